"""Shot after shot in one handle: the trace tables and snapshot slots of the shot
before are taken again where they fit.  A handle that has held another shot's
tables must give what a fresh one gives."""
import numpy as np
import pytest

from konglong_b200 import workloads as W
from konglong_b200.propagator import Propagator, spread_coeffs
from konglong_b200.spec import ISO, SNAP_C16, SNAP_FP32
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

NT = 24


def _shot():
    return W.small_shots(nshots=1, seed=5, size=(36, 44), steps=(NT, NT + 1), nrec=4, model=ISO)[0]


def _handle(shot):
    p = Propagator(shot.spec)
    p.set_model(**shot.model_arrays())
    return p


def _receivers(shot, n, seed):
    """n receivers at one depth (one grouped z kernel from 16 on)."""
    s = shot.spec
    rng = np.random.default_rng(seed)
    pos = [(rng.uniform(6, s.nx - 7), rng.uniform(6, s.ny - 7), 9.3) for _ in range(n)]
    k1, k2 = W.spread_band(s)
    ts = W.make_traceset(pos, s.nx, s.ny, s.nz, 10, k1, k2, spread_coeffs)
    return ts, rng.standard_normal((n, NT)).astype(np.float32)


def _rtm(p, shot, nrec, fmt):
    src, _ = _receivers(shot, 1, 1)
    rcv, tr = _receivers(shot, nrec, 2 + nrec)
    image, _, _ = p.rtm_shot(src, shot.wavelet[None, :NT], rcv, tr, NT, NT, 4, snap_fmt=fmt)
    return image


@pytest.mark.parametrize("before, then", [(120, 100), (100, 120), (120, 2), (3, 17), (1, 1)])
@pytest.mark.parametrize("fmts", [(SNAP_FP32, SNAP_FP32), (SNAP_FP32, SNAP_C16)])
def test_second_shot_equals_fresh_handle(before, then, fmts):
    shot = _shot()
    fresh = _handle(shot)
    want = _rtm(fresh, shot, then, fmts[1])
    fresh.close()
    p = _handle(shot)
    _rtm(p, shot, before, fmts[0])
    got = _rtm(p, shot, then, fmts[1])
    # the same kernels; atomic adds of overlapping kernels may order differently:
    # a few roundings of 6e-8 an injected value
    assert np.abs(want).max() > 0
    assert rel_l2(got, want) < 1e-5
    # extraction tables: set, replaced by a smaller and a larger set, zeroed each time
    for n in (30, 20, 60):
        p.set_extraction(_receivers(shot, n, n)[0], NT)
        t = p.traces()
        assert t.shape == (n, NT) and not t.any()
    p.close()
