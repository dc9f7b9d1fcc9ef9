"""Batches of tiny shots, whose steps are shared launches over all shots' tiles:
every shot's own rtm_modelling bit for bit (one-cell kernels, which every FD8 kernel
equals), receivers to the rounding of a 20^3-tap sum.  Extents below, at and above a
tile (32 z, 8 x) and a y segment (8), shots that end at different steps, shots with
and without grouped receivers, none at all, and several sources."""
import numpy as np
import pytest

from konglong_b200 import workloads as W
from konglong_b200.propagator import Batch, Propagator, spread_coeffs
from konglong_b200.spec import FIELD_W0, FIELD_W1, ISO, TTI, VTI
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


def _shots(model, n):
    shots = W.small_shots(nshots=n, seed=5, size=(24, 41), steps=(9, 24), nrec=3, model=VTI if model != ISO else ISO)
    for k, sh in enumerate(shots):
        s = sh.spec
        s.nbnd = ((4 + k % 3,) * 6)
        if model == TTI:
            rng = np.random.default_rng(k)
            t = np.deg2rad(W.minmax(W.smooth_field(s.shape, 3.0, rng), 0.0, 30.0))
            s.model_type, sh.pjx, sh.pjy = TTI, (-np.sin(t)).astype(np.float32), 0 * sh.vel
            s.dt *= 0.7
            sh.wavelet = W.ricker(sh.fpeak, s.dt, sh.nt)
    return shots


def _handle(shot, k):
    s = shot.spec
    p = Propagator(s)
    p.set_model(**shot.model_arrays())
    k1, k2 = W.spread_band(s)
    at = [shot.src_pos] + [(6.0 + 3 * j, s.ny / 2, s.nz / 2) for j in range(k % 3)]
    src = W.make_traceset(at, s.nx, s.ny, s.nz, 10, k1, k2, spread_coeffs)
    p.set_injection(src, np.tile(shot.wavelet, (len(at), 1)), s.dt_dxyz)
    if k % 5 != 4:
        pos = shot.rcv_pos if k % 2 else np.repeat(shot.rcv_pos, 3, 0)
        p.set_extraction(W.make_traceset(pos, s.nx, s.ny, s.nz, 10, k1, k2, spread_coeffs), shot.nt)
    p.reset()
    return p


@pytest.mark.parametrize("model", [ISO, VTI, TTI])
@pytest.mark.parametrize("n", [1, 40])
def test_shared_steps_equal_own(model, n):
    shots = _shots(model, n)
    want = []
    for k, sh in enumerate(shots):
        p = _handle(sh, k)
        p.modelling(sh.nt, -1, 2)
        want.append((p.get(FIELD_W1), p.get(FIELD_W0), p.traces() if k % 5 != 4 else None))
        p.close()
    ps = [_handle(sh, k) for k, sh in enumerate(shots)]
    b = Batch(ps)
    b.modelling([sh.nt for sh in shots], -1, 2)
    for k, (p, (w1, w0, tr)) in enumerate(zip(ps, want)):
        assert np.abs(w1).max() > 0
        # sources that overlap are added in either order: a rounding of 6e-8 for each of up to 3 a step
        same = (lambda a, b: np.testing.assert_array_equal(a, b)) if k % 3 == 0 else \
            (lambda a, b: np.testing.assert_array_less(rel_l2(a, b), 24 * 3 * 6e-8))
        same(p.get(FIELD_W1), w1)
        same(p.get(FIELD_W0), w0)
        if tr is not None:
            assert rel_l2(p.traces(), tr) < 1e-5
    b.close()


@pytest.mark.parametrize("model", [ISO, VTI])
def test_own_kernels_give_the_same_traces(model):
    """Shots stepped by their own kernels record by their own kernels: equal traces."""
    shots = W.small_shots(nshots=2, seed=9, size=(72, 90), steps=(12, 20), nrec=5, model=model)
    want = []
    for sh in shots:
        p = _handle(sh, 1)
        p.modelling(sh.nt, -1, 1)
        want.append((p.traces(), p.get(FIELD_W1)))
        p.close()
    ps = [_handle(sh, 1) for sh in shots]
    b = Batch(ps)
    b.modelling([sh.nt for sh in shots], -1, 1)
    for p, (tr, w1) in zip(ps, want):
        assert np.abs(tr).max() > 0
        np.testing.assert_array_equal(p.traces(), tr)
        np.testing.assert_array_equal(p.get(FIELD_W1), w1)
    b.close()
