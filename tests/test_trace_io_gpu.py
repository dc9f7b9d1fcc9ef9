"""Injection and extraction kernels at the sizes where their indexing can go
wrong: x / y kernels of one tap, of lengths around the eight-column and
32-lane strides, z kernels that are not a multiple of the lanes sharing a
column, member counts around the staging chunk, grids that cut the xy tiles,
and non-finite samples that must stay inside their own box.  Checked against
float64 sums of the same taps."""
import numpy as np
import pytest

from konglong_b200.propagator import Propagator
from konglong_b200.spec import FIELD_VEL, FIELD_W0, PropSpec, TraceSet

pytestmark = pytest.mark.gpu

NX, NY, NZ = 75, 53, 47


def _set(rng, ntr, lx, ly, lz, grouped):
    """ntr traces with boxes of up to lx * ly * lz taps; grouped: one z kernel for all."""
    ln = np.stack([rng.integers(max(1, lx - 2), lx + 1, ntr), rng.integers(max(1, ly - 2), ly + 1, ntr),
                   np.full(ntr, lz)], 1).astype(np.int32)
    off = np.stack([rng.integers(0, NX - ln[:, 0] + 1), rng.integers(0, NY - ln[:, 1] + 1),
                    np.full(ntr, 5) if grouped else rng.integers(0, NZ - lz + 1, ntr)], 1).astype(np.int32)
    off[0, :2] = 0                                   # the grid's corners
    off[-1, :2] = NX - ln[-1, 0], NY - ln[-1, 1]
    k = [rng.standard_normal((ntr, n)).astype(np.float32) for n in (lx, ly, lz)]
    if grouped:
        k[2][:] = k[2][0]
    return TraceSet(ntr, lx, ly, lz, off, ln, *k)


def _box(ts, r):
    o, n = ts.off[r], ts.len[r]
    sl = tuple(slice(o[a], o[a] + n[a]) for a in (1, 0, 2))
    taps = np.einsum("y,x,z->yxz", *(k[r, :n[a]].astype(np.float64) for a, k in ((1, ts.ky), (0, ts.kx), (2, ts.kz))))
    return sl, taps


@pytest.fixture(scope="module")
def engine():
    p = Propagator(PropSpec(nx=NX, ny=NY, nz=NZ, nbnd=(6,) * 6))
    rng = np.random.default_rng(1)
    p.set_model(vel=rng.uniform(1500, 4000, (NY, NX, NZ)).astype(np.float32))
    yield p
    p.close()


@pytest.mark.parametrize("ntr,lx,ly,lz,grouped", [
    (40, 20, 20, 20, True), (33, 1, 1, 1, True), (64, 3, 40, 7, True), (31, 33, 2, 31, True), (97, 8, 9, 42, True),
    (12, 20, 20, 20, False), (9, 1, 1, 1, False), (7, 3, 5, 21, False), (5, 7, 33, 3, False), (5, 40, 2, 42, False)])
def test_injection_and_extraction_sums(engine, ntr, lx, ly, lz, grouped):
    p, rng = engine, np.random.default_rng(ntr * 1000 + lx)
    ts = _set(rng, ntr, lx, ly, lz, grouped)
    w = rng.standard_normal((NY, NX, NZ)).astype(np.float32)
    # extraction: a warp sums at most taps / 32 + 1 products per lane one after the other, then 5 adds
    p.set_extraction(ts, 1)
    p.put(FIELD_W0, w)
    p.extract(0)
    got = p.traces()[:, 0]
    for r in range(ntr):
        sl, taps = _box(ts, r)
        terms = taps * w[sl]
        bound = (terms.size / 32 + 40) * 2.0 ** -24 * np.abs(terms).sum()
        assert abs(got[r] - terms.sum()) <= bound, (r, got[r], terms.sum())
    # injection: each cell sums its members in order
    tr = rng.standard_normal((ntr, 1)).astype(np.float32)
    p.set_injection(ts, tr, 2.0)
    p.put(FIELD_W0, w)
    p.inject(0)
    vel = p.get(FIELD_VEL).reshape(w.shape).astype(np.float64)
    add, mag = np.zeros(w.shape), np.abs(w).astype(np.float64)
    for r in range(ntr):
        sl, taps = _box(ts, r)
        add[sl] += 2.0 * float(tr[r, 0]) * taps * vel[sl]
        mag[sl] += np.abs(2.0 * float(tr[r, 0]) * taps * vel[sl])
    err = np.abs(p.get(FIELD_W0).reshape(w.shape) - (w + add))
    assert np.all(err <= (ntr + 8) * 2.0 ** -24 * mag)


def test_non_finite_sample_stays_in_its_box(engine):
    p, rng = engine, np.random.default_rng(5)
    ts = _set(rng, 40, 9, 6, 11, True)
    tr = rng.standard_normal((40, 1)).astype(np.float32)
    tr[17] = np.inf
    p.set_injection(ts, tr, 1.0)
    p.put(FIELD_W0, np.zeros((NY, NX, NZ), np.float32))
    p.inject(0)
    bad = ~np.isfinite(p.get(FIELD_W0).reshape(NY, NX, NZ))
    sl, _ = _box(ts, 17)
    inside = np.zeros(bad.shape, bool)
    inside[sl] = True
    assert bad.any() and not (bad & ~inside).any()
