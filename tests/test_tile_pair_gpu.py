"""PML tiles and interior tiles of a pass run side by side, the interior tiles
let in when the PML tiles have all started.  Loops of steps launched back to
back, with many interior tiles to few PML tiles, the other way round, and only
one kind, equal the one-cell kernels, one launch a pass after the other, bit
for bit."""
import numpy as np
import pytest

from konglong_b200 import workloads as W
from konglong_b200.propagator import Propagator, spread_coeffs
from konglong_b200.spec import FIELD_W0, FIELD_W1, ISO, TTI, VTI, PropSpec

pytestmark = pytest.mark.gpu

STEPS = 24


@pytest.mark.parametrize("model", [ISO, VTI, TTI])
@pytest.mark.parametrize("shape,widths", [
    ((160, 96, 132), (0, 0, 3, 3, 0, 0)),         # interior columns, thin PML ends
    ((160, 96, 132), (40, 40, 10, 10, 32, 32)),   # mostly PML tiles
    ((64, 40, 64), (16, 16, 8, 8, 24, 24)),       # PML tiles alone
    ((72, 40, 96), (0, 0, 0, 0, 0, 0)),           # interior tiles alone
    ((40, 200, 96), (0, 9, 0, 9, 0, 9))])         # one interior column, long in y
def test_loop_equals_one_cell_kernels(model, shape, widths):
    nx, ny, nz = shape
    rng = np.random.default_rng(nx + nz + model)
    fields = []
    for variant in (0, 1):
        s = PropSpec(nx=nx, ny=ny, nz=nz, model_type=model, nbnd=widths, dt=0.0006, kernel_variant=variant)
        if not fields:
            m = dict(vel=rng.uniform(1500, 4500, s.shape).astype(np.float32))
            if model != ISO:
                m.update(eps=rng.uniform(0, 0.25, s.shape).astype(np.float32),
                         dl=rng.uniform(0, 0.1, s.shape).astype(np.float32))
            if model == TTI:
                th, ph = rng.uniform(0, 0.7, s.shape), rng.uniform(0, 6.28, s.shape)
                m.update(pjx=(-np.sin(th) * np.cos(ph)).astype(np.float32),
                         pjy=(-np.sin(th) * np.sin(ph)).astype(np.float32))
            w = [rng.standard_normal(s.n).astype(np.float32) for _ in range(2)]
        p = Propagator(s)
        p.set_model(**m)
        p.reset()
        p.put(FIELD_W0, w[0])
        p.put(FIELD_W1, w[1])
        # a point source of one sample keeps the step's other launches in the loop
        k1, k2 = W.spread_band(s)
        src = W.make_traceset([(nx / 2, ny / 2, nz / 2)], nx, ny, nz, 10, k1, k2, spread_coeffs)
        p.set_injection(src, np.ones((1, STEPS), np.float32), s.dt_dxyz)
        p.modelling(STEPS)
        fields.append((p.get(FIELD_W0), p.get(FIELD_W1)))
        p.close()
    for a, b in zip(*fields):
        assert np.isfinite(a).all() and np.abs(a).max() > 0
        np.testing.assert_array_equal(a, b)
