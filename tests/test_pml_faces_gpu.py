"""PML widths that are not whole float4s: the 4-cell FD8 kernels read z faces
padded with undamped layers.  Operator steps against the FP32 oracle (which has
no padding) for odd widths, uneven sides, a face on one side only and widths
whose padded faces would not fit the grid, with and without cross terms."""
import numpy as np
import pytest

from konglong_b200.propagator import Propagator
from konglong_b200.spec import FIELD_W0, FIELD_W1, ISO, TTI, VTI, PropSpec
from oracle import pyoracle as O
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("model", [ISO, VTI, TTI])
@pytest.mark.parametrize("nz,widths,pml3d", [
    (52, (5, 7, 6, 9, 5, 7), True), (52, (5, 7, 6, 9, 3, 10), False), (44, (4, 0, 0, 3, 22, 22), True),
    (44, (6, 6, 6, 6, 21, 21), True), (60, (2, 2, 2, 2, 0, 13), True), (60, (9, 9, 9, 9, 6, 0), False)])
def test_odd_pml_widths_match_oracle(model, nz, widths, pml3d):
    nx, ny = 41, 26
    s = PropSpec(nx=nx, ny=ny, nz=nz, model_type=model, nbnd=widths, pml3d=pml3d, dt=0.0007)
    rng = np.random.default_rng(nz + model)
    m = dict(vel=rng.uniform(1500, 4500, s.shape).astype(np.float32))
    if model != ISO:
        m.update(eps=rng.uniform(0, 0.25, s.shape).astype(np.float32), dl=rng.uniform(0, 0.1, s.shape).astype(np.float32))
    if model == TTI:
        th, ph = rng.uniform(0, 0.7, s.shape), rng.uniform(0, 6.28, s.shape)
        m.update(pjx=(-np.sin(th) * np.cos(ph)).astype(np.float32), pjy=(-np.sin(th) * np.sin(ph)).astype(np.float32))
    w = [rng.standard_normal(s.n).astype(np.float32) for _ in range(2)]
    out = []
    for x in (Propagator(s), O.Oracle(s)):
        x.set_model(**m)
        x.reset()
        x.put(FIELD_W0, w[0])
        x.put(FIELD_W1, w[1])
        for _ in range(3):  # the memory of both rounds is written and read back
            x.kernel()
            x.update2nd()
            x.swap()
        out.append(x.get(FIELD_W1))
    # FP32 stencils and recursions against FP32: the bound of the operator parity tests
    assert rel_l2(out[0], out[1]) < 2e-6, rel_l2(out[0], out[1])
