"""PML widths that are not whole float4s: the 4-cell FD8 kernels read z faces
padded with undamped layers.  Operator steps against the FP32 oracle (which has
no padding) for odd widths, uneven sides, a face on one side only and widths
whose padded faces would not fit the grid, with and without cross terms."""
import numpy as np
import pytest

from konglong_b200.propagator import Propagator
from konglong_b200.spec import ENGINE_CFD, ENGINE_R2R, FIELD_W0, FIELD_W1, ISO, TTI, VTI, PropSpec
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


@pytest.mark.parametrize("engine", [ENGINE_CFD, ENGINE_R2R])
@pytest.mark.parametrize("model", [ISO, VTI, TTI])
@pytest.mark.parametrize("shape,widths", [((40, 26, 52), (5, 7, 6, 9, 5, 7)), ((34, 22, 50), (5, 7, 0, 9, 3, 10)),
                                          ((36, 20, 44), (6, 6, 6, 6, 22, 21)), ((44, 1, 48), (6, 6, 0, 0, 6, 6))])
def test_line_engine_epilogues_at_odd_widths(engine, model, shape, widths):
    """The pointwise epilogues of the line-derivative engines: nz a multiple of 4 and not, faces
    on one side, faces that pad and that do not, and a 2-D grid."""
    nx, ny, nz = shape
    s = PropSpec(nx=nx, ny=ny, nz=nz, engine=engine, model_type=model, nbnd=widths, dt=0.0005)
    rng = np.random.default_rng(nz + model)
    m = dict(vel=rng.uniform(1500, 4500, s.shape).astype(np.float32))
    if model != ISO:
        m.update(eps=rng.uniform(0, 0.25, s.shape).astype(np.float32), dl=rng.uniform(0, 0.1, s.shape).astype(np.float32))
    if model == TTI:
        th, ph = rng.uniform(0, 0.7, s.shape), rng.uniform(0, 6.28, s.shape)
        m.update(pjx=(-np.sin(th) * np.cos(ph)).astype(np.float32), pjy=(-np.sin(th) * np.sin(ph)).astype(np.float32))
    w = [rng.standard_normal(s.n).astype(np.float32) for _ in range(2)]
    out = []
    for x in (Propagator(s), O.Oracle(s), O.Oracle(s, double=True)):
        x.set_model(**m)
        x.reset()
        x.put(FIELD_W0, w[0])
        x.put(FIELD_W1, w[1])
        for _ in range(2):
            x.kernel()
            x.update2nd()
            x.swap()
        out.append(x.get(FIELD_W1))
    # transform lines: the bound of the operator parity tests; compact FD: its FP32 band solve
    # amplifies rounding, so twice the FP32 oracle's own distance from FP64
    bound = 1e-5 if engine == ENGINE_R2R else 2 * rel_l2(out[1], out[2])
    assert rel_l2(out[0], out[2]) < bound, (rel_l2(out[0], out[2]), bound)
