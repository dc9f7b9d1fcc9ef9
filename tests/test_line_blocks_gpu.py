"""Tensor-core line operators at the edges of their column blocks and stages:
line lengths around one, two and three blocks of 128 columns, an odd number of
8-point K blocks, fewer K blocks than stages, tiles of 128 lines cut short and
tiles that run over several y planes, against the FP32 cuBLAS line products."""
import numpy as np
import pytest

from konglong_b200.propagator import Propagator
from konglong_b200.spec import ENGINE_R2C, ENGINE_R2R, FIELD_W1, VTI
from tests.conftest import rel_l2
from tests.golden_inputs import case_inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("engine", [ENGINE_R2R, ENGINE_R2C])
@pytest.mark.parametrize("shape", [(128, 20, 36), (130, 20, 28), (20, 258, 28), (24, 384, 28), (386, 20, 28),
                                   (20, 24, 128), (20, 24, 132), (64, 66, 64), (20, 20, 24)])
def test_line_lengths_around_the_blocks(engine, shape):
    c = dict(engine=engine, model=VTI, shape=shape, pml=6, seed=sum(shape))
    spec, m, w0, w1 = case_inputs(c)
    out = {}
    for variant in (0, 1):
        spec.kernel_variant = variant
        p = Propagator(spec)
        p.set_model(**m)
        p.put(0, w0)
        p.put(1, w1)
        for _ in range(2):
            p.kernel()
            p.update2nd()
            p.swap()
        out[variant] = p.get(FIELD_W1)
        p.close()
    assert np.abs(out[1]).max() > 0
    # both FP32-accurate products: the bound of the line-operator tests
    assert rel_l2(out[0], out[1]) < 2e-6, rel_l2(out[0], out[1])
