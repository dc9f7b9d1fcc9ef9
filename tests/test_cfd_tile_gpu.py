"""Compact-FD tile line solves (kernel_variant 0 / 1 / 2) at the line lengths
where their chunks, quads, runs and boxes end: the smallest lines, remainders of
4 and 8 rows, lines without a constant run of factors, one and two TMA boxes,
four and eight warps, ragged z tiles, nz that allows bulk copies and not.  The
x / y lines are compared bit for bit with the register-streamed kernel
(variant 5), the z lines with the z solve that carries the epilogue (variant 9)."""
import numpy as np
import pytest

from konglong_b200.propagator import Propagator
from konglong_b200.spec import ENGINE_CFD, FIELD_W0, FIELD_W1, VTI
from tests.golden_inputs import case_inputs

pytestmark = pytest.mark.gpu


def _steps(spec, m, w0, w1, variant):
    spec.kernel_variant = variant
    p = Propagator(spec)
    p.set_model(**m)
    p.put(0, w0)
    p.put(1, w1)
    for _ in range(2):
        p.kernel()
        p.update2nd()
        p.swap()
    out = p.get(FIELD_W0), p.get(FIELD_W1)
    p.close()
    return out


@pytest.mark.parametrize("shape", [(16, 17, 20), (19, 16, 33), (36, 29, 36), (95, 33, 64), (100, 18, 97), (130, 20, 132),
                                   (257, 16, 251), (250, 16, 260), (20, 516, 36), (16, 18, 514)])
def test_tile_lines_equal_other_forms(shape):
    spec, m, w0, w1 = case_inputs(dict(engine=ENGINE_CFD, model=VTI, shape=shape, pml=6, seed=shape[0]))
    want = _steps(spec, m, w0, w1, 5)
    assert np.abs(want[1]).max() > 0
    for variant in (0, 1, 2, 9):
        for a, b in zip(_steps(spec, m, w0, w1, variant), want):
            np.testing.assert_array_equal(a, b)
