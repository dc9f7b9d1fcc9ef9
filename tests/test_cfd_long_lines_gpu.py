"""Compact-FD lines longer than a shared-memory tile of 32 lines: z tiles of 16 and 8
lines (the last one ragged, nz that allows bulk copies and not), the longest that
take 32, and x / y lines around the length at which the streamed kernel takes over.
Likewise the lines at which a tile goes from four warps to eight: 316 and 336 points
with plain copies, 416 and 448 with asynchronous ones.  Up to 1815 points the z solve that carries the epilogue (kernel_variant 9) fits and
gives the same bits, as does the streamed kernel (5) for x / y lines; longer z lines
are within twice the FP32 oracle's distance from the FP64 one (rounding grows some
hundred times in the band solves, whose symbol falls to 3e-5 at the Nyquist
wavenumber)."""
import numpy as np
import pytest

from konglong_b200.propagator import Propagator
from konglong_b200.spec import ENGINE_CFD, FIELD_W1, VTI
from oracle import pyoracle as O
from tests.conftest import rel_l2
from tests.golden_inputs import case_inputs

pytestmark = pytest.mark.gpu


def _two_steps(x, model, w0, w1):
    x.set_model(**model)
    x.put(0, w0)
    x.put(1, w1)
    for _ in range(2):
        x.kernel()
        x.update2nd()
        x.swap()
    return np.array(x.get(FIELD_W1))


def _variant(spec, model, w0, w1, variant):
    spec.kernel_variant = variant
    p = Propagator(spec)
    out = _two_steps(p, model, w0, w1)
    p.close()
    return out


@pytest.mark.parametrize("shape, other", [
    ((316, 17, 33), 5), ((336, 16, 33), 5), ((17, 331, 37), 5), ((17, 16, 315), 9), ((17, 16, 333), 9),
    ((416, 16, 36), 5), ((448, 17, 36), 5), ((16, 444, 40), 5), ((17, 17, 416), 9), ((17, 17, 448), 9),
    ((17, 17, 1764), 9), ((17, 17, 1784), 9), ((17, 17, 1792), 9), ((19, 17, 1813), 9),
    ((1780, 16, 36), 5), ((1781, 16, 33), 5), ((1796, 16, 36), 5), ((1900, 16, 33), 5), ((16, 1780, 36), 5), ((16, 1900, 36), 5)])
def test_long_lines_equal_other_forms(shape, other):
    spec, m, w0, w1 = case_inputs(dict(engine=ENGINE_CFD, model=VTI, shape=shape, pml=6, seed=7))
    want = _variant(spec, m, w0, w1, other)
    assert np.abs(want).max() > 0
    for variant in (0, 1):
        np.testing.assert_array_equal(_variant(spec, m, w0, w1, variant), want)


@pytest.mark.parametrize("nz", [3600, 3601])
def test_longer_z_lines_match_oracle(nz):
    spec, m, w0, w1 = case_inputs(dict(engine=ENGINE_CFD, model=VTI, shape=(17, 17, nz), pml=6, seed=8))
    exact = _two_steps(O.Oracle(spec, double=True), m, w0, w1)
    spread = rel_l2(_two_steps(O.Oracle(spec), m, w0, w1), exact)
    assert 0 < spread < 1e-3
    assert rel_l2(_variant(spec, m, w0, w1, 0), exact) < 2 * spread + 1e-6
