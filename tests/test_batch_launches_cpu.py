"""How a batch of small shots is launched.  The host submits a kernel in about 2 us,
so the steps of many tiny shots have to be shared launches; larger shots run their
own, faster kernels.  Counted on the fake runtime."""
import pytest

from tests.fake_cuda import fake_cuda  # noqa: F401


@pytest.mark.parametrize("model, nshots, size, nrec, shared", [
    ("ISO", 64, (28, 40), 6, True), ("ISO", 8, (28, 40), 6, True), ("ISO", 12, (96, 104), 4, False),
    ("VTI", 64, (28, 40), 6, True), ("VTI", 32, (60, 64), 4, False), ("TTI", 64, (28, 40), 1, True)])
def test_launches_of_a_batched_step(fake_cuda, model, nshots, size, nrec, shared):  # noqa: F811
    fake_cuda("""
    shots = W.small_shots(nshots=%d, seed=3, size=%r, steps=(10, 10), nrec=%d, model=S.VTI if %r != "ISO" else S.ISO)
    for sh in shots:
        sh.spec.nbnd = (8,) * 6
        if %r == "TTI":
            sh.spec.model_type, sh.pjx, sh.pjy = S.TTI, 0 * sh.vel, 0 * sh.vel
    ps = [handle(sh) for sh in shots]
    b = Batch(ps)
    fake.fake_clear()
    b.modelling([10] * len(ps))
    n, shared = launched() / 10, launched("_batch")
    assert in_flight() == 0
    if %r:
        assert n <= 4 and shared, n
    else:
        assert not shared and n >= 4 * len(ps), n
    """ % (nshots, size, nrec, model, model, shared))
