"""A time loop whose launch, copy or allocation fails: the call returns the first
error with its text, nothing that it submitted is still in flight, and the handles
answer the next call for themselves.  On the fake runtime."""
import pytest

from tests.fake_cuda import fake_cuda  # noqa: F401

SHOT = """
shot = W.small_shots(nshots=1, seed=3, size=(36, 40), steps=(12, 12), nrec=3)[0]
shot.spec.nbnd = (8,) * 6


def code(f, *a):
    try:
        f(*a)
    except RtmError as e:
        return e.code, str(e)
    return 0, ""
"""


@pytest.mark.parametrize("what", ["launch iso_fd8", "launch inject", "launch extract"])
def test_modelling_waits_for_what_it_submitted(fake_cuda, what):  # noqa: F811
    fake_cuda(SHOT + """
p = handle(shot)
p.modelling(2)
before = p.last_loop_ms
fail(%r, 5)
rc, text = code(p.modelling, 12)
assert rc == STATUS_CODE["RTM_ERR_NOMEM"] and "fake error" in text, text
assert in_flight() == 0
assert p.last_loop_ms != before
assert code(p.modelling, 2) == (0, "")
""" % what)


@pytest.mark.parametrize("dir", ["forward", "backward"])
def test_migration_joins_its_snapshot_copies(fake_cuda, dir):  # noqa: F811
    fake_cuda(SHOT + """
p = handle(shot, receivers=False)
p.snapshot_setup(S.SNAP_C16, 12)
p.snapshot_offload(3)
p.image_setup(0, 0, 1)
forward = %r == "forward"
if not forward:
    p.migration(S.FORWARD, 0, 12, -1, 1)
fail("launch iso_fd8", 7)
rc, text = code(p.migration, S.FORWARD, 0, 12, -1, 1) if forward else code(p.migration, S.BACKWARD, 11, -1, -1, 1)
assert rc == STATUS_CODE["RTM_ERR_NOMEM"] and "iso_fd8" in text, text
assert in_flight() == 0
fail("cudaMemcpyAsync", 4)
rc, text = code(p.migration, S.FORWARD, 0, 12, -1, 1)
assert rc == STATUS_CODE["RTM_ERR_NOMEM"], text
assert in_flight() == 0
""" % dir)


@pytest.mark.parametrize("nshots, size, what", [
    (3, (72, 80), "launch iso_fd8"), (3, (72, 80), "launch inject_scatter"), (3, (72, 80), "launch extract"),
    (40, (28, 32), "launch iso_fd8"), (40, (28, 32), "launch batch_inject"), (40, (28, 32), "cudaMemcpyAsync")])
def test_batch_waits_for_every_shot(fake_cuda, nshots, size, what):  # noqa: F811
    fake_cuda(SHOT + """
shots = W.small_shots(nshots=%d, seed=3, size=%r, steps=(10, 10), nrec=3)
for sh in shots:
    sh.spec.nbnd = (8,) * 6
ps = [handle(sh) for sh in shots]
b = Batch(ps)
fail(%r, 1)
rc, _ = code(b.modelling, [10] * len(ps))
assert rc == STATUS_CODE["RTM_ERR_NOMEM"]
assert in_flight() == 0
assert any(b"fake error" in p.L.rtm_last_error(p.h) for p in ps)
assert code(b.modelling, [10] * len(ps)) == (0, "")
assert in_flight() == 0
""" % (nshots, size, what))


@pytest.mark.parametrize("nshots, size", [(3, (72, 80)), (40, (28, 32))])
def test_batch_takes_every_timeout_flag(fake_cuda, nshots, size):  # noqa: F811
    fake_cuda(SHOT + """
shots = W.small_shots(nshots=%d, seed=3, size=%r, steps=(4, 4), nrec=3)
for sh in shots:
    sh.spec.nbnd = (8,) * 6
ps = [handle(sh) for sh in shots]
b = Batch(ps)
fake.fake_set_flags(1)
rc, _ = code(b.modelling, [4] * len(ps))
shared = launched("_batch") > 0
assert shared == (len(ps) == 40)
if not shared:  # their kernels wait for copies, the shared ones do not
    assert rc == STATUS_CODE["RTM_ERR_TIMEOUT"]
    for p in ps:  # the flag of the batch is not left for the shot's next call
        assert code(p.modelling, 0) == (0, ""), p
    assert code(b.modelling, [4] * len(ps)) == (0, "")
""" % (nshots, size))
