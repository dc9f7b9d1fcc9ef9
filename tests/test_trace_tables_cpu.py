"""Trace tables that do not fit the host's memory: an error, an empty set and a
handle that goes on, not an exception through the C interface.  On the fake runtime,
with the address space capped so that the tables' 1.5 GB cannot be had."""
import pytest

from tests.fake_cuda import fake_cuda  # noqa: F401


@pytest.mark.parametrize("call", ["injection", "extraction"])
def test_tables_beyond_host_memory(fake_cuda, call):  # noqa: F811
    out = fake_cuda("""
    import resource
    shot = W.small_shots(nshots=1, seed=3, size=(36, 40), steps=(12, 12), nrec=3)[0]
    shot.spec.nbnd = (8,) * 6
    p = handle(shot)
    n, lx = 1000, 400000  # taps padded to a long stride
    big = S.TraceSet(n, lx, 1, 1, np.ones((n, 3), np.int32), np.ones((n, 3), np.int32), np.zeros((n, lx), np.float32),
                     np.ones((n, 1), np.float32), np.ones((n, 1), np.float32))
    used = int(open("/proc/self/statm").read().split()[0]) * resource.getpagesize()
    resource.setrlimit(resource.RLIMIT_AS, (used + (512 << 20),) * 2)
    try:
        p.set_injection(big, np.ones((n, 12), np.float32), 1.0) if %r == "injection" else p.set_extraction(big, 12)
        raise SystemExit("no error")
    except RtmError as e:
        assert e.code == STATUS_CODE["RTM_ERR_NOMEM"], e
        print(e)
    p.modelling(4)
    assert launched(%r) == 0
    """ % (call, "inject" if call == "injection" else "extract"))
    assert "RTM_ERR_NOMEM" in out
