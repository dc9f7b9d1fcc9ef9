"""Threads of the compact-FD tile kernels: 128 while four or more tiles (five with
plain copies) fit an SM, 256 beyond, on either side of each line.  Counted on the
fake runtime; the speeds are beside the rule."""
import pytest

from tests.fake_cuda import fake_cuda  # noqa: F401

# points, whether nz % 4 == 0 (asynchronous copies), threads
LINES = [(256, True, 128), (400, True, 128), (416, True, 128), (448, True, 256), (512, True, 256),
         (255, False, 128), (313, False, 128), (341, False, 256), (513, False, 256)]


@pytest.mark.parametrize("axis", ["x", "y", "z"])
def test_threads_of_a_tile(fake_cuda, axis):  # noqa: F811
    fake_cuda("""
    for n, whole, want in %r:
        nz = 40 if whole else 37
        nx, ny, nz = {"x": (n, 24, nz), "y": (24, n, nz), "z": (24, 24, n)}[%r]
        p = Propagator(S.PropSpec(nx=nx, ny=ny, nz=nz, engine=S.ENGINE_CFD, model_type=S.ISO, nbnd=(6,) * 6))
        p.set_model(vel=np.full((ny, nx, nz), 2000, np.float32))
        p.reset()
        fake.fake_clear()
        p.modelling(1)
        assert launched("cfd_tile_k") == 6  # two passes, three axes
        other = launched("epi_k")           # 256 threads each
        tiles = launched("[128]"), launched("[256]") - other
        assert tiles == ((6, 0) if want == 128 else (4, 2)), (n, whole, tiles)
        p.close()
    """ % (LINES, axis))
