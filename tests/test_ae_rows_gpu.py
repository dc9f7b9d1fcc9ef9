"""The volume codec takes 16 blocks as the rows of its MMAs and cells as 16-byte
words where the volume allows it.  Block counts around multiples of 16, extents
that are no multiples of 8 or 4, buffers off 16-byte boundaries, and blocks of
tiny, huge and zero scale give the bits of the layer-by-layer path."""
import numpy as np
import pytest

from konglong_b200 import compressor as AE
from oracle import ae_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [0, 1])  # elements the device buffers are shifted by
@pytest.mark.parametrize("shape", [(1, 1, 1), (8, 8, 8), (8, 16, 64), (8, 8, 136), (24, 40, 72), (17, 9, 30), (40, 33, 52)])
def test_codec_rows(shape, off):
    import torch
    from konglong_b200 import _lib
    L = _lib.lib()
    rng = np.random.default_rng(sum(shape))
    ny, nx, nz = shape
    w = rng.standard_normal(shape).astype(np.float32)
    # quotients by a power of two that lie on, and next to, a tie of the BF16 rounding
    flat = w.reshape(-1)
    half = np.arange(flat.size) % 7 == 0
    bits = (flat.view(np.uint32) & np.uint32(0xffff0000)) | np.uint32(0x7ffe) + rng.integers(0, 5, flat.size).astype(np.uint32)
    flat[half] = bits.view(np.float32)[half]
    for z0, s in ((0, 1.0), (8, 4e-38), (16, 1e37), (24, 0.0), (32, 1e-44), (40, 3e-30)):
        w[:, :, z0:z0 + 8] *= np.float32(s)
    ae = AE.AutoEncoder(seed=5)
    b, sc = AE.volume_to_blocks(w)
    rec, lat = ae.reconstruct(b)
    nb = b.shape[0]

    def dev(n, dt):
        return torch.zeros(n + off, device="cuda", dtype=dt)[off:]

    dv, out = dev(w.size, torch.float32), dev(w.size, torch.float32)
    dv.copy_(torch.from_numpy(w).reshape(-1))
    dl, ds = dev(nb * AE.LATENT, torch.bfloat16), dev(nb, torch.float32)
    _lib.check(L.rtm_ae_compress_volume(ae.a, dv.data_ptr(), nx, ny, nz, dl.data_ptr(), ds.data_ptr(), None),
               "rtm_ae_compress_volume")
    _lib.check(L.rtm_ae_decompress_volume(ae.a, dl.data_ptr(), ds.data_ptr(), nx, ny, nz, out.data_ptr(), None),
               "rtm_ae_decompress_volume")
    torch.cuda.synchronize()
    np.testing.assert_array_equal(ds.cpu().numpy(), sc)
    np.testing.assert_array_equal(dl.float().cpu().numpy().reshape(nb, AE.LATENT), O.bf16(lat).astype(np.float32))
    np.testing.assert_array_equal(out.cpu().numpy().reshape(shape), AE.blocks_to_volume(rec, sc, shape))
    ae.close()
