"""cbm_pfpc_sums_noalloc at the edges of its split: every reduction width, one pair
row a column and more than a round of them, buffers aligned to 16 bytes and not,
bit for bit against the reference's order of the sums in numpy float32."""
import numpy as np
import pytest

from test_zz_no_alloc import _entry, _last_error

pytestmark = pytest.mark.gpu


def reference(ap, mask, w, pcs):
    n = ap.size // pcs
    bs = 512 if n >= 2048 else 128 if n >= 512 else 32 if n >= 128 else 8 if n >= 32 else 2
    x = (w * ((ap & mask) > 0).astype(np.float32)).reshape(pcs, n // (2 * bs), 2, bs)
    s = np.zeros((pcs, bs), np.float32)
    for k in range(x.shape[1]):  # the running sum over the pairs
        s = s + (x[:, k, 0] + x[:, k, 1])
    while s.shape[1] > 1:  # the halving tree
        h = s.shape[1] // 2
        s = s[:, :h] + s[:, h:]
    return s[:, 0]


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("pcs,fibres", [(1, 4), (5, 16), (3, 32), (700, 64), (7, 128), (9, 256), (5, 512), (3, 1024),
                                        (2, 2048), (128, 4096), (3, 32768), (1, 131072)])
def test_sums_match_reference_order(pcs, fibres, shift):
    import torch
    rng = np.random.Generator(np.random.PCG64(fibres + pcs))
    n = pcs * fibres
    ap = rng.integers(0, 2 ** 32, n, dtype=np.uint32)
    mask = (np.uint32(1) << rng.integers(0, 32, n, dtype=np.uint32)).astype(np.uint32)
    w = rng.random(n, dtype=np.float32)
    w[:: 7] = -w[:: 7]

    def dev(a):
        buf = torch.zeros(n + 4, dtype=torch.int32, device="cuda")
        buf[shift:shift + n] = torch.from_numpy(a.view(np.int32)).cuda()
        return buf

    bufs = [dev(a) for a in (ap, mask, w)]
    out = torch.full((pcs,), float("nan"), device="cuda")
    torch.cuda.synchronize()
    rc = _entry()(*[b.data_ptr() + 4 * shift for b in bufs], n, pcs, out.data_ptr(), None)
    assert rc == 0, _last_error()
    torch.cuda.synchronize()
    assert out.cpu().numpy().tobytes() == reference(ap, mask, w, pcs).tobytes()
