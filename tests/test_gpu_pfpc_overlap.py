"""Overlapping calls of cbm_pfpc_sums_noalloc keep nothing in common: on several
streams at once, each with its own buffers, at every number of CTAs a cluster has
and with the shortest rows (a CTA reaches its first store to another one's shared
memory as early as it can), every call gives the sums in the reference's order."""
import numpy as np
import pytest

from test_gpu_pfpc_sums import reference
from test_zz_no_alloc import _entry, _last_error

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pcs,fibres", [(64, 128), (64, 512), (64, 2048), (16, 8192)])
def test_overlapping_calls(pcs, fibres):
    import torch
    rng = np.random.Generator(np.random.PCG64(pcs + fibres))
    n, calls = pcs * fibres, 4
    streams = [torch.cuda.Stream() for _ in range(calls)]
    data, want, outs = [], [], []
    for _ in range(calls):
        ap = rng.integers(0, 2 ** 32, n, dtype=np.uint32)
        mask = (np.uint32(1) << rng.integers(0, 32, n, dtype=np.uint32)).astype(np.uint32)
        w = rng.random(n, dtype=np.float32)
        data.append([torch.from_numpy(a.view(np.int32)).cuda() for a in (ap, mask, w)])
        want.append(reference(ap, mask, w, pcs).tobytes())
        outs.append([torch.full((pcs,), float("nan"), device="cuda") for _ in range(50)])
    torch.cuda.synchronize()
    fn = _entry()
    for k in range(50):
        for s, bufs, out in zip(streams, data, outs):
            assert fn(*[b.data_ptr() for b in bufs], n, pcs, out[k].data_ptr(), s.cuda_stream) == 0, _last_error()
    torch.cuda.synchronize()
    for out, w in zip(outs, want):
        assert all(o.cpu().numpy().tobytes() == w for o in out)
