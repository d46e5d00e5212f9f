"""The allocation-free sort after one of its waits has run out: the outputs are those of a stable sort all the same.

One tile of every pass withholds its digit counts and the tiles after it give up after 64 spins (one tile alone has
nobody to wait for); whole and ragged tiles, one to four 8-bit digits, an even and an odd number of passes. The call
after it, with the default bound, finds nothing of the stall.
"""

import numpy as np
import pytest

from libclsph_gb300.gpu import NO_TILE

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("bits", [8, 16, 22, 32])
@pytest.mark.parametrize("n, tile", [(4096, 0), (4097, 0), (40000, 3), (1 << 20, 0), (1 << 20, 255), ((1 << 20) - 1, 100)])
def test_stalled_sort_is_sorted(gpu_lib, n, tile, bits):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, 1 << bits, n, dtype=np.uint64).astype(np.uint32)
    keys[::5] = keys[0]
    want = np.argsort(keys, kind="stable").astype(np.uint32)
    src = torch.from_numpy(keys.view(np.int32)).cuda()
    stream = torch.cuda.current_stream()
    for limits in ((64, tile), (1 << 20, NO_TILE)):
        out, perm = torch.full_like(src, -1), torch.full_like(src, -1)
        assert gpu_lib.clsph_gpu_sort_keys_noalloc_limited(src.data_ptr(), out.data_ptr(), perm.data_ptr(), n,
                                                           stream.cuda_stream, *limits) == 0
        stream.synchronize()
        assert np.array_equal(perm.cpu().numpy().view(np.uint32), want)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), keys[want])
