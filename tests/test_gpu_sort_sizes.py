"""The stable key sort at the edges of its tiles and passes, against numpy's stable sort (integers: equal).

Through clsph_gpu_sort_keys_noalloc, which shares the substep's sort: one key, whole and ragged tiles of 4,096,
several tiles; keys of one to four 8-bit digits, random, nearly sorted (runs of equal keys) and all equal.
"""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _keys(n, bits, kind, rng):
    if kind == "equal":
        return np.full(n, (1 << bits) - 1, dtype=np.uint32)
    k = rng.integers(0, 1 << bits, n, dtype=np.uint64)
    if kind == "runs":
        k = np.sort(k)[np.arange(n) // 37 * 37]
        stray = rng.random(n) < 0.05
        k[stray] = rng.integers(0, 1 << bits, int(stray.sum()), dtype=np.uint64)
    return k.astype(np.uint32)


@pytest.mark.parametrize("kind", ["random", "runs", "equal"])
@pytest.mark.parametrize("n", [1, 31, 4095, 4096, 4097, 40000, 1 << 20])
def test_sort_sizes(gpu_lib, n, kind):
    rng = np.random.default_rng(n)
    for bits in (1, 8, 9, 16, 22, 32):
        keys = _keys(n, bits, kind, rng)
        src = torch.from_numpy(keys.view(np.int32)).cuda()
        out, perm = torch.full_like(src, -1), torch.full_like(src, -1)
        stream = torch.cuda.current_stream()
        assert gpu_lib.clsph_gpu_sort_keys_noalloc(src.data_ptr(), out.data_ptr(), perm.data_ptr(), n,
                                                   stream.cuda_stream) == 0
        stream.synchronize()
        want = np.argsort(keys, kind="stable").astype(np.uint32)
        assert np.array_equal(perm.cpu().numpy().view(np.uint32), want), (bits, kind)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), keys[want]), (bits, kind)
