"""Calls on a caller's stream come after everything queued there, also behind kernels that the caller placed early.

The caller's stream holds a kernel that lets its successor start at once and writes its data some milliseconds
later, and a second one, launched to overlap it, that ends without waiting. Work queued next has to see the data.
"""

import ctypes
import subprocess

import numpy as np
import pytest

from libclsph_gb300 import workloads as W
from libclsph_gb300.build import ARCH, _nvcc
from libclsph_gb300.gpu import GpuSolver

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SOURCE = r"""
#include <cuda_runtime.h>
#include <cstdint>
__global__ void late_copy(const uint32_t* src, uint32_t* dst, uint32_t words) {
  asm volatile("griddepcontrol.launch_dependents;");
  for (int k = 0; k < 300; ++k) __nanosleep(10000);
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < words; i += gridDim.x * blockDim.x) dst[i] = src[i];
}
__global__ void no_wait() {}
extern "C" int late_words(const uint32_t* src, uint32_t* dst, uint32_t words, void* stream) {
  late_copy<<<8, 256, 0, static_cast<cudaStream_t>(stream)>>>(src, dst, words);
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(1);
  cfg.blockDim = dim3(32);
  cfg.stream = static_cast<cudaStream_t>(stream);
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return (int)cudaLaunchKernelEx(&cfg, no_wait);
}
"""


@pytest.fixture(scope="module")
def late_words(gpu_lib, tmp_path_factory):
    d = tmp_path_factory.mktemp("late")
    (d / "late.cu").write_text(SOURCE)
    subprocess.run([_nvcc(), *ARCH, "-O2", "-std=c++17", "-Xcompiler", "-fPIC", "-shared", "-o", str(d / "late.so"),
                    str(d / "late.cu")], check=True)
    fn = ctypes.CDLL(str(d / "late.so")).late_words
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_void_p]
    return fn


def test_sort_sees_late_keys(gpu_lib, late_words):
    n = 100001
    keys = np.random.default_rng(1).integers(0, 1 << 22, n, dtype=np.uint32)
    src = torch.from_numpy(keys.view(np.int32)).cuda()
    buf, out, perm = torch.zeros_like(src), torch.full_like(src, -1), torch.full_like(src, -1)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(3):  # (the first call also loads the code)
        buf.zero_()
        torch.cuda.synchronize()
        assert late_words(src.data_ptr(), buf.data_ptr(), n, stream.cuda_stream) == 0
        assert gpu_lib.clsph_gpu_sort_keys_noalloc(buf.data_ptr(), out.data_ptr(), perm.data_ptr(), n,
                                                   stream.cuda_stream) == 0
        stream.synchronize()
        assert np.array_equal(perm.cpu().numpy().view(np.uint32), np.argsort(keys, kind="stable").astype(np.uint32))


def test_upload_sees_late_records(gpu_lib, late_words):
    sc = W.small_block(12, seed=17, velocity_sigma=0.2)
    records = sc.particles.view(np.uint8).reshape(-1)
    src = torch.from_numpy(records.copy()).cuda()
    pinned = torch.zeros(len(records), dtype=torch.uint8).pin_memory()
    stream = torch.cuda.Stream()
    with GpuSolver(sc.params, sc.terms, sc.n, sc.mesh) as g:
        g.upload(sc.particles)
        g.step(1)
        want = g.download()
        g.set_stream(stream.cuda_stream)
        for _ in range(3):
            pinned.zero_()
            torch.cuda.synchronize()
            assert late_words(src.data_ptr(), pinned.data_ptr(), len(records) // 4, stream.cuda_stream) == 0
            g.upload(pinned.numpy().view(sc.particles.dtype))
            g.step(1)
            got = g.download()
            assert np.array_equal(got.view(np.uint8), want.view(np.uint8))
        g.set_stream(None)
