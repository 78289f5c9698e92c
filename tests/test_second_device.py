"""The 32-bit kernels on a second device of one process, without a device: their launchers are compiled against a stand-in for the CUDA runtime that keeps the
shared-memory attribute per device, as the runtime does, and refuses a launch without it."""
from __future__ import annotations

import ctypes
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tinyllama_inference_engine_b200" / "csrc"

FAKE_RUNTIME = r"""
#include <cuda_runtime.h>
#include <map>
#include <utility>
static int device = 0, launches = 0;
static std::map<std::pair<const void*, int>, int> allowed;
static dim3 pushed_grid, pushed_block; static size_t pushed_smem; static cudaStream_t pushed_stream;
static cudaError_t launch(const void* kernel, size_t smem) {
  auto found = allowed.find({kernel, device});
  if (smem > 48 * 1024 && (found == allowed.end() || (size_t)found->second < smem)) return cudaErrorInvalidValue;
  ++launches;
  return cudaSuccess;
}
static cudaError_t last = cudaSuccess;
extern "C" {
void fake_set_device(int d) { device = d; }
int fake_launches() { return launches; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr, int) { *value = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* kernel, cudaFuncAttribute, int value) { allowed[{kernel, device}] = value; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* kernel, dim3, dim3, void**, size_t smem, cudaStream_t) { return last = launch(kernel, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* kernel, void**) { return last = launch(kernel, config->dynamicSmemBytes); }
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t m, cudaStream_t s) { pushed_grid = g; pushed_block = b; pushed_smem = m; pushed_stream = s; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) { *g = pushed_grid; *b = pushed_block; *m = pushed_smem; *(cudaStream_t*)s = pushed_stream; return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
char __cudaInitModule(void**) { return 0; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long, cudaDriverEntryPointQueryResult*) { return cudaErrorUnknown; }
cudaError_t __cudaLaunchKernel(const void* kernel, dim3, dim3, void**, size_t smem, cudaStream_t) { return last = launch(kernel, smem); }
cudaError_t __cudaGetKernel(void** kernel, const void* entry) { *kernel = const_cast<void*>(entry); return cudaSuccess; }
}
"""


@pytest.fixture(scope="module")
def launchers(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    folder = tmp_path_factory.mktemp("fake_runtime")
    (folder / "runtime.cpp").write_text(FAKE_RUNTIME)
    library = folder / "launchers.so"   # -Bsymbolic: the real runtime may be loaded in this process too
    subprocess.run([nvcc, "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-cudart", "none", "-Xlinker", "-Bsymbolic", "-gencode", "arch=compute_100a,code=sm_100a", "-Xptxas", "-O0",
                    "-I", str(CSRC), "-o", str(library), str(CSRC / "gemm_fp32.cu"), str(CSRC / "attention_generic.cu"), str(folder / "runtime.cpp")], check=True)
    return ctypes.CDLL(str(library))


@pytest.mark.parametrize("M", [1, 2, 4, 8, 16, 40, 300])
def test_32_bit_products_launch_on_every_device(launchers, M):
    memory = ctypes.c_void_p(1 << 20)   # an address that nothing reads: nothing runs
    for device in (0, 1, 1, 0, 63, 64, 65):
        launchers.fake_set_device(device)
        for N in (64, 2048, 32000):
            before = launchers.fake_launches()
            assert launchers.tlie_gemm_nt_f32(memory, memory, memory, M, N, 2048, ctypes.c_longlong(2048), None) == 0, (device, N)
            assert launchers.fake_launches() == before + 1


@pytest.mark.parametrize("head_dim", [64, 128])
def test_32_bit_attention_launches_on_every_device(launchers, head_dim):
    memory = ctypes.c_void_p(1 << 20)
    for device in (0, 1, 64, 65):
        launchers.fake_set_device(device)
        for rows in (1, 4):
            before = launchers.fake_launches()
            assert launchers.tlie_paged_attention_shared_f32(memory, 4096, memory, memory, memory, memory, 8, memory, 12, 16, 2, head_dim, 64, ctypes.c_float(0.125), rows, None) == 0
            assert launchers.fake_launches() == before + 1
