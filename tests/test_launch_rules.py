"""What holds for a kernel by the way it is launched and ended, checked without a device: on the sources, and on the launchers compiled against a stand-in for the CUDA runtime."""
from __future__ import annotations

import ctypes
import re
import shutil
import subprocess
from pathlib import Path

import pytest
from test_second_device import CSRC, FAKE_RUNTIME


@pytest.fixture(scope="module")
def products(tmp_path_factory):
    """gemm_fp32.cu's launchers; the stand-in counts the launches that may start before the kernel in front of them has ended."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("no nvcc")
    folder = tmp_path_factory.mktemp("launch_rules")
    launch = "cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* kernel, void**) {"
    assert launch in FAKE_RUNTIME
    runtime = FAKE_RUNTIME.replace(launch, "static int early = 0;\nstatic dim3 grid, block;\nint fake_early_launches() { return early; }\nint fake_threads() { return block.x; }\n" + launch
                                   + " early += config->numAttrs; grid = config->gridDim; block = config->blockDim; if (grid.y > 65535 || grid.z > 65535) return cudaErrorInvalidConfiguration;")
    (folder / "runtime.cpp").write_text(runtime)
    library = folder / "products.so"
    subprocess.run([nvcc, "-std=c++17", "-shared", "-Xcompiler", "-fPIC", "--expt-relaxed-constexpr", "-cudart", "none", "-Xlinker", "-Bsymbolic", "-gencode", "arch=compute_100a,code=sm_100a", "-Xptxas", "-O0",
                    "-I", str(CSRC), "-o", str(library), str(CSRC / "gemm_fp32.cu"), str(folder / "runtime.cpp")], check=True)
    return ctypes.CDLL(str(library))


@pytest.mark.parametrize("M", [1, 12, 40, 300])
def test_32_bit_products_that_read_through_l1_do_not_start_early(products, M, monkeypatch):
    """Operands that are not 16-byte aligned take 4-byte asynchronous copies, which exist through L1 only; a line of it may be older than what the kernel in front writes."""
    monkeypatch.delenv("TLIE_PDL", raising=False)
    for N in (100, 2050):
        for address, K, lda, early in ((1 << 20, 2048, 2048, 1), (1 << 20, 2048, 2052, 1), ((1 << 20) + 4, 2048, 2048, 0), (1 << 20, 2047, 2048, 0), (1 << 20, 2048, 2049, 0), (1 << 20, 5, 5, 0)):
            memory, before, launches = ctypes.c_void_p(address), products.fake_early_launches(), products.fake_launches()
            assert products.tlie_gemm_nt_f32(memory, memory, memory, M, N, K, ctypes.c_longlong(lda), None) == 0
            assert (products.fake_early_launches() - before, products.fake_launches() - launches) == (early, 1), (N, address, K, lda)


@pytest.mark.parametrize("M,N,K,few", [(17, 1, 64, True), (24, 2048, 2048, True), (64, 5632, 2048, True), (96, 2048, 2048, True), (200, 2048, 2048, False), (600, 97, 2048, True),
                                       (1280, 208, 2048, False), (24, 32000, 2048, True), (48, 11264, 2048, False), (150, 2048, 5632, False), (400, 256, 64, True), (760, 2048, 5632, False), (3000000, 1, 64, False)])
def test_32_bit_products_take_the_kernel_that_is_cheaper(products, M, N, K, few):
    """Blocks of 16 rows (CTAs of 256 threads) or tiles of 128: measured, one of them 1.1 to 8 times as fast; and never more blocks than a grid's second dimension has."""
    memory = ctypes.c_void_p(1 << 20)
    assert products.tlie_gemm_nt_f32(memory, memory, memory, M, N, K, ctypes.c_longlong(K), None) == 0
    assert products.fake_threads() == (256 if few else 544)


def test_32_bit_products_read_operands_by_ordinary_loads():
    """Their kernels start while the one in front may still write x or w: no read-only path, nor C++ loads of pointers to constants, which the compiler may send there."""
    source = (CSRC / "gemm_fp32.cu").read_text()
    kernels = source[source.index("load_four("):source.index("gemm_short_f32_kernel")]   # (that one is launched behind the kernel in front of it)
    assert not re.search(r"__ldg\(|ld\.global\.nc|\bx_rows\[\w+\]\[|\brow\[k|\bx\[|\bw\[", kernels)


WAITING = sorted(path.name for path in CSRC.glob("*.cu") if "abort_flag" in path.read_text())


def test_the_kernels_with_bounded_waits_are_known():
    assert WAITING == ["attention_prefill_tc.cu", "gemm_fp32.cu", "gemm_skinny.cu", "gemm_tcgen05.cu", "gemm_tcgen05_pair.cu", "moe_grouped_tc.cu"]


@pytest.mark.parametrize("name", WAITING)
def test_a_wait_that_gives_up_is_reported_whichever_thread_it_is(name):
    """The report reads the CTA's flag behind the barrier that every wait has ended at; in front of it, the reporting thread may be done before another thread's wait gives up."""
    shared = (CSRC / "tcgen05_utils.cuh").read_text()
    closing = shared[shared.index("void close_and_report("):]
    closing = closing[:closing.index("\n}\n")]
    assert closing.index("__syncthreads();") < closing.index("if (*abort_flag)") < closing.index("atomicOr(error_flag, 1)") < closing.index("__nanosleep")
    source = (CSRC / name).read_text()
    assert "if (*abort_flag" not in source   # nobody reports by itself
    for kernel in re.split(r"(?=__global__ )", source)[1:]:
        if "mbar_wait(" in kernel:
            end = kernel.index("close_and_report(abort_flag,")
            assert "mbar_wait(" not in kernel[end:] and kernel.index("tcgen05.dealloc", end) > end   # tensor memory is given back behind it
