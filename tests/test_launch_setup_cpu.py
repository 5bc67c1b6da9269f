"""Set-up of the kernels that take more than 48 KB of shared memory, against a fake CUDA runtime (no GPU): the opt-in belongs
to one device's copy of a function, so every device needs its own."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KERNELS = os.path.join(ROOT, "torch_musa_b200", "csrc", "kernels")
LIB = os.path.join(ROOT, "torch_musa_b200", "libb200_kernels.so")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

# The executable's definitions stand before the runtime's when the kernel library looks its symbols up.  The fake keeps the
# rule of the real one: a launch with more than 48 KB of dynamic shared memory is refused unless this device's copy of the
# function has been given that much.
DRIVER = r"""
#include "b200_kernels.h"
#include <cuda.h>
#include <cuda_runtime_api.h>
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <utility>

static int g_dev = 0, g_fail = 0, g_launched = 0;
static cudaError_t g_last = cudaSuccess;
static std::map<std::pair<int, const void*>, size_t> g_opt_in;

static cudaError_t launch(const void* f, size_t smem) {
  auto it = g_opt_in.find({g_dev, f});
  const size_t room = it == g_opt_in.end() ? 48 * 1024 : it->second;
  ++g_launched;
  if (smem > room) g_last = cudaErrorInvalidValue;
  return smem > room ? cudaErrorInvalidValue : cudaSuccess;
}
static CUresult encode(CUtensorMap* m, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                       const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion,
                       CUtensorMapFloatOOBfill) {
  memset(m, 0, sizeof(*m));
  return CUDA_SUCCESS;
}
extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = g_dev; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaDeviceGetAttribute(int* v, enum cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaHostAlloc(void**, size_t, unsigned) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFuncGetAttributes(struct cudaFuncAttributes* a, const void*) { memset(a, 0, sizeof(*a)); a->numRegs = 255; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute, int v) {
  if (g_fail) { --g_fail; g_last = cudaErrorMemoryAllocation; return cudaErrorMemoryAllocation; }
  g_opt_in[{g_dev, f}] = (size_t)v;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launch(f, c->dynamicSmemBytes); }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, enum cudaDriverEntryPointQueryResult* q) {
  *p = (void*)encode;
  if (q) *q = cudaDriverEntryPointSuccess;
  return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char* s, void** p, unsigned, unsigned long long f, enum cudaDriverEntryPointQueryResult* q) {
  return cudaGetDriverEntryPoint(s, p, f, q);
}
}

// never read or written by the fake: only the addresses count
static void* const A = (void*)0x10000, * const B = (void*)0x20000, * const C = (void*)0x30000, * const D = (void*)0x40000;

static int rms(int dtype, int cols) {
  return b200_rmsnorm_residual_bwd(dtype, A, (float*)B, nullptr, C, D, A, (float*)B, C, 8, cols, nullptr);
}
static int gemm(int m, int n, int k, int out_dtype, int in_dtype) {
  b200_gemm_desc_t g;
  memset(&g, 0, sizeof(g));
  g.m = m; g.n = n; g.k = k; g.batch = 1;
  g.a_kmajor = g.b_kmajor = 1;
  g.lda = g.ldb = k; g.ldd = n;
  g.in_dtype = in_dtype; g.out_dtype = out_dtype; g.bias_dtype = out_dtype;
  g.alpha = 1.f;
  return b200_gemm(&g, C, A, B, nullptr);
}
static int fp8(int m, int n) {
  b200_fp8_gemm_t g;
  memset(&g, 0, sizeof(g));
  g.m = m; g.n = n; g.k = 256;
  g.lda = g.ldb = 256; g.ldd = n;
  g.out_dtype = g.bias_dtype = B200_BF16;
  return b200_gemm_fp8(&g, C, A, B, nullptr);
}
static b200_attn_t attn(int dtype) {
  b200_attn_t a;
  memset(&a, 0, sizeof(a));
  a.B = 1; a.H = a.Hkv = 2; a.Sq = a.Sk = 256; a.head_dim = 128;
  a.dtype = dtype; a.scale = 1.f;
  a.q_sb = a.k_sb = a.v_sb = a.o_sb = 2 * 256 * 128;
  a.q_sh = a.k_sh = a.v_sh = a.o_sh = 256 * 128;
  a.q_ss = a.k_ss = a.v_ss = a.o_ss = 128;
  return a;
}
static int attn_fwd(int dtype) {
  b200_attn_t a = attn(dtype);
  return b200_flash_attn_fwd(&a, A, (float*)B, C, D, A, nullptr);
}
static int attn_bwd(int dtype) {
  b200_attn_t a = attn(dtype);
  const int64_t x[9] = {2 * 256 * 128, 256 * 128, 128, 2 * 256 * 128, 256 * 128, 128, 2 * 256 * 128, 256 * 128, 128};
  return b200_flash_attn_bwd(&a, (float*)A, B, C, (float*)D, A, B, C, D, A, (float*)B, x, nullptr);
}
static int grouped(int ragged_depth) {
  b200_grouped_gemm_t g;
  memset(&g, 0, sizeof(g));
  g.ragged_depth = ragged_depth;
  g.rows = 256; g.m = 256; g.n = 256; g.k = 256; g.groups = 2;
  g.counts = (const int*)D;
  g.b_kmajor = 1;
  g.lda = g.ldb = g.ldd = 256;
  g.stride_b = g.stride_d = 256 * 256;
  g.in_dtype = g.out_dtype = B200_BF16;
  return b200_grouped_gemm(&g, C, A, B, nullptr);
}

struct Call { const char* name; int (*go)(); };
static const Call kCalls[] = {
    {"rmsnorm_bwd bf16 4096", [] { return rms(B200_BF16, 4096); }},
    {"rmsnorm_bwd bf16 8192", [] { return rms(B200_BF16, 8192); }},
    {"rmsnorm_bwd f32 16384", [] { return rms(B200_F32, 16384); }},
    {"gemm few rows 16", [] { return gemm(16, 4096, 4096, B200_BF16, B200_BF16); }},
    {"gemm few rows 32 f16", [] { return gemm(32, 4096, 4096, B200_F16, B200_F16); }},
    {"gemm few rows 64 f32", [] { return gemm(64, 4096, 4096, B200_F32, B200_BF16); }},
    {"gemm one CTA", [] { return gemm(100, 4096, 512, B200_BF16, B200_BF16); }},
    {"gemm pair", [] { return gemm(4096, 4096, 512, B200_BF16, B200_BF16); }},
    {"gemm tf32", [] { return gemm(256, 256, 512, B200_F32, B200_F32); }},
    {"gemm fp8 narrow", [] { return fp8(128, 256); }},
    {"gemm fp8 wide", [] { return fp8(4096, 14336); }},
    {"attention fwd bf16", [] { return attn_fwd(B200_BF16); }},
    {"attention fwd f16", [] { return attn_fwd(B200_F16); }},
    {"attention bwd bf16", [] { return attn_bwd(B200_BF16); }},
    {"attention bwd f16", [] { return attn_bwd(B200_F16); }},
    {"grouped gemm fwd", [] { return grouped(0); }},
    {"grouped gemm wgrad", [] { return grouped(1); }},
};

int main(int argc, char** argv) {
  const std::string what = argv[1];
  int wrong = 0;
  for (const Call& c : kCalls) {
    int before = 0, bad = 0;
    if (what == "retry") {
      g_fail = 1;
      if (c.go() == 0) { printf("%s: the failing set-up was not seen\n", c.name); return 2; }
      g_fail = 0;
      bad = c.go();
      if (bad) printf("%s: %d at the second try\n", c.name, bad);
    } else {
      for (g_dev = 0; g_dev < 3 && !bad; ++g_dev) {
        before = g_launched;
        bad = c.go();
        if (bad) printf("%s: %d on device %d\n", c.name, bad, g_dev);
        if (g_launched == before) { printf("%s: no launch\n", c.name); return 2; }
      }
      g_dev = 0;
    }
    wrong += bad != 0;
  }
  return wrong;
}
"""


@pytest.fixture(scope="module")
def driver(tmp_path_factory):
    cxx = os.environ.get("B200_CXX", shutil.which("g++"))
    if cxx is None or not os.path.exists(LIB):
        pytest.skip("needs a C++ compiler and the built kernel library")
    import torch  # noqa: F401  (its CUDA runtime is the one the library was linked to)
    import nvidia.cuda_runtime

    d = tmp_path_factory.mktemp("setup")
    src, exe = d / "driver.cpp", d / "driver"
    src.write_text(DRIVER)
    rt = os.path.join(list(nvidia.cuda_runtime.__path__)[0], "lib")
    subprocess.run([cxx, "-std=c++17", "-O1", "-I", KERNELS, "-I", os.path.join(CUDA, "include"), str(src), LIB, "-L" + rt, "-l:libcudart.so.12",
                    "-Wl,-rpath," + os.path.dirname(LIB), "-Wl,-rpath," + rt, "-o", str(exe)], check=True)
    return exe


def test_second_device(driver):
    """A kernel that ran on one device of the process runs on the others."""
    r = subprocess.run([str(driver), "devices"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_failed_setup_is_tried_again(driver):
    """A set-up that fails once (no memory for a moment, say) fails that call and not those after it."""
    r = subprocess.run([str(driver), "retry"], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr


def test_rmsnorm_bwd_keeps_its_signature(tmp_path):
    """The kernel library is called from C and ctypes: an entry keeps its arguments, one that needs more gets a name."""
    src = tmp_path / "sig.cpp"
    src.write_text("""
#include "b200_kernels.h"
#include <type_traits>
static_assert(std::is_same<decltype(&b200_rmsnorm_bwd), int (*)(int, void*, float*, int*, const void*, const void*, const void*, const float*,
                                                                int64_t, int64_t, cudaStream_t)>::value, "b200_rmsnorm_bwd");
""")
    cxx = os.environ.get("B200_CXX", shutil.which("g++"))
    r = subprocess.run([cxx, "-std=c++17", "-fsyntax-only", "-I", KERNELS, "-I", os.path.join(CUDA, "include"), str(src)], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr


def test_blocks_that_gave_up_wait_for_their_copies():
    """Every kernel with tensor memory ends in settle_abort, after its last barrier: a block that gave up on a wait must not
    release shared memory that its copies in flight still write."""
    seen = 0
    for name in sorted(os.listdir(KERNELS)):
        if name.endswith(".cu"):
            text = open(os.path.join(KERNELS, name)).read()
            ends = re.findall(r"__syncthreads\(\);(?:(?!__syncthreads).)*?settle_abort\(", text, re.S)
            calls = re.findall(r"^ +tmem_dealloc(?:_pair)?\(", text, re.M)
            assert len(ends) == len(calls), name
            seen += len(calls)
    assert seen >= 8
