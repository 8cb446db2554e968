"""The tensor-core launches on a second device of one process.

Dynamic shared memory beyond 48 KB is allowed per device; a launch above what its device allows is refused.  The launch
code (mlp.o, as it goes into the library) is linked here with a fake of the runtime that keeps that rule, so that it
needs neither a GPU nor a second one.
"""
import ctypes as C
import os
import shutil
import subprocess

import pytest

from conftest import PKG

FAKE = r"""
#include <map>
#include <set>
#include <utility>
#include "abi_internal.h"
namespace {
int device = 0, launches = 0;
std::map<std::pair<int, const void*>, int> allowed;
struct { dim3 g, b; size_t smem; void* st; } pushed;
}
namespace csv {
int abi_fail(csv_ctx*, int code, const std::string&) { return code; }
int abi_cuda_fail(csv_ctx*, cudaError_t e, const char*) { return -1000 - (int)e; }
}
static cudaError_t last = cudaSuccess;
extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) { pushed = {g, b, smem, st}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    *g = pushed.g; *b = pushed.b; *smem = pushed.smem; *(void**)st = pushed.st;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
    allowed[{device, f}] = v;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) {
    ++launches;
    last = smem <= 48 * 1024 || allowed[{device, f}] >= (int)smem ? cudaSuccess : cudaErrorInvalidValue;
    return last;
}
cudaError_t cudaGetLastError() { cudaError_t e = last; last = cudaSuccess; return e; }

// what = 0: csv_gemm_bf16; 1: a product of the network's tiled operands; 2: the fused forward; 3: csv_gemm_bf16 in place
int run(int what, int dev) {
    csv_ctx ctx;
    ctx.device = dev;
    csv::DeviceGuard guard(dev);
    static __nv_bfloat16 A[128 * 64], B[64 * 64], out[128 * 64];
    if (what == 0 || what == 3)
        return csv_gemm_bf16(&ctx, A, B, 128, 64, 64, nullptr, nullptr, 0, nullptr, what ? A : out, nullptr, nullptr, nullptr, nullptr);
    if (what == 1) {
        csv::GemmArgs g;
        g.A = A; g.B = B; g.M = 128; g.N = 64; g.K = 64; g.tiled = true; g.Cb = out;
        return csv::launch_gemm_bf16(g, nullptr);
    }
    return csv::launch_mlp_infer((const float*)A, 1, B, B, B, (float*)B, (float*)B, (float*)B, (float*)out, nullptr, nullptr,
                                 dev, nullptr);
}
int launch_count() { return launches; }
}
"""


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc")))
    if not os.path.exists(os.path.join(cuda, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    subprocess.run(["make", "-s", "-C", PKG, "_build/mlp.o"], check=True)
    d = tmp_path_factory.mktemp("fake")
    (d / "fake.cpp").write_text(FAKE)
    so = str(d / "fake.so")
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-o", so, str(d / "fake.cpp"),
                    os.path.join(PKG, "_build", "mlp.o"), "-I", os.path.join(PKG, "csrc"),
                    "-I", os.path.join(PKG, "..", "include"), "-I", os.path.join(cuda, "include"),
                    "-Wl,-Bsymbolic"], check=True)
    return C.CDLL(so)


@pytest.mark.parametrize("what", [0, 1, 2, 3])
def test_shared_memory_is_allowed_on_every_device(fake, what):
    n = fake.launch_count()
    for dev in (0, 1, 0, 70, 1):
        assert fake.run(what, dev) == 0, dev
    assert fake.launch_count() == n + 5
