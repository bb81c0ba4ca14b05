"""The sort's host side against a CUDA runtime of this file (no GPU is used: its object file is linked
with it).  A process with several GPUs: limits that a launch needs are asked for on every device, as the
runtime keeps a function's attributes per device and refuses a launch that goes beyond them.  And which
calls wait for their work before they return."""
import ctypes as C
import shutil
import subprocess
from pathlib import Path

import pytest

RUNTIME = r"""
#include <cuda_runtime_api.h>
#include <cstdint>
#include <cstring>
#include <map>
#include <utility>

static int g_device = 0;
static std::map<std::pair<int, const void*>, std::pair<int, bool>> g_attr;   // (device, kernel): smem, clusters of 16
static int g_count[8];
static bool g_pending = false;          // work enqueued and not waited for
static cudaError_t g_last = cudaSuccess;

static cudaError_t allowed(const void* f, size_t smem, bool cluster) {
  const auto& a = g_attr[{g_device, f}];
  if ((smem > 48 * 1024 && (size_t)a.first < smem) || (cluster && !a.second)) return g_last = cudaErrorInvalidValue;
  ++g_count[g_device];
  g_pending = true;
  return cudaSuccess;
}

namespace tqpk {
thread_local int64_t g_launches = 0;
int num_sms() { return 152; }
int grid_for(int64_t, int) { return 1; }
void timing_before(int, cudaStream_t) {}
void timing_after(int, cudaStream_t) {}
}

extern "C" {
void fake_device(int d) { g_device = d; }
int fake_launches(int d) { return g_count[d]; }
int fake_pending() { return g_pending; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, void*, void*, void*, void*, int*) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
static struct { dim3 g, b; size_t smem; void* s; } g_cfg;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* s) { g_cfg = {g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
  *g = g_cfg.g; *b = g_cfg.b; *smem = g_cfg.smem; *(void**)s = g_cfg.s;
  return cudaSuccess;
}
cudaError_t __cudaGetKernel(void** k, const void* f) { *k = const_cast<void*>(f); return cudaSuccess; }
cudaError_t __cudaLaunchKernel(void* k, dim3, dim3, void**, size_t smem, cudaStream_t) { return allowed(k, smem, false); }
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return allowed(f, smem, false); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
  return allowed(f, c->dynamicSmemBytes, true);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
  auto& x = g_attr[{g_device, f}];
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) x.first = v;
  if (a == cudaFuncAttributeNonPortableClusterSizeAllowed) x.second = v != 0;
  return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 2; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 2; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { *n = 4; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = g_device; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError() { return g_last; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { g_pending = false; return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void*, size_t n, cudaMemcpyKind k, cudaStream_t) {
  if (k == cudaMemcpyDeviceToHost) memset(d, 0, n);
  g_pending = true;
  return cudaSuccess;
}
}
"""


@pytest.fixture(scope="module")
def sort_lib(tmp_path_factory):
    from tqpk import build as B
    B.build()
    obj = B.BUILD / "sort.o"
    gxx = shutil.which("g++")
    if not obj.exists() or gxx is None:
        pytest.skip("the build left no object files, or there is no g++")
    cuda = Path(B._nvcc()).resolve().parent.parent / "include"
    d = tmp_path_factory.mktemp("runtime")
    (d / "runtime.cpp").write_text(RUNTIME)
    subprocess.run([gxx, "-std=c++17", "-O1", "-fPIC", f"-I{cuda}", "-c", str(d / "runtime.cpp"), "-o", str(d / "runtime.o")],
                   check=True)
    subprocess.run([gxx, "-shared", "-Wl,-Bsymbolic", "-o", str(d / "sort.so"), str(obj), str(d / "runtime.o")], check=True)
    lib = C.CDLL(str(d / "sort.so"))
    lib.tqpk_sort_workspace_bytes.restype = C.c_size_t
    lib.tqpk_sort_workspace_bytes.argtypes = [C.c_int64]
    lib.tqpk_argsort_stable.argtypes = [C.c_void_p, C.c_int32, C.c_int32, C.c_void_p, C.c_int64, C.c_void_p, C.c_void_p,
                                        C.c_size_t, C.c_void_p]
    return lib


@pytest.mark.parametrize("n", [2000, 5000, 60_000, 200_000, 1_500_000])
def test_every_device_sorts(sort_lib, n):
    from tqpk import _lib as L
    ws = sort_lib.tqpk_sort_workspace_bytes(n)
    base = C.create_string_buffer(4096)
    p = (C.addressof(base) + 255) & ~255                    # never read: nothing runs
    for device in (0, 1, 0, 3):
        sort_lib.fake_device(device)
        before = sort_lib.fake_launches(device)
        assert sort_lib.tqpk_argsort_stable(p, L.I64, 0, None, n, p, p, ws, None) == L.OK
        assert sort_lib.fake_launches(device) > before


@pytest.mark.parametrize("n", [2048, 2049, 32_769, 98_304, 98_305])
@pytest.mark.parametrize("in_place", [False, True])
def test_sorts_beyond_one_cta_are_complete_when_they_return(sort_lib, n, in_place):
    """More than 2048 rows: the keys are not read again, and the order is written, when the call returns
    (another stream may use either); up to 2048 nothing waits, so that a capture may hold the call."""
    from tqpk import _lib as L
    ws = sort_lib.tqpk_sort_workspace_bytes(n)
    base = C.create_string_buffer(4096)
    p = (C.addressof(base) + 255) & ~255
    perm = p + (1 << 40)                                    # never read or written either
    sort_lib.fake_device(0)
    assert sort_lib.tqpk_argsort_stable(p, L.I64, 0, perm if in_place else None, n, perm, p, ws, None) == L.OK
    assert bool(sort_lib.fake_pending()) == (n <= 2048)
