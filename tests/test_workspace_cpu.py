"""The device workspace (csrc/workspace.cu) over a fake CUDA runtime with a
settable amount of memory: how much a call gets, and that calls repeated where
memory is short neither reallocate each time nor stay small once there is room.
And the kernels' shared-memory limits, which a call never lowers."""

import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

FAKE = r"""
#include "%(csrc)s/common.cuh"
#include <map>
static size_t g_free, g_refuse_from = SIZE_MAX;
static long g_mallocs;
static bool g_capturing;
static std::map<void *, size_t> g_blocks;
namespace wb {
bool injected(int) { return false; }
int fail(int code, const std::string &) { return code; }
int cuda_fail(cudaError_t, const char *) { return WB_ECUDA; }
size_t align256(size_t b) { return (b + 255) & ~size_t(255); }
const DeviceInfo &device_info() {
    static DeviceInfo d;
    d.max_smem_optin = 232448;
    return d;
}
}
static std::map<const void *, int> g_limit;
static long g_sets;
extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = g_free; *t = 1ull << 38; return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) {
    *s = g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) {
    static char *at = (char *)0x100000;
    g_mallocs++;
    if (g_capturing) return cudaErrorStreamCaptureUnsupported;
    if (n > g_free || n >= g_refuse_from) return cudaErrorMemoryAllocation;
    g_free -= n;
    *p = at;
    at += (n + 255) & ~size_t(255);
    g_blocks[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) { g_free += g_blocks[p]; g_blocks.erase(p); return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *k) {
    *a = cudaFuncAttributes();
    a->sharedSizeBytes = 8192;
    a->maxDynamicSharedSizeBytes = g_limit.count(k) ? g_limit[k] : 49152 - 8192;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *k, cudaFuncAttribute, int v) {
    g_sets++;
    if (v > 232448 - 8192) return cudaErrorInvalidValue;
    g_limit[k] = v;
    return cudaSuccess;
}
int t_allow(long kernel, size_t bytes) { return wb::allow_shared((const void *)kernel, bytes); }
int t_limit(long kernel) { return g_limit[(const void *)kernel]; }
long t_sets() { return g_sets; }
// a call that reserves: what it has, or a negative status
int64_t t_reserve(long stream, size_t bytes, size_t least) {
    wb::Workspace ws((cudaStream_t)stream);
    const int st = ws.reserve(bytes, least);
    return st == WB_OK ? (int64_t)ws.remaining() : -(int64_t)st;
}
void t_set(size_t free, size_t refuse_from, int capturing) {
    g_free = free; g_refuse_from = refuse_from; g_capturing = capturing != 0;
}
size_t t_free() { return g_free; }
long t_mallocs() { return g_mallocs; }
}
"""

MB, GB = 1 << 20, 1 << 30
NEVER = (1 << 64) - 1


@pytest.fixture
def ws(tmp_path, monkeypatch):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("no CUDA headers")
    monkeypatch.delenv("WB_GPU_WORKSPACE_MB", raising=False)
    csrc = os.path.join(ROOT, "wildboar_gb300", "csrc")
    (tmp_path / "fake.cpp").write_text(FAKE % {"csrc": csrc})
    lib = str(tmp_path / "ws.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I",
                    os.path.join(CUDA, "include"), str(tmp_path / "fake.cpp"), "-x", "c++",
                    os.path.join(csrc, "workspace.cu"), "-o", lib], check=True)
    L = ctypes.CDLL(lib)
    size = ctypes.c_size_t
    L.t_reserve.argtypes = [ctypes.c_long, size, size]
    L.t_reserve.restype = ctypes.c_int64
    L.t_set.argtypes = [size, size, ctypes.c_int]
    L.t_free.restype = size
    L.t_mallocs.restype = ctypes.c_long
    L.t_allow.argtypes = [ctypes.c_long, size]
    L.t_limit.argtypes = [ctypes.c_long]
    L.t_sets.restype = ctypes.c_long
    L.wb_release_workspace.argtypes = [ctypes.c_void_p]
    return L


def test_room_for_all(ws):
    ws.t_set(100 * GB, NEVER, 0)
    assert ws.t_reserve(1, 6 * GB, 10 * MB) >= 6 * GB
    for _ in range(5):
        assert ws.t_reserve(1, 6 * GB, 10 * MB) >= 6 * GB
    assert ws.t_mallocs() == 1
    # another stream has its own
    assert ws.t_reserve(2, 10 * MB, 10 * MB) >= 10 * MB
    ws.wb_release_workspace(None)
    assert ws.t_free() == 100 * GB


def test_half_of_what_is_free(ws):
    ws.t_set(4 * GB, NEVER, 0)
    got = ws.t_reserve(1, 6 * GB, 10 * MB)
    assert 10 * MB <= got <= 2.3 * GB and ws.t_free() >= 1.7 * GB
    n = ws.t_mallocs()
    for _ in range(20):  # equal calls: no new arena, none given back
        assert ws.t_reserve(1, 6 * GB, 10 * MB) == got
    assert ws.t_mallocs() == n
    ws.t_set(ws.t_free() + 80 * GB, NEVER, 0)  # memory was freed: all of it
    assert ws.t_reserve(1, 6 * GB, 10 * MB) >= 6 * GB


def test_refused_sizes(ws):
    ws.t_set(40 * GB, 3 * GB, 0)  # the device refuses 3 GB and more
    got = ws.t_reserve(1, 6 * GB, 10 * MB)
    assert 10 * MB <= got < 3 * GB
    n = ws.t_mallocs()
    for _ in range(20):
        assert ws.t_reserve(1, 6 * GB, 10 * MB) == got
        assert ws.t_reserve(1, 5 * GB, 10 * MB) == got
    assert ws.t_mallocs() == n
    # a call that needs more gets what it needs, whatever was refused before
    assert ws.t_reserve(1, 6 * GB, 2900 * MB) >= 2900 * MB
    # with more room the larger size is asked for again; also after a release
    ws.t_set(ws.t_free() + 40 * GB, NEVER, 0)
    assert ws.t_reserve(1, 6 * GB, 10 * MB) >= 6 * GB
    ws.wb_release_workspace(None)
    ws.t_set(40 * GB, 3 * GB, 0)
    assert ws.t_reserve(1, 6 * GB, 10 * MB) < 3 * GB
    ws.wb_release_workspace(None)
    ws.t_set(40 * GB, NEVER, 0)
    assert ws.t_reserve(1, 6 * GB, 10 * MB) >= 6 * GB


def test_exact_size_where_the_slack_does_not_fit(ws):
    ws.t_set(40 * GB, 6 * GB + 100 * MB, 0)
    assert 6 * GB <= ws.t_reserve(1, 6 * GB, 10 * MB) < 6 * GB + 100 * MB
    n = ws.t_mallocs()
    assert ws.t_reserve(1, 6 * GB, 10 * MB) >= 6 * GB and ws.t_mallocs() == n


def test_the_least_need_fails_as_out_of_memory(ws):
    ws.t_set(50 * MB, NEVER, 0)
    assert ws.t_reserve(1, 6 * GB, 100 * MB) < 0
    assert ws.t_reserve(1, 6 * GB, 20 * MB) >= 20 * MB  # and the next call runs


def test_no_growth_for_faster_forms_under_capture(ws):
    ws.t_set(40 * GB, NEVER, 0)
    assert ws.t_reserve(1, 100 * MB, 100 * MB) >= 100 * MB
    n = ws.t_mallocs()
    ws.t_set(ws.t_free(), NEVER, 1)
    assert ws.t_reserve(1, 6 * GB, 50 * MB) >= 100 * MB
    assert ws.t_mallocs() == n


def test_the_budget(ws, monkeypatch):
    ws.t_set(40 * GB, NEVER, 0)
    monkeypatch.setenv("WB_GPU_WORKSPACE_MB", "64")
    got = ws.t_reserve(1, 6 * GB, 10 * MB)
    assert 74 * MB <= got <= 100 * MB
    monkeypatch.setenv("WB_GPU_WORKSPACE_MB", "0")
    assert ws.t_reserve(2, 6 * GB, 10 * MB) <= 14 * MB


def test_a_shared_memory_limit_is_never_lowered(ws):
    # a large call raises the limit, a small one of another thread comes before
    # the large call's launch
    assert ws.t_allow(1, 100_000) == 0 and ws.t_allow(1, 2_000) == 0
    assert ws.t_limit(1) >= 100_000
    assert ws.t_allow(1, 224_256) == 0 and ws.t_sets() == 1  # set once, to all there is
    assert ws.t_allow(1, 224_257) != 0  # more than the device has
    assert ws.t_allow(2, 40_000) == 0 and ws.t_allow(2, 200_000) == 0 and ws.t_sets() == 2


def test_no_call_sets_a_limit_by_itself():
    csrc = os.path.join(ROOT, "wildboar_gb300", "csrc")
    for f in sorted(os.listdir(csrc)):
        with open(os.path.join(csrc, f)) as fh:
            assert f == "workspace.cu" or "MaxDynamicSharedMemorySize" not in fh.read(), f
