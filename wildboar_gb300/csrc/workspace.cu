// workspace.cu -- the device workspace: one arena per (device, stream),
// bump-allocated per call; the kernels' limits of shared memory.
//
// A call needs `least` bytes and runs its faster forms where it gets `bytes`.
// The difference is asked for only as far as the device has room: at most half of
// what is free beyond the least need (the program's own allocations share the
// device), at most WB_GPU_WORKSPACE_MB where that is set, never while the stream is
// being captured, and not again after a refusal until the device has more room.

#include <algorithm>
#include <cstdlib>
#include <map>
#include <utility>

#include "common.cuh"

namespace wb {

static std::mutex g_arena_mu;
static std::map<std::pair<int, cudaStream_t>, Arena *> g_arenas;

// (arenas stay in the map for good: a call that waits for one may hold no other
// reference to it)
static Arena *arena_for(cudaStream_t s) {
    int dev = 0;
    cudaGetDevice(&dev);
    std::lock_guard<std::mutex> g(g_arena_mu);
    Arena *&a = g_arenas[std::make_pair(dev, s)];
    if (!a) a = new Arena();
    return a;
}

Workspace::Workspace(cudaStream_t stream)
    : arena_(arena_for(stream)), stream_(stream), lock_(arena_->mu) {
    arena_->used = 0;
}

Workspace::~Workspace() { arena_->used = 0; }

// most bytes that a call may get beyond its least need
static size_t optional_budget() {
    const char *e = getenv("WB_GPU_WORKSPACE_MB");
    if (!e || !*e) return SIZE_MAX;
    const double mb = atof(e);
    return mb > 0.0 ? (size_t)std::min(mb * 1048576.0, 9e18) : 0;
}

static bool capturing(cudaStream_t s) {
    cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(s, &st) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return st != cudaStreamCaptureStatusNone;
}

int Workspace::reserve(size_t bytes, size_t least) {
    if (injected(INJ_RESERVE))
        return fail(WB_ENOMEM, "cannot allocate device workspace (injected fault)");
    Arena &a = *arena_;
    a.used = 0;
    least = align256(least) + 4096;
    size_t want = std::max(align256(bytes) + 4096, least);
    const size_t budget = optional_budget();
    if (want - least > budget) want = least + budget / 256 * 256;
    if (want <= a.cap) return WB_OK;
    size_t room = 0;
    if (want > least) {
        const bool must = least > a.cap;
        if (!must && capturing(stream_)) return WB_OK;
        size_t free = 0, total = 0;
        if (must && capturing(stream_)) {
            want = least;
        } else if (cudaMemGetInfo(&free, &total) != cudaSuccess) {
            cudaGetLastError();
            want = least;
        } else {
            room = free + a.cap;
            const size_t share = room > least ? (room - least) / 2 / 256 * 256 : 0;
            const bool all = want - least <= share;
            if (!all) want = least + share;
            // (a little more room than last time is not worth a new arena)
            const bool refused = a.refused && room < a.refused + a.refused / 8;
            if (!must && (refused || want <= a.cap || (!all && want < a.cap / 4 * 5)))
                return WB_OK;
            if (refused) want = least;
        }
    }
    if (want <= a.cap) return WB_OK;
    if (a.base) {
        // cudaFree waits for the device, so earlier work on this stream that
        // still reads the arena has finished
        cudaError_t e = cudaFree(a.base);
        a.base = nullptr;
        a.cap = 0;
        if (e != cudaSuccess) return cuda_fail(e, "cudaFree(workspace)");
    }
    // some slack for later calls, then the size itself, then down to the least
    size_t cap = want + std::min(want / 4, (size_t)256 << 20);
    cudaError_t e = cudaMalloc((void **)&a.base, cap);
    while (e == cudaErrorMemoryAllocation && cap > least) {
        cudaGetLastError();
        cap = cap > want ? want : std::max(cap / 2 / 256 * 256, least);
        e = cudaMalloc((void **)&a.base, cap);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        a.base = nullptr;
        if (e != cudaErrorMemoryAllocation) return cuda_fail(e, "cudaMalloc(workspace)");
        return fail(WB_ENOMEM, "cannot allocate " + std::to_string(cap) +
                                   " bytes of device workspace");
    }
    a.cap = cap;
    if (want > least) a.refused = cap < want ? room : 0;
    return WB_OK;
}

// (asking the runtime takes some 20 us a call, so what was set is kept)
cudaError_t allow_shared(const void *kernel, size_t bytes) {
    static std::mutex mu;
    static std::map<std::pair<int, const void *>, size_t> limits;
    const DeviceInfo &dev = device_info();
    std::lock_guard<std::mutex> g(mu);
    size_t &limit = limits[std::make_pair(dev.device, kernel)];
    if (limit == 0) {
        cudaFuncAttributes at;
        cudaError_t e = cudaFuncGetAttributes(&at, kernel);
        if (e != cudaSuccess) return e;
        const int most = dev.max_smem_optin - (int)at.sharedSizeBytes;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
        if (e != cudaSuccess) return e;
        limit = (size_t)imax(most, 0);
    }
    return bytes <= limit ? cudaSuccess : cudaErrorInvalidValue;
}

}  // namespace wb

extern "C" int wb_release_workspace(void *stream_) {
    WB_TRACE();
    using namespace wb;
    std::lock_guard<std::mutex> g(g_arena_mu);
    for (auto &entry : g_arenas) {
        if (stream_ && entry.first.second != (cudaStream_t)stream_) continue;
        Arena *a = entry.second;
        std::lock_guard<std::mutex> ga(a->mu);
        if (a->base) cudaFree(a->base);
        a->base = nullptr;
        a->cap = 0;
        a->refused = 0;
    }
    return WB_OK;
}
