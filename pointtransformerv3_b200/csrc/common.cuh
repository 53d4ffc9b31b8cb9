// Shared helpers of the sm_100a kernel library: status codes, the thread-local
// error string behind ptv3_last_error(), launch checking and small device
// utilities.  The library never allocates device memory (one documented entry
// point uses a static device array instead); callers pass outputs and
// workspaces.
#pragma once
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/ptv3_b200.h"

namespace ptv3 {

void set_error(const char* fmt, ...);
int check_launch(const char* what);
// Adds to the process-wide count of kernels this library has launched
// (read through ptv3_launch_count()).
void count_launches(int n);
// polls a word of mapped host memory until a kernel of `stream` has stored it (see ptv3_host_wait)
int host_wait(const int64_t* word, cudaStream_t stream);

#define PTV3_REQUIRE(cond, code, ...)            \
    do {                                         \
        if (!(cond)) {                           \
            ::ptv3::set_error(__VA_ARGS__);      \
            return (code);                       \
        }                                        \
    } while (0)

static inline size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Carves a caller-provided workspace into 256-byte aligned pieces.
struct Carver {
    char* base;
    size_t off;
    explicit Carver(void* p) : base(static_cast<char*>(p)), off(0) {}
    template <typename T>
    T* take(size_t count) {
        T* p = reinterpret_cast<T*>(base + off);
        off += align_up(count * sizeof(T), 256);
        return p;
    }
};

// streaming multiprocessors of a B200: grids and the lines of dispatch rules are stated in them
constexpr int SMS = 148;

static inline int ceil_div(int64_t a, int64_t b) { return static_cast<int>((a + b - 1) / b); }

// ---- programmatic dependent launch -------------------------------------------------------------
// A forward is a chain of a few hundred kernels on one stream, many of them a few microseconds
// long.  A kernel launched with launch_dependent() may be scheduled while the kernel before it in
// the stream still runs; it must call pdl_wait() before it touches anything that kernel wrote (all
// such kernels here call it first thing), and pdl_launch_next() tells the scheduler that the
// kernel after it may be brought up.  The launch latency and the start-up of a kernel then overlap
// the tail of its predecessor.
//
// Such a kernel takes plain pointers: the memory clobber of the wait holds back loads through those.  A load through
// const __restrict__ or by __ldg says that nobody writes there while the kernel runs; it may be moved ahead of the
// wait, and takes the path that is not kept coherent with the kernel ahead.  (Voxelisation read slots before they were
// written that way, an illegal address.)  What the compiler then no longer moves by itself stands early in the source:
// the MLP's residual rows, for one (400 000 x 64: 74 us; 91 where they were asked for as they were stored).
#ifdef __CUDACC__
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... KArgs, typename... Args>
static inline cudaError_t launch_dependent_cluster(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                                   cudaStream_t stream, dim3 cluster, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster.x;
    attr[1].val.clusterDim.y = cluster.y;
    attr[1].val.clusterDim.z = cluster.z;
    cfg.attrs = attr;
    cfg.numAttrs = cluster.x * cluster.y * cluster.z > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}
template <typename... KArgs, typename... Args>
static inline cudaError_t launch_dependent(void (*kern)(KArgs...), dim3 grid, dim3 block, size_t smem,
                                           cudaStream_t stream, Args... args)
{
    return launch_dependent_cluster(kern, grid, block, smem, stream, dim3(1, 1, 1), args...);
}

// Lets a kernel take all the shared memory of an SM that its static part leaves, asked for once per thread,
// device and kernel: the driver call costs as much as a third of a launch.  (Always the same value, so that
// threads do not undo one another's.)
template <typename K>
static inline cudaError_t allow_smem(K kern)
{
    struct Seen {
        const void* kern;
        int device;
    };
    static thread_local Seen seen[16] = {};      // kernels of one signature share an instance
    static thread_local int next = 0;
    int device = -1;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    for (const Seen& s : seen)
        if (s.kern == (const void*)kern && s.device == device) return cudaSuccess;
    cudaFuncAttributes attr;
    e = cudaFuncGetAttributes(&attr, (const void*)kern);
    if (e != cudaSuccess) return e;
    e = cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             227 * 1024 - (int)attr.sharedSizeBytes);
    if (e == cudaSuccess) {
        seen[next] = Seen{(const void*)kern, device};
        next = (next + 1) % 16;
    }
    return e;
}
#endif

}  // namespace ptv3
