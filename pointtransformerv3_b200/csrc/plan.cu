// Integer bookkeeping of the hierarchy: the patch padding plan of serialized
// attention and the cluster / pooled-order plan of serialized pooling.
//
// Replaces model.py:382-438 (get_padding_and_inverse) and the index part of
// model.py:639-695 (unique / sort / cumsum / argsort / scatter_ of
// SerializedPooling.forward).  Pooled orders need no sort: children of a parent
// cell are contiguous in every order, so the pooled order of row r is the
// cluster id sequence along the fine order of row r with repeats removed.
#include <limits.h>

#include "common.cuh"
#include "plan.cuh"
#include "scan.cuh"
#include "../../include/ptv3_b200.h"

namespace ptv3 {

// ----------------------------------------------------------------------------
// padding plan
// ----------------------------------------------------------------------------
constexpr int PAD_MAX_SCENES = 4096;

// `index`: a voxel index to clear beside it (the one-call backbone's next launches on the stream fill it)
__global__ void __launch_bounds__(256) pad_plan_kernel(const int64_t* offset, int B, int K, int64_t n, int64_t n_pad,
                                                       int n_seq, int64_t* pad, int64_t* unpad, int32_t* cu_seqlens,
                                                       uint32_t* status, const VoxelClear index)
{
    extern __shared__ int64_t sm[];
    // A layout made on the main stream stands when the block after it starts: its attention looks patches up ahead of
    // its own wait (`planned`, linear.cuh).
    if (index.pairs) pdl_launch_next();
    pdl_wait();
    index.clear();
    int64_t* off = sm;                  // B + 1, unpadded scene starts
    int64_t* off_pad = sm + (B + 1);    // B + 1, padded scene starts
    int64_t* seq0 = sm + 2 * (B + 1);   // B + 1, first sequence of each scene
    if (threadIdx.x == 0) {
        off[0] = 0;
        off_pad[0] = 0;
        seq0[0] = 0;
        for (int s = 0; s < B; ++s) {
            const int64_t end = offset[s];
            const int64_t c = end - off[s];
            const int64_t cp = c > K ? (c + K - 1) / K * K : c;   // model.py:394-404
            off[s + 1] = end;
            off_pad[s + 1] = off_pad[s] + cp;
            seq0[s + 1] = seq0[s] + (cp + K - 1) / K;
        }
        if (blockIdx.x == 0 && (off[B] != n || off_pad[B] != n_pad || seq0[B] != n_seq))
            atomicOr(status, PTV3_STATUS_BAD_INDEX);
    }
    __syncthreads();
    if (off[B] != n || off_pad[B] != n_pad || seq0[B] != n_seq) return;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < n_pad; p += stride) {
        int lo = 0, hi = B;  // last s with off_pad[s] <= p
        while (hi - lo > 1) {
            const int mid = (lo + hi) >> 1;
            if (off_pad[mid] <= p) lo = mid; else hi = mid;
        }
        // scenes without points have equal starts; the search lands on the last one
        const int s = lo;
        const int64_t j = p - off_pad[s];
        const int64_t c = off[s + 1] - off[s];
        // tail of the last patch re-uses the ranks one patch earlier (model.py:412-423)
        pad[p] = off[s] + (j < c ? j : j - K);
        if (j < c) unpad[off[s] + j] = p;                          // model.py:411
        if (j % K == 0) cu_seqlens[seq0[s] + j / K] = (int32_t)p;  // model.py:424-432
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) cu_seqlens[n_seq] = (int32_t)n_pad;
}

// ----------------------------------------------------------------------------
// pooling plan
// ----------------------------------------------------------------------------
struct RowPerm {
    int src[PTV3_MAX_ORDERS];
};

// Rows of (n) keys are read in tiles of PP_THREADS x ITEMS; a warp owns 32 x ITEMS consecutive elements of its tile,
// its lanes side by side.
//
// The plan is three kernels, each a chain of few dependent loads, because on a small level it is their latency that the
// features wait for.  (As flags scanned in three launches each, first of the clusters, then of the orders, eight
// elements of a thread one after another: 6 000 points 57 us in eight launches, 16 here; the four plans of 2 M LiDAR
// points 1.6 ms, 0.49 here.)
//   pool_count_kernel     starts of runs per tile, every row.  A run is a parent cell: the codes of a row name it alike
//                         however the row is ordered, so all rows are counted at once, without the cluster ids.
//   pool_clusters_kernel  row 0: cluster ids, heads and what is read at the heads; its last block writes the sizes
//   pool_orders_kernel    every row: orders and inverses of the pooled level from the cluster ids; its last block reports,
//                         because only here it shows whether the rows belong together
// A block adds up the tiles before its own by itself up to PP_OWN_TILES; beyond, a kernel of its own scans the counts.
constexpr int PP_THREADS = 256, PP_WARPS = PP_THREADS / 32;
// Up to this size a thread takes one element (the chip has idle threads, and a block has the shortest chain), above it
// four, whose loads are in flight together.  us a plan, one / four: 3 000 points 15.5 / 18.7, 100 000 23.8 / 26.3,
// 200 000 34.8 / 32.9, 800 000 112 / 93
constexpr int64_t PP_SHORT = 1 << 17;
constexpr int PP_OWN_TILES = 4096;

// bits of `run`: elements of this warp's stretch `it` whose key differs from that of the element before
template <int ITEMS>
__device__ __forceinline__ void run_starts(const int64_t (&key)[ITEMS], int64_t before, int64_t j0, int64_t n,
                                           uint32_t (&run)[ITEMS])
{
    const int lane = threadIdx.x & 31;
    int64_t edge = before;                       // the key ahead of lane 0
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        const int64_t j = j0 + it * 32;
        int64_t prev = __shfl_up_sync(0xffffffffu, key[it], 1);
        if (lane == 0) prev = edge;
        edge = __shfl_sync(0xffffffffu, key[it], 31);
        run[it] = __ballot_sync(0xffffffffu, j < n && (j == 0 || key[it] != prev));
    }
}

template <int ITEMS>
__device__ __forceinline__ uint32_t count_runs(const uint32_t (&run)[ITEMS])
{
    uint32_t c = 0;
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) c += __popc(run[it]);
    return c;
}

// first element of this thread in the tile
template <int ITEMS>
__device__ __forceinline__ int64_t tile_element()
{
    return (int64_t)blockIdx.x * (PP_THREADS * ITEMS) + (threadIdx.x >> 5) * (32 * ITEMS) + (threadIdx.x & 31);
}

// Sums of this thread's share of a row's counts: those before `tile`, and all of them.  (Scanned counts hold the sum.)
__device__ __forceinline__ void tile_counts(const uint32_t* sums, int ntiles, int tile, bool scanned, uint32_t& ahead,
                                            uint32_t& all)
{
    ahead = all = 0;
    if (scanned) {
        if (threadIdx.x == 0) ahead = sums[tile];
        return;
    }
    for (int t = threadIdx.x; t < ntiles; t += PP_THREADS) {
        const uint32_t c = sums[t];
        all += c;
        if (t < tile) ahead += c;
    }
}

struct PoolArgs {
    const int64_t *code, *order;      // k x n
    const int32_t* grid;              // n x 3
    const int64_t* batch;             // n
    int64_t n;
    int k, shift, pooling_depth, B, ntiles;
    bool scanned;                     // tile_sums hold exclusive sums, totals their ends
    RowPerm perm;
    uint32_t *tile_sums, *totals;     // k x ntiles, by source row; k
    unsigned long long* scene_count;  // B
    uint32_t* done;                   // blocks of pool_clusters_kernel and of pool_orders_kernel that are through
    int64_t *cluster, *idx_ptr, *head, *pcode, *porder, *pinverse, *pbatch, *meta, *meta_host, *offset;
    int32_t *pgrid, *indices;         // indices: (batch, x, y, z) rows of the pooled level, or NULL
    uint32_t* status;
};

template <int ITEMS>
__global__ void __launch_bounds__(PP_THREADS) pool_count_kernel(const __grid_constant__ PoolArgs a)
{
    __shared__ uint32_t warp_runs[PP_WARPS];
    pdl_launch_next();
    pdl_wait();
    const int row = blockIdx.y, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t* order = a.order + (int64_t)row * a.n;
    const int64_t* code = a.code + (int64_t)row * a.n;
    if (blockIdx.x == 0 && row == 0) {
        for (int b = threadIdx.x; b < a.B; b += PP_THREADS) a.scene_count[b] = 0;
        if (threadIdx.x < 2) a.done[threadIdx.x] = 0;
    }
    const int64_t j0 = tile_element<ITEMS>();
    int64_t p[ITEMS], key[ITEMS], before = 0;
    const bool edge = lane == 0 && j0 > 0 && j0 - 1 < a.n;
    if (edge) before = order[j0 - 1];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) p[it] = j0 + it * 32 < a.n ? order[j0 + it * 32] : -1;
    if (edge) before = code[before] >> a.shift;
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) key[it] = p[it] >= 0 ? code[p[it]] >> a.shift : 0;
    uint32_t run[ITEMS];
    run_starts<ITEMS>(key, before, j0, a.n, run);
    if (lane == 0) warp_runs[warp] = count_runs<ITEMS>(run);
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t c = 0;
#pragma unroll
        for (int w = 0; w < PP_WARPS; ++w) c += warp_runs[w];
        a.tile_sums[(int64_t)row * a.ntiles + blockIdx.x] = c;
    }
}

template <int ITEMS>
__global__ void __launch_bounds__(PP_THREADS) pool_clusters_kernel(const __grid_constant__ PoolArgs a)
{
    __shared__ uint32_t warp_runs[PP_WARPS], sum_ahead, sum_all, same_scene;
    __shared__ bool last;
    if (threadIdx.x == 0) sum_ahead = sum_all = same_scene = 0;
    pdl_launch_next();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t n = a.n, j0 = tile_element<ITEMS>();
    // row 0: points along its order, with their parent cells
    int64_t p[ITEMS], key[ITEMS], before = 0;
    const bool edge = lane == 0 && j0 > 0 && j0 - 1 < n;
    if (edge) before = a.order[j0 - 1];
    const int64_t p_first = a.order[(int64_t)blockIdx.x * (PP_THREADS * ITEMS)];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) p[it] = j0 + it * 32 < n ? a.order[j0 + it * 32] : -1;
    if (edge) before = a.code[before] >> a.shift;
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) key[it] = p[it] >= 0 ? a.code[p[it]] >> a.shift : 0;
    const int64_t scene = a.batch[p_first];          // of the tile's first point: most of a tile shares it
    uint32_t ahead, all;
    tile_counts(a.tile_sums, a.ntiles, blockIdx.x, a.scanned, ahead, all);
    uint32_t run[ITEMS];
    run_starts<ITEMS>(key, before, j0, n, run);
    // what is read at a head; the codes of four rows at a time
    int64_t b[ITEMS], c[4][ITEMS];
    int32_t g[ITEMS][3];
    bool f[ITEMS];
    auto load_codes = [&](int r0) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int it = 0; it < ITEMS; ++it)
                c[r][it] = f[it] && r0 + r < a.k ? a.code[(int64_t)a.perm.src[r0 + r] * n + p[it]] : 0;
    };
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        f[it] = (run[it] >> lane) & 1;
        b[it] = f[it] ? a.batch[p[it]] : 0;
#pragma unroll
        for (int x = 0; x < 3; ++x) g[it][x] = f[it] ? a.grid[3 * p[it] + x] >> a.pooling_depth : 0;
    }
    load_codes(0);
    __syncthreads();
    ahead = __reduce_add_sync(0xffffffffu, ahead);
    all = __reduce_add_sync(0xffffffffu, all);
    if (lane == 0) {
        atomicAdd(&sum_ahead, ahead);
        atomicAdd(&sum_all, all);
        warp_runs[warp] = count_runs<ITEMS>(run);
    }
    __syncthreads();
    const int64_t m = a.scanned ? a.totals[0] : sum_all;
    uint32_t pos = sum_ahead;
    for (int w = 0; w < warp; ++w) pos += warp_runs[w];
    const uint32_t below = (1u << lane) - 1;
    int64_t cid[ITEMS];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        cid[it] = (int64_t)pos + __popc(run[it] & below) + (f[it] ? 1 : 0) - 1;
        pos += __popc(run[it]);
        if (p[it] >= 0) a.cluster[p[it]] = cid[it];
    }
#pragma unroll 1
    for (int r0 = 0; r0 < a.k; r0 += 4) {
        if (r0) load_codes(r0);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int it = 0; it < ITEMS; ++it)
                if (f[it] && r0 + r < a.k) a.pcode[(int64_t)(r0 + r) * m + cid[it]] = c[r][it] >> a.shift;
    }
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        // clusters per scene: those of the tile's first scene are added up in the block
        const uint32_t same = __ballot_sync(0xffffffffu, f[it] && b[it] == scene);
        if (lane == 0 && same) atomicAdd(&same_scene, __popc(same));
        if (!f[it]) continue;
        const int64_t j = j0 + it * 32, c = cid[it];
        a.idx_ptr[c] = j;
        a.head[c] = p[it];
        a.pbatch[c] = b[it];
#pragma unroll
        for (int x = 0; x < 3; ++x) a.pgrid[3 * c + x] = g[it][x];
        if (a.indices) reinterpret_cast<int4*>(a.indices)[c] = make_int4((int)b[it], g[it][0], g[it][1], g[it][2]);
        if (b[it] != scene) {
            if ((unsigned long long)b[it] < (unsigned long long)a.B)
                atomicAdd(&a.scene_count[b[it]], 1ull);
            else       // a number that the offsets know nothing of: it has no counter
                atomicOr(a.status, PTV3_STATUS_BAD_INDEX);
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        if (same_scene) {
            if ((unsigned long long)scene < (unsigned long long)a.B)
                atomicAdd(&a.scene_count[scene], (unsigned long long)same_scene);
            else
                atomicOr(a.status, PTV3_STATUS_BAD_INDEX);
        }
        __threadfence();
        last = atomicAdd(a.done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    // the last block: every row must have as many runs as row 0
    for (int r = 1 + warp; r < a.k; r += PP_WARPS) {
        const uint32_t* sums = a.tile_sums + (int64_t)r * a.ntiles;
        uint32_t runs = 0;
        if (a.scanned) {
            runs = a.totals[r];
        } else {
#pragma unroll 8
            for (int t = lane; t < a.ntiles; t += 32) runs += sums[t];
            runs = __reduce_add_sync(0xffffffffu, runs);
        }
        if (lane == 0 && (int64_t)runs != m) atomicOr(a.status, PTV3_STATUS_BAD_INDEX);
    }
    __threadfence();
    __syncthreads();
    if (warp != 0) return;
    if (lane == 0) {
        a.idx_ptr[m] = n;
        a.meta[0] = m;
    }
    int64_t end = 0;
    for (int s0 = 0; s0 < a.B; s0 += 32) {
        const int s = s0 + lane;
        const int64_t own =
            s < a.B ? (int64_t)*reinterpret_cast<volatile unsigned long long*>(&a.scene_count[s]) : 0;
        int64_t upto = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int64_t u = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += u;
        }
        if (s < a.B) {
            a.meta[1 + s] = own;
            if (a.offset) a.offset[s] = end + upto;
            if (a.meta_host) a.meta_host[1 + s] = own;
        }
        end += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (!a.meta_host) return;
    // (the same numbers go straight into the caller's mapped host memory: a copy would queue behind whatever else the copy
    // engine is busy with)
    if (lane == 0) a.meta_host[0] = m;
    __threadfence_system();
}

template <int ITEMS>
__global__ void __launch_bounds__(PP_THREADS) pool_orders_kernel(const __grid_constant__ PoolArgs a)
{
    __shared__ uint32_t warp_runs[PP_WARPS], sum_ahead;
    if (threadIdx.x == 0) sum_ahead = 0;
    pdl_launch_next();
    pdl_wait();
    const int r = blockIdx.y, src = a.perm.src[r], lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t n = a.n, j0 = tile_element<ITEMS>();
    const int64_t* order = a.order + (int64_t)src * n;
    int64_t key[ITEMS], before = 0;
    const bool edge = lane == 0 && j0 > 0 && j0 - 1 < n;
    if (edge) before = order[j0 - 1];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) key[it] = j0 + it * 32 < n ? order[j0 + it * 32] : -1;
    if (edge) before = a.cluster[before];
#pragma unroll
    for (int it = 0; it < ITEMS; ++it)
        if (key[it] >= 0) key[it] = a.cluster[key[it]];
    const int64_t m = a.meta[0];
    const uint32_t* sums = a.tile_sums + (int64_t)src * a.ntiles;
    uint32_t ahead, all;
    tile_counts(sums, a.ntiles, blockIdx.x, a.scanned, ahead, all);
    uint32_t run[ITEMS];
    run_starts<ITEMS>(key, before, j0, n, run);
    __syncthreads();
    ahead = __reduce_add_sync(0xffffffffu, ahead);
    if (lane == 0) {
        atomicAdd(&sum_ahead, ahead);
        warp_runs[warp] = count_runs<ITEMS>(run);
    }
    __syncthreads();
    uint32_t pos = sum_ahead, mine = 0;
#pragma unroll
    for (int w = 0; w < PP_WARPS; ++w) {
        if (w < warp) pos += warp_runs[w];
        mine += warp_runs[w];
    }
    if (threadIdx.x == 0) {
        // runs of cluster ids are the runs of codes that were counted, or the rows do not belong together
        const uint32_t counted = !a.scanned ? sums[blockIdx.x]
                                 : (int)blockIdx.x + 1 < a.ntiles ? sums[blockIdx.x + 1] - sums[blockIdx.x]
                                                                  : a.totals[src] - sums[blockIdx.x];
        if (mine != counted) atomicOr(a.status, PTV3_STATUS_BAD_INDEX);
        if (a.meta_host) {
            // Whoever comes last has every check behind it, and the kernel before has stored the sizes: now the status word
            // goes to the host, then "everything has been stored".  A host that zeroed this word before the call may poll
            // it instead of waiting for the stream.
            __threadfence();
            if (atomicAdd(a.done + 1, 1u) == gridDim.x * gridDim.y - 1) {
                __threadfence();
                a.meta_host[1 + a.B] = (int64_t)atomicOr(a.status, 0u);
                __threadfence_system();
                *reinterpret_cast<volatile int64_t*>(&a.meta_host[2 + a.B]) = 1;
                __threadfence_system();
            }
        }
    }
    const uint32_t below = (1u << lane) - 1;
#pragma unroll
    for (int it = 0; it < ITEMS; ++it) {
        if ((run[it] >> lane) & 1) {
            const int64_t at = (int64_t)pos + __popc(run[it] & below);
            a.porder[(int64_t)r * m + at] = key[it];
            a.pinverse[(int64_t)r * m + key[it]] = at;
        }
        pos += __popc(run[it]);
    }
}

struct PoolWs {
    int items, ntiles;
    size_t bytes;
};
static PoolWs pool_ws(int k, int64_t n, int B)
{
    PoolWs w;
    w.items = n <= PP_SHORT ? 1 : 4;
    w.ntiles = ceil_div(n, (int64_t)PP_THREADS * w.items);
    w.bytes = align_up((size_t)k * w.ntiles * sizeof(uint32_t), 256) + align_up((size_t)k * sizeof(uint32_t), 256) +
              align_up((size_t)B * sizeof(unsigned long long), 256) + 256;
    return w;
}

template <int ITEMS>
static int launch_pool_plan(const PoolArgs& a, cudaStream_t stream)
{
    const dim3 rows(a.ntiles, a.k);
    launch_dependent(pool_count_kernel<ITEMS>, rows, dim3(PP_THREADS), 0, stream, a);
    if (a.scanned) scan_sums_kernel<<<a.k, SC_THREADS, 0, stream>>>(a.tile_sums, a.ntiles, a.totals);
    launch_dependent(pool_clusters_kernel<ITEMS>, dim3(a.ntiles), dim3(PP_THREADS), 0, stream, a);
    launch_dependent(pool_orders_kernel<ITEMS>, rows, dim3(PP_THREADS), 0, stream, a);
    count_launches(a.scanned ? 4 : 3);
    return check_launch("ptv3_pool_plan");
}

// ----------------------------------------------------------------------------
// batch index of every point from the scene offsets, and the (batch, x, y, z) rows
// of the sparse tensor (model.py:35-40 and :150-152)
// ----------------------------------------------------------------------------
// NORMS: the last blocks turn a BatchNorm layer each into scale and shift, which costs a pass no launch of its own
struct NoNorms {};
__device__ __forceinline__ int norm_blocks(const NoNorms&) { return 0; }
__device__ __forceinline__ int norm_blocks(const BnJobs& norms) { return norms.count; }
__device__ __forceinline__ void norm_block(const NoNorms&, int) {}
__device__ __forceinline__ void norm_block(const BnJobs& norms, int i) { bn_layer(norms, i); }

template <typename Norms>
__global__ void __launch_bounds__(256) batch_indices_kernel(const int64_t* __restrict__ offset, int B,
                                                            const int32_t* __restrict__ grid_coord, int64_t n,
                                                            int64_t* __restrict__ batch, int32_t* __restrict__ indices,
                                                            const VoxelClear index,
                                                            const __grid_constant__ Norms norms)
{
    extern __shared__ int64_t sm[];      // B scene ends
    index.clear();
    const int blocks = (int)gridDim.x - norm_blocks(norms);
    if ((int)blockIdx.x >= blocks) {
        norm_block(norms, (int)blockIdx.x - blocks);
        return;
    }
    for (int s = threadIdx.x; s < B; s += blockDim.x) sm[s] = offset[s];
    __syncthreads();
    const int64_t stride = (int64_t)blocks * blockDim.x;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
        int lo = 0, hi = B - 1;          // first scene whose end lies beyond i (the last one at worst)
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (sm[mid] > i) hi = mid; else lo = mid + 1;
        }
        if (batch) batch[i] = lo;
        if (indices)
            reinterpret_cast<int4*>(indices)[i] =
                make_int4(lo, grid_coord[3 * i], grid_coord[3 * i + 1], grid_coord[3 * i + 2]);
    }
}

constexpr int BS_CLEARED = (int)0x80808080;       // scratch words before the kernel: below every coordinate

// Largest coordinate per axis, NUMBERED: and largest scene number (as 32 bits); the block that finishes last stores
// them, with the offsets, in host memory.  A thread has four points on their way at once, and a block adds one maximum
// per value: the call is waited for, so its time is that of one chain of loads and of the atomics on one address (one
// point at a time and a maximum per warp: 100 000 points 8.9 us, 8.0 so, 400 000 13.9 and 8.5, 8 M 23.1 and 16.8; with
// the scene numbers 8.1, 8.8 and 30.3).
template <bool NUMBERED>
__global__ void __launch_bounds__(256) batch_stats_kernel(const int32_t* __restrict__ grid_coord,
                                                          const int64_t* __restrict__ batch, int64_t n,
                                                          const int64_t* __restrict__ offset, int B,
                                                          int32_t* __restrict__ scratch, int64_t* out_host)
{
    // scratch: three maxima, the count of blocks, the fourth maximum
    constexpr int VALUES = NUMBERED ? 4 : 3, AHEAD = 4;
    __shared__ int32_t top[VALUES];
    __shared__ bool last;
    if (threadIdx.x < VALUES) top[threadIdx.x] = INT_MIN;
    int32_t mx[VALUES];
#pragma unroll
    for (int a = 0; a < VALUES; ++a) mx[a] = INT_MIN;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i0 < n; i0 += AHEAD * stride) {
        int32_t g[AHEAD][3];
        int64_t number[AHEAD];
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) {
            const int64_t i = i0 + q * stride;
#pragma unroll
            for (int a = 0; a < 3; ++a) g[q][a] = i < n ? grid_coord[3 * i + a] : INT_MIN;
            number[q] = NUMBERED && i < n ? batch[i] : INT_MIN;
        }
#pragma unroll
        for (int q = 0; q < AHEAD; ++q) {
#pragma unroll
            for (int a = 0; a < 3; ++a) mx[a] = max(mx[a], g[q][a]);
            if (NUMBERED) mx[VALUES - 1] = max(mx[VALUES - 1], (int32_t)min(max(number[q], (int64_t)INT_MIN), (int64_t)INT_MAX));
        }
    }
    __syncthreads();
#pragma unroll
    for (int a = 0; a < VALUES; ++a) {
        const int32_t v = __reduce_max_sync(0xffffffffu, mx[a]);
        if ((threadIdx.x & 31) == 0) atomicMax(&top[a], v);
    }
    __syncthreads();
    if (threadIdx.x < VALUES) {
        atomicMax(&scratch[threadIdx.x < 3 ? threadIdx.x : 4], top[threadIdx.x]);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&scratch[3], 1) == BS_CLEARED + (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    for (int b = threadIdx.x; b < B; b += blockDim.x) out_host[VALUES + b] = offset[b];
    if (threadIdx.x <= VALUES) {      // read, and left as the next call wants to find them
        const int32_t v = atomicExch(&scratch[threadIdx.x], BS_CLEARED);
        if (threadIdx.x != 3) out_host[threadIdx.x < 3 ? threadIdx.x : 3] = v;
    }
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) {
        *reinterpret_cast<volatile int64_t*>(&out_host[VALUES + B]) = 1;
        __threadfence_system();
    }
}

static int check_batch_indices(const int64_t* offset, int n_scenes, const int32_t* grid_coord, int64_t n,
                               const int32_t* indices)
{
    PTV3_REQUIRE(n_scenes >= 1 && n_scenes <= PAD_MAX_SCENES, PTV3_ERR_UNSUPPORTED,
                 "ptv3_batch_indices: %d scenes outside [1, %d]", n_scenes, PAD_MAX_SCENES);
    PTV3_REQUIRE(n >= 0, PTV3_ERR_INVALID_ARGUMENT, "ptv3_batch_indices: n < 0");
    PTV3_REQUIRE(n == 0 || (offset && (!indices || grid_coord)), PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_batch_indices: null pointer");
    PTV3_REQUIRE(((uintptr_t)indices & 15) == 0, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_batch_indices: indices must be 16-byte aligned");
    return PTV3_OK;
}

static unsigned batch_indices_blocks(int64_t n) { return (unsigned)((n + 255) / 256 > SMS * 8 ? SMS * 8 : (n + 255) / 256); }

int batch_indices_and_norms(const int64_t* offset, int n_scenes, const int32_t* grid_coord, int64_t n, int32_t* indices,
                            const VoxelClear& index, const BnJobs& norms, cudaStream_t stream)
{
    const int rc = check_batch_indices(offset, n_scenes, grid_coord, n, indices);
    if (rc != PTV3_OK) return rc;
    batch_indices_kernel<<<batch_indices_blocks(n) + norms.count, 256, (size_t)n_scenes * sizeof(int64_t), stream>>>(
        offset, n_scenes, grid_coord, n, nullptr, indices, index, norms);
    count_launches(1);
    return check_launch("ptv3_batch_indices");
}

}  // namespace ptv3

static int launch_batch_stats(const int32_t* grid_coord, const int64_t* batch, int64_t n, const int64_t* offset,
                              int n_scenes, int64_t* out_host, void* scratch, cudaStream_t stream, const char* what)
{
    using namespace ptv3;
    PTV3_REQUIRE(n >= 0 && n_scenes >= 1, PTV3_ERR_INVALID_ARGUMENT, "%s: bad sizes", what);
    PTV3_REQUIRE((grid_coord || n == 0) && offset && out_host && scratch, PTV3_ERR_INVALID_ARGUMENT,
                 "%s: null pointer", what);
    int64_t blocks = (n + 1023) / 1024;         // four points per thread, at most four blocks per SM
    if (blocks < 1) blocks = 1;
    if (blocks > SMS * 4) blocks = SMS * 4;
    (batch ? batch_stats_kernel<true> : batch_stats_kernel<false>)<<<(unsigned)blocks, 256, 0, stream>>>(
        grid_coord, batch, n, offset, n_scenes, (int32_t*)scratch, out_host);
    count_launches(1);
    return check_launch(what);
}

extern "C" int ptv3_batch_stats(const int32_t* grid_coord, int64_t n, const int64_t* offset, int n_scenes,
                                int64_t* out_host, void* scratch, void* stream)
{
    return launch_batch_stats(grid_coord, nullptr, n, offset, n_scenes, out_host, scratch, (cudaStream_t)stream,
                              "ptv3_batch_stats");
}

extern "C" int ptv3_scene_stats(const int32_t* grid_coord, const int64_t* batch, int64_t n, const int64_t* offset,
                                int n_scenes, int64_t* out_host, void* scratch, void* stream)
{
    PTV3_REQUIRE(batch, PTV3_ERR_INVALID_ARGUMENT, "ptv3_scene_stats: null pointer");
    return launch_batch_stats(grid_coord, batch, n, offset, n_scenes, out_host, scratch, (cudaStream_t)stream,
                              "ptv3_scene_stats");
}

extern "C" int ptv3_batch_indices(const int64_t* offset, int n_scenes, const int32_t* grid_coord, int64_t n,
                                  int64_t* batch, int32_t* indices, void* stream)
{
    using namespace ptv3;
    if (n == 0 || (n > 0 && !batch && !indices)) return check_batch_indices(offset, n_scenes, grid_coord, 0, nullptr);
    const int rc = check_batch_indices(offset, n_scenes, grid_coord, n, indices);
    if (rc != PTV3_OK) return rc;
    batch_indices_kernel<<<batch_indices_blocks(n), 256, (size_t)n_scenes * sizeof(int64_t), (cudaStream_t)stream>>>(
        offset, n_scenes, grid_coord, n, batch, indices, VoxelClear{}, NoNorms());
    count_launches(1);
    return check_launch("ptv3_batch_indices");
}

int ptv3::pad_plan(const int64_t* offset, int n_scenes, int patch, int64_t n, int64_t n_pad, int n_seq, int64_t* pad,
                   int64_t* unpad, int32_t* cu_seqlens, uint32_t* status, const VoxelClear& index, cudaStream_t stream)
{
    PTV3_REQUIRE(n_scenes >= 1 && n_scenes <= PAD_MAX_SCENES, PTV3_ERR_UNSUPPORTED,
                 "ptv3_pad_plan: %d scenes outside [1, %d]", n_scenes, PAD_MAX_SCENES);
    PTV3_REQUIRE(patch >= 1 && n >= 0 && n_pad >= n && n_seq >= 0, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_pad_plan: bad sizes");
    PTV3_REQUIRE(offset && cu_seqlens && status && (n_pad == 0 || (pad && unpad)),
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_pad_plan: null pointer");
    const int64_t most = n_pad > index.pairs ? n_pad : index.pairs;
    int64_t blocks = (most + 255) / 256;
    if (blocks < 1) blocks = 1;
    if (blocks > SMS * 8) blocks = SMS * 8;
    const size_t smem = 3 * (size_t)(n_scenes + 1) * sizeof(int64_t);
    launch_dependent(pad_plan_kernel, dim3((unsigned)blocks), dim3(256), smem, stream, offset, n_scenes, patch, n, n_pad,
                     n_seq, pad, unpad, cu_seqlens, status, index);
    count_launches(1);
    return check_launch("ptv3_pad_plan");
}

extern "C" int ptv3_pad_plan(const int64_t* offset, int n_scenes, int patch, int64_t n, int64_t n_pad,
                             int n_seq, int64_t* pad, int64_t* unpad, int32_t* cu_seqlens,
                             uint32_t* status, void* stream)
{
    return ptv3::pad_plan(offset, n_scenes, patch, n, n_pad, n_seq, pad, unpad, cu_seqlens, status, ptv3::VoxelClear{},
                          (cudaStream_t)stream);
}

extern "C" size_t ptv3_pool_plan_workspace_bytes(int k, int64_t n, int n_scenes)
{
    if (k <= 0 || n <= 0 || n_scenes <= 0) return 0;
    return ptv3::pool_ws(k, n, n_scenes).bytes;
}

int ptv3::pool_plan(const int64_t* code, const int64_t* order, const int32_t* grid_coord, const int64_t* batch, int k,
                    int64_t n, int n_scenes, int pooling_depth, const int* row_perm, int64_t* cluster,
                    int64_t* idx_ptr, int64_t* head, int64_t* pooled_code, int64_t* pooled_order,
                    int64_t* pooled_inverse, int32_t* pooled_grid_coord, int64_t* pooled_batch, int64_t* meta,
                    int64_t* meta_host, int64_t* pooled_offset, int32_t* pooled_indices, uint32_t* status,
                    void* workspace, size_t workspace_bytes, cudaStream_t stream)
{
    PTV3_REQUIRE(k >= 1 && k <= PTV3_MAX_ORDERS && n >= 1 && n_scenes >= 1,
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_pool_plan: bad k/n/n_scenes");
    PTV3_REQUIRE(pooling_depth >= 0 && pooling_depth <= 16, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_pool_plan: bad pooling_depth");
    PTV3_REQUIRE(n < (1ll << 31), PTV3_ERR_UNSUPPORTED, "ptv3_pool_plan: n too large");
    PTV3_REQUIRE(code && order && grid_coord && batch && cluster && idx_ptr && head && pooled_code &&
                     pooled_order && pooled_inverse && pooled_grid_coord && pooled_batch && meta &&
                     status && workspace,
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_pool_plan: null pointer");
    const PoolWs w = pool_ws(k, n, n_scenes);
    PTV3_REQUIRE(workspace_bytes >= w.bytes, PTV3_ERR_WORKSPACE,
                 "ptv3_pool_plan: workspace %zu < %zu bytes", workspace_bytes, w.bytes);
    PoolArgs a{};
    for (int r = 0; r < PTV3_MAX_ORDERS; ++r) a.perm.src[r] = r < k ? (row_perm ? row_perm[r] : r) : 0;
    for (int r = 0; r < k; ++r)
        PTV3_REQUIRE(a.perm.src[r] >= 0 && a.perm.src[r] < k, PTV3_ERR_INVALID_ARGUMENT,
                     "ptv3_pool_plan: row_perm[%d] = %d outside [0, %d)", r, a.perm.src[r], k);
    Carver cv(workspace);
    a.tile_sums = cv.take<uint32_t>((size_t)k * w.ntiles);
    a.totals = cv.take<uint32_t>(k);
    a.scene_count = cv.take<unsigned long long>(n_scenes);
    a.done = cv.take<uint32_t>(2);
    a.code = code;
    a.order = order;
    a.grid = grid_coord;
    a.batch = batch;
    a.n = n;
    a.k = k;
    a.shift = 3 * pooling_depth;
    a.pooling_depth = pooling_depth;
    a.B = n_scenes;
    a.ntiles = w.ntiles;
    a.scanned = w.ntiles > PP_OWN_TILES;
    a.cluster = cluster;
    a.idx_ptr = idx_ptr;
    a.head = head;
    a.pcode = pooled_code;
    a.porder = pooled_order;
    a.pinverse = pooled_inverse;
    a.pgrid = pooled_grid_coord;
    a.pbatch = pooled_batch;
    a.indices = pooled_indices;
    a.meta = meta;
    a.meta_host = meta_host;
    a.offset = pooled_offset;
    a.status = status;
    return w.items == 1 ? launch_pool_plan<1>(a, stream) : launch_pool_plan<4>(a, stream);
}

extern "C" int ptv3_pool_plan(const int64_t* code, const int64_t* order, const int32_t* grid_coord,
                              const int64_t* batch, int k, int64_t n, int n_scenes,
                              int pooling_depth, const int* row_perm, int64_t* cluster,
                              int64_t* idx_ptr, int64_t* head, int64_t* pooled_code,
                              int64_t* pooled_order, int64_t* pooled_inverse,
                              int32_t* pooled_grid_coord, int64_t* pooled_batch, int64_t* meta,
                              int64_t* meta_host, uint32_t* status, void* workspace,
                              size_t workspace_bytes, void* stream)
{
    return ptv3::pool_plan(code, order, grid_coord, batch, k, n, n_scenes, pooling_depth, row_perm, cluster, idx_ptr,
                           head, pooled_code, pooled_order, pooled_inverse, pooled_grid_coord, pooled_batch, meta,
                           meta_host, nullptr, nullptr, status, workspace, workspace_bytes, (cudaStream_t)stream);
}
