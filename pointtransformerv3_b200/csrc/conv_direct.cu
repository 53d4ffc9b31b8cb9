// Submanifold convolution with few input channels and a large kernel (the 5x5x5
// stem, model.py:766-779) without a kernel map: the neighbour table of such a
// convolution (125 x N int32) is several times larger than its input and its
// output, so the voxel hash table is probed inside the convolution instead.
//
// The voxels are indexed in two levels: a hash table of 4 x 4 x 4 blocks whose
// values point at 64-entry cell tables (cell -> row).  A CTA owns 128 voxels:
// each voxel first looks up the (at most 8) blocks its neighbourhood touches,
// then the kernel offsets are walked 25 at a time; in each round the 256 threads
// read 25 x 128 neighbour rows from the cell tables and gather the features of
// the neighbours found into shared memory (all independent, latencies overlap);
// then thread (voxel, half) accumulates half of the output channels in fp32
// registers, reading the weights (staged once per CTA) as warp-wide broadcasts
// and skipping absent neighbours.
// Epilogue: optional bias, optional BatchNorm(eval) scale/shift + exact GELU
// (model.py:848,860 for the stem), rounding, one contiguous store per thread.
//
// bf16 features take the tensor-core form of the same kernel (conv_direct_tc05_kernel):
// the staged neighbour rows of a few (dx, dy) rows of offsets are the A operand (128 voxels x K = offsets x 8
// padded channels, zero rows where a neighbour is absent) of tcgen05.mma against that
// round's slice of the weights; nothing is skipped because the products are cheap - the
// CUDA-core form spends most of its instructions unpacking bf16 weights for the FMAs.
#include <algorithm>

#include "common.cuh"
#include "convert.cuh"
#include "kmap.cuh"
#include "mma_util.cuh"
#include "tc05.cuh"
#include "voxel_index.cuh"
#include "plan.cuh"
#include "vec.cuh"

namespace ptv3 {

constexpr int CD_TM = 128;
constexpr int CD_THREADS = 256;
constexpr int CD_MAX_CIN = 8;

__device__ __forceinline__ float cd_gelu(float x)
{
    return 0.5f * x * (1.f + erff(x * 0.70710678118654752440f));
}

constexpr int CD_CHUNK = 25;   // kernel offsets staged per round

// [cout][kvol][cin] -> [kvol][cin][cout], once per call (a few thousand elements)
template <typename T>
__global__ void conv_direct_transpose_kernel(const T* __restrict__ w, T* __restrict__ wt, int cout,
                                             int kvol, int cin)
{
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= cout * kvol * cin) return;
    const int ci = idx % cin, rest = idx / cin;
    const int o = rest % kvol, co = rest / kvol;
    wt[((size_t)o * cin + ci) * cout + co] = w[idx];
}

// CO: output channels per thread (c_out = 2 * CO)
template <typename T, int CO>
__global__ void __launch_bounds__(CD_THREADS) conv_direct_kernel(
    const T* __restrict__ feat, const int32_t* __restrict__ indices, const T* __restrict__ weight,
    const T* __restrict__ bias, const float* __restrict__ bn_scale, const float* __restrict__ bn_shift,
    int apply_gelu, T* __restrict__ out, const int64_t* __restrict__ row_order, int64_t n, int cin,
    int ksize, const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ vals,
    uint64_t cap_mask, const uint32_t* __restrict__ cells, uint32_t* __restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const int kvol = ksize * ksize * ksize;
    const int cout = 2 * CO;
    // staged neighbour features of one round: [CD_CHUNK][128][CD_MAX_CIN], zero where absent
    T* x_s = reinterpret_cast<T*>(smem);
    unsigned char* has_s = smem + (size_t)CD_CHUNK * CD_TM * CD_MAX_CIN * sizeof(T);   // [CD_CHUNK][128]
    T* w_s = reinterpret_cast<T*>(has_s + CD_CHUNK * CD_TM);                            // kvol x cin x cout
    __shared__ int4 coord_s[CD_TM];
    __shared__ uint32_t block_s[8][CD_TM];   // table id of the 2 x 2 x 2 blocks around each voxel
    __shared__ char4 delta_s[343];           // (dx, dy, dz) of every kernel offset

    const int tid = threadIdx.x;
    const int v = tid % CD_TM, half = tid / CD_TM;
    const int64_t i = (int64_t)blockIdx.x * CD_TM + v;
    const int64_t row = i < n ? (row_order ? row_order[i] : i) : -1;
    const int r = ksize / 2;
    const int4 c = row >= 0 ? reinterpret_cast<const int4*>(indices)[row] : make_int4(-1, 0, 0, 0);
    if (half == 0) coord_s[v] = c;
    for (int o = tid; o < kvol; o += CD_THREADS)
        delta_s[o] = make_char4((char)(o / (ksize * ksize) - r), (char)((o / ksize) % ksize - r),
                                (char)(o % ksize - r), 0);
    // weights, already transposed to [kvol][cin][cout]: straight 16-byte copy
    {
        const int nvec = kvol * cin * cout / Vec<T>::N;
        const typename Vec<T>::Raw* src = reinterpret_cast<const typename Vec<T>::Raw*>(weight);
        typename Vec<T>::Raw* dst = reinterpret_cast<typename Vec<T>::Raw*>(w_s);
        for (int idx = tid; idx < nvec; idx += CD_THREADS) dst[idx] = src[idx];
    }
    // the 8 candidate blocks of this voxel: 4 probes per thread
    bool overflow = false;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int bi = half * 4 + q;   // bit 2: x, bit 1: y, bit 0: z  (0 = block of coord - r)
        uint32_t id = VI_NO_ROW;
        if (c.x >= 0) {
            const int bx = ((c.y - r) >> 2) + ((bi >> 2) & 1);
            const int by = ((c.z - r) >> 2) + ((bi >> 1) & 1);
            const int bz = ((c.w - r) >> 2) + (bi & 1);
            uint64_t key;
            if (vi_block_key(c.x, bx, by, bz, key)) id = vi_block_lookup(keys, vals, cap_mask, key, &overflow);
        }
        block_s[bi][v] = id;
    }
    __syncthreads();

    float acc[CO];
#pragma unroll
    for (int k = 0; k < CO; ++k) acc[k] = 0.f;

    for (int o0 = 0; o0 < kvol; o0 += CD_CHUNK) {
        const int no = min(CD_CHUNK, kvol - o0);
        // neighbour row from the cell tables + feature gather; all independent
        for (int idx = tid; idx < no * CD_TM; idx += CD_THREADS) {
            const int ol = idx / CD_TM, vv = idx % CD_TM;
            const int4 cc = coord_s[vv];
            const char4 d = delta_s[o0 + ol];
            uint32_t j = VI_NO_ROW;
            if (cc.x >= 0) {
                const int x = cc.y + d.x, y = cc.z + d.y, z = cc.w + d.z;
                const int bi = (((x >> 2) - ((cc.y - r) >> 2)) << 2) | (((y >> 2) - ((cc.z - r) >> 2)) << 1) |
                               ((z >> 2) - ((cc.w - r) >> 2));
                const uint32_t id = block_s[bi][vv];
                if (id != VI_NO_ROW) j = cells[(size_t)id * 64 + ((x & 3) << 4 | (y & 3) << 2 | (z & 3))];
            }
            T* dst = x_s + ((size_t)ol * CD_TM + vv) * CD_MAX_CIN;
            has_s[ol * CD_TM + vv] = j != VI_NO_ROW;
            if (j != VI_NO_ROW) {
                const T* src = feat + (int64_t)j * cin;
#pragma unroll
                for (int ci = 0; ci < CD_MAX_CIN; ++ci) dst[ci] = ci < cin ? src[ci] : from_f<T>(0.f);
            }
        }
        __syncthreads();
        for (int ol = 0; ol < no; ++ol) {
            if (!has_s[ol * CD_TM + v]) continue;
            const T* xp = x_s + ((size_t)ol * CD_TM + v) * CD_MAX_CIN;
            float x[CD_MAX_CIN];
#pragma unroll
            for (int ci = 0; ci < CD_MAX_CIN; ci += Vec<T>::N)
                Vec<T>::unpack(*reinterpret_cast<const typename Vec<T>::Raw*>(xp + ci), x + ci);
            const T* w = w_s + (size_t)(o0 + ol) * cin * cout + half * CO;
#pragma unroll
            for (int ci = 0; ci < CD_MAX_CIN; ++ci) {
                if (ci < cin) {
                    // CO consecutive weights with 16-byte shared-memory loads (same address warp-wide)
#pragma unroll
                    for (int k = 0; k < CO; k += Vec<T>::N) {
                        float wv[Vec<T>::N];
                        Vec<T>::unpack(*reinterpret_cast<const typename Vec<T>::Raw*>(w + ci * cout + k), wv);
#pragma unroll
                        for (int q = 0; q < Vec<T>::N; ++q) acc[k + q] = fmaf(x[ci], wv[q], acc[k + q]);
                    }
                }
            }
        }
        __syncthreads();
    }
    if (overflow) atomicOr(status, PTV3_STATUS_PROBE_LIMIT);
    if (row < 0) return;
    T* op = out + row * (int64_t)cout + half * CO;
#pragma unroll
    for (int k = 0; k < CO; ++k) {
        const int ch = half * CO + k;
        float y = acc[k];
        if (bias) y += to_f<T>(bias[ch]);
        if (bn_scale) {
            // the convolution output is rounded to the element type first, as a
            // separate normalisation module would see it
            y = to_f<T>(from_f<T>(y));
            y = fmaf(y, bn_scale[ch], bn_shift[ch]);
        }
        if (apply_gelu) {
            if (bn_scale) y = to_f<T>(from_f<T>(y));
            y = cd_gelu(y);
        }
        op[k] = from_f<T>(y);
    }
}

constexpr int CDM_ROWS = 2;      // (dx, dy) rows of ksize offsets per round; even, so that K is a multiple of 16

// What the kernel reads, once per call: the weights [cout][kvol][cin] -> [offset][cout][8], zero padded to whole
// rounds, and the features with their rows padded to 16 bytes, so that a neighbour is one aligned copy
__global__ void __launch_bounds__(256) conv_direct_prepare_kernel(const __nv_bfloat16* __restrict__ w,
                                                                  __nv_bfloat16* __restrict__ wt, int cout, int kvol,
                                                                  int cin, int kvol_pad,
                                                                  const __nv_bfloat16* __restrict__ feat,
                                                                  uint4* __restrict__ rows, int64_t n)
{
    const int64_t first = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t idx = first; idx < (int64_t)kvol_pad * 8 * cout; idx += step) {
        const int ci = (int)idx % 8, co = ((int)idx / 8) % cout, o = (int)idx / (8 * cout);
        wt[idx] = (o < kvol && ci < cin) ? w[((size_t)co * kvol + o) * cin + ci] : __float2bfloat16(0.f);
    }
    const unsigned short* f = reinterpret_cast<const unsigned short*>(feat);
    for (int64_t i = first; i < n; i += step) {
        uint32_t e[8];
#pragma unroll
        for (int ci = 0; ci < 8; ++ci) e[ci] = ci < cin ? f[i * cin + ci] : 0u;
        rows[i] = make_uint4(e[0] | e[1] << 16, e[2] | e[3] << 16, e[4] | e[5] << 16, e[6] | e[7] << 16);
    }
}

// The cells of a (dx, dy) row of offsets lie in at most two aligned groups of four (z runs fastest in a table), so a
// thread takes the row's offsets of one voxel with two 16-byte loads, and copies each neighbour's padded row straight to
// shared memory: [offset][voxel] of 16 bytes is the K-major layout of an operand without swizzle (a product takes two
// offsets), [offset][channel] that of the weights.  One thread issues a round's products; while they run, the next
// round's cells are on their way.  Two rows per round, six CTAs per SM.
// us, here / with mma.sync, whose fragments (20 of 30 M shared-memory wavefronts, weights again for every 16 voxels) kept
// that pipe 74 % busy: 6 000 voxels 15.7 / 20.7, 100 000 45.0 / 55.1, 400 000 of four rooms 142 / 179, 2.05 M of LiDAR
// frames 599 / 817 (no GELU).  Error against 64 bits: that of rounding to bf16 in both, 0.0095 % of the results are not the
// rounded sum in both.  What bounds it: the gathers' passes through L1, a warp's 32 voxels touch as many cell tables.
// NT: 8-wide output channel tiles (c_out = 8 NT, NT even)
template <int NT>
__global__ void __launch_bounds__(CD_THREADS, NT <= 4 ? 6 : 4) conv_direct_tc05_kernel(
    const uint4* __restrict__ feat, const int32_t* __restrict__ indices,
    const __nv_bfloat16* __restrict__ wt, const __nv_bfloat16* __restrict__ bias,
    const float* __restrict__ bn_scale, const float* __restrict__ bn_shift, int apply_gelu,
    __nv_bfloat16* __restrict__ out, const int64_t* __restrict__ row_order, int64_t n, int ksize,
    const unsigned long long* __restrict__ keys, const uint32_t* __restrict__ vals, uint64_t cap_mask,
    const uint32_t* __restrict__ cells, uint32_t* __restrict__ status)
{
    using namespace tc05;
    constexpr int COUT = 8 * NT, TM_COLS = COUT <= 32 ? 32 : 64, PER = CDM_ROWS * CD_TM / CD_THREADS;
    extern __shared__ __align__(128) unsigned char smem[];
    const int per_round = CDM_ROWS * ksize;                      // offsets
    unsigned char* x_s = smem;                                   // [per_round][128] rows of 8 channels (16 B)
    unsigned char* w_s = smem + per_round * CD_TM * 16;          // [per_round][COUT] of this round
    __shared__ int row_s[CD_TM];
    __shared__ uint32_t block_s[8][CD_TM];
    __shared__ char2 delta_s[25];                                // (dx, dy) of a row
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s;

    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const uint32_t bar = smem_u32_generic(&bar_s);
    if (tid == 0) {
        mbar_init(bar, 1);
        abort_s = 0;
        fence_barrier_init();
    }
    if (warp == 0) tmem_alloc(smem_u32_generic(&tmem_slot), TM_COLS);
    const int v = tid % CD_TM, half = tid / CD_TM;
    const int64_t i = (int64_t)blockIdx.x * CD_TM + v;
    const int64_t row = i < n ? (row_order ? row_order[i] : i) : -1;
    const int r = ksize / 2;
    const int4 c = row >= 0 ? reinterpret_cast<const int4*>(indices)[row] : make_int4(-1, 0, 0, 0);
    if (half == 0) row_s[v] = (int)row;
    const int n_rows = ksize * ksize;
    if (tid < n_rows) delta_s[tid] = make_char2((char)(tid / ksize - r), (char)(tid % ksize - r));
    bool overflow = false;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int bi = half * 4 + q;   // bit 2: x, bit 1: y, bit 0: z  (0 = block of coord - r)
        uint32_t id = VI_NO_ROW;
        if (c.x >= 0) {
            const int bx = ((c.y - r) >> 2) + ((bi >> 2) & 1);
            const int by = ((c.z - r) >> 2) + ((bi >> 1) & 1);
            const int bz = ((c.w - r) >> 2) + (bi & 1);
            uint64_t key;
            if (vi_block_key(c.x, bx, by, bz, key)) id = vi_block_lookup(keys, vals, cap_mask, key, &overflow);
        }
        block_s[bi][v] = id;
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tm = tmem_slot;
    const uint32_t xs_base = smem_u32(x_s), ws_base = smem_u32(w_s);

    // the neighbours of a voxel along the rows of a round
    uint4 cell[PER][2];
    auto load_cells = [&](int row0) {
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            const int row = row0 + half + k * (CD_THREADS / CD_TM);
            cell[k][0] = cell[k][1] = make_uint4(VI_NO_ROW, VI_NO_ROW, VI_NO_ROW, VI_NO_ROW);
            if (c.x >= 0 && row < n_rows) {
                const char2 d = delta_s[row];
                const int x = c.y + d.x, y = c.z + d.y;
                const int bi = (((x >> 2) - ((c.y - r) >> 2)) << 2) | (((y >> 2) - ((c.z - r) >> 2)) << 1);
                const size_t at = (size_t)((x & 3) << 4 | (y & 3) << 2);
                const uint32_t id0 = block_s[bi][v], id1 = block_s[bi | 1][v];
                if (id0 != VI_NO_ROW) cell[k][0] = *reinterpret_cast<const uint4*>(cells + (size_t)id0 * 64 + at);
                if (id1 != VI_NO_ROW && ((c.w - r) & 3) + ksize > 4)
                    cell[k][1] = *reinterpret_cast<const uint4*>(cells + (size_t)id1 * 64 + at);
            }
        }
    };
    load_cells(0);
    bool ok = true;
    int phase = 1;                     // of the round before
    for (int row0 = 0; row0 < n_rows; row0 += CDM_ROWS, phase ^= 1) {
        if (row0) ok &= mbar_wait(bar, phase, &abort_s);
        // this round's weights: per_round planes of COUT rows
        for (int idx = tid; idx < per_round * COUT; idx += CD_THREADS)
            cp_async16(ws_base + idx * 16, wt + (size_t)row0 * ksize * 8 * COUT + (size_t)idx * 8);
#pragma unroll
        for (int k = 0; k < PER; ++k) {
            // entry 0 becomes the cell of dz = -r
            const int s0 = (c.w - r) & 3;
            uint32_t e[8] = {cell[k][0].x, cell[k][0].y, cell[k][0].z, cell[k][0].w,
                             cell[k][1].x, cell[k][1].y, cell[k][1].z, cell[k][1].w};
#pragma unroll
            for (int q = 0; q < 6; ++q) e[q] = s0 & 2 ? e[q + 2] : e[q];
#pragma unroll
            for (int q = 0; q < 5; ++q) e[q] = s0 & 1 ? e[q + 1] : e[q];
            const uint32_t dst = xs_base + ((half + k * (CD_THREADS / CD_TM)) * ksize * CD_TM + v) * 16;
#pragma unroll
            for (int q = 0; q < 5; ++q)
                if (q < ksize) cp_async16_zfill(dst + q * CD_TM * 16, feat + (e[q] != VI_NO_ROW ? e[q] : 0u), e[q] != VI_NO_ROW);
        }
        cp_async_commit();
        if (row0 + CDM_ROWS < n_rows) load_cells(row0 + CDM_ROWS);
        cp_async_wait<0>();
        fence_proxy_async();
        __syncthreads();
        // out[128 voxels][COUT] += X[128][K] . W[COUT][K]^T, two offsets to a product
        if (warp == 0) {
            if (elect_one()) {
                const uint64_t dx = umma_desc_plain(xs_base, CD_TM * 16, 128), dw = umma_desc_plain(ws_base, COUT * 16, 128);
                for (int ks = 0; ks < per_round / 2; ++ks)
                    umma_bf16(tm, dx + (uint64_t)(ks * 2 * CD_TM), dw + (uint64_t)(ks * 2 * COUT), umma_idesc_bf16(CD_TM, COUT),
                              row0 > 0 || ks > 0);
                umma_commit(bar);
            }
            __syncwarp();
        }
    }
    if (overflow) atomicOr(status, PTV3_STATUS_PROBE_LIMIT);
    ok &= mbar_wait(bar, phase, &abort_s);
    __syncwarp();
    fence_after_sync();

    // thread = voxel, half of its channels
    const int q = warp & 3, c0 = (warp >> 2) * (COUT / 2), orow = row_s[q * 32 + lane];
    const bool wide = ((uintptr_t)out & 15) == 0;
#pragma unroll
    for (int g = 0; g < NT / 2; ++g) {
        uint32_t acc[8], packed[4];
        __syncwarp();
        tmem_ld8(tm + ((uint32_t)(q * 32) << 16) + c0 + 8 * g, acc);
        tmem_ld8_fence(acc);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            float y[2] = {__uint_as_float(acc[2 * p]), __uint_as_float(acc[2 * p + 1])};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int ch = c0 + 8 * g + 2 * p + e;
                if (bias) y[e] += __bfloat162float(bias[ch]);
                if (bn_scale) {
                    // the convolution output is rounded to the element type first, as a
                    // separate normalisation module would see it
                    y[e] = __bfloat162float(__float2bfloat16(y[e]));
                    y[e] = fmaf(y[e], bn_scale[ch], bn_shift[ch]);
                }
                if (apply_gelu) {
                    if (bn_scale) y[e] = __bfloat162float(__float2bfloat16(y[e]));
                    y[e] = cd_gelu(y[e]);
                }
            }
            packed[p] = pack_bf16(y[0], y[1]);
        }
        __nv_bfloat16* op = out + (int64_t)orow * COUT + c0 + 8 * g;
        if (orow >= 0 && wide) {
            *reinterpret_cast<uint4*>(op) = make_uint4(packed[0], packed[1], packed[2], packed[3]);
        } else if (orow >= 0) {
#pragma unroll
            for (int p = 0; p < 4; ++p) reinterpret_cast<uint32_t*>(op)[p] = packed[p];
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        if (!ok) {
            int give_up = 0;           // products that were waited for in vain: once more, with a limit
            mbar_wait(bar, phase, &give_up);
        }
        fence_after_sync();
        tmem_dealloc(tm, TM_COLS);
    }
    if (lane == 0 && !ok) atomicOr(status, PTV3_STATUS_WAIT_LIMIT);
}

// laid-out weights (whole rounds)
static size_t conv_direct_weight_bytes(int ksize) { return align_up((size_t)(ksize * ksize + CDM_ROWS) * ksize * 8 * 64 * 4, 256); }
// ... and the padded features
size_t conv_direct_scratch_bytes(int64_t n, int ksize) { return conv_direct_weight_bytes(ksize) + align_up((size_t)n * 16, 256); }

static int launch_conv_direct_tc05(const void* feat, const int32_t* indices, const void* weight, const void* bias,
                                  const float* bn_scale, const float* bn_shift, int apply_gelu, void* out,
                                  const int64_t* row_order, int64_t n, int cin, int cout, int ksize,
                                  const unsigned long long* keys, const uint32_t* vals, uint64_t cap_mask,
                                  const uint32_t* cells, uint32_t* status, void* wt, cudaStream_t stream)
{
    const int kvol = ksize * ksize * ksize;
    const int rounds = (ksize * ksize + CDM_ROWS - 1) / CDM_ROWS, per_round = CDM_ROWS * ksize;
    uint4* rows = reinterpret_cast<uint4*>(static_cast<char*>(wt) + conv_direct_weight_bytes(ksize));
    const int64_t prepare = (std::max<int64_t>(n, rounds * per_round * 8 * cout) + 255) / 256;
    conv_direct_prepare_kernel<<<(unsigned)std::min<int64_t>(prepare, SMS * 8), 256, 0, stream>>>(
        (const __nv_bfloat16*)weight, (__nv_bfloat16*)wt, cout, kvol, cin, rounds * per_round, (const __nv_bfloat16*)feat,
        rows, n);
    const size_t smem = (size_t)per_round * (CD_TM + cout) * 16;
    const unsigned blocks = (unsigned)((n + CD_TM - 1) / CD_TM);
#define CDM_LAUNCH(NT)                                                                                      \
    do {                                                                                                    \
        auto kern = conv_direct_tc05_kernel<NT>;                                                            \
        if (allow_smem(kern) != cudaSuccess)                                                \
            return check_launch("ptv3_subm_conv_direct_fwd: shared memory attribute");                      \
        kern<<<blocks, CD_THREADS, smem, stream>>>(                                                          \
            rows, indices, (const __nv_bfloat16*)wt, (const __nv_bfloat16*)bias,                             \
            bn_scale, bn_shift, apply_gelu, (__nv_bfloat16*)out, row_order, n, ksize, keys, vals,            \
            cap_mask, cells, status);                                                                       \
    } while (0)
    switch (cout) {
        case 16: CDM_LAUNCH(2); break;
        case 32: CDM_LAUNCH(4); break;
        case 48: CDM_LAUNCH(6); break;
        case 64: CDM_LAUNCH(8); break;
        default:
            set_error("ptv3_subm_conv_direct_fwd: c_out %d (supported: 16, 32, 48, 64)", cout);
            return PTV3_ERR_UNSUPPORTED;
    }
#undef CDM_LAUNCH
    count_launches(2);
    return check_launch("ptv3_subm_conv_direct_fwd");
}

template <typename T>
static int launch_conv_direct(const void* feat, const int32_t* indices, const void* weight, const void* bias,
                              const float* bn_scale, const float* bn_shift, int apply_gelu, void* out,
                              const int64_t* row_order, int64_t n, int cin, int cout, int ksize,
                              const unsigned long long* keys, const uint32_t* vals, uint64_t cap_mask,
                              const uint32_t* cells, uint32_t* status, void* wt, cudaStream_t stream)
{
    const int kvol = ksize * ksize * ksize;
    conv_direct_transpose_kernel<T><<<(cout * kvol * cin + 255) / 256, 256, 0, stream>>>(
        (const T*)weight, (T*)wt, cout, kvol, cin);
    weight = wt;
    const size_t smem = (size_t)CD_CHUNK * CD_TM * (CD_MAX_CIN * sizeof(T) + 1) +
                        (size_t)kvol * cin * cout * sizeof(T);
    const unsigned blocks = (unsigned)((n + CD_TM - 1) / CD_TM);
#define CD_LAUNCH(CO)                                                                                    \
    do {                                                                                                 \
        auto kern = conv_direct_kernel<T, CO>;                                                           \
        if (allow_smem(kern) != cudaSuccess)                                                \
            return check_launch("ptv3_subm_conv_direct_fwd: shared memory attribute");                   \
        kern<<<blocks, CD_THREADS, smem, stream>>>((const T*)feat, indices, (const T*)weight,             \
                                                   (const T*)bias, bn_scale, bn_shift, apply_gelu,        \
                                                   (T*)out, row_order, n, cin, ksize, keys, vals,         \
                                                   cap_mask, cells, status);                              \
    } while (0)
    if (smem > 220 * 1024) {
        set_error("ptv3_subm_conv_direct_fwd: %zu bytes of shared memory needed", smem);
        return PTV3_ERR_UNSUPPORTED;
    }
    switch (cout) {
        case 16: CD_LAUNCH(8); break;
        case 32: CD_LAUNCH(16); break;
        case 48: CD_LAUNCH(24); break;
        case 64: CD_LAUNCH(32); break;
        default:
            set_error("ptv3_subm_conv_direct_fwd: c_out %d (supported: 16, 32, 48, 64)", cout);
            return PTV3_ERR_UNSUPPORTED;
    }
#undef CD_LAUNCH
    count_launches(2);
    return check_launch("ptv3_subm_conv_direct_fwd");
}

// hash table of blocks (sized for one block per voxel), block counter, one 64-entry table per block
static size_t conv_direct_index_bytes(int64_t n) { return voxel_index_bytes(n); }

int conv_direct_from_index(const VoxelIndex& vi, const void* feat, const int32_t* indices, const void* weight,
                           const float* bn_scale, const float* bn_shift, void* out, const int64_t* row_order,
                           int64_t n, int c_in, int c_out, int ksize, int dtype, uint32_t* status,
                           void* weight_scratch, cudaStream_t stream)
{
    if (dtype == PTV3_DTYPE_F32)
        return launch_conv_direct<float>(feat, indices, weight, nullptr, bn_scale, bn_shift, 1, out, row_order, n, c_in,
                                         c_out, ksize, vi.keys, vi.vals, vi.cap_mask, vi.cells, status, weight_scratch,
                                         stream);
    return launch_conv_direct_tc05(feat, indices, weight, nullptr, bn_scale, bn_shift, 1, out, row_order, n, c_in, c_out,
                                  ksize, vi.keys, vi.vals, vi.cap_mask, vi.cells, status, weight_scratch, stream);
}

}  // namespace ptv3

extern "C" size_t ptv3_subm_conv_direct_workspace_bytes(int64_t n, int ksize)
{
    return n > 0 ? ptv3::conv_direct_index_bytes(n) + ptv3::conv_direct_scratch_bytes(n, ksize) : 0;
}

extern "C" int ptv3_subm_conv_direct_fwd(const void* feat, const int32_t* indices, const void* weight,
                                         const void* bias, const float* bn_scale, const float* bn_shift,
                                         int apply_gelu, void* out, const int64_t* row_order, int64_t n,
                                         int c_in, int c_out, int ksize, int dtype, uint32_t* status,
                                         void* workspace, size_t workspace_bytes, void* stream_)
{
    using namespace ptv3;
    PTV3_REQUIRE(n >= 0 && n < (1ll << 31), PTV3_ERR_INVALID_ARGUMENT, "ptv3_subm_conv_direct_fwd: bad n");
    PTV3_REQUIRE(c_in >= 1 && c_in <= CD_MAX_CIN, PTV3_ERR_UNSUPPORTED,
                 "ptv3_subm_conv_direct_fwd: c_in %d outside [1, %d]", c_in, CD_MAX_CIN);
    PTV3_REQUIRE(ksize == 1 || ksize == 3 || ksize == 5, PTV3_ERR_UNSUPPORTED,
                 "ptv3_subm_conv_direct_fwd: kernel size %d (supported: 1, 3, 5)", ksize);
    PTV3_REQUIRE(dtype == PTV3_DTYPE_F32 || dtype == PTV3_DTYPE_BF16, PTV3_ERR_UNSUPPORTED,
                 "ptv3_subm_conv_direct_fwd: dtype %d", dtype);
    PTV3_REQUIRE((bn_scale == nullptr) == (bn_shift == nullptr), PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_subm_conv_direct_fwd: bn_scale and bn_shift go together");
    if (n == 0) return PTV3_OK;
    PTV3_REQUIRE(feat && indices && weight && out && status && workspace, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_subm_conv_direct_fwd: null pointer");
    PTV3_REQUIRE(((uintptr_t)indices & 15) == 0, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_subm_conv_direct_fwd: indices must be 16-byte aligned");
    const size_t need = conv_direct_index_bytes(n) + conv_direct_scratch_bytes(n, ksize);
    PTV3_REQUIRE(workspace_bytes >= need, PTV3_ERR_WORKSPACE,
                 "ptv3_subm_conv_direct_fwd: workspace %zu < %zu bytes", workspace_bytes, need);
    PTV3_REQUIRE(((size_t)ksize * ksize * ksize * c_in * c_out) % 8 == 0, PTV3_ERR_UNSUPPORTED,
                 "ptv3_subm_conv_direct_fwd: weight size must be a multiple of 8 elements");
    void* wt = static_cast<char*>(workspace) + conv_direct_index_bytes(n);
    cudaStream_t stream = (cudaStream_t)stream_;
    VoxelIndex vi;
    {
        const int rc = build_voxel_index(indices, n, workspace, status, stream, &vi);
        if (rc != PTV3_OK) return rc;
    }
    const unsigned long long* keys = vi.keys;
    const uint32_t* vals = vi.vals;
    const uint64_t cap_mask = vi.cap_mask;
    const uint32_t* cells = vi.cells;
    if (dtype == PTV3_DTYPE_F32)
        return launch_conv_direct<float>(feat, indices, weight, bias, bn_scale, bn_shift, apply_gelu, out,
                                         row_order, n, c_in, c_out, ksize, keys, vals, cap_mask, cells, status,
                                         wt, stream);
    return launch_conv_direct_tc05(feat, indices, weight, bias, bn_scale, bn_shift, apply_gelu, out, row_order, n,
                                  c_in, c_out, ksize, keys, vals, cap_mask, cells, status, wt, stream);
}
