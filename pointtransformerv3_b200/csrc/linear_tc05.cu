// Linear layers of a block on the 5th-generation tensor cores, with the row-wise
// glue that follows them fused into the epilogue:
//
//   plain      out = x W^T + b                                  (qkv, model.py:456)
//   residual   y   = x W^T + b
//              t   = ln1 ? LayerNorm(y; ln1) : y
//              s   = residual + t                   -> sum_out
//              out = LayerNorm(s; ln2)              -> norm_out
//     which is  cpe.1 + cpe.2 + shortcut + norm1     (model.py:553-554, 589-592)
//     and       attn.proj + shortcut + norm2         (model.py:487, 594, 598-600)
//
// bf16, input width K in {32, 64, 128}.  A persistent CTA keeps W in shared memory
// (TMA, once) and runs independent 128-thread groups; a group loads a
// 128-row x tile by TMA, issues K/16 tcgen05.mma into its slice of tensor memory and
// owns one accumulator row per thread, so LayerNorm statistics are thread-local
// (no shuffles).  Every intermediate the unfused sequence would round to bf16 is
// rounded at the same place.  Waits are bounded.
#include "common.cuh"
#include "mma_util.cuh"
#include "linear.cuh"
#include "tc05.cuh"
#include "vec.cuh"

namespace ptv3 {

using namespace tc05;

struct LinearArgs {
    const __nv_bfloat16* bias;       // n_out or NULL
    __nv_bfloat16* out;              // n x n_out
    int64_t n;
    int n_out;
    int groups;       // 128-thread groups that work (1..4)
    int nacc;         // accumulators per group in tensor memory (2 where 2 x groups x columns fit in 512)
    int w_box_rows;   // rows per TMA box of W
    int out_box;      // columns per staging tile and TMA store (64, or 32 when n_out % 64 != 0)
    bool settled;     // see linear.cuh
    uint32_t* status;
};

// Staging tile of a group: 128 rows x 64 bf16 columns, rows 144 bytes apart, so that
// both the row-per-thread accesses of the epilogue and the coalesced copies to and
// from global memory (consecutive threads on consecutive 16-byte pieces) are free of
// bank conflicts.  Global rows are `pitch` elements wide; `col0` is the slab's column.
constexpr int LIN_STAGE_ROW = 144;
constexpr int LIN_STAGE_BYTES = 128 * LIN_STAGE_ROW;

// A warp copies the 32 rows its own threads filled (t = thread of the group; rows (t / 32) * 32 ...), so
// that only the warp has to be in step, not the group.
template <int K>
__global__ void __launch_bounds__(512, 1) linear_tc05_kernel(const __grid_constant__ CUtensorMap map_x,
                                                             const __grid_constant__ CUtensorMap map_w,
                                                             const __grid_constant__ CUtensorMap map_o,
                                                             const LinearArgs a)
{
    constexpr int SW = K >= 64 ? 128 : 64;       // bytes per shared-memory row (swizzle span)
    constexpr int KB = K >= 64 ? K / 64 : 1;     // 64-wide K blocks
    constexpr int KCOLS = K >= 64 ? 64 : K;      // columns per K block
    constexpr int X_BLOCK = 128 * SW;            // one K block of an x tile
    constexpr int X_BYTES = KB * X_BLOCK;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32_generic(smem);
    const int n_out = a.n_out;
    const int w_block = n_out * SW;              // one K block of W
    const int off_x = KB * w_block;              // x tiles of the groups
    const int off_stage = off_x + 2 * a.groups * X_BYTES;   // (x tiles are double buffered) one staging tile per group
    const int off_par = off_stage + a.groups * LIN_STAGE_BYTES;   // bias as floats
    const int off_bar = off_par + n_out * 4;
    float* bias_s = reinterpret_cast<float*>(smem + off_par);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + off_bar);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const int tid = threadIdx.x, warp = tid >> 5;
    const int g = tid >> 7, t = tid & 127;
    const uint32_t wbar = sbase + off_bar;
    // xbar0 + 8: second x buffer; mbar0 + 8: second accumulator
    const uint32_t xbar0 = wbar + 8 * (1 + 2 * g), mbar0 = wbar + 8 * (9 + 2 * g);

    if (tid == 0) {
        for (int i = 0; i < 17; ++i) mbar_init(wbar + 8 * i, 1);
        *abort = 0;
        fence_barrier_init();
        prefetch_tensormap(&map_x);
        prefetch_tensormap(&map_w);
    }
    auto parameters = [&] {
        for (int i = tid; i < n_out; i += 512) bias_s[i] = a.bias ? __bfloat162float(a.bias[i]) : 0.f;
    };
    if (a.settled) parameters();
    if (warp == 0) {
        tmem_alloc(sbase + off_bar + 136, 512);
        // only now: the kernel brought up behind this one may take tensor memory and then wait for this one
        pdl_launch_next();
    }
    if (!a.settled) {
        pdl_wait();
        parameters();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0 && elect_one()) {   // weights: once per CTA
        mbar_expect_tx(wbar, (uint32_t)(KB * w_block));
        for (int kb = 0; kb < KB; ++kb)
            for (int r = 0; r < n_out; r += a.w_box_rows)
                tma_load_2d(sbase + kb * w_block + r * SW, &map_w, kb * KCOLS, r, wbar);
    }
    // up to here only settled weights, biases and LayerNorm parameters were read: everything the kernel before
    // this one in the stream may have written is touched after this wait
    pdl_wait();
    bool ok = mbar_wait(wbar, 0, abort);

    // columns of tensor memory per group: n_out rounded up to 32, groups side by side
    const int tm_cols = (n_out + 31) / 32 * 32;
    const uint32_t tm_lane = (uint32_t)((warp & 3) * 32) << 16;
    // two accumulators per group where tensor memory has room (a.nacc == 2): the product of the next
    // tile is issued before this tile's epilogue starts, so no tile waits for its product
    const int nacc = a.nacc;
    const uint32_t tm_acc_step = (uint32_t)(a.groups * tm_cols);
    const uint32_t tm_acc0 = tmem_base + tm_lane + g * tm_cols;
    const uint32_t tm_acc_mma0 = tmem_base + g * tm_cols;
    const uint32_t xs0 = sbase + off_x + 2 * g * X_BYTES;   // two x buffers
    unsigned char* stage = smem + off_stage + g * LIN_STAGE_BYTES;
    // one MMA covers at most 256 output columns
    const int n_half = n_out > 256 ? n_out / 2 : n_out;
    const uint32_t idesc = umma_idesc_bf16(128, n_half);
    uint32_t xph[2] = {0, 0};

    const int64_t ntiles = (a.n + 127) / 128;
    if (g < a.groups) {
        const int64_t tile_step = (int64_t)gridDim.x * a.groups;
        const int64_t tile0 = (int64_t)g * gridDim.x + blockIdx.x;      // (few tiles: one per SM, not four on one)
        // both by the group's first warp, one lane of it issuing
        const bool first_warp = (t >> 5) == 0;
        auto load_x = [&](int64_t tile, int b) {
            if (elect_one()) {
                mbar_expect_tx(xbar0 + 8 * b, X_BYTES);
                for (int kb = 0; kb < KB; ++kb)
                    tma_load_2d(xs0 + b * X_BYTES + kb * X_BLOCK, &map_x, kb * KCOLS, (int)(tile * 128), xbar0 + 8 * b);
            }
            __syncwarp();
        };
        // the product of the x tile in buffer xb into accumulator acc
        const uint64_t dx0 = umma_desc_kmajor(xs0, SW), dw0 = umma_desc_kmajor(sbase, SW);
        auto issue_mma = [&](int xb, int acc) {
            fence_after_sync();
            if (elect_one()) {
                for (int h = 0; h < n_out; h += n_half) {
#pragma unroll
                    for (int k = 0; k < K / 16; ++k) {
                        const int kb = (k * 16) / KCOLS, kk = (k * 16) % KCOLS;
                        umma_bf16(tm_acc_mma0 + acc * tm_acc_step + h, dx0 + ((xb * X_BYTES + kb * X_BLOCK + kk * 2) >> 4),
                                  dw0 + ((kb * w_block + h * SW + kk * 2) >> 4), idesc, k > 0);
                    }
                }
                umma_commit(mbar0 + 8 * acc);
            }
            __syncwarp();
        };
        if (first_warp && tile0 < ntiles) {
            load_x(tile0, 0);
            if (nacc == 2) {
                ok &= mbar_wait(xbar0, xph[0], abort);
                xph[0] ^= 1;
                issue_mma(0, 0);
                if (tile0 + tile_step < ntiles) load_x(tile0 + tile_step, 1);
            }
        }
        int j = 0;
        for (int64_t tile = tile0; tile < ntiles; tile += tile_step, ++j) {
            const int64_t row0 = tile * 128;
            const int buf = j & 1, cur = nacc == 2 ? buf : 0;
            if (nacc == 2) {
                ok &= mbar_wait(mbar0 + 8 * cur, (j >> 1) & 1, abort);
                if (first_warp && tile + tile_step < ntiles) {
                    // the next tile's product into the other accumulator (its epilogue ended with
                    // the barrier that closed the previous tile), then the x tile after that into
                    // the buffer this tile's product has finished with
                    ok &= mbar_wait(xbar0 + 8 * (buf ^ 1), xph[buf ^ 1], abort);
                    xph[buf ^ 1] ^= 1;
                    issue_mma(buf ^ 1, buf ^ 1);
                    if (tile + 2 * tile_step < ntiles) load_x(tile + 2 * tile_step, buf);
                }
            } else {
                ok &= mbar_wait(xbar0 + 8 * buf, xph[buf], abort);
                xph[buf] ^= 1;
                if (first_warp) {
                    // the other buffer was consumed by the previous tile's MMAs, which have completed:
                    // fetch the next tile into it while this tile is multiplied and written out
                    if (tile + tile_step < ntiles) load_x(tile + tile_step, buf ^ 1);
                    issue_mma(buf, 0);
                }
                ok &= mbar_wait(mbar0, j & 1, abort);
            }
            fence_after_sync();
            const uint32_t tm_acc = tm_acc0 + cur * tm_acc_step;
            // A warp packs `slw` columns of its 32 rows into its own staging tile (rows
            // slw * 2 bytes wide, swizzled like the tensor map so that the 16-byte stores of a warp
            // do not collide) and one lane hands the tile to a TMA store, which writes whole lines.
            const int slw = a.out_box, lane = t & 31;
            const uint32_t wtile = smem_u32_generic(stage) + (t >> 5) * 4096;
            const uint32_t my = wtile + lane * (slw * 2), swz = slw == 64 ? (lane & 7) : ((lane >> 1) & 3);
            for (int sl = 0; sl < n_out / slw; ++sl) {
                // the copy of the slab before has finished reading the staging tile
                if (lane == 0) bulk_wait_read<0>();
                __syncwarp();
                for (int c = 0; c < slw / 32; ++c) {
                    const int ch0 = sl * slw + c * 32;
                    float4 bb[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) bb[i] = *reinterpret_cast<const float4*>(bias_s + ch0 + i * 4);
                    uint32_t v[32];
                    tmem_ld32(tm_acc + ch0, v);
                    tmem_ld_wait();
                    tmem_ld_fence(v);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 b0 = bb[2 * q], b1 = bb[2 * q + 1];
                        const uint32_t* vv = v + q * 8;
                        const uint32_t o0 = pack_bf16(__uint_as_float(vv[0]) + b0.x, __uint_as_float(vv[1]) + b0.y);
                        const uint32_t o1 = pack_bf16(__uint_as_float(vv[2]) + b0.z, __uint_as_float(vv[3]) + b0.w);
                        const uint32_t o2 = pack_bf16(__uint_as_float(vv[4]) + b1.x, __uint_as_float(vv[5]) + b1.y);
                        const uint32_t o3 = pack_bf16(__uint_as_float(vv[6]) + b1.z, __uint_as_float(vv[7]) + b1.w);
                        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(my + (((c * 4 + q) ^ swz) << 4)),
                                     "r"(o0), "r"(o1), "r"(o2), "r"(o3));
                    }
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0 && row0 + (t & ~31) < a.n) {
                    tma_store_2d(&map_o, sl * slw, (int)row0 + (t & ~31), wtile);
                    bulk_commit();
                }
            }
            fence_before_sync();
            named_barrier(1 + g, 128);
        }
    }
    // shared memory stays allocated until the last TMA stores have read it
    if ((tid & 31) == 0) bulk_wait_read<0>();
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, 512);
    if (tid == 0 && (*abort || !ok)) atomicOr(a.status, PTV3_STATUS_WAIT_LIMIT);
}

template <int VEC, int PITCH>
__device__ __forceinline__ void stage_to_global(const unsigned char* stage, __nv_bfloat16* dst, int64_t row0,
                                                int64_t n, int col0, int t)
{
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const int idx = i * 32 + (t & 31), r = (t & ~31) + idx / VEC, c = idx % VEC;
        if (row0 + r < n)
            *reinterpret_cast<uint4*>(dst + (row0 + r) * PITCH + col0 + c * 8) =
                *reinterpret_cast<const uint4*>(stage + r * LIN_STAGE_ROW + c * 16);
    }
}

template <int VEC, int PITCH>
__device__ __forceinline__ void global_to_stage_async(unsigned char* stage, const __nv_bfloat16* src, int64_t row0,
                                                      int64_t n, int col0, int t)
{
#pragma unroll
    for (int i = 0; i < VEC; ++i) {
        const int idx = i * 32 + (t & 31), r = (t & ~31) + idx / VEC, c = idx % VEC;
        const bool in = row0 + r < n;
        cp_async16_zfill(smem_u32_generic(stage + r * LIN_STAGE_ROW + c * 16),
                         src + (in ? row0 + r : 0) * PITCH + col0 + c * 8, in);
    }
    cp_async_commit();
}

struct LinearLnArgs {
    const __nv_bfloat16* bias;       // K or NULL
    const __nv_bfloat16* residual;   // n x K
    const __nv_bfloat16 *ln1_w, *ln1_b;   // optional
    const __nv_bfloat16 *ln2_w, *ln2_b;
    __nv_bfloat16* sum_out;          // optional
    __nv_bfloat16* norm_out;
    float eps1, eps2;
    int64_t n;
    bool settled;                    // see linear.cuh
    uint32_t* status;
};

__host__ __device__ constexpr int lin_ln_groups(int k) { return k == 128 ? 2 : k == 64 ? 3 : 4; }
constexpr size_t lin_ln_smem(int k)
{
    const int sw = k >= 64 ? 128 : 64, kb = k >= 64 ? k / 64 : 1;
    return (size_t)kb * k * sw + (size_t)lin_ln_groups(k) * (kb * 128 * sw + LIN_STAGE_BYTES) + 5 * k * 4 +
           160 + 1024;
}

// Linear + residual + LayerNorms (the residual form above).  A thread takes its accumulator row out of tensor
// memory once, rounded to the bf16 pairs that everything after it works from; the epilogue then
// runs on registers alone: arithmetic on pairs of channels
// (fma.rn.f32x2 / add.rn.f32x2), one conversion per rounding, parameters two pairs at a time from shared memory.
// It is bound by instruction issue and the latency of few warps per scheduler.  Groups per CTA: as many as leave
// a thread the registers of its row (two at 128 channels: 112 us for 440 000 rows against 125 with three, whose
// threads spill; three at 64, four at 32); one x buffer and the next product issued at the end of the epilogue
// (with two buffers and the product ahead of it the issuing warp waits where the others work: 64 channels
// 51 -> 48 us, 32: 26.5 -> 25).  Against the form that parked the sum in tensor memory between the passes:
// 407 678 x 64: 60 -> 48 us (49 -> 38 without the first LayerNorm), x 32: 35 -> 25, 440 000 x 128: 157 -> 112.
template <int K, bool LN1>
__global__ void __launch_bounds__(128 * lin_ln_groups(K), 1) linear_ln_tc05_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                                 const __grid_constant__ CUtensorMap map_w,
                                                                                 const LinearLnArgs a)
{
    constexpr int SW = K >= 64 ? 128 : 64, KB = K >= 64 ? K / 64 : 1, KCOLS = K >= 64 ? 64 : K;
    constexpr int X_BLOCK = 128 * SW, X_BYTES = KB * X_BLOCK, W_BLOCK = K * SW;
    constexpr int GROUPS = lin_ln_groups(K), THREADS = 128 * GROUPS;
    constexpr int COLS = K < 64 ? K : 64, VEC = COLS / 8;       // a slab of the staging tile
    constexpr int OFF_X = KB * W_BLOCK, OFF_STAGE = OFF_X + GROUPS * X_BYTES;
    constexpr int OFF_PAR = OFF_STAGE + GROUPS * LIN_STAGE_BYTES, OFF_BAR = OFF_PAR + 5 * K * 4;
    constexpr uint32_t TM_COLS = GROUPS * K <= 128 ? 128 : GROUPS * K <= 256 ? 256 : 512;
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32_generic(smem);
    float* bias_s = reinterpret_cast<float*>(smem + OFF_PAR);
    float *g1 = bias_s + K, *b1 = bias_s + 2 * K, *g2 = bias_s + 3 * K, *b2 = bias_s + 4 * K;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + OFF_BAR);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 17);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const int tid = threadIdx.x, warp = tid >> 5, g = tid >> 7, t = tid & 127;
    const uint32_t wbar = sbase + OFF_BAR;
    const uint32_t xbar = wbar + 8 * (1 + g), mbar = wbar + 8 * (5 + g);

    if (tid == 0) {
        for (int i = 0; i < 17; ++i) mbar_init(wbar + 8 * i, 1);
        *abort = 0;
        fence_barrier_init();
        prefetch_tensormap(&map_x);
        prefetch_tensormap(&map_w);
    }
    auto parameters = [&] {
        for (int i = tid; i < K; i += THREADS) {
            bias_s[i] = a.bias ? __bfloat162float(a.bias[i]) : 0.f;
            g1[i] = LN1 ? __bfloat162float(a.ln1_w[i]) : 1.f;
            b1[i] = LN1 ? __bfloat162float(a.ln1_b[i]) : 0.f;
            g2[i] = __bfloat162float(a.ln2_w[i]);
            b2[i] = __bfloat162float(a.ln2_b[i]);
        }
    };
    if (a.settled) parameters();
    if (warp == 0) {
        tmem_alloc(sbase + OFF_BAR + 136, TM_COLS);
        // only now: the kernel brought up behind this one may take tensor memory and then wait for this one
        pdl_launch_next();
    }
    if (!a.settled) {
        pdl_wait();
        parameters();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    if (warp == 0 && elect_one()) {   // weights: once per CTA
        mbar_expect_tx(wbar, (uint32_t)(KB * W_BLOCK));
        for (int kb = 0; kb < KB; ++kb) tma_load_2d(sbase + kb * W_BLOCK, &map_w, kb * KCOLS, 0, wbar);
    }
    // up to here only settled weights, biases and LayerNorm parameters were read: everything the kernel before
    // this one in the stream may have written is touched after this wait
    pdl_wait();
    bool ok = mbar_wait(wbar, 0, abort);

    const uint32_t tm_acc = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + g * K;
    const uint32_t xs = sbase + OFF_X + g * X_BYTES;
    unsigned char* stage = smem + OFF_STAGE + g * LIN_STAGE_BYTES;
    unsigned char* my_row = stage + t * LIN_STAGE_ROW;
    constexpr float inv_c = 1.f / (float)K;
    const int64_t ntiles = (a.n + 127) / 128, tile_step = (int64_t)gridDim.x * GROUPS;
    const int64_t tile0 = (int64_t)g * gridDim.x + blockIdx.x;      // (few tiles: one per SM, not four on one)
    uint32_t xph = 0;

    // by the group's first warp, one lane of it issuing: an x tile; its product
    const bool first_warp = (t >> 5) == 0;
    auto load_x = [&](int64_t tile) {
        if (elect_one()) {
            mbar_expect_tx(xbar, X_BYTES);
            for (int kb = 0; kb < KB; ++kb) tma_load_2d(xs + kb * X_BLOCK, &map_x, kb * KCOLS, (int)(tile * 128), xbar);
        }
        __syncwarp();
    };
    auto multiply = [&] {
        ok &= mbar_wait(xbar, xph, abort);
        xph ^= 1;
        fence_after_sync();
        if (elect_one()) {
            const uint64_t dx = umma_desc_kmajor(xs, SW), dw = umma_desc_kmajor(sbase, SW);
#pragma unroll
            for (int k = 0; k < K / 16; ++k) {
                const int kb = (k * 16) / KCOLS, kk = (k * 16) % KCOLS;
                umma_bf16(tmem_base + g * K, dx + ((kb * X_BLOCK + kk * 2) >> 4), dw + ((kb * W_BLOCK + kk * 2) >> 4),
                          umma_idesc_bf16(128, K), k > 0);
            }
            umma_commit(mbar);
        }
        __syncwarp();
    };
    if (first_warp && tile0 < ntiles) {
        load_x(tile0);
        multiply();
    }
    int j = 0;
    for (int64_t tile = tile0; tile < ntiles; tile += tile_step, ++j) {
        const int64_t row0 = tile * 128;
        const bool more = tile + tile_step < ntiles;
        // the residual's first slab into the staging tile; the next tile's rows into L2
        global_to_stage_async<VEC, K>(stage, a.residual, row0, a.n, 0, t);
        if (more && row0 + tile_step * 128 + t < a.n) {
            const char* p = reinterpret_cast<const char*>(a.residual + (row0 + tile_step * 128 + t) * K);
#pragma unroll
            for (int b = 0; b < K * 2; b += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(p + b));
        }
        ok &= mbar_wait(mbar, j & 1, abort);
        fence_after_sync();
        if (first_warp && more) load_x(tile + tile_step);     // (its product is done)
        // ---- y = round(acc + bias); sums for its LayerNorm, shifted by the row's first value (no cancellation)
        uint32_t y[K / 2];
        float shift1 = 0.f;
        uint64_t nshift = 0, s1 = 0, q1 = 0;
        // (keeps the compiler from holding raw or unpacked values, twice the registers, across chunks and passes)
        auto pin = [&](int lo, int hi) {
#pragma unroll
            for (int i = 0; i < K / 2; ++i)
                if (i >= lo && i < hi) asm volatile("" : "+r"(y[i]));
        };
#pragma unroll
        for (int c = 0; c < K; c += 32) {
            uint32_t v[32];
            tmem_ld32(tm_acc + c, v);
            tmem_ld_wait();
            tmem_ld_fence(v);
#pragma unroll
            for (int i = 0; i < 32; i += 4) {
                const ulonglong2 bb = *reinterpret_cast<const ulonglong2*>(bias_s + c + i);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint64_t r = round2(add2(pack2u(v[i + 2 * e], v[i + 2 * e + 1]), e ? bb.y : bb.x),
                                              y[(c + i) / 2 + e]);
                    if (LN1) {
                        if (c == 0 && i == 0 && e == 0) {
                            float lo, hi;
                            unpack2(r, lo, hi);
                            shift1 = lo;
                            nshift = pack2(-lo, -lo);
                        }
                        const uint64_t d = add2(r, nshift);
                        s1 = add2(s1, d);
                        q1 = fma2(d, d, q1);
                    }
                }
            }
            pin(c / 2, c / 2 + 16);
            if (LN1) asm volatile("" : "+l"(s1), "+l"(q1));
        }
        // every thread of the group has its row: the accumulator is free
        fence_before_sync();
        named_barrier(1 + g, 128);
        uint64_t nmean1 = 0, rs1 = 0;
        if (LN1) {
            const float md = hsum2(s1) * inv_c, mean = shift1 + md;
            const float rstd = rsqrtf(fmaxf(hsum2(q1) * inv_c - md * md, 0.f) + a.eps1);
            nmean1 = pack2(-mean, -mean);
            rs1 = pack2(rstd, rstd);
        }
        // ---- s = residual + (LayerNorm of) y, written out; shifted sums for the second LayerNorm
        float shift2 = 0.f;
        uint64_t s2 = 0, q2 = 0;
#pragma unroll
        for (int sl = 0; sl < K; sl += COLS) {
            if (sl > 0) global_to_stage_async<VEC, K>(stage, a.residual, row0, a.n, sl, t);
            cp_async_wait<0>();
            __syncwarp();      // the staging rows of a warp are its own
#pragma unroll
            for (int q = 0; q < VEC; ++q) {
                const uint4 rr = *reinterpret_cast<const uint4*>(my_row + q * 16);
                const uint32_t rw[4] = {rr.x, rr.y, rr.z, rr.w};
                uint32_t* o = y + (sl + q * 8) / 2;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ch = sl + q * 8 + h * 4;
                    ulonglong2 gg = {0, 0}, hh = {0, 0};
                    if (LN1) {
                        gg = *reinterpret_cast<const ulonglong2*>(g1 + ch);
                        hh = *reinterpret_cast<const ulonglong2*>(b1 + ch);
                    }
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int i = h * 2 + e;
                        uint64_t v = unpack_bf16x2(o[i]);
                        uint32_t pk;
                        if (LN1) v = round2(fma2(mul2(add2(v, nmean1), rs1), e ? gg.y : gg.x, e ? hh.y : hh.x), pk);
                        v = round2(add2(unpack_bf16x2(rw[i]), v), o[i]);
                        if (sl == 0 && q == 0 && i == 0) {
                            float lo, hi;
                            unpack2(v, lo, hi);
                            shift2 = lo;
                            nshift = pack2(-lo, -lo);
                        }
                        const uint64_t d = add2(v, nshift);
                        s2 = add2(s2, d);
                        q2 = fma2(d, d, q2);
                    }
                }
                if (a.sum_out) *reinterpret_cast<uint4*>(my_row + q * 16) = make_uint4(o[0], o[1], o[2], o[3]);
            }
            __syncwarp();
            if (a.sum_out) {
                stage_to_global<VEC, K>(stage, a.sum_out, row0, a.n, sl, t);
                __syncwarp();
            }
        }
        pin(0, K / 2);
        const float md = hsum2(s2) * inv_c, mean2 = shift2 + md;
        const float rstd2 = rsqrtf(fmaxf(hsum2(q2) * inv_c - md * md, 0.f) + a.eps2);
        const uint64_t nmean2 = pack2(-mean2, -mean2), rs2 = pack2(rstd2, rstd2);
#pragma unroll
        for (int sl = 0; sl < K; sl += COLS) {
#pragma unroll
            for (int q = 0; q < VEC; ++q) {
                uint32_t ow[4];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int ch = sl + q * 8 + h * 4;
                    const ulonglong2 gg = *reinterpret_cast<const ulonglong2*>(g2 + ch);
                    const ulonglong2 hh = *reinterpret_cast<const ulonglong2*>(b2 + ch);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const uint64_t f = fma2(mul2(add2(unpack_bf16x2(y[ch / 2 + e]), nmean2), rs2), e ? gg.y : gg.x,
                                                e ? hh.y : hh.x);
                        float lo, hi;
                        unpack2(f, lo, hi);
                        ow[h * 2 + e] = pack_bf16(lo, hi);
                    }
                }
                *reinterpret_cast<uint4*>(my_row + q * 16) = make_uint4(ow[0], ow[1], ow[2], ow[3]);
            }
            __syncwarp();
            stage_to_global<VEC, K>(stage, a.norm_out, row0, a.n, sl, t);
            __syncwarp();
        }
        if (first_warp && more) multiply();      // (its x tile has long landed)
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, TM_COLS);
    if (tid == 0 && (*abort || !ok)) atomicOr(a.status, PTV3_STATUS_WAIT_LIMIT);
}

static bool linear_shape_ok(int k, int n_out, bool residual_mode)
{
    if (k != 32 && k != 64 && k != 128) return false;
    if (residual_mode) return n_out == k;
    return n_out % 32 == 0 && n_out >= 32 && n_out <= 384 && (n_out <= 256 || (n_out / 2) % 16 == 0);
}

static int launch_linear(const void* x, const void* w, LinearArgs a, int k, cudaStream_t stream)
{
    const int sw = k >= 64 ? 128 : 64, kb = k >= 64 ? k / 64 : 1, kcols = k >= 64 ? 64 : k;
    a.w_box_rows = a.n_out <= 256 ? a.n_out : a.n_out / 2;
    const int tm_cols = (a.n_out + 31) / 32 * 32;
    int groups = 512 / tm_cols;
    if (groups > 4) groups = 4;
    // ... and as many as fit in shared memory next to the resident weights
    while (groups > 1 && (size_t)kb * a.n_out * sw + (size_t)groups * (2 * kb * 128 * sw + LIN_STAGE_BYTES) +
                                 (size_t)a.n_out * 4 + 160 + 1024 > 220 * 1024)
        --groups;
    a.groups = groups;
    a.nacc = 2 * groups * tm_cols <= 512 ? 2 : 1;
    CUtensorMap mx, mw, mo;
    int rc = make_tensor_map_bf16(&mx, x, (uint64_t)a.n, k, (uint64_t)k * 2, 128, kcols);
    if (rc) return rc;
    a.out_box = a.n_out % 64 == 0 ? 64 : 32;
    rc = make_tensor_map_bf16(&mo, a.out, (uint64_t)a.n, (uint64_t)a.n_out, (uint64_t)a.n_out * 2, 32, a.out_box);
    if (rc) return rc;
    rc = make_tensor_map_bf16(&mw, w, a.n_out, k, (uint64_t)k * 2, a.w_box_rows, kcols);
    if (rc) return rc;
    const size_t smem = (size_t)kb * a.n_out * sw + (size_t)groups * (2 * kb * 128 * sw + LIN_STAGE_BYTES) +
                        (size_t)a.n_out * 4 + 160 + 1024;
    const size_t smem_req = smem < 120 * 1024 ? 120 * 1024 : smem;   // one CTA per SM (it takes all of tensor memory)
    const int64_t ntiles = (a.n + 127) / 128, grid = ntiles < SMS ? ntiles : SMS;
#define LIN_LAUNCH(KK)                                                                                       \
    do {                                                                                                     \
        auto kern = linear_tc05_kernel<KK>;                                                                  \
        if (allow_smem(kern) != cudaSuccess)                                                \
            return check_launch("ptv3_linear_fwd: shared memory attribute");                                 \
        launch_dependent(kern, dim3((unsigned)grid), dim3(512), smem_req, stream, mx, mw, mo, a);                \
    } while (0)
    if (k == 32) LIN_LAUNCH(32);
    else if (k == 64) LIN_LAUNCH(64);
    else LIN_LAUNCH(128);
#undef LIN_LAUNCH
    count_launches(1);
    return check_launch("ptv3_linear_fwd");
}

template <int K, bool LN1>
static int launch_linear_ln(const void* x, const void* w, const LinearLnArgs& a, cudaStream_t stream)
{
    constexpr int kcols = K >= 64 ? 64 : K;
    CUtensorMap mx, mw;
    int rc = make_tensor_map_bf16(&mx, x, (uint64_t)a.n, K, (uint64_t)K * 2, 128, kcols);
    if (rc == PTV3_OK) rc = make_tensor_map_bf16(&mw, w, K, K, (uint64_t)K * 2, K, kcols);
    if (rc != PTV3_OK) return rc;
    auto kern = linear_ln_tc05_kernel<K, LN1>;
    if (allow_smem(kern) != cudaSuccess) return check_launch("ptv3_linear_ln_fwd: shared memory attribute");
    const int64_t ntiles = (a.n + 127) / 128;
    constexpr size_t smem = lin_ln_smem(K) < 120 * 1024 ? 120 * 1024 : lin_ln_smem(K);      // one CTA per SM
    launch_dependent(kern, dim3((unsigned)(ntiles < SMS ? ntiles : SMS)), dim3(128 * lin_ln_groups(K)), smem, stream, mx,
                     mw, a);
    count_launches(1);
    return check_launch("ptv3_linear_ln_fwd");
}

int linear_fwd(const void* x, const void* weight, const void* bias, void* out, int64_t n, int k, int n_out, int dtype,
               bool settled, uint32_t* status, cudaStream_t stream)
{
    PTV3_REQUIRE(n >= 0 && n < (1ll << 31), PTV3_ERR_INVALID_ARGUMENT, "ptv3_linear_fwd: bad n");
    PTV3_REQUIRE(ptv3_linear_supported(k, n_out, 0, dtype), PTV3_ERR_UNSUPPORTED,
                 "ptv3_linear_fwd: supported: bf16, k in {32, 64, 128}, n_out a multiple of 32 up to 384");
    if (n == 0) return PTV3_OK;
    PTV3_REQUIRE(x && weight && out && status, PTV3_ERR_INVALID_ARGUMENT, "ptv3_linear_fwd: null pointer");
    PTV3_REQUIRE((((uintptr_t)x | (uintptr_t)weight | (uintptr_t)out) & 15) == 0, PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_linear_fwd: tensors must be 16-byte aligned");
    if (linear_small_wanted(n, k, n_out, false))
        return launch_linear_small(x, weight, bias, nullptr, out, n, k, n_out, 0, settled, status, stream);
    LinearArgs a{};
    a.bias = (const __nv_bfloat16*)bias;
    a.out = (__nv_bfloat16*)out;
    a.n = n;
    a.n_out = n_out;
    a.settled = settled;
    a.status = status;
    return launch_linear(x, weight, a, k, stream);
}

int linear_ln_fwd(const void* x, const void* weight, const void* bias, const void* residual, const void* ln1_weight,
                  const void* ln1_bias, float ln1_eps, void* sum_out, const void* ln2_weight, const void* ln2_bias,
                  float ln2_eps, void* norm_out, int64_t n, int channels, int dtype, bool settled, uint32_t* status,
                  cudaStream_t stream)
{
    PTV3_REQUIRE(n >= 0 && n < (1ll << 31), PTV3_ERR_INVALID_ARGUMENT, "ptv3_linear_ln_fwd: bad n");
    PTV3_REQUIRE(ptv3_linear_supported(channels, channels, 1, dtype), PTV3_ERR_UNSUPPORTED,
                 "ptv3_linear_ln_fwd: supported: bf16, channels in {32, 64, 128}");
    PTV3_REQUIRE((ln1_weight == nullptr) == (ln1_bias == nullptr), PTV3_ERR_INVALID_ARGUMENT,
                 "ptv3_linear_ln_fwd: LayerNorm weight and bias go together");
    if (n == 0) return PTV3_OK;
    PTV3_REQUIRE(x && weight && residual && ln2_weight && ln2_bias && norm_out && status,
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_linear_ln_fwd: null pointer");
    PTV3_REQUIRE((((uintptr_t)x | (uintptr_t)weight | (uintptr_t)residual | (uintptr_t)norm_out |
                   (uintptr_t)sum_out) & 15) == 0,
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_linear_ln_fwd: tensors must be 16-byte aligned");
    const LinearLnArgs a{(const __nv_bfloat16*)bias, (const __nv_bfloat16*)residual, (const __nv_bfloat16*)ln1_weight,
                         (const __nv_bfloat16*)ln1_bias, (const __nv_bfloat16*)ln2_weight, (const __nv_bfloat16*)ln2_bias,
                         (__nv_bfloat16*)sum_out, (__nv_bfloat16*)norm_out, ln1_eps, ln2_eps, n, settled, status};
    auto launch = channels == 32   ? (ln1_weight ? launch_linear_ln<32, true> : launch_linear_ln<32, false>)
                  : channels == 64 ? (ln1_weight ? launch_linear_ln<64, true> : launch_linear_ln<64, false>)
                                   : (ln1_weight ? launch_linear_ln<128, true> : launch_linear_ln<128, false>);
    return launch(x, weight, a, stream);
}

}  // namespace ptv3

extern "C" int ptv3_linear_supported(int k, int n_out, int residual_mode, int dtype)
{
    return dtype == PTV3_DTYPE_BF16 && ptv3::linear_shape_ok(k, n_out, residual_mode != 0);
}

extern "C" int ptv3_linear_fwd(const void* x, const void* weight, const void* bias, void* out, int64_t n, int k,
                               int n_out, int dtype, uint32_t* status, void* stream)
{
    return ptv3::linear_fwd(x, weight, bias, out, n, k, n_out, dtype, false, status, (cudaStream_t)stream);
}

extern "C" int ptv3_linear_ln_fwd(const void* x, const void* weight, const void* bias, const void* residual,
                                  const void* ln1_weight, const void* ln1_bias, float ln1_eps, void* sum_out,
                                  const void* ln2_weight, const void* ln2_bias, float ln2_eps, void* norm_out,
                                  int64_t n, int channels, int dtype, uint32_t* status, void* stream)
{
    return ptv3::linear_ln_fwd(x, weight, bias, residual, ln1_weight, ln1_bias, ln1_eps, sum_out, ln2_weight, ln2_bias,
                               ln2_eps, norm_out, n, channels, dtype, false, status, (cudaStream_t)stream);
}
