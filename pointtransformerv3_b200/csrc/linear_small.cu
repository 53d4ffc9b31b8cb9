// Linear layers on short inputs (the coarse levels, small rooms), tcgen05: one 128 x 64 tile per CTA.
//
// On a few hundred rows a layer is bound by the length of its own chain, not by any unit: the persistent
// kernels (gemm_tc05.cu, linear_tc05.cu) give such a layer a handful of CTAs that walk all of K and then
// spend most of their time in an epilogue of 128 or 256 columns (27 x 2048 -> 512: 11 us on four CTAs).  Here
//   * tiles are 64 columns wide, eight warps take 32 columns of a row each;
//   * the weights of the first chunks are on their way before the preceding kernel has finished (where the
//     caller vouches for them, see linear.cuh);
//   * long K: a cluster of up to eight CTAs takes shares of K; each stores its partial sums with the CTA that finishes
//     their rows, which adds them in rank order (the result is the same on every run).  Read from the peers instead, one
//     after another and with a barrier more, behind which they may end: us, 441 x 1 024 -> 256 8.7 for 6.5, 457 x 2 048 -> 512
//     9.2 / 7.9, 75 x 2 048 -> 512 7.6 / 6.5; fp32 820 x 1 024 -> 256 14.8 / 10.4, 260 x 2 048 -> 512 17.9 / 14.5.
// (Linear + LayerNorm stays with linear_tc05.cu, whose epilogue holds a row in registers: 1 560 x 64 5.1 us
// against 6.5 in this form, 6 700 x 128 8.1 against 10.4.)
#include "common.cuh"
#include "linear.cuh"
#include "split_f32.cuh"
#include "tc05.cuh"
#include "vec.cuh"

namespace ptv3 {

using namespace tc05;

constexpr int LS_BM = 128, LS_BN = 64, LS_BK = 64;
constexpr int LS_A_BYTES = LS_BM * LS_BK * 2, LS_B_BYTES = LS_BN * LS_BK * 2, LS_STAGE = LS_A_BYTES + LS_B_BYTES;
constexpr int LS_MAX_STAGES = 8;
// fp32 (split_f32.cuh): a stage is a slice of 32 columns, its three parts of x and of W beside one another, and gives all
// six products.  (A stage for every product of 64 columns moved each part twice in the mean.  us, before / now: 40 000 x 64 ->
// 192 37.4 / 31.1, 40 000 x 256 -> 64 41.3 / 29.3, 2 800 x 128 -> 128 10.5 / 7.6, 820 x 256 -> 768 17.0 / 10.9, 260 x 512 ->
// 2 048 27.6 / 15.3, 260 x 2 048 -> 512 28.4 / 17.3, 27 x 2 048 -> 512 16.4 / 10.4.  Errors against 64 bits as before or,
// with K shared by a cluster, smaller: 820 x 256 -> 768 7.0e-8 / 5.5e-8, 260 x 2 048 -> 512 3.7e-7 / 1.0e-7.)
constexpr int LS_SLICE = 32;
constexpr int LS_A_PART = LS_BM * LS_SLICE * 2, LS_B_PART = LS_BN * LS_SLICE * 2, LS_SPLIT_STAGE = 3 * (LS_A_PART + LS_B_PART);
constexpr int LS_EPI_WARPS = 8, LS_THREADS = 64 + 32 * LS_EPI_WARPS;
constexpr int LS_PITCH = LS_BN + 4;                    // floats of a row of partial sums
constexpr int LS_PLAIN = 0, LS_GELU = 1, LS_RESIDUAL = 2, LS_F32 = 8;

struct LinearSmallArgs {
    const void *bias, *residual;                       // bf16; fp32 with LS_F32
    void* out;
    __nv_bfloat16* split_out;                          // LS_F32: the result as split rows instead
    int64_t n;
    int k, n_out, stages;
    bool settled;                                      // see linear.cuh
    uint32_t* status;
};

// Shared memory: the ring; with K shared by a cluster the partial sums of this CTA's rows (128 / parts of each CTA); bias as
// floats; barriers
constexpr int LS_PART_BYTES = LS_BM * LS_PITCH * 4;
static_assert(LS_PART_BYTES % 1024 == 0, "alignment of what follows");
constexpr int LS_PARAM_BYTES = LS_BN * 4;
__host__ __device__ constexpr int ls_part_offset(int stages, bool split) { return stages * (split ? LS_SPLIT_STAGE : LS_STAGE); }
__host__ __device__ constexpr int ls_param_offset(int stages, bool split, int parts)
{
    return ls_part_offset(stages, split) + (parts > 1 ? LS_PART_BYTES : 0);
}
static size_t ls_smem(int stages, bool split, int parts)
{
    return ls_param_offset(stages, split, parts) + LS_PARAM_BYTES + 8 * (2 * LS_MAX_STAGES + 1) + 16 + 1024;
}

// LS_F32: eight finished columns of a row, as floats or as split bf16 parts (see split_f32.cuh)
template <int MODE>
__device__ __forceinline__ void ls_store_f32(const LinearSmallArgs& a, int64_t row, int col, const float* acc,
                                             const float* bias)
{
    float y[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        y[i] = acc[i] + bias[i];
        if (MODE & LS_GELU) y[i] = 0.5f * y[i] * (1.f + erff(y[i] * 0.70710678118654752f));
    }
    if (MODE & LS_RESIDUAL) {
        const float4* r = reinterpret_cast<const float4*>((const float*)a.residual + row * a.n_out + col);
        const float4 r0 = r[0], r1 = r[1];
        y[0] += r0.x; y[1] += r0.y; y[2] += r0.z; y[3] += r0.w;
        y[4] += r1.x; y[5] += r1.y; y[6] += r1.z; y[7] += r1.w;
    }
    if (a.split_out) {
        split_store8(a.split_out + row * split_stored(a.n_out) * a.n_out, col, a.n_out, y);
        return;
    }
    float4* o = reinterpret_cast<float4*>((float*)a.out + row * a.n_out + col);
    o[0] = make_float4(y[0], y[1], y[2], y[3]);
    o[1] = make_float4(y[4], y[5], y[6], y[7]);
}

template <int MODE>
__device__ __forceinline__ uint4 ls_finish(const float* acc, const float* bias, uint4 res)
{
    uint32_t o[4];
    const uint32_t r[4] = {res.x, res.y, res.z, res.w};
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        // the Linear's own output in bf16, then the activation and the residual
        uint32_t packed;
        uint64_t y = round2(pack2(acc[2 * p] + bias[2 * p], acc[2 * p + 1] + bias[2 * p + 1]), packed);
        if (MODE & LS_GELU) y = gelu_tanh_erf2(y);
        if (MODE & LS_RESIDUAL) y = add2(y, unpack_bf16x2(r[p]));
        if (MODE & (LS_GELU | LS_RESIDUAL)) {
            float lo, hi;
            unpack2(y, lo, hi);
            packed = pack_bf16(lo, hi);
        }
        o[p] = packed;
    }
    return make_uint4(o[0], o[1], o[2], o[3]);
}

template <int MODE>
__global__ void __launch_bounds__(LS_THREADS) linear_small_kernel(const __grid_constant__ CUtensorMap map_x,
                                                                 const __grid_constant__ CUtensorMap map_w,
                                                                 const LinearSmallArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32_generic(smem);
    constexpr bool SPLIT = (MODE & LS_F32) != 0;
    constexpr int STAGE = SPLIT ? LS_SPLIT_STAGE : LS_STAGE, BK = SPLIT ? LS_SLICE : LS_BK;
    const int stages = a.stages, parts = (int)gridDim.z;
    if (parts > 1) cluster_started_arrive();
    const int off_part = ls_part_offset(stages, SPLIT), off_param = ls_param_offset(stages, SPLIT, parts),
              off_bar = off_param + LS_PARAM_BYTES;
    float* params = reinterpret_cast<float*>(smem + off_param);
    const uint32_t full0 = sbase + off_bar, empty0 = full0 + 8 * LS_MAX_STAGES,
                   accfull = empty0 + 8 * LS_MAX_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + off_bar + 8 * (2 * LS_MAX_STAGES + 1));
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint32_t* used_s = tmem_slot + 2;                      // LS_F32: the accumulators in use
    constexpr int TM_COLS = (MODE & LS_F32) ? SPLIT_ACCS * LS_BN : LS_BN;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int col0 = blockIdx.x * LS_BN, row0 = blockIdx.y * LS_BM;
    // this CTA's chunks of K
    const int nk = a.k / BK / parts, k0 = nk * (int)blockIdx.z * BK;

    // chunk kc of x or of W into slot `s`; of a split layer part by part
    auto load_x = [&](int kc, int s) {
        const uint32_t at = sbase + s * STAGE;
        if (SPLIT) {
#pragma unroll
            for (int p = 0; p < 3; ++p)
                tma_load_2d(at + p * LS_A_PART, &map_x, split_part_a(p, a.k) + k0 + kc * BK, row0, full0 + 8 * s);
        } else {
            tma_load_2d(at, &map_x, k0 + kc * BK, row0, full0 + 8 * s);
        }
    };
    auto load_w = [&](int kc, int s) {
        const uint32_t at = sbase + s * STAGE;
        mbar_expect_tx(full0 + 8 * s, STAGE);
        if (SPLIT) {
#pragma unroll
            for (int p = 0; p < 3; ++p)
                tma_load_2d(at + 3 * LS_A_PART + p * LS_B_PART, &map_w, p * a.k + k0 + kc * BK, col0, full0 + 8 * s);
        } else {
            tma_load_2d(at + LS_A_BYTES, &map_w, k0 + kc * BK, col0, full0 + 8 * s);
        }
    };

    // those of the first chunks: settled ones are fetched ahead of the wait below
    auto weights = [&] {
        for (int kc = 0; kc < nk && kc < stages; ++kc) load_w(kc, kc);
    };
    if (warp == 0 && elect_one()) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(full0 + 8 * s, 1);
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(accfull, (MODE & LS_F32) ? 2 : 1);       // the products; LS_F32: and the word below
        *abort = 0;
        fence_barrier_init();
        prefetch_tensormap(&map_x);
        if (a.settled) weights();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32_generic(tmem_slot), TM_COLS);
        // only now: the kernel brought up behind this one may take tensor memory and then wait for this one
        pdl_launch_next();
    }
    if (!a.settled) {
        pdl_wait();
        if (warp == 0 && elect_one()) weights();
    }
    for (int i = tid; i < LS_BN; i += LS_THREADS) {
        const int c = col0 + i;
        if (MODE & LS_F32)
            params[i] = a.bias && c < a.n_out ? ((const float*)a.bias)[c] : 0.f;
        else
            params[i] = a.bias ? __bfloat162float(((const __nv_bfloat16*)a.bias)[c]) : 0.f;
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    bool ok = true;
    pdl_wait();

    // epilogue threads: row r of the tile, 32 of its columns
    const int q = warp & 3, half = (warp - 2) >> 2, r = q * 32 + lane, c0 = half * 32;
    const int64_t row = (int64_t)row0 + r;
    const bool live = warp >= 2 && row < a.n;
    float v[32];
    uint4 res[4] = {};

    if (warp == 0) {
        // (slots and phases are counted, not divided: a division by `stages` takes longer than the rest of a turn)
        int s = 0, phase = 1;
        for (int kc = 0; kc < nk; ++kc) {
            if (kc >= stages) ok &= mbar_wait(empty0 + 8 * s, phase, abort);
            if (elect_one()) {
                if (kc >= stages) load_w(kc, s);
                load_x(kc, s);
            }
            __syncwarp();
            if (++s == stages) {
                s = 0;
                phase ^= 1;
            }
        }
    } else if (warp == 1) {
        constexpr uint32_t idesc = umma_idesc_bf16(LS_BM, LS_BN);
        const uint64_t da0 = umma_desc_kmajor(sbase, BK * 2),
                       db0 = umma_desc_kmajor(sbase + (SPLIT ? 3 * LS_A_PART : LS_A_BYTES), BK * 2);
        uint32_t used = 0;
        int s = 0, phase = 0, lead = k0 / 16 % SPLIT_MAIN;
        for (int kc = 0; kc < nk; ++kc) {
            ok &= mbar_wait(full0 + 8 * s, phase, abort);
            fence_after_sync();
            const uint64_t da = da0 + s * (STAGE >> 4), db = db0 + s * (STAGE >> 4);
            uint32_t seen = used;
            if (elect_one()) {
#pragma unroll
                for (int k4 = 0; k4 < BK / 16; ++k4) {
                    auto product = [&](int x, int w, uint32_t acc, bool add) {
                        umma_bf16(tmem_base + acc * LS_BN, da + 2 * k4 + x * (LS_A_PART >> 4), db + 2 * k4 + w * (LS_B_PART >> 4),
                                  idesc, add);
                    };
                    if (SPLIT) {
                        // x1 w1 into the leading accumulators in turn, the others x_i w_j, i + j <= 4, into the last one
                        const uint32_t acc = lead + k4 < SPLIT_MAIN ? lead + k4 : lead + k4 - SPLIT_MAIN;
                        product(0, 0, acc, (seen >> acc) & 1);
                        product(0, 1, SPLIT_MAIN, (seen >> SPLIT_MAIN) & 1);
                        seen |= 1u << acc | 1u << SPLIT_MAIN;
                        product(0, 2, SPLIT_MAIN, true);
                        product(1, 0, SPLIT_MAIN, true);
                        product(1, 1, SPLIT_MAIN, true);
                        product(2, 0, SPLIT_MAIN, true);
                    } else {
                        product(0, 0, 0, kc > 0 || k4 > 0);
                    }
                }
                if (kc + stages < nk) umma_commit(empty0 + 8 * s);
                if (kc == nk - 1) {
                    umma_commit(accfull);
                    if (SPLIT) {
                        *used_s = seen;
                        mbar_arrive_one(accfull);
                    }
                }
            }
            __syncwarp();
            // (what the elected lane has seen, for every lane)
            if (SPLIT) {
                used |= 1u << SPLIT_MAIN;
#pragma unroll
                for (int k4 = 0; k4 < BK / 16; ++k4) {
                    used |= 1u << lead;
                    lead = lead + 1 < SPLIT_MAIN ? lead + 1 : 0;
                }
            }
            if (++s == stages) {
                s = 0;
                phase ^= 1;
            }
        }
    } else {
        if ((MODE & LS_RESIDUAL) && !(MODE & LS_F32) && parts == 1 && live) {
#pragma unroll
            for (int g = 0; g < 4; ++g)
                res[g] = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)a.residual + row * a.n_out + col0 + c0 + g * 8);
        }
        ok &= mbar_wait(accfull, 0, abort);
        fence_after_sync();
        uint32_t acc[32];
        const uint32_t used = (MODE & LS_F32) ? *reinterpret_cast<volatile uint32_t*>(used_s) : 1u;
#pragma unroll
        for (int i = 0; i < 32; ++i) v[i] = 0.f;
        // (from the small products to the leading ones)
#pragma unroll 1
        for (int z = TM_COLS / LS_BN - 1; z >= 0; --z) {
            if (!((used >> z) & 1)) continue;
            tmem_ld32(tmem_base + ((uint32_t)(q * 32) << 16) + z * LS_BN + c0, acc);
            tmem_ld_wait();
            tmem_ld_fence(acc);
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] += __uint_as_float(acc[i]);
        }
    }

    if (parts == 1) {
        // (LS_F32: the last column tile may be half a tile)
        if (live && (!(MODE & LS_F32) || col0 + c0 < a.n_out))
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                if (MODE & LS_F32)
                    ls_store_f32<MODE>(a, row, col0 + c0 + g * 8, v + g * 8, params + c0 + g * 8);
                else
                    *reinterpret_cast<uint4*>((__nv_bfloat16*)a.out + row * a.n_out + col0 + c0 + g * 8) =
                        ls_finish<MODE>(v + g * 8, params + c0 + g * 8, res[g]);
            }
    } else {
        // every CTA's partial sums go to the CTA that finishes their rows (beside its ring, which it may still need); one
        // barrier, and it adds them up in rank order
        const int rows = LS_BM / parts, rank = (int)cluster_rank();
        __syncwarp();
        cluster_started_wait();
        if (warp >= 2) {
            const uint32_t at = peer_address(sbase + off_part + ((rank * rows + r % rows) * LS_PITCH + c0) * 4, r / rows);
#pragma unroll
            for (int g = 0; g < 8; ++g) st_cluster_f4(at + g * 16, v[g * 4], v[g * 4 + 1], v[g * 4 + 2], v[g * 4 + 3]);
        }
        __syncwarp();
        cluster_sync();
        const float* sums = reinterpret_cast<const float*>(smem + off_part);
        for (int e = tid; e < rows * (LS_BN / 8); e += LS_THREADS) {
            const int rr = e / (LS_BN / 8), c = e % (LS_BN / 8) * 8;
            const int64_t orow = (int64_t)row0 + rows * rank + rr;
            if (orow >= a.n || ((MODE & LS_F32) && col0 + c >= a.n_out)) continue;
            uint4 r4 = make_uint4(0, 0, 0, 0);
            if ((MODE & LS_RESIDUAL) && !(MODE & LS_F32))
                r4 = *reinterpret_cast<const uint4*>((const __nv_bfloat16*)a.residual + orow * a.n_out + col0 + c);
            float t[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            for (int z = 0; z < parts; ++z) {
                const float4* p = reinterpret_cast<const float4*>(sums + (z * rows + rr) * LS_PITCH + c);
                const float4 m = p[0], w = p[1];
                t[0] += m.x; t[1] += m.y; t[2] += m.z; t[3] += m.w;
                t[4] += w.x; t[5] += w.y; t[6] += w.z; t[7] += w.w;
            }
            if (MODE & LS_F32)
                ls_store_f32<MODE>(a, orow, col0 + c, t, params + c);
            else
                *reinterpret_cast<uint4*>((__nv_bfloat16*)a.out + orow * a.n_out + col0 + c) =
                    ls_finish<MODE>(t, params + c, r4);
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 1) {
        fence_after_sync();
        tmem_dealloc(tmem_base, TM_COLS);
    }
    if (lane == 0 && (!ok || (tid == 0 && *abort))) atomicOr(a.status, PTV3_STATUS_WAIT_LIMIT);
}

template <int MODE>
static int launch_ls(const void* x, const void* w, LinearSmallArgs a, int parts, cudaStream_t stream)
{
    constexpr bool split = (MODE & LS_F32) != 0;
    constexpr int BK = split ? LS_SLICE : LS_BK;
    const int nk = a.k / BK / parts;
    // (fp32: two CTAs share an SM, in shared memory as in tensor memory; two rooms of 20 000: 6.79 -> 6.65 ms)
    const dim3 grid((a.n_out + LS_BN - 1) / LS_BN, (unsigned)((a.n + LS_BM - 1) / LS_BM), parts);
    const int64_t ctas = (int64_t)grid.x * grid.y * parts;
    const int most = split ? (parts > 1 && ctas > SMS ? 2 : 3) : parts > 1 ? LS_MAX_STAGES - 1 : LS_MAX_STAGES;
    a.stages = nk < most ? nk : most;
    CUtensorMap mx, mw;
    const uint64_t cols = split ? (uint64_t)a.k * split_stored(a.k) : (uint64_t)a.k;      // stored
    int rc = make_tensor_map_bf16(&mx, x, (uint64_t)a.n, cols, cols * 2, LS_BM, BK);
    if (rc) return rc;
    rc = make_tensor_map_bf16(&mw, w, (uint64_t)a.n_out, cols, cols * 2, LS_BN, BK);
    if (rc) return rc;
    auto kern = linear_small_kernel<MODE>;
    if (allow_smem(kern) != cudaSuccess) return check_launch("short Linear: shared memory attribute");
    const dim3 cluster(1, 1, parts);
    launch_dependent_cluster(kern, grid, dim3(LS_THREADS), ls_smem(a.stages, split, parts), stream, cluster, mx, mw, a);
    count_launches(1);
    return check_launch("short Linear");
}

// Shares of K: clusters of up to eight CTAs, at least four chunks each.  Below 16 chunks the exchange costs
// more than it saves (441 x 512 -> 512: 7.1 us in clusters of two, 6.1 with the persistent kernel).
constexpr int LS_CLUSTER_CTAS = 128;                   // one wave: sixteen clusters of eight (a cluster lives in one GPC)
static int ls_parts(int64_t tiles, int k)
{
    const int chunks = k / LS_BK;
    int parts = 1;
    if (chunks >= 16)
        while (parts < 8 && tiles * parts * 2 <= LS_CLUSTER_CTAS && chunks % (parts * 2) == 0 && chunks / (parts * 2) >= 4)
            parts *= 2;
    return parts;
}
// fp32: at least four slices each; pairs also where two CTAs share an SM.  us in clusters of 1, 2, 4, 8: 2 800 x 128 -> 128
// (4 slices) 7.6 8.4 10.0, 820 x 256 -> 256 8.8 8.2 9.8 12.1, 820 x 256 -> 1 024 (224 CTAs in pairs) 12.7 11.7, 260 x 512 ->
// 512 12.5 10.2 9.4 12.5, 2 800 x 512 -> 128 (176 in fours) 17.2 13.1 13.9, 260 x 2 048 -> 512 (192 in eights) 38.9 22.6 17.3
// 18.4, 27 x 2 048 -> 512 34.5 20.5 13.5 10.4.
static int ls_split_parts(int64_t tiles, int k)
{
    const int slices = k / LS_SLICE;
    int parts = 1;
    while (parts < 8 && tiles * parts * 2 <= (parts == 1 ? 2 : 1) * LS_CLUSTER_CTAS && slices % (parts * 2) == 0 &&
           slices / (parts * 2) >= 4)
        parts *= 2;
    return parts;
}

// Where the lines lie (us, this kernel against the persistent ones):
//   K <= 128: three CTAs share an SM: one wave.  1 560 x 64 -> 192: 3.5 / 5.0, 6 760 x 128 -> 512 with GELU (424 tiles)
//     5.5 / 5.8; 1 776 tiles lose
//   longer K with GELU or a residual: one wave of one CTA per SM.  105 x 256 -> 1 024: 3.9 / 4.3, 457 x 512 -> 2 048
//     (128 tiles) 5.3 / 5.7, 6 760 x 512 -> 128 (106) 5.2 / 6.8, 4 000 x 1 024 -> 256 (128) 7.3 / 8.9, 2 200 x 2 048 -> 512
//     (144) 11.3 / 13.2, 11 400 x 1 024 -> 256 (360) 21.0 / 13.6; shared over K: 27 x 2 048 -> 512 5.6 / 11.0
//   without: half a wave from K = 512 (800 x 512 -> 512, 56 tiles: 5.0 / 5.1, 457 x 512 -> 1 536, 96: 5.3 / 5.1), a
//     handful of tiles below (105 x 256 -> 256, 4 tiles: 3.6 / 3.7, -> 768, 12: 3.9 / 3.8, 1 757 x 256 -> 256, 56: 4.4 / 4.0)
bool linear_small_wanted(int64_t n, int k, int n_out, bool epilogue)
{
    if (k % LS_BK || k < LS_BK || k > 8192 || n_out % LS_BN) return false;
    const int64_t tiles = (n + LS_BM - 1) / LS_BM * (n_out / LS_BN);
    if (k <= 128) return tiles <= 3 * SMS;
    if (epilogue || k >= 1024) return tiles <= SMS;
    return tiles <= (k < 512 ? 8 : SMS / 2);
}

int launch_linear_small(const void* x, const void* w, const void* bias, const void* residual, void* out, int64_t n, int k,
                        int n_out, int gelu, bool settled, uint32_t* status, cudaStream_t stream)
{
    LinearSmallArgs a{};
    a.bias = bias;
    a.residual = residual;
    a.out = out;
    a.n = n;
    a.k = k;
    a.n_out = n_out;
    a.settled = settled;
    a.status = status;
    const int parts = ls_parts((n + LS_BM - 1) / LS_BM * (n_out / LS_BN), k);
    switch ((gelu ? LS_GELU : 0) | (residual ? LS_RESIDUAL : 0)) {
    case LS_PLAIN: return launch_ls<LS_PLAIN>(x, w, a, parts, stream);
    case LS_GELU: return launch_ls<LS_GELU>(x, w, a, parts, stream);
    case LS_RESIDUAL: return launch_ls<LS_RESIDUAL>(x, w, a, parts, stream);
    default: return launch_ls<LS_GELU | LS_RESIDUAL>(x, w, a, parts, stream);
    }
}

int launch_linear_split(const void* xs, const void* ws, const float* bias, const float* residual, float* out,
                        void* split_out, int64_t n, int k, int n_out, int gelu, bool settled, uint32_t* status,
                        cudaStream_t stream)
{
    LinearSmallArgs a{};
    a.bias = bias;
    a.residual = residual;
    a.out = out;
    a.split_out = (__nv_bfloat16*)split_out;
    a.n = n;
    a.k = k;
    a.n_out = n_out;
    a.settled = settled;
    a.status = status;
    const int parts = ls_split_parts((n + LS_BM - 1) / LS_BM * ((n_out + LS_BN - 1) / LS_BN), k);
    switch ((gelu ? LS_GELU : 0) | (residual ? LS_RESIDUAL : 0)) {
    case LS_PLAIN: return launch_ls<LS_F32>(xs, ws, a, parts, stream);
    case LS_GELU: return launch_ls<LS_F32 | LS_GELU>(xs, ws, a, parts, stream);
    case LS_RESIDUAL: return launch_ls<LS_F32 | LS_RESIDUAL>(xs, ws, a, parts, stream);
    default: return launch_ls<LS_F32 | LS_GELU | LS_RESIDUAL>(xs, ws, a, parts, stream);
    }
}

}  // namespace ptv3
