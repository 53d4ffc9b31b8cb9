// Submanifold convolution (3x3x3) for bf16 features on inputs of many tiles: the implicit GEMM of conv_tc05.cu as a
// persistent kernel, one CTA per SM.
//
// A tile is 128 voxels (consecutive along a space-filling curve) x BN output channels; its stages are the (offset,
// 64-channel slice) pairs of the offsets that any of its voxels has a neighbour for.  A CTA walks tiles blockIdx.x,
// + gridDim.x, ...; four kinds of warps run ahead of one another, so that neither the look-up of a tile's neighbours nor
// its epilogue is waited for:
//   index warps     bring the 27 x 128 neighbour rows of the next tile, the list of its offsets in use, its voxels and
//                   its bias into one of two index buffers,
//   gather warps    fill the ring: each takes every GW-th stage, copies the stage's 128 neighbour rows with cp.async
//                   (zero rows where there is none) into the 128-byte (64 for 32 channels) swizzled K-major layout
//                   and asks TMA for the slice of W,
//   issuers         take the stages in turn, each into its own accumulator: tcgen05.mma (M = 128, N = BN, K = 16) into
//                   one of two sets of accumulators in tensor memory (256 columns: the only set),
//   epilogue warps  add the issuers' partial sums and the bias and store the rows, while the next tile is multiplied.
// The stages of a tile go round the issuers and every sum is taken in one fixed order, so the result is the same bit
// for bit on every run.
//
// What bounds it (cycle stamps, shared-memory bytes): the shared memory of an SM.  A stage is written once and read
// once by its products: 48 KB at 64 channels, 64 KB at 128, 96 KB at 256, of which 128 bytes pass in a cycle, so 384
// of the ~495 cycles that a stage takes, 512 of 544 and 768 of 754.  Products issued by an elected lane of a converged
// warp take their share of issue out of that (with `lane == 0` in a diverged one an issuer needed 1 100 cycles per stage
// of four, which was the limit).  Not tried: pairs of CTAs that share the slice of W (cta_group::2), which would move 17,
// 25 and 33 % fewer bytes.  Measured and dropped: neighbour rows by TMA gather
// (~11 cycles a row, twice the time), one warp for all weight loads (65 -> 77 us at 32 channels), waits by one
// elected lane (101 -> 162 us), with a time hint or as a spin (163 to 199), a look at the next stage ahead of the
// products (equal), copies through L1 (2 to 7 % slower).
// us here and as one CTA per tile (conv_tc05.cu, 32 channels: conv_mma.cu): 407 000 x 32 64 / 83, x 64 88 / 114,
// 2 000 000 x 32 343 / 528, x 64 492 / 653, 440 000 x 128 198 / 290, 172 000 x 256 195 / 231, 70 000 x 512 288 / 313.
//
// Replaces spconv.SubMConv3d.forward at model.py:546-552 for bf16.  Every wait is bounded and reports through the
// status word.
#include "common.cuh"
#include "conv_gather.cuh"
#include "conv_mma.cuh"
#include "mma_util.cuh"
#include "tc05.cuh"

namespace ptv3 {

using namespace tc05;

constexpr int CS_TM = CG_ROWS;         // voxels per tile
constexpr int CS_KVOL = 27;            // offsets, at most
constexpr int CS_SPLIT_O = 14;         // those of the first index warp

struct ConvStreamArgs {
    const __nv_bfloat16* feat;
    const int32_t* nbr;                // kvol x n, columns in tile order
    const __nv_bfloat16* bias;         // cout or NULL
    __nv_bfloat16* out;
    const int64_t* row_order;          // voxel of every tile position, or NULL
    int64_t n;
    int cin, cout, kvol;
    int tiles;                         // row tiles x column tiles
    bool planned;                      // see linear.cuh
    uint32_t* status;
};

// Warps: GW that gather, then NI issuers and two index warps, then (on a multiple of four, as a warp reads the quarter
// of tensor memory that its number names) four of the epilogue.
template <int GW, int NI>
__host__ __device__ constexpr int cs_epi_warp() { return (GW + NI + 2 + 3) / 4 * 4; }

// an index buffer
template <int BN>
struct ConvIndex {
    int32_t nbr[CS_KVOL * CS_TM];
    int32_t row[CS_TM];
    float bias[BN];
    int act[32];                       // number of offsets in use, then the offsets
    unsigned mask[4];
};

template <int BN, int KC, int STAGES, int NI, int GW, int SETS, int EW>
__global__ void __launch_bounds__((cs_epi_warp<GW, NI>() + EW) * 32, 1) conv_stream_kernel(
    const __grid_constant__ CUtensorMap map_w, const ConvStreamArgs a)
{
    constexpr int ROWB = KC * 2;
    constexpr int A_BYTES = CS_TM * ROWB, B_BYTES = BN * ROWB, STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr int EPI = cs_epi_warp<GW, NI>();
    constexpr int TM_COLS = SETS * NI * BN;
    static_assert(TM_COLS >= 32 && TM_COLS <= 512 && (TM_COLS & (TM_COLS - 1)) == 0, "tensor memory");
    static_assert(STAGE_BYTES % 1024 == 0 && A_BYTES % 1024 == 0, "operand tiles start on a swizzle atom");
    // a parity wait can only tell a phase from the one before it: see conv_tc05.cu
    static_assert(STAGES % NI == 0 && GW <= STAGES && GW % NI == 0, "slots, issuers and gathering warps");

    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32_generic(smem);
    ConvIndex<BN>* index = reinterpret_cast<ConvIndex<BN>*>(smem + STAGES * STAGE_BYTES);
    uint64_t* bars = reinterpret_cast<uint64_t*>(index + 2);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 * STAGES + 8);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t full0 = smem_u32_generic(bars), empty0 = full0 + 8 * STAGES, accfull0 = empty0 + 8 * STAGES,
                   accempty0 = accfull0 + 16, idxfull0 = accempty0 + 16, idxempty0 = idxfull0 + 16;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int col_tiles = a.cout / BN, kchunks = a.cin / KC;
    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 2);            // the gathering warp of the stage + its weight load
            mbar_init(empty0 + 8 * s, 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(accfull0 + 8 * b, NI);
            mbar_init(accempty0 + 8 * b, EW);
            mbar_init(idxfull0 + 8 * b, 2);
            mbar_init(idxempty0 + 8 * b, GW + NI + EW);
        }
        *abort = 0;
        fence_barrier_init();
        prefetch_tensormap(&map_w);
    }
    if (warp == EPI) {
        tmem_alloc(smem_u32_generic(tmem_slot), TM_COLS);
        // only now: the kernel brought up behind this one may take tensor memory and then wait for this one
        pdl_launch_next();
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    // the kernel before this one in the stream may still run: the set-up above and, planned, the index warps (which read
    // nothing but the geometry and the bias) go on beside it
    if (!a.planned || warp < GW + NI || warp >= GW + NI + 2) pdl_wait();
    bool ok = true;
    int seen = 0;              // stages of the tiles before this one
    const int first = (int)blockIdx.x, step = (int)gridDim.x;

    if (warp < GW) {
        // ---- gather: stages warp, warp + GW, ... of the CTA's sequence ---------------------------
        const RowGather<KC> gather(lane);
        const uint32_t pitch = (uint32_t)a.cin * 2;
        int g = warp;
        StageCursor cur{0, 0, warp, 1};                   // (GW <= STAGES)
        for (int i = 0, t = first; t < a.tiles; ++i, t += step) {
            const int b = i & 1;
            ok &= mbar_wait(idxfull0 + 8 * b, (i >> 1) & 1, abort);
            if (!__all_sync(0xffffffffu, ok)) break;
            const ConvIndex<BN>& x = index[b];
            const int end = seen + x.act[0] * kchunks, col0 = t % col_tiles * BN;
            cur.at = (g - seen) / kchunks;
            cur.chunk = (g - seen) - cur.at * kchunks;
            for (; g < end; g += GW) {
                const int o = x.act[1 + cur.at], chunk = cur.chunk;
                ok &= mbar_wait(empty0 + 8 * cur.slot, cur.phase, abort);
                fill_stage<KC, B_BYTES>(gather, sbase + cur.slot * STAGE_BYTES, x.nbr + o * CS_TM,
                                        reinterpret_cast<const char*>(a.feat) + chunk * ROWB, pitch, &map_w,
                                        o * a.cin + chunk * KC, col0, full0 + 8 * cur.slot, lane);
                cur.step<GW, STAGES>(kchunks);
            }
            seen = end;
            __syncwarp();
            if (lane == 0) mbar_arrive_one(idxempty0 + 8 * b);
        }
    } else if (warp < GW + NI) {
        // ---- issuers -------------------------------------------------------------------------------
        constexpr uint32_t idesc = umma_idesc_bf16(CS_TM, BN);
        const int me = warp - GW;
        const uint64_t da0 = umma_desc_kmajor(sbase, ROWB), db0 = umma_desc_kmajor(sbase + A_BYTES, ROWB);
        int g = me, s = me, phase = 0;
        for (int i = 0, t = first; t < a.tiles; ++i, t += step) {
            const int b = i & 1;
            ok &= mbar_wait(idxfull0 + 8 * b, (i >> 1) & 1, abort);
            const int end = seen + index[b].act[0] * kchunks;
            __syncwarp();
            if (lane == 0) mbar_arrive_one(idxempty0 + 8 * b);
            // the epilogue has read this set of accumulators (first use: free)
            ok &= mbar_wait(accempty0 + 8 * (i % SETS), ((i / SETS) & 1) ^ 1, abort);
            if (!__all_sync(0xffffffffu, ok)) break;
            fence_after_sync();
            const uint32_t acc = tmem_base + (i % SETS * NI + me) * BN;
            bool more = false;
            for (; g < end; g += NI) {
                const uint64_t da = da0 + s * (STAGE_BYTES >> 4), db = db0 + s * (STAGE_BYTES >> 4);
                ok &= mbar_wait(full0 + 8 * s, phase, abort);
                fence_after_sync();
                if (elect_one()) {
#pragma unroll
                    for (int k4 = 0; k4 < KC / 16; ++k4) umma_bf16(acc, da + 2 * k4, db + 2 * k4, idesc, more || k4 > 0);
                    umma_commit(empty0 + 8 * s);
                }
                __syncwarp();
                more = true;
                s += NI;
                if (s >= STAGES) {
                    s -= STAGES;
                    phase ^= 1;
                }
            }
            if (elect_one()) {
                if (more) umma_commit(accfull0 + 8 * (i % SETS));
                else mbar_arrive_one(accfull0 + 8 * (i % SETS));
            }
            __syncwarp();
            seen = end;
        }
    } else if (warp < GW + NI + 2) {
        // ---- index: an offset's 128 neighbours are four coalesced loads ---------------------------
        const int w = warp - GW - NI;
        for (int i = 0, t = first; t < a.tiles; ++i, t += step) {
            const int b = i & 1;
            const int64_t row0 = (int64_t)(t / col_tiles) * CS_TM;
            const int col0 = t % col_tiles * BN;
            ConvIndex<BN>& x = index[b];
            int32_t v[CS_SPLIT_O][4];
#pragma unroll
            for (int j = 0; j < CS_SPLIT_O; ++j) {
                const int o = w * CS_SPLIT_O + j;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int64_t r = row0 + lane + 32 * e;
                    v[j][e] = o < a.kvol && r < a.n ? a.nbr[(int64_t)o * a.n + r] : -1;
                }
            }
            int32_t row[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int64_t r = row0 + w * 64 + lane + 32 * e;
                row[e] = r < a.n ? (int32_t)(a.row_order ? a.row_order[r] : r) : -1;
            }
            ok = mbar_wait(idxempty0 + 8 * b, ((i >> 1) & 1) ^ 1, abort);
            if (!__all_sync(0xffffffffu, ok)) break;
            for (int e = w * 32 + lane; e < BN; e += 64) x.bias[e] = a.bias ? __bfloat162float(a.bias[col0 + e]) : 0.f;
#pragma unroll
            for (int e = 0; e < 2; ++e) x.row[w * 64 + lane + 32 * e] = row[e];
            unsigned used = 0;
#pragma unroll
            for (int j = 0; j < CS_SPLIT_O; ++j) {
                const int o = w * CS_SPLIT_O + j;
                bool any = false;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (o < CS_KVOL) x.nbr[o * CS_TM + lane + 32 * e] = v[j][e];
                    any |= v[j][e] >= 0;
                }
                if (__ballot_sync(0xffffffffu, any)) used |= 1u << o;
            }
            if (lane == 0) x.mask[w] = used;
            named_barrier(1, 64);
            if (w == 0) {
                const unsigned m = x.mask[0] | x.mask[1];
                if ((m >> lane) & 1) x.act[1 + __popc(m & ((1u << lane) - 1))] = lane;
                if (lane == 0) x.act[0] = __popc(m);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive_one(idxfull0 + 8 * b);
        }
    } else if (warp >= EPI) {
        // ---- epilogue ------------------------------------------------------------------------------
        // A warp takes its share of the columns out of tensor memory, rounded, before it stores any: where there is
        // one set of accumulators the next tile waits for no more than that.
        constexpr int BLOCKS = BN / 32 / (EW / 4);        // of 32 columns
        const int q = warp & 3, cb0 = (warp - EPI) / 4 * BLOCKS;
        for (int i = 0, t = first; t < a.tiles; ++i, t += step) {
            const int b = i & 1, set = i % SETS, col0 = t % col_tiles * BN;
            ok = mbar_wait(idxfull0 + 8 * b, (i >> 1) & 1, abort) && mbar_wait(accfull0 + 8 * set, (i / SETS) & 1, abort);
            if (!__all_sync(0xffffffffu, ok)) break;
            fence_after_sync();
            const ConvIndex<BN>& x = index[b];
            const int stages = x.act[0] * kchunks;
            // (the issuers' sums are added from that of the tile's first stage on, whoever had it)
            const uint32_t tm = tmem_base + set * NI * BN + ((uint32_t)(q * 32) << 16);
            uint32_t o[SETS == 1 ? BLOCKS : 1][4][4];
            auto take = [&](int cb, uint32_t (&y)[4][4]) {
                uint32_t acc[32];
                if (stages > 0) {
                    tmem_ld32(tm + seen % NI * BN + cb * 32, acc);
                    tmem_ld_wait();
                    tmem_ld_fence(acc);
                } else {
#pragma unroll
                    for (int e = 0; e < 32; ++e) acc[e] = 0;
                }
#pragma unroll 1
                for (int z = 1; z < NI && z < stages; ++z) {
                    uint32_t more[32];
                    tmem_ld32(tm + (seen + z) % NI * BN + cb * 32, more);
                    tmem_ld_wait();
                    tmem_ld_fence(more);
#pragma unroll
                    for (int e = 0; e < 32; ++e)
                        acc[e] = __float_as_uint(__uint_as_float(acc[e]) + __uint_as_float(more[e]));
                }
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const float2 bias = *reinterpret_cast<const float2*>(&x.bias[cb * 32 + c * 8 + 2 * e]);
                        y[c][e] = pack_bf16(__uint_as_float(acc[c * 8 + 2 * e]) + bias.x,
                                            __uint_as_float(acc[c * 8 + 2 * e + 1]) + bias.y);
                    }
            };
            // Four lanes exchange their rows' 16-byte chunks, so that a store writes 64 bytes of eight rows and not
            // 16 of 32 (with row-per-thread stores 101 us at 407 000 x 64, 88 so, 85 without any).  Afterwards
            // y[k] is chunk `m` of the row of the k-th of the four.
            auto store = [&](int cb, uint32_t (&y)[4][4]) {
                const int m = lane & 3;
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    uint32_t p0 = __shfl_xor_sync(0xffffffffu, m & 1 ? y[0][e] : y[1][e], 1);
                    uint32_t p1 = __shfl_xor_sync(0xffffffffu, m & 1 ? y[2][e] : y[3][e], 1);
                    if (m & 1) y[0][e] = p0, y[2][e] = p1;
                    else y[1][e] = p0, y[3][e] = p1;
                    p0 = __shfl_xor_sync(0xffffffffu, m & 2 ? y[0][e] : y[2][e], 2);
                    p1 = __shfl_xor_sync(0xffffffffu, m & 2 ? y[1][e] : y[3][e], 2);
                    if (m & 2) y[0][e] = p0, y[1][e] = p1;
                    else y[2][e] = p0, y[3][e] = p1;
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int row = x.row[q * 32 + (lane & ~3) + k];
                    if (row >= 0)
                        *reinterpret_cast<uint4*>(a.out + (int64_t)row * a.cout + col0 + cb * 32 + m * 8) =
                            make_uint4(y[k][0], y[k][1], y[k][2], y[k][3]);
                }
            };
            auto release = [&] {
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive_one(accempty0 + 8 * set);
            };
            if (SETS == 1) {
#pragma unroll
                for (int j = 0; j < BLOCKS; ++j) take(cb0 + j, o[SETS == 1 ? j : 0]);
                release();
#pragma unroll
                for (int j = 0; j < BLOCKS; ++j) store(cb0 + j, o[SETS == 1 ? j : 0]);
            } else {
#pragma unroll 1
                for (int j = 0; j < BLOCKS; ++j) {
                    take(cb0 + j, o[0]);
                    store(cb0 + j, o[0]);
                }
                release();
            }
            seen += stages;
            __syncwarp();
            if (lane == 0) mbar_arrive_one(idxempty0 + 8 * b);
        }
    }
    __syncwarp();
    fence_before_sync();
    __syncthreads();
    if (warp == EPI) {
        fence_after_sync();
        tmem_dealloc(tmem_base, TM_COLS);
    }
    if (lane == 0 && (!ok || (tid == 0 && *abort))) atomicOr(a.status, PTV3_STATUS_WAIT_LIMIT);
}

template <int BN, int KC, int STAGES, int NI, int GW, int SETS, int EW>
static int launch_as(const void* weight, ConvStreamArgs a, cudaStream_t stream)
{
    CUtensorMap mw;
    const uint64_t wcols = (uint64_t)a.kvol * a.cin;
    const int rc = make_tensor_map_bf16(&mw, weight, (uint64_t)a.cout, wcols, wcols * 2, BN, KC);
    if (rc) return rc;
    constexpr size_t smem = (size_t)STAGES * (CS_TM + BN) * KC * 2 + 2 * sizeof(ConvIndex<BN>) + 8 * (2 * STAGES + 8) + 16 + 1024;
    static_assert(smem <= 227 * 1024, "shared memory of a CTA");
    auto kern = conv_stream_kernel<BN, KC, STAGES, NI, GW, SETS, EW>;
    if (allow_smem(kern) != cudaSuccess) return check_launch("ptv3_subm_conv_fwd: shared memory attribute");
    a.tiles = (int)((a.n + CS_TM - 1) / CS_TM) * (a.cout / BN);
    // one CTA per SM (it may take all of tensor memory)
    launch_dependent(kern, dim3(a.tiles < SMS ? a.tiles : SMS), dim3((cs_epi_warp<GW, NI>() + EW) * 32),
                     smem < 120 * 1024 ? (size_t)120 * 1024 : smem, stream, mw, a);
    count_launches(1);
    return check_launch("ptv3_subm_conv_fwd");
}

int launch_conv_stream(const void* feat, const int32_t* nbr, const void* weight, const void* bias, void* out,
                       const int64_t* row_order, int64_t n, int c_in, int c_out, int kvol, int bn, bool planned,
                       uint32_t* status, cudaStream_t stream)
{
    const ConvStreamArgs a{(const __nv_bfloat16*)feat, nbr, (const __nv_bfloat16*)bias, (__nv_bfloat16*)out, row_order, n,
                           c_in, c_out, kvol, 0, planned, status};
    switch (bn) {
    case 32: return launch_as<32, 32, 16, 4, 8, 2, 4>(weight, a, stream);
    case 64: return launch_as<64, 64, 8, 2, 8, 2, 4>(weight, a, stream);
    case 128: return launch_as<128, 64, 6, 2, 6, 2, 4>(weight, a, stream);
    default: return launch_as<256, 64, 4, 2, 4, 1, 8>(weight, a, stream);
    }
}

}  // namespace ptv3
