// Submanifold convolution (3x3x3) on the 5th-generation tensor cores where tiles are few (the coarse levels, small
// rooms), and for fp32 features: an implicit GEMM, output-stationary over tiles of 128 voxels, accumulated in tensor
// memory.  bf16 inputs of many tiles take the persistent kernel in conv_stream.cu.
//
// A CTA owns 128 voxels (consecutive in the tile order, which follows a space-filling curve) and
// BN output channels.  It stages the 27 x 128 neighbour rows of its tile in shared memory and
// drops the offsets for which no voxel of the tile has a neighbour.  Then, for each remaining
// offset o and each KC-wide slice of the input channels,
//   gather warps  each fill every NGW-th stage: the 128 neighbour rows (zero rows where there is none)
//                 gathered with cp.async into the 128-byte swizzled K-major operand layout, and the
//                 matching BN x KC slice of W[:, o, :] fetched with TMA into the same layout,
//   issuers       issue KC / 16 tcgen05.mma (M = 128, N = BN, K = 16) that add A_o W_o^T to the
//                 accumulator in tensor memory, and release the stage with tcgen05.commit,
// through a ring of stages guarded by mbarriers.  When the last product has completed, the gather warps
// read the accumulator (thread = voxel), add the bias, round to bf16 and store their rows.
//
// Two threads issue the products, taking the stages in turn, each into its own accumulator; the epilogue adds
// the two partial sums.  Every sum is taken in one fixed order, so the result is the same bit for bit on every run, on
// every level: no atomics, no pair lists, no second pass.  Products with zero rows are not skipped.
// What bounds it on few tiles: ~7 us before the first and after the last product, and ~370 cycles per stage of 64
// channels, 500 of 128, 700 of 256 (see conv_stream.cu for what a stage is made of).
//
// A cluster of up to eight CTAs shares one tile.  Each takes a contiguous share of the tile's stages (of fp32 parts: slices
// in turn); the partial sums meet in shared memory and every CTA adds the
// parts of its rows, which the peers have stored with it, in rank order.  A tile alone walks
// 27 x c_in / 64 stages one after the other, 49 us at 512 channels on 27 voxels, while most SMs have nothing; in
// clusters of eight that is 10 us.
// Stored with the CTA that adds them, not read from the peers: us, 487 x 128 9.0 / 8.0, 178 x 256 10.1 / 9.4, 822 x 256 11.7 /
// 11.2; fp32 822 x 256 26.7 / 23.5, 261 x 512 48.5 / 45.4.
//
// Replaces spconv.SubMConv3d.forward at model.py:546-552.
// Useful work: 2 . pairs . C_in . C_out FLOP.  Every mbarrier wait is bounded and reports through
// the status word.
#include <atomic>

#include "common.cuh"
#include "conv_gather.cuh"
#include "conv_mma.cuh"
#include "mma_util.cuh"
#include "split_f32.cuh"
#include "tc05.cuh"

namespace ptv3 {

using namespace tc05;

constexpr int CT_TM = CG_ROWS;     // voxels per tile
constexpr int CT_KC = 64;          // channels per stage
constexpr int CT_MAX_KVOL = 27;
constexpr int CT_GATHER_WARPS = 8;

struct ConvTcArgs {
    const __nv_bfloat16* feat;
    const int32_t* nbr;            // kvol x n, columns in tile order
    const void* bias;              // cout or NULL, of the output's type
    void* out;                     // bf16 or fp32
    __nv_bfloat16* split_out;      // fp32: the result as split rows instead, or NULL
    const int64_t* row_order;      // voxel of every tile position, or NULL
    int64_t n;
    int cin, cout, kvol;
    bool planned;                  // see linear.cuh
    uint32_t* status;
};

// eight finished fp32 columns of a row
__device__ __forceinline__ void ct_store_f32(const ConvTcArgs& a, int64_t row, int col, const float* y)
{
    if (a.split_out) {
        split_store8(a.split_out + row * split_stored(a.cout) * a.cout, col, a.cout, y);
        return;
    }
    float4* o = reinterpret_cast<float4*>((float*)a.out + row * a.cout + col);
    o[0] = make_float4(y[0], y[1], y[2], y[3]);
    o[1] = make_float4(y[4], y[5], y[6], y[7]);
}

// Operands: bf16; fp32 as the six pieces of split_f32.cuh, 64 of their columns to a stage (widths that are not whole slices
// of 64 channels); fp32 as three parts, a stage for each, from which the six products are taken.  A stage for every product, the form before for all widths, moves
// each part twice in the mean.  us, before / now (L2 flushed, ~5 us of it the timing): 1 830 x 256 73.7 / 48.1, 822 x 256
// 41.0 / 33.8, 261 x 512 88 / 59.5, 2 855 x 128 36.9 / 29.6, 10 542 x 64 35.8 / 33.8, 100 000 x 64 122.8 / 119.8.  What is left is
// shared memory: a product of 64 columns takes its 48 to 58 cycles to read 6 KB, of 128 columns 65 (measured alone), 24
// of them to a slice, whose copies write 72 or 96 KB beside them; a slice takes 3 200 cycles.
// Error against 64 bits, 2-norm, before / now: 1 830 x 256 1.90e-7 / 1.70e-7, 261 x 512 3.07e-7 / 2.16e-7, 2 855 x 128 1.16e-7 /
// 1.08e-7, 40 000 x 64 1.76e-7 / 1.04e-7; with contiguous shares of a cluster's CTAs 2.11e-7, 3.56e-7, 1.21e-7.
constexpr int CT_BF16 = 0, CT_PIECES = 1, CT_PARTS = 2;

template <int BN, int STAGES, int NI, bool SPLIT, int FORM>
__global__ void __launch_bounds__((CT_GATHER_WARPS + NI) * 32, 1) conv_tc05_kernel(const __grid_constant__ CUtensorMap map_w,
                                                               const ConvTcArgs a)
{
    constexpr bool F32 = FORM != CT_BF16;
    static_assert(SPLIT || F32, "whole bf16 tiles: conv_stream.cu");
    static_assert(FORM != CT_PARTS || NI == 1, "one warp meets the three stages of a slice");
    constexpr int KC = CT_KC, ROWB = KC * 2;        // bytes per staged row: one swizzle span
    constexpr int A_BYTES = CT_TM * ROWB, B_BYTES = BN * ROWB, STAGE_BYTES = A_BYTES + B_BYTES;
    constexpr int CT_THREADS = (CT_GATHER_WARPS + NI) * 32;
    // NI issuing warps, each with its own accumulator in tensor memory.  A slot of the ring must always be
    // consumed by the same issuer (STAGES a multiple of NI): an issuer that met a slot whose previous use
    // another, slower issuer had not consumed yet would take the parity of that older phase for its own.
    // fp32: SPLIT_ACCS accumulators each (split_f32.cuh)
    // ... parts: as many as tensor memory holds, three of four for the leading products (the more sums, the less is lost
    // where the tensor core truncates, and a product into an accumulator waits for the one before it)
    constexpr int ACCS = FORM == CT_PARTS ? 512 / BN : F32 ? SPLIT_ACCS : 1, LEADS = ACCS / 4 * 3;
    constexpr int TM_COLS = NI * ACCS * BN;
    static_assert(TM_COLS >= 32 && TM_COLS <= 512 && (TM_COLS & (TM_COLS - 1)) == 0, "tensor memory");
    static_assert(STAGES % NI == 0, "issuers and accumulators");
    static_assert(STAGE_BYTES % 1024 == 0 && A_BYTES % 1024 == 0, "operand tiles start on a swizzle atom");
    // Warps that gather: at most one per stage of the ring.  A parity wait on an mbarrier can only tell
    // the current phase from the one before it, so a warp must never be two uses ahead of a slot: its
    // stages are NGW apart, and having been given a slot for stage X (stage X - STAGES consumed) it may
    // ask for the slot of stage X + NGW only if stage X + NGW - 2 STAGES is known to be consumed,
    // i.e. NGW <= STAGES (the products run in order).
    constexpr int NGW = STAGES < CT_GATHER_WARPS ? STAGES : CT_GATHER_WARPS;

    // partial sums of a split tile, over the ring: rows of BN floats, padded so that 16-byte accesses of
    // consecutive rows spread over the banks
    constexpr int PART_PITCH = BN + 4;
    static_assert(!SPLIT || CT_TM * PART_PITCH * 4 <= STAGES * STAGE_BYTES, "partial sums fit the ring");

    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const uint32_t sbase = smem_u32_generic(smem);
    constexpr int OFF_NBR = STAGES * STAGE_BYTES;                   // kvol x 128 int32
    constexpr int OFF_ROWS = OFF_NBR + CT_MAX_KVOL * CT_TM * 4;     // 128 int64
    constexpr int OFF_ACT = OFF_ROWS + CT_TM * 8;                   // 32 int
    constexpr int OFF_BIAS = OFF_ACT + 32 * 4;                      // BN float
    constexpr int OFF_BAR = OFF_BIAS + BN * 4;                      // full, empty per stage; accumulator full
    int32_t* nbr_s = reinterpret_cast<int32_t*>(smem + OFF_NBR);
    int64_t* rows_s = reinterpret_cast<int64_t*>(smem + OFF_ROWS);
    int* act = reinterpret_cast<int*>(smem + OFF_ACT);
    float* bias_s = reinterpret_cast<float*>(smem + OFF_BIAS);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + OFF_BAR + 8 * (2 * STAGES + 1));
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    uint32_t* used_s = tmem_slot + 2;              // fp32: the accumulators an issuer has written
    const uint32_t full0 = sbase + OFF_BAR, empty0 = full0 + 8 * STAGES, accfull = empty0 + 8 * STAGES;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int64_t row0 = (int64_t)blockIdx.x * CT_TM;
    const int col0 = blockIdx.y * BN;
    const int kvol = a.kvol;

    if (tid == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(full0 + 8 * s, 2);        // the gathering warp of the stage + its weight load
            mbar_init(empty0 + 8 * s, 1);
        }
        mbar_init(accfull, F32 ? 2 * NI : NI);     // the products of every issuer; fp32: and its word in used_s
        *abort = 0;
        fence_barrier_init();
        prefetch_tensormap(&map_w);
    }
    if (warp == CT_GATHER_WARPS) {
        tmem_alloc(smem_u32_generic(tmem_slot), TM_COLS);
        // only now: the kernel brought up behind this one may take tensor memory and then wait for this one
        pdl_launch_next();
    }
    // (only the set-up above, and planned the look-up below, runs beside the kernel before this one in the stream)
    if (!a.planned) pdl_wait();

    // ---- voxels of this tile, their neighbour rows, the offsets in use -------------------------
    if (tid < CT_TM) {
        const int64_t i = row0 + tid;
        rows_s[tid] = i < a.n ? (a.row_order ? a.row_order[i] : i) : -1;
    }
    for (int c = tid; c < BN; c += CT_THREADS) {
        if (F32)
            bias_s[c] = a.bias ? ((const float*)a.bias)[col0 + c] : 0.f;
        else
            bias_s[c] = a.bias ? __bfloat162float(((const __nv_bfloat16*)a.bias)[col0 + c]) : 0.f;
    }
    {
        // A warp stages whole offsets (four coalesced rows of 32 entries each), all of its loads issued
        // before the first store, and notes in the same pass whether the tile has the offset at all.
        constexpr int NW = CT_THREADS / 32, OPW = (CT_MAX_KVOL + NW - 1) / NW;
        int32_t v[OPW][4];
#pragma unroll
        for (int j = 0; j < OPW; ++j) {
            const int o = warp + j * NW;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = lane + 32 * i;
                v[j][i] = (o < kvol && row0 + r < a.n) ? a.nbr[(int64_t)o * a.n + row0 + r] : -1;
            }
        }
#pragma unroll
        for (int j = 0; j < OPW; ++j) {
            const int o = warp + j * NW;
            if (o < kvol) {
                bool any = false;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    nbr_s[o * CT_TM + lane + 32 * i] = v[j][i];
                    any |= v[j][i] >= 0;
                }
                const unsigned b = __ballot_sync(0xffffffffu, any);
                if (lane == 0) act[1 + o] = b != 0;
            }
        }
    }
    __syncthreads();
    if (warp == 0) {
        // the offsets in use, in ascending order: act[1 ..], their number in act[0]
        const int flag = lane < kvol ? act[1 + lane] : 0;
        const unsigned m = __ballot_sync(0xffffffffu, flag != 0);
        if (flag) act[1 + __popc(m & ((1u << lane) - 1))] = lane;
        if (lane == 0) act[0] = __popc(m);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (a.planned) pdl_wait();
    const uint32_t tmem_base = *tmem_slot;
    const int n_act = act[0];
    // stages of an offset; parts: three to a slice of KC channels, which stay together
    constexpr int UNIT = FORM == CT_PARTS ? 3 : 1;
    const int kchunks = FORM == CT_PARTS ? a.cin / 6 / KC * UNIT : a.cin / KC;
    const int stored = F32 ? a.cin / 6 * split_stored(a.cin / 6) : a.cin;      // columns of a feature row
    // this CTA's share of the tile's stages (all of them without a cluster)
    int first = 0, nit = n_act * kchunks;
    if (SPLIT) {
        const int total = nit / UNIT, parts = (int)gridDim.z;
        if (FORM == CT_PARTS) {
            // slices in turn: a voxel's neighbours lie on few offsets, and their products then spread over all sums
            nit = (total - (int)blockIdx.z + parts - 1) / parts * UNIT;
        } else {
            first = total * (int)blockIdx.z / parts;
            nit = total * ((int)blockIdx.z + 1) / parts - first;
        }
    }
    bool ok = true;

    if (warp < CT_GATHER_WARPS) {
        // ---- gather: warp w < NGW fills stages w, w + NGW, ...: the 128 neighbour rows of offset
        // act[it / kchunks], channels of chunk it % kchunks, and (lane 0) the matching slice of W.
        // The warps run independent pipelines, so the fixed cost of a stage (barrier waits, the TMA
        // issue, the proxy fence) and the latency of its copies overlap with the other warps' stages.
        const RowGather<KC> gather(lane);
        const uint32_t pitch = (uint32_t)stored * 2;
        StageCursor cur{(first + warp) / kchunks, (first + warp) % kchunks, warp % STAGES, 1};
        for (int it = warp < NGW ? warp : nit; it < nit; it += NGW) {
            if (FORM == CT_PARTS) {
                const int slice = (int)blockIdx.z + it / UNIT * (int)gridDim.z, per = kchunks / UNIT;
                cur.at = slice / per;
                cur.chunk = slice % per * UNIT + it % UNIT;
            }
            const int o = act[1 + cur.at];
            int kc = cur.chunk * KC, kw = kc;
            if (FORM == CT_PIECES) {
                kc = split_column_a(cur.chunk, a.cin / 6);
                kw = split_column_b(cur.chunk, a.cin / 6);
            }
            if (FORM == CT_PARTS) kc = kw = cur.chunk % 3 * (a.cin / 6) + cur.chunk / 3 * KC;
            ok &= mbar_wait(empty0 + 8 * cur.slot, cur.phase, abort);
            fill_stage<KC, B_BYTES>(gather, sbase + cur.slot * STAGE_BYTES, nbr_s + o * CT_TM,
                                    reinterpret_cast<const char*>(a.feat + kc), pitch, &map_w, o * stored + kw, col0,
                                    full0 + 8 * cur.slot, lane);
            cur.step<NGW, STAGES>(kchunks);
        }
        if (nit > 0) {
            ok &= mbar_wait(accfull, 0, abort);
            fence_after_sync();
        }
    } else if (FORM == CT_PARTS) {
        // ---- the issuer, fp32 from parts: per slice of KC channels x1 w1 into the leading accumulators in turn, the five
        // small products into the others in turn
        constexpr uint32_t idesc = umma_idesc_bf16(CT_TM, BN);
        const uint64_t da0 = umma_desc_kmajor(sbase, ROWB), db0 = umma_desc_kmajor(sbase + A_BYTES, ROWB);
        constexpr uint32_t RESTS = ACCS - LEADS;
        uint32_t used = 0;
        int s = 0, phase = 0, lead = 0;
        for (int it = 0; it < nit; it += 3) {
            uint64_t da[3], db[3];
            uint32_t slot[3];
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                ok &= mbar_wait(full0 + 8 * s, phase, abort);
                fence_after_sync();
                da[p] = da0 + s * (STAGE_BYTES >> 4);
                db[p] = db0 + s * (STAGE_BYTES >> 4);
                slot[p] = empty0 + 8 * s;
                if (elect_one()) {
                    // (x_i w_j with i + j <= 4, as soon as its parts are here)
                    if (p == 0) {
#pragma unroll
                        for (int k4 = 0; k4 < KC / 16; ++k4) {
                            const uint32_t acc = lead + k4 < LEADS ? lead + k4 : lead + k4 - LEADS;
                            const uint32_t before = k4 < LEADS ? used : ~0u;
                            umma_bf16(tmem_base + acc * BN, da[0] + 2 * k4, db[0] + 2 * k4, idesc, (before >> acc) & 1);
                        }
                    } else {
                        constexpr int X[2][3] = {{0, 1, 1}, {0, 2, 0}}, W[2][3] = {{1, 0, 1}, {2, 0, 0}};
#pragma unroll
                        for (int k4 = 0; k4 < KC / 16; ++k4)
#pragma unroll
                            for (int i = 0; i < (p == 1 ? 3 : 2); ++i) {
                                const uint32_t turn = k4 * (p == 1 ? 3 : 2) + i;
                                umma_bf16(tmem_base + (LEADS + turn % RESTS) * BN, da[X[p - 1][i]] + 2 * k4,
                                          db[W[p - 1][i]] + 2 * k4, idesc, it > 0 || p > 1 || turn >= RESTS);
                            }
                    }
                    if (p == 2) {
#pragma unroll
                        for (int i = 0; i < 3; ++i) umma_commit(slot[i]);
                        if (it + 3 >= nit) {
                            umma_commit(accfull);
                            uint32_t all = used;
#pragma unroll
                            for (int k4 = 0; k4 < KC / 16; ++k4) all |= 1u << (lead + k4 < LEADS ? lead + k4 : lead + k4 - LEADS);
                            used_s[0] = all | ((1u << RESTS) - 1) << LEADS;
                            mbar_arrive_one(accfull);
                        }
                    }
                }
                __syncwarp();
                if (++s == STAGES) {
                    s = 0;
                    phase ^= 1;
                }
            }
#pragma unroll
            for (int k4 = 0; k4 < KC / 16; ++k4) {
                used |= 1u << lead;
                lead = lead + 1 < LEADS ? lead + 1 : 0;
            }
        }
    } else {
        // ---- issuers: warp i takes stages i, i + NI, ... in order and accumulates them in
        // its own accumulator; the partial sums are added in the epilogue.  (Two, because a lane of a diverged warp
        // took ~150 cycles to issue a product, which held a single issuer up; an elected lane takes ~30.  The second
        // accumulator stays for the sums: the tensor core truncates as it adds, see conv_cluster_cost.)
        constexpr uint32_t idesc = umma_idesc_bf16(CT_TM, BN);
        const int me = warp - CT_GATHER_WARPS;
        const uint32_t tm_acc = tmem_base + me * ACCS * BN;
        const uint64_t da0 = umma_desc_kmajor(sbase, ROWB), db0 = umma_desc_kmajor(sbase + A_BYTES, ROWB);
        uint32_t used = 0;
        int lead = 0;          // stages of this issuer with leading products
        int s = me, phase = 0, chunk = F32 ? (first + me) % kchunks : 0;
        for (int it = me; it < nit; it += NI) {
            ok &= mbar_wait(full0 + 8 * s, phase, abort);
            fence_after_sync();
            const uint64_t da = da0 + s * (STAGE_BYTES >> 4), db = db0 + s * (STAGE_BYTES >> 4);
            // accumulator of a product: the leading ones go round the first three (split_f32.cuh)
            auto target = [&](int k4) { return F32 ? ((chunk * KC + k4 * 16) * 6 < a.cin ? lead % SPLIT_MAIN : SPLIT_MAIN) : 0; };
            if (elect_one()) {
                uint32_t seen = used;
#pragma unroll
                for (int k4 = 0; k4 < KC / 16; ++k4) {
                    const uint32_t acc = target(k4);
                    umma_bf16(tm_acc + acc * BN, da + 2 * k4, db + 2 * k4, idesc, F32 ? (seen >> acc) & 1 : it >= NI || k4 > 0);
                    seen |= 1u << acc;
                }
                umma_commit(empty0 + 8 * s);
                if (it + NI >= nit) {
                    umma_commit(accfull);
                    if (F32) {
                        used_s[me] = seen;
                        mbar_arrive_one(accfull);
                    }
                }
            }
            __syncwarp();
            if (F32) {
#pragma unroll
                for (int k4 = 0; k4 < KC / 16; ++k4) used |= 1u << target(k4);
                lead += chunk * KC * 6 < a.cin;
                chunk += NI;
                while (chunk >= kchunks) chunk -= kchunks;
            }
            s += NI;
            if (s >= STAGES) {
                s -= STAGES;
                phase ^= 1;
            }
        }
        // an issuer without a stage
        if (nit > 0 && nit <= me && lane == 0) {
            mbar_arrive_one(accfull);
            if (F32) {
                used_s[me] = 0;
                mbar_arrive_one(accfull);
            }
        }
    }
    // until the rings of the cluster are free: partial sums go there (a gathering warp has read its first sums by then)
    bool met = !SPLIT;
    auto meet = [&]() {
        __syncwarp();
        cluster_sync();
        met = true;
    };
    if (warp < CT_GATHER_WARPS) {
        // ---- epilogue: thread = voxel ----------------------------------------------------------
        const bool read_acc = nit > 0 && __all_sync(0xffffffffu, ok);    // tcgen05.ld is warp-wide
        const int q = warp & 3, half = warp >> 2;      // lane quarter of tensor memory, half of the columns
        const int64_t v = rows_s[q * 32 + lane];
        const uint32_t tm = tmem_base + ((uint32_t)(q * 32) << 16);
        constexpr int NCB = BN / 32;                   // 32-column blocks, split between the two halves
#pragma unroll 1
        for (int cb = half * ((NCB + 1) / 2); cb < (half == 0 ? (NCB + 1) / 2 : NCB); ++cb) {
            uint32_t acc[32];
            if (F32) {
                // from the small products to the leading ones, issuer after issuer
#pragma unroll
                for (int e = 0; e < 32; ++e) acc[e] = 0;
#pragma unroll 1
                for (int z = ACCS - 1; z >= 0; --z)
#pragma unroll 1
                    for (int i = 0; i < NI; ++i) {
                        if (!read_acc || !((*reinterpret_cast<volatile uint32_t*>(used_s + i) >> z) & 1)) continue;
                        uint32_t more[32];
                        tmem_ld32(tm + (i * ACCS + z) * BN + cb * 32, more);
                        tmem_ld_wait();
                        tmem_ld_fence(more);
#pragma unroll
                        for (int e = 0; e < 32; ++e)
                            acc[e] = __float_as_uint(__uint_as_float(acc[e]) + __uint_as_float(more[e]));
                    }
            } else if (read_acc) {
                tmem_ld32(tm + cb * 32, acc);
                tmem_ld_wait();
                // the other issuers' partial sums, added in a fixed order
#pragma unroll 1
                for (int i = 1; i < NI && i < nit; ++i) {
                    uint32_t more[32];
                    tmem_ld32(tm + i * BN + cb * 32, more);
                    tmem_ld_wait();
#pragma unroll
                    for (int e = 0; e < 32; ++e)
                        acc[e] = __float_as_uint(__uint_as_float(acc[e]) + __uint_as_float(more[e]));
                }
            } else {
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] = 0;
            }
            if (SPLIT) {
                if (!met) meet();
                // to the CTA that finishes the row
                const int rows = CT_TM / (int)gridDim.z, r = q * 32 + lane;
                const uint32_t at = peer_address(
                    sbase + (((int)cluster_rank() * rows + r % rows) * PART_PITCH + cb * 32) * 4, r / rows);
#pragma unroll
                for (int g = 0; g < 8; ++g)
                    st_cluster_f4(at + g * 16, __uint_as_float(acc[g * 4]), __uint_as_float(acc[g * 4 + 1]),
                                  __uint_as_float(acc[g * 4 + 2]), __uint_as_float(acc[g * 4 + 3]));
                continue;
            }
            if (v < 0) continue;
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                float y[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = __uint_as_float(acc[g * 8 + i]) + bias_s[cb * 32 + g * 8 + i];
                ct_store_f32(a, v, col0 + cb * 32 + g * 8, y);
            }
        }
    }
    if (!met) meet();
    if (SPLIT) {
        // this CTA's rows: the cluster's partial sums in rank order, bias, bf16
        __syncwarp();
        cluster_sync();
        const int parts = (int)gridDim.z, rows = CT_TM / parts, r0 = rows * (int)cluster_rank();
        for (int e = tid; e < rows * (BN / 8); e += CT_THREADS) {
            const int r = e / (BN / 8), c = e % (BN / 8) * 8;
            const int64_t v = rows_s[r0 + r];
            if (v < 0) continue;
            const float* sums = reinterpret_cast<const float*>(smem) + r * PART_PITCH + c;
            float y[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] = 0.f;
            for (int z = 0; z < parts; ++z) {
                const float4* p = reinterpret_cast<const float4*>(sums + z * rows * PART_PITCH);
                const float4 m = p[0], w = p[1];
                y[0] += m.x; y[1] += m.y; y[2] += m.z; y[3] += m.w;
                y[4] += w.x; y[5] += w.y; y[6] += w.z; y[7] += w.w;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) y[i] += bias_s[c + i];
            if (F32)
                ct_store_f32(a, v, col0 + c, y);
            else
                *reinterpret_cast<uint4*>((__nv_bfloat16*)a.out + v * a.cout + col0 + c) =
                    make_uint4(pack_bf16(y[0], y[1]), pack_bf16(y[2], y[3]), pack_bf16(y[4], y[5]), pack_bf16(y[6], y[7]));
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == CT_GATHER_WARPS) {
        fence_after_sync();
        tmem_dealloc(tmem_base, TM_COLS);
    }
    if (lane == 0 && (!ok || (tid == 0 && *abort))) atomicOr(a.status, PTV3_STATUS_WAIT_LIMIT);
}

bool conv_tc05_supported(int c_in, int c_out, int kernel_volume)
{
    if (kernel_volume > CT_MAX_KVOL) return false;
    if (c_in == 32 && c_out == 32) return true;
    return c_in % 64 == 0 && c_in <= 4096 && c_out % 64 == 0 && c_out <= 4096;
}

template <int BN, int STAGES>
static constexpr size_t conv_tc05_smem()
{
    return (size_t)STAGES * (CT_TM + BN) * CT_KC * 2 + CT_MAX_KVOL * CT_TM * 4 + CT_TM * 8 + 32 * 4 + BN * 4 +
           8 * (2 * STAGES + 1) + 32 + 1024;
}

template <int BN, int STAGES, int NI, bool SPLIT, int FORM>
static int launch_conv_tc05_as(const void* weight, const ConvTcArgs& a, cudaStream_t stream, int parts)
{
    constexpr bool F32 = FORM != CT_BF16;
    CUtensorMap mw;
    const uint64_t wcols = (uint64_t)a.kvol * (F32 ? a.cin / 6 * split_stored(a.cin / 6) : a.cin);
    const int rc = make_tensor_map_bf16(&mw, weight, (uint64_t)a.cout, wcols, wcols * 2, BN, CT_KC);
    if (rc) return rc;
    constexpr size_t smem = conv_tc05_smem<BN, STAGES>();
    auto kern = conv_tc05_kernel<BN, STAGES, NI, SPLIT, FORM>;
    if (allow_smem(kern) != cudaSuccess)
        return check_launch("ptv3_subm_conv_fwd: shared memory attribute");
    const dim3 grid((unsigned)((a.n + CT_TM - 1) / CT_TM), a.cout / BN, parts);
    launch_dependent_cluster(kern, grid, dim3((CT_GATHER_WARPS + NI) * 32), smem, stream, dim3(1, 1, parts), mw, a);
    count_launches(1);
    return check_launch("ptv3_subm_conv_fwd");
}

// CTAs in clusters of `parts` that run at once (the driver's answer: a cluster lives in one GPC)
template <int BN, int STAGES, int NI, int FORM>
static int conv_tc05_capacity(int parts)
{
    static std::atomic<int> known[4];
    const int slot = parts == 2 ? 1 : parts == 4 ? 2 : 3;
    int c = known[slot].load(std::memory_order_relaxed);
    if (c == 0) {
        auto kern = conv_tc05_kernel<BN, STAGES, NI, true, FORM>;
        if (allow_smem(kern) != cudaSuccess) return 0;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(SMS, 1, parts);
        cfg.blockDim = dim3((CT_GATHER_WARPS + NI) * 32);
        cfg.dynamicSmemBytes = conv_tc05_smem<BN, STAGES>();
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = parts;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, kern, &cfg) != cudaSuccess) {
            cudaGetLastError();
            clusters = 0;
        }
        c = clusters > 0 ? clusters * parts : -1;
        known[slot].store(c, std::memory_order_relaxed);
    }
    return c;
}

struct ConvVariant {
    int bn;
    double fixed_us, load_us, stage_us;      // load_us: more for a CTA on every SM
    int (*plain)(const void*, const ConvTcArgs&, cudaStream_t, int);
    int (*split)(const void*, const ConvTcArgs&, cudaStream_t, int);
    int (*capacity)(int);
};
constexpr int CT_VARIANTS = 3;
// fp32 output (the accumulators of 64 or 128 columns fill the tensor memory of an SM).  us, 64 wide in clusters of 1, 2, 4, 8 |
// 128 wide: 822 x 256 94 55 37 - | 110 64 42 34, 487 x 128 54 34 26 22 | 66 41 30 26, 75 x 512 208 110 64 41 | 266 143 81 51.
static const ConvVariant g_variants_f32[CT_VARIANTS] = {
    {64, 6.5, 0, 0.56, launch_conv_tc05_as<64, 8, 1, false, CT_PARTS>, launch_conv_tc05_as<64, 8, 1, true, CT_PARTS>,
     conv_tc05_capacity<64, 8, 1, CT_PARTS>},
    {128, 9.5, 0, 0.63, launch_conv_tc05_as<128, 6, 1, false, CT_PARTS>, launch_conv_tc05_as<128, 6, 1, true, CT_PARTS>,
     conv_tc05_capacity<128, 6, 1, CT_PARTS>},
    {1 << 20, 0, 0, 0, nullptr, nullptr, nullptr}};
// ... of pieces, and all of 32 columns.  us, 64 wide | 32 wide: 111 445 x 32 -> 64 118.7 | 204.7, -> 128 231.5 | 401.8
static const ConvVariant g_variants_f32_pieces[CT_VARIANTS] = {
    {64, 6.5, 0, 0.20, launch_conv_tc05_as<64, 8, 2, false, CT_PIECES>, launch_conv_tc05_as<64, 8, 2, true, CT_PIECES>,
     conv_tc05_capacity<64, 8, 2, CT_PIECES>},
    {32, 6.5, 0, 0.18, launch_conv_tc05_as<32, 8, 2, false, CT_PIECES>, launch_conv_tc05_as<32, 8, 2, true, CT_PIECES>,
     conv_tc05_capacity<32, 8, 2, CT_PIECES>},
    {1 << 20, 0, 0, 0, nullptr, nullptr, nullptr}};
// bf16: clusters here, whole tiles in conv_stream.cu
static const ConvVariant g_variants[CT_VARIANTS] = {
    {64, 6.9, 1.6, 0.19, nullptr, launch_conv_tc05_as<64, 8, 2, true, CT_BF16>, conv_tc05_capacity<64, 8, 2, CT_BF16>},
    {128, 8.7, 1.6, 0.26, nullptr, launch_conv_tc05_as<128, 6, 2, true, CT_BF16>, conv_tc05_capacity<128, 6, 2, CT_BF16>},
    {256, 12., 1.6, 0.37, nullptr, launch_conv_tc05_as<256, 4, 2, true, CT_BF16>, conv_tc05_capacity<256, 4, 2, CT_BF16>}};

// The cluster size and tile width with the shortest estimated time: waves of CTAs, each taking a
// fixed time (prologue, epilogue) and its stages.  Wide tiles gather a row once for more output
// channels; clusters fill SMs that a single wave leaves idle.  `stages`: of a tile.  The constants are measured.
//
// The choice also sets how many partial sums a tile has, issuers x CTAs of its cluster, and the tensor core truncates where
// an fp32 addition rounds.  Share of the results (bf16) that are not the rounded 64-bit sum, with the lines as they are and
// with twice to four times the sums (clusters of up to eight wherever they fit a wave): 3 900 x 64 0.007 / 0.005 %,
// 9 000 x 64 0.013 / 0.008, 5 000 x 128 0.032 / 0.017, 1 200 x 256 0.035 / 0.011, 2 500 x 256 0.067 / 0.021, 2 400 x 512
// 0.133 / 0.072; the persistent kernel's two sums 9 000 x 512 0.147.  The error against 64 bits is that of the rounding to
// bf16 in all of them (0.00165 of the norm, the same to six digits).
static double conv_cluster_cost(const ConvVariant* variants, const ConvTcArgs& a, double stages, int* best_v, int* best_parts)
{
    const int64_t tiles = (a.n + CT_TM - 1) / CT_TM;
    double best = 0;
    *best_v = -1;
    for (int v = 0; v < CT_VARIANTS; ++v) {
        const ConvVariant& var = variants[v];
        if (a.cout % var.bn) continue;
        const int64_t ctas = tiles * (a.cout / var.bn);
        for (int parts = var.plain ? 1 : 2; parts <= 8; parts *= 2) {
            const int64_t room = parts == 1 ? (int64_t)SMS : (int64_t)var.capacity(parts);
            if (room < parts) continue;
            if (parts > 1 && (ctas * parts > room || stages < 2 * parts)) continue;       // a cluster only within one wave
            const double cost = (double)((ctas * parts + room - 1) / room) *
                                (var.fixed_us + var.load_us * (double)(ctas * parts) / SMS + stages / parts * var.stage_us);
            if (*best_v < 0 || cost < best) {
                best = cost;
                *best_v = v;
                *best_parts = parts;
            }
        }
    }
    return best;
}

// bf16: persistent CTAs on whole tiles (conv_stream.cu) or clusters that share them, whichever should be faster.  About
// half of the offsets of a tile are in use (9 to 19 of 27 on rooms from fine to coarse levels).  A persistent CTA
// takes a fixed time and its stages, at the pace of its own chain or, with all SMs at work, of what they share.
// us, estimated best of the clusters against the persistent kernel, measured: 1 757 x 256 13.4 / 18.3 (it was 19.9 in
// clusters of eight with 256-wide tiles, when all offsets were counted), 457 x 512 15.5 / 32, 2 240 x 512 25.3 / 30,
// 6 760 x 128 11.9 / 11.7, 7 700 x 256 23.0 / 22.8, 5 200 x 512 56.7 / 44.8, 26 000 x 64 12.3 / 10.8.
static int conv_stream_width(const ConvTcArgs& a, double stages, double* cost)
{
    static const struct {
        int bn;
        double fixed_us, chain_us, shared_us;
    } widths[3] = {{64, 6.3, 0.19, 0.31}, {128, 9.5, 0.21, 0.36}, {256, 12., 0.53, 0.57}};
    const int64_t tiles = (a.n + CT_TM - 1) / CT_TM;
    int best = 0;
    for (const auto& w : widths) {
        if (a.cout % w.bn) continue;
        const int64_t ctas = tiles * (a.cout / w.bn);
        const double chain = (double)((ctas + SMS - 1) / SMS) * w.chain_us, shared = (double)ctas / SMS * w.shared_us;
        const double t = w.fixed_us + stages * (chain > shared ? chain : shared);
        if (!best || t < *cost) {
            best = w.bn;
            *cost = t;
        }
    }
    return best;
}

int launch_conv_tc05(const void* feat, const int32_t* nbr, const void* weight, const void* bias, void* out,
                     const int64_t* row_order, int64_t n, int c_in, int c_out, int kvol, bool planned,
                     uint32_t* status, cudaStream_t stream)
{
    ConvTcArgs a{};
    a.feat = (const __nv_bfloat16*)feat;
    a.nbr = nbr;
    a.bias = bias;
    a.out = out;
    a.row_order = row_order;
    a.n = n;
    a.cin = c_in;
    a.cout = c_out;
    a.kvol = kvol;
    a.planned = planned;
    a.status = status;
    auto stream_form = [&](int bn) {
        return launch_conv_stream(feat, nbr, weight, bias, out, row_order, n, c_in, c_out, kvol, bn, planned, status,
                                  stream);
    };
    if (c_in == 32) return stream_form(32);
    const double stages = 0.5 * kvol * (c_in / 64);
    double whole = 0;
    int v, parts = 1;
    const int bn = conv_stream_width(a, stages, &whole);
    const double shared = conv_cluster_cost(g_variants, a, stages, &v, &parts);
    if (v < 0 || whole <= shared) return stream_form(bn);
    return g_variants[v].split(weight, a, stream, parts);
}

// fp32 on split operands (see split_f32.cuh)
int launch_conv_split(const void* feat, const int32_t* nbr, const void* weight, const float* bias, float* out,
                      void* split_out, const int64_t* row_order, int64_t n, int c_in, int c_out, int kvol,
                      uint32_t* status, cudaStream_t stream)
{
    ConvTcArgs a{};
    a.feat = (const __nv_bfloat16*)feat;
    a.nbr = nbr;
    a.bias = bias;
    a.out = out;
    a.split_out = (__nv_bfloat16*)split_out;
    a.row_order = row_order;
    a.n = n;
    a.cin = 6 * c_in;
    a.cout = c_out;
    a.kvol = kvol;
    a.status = status;
    int v, parts = 1;
    // A slice is 64 channels, so parts are for whole ones, and their accumulators fill tensor memory with 64 columns or
    // 128; other widths (odd multiples of 32, stored as six pieces) and 32 columns walk the pieces in 64-column chunks.
    // (Stages: half of the offsets in use; of pieces all.)
    const bool slices = c_in % 64 == 0 && c_out % 64 == 0;
    const ConvVariant* variants = slices ? g_variants_f32 : g_variants_f32_pieces;
    conv_cluster_cost(variants, a, slices ? 0.5 * a.kvol * (c_in / 64) * 3 : (double)a.kvol * (a.cin / 64), &v, &parts);
    PTV3_REQUIRE(v >= 0, PTV3_ERR_UNSUPPORTED, "ptv3_subm_conv_split_fwd: no kernel of %d -> %d channels", c_in, c_out);
    return (parts > 1 ? variants[v].split : variants[v].plain)(weight, a, stream, parts);
}

}  // namespace ptv3
