// Tensor-core path of the patch attention core for bf16 features and head
// dimension 16 (every stage of the default backbone).
//
// One CTA owns one (sequence, head) pair (optionally a slice of its queries):
// the keys and values of the whole sequence are gathered once into shared
// memory with cp.async, straight from the point-major qkv tensor through
// order[pad[.]].  Each warp then walks 16-query tiles: S = Q K^T for 64 keys at
// a time by mma.sync (k = head_dim = 16, one instruction per 16x8 tile), exp2 on
// the accumulator registers, P rounded to bf16 in the same registers re-used as
// the A operand of P V.
// Nothing but q, k, v and the output rows touches global memory; scores never
// leave registers.  Rows are written back to out[order[pad[.]]] only by the
// padded row that owns the point (borrowed rows of a last patch are dropped).
//
// Replaces model.py:452-484 for the bf16 case (see attention.cu for the
// contract).  Work per (sequence, head): 4 L^2 16 tensor FLOPs and L^2 exps;
// at head_dim 16 the exp unit, not the tensor pipe, is the limiter.
//
// Softmax needs no reference value where no score can leave the range of exp2: |q . k| <= |q| max|k|, so a
// tile whose rows pass that test (AM_BOUND) runs without maxima, votes and rescaling, and its 16-key
// groups do not depend on one another; the other tiles, and the ragged end of a sequence, run the
// online form.  400 000 points x 64 channels: 0.502 -> 0.455 ms, 70 -> 77 % of the exp unit's rate over
// the launch (83 % of it while warps are active, at 120 000 points).  What is left: the gather before a CTA's
// first product, the last wave, and 20 mma.sync of 8 cycles per 16 x 64 scores, which share register ports with
// the FMA pipe, so that exponentials moved there (a quartic on 2 to 8 of 16 pairs) gain nothing: 0.446 to 0.498 ms.
#include "common.cuh"
#include "attention_mma.cuh"
#include "mma_util.cuh"

namespace ptv3 {

constexpr int AM_THREADS = 256;
constexpr int AM_WARPS = AM_THREADS / 32;
constexpr int AM_KC = 64;           // keys per online-softmax step
constexpr int AM_D = 16;
constexpr int AM_MAX_SLICES = 16;
constexpr size_t AM_SM_SMEM = 228 * 1024;    // shared memory of an SM, of which a CTA takes 1 KiB more than it asks for
constexpr float AM_LOG2E = 1.4426950408889634f;
constexpr float AM_LAZY = 8.f;       // slack of the running maximum, in powers of two
constexpr float AM_BOUND = 80.f;     // largest |score| (exp2 domain) taken without a reference value

// byte offset of 16-byte chunk c (0/1) of row r in a [rows][16] bf16 tile whose
// chunks are swapped in rows 4..7 (mod 8) so that 8-row ldmatrix reads hit 32
// distinct banks
__device__ __forceinline__ uint32_t kv_offset(int r, int c)
{
    return (uint32_t)(r * 32 + ((c ^ ((r >> 2) & 1)) << 4));
}

__device__ __forceinline__ uint32_t scale_bf16x2(uint32_t v, float s)
{
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
    return pack_bf16(f.x * s, f.y * s);
}

// How K and V come to shared memory.  A copy instruction costs a cycle per line it touches, so two lanes that take the
// halves of one row cost half of one lane per row with a half at a time.  That shortens the start of launches of a few
// waves, where CTAs gather at the same time (us: 405 points of 8 heads 5.5 -> 5.1, 1 560 of 4 9.1 -> 8.0, 6 000 of 2
// 10.7 -> 9.8, 1 757 of 16 16.3 -> 15.7, 4 x 560 of 32 20.8 -> 19.8, 632 CTAs of 256 points 19.7 -> 19.0); in long ones a CTA's
// gather is hidden by the two beside it, and the loop behind it gets worse registers (half rows: 16 bytes of a thread's are
// spilled, 8 in the planned form, none in the long one; 6 252 CTAs of 256 points 146.5 -> 148.1, 60 000 points of 2 048 174.7 ->
// 183).
enum AmGather {
    AM_LONG,          // a row per lane
    AM_SHORT,         // half a row per lane
    AM_PLANNED        // the same, and the geometry may be read before the wait for the kernel ahead (see linear.cuh)
};

template <bool PACKED, AmGather GATHER>
__global__ void __launch_bounds__(AM_THREADS, 3) attn_mma_d16_kernel(
    const __nv_bfloat16* qkv, const int64_t* order, const int64_t* pad, const int64_t* unpad, const int32_t* cu_seqlens,
    __nv_bfloat16* out, int C, float scale, int lpad_max, uint32_t* status)
{
    pdl_launch_next();
    if (GATHER != AM_PLANNED) pdl_wait();
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char* Ks = smem;
    unsigned char* Vs = smem + (size_t)lpad_max * 32;
    // point row of every padded row of the sequence, negated - 1 where the padded row does not own
    // its point (borrowed rows): the gather walks pad -> order for every row anyway, and the query
    // tiles then need one dependent load instead of three
    int32_t* src_s = reinterpret_cast<int32_t*>(smem + (size_t)lpad_max * 64);

    // heads and query slices vary fastest over the grid (blockIdx.x = slice * heads + head): the
    // CTAs of one patch run together, so the rows they all gather from (a row holds every head's
    // q, k and v side by side) are fetched from DRAM once
    const int n_heads = C / 16;
    const int seq = blockIdx.y, h = blockIdx.x % n_heads;
    const int slice = blockIdx.x / n_heads, n_slices = gridDim.x / n_heads;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t start = cu_seqlens[seq];
    const int L = (int)(cu_seqlens[seq + 1] - start);
    if (L <= 0) {
        pdl_wait();          // (no CTA ends before the kernel ahead has: the one behind relies on it)
        return;
    }
    // shared memory was sized from the caller's max_seqlen: a longer sequence (a plan made
    // for a larger patch) is reported and skipped, uniformly over the CTA, before any write
    if (L > lpad_max) {
        pdl_wait();
        if (tid == 0 && status) atomicOr(status, PTV3_STATUS_BAD_INDEX);
        return;
    }
    const int Lp = (L + AM_KC - 1) / AM_KC * AM_KC;   // <= lpad_max
    const int ntiles = (L + 15) / 16;
    const int tiles_per_slice = (ntiles + n_slices - 1) / n_slices;
    const int tile_lo = slice * tiles_per_slice;
    const int tile_hi = min(ntiles, tile_lo + tiles_per_slice);
    if (tile_lo >= tile_hi) {
        pdl_wait();
        return;
    }
    const int64_t row_stride = 3 * (int64_t)C;

    if (GATHER != AM_LONG) {
        // ---- K and V of the whole sequence: two lanes a row, a 16-byte half each ------------------------------
        const int half = lane & 1;
        auto gather32 = [&](int base, int32_t e) {      // rows base .. base + 31, of which this lane knows one
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                const int r = base + 16 * k + (lane >> 1);
                const int32_t er = __shfl_sync(0xffffffffu, e, 16 * k + (lane >> 1));
                if (r < L) {
                    const __nv_bfloat16* kp = qkv + C + h * AM_D + (int64_t)(er >= 0 ? er : -(er + 1)) * row_stride + 8 * half;
                    cp_async16(smem_u32(Ks) + kv_offset(r, half), kp);
                    cp_async16(smem_u32(Vs) + kv_offset(r, half), kp + C);
                } else if (r < Lp) {
                    const uint4 z = make_uint4(0, 0, 0, 0);
                    *reinterpret_cast<uint4*>(Ks + kv_offset(r, half)) = z;
                    *reinterpret_cast<uint4*>(Vs + kv_offset(r, half)) = z;
                }
            }
        };
        // rows of the sequence, four rounds at a time: a chain of two dependent loads (points and padded rows are numbered
        // in 32 bits, as the caller's n and cu_seqlens are)
        for (int base = 32 * warp; base < Lp; base += 4 * AM_THREADS) {
            const int rb = base + lane;
            int32_t pd[4], src[4], own[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) pd[i] = rb + i * AM_THREADS < L ? (int32_t)pad[start + rb + i * AM_THREADS] : -1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                src[i] = pd[i] >= 0 ? (int32_t)order[pd[i]] : 0;
                own[i] = pd[i] >= 0 ? (int32_t)unpad[pd[i]] : 0;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (GATHER == AM_SHORT && base + i * AM_THREADS < Lp) gather32(base + i * AM_THREADS, src[i]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = rb + i * AM_THREADS;
                if (r < L) src_s[r] = own[i] == (int32_t)start + r ? src[i] : -src[i] - 1;
            }
        }
        if (GATHER == AM_PLANNED) {
            // (so far only the geometry was read: planned, that happens beside the kernel before this one in the stream)
            pdl_wait();
            for (int base = 32 * warp; base < Lp; base += AM_THREADS)
                gather32(base, base + lane < L ? src_s[base + lane] : 0);          // (this lane's own)
        }
    } else {
        // ---- gather K and V of the whole sequence ------------------------------
        // four rows per thread at a time: the chain pad -> order -> row is three dependent loads long
        for (int rb = tid; rb < Lp; rb += 4 * AM_THREADS) {
            int64_t pd[4], src[4], own[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) pd[i] = rb + i * AM_THREADS < L ? pad[start + rb + i * AM_THREADS] : -1;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                src[i] = pd[i] >= 0 ? order[pd[i]] : 0;
                own[i] = pd[i] >= 0 ? unpad[pd[i]] : 0;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int r = rb + i * AM_THREADS;
                if (r >= Lp) break;
                if (pd[i] >= 0) {
                    src_s[r] = own[i] == start + r ? (int32_t)src[i] : -(int32_t)src[i] - 1;
                    const __nv_bfloat16* kp = qkv + src[i] * row_stride + C + h * AM_D;
                    cp_async16(smem_u32(Ks) + kv_offset(r, 0), kp);
                    cp_async16(smem_u32(Ks) + kv_offset(r, 1), kp + 8);
                    cp_async16(smem_u32(Vs) + kv_offset(r, 0), kp + C);
                    cp_async16(smem_u32(Vs) + kv_offset(r, 1), kp + C + 8);
                } else {
                    const uint4 z = make_uint4(0, 0, 0, 0);
                    *reinterpret_cast<uint4*>(Ks + kv_offset(r, 0)) = z;
                    *reinterpret_cast<uint4*>(Ks + kv_offset(r, 1)) = z;
                    *reinterpret_cast<uint4*>(Vs + kv_offset(r, 0)) = z;
                    *reinterpret_cast<uint4*>(Vs + kv_offset(r, 1)) = z;
                }
            }
        }
    }
    __shared__ float knorm_s[AM_WARPS];
    cp_async_commit();
    cp_async_wait<0>();
    // largest squared norm of a key (every thread reads back what it copied itself)
    float knorm = 0.f;
    if (GATHER != AM_LONG) {
        for (int base = 32 * warp; base < Lp; base += AM_THREADS)
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                float n = sq_norm8(*reinterpret_cast<const uint4*>(Ks + kv_offset(base + 16 * k + (lane >> 1), lane & 1)));
                n += __shfl_xor_sync(0xffffffffu, n, 1);
                knorm = max_nan(knorm, n);
            }
    } else {
        for (int r = tid; r < L; r += AM_THREADS)
            knorm = max_nan(knorm, sq_norm16(*reinterpret_cast<const uint4*>(Ks + kv_offset(r, 0)),
                                             *reinterpret_cast<const uint4*>(Ks + kv_offset(r, 1))));
    }
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) knorm = max_nan(knorm, __shfl_xor_sync(0xffffffffu, knorm, d));
    if (lane == 0) knorm_s[warp] = knorm;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < AM_WARPS; ++w) knorm = max_nan(knorm, knorm_s[w]);

    const int g = lane >> 2, t = lane & 3;
    // ldmatrix row/chunk this lane addresses inside a 16-key group
    const int k_row = (lane & 7) + ((lane >> 4) << 3), k_chunk = (lane >> 3) & 1;   // K: keys x d
    const int v_row = (lane & 7) + (((lane >> 3) & 1) << 3), v_chunk = lane >> 4;   // V (transposed)
    const uint32_t ks_base = smem_u32(Ks), vs_base = smem_u32(Vs);
    const float sl2 = AM_LOG2E;

    // query rows of a warp's tile, fetched one tile ahead (the row numbers are in shared memory,
    // so this is a single load per row)
    auto fetch_q = [&](int tile, uint32_t (&q)[4]) {
        const int r0 = tile * 16 + g, r1 = r0 + 8;
        q[0] = q[1] = q[2] = q[3] = 0u;
        if (tile < tile_hi && r0 < L) {
            const int32_t e = src_s[r0];
            const uint32_t* qp = reinterpret_cast<const uint32_t*>(qkv + (int64_t)(e >= 0 ? e : -(e + 1)) * row_stride + h * AM_D);
            q[0] = qp[t];
            q[2] = qp[4 + t];
        }
        if (tile < tile_hi && r1 < L) {
            const int32_t e = src_s[r1];
            const uint32_t* qp = reinterpret_cast<const uint32_t*>(qkv + (int64_t)(e >= 0 ? e : -(e + 1)) * row_stride + h * AM_D);
            q[1] = qp[t];
            q[3] = qp[4 + t];
        }
    };
    uint32_t qn[4];
    fetch_q(tile_lo + warp, qn);
    for (int tile = tile_lo + warp; tile < tile_hi; tile += AM_WARPS) {
        const int r0 = tile * 16 + g, r1 = r0 + 8;
        const bool ok0 = r0 < L, ok1 = r1 < L;
        const uint32_t qa[4] = {scale_bf16x2(qn[0], scale), scale_bf16x2(qn[1], scale), scale_bf16x2(qn[2], scale),
                                scale_bf16x2(qn[3], scale)};
        fetch_q(tile + AM_WARPS, qn);
        float m0 = -INFINITY, m1 = -INFINITY, l0, l1;
        float o[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        float osum[4] = {0.f, 0.f, 0.f, 0.f};   // row sums of the rounded probabilities: a ones column of V

        int kc0 = 0;
        if (!PACKED) {
            // the tile's query norms against the largest key norm; a NaN fails the test
            float n0 = sq_norm_bf16x2(qa[0], sq_norm_bf16x2(qa[2], 0.f));
            float n1 = sq_norm_bf16x2(qa[1], sq_norm_bf16x2(qa[3], 0.f));
            n0 += __shfl_xor_sync(0xffffffffu, n0, 1);
            n1 += __shfl_xor_sync(0xffffffffu, n1, 1);
            n0 += __shfl_xor_sync(0xffffffffu, n0, 2);
            n1 += __shfl_xor_sync(0xffffffffu, n1, 2);
            const float lim = (AM_BOUND / AM_LOG2E) * (AM_BOUND / AM_LOG2E);
            if (__all_sync(0xffffffffu, n0 * knorm <= lim && n1 * knorm <= lim)) {
                m0 = m1 = 0.f;
                const int full = L / AM_KC * AM_KC;
                for (; kc0 < full; kc0 += AM_KC) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        uint32_t kb[4], vb[4];
                        ldmatrix_x4(kb, ks_base + kv_offset(kc0 + 16 * j + k_row, k_chunk));
                        ldmatrix_x4_trans(vb, vs_base + kv_offset(kc0 + 16 * j + v_row, v_chunk));
                        float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
                        mma_bf16(s[0], qa, kb[0], kb[1]);
                        mma_bf16(s[1], qa, kb[2], kb[3]);
                        uint32_t a[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float px, py;
                            unpack2(mul2(pack2(s[i >> 1][2 * (i & 1)], s[i >> 1][2 * (i & 1) + 1]), pack2(sl2, sl2)), px,
                                    py);
                            a[i] = pack_bf16(fast_exp2(px), fast_exp2(py));
                        }
                        mma_bf16(o[0], a, vb[0], vb[1]);
                        mma_bf16(o[1], a, vb[2], vb[3]);
                        mma_bf16(osum, a, 0x3f803f80u, 0x3f803f80u);
                    }
                }
            }
        }
        for (int kc = kc0; kc < Lp; kc += AM_KC) {
            float s[8][4];
#pragma unroll
            for (int j = 0; j < 8; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                uint32_t kb[4];
                ldmatrix_x4(kb, ks_base + kv_offset(kc + 16 * j + k_row, k_chunk));
                mma_bf16(s[2 * j], qa, kb[0], kb[1]);
                mma_bf16(s[2 * j + 1], qa, kb[2], kb[3]);
            }
            if (kc + AM_KC > L) {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int col = kc + 8 * j + 2 * t;
                    if (col >= L) s[j][0] = s[j][2] = -INFINITY;
                    if (col + 1 >= L) s[j][1] = s[j][3] = -INFINITY;
                }
            }
            // three-input maxima (one instruction each on this architecture)
            float mx0 = fmaxf(s[0][0], s[0][1]), mx1 = fmaxf(s[0][2], s[0][3]);
#pragma unroll
            for (int j = 1; j < 8; ++j) {
                mx0 = fmaxf(fmaxf(mx0, s[j][0]), s[j][1]);
                mx1 = fmaxf(fmaxf(mx1, s[j][2]), s[j][3]);
            }
            // Lazy reference: the running "maximum" m only has to keep the exponentials in
            // range, so it is raised (and the output rescaled) only when some score of the
            // chunk exceeds it by more than AM_LAZY in the exp2 domain; probabilities then
            // stay below 2^AM_LAZY, exact in bf16's range and harmless in the fp32 sums.
            // After the first chunks of a sequence this is rare, and the common path needs
            // neither the cross-lane reduction nor the rescaling.
            if (__any_sync(0xffffffffu, (mx0 - m0) * sl2 > AM_LAZY || (mx1 - m1) * sl2 > AM_LAZY)) {
                mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
                mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
                mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
                mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
                const float mn0 = fmaxf(m0, mx0), mn1 = fmaxf(m1, mx1);
                // every chunk holds at least one real key, so mn is finite
                const float c0 = fast_exp2((m0 - mn0) * sl2), c1 = fast_exp2((m1 - mn1) * sl2);
                m0 = mn0;
                m1 = mn1;
                osum[0] *= c0;
                osum[2] *= c1;
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    o[n][0] *= c0;
                    o[n][1] *= c0;
                    o[n][2] *= c1;
                    o[n][3] *= c1;
                }
            }
            const float mn0 = m0, mn1 = m1;
            const float b0 = mn0 * sl2, b1 = mn1 * sl2;
            uint32_t pa[8][2];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                if (PACKED) {
                    // exponent argument rounded to bf16, two exps per instruction, the result
                    // already is the bf16 pair the next MMA consumes
                    pa[j][0] = exp2_bf16x2(pack_bf16(fmaf(s[j][0], sl2, -b0), fmaf(s[j][1], sl2, -b0)));
                    pa[j][1] = exp2_bf16x2(pack_bf16(fmaf(s[j][2], sl2, -b1), fmaf(s[j][3], sl2, -b1)));
                } else {
                    const float p0 = fast_exp2(fmaf(s[j][0], sl2, -b0));
                    const float p1 = fast_exp2(fmaf(s[j][1], sl2, -b0));
                    const float p2 = fast_exp2(fmaf(s[j][2], sl2, -b1));
                    const float p3 = fast_exp2(fmaf(s[j][3], sl2, -b1));
                    pa[j][0] = pack_bf16(p0, p1);
                    pa[j][1] = pack_bf16(p2, p3);
                }
            }
#pragma unroll
            for (int kk = 0; kk < 4; ++kk) {
                const uint32_t a[4] = {pa[2 * kk][0], pa[2 * kk][1], pa[2 * kk + 1][0], pa[2 * kk + 1][1]};
                uint32_t vb[4];
                ldmatrix_x4_trans(vb, vs_base + kv_offset(kc + 16 * kk + v_row, v_chunk));
                mma_bf16(o[0], a, vb[0], vb[1]);
                mma_bf16(o[1], a, vb[2], vb[3]);
                // a column of ones appended to V: the tensor core sums the rounded probabilities
                mma_bf16(osum, a, 0x3f803f80u, 0x3f803f80u);
            }
        }
        l0 = osum[0];
        l1 = osum[2];
        const int32_t e0 = ok0 ? src_s[r0] : -1, e1 = ok1 ? src_s[r1] : -1;     // >= 0: the row owns its point
        if (e0 >= 0) {
            const float inv = 1.f / l0;
            uint32_t* op = reinterpret_cast<uint32_t*>(out + e0 * (int64_t)C + h * AM_D);
            op[t] = pack_bf16(o[0][0] * inv, o[0][1] * inv);
            op[4 + t] = pack_bf16(o[1][0] * inv, o[1][1] * inv);
        }
        if (e1 >= 0) {
            const float inv = 1.f / l1;
            uint32_t* op = reinterpret_cast<uint32_t*>(out + e1 * (int64_t)C + h * AM_D);
            op[t] = pack_bf16(o[0][2] * inv, o[0][3] * inv);
            op[4 + t] = pack_bf16(o[1][2] * inv, o[1][3] * inv);
        }
    }
}

// How a launch is cut: slices of the queries of a (sequence, head) pair, each a CTA that gathers K and V again, and
// CTAs per SM.
struct AmCut {
    int slices, per_sm;
};

// The cut with the shortest estimated time.  Up to three CTAs share an SM (four schedulers, two warps of a CTA on
// each); a launch that gives no SM more than one or two is held to that number, because CTAs otherwise
// pile up on the SMs that are free first (2 sequences of 1 024 x 16 heads in eight slices: 23.9 us, 17.3 with two per SM).
// The estimate, in cycles (measured on sequences of 27 to 1 024; within 5 % from 32 pairs of 1 024 up):
//   * a CTA starts with a gather, 4 800 and 3 800 more per 1 024 rows and CTA of the SM, one after another;
//   * a scheduler takes 78 per tile and 16 keys, but one of its two warps in a CTA at least 172, the chain through
//     the units (a warp alone 136);
//   * where an SM has more CTAs than run at once they follow one another, at 1 500 more each (a gather, where
//     there is room for one).
// us with the cut before (a power of two of slices up to nearly two waves of three per SM) and now, 1 024 points a
// sequence: 12 pairs 17.1 / 10.6, 32 pairs 23.9 / 16.3, 56 pairs 29.3 / 25.7, 196 pairs 69.5 / 65.1, 392 pairs
// 130 / 121, 784 pairs 231 / 231; 32 pairs of 457 points 10.0 / 7.1, 128 pairs of 560 25.3 / 20.7.
static AmCut am_cut(int64_t pairs, int max_seqlen, size_t smem)
{
    const int tiles = (max_seqlen + 15) / 16;
    int fit = (int)(AM_SM_SMEM / (smem + 1024));
    fit = fit < 1 ? 1 : fit > 3 ? 3 : fit;
    const double rows = max_seqlen / 1024.0, steps = (max_seqlen + 15) / 16;
    AmCut best{1, fit};
    double least = 0;
    for (int q = 1; q <= AM_MAX_SLICES && (q - 1) * 4 < tiles; ++q) {
        const int per = (tiles + q - 1) / q, slices = (tiles + per - 1) / per;
        if (slices < q) continue;
        const int64_t on_sm = (pairs * slices + SMS - 1) / SMS;
        const int c = on_sm < fit ? (int)on_sm : fit;
        const double busy = 78. * on_sm * (on_sm > c && per >= 8 ? per / 4. : (per + 3) / 4);
        const double chain = (double)((on_sm + c - 1) / c) * (per / 8 * 172 + (per % 8 > 4 ? 172 : per % 8 ? 136 : 0));
        const double start = 4800 + 3800 * rows * c;
        const double t = start + steps * (busy > chain ? busy : chain) +
                         (on_sm - c) * (fit == 1 ? start : 700 + 800 * rows);
        if (q == 1 || t < least) {
            least = t;
            best = AmCut{slices, c};
        }
    }
    return best;
}

bool attn_mma_supported(int channels, int heads, int max_seqlen)
{
    return channels % heads == 0 && channels / heads == AM_D && channels % 8 == 0 &&
           max_seqlen <= ATTN_MMA_MAX_SEQLEN;
}

int launch_attn_mma(const void* qkv, const int64_t* order, const int64_t* pad, const int64_t* unpad,
                    const int32_t* cu, void* out, int n_seq, int max_seqlen, int C, int H, float scale,
                    bool packed_exp, bool planned, uint32_t* status, cudaStream_t stream)
{
    const int lpad = (max_seqlen + AM_KC - 1) / AM_KC * AM_KC;
    const size_t smem = (size_t)lpad * 68;      // K, V and the row numbers
    const AmCut cut = am_cut((int64_t)n_seq * H, max_seqlen, smem);
    // The look-up ahead of the wait pays where a launch has at most one CTA per SM, all of them at their beginning when the
    // kernel ahead ends (a pass over 6 000 points 1 550 -> 1 498 us).
    const int64_t ctas = (int64_t)n_seq * H * cut.slices;
    // (patches of more than 1 024 rows: one CTA per SM, which takes too long for its start to count)
    auto kern = packed_exp                                  ? attn_mma_d16_kernel<true, AM_LONG>
                : planned && ctas <= SMS                   ? attn_mma_d16_kernel<false, AM_PLANNED>
                : ctas <= 8 * SMS && max_seqlen <= 1024 ? attn_mma_d16_kernel<false, AM_SHORT>
                                                            : attn_mma_d16_kernel<false, AM_LONG>;
    if (allow_smem(kern) != cudaSuccess)
        return check_launch("ptv3_attention_fwd: shared memory attribute");
    // (shared memory that only so many CTAs find room for)
    const size_t least = cut.per_sm < 3 ? AM_SM_SMEM / (cut.per_sm + 1) : 0;
    const dim3 grid(H * cut.slices, n_seq);
    launch_dependent(kern, grid, dim3(AM_THREADS), smem > least ? smem : least, stream, (const __nv_bfloat16*)qkv,
                     order, pad, unpad, cu, (__nv_bfloat16*)out, C, scale, lpad, status);
    count_launches(1);
    return check_launch("ptv3_attention_fwd");
}

}  // namespace ptv3
