// fp32 patch attention (model.py:452-484), head dimension 16: the fp32 backbone's attention core, on the 5th-generation
// tensor cores with split operands (split_f32.cuh).
//
// A CTA owns 128 queries of a (patch, head) pair, a thread one of them (a lane of tensor memory).  Per block of 48 keys:
//   S = Q K^T from the three parts of each, the leading product q1 k1 in columns of its own beside the five small ones;
//   a thread adds the two, takes the exponentials, and writes the probabilities' three parts back over S;
//   O = P V from the parts, leading and small products apart again, is read back and added to the row in registers.
// The next block's S is issued behind this one's O, so that it is made while O is read and the block after it is split
// into the buffer that O has left.  Four CTAs to an SM, 128 columns of tensor memory each.
//
// Softmax needs no reference value where |q| max|k| bounds a block's scores (AX_BOUND, per warp); other blocks take their
// maximum first, and their probabilities are scaled by AX_LIFT: the parts of the smallest one above zero are normal numbers
// then too.  (A lower reference instead of the factor costs a score's last bits: error 3.6e-7 for 2.5e-7, q and k of 2 and 1.)
// V is scaled by AX_VSCALE, so that the last part of the smallest normal number is a normal one still.  (Q and
// K need no scale: what their parts lose down there is nothing to a score.)  A row whose squares are not below AX_HUGE or
// AX_HUGE_V (infinities and NaN among them: their parts would be NaN) sends the CTA to plain arithmetic over all keys.
//
// Before, queries were registers of a thread and keys came from shared memory, on CUDA cores; two or four queries to a thread.
// us, before (the better of the two) / now, patches of 1 024: 90 000 x 64 672 / 294, 40 000 x 64 315 / 148, 10 500 x 64 112 / 55,
// 2 800 x 128 72 / 46; patches of 410, 820 x 256 24.8 / 17.2, of 130, 260 x 512 12.5 / 8.5.  Error against 64 bits, rms of a
// row, q and k of size 1: 2.7e-7 / 1.5e-7, of 8 and 8: 1.3e-6 / 1.1e-6 (a row's sums are taken per block, and S and O lose
// only what four products in a row truncate).
// No unit is full: issue slots are 54 % busy (13 instructions for a pair of probabilities and their parts, and the splitting of
// a block's keys and values by each of a patch's CTAs), the L1 data pipe 58 %, the tensor pipe 37 %; four warps to a scheduler
// wait for tensor memory most, then at a block's two barriers (21 instructions a key and thread, the form before: 67 %).
// Without gain: 64 keys a block with O over S (S then waits for O: 332 us where this takes 296).  Leaving out 16 of the 20
// products of O, the splitting, the staging or the exponentials gave that form 4, 10, 8 and 4 %.
#include "attention_mma.cuh"
#include "common.cuh"
#include "mma_util.cuh"
#include "split_f32.cuh"
#include "tc05.cuh"
#include <type_traits>

namespace ptv3 {

using namespace tc05;

constexpr int AX_THREADS = 128, AX_QT = 128;
constexpr int AX_KC = 48;                    // keys of a block
constexpr int AX_D = 16;
// largest |score| taken without a reference value: the exponent's rounding (16 log2 e 2^-24) stays within
// that of a score of this size
constexpr float AX_BOUND = 16.f, AX_HUGE = 1e36f;
constexpr float AX_LIFT = 16777216.f, AX_VSCALE = 16777216.f;         // 2^24 both
constexpr float AX_HUGE_V = 1e26f;                                    // (sums of P V stay far inside fp32)
constexpr float AX_LOG2E = 1.4426950408889634f;

// operands in shared memory, 16-byte chunks of eight values: [d half][part][row] for Q and K (K-major), [part][d half][key]
// for V (MN-major)
constexpr int AX_Q_PLANE = 3 * AX_QT * 16, AX_K_PLANE = 3 * AX_KC * 16, AX_V_PLANE = AX_KC * 16;
constexpr int AX_K_BYTES = 2 * AX_K_PLANE, AX_V_BYTES = 6 * AX_V_PLANE;
// Tensor memory: S = q1 k1 (48 columns) | small products (48) | O = p1 v1 (16) | small products (16).  The parts of P go over
// columns whose S has been read: of 16 keys p1 and p2 over their q1 k1, p3 to AX_TM_SMALL + 8 chunk.
constexpr int AX_TM = 128, AX_TM_SMALL = AX_KC, AX_TM_O = 2 * AX_KC;
static_assert(AX_TM_O + 32 <= AX_TM && AX_KC % 16 == 0 && AX_KC <= AX_THREADS / 2, "block of keys");

// the three parts of 16 values, as 16-byte chunks
struct AxParts {
    uint4 c[3][2];
    __device__ __forceinline__ explicit AxParts(const uint64_t (&x)[8])
    {
        const uint64_t minus = pack2(-1.f, -1.f);
        uint32_t w[3][8];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const uint64_t rest = fma2(round2(x[i], w[0][i]), minus, x[i]);
            float lo, hi;
            unpack2(fma2(round2(rest, w[1][i]), minus, rest), lo, hi);
            w[2][i] = pack_bf16(lo, hi);
        }
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int h = 0; h < 2; ++h)
                c[p][h] = make_uint4(w[p][4 * h], w[p][4 * h + 1], w[p][4 * h + 2], w[p][4 * h + 3]);
    }
};
__device__ __forceinline__ float ax_norm(const uint64_t (&x)[8])
{
    uint64_t a = mul2(x[0], x[0]);
#pragma unroll
    for (int i = 1; i < 8; ++i) a = fma2(x[i], x[i], a);
    return hsum2(a);
}
__device__ __forceinline__ void ax_row(const float* src, uint64_t (&x)[8])
{
#pragma unroll
    for (int d = 0; d < 4; ++d) {
        const float4 v = reinterpret_cast<const float4*>(src)[d];
        x[2 * d] = pack2(v.x, v.y);
        x[2 * d + 1] = pack2(v.z, v.w);
    }
}

struct AxArgs {
    const float* qkv;
    const int64_t *order, *pad, *unpad;
    const int32_t* cu;
    float* out;
    __nv_bfloat16* split_out;        // the result as split rows instead
    int C, heads;
    float scale;
    uint32_t* status;
};

// plain arithmetic over a patch's keys, for one query
__device__ __noinline__ void ax_plain(const AxArgs& a, int64_t start, int L, int h, const float (&q)[AX_D], float (&y)[AX_D])
{
    float m = 0.f, l = 0.f;
    for (int j = 0; j < L; ++j) {
        const float* k = a.qkv + a.order[a.pad[start + j]] * 3 * a.C + a.C + h * AX_D;
        float s = 0.f;
#pragma unroll
        for (int d = 0; d < AX_D; ++d) s = fmaf(q[d], k[d], s);
        // (as long as every score is -inf the weights are one another's, and a later score's are 0 of it)
        const float up = j == 0 ? s : fmaxf(m, s), corr = up == -INFINITY ? 1.f : __expf(m - up),
                    p = up == -INFINITY ? 1.f : __expf(s - up);
        m = up;
        l = j == 0 ? p : fmaf(l, corr, p);
#pragma unroll
        for (int d = 0; d < AX_D; ++d) y[d] = fmaf(p, k[a.C + d], j == 0 ? 0.f : y[d] * corr);
    }
    const float inv = m == -INFINITY ? __int_as_float(0x7fffffff) : 1.f / l;
#pragma unroll
    for (int d = 0; d < AX_D; ++d) y[d] *= inv;
}

// SHORT: patches of up to 128 rows.  Warps whose queries or keys all lie behind a patch's end leave them out (us, without /
// with: 90 000 x 64 in patches of 20 178 / 166, of 28 134 / 125; the tests cost long patches 2 %).
template <bool SHORT>
__global__ void __launch_bounds__(AX_THREADS, 4) attn_f32_d16_kernel(const __grid_constant__ AxArgs a)
{
    __shared__ __align__(128) unsigned char q_s[2 * AX_Q_PLANE], k_s[2][AX_K_BYTES], v_s[2][AX_V_BYTES];
    __shared__ __align__(8) uint64_t bars[2];
    __shared__ float norm_s[2][2];               // largest squared norm of a key, of each buffer and loading warp
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_s, plain_s[2];          // plain_s: of each buffer, a value is out of range
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    volatile int* abort = &abort_s;
    const uint32_t bar_s = smem_u32_generic(bars), bar_o = bar_s + 8;
    if (tid == 0) {
        mbar_init(bar_s, 1);
        mbar_init(bar_o, 1);
        abort_s = plain_s[0] = plain_s[1] = 0;
        fence_barrier_init();
    }
    pdl_wait();
    const int seq = blockIdx.y, h = blockIdx.x % a.heads, tile = blockIdx.x / a.heads;
    const int64_t start = a.cu[seq];
    const int L = (int)(a.cu[seq + 1] - start);
    // a sequence longer than the caller's max_seqlen would leave rows of the output unwritten: reported
    if (tile == 0 && tid == 0 && a.status && L > (int)(gridDim.x / a.heads) * AX_QT) atomicOr(a.status, PTV3_STATUS_BAD_INDEX);
    if (tile * AX_QT >= L) return;
    if (warp == 0) {
        tmem_alloc(smem_u32_generic(&tmem_slot), AX_TM);
        // only now: the kernel brought up behind this one may take tensor memory and then wait for this one
        pdl_launch_next();
    }
    const int64_t stride = 3 * (int64_t)a.C;

    // thread t < 48 brings key t of a block, thread 64 + t its value (the patch's last one behind its end); `src` is the row
    // of the block after the one in `x`
    const int key = min(tid & (AX_THREADS / 2 - 1), AX_KC - 1);
    const bool is_v = warp >= AX_THREADS / 64;
    const int key_warp = warp % (AX_THREADS / 64) * 32;
    const float* kv = a.qkv + (is_v ? 2 : 1) * a.C + h * AX_D;
    uint64_t x[8];
    auto source = [&](int c0) { return a.order[a.pad[start + min(c0 + key, L - 1)]]; };
    auto fetch = [&](int64_t src) { ax_row(kv + src * stride, x); };
    // c0: first key of the block
    auto stage = [&](int buf, int c0) {
        if (SHORT && c0 + key_warp >= L) {
            if (!is_v && lane == 0) norm_s[buf][warp] = 0.f;
            return;
        }
        const float norm = ax_norm(x);
        if (!(norm < (is_v ? AX_HUGE_V : AX_HUGE))) plain_s[buf] = 1;
        if (is_v) {
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = mul2(x[i], pack2(AX_VSCALE, AX_VSCALE));
        }
        const AxParts parts(x);
        if (is_v) {
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    *reinterpret_cast<uint4*>(v_s[buf] + key * 16 + (2 * p + half) * AX_V_PLANE) = parts.c[p][half];
        } else {
#pragma unroll
            for (int p = 0; p < 3; ++p)
#pragma unroll
                for (int half = 0; half < 2; ++half)
                    *reinterpret_cast<uint4*>(k_s[buf] + key * 16 + half * AX_K_PLANE + p * AX_V_PLANE) = parts.c[p][half];
            // (squares are ordered as their bits; a NaN lies above them)
            const uint32_t most = __reduce_max_sync(0xffffffffu, __float_as_uint(norm));
            if (lane == 0) norm_s[buf][warp] = __uint_as_float(most);
        }
    };
    fetch(source(0));
    int64_t src = source(AX_KC);
    // this thread's query, and the point whose result it writes: none behind the patch's end or in a row that fills the last
    // patch, whose owner is elsewhere (points are numbered in 32 bits)
    float qnorm = 0.f;
    int mine = -1;
    const bool queries = !SHORT || warp * 32 < L;          // of this warp
    if (queries) {
        const int qi = tile * AX_QT + tid;
        uint64_t q[8];
        if (qi < L) {
            const int64_t pd = a.pad[start + qi], row = a.order[pd];
            ax_row(a.qkv + row * stride + h * AX_D, q);
            if (a.unpad[pd] == start + qi) mine = (int)row;
        } else {
#pragma unroll
            for (int i = 0; i < 8; ++i) q[i] = 0ull;
        }
        const uint64_t scale = pack2(a.scale, a.scale);
#pragma unroll
        for (int i = 0; i < 8; ++i) q[i] = mul2(q[i], scale);
        qnorm = ax_norm(q);
        // (scores in base 2 from here on)
#pragma unroll
        for (int i = 0; i < 8; ++i) q[i] = mul2(q[i], pack2(AX_LOG2E, AX_LOG2E));
        // (plain_s was cleared ahead of the barrier that follows; this write may only come after it)
        const AxParts parts(q);
#pragma unroll
        for (int p = 0; p < 3; ++p)
#pragma unroll
            for (int half = 0; half < 2; ++half)
                *reinterpret_cast<uint4*>(q_s + half * AX_Q_PLANE + (p * AX_QT + tid) * 16) = parts.c[p][half];
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (!(qnorm < AX_HUGE)) plain_s[0] = 1;
    stage(0, 0);
    fetch(src);
    src = source(2 * AX_KC);
    fence_proxy_async();
    __syncthreads();

    const uint32_t tm0 = tmem_slot, tm = tm0 + ((uint32_t)(warp * 32) << 16);
    const uint32_t q_base = smem_u32_generic(q_s), k_base = smem_u32_generic(k_s), v_base = smem_u32_generic(v_s);
    auto issue_s = [&](int buf) {
        const uint64_t dq = umma_desc_plain(q_base, AX_Q_PLANE, 128),
                       dk = umma_desc_plain(k_base + buf * AX_K_BYTES, AX_K_PLANE, 128);
        constexpr uint64_t QP = AX_QT, KP = AX_KC;            // parts lie 16 bytes x rows apart
        constexpr uint32_t one = umma_idesc_bf16(AX_QT, AX_KC), two = umma_idesc_bf16(AX_QT, 2 * AX_KC);
        umma_bf16(tm0, dq, dk, two, false);                                     // q1 k1 | q1 k2
        umma_bf16(tm0 + AX_TM_SMALL, dq, dk + 2 * KP, one, true);               // q1 k3
        umma_bf16(tm0 + AX_TM_SMALL, dq + QP, dk, one, true);                   // q2 k1
        umma_bf16(tm0 + AX_TM_SMALL, dq + QP, dk + KP, one, true);              // q2 k2
        umma_bf16(tm0 + AX_TM_SMALL, dq + 2 * QP, dk, one, true);               // q3 k1
        umma_commit(bar_s);
    };
    auto issue_o = [&](int buf, int chunks) {
        const uint64_t dv = umma_desc_plain(v_base + buf * AX_V_BYTES, 128, AX_V_PLANE);
        constexpr uint64_t VP = 2 * AX_V_PLANE >> 4;
        constexpr uint32_t one = umma_idesc_bf16(AX_QT, 16) | (1u << 16), two = umma_idesc_bf16(AX_QT, 32) | (1u << 16);
        for (int c = 0; c < chunks; ++c) {
            const uint32_t p1 = tm0 + 16 * c, p2 = p1 + 8, p3 = tm0 + AX_TM_SMALL + 8 * c, o = tm0 + AX_TM_O;
            const uint64_t v = dv + 16 * c;
            umma_bf16_ts(o, p1, v, two, c > 0);                  // p1 v1 | p1 v2
            umma_bf16_ts(o + 16, p1, v + 2 * VP, one, true);     // p1 v3
            umma_bf16_ts(o + 16, p2, v, one, true);              // p2 v1
            umma_bf16_ts(o + 16, p2, v + VP, one, true);         // p2 v2
            umma_bf16_ts(o + 16, p3, v, one, true);              // p3 v1
        }
        umma_commit(bar_o);
    };
    float acc[AX_D], l = 0.f, m = 0.f, lift = 1.f;
#pragma unroll
    for (int d = 0; d < AX_D; ++d) acc[d] = 0.f;
    bool first = true, ok = true, plain = *reinterpret_cast<volatile int*>(&plain_s[0]) != 0;
    uint32_t s_phase = 0, o_phase = 0;
    auto take_o = [&]() {
        uint32_t o0[16], o1[16];
        ok &= mbar_wait(bar_o, o_phase, abort);
        o_phase ^= 1;
        __syncwarp();
        if (!queries) return;
        fence_after_sync();
        tmem_ld16(tm + AX_TM_O, o0);
        tmem_ld16(tm + AX_TM_O + 16, o1);
        tmem_ld16_fence(o0);
        tmem_ld16_fence(o1);
#pragma unroll
        for (int d = 0; d < AX_D; ++d) acc[d] += __uint_as_float(o0[d]) + __uint_as_float(o1[d]);
    };
    if (!plain && warp == 0) {
        if (elect_one()) {
            fence_after_sync();
            issue_s(0);
        }
        __syncwarp();
    }
    const uint64_t minus = pack2(-1.f, -1.f);
    for (int c0 = 0; c0 < L && !plain; c0 += AX_KC) {
        const int buf = s_phase, nk = min(AX_KC, L - c0), chunks = (nk + 15) / 16;
        const float kn = fmaxf(norm_s[buf][0], norm_s[buf][1]);
        const bool more = c0 + AX_KC < L;
        // O of the block before; then (its V has been read) the next block into that buffer
        if (c0) take_o();
        if (more) {
            stage(buf ^ 1, c0 + AX_KC);
            fence_proxy_async();
            fetch(src);
            src = source(c0 + 3 * AX_KC);
        }
        const bool bounded = __all_sync(0xffffffffu, qnorm * kn <= AX_BOUND * AX_BOUND && lift == 1.f);
        ok &= mbar_wait(bar_s, s_phase, abort);
        s_phase ^= 1;
        __syncwarp();
        fence_after_sync();
        uint32_t x0[8], x1[8], y0[8], y1[8];
        if (!bounded && queries) {
            float cm = -INFINITY;
            for (int c = 0; c < 2 * chunks; ++c) {
                tmem_ld8(tm + 8 * c, x0);
                tmem_ld8(tm + AX_TM_SMALL + 8 * c, x1);
                tmem_ld8_fence(x0, x1);
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    if (8 * c + i < nk) cm = fmaxf(cm, __uint_as_float(x0[i]) + __uint_as_float(x1[i]));
            }
            // the first block sets the reference; after blocks without one (reference 0, not lifted) it only rises
            const float up = first ? cm : fmaxf(m, cm), corr = first ? 0.f : fast_exp2(m - up) * (lift == 1.f ? AX_LIFT : 1.f);
            lift = AX_LIFT;
            l *= corr;
#pragma unroll
            for (int d = 0; d < AX_D; ++d) acc[d] *= corr;
            m = up;
        }
        first = false;
        uint64_t sum = 0ull;
        const uint64_t ref = pack2(-m, -m);
        // eight scores of a row -> the parts of their probabilities; RAGGED: with a reference value, and `valid` keys
        auto probabilities = [&](auto ragged, const uint32_t (&s0)[8], const uint32_t (&s1)[8], int valid, uint32_t* w0,
                                 uint32_t* w1, uint32_t* w2) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint64_t s = add2(pack2u(s0[2 * i], s0[2 * i + 1]), pack2u(s1[2 * i], s1[2 * i + 1]));
                float e0, e1;
                if (ragged.value) s = add2(s, ref);
                unpack2(s, e0, e1);
                e0 = fast_exp2(e0);
                e1 = fast_exp2(e1);
                if (ragged.value) {
                    e0 = 2 * i < valid ? e0 : 0.f;
                    e1 = 2 * i + 1 < valid ? e1 : 0.f;
                }
                uint64_t p = pack2(e0, e1);
                if (ragged.value) p = mul2(p, pack2(lift, lift));
                sum = add2(sum, p);
                const uint64_t rest = fma2(round2(p, w0[i]), minus, p);
                unpack2(fma2(round2(rest, w1[i]), minus, rest), e0, e1);
                w2[i] = pack_bf16(e0, e1);
            }
        };
        // 16 keys at a time, the next eight scores on their way
        auto rows = [&](auto ragged, int chunks) {
            tmem_ld8(tm, x0);
            tmem_ld8(tm + AX_TM_SMALL, x1);
#pragma unroll(ragged.value ? 1 : AX_KC / 16)
            for (int c = 0; c < chunks; ++c) {
                uint32_t w0[4], w1[8], w2[4];
                const uint32_t at = tm + 16 * c;
                tmem_ld8_fence(x0, x1);
                tmem_ld8(at + 8, y0);
                tmem_ld8(at + AX_TM_SMALL + 8, y1);
                probabilities(ragged, x0, x1, nk - 16 * c, w0, w1, w2);
                tmem_st4(at, w0);
                tmem_st4(tm + AX_TM_SMALL + 8 * c, w2);
                tmem_ld8_fence(y0, y1);
                if (c + 1 < chunks) {
                    tmem_ld8(at + 16, x0);
                    tmem_ld8(at + AX_TM_SMALL + 16, x1);
                }
                probabilities(ragged, y0, y1, nk - 16 * c - 8, w0, w1 + 4, w2);
                tmem_st4(at + 4, w0);
                tmem_st8(at + 8, w1);
                tmem_st4(tm + AX_TM_SMALL + 8 * c + 4, w2);
            }
        };
        if (queries) {
            if (bounded && nk == AX_KC)
                rows(std::false_type(), AX_KC / 16);
            else
                rows(std::true_type(), chunks);
        }
        l += hsum2(sum);
        tmem_st_wait();
        fence_before_sync();
        __syncthreads();
        // (a value out of range in the block ahead: this one's products are still issued and waited for)
        plain = *reinterpret_cast<volatile int*>(&plain_s[buf ^ 1]) != 0;
        if (*abort) break;
        if (warp == 0) {
            if (elect_one()) {
                fence_after_sync();
                // (S of the next block overwrites P, which O is made from: products run in the order of issue, see umma_bf16)
                issue_o(buf, chunks);
                if (more && !plain) issue_s(buf ^ 1);
            }
            __syncwarp();
        }
        if (!more || plain) take_o();
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        if (*abort) {
            // products that were waited for in vain: once more, with a limit, before the memory under them goes
            int give_up = 0;
            mbar_wait(bar_s, s_phase ^ 1, &give_up);
            give_up = 0;
            mbar_wait(bar_o, o_phase, &give_up);
        }
        fence_after_sync();
        tmem_dealloc(tm0, AX_TM);
    }
    if (lane == 0 && !ok && a.status) atomicOr(a.status, PTV3_STATUS_WAIT_LIMIT);

    if (mine < 0) return;
    if (plain) {
        float q[AX_D];
#pragma unroll
        for (int d = 0; d < AX_D; ++d) q[d] = a.qkv[mine * stride + h * AX_D + d] * a.scale;
        ax_plain(a, start, L, h, q, acc);
    } else {
        const float inv = 1.f / (l * AX_VSCALE);
#pragma unroll
        for (int d = 0; d < AX_D; ++d) acc[d] *= inv;
    }
    if (a.split_out) {
#pragma unroll
        for (int d = 0; d < AX_D; d += 8)
            split_store8(a.split_out + (int64_t)mine * split_stored(a.C) * a.C, h * AX_D + d, a.C, acc + d);
        return;
    }
    float4* op = reinterpret_cast<float4*>(a.out + (int64_t)mine * a.C + h * AX_D);
#pragma unroll
    for (int d = 0; d < 4; ++d) op[d] = make_float4(acc[4 * d], acc[4 * d + 1], acc[4 * d + 2], acc[4 * d + 3]);
}

int launch_attn_f32(const void* qkv, const int64_t* order, const int64_t* pad, const int64_t* unpad, const int32_t* cu,
                    void* out, bool split, int n_seq, int max_seqlen, int C, int H, float scale, uint32_t* status,
                    cudaStream_t stream)
{
    const int tiles = (max_seqlen + AX_QT - 1) / AX_QT;
    launch_dependent(max_seqlen <= AX_QT ? attn_f32_d16_kernel<true> : attn_f32_d16_kernel<false>,
                     dim3(H * tiles, n_seq), dim3(AX_THREADS), 0, stream,
                     AxArgs{(const float*)qkv, order, pad, unpad, cu, split ? nullptr : (float*)out,
                            split ? (__nv_bfloat16*)out : nullptr, C, H, scale, status});
    count_launches(1);
    return check_launch("ptv3_attention_fwd");
}

}  // namespace ptv3
