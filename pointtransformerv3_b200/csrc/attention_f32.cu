// fp32 patch attention (model.py:452-484), head dimension 16: the fp32 backbone's attention core.
//
// The first form of this path (attention.cu, which keeps the other head dimensions, the position bias and
// the bf16 cross-check) gave a thread one query: every key cost eight 16-byte shared-memory reads for 32
// multiply-adds, and the scores were computed twice (maximum first, probabilities second).  Here a thread
// owns two or four queries, so a read serves as much more arithmetic, products run on pairs of floats, and the scores
// are computed once: where |q| max|k| bounds them (AX_BOUND, per chunk of keys and CTA) the exponentials
// need no reference value; other chunks take the maximum first as before.
//
// The four warps of a CTA share its 64 or 128 queries and take the keys in turn; their sums meet at the end.
// With the queries spread over all threads instead, a patch of a coarse level was a serial chain of up to
// 1 024 keys on a few CTAs (100 us at 700 points x 256 channels as at 40 000 x 64).
#include "attention_mma.cuh"
#include "common.cuh"
#include "mma_util.cuh"

namespace ptv3 {

constexpr int AX_THREADS = 128, AX_WARPS = AX_THREADS / 32;
constexpr int AX_KC = 128;                   // keys per staged chunk
constexpr int AX_D = 16, AX_P = AX_D / 2;
// largest |score| taken without a reference value: the exponent's rounding (16 log2 e 2^-24) stays within
// that of a score of this size
constexpr float AX_BOUND = 16.f;
constexpr float AX_LOG2E = 1.4426950408889634f;

struct AxRow {
    uint64_t q[AX_P], acc[AX_P];
    float m, l, norm;
};

__device__ __forceinline__ float ax_dot(const uint64_t (&q)[AX_P], const ulonglong2* k)
{
    const ulonglong2 k0 = k[0], k1 = k[1], k2 = k[2], k3 = k[3];
    uint64_t a = mul2(q[0], k0.x), b = mul2(q[1], k0.y);
    a = fma2(q[2], k1.x, a);
    b = fma2(q[3], k1.y, b);
    a = fma2(q[4], k2.x, a);
    b = fma2(q[5], k2.y, b);
    a = fma2(q[6], k3.x, a);
    b = fma2(q[7], k3.y, b);
    return hsum2(add2(a, b));
}
__device__ __forceinline__ void ax_add(AxRow& r, float p, const ulonglong2* v)
{
    const uint64_t pp = pack2(p, p);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const ulonglong2 w = v[i];
        r.acc[2 * i] = fma2(pp, w.x, r.acc[2 * i]);
        r.acc[2 * i + 1] = fma2(pp, w.y, r.acc[2 * i + 1]);
    }
    r.l += p;
}

// AX_Q queries per thread (2 or 4): AX_QT of a CTA
template <int AX_Q>
__global__ void __launch_bounds__(AX_THREADS, AX_Q == 2 ? 4 : 3) attn_f32_d16_kernel(
    const float* __restrict__ qkv, const int64_t* __restrict__ order, const int64_t* __restrict__ pad,
    const int64_t* __restrict__ unpad, const int32_t* __restrict__ cu_seqlens, float* __restrict__ out, int C,
    float scale, uint32_t* __restrict__ status)
{
    constexpr int AX_QT = 32 * AX_Q;
    // keys and values of a chunk; in the end, in their place, the warps' sums
    struct Chunk {
        float k[AX_KC][AX_D], v[AX_KC][AX_D];
    };
    typedef float Sums[AX_WARPS][AX_QT][AX_D + 3];         // sums, l, m; padded against bank conflicts
    __shared__ __align__(16) unsigned char shared[sizeof(Chunk) > sizeof(Sums) ? sizeof(Chunk) : sizeof(Sums)];
    float(&Ks)[AX_KC][AX_D] = reinterpret_cast<Chunk*>(shared)->k;
    float(&Vs)[AX_KC][AX_D] = reinterpret_cast<Chunk*>(shared)->v;
    Sums& part = *reinterpret_cast<Sums*>(shared);
    __shared__ float warp_norm[AX_WARPS];
    const int n_heads = C / AX_D;
    const int seq = blockIdx.y, h = blockIdx.x % n_heads, tile = blockIdx.x / n_heads, tid = threadIdx.x, warp = tid >> 5,
              lane = tid & 31;
    const int64_t start = cu_seqlens[seq];
    const int L = (int)(cu_seqlens[seq + 1] - start);
    // a sequence longer than the caller's max_seqlen would leave rows of the output unwritten: reported
    if (tile == 0 && tid == 0 && status && L > (int)(gridDim.x / n_heads) * AX_QT) atomicOr(status, PTV3_STATUS_BAD_INDEX);
    if (tile * AX_QT >= L) return;
    const int64_t stride = 3 * (int64_t)C;

    AxRow row[AX_Q];
#pragma unroll
    for (int i = 0; i < AX_Q; ++i) {
        const int qi = tile * AX_QT + i * 32 + lane;
        AxRow& r = row[i];
        r.m = 0.f;
        r.l = r.norm = 0.f;
#pragma unroll
        for (int d = 0; d < AX_P; ++d) r.q[d] = r.acc[d] = 0ull;
        if (qi < L) {
            const float4* qp = reinterpret_cast<const float4*>(qkv + order[pad[start + qi]] * stride + h * AX_D);
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                float4 v = qp[d];
                v.x *= scale; v.y *= scale; v.z *= scale; v.w *= scale;
                r.norm += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
                r.q[2 * d] = pack2(v.x, v.y);
                r.q[2 * d + 1] = pack2(v.z, v.w);
            }
        }
    }
    bool first = true;       // no key taken by this warp yet
    for (int c0 = 0; c0 < L; c0 += AX_KC) {
        const int nk = min(AX_KC, L - c0);
        __syncthreads();
        // a thread stages one key: its row, and the row's squared norm
        float kn = 0.f;
        if (tid < nk) {
            const float4* kp = reinterpret_cast<const float4*>(qkv + order[pad[start + c0 + tid]] * stride + C + h * AX_D);
            const float4* vp = kp + C / 4;
#pragma unroll
            for (int d = 0; d < 4; ++d) {
                const float4 k = kp[d], v = vp[d];
                kn += k.x * k.x + k.y * k.y + k.z * k.z + k.w * k.w;
                *reinterpret_cast<float4*>(&Ks[tid][4 * d]) = k;
                *reinterpret_cast<float4*>(&Vs[tid][4 * d]) = v;
            }
        }
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) kn = max_nan(kn, __shfl_xor_sync(0xffffffffu, kn, d));
        if (lane == 0) warp_norm[warp] = kn;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < AX_WARPS; ++w) kn = max_nan(kn, warp_norm[w]);
        // (a NaN fails the test); a reference value raised by an earlier chunk stays in force
        bool bounded = true;
#pragma unroll
        for (int i = 0; i < AX_Q; ++i) bounded = bounded && row[i].norm * kn <= AX_BOUND * AX_BOUND && row[i].m == 0.f;
        if (__syncthreads_and(bounded)) {
#pragma unroll(AX_Q == 2 ? 4 : 2)
            for (int j = warp; j < nk; j += AX_WARPS) {
                const ulonglong2* k = reinterpret_cast<const ulonglong2*>(Ks[j]);
                const ulonglong2* v = reinterpret_cast<const ulonglong2*>(Vs[j]);
                float p[AX_Q];
#pragma unroll
                for (int i = 0; i < AX_Q; ++i) p[i] = fast_exp2(ax_dot(row[i].q, k) * AX_LOG2E);
#pragma unroll
                for (int i = 0; i < AX_Q; ++i) ax_add(row[i], p[i], v);
            }
        } else if (warp < nk) {
#pragma unroll
            for (int i = 0; i < AX_Q; ++i) {
                AxRow& r = row[i];
                float cm = -INFINITY;
                for (int j = warp; j < nk; j += AX_WARPS)
                    cm = fmaxf(cm, ax_dot(r.q, reinterpret_cast<const ulonglong2*>(Ks[j])));
                // the first chunk sets the reference; after chunks without one (reference 0) it only rises
                const float mn = first ? cm : fmaxf(r.m, cm);
                const float corr = first ? 0.f : __expf(r.m - mn);
                r.l *= corr;
#pragma unroll
                for (int d = 0; d < AX_P; ++d) r.acc[d] = mul2(r.acc[d], pack2(corr, corr));
                r.m = mn;
                for (int j = warp; j < nk; j += AX_WARPS)
                    ax_add(r, __expf(ax_dot(r.q, reinterpret_cast<const ulonglong2*>(Ks[j])) - mn),
                           reinterpret_cast<const ulonglong2*>(Vs[j]));
            }
        }
        first = first && warp >= nk;
    }
    // ---- the warps' sums meet; the first warps finish one query of a lane each ----------
    __syncthreads();
#pragma unroll
    for (int i = 0; i < AX_Q; ++i) {
        const int qi = i * 32 + lane;
#pragma unroll
        for (int d = 0; d < AX_P; ++d) {
            float lo, hi;
            unpack2(row[i].acc[d], lo, hi);
            part[warp][qi][2 * d] = lo;
            part[warp][qi][2 * d + 1] = hi;
        }
        part[warp][qi][AX_D] = row[i].l;
        part[warp][qi][AX_D + 1] = row[i].m;
    }
    __syncthreads();
    const int qi = warp * 32 + lane, at = tile * AX_QT + qi;
    if (warp >= AX_Q || at >= L) return;
    const int64_t pd = pad[start + at];
    if (unpad[pd] != start + at) return;       // a row that fills the last patch: its owner is elsewhere
    const int64_t mine = order[pd];
    float m = -INFINITY;
    for (int w = 0; w < AX_WARPS; ++w)
        if (part[w][qi][AX_D] != 0.f) m = fmaxf(m, part[w][qi][AX_D + 1]);      // (a NaN sum stays in)
    float y[AX_D], l = 0.f;
#pragma unroll
    for (int d = 0; d < AX_D; ++d) y[d] = 0.f;
    for (int w = 0; w < AX_WARPS; ++w) {
        if (part[w][qi][AX_D] == 0.f) continue;
        const float c = __expf(part[w][qi][AX_D + 1] - m);
        l = fmaf(c, part[w][qi][AX_D], l);
#pragma unroll
        for (int d = 0; d < AX_D; ++d) y[d] = fmaf(c, part[w][qi][d], y[d]);
    }
    const float inv = 1.f / l;
    float4* op = reinterpret_cast<float4*>(out + mine * C + h * AX_D);
#pragma unroll
    for (int d = 0; d < 4; ++d)
        op[d] = make_float4(y[4 * d] * inv, y[4 * d + 1] * inv, y[4 * d + 2] * inv, y[4 * d + 3] * inv);
}

template <int Q>
static int launch_attn_f32_as(const float* qkv, const int64_t* order, const int64_t* pad, const int64_t* unpad,
                              const int32_t* cu, float* out, int n_seq, int tiles, int C, int H, float scale,
                              uint32_t* status, cudaStream_t stream)
{
    attn_f32_d16_kernel<Q><<<dim3(H * tiles, n_seq), AX_THREADS, 0, stream>>>(qkv, order, pad, unpad, cu, out, C, scale,
                                                                            status);
    count_launches(1);
    return check_launch("ptv3_attention_fwd");
}

int launch_attn_f32(const void* qkv, const int64_t* order, const int64_t* pad, const int64_t* unpad, const int32_t* cu,
                    void* out, int n_seq, int max_seqlen, int C, int H, float scale, uint32_t* status,
                    cudaStream_t stream)
{
    // Four queries per thread read shared memory half as often and keep the FMA pipe busier, in half as many CTAs: from
    // two of them to an SM.  us, two / four: 90 000 x 64 791 / 672, 40 000 x 64 374 / 315, 20 000 x 64 (640 CTAs of four) 196 / 183,
    // 10 500 x 64 (352) 114.6 / 111.9, 5 000 x 64 (160) 72.1 / 82.5, 820 x 256 24.8 / 28.9; patches of 1 024.
    const int64_t ctas = (int64_t)H * n_seq * ((max_seqlen + 127) / 128);
    const bool four = ctas > SMS * 2;
    return (four ? launch_attn_f32_as<4> : launch_attn_f32_as<2>)((const float*)qkv, order, pad, unpad, cu, (float*)out, n_seq,
                                                                  (max_seqlen + (four ? 127 : 63)) / (four ? 128 : 64), C, H,
                                                                  scale, status, stream);
}

}  // namespace ptv3
