// Patch attention core on the 5th-generation tensor cores (tcgen05 + tensor memory) for bf16 features, head
// dimension 16 and patches of up to 1024 rows (model.py:452-484; see attention.cu for the contract).
//
// At head dimension 16 a score costs 64 tensor FLOPs and one exponential.  tcgen05 takes both products off the CUDA
// cores, whose issue slots are then free to evaluate a share of the exponentials on the FMA pipe beside the
// exponential unit (AT_POLY of 16).
//
// One persistent CTA per SM owns a contiguous range of query tiles (128 rows of a (patch, head) pair).
//   three softmax groups of 128 threads (thread = query row = tensor-memory lane); group g takes tiles g, g + 3, ...
//   one issuing warp per group; per block of 128 keys S[128 x 128] = Q K^T, and O|l[128 x 32] += P V' (A from tensor
//     memory) once the group has written P over the first half of S, with the next S right behind it
//   four loading warps: K and V of a pair through order[pad[.]] into one of two slots, Q tiles into two slots per
//     group, both ahead of their use.
// All of them talk through mbarriers only.  V' has a column of ones beside V, so that P V' also yields the row sums of
// the rounded probabilities.  Keys behind a patch's end have zero K, V and ones: their probabilities (1) add nothing.
//
// Softmax needs no reference value where no score can leave the range of exp2: |q . k| <= |q| max|k| (AT_BOUND, checked by
// the loading warps).  A tile with a row that fails the test takes its scores twice, first for the row maxima.
//
// Tensor memory per group: S (128 columns, P over the first 64) | O|l (32) = 160 columns.
// Every mbarrier wait is bounded; a wait that runs out sets PTV3_STATUS_WAIT_LIMIT.
//
// Measured (C = 64, 4 heads, patches of 1 024; us here and by the mma.sync kernel, attention_mma.cu): 100 000 points
// 103 / 121, 400 000 363 / 447, 912 000 807 / 991: 86, 97 and 99 % of the exponential unit's rate at 1 965 MHz.  128 x 128
// scores take an SM 1 035 cycles at 400 000 points (mma.sync 1 280; without a CTA's first ~7 us in both): the exponential unit
// needs 640 of them for its ten of sixteen; a loop of the same reads, arithmetic (degree 4) and stores without any hand-over
// runs at 784.  What is left is a block's way through the roles (softmax -> issuing warp -> product -> softmax, ~900 cycles),
// which the two other groups cover only in part.  Forms tried (these times with a polynomial of degree 4, 2 % less):
//   * Blocks of 128 keys and one buffer, not 64 and two (505 us where this takes 406, 444 patches of 4 heads): a
//     hand-over costs ~170 cycles in the issuing warp's wait and ~160 in issuing, whatever the block's size, and
//     an issuing warp that keeps three groups waiting bounded the earlier forms of this kernel, not the products
//     (16 cycles each for P V', 64 for S).
//   * 16 columns per read of tensor memory, two reads in flight: 32 columns take registers that spill (437 us for 406).
//   * Two groups with larger blocks (511) or four with blocks of 96 keys (418) are slower; so is handing a block over
//     in halves (408 to 420), probabilities in registers with P V on mma.sync (583), and a patch's rows looked up
//     ahead by the loading warps (their instructions count: 100 000 points 105 us).
//   * AT_POLY 5, 6, 7: 366, 363, 371 us at 400 000 points; 0 (all on the exponential unit) takes a quarter more.
//   * 80 registers a thread, so that kernels of the planning stream fit beside a CTA: 377 us for 361 at 400 000
//     points, and no pass gained (16 LiDAR frames 42.0 ms, with 96 registers 41.3).
#include "common.cuh"
#include "attention_mma.cuh"
#include "exp2_poly.cuh"
#include "mma_util.cuh"
#include "tc05.cuh"

namespace ptv3 {

using namespace tc05;

constexpr int AT_GROUPS = 3;
constexpr int AT_LOAD_WARP = AT_GROUPS;           // first loading warp, behind the issuing ones; the others come last
constexpr int AT_SOFT_WARP = 4;                   // first softmax warp (a multiple of 4: a quarter of the lanes each)
constexpr int AT_REST_WARP = AT_SOFT_WARP + 4 * AT_GROUPS;
constexpr int AT_THREADS = 32 * (AT_REST_WARP + 3);
static_assert(AT_LOAD_WARP + 1 == AT_SOFT_WARP, "roles of the warps");
constexpr int AT_BM = 128;                        // query rows of a tile
constexpr int AT_BK = 128;                        // keys of a block
constexpr int AT_D = 16;
constexpr int AT_MAX_TILES = ATTN_TC05_MAX_SEQLEN / AT_BM;
constexpr int AT_POLY = 6;                        // of 16 pairs of exponentials, this many on the FMA pipe
constexpr float AT_LOG2E = 1.4426950408889634f;
constexpr float AT_BOUND = 80.f;                  // largest |score| (exp2 domain) taken without a reference value
constexpr int AT_Q_BYTES = AT_BM * AT_D * 2;
constexpr int AT_TM_GROUP = AT_BK + 32, AT_TM_O = AT_BK;
static_assert(AT_TM_GROUP * AT_GROUPS <= 512, "tensor memory");

// mbarriers of a group, and of the CTA behind those of the groups
constexpr int AT_B_QFULL = 0, AT_B_QFREE = 2, AT_B_S = 4, AT_B_P = 5, AT_B_O = 6, AT_B_DONE = 7, AT_B_GROUP = 8;
constexpr int AT_B_V = AT_B_GROUP * AT_GROUPS, AT_B_KVFREE = AT_B_V + 2, AT_NBAR = AT_B_V + 4;

// shared-memory map for patches padded to lpad (a multiple of 128) keys
struct AtLayout {
    int plane, slot, off_q, off_src, off_qrow, off_flag, off_kn, off_bar, total;
    __host__ __device__ explicit AtLayout(int lpad)
    {
        plane = lpad * 16;                          // a 16-byte chunk of every key
        slot = 5 * plane;                           // V d 0-7, V d 8-15, ones, K d 0-7, K d 8-15
        off_q = 2 * slot;
        off_src = off_q + AT_GROUPS * 2 * AT_Q_BYTES;
        off_qrow = off_src + lpad * 4;
        off_flag = off_qrow + AT_GROUPS * 2 * AT_BM * 4;
        off_kn = off_flag + AT_GROUPS * 2 * 16;
        off_bar = off_kn + 2 * 16;
        total = off_bar + 8 * AT_NBAR + 16;
    }
};

__device__ __forceinline__ uint32_t at_scale_bf16x2(uint32_t v, float s)
{
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&v));
    return pack_bf16(f.x * s, f.y * s);
}

// exp2(s log2e) of a pair on the FMA pipe, |s log2e| <= AT_BOUND: n = round(s log2e) by adding 1.5 * 2^23, 2^r on
// [-0.5, 0.5] by a polynomial as close as the exponential unit (exp2_poly.cuh; one of degree 4, with 2.7e-6 for its 2.1e-7,
// is 2 % faster: 400 000 points 355 us for 363), n added to the exponent field.
struct AtPoly {
    uint64_t log2e, magic, neg_one, c5, c4, c3, c2, c1, c0;
    __device__ __forceinline__ AtPoly()
    {
        log2e = pack2(AT_LOG2E, AT_LOG2E);
        magic = pack2(12582912.f, 12582912.f);
        neg_one = pack2(-1.f, -1.f);
        c5 = pack2(EXP2_C5, EXP2_C5);
        c4 = pack2(EXP2_C4, EXP2_C4);
        c3 = pack2(EXP2_C3, EXP2_C3);
        c2 = pack2(EXP2_C2, EXP2_C2);
        c1 = pack2(EXP2_C1, EXP2_C1);
        c0 = pack2(EXP2_C0, EXP2_C0);
    }
};
__device__ __forceinline__ uint32_t at_exp2_poly(uint64_t s2, const AtPoly& k)
{
    const uint64_t t2 = fma2(s2, k.log2e, k.magic);
    const uint64_t r2 = fma2(s2, k.log2e, fma2(t2, k.neg_one, k.magic));
    uint64_t p2 = fma2(r2, k.c5, k.c4);
    p2 = fma2(p2, r2, k.c3);
    p2 = fma2(p2, r2, k.c2);
    p2 = fma2(p2, r2, k.c1);
    p2 = fma2(p2, r2, k.c0);
    float px, py, tx, ty;
    unpack2(p2, px, py);
    unpack2(t2, tx, ty);
    px = __int_as_float(__float_as_int(px) + (__float_as_int(tx) << 23));
    py = __int_as_float(__float_as_int(py) + (__float_as_int(ty) << 23));
    return pack_bf16(px, py);
}

// 16 scores of a row -> 8 packed probabilities; CH: number of the chunk in its block
template <int CH>
__device__ __forceinline__ void at_probabilities(const uint32_t (&s)[16], uint32_t (&pk)[8], const AtPoly& k)
{
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint64_t s2 = pack2u(s[2 * i], s[2 * i + 1]);
        if (((8 * (CH & 1) + i) * AT_POLY) % 16 < AT_POLY) {          // AT_POLY of 16, spread evenly
            pk[i] = at_exp2_poly(s2, k);
        } else {
            float x, y;
            unpack2(mul2(s2, k.log2e), x, y);
            pk[i] = pack_bf16(fast_exp2(x), fast_exp2(y));
        }
    }
}
// chunk CH of a block of NCH: x holds it (in flight), y takes the next one
template <int CH, int NCH>
__device__ __forceinline__ void at_chunks(uint32_t (&x)[16], uint32_t (&y)[16], uint32_t tm_s, const AtPoly& k)
{
    uint32_t pk[8];
    tmem_ld16_fence(x);
    if (CH + 1 < NCH) tmem_ld16(tm_s + 16 * (CH + 1), y);
    at_probabilities<CH>(x, pk, k);
    tmem_st8(tm_s + 8 * CH, pk);
    if constexpr (CH + 1 < NCH) at_chunks<CH + 1, NCH>(y, x, tm_s, k);
}
// the same with a reference value (mb = -m log2e) and `valid` real keys
__device__ __forceinline__ void at_probabilities_ref(const uint32_t (&s)[16], uint32_t (&pk)[8], float mb, int valid)
{
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const float x = fast_exp2(fmaf(__uint_as_float(s[2 * i]), AT_LOG2E, mb));
        const float y = fast_exp2(fmaf(__uint_as_float(s[2 * i + 1]), AT_LOG2E, mb));
        pk[i] = pack_bf16(2 * i < valid ? x : 0.f, 2 * i + 1 < valid ? y : 0.f);
    }
}

struct AtArgs {
    const __nv_bfloat16* qkv;
    const int64_t *order, *pad, *unpad;
    const int32_t* cu;
    __nv_bfloat16* out;
    int n_seq, heads, tiles, lpad;
    float scale;
    bool planned;                 // the geometry may be read before the wait for the kernel ahead (see linear.cuh)
    uint32_t* status;
};

// The CTA's tiles, pair after pair.  Every role walks them by itself, in the same order.
struct AtWalk {
    const AtArgs* a;
    int w0, w1, pair, last, seq, head, start, L, lo, hi, counted, before;
    __device__ __forceinline__ explicit AtWalk(const AtArgs& args) : a(&args)
    {
        const int64_t total = (int64_t)a->n_seq * a->heads * a->tiles;
        w0 = (int)(total * blockIdx.x / gridDim.x);
        w1 = (int)(total * (blockIdx.x + 1) / gridDim.x);
        pair = w0 / a->tiles - 1;
        last = w1 > w0 ? (w1 - 1) / a->tiles : pair;
        counted = -1;
        before = lo = hi = 0;
    }
    // next pair with tiles of this CTA: `counted` is its number, `before` the tiles of those ahead of it
    __device__ __forceinline__ bool next(bool report = false)
    {
        before += hi - lo;
        lo = hi = 0;
        while (++pair <= last) {
            seq = pair / a->heads;
            head = pair - seq * a->heads;
            start = __shfl_sync(0xffffffffu, a->cu[seq], 0);
            L = __shfl_sync(0xffffffffu, a->cu[seq + 1], 0) - start;
            // a patch that the caller's max_seqlen does not cover is reported and skipped
            if (L > a->lpad) {
                if (report) atomicOr(a->status, PTV3_STATUS_BAD_INDEX);
                continue;
            }
            lo = max(w0 - pair * a->tiles, 0);
            hi = min(w1 - pair * a->tiles, L <= 0 ? 0 : (L + AT_BM - 1) / AT_BM);
            if (hi > lo) {
                ++counted;
                return true;
            }
            lo = hi = 0;
        }
        return false;
    }
    // first tile of the pair that is group g's (tile number `before + i - lo` goes to group number % 3)
    __device__ __forceinline__ int first(int g) const
    {
        return lo + (g + AT_GROUPS - before % AT_GROUPS) % AT_GROUPS;
    }
    __device__ __forceinline__ int blocks() const { return (L + AT_BK - 1) / AT_BK; }
    // 16-key steps of the last block
    __device__ __forceinline__ int tail() const { return ((L - 1) % AT_BK + 16) / 16; }
};

__global__ void __launch_bounds__(AT_THREADS, 1) attn_tc05_d16_kernel(const AtArgs a)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
    const AtLayout lay(a.lpad);
    const uint32_t sbase = smem_u32_generic(smem);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int C = a.heads * AT_D;
    const int64_t row_stride = 3 * (int64_t)C;

    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + lay.off_bar);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + AT_NBAR);
    volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t bar0 = sbase + lay.off_bar;
    const uint32_t vbar = bar0 + 8 * AT_B_V, kvfree = bar0 + 8 * AT_B_KVFREE;
    int32_t* qrow = reinterpret_cast<int32_t*>(smem + lay.off_qrow);      // [group][slot][128]
    uint32_t* qflag = reinterpret_cast<uint32_t*>(smem + lay.off_flag);   // [group][slot][4]
    float* kn_s = reinterpret_cast<float*>(smem + lay.off_kn);            // [slot][4]

    if (tid == 0) {
        for (int g = 0; g < AT_GROUPS; ++g) {
            const uint32_t b = bar0 + 8 * AT_B_GROUP * g;
            for (int s = 0; s < 2; ++s) {
                mbar_init(b + 8 * (AT_B_QFULL + s), 4);       // a loading warp each
                mbar_init(b + 8 * (AT_B_QFREE + s), 4);       // a softmax warp each
            }
            mbar_init(b + 8 * AT_B_S, 1);
            mbar_init(b + 8 * AT_B_P, 4);
            mbar_init(b + 8 * AT_B_O, 1);
            mbar_init(b + 8 * AT_B_DONE, 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(vbar + 8 * s, 4);
            mbar_init(kvfree + 8 * s, 4 * AT_GROUPS);
        }
        *abort = 0;
        fence_barrier_init();
    }
    if (warp == AT_LOAD_WARP) {
        tmem_alloc(sbase + lay.off_bar + 8 * AT_NBAR, 512);
        // only now: the kernel brought up behind this one may take tensor memory and then wait for this one
        pdl_launch_next();
    }
    if (!a.planned) pdl_wait();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    if (warp == AT_LOAD_WARP || warp >= AT_REST_WARP) {
        // ---- loading warps: thread t owns rows t, t + 128, ... of every pair ------------------------------------
        const int lw = warp == AT_LOAD_WARP ? 0 : warp - AT_REST_WARP + 1, t = 32 * lw + lane;
        int32_t* src_s = reinterpret_cast<int32_t*>(smem + lay.off_src);
        int ones0 = -1, ones1 = -1;          // rows of the slots' planes of ones
        int seq = -1;
        bool waited = false;
        AtWalk w(a);
        while (w.next(t == 0)) {
            const int slot = w.counted & 1, L = w.L, Lk = (L + 15) / 16 * 16;
            if (w.seq != seq) {
                // point row of every padded row, negated - 1 where the padded row does not own its point
                // (borrowed rows); read back by this thread alone
                seq = w.seq;
                for (int r = t; r < L; r += 4 * AT_BM) {
                    int64_t pd[4], src[4], own[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) pd[i] = r + i * AT_BM < L ? a.pad[w.start + r + i * AT_BM] : -1;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        src[i] = pd[i] >= 0 ? a.order[pd[i]] : 0;
                        own[i] = pd[i] >= 0 ? a.unpad[pd[i]] : 0;
                    }
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (pd[i] >= 0)
                            src_s[r + i * AT_BM] = own[i] == w.start + r + i * AT_BM ? (int32_t)src[i] : -(int32_t)src[i] - 1;
                }
            }
            // (planned: so far only the geometry was read)
            if (!waited) pdl_wait();
            waited = true;
            if (w.counted >= 2) mbar_wait(kvfree + 8 * slot, ((w.counted >> 1) - 1) & 1, abort);

            unsigned char* vs = smem + slot * lay.slot;
            unsigned char* ks = vs + 3 * lay.plane;
            const uint32_t vs_a = sbase + slot * lay.slot, ks_a = vs_a + 3 * lay.plane;
            auto row_of = [&](int r) {
                const int32_t e = src_s[r];
                return (int64_t)(e >= 0 ? e : -(e + 1)) * row_stride + w.head * AT_D;
            };
            const uint4 zero = make_uint4(0, 0, 0, 0);
#pragma unroll
            for (int i = 0; i < AT_MAX_TILES; ++i) {
                const int r = i * AT_BM + t;
                if (i * AT_BM >= Lk) break;
                if (r < L) {
                    const __nv_bfloat16* kp = a.qkv + row_of(r) + C;
                    cp_async16(ks_a + r * 16, kp);
                    cp_async16(ks_a + lay.plane + r * 16, kp + 8);
                } else if (r < Lk) {
                    *reinterpret_cast<uint4*>(ks + r * 16) = zero;
                    *reinterpret_cast<uint4*>(ks + lay.plane + r * 16) = zero;
                }
            }
            cp_async_commit();
            // query row of the pair's first tile
            uint4 q0 = zero, q1 = zero;
            auto fetch_q = [&](int tile) {
                const int r = tile * AT_BM + t;
                q0 = q1 = zero;
                if (tile < w.hi && r < L) {
                    const uint4* qp = reinterpret_cast<const uint4*>(a.qkv + row_of(r));
                    q0 = qp[0];
                    q1 = qp[1];
                }
            };
            fetch_q(w.lo);
#pragma unroll
            for (int i = 0; i < AT_MAX_TILES; ++i) {
                const int r = i * AT_BM + t;
                if (i * AT_BM >= Lk) break;
                if (r < L) {
                    const __nv_bfloat16* vp = a.qkv + row_of(r) + 2 * C;
                    cp_async16(vs_a + r * 16, vp);
                    cp_async16(vs_a + lay.plane + r * 16, vp + 8);
                } else if (r < Lk) {
                    *reinterpret_cast<uint4*>(vs + r * 16) = zero;
                    *reinterpret_cast<uint4*>(vs + lay.plane + r * 16) = zero;
                }
            }
            cp_async_commit();
            if ((slot ? ones1 : ones0) != L) {
                (slot ? ones1 : ones0) = L;
                for (int r = t; r < Lk; r += AT_BM)
                    *reinterpret_cast<uint4*>(vs + 2 * lay.plane + r * 16) = make_uint4(r < L ? 0x3f80u : 0u, 0, 0, 0);
            }
            // largest squared norm of a key (every thread reads back the rows it copied itself)
            cp_async_wait<1>();
            float kn = 0.f;
            for (int r = t; r < L; r += AT_BM)
                kn = max_nan(kn, sq_norm16(*reinterpret_cast<const uint4*>(ks + r * 16),
                                           *reinterpret_cast<const uint4*>(ks + lay.plane + r * 16)));
#pragma unroll
            for (int d = 16; d > 0; d >>= 1) kn = max_nan(kn, __shfl_xor_sync(0xffffffffu, kn, d));
            if (lane == 0) kn_s[slot * 4 + lw] = kn;
            named_barrier(1, 128);
#pragma unroll
            for (int i = 0; i < 4; ++i) kn = max_nan(kn, kn_s[slot * 4 + i]);

            const float lim = (AT_BOUND / AT_LOG2E) * (AT_BOUND / AT_LOG2E);
            for (int tile = w.lo; tile < w.hi; ++tile) {
                const int number = w.before + tile - w.lo, g = number % AT_GROUPS, k = number / AT_GROUPS, qs = k & 1;
                const uint32_t gbar = bar0 + 8 * AT_B_GROUP * g;
                if (k >= 2) mbar_wait(gbar + 8 * (AT_B_QFREE + qs), ((k >> 1) - 1) & 1, abort);
                uint4 s0, s1;
                s0.x = at_scale_bf16x2(q0.x, a.scale); s0.y = at_scale_bf16x2(q0.y, a.scale);
                s0.z = at_scale_bf16x2(q0.z, a.scale); s0.w = at_scale_bf16x2(q0.w, a.scale);
                s1.x = at_scale_bf16x2(q1.x, a.scale); s1.y = at_scale_bf16x2(q1.y, a.scale);
                s1.z = at_scale_bf16x2(q1.z, a.scale); s1.w = at_scale_bf16x2(q1.w, a.scale);
                unsigned char* qp = smem + lay.off_q + (g * 2 + qs) * AT_Q_BYTES;
                *reinterpret_cast<uint4*>(qp + t * 16) = s0;
                *reinterpret_cast<uint4*>(qp + AT_Q_BYTES / 2 + t * 16) = s1;
                const int r = tile * AT_BM + t;
                qrow[(g * 2 + qs) * AT_BM + t] = r < L ? src_s[r] : -1;
                // (a NaN fails the test)
                const bool bounded = sq_norm16(s0, s1) * kn <= lim;
                const uint32_t flag = __all_sync(0xffffffffu, bounded) ? 0u : 1u;
                if (lane == 0) qflag[(g * 2 + qs) * 4 + lw] = flag;
                fetch_q(tile + 1);
                // (this and, with a pair's first tile, K: in every warp ahead of V, and V ahead of the next pair's K)
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive_one(gbar + 8 * (AT_B_QFULL + qs));
                if (tile == w.lo) {
                    cp_async_wait<0>();
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_one(vbar + 8 * slot);
                }
            }
        }
        if (!waited) pdl_wait();          // (no CTA ends before the kernel ahead has: the one behind relies on it)
        cp_async_wait<0>();
    } else if (warp < AT_GROUPS) {
        // ---- issuing warp of group g ------------------------------------------------------------------------------
        const int g = warp;
        const uint32_t gbar = bar0 + 8 * AT_B_GROUP * g;
        const uint32_t tm = tmem_base + g * AT_TM_GROUP;
        constexpr uint32_t IDESC_S = umma_idesc_bf16(AT_BM, AT_BK);
        constexpr uint32_t IDESC_O = umma_idesc_bf16(AT_BM, 32) | (1u << 16);   // B is MN-major
        // A = Q planes [d half][row], B = K planes [d half][key]
        const uint64_t desc_q = umma_desc_plain(sbase + lay.off_q + g * 2 * AT_Q_BYTES, AT_Q_BYTES / 2, 128);
        const uint64_t desc_k = umma_desc_plain(sbase + 3 * lay.plane, lay.plane, 128);
        // B = planes [d chunk][key]: V, V, ones, and K's first (columns that nobody reads)
        const uint64_t desc_v = umma_desc_plain(sbase, 128, lay.plane);
        uint32_t pphase = 0;
        int k = 0;                    // tiles so far
        AtWalk w(a);
        while (w.next()) {
            const int nb = w.blocks(), tail = w.tail();
            const uint32_t vparity = (w.counted >> 1) & 1, vb = vbar + 8 * (w.counted & 1);
            const uint64_t slot = w.counted & 1 ? lay.slot >> 4 : 0;
            for (int tile = w.first(g); tile < w.hi; tile += AT_GROUPS, ++k) {
                mbar_wait(gbar + 8 * (AT_B_QFULL + (k & 1)), (k >> 1) & 1, abort);      // and K of the pair
                const uint4 f = *reinterpret_cast<const uint4*>(qflag + (g * 2 + (k & 1)) * 4);
                const uint64_t dq = desc_q + (k & 1) * (AT_Q_BYTES >> 4);
                const uint64_t dk = desc_k + slot;
                uint64_t dv = desc_v + slot;
                // P V' of a full block, or of the tile's last one.  The S issued behind it overwrites P (order: see umma_bf16).
                auto issue_pv = [&](bool first, int steps) {
                    if (steps == AT_BK / 16) {
#pragma unroll
                        for (int i = 0; i < AT_BK / 16; ++i)
                            umma_bf16_ts(tm + AT_TM_O, tm + 8 * i, dv + 16 * i, IDESC_O, !first || i > 0);
                    } else {
                        for (int i = 0; i < steps; ++i)
                            umma_bf16_ts(tm + AT_TM_O, tm + 8 * i, dv + 16 * i, IDESC_O, !first || i > 0);
                    }
                };
                auto issue_s = [&](int j) {
                    const uint32_t idesc = j + 1 < nb ? IDESC_S : umma_idesc_bf16(AT_BM, 16 * tail);
                    umma_bf16(tm, dq, dk + (uint64_t)(j * AT_BK), idesc, false);
                    umma_commit(gbar + 8 * AT_B_S);
                };
                auto wait_p = [&]() {
                    mbar_wait(gbar + 8 * AT_B_P, pphase, abort);
                    pphase ^= 1;
                    __syncwarp();
                };
                __syncwarp();
                if ((f.x | f.y | f.z | f.w) != 0)           // the scores once for their maxima
                    for (int j = 0; j < nb; ++j) {
                        if (elect_one()) {
                            fence_after_sync();
                            issue_s(j);
                        }
                        wait_p();
                    }
                if (elect_one()) {
                    fence_after_sync();
                    issue_s(0);
                }
                __syncwarp();
                // (the pair before in this slot is complete: its V was there before this tile's Q)
                mbar_wait(vb, vparity, abort);
                for (int j = 0; j + 1 < nb; ++j) {
                    wait_p();
                    if (elect_one()) {
                        fence_after_sync();
                        issue_pv(j == 0, AT_BK / 16);
                        issue_s(j + 1);
                    }
                    __syncwarp();
                    dv += AT_BK;
                }
                wait_p();
                if (elect_one()) {
                    fence_after_sync();
                    issue_pv(nb == 1, tail);
                    umma_commit(gbar + 8 * AT_B_O);
                }
                __syncwarp();
            }
        }
        // nothing of this warp's is in flight when the CTA ends, whatever happened
        if (elect_one()) umma_commit(gbar + 8 * AT_B_DONE);
        __syncwarp();
        int give_up = 0;
        mbar_wait(gbar + 8 * AT_B_DONE, 0, &give_up);
    } else {
        // ---- softmax: thread t owns query row t of its group's tiles -----------------------------------------------
        const int g = warp / 4 - 1, t = tid & 127;
        const uint32_t gbar = bar0 + 8 * AT_B_GROUP * g;
        const uint32_t tm = tmem_base + ((uint32_t)((warp & 3) * 32) << 16) + g * AT_TM_GROUP;
        const AtPoly poly;
        uint32_t sphase = 0;
        int k = 0;               // tiles so far
        auto wait_s = [&]() {
            mbar_wait(gbar + 8 * AT_B_S, sphase, abort);
            sphase ^= 1;
            fence_after_sync();
        };
        auto hand_over = [&]() {  // this warp's P (or its reads of S) are done
            fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_one(gbar + 8 * AT_B_P);
        };
        AtWalk w(a);
        while (w.next()) {
            const int nb = w.blocks(), tail = w.tail(), L = w.L;
            for (int tile = w.first(g); tile < w.hi; tile += AT_GROUPS, ++k) {
                const int qs = k & 1;
                uint32_t x[16], y[16];
                wait_s();
                // (the issuing warp has waited for the Q tile that S was made from)
                const int32_t e = qrow[(g * 2 + qs) * AT_BM + t];
                const uint4 f = *reinterpret_cast<const uint4*>(qflag + (g * 2 + qs) * 4);
                if ((f.x | f.y | f.z | f.w) == 0) {
                    for (int j = 0; j < nb; ++j) {
                        if (j) wait_s();
                        if (j + 1 < nb || tail == AT_BK / 16) {
                            tmem_ld16(tm, x);
                            at_chunks<0, AT_BK / 16>(x, y, tm, poly);
                        } else {
                            for (int i = 0; i < tail; ++i) {
                                uint32_t pk[8];
                                tmem_ld16(tm + 16 * i, x);
                                tmem_ld16_fence(x);
                                at_probabilities<0>(x, pk, poly);
                                tmem_st8(tm + 8 * i, pk);
                            }
                        }
                        tmem_st_wait();
                        hand_over();
                    }
                } else {
                    float m = -INFINITY;
                    for (int j = 0; j < nb; ++j) {
                        if (j) wait_s();
                        const int steps = j + 1 < nb ? AT_BK / 16 : tail;
                        for (int i = 0; i < steps; ++i) {
                            tmem_ld16(tm + 16 * i, x);
                            tmem_ld16_fence(x);
                            const int valid = L - j * AT_BK - 16 * i;
#pragma unroll
                            for (int c = 0; c < 16; ++c)
                                if (c < valid) m = fmaxf(m, __uint_as_float(x[c]));
                        }
                        hand_over();
                    }
                    const float mb = -m * AT_LOG2E;
                    for (int j = 0; j < nb; ++j) {
                        wait_s();
                        const int steps = j + 1 < nb ? AT_BK / 16 : tail;
                        for (int i = 0; i < steps; ++i) {
                            uint32_t pk[8];
                            tmem_ld16(tm + 16 * i, x);
                            tmem_ld16_fence(x);
                            at_probabilities_ref(x, pk, mb, L - j * AT_BK - 16 * i);
                            tmem_st8(tm + 8 * i, pk);
                        }
                        tmem_st_wait();
                        hand_over();
                    }
                }
                mbar_wait(gbar + 8 * AT_B_O, k & 1, abort);
                fence_after_sync();
                // (the next tile's first P V overwrites these columns: issued behind this warp's next hand-over)
                tmem_ld16(tm + AT_TM_O, x);
                tmem_ld16(tm + AT_TM_O + 16, y);
                tmem_ld16_fence(x);
                tmem_ld16_fence(y);
                __syncwarp();
                if (lane == 0) mbar_arrive_one(gbar + 8 * (AT_B_QFREE + qs));
                if (e >= 0) {
                    const float inv = 1.f / __uint_as_float(y[0]);
                    uint4 o[2];
                    uint32_t* ow = reinterpret_cast<uint32_t*>(o);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        ow[i] = pack_bf16(__uint_as_float(x[2 * i]) * inv, __uint_as_float(x[2 * i + 1]) * inv);
                    uint4* op = reinterpret_cast<uint4*>(a.out + (int64_t)e * C + w.head * AT_D);
                    op[0] = o[0];
                    op[1] = o[1];
                }
            }
            // this warp's products with K and V of the pair are complete (and a group without a tile in it waits, or it
            // would count twice for the pair before in this slot)
            mbar_wait(vbar + 8 * (w.counted & 1), (w.counted >> 1) & 1, abort);
            __syncwarp();
            if (lane == 0) mbar_arrive_one(kvfree + 8 * (w.counted & 1));
        }
    }

    fence_before_sync();
    __syncthreads();
    if (tid == 0 && *abort) atomicOr(a.status, PTV3_STATUS_WAIT_LIMIT);
    if (warp == AT_LOAD_WARP) {
        fence_after_sync();
        tmem_dealloc(tmem_base, 512);
    }
}

bool attn_tc05_supported(int n_seq, int channels, int heads, int max_seqlen)
{
    return channels % heads == 0 && channels / heads == AT_D && max_seqlen <= ATTN_TC05_MAX_SEQLEN &&
           (int64_t)n_seq * heads * AT_MAX_TILES < (1ll << 31);
}

// Whether this kernel is faster than the mma.sync one (attention_mma.cu) on n points in n_seq patches.  Three things speak
// against it: few blocks (a CTA starts with ~7 us of gather, and a group alone on an SM takes 1 800 cycles a block, three
// together 1 035 each), short patches (a pair's gather takes the loading warps ~5 us) and rows of a tile that
// the patch does not have.  us here and there, H heads of 16, blocks of 128 x 128 scores per SM:
//   patches of 1 024: 8 192 points H 8 (28 blocks) 28.9 / 27.6, 12 288 H 8 (42) 35.2 / 37.9, 100 000 H 4 (169) 103 / 121,
//     400 000 H 4 (676) 363 / 448;  of 800: 3 200 H 32 (38) 33.9 / 39.0;  of 640: 2 560 H 32 (22) 22.4 / 22.7
//   of 512: 20 000 H 8 (35) 29.4 / 33.7;  of 384: 30 000 H 8 (38) 34.7 / 35.6, 200 000 H 4 (127) 91.6 / 99.5
//   of 320: 200 000 H 4 (106) 103 / 88;  of 256: 400 000 H 4 (169) 168 / 146
bool attn_tc05_wanted(int64_t n, int n_seq, int heads, int max_seqlen)
{
    const int64_t mean = (n + n_seq - 1) / n_seq;      // (a caller may state a longer patch than there is)
    const int64_t len = mean < max_seqlen ? mean : max_seqlen;
    const int64_t tiles = (len + AT_BM - 1) / AT_BM, steps = (len + 15) / 16;
    if (len < 384 || (len < 640 && tiles * AT_BM * steps * 16 * 10 > len * len * 11)) return false;
    return (int64_t)n_seq * heads * tiles * steps >= 33 * SMS * (AT_BK / 16);
}

int launch_attn_tc05(const void* qkv, const int64_t* order, const int64_t* pad, const int64_t* unpad,
                     const int32_t* cu, void* out, int n_seq, int max_seqlen, int C, int H, float scale,
                     bool planned, uint32_t* status, cudaStream_t stream)
{
    AtArgs a{(const __nv_bfloat16*)qkv, order, pad, unpad, cu, (__nv_bfloat16*)out, n_seq, H,
             (max_seqlen + AT_BM - 1) / AT_BM, (max_seqlen + AT_BM - 1) / AT_BM * AT_BM, scale, planned, status};
    const AtLayout lay(a.lpad);
    // A CTA takes the whole tensor memory of its SM: ask for enough shared memory that no
    // second CTA shares the SM (it would wait in tcgen05.alloc).
    const size_t floor_smem = (size_t)(228 * 1024 / 2 + 1024);
    const size_t smem = lay.total + 128 < floor_smem ? floor_smem : (size_t)lay.total + 128;
    if (allow_smem(attn_tc05_d16_kernel) != cudaSuccess)
        return check_launch("ptv3_attention_fwd: shared memory attribute");
    const int64_t total = (int64_t)n_seq * H * a.tiles;
    const dim3 grid((unsigned)(total < SMS ? total : SMS));
    launch_dependent(attn_tc05_d16_kernel, grid, dim3(AT_THREADS), smem, stream, a);
    count_launches(1);
    return check_launch("ptv3_attention_fwd");
}

}  // namespace ptv3
