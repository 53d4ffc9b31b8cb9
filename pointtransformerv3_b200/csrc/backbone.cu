// The whole backbone in one call (model.py:884-982 for segmentation networks, inference).
//
// A pass over a small room is bounded by its host: 276 launches queued through a Python-level module
// tree took 3.9 ms for 1.75 ms of GPU work (6 000 points; 4.7 ms for 3.0 ms at 100 000).  Here the same
// kernels are queued from C++ (two streams, as before: serialization, kernel maps and pooling plans on
// the planning stream, features on the main stream), with memory carved from a few chunks instead of one
// allocation per tensor, and with one difference in schedule: the size of a coarse level is looked
// for after every block without waiting, so the next plan is launched as soon as the last one is known
// instead of when its stage comes up.
#include "common.cuh"
#include "linear.cuh"
#include "plan.cuh"
#include "split_f32.cuh"
#include <string.h>
#include <memory>
#include <new>

namespace ptv3 {

constexpr int BB_MAX_STAGES = 12;
constexpr size_t BB_CHUNK = (size_t)16 << 20;       // smallest piece of memory asked for at a time

#define BB_STEP(call)                    \
    do {                                 \
        const int rc_ = (call);          \
        if (rc_ != PTV3_OK) return rc_;  \
    } while (0)
#define BB_CUDA(call)                                                                 \
    do {                                                                              \
        if ((call) != cudaSuccess) return check_launch("ptv3_backbone_fwd: " #call);  \
    } while (0)

// pieces of the chunks that the caller hands out
class Arena {
public:
    Arena(ptv3_alloc_fn fn, void* ctx, int pool) : fn_(fn), ctx_(ctx), pool_(pool) {}
    template <typename T>
    T* take(size_t count)
    {
        const size_t bytes = align_up(count * sizeof(T) + 1, 256);
        if (bytes > left_) {
            const size_t ask = bytes > BB_CHUNK ? bytes : BB_CHUNK;
            char* p = static_cast<char*>(fn_(ctx_, ask, pool_));
            if (!p) return nullptr;
            // the larger rest is kept for what comes next
            if (ask - bytes < left_) return reinterpret_cast<T*>(p);
            at_ = p;
            left_ = ask;
        }
        char* p = at_;
        at_ += bytes;
        left_ -= bytes;
        return reinterpret_cast<T*>(p);
    }

private:
    ptv3_alloc_fn fn_;
    void* ctx_;
    int pool_;
    char* at_ = nullptr;
    size_t left_ = 0;
};

// events of one pass, given back at its end (work queued behind them is not affected)
class Events {
public:
    ~Events()
    {
        for (int i = 0; i < n_; ++i) cudaEventDestroy(ev_[i]);
    }
    cudaError_t record(cudaStream_t s, cudaEvent_t* out)
    {
        cudaEvent_t e;
        cudaError_t rc = cudaEventCreateWithFlags(&e, cudaEventDisableTiming);
        if (rc != cudaSuccess) return rc;
        ev_[n_++] = e;
        *out = e;
        return cudaEventRecord(e, s);
    }

private:
    cudaEvent_t ev_[BB_MAX_STAGES + 4];
    int n_ = 0;
};

struct BbLevel {
    int64_t n = 0;
    int depth = 0;
    const int64_t* counts = nullptr;                        // HOST
    const int64_t *code = nullptr, *order = nullptr, *batch = nullptr, *offset = nullptr;
    const int32_t *grid = nullptr, *nbr = nullptr;
    int64_t *cluster = nullptr, *idx_ptr = nullptr;         // pooling of this level into the next
    // patch layout, made for patch size `patch`
    int patch = 0, n_seq = 0, longest = 0;                  // (longest: no sequence has more rows)
    int64_t *pad = nullptr, *unpad = nullptr;
    int32_t* cu = nullptr;
    const void* feat = nullptr;                             // encoder output (skip connection)
    cudaEvent_t ready = nullptr;                            // kernel map and patch layout are queued
    bool begun = false;                                     // a kernel of the level is queued behind that event
};

class Pass {
public:
    explicit Pass(const ptv3_backbone_args* a)
        : a_(*a), main_((cudaStream_t)a->main_stream), side_((cudaStream_t)a->plan_stream), mem_(a->alloc, a->alloc_ctx, 0),
          plan_mem_(a->alloc, a->alloc_ctx, 1)
    {
        memcpy(enc_, a->enc, a->n_enc * sizeof(ptv3_stage_args));
        memcpy(dec_, a->dec, a->n_dec * sizeof(ptv3_stage_args));
    }
    int run();

private:
    const ptv3_backbone_args& a_;
    cudaStream_t main_, side_;
    Arena mem_, plan_mem_;
    Events events_;
    ptv3_stage_args enc_[BB_MAX_STAGES], dec_[BB_MAX_STAGES];       // as given, with this pass's split weights
    std::unique_ptr<ptv3_block_args[]> blocks_;                     // ... and the blocks they point to
    BbLevel lv_[BB_MAX_STAGES];
    int made_ = 0;                  // levels whose geometry is queued
    // the plan in flight (pooling of level made_ - 1): packed outputs whose row stride is not known yet
    bool flying_ = false;
    int64_t *pcode_ = nullptr, *porder_ = nullptr, *pbatch_ = nullptr, *poffset_ = nullptr;
    int32_t *pgrid_ = nullptr, *pindices_ = nullptr;
    // scratch of the main stream, reused in stream order
    char* ws_ = nullptr;
    size_t ws_bytes_ = 0;

    const size_t esize_ = a_.dtype == PTV3_DTYPE_F32 ? 4 : 2;

    int64_t* flag(int l) const { return a_.meta_host + (int64_t)l * (3 + a_.n_scenes); }
    int out_of_memory() const
    {
        set_error("ptv3_backbone_fwd: the caller's allocator returned no memory");
        return PTV3_ERR_WORKSPACE;
    }
    int need_ws(size_t bytes)
    {
        if (bytes > ws_bytes_) {
            ws_ = mem_.take<char>(bytes);
            if (!ws_) return out_of_memory();
            ws_bytes_ = bytes;
        }
        return PTV3_OK;
    }
    static int patch_of(int patch, const BbLevel& l, int n_scenes)
    {
        if (patch > 0) return patch;
        int64_t least = -(int64_t)patch;
        for (int b = 0; b < n_scenes; ++b) least = l.counts[b] < least ? l.counts[b] : least;
        return (int)least;
    }
    int pad_level(BbLevel& l, int patch, Arena& mem, cudaStream_t stream, int64_t* pad, int64_t* unpad, int32_t* cu,
                  const VoxelClear& index);
    const float *stem_scale_ = a_.stem_scale, *stem_shift_ = a_.stem_shift;
    int norms(BnJobs* jobs);
    template <typename F>
    int each_weight(F&& f);
    int split_weights();
    int finest();
    int launch_plan();
    int take_plan(bool block);
    int block(const ptv3_stage_args& st, int j, BbLevel& l, const void* conv_in, const void* feat, void* out);
    int project(const void* x, const void* w, const void* bias, int64_t n, int c_in, int c_out, void* split, void* out);
    int encoder(int s);
    int decoder(int d);
};

// patch layout of a level (model.py:382-438); pad / unpad / cu may be given; a layout that is made clears `index` too
int Pass::pad_level(BbLevel& l, int patch, Arena& mem, cudaStream_t stream, int64_t* pad, int64_t* unpad, int32_t* cu,
                    const VoxelClear& index)
{
    if (l.patch == patch) return PTV3_OK;
    PTV3_REQUIRE(patch >= 1, PTV3_ERR_INVALID_ARGUMENT, "ptv3_backbone_fwd: patch size %d", patch);
    int64_t n_pad = 0, n_seq = 0, longest = 1;
    for (int b = 0; b < a_.n_scenes; ++b) {
        const int64_t c = l.counts[b], cp = c > patch ? (c + patch - 1) / patch * patch : c;
        n_pad += cp;
        n_seq += (cp + patch - 1) / patch;
        longest = c > longest ? c : longest;
    }
    l.longest = longest < patch ? (int)longest : patch;
    l.pad = pad ? pad : mem.take<int64_t>(n_pad);
    l.unpad = unpad ? unpad : mem.take<int64_t>(l.n);
    l.cu = cu ? cu : mem.take<int32_t>(n_seq + 1);
    if (!l.pad || !l.unpad || !l.cu) return out_of_memory();
    l.patch = patch;
    l.n_seq = (int)n_seq;
    return pad_plan(l.offset, a_.n_scenes, patch, l.n, n_pad, (int)n_seq, l.pad, l.unpad, l.cu, a_.status, index, stream);
}

// BatchNorm layers as scale and shift, computed for this pass (as the weights below): where they will lie
int Pass::norms(BnJobs* jobs)
{
    constexpr int MOST = 1 + 3 * BB_MAX_STAGES;
    static_assert(MOST <= BN_JOBS, "one launch holds them");
    ptv3_bn_args layers[MOST];
    const float** slots[MOST][2];
    int count = 0;
    size_t floats = 0;
    auto add = [&](const ptv3_bn_args* bn, int channels, const float*& scale, const float*& shift) {
        if (!bn) return PTV3_OK;
        PTV3_REQUIRE(bn->channels == channels, PTV3_ERR_INVALID_ARGUMENT,
                     "ptv3_backbone_fwd: BatchNorm over %d channels where %d go in", bn->channels, channels);
        slots[count][0] = &scale;
        slots[count][1] = &shift;
        layers[count++] = *bn;
        floats += 2 * (size_t)channels;
        return PTV3_OK;
    };
    BB_STEP(add(a_.stem_bn, a_.stem_c_out, stem_scale_, stem_shift_));
    for (int s = 1; s < a_.n_enc; ++s) BB_STEP(add(enc_[s].bn, enc_[s].c_out, enc_[s].scale, enc_[s].shift));
    for (int d = 0; d < a_.n_dec; ++d) {
        BB_STEP(add(dec_[d].bn, dec_[d].c_out, dec_[d].scale, dec_[d].shift));
        BB_STEP(add(dec_[d].bn_skip, dec_[d].c_out, dec_[d].scale_skip, dec_[d].shift_skip));
    }
    float* out = count ? mem_.take<float>(floats) : nullptr;
    if (count && !out) return out_of_memory();
    BB_STEP(bn_jobs(layers, count, out, jobs));
    for (int i = 0; i < count; ++i) {
        *slots[i][0] = jobs->out[i];
        *slots[i][1] = jobs->out[i] + layers[i].channels;
    }
    return PTV3_OK;
}

// f(pointer, rows, inner dimension) of every weight that enters a matrix product; `blocks_` holds the blocks
template <typename F>
int Pass::each_weight(F&& f)
{
    for (int s = 0; s < a_.n_enc + a_.n_dec; ++s) {
        const bool encoder = s < a_.n_enc;
        ptv3_stage_args& st = encoder ? enc_[s] : dec_[s - a_.n_enc];
        if (s > 0) BB_STEP(f(st.w, st.c_out, st.c_in));
        if (!encoder) BB_STEP(f(st.w_skip, st.c_out, st.c_skip));
        ptv3_block_args* b = const_cast<ptv3_block_args*>(st.blocks);
        for (int j = 0; j < st.n_blocks; ++j, ++b) {
            const int C = b->channels, H = b->hidden;
            BB_STEP(f(b->conv_weight, (int64_t)27 * C, C));
            BB_STEP(f(b->cpe_w, C, C));
            BB_STEP(f(b->qkv_w, (int64_t)3 * C, C));
            BB_STEP(f(b->proj_w, C, C));
            BB_STEP(f(b->fc1_w, H, C));
            BB_STEP(f(b->fc2_w, C, H));
        }
    }
    return PTV3_OK;
}

// fp32 weights, split for this pass: what the caller writes to them is seen by the next pass, whichever way it
// is written and on whatever stream.  The default network's 183 MB become 275, one launch that runs on the main
// stream while that waits for the sort (two rooms of 20 000 points: 6.58 ms a pass, 6.50 with splits that were kept).
int Pass::split_weights()
{
    if (a_.dtype != PTV3_DTYPE_F32 || !a_.plain_weights) return PTV3_OK;
    int n_blocks = 0, count = 0;
    for (int s = 0; s < a_.n_enc; ++s) n_blocks += enc_[s].n_blocks;
    for (int d = 0; d < a_.n_dec; ++d) n_blocks += dec_[d].n_blocks;
    blocks_.reset(new (std::nothrow) ptv3_block_args[n_blocks]);
    std::unique_ptr<SplitWeight[]> jobs(new (std::nothrow) SplitWeight[6 * n_blocks + a_.n_enc + 2 * a_.n_dec]);
    PTV3_REQUIRE(blocks_ && jobs, PTV3_ERR_WORKSPACE, "ptv3_backbone_fwd: out of host memory");
    ptv3_block_args* at = blocks_.get();
    for (int s = 0; s < a_.n_enc + a_.n_dec; ++s) {
        ptv3_stage_args& st = s < a_.n_enc ? enc_[s] : dec_[s - a_.n_enc];
        memcpy(at, st.blocks, st.n_blocks * sizeof(ptv3_block_args));
        st.blocks = at;
        at += st.n_blocks;
    }
    size_t bytes = 0;
    BB_STEP(each_weight([&](const void*& w, int64_t rows, int k) {
        PTV3_REQUIRE(w && ((uintptr_t)w & 15) == 0 && rows > 0 && k >= 32 && k % 32 == 0, PTV3_ERR_INVALID_ARGUMENT,
                     "ptv3_backbone_fwd: a weight of %lld x %d: null, alignment or width", (long long)rows, k);
        jobs[count++] = SplitWeight{(const float*)w, rows, k, nullptr};
        bytes += align_up((size_t)rows * split_stored(k) * k * 2, 256);
        return PTV3_OK;
    }));
    char* out = mem_.take<char>(bytes);
    if (!out) return out_of_memory();
    int j = 0;
    BB_STEP(each_weight([&](const void*& w, int64_t rows, int k) {
        w = jobs[j++].out = out;
        out += align_up((size_t)rows * split_stored(k) * k * 2, 256);
        return PTV3_OK;
    }));
    return launch_split_weights(jobs.get(), count, main_);
}

// serialization, voxel index, kernel map and stem of the finest level
int Pass::finest()
{
    BbLevel& l = lv_[0];
    l.n = a_.n;
    l.depth = a_.depth;
    l.counts = a_.level_counts;
    memcpy(a_.level_counts, a_.counts, a_.n_scenes * sizeof(int64_t));
    l.code = a_.code;
    l.order = a_.order;
    l.batch = a_.batch;
    l.offset = a_.offset;
    l.grid = a_.grid_coord;
    l.nbr = a_.nbr;
    cudaEvent_t inputs, indexed, sorted;
    BB_CUDA(events_.record(main_, &inputs));
    BB_CUDA(cudaStreamWaitEvent(side_, inputs, 0));
    // planning stream: codes, orders, inverses
    // (bits of the largest scene number: a larger one in `batch` is reported by the first pooling plan)
    int scene_bits = 0;
    while (((a_.n_scenes - 1) >> scene_bits) != 0) ++scene_bits;
    const int sig_bits = 3 * a_.depth + scene_bits;
    const size_t sort_bytes = ptv3_argsort_workspace_bytes(a_.k, a_.n, sig_bits);
    char* sort_ws = plan_mem_.take<char>(sort_bytes);
    if (!sort_ws) return out_of_memory();
    BB_STEP(ptv3_encode(a_.grid_coord, a_.batch, a_.n, a_.depth, a_.order_ids, a_.k, a_.code, side_));
    BB_STEP(ptv3_argsort_inverse(a_.code, a_.k, a_.n, sig_bits, a_.order, a_.inverse, a_.status, sort_ws, sort_bytes,
                                 side_));
    BB_CUDA(events_.record(side_, &sorted));
    // main stream, beside them: the voxel index that the stem and the 3x3x3 kernel map share.  (Its first
    // kernel is an ordinary launch: what `settled` stands on, see linear.cuh.)
    char* index_ws = mem_.take<char>(voxel_index_bytes(a_.n));
    char* wt = mem_.take<char>(conv_direct_scratch_bytes(a_.n, a_.stem_ksize));
    if (!index_ws || !wt) return out_of_memory();
    BnJobs bn;
    BB_STEP(norms(&bn));
    VoxelIndex vi;
    const VoxelClear empty = place_voxel_index(a_.n, index_ws, &vi);
    BB_STEP(batch_indices_and_norms(a_.offset, a_.n_scenes, a_.grid_coord, a_.n, a_.indices, empty, bn, main_));
    BB_STEP(fill_voxel_index(vi, empty, a_.indices, a_.n, a_.status, main_));
    BB_CUDA(events_.record(main_, &indexed));
    BB_STEP(split_weights());
    BB_CUDA(cudaStreamWaitEvent(side_, indexed, 0));
    BB_STEP(kmap_from_index(vi, a_.indices, a_.n, 3, a_.order, a_.nbr, a_.status, side_));
    if (enc_[0].n_blocks > 0)
        BB_STEP(pad_level(l, patch_of(enc_[0].patch[0], l, a_.n_scenes), plan_mem_, side_, a_.pad, a_.unpad,
                          a_.cu_seqlens, VoxelClear{}));
    BB_CUDA(events_.record(side_, &l.ready));
    made_ = 1;
    BB_STEP(launch_plan());
    BB_CUDA(cudaStreamWaitEvent(main_, sorted, 0));
    void* feat = mem_.take<char>((size_t)a_.n * a_.stem_c_out * esize_);
    if (!feat) return out_of_memory();
    BB_STEP(conv_direct_from_index(vi, a_.feat, a_.indices, a_.stem_weight, stem_scale_, stem_shift_, feat, a_.order,
                                   a_.n, a_.stem_c_in, a_.stem_c_out, a_.stem_ksize, a_.dtype, a_.status, wt, main_));
    l.feat = feat;
    return PTV3_OK;
}

// queues the pooling plan of the coarsest level made so far (model.py:639-695)
int Pass::launch_plan()
{
    if (made_ >= a_.n_enc) return PTV3_OK;
    BbLevel& p = lv_[made_ - 1];
    const int depth = enc_[made_].pooling_depth <= p.depth ? enc_[made_].pooling_depth : 0;
    const size_t bytes = ptv3_pool_plan_workspace_bytes(a_.k, p.n, a_.n_scenes);
    p.cluster = plan_mem_.take<int64_t>(p.n);
    p.idx_ptr = plan_mem_.take<int64_t>(p.n + 1);
    int64_t* head = plan_mem_.take<int64_t>(p.n);
    pcode_ = plan_mem_.take<int64_t>((size_t)a_.k * p.n);
    porder_ = plan_mem_.take<int64_t>((size_t)a_.k * p.n);
    int64_t* pinverse = plan_mem_.take<int64_t>((size_t)a_.k * p.n);
    pgrid_ = plan_mem_.take<int32_t>((size_t)3 * p.n);
    pbatch_ = plan_mem_.take<int64_t>(p.n);
    poffset_ = plan_mem_.take<int64_t>(a_.n_scenes);
    pindices_ = plan_mem_.take<int32_t>((size_t)4 * p.n);
    int64_t* meta = plan_mem_.take<int64_t>(1 + a_.n_scenes);
    char* ws = plan_mem_.take<char>(bytes);
    if (!p.cluster || !p.idx_ptr || !head || !pcode_ || !porder_ || !pinverse || !pgrid_ || !pbatch_ || !poffset_ ||
        !pindices_ || !meta || !ws)
        return out_of_memory();
    int64_t* host = flag(made_ - 1);
    reinterpret_cast<volatile int64_t*>(host)[2 + a_.n_scenes] = 0;
    BB_STEP(pool_plan(p.code, p.order, p.grid, p.batch, a_.k, p.n, a_.n_scenes, depth,
                      a_.row_perm ? a_.row_perm + (size_t)(made_ - 1) * a_.k : nullptr, p.cluster, p.idx_ptr, head, pcode_,
                      porder_, pinverse, pgrid_, pbatch_, meta, host, poffset_, pindices_, a_.status, ws, bytes, side_));
    lv_[made_].depth = p.depth - depth;
    flying_ = true;
    return PTV3_OK;
}

// When the plan in flight has been reported (or after waiting for it, with `block`): makes the kernel map
// and the patch layout of its level and queues the next plan.
int Pass::take_plan(bool block)
{
    if (!flying_) return PTV3_OK;
    volatile int64_t* host = flag(made_ - 1);
    if (!host[2 + a_.n_scenes]) {
        if (!block) return PTV3_OK;
        BB_STEP(host_wait(flag(made_ - 1) + 2 + a_.n_scenes, side_));
    }
    flying_ = false;
    PTV3_REQUIRE(host[1 + a_.n_scenes] == 0, PTV3_ERR_CUDA, "device status 0x%x (read after a pooling plan; the word is "
                 "shared by every kernel queued with it)", (unsigned)host[1 + a_.n_scenes]);
    BbLevel& l = lv_[made_];
    l.n = host[0];
    int64_t* counts = a_.level_counts + (size_t)made_ * a_.n_scenes;
    for (int b = 0; b < a_.n_scenes; ++b) counts[b] = host[1 + b];
    l.counts = counts;
    l.code = pcode_;
    l.order = porder_;
    l.grid = pgrid_;
    l.batch = pbatch_;
    l.offset = poffset_;
    int32_t* nbr = plan_mem_.take<int32_t>((size_t)27 * l.n);
    char* ws = plan_mem_.take<char>(voxel_index_bytes(l.n));
    if (!nbr || !ws) return out_of_memory();
    VoxelIndex vi;
    const ptv3_stage_args& st = enc_[made_];
    if (st.n_blocks > 0) {
        const VoxelClear empty = place_voxel_index(l.n, ws, &vi);
        BB_STEP(pad_level(l, patch_of(st.patch[0], l, a_.n_scenes), plan_mem_, side_, nullptr, nullptr, nullptr, empty));
        BB_STEP(fill_voxel_index(vi, empty, pindices_, l.n, a_.status, side_));
    } else {
        BB_STEP(build_voxel_index(pindices_, l.n, ws, a_.status, side_, &vi));
    }
    BB_STEP(kmap_from_index(vi, pindices_, l.n, 3, l.order, nbr, a_.status, side_));
    l.nbr = nbr;
    BB_CUDA(events_.record(side_, &l.ready));
    ++made_;
    return launch_plan();
}

int Pass::block(const ptv3_stage_args& st, int j, BbLevel& l, const void* conv_in, const void* feat, void* out)
{
    ptv3_block_args b = st.blocks[j];
    BB_STEP(pad_level(l, patch_of(st.patch[j], l, a_.n_scenes), mem_, main_, nullptr, nullptr, nullptr,
                      VoxelClear{}));
    b.n = l.n;
    b.n_seq = l.n_seq;
    b.max_seqlen = l.longest;
    b.conv_in = conv_in;
    b.feat = feat;
    b.out = out;
    b.nbr = l.nbr;
    b.row_order = l.order;
    b.pair_in = b.pair_out = b.off_start = b.tile_start = nullptr;
    b.order = l.order + (size_t)st.order_index[j] * l.n;
    b.pad = l.pad;
    b.unpad = l.unpad;
    b.cu_seqlens = l.cu;
    b.status = a_.status;
    const size_t bytes = ptv3_block_workspace_bytes(&b);
    BB_STEP(need_ws(bytes));
    b.workspace = ws_;
    b.workspace_bytes = bytes;
    // (the first block of the finest level comes straight behind the event of its geometry)
    BB_STEP(block_fwd(&b, true, l.begun, main_));
    l.begun = true;
    return take_plan(false);
}

// fp32 projection of a stage transition, on split operands
int Pass::project(const void* x, const void* w, const void* bias, int64_t n, int c_in, int c_out, void* split, void* out)
{
    BB_STEP(launch_split_f32((const float*)x, n, c_in, split, main_));
    return launch_linear_split(split, w, (const float*)bias, nullptr, (float*)out, nullptr, n, c_in, c_out, 0, true,
                               a_.status, main_);
}

int Pass::encoder(int s)
{
    const ptv3_stage_args& st = enc_[s];
    while (made_ <= s) BB_STEP(take_plan(true));
    BbLevel& l = lv_[s];
    BB_CUDA(cudaStreamWaitEvent(main_, l.ready, 0));
    const void* x = l.feat;
    if (s > 0) {
        BbLevel& p = lv_[s - 1];
        void* pooled = mem_.take<char>((size_t)l.n * st.c_out * esize_);
        if (!pooled) return out_of_memory();
        if (a_.dtype == PTV3_DTYPE_F32) {
            const size_t split = align_up((size_t)p.n * st.c_in * 12, 256);
            BB_STEP(need_ws(split + (size_t)p.n * st.c_out * 4));
            BB_STEP(project(p.feat, st.w, st.b, p.n, st.c_in, st.c_out, ws_, ws_ + split));
            BB_STEP(ptv3_pool_fwd(ws_ + split, nullptr, p.order, p.idx_ptr, l.n, st.c_out, st.scale, st.shift, pooled,
                                  nullptr, st.reduce, a_.dtype, main_));
        } else {
            const size_t bytes = ptv3_pool_stage_workspace_bytes(p.n, st.c_out);
            BB_STEP(need_ws(bytes));
            BB_STEP(pool_stage_fwd(p.feat, st.w, st.b, nullptr, p.order, p.idx_ptr, p.n, l.n, st.c_in, st.c_out, st.scale,
                                   st.shift, pooled, nullptr, st.reduce, PTV3_DTYPE_BF16, true, a_.status, ws_, bytes,
                                   main_));
        }
        x = pooled;
        l.begun = true;
    }
    char* buf[2] = {nullptr, nullptr};
    for (int j = 0; j < st.n_blocks; ++j) {
        if (j < 2) {
            buf[j] = mem_.take<char>((size_t)l.n * st.blocks[j].channels * esize_);
            if (!buf[j]) return out_of_memory();
        }
        BB_STEP(block(st, j, l, x, x, buf[j & 1]));
        x = buf[j & 1];
    }
    l.feat = x;
    return PTV3_OK;
}

int Pass::decoder(int d)
{
    const ptv3_stage_args& st = dec_[d];
    BbLevel& c = lv_[a_.n_enc - 1 - d];
    BbLevel& l = lv_[a_.n_enc - 2 - d];
    const size_t row = (size_t)l.n * st.c_out * esize_;
    // out: skip + up-sampled rows; act: the skip branch alone, which the first block's convolution
    // reads (model.py:744-746 adds to `feat` only)
    char* buf[2] = {mem_.take<char>(row), mem_.take<char>(row)};
    char* act = mem_.take<char>(row);
    if (!buf[0] || !buf[1] || !act) return out_of_memory();
    if (a_.dtype == PTV3_DTYPE_F32) {
        const int64_t wide = l.n * st.c_skip > c.n * st.c_in ? l.n * st.c_skip : c.n * st.c_in;
        const size_t split = align_up((size_t)wide * 12, 256), rows = align_up(row, 256);
        BB_STEP(need_ws(split + rows + (size_t)c.n * st.c_out * 4));
        char *skip = ws_ + split, *child = ws_ + split + rows;
        BB_STEP(project(c.feat, st.w, st.b, c.n, st.c_in, st.c_out, ws_, child));
        BB_STEP(project(l.feat, st.w_skip, st.b_skip, l.n, st.c_skip, st.c_out, ws_, skip));
        BB_STEP(ptv3_unpool_fwd(skip, child, l.cluster, l.n, st.c_out, st.scale_skip, st.shift_skip, st.scale, st.shift,
                                buf[0], act, a_.dtype, main_));
    } else {
        const size_t bytes = ptv3_unpool_stage_workspace_bytes(l.n, c.n, st.c_out);
        BB_STEP(need_ws(bytes));
        BB_STEP(unpool_stage_fwd(l.feat, c.feat, st.w_skip, st.b_skip, st.w, st.b, l.cluster, l.n, c.n, st.c_skip, st.c_in,
                                 st.c_out, st.scale_skip, st.shift_skip, st.scale, st.shift, buf[0], act, PTV3_DTYPE_BF16,
                                 true, a_.status, ws_, bytes, main_));
    }
    const void *x = buf[0], *conv_in = act;
    for (int j = 0; j < st.n_blocks; ++j) {
        void* out = d == a_.n_dec - 1 && j == st.n_blocks - 1 ? a_.out : buf[(j + 1) & 1];
        BB_STEP(block(st, j, l, conv_in, x, out));
        x = conv_in = out;
    }
    l.feat = x;
    return PTV3_OK;
}

int Pass::run()
{
    BB_STEP(finest());
    for (int s = 0; s < a_.n_enc; ++s) BB_STEP(encoder(s));
    for (int d = 0; d < a_.n_dec; ++d) BB_STEP(decoder(d));
    return PTV3_OK;
}

}  // namespace ptv3

extern "C" int ptv3_backbone_fwd(const ptv3_backbone_args* a)
{
    using namespace ptv3;
    PTV3_REQUIRE(a != nullptr, PTV3_ERR_INVALID_ARGUMENT, "ptv3_backbone_fwd: null argument block");
    PTV3_REQUIRE(a->n_enc >= 1 && a->n_enc <= BB_MAX_STAGES && a->n_dec == a->n_enc - 1 && a->n_dec >= 1 && a->enc && a->dec,
                 PTV3_ERR_UNSUPPORTED, "ptv3_backbone_fwd: %d encoder and %d decoder stages", a->n_enc, a->n_dec);
    PTV3_REQUIRE(a->dtype == PTV3_DTYPE_BF16 || (a->dtype == PTV3_DTYPE_F32 && a->n <= 65535ll * 128),
                 PTV3_ERR_UNSUPPORTED, "ptv3_backbone_fwd: dtype %d, %lld points", a->dtype, (long long)a->n);
    PTV3_REQUIRE(a->dec[a->n_dec - 1].n_blocks >= 1, PTV3_ERR_UNSUPPORTED,
                 "ptv3_backbone_fwd: the last decoder stage has no block");
    PTV3_REQUIRE(a->n >= 1 && a->n < (1ll << 31) && a->n_scenes >= 1 && a->depth >= 1 && a->k >= 1 &&
                     a->k <= PTV3_MAX_ORDERS,
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_backbone_fwd: bad sizes");
    PTV3_REQUIRE(a->counts && a->order_ids && a->feat && a->grid_coord && a->offset && a->batch && a->code && a->order &&
                     a->inverse && a->indices && a->nbr && a->out && a->level_counts && a->meta_host && a->status &&
                     a->alloc && a->stem_weight && (a->enc[0].n_blocks == 0 || (a->pad && a->unpad && a->cu_seqlens)),
                 PTV3_ERR_INVALID_ARGUMENT, "ptv3_backbone_fwd: null pointer");
    return Pass(a).run();
}
