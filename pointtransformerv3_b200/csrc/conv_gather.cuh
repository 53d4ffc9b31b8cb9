// One stage of the convolutions on tcgen05 (conv_tc05.cu, conv_stream.cu): the 128 neighbour rows of an offset, KC
// channels wide, and the matching slice of W, brought into a slot of the ring by one warp.
#pragma once
#include "mma_util.cuh"
#include "tc05.cuh"

namespace ptv3 {

constexpr int CG_ROWS = 128;           // voxels per tile

// What a lane copies: one 16-byte chunk of a row, into the swizzled K-major operand layout (spans of 128 bytes, of 64 for
// 32 channels).  The lanes of a row take four rows, the next ones the four after them, so that the numbers of four rows
// are one load.
template <int KC>
struct RowGather {
    static constexpr int ROWB = KC * 2, NCH = ROWB / 16, GROUPS = 32 / NCH;       // GROUPS: rows per instruction
    static_assert(NCH == 8 || NCH == 4, "one swizzle span per row");
    int chunk, row4;
    uint32_t dst[4];                   // within a stage's rows, of the four rows

    __device__ explicit RowGather(int lane) : chunk(lane % NCH), row4(lane / NCH * 4)
    {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int r = row4 + j;
            dst[j] = (uint32_t)(r * ROWB + ((NCH == 8 ? chunk ^ (r & 7) : chunk ^ ((r >> 1) & 3)) << 4));
        }
    }

    // rows nbr[0 .. 128) of `src` (its first channel of the stage), `pitch` bytes apart; zero rows where there is none
    __device__ __forceinline__ void copy(uint32_t slot, const int32_t* nbr, const char* src, uint32_t pitch) const
    {
        src += chunk * 16;
        nbr += row4;
#pragma unroll
        for (int j0 = 0; j0 < CG_ROWS; j0 += GROUPS * 4) {
            const int4 n4 = *reinterpret_cast<const int4*>(nbr + j0);
            const int row[4] = {n4.x, n4.y, n4.z, n4.w};
#pragma unroll
            for (int j = 0; j < 4; ++j)
                cp_async16_zfill(slot + j0 * ROWB + dst[j], src + (uint64_t)(uint32_t)max(row[j], 0) * pitch, row[j] >= 0);
        }
    }
};

// The whole stage, in a slot that is free: the copies, then (they are on their way) the W_BYTES of W at column x and row y
// behind them, and the arrival at `full` once the copies have landed.
template <int KC, int W_BYTES>
__device__ __forceinline__ void fill_stage(const RowGather<KC>& gather, uint32_t slot, const int32_t* nbr, const char* src,
                                           uint32_t pitch, const CUtensorMap* map_w, int x, int y, uint32_t full, int lane)
{
    gather.copy(slot, nbr, src, pitch);
    cp_async_commit();
    if (tc05::elect_one()) {
        tc05::mbar_expect_tx(full, W_BYTES);
        tc05::tma_load_2d(slot + CG_ROWS * KC * 2, map_w, x, y, full);
    }
    cp_async_wait<0>();
    tc05::fence_proxy_async();
    __syncwarp();
    if (lane == 0) tc05::mbar_arrive_one(full);
}

// Where a warp that takes every STEP-th stage stands: the offset (by its place in the list of those in use) and chunk of
// its stage, counted, not divided, from stage to stage; the slot of the ring and the phase of its barriers.
struct StageCursor {
    int at, chunk, slot, phase;
    template <int STEP, int STAGES>
    __device__ __forceinline__ void step(int kchunks)
    {
        chunk += STEP;
        while (chunk >= kchunks) {
            chunk -= kchunks;
            ++at;
        }
        slot += STEP;
        if (slot >= STAGES) {
            slot -= STAGES;
            phase ^= 1;
        }
    }
};

}  // namespace ptv3
