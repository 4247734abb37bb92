// Hand-over of the dequantised stages of awq_gemm.cu's row-per-thread form: who writes which k-block and how often a stage's barriers
// are arrived at.  Plain numbers, so that a host program can walk through the orders in which the warps may run.
#pragma once

namespace fi {

constexpr int kDequantWarps = 8;       // two halves of four warps; a warp owns 32 of the 128 weight rows
constexpr int kRowBlocks = 4;          // k-blocks of 64 per raw stage in this form

// The k-block of a raw stage that a half of the warps writes in its turn u (0, 1).  The halves take the k-blocks in turn (even,
// odd): a warp then comes back to an A stage at most a_stages + 2 k-blocks after the last one it knows to be read, and the parity
// of the stage's barrier tells that apart from a stage one round older for any number of stages from 2 on.  Two neighbouring
// k-blocks per half would skip two, and with two stages a warp that ran ahead could take an unread stage for a free one.
constexpr int row_block(int u, int half) { return u * 2 + half; }

constexpr int a_stages(bool gated) { return gated ? 2 : 3; }

// Arrivals that fill an A stage: one per warp that writes the k-block, all eight in the form of half k-blocks.
constexpr int a_full_arrivals(bool row) { return row ? kDequantWarps / 2 : kDequantWarps; }

}  // namespace fi
