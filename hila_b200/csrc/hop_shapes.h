// Launch shapes of the FP64 hop and the sizes of its grid reductions (no CUDA types: a CPU test
// checks the arithmetic).
#pragma once

#include <stddef.h>

namespace hw {

constexpr int kHopBlock = 128;
constexpr int kHopVariants = 4;  // 0..2 timed per lattice, 3 for small lattices (dslash_f64.cu)
constexpr int kSplitSites = 32;  // sites of a block of shape 3: one per lane
// Sites per parity up to which the hop runs eight warps per 32 sites (k_hop_split): an FP64 CG
// iteration took 40 -> 30 us at 8^4, 43 -> 39 us at 6x10x14x22 (9240), 43 -> 44 us at 12^4
// (10368), 52 -> 65 us at 16^4.  From 20^4 on the CG gains a little from it (142 -> 136 us, 24^4
// 282 -> 273) and the apply loses (49 -> 58, 103 -> 118).
constexpr int kHopSplitSites = 9500;

// sites that one block of a launch shape serves
constexpr int hop_sites(int variant) { return variant == 3 ? kSplitSites : variant == 2 ? 256 : kHopBlock; }
constexpr long hop_blocks(int variant, long Vh) { return (Vh + hop_sites(variant) - 1) / hop_sites(variant); }

// Doubles reserved for the partial sums of a reduction over nblocks blocks
constexpr int kRedValues = 4;  // most values that a kernel sums
constexpr size_t red_doubles(long nblocks) { return (size_t)kRedValues * (nblocks + 1); }

}  // namespace hw
