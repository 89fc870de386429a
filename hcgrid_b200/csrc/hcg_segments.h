// Accumulation segments of the tensor-core kernels (host and device).
//
// The tensor cores' FP32 accumulation drops low bits of the products it adds
// (the sums come out low by up to ~2^-24 of the running sum per MMA), so long K
// loops drift. An item of more than kTcWholeSlots staged slots is accumulated in
// equal segments of kTcSegSlots at most (up to a chunk), each in a fresh
// accumulator (the two TMEM halves in turn), and the epilogue adds the segments
// with round-to-nearest FP32 adds (in the cube buffer) before it normalises them.
// What drifts is the slots with weight: the closer the staged list fits the beam,
// the shorter a segment must be. 150,000 samples, beam 54 pixels wide: the cube's
// mean came out low by 6.5e-6 in segments of 1,024 of the 5,090 slots a tile,
// 5.7e-6 when a tile staged 5,930 for the same pairs, and by 5.6e-6 in these
// (4.9e-6 in segments of 896, which give many cubes a segment more: 144 channels on
// 579 x 479 pixels 1.33 against 1.29 ms).
#pragma once

#include "hcg_math.cuh"

namespace hcg {

constexpr uint32_t kTcSegSlots = 992, kTcWholeSlots = 1344;
// The one-item kernel (k_tile_tc) accumulates an item in one segment: it takes
// tiles of at most this many staged slots (longer ones go to the persistent
// kernels, and jobs that hold one leave a batch, whose kernel could take them in
// segments as well).
constexpr uint32_t kTcOneSegmentSlots = 1536;

// segments of an item of `nchunks` chunks of `kc` slots, and the end of segment q
HCG_HD uint32_t tc_segments(uint32_t kc, uint32_t nchunks) {
    const uint64_t slots = (uint64_t)nchunks * kc;
    return slots > kTcWholeSlots ? (uint32_t)((slots + kTcSegSlots - 1) / kTcSegSlots) : 1;
}
HCG_HD uint32_t tc_segment_end(uint32_t nchunks, uint32_t nseg, uint32_t q) {
    return (uint32_t)((uint64_t)nchunks * (q + 1) / nseg);
}

}  // namespace hcg
