// How many CTAs and clusters of two a persistent grid takes beside an SM margin. Plain C++, so that it can be checked without a GPU.
#pragma once

namespace pcb {

// SMs beside a margin of `margin`: never fewer than two.
inline int sms_beside(int sms, int margin) { return sms - margin < 2 ? 2 : sms - margin; }

// Clusters of two CTAs that fill whole SMs. A cluster takes both SMs of a TPC, and the CTAs that the margin is for need not share theirs: started while a
// staging kernel runs, two of them lay on two TPCs in 35 of 40 calls, and a grid of 73 pairs found 72 places, which cost a second round. 3x3, 64 channels,
// 56 x 56, batch 128, channels-last, both gradients with two SMs taken behind the first: 862 us with 73 pairs, 641 with 72 (608 alone).
inline int pairs_beside(int sms, int margin) { return sms / 2 - margin < 1 ? 1 : sms / 2 - margin; }

}  // namespace pcb
