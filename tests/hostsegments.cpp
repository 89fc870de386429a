// Host build of the tensor-core kernels' segment rule.
#include "hcg_segments.h"

extern "C" unsigned hs_segments(unsigned kc, unsigned nchunks) { return hcg::tc_segments(kc, nchunks); }
extern "C" unsigned hs_end(unsigned nchunks, unsigned nseg, unsigned q) { return hcg::tc_segment_end(nchunks, nseg, q); }
