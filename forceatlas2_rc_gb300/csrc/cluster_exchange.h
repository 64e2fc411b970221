// cluster_exchange.h -- which mbarrier a pass of the cluster sort counts its
// digit counts on (k_codes_sort). Plain C++: the host model of the exchange
// compiles it too.
#pragma once

#ifdef __CUDACC__
#define CS_HD __host__ __device__
#else
#define CS_HD
#endif

namespace fa2cu {

// Barriers of the counts, taken in turn by the passes. One is not enough: a
// block that holds a pass's counts from all others may have sent the next
// pass's before the same counts are at every other block, and there they would
// fill the phase in their place.
#ifndef CS_COUNT_BARS
#define CS_COUNT_BARS 2
#endif
CS_HD constexpr int cs_count_bar(int pass) { return pass % CS_COUNT_BARS; }
CS_HD constexpr unsigned cs_count_parity(int pass) { return pass / CS_COUNT_BARS & 1; }

} // namespace fa2cu
