// gg_cluster_addr.h -- shared-memory addresses of 8-byte words in a cluster, marked where they
// belong to another CTA.
//
// The mark is bit 0: an 8-byte word's address has its low three bits clear wherever the
// hardware puts the cluster window, so no value of an address is taken for a mark.  Offsets
// that are multiples of 8 may be added to a marked address.
#pragma once

#ifdef __CUDACC__
#define GG_HD __host__ __device__ __forceinline__
#else
#define GG_HD inline
#endif

namespace gg {

constexpr unsigned kRemoteBit = 1u;
constexpr unsigned kNoAddr = 0xffffffffu;  // no word: not 8-byte aligned under the mark either

constexpr GG_HD unsigned mark_remote(unsigned a) { return a | kRemoteBit; }
constexpr GG_HD bool is_remote(unsigned a) { return (a & kRemoteBit) != 0u; }
constexpr GG_HD unsigned unmarked(unsigned a) { return a & ~kRemoteBit; }

}  // namespace gg
