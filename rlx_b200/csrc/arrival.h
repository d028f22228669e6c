// Words in which the contributors of a tile count themselves in, in scratch that nobody clears first: the caller's workspace
// holds whatever the call before left there (f32 sums of another shape, as a rule).  A word is {tag of the call : 48 bits,
// count : 16 bits}, and any other upper 48 bits read as a count of zero.  48 bits, because with 32 one stray f32 value in the
// upper half of a word was enough to be taken for a count; two neighbouring values would have to agree with the tag now.
// Plain C++ as well as device code.
#pragma once

#ifdef __CUDACC__
#define RLXQ_BOTH __host__ __device__ __forceinline__
#else
#define RLXQ_BOTH inline
#endif

namespace rlxq {

constexpr int kArrivalCountBits = 16;                    // contributors are CTAs, one per SM at most
constexpr unsigned long long kArrivalTagMask = (1ull << (64 - kArrivalCountBits)) - 1;

// The n-th call's tag: odd, so never zero, and different from those of the calls that may be in flight beside it.
RLXQ_BOTH unsigned long long arrival_tag(unsigned long long n) { return ((n << 1) | 1ull) & kArrivalTagMask; }
RLXQ_BOTH unsigned long long arrival_word(unsigned long long tag, unsigned count) { return (tag << kArrivalCountBits) | count; }
// How many have arrived in the call `tag`, going by the word.
RLXQ_BOTH unsigned arrival_count(unsigned long long word, unsigned long long tag) {
    return word >> kArrivalCountBits == tag ? (unsigned)(word & ((1u << kArrivalCountBits) - 1u)) : 0u;
}

}  // namespace rlxq
