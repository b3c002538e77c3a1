// Base-2 strong probable-prime tests of many numbers of one size on the tensor
// cores (pg_rns.cu): residue number system, Montgomery reduction with both base
// extensions as matrix products shared by every number.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pg {

constexpr uint32_t kRnsDumps = 12;      // last values kept for the strong test's verdict
constexpr uint32_t kRnsTile = 256;      // numbers of a tile, half in each CTA of a pair
constexpr uint32_t kRnsGroup = 4;       // most tiles that a pair takes in turn
constexpr uint32_t kRnsSpread = 22;     // numbers this many bits narrower than the widest are taken with it

struct PrpItem {
    uint32_t row;  // row of the base numbers
    int32_t x;     // N = base[row] + x
};

// Chunks of residue slots that numbers below 2^bits take; 0: too wide.
uint32_t rns_chunks(uint32_t bits);

// Numbers that run at once in one wave, of single tiles or of full groups of
// tiles (0 where rns_chunks is 0 and full is asked).
uint64_t rns_wave(uint32_t bits, bool full);

// Microseconds that rns_test takes, over slices of a long list.
double rns_us(uint32_t bits, uint64_t items);

// How many of `left` numbers the next rns_test of a long list takes: one wave.
uint64_t rns_slice(uint32_t bits, uint64_t left);

// Device workspace of rns_test over at most max_items numbers at a time, all_items
// in all.
struct RnsLayout {
    uint32_t chunks, limbs;
    uint64_t tiles;  // of kRnsTile numbers
    size_t matrices, num_a, num_b, state, dumps, nums, quot, flag, factor, list, counters, total;
};
RnsLayout rns_layout(uint32_t bits, uint32_t limbs, uint64_t max_items, uint64_t all_items);

// Tests items[first .. first + min(*count, max_items)) (count == nullptr: max_items)
// and writes their results; numbers that this form does not decide (how many since
// first = 0 at rns_fallback_count, their places at rns_fallback_list) are left for
// the caller.
cudaError_t rns_begin(const RnsLayout &l, uint32_t bits, void *work, cudaStream_t s);
cudaError_t rns_test(const RnsLayout &l, uint32_t bits, void *work, const uint32_t *bases, const PrpItem *items,
                     uint64_t first, const unsigned long long *count, uint64_t max_items, uint8_t *result,
                     cudaStream_t s);
inline const unsigned long long *rns_fallback_count(const RnsLayout &l, void *work) {
    return (const unsigned long long *)((char *)work + l.counters);
}
inline const uint32_t *rns_fallback_list(const RnsLayout &l, void *work) {
    return (const uint32_t *)((char *)work + l.list);
}
// Set by a wait that gave up.
inline const unsigned long long *rns_error(const RnsLayout &l, void *work) {
    return (const unsigned long long *)((char *)work + l.counters) + 1;
}

}  // namespace pg
