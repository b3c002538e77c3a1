// Probable-prime tests of N = m*K +- X on the device, and the prime-gap search
// over a job's unknown lists that they serve.
//
// Replaces the reference's GPU Miller-Rabin (kernel_miller_rabin,
// miller_rabin_t::miller_rabin and powm, miller_rabin.h:154-267: CGBN, eight
// threads per number) with the one base gap_test_gpu uses (ROUNDS = 1 with
// primes {2}, gap_test_gpu.cu:81, miller_rabin.h:269), and its host threads
// (load_batch_thread, run_gpu_thread, run_overflow_thread,
// gap_test_gpu.cu:213-640) with device rounds.
//
// Numbers wide and many enough are tested in a residue number system on the
// tensor cores (pg_rns.cu); the limb arithmetic here takes the others, and the
// few that the residue form leaves.
//
// Numbers: n = 8L little-endian 32-bit limbs over a group of 8 lanes of a
// warp, lane t holding limbs [tL, tL + L).  N < 2^(32n - 4), so R = 2^(32n) is
// at least 16N and Montgomery products of inputs below 4N stay below 2N: 2^d
// (N - 1 = d 2^s) by left-to-right squaring with a doubling (a one-bit shift)
// on each set bit of d needs no conditional subtraction.  Base 2 makes every
// multiplication of the exponentiation a shift.
//
// Montgomery product, CIOS word by word: each lane runs its L-limb
// multiply-add chains; the carry out of its top limb waits in a pending word
// until the one-limb shift of the step brings the next lane's bottom limb down
// beside it, so a step exchanges three words between lanes (the multiplier
// word, the quotient word, the shifted limb) and no carry crosses lanes until
// the end of the product, where one ballot resolves them all.
//
// The strong test follows miller_rabin.h:211-245, including its loop bound:
// after x = 2^d, up to s squarings (one more than the textbook s - 1).  The
// extra squaring never changes a verdict (2^(N-1) = -1 mod N has no odd
// solution N > 1).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "pg_arith.cuh"
#include "pg_host.h"
#include "pg_rns.h"

namespace pg {

namespace {

constexpr int kTPI = 8;                       // lanes per number
constexpr int kPrpThreads = 128;              // 16 numbers per block
constexpr int kGroups = kPrpThreads / kTPI;
constexpr int kMaxL = 16;                     // up to 8*16*32 - 4 = 4092-bit numbers

template <int L>
struct Num {
    uint32_t v[L];
};

struct Grp {
    uint32_t mask;  // the group's lanes in the warp
    uint32_t base;  // its first lane
    uint32_t t;     // this lane within the group
};

__device__ __forceinline__ Grp group_of_lane() {
    const uint32_t lane = threadIdx.x & 31u;
    Grp g;
    g.t = lane & (kTPI - 1);
    g.base = lane - g.t;
    g.mask = ((1u << kTPI) - 1u) << g.base;
    return g;
}

__device__ __forceinline__ uint32_t gballot(const Grp &g, bool p) {
    return (__ballot_sync(g.mask, p) >> g.base) & ((1u << kTPI) - 1u);
}

// Carries between lanes from each lane's carry out (gen) and whether it would
// pass an incoming carry on (prop): bit t = carry into lane t, bit kTPI =
// carry out of the top lane.  Same rule for borrows.
__device__ __forceinline__ uint32_t lane_carries(uint32_t gen, uint32_t prop) {
    return ((gen << 1) + prop) ^ prop;
}

template <int L>
__device__ __forceinline__ uint32_t add_lane(Num<L> &a, uint32_t c) {
#pragma unroll
    for (int k = 0; k < L; k++) {
        const uint64_t s = (uint64_t)a.v[k] + c;
        a.v[k] = (uint32_t)s;
        c = (uint32_t)(s >> 32);
    }
    return c;
}

template <int L>
__device__ __forceinline__ uint32_t sub_lane(Num<L> &a, uint32_t b) {
#pragma unroll
    for (int k = 0; k < L; k++) {
        const uint64_t s = (uint64_t)a.v[k] - b;
        a.v[k] = (uint32_t)s;
        b = (uint32_t)(s >> 63);
    }
    return b;
}

template <int L>
__device__ __forceinline__ bool all_limbs(const Num<L> &a, uint32_t w) {
    bool r = true;
#pragma unroll
    for (int k = 0; k < L; k++) r &= a.v[k] == w;
    return r;
}

// a += x, x at limb 0
template <int L>
__device__ __forceinline__ void add_small(const Grp &g, Num<L> &a, uint32_t x) {
    const uint32_t co = add_lane(a, g.t == 0 ? x : 0u);
    const uint32_t cin = lane_carries(gballot(g, co != 0), gballot(g, all_limbs(a, 0xFFFFFFFFu)));
    add_lane(a, (cin >> g.t) & 1u);
}

// a -= x, x at limb 0, a >= x
template <int L>
__device__ __forceinline__ void sub_small(const Grp &g, Num<L> &a, uint32_t x) {
    const uint32_t bo = sub_lane(a, g.t == 0 ? x : 0u);
    const uint32_t bin = lane_carries(gballot(g, bo != 0), gballot(g, all_limbs(a, 0u)));
    sub_lane(a, (bin >> g.t) & 1u);
}

// a -= n when a >= n (a < 2n)
template <int L>
__device__ __forceinline__ void reduce_once(const Grp &g, Num<L> &a, const Num<L> &n) {
    Num<L> d;
    uint32_t br = 0;
#pragma unroll
    for (int k = 0; k < L; k++) {
        const uint64_t s = (uint64_t)a.v[k] - n.v[k] - br;
        d.v[k] = (uint32_t)s;
        br = (uint32_t)(s >> 63);
    }
    const uint32_t bin = lane_carries(gballot(g, br != 0), gballot(g, all_limbs(d, 0u)));
    sub_lane(d, (bin >> g.t) & 1u);
    if (!((bin >> kTPI) & 1u)) a = d;  // no borrow out of the top: a >= n
}

// a <<= bit (bit 0 or 1)
template <int L>
__device__ __forceinline__ void shl(const Grp &g, Num<L> &a, uint32_t bit) {
    uint32_t in = __shfl_up_sync(g.mask, a.v[L - 1], 1, kTPI);
    if (g.t == 0) in = 0;
#pragma unroll
    for (int k = L - 1; k > 0; k--) a.v[k] = __funnelshift_l(a.v[k - 1], a.v[k], bit);
    a.v[0] = __funnelshift_l(in, a.v[0], bit);
}

// out = x * y / R mod n (below 2n for x, y below 4n), y = x or one (y_one).
template <int L>
__device__ __forceinline__ void mont_mul(const Grp &g, Num<L> &out, const Num<L> &x, bool y_one,
                                         const Num<L> &n, uint32_t ninv) {
    Num<L> y, a;
#pragma unroll
    for (int k = 0; k < L; k++) {
        y.v[k] = y_one ? (g.t == 0 && k == 0 ? 1u : 0u) : x.v[k];
        a.v[k] = 0;
    }
    uint64_t e = 0;  // carries pending into the next lane's bottom limb
    const bool top = g.t == kTPI - 1;
    for (uint32_t src = 0; src < kTPI; src++) {
#pragma unroll
        for (int k = 0; k < L; k++) {
            const uint32_t xi = __shfl_sync(g.mask, x.v[k], src, kTPI);
            uint32_t c = 0;
#pragma unroll
            for (int j = 0; j < L; j++) {
                const uint64_t s = (uint64_t)xi * y.v[j] + a.v[j] + c;
                a.v[j] = (uint32_t)s;
                c = (uint32_t)(s >> 32);
            }
            e += c;
            // lane 0's bottom limb has nothing pending: the quotient word
            const uint32_t q = __shfl_sync(g.mask, a.v[0] * ninv, 0, kTPI);
            c = 0;
#pragma unroll
            for (int j = 0; j < L; j++) {
                const uint64_t s = (uint64_t)q * n.v[j] + a.v[j] + c;
                a.v[j] = (uint32_t)s;
                c = (uint32_t)(s >> 32);
            }
            e += c;
            // shift down one limb; lane 0's bottom limb (zero) drops out
            uint32_t in = __shfl_down_sync(g.mask, a.v[0], 1, kTPI);
            if (top) in = 0;
#pragma unroll
            for (int j = 0; j + 1 < L; j++) a.v[j] = a.v[j + 1];
            const uint64_t s = (uint64_t)in + e;
            a.v[L - 1] = (uint32_t)s;
            e = s >> 32;
        }
    }
    // resolve the pending carries (the value is below R: none leaves the top)
    uint32_t in = __shfl_up_sync(g.mask, (uint32_t)e, 1, kTPI);
    if (g.t == 0) in = 0;
    const uint32_t co = add_lane(a, in);
    const uint32_t cin = lane_carries(gballot(g, co != 0), gballot(g, all_limbs(a, 0xFFFFFFFFu)));
    add_lane(a, (cin >> g.t) & 1u);
    out = a;
}

template <int L>
__device__ __forceinline__ bool equals_small(const Grp &g, const Num<L> &a, uint32_t w) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < L; k++) ok &= a.v[k] == (g.t == 0 && k == 0 ? w : 0u);
    return gballot(g, ok) == (1u << kTPI) - 1u;
}

template <int L>
__device__ __forceinline__ bool equals_n_minus_1(const Grp &g, const Num<L> &a, const Num<L> &n) {
    bool ok = true;
#pragma unroll
    for (int k = 0; k < L; k++) ok &= a.v[k] == n.v[k] - (g.t == 0 && k == 0 ? 1u : 0u);
    return gballot(g, ok) == (1u << kTPI) - 1u;
}

template <int L>
__device__ __forceinline__ uint32_t bit_length(const Grp &g, const Num<L> &a) {
    int hi = -1;
    uint32_t w = 0;
#pragma unroll
    for (int k = 0; k < L; k++)
        if (a.v[k]) hi = k, w = a.v[k];
    const uint32_t lanes = gballot(g, hi >= 0);
    if (!lanes) return 0;
    const uint32_t top = 31 - __clz(lanes);
    const uint32_t word = __shfl_sync(g.mask, w, top, kTPI);
    const int idx = __shfl_sync(g.mask, hi, top, kTPI);
    return 32u * (top * L + (uint32_t)idx) + (32u - __clz(word));
}

// Base-2 strong probable-prime test of odd n (5 <= n < 2^(32*8L - 4)); sn =
// the group's copy of n's limbs in shared memory (exponent bits).
template <int L>
__device__ bool prp2(const Grp &g, const Num<L> &n, const uint32_t *sn) {
    const uint32_t b = bit_length(g, n);
    uint32_t s = 0;  // trailing zeros of n - 1
    for (uint32_t w = 0; w < 8u * L; w++) {
        const uint32_t v = sn[w] - (w == 0 ? 1u : 0u);
        if (v) {
            s = 32u * w + (uint32_t)__ffs(v) - 1u;
            break;
        }
    }
    const uint32_t ninv = __shfl_sync(g.mask, neg_inv32(n.v[0]), 0, kTPI);
    // x = 2R mod n, the Montgomery form of 2 (the leading bit of d): 2^(b-1)
    // doubled 32n - b + 2 times, reduced after each doubling
    Num<L> x;
    const uint32_t top_limb = (b - 1) >> 5;
#pragma unroll
    for (int k = 0; k < L; k++) x.v[k] = (g.t * L + k == top_limb) ? (1u << ((b - 1) & 31)) : 0u;
    const uint32_t doublings = 32u * 8u * L - b + 2u;
    for (uint32_t i = 0; i < doublings; i++) {
        shl(g, x, 1u);
        reduce_once(g, x, n);
    }
    // One Montgomery product per step: squarings of the exponent (bits b-2 ..
    // s of n are the bits of d below its leading one), then alternately a
    // conversion y = x/R (the value) and a squaring, per miller_rabin.h:222-243.
    int p = (int)b - 2;
    bool convert = p < (int)s;
    bool first_check = true;
    uint32_t count = s;
    for (;;) {
        Num<L> r;
        mont_mul(g, r, x, convert, n, ninv);
        if (!convert) {
            x = r;
            if (p >= (int)s) {
                const uint32_t bit = (sn[p >> 5] >> (p & 31)) & 1u;
                shl(g, x, bit);
                p--;
                convert = p < (int)s;
            } else {
                convert = true;  // a squaring of the strong loop: check it next
            }
            continue;
        }
        reduce_once(g, r, n);  // the value, below n
        convert = false;
        if (first_check) {
            if (equals_small(g, r, 1u) || equals_n_minus_1(g, r, n)) return true;
            if (s == 1) return false;
            first_check = false;
            continue;
        }
        if (equals_n_minus_1(g, r, n)) return true;
        if (--count == 0 || equals_small(g, r, 1u)) return false;
    }
}

// kListed: the items to test are the listed ones, if there is a list.  Its own instance:
// the branch costs some widths up to 11 % (16 numbers of 1463 bits 6.57 ms without it,
// 7.03 with it; 1788 bits 10.5, 11.6).  At three limbs per lane the instance with it is
// the faster one (735 bits 1.65, 1.50) and takes all calls.
template <int L, bool kListed>
__global__ void __launch_bounds__(kPrpThreads)
    prp_kernel(const uint32_t *__restrict__ bases, const PrpItem *__restrict__ items,
               const uint32_t *__restrict__ list, const unsigned long long *count, uint64_t max_items, uint8_t *__restrict__ result) {
    __shared__ uint32_t s_n[kGroups][8 * L];
    const Grp g = group_of_lane();
    const uint32_t gi = threadIdx.x / kTPI;
    uint64_t i = (uint64_t)blockIdx.x * kGroups + gi;
    const uint64_t n_items = count ? min((uint64_t)*count, max_items) : max_items;
    if (i >= n_items) return;  // the whole group leaves together
    if (kListed && list) i = list[i];
    const PrpItem it = items[i];
    const uint32_t *src = bases + (uint64_t)it.row * (8 * L) + g.t * L;
    Num<L> n;
#pragma unroll
    for (int k = 0; k < L; k++) n.v[k] = src[k];
    if (it.x > 0) add_small(g, n, (uint32_t)it.x);
    if (it.x < 0) sub_small(g, n, (uint32_t)(-(int64_t)it.x));
#pragma unroll
    for (int k = 0; k < L; k++) s_n[gi][g.t * L + k] = n.v[k];
    __syncwarp(g.mask);
    const bool r = prp2<L>(g, n, s_n[gi]);
    if (g.t == 0) result[i] = r ? 1 : 0;
}

cudaError_t launch_prp(int L, const uint32_t *bases, const PrpItem *items, const uint32_t *list,
                       const unsigned long long *count, uint64_t max_items, uint8_t *result, cudaStream_t s) {
    if (max_items == 0) return cudaSuccess;
    const unsigned blocks = (unsigned)((max_items + kGroups - 1) / kGroups);
#define PG_PRP_CASE(LL)                                                                                       \
    case LL:                                                                                                  \
        if (list || LL == 3)                                                                                  \
            prp_kernel<LL, true><<<blocks, kPrpThreads, 0, s>>>(bases, items, list, count, max_items, result); \
        else                                                                                                  \
            prp_kernel<LL, LL == 3><<<blocks, kPrpThreads, 0, s>>>(bases, items, list, count, max_items, result); \
        break;
    switch (L) {
        PG_PRP_CASE(1)
        PG_PRP_CASE(2)
        PG_PRP_CASE(3)
        PG_PRP_CASE(4)
        PG_PRP_CASE(5)
        PG_PRP_CASE(6)
        PG_PRP_CASE(7)
        PG_PRP_CASE(8)
        PG_PRP_CASE(9)
        PG_PRP_CASE(10)
        PG_PRP_CASE(11)
        PG_PRP_CASE(12)
        PG_PRP_CASE(13)
        PG_PRP_CASE(14)
        PG_PRP_CASE(15)
        PG_PRP_CASE(16)
        default:
            return cudaErrorInvalidValue;
    }
#undef PG_PRP_CASE
    return cudaGetLastError();
}

// Limbs per lane for numbers of `bits` bits: 32*8L >= bits + 4.
int limbs_per_lane(uint32_t bits) { return (int)((bits + 4 + 255) / 256); }

// How a call's numbers are tested: on the tensor cores where their width allows
// it (pg_rns.cu) with what is left over tested limb by limb, or limb by limb.
struct PrpPlan {
    int L = 0;
    uint32_t bits = 0;
    bool rns = false;
    RnsLayout layout{};
};

// Where the residue form is the faster one: from so many numbers of one width on.
// Whole calls in ms (limbs, residues) at the widths where a step up of one form's time
// comes before the other's, elsewhere the residue form is ahead from one number on:
//   253-360 bits, a chunk: 300 bits, one number 0.32, 0.39; two 0.40, 0.39
//   361-508, two chunks and two limbs per lane: 430 bits, 9728 numbers (four blocks on
//     each SM) 0.97, 1.03; 9729 1.14, 1.03; 19456 1.75, 1.15; 24320 (a wave and a
//     quarter of single tiles) 2.11, 2.11, 26752 2.29, 2.11
//   509-735, two and three: 735 bits, two 1.30, 1.45; four 1.49, 1.45
//   736-764, three and three: 764 bits, 4864 (two blocks) 1.87, 1.98; 5000 2.20, 1.99
//   1104-1276, four and five: 1276 bits, one 4.44, 4.53; two 4.65, 4.53
//   1464-1532, five and six: 1464 bits, two 6.18, 6.26; four 6.57, 6.27
// and the others: 765 bits, one 1.97, 1.87; 1100 bits 3.83, 2.67; 2136 bits 15.0, 11.0;
// 2838 bits 52.4, 24.7; 200 bits 0.20, 0.32.
bool rns_pays(uint32_t bits, uint64_t items) {
    const uint32_t n = rns_chunks(bits);
    if (bits < 253 || n == 0) return false;
    const int L = limbs_per_lane(bits);
    const uint64_t wave = rns_wave(bits, false);
    switch (16 * n + (uint32_t)L) {
        case 16 * 1 + 2: return items >= 2;
        case 16 * 2 + 2: return items > wave / 2 && !(items > wave && items <= 5 * wave / 4);
        case 16 * 2 + 3: return items >= 4;
        case 16 * 3 + 3: return items > wave / 4;
        case 16 * 4 + 5: return items >= 2;
        case 16 * 5 + 6: return items >= 4;
        default: return true;
    }
}

PrpPlan limb_plan(uint32_t bits) {
    PrpPlan p;
    p.bits = bits;
    p.L = limbs_per_lane(bits);
    return p;
}

// The residue form's workspace, some 6 KB per number of 2136 bits, is for a wave of
// numbers: a longer list goes through it in slices.
PrpPlan prp_plan(uint32_t bits, uint64_t max_items) {
    PrpPlan p = limb_plan(bits);
    p.rns = rns_pays(bits, max_items);
    if (p.rns) p.layout = rns_layout(bits, 8u * (uint32_t)p.L, rns_slice(bits, max_items), max_items);
    return p;
}

// Numbers of one block on each SM.
uint64_t limb_layer() { return rns_wave(0, false) * kGroups / kRnsTile * 2; }

// The limb form at the limbs per lane of `bits`: microseconds per bit of a chain of
// squarings (16 numbers), nanoseconds per bit of each of many numbers (4864 to 38912;
// above 3068 bits put low).
double limb_step_us(uint32_t bits) {
    constexpr double kStep[kMaxL + 1] = {0,   0.5, 1.3,  1.95, 2.87, 3.82, 4.4,  5.83, 7.6,
                                         7.4, 8.6, 10.3, 18.9, 14,   15.6, 19.3, 20.4};
    return kStep[limbs_per_lane(bits)];
}
double limb_bit_ns(uint32_t bits) {
    constexpr double kNs[kMaxL + 1] = {0, 0.1, 0.17, 0.31, 0.5, 0.76, 1.04, 1.45, 1.74, 2.4, 2.95, 2.95, 2.95, 4, 5, 5, 5};
    return kNs[limbs_per_lane(bits)];
}
// ... and of a launch over numbers up to `bits` wide whose widths add up to `sum`: one
// block of 16 numbers on each SM after another.
double limb_us(uint32_t bits, double sum) {
    const double layer = (double)limb_layer() * bits;
    return std::max(bits * limb_step_us(bits), 1e-3 * std::ceil(sum / layer) * layer * limb_bit_ns(bits));
}

// Numbers that are tested with one plan: `count` of the call's order from `first` on.
struct PrpPart {
    uint64_t first, count;
    PrpPlan plan;
};

// The parts of a list of numbers of these widths, `lo` to `hi`, that spread over more than
// kRnsSpread; `order` becomes the order in which they are tested, where it is not the
// list's.  The residue form, which takes numbers of nearly one width, gets the bands of
// kRnsSpread bits whose many numbers are worth a wave of their own, with or without the
// widest numbers' band; one launch of the limb form takes the rest, at the rest's own
// width; or the limb form takes all, where that is the fastest.  (All through the residue
// form at the widest number's width and what it left through the limb form as well, the
// limb form for all, and in parts, in ms: 15 numbers of 2136 bits and one of 2161 29.0,
// 16.1, 16.1; 2000 of 300 to 2800 bits 53, 29, 29; 9000 of 2838 and one of 2863 132, 106,
// 51; 9000 of 2136 and 9000 of 1400 51, 78, 17.)
std::vector<PrpPart> prp_parts(const std::vector<uint16_t> &width, uint32_t lo, uint32_t hi,
                               std::vector<uint64_t> &order) {
    const uint64_t n = width.size();
    // numbers of each width below w, and the sum of their widths
    std::vector<uint64_t> below(hi + 2, 0), sum(hi + 2, 0);
    for (uint32_t w : width) below[w + 1]++;
    for (uint32_t w = 0; w <= hi; w++) {
        sum[w + 1] = sum[w] + below[w + 1] * w;
        below[w + 1] += below[w];
    }
    std::vector<PrpPart> best{{0, n, limb_plan(hi)}};
    std::vector<uint32_t> best_of;  // a width's part
    double best_us = 0.95 * limb_us(hi, (double)sum[hi + 1]);
    for (const bool widest : {false, true}) {
        constexpr uint32_t kRest = ~0u;
        std::vector<PrpPart> parts;
        std::vector<uint32_t> of(hi + 1, kRest);
        double us = 0, rest_sum = 0;
        uint32_t rest_bits = 0;
        for (uint32_t w = hi; w >= lo;) {
            const uint32_t from = std::max(lo, w - std::min(w, kRnsSpread));
            const uint64_t here = below[w + 1] - below[w], count = below[w + 1] - below[from];
            if (here && rns_pays(w, count) &&
                ((widest && w == hi) || rns_us(w, count) < 1e-3 * (double)(sum[w + 1] - sum[from]) * limb_bit_ns(w))) {
                std::fill(of.begin() + from, of.begin() + w + 1, (uint32_t)parts.size());
                parts.push_back({0, count, prp_plan(w, count)});
                us += rns_us(w, count);
                w = from;
            } else if (here) {
                rest_bits = std::max(rest_bits, w);
                rest_sum += (double)here * w;
            }
            w--;
        }
        if (rest_bits) {
            uint64_t count = n;
            for (const PrpPart &p : parts) count -= p.count;
            us += limb_us(rest_bits, rest_sum);
            std::replace(of.begin(), of.end(), kRest, (uint32_t)parts.size());
            parts.push_back({0, count, limb_plan(rest_bits)});
        }
        if (us < best_us && parts.size() > 1) best_us = us, best = parts, best_of = of;
    }
    if (best.size() == 1) return best;
    order.resize(n);
    std::vector<uint64_t> at(best.size());
    for (size_t i = 1; i < best.size(); i++) best[i].first = best[i - 1].first + best[i - 1].count;
    for (size_t i = 0; i < best.size(); i++) at[i] = best[i].first;
    for (uint64_t i = 0; i < n; i++) order[at[best_of[width[i]]]++] = i;
    return best;
}

// The residue form's workspace; false where the device has no room for it: then the
// limb form takes the call.
bool prp_workspace(pgh::DevBuf &work, size_t bytes, cudaError_t &e) {
    e = work.ensure(bytes);
    if (e != cudaErrorMemoryAllocation) return true;
    e = cudaSuccess;
    cudaGetLastError();
    return false;
}

cudaError_t prp_begin(const PrpPlan &p, void *work, cudaStream_t s) {
    return p.rns ? rns_begin(p.layout, p.bits, work, s) : cudaSuccess;
}

cudaError_t prp_launch(const PrpPlan &p, void *work, const uint32_t *bases, const PrpItem *items,
                       const unsigned long long *count, uint64_t max_items, uint8_t *result, cudaStream_t s) {
    if (!p.rns) return launch_prp(p.L, bases, items, nullptr, count, max_items, result, s);
    for (uint64_t first = 0; first < max_items;) {  // a count: one slice, at most a wave
        const uint64_t n = count ? max_items : rns_slice(p.bits, max_items - first);
        const cudaError_t e = rns_test(p.layout, p.bits, work, bases, items, first, count, n, result, s);
        if (e != cudaSuccess) return e;
        first += n;
    }
    return launch_prp(p.L, bases, items, rns_fallback_list(p.layout, work), rns_fallback_count(p.layout, work),
                      max_items, result, s);
}

// *error (host) = nonzero after a wait on the device that gave up
cudaError_t prp_error(const PrpPlan &p, void *work, unsigned long long *error, cudaStream_t s) {
    *error = 0;
    return p.rns ? cudaMemcpyAsync(error, rns_error(p.layout, work), sizeof(*error), cudaMemcpyDeviceToHost, s)
                 : cudaSuccess;
}

// ---------------------------------------------------------------------------
// gap search

// centers[r] = m[r] * K as n limbs (one thread per row)
__global__ void centers_kernel(const uint32_t *__restrict__ k, uint32_t nk, const uint64_t *__restrict__ m,
                               uint64_t rows, uint32_t n, uint32_t *__restrict__ out) {
    const uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const uint64_t mm = m[r];
    const uint32_t lo = (uint32_t)mm, hi = (uint32_t)(mm >> 32);
    uint32_t *o = out + r * n;
    uint64_t c = 0;
    for (uint32_t j = 0; j < n; j++) {
        const uint64_t t = (uint64_t)lo * (j < nk ? k[j] : 0u) + c;
        o[j] = (uint32_t)t;
        c = t >> 32;
    }
    c = 0;
    for (uint32_t j = 1; j < n; j++) {
        const uint64_t t = (uint64_t)hi * (j - 1 < nk ? k[j - 1] : 0u) + o[j] + c;
        o[j] = (uint32_t)t;
        c = t >> 32;
    }
}

// One side of one m: the search for the nearest probable prime.  Both sides of
// an m are searched at once unless the next side may be skipped.
struct GapSearch {
    uint32_t state;      // kWaiting (for the previous side), kActive, kDone
    uint32_t idx;        // next unknown to test
    uint32_t past;       // 1 past the sieve length
    uint32_t past_x;     // next distance there (sl + 1 at first)
    uint32_t item_base, item_cnt;
    uint32_t item_list;  // the first of them that are unknowns, the others past the sieve length
};
enum { kWaiting, kActive, kDone };

struct GapLists {
    const uint64_t *start;
    const uint32_t *n_prev, *n_next, *dist;
};

// Distances past the sieve length that are coprime to K, a bit each from sl + 1 (for the
// residue form's rounds, which nearly all look at some).
constexpr uint32_t kPastBits = 1u << 17;

__device__ __forceinline__ bool coprime_to_k(uint32_t x, const uint32_t *kp, uint32_t nkp) {
    for (uint32_t i = 0; i < nkp; i++)
        if (x % kp[i] == 0) return false;
    return true;
}

__global__ void past_kernel(const uint32_t *kp, uint32_t nkp, uint32_t sl, uint32_t *__restrict__ bits) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kPastBits) return;
    const uint32_t w = __ballot_sync(0xFFFFFFFFu, coprime_to_k(sl + 1 + i, kp, nkp));
    if ((i & 31) == 0) bits[i >> 5] = w;
}

// A round's candidates, nearest first: spec for each active search and one more
// for the first `extra` that ask; past the sieve length, the next distances that keep N
// odd and coprime to K.  With go_on, a round goes on past the sieve length where the
// unknowns end (a round of the residue form is a whole wave: a search that ends there
// does not wait for another one).  Without, a search has its unknowns tested first: the
// limb form's time grows with the candidates (10 searches of 2503#/30030: 131 ms with 512
// each, 55 with 64).  A warp per search.
__global__ void select_kernel(GapSearch *searches, uint64_t rows, GapLists ls, const uint32_t *centers, uint32_t n,
                              uint32_t spec, uint32_t extra, bool go_on, const uint32_t *kp, uint32_t nkp,
                              const uint32_t *__restrict__ past_bits, uint32_t sl, uint32_t x_limit, PrpItem *items,
                              uint64_t max_items, unsigned long long *n_items, unsigned long long *asked,
                              unsigned long long *errors) {
    const uint64_t e = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (e >= 2 * rows) return;
    const uint32_t lane = threadIdx.x & 31;
    GapSearch st = searches[e];
    if (st.state != kActive) return;
    const uint64_t r = e >> 1;
    const bool next = e & 1;
    const int32_t sign = next ? 1 : -1;
    const uint32_t center_odd = centers[r * n] & 1u;
    uint32_t want = spec;
    if (extra) {
        uint32_t more = 0;
        if (lane == 0) more = atomicAdd(asked, 1ull) < extra;
        want += __shfl_sync(0xFFFFFFFFu, more, 0);
    }
    const uint32_t nlist = next ? ls.n_next[r] : ls.n_prev[r];
    if (!go_on && !st.past) want = min(want, nlist - st.idx);
    unsigned long long base = 0;
    if (lane == 0 && want) base = atomicAdd(n_items, (unsigned long long)want);
    base = __shfl_sync(0xFFFFFFFFu, base, 0);
    if (base + want > max_items) {  // the host sizes rounds so that this never happens
        if (lane == 0) atomicAdd(errors, 1ull);
        return;
    }
    uint32_t cnt = st.past ? 0u : min(want, nlist - st.idx);
    st.item_list = cnt;
    if (cnt) {
        const uint32_t *lst = ls.dist + ls.start[r] + (next ? ls.n_prev[r] : 0u) + st.idx;
        for (uint32_t j = lane; j < cnt; j += 32) items[base + j] = PrpItem{(uint32_t)r, sign * (int32_t)lst[j]};
    }
    if (cnt < want) {
        uint32_t x = st.past_x;
        while (cnt < want && x < x_limit) {
            // 1024 distances, 32 a lane (32 past the bitmap, one a lane): those
            // coprime to K, not before x, of the other parity than m*K
            const uint32_t at = x - (sl + 1);
            const bool table = past_bits && at < kPastBits;
            uint32_t from, word;
            if (table) {
                const uint32_t w = (at >> 5) + lane;
                from = sl + 1 + 32 * w;
                word = w < kPastBits / 32 ? past_bits[w] : 0u;
                if (lane == 0) word &= 0xFFFFFFFFu << (at & 31);
                word &= ((from & 1u) == center_odd) ? 0xAAAAAAAAu : 0x55555555u;
            } else {
                from = x + lane;
                word = from < x_limit && (from & 1u) != center_odd && coprime_to_k(from, kp, nkp);
            }
            const uint32_t mine = __popc(word);
            uint32_t before = mine;
            for (uint32_t o = 1; o < 32; o <<= 1) {
                const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, before, o);
                if (lane >= o) before += v;
            }
            const uint32_t all = __shfl_sync(0xFFFFFFFFu, before, 31);
            before -= mine;
            uint32_t k = cnt + before, last = 0;
            while (word && k < want) {
                const uint32_t bit = (uint32_t)__ffs(word) - 1;
                word &= word - 1;
                last = from + bit;
                items[base + k++] = PrpItem{(uint32_t)r, sign * (int32_t)last};
            }
            if (cnt + all >= want) {
                x = __reduce_max_sync(0xFFFFFFFFu, last) + 1;
                cnt = want;
            } else {
                cnt += all;
                x = table ? min(sl + 1 + kPastBits, sl + 1 + 32 * (at >> 5) + 1024u) : x + 32;
            }
        }
        if (cnt < want) {
            // no prime within the scan limit: report, stop the search; the slots
            // left over get a harmless odd number
            if (lane == 0) atomicAdd(errors, 1ull);
            for (uint32_t j = cnt + lane; j < want; j += 32) items[base + j] = PrpItem{(uint32_t)r, 1 + (int32_t)center_odd};
            st.state = kDone;
        }
        st.past_x = x;
    }
    st.item_base = (uint32_t)base;
    st.item_cnt = cnt;
    if (lane == 0) searches[e] = st;
}

// The round's results: a warp per search finds its first probable prime.
__global__ void resolve_kernel(GapSearch *searches, uint64_t rows, GapLists ls, const uint32_t *skip_below,
                               const PrpItem *items, const uint8_t *result, uint32_t sl, pgs_gap_result *out,
                               unsigned long long *active, unsigned long long *found) {
    const uint64_t e = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (e >= 2 * rows) return;
    const uint32_t lane = threadIdx.x & 31;
    GapSearch st = searches[e];
    if (st.state != kActive || st.item_cnt == 0) return;
    uint32_t first = 0xFFFFFFFFu;
    for (uint32_t j = 0; j < st.item_cnt && first == 0xFFFFFFFFu; j += 32) {
        const uint32_t hit = __ballot_sync(0xFFFFFFFFu, j + lane < st.item_cnt && result[st.item_base + j + lane]);
        if (hit) first = j + (uint32_t)__ffs(hit) - 1;
    }
    if (lane) return;
    const uint64_t r = e >> 1;
    const bool next = e & 1;
    const uint32_t nlist = next ? ls.n_next[r] : ls.n_prev[r];
    if (first == 0xFFFFFFFFu) {
        st.idx += st.item_list;
        if (st.idx >= nlist) st.past = 1;
    } else {
        if (first >= st.item_list) st.past = 1;
        const int32_t xs = items[st.item_base + first].x;
        const uint32_t x = (uint32_t)(xs < 0 ? -xs : xs);
        const uint32_t tests = st.past ? nlist : st.idx + first + 1u;
        pgs_gap_result *o = out + r;
        st.state = kDone;
        bool more = false;
        if (!next) {
            o->prev_p = (int32_t)x;
            o->p_tests = tests;
            if (st.past) atomicOr(&o->flags, 1u);
            if (skip_below) {
                if (x < skip_below[r]) atomicOr(&o->flags, 4u);
                else more = true, searches[e + 1].state = kActive;
            }
        } else {
            o->next_p = (int32_t)x;
            o->n_tests = tests;
            if (st.past) atomicOr(&o->flags, 2u);
        }
        if (!more) atomicAdd(active, ~0ull);  // one fewer
        atomicAdd(found, 1ull);
    }
    st.item_cnt = 0;
    searches[e] = st;
}

__global__ void gap_init_kernel(GapSearch *searches, uint64_t rows, GapLists ls, bool may_skip, uint32_t sl,
                                pgs_gap_result *out) {
    const uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= 2 * rows) return;
    const uint64_t r = e >> 1;
    GapSearch st{};
    st.state = (e & 1) && may_skip ? kWaiting : kActive;
    st.past = ((e & 1) ? ls.n_next[r] : ls.n_prev[r]) == 0 ? 1u : 0u;
    st.past_x = sl + 1;
    searches[e] = st;
    if (!(e & 1)) out[r] = pgs_gap_result{};
}

}  // namespace

}  // namespace pg

using namespace pgh;

namespace {

// K = p#/d as 32-bit limbs (gap_common.cpp:116-121).
bool build_k(uint32_t p, uint32_t d, std::vector<uint32_t> &k, std::vector<uint32_t> &k_primes) {
    k.assign(1, 1u);
    uint32_t rest = d;
    for (uint32_t q : primes_upto(p)) {
        if (rest % q == 0) {
            rest /= q;
            continue;
        }
        k_primes.push_back(q);
        uint64_t c = 0;
        for (auto &l : k) {
            const uint64_t t = (uint64_t)l * q + c;
            l = (uint32_t)t;
            c = t >> 32;
        }
        if (c) k.push_back((uint32_t)c);
    }
    return rest == 1;
}

uint32_t bits_of(const std::vector<uint32_t> &k) {
    return 32u * (uint32_t)(k.size() - 1) + (32u - (uint32_t)__builtin_clz(k.back()));
}

// _log(K) (gap_common.cpp:100-104): log of GMP's truncated 53-bit mantissa in
// [0.5, 1) plus exp * log(2).
double k_log(const std::vector<uint32_t> &k) {
    const uint32_t b = bits_of(k);
    auto bit = [&](uint32_t i) { return (k[i >> 5] >> (i & 31)) & 1u; };
    uint64_t top = 0;
    for (uint32_t i = 0; i < 53; i++) top = (top << 1) | (b >= 1 + i ? bit(b - 1 - i) : 0u);
    const double mantissa = (double)top / 9007199254740992.0;  // 2^53
    return std::log(mantissa) + std::log(2.0) * b;
}

// Smallest prev_p whose merit, float(prev_p / (K_log + log(m))), reaches
// min_merit / 2 - 2 (gap_test_gpu.cu:577-590); 0 when every prev_p does.
uint32_t skip_threshold(double klog, uint64_t m, float min_merit) {
    const float need = min_merit / 2 - 2;
    const double denom = klog + std::log((double)m);
    auto ok = [&](uint32_t g) { return !((float)(g / denom) < need); };
    if (ok(0)) return 0;
    uint32_t lo = 0, hi = 1;
    while (!ok(hi)) {
        lo = hi;
        if (hi >= 0x40000000u) return 0x7FFFFFFFu;
        hi *= 2;
    }
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        (ok(mid) ? hi : lo) = mid;
    }
    return hi;
}

constexpr uint64_t kRoundTarget = 1ull << 15;  // candidates per round of the limb form
constexpr uint32_t kMaxSpec = 512;             // most candidates per search and round
constexpr uint32_t kPastScanSpan = 1u << 24;   // distances scanned past SL before giving up

}  // namespace

extern "C" {

int pgs_prp_test(pgs_ctx *ctx, const uint32_t *limbs, uint32_t n_limbs, size_t count, int rounds,
                 uint8_t *out) {
    if (!ctx || (count && (!limbs || !out)) || n_limbs == 0 || rounds != 1) return PGS_EINVAL;
    std::lock_guard<std::mutex> g(ctx->mu);
    CK(cudaSetDevice(ctx->device));
    if (count == 0) return PGS_OK;
    // the widths; tiny, even and too wide numbers on the host
    uint32_t lo = ~0u, hi = 0;
    std::vector<uint16_t> widths;
    std::vector<uint64_t> dev_rows;
    widths.reserve(count);
    dev_rows.reserve(count);
    for (size_t i = 0; i < count; i++) {
        const uint32_t *v = limbs + i * n_limbs;
        uint32_t top = n_limbs;
        while (top > 0 && v[top - 1] == 0) top--;
        const uint32_t bits = top ? 32u * (top - 1) + (32u - (uint32_t)__builtin_clz(v[top - 1])) : 0u;
        if (bits > 8u * pg::kMaxL * 32u - 4u) {
            ctx->err = "pgs_prp_test: numbers above 4092 bits";
            return PGS_EINVAL;
        }
        if (bits <= 3) {  // 0..7: the reference's answers for 2, 3, 5, 7 are prime
            const uint32_t v0 = bits ? v[0] : 0u;
            out[i] = (v0 == 2 || v0 == 3 || v0 == 5 || v0 == 7) ? 1 : 0;
            continue;
        }
        if (!(v[0] & 1u)) {
            out[i] = 0;
            continue;
        }
        lo = std::min(lo, bits);
        hi = std::max(hi, bits);
        widths.push_back((uint16_t)bits);
        dev_rows.push_back(i);
    }
    if (dev_rows.empty()) return PGS_OK;
    std::vector<uint64_t> order;
    std::vector<pg::PrpPart> parts;
    if (hi - lo <= pg::kRnsSpread) {
        parts.push_back({0, dev_rows.size(), pg::prp_plan(hi, dev_rows.size())});
    } else {
        parts = pg::prp_parts(widths, lo, hi, order);
    }
    const auto at = [from = order.empty() ? nullptr : order.data()](uint64_t i) { return from ? from[i] : i; };
    size_t words = 0, work_bytes = 0;
    for (const auto &part : parts) {
        words += part.count * 8u * (size_t)part.plan.L;
        if (part.plan.rns) work_bytes = std::max(work_bytes, part.plan.layout.total);
    }
    const cudaStream_t s = ctx->stream;
    DevBuf d_nums, d_items, d_res, d_work;
    DevBuf *bufs[] = {&d_nums, &d_items, &d_res, &d_work};
    for (DevBuf *b : bufs) b->pool = &ctx->dpool;
    cudaError_t e = cudaSuccess;
    if (work_bytes && !pg::prp_workspace(d_work, work_bytes, e)) {
        for (auto &part : parts) part.plan.rns = false;
    }
    std::vector<uint32_t> packed(words, 0u);
    std::vector<pg::PrpItem> items(dev_rows.size());
    uint32_t *to = packed.data();
    for (const auto &part : parts) {
        const uint32_t n = 8u * (uint32_t)part.plan.L;
        for (uint64_t j = 0; j < part.count; j++, to += n) {
            std::memcpy(to, limbs + dev_rows[at(part.first + j)] * n_limbs, std::min(n, n_limbs) * 4u);
            items[part.first + j] = pg::PrpItem{(uint32_t)j, 0};
        }
    }
    std::vector<uint8_t> res(dev_rows.size());
    std::vector<unsigned long long> gave_up(parts.size(), 0ull);
    if (e == cudaSuccess) e = upload(d_nums, packed, s);
    if (e == cudaSuccess) e = upload(d_items, items, s);
    if (e == cudaSuccess) e = d_res.ensure(dev_rows.size());
    const uint32_t *nums = d_nums.as<uint32_t>();
    for (size_t i = 0; i < parts.size() && e == cudaSuccess; i++) {
        const pg::PrpPart &part = parts[i];
        e = pg::prp_begin(part.plan, d_work.p, s);
        if (e == cudaSuccess)
            e = pg::prp_launch(part.plan, d_work.p, nums, d_items.as<pg::PrpItem>() + part.first, nullptr, part.count,
                               d_res.as<uint8_t>() + part.first, s);
        if (e == cudaSuccess) e = pg::prp_error(part.plan, d_work.p, &gave_up[i], s);
        nums += part.count * 8u * (size_t)part.plan.L;
    }
    if (e == cudaSuccess) e = cudaMemcpyAsync(res.data(), d_res.p, res.size(), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaStreamSynchronize(s);
    for (DevBuf *b : bufs) b->release();
    if (e != cudaSuccess) return fail(ctx, e, "pgs_prp_test");
    if (std::any_of(gave_up.begin(), gave_up.end(), [](unsigned long long g) { return g != 0; })) {
        ctx->err = "pgs_prp_test: a wait on the device gave up";
        return PGS_ETIMEOUT;
    }
    for (size_t j = 0; j < dev_rows.size(); j++) out[dev_rows[at(j)]] = res[j];
    return PGS_OK;
}

}  // extern "C"

namespace {

// What a search's rounds are expected to take, in microseconds, with so many unknowns on
// each side and a chance that one is prime (sl / lnN primes on a side): round after round
// of so many candidates, shared by the sides that are left, until there is none.
struct RoundCost {
    uint32_t bits;
    double unknowns, chance;
    double us(uint64_t searches, uint64_t items, bool residues) const {
        double total = 0, left = (double)searches;
        for (int round = 0; round < 20 && left >= 0.2; round++) {
            double each = std::min((double)items / left, (double)kMaxSpec);
            if (!residues) each = std::min(each, unknowns);
            const double count = std::ceil(each * left);
            total += 130 + (residues ? pg::rns_us(bits, (uint64_t)count) : pg::limb_us(bits, count * bits));
            left *= std::exp(-each * chance);
        }
        if (left >= 0.2)  // many more rounds like these
            total *= std::log(5.0 * (double)searches) / std::log((double)searches / left);
        return total;
    }
    // Candidates of a round of the limb form: blocks on each SM that are full.  (Both
    // sides of 5 rows of 2503#/30030: 7 rounds of 64 for each side 386 ms, one of 512 131,
    // 243 111; of 20 rows 417, 372, 142.)
    uint64_t limb_items(uint64_t searches) const {
        uint64_t best = 0;
        double best_us = 0;
        for (uint64_t items = pg::limb_layer(); items <= kRoundTarget; items += pg::limb_layer()) {
            const double t = us(searches, items, false);
            if (!best || t < best_us) best = items, best_us = t;
        }
        return best;
    }
};

// Whether a search's rounds are the residue form's, which a search of few rows leaves
// mostly empty or fills with what is not needed (7 rows of 307#/210: 0.70 ms limb by limb,
// 1.00 in residues).  Rows with m far below the largest are tested limb by limb in every
// round: more than a few, and the whole search is.
bool residue_rounds(const RoundCost &c, uint64_t rows, const uint64_t *h_m, uint64_t searches) {
    if (c.bits < 253 || pg::rns_chunks(c.bits) == 0) return false;
    uint64_t max_m = 0, narrow = 0;
    for (uint64_t r = 0; r < rows; r++) max_m = std::max(max_m, h_m[r]);
    for (uint64_t r = 0; r < rows; r++) narrow += h_m[r] >> 1 < max_m >> pg::kRnsSpread;
    if (narrow > rows / 256) return false;
    return c.us(searches, pg::rns_wave(c.bits, false), true) < 1.1 * c.us(searches, c.limb_items(searches), false);
}

// Device lists of rows (d_m .. d_dist, as pgs_unknowns; `listed` unknowns in all) and the
// host copy of their m: the gap search.  The caller holds ctx->mu and checked the lists.
int prp_gaps_core(pgs_ctx *ctx, const pgs_gap_params *prm, uint64_t rows, const uint64_t *h_m,
                  const uint64_t *d_m, const uint64_t *d_start, const uint32_t *d_np, const uint32_t *d_nn,
                  const uint32_t *d_dist, uint64_t listed, pgs_gap_result *out, pgs_gap_stats *stats) {
    if (prm->p < 2 || !is_prime_u64(prm->p) || prm->d == 0 || prm->sieve_length == 0 ||
        prm->sieve_length >= (1u << 30)) {
        ctx->err = "pgs_prp_gaps: bad p, d or sieve_length";
        return PGS_EINVAL;
    }
    std::vector<uint32_t> k, kprimes;
    if (!build_k(prm->p, prm->d, k, kprimes) || (k.size() == 1 && k[0] <= 1)) {
        ctx->err = "pgs_prp_gaps: d does not divide p#";
        return PGS_EINVAL;
    }
    uint64_t max_m = 0;
    for (uint64_t r = 0; r < rows; r++) max_m = std::max(max_m, h_m[r]);
    const uint32_t bits = bits_of(k) + (64u - (uint32_t)__builtin_clzll(max_m)) + 1u;
    if (bits > 8u * pg::kMaxL * 32u - 4u) {
        ctx->err = "pgs_prp_gaps: m*K above 4092 bits";
        return PGS_EINVAL;
    }
    // A round is a wave of the residue form (its time is the same for fewer), or
    // enough to fill the GPU with the limb form
    const bool may_skip = prm->one_side_skip != 0;
    const uint64_t searches = 2 * rows, wave = pg::rns_wave(bits, true);
    const uint64_t limb_round = std::max<uint64_t>(searches, kRoundTarget);
    RoundCost cost{bits, std::max(1.0, (double)listed / (double)searches), 1.0};
    cost.chance = std::min(1.0, prm->sieve_length / (0.693 * bits) / cost.unknowns);
    pg::PrpPlan plan = pg::limb_plan(bits);
    if (residue_rounds(cost, rows, h_m, may_skip ? rows : searches)) {
        plan.rns = true;
        plan.layout = pg::rns_layout(bits, 8u * (uint32_t)plan.L, wave, wave);
    }
    const uint32_t n = 8u * (uint32_t)plan.L;
    std::vector<uint32_t> skip(rows, 0u);
    if (prm->one_side_skip) {
        const double klog = k_log(k);
        for (uint64_t r = 0; r < rows; r++) skip[r] = skip_threshold(klog, h_m[r], prm->min_merit);
    }
    const cudaStream_t s = ctx->stream;
    DevBuf d_k, d_kp, d_skip, d_centers, d_state, d_items, d_res, d_out, d_ctr, d_work, d_past;
    DevBuf *bufs[] = {&d_past, &d_k, &d_kp, &d_skip, &d_centers, &d_state, &d_items, &d_res, &d_out, &d_ctr, &d_work};
    for (DevBuf *b : bufs) b->pool = &ctx->dpool;
    auto cleanup = [&] {
        cudaStreamSynchronize(s);
        for (DevBuf *b : bufs) b->release();
    };
    cudaError_t e = cudaSuccess;
    if (plan.rns) plan.rns = pg::prp_workspace(d_work, plan.layout.total, e);
    const uint64_t max_items = plan.rns ? wave : limb_round;
    if (e == cudaSuccess) e = upload(d_k, k, s);
    if (e == cudaSuccess) e = upload(d_kp, kprimes, s);
    if (e == cudaSuccess && may_skip) e = upload(d_skip, skip, s);
    if (e == cudaSuccess) e = d_past.ensure(pg::kPastBits / 8);
    if (e == cudaSuccess) e = d_centers.ensure(rows * n * 4ull);
    if (e == cudaSuccess) e = d_state.ensure(searches * sizeof(pg::GapSearch));
    if (e == cudaSuccess) e = d_items.ensure(max_items * sizeof(pg::PrpItem));
    if (e == cudaSuccess) e = d_res.ensure(max_items);
    if (e == cudaSuccess) e = d_out.ensure(rows * sizeof(pgs_gap_result));
    if (e == cudaSuccess) e = d_ctr.ensure(40);
    if (e == cudaSuccess) e = pg::prp_begin(plan, d_work.p, s);
    if (e != cudaSuccess) {
        cleanup();
        return fail(ctx, e, "pgs_prp_gaps setup");
    }
    const pg::GapLists ls{d_start, d_np, d_nn, d_dist};
    unsigned long long *ctr = d_ctr.as<unsigned long long>();  // items, asked, active, errors, found
    const uint32_t *skip_below = may_skip ? d_skip.as<uint32_t>() : nullptr;
    const unsigned rb = (unsigned)((rows + 255) / 256), sb = (unsigned)((searches + 7) / 8);
    pg::centers_kernel<<<rb, 256, 0, s>>>(d_k.as<uint32_t>(), (uint32_t)k.size(), d_m, rows, n,
                                          d_centers.as<uint32_t>());
    if (plan.rns)
        pg::past_kernel<<<pg::kPastBits / 256, 256, 0, s>>>(d_kp.as<uint32_t>(), (uint32_t)kprimes.size(),
                                                            prm->sieve_length, d_past.as<uint32_t>());
    pg::gap_init_kernel<<<(unsigned)((searches + 255) / 256), 256, 0, s>>>(
        d_state.as<pg::GapSearch>(), rows, ls, may_skip, prm->sieve_length, d_out.as<pgs_gap_result>());
    uint64_t active = may_skip ? rows : searches, rounds = 0, launched = 0;
    unsigned long long host_ctr[5] = {0, 0, active, 0, 0};
    e = cudaMemcpyAsync(ctr, host_ctr, 40, cudaMemcpyHostToDevice, s);
    const uint32_t x_limit = prm->sieve_length + kPastScanSpan;
    while (e == cudaSuccess && active > 0) {
        uint64_t quota = active;
        if (!plan.rns) {
            quota = std::max(active, std::min(cost.limb_items(active), active * kMaxSpec));
        } else {
            // A wave of several tiles per pair tests 1.1-1.2 times as many a second as
            // a single one, but what lies past a search's end is wasted: with s
            // candidates per search in the single wave and a chance p of each (found
            // so far / tested), it resolves more a second where s p is below 0.45
            // (2136 bits, p 1/39, 20.5 and 12.4 ms: 33 searches a ms each at s p = 0.43).
            const uint64_t one = pg::rns_wave(bits, false);
            const double chance = launched ? (double)host_ctr[4] / (double)launched : 1.0 / 32;
            quota = std::min((double)one * chance < 0.45 * (double)active ? max_items : one, active * kMaxSpec);
        }
        const uint32_t spec = (uint32_t)(quota / active), extra = (uint32_t)(quota % active);
        e = cudaMemsetAsync(ctr, 0, 16, s);  // items, asked
        if (e) break;
        pg::select_kernel<<<sb, 256, 0, s>>>(d_state.as<pg::GapSearch>(), rows, ls, d_centers.as<uint32_t>(), n, spec,
                                             extra, plan.rns, d_kp.as<uint32_t>(), (uint32_t)kprimes.size(),
                                             plan.rns ? d_past.as<uint32_t>() : nullptr, prm->sieve_length, x_limit,
                                             d_items.as<pg::PrpItem>(), quota, ctr, ctr + 1, ctr + 3);
        e = pg::prp_launch(plan, d_work.p, d_centers.as<uint32_t>(), d_items.as<pg::PrpItem>(), ctr, quota,
                           d_res.as<uint8_t>(), s);
        if (e) break;
        unsigned long long gave_up = 0;
        e = pg::prp_error(plan, d_work.p, &gave_up, s);
        if (e) break;
        pg::resolve_kernel<<<sb, 256, 0, s>>>(d_state.as<pg::GapSearch>(), rows, ls, skip_below,
                                              d_items.as<pg::PrpItem>(), d_res.as<uint8_t>(), prm->sieve_length,
                                              d_out.as<pgs_gap_result>(), ctr + 2,
                                              ctr + 4);
        e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaMemcpyAsync(host_ctr, ctr, 40, cudaMemcpyDeviceToHost, s);
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e) break;
        if (host_ctr[3]) break;  // reported below
        if (gave_up) {
            cleanup();
            ctx->err = "pgs_prp_gaps: a wait on the device gave up";
            return PGS_ETIMEOUT;
        }
        launched += host_ctr[0];
        active = host_ctr[2];
        if (++rounds > (1u << 22)) {
            cleanup();
            ctx->err = "pgs_prp_gaps: no progress";
            return PGS_ETIMEOUT;
        }
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(out, d_out.p, rows * sizeof(pgs_gap_result), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cleanup();
    if (e != cudaSuccess) return fail(ctx, e, "pgs_prp_gaps");
    if (host_ctr[3]) {
        ctx->err = "pgs_prp_gaps: a side found no probable prime within 2^24 past the sieve length";
        return PGS_EABORT;
    }
    if (stats) {
        stats->rounds = rounds;
        stats->prp_tests = launched;
        stats->limbs = n;
    }
    return PGS_OK;
}

}  // namespace

extern "C" {

int pgs_prp_gaps(pgs_ctx *ctx, const pgs_gap_params *prm, const pgs_unknowns *lists, pgs_gap_result *out,
                 pgs_gap_stats *stats) {
    if (!ctx || !prm || !lists || (lists->rows && !out)) return PGS_EINVAL;
    if (stats) std::memset(stats, 0, sizeof(*stats));
    std::lock_guard<std::mutex> g(ctx->mu);
    CK(cudaSetDevice(ctx->device));
    const uint64_t rows = lists->rows;
    if (rows == 0) return PGS_OK;
    if (rows >= (1ull << 31) || !lists->m || !lists->start || !lists->n_prev || !lists->n_next ||
        (lists->total && !lists->dist)) {
        ctx->err = "pgs_prp_gaps: bad lists";
        return PGS_EINVAL;
    }
    uint64_t listed = 0;
    for (uint64_t r = 0; r < rows; r++) {
        if (lists->m[r] == 0 || lists->start[r] + lists->n_prev[r] + lists->n_next[r] > lists->total) {
            ctx->err = "pgs_prp_gaps: row outside the distance array";
            return PGS_EINVAL;
        }
        listed += lists->n_prev[r] + (uint64_t)lists->n_next[r];
    }
    const cudaStream_t s = ctx->stream;
    PackedLists pk;
    pk.block.pool = &ctx->dpool;
    cudaError_t e = packed_alloc(pk, rows, lists->total);
    auto up = [&](void *dst, const void *src, size_t bytes) {
        return bytes ? cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s) : cudaSuccess;
    };
    if (e == cudaSuccess) e = up(pk.m, lists->m, rows * 8);
    if (e == cudaSuccess) e = up(pk.start, lists->start, rows * 8);
    if (e == cudaSuccess) e = up(pk.n_prev, lists->n_prev, rows * 4);
    if (e == cudaSuccess) e = up(pk.n_next, lists->n_next, rows * 4);
    if (e == cudaSuccess) e = up(pk.dist, lists->dist, lists->total * 4);
    int rc = e == cudaSuccess ? prp_gaps_core(ctx, prm, rows, lists->m, pk.m, pk.start, pk.n_prev, pk.n_next,
                                              pk.dist, listed, out, stats)
                              : fail(ctx, e, "pgs_prp_gaps upload");
    cudaStreamSynchronize(s);
    pk.block.release();
    return rc;
}

int pgs_prp_gaps_prepared(pgs_ctx *ctx, pgs_prepared *prep, const pgs_gap_params *prm, pgs_gap_result *out,
                          pgs_gap_stats *stats) {
    if (!ctx || !prep || !prm || !out || prep->ctx != ctx || !prep->ran) return PGS_EINVAL;
    if (stats) std::memset(stats, 0, sizeof(*stats));
    std::lock_guard<std::mutex> g(ctx->mu);
    CK(cudaSetDevice(ctx->device));
    const HostJob &h = prep->hj;
    const uint64_t rows = h.valid_mi.size();
    if (rows == 0) return PGS_OK;
    std::vector<uint64_t> m(rows);
    for (uint64_t r = 0; r < rows; r++) m[r] = h.job.mstart + h.valid_mi[r];
    pgs_gap_params jp = *prm;  // the job's own p, d and sieve length
    jp.p = h.job.p;
    jp.d = h.job.d;
    jp.sieve_length = h.job.sieve_length;
    const cudaStream_t s = ctx->stream;
    PackedLists pk;
    int rc = job_lists_device(ctx, prep, s, pk);
    if (rc == PGS_OK)
        rc = prp_gaps_core(ctx, &jp, rows, m.data(), pk.m, pk.start, pk.n_prev, pk.n_next, pk.dist, pk.total, out,
                           stats);
    cudaStreamSynchronize(s);
    pk.block.release();
    return rc;
}

}  // extern "C"
