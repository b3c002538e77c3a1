// Base-2 strong probable-prime tests on the tensor cores.
//
// Replaces, for many numbers of one size, the limb arithmetic of the reference's
// kernel_miller_rabin (miller_rabin.h:154-267).  A test is a chain of about
// log2 N squarings mod N, and a chain of squarings of different numbers has no
// matrix product in it -- unless the numbers are held as residues: Montgomery
// reduction in a residue number system (Posch and Posch 1995; Bajard, Didier and
// Kornerup 1998; the quotient's rank as in Kawamura et al. 2000) needs two base
// extensions per squaring, and a base extension is a product with a matrix of
// constants that every number shares.
//
// Two bases of pairwise coprime moduli up to 4096: A (primes) and B.  x is held
// as |x| <= cN in both.  With xi_i = x_i^2 (-N^-1) (A/m_i)^-1 mod m_i,
// q = sum xi_i A/m_i is congruent to -x^2/N mod A, |q| <= A k/2, and
// (x^2 + q N)/A is again below cN when 4c^2 N <= A (x^2 may come doubled twice).
// First extension (q to B): q_j = sum_i xi_i ((A/m_i) mod m_j).  Then in B
// r_j = (x_j^2 + q_j N_j)/A, held as xi_j = r_j (B/m_j)^-1.  Second extension
// (r back to A): r_i = sum_j xi_j ((B/m_j) mod m_i) - a (B mod m_i), with
// a = round(sum_j xi_j / m_j), exact since |r| <= B/4.
//
// Exact arithmetic in floating point.  Residues are balanced, |xi| <= 2048, so
// one f16 holds one; a matrix entry is split as c = lo + hi, |lo| <= 32 and hi a
// multiple of 64, each exact in f16, and the two sums stay below 2^24 (times 64
// for hi), which the choice of the moduli sees to (pg_rns_moduli.h): the tensor
// core's f32 accumulators hold them exactly.  Everything
// between the products is f32 multiply-adds whose results are whole numbers
// below 2^24 (the remainder of T by m: q = rint(T/m) by adding 1.5 2^23, then
// T - q m, exact in a fused multiply-add).
//
// A pair of CTAs takes 256 numbers, 128 TMEM lanes each, a lane a number.  The
// two matrices (K x 2K f16) stay in the pair's shared memory for the whole
// chain, half the columns in each CTA (cta_group::2), so nothing but the
// numbers' own constants is read again.  The residues are the A operand and lie
// in TMEM, written there by the threads that compute them.  Output columns come
// in blocks of 64 slots (128 columns); while 16 warps turn a block of sums into
// residues, 32 slots at a time, the tensor cores work on the next one, and the next
// product's first block accumulates slice by slice as the residues appear.
//
// Measured (2136-bit numbers, 19456 at once): 12.2 ms, 1.6e6 tests/s, where the
// limb form takes 105 ms; a squaring step 5.2 us per pair, of which the products
// alone take 2.9 (128 columns cost 78 cycles per 16 of K; 64 columns cost the same,
// the A operand's read, hence blocks of 128) and the residues' f32 operations 3.4.
#include "pg_rns.h"
#include "pg_rns_moduli.h"

#include <cuda_fp16.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <type_traits>
#include <vector>

namespace pg {

namespace {

constexpr uint32_t kMaxK = kSlots * kRnsMaxChunks;     // 288
constexpr uint32_t kWarps = 16;                        // warps that compute residues
constexpr uint32_t kThreads = 32 * (kWarps + 1);       // and one that issues products
constexpr float kMagic = 12582912.0f;                  // 1.5 2^23

// Constants of two neighbouring slots, as the paired f32 operations read them.
struct SlotPair {
    float neg_m[2], inv_m[2], c[2];  // -m, 1/m; A: -(B mod m), B: (B/m) / A mod m
    float pad[2];
};
struct RnsConst {
    SlotPair a[kMaxK / 2], b[kMaxK / 2];
};

// What the kernels around the chain need of each slot.
struct RnsSlots {
    uint16_t ma[kMaxK], mb[kMaxK];   // moduli (base A: slot 0 is the rank's column, modulus 1)
    uint16_t am[kMaxK];              // A/m_i mod m_i
    uint16_t ab[kMaxK];              // A mod m_j
    uint16_t gb[kMaxK];              // (B/m_j)^-1 mod m_j
    uint16_t ba[kMaxK];              // B mod m_i
    uint32_t b_primes;               // the first moduli of B, prime
};

struct RnsPlan {
    RnsConst k;
    RnsSlots s;
    double a_mant;        // A = a_mant 2^a_exp, a_mant in [1/2, 1)
    int a_exp;
    uint32_t t_max;       // largest multiple of N between two values of one residue
};

uint32_t inverse(uint32_t a, uint32_t m) {  // extended Euclid; a and m coprime
    int64_t r0 = m, r1 = a % m, t0 = 0, t1 = 1;
    while (r1) {
        const int64_t q = r0 / r1;
        const int64_t r2 = r0 - q * r1, t2 = t0 - q * t1;
        r0 = r1, r1 = r2, t0 = t1, t1 = t2;
    }
    return (uint32_t)(t0 < 0 ? t0 + m : t0);
}

float balanced(uint32_t x, uint32_t m) { return x > m / 2 ? (float)x - (float)m : (float)x; }

void make_plan(uint32_t n, uint32_t ka, RnsPlan &p) {
    const RnsModuli &mod = moduli_of(n);
    const uint32_t k = kSlots * n;
    const std::vector<uint32_t> a(mod.a.begin(), mod.a.begin() + ka);
    std::memset(&p, 0, sizeof(p));
    p.t_max = (uint32_t)(2 * coefficient(a.size()) + 4);
    p.a_mant = 1;
    for (uint32_t q : a) {
        int e;
        p.a_mant = std::frexp(p.a_mant * q, &e);
        p.a_exp += e;
    }
    auto prod = [](const std::vector<uint32_t> &v, uint32_t m, uint32_t but) {
        uint32_t r = 1;
        for (uint32_t q : v)
            if (q != but) r = r * q % m;  // below 2^24
        return r;
    };
    p.s.b_primes = mod.b_primes;
    for (uint32_t i = 0; i < k; i++) {
        p.s.ma[i] = 1;
        if (i == 0 || i > a.size()) continue;
        const uint32_t m = a[i - 1];
        p.s.ma[i] = (uint16_t)m;
        p.s.am[i] = (uint16_t)prod(a, m, m);
        p.s.ba[i] = (uint16_t)prod(mod.b, m, 0);
    }
    for (uint32_t j = 0; j < k; j++) {
        const uint32_t m = mod.b[j];
        p.s.mb[j] = (uint16_t)m;
        p.s.ab[j] = (uint16_t)prod(a, m, 0);
        p.s.gb[j] = (uint16_t)inverse(prod(mod.b, m, m), m);
    }
    for (uint32_t i = 0; i < k; i++) {
        SlotPair &pa = p.k.a[i / 2], &pb = p.k.b[i / 2];
        const uint32_t h = i & 1;
        const uint32_t ma = p.s.ma[i], mb = p.s.mb[i];
        pa.neg_m[h] = -(float)ma;
        pa.inv_m[h] = 1.0f / (float)ma;
        pa.c[h] = ma > 1 ? -balanced(p.s.ba[i], ma) : 0.0f;
        pb.neg_m[h] = -(float)mb;
        pb.inv_m[h] = 1.0f / (float)mb;
        pb.c[h] = balanced(inverse(p.s.gb[i], mb) * inverse(p.s.ab[i], mb) % mb, mb);
    }
}

// One plan per (n, moduli of A): constants, made on first use and kept for the
// process, at most about kMaxK of 10 KB.
const RnsPlan &plan_of(uint32_t n, uint32_t bits) {
    static std::mutex mu;
    static std::map<uint32_t, std::unique_ptr<RnsPlan>> plans;
    const uint32_t ka = a_count(n, bits);
    std::lock_guard<std::mutex> g(mu);
    std::unique_ptr<RnsPlan> &p = plans[n << 16 | ka];
    if (!p) {
        p.reset(new RnsPlan);
        make_plan(n, ka, *p);
    }
    return *p;
}

// ---------------------------------------------------------------------------
// device arithmetic on residues below 4096

// v mod m; inv32 = floor((2^32 - 1) / m): the quotient is at most one short
__device__ __forceinline__ uint32_t mod_small(uint32_t v, uint32_t m, uint32_t inv32) {
    uint32_t r = v - __umulhi(v, inv32) * m;
    return r >= m ? r - m : r;
}

__device__ uint32_t pow_small(uint32_t x, uint32_t e, uint32_t m, uint32_t inv32) {
    uint32_t r = 1;
    for (; e; e >>= 1) {
        if (e & 1) r = mod_small(r * x, m, inv32);
        x = mod_small(x * x, m, inv32);
    }
    return r;
}

// a^-1 mod m (m not always prime), by Euclid; a and m coprime
__device__ uint32_t inverse_small(uint32_t a, uint32_t m) {
    int r0 = (int)m, r1 = (int)(a % m), t0 = 0, t1 = 1;
    while (r1) {
        const int q = r0 / r1, r2 = r0 - q * r1, t2 = t0 - q * t1;
        r0 = r1, r1 = r2, t0 = t1, t1 = t2;
    }
    return (uint32_t)(t0 < 0 ? t0 + (int)m : t0);
}

__device__ __forceinline__ int balance(uint32_t x, uint32_t m) { return x > m / 2 ? (int)x - (int)m : (int)x; }

__device__ __forceinline__ uint32_t inv32_of(uint32_t m) { return m > 1 ? 0xFFFFFFFFu / m : 0u; }

// The matrices as the tensor cores read them from shared memory.  Per CTA of
// the pair (0: the low parts, 1: the high parts), product (0: xi of B into A,
// 1: xi of A into B) and block of 64 output slots (the last may have 32), 8 x 8
// pieces of 128 bytes, neighbouring outputs together: [k/8][slot/8][slot%8][k%8].
__global__ void matrix_kernel(const __grid_constant__ RnsSlots p, uint32_t chunks, __half *__restrict__ out) {
    const uint32_t k = kSlots * chunks;
    const uint32_t idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 2 * k * k) return;
    const uint32_t product = idx / (k * k), in = idx % (k * k) / k, o = idx % k;
    float lo = 0, hi = 0;
    if (product == 0) {
        const uint32_t mj = p.mb[in];
        const uint32_t m = p.ma[o], inv = inv32_of(m);  // m prime, or 1
        if (o == 0) {
            lo = 4096.0f / (float)mj;  // the rank's column: xi_j / m_j
        } else if (m > 1) {
            const int c = balance(mod_small(p.ba[o] * pow_small(mj % m, m - 2, m, inv), m, inv), m);
            const int l = ((c + 32) & 63) - 32;
            lo = (float)l, hi = (float)(c - l);
        }
    } else if (p.ma[in] > 1) {
        const uint32_t m = p.mb[o];
        const int c = balance(mod_small(p.ab[o] * inverse_small(p.ma[in], m), m, inv32_of(m)), m);
        const int l = ((c + 32) & 63) - 32;
        lo = (float)l, hi = (float)(c - l);
    }
    const uint32_t block = o / 64, slot = o % 64, rows = min(64u, k - 64 * block);
    const uint64_t at = (uint64_t)product * k * k + block * 64 * k +
                        (in / 8 * (rows / 8) + slot / 8) * 64 + slot % 8 * 8 + in % 8;
    out[at] = __float2half_rn(lo);
    out[at + 2ull * k * k] = __float2half_rn(hi);
}

// Halves of a number's slots lie as the chain's threads load them: 8 slots of
// one warp group per 16 bytes, neighbouring numbers together.
__device__ __forceinline__ uint64_t slot_at(uint32_t chunks, uint64_t number, uint32_t slot) {
    const uint64_t tile = number / 128, row = number % 128;
    return ((tile * chunks * 4 + slot / 8) * 128 + row) * 8 + slot % 8;
}

enum { kFlagRun = 0, kFlagComposite = 1, kFlagOther = 2 };

// Remainder below 2m (3m for v above 2^31) of v by m, where it only has to be small.
__device__ __forceinline__ uint32_t mod_lazy(uint32_t v, uint32_t m, uint32_t inv32) {
    return v - __umulhi(v, inv32) * m;
}

// Little-endian limbs mod m.
__device__ __forceinline__ uint32_t limbs_mod(const uint32_t *n, uint32_t limbs, uint32_t m, uint32_t inv32) {
    uint32_t r = 0;
    for (int w = (int)limbs - 1; w >= 0; w--) {
        const uint32_t v = n[w];
        r = mod_lazy((r << 16) | (v >> 16), m, inv32);
        r = mod_lazy((r << 16) | (v & 0xFFFFu), m, inv32);
    }
    return r >= m ? r - m : r;
}

// Whether n (top its highest limb that is not 0) is near enough to 2^bits for
// its start, and floor(A / n) from its leading words.
__device__ bool near_widest(const uint32_t *n, int top, uint32_t bits, double a_mant, int a_exp, long long &q) {
    if (top < 3) return false;
    const double v = ((double)n[top] * 4294967296.0 + (double)n[top - 1]) * 4294967296.0 + (double)n[top - 2];
    if (log2(v) + 32.0 * (top - 2) <= (double)bits - 24.0) return false;
    q = (long long)floor(ldexp(a_mant / v, a_exp - 32 * (top - 2)));
    return true;
}

// Per number: its limbs, its constants in every slot, its start (the Montgomery
// form of 1).  A block takes 8 numbers; a thread one slot of each base.
// A prime m of base A that divides N leaves no inverse there.  N can still be a
// pseudoprime only if 2^(N-1) = 1 mod m; then the chain runs mod N/m (the
// exponent stays N's) and the verdict looks at both; so too for two primes.  It is
// composite if m^2 divides it: 2's order mod m^2 would divide N - 1, hence be prime to m,
// hence divide m - 1, as it does below 4096 for m = 1093 and 3511 alone.  (Of unsieved
// numbers of 2900 bits, where A goes down to 17, one in 2000 is such a multiple; the limb
// form took 54 ms more for a single one.)
// Bound by the remainders' multiplies, one per 16 bits, number and modulus.
constexpr uint32_t kSetupNumbers = 8;
__global__ void setup_kernel(const __grid_constant__ RnsSlots p, uint32_t chunks, uint32_t bits, double a_mant,
                             int a_exp, uint32_t limbs, const uint32_t *__restrict__ bases,
                             const PrpItem *__restrict__ items, const unsigned long long *count, uint64_t max_items,
                             __half *__restrict__ num_a, __half *__restrict__ num_b, __half *__restrict__ state,
                             uint32_t *__restrict__ nums, long long *__restrict__ quot, uint32_t *__restrict__ flag,
                             uint32_t *__restrict__ factor) {
    __shared__ uint32_t s_n[kSetupNumbers][128];
    __shared__ long long s_q[kSetupNumbers];
    __shared__ uint32_t s_f[kSetupNumbers];
    // primes of A that divide the number, the last of them, and whether one rules it out
    __shared__ uint32_t s_divide[kSetupNumbers], s_by[kSetupNumbers], s_out[kSetupNumbers];
    const uint64_t n_items = count ? min((uint64_t)*count, max_items) : max_items;
    const uint64_t padded = ((n_items + kRnsTile - 1) / kRnsTile + kRnsGroup - 1) * kRnsTile;
    const uint64_t first = (uint64_t)blockIdx.x * kSetupNumbers;
    if (first >= padded) return;
    // the numbers' limbs, together; then a thread per number adds its offset
    for (uint32_t e = threadIdx.x; e < kSetupNumbers * limbs; e += blockDim.x) {
        const uint32_t g = e / limbs, w = e % limbs;
        if (first + g < n_items) s_n[g][w] = bases[(uint64_t)items[first + g].row * limbs + w];
    }
    __syncthreads();
    if (threadIdx.x < kSetupNumbers) {
        const uint32_t g = threadIdx.x;
        const uint64_t i = first + g;
        long long q = 0;
        uint32_t f = kFlagComposite;
        if (i < n_items) {
            int64_t carry = items[i].x;
            int top = -1;
            for (uint32_t w = 0; w < limbs; w++) {
                const uint32_t was = s_n[g][w];
                const int64_t v = (int64_t)was + carry;
                if (carry) s_n[g][w] = (uint32_t)v;
                carry = v >> 32;
                if ((uint32_t)v) top = (int)w;
            }
            f = near_widest(s_n[g], top, bits, a_mant, a_exp, q) ? kFlagRun : kFlagOther;
        }
        s_q[g] = q;
        s_f[g] = f;
        s_divide[g] = 0, s_by[g] = 1, s_out[g] = 0;
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < kSetupNumbers * limbs; e += blockDim.x) {
        const uint32_t g = e / limbs, w = e % limbs;
        if (first + g < n_items) nums[(first + g) * limbs + w] = s_n[g][w];
    }
    const uint32_t t = threadIdx.x;
    const uint32_t ma = p.ma[t], mb = p.mb[t];
    const uint32_t ia = inv32_of(ma), ib = inv32_of(mb);
    const uint32_t ainv = inverse_small(p.ab[t], mb);
    // the 8 numbers mod this thread's two moduli: sums of 16-bit digits times the
    // powers of 2^16, which the numbers share (remainders every 8 digits: below 2^32)
    uint32_t ra[kSetupNumbers], rb[kSetupNumbers];
#pragma unroll
    for (uint32_t g = 0; g < kSetupNumbers; g++) ra[g] = rb[g] = 0;
    uint32_t pa = ma > 1, pb = mb > 1;
    for (uint32_t w = 0; w < limbs; w++) {
        const uint32_t qa = mod_small(pa << 16, ma, ia), qb = mod_small(pb << 16, mb, ib);
        const bool reduce = (w & 3) == 3;
#pragma unroll
        for (uint32_t g = 0; g < kSetupNumbers; g++) {
            const uint32_t v = s_n[g][w], lo = v & 0xFFFFu, hi = v >> 16;
            ra[g] += lo * pa + hi * qa;
            rb[g] += lo * pb + hi * qb;
            if (reduce) ra[g] = mod_lazy(ra[g], ma, ia), rb[g] = mod_lazy(rb[g], mb, ib);
        }
        pa = mod_small(qa << 16, ma, ia), pb = mod_small(qb << 16, mb, ib);
    }
    const auto slots = [&](uint32_t g, uint32_t ra, uint32_t rb, uint32_t by) {  // by: what N was divided by
        const uint64_t at = slot_at(chunks, first + g, t);
        int ca = 0;
        if (ma > 1 && ra == 0) {
            atomicAdd(&s_divide[g], 1u);
            s_by[g] = ma;
            if (by == 1) {
                uint32_t r = limbs_mod(s_n[g], limbs, ma - 1, inv32_of(ma - 1));
                r = r ? r - 1 : ma - 2;
                if (pow_small(2, r, ma, ia) != 1) s_out[g] = 1;
            } else if ((ma == (by & 0xFFFFu) || ma == by >> 16) && ma != 1093 && ma != 3511) {
                s_out[g] = 1;
            }
        } else if (ma > 1) {  // -1 / (N (A/m))
            const uint32_t d = mod_small(ra * p.am[t], ma, ia);
            ca = -balance(pow_small(d, ma - 2, ma, ia), ma);
        }
        num_a[at] = __float2half_rn((float)ca);
        // n = N (B/m)^-1 / A;  start xi = ((B/m)^-1 - q n) A
        const uint32_t gb = p.gb[t], ab = p.ab[t];
        const uint32_t nb = mod_small(mod_small(rb * gb, mb, ib) * ainv, mb, ib);
        num_b[at] = __float2half_rn((float)balance(nb, mb));
        const uint32_t qm = (uint32_t)((uint64_t)s_q[g] % mb);
        const uint32_t d = mod_small(gb + mb - mod_small(qm * nb, mb, ib), mb, ib);
        state[at] = __float2half_rn((float)balance(mod_small(d * ab, mb, ib), mb));
    };
#pragma unroll
    for (uint32_t g = 0; g < kSetupNumbers; g++) {
        if (s_f[g] == kFlagRun) {
            const uint32_t a = mod_lazy(ra[g], ma, ia), b = mod_lazy(rb[g], mb, ib);
            slots(g, mod_small(a, ma, ia), mod_small(b, mb, ib), 1);
        } else {  // an all-zero lane
            const uint64_t at = slot_at(chunks, first + g, t);
            num_a[at] = num_b[at] = state[at] = __half(0.0f);
        }
    }
    __syncthreads();
    for (uint32_t g = 0; g < kSetupNumbers; g++) {
        if (s_f[g] != kFlagRun || s_divide[g] == 0 || s_out[g]) continue;  // the same for the whole block
        uint32_t by = 1;  // one or two primes of A, 16 bits each
        for (;;) {
            __syncthreads();
            const uint32_t m = s_by[g];
            const bool take = by == 1 || (by >> 16 == 0 && m != by);
            if (t == 0) {
                uint64_t r = 0;
                int top = -1;
                for (int w = (int)limbs - 1; w >= 0; w--) {
                    r = r << 32 | s_n[g][w];
                    s_n[g][w] = (uint32_t)(r / m);
                    if (top < 0 && s_n[g][w]) top = w;
                    r %= m;
                }
                s_divide[g] = 0;
                s_f[g] = take && near_widest(s_n[g], top, bits, a_mant, a_exp, s_q[g]) ? kFlagRun : kFlagOther;
            }
            __syncthreads();
            if (s_f[g] != kFlagRun) break;
            by = by == 1 ? m : by | m << 16;
            slots(g, limbs_mod(s_n[g], limbs, ma, ia), limbs_mod(s_n[g], limbs, mb, ib), by);
            __syncthreads();
            if (s_divide[g] == 0 || s_out[g]) break;
        }
        __syncthreads();
        if (t == 0) s_by[g] = by;
    }
    __syncthreads();
    if (t < kSetupNumbers && first + t < n_items) {
        flag[first + t] = s_out[t] ? kFlagComposite : s_f[t];
        quot[first + t] = s_q[t];
        factor[first + t] = s_by[t];
    }
}

// ---------------------------------------------------------------------------
// the chain of squarings

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t n) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(n) : "memory");
}

// Wait for the barrier's completion of the given parity; gives up after about
// a second, 2^18 tries of 3.8 us (gone: the caller stops waiting altogether).
__device__ __forceinline__ void mbar_wait(uint32_t bar, uint32_t parity, bool &gone) {
    if (gone) return;
    uint32_t ok = 0;
    for (uint32_t i = 0; i < (1u << 18); i++) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return;
    }
    gone = true;
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// One lane of a warp that is all here.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xFFFFFFFF;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r;
}

// Product d (+)= x b of the pair, issued by the lane that has `one`: the whole warp
// keeps its addresses, so that they stay in uniform registers (a single lane's
// would be moved there for every product: 2838 bits 14.8 us a step so, 10.0 now;
// 2136 bits 6.2 and 5.4).
__device__ __forceinline__ void multiply_pair(uint32_t one, uint32_t d, uint32_t x, uint64_t b, uint32_t instr,
                                              uint32_t add) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %4, 0;\n\tsetp.ne.u32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
        "r"(x), "l"(b), "r"(instr), "r"(add), "r"(one)
        : "memory");
}

// The barrier of both CTAs completes when the products issued so far are done.
__device__ __forceinline__ void commit_pair(uint32_t one, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}" ::
            "r"(bar),
        "h"((uint16_t)3), "r"(one)
        : "memory");
}

// The issuing warp's last act: where one of its waits gave up, the products still in
// flight end before TMEM is given back.  A commit covers what its own thread issued, so
// it comes from the lane that issued them, whichever lane gave up.
__device__ __forceinline__ void end_products(bool gone, uint32_t one, uint32_t bar) {
    if (!__any_sync(0xFFFFFFFFu, gone)) return;
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(bar),
        "r"(one)
        : "memory");
    bool late = false;
    mbar_wait(bar, 0, late);
}

__device__ __forceinline__ void tmem_ld8(uint32_t (&r)[8], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_ld4(uint32_t (&r)[4], uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
__device__ __forceinline__ void tmem_ld1(uint32_t &r, uint32_t addr) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r) : "r"(addr));
}
__device__ __forceinline__ void tmem_st4(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]),
                 "r"(r[2]), "r"(r[3])
                 : "memory");
}
// ... and what has come is not read before
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&a)[8], uint32_t (&b)[8], uint32_t &c) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7]),
                   "+r"(c)::"memory");
}
__device__ __forceinline__ void tmem_wait_ld(uint32_t (&a)[4]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3])::"memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Two f32 in one register pair, an operation on both per instruction.
typedef unsigned long long f2;
__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f2 pack2u(uint32_t a, uint32_t b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint32_t to_half2(f2 a) {
    float x, y;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(a));
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(y), "f"(x));
    return r;
}
__device__ __forceinline__ f2 from_half2(uint32_t h) {
    const float2 f = __half22float2(*reinterpret_cast<const __half2 *>(&h));
    return pack2(f.x, f.y);
}
__device__ __forceinline__ uint32_t hmul2(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}

// a b of both halves, exact in f32: one mixed-precision multiply-add each, where
// converting the halves first would take two more operations (2136 bits 12.8 ->
// 12.2 ms).  |a| <= 2048 and |b| <= 8192 are exact in f16.
__device__ __forceinline__ f2 mul_half2(uint32_t a, uint32_t b) {
    float x, y;
    asm("{\n\t.reg .b16 al, ah, bl, bh;\n\tmov.b32 {al, ah}, %2;\n\tmov.b32 {bl, bh}, %3;\n\t"
        "fma.rn.f32.f16 %0, al, bl, 0f00000000;\n\tfma.rn.f32.f16 %1, ah, bh, 0f00000000;\n\t}"
        : "=f"(x), "=f"(y)
        : "r"(a), "r"(b));
    return pack2(x, y);
}

// T mod m, balanced: T - m rint(T / m)
__device__ __forceinline__ f2 red2(f2 t, f2 neg_m, f2 inv_m, f2 magic, f2 neg_magic) {
    const f2 q = add2(fma2(t, inv_m, magic), neg_magic);
    return fma2(q, neg_m, t);
}
// (lo + hi) mod m, hi a multiple of 64 up to 2^30: the quotient from the rounded
// sum, the remainder's two parts exact
__device__ __forceinline__ f2 red_sum2(f2 lo, f2 hi, f2 neg_m, f2 inv_m, f2 magic, f2 neg_magic) {
    const f2 q = add2(fma2(add2(lo, hi), inv_m, magic), neg_magic);
    return add2(fma2(q, neg_m, hi), lo);
}

// The sums of C chunks to residues, 8 slots of a lane each.  w: the number's own
// constants, four: 1 or 4 (the squared doubling) in both halves.  A chain of some
// 20 dependent operations per pair of slots: two chunks at once keep eight going (with one
// store and one arrival per block: 1100 bits 3.9 -> 3.2 ms, 1750 bits 8.3 -> 7.5 for
// one pair, 2838 bits 27.8 -> 24.9).
struct Magic {
    f2 plus, minus;
};
template <uint32_t C>
__device__ __forceinline__ void residues_a(const SlotPair *chunk, const uint32_t (&lo2)[2][8],
                                           const uint32_t (&hi2)[2][8], f2 rank2, const uint32_t (&w2)[2][4],
                                           uint32_t four, const Magic &mg, uint32_t (&x2)[2][4], uint32_t first = 0) {
#pragma unroll
    for (uint32_t i = 0; i < 4 * C; i++) {
        const uint32_t h = first + (i & (C - 1)), j = i / C;  // the chunks' pairs in turn
        const SlotPair *sp = chunk + 16 * h;
        const auto &lo = lo2[h], &hi = hi2[h];
        const auto &w = w2[h];
        auto &x = x2[h];
        const f2 nm = pack2(sp[j].neg_m[0], sp[j].neg_m[1]), im = pack2(sp[j].inv_m[0], sp[j].inv_m[1]);
        const f2 l = fma2(rank2, pack2(sp[j].c[0], sp[j].c[1]), pack2u(lo[2 * j], lo[2 * j + 1]));
        const f2 r = red_sum2(l, pack2u(hi[2 * j], hi[2 * j + 1]), nm, im, mg.plus, mg.minus);
        const f2 u = red2(mul2(r, r), nm, im, mg.plus, mg.minus);
        const f2 v = mul_half2(to_half2(u), hmul2(w[j], four));
        x[j] = to_half2(red2(v, nm, im, mg.plus, mg.minus));
    }
}
template <uint32_t C>
__device__ __forceinline__ void residues_b(const SlotPair *chunk, const uint32_t (&lo2)[2][8],
                                           const uint32_t (&hi2)[2][8], const uint32_t (&old2)[2][4],
                                           const uint32_t (&w2)[2][4], uint32_t four, const Magic &mg,
                                           uint32_t (&x2)[2][4], uint32_t first = 0) {
#pragma unroll
    for (uint32_t i = 0; i < 4 * C; i++) {
        const uint32_t h = first + (i & (C - 1)), j = i / C;
        const SlotPair *sp = chunk + 16 * h;
        const auto &lo = lo2[h], &hi = hi2[h];
        const auto &w = w2[h], &old = old2[h];
        auto &x = x2[h];
        const f2 nm = pack2(sp[j].neg_m[0], sp[j].neg_m[1]), im = pack2(sp[j].inv_m[0], sp[j].inv_m[1]);
        const f2 r = red_sum2(pack2u(lo[2 * j], lo[2 * j + 1]), pack2u(hi[2 * j], hi[2 * j + 1]), nm, im, mg.plus,
                              mg.minus);
        const f2 t = mul_half2(old[j], hmul2(old[j], four));
        const f2 u = red2(t, nm, im, mg.plus, mg.minus);
        const f2 v = fma2(r, from_half2(w[j]), mul2(u, pack2(sp[j].c[0], sp[j].c[1])));
        x[j] = to_half2(red2(v, nm, im, mg.plus, mg.minus));
    }
}
// round(sum / 4096): the rank from its column
__device__ __forceinline__ f2 rank_of(uint32_t sum) {
    const float f = __fadd_rn(__fmaf_rn(__uint_as_float(sum), 1.0f / 4096.0f, kMagic), -kMagic);
    return pack2(f, f);
}

struct ChainArgs {
    const uint4 *matrices;   // [cta of the pair][product][chunk]
    const uint4 *num_a, *num_b;
    const uint4 *state;      // start
    uint4 *dumps;            // the last kRnsDumps values, the last first
    const uint32_t *nums;
    const unsigned long long *count;
    uint64_t max_items, dump_stride;  // in uint4
    unsigned long long *error;
    uint32_t limbs, steps;
};

// Up to seven chunks the matrices stay in shared memory and both A operands (of
// the product under way and of the next) lie in TMEM in full.  Above, the
// matrices' blocks go round a ring, copied from L2 ahead of each product (2838
// bits: 8.8 us a step; 9001 numbers 26 ms where the limb form takes 106), and the
// chunks from the eighth on have one place in TMEM: their residues are written
// when the product's last sums are in, and B's (needed again for the next square)
// are kept in shared memory.
template <uint32_t N>
struct ChainShape {
    static constexpr uint32_t K = kSlots * N;
    static constexpr uint32_t kBlocks = (N + 1) / 2;          // of 64 slots, the last of 32 for odd N
    static constexpr uint32_t kTwice = N < 7 ? N : 7;         // chunks with two places
    static constexpr bool kRing = N > 7;
    static constexpr uint32_t kWarpsAll = kWarps + (kRing ? 2 : 1);
    static constexpr uint32_t kBlockBytes = 64 * K * 2;       // of one CTA
    static constexpr uint32_t kKept = (N - kTwice) * 128 * 4 * 16;
    static constexpr uint32_t kSlotsOfRing = kRing ? (226 * 1024 - kKept) / kBlockBytes : 1;
    static constexpr uint32_t kShared = kRing ? kSlotsOfRing * kBlockBytes + kKept : 2 * K * K * 2;
    static constexpr uint32_t kXb = K / 2, kAcc = K / 2 + 16 * kTwice;  // TMEM columns
    static_assert(kAcc + 256 <= 512, "TMEM");
};

template <uint32_t N>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(32 * ChainShape<N>::kWarpsAll, 1)
    chain_kernel(const __grid_constant__ RnsConst kc, const __grid_constant__ ChainArgs a) {
    using S = ChainShape<N>;
    constexpr uint32_t K = S::K, kBlocks = S::kBlocks, kAcc = S::kAcc;
    constexpr uint32_t kBuffers = 2;  // of 128 accumulator columns
    constexpr uint32_t kCols = 512, kRingSlots = S::kSlotsOfRing;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_done[N], s_free[kBuffers], s_full[kBuffers], s_end;
    __shared__ __align__(8) uint64_t s_landed[kRingSlots], s_peer[kRingSlots], s_empty[kRingSlots];

    const uint64_t n_items = a.count ? min((uint64_t)*a.count, a.max_items) : a.max_items;
    const uint32_t pair = blockIdx.x / 2, rank = blockIdx.x & 1;
    if ((uint64_t)pair * kRnsTile >= n_items) return;  // both CTAs of the pair

    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x / 32, 0);
    const uint32_t lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                     "r"(kCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < N; i++) mbar_init(smem_addr(&s_done[i]), 2 * kWarps);
        for (uint32_t i = 0; i < kBuffers; i++) mbar_init(smem_addr(&s_full[i]), 1), mbar_init(smem_addr(&s_free[i]), 2 * kWarps);
        mbar_init(smem_addr(&s_end), 1);
        for (uint32_t i = 0; i < kRingSlots; i++)
            mbar_init(smem_addr(&s_landed[i]), 1), mbar_init(smem_addr(&s_peer[i]), 1),
                mbar_init(smem_addr(&s_empty[i]), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint4 *const matrices = a.matrices + (uint64_t)rank * (2 * K * K / 8);
    if constexpr (!S::kRing) {
        uint4 *dst = reinterpret_cast<uint4 *>(smem);
        for (uint32_t i = threadIdx.x; i < 2 * K * K / 8; i += kThreads) dst[i] = matrices[i];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor cores read it
    fence_before();
    __syncthreads();
    cluster_sync();
    fence_after();
    const uint32_t tmem = s_tmem;
    // chunk c of the A operand of product ph: even ones sum xi of B, odd ones of A
    const auto x_at = [](uint32_t ph, uint32_t c) { return 16 * c + ((ph & 1) && c < S::kTwice ? S::kXb : 0u); };
    bool gone = false;

    if (warp < kWarps) {
        const uint32_t wg = warp / 4;                           // its 8 slots of each chunk
        const uint32_t lanes = tmem + ((32 * (warp % 4)) << 16);  // its TMEM lanes
        const uint32_t row = 32 * (warp % 4) + lane;
        const uint64_t tile = (uint64_t)pair * 2 + rank;
        const uint64_t at0 = (tile * N * 4 + wg) * 128 + row;  // + 512 per chunk
        const uint64_t number = tile * 128 + row;
        const uint32_t *n_limbs = a.nums + (number < n_items ? number : 0) * a.limbs;
        uint32_t done0, free0;  // the leader's barriers
        asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(done0) : "r"(smem_addr(&s_done[0])));
        asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(free0) : "r"(smem_addr(&s_free[0])));
        auto arrive = [&](uint32_t bar) {
            fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
        };
        uint4 *const kept = reinterpret_cast<uint4 *>(smem + S::kShared - S::kKept) + wg * 128 + row;
        for (uint32_t c = 0; c < N; c++) {
            const uint4 v = a.state[at0 + 512 * c];
            const uint32_t x[4] = {v.x, v.y, v.z, v.w};
            tmem_st4(lanes + x_at(0, c) + 4 * wg, x);
            if (c >= S::kTwice) kept[(c - S::kTwice) * 512] = v;
            tmem_wait_st();
            // one arrival for the two chunks of a block (the late ones have their own)
            if (c % 2 == 1 || c + 1 >= S::kTwice) arrive(done0 + 8 * (c >= S::kTwice ? c : c & ~1u));
        }
        const Magic mg{pack2(kMagic, kMagic), pack2(-kMagic, -kMagic)};
        uint32_t seq = 0;  // blocks seen
        uint32_t word = 0;
        const auto load = [&](const uint4 *p, uint32_t c, uint32_t (&w)[4]) {
            const uint4 v = __ldg(p + at0 + 512 * c);
            w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
        };
        uint32_t lo[2][8], hi[2][8], rk = 0;
        const auto fetch = [&](uint32_t b, bool rank_too) {
            const bool two = 2 * b + 1 < N;
            const uint32_t acc = lanes + kAcc + 128 * (seq & 1) + 8 * wg, hi_at = two ? 64 : 32;
            mbar_wait(smem_addr(&s_full[seq & 1]), (seq >> 1) & 1, gone);
            fence_after();
            tmem_ld8(lo[0], acc);
            tmem_ld8(hi[0], acc + hi_at);
            if (two) {
                tmem_ld8(lo[1], acc + 32);
                tmem_ld8(hi[1], acc + hi_at + 32);
            }
            if (rank_too) tmem_ld1(rk, acc - 8 * wg);
        };
        // One product's sums to the residues of the next, a block of two chunks (8 slots each
        // per thread) at a time.  The numbers' constants are loaded a block ahead; the next
        // block's sums are on their way while this one's residues are stored.
        uint32_t cw[2][4];
        load(a.num_a, 0, cw[0]);
        if (N > 1) load(a.num_a, 1, cw[1]);
        f2 rank2 = 0;
        const auto product = [&](auto in_b, uint32_t four, uint32_t step) {
            constexpr bool kB = decltype(in_b)::value;
            constexpr uint32_t to = kB ? 0 : 1;  // parity of the product that these residues go to
            const uint4 *const nums = kB ? a.num_b : a.num_a, *const next = kB ? a.num_a : a.num_b;
            uint4 *const dump = kB && step + kRnsDumps >= a.steps
                                    ? a.dumps + (a.steps - 1 - step) * a.dump_stride + at0
                                    : nullptr;
            [[maybe_unused]] uint32_t late[N - S::kTwice + 1][4];
            const auto block = [&](uint32_t b, auto chunks) {
                constexpr uint32_t C = decltype(chunks)::value;
                uint32_t x[2][4];
                [[maybe_unused]] uint32_t old[2][4];
                if constexpr (kB) {
#pragma unroll
                    for (uint32_t h = 0; h < C; h++) {
                        const uint32_t c = 2 * b + h;
                        if (c < S::kTwice) {
                            tmem_ld4(old[h], lanes + x_at(0, c) + 4 * wg);
                        } else {
                            const uint4 v = kept[(c - S::kTwice) * 512];
                            old[h][0] = v.x, old[h][1] = v.y, old[h][2] = v.z, old[h][3] = v.w;
                        }
                    }
                }
                tmem_wait_ld(lo[0], hi[0], rk);
                if constexpr (C == 2) tmem_wait_ld(lo[1], hi[1], rk);
                if constexpr (kB) {
#pragma unroll
                    for (uint32_t h = 0; h < C; h++)
                        if (2 * b + h < S::kTwice) tmem_wait_ld(old[h]);
                }
                if constexpr (kBlocks > 2) arrive(free0 + 8 * (seq & 1));
                seq++;
                if (!kB && b == 0) rank2 = rank_of(rk);
                constexpr uint32_t kAtOnce = N == 8 ? 1 : C;  // (eight chunks: it would spill)
#pragma unroll
                for (uint32_t h = 0; h < C; h += kAtOnce) {
                    if constexpr (kB)
                        residues_b<kAtOnce>(kc.b + (32 * b + 4 * wg), lo, hi, old, cw, four, mg, x, h);
                    else
                        residues_a<kAtOnce>(kc.a + (32 * b + 4 * wg), lo, hi, rank2, cw, four, mg, x, h);
                }
#pragma unroll
                for (uint32_t h = 0; h < C; h++) {
                    const uint32_t c = 2 * b + h;
                    const uint4 v = make_uint4(x[h][0], x[h][1], x[h][2], x[h][3]);
                    if (c < S::kTwice) tmem_st4(lanes + x_at(to, c) + 4 * wg, x[h]);
                    if constexpr (N > 7) {
                        if (c == 7) late[0][0] = v.x, late[0][1] = v.y, late[0][2] = v.z, late[0][3] = v.w;
                        if constexpr (N > 8)
                            if (c == 8) late[1][0] = v.x, late[1][1] = v.y, late[1][2] = v.z, late[1][3] = v.w;
                    }
                    if constexpr (kB) {
                        if (c >= S::kTwice) kept[(c - S::kTwice) * 512] = v;
                        if (dump) dump[512 * c] = v;
                    }
                }
                // the next block's constants, or the next product's first
                const bool more = b + 1 < kBlocks;
                const uint32_t at = more ? 2 * b + 2 : 0;
                load(more ? nums : next, at, cw[0]);
                if (at + 1 < N) load(more ? nums : next, at + 1, cw[1]);
                if (more) fetch(b + 1, false);
                if (2 * b < S::kTwice) {
                    tmem_wait_st();
                    arrive(done0 + 16 * b);
                }
            };
            fetch(0, !kB);
            if constexpr (N > 1) {
#pragma unroll 1
                for (uint32_t b = 0; b < N / 2; b++) block(b, std::integral_constant<uint32_t, 2>{});
            }
            if constexpr (N % 2 == 1) block(N / 2, std::integral_constant<uint32_t, 1>{});
            if constexpr (N > 7) {  // the last block's sums are in: the product is done with their place
#pragma unroll
                for (uint32_t c = 7; c < N; c++) tmem_st4(lanes + x_at(to, c) + 4 * wg, late[c - 7]);
                tmem_wait_st();
#pragma unroll
                for (uint32_t c = 7; c < N; c++) arrive(done0 + 8 * c);
            }
        };
#pragma unroll 1
        for (uint32_t step = 0; step < a.steps; step++) {
            // the doubling that the last step's exponent bit asked for, squared
            uint32_t four = 0x3C003C00u;  // 1, 1
            if (step > 0) {
                const uint32_t at = a.steps - step + 1;  // bit of N: bit steps - step of (N - 1)/2
                if (step == 1 || (at & 31) == 31) word = n_limbs[at >> 5];
                if ((word >> (at & 31)) & 1) four = 0x44004400u;  // 4, 4
            }
            product(std::false_type{}, four, step);  // sums of xi over B -> x in A -> xi in A
            product(std::true_type{}, four, step);   // sums of xi over A -> q in B -> xi in B
        }
    } else if (warp == kWarps && rank == 0) {
        const uint32_t one = elect_one();
        // f16 operands, f32 sums, both K-major, M = 256
        constexpr uint32_t kInstr = (1u << 4) | ((256 / 16) << 24);
        const uint32_t base = smem_addr(smem);
        uint32_t seq = 0;
        for (uint32_t ph = 0; ph < 2 * a.steps; ph++) {
            for (uint32_t b = 0; b < kBlocks; b++, seq++) {
                const uint32_t d = tmem + kAcc + 128 * (seq & 1);
                const uint32_t slots = 2 * b + 1 < N ? 64 : 32;  // columns: twice that
                const uint32_t ring = seq % kRingSlots;
                const uint32_t block = base + (S::kRing ? ring * S::kBlockBytes : (ph & 1) * (2 * K * K) + b * S::kBlockBytes);
                // 8 x 8 pieces of 128 bytes, unswizzled: slots 128 bytes apart, k a row of them
                const uint32_t row = slots / 8 * 128;
                const uint64_t desc = (uint64_t)((block & 0x3FFFF) >> 4) | ((uint64_t)(row / 16) << 16) |
                                      ((uint64_t)(128 / 16) << 32) | (1ull << 46);
                const uint32_t instr = kInstr | (slots * 2 / 8) << 17;
                const auto multiply = [&](uint32_t kk) {
                    multiply_pair(one, d, tmem + x_at(ph, kk / 2) + 8 * (kk & 1), desc + kk * (2 * row / 16), instr, kk);
                };
                // the buffer's last sums have been read; the block is there in both CTAs
                // (up to two blocks: before any of this product's residues were there)
                if (kBlocks > 2 && seq >= kBuffers)
                    mbar_wait(smem_addr(&s_free[seq & 1]), (seq / kBuffers - 1) & 1, gone);
                if constexpr (S::kRing) {
                    mbar_wait(smem_addr(&s_landed[ring]), (seq / kRingSlots) & 1, gone);
                    mbar_wait(smem_addr(&s_peer[ring]), (seq / kRingSlots) & 1, gone);
                }
                fence_after();
                if (b == 0) {  // slice by slice, as the residues appear
#pragma unroll
                    for (uint32_t i = 0; i < N; i++) {
                        if (i % 2 == 0 || i >= S::kTwice) {
                            mbar_wait(smem_addr(&s_done[i]), ph & 1, gone);
                            fence_after();
                        }
                        multiply(2 * i);
                        multiply(2 * i + 1);
                    }
                } else {
#pragma unroll
                    for (uint32_t kk = 0; kk < 2 * N; kk++) multiply(kk);
                }
                commit_pair(one, smem_addr(&s_full[seq & 1]));
                if constexpr (S::kRing) commit_pair(one, smem_addr(&s_empty[ring]));
            }
        }
        end_products(gone, one, smem_addr(&s_end));
    } else if (S::kRing && warp == kWarps && lane == 0) {
        // the other CTA's half of each block has landed: tell the one that multiplies
        uint32_t peer0;
        asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(peer0) : "r"(smem_addr(&s_peer[0])));
        for (uint32_t seq = 0; seq < 2 * a.steps * kBlocks; seq++) {
            mbar_wait(smem_addr(&s_landed[seq % kRingSlots]), (seq / kRingSlots) & 1, gone);
            asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(peer0 + 8 * (seq % kRingSlots)) : "memory");
        }
    } else if (S::kRing && warp == kWarps + 1 && lane == 0) {
        // this CTA's half of each block, in the order in which the products use them
        uint32_t seq = 0;
        for (uint32_t ph = 0; ph < 2 * a.steps; ph++) {
            for (uint32_t b = 0; b < kBlocks; b++, seq++) {
                const uint32_t ring = seq % kRingSlots;
                const uint32_t bytes = 2 * b + 1 < N ? S::kBlockBytes : S::kBlockBytes / 2;
                if (seq >= kRingSlots) mbar_wait(smem_addr(&s_empty[ring]), (seq / kRingSlots - 1) & 1, gone);
                if (gone) break;  // nothing more is asked for
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&s_landed[ring])),
                             "r"(bytes)
                             : "memory");
                asm volatile(
                    "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                        smem_addr(smem + ring * S::kBlockBytes)),
                    "l"((const char *)matrices + (size_t)(ph & 1) * (2 * K * K) + (size_t)b * S::kBlockBytes), "r"(bytes),
                    "r"(smem_addr(&s_landed[ring]))
                    : "memory");
            }
            if (gone) break;
        }
        if (gone) {  // copies in flight land before the CTA ends
            bool late = false;
            for (uint32_t i = seq > kRingSlots ? seq - kRingSlots : 0; i < seq; i++)
                mbar_wait(smem_addr(&s_landed[i % kRingSlots]), (i / kRingSlots) & 1, late);
        }
    }
    if (gone) atomicExch(a.error, 1ull);
    fence_before();
    __syncthreads();
    cluster_sync();
    fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kCols));
}

// The same chain with T tiles of 256 numbers per pair, taken in turn: a tile's
// two exchanges per squaring (residues written, product, sums ready: some 1300
// cycles) pass while the other tiles' residues are computed.  A tile has one A
// operand in TMEM: the next one replaces it when its product's last sums are in,
// so a product's residues wait in registers; B's residues, needed again for the
// next square, are kept in shared memory (what does not fit, in TMEM).
// 38912 numbers of 2120 bits: 19.4 ms against 21.9 ms in two single waves (38912 of 1060
// bits 5.2, 5.1; 58368 of 700 bits 3.4, three waves 4.0; 77824 of 340 bits 1.33, four
// waves 1.47), the f32 pipe 68 % busy, the tensor cores 52 %.
// Reading the next sums while residues are computed made it slower here (24.9 ms;
// two chunks at once 24.1).
template <uint32_t N, uint32_t T>
struct TilesShape {
    static constexpr uint32_t K = kSlots * N;
    static constexpr uint32_t kMatrices = 2 * K * K * 2;
    static constexpr uint32_t kChunk = 128 * 4 * 16;  // one tile's residues of one chunk, bytes
    static constexpr uint32_t kRoom = (226 * 1024 - kMatrices) / (T * kChunk);
    static constexpr uint32_t kOldShared = kRoom < N ? kRoom : N;  // chunks in shared memory
    static constexpr uint32_t kShared = kMatrices + T * kOldShared * kChunk;
    static constexpr uint32_t kAcc = T * K / 2, kOld = kAcc + 256;  // TMEM columns
    static_assert(kOld + T * (N - kOldShared) * 16 <= 512, "TMEM");
};

template <uint32_t N, uint32_t T>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kThreads, 1)
    chain_tiles_kernel(const __grid_constant__ RnsConst kc, const __grid_constant__ ChainArgs a) {
    using S = TilesShape<N, T>;
    constexpr uint32_t K = S::K;
    constexpr uint32_t kBlocks = (N + 1) / 2;  // of 64 slots, the last of 32 for odd N
    constexpr uint32_t kBuffers = 2;           // of 128 accumulator columns
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_done[T], s_free[kBuffers], s_full[kBuffers], s_end;

    const uint64_t n_items = a.count ? min((uint64_t)*a.count, a.max_items) : a.max_items;
    const uint32_t pair = blockIdx.x / 2, rank = blockIdx.x & 1;
    if ((uint64_t)pair * (T * kRnsTile) >= n_items) return;  // both CTAs of the pair

    const uint32_t warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x / 32, 0);
    const uint32_t lane = threadIdx.x & 31;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    }
    if (threadIdx.x == 0) {
        for (uint32_t i = 0; i < T; i++) mbar_init(smem_addr(&s_done[i]), 2 * kWarps);
        for (uint32_t i = 0; i < kBuffers; i++)
            mbar_init(smem_addr(&s_full[i]), 1), mbar_init(smem_addr(&s_free[i]), 2 * kWarps);
        mbar_init(smem_addr(&s_end), 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    {
        const uint4 *src = a.matrices + (uint64_t)rank * (2 * K * K / 8);
        uint4 *dst = reinterpret_cast<uint4 *>(smem);
        for (uint32_t i = threadIdx.x; i < 2 * K * K / 8; i += kThreads) dst[i] = src[i];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tensor cores read it
    fence_before();
    __syncthreads();
    cluster_sync();
    fence_after();
    const uint32_t tmem = s_tmem;
    bool gone = false;

    if (warp < kWarps) {
        const uint32_t wg = warp / 4;                           // its 8 slots of each chunk
        const uint32_t lanes = tmem + ((32 * (warp % 4)) << 16);  // its TMEM lanes
        const uint32_t row = 32 * (warp % 4) + lane;
        const uint64_t tile0 = (uint64_t)pair * (2 * T) + rank;  // + 2 per tile
        const uint64_t at0 = (tile0 * N * 4 + wg) * 128 + row;   // + 512 per chunk
        constexpr uint32_t kTileStep = 2 * N * 512;
        uint4 *const old_shared = reinterpret_cast<uint4 *>(smem + S::kMatrices) + wg * 128 + row;
        uint32_t done0, free0;  // the leader's barriers
        asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(done0) : "r"(smem_addr(&s_done[0])));
        asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(free0) : "r"(smem_addr(&s_free[0])));
        auto arrive = [&](uint32_t bar) {
            fence_before();
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(bar) : "memory");
        };
        auto keep = [&](uint32_t t, uint32_t c, const uint32_t (&x)[4]) {
            if (c < S::kOldShared)
                old_shared[(t * S::kOldShared + c) * 512] = make_uint4(x[0], x[1], x[2], x[3]);
            else
                tmem_st4(lanes + S::kOld + (t * (N - S::kOldShared) + c - S::kOldShared) * 16 + 4 * wg, x);
        };
        auto kept = [&](uint32_t t, uint32_t c, uint32_t (&x)[4]) {
            if (c < S::kOldShared) {
                const uint4 v = old_shared[(t * S::kOldShared + c) * 512];
                x[0] = v.x, x[1] = v.y, x[2] = v.z, x[3] = v.w;
            } else {
                tmem_ld4(x, lanes + S::kOld + (t * (N - S::kOldShared) + c - S::kOldShared) * 16 + 4 * wg);
                tmem_wait_ld(x);
            }
        };
        for (uint32_t t = 0; t < T; t++) {
            for (uint32_t c = 0; c < N; c++) {
                const uint4 v = a.state[at0 + t * kTileStep + 512 * c];
                const uint32_t x[4] = {v.x, v.y, v.z, v.w};
                tmem_st4(lanes + t * (K / 2) + 16 * c + 4 * wg, x);
                keep(t, c, x);
            }
            tmem_wait_st();
            arrive(done0 + 8 * t);
        }
        const Magic mg{pack2(kMagic, kMagic), pack2(-kMagic, -kMagic)};
        // a tile's limb that holds the exponent bit of a step
        const auto limb = [&](uint32_t t, uint32_t step) {
            const uint64_t number = (tile0 + 2 * t) * 128 + row;
            return __ldg(a.nums + (number < n_items ? number : 0) * a.limbs + ((a.steps - step + 1) >> 5));
        };
        const auto load = [&](const uint4 *p, uint32_t t, uint32_t c, uint32_t (&w)[4]) {
            const uint4 v = __ldg(p + at0 + t * kTileStep + 512 * c);
            w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
        };
        uint32_t seq = 0;  // blocks seen
        uint32_t cw[2][4], word = 0;
        load(a.num_a, 0, 0, cw[0]);
        if (N > 1) load(a.num_a, 0, 1, cw[1]);
        // one tile's sums of one product to the A operand of its next; the constants and the
        // limb of what comes after are loaded on the way
        const auto product = [&](auto in_b, uint32_t step, uint32_t t) {
            constexpr bool kB = decltype(in_b)::value;
            const uint4 *const nums = kB ? a.num_b : a.num_a;
            const bool last_tile = t + 1 == T;
            const uint4 *const next = last_tile ? (kB ? a.num_a : a.num_b) : nums;
            const uint32_t next_t = last_tile ? 0 : t + 1;
            const uint32_t next_step = last_tile && kB && step + 1 < a.steps ? step + 1 : step;
            const uint32_t bit = a.steps - step + 1;
            const uint32_t four = step > 0 && ((word >> (bit & 31)) & 1) ? 0x44004400u : 0x3C003C00u;  // 4, 4 or 1, 1
            word = limb(next_t, next_step);
            const bool dump = kB && step + kRnsDumps >= a.steps;
            f2 rank2 = 0;
            uint32_t x[kBlocks][2][4];
#pragma unroll
            for (uint32_t b = 0; b < kBlocks; b++) {
                const bool two = 2 * b + 1 < N;
                const uint32_t acc = lanes + S::kAcc + 128 * (seq & 1) + 8 * wg, hi_at = two ? 64 : 32;
                mbar_wait(smem_addr(&s_full[seq & 1]), (seq >> 1) & 1, gone);
                fence_after();
                uint32_t lo[2][8], hi[2][8], rk = 0;
                tmem_ld8(lo[0], acc);
                tmem_ld8(hi[0], acc + hi_at);
                if (two) {
                    tmem_ld8(lo[1], acc + 32);
                    tmem_ld8(hi[1], acc + hi_at + 32);
                }
                if (!kB && b == 0) tmem_ld1(rk, acc - 8 * wg);
                tmem_wait_ld(lo[0], hi[0], rk);
                if (two) tmem_wait_ld(lo[1], hi[1], rk);
                arrive(free0 + 8 * (seq & 1));
                seq++;
                if (!kB && b == 0) rank2 = rank_of(rk);
#pragma unroll
                for (uint32_t h = 0; h < (two ? 2 : 1); h++) {
                    const uint32_t c = 2 * b + h;
                    if (kB) {
                        uint32_t old[2][4];
                        kept(t, c, old[h]);
                        residues_b<1>(kc.b + (32 * b + 4 * wg), lo, hi, old, cw, four, mg, x[b], h);
                        keep(t, c, x[b][h]);
                        if (dump)
                            a.dumps[(a.steps - 1 - step) * a.dump_stride + at0 + t * kTileStep + 512 * c] =
                                make_uint4(x[b][h][0], x[b][h][1], x[b][h][2], x[b][h][3]);
                    } else {
                        residues_a<1>(kc.a + (32 * b + 4 * wg), lo, hi, rank2, cw, four, mg, x[b], h);
                    }
                    const bool more = b + 1 < kBlocks;
                    const uint32_t at = more ? 2 * b + 2 + h : h;
                    if (at < N) load(more ? nums : next, more ? t : next_t, at, cw[h]);
                    // odd N: the second chunk of what comes next, where this block has none
                    if (!two && !more && N > 1) load(next, next_t, 1, cw[1]);
                }
            }
            // the last block's sums are in: every product with the old operand is done
#pragma unroll
            for (uint32_t c = 0; c < N; c++) tmem_st4(lanes + t * (K / 2) + 16 * c + 4 * wg, x[c / 2][c % 2]);
            tmem_wait_st();
            arrive(done0 + 8 * t);
        };
#pragma unroll 1
        for (uint32_t step = 0; step < a.steps; step++) {
#pragma unroll 1
            for (uint32_t t = 0; t < T; t++) product(std::false_type{}, step, t);
#pragma unroll 1
            for (uint32_t t = 0; t < T; t++) product(std::true_type{}, step, t);
        }
    } else if (rank == 0) {
        const uint32_t one = elect_one();
        constexpr uint32_t kInstr = (1u << 4) | ((256 / 16) << 24);
        const uint32_t base = smem_addr(smem);
        uint32_t seq = 0;
        for (uint32_t ph = 0; ph < 2 * a.steps; ph++) {
            for (uint32_t t = 0; t < T; t++) {
                const uint32_t x = tmem + t * (K / 2);
                mbar_wait(smem_addr(&s_done[t]), ph & 1, gone);
                for (uint32_t b = 0; b < kBlocks; b++, seq++) {
                    const uint32_t d = tmem + S::kAcc + 128 * (seq & 1);
                    const uint32_t slots = 2 * b + 1 < N ? 64 : 32, r = slots / 8 * 128;
                    if (seq >= kBuffers) mbar_wait(smem_addr(&s_free[seq & 1]), (seq / kBuffers - 1) & 1, gone);
                    fence_after();
                    const uint32_t from = base + (ph & 1 ? 2 * K * K : 0) + b * (64 * K * 2);
                    const uint64_t desc = (uint64_t)((from & 0x3FFFF) >> 4) | ((uint64_t)(r / 16) << 16) |
                                          ((uint64_t)(128 / 16) << 32) | (1ull << 46);
#pragma unroll
                    for (uint32_t kk = 0; kk < 2 * N; kk++)
                        multiply_pair(one, d, x + 8 * kk, desc + kk * (2 * r / 16), kInstr | (slots * 2 / 8) << 17, kk);
                    commit_pair(one, smem_addr(&s_full[seq & 1]));
                }
            }
        }
        end_products(gone, one, smem_addr(&s_end));
    }
    if (gone) atomicExch(a.error, 1ull);
    fence_before();
    __syncthreads();
    cluster_sync();
    fence_after();
    if (warp == 0)
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// ---------------------------------------------------------------------------
// verdicts: a warp per number.  The value after the last squarings (f times, f
// its exponent bit's doubling) is +-1 exactly when f x -+ (A mod N) is t N for
// one small t, in every modulus of B (their product is above the difference's
// range): f xi/A -+ ((B/m)^-1 - q n) = t n mod m.
__global__ void verdict_kernel(const __grid_constant__ RnsSlots p, uint32_t chunks, uint32_t steps, uint32_t t_max,
                               uint32_t limbs, const unsigned long long *count, uint64_t max_items,
                               const __half *__restrict__ num_b, const __half *__restrict__ dumps, uint64_t dump_stride,
                               const uint32_t *__restrict__ nums, const long long *__restrict__ quot,
                               const uint32_t *__restrict__ flag, const uint32_t *__restrict__ factor,
                               uint32_t first, uint8_t *__restrict__ result, uint32_t *__restrict__ list,
                               unsigned long long *__restrict__ listed) {
    const uint64_t n_items = count ? min((uint64_t)*count, max_items) : max_items;
    const uint64_t i = (uint64_t)blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    if (i >= n_items) return;
    const uint32_t lane = threadIdx.x & 31;
    uint32_t f = flag[i];
    const uint32_t *n = nums + i * limbs;
    if (f == kFlagRun) {
        uint32_t s = 0;  // trailing zeros of N - 1
        for (uint32_t w = 0; w < limbs; w++) {
            const uint32_t v = n[w] - (w == 0);
            if (v) {
                s = 32 * w + (uint32_t)__ffs(v) - 1;
                break;
            }
        }
        const uint32_t k = kSlots * chunks;
        const long long q = quot[i];
        const uint32_t last = min(min(kRnsDumps, s), steps);
        f = kFlagOther;
        bool prime = false;
        for (uint32_t d = 0; d < last && f == kFlagOther; d++) {
            const int twice = (int)((n[(d + 1) >> 5] >> ((d + 1) & 31)) & 1) + 1;
            int sign = 1;
            bool have = true, ok = false;
            for (; sign >= -1 && !ok && have; sign -= 2) {
                int t = 0;
                ok = true;
                for (uint32_t base = 0; base < k && ok; base += 32) {
                    const uint32_t j = base + lane;
                    const int m = (int)p.mb[j];
                    const uint64_t at = slot_at(chunks, i, j);
                    const int xi = (int)__half2float(dumps[d * dump_stride + at]), nb = (int)__half2float(num_b[at]);
                    const int ainv = (int)inverse_small(p.ab[j], (uint32_t)m);
                    const int one = ((int)p.gb[j] - (int)(q % m) * nb) % m;
                    int lhs = (twice * xi % m * ainv - sign * one) % m;
                    if (lhs < 0) lhs += m;
                    const uint32_t nn = (uint32_t)(nb < 0 ? nb + m : nb);
                    if (base == 0) {  // t from the first prime modulus that N is a unit of
                        const uint32_t units = __ballot_sync(0xFFFFFFFFu, nn != 0 && j < p.b_primes);
                        have = units != 0;
                        const uint32_t inv = inv32_of((uint32_t)m);
                        const int w = balance(
                            mod_small((uint32_t)lhs * pow_small(nn, (uint32_t)m - 2, (uint32_t)m, inv), (uint32_t)m, inv),
                            (uint32_t)m);
                        t = __shfl_sync(0xFFFFFFFFu, w, have ? __ffs(units) - 1 : 0);
                        ok = have && (uint32_t)abs(t) <= t_max;
                    }
                    ok = __all_sync(0xFFFFFFFFu, (lhs - t * (int)nn) % m == 0) && ok;
                }
            }
            if (!have) break;                                     // N shares a factor with them all
            for (uint32_t rest = factor[i]; ok && rest > 1; rest >>= 16) {
                // the chain ran without this factor: 2^((N - 1) / 2^(d + 1)) mod it has to agree
                const uint32_t by = rest & 0xFFFFu;
                const uint32_t e = by - 1, ie = inv32_of(e), sh = d + 1;
                uint32_t r = 0;
                for (int w = (int)limbs - 1; w >= 0; w--) {
                    const uint32_t up = w + 1 < (int)limbs ? n[w + 1] : 0u;
                    const uint32_t v = __funnelshift_r(n[w], up, sh);
                    r = mod_lazy((r << 16) | (v >> 16), e, ie);
                    r = mod_lazy((r << 16) | (v & 0xFFFFu), e, ie);
                }
                const uint32_t z = pow_small(2, r, by, inv32_of(by));
                ok = z == (sign == -3 ? by - 1 : 1u);
            }
            if (!ok) f = kFlagRun;                                // neither: composite
            else if (sign == -3) f = kFlagRun, prime = true;      // -1 on the way
            else if (d + 1 == s) f = kFlagRun, prime = true;      // 1 from the start
        }
        if (f == kFlagRun && lane == 0) result[i] = prime;
    } else if (f == kFlagComposite && lane == 0) {
        result[i] = 0;
    }
    if (f == kFlagOther && lane == 0) list[atomicAdd(listed, 1ull)] = first + (uint32_t)i;
}

// Tiles per pair: enough that their residues take longer than one tile's exchange.
constexpr uint32_t kTilesOf[kRnsMaxChunks + 1] = {0, 4, 3, 2, 2, 2, 2, 1, 1, 1};

// Pairs of CTAs that run at once, one CTA per SM (asked of each device once: the search's
// expectations ask hundreds of times).
uint64_t pairs_at_once() {
    static std::atomic<int> known[64];
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return 76;
    const bool keep = device >= 0 && device < 64;
    if (keep) sms = known[device].load(std::memory_order_relaxed);
    if (sms == 0) {
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms < 2) return 76;
        if (keep) known[device].store(sms, std::memory_order_relaxed);
    }
    return (uint64_t)sms / 2;
}

// A group of tiles takes a little less than its tiles one after another, whether it is
// full or not: it runs where single tiles would need a wave for each of its places.
// (20000 numbers, two waves of single tiles, and a group's wave: 300 bits 1.23, 1.59
// ms; 500 bits 2.53, 2.66; 764 bits 4.1, 4.1; 1250 bits 9.5, 8.5; 1814 bits 19.6, 17.8.)
bool group_pays(uint32_t chunks, uint64_t tiles) {
    return kTilesOf[chunks] > 1 && tiles > (kTilesOf[chunks] - 1) * pairs_at_once();
}

template <uint32_t N, uint32_t T>
cudaError_t launch_tiles(const RnsPlan &p, const ChainArgs &a, uint64_t tiles, cudaStream_t s) {
    constexpr uint32_t least = 118 * 1024;  // one CTA per SM, as below
    constexpr uint32_t bytes = TilesShape<N, T>::kShared > least ? TilesShape<N, T>::kShared : least;
    cudaError_t e = cudaFuncSetAttribute(chain_tiles_kernel<N, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    chain_tiles_kernel<N, T><<<(unsigned)(2 * ((tiles + T - 1) / T)), kThreads, bytes, s>>>(p.k, a);
    return cudaGetLastError();
}

template <uint32_t N>
cudaError_t launch_chain(const RnsPlan &p, const ChainArgs &a, uint64_t tiles, cudaStream_t s) {
    if constexpr (N < 7) {
        if (group_pays(N, tiles)) return launch_tiles<N, kTilesOf[N]>(p, a, tiles, s);
    }
    // at least half of the SM's shared memory: a second CTA would wait for TMEM
    // columns, and two pairs could each hold what the other waits for
    using S = ChainShape<N>;
    constexpr uint32_t bytes = S::kShared > 118 * 1024 ? S::kShared : 118 * 1024;
    cudaError_t e = cudaFuncSetAttribute(chain_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e != cudaSuccess) return e;
    chain_kernel<N><<<(unsigned)(2 * tiles), 32 * S::kWarpsAll, bytes, s>>>(p.k, a);
    return cudaGetLastError();
}

template <typename T>
T *at(void *work, size_t off) {
    return reinterpret_cast<T *>((char *)work + off);
}

}  // namespace

uint32_t rns_chunks(uint32_t bits) {
    for (uint32_t n = 1; n <= kRnsMaxChunks; n++)
        if ((double)bits + 1e-6 <= moduli_of(n).bits) return n;
    return 0;
}

uint64_t rns_wave(uint32_t bits, bool full) {
    return pairs_at_once() * kRnsTile * (full ? kTilesOf[rns_chunks(bits)] : 1);
}

uint64_t rns_slice(uint32_t bits, uint64_t left) {
    const uint64_t tiles = (left + kRnsTile - 1) / kRnsTile;
    return std::min(left, rns_wave(bits, group_pays(rns_chunks(bits), tiles)));
}

// A launch of one wave: per bit a step's time of one tile or of a group (the widest
// numbers of each chunk count, 16 and 38912 of them), and the set-up and verdicts.
double rns_us(uint32_t bits, uint64_t items) {
    constexpr double kStep[kRnsMaxChunks + 1] = {0, 1.05, 1.88, 2.36, 3.5, 4.22, 5.13, 5.95, 7.43, 8.75};
    constexpr double kGroupStep[kRnsMaxChunks + 1] = {0, 4.2, 4.6, 4.8, 6.5, 8.6, 9.6};
    const uint32_t n = rns_chunks(bits);
    double us = 0;
    for (uint64_t left = items; left > 0;) {
        const uint64_t take = rns_slice(bits, left);
        us += 20 + bits * (group_pays(n, (left + kRnsTile - 1) / kRnsTile) ? kGroupStep[n] : kStep[n]);
        left -= take;
    }
    return us + 0.0025 * n * (double)items;
}

RnsLayout rns_layout(uint32_t bits, uint32_t limbs, uint64_t max_items, uint64_t all_items) {
    RnsLayout l{};
    l.chunks = rns_chunks(bits);
    l.limbs = limbs;
    l.tiles = (max_items + kRnsTile - 1) / kRnsTile + kRnsGroup - 1;  // a last group's empty tiles
    const size_t k = kSlots * l.chunks, numbers = l.tiles * kRnsTile;
    size_t off = 0;
    auto take = [&](size_t bytes) {
        const size_t o = off;
        off += (bytes + 255) & ~(size_t)255;
        return o;
    };
    l.matrices = take(2 * 2 * k * k * 2);
    l.num_a = take(numbers * k * 2);
    l.num_b = take(numbers * k * 2);
    l.state = take(numbers * k * 2);
    l.dumps = take(kRnsDumps * numbers * k * 2);
    l.nums = take(numbers * limbs * 4);
    l.quot = take(numbers * 8);
    l.flag = take(numbers * 4);
    l.factor = take(numbers * 4);
    l.list = take(all_items * 4);
    l.counters = take(16);
    l.total = off;
    return l;
}

cudaError_t rns_begin(const RnsLayout &l, uint32_t bits, void *work, cudaStream_t s) {
    const RnsPlan &p = plan_of(l.chunks, bits);
    const uint32_t k = kSlots * l.chunks;
    matrix_kernel<<<(2 * k * k + 255) / 256, 256, 0, s>>>(p.s, l.chunks, at<__half>(work, l.matrices));
    const cudaError_t e = cudaGetLastError();
    return e != cudaSuccess ? e : cudaMemsetAsync(at<char>(work, l.counters), 0, 16, s);
}

cudaError_t rns_test(const RnsLayout &l, uint32_t bits, void *work, const uint32_t *bases, const PrpItem *items,
                     uint64_t first, const unsigned long long *count, uint64_t max_items, uint8_t *result,
                     cudaStream_t s) {
    if (max_items == 0) return cudaSuccess;
    const RnsPlan &p = plan_of(l.chunks, bits);
    const uint32_t k = kSlots * l.chunks;
    const uint64_t tiles = (max_items + kRnsTile - 1) / kRnsTile, numbers = l.tiles * kRnsTile;
    const uint32_t steps = bits - 1;
    cudaError_t e = first == 0 ? cudaMemsetAsync(at<char>(work, l.counters), 0, 8, s) : cudaSuccess;
    if (e != cudaSuccess) return e;
    setup_kernel<<<(unsigned)((tiles + kRnsGroup - 1) * (kRnsTile / kSetupNumbers)), k, 0, s>>>(
        p.s, l.chunks, bits, p.a_mant, p.a_exp, l.limbs, bases, items + first, count, max_items, at<__half>(work, l.num_a),
        at<__half>(work, l.num_b), at<__half>(work, l.state), at<uint32_t>(work, l.nums), at<long long>(work, l.quot),
        at<uint32_t>(work, l.flag), at<uint32_t>(work, l.factor));
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const ChainArgs a{at<uint4>(work, l.matrices), at<uint4>(work, l.num_a), at<uint4>(work, l.num_b),
                      at<uint4>(work, l.state),    at<uint4>(work, l.dumps), at<uint32_t>(work, l.nums),
                      count,                       max_items,                numbers * k / 8,
                      at<unsigned long long>(work, l.counters) + 1,          l.limbs,
                      steps};
    switch (l.chunks) {
        case 1: e = launch_chain<1>(p, a, tiles, s); break;
        case 2: e = launch_chain<2>(p, a, tiles, s); break;
        case 3: e = launch_chain<3>(p, a, tiles, s); break;
        case 4: e = launch_chain<4>(p, a, tiles, s); break;
        case 5: e = launch_chain<5>(p, a, tiles, s); break;
        case 6: e = launch_chain<6>(p, a, tiles, s); break;
        case 7: e = launch_chain<7>(p, a, tiles, s); break;
        case 8: e = launch_chain<8>(p, a, tiles, s); break;
        case 9: e = launch_chain<9>(p, a, tiles, s); break;
        default: return cudaErrorInvalidValue;
    }
    if (e != cudaSuccess) return e;
    verdict_kernel<<<(unsigned)((max_items + 3) / 4), 128, 0, s>>>(
        p.s, l.chunks, steps, p.t_max, l.limbs, count, max_items, at<__half>(work, l.num_b), at<__half>(work, l.dumps),
        numbers * k, at<uint32_t>(work, l.nums), at<long long>(work, l.quot), at<uint32_t>(work, l.flag),
        at<uint32_t>(work, l.factor), (uint32_t)first, result + first, at<uint32_t>(work, l.list),
        at<unsigned long long>(work, l.counters));
    return cudaGetLastError();
}

}  // namespace pg
