// The moduli of the residue number system (pg_rns.cu): which they are, what they hold, and
// that every sum over them is exact.  Host code.
#pragma once
#include <stdint.h>

#include <cmath>
#include <vector>

namespace pg {

constexpr uint32_t kSlots = 32;        // residue slots per chunk
constexpr uint32_t kRnsMaxChunks = 9;  // chunks

// The moduli of 32n slots in each base and the bits that they hold.  A takes
// primes alone (N has to be a unit there); B ends with composite moduli near
// 4096 made of small primes of their own, which hold more than the primes that
// they stand in for (2136-bit numbers fit six chunks, not seven).
struct RnsModuli {
    std::vector<uint32_t> a, b;
    uint32_t b_primes = 0;
    double bits = 0;  // numbers below 2^bits
};

inline double log2_product(const std::vector<uint32_t> &v) {
    double l = 0;
    for (uint32_t q : v) l += std::log2((double)q);
    return l;
}

// |x| <= c N; 4 c^2 N <= A and c N <= B / 4
inline double coefficient(size_t k) { return 0.5 * (double)k + 1; }
inline double a_capacity(double log_a, size_t k) { return log_a - 2 - 2 * std::log2(coefficient(k)); }

// Whether the f32 sums over residues of these moduli, |xi| <= m/2 + 1, are whole numbers
// below 2^24: the low parts |lo| <= 32 with the rank's correction (a rank up to half the
// slots times a residue), and the high parts in units of 64, |hi| <= 32 of them.  (Widest
// numbers of nine chunks: 0.55 of 2^24.)
inline bool sums_exact(const std::vector<uint32_t> &moduli) {
    uint64_t sum = 0;
    for (uint32_t m : moduli) sum += 32ull * (m / 2 + 1);
    return sum + (moduli.size() / 2 + 1) * 2048ull < 1ull << 24;
}

inline RnsModuli make_moduli(uint32_t n) {
    const uint32_t k = kSlots * n;
    std::vector<uint8_t> comp(4097, 0), used(4097, 0);
    std::vector<uint32_t> primes, extra;
    for (uint32_t q = 2; q <= 4096; q++) {
        if (comp[q]) continue;
        primes.push_back(q);
        for (uint32_t t = q * q; t <= 4096; t += q) comp[t] = 1;
    }
    for (uint32_t c = 4096; c > 3900; c--) {
        std::vector<uint32_t> f;
        uint32_t rest = c;
        for (uint32_t q : primes) {
            if (q > 200) break;
            if (rest % q == 0 && !used[q]) f.push_back(q);
            while (rest % q == 0 && !used[q]) rest /= q;
        }
        if (!comp[c] || rest != 1) continue;
        for (uint32_t q : f) used[q] = 1;
        extra.push_back(c);
    }
    // A needs log2 c + 2 more bits than B: it gets the first `lead` primes
    RnsModuli best;
    for (uint32_t lead = 0; lead < 24; lead++) {
        RnsModuli m;
        size_t top = primes.size();
        while (top > 0 && (m.a.size() + 1 < k || m.b.size() + extra.size() < k)) {
            const uint32_t q = primes[--top];
            if (used[q]) continue;
            const bool b_full = m.b.size() + extra.size() >= k;
            (m.a.size() + 1 < k && (b_full || m.a.size() < m.b.size() + lead) ? m.a : m.b).push_back(q);
        }
        m.b_primes = (uint32_t)m.b.size();
        m.b.insert(m.b.end(), extra.begin(), extra.end());
        const double c = coefficient(m.a.size());
        m.bits = std::fmin(a_capacity(log2_product(m.a), m.a.size()), log2_product(m.b) - 2 - std::log2(c));
        if (!sums_exact(m.a) || !sums_exact(m.b)) m.bits = 0;
        m.b.resize(k, 1);  // slots left over: modulus 1, all zero
        if (m.bits > best.bits) best = m;
    }
    return best;
}

inline const RnsModuli &moduli_of(uint32_t n) {
    static const std::vector<RnsModuli> all = [] {
        std::vector<RnsModuli> v(kRnsMaxChunks + 1);
        for (uint32_t i = 1; i <= kRnsMaxChunks; i++) v[i] = make_moduli(i);
        return v;
    }();
    return all[n];
}

// How many of A's moduli numbers below 2^bits take: no more, so that A / N stays
// small (the start needs A mod N).
inline uint32_t a_count(uint32_t n, uint32_t bits) {
    const RnsModuli &mod = moduli_of(n);
    double la = 0;
    uint32_t k = 0;
    while (k < mod.a.size() && (k == 0 || a_capacity(la, k) - 1e-6 < (double)bits)) la += std::log2((double)mod.a[k++]);
    return k;
}

}  // namespace pg
