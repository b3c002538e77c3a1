// Host build of the residue number system's moduli (prime-gap_gb300/csrc/pg_rns_moduli.h)
// for CPU tests.
#include <algorithm>

#include "pg_rns_moduli.h"

extern "C" {

uint32_t rh_chunks() { return pg::kRnsMaxChunks; }

// The moduli of n chunks (room for 32 n each); returns how many A has.
uint32_t rh_moduli(uint32_t n, uint32_t *a, uint32_t *b, uint32_t *b_primes, double *bits) {
    const pg::RnsModuli &m = pg::moduli_of(n);
    std::copy(m.a.begin(), m.a.end(), a);
    std::copy(m.b.begin(), m.b.end(), b);
    *b_primes = m.b_primes;
    *bits = m.bits;
    return (uint32_t)m.a.size();
}

uint32_t rh_a_count(uint32_t n, uint32_t bits) { return pg::a_count(n, bits); }

int rh_sums_exact(const uint32_t *m, uint32_t n) { return pg::sums_exact(std::vector<uint32_t>(m, m + n)); }

}  // extern "C"
