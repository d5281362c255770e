// How the rank tables of a fixed-particle-number sector of up to 32 qubits cut a
// state, and how many entries they need.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace tcp {

// Bits of the top, middle and low part of a state; mid = 0: two levels.  The top
// table has 2^top entries, the low one 2^low, the middle one u1_mid_rows rows of
// 2^mid: one row per number of ones in the top part of a state of the sector.
struct U1Split {
    uint32_t top, mid, low;
};

inline uint32_t u1_mid_rows(uint32_t k, uint32_t top) { return std::min(k, top) + 1u; }

// Two levels up to 24 qubits, else the three with the fewest entries.
inline U1Split u1_split(uint32_t n, uint32_t k) {
    if (n <= 24) return {n - n / 2, 0, n / 2};
    U1Split best{0, 0, 0};
    size_t least = ~size_t(0);
    for (uint32_t a = 1; a + 2 <= n; ++a)
        for (uint32_t b = 1; a + b + 1 <= n; ++b) {
            const uint32_t c = n - a - b;
            const size_t entries = (size_t(1) << a) + u1_mid_rows(k, a) * (size_t(1) << b) + (size_t(1) << c);
            if (entries < least) {
                least = entries;
                best = {a, b, c};
            }
        }
    return best;
}

// Entries of the tables laid out as top, middle, low.  The pair kernel looks up
// the source of every pair of bits, also of dead ones (both bits set or both
// clear), whose value it does not use: such a source has up to two ones more than
// the sector's states, and its entry lies up to two rows behind the middle table,
// in the low one or, for sectors without particles, behind it.  (Looking up the
// row itself instead would cost 2 to 5 % on 28 to 32 qubits.)
inline size_t u1_table_entries(U1Split s, uint32_t k) {
    const size_t top = size_t(1) << s.top, low = size_t(1) << s.low;
    if (s.mid == 0) return top + low;
    const size_t mid = size_t(u1_mid_rows(k, s.top)) << s.mid, reached = size_t(u1_mid_rows(k + 2, s.top)) << s.mid;
    return top + std::max(mid + low, reached);
}

}  // namespace tcp
