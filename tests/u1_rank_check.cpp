// The rank tables of the sectors of up to 32 qubits: every entry that the pair
// kernel looks up, for live and dead pairs of every row, lies inside them.  Built
// and run by tests/test_u1_rank_cpu.py; exits non-zero on the first failure.
#include <algorithm>
#include <cstdio>
#include <vector>

#include "../tencirpauli_b200/csrc/tcp_u1_rank.h"

int main() {
    for (uint32_t n = 1; n <= 32; ++n) {
        for (uint32_t k = 0; k <= n; ++k) {
            const tcp::U1Split s = tcp::u1_split(n, k);
            if (s.top + s.mid + s.low != n || (s.mid == 0) != (n <= 24)) return std::printf("%u qubits: split\n", n), 1;
            const uint64_t entries = tcp::u1_table_entries(s, k);
            const uint64_t m_off = 1ull << s.top;
            const uint64_t l_off = m_off + (s.mid ? uint64_t(tcp::u1_mid_rows(k, s.top)) << s.mid : 0);
            // states with a, c and k - a - c ones in the three parts, lowest and
            // highest in each
            std::vector<uint32_t> states;
            for (uint32_t a = 0; a <= s.top && a <= k; ++a)
                for (uint32_t c = 0; c <= s.mid && a + c <= k; ++c) {
                    const uint32_t e = k - a - c;
                    if (e > s.low) continue;
                    auto part = [](uint32_t ones, uint32_t bits, bool high) {
                        return ((1ull << ones) - 1) << (high ? bits - ones : 0);
                    };
                    for (int h = 0; h < 8; ++h)
                        states.push_back(static_cast<uint32_t>(part(a, s.top, h & 1) << (s.mid + s.low) |
                                                               part(c, s.mid, h & 2) << s.low | part(e, s.low, h & 4)));
                }
            for (const uint32_t b : states)
                for (uint32_t p = 0; p < n; ++p)
                    for (uint32_t q = 0; q <= p; ++q) {  // p == q: the padding's empty pair
                        const uint32_t x = p == q ? 0u : 1u << p | 1u << q;
                        const uint64_t v = b ^ x, top = v >> (s.mid + s.low);
                        const uint64_t mid = (v >> s.low) & ((1ull << s.mid) - 1), low = v & ((1ull << s.low) - 1);
                        uint64_t at = std::max(top, l_off + low);
                        if (s.mid) at = std::max(at, m_off + (uint64_t(__builtin_popcountll(top)) << s.mid) + mid);
                        if (top >= m_off || at >= entries)
                            return std::printf("%u qubits, %u particles, row %x, pair %x: entry %llu of %llu\n", n, k, b, x,
                                               static_cast<unsigned long long>(at), static_cast<unsigned long long>(entries)), 1;
                    }
        }
    }
    return 0;
}
