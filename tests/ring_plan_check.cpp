// Properties of the ring schedules beyond the sums they give: the work of
// building them and the folds of the complex64 sums.  Built and run by tests/test_ring_plan_cpu.py with the name of
// the check; exits non-zero on the first failure.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <utility>
#include <vector>

#include "../tencirpauli_b200/csrc/tcp_internal.h"

using tcp::MatrixTerm;

static std::mt19937_64 rng(20);
static std::normal_distribution<double> normal;

static uint32_t word32(const uint8_t *p) {
    uint32_t v;
    std::memcpy(&v, p, 4);
    return v;
}
static bool odd(uint64_t v) { return (__builtin_popcountll(v) & 1) != 0; }

// The signed weight of a complex128 record for the row word c; p moves past it.
static double take_record(const uint8_t *&p, uint32_t c) {
    const uint32_t kind = (word32(p + 4) & tcp::kRingKindMask) >> tcp::kRingKindShift;
    uint32_t at = 8;
    if (kind) {
        at = kind == 1 ? 16 : 32;
        for (uint32_t b = 0; b <= kind; ++b) at += odd(word32(p + 8 + 4 * b) & c) ? 8u << b : 0u;
    }
    double w;
    std::memcpy(&w, p + at, 8);
    if (odd(word32(p) & c)) w = -w;
    p += tcp::ring_record_bytes(kind, 8);
    return w;
}

// H_ii of a diagonal operator from its complex128 blocks.
static double diagonal(const tcp::RingSchedule &r, uint64_t row) {
    const uint32_t c = (row & 511u) | static_cast<uint32_t>(row >> 12) << 9, j = (row >> 9) & 7u;
    double sum = 0.0, run = 0.0;
    for (size_t st = 0; st < r.step_info.size(); st += 4) {
        const uint8_t *p = r.blocks_c128.data() + size_t(r.step_info[st + 1]) * 16;
        uint32_t left = word32(p), zj = 0;
        for (p += 16; left; --left) {
            const uint32_t word = word32(p + 4);
            zj = (word & tcp::kRingNew ? 0u : zj) ^ (word & tcp::kRingFlipMask) >> tcp::kRingFlipShift;
            run += take_record(p, c);
            if (!(word & tcp::kRingLast)) continue;
            sum += odd(zj & j) ? -run : run;
            run = 0.0;
        }
    }
    return sum;
}

// One search looks at 31 places in four directions of 1, 2, 4 and 8 points from
// two starts, below 1000 steps with its sample and the 16 look-ups of the table
// it finds; a run's searches end after 64 tables of fewer than 8 terms, each of
// at least 3.  Lists of up to 512 terms are rewritten after every table, longer
// ones at 16 moves a term.  So a run takes below 64 (1000 + 512) steps and
// (1000 + 512) / 8 more a term.
static int work(uint32_t n) {
    const uint64_t mask = (1ull << n) - 1;
    auto bounded = [&](const char *name, const std::vector<MatrixTerm> &terms) {
        for (const tcp::RingShapeBits shape : tcp::kRingShapes) {
            const tcp::RingSchedule r = tcp::build_ring_schedule(terms, n, shape, shape.low == 0);
            const double limit = 1512.0 / 8 * static_cast<double>(terms.size()) + 64 * 1512.0 * 16;  // 16 row parts
            if (r.tile_bits != shape.tile_bits || static_cast<double>(r.work) > limit) {
                std::printf("%s: %.0f steps for %zu terms\n", name, static_cast<double>(r.work), terms.size());
                return false;
            }
            // and the sum is the operator's: at most 2^18 weights of size ~1,
            // so a wrong or missing one shows; rounding alone stays below 1e-8
            for (int k = 0; k < 4 && shape.low == 0; ++k) {
                const uint64_t row = rng() & mask;
                long double sum = 0.0L;
                for (const MatrixTerm &t : terms) sum += odd(t.z_mask & row) ? -t.w_re : t.w_re;
                if (std::abs(static_cast<double>(diagonal(r, row) - sum)) > 1e-8) {
                    std::printf("%s: H_ii differs in row %llu\n", name, static_cast<unsigned long long>(row));
                    return false;
                }
            }
        }
        return true;
    };
    std::vector<MatrixTerm> t;
    for (int k = 0; k < 1 << 18; ++k) t.push_back({0, rng() & mask, normal(rng), 0.0});
    if (!bounded("random diagonal", t)) return 1;
    t.clear();
    for (uint64_t z = 0; z < 1ull << 18; ++z) t.push_back({0, z, normal(rng), 0.0});
    if (!bounded("dense diagonal", t)) return 1;
    std::shuffle(t.begin(), t.end(), rng);
    if (!bounded("shuffled dense diagonal", t)) return 1;
    t.resize(t.size() / 4);
    if (!bounded("a quarter of it", t)) return 1;
    t.clear();
    for (uint64_t k = 0; k < 1ull << 18; ++k) t.push_back({0, (k % 100) * 0x9e377ull & mask, normal(rng), 0.0});
    if (!bounded("repeated words", t)) return 1;
    t.clear();
    for (uint32_t a = 0; a < n; ++a)
        for (uint32_t b = 0; b < a; ++b)
            for (uint32_t c = 0; c < b; ++c)
                for (uint32_t d = 0; d < c; ++d) t.push_back({0, 1ull << a | 1ull << b | 1ull << c | 1ull << d, normal(rng), 0.0});
    if (!bounded("quartic diagonal", t)) return 1;
    return 0;
}

// Jordan-Wigner-like, lattice and random operators on n qubits.
static std::vector<std::pair<const char *, std::vector<MatrixTerm>>> operators(uint32_t n) {
    std::vector<std::pair<const char *, std::vector<MatrixTerm>>> out;
    std::vector<MatrixTerm> t;
    for (uint32_t q = 0; q < n; ++q) {
        const uint64_t m = 1ull << q | 1ull << (q + 1) % n;
        t.push_back({m, 0, 0.25, 0.0});
        t.push_back({m, m, -0.25, 0.0});
        t.push_back({0, m, 0.25, 0.0});
        t.push_back({0, 1ull << q, 0.5 * normal(rng), 0.0});
    }
    out.emplace_back("lattice", t);
    t.clear();
    for (int k = 0; k < 600; ++k) {
        uint64_t x = 0, z = 0;
        for (int j = 0; j < 2 + k % 3; ++j) {
            const uint64_t q = 1ull << rng() % n, letter = rng() % 3;
            if (letter < 2) x |= q;
            if (letter > 0) z |= q;
        }
        t.push_back({x, z, normal(rng), k % 7 ? 0.0 : normal(rng)});
    }
    out.emplace_back("random", t);
    t.clear();
    for (int k = 0; k < 150; ++k) {
        uint64_t m = 0;
        while (__builtin_popcountll(m) < 4) m |= 1ull << rng() % n;
        const uint64_t string = rng() & ((1ull << n) - 1) & ~m;
        for (uint64_t u = m;; u = (u - 1) & m) {
            if (__builtin_popcountll(u) % 2 == 0) t.push_back({m, string ^ u, normal(rng), 0.0});
            if (u == 0) break;
        }
    }
    for (uint32_t a = 0; a < n; ++a)
        for (uint32_t b = 0; b <= a; ++b) t.push_back({0, 1ull << a | 1ull << b, normal(rng), 0.0});
    out.emplace_back("two-body", t);
    return out;
}

// complex64: the kernel carries its partial sums from step to step, so a fold is
// due every kRingFoldRuns runs of the whole schedule, not of a step.  (The last
// fold, after the last step, is the kernel's own.)
static int folds() {
    for (uint32_t n : {14u, 22u}) {
        for (const auto &op : operators(n)) {
            for (const tcp::RingShapeBits shape : tcp::kRingShapes) {
                const tcp::RingSchedule r = tcp::build_ring_schedule(op.second, n, shape, shape.low == 0);
                uint32_t unfolded = 0, most = 0;
                uint64_t runs = 0;
                for (size_t st = 0; st < r.step_info.size(); st += 4) {
                    const uint8_t *p = r.blocks_c64.data() + size_t(r.step_info[st + 2]) * 16;
                    uint32_t left = word32(p);
                    for (p += 16; left; --left) {
                        const uint32_t word = word32(p + 4);
                        p += tcp::ring_record_bytes((word & tcp::kRingKindMask) >> tcp::kRingKindShift, 4);
                        if (!(word & tcp::kRingLast)) continue;
                        ++runs;
                        most = std::max(most, ++unfolded);
                        if (word & tcp::kRingFold) unfolded = 0;
                    }
                }
                if (most > tcp::kRingFoldRuns || runs != r.runs || runs <= tcp::kRingFoldRuns) {
                    std::printf("%s, %u qubits: %u of %llu runs without a fold\n", op.first, n, most,
                                static_cast<unsigned long long>(runs));
                    return 1;
                }
            }
        }
    }
    return 0;
}

int main(int argc, char **argv) {
    const char *check = argc > 1 ? argv[1] : "";
    if (!std::strcmp(check, "work")) return work(20) || work(28);  // terms left in a bitmap, in a hash table
    if (!std::strcmp(check, "folds")) return folds();
    std::printf("unknown check\n");
    return 2;
}
