// Walks the ring kernel's step blocks on the CPU, thread by thread and row by
// row, and compares the result with the direct sum over terms.  Built and run
// by tests/test_ring_schedule_cpu.py; prints one line per operator and exits
// non-zero on the first mismatch or block that does not fit its size.
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "../tencirpauli_b200/csrc/tcp_internal.h"

using cplx = std::complex<double>;

static bool fail_line(const char *name, const char *what) {
    std::printf("%s: %s\n", name, what);
    return false;
}

template <typename W> static W read(const uint8_t *p) {
    W v;
    std::memcpy(&v, p, sizeof v);
    return v;
}
static int parity(uint32_t v) { return __builtin_popcount(v) & 1; }

// Signed weight of one record for the row word c; `p` moves past it.
template <typename W> static double record_value(const uint8_t *&p, uint32_t c) {
    const uint32_t kind = (read<uint32_t>(p + 4) & tcp::kRingKindMask) >> tcp::kRingKindShift;
    const double sign = parity(read<uint32_t>(p) & c) ? -1.0 : 1.0;
    double w;
    if (kind == 0) {
        w = read<W>(p + 8);
    } else {
        uint32_t at = 0;
        for (uint32_t b = 0; b < kind + 1; ++b) at |= parity(read<uint32_t>(p + 8 + 4 * b) & c) << b;
        w = read<W>(p + (kind == 1 ? 16 : 32) + at * sizeof(W));
    }
    p += tcp::ring_record_bytes(kind, sizeof(W));
    return sign * w;
}

template <typename W>
static bool check(const char *name, uint32_t n, const std::vector<tcp::MatrixTerm> &terms, tcp::RingShapeBits shape,
                  double tolerance) {
    const bool c64 = sizeof(W) == 4;
    const uint32_t S = shape.tile_bits, T = 1u << shape.log_threads, E = 1u << (S - shape.log_threads);
    // tile row of thread t's register row j
    auto row = [&](uint32_t t, uint32_t j) {
        const uint32_t low = (1u << shape.low) - 1u;
        return (j & low) | (t << shape.low) | ((j >> shape.low) << (shape.low + shape.log_threads));
    };
    const tcp::RingSchedule r = tcp::build_ring_schedule(terms, n, shape, shape.low == 0);
    if (r.tile_bits != S) return fail_line(name, "no ring schedule");
    const std::vector<uint8_t> &blocks = c64 ? r.blocks_c64 : r.blocks_c128;
    std::mt19937_64 rng(5);
    std::normal_distribution<double> normal;
    std::vector<cplx> x(1ull << n), y(1ull << n, 0.0);
    for (auto &v : x) v = cplx(normal(rng), normal(rng));
    uint32_t last_d = 0;
    uint64_t cosets = 0;
    for (size_t st = 0; st < r.step_info.size(); st += 4) {
        const uint32_t d = r.step_info[st], info = r.step_info[st + 3];
        const size_t off = static_cast<size_t>(r.step_info[st + (c64 ? 2 : 1)]) * 16;
        const size_t bytes = (c64 ? info >> 16 : info & 0xffffu) * size_t(16);
        if (st && d < last_d) return fail_line(name, "steps are not sorted by d");
        last_d = d;
        // the kernel reads 16 bytes past the last record
        if (bytes + 16 > tcp::kRingBlockBytes || off + bytes > blocks.size()) return fail_line(name, "block size");
        const uint8_t *blk = blocks.data() + off;
        for (uint64_t tile = 0; tile < (1ull << (n - S)); ++tile) {
            for (uint32_t t = 0; t < T; ++t) {
                const uint32_t c = t | static_cast<uint32_t>(tile << shape.log_threads);
                const uint8_t *p = blk + 16;
                const cplx *src = nullptr;
                uint32_t from_t = 0;
                double sum = 0.0;
                uint32_t unfolded = 0, flips = 0;
                for (uint32_t left = read<uint32_t>(blk); left; --left) {
                    if (p + 16 > blk + bytes) return fail_line(name, "record past the block");
                    const uint32_t word = read<uint32_t>(p + 4);
                    if (word & tcp::kRingNew) {
                        src = x.data() + ((tile ^ d) << S);
                        from_t = t ^ (word >> tcp::kRingMaskShift);
                        if (from_t >= T) return fail_line(name, "thread mask");
                        cosets += tile == 0 && t == 0;
                        flips = 0;
                    }
                    flips ^= (word & tcp::kRingFlipMask) >> tcp::kRingFlipShift;
                    if (src == nullptr) return fail_line(name, "a block does not begin with a coset");
                    sum += record_value<W>(p, c);
                    if (!(word & tcp::kRingLast)) continue;
                    for (uint32_t j = 0; j < E; ++j) {
                        const uint32_t from = j ^ (word & 15u);
                        if (from >= E) return fail_line(name, "row permutation");
                        const double w = parity(flips & from) ? -sum : sum;
                        const cplx v = src[row(from_t, from)];
                        y[(tile << S) + row(t, j)] += word & tcp::kRingImag ? cplx(0.0, w) * v : w * v;
                    }
                    sum = 0.0;
                    if (++unfolded > tcp::kRingFoldRuns) return fail_line(name, "too many runs without a fold");
                    if (word & tcp::kRingFold) {
                        unfolded = 0;
                        if (shape.low) src = nullptr;  // a new coset follows
                    }
                }
                if (sum != 0.0) return fail_line(name, "a block ends inside a run");
                if (p != blk + bytes) return fail_line(name, "block not consumed exactly");
            }
        }
    }
    if (cosets != r.cosets) return fail_line(name, "coset count");
    double diff = 0.0, norm = 0.0;
    for (uint64_t i = 0; i < (1ull << n); ++i) {
        cplx ref = 0.0;
        for (const tcp::MatrixTerm &t : terms) {
            const uint64_t col = i ^ t.x_mask;
            const double s = __builtin_popcountll(t.z_mask & col) & 1 ? -1.0 : 1.0;
            ref += s * cplx(t.w_re, t.w_im) * x[col];
        }
        diff += std::norm(ref - y[i]);
        norm += std::norm(ref);
    }
    const double err = norm > 0.0 ? std::sqrt(diff / norm) : std::sqrt(diff);
    std::printf("%s n=%u terms=%zu %s: runs %llu, relative error %.2e\n", name, n, terms.size(), c64 ? "c64" : "c128",
                static_cast<unsigned long long>(r.runs), err);
    return err <= tolerance || fail_line(name, "mismatch");
}

int main() {
    std::mt19937_64 rng(7);
    std::normal_distribution<double> normal;
    auto both = [](const char *name, uint32_t n, const std::vector<tcp::MatrixTerm> &t) {
        // complex128: T products of FP64 weights; complex64: weights rounded to FP32
        for (const tcp::RingShapeBits shape : tcp::kRingShapes) {
            if (n < shape.tile_bits) continue;
            // the 8192-row schedule has complex64 blocks only
            if (shape.low == 0 && !check<double>(name, n, t, shape, 1e-13)) return false;
            if (!check<float>(name, n, t, shape, 1e-6)) return false;
        }
        return true;
    };
    for (uint32_t n : {12u, 13u, 15u}) {
        const uint64_t mask = (1ull << n) - 1;
        std::vector<tcp::MatrixTerm> t;
        if (!both("empty", n, t)) return 1;
        t.push_back({0, 0, 0.0, 0.0});
        if (!both("zero weight", n, t)) return 1;
        t.assign(5, {5, 9, 0.3, 0.0});
        if (!both("one word five times", n, t)) return 1;
        t.clear();
        for (int k = 0; k < 40; ++k) t.push_back({rng() & mask, rng() & mask, normal(rng), k % 3 ? 0.0 : normal(rng)});
        if (!both("random, complex weights", n, t)) return 1;
        t.clear();
        for (uint64_t z = 0; z < 1100; ++z) t.push_back({1ull << (n - 1), (z * 2654435761u) & mask, normal(rng), 0.0});
        if (!both("one group of 1100 terms", n, t)) return 1;
        t.clear();  // every pair of Z, and single Z: the diagonal of a lattice
        for (uint32_t a = 0; a < n; ++a)
            for (uint32_t b = a; b < n; ++b) t.push_back({0, (1ull << a) | (1ull << b), normal(rng), 0.0});
        if (!both("diagonal pairs", n, t)) return 1;
        t.clear();  // four flips, all sixteen letter choices, a Z string between
        for (int k = 0; k < 24; ++k) {
            uint64_t m = 0;
            while (__builtin_popcountll(m) < 4) m |= 1ull << (rng() % n);
            const uint64_t string = rng() & mask & ~m;
            for (uint64_t u = m;; u = (u - 1) & m) {
                t.push_back({m, string ^ u, normal(rng), k & 1 ? normal(rng) : 0.0});
                if (u == 0) break;
            }
        }
        if (!both("two-body groups", n, t)) return 1;
        t.clear();  // more words of the same x mask and z row part than one run holds, repeated words
        for (int k = 0; k < 3000; ++k) t.push_back({3, (rng() & mask & 0x1ffull) | (uint64_t(k & 1) << 9), normal(rng), 0.0});
        if (!both("repeated words", n, t)) return 1;
    }
    // z bits at the top of the row word
    {
        std::vector<tcp::MatrixTerm> t;
        for (int k = 0; k < 60; ++k) t.push_back({rng() & 0xffffull, rng() & 0xffffull, normal(rng), 0.0});
        if (!both("16 qubits", 16, t)) return 1;
    }
    for (const tcp::RingShapeBits shape : tcp::kRingShapes) {
        const uint32_t most = tcp::kRingMaxZBits + shape.tile_bits - shape.log_threads;
        if (tcp::build_ring_schedule({}, most + 1, shape).tile_bits != 0 ||
            tcp::build_ring_schedule({}, most, shape).tile_bits != shape.tile_bits)
            return fail_line("qubit limit", "wrong"), 1;
    }
    std::printf("ok\n");
    return 0;
}
