// Host side of libtcpmvp.so: error slot, canonicalization, term compilation and
// the tile schedule.  Pure C++ (no CUDA); compiled by nvcc with the kernels.
#include <algorithm>
#include <array>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <utility>

#include "tcp_internal.h"

namespace tcp {

namespace {
thread_local std::string g_last_error;
thread_local int g_last_status = 0;
thread_local uint64_t g_last_fields[2] = {0, 0};
std::atomic<long long> g_alloc_count{0};
}  // namespace

void set_error(const std::string &message) { g_last_error = message; }

int fail(int status, const std::string &message) { return fail_fields(status, message, 0, 0); }

int fail_fields(int status, const std::string &message, uint64_t a, uint64_t b) {
    g_last_error = message;
    g_last_status = status;
    g_last_fields[0] = a;
    g_last_fields[1] = b;
    return status;
}

uint64_t clamp_u64(unsigned __int128 v) { return (v >> 64) ? ~0ull : static_cast<uint64_t>(v); }

bool injected_alloc_failure() {
    const char *env = std::getenv("TCP_FAIL_ALLOC_AFTER");
    if (env == nullptr || *env == '\0') return false;
    long long limit = std::atoll(env);
    long long index = g_alloc_count.fetch_add(1);
    return index >= limit;
}

static inline uint32_t packed_word_count(uint32_t nqubits) { return nqubits / 64 + (nqubits % 64 != 0); }

int compile_terms(uint32_t nqubits, uint64_t count, uint32_t word_count, const uint64_t *x_words,
                  const uint64_t *z_words, const double *coefficients, std::vector<MatrixTerm> &out) {
    // pauli_action.rs:38-55 -- word-length and dimension checks
    uint32_t expected = packed_word_count(nqubits);
    if (word_count != expected) {
        return fail_fields(TCP_ERR_INVALID_WORD_LENGTH,
                           "expected " + std::to_string(expected) + " packed words, got " + std::to_string(word_count),
                           expected, word_count);
    }
    if (nqubits >= 64) return fail(TCP_ERR_OVERFLOW, "integer overflow while computing dense statevector dimension");
    out.clear();
    out.reserve(count);
    // word.rs:81-85: bits above nqubits in the final word are masked off
    uint64_t tail = (nqubits % 64) ? ((1ull << (nqubits % 64)) - 1) : ~0ull;
    for (uint64_t t = 0; t < count; ++t) {
        double re = coefficients[2 * t], im = coefficients[2 * t + 1];
        if (!std::isfinite(re) || !std::isfinite(im)) {
            return fail_fields(TCP_ERR_NON_FINITE_COEFFICIENT, "coefficient at index " + std::to_string(t) + " is not finite",
                               t, 0);
        }
        uint64_t xm = 0, zm = 0;
        uint32_t ny = 0;
        for (uint32_t q = 0; q < nqubits; ++q) {
            uint64_t packed = 1ull << (q % 64);
            uint64_t xw = x_words[t * word_count + q / 64];
            uint64_t zw = z_words[t * word_count + q / 64];
            if (q / 64 == word_count - 1) {
                xw &= tail;
                zw &= tail;
            }
            bool x = (xw & packed) != 0, z = (zw & packed) != 0;
            uint64_t bit = 1ull << (nqubits - 1 - q);
            if (x) xm |= bit;
            if (z) zm |= bit;
            if (x && z) ++ny;
        }
        // y_phase = i^{#Y mod 4}; weighted = coefficient * y_phase with the
        // textbook complex product (num-complex): (a c - b d, a d + b c).
        double pr = 0.0, pi = 0.0;
        switch (ny % 4) {
        case 0: pr = 1.0; break;
        case 1: pi = 1.0; break;
        case 2: pr = -1.0; break;
        default: pi = -1.0; break;
        }
        MatrixTerm mt;
        mt.x_mask = xm;
        mt.z_mask = zm;
        volatile double ac = re * pr, bd = im * pi, ad = re * pi, bc = im * pr;  // no contraction
        mt.w_re = ac - bd;
        mt.w_im = ad + bc;
        out.push_back(mt);
    }
    return TCP_OK;
}

uint64_t distinct_x_masks(const std::vector<MatrixTerm> &terms) {
    std::vector<uint64_t> m;
    m.reserve(terms.size());
    for (auto &t : terms) m.push_back(t.x_mask);
    std::sort(m.begin(), m.end());
    return static_cast<uint64_t>(std::unique(m.begin(), m.end()) - m.begin());
}

namespace {
template <typename T> void put(std::vector<uint8_t> &out, const T &v) {
    const uint8_t *p = reinterpret_cast<const uint8_t *>(&v);
    out.insert(out.end(), p, p + sizeof(T));
}
}  // namespace

Schedule build_schedule(const std::vector<MatrixTerm> &terms, uint32_t nqubits, uint32_t tile_bits,
                        uint32_t log_threads, bool blocks) {
    Schedule s;
    s.tile_bits = std::min(tile_bits, nqubits);
    s.log_threads = std::min(log_threads, s.tile_bits);
    const uint32_t S = s.tile_bits;
    const uint32_t L = s.log_threads;
    const uint64_t inner = (S >= 64) ? ~0ull : ((1ull << S) - 1);
    const uint32_t jcount = 1u << (S - L);
    // (outer, inner, canonical index): a stable order that keeps canonical
    // term order inside every x-mask group.
    std::vector<uint64_t> order(terms.size());
    std::iota(order.begin(), order.end(), 0);
    std::stable_sort(order.begin(), order.end(), [&](uint64_t a, uint64_t b) {
        uint64_t da = terms[a].x_mask >> S, db = terms[b].x_mask >> S;
        if (da != db) return da < db;
        return (terms[a].x_mask & inner) < (terms[b].x_mask & inner);
    });
    // group view
    s.g_tbeg.push_back(0);
    for (size_t i = 0; i < order.size(); ++i) {
        const MatrixTerm &t = terms[order[i]];
        if (s.g_mask.empty() || s.g_mask.back() != t.x_mask) {
            if (!s.g_mask.empty()) s.g_tbeg.push_back(static_cast<uint32_t>(i));
            s.g_mask.push_back(t.x_mask);
        }
        s.t_z.push_back(t.z_mask);
        s.t_w.push_back(t.w_re);
        s.t_w.push_back(t.w_im);
        s.t_wf.push_back(static_cast<float>(t.w_re));
        s.t_wf.push_back(static_cast<float>(t.w_im));
    }
    if (!s.g_mask.empty()) s.g_tbeg.push_back(static_cast<uint32_t>(order.size()));

    // step view: walk the groups, packing blocks of at most kBlockBytesMax
    struct Pending {
        uint32_t m_in;
        size_t gid;                   // group index in the group view
        std::vector<uint64_t> terms;  // indices into `terms`
    };
    uint64_t cur_d = 0;
    std::vector<Pending> pend;
    size_t pend_bytes = 0;
    auto flush = [&]() {
        if (pend.empty()) return;
        if (!blocks) {
            s.step_info.insert(s.step_info.end(), {static_cast<uint32_t>(cur_d), static_cast<uint32_t>(cur_d >> 32), 0u,
                                                   static_cast<uint32_t>(pend.size())});
            pend.clear();
            pend_bytes = 0;
            return;
        }
        const size_t off = s.blocks_c128.size();
        uint32_t nterms = 0;
        for (auto &g : pend) {
            put(s.blocks_c128, g.m_in);
            put(s.blocks_c128, nterms);
            nterms += static_cast<uint32_t>(g.terms.size());
            put(s.blocks_c128, nterms);
            put(s.blocks_c128, uint32_t(0));
        }
        for (auto &g : pend) {
            for (uint64_t ti : g.terms) {
                const MatrixTerm &t = terms[ti];
                const uint64_t zt = (S >= 64) ? 0 : (t.z_mask >> S);
                const uint32_t zlo = static_cast<uint32_t>(t.z_mask & ((1ull << L) - 1));
                const uint32_t zj = static_cast<uint32_t>((t.z_mask & inner) >> L);
                uint32_t pattern = 0;
                for (uint32_t jj = 0; jj < jcount; ++jj)
                    pattern |= (static_cast<uint32_t>(__builtin_popcount(zj & jj)) & 1u) << jj;
                const uint32_t kind = (t.w_im == 0.0) ? kKindReal : ((t.w_re == 0.0) ? kKindImag : kKindComplex);
                const uint64_t zrec = static_cast<uint64_t>(zlo) | (static_cast<uint64_t>(pattern) << 32) |
                                      (static_cast<uint64_t>(kind) << 56);
                // parity(zt & d), parity(zlo & m_lo) and parity(zj & jh) are
                // fixed for the term inside its step and group, so they are
                // folded into the weight.  (The kernel loads row j's source
                // j ^ jh into register j, so the remaining sign of row j is
                // bit j of the pattern, parity(zj & j), XOR the thread's base.)
                const uint32_t m_lo = g.m_in & ((1u << L) - 1u);
                const uint32_t jh = g.m_in >> L;
                const bool flip = ((__builtin_popcountll(zt & cur_d) + __builtin_popcount(zlo & m_lo) +
                                    __builtin_popcount(zj & jh)) & 1) != 0;
                const double wr = flip ? -t.w_re : t.w_re, wi = flip ? -t.w_im : t.w_im;
                put(s.blocks_c128, zrec);
                put(s.blocks_c128, zt);
                put(s.blocks_c128, wr);
                put(s.blocks_c128, wi);
            }
        }
        const size_t bytes = s.blocks_c128.size() - off;
        s.step_info.push_back(static_cast<uint32_t>(cur_d));
        s.step_info.push_back(static_cast<uint32_t>(cur_d >> 32));
        s.step_info.push_back(static_cast<uint32_t>(off / 16));
        s.step_info.push_back(static_cast<uint32_t>(pend.size()) | static_cast<uint32_t>((bytes / 16) << 16));
        pend.clear();
        pend_bytes = 0;
    };
    bool have_step = false;
    for (size_t g = 0; g < s.g_mask.size(); ++g) {
        const uint64_t d = s.g_mask[g] >> S;
        const uint32_t m_in = static_cast<uint32_t>(s.g_mask[g] & inner);
        if (!have_step || d != cur_d) {
            flush();
            cur_d = d;
            have_step = true;
            ++s.distinct_outer;
        }
        for (uint32_t t = s.g_tbeg[g]; t < s.g_tbeg[g + 1]; ++t) {
            bool opens = pend.empty() || pend.back().gid != g;
            if (pend_bytes + kTermRecBytes + (opens ? kGroupRecBytes : 0) > kBlockBytesMax) {
                flush();
                opens = true;
            }
            if (opens) {
                pend.push_back(Pending{m_in, g, {}});
                pend_bytes += kGroupRecBytes;
            }
            if (blocks) pend.back().terms.push_back(order[t]);
            pend_bytes += kTermRecBytes;
        }
    }
    flush();
    if (!blocks) return s;
    // complex64 blocks: same layout, weights as two floats + 8 pad bytes
    s.blocks_c64 = s.blocks_c128;
    for (size_t i = 0; i + 4 <= s.step_info.size(); i += 4) {
        const size_t off = static_cast<size_t>(s.step_info[i + 2]) * 16;
        const uint32_t ng = s.step_info[i + 3] & 0xffffu;
        const size_t bytes = static_cast<size_t>(s.step_info[i + 3] >> 16) * 16;
        for (size_t p = off + ng * kGroupRecBytes; p < off + bytes; p += kTermRecBytes) {
            double wr, wi;
            std::memcpy(&wr, &s.blocks_c128[p + 16], 8);
            std::memcpy(&wi, &s.blocks_c128[p + 24], 8);
            const float fr = static_cast<float>(wr), fi = static_cast<float>(wi);
            std::memcpy(&s.blocks_c64[p + 16], &fr, 4);
            std::memcpy(&s.blocks_c64[p + 20], &fi, 4);
            std::memset(&s.blocks_c64[p + 24], 0, 8);
        }
    }
    return s;
}

namespace {

struct SignedWeight {
    uint32_t zs;
    double w;
};

// Terms in one affine space z0 ^ span(v[0 .. rank)): the table of their signed
// sums over the rank index bits.
struct SignTable {
    uint32_t z0 = 0;
    uint32_t v[4] = {0, 0, 0, 0};
    uint32_t rank = 0;
    double t[16] = {};
};

// Coordinates of zs ^ z0 in a growing basis of at most 4 vectors; returns
// false when it lies outside and the basis is full.
struct AffineSpan {
    uint32_t z0 = 0;
    uint32_t v[4] = {0, 0, 0, 0};       // the basis as given
    uint32_t red[4] = {0, 0, 0, 0};     // reduced vectors
    uint32_t combo[4] = {0, 0, 0, 0};   // each as a combination of v
    uint32_t rank = 0;
    bool contains(uint32_t zs) const {
        uint32_t x = zs ^ z0;
        for (uint32_t k = 0; k < rank; ++k) x = std::min(x, x ^ red[k]);
        return x == 0;
    }
    bool coordinates(uint32_t zs, uint32_t max_rank, uint32_t &coord) {
        uint32_t x = zs ^ z0, c = 0;
        for (uint32_t k = 0; k < rank; ++k) {
            if ((x ^ red[k]) < x) {  // red[k]'s top bit is set in x
                x ^= red[k];
                c ^= combo[k];
            }
        }
        if (x != 0) {
            if (rank == max_rank) return false;
            v[rank] = zs ^ z0;
            // keep the reduced vectors in descending order of their top bit
            uint32_t r = x, rc = c ^ (1u << rank);
            uint32_t at = rank;
            while (at > 0 && red[at - 1] < r) {
                red[at] = red[at - 1];
                combo[at] = combo[at - 1];
                --at;
            }
            red[at] = r;
            combo[at] = rc;
            c = 1u << rank;
            ++rank;
        }
        coord = c;
        return true;
    }
};

// Fewest terms for which a table of rank r is taken instead of singles: per
// thread a single takes about 8 instructions, a table of rank 2, 3, 4 about
// 18, 24 and 28.
constexpr size_t kTableMinTerms[5] = {3, 3, 3, 4, 5};

void fill_table(const AffineSpan &span, const std::vector<SignedWeight> &terms, const std::vector<uint32_t> &coords,
                SignTable &out) {
    out.z0 = span.z0;
    out.rank = span.rank;
    for (uint32_t k = 0; k < 4; ++k) out.v[k] = k < span.rank ? span.v[k] : 0u;
    for (size_t k = 0; k < terms.size(); ++k) {
        for (uint32_t i = 0; i < 16u; ++i) out.t[i] += __builtin_parity(coords[k] & i) ? -terms[k].w : terms[k].w;
    }
}

// The terms of one run that are not in a table yet, looked up by zs.
class RunTerms {
  public:
    uint64_t work = 0;  // look-ups, list steps and moves so far
    // `zbits`: bits of the zs, `terms`: terms of the whole plan.  A bitmap of the
    // terms left answers has() where it is small (16 KiB, or 4 bytes a term: a large
    // one costs a small plan more to map than it saves); a bit test takes a quarter
    // of a hash look-up.
    RunTerms(uint32_t zbits, size_t terms) : bitmap_(((uint64_t(1) << zbits) >> 3) <= std::max<uint64_t>(16384, 4 * terms)) {
        if (bitmap_) bits_.assign((size_t(1) << zbits) / 64 + 1, 0);
    }
    // Terms of equal zs are chained behind one of them.
    void reset(const std::vector<SignedWeight> &terms) {
        forget();
        terms_ = &terms;
        const size_t n = terms.size();
        log_ = 2;
        while ((size_t(1) << log_) < 4 * n) ++log_;
        slots_.assign(size_t(1) << log_, Slot{0, kNone});
        next_.assign(n, kNone);
        live_.assign(n, 1);
        order_.resize(n);
        std::iota(order_.begin(), order_.end(), 0u);
        head_ = dead_ = shift_ = 0;
        for (uint32_t i = 0; i < n; ++i) {
            Slot &slot = slots_[find(terms[i].zs)];
            next_[i] = slot.at;
            slot = {terms[i].zs, i};
            if (bitmap_) bits_[terms[i].zs >> 6] |= 1ull << (terms[i].zs & 63u);
        }
    }
    // Clears the bitmap of the terms still left.
    void forget() {
        if (bitmap_ && terms_)
            for (uint32_t i : order_) bits_[(*terms_)[i].zs >> 6] = 0;
        terms_ = nullptr;
    }
    uint32_t has(uint32_t zs) {
        ++work;
        if (bitmap_) return static_cast<uint32_t>(bits_[zs >> 6] >> (zs & 63u)) & 1u;
        return slots_[find(zs)].at < kTaken;
    }
    size_t left() const { return order_.size() - dead_; }
    bool compact() const { return dead_ == 0; }
    void squeeze() {
        work += order_.size();
        order_.erase(std::remove_if(order_.begin(), order_.end(), [&](uint32_t i) { return !live_[i]; }), order_.end());
        head_ = dead_ = shift_ = 0;
    }
    // Lists of up to 512 terms are squeezed after every table, longer ones once a
    // sixteenth of them is gone (16 moves a term).
    void tidy() {
        if (dead_ != 0 && (order_.size() <= 512 || dead_ >= order_.size() / 16)) squeeze();
    }
    uint32_t first() {
        for (; !live_[order_[head_]]; ++head_) ++work;
        return (*terms_)[order_[head_]].zs;
    }
    // Calls f(zs) for the first term left and its successors until f returns false.
    template <typename F> void walk(const F &f) {
        first();
        for (size_t k = head_; k < order_.size(); ++k) {
            ++work;
            if (live_[order_[k]] && !f((*terms_)[order_[k]].zs)) return;
        }
    }
    // Up to 31 of the terms left, spread over the list; the places move on with
    // every table, away from those that the last ones took.
    void sample(std::vector<uint32_t> &out) {
        out.clear();
        const size_t stride = std::max<size_t>(1, order_.size() / 16);
        for (size_t k = shift_++ % stride; k < order_.size(); k += stride) {
            ++work;
            if (live_[order_[k]]) out.push_back((*terms_)[order_[k]].zs);
        }
    }
    // Take the terms in the span, in list order, with their coordinates.
    void take(const AffineSpan &span, std::vector<SignedWeight> &in, std::vector<uint32_t> &coords) {
        found_.clear();
        for (uint32_t c = 0; c < (1u << span.rank); ++c) {
            uint32_t zs = span.z0;
            for (uint32_t k = 0; k < span.rank; ++k) zs ^= (c >> k) & 1u ? span.v[k] : 0u;
            ++work;
            Slot &slot = slots_[find(zs)];
            if (slot.at >= kTaken) continue;
            for (uint32_t i = slot.at; i != kNone; i = next_[i]) {
                found_.push_back({i, c});
                live_[i] = 0;
            }
            slot.at = kTaken;
            if (bitmap_) bits_[zs >> 6] &= ~(1ull << (zs & 63u));
        }
        std::sort(found_.begin(), found_.end());
        dead_ += found_.size();
        in.clear();
        coords.clear();
        for (const auto &f : found_) {
            in.push_back((*terms_)[f.first]);
            coords.push_back(f.second);
        }
    }
    void rest(std::vector<SignedWeight> &out) const {
        for (uint32_t i : order_)
            if (live_[i]) out.push_back((*terms_)[i]);
    }

  private:
    struct Slot {
        uint32_t zs, at;  // last term with this zs
    };
    static constexpr uint32_t kNone = 0xffffffffu, kTaken = 0xfffffffeu;
    size_t find(uint32_t zs) const {
        const size_t mask = slots_.size() - 1;
        size_t i = static_cast<uint64_t>(zs * 0x9e3779b97f4a7c15ull) >> (64 - log_);
        while (slots_[i].at != kNone && slots_[i].zs != zs) i = (i + 1) & mask;
        return i;
    }
    const std::vector<SignedWeight> *terms_ = nullptr;
    const bool bitmap_;
    std::vector<uint64_t> bits_;
    uint32_t log_ = 2;
    std::vector<Slot> slots_;
    std::vector<uint32_t> next_, order_;
    std::vector<uint8_t> live_;
    std::vector<std::pair<uint32_t, uint32_t>> found_;
    size_t head_ = 0, dead_ = 0, shift_ = 0;
};

// Tables with fewer terms than half their points after which the search of a run
// takes one start instead of two: terms without structure give no better ones
// from either.  Runs of the Jordan-Wigner and lattice operators end before that.
// It also bounds how often a list is rewritten for want of places to look at, so
// the work per term does not grow with the length of the run: 100,000 random
// diagonal words take 0.065 s (two starts throughout: 0.079 s, for 0.2 % fewer
// records), all 131,072 diagonal words of 17 qubits 0.04 s.
constexpr uint32_t kSparseTables = 64;

// Cut the terms of one run into singles and tables.  Whole runs of affine
// rank <= 4 become one table; larger ones are covered greedily by tables of
// rank 4, each grown direction by direction to cover the most remaining terms.
struct Tabulator {
    Tabulator(uint32_t zbits, size_t terms) : left(zbits, terms) {}
    RunTerms left;
    std::vector<SignedWeight> in;
    std::vector<uint32_t> coords, picks, points;

    void run(const std::vector<SignedWeight> &terms, std::vector<SignedWeight> &singles,
             std::vector<SignTable> &tables) {
        singles.clear();
        tables.clear();
        if (terms.size() < kTableMinTerms[2]) {
            singles = terms;
            return;
        }
        AffineSpan span;
        if (spans_all(terms, span)) {
            if (terms.size() < kTableMinTerms[span.rank]) {
                singles = terms;
                return;
            }
            SignTable t;
            fill_table(span, terms, coords, t);
            tables.push_back(t);
            return;
        }
        left.reset(terms);
        uint32_t sparse = 0, misses = 0;
        while (left.left() >= kTableMinTerms[2]) {
            bool whole = false;
            if (left.left() <= 16) {
                span = AffineSpan();
                span.z0 = left.first();
                left.walk([&](uint32_t zs) {
                    uint32_t c;
                    return whole = span.coordinates(zs, 4, c);
                });
            }
            if (!whole && search(span, sparse < kSparseTables) < kTableMinTerms[span.rank]) {
                if (left.compact() || ++misses > kSparseTables) break;
                left.squeeze();  // the places looked at may have missed the terms left
                continue;
            }
            left.take(span, in, coords);
            if (in.size() < kTableMinTerms[span.rank]) {
                singles.insert(singles.end(), in.begin(), in.end());
            } else {
                SignTable t;
                fill_table(span, in, coords, t);
                tables.push_back(t);
            }
            sparse += 2 * in.size() < (size_t(1) << span.rank);
            left.tidy();
        }
        left.rest(singles);
        left.forget();
    }

  private:
    bool spans_all(const std::vector<SignedWeight> &terms, AffineSpan &span) {
        span.z0 = terms[0].zs;
        coords.clear();
        for (const SignedWeight &s : terms) {
            uint32_t c;
            if (!span.coordinates(s.zs, 4, c)) return false;
            coords.push_back(c);
        }
        return true;
    }
    // Best table through the first term left or (`both`) through zero; its terms.
    size_t search(AffineSpan &best, bool both) {
        left.sample(picks);
        const uint32_t first = left.first();
        size_t best_count = 0;
        for (const uint32_t z0 : {first, 0u}) {
            AffineSpan cur;
            cur.z0 = z0;
            points.assign(1, z0);
            size_t covered = left.has(z0);
            for (uint32_t dim = 0; dim < 4; ++dim) {
                uint32_t best_v = 0;
                size_t best_new = 0;
                for (const uint32_t zs : picks) {
                    const uint32_t v = zs ^ z0;
                    if (cur.contains(zs)) continue;
                    size_t fresh = 0;
                    for (uint32_t p : points) fresh += left.has(p ^ v);
                    if (fresh > best_new) {
                        best_new = fresh;
                        best_v = v;
                    }
                    if (best_new == points.size()) break;  // no direction gives more
                }
                if (best_new == 0) break;
                uint32_t c;
                cur.coordinates(z0 ^ best_v, 4, c);
                const size_t n = points.size();
                for (size_t i = 0; i < n; ++i) points.push_back(points[i] ^ best_v);
                covered += best_new;
            }
            if (covered > best_count) {
                best_count = covered;
                best = cur;
            }
            if (!both || best_count == 16 || first == 0u) break;  // the second start gives no more
        }
        return best_count;
    }
};

}  // namespace

RingSchedule build_ring_schedule(const std::vector<MatrixTerm> &terms, uint32_t nqubits, RingShapeBits shape, bool c128) {
    RingSchedule r;
    const uint32_t S = shape.tile_bits, L = shape.log_threads;
    if (nqubits < S || nqubits - (S - L) > kRingMaxZBits) return r;
    const uint64_t inner = (1ull << S) - 1;
    const uint32_t tmask = (1u << L) - 1u, lowmask = (1u << shape.low) - 1u;
    auto thread_part = [&](uint64_t m) { return static_cast<uint32_t>(m >> shape.low) & tmask; };
    auto row_part = [&](uint64_t m) {
        const uint32_t high = static_cast<uint32_t>((m & inner) >> (shape.low + L));
        return (static_cast<uint32_t>(m) & lowmask) | (high << shape.low);
    };
    r.tile_bits = S;
    r.log_threads = L;

    // One item per real or imaginary weight part, in the order of d, m_lo, zj,
    // jh, kind of weight and canonical index.  Inside a coset the row parts zj
    // come in Gray-code order, so that most changes flip the rows of one bit.
    struct Item {
        uint64_t key;  // d << 18 | m_lo << 9 | Gray rank of zj << 5 | jh << 1 | imag
        uint32_t canon, zs;
        double w;  // folded
        uint32_t d() const { return static_cast<uint32_t>(key >> 18); }
        uint32_t m_lo() const { return static_cast<uint32_t>(key >> 9) & 0x1ffu; }
        uint32_t zj() const {
            const uint32_t g = static_cast<uint32_t>(key >> 5) & 15u;
            return g ^ (g >> 1);
        }
        uint32_t jh() const { return static_cast<uint32_t>(key >> 1) & 15u; }
        uint32_t imag() const { return static_cast<uint32_t>(key) & 1u; }
    };
    static_assert(kRingMaxZBits <= 32, "d and the key's 18 bits fit 64 bits");
    auto gray_rank = [](uint32_t zj) { return zj ^ (zj >> 1) ^ (zj >> 2) ^ (zj >> 3); };
    std::vector<Item> items;
    items.reserve(terms.size() + 8);
    for (size_t i = 0; i < terms.size(); ++i) {
        const MatrixTerm &t = terms[i];
        const uint64_t d = t.x_mask >> S;
        const uint32_t m_lo = thread_part(t.x_mask);
        const uint32_t zlo = thread_part(t.z_mask), zt = static_cast<uint32_t>(t.z_mask >> S);
        const bool flip = (__builtin_parityll(zt & d) ^ __builtin_parity(zlo & m_lo)) != 0;
        const uint64_t key = d << 18 | uint64_t(m_lo) << 9 | gray_rank(row_part(t.z_mask)) << 5 | row_part(t.x_mask) << 1;
        for (uint32_t imag = 0; imag < 2; ++imag) {
            const double w = imag ? t.w_im : t.w_re;
            if (imag ? w == 0.0 : (w == 0.0 && t.w_im != 0.0)) continue;
            items.push_back({key | imag, static_cast<uint32_t>(i), zlo | (zt << L), flip ? -w : w});
        }
    }
    std::sort(items.begin(), items.end(),
              [](const Item &a, const Item &b) { return a.key != b.key ? a.key < b.key : a.canon < b.canon; });

    std::vector<uint8_t> out128, out64;  // records of the open step
    const uint32_t wb = c128 ? 8u : 4u;  // weight bytes of the larger blocks
    uint32_t count = 0, cur_d = 0, cur_zj = 0, run_index = 0;
    int64_t cur_coset = -1;              // m_lo of the open coset (-1: none)
    auto flush = [&]() {
        if (count == 0) return;
        const size_t off[2] = {r.blocks_c128.size(), r.blocks_c64.size()};
        size_t bytes[2] = {0, 0};
        for (int f = c128 ? 0 : 1; f < 2; ++f) {
            std::vector<uint8_t> &dst = f ? r.blocks_c64 : r.blocks_c128;
            put(dst, count);
            for (int k = 0; k < 3; ++k) put(dst, uint32_t(0));
            const std::vector<uint8_t> &src = f ? out64 : out128;
            dst.insert(dst.end(), src.begin(), src.end());
            bytes[f] = dst.size() - off[f];
        }
        r.step_info.push_back(cur_d);
        r.step_info.push_back(static_cast<uint32_t>(off[0] / 16));
        r.step_info.push_back(static_cast<uint32_t>(off[1] / 16));
        r.step_info.push_back(static_cast<uint32_t>(bytes[0] / 16) | static_cast<uint32_t>(bytes[1] / 16) << 16);
        out128.clear();
        out64.clear();
        count = 0;
        cur_coset = -1;
    };
    // A record in both precisions: zs or z0, word, then the kind's content.
    auto put_record = [&](uint32_t kind, uint32_t zs, uint32_t word, const SignTable *t, double w) {
        for (int f = c128 ? 0 : 1; f < 2; ++f) {
            uint8_t rec[ring_record_bytes(3, 8)] = {};
            const uint32_t head[2] = {zs, word | (kind << kRingKindShift)};
            std::memcpy(rec, head, 8);
            const uint32_t first = kind == 0 ? 8u : (kind == 1 ? 16u : 32u), weights = kind == 0 ? 1u : 2u << kind;
            if (kind > 0) std::memcpy(rec + 8, t->v, kind == 1 ? 8 : (kind == 2 ? 12 : 16));
            for (uint32_t k = 0; k < weights; ++k) {
                const double v = kind == 0 ? w : t->t[k];
                const float single = static_cast<float>(v);
                std::memcpy(rec + first + k * (f ? 4 : 8), f ? static_cast<const void *>(&single) : &v, f ? 4 : 8);
            }
            std::vector<uint8_t> &dst = f ? out64 : out128;
            dst.insert(dst.end(), rec, rec + ring_record_bytes(kind, f ? 4u : 8u));
        }
        ++count;
    };
    std::vector<SignedWeight> list, singles;
    std::vector<SignTable> tables;
    Tabulator tabulator(nqubits - (S - L), terms.size());
    for (size_t k = 0; k < items.size();) {
        const Item first = items[k];
        if (k == 0 || first.d() != cur_d) {
            flush();
            cur_d = first.d();
        }
        list.clear();
        size_t e = k;
        for (; e < items.size() && items[e].key == first.key; ++e) list.push_back({items[e].zs, items[e].w});
        tabulator.run(list, singles, tables);
        // The run's records in order, a run per stretch that fits the block.
        const uint32_t run_word = first.jh() | (first.imag() ? kRingImag : 0u) | (first.m_lo() << kRingMaskShift);
        const size_t total = singles.size() + tables.size();
        auto kind_of = [&](size_t i) {
            return i < singles.size() ? 0u : std::max<uint32_t>(2u, tables[i - singles.size()].rank) - 1u;
        };
        // header, the records so far, `bytes` more and the 16 unused bytes
        auto room = [&](uint32_t bytes) {
            return 16 + (c128 ? out128 : out64).size() + bytes + 16 <= kRingBlockBytes;
        };
        for (size_t i = 0; i < total; ++i) {
            const uint32_t kind = kind_of(i);
            if (!room(ring_record_bytes(kind, wb))) flush();
            uint32_t word = run_word;
            if (cur_coset != static_cast<int64_t>(first.m_lo())) {
                word |= kRingNew;
                cur_coset = first.m_lo();
                cur_zj = 0;
                ++r.cosets;
            }
            word |= (first.zj() ^ cur_zj) << kRingFlipShift;
            cur_zj = first.zj();
            const bool ends = i + 1 == total;
            // the run also ends where the next record would open another step
            const bool cut = !ends && !room(ring_record_bytes(kind, wb) + ring_record_bytes(kind_of(i + 1), wb));
            if (ends || cut) {
                word |= kRingLast;
                ++r.runs;
                if (++run_index % kRingFoldRuns == 0) {
                    word |= kRingFold;
                    if (!c128) cur_coset = -1;
                }
            }
            if (i < singles.size())
                put_record(kind, singles[i].zs, word, nullptr, singles[i].w);
            else
                put_record(kind, tables[i - singles.size()].z0, word, &tables[i - singles.size()], 0.0);
        }
        k = e;
    }
    flush();
    r.work = tabulator.left.work;
    return r;
}

}  // namespace tcp

// ---------------------------------------------------------------------------
// C ABI: canonicalization (operator.rs:117-155)
// ---------------------------------------------------------------------------
namespace {
inline uint8_t code_at(const uint64_t *xw, const uint64_t *zw, uint32_t q) {
    uint64_t x = (xw[q / 64] >> (q % 64)) & 1u, z = (zw[q / 64] >> (q % 64)) & 1u;
    return x ? (z ? 2 : 1) : (z ? 3 : 0);
}
inline uint64_t bits_of(double v) {
    uint64_t b;
    std::memcpy(&b, &v, sizeof b);
    return b;
}
}  // namespace

extern "C" int tcp_pauli_canonicalize(uint32_t nqubits, uint64_t count, const uint8_t *codes,
                                      const double *coefficients, uint64_t *out_x, uint64_t *out_z,
                                      double *out_coefficients, uint64_t *out_count, uint64_t *bad_index) {
    using namespace tcp;
    if (out_count == nullptr || (count > 0 && (coefficients == nullptr || out_coefficients == nullptr ||
                                               out_x == nullptr || out_z == nullptr ||
                                               (nqubits > 0 && codes == nullptr)))) {
        return fail(TCP_ERR_INVALID_ARGUMENT, "null pointer argument");
    }
    const uint32_t w = packed_word_count(nqubits);
    // Validation in input order, coefficient before codes (operator.rs:130-136).
    for (uint64_t t = 0; t < count; ++t) {
        if (!std::isfinite(coefficients[2 * t]) || !std::isfinite(coefficients[2 * t + 1])) {
            if (bad_index) *bad_index = t;
            return fail_fields(TCP_ERR_NON_FINITE_COEFFICIENT, "coefficient at index " + std::to_string(t) + " is not finite",
                               t, 0);
        }
        for (uint32_t q = 0; q < nqubits; ++q) {
            uint8_t c = codes[t * nqubits + q];
            if (c > 3) {
                if (bad_index) *bad_index = q;
                return fail_fields(TCP_ERR_INVALID_CODE,
                                   "invalid Pauli code " + std::to_string(c) + " at index " + std::to_string(q) +
                                       "; expected 0..=3",
                                   c, q);
            }
        }
    }
    std::vector<uint64_t> xw(count * w + 1, 0), zw(count * w + 1, 0);
    for (uint64_t t = 0; t < count; ++t) {
        for (uint32_t q = 0; q < nqubits; ++q) {
            uint8_t c = codes[t * nqubits + q];
            uint64_t x = (c == 1 || c == 2), z = (c == 2 || c == 3);
            xw[t * w + q / 64] |= x << (q % 64);
            zw[t * w + q / 64] |= z << (q % 64);
        }
    }
    auto word_less = [&](uint64_t a, uint64_t b) -> int {
        for (uint32_t q = 0; q < nqubits; ++q) {
            uint8_t ca = code_at(&xw[a * w], &zw[a * w], q), cb = code_at(&xw[b * w], &zw[b * w], q);
            if (ca != cb) return ca < cb ? -1 : 1;
        }
        return 0;
    };
    std::vector<uint64_t> idx(count);
    std::iota(idx.begin(), idx.end(), 0);
    auto tie_break = [&](uint64_t a, uint64_t b) {
        uint64_t ar = bits_of(coefficients[2 * a]), br = bits_of(coefficients[2 * b]);
        if (ar != br) return ar < br;
        uint64_t ai = bits_of(coefficients[2 * a + 1]), bi = bits_of(coefficients[2 * b + 1]);
        if (ai != bi) return ai < bi;
        return a < b;
    };
    if (nqubits <= 64) {
        // Word order (word.rs:240-254) as a 128-bit integer key: the 2-bit code
        // of qubit 0 is the most significant digit.
        std::vector<std::pair<uint64_t, uint64_t>> key(count);
        for (uint64_t t = 0; t < count; ++t) {
            uint64_t hi = 0, lo = 0;
            for (uint32_t q = 0; q < nqubits; ++q) {
                const uint64_t c = codes[t * nqubits + q];
                const uint32_t pos = 2 * (63 - q);  // digit position inside 128 bits
                if (pos >= 64) hi |= c << (pos - 64); else lo |= c << pos;
            }
            key[t] = {hi, lo};
        }
        std::sort(idx.begin(), idx.end(), [&](uint64_t a, uint64_t b) {
            if (key[a] != key[b]) return key[a] < key[b];
            return tie_break(a, b);
        });
    } else {
        std::sort(idx.begin(), idx.end(), [&](uint64_t a, uint64_t b) {
            int r = word_less(a, b);
            if (r) return r < 0;
            return tie_break(a, b);
        });
    }
    uint64_t out = 0;
    for (uint64_t i = 0; i < count;) {
        uint64_t j = i;
        double sr = 0.0, si = 0.0;
        while (j < count && word_less(idx[i], idx[j]) == 0) {
            sr = sr + coefficients[2 * idx[j]];
            si = si + coefficients[2 * idx[j] + 1];
            ++j;
        }
        if (!(sr == 0.0 && si == 0.0)) {
            for (uint32_t k = 0; k < w; ++k) {
                out_x[out * w + k] = xw[idx[i] * w + k];
                out_z[out * w + k] = zw[idx[i] * w + k];
            }
            out_coefficients[2 * out] = sr;
            out_coefficients[2 * out + 1] = si;
            ++out;
        }
        i = j;
    }
    *out_count = out;
    return TCP_OK;
}

extern "C" size_t tcp_last_error(char *buffer, size_t capacity) {
    const std::string &m = tcp::g_last_error;
    if (buffer != nullptr && capacity > 0) {
        size_t n = std::min(capacity - 1, m.size());
        std::memcpy(buffer, m.data(), n);
        buffer[n] = '\0';
    }
    return m.size();
}

extern "C" int tcp_abi_version(void) { return TCP_ABI_VERSION; }

extern "C" int tcp_last_error_fields(uint64_t *fields) {
    if (fields != nullptr) {
        fields[0] = tcp::g_last_fields[0];
        fields[1] = tcp::g_last_fields[1];
    }
    return tcp::g_last_status;
}
