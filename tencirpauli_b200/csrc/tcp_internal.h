// Internal declarations shared by the host plan builder (tcp_plan.cpp) and the
// CUDA side (tcp_mvp.cu) of libtcpmvp.so.  Not part of the public C ABI.
#pragma once

#include <cstdint>
#include <cstdio>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/tcp_mvp.h"

#include <nvtx3/nvToolsExt.h>

namespace tcp {

// NVTX range over a scope (plan building, uploads, applies), so that a
// timeline profiler shows where the host side of the library spends its
// time.  NVTX is header-only and costs a null-function call when no tool is
// attached.
struct Range {
    explicit Range(const char *name) { nvtxRangePushA(name); }
    ~Range() { nvtxRangePop(); }
    Range(const Range &) = delete;
    Range &operator=(const Range &) = delete;
};

// Thread-local last-error slot behind tcp_last_error().
void set_error(const std::string &message);
int fail(int status, const std::string &message);
// The same with the numeric fields of the PauliError variant (expected /
// actual, requested / limit, code / index, index / 0), read back through
// tcp_last_error_fields so that a binding can rebuild the variant exactly.
int fail_fields(int status, const std::string &message, uint64_t a, uint64_t b);
uint64_t clamp_u64(unsigned __int128 v);
// InvalidStructureLength {expected, actual}: "expected structure length E, got A"
int length_error(uint64_t expected, uint64_t actual);

// One compiled term: StatevectorPauliAction masks in the MSB index space and
// the weighted phase c * i^{#Y} (pauli_action.rs:58-86, hamiltonian.rs:564-571).
struct MatrixTerm {
    uint64_t x_mask;
    uint64_t z_mask;
    double w_re;
    double w_im;
};

// Tile schedule for the batched kernel.  The 2^n rows are cut into tiles of
// 2^tile_bits consecutive rows.  Every x-mask group m splits into an outer
// pattern d = m >> tile_bits (which source tile feeds an output tile: the tile
// index XOR d) and an inner mask m & (2^tile_bits - 1) (a permutation inside
// the tile).  A "step" is one distinct outer pattern with all groups that share
// it; one tile load serves every group of a step.
//
// Inside a tile, thread t of a CTA with 2^log_threads threads owns rows
// t + j * 2^log_threads (j = 0 .. 2^(tile_bits-log_threads) - 1).  For group
// inner mask m the thread reads source rows (t ^ (m & (T-1))) + jj * T and row
// j takes source jj = j ^ (m >> log_threads).  The sign of a term at source
// column c = (tile ^ d) * 2^S + local is
//   parity(zt & tile) ^ parity(zt & d) ^ parity(zlo & t) ^ parity(zlo & m_lo) ^ parity(zj & jj)
// with zt = z >> S, zlo = z & (T-1), m_lo = m & (T-1),
// zj = (z & (2^S-1)) >> log_threads.  The schedule folds parity(zt & d) and
// parity(zlo & m_lo) into the term's weight and stores the 2^(S-logT)-bit
// pattern parity(zj & jj); the kernel applies parity(zt & tile) once per step
// and tile, and parity(zlo & t) per thread.
struct Schedule {
    uint32_t tile_bits = 0;
    uint32_t log_threads = 0;
    uint64_t distinct_outer = 0;      // distinct outer patterns d
    // step view (k_batched).  A step is one outer pattern d and a block of
    // its groups and terms no larger than kBlockBytesMax; a pattern with more
    // data is split over several steps (the tile is loaded once per step).
    // step_info: 4 words per step: d (lo, hi), block offset / 16,
    // group count | (block bytes / 16) << 16.
    std::vector<uint32_t> step_info;
    // Step blocks, 16-byte aligned: group records (16 B: inner mask, first
    // term, end term, 0) then term records (32 B: zlo | pattern << 32 |
    // kind << 56, zt, weight).  The weight has parity(zt & d) folded in and is
    // two doubles (complex128 blocks) or two floats + 8 pad bytes (complex64).
    std::vector<uint8_t> blocks_c128;
    std::vector<uint8_t> blocks_c64;
    // group view (row kernel, transition count, diagonal): unfolded
    std::vector<uint64_t> g_mask;     // full x mask per group (schedule order)
    std::vector<uint32_t> g_tbeg;     // terms of group g: [g_tbeg[g], g_tbeg[g+1])
    std::vector<uint64_t> t_z;        // z mask of each term, schedule order
    std::vector<double> t_w;          // weighted phase (re, im), schedule order
    std::vector<float> t_wf;          // the same rounded to FP32 (re, im)
};

// Schedule of the ring kernel (k_ring).  Same tiles and steps as Schedule
// (one step per distinct outer pattern d, split when its block outgrows
// kRingBlockBytes), but the groups of a step are arranged in cosets: groups
// whose inner masks agree on the thread bits (m & (2^log_threads - 1)) read
// the same 2^(S - log_threads) source values per thread, in a permuted order,
// so the values are loaded once per coset, in row order (fixed offsets), and
// every group of the coset applies them through a compile-time register
// permutation a = jh (its inner-mask bits above the thread bits).
//
// A group's terms are cut into runs: one run per kind of weight (real or
// imaginary) and per row part zj of the z mask (its bits above the thread
// bits).  Inside a run the signs of a thread's 8 source values differ only by
// parity(zj & s) of the source row s, the same for every thread, so the kernel
// keeps the loaded values multiplied by that sign (a run names the bits in
// which its zj differs from the run before), sums the run's signed weights
// into one scalar D per thread and multiplies the 8 values by it: the work per
// term is a sign and an addition per thread, the multiply-adds are paid once
// per run.
// The sign of a term is parity(zs & c) with zs = zlo | zt << 9 against the
// thread's constant word c = t | tile << 9 (hence n - 3 <= 32); parity(zt & d)
// ^ parity(zlo & m_lo) is folded into the weight.
//
// The signed sum of a run takes two forms, mixed freely:
//   singles   one record per term: zs and weight;
//   tables    terms whose zs lie in one affine space z0 ^ span(v1 .. vr),
//             r <= 4: their sum is (-1)^parity(z0 & c) T[i] with bit k of i =
//             parity(v_{k+1} & c) and T the 2^r signed sums of the weights,
//             formed in double precision when the plan is built.
// A table costs about as much as 2 to 4 singles whatever the number of its
// terms: Jordan-Wigner two-body groups (16 terms in a 4-dimensional space)
// take one table of 16.
//
// A step's block is one stream of records, walked front to back:
//   header    {record count, 0, 0, 0}
//   record    {zs or z0, word, ...}: single {.., f64 weight} or (complex64)
//             {.., f32 weight, 0}; table of 4 {.., v1, v2} and 4 weights; table
//             of 8 or 16 {.., v1, v2}, {v3, v4 or 0, 0, 0} and the weights
// The word (kRing* below) names the run (a, imag, row signs to flip) and tells
// where it ends, where a coset begins (the 8 source values are loaded then)
// and, complex64, where the partial sums are folded into the compensated row
// sums (in a schedule without complex128 blocks a new coset follows a fold, so
// that the 16-row kernel holds no loaded values across it).  Records are 16-byte
// aligned and the next one is loaded while the present one is applied, so a
// block leaves 16 bytes of its stage unused.
constexpr uint32_t kRingImag = 1u << 4;       // bits 0..3: the register permutation a
constexpr uint32_t kRingKindShift = 5;        // 0 single, 1 / 2 / 3: table of 4 / 8 / 16
constexpr uint32_t kRingKindMask = 3u << kRingKindShift;
constexpr uint32_t kRingLast = 1u << 7;       // last record of its run: apply
constexpr uint32_t kRingNew = 1u << 8;        // first record of its coset: load
constexpr uint32_t kRingFold = 1u << 9;       // complex64: fold the partial sums after this run
constexpr uint32_t kRingFlipShift = 10;       // 4 bits: negate the loaded values of rows with this bit set
constexpr uint32_t kRingFlipMask = 15u << kRingFlipShift;
constexpr uint32_t kRingMaskShift = 14;       // 9 bits: m_lo

constexpr uint32_t kRingFoldRuns = 16;        // complex64: runs per fold

// Bytes of a record of each kind.
constexpr uint32_t ring_record_bytes(uint32_t kind, uint32_t weight_bytes) {
    return kind == 0 ? 16u : (kind == 1 ? 16u : 32u) + (weight_bytes << (kind + 1));
}

struct RingSchedule {
    uint32_t tile_bits = 0;
    uint32_t log_threads = 0;
    uint64_t cosets = 0;               // coset loads per output tile
    uint64_t runs = 0;                 // runs per output tile
    uint64_t work = 0;                 // steps spent on finding the sign tables
    // 4 words per step: d, complex128 block offset / 16, complex64 block
    // offset / 16, complex128 block bytes / 16 | complex64 block bytes / 16 << 16
    std::vector<uint32_t> step_info;
    std::vector<uint8_t> blocks_c128;
    std::vector<uint8_t> blocks_c64;
};

constexpr uint32_t kRingBlockBytes = 8192;
// A tile's row bits: thread bits [low, low + log_threads), register bits the
// rest, bit 0 of the register index first (low = 1: row bit 0 is register bit 0).
struct RingShapeBits {
    uint32_t tile_bits, log_threads, low;
};
constexpr RingShapeBits kRingShapes[] = {{12, 9, 0}, {13, 9, 1}};
constexpr int kRingShapeCount = 2;
constexpr uint32_t kRingMaxZBits = 32;   // zs holds the z bits that are not register bits

// `c128`: with the complex128 blocks (the complex64 blocks are always built).
RingSchedule build_ring_schedule(const std::vector<MatrixTerm> &terms, uint32_t nqubits, RingShapeBits shape,
                                 bool c128 = true);

constexpr uint32_t kBlockBytesMax = 16384;
constexpr uint32_t kGroupRecBytes = 16;
constexpr uint32_t kTermRecBytes = 32;

// Term kinds (uniform per term): the weight is real, imaginary, or general.
enum : uint32_t { kKindReal = 0, kKindImag = 1, kKindComplex = 2 };

// Build the schedule for one tile width.  Groups are the distinct x masks
// (group_matrix_terms, hamiltonian.rs:573-582); terms keep canonical order
// inside a group so the per-group diagonal sum rounds exactly as the
// reference's eager diagonal (hamiltonian.rs:125-133).
// `blocks` = false leaves the step blocks out (step_info still counts them).
Schedule build_schedule(const std::vector<MatrixTerm> &terms, uint32_t nqubits, uint32_t tile_bits,
                        uint32_t log_threads, bool blocks = true);

// Compile packed words into matrix terms (pauli_action.rs:24-88).
int compile_terms(uint32_t nqubits, uint64_t count, uint32_t word_count, const uint64_t *x_words,
                  const uint64_t *z_words, const double *coefficients, std::vector<MatrixTerm> &out);

uint64_t distinct_x_masks(const std::vector<MatrixTerm> &terms);

// Device allocation wrapper with host-side failure injection: when the
// environment variable TCP_FAIL_ALLOC_AFTER=N is set, the allocation after the
// first N successful ones reports failure (nothing touches the GPU).
bool injected_alloc_failure();

}  // namespace tcp
