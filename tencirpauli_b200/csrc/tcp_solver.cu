// libtcpmvp.so -- eigensolver kernels built on the MVP: FP64 block
// inner products and block combinations over complex64 or complex128 vector
// storage, per-basis-state features, the Jacobi and learned (MLP)
// preconditioners, and the MLP's training kernels (forward, backward, Adam).
//
// Vectors are stored RHS-major (vector v at offset v * n) as complex64 or
// complex128; every reduction and combination accumulates in FP64.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <type_traits>
#include <string>
#include <vector>

#include "../../include/tcp_solver.h"
#include "tcp_device.cuh"
#include "tcp_plan_impl.h"

using namespace tcpdev;
using tcp::cuda_fail;
using tcp::fail;

namespace {

constexpr int kGramThreads = 512;      // 16 warps, one CTA per SM
constexpr int kGramWarps = kGramThreads / 32;
constexpr int kGramPairs = 16;         // (i, j) pairs of one warp tile
constexpr int kGramMaxVectors = 96;    // p + q
constexpr int kGramMaxPairs = 512;     // p * q
constexpr int kGramBlocks = 296;       // partial-sum slots in the work buffer
constexpr int kGramGrid = 148;         // CTAs launched (<= kGramBlocks)
constexpr int kGramRedBytes = 96 * 1024;  // shared memory for the row-group sums
constexpr int kGramStages = 4;            // TMA pipeline depth (chunks)
constexpr uint32_t kGramStageBytes = 48 * 1024;  // one chunk of every vector

constexpr int kCombineThreads = 256;
constexpr int kCombineTile = 4;        // output vectors per thread
constexpr int kCombineUnroll = 8;      // complex128 source vectors loaded ahead (16 for complex64)
constexpr int kCombineMaxK = 32;       // output vectors per launch

__device__ __forceinline__ double2 load_c(const void *base, int c64, uint64_t idx) {
    if (c64) {
        const float2 v = static_cast<const float2 *>(base)[idx];
        return make_double2(v.x, v.y);
    }
    return static_cast<const double2 *>(base)[idx];
}
__device__ __forceinline__ void store_c(void *base, int c64, uint64_t idx, double2 v) {
    if (c64) {
        static_cast<float2 *>(base)[idx] = make_float2(static_cast<float>(v.x), static_cast<float>(v.y));
    } else {
        static_cast<double2 *>(base)[idx] = v;
    }
}
template <bool C64> __device__ __forceinline__ double2 load_v(const void *base, uint64_t idx) {
    if constexpr (C64) {
        const float2 v = __ldg(static_cast<const float2 *>(base) + idx);
        return make_double2(v.x, v.y);
    } else {
        return __ldg(static_cast<const double2 *>(base) + idx);
    }
}

__device__ __forceinline__ uint64_t umin64(uint64_t a, uint64_t b) { return a < b ? a : b; }

// t += conj(a) * b in FP64.
__device__ __forceinline__ void cmac(double2 &t, double2 a, double2 b) {
    t.x = fma(a.x, b.x, fma(a.y, b.y, t.x));
    t.y = fma(a.x, b.y, fma(-a.y, b.x, t.y));
}

// Per-CTA partial sums of G = A^H B.  The p x q pairs are cut into warp
// tiles of PI x QJ pairs (PI vectors of A, QJ of B: 8 x 1, 8 x 2 or 4 x 4,
// at most kGramPairs).  The CTA's rows are dealt to `groups` row groups, and
// its 16 warps take the (tile, row group) slots in turn: with groups chosen so
// that slots is a multiple of 16, every warp does the same work.  Warps walk
// the same 32-row chunks, so the B rows one tile reads are shared through L1
// by the warps of the other tiles and every vector crosses HBM once.  Each
// lane keeps its pair sums in FP64 registers; the warp reduces them by a
// fixed butterfly (commutative steps, so every lane holds the same bits), the
// row groups of a tile are summed in a fixed order from shared memory, and
// the CTA writes partial[block][i + p*j].  RPL = 2 (both blocks complex64,
// n even, 16-byte aligned) gives each lane two rows per chunk.
template <int QJ, bool A64, bool B64, int RPL>
__global__ void __launch_bounds__(kGramThreads, 1)
    k_gram_tiles(const void *__restrict__ A, uint32_t p, const void *__restrict__ B, uint32_t q, uint64_t n,
                 uint32_t groups, double2 *__restrict__ partial) {
    constexpr int PI = QJ == 4 ? 4 : 8;
    constexpr int TP = PI * QJ;
    static_assert(TP <= kGramPairs, "tile shape");
    extern __shared__ double2 red[];  // [slot][TP] when groups > 1
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t ni = (p + PI - 1) / PI, nj = (q + QJ - 1) / QJ, ntiles = ni * nj;
    const uint32_t slots = groups * ntiles;
    const uint32_t pairs = p * q;
    const uint64_t chunks = (n + 32 * RPL - 1) / (32 * RPL);
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * groups;
    for (uint32_t s = warp; s < slots; s += kGramWarps) {
        const uint32_t tile = s % ntiles, rg = s / ntiles;
        const uint32_t i0 = (tile % ni) * PI, j0 = (tile / ni) * QJ;
        double2 acc[TP];
#pragma unroll
        for (int e = 0; e < TP; ++e) acc[e] = make_double2(0.0, 0.0);
        for (uint64_t c = static_cast<uint64_t>(blockIdx.x) * groups + rg; c < chunks; c += stride) {
            if constexpr (RPL == 1) {
                const uint64_t row = c * 32 + lane;
                if (row < n) {
                    double2 b[QJ], a[PI];
#pragma unroll
                    for (int jj = 0; jj < QJ; ++jj)
                        b[jj] = j0 + jj < q ? load_v<B64>(B, static_cast<uint64_t>(j0 + jj) * n + row)
                                            : make_double2(0.0, 0.0);
#pragma unroll
                    for (int ii = 0; ii < PI; ++ii)
                        a[ii] = i0 + ii < p ? load_v<A64>(A, static_cast<uint64_t>(i0 + ii) * n + row)
                                            : make_double2(0.0, 0.0);
#pragma unroll
                    for (int ii = 0; ii < PI; ++ii) {
#pragma unroll
                        for (int jj = 0; jj < QJ; ++jj) cmac(acc[ii * QJ + jj], a[ii], b[jj]);
                    }
                }
            } else {
                // complex64 storage, n even: a lane loads rows 2 lane and
                // 2 lane + 1 of every vector as one 16-byte float4
                const uint64_t row = c * 64 + 2 * lane;
                if (row < n) {
                    const float4 *A4 = static_cast<const float4 *>(A), *B4 = static_cast<const float4 *>(B);
                    float4 b[QJ], a[PI];
#pragma unroll
                    for (int jj = 0; jj < QJ; ++jj)
                        b[jj] = j0 + jj < q ? __ldg(B4 + (static_cast<uint64_t>(j0 + jj) * n + row) / 2)
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int ii = 0; ii < PI; ++ii)
                        a[ii] = i0 + ii < p ? __ldg(A4 + (static_cast<uint64_t>(i0 + ii) * n + row) / 2)
                                            : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int ii = 0; ii < PI; ++ii) {
#pragma unroll
                        for (int jj = 0; jj < QJ; ++jj) {
                            cmac(acc[ii * QJ + jj], make_double2(a[ii].x, a[ii].y), make_double2(b[jj].x, b[jj].y));
                            cmac(acc[ii * QJ + jj], make_double2(a[ii].z, a[ii].w), make_double2(b[jj].z, b[jj].w));
                        }
                    }
                }
            }
        }
#pragma unroll
        for (int e = 0; e < TP; ++e) {
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                acc[e].x += __shfl_xor_sync(0xffffffffu, acc[e].x, off);
                acc[e].y += __shfl_xor_sync(0xffffffffu, acc[e].y, off);
            }
        }
#pragma unroll
        for (int e = 0; e < TP; ++e) {
            if (lane == static_cast<uint32_t>(e)) {
                if (groups == 1u) {
                    const uint32_t i = i0 + e / QJ, j = j0 + e % QJ;
                    if (i < p && j < q) partial[static_cast<size_t>(blockIdx.x) * pairs + i + p * j] = acc[e];
                } else {
                    red[s * TP + e] = acc[e];
                }
            }
        }
    }
    if (groups > 1u) {
        __syncthreads();
        for (uint32_t t = threadIdx.x; t < ntiles * TP; t += blockDim.x) {
            const uint32_t tile = t / TP, e = t % TP;
            double2 sum = make_double2(0.0, 0.0);
            for (uint32_t rg = 0; rg < groups; ++rg) {
                const double2 v = red[(rg * ntiles + tile) * TP + e];
                sum.x += v.x;
                sum.y += v.y;
            }
            const uint32_t i = (tile % ni) * PI + e / QJ, j = (tile / ni) * QJ + e % QJ;
            if (i < p && j < q) partial[static_cast<size_t>(blockIdx.x) * pairs + i + p * j] = sum;
        }
    }
}

// 2-D tiled TMA load of one box (x: innermost coordinate in 8-byte units,
// y: vector index) into shared memory; completes the box bytes on `bar`.
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, int x, int y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

// G = A^H B for two blocks of the same storage type, fed by the TMA engine.
// The blocks are described by two 2-D tensor maps (vectors x 8-byte units),
// and a chunk is one box of each: `rows` rows of every vector.  A CTA walks
// its full chunks (chunk c = blockIdx.x + k * gridDim.x) through a
// kGramStages-deep ring in shared memory; thread 0 issues the two box loads
// of a chunk onto the stage's mbarrier kGramStages - 1 chunks ahead of the
// consumers, so the loads in flight hold no registers.  The last n % rows
// rows are read straight from global memory by the CTA next in turn.  Warp w
// takes tile w % ntiles and row group w / ntiles (ntiles * groups <= 16); its
// lanes keep the tile's pair sums in FP64 registers.  The reduction order is
// fixed (warp butterfly, row groups, then k_gram_reduce over CTAs).  A box
// that does not land within the bounded wait poisons this CTA's partial sums
// with NaN, after a bounded wait for the boxes still in flight, so the caller
// sees a non-finite Gram matrix.
template <int QJ, bool C64>
__global__ void __launch_bounds__(kGramThreads, 1)
    k_gram_tma(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
               const void *__restrict__ A, uint32_t p, const void *__restrict__ B, uint32_t q, uint64_t n,
               uint32_t rows, uint32_t groups, double2 *__restrict__ partial) {
    using E = std::conditional_t<C64, float2, double2>;
    constexpr int PI = QJ == 4 ? 4 : 8;
    constexpr int TP = PI * QJ;
    constexpr int UNITS = sizeof(E) / 8;  // 8-byte units per element
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full[kGramStages];
    __shared__ double2 red[kGramWarps][kGramPairs];
    E *ring = reinterpret_cast<E *>(smem_raw);
    const uint32_t vecs = p + q;
    const size_t stage_elems = static_cast<size_t>(vecs) * rows;
    const uint32_t stage_bytes = static_cast<uint32_t>(stage_elems * sizeof(E));
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const uint32_t ni = (p + PI - 1) / PI, nj = (q + QJ - 1) / QJ, ntiles = ni * nj;
    const uint32_t pairs = p * q;
    const uint64_t chunks = n / rows;  // full chunks only
    const uint64_t mine = chunks > blockIdx.x ? (chunks - blockIdx.x + gridDim.x - 1) / gridDim.x : 0;

    if (tid == 0) {
        for (int st = 0; st < kGramStages; ++st) mbar_init(&full[st], 1);
        fence_mbar_init();
    }
    __syncthreads();
    // chunk k of this CTA -> stage k % kGramStages
    auto issue = [&](uint64_t k) {
        const uint64_t r0 = (blockIdx.x + k * gridDim.x) * static_cast<uint64_t>(rows);
        uint64_t *bar = &full[k % kGramStages];
        E *dst = ring + (k % kGramStages) * stage_elems;
        mbar_arrive_expect_tx(bar, stage_bytes);
        tma_load_2d(dst, &ta, static_cast<int>(r0 * UNITS), 0, bar);
        tma_load_2d(dst + static_cast<size_t>(p) * rows, &tb, static_cast<int>(r0 * UNITS), 0, bar);
    };
    if (tid == 0) {
        for (uint64_t k = 0; k < mine && k + 1 < static_cast<uint64_t>(kGramStages); ++k) issue(k);
    }

    const bool active = warp < ntiles * groups;
    const uint32_t tile = warp % ntiles, rg = warp / ntiles;
    const uint32_t i0 = (tile % ni) * PI, j0 = (tile / ni) * QJ;
    double2 acc[TP];
#pragma unroll
    for (int e = 0; e < TP; ++e) acc[e] = make_double2(0.0, 0.0);
    // one row of the tile's vectors, from shared memory or from global memory
    auto accumulate = [&](const E *sa, const E *sb, size_t stride, uint64_t r) {
        double2 a[PI], b[QJ];
#pragma unroll
        for (int jj = 0; jj < QJ; ++jj) {
            if (j0 + jj < q) {
                const E v = sb[(j0 + jj) * stride + r];
                b[jj] = make_double2(v.x, v.y);
            } else {
                b[jj] = make_double2(0.0, 0.0);
            }
        }
#pragma unroll
        for (int ii = 0; ii < PI; ++ii) {
            if (i0 + ii < p) {
                const E v = sa[(i0 + ii) * stride + r];
                a[ii] = make_double2(v.x, v.y);
            } else {
                a[ii] = make_double2(0.0, 0.0);
            }
        }
#pragma unroll
        for (int ii = 0; ii < PI; ++ii) {
#pragma unroll
            for (int jj = 0; jj < QJ; ++jj) cmac(acc[ii * QJ + jj], a[ii], b[jj]);
        }
    };
    for (uint64_t k = 0; k < mine; ++k) {
        const uint32_t st = static_cast<uint32_t>(k % kGramStages);
        const bool ok = mbar_wait_bounded(&full[st], static_cast<uint32_t>(k / kGramStages) & 1u);
        if (__syncthreads_or(!ok)) {
            if (tid == 0) {
                // let the boxes already issued land before the CTA exits
                const uint64_t issued = umin64(mine, k + kGramStages - 1);
                for (uint64_t kk = k; kk < issued; ++kk)
                    mbar_wait_bounded(&full[kk % kGramStages], static_cast<uint32_t>(kk / kGramStages) & 1u,
                                      kWaitLimitNs / 4);
            }
            const double nan = __longlong_as_double(0x7ff8000000000000ll);
            for (uint32_t pr = tid; pr < pairs; pr += blockDim.x)
                partial[static_cast<size_t>(blockIdx.x) * pairs + pr] = make_double2(nan, nan);
            return;
        }
        // every thread has finished chunk k - 1, so its stage can be refilled
        if (tid == 0 && k + kGramStages - 1 < mine) {
            fence_proxy_async_smem();
            issue(k + kGramStages - 1);
        }
        if (active) {
            const E *sa = ring + st * stage_elems;
            for (uint32_t r = rg * 32 + lane; r < rows; r += groups * 32) accumulate(sa, sa + static_cast<size_t>(p) * rows, rows, r);
        }
    }
    const uint64_t tail0 = chunks * rows;
    if (active && tail0 < n && blockIdx.x == chunks % gridDim.x) {
        for (uint64_t r = tail0 + rg * 32 + lane; r < n; r += groups * 32)
            accumulate(static_cast<const E *>(A), static_cast<const E *>(B), n, r);
    }
#pragma unroll
    for (int e = 0; e < TP; ++e) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            acc[e].x += __shfl_xor_sync(0xffffffffu, acc[e].x, off);
            acc[e].y += __shfl_xor_sync(0xffffffffu, acc[e].y, off);
        }
    }
    if (active) {
#pragma unroll
        for (int e = 0; e < TP; ++e)
            if (lane == static_cast<uint32_t>(e)) red[warp][e] = acc[e];
    }
    __syncthreads();
    for (uint32_t t = tid; t < ntiles * TP; t += blockDim.x) {
        const uint32_t tl = t / TP, e = t % TP;
        double2 sum = make_double2(0.0, 0.0);
        for (uint32_t g = 0; g < groups; ++g) {
            const double2 v = red[g * ntiles + tl][e];
            sum.x += v.x;
            sum.y += v.y;
        }
        const uint32_t i = (tl % ni) * PI + e / QJ, j = (tl / ni) * QJ + e % QJ;
        if (i < p && j < q) partial[static_cast<size_t>(blockIdx.x) * pairs + i + p * j] = sum;
    }
}

// Deterministic reduction of the per-block partials: a block takes 32 pairs;
// warp w adds the partials w, w + 32, ... of each (coalesced across the lanes),
// then warp 0 adds the 32 sums in warp order: 4 us.  (One thread per pair walking
// all 148 partials takes 20, most of it load latency.)
constexpr int kGramReduceWarps = 32;
__global__ void __launch_bounds__(kGramReduceWarps * 32)
    k_gram_reduce(const double2 *__restrict__ partial, uint32_t blocks, uint32_t pairs, double2 *__restrict__ out) {
    __shared__ double2 red[kGramReduceWarps][32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t pr = blockIdx.x * 32u + lane;
    double re = 0.0, im = 0.0;
    if (pr < pairs) {
        for (uint32_t b = warp; b < blocks; b += kGramReduceWarps) {
            const double2 v = partial[static_cast<size_t>(b) * pairs + pr];
            re += v.x;
            im += v.y;
        }
    }
    red[warp][lane] = make_double2(re, im);
    __syncthreads();
    if (warp != 0 || pr >= pairs) return;
    for (int w = 1; w < kGramReduceWarps; ++w) {
        re += red[w][lane].x;
        im += red[w][lane].y;
    }
    out[pr] = make_double2(re, im);
}

// out[:, j] = alpha * sum_i A[:, i] S[i, j] + beta * out[:, j]  (FP64 arithmetic).
// A CTA covers rb = 256 / njp consecutive rows for njp tiles of kCombineTile
// output vectors (njp: the tile count rounded up to a power of two); the
// tiles of the same rows sit in one CTA, so each source row is fetched from
// HBM once and re-read from L1.  Source values are loaded 8 (complex128) or
// 16 (complex64) ahead of their multiply-adds, and every output sums
// i = 0..p-1 in order.
// S is staged column-major as p x (njp * kCombineTile), zero beyond k.
template <bool A64, bool O64>
__global__ void __launch_bounds__(kCombineThreads)
    k_combine_tiles(const void *__restrict__ A, uint32_t p, const double2 *__restrict__ S, uint32_t k, uint32_t njp,
                    uint64_t n, double alpha, double beta, void *__restrict__ out) {
    extern __shared__ double2 ss[];
    const uint32_t kpad = njp * kCombineTile;
    for (uint32_t e = threadIdx.x; e < p * kpad; e += blockDim.x) {
        const uint32_t j = e / p;
        ss[e] = j < k ? S[e] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    const uint32_t rb = kCombineThreads / njp;
    const uint32_t jt = threadIdx.x / rb;
    if (jt * kCombineTile >= k) return;  // padding tile: no further barrier below
    constexpr int U = A64 ? 2 * kCombineUnroll : kCombineUnroll;
    const double2 *sj = ss + static_cast<size_t>(p) * jt * kCombineTile;
    for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * rb + threadIdx.x % rb; r < n;
         r += static_cast<uint64_t>(gridDim.x) * rb) {
        double2 acc[kCombineTile];
#pragma unroll
        for (int jj = 0; jj < kCombineTile; ++jj) acc[jj] = make_double2(0.0, 0.0);
        uint32_t i = 0;
        for (; i + U <= p; i += U) {
            double2 a[U];
#pragma unroll
            for (int u = 0; u < U; ++u) a[u] = load_v<A64>(A, static_cast<uint64_t>(i + u) * n + r);
#pragma unroll
            for (int u = 0; u < U; ++u) {
#pragma unroll
                for (int jj = 0; jj < kCombineTile; ++jj) {
                    const double2 sv = sj[i + u + p * jj];
                    acc[jj].x = fma(a[u].x, sv.x, fma(-a[u].y, sv.y, acc[jj].x));
                    acc[jj].y = fma(a[u].x, sv.y, fma(a[u].y, sv.x, acc[jj].y));
                }
            }
        }
        for (; i < p; ++i) {
            const double2 a = load_v<A64>(A, static_cast<uint64_t>(i) * n + r);
#pragma unroll
            for (int jj = 0; jj < kCombineTile; ++jj) {
                const double2 sv = sj[i + p * jj];
                acc[jj].x = fma(a.x, sv.x, fma(-a.y, sv.y, acc[jj].x));
                acc[jj].y = fma(a.x, sv.y, fma(a.y, sv.x, acc[jj].y));
            }
        }
#pragma unroll
        for (int jj = 0; jj < kCombineTile; ++jj) {
            const uint32_t j = jt * kCombineTile + jj;
            if (j < k) {
                double2 v = make_double2(alpha * acc[jj].x, alpha * acc[jj].y);
                if (beta != 0.0) {
                    const double2 o = load_c(out, O64, static_cast<uint64_t>(j) * n + r);
                    v.x = fma(beta, o.x, v.x);
                    v.y = fma(beta, o.y, v.y);
                }
                store_c(out, O64, static_cast<uint64_t>(j) * n + r, v);
            }
        }
    }
}

// The same for complex64 sources and outputs, two consecutive rows per thread:
// one 16-byte load brings both, and every coefficient load from shared memory
// (two cycles of the load pipe per warp, as long as its four multiply-adds take
// one row) serves both.  Needs n even and 16-byte aligned blocks.  n = 2^22,
// 40 sources, 4 outputs: 338 us one row per thread, 250 two (HBM: 215).
constexpr int kCombinePairUnroll = 8, kCombinePairBlocks = 3;  // resident blocks per SM: 80 registers
// With more than 4 outputs a block's time is its arithmetic, and with half the row
// blocks of one row per thread an SM that gets one more than the others shows: the
// pairs then need 9 rounds of blocks or 93 % of the last one.  64 sources, pairs
// against one row: 16 outputs, 460 blocks of rows 39.3 and 35.2 us, 700 blocks 45.5
// and 47.5; 24 outputs, 600 blocks 41.3 and 37.2; 8 outputs, 1200 blocks 79.7 and
// 88.3.  4 outputs, 600 blocks: 47.8 and 49.5.  With 17 to 20 outputs three of a
// block's eight tiles are padding, and the pairs gain from 13 rounds on: 20 outputs,
// 1400 blocks 59.8 and 55.7, 2100 blocks 87.6 and 91.8.
bool combine_by_pairs(uint32_t k, uint32_t njp, uint64_t blocks) {
    const uint64_t rounds = (blocks + 147) / 148;
    if (k > 16 && k <= 20) return rounds > 12;
    return njp == 1 || rounds > 8 || 100 * blocks >= 93 * 148 * rounds;
}
__global__ void __launch_bounds__(kCombineThreads, kCombinePairBlocks)
    k_combine_pairs(const float4 *__restrict__ A, uint32_t p, const double2 *__restrict__ S, uint32_t k, uint32_t njp,
                    uint64_t half, double alpha, double beta, float4 *__restrict__ out) {
    extern __shared__ double2 ss[];
    const uint32_t kpad = njp * kCombineTile;
    // row i of the staged coefficients: its kpad outputs
    for (uint32_t e = threadIdx.x; e < p * kpad; e += blockDim.x) {
        const uint32_t i = e / kpad, j = e % kpad;
        ss[e] = j < k ? S[i + static_cast<size_t>(j) * p] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    const uint32_t rb = kCombineThreads / njp;
    const uint32_t jt = threadIdx.x / rb;
    if (jt * kCombineTile >= k) return;  // padding tile: no further barrier below
    constexpr int U = kCombinePairUnroll;
    const double2 *sj = ss + jt * kCombineTile;
    for (uint64_t r = static_cast<uint64_t>(blockIdx.x) * rb + threadIdx.x % rb; r < half;
         r += static_cast<uint64_t>(gridDim.x) * rb) {
        double2 acc[kCombineTile][2];
#pragma unroll
        for (int jj = 0; jj < kCombineTile; ++jj) acc[jj][0] = acc[jj][1] = make_double2(0.0, 0.0);
        auto add = [&](float4 v, uint32_t i) {
            const double2 a0 = make_double2(v.x, v.y), a1 = make_double2(v.z, v.w);
#pragma unroll
            for (int jj = 0; jj < kCombineTile; ++jj) {
                const double2 sv = sj[i * kpad + jj];
                acc[jj][0].x = fma(a0.x, sv.x, fma(-a0.y, sv.y, acc[jj][0].x));
                acc[jj][0].y = fma(a0.x, sv.y, fma(a0.y, sv.x, acc[jj][0].y));
                acc[jj][1].x = fma(a1.x, sv.x, fma(-a1.y, sv.y, acc[jj][1].x));
                acc[jj][1].y = fma(a1.x, sv.y, fma(a1.y, sv.x, acc[jj][1].y));
            }
        };
        uint32_t i = 0;
        for (; i + U <= p; i += U) {
            float4 a[U];
#pragma unroll
            for (int u = 0; u < U; ++u) a[u] = __ldg(A + static_cast<uint64_t>(i + u) * half + r);
#pragma unroll
            for (int u = 0; u < U; ++u) add(a[u], i + u);
        }
        for (; i < p; ++i) add(__ldg(A + static_cast<uint64_t>(i) * half + r), i);
#pragma unroll
        for (int jj = 0; jj < kCombineTile; ++jj) {
            const uint32_t j = jt * kCombineTile + jj;
            if (j < k) {
                float4 *o = out + static_cast<uint64_t>(j) * half + r;
                double2 v[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) v[e] = make_double2(alpha * acc[jj][e].x, alpha * acc[jj][e].y);
                if (beta != 0.0) {
                    const float4 w = *o;
                    v[0].x = fma(beta, static_cast<double>(w.x), v[0].x);
                    v[0].y = fma(beta, static_cast<double>(w.y), v[0].y);
                    v[1].x = fma(beta, static_cast<double>(w.z), v[1].x);
                    v[1].y = fma(beta, static_cast<double>(w.w), v[1].y);
                }
                *o = make_float4(static_cast<float>(v[0].x), static_cast<float>(v[0].y), static_cast<float>(v[1].x),
                                 static_cast<float>(v[1].y));
            }
        }
    }
}

// Jacobi correction t = -r / (d - theta), |d - theta| clamped below by eps.
__global__ void k_jacobi(const void *__restrict__ R, int r64, uint64_t n, uint32_t k, const double2 *__restrict__ diag,
                         const double *__restrict__ theta, double eps, void *__restrict__ T, int t64) {
    for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; r < n;
         r += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const double d = diag[r].x;
        for (uint32_t j = 0; j < k; ++j) {
            double den = d - theta[j];
            if (fabs(den) < eps) den = den < 0.0 ? -eps : eps;
            const double2 v = load_c(R, r64, j * n + r);
            store_c(T, t64, j * n + r, make_double2(-v.x / den, -v.y / den));
        }
    }
}

// Per-basis-state features that do not depend on the Ritz value (see
// tcp_solver.h): H_ii, the mean and minimum diagonal of the states the row
// couples to, sum |H_ij|, sum |H_ij|^2, the number of couplings, and the
// normalised Hamming weight of the basis state.
__global__ void k_features(DevSchedule s, uint32_t gzero, uint32_t nqubits, uint64_t n, float *__restrict__ feat) {
    for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; r < n;
         r += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        auto diag_at = [&](uint64_t c) -> double {
            double re = 0.0;
            if (gzero != 0xffffffffu) {
                for (uint32_t t = s.g_tbeg[gzero]; t < s.g_tbeg[gzero + 1]; ++t) {
                    const double2 w = s.t_w[t];
                    re += (__popcll(s.t_z[t] & c) & 1) ? -w.x : w.x;
                }
            }
            return re;
        };
        const double hii = diag_at(r);
        double sum_abs = 0.0, sum_sq = 0.0, sum_nd = 0.0, min_nd = 1e300;
        uint32_t count = 0;
        for (uint32_t g = 0; g < s.ngroups; ++g) {
            if (g == gzero) continue;
            const uint64_t c = r ^ s.g_mask[g];
            double dre = 0.0, dim = 0.0;
            for (uint32_t t = s.g_tbeg[g]; t < s.g_tbeg[g + 1]; ++t) {
                const double2 w = s.t_w[t];
                const bool neg = __popcll(s.t_z[t] & c) & 1;
                dre += neg ? -w.x : w.x;
                dim += neg ? -w.y : w.y;
            }
            const double a2 = dre * dre + dim * dim;
            if (a2 == 0.0) continue;
            const double dj = diag_at(c);
            sum_abs += sqrt(a2);
            sum_sq += a2;
            sum_nd += dj;
            min_nd = fmin(min_nd, dj);
            ++count;
        }
        float *f = feat + r * TCP_FEATURES;
        f[0] = static_cast<float>(hii);
        f[1] = static_cast<float>(count ? sum_nd / count : hii);
        f[2] = static_cast<float>(count ? min_nd : hii);
        f[3] = static_cast<float>(sum_abs);
        f[4] = static_cast<float>(sum_sq);
        f[5] = static_cast<float>(count);
        f[6] = static_cast<float>(static_cast<double>(__popcll(r)) / fmax(1.0, static_cast<double>(nqubits)) - 0.5);
        f[7] = 0.f;
    }
}

// ---------------------------------- MLP -------------------------------------
// Network: x (TCP_MLP_IN inputs, built from the features and the Ritz value)
// -> tanh(W1 x + b1) (TCP_MLP_HIDDEN) -> tanh(W2 h1 + b2) (TCP_MLP_HIDDEN)
// -> c = w3 . h2 + b3.  The correction is t = -exp(c) r / max(d - theta, eps):
// c = 0 is the Jacobi correction, and the network learns a per-state factor.
constexpr int IN = TCP_MLP_IN, HID = TCP_MLP_HIDDEN;
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + HID * IN, OFF_W2 = OFF_B1 + HID, OFF_B2 = OFF_W2 + HID * HID,
              OFF_W3 = OFF_B2 + HID, OFF_B3 = OFF_W3 + HID, NPARAM = OFF_B3 + 1;
static_assert(NPARAM == TCP_MLP_PARAMS, "parameter count mismatch");

// Network inputs of one basis state; `scale` normalises energies (a spread of
// the spectrum).  What does not depend on the Ritz value is formed once per
// state: with several residuals the conversions between FP32 and FP64 (16 per
// SM and clock, the pipe of the activations' exponentials) would cost more
// than the inputs' arithmetic.
struct MlpState {
    double f0, f1, f2, f4, inv;
    float x3, x4, x5, x6;
    __device__ __forceinline__ MlpState(const float (&f)[TCP_FEATURES], double scale) {
        inv = 1.0 / scale;
        f0 = f[0];
        f1 = f[1];
        f2 = f[2];
        f4 = f[4];
        x3 = static_cast<float>(static_cast<double>(f[3]) * inv);
        x4 = static_cast<float>(f4 * inv * inv);
        x5 = static_cast<float>(static_cast<double>(f[5]) * 0.05);
        x6 = f[6];
    }
    // Inputs for Ritz value theta; also returns den = f0 - theta, |den| >= eps.
    __device__ __forceinline__ void inputs(double theta, double eps, float (&x)[IN], double &den) const {
        const double d = f0 - theta;
        den = fabs(d) < eps ? (d < 0.0 ? -eps : eps) : d;
        x[0] = static_cast<float>(d * inv);
        x[1] = static_cast<float>((f1 - theta) * inv);
        x[2] = static_cast<float>((f2 - theta) * inv);
        x[3] = x3;
        x[4] = x4;
        x[5] = x5;
        x[6] = x6;
        // size of the second-order (one coupling out and back) term relative to
        // the first-order denominator, squashed to [0, 1)
        const double ratio = f4 / (fabs(den) * fmax(fabs(f1 - theta), eps));
        x[7] = static_cast<float>(ratio / (1.0 + ratio));
    }
};

// tanh(a) = 1 - 2 / (exp(2a) + 1), an exact identity, with the approximate
// exponential and reciprocal: five instructions, about 1e-7 absolute error (all
// the activations need), and it saturates to +-1 for large |a| (the
// exponential overflows to inf or underflows to 0).  The factor 2 log2(e) and
// the final 1 - 2r round once each, as 2a, exp and 2r (powers of two) did.
__device__ __forceinline__ float act_tanh(float a) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(a * 2.885390081777927f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(e + 1.f));
    return fmaf(-2.f, r, 1.f);
}

// The parameters in the order mlp_eval reads them: per unit o of layer 1 its 8
// weights, its bias, three zeros, then its column of W2; then b2, w3, b3.
// Two rows per thread at 64 registers, four blocks of 256 per SM: 506 us for 4
// residuals of 2^22 complex128 states (one row per thread: 690; two rows at
// 80 registers: 527; three at 80: 762; four at 128 registers: 614; two packed
// in f32x2 with doubled weights: 546).
constexpr int kEvalThreads = 256, kEvalBlocks = 4, kEvalRows = 2;
constexpr int kEvalUnit = IN + 4 + HID;
constexpr int kEvalTail = HID * kEvalUnit;
constexpr int kEvalWords = kEvalTail + 2 * HID + 4;
__device__ __forceinline__ void mlp_stage(float *__restrict__ sw, const float *__restrict__ w) {
    for (int e = threadIdx.x; e < kEvalWords; e += blockDim.x) {
        float v = 0.f;
        if (e < kEvalTail) {
            const int o = e / kEvalUnit, k = e % kEvalUnit;
            if (k < IN)
                v = w[OFF_W1 + o * IN + k];
            else if (k == IN)
                v = w[OFF_B1 + o];
            else if (k >= IN + 4)
                v = w[OFF_W2 + (k - IN - 4) * HID + o];
        } else {
            const int k = e - kEvalTail;
            if (k < HID)
                v = w[OFF_B2 + k];
            else if (k < 2 * HID)
                v = w[OFF_W3 + k - HID];
            else if (k == 2 * HID)
                v = w[OFF_B3];
        }
        sw[e] = v;
    }
}

// Network output for V input rows (x(i, v): input i of row v).  The layer-2
// sums are accumulated alongside layer 1, so no activation array is indexed at
// run time, and every weight load serves V rows: shared memory delivers 8
// bytes of a warp-uniform load per clock, and with one row per thread the
// loads took longer than the arithmetic.
template <int V, typename X>
__device__ __forceinline__ void mlp_eval(const float *__restrict__ sw, const X &x, float (&c)[V]) {
    float a2[HID][V];
#pragma unroll
    for (int p = 0; p < HID; ++p)
#pragma unroll
        for (int v = 0; v < V; ++v) a2[p][v] = sw[kEvalTail + p];
#pragma unroll 1
    for (int o = 0; o < HID; ++o) {
        const float4 *unit = reinterpret_cast<const float4 *>(sw + o * kEvalUnit);
        float h[V];
        const float4 u = unit[0], t = unit[1];
        const float bias = sw[o * kEvalUnit + IN];
#pragma unroll
        for (int v = 0; v < V; ++v) {
            float a = fmaf(u.x, x(0, v), bias);
            a = fmaf(u.y, x(1, v), a);
            a = fmaf(u.z, x(2, v), a);
            a = fmaf(u.w, x(3, v), a);
            a = fmaf(t.x, x(4, v), a);
            a = fmaf(t.y, x(5, v), a);
            a = fmaf(t.z, x(6, v), a);
            a = fmaf(t.w, x(7, v), a);
            h[v] = act_tanh(a);
        }
#pragma unroll
        for (int p = 0; p < HID; p += 4) {
            const float4 w = unit[(IN + 4 + p) / 4];
#pragma unroll
            for (int v = 0; v < V; ++v) {
                a2[p][v] = fmaf(w.x, h[v], a2[p][v]);
                a2[p + 1][v] = fmaf(w.y, h[v], a2[p + 1][v]);
                a2[p + 2][v] = fmaf(w.z, h[v], a2[p + 2][v]);
                a2[p + 3][v] = fmaf(w.w, h[v], a2[p + 3][v]);
            }
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v) c[v] = sw[kEvalTail + 2 * HID];
#pragma unroll
    for (int p = 0; p < HID; ++p) {
        const float w = sw[kEvalTail + HID + p];
#pragma unroll
        for (int v = 0; v < V; ++v) c[v] = fmaf(w, act_tanh(a2[p][v]), c[v]);
    }
}

// 8 floats of a row, as two 16-byte loads when the array allows it.
__device__ __forceinline__ void load_row8(const float *__restrict__ row, bool wide, float (&f)[8]) {
    if (wide) {
        const float4 u = __ldg(reinterpret_cast<const float4 *>(row)), v = __ldg(reinterpret_cast<const float4 *>(row) + 1);
        f[0] = u.x, f[1] = u.y, f[2] = u.z, f[3] = u.w, f[4] = v.x, f[5] = v.y, f[6] = v.z, f[7] = v.w;
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = __ldg(row + i);
    }
}

// Learned correction for k residual vectors: t_j = -exp(c) r_j / den with
// den = H_ii - theta_j (FP64 diagonal, clamped by eps, exactly as k_jacobi).
// kEvalRows residuals of a state share its features and every weight load; what is
// left of k goes one by one (2^22 states, one residual: 208 us, 251 as half of a
// pair).  The state's features and diagonal are read again per group of residuals
// rather than held in registers beside the layer-2 sums.
__global__ void __launch_bounds__(kEvalThreads, kEvalBlocks)
    k_mlp_precond(const void *__restrict__ R, int r64, uint64_t n, uint32_t k, const float *feat, int wide,
                  const double2 *diag, const double *theta, double scale, double eps, float clamp,
                  const float *__restrict__ wglob, void *__restrict__ T, int t64) {
    __shared__ __align__(16) float sw[kEvalWords];
    mlp_stage(sw, wglob);
    __syncthreads();
    for (uint64_t r = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; r < n;
         r += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        auto correct = [&](auto rows, uint32_t j0) {  // residuals j0 .. j0 + V - 1
            constexpr int V = decltype(rows)::value;
            float own[4][V], shared[4], c[V];  // inputs 0, 1, 2, 7 and 3 .. 6
            {
                const float *row = feat + r * TCP_FEATURES;
                asm volatile("" : "+l"(row));  // read again, not held
                float f[TCP_FEATURES];
                load_row8(row, wide, f);
                const MlpState state(f, scale);
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    float x[IN];
                    double den;
                    state.inputs(theta[j0 + v], eps, x, den);
#pragma unroll
                    for (int i = 0; i < 3; ++i) own[i][v] = x[i];
                    own[3][v] = x[7];
                }
                shared[0] = state.x3;
                shared[1] = state.x4;
                shared[2] = state.x5;
                shared[3] = state.x6;
            }
            mlp_eval<V>(sw, [&](int i, int v) { return i < 3 ? own[i][v] : (i < 7 ? shared[i - 3] : own[3][v]); }, c);
            const double2 *dr = diag + r;
            asm volatile("" : "+l"(dr));
            const double d = __ldg(&dr->x);
#pragma unroll
            for (int v = 0; v < V; ++v) {
                const uint32_t j = j0 + v;
                const float cj = fminf(fmaxf(c[v], -clamp), clamp);
                double den = d - theta[j];
                if (fabs(den) < eps) den = den < 0.0 ? -eps : eps;
                const double2 rv = load_c(R, r64, j * n + r);
                if (cj == 0.f) {  // the Jacobi correction, rounded exactly as k_jacobi
                    store_c(T, t64, j * n + r, make_double2(-rv.x / den, -rv.y / den));
                } else {
                    const double g = -static_cast<double>(__expf(cj)) / den;  // |c| <= clamp
                    store_c(T, t64, j * n + r, make_double2(g * rv.x, g * rv.y));
                }
            }
        };
        uint32_t j0 = 0;
        for (; j0 + kEvalRows <= k; j0 += kEvalRows) correct(std::integral_constant<int, kEvalRows>{}, j0);
        for (; j0 < k; ++j0) correct(std::integral_constant<int, 1>{}, j0);
    }
}

// Training: per sample s the network sees inputs X[s] (TCP_MLP_IN floats) and
// predicts c; the correction is g = -exp(c) / den[s].  With a = |r|^2 and
// b = Re(conj(e) r) (e: the exact correction), the sample loss is
// wt[s] * (g^2 a - 2 g b + |e|^2).  A block takes kTrainChunk samples at a
// time: each thread runs one sample forward and back to the hidden layers and
// stages its activations, feature by feature, in shared memory.  Then warp w
// takes the units 4 w .. 4 w + 3 of every layer and lane l the samples 4 l ..
// 4 l + 3: a 16-byte load brings one feature of four samples, and the 109
// weight-gradient sums of the warp's units stay in each lane's registers
// across the chunks (12 multiply-adds per load: 177 us for 1.6 M samples; one
// thread per parameter pays two loads for each: 590 us).  The lanes are
// added by a fixed butterfly at the end, so the result is deterministic; each
// block writes its gradient partial sum.
constexpr int kTrainChunk = 128;
constexpr int kTrainStride = kTrainChunk + 4;
constexpr int kActX = 0, kActH1 = IN, kActH2 = kActH1 + HID, kActD1 = kActH2 + HID, kActD2 = kActD1 + HID,
              kActDc = kActD2 + HID, kActRows = kActDc + 1;
constexpr int kOwnUnits = HID / (kTrainChunk / 32);
static_assert(kOwnUnits == 4, "four warps cover the hidden units");

__device__ __forceinline__ float dot4(float4 a, float4 b, float acc) {
    return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}
__device__ __forceinline__ float sum4(float4 a, float acc) { return acc + ((a.x + a.y) + (a.z + a.w)); }
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

__global__ void __launch_bounds__(kTrainChunk)
    k_mlp_train(const float *__restrict__ X, int wide, const float *__restrict__ den, const float *__restrict__ a,
                const float *__restrict__ b, const float *__restrict__ e2, const float *__restrict__ wt,
                const float *__restrict__ dc_in, uint32_t count, const float *__restrict__ wglob,
                float *__restrict__ grad_partial, float *__restrict__ loss_partial) {
    __shared__ __align__(16) float w[NPARAM];
    __shared__ __align__(16) float act[kActRows][kTrainStride];
    __shared__ float lsum[kTrainChunk / 32];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, o0 = (tid >> 5) * kOwnUnits;
    for (int e = tid; e < NPARAM; e += kTrainChunk) w[e] = wglob[e];
    float g1[kOwnUnits][IN] = {}, g2[kOwnUnits][HID] = {}, gb1[kOwnUnits] = {}, gb2[kOwnUnits] = {}, g3[kOwnUnits] = {};
    float gb3 = 0.f, loss = 0.f;
    __syncthreads();
    const uint32_t chunks = (count + kTrainChunk - 1) / kTrainChunk;
    for (uint32_t ch = blockIdx.x; ch < chunks; ch += gridDim.x) {
        const uint32_t sidx = ch * kTrainChunk + tid;
        if (sidx < count) {
            // activations go to shared memory as soon as they are formed and
            // are read back from there: the sums above need the registers
            float h1[HID];
            {
                float x[IN];
                load_row8(X + static_cast<size_t>(sidx) * IN, wide, x);
#pragma unroll
                for (int i = 0; i < IN; ++i) act[kActX + i][tid] = x[i];
#pragma unroll
                for (int o = 0; o < HID; o += 4) {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        h1[o + k] = w[OFF_B1 + o + k];
#pragma unroll
                        for (int i = 0; i < IN; ++i) h1[o + k] = fmaf(w[OFF_W1 + (o + k) * IN + i], x[i], h1[o + k]);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k) h1[o + k] = act_tanh(h1[o + k]);
                }
            }
#pragma unroll
            for (int i = 0; i < HID; ++i) act[kActH1 + i][tid] = h1[i];
            float c = w[OFF_B3];
#pragma unroll 1
            for (int o = 0; o < HID; o += 4) {
                float h2[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    h2[k] = w[OFF_B2 + o + k];
#pragma unroll
                    for (int i = 0; i < HID; ++i) h2[k] = fmaf(w[OFF_W2 + (o + k) * HID + i], h1[i], h2[k]);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    h2[k] = act_tanh(h2[k]);
                    c = fmaf(w[OFF_W3 + o + k], h2[k], c);
                    act[kActH2 + o + k][tid] = h2[k];
                }
            }
            float dc;
            if (dc_in != nullptr) {  // caller-supplied dL/dc (any loss on the outputs)
                dc = dc_in[sidx];
            } else {
                const float g = -expf(c) / den[sidx];
                const float as = a[sidx], bs = b[sidx], ws = wt[sidx];
                loss += ws * (g * g * as - 2.f * g * bs + e2[sidx]);
                dc = ws * (2.f * g * as - 2.f * bs) * g;  // dL/dc
            }
            act[kActDc][tid] = dc;
            float d1[HID];
#pragma unroll
            for (int i = 0; i < HID; ++i) d1[i] = 0.f;
#pragma unroll 2
            for (int o = 0; o < HID; ++o) {
                const float h2 = act[kActH2 + o][tid];
                const float dh2 = dc * w[OFF_W3 + o] * (1.f - h2 * h2);
                act[kActD2 + o][tid] = dh2;
#pragma unroll
                for (int i = 0; i < HID; ++i) d1[i] = fmaf(dh2, w[OFF_W2 + o * HID + i], d1[i]);
            }
#pragma unroll
            for (int i = 0; i < HID; ++i) act[kActD1 + i][tid] = d1[i] * (1.f - h1[i] * h1[i]);
        } else {
            for (int i = 0; i < kActRows; ++i) act[i][tid] = 0.f;
        }
        __syncthreads();
        auto four = [&](int row) { return *reinterpret_cast<const float4 *>(&act[row][4 * lane]); };
        float4 u[kOwnUnits];
#pragma unroll
        for (int k = 0; k < kOwnUnits; ++k) {
            u[k] = four(kActD2 + o0 + k);
            gb2[k] = sum4(u[k], gb2[k]);
        }
#pragma unroll
        for (int i = 0; i < HID; ++i) {
            const float4 v = four(kActH1 + i);
#pragma unroll
            for (int k = 0; k < kOwnUnits; ++k) g2[k][i] = dot4(u[k], v, g2[k][i]);
        }
#pragma unroll
        for (int k = 0; k < kOwnUnits; ++k) {
            u[k] = four(kActD1 + o0 + k);
            gb1[k] = sum4(u[k], gb1[k]);
        }
#pragma unroll
        for (int i = 0; i < IN; ++i) {
            const float4 v = four(kActX + i);
#pragma unroll
            for (int k = 0; k < kOwnUnits; ++k) g1[k][i] = dot4(u[k], v, g1[k][i]);
        }
        const float4 dc4 = four(kActDc);
#pragma unroll
        for (int k = 0; k < kOwnUnits; ++k) g3[k] = dot4(four(kActH2 + o0 + k), dc4, g3[k]);
        gb3 = sum4(dc4, gb3);
        __syncthreads();
    }
    float *out = grad_partial + static_cast<size_t>(blockIdx.x) * NPARAM;
    auto write = [&](int pidx, float v) {
        const float total = warp_sum(v);
        if (lane == 0u) out[pidx] = total;
    };
#pragma unroll
    for (int k = 0; k < kOwnUnits; ++k) {
#pragma unroll
        for (int i = 0; i < IN; ++i) write(OFF_W1 + (o0 + k) * IN + i, g1[k][i]);
#pragma unroll
        for (int i = 0; i < HID; ++i) write(OFF_W2 + (o0 + k) * HID + i, g2[k][i]);
        write(OFF_B1 + o0 + k, gb1[k]);
        write(OFF_B2 + o0 + k, gb2[k]);
        write(OFF_W3 + o0 + k, g3[k]);
    }
    if (o0 == 0) write(OFF_B3, gb3);
    loss = warp_sum(loss);
    if (lane == 0u) lsum[tid >> 5] = loss;
    __syncthreads();
    if (tid == 0) loss_partial[blockIdx.x] = (lsum[0] + lsum[1]) + (lsum[2] + lsum[3]);
}

// Fixed-order sum of per-block losses (one warp).
__global__ void k_sum_losses(const float *__restrict__ partial, uint32_t blocks, float *__restrict__ out) {
    float l = 0.f;
    for (uint32_t b = threadIdx.x; b < blocks; b += 32u) l += partial[b];
    l = warp_sum(l);
    if (threadIdx.x == 0) *out = l;
}

// Network output c for every sample, kEvalRows per thread.
__global__ void __launch_bounds__(kEvalThreads, kEvalBlocks)
    k_mlp_forward(const float *__restrict__ X, int wide, uint32_t count, const float *__restrict__ wglob,
                  float *__restrict__ out) {
    constexpr int V = kEvalRows;
    __shared__ __align__(16) float sw[kEvalWords];
    mlp_stage(sw, wglob);
    __syncthreads();
    const uint64_t step = static_cast<uint64_t>(gridDim.x) * (V * kEvalThreads);
    for (uint64_t s0 = static_cast<uint64_t>(blockIdx.x) * (V * kEvalThreads) + threadIdx.x; s0 < count; s0 += step) {
        float x[V][IN], c[V];
#pragma unroll
        for (int v = 0; v < V; ++v) load_row8(X + umin64(s0 + v * kEvalThreads, count - 1u) * IN, wide, x[v]);
        mlp_eval<V>(sw, [&](int i, int v) { return x[v][i]; }, c);
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (s0 + v * kEvalThreads < count) out[s0 + v * kEvalThreads] = c[v];
    }
}

// Sum the per-block gradient partials (fixed order) and apply one Adam step.
// A block takes 32 parameters: warp w adds the partials w, w + 32, ... of each
// (coalesced), warp 0 adds the 32 sums in warp order and updates.
constexpr int kAdamWarps = 32;
__global__ void __launch_bounds__(kAdamWarps * 32)
    k_adam(float *__restrict__ w, float *__restrict__ m, float *__restrict__ v, const float *__restrict__ grad_partial,
           uint32_t blocks, float scale, float lr, float b1, float b2, float eps, uint32_t step,
           float *__restrict__ grad_out) {
    __shared__ float red[kAdamWarps][32];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const int e = static_cast<int>(blockIdx.x * 32u + lane);
    float gsum = 0.f;
    if (e < NPARAM) {
        for (uint32_t b = warp; b < blocks; b += kAdamWarps) gsum += grad_partial[static_cast<size_t>(b) * NPARAM + e];
    }
    red[warp][lane] = gsum;
    __syncthreads();
    if (warp != 0 || e >= NPARAM) return;
    for (int k = 1; k < kAdamWarps; ++k) gsum += red[k][lane];
    const float g = gsum * scale;
    if (grad_out) grad_out[e] = g;
    if (lr == 0.f) return;  // gradient only
    m[e] = b1 * m[e] + (1.f - b1) * g;
    v[e] = b2 * v[e] + (1.f - b2) * g * g;
    const float mh = m[e] / (1.f - powf(b1, static_cast<float>(step)));
    const float vh = v[e] / (1.f - powf(b2, static_cast<float>(step)));
    w[e] -= lr * mh / (sqrtf(vh) + eps);
}

// Network inputs and denominators for training samples taken from features.
__global__ void k_mlp_inputs(const float *__restrict__ feat, const uint64_t *__restrict__ rows, const double *__restrict__ theta,
                             const uint32_t *__restrict__ which, uint32_t count, double scale, double eps,
                             float *__restrict__ X, float *__restrict__ den) {
    for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < count; s += gridDim.x * blockDim.x) {
        float f[TCP_FEATURES], x[IN];
        double d;
        load_row8(feat + rows[s] * TCP_FEATURES, false, f);
        MlpState(f, scale).inputs(theta[which[s]], eps, x, d);
#pragma unroll
        for (int i = 0; i < IN; ++i) X[static_cast<size_t>(s) * IN + i] = x[i];
        den[s] = static_cast<float>(d);
    }
}

// ---------------------- alignment objective of the training ---------------------
// A training set s covers the states [seg_begin[s], seg_begin[s + 1]).  With
// g = -exp(clamp(c)) / den per state its sums are A = sum g alpha, B = sum g^2 a,
// C = sum g gamma, D = max(B - |C|^2, 1e-300), and its loss is
// 1 - |A|^2 / (E_s D): one minus the squared cosine between the correction
// g o r, made orthogonal to the Ritz vector, and the missing direction.  The
// objective is the mean over the sets.
constexpr int kAlignThreads = 512;
constexpr int kAlignWords = 6;  // A (2), B, C (2), loss per set

__device__ __forceinline__ double align_g(float c, float den, float clamp) {
    const double cc = fmin(fmax(static_cast<double>(c), -static_cast<double>(clamp)), static_cast<double>(clamp));
    return -exp(cc) / static_cast<double>(den);
}

// The sums of set s: N blocks of THREADS threads take its states in turn, and the
// first adds their five sums through distributed shared memory in rank order (a
// fixed-order tree inside each block), so the sums do not depend on scheduling.
template <int N, int THREADS>
__device__ __forceinline__ void align_sums(uint32_t s, uint32_t rank, const float *__restrict__ c,
                                           const float *__restrict__ den, const double2 *__restrict__ alpha,
                                           const double *__restrict__ a, const double2 *__restrict__ gamma,
                                           const double *__restrict__ E, const uint64_t *__restrict__ seg_begin,
                                           float clamp, double *__restrict__ sums) {
    namespace cg = cooperative_groups;
    __shared__ double red[5][THREADS / 32];
    __shared__ double mine[5];
    const uint32_t t = threadIdx.x;
    double v[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    for (uint64_t i = seg_begin[s] + rank * THREADS + t; i < seg_begin[s + 1]; i += N * THREADS) {
        const double g = align_g(c[i], den[i], clamp);
        const double2 al = alpha[i], ga = gamma[i];
        v[0] += g * al.x;
        v[1] += g * al.y;
        v[2] += g * g * a[i];
        v[3] += g * ga.x;
        v[4] += g * ga.y;
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], off);
        if ((t & 31u) == 0u) red[k][t >> 5] = v[k];
    }
    __syncthreads();
    if (t < 5) {
        double sum = 0.0;
        for (int q = 0; q < THREADS / 32; ++q) sum += red[t][q];
        mine[t] = sum;
    }
    if constexpr (N > 1) {
        const cg::cluster_group cluster = cg::this_cluster();
        cluster.sync();
        double sum = 0.0;
        if (rank == 0 && t < 5) {
            for (int q = 0; q < N; ++q) sum += cluster.map_shared_rank(mine, q)[t];
        }
        cluster.sync();  // no block leaves, or overwrites its sums, while they are being read
        if (rank == 0 && t < 5) mine[t] = sum;
    }
    __syncthreads();
    if (rank == 0 && t == 0) {
        double *q = sums + static_cast<size_t>(s) * kAlignWords;
#pragma unroll
        for (int k = 0; k < 5; ++k) q[k] = mine[k];
        const double D = fmax(mine[2] - (mine[3] * mine[3] + mine[4] * mine[4]), 1e-300);
        const double A2 = mine[0] * mine[0] + mine[1] * mine[1];
        q[5] = 1.0 - A2 / (E[s] * D);
    }
}

// One block per set, or a cluster of eight.  A cluster takes 0.08 us to launch and
// meet, whatever its set; a block walks its set at 3.8 us per 1000 states.  So
// clusters serve few and large sets, more than kAlignLarge states on average for
// each set there is: 24 sets of 65,536 states 20 us (blocks 247), 150 of them 108
// (281), 64 of 4,096 7.9 (9.7), but 400 of 16,384 95 (80), 300 of 4,096 33 (14), 128
// of 512 13.6 (3.1), 1000 of 256 82 (5.4).
constexpr int kAlignCluster = 8, kAlignBlockThreads = 256;
constexpr uint64_t kAlignLarge = 48;
__global__ void __launch_bounds__(kAlignBlockThreads)
    k_align_sums(const float *__restrict__ c, const float *__restrict__ den, const double2 *__restrict__ alpha,
                 const double *__restrict__ a, const double2 *__restrict__ gamma, const double *__restrict__ E,
                 const uint64_t *__restrict__ seg_begin, float clamp, double *__restrict__ sums) {
    align_sums<1, kAlignBlockThreads>(blockIdx.x, 0u, c, den, alpha, a, gamma, E, seg_begin, clamp, sums);
}
__global__ void __launch_bounds__(kAlignThreads) __cluster_dims__(kAlignCluster, 1, 1)
    k_align_sums_large(const float *__restrict__ c, const float *__restrict__ den, const double2 *__restrict__ alpha,
                       const double *__restrict__ a, const double2 *__restrict__ gamma, const double *__restrict__ E,
                       const uint64_t *__restrict__ seg_begin, float clamp, double *__restrict__ sums) {
    align_sums<kAlignCluster, kAlignThreads>(blockIdx.x / kAlignCluster, blockIdx.x % kAlignCluster, c, den, alpha, a,
                                             gamma, E, seg_begin, clamp, sums);
}

// dL/dc per state (zero where the clamp is active).
__global__ void k_align_dc(const float *__restrict__ c, const float *__restrict__ den, const double2 *__restrict__ alpha,
                           const double *__restrict__ a, const double2 *__restrict__ gamma, const double *__restrict__ E,
                           const int64_t *__restrict__ seg, uint64_t count, uint32_t nsets, float clamp,
                           const double *__restrict__ sums, float *__restrict__ dc) {
    for (uint64_t i = blockIdx.x * static_cast<uint64_t>(blockDim.x) + threadIdx.x; i < count;
         i += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
        const int64_t s = seg[i];
        const double *q = sums + static_cast<size_t>(s) * kAlignWords;
        const double D = fmax(q[2] - (q[3] * q[3] + q[4] * q[4]), 1e-300);
        const double A2 = q[0] * q[0] + q[1] * q[1];
        const double g = align_g(c[i], den[i], clamp);
        const double2 al = alpha[i], ga = gamma[i];
        const double dA2 = 2.0 * (q[0] * al.x + q[1] * al.y);
        const double dD = 2.0 * g * a[i] - 2.0 * (q[3] * ga.x + q[4] * ga.y);
        const double dLdg = -(dA2 * D - A2 * dD) / (E[s] * D * D) / static_cast<double>(nsets);
        const float ci = c[i];
        dc[i] = (ci > -clamp && ci < clamp) ? static_cast<float>(dLdg * g) : 0.f;
    }
}

// Mean of the per-set losses, summed in set order.
__global__ void k_align_loss(const double *__restrict__ sums, uint32_t nsets, double *__restrict__ loss) {
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        double l = 0.0;
        for (uint32_t s = 0; s < nsets; ++s) l += sums[static_cast<size_t>(s) * kAlignWords + 5];
        *loss = l / static_cast<double>(nsets);
    }
}

int grid_for(uint64_t n, int threads) {
    return static_cast<int>(std::min<uint64_t>((n + threads - 1) / threads, 148ull * 16));
}

// Rows of 8 floats that 16-byte loads can address.
int rows_wide(const float *rows) { return reinterpret_cast<uintptr_t>(rows) % 16 == 0; }

bool valid_dtype(int d) { return d == TCP_DTYPE_C128 || d == TCP_DTYPE_C64; }

template <int QJ>
void launch_gram_tiles(int grid, size_t smem, cudaStream_t s, const void *A, bool a64, uint32_t p, const void *B,
                       bool b64, uint32_t q, uint64_t n, uint32_t groups, bool pairs_of_rows, double2 *partial) {
#define TCP_GRAM_LAUNCH(A64, B64, RPL)                                                                            \
    do {                                                                                                        \
        cudaFuncSetAttribute(k_gram_tiles<QJ, A64, B64, RPL>, cudaFuncAttributeMaxDynamicSharedMemorySize,       \
                             kGramRedBytes);                                                                    \
        k_gram_tiles<QJ, A64, B64, RPL><<<grid, kGramThreads, smem, s>>>(A, p, B, q, n, groups, partial);       \
    } while (0)
    if (a64 && b64 && pairs_of_rows) {
        TCP_GRAM_LAUNCH(true, true, 2);
    } else if (a64 && b64) {
        TCP_GRAM_LAUNCH(true, true, 1);
    } else if (a64) {
        TCP_GRAM_LAUNCH(true, false, 1);
    } else if (b64) {
        TCP_GRAM_LAUNCH(false, true, 1);
    } else {
        TCP_GRAM_LAUNCH(false, false, 1);
    }
#undef TCP_GRAM_LAUNCH
}

// cuTensorMapEncodeTiled from the driver, looked up once.
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static PFN_cuTensorMapEncodeTiled_v12000 fn = [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &qres) != cudaSuccess ||
            qres != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return static_cast<PFN_cuTensorMapEncodeTiled_v12000>(nullptr);
        }
        return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
    }();
    return fn;
}

// Tensor map of `vecs` vectors of length n (element size es) seen as a 2-D
// array of 8-byte units; box = `rows` rows of every vector.
bool vector_block_map(CUtensorMap *map, const void *base, uint32_t vecs, uint64_t n, size_t es, uint32_t rows) {
    PFN_cuTensorMapEncodeTiled_v12000 encode = tensor_map_encoder();
    if (!encode) return false;
    const cuuint64_t dims[2] = {n * (es / 8), vecs};
    const cuuint64_t strides[1] = {n * es};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(rows * (es / 8)), vecs};
    const cuuint32_t elem_strides[2] = {1, 1};
    return encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, const_cast<void *>(base), dims, strides, box, elem_strides,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The TMA-fed Gram for two complex128 blocks: 16-byte aligned vectors, at
// most 16 warp tiles, n * 8-byte units below 2^31.  Returns false (nothing
// launched) when those conditions do not hold.  Complex64 blocks take the
// register-fed kernel, which measured faster for them (3.1 against 2.6 TB/s
// at n = 2^24 with 64 + 4 vectors; both are bound by FP64 work, 16 FMAs and
// 2 conversions per 8-byte value), while complex128 gains 5.2 -> 5.7 TB/s.
// (The kernel template also reads complex64 blocks with n even.)
bool launch_gram_tma(const void *A, bool a64, uint32_t p, const void *B, bool b64, uint32_t q, uint64_t n,
                     uint32_t qj, uint32_t ntiles, cudaStream_t s, double2 *partial, uint32_t *grid_used) {
    if (a64 || b64 || ntiles > static_cast<uint32_t>(kGramWarps)) return false;
    const size_t es = a64 ? sizeof(float2) : sizeof(double2);
    if ((n * es) % 16 != 0 || n * (es / 8) >= (1ull << 31) || reinterpret_cast<uintptr_t>(A) % 16 != 0 ||
        reinterpret_cast<uintptr_t>(B) % 16 != 0)
        return false;
    const uint32_t vecs = p + q;
    // rows per chunk: a multiple of 32, one stage <= kGramStageBytes, a box
    // edge <= 256 units
    uint32_t rows = static_cast<uint32_t>(kGramStageBytes / (vecs * es)) / 32u * 32u;
    rows = std::min<uint32_t>(rows, static_cast<uint32_t>(256 / (es / 8)));
    if (rows < 32) return false;
    CUtensorMap ta, tb;
    if (!vector_block_map(&ta, A, p, n, es, rows) || !vector_block_map(&tb, B, q, n, es, rows)) return false;
    const uint32_t groups = std::max<uint32_t>(1u, std::min<uint32_t>(kGramWarps / ntiles, rows / 32u));
    const uint64_t chunks = n / rows;
    const int grid = static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>(kGramGrid, chunks)));
    const size_t smem = static_cast<size_t>(kGramStages) * vecs * rows * es;
#define TCP_GRAM_TMA(QJ, C64)                                                                                   \
    do {                                                                                                      \
        cudaFuncSetAttribute(k_gram_tma<QJ, C64>, cudaFuncAttributeMaxDynamicSharedMemorySize,                 \
                             static_cast<int>(kGramStages * kGramStageBytes));                                \
        k_gram_tma<QJ, C64><<<grid, kGramThreads, smem, s>>>(ta, tb, A, p, B, q, n, rows, groups, partial);   \
    } while (0)
    if (qj == 1) {
        TCP_GRAM_TMA(1, false);
    } else if (qj == 2) {
        TCP_GRAM_TMA(2, false);
    } else {
        TCP_GRAM_TMA(4, false);
    }
#undef TCP_GRAM_TMA
    *grid_used = static_cast<uint32_t>(grid);
    return true;
}

}  // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
extern "C" size_t tcp_gram_work_bytes(uint32_t p, uint32_t q) {
    return static_cast<size_t>(kGramBlocks) * p * q * sizeof(double2);
}

extern "C" int tcp_gram(const void *A, int a_dtype, uint32_t p, const void *B, int b_dtype, uint32_t q, uint64_t n,
                        void *d_G, void *d_work, void *stream) {
    if (!valid_dtype(a_dtype) || !valid_dtype(b_dtype)) return fail(TCP_ERR_INVALID_ARGUMENT, "unknown dtype");
    if (p == 0 || q == 0) return TCP_OK;
    if (p + q > kGramMaxVectors || p * q > kGramMaxPairs) {
        return fail(TCP_ERR_INVALID_ARGUMENT, "tcp_gram supports p + q <= 96 and p * q <= 512");
    }
    if (!A || !B || !d_G || !d_work) return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    auto *partial = static_cast<double2 *>(d_work);
    const uint32_t qj = q == 1 ? 1u : (q == 2 ? 2u : 4u);
    const uint32_t pi = qj == 4 ? 4u : 8u;  // tile shape of k_gram_tiles<qj>
    const uint32_t ntiles = ((p + pi - 1) / pi) * ((q + qj - 1) / qj);
    const bool a64 = a_dtype == TCP_DTYPE_C64, b64 = b_dtype == TCP_DTYPE_C64;
    uint32_t grid_used = 0;
    if (launch_gram_tma(A, a64, p, B, b64, q, n, qj, ntiles, s, partial, &grid_used)) {
        const uint32_t pairs = p * q;
        k_gram_reduce<<<(pairs + 31) / 32, kGramReduceWarps * 32, 0, s>>>(partial, grid_used, pairs, static_cast<double2 *>(d_G));
        cudaError_t e = cudaGetLastError();
        return e == cudaSuccess ? TCP_OK : cuda_fail(e, "gram kernel launch");
    }
    // Register-fed tiles (mixed storage types, odd complex64 lengths, more
    // than 16 tiles).  Row groups per CTA: slots = ntiles * groups =
    // lcm(ntiles, 16) keeps all 16 warps equally busy; if those partial sums
    // do not fit in shared memory, fall back to 16 / ntiles groups (or one).
    const uint32_t tp = pi * qj;
    uint32_t groups = kGramWarps / std::gcd(ntiles, static_cast<uint32_t>(kGramWarps));
    if (static_cast<size_t>(groups) * ntiles * tp * sizeof(double2) > static_cast<size_t>(kGramRedBytes))
        groups = ntiles >= static_cast<uint32_t>(kGramWarps) ? 1u : kGramWarps / ntiles;
    const size_t smem = groups > 1 ? static_cast<size_t>(groups) * ntiles * tp * sizeof(double2) : 0;
    const bool pairs_of_rows = a64 && b64 && n % 2 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 &&
                               reinterpret_cast<uintptr_t>(B) % 16 == 0;
    const uint64_t rows_per_chunk = pairs_of_rows ? 64 : 32;
    const uint64_t chunks = (n + rows_per_chunk - 1) / rows_per_chunk;
    const int grid = static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>(kGramGrid, (chunks + groups - 1) / groups)));
    if (qj == 1) {
        launch_gram_tiles<1>(grid, smem, s, A, a64, p, B, b64, q, n, groups, pairs_of_rows, partial);
    } else if (qj == 2) {
        launch_gram_tiles<2>(grid, smem, s, A, a64, p, B, b64, q, n, groups, pairs_of_rows, partial);
    } else {
        launch_gram_tiles<4>(grid, smem, s, A, a64, p, B, b64, q, n, groups, pairs_of_rows, partial);
    }
    const uint32_t pairs = p * q;
    k_gram_reduce<<<(pairs + 31) / 32, kGramReduceWarps * 32, 0, s>>>(partial, static_cast<uint32_t>(grid), pairs,
                                                      static_cast<double2 *>(d_G));
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "gram kernel launch");
}

extern "C" int tcp_block_combine(const void *A, int a_dtype, uint32_t p, const void *d_S, uint32_t k, uint64_t n,
                                 double alpha, double beta, void *out, int out_dtype, void *stream) {
    if (!valid_dtype(a_dtype) || !valid_dtype(out_dtype)) return fail(TCP_ERR_INVALID_ARGUMENT, "unknown dtype");
    if (k == 0) return TCP_OK;
    if (k > static_cast<uint32_t>(kCombineMaxK)) return fail(TCP_ERR_INVALID_ARGUMENT, "tcp_block_combine supports k <= 32");
    uint32_t njp = 1;
    while (njp * kCombineTile < k) njp <<= 1;
    const size_t smem = static_cast<size_t>(p) * njp * kCombineTile * sizeof(double2);
    if (smem > 96 * 1024) return fail(TCP_ERR_INVALID_ARGUMENT, "coefficient block too large");
    if (!A || !d_S || !out) return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    if (n == 0) return TCP_OK;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const uint32_t rb = kCombineThreads / njp;
    const int grid = static_cast<int>(std::min<uint64_t>((n + rb - 1) / rb, 148ull * 8));
    const bool a64 = a_dtype == TCP_DTYPE_C64, o64 = out_dtype == TCP_DTYPE_C64;
    const auto *S = static_cast<const double2 *>(d_S);
    const bool aligned = reinterpret_cast<uintptr_t>(A) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
    const uint64_t pair_blocks = (n / 2 + rb - 1) / rb;
    if (a64 && o64 && n % 2 == 0 && aligned && combine_by_pairs(k, njp, pair_blocks)) {
        const int pgrid = static_cast<int>(std::min<uint64_t>(pair_blocks, 148ull * 4 * kCombinePairBlocks));
        cudaFuncSetAttribute(k_combine_pairs, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        k_combine_pairs<<<pgrid, kCombineThreads, smem, s>>>(static_cast<const float4 *>(A), p, S, k, njp, n / 2, alpha, beta,
                                                            static_cast<float4 *>(out));
    } else if (a64 && o64) {
        cudaFuncSetAttribute(k_combine_tiles<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        k_combine_tiles<true, true><<<grid, kCombineThreads, smem, s>>>(A, p, S, k, njp, n, alpha, beta, out);
    } else if (a64) {
        cudaFuncSetAttribute(k_combine_tiles<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        k_combine_tiles<true, false><<<grid, kCombineThreads, smem, s>>>(A, p, S, k, njp, n, alpha, beta, out);
    } else if (o64) {
        cudaFuncSetAttribute(k_combine_tiles<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        k_combine_tiles<false, true><<<grid, kCombineThreads, smem, s>>>(A, p, S, k, njp, n, alpha, beta, out);
    } else {
        cudaFuncSetAttribute(k_combine_tiles<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, 96 * 1024);
        k_combine_tiles<false, false><<<grid, kCombineThreads, smem, s>>>(A, p, S, k, njp, n, alpha, beta, out);
    }
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "combine kernel launch");
}

extern "C" int tcp_precond_jacobi(const void *R, int r_dtype, uint64_t n, uint32_t k, const void *d_diag,
                                  const double *d_theta, double eps, void *T, int t_dtype, void *stream) {
    if (!valid_dtype(r_dtype) || !valid_dtype(t_dtype)) return fail(TCP_ERR_INVALID_ARGUMENT, "unknown dtype");
    if (!R || !d_diag || !d_theta || !T) return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    k_jacobi<<<grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        R, r_dtype == TCP_DTYPE_C64, n, k, static_cast<const double2 *>(d_diag), d_theta, eps, T, t_dtype == TCP_DTYPE_C64);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "jacobi kernel launch");
}

extern "C" int tcp_state_features(const tcp_mvp_plan *plan, float *d_features, uint64_t n, void *stream) {
    int st = tcp::check_plan(plan);
    if (st) return st;
    if (n != plan->dim) return tcp::length_error(plan->dim, n);
    if (!d_features) return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    const tcp::Schedule &h = plan->sched.host;
    uint32_t gzero = 0xffffffffu;
    for (size_t g = 0; g < h.g_mask.size(); ++g)
        if (h.g_mask[g] == 0) gzero = static_cast<uint32_t>(g);
    k_features<<<grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(plan->sched.dev, gzero, plan->nqubits, n,
                                                                              d_features);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "feature kernel launch");
}

extern "C" int tcp_precond_mlp(const void *R, int r_dtype, uint64_t n, uint32_t k, const float *d_features,
                               const void *d_diag, const double *d_theta, double scale, double eps, float clamp,
                               const float *d_params, void *T, int t_dtype, void *stream) {
    if (!valid_dtype(r_dtype) || !valid_dtype(t_dtype)) return fail(TCP_ERR_INVALID_ARGUMENT, "unknown dtype");
    if (!R || !d_features || !d_diag || !d_theta || !d_params || !T) return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    k_mlp_precond<<<grid_for(n, kEvalThreads), kEvalThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        R, r_dtype == TCP_DTYPE_C64, n, k, d_features, rows_wide(d_features), static_cast<const double2 *>(d_diag), d_theta, scale, eps, clamp,
        d_params, T, t_dtype == TCP_DTYPE_C64);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "mlp preconditioner launch");
}

extern "C" int tcp_mlp_inputs(const float *d_features, const uint64_t *d_rows, const double *d_theta,
                              const uint32_t *d_which, uint32_t count, double scale, double eps, float *d_X,
                              float *d_den, void *stream) {
    if (!d_features || !d_rows || !d_theta || !d_which || !d_X || !d_den) return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    if (count == 0) return TCP_OK;
    k_mlp_inputs<<<grid_for(count, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(d_features, d_rows, d_theta, d_which,
                                                                                   count, scale, eps, d_X, d_den);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "mlp input kernel launch");
}

extern "C" int tcp_mlp_forward(const float *d_X, uint32_t count, const float *d_params, float *d_out, void *stream) {
    if (!d_X || !d_params || !d_out) return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    if (count == 0) return TCP_OK;
    k_mlp_forward<<<grid_for(count, kEvalRows * kEvalThreads), kEvalThreads, 0, static_cast<cudaStream_t>(stream)>>>(d_X, rows_wide(d_X), count, d_params, d_out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "mlp forward launch");
}

extern "C" int tcp_mlp_backward_step(const float *d_X, const float *d_dc, uint32_t count, float *d_params, float *d_m,
                                     float *d_v, float *d_work, float lr, uint32_t step, float *d_grad_out,
                                     void *stream) {
    if (!d_X || !d_dc || !d_params || !d_work) return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    if (lr != 0.f && (!d_m || !d_v || step == 0)) return fail(TCP_ERR_INVALID_ARGUMENT, "Adam state missing");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float *grad_partial = d_work;
    float *loss_partial = d_work + static_cast<size_t>(TCP_MLP_TRAIN_BLOCKS) * TCP_MLP_PARAMS;
    k_mlp_train<<<TCP_MLP_TRAIN_BLOCKS, kTrainChunk, 0, s>>>(d_X, rows_wide(d_X), nullptr, nullptr, nullptr, nullptr, nullptr, d_dc,
                                                             count, d_params, grad_partial, loss_partial);
    k_adam<<<(TCP_MLP_PARAMS + 31) / 32, kAdamWarps * 32, 0, s>>>(d_params, d_m, d_v, grad_partial, TCP_MLP_TRAIN_BLOCKS, 1.f, lr,
                                                       0.9f, 0.999f, 1e-8f, step, d_grad_out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "mlp backward launch");
}

extern "C" size_t tcp_mlp_train_work_bytes(void) {
    return static_cast<size_t>(TCP_MLP_TRAIN_BLOCKS) * (TCP_MLP_PARAMS + 1) * sizeof(float);
}

extern "C" int tcp_mlp_train_step(const float *d_X, const float *d_den, const float *d_a, const float *d_b,
                                  const float *d_e2, const float *d_wt, uint32_t count, float *d_params, float *d_m,
                                  float *d_v, float *d_work, float lr, uint32_t step, float *d_grad_out,
                                  float *d_loss_out, void *stream) {
    if (!d_X || !d_den || !d_a || !d_b || !d_e2 || !d_wt || !d_params || !d_work) {
        return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    }
    if (lr != 0.f && (!d_m || !d_v || step == 0)) return fail(TCP_ERR_INVALID_ARGUMENT, "Adam state missing");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    float *grad_partial = d_work;
    float *loss_partial = d_work + static_cast<size_t>(TCP_MLP_TRAIN_BLOCKS) * TCP_MLP_PARAMS;
    k_mlp_train<<<TCP_MLP_TRAIN_BLOCKS, kTrainChunk, 0, s>>>(d_X, rows_wide(d_X), d_den, d_a, d_b, d_e2, d_wt, nullptr, count,
                                                             d_params, grad_partial, loss_partial);
    k_adam<<<(TCP_MLP_PARAMS + 31) / 32, kAdamWarps * 32, 0, s>>>(d_params, d_m, d_v, grad_partial, TCP_MLP_TRAIN_BLOCKS, 1.f, lr,
                                                       0.9f, 0.999f, 1e-8f, step, d_grad_out);
    if (d_loss_out) k_sum_losses<<<1, 32, 0, s>>>(loss_partial, TCP_MLP_TRAIN_BLOCKS, d_loss_out);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "mlp training launch");
}

extern "C" size_t tcp_mlp_alignment_work_bytes(uint32_t nsets) {
    return static_cast<size_t>(nsets) * kAlignWords * sizeof(double);
}

extern "C" int tcp_mlp_alignment_grad(const float *d_c, const float *d_den, const void *d_alpha, const double *d_a,
                                      const void *d_gamma, const double *d_E, const int64_t *d_seg,
                                      const uint64_t *d_seg_begin, uint32_t nsets, uint64_t count, float clamp,
                                      double *d_work, float *d_dc, double *d_loss, void *stream) {
    if (!d_c || !d_den || !d_alpha || !d_a || !d_gamma || !d_E || !d_seg || !d_seg_begin || !d_work || !d_dc) {
        return fail(TCP_ERR_INVALID_ARGUMENT, "null buffer");
    }
    if (nsets == 0) return fail(TCP_ERR_INVALID_ARGUMENT, "the alignment objective needs at least one set");
    if (!(clamp > 0.f)) return fail(TCP_ERR_INVALID_ARGUMENT, "clamp must be positive");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const auto *alpha = static_cast<const double2 *>(d_alpha), *gamma = static_cast<const double2 *>(d_gamma);
    if (count / nsets > kAlignLarge * nsets)
        k_align_sums_large<<<nsets * kAlignCluster, kAlignThreads, 0, s>>>(d_c, d_den, alpha, d_a, gamma, d_E,
                                                                          d_seg_begin, clamp, d_work);
    else
        k_align_sums<<<nsets, kAlignBlockThreads, 0, s>>>(d_c, d_den, alpha, d_a, gamma, d_E, d_seg_begin, clamp, d_work);
    if (count > 0) {
        k_align_dc<<<grid_for(count, 256), 256, 0, s>>>(d_c, d_den, alpha, d_a, gamma, d_E, d_seg, count, nsets, clamp,
                                                        d_work, d_dc);
    }
    if (d_loss) k_align_loss<<<1, 32, 0, s>>>(d_work, nsets, d_loss);
    cudaError_t e = cudaGetLastError();
    return e == cudaSuccess ? TCP_OK : cuda_fail(e, "alignment gradient launch");
}
