// Device building blocks of the ring kernel (k_ring in tcp_mvp.cu): ring
// geometry, the sums of a thread's rows, and the walk of a step's records.  The
// block layout is tcp::RingSchedule's.
#pragma once

#include "tcp_device.cuh"

namespace tcpdev {

// Geometry of one ring kernel: SHAPE indexes tcp::kRingShapes.
// Who refills the ring.  complex128: a dedicated producer warp waits on the
// stages' "empty" barriers and issues the fills (2,000 random words on 28 qubits:
// 168 ms against 191 without it; 20-qubit chain: 31 us against 37, in launches one
// after another).  complex64: no extra warp -- the row
// warp that releases a stage last issues its refill -- so the 512 threads keep
// 128 registers for the paired FP32 accumulators.
template <typename R, int SHAPE> struct RingGeo {
    static constexpr tcp::RingShapeBits kBits = tcp::kRingShapes[SHAPE];
    static constexpr uint32_t kTileBits = kBits.tile_bits;
    static constexpr uint32_t kLogT = kBits.log_threads;
    static constexpr uint32_t kLow = kBits.low;
    static constexpr int kRows = 1 << (kTileBits - kLogT);  // rows of a thread
    static constexpr uint32_t kWarps = (1u << kLogT) / 32u;  // warps that own rows
    static constexpr bool kProducerWarp = sizeof(R) == 8;
    // complex64, 16 rows: the compensated sums live in tensor memory
    static constexpr bool kTmem = sizeof(R) == 4 && kRows == 16;
    static constexpr uint32_t kTmemColumns = 256;  // 4 warps per lane quarter x 16 rows x 4 words
    static constexpr int kThreads = (1 << kLogT) + (kProducerWarp ? 32 : 0);
    static constexpr uint32_t kTileBytes = (1u << kTileBits) * 2u * static_cast<uint32_t>(sizeof(R));
    static constexpr uint32_t kStageBytes = kTileBytes + tcp::kRingBlockBytes;
    static constexpr uint32_t kDepth = kTileBytes > 32768u ? 3u : 4u;  // ring stages: 3 x 72 or 4 x 40 KiB
    static constexpr size_t kSmemBytes = size_t(kDepth) * kStageBytes;
    // tile row of register row j of thread 0
    static constexpr uint32_t row(uint32_t j) {
        return (j & ((1u << kLow) - 1u)) | ((j >> kLow) << (kLow + kLogT));
    }
};

template <typename R> __device__ __forceinline__ const unsigned char *ring_blocks(const RingView &s);
template <> __device__ __forceinline__ const unsigned char *ring_blocks<double>(const RingView &s) {
    return s.blocks128;
}
template <> __device__ __forceinline__ const unsigned char *ring_blocks<float>(const RingView &s) {
    return s.blocks64;
}

// (-1)^parity(zs & c) as a sign bit in bit 31.
__device__ __forceinline__ uint32_t ring_sign(uint32_t zs, uint32_t c) {
    return static_cast<uint32_t>(__popc(zs & c)) << 31;
}
__device__ __forceinline__ double xor_sign(double w, uint32_t sign) {
    return __hiloint2double(__double2hiint(w) ^ static_cast<int>(sign), __double2loint(w));
}
__device__ __forceinline__ float xor_sign(float w, uint32_t sign) {
    return __int_as_float(__float_as_int(w) ^ static_cast<int>(sign));
}
// Bit k of a table index, scaled to the weight's size (log2 LOGB bytes).
template <int K, int LOGB> __device__ __forceinline__ uint32_t ring_index(uint32_t v, uint32_t c) {
    return (static_cast<uint32_t>(__popc(v & c)) << (K + LOGB)) & (1u << (K + LOGB));
}

// Weight of a single's record: one f64 (bytes 8..15) or one f32 (bytes 8..11).
template <typename R> __device__ __forceinline__ R ring_weight(uint4 rec);
template <> __device__ __forceinline__ double ring_weight<double>(uint4 rec) {
    return __hiloint2double(static_cast<int>(rec.w), static_cast<int>(rec.z));
}
template <> __device__ __forceinline__ float ring_weight<float>(uint4 rec) { return __uint_as_float(rec.z); }

// Table entry of a table record at `p` (its first 16 bytes in `rec`) for the
// row word c; `p` moves past the record.
template <typename R>
__device__ __forceinline__ R ring_table(const unsigned char *&p, uint4 rec, uint32_t c) {
    constexpr int LOGB = sizeof(R) == 8 ? 3 : 2;
    const uint32_t kind = (rec.y & tcp::kRingKindMask) >> tcp::kRingKindShift;
    uint32_t at = ring_index<0, LOGB>(rec.z, c) | ring_index<1, LOGB>(rec.w, c);
    p += 16;
    if (kind > 1u) {
        const uint2 more = *reinterpret_cast<const uint2 *>(p);
        at |= ring_index<2, LOGB>(more.x, c) | ring_index<3, LOGB>(more.y, c);
        p += 16;
    }
    const R v = *reinterpret_cast<const R *>(p + at);
    p += sizeof(R) << (kind + 1u);
    return v;
}

// Negate the loaded values of the rows that have bit B set.
template <int B, int E, typename C> __device__ __forceinline__ void ring_flip_rows(C (&xv)[E]) {
#pragma unroll
    for (int j = 0; j < E; ++j) {
        if ((j >> B) & 1) {
            xv[j].x = xor_sign(xv[j].x, 0x80000000u);
            xv[j].y = xor_sign(xv[j].y, 0x80000000u);
        }
    }
}

// One run applied to the thread's rows: row j takes source value j ^ A times D.
template <int A, int E, typename R>
__device__ __forceinline__ void ring_apply(R d, uint32_t word, const typename Cx<R>::T (&xv)[E], RingAcc<R> (&acc)[E]) {
    if (!(word & tcp::kRingImag)) {
#pragma unroll
        for (int j = 0; j < E; ++j) acc[j].add_real(d, xv[j ^ A]);
    } else {
#pragma unroll
        for (int j = 0; j < E; ++j) acc[j].add_imag(d, xv[j ^ A]);
    }
}

template <int E, typename R>
__device__ __forceinline__ void ring_dispatch(R d, uint32_t word, const typename Cx<R>::T (&xv)[E], RingAcc<R> (&acc)[E]) {
    // Most runs have a = 0 (a group rarely flips one of the few register bits):
    // one test ahead of the switch, which for complex64 takes real weights along
    // (26 qubits 23.7 ms, 24.0 without it; J1-J2 block 3.57 and 3.71 ms).  complex128
    // takes the same time with and without it (28 qubits: 168 ms).
    constexpr uint32_t kCommon = static_cast<uint32_t>(E - 1) | (sizeof(R) == 4 ? tcp::kRingImag : 0u);
    if ((word & kCommon) == 0u) {
        ring_apply<0, E, R>(d, sizeof(R) == 4 ? 0u : word, xv, acc);
        return;
    }
#define TCP_RING_CASE(A) \
    case A: if constexpr (A < E) ring_apply<A % E, E, R>(d, word, xv, acc); break;
    switch (word & static_cast<uint32_t>(E - 1)) {
        TCP_RING_CASE(0) TCP_RING_CASE(1) TCP_RING_CASE(2) TCP_RING_CASE(3)
        TCP_RING_CASE(4) TCP_RING_CASE(5) TCP_RING_CASE(6) TCP_RING_CASE(7)
        TCP_RING_CASE(8) TCP_RING_CASE(9) TCP_RING_CASE(10) TCP_RING_CASE(11)
        TCP_RING_CASE(12) TCP_RING_CASE(13) TCP_RING_CASE(14) TCP_RING_CASE(15)
    }
#undef TCP_RING_CASE
}

// The thread's accumulators and, complex64, its compensated sums.
template <typename R, int SHAPE> struct RingSums {
    static constexpr int E = RingGeo<R, SHAPE>::kRows;
    RingAcc<R> acc[E];
    __device__ __forceinline__ void fold() {}
    __device__ __forceinline__ double2 value(int j) const { return acc[j].value(); }
};
// 8 rows: in registers.
template <> struct RingSums<float, 0> {
    static constexpr int E = RingGeo<float, 0>::kRows;
    RingAcc<float> acc[E];
    uint64_t s[E] = {}, c[E] = {};
    // The barrier keeps the fold a branch of its own, apart from the common run's
    // code (3,000 random words on 16 qubits: 293 us, 300 without it).
    __device__ __forceinline__ void fold() {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < E; ++j) acc[j].fold(s[j], c[j]);
    }
    __device__ __forceinline__ float2 value(int j) const { return RingAcc<float>::value(s[j], c[j]); }
};
// 16 rows: (s, c) of rows 4 k .. 4 k + 3 in 16 tensor-memory columns of the
// thread's lane.
template <> struct RingSums<float, 1> {
    static constexpr int E = RingGeo<float, 1>::kRows;
    RingAcc<float> acc[E];
    uint32_t tmem = 0;
    // Warp w owns lanes 32 (w % 4) .. + 31 and 64 columns from 64 (w / 4).
    __device__ __forceinline__ void init(uint32_t base, uint32_t warp) {
        tmem = base + ((warp & 3u) << 21) + (warp >> 2) * 64u;
        const uint64_t zero[8] = {};
#pragma unroll
        for (uint32_t k = 0; k < E / 4; ++k) tmem_store8(tmem + 16u * k, zero);
        tmem_wait_stores();
    }
    __device__ __forceinline__ void fold() {
        __syncwarp();
#pragma unroll
        for (uint32_t k = 0; k < E / 4; ++k) {
            uint64_t v[8];
            tmem_load8(tmem + 16u * k, v);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) acc[4 * k + j].fold(v[2 * j], v[2 * j + 1]);
            tmem_store8(tmem + 16u * k, v);
        }
        tmem_wait_stores();
    }
    // Rows 4 k .. 4 k + 3 (after the last fold).
    __device__ __forceinline__ void values(uint32_t k, float2 (&out)[4]) const {
        uint64_t v[8];
        tmem_load8(tmem + 16u * k, v);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) out[j] = RingAcc<float>::value(v[2 * j], v[2 * j + 1]);
    }
};

// The words of the records are the same for every lane, but come from shared
// memory, so the compiler must guard each branch on them with convergence
// barriers (8 of 74 instructions per run).  A warp reduction of the next word,
// taken while the present run is applied, makes them uniform.  It pays for
// complex128 (28 qubits: 168 ms against 180; Jordan-Wigner operator on 20 qubits:
// 6.45 against 7.10) and not for complex64, whose runs are shorter (26 qubits: 26.0
// against 23.7 ms).
template <typename R> __device__ __forceinline__ uint32_t ring_uniform(uint32_t word) {
    if constexpr (sizeof(R) == 8)
        return __reduce_or_sync(0xffffffffu, word);
    else
        return word;
}

// Walk one step: its block and source tile in shared memory, for the thread
// `tid` whose row word is `row_word`.
template <typename R, int SHAPE>
__device__ __forceinline__ void ring_walk(const unsigned char *blk, const typename Cx<R>::T *xs, uint32_t tid,
                                          uint32_t row_word, RingSums<R, SHAPE> &sums) {
    using C = typename Cx<R>::T;
    using G = RingGeo<R, SHAPE>;
    constexpr int E = G::kRows;
    const unsigned char *p = blk + 16;
    uint4 rec = *reinterpret_cast<const uint4 *>(p);
    C xv[E];
    R dsum = R(0);
    uint32_t left = ring_uniform<R>(*reinterpret_cast<const uint32_t *>(blk)), next_word = ring_uniform<R>(rec.y);
    for (; left; --left) {
        const uint32_t word = next_word;
        if (word & tcp::kRingNew) {
            const C *src = xs + ((tid ^ (word >> tcp::kRingMaskShift)) << G::kLow);
            if constexpr (G::kLow == 0) {
#pragma unroll
                for (int j = 0; j < E; ++j) xv[j] = src[G::row(j)];
            } else {
                // row bit 0 is a register bit: two complex64 rows per 16-byte load
#pragma unroll
                for (int j = 0; j < E; j += 2) {
                    const float4 v = *reinterpret_cast<const float4 *>(src + G::row(j));
                    xv[j] = C{v.x, v.y};
                    xv[j + 1] = C{v.z, v.w};
                }
            }
        }
        const uint32_t sign = ring_sign(rec.x, row_word);
        R w = ring_weight<R>(rec);
        const unsigned char *next = p + 16;
        // one branch past the common record: a single without sign changes
        if (word & (tcp::kRingKindMask | tcp::kRingFlipMask)) {
            if (word & tcp::kRingKindMask) {
                next = p;
                w = ring_table<R>(next, rec, row_word);
            }
            if (word & (1u << tcp::kRingFlipShift)) ring_flip_rows<0>(xv);
            if (word & (2u << tcp::kRingFlipShift)) ring_flip_rows<1>(xv);
            if (word & (4u << tcp::kRingFlipShift)) ring_flip_rows<2>(xv);
            if constexpr (E > 8) {
                if (word & (8u << tcp::kRingFlipShift)) ring_flip_rows<3>(xv);
            }
        }
        p = next;
        rec = *reinterpret_cast<const uint4 *>(p);  // the next record (16 unused bytes after the last)
        dsum += xor_sign(w, sign);
        next_word = ring_uniform<R>(rec.y);
        if (word & tcp::kRingLast) {
            ring_dispatch<E, R>(dsum, word, xv, sums.acc);
            dsum = R(0);
            // FP32: fold the running partial sums into the compensated row
            // sums (every tcp::kRingFoldRuns runs)
            if constexpr (sizeof(R) == 4) {
                if (word & tcp::kRingFold) {
                    sums.fold();
                    if constexpr (G::kTmem) {
#pragma unroll
                        for (int j = 0; j < E; ++j) xv[j] = C{0.f, 0.f};  // dead: a new coset follows
                    }
                }
            }
        }
    }
}

}  // namespace tcpdev
