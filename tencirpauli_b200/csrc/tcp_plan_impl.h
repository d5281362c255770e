// Host-side layout of a plan object, shared by the .cu files of libtcpmvp.so.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

#include "tcp_device.cuh"
#include "tcp_internal.h"

namespace tcp {

struct DeviceSchedule {
    Schedule host;
    RingSchedule ring[kRingShapeCount];  // k_ring's schedules (tile_bits = 0: the plan has none of this shape)
    tcpdev::DevSchedule dev{};
};

// Page-locked staging ring of a host apply whose caller's buffers are
// ordinary (pageable) memory: kStageSlots slots of kStageSlotBytes; slot use u
// goes to slot u % kStageSlots, and ev[slot] marks the end of its last DMA.
// Small slots shorten what nothing overlaps: the host copy of the first and the
// last piece of each direction (2^22 complex128, 64 MiB each way: 6.3 ms with
// 4 slots of 32 MiB, 5.5 with 8 of 16, 5.06 with 16 of 8 or 32 of 4, 5.3 with 64
// of 2; on buffers not used before 6.1 with 4 of 32, 5.1 with 16 of 8; 2^26, 1 GiB
// each way, on another host: 61 to 67 with 4 of 32, 60 to 63 with 8 of 16, 55 to 61
// with 16 of 8).
constexpr int kStageSlots = 16;
constexpr size_t kStageSlotBytes = size_t(8) << 20;
constexpr size_t kStageMinBytes = size_t(64) << 20;  // vectors from which the ring is used

struct Staging {
    unsigned char *host = nullptr;
    cudaEvent_t ev[kStageSlots] = {};
    uint64_t uses = 0;
};

struct Workspace {
    void *x = nullptr;
    void *y = nullptr;
    size_t bytes = 0;
    Staging *stage = nullptr;  // allocated on the first pageable apply
};

int cuda_fail(cudaError_t e, const char *what);
cudaError_t dev_malloc(void **p, size_t bytes);

}  // namespace tcp

struct tcp_mvp_plan {
    uint32_t nqubits = 0;
    uint32_t word_count = 0;
    uint64_t dim = 0;
    int storage = 0;
    int device = 0;
    int64_t transitions = -1;
    std::vector<tcp::MatrixTerm> terms;
    uint64_t group_count = 0;
    tcp::DeviceSchedule sched;  // one schedule (4096-row tiles) serves both precisions
    void *dev_block = nullptr;
    size_t dev_bytes = 0;
    int *d_err = nullptr;
    mutable std::mutex ws_mutex;
    mutable std::vector<tcp::Workspace> ws_free;
    mutable std::vector<tcp::Workspace> ws_all;
};

namespace tcp {
int check_plan(const tcp_mvp_plan *plan);
int length_error(uint64_t expected, uint64_t actual);
bool overlaps(const void *a, const void *b, size_t bytes);
int ring_prepare(const tcp_mvp_plan *p, bool c64);
int launch_ring_rhs(const tcp_mvp_plan *p, const void *x, void *y, uint32_t nrhs, bool c64, int *err,
                    cudaStream_t stream, bool accumulate = false);
}  // namespace tcp
