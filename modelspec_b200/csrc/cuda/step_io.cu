// The two ends of a step: its inputs taken over from the staging slot of its turn, its loss and
// status word put where the host reads them. Both run inside the step's graph.
//
// Bound by latency, not by bytes: a copy engine's turn in the stream (a host-to-device copy in
// front, two 4-byte device-to-host copies behind) costs the device 2 to 10 us of waiting each, a
// kernel that reads and writes pinned memory itself about one trip over PCIe. Which of the
// kStagingSlots slots a step uses changes from step to step while its graph's arguments do not, so
// the slot number lives in device memory and the step moves it on itself.
#include "common.cuh"
#include "kernels.cuh"

namespace msx {
namespace k {

namespace {

constexpr int kTakeThreads = 256, kTakeChunks = 4;

// 16-byte chunks, four in flight per thread. No word in pinned memory is read by more than one warp:
// reads of one host address are served one after the other, about a microsecond each.
__global__ void __launch_bounds__(kTakeThreads) take_inputs_kernel(const __grid_constant__ InputSlots slots, uint64_t chunks, uint4* to,
                                                                    const uint32_t* turn) {
    after_producers();
    const uint4* from = reinterpret_cast<const uint4*>(slots.at[*turn % slots.count]);
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * kTakeThreads;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * kTakeThreads + threadIdx.x; i < chunks; i += kTakeChunks * stride) {
        uint4 v[kTakeChunks];
#pragma unroll
        for (int j = 0; j < kTakeChunks; ++j)
            if (i + j * stride < chunks) v[j] = __ldcv(from + i + j * stride);
#pragma unroll
        for (int j = 0; j < kTakeChunks; ++j)
            if (i + j * stride < chunks) to[i + j * stride] = v[j];
    }
}

__global__ void publish_step_kernel(const float* loss, const uint32_t* status, float* to_loss,
                                    uint32_t* to_status, uint32_t* turn, uint32_t slots) {
    after_producers();
    const uint32_t slot = *turn;
    if (loss) to_loss[slot] = *loss;
    to_status[slot] = *status;
    *turn = slot + 1 == slots ? 0u : slot + 1;
}

}  // namespace

void take_inputs(cudaStream_t s, const InputSlots& slots, uint64_t bytes, char* to, const uint32_t* turn) {
    const uint64_t chunks = bytes / 16;
    // A chunk a thread while that keeps the grid within one wave (64 KB from pinned memory is 16
    // blocks); four a thread and a loop beyond.
    uint64_t blocks = (chunks + kTakeThreads - 1) / kTakeThreads;
    if (blocks > 296) blocks = 296;
    take_inputs_kernel<<<static_cast<uint32_t>(blocks), kTakeThreads, 0, s>>>(slots, chunks, reinterpret_cast<uint4*>(to), turn);
    check_launch("take_inputs");
}

void publish_step(cudaStream_t s, const float* loss, const uint32_t* status, float* to_loss, uint32_t* to_status, uint32_t* turn, uint32_t slots) {
    publish_step_kernel<<<1, 1, 0, s>>>(loss, status, to_loss, to_status, turn, slots);
    check_launch("publish_step");
}

}  // namespace k
}  // namespace msx
