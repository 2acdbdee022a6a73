// qsv_side.h -- side streams: streams of the library's own that run beside a caller's stream, between two points of it.
#pragma once
#include <cuda_runtime.h>

namespace qsv {

struct SideStreams {
    static constexpr int kMax = 3;
    int dev = -1;
    cudaStream_t stream[kMax] = {};
    cudaEvent_t fork = nullptr, joined[kMax] = {};
};

// A set of side streams on the current device, or null if they cannot be made: the caller then does without them, and
// no error is left behind for its next launch to report.
SideStreams *side_take();
void side_give(SideStreams *s);

}  // namespace qsv
