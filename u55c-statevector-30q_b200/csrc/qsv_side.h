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
// Whether work on the first `count` streams of s can be tied to the caller's stream: they are captured into the same
// graph as it is, or neither it nor they are captured. (A side stream that a launch has brought into a capture stays in
// it until the capture ends; work of other streams must not meet it there.)
bool side_joins(const SideStreams *s, int count, cudaStream_t stream);

}  // namespace qsv
