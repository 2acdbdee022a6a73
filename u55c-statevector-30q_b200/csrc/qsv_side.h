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

// A set of side streams on the current device, the caller's alone until it gives it back (also with work of its own
// still running), or null if none can be made: the caller then does without, and no error is left behind for its next
// launch to report. Sets that were given back are kept, at most kSideKept on a device, and handed out again: making
// three streams and four events takes 160-180 us and destroying them as long. Batches made, uploaded, launched once and
// freed, as the serving loop does (us): four circuits of 12 and 13 qubits 650-710 with a set of their own each time, 329
// with kept ones (553 one qubit count after the other), 16 circuits of 10-13 qubits 1850, 1430 (2100). Any thread may
// call these.
constexpr int kSideKept = 8;
SideStreams *side_take();
void side_give(SideStreams *s);
// Whether work on the first `count` streams of s can be tied to the caller's stream: they are captured into the same
// graph as it is, or neither it nor they are captured. (A side stream that a launch has brought into a capture stays in
// it until the capture ends; work of other streams must not meet it there.)
bool side_joins(const SideStreams *s, int count, cudaStream_t stream);

}  // namespace qsv
