// qsv_side.cpp -- side streams (qsv_side.h).
#include "qsv_side.h"

#include <new>

namespace qsv {

static void destroy(SideStreams *s) {
    for (int k = 0; k < SideStreams::kMax; k++) {
        if (s->stream[k]) cudaStreamDestroy(s->stream[k]);
        if (s->joined[k]) cudaEventDestroy(s->joined[k]);
    }
    if (s->fork) cudaEventDestroy(s->fork);
    delete s;
}

SideStreams *side_take() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    SideStreams *s = new (std::nothrow) SideStreams;
    if (!s) return nullptr;
    s->dev = dev;
    bool ok = cudaEventCreateWithFlags(&s->fork, cudaEventDisableTiming) == cudaSuccess;
    for (int k = 0; ok && k < SideStreams::kMax; k++)
        ok = cudaStreamCreateWithFlags(&s->stream[k], cudaStreamNonBlocking) == cudaSuccess &&
             cudaEventCreateWithFlags(&s->joined[k], cudaEventDisableTiming) == cudaSuccess;
    if (ok) return s;
    destroy(s);
    cudaGetLastError();              // the launch after a failed call must not report it as its own
    return nullptr;
}

void side_give(SideStreams *s) {
    if (s) destroy(s);
}

static bool capture_of(cudaStream_t stream, cudaStreamCaptureStatus *status, unsigned long long *id) {
    *id = 0;
    return cudaStreamGetCaptureInfo(stream, status, id) == cudaSuccess;
}

bool side_joins(const SideStreams *s, int count, cudaStream_t stream) {
    cudaStreamCaptureStatus own, st;
    unsigned long long own_id, id;
    bool ok = capture_of(stream, &own, &own_id) && own != cudaStreamCaptureStatusInvalidated;
    for (int k = 0; ok && k < count; k++)
        ok = capture_of(s->stream[k], &st, &id) &&
             (st == cudaStreamCaptureStatusNone || (st == own && id == own_id));
    if (!ok) cudaGetLastError();     // (the legacy stream cannot be asked during a capture elsewhere)
    return ok;
}

}  // namespace qsv
