// qsv_side.cpp -- side streams (qsv_side.h).
#include "qsv_side.h"

#include <mutex>
#include <new>
#include <vector>

namespace qsv {

static void destroy(SideStreams *s) {
    for (int k = 0; k < SideStreams::kMax; k++) {
        if (s->stream[k]) cudaStreamDestroy(s->stream[k]);
        if (s->joined[k]) cudaEventDestroy(s->joined[k]);
    }
    if (s->fork) cudaEventDestroy(s->fork);
    delete s;
}

// Sets that were given back (never destroyed with the process: its contexts may be gone by then). Streams and events
// belong to a device's primary context, which is assumed not to be reset while the library is loaded.
struct Kept {
    std::mutex mu;
    std::vector<SideStreams *> sets;
};
static Kept &kept() {
    static Kept *k = new Kept;
    return *k;
}

// a set whose streams a capture still holds is neither handed out nor destroyed
static bool in_capture(const SideStreams *s) {
    for (int k = 0; k < SideStreams::kMax; k++) {
        cudaStreamCaptureStatus st;
        if (cudaStreamIsCapturing(s->stream[k], &st) != cudaSuccess) {
            cudaGetLastError();
            return true;
        }
        if (st != cudaStreamCaptureStatusNone) return true;
    }
    return false;
}

static SideStreams *make(int dev) {
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

SideStreams *side_take() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    Kept &p = kept();
    {
        std::lock_guard<std::mutex> lk(p.mu);
        for (size_t i = p.sets.size(); i-- > 0;) {
            SideStreams *s = p.sets[i];
            if (s->dev != dev || in_capture(s)) continue;
            p.sets.erase(p.sets.begin() + (long)i);
            return s;
        }
    }
    return make(dev);
}

void side_give(SideStreams *s) {
    if (!s) return;
    Kept &p = kept();
    std::vector<SideStreams *> out;              // over the bound: destroyed, the oldest first
    {
        std::lock_guard<std::mutex> lk(p.mu);
        int n = 1;
        for (const SideStreams *x : p.sets) n += x->dev == s->dev;
        try {
            out.reserve(p.sets.size() + 1);
            p.sets.push_back(s);
        } catch (...) {
            destroy(s);
            return;
        }
        for (size_t i = 0; i < p.sets.size() && n > kSideKept;) {
            SideStreams *x = p.sets[i];
            if (x->dev == s->dev && !in_capture(x)) {
                out.push_back(x);
                p.sets.erase(p.sets.begin() + (long)i);
                n--;
            } else {
                i++;
            }
        }
    }
    for (SideStreams *x : out) destroy(x);
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
