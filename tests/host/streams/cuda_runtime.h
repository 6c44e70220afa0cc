// Stand-in for the stream and event calls of cuda_runtime.h that keeps, per
// stream, the set of launches it is ordered behind.
#pragma once
#include <set>

typedef int cudaError_t;
enum { cudaSuccess = 0, cudaErrorUnknown = 999 };
enum { cudaEventDisableTiming = 2, cudaStreamNonBlocking = 1 };
enum cudaStreamCaptureStatus { cudaStreamCaptureStatusNone, cudaStreamCaptureStatusActive };
struct FakeStream {
    std::set<int> behind;
    bool capturing = false;
};
struct FakeEvent {
    std::set<int> at;
};
typedef FakeStream *cudaStream_t;
typedef FakeEvent *cudaEvent_t;

static std::set<int> fake_done;        // launches the host has waited for
static int fake_streams, fake_events;  // alive
static int fake_fail_record;           // the n-th record from now on fails
static int fake_dev;

inline cudaError_t cudaGetDevice(int *d) { *d = fake_dev; return cudaSuccess; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, int) { *e = new FakeEvent; fake_events++; return cudaSuccess; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { delete e; fake_events--; return cudaSuccess; }
inline cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, int) { *s = new FakeStream; fake_streams++; return cudaSuccess; }
inline cudaError_t cudaStreamDestroy(cudaStream_t s) { delete s; fake_streams--; return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s)
{
    if (fake_fail_record > 0 && --fake_fail_record == 0) return cudaErrorUnknown;
    e->at = s->behind;
    return cudaSuccess;
}
inline cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, int)
{
    s->behind.insert(e->at.begin(), e->at.end());
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s)
{
    fake_done.insert(s->behind.begin(), s->behind.end());
    return cudaSuccess;
}
inline cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus *c)
{
    *c = s->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
