// side_streams.cuh -- streams for the launches of one build that are
// independent of one another.
#pragma once

#include <cuda_runtime.h>

#include <mutex>
#include <vector>

// Streams the launches of a build are dealt out to in turn (n == 1: all in
// order on one stream).
#define GTF_FOCK_STREAMS 8
struct FockStreams {
    cudaStream_t s[GTF_FOCK_STREAMS];
    int n, next;
    explicit FockStreams(cudaStream_t st) : n(1), next(0) { s[0] = st; }
    cudaStream_t take()
    {
        const cudaStream_t st = s[next];
        next = next + 1 < n ? next + 1 : 0;
        return st;
    }
};

// A set of side streams.  Sets are leased for one build: they come from a
// process-wide pool (creating one takes 0.3 ms), so there are as many as
// builds that were ever under way at once, and at most GTF_SIDE_SETS wait in
// the pool.
#define GTF_SIDE_SETS 16
struct SideStreams {
    int dev;
    cudaStream_t s[GTF_FOCK_STREAMS - 1];
    cudaEvent_t ev_fork, ev_join[GTF_FOCK_STREAMS - 1];
};
struct SidePool {
    std::mutex mu;
    std::vector<SideStreams *> idle;
};
inline SidePool &side_pool()
{
    static SidePool pool;
    return pool;
}

inline void side_destroy(SideStreams *p)
{
    for (int k = 0; k < GTF_FOCK_STREAMS - 1; k++) {
        if (p->ev_join[k]) cudaEventDestroy(p->ev_join[k]);
        if (p->s[k]) cudaStreamDestroy(p->s[k]);
    }
    if (p->ev_fork) cudaEventDestroy(p->ev_fork);
    delete p;
}

// The lease of one build.  fork() lets the first n - 1 side streams start
// where fs.s[0] stands, join() lets fs.s[0] go on once they are through.  The
// end of the lease joins on every way out, a failed launch among them, so that
// a retry's clears and the frees of a destroyed engine come after all that was
// launched, and returns the set.  The set may still be busy then: what its
// next user launches comes after that.
struct SideLease {
    SideStreams *p;
    FockStreams *fs;   // forked and not joined
    SideLease() : p(nullptr), fs(nullptr) {}
    SideLease(const SideLease &) = delete;
    SideLease &operator=(const SideLease &) = delete;
    ~SideLease() { release(); }
    // Takes a set of the current device for a build on `st`: from the pool,
    // or a new one if none waits there.  The lease stays empty without
    // `create`, or when `st` is being captured: a set belongs to a capture
    // until that ends, so whoever captures takes it before and keeps it.
    cudaError_t take(cudaStream_t st, bool create = true)
    {
        if (p) return cudaSuccess;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        cudaError_t e = cudaStreamIsCapturing(st, &cap);
        if (e != cudaSuccess || cap != cudaStreamCaptureStatusNone) return e;
        int dev = 0;
        e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        {
            std::lock_guard<std::mutex> lk(side_pool().mu);
            std::vector<SideStreams *> &idle = side_pool().idle;
            for (size_t k = 0; k < idle.size(); k++)
                if (idle[k]->dev == dev) {
                    p = idle[k];
                    idle.erase(idle.begin() + k);
                    return cudaSuccess;
                }
        }
        if (!create) return cudaSuccess;
        SideStreams *q = new SideStreams();
        q->dev = dev;
        e = cudaEventCreateWithFlags(&q->ev_fork, cudaEventDisableTiming);
        for (int k = 0; k < GTF_FOCK_STREAMS - 1 && e == cudaSuccess; k++) {
            e = cudaStreamCreateWithFlags(&q->s[k], cudaStreamNonBlocking);
            if (e == cudaSuccess) e = cudaEventCreateWithFlags(&q->ev_join[k], cudaEventDisableTiming);
        }
        if (e == cudaSuccess) p = q;
        else side_destroy(q);
        return e;
    }
    // needs a set
    cudaError_t fork(FockStreams &f, int n)
    {
        cudaError_t e = cudaEventRecord(p->ev_fork, f.s[0]);
        f.n = n < 1 ? 1 : n > GTF_FOCK_STREAMS ? GTF_FOCK_STREAMS : n;
        for (int k = 1; k < f.n && e == cudaSuccess; k++) {
            f.s[k] = p->s[k - 1];
            e = cudaStreamWaitEvent(f.s[k], p->ev_fork, 0);
        }
        if (e == cudaSuccess) fs = &f;
        else f.n = 1;   // nothing was launched on the others
        return e;
    }
    // whatever fails, fs.s[0] waits for every stream it can
    cudaError_t join()
    {
        cudaError_t first = cudaSuccess;
        for (int k = 1; fs && k < fs->n; k++) {
            cudaError_t e = cudaEventRecord(p->ev_join[k - 1], fs->s[k]);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(fs->s[0], p->ev_join[k - 1], 0);
            if (e != cudaSuccess) cudaStreamSynchronize(fs->s[k]);
            if (first == cudaSuccess) first = e;
        }
        if (fs) {
            fs->n = 1;
            fs->next = 0;
        }
        fs = nullptr;
        return first;
    }
    void release()
    {
        join();
        if (!p) return;
        {
            std::lock_guard<std::mutex> lk(side_pool().mu);
            if (side_pool().idle.size() < GTF_SIDE_SETS) {
                side_pool().idle.push_back(p);
                p = nullptr;
            }
        }
        if (p) side_destroy(p);   // a busy stream is destroyed when its work is done
        p = nullptr;
    }
};

// joins a lease that outlives the build
struct ForkScope {
    SideLease &side;
    explicit ForkScope(SideLease &l) : side(l) {}
    ~ForkScope() { side.join(); }
};
