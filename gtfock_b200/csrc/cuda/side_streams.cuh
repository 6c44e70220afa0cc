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
    cudaStream_t last;   // stream of the latest launch
    explicit FockStreams(cudaStream_t st) : n(1), next(0), last(st) { s[0] = st; }
    cudaStream_t take()
    {
        last = s[next];
        next = next + 1 < n ? next + 1 : 0;
        return last;
    }
};

// fork() lets the first n - 1 side streams start where fs.s[0] stands, join()
// lets fs.s[0] go on once they are through.  The sets come from a
// process-wide pool (creating one takes 0.3 ms) and return to it with the
// engine or batch that took them, at most GTF_SIDE_SETS waiting there.
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

struct ForkJoin {
    SideStreams *p;
    cudaError_t fork(FockStreams &fs, int n)
    {
        cudaError_t e = p ? cudaSuccess : take();
        if (e == cudaSuccess) e = cudaEventRecord(p->ev_fork, fs.s[0]);
        fs.n = n < 1 ? 1 : n > GTF_FOCK_STREAMS ? GTF_FOCK_STREAMS : n;
        for (int k = 1; k < fs.n && e == cudaSuccess; k++) {
            fs.s[k] = p->s[k - 1];
            e = cudaStreamWaitEvent(fs.s[k], p->ev_fork, 0);
        }
        if (e != cudaSuccess) fs.n = 1;   // nothing was launched on the others
        return e;
    }
    // whatever fails, fs.s[0] waits for every stream it can
    cudaError_t join(FockStreams &fs)
    {
        cudaError_t first = cudaSuccess;
        for (int k = 1; k < fs.n; k++) {
            cudaError_t e = cudaEventRecord(p->ev_join[k - 1], fs.s[k]);
            if (e == cudaSuccess) e = cudaStreamWaitEvent(fs.s[0], p->ev_join[k - 1], 0);
            if (e != cudaSuccess) cudaStreamSynchronize(fs.s[k]);
            if (first == cudaSuccess) first = e;
        }
        fs.n = 1;
        fs.next = 0;
        return first;
    }
    cudaError_t take()
    {
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
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
    // The builds that used the set have been joined: what is left on it is
    // ordered before the work the owner's stream, and its next user's, has.
    void give_back()
    {
        if (!p) return;
        for (cudaStream_t q : p->s) cudaStreamSynchronize(q);
        {
            std::lock_guard<std::mutex> lk(side_pool().mu);
            if (side_pool().idle.size() < GTF_SIDE_SETS) {
                side_pool().idle.push_back(p);
                p = nullptr;
            }
        }
        if (p) side_destroy(p);
        p = nullptr;
    }
};

// Joins the streams of a fork on every way out, a failed launch among them:
// the caller's stream is then ordered behind all that was launched, so a
// retry's clears and the frees of a destroyed engine come after it.
struct ForkScope {
    ForkJoin &fj;
    FockStreams &fs;
    ForkScope(ForkJoin &f, FockStreams &s) : fj(f), fs(s) {}
    ~ForkScope() { fj.join(fs); }
    ForkScope(const ForkScope &) = delete;
    ForkScope &operator=(const ForkScope &) = delete;
};
