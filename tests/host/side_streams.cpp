// Order of the launches of a build around fork and join (side_streams.cuh);
// exits 0 when every check holds, else names the first that does not.
#include <cuda_runtime.h>

#include "side_streams.cuh"

#include <cstdio>

#define CHECK(x)                                          \
    do {                                                  \
        if (!(x)) {                                       \
            printf("line %d: %s\n", __LINE__, #x);        \
            return 1;                                     \
        }                                                 \
    } while (0)

static int next_launch = 1;
static int launch(FockStreams &fs)
{
    fs.take()->behind.insert(next_launch);
    return next_launch++;
}

// a build of n launches after `clear` on the main stream; fail: stops after that many
static cudaError_t build(ForkJoin &side, cudaStream_t main, int n, int fail)
{
    FockStreams fs(main);
    ForkScope scope(side, fs);
    if (side.fork(fs, n) != cudaSuccess) return cudaErrorUnknown;
    for (int k = 0; k < n; k++) {
        if (k == fail) return cudaErrorUnknown;
        launch(fs);
    }
    return side.join(fs);
}

// every launch from `first` on
static bool behind_all(cudaStream_t s, int first)
{
    for (int k = first; k < next_launch; k++)
        if (!s->behind.count(k) && !fake_done.count(k)) return false;
    return true;
}

int main()
{
    for (int fail = -1; fail < 12; fail++) {
        FakeStream main_stream;
        const int first = next_launch;
        main_stream.behind.insert(next_launch++);   // the clears
        ForkJoin side{nullptr};
        const cudaError_t e = build(side, &main_stream, 12, fail);
        CHECK((e == cudaSuccess) == (fail < 0));
        CHECK(behind_all(&main_stream, first));            // a retry, or a free, comes after every launch
        side.give_back();
    }
    // a record of the join fails: the host waits for that stream instead
    for (int rec = 1; rec <= 8; rec++) {
        FakeStream main_stream;
        const int first = next_launch;
        ForkJoin side{nullptr};
        fake_fail_record = rec;
        CHECK(build(side, &main_stream, 12, -1) != cudaSuccess);
        fake_fail_record = 0;
        CHECK(behind_all(&main_stream, first));
        side.give_back();
    }
    CHECK(side_pool().idle.size() == 1);            // one set served every build
    CHECK(fake_streams == GTF_FOCK_STREAMS - 1 && fake_events == GTF_FOCK_STREAMS);
    return 0;
}
