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

// a build of n launches after what `main` holds; fail: stops after that many
static cudaError_t build(cudaStream_t main, int n, int fail, SideLease *held = nullptr)
{
    FockStreams fs(main);
    SideLease own, &side = held ? *held : own;
    const ForkScope scope(side);
    if (side.take(main) != cudaSuccess) return cudaErrorUnknown;
    if (side.p && side.fork(fs, n) != cudaSuccess) return cudaErrorUnknown;
    for (int k = 0; k < n; k++) {
        if (k == fail) return cudaErrorUnknown;
        launch(fs);
    }
    return side.join();
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
        const cudaError_t e = build(&main_stream, 12, fail);
        CHECK((e == cudaSuccess) == (fail < 0));
        CHECK(behind_all(&main_stream, first));     // a retry, or a free, comes after every launch
    }
    // a record of the join fails: the host waits for that stream instead
    for (int rec = 1; rec <= 8; rec++) {
        FakeStream main_stream;
        const int first = next_launch;
        fake_fail_record = rec;
        CHECK(build(&main_stream, 12, -1) != cudaSuccess);
        fake_fail_record = 0;
        CHECK(behind_all(&main_stream, first));
    }
    // leased for the build: one set served every one of them
    CHECK(side_pool().idle.size() == 1);
    CHECK(fake_streams == GTF_FOCK_STREAMS - 1 && fake_events == GTF_FOCK_STREAMS);

    // under capture: no set is taken or created inside; one taken before is used and kept
    side_pool().idle.clear();
    fake_streams = fake_events = 0;
    FakeStream captured;
    SideLease held;
    CHECK(held.take(&captured) == cudaSuccess && held.p);
    SideStreams *set = held.p;
    const int made = fake_streams;
    captured.capturing = true;
    CHECK(build(&captured, 12, -1) == cudaSuccess && side_pool().idle.empty() && fake_streams == made);
    const int first = next_launch;
    CHECK(build(&captured, 12, 5, &held) != cudaSuccess);
    CHECK(behind_all(&captured, first));
    CHECK(build(&captured, 12, -1, &held) == cudaSuccess);
    CHECK(behind_all(&captured, first));
    CHECK(held.p == set && side_pool().idle.empty());
    captured.capturing = false;
    held.release();
    CHECK(side_pool().idle.size() == 1);

    // no set waits and none may be created
    side_pool().idle.clear();
    FakeStream plain;
    SideLease none;
    CHECK(none.take(&plain, false) == cudaSuccess && !none.p);

    // at most GTF_SIDE_SETS wait in the pool
    fake_streams = 0;
    {
        SideLease many[GTF_SIDE_SETS + 3];
        for (SideLease &l : many) CHECK(l.take(&plain) == cudaSuccess);
        CHECK(fake_streams == (GTF_SIDE_SETS + 3) * (GTF_FOCK_STREAMS - 1));
    }
    CHECK(side_pool().idle.size() == GTF_SIDE_SETS);
    CHECK(fake_streams == GTF_SIDE_SETS * (GTF_FOCK_STREAMS - 1));
    return 0;
}
