// screen_dd.cu -- the (dd|dd) diagonals of the Schwarz screening
#include "screen_kernel.cuh"

int launch_screen_dd(const PairRec *pairs, PrimPairs pp, int n, int pure, double *sums, cudaStream_t st)
{
    return launch_screen_slices<2, 2>(pairs, pp, n, pure, sums, st);
}
