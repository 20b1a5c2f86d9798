// mxradix.h -- radices of the any-length transforms (mx.cu), for its planner and its
// kernels.
#pragma once

namespace mx {

// First factor of a composite radix (0: prime)
__host__ __device__ constexpr int first_factor(int R)
{
    if (R > 4 && R % 4 == 0) return 4;
    for (int p = 2; p * p <= R; p++)
        if (R % p == 0) return p;
    return 0;
}

} // namespace mx
