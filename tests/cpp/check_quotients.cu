// quotient() and over() of epilogue.cuh against division, bit for bit: every float for the two constants and for
// x / 1, random pairs for the others.  Prints the number of differences of each.
#include <cstdio>

#include <cuda_runtime.h>

#include "epilogue.cuh"

namespace {

__device__ unsigned long long bad[4];

__device__ void count(int slot, float got, float want)
{
    if (__float_as_uint(got) != __float_as_uint(want)) atomicAdd(&bad[slot], 1ull);
}

__global__ void every_float(float cs, float cs2)
{
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 32); i += stride)
    {
        const float x = __uint_as_float((unsigned)i);
        if ((unsigned)i == 0x80000000u || !(fabsf(x) <= 0x1p98f)) continue;   // -0: sums that start at 0 never give it
        count(0, lbm::over(x, cs, 1.0f / cs), __fdiv_rn(x, cs));
        count(1, lbm::over(x, cs2, 1.0f / cs2), __fdiv_rn(x, cs2));
        count(2, lbm::quotient(x, 1.0f, __frcp_rn(1.0f)), x);
    }
}

__global__ void random_pairs()
{
    const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x; i < (1ull << 31); i += stride)
    {
        unsigned long long r = i * 0x9e3779b97f4a7c15ull + 11;
        r = (r ^ (r >> 30)) * 0xbf58476d1ce4e5b9ull;
        r = (r ^ (r >> 27)) * 0x94d049bb133111ebull;
        r ^= r >> 31;
        const unsigned ex = 30u + (unsigned)((r >> 50) % 188ull), eb = 123u + (unsigned)((r >> 47) & 7u);   // 2^-97 .. 2^90, 2^-4 .. 2^4
        const float x = __uint_as_float(((unsigned)(r >> 46) << 31) | (ex << 23) | ((unsigned)r & 0x7fffffu));
        const float b = __uint_as_float((eb << 23) | ((unsigned)(r >> 23) & 0x7fffffu));
        count(3, lbm::quotient(x, b, __frcp_rn(b)), __fdiv_rn(x, b));
    }
}

}  // namespace

int main()
{
    every_float<<<1184, 256>>>((float)lbm::kCs, (float)lbm::kCs2);
    random_pairs<<<1184, 256>>>();
    unsigned long long h[4];
    const cudaError_t e = cudaMemcpyFromSymbol(h, bad, sizeof(h));
    std::printf("%s %llu %llu %llu %llu\n", e == cudaSuccess ? "ok" : cudaGetErrorString(e), h[0], h[1], h[2], h[3]);
    return e != cudaSuccess;
}
