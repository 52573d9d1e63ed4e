// GPU check of quotient_proven (moist2d_b200/csrc/fastdiv.cuh), the acceptance test of the acoustic
// substep's quotients, on n random double pairs with a seed:
//
//   n seed: "<wrong accepted> <right refused> <right refused at powers of two> <accepted>"
//
// For q = a / b (IEEE) the test must accept q and refuse both neighbours of q. At a power of two, where
// the spacing below is half the one above, it may refuse q as well.
#include <cstdio>
#include <cstdlib>

#include "../moist2d_b200/csrc/fastdiv.cuh"

using namespace moist;
typedef unsigned long long u64;

__device__ __forceinline__ u64 mix64(u64 z) {  // splitmix64 finaliser
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ __forceinline__ double bits(u64 u) { return __longlong_as_double((long long)u); }

__global__ void k_check(u64 n, u64 seed, u64* out) {
    u64 c[4] = {0, 0, 0, 0};
    for (u64 j = blockIdx.x * (u64)blockDim.x + threadIdx.x; j < n; j += (u64)gridDim.x * blockDim.x) {
        u64 ua = mix64(seed * 0x9e3779b97f4a7c15ull + 2 * j), ub = mix64(seed * 0x9e3779b97f4a7c15ull + 2 * j + 1);
        if (j & 1) ua &= ~0xffffffffffull, ub &= ~0xffffffffffull;  // short significands: exact quotients
        if (j & 2) ub |= 0xfffffffff0000ull;                        // significands of many ones
        double a = bits(ua);
        const double b = bits(ub);
        if (j & 4) {  // quotients at and beside powers of two
            const u64 e = (ua >> 52) & 0x7ff, m = (ub & 0xfffffffffffffull) + (j & 8 ? 1 : 0) - (j & 16 ? 1 : 0);
            a = bits((ua & (1ull << 63)) | (e << 52) | (m & 0xfffffffffffffull));
        }
        const double aa = fabs(a), ab = fabs(b), q = a / b, aq = fabs(q);
        const bool ranges = aa >= 0x1p-960 && aa <= 0x1p1000 && ab >= 0x1p-1000 && ab <= 0x1p1000 && aq >= 0x1p-960 &&
                            aq <= 0x1p1000;
        const u64 uq = (u64)__double_as_longlong(q);
        const bool ok = quotient_proven(a, b, q);
        c[3] += ok;
        if (ranges) c[(uq & 0xfffffffffffffull) == 0 ? 2 : 1] += !ok;
        if (aq >= 0x1p-1000 && aq <= 0x1p1000) c[0] += quotient_proven(a, b, bits(uq + 1)) + quotient_proven(a, b, bits(uq - 1));
    }
    for (int k = 0; k < 4; k++) atomicAdd(out + k, c[k]);
}

int main(int argc, char** argv) {
    if (argc != 3) return 2;
    u64 *d, h[4];
    if (cudaMalloc(&d, sizeof h) != cudaSuccess) return 2;
    cudaMemset(d, 0, sizeof h);
    k_check<<<148 * 8, 256>>>(strtoull(argv[1], nullptr, 10), strtoull(argv[2], nullptr, 10), d);
    if (cudaMemcpy(h, d, sizeof h, cudaMemcpyDeviceToHost) != cudaSuccess) {
        printf("cuda error\n");
        return 2;
    }
    printf("%llu %llu %llu %llu\n", h[0], h[1], h[2], h[3]);
    cudaFree(d);
    return 0;
}
