// GPU checks of the tracer cell's divisions (FastDiv of moist2d_b200/csrc/fastdiv.cuh) against
// IEEE division, bit for bit: a quotient counts as a mismatch when it is finite, its `bad` flag is
// clear and it is not the IEEE quotient (in ratio(), a zero of either sign matches a zero). Modes:
//
//   cdiv b...        every float numerator by each b > 0: "<b> <cdiv> <quot> <ratio> <ratio by -b> <bad>"
//   rcp              rcp_rn of every float |b| in [2^-125, 2^125] against 1/b: "rcp <mismatches>"
//   div6             every float numerator of |a| in [2^-30, 2^120], and +0: "div6 <mismatches>"
//   random n seed    n random float (a, b) bit patterns, half of them with exponents near the type's
//                    lower end: "random <cdiv> <quot> <ratio> <accepted>"
//   random64 n seed  the same in double, with div6: "random64 <cdiv> <quot> <ratio> <div6> <accepted>"
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../moist2d_b200/csrc/fastdiv.cuh"

using namespace moist;
typedef unsigned long long u64;

__device__ __forceinline__ bool same(float x, float y) { return __float_as_uint(x) == __float_as_uint(y); }
__device__ __forceinline__ bool same(double x, double y) { return __double_as_longlong(x) == __double_as_longlong(y); }
template <class T>
__device__ __forceinline__ bool is_finite(T x) { return fabs(x) <= DivRange<T>::MAX; }

__device__ __forceinline__ u64 mix64(u64 z) {  // splitmix64 finaliser
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// c: mismatches of cdiv, quot and quot_var, ratio(b), ratio(-b); refused by cdiv (not finite); accepted by ratio
template <class T>
__device__ __forceinline__ void check(T a, T b, const Rcp<T>& y, T y1, bool prepared, u64* c) {
    using F = FastDiv<T>;
    const T r = a / b;
    bool bad = false;
    if (prepared) {
        const T q = F::cdiv(a, b, y);
        c[0] += is_finite(q) && !same(q, r);
        c[4] += !is_finite(q);
        const T q1 = F::quot(a, b, y1, bad);
        c[1] += !bad && is_finite(q1) && !same(q1, r);
        bad = false;
        const T q2 = F::quot_var(a, b, bad);
        c[1] += !bad && !same(q2, r);
    }
    bad = false;
    const T v = F::ratio(a, b, false, bad);
    c[2] += !bad && is_finite(v) && v != r;
    c[5] += !bad && is_finite(v);
    bad = false;
    const T w = F::ratio(a, -b, false, bad);
    c[3] += !bad && is_finite(w) && w != -r;
}

__global__ void k_cdiv(float b, u64* out) {
    const u64 st = (u64)gridDim.x * blockDim.x;
    u64 c[6] = {0, 0, 0, 0, 0, 0};
    const Rcp<float> y = FastDiv<float>::prep(b);
    const float y1 = FastDiv<float>::prep1(b);
    for (u64 u = blockIdx.x * (u64)blockDim.x + threadIdx.x; u < (1ull << 32); u += st)
        check(__uint_as_float((unsigned)u), b, y, y1, true, c);
    for (int j = 0; j < 6; j++) atomicAdd(out + j, c[j]);
}
__global__ void k_rcp(u64* out) {
    const u64 st = (u64)gridDim.x * blockDim.x;
    u64 n = 0;
    for (u64 u = blockIdx.x * (u64)blockDim.x + threadIdx.x; u < (1ull << 32); u += st) {
        const float b = __uint_as_float((unsigned)u);
        float y0;
        bool bad = false;
        if (fabsf(b) >= 0x1p-125f && fabsf(b) <= 0x1p125f) n += !same(rcp_rn(b, y0, bad), 1.0f / b);
    }
    atomicAdd(out, n);
}
__global__ void k_div6(u64* out) {
    const u64 st = (u64)gridDim.x * blockDim.x;
    u64 n = 0;
    for (u64 u = blockIdx.x * (u64)blockDim.x + threadIdx.x; u < (1ull << 32); u += st) {
        const float a = __uint_as_float((unsigned)u);
        if (u == 0 || (fabsf(a) >= 0x1p-30f && fabsf(a) <= 0x1p120f)) n += !same(FastDiv<float>::div6(a), a / 6.0f);
    }
    atomicAdd(out, n);
}
__global__ void k_random(u64 n, u64 seed, u64* out) {
    const u64 st = (u64)gridDim.x * blockDim.x;
    u64 c[6] = {0, 0, 0, 0, 0, 0};
    for (u64 j = blockIdx.x * (u64)blockDim.x + threadIdx.x; j < n; j += st) {
        const u64 h = mix64(seed * 0x9e3779b97f4a7c15ull + j);
        unsigned ua = (unsigned)h, ub = (unsigned)(h >> 32);
        if (j & 1) ub = (ub & 0x807fffffu) | ((((ub >> 23) & 0x1f) + 112u) << 23);  // |b| in [2^-15, 2^16]
        if (j & 2) ua = (ua & 0x807fffffu) | (((ua >> 23) & 0x1f) << 23);           // a subnormal or just above
        const float a = __uint_as_float(ua), b = fabsf(__uint_as_float(ub));
        check(a, b, FastDiv<float>::prep(b), FastDiv<float>::prep1(b), true, c);
    }
    for (int j = 0; j < 6; j++) atomicAdd(out + j, c[j]);
}
__global__ void k_random64(u64 n, u64 seed, u64* out) {
    const u64 st = (u64)gridDim.x * blockDim.x;
    u64 c[6] = {0, 0, 0, 0, 0, 0}, d6 = 0;
    for (u64 j = blockIdx.x * (u64)blockDim.x + threadIdx.x; j < n; j += st) {
        u64 ua = mix64(seed * 0x9e3779b97f4a7c15ull + 2 * j), ub = mix64(seed * 0x9e3779b97f4a7c15ull + 2 * j + 1);
        if (j & 1) ub = (ub & 0x800fffffffffffffull) | ((((ub >> 52) & 0x1f) + 1007ull) << 52);
        if (j & 2) ua = (ua & 0x800fffffffffffffull) | (((ua >> 52) & 0x3f) << 52);
        if (j & 4) {  // short significands: quotients on and near ties
            ua &= ~0xffffffffffull;
            ub &= ~0xffffffffffull;
        }
        if (j & 8) ub |= 0xffffffff00000ull;  // significands of many ones
        const double a = __longlong_as_double((long long)ua), b = fabs(__longlong_as_double((long long)ub));
        check(a, b, FastDiv<double>::prep(b), FastDiv<double>::prep1(b), true, c);
        const double m = __longlong_as_double((long long)((ua & 0x800fffffffffffffull) | ((((ua >> 52) & 0x7f) + 970ull) << 52)));
        d6 += !same(FastDiv<double>::div6(m), m / 6.0);
    }
    for (int j = 0; j < 6; j++) atomicAdd(out + j, c[j]);
    atomicAdd(out + 6, d6);
}

int main(int argc, char** argv) {
    if (argc < 2) return 2;
    u64* d;
    if (cudaMalloc(&d, 64) != cudaSuccess) return 2;
    u64 h[8];
    auto run = [&](auto launch) {
        cudaMemset(d, 0, 64);
        launch();
        if (cudaMemcpy(h, d, 64, cudaMemcpyDeviceToHost) != cudaSuccess) {
            printf("cuda error\n");
            exit(2);
        }
    };
    const dim3 g(148 * 8), b(256);
    const char* mode = argv[1];
    if (!strcmp(mode, "cdiv")) {
        for (int j = 2; j < argc; j++) {
            const float bv = strtof(argv[j], nullptr);
            run([&] { k_cdiv<<<g, b>>>(bv, d); });
            printf("%a %llu %llu %llu %llu %llu\n", bv, h[0], h[1], h[2], h[3], h[4]);
        }
    } else if (!strcmp(mode, "rcp")) {
        run([&] { k_rcp<<<g, b>>>(d); });
        printf("rcp %llu\n", h[0]);
    } else if (!strcmp(mode, "div6")) {
        run([&] { k_div6<<<g, b>>>(d); });
        printf("div6 %llu\n", h[0]);
    } else if (!strcmp(mode, "random") && argc == 4) {
        run([&] { k_random<<<g, b>>>(strtoull(argv[2], nullptr, 10), strtoull(argv[3], nullptr, 10), d); });
        printf("random %llu %llu %llu %llu\n", h[0], h[1], h[2] + h[3], h[5]);
    } else if (!strcmp(mode, "random64") && argc == 4) {
        run([&] { k_random64<<<g, b>>>(strtoull(argv[2], nullptr, 10), strtoull(argv[3], nullptr, 10), d); });
        printf("random64 %llu %llu %llu %llu %llu\n", h[0], h[1], h[2] + h[3], h[6], h[5]);
    } else {
        return 2;
    }
    cudaFree(d);
    return 0;
}
