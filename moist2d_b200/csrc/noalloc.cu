// noalloc.cu - an allocation-free entry point: the vertically implicit w-p column solve
// (implicit_correction!) for many columns at once, on device buffers the caller owns.
//
// Who needs it: callers that must not have a library allocate device memory behind them. A
// Julia host routes every device allocation through CUDA.jl's memory pool and counts on it to
// reclaim memory under pressure; a host with a fixed device-memory budget reserves all of it
// up front and cannot meet an out-of-memory failure in the middle of a run; and a host that
// keeps other streams busy cannot afford cudaFree, which waits for the whole device.
// moist_implicit_correction allocates its column buffers on every call; this variant
// allocates nothing. The grid vectors travel in the kernel's parameter block (so the call
// issues no host-to-device copy either), and the elimination works in shared memory and registers.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>

#include "../../include/moist2d.h"
#include "fastdiv.cuh"
#include "model.cuh"

namespace {

// the grid vectors dz and z, passed by value in the kernel's parameter block (at most
// MOIST_NOALLOC_MAX_NZ levels: 16 KiB in Float64, within the 32 KiB parameter limit). The smaller of two
// capacities that holds nz travels: 16 KiB of parameters a launch cost the host and the GPU's front
// end more than the solve of a small call.
template <class T, int CAP>
struct ColumnGrid {
    T dz[CAP];
    T z[CAP];
};

void put_msg(char* err, size_t errlen, const char* msg) {
    if (err && errlen) {
        std::strncpy(err, msg, errlen - 1);
        err[errlen - 1] = '\0';
    }
}

// One row of the w-p system of a column (moist.jl:974-1030): level k, th, r2, w and dw at that level
template <class T>
struct Row {
    T a, b, c, d;  // the diagonal is b + 1
};
template <class T>
struct Factors {
    T grav, dt_tp2, fact;
    __device__ Factors(T grav_, T beta, T dt) : grav(grav_) {
        const T fact_tp = T(0.5) * (T(1.0) + beta);
        const T fact_tm = T(0.5) * (T(1.0) - beta);
        dt_tp2 = (dt * fact_tp) * (dt * fact_tp);
        fact = fact_tm / fact_tp;
    }
};
template <class T, int CAP>
__device__ __forceinline__ Row<T> row_of(int k, int ke, const Factors<T>& f, const ColumnGrid<T, CAP>& grid, const T* th,
                                         const T* r2, const T* w, const T* dw) {
    const T dz_k = grid.dz[k], dz_kp = grid.dz[k + 1], zd = grid.z[k + 1] - grid.z[k];
    const T th_cur = moist::f2h(th[0], th[1], dz_k, dz_kp);
    const T th_prev = k > 0 ? moist::f2h(th[-1], th[0], grid.dz[k - 1], dz_k) : T(0);
    const T th_next = (k + 1 <= ke - 1) ? moist::f2h(th[1], th[2], dz_kp, grid.dz[k + 2]) : T(0);
    Row<T> r;
    r.b = f.dt_tp2 * (r2[0] / dz_k + r2[1] / dz_kp) * th_cur / zd;
    r.a = (k > 0) ? -f.dt_tp2 * (r2[0] * th_prev / (zd * dz_k) - f.grav / (dz_k + dz_kp)) : T(0);
    r.c = (k < ke - 1) ? -f.dt_tp2 * (r2[1] * th_next / (zd * dz_kp) + f.grav / (dz_k + dz_kp)) : T(0);
    r.d = w[0] + dw[0];
    if (k > 0) r.d -= r.a * f.fact * w[0];
    r.d -= r.b * f.fact * w[0];
    if (k < ke - 1) r.d -= r.c * f.fact * w[1];
    return r;
}

// shared memory of one level of one column: a, b + 1, c, d (T), c', d' (TT)
template <class T, class TT>
constexpr size_t level_bytes() {
    return 4 * sizeof(T) + 2 * sizeof(TT);
}
// elements from one column to the next: odd, so that the columns' threads read different banks
__host__ __device__ inline int column_stride(int nz, int wc) { return wc == 1 ? nz : (nz | 1); }
constexpr int kThreads = 128;

// wc adjacent columns per block, column j of each (nz, ncols) array starting at j * nz (z fastest, the
// reference layout): a block's columns are one contiguous piece of every array. All threads form the
// coefficients and right-hand sides of the piece's levels (whole-line loads, divisions in
// parallel), one thread per column eliminates and substitutes in shared memory, all threads write the
// piece back. What bounds it is the elimination's chain: two multiply-subtracts and the
// quotients c' and d' per level, both from one reciprocal of the pivot (rcp_rn and two remainder
// corrections, fastdiv.cuh; a column with a refused or non-finite quotient is eliminated again with
// IEEE division). Same arithmetic as implicit_correction! (moist.jl:974-1030) and solve_tridiagonal!
// (moist.jl:952-971), with the elimination in TT. One thread per column out of global memory, every
// load a line of its own: 204 us a call for 2048 columns of 128 levels (Float32, FP64 elimination);
// this way 41 us.
template <class T, class TT, int CAP>
__global__ void __launch_bounds__(kThreads) k_implicit_columns_noalloc(int nz, int ncols, int wc, T grav, T beta, T* rho_w,
                                                                       const T* drho_w, const T* theta,
                                                                       const T* rt2pres, T dt,
                                                                       const __grid_constant__ ColumnGrid<T, CAP> grid) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    using F = moist::FastDiv<TT>;
    const int n = nz - 1, ke = nz - 1, ld = column_stride(nz, wc);
    const int j0 = blockIdx.x * wc, nc = min(wc, ncols - j0);
    TT* cps = reinterpret_cast<TT*>(smem_raw);  // [wc][ld]
    TT* dps = cps + (size_t)wc * ld;
    T* sa = reinterpret_cast<T*>(dps + (size_t)wc * ld);
    T* sb = sa + (size_t)wc * ld;
    T* sc = sb + (size_t)wc * ld;
    T* sd = sc + (size_t)wc * ld;
    const Factors<T> f(grav, beta, dt);
    const size_t base = (size_t)j0 * nz;
    for (int e = threadIdx.x; e < nc * nz; e += kThreads) {
        const int col = e / nz, k = e - col * nz;
        if (k >= n) continue;
        const int o = col * ld + k;
        const size_t c0 = base + e;  // this level of this column
        const Row<T> r = row_of(k, ke, f, grid, theta + c0, rt2pres + c0, rho_w + c0, drho_w + c0);
        sa[o] = r.a;
        sb[o] = r.b + T(1.0);
        sc[o] = r.c;
        sd[o] = r.d;
    }
    __syncthreads();
    if (threadIdx.x < nc) {
        const size_t o = (size_t)threadIdx.x * ld;
        const T* __restrict__ pa = sa + o;
        const T* __restrict__ pb = sb + o;
        const T* __restrict__ pc = sc + o;
        T* __restrict__ pd = sd + o;
        TT* __restrict__ cp = cps + o;
        TT* __restrict__ dp = dps + o;
        auto eliminate = [&](auto quotients) {
            TT c_prev = TT(0), d_prev = TT(0);
            T an = pa[0], bn = pb[0], cn = pc[0], dn = pd[0];
#pragma unroll 2
            for (int k = 0; k < n; k++) {  // the next level's operands are read one level ahead
                const TT a = (TT)an, b = (TT)bn, c = (TT)cn, d = (TT)dn;
                const int kn = k + 1 < n ? k + 1 : n - 1;
                an = pa[kn];
                bn = pb[kn];
                cn = pc[kn];
                dn = pd[kn];
                const TT piv = k == 0 ? b : b - a * c_prev, num = k == 0 ? d : d - a * d_prev;
                quotients(c, num, piv, c_prev, d_prev);
                cp[k] = c_prev;
                dp[k] = d_prev;
            }
        };
        bool bad = false;
        eliminate([&](TT c, TT num, TT piv, TT& q_c, TT& q_d) {
            bad |= !(piv >= F::LO && piv <= F::HI);
            TT y0;
            const TT y = moist::rcp_rn(piv, y0, bad);
            q_c = F::twice(c, piv, y0, y, piv * F::TIE, bad);
            q_d = F::twice(num, piv, y0, y, piv * F::TIE, bad);
            bad |= !(fabs(q_c) <= F::MAX) || !(fabs(q_d) <= F::MAX);
        });
        if (bad)
            eliminate([&](TT c, TT num, TT piv, TT& q_c, TT& q_d) {
                q_c = c / piv;
                q_d = num / piv;
            });
        TT x = dp[n - 1];
        pd[n - 1] = (T)x;
        const int k1 = n >= 2 ? n - 2 : 0;
        TT dn = dp[k1], cn = cp[k1];
#pragma unroll 4
        for (int k = n - 2; k >= 0; k--) {
            const TT dk = dn, ck = cn;
            const int kn = k >= 1 ? k - 1 : 0;
            dn = dp[kn];
            cn = cp[kn];
            x = dk - ck * x;
            pd[k] = (T)x;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nc * nz; e += kThreads) {
        const int col = e / nz, k = e - col * nz;
        if (k < n) rho_w[base + e] = sd[col * ld + k];  // the lid face is never solved
    }
}

// Columns of few levels: one thread per column, everything in registers, IEEE division. A column is then a
// sector or two of every array, and pieces of 8 columns leave most of a block's threads without a level: 262144
// columns of 2 levels took 43.6 us, 65536 of 5 18.4 us, 29127 of 10 13.7 us that way (Float32, FP64 elimination),
// 3.3, 4.5 and 7.3 us this way (5.1, 8.6 and 14.0 with one thread per column out of a scratch array). What bounds it
// is the chain of quotients, so up to 64 columns an SM only the shortest columns take it: 6000 columns of
// 5 levels 3.5 us against 3.9 in pieces, but 6000 of 8 5.0 against 4.6 (Float64 6.9 against 5.0).
template <class T, class TT, int NZ>
__global__ void __launch_bounds__(kThreads) k_implicit_columns_few(int ncols, T grav, T beta, T* rho_w,
                                                                   const T* drho_w, const T* theta, const T* rt2pres,
                                                                   T dt, const __grid_constant__ ColumnGrid<T, NZ> grid) {
    constexpr int n = NZ - 1;
    const int j = blockIdx.x * kThreads + threadIdx.x;
    if (j >= ncols) return;
    const Factors<T> f(grav, beta, dt);
    const size_t base = (size_t)j * NZ;
    TT cp[n], dp[n];
#pragma unroll
    for (int k = 0; k < n; k++) {
        const size_t c0 = base + k;
        const Row<T> r = row_of(k, NZ - 1, f, grid, theta + c0, rt2pres + c0, rho_w + c0, drho_w + c0);
        const TT bb = (TT)(r.b + T(1.0));
        if (k == 0) {
            cp[0] = (TT)r.c / bb;
            dp[0] = (TT)r.d / bb;
        } else {
            const TT piv = bb - (TT)r.a * cp[k - 1];
            cp[k] = (TT)r.c / piv;
            dp[k] = ((TT)r.d - (TT)r.a * dp[k - 1]) / piv;
        }
    }
    TT x = dp[n - 1];
    rho_w[base + n - 1] = (T)x;
#pragma unroll
    for (int k = n - 2; k >= 0; k--) {
        x = dp[k] - cp[k] * x;
        rho_w[base + k] = (T)x;
    }
}
constexpr int FEW = 4, FEW_MANY = 10;  // levels: for any number of columns, for more than 64 an SM
template <class T, class TT, int NZ = FEW_MANY>
cudaError_t launch_few(const moist_params* p, int ncols, void* rho_w, const void* drho_w, const void* theta,
                       const void* rt2pres, double dt, cudaStream_t st) {
    if constexpr (NZ > 2) {
        if (p->nz < NZ) return launch_few<T, TT, NZ - 1>(p, ncols, rho_w, drho_w, theta, rt2pres, dt, st);
    }
    ColumnGrid<T, NZ> grid;
    std::memcpy(grid.dz, p->dz, sizeof grid.dz);
    std::memcpy(grid.z, p->z, sizeof grid.z);
    k_implicit_columns_few<T, TT, NZ><<<(ncols + kThreads - 1) / kThreads, kThreads, 0, st>>>(
        ncols, (T)p->grav, (T)p->beta_offcenter, (T*)rho_w, (const T*)drho_w, (const T*)theta, (const T*)rt2pres,
        (T)dt, grid);
    return cudaGetLastError();
}

template <class T, class TT, int CAP>
cudaError_t launch_noalloc(const moist_params* p, int ncols, void* rho_w, const void* drho_w, const void* theta,
                           const void* rt2pres, double dt, cudaStream_t st) {
    const int nz = p->nz;
    int dev = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess) return e;
    if (nz <= FEW || (nz <= FEW_MANY && ncols > 64 * nsm))
        return launch_few<T, TT>(p, ncols, rho_w, drho_w, theta, rt2pres, dt, st);
    ColumnGrid<T, CAP> grid;  // levels from nz on are never read
    std::memcpy(grid.dz, p->dz, nz * sizeof(T));
    std::memcpy(grid.z, p->z, nz * sizeof(T));
    // columns per block: 8, fewer where the default 48 KiB of shared memory ask for it (one column of 1024
    // levels takes 48 KiB in Float64) or while the blocks are fewer than the SMs, whose chains run side by side
    auto bytes = [&](int w) { return level_bytes<T, TT>() * column_stride(nz, w) * w; };
    int wc = 8;
    while (wc > 1 && (bytes(wc) > 48 * 1024 || (ncols + wc - 1) / wc < nsm)) wc /= 2;
    k_implicit_columns_noalloc<T, TT, CAP><<<(ncols + wc - 1) / wc, kThreads, bytes(wc), st>>>(
        nz, ncols, wc, (T)p->grav, (T)p->beta_offcenter, (T*)rho_w, (const T*)drho_w, (const T*)theta,
        (const T*)rt2pres, (T)dt, grid);
    return cudaGetLastError();
}

template <class T, class TT>
int run_noalloc(const moist_params* p, int ncols, void* rho_w, const void* drho_w, const void* theta,
                const void* rt2pres, double dt, cudaStream_t st, char* err, size_t errlen) {
    const int nz = p->nz;
    // the call's documented limit: the elimination's values (TT, 2 (nz-1) per column)
    const size_t work_bytes = 2 * (size_t)(nz - 1) * ncols * sizeof(TT);
    if (work_bytes > MOIST_NOALLOC_SCRATCH_BYTES) {
        char msg[256];
        std::snprintf(msg, sizeof msg,
                      "moist_implicit_correction_noalloc: %d columns of %d levels are %zu scratch bytes of elimination, "
                      "more than the %d that a call takes (MOIST_NOALLOC_SCRATCH_BYTES)",
                      ncols, nz, work_bytes, (int)MOIST_NOALLOC_SCRATCH_BYTES);
        put_msg(err, errlen, msg);
        return MOIST_ERR_ARG;
    }
    const cudaError_t e = nz <= 256 ? launch_noalloc<T, TT, 256>(p, ncols, rho_w, drho_w, theta, rt2pres, dt, st)
                                    : launch_noalloc<T, TT, MOIST_NOALLOC_MAX_NZ>(p, ncols, rho_w, drho_w, theta, rt2pres, dt, st);
    if (e != cudaSuccess) {
        put_msg(err, errlen, cudaGetErrorString(e));
        return MOIST_ERR_CUDA;
    }
    return MOIST_OK;
}

}  // namespace

extern "C" {
#pragma GCC visibility push(default)

int moist_implicit_correction_noalloc(const moist_params* p, int precision, int flags, int ncols, void* rho_w,
                                      const void* drho_w, const void* theta, const void* rt2pres, double dt,
                                      void* stream, char* err, size_t errlen) {
    put_msg(err, errlen, "");
    if (!p || !p->dz || !p->z || p->nz < 2 || ncols < 0 || !rho_w || !drho_w || !theta || !rt2pres) {
        put_msg(err, errlen, "moist_implicit_correction_noalloc: invalid argument");
        return MOIST_ERR_ARG;
    }
    if (p->nz > MOIST_NOALLOC_MAX_NZ) {
        char msg[160];
        std::snprintf(msg, sizeof msg, "moist_implicit_correction_noalloc: nz = %d is above the limit of %d levels",
                      p->nz, (int)MOIST_NOALLOC_MAX_NZ);
        put_msg(err, errlen, msg);
        return MOIST_ERR_ARG;
    }
    if (precision != MOIST_F32 && precision != MOIST_F64) {
        put_msg(err, errlen, "moist_implicit_correction_noalloc: unknown precision");
        return MOIST_ERR_ARG;
    }
    if (ncols == 0) return MOIST_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (precision == MOIST_F64) return run_noalloc<double, double>(p, ncols, rho_w, drho_w, theta, rt2pres, dt, st, err, errlen);
    if (flags & MOIST_FLAG_TRI_NATIVE) return run_noalloc<float, float>(p, ncols, rho_w, drho_w, theta, rt2pres, dt, st, err, errlen);
    return run_noalloc<float, double>(p, ncols, rho_w, drho_w, theta, rt2pres, dt, st, err, errlen);
}

#pragma GCC visibility pop
}  // extern "C"
