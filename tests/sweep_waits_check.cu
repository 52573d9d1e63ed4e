// GPU check of the tracer sweeps' bounded waits, on the kernels themselves. Modes:
//
//   stream nx nz limit   the streaming sweep (k_stream_prep, k_tracer_stream) with waits of at most `limit`
//                        cycles: "<timeout word> <mismatches>", the results against those of the
//                        wavefront sweep (k_tracer_wavefront, IEEE division)
//   tiles nx nz passes   the tiled sweep (k_tracer_tiles, one chunk) with a bound of `passes` passes: likewise
//
// The domain has cloud-like tracers, both signs of wind, a stretched grid.
#include <climits>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../moist2d_b200/csrc/tracer_stream.cuh"

using namespace moist;
typedef float T;

template <class U>
U* device(const std::vector<U>& h) {
    U* d = nullptr;
    if (cudaMalloc(&d, h.size() * sizeof(U)) != cudaSuccess ||
        cudaMemcpy(d, h.data(), h.size() * sizeof(U), cudaMemcpyHostToDevice) != cudaSuccess) {
        printf("cuda error\n");
        exit(2);
    }
    return d;
}

int main(int argc, char** argv) {
    if (argc != 5) return 2;
    const int nx = atoi(argv[2]), nz = atoi(argv[3]), P = (nx + 31) / 32 * 32;
    const long long limit = atoll(argv[4]);
    if (nx < 4 || nz < 4 || nz > STREAM_MAX_ROWS) return 2;
    const size_t n = (size_t)nz * P;
    unsigned long long seed = 88172645463325252ull;
    auto rnd = [&] {  // xorshift64
        seed ^= seed << 13;
        seed ^= seed >> 7;
        seed ^= seed << 17;
        return (T)((seed >> 11) * 0x1p-53);
    };
    auto field = [&](T lo, T hi) {
        std::vector<T> v(n);
        for (T& x : v) x = lo + (hi - lo) * rnd();
        return v;
    };
    DevParams<T> p{};
    p.nx = nx;
    p.nz = nz;
    p.P = P;
    p.dx = T(250);
    p.dt = T(2);
    p.kappa = T(1.4);
    p.EPS = T(1e-12);
    std::vector<T> dz(nz), z(nz);
    T top = T(0);
    for (int k = 0; k < nz; k++) {
        dz[k] = T(100 + 2 * k);
        z[k] = top + dz[k] * T(0.5);
        top += dz[k];
    }
    p.dz = device(dz);
    p.z = device(z);
    TracerArgs<T> a{};
    T* ref[3];
    for (int t = 0; t < 3; t++) {
        a.q_old[t] = device(field(T(-5e-4), T(2e-3)));
        a.q0[t] = device(field(T(0), T(2e-3)));
        a.dphys[t] = device(field(T(-1e-6), T(1e-6)));
        a.q_new[t] = device(std::vector<T>(n));
        ref[t] = device(std::vector<T>(n));
    }
    a.rho = device(field(T(0.3), T(1.2)));
    a.mfx = device(field(T(-30), T(30)));
    a.mfz = device(field(T(-10), T(10)));
    a.dt = T(2);
    int* err = device(std::vector<int>{INT_MAX, INT_MAX, 0, 0});
    TracerArgs<T> ar = a;
    for (int t = 0; t < 3; t++) ar.q_new[t] = ref[t];
    k_tracer_wavefront<T><<<3, (nz + 31) / 32 * 32, 3 * nz * sizeof(T)>>>(p, ar, err);

    if (!strcmp(argv[1], "stream")) {
        StreamArgs<T> s{};
        s.tr = a;
        s.dom = device(std::vector<T>(skew_elems(nx, nz) * SK_ND));
        for (int t = 0; t < 3; t++) s.trc[t] = device(std::vector<T>(skew_elems(nx, nz) * SK_NT));
        s.spin_limit = limit;
        const size_t smem = stream_smem_bytes<T>(nz);
        cudaFuncSetAttribute(k_tracer_stream<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        k_stream_prep<T><<<dim3((nx + 34) / 32, (nz + 31) / 32), 256>>>(p, s, err);
        k_tracer_stream<T><<<3, stream_threads(nz), smem>>>(p, s, err);
    } else if (!strcmp(argv[1], "tiles")) {
        TileCtl c{};
        c.tiles_x = c.chunk_x = (nx + TT_W - 1) / TT_W;
        c.tiles_z = (nz + TT_H - 1) / TT_H;
        c.ntiles = c.tiles_x * c.tiles_z;
        c.max_pass = (int)limit;
        c.bar = device(std::vector<unsigned long long>(3));
        c.changed = device(std::vector<int>((size_t)2 * 3 * c.ntiles * 2));
        c.passes = device(std::vector<int>(1));
        c.hist = device(std::vector<int>(64));
        c.timeout = err + 2;
        c.spin_limit = 4000000000ll;
        T* strips = device(std::vector<T>((size_t)TT_RING * 3 * c.ntiles * 4 * TT_W));
        const int smem = (int)sizeof(TileSmem<T>);
        cudaFuncSetAttribute(k_tracer_tiles<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        const int* e = err;
        void* args[] = {&p, &a, &c, &strips, &e};
        if (cudaLaunchCooperativeKernel((void*)k_tracer_tiles<T, false>, dim3(c.ntiles), dim3(96), args, smem, 0) !=
            cudaSuccess)
            return 2;
    } else {
        return 2;
    }
    int word[4];
    if (cudaMemcpy(word, err, sizeof word, cudaMemcpyDeviceToHost) != cudaSuccess || cudaGetLastError() != cudaSuccess) {
        printf("cuda error\n");
        return 2;
    }
    size_t bad = 0;
    std::vector<T> x(n), y(n);
    for (int t = 0; t < 3; t++) {
        cudaMemcpy(x.data(), a.q_new[t], n * sizeof(T), cudaMemcpyDeviceToHost);
        cudaMemcpy(y.data(), ref[t], n * sizeof(T), cudaMemcpyDeviceToHost);
        for (int k = 0; k < nz; k++)
            for (int i = 0; i < nx; i++) bad += !(x[(size_t)k * P + i] == y[(size_t)k * P + i]);
    }
    printf("%d %zu\n", word[2], bad);
    return 0;
}
