// tracer_tiles.cuh - the reference's in-place Gauss-Seidel tracer sweep, computed in parallel
// tiles and repaired to a bitwise fixed point.
//
// The reference updates rho_q in place in lexicographic order (moist.jl:1469-1518), so cell
// (k, i) reads the updated values at (k, i-1), (k, i-2), (k-1, i), (k-2, i) and the
// stage-start values everywhere else. Write F for the map "recompute every cell from the
// current values of its predecessors": the reference result is the unique fixed point of F
// (unique by induction along the dependency order). Here the domain is cut into tiles of 16 rows x 32
// columns. Inside a tile the order is exact: one warp per tracer, lanes r and r + 16 own row z0+r
// (tracer_cell.cuh) and process column c at wavefront step c + r, receiving the row below through
// warp shuffles. Across tile boundaries each tile starts from speculative values of its left and
// bottom neighbours' boundary strips (the stage-start values, which it forms itself), publishes
// its own right and top strips whenever they change, and is recomputed only when a neighbour's
// strip changed. A pass in which no strip changes leaves every tile computed from its neighbours'
// final values: a fixed point, hence the reference's result bit for bit. Information crosses one
// tile per pass, so a chunk needs at most its tile columns + tiles_z passes; max_pass leaves two to
// spare, and a sweep that reached it would report an error, never a result. Mostly a few passes
// do, but a change of one ulp can keep reproducing itself along uniform rows: on spun-up States 3-4 on
// 200 x 100 in Float32 and 5-8 in Float64, 11-16 on 2048 x 128 in Float64, 12-33 on 4096 x 256.
//
// The kernel is persistent (cooperative launch, the tiles of a chunk resident); passes are
// separated by a grid barrier whose wait is bounded: on timeout it records MOIST_ERR_TIMEOUT and
// returns. A domain of more tiles than fit is swept in chunks of tile columns from left to right:
// no cell depends on an updated value to its right, so a chunk's fixed point is final before the
// next chunk starts from it.
//
// What bounds it: the chain of dependent cells. A tile is 47 wavefront steps; with 16 rows and two
// lanes per cell a step is about half as long as with 32 rows and a lane per cell, a tile needs 47
// steps instead of 63, and twice as many tiles spread over the SMs. The walk of a whole tile (alone on
// its SM): 16 us in Float32, 31 us in Float64; the sweeps of a step on 2048 x 128 0.94 -> 0.37 ms in
// Float32, 11.6 -> 2.7 ms in Float64 (two chunks), on 4096 x 256 (four chunks; one block's wavefront
// with IEEE division before) 96.7 -> 3.2 ms.
#pragma once

#include "tracer_cell.cuh"

namespace moist {

constexpr int TT_W = 32;     // tile width (columns)
constexpr int TT_H = WROWS;  // tile height (rows)
constexpr int TT_S = TT_W + 2;  // row stride in shared memory: lane r reads column step - r, conflict-free

struct TileCtl {
    int tiles_x, tiles_z, ntiles, max_pass;  // max_pass: of one chunk
    int chunk_x;        // tile columns of a chunk (grid = chunk_x * tiles_z blocks)
    int* ver;           // dataflow sweep: [3][ntiles] words (version << 1 | final) of each tile's strips
    unsigned long long* bar;  // [2] arrivals (low word) and changed tiles (high word) of even and odd barriers,
                              // [2] blocks that have left the kernel; all zero between launches
    int* changed;       // [2][3][ntiles][2] per pass parity: rows whose right-strip entries changed, columns whose top-strip entries changed (bit masks)
    int* passes;        // out: passes run (all chunks)
    int* hist;          // [64] sweeps that converged after p passes
    int* timeout;       // out: 1: a wait ran out, 2: no fixed point within max_pass
    long long spin_limit;
    unsigned long long* pass_ts;  // optional diagnostic [max_pass + 3] of the first chunk: globaltimer at the
                                  // start of each pass, and at [max_pass + 2] when block 0 leaves it
    int* pass_work;               // optional diagnostic: [pass] warps that recomputed their tile
};

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ unsigned long long ld_acquire64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

// Bounded grid barrier with a count: every block adds one arrival, and one to the high word when
// it reports a change; the poll that sees the last arrival also returns the changes. Two counters
// alternate, so that no block can add to a counter that another still reads: a block reaches the
// next barrier on the same counter only after every block has left the one in between. One thread
// per block arrives with a reduction (nothing returned) and polls without sleeping; the counter
// costs one round trip to L2 instead of an arrival, a release and a read of a changed flag in turn
// (a pass without work on 2048 x 128, 512 blocks: 4.1 us before, 3.2 us now).
struct GridSync {
    unsigned n = 0;                            // barriers so far
    unsigned seen[2] = {0, 0};                 // high words at the end of the last even and odd barrier
    // -1: timed out; 0 / 1: no block / some block reported a change. Called by all threads.
    __device__ __forceinline__ int operator()(const TileCtl& c, unsigned nblocks, bool change) {
        __shared__ int s_res;
        const int any = __syncthreads_or(change);  // the block's stores are done
        if (threadIdx.x == 0) {
            unsigned long long* w = c.bar + (n & 1);
            const unsigned target = (n / 2 + 1) * nblocks;
            __threadfence();
            atomicAdd(w, any ? (1ull << 32) + 1ull : 1ull);
            const long long t0 = clock64();
            unsigned long long v;
            int ok = 1;
            while ((unsigned)(v = ld_acquire64(w)) < target) {
                if (clock64() - t0 > c.spin_limit) {
                    ok = 0;
                    atomicExch(c.timeout, 1);
                    break;
                }
            }
            const unsigned hi = (unsigned)(v >> 32);
            s_res = !ok || *(volatile int*)c.timeout != 0 ? -1 : hi != seen[n & 1];
            seen[n & 1] = hi;
        }
        n++;
        __syncthreads();
        return s_res;
    }
};

// faces staged in shared memory: x faces [TT_H][TT_S] (face c - 1/2 at index c), then z faces
// [TT_H + 1][TT_S] (face r - 1/2 at row r); the gap puts the two halves' lanes on different banks
constexpr int FACE_Z = TT_H * TT_S + 15;
constexpr int FACE_N = FACE_Z + (TT_H + 1) * TT_S;

template <class T>
struct TileSmem {
    T s[3][TT_H + 2][TT_S];  // per tracer: stage-start s = q/rho, rows z0 .. z0+17, cols x0 .. x0+33
    T q0[3][TT_H][TT_S];
    T dph[3][TT_H][TT_S];
    T qn[3][TT_H][TT_S];     // results
    T snp[3][TT_H][TT_S];    // s = q / rho of the last pass (the rows a repair pass replays)
    T rho[TT_H][TT_S], rrho[TT_H][TT_S];
    T vel[FACE_N];           // mass fluxes
    T rf[FACE_N];            // face densities: (rho_i + rho_i+1) / 2 and f2h of rho_k, rho_k+1
    T bot[3][2][TT_W];       // per tracer: the lower tile's top strip for the current pass
    T lin[3][TT_H + 2];      // per tracer: column 1 of the reference array (interior nx-2), rows z0-1 .. z0+16
    T cl[3][2][2][TT_W];     // per tracer: clamp quotients of the vertical limiter [p, m face][low, high row][column]
};

// the staging loops of k_tracer_tiles: every thread loads TT_BATCH elements (load(j) returns
// an element's value), then stores them (store(j, v)); elements j = threadIdx.x + u blockDim.x
constexpr int TT_BATCH = 8;
template <class V, class L, class S>
__device__ __forceinline__ void stage_batched(int total, L load, S store) {
    for (int j0 = threadIdx.x; j0 < total; j0 += TT_BATCH * (int)blockDim.x) {
        V v[TT_BATCH];
#pragma unroll
        for (int u = 0; u < TT_BATCH; u++) {
            const int j = j0 + u * (int)blockDim.x;
            if (j < total) v[u] = load(j);
        }
#pragma unroll
        for (int u = 0; u < TT_BATCH; u++) {
            const int j = j0 + u * (int)blockDim.x;
            if (j < total) store(j, v[u]);
        }
    }
}

// strips in global memory: [tracer][tile][4][32], right strip columns 30, 31 (rows in entries 0 .. 15),
// top strip rows 14, 15. One copy: a tile writes them in the pass they change, a neighbour that
// reads a value of the pass in progress is told by the next pass's mask to compute again.
template <class T>
__device__ __forceinline__ T* strip_ptr(T* strips, int t, int tile, int ntiles) {
    return strips + (((size_t)t * ntiles + tile) * 4) * TT_W;
}
// the dataflow sweep keeps the last TT_RING versions of each tile's strips:
// [tracer][tile][version % TT_RING][4][32]
constexpr int TT_RING = 4;
template <class T>
__device__ __forceinline__ T* strip_ver_ptr(T* strips, int t, int tile, int ver, int ntiles) {
    return strips + ((((size_t)t * ntiles + tile) * TT_RING + (ver % TT_RING)) * 4) * TT_W;
}
__device__ __forceinline__ int ld_acquire(const int* p) {
    int v;
    asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
    asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One walk of a tile by one tracer's warp: every cell from wavefront step `step` on, in order. It
// starts where the first changed input is read (earlier cells keep their values: they are
// recomputed from unchanged inputs or not at all) and ends early when, past the last changed
// input, two steps in a row changed no cell. The next step's operands are read one step ahead and
// the loop has no branch but its own end, so that a step costs the dependent length of the cell
// and little more (with a skipped-step test, a check of `bad` and loads in place a step took 1150
// cycles against about 490 of the cell alone). Returns whether the fast division refused an operand or a
// result is not finite: the caller then walks the whole tile with IeeeDiv.
template <class T>
struct TileLane {
    const T *S, *Sp1, *Sp2;          // stage-start s along the half's direction, at column 0
    const T *vel_p, *vel_m, *rf_p, *rf_m;
    const T *q0, *dph, *rho, *rrho, *cl_p, *cl_m, *bot0, *bot1;
    T *qn, *snp;
    int r, width;
    bool zh, row_ok;
};
template <class D, bool CEN, class T>
__device__ __forceinline__ bool tile_walk(const HalfRow<T>& w, const TileLane<T>& L, int step, int last_in, T in_p1, T in_p2) {
    const int r = L.r, nsteps = L.width + TT_H - 1;
    struct Ops {
        T sc, p1, p2, vp, vm, rp, rm, q0, dph, rho, rrho, cp, cm, b0, b1, old;
    };
    auto load = [&](int st) {
        const int c = min(max(st - r, 0), TT_W - 1);
        Ops o;
        o.sc = L.S[c];
        o.p1 = L.Sp1[c];
        o.p2 = L.Sp2[c];
        o.vp = L.vel_p[c];
        o.vm = L.vel_m[c];
        o.rp = L.rf_p[c];
        o.rm = L.rf_m[c];
        o.q0 = L.q0[c];
        o.dph = L.dph[c];
        o.rho = L.rho[c];
        o.rrho = L.rrho[c];
        o.cp = CEN ? L.cl_p[c] : T(0);
        o.cm = CEN ? L.cl_m[c] : T(0);
        o.b0 = L.bot0[c];
        o.b1 = L.bot1[c];
        o.old = L.snp[c];
        return o;
    };
    T prev1 = in_p1, prev2 = in_p2, sn_last = T(0), m1_used = T(0);
    if (step > 0) {  // the values the walk would have left behind one step earlier
        const int c = step - r;
        if (c >= 1) prev1 = L.snp[min(c, TT_W) - 1];
        if (c >= 2) prev2 = L.snp[min(c, TT_W) - 2];
        if (c == 1) prev2 = in_p1;
        if (c >= 1 && c <= TT_W) {
            sn_last = L.snp[c - 1];
            m1_used = r == 0 ? L.bot1[c - 1] : L.snp[c - 1 - TT_S];
        }
    }
    bool bad_any = false;
    unsigned chg1 = ~0u, chg2 = ~0u;  // rows changed one and two steps ago
    Ops nxt = load(step);
    for (; step < nsteps; step++) {
        if (step > last_in + 2 && (chg1 | chg2) == 0u) break;
        const Ops o = nxt;
        nxt = load(step + 1);
        const int c_raw = step - r;
        const bool active = L.row_ok && c_raw >= 0 && c_raw < L.width;
        // row-below values: lane r-1's result of the previous step and the value it used
        const T up_sn = __shfl_up_sync(0xffffffffu, sn_last, 1);
        const T up_m1 = __shfl_up_sync(0xffffffffu, m1_used, 1);
        const T m1 = L.zh ? (r == 0 ? o.b1 : up_sn) : prev1;
        const T m2 = L.zh ? (r == 0 ? o.b0 : (r == 1 ? o.b1 : up_m1)) : prev2;
        T q, sn;
        bool bad = false;
        two_lane_cell<D, CEN>(w, m2, m1, o.sc, o.p1, o.p2, o.vp, o.vm, o.rp, o.rm, o.cp, o.cm, o.q0, o.dph, o.rho, o.rrho,
                              q, sn, bad);
        bad_any |= bad && active;
        if (active && !L.zh) {
            L.qn[c_raw] = q;
            L.snp[c_raw] = sn;
        }
        prev2 = active ? prev1 : prev2;
        prev1 = active ? sn : prev1;
        // lane r+1 reads these next step only for the column it shares with this step
        sn_last = sn;
        m1_used = m1;
        chg2 = chg1;
        chg1 = __ballot_sync(0xffffffffu, active && !same_bits(sn, o.old));
    }
    __syncwarp();
    return __any_sync(0xffffffffu, bad_any);
}

// DF = false: passes separated by grid barriers (all tiles advance pass by pass). DF = true (one
// chunk only): no grid barrier; every tile publishes numbered versions of its strips and recomputes
// whenever its left or lower neighbour publishes a new version, so a chain of changes crosses the
// tiles at the pace of its own work. A tile is final once it has computed from its neighbours'
// final strips (the left column and the bottom row of tiles have fixed inputs), which every tile
// reaches because the dependencies run only left-to-right and bottom-to-top.
// Register bound: as many blocks as the shared memory lets onto an SM (49 KB and 99 KB a tile).
template <class T, bool DF>
__global__ void __launch_bounds__(96, sizeof(T) == 4 ? 4 : 2) k_tracer_tiles(DevParams<T> p, TracerArgs<T> a, TileCtl ctl, T* strips,
                                                     const int* err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileSmem<T>& sm = *reinterpret_cast<TileSmem<T>*>(smem_raw);
    const int nx = p.nx, nz = p.nz, P = p.P;
    const int t = threadIdx.x >> 5, lane = threadIdx.x & 31;  // this warp's tracer
    const int r = lane & (TT_H - 1);
    const bool zh = lane >= TT_H;                              // the z half
    const unsigned nblocks = gridDim.x;
    const int tz = blockIdx.x / ctl.chunk_x, z0 = tz * TT_H;
    const int k = z0 + r;
    const bool row_ok = k < nz;
    const bool halt = halted(err);  // uniform across the grid: every block still meets every barrier
    const HalfRow<T> w = half_row(p, k, zh, a.dt);
    GridSync sync;
    int npass_all = 0;

    for (int tx0 = 0; tx0 < ctl.tiles_x; tx0 += ctl.chunk_x) {
        const int tx = tx0 + blockIdx.x % ctl.chunk_x, tile = tz * ctl.tiles_x + tx;
        const bool mine = tx < ctl.tiles_x;  // the last chunk may be narrower: its spare blocks only meet the barriers
        const int x0 = tx * TT_W;
        const int width = min(TT_W, nx - x0);
        bool cen_any = false;
        if (mine) {
            // ---- stage the stage-start values this tile reads (coalesced rows). Each thread issues
            // the loads of TT_BATCH elements before it stores any, so that it waits for one memory
            // round trip per batch rather than per element. Densities of rows z0-1 .. z0+17 and
            // columns x0-1 .. x0+33 go through the space of the results, which is free until pass 1.
            constexpr int RW = TT_W + 3, RH = TT_H + 3;
            static_assert(RW * RH <= 3 * TT_H * TT_S, "the densities fit in the results' space");
            T* rho_t = &sm.qn[0][0][0];
            stage_batched<T>(RW * RH, [&](int j) {
                const int kk = z0 - 1 + j / RW, ii = x0 - 1 + j % RW;
                // columns beyond nx+1 are never read; the bound also keeps wrapx within one period
                return (kk >= 0 && kk < nz && ii < nx + 2) ? a.rho[MOIST_IDX(kk, wrapx(ii, nx))] : T(1);
            }, [&](int j, T v) { rho_t[j] = v; });
            stage_batched<T>(TT_H * (TT_W + 1), [&](int j) {
                const int kk = z0 + j / (TT_W + 1), ii = x0 - 1 + j % (TT_W + 1);
                // faces x0-1 .. nx-1 only: faces i-1 and i of the cells i < nx
                return (kk < nz && ii < nx) ? a.mfx[MOIST_IDX(kk, wrapx(ii, nx))] : T(0);
            }, [&](int j, T v) {
                cen_any |= !(fabs(v) > p.EPS);
                sm.vel[(j / (TT_W + 1)) * TT_S + j % (TT_W + 1)] = v;
            });
            stage_batched<T>((TT_H + 1) * TT_W, [&](int j) {
                const int kk = z0 - 1 + j / TT_W, ii = x0 + j % TT_W;
                return (kk >= 0 && kk < nz && ii < nx) ? a.mfz[MOIST_IDX(kk, ii)] : T(0);
            }, [&](int j, T v) {
                cen_any |= !(fabs(v) > p.EPS);
                sm.vel[FACE_Z + (j / TT_W) * TT_S + j % TT_W] = v;
            });
            for (int q = 0; q < 3; q++) {
                const T* qo = a.q_old[q];
                stage_batched<T>((TT_H + 2) * TT_S, [&](int j) {
                    const int kk = z0 + j / TT_S, cc = j % TT_S;
                    return (kk < nz && x0 + cc < nx + 2) ? qo[MOIST_IDX(kk, wrapx(x0 + cc, nx))] : T(0);
                }, [&](int j, T v) { sm.s[q][j / TT_S][j % TT_S] = v; });
                for (int j = threadIdx.x; j < TT_H + 2; j += blockDim.x) {
                    const int kk = z0 - 1 + j;
                    sm.lin[q][j] = (kk >= 0 && kk < nz) ? qo[MOIST_IDX(kk, nx - 2)] : T(0);
                }
                stage_batched<T>(TT_H * TT_W, [&](int j) {
                    const int kk = z0 + j / TT_W, ii = x0 + j % TT_W;
                    return (kk < nz && ii < nx) ? a.q0[q][MOIST_IDX(kk, ii)] : T(0);
                }, [&](int j, T v) { sm.q0[q][j / TT_W][j % TT_W] = v; });
                stage_batched<T>(TT_H * TT_W, [&](int j) {
                    const int kk = z0 + j / TT_W, ii = x0 + j % TT_W;
                    return (kk < nz && ii < nx) ? a.dphys[q][MOIST_IDX(kk, ii)] : T(0);
                }, [&](int j, T v) { sm.dph[q][j / TT_W][j % TT_W] = v; });
            }
            __syncthreads();
            // s = rho_q / rho, the face densities and the cells' reciprocals (once for three tracers)
            for (int j = threadIdx.x; j < (TT_H + 2) * TT_S; j += blockDim.x) {
                const int rr = j / TT_S, cc = j % TT_S;
                const T rho = rho_t[(rr + 1) * RW + cc + 1];
                for (int q = 0; q < 3; q++) sm.s[q][rr][cc] = sm.s[q][rr][cc] / rho;
            }
            for (int j = threadIdx.x; j < TT_H * (TT_W + 1); j += blockDim.x) {
                const int rr = j / (TT_W + 1), cc = j % (TT_W + 1);
                const T* rp = rho_t + (rr + 1) * RW + cc;  // cell c - 1, and c next to it
                sm.rf[rr * TT_S + cc] = (rp[1] + rp[0]) * T(0.5);
                if (cc > 0) {
                    sm.rho[rr][cc - 1] = rp[0];
                    sm.rrho[rr][cc - 1] = FastDiv<T>::prep1(rp[0]);
                }
            }
            for (int j = threadIdx.x; j < (TT_H + 1) * TT_W; j += blockDim.x) {
                const int rr = j / TT_W, cc = j % TT_W, kk = z0 - 1 + rr;
                const T* rp = rho_t + rr * RW + cc + 1;
                sm.rf[FACE_Z + rr * TT_S + cc] =
                    (kk >= 0 && kk < nz - 1) ? f2h(rp[RW], rp[0], p.dz[kk + 1], p.dz[kk]) : T(0);
            }
        }
        // the clamp rows need the centred face values wherever they lie
        const bool need_cen = __syncthreads_or(cen_any) != 0 || z0 <= 1 || z0 + TT_H >= nz - 1;
        if (mine) {
            // the clamp quotients lin / (+-vel dt) of limited_flux_z on the four rows that can use them:
            // face k+1/2 from rows k = 0 and nz-2, face k-1/2 from rows k = 1 and nz-1 (IEEE division)
            const int c = lane;
            for (int slot = 0; slot < 2; slot++) {
                T vkp = T(0), vkm = T(0);
                const int kp = slot == 0 ? 0 : nz - 2;  // face kp+1/2 between cells kp, kp+1
                const int km = slot == 0 ? 1 : nz - 1;  // face km-1/2 between cells km-1, km
                if (kp >= 0 && kp < nz - 1 && kp >= z0 && kp < z0 + TT_H && x0 + c < nx) {
                    const T vel = sm.vel[FACE_Z + (kp - z0 + 1) * TT_S + c];
                    const T lin_a = sm.lin[t][kp - z0 + 1], lin_b = sm.lin[t][kp - z0 + 2];
                    vkp = vel > p.EPS ? lin_a / (vel * p.dt) : lin_b / (-vel * p.dt);
                }
                if (km >= 1 && km < nz && km >= z0 && km < z0 + TT_H && x0 + c < nx) {
                    const T vel = sm.vel[FACE_Z + (km - z0) * TT_S + c];
                    const T lin_a = sm.lin[t][km - z0], lin_b = sm.lin[t][km - z0 + 1];
                    vkm = vel > p.EPS ? lin_a / (vel * p.dt) : lin_b / (-vel * p.dt);
                }
                sm.cl[t][0][slot][c] = vkp;
                sm.cl[t][1][slot][c] = vkm;
            }
            __syncwarp();
        }

        const int left = (mine && tx > 0) ? tile - 1 : -1;
        const bool left_done = tx == tx0 && tx0 > 0;  // the left tile belongs to the finished chunk
        const int below = (mine && tz > 0) ? tile - ctl.tiles_x : -1;
        // the left-strip values of this lane's row and the bottom strip (sm.bot) of the last
        // computation: first the stage-start values, formed as the neighbour's staging forms them
        T in_p1 = T(0), in_p2 = T(0);
        T pub[4] = {T(0), T(0), T(0), T(0)};  // this tile's published strips (stage-start values at first)
        if (mine) {
            auto s0 = [&](int kk, int ii) {
                return (kk >= 0 && kk < nz) ? a.q_old[t][MOIST_IDX(kk, ii)] / a.rho[MOIST_IDX(kk, ii)] : T(0);
            };
            if (left_done) {
                const T* ls = strip_ptr(strips, t, left, ctl.ntiles);
                const int own = row_ok;
                in_p2 = own ? __ldcg(ls + 0 * TT_W + r) : T(0);
                in_p1 = own ? __ldcg(ls + 1 * TT_W + r) : T(0);
            } else if (row_ok) {
                in_p1 = s0(k, wrapx(x0 - 1, nx));
                in_p2 = s0(k, wrapx(x0 - 2, nx));
            }
            const bool cin = below >= 0 && x0 + lane < nx + 2;
            sm.bot[t][0][lane] = cin ? s0(z0 - 2, wrapx(x0 + lane, nx)) : T(0);  // row z0-2
            sm.bot[t][1][lane] = cin ? s0(z0 - 1, wrapx(x0 + lane, nx)) : T(0);  // row z0-1
            pub[0] = sm.s[t][r][TT_W - 2];
            pub[1] = sm.s[t][r][TT_W - 1];
            pub[2] = sm.s[t][TT_H - 2][lane];
            pub[3] = sm.s[t][TT_H - 1][lane];
            __syncwarp();
        }
        // entries this tile owns: lanes 0 .. 15 the right strip's rows (full tiles), lanes 0 .. 31 the top strip's columns
        const bool own_r = !zh && row_ok && width == TT_W;
        const bool own_t0 = z0 + TT_H - 2 < nz && lane < width, own_t1 = z0 + TT_H - 1 < nz && lane < width;
        // dataflow state: the neighbours' versions used and the words read with them, the own version
        int used_lv = 0, used_bv = 0, lw_cur = 0, bw_cur = 0, my_ver = 0;
        int* const my_word = ctl.ver + (size_t)t * ctl.ntiles + (mine ? tile : 0);

        TileLane<T> L;
        L.S = &sm.s[t][r][0];
        L.Sp1 = zh ? &sm.s[t][r + 1][0] : &sm.s[t][r][1];
        L.Sp2 = zh ? &sm.s[t][r + 2][0] : &sm.s[t][r][2];
        L.vel_p = sm.vel + (zh ? FACE_Z + (r + 1) * TT_S : r * TT_S + 1);
        L.vel_m = sm.vel + (zh ? FACE_Z + r * TT_S : r * TT_S);
        L.rf_p = sm.rf + (zh ? FACE_Z + (r + 1) * TT_S : r * TT_S + 1);
        L.rf_m = sm.rf + (zh ? FACE_Z + r * TT_S : r * TT_S);
        L.q0 = &sm.q0[t][r][0];
        L.dph = &sm.dph[t][r][0];
        L.rho = &sm.rho[r][0];
        L.rrho = &sm.rrho[r][0];
        L.cl_p = sm.cl[t][0][k == 0 ? 0 : 1];
        L.cl_m = sm.cl[t][1][k == 1 ? 0 : 1];
        L.bot0 = sm.bot[t][0];
        L.bot1 = sm.bot[t][1];
        L.qn = &sm.qn[t][r][0];
        L.snp = &sm.snp[t][r][0];
        L.r = r;
        L.width = width;
        L.zh = zh;
        L.row_ok = row_ok;

        int pass = 1;
        for (;; pass++) {
            if constexpr (!DF) {
                if (pass > ctl.max_pass) break;
            }
            const int cur = pass & 1, prv = cur ^ 1;
            unsigned lmask = 0u, bmask = 0u;
            if constexpr (DF) {
                if (pass > 1) {
                    // wait until a neighbour has published a version this tile has not used (bounded)
                    const int* lwp = ctl.ver + (size_t)t * ctl.ntiles + left;
                    const int* bwp = ctl.ver + (size_t)t * ctl.ntiles + below;
                    int lw = lw_cur, bw = bw_cur;
                    const long long t0 = clock64();
                    bool df_timeout = false;
                    while (true) {
                        lw = left >= 0 ? ld_acquire(lwp) : 0;
                        bw = below >= 0 ? ld_acquire(bwp) : 0;
                        const bool news = (left >= 0 && (lw >> 1) > used_lv) || (below >= 0 && (bw >> 1) > used_bv);
                        if (__shfl_sync(0xffffffffu, (int)news, 0)) break;
                        if (__shfl_sync(0xffffffffu, (int)(clock64() - t0 > ctl.spin_limit), 0)) {
                            df_timeout = true;
                            break;
                        }
                        __nanosleep(32);
                    }
                    if (df_timeout) {
                        if (lane == 0) atomicExch(ctl.timeout, 1);
                        break;
                    }
                    lw = __shfl_sync(0xffffffffu, lw, 0);
                    bw = __shfl_sync(0xffffffffu, bw, 0);
                    // the newest strips, read from the ring slot of their version; a slot the neighbour
                    // may have begun to overwrite meanwhile (it got TT_RING - 1 versions ahead) is read again
                    T np1 = in_p1, np2 = in_p2, nb0 = sm.bot[t][0][lane], nb1 = sm.bot[t][1][lane];
                    if (left >= 0 && (lw >> 1) > used_lv) {
                        for (int tries = 0;; tries++) {
                            const int v = lw >> 1;
                            const T* ls = strip_ver_ptr(strips, t, left, v, ctl.ntiles);
                            np2 = __ldcg(ls + 0 * TT_W + r);
                            np1 = __ldcg(ls + 1 * TT_W + r);
                            const int again = __shfl_sync(0xffffffffu, ld_acquire(lwp), 0);
                            if ((again >> 1) <= v + TT_RING - 2 || tries > 1000) break;
                            lw = again;
                        }
                        used_lv = lw >> 1;
                        lw_cur = lw;
                    }
                    if (below >= 0 && (bw >> 1) > used_bv) {
                        for (int tries = 0;; tries++) {
                            const int v = bw >> 1;
                            const T* bs = strip_ver_ptr(strips, t, below, v, ctl.ntiles);
                            nb0 = __ldcg(bs + 2 * TT_W + lane);
                            nb1 = __ldcg(bs + 3 * TT_W + lane);
                            const int again = __shfl_sync(0xffffffffu, ld_acquire(bwp), 0);
                            if ((again >> 1) <= v + TT_RING - 2 || tries > 1000) break;
                            bw = again;
                        }
                        used_bv = bw >> 1;
                        bw_cur = bw;
                    }
                    auto differs = [](T x, T y) { return !(x == y || (x != x && y != y)); };
                    lmask = __ballot_sync(0xffffffffu, !zh && (differs(np1, in_p1) || differs(np2, in_p2)));
                    bmask = __ballot_sync(0xffffffffu, differs(nb0, sm.bot[t][0][lane]) || differs(nb1, sm.bot[t][1][lane]));
                    in_p1 = np1;
                    in_p2 = np2;
                    sm.bot[t][0][lane] = nb0;
                    sm.bot[t][1][lane] = nb1;
                    __syncwarp();
                }
            } else if (pass > 1) {
                // neighbours' strips and masks are written by other SMs: read them through L2 (__ldcg),
                // all at once; a strip is used only where its mask says that it was written
                const int* chg_prev = ctl.changed + ((size_t)prv * 3 + t) * ctl.ntiles * 2;
                const bool lin = left >= 0 && !left_done;
                T np1 = T(0), np2 = T(0), nb0 = T(0), nb1 = T(0);
                if (lin) {
                    const T* ls = strip_ptr(strips, t, left, ctl.ntiles);
                    lmask = (unsigned)__ldcg(chg_prev + 2 * left);
                    np2 = __ldcg(ls + 0 * TT_W + r);
                    np1 = __ldcg(ls + 1 * TT_W + r);
                }
                if (below >= 0) {
                    const T* bs = strip_ptr(strips, t, below, ctl.ntiles);
                    bmask = (unsigned)__ldcg(chg_prev + 2 * below + 1);
                    nb0 = __ldcg(bs + 2 * TT_W + lane);
                    nb1 = __ldcg(bs + 3 * TT_W + lane);
                }
                if (lmask != 0u) {
                    in_p1 = np1;
                    in_p2 = np2;
                }
                if (bmask != 0u) {
                    sm.bot[t][0][lane] = nb0;
                    sm.bot[t][1][lane] = nb1;
                    __syncwarp();
                }
            }
            const bool compute = mine && !halt && (pass == 1 || lmask != 0u || bmask != 0u);
            if (ctl.pass_ts && tx0 == 0 && pass <= ctl.max_pass) {
                if constexpr (DF) {
                    if (lane == 0) atomicMax(ctl.pass_ts + pass, globaltimer_ns());
                } else if (blockIdx.x == 0 && threadIdx.x == 0) {
                    ctl.pass_ts[pass] = globaltimer_ns();
                }
            }
            if (ctl.pass_work && tx0 == 0 && compute && lane == 0 && pass <= ctl.max_pass) atomicAdd(ctl.pass_work + pass, 1);
            unsigned rmask = 0u, tmask = 0u;
            if (compute) {
                // A cell reads four updated values: (k, i-1), (k, i-2) of its own row and (k-1, i),
                // (k-2, i) from the rows below; the stage-start values never change. Row r reads its
                // left-strip entries at steps r and r + 1, column c of the bottom strip is read at steps c
                // and c + 1: a repair starts at the first changed entry, and last_in is the last step
                // that reads one.
                const bool all = pass == 1;
                const int step0 = all ? 0 : min(lmask != 0u ? __ffs((int)lmask) - 1 : TT_W, bmask != 0u ? __ffs((int)bmask) - 1 : TT_W);
                const int last_in = all ? TT_W + TT_H : max(32 - __clz((int)lmask), 32 - __clz((int)bmask));
                const bool bad = need_cen ? tile_walk<FastDiv<T>, true>(w, L, step0, last_in, in_p1, in_p2)
                                          : tile_walk<FastDiv<T>, false>(w, L, step0, last_in, in_p1, in_p2);
                if (bad) tile_walk<IeeeDiv<T>, true>(w, L, 0, TT_W + TT_H, in_p1, in_p2);
                // the boundary strips of the values just computed; an entry the tile does not own
                // (partial tile) keeps the speculative value so it never registers a change
                T v[4];
                v[0] = own_r ? sm.snp[t][r][TT_W - 2] : pub[0];
                v[1] = own_r ? sm.snp[t][r][TT_W - 1] : pub[1];
                v[2] = own_t0 ? sm.snp[t][TT_H - 2][lane] : pub[2];
                v[3] = own_t1 ? sm.snp[t][TT_H - 1][lane] : pub[3];
                auto differs = [](T x, T y) { return !(x == y || (x != x && y != y)); };
                rmask = __ballot_sync(0xffffffffu, differs(v[0], pub[0]) || differs(v[1], pub[1]));
                tmask = __ballot_sync(0xffffffffu, differs(v[2], pub[2]) || differs(v[3], pub[3]));
                for (int q = 0; q < 4; q++) pub[q] = v[q];
            }
            if constexpr (DF) {
                // a new version when the strips changed, or when the tile became final: it computed
                // from (or is unchanged by) its neighbours' final strips
                const bool fin = (left < 0 || (lw_cur & 1)) && (below < 0 || (bw_cur & 1));
                if (rmask != 0u || tmask != 0u || fin) {
                    T* out = strip_ver_ptr(strips, t, tile, my_ver + 1, ctl.ntiles);
                    if (!zh) {
                        __stcg(out + 0 * TT_W + r, pub[0]);
                        __stcg(out + 1 * TT_W + r, pub[1]);
                    }
                    __stcg(out + 2 * TT_W + lane, pub[2]);
                    __stcg(out + 3 * TT_W + lane, pub[3]);
                    __threadfence();
                    __syncwarp();
                    my_ver++;
                    if (lane == 0) st_release(my_word, (my_ver << 1) | (fin ? 1 : 0));
                }
                if (fin || halt) break;
            } else {
                // a later chunk reads the strips of this one's last column whether they changed or not
                const bool last_col = mine && tx == tx0 + ctl.chunk_x - 1;
                if (rmask != 0u || tmask != 0u || (pass == 1 && last_col)) {
                    T* out = strip_ptr(strips, t, tile, ctl.ntiles);
                    if (!zh) {
                        __stcg(out + 0 * TT_W + r, pub[0]);
                        __stcg(out + 1 * TT_W + r, pub[1]);
                    }
                    __stcg(out + 2 * TT_W + lane, pub[2]);
                    __stcg(out + 3 * TT_W + lane, pub[3]);
                }
                // lane r: row r of the right strip, column r of the top strip
                if (mine && lane == 0) {
                    int* chg = ctl.changed + (((size_t)cur * 3 + t) * ctl.ntiles + tile) * 2;
                    __stcg(chg, (int)rmask);
                    __stcg(chg + 1, (int)tmask);
                }
                const int res = sync(ctl, nblocks, (rmask | tmask) != 0u);
                if (res < 0) return;
                if (res == 0) break;
            }
        }
        // the results (coalesced rows): this warp's own tracer
        if (mine && !halt) {
            __syncwarp();
            T* qn = a.q_new[t];
            for (int rr = 0; rr < TT_H; rr++) {
                const int kk = z0 + rr;
                if (kk < nz && lane < width) qn[MOIST_IDX(kk, x0 + lane)] = sm.qn[t][rr][lane];
            }
        }
        npass_all += pass;
        if constexpr (DF) {  // the deepest tile's count of computations, and the moment the last tile leaves
            if (lane == 0) {
                atomicMax(ctl.passes, pass);
                if (ctl.pass_ts) atomicMax(ctl.pass_ts + ctl.max_pass + 2, globaltimer_ns());
            }
        } else if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (ctl.pass_ts && tx0 == 0) ctl.pass_ts[ctl.max_pass + 2] = globaltimer_ns();  // block 0 leaves the chunk
            if (pass > ctl.max_pass) atomicMax(ctl.timeout, 2);  // no fixed point: what was written is no result
        }
        __syncthreads();  // the next chunk stages over this one's shared memory
    }
    if constexpr (!DF) {
        if (threadIdx.x == 0) {
            if (blockIdx.x == 0) {
                *ctl.passes = npass_all;
                atomicAdd(ctl.hist + (npass_all < 63 ? npass_all : 63), 1);
            }
            // the last block to leave clears the barrier words for the next launch
            if (atomicAdd(ctl.bar + 2, 1ull) == nblocks - 1) {
                ctl.bar[0] = 0;
                ctl.bar[1] = 0;
                ctl.bar[2] = 0;
            }
        }
    }
}

// histogram of the dataflow sweep's counts (diagnostic)
__global__ void k_pass_count(const int* passes, int* hist) {
    const int p = *passes;
    atomicAdd(hist + (p < 63 ? p : 63), 1);
}

}  // namespace moist
