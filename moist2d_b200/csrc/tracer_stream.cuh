// tracer_stream.cuh - the reference's in-place Gauss-Seidel tracer sweep as one exact wavefront
// per tracer, streaming the anti-diagonals of the domain through shared memory.
//
// Cell (k, i) of the in-place sweep (moist.jl:1469-1518) reads the updated values at (k, i-1),
// (k, i-2), (k-1, i), (k-2, i) and stage-start values elsewhere, so the anti-diagonals
// k + i = const can be updated together. One block sweeps one tracer of one domain: two lanes own
// row k (tracer_cell.cuh; 16 rows per warp, nz <= STREAM_MAX_ROWS) and update column c = s - k at
// step s, for s = 0 .. nx + nz - 2. No speculation, no repair passes and no grid-wide barrier:
// blocks are independent, so any number of (domain, tracer) sweeps can share one launch.
//
// The stage-start inputs are first copied by b_stream_prep into records by anti-diagonal (element
// k of record s belongs to column s - k), so that a step reads whole lines: with the fields' own
// layout every lane of a load touches another row, 32 lines a load, which bounded the sweep (2900
// cycles a step with two or three blocks of 128 rows on an SM). The block copies one record a step with
// 16-byte cp.async into a ring of shared memory, three steps before its first use. The updated
// values of the rows below come through warp shuffles, across warps through a small ring, one
// block barrier per step.
#pragma once

#include "tracer_tiles.cuh"

namespace moist {

constexpr int STREAM_MAX_ROWS = 256;  // rows per block (two threads each)
constexpr int STREAM_RING = 8;        // records in shared memory; columns kept of the two top rows of every warp

// fields of a record: the first six are the domain's, the last three the tracer's
enum { SK_VX = 0, SK_VZ, SK_RX, SK_RZ, SK_RHO, SK_RRHO, SK_ND, SK_S = 0, SK_Q0, SK_DPH, SK_NT };

// elements of one field of a record: rows -1 .. nz+1 at positions 0 .. nz+2, padded to 16 (mod 32) so that
// the two halves of a warp read two neighbouring fields on different banks
__host__ __device__ inline int skew_pitch(int nz) { return (nz + 3 + 15) / 32 * 32 + 16; }
// records s = -1 .. nx + nz + 1 (+ the ring's look-ahead)
__host__ __device__ inline size_t skew_rows(int nx, int nz) { return (size_t)nx + nz + 4 + STREAM_RING; }

template <class T>
struct StreamArgs {
    TracerArgs<T> tr;
    T* dom;      // [skew_rows][SK_ND][pitch]
    T* trc[3];   // [skew_rows][SK_NT][pitch]
};

__device__ __forceinline__ int pmod(int c, int n) {
    const int r = c % n;
    return r < 0 ? r + n : r;
}

// The records of the sweep: block (bx, by) takes columns 32 bx - 1 .. 32 bx + 30 of rows 32 by ..
// 32 by + 31 (256 threads), reads every field by rows and writes it by anti-diagonals through a
// shared tile. s = rho_q / rho (IEEE), the reciprocal of rho for quot(), face densities. Positions no
// cell of the domain has (rows -1, nz, nz+1; corners) keep the zeros of the allocation.
template <class T>
__device__ __forceinline__ void b_stream_prep(DevParams<T> p, StreamArgs<T> a, const int* err, int bx, int by) {
    __shared__ T tile[32][34];  // stride 34: a column of an anti-diagonal touches every bank once
    if (halted(err)) return;  // the same for every thread of the launch
    const int nx = p.nx, nz = p.nz, P = p.P, np = skew_pitch(nz);
    const int lane = threadIdx.x & 31, wid = (threadIdx.x + threadIdx.y * blockDim.x) >> 5, nw = (blockDim.x * blockDim.y) >> 5;
    const int c0 = 32 * bx - 1, k0 = 32 * by;
    // one field: val(k, i) at the periodic column i of cells (k, c) with c in [c_lo, c_hi]
    auto field = [&](T* out, int nf, int f, int c_lo, int c_hi, int rows, auto val) {
        for (int r = wid; r < 32; r += nw) {
            const int k = k0 + r, c = c0 + lane;
            tile[r][lane] = (k < rows && c >= c_lo && c <= c_hi) ? val(k, pmod(c, nx)) : T(0);
        }
        __syncthreads();
        for (int d = wid; d < 63; d += nw) {  // anti-diagonal d of the tile: rows r with column d - r
            const int cc = d - lane, k = k0 + lane, c = c0 + cc;
            if (cc >= 0 && cc < 32 && k < rows && c >= c_lo && c <= c_hi)
                out[((size_t)(c + k + 1) * nf + f) * np + k + 1] = tile[lane][cc];
        }
        __syncthreads();
    };
    const T* rho = a.tr.rho;
    field(a.dom, SK_ND, SK_VX, -1, nx - 1, nz, [&](int k, int i) { return a.tr.mfx[MOIST_IDX(k, i)]; });
    field(a.dom, SK_ND, SK_VZ, 0, nx - 1, nz - 1, [&](int k, int i) { return a.tr.mfz[MOIST_IDX(k, i)]; });
    field(a.dom, SK_ND, SK_RX, -1, nx - 1, nz,
          [&](int k, int i) { return (rho[MOIST_IDX(k, wrapx(i + 1, nx))] + rho[MOIST_IDX(k, i)]) * T(0.5); });
    field(a.dom, SK_ND, SK_RZ, 0, nx - 1, nz - 1,
          [&](int k, int i) { return f2h(rho[MOIST_IDX(k + 1, i)], rho[MOIST_IDX(k, i)], p.dz[k + 1], p.dz[k]); });
    field(a.dom, SK_ND, SK_RHO, 0, nx - 1, nz, [&](int k, int i) { return rho[MOIST_IDX(k, i)]; });
    field(a.dom, SK_ND, SK_RRHO, 0, nx - 1, nz, [&](int k, int i) { return FastDiv<T>::prep1(rho[MOIST_IDX(k, i)]); });
    for (int t = 0; t < 3; t++) {
        field(a.trc[t], SK_NT, SK_S, 0, nx + 1, nz,
              [&](int k, int i) { return a.tr.q_old[t][MOIST_IDX(k, i)] / rho[MOIST_IDX(k, i)]; });
        field(a.trc[t], SK_NT, SK_Q0, 0, nx - 1, nz, [&](int k, int i) { return a.tr.q0[t][MOIST_IDX(k, i)]; });
        field(a.trc[t], SK_NT, SK_DPH, 0, nx - 1, nz, [&](int k, int i) { return a.tr.dphys[t][MOIST_IDX(k, i)]; });
    }
}
template <class T>
__global__ void __launch_bounds__(256) k_stream_prep(DevParams<T> p, StreamArgs<T> a, const int* err) {
    b_stream_prep(p, a, err, blockIdx.x, blockIdx.y);
}

__device__ __forceinline__ void cp_async16(void* s, const void* g) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(s);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(g) : "memory");
}

// shared memory of one sweep: the ring of records, then the updated values of the two top rows of
// every warp ([2][warps][STREAM_RING])
template <class T>
__host__ __device__ inline size_t stream_smem_bytes(int nz) {
    return ((size_t)STREAM_RING * (SK_ND + SK_NT) * skew_pitch(nz) + 2 * ((nz + WROWS - 1) / WROWS) * STREAM_RING) * sizeof(T);
}
inline int stream_threads(int nz) { return (nz + WROWS - 1) / WROWS * 32; }

// one tracer t of one domain; blockDim.x = stream_threads(nz) or more. Returns (to every thread)
// whether the fast division refused an operand or a result is not finite.
template <class D, class T>
__device__ __forceinline__ bool stream_sweep(const DevParams<T>& p, const StreamArgs<T>& a, int t, T* smem) {
    const int nx = p.nx, nz = p.nz, P = p.P, np = skew_pitch(nz);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nwarp = (nz + WROWS - 1) / WROWS;
    const int r = lane & (WROWS - 1), k = WROWS * wid + r;
    const bool zh = lane >= WROWS, row_ok = k < nz;
    const int recd = SK_ND * np, rect = SK_NT * np, rec = recd + rect;
    T* top1 = smem + (size_t)STREAM_RING * rec;  // [warp][STREAM_RING]: row 16w+15
    T* top2 = top1 + nwarp * STREAM_RING;        // row 16w+14
    const T* gd = a.dom;
    const T* gt = a.trc[t];
    constexpr int EPC = 16 / sizeof(T);  // elements per 16-byte copy
    // record s (>= -1) into its slot of the ring; every thread commits one group per call
    auto issue = [&](int s) {
        T* dst = smem + (size_t)((s + 1) & (STREAM_RING - 1)) * rec;
        const T* sd = gd + (size_t)(s + 1) * recd;
        const T* st = gt + (size_t)(s + 1) * rect;
        for (int j = threadIdx.x; j < recd / EPC; j += blockDim.x) cp_async16(dst + j * EPC, sd + j * EPC);
        for (int j = threadIdx.x; j < rect / EPC; j += blockDim.x) cp_async16(dst + recd + j * EPC, st + j * EPC);
        cp_async_commit();
    };
    const HalfRow<T> w = half_row(p, k, zh, a.tr.dt);
    const T* qo = a.tr.q_old[t];
    const T lin_km1 = (k - 1 >= 0 && k - 1 < nz) ? qo[MOIST_IDX(k - 1, nx - 2)] : T(0);
    const T lin_k = row_ok ? qo[MOIST_IDX(k, nx - 2)] : T(0);
    const T lin_kp1 = (k + 1 < nz) ? qo[MOIST_IDX(k + 1, nx - 2)] : T(0);
    // this half's clamp rows (z half only)
    const bool clamp_p = zh && row_ok && (k == 0 || k == nz - 2) && k < nz - 1;
    const bool clamp_m = zh && row_ok && (k == 1 || k == nz - 1) && k >= 1;
    // the updated values of the two columns to the left; the seam reads the stage-start values
    T prev1 = row_ok ? qo[MOIST_IDX(k, nx - 1)] / a.tr.rho[MOIST_IDX(k, nx - 1)] : T(0);
    T prev2 = row_ok ? qo[MOIST_IDX(k, nx - 2)] / a.tr.rho[MOIST_IDX(k, nx - 2)] : T(0);
    T sn_last = T(0), m1_used = T(0);
    T* qn = a.tr.q_new[t] + (size_t)(row_ok ? k : 0) * P;
    const int z = zh ? 1 : 0, ki = min(k, nz - 1);  // the last warp's rows beyond the domain read row nz-1's inputs
    const int o_v = (zh ? SK_VZ : SK_VX) * np + ki + 1, o_r = (zh ? SK_RZ : SK_RX) * np + ki + 1;
    const int o_rho = SK_RHO * np + ki + 1, o_rr = SK_RRHO * np + ki + 1;
    const int o_s = recd + SK_S * np + ki + 1, o_q = recd + SK_Q0 * np + ki + 1, o_d = recd + SK_DPH * np + ki + 1;
    const bool in = wid < nwarp;  // warps beyond the rows only copy and meet the barrier
    bool bad_any = false;
    struct Ops {
        T sc, p1, p2, vp, vm, rp, rm, q0, dph, rho, rrho;
    };
    auto load = [&](int s) {  // the operands of step s (records s - 1 .. s + 2)
        auto R = [&](int j) { return smem + (size_t)((j + 1) & (STREAM_RING - 1)) * rec; };
        const T *R0 = R(s), *Rm = R(s - 1);
        Ops o;
        o.sc = R0[o_s];
        o.p1 = R(s + 1)[o_s + z];
        o.p2 = R(s + 2)[o_s + 2 * z];
        o.vp = R0[o_v];
        o.vm = Rm[o_v - z];
        o.rp = R0[o_r];
        o.rm = Rm[o_r - z];
        o.q0 = R0[o_q];
        o.dph = R0[o_d];
        o.rho = R0[o_rho];
        o.rrho = R0[o_rr];
        return o;
    };

    const int nsteps = nx + nz - 1;
    for (int s = -1; s <= STREAM_RING - 3; s++) issue(s);
    cp_async_wait<STREAM_RING - 5>();  // records up to 2
    __syncthreads();
    Ops nxt = load(0);
    for (int step = 0; step < nsteps; step++) {
        // records up to step + 3 have landed (the next step's operands, read one step ahead); the slot of record
        // step - 2, which nobody reads any more, takes record step + 6 (records beyond the last are allocated)
        cp_async_wait<STREAM_RING - 6>();
        __syncthreads();
        issue(step + STREAM_RING - 2);
        if (!in) continue;
        const int c = step - k;
        const bool active = row_ok && c >= 0 && c < nx;
        const Ops o = nxt;
        nxt = load(step + 1);
        // neighbours: row k-1 stands one column ahead
        const T up_sn = __shfl_up_sync(0xffffffffu, sn_last, 1);
        const T up_m1 = __shfl_up_sync(0xffffffffu, m1_used, 1);
        const int slot = c & (STREAM_RING - 1);
        const T t1 = wid > 0 ? top1[(wid - 1) * STREAM_RING + slot] : T(0);
        const T t2 = wid > 0 ? top2[(wid - 1) * STREAM_RING + slot] : T(0);
        const T m1 = zh ? (r == 0 ? t1 : up_sn) : prev1;
        const T m2 = zh ? (r == 0 ? t2 : (r == 1 ? t1 : up_m1)) : prev2;
        T q, sn;
        bool bad = false;
        if (__any_sync(0xffffffffu, active && (clamp_p || clamp_m || !(fabs(o.vp) > w.EPS) || !(fabs(o.vm) > w.EPS)))) {
            // the clamp quotients of limited_flux_z, on the four rows that can use them
            T cl_p = T(0), cl_m = T(0);
            if (clamp_p) cl_p = o.vp > w.EPS ? lin_k / (o.vp * p.dt) : lin_kp1 / (-o.vp * p.dt);
            if (clamp_m) cl_m = o.vm > w.EPS ? lin_km1 / (o.vm * p.dt) : lin_k / (-o.vm * p.dt);
            two_lane_cell<D, true>(w, m2, m1, o.sc, o.p1, o.p2, o.vp, o.vm, o.rp, o.rm, cl_p, cl_m, o.q0, o.dph, o.rho,
                                   o.rrho, q, sn, bad);
        } else {
            two_lane_cell<D, false>(w, m2, m1, o.sc, o.p1, o.p2, o.vp, o.vm, o.rp, o.rm, T(0), T(0), o.q0, o.dph, o.rho,
                                    o.rrho, q, sn, bad);
        }
        bad_any |= bad && active;
        if (active && !zh) {
            qn[c] = q;
            if (r == WROWS - 1) top1[wid * STREAM_RING + slot] = sn;
            if (r == WROWS - 2) top2[wid * STREAM_RING + slot] = sn;
        }
        prev2 = active ? prev1 : prev2;
        prev1 = active ? sn : prev1;
        // lane r+1 reads these next step only for the column it shares with this step
        sn_last = sn;
        m1_used = m1;
    }
    cp_async_wait<0>();
    return __syncthreads_or(bad_any) != 0;
}

// tracer t of one domain
template <class T>
__device__ __forceinline__ void b_tracer_stream(const DevParams<T>& p, const StreamArgs<T>& a, const int* err, int t) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (halted(err)) return;
    T* sm = reinterpret_cast<T*>(smem_raw);
    if (stream_sweep<FastDiv<T>>(p, a, t, sm)) stream_sweep<IeeeDiv<T>>(p, a, t, sm);
}

// single domain: block t sweeps tracer t
template <class T>
__global__ void __launch_bounds__(2 * STREAM_MAX_ROWS) k_tracer_stream(DevParams<T> p, StreamArgs<T> a, const int* err) {
    b_tracer_stream(p, a, err, blockIdx.x);
}

}  // namespace moist
