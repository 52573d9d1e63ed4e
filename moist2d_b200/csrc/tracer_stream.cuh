// tracer_stream.cuh - the reference's in-place Gauss-Seidel tracer sweep as one exact wavefront
// per tracer, streaming the anti-diagonals of the domain through shared memory.
//
// Cell (k, i) of the in-place sweep (moist.jl:1469-1518) reads the updated values at (k, i-1),
// (k, i-2), (k-1, i), (k-2, i) and stage-start values elsewhere, so the anti-diagonals
// k + i = const can be updated together. One block sweeps one tracer of one domain: warp g owns rows
// 16 g .. 16 g + 15 (two lanes a row, tracer_cell.cuh; nz <= STREAM_MAX_ROWS), row 16 g + r at column
// j - r in its step j = 0 .. nx + 14. No speculation, no repair passes and no grid-wide barrier:
// blocks are independent, so any number of (domain, tracer) sweeps can share one launch.
//
// The stage-start inputs are first copied by b_stream_prep into records by row group and
// anti-diagonal (the element of row k in record s belongs to column s - k), so that a step reads
// whole lines: with the fields' own layout every lane of a load touches another row, 32 lines a
// load, which bounded the sweep. A warp copies its own records with 16-byte cp.async into its own
// ring of shared memory, four steps ahead. It depends on the warp below alone, through the updated
// values of that warp's two top rows: they pass through a ring of shared memory, with counts of the
// columns done and used, read and written every STREAM_HAND steps. (With one block barrier a step,
// and a whole block copying each record, a step took 2500 cycles, of which the cell takes about 500: the
// slowest warp, and the copies' and the barrier's instructions, for every warp: 10.7 ms of a step of 64
// members, 6.9 this way.) Waits on a count are bounded and report through the error words.
#pragma once

#include "tracer_tiles.cuh"

namespace moist {

constexpr int STREAM_MAX_ROWS = 256;  // rows per block (two threads each)
constexpr int STREAM_RING = 8;        // records of a warp in shared memory
constexpr int STREAM_HAND = 8;        // steps between two exchanges of counts with the neighbouring warps
constexpr int STREAM_TOP = 64;        // columns of a warp's top rows kept for the warp above
constexpr int SK_ROWS = 20;           // rows 16 g - 1 .. 16 g + 17 of a group at positions 0 .. 18

// fields of a record: the first six are the domain's, the last three the tracer's
enum { SK_VX = 0, SK_VZ, SK_RX, SK_RZ, SK_RHO, SK_RRHO, SK_ND, SK_S = 0, SK_Q0, SK_DPH, SK_NT };

__host__ __device__ inline int stream_groups(int nz) { return (nz + WROWS - 1) / WROWS; }
// records of a group: anti-diagonals 16 g - 1 .. 16 g + nx + 17 and the ring's look-ahead
__host__ __device__ inline int skew_records(int nx) { return nx + 19 + STREAM_RING + 2; }
__host__ __device__ inline size_t skew_elems(int nx, int nz) { return (size_t)stream_groups(nz) * skew_records(nx) * SK_ROWS; }

template <class T>
struct StreamArgs {
    TracerArgs<T> tr;
    T* dom;      // [group][record][SK_ND][SK_ROWS]
    T* trc[3];   // [group][record][SK_NT][SK_ROWS]
    long long spin_limit;  // bound of a wait for a neighbouring warp, in SM clock cycles
};

__device__ __forceinline__ int pmod(int c, int n) {
    const int r = c % n;
    return r < 0 ? r + n : r;
}

// The records of the sweep: block (bx, by) takes columns 32 bx - 1 .. 32 bx + 30 of rows 32 by ..
// 32 by + 31 (256 threads), reads every field by rows and writes it by anti-diagonals through
// shared tiles, SK_BATCH fields between two barriers. s = rho_q / rho (IEEE), the reciprocal of rho for
// quot(), face densities. A group also holds its neighbours' rows that its cells read: s of the
// two rows above, the vertical fluxes and densities of the row below. Positions no cell of the domain has
// (rows -1, nz, nz+1; corners) keep the zeros of the allocation.
constexpr int SK_BATCH = 3;
template <class T>
__device__ __forceinline__ void b_stream_prep(DevParams<T> p, StreamArgs<T> a, const int* err, int bx, int by) {
    __shared__ T tile[SK_BATCH][32][34];  // stride 34: a column of an anti-diagonal touches every bank once
    if (halted(err)) return;  // the same for every thread of the launch
    const int nx = p.nx, nz = p.nz, P = p.P, nrec = skew_records(nx);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int c0 = 32 * bx - 1, k0 = 32 * by;
    struct Field {
        T* out;
        int nf, f, c_lo, c_hi, rows, up, dn;  // up / dn: rows of the group above / below that the record repeats
    };
    // fields f[0 .. SK_BATCH): val(q, k, i) at the periodic column i of cells (k, c), c in [c_lo, c_hi], k < rows
    auto fields = [&](const Field (&f)[SK_BATCH], auto val) {
        for (int r = wid; r < 32; r += nw) {
            const int k = k0 + r, c = c0 + lane, i = pmod(c, nx);
#pragma unroll
            for (int q = 0; q < SK_BATCH; q++)
                tile[q][r][lane] = (k < f[q].rows && c >= f[q].c_lo && c <= f[q].c_hi) ? val(q, k, i) : T(0);
        }
        __syncthreads();
        const int k = k0 + lane, g = k / WROWS, r = k - g * WROWS;
        for (int d = wid; d < 63; d += nw) {  // anti-diagonal d of the tile: rows with column d - row
            const int cc = d - lane, c = c0 + cc, s = c + k;
            if (cc < 0 || cc >= 32) continue;
#pragma unroll
            for (int q = 0; q < SK_BATCH; q++) {
                if (!(k < f[q].rows && c >= f[q].c_lo && c <= f[q].c_hi)) continue;
                const T v = tile[q][lane][cc];
                auto put = [&](int gg) {  // into group gg's record of anti-diagonal s
                    f[q].out[(((size_t)gg * nrec + (s - WROWS * gg + 1)) * f[q].nf + f[q].f) * SK_ROWS + k - WROWS * gg + 1] = v;
                };
                put(g);
                if (r < f[q].up && g > 0) put(g - 1);
                if (r >= WROWS - f[q].dn && WROWS * (g + 1) < nz) put(g + 1);
            }
        }
        __syncthreads();
    };
    const T* rho = a.tr.rho;
    {
        const Field f[SK_BATCH] = {{a.dom, SK_ND, SK_VX, -1, nx - 1, nz, 0, 0},
                                   {a.dom, SK_ND, SK_VZ, 0, nx - 1, nz - 1, 0, 1},
                                   {a.dom, SK_ND, SK_RX, -1, nx - 1, nz, 0, 0}};
        fields(f, [&](int q, int k, int i) {
            const size_t c = MOIST_IDX(k, i);
            return q == 0 ? a.tr.mfx[c]
                          : q == 1 ? a.tr.mfz[c] : (rho[MOIST_IDX(k, wrapx(i + 1, nx))] + rho[c]) * T(0.5);
        });
    }
    {
        const Field f[SK_BATCH] = {{a.dom, SK_ND, SK_RZ, 0, nx - 1, nz - 1, 0, 1},
                                   {a.dom, SK_ND, SK_RHO, 0, nx - 1, nz, 0, 0},
                                   {a.dom, SK_ND, SK_RRHO, 0, nx - 1, nz, 0, 0}};
        fields(f, [&](int q, int k, int i) {
            const size_t c = MOIST_IDX(k, i);
            return q == 0 ? f2h(rho[c + P], rho[c], p.dz[k + 1], p.dz[k]) : q == 1 ? rho[c] : FastDiv<T>::prep1(rho[c]);
        });
    }
    for (int t = 0; t < 3; t++) {
        const Field f[SK_BATCH] = {{a.trc[t], SK_NT, SK_S, 0, nx + 1, nz, 2, 0},
                                   {a.trc[t], SK_NT, SK_Q0, 0, nx - 1, nz, 0, 0},
                                   {a.trc[t], SK_NT, SK_DPH, 0, nx - 1, nz, 0, 0}};
        fields(f, [&](int q, int k, int i) {
            const size_t c = MOIST_IDX(k, i);
            return q == 0 ? a.tr.q_old[t][c] / rho[c] : q == 1 ? a.tr.q0[t][c] : a.tr.dphys[t][c];
        });
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

// shared memory of one sweep: per warp its ring of records, the updated values of its two top rows
// ([2][STREAM_TOP]) and two counts: columns done by its top row, steps begun
constexpr int SK_REC = (SK_ND + SK_NT) * SK_ROWS;  // elements of a record
template <class T>
__host__ __device__ inline size_t stream_smem_bytes(int nz) {
    return (size_t)stream_groups(nz) * ((STREAM_RING * SK_REC + 2 * STREAM_TOP) * sizeof(T) + 2 * sizeof(int));
}
inline int stream_threads(int nz) { return stream_groups(nz) * 32; }

// one tracer t of one domain; blockDim.x = stream_threads(nz) or more. Returns (to every thread)
// whether the fast division refused an operand or a result is not finite.
template <class D, class T>
__device__ __forceinline__ bool stream_sweep(const DevParams<T>& p, const StreamArgs<T>& a, int t, T* smem, int* timeout) {
    const int nx = p.nx, nz = p.nz, P = p.P;
    const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, ng = stream_groups(nz);
    T* const ring = smem + (size_t)g * (STREAM_RING * SK_REC);
    T* const tops = smem + (size_t)ng * (STREAM_RING * SK_REC);
    volatile int* const done = reinterpret_cast<volatile int*>(tops + (size_t)ng * 2 * STREAM_TOP);  // [ng], then begun [ng]
    volatile int* const begun = done + ng;
    if (g < ng && lane == 0) {
        done[g] = 0;
        begun[g] = 0;
    }
    __syncthreads();
    bool bad_any = false;
    if (g < ng) {
        const int r = lane & (WROWS - 1), k = WROWS * g + r;
        const bool zh = lane >= WROWS, row_ok = k < nz;
        T* const top_out = tops + (size_t)g * 2 * STREAM_TOP;                       // row 15, then row 14
        const T* const top_in = tops + (size_t)(g > 0 ? g - 1 : 0) * 2 * STREAM_TOP;
        // 16-byte copies: this lane's chunks lane and lane + 32 of a record (domain part, then tracer part)
        constexpr int EPC = 16 / sizeof(T), CD = SK_ND * SK_ROWS / EPC, CR = SK_REC / EPC;
        static_assert(CR <= 96, "three chunks a lane at most");
        const T* gd = a.dom + (size_t)g * skew_records(nx) * (SK_ND * SK_ROWS);
        const T* gt = a.trc[t] + (size_t)g * skew_records(nx) * (SK_NT * SK_ROWS);
        const T* src[3];
        int inc[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            const int ch = lane + 32 * q;
            src[q] = ch < CD ? gd + ch * EPC : gt + (ch - CD) * EPC;
            inc[q] = ch < CD ? SK_ND * SK_ROWS : SK_NT * SK_ROWS;
        }
        auto issue = [&](int slot) {  // the next record into a slot; one group
            T* dst = ring + slot * SK_REC + lane * EPC;
#pragma unroll
            for (int q = 0; q < (CR + 31) / 32; q++)
                if (lane + 32 * q < CR) {
                    cp_async16(dst + 32 * q * EPC, src[q]);
                    src[q] += inc[q];
                }
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
        const bool edge = clamp_p || clamp_m || (zh && row_ok && (k == 0 || k == nz - 1));
        const int clamp_g = (nz - 2) / WROWS;  // rows nz-2 and nz-1 lie in this group and above
        // the updated values of the two columns to the left; the seam reads the stage-start values
        T prev1 = row_ok ? qo[MOIST_IDX(k, nx - 1)] / a.tr.rho[MOIST_IDX(k, nx - 1)] : T(0);
        T prev2 = row_ok ? qo[MOIST_IDX(k, nx - 2)] / a.tr.rho[MOIST_IDX(k, nx - 2)] : T(0);
        T sn_last = T(0), m1_used = T(0);
        T* qn = a.tr.q_new[t] + (size_t)(row_ok ? k : 0) * P;
        const int z = zh ? 1 : 0;
        const int o_v = (zh ? SK_VZ : SK_VX) * SK_ROWS + r + 1, o_r = (zh ? SK_RZ : SK_RX) * SK_ROWS + r + 1;
        const int o_s = (SK_ND + SK_S) * SK_ROWS + r + 1;
        struct Ops {
            T sc, p1, p2, vp, vm, rp, rm, q0, dph, rho, rrho, cl_p, cl_m;
            bool cen;
        };
        auto load = [&](int j) {  // the operands of step j (records j .. j + 3)
            auto R = [&](int i) { return ring + (i & (STREAM_RING - 1)) * SK_REC; };
            const T *Rm = R(j), *R0 = R(j + 1);
            Ops o;
            o.sc = R0[o_s];
            o.p1 = R(j + 2)[o_s + z];
            o.p2 = R(j + 3)[o_s + 2 * z];
            o.vp = R0[o_v];
            o.vm = Rm[o_v - z];
            o.rp = R0[o_r];
            o.rm = Rm[o_r - z];
            o.q0 = R0[(SK_ND + SK_Q0) * SK_ROWS + r + 1];
            o.dph = R0[(SK_ND + SK_DPH) * SK_ROWS + r + 1];
            o.rho = R0[SK_RHO * SK_ROWS + r + 1];
            o.rrho = R0[SK_RRHO * SK_ROWS + r + 1];
            // the clamp quotients of limited_flux_z, on the four rows that can use them, and whether a cell of
            // the step needs the centred face values: a step ahead, off the chain
            const bool act = row_ok && j >= r && j - r < nx;
            o.cl_p = o.cl_m = T(0);
            o.cen = __any_sync(0xffffffffu, act && (edge || !(fabs(o.vp) > w.EPS) || !(fabs(o.vm) > w.EPS)));
            if (o.cen && (g == 0 || g >= clamp_g)) {
                // selected only where |vel| > EPS; IEEE division here, whose quotients of zero and tiny water take
                // its slow path, made the two warps with clamp rows twice as slow as the others
                bool bad_p = false, bad_m = false;
                const T up_p = o.vp > w.EPS ? lin_k : lin_kp1, up_m = o.vm > w.EPS ? lin_km1 : lin_k;
                o.cl_p = D::quot_var(up_p, fabs(o.vp) * p.dt, bad_p);
                o.cl_m = D::quot_var(up_m, fabs(o.vm) * p.dt, bad_m);
                bad_any |= act && ((clamp_p && bad_p && fabs(o.vp) > w.EPS) || (clamp_m && bad_m && fabs(o.vm) > w.EPS));
            }
            return o;
        };
        // lane 0 waits until *count reaches least (bounded); false: it did not
        auto wait = [&](const volatile int* count, int least) {
            int ok = 1;
            if (lane == 0 && *count < least) {
                const long long t0 = clock64();
                while (*count < least)
                    if (clock64() - t0 > a.spin_limit) {
                        ok = 0;
                        atomicExch(timeout, 1);
                        break;
                    }
            }
            ok = __shfl_sync(0xffffffffu, ok, 0);
            __threadfence_block();  // the values counted are read after the count
            return ok != 0;
        };
        for (int i = 0; i < STREAM_RING; i++) issue(i);
        cp_async_wait<4>();  // records up to 3
        __syncwarp();
        Ops nxt = load(0);
        const int nsteps = nx + WROWS - 1;
        for (int j = 0; j < nsteps; j++) {
            if ((j & (STREAM_HAND - 1)) == 0) {
                // columns below j - 14 are done by the top row; the warp above may need them, the warp below must
                // have done the columns of this round, the warp above used those that it overwrites
                __syncwarp();
                if (lane == 0) {
                    __threadfence_block();
                    done[g] = min(max(j - (WROWS - 1), 0), nx);
                    begun[g] = j;
                }
                if (g > 0 && !wait(done + g - 1, min(j + STREAM_HAND, nx))) break;
                if (g + 1 < ng && !wait(begun + g + 1, min(j + STREAM_HAND - (WROWS - 2) - STREAM_TOP + 2, nx))) break;
            }
            const Ops o = nxt;
            __syncwarp();  // every lane has read record j
            issue(j & (STREAM_RING - 1));
            cp_async_wait<4>();  // records up to j + 4
            __syncwarp();
            nxt = load(j + 1);
            const int c = j - r;
            const bool active = row_ok && c >= 0 && c < nx;
            // neighbours: row k-1 stands one column ahead
            const T up_sn = __shfl_up_sync(0xffffffffu, sn_last, 1);
            const T up_m1 = __shfl_up_sync(0xffffffffu, m1_used, 1);
            const int slot = c & (STREAM_TOP - 1);
            const T t1 = g > 0 ? top_in[slot] : T(0);
            const T t2 = g > 0 ? top_in[STREAM_TOP + slot] : T(0);
            const T m1 = zh ? (r == 0 ? t1 : up_sn) : prev1;
            const T m2 = zh ? (r == 0 ? t2 : (r == 1 ? t1 : up_m1)) : prev2;
            T q, sn;
            bool bad = false;
            if (o.cen)
                two_lane_cell<D, true>(w, m2, m1, o.sc, o.p1, o.p2, o.vp, o.vm, o.rp, o.rm, o.cl_p, o.cl_m, o.q0, o.dph,
                                       o.rho, o.rrho, q, sn, bad);
            else
                two_lane_cell<D, false>(w, m2, m1, o.sc, o.p1, o.p2, o.vp, o.vm, o.rp, o.rm, T(0), T(0), o.q0, o.dph,
                                        o.rho, o.rrho, q, sn, bad);
            bad_any |= bad && active;
            if (active && !zh) {
                qn[c] = q;
                if (r >= WROWS - 2) top_out[(WROWS - 1 - r) * STREAM_TOP + slot] = sn;
            }
            prev2 = active ? prev1 : prev2;
            prev1 = active ? sn : prev1;
            // lane r+1 reads these next step only for the column it shares with this step
            sn_last = sn;
            m1_used = m1;
        }
        __syncwarp();
        if (lane == 0) {
            __threadfence_block();
            done[g] = nx;
            begun[g] = INT_MAX;
        }
        cp_async_wait<0>();
    }
    return __syncthreads_or(bad_any) != 0;
}

// tracer t of one domain
template <class T>
__device__ __forceinline__ void b_tracer_stream(const DevParams<T>& p, const StreamArgs<T>& a, const int* err, int t) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    if (halted(err)) return;
    T* sm = reinterpret_cast<T*>(smem_raw);
    int* timeout = const_cast<int*>(err) + 2;
    if (stream_sweep<FastDiv<T>>(p, a, t, sm, timeout)) stream_sweep<IeeeDiv<T>>(p, a, t, sm, timeout);
}

// single domain: block t sweeps tracer t
template <class T>
__global__ void __launch_bounds__(2 * STREAM_MAX_ROWS) k_tracer_stream(DevParams<T> p, StreamArgs<T> a, const int* err) {
    b_tracer_stream(p, a, err, blockIdx.x);
}

}  // namespace moist
