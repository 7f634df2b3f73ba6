// Newton iteration of instances whose effective band does not fit in shared memory (a 3D frame
// of a few thousand dofs and a bandwidth of a few hundred: ~10-30 MB, resident in the 126 MB L2).
//
//   large_assemble_kernel  one warp per band row: K of gather_kernel, C, the
//                          effective entries K + a1 C + a0 M written to the global band, the row's
//                          residual P - F_int - C v - M a (transient_nonlinear.mojo:2302-2356,
//                          linear_solver_backend.mojo:1877-1983)
//   large_factor_kernel    cooperative (all CTAs co-resident): blocked right-looking band LU with
//                          partial pivoting, panel width kPanel, the right-hand side carried as
//                          one more column.  CTA 0 factors the panel in shared memory; every CTA
//                          then takes column tiles of the trailing block (the panel's row
//                          interchanges, then the eliminations in column order).  Two one-way
//                          signals per panel, each waited for a bounded number of polls.
//   large_solve_kernel     one CTA per instance: blocked back substitution through U, then the
//                          displacement update and the convergence test shared with the
//                          shared-memory path.
//
// Strut's BandGeneral factorises without pivoting and, at the first column whose pivot test
// fails (a sub-diagonal entry larger than the pivot, linear_solver_backend.mojo:631-680),
// restarts from the original matrix with a dense partial-pivot LU (175-240).  The columns
// before that one choose no interchange under partial pivoting either (the same strict test,
// the first largest entry wins), so one partial-pivot factorisation performs the reference's
// interchanges and eliminations on every entry; it needs only the band, because below the
// band the dense matrix's columns are zero (rows never come from further than bw below) and
// the pivot rows' fill stays within 2 bw of the diagonal (storage: columns i - bw .. i + 2 bw
// of row i, 3 bw + 1 slots).  A factorisation that interchanged rows counts as a dense
// fallback in the statistics.  The order of the subtractions on an entry is the reference's
// (column by column); the substitution through U is blocked, so the GPU agrees with the
// oracle to rounding.
#pragma once

#include "solver_kernels.cuh"

namespace strut {

constexpr int kPanel = 32;         // panel width of the blocked band LU
constexpr int kLargeThreads = 384; // threads of a factorisation CTA (one per panel row)
// The variant for wider bands: 16-column panels and 640 threads (the panel rows halve,
// so more of them fit a CTA's shared memory).  Every entry receives the same subtractions in the same column order
// with either variant, so their results are the same bit for bit.
constexpr int kPanelWide = 16;
constexpr int kLargeThreadsWide = 640;
constexpr int kSolveThreads = 1024;
constexpr int kSolveAhead = 8;     // columns a lane of the substitution fetches a block ahead

constexpr int kColTile = 16;       // trailing-update columns per tile
// Variants for half bands up to 96 and 160 (15 and 25 nodes a floor): 128 and 192 threads, so few warps that
// every one looks through the whole column by itself and a panel column needs one barrier
// instead of two of twelve warps; 8-column tiles, which double the CTAs of the trailing update.
// Against 384 threads: n = 3000, half band 155 (8 steps) 87.4 -> 81.0 ms; n = 768, half band 101 12.6
// -> 11.6 ms.  Every warp's look through the column grows with the square of the warps.
constexpr int kLargeThreadsNarrow = 128;
constexpr int kLargeThreadsMid = 192;
constexpr int kColTileNarrow = 8;
enum { LSTAT_OK = 0, LSTAT_SINGULAR = 2, LSTAT_CONVERGED = 7, LSTAT_IDLE = -1 };

struct GridBarrier {
    unsigned int done;   // CTAs other than 0 that are through with a panel, over all panels
    unsigned int panel;  // panels that CTA 0 has published, times two, plus one if it is singular
    int err;
    int limit;  // polls a waiting CTA makes before it gives up (strut_gpu_set_wait_limit)
};

constexpr int kBarrierPolls = 1 << 22;

// The CTAs of the cooperative factorisation hand each other two words, both reset before each
// launch: CTA 0 publishes a panel, the others count themselves off when they are through with its
// columns and go on to wait for the next; only CTA 0 waits for the count.  One way each, where a
// barrier of all costs two trips through L2 for the arrival and the reset and one for the release
// (2,700 cycles a barrier).  A wait makes gb->limit polls at most, then it records an error and
// the CTA stops; the others run out in turn.
__device__ __forceinline__ unsigned int ld_acquire(const unsigned int* p) {
    unsigned int v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Thread 0 polls until ready(word); the CTA gets the word.  False once the wait was given up.
template <class Ready>
__device__ __forceinline__ bool await_word(GridBarrier* gb, const unsigned int* p, unsigned int* s_word, Ready ready) {
    int ok = 1;
    if (threadIdx.x == 0) {
        const int limit = *(volatile int*)&gb->limit;
        int polls = 0;
        unsigned int v = ld_acquire(p);
        while (!ready(v)) {
            if (++polls > limit || ((polls & 63) == 0 && *(volatile int*)&gb->err != 0)) {
                atomicExch(&gb->err, 1);
                ok = 0;
                break;
            }
            v = ld_acquire(p);
        }
        __threadfence();
        *s_word = v;
    }
    return __syncthreads_and(ok) != 0;
}

// Slot of (i, j) in the factorisation band: row i holds columns i - bw .. i + 2 bw.
__device__ __forceinline__ long long lslot(int lrw, int bw, int i, int j) {
    return (long long)i * lrw + (j - i + bw);
}

// ---- assembly and residual ---------------------------------------------------------------

// grid.x: warps over the rows of all large instances (row r of the concatenation over
// large_list).  mode INST_MODE_NEWTON skips inactive instances; INST_MODE_EXPORT also writes the
// band and F_int to the export buffers.  The residual is also written to wbuf, the column the
// factorisation carries along.
__global__ void __launch_bounds__(256) large_assemble_kernel(const DevInst* __restrict__ insts,
                                                             InstArrays A, const int* __restrict__ large_list,
                                                             const int* __restrict__ row_base,
                                                             int n_large, int total_rows, int mode,
                                                             GridBarrier* gb, double* __restrict__ wbuf) {
    const int warp_g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        // the factorisation that follows starts from a clean barrier
        gb->done = 0u;
        gb->panel = 0u;
        gb->err = 0;
    }
    if (warp_g >= total_rows) return;
    int li = 0;
    while (li + 1 < n_large && row_base[li + 1] <= warp_g) ++li;
    const int inst = large_list[li];
    const DevInst& I = insts[inst];
    if (mode == INST_MODE_NEWTON && !A.active[inst]) return;
    const int i = warp_g - row_base[li];
    const int n = I.n, bw = I.bw, rw = I.rw, f0 = I.f_off;
    if (mode == INST_MODE_NEWTON && i == 0 && lane == 0) {
        A.iters[inst] += 1;
        if (A.bytes_counter) atomicAdd(A.bytes_counter, (unsigned long long)I.io_bytes);
    }
    const double* Kinit = A.Kinit + I.band_off;
    double* B = A.lband + I.lband_off + (long long)i * I.lrw;
    for (int o = rw + lane; o < I.lrw; o += 32) B[o] = 0.0;  // fill slots
    double cv = 0.0;
    for (int o = lane; o < rw; o += 32) {
        const int j = i + o - bw;
        const long long slot = (long long)i * rw + o;
        if (j < 0 || j >= n) {
            B[o] = 0.0;
            if (mode == INST_MODE_EXPORT) A.export_band[I.band_off + slot] = 0.0;
            continue;
        }
        const double K = A.kband[I.band_off + slot];
        double C = 0.0;
        if (I.has_damping) {
            C = I.alpha_m * (i == j ? A.Mrff[f0 + i] : 0.0);
            if (I.beta_k != 0.0) C += I.beta_k * K;
            if (I.beta_k_init != 0.0) C += I.beta_k_init * Kinit[slot];
            const int gj = f0 + j;
            const double an = I.a0 * (A.u_f[gj] - A.u_n[gj]) - I.a2 * A.v_n[gj] - I.a3 * A.a_n[gj];
            const double vt = A.v_n[gj] + I.dt * ((1.0 - I.gamma) * A.a_n[gj] + I.gamma * an);
            cv += C * vt;
        }
        double keff = K;
        if (I.has_damping && I.a1 != 0.0) keff += I.a1 * C;
        if (i == j) keff += I.a0 * A.Mff[f0 + i];
        B[o] = keff;
        if (mode == INST_MODE_EXPORT) A.export_band[I.band_off + slot] = keff;
    }
    cv = warp_sum(cv);
    if (lane == 0) {
        const int gi = f0 + i;
        const double an = I.a0 * (A.u_f[gi] - A.u_n[gi]) - I.a2 * A.v_n[gi] - I.a3 * A.a_n[gi];
        const double F = A.fsum[gi];
        const double ma = A.Mff[gi] * an;
        A.R[gi] = A.P_f[gi] - F - 0.0 - cv - ma;
        wbuf[gi] = A.R[gi];
        if (mode == INST_MODE_EXPORT) A.export_f[gi] = F;
    }
}

// The learned guess's check on the global-memory band path, between the assembly and the
// factorisation (the instance kernel's check, the same arithmetic): one CTA per large instance.
// At the step's first iteration from a learned guess u_l, compare |R(u_l)| with the first-order
// residual of the Newmark predictor u_p, |R(u_l) + K_eff (u_l - u_p)|, K_eff being the band just
// assembled (row i: columns i - bw .. i + bw at slots 0 .. 2 bw); when the learned one is the
// larger, go back to u_p, skip this iteration's factorisation and list the elements again.
__global__ void __launch_bounds__(256) large_learned_check_kernel(const DevInst* __restrict__ insts, InstArrays A,
                                                                  const int* __restrict__ large_list,
                                                                  int n_large) {
    __shared__ double red[32];
    __shared__ int red_r[2];
    const int li = blockIdx.x;
    if (li >= n_large) return;
    const int inst = large_list[li];
    const DevInst& I = insts[inst];
    const int tid = threadIdx.x, nt = blockDim.x;
    if (tid == 0) A.skip[inst] = 0;
    if (!A.active[inst] || A.iters[inst] != 1 || A.rejected[inst] || (A.attempt && A.attempt[inst] != 0)) return;
    const int n = I.n, bw = I.bw, f0 = I.f_off;
    const double* B = A.lband + I.lband_off;
    double sl = 0.0, sp = 0.0;
    for (int i = tid; i < n; i += nt) {
        double kd = 0.0;
        for (int o = 0; o <= 2 * bw; ++o) {
            const int j = i + o - bw;
            if (j >= 0 && j < n) kd += B[(long long)i * I.lrw + o] * (A.u_f[f0 + j] - A.u_base[f0 + j]);
        }
        const double r = A.R[f0 + i];
        const double rp = r + kd;
        sl += r * r;
        sp += rp * rp;
    }
    sl = block_sum(sl, red);
    sp = block_sum(sp, red);
    const bool keep = isfinite(sl) && sl <= sp;
    if (tid == 0 && A.pred_stats) {
        A.pred_stats[2 * inst] += 1;
        if (keep) A.pred_stats[2 * inst + 1] += 1;
    }
    if (keep) return;
    for (int i = tid; i < n; i += nt) {
        const int gi = f0 + i;
        const double u = A.u_base[gi];
        A.u_f[gi] = u;
        A.u_full[A.free_dof[gi]] = u;
    }
    const size_t e0 = (size_t)I.elem_off * kEStride;
    for (size_t t = tid; t < (size_t)I.n_elem * kEStride; t += nt) A.estate[e0 + t] = A.estate_base[e0 + t];
    if (I.n_sl > 0) {
        __syncthreads();
        enforce_slaves(I, A);
    }
    if (tid == 0) {
        A.iters[inst] -= 1;  // the rejected evaluation is not a Newton iteration of the step
        A.rejected[inst] = 1;
        A.skip[inst] = 1;
        red_r[0] = A.ctl ? atomicAdd(&A.el.count[(A.ctl->iter + 1) & 1], I.n_elem) : -1;
    }
    __syncthreads();
    const int base = red_r[0];
    if (base >= 0) {
        const int buf = (A.ctl->iter + 1) & 1;
        for (int k = tid; k < I.n_elem; k += nt) A.el.list[buf][base + k] = list_entry(A.el, buf, I.elem_off + k);
    }
}

// ---- blocked band LU with partial pivoting -------------------------------------------------

// Copies the exported band of every large instance into its factorisation band (fill slots
// zero) and the right-hand side into wbuf (strut_gpu_factor_solve on a band from
// strut_gpu_state_determination).
__global__ void large_load_exported_kernel(const DevInst* __restrict__ insts, InstArrays A,
                                           const int* __restrict__ large_list, int n_large,
                                           GridBarrier* gb, double* __restrict__ wbuf) {
    if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
        gb->done = 0u;
        gb->panel = 0u;
        gb->err = 0;
    }
    const int li = blockIdx.y;
    if (li >= n_large) return;
    const DevInst& I = insts[large_list[li]];
    const long long total = (long long)I.n * I.lrw;
    const long long stride = (long long)gridDim.x * blockDim.x;
    const long long first = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    for (long long t = first; t < total; t += stride) {
        const long long i = t / I.lrw;
        const int o = (int)(t - i * I.lrw);
        A.lband[I.lband_off + t] = o < I.rw ? A.export_band[I.band_off + i * I.rw + o] : 0.0;
    }
    for (long long i = first; i < I.n; i += stride) wbuf[I.f_off + i] = A.rhs_in[I.f_off + i];
}

// Shared memory of large_factor_kernel: the panel's unit lower triangle L11
// (kPanel x (kPanel + 1)); CTA 0's panel rows (kLargeThreads x (kPanel + 1)), whose space the
// column slab of the trailing phase ((kPanel + bw) x (kColTile + 2)) reuses; four rows of U; four
// columns by place (two sets, by column parity); the panel's row permutation.
// Row stride of the panel-row buffer, which the slab (stride kColTile + 2) reuses.
__host__ __device__ constexpr int large_row_stride(int panel) {
    return panel + 1 > kColTile + 2 ? panel + 1 : kColTile + 2;
}
__host__ __device__ constexpr int large_col_tile(int threads) {
    return threads <= kLargeThreadsMid ? kColTileNarrow : kColTile;
}
__host__ __device__ inline size_t large_factor_smem(int panel, int threads) {
    return sizeof(double) * ((size_t)panel * (panel + 1) + (size_t)threads * large_row_stride(panel) + 4 * panel +
                             8 * (size_t)threads) +
           sizeof(int) * (size_t)threads;
}

// Column tiles of the trailing update of one panel (+1: the right-hand side): the CTAs a
// factorisation can keep busy.
__host__ __device__ inline int large_factor_tiles(int bw, int threads) {
    return (2 * bw + large_col_tile(threads) - 1) / large_col_tile(threads) + 1;
}

// Largest half-band each variant takes: one thread per panel row.
constexpr int kLargeMaxBwNarrow = kLargeThreadsNarrow - kPanel;
constexpr int kLargeMaxBwMid = kLargeThreadsMid - kPanel;
constexpr int kLargeMaxBw = kLargeThreads - kPanel;
constexpr int kLargeMaxBwWide = kLargeThreadsWide - kPanelWide;

// Argmax over a warp, the first (smallest index) of equal values winning.
__device__ __forceinline__ void warp_argmax_first(double& v, int& idx) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, v, off);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, off);
        if (ov > v || (ov == v && oi < idx)) {
            v = ov;
            idx = oi;
        }
    }
}

// Cooperative.  wbuf holds the right-hand side on entry and L^-1 P b on exit; the band holds U
// on exit (its strictly lower part is left stale: the substitution reads U only).  lpan
// (column-major, leading dimension kLargeThreads) / lperm: the factored panel and the row
// permutation of its interchanges, from CTA 0 to the others.
//
// Per panel: CTA 0 factors the panel columns with one thread per panel row, the row in shared
// memory and four of its columns in registers.  A column is one chain of latencies (offer the
// entries by place, barrier, pivot and its reciprocal beside the vote, multiplier, the rest of the
// four columns), so it has no branch but the vote's: only where a row beats the diagonal
// strictly, or the diagonal is small, the search for the first largest entry runs, and an
// interchange swaps the places of two rows, not the rows.  After four columns the pivot rows
// behind them are formed by one warp, lane = column, and every row takes its four updates an
// entry in the columns' order.  Rows exchanged whole, a vote of twelve warps and a division a
// column took 30,200 cycles a panel of 32 columns (n = 936, half band 83), this 17,500; the
// factorisation with its loads and signals 63,200 cycles a panel, now 34,200.  CTA 0
// publishes the panel; every CTA takes column tiles of the trailing block: loads them with the panel's row
// permutation applied, solves the panel rows against the unit lower L11 on the warps (lane =
// row), subtracts L21 U12 from the rows below entry by entry in column order (one thread per
// row, the row's multipliers in registers) and counts itself off.
template <int PANEL, int THREADS>
__global__ void __launch_bounds__(THREADS) large_factor_kernel(
    const DevInst* __restrict__ insts, InstArrays A, const int* __restrict__ large_list,
    int n_large, int mode, GridBarrier* gb, double* wbuf, double* lpan, int* lperm) {
    extern __shared__ __align__(16) double smem_lf[];
    __shared__ int s_flag[1];
    __shared__ double red[32];
    constexpr int kPs = PANEL + 1;     // row stride of L11
    constexpr int kRs = large_row_stride(PANEL);  // row stride of the panel rows and the slab
    constexpr int CT = large_col_tile(THREADS);
    constexpr bool kNarrow = THREADS <= kLargeThreadsMid;
    constexpr int kFly = kNarrow ? 8 : 4;  // loads in flight per thread
    constexpr int kSs = CT + 2;   // row stride of the slab (even: 16-byte rows)
    constexpr int kLd = THREADS;  // leading dimension of lpan
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
    const int nwarps = nt >> 5;
    double* L11 = smem_lf;                              // PANEL x kPs
    double* Pout = L11 + PANEL * kPs;                  // panel rows (CTA 0), THREADS x kRs
    double* S = Pout;                                   // slab of the trailing phase, pr x kSs
    double* ublk = Pout + (size_t)THREADS * kRs;        // four rows of U, PANEL x 4
    double* colb = ublk + 4 * PANEL;                    // four columns by place, by column parity
    int* s_perm = (int*)(colb + 8 * THREADS);           // panel row -> original row
    __shared__ unsigned int s_word;
    unsigned int panels = 0;  // published so far, over all instances
    // CTA 0 waits for the others to be through with the panel, the others say that they are
    auto finish = [&]() -> bool {
        if (blockIdx.x == 0) {
            const unsigned int all = panels * (gridDim.x - 1);
            return await_word(gb, &gb->done, &s_word, [=](unsigned int v) { return v == all; });
        }
        __syncthreads();
        if (tid == 0) {
            __threadfence();
            atomicAdd(&gb->done, 1u);
        }
        return true;
    };
    for (int li = 0; li < n_large; ++li) {
        const int inst = large_list[li];
        const DevInst& I = insts[inst];
        if (mode == INST_MODE_NEWTON && (!A.active[inst] || (A.skip && A.skip[inst]))) {
            if (blockIdx.x == 0 && tid == 0) A.lstatus[li] = LSTAT_IDLE;
            continue;
        }
        const int n = I.n, bw = I.bw, lrw = I.lrw;
        double* B = A.lband + I.lband_off;
        double* w = wbuf + I.f_off;
        const Attempt at = attempt_of(I, A, inst);
        if (mode == INST_MODE_NEWTON && at.test == 2) {
            // NormUnbalance is tested on the residual before the solve; every CTA reaches the
            // same decision from the same sums
            double s = 0.0;
            for (int i = tid; i < n; i += nt) s += A.R[I.f_off + i] * A.R[I.f_off + i];
            s = block_sum(s, red);
            if (sqrt(s) <= at.tol) {
                if (blockIdx.x == 0 && tid == 0) A.lstatus[li] = LSTAT_CONVERGED;
                continue;
            }
        }
        const int P = min(PANEL, max(bw, 1));
        int result = LSTAT_OK;
        int pivoted = 0;
        for (int k0 = 0; k0 < n && result == LSTAT_OK; k0 += P) {
            const int kb = min(P, n - k0);
            const int r1 = min(n - 1, k0 + kb - 1 + bw);      // last row with a nonzero in the panel
            const int pr = r1 - k0 + 1;
            const int c1 = min(n - 1, k0 + kb - 1 + 2 * bw);  // last column the panel's rows reach
            const int r = tid;                                // the panel row of this thread
            const bool own = r < pr;
            if (blockIdx.x == 0) {
                // ---- panel: rows k0..r1, columns k0..k0+kb-1 (rows loaded coalesced, lane = column)
                for (int rb = wid; rb < pr; rb += 2 * kFly * nwarps) {
                    double v[2 * kFly];  // rows in flight per warp
#pragma unroll
                    for (int m = 0; m < 2 * kFly; ++m) {
                        const int rr = rb + m * nwarps;
                        const int d = lane - rr;
                        v[m] = (rr < pr && lane < kb && d >= -bw && d <= 2 * bw) ? B[lslot(lrw, bw, k0 + rr, k0 + lane)]
                                                                                 : 0.0;
                    }
#pragma unroll
                    for (int m = 0; m < 2 * kFly; ++m)
                        if (rb + m * nwarps < pr && lane < PANEL) Pout[(rb + m * nwarps) * kRs + lane] = v[m];
                }
                if (tid == 0) s_flag[0] = LSTAT_OK;
                __syncthreads();
                bool failed = false;
                int pos = r;  // the row's place; interchanges move places, not rows
                double* row = Pout + r * kRs;
                for (int c0 = 0; c0 < kb && !failed; c0 += 4) {
                    // One column: no branch but the vote's, which takes the rows in which the diagonal
                    // is beaten or small out of the way.  Rows past the band hold zeros, as do the
                    // places past the panel; rows that are done offer a zero and keep their entries.
                    double a[4];  // a[q] = column c + q of this thread's row
#pragma unroll
                    for (int q = 0; q < 4; ++q) a[q] = own ? row[c0 + q] : 0.0;
                    const int ce = min(kb, c0 + 4);
#pragma unroll 1
                    for (int c = c0; c < ce; ++c) {
                        // double buffered: a slow thread may still read the previous one
                        double* cb = colb + (c & 1) * 4 * THREADS;
                        const double offer = pos >= c ? a[0] : 0.0;
                        cb[pos] = offer;
#pragma unroll
                        for (int q = 1; q < 4; ++q) cb[q * THREADS + pos] = a[q];
                        __syncthreads();
                        double u[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) u[q] = cb[q * THREADS + c];
                        // the reference's strict '>' scan keeps the diagonal unless a row below
                        // beats it, then takes the first largest
                        const double dabs = fabs(u[0]);
                        bool rare = dabs <= 1.0e-14;
                        if constexpr (kNarrow) {
#pragma unroll
                            for (int m = 0; m < THREADS / 32; ++m) rare |= fabs(cb[lane + 32 * m]) > dabs;
                            rare = __any_sync(0xffffffffu, rare);
                        } else {
                            rare = __syncthreads_or(rare || fabs(offer) > dabs);
                        }
                        double rpiv = pivot_recip(u[0]);  // beside the vote
                        if (rare) {
                            // a NaN is no candidate: every thread has to find the same row
                            double pv = -1.0;
                            int p = 0x7fffffff;
                            for (int rr = c + lane; rr < pr; rr += 32) {
                                const double v = fabs(cb[rr]);
                                if (v > pv) {
                                    pv = v;
                                    p = rr;
                                }
                            }
                            warp_argmax_first(pv, p);
                            if (pv <= 1.0e-14) {
                                failed = true;
                                if (tid == 0) s_flag[0] = LSTAT_SINGULAR;
                                break;
                            }
                            if (p != c) {
                                pivoted = 1;
#pragma unroll
                                for (int q = 0; q < 4; ++q) u[q] = cb[q * THREADS + p];
                                rpiv = pivot_recip(u[0]);
                                if (pos == c) pos = p;
                                else if (pos == p) pos = c;
                            }
                        }
                        const bool below = pos > c;
                        const double f = pivot_quot(a[0], u[0], rpiv);
                        a[0] = below ? f : a[0];
                        row[c] = a[0];
                        if (pos == c) s_perm[c] = r;
#pragma unroll
                        for (int q = 1; q < 4; ++q) {
                            const double t = fma(-f, u[q], a[q]);
                            a[q - 1] = below ? t : a[q];
                        }
                    }
                    if (c0 + 4 < kb && !failed) {
                        // the four pivot rows behind these columns, then four updates an entry,
                        // in the columns' order
                        __syncthreads();
                        if (wid == 0 && lane >= c0 + 4 && lane < PANEL) {
                            double* r0 = Pout + s_perm[c0] * kRs;
                            double* r1 = Pout + s_perm[c0 + 1] * kRs;
                            double* r2 = Pout + s_perm[c0 + 2] * kRs;
                            double* r3 = Pout + s_perm[c0 + 3] * kRs;
                            const double u0 = r0[lane];
                            const double u1 = fma(-r1[c0], u0, r1[lane]);
                            const double u2 = fma(-r2[c0 + 1], u1, fma(-r2[c0], u0, r2[lane]));
                            const double u3 =
                                fma(-r3[c0 + 2], u2, fma(-r3[c0 + 1], u1, fma(-r3[c0], u0, r3[lane])));
                            r1[lane] = u1;
                            r2[lane] = u2;
                            r3[lane] = u3;
                            double2* to = reinterpret_cast<double2*>(ublk + 4 * lane);
                            to[0] = make_double2(u0, u1);
                            to[1] = make_double2(u2, u3);
                        }
                        __syncthreads();
                        if (own && pos >= c0 + 4 && pos <= c0 + 3 + bw) {
                            double f[4];
#pragma unroll
                            for (int k = 0; k < 4; ++k) f[k] = row[c0 + k];
#pragma unroll 2
                            for (int q = c0 + 4; q < kb; q += 4) {
                                double x[4];
#pragma unroll
                                for (int j = 0; j < 4; ++j) x[j] = row[q + j];
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const double2* u = reinterpret_cast<const double2*>(ublk + 4 * (q + j));
                                    const double2 lo = u[0], hi = u[1];
                                    x[j] = fma(-f[0], lo.x, x[j]);
                                    x[j] = fma(-f[1], lo.y, x[j]);
                                    x[j] = fma(-f[2], hi.x, x[j]);
                                    x[j] = fma(-f[3], hi.y, x[j]);
                                }
#pragma unroll
                                for (int j = 0; j < 4; ++j) row[q + j] = x[j];
                            }
                        }
                    }
                }
                if (own && pos >= kb) s_perm[pos] = r;
                __syncthreads();
                if (s_flag[0] == LSTAT_OK) {
                    // thread = place in the panel
                    if (own) {
                        const double* placed = Pout + s_perm[r] * kRs;
#pragma unroll 8
                        for (int q = 0; q < kb; ++q) lpan[q * kLd + r] = placed[q];
                        lperm[r] = s_perm[r];
                    }
                    for (int rr = wid; rr < kb; rr += nwarps)
                        if (lane >= rr && lane < kb)
                            B[lslot(lrw, bw, k0 + rr, k0 + lane)] = Pout[s_perm[rr] * kRs + lane];
                }
                __syncthreads();
                ++panels;
                result = s_flag[0];
                if (tid == 0) {
                    A.lstatus[li] = result;
                    __threadfence();
                    atomicExch(&gb->panel, 2 * panels + (result != LSTAT_OK ? 1 : 0));
                }
            } else {
                ++panels;
                const unsigned int want = panels;
                if (!await_word(gb, &gb->panel, &s_word, [=](unsigned int v) { return (v >> 1) == want; })) return;
                result = s_word & 1u ? LSTAT_SINGULAR : LSTAT_OK;
            }
            if (result != LSTAT_OK) {
                if (!finish()) return;
                break;
            }
            // ---- trailing columns k0+kb .. c1 in tiles of CT, and the right-hand side
            const int j_first = k0 + kb;
            const int ncols = c1 - j_first + 1;
            const int ntiles = (ncols > 0 ? (ncols + CT - 1) / CT : 0) + 1;
            if (blockIdx.x >= ntiles) {
                if (!finish()) return;
                continue;
            }
            // this thread's panel row: its multipliers (L21, or L11 for the first kb rows)
            double lrow[PANEL];
#pragma unroll
            for (int q = 0; q < PANEL; ++q) lrow[q] = (own && q < kb) ? lpan[q * kLd + r] : 0.0;
            if (own) {
                s_perm[r] = lperm[r];
                if (r < kb) {
#pragma unroll
                    for (int q = 0; q < PANEL; ++q) L11[r * kPs + q] = lrow[q];
                }
            }
            for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
                const bool rhs = tile == ntiles - 1;
                const int j0 = j_first + tile * CT;
                const int ct = rhs ? 1 : min(CT, c1 - j0 + 1);
                __syncthreads();
                if (rhs) {
                    if (own) S[r * kSs] = w[k0 + s_perm[r]];
                } else {
                    for (int t0 = tid; t0 < pr * CT; t0 += kFly * nt) {
                        double v[kFly];
#pragma unroll
                        for (int m = 0; m < kFly; ++m) {
                            const int t = t0 + m * nt, rr = t / CT, q = t % CT;
                            v[m] = 0.0;
                            if (rr < pr && q < ct) {
                                const int src = k0 + s_perm[rr];
                                const int d = j0 + q - src;
                                if (d >= -bw && d <= 2 * bw) v[m] = B[lslot(lrw, bw, src, j0 + q)];
                            }
                        }
#pragma unroll
                        for (int m = 0; m < kFly; ++m) {
                            const int t = t0 + m * nt, rr = t / CT, q = t % CT;
                            if (rr < pr) S[rr * kSs + q] = v[m];
                        }
                    }
                }
                __syncthreads();
                // U12 = L11^-1 (P A12): lane = panel row, two columns a warp, whose chains of
                // shuffle and FMA (one step a panel column) overlap
                for (int q = wid; q < ct; q += 2 * nwarps) {
                    const int q1 = q + nwarps;
                    double v = lane < kb ? S[lane * kSs + q] : 0.0;
                    double v1 = lane < kb && q1 < ct ? S[lane * kSs + q1] : 0.0;
#pragma unroll 4
                    for (int sc = 0; sc + 1 < kb; ++sc) {
                        const double u = __shfl_sync(0xffffffffu, v, sc);
                        const double u1 = __shfl_sync(0xffffffffu, v1, sc);
                        if (lane > sc && lane < kb) {
                            const double f = -L11[lane * kPs + sc];
                            v = fma(f, u, v);
                            v1 = fma(f, u1, v1);
                        }
                    }
                    if (lane < kb) S[lane * kSs + q] = v;
                    if (lane < kb && q1 < ct) S[lane * kSs + q1] = v1;
                }
                __syncthreads();
                // A22 -= L21 U12 entry by entry, column order; one thread per row
                double v[CT];
                if (own && r >= kb) {
#pragma unroll
                    for (int q = 0; q < CT; ++q) v[q] = S[r * kSs + q];
                    auto step = [&](int sc) {
                        const double f = lrow[sc];
#pragma unroll
                        for (int q2 = 0; q2 < CT / 2; ++q2) {
                            const double2 u = reinterpret_cast<const double2*>(S + sc * kSs)[q2];
                            v[2 * q2] = fma(-f, u.x, v[2 * q2]);
                            v[2 * q2 + 1] = fma(-f, u.y, v[2 * q2 + 1]);
                        }
                    };
                    if (kNarrow && kb == PANEL) {  // without a test a step, so that loads run ahead
#pragma unroll
                        for (int sc = 0; sc < PANEL; ++sc) step(sc);
                    } else {
#pragma unroll
                        for (int sc = 0; sc < PANEL; ++sc)
                            if (sc < kb) step(sc);
                    }
                }
                __syncthreads();
                if (own && r >= kb) {
#pragma unroll
                    for (int q = 0; q < CT; ++q) S[r * kSs + q] = v[q];
                }
                __syncthreads();
                if (rhs) {
                    if (own) w[k0 + r] = S[r * kSs];
                } else {
                    for (int t = tid; t < pr * CT; t += nt) {
                        const int rr = t / CT, q = t % CT, i = k0 + rr;
                        const int d = j0 + q - i;
                        if (q < ct && d >= -bw && d <= 2 * bw) B[lslot(lrw, bw, i, j0 + q)] = S[rr * kSs + q];
                    }
                }
            }
            if (!finish()) return;
        }
        if (blockIdx.x == 0 && tid == 0 && pivoted && result == LSTAT_OK && A.fallbacks) A.fallbacks[inst] += 1;
    }
}

// ---- substitution, update and test ---------------------------------------------------------

// Dynamic shared memory of large_solve_kernel: x (n) and one 32 x 33 diagonal block of U.
__host__ __device__ inline size_t large_solve_smem(int n) {
    return sizeof(double) * ((size_t)n + 32 * 33);
}

// One CTA per large instance (32 warps): U x = L^-1 P b (left in wbuf by the factorisation) in
// blocks of 32 rows from the end.  Warp r of a block forms row r's sum over the columns below
// the block (the row's U entries are contiguous in the band), then warp 0 solves the block's
// triangle with shuffles.  x stays in shared memory.  A block is a chain of
// latencies, so the next block's U and right-hand side are fetched during the triangle, the
// reciprocal pivots are formed beside the sums and a step of the triangle has no branch: with
// the assembly and the factorisation 766 -> 720 us a Newton iteration at n = 936, half band 83.
__global__ void __launch_bounds__(kSolveThreads) large_solve_kernel(
    const DevInst* __restrict__ insts, InstArrays A, const int* __restrict__ large_list, int n_large,
    int mode, double* __restrict__ wbuf, const GridBarrier* __restrict__ gb) {
    extern __shared__ __align__(16) double smem_ls[];
    __shared__ double red[32];
    __shared__ int red_r[32];
    __shared__ double tb[32], rdiag[32];  // the block's right-hand side, its reciprocal pivots
    const int li = blockIdx.x;
    if (li >= n_large) return;
    const int inst = large_list[li];
    const DevInst& I = insts[inst];
    const int st = A.lstatus[li];
    if (mode == INST_MODE_NEWTON && (st == LSTAT_IDLE || !A.active[inst])) return;
    if (gb->err) {
        // a barrier of the factorisation gave up: the factors are incomplete
        if (threadIdx.x == 0) {
            A.status[inst] = STRUT_CUDA_ERROR;
            if (mode == INST_MODE_NEWTON && A.active[inst]) {
                A.active[inst] = 0;
                atomicSub(A.nactive, 1);
            }
        }
        return;
    }
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, wid = tid >> 5;
    const int n = I.n, bw = I.bw, lrw = I.lrw, f0 = I.f_off;
    const int ub = 2 * bw;  // reach of U
    int* hrow = (mode == INST_MODE_NEWTON && A.hist_iters && A.ctl)
                    ? A.hist_iters + (size_t)A.ctl->step * A.n_inst : nullptr;
    if (st == LSTAT_CONVERGED) {
        if (tid == 0) {
            A.active[inst] = 0;
            atomicSub(A.nactive, 1);
            if (hrow) hrow[inst] = A.iters[inst] + (A.iters_prev ? A.iters_prev[inst] : 0);
        }
        return;
    }
    if (st == LSTAT_SINGULAR) {
        if (tid == 0) {
            A.status[inst] = LSTAT_SINGULAR;
            if (mode == INST_MODE_NEWTON && A.active[inst]) {
                A.active[inst] = 0;
                atomicSub(A.nactive, 1);
            }
        }
        return;
    }
    const double* B = A.lband + I.lband_off;
    double* w = wbuf + f0;  // L^-1 P b, then x
    double* xs = smem_ls;         // n
    double* Ud = smem_ls + n;     // 32 x 33
    // The row of this warp in the block that ends at r1: its entries right of the block (the first
    // kAhead columns a lane), its part of the diagonal block, its right-hand side.
    double pre[kSolveAhead], dg = 0.0, wi = 0.0;
    auto fetch = [&](int r1) {
        const int r0 = max(0, r1 - 32), i = r0 + wid;
        if (i >= r1) return;
        const double* urow = B + (long long)i * lrw + bw;  // U(i, i + o), o = 0 .. 2 bw
        const int jmax = min(n - 1, i + ub);
#pragma unroll
        for (int m = 0; m < kSolveAhead; ++m) {
            const int j = r1 + lane + 32 * m;
            pre[m] = j <= jmax ? urow[j - i] : 0.0;
        }
        const int o = r0 + lane - i;
        dg = (lane < r1 - r0 && o >= 0 && o <= ub) ? urow[o] : 0.0;
        wi = w[i];
    };
    fetch(n);
    for (int r1 = n; r1 > 0; r1 -= 32) {
        const int r0 = max(0, r1 - 32), rb = r1 - r0;
        if (wid < rb) {
            const int i = r0 + wid;
            const double* urow = B + (long long)i * lrw + bw;
            const int jmax = min(n - 1, i + ub);
            double acc = 0.0;
#pragma unroll
            for (int m = 0; m < kSolveAhead; ++m) {
                const int j = r1 + lane + 32 * m;
                if (j <= jmax) acc = fma(pre[m], xs[j], acc);
            }
#pragma unroll 8
            for (int j = r1 + lane + 32 * kSolveAhead; j <= jmax; j += 32) acc = fma(urow[j - i], xs[j], acc);
            acc = warp_sum(acc);
            if (lane < rb) Ud[wid * 33 + lane] = dg;
            if (lane == wid) rdiag[wid] = 1.0 / dg;  // off the sequential chain
            if (lane == 0) tb[wid] = wi - acc;
        }
        if (r0 > 0) fetch(r0);
        __syncthreads();
        if (wid == 0) {
            double v = lane < rb ? tb[lane] : 0.0;
            const double rd = lane < rb ? rdiag[lane] : 0.0;
#pragma unroll 8
            for (int s = rb - 1; s >= 0; --s) {
                const double u = Ud[lane * 33 + s];
                const double x = __shfl_sync(0xffffffffu, v * rd, s);
                const double t = fma(-u, x, v);
                v = lane == s ? x : lane < s ? t : v;
            }
            if (lane < rb) xs[r0 + lane] = v;
        }
        __syncthreads();
    }
    for (int i = tid; i < n; i += nt) w[i] = xs[i];
    __syncthreads();
    if (mode == INST_MODE_SOLVE_EXPORTED) {
        for (int i = tid; i < n; i += nt) A.du[f0 + i] = w[i];
        return;
    }
    InstArrays Ar = A;
    newton_tail(I, Ar, inst, w, A.R + f0, hrow, red, red_r);
}

}  // namespace strut
