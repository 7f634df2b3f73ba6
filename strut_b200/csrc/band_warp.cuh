// Band factor-solve in shared memory: the LU of narrow bands and the one-warp back substitutions.
//
// Algorithm (paths relative to the Strut project root):
//   BandGeneral  src/mojo/solver/run_case/linear_solver_backend.mojo:631-680, 735-770
//   BandSPD      linear_solver_backend.mojo:689-726, 772-812
//
// A 2D frame's system (36 to 216 unknowns, half band 11 to 20) is a chain of n dependent steps of a
// few hundred operations, so the time is the latency of a step.  Measured for 216 unknowns of half
// band 20 (cycles per unknown): factorisation 1,230 -> 355, back substitution 810 -> 263 (the sums of a row
// taken column by column instead, 123, rounded differently and were dropped: a batch of long records
// is chaotic at the rounding level, and one record of 256 ended elsewhere).
#pragma once

#include "quotient.cuh"

namespace strut {

constexpr int kBackWarpMax = 24;   // widest half band of the one-warp back substitutions: 24 + 8 rows in a
                                   // warp's window
constexpr int kBackWarpGroup = 8;  // unknowns per window position
constexpr int kLuRowsMax = 62;     // widest half band of band_lu_cta
constexpr int kLuRowsThreads = 256;

// Barrier of the first nt threads of the CTA (a multiple of 32).
__device__ __forceinline__ void bar_first(int nt) { asm volatile("bar.sync 1, %0;" ::"r"(nt) : "memory"); }

// Band LU without interchanges (Doolittle) of the n x (2 bw + 1) band B in shared memory with the
// first NW warps of the CTA, the right-hand side (at B[woff ...]) carried along as one more column,
// so it leaves as L^-1 rhs.  Step k: warp w takes rows k + 1 + w + u NW, u < NR; its lanes form the
// row's multiplier from the pivot's reciprocal and update the row, lane = column (NC columns per
// lane).  The warp of row k + 1 publishes the next reciprocal, and one barrier ends the step.  Every
// entry receives the reference's operations in the reference's order.  KEEP: multipliers stored.
//
// What bounds it is the chain of a step (load, quotient, multiply-add, reciprocal, barrier), and
// next to it the instructions of a warp that works alone on its scheduler.  So the step has no
// inner loop, no division (74 cycles, 413 with a zero numerator, which bands are full of; recip 40,
// quot 24) and no reducing barrier (63 against 28 cycles): a row that needs an interchange raises a
// flag that the next step reads with its other operands.  Flags alternate between two places by the
// step's parity: a place is written in one step and read in the next only, so all warps leave the
// loop at the same step.  While all bw rows exist, every operand
// has a pointer that moves by a fixed stride; rows and columns that a warp or lane does not have
// point at the zeros z (stride 0) instead of being tested.
// NR NW >= bw, 32 NC > bw.  rk: 2 doubles; z: 2 doubles; flag: 4 ints of shared memory.  Returns
// 0 ok, 2 singular, 6 a row swap would be needed (the caller then starts again from the assembled
// values), on the threads of the first NW warps.
template <int NR, int NC, int NW, bool KEEP>
__device__ __forceinline__ int band_lu_rows(double* B, int n, int bw, int rw, int woff, double* rk, double* z,
                                            int* flag) {
    constexpr int NT = 32 * NW;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        rk[0] = recip(B[bw]);
        z[0] = z[1] = 0.0;
        flag[0] = flag[1] = flag[2] = flag[3] = 0;
    }
    // what step k of an elimination that cannot go on means: a row swap (6) or a singular matrix
    auto verdict = [&](int k) { return flag[2 * (k & 1)] && flag[2 * (k & 1) + 1] ? 6 : 2; };
    const double* pf[NR];  // B(i, k) of this warp's rows
    double* pa[NR][NC];    // this lane's entries of them
    const double* pu[NC];  // and of row k
    const double* pk = B + bw;
    int sf[NR], sa[NR][NC], su[NC];
#pragma unroll
    for (int u = 0; u < NR; ++u) {
        const int r = 1 + warp + NW * u;
        pf[u] = r <= bw ? B + r * rw + bw - r : z;
        sf[u] = r <= bw ? rw : 0;
#pragma unroll
        for (int v = 0; v < NC; ++v) {
            const int c = lane + 1 + 32 * v;  // column k + c, or the right-hand side behind the last
            if (u == 0) {
                pu[v] = c <= bw ? B + bw + c : c == bw + 1 ? B + woff : z;
                su[v] = c <= bw ? rw : c == bw + 1 ? 1 : 0;
            }
            pa[u][v] = r > bw ? z + 1 : c <= bw ? B + r * rw + bw - r + c : c == bw + 1 ? B + woff + r : z + 1;
            sa[u][v] = r > bw ? 0 : su[v];
        }
    }
    bar_first(NT);
    int k = 0;
#pragma unroll 1
    for (; k + bw < n; ++k) {
        const double akk = *pk, rkk = rk[k & 1], pa_ = fabs(akk);
        const int failed = flag[2 * ((k + 1) & 1)];  // raised in step k - 1
        double f[NR], uk[NC], a[NR][NC];
#pragma unroll
        for (int u = 0; u < NR; ++u) f[u] = *pf[u];
#pragma unroll
        for (int v = 0; v < NC; ++v) {
            uk[v] = *pu[v];
#pragma unroll
            for (int u = 0; u < NR; ++u) a[u][v] = *pa[u][v];
        }
        if (failed) return verdict(k - 1);
        bool swap = false;
#pragma unroll
        for (int u = 0; u < NR; ++u) {
            swap = swap || fabs(f[u]) > pa_;
            const double q = quot(f[u], akk, rkk);
#pragma unroll
            for (int v = 0; v < NC; ++v) {
                a[u][v] -= q * uk[v];
                *pa[u][v] = a[u][v];
                pa[u][v] += sa[u][v];
            }
            if (KEEP && lane == 0 && sf[u]) *const_cast<double*>(pf[u]) = q;
            pf[u] += sf[u];
        }
        if (threadIdx.x == 0) rk[(k + 1) & 1] = recip(a[0][0]);
        if (swap) {
            // pivot search of linear_solver_backend.mojo:640-657: an entry strictly larger than
            // the diagonal selects another row; the largest one decides singularity
            flag[2 * (k & 1)] = 1;
#pragma unroll
            for (int u = 0; u < NR; ++u)
                if (fabs(f[u]) > 1.0e-14) flag[2 * (k & 1) + 1] = 1;
        }
#pragma unroll
        for (int v = 0; v < NC; ++v) pu[v] += su[v];
        pk += rw;
        bar_first(NT);
        if (pa_ <= 1.0e-14) return verdict(k);
    }
    if (k > 0 && flag[2 * ((k + 1) & 1)]) return verdict(k - 1);
    // the last bw columns, fewer rows and columns each
    int dk = k * rw + bw;
#pragma unroll 1
    for (; k < n; ++k) {
        const int m = n - 1 - k;
        const double akk = B[dk], rkk = rk[k & 1], pa_ = fabs(akk);
        double f[NR], uk[NC];
        bool swap = false;
#pragma unroll
        for (int v = 0; v < NC; ++v) {
            const int c = lane + 1 + 32 * v;
            uk[v] = c <= m + 1 ? B[c <= m ? dk + c : woff + k] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < NR; ++u) {
            const int r = 1 + warp + NW * u;
            if (r > m) continue;
            const int d = dk + r * (rw - 1);
            f[u] = B[d];
            swap = swap || fabs(f[u]) > pa_;
            const double q = quot(f[u], akk, rkk);
#pragma unroll
            for (int v = 0; v < NC; ++v) {
                const int c = lane + 1 + 32 * v;
                if (c <= m + 1) {
                    double* p = B + (c <= m ? d + c : woff + k + r);
                    const double t = *p - q * uk[v];
                    *p = t;
                    if (u == 0 && v == 0 && threadIdx.x == 0) rk[(k + 1) & 1] = recip(t);
                }
            }
            if (KEEP && lane == 0) B[d] = q;
        }
        if (swap) {
            flag[2 * (k & 1)] = 1;
#pragma unroll
            for (int u = 0; u < NR; ++u)
                if (1 + warp + NW * u <= m && fabs(f[u]) > 1.0e-14) flag[2 * (k & 1) + 1] = 1;
        }
        dk += rw;
        bar_first(NT);
        if (flag[2 * (k & 1)] || pa_ <= 1.0e-14) return verdict(k);
    }
    return 0;
}

// band_lu_rows for half bands up to kLuRowsMax, by a CTA of kLuRowsThreads threads (all of them
// call; the result is the same on all).
template <bool KEEP>
__device__ __forceinline__ int band_lu_cta(double* B, int n, int bw, int rw, int woff, double* rk, double* z,
                                           int* flag) {
    constexpr int NW = kLuRowsThreads / 32;
    if (bw <= 2 * NW) return band_lu_rows<2, 1, NW, KEEP>(B, n, bw, rw, woff, rk, z, flag);
    if (bw <= 3 * NW) return band_lu_rows<3, 1, NW, KEEP>(B, n, bw, rw, woff, rk, z, flag);
    return band_lu_rows<8, 2, NW, KEEP>(B, n, bw, rw, woff, rk, z, flag);
}

// U x = w with one warp for bw <= kBackWarpMax, every row's sum in the reference's order (columns
// upwards from the diagonal, so the chain of a row runs through all its bw products, the newest
// unknown's first).  The unknowns a row needs and the next row's entries are in registers, so a row
// costs its chain and a quotient (bw 20: 263 cycles; one lane with its operands in shared memory
// took 810).  EXACT: bw == BW; else bw <= BW.  Slots of columns outside the matrix hold zeros.
// rd: n doubles of scratch.
template <int BW, bool EXACT>
__device__ __noinline__ void band_back_lu(const double* B, int n, int bw, int rw, const double* w, double* x,
                                          double* rd) {
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < n; i += 32) rd[i] = 1.0 / B[i * rw + bw];
    __syncwarp();
    double xw[BW], u[BW];  // x_(i + 1 + t), U(i, i + 1 + t)
    const double* row = B + (n - 1) * rw + bw;
#pragma unroll
    for (int t = 0; t < BW; ++t) {
        xw[t] = 0.0;
        u[t] = EXACT || t < bw ? row[1 + t] : 0.0;
    }
    double s = w[n - 1], d = row[0], r = rd[n - 1];
#pragma unroll 2
    for (int i = n - 1; i >= 0; --i) {
        const int ip = i > 0 ? i - 1 : 0;
        row = B + ip * rw + bw;
        double un[BW];
#pragma unroll
        for (int t = 0; t < BW; ++t) un[t] = EXACT || t < bw ? row[1 + t] : 0.0;
        const double sn = w[ip], dn = row[0], rn = rd[ip];
#pragma unroll
        for (int t = 0; t < BW; ++t) s -= u[t] * xw[t];
        s = quot(s, d, r);
        if (lane == 0) x[i] = s;
#pragma unroll
        for (int t = BW - 1; t > 0; --t) xw[t] = xw[t - 1];
        xw[0] = s;
#pragma unroll
        for (int t = 0; t < BW; ++t) u[t] = un[t];
        s = sn;
        d = dn;
        r = rn;
    }
    __syncwarp();
}

// The half bands of 2D frames of two to five bays have their own instance.
__device__ __forceinline__ void band_back_lu_any(const double* B, int n, int bw, int rw, const double* w, double* x,
                                                 double* rd) {
    if (bw == 11) band_back_lu<11, true>(B, n, bw, rw, w, x, rd);
    else if (bw == 14) band_back_lu<14, true>(B, n, bw, rw, w, x, rd);
    else if (bw == 17) band_back_lu<17, true>(B, n, bw, rw, w, x, rd);
    else if (bw == 20) band_back_lu<20, true>(B, n, bw, rw, w, x, rd);
    else if (bw <= 12) band_back_lu<12, false>(B, n, bw, rw, w, x, rd);
    else band_back_lu<kBackWarpMax, false>(B, n, bw, rw, w, x, rd);
}

// L^T x = w with one warp for bw <= kBackWarpMax, column by column from the end (the reference's
// order), a lane per row of the window, so that only a quotient and a shuffle separate one unknown
// from the next.  rd: n doubles of scratch.
__device__ __noinline__ void band_back_chol(const double* B, int n, int bw, int rw, const double* w, double* x,
                                            double* rd) {
    constexpr unsigned all = 0xffffffffu;
    constexpr int G = kBackWarpGroup;
    const int lane = threadIdx.x & 31;
    for (int i = lane; i < n; i += 32) rd[i] = 1.0 / B[i * rw + bw];
    __syncwarp();
    int j0 = n - 1;
    int row = j0 - ((j0 - lane) & 31);
    auto coef = [&](int r, int j) -> double {
        return r < 0 || r >= j || r < j - bw ? 0.0 : B[j * rw + (r - j + bw)];
    };
    double c[G], v, r = 0.0, d = 1.0;
#pragma unroll
    for (int q = 0; q < G; ++q) c[q] = coef(row, j0 - q);
    v = row >= 0 ? w[row] : 0.0;
    for (; j0 >= 0; j0 -= G) {
        // the next group's coefficients are loaded while this one's chain runs
        const bool done = row > j0 - G;
        if (done && row >= 0) {
            r = rd[row];
            d = B[row * rw + bw];
        }
        const int row_n = done ? row - 32 : row;
        double cn[G];
#pragma unroll
        for (int q = 0; q < G; ++q) cn[q] = coef(row_n, j0 - G - q);
        const double vn = done && row_n >= 0 ? w[row_n] : 0.0;
#pragma unroll
        for (int q = 0; q < G; ++q) {
            const int j = j0 - q;
            if (j >= 0) {
                const double xj = __shfl_sync(all, quot(v, d, r), j & 31);
                if (lane == (j & 31)) v = xj;
                else v -= c[q] * xj;
            }
        }
        if (done) {
            if (row >= 0) x[row] = v;
            v = vn;
            row = row_n;
        }
#pragma unroll
        for (int q = 0; q < G; ++q) c[q] = cn[q];
    }
    __syncwarp();
}

}  // namespace strut
