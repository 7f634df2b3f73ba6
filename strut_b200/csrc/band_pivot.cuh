// Band factor-solve with partial pivoting by one CTA, the active window in registers.
//
// Strut's BandGeneral factors without interchanges and, at the first column whose pivot test fails,
// restarts from the original matrix with a dense partial-pivot LU (linear_solver_backend.mojo:
// 175-240, 631-680).  Partial pivoting with the same strict test and the first largest entry makes
// the interchanges and eliminations of that restart, and needs only the band: below it the dense
// matrix's columns are zero, and a row reaches at most 2 bw beyond its pivot column.
//
// A thread owns a column: the entries of rows k .. k + R - 1 of its column are R registers, so the
// elimination of a step is R multiply-adds that also move the window on by a row.  The owner of
// column k publishes it; after the step's one barrier every warp by itself finds the pivot, forms
// the multipliers (two per lane, shared inside the warp) and updates its columns, so no second
// barrier is needed; warps whose columns the window does not touch only take the barrier.  The last
// warp carries the right-hand side.  U goes to global memory as it is final and back into the
// band's shared memory for the substitution.
//
// Bound by the multipliers' way from shared memory into registers (R / 2 16-byte broadcasts a warp
// and step).  A 4-story 3D frame with rigid diaphragms (204 unknowns, half band 56), which pivots in
// every iteration: 6.5 M cycles (3.3 ms) for the failed elimination, the dense LU in global memory and its
// substitution, 313 K (159 us) for this, substitution included.
#pragma once

#include "band_warp.cuh"
#include "pivot_candidate.cuh"

namespace strut {

constexpr int kPivotThreads = 256;                     // CTA size
constexpr int kPivotCols = kPivotThreads - 32;         // columns in registers at a time
constexpr int kPivotMaxBw = 63;                        // R = 64 rows
constexpr int kPivotBuf = 64 * (2 + kPivotThreads / 32);  // doubles of shared memory

// Factors the band Kb (n x (2 bw + 1), left as it is) and takes w (in: right-hand side, shared
// memory) to L^-1 P w; U(k, j) to U[k * rw + j - k].  buf: kPivotBuf doubles of shared memory, 16-byte
// aligned.  Returns 0, 2 (singular) on every thread; *swaps counts the interchanges.
template <int R>
__device__ __forceinline__ int band_lu_pivot(const double* Kb, int n, int bw, int rw, double* w, double* U, double* buf,
                                          int* swaps) {
    constexpr unsigned all = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool rhs_warp = tid >= kPivotCols;
    double* fw = buf + 128 + 64 * warp;  // this warp's multipliers
    int j = tid;                         // this thread's column
    double a[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int d = j - r;
        const bool in = !rhs_warp && j < n && r < n && d <= bw && d >= -bw;
        a[r] = in ? Kb[r * rw + bw + d] : 0.0;
    }
    if (tid == 0)
#pragma unroll
        for (int r = 0; r < R; ++r) buf[r] = a[r];
    int nswap = 0;
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const double* col = buf + 64 * (k & 1);
        // pivot: the diagonal unless a row below beats it strictly, then the first largest.  A NaN on
        // the diagonal is beaten by nothing (band LU), but once rows have been exchanged, as in the
        // dense LU that Strut restarts with, the largest of the others takes its place.
        double v0 = lane < R ? col[lane] : 0.0;
        double v1 = lane + 32 < R ? col[lane + 32] : 0.0;
        const double akk = col[0];
        double piv = akk;
        int p = 0;
        if (__any_sync(all, fabs(v0) > fabs(akk) || fabs(v1) > fabs(akk) || (nswap > 0 && akk != akk))) {
            PivotCandidate best;
            pivot_offer(best, fabs(v0), lane);
            pivot_offer(best, fabs(v1), lane + 32);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
                pivot_merge(best, __shfl_xor_sync(all, best.v, o), __shfl_xor_sync(all, best.row, o));
            if (best.v <= 1.0e-14) return 2;  // the same on every lane of every warp
            p = best.row;
            piv = col[p];
            nswap += p != 0;
        }
        if (fabs(piv) <= 1.0e-14) return 2;
        // the warp's columns: j0 .. j0 + 31
        const int j0 = j - lane;
        const bool touched = rhs_warp || (k + bw + R >= j0 && j0 < n);
        if (touched) {
            const double rp = recip(piv);
            if (p == lane) v0 = akk;  // row k takes the pivot row's place
            if (p == lane + 32) v1 = akk;
            fw[lane] = lane ? quot(v0, piv, rp) : 0.0;
            fw[lane + 32] = quot(v1, piv, rp);
            __syncwarp();
            if (rhs_warp) {
                const double wk = w[k + p], wo = w[k];
                __syncwarp();
                if (lane == 0) {
                    w[k + p] = wo;
                    w[k] = wk;
                }
                __syncwarp();
                if (lane >= 1 && lane <= bw && k + lane < n) w[k + lane] -= fw[lane] * wk;
                if (lane + 32 <= bw && k + lane + 32 < n) w[k + lane + 32] -= fw[lane + 32] * wk;
            } else {
                double u = a[0];
                if (p) {
#pragma unroll
                    for (int r = 1; r < R; ++r)
                        if (r == p) {
                            u = a[r];
                            a[r] = a[0];
                        }
                }
                if (j >= k && j <= k + 2 * bw && j < n) U[(size_t)k * rw + (j - k)] = u;
                const int i = k + R, d = j - i;  // the row that enters
                const bool in = i < n && j < n && d <= bw && d >= -bw;
                const double e = Kb[in ? i * rw + bw + d : 0];
#pragma unroll
                for (int r = 1; r < R; ++r) a[r - 1] = a[r] - fw[r] * u;
                a[R - 1] = in ? e : 0.0;
                if (j == k + 1) {
                    double* next = buf + 64 * ((k + 1) & 1);
#pragma unroll
                    for (int r = 0; r < R; ++r) next[r] = a[r];
                }
                // a warp whose columns are all done takes the next block of columns, which the
                // window has not reached (2 bw + 1 + 32 <= kPivotCols)
                if (j0 + 31 <= k) {
                    j += kPivotCols;
#pragma unroll
                    for (int r = 0; r < R; ++r) a[r] = 0.0;
                }
            }
        }
        __syncthreads();
    }
    *swaps = nswap;
    return 0;
}

// U x = w (U as band_lu_pivot leaves it) in blocks of 32 rows from the end: the warps form the
// rows' sums over the columns behind the block, the first warp solves the block's triangle.  Us:
// n x rw doubles of shared memory for U, t: 32 doubles.
__device__ __forceinline__ void band_pivot_back(const double* U, double* Us, int n, int bw, int rw, const double* w,
                                             double* x, double* t) {
    constexpr unsigned all = 0xffffffffu;
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nt >> 5;
#pragma unroll 4
    for (int q = tid; q < n * rw; q += nt) Us[q] = __ldcg(U + q);
    __syncthreads();
    for (int r1 = n; r1 > 0; r1 -= 32) {
        const int r0 = max(0, r1 - 32), rb = r1 - r0;
        for (int r = warp; r < rb; r += nw) {
            const int i = r0 + r, jmax = min(n - 1, i + 2 * bw);
            double acc = 0.0;
            for (int j = r1 + lane; j <= jmax; j += 32) acc += Us[i * rw + (j - i)] * x[j];
            acc = warp_sum(acc);
            if (lane == 0) t[r] = w[i] - acc;
        }
        __syncthreads();
        if (warp == 0) {
            const int i = r0 + lane;
            const bool in = lane < rb;
            double v = in ? t[lane] : 0.0;
            const double d = in ? Us[i * rw] : 1.0, rd = 1.0 / d;
#pragma unroll 4
            for (int s = rb - 1; s >= 0; --s) {
                const double c = in && lane < s && s - lane <= 2 * bw ? Us[i * rw + (s - lane)] : 0.0;
                const double xs = __shfl_sync(all, quot(v, d, rd), s);
                if (lane == s) v = xs;
                else v -= c * xs;
            }
            if (in) x[i] = v;
        }
        __syncthreads();
    }
}

// Factor and solve: Kb (n x rw, shared memory) is replaced by U, w by L^-1 P w, x the solution.  U:
// n x rw doubles of global memory.  The whole CTA of kPivotThreads threads; bw <= kPivotMaxBw; regular
// systems (quotient.cuh).  Returns 0 or 2 (singular); *swaps: interchanges made.  The window is as high as the
// half band needs, rounded up to 32, 58 or 64 rows: the multipliers' broadcasts are the time (half band
// 56: 313 K cycles with 58 rows, 322 K with 64).
__device__ __forceinline__ int band_pivot_solve(double* Kb, int n, int bw, int rw, double* w, double* x, double* U,
                                                double* buf, int* swaps) {
    const int rc = bw < 32   ? band_lu_pivot<32>(Kb, n, bw, rw, w, U, buf, swaps)
                   : bw < 58 ? band_lu_pivot<58>(Kb, n, bw, rw, w, U, buf, swaps)
                             : band_lu_pivot<64>(Kb, n, bw, rw, w, U, buf, swaps);
    if (rc != 0) return rc;
    band_pivot_back(U, Kb, n, bw, rw, w, x, buf);
    return 0;
}

}  // namespace strut
