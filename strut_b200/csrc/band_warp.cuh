// Band factor-solve in shared memory: the LU of narrow bands and the one-warp back substitutions.
//
// Algorithm (paths relative to the Strut project root):
//   BandGeneral  src/mojo/solver/run_case/linear_solver_backend.mojo:631-680, 735-770
//   BandSPD      linear_solver_backend.mojo:689-726, 772-812
//
// A 2D frame's system (36 to 216 unknowns, half band 11 to 20) is a chain of n dependent steps of a
// few hundred operations, so the time is the latency of a step.  Measured for 216 unknowns of half
// band 20 (cycles per unknown): factorisation 1,230 -> 246, back substitution 810 -> 262 (the sums of a row
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
constexpr int kNoColumn = 0x7fffffff;  // no column of the factorisation failed

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
// next to it the instructions of a warp that works alone on its scheduler.  So a step is straight
// code without a branch: no inner loop, no division (74 cycles, 413 with a zero numerator, which
// bands are full of; recip 40, quot 24), no reducing barrier (63 against 28 cycles), and the pivot
// test only folds the first failing column into a key that is looked at after the last step (as
// flags that end the loop it cost 120 of 375 cycles a step).  Every operand has a pointer that moves
// by a fixed stride; rows and columns that a warp or lane does not have point at the zeros z (stride
// 0), and bw rows of zeros behind the band (B has n + bw rows) stand in for the rows the last steps
// lack.
// NR NW >= bw, 32 NC > bw.  rk: 2 doubles; z: 2 doubles; key: an int, all of shared memory; the first
// failing column comes back in *key.
template <int NR, int NC, int NW, bool KEEP>
__device__ __forceinline__ void band_lu_rows(double* B, int n, int bw, int rw, int woff, double* rk, double* z,
                                            int* key) {
    constexpr int NT = 32 * NW, kNone = kNoColumn;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) {
        rk[0] = recip(B[bw]);
        z[0] = z[1] = 0.0;
        *key = kNone;
    }
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
    int first = kNone;  // 2 k: column k needs a swap; 2 k + 1: column k is singular
    bar_first(NT);
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
        const double akk = *pk, rkk = rk[k & 1], d = fabs(akk), dbig = fmax(d, 1.0e-14);
        double f[NR], uk[NC], a[NR][NC];
#pragma unroll
        for (int u = 0; u < NR; ++u) f[u] = *pf[u];
#pragma unroll
        for (int v = 0; v < NC; ++v) {
            uk[v] = *pu[v];
#pragma unroll
            for (int u = 0; u < NR; ++u) a[u][v] = *pa[u][v];
        }
        // pivot search of linear_solver_backend.mojo:640-657: an entry strictly larger than the
        // diagonal selects another row, and the largest one decides singularity (1e-14)
        bool swap = d <= 1.0e-14, big = false;
#pragma unroll
        for (int u = 0; u < NR; ++u) {
            const double q = quot(f[u], akk, rkk);
#pragma unroll
            for (int v = 0; v < NC; ++v) {
                a[u][v] -= q * uk[v];
                *pa[u][v] = a[u][v];
                pa[u][v] += sa[u][v];
            }
            swap = swap || fabs(f[u]) > d;
            big = big || fabs(f[u]) > dbig;
            if constexpr (KEEP) {
                if (u == 0) __syncwarp();  // every lane has read its multipliers' entries
                if (lane == 0 && sf[u]) *const_cast<double*>(pf[u]) = q;
            }
            pf[u] += sf[u];
        }
        const double rn = recip(a[0][0]);
        if (threadIdx.x == 0) rk[(k + 1) & 1] = rn;
        first = min(first, big ? 2 * k : swap ? 2 * k + 1 : kNone);
#pragma unroll
        for (int v = 0; v < NC; ++v) pu[v] += su[v];
        pk += rw;
        bar_first(NT);
    }
    first = __reduce_min_sync(0xffffffffu, first);
    if (lane == 0) atomicMin(key, first);
}

// Rows of zeros that band_lu_rows needs behind the band; the limit on the shared memory of band and
// vectors decides whether they fit (else band_lu_smem runs).
constexpr size_t kBandSmemMax = 220 * 1024;
__host__ __device__ inline int band_pad_rows(int n, int bw, int vectors) {
    return bw <= kLuRowsMax &&
                   ((size_t)(n + bw) * (2 * bw + 1) + (size_t)vectors * n) * sizeof(double) <= kBandSmemMax
               ? bw : 0;
}

// band_lu_rows for half bands up to kLuRowsMax and regular systems (quotient.cuh), by a CTA of
// kLuRowsThreads threads (all of them call).  Returns 0 ok, 2 singular, 6 a row swap would be needed (the
// caller then starts again from the assembled values), the same on all threads.  Four warps up to half
// band 31 (half band 14 / 20: 229 / 246 cycles a step, with eight warps 330 / 318), eight above.
template <bool KEEP>
__device__ __forceinline__ int band_lu_cta(double* B, int n, int bw, int rw, int woff, double* rk, double* z,
                                           int* key) {
    if (bw > 31) {
        band_lu_rows<8, 2, kLuRowsThreads / 32, KEEP>(B, n, bw, rw, woff, rk, z, key);
    } else if (threadIdx.x < 128) {
        if (bw <= 12) band_lu_rows<3, 1, 4, KEEP>(B, n, bw, rw, woff, rk, z, key);
        else if (bw <= 16) band_lu_rows<4, 1, 4, KEEP>(B, n, bw, rw, woff, rk, z, key);
        else if (bw <= 20) band_lu_rows<5, 1, 4, KEEP>(B, n, bw, rw, woff, rk, z, key);
        else band_lu_rows<8, 1, 4, KEEP>(B, n, bw, rw, woff, rk, z, key);
    }
    __syncthreads();
    return *key == kNoColumn ? 0 : *key & 1 ? 2 : 6;
}

// U x = w with one warp for bw <= kBackWarpMax, every row's sum in the reference's order (columns
// upwards from the diagonal, so the chain of a row runs through all its bw products, the newest
// unknown's first).  The unknowns a row needs and the next row's entries are in registers, so a row
// costs its chain and a quotient (bw 20: 262 cycles; one lane with its operands in shared memory
// took 810).  EXACT: bw == BW; else bw <= BW.  Slots of columns outside the matrix hold zeros.
// rd: n doubles of scratch.  Where an unknown is not finite, it and those before
// it come out as NaN, x[0] with them (each takes up the one behind it, if only times zero).
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
// from the next.  rd: n doubles of scratch.  Not finite: as in band_back_lu.
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
