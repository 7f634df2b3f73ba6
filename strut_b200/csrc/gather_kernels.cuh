// Assembly as a kernel of its own, for 3D instances and for every handle with a band in global memory
// (whose kernels read the assembled slots): every band slot and every free dof's F_int sums
// its list of element contributions (in assembly order, as the scatter of
// stiffness_internal_frame2d.mojo:594-619 and its 3D counterpart add them up), times the collapse
// coefficients of multi-point constraints.
//
// The lists are uneven.  A slot between ordinary dofs has up to a few dozen contributions, one
// between the master dofs of a rigid diaphragm thousands, and a thread that walks such a list alone
// pays two dependent loads for each.  So a lane takes a slot of its own up to kShortList
// contributions, and a longer list belongs to the whole warp: it loads 32 contributions at a time
// (indices two chunks ahead, entries one), and the sum runs through them from shared memory.  Either
// way a slot's sum is one chain of multiply-adds in list order.  Spread over the GPU instead of one
// CTA per instance it is bound by the longest list's chain (8.3 cycles a contribution).
// 32 4-story 3x3-bay diaphragm frames: 833 us inside the instance kernel, 30 us here.
#pragma once

#include "solver_kernels.cuh"

namespace strut {

constexpr int kShortList = 24;

// Sum of the contributions [c0, c1) of each lane's list: val[con[c]] times coef[c] (1 without coef).
// All lanes of the warp call; buf: 32 double2 of shared memory of the warp.
__device__ __forceinline__ double gather_list(long long c0, long long c1, const int* __restrict__ con,
                                              const double* __restrict__ coef, const double* __restrict__ val,
                                              double2* buf) {
    constexpr unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double K = 0.0;
    const bool lng = c1 - c0 > kShortList;
    long long c = lng ? c1 : c0;
    // short lists, four contributions in flight per lane
    while (__any_sync(all, c < c1)) {
        int idx[4];
        double f[4], v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool in = c + u < c1;
            idx[u] = in ? __ldg(con + c + u) : -1;
            f[u] = in ? (coef ? __ldg(coef + c + u) : 1.0) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = idx[u] >= 0 ? val[idx[u]] : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (idx[u] >= 0) K += f[u] * v[u];
        c += 4;
    }
    // long lists one after another, the warp together
    for (unsigned todo = __ballot_sync(all, lng); todo; todo &= todo - 1) {
        const int owner = __ffs(todo) - 1;
        const long long b0 = __shfl_sync(all, c0, owner), b1 = __shfl_sync(all, c1, owner);
        auto index = [&](long long p) { return p < b1 ? __ldg(con + p) : -1; };
        auto factor = [&](long long p) { return p < b1 ? (coef ? __ldg(coef + p) : 1.0) : 0.0; };
        int i1 = index(b0 + lane), i2 = index(b0 + 32 + lane);
        double f1 = factor(b0 + lane), f2 = factor(b0 + 32 + lane);
        double v1 = i1 >= 0 ? val[i1] : 0.0;
        double S = 0.0;
        for (long long p = b0; p < b1; p += 32) {
            buf[lane] = make_double2(f1, v1);
            __syncwarp();
            const double v2 = i2 >= 0 ? val[i2] : 0.0;
            f1 = f2;
            i2 = index(p + 64 + lane);
            f2 = factor(p + 64 + lane);
            const int m = (int)min((long long)32, b1 - p);
#pragma unroll
            for (int t = 0; t < 32; t += 8) {
                if (t < m) {  // entries behind the list are 0 * 0
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const double2 e = buf[t + q];
                        S += e.x * e.y;
                    }
                }
            }
            __syncwarp();
            v1 = v2;
        }
        if (lane == owner) K = S;
    }
    return K;
}

// A block's items: 256 band slots of an instance from `first`, or 256 free dofs from -1 - first.  Blocks
// exist for the items there are, in one dimension, so neither the number of instances nor their
// difference in size matters (as a grid of the largest instance's blocks by instances, 65,535 was the limit).
struct GatherBlock {
    int inst, first;
};

// kband: band slots (band_off), fsum: F_int of the free dofs (f_off).
__global__ void __launch_bounds__(256) gather_kernel(const DevInst* __restrict__ insts, InstArrays A, int newton,
                                                     const GatherBlock* __restrict__ blocks,
                                                     double* __restrict__ kband, double* __restrict__ fsum) {
    __shared__ __align__(16) double2 buf[8][32];
    const GatherBlock G = blocks[blockIdx.x];
    const int inst = G.inst, warp = threadIdx.x >> 5;
    if (newton && !A.active[inst]) return;
    const DevInst& I = insts[inst];
    const bool slots = G.first >= 0;
    const int n_items = slots ? I.n * I.rw : I.n;
    const int t = (slots ? G.first : -1 - G.first) + threadIdx.x;
    long long c0 = 0, c1 = 0;
    if (t < n_items) {
        if (slots) {
            c0 = A.slot_ptr[I.slot_ptr_off + t];
            c1 = A.slot_ptr[I.slot_ptr_off + t + 1];
        } else {
            c0 = A.fint_ptr[I.fint_ptr_off + t];
            c1 = A.fint_ptr[I.fint_ptr_off + t + 1];
        }
    }
    const double s = slots ? gather_list(c0, c1, A.slot_contrib, A.slot_coef, A.ek, buf[warp])
                           : gather_list(c0, c1, A.fint_contrib, A.fint_coef, A.ef, buf[warp]);
    if (t < n_items) {
        if (slots) kband[I.band_off + t] = s;
        else fsum[I.f_off + t] = s;
    }
}

// K_init column by column (slot o of row i at o n + i), so that threads that each take a row read it
// coalesced.  One CTA per instance.
__global__ void kinit_by_column_kernel(const DevInst* __restrict__ insts, const double* __restrict__ kinit,
                                       double* __restrict__ out) {
    const DevInst& I = insts[blockIdx.x];
    if (I.large) return;
    for (int t = threadIdx.x; t < I.n * I.rw; t += blockDim.x) {
        const int o = t / I.n, i = t - o * I.n;
        out[I.band_off + t] = kinit[I.band_off + (long long)i * I.rw + o];
    }
}

}  // namespace strut
