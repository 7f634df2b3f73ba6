// Initial committed fiber history (UniMaterialState(mat_def), core.mojo:203-263) written on the
// device: a batch's history is hundreds of megabytes, most of it zeros, and only the few fields
// below differ from zero (the arrays arrive zeroed).  Bound: HBM writes.  256 frames (11.6 M fibers):
// the host loop and its copy took 205 ms of a handle's creation, this 0.1 ms.
#pragma once

#include "element_kernels.cuh"
#include "kat_kernels.cuh"

namespace strut {

__device__ __forceinline__ void init_s2(const DevMat& m, double* F, long long N) {
    F[2 * N] = m.p[1];
    F[4 * N] = m.k[S2K_EPSY];
    F[3 * N] = -m.k[S2K_EPSY];
    if (m.p[10] != 0.0) {
        F[0] = m.k[S2K_SIGINI_E0];
        F[N] = m.p[10];
    }
}

// One CTA per element.
__global__ void init_history_kernel(const DevElem* __restrict__ elems, Geo g, FiberState fs) {
    const DevElem& E = elems[blockIdx.x];
    const DevSection& sd = g.secs[E.sec];
    const int nip = E.nip;
    int base = sd.geo_off;
    for (int t = threadIdx.x; t < nip * sd.n_s2; t += blockDim.x) {
        const DevMat& m = g.mats[g.m[base + t % sd.n_s2]];
        double* F = fs.s2 + E.s2_off + t;
        init_s2(m, F, fs.s2_n);
        S2State c;
        c.eps = F[0];
        c.sig = F[fs.s2_n];
        c.epsmin = F[3 * fs.s2_n];
        c.epsmax = F[4 * fs.s2_n];
        c.epspl = c.epss0 = c.sigs0 = c.epsr = c.sigr = 0.0;
        c.kon = 0;
        double* D = fs.s2d + 14ll * E.s2_off + t;
        store_s2d(m, c, true, D, E.s2_blk);
        store_s2d(m, c, false, D, E.s2_blk);
    }
    base += sd.n_s2;
    for (int t = threadIdx.x; t < nip * sd.n_c2; t += blockDim.x) {
        const DevMat& m = g.mats[g.m[base + t % sd.n_c2]];
        C2State c;
        c.eps = c.sig = c.ecmin = c.dept = 0.0;
        c.tan = m.k[C2K_EC0];
        fs.c2[2 * fs.c2_n + E.c2_off + t] = c.tan;
        store_c2d(m, c, fs.c2d + 5ll * E.c2_off + t, E.c2_blk);
    }
    base += sd.n_c2;
    for (int t = threadIdx.x; t < nip * sd.n_s1; t += blockDim.x)
        fs.s1[2 * fs.s1_n + E.s1_off + t] = g.mats[g.m[base + t % sd.n_s1]].p[1];
    base += sd.n_s1;
    for (int t = threadIdx.x; t < nip * sd.n_c1; t += blockDim.x) {
        const double e = g.mats[g.m[base + t % sd.n_c1]].k[C1K_EC0];
        fs.c1[2 * fs.c1_n + E.c1_off + t] = e;
        fs.c1[5 * fs.c1_n + E.c1_off + t] = e;
    }
}

// The bs.n_inst copies of section sd of a section batch: one thread per fiber and instance.
__global__ void init_batch_kernel(Geo g, DevSection sd, BatchState bs) {
    const int nf = sd.n_s2 + sd.n_c2 + sd.n_s1 + sd.n_c1;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long i = t / nf;
    if (i >= bs.n_inst) return;
    int j = (int)(t - i * nf);
    const DevMat& m = g.mats[g.m[sd.geo_off + j]];
    if (j < sd.n_s2) {
        init_s2(m, bs.s2 + i * bs.p_s2 + j, bs.n_inst * bs.p_s2);
        return;
    }
    j -= sd.n_s2;
    if (j < sd.n_c2) {
        bs.c2[2 * bs.n_inst * bs.p_c2 + i * bs.p_c2 + j] = m.k[C2K_EC0];
        return;
    }
    j -= sd.n_c2;
    if (j < sd.n_s1) {
        bs.s1[2 * bs.n_inst * bs.p_s1 + i * bs.p_s1 + j] = m.p[1];
        return;
    }
    j -= sd.n_s1;
    bs.c1[2 * bs.n_inst * bs.p_c1 + i * bs.p_c1 + j] = m.k[C1K_EC0];
    bs.c1[5 * bs.n_inst * bs.p_c1 + i * bs.p_c1 + j] = m.k[C1K_EC0];
}

}  // namespace strut
