// Candidate of a pivot search spread over lanes: the first row of the largest magnitude.  Plain C++, so
// that the search can be run lane by lane on the host as well.
#pragma once

#if defined(__CUDACC__)
#define STRUT_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define STRUT_HOST_DEVICE inline
#endif

namespace strut {

// Starts below every magnitude: a NaN beats no value and is never taken, so the lanes of an exchange
// agree on the row whatever the column holds (a candidate that were a NaN itself would be kept by its
// own lane and refused by the others).
struct PivotCandidate {
    double v = -1.0;       // magnitude; -1: none
    int row = 0x7fffffff;
};

// A lane's rows in increasing order.
STRUT_HOST_DEVICE void pivot_offer(PivotCandidate& c, double v, int row) {
    if (v > c.v) {
        c.v = v;
        c.row = row;
    }
}

// Another lane's candidate.
STRUT_HOST_DEVICE void pivot_merge(PivotCandidate& c, double v, int row) {
    if (v > c.v || (v == c.v && row < c.row)) {
        c.v = v;
        c.row = row;
    }
}

}  // namespace strut
