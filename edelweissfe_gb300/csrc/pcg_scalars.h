// The scalars of the block-Jacobi PCG recurrence and its three steps (krylov.cu): FP64 for FP64 and FP32 vectors alike,
// rounded to the vectors' type VT only where they multiply one.  The first thread of every CTA keeps them.
#pragma once

#include "../../include/efgpu.h"

#ifdef __CUDACC__
#define EF_PCG_HD __host__ __device__
#else
#define EF_PCG_HD
#endif

namespace ef {

template <typename VT>
struct PcgScalars {
    double rz = 0.0, rr = 0.0, bb = 0.0;
    double limit = 0.0;  // rtol^2 b.b
    int status = EF_OK;
    bool done = false;
    // each returns whether to go on, with the factor of the next vector update in `scalar`
    EF_PCG_HD bool start(const double (&t)[2], double rtol2, VT& scalar) {  // t: r.z, r.r
        rz = t[0];
        rr = bb = t[1];
        limit = rtol2 * bb;
        scalar = (VT)0;
        return bb > 0.0;
    }
    EF_PCG_HD bool step(const double (&t)[1], VT& scalar) {  // t: p.q
        scalar = (VT)(rz / t[0]);
        // NaN, or a breakdown (the current iterate is kept)
        if (!(t[0] > 0.0)) status = t[0] == t[0] ? EF_NOT_CONVERGED : EF_NAN;
        return t[0] > 0.0;
    }
    EF_PCG_HD bool direction(const double (&t)[2], VT& scalar) {  // t: r.z, r.r
        scalar = (VT)(t[0] / rz);
        rz = t[0];
        rr = t[1];
        if (!(rr == rr)) status = EF_NAN;
        done = finished();
        return rr == rr && !done;
    }
    EF_PCG_HD bool finished() const { return rr <= limit; }
};

}  // namespace ef
