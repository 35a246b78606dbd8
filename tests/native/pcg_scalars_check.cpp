// Host check of the PCG's recurrence scalars (edelweissfe_gb300/csrc/pcg_scalars.h): the sums they are made of are kept
// and compared in FP64 for FP32 vectors too, over FP64's range, and rounded only as a vector's factor.
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

#include "../../edelweissfe_gb300/csrc/pcg_scalars.h"

static long bad = 0;
static void expect(bool ok, const char* what) {
    if (!ok && ++bad < 10) std::printf("%s\n", what);
}

template <typename VT>
static void check() {
    std::mt19937_64 g(11);
    std::uniform_real_distribution<double> um(1.0, 2.0), ue(-300.0, 300.0);
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    for (int t = 0; t < 200000; ++t) {
        const double e = std::exp2(std::floor(ue(g)));  // sums of any magnitude, all 53 bits in use
        const double rz = um(g) * e, rr = um(g) * e, pq = um(g) * e, rz2 = um(g) * e, rtol2 = 1e-16 * um(g);
        ef::PcgScalars<VT> s;
        VT f = 7;
        expect(s.start({rz, rr}, rtol2, f) && f == (VT)0 && s.rz == rz && s.bb == rr, "start");
        expect(s.step({pq}, f) && f == (VT)(rz / pq) && s.status == EF_OK, "step");
        const double limit = rtol2 * rr;
        ef::PcgScalars<VT> above = s, at = s;
        expect(above.direction({rz2, std::nextafter(limit, inf)}, f) && f == (VT)(rz2 / rz) && above.rz == rz2 && !above.done,
               "a residual one step above the limit goes on");
        expect(!at.direction({rz2, limit}, f) && at.done && at.finished() && at.status == EF_OK, "the limit ends the solve");
    }
    VT f;
    ef::PcgScalars<VT> s;
    expect(!s.start({0.0, 0.0}, 1e-16, f) && s.status == EF_OK, "a zero right-hand side");
    expect(!s.start({nan, nan}, 1e-16, f), "a right-hand side that is not a number");
    s.start({1.0, 1.0}, 1e-16, f);
    expect(!s.step({-1.0}, f) && s.status == EF_NOT_CONVERGED, "a breakdown keeps the iterate");
    s.status = EF_OK;
    expect(!s.step({nan}, f) && s.status == EF_NAN, "p.q not a number");
    s.status = EF_OK;
    expect(!s.direction({1.0, nan}, f) && s.status == EF_NAN && !s.done, "r.r not a number");
}

int main() {
    check<double>();
    check<float>();
    std::printf("failures %ld\n", bad);
    return bad != 0;
}
