// The forms of csrc/lb_ff.cuh on the host, for tests/test_ff_host.py: the same
// single roundings (fused multiply-adds are fmaf; built without contraction), the
// reciprocal's approximation replaced by the nearest float and its neighbours.
#include <cmath>
#include <cstdint>
#include <cstring>

static inline float __fmaf_rn(float a, float b, float c) { return fmaf(a, b, c); }
static inline float __int_as_float(int i) { float f; memcpy(&f, &i, 4); return f; }
static inline int __float_as_int(float f) { int i; memcpy(&i, &f, 4); return i; }

#include "../lattibol_0.3.31f_gb300/csrc/lb_ff.cuh"

static int seed_ulps = 0;
namespace lb {
float ff_rcp(float x) { return __int_as_float(__float_as_int(1.f / x) + seed_ulps); }
}  // namespace lb

extern "C" {

// how many of n pairs (a, b) the form add + (a + 2 b) / v decides otherwise than
// the FP64 line
long ratio_wrong(const float *a, const float *b, long n, double v, float add) {
    const lb::FF inv = lb::ff_reciprocal(v);
    long wrong = 0;
    for (long i = 0; i < n; i++) {
        float out;
        if (!lb::ff_ratio(a[i], b[i], inv, add, out)) continue;
        const float line = (float)((double)add + ((double)a[i] + 2. * (double)b[i]) / v);
        wrong += memcmp(&line, &out, 4) != 0;
    }
    return wrong;
}

// every `step`-th float of [lo, hi], the reciprocal's seed off by -1, 0 and +1 ulp:
// the largest relative error of the two floats of 4 exp(-200 / rho), and how many
// of the values that the form decides differ from the FP64 line
double psi_error(float lo, float hi, int step, long *wrong) {
    double worst = 0;
    *wrong = 0;
    for (seed_ulps = -1; seed_ulps <= 1; seed_ulps++)
        for (int i = __float_as_int(lo); i <= __float_as_int(hi); i += step) {
            const float rho = __int_as_float(i);
            float h, l, out;
            if (!lb::ff_psi_parts(rho, h, l)) return INFINITY;
            // the FP64 line's own error, 2^-52 or so, does not show at 2^-35
            const double line = 4. * exp(-200. / (double)rho);
            worst = fmax(worst, fabs(((double)h + (double)l - line) / line));
            const float f = (float)line;
            if (lb::ff_psi_ref(rho, out)) *wrong += memcmp(&f, &out, 4) != 0;
        }
    seed_ulps = 0;
    return worst;
}

}
