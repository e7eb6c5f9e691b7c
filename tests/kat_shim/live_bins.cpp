// live_z() of the marcher for tests/test_live_bins_cpu.py: the largest bin mass,
// as the marcher computes it, between any two borders beyond the limit.
#include <algorithm>

#include "../../differentiable_gaussian_mixture_renderer_b200/csrc/dgmr_live_bins.h"

namespace {
template <class T>
T cdf(T z)
{
    return T(0.5) * (T(1) + dgmr_fm::erf_f(z));
}

template <class T>
void run(const double* mor, long n, long points, double* limit, double* largest)
{
    for (long i = 0; i < n; ++i) {
        const T m = T(mor[i]), z0 = dgmr::live_z(m);
        T worst = T(0);
        for (int side = -1; side <= 1; side += 2) {
            T lo = cdf(T(side) * T(50)), hi = lo;
            for (long k = 0; k <= points; ++k) {
                const T c = cdf(T(side) * (z0 + T(6) * T(k) / T(points)));
                lo = std::min(lo, c);
                hi = std::max(hi, c);
            }
            worst = std::max(worst, (hi - lo) * m);
        }
        limit[i] = double(z0);
        largest[i] = double(worst);
    }
}
} // namespace

extern "C" void live_bins(int is_double, const double* mor, long n, long points, double* limit, double* largest)
{
    if (is_double)
        run<double>(mor, n, points, limit, largest);
    else
        run<float>(mor, n, points, limit, largest);
}
