// How far out on a ray a Gaussian's bins can pass the mass test of 1e-5 (host
// and device code): in z = (x - centre) / (sd sqrt(2)).
#pragma once

#include "dgmr_fmath.h"

namespace dgmr {

template <class T>
DGMR_HD T tail_z();
template <>
DGMR_HD float tail_z<float>() { return 3.92f; }
template <>
DGMR_HD double tail_z<double>() { return 5.0; }

// A Gaussian with mass mor on the ray reaches the mass test of a bin less far
// out: the tail of the CDF beyond z >= 2 is erfc(z) / 2 <= exp(-z^2) / (4 sqrt(pi)), so
// a bin that lies wholly beyond the z where this is (1e-5 / mor) holds less than
// 1e-5.  The computed CDF difference exceeds the true one by less than the
// margin (float: 2 x 0.75e-7 of A&S 7.1.26 plus the roundings of two values below 1).
template <class T>
DGMR_HD T tail_margin();
template <>
DGMR_HD float tail_margin<float>() { return 1e-6f; }
template <>
DGMR_HD double tail_margin<double>() { return 1e-13; }
template <class T>
DGMR_HD T live_z(T mor)
{
    const T tail = T(0.999e-5) / mor - tail_margin<T>();
    if (!(tail > T(1e-9)))
        return tail_z<T>();
    return dgmr_fm::min_f(tail_z<T>(), dgmr_fm::sqrt_f(dgmr_fm::max_f(T(4), -dgmr_fm::log_f(T(7.0898154) * tail))));
}

} // namespace dgmr
