// Element-pattern device functions shared by the exact station beam
// (beam.cu) and the learned-surrogate beam (surrogate.cu).
#pragma once

#include "common.cuh"

namespace oskb {

// Dipole far field along phi for a direction with (sin, cos) theta
// (oskar/telescope/station/element/define_evaluate_dipole_pattern.h:3-15).
template <typename T>
__device__ __forceinline__ void dipole(T kL, T cos_kL, T sin_th, T cos_th,
        T phi, T& e_theta, T& e_phi)
{
    T sp, cp;
    sincos(phi, &sp, &cp);
    const T denom = (T) 1 + cp * cp * (cos_th * cos_th - (T) 1);
    if (denom == (T) 0)
    {
        e_theta = e_phi = (T) 0;
        return;
    }
    const T t = (cos(kL * cp * sin_th) - cos_kL) / denom;
    e_theta = -cp * cos_th * t;
    e_phi = sp * t;
}

// Real element-pattern matrix {a, b, c, d} for one direction
// (define_convert_enu_directions_to_theta_phi.h:3-31 then
// define_evaluate_dipole_pattern.h:17-48). pole: the extra point at theta = 0
// whose phi values are the unwrapped offsets.
template <typename T>
__device__ __forceinline__ void element_pattern(T X, T Y, T Z, bool pole,
        T dphi1, T dphi2, T kL, T cos_kL, int swap_xy, T p[4])
{
    T theta, phi1, phi2;
    if (pole)
    {
        theta = (T) 0;
        phi1 = dphi1;
        phi2 = dphi2;
    }
    else
    {
        const T twopi = (T) 2 * (T) kPi;
        const T p0 = atan2(Y, X);
        phi1 = fmod(p0 + dphi1, twopi);
        phi2 = fmod(p0 + dphi2, twopi);
        if (phi1 < (T) 0) phi1 += twopi;
        if (phi2 < (T) 0) phi2 += twopi;
        theta = atan2(sqrt(X * X + Y * Y), Z);
    }
    T st, ct, xt, xp, yt, yp;
    sincos(theta, &st, &ct);
    dipole(kL, cos_kL, st, ct, phi1, xt, xp);
    dipole(kL, cos_kL, st, ct, phi2, yt, yp);
    p[0] = swap_xy ? yt : xt;
    p[1] = swap_xy ? yp : xp;
    p[2] = swap_xy ? xt : yt;
    p[3] = swap_xy ? xp : yp;
}

// The same for a direction away from the zenith from its components alone:
// with r = |(X, Y)| and h = |(X, Y, Z)|, the polar angle has sine r / h and
// cosine Z / h, the azimuth cosine X / r and sine Y / r, and the elements'
// azimuth offsets add by rotation (rot: cos dphi1, sin dphi1, cos dphi2,
// sin dphi2, once per station). Less than half of the 350 FP64 operations
// with the inverse tangents and their sines and cosines. Directions where r
// vanishes (the zenith, whose azimuth is that of the signed zeros) take
// element_pattern.
//
// The pattern's quotient (cos(kL a) - cos kL) / (1 - a^2), a = cos phi sin
// theta, loses its digits towards the dipole's axis (a = 1) as it stands,
// where an angle's rounding does not show in its cosine but a rotated
// cosine's does. Hence 1 - a^2 = sin^2 phi + cos^2 phi cos^2 theta, a sum of
// squares, 1 - |a| from it near the axis, and with d = kL (1 - |a|) the
// numerator as 2 sin(d/2) sin(kL - d/2): a few ulp everywhere. As it stands
// the error, 4.6e-15 rms of one at 1 to 6 degrees from the axis by the
// angles, was 6.9e-15 by the rotated cosines and is 6e-17 or less.
template <typename T>
__device__ __forceinline__ void element_pattern_rotated(T X, T Y, T Z,
        T dphi1, T dphi2, const T* rot, T kL, T cos_kL, T sin_kL, int swap_xy,
        T p[4])
{
    const T r2 = X * X + Y * Y;
    if (!(r2 > (sizeof(T) == 8 ? (T) 1e-280 : (T) 1e-30)))
    {
        element_pattern<T>(X, Y, Z, false, dphi1, dphi2, kL, cos_kL, swap_xy,
                p);
        return;
    }
    const T ri = rsqrt(r2), hi = rsqrt(r2 + Z * Z);
    const T st = r2 * ri * hi, ct = Z * hi;
    const T c0 = X * ri, s0 = Y * ri;
#pragma unroll
    for (int f = 0; f < 2; ++f)
    {
        const T cp = c0 * rot[2 * f] - s0 * rot[2 * f + 1];
        const T sp = s0 * rot[2 * f] + c0 * rot[2 * f + 1];
        const T cc = cp * ct, denom = sp * sp + cc * cc;
        T e_theta = (T) 0, e_phi = (T) 0;
        if (denom != (T) 0)
        {
            const T a = fabs(cp) * st;
            T below = (T) 1 - a;
            if (a > (T) 0.75) below = denom / ((T) 1 + a);
            T s, c;
            sincospi((T) (0.5 / kPi) * kL * below, &s, &c);   // of d / 2
            const T t = (T) 2 * s * (c * sin_kL - s * cos_kL) / denom;
            e_theta = -cc * t;
            e_phi = sp * t;
        }
        const int o = (f == 0) == (swap_xy == 0) ? 0 : 2;
        p[o] = e_theta;
        p[o + 1] = e_phi;
    }
}

}  // namespace oskb
