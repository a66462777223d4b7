// tild_uk.cuh -- û(k) of the potentials and its strain derivative, FP64 (device).
#pragma once
#include "tild_device.h"

namespace tild {

// û(k) of each potential kind, FP64 (ps_potentialGaussian.cu:38-46,
// ps_potentialErf2.cu:111-124, ps_potentialErfG.cu:177-190, ps_potentialCharges.cu:241-258),
// as amplitude x shape: the shape is fixed for a box, the amplitude follows the ramp.
__device__ __forceinline__ double uk_shape(const PotDev &p, double k2)
{
    const double PI4 = 12.566370614359172953850573533118;
    if (p.kind == POT_WALL) return 0.0;   // a per-particle term, nothing in k-space
    if (p.kind == POT_GAUSSIAN) return exp(-0.5 * k2 * p.sig2);
    if (p.kind == POT_CHARGES) return k2 > 0.0 ? PI4 * p.lB * exp(-k2 * p.sig2) / k2 : 0.0;
    const double R = p.Rp;
    double t;
    if (k2 == 0.0) {
        t = PI4 * R * R * R / 3.0;
        return p.kind == POT_ERF2 ? t * t : t;
    }
    const double k = sqrt(k2);
    double sn, cs;
    sincos(R * k, &sn, &cs);
    t = PI4 * (sn - R * k * cs) / (k2 * k);
    const double gs = exp(-0.5 * k2 * p.sig2);
    return p.kind == POT_ERF2 ? gs * t * t : gs * t;
}

__device__ __forceinline__ double uk_amp(const PotDev &p) { return p.kind == POT_CHARGES ? 1.0 : p.amp; }

__device__ __forceinline__ double uk_eval(const PotDev &p, double k2) { return uk_amp(p) * uk_shape(p, k2); }

// (d û / d k) / k for k > 0, FP64, amplitude included: the strain derivative of the pair
// energy.  gaussian: -sigma^2 û; charges: û (-2 sigma^2 - 2/k^2); erf2/erfG with
// t = 4 pi (sin Rk - Rk cos Rk)/k^3: A g t^(p-1) (-sigma^2 t + p t'/k),
// t'/k = 4 pi (R^2 sin(Rk)/k^3 - 3 (sin Rk - Rk cos Rk)/k^5).
__device__ __forceinline__ double uk_dk_over_k(const PotDev &p, double k2)
{
    if (k2 <= 0.0 || p.kind == POT_WALL) return 0.0;
    if (p.kind == POT_GAUSSIAN) return -p.sig2 * uk_eval(p, k2);
    if (p.kind == POT_CHARGES) return uk_eval(p, k2) * (-2.0 * p.sig2 - 2.0 / k2);
    const double PI4 = 12.566370614359172953850573533118;
    const double R = p.Rp, k = sqrt(k2);
    double sn, cs;
    sincos(R * k, &sn, &cs);
    const double f = sn - R * k * cs;
    const double t = PI4 * f / (k2 * k);
    const double dt_k = PI4 * (R * R * sn / (k2 * k) - 3.0 * f / (k2 * k2 * k));
    const double gs = exp(-0.5 * k2 * p.sig2);
    return p.kind == POT_ERF2 ? p.amp * gs * t * (-p.sig2 * t + 2.0 * dt_k) : p.amp * gs * (-p.sig2 * t + dt_k);
}

// both at once, sharing the exponential where the kinds allow it
__device__ __forceinline__ void uk_and_derivative(const PotDev &p, double k2, double &u, double &du)
{
    u = uk_eval(p, k2);
    if (k2 <= 0.0 || p.kind == POT_WALL) du = 0.0;
    else if (p.kind == POT_GAUSSIAN) du = -p.sig2 * u;
    else if (p.kind == POT_CHARGES) du = u * (-2.0 * p.sig2 - 2.0 / k2);
    else du = uk_dk_over_k(p, k2);
}

}  // namespace tild
