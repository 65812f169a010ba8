// Plain FP64 spectrum, tensor and time-resolved integrand (the default kernel), spectrum_direct.cu.
#pragma once

#include "device_common.cuh"

namespace bgw {

// Device pointers of one spectrum, tensor or integrand job.
struct DirectInputs {
    const D4* bub;  // rotated frames (kn, n_tot)
    const uint32_t* sel;
    const double* tau;  // (kn, n_sel, n_cos n_phi)
    const double* cos_t;
    const double* sin2;
    const double* cos2;
    const double* sinphi;  // tensor form
    const double* cosphi;
    const double* coeffs;
    const double* powers;
    const double* t_arr;
    const double* cutw;
    const double* w;
};

// Spectrum (or tensor) of kn frames: out (kn, G, S, W) with G = 2 (+, x) or 6 (xx, xy, xz, yy, yz,
// zz).  Returns the number of kernel launches.
uint64_t launch_direct(Device* dev, const SpectrumJob& job, const DirectInputs& in, size_t kn, double2* out);

// Time-resolved integrand of one frame: out (G, S, W, n_t).
uint64_t launch_direct_integrand(Device* dev, const SpectrumJob& job, const DirectInputs& in, double2* out);

// Device bytes per k-hat frame of the work arrays that grow with the frames.
size_t direct_bytes_per_frame(const SpectrumJob& job);

}  // namespace bgw
