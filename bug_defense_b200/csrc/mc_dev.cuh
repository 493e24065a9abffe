// What both photon tracers (mc.cu, mc_fluence.cu) share: the kernel parameters, the physics at a face, the
// scattering and the launch offsets.
#pragma once

#include "common.cuh"

namespace bd {

struct McDev {
    int nx, ny, nz, launch_axis;
    float dx, dy, dz, lx, ly, lz;
    float ux0, uy0, uz0, cos_ph, sin_ph, cos_th_safe;
    float xc, yc, zc, sigma, radius;
    int profile;
    float n_amb, rmax2;
    int options;
    long long n_photons, offset;
    long long max_events;
    float fnx, fny, fnz;
    uint32_t keys[20];   // the seed's Philox round keys
    unsigned long long seed;
    float eq_eps;     // Fresnel index-equality guard
    float step_eps;   // internal index-step threshold
    float entry_eps;  // entrance refraction threshold
};

__device__ __forceinline__ float fresnel_unpol(float n1, float n2, float cos_i, float eq_eps) {
    // voxel_mc_3d.py:33-48 / voxel_mc_metal.py:70-83
    if (fabsf(n1 - n2) < eq_eps) return 0.0f;
    cos_i = fminf(1.0f, fabsf(cos_i));
    if (cos_i > 0.999999f) {
        float r = (n1 - n2) / (n1 + n2);
        return r * r;
    }
    float q = n1 / n2;
    float sin_t2 = q * q * (1.0f - cos_i * cos_i);
    if (sin_t2 >= 1.0f) return 1.0f;
    float cos_t = sqrtf(1.0f - sin_t2);
    float a = n1 * cos_i, b = n2 * cos_t, c = n1 * cos_t, d = n2 * cos_i;
    float rs = (a - b) / (a + b);
    float rp = (c - d) / (c + d);
    return 0.5f * (rs * rs + rp * rp);
}

// Snell refraction across an axis-aligned face (voxel_mc_3d.py:51-69)
__device__ __forceinline__ void refract_axis(float& ux, float& uy, float& uz, int axis, float eta) {
    if (axis == 0) {
        float s = ux > 0.0f ? 1.0f : -1.0f;
        uy *= eta; uz *= eta;
        ux = s * sqrtf(fmaxf(0.0f, 1.0f - uy * uy - uz * uz));
    } else if (axis == 1) {
        float s = uy > 0.0f ? 1.0f : -1.0f;
        ux *= eta; uz *= eta;
        uy = s * sqrtf(fmaxf(0.0f, 1.0f - ux * ux - uz * uz));
    } else {
        float s = uz > 0.0f ? 1.0f : -1.0f;
        ux *= eta; uy *= eta;
        uz = s * sqrtf(fmaxf(0.0f, 1.0f - ux * ux - uy * uy));
    }
}

// Henyey-Greenstein deflection + uniform azimuth (voxel_mc_3d.py:229-262); xi, xphi: uniforms
__device__ __forceinline__ void scatter_hg(float& ux, float& uy, float& uz, float g, float xi, float xphi) {
    float cost;
    if (fabsf(g) < 1e-4f) {
        cost = 2.0f * xi - 1.0f;
    } else {
        float t = (1.0f - g * g) / (1.0f - g + 2.0f * g * xi);
        cost = (1.0f + g * g - t * t) / (2.0f * g);
        cost = fminf(1.0f, fmaxf(-1.0f, cost));
    }
    float sint = sqrtf(fmaxf(0.0f, 1.0f - cost * cost));
    float sinp, cosp;
    sincospif(2.0f * xphi, &sinp, &cosp);
    float nx, ny, nz;
    if (fabsf(uz) > 0.99999f) {
        float sz = uz > 0.0f ? 1.0f : -1.0f;
        nx = sint * cosp;
        ny = sint * sinp;
        nz = cost * sz;
    } else {
        float den = sqrtf(fmaxf(1.0f - uz * uz, 1e-12f));
        float f = sint / den;
        nx = f * (ux * uz * cosp - uy * sinp) + ux * cost;
        ny = f * (uy * uz * cosp + ux * sinp) + uy * cost;
        nz = -sint * cosp * den + uz * cost;
    }
    float nn = nx * nx + ny * ny + nz * nz;
    if (nn > 1e-24f) {
        float r = rsqrtf(nn);
        nx *= r; ny *= r; nz *= r;
    }
    ux = nx; uy = ny; uz = nz;
}

// Transverse launch offsets (voxel_mc_3d.py:101-120)
template <class Rng>
__device__ __forceinline__ void beam_offsets(const McDev& P, Rng& rng, float& u1, float& u2) {
    if (P.profile == BD_BEAM_TOPHAT) {
        float r = P.radius * sqrtf(rng.uniform(P.keys));
        float s, c;
        sincospif(2.0f * rng.uniform(P.keys), &s, &c);
        u1 = r * c; u2 = r * s;
        return;
    }
    if (P.profile == BD_BEAM_KIM_EXP_DISK || P.profile == BD_BEAM_KIM_GAUSS_DISK) {
        float rn = 0.0f;
        // rejection sampling; acceptance >= e^-2, so 256 tries all fail with p < 1e-16
        for (int t = 0; t < 256; ++t) {
            rn = sqrtf(rng.uniform(P.keys));
            float acc = (P.profile == BD_BEAM_KIM_EXP_DISK) ? expf(-2.0f * rn) : expf(-2.0f * rn * rn);
            if (rng.uniform(P.keys) < acc) break;
        }
        float s, c;
        sincospif(2.0f * rng.uniform(P.keys), &s, &c);
        u1 = P.radius * rn * c; u2 = P.radius * rn * s;
        return;
    }
    // Gaussian: Box-Muller pair with per-axis sigma
    float a = rng.uniform_pos(P.keys);
    float b = rng.uniform(P.keys);
    float r = sqrtf(-2.0f * logf(a)) * P.sigma;
    float s, c;
    sincospif(2.0f * b, &s, &c);
    u1 = r * c; u2 = r * s;
}

// Traces the photons with the FP32 tallies' kernel (mc_fluence.cu) into `blocks` ledger rows, zeroed before.
int mc_fluence_launch(const McDev& d, const float4* props, const uint8_t* flags, float* A, unsigned long long* tally64,
                      float* L, double* latz, unsigned long long* queue, double* partials, int max_blocks, int sm_count,
                      cudaStream_t st, const long long* offset_dev, int* blocks);

}  // namespace bd
