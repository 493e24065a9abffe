// Voxel Monte Carlo photon transport (hop-drop-spin with optical-depth voxel marching).
//
// Algorithm follows the reference CPU tracer simulation/voxel_mc_3d.py:123-337
// (_trace_one_photon) and its Metal twin simulation/voxel_mc_metal.py:173-332:
//   launch (Gaussian / top-hat / Kim disks, oblique footprint stretch u1/cos(theta))
//   -> deterministic entrance Fresnel split + Snell refraction
//   -> loop: tau = -ln(xi) consumed voxel by voxel; collision absorbs w*mu_a/mu_t,
//      Russian roulette at w < 1e-4 (survive 1/10 with w*10), Henyey-Greenstein scatter;
//      face crossings do Fresnel/TIR or Snell at index steps, exits tally R_diff / T / lateral.
//
// B200 design:
//   * one persistent grid, photons handed out by a global atomic queue; every lane advances its
//     photon by one event per loop iteration and takes a new photon as soon as its own ends, so
//     warps stay full while the per-photon event counts differ by orders of magnitude;
//   * a crossing is free of branches (the crossed axis by selection), interactions wait for company,
//     and few photons are spread over half of the resident warps: a warp runs the union of its lanes' paths;
//   * Philox-4x32-10 counter-based RNG keyed on (seed, photon index): no RNG state in memory
//     and a photon's path does not depend on which thread traced it;
//   * optical properties packed as one float4 {mu_t, mu_a/mu_t, g, n} per voxel read through
//     the read-only (L1/texture) path: one 16-byte load per event;
//   * absorbed weight tallied with fire-and-forget reductions into an exact fixed-point map (launches
//     whose sums are FP32 in memory run mc_fluence.cu's kernel);
//   * FP64 ledger: per-thread FP64 registers for the per-event channels, per-block partial rows for
//     the per-photon channels, reduced in a fixed order.
// What bounds it: instructions. At 1.5 M photons about 19 warp instructions an event at 12 active
// lanes; at 15 k the longest history (1900 events) at ~1300 clocks an event, an L2 round trip and a
// hundred dependent instructions. Traces of the 200x200x128 stack, before the changes of this list
// and after: 15 k photons 2.04 -> 1.40 ms, 150 k 2.95 -> 2.09 ms, 1.5 M 14.2 -> 8.6 ms; same maps.
#include "mc_dev.cuh"

#include <stdlib.h>

#include <algorithm>
#include <atomic>
#include <mutex>

namespace bd {

// Per-thread FP64 accumulator for the per-collision channel (absorbed weight); the rare
// channels (exits, roulette, truncation, absorption in void) go straight to the block's
// partial row with FP64 atomics, so no block-wide barrier is needed anywhere in the kernel.
struct ThreadLedger {
    double absorbed, absorbed_void;
    unsigned collisions, crossings, reflections;
};

// The photon a lane is tracing. The kernel advances every lane by one event per loop iteration,
// and a lane whose photon has ended takes the next photon from the queue in the same loop, so the
// lanes of a warp are not held back until the warp's longest photon ends (event counts per photon
// differ by orders of magnitude). A photon's random stream and arithmetic do not depend on the
// lane that traces it or on when it is traced.
struct PhotonState {
    PhotonRng rng;
    float x, y, z, ux, uy, uz;
    float iux, iuy, iuz;   // 1 / u, or 1 along an axis the photon does not move on
    float gx, gy, gz;      // voxel indices (whole numbers up to kMcMaxAxis, exact in FP32)
    float ox, oy, oz;      // the exit face's offset from them: 1 or 0 by direction, kFar when not moving
    float tau, w;
    float4 pr;
    int idx;
    unsigned ev;
};

// The longest axis whose indices, and the one past its end, are exact in FP32: beyond it gx + 1 == gx, and
// the photon's linear index would walk out of the grid unseen.
constexpr int kMcMaxAxis = 1 << 24;
// The largest event cap that a photon's 32-bit counter can reach.
constexpr long long kMcMaxEvents = 0xffffffffLL;

// Puts the exit face of an axis without motion out of reach: its distance is about 1e30 voxels.
constexpr float kFar = 1e30f;

// What a crossing needs of a new direction.
__device__ __forceinline__ void photon_aim(PhotonState& s) {
    const bool mx = fabsf(s.ux) > 1e-15f, my = fabsf(s.uy) > 1e-15f, mz = fabsf(s.uz) > 1e-15f;
    s.iux = mx ? 1.0f / s.ux : 1.0f;
    s.iuy = my ? 1.0f / s.uy : 1.0f;
    s.iuz = mz ? 1.0f / s.uz : 1.0f;
    s.ox = mx ? (s.ux > 0.0f ? 1.0f : 0.0f) : kFar;
    s.oy = my ? (s.uy > 0.0f ? 1.0f : 0.0f) : kFar;
    s.oz = mz ? (s.uz > 0.0f ? 1.0f : 0.0f) : kFar;
}

// Launch: transverse offsets, footprint test, entrance Fresnel split and refraction, first
// optical depth. Returns false when the photon never enters the grid (booked here).
template <int DEPTH>  // 2: launch along +z at z=0 ; 0: launch along +x at x=0
__device__ __forceinline__ bool photon_launch(const McDev& P, long long pid, const float4* __restrict__ props,
                                              double* __restrict__ latz, double* sl, PhotonState& s) {
    s.rng.init((unsigned long long)(P.offset + pid), P.keys);
    float u1, u2;
    int ix, iy, iz;
    beam_offsets(P, s.rng, u1, u2);
    const float stretch = u1 / P.cos_th_safe;
    if (DEPTH == 2) {
        s.x = P.xc + stretch * P.cos_ph - u2 * P.sin_ph;
        s.y = P.yc + stretch * P.sin_ph + u2 * P.cos_ph;
        s.z = 0.0f;
        bool out = s.x < 0.0f || s.x >= P.lx || s.y < 0.0f || s.y >= P.ly;
        if (!out && P.rmax2 > 0.0f) {
            float a = s.x - P.xc, b = s.y - P.yc;
            out = a * a + b * b >= P.rmax2;
        }
        if (out) {
            atomicAdd(&sl[BD_LEDGER_LATERAL], 1.0);
            if (latz) atomicAdd(&latz[0], 1.0);
            return false;
        }
        ix = min((int)(s.x / P.dx), P.nx - 1);
        iy = min((int)(s.y / P.dy), P.ny - 1);
        iz = 0;
    } else {
        s.x = 0.0f;
        s.y = P.yc + stretch * P.cos_ph - u2 * P.sin_ph;
        s.z = P.zc + stretch * P.sin_ph + u2 * P.cos_ph;
        bool out = s.y < 0.0f || s.y >= P.ly || s.z < 0.0f || s.z >= P.lz;
        if (!out && P.rmax2 > 0.0f) {
            float a = s.y - P.yc, b = s.z - P.zc;
            out = a * a + b * b >= P.rmax2;
        }
        if (out) {
            atomicAdd(&sl[BD_LEDGER_LATERAL], 1.0);
            if (latz) atomicAdd(&latz[0], 1.0);
            return false;
        }
        ix = 0;
        iy = min((int)(s.y / P.dy), P.ny - 1);
        iz = min((int)(s.z / P.dz), P.nz - 1);
    }
    s.ux = P.ux0; s.uy = P.uy0; s.uz = P.uz0;
    s.gx = (float)ix; s.gy = (float)iy; s.gz = (float)iz;
    s.idx = ix * (P.ny * P.nz) + iy * P.nz + iz;

    // entrance face: deterministic specular split + refraction (voxel_mc_3d.py:183-192)
    s.pr = __ldg(&props[s.idx]);
    {
        float n_in = s.pr.w;
        float cos_in = (DEPTH == 2) ? s.uz : s.ux;
        float r = fresnel_unpol(P.n_amb, n_in, cos_in, P.eq_eps);
        s.w = 1.0f - r;
        // the ledger books what the FP32 weight actually lost, so it closes exactly
        atomicAdd(&sl[BD_LEDGER_SPECULAR], 1.0 - (double)s.w);
        if (s.w <= 0.0f) return false;
        if (fabsf(n_in - P.n_amb) > P.entry_eps) refract_axis(s.ux, s.uy, s.uz, DEPTH, P.n_amb / n_in);
    }
    photon_aim(s);
    s.tau = -__logf(fmaxf(s.rng.uniform(P.keys), 1e-12f));
    s.ev = 0u;
    return true;
}

// An interaction inside the voxel (voxel_mc_3d.py:203-262), st along the path. Returns false when the
// photon has ended (its weight booked).
template <int DEPTH>
__device__ __forceinline__ bool photon_collide(const McDev& P, const uint8_t* __restrict__ flags,
                                               unsigned long long* __restrict__ A64, double* __restrict__ latz, double* sl,
                                               ThreadLedger& tl, PhotonState& s) {
    // the void flag only sorts the ledger: loaded first, used last
    const unsigned fl = flags != nullptr ? (unsigned)__ldg(&flags[s.idx]) : 0u;
    ++tl.collisions;
    const float st = s.tau / s.pr.x;
    s.x += st * s.ux; s.y += st * s.uy; s.z += st * s.uz;
    if (P.rmax2 > 0.0f) {
        float a = (DEPTH == 2) ? s.x - P.xc : s.y - P.yc;
        float b = (DEPTH == 2) ? s.y - P.yc : s.z - P.zc;
        if (a * a + b * b >= P.rmax2) {
            atomicAdd(&sl[BD_LEDGER_LATERAL], (double)s.w);
            if (latz) atomicAdd(&latz[(int)(DEPTH == 2 ? s.gz : s.gx)], (double)s.w);
            return false;
        }
    }
    const float dw = __fmul_rn(s.w, s.pr.y);
    const float w_new = __fsub_rn(s.w, dw);
    atomicAdd(&A64[s.idx], __float2ull_rn(dw * kTallyScale));
    const double lost = (double)s.w - (double)w_new;  // exact: both are FP32 values
    s.w = w_new;
    bool alive = true;
    if (s.w < 1e-4f) {
        if (s.rng.uniform(P.keys) < 0.1f) {
            const float w10 = s.w * 10.0f;
            atomicAdd(&sl[BD_LEDGER_ROULETTE_GAIN], (double)w10 - (double)s.w);
            s.w = w10;
        } else {
            atomicAdd(&sl[BD_LEDGER_ROULETTE_LOSS], (double)s.w);
            alive = false;
        }
    }
    if (alive) {
        uint32_t u0, u1, u2;
        s.rng.next3(u0, u1, u2, P.keys);
        scatter_hg(s.ux, s.uy, s.uz, s.pr.z, PhotonRng::to_uniform(u0), PhotonRng::to_uniform(u1));
        photon_aim(s);
        s.tau = -__logf(fmaxf(PhotonRng::to_uniform(u2), 1e-12f));
    }
    const bool in_void = (fl & BD_FLAG_ABLATED) != 0u;
    tl.absorbed += in_void ? 0.0 : lost;
    tl.absorbed_void += in_void ? lost : 0.0;
    return alive;
}

// The FP32 operations whose contraction the compiler may choose (face distance, optical depth, weight)
// are written out: every photon's history depends on each of their bits.
//
// One event of the hop-drop-spin loop (voxel_mc_3d.py:194-337): the exit face's crossing, or `hit` when
// the photon interacts inside the voxel first (photon_collide completes that event). Returns false
// when the photon has ended (its weight booked).
template <int DEPTH>
__device__ __forceinline__ bool photon_move(const McDev& P, const float4* __restrict__ props, double* __restrict__ latz,
                                            double* sl, ThreadLedger& tl, PhotonState& s, bool metal, bool& hit) {
    // exact ray/box distance to the exit face (voxel_mc_3d.py:72-98)
    const float fx = s.gx + s.ox, fy = s.gy + s.oy, fz = s.gz + s.oz;
    const float sx = __fmaf_rn(fx, P.dx, -s.x) * s.iux;
    const float sy = __fmaf_rn(fy, P.dy, -s.y) * s.iuy;
    const float sz = __fmaf_rn(fz, P.dz, -s.z) * s.iuz;
    const bool ax0 = sx <= sy && sx <= sz, ax1 = !ax0 && sy <= sz;
    const float s_exit = fmaxf(ax0 ? sx : (ax1 ? sy : sz), 0.0f);
    const float mu_t = s.pr.x;
    const float depth_out = __fmul_rn(mu_t, s_exit);
    if (mu_t > 1e-12f && depth_out >= s.tau) {
        hit = true;
        return true;
    }

    // ---- traverse the chord and land exactly on the exit face: everything of the crossed axis by
    // selection, so that lanes that cross different faces stay together ----
    ++tl.crossings;
    s.tau = __fsub_rn(s.tau, depth_out);
    const float ua = ax0 ? s.ux : (ax1 ? s.uy : s.uz);
    const bool fwd = ua > 0.0f;
    const float face = (ax0 ? fx : (ax1 ? fy : fz)) * (ax0 ? P.dx : (ax1 ? P.dy : P.dz));
    const float cell = (ax0 ? s.gx : (ax1 ? s.gy : s.gz)) + (fwd ? 1.0f : -1.0f);
    s.x = ax0 ? face : s.x + s_exit * s.ux;
    s.y = ax1 ? face : s.y + s_exit * s.uy;
    s.z = ax0 || ax1 ? s.z + s_exit * s.uz : face;
    const bool depth = DEPTH == 2 ? !(ax0 || ax1) : ax0;
    if (cell < 0.0f || cell >= (ax0 ? P.fnx : (ax1 ? P.fny : P.fnz))) {
        if (!depth) {
            atomicAdd(&sl[BD_LEDGER_LATERAL], (double)s.w);
            if (latz) atomicAdd(&latz[(int)(DEPTH == 2 ? s.gz : s.gx)], (double)s.w);
            return false;
        }
        if (fwd) {
            atomicAdd(&sl[BD_LEDGER_TRANSMITTED], (double)s.w);
            return false;
        }
        // leaving through the entrance face: Fresnel / TIR against ambient
        float r = fresnel_unpol(s.pr.w, P.n_amb, ua, P.eq_eps);
        if (r > 0.0f && s.rng.uniform(P.keys) < r) {
            ++tl.reflections;
            if (DEPTH == 2) { s.uz = -s.uz; s.iuz = -s.iuz; s.oz = 1.0f; }
            else { s.ux = -s.ux; s.iux = -s.iux; s.ox = 1.0f; }
            return true;
        }
        atomicAdd(&sl[BD_LEDGER_DIFFUSE], (double)s.w);
        return false;
    }
    if (!metal && P.rmax2 > 0.0f) {
        float a = (DEPTH == 2) ? s.x - P.xc : s.y - P.yc;
        float b = (DEPTH == 2) ? s.y - P.yc : s.z - P.zc;
        if (a * a + b * b >= P.rmax2) {
            atomicAdd(&sl[BD_LEDGER_LATERAL], (double)s.w);
            if (latz) atomicAdd(&latz[(int)(DEPTH == 2 ? s.gz : s.gx)], (double)s.w);
            return false;
        }
    }
    const int stride = ax0 ? P.ny * P.nz : (ax1 ? P.nz : 1);
    const int jidx = s.idx + (fwd ? stride : -stride);
    const float4 pn = __ldg(&props[jidx]);
    const float n1 = s.pr.w, n2 = pn.w;
    if (fabsf(n1 - n2) > P.step_eps) {
        float r = fresnel_unpol(n1, n2, ua, P.eq_eps);
        if ((!metal || r > 0.0f) && s.rng.uniform(P.keys) < r) {
            ++tl.reflections;
            const float off = fwd ? 0.0f : 1.0f;
            if (ax0) { s.ux = -s.ux; s.iux = -s.iux; s.ox = off; }
            else if (ax1) { s.uy = -s.uy; s.iuy = -s.iuy; s.oy = off; }
            else { s.uz = -s.uz; s.iuz = -s.iuz; s.oz = off; }
            return true;
        }
        refract_axis(s.ux, s.uy, s.uz, ax0 ? 0 : (ax1 ? 1 : 2), n1 / n2);
        photon_aim(s);
    }
    s.gx = ax0 ? cell : s.gx;
    s.gy = ax1 ? cell : s.gy;
    s.gz = ax0 || ax1 ? s.gz : cell;
    s.idx = jidx;
    s.pr = pn;
    return true;
}

#ifndef BD_MC_MIN_BLOCKS
#define BD_MC_MIN_BLOCKS 8
#endif
template <int DEPTH>
__global__ void __launch_bounds__(128, BD_MC_MIN_BLOCKS) k_mc_trace(McDev P, const float4* __restrict__ props,
                                                     const uint8_t* __restrict__ flags,
                                                     unsigned long long* __restrict__ A64, double* __restrict__ latz,
                                                     unsigned long long* __restrict__ queue,
                                                     double* __restrict__ partials,
                                                     const long long* __restrict__ offset_dev, int lanes) {
    // a photon-stream offset kept in device memory lets a captured graph advance it per replay
    if (offset_dev != nullptr) P.offset += *offset_dev;
    double* sl = partials + (size_t)blockIdx.x * BD_LEDGER_LEN;  // zeroed before the launch
    ThreadLedger tl;
    tl.absorbed = tl.absorbed_void = 0.0;
    tl.collisions = tl.crossings = tl.reflections = 0u;
    const bool metal = (P.options & BD_MC_METAL_SEMANTICS) != 0;

    const unsigned long long N = (unsigned long long)P.n_photons;
    // A lane that has reached an interaction waits until half the live lanes of its warp have (or none
    // can move): interactions cost several times a crossing, are seven times rarer, and would otherwise
    // run for the few lanes that reach one in the same iteration. 1.5 M photons on the 200x200x128
    // stack: 8.6 ms, 12.6 ms without waiting; a third of the lanes 8.7 ms, a quarter 9.0 ms.
    PhotonState s;
    bool live = false, more = (int)(threadIdx.x & 31u) < lanes, hit = false;
    for (;;) {
        if (!live && more) {
            const unsigned long long p = atomicAdd(queue, 1ull);
            if (p >= N) more = false;
            else live = photon_launch<DEPTH>(P, (long long)p, props, latz, sl, s);
        }
        if (live && !hit) {
            if (s.ev >= (unsigned)P.max_events) {   // at most kMcMaxEvents
                // event cap reached: the remaining weight is accounted, not lost
                atomicAdd(&sl[BD_LEDGER_TRUNCATED], (double)s.w);
                live = false;
            } else {
                ++s.ev;
                live = photon_move<DEPTH>(P, props, latz, sl, tl, s, metal, hit);
            }
        }
        const unsigned wait = __ballot_sync(0xffffffffu, live && hit);
        const unsigned go = __ballot_sync(0xffffffffu, live ? !hit : more);
        if (go == 0u ? wait != 0u : 2 * __popc(wait) >= __popc(wait | go)) {
            if (live && hit) {
                live = photon_collide<DEPTH>(P, flags, A64, latz, sl, tl, s);
                hit = false;
            }
        } else if (go == 0u) {
            break;
        }
    }
    // warp reduction of the per-thread channels, one FP64 atomic per warp and channel
    double v0 = tl.absorbed, v1 = tl.absorbed_void;
    unsigned c0 = tl.collisions, c1 = tl.crossings, c2 = tl.reflections;
    __syncwarp();  // every lane reaches here (no early return): reconverge for the shuffles
    const unsigned mask = 0xffffffffu;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v0 += __shfl_xor_sync(mask, v0, o);
        v1 += __shfl_xor_sync(mask, v1, o);
        c0 += __shfl_xor_sync(mask, c0, o);
        c1 += __shfl_xor_sync(mask, c1, o);
        c2 += __shfl_xor_sync(mask, c2, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sl[BD_LEDGER_ABSORBED], v0);
        if (v1 != 0.0) atomicAdd(&sl[BD_LEDGER_ABSORBED_VOID], v1);
        atomicAdd(&sl[BD_LEDGER_COLLISIONS], (double)c0);
        atomicAdd(&sl[BD_LEDGER_CROSSINGS], (double)c1);
        atomicAdd(&sl[BD_LEDGER_REFLECTIONS], (double)c2);
    }
}

// Fixed-order reduction of the per-block partials (deterministic for a given grid): a warp per channel,
// each lane a strided share of the blocks, then a tree over the lanes. One thread per channel walked
// the ~1200 rows one L2 round trip after another: 66 us of every trace.
__global__ void __launch_bounds__(32 * BD_LEDGER_LEN) k_ledger_reduce(const double* __restrict__ partials, int nblocks,
                                                                      double launched, double* __restrict__ ledger) {
    const int ch = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double s = 0.0;
#pragma unroll 4
    for (int b = lane; b < nblocks; b += 32) s += partials[(size_t)b * BD_LEDGER_LEN + ch];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) ledger[ch] = ch == BD_LEDGER_LAUNCHED ? launched : s;
}

__global__ void k_pack_props(const float* __restrict__ mu_a, const float* __restrict__ mu_s,
                             const float* __restrict__ g, const float* __restrict__ n,
                             const float* __restrict__ mu_ext, const uint8_t* __restrict__ flags,
                             float ra, float rs, float g_plume, long long nv, float4* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv;
         i += (long long)gridDim.x * blockDim.x) {
        float a = mu_a[i], s = mu_s[i], gg = g[i], nn = n[i];
        if (mu_ext != nullptr) {
            float e = mu_ext[i];
            a = a + e * ra;
            s = s + e * rs;
            if (e > 0.001f && (flags[i] & BD_FLAG_ABLATED)) gg = g_plume;
        }
        float mt = a + s;
        float ratio = mt > 0.0f ? a / mt : 0.0f;
        out[i] = make_float4(mt, ratio, gg, nn);
    }
}

// A[i] += fixed-point tally[i] in weight units; the tally is left zeroed for the next launch.
__global__ void k_tally_finalize(unsigned long long* __restrict__ t64, float* __restrict__ A, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long v = t64[i];
        if (v != 0ull) {
            A[i] += (float)((double)v * (1.0 / (double)kTallyScale));
            t64[i] = 0ull;
        }
    }
}

__global__ void k_fold(float* __restrict__ src, double* __restrict__ dst, long long n) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        float v = src[i];
        if (v != 0.0f) {
            dst[i] += (double)v;
            src[i] = 0.0f;
        }
    }
}

}  // namespace bd

// ------------------------------------------------------------------------------------
struct BdMcContext {
    unsigned long long* queue = nullptr;
    double* partials = nullptr;
    unsigned long long* tally64 = nullptr;   // fixed-point absorbed tally, grown to the largest grid
    long long tally_cap = 0;
    int partial_blocks = 0;
    int device = -1;
    int sm_count = 148;
};

using namespace bd;

extern "C" int bd_mc_create(BdMcContext** out) {
    BD_REQUIRE(out != nullptr, "bd_mc_create: out is NULL");
    BdMcContext* c = new BdMcContext();
    BD_CUDA(cudaGetDevice(&c->device));
    cudaDeviceGetAttribute(&c->sm_count, cudaDevAttrMultiProcessorCount, c->device);
    // 16 resident 128-thread blocks per SM is the occupancy ceiling of k_mc_trace
    c->partial_blocks = c->sm_count * 16;
    cudaError_t e = cudaMalloc(&c->queue, sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMalloc(&c->partials, sizeof(double) * BD_LEDGER_LEN * c->partial_blocks);
    if (e != cudaSuccess) {
        cudaFree(c->queue);
        delete c;
        return cuda_status(e, "bd_mc_create: cudaMalloc");
    }
    *out = c;
    return BD_OK;
}

extern "C" int bd_mc_destroy(BdMcContext* c) {
    if (!c) return BD_OK;
    cudaFree(c->queue);
    cudaFree(c->partials);
    cudaFree(c->tally64);
    delete c;
    return BD_OK;
}

namespace bd {
int mc_validate(const BdMcParams* p) {
    BD_REQUIRE(p != nullptr, "bd_mc_trace: params is NULL");
    BD_REQUIRE(p->nx > 0 && p->ny > 0 && p->nz > 0, "bd_mc_trace: grid dims must be positive");
    BD_REQUIRE(p->dx > 0 && p->dy > 0 && p->dz > 0, "bd_mc_trace: voxel size must be positive");
    BD_REQUIRE(p->launch_axis == 0 || p->launch_axis == 1, "bd_mc_trace: launch_axis must be 0 (z) or 1 (x)");
    BD_REQUIRE(p->beam_profile >= 0 && p->beam_profile <= 3, "bd_mc_trace: unknown beam profile %d", p->beam_profile);
    BD_REQUIRE(p->n_photons >= 0, "bd_mc_trace: n_photons must be >= 0");
    BD_REQUIRE(p->max_events > 0, "bd_mc_trace: max_events must be > 0");
    BD_REQUIRE(p->cos_th_safe > 0.0f, "bd_mc_trace: cos_th_safe must be > 0");
    return BD_OK;
}

McDev mc_dev_params(const BdMcParams* p) {
    McDev d;
    d.nx = p->nx; d.ny = p->ny; d.nz = p->nz; d.launch_axis = p->launch_axis;
    d.dx = p->dx; d.dy = p->dy; d.dz = p->dz; d.lx = p->lx; d.ly = p->ly; d.lz = p->lz;
    d.ux0 = p->init_ux; d.uy0 = p->init_uy; d.uz0 = p->init_uz;
    d.cos_ph = p->cos_ph; d.sin_ph = p->sin_ph; d.cos_th_safe = p->cos_th_safe;
    d.xc = p->x_center; d.yc = p->y_center; d.zc = p->z_center;
    d.sigma = p->sigma_axis; d.radius = p->beam_radius; d.profile = p->beam_profile;
    d.n_amb = p->n_ambient; d.rmax2 = p->r_max_sq; d.options = p->options;
    d.n_photons = p->n_photons; d.offset = p->photon_offset;
    d.max_events = p->max_events;
    d.seed = p->seed;
    d.fnx = (float)p->nx; d.fny = (float)p->ny; d.fnz = (float)p->nz;
    Philox::keys((uint32_t)p->seed, (uint32_t)(p->seed >> 32), d.keys);
    const bool metal = (p->options & BD_MC_METAL_SEMANTICS) != 0;
    d.eq_eps = metal ? 1e-6f : 1e-9f;
    d.step_eps = metal ? 1e-4f : 1e-9f;
    d.entry_eps = metal ? 1e-6f : 1e-9f;
    return d;
}

// Launch with caller-provided scratch (queue counter + per-block partials).
int mc_launch(const BdMcParams* p, const float* props, const uint8_t* flags, float* A, float* L,
              double* latz, double* ledger, unsigned long long* queue, double* partials, int max_blocks,
              int sm_count, cudaStream_t st, const long long* offset_dev, unsigned long long* tally64) {
    McDev d = mc_dev_params(p);
    const float4* pr = reinterpret_cast<const float4*>(props);
    int blocks = 1;
    // k_mc_trace tests the bounds on voxel indices in FP32, exact up to 2^24, and counts events in 32 bits;
    // mc_fluence.cu's indices are integers and its events 64 bits
    const bool wide = std::max(p->nx, std::max(p->ny, p->nz)) > kMcMaxAxis || p->max_events > kMcMaxEvents;
    if (((d.options & BD_MC_TALLY_FLUENCE) != 0 && L != nullptr) || tally64 == nullptr || wide) {
        // FP32 sums in memory depend on the order of the deposits: these launches keep the event order of
        // mc_fluence.cu (its comment has both sides)
        if (int rc = mc_fluence_launch(d, pr, flags, A, tally64, L, latz, queue, partials, max_blocks, sm_count, st,
                                       offset_dev, &blocks))
            return rc;
    } else {
        // resident 128-thread CTAs per SM of each kernel variant: computed once, shared by host threads
        static std::atomic<int> per_sm[2] = {{0}, {0}};
        const int ax = p->launch_axis == 0 ? 0 : 1;
        int occ = per_sm[ax].load(std::memory_order_relaxed);
        if (occ == 0) {
            int nb = 0;
            if (ax == 0) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_mc_trace<2>, 128, 0);
            else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_mc_trace<0>, 128, 0);
            occ = std::max(1, std::min(nb, 16));
            cudaGetLastError();
            per_sm[ax].store(occ, std::memory_order_relaxed);
        }
        const int want = tune_value(BD_TUNE_MC_BLOCKS_PER_SM);
        const int use_sm = want > 0 ? std::min(want, occ) : occ;
        // A warp runs the union of its lanes' branches, so few photons finish sooner spread over half of the resident
        // warps, some lanes of each, than packed into full ones; over all of them, photons whose histories are
        // alike cost more issue slots than the union saves. 20 k / 40 k / 80 k photons over all, and over half:
        // crater stack of 200x200x128 0.94 / 1.08 / 1.16 and 0.94 / 1.10 / 1.18 ms, one dense medium 0.63 / 0.68 /
        // 0.74 and 0.55 / 0.56 / 0.59, a clear one 0.20 / 0.20 / 0.20 and 0.16 / 0.17 / 0.17 (full warps of the kernel
        // before: 1.35 / 1.42 / 1.46, 0.67 / 0.71 / 0.84, 0.17 / 0.18 / 0.20).
        const long long most = std::max(1LL, std::min<long long>((long long)sm_count * use_sm, max_blocks));
        const int lanes = (int)std::min<long long>(32, std::max<long long>(1, (p->n_photons + 2 * most - 1) / (2 * most)));
        blocks = (int)std::max(1LL, std::min(most, (p->n_photons + 4LL * lanes - 1) / (4LL * lanes)));
        BD_CUDA(cudaMemsetAsync(queue, 0, sizeof(unsigned long long), st));
        BD_CUDA(cudaMemsetAsync(partials, 0, sizeof(double) * BD_LEDGER_LEN * blocks, st));
        if (p->launch_axis == 0)
            k_mc_trace<2><<<blocks, 128, 0, st>>>(d, pr, flags, tally64, latz, queue, partials, offset_dev, lanes);
        else
            k_mc_trace<0><<<blocks, 128, 0, st>>>(d, pr, flags, tally64, latz, queue, partials, offset_dev, lanes);
        BD_CHECK_LAUNCH("k_mc_trace");
    }
    if (tally64) {
        const long long nv = (long long)p->nx * p->ny * p->nz;
        k_tally_finalize<<<grid_for(nv, 256), 256, 0, st>>>(tally64, A, nv);
        BD_CHECK_LAUNCH("k_tally_finalize");
    }
    k_ledger_reduce<<<1, 32 * BD_LEDGER_LEN, 0, st>>>(partials, blocks, (double)p->n_photons, ledger);
    BD_CHECK_LAUNCH("k_ledger_reduce");
    return BD_OK;
}
}  // namespace bd

extern "C" int bd_mc_trace(BdMcContext* c, const BdMcParams* p, const float* props, const uint8_t* flags,
                           float* A, float* L, double* lat_depth, double* ledger, void* stream) {
    BD_REQUIRE(c != nullptr, "bd_mc_trace: context is NULL");
    int rc = mc_validate(p);
    if (rc) return rc;
    BD_REQUIRE(props != nullptr && A != nullptr && ledger != nullptr, "bd_mc_trace: props, A and ledger are required");
    BD_REQUIRE(!(p->options & BD_MC_TALLY_FLUENCE) || L != nullptr, "bd_mc_trace: BD_MC_TALLY_FLUENCE needs L");
    BD_REQUIRE(p->n_photons <= kTallyMaxPhotons,
               "bd_mc_trace: at most %lld photons per launch (fixed-point tally range); split into batches",
               (long long)kTallyMaxPhotons);
    const long long nv = (long long)p->nx * p->ny * p->nz;
    if (nv > c->tally_cap) {
        cudaFree(c->tally64);
        c->tally64 = nullptr;
        c->tally_cap = 0;
        BD_CUDA(cudaMalloc(&c->tally64, sizeof(unsigned long long) * nv));
        BD_CUDA(cudaMemset(c->tally64, 0, sizeof(unsigned long long) * nv));
        c->tally_cap = nv;
    }
    return mc_launch(p, props, flags, A, L, lat_depth, ledger, c->queue, c->partials, c->partial_blocks,
                     c->sm_count, as_stream(stream), nullptr, c->tally64);
}

extern "C" int bd_mc_pack_props(const float* mu_a, const float* mu_s, const float* g, const float* n,
                                const float* mu_ext, const uint8_t* flags, float ra, float rs, float g_plume,
                                int64_t nv, float* out, void* stream) {
    BD_REQUIRE(mu_a && mu_s && g && n && out, "bd_mc_pack_props: NULL property pointer");
    BD_REQUIRE(nv >= 0, "bd_mc_pack_props: negative size");
    BD_REQUIRE(mu_ext == nullptr || flags != nullptr, "bd_mc_pack_props: plume extinction needs flags");
    if (nv == 0) return BD_OK;
    k_pack_props<<<grid_for(nv, 256), 256, 0, as_stream(stream)>>>(mu_a, mu_s, g, n, mu_ext, flags, ra, rs,
                                                                    g_plume, nv, reinterpret_cast<float4*>(out));
    BD_CHECK_LAUNCH("k_pack_props");
    return BD_OK;
}

extern "C" int bd_fold_f32_to_f64(float* src, double* dst, int64_t n, void* stream) {
    BD_REQUIRE(src && dst, "bd_fold_f32_to_f64: NULL pointer");
    if (n <= 0) return BD_OK;
    k_fold<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(src, dst, n);
    BD_CHECK_LAUNCH("k_fold");
    return BD_OK;
}

// ------------------------------------------------------------------------------------
// Allocation-free variant of bd_mc_trace.
//
// Some callers cannot call cudaMalloc once they are running: a control loop that must keep a
// fixed latency per laser pulse (the allocator may synchronise the device or block on the
// driver), or a host framework that owns all device memory through its own pool and does not
// allow side allocations. bd_mc_trace_noalloc needs no allocation at all: its scratch (the
// photon-queue counter and one FP64 ledger row per block) is a file-scope device array of fixed
// size, which every GPU that loads this library holds until the process exits.
namespace bd {
constexpr int MC_NOALLOC_MAX_BLOCKS = 2048;
constexpr size_t MC_NOALLOC_QUEUE_BYTES = 256;
static __device__ __align__(256) unsigned char g_mc_noalloc_scratch[MC_NOALLOC_QUEUE_BYTES +
                                                                    sizeof(double) * BD_LEDGER_LEN *
                                                                        MC_NOALLOC_MAX_BLOCKS];
constexpr int MC_NOALLOC_MAX_DEVICES = 64;
static void* g_mc_noalloc_ptr[MC_NOALLOC_MAX_DEVICES] = {nullptr};
static int g_mc_noalloc_sms[MC_NOALLOC_MAX_DEVICES] = {0};
static std::mutex g_mc_noalloc_mu;
}  // namespace bd

extern "C" int bd_mc_trace_noalloc(const BdMcParams* p, const float* props, const uint8_t* flags, float* A,
                                   float* L, double* lat_depth, double* ledger, void* stream) {
    int rc = mc_validate(p);
    if (rc) return rc;
    BD_REQUIRE(props != nullptr && A != nullptr && ledger != nullptr,
               "bd_mc_trace_noalloc: props, A and ledger are required");
    BD_REQUIRE(!(p->options & BD_MC_TALLY_FLUENCE) || L != nullptr, "bd_mc_trace_noalloc: BD_MC_TALLY_FLUENCE needs L");
    int dev = 0;
    BD_CUDA(cudaGetDevice(&dev));
    BD_REQUIRE(dev >= 0 && dev < MC_NOALLOC_MAX_DEVICES, "bd_mc_trace_noalloc: device ordinal %d >= %d", dev,
               MC_NOALLOC_MAX_DEVICES);
    void* base = nullptr;
    int sms = 0;
    {
        // set-up once per device, with that device current: the array's name is only a host-side
        // stand-in, the kernel must be given the device address of this device's copy. The address
        // is cached for the life of the device's primary context: do not use this entry point across
        // a cudaDeviceReset of that device.
        std::lock_guard<std::mutex> lock(g_mc_noalloc_mu);
        if (g_mc_noalloc_ptr[dev] == nullptr) {
            void* ptr = nullptr;
            BD_CUDA(cudaGetSymbolAddress(&ptr, g_mc_noalloc_scratch));
            int n = 0;
            BD_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
            g_mc_noalloc_ptr[dev] = ptr;
            g_mc_noalloc_sms[dev] = n;
        }
        base = g_mc_noalloc_ptr[dev];
        sms = g_mc_noalloc_sms[dev];
    }
    // the kernel is persistent (a photon queue), so any photon count runs on at most
    // MC_NOALLOC_MAX_BLOCKS blocks: mc_launch caps the grid at the static ledger rows
    unsigned long long* queue = static_cast<unsigned long long*>(base);
    double* partials = reinterpret_cast<double*>(static_cast<unsigned char*>(base) + MC_NOALLOC_QUEUE_BYTES);
    // mc_launch zeroes the queue counter and the ledger rows it uses before the kernel runs
    return mc_launch(p, props, flags, A, L, lat_depth, ledger, queue, partials, MC_NOALLOC_MAX_BLOCKS, sms,
                     as_stream(stream), nullptr, nullptr);
}
