// Photon tracer of the launches whose results are FP32 sums in memory: the track length (fluence), and the
// absorbed map where no exact tally is kept; and of grids with an axis of more than 2^24 voxels or event caps of
// more than 32 bits, which mc.cu's indices and counter cannot hold.
//
// An FP32 sum of thousands of deposits depends on their order by up to 3e-6 of the map (2-norm, 75 k photons on
// a 26x40x50 grid): the beam's voxels first take the photons' equal first chords. Two traces with this order
// of events agree to 0.1-0.7e-6; with the crossings apart from the interactions, as mc.cu traces, they come
// nearer to the exact sum (2.9e-6 against 3.5e-6) but 0.3-1.7e-6 from what this order gives, up to 5 times what
// two traces differ by. So these launches keep one event, crossing or interaction, a lane and iteration; the
// exact fixed-point tally does not depend on the order, and mc.cu serves it. 100 k photons on a 40x40x50 grid
// through the host call: 2.84 ms here, 2.74 ms with mc.cu's kernel. Same histories bit for bit.
#include <algorithm>
#include <atomic>

#include "mc_dev.cuh"

namespace bd {

namespace {

// Per-photon stream (counter layout of PhotonRng; the same draws), a block of four generated when needed.
struct FluenceRng {
    uint32_t k0, k1, p_lo, p_hi, blk;
    uint32_t r0, r1, r2, r3;
    int left;
    __device__ inline void init(uint64_t seed, uint64_t photon) {
        k0 = (uint32_t)seed; k1 = (uint32_t)(seed >> 32);
        p_lo = (uint32_t)photon; p_hi = (uint32_t)(photon >> 32);
        blk = 0; left = 0;
    }
    __device__ inline uint32_t next_u32() {
        if (left == 0) {
            uint4 v = Philox::gen(make_uint4(p_lo, p_hi, blk++, 0x42444d43u), k0, k1);
            r0 = v.x; r1 = v.y; r2 = v.z; r3 = v.w; left = 4;
        }
        uint32_t out = r0;
        r0 = r1; r1 = r2; r2 = r3; --left;
        return out;
    }
    // uniform in [0, 1): 24 significant bits
    __device__ inline float uniform(const uint32_t* = nullptr) { return (float)(next_u32() >> 8) * (1.0f / 16777216.0f); }
    // uniform in (0, 1): never 0, for logarithms
    __device__ inline float uniform_pos(const uint32_t* = nullptr) {
        return ((float)(next_u32() >> 8) + 0.5f) * (1.0f / 16777216.0f);
    }
};

// Per-thread accumulators of the per-event ledger channels; the rare channels go to the block's row.
struct FluenceLedger {
    double absorbed;
    unsigned collisions, crossings, reflections;
};

// The photon a lane is tracing; a lane whose photon has ended takes the next from the queue.
struct FluencePhoton {
    FluenceRng rng;
    float x, y, z, ux, uy, uz, iux, iuy, iuz, tau, w;
    float4 pr;
    int ix, iy, iz, idx;
    long long ev;
};

// Launch: transverse offsets, footprint test, entrance Fresnel split and refraction, first
// optical depth. Returns false when the photon never enters the grid (booked here).
template <int DEPTH>  // 2: launch along +z at z=0 ; 0: launch along +x at x=0
__device__ __forceinline__ bool fluence_launch(const McDev& P, long long pid, const float4* __restrict__ props,
                                              double* __restrict__ latz, double* sl, FluencePhoton& s) {
    s.rng.init(P.seed, (unsigned long long)(P.offset + pid));
    float u1, u2;
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
        s.ix = min((int)(s.x / P.dx), P.nx - 1);
        s.iy = min((int)(s.y / P.dy), P.ny - 1);
        s.iz = 0;
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
        s.ix = 0;
        s.iy = min((int)(s.y / P.dy), P.ny - 1);
        s.iz = min((int)(s.z / P.dz), P.nz - 1);
    }
    s.ux = P.ux0; s.uy = P.uy0; s.uz = P.uz0;
    s.idx = s.ix * (P.ny * P.nz) + s.iy * P.nz + s.iz;

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
    s.iux = fabsf(s.ux) > 1e-15f ? 1.0f / s.ux : 0.0f;
    s.iuy = fabsf(s.uy) > 1e-15f ? 1.0f / s.uy : 0.0f;
    s.iuz = fabsf(s.uz) > 1e-15f ? 1.0f / s.uz : 0.0f;
    s.tau = -__logf(fmaxf(s.rng.uniform(), 1e-12f));
    s.ev = 0;
    return true;
}

// One event of the hop-drop-spin loop (voxel_mc_3d.py:194-337): a collision inside the voxel or a
// crossing of its exit face. Returns false when the photon has ended (its weight booked).
template <int DEPTH>
__device__ __forceinline__ bool fluence_event(const McDev& P, const float4* __restrict__ props,
                                             const uint8_t* __restrict__ flags, float* __restrict__ A,
                                             unsigned long long* __restrict__ A64, float* __restrict__ L,
                                             double* __restrict__ latz, double* sl, FluenceLedger& tl,
                                             FluencePhoton& s, bool metal, bool tally_l) {
    const float dx = P.dx, dy = P.dy, dz = P.dz;
    // exact ray/box distance to the exit face (voxel_mc_3d.py:72-98)
    float sx = s.ux > 1e-15f ? ((float)(s.ix + 1) * dx - s.x) * s.iux
                             : (s.ux < -1e-15f ? ((float)s.ix * dx - s.x) * s.iux : 1e30f);
    float sy = s.uy > 1e-15f ? ((float)(s.iy + 1) * dy - s.y) * s.iuy
                             : (s.uy < -1e-15f ? ((float)s.iy * dy - s.y) * s.iuy : 1e30f);
    float sz = s.uz > 1e-15f ? ((float)(s.iz + 1) * dz - s.z) * s.iuz
                             : (s.uz < -1e-15f ? ((float)s.iz * dz - s.z) * s.iuz : 1e30f);
    int axis;
    float s_exit;
    if (sx <= sy && sx <= sz) { axis = 0; s_exit = fmaxf(sx, 0.0f); }
    else if (sy <= sz)        { axis = 1; s_exit = fmaxf(sy, 0.0f); }
    else                      { axis = 2; s_exit = fmaxf(sz, 0.0f); }
    const float mu_t = s.pr.x;

    if (mu_t > 1e-12f && mu_t * s_exit >= s.tau) {
        // ---- interaction inside the voxel ----
        ++tl.collisions;
        float st = s.tau / mu_t;
        if (tally_l) atomicAdd(&L[s.idx], s.w * st);
        s.x += st * s.ux; s.y += st * s.uy; s.z += st * s.uz;
        if (P.rmax2 > 0.0f) {
            float a = (DEPTH == 2) ? s.x - P.xc : s.y - P.yc;
            float b = (DEPTH == 2) ? s.y - P.yc : s.z - P.zc;
            if (a * a + b * b >= P.rmax2) {
                atomicAdd(&sl[BD_LEDGER_LATERAL], (double)s.w);
                if (latz) atomicAdd(&latz[DEPTH == 2 ? s.iz : s.ix], (double)s.w);
                return false;
            }
        }
        {
            const float dw = s.w * s.pr.y;
            const float w_new = s.w - dw;
            if (A64) atomicAdd(&A64[s.idx], __float2ull_rn(dw * kTallyScale));
            else atomicAdd(&A[s.idx], dw);
            const double lost = (double)s.w - (double)w_new;  // exact: both are FP32 values
            if (flags != nullptr && (__ldg(&flags[s.idx]) & BD_FLAG_ABLATED)) atomicAdd(&sl[BD_LEDGER_ABSORBED_VOID], lost);
            else tl.absorbed += lost;
            s.w = w_new;
        }
        if (s.w < 1e-4f) {
            if (s.rng.uniform() < 0.1f) {
                const float w10 = s.w * 10.0f;
                atomicAdd(&sl[BD_LEDGER_ROULETTE_GAIN], (double)w10 - (double)s.w);
                s.w = w10;
            } else {
                atomicAdd(&sl[BD_LEDGER_ROULETTE_LOSS], (double)s.w);
                return false;
            }
        }
        const float xi = s.rng.uniform(), xphi = s.rng.uniform();
        scatter_hg(s.ux, s.uy, s.uz, s.pr.z, xi, xphi);
        s.iux = fabsf(s.ux) > 1e-15f ? 1.0f / s.ux : 0.0f;
        s.iuy = fabsf(s.uy) > 1e-15f ? 1.0f / s.uy : 0.0f;
        s.iuz = fabsf(s.uz) > 1e-15f ? 1.0f / s.uz : 0.0f;
        s.tau = -__logf(fmaxf(s.rng.uniform(), 1e-12f));
        return true;
    }

    // ---- traverse the chord and land exactly on the exit face ----
    ++tl.crossings;
    s.tau -= mu_t * s_exit;
    if (tally_l) atomicAdd(&L[s.idx], s.w * s_exit);
    s.x += s_exit * s.ux; s.y += s_exit * s.uy; s.z += s_exit * s.uz;
    int jx = s.ix, jy = s.iy, jz = s.iz;
    if (axis == 0)      { int sd = s.ux > 0.0f ? 1 : -1; jx += sd; s.x = sd > 0 ? (float)(s.ix + 1) * dx : (float)s.ix * dx; }
    else if (axis == 1) { int sd = s.uy > 0.0f ? 1 : -1; jy += sd; s.y = sd > 0 ? (float)(s.iy + 1) * dy : (float)s.iy * dy; }
    else                { int sd = s.uz > 0.0f ? 1 : -1; jz += sd; s.z = sd > 0 ? (float)(s.iz + 1) * dz : (float)s.iz * dz; }

    if (axis == DEPTH) {
        const int jd = (DEPTH == 2) ? jz : jx;
        const int nd = (DEPTH == 2) ? P.nz : P.nx;
        if (jd < 0) {
            // leaving through the entrance face: Fresnel / TIR against ambient
            float cos_out = (DEPTH == 2) ? s.uz : s.ux;
            float r = fresnel_unpol(s.pr.w, P.n_amb, cos_out, P.eq_eps);
            if (r > 0.0f && s.rng.uniform() < r) {
                ++tl.reflections;
                if (DEPTH == 2) { s.uz = -s.uz; s.iuz = -s.iuz; } else { s.ux = -s.ux; s.iux = -s.iux; }
                return true;
            }
            atomicAdd(&sl[BD_LEDGER_DIFFUSE], (double)s.w);
            return false;
        }
        if (jd >= nd) {
            atomicAdd(&sl[BD_LEDGER_TRANSMITTED], (double)s.w);
            return false;
        }
    } else if (jx < 0 || jx >= P.nx || jy < 0 || jy >= P.ny || jz < 0 || jz >= P.nz) {
        atomicAdd(&sl[BD_LEDGER_LATERAL], (double)s.w);
        if (latz) atomicAdd(&latz[DEPTH == 2 ? s.iz : s.ix], (double)s.w);
        return false;
    }
    if (!metal && P.rmax2 > 0.0f) {
        float a = (DEPTH == 2) ? s.x - P.xc : s.y - P.yc;
        float b = (DEPTH == 2) ? s.y - P.yc : s.z - P.zc;
        if (a * a + b * b >= P.rmax2) {
            atomicAdd(&sl[BD_LEDGER_LATERAL], (double)s.w);
            if (latz) atomicAdd(&latz[DEPTH == 2 ? s.iz : s.ix], (double)s.w);
            return false;
        }
    }
    const int jidx = jx * (P.ny * P.nz) + jy * P.nz + jz;
    float4 pn = __ldg(&props[jidx]);
    float n1 = s.pr.w, n2 = pn.w;
    if (fabsf(n1 - n2) > P.step_eps) {
        float cos_face = axis == 0 ? s.ux : (axis == 1 ? s.uy : s.uz);
        float r = fresnel_unpol(n1, n2, cos_face, P.eq_eps);
        if ((!metal || r > 0.0f) && s.rng.uniform() < r) {
            ++tl.reflections;
            if (axis == 0) { s.ux = -s.ux; s.iux = -s.iux; }
            else if (axis == 1) { s.uy = -s.uy; s.iuy = -s.iuy; }
            else { s.uz = -s.uz; s.iuz = -s.iuz; }
            return true;
        }
        refract_axis(s.ux, s.uy, s.uz, axis, n1 / n2);
        s.iux = fabsf(s.ux) > 1e-15f ? 1.0f / s.ux : 0.0f;
        s.iuy = fabsf(s.uy) > 1e-15f ? 1.0f / s.uy : 0.0f;
        s.iuz = fabsf(s.uz) > 1e-15f ? 1.0f / s.uz : 0.0f;
    }
    s.ix = jx; s.iy = jy; s.iz = jz;
    s.idx = jidx;
    s.pr = pn;
    return true;
}

template <int DEPTH>
__global__ void __launch_bounds__(128, 8) k_mc_fluence(McDev P, const float4* __restrict__ props,
                                                     const uint8_t* __restrict__ flags, float* __restrict__ A,
                                                     unsigned long long* __restrict__ A64,
                                                     float* __restrict__ L, double* __restrict__ latz,
                                                     unsigned long long* __restrict__ queue,
                                                     double* __restrict__ partials,
                                                     const long long* __restrict__ offset_dev) {
    // a photon-stream offset kept in device memory lets a captured graph advance it per replay
    if (offset_dev != nullptr) P.offset += *offset_dev;
    double* sl = partials + (size_t)blockIdx.x * BD_LEDGER_LEN;  // zeroed before the launch
    FluenceLedger tl;
    tl.absorbed = 0.0;
    tl.collisions = tl.crossings = tl.reflections = 0u;
    const bool metal = (P.options & BD_MC_METAL_SEMANTICS) != 0;
    const bool tally_l = (P.options & BD_MC_TALLY_FLUENCE) != 0 && L != nullptr;

    const unsigned long long N = (unsigned long long)P.n_photons;
    FluencePhoton s;
    bool live = false;
    for (;;) {
        if (!live) {
            const unsigned long long p = atomicAdd(queue, 1ull);
            if (p >= N) break;
            live = fluence_launch<DEPTH>(P, (long long)p, props, latz, sl, s);
            if (!live) continue;
        }
        if (s.ev >= P.max_events) {
            // event cap reached: the remaining weight is accounted, not lost
            atomicAdd(&sl[BD_LEDGER_TRUNCATED], (double)s.w);
            live = false;
            continue;
        }
        ++s.ev;
        live = fluence_event<DEPTH>(P, props, flags, A, A64, L, latz, sl, tl, s, metal, tally_l);
    }
    // warp reduction of the per-thread channels, one FP64 atomic per warp and channel
    double v0 = tl.absorbed;
    unsigned c0 = tl.collisions, c1 = tl.crossings, c2 = tl.reflections;
    __syncwarp();  // every lane reaches here (no early return): reconverge for the shuffles
    const unsigned mask = 0xffffffffu;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v0 += __shfl_xor_sync(mask, v0, o);
        c0 += __shfl_xor_sync(mask, c0, o);
        c1 += __shfl_xor_sync(mask, c1, o);
        c2 += __shfl_xor_sync(mask, c2, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&sl[BD_LEDGER_ABSORBED], v0);
        atomicAdd(&sl[BD_LEDGER_COLLISIONS], (double)c0);
        atomicAdd(&sl[BD_LEDGER_CROSSINGS], (double)c1);
        atomicAdd(&sl[BD_LEDGER_REFLECTIONS], (double)c2);
    }
}

}  // namespace

int mc_fluence_launch(const McDev& d, const float4* props, const uint8_t* flags, float* A, unsigned long long* tally64,
                      float* L, double* latz, unsigned long long* queue, double* partials, int max_blocks, int sm_count,
                      cudaStream_t st, const long long* offset_dev, int* blocks) {
    // resident 128-thread CTAs per SM of each kernel variant: computed once, shared by host threads
    static std::atomic<int> per_sm[2] = {{0}, {0}};
    const int ax = d.launch_axis == 0 ? 0 : 1;
    int occ = per_sm[ax].load(std::memory_order_relaxed);
    if (occ == 0) {
        int nb = 0;
        if (ax == 0) cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_mc_fluence<2>, 128, 0);
        else cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_mc_fluence<0>, 128, 0);
        occ = std::max(1, std::min(nb, 16));
        cudaGetLastError();
        per_sm[ax].store(occ, std::memory_order_relaxed);
    }
    const int want = tune_value(BD_TUNE_MC_BLOCKS_PER_SM);
    const int use_sm = want > 0 ? std::min(want, occ) : occ;
    const int n = (int)std::min<long long>((d.n_photons + 127) / 128, (long long)sm_count * use_sm);
    *blocks = std::max(1, std::min(n, max_blocks));
    BD_CUDA(cudaMemsetAsync(queue, 0, sizeof(unsigned long long), st));
    BD_CUDA(cudaMemsetAsync(partials, 0, sizeof(double) * BD_LEDGER_LEN * *blocks, st));
    if (ax == 0)
        k_mc_fluence<2><<<*blocks, 128, 0, st>>>(d, props, flags, A, tally64, L, latz, queue, partials, offset_dev);
    else
        k_mc_fluence<0><<<*blocks, 128, 0, st>>>(d, props, flags, A, tally64, L, latz, queue, partials, offset_dev);
    BD_CHECK_LAUNCH("k_mc_fluence");
    return BD_OK;
}

}  // namespace bd
