// Explicit 7-point bioheat stencil and the fused ablation substep (the plume is in plume.cu).
//
// Thermal update (voxel_thermal_3d.py:30-112, voxel_thermal_metal.py:56-134):
//   T' = T + dt (sum_faces k_face (T_nb - T) / d^2 + Q) / rho_cp,
//   k_face = 2 k_c k_n / (k_c + k_n + 1e-12); x/y faces insulated; z faces convective
//   (series half-cell + h_eff, or the Metal fused kernel's -h_eff (T - T_amb)/dz).
// Fused substep (metal_ablation_solver.py:71-191; CPU twin coupled_ablation.py:515-531):
//   + latent-heat plateau (voxel_thermal_3d.py:115-143), Arrhenius damage
//   (coupled_ablation.py:33-40) and first-order char kinetics (coupled_ablation.py:43-58),
//   all pointwise on the trial temperature, so one pass per substep does everything.
//
// Layout: z fastest. A thread owns 4 consecutive z voxels (a float4) of one row and marches along x
// (the slowest axis); the plane's groups are dealt to threads in memory order, so any nz fills the
// warps. A face's flux is computed once: +x kept for the next plane, z faces within the thread and
// by shuffle from the lane below, only the y faces twice (their rows come from L1). The source and the
// enthalpy are read only where a voxel uses them.
// What bounds it: latency and issue, with DRAM behind them (200x200x192: 172 MB of DRAM a substep, 3.1 TB/s;
// 527 warp instructions per 32 groups of 4, issue 57 %). 20 substeps, char on / char and damage on: 1.85 / 2.13 ms
// by 32 x 16 tiles staged through shared memory with every face computed twice, now 1.07 / 1.33 ms
// (5 CTAs of 128 threads per SM; 3 of 256 1.20 / 1.51, 6 of 128 1.17 / 1.46, 10 of 64 1.09 / 1.34).
// 150x150x138 (rows of no whole float4s) 0.86 -> 0.64 ms. Same bits.
#include "common.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace bd {


struct Geo {
    int nx, ny, nz, ni;
    float idx2, idy2, idz2, dz, h_eff, t_amb, dt;
};

// Harmonic face conductance 2 k_c k_n / (k_c + k_n + 1e-12) by the approximate reciprocal (<= 1 ulp): six
// precise IEEE divisions per voxel made the stencil instruction-bound, while the parity bar on T is
// 1e-4 relative. The operations are written out: the compiler contracts none of them, so the launch
// shape does not change a bit. The load width does, by a rounding of the -y face in half of the rows (see
// `fuse`): a grid of whole float4 rows rounds otherwise where its buffers are not aligned.
__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 rcp_approx2(float2 x) { return make_float2(rcp_approx(x.x), rcp_approx(x.y)); }
// conductance x temperature step across a face; k2: 2 k_c, nt: -T_c
__device__ __forceinline__ float face(float k2, float kc, float kn, float nt, float tn) {
    const float kf = __fmul_rn(__fmul_rn(k2, kn), rcp_approx(__fadd_rn(__fadd_rn(kc, kn), 1e-12f)));
    return __fmul_rn(kf, __fadd_rn(tn, nt));
}
__device__ __forceinline__ float2 face2(float2 k2, float2 kc, float2 kn, float2 nt, float2 tn) {
    const float2 den = __fadd2_rn(__fadd2_rn(kc, kn), make_float2(1e-12f, 1e-12f));
    return __fmul2_rn(__fmul2_rn(__fmul2_rn(k2, kn), rcp_approx2(den)), __fadd2_rn(tn, nt));
}
// A product that enters a sum rounded. Scalar: a packed multiply may be contracted with the packed add
// that takes it, a scalar one with explicit rounding is not.
__device__ __forceinline__ float2 scale2(float2 a, float s) { return make_float2(__fmul_rn(a.x, s), __fmul_rn(a.y, s)); }
__device__ __forceinline__ float2 lo2(const float4& v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4& v) { return make_float2(v.z, v.w); }

template <int BC>
__device__ __forceinline__ float zwall_flux(float Tc, float kc, const Geo& g) {
    if (BC == BD_BC_SERIES) {
        // voxel_thermal_3d.py:97,105
        return g.h_eff > 0.0f
                   ? (g.t_amb - Tc) / (g.dz * (0.5f * g.dz / fmaxf(kc, 1e-30f) + 1.0f / fmaxf(g.h_eff, 1e-30f)))
                   : 0.0f;
    } else {
        // metal_ablation_solver.py:141,150
        return -g.h_eff * (Tc - g.t_amb) / g.dz;
    }
}

struct AblConst {
    float t_abl, t_void, q_scale;
    float arr_A, arr_EaR, char_A, char_EaR;
    float t_cold;   // below this temperature a substep's char rate is nothing in FP32 (degC)
    int zero_src_in_ablated, is_active;
};

// MODE 0: thermal only. MODE 1: fused ablation substep. A thread owns 4 consecutive z voxels (one
// float4) of the plane's groups, taken in memory order, and marches xc planes along x.
constexpr int SUB_T = 128;
constexpr int SUB_WAVE = 12;   // CTAs per SM that the choice of planes per CTA aims at, at least

// 4 voxels from p on; `left` of them (>= 1) are in the row
template <bool VEC>
__device__ __forceinline__ float4 load4(const float* p, int left) {
    if (VEC) return *reinterpret_cast<const float4*>(p);
    return make_float4(p[0], left > 1 ? p[1] : 0.0f, left > 2 ? p[2] : 0.0f, left > 3 ? p[3] : 0.0f);
}
template <bool VEC>
__device__ __forceinline__ float4 load4_ro(const float* __restrict__ p, int left) {
    if (VEC) return __ldg(reinterpret_cast<const float4*>(p));
    return make_float4(__ldg(p), left > 1 ? __ldg(p + 1) : 0.0f, left > 2 ? __ldg(p + 2) : 0.0f,
                       left > 3 ? __ldg(p + 3) : 0.0f);
}
template <bool VEC>
__device__ __forceinline__ void store4(float* p, const float* v, int left) {
    if constexpr (VEC) {
        *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (i < left) p[i] = v[i];
    }
}
template <bool VEC>
__device__ __forceinline__ unsigned load_flags4(const uint8_t* __restrict__ p, int left) {
    if (VEC) return __ldg(reinterpret_cast<const unsigned*>(p));
    unsigned f = __ldg(p);
    if (left > 1) f |= (unsigned)__ldg(p + 1) << 8;
    if (left > 2) f |= (unsigned)__ldg(p + 2) << 16;
    if (left > 3) f |= (unsigned)__ldg(p + 3) << 24;
    return f;
}

template <int MODE, int BC, bool ARR, bool CHAR, bool VEC>
__global__ void __launch_bounds__(SUB_T, 5) k_substep(Geo g, AblConst c, const float* __restrict__ T,
                                                             float* __restrict__ Tn, const float* __restrict__ src,
                                                             const float* __restrict__ K, const float* __restrict__ R,
                                                             const uint8_t* __restrict__ F, float* __restrict__ H,
                                                             float* __restrict__ Om, float* __restrict__ Chi) {
    __shared__ float4 work[MODE == 1 && CHAR ? SUB_T / 32 : 1][16];   // per warp: 8 groups' T, 8 groups' chi
    const int G = (g.nz + 3) / 4;
    const int lane = threadIdx.x & 31;
    // threads past the plane's groups work on its last one and store nothing
    const int q0 = blockIdx.x * SUB_T + threadIdx.x, q = min(q0, g.ny * G - 1);
    const bool on = q0 == q;
    const int j = q / G, gi = q - j * G;
    const int z = 4 * gi, left = g.nz - z;
    const int plane = g.ny * g.nz;
    const int i0 = blockIdx.y * g.ni, i1 = min(i0 + g.ni, g.nx);
    // neighbours outside the grid are read from the voxel itself: no step, no flux
    const int to_s = j > 0 ? -g.nz : 0, to_n = j + 1 < g.ny ? g.nz : 0;
    const bool edge_b = gi > 0 && lane == 0, edge_a = gi + 1 < G && (lane == 31 || !on);
    const bool wall = gi == 0 || gi == G - 1;
    // The -y face's product enters the sum rounded, or within the multiply-add in rows 8..15 of every
    // 16 when rows are whole float4s: the rounding that recorded runs of such grids have.
    const bool fuse = VEC && (j & 8);
    const float2 ys = fuse ? make_float2(g.idy2, g.idy2) : make_float2(1.0f, 1.0f);
    int idx = i0 * plane + j * g.nz + z;
    float4 Tc = load4_ro<VEC>(T + idx, left), Kc = load4_ro<VEC>(K + idx, left);
    unsigned fl = 0u;
    if (MODE == 1) fl = load_flags4<VEC>(F + idx, left);
    float2 fwa, fwb;   // flux through the -x faces, of voxels 0, 1 and 2, 3
    {
        const int to_w = i0 > 0 ? -plane : 0;
        const float4 Tm = load4_ro<VEC>(T + idx + to_w, left), Km = load4_ro<VEC>(K + idx + to_w, left);
        const float2 m2 = make_float2(2.0f, 2.0f), m1 = make_float2(-1.0f, -1.0f);
        fwa = scale2(face2(__fmul2_rn(m2, lo2(Kc)), lo2(Kc), lo2(Km), __fmul2_rn(m1, lo2(Tc)), lo2(Tm)), g.idx2);
        fwb = scale2(face2(__fmul2_rn(m2, hi2(Kc)), hi2(Kc), hi2(Km), __fmul2_rn(m1, hi2(Tc)), hi2(Tm)), g.idx2);
    }
    for (int i = i0; i < i1; ++i, idx += plane) {
        // all of this plane's loads first; the flags were loaded a plane ahead, so that the source and
        // the enthalpy are read only where they are used
        const unsigned f4 = fl;
        const int to_e = i + 1 < g.nx ? plane : 0;
        const float4 Te = load4_ro<VEC>(T + idx + to_e, left), Ke = load4_ro<VEC>(K + idx + to_e, left);
        const float4 Ts = load4_ro<VEC>(T + idx + to_s, left), Ks = load4_ro<VEC>(K + idx + to_s, left);
        const float4 Tq = load4_ro<VEC>(T + idx + to_n, left), Kq = load4_ro<VEC>(K + idx + to_n, left);
        const float4 rho = load4_ro<VEC>(R + idx, left);
        float4 sr = make_float4(0.f, 0.f, 0.f, 0.f), h4 = sr;
        if (c.is_active && (MODE == 0 || !c.zero_src_in_ablated || (f4 & 0x01010101u) != 0x01010101u))
            sr = load4_ro<VEC>(src + idx, left);
        if (MODE == 1 && ((f4 | (f4 >> 1)) & 0x01010101u) != 0x01010101u) h4 = load4<VEC>(H + idx, left);
        if (MODE == 1 && i + 1 < i1) fl = load_flags4<VEC>(F + idx + plane, left);
        const unsigned dry4 = MODE == 1 && CHAR && on ? (f4 >> 1) & ~f4 & 0x01010101u : 0u;
        float4 x4 = make_float4(0.f, 0.f, 0.f, 0.f), o4 = x4;
        if (MODE == 1 && CHAR && dry4) x4 = load4<VEC>(Chi + idx, left);
        if (MODE == 1 && ARR && on && (f4 & 0x01010101u) != 0x01010101u) o4 = load4<VEC>(Om + idx, left);
        float Tb = 0.f, Kb = 0.f, Ta = 0.f, Ka = 0.f;
        if (edge_b) { Tb = __ldg(T + idx - 1); Kb = __ldg(K + idx - 1); }
        if (edge_a) { Ta = __ldg(T + idx + 4); Ka = __ldg(K + idx + 4); }
        const float2 k2a = __fmul2_rn(make_float2(2.0f, 2.0f), lo2(Kc)), k2b = __fmul2_rn(make_float2(2.0f, 2.0f), hi2(Kc));
        const float2 nta = __fmul2_rn(make_float2(-1.0f, -1.0f), lo2(Tc)), ntb = __fmul2_rn(make_float2(-1.0f, -1.0f), hi2(Tc));
        // z faces: f[v] between voxel v and v + 1, the lower one of voxel 0 from the lane below
        const float Tu = __shfl_down_sync(0xffffffffu, Tc.x, 1), Ku = __shfl_down_sync(0xffffffffu, Kc.x, 1);
        if (!edge_a) { Ta = Tu; Ka = Ku; }
        float fz0 = __fmul_rn(face(k2a.x, Kc.x, Kc.y, nta.x, Tc.y), g.idz2);
        float fz1 = __fmul_rn(face(k2a.y, Kc.y, Kc.z, nta.y, Tc.z), g.idz2);
        float fz2 = __fmul_rn(face(k2b.x, Kc.z, Kc.w, ntb.x, Tc.w), g.idz2);
        float fz3 = __fmul_rn(face(k2b.y, Kc.w, Ka, ntb.y, Ta), g.idz2);
        float fzb = -__shfl_up_sync(0xffffffffu, fz3, 1);
        if (edge_b) fzb = __fmul_rn(face(k2a.x, Kc.x, Kb, nta.x, Tb), g.idz2);
        float lo1 = -fz0, lo2_ = -fz1, lo3 = -fz2;
        if (wall) {
            // the row's first and last voxel lose heat through their z faces instead
            const int last = left - 1;
            const float Tw = gi == 0 ? Tc.x : (VEC || last == 3 ? Tc.w : last == 2 ? Tc.z : last == 1 ? Tc.y : Tc.x);
            const float kw = gi == 0 ? Kc.x : (VEC || last == 3 ? Kc.w : last == 2 ? Kc.z : last == 1 ? Kc.y : Kc.x);
            const float fl0 = zwall_flux<BC>(Tw, kw, g);
            if (gi == 0) fzb = fl0;
            if (gi == G - 1) {
                float up = fl0;
                if (G == 1) {
                    const float Tl = last == 3 ? Tc.w : last == 2 ? Tc.z : last == 1 ? Tc.y : Tc.x;
                    const float kl = last == 3 ? Kc.w : last == 2 ? Kc.z : last == 1 ? Kc.y : Kc.x;
                    up = zwall_flux<BC>(Tl, kl, g);
                }
                if (VEC || last == 3) fz3 = up;
                else if (last == 2) fz2 = up;
                else if (last == 1) fz1 = up;
                else fz0 = up;
            }
        }
        const float2 fea = scale2(face2(k2a, lo2(Kc), lo2(Ke), nta, lo2(Te)), g.idx2);
        const float2 feb = scale2(face2(k2b, hi2(Kc), hi2(Ke), ntb, hi2(Te)), g.idx2);
        float2 da = __fadd2_rn(fwa, fea), db = __fadd2_rn(fwb, feb);
        fwa = make_float2(-fea.x, -fea.y);
        fwb = make_float2(-feb.x, -feb.y);
        float2 sa = face2(k2a, lo2(Kc), lo2(Ks), nta, lo2(Ts)), sb = face2(k2b, hi2(Kc), hi2(Ks), ntb, hi2(Ts));
        if (!fuse) { sa = scale2(sa, g.idy2); sb = scale2(sb, g.idy2); }
        da = __ffma2_rn(sa, ys, da);
        db = __ffma2_rn(sb, ys, db);
        da = __fadd2_rn(da, scale2(face2(k2a, lo2(Kc), lo2(Kq), nta, lo2(Tq)), g.idy2));
        db = __fadd2_rn(db, scale2(face2(k2b, hi2(Kc), hi2(Kq), ntb, hi2(Tq)), g.idy2));
        da = __fadd2_rn(__fadd2_rn(da, make_float2(fzb, lo1)), make_float2(fz0, fz1));
        db = __fadd2_rn(__fadd2_rn(db, make_float2(lo2_, lo3)), make_float2(fz2, fz3));
        float2 qa = scale2(lo2(sr), c.q_scale), qb = scale2(hi2(sr), c.q_scale);
        if (MODE == 1 && c.zero_src_in_ablated && (f4 & 0x01010101u)) {
            if (f4 & 0x00000001u) qa.x = 0.0f;
            if (f4 & 0x00000100u) qa.y = 0.0f;
            if (f4 & 0x00010000u) qb.x = 0.0f;
            if (f4 & 0x01000000u) qb.y = 0.0f;
        }
        const float2 dt2 = make_float2(g.dt, g.dt);
        const float2 ra = rcp_approx2(make_float2(fmaxf(rho.x, 1e-12f), fmaxf(rho.y, 1e-12f)));
        const float2 rb = rcp_approx2(make_float2(fmaxf(rho.z, 1e-12f), fmaxf(rho.w, 1e-12f)));
        const float2 ta = __ffma2_rn(__fmul2_rn(dt2, __fadd2_rn(da, qa)), ra, lo2(Tc));
        const float2 tb = __ffma2_rn(__fmul2_rn(dt2, __fadd2_rn(db, qb)), rb, hi2(Tc));
        float out[4] = {ta.x, ta.y, tb.x, tb.y};
        if (MODE == 1) {
            float h[4] = {h4.x, h4.y, h4.z, h4.w};
            const float rh[4] = {rho.x, rho.y, rho.z, rho.w};
            const unsigned abl4 = f4 & 0x01010101u, dead4 = (f4 | (f4 >> 1)) & 0x01010101u;
            bool boils = false;   // a wet voxel above the plateau, or with enthalpy banked
            if (abl4) {
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (((f4 >> (8 * v)) & BD_FLAG_ABLATED) && out[v] > c.t_void) out[v] = c.t_void;
            }
            if (dead4 != 0x01010101u) {
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    boils |= !((f4 >> (8 * v)) & (BD_FLAG_ABLATED | BD_FLAG_DRY)) && (out[v] > c.t_abl || h[v] > 0.0f);
            }
            if (boils && on) {
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    if ((f4 >> (8 * v)) & (BD_FLAG_ABLATED | BD_FLAG_DRY)) continue;
                    if (out[v] > c.t_abl) {
                        h[v] = h[v] + (out[v] - c.t_abl) * rh[v];
                        out[v] = c.t_abl;
                    } else if (h[v] > 0.0f) {
                        const float rel = fminf(h[v], (c.t_abl - out[v]) * rh[v]);
                        h[v] = h[v] - rel;
                        out[v] = out[v] + rel / rh[v];
                    }
                }
                store4<VEC>(H + idx, h, left);
            }
            if (ARR && on && (f4 & 0x01010101u) != 0x01010101u) {
                float o[4] = {o4.x, o4.y, o4.z, o4.w};
#pragma unroll
                for (int v = 0; v < 4; ++v)
                    if (!((f4 >> (8 * v)) & BD_FLAG_ABLATED)) o[v] += g.dt * c.arr_A * expf(-c.arr_EaR / (out[v] + 273.15f));
                store4<VEC>(Om + idx, o, left);
            }
            if (CHAR) {
                const unsigned who = __ballot_sync(0xffffffffu, dry4 != 0u);
                // below t_cold the rate times dt is under 2^-27, and exp(-rate dt) is 1
                bool cold = true;
#pragma unroll
                for (int v = 0; v < 4; ++v) cold = cold && out[v] > -273.0f && out[v] < c.t_cold;
                if (who && !__any_sync(0xffffffffu, dry4 && !cold)) {
                    const float x[4] = {dry4 & 0x00000001u ? 1.0f - (1.0f - x4.x) : x4.x,
                                        dry4 & 0x00000100u ? 1.0f - (1.0f - x4.y) : x4.y,
                                        dry4 & 0x00010000u ? 1.0f - (1.0f - x4.z) : x4.z,
                                        dry4 & 0x01000000u ? 1.0f - (1.0f - x4.w) : x4.w};
                    if (dry4 && (x[0] != x4.x || x[1] != x4.y || x[2] != x4.z || x[3] != x4.w))
                        store4<VEC>(Chi + idx, x, left);
                } else if (who) {
                    // Two exponentials and a division a voxel, needed by the few dry ones: the warp's dry
                    // groups pass their voxels to all its lanes, 8 groups at a time (thin dry layers cost
                    // every warp that crosses one 4 rounds for a handful of lanes otherwise).
                    const int rank = __popc(who & ((1u << lane) - 1u));
                    float4* box = work[threadIdx.x >> 5];
                    for (int k0 = 0; k0 < __popc(who); k0 += 8) {
                        const int slot = rank - k0;
                        const bool mine = dry4 && slot >= 0 && slot < 8;
                        if (mine) {
                            box[slot] = make_float4(out[0], out[1], out[2], out[3]);
                            box[8 + slot] = x4;
                        }
                        __syncwarp();
                        const float Tv = reinterpret_cast<const float*>(box)[lane];
                        float* xp = reinterpret_cast<float*>(box + 8) + lane;
                        if (k0 + (lane >> 2) < __popc(who)) {
                            const float rate = c.char_A * expf(-c.char_EaR / (Tv + 273.15f));
                            *xp = 1.0f - (1.0f - *xp) * expf(-rate * g.dt);
                        }
                        __syncwarp();
                        if (mine) {
                            const float4 y = box[8 + slot];
                            const float x[4] = {dry4 & 0x00000001u ? y.x : x4.x, dry4 & 0x00000100u ? y.y : x4.y,
                                                dry4 & 0x00010000u ? y.z : x4.z, dry4 & 0x01000000u ? y.w : x4.w};
                            store4<VEC>(Chi + idx, x, left);
                        }
                        __syncwarp();
                    }
                }
            }
        }
        if (on) store4<VEC>(Tn + idx, out, left);
        Tc = Te;
        Kc = Ke;
    }
}

__global__ void k_pack_flags(const uint8_t* __restrict__ abl, const uint8_t* __restrict__ dry,
                             const uint8_t* __restrict__ vd, long long n, uint8_t* __restrict__ out) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        uint8_t a = abl[i] ? 1 : 0, d = dry[i] ? 1 : 0;
        uint8_t v = vd ? (vd[i] ? 1 : 0) : a;
        out[i] = (uint8_t)(a * BD_FLAG_ABLATED | d * BD_FLAG_DRY | v * BD_FLAG_VOID);
    }
}

static Geo make_geo(int nx, int ny, int nz, float dx, float dy, float dz, float dt, float h, float tamb) {
    Geo g;
    g.nx = nx; g.ny = ny; g.nz = nz;
    g.ni = 1;
    g.idx2 = 1.0f / (dx * dx); g.idy2 = 1.0f / (dy * dy); g.idz2 = 1.0f / (dz * dz);
    g.dz = dz; g.h_eff = h; g.t_amb = tamb; g.dt = dt;
    return g;
}

// Unused dynamic shared memory that lets at most `cap` substep CTAs share an SM (0: no cap). A plume stage
// of a launch per step runs beside the substeps, and capping them leaves its CTAs room on every SM (16 KB of
// shared memory per SM stay free for them). The chained plume kernel shares an SM with no substep CTA (it
// takes the registers), so beside it a cap only slows the substeps: laser-off epochs of 200x200x192 6.3 and
// 8.0 ms with 2 and 1 CTAs per SM, 5.3 without. The kernel's limit is raised once per instantiation.
static size_t substep_pad_bytes(int cap, const void* kernel) {
    if (cap <= 0) return 0;
    int dev = 0, per_sm = 0, per_block = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    cudaDeviceGetAttribute(&per_block, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    cudaFuncAttributes fa;
    if (cudaFuncGetAttributes(&fa, kernel) != cudaSuccess) return 0;
    const long long reserve = 1024;                  // per-CTA shared memory the system keeps
    long long pad = ((long long)per_sm - 16384) / cap - (long long)fa.sharedSizeBytes - reserve;
    pad = std::max(0LL, std::min(pad, (long long)per_block - (long long)fa.sharedSizeBytes));
    if (pad > 48 * 1024 && fa.maxDynamicSharedSizeBytes < pad)
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pad);
    return (size_t)pad;
}

// x planes per CTA: the knob's, fewer where that leaves the chip idle (a CTA of few planes reads its
// halo planes of T and k for fewer of its own). Aiming at 12 CTAs per SM: 150x150x138 0.64 ms per 20
// substeps against 0.69 - 0.74 at 6, 24 and 48; 200x200x192 takes the knob's 8 planes either way.
static int substep_planes(int tiles, int nx) {
    const int want = std::max(1, 148 * SUB_WAVE / std::max(1, tiles));   // chunks that fill the chip
    const int ni = std::max(1, std::min(tune_value(BD_TUNE_STENCIL_XC), nx / std::min(want, nx)));
    return std::max(ni, (nx + 65534) / 65535);   // chunks fit the grid's second dimension
}

template <int MODE, int BC, bool ARR, bool CHAR>
static void launch_substeps(const Geo& g, const AblConst& c, float* Ta, float* Tb, int n, const float* src,
                            const float* K, const float* R, const uint8_t* F, float* H, float* Om, float* Chi,
                            cudaStream_t st) {
    Geo gg = g;
    const int groups = (g.nz + 3) / 4 * g.ny;
    const int tiles = (groups + SUB_T - 1) / SUB_T;
    gg.ni = substep_planes(tiles, g.nx);
    const dim3 grid(tiles, (g.nx + gg.ni - 1) / gg.ni);
    const uintptr_t bits = (uintptr_t)Ta | (uintptr_t)Tb | (uintptr_t)src | (uintptr_t)K | (uintptr_t)R | (uintptr_t)H |
                           (uintptr_t)Om | (uintptr_t)Chi;
    const bool vec = g.nz % 4 == 0 && (bits & 15) == 0 && ((uintptr_t)F & 3) == 0;
    auto run = [&](auto v) {
        constexpr bool VEC = decltype(v)::value;
        const size_t pad = substep_pad_bytes(tune_value(BD_TUNE_STENCIL_CAP), (const void*)k_substep<MODE, BC, ARR, CHAR, VEC>);
        for (int s = 0; s < n; ++s)
            k_substep<MODE, BC, ARR, CHAR, VEC><<<grid, SUB_T, pad, st>>>(gg, c, (s & 1) ? Tb : Ta, (s & 1) ? Ta : Tb, src,
                                                                          K, R, F, H, Om, Chi);
    };
    if (vec) run(std::true_type{});
    else run(std::false_type{});
}

// The scale of the heat source; without one the kernel scales zeros, which an infinite or NaN scale must not reach.
static float source_scale(int is_active, float q_scale) { return is_active ? q_scale : 0.0f; }

// The synchronous entry points' end: waits for the launches and reports what went wrong in them.
static int finish(int rc, cudaStream_t st, const char* what) {
    if (rc) return rc;
    const cudaError_t e = cudaStreamSynchronize(st);
    return e == cudaSuccess ? BD_OK : cuda_status(e, what);
}

}  // namespace bd

using namespace bd;

extern "C" int bd_thermal_advance(const BdThermalParams* p, float* Ta, float* Tb, int n, const float* src,
                                  const float* K, const float* R, void* stream) {
    BD_REQUIRE(p != nullptr, "bd_thermal_advance: params is NULL");
    BD_REQUIRE(p->nx > 0 && p->ny > 0 && p->nz > 0, "bd_thermal_advance: grid dims must be positive");
    BD_REQUIRE(Ta && Tb && K && R, "bd_thermal_advance: NULL field");
    BD_REQUIRE(!p->is_active || src != nullptr, "bd_thermal_advance: active source needs src");
    BD_REQUIRE(p->bc_mode == BD_BC_SERIES || p->bc_mode == BD_BC_METAL, "bd_thermal_advance: bad bc_mode");
    BD_REQUIRE(n >= 0, "bd_thermal_advance: n_substeps must be >= 0");
    BD_REQUIRE((long long)p->nx * p->ny * p->nz < (1LL << 31), "bd_thermal_advance: grid exceeds 2^31 voxels");
    if (n == 0) return BD_OK;
    Geo g = make_geo(p->nx, p->ny, p->nz, p->dx, p->dy, p->dz, p->dt, p->h_eff, p->t_ambient);
    AblConst c{};
    c.q_scale = source_scale(p->is_active, p->q_scale);
    c.is_active = p->is_active;
    cudaStream_t st = as_stream(stream);
    if (p->bc_mode == BD_BC_SERIES)
        launch_substeps<0, BD_BC_SERIES, false, false>(g, c, Ta, Tb, n, src, K, R, nullptr, nullptr, nullptr, nullptr, st);
    else
        launch_substeps<0, BD_BC_METAL, false, false>(g, c, Ta, Tb, n, src, K, R, nullptr, nullptr, nullptr, nullptr, st);
    BD_CHECK_LAUNCH("k_substep<thermal>");
    return finish(BD_OK, st, "bd_thermal_advance");
}

namespace bd {
// The temperature (degC) up to which A exp(-E / T) dt stays below 2^-27: T = E / ln(A dt 2^27), a tenth of a
// kelvin lower for the rounding of the kernel's own evaluation. Nowhere (-inf) unless A, E, dt > 0.
static float char_cold_limit(double A, double E, double dt) {
    const double x = A * dt * 134217728.0;
    if (!(A > 0.0) || !(E > 0.0) || !(dt > 0.0) || !std::isfinite(x) || !std::isfinite(E)) return -INFINITY;
    if (x <= 1.0) return -INFINITY;   // below the limit at any temperature: rare enough for the general path
    return (float)(E / std::log(x) - 273.15 - 0.1);
}

int ablation_launch(const BdAblationParams* p, float* Ta, float* Tb, int n, float* H, float* Om, float* Chi,
                    const uint8_t* F, const float* src, const float* K, const float* R, cudaStream_t st) {
    Geo g = make_geo(p->nx, p->ny, p->nz, p->dx, p->dy, p->dz, p->dt, p->h_eff, p->t_ambient);
    AblConst c;
    c.t_abl = p->t_abl; c.t_void = p->t_void; c.q_scale = source_scale(p->is_active, p->q_scale);
    c.arr_A = p->arr_A; c.arr_EaR = p->arr_Ea_over_R; c.char_A = p->char_A; c.char_EaR = p->char_Ea_over_R;
    c.zero_src_in_ablated = p->zero_src_in_ablated; c.is_active = p->is_active;
    c.t_cold = p->has_char ? char_cold_limit(p->char_A, p->char_Ea_over_R, p->dt) : 0.0f;
    const bool arr = p->has_arrhenius != 0, chr = p->has_char != 0;
#define BD_ABL_CASE(BCV, A_, C_)                                                                 \
    if (p->bc_mode == BCV && arr == A_ && chr == C_) {                                           \
        launch_substeps<1, BCV, A_, C_>(g, c, Ta, Tb, n, src, K, R, F, H, Om, Chi, st);          \
        BD_CHECK_LAUNCH("k_substep<ablation>");                                                  \
        return BD_OK;                                                                            \
    }
    BD_ABL_CASE(BD_BC_SERIES, false, false)
    BD_ABL_CASE(BD_BC_SERIES, false, true)
    BD_ABL_CASE(BD_BC_SERIES, true, false)
    BD_ABL_CASE(BD_BC_SERIES, true, true)
    BD_ABL_CASE(BD_BC_METAL, false, false)
    BD_ABL_CASE(BD_BC_METAL, false, true)
    BD_ABL_CASE(BD_BC_METAL, true, false)
    BD_ABL_CASE(BD_BC_METAL, true, true)
#undef BD_ABL_CASE
    return fail(BD_ERR_INVALID_ARG, "bd_ablation_advance: bad bc_mode %d", p->bc_mode);
}

}  // namespace bd

extern "C" int bd_ablation_advance(const BdAblationParams* p, float* Ta, float* Tb, int n, float* H, float* Om,
                                   float* Chi, const uint8_t* F, const float* src, const float* K, const float* R,
                                   void* stream) {
    BD_REQUIRE(p != nullptr, "bd_ablation_advance: params is NULL");
    BD_REQUIRE(p->nx > 0 && p->ny > 0 && p->nz > 0, "bd_ablation_advance: grid dims must be positive");
    BD_REQUIRE(Ta && Tb && H && F && K && R, "bd_ablation_advance: NULL field");
    BD_REQUIRE(!p->is_active || src != nullptr, "bd_ablation_advance: active source needs src");
    BD_REQUIRE(!p->has_arrhenius || Om != nullptr, "bd_ablation_advance: Arrhenius needs Omega");
    BD_REQUIRE(!p->has_char || Chi != nullptr, "bd_ablation_advance: char kinetics need chi");
    BD_REQUIRE(n >= 0, "bd_ablation_advance: n_substeps must be >= 0");
    BD_REQUIRE((long long)p->nx * p->ny * p->nz < (1LL << 31), "bd_ablation_advance: grid exceeds 2^31 voxels");
    if (n == 0) return BD_OK;
    cudaStream_t st = as_stream(stream);
    return finish(ablation_launch(p, Ta, Tb, n, H, Om, Chi, F, src, K, R, st), st, "bd_ablation_advance");
}

extern "C" int bd_pack_flags(const uint8_t* abl, const uint8_t* dry, const uint8_t* vd, int64_t n, uint8_t* out,
                             void* stream) {
    BD_REQUIRE(abl && dry && out, "bd_pack_flags: NULL mask");
    if (n <= 0) return BD_OK;
    k_pack_flags<<<grid_for(n, 256), 256, 0, as_stream(stream)>>>(abl, dry, vd, n, out);
    BD_CHECK_LAUNCH("k_pack_flags");
    return BD_OK;
}
