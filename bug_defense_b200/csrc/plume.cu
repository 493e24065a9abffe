// Plume transport in the void domain (plume.py:18-80, metal_ablation_solver.py:193-240): FTCS
// diffusion with upwind drift, zero flux at solid walls (the neighbour value is replaced by the
// centre), Dirichlet 0 on the outer walls, clamped at 0, optional first-order decay.
//
// Kernels (all evaluate the same per-voxel expression, ftcs1 / ftcs4, so they are bit-identical):
//   k_plume_chain     BD_PLUME_KERNEL_DIRECT, the default: a whole stage in one launch, 4 FTCS steps per
//                     pass over the field
//   k_plume_direct    the default's stages of too few steps for a chain (chain_pays), and grids of more than
//                     255 z groups (nz > 1020): one launch per step, a CTA per 32 (z) x 16 (y) tile column;
//                     whole, aligned float4 rows
//   k_plume_step      the same for other rows: one voxel per thread
//   k_plume_direct_c  (BD_PLUME_KERNEL_COMPACT): one launch per step, one wave of CTAs looping over a
//                     compact list of the live units, x planes per unit chosen per stage
// Layout: C-order (nx, ny, nz), z fastest; the neighbourhood of every voxel is one mask byte.
#include "chain_wait.cuh"
#include "common.cuh"
#include "engine.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <type_traits>
#include <vector>

namespace bd {

constexpr int PM_TZ = 32, PM_TY = 8;  // k_plume_mask / k_plume_step block: 32 z x 8 y

// Plume neighbourhood byte per voxel, rebuilt whenever the void domain changes (epoch end); the
// bytes of one (x, y) column start every mz = plume_mask_pitch(nz) bytes (16-byte rows):
//   bit 6: voxel is void            bit 7: voxel is void and not on an outer wall (FTCS update)
//   bits 0-5: -x +x -y +y -z +z neighbour is void (otherwise its value is replaced by the centre,
//   the zero-flux wall of plume.py:61-71)
#define BD_PM_VOID 0x40u
#define BD_PM_UPDATE 0x80u
__global__ void k_plume_mask(int nx, int ny, int nz, int mz, const uint8_t* __restrict__ F,
                             uint8_t* __restrict__ M, const int* __restrict__ zlimit) {
    const int zl = zlimit ? min(max(*zlimit, 0), nz) : nz;
    const int j = blockIdx.x * PM_TY + threadIdx.y;
    const int i = blockIdx.y;
    if (j >= ny) return;
    const int plane = ny * nz;
    const bool xy_interior = (i > 0 && i < nx - 1 && j > 0 && j < ny - 1);
    const int col = i * plane + j * nz;
    const size_t mcol = ((size_t)i * ny + j) * mz;
    for (int k = threadIdx.x; k < zl; k += PM_TZ) {
        const int idx = col + k;
        uint8_t m = 0;
        if (F[idx] & BD_FLAG_VOID) {
            m = BD_PM_VOID;
            if (xy_interior && k > 0 && k < nz - 1) {
                m |= BD_PM_UPDATE;
                m |= (F[idx - plane] & BD_FLAG_VOID) ? 0x01 : 0;
                m |= (F[idx + plane] & BD_FLAG_VOID) ? 0x02 : 0;
                m |= (F[idx - nz] & BD_FLAG_VOID) ? 0x04 : 0;
                m |= (F[idx + nz] & BD_FLAG_VOID) ? 0x08 : 0;
                m |= (F[idx - 1] & BD_FLAG_VOID) ? 0x10 : 0;
                m |= (F[idx + 1] & BD_FLAG_VOID) ? 0x20 : 0;
            }
        }
        M[mcol + k] = m;
    }
}

struct PlumeConst {
    float dxy_x, dxy_y, dz_z;  // D_xy*idx2, D_xy*idy2, D_z*idz2
    float vz_over_dz, dtp, decay;
};

// Weights of one step. plume.py:46-80 updates a void voxel as
//   C' = decay * (C + dt (D_xy (lap_x + lap_y) + D_z lap_z - v (C - C_{+z}) / dz)),
// with a solid neighbour's value replaced by the centre's (zero flux). Every kernel keeps solid
// voxels at 0, so that replacement is the same as adding the solid neighbour's weight to the centre:
//   C' = decay * (w0eff C + wx (C_-x + C_+x) + wy (C_-y + C_+y) + wb C_-z + wt C_+z),
// w0eff = w0 + the weights of the solid neighbours, one of 64 values picked by the six neighbour
// bits of the voxel's mask byte. The table is built once per stage on the host, in float32, in a
// fixed order, so every kernel applies the same weights.
struct PlumeTab {
    float wx, wy, wb, wt, decay;
    int decays;          // decay != 1 (a factor of exactly 1 is skipped: x * 1 == x)
    float w0eff[64];
};

static PlumeTab make_plume_tab(const PlumeConst& c) {
    PlumeTab t;
    t.wx = c.dtp * c.dxy_x;
    t.wy = c.dtp * c.dxy_y;
    t.wb = c.dtp * c.dz_z;
    const float adv = c.dtp * c.vz_over_dz;
    t.wt = t.wb + adv;
    const float w0 = 1.0f - 2.0f * (t.wx + t.wy + t.wb) - adv;
    for (int b = 0; b < 64; ++b) {
        float e = w0;
        if (!(b & 0x01)) e += t.wx;
        if (!(b & 0x02)) e += t.wx;
        if (!(b & 0x04)) e += t.wy;
        if (!(b & 0x08)) e += t.wy;
        if (!(b & 0x10)) e += t.wb;
        if (!(b & 0x20)) e += t.wt;
        t.w0eff[b] = e;
    }
    t.decay = c.decay;
    t.decays = c.decay != 1.0f;
    return t;
}

// One voxel (the scalar form; the packed form below performs the same operations per component).
__device__ __forceinline__ float ftcs1(float c0, float w, float e, float s, float n, float b, float t, unsigned m,
                                       const PlumeTab& k) {
    float a = __fmul_rn(k.w0eff[m & 0x3Fu], c0);
    a = __fmaf_rn(k.wx, __fadd_rn(w, e), a);
    a = __fmaf_rn(k.wy, __fadd_rn(s, n), a);
    a = __fmaf_rn(k.wb, b, a);
    a = __fmaf_rn(k.wt, t, a);
    if (k.decays) a = __fmul_rn(a, k.decay);
    return (m & BD_PM_UPDATE) ? fmaxf(a, 0.0f) : 0.0f;
}

// Four consecutive z voxels (one float4 and their four mask bytes); zb / zt: the voxels below and
// above the group. Pairs of voxels go through the packed FP32x2 operations of sm_100 (each lane
// rounded as the scalar operation), which halves the arithmetic instructions.
// w0eff: the table of effective centre weights, wherever the caller keeps it (shared memory in
// every step kernel).
__device__ __forceinline__ float4 ftcs4(float4 c, float4 w, float4 e, float4 s, float4 n, float zb, float zt,
                                        unsigned m, const PlumeTab& k, const float* w0eff) {
    const float2 wx = make_float2(k.wx, k.wx), wy = make_float2(k.wy, k.wy);
    const float2 wb = make_float2(k.wb, k.wb), wt = make_float2(k.wt, k.wt);
    // a group whose four voxels have six void neighbours each (the bulk of the domain) needs no lookup
    float2 wa, wc;
    if ((m & 0x3F3F3F3Fu) == 0x3F3F3F3Fu) {
        wa = wc = make_float2(w0eff[0x3F], w0eff[0x3F]);
    } else {
        wa = make_float2(w0eff[m & 0x3Fu], w0eff[(m >> 8) & 0x3Fu]);
        wc = make_float2(w0eff[(m >> 16) & 0x3Fu], w0eff[(m >> 24) & 0x3Fu]);
    }
    float2 a = __fmul2_rn(wa, make_float2(c.x, c.y));
    float2 b = __fmul2_rn(wc, make_float2(c.z, c.w));
    a = __ffma2_rn(wx, __fadd2_rn(make_float2(w.x, w.y), make_float2(e.x, e.y)), a);
    b = __ffma2_rn(wx, __fadd2_rn(make_float2(w.z, w.w), make_float2(e.z, e.w)), b);
    a = __ffma2_rn(wy, __fadd2_rn(make_float2(s.x, s.y), make_float2(n.x, n.y)), a);
    b = __ffma2_rn(wy, __fadd2_rn(make_float2(s.z, s.w), make_float2(n.z, n.w)), b);
    a = __ffma2_rn(wb, make_float2(zb, c.x), a);
    b = __ffma2_rn(wb, make_float2(c.y, c.z), b);
    a = __ffma2_rn(wt, make_float2(c.y, c.z), a);
    b = __ffma2_rn(wt, make_float2(c.w, zt), b);
    if (k.decays) {
        const float2 d = make_float2(k.decay, k.decay);
        a = __fmul2_rn(a, d);
        b = __fmul2_rn(b, d);
    }
    float4 v;
    v.x = (m & 0x00000080u) ? fmaxf(a.x, 0.0f) : 0.0f;
    v.y = (m & 0x00008000u) ? fmaxf(a.y, 0.0f) : 0.0f;
    v.z = (m & 0x00800000u) ? fmaxf(b.x, 0.0f) : 0.0f;
    v.w = (m & 0x80000000u) ? fmaxf(b.y, 0.0f) : 0.0f;
    return v;
}

// mask bytes of a 4-voxel group starting at z = k that lie below the void limit zl
__device__ __forceinline__ unsigned zkeep_mask(int zl, int k) {
    const int nk = zl - k;
    return nk >= 4 ? 0xffffffffu : (nk <= 0 ? 0u : (0xffffffffu >> (8 * (4 - nk))));
}

// Non-void voxels of a field set to 0 (the context API's input may hold anything there): afterwards
// both ping-pong buffers satisfy the invariant every step relies on.
__global__ void k_plume_clear(float* __restrict__ Ca, float* __restrict__ Cb, const uint8_t* __restrict__ M, int nx,
                              int ny, int nz, int mz) {
    const long long n = (long long)nx * ny * nz;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const long long col = i / nz;
        const int k = (int)(i - col * nz);
        if (!(M[col * mz + k] & BD_PM_VOID)) {
            Ca[i] = 0.0f;
            Cb[i] = 0.0f;
        }
    }
}

// ---- k_plume_step: any grid ----------------------------------------------------------------
// One FTCS step. CTA (y tile, x plane); a thread owns the voxels k = tx, tx+32, ... < zlim of one
// (x, y) column (zlim = *zlimit when given, every void voxel lies above it, else nz); only void
// voxels are written (solid voxels stay 0).
__global__ void __launch_bounds__(PM_TZ * PM_TY) k_plume_step(int nx, int ny, int nz, int mz,
                                                              const __grid_constant__ PlumeTab k,
                                                              const float* __restrict__ C, float* __restrict__ Cn,
                                                              const uint8_t* __restrict__ M,
                                                              const int* __restrict__ zlimit) {
    const int zl = zlimit ? min(max(*zlimit, 0), nz) : nz;
    const int j = blockIdx.x * PM_TY + threadIdx.y;
    const int i = blockIdx.y;
    if (j >= ny) return;
    const int plane = ny * nz;
    const int col = i * plane + j * nz;
    const size_t mcol = ((size_t)i * ny + j) * mz;
    for (int z = threadIdx.x; z < zl; z += PM_TZ) {
        const int idx = col + z;
        const unsigned m = __ldg(&M[mcol + z]);
        if (!(m & BD_PM_VOID)) continue;
        if (!(m & BD_PM_UPDATE)) {
            Cn[idx] = 0.0f;
            continue;
        }
        // an updated voxel is never on an outer wall: all six neighbours exist
        Cn[idx] = ftcs1(__ldg(&C[idx]), __ldg(&C[idx - plane]), __ldg(&C[idx + plane]), __ldg(&C[idx - nz]),
                        __ldg(&C[idx + nz]), __ldg(&C[idx - 1]), __ldg(&C[idx + 1]), m, k);
    }
}

// ---- one step per launch: the units of the direct, the compact and the batched kernel ----------
// A unit is 16 rows (y) by 8 live z groups and marches xc x planes; thread = 4 consecutive z voxels of
// one row, a warp 8 such groups x 4 rows (one 128-byte line per row and load). The thread keeps the
// x-1 / x float4 of its row in registers and loads, per plane, the next plane's float4 and the
// centre plane's y neighbours from the (L2-resident) field beside the plane's mask bytes (one
// 32-bit load): one L2 round trip per plane, at the price of loads a tissue plane does not need. The
// z neighbours come from the neighbouring lanes by shuffle (the unit's edge lanes load them).
// Latency is hidden by the many independent units of a step. Only void voxels are written. Needs
// nz % 4 == 0 and 16-byte aligned fields.
constexpr int PD_BY = 16;  // rows of a unit (8 * PD_BY threads)
static_assert(PD_BY == kPlumeZRows, "z-list columns follow the units' y tiles");

__device__ __forceinline__ void store_void(float* dst, float4 v, unsigned vd) {
    if (vd == 0x40404040u) {
        *reinterpret_cast<float4*>(dst) = v;
    } else {
        if (vd & 0x00000040u) dst[0] = v.x;
        if (vd & 0x00004000u) dst[1] = v.y;
        if (vd & 0x00400000u) dst[2] = v.z;
        if (vd & 0x40000000u) dst[3] = v.w;
    }
}

// Live z groups of every (x chunk, y tile) column of units: a CTA per column (grid
// n_yt x n_chunks), thread g = the 4-voxel z group g; live when any of the column's planes and rows
// holds a void voxel in the group below the void z-limit (the mask bytes at or above it are not
// rebuilt, so they are masked off here). The void domain is fixed within a plume stage, so the
// lists are built once per stage, after the mask.
__global__ void __launch_bounds__(256) k_plume_zlist(const uint8_t* __restrict__ M, int nx, int ny, int nz, int mz,
                                                     int xc, const int* __restrict__ zlimit,
                                                     uint8_t* __restrict__ zlist) {
    __shared__ int wcount[8];
    const int zl = zlimit ? min(max(*zlimit, 0), nz) : nz;
    const int G = (nz + 3) / 4;
    const int n_yt = gridDim.x;
    const int n_cols = gridDim.x * gridDim.y;
    const int col = blockIdx.y * n_yt + blockIdx.x;
    const int ib = blockIdx.y * xc, ie = min(nx, ib + xc);
    const int j0 = blockIdx.x * PD_BY, j1 = min(ny, j0 + PD_BY);
    const int g = threadIdx.x;
    bool live = false;
    if (g < G && zl - 4 * g > 0) {
        const unsigned keep = zkeep_mask(zl, 4 * g);
        for (int i = ib; i < ie && !live; ++i)
            for (int j = j0; j < j1; ++j)
                if (__ldg(reinterpret_cast<const unsigned*>(M + ((size_t)i * ny + j) * mz + 4 * g)) & keep &
                    0x40404040u) {
                    live = true;
                    break;
                }
    }
    const unsigned bal = __ballot_sync(0xffffffffu, live);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) wcount[w] = __popc(bal);
    __syncthreads();
    int before = 0;
    for (int q = 0; q < w; ++q) before += wcount[q];
    if (live) zlist[n_cols + (size_t)col * G + before + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)g;
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int q = 0; q < 8; ++q) tot += wcount[q];
        zlist[col] = (uint8_t)tot;
    }
}

// One unit: band `band` of column `col` (y tile yt, x chunk xch of xc planes)
// takes the column's live groups 8 band .. 8 band + 7 from its z list instead of 8 consecutive
// groups, so z tiles that are partly tissue cost only their void groups. A lane whose z neighbour
// group is not held by the neighbouring lane loads that neighbour voxel instead of taking it by
// shuffle. Voxels outside the lists are not void and are never written. Uniform over the CTA.
// g: this lane's z group (-2 when the band has no group for the lane); uniform early exit over the
// CTA when the x chunk is empty.
__device__ __forceinline__ void plume_unit_groups(const float* __restrict__ C, float* __restrict__ Cn,
                                                  const uint8_t* __restrict__ M, int nx, int ny, int nz, int mz,
                                                  int xc, const PlumeTab& k, int zl, int g, int yt, int xch,
                                                  const float* w0s) {
    const int ib = xch * xc, ie = min(nx, ib + xc);
    if (ib >= ie) return;
    const int zg = threadIdx.x & 7;
    const int gp = __shfl_up_sync(0xffffffffu, g, 1, 8);
    const int gn = __shfl_down_sync(0xffffffffu, g, 1, 8);
    const bool zb_lane = zg > 0 && gp == g - 1;  // the -z neighbour is the previous lane's last voxel
    const bool zt_lane = zg < 7 && gn == g + 1;  // the +z neighbour is the next lane's first voxel
    const int j = yt * PD_BY + ((threadIdx.x & 127) >> 3), z = 4 * max(g, 0);
    const bool act = g >= 0 && zl - z > 0 && j < ny;
    const bool in = g >= 0 && j < ny && z < nz;
    const unsigned zkeep = zkeep_mask(zl, z);
    // 32-bit element offsets (grids have < 2^31 voxels); rows past the grid load nothing
    const int plane = ny * nz, mplane = ny * mz;
    const int jj = min(j, ny - 1);
    int off = (ib * ny + jj) * nz + z;
    int moff = (ib * ny + jj) * mz + z;
    const bool ys = in && j > 0, yn = in && j + 1 < ny;
    const bool ebl = !zb_lane && in && z > 0, etl = !zt_lane && in && z + 4 < nz;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 cw = in && ib > 0 ? __ldg(reinterpret_cast<const float4*>(C + (off - plane))) : z4;
    float4 cc = in ? __ldg(reinterpret_cast<const float4*>(C + off)) : z4;
    for (int i = ib; i < ie; ++i, off += plane, moff += mplane) {
        const unsigned mr = act ? (__ldg(reinterpret_cast<const unsigned*>(M + moff)) & zkeep) : 0u;
        const float4 ce = in && i + 1 < nx ? __ldg(reinterpret_cast<const float4*>(C + (off + plane))) : z4;
        const float4 cs = ys ? __ldg(reinterpret_cast<const float4*>(C + (off - nz))) : z4;
        const float4 cn = yn ? __ldg(reinterpret_cast<const float4*>(C + (off + nz))) : z4;
        const float eb = ebl ? __ldg(C + (off - 1)) : 0.0f;
        const float et = etl ? __ldg(C + (off + 4)) : 0.0f;
        const unsigned vd = mr & 0x40404040u;
        if (__any_sync(0xffffffffu, act && vd)) {
            float zb = __shfl_up_sync(0xffffffffu, cc.w, 1, 8);
            float zt = __shfl_down_sync(0xffffffffu, cc.x, 1, 8);
            if (!zb_lane) zb = eb;
            if (!zt_lane) zt = et;
            const float4 v = ftcs4(cc, cw, ce, cs, cn, zb, zt, mr, k, w0s);
            if (act && vd) store_void(Cn + off, v, vd);
        }
        cw = cc;
        cc = ce;
    }
}

// The unit (column col, band) with its groups read from the column's z list.
__device__ __forceinline__ void plume_direct_unit(const float* __restrict__ C, float* __restrict__ Cn,
                                                  const uint8_t* __restrict__ M, int nx, int ny, int nz, int mz,
                                                  int xc, const PlumeTab& k, int zl, const uint8_t* __restrict__ zlist,
                                                  int n_cols, int col, int yt, int xch, int band, const float* w0s) {
    const int G = (nz + 3) / 4;
    const int cnt = zlist[col];
    const int b0 = band * 8;
    if (b0 >= cnt) return;  // uniform over the CTA
    const int zg = threadIdx.x & 7;
    const int g = b0 + zg < cnt ? (int)zlist[n_cols + col * G + b0 + zg] : -2;
    plume_unit_groups(C, Cn, M, nx, ny, nz, mz, xc, k, zl, g, yt, xch, w0s);
}

// One step over a grid of units: blockIdx = (band, y tile, x chunk), the bands from the columns' z lists, or of
// 8 consecutive z groups where there are none (nz > 1020: a group's id is a byte in a list; 64 x 64 x 1200, 680
// steps: 7.0 ms a call, 14.0 ms by one voxel per thread).
template <bool LISTED>
__global__ void __launch_bounds__(8 * PD_BY, 9) k_plume_direct(const float* __restrict__ C, float* __restrict__ Cn,
                                                               const uint8_t* __restrict__ M, int nx, int ny, int nz,
                                                               int mz, int xc, const __grid_constant__ PlumeTab k,
                                                               const int* __restrict__ zlimit,
                                                               const uint8_t* __restrict__ zlist) {
    __shared__ float w0s[64];
    if (threadIdx.x < 64) w0s[threadIdx.x] = k.w0eff[threadIdx.x];
    __syncthreads();
    const int zl = zlimit ? min(max(*zlimit, 0), nz) : nz;
    if (LISTED) {
        plume_direct_unit(C, Cn, M, nx, ny, nz, mz, xc, k, zl, zlist, gridDim.y * gridDim.z,
                          blockIdx.z * gridDim.y + blockIdx.y, blockIdx.y, blockIdx.z, blockIdx.x, w0s);
    } else {
        const int g0 = 8 * (int)blockIdx.x, g = g0 + (threadIdx.x & 7);
        if (4 * g0 >= zl) return;  // uniform over the CTA
        plume_unit_groups(C, Cn, M, nx, ny, nz, mz, xc, k, zl, 4 * g < zl ? g : -2, blockIdx.y, blockIdx.z, w0s);
    }
}

// ---- BD_PLUME_KERNEL_COMPACT: a compact list of live units, one launch per step --------------
// A step's CTAs are dispatched at a limited rate and the step ends with its last CTA, so the step is
// fastest when the live units about fill one wave of resident CTAs: each CTA then runs exactly one
// unit, and no empty CTA is dispatched between working ones. Once per stage the x planes per unit
// (xc) are chosen on the device: per (x plane, y tile) bitmaps of the live z groups give the unit
// count of every candidate xc, and the smallest xc whose count fits the wave (3 % over allowed)
// wins (fewer planes per unit = a shorter CTA). The z list and the unit list are then built for it
// and the step kernel, one wave of CTAs, loops over the units. Region layout (32-bit words, from
// plume_units_offset): [0] unit count, [1] chosen xc, [4 + c - kPlumeXcMin] unit count for xc = c,
// then the bitmaps (nx x y tiles x kPlumeBitWords), then the units: 16 bytes each, {column << 5 |
// band, 0, the band's 8 z-group ids as bytes (0xFF: none)}.
constexpr int kPlumeXcMin = 2, kPlumeXcMax = 12;
constexpr int kPlumeBitWords = 8;  // 32-group words of a bitmap: 4-voxel groups <= 255
constexpr int kPlumeHdrWords = 16;

// bit g of (x plane i, y tile yt): a voxel of group g below the void z-limit in the tile's rows is void
__global__ void __launch_bounds__(256) k_plume_planebits(const uint8_t* __restrict__ M, int nx, int ny, int nz,
                                                         int mz, const int* __restrict__ zlimit,
                                                         unsigned* __restrict__ bits) {
    const int zl = zlimit ? min(max(*zlimit, 0), nz) : nz;
    const int G = (nz + 3) / 4;
    const int yt = blockIdx.x, i = blockIdx.y, n_yt = gridDim.x;
    const int j0 = yt * PD_BY, j1 = min(ny, j0 + PD_BY);
    const int g = threadIdx.x;
    bool live = false;
    if (g < G && zl - 4 * g > 0) {
        const unsigned keep = zkeep_mask(zl, 4 * g);
        for (int j = j0; j < j1 && !live; ++j)
            live = (__ldg(reinterpret_cast<const unsigned*>(M + ((size_t)i * ny + j) * mz + 4 * g)) & keep &
                    0x40404040u) != 0u;
    }
    const unsigned bal = __ballot_sync(0xffffffffu, live);
    if ((threadIdx.x & 31) == 0) bits[((size_t)i * n_yt + yt) * kPlumeBitWords + (threadIdx.x >> 5)] = bal;
}

// live units (bands of 8 live groups) for candidate xc = kPlumeXcMin + blockIdx.x
__global__ void __launch_bounds__(1024) k_plume_unit_counts(const unsigned* __restrict__ bits, int nx, int n_yt,
                                                            int G, unsigned* __restrict__ hdr) {
    __shared__ int tot;
    if (threadIdx.x == 0) tot = 0;
    __syncthreads();
    const int c = kPlumeXcMin + blockIdx.x;
    const int n_xch = (nx + c - 1) / c;
    const int W = (G + 31) / 32;
    int mine = 0;
    for (int p = threadIdx.x; p < n_xch * n_yt; p += blockDim.x) {
        const int xch = p / n_yt, yt = p - xch * n_yt;
        const int ib = xch * c, ie = min(nx, ib + c);
        int live = 0;
        for (int w = 0; w < W; ++w) {
            unsigned o = 0u;
            for (int i = ib; i < ie; ++i) o |= __ldg(&bits[((size_t)i * n_yt + yt) * kPlumeBitWords + w]);
            live += __popc(o);
        }
        mine += (live + 7) / 8;
    }
    atomicAdd(&tot, mine);
    __syncthreads();
    if (threadIdx.x == 0) hdr[4 + blockIdx.x] = (unsigned)tot;
}

// the smallest candidate xc whose unit count fits slot_cap (else the largest)
__global__ void k_plume_pick_xc(unsigned* __restrict__ hdr, int slot_cap) {
    if (threadIdx.x != 0) return;
    int pick = kPlumeXcMax;
    for (int c = kPlumeXcMin; c <= kPlumeXcMax; ++c)
        if ((int)hdr[4 + c - kPlumeXcMin] <= slot_cap) {
            pick = c;
            break;
        }
    hdr[1] = (unsigned)pick;
}

// z lists of the chosen xc's columns from the bitmaps (the layout of k_plume_zlist's lists); grid
// (y tiles, x chunks of the smallest candidate), chunks past the chosen xc's exit
__global__ void __launch_bounds__(256) k_plume_zlist_bits(const unsigned* __restrict__ bits, int nx, int nz,
                                                          const unsigned* __restrict__ hdr,
                                                          uint8_t* __restrict__ zlist) {
    __shared__ int wcount[8];
    const int c = (int)hdr[1];
    const int n_xch = (nx + c - 1) / c;
    const int yt = blockIdx.x, xch = blockIdx.y, n_yt = gridDim.x;
    if (xch >= n_xch) return;  // uniform over the CTA
    const int G = (nz + 3) / 4;
    const int n_cols = n_yt * n_xch;
    const int col = xch * n_yt + yt;
    const int ib = xch * c, ie = min(nx, ib + c);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned o = 0u;
    if (32 * w < G)
        for (int i = ib; i < ie; ++i) o |= __ldg(&bits[((size_t)i * n_yt + yt) * kPlumeBitWords + w]);
    const int g = threadIdx.x;
    const bool live = g < G && ((o >> lane) & 1u);
    const unsigned bal = __ballot_sync(0xffffffffu, live);
    if (lane == 0) wcount[w] = __popc(bal);
    __syncthreads();
    int before = 0;
    for (int q = 0; q < w; ++q) before += wcount[q];
    if (live) zlist[n_cols + (size_t)col * G + before + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)g;
    if (threadIdx.x == 0) {
        int tot = 0;
        for (int q = 0; q < 8; ++q) tot += wcount[q];
        zlist[col] = (uint8_t)tot;
    }
}

// the unit list of the chosen xc's columns, in column order: one CTA, a block-wide exclusive scan
// of the bands per column
__global__ void __launch_bounds__(1024) k_plume_units(const uint8_t* __restrict__ zlist, int nx, int n_yt, int G,
                                                      unsigned* __restrict__ hdr, uint4* __restrict__ units) {
    __shared__ int part[32];
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    const int c = (int)hdr[1];
    const int n_cols = n_yt * ((nx + c - 1) / c);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int c0 = 0; c0 < n_cols; c0 += 1024) {
        const int col = c0 + threadIdx.x;
        const int nb = col < n_cols ? (zlist[col] + 7) / 8 : 0;
        int v = nb;  // inclusive scan within the warp
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += t;
        }
        if (lane == 31) part[w] = v;
        __syncthreads();
        if (w == 0) {
            int x = part[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += t;
            }
            part[lane] = x;
        }
        __syncthreads();
        const int excl = base + (w > 0 ? part[w - 1] : 0) + v - nb;
        for (int b = 0; b < nb; ++b) {
            // the band's group ids, one byte per lane (0xFF: no group), so that a step's CTA learns
            // its unit with one 16-byte load
            const uint8_t* gl = zlist + n_cols + (size_t)col * G + 8 * b;
            const int n_in = min(8, (int)zlist[col] - 8 * b);
            unsigned lo = 0u, hi = 0u;
            for (int q = 0; q < 8; ++q) {
                const unsigned gq = q < n_in ? (unsigned)gl[q] : 0xFFu;
                if (q < 4) lo |= gq << (8 * q);
                else hi |= gq << (8 * (q - 4));
            }
            units[excl + b] = make_uint4(((unsigned)col << 5) | (unsigned)b, 0u, lo, hi);
        }
        __syncthreads();
        if (threadIdx.x == 1023) base = excl + nb;
        __syncthreads();
    }
    if (threadIdx.x == 0) hdr[0] = (unsigned)base;
}

// One step over the unit list: a wave of CTAs, each running kPlumeUnitsPerCta units at a time, one per
// 128-thread group (the groups share no barrier): group g of CTA b runs units 3b + g, 3b + g + 3 grid,
// ... A step's wave is then dispatched as a third as many CTAs with the same resident threads per SM.
constexpr int kPlumeUnitsPerCta = 3;
__global__ void __launch_bounds__(8 * PD_BY * kPlumeUnitsPerCta, 3) k_plume_direct_c(const float* __restrict__ C, float* __restrict__ Cn,
                                                                 const uint8_t* __restrict__ M, int nx, int ny,
                                                                 int nz, int mz, const __grid_constant__ PlumeTab k,
                                                                 const int* __restrict__ zlimit,
                                                                 const unsigned* __restrict__ hdr,
                                                                 const uint4* __restrict__ units, int n_yt,
                                                                 int unit_cap) {
    // the CTA's first unit record is loaded beside the header (not after the unit count is known):
    // one L2 round trip before the field loads; a record past the count is never used
    const int grp = threadIdx.x >> 7;  // this thread's unit slot within the CTA
    const int u0 = (int)blockIdx.x * kPlumeUnitsPerCta + grp;
    const uint4 r0 = __ldg(&units[min(u0, unit_cap - 1)]);
    const int nu = (int)__ldg(&hdr[0]);
    const int xc = (int)__ldg(&hdr[1]);
    const int zl = zlimit ? min(max(*zlimit, 0), nz) : nz;
    __shared__ float w0s[64];
    if (threadIdx.x < 64) w0s[threadIdx.x] = k.w0eff[threadIdx.x];
    __syncthreads();
    const int zg = threadIdx.x & 7;
    for (int u = u0; u < nu; u += gridDim.x * kPlumeUnitsPerCta) {
        // column << 5 | band, then the band's 8 group ids
        const uint4 r = u == u0 ? r0 : __ldg(&units[u]);
        const int col = (int)(r.x >> 5);
        const int xch = col / n_yt;
        const unsigned gb = ((zg < 4 ? r.z : r.w) >> (8 * (zg & 3))) & 0xFFu;
        plume_unit_groups(C, Cn, M, nx, ny, nz, mz, xc, k, zl, gb == 0xFFu ? -2 : (int)gb, col - xch * n_yt, xch,
                          w0s);
    }
}

// ---- BD_PLUME_KERNEL_DIRECT: a chain of blocks of S FTCS steps in one launch -------------------
// One step moves 9 bytes per void voxel for 13 operations; a launch per step spends its time on
// dispatch and L2 round trips, and a launch per few steps recomputes the halo planes of every x
// chunk. Here a stage is one launch. A unit is 16 rows (y) by up to 32 consecutive 4-voxel groups
// (z) over the x range where they hold void. A CTA advances a unit by S steps while it marches once
// along x with the time levels staggered by one plane: when plane p arrives, level 1 is computed on
// plane p-1, level 2 on p-2, ... and level S is written for plane p-S. The next S steps of the same
// unit are another CTA's, which follows a few planes behind: it reads what the units of its own and
// the two neighbouring row tiles have written, as far as their progress counters say. Only the row
// halo (4 on each side) is computed twice; nothing is recomputed along x.
//
// As many CTAs as there are SMs are launched, and those that can have no work leave at once: the stages of
// several small instances, and a stage's photons and substeps, run beside it (8 instances of 64x64x144, laser off:
// 23.6 ms an epoch with all CTAs staying, 10.2 ms now, 14.2 ms by a launch per step).
// A CTA takes (block of steps, unit) pairs by a ticket, blocks in order, and waits only on the block
// before its own, that is on lower tickets, whose CTAs are running or done: the lowest unfinished
// ticket never waits, whatever else occupies the GPU. Every wait is bounded and raises *err.
// Two buffers do: a unit writes plane q of block j over block j - 2's after its inputs up to plane
// q + S are there, and the units of block j - 1 that read plane q have by then written plane q + S.
//
// A warp holds two rows (lane = z group); the planes a level needs stay in registers, z neighbours
// come by shuffle, and the rows above and below a warp's pair come from shared memory, where every
// level's plane was put one iteration earlier: one barrier per plane for all S levels. Each voxel is
// evaluated by the same expression as everywhere else (ftcs4), so the bits depend neither on S nor
// on the tiling; what the row halo recomputes is discarded. Groups outside a unit's are solid, or
// its first and last are halo groups: a run of live groups longer than 32 is split into windows
// that overlap by one group on each side (S <= 4 voxels).
//
// What bounds it: 12 warps of 168 registers fill an SM, and their FMA, shared-memory and issue slots
// are each about half busy (issue 47 %, 417 instructions per warp and plane); DRAM 1 %, L2 13 %.
// Measured on 3.58 M void voxels of 200 x 200 x 192, 680 steps: 4.16 ms, against 8.45 ms for one
// launch per step (k_plume_direct_c), 6.4 ms for one launch per 4 steps with x chunks and their halo
// planes, and 4.4 - 5.6 ms for 2 or 3 steps per pass, 1 row per warp or 16 warps of 128 registers.
// Laser-off epoch of the full-resolution run 9.38 -> 6.01 ms, 48 x 48 x 144 laser-on 3.08 -> 2.18 ms.
constexpr int kChainHalo = 4;                                  // halo rows; at most as many steps per block
constexpr int kChainR = 2;                                     // rows of a warp
constexpr int kChainWarps = (kChainRows + 2 * kChainHalo) / kChainR;
constexpr int kChainThreads = 32 * kChainWarps;
constexpr int chain_smem_bytes(int S) { return 2 * S * 2 * kChainWarps * 32 * (int)sizeof(float4); }
constexpr int kChainDone = 0x7fffffff;

struct ChainUnit {
    int tile, first, lo, hi;   // y tile; first group loaded; groups written
    int ix0, ix1, _p0, _p1;    // planes on which the written groups may hold void
};
static_assert(sizeof(ChainUnit) == kChainUnitBytes, "unit records fill their region");

// Regions of a stage's plan in its scratch.
struct ChainPlan {
    unsigned* hdr;       // [0] units, [1] ticket, [2] CTAs arrived
    int* tile_start;     // first unit of each y tile, and the end
    unsigned* bits;      // live groups of (x plane, y tile with its halo rows)
    ChainUnit* units;
    int* progress;       // [block][unit]: planes below this are written
    int cap;
};

static ChainPlan chain_plan(uint8_t* mask, int nx, int ny, int nz) {
    ChainPlan p;
    const size_t n_yt = (ny + kChainRows - 1) / kChainRows;
    uint8_t* at = mask + plume_chain_offset(nx, ny, nz);
    p.hdr = reinterpret_cast<unsigned*>(at);
    at += 256;
    p.tile_start = reinterpret_cast<int*>(at);
    at += chain_round((n_yt + 1) * sizeof(int));
    p.bits = reinterpret_cast<unsigned*>(at);
    at += chain_round((size_t)nx * n_yt * kPlumeBitWords * sizeof(unsigned));
    p.units = reinterpret_cast<ChainUnit*>(at);
    at += chain_round(plume_chain_capacity(ny, nz) * sizeof(ChainUnit));
    p.progress = reinterpret_cast<int*>(at);
    p.cap = (int)plume_chain_capacity(ny, nz);
    return p;
}

// The field is written by other SMs during the kernel: it is read past the L1.
template <bool VEC>
__device__ __forceinline__ float4 chain_load(const float* p, int left) {
    if (VEC) return __ldcg(reinterpret_cast<const float4*>(p));
    float4 v;                       // left: voxels of the row from p on
    v.x = __ldcg(p);
    v.y = left > 1 ? __ldcg(p + 1) : 0.0f;
    v.z = left > 2 ? __ldcg(p + 2) : 0.0f;
    v.w = left > 3 ? __ldcg(p + 3) : 0.0f;
    return v;
}

template <bool VEC>
__device__ __forceinline__ void chain_store(float* p, const float4& v, int left) {
    if (VEC) {
        __stcg(reinterpret_cast<float4*>(p), v);
        return;
    }
    p[0] = v.x;
    if (left > 1) p[1] = v.y;
    if (left > 2) p[2] = v.z;
    if (left > 3) p[3] = v.w;
}

// Per-voxel factors of a group from its four mask bytes: the effective centre weight, and the decay
// (or 1) for a voxel that is updated, 0 for one that is not. A factor of exactly 1 leaves the bits.
struct ChainFactors {
    float2 wa, wc, da, dc;
};
__device__ __forceinline__ ChainFactors chain_factors(unsigned m, float decay, const float* w0eff) {
    ChainFactors f;
    f.wa = make_float2(w0eff[m & 0x3Fu], w0eff[(m >> 8) & 0x3Fu]);
    f.wc = make_float2(w0eff[(m >> 16) & 0x3Fu], w0eff[(m >> 24) & 0x3Fu]);
    f.da = make_float2((m & 0x00000080u) ? decay : 0.0f, (m & 0x00008000u) ? decay : 0.0f);
    f.dc = make_float2((m & 0x00800000u) ? decay : 0.0f, (m & 0x80000000u) ? decay : 0.0f);
    return f;
}

// ftcs4 with the factors at hand. The z terms are scalar: their operand pairs straddle the registers
// of c, and pairing them up costs the moves that a packed operation saves.
__device__ __forceinline__ float4 chain_ftcs4(const float4& c, const float4& w, const float4& e, const float4& s,
                                              const float4& n, float zb, float zt, const ChainFactors& f,
                                              const PlumeTab& k) {
    const float2 wx = make_float2(k.wx, k.wx), wy = make_float2(k.wy, k.wy);
    float2 a = __fmul2_rn(f.wa, make_float2(c.x, c.y));
    float2 b = __fmul2_rn(f.wc, make_float2(c.z, c.w));
    a = __ffma2_rn(wx, __fadd2_rn(make_float2(w.x, w.y), make_float2(e.x, e.y)), a);
    b = __ffma2_rn(wx, __fadd2_rn(make_float2(w.z, w.w), make_float2(e.z, e.w)), b);
    a = __ffma2_rn(wy, __fadd2_rn(make_float2(s.x, s.y), make_float2(n.x, n.y)), a);
    b = __ffma2_rn(wy, __fadd2_rn(make_float2(s.z, s.w), make_float2(n.z, n.w)), b);
    a.x = __fmaf_rn(k.wt, c.y, __fmaf_rn(k.wb, zb, a.x));
    a.y = __fmaf_rn(k.wt, c.z, __fmaf_rn(k.wb, c.x, a.y));
    b.x = __fmaf_rn(k.wt, c.w, __fmaf_rn(k.wb, c.y, b.x));
    b.y = __fmaf_rn(k.wt, zt, __fmaf_rn(k.wb, c.z, b.y));
    a = __fmul2_rn(a, f.da);
    b = __fmul2_rn(b, f.dc);
    return make_float4(fmaxf(a.x, 0.0f), fmaxf(a.y, 0.0f), fmaxf(b.x, 0.0f), fmaxf(b.y, 0.0f));
}

template <int S, bool VEC>
__global__ void __launch_bounds__(kChainThreads, 1) k_plume_chain(float* Ca, float* Cb,
                                                                  const uint8_t* __restrict__ M, int nx, int ny,
                                                                  int nz, int mz, const __grid_constant__ PlumeTab k,
                                                                  const int* __restrict__ zlimit, ChainPlan plan,
                                                                  int nblocks, int in_flight, int* err) {
    constexpr int R = kChainR;
    extern __shared__ float4 lev[];  // [plane parity][level][warp][first, last row][lane]
    __shared__ float w0s[64];
    __shared__ int ticket_s;
    constexpr int kPar = S * kChainWarps * 2 * 32;
    if (threadIdx.x < 64) w0s[threadIdx.x] = k.w0eff[threadIdx.x];
    const int nu = (int)__ldg(&plan.hdr[0]);
    // No more CTAs stay than can have work: the others would hold an SM each until the stage ends. The first to
    // arrive stay, which are near each other (by index: 400x64x64, 120 steps 1.35 ms a call, 1.08 so).
    if ((long long)nu * in_flight < gridDim.x) {
        if (threadIdx.x == 0) ticket_s = (int)atomicAdd(&plan.hdr[2], 1u);
        __syncthreads();
        if (ticket_s >= nu * in_flight) return;
    }
    const int zl = zlimit ? min(max(*zlimit, 0), nz) : nz;
    const int n_yt = (ny + kChainRows - 1) / kChainRows;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, row0 = R * warp;
    const int ws = max(warp - 1, 0) * 64 + 32, wn = min(warp + 1, kChainWarps - 1) * 64;
    // levels whose rows of this warp some written row depends on
    const int nlev = min(S, max(0, min(row0 + R - 1 - kChainHalo, kChainHalo + kChainRows - 1 - row0) + S));
    const int plane = ny * nz, mplane = ny * mz;
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) ticket_s = (int)atomicAdd(&plan.hdr[1], 1u);
        __syncthreads();
        const int ticket = ticket_s;
        const int j = nu > 0 ? ticket / nu : nblocks;
        if (j >= nblocks) break;
        const int u = ticket - j * nu;
        const ChainUnit rec = plan.units[u];
        const float* C = (j & 1) ? Cb : Ca;
        float* Cn = (j & 1) ? Ca : Cb;
        // warp 0 waits for the units of the block before: those of this and the neighbouring y tiles
        const int* up = plan.progress + (size_t)max(j - 1, 0) * plan.cap;
        int* mine = plan.progress + (size_t)j * plan.cap + u;
        const int d0 = plan.tile_start[max(rec.tile - 1, 0)], d1 = plan.tile_start[min(rec.tile + 2, n_yt)];
        int seen = 0, vx0 = 0, vx1 = 0;  // of this lane's first unit
        if (d0 + lane < d1) {
            vx0 = plan.units[d0 + lane].ix0;
            vx1 = plan.units[d0 + lane].ix1;
        }
        bool ok = true;
        auto wait_plane = [&](int p) {
            if (j == 0 || !ok) return;
            if (p >= vx0 && p < vx1 && seen <= p) ok = chain_wait(up + d0 + lane, p, seen, err);
            for (int v = d0 + lane + 32; v < d1; v += 32) {
                int s2 = 0;
                if (ok && p >= plan.units[v].ix0 && p < plan.units[v].ix1) ok = chain_wait(up + v, p, s2, err);
            }
            ok = __all_sync(0xffffffffu, ok);
        };
        const int ib = rec.ix0, ie = rec.ix1;
        const int y0 = rec.tile * kChainRows - kChainHalo + row0;
        const int g = rec.first + lane, z = 4 * g;
        const unsigned keep = zkeep_mask(zl, z);
        unsigned inr = 0u, wrr = 0u;   // bit r: row r is in the grid / written
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (z < nz && y0 + r >= 0 && y0 + r < ny) {
                inr |= 1u << r;
                if (g >= rec.lo && g <= rec.hi && row0 + r >= kChainHalo && row0 + r < kChainHalo + kChainRows)
                    wrr |= 1u << r;
            }
        }
        const int left = nz - z;
        const int p0 = ib - S, p1 = ie + S;
        const float* cp = C + ((long long)p0 * plane + y0 * nz + z);      // plane p0, read only inside the grid
        const uint8_t* mp = M + ((long long)p0 * mplane + y0 * mz + z);
        float* dst = Cn + ((long long)ib * plane + y0 * nz + z);
        // V[l][q]: this thread's row groups of level l, plane p - l in slot (p - l - p0) mod 3
        float4 V[S][3][R];
        unsigned mk[S][R];  // mask words of plane p - l - 1
        unsigned nm[R];     // of the plane in flight
        // the factors in use and the masks they are for: computed again only where a level's mask
        // differs from the last one in a lane of the warp, that is near the walls of a cavity
        unsigned cm[R];
        ChainFactors f[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
#pragma unroll
            for (int l = 0; l < S; ++l) {
                V[l][0][r] = V[l][1][r] = V[l][2][r] = z4;
                mk[l][r] = 0u;
            }
            nm[r] = cm[r] = 0u;
            f[r].wa = f[r].wc = f[r].da = f[r].dc = make_float2(0.f, 0.f);
        }
        auto fetch = [&](int p, float4 (&e)[R]) {
            const bool in = p >= 0 && p < nx;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                e[r] = z4;
                nm[r] = 0u;
                if (in && (inr >> r) & 1u) {
                    e[r] = chain_load<VEC>(cp + r * nz, left);
                    nm[r] = __ldg(reinterpret_cast<const unsigned*>(mp + r * mz));
                }
            }
            cp += plane;
            mp += mplane;
        };
        auto advance = [&](auto phase, int p) {
            constexpr int B = 3 * S + decltype(phase)::value;
            const int age = p - p0;
            float4* put = lev + (p & 1) * kPar + warp * 64 + lane;
            const float4* get = lev + ((p + 1) & 1) * kPar + lane;
            // plane p - 1 - S was stored before the last barrier; the last warp, which has few rows to
            // compute, publishes it
            if (threadIdx.x == kChainThreads - 32 && age > 2 * S) st_release(mine, p - S);
            float4 o[R];
            unsigned m[R];  // of plane p
#pragma unroll
            for (int r = 0; r < R; ++r) m[r] = nm[r] & keep;
            auto each = [&](auto fn) {
                fn(std::integral_constant<int, 0>{});
                if constexpr (S > 1) fn(std::integral_constant<int, 1>{});
                if constexpr (S > 2) fn(std::integral_constant<int, 2>{});
                if constexpr (S > 3) fn(std::integral_constant<int, 3>{});
            };
            each([&](auto lc) {
                constexpr int l = decltype(lc)::value;
                const float4(&e)[R] = V[l][(B - l) % 3];
                const float4(&c)[R] = V[l][(B - l - 1) % 3];
                const float4(&w)[R] = V[l][(B - l - 2) % 3];
                put[l * kChainWarps * 64] = e[0];
                put[l * kChainWarps * 64 + 32] = e[R - 1];
                unsigned any = 0u, df = 0u;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    o[r] = z4;
                    any |= mk[l][r];
                    df |= mk[l][r] ^ cm[r];
                }
                if (l < nlev && age >= 2 * (l + 1) && __any_sync(0xffffffffu, any & 0x80808080u)) {
                    const float4 s = get[l * kChainWarps * 64 + ws];
                    const float4 n = get[l * kChainWarps * 64 + wn];
                    if (__any_sync(0xffffffffu, df)) {
#pragma unroll
                        for (int r = 0; r < R; ++r) {
                            cm[r] = mk[l][r];
                            f[r] = chain_factors(cm[r], k.decay, w0s);
                        }
                    }
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        float bz = __shfl_up_sync(0xffffffffu, c[r].w, 1);
                        float tz = __shfl_down_sync(0xffffffffu, c[r].x, 1);
                        if (lane == 0) bz = 0.0f;    // solid (its weight is in w0eff), or a halo group
                        if (lane == 31) tz = 0.0f;
                        o[r] = chain_ftcs4(c[r], w[r], e[r], r == 0 ? s : c[max(r - 1, 0)],
                                           r == R - 1 ? n : c[min(r + 1, R - 1)], bz, tz, f[r], k);
                    }
                }
                if constexpr (l + 1 < S) {
#pragma unroll
                    for (int r = 0; r < R; ++r) V[l + 1][(B - l - 1) % 3][r] = o[r];
                }
                if constexpr (l == 0) {
                    if (p + 1 < p1) fetch(p + 1, V[0][(B + 1) % 3]);
                }
            });
#pragma unroll
            for (int r = 0; r < R; ++r) {
#pragma unroll
                for (int l = S - 1; l > 0; --l) mk[l][r] = mk[l - 1][r];
                mk[0][r] = m[r];
            }
            if (age >= 2 * S) {
#pragma unroll
                for (int r = 0; r < R; ++r)
                    if ((wrr >> r) & 1u) chain_store<VEC>(dst + r * nz, o[r], left);  // solid voxels hold 0 already
                dst += plane;
            }
            if (warp == 0) wait_plane(p + 2);  // fetched by every warp in the next iteration
            __syncthreads();
        };
        if (warp == 0) {
            for (int p = p0; p < p0 + 2; ++p) wait_plane(p);
        }
        __syncthreads();
        fetch(p0, V[0][0]);
        for (int p = p0; p < p1;) {
            advance(std::integral_constant<int, 0>{}, p);
            if (++p >= p1) break;
            advance(std::integral_constant<int, 1>{}, p);
            if (++p >= p1) break;
            advance(std::integral_constant<int, 2>{}, p);
            ++p;
        }
        if (threadIdx.x == 0) st_release(mine, kChainDone);
    }
}

// bit g of (x plane, y tile): a voxel of group g below the void z-limit is void in the tile's rows or
// its halo rows. CTA per (y tile, x plane), a warp per row, 32 groups a pass.
__global__ void __launch_bounds__(256) k_plume_chain_bits(const uint8_t* __restrict__ M, int ny, int nz, int mz,
                                                          const int* __restrict__ zlimit,
                                                          unsigned* __restrict__ bits) {
    __shared__ unsigned w8[kPlumeBitWords];
    const int zl = zlimit ? min(max(*zlimit, 0), nz) : nz;
    if (threadIdx.x < kPlumeBitWords) w8[threadIdx.x] = 0u;
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int j0 = max(0, (int)blockIdx.x * kChainRows - kChainHalo);
    const int j1 = min(ny, (int)(blockIdx.x + 1) * kChainRows + kChainHalo);
    for (int w = 0; 128 * w < zl; ++w) {
        const int z = 128 * w + 4 * lane;
        unsigned m = 0u;
        if (z < zl)
            for (int j = j0 + warp; j < j1; j += 8)
                m |= __ldg(reinterpret_cast<const unsigned*>(M + ((size_t)blockIdx.y * ny + j) * mz + z));
        const unsigned bal = __ballot_sync(0xffffffffu, (m & zkeep_mask(zl, z) & 0x40404040u) != 0u);
        if (lane == 0 && bal) atomicOr(&w8[w], bal);
    }
    __syncthreads();
    if (threadIdx.x < kPlumeBitWords)
        bits[((size_t)blockIdx.y * gridDim.x + blockIdx.x) * kPlumeBitWords + threadIdx.x] = w8[threadIdx.x];
}

__device__ __forceinline__ bool chain_bit(const unsigned* o, int g) { return (o[g >> 5] >> (g & 31)) & 1u; }

// The stage's units, one CTA: a warp ORs a y tile's live groups over x, cuts them into windows of 32
// groups and finds the x range of each.
__global__ void __launch_bounds__(1024) k_plume_chain_units(ChainPlan plan, int nx, int n_yt, int G) {
    __shared__ unsigned live[32][kPlumeBitWords];
    __shared__ int count[32];
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int t0 = 0; t0 < n_yt; t0 += 32) {
        const int t = t0 + warp;
        __syncthreads();
        if (t < n_yt) {
            unsigned o[kPlumeBitWords] = {0u, 0u, 0u, 0u, 0u, 0u, 0u, 0u};
            for (int i = lane; i < nx; i += 32) {
                const uint4* b = reinterpret_cast<const uint4*>(plan.bits + ((size_t)i * n_yt + t) * kPlumeBitWords);
                const uint4 q = __ldg(b), r = __ldg(b + 1);
                o[0] |= q.x; o[1] |= q.y; o[2] |= q.z; o[3] |= q.w;
                o[4] |= r.x; o[5] |= r.y; o[6] |= r.z; o[7] |= r.w;
            }
#pragma unroll
            for (int w = 0; w < kPlumeBitWords; ++w) {
                const unsigned v = __reduce_or_sync(0xffffffffu, o[w]);
                if (lane == 0) live[warp][w] = v;
            }
        }
        __syncwarp();
        // windows of this tile: counted first, then written behind those of the tiles before
        for (int pass = 0; pass < 2; ++pass) {
            int at = 0;
            if (pass == 1) {
                at = base;
                for (int w = 0; w < warp; ++w) at += count[w];
                if (t < n_yt && lane == 0) plan.tile_start[t] = at;
            }
            int n = 0;
            for (int g = 0; t < n_yt && g < G;) {
                const unsigned* o = live[warp];
                if (!chain_bit(o, g)) {
                    ++g;
                    continue;
                }
                const int first = g > 0 && chain_bit(o, g - 1) ? g - 1 : g;  // a live group before: one halo group
                int last = min(G - 1, first + 31);
                if (last + 1 < G && last > g && chain_bit(o, last) && chain_bit(o, last + 1)) --last;  // one after
                if (pass == 1) {
                    int lo = nx, hi = 0;
                    for (int i = lane; i < nx; i += 32) {
                        bool any = false;
                        for (int w = g >> 5; w <= (last >> 5); ++w) {
                            unsigned v = __ldg(plan.bits + ((size_t)i * n_yt + t) * kPlumeBitWords + w);
                            if (w == (g >> 5)) v &= 0xffffffffu << (g & 31);
                            if (w == (last >> 5)) v &= 0xffffffffu >> (31 - (last & 31));
                            any |= v != 0u;
                        }
                        if (any) {
                            lo = min(lo, i);
                            hi = max(hi, i + 1);
                        }
                    }
                    lo = __reduce_min_sync(0xffffffffu, lo);
                    hi = __reduce_max_sync(0xffffffffu, hi);
                    if (lane == 0) plan.units[at + n] = ChainUnit{t, first, g, last, lo, hi, 0, 0};
                }
                ++n;
                g = last + 1;
            }
            if (pass == 0) {
                if (lane == 0) count[warp] = n;
                __syncthreads();
            }
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 0; w < 32; ++w) base += count[w];
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        plan.tile_start[n_yt] = base;
        plan.hdr[0] = (unsigned)base;
        plan.hdr[1] = 0u;
    }
}

template <int S, bool VEC>
static cudaError_t chain_launch(int slots, float* Ca, float* Cb, const uint8_t* mask, int nx, int ny, int nz, int mz,
                                const PlumeTab& tab, const int* zl, const ChainPlan& plan, int nblocks, int* err,
                                cudaStream_t st) {
    constexpr int smem = chain_smem_bytes(S);
    cudaError_t e = cudaFuncSetAttribute(k_plume_chain<S, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess) e = cudaMemsetAsync(plan.hdr + 1, 0, 2 * sizeof(unsigned), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(plan.progress, 0, sizeof(int) * (size_t)plan.cap * nblocks, st);
    if (e != cudaSuccess) return e;
    // a block reads plane p + 2 after the one before has written it, S + 3 planes behind its own front
    const int in_flight = std::min(nblocks, (nx + 2 * S) / (S + 3) + 2);
    k_plume_chain<S, VEC><<<slots, kChainThreads, smem, st>>>(Ca, Cb, mask, nx, ny, nz, mz, tab, zl, plan, nblocks,
                                                              in_flight, err);
    return cudaGetLastError();
}

template <bool VEC>
static cudaError_t chain_blocks(int S, int slots, float* Ca, float* Cb, const uint8_t* mask, int nx, int ny, int nz,
                                int mz, const PlumeTab& tab, const int* zl, const ChainPlan& plan, int nblocks,
                                int* err, cudaStream_t st) {
    switch (S) {
        case 4: return chain_launch<4, VEC>(slots, Ca, Cb, mask, nx, ny, nz, mz, tab, zl, plan, nblocks, err, st);
        case 3: return chain_launch<3, VEC>(slots, Ca, Cb, mask, nx, ny, nz, mz, tab, zl, plan, nblocks, err, st);
        case 2: return chain_launch<2, VEC>(slots, Ca, Cb, mask, nx, ny, nz, mz, tab, zl, plan, nblocks, err, st);
        default: return chain_launch<1, VEC>(slots, Ca, Cb, mask, nx, ny, nz, mz, tab, zl, plan, nblocks, err, st);
    }
}

// Whether a stage of `total` steps is shorter as a chain than as a launch per step. A chain marches along all of x
// before its first block of 4 steps is done, and once more for a remainder of 1 to 3 steps, on one SM per 16 rows;
// a launch per step has a fixed cost and then the voxels'. Estimates in us, set so that they cross where the measured
// times do. A step in a captured stage: 4.2 + 0.7 a million voxels (3.1 to 11.6 in all, by the depth of the void
// domain), scalar rows 3.3 + 1.8 (1.9 to 18). `whole`: launched one by one by the host, 6.2 at least, without a void
// limit. A plane of a block of steps: 1.45 (measured 1.1 to 1.3), scalar rows 1.6 (1.5), of a remainder 1.2 and
// 1.3 (1.0 and 1.25); the next block is 8.5 planes behind (7 to 10).
// Laser-off epochs, chain and a launch per step: 200x200x192, 2 steps 475 and 272 us, 34 steps 816 and 594, 68 steps
// 993 and 966, 170 steps 1778 and 2131, 680 steps 5289 and 8875; 1000x24x144, 10 steps 2296 and 281, 680 steps
// 4904 and 5393; 48x48x144, 10 steps 190 and 110, 68 steps 287 and 335; 48x48x143, 34 steps 274 and 106, 680 steps
// 2234 and 2340.
static bool chain_pays(int nx, int ny, int nz, long long total, bool vec, bool whole, int nsm) {
    const double vox = 1e-6 * nx * ny * nz;
    const double step = whole ? std::max(6.2, vec ? 4.2 + 1.0 * vox : 4.0 + 3.1 * vox)
                              : vec ? 4.2 + 0.7 * vox : 3.3 + 1.8 * vox;
    const double plane = vec ? 1.45 : 1.6, tail = vec ? 1.2 : 1.3, lag = 8.5;
    // units: one or more windows of z groups per 16 rows; blocks beyond those on the chip start as others end
    const double units = (double)((ny + kChainRows - 1) / kChainRows) * std::max(1.0, nz / 240.0);
    const double on_chip = std::max(1.0, std::floor(nsm / units));
    const long long blocks = total / kChainHalo, rest = total % kChainHalo;
    double chain = 10.0;
    if (blocks > 0) {
        const double march = nx + 2.0 * kChainHalo, turns = std::floor((blocks - 1) / on_chip);
        chain += plane * (march + turns * std::max(march, lag * on_chip) + (blocks - 1 - turns * on_chip) * lag);
    }
    if (rest > 0) chain += tail * (nx + 2.0 * rest);
    return chain < step * total;
}

int plume_policy_steps(const BdPlumeParams* p, int* n_steps, float* dt_step, float* decay_step) {
    const double idx2 = 1.0 / ((double)p->dx * p->dx), idy2 = 1.0 / ((double)p->dy * p->dy);
    const double idz2 = 1.0 / ((double)p->dz * p->dz);
    const double d_rate = (double)p->D_xy * (idx2 + idy2) + (double)p->D_z * idz2;
    const double dt = p->dt;
    const bool decays = p->tau_linger > 0.0f && std::isfinite(p->tau_linger);
    if (p->dt_policy == BD_PLUME_DT_AS_GIVEN) {
        *n_steps = 1; *dt_step = (float)dt;
        *decay_step = decays ? (float)std::exp(-dt / p->tau_linger) : 1.0f;
    } else if (p->dt_policy == BD_PLUME_DT_METAL) {
        // dt_plume = min(dt, 0.45 / (2 d_rate)); decay still uses the substep dt
        float dr = (float)p->D_xy * ((float)idx2 + (float)idy2) + (float)p->D_z * (float)idz2;
        *n_steps = 1;
        *dt_step = dr > 1e-6f ? std::min((float)dt, 0.45f / (2.0f * dr)) : (float)dt;
        *decay_step = decays ? (float)std::exp(-dt / p->tau_linger) : 1.0f;
    } else if (p->dt_policy == BD_PLUME_DT_SUBCYCLE) {
        int n = p->n_sub;
        if (n <= 0) {
            // FTCS with upwind drift keeps every coefficient >= 0 while
            // dt (2 d_rate + vz/dz) <= 1; use 90 % of that limit.
            const double rate = 2.0 * d_rate + std::max(0.0, (double)p->vz) / p->dz;
            n = std::max(1, (int)std::ceil(dt * rate / 0.9 - 1e-9));
        }
        *n_steps = n;
        *dt_step = (float)(dt / n);
        *decay_step = decays ? (float)std::exp(-(dt / n) / p->tau_linger) : 1.0f;
    } else {
        return fail(BD_ERR_INVALID_ARG, "unknown plume dt policy %d", p->dt_policy);
    }
    return BD_OK;
}

// One wave of the compact step kernel on the current device: resident CTAs per SM x SMs (cached).
static int compact_slots() {
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0) dev = 0;
    const int d = dev < 64 ? dev : 63;
    int v = cache[d].load();
    if (v > 0) return v;
    int nsm = 0, per = 0;
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_plume_direct_c, 8 * PD_BY * kPlumeUnitsPerCta, 0);
    v = std::max(1, nsm) * std::max(1, per) * kPlumeUnitsPerCta;  // units of one wave
    cache[d].store(v);
    return v;
}

// A plume stage: n_substeps x (steps per substep) FTCS steps on the ping-pong pair (Ca, Cb), the
// field in Ca on entry. *in_b = 1 when the result ends in Cb. With full_first (the context API, whose
// non-void voxels may hold anything) the mask covers the whole grid and the non-void voxels of both
// buffers are set to 0 first (every step keeps them 0).
int plume_launch(const BdPlumeParams* p, float* Ca, float* Cb, int n_substeps, const uint8_t* F, int* in_b,
                 cudaStream_t st, const int* zlimit, int full_first, uint8_t* mask, int* err) {
    int steps;
    float dtp, decay;
    int rc = plume_policy_steps(p, &steps, &dtp, &decay);
    if (rc) return rc;
    PlumeConst c;
    c.dxy_x = p->D_xy / (p->dx * p->dx);
    c.dxy_y = p->D_xy / (p->dy * p->dy);
    c.dz_z = p->D_z / (p->dz * p->dz);
    c.vz_over_dz = p->vz > 0.0f ? p->vz / p->dz : 0.0f;
    c.dtp = dtp;
    c.decay = decay;
    const PlumeTab tab = make_plume_tab(c);
    const int nx = p->nx, ny = p->ny, nz = p->nz;
    const int mz = plume_mask_pitch(nz);
    BD_REQUIRE((long long)nx * ny * mz < (1LL << 31), "plume: grid %dx%dx%d exceeds 2^31 mask bytes", nx, ny, nz);
    const int* zl = full_first ? nullptr : zlimit;
    k_plume_mask<<<dim3((ny + PM_TY - 1) / PM_TY, nx), dim3(PM_TZ, PM_TY), 0, st>>>(nx, ny, nz, mz, F, mask, zl);
    BD_CHECK_LAUNCH("k_plume_mask");
    if (full_first) {
        k_plume_clear<<<grid_for((int64_t)nx * ny * nz, 256), 256, 0, st>>>(Ca, Cb, mask, nx, ny, nz, mz);
        BD_CHECK_LAUNCH("k_plume_clear");
    }
    const long long total = (long long)steps * n_substeps;
    const int kernel = tune_value(BD_TUNE_PLUME_KERNEL);
    const bool vec = nz % 4 == 0 && plume_aligned(Ca, Cb);  // rows of whole float4 groups
    if (kernel == BD_PLUME_KERNEL_COMPACT && vec && (nz + 3) / 4 <= 255) {
        const int n_yt = (ny + PD_BY - 1) / PD_BY;
        unsigned* hdr = reinterpret_cast<unsigned*>(mask + plume_units_offset(nx, ny, nz));
        unsigned* bits = hdr + kPlumeHdrWords;
        uint4* units = reinterpret_cast<uint4*>(bits + (size_t)nx * n_yt * kPlumeBitWords);
        const int unit_cap = (int)plume_unit_capacity(nx, ny, nz);
        uint8_t* zlist = mask + plume_zlist_offset(nx, ny, nz);
        const int slots = compact_slots();
        k_plume_planebits<<<dim3(n_yt, nx), 256, 0, st>>>(mask, nx, ny, nz, mz, zl, bits);
        k_plume_unit_counts<<<kPlumeXcMax - kPlumeXcMin + 1, 1024, 0, st>>>(bits, nx, n_yt, (nz + 3) / 4, hdr);
        k_plume_pick_xc<<<1, 32, 0, st>>>(hdr, slots + slots * 3 / 100);
        k_plume_zlist_bits<<<dim3(n_yt, (nx + kPlumeXcMin - 1) / kPlumeXcMin), 256, 0, st>>>(bits, nx, nz, hdr, zlist);
        k_plume_units<<<1, 1024, 0, st>>>(zlist, nx, n_yt, (nz + 3) / 4, hdr, units);
        BD_CHECK_LAUNCH("k_plume_units");
        for (long long s = 0; s < total; ++s) {
            const float* in = (s & 1) ? Cb : Ca;
            float* out = (s & 1) ? Ca : Cb;
            k_plume_direct_c<<<slots / kPlumeUnitsPerCta, 8 * PD_BY * kPlumeUnitsPerCta, 0, st>>>(
                in, out, mask, nx, ny, nz, mz, tab, zl, hdr, units, n_yt, unit_cap);
        }
        BD_CHECK_LAUNCH("k_plume_direct_c");
        if (in_b) *in_b = (int)(total & 1);
        return BD_OK;
    }
    const bool groups_in_byte = (nz + 3) / 4 <= 255;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    const int slots = std::max(1, nsm);
    if (groups_in_byte && chain_pays(nx, ny, nz, total, vec, full_first != 0, slots)) {
        const int n_yt = (ny + kChainRows - 1) / kChainRows;
        const ChainPlan plan = chain_plan(mask, nx, ny, nz);
        k_plume_chain_bits<<<dim3(n_yt, nx), 256, 0, st>>>(mask, ny, nz, mz, zl, plan.bits);
        k_plume_chain_units<<<1, 1024, 0, st>>>(plan, nx, n_yt, (nz + 3) / 4);
        BD_CHECK_LAUNCH("k_plume_chain_units");
        int flips = 0;
        for (long long left = total; left > 0;) {
            const int S = (int)std::min<long long>(left, kChainHalo);
            const int nb = (int)std::min<long long>(left / S, kChainBlocks);
            float* a = (flips & 1) ? Cb : Ca;
            float* b = (flips & 1) ? Ca : Cb;
            const cudaError_t e = vec ? chain_blocks<true>(S, slots, a, b, mask, nx, ny, nz, mz, tab, zl, plan, nb, err, st)
                                      : chain_blocks<false>(S, slots, a, b, mask, nx, ny, nz, mz, tab, zl, plan, nb, err, st);
            if (e != cudaSuccess) return cuda_status(e, "k_plume_chain");
            flips += nb;
            left -= (long long)S * nb;
        }
        if (in_b) *in_b = flips & 1;
        return BD_OK;
    }
    const int xc = tune_value(BD_TUNE_PLUME_XC);
    const dim3 dgrid((nz + 31) / 32, (ny + PD_BY - 1) / PD_BY, (nx + xc - 1) / xc);
    const bool direct = vec && dgrid.y <= 65535;
    const bool listed = direct && groups_in_byte;
    uint8_t* zlist = mask + plume_zlist_offset(nx, ny, nz);
    if (listed) k_plume_zlist<<<dim3(dgrid.y, dgrid.z), 256, 0, st>>>(mask, nx, ny, nz, mz, xc, zl, zlist);
    for (long long s = 0; s < total; ++s) {
        const float* in = (s & 1) ? Cb : Ca;
        float* out = (s & 1) ? Ca : Cb;
        if (listed)
            k_plume_direct<true><<<dgrid, 8 * PD_BY, 0, st>>>(in, out, mask, nx, ny, nz, mz, xc, tab, zl, zlist);
        else if (direct)
            k_plume_direct<false><<<dgrid, 8 * PD_BY, 0, st>>>(in, out, mask, nx, ny, nz, mz, xc, tab, zl, nullptr);
        else
            k_plume_step<<<dim3((ny + PM_TY - 1) / PM_TY, nx), dim3(PM_TZ, PM_TY), 0, st>>>(nx, ny, nz, mz, tab, in, out,
                                                                                            mask, zl);
    }
    BD_CHECK_LAUNCH("k_plume_step");
    if (in_b) *in_b = (int)(total & 1);
    return BD_OK;
}

// ---- batched stages: several instances' plume steps in one launch per step ------------------
// The instances may differ in diffusivity, so each carries its own weights and step count. They
// are ranked by step count (rank 0 steps longest); a unit of rank r is (r << 27) | (column << 5) |
// band, and the unit list is in (rank, column) order, so the units of step s are a prefix of it:
// those of the ranks that still step. The header holds the unit count [0] and, at [16 + r], the
// units of ranks 0..r; the units follow at word 64.
struct PlumeInstDev {
    float* Ca;
    float* Cb;
    const uint8_t* mask;
    const int* zlimit;
    long long steps;  // FTCS steps of the stage (steps per substep x substeps)
    PlumeTab tab;
};
constexpr int kBatchHdrWords = 64;

__global__ void __launch_bounds__(1024) k_plume_batch_units(const PlumeInstDev* __restrict__ insts, int n,
                                                            int n_cols, size_t zoff, unsigned* __restrict__ hdr) {
    __shared__ int part[32];
    __shared__ int base;
    if (threadIdx.x == 0) base = 0;
    __syncthreads();
    unsigned* units = hdr + kBatchHdrWords;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int total = n * n_cols;
    for (int c0 = 0; c0 < total; c0 += 1024) {
        const int q = c0 + threadIdx.x;
        int nb = 0, r = 0, col = 0;
        if (q < total) {
            r = q / n_cols;
            col = q - r * n_cols;
            nb = (insts[r].mask[zoff + col] + 7) / 8;
        }
        int v = nb;  // inclusive scan within the warp
        for (int o = 1; o < 32; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += t;
        }
        if (lane == 31) part[w] = v;
        __syncthreads();
        if (w == 0) {
            int x = part[lane];
            for (int o = 1; o < 32; o <<= 1) {
                const int t = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += t;
            }
            part[lane] = x;
        }
        __syncthreads();
        const int excl = base + (w > 0 ? part[w - 1] : 0) + v - nb;
        for (int b = 0; b < nb; ++b) units[excl + b] = ((unsigned)r << 27) | ((unsigned)col << 5) | (unsigned)b;
        if (q < total && col == n_cols - 1) hdr[16 + r] = (unsigned)(excl + nb);  // units of ranks 0..r
        __syncthreads();
        if (threadIdx.x == 1023) base = excl + nb;
        __syncthreads();
    }
    if (threadIdx.x == 0) hdr[0] = (unsigned)base;
}

// step s of every instance that still steps: a wave of CTAs looping over a prefix of the units. At
// the start every CTA copies each instance's buffers, void z-limit and weights into shared memory,
// so a unit costs the same dependent loads as one of the compact kernel.
constexpr int kBatchMax = 32;
__global__ void __launch_bounds__(8 * PD_BY, 8) k_plume_direct_b(const PlumeInstDev* __restrict__ insts, int n,
                                                                 long long s, int nx, int ny, int nz, int mz, int xc,
                                                                 size_t zoff, const unsigned* __restrict__ hdr,
                                                                 int n_yt) {
    __shared__ float w0s[kBatchMax][64];
    __shared__ float sc[kBatchMax][6];  // wx, wy, wb, wt, decay, decays
    __shared__ const float* cin[kBatchMax];
    __shared__ float* cout[kBatchMax];
    __shared__ const uint8_t* msk[kBatchMax];
    __shared__ int zls[kBatchMax];
    __shared__ int nu_s;
    const int odd = (int)(s & 1);
    for (int q = threadIdx.x; q < n * 64; q += blockDim.x) w0s[q >> 6][q & 63] = insts[q >> 6].tab.w0eff[q & 63];
    if (threadIdx.x < n) {
        const PlumeInstDev& in = insts[threadIdx.x];
        float* t = sc[threadIdx.x];
        t[0] = in.tab.wx;
        t[1] = in.tab.wy;
        t[2] = in.tab.wb;
        t[3] = in.tab.wt;
        t[4] = in.tab.decay;
        t[5] = in.tab.decays ? 1.0f : 0.0f;
        cin[threadIdx.x] = odd ? in.Cb : in.Ca;
        cout[threadIdx.x] = odd ? in.Ca : in.Cb;
        msk[threadIdx.x] = in.mask;
        zls[threadIdx.x] = in.zlimit ? min(max(*in.zlimit, 0), nz) : nz;
    }
    if (threadIdx.x == 0) {
        int r = 0;
        while (r < n && insts[r].steps > s) ++r;
        nu_s = r > 0 ? (int)hdr[16 + r - 1] : 0;
    }
    __syncthreads();
    const int nu = nu_s;
    const unsigned* units = hdr + kBatchHdrWords;
    const int n_cols = n_yt * ((nx + xc - 1) / xc);
    for (int u = blockIdx.x; u < nu; u += gridDim.x) {
        const unsigned v = __ldg(&units[u]);
        const int ri = (int)(v >> 27);
        PlumeTab kt;
        kt.wx = sc[ri][0];
        kt.wy = sc[ri][1];
        kt.wb = sc[ri][2];
        kt.wt = sc[ri][3];
        kt.decay = sc[ri][4];
        kt.decays = sc[ri][5] != 0.0f;
        const int col = (int)((v >> 5) & 0x3FFFFFu);
        const int xch = col / n_yt;
        const uint8_t* M = msk[ri];
        plume_direct_unit(cin[ri], cout[ri], M, nx, ny, nz, mz, xc, kt, zls[ri], M + zoff, n_cols, col,
                          col - xch * n_yt, xch, (int)(v & 31u), w0s[ri]);
    }
}

size_t plume_batch_desc_bytes(int n) { return sizeof(PlumeInstDev) * (size_t)n; }

size_t plume_batch_units_words(int n, int nx, int ny, int nz) {
    const size_t cols = (size_t)nx * ((ny + PD_BY - 1) / PD_BY);
    const size_t bands = ((size_t)(nz + 3) / 4 + 7) / 8;
    return kBatchHdrWords + (size_t)n * cols * bands;
}

static int batch_steps(const PlumeInstHost& q, long long* total, PlumeTab* tab) {
    int steps;
    float dtp, decay;
    int rc = plume_policy_steps(q.params, &steps, &dtp, &decay);
    if (rc) return rc;
    const BdPlumeParams* p = q.params;
    PlumeConst c;
    c.dxy_x = p->D_xy / (p->dx * p->dx);
    c.dxy_y = p->D_xy / (p->dy * p->dy);
    c.dz_z = p->D_z / (p->dz * p->dz);
    c.vz_over_dz = p->vz > 0.0f ? p->vz / p->dz : 0.0f;
    c.dtp = dtp;
    c.decay = decay;
    if (tab) *tab = make_plume_tab(c);
    *total = (long long)steps * q.n_substeps;
    return BD_OK;
}

int plume_batch_prepare(int n, const PlumeInstHost* insts, void* dev, int* order, long long* max_steps) {
    BD_REQUIRE(n >= 1 && n <= kBatchMax, "plume batch: 1..%d instances, got %d", kBatchMax, n);
    std::vector<long long> total(n);
    std::vector<PlumeTab> tabs(n);
    for (int i = 0; i < n; ++i) {
        int rc = batch_steps(insts[i], &total[i], &tabs[i]);
        if (rc) return rc;
        order[i] = i;
    }
    std::stable_sort(order, order + n, [&](int a, int b) { return total[a] > total[b]; });
    std::vector<PlumeInstDev> h(n);
    for (int r = 0; r < n; ++r) {
        const PlumeInstHost& q = insts[order[r]];
        h[r].Ca = q.Ca;
        h[r].Cb = q.Cb;
        h[r].mask = q.mask;
        h[r].zlimit = q.zlimit;
        h[r].steps = total[order[r]];
        h[r].tab = tabs[order[r]];
    }
    *max_steps = total[order[0]];
    BD_CUDA(cudaMemcpy(dev, h.data(), sizeof(PlumeInstDev) * n, cudaMemcpyHostToDevice));
    return BD_OK;
}

int plume_batch_launch(int n, const PlumeInstHost* insts, const int* order, const void* dev, long long max_steps,
                       unsigned* units, cudaStream_t st) {
    const BdPlumeParams* p = insts[0].params;
    const int nx = p->nx, ny = p->ny, nz = p->nz;
    const int mz = plume_mask_pitch(nz);
    BD_REQUIRE((long long)nx * ny * mz < (1LL << 31), "plume batch: grid exceeds 2^31 mask bytes");
    const int xc = tune_value(BD_TUNE_PLUME_XC);
    const int n_yt = (ny + PD_BY - 1) / PD_BY, n_xch = (nx + xc - 1) / xc;
    const size_t zoff = plume_zlist_offset(nx, ny, nz);
    for (int i = 0; i < n; ++i) {
        const PlumeInstHost& q = insts[i];
        k_plume_mask<<<dim3((ny + PM_TY - 1) / PM_TY, nx), dim3(PM_TZ, PM_TY), 0, st>>>(nx, ny, nz, mz, q.flags, q.mask,
                                                                                       q.zlimit);
        k_plume_zlist<<<dim3(n_yt, n_xch), 256, 0, st>>>(q.mask, nx, ny, nz, mz, xc, q.zlimit, q.mask + zoff);
    }
    BD_CHECK_LAUNCH("k_plume_zlist");
    const PlumeInstDev* d = static_cast<const PlumeInstDev*>(dev);
    k_plume_batch_units<<<1, 1024, 0, st>>>(d, n, n_yt * n_xch, zoff, units);
    BD_CHECK_LAUNCH("k_plume_batch_units");
    static std::atomic<int> per_sm{0};  // resident CTAs per SM of the batched step kernel
    if (per_sm.load() == 0) {
        int v = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, k_plume_direct_b, 8 * PD_BY, 0);
        per_sm.store(std::max(1, v));
    }
    int dev_id = 0, nsm = 0;
    cudaGetDevice(&dev_id);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev_id);
    const int slots = std::max(1, nsm) * per_sm.load();
    for (long long s = 0; s < max_steps; ++s)
        k_plume_direct_b<<<slots, 8 * PD_BY, 0, st>>>(d, n, s, nx, ny, nz, mz, xc, zoff, units, n_yt);
    BD_CHECK_LAUNCH("k_plume_direct_b");
    // an instance whose step count is odd ends in its Cb buffer
    const long long nv = (long long)nx * ny * nz;
    for (int i = 0; i < n; ++i) {
        long long total = 0;
        int rc = batch_steps(insts[i], &total, nullptr);
        if (rc) return rc;
        if (total & 1)
            BD_CUDA(cudaMemcpyAsync(insts[i].Ca, insts[i].Cb, sizeof(float) * nv, cudaMemcpyDeviceToDevice, st));
    }
    (void)order;
    return BD_OK;
}
}  // namespace bd

using namespace bd;

extern "C" int bd_plume_advance(const BdPlumeParams* p, float* Ca, float* Cb, int n_substeps, const uint8_t* F,
                                int* in_b, void* stream) {
    BD_REQUIRE(p != nullptr, "bd_plume_advance: params is NULL");
    BD_REQUIRE(p->nx > 0 && p->ny > 0 && p->nz > 0, "bd_plume_advance: grid dims must be positive");
    BD_REQUIRE(Ca && Cb && F, "bd_plume_advance: NULL field");
    BD_REQUIRE(n_substeps >= 0, "bd_plume_advance: n_substeps must be >= 0");
    BD_REQUIRE((long long)p->nx * p->ny * p->nz < (1LL << 31), "bd_plume_advance: grid exceeds 2^31 voxels");
    if (n_substeps == 0) {
        if (in_b) *in_b = 0;
        return BD_OK;
    }
    cudaStream_t st = as_stream(stream);
    unsigned char* scratch = nullptr;  // an error flag, then the plume neighbourhood bytes and plans
    BD_CUDA(scratch_alloc((void**)&scratch, 256 + plume_mask_bytes(p->nx, p->ny, p->nz), st));
    int* err = reinterpret_cast<int*>(scratch);
    int host_err = 0;
    cudaError_t e = cudaMemsetAsync(err, 0, sizeof(int), st);
    int rc = BD_OK;
    if (e == cudaSuccess) rc = plume_launch(p, Ca, Cb, n_substeps, F, in_b, st, nullptr, 1, scratch + 256, err);
    if (e == cudaSuccess && rc == BD_OK) e = cudaMemcpyAsync(&host_err, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaError_t e2 = cudaFreeAsync(scratch, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (rc) return rc;
    if (e != cudaSuccess) return cuda_status(e, "bd_plume_advance");
    if (e2 != cudaSuccess) return cuda_status(e2, "bd_plume_advance: cudaFreeAsync");
    if (host_err) return fail(BD_ERR_TIMEOUT, "bd_plume_advance: a bounded device wait timed out");
    return BD_OK;
}

extern "C" int bd_plume_steps_per_substep(const BdPlumeParams* p, int* n_steps, float* dt_step) {
    BD_REQUIRE(p && n_steps && dt_step, "bd_plume_steps_per_substep: NULL argument");
    float decay;
    return plume_policy_steps(p, n_steps, dt_step, &decay);
}
