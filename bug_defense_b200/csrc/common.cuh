// Shared helpers for the libbugdef kernels: status/error plumbing, the counter-based
// RNG and small device utilities.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string>

#include "../../include/bugdef.h"

namespace bd {

// ---- error state (thread-local message of the last failure) ------------------------
void set_error(const char* fmt, ...);
int fail(int code, const char* fmt, ...);
int cuda_status(cudaError_t e, const char* what);
// Absorbed-weight tallies are 64-bit fixed point: weight * 2^36 per deposit, rounded to nearest.
// Integer sums are exact and independent of the order of the atomic additions (FP32 sums of
// millions of deposits lose the small ones once the voxel total dwarfs them). A photon deposits at
// most its weight (<= 1 plus rare roulette gains), so 2^26 photons per launch keep every voxel sum
// below 2^62.
constexpr float kTallyScale = 68719476736.0f;          // 2^36
constexpr long long kTallyMaxPhotons = 1LL << 26;
// Plume neighbourhood mask: one byte per voxel, z rows padded to a 16-byte pitch.
inline int plume_mask_pitch(int nz) { return (nz + 15) / 16 * 16; }
inline size_t plume_mask_only_bytes(int nx, int ny, int nz) {
    return ((size_t)nx * ny * plume_mask_pitch(nz) + 255) / 256 * 256;
}
// Then the live z groups of the columns (x chunk, 16-row y tile) of the one-step kernels: one count
// byte per column, then per column the ascending ids of its 4-voxel z groups that hold void
// (at most (nz + 3) / 4 <= 255 ids; sized for one x plane per chunk).
constexpr int kPlumeZRows = 16;
inline size_t plume_zlist_offset(int nx, int ny, int nz) { return plume_mask_only_bytes(nx, ny, nz); }
inline size_t plume_zlist_bytes(int nx, int ny, int nz) {
    const size_t cols = (size_t)nx * ((ny + kPlumeZRows - 1) / kPlumeZRows);
    return (cols * (1 + (size_t)(nz + 3) / 4) + 255) / 256 * 256;
}
// Then the compact kernel's state: 16 header words (unit count, chosen
// x planes per unit, unit count per candidate), the live-group bitmaps of every (x plane, y tile)
// (8 words each), then the units (16 bytes: column << 5 | band and the band's 8 group ids), at
// most one per band of every column.
inline size_t plume_units_offset(int nx, int ny, int nz) {
    return plume_zlist_offset(nx, ny, nz) + plume_zlist_bytes(nx, ny, nz);
}
inline size_t plume_unit_capacity(int nx, int ny, int nz) {
    const size_t cols = (size_t)nx * ((ny + kPlumeZRows - 1) / kPlumeZRows);
    return cols * (((size_t)(nz + 3) / 4 + 7) / 8);
}
inline size_t plume_units_bytes(int nx, int ny, int nz) {
    const size_t cols = (size_t)nx * ((ny + kPlumeZRows - 1) / kPlumeZRows);
    return ((16 + cols * 8) * sizeof(unsigned) + plume_unit_capacity(nx, ny, nz) * 16 + 255) / 256 * 256;
}
// Then the chained plume kernel's plan: a header, the first unit of every 16-row y tile, the
// live-group bitmaps of every (x plane, y tile with its halo rows) (8 words each), the units (at most
// one per started window of 30 z groups of a tile) and every unit's progress in up to kChainBlocks
// blocks of steps.
constexpr int kChainRows = 16;       // rows a unit writes
constexpr int kChainBlocks = 256;    // blocks of steps per launch
constexpr int kChainUnitBytes = 32;
inline size_t chain_round(size_t b) { return (b + 255) / 256 * 256; }
inline size_t plume_chain_offset(int nx, int ny, int nz) {
    return plume_units_offset(nx, ny, nz) + plume_units_bytes(nx, ny, nz);
}
inline size_t plume_chain_capacity(int ny, int nz) {
    return (size_t)((ny + kChainRows - 1) / kChainRows) * (((size_t)(nz + 3) / 4) / 30 + 1);
}
inline size_t plume_chain_bytes(int nx, int ny, int nz) {
    const size_t n_yt = (ny + kChainRows - 1) / kChainRows, cap = plume_chain_capacity(ny, nz);
    return 256 + chain_round((n_yt + 1) * 4) + chain_round((size_t)nx * n_yt * 32) +
           chain_round(cap * kChainUnitBytes) + chain_round(cap * kChainBlocks * 4);
}
inline size_t plume_mask_bytes(int nx, int ny, int nz) {
    return plume_chain_offset(nx, ny, nz) + plume_chain_bytes(nx, ny, nz);
}

// Stream-ordered scratch of the synchronous entry points (the plume's masks and plans, the convolutions' error
// flags), from one pool per context that keeps up to kScratchKeep bytes mapped between calls; what a call needs
// beyond that goes back to the driver at the next synchronisation. The default pool keeps nothing: every one of
// these calls ends in a synchronisation, so each call mapped and unmapped its few bytes again (a convolution of
// an 8x8x8 volume 450 us a call, 40 us so; one plume step of a 24x24x32 grid 525 and 60). Safe from any thread and
// stream: the pool orders reuse by stream.
constexpr unsigned long long kScratchKeep = 32ull << 20;
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t st);

// Launch-shape knobs (BD_TUNE_*) and the generation counter bumped by every change.
int tune_value(int knob);
int tune_generation();

#define BD_CUDA(call)                                                   \
    do {                                                                \
        cudaError_t _e = (call);                                        \
        if (_e != cudaSuccess) return ::bd::cuda_status(_e, #call);     \
    } while (0)

#define BD_CHECK_LAUNCH(what)                                           \
    do {                                                                \
        cudaError_t _e = cudaGetLastError();                            \
        if (_e != cudaSuccess) return ::bd::cuda_status(_e, what);      \
    } while (0)

#define BD_REQUIRE(cond, ...)                                           \
    do {                                                                \
        if (!(cond)) return ::bd::fail(BD_ERR_INVALID_ARG, __VA_ARGS__); \
    } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

inline int grid_for(int64_t n, int block, int cap = 148 * 32) {
    int64_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return (int)g;
}

// ---- Philox-4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy as
// 1, 2, 3", SC'11). Counter-based: the stream of photon p is a pure function of
// (seed, p, draw index), so no RNG state lives in memory. ----------------------------
struct Philox {
    static constexpr uint32_t M0 = 0xD2511F53u, M1 = 0xCD9E8D57u;
    static constexpr uint32_t W0 = 0x9E3779B9u, W1 = 0xBB67AE85u;
    __host__ __device__ static inline void round(uint32_t& x0, uint32_t& x1, uint32_t& x2,
                                                 uint32_t& x3, uint32_t k0, uint32_t k1) {
#ifdef __CUDA_ARCH__
        uint32_t hi0 = __umulhi(M0, x0), lo0 = M0 * x0;
        uint32_t hi1 = __umulhi(M1, x2), lo1 = M1 * x2;
#else
        uint64_t p0 = (uint64_t)M0 * x0, p1 = (uint64_t)M1 * x2;
        uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
        uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
#endif
        uint32_t y0 = hi1 ^ x1 ^ k0, y2 = hi0 ^ x3 ^ k1;
        x0 = y0; x1 = lo1; x2 = y2; x3 = lo0;
    }
    __host__ __device__ static inline uint4 gen(uint4 c, uint32_t k0, uint32_t k1) {
        uint32_t x0 = c.x, x1 = c.y, x2 = c.z, x3 = c.w;
#pragma unroll
        for (int r = 0; r < 10; ++r) {
            round(x0, x1, x2, x3, k0, k1);
            k0 += W0; k1 += W1;
        }
        return make_uint4(x0, x1, x2, x3);
    }
    // the same with the ten round keys at hand (kernel parameters: operands straight from the constant
    // bank, where adding them up costs two instructions a round and the two key registers)
    __host__ static inline void keys(uint32_t k0, uint32_t k1, uint32_t* ks) {
        for (int r = 0; r < 10; ++r) {
            ks[2 * r] = k0; ks[2 * r + 1] = k1;
            k0 += W0; k1 += W1;
        }
    }
    __device__ static inline uint4 gen(uint4 c, const uint32_t* ks) {
        uint32_t x0 = c.x, x1 = c.y, x2 = c.z, x3 = c.w;
#pragma unroll
        for (int r = 0; r < 10; ++r) round(x0, x1, x2, x3, ks[2 * r], ks[2 * r + 1]);
        return make_uint4(x0, x1, x2, x3);
    }
};

// Per-photon stream: counter = (photon lo, photon hi, draw block, 0x42444d43 'BDMC'); draw n is word
// n & 3 of block n >> 2. r0..r3 always hold the block of the next draw, so a draw never waits for a
// block, and the three draws of a scattering need one block at one place: lanes whose positions in
// their blocks differ would otherwise each run the ten rounds at another of the three draws.
// `ks`: the round keys of the run's seed (Philox::keys).
struct PhotonRng {
    uint32_t p_lo, p_hi;
    uint32_t n;               // draws so far
    uint32_t r0, r1, r2, r3;  // block n >> 2
    __device__ inline uint4 block(uint32_t b, const uint32_t* ks) const {
        return Philox::gen(make_uint4(p_lo, p_hi, b, 0x42444d43u), ks);
    }
    __device__ inline void hold(const uint4& v) { r0 = v.x; r1 = v.y; r2 = v.z; r3 = v.w; }
    __device__ inline void init(uint64_t photon, const uint32_t* ks) {
        p_lo = (uint32_t)photon; p_hi = (uint32_t)(photon >> 32);
        n = 0;
        hold(block(0, ks));
    }
    __device__ inline uint32_t next_u32(const uint32_t* ks) {
        const uint32_t lo = (n & 1u) ? r1 : r0, hi = (n & 1u) ? r3 : r2;
        const uint32_t out = (n & 2u) ? hi : lo;
        ++n;
        if ((n & 3u) == 0u) hold(block(n >> 2, ks));
        return out;
    }
    // the next three draws
    __device__ inline void next3(uint32_t& u0, uint32_t& u1, uint32_t& u2, const uint32_t* ks) {
        const bool odd = (n & 1u) != 0u, upper = (n & 2u) != 0u, turn = (n & 3u) != 0u;
        uint4 x = make_uint4(0u, 0u, 0u, 0u);
        if (turn) x = block((n >> 2) + 1u, ks);
        const uint32_t t0 = odd ? r1 : r0, t1 = odd ? r2 : r1, t2 = odd ? r3 : r2, t3 = odd ? x.x : r3,
                       t4 = odd ? x.y : x.x;
        u0 = upper ? t2 : t0;
        u1 = upper ? t3 : t1;
        u2 = upper ? t4 : t2;
        n += 3u;
        if (turn) hold(x);
    }
    // uniform in [0, 1): 24 significant bits
    __device__ static inline float to_uniform(uint32_t u) { return (float)(u >> 8) * (1.0f / 16777216.0f); }
    __device__ inline float uniform(const uint32_t* ks) { return to_uniform(next_u32(ks)); }
    // uniform in (0, 1): never 0, for logarithms
    __device__ inline float uniform_pos(const uint32_t* ks) {
        return ((float)(next_u32(ks) >> 8) + 0.5f) * (1.0f / 16777216.0f);
    }
};

__device__ __forceinline__ size_t vidx(int i, int j, int k, int ny, int nz) {
    return ((size_t)i * ny + j) * nz + k;
}

}  // namespace bd
