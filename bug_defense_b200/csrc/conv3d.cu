// 3-D convolutions of the absorbed-map denoiser on the fifth-generation tensor cores.
//
// Volumes are bf16 with a one-voxel zero pad, stored as "8-channel planes": channel c of padded row
// v lives at ((c/8)*R + v)*8 + c%8, with R = padded rows + a zero margin. The neighbour (dx, dy, dz)
// of row v is row v + dx*nyp*nzp + dy*nzp + dz for every interior voxel, so a 3x3x3 convolution is
// 27 row-shifted GEMMs [128 voxels x cin] x [cin x cout] accumulated in TMEM (implicit GEMM), and
// every operand tile is a run of contiguous 16-byte rows: one bulk copy per 8 channels.
//
// Forward / data-gradient kernel (k_conv): a CTA computes 16 output channels of units of up to 3 tiles of 128
// rows of the (y, z) plane, marching along x. A plane's rows arrive once, with their dy and dz halo, as cin/8
// bulk copies: K-major, no-swizzle UMMA operands, whose (dy, dz) shift is a shift of the start address by
// whole 16-byte rows. The plane x adds to the outputs of x-1, x and x+1 at once: the three are neighbours in
// TMEM and stacked along N, one 128 x 48 x 16 MMA per (dy, dz) and K step, and the weights lie in shared
// memory so that every rotation of the three slots is a run. Each z tap has accumulators of its own, summed
// over (dx, dy) in order, and the three are added at the end: (t0 + t-1) + t+1, but the third before the second
// in 3 of 126 rows, which is the order of the kernel before (its tiles of 126 outputs crossed warps there), so
// that stored weights give the same maps to the last bit: a bf16 rounding that flips at a coarse level moves
// the map by up to 0.2 % around it. A finished output plane's slot is read, cleared for the plane three on, and goes through the fused epilogue (bias, ReLU,
// nearest upsampling with the skip add, gradient gating, the 1x1 head), a group of 4 warps per tile. Three
// warps issue MMAs, one a tile: the tensor pipe queues only a few, and a warp that waits for its barrier
// leaves it idle for hundreds of clocks.
// Bounds: an MMA of this shape takes 43 clocks whatever N <= 48 (the A rows' read), 9 per 128 rows and 16
// channels. Reading nine shifted copies of every row instead, with N = 48 from the z taps and the z sums by
// shuffles, was bound by the copies (36 KB and 18 copies a tile) and then by the shuffles. 16 -> 16 channels
// at 200x200x128: 237 us before, 105 us now, of which 63 MMAs; 32 -> 16: 176 and 120; the whole network's
// forward pass 1.31 ms and 0.86 ms, of a 100x60x64 volume 0.24 and 0.22 ms.
//
// Weight-gradient kernel (k_conv_wgrad): dW[(dx, dy), dz][co][ci] = sum_u g[u - (dx, dy)][co] x[u + dz][ci].
// A chunk of up to 256 rows u takes a window of the gradient rows for each dx, dy being a row offset in it, and
// the activations at the three z shifts. The 8-channel blocks of the three windows lie one window apart and
// are stacked along M, the z shifts along N: an MMA per dy, each dy issued by a warp of its own; plane rows are
// the MN-major, no-swizzle operands as they lie (8 channels per core-matrix column). Each CTA reduces a
// contiguous range of rows in TMEM and adds its partial weights with FP32 atomics, four at a time.
// Bounds: 16 -> 16 channels move 74 KB a chunk of 256 rows from L2 (~7 TB/s in all); smaller levels wait for
// MMAs of N = 96 and the first loads. 27 shifted tiles in rows of 64, and the activations again for each MMA,
// took 3 times the bytes or more in copies of 1 KB. Calls, before and now: 16 -> 16 at 200x200x128 2.84 ms,
// 0.26 ms (0.36 with chunks of 128 rows); 32 -> 32 at 100x100x64 1.02, 0.09 (0.16 with single atomics);
// 64 -> 64 at 50x50x32 1.00, 0.07; a training step of a 200x200x128 volume 12.1 ms, 2.9 ms.
//
// Every mbarrier wait is bounded; a timeout sets the error flag, the roles drain what they issued
// and the CTA frees its TMEM and returns.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "common.cuh"
#include "conv3d.cuh"
#include "tma.cuh"
#include "umma.cuh"

namespace bd {

namespace {

constexpr int kTileM = 128;
constexpr int kSmemLimit = 232448;     // 227 KB opt-in dynamic shared memory per CTA
constexpr int kRowMargin = 256;        // zero rows after the padded volume (tile copies overrun it)
constexpr int kSlice = 16;             // output channels of a k_conv CTA
constexpr int kMaxTiles = 3;           // tiles of a unit: 3 z taps x 3 planes x 16 TMEM columns each
constexpr int kTileCols = 9 * kSlice;
constexpr int kMmaWarps = kMaxTiles;
constexpr int kEpiGroups = kMaxTiles;  // epilogue groups of 4 warps, one a tile
constexpr int kConvThreads = (1 + kMmaWarps + 4 * kEpiGroups) * 32;

struct Geom {
    int nxp, nyp, nzp;
    int v_lo, v_hi;       // interior rows lie in [v_lo, v_hi)
    int plane;            // nyp * nzp
    int R;                // rows per 8-channel plane (padded rows + margin)
};

__host__ __device__ inline Geom make_geom(int nx, int ny, int nz) {
    Geom g;
    g.nxp = nx + 2; g.nyp = ny + 2; g.nzp = nz + 2;
    g.plane = g.nyp * g.nzp;
    g.v_lo = g.plane + g.nzp + 1;
    g.v_hi = nx * g.plane + ny * g.nzp + nz + 1;
    g.R = g.nxp * g.plane + kRowMargin;
    return g;
}

__device__ __forceinline__ size_t prow(const Geom& g, int chunk, int v) { return ((size_t)chunk * g.R + v) * 8; }

// How k_conv cuts a level into units: `groups` in-plane groups of `tiles` x 128 rows, times segments of
// `steps` planes along x.
struct MarchPlan {
    int tiles, groups, steps, units;
    int segs;          // copies per plane and 8 channels: one window of rows, or the rows of dy = -1, 0, +1
    int dy_rows;       // rows between the dy = -1, 0, +1 operands of a slot
    int rows;          // rows of a slot
    int slots;         // planes in shared memory
};

struct ConvArgs {
    Geom g;        // level of the convolution
    Geom gf;       // finer level (UPADD modes)
    int taps, mode, n_off, n_slice;
    const __nv_bfloat16* input;
    const __nv_bfloat16* wimage;
    const float* bias;
    __nv_bfloat16* out;
    __nv_bfloat16* out_coarse;
    const __nv_bfloat16* aux;
    const __nv_bfloat16* aux2;
    const float* head;
    const float* a_noisy;
    const uint8_t* mask;
    float scale, loss_norm;
    float* pred;
    const float* target;
    float* head_grad;
    double* loss;
    __nv_bfloat16* grad_out;
    int* err;
    MarchPlan m;
};

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}

// N channels of row v, starting at 8-channel plane c0, from / to plane-layout storage.
template <int N>
__device__ __forceinline__ void store_row(__nv_bfloat16* base, const Geom& g, int c0, int v, const float* val) {
#pragma unroll
    for (int c = 0; c < N; c += 8) {
        uint4 q;
        q.x = pack_bf16x2(val[c + 0], val[c + 1]);
        q.y = pack_bf16x2(val[c + 2], val[c + 3]);
        q.z = pack_bf16x2(val[c + 4], val[c + 5]);
        q.w = pack_bf16x2(val[c + 6], val[c + 7]);
        *reinterpret_cast<uint4*>(base + prow(g, c0 + c / 8, v)) = q;
    }
}

__device__ __forceinline__ void unpack8(const uint4& q, float* val) {
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __bfloat1622float2(h[j]);
        val[2 * j] = f.x;
        val[2 * j + 1] = f.y;
    }
}

template <int N>
__device__ __forceinline__ void load_row(const __nv_bfloat16* base, const Geom& g, int c0, int v, float* val) {
#pragma unroll
    for (int c = 0; c < N; c += 8) unpack8(*reinterpret_cast<const uint4*>(base + prow(g, c0 + c / 8, v)), val + c);
}

struct SharedCtl {
    unsigned long long full[32], empty[32];
    unsigned long long acc_full[kEpiGroups], acc_empty[kMaxTiles], done;
    uint32_t tmem;
    volatile int abort;
};

__device__ __forceinline__ bool wait_or_abort(unsigned long long* bar, unsigned parity, SharedCtl* ctl, int* err) {
    if (mbar_wait(bar, parity)) return true;
    ctl->abort = 1;
    if (err) atomicExch(err, 1);
    return false;
}

// The same for a whole warp, which stays converged; false also once another role has given up.
__device__ __forceinline__ bool warp_wait(unsigned long long* bar, unsigned parity, SharedCtl* ctl, int* err) {
    bool ok = mbar_wait_limit(bar, parity, 1);
    if (!ok) ok = !ctl->abort && wait_or_abort(bar, parity, ctl, err);
    return __all_sync(0xffffffffu, ok);
}

// A producer warp whose lanes all issue copies, before it fills a stage of `bytes`: false (in every lane)
// when the kernel gives up.
__device__ __forceinline__ bool open_stage(unsigned long long* empty, unsigned parity, unsigned long long* full,
                                           uint32_t bytes, int lane, SharedCtl* ctl, int* err) {
    int ok = 0;
    if (lane == 0) {
        ok = !ctl->abort && wait_or_abort(empty, parity, ctl, err);
        if (ok) mbar_expect_tx(full, bytes);
    }
    return __shfl_sync(0xffffffffu, ok, 0) != 0;
}

constexpr int pow2_at_least(int x) { return x <= 32 ? 32 : x <= 64 ? 64 : x <= 128 ? 128 : x <= 256 ? 256 : 512; }

// Fused epilogue for voxel (x, y, z) of the padded level, row v; acc holds its N outputs from 8-channel plane
// c0 on.
template <int N, bool HEAD>
__device__ __forceinline__ void conv_epilogue(const ConvArgs& a, int c0, int x, int y, int z, int v, float* acc,
                                              float* head_acc, double& loss_acc) {
    const Geom& g = a.g;
    const int mode = HEAD ? BD_CONV_FWD_HEAD : a.mode;
    if (mode <= BD_CONV_FWD_HEAD) {
#pragma unroll
        for (int c = 0; c < N; ++c) acc[c] = fmaxf(acc[c], 0.f);
    }
    if constexpr (HEAD) {
        const int nz = g.nzp - 2, ny = g.nyp - 2;
        const size_t u = ((size_t)(x - 1) * ny + (y - 1)) * nz + (z - 1);
        float yv = a.head[N];
#pragma unroll
        for (int c = 0; c < N; ++c) yv = fmaf(a.head[c], acc[c], yv);
        const float m = a.mask[u] ? 1.f : 0.f;
        const float p = (a.a_noisy[u] * a.scale + yv) * m;
        a.pred[u] = p / a.scale;
        if (a.target) {
            const float res = (p - a.target[u] * a.scale) * m;
            loss_acc += (double)res * res;
            const float dy = 2.f * res * a.loss_norm;
            float gr[N];
#pragma unroll
            for (int c = 0; c < N; ++c) {
                gr[c] = acc[c] > 0.f ? dy * a.head[c] : 0.f;
                head_acc[c] = fmaf(dy, acc[c], head_acc[c]);
            }
            head_acc[N] += dy;
            store_row<N>(a.grad_out, g, 0, v, gr);
        }
        return;
    }
    if (mode == BD_CONV_FWD_RELU || mode == BD_CONV_BWD_RAW) {
        store_row<N>(a.out, g, c0, v, acc);
    } else if (mode == BD_CONV_BWD_MASK) {
#pragma unroll
        for (int c = 0; c < N; c += 8) {
            float m[8];
            load_row<8>(a.aux, g, c0 + c / 8, v, m);
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[c + j] = m[j] > 0.f ? acc[c + j] : 0.f;
        }
        store_row<N>(a.out, g, c0, v, acc);
    } else if (mode == BD_CONV_FWD_UPADD || mode == BD_CONV_BWD_UPADD) {
        if (mode == BD_CONV_FWD_UPADD && a.out_coarse) store_row<N>(a.out_coarse, g, c0, v, acc);
        const Geom& f = a.gf;
        // the eight fine voxels of 8 channels at a time, all loads before the first store
        const int vf0 = (2 * x - 1) * f.plane + (2 * y - 1) * f.nzp + 2 * z - 1;
#pragma unroll
        for (int c = 0; c < N; c += 8) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint4 s[4], m[4];
                int vf[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    vf[k] = vf0 + h * f.plane + (k >> 1) * f.nzp + (k & 1);
                    s[k] = *reinterpret_cast<const uint4*>(a.aux + prow(f, c0 + c / 8, vf[k]));
                    if (mode == BD_CONV_BWD_UPADD)
                        m[k] = *reinterpret_cast<const uint4*>(a.aux2 + prow(f, c0 + c / 8, vf[k]));
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float sv[8], mv[8], o[8];
                    unpack8(s[k], sv);
                    if (mode == BD_CONV_FWD_UPADD) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) o[j] = acc[c + j] + sv[j];
                    } else {
                        unpack8(m[k], mv);
#pragma unroll
                        for (int j = 0; j < 8; ++j) o[j] = mv[j] > 0.f ? sv[j] + 0.125f * acc[c + j] : 0.f;
                    }
                    store_row<8>(a.out, f, c0 + c / 8, vf[k], o);
                }
            }
        }
    }
}

// A warp's share of the head's weight gradient and of the loss.
template <int HA>
__device__ __forceinline__ void flush_head(const ConvArgs& a, const float* head_acc, double loss_acc, int lane) {
    if (!a.target) return;
#pragma unroll
    for (int c = 0; c < HA; ++c) {
        float h = head_acc[c];
        for (int o = 16; o; o >>= 1) h += __shfl_xor_sync(0xffffffffu, h, o);
        if (lane == 0) atomicAdd(&a.head_grad[c], h);
    }
    for (int o = 16; o; o >>= 1) loss_acc += __shfl_xor_sync(0xffffffffu, loss_acc, o);
    if (lane == 0) atomicAdd(a.loss, loss_acc);
}

template <int CIN>
struct ConvCfg {
    static constexpr int KP = CIN / 8;
    static constexpr int WBLK = kSlice * 16;       // 16 outputs x 8 input channels of one tap
    static constexpr int WK = 5 * WBLK;            // dx = +1, 0, -1, +1, 0: every rotation is a run of three
    static constexpr int WMAX = 9 * KP * WK;
    static constexpr int CTL = 1024;               // SharedCtl + bias
    static constexpr int AVAIL = kSmemLimit - 1024 - CTL - WMAX;   // for the planes
};

// Slice blockIdx.y of 16 outputs. See the file comment for the layout and march_plan for the units.
template <int CIN, bool HEAD>
__global__ void __launch_bounds__(kConvThreads, 1) k_conv(const ConvArgs a) {
    using C = ConvCfg<CIN>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base_addr = smem_addr(smem_raw);
    unsigned char* smem = smem_raw + ((1024 - (base_addr & 1023)) & 1023);
    SharedCtl* ctl = reinterpret_cast<SharedCtl*>(smem);
    float* sbias = reinterpret_cast<float*>(smem + C::CTL - kSlice * 4);   // bias (forward modes), else 0
    unsigned char* wsm = smem + C::CTL;
    unsigned char* planes = wsm + C::WMAX;
    static_assert(sizeof(SharedCtl) + kSlice * 4 <= C::CTL, "conv: control block over its space");
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kz = a.taps == 27 ? 3 : 1;
    const MarchPlan m = a.m;
    const int nx = a.g.nxp - 2, group_rows = m.tiles * kTileM;
    const int in_rows = (a.g.nyp - 2) * a.g.nzp - 2;   // in-plane rows from the first interior one to the last
    const uint32_t kp_bytes = m.rows * 16, slot_bytes = C::KP * kp_bytes;
    const int n0 = blockIdx.y * kSlice;
    const int issuers = m.tiles == 1 ? kz : m.tiles;           // MMA warps at work: one a z tap, or one a tile

    if (threadIdx.x == 0) {
        for (int s = 0; s < m.slots; ++s) {
            mbar_init(&ctl->full[s], 1);
            mbar_init(&ctl->empty[s], issuers);
        }
        for (int i = 0; i < kEpiGroups; ++i) mbar_init(&ctl->acc_full[i], m.tiles == 1 ? kz : 1);
        for (int i = 0; i < kMaxTiles; ++i) mbar_init(&ctl->acc_empty[i], 4);
        mbar_init(&ctl->done, issuers);
        ctl->abort = 0;
        mbar_init_fence();
    }
    if (threadIdx.x < kSlice)
        sbias[threadIdx.x] = (a.mode <= BD_CONV_FWD_HEAD && a.bias) ? a.bias[n0 + threadIdx.x] : 0.f;
    if (warp == 1) tmem_alloc(&ctl->tmem, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(ctl->tmem);
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;      // TMEM lanes of an epilogue warp
    if (warp != 0) {
        // While the producer fetches the first planes (a 40x48x52 map 144 us, 149 one after the other): clear
        // the accumulators, and bring the resident weights, wsm[dy][dz][k plane][5 dx][16 outputs][8], by plain
        // loads (as bulk copies, 256 bytes each at ~100 clocks to issue, they took 8 us a launch).
        if (warp >= 4 && warp < 8) {
            for (int c = 0; c < kMaxTiles * kTileCols; c += 16) tmem_zero16(tmem + lanes + c);
        }
#pragma unroll 4
        for (int i = threadIdx.x - 32; i < 3 * kz * C::KP * 5 * kSlice; i += kConvThreads - 32) {
            const int n = i % kSlice, blk = i / kSlice % 5, r = i / kSlice / 5, kp = r % C::KP, t = r / C::KP;
            const int dz = t % kz, dy = t / kz, dx = 2 - blk % 3;       // 2, 1, 0 = +1, 0, -1
            reinterpret_cast<uint4*>(wsm)[i] = __ldg(reinterpret_cast<const uint4*>(
                a.wimage + ((((dx * 3 + dy) * C::KP + kp) * kz + dz) * a.n_slice + n0 + n) * 8));
        }
        if (warp >= 4 && warp < 8) tmem_st_wait();
        fence_proxy_async_smem();
        tc_fence_before();
        asm volatile("bar.sync 1, %0;" ::"n"(kConvThreads - 32) : "memory");
        tc_fence_after();
    }

    if (warp == 0) {
        // ---- producer: the units' planes x0-1 .. x1+1 one after another ----
        if (lane == 0) {
            int s = 0;
            unsigned ph = 0;
            long long issued = 0;
            bool ok = true;
            const int seg_rows = m.segs == 1 ? m.rows : m.dy_rows;
            for (int unit = blockIdx.x; ok && unit < m.units; unit += gridDim.x) {
                const int x0 = 1 + unit / m.groups * m.steps, x1 = min(nx, x0 + m.steps - 1);
                const int p = unit % m.groups * group_rows;    // (dy, dz) = (-1, -1) row of the first output
                for (int x = x0 - 1; x <= x1 + 1; ++x) {
                    ok = !ctl->abort && wait_or_abort(&ctl->empty[s], ph ^ 1, ctl, a.err);
                    if (!ok) break;
                    const int row0 = x * a.g.plane + p;
                    // a group that overruns the last plane stops at the volume's end
                    uint32_t bytes = 0;
                    for (int i = 0; i < m.segs; ++i) bytes += min(seg_rows, a.g.R - (row0 + i * a.g.nzp)) * 16;
                    mbar_expect_tx(&ctl->full[s], C::KP * bytes);
                    for (int i = 0; i < m.segs; ++i) {
                        const int row = row0 + i * a.g.nzp;
                        const uint32_t n = min(seg_rows, a.g.R - row) * 16;
#pragma unroll
                        for (int k = 0; k < C::KP; ++k)
                            bulk_load(planes + s * slot_bytes + k * kp_bytes + i * m.dy_rows * 16,
                                      a.input + prow(a.g, k, row), n, &ctl->full[s]);
                    }
                    ++issued;
                    if (++s == m.slots) { s = 0; ph ^= 1; }
                }
            }
            // drain: every issued load has landed before the CTA leaves
            const long long n_drain = issued < m.slots ? issued : m.slots;
            for (long long i = 0; i < n_drain; ++i) {
                if (--s < 0) { s = m.slots - 1; ph ^= 1; }
                mbar_wait(&ctl->full[s], ph);
            }
        }
        __syncwarp();
    } else if (warp <= kMmaWarps) {
        // ---- MMA issuers: per plane and tile 3 * kz * CIN/16 MMAs of 128 x 48 x 16. Every tile's (or z tap's)
        // MMAs come from one warp, in order ----
        const int me = uniform(warp - 1);
        const int my_t = m.tiles == 1 ? 0 : me, dz0 = m.tiles == 1 ? me : 0, dz1 = m.tiles == 1 ? me + 1 : kz;
        const uint32_t lead = elect_one();
        constexpr uint32_t idesc48 = umma_idesc_bf16(kTileM, 3 * kSlice, false, false);
        constexpr uint32_t idesc16 = umma_idesc_bf16(kTileM, kSlice, false, false);
        const uint32_t wbase = smem_addr(wsm), pbase = smem_addr(planes);
        bool ok = me < issuers;
        int s = 0, turn = my_t, oldest = 0;
        unsigned ph = 0, eph = 0;
        bool drained = false;
        for (int unit = blockIdx.x; ok && unit < m.units; unit += gridDim.x) {
            const int x0 = 1 + unit / m.groups * m.steps;
            const int planes_n = uniform(min(nx + 1 - x0, m.steps) + 2);
            const int left = in_rows - unit % m.groups * group_rows;
            const int tiles = uniform(min(m.tiles, (left + kTileM - 1) / kTileM));
            for (int i = 0; i < planes_n; ++i) {                    // plane x = x0 - 1 + i
                ok = warp_wait(&ctl->full[s], ph, ctl, a.err);
                if (!ok) break;
                if (my_t < tiles) {
                    if (drained) {       // slot x+1 is the one that the plane before this completed
                        ok = warp_wait(&ctl->acc_empty[my_t], eph, ctl, a.err);
                        if (!ok) break;
                        eph ^= 1;
                    }
                    tc_fence_after();
                    // outputs x-1, x, x+1 live in slots oldest, oldest+1, oldest+2 (mod 3); a unit's first two
                    // and last two planes add to its own outputs only
                    const uint32_t wrot = wbase + (oldest ? 3 - oldest : 0) * C::WBLK;
                    const uint32_t op = pbase + s * slot_bytes + my_t * kTileM * 16 + (kz == 3 ? 0 : 16);
                    const uint32_t d = tmem + my_t * kTileCols;
                    const uint32_t mine = (i >= 2) | (i >= 1 && i < planes_n - 1) << 1 | (i < planes_n - 2) << 2;
                    const int pieces = mine == 7 ? 1 : 3;
                    for (int k = 0; k < pieces; ++k) {
                        if (!(mine >> k & 1)) continue;
                        const int at = mine == 7 ? 0 : oldest + k - (oldest + k >= 3 ? 3 : 0);   // slot of x - 1 + k
                        const uint32_t idesc = mine == 7 ? idesc48 : idesc16;
                        for (int dz = dz0; dz < dz1; ++dz) {
#pragma unroll
                            for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                                for (int kk = 0; kk < CIN / 16; ++kk) {
                                    const uint64_t ad = umma_desc(op + (dy * m.dy_rows + dz) * 16 + kk * 2 * kp_bytes,
                                                                  kp_bytes, 128, UMMA_NONE);
                                    const uint64_t bd = umma_desc(
                                        wrot + ((dy * kz + dz) * C::KP + kk * 2) * C::WK + at * C::WBLK, C::WK, 128, UMMA_NONE);
                                    umma_bf16(d + (dz * 3 + at) * kSlice, ad, bd, idesc, true, lead);
                                }
                        }
                    }
                    drained = i >= 2;
                    if (drained) {
                        umma_commit(&ctl->acc_full[turn], lead);
                        if (m.tiles == 1 && ++turn == kEpiGroups) turn = 0;
                    }
                }
                umma_commit(&ctl->empty[s], lead);
                if (++s == m.slots) { s = 0; ph ^= 1; }
                if (++oldest == 3) oldest = 0;
            }
        }
        if (me < issuers) {
            umma_commit(&ctl->done, lead);
            mbar_wait(&ctl->done, 0);
        }
        __syncwarp();
    } else {
        // ---- epilogue: a group of 4 warps for each tile; one tile a unit goes round the groups. Warp w
        // reads TMEM lanes 32*(w % 4) .. +31; row = TMEM lane. ----
        const int grp = (warp - 1 - kMmaWarps) >> 2;
        const int t = m.tiles == 1 ? 0 : grp;
        const int row = (warp & 3) * 32 + lane;
        const int c0 = (a.n_off + n0) / 8;
        unsigned ph = 0;
        float head_acc[HEAD ? kSlice + 1 : 1];
        double loss_acc = 0.0;
        if constexpr (HEAD) {
#pragma unroll
            for (int c = 0; c <= kSlice; ++c) head_acc[c] = 0.f;
        }
        int turn = 0, oldest = 0;
        bool ok = true;
        for (int unit = blockIdx.x; ok && unit < m.units; unit += gridDim.x) {
            const int x0 = 1 + unit / m.groups * m.steps, x1 = min(nx, x0 + m.steps - 1);
            const int p = unit % m.groups * group_rows;
            const bool used = t < m.tiles && t * kTileM < in_rows - p;
            const int r = a.g.nzp + 1 + p + t * kTileM + row, y = r / a.g.nzp, z = r - y * a.g.nzp;
            const bool inside = y <= a.g.nyp - 2 && z >= 1 && z <= a.g.nzp - 2;
            if (++oldest == 3) oldest = 0;                       // the planes x0 - 1 and x0 complete none
            if (++oldest == 3) oldest = 0;
            for (int x = x0; x <= x1; ++x) {                     // plane x + 1 completes output plane x
                const bool mine = m.tiles == 1 ? turn == grp : used;
                if (++turn == kEpiGroups) turn = 0;
                if (mine) {
                    const int vr = x * a.g.plane + r;
                    // the order of the two additions below is a function of the voxel's row
                    const bool late = ((vr - a.g.v_lo) % 126 & 31) == 31;
                    ok = warp_wait(&ctl->acc_full[grp], ph, ctl, a.err);
                    if (!ok) break;
                    ph ^= 1;
                    tc_fence_after();
                    const uint32_t tb = tmem + lanes + t * kTileCols + oldest * kSlice;
                    float v[kSlice], up[kSlice], dn[kSlice];
                    if (kz == 3) {
                        tmem_ld16(tb, up);
                        tmem_ld16(tb + 3 * kSlice, v);
                        tmem_ld16(tb + 6 * kSlice, dn);
                    } else {
                        tmem_ld16(tb, v);
                    }
                    tmem_ld_wait();
                    tmem_zero16(tb);                             // output plane x + 3 adds up here from zero
                    if (kz == 3) {
                        tmem_zero16(tb + 3 * kSlice);
                        tmem_zero16(tb + 6 * kSlice);
                    }
                    tmem_st_wait();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&ctl->acc_empty[t]);
                    if (inside) {
                        if (kz == 3) {
#pragma unroll
                            for (int c = 0; c < kSlice; ++c)
                                v[c] = (v[c] + (late ? dn[c] : up[c])) + (late ? up[c] : dn[c]);
                        }
#pragma unroll
                        for (int c = 0; c < kSlice; ++c) v[c] += sbias[c];
                        conv_epilogue<kSlice, HEAD>(a, c0, x, y, z, vr, v, head_acc, loss_acc);
                    }
                }
                if (++oldest == 3) oldest = 0;
            }
        }
        if constexpr (HEAD) flush_head<kSlice + 1>(a, head_acc, loss_acc, lane);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

struct WgradArgs {
    Geom g;
    int taps, u_lo, chunks_total, chunks_per_cta, cin;
    int kv;            // rows of a chunk
    int segs;          // gradient copies per plane and 8 channels: one window, or the rows of dy = -1, 0, +1
    int dy_rows, rows; // rows between the dy operands; rows of a gradient window
    int stages;
    const __nv_bfloat16* grad;
    const __nv_bfloat16* act;
    float* dw;
    int* err;
};

template <int COUT, int CIS>
struct WgradCfg {
    static constexpr int CB = COUT / 8;
    static constexpr int NB = 3 * CB;                       // 8-channel blocks of the gradient's three planes
    static constexpr int MB = kTileM / 8;                   // blocks of an MMA
    static constexpr int NH = NB > MB ? 2 : 1;              // MMAs over the blocks; a second one overlaps
    static constexpr int CTL = 1024;
    static constexpr int TMEM_COLS = pow2_at_least(3 * NH * 3 * CIS);
    static constexpr int THREADS = 256;
    static_assert(3 * NH * 3 * CIS <= 512 && 3 * CIS <= 256, "wgrad: accumulators fit TMEM, N fits an MMA");
    static_assert(NB <= NH * MB, "wgrad: the MMAs cover the blocks");
    __host__ __device__ static int stage_bytes(int kv, int rows) { return (NB * rows + 3 * (CIS / 8) * kv) * 16; }
    // an MMA reads MB blocks from the stage's start, whatever their number: the rows past NB are not used,
    // but lie in the buffer
    __host__ __device__ static int smem_bytes(int kv, int rows, int stages) {
        const int st = stage_bytes(kv, rows), mma = MB * rows * 16;
        return 1024 + CTL + (stages - 1) * st + (st > mma ? st : mma);
    }
};

// Slice blockIdx.y of CIS input channels. See the file comment for the layout.
template <int COUT, int CIS>
__global__ void __launch_bounds__(256, 1) k_conv_wgrad(const WgradArgs a) {
    using C = WgradCfg<COUT, CIS>;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base_addr = smem_addr(smem_raw);
    unsigned char* smem = smem_raw + ((1024 - (base_addr & 1023)) & 1023);
    SharedCtl* ctl = reinterpret_cast<SharedCtl*>(smem);
    unsigned char* stages = smem + C::CTL;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int kz = a.taps == 27 ? 3 : 1;
    const int NN = kz * CIS;                         // MMA N: z taps stacked along N
    const int ci0 = blockIdx.y * CIS;
    const uint32_t blk = a.rows * 16, chunk = a.kv * 16;
    const uint32_t stage = C::stage_bytes(a.kv, a.rows);

    const int c_begin = blockIdx.x * a.chunks_per_cta;
    const int c_end = min(a.chunks_total, c_begin + a.chunks_per_cta);

    if (threadIdx.x == 0) {
        for (int s = 0; s < a.stages; ++s) {
            mbar_init(&ctl->full[s], 1);
            mbar_init(&ctl->empty[s], 3);
        }
        mbar_init(&ctl->done, 3);
        ctl->abort = 0;
        mbar_init_fence();
    }
    if (warp == 1) tmem_alloc(&ctl->tmem, C::TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = uniform(ctl->tmem);

    if (warp == 0) {
        const int seg_rows = a.segs == 1 ? a.rows : a.kv;
        const uint32_t bytes = C::NB * blk + kz * (CIS / 8) * chunk;
        const int NA = C::NB * a.segs;                   // gradient copies of a stage, then the activations'
        const int n_copies = NA + kz * (CIS / 8);
        int s = 0;
        unsigned ph = 0;
        long long issued = 0;
        for (int c = c_begin; c < c_end; ++c) {
            const int u0 = a.u_lo + c * a.kv;
            if (!open_stage(&ctl->empty[s], ph ^ 1, &ctl->full[s], bytes, lane, ctl, a.err)) break;
            unsigned char* st = stages + s * stage;
            for (int i = lane; i < n_copies; i += 32) {
                if (i < NA) {
                    const int b = i / a.segs, j = i % a.segs;
                    bulk_load(st + b * blk + j * chunk,
                              a.grad + prow(a.g, b % C::CB, u0 - (b / C::CB - 1) * a.g.plane + (j - 1) * a.g.nzp),
                              seg_rows * 16, &ctl->full[s]);
                } else {
                    const int dz = (i - NA) / (CIS / 8), cb = (i - NA) % (CIS / 8);
                    bulk_load(st + C::NB * blk + (i - NA) * chunk, a.act + prow(a.g, ci0 / 8 + cb, u0 + dz - kz / 2),
                              chunk, &ctl->full[s]);
                }
            }
            ++issued;
            if (++s == a.stages) { s = 0; ph ^= 1; }
        }
        __syncwarp();
        if (lane == 0) {
            const long long n_drain = issued < a.stages ? issued : a.stages;
            for (long long i = 0; i < n_drain; ++i) {
                if (--s < 0) { s = a.stages - 1; ph ^= 1; }
                mbar_wait(&ctl->full[s], ph);
            }
        }
        __syncwarp();
    } else if (warp <= 3) {
        // ---- MMA issuers, one for each dy. MN-major, no swizzle: 8 M (or N) elements x 8 K rows per
        // 128-byte core matrix; K groups 128 B apart (LBO), M blocks a window apart and N blocks a chunk (SBO)
        const int j = uniform(warp - 1);
        const uint32_t lead = elect_one();
        const uint32_t idesc = umma_idesc_bf16(kTileM, NN, true, true);
        const uint32_t sbase = smem_addr(stages);
        const uint32_t d = tmem + j * C::NH * NN;
        int s = 0;
        unsigned ph = 0;
        for (int c = c_begin; c < c_end; ++c) {
            if (!warp_wait(&ctl->full[s], ph, ctl, a.err)) break;
            tc_fence_after();
            const uint32_t ga = sbase + s * stage + j * a.dy_rows * 16, xa = sbase + s * stage + C::NB * blk;
            for (int kk = 0; kk < a.kv / 16; ++kk) {
                const uint64_t bd = umma_desc(xa + kk * 256, 128, chunk, UMMA_NONE);
#pragma unroll
                for (int h = 0; h < C::NH; ++h) {
                    const uint64_t ad = umma_desc(ga + h * (C::NB - C::MB) * blk + kk * 256, 128, blk, UMMA_NONE);
                    umma_bf16(d + h * NN, ad, bd, idesc, (c != c_begin) || kk != 0, lead);
                }
            }
            umma_commit(&ctl->empty[s], lead);
            if (++s == a.stages) { s = 0; ph ^= 1; }
        }
        umma_commit(&ctl->done, lead);
        mbar_wait(&ctl->done, 0);
        __syncwarp();
    } else if (c_begin < c_end) {
        const int quad = warp & 3;
        const int row = quad * 32 + lane;
        if (warp_wait(&ctl->done, 0, ctl, a.err) && !ctl->abort) {
            tc_fence_after();
            const bool vec = reinterpret_cast<uintptr_t>(a.dw) % 16 == 0;   // a fourth of the memory operations
            for (int j = 0; j < 3; ++j)
                for (int h = 0; h < C::NH; ++h) {
                    const int b = row / 8 + h * (C::NB - C::MB);
                    const bool mine = b < C::NB && b >= h * C::MB;   // not already the MMA before's
                    const int q = b / C::CB * 3 + 2 - j, co = b % C::CB * 8 + row % 8;
                    for (int dz = 0; dz < kz; ++dz) {
                        float v[CIS];
#pragma unroll
                        for (int c = 0; c < CIS; c += 16)
                            tmem_ld16(tmem + ((uint32_t)(quad * 32) << 16) + (j * C::NH + h) * NN + dz * CIS + c, v + c);
                        tmem_ld_wait();
                        if (mine) {
                            float* dst = a.dw + ((size_t)(q * kz + dz) * COUT + co) * a.cin + ci0;
                            if (vec) {
#pragma unroll
                                for (int c = 0; c < CIS; c += 4)
                                    atomicAdd(reinterpret_cast<float4*>(dst + c), make_float4(v[c], v[c + 1], v[c + 2], v[c + 3]));
                            } else {
#pragma unroll
                                for (int c = 0; c < CIS; ++c) atomicAdd(dst + c, v[c]);
                            }
                        }
                    }
                }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem, C::TMEM_COLS);
    }
}

__global__ void k_pack_weights(int taps, int cin, int cout, int n_off, int n_slice, int transpose, const float* w,
                               __nv_bfloat16* img) {
    // image[q][kp][dz][n][8]: for each (dx, dy) pair q, K-major planes of 8 input channels whose
    // rows are the (z tap, output) pairs the stacked MMA computes (kz = 3 z taps, or 1)
    const int K = transpose ? cout : cin;
    const int kz = taps == 27 ? 3 : 1;
    const long long total = (long long)taps * K * n_slice;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
        const int j = (int)(i & 7);
        long long r = i >> 3;
        const int n = (int)(r % n_slice);
        r /= n_slice;
        const int dz = (int)(r % kz);
        r /= kz;
        const int kp = (int)(r % (K / 8));
        const int q = (int)(r / (K / 8));
        const int t = q * kz + dz;
        const int k = kp * 8 + j;
        float val;
        if (!transpose) val = w[((size_t)t * cout + (n_off + n)) * cin + k];
        else val = w[((size_t)(taps - 1 - t) * cout + k) * cin + (n_off + n)];
        img[i] = __float2bfloat16_rn(val);
    }
}

// Units of k_conv, by the clocks of a CTA: a tile's MMAs at ~75 clocks each with their waits, or its epilogue
// (~650), and a plane's load at ~24 bytes a clock (43 to 75 clocks an MMA give the same times to 3 %). A unit
// reads two planes more than it writes, and a short group its dy halo too often; the units should fill the
// CTAs evenly.
MarchPlan march_plan(const Geom& g, int cin, int taps, int avail, int ctas) {
    const int nx = g.nxp - 2, in_rows = (g.nyp - 2) * g.nzp - 2;
    const double tile_clk = std::max(650.0, 75.0 * (taps / 3) * (cin / 16));
    MarchPlan best{};
    double best_cost = 0;
    for (int tiles = 1; tiles <= kMaxTiles; ++tiles) {
        MarchPlan m{};
        m.tiles = tiles;
        const int run = tiles * kTileM + 2;
        m.segs = g.nzp <= run ? 1 : 3;
        m.dy_rows = std::min(g.nzp, run);
        m.rows = run + 2 * m.dy_rows;
        m.slots = std::min(4, avail / (m.rows * cin * 2));
        if (m.slots < 2) break;
        m.groups = (in_rows + tiles * kTileM - 1) / (tiles * kTileM);
        for (int cut = 1; cut <= nx && (cut == 1 || m.groups * cut <= 8 * ctas); ++cut) {
            m.steps = (nx + cut - 1) / cut;
            m.units = m.groups * ((nx + m.steps - 1) / m.steps);
            const int waves = (m.units + ctas - 1) / ctas;
            // one tile at a time: the next plane's MMAs wait for its epilogue's reads
            const double cost = waves * (m.steps + 2.0) *
                                std::max(tiles * tile_clk + (tiles == 1 ? 500.0 : 0.0), m.rows * cin / 12.0);
            if (best_cost == 0 || cost < best_cost) {
                best_cost = cost;
                best = m;
            }
        }
        if (m.groups == 1) break;
    }
    return best;
}

template <int CIN, bool HEAD>
int launch_conv_t(const BdConvCall& c, cudaStream_t st, int* err, int sms) {
    using C = ConvCfg<CIN>;
    // one tile a unit and two planes always fit
    static_assert(2 * 3 * (kTileM + 2) * CIN * 2 <= C::AVAIL, "conv: not enough shared memory for two planes");
    ConvArgs a{};
    a.g = make_geom(c.nx, c.ny, c.nz);
    a.gf = make_geom(2 * c.nx, 2 * c.ny, 2 * c.nz);
    a.taps = c.taps; a.mode = c.mode; a.n_off = c.n_off; a.n_slice = c.n_slice;
    a.input = static_cast<const __nv_bfloat16*>(c.input);
    a.wimage = static_cast<const __nv_bfloat16*>(c.wimage);
    a.bias = c.bias;
    a.out = static_cast<__nv_bfloat16*>(c.out);
    a.out_coarse = static_cast<__nv_bfloat16*>(c.out_coarse);
    a.aux = static_cast<const __nv_bfloat16*>(c.aux);
    a.aux2 = static_cast<const __nv_bfloat16*>(c.aux2);
    a.head = c.head; a.a_noisy = c.a_noisy; a.mask = c.mask; a.scale = c.scale; a.loss_norm = c.loss_norm;
    a.pred = c.pred; a.target = c.target; a.head_grad = c.head_grad; a.loss = c.loss;
    a.grad_out = static_cast<__nv_bfloat16*>(c.grad_out);
    a.err = err;
    const int slices = c.n_slice / kSlice, ctas = std::max(1, sms / slices);
    a.m = march_plan(a.g, CIN, c.taps, C::AVAIL, ctas);
    const int smem = 1024 + C::CTL + C::WMAX + a.m.slots * a.m.rows * CIN * 2;
    BD_CUDA(cudaFuncSetAttribute(k_conv<CIN, HEAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    k_conv<CIN, HEAD><<<dim3(std::min(a.m.units, ctas), slices), kConvThreads, smem, st>>>(a);
    BD_CHECK_LAUNCH("k_conv");
    return BD_OK;
}

template <int COUT, int CIS>
int launch_wgrad_t(int nx, int ny, int nz, int cin, int taps, const void* grad, const void* act, float* dw,
                   cudaStream_t st, int* err, int sms) {
    using C = WgradCfg<COUT, CIS>;
    BD_CUDA(cudaFuncSetAttribute(k_conv_wgrad<COUT, CIS>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit));
    WgradArgs a{};
    a.g = make_geom(nx, ny, nz);
    a.taps = taps;
    a.cin = cin;
    // the longest chunks of which two stages fit: a window carries 2 nzp rows of halo
    for (a.kv = 256;; a.kv -= 64) {
        a.segs = a.g.nzp <= a.kv ? 1 : 3;
        a.dy_rows = std::min(a.g.nzp, a.kv);
        a.rows = a.kv + 2 * a.dy_rows;
        if (a.kv == 64 || C::smem_bytes(a.kv, a.rows, 2) <= kSmemLimit) break;
    }
    static_assert(2 * (C::NB * 3 + 3 * (CIS / 8)) * 64 * 16 <= kSmemLimit - 2048, "wgrad: two stages of 64 rows fit");
    for (a.stages = 2; a.stages < 6 && C::smem_bytes(a.kv, a.rows, a.stages + 1) <= kSmemLimit;) ++a.stages;
    // rows u of the sums g[u - (dx, dy)] x[u + dz]: one more on either side than the interior has
    a.u_lo = a.g.v_lo - 1;
    a.chunks_total = (a.g.v_hi + 1 - a.u_lo + a.kv - 1) / a.kv;
    a.grad = static_cast<const __nv_bfloat16*>(grad);
    a.act = static_cast<const __nv_bfloat16*>(act);
    a.dw = dw;
    a.err = err;
    // split the rows over the SMs; small levels keep at least 2048 rows per CTA (a CTA ends by adding
    // its 27 x cout x CIS partial weights to memory)
    const int slices = cin / CIS;
    const int ctas = std::max(1, std::min(std::max(1, sms / slices), (a.chunks_total * a.kv + 2048 - 1) / 2048));
    a.chunks_per_cta = (a.chunks_total + ctas - 1) / ctas;
    const int grid = (a.chunks_total + a.chunks_per_cta - 1) / a.chunks_per_cta;
    k_conv_wgrad<COUT, CIS><<<dim3(grid, slices), C::THREADS, C::smem_bytes(a.kv, a.rows, a.stages), st>>>(a);
    BD_CHECK_LAUNCH("k_conv_wgrad");
    return BD_OK;
}

int sm_count() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 148;
    }
    return n;
}

}  // namespace

int conv_check(const BdConvCall& c) {
    BD_REQUIRE(c.nx > 0 && c.ny > 0 && c.nz > 0, "bd_conv3d: dims must be positive");
    BD_REQUIRE(c.cin == 16 || c.cin == 32 || c.cin == 64, "bd_conv3d: cin must be 16, 32 or 64");
    BD_REQUIRE(c.n_slice == 16 || c.n_slice == 32 || c.n_slice == 64, "bd_conv3d: n_slice must be 16, 32 or 64");
    BD_REQUIRE(!(c.cin == 64 && c.n_slice == 64), "bd_conv3d: cin 64 x n_slice 64 is not supported; split the slice");
    BD_REQUIRE(c.n_off >= 0 && c.n_off + c.n_slice <= c.cout_total && c.n_off % 8 == 0, "bd_conv3d: bad output slice");
    BD_REQUIRE(c.taps == 27 || c.taps == 9, "bd_conv3d: taps must be 27 or 9");
    BD_REQUIRE(c.mode >= BD_CONV_FWD_RELU && c.mode <= BD_CONV_BWD_UPADD, "bd_conv3d: unknown mode");
    BD_REQUIRE(c.input && c.wimage && (c.out || c.mode == BD_CONV_FWD_HEAD),
               "bd_conv3d: in, wimage and out are required");
    const long long vp = (long long)(c.nx + 2) * (c.ny + 2) * (c.nz + 2);
    const long long vpf = (long long)(2 * c.nx + 2) * (2 * c.ny + 2) * (2 * c.nz + 2);
    BD_REQUIRE(vp * c.cout_total < (1LL << 31) && vpf < (1LL << 31), "bd_conv3d: volume too large for 32-bit rows");
    if (c.mode == BD_CONV_FWD_UPADD || c.mode == BD_CONV_BWD_UPADD)
        BD_REQUIRE(c.aux != nullptr && (c.mode == BD_CONV_FWD_UPADD || c.aux2 != nullptr),
                   "bd_conv3d: the upsampling modes need aux (and aux2)");
    if (c.mode == BD_CONV_BWD_MASK) BD_REQUIRE(c.aux != nullptr, "bd_conv3d: BWD_MASK needs aux");
    BD_REQUIRE(((uintptr_t)c.input | (uintptr_t)c.wimage | (uintptr_t)c.out | (uintptr_t)c.aux | (uintptr_t)c.aux2 |
                (uintptr_t)c.out_coarse | (uintptr_t)c.grad_out) % 16 == 0,
               "bd_conv3d: volumes and weight images must be 16-byte aligned");
    if (c.mode == BD_CONV_FWD_HEAD) {
        BD_REQUIRE(c.n_slice == 16 && c.cout_total == 16 && c.n_off == 0, "bd_conv3d: the head takes 16 channels");
        BD_REQUIRE(c.head && c.a_noisy && c.mask && c.pred && c.scale > 0.f, "bd_conv3d: head inputs missing");
        BD_REQUIRE(!c.target || (c.head_grad && c.loss && c.grad_out), "bd_conv3d: training head needs gradients");
    }
    return BD_OK;
}

int conv_launch(const BdConvCall& c, cudaStream_t st, int* err) {
    const int sms = sm_count();
    const bool head = c.mode == BD_CONV_FWD_HEAD;
#define BD_CONV_CASE(CI) \
    if (c.cin == CI) return head ? launch_conv_t<CI, true>(c, st, err, sms) : launch_conv_t<CI, false>(c, st, err, sms);
    BD_CONV_CASE(16) BD_CONV_CASE(32) BD_CONV_CASE(64)
#undef BD_CONV_CASE
    return fail(BD_ERR_INVALID_ARG, "bd_conv3d: unsupported channel combination");
}

int wgrad_launch(int nx, int ny, int nz, int cin, int cout, int taps, const void* grad, const void* act, float* dw,
                 cudaStream_t st, int* err) {
    const int sms = sm_count();
#define BD_WG_CASE(CO, CIS_)                    \
    if (cout == CO && (cin == CIS_ || (cin > CIS_ && CIS_ == (CO == 64 ? 16 : 32)))) \
        return launch_wgrad_t<CO, CIS_>(nx, ny, nz, cin, taps, grad, act, dw, st, err, sms);
    // more input channels run as slices: their accumulators would not fit TMEM
    BD_WG_CASE(16, 16) BD_WG_CASE(16, 32)
    BD_WG_CASE(32, 16) BD_WG_CASE(32, 32)
    BD_WG_CASE(64, 16)
#undef BD_WG_CASE
    return fail(BD_ERR_INVALID_ARG, "bd_conv3d_wgrad: unsupported channel combination");
}

int pack_weights_launch(int taps, int cin, int cout, int n_off, int n_slice, int transpose, const float* w, void* img,
                        cudaStream_t st) {
    const long long total = (long long)taps * (transpose ? cout : cin) * n_slice;
    const int blocks = (int)std::min<long long>((total + 255) / 256, 4096);
    k_pack_weights<<<blocks, 256, 0, st>>>(taps, cin, cout, n_off, n_slice, transpose, w,
                                           static_cast<__nv_bfloat16*>(img));
    BD_CHECK_LAUNCH("k_pack_weights");
    return BD_OK;
}

// Synchronous wrapper with a transient device error flag, for the standalone entry points.
template <class F>
static int run_checked(cudaStream_t st, const char* what, F launch) {
    int* err = nullptr;
    BD_CUDA(scratch_alloc((void**)&err, sizeof(int), st));
    int host_err = 0;
    cudaError_t e = cudaMemsetAsync(err, 0, sizeof(int), st);
    int rc = e == cudaSuccess ? launch(err) : BD_OK;
    if (e == cudaSuccess && rc == BD_OK) e = cudaMemcpyAsync(&host_err, err, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaError_t e2 = cudaFreeAsync(err, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (rc) return rc;
    if (e != cudaSuccess) return cuda_status(e, what);
    if (e2 != cudaSuccess) return cuda_status(e2, what);
    if (host_err) return fail(BD_ERR_TIMEOUT, "%s: a bounded pipeline wait timed out", what);
    return BD_OK;
}

}  // namespace bd

using namespace bd;

extern "C" int64_t bd_conv_plane_rows(int nx, int ny, int nz) {
    return (int64_t)(nx + 2) * (ny + 2) * (nz + 2) + kRowMargin;
}

extern "C" int64_t bd_conv_image_bytes(int taps, int k_channels, int n_slice) {
    return (int64_t)taps * k_channels * n_slice * 2;
}

extern "C" int bd_conv_pack_weights(int taps, int cin, int cout, int n_off, int n_slice, int transpose, const float* w,
                                    void* wimage, void* stream) {
    BD_REQUIRE(w && wimage, "bd_conv_pack_weights: NULL pointer");
    BD_REQUIRE(taps == 27 || taps == 9, "bd_conv_pack_weights: taps must be 27 or 9");
    BD_REQUIRE(cin % 8 == 0 && cout % 8 == 0 && n_slice > 0 && n_off >= 0, "bd_conv_pack_weights: bad channels");
    BD_REQUIRE(n_off + n_slice <= (transpose ? cin : cout), "bd_conv_pack_weights: slice out of range");
    return pack_weights_launch(taps, cin, cout, n_off, n_slice, transpose, w, wimage, (cudaStream_t)stream);
}

extern "C" int bd_conv3d(const BdConvCall* c, void* stream) {
    BD_REQUIRE(c != nullptr, "bd_conv3d: call is NULL");
    if (int rc = conv_check(*c)) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    return run_checked(st, "bd_conv3d", [&](int* err) { return conv_launch(*c, st, err); });
}

extern "C" int bd_conv3d_wgrad(int nx, int ny, int nz, int cin, int cout, int taps, const void* grad, const void* act,
                               float* dw, void* stream) {
    BD_REQUIRE(grad && act && dw, "bd_conv3d_wgrad: NULL pointer");
    BD_REQUIRE(nx > 0 && ny > 0 && nz > 0, "bd_conv3d_wgrad: dims must be positive");
    BD_REQUIRE((cin == 16 || cin == 32 || cin == 64) && (cout == 16 || cout == 32 || cout == 64),
               "bd_conv3d_wgrad: channels must be 16, 32 or 64");
    BD_REQUIRE(taps == 27 || taps == 9, "bd_conv3d_wgrad: taps must be 27 or 9");
    BD_REQUIRE((long long)(nx + 2) * (ny + 2) * (nz + 2) * 64 < (1LL << 31), "bd_conv3d_wgrad: volume too large");
    BD_REQUIRE(((uintptr_t)grad | (uintptr_t)act) % 16 == 0, "bd_conv3d_wgrad: volumes must be 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
    return run_checked(st, "bd_conv3d_wgrad",
                       [&](int* err) { return wgrad_launch(nx, ny, nz, cin, cout, taps, grad, act, dw, st, err); });
}
