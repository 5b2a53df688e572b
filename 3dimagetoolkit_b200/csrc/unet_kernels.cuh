// unet_kernels.cuh -- kernels of the learned Poisson warm start: a 3-level 3-D U-Net
// (16/32/64 channels, 3x3x3 convolutions) on BF16 channels-last activations.
//
// Tensors: voxel-major, channels fastest ("channels-last"), BF16, with a channel pitch
// (channels stored per voxel) and a channel offset, so that a decoder's concatenated
// input [upsampled | skip] is one tensor whose halves two producers write. Voxel index
// ((s * D + z) * H + y) * W + x for sample s: the reference's image3d order (i, j, k)
// with k contiguous.
//
// The 3x3x3 convolutions (forward, and the data gradient as a forward convolution with
// the flipped, transposed filter) run as implicit GEMMs on the tensor cores
// (conv3_march_kernel): a CTA stages, by TMA, one input plane of a tile after another --
// (TH + 2) rows x (TW + 2) columns of every 8-channel chunk, "chunk-planar" (see
// tc_sm100.cuh) -- with the out-of-volume halo zero-filled by the TMA unit, which is the
// convolution's zero padding. Each of the 9 taps of a plane is then the same block read
// at a row offset, so the A operand of every tap is a descriptor into one staged plane:
// no im2col buffer, one read of each plane per tile. M = 128 output positions of the
// padded tile, N = the output channels of the launch (16 or 32) of the three output planes
// that the input plane feeds, K = 16 input channels per instruction; the FP32 accumulators
// live in TMEM and are drained by 8 warps (bias + ReLU or the ReLU mask of the data
// gradient, BF16 store). The weight gradient (wgrad_mma_kernel) streams rows of the
// activations and of the output's gradient, with its accumulators in registers (mma.sync: its M
// fits 16 and 32 output channels).
// Pooling, the 2x2x2 transposed convolutions, the 1x1 output layer, the loss and Adam
// are small SIMT kernels.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdint>

#include "tc_sm100.cuh"

namespace im3d {
namespace unet {

typedef uint16_t bf16_t;  // raw BF16 bits in global memory

__device__ __forceinline__ float bf(bf16_t v) { return __uint_as_float(((uint32_t)v) << 16); }
__device__ __forceinline__ bf16_t to_bf(float v)
{
    return __bfloat16_as_ushort(__float2bfloat16_rn(v));
}

// two floats as packed BF16 (round to nearest), the first in the low half
__device__ __forceinline__ uint32_t pack_bf(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return (uint32_t)__bfloat16_as_ushort(v.x) | ((uint32_t)__bfloat16_as_ushort(v.y) << 16);
}

enum { CONV_BIAS_RELU = 0, CONV_MASK = 1, CONV_BIAS_F32 = 2 };

constexpr int kGuardBytes = 8192;  // after the staged blocks: the last M-tile's overreach

__host__ __device__ constexpr int align_up(int x, int a) { return (x + a - 1) / a * a; }

template <int CIN, int NOUT>
__host__ __device__ constexpr int conv_weight_bytes()
{
    return 27 * (CIN / 8) * NOUT * 16;
}

// Plan of one convolution launch by conv3_march_kernel (host-filled).
struct MarchGeom {
    int D, H, W;      // volume of one sample
    int TH, TW;       // tile rows (along H) and columns (along W; TW divides W, TW <= 128)
    int tiles_w, tiles_h;
    int zc, nzc;      // output planes of a unit, units along z
    long long units;  // nsamp * nzc * tiles_h * tiles_w
    int mtiles;       // 128-position MMA tiles of a plane
    int reg_bytes;    // one chunk region of a staged plane
    int stages;       // staged planes
    int slots;        // output planes in TMEM (>= 4)
    int tmem_cols;    // power of two >= slots * mtiles * NOUT
};

struct ConvArgs {
    MarchGeom g;
    const bf16_t* wpk;     // [N-block][9][CIN/8][3 NOUT][8] BF16 filter of this launch (pack_filter_kernel)
    const float* bias;     // output channels' bias (MODE 0, 2) or NULL
    void* out;             // BF16 (MODE 0, 1) or FP32 (MODE 2) channels-last
    int out_pitch, out_coff;
    const bf16_t* mask;    // MODE 1: result multiplied by (mask > 0), or NULL
    int mask_pitch, mask_coff;
    int in_coff;           // first input channel (a multiple of 8)
    int* err;              // raised when a wait gives up
};

constexpr int kMarchStages = 8, kMarchSlots = 8;  // most staged planes, most TMEM planes
constexpr int kMarchMaxMT = 4;    // most M-tiles of a plane
// warps of a block: one loader, MMA issuers, accumulator drains (a multiple of 4)
constexpr int kMarchIssuers = 4, kMarchDrains = 8;
constexpr int kMarchThreads = 32 * (1 + kMarchIssuers + kMarchDrains);

// dynamic shared memory of conv3_march_kernel<CIN, NOUT>
template <int CIN, int NOUT>
__host__ __device__ inline int march_smem_bytes(int reg_bytes, int stages)
{
    return align_up(conv_weight_bytes<CIN, NOUT>(), 1024) + stages * (CIN / 8) * reg_bytes + kGuardBytes +
           8 * (2 * kMarchStages + 2 * kMarchSlots) + 16 + 1024;
}

// Position of M-tile m's first row in a padded tile plane (pitch P = TW + 2): one interior
// row per M-tile when TW == 128, else 128 consecutive positions starting at the first
// interior one (rows of the tile and the 2 halo columns between them).
__device__ __forceinline__ int mtile_start(int TW, int m)
{
    const int P = TW + 2;
    return TW == 128 ? (m + 1) * P + 1 : P + 1 + 128 * m;
}

// 3x3x3 convolution, marching along z. A CTA takes units (a TH x TW column of tiles, zc
// output planes) in turn and streams the input planes z0-1 .. z0+zc of a unit once each
// through a ring in shared memory (TMA, one 8-channel chunk per load). Input plane z feeds
// three output planes: their accumulators sit side by side in TMEM (a ring of `slots` planes
// per M-tile), so one MMA of N = 3 NOUT columns adds a (dy, dx) tap of all three, with the
// filter packed as [tap][chunk][dz 2, 1, 0][NOUT]. An output plane still receives its 27 taps
// in the order dz, dy, dx, channel.
// Roles: one thread loads, 4 warps issue the MMAs (each its own M-tiles), 8 warps drain
// finished planes (bias + ReLU, or the ReLU mask of a data gradient) while the next planes are
// multiplied.
// What bounds it: the TMA moves 16-byte rows (8 channels of a voxel) at 2-3 cycles each, about
// 3800 cycles per plane of 4 x 128 voxels of 16 channels, against 36 + N / 4 cycles per MMA
// (measured, M = 128, K = 16: its operands go through shared memory), about 2000. Three dz taps
// per MMA cost little more than one, and each plane is loaded once instead of three times.
// 16-byte cp.async from 4 warps instead of the TMA measured 1.5 times slower.
// Measured against one block of three planes per output plane, load, MMAs (N = NOUT) and drain
// in turn (us): 16 -> 16 channels at 128^3 139 -> 74, 32 -> 16 406 -> 124, 64 -> 32 at 64^3
// 154 + 154 (N = 16) -> 67.
template <int CIN, int NOUT, int MODE>
__global__ void __launch_bounds__(kMarchThreads, 1) conv3_march_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ ConvArgs a)
{
    constexpr int KC = CIN / 8, N3 = 3 * NOUT;
    constexpr int WB = conv_weight_bytes<CIN, NOUT>();
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const MarchGeom& g = a.g;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int stage_bytes = KC * g.reg_bytes;
    unsigned char* wsm = smem;
    unsigned char* act = smem + align_up(WB, 1024);
    uint64_t* full = reinterpret_cast<uint64_t*>(act + g.stages * stage_bytes + kGuardBytes);  // plane loaded
    uint64_t* empty = full + kMarchStages;   // plane multiplied
    uint64_t* ready = empty + kMarchStages;  // output plane complete in TMEM
    uint64_t* drained = ready + kMarchSlots; // ... and read out
    uint32_t* tslot = reinterpret_cast<uint32_t*>(drained + kMarchSlots);
    __shared__ volatile int s_fail;
    __shared__ uint64_t s_last[kMarchIssuers];  // a failed issuer's MMAs have ended
    __shared__ float s_bias[NOUT];
    const int nb = blockIdx.y;  // block of NOUT output channels

    {
        const uint4* src = reinterpret_cast<const uint4*>(a.wpk + (size_t)nb * (WB / 2));
        uint4* dst = reinterpret_cast<uint4*>(wsm);
        for (int q = tid; q < WB / 16; q += blockDim.x) dst[q] = src[q];
    }
    if (tid < NOUT) s_bias[tid] = a.bias ? a.bias[nb * NOUT + tid] : 0.f;
    if (tid == 0) {
        for (int q = 0; q < kMarchStages; ++q) {
            tc::mbar_init(full + q, 1);
            tc::mbar_init(empty + q, kMarchIssuers);
        }
        for (int q = 0; q < kMarchSlots; ++q) {
            tc::mbar_init(ready + q, kMarchIssuers);
            tc::mbar_init(drained + q, kMarchDrains);
        }
        for (int q = 0; q < kMarchIssuers; ++q) tc::mbar_init(s_last + q, 1);
        tc::fence_mbar_init();
        s_fail = 0;
    }
    if (warp == 1) {
        tc::tmem_alloc(tslot, (uint32_t)g.tmem_cols);
        tc::tmem_relinquish();
    }
    tc::fence_proxy_async_smem();
    tc::tc_fence_before_sync();
    __syncthreads();
    tc::tc_fence_after_sync();
    const uint32_t tmem = *tslot;
    const int P = g.TW + 2, plane = (g.TH + 2) * P;
    // a unit's first tile row and column, first output plane, planes and sample
    auto unit = [&](long long u, int& w0, int& h0, int& z0, int& zn, int& s) {
        w0 = (int)(u % g.tiles_w) * g.TW;
        u /= g.tiles_w;
        h0 = (int)(u % g.tiles_h) * g.TH;
        u /= g.tiles_h;
        z0 = (int)(u % g.nzc) * g.zc;
        s = (int)(u / g.nzc);
        zn = min(g.zc, g.D - z0);
    };

    if (warp == 0) {
        if (lane == 0) {
            const uint32_t bytes = (uint32_t)KC * 16u * (uint32_t)plane;
            int st = 0, loaded = 0;  // next stage; planes loaded (counted up to the stages)
            uint32_t ph = 1;         // parity of a free stage: the first pass finds them free
            bool ok = true;
            for (long long u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
                int w0, h0, z0, zn, s;
                unit(u, w0, h0, z0, zn, s);
                for (int z = z0 - 1; z <= z0 + zn; ++z) {
                    if (!tc::mbar_wait(empty + st, ph)) s_fail = 1;
                    if (s_fail) {
                        ok = false;
                        break;
                    }
                    tc::mbar_arrive_expect_tx(full + st, bytes);
                    for (int c = 0; c < KC; ++c)
                        tc::tma_load_5d(act + st * stage_bytes + c * g.reg_bytes, &xmap, full + st, a.in_coff + 8 * c,
                                        w0 - 1, h0 - 1, z, s);
                    loaded = min(loaded + 1, g.stages);
                    if (++st == g.stages) {
                        st = 0;
                        ph ^= 1u;
                    }
                }
            }
            // after a failure the loads still in flight land before the block exits (the
            // stages before st hold this pass's planes, the others the last one's)
            if (!ok)
                for (int q = 0; q < loaded; ++q) tc::mbar_wait(full + q, q < st ? ph ^ 1u : ph, 1000000000ull);
        }
    } else if (warp < 1 + kMarchIssuers) {
        // lane 0 of each warp issues the MMAs of every kMarchIssuers-th M-tile
        if (lane == 0) {
            const uint32_t act_s = tc::smem_u32(act), w_s = tc::smem_u32(wsm);
            int st = 0;                // stage of the plane
            uint32_t ph = 0;           // ... and the parity of its load
            int sa = 0, sf = 0;        // TMEM slots of output planes max(z - 1, z0) and of the next fresh plane
            uint32_t phf = 1;          // parity of a drained fresh slot: the first pass finds them free
            bool ok = true;
            for (long long u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
                int w0, h0, z0, zn, s;
                unit(u, w0, h0, z0, zn, s);
                for (int z = z0 - 1; z <= z0 + zn; ++z) {
                    // output planes z-1 .. z+1 of this unit, as offsets from z0
                    const int o0 = max(z - 1 - z0, 0), o1 = min(z + 1 - z0, zn - 1);
                    const bool fresh = o1 == z + 1 - z0;  // plane z + 1 receives its first tap
                    if (fresh) {
                        ok = tc::mbar_wait(drained + sf, phf);
                        if (++sf == g.slots) {
                            sf = 0;
                            phf ^= 1u;
                        }
                    }
                    if (!ok || !tc::mbar_wait(full + st, ph) || s_fail) {
                        s_fail = 1;
                        ok = false;
                        break;
                    }
                    tc::tc_fence_after_sync();
                    // the planes o0 .. o1 are consecutive TMEM slots, split where the ring wraps;
                    // their filter rows start at dz = 1 - (o0 + z0 - z). Descriptors advance by
                    // additions to their low words (addresses below 256 KB: no carry)
                    const int cnt = o1 - o0 + 1;
                    const int n0 = min(cnt, g.slots - sa), n1 = cnt - n0;
                    const uint64_t bd0 = tc::smem_desc(w_s + (uint32_t)((o0 + z0 - (z - 1)) * NOUT * 16), (uint32_t)(N3 * 16), 128);
                    const uint64_t ad0 = tc::smem_desc(act_s + (uint32_t)(st * stage_bytes), (uint32_t)g.reg_bytes, 128);
                    const uint32_t id0 = tc::idesc_bf16(128, n0 * NOUT, false, false);
                    const uint32_t id1 = tc::idesc_bf16(128, n1 * NOUT, false, false);
                    const uint32_t ida = tc::idesc_bf16(128, NOUT, false, false);
                    const uint32_t kstep = (uint32_t)((2 * g.reg_bytes) >> 4);
                    for (int m = warp - 1; m < g.mtiles; m += kMarchIssuers) {
                        const uint64_t am = ad0 + (uint32_t)(mtile_start(g.TW, m) - P - 1);
                        const uint32_t dm = tmem + (uint32_t)(m * g.slots * NOUT);
                        const uint32_t d0 = dm + (uint32_t)(sa * NOUT);
                        if (fresh) {
                            // the fresh plane's first tap does not accumulate
                            for (int o = 0; o < cnt; ++o) {
                                const int so = sa + o < g.slots ? sa + o : sa + o - g.slots;
                                tc::mma_bf16(dm + (uint32_t)(so * NOUT), am, bd0 + (uint32_t)(o * NOUT), ida, o < cnt - 1);
                            }
                        }
#pragma unroll
                        for (int t = 0; t < 9; ++t) {
#pragma unroll
                            for (int ks = 0; ks < KC / 2; ++ks) {
                                if (t == 0 && ks == 0 && fresh) continue;
                                const uint64_t ad = am + (uint32_t)((t / 3) * P + t % 3) + ks * kstep;
                                const uint64_t bd = bd0 + (uint32_t)((t * KC + 2 * ks) * N3);
                                tc::mma_bf16_acc(d0, ad, bd, id0);
                                if (n1) tc::mma_bf16_acc(dm, ad, bd + (uint32_t)(n0 * NOUT), id1);
                            }
                        }
                    }
                    tc::mma_commit(empty + st);
                    if (++st == g.stages) {
                        st = 0;
                        ph ^= 1u;
                    }
                    if (z > z0) {  // output plane z - 1 is complete
                        tc::mma_commit(ready + sa);
                        if (++sa == g.slots) sa = 0;
                    }
                }
            }
            // after a failure the MMAs issued so far end before their operands and TMEM are given back
            if (!ok) {
                tc::mma_commit(s_last + warp - 1);
                tc::mbar_wait(s_last + warp - 1, 0, 1000000000ull);
            }
        }
    } else {
        const int lanes = (warp & 3) * 32;  // this warp's TMEM lanes
        // this warp's M-tiles mfirst, mfirst + MS, ..., and where its lane's position of each
        // lies: row py and column px of the tile, py < 0 for a halo position
        constexpr int MS = kMarchDrains / 4, MT = kMarchMaxMT / MS;
        const int mfirst = (warp - 1 - kMarchIssuers) >> 2;
        int off[MT], py[MT];
#pragma unroll
        for (int e = 0; e < MT; ++e) {
            const int pq = mtile_start(g.TW, mfirst + e * MS) + lanes + lane;
            const int r = pq / P, px = pq - r * P;
            py[e] = mfirst + e * MS < g.mtiles && r >= 1 && r <= g.TH && px >= 1 && px <= g.TW ? r - 1 : -1;
            off[e] = (r - 1) * g.W + px - 1;
        }
        const int c_first = nb * NOUT;
        const uint4* mask = MODE == CONV_MASK ? reinterpret_cast<const uint4*>(a.mask) : nullptr;
        int slot = 0;
        uint32_t ph = 0;
        bool ok = true;
        for (long long u = blockIdx.x; u < g.units && ok; u += gridDim.x) {
            int w0, h0, z0, zn, s;
            unit(u, w0, h0, z0, zn, s);
            for (int z = z0; z < z0 + zn; ++z) {
                const long long vbase = (((long long)s * g.D + z) * g.H + h0) * g.W + w0;
                // the ReLU mask of an M-tile is read one M-tile ahead (the first before the wait)
                uint4 mk[NOUT / 8], mkn[NOUT / 8];
                auto live = [&](int e) { return py[e] >= 0 && h0 + py[e] < g.H; };
                auto ld_mask = [&](int e) {
#pragma unroll
                    for (int n8 = 0; n8 < NOUT / 8; ++n8) {
                        mkn[n8] = make_uint4(0, 0, 0, 0);
                        if (mask && live(e))
                            mkn[n8] = *(reinterpret_cast<const uint4*>(a.mask + (vbase + off[e]) * a.mask_pitch +
                                                                       a.mask_coff + c_first) + n8);
                    }
                };
                if (MODE == CONV_MASK) ld_mask(0);
                if (!tc::mbar_wait(ready + slot, ph) || s_fail) {
                    s_fail = 1;
                    ok = false;
                    break;
                }
                tc::tc_fence_after_sync();
                __syncwarp();
#pragma unroll
                for (int e = 0; e < MT; ++e) {
                    const int m = mfirst + e * MS;
                    if (m >= g.mtiles) break;
                    if (MODE == CONV_MASK) {
#pragma unroll
                        for (int n8 = 0; n8 < NOUT / 8; ++n8) mk[n8] = mkn[n8];
                        if (e + 1 < MT) ld_mask(e + 1);
                    }
                    float v[NOUT];
                    __syncwarp();
#pragma unroll
                    for (int c0 = 0; c0 < NOUT; c0 += 16) {
                        float part[16];
                        tc::tmem_ld16(tmem + ((uint32_t)lanes << 16) + (uint32_t)((m * g.slots + slot) * NOUT + c0), part);
#pragma unroll
                        for (int n = 0; n < 16; ++n) v[c0 + n] = part[n];
                    }
                    if (!live(e)) continue;
                    const long long vox = vbase + off[e];
                    if (MODE != CONV_MASK) {
#pragma unroll
                        for (int n = 0; n < NOUT; ++n) v[n] += s_bias[n];
                    }
                    if (MODE == CONV_BIAS_F32) {
                        float* o = reinterpret_cast<float*>(a.out) + vox * a.out_pitch + a.out_coff + c_first;
                        if ((reinterpret_cast<uintptr_t>(o) & 15) == 0) {
#pragma unroll
                            for (int n = 0; n < NOUT; n += 4)
                                reinterpret_cast<float4*>(o)[n / 4] = make_float4(v[n], v[n + 1], v[n + 2], v[n + 3]);
                        } else {
#pragma unroll
                            for (int n = 0; n < NOUT; ++n) o[n] = v[n];
                        }
                        continue;
                    }
                    if (MODE == CONV_BIAS_RELU) {
#pragma unroll
                        for (int n = 0; n < NOUT; ++n) v[n] = fmaxf(v[n], 0.f);
                    } else if (mask) {
#pragma unroll
                        for (int n8 = 0; n8 < NOUT / 8; ++n8) {
                            const uint32_t w4[4] = {mk[n8].x, mk[n8].y, mk[n8].z, mk[n8].w};
#pragma unroll
                            for (int n = 0; n < 4; ++n) {
                                if (!(bf((bf16_t)(w4[n] & 0xffff)) > 0.f)) v[n8 * 8 + 2 * n] = 0.f;
                                if (!(bf((bf16_t)(w4[n] >> 16)) > 0.f)) v[n8 * 8 + 2 * n + 1] = 0.f;
                            }
                        }
                    }
                    uint4* o = reinterpret_cast<uint4*>(reinterpret_cast<bf16_t*>(a.out) + vox * a.out_pitch + a.out_coff + c_first);
#pragma unroll
                    for (int n8 = 0; n8 < NOUT / 8; ++n8) {
                        uint4 pk;
                        pk.x = pack_bf(v[n8 * 8 + 0], v[n8 * 8 + 1]);
                        pk.y = pack_bf(v[n8 * 8 + 2], v[n8 * 8 + 3]);
                        pk.z = pack_bf(v[n8 * 8 + 4], v[n8 * 8 + 5]);
                        pk.w = pack_bf(v[n8 * 8 + 6], v[n8 * 8 + 7]);
                        o[n8] = pk;
                    }
                }
                // this warp's part of the slot may be multiplied into again
                __syncwarp();
                tc::tc_fence_before_sync();
                if (lane == 0) tc::mbar_arrive(drained + slot);
                if (++slot == g.slots) {
                    slot = 0;
                    ph ^= 1u;
                }
            }
        }
    }
    __syncwarp();
    tc::tc_fence_before_sync();
    __syncthreads();
    if (s_fail && tid == 0) atomicExch(a.err, 1);
    if (warp == 1) tc::tmem_dealloc(tmem, (uint32_t)g.tmem_cols);
}

// ---------------------------------------------------------------- weight gradient
constexpr int kWgWarps = 12;                     // multiplying warps
constexpr int kWgThreads = 32 * (kWgWarps + 1);  // and one that loads
constexpr int kWgXRows = 8, kWgZRows = 5;        // rows of X (of three planes) and of dZ in shared memory

struct WgradArgs {
    int D, H, W;       // volume of one sample
    int TH, TW;        // tile rows and columns (TW divides W, TW <= 128, a multiple of 16)
    int tiles_w, tiles_h;
    long long ntiles;  // nsamp * D * tiles_h * tiles_w
    int xbytes, zbytes;  // a staged row of X (three planes, halo included) and of dZ
    int zcoff, xcoff;    // first channel of dZ and of X in their tensors
    int cin;             // input channels of the layer
    float* dw;           // FP32 gradient [CO][cin][27] (the parameter layout), accumulated with atomics
    int* err;
};

__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t addr, uint32_t (&r)[4])
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}

// D (16 x 8, FP32) += A (16 x 16) * B (16 x 8), BF16
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
                 "{%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Byte offset of 16-byte chunk c of row r in rows of ROW bytes that the TMA wrote with its
// ROW-byte swizzle (32: chunk bit 0 ^ address bit 7; 64: chunk bits ^ bits 7, 8; 128: ^ bits 7 to 9).
template <int ROW>
__device__ __forceinline__ uint32_t swizzled(int r, int c)
{
    return (uint32_t)(r * ROW + ((ROW == 32 ? c ^ ((r >> 2) & 1) : ROW == 64 ? c ^ ((r >> 1) & 3) : c ^ (r & 7)) << 4));
}

// The sums of one row of dZ by a warp: NT taps of 16 * MB output channels against 16 input
// channels, 16 voxels per step along the row. zp: this lane's ldmatrix row per block of 16
// output channels; xp: per tap.
template <int NT, int MB, int RZ>
__device__ __forceinline__ void wgrad_row(float (&acc)[3][MB][2][4], const uint32_t (&zp)[MB], const uint32_t (&xp)[3], int ksteps)
{
#pragma unroll(MB == 4 ? 1 : 2)
    for (int kc = 0; kc < ksteps; ++kc) {
        uint32_t zf[MB][4], xf[NT][4];
#pragma unroll
        for (int m = 0; m < MB; ++m) ldmatrix_x4_trans(zp[m] + kc * (16 * RZ), zf[m]);
#pragma unroll
        for (int t = 0; t < NT; ++t) ldmatrix_x4_trans(xp[t] + kc * (16 * 32), xf[t]);
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int m = 0; m < MB; ++m)
#pragma unroll
                for (int n = 0; n < 2; ++n) mma_16816(acc[t][m][n], zf[m], xf[t][2 * n], xf[t][2 * n + 1]);
    }
}

// dW[co][ci][tap] = sum over voxels of dZ[v][co] X[v + tap][ci], for all CO output channels and
// 16 input channels (blockIdx.y).
// The order of the sums is part of the result: the tensor core's FP32 accumulator truncates, so
// that another order moves the gradient by up to 6e-5 (2 x 128 x 128 x 256), and a training run
// with it. Every (co, ci, tap) is one chain of multiplications of 16 voxels each: block
// blockIdx.x takes the tiles blockIdx.x, blockIdx.x + gridDim.x, ... (columns, rows, planes,
// samples, the first fastest) row by row, 16 voxels after 16 along a row, and the blocks' sums
// are added to the gradient with one atomic each. The host's plan (wgrad_plan) fixes the
// tiles and the number of blocks.
// Rows stream through rings in shared memory (TMA): a row of X of the three planes around the
// tile's, and a row of dZ. The 27 taps are spread over 12 warps, three to the first three, two to
// the others (7, 7, 7 and 6 per scheduler), each with its sums in registers throughout.
// The products run on mma.sync (M = 16 output channels, N = 8 input channels, K = 16 voxels),
// which gives the bits of tcgen05.mma for the same chain: both operands are read transposed from
// channels-last rows by ldmatrix, and M = 16 fits 16 and 32 channels exactly, where tcgen05's
// smallest M (64) multiplies three quarters or half of it for nothing.
// us (output x input channels): 16 x 16 at 128^3 124, 16 x 32 at 128^3 261, 32 x 32 at 64^3 60,
// 32 x 16 at 64^3 37; the same chains on tcgen05, load and multiply in turn: 929, 950, 420 for
// the first three. What bounds it: the reads of the fragments from shared memory (its port busy
// 36 to 61 % of the time) and the fixed latency of mma.sync, whose pipe is busy 28 to 46 %. Consecutive tiles of a chain lie in other rows and planes, so X is read for each of
// its three planes anew; chains marching along z (90, 157, 48, 32 us) are other sums.
template <int CO>
__global__ void __launch_bounds__(kWgThreads, 1) wgrad_mma_kernel(const __grid_constant__ CUtensorMap xmap,
                                                                  const __grid_constant__ CUtensorMap zmap,
                                                                  const __grid_constant__ WgradArgs a)
{
    constexpr int CI = 16, RX = 2 * CI, RZ = 2 * CO, MB = CO / 16;  // RX, RZ: bytes of a voxel
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    unsigned char* zs = smem;
    unsigned char* xs = zs + kWgZRows * a.zbytes;
    uint64_t* fullx = reinterpret_cast<uint64_t*>(xs + kWgXRows * a.xbytes);
    uint64_t* emptyx = fullx + kWgXRows;
    uint64_t* fullz = emptyx + kWgXRows;
    uint64_t* emptyz = fullz + kWgZRows;
    __shared__ volatile int s_fail;
    if (tid == 0) {
        for (int q = 0; q < kWgXRows; ++q) {
            tc::mbar_init(fullx + q, 1);
            tc::mbar_init(emptyx + q, kWgWarps);
        }
        for (int q = 0; q < kWgZRows; ++q) {
            tc::mbar_init(fullz + q, 1);
            tc::mbar_init(emptyz + q, kWgWarps);
        }
        tc::fence_mbar_init();
        s_fail = 0;
    }
    __syncthreads();
    const int cib = blockIdx.y;
    const int P = a.TW + 8;  // voxels of a staged row of X: a multiple of 8 keeps the swizzle's phase
    float acc[3][MB][2][4];  // [this warp's taps][16 output channels][8 input channels]
#pragma unroll
    for (int t = 0; t < 3; ++t)
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
            for (int e = 0; e < 8; ++e) acc[t][m][e >> 2][e & 3] = 0.f;
    // a tile's first column and row, its rows inside the volume, plane and sample
    auto place = [&](long long r, int& w0, int& h0, int& rows, int& z, int& s) {
        w0 = (int)(r % a.tiles_w) * a.TW;
        r /= a.tiles_w;
        h0 = (int)(r % a.tiles_h) * a.TH;
        r /= a.tiles_h;
        z = (int)(r % a.D);
        s = (int)(r / a.D);
        rows = min(a.TH, a.H - h0);
    };
    if (warp == kWgWarps) {
        if (lane == 0) {
            const uint32_t xb = (uint32_t)(3 * P * RX), zb = (uint32_t)(a.TW * RZ);
            int sx = 0, sz = 0, nx = 0, nzl = 0;  // next slots, loads issued (up to the slots)
            uint32_t phx = 1, phz = 1;            // parity of a free slot: the first pass finds them free
            bool ok = true;
            for (long long tile = blockIdx.x; tile < a.ntiles && ok; tile += gridDim.x) {
                int w0, h0, rows, z, s;
                place(tile, w0, h0, rows, z, s);
                // X rows h0 - 1 .. h0 + rows; the dZ row h goes out with the X row h + 1
                for (int j = 0; j < rows + 2 && ok; ++j) {
                    ok = tc::mbar_wait(emptyx + sx, phx) && !s_fail;
                    if (!ok) break;
                    tc::mbar_arrive_expect_tx(fullx + sx, xb);
                    tc::tma_load_5d(xs + sx * a.xbytes, &xmap, fullx + sx, a.xcoff + cib * CI, w0 - 1, h0 - 1 + j, z - 1, s);
                    nx = min(nx + 1, kWgXRows);
                    if (++sx == kWgXRows) {
                        sx = 0;
                        phx ^= 1u;
                    }
                    if (j < 2) continue;
                    ok = tc::mbar_wait(emptyz + sz, phz) && !s_fail;
                    if (!ok) break;
                    tc::mbar_arrive_expect_tx(fullz + sz, zb);
                    tc::tma_load_5d(zs + sz * a.zbytes, &zmap, fullz + sz, a.zcoff, w0, h0 + j - 2, z, s);
                    nzl = min(nzl + 1, kWgZRows);
                    if (++sz == kWgZRows) {
                        sz = 0;
                        phz ^= 1u;
                    }
                }
            }
            if (!ok) {
                // the loads still in flight land before the block exits
                s_fail = 1;
                for (int q = 0; q < nx; ++q) tc::mbar_wait(fullx + q, q < sx ? phx ^ 1u : phx, 1000000000ull);
                for (int q = 0; q < nzl; ++q) tc::mbar_wait(fullz + q, q < sz ? phz ^ 1u : phz, 1000000000ull);
            }
        }
    } else {
        // ldmatrix rows of this lane: A (voxel, chunk of 8 output channels), B (voxel, chunk of
        // 8 input channels) of the fragment order of mma.m16n8k16
        const int av = (lane & 7) + ((lane >> 4) << 3), ac = (lane >> 3) & 1;
        const int bv = (lane & 7) + (((lane >> 3) & 1) << 3), bc = lane >> 4;
        uint32_t zo[MB], xo[3];
        int dy[3];
#pragma unroll
        for (int m = 0; m < MB; ++m) zo[m] = tc::smem_u32(zs) + swizzled<RZ>(av, 2 * m + ac);
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            const int tap = min(warp + t * kWgWarps, 26);  // dz * 9 + dy * 3 + dx
            dy[t] = tap / 3 % 3;
            xo[t] = tc::smem_u32(xs) + (uint32_t)(tap / 9 * P * RX) + swizzled<RX>(bv + tap % 3, bc);
        }
        const int ksteps = a.TW / 16;
        int sx = 0, sz = 0;       // slots of X row h - 1 and of dZ row h
        uint32_t wx = 0, wz = 0;  // parities of the next X slot to wait for and of dZ
        int nwx = 0;              // next X slot to wait for
        bool ok = true;
        for (long long tile = blockIdx.x; tile < a.ntiles && ok; tile += gridDim.x) {
            int w0, h0, rows, z, s;
            place(tile, w0, h0, rows, z, s);
            for (int r = 0; r < rows; ++r) {
                for (int q = r == 0 ? 0 : 2; q < 3 && ok; ++q) {
                    ok = tc::mbar_wait(fullx + nwx, wx) && !s_fail;
                    if (++nwx == kWgXRows) {
                        nwx = 0;
                        wx ^= 1u;
                    }
                }
                ok = ok && tc::mbar_wait(fullz + sz, wz) && !s_fail;
                ok = __all_sync(0xffffffffu, ok);
                if (!ok) break;
                uint32_t zp[MB], xp[3];
#pragma unroll
                for (int m = 0; m < MB; ++m) zp[m] = zo[m] + (uint32_t)(sz * a.zbytes);
#pragma unroll
                for (int t = 0; t < 3; ++t) {
                    const int q = sx + dy[t] < kWgXRows ? sx + dy[t] : sx + dy[t] - kWgXRows;
                    xp[t] = xo[t] + (uint32_t)(q * a.xbytes);
                }
                if (warp < 27 - 2 * kWgWarps) wgrad_row<3, MB, RZ>(acc, zp, xp, ksteps);
                else wgrad_row<2, MB, RZ>(acc, zp, xp, ksteps);
                __syncwarp();
                // X row h - 1 (and at the tile's end h and h + 1) and dZ row h are free
                for (int q = 0; q < (r == rows - 1 ? 3 : 1); ++q) {
                    if (lane == 0) tc::mbar_arrive(emptyx + sx);
                    if (++sx == kWgXRows) sx = 0;
                }
                if (lane == 0) tc::mbar_arrive(emptyz + sz);
                if (++sz == kWgZRows) {
                    sz = 0;
                    wz ^= 1u;
                }
            }
        }
        if (!ok) s_fail = 1;
    }
    __syncthreads();
    // every load has landed and been read: the rings hold the block's sums, [co][ci][tap]
    if (!s_fail) {
        float* sum = reinterpret_cast<float*>(smem);
        const int g = lane >> 2, t4 = lane & 3;
        if (warp < kWgWarps) {
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const int tap = warp + t * kWgWarps;
                if (tap > 26) continue;
#pragma unroll
                for (int m = 0; m < MB; ++m)
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const int co = m * 16 + g + ((e >> 1) & 1) * 8, ci = (e >> 2) * 8 + 2 * t4 + (e & 1);
                        sum[(co * CI + ci) * 27 + tap] = acc[t][m][e >> 2][e & 3];
                    }
            }
        }
        __syncthreads();
        // (rows of CI x 27 floats start on 16 bytes: the filters' offsets are multiples of 16)
        for (int e = 4 * tid; e < CO * CI * 27; e += 4 * kWgThreads) {
            const int co = e / (CI * 27), rest = e - co * (CI * 27);
            atomicAdd(reinterpret_cast<float4*>(a.dw + ((size_t)co * a.cin + cib * CI) * 27 + rest),
                      *reinterpret_cast<const float4*>(sum + e));
        }
    }
    if (s_fail && tid == 0) atomicExch(a.err, 2);
}

// ------------------------------------------------------------------ SIMT kernels
// 8 BF16 channels as floats
__device__ __forceinline__ void unpack8(const uint4& q, float (&v)[8])
{
    const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        v[2 * e] = __uint_as_float(w[e] << 16);
        v[2 * e + 1] = __uint_as_float(w[e] & 0xffff0000u);
    }
}
__device__ __forceinline__ uint4 pack8(const float (&v)[8])
{
    return make_uint4(pack_bf(v[0], v[1]), pack_bf(v[2], v[3]), pack_bf(v[4], v[5]), pack_bf(v[6], v[7]));
}

// sum over voxels of dZ[v][c] (c < C) into db[c]; 8 channels per thread and read, the block's
// sums added once (a scalar read and a shared atomic per thread took 35 us at 128^3 x 16,
// bandwidth 11)
template <int C>
__global__ void __launch_bounds__(256) bias_grad_kernel(const bf16_t* __restrict__ dz, int pitch, int coff, long long n,
                                                        float* db)
{
    constexpr int G = C / 8, LANES = 256 / G;
    __shared__ float part[8][C];
    const int g = threadIdx.x % G;
    float s[8];
#pragma unroll
    for (int e = 0; e < 8; ++e) s[e] = 0.f;
    for (long long v = (long long)blockIdx.x * LANES + threadIdx.x / G; v < n; v += (long long)gridDim.x * LANES) {
        float x[8];
        unpack8(*reinterpret_cast<const uint4*>(dz + v * pitch + coff + 8 * g), x);
#pragma unroll
        for (int e = 0; e < 8; ++e) s[e] += x[e];
    }
#pragma unroll
    for (int e = 0; e < 8; ++e)
#pragma unroll
        for (int o = G; o < 32; o <<= 1) s[e] += __shfl_xor_sync(0xffffffffu, s[e], o);
    if ((threadIdx.x & 31) < G)
#pragma unroll
        for (int e = 0; e < 8; ++e) part[threadIdx.x >> 5][8 * g + e] = s[e];
    __syncthreads();
    if (threadIdx.x < C) {
        float t = 0.f;
#pragma unroll
        for (int w = 0; w < 8; ++w) t += part[w][threadIdx.x];
        atomicAdd(db + threadIdx.x, t);
    }
}

// 2x2x2 max pooling of channels [coff, coff + C) of `in` (pitch ip) into out [n/8][C]
// (pitch C); idx receives the argmax child (0..7) per output value. 8 channels per thread.
__global__ void pool_fwd_kernel(const bf16_t* __restrict__ in, int ip, int coff, int C, int D, int H, int W,
                                int nsamp, bf16_t* __restrict__ out, uint8_t* __restrict__ idx)
{
    const int D2 = D / 2, H2 = H / 2, W2 = W / 2, G = C / 8;
    const long long total = (long long)nsamp * D2 * H2 * W2 * G;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int g = (int)(e % G);
        const long long p = e / G;
        const int x = (int)(p % W2);
        long long r = p / W2;
        const int y = (int)(r % H2);
        r /= H2;
        const int z = (int)(r % D2);
        const int s = (int)(r / D2);
        uint4 q[8];
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            const long long v = (((long long)s * D + 2 * z + (o >> 2)) * H + 2 * y + ((o >> 1) & 1)) * W + 2 * x + (o & 1);
            q[o] = *reinterpret_cast<const uint4*>(in + v * ip + coff + 8 * g);
        }
        float best[8];
        uint32_t bi[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            best[c] = -3.0e38f;
            bi[c] = 0;
        }
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            float f[8];
            unpack8(q[o], f);
#pragma unroll
            for (int c = 0; c < 8; ++c)
                if (f[c] > best[c]) {
                    best[c] = f[c];
                    bi[c] = (uint32_t)o;
                }
        }
        reinterpret_cast<uint4*>(out)[e] = pack8(best);
        reinterpret_cast<uint2*>(idx)[e] = make_uint2(bi[0] | bi[1] << 8 | bi[2] << 16 | bi[3] << 24,
                                                      bi[4] | bi[5] << 8 | bi[6] << 16 | bi[7] << 24);
    }
}

// Gradient of the pooled skip tensor: for every child cell of a pooled cell,
//   g[child] = (g_skip[child] + (child == argmax ? g_pool : 0)) * (act[child] > 0)
// (act = the pooled ReLU output). g may alias g_skip (same pitch and offset). 8 channels per
// thread, every child's reads before the first store.
__global__ void pool_bwd_kernel(const bf16_t* __restrict__ gpool, const uint8_t* __restrict__ idx, int C, int D,
                                int H, int W, int nsamp, const bf16_t* gskip, int sp, int soff,
                                const bf16_t* __restrict__ act, int ap, int aoff, bf16_t* g, int gp, int goff)
{
    const int D2 = D / 2, H2 = H / 2, W2 = W / 2, G = C / 8;
    const long long total = (long long)nsamp * D2 * H2 * W2 * G;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < total; e += (long long)gridDim.x * blockDim.x) {
        const int c8 = 8 * (int)(e % G);
        const long long p = e / G;
        const int x = (int)(p % W2);
        long long r = p / W2;
        const int y = (int)(r % H2);
        r /= H2;
        const int z = (int)(r % D2);
        const int s = (int)(r / D2);
        float gv[8];
        unpack8(reinterpret_cast<const uint4*>(gpool)[e], gv);
        const uint2 ix = reinterpret_cast<const uint2*>(idx)[e];
        const long long v0 = (((long long)s * D + 2 * z) * H + 2 * y) * W + 2 * x;
#pragma unroll
        for (int oz = 0; oz < 2; ++oz) {
            uint4 qs[4], qa[4];
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                const long long v = v0 + ((long long)oz * H + (o >> 1)) * W + (o & 1);
                qs[o] = gskip ? *reinterpret_cast<const uint4*>(gskip + v * sp + soff + c8) : make_uint4(0, 0, 0, 0);
                qa[o] = *reinterpret_cast<const uint4*>(act + v * ap + aoff + c8);
            }
#pragma unroll
            for (int o = 0; o < 4; ++o) {
                const long long v = v0 + ((long long)oz * H + (o >> 1)) * W + (o & 1);
                float val[8], av[8];
                unpack8(qs[o], val);
                unpack8(qa[o], av);
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const uint32_t bi = ((c < 4 ? ix.x : ix.y) >> (8 * (c & 3))) & 0xffu;
                    if (bi == (uint32_t)(4 * oz + o)) val[c] += gv[c];
                    if (!(av[c] > 0.f)) val[c] = 0.f;
                }
                *reinterpret_cast<uint4*>(g + v * gp + goff + c8) = pack8(val);
            }
        }
    }
}

// 2x2x2 stride-2 transposed convolution: out[child(p, o)][co] = b[co] + sum_ci
// in[p][ci] U[o][ci][co], the sum in the order of ci. A thread holds the channels of VX coarse
// voxels and goes through the children of its block (blockIdx.y: OG of them) and 16 output
// channels at a time; the filter sits in shared memory as floats and is read as broadcast
// 16-byte vectors, the sums run on the paired FP32 instructions. (One thread per output voxel
// with a 2-byte shared read per product took 266 us for 32 -> 16 channels at 128^3.)
template <int CI, int CO, int VX, int OG>
__global__ void __launch_bounds__(128) upconv_fwd_kernel(const bf16_t* __restrict__ in, const bf16_t* __restrict__ U,
                                                         const float* __restrict__ b, int D2, int H2, int W2, int nsamp,
                                                         bf16_t* out, int op, int ooff)
{
    extern __shared__ __align__(16) float us[];  // [OG][CI][CO]
    const int o0 = blockIdx.y * OG;
    for (int q = threadIdx.x; q < OG * CI * CO; q += blockDim.x) us[q] = bf(U[o0 * CI * CO + q]);
    __syncthreads();
    const int H = 2 * H2, W = 2 * W2;
    const long long total = (long long)nsamp * D2 * H2 * W2;  // a multiple of VX
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t * VX < total; t += (long long)gridDim.x * blockDim.x) {
        const long long p = t * VX;
        uint4 xq[VX][CI / 8];
#pragma unroll
        for (int v = 0; v < VX; ++v)
#pragma unroll
            for (int c = 0; c < CI / 8; ++c) xq[v][c] = reinterpret_cast<const uint4*>(in + (p + v) * CI)[c];
        const int x = (int)(p % W2);  // the VX voxels lie in one row (W2 a multiple of VX)
        long long r = p / W2;
        const int y = (int)(r % H2);
        r /= H2;  // r = s * D2 + z
        for (int og = 0; og < OG; ++og) {
            const int o = o0 + og;
            const long long vox = ((2 * r + (o >> 2)) * H + 2 * y + ((o >> 1) & 1)) * W + 2 * x + (o & 1);
#pragma unroll
            for (int h = 0; h < CO / 16; ++h) {
                float2 acc[VX][8];
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float2 bb = make_float2(__ldg(b + h * 16 + 2 * c), __ldg(b + h * 16 + 2 * c + 1));
#pragma unroll
                    for (int v = 0; v < VX; ++v) acc[v][c] = bb;
                }
                const float* ub = us + og * CI * CO + h * 16;
#pragma unroll
                for (int c8 = 0; c8 < CI / 8; ++c8) {
                    float xv[VX][8];
#pragma unroll
                    for (int v = 0; v < VX; ++v) unpack8(xq[v][c8], xv[v]);
#pragma unroll
                    for (int e = 0; e < 8; ++e) {
                        const float4* u4 = reinterpret_cast<const float4*>(ub + (c8 * 8 + e) * CO);
#pragma unroll
                        for (int c = 0; c < 4; ++c) {
                            const float4 w = u4[c];
#pragma unroll
                            for (int v = 0; v < VX; ++v) {
                                const float2 x2 = make_float2(xv[v][e], xv[v][e]);
                                acc[v][2 * c] = __ffma2_rn(x2, make_float2(w.x, w.y), acc[v][2 * c]);
                                acc[v][2 * c + 1] = __ffma2_rn(x2, make_float2(w.z, w.w), acc[v][2 * c + 1]);
                            }
                        }
                    }
                }
#pragma unroll
                for (int v = 0; v < VX; ++v) {
                    uint4* dst = reinterpret_cast<uint4*>(out + (vox + 2 * v) * op + ooff + h * 16);
                    dst[0] = make_uint4(pack_bf(acc[v][0].x, acc[v][0].y), pack_bf(acc[v][1].x, acc[v][1].y),
                                        pack_bf(acc[v][2].x, acc[v][2].y), pack_bf(acc[v][3].x, acc[v][3].y));
                    dst[1] = make_uint4(pack_bf(acc[v][4].x, acc[v][4].y), pack_bf(acc[v][5].x, acc[v][5].y),
                                        pack_bf(acc[v][6].x, acc[v][6].y), pack_bf(acc[v][7].x, acc[v][7].y));
                }
            }
        }
    }
}

// Data gradient of the transposed convolution, masked by the ReLU of its input:
//   g_in[p][ci] = (sum_{o, co} g_out[child(p, o)][co] U[o][ci][co]) * (in[p][ci] > 0),
// the sum in the order of o, co. One coarse voxel and CB input channels (blockIdx.y) per
// thread; the filter sits in shared memory as floats, [o][co][ci of the block].
template <int CI, int CO, int CB>
__global__ void __launch_bounds__(128) upconv_bwd_kernel(const bf16_t* __restrict__ gout, int gp, int goff,
                                                         const bf16_t* __restrict__ U, const bf16_t* __restrict__ in,
                                                         int D2, int H2, int W2, int nsamp, bf16_t* __restrict__ gin)
{
    extern __shared__ __align__(16) float us[];  // [8][CO][CB]
    const int c0 = blockIdx.y * CB;
    for (int q = threadIdx.x; q < 8 * CO * CB; q += blockDim.x) {
        const int ci = q % CB, co = q / CB % CO, o = q / (CB * CO);
        us[q] = bf(U[(o * CI + c0 + ci) * CO + co]);
    }
    __syncthreads();
    const int H = 2 * H2, W = 2 * W2;
    const long long total = (long long)nsamp * D2 * H2 * W2;
    for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < total; p += (long long)gridDim.x * blockDim.x) {
        const int x = (int)(p % W2);
        long long r = p / W2;
        const int y = (int)(r % H2);
        r /= H2;
        float2 acc[CB / 2];
#pragma unroll
        for (int c = 0; c < CB / 2; ++c) acc[c] = make_float2(0.f, 0.f);
        for (int o = 0; o < 8; ++o) {
            const long long v = ((2 * r + (o >> 2)) * H + 2 * y + ((o >> 1) & 1)) * W + 2 * x + (o & 1);
            const uint4* gr = reinterpret_cast<const uint4*>(gout + v * gp + goff);
#pragma unroll
            for (int c8 = 0; c8 < CO / 8; ++c8) {
                float gv[8];
                unpack8(gr[c8], gv);
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const float4* u4 = reinterpret_cast<const float4*>(us + (o * CO + c8 * 8 + e) * CB);
                    const float2 g2 = make_float2(gv[e], gv[e]);
#pragma unroll
                    for (int c = 0; c < CB / 4; ++c) {
                        const float4 w = u4[c];
                        acc[2 * c] = __ffma2_rn(g2, make_float2(w.x, w.y), acc[2 * c]);
                        acc[2 * c + 1] = __ffma2_rn(g2, make_float2(w.z, w.w), acc[2 * c + 1]);
                    }
                }
            }
        }
        const uint4* ip = reinterpret_cast<const uint4*>(in + p * CI + c0);
        uint4* dst = reinterpret_cast<uint4*>(gin + p * CI + c0);
#pragma unroll
        for (int c8 = 0; c8 < CB / 8; ++c8) {
            float iv[8], ov[8];
            unpack8(ip[c8], iv);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float a = e & 1 ? acc[c8 * 4 + e / 2].y : acc[c8 * 4 + e / 2].x;
                ov[e] = a * (iv[e] > 0.f ? 1.f : 0.f);
            }
            dst[c8] = pack8(ov);
        }
    }
}

// Weight and bias gradient of the transposed convolution:
//   dU[o][ci][co] += sum_p in[p][ci] g_out[child(p, o)][co],  db[co] += sum g_out[.][co],
// as products of M = 16 input channels, N = 8 output channels and K = 16 coarse voxels on
// mma.sync; warp o takes child o. A block stages 64 coarse voxels (4 row segments of 16) and
// their 512 children at a time, two stages ahead of each other, in rows padded by 16 bytes
// (ldmatrix reads 8 rows on distinct banks), and adds its sums once. (One scalar product per
// thread and voxel took 550 us for 32 -> 16 channels at 128^3, this 30.)
// The tensor core's accumulator truncates, so it holds one stage only (4 multiplications); the
// stages are joined by FP32 additions that round to nearest. Error of up1's gradient against
// FP64 sums at 128^3 / 2 x 128 x 128 x 256: 2.6e-7 / 2.7e-7 (one accumulator over all
// stages 2.4e-6 / 6.3e-6; scalar products 1.1e-6 / 1.0e-6).
template <int CI, int CO>
struct UpWgrad {
    static constexpr int TP = 64, RI = 2 * CI + 16, RG = 2 * CO + 16;      // voxels, row bytes
    static constexpr int stage = TP * RI + 8 * TP * RG;                     // bytes
};
template <int CI, int CO>
__global__ void __launch_bounds__(256) upconv_wgrad_kernel(const bf16_t* __restrict__ in,
                                                           const bf16_t* __restrict__ gout, int gp, int goff,
                                                           int D2, int H2, int W2, int nsamp, float* dU, float* db)
{
    typedef UpWgrad<CI, CO> G;
    constexpr int TP = G::TP, RI = G::RI, RG = G::RG;
    extern __shared__ __align__(16) unsigned char sm[];
    const int tid = threadIdx.x, lane = tid & 31, o = tid >> 5;
    const int H = 2 * H2, W = 2 * W2;
    const long long total = (long long)nsamp * D2 * H2 * W2;  // a multiple of 16
    const long long tiles = (total + TP - 1) / TP;
    // stage s: in[TP][CI], then children [8][TP][CO]
    auto load = [&](long long tile, int s) {
        unsigned char* bi = sm + s * G::stage;
        unsigned char* bg = bi + TP * RI;
        for (int q = tid; q < TP * (CI / 8); q += 256) {
            const int v = q / (CI / 8), c = q % (CI / 8);
            const long long p = tile * TP + v;
            tc::cp_async16_zfill(bi + v * RI + c * 16, p < total ? in + p * CI + 8 * c : in, p < total);
        }
        for (int q = tid; q < 8 * TP * (CO / 8); q += 256) {
            const int c = q % (CO / 8), f = q / (CO / 8);
            const int ox = f & 1, v = (f >> 1) % TP, zy = f / (2 * TP);  // children of a row side by side
            const long long p = tile * TP + v;
            const int x = (int)(p % W2);
            long long r = p / W2;
            const int y = (int)(r % H2);
            r /= H2;
            const long long vox = ((2 * r + (zy >> 1)) * H + 2 * y + (zy & 1)) * W + 2 * x + ox;
            tc::cp_async16_zfill(bg + ((zy * 2 + ox) * TP + v) * RG + c * 16,
                                 p < total ? gout + vox * gp + goff + 8 * c : gout, p < total);
        }
        tc::cp_async_commit();
    };
    float acc[CI / 16][CO / 8][4], bs[CO / 8];
#pragma unroll
    for (int n = 0; n < CO / 8; ++n) {
        bs[n] = 0.f;
#pragma unroll
        for (int m = 0; m < CI / 16; ++m)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[m][n][e] = 0.f;
    }
    const int av = (lane & 7) + ((lane >> 4) << 3), ac = (lane >> 3) & 1;
    const int bv = (lane & 7) + (((lane >> 3) & 1) << 3), bc = lane >> 4;
    long long tile = blockIdx.x;
    if (tile < tiles) load(tile, 0);
    for (int s = 0; tile < tiles; tile += gridDim.x, s ^= 1) {
        if (tile + gridDim.x < tiles) {
            load(tile + gridDim.x, s ^ 1);
            tc::cp_async_wait<1>();
        } else {
            tc::cp_async_wait<0>();
        }
        __syncthreads();
        const uint32_t bi = tc::smem_u32(sm + s * G::stage), bg = bi + TP * RI + (uint32_t)(o * TP * RG);
        uint32_t gf[TP / 16][CO / 16][4];
#pragma unroll
        for (int n = 0; n < CO / 16; ++n) {
            float b0 = 0.f, b1 = 0.f;  // this lane's share of the bias sums: channel lane / 4 of each 8
#pragma unroll
            for (int k = 0; k < TP / 16; ++k) {
                uint32_t(&f)[4] = gf[k][n];
                ldmatrix_x4_trans(bg + (uint32_t)((16 * k + bv) * RG + (2 * n + bc) * 16), f);
                auto four = [](uint32_t u, uint32_t v) {
                    return (__uint_as_float(u << 16) + __uint_as_float(u & 0xffff0000u)) +
                           (__uint_as_float(v << 16) + __uint_as_float(v & 0xffff0000u));
                };
                b0 += four(f[0], f[1]);
                b1 += four(f[2], f[3]);
            }
            bs[2 * n] += b0;
            bs[2 * n + 1] += b1;
        }
#pragma unroll
        for (int m = 0; m < CI / 16; ++m) {
            float part[CO / 8][4];
#pragma unroll
            for (int n = 0; n < CO / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) part[n][e] = 0.f;
#pragma unroll
            for (int k = 0; k < TP / 16; ++k) {
                uint32_t af[4];
                ldmatrix_x4_trans(bi + (uint32_t)((16 * k + av) * RI + (2 * m + ac) * 16), af);
#pragma unroll
                for (int n = 0; n < CO / 16; ++n) {
                    mma_16816(part[2 * n], af, gf[k][n][0], gf[k][n][1]);
                    mma_16816(part[2 * n + 1], af, gf[k][n][2], gf[k][n][3]);
                }
            }
#pragma unroll
            for (int n = 0; n < CO / 8; ++n)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[m][n][e] += part[n][e];
        }
        __syncthreads();
    }
    const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
    for (int m = 0; m < CI / 16; ++m)
#pragma unroll
        for (int n = 0; n < CO / 8; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int ci = m * 16 + g + (e >> 1) * 8, co = n * 8 + 2 * t4 + (e & 1);
                atomicAdd(dU + (o * CI + ci) * CO + co, acc[m][n][e]);
            }
    // the children's bias sums are joined in shared memory (every stage has been read)
    float(*bsum)[CO] = reinterpret_cast<float(*)[CO]>(sm);
#pragma unroll
    for (int n = 0; n < CO / 8; ++n) {
        bs[n] += __shfl_xor_sync(0xffffffffu, bs[n], 1);
        bs[n] += __shfl_xor_sync(0xffffffffu, bs[n], 2);
        if (t4 == 0) bsum[o][n * 8 + g] = bs[n];
    }
    __syncthreads();
    if (tid < CO) {
        float t = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) t += bsum[c][tid];
        atomicAdd(db + tid, t);
    }
}

// 1x1 output layer, loss and its gradient in one pass:
//   y = b + sum_c w[c] d[v][c];  diff = y - target (on the cells with weight != 0);
//   loss += diff^2 * wt; dy = 2 diff wt / count;  g_d[v][c] = dy w[c] (d[v][c] > 0);
//   dw[c] += dy d[v][c], db += dy.
// target == NULL: forward only (y written, nothing else). The sums are folded by shuffles and
// one add per block (a shared atomic per thread and channel took 650 of 668 us at 128^3).
template <int C>
__global__ void __launch_bounds__(256) out_layer_kernel(const bf16_t* __restrict__ d, const float* __restrict__ w,
                                                        const float* __restrict__ b, long long n, float* y,
                                                        const float* __restrict__ target,
                                                        const float* __restrict__ wt, float inv_count,
                                                        bf16_t* __restrict__ gd, float* dw, float* db, double* loss)
{
    __shared__ float sg[8][C + 1];
    __shared__ double sl[8];
    float wv_[C];
#pragma unroll
    for (int c = 0; c < C; ++c) wv_[c] = __ldg(w + c);
    const float bias = __ldg(b);
    float gl[C];
#pragma unroll
    for (int c = 0; c < C; ++c) gl[c] = 0.f;
    float gb = 0.f;
    double ls = 0.0;
    for (long long v = blockIdx.x * (long long)blockDim.x + threadIdx.x; v < n; v += (long long)gridDim.x * blockDim.x) {
        float dv[C];
        const uint4* dp = reinterpret_cast<const uint4*>(d + v * C);
#pragma unroll
        for (int c8 = 0; c8 < C / 8; ++c8) {
            float t[8];
            unpack8(dp[c8], t);
#pragma unroll
            for (int h = 0; h < 8; ++h) dv[c8 * 8 + h] = t[h];
        }
        float yv = bias;
#pragma unroll
        for (int c = 0; c < C; ++c) yv = fmaf(wv_[c], dv[c], yv);
        if (y) y[v] = yv;
        if (!target) continue;
        const float wv = wt ? wt[v] : 1.f;
        const float diff = (yv - target[v]) * wv;
        ls += (double)diff * diff;
        const float dy = 2.f * diff * wv * inv_count;
        gb += dy;
        uint4* gp = reinterpret_cast<uint4*>(gd + v * C);
#pragma unroll
        for (int c8 = 0; c8 < C / 8; ++c8) {
            float go[8];
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                const int c = c8 * 8 + h;
                gl[c] = fmaf(dy, dv[c], gl[c]);
                go[h] = dv[c] > 0.f ? dy * wv_[c] : 0.f;
            }
            gp[c8] = pack8(go);
        }
    }
    if (!target) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int c = 0; c < C; ++c) gl[c] += __shfl_xor_sync(0xffffffffu, gl[c], o);
        gb += __shfl_xor_sync(0xffffffffu, gb, o);
        ls += __shfl_xor_sync(0xffffffffu, ls, o);
    }
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < C; ++c) sg[warp][c] = gl[c];
        sg[warp][C] = gb;
        sl[warp] = ls;
    }
    __syncthreads();
    if (threadIdx.x <= C) {
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) t += sg[q][threadIdx.x];
        atomicAdd(threadIdx.x < C ? dw + threadIdx.x : db, t);
    }
    if (threadIdx.x == 32) {
        double t = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) t += sl[q];
        atomicAdd(loss, t);
    }
}

// Adam step on FP32 master parameters (bias-corrected learning rate lr_t).
__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g, float* __restrict__ m,
                            float* __restrict__ v, long long n, float lr_t, float b1, float b2, float eps,
                            float gscale)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x) {
        const float gq = g[q] * gscale;
        const float mq = b1 * m[q] + (1.f - b1) * gq;
        const float vq = b2 * v[q] + (1.f - b2) * gq * gq;
        m[q] = mq;
        v[q] = vq;
        p[q] -= lr_t * mq / (sqrtf(vq) + eps);
    }
}

// FP32 filter W[co][ci][27] -> BF16 operand blocks of conv3_march_kernel: block nb holds
// outputs nb*NOUT .. of the launch, [9 taps (dy, dx)][CIN/8][dz 2, 1, 0][NOUT][8]:
//   forward (transpose = 0): element (t, kc, dz, n, e) = W[nb*NOUT + n][kc*8 + e][9 dz + t]
//     (CIN = layer Cin)
//   data gradient (transpose = 1): the flipped, transposed filter, CIN = layer Cout,
//     outputs = layer Cin: W[kc*8 + e][nb*NOUT + n][26 - (9 dz + t)]
struct PackJob {
    const float* W;
    bf16_t* out;
    int cout, cin, nout, transpose;
};
struct PackJobs {
    PackJob job[20];
};
__device__ __forceinline__ void pack_filter(const PackJob& j, long long first, long long step)
{
    const int kcin = j.transpose ? j.cout : j.cin;   // K of the GEMM
    const int nall = j.transpose ? j.cin : j.cout;   // N of the GEMM
    const long long total = 27ll * kcin * nall;
    for (long long e = first; e < total; e += step) {
        const int el = (int)(e % 8);
        long long r = e / 8;
        const int n = (int)(r % j.nout);
        r /= j.nout;
        const int dz = 2 - (int)(r % 3);
        r /= 3;
        const int kc = (int)(r % (kcin / 8));
        r /= kcin / 8;
        const int t = 9 * dz + (int)(r % 9);
        const int nb = (int)(r / 9);
        const int k = kc * 8 + el, nn = nb * j.nout + n;
        const float w = j.transpose ? j.W[((size_t)k * j.cin + nn) * 27 + (26 - t)] : j.W[((size_t)nn * j.cin + k) * 27 + t];
        j.out[e] = to_bf(w);
    }
}
// one filter per blockIdx.y
__global__ void pack_filter_kernel(const __grid_constant__ PackJobs jobs)
{
    pack_filter(jobs.job[blockIdx.y], blockIdx.x * (long long)blockDim.x + threadIdx.x, (long long)gridDim.x * blockDim.x);
}

__global__ void to_bf16_kernel(const float* __restrict__ src, bf16_t* __restrict__ dst, long long n)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        dst[q] = to_bf(src[q]);
}

__global__ void zero_f32_kernel(float* p, long long n)
{
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < n; q += (long long)gridDim.x * blockDim.x)
        p[q] = 0.f;
}

}  // namespace unet
}  // namespace im3d
