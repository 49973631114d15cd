// learned_train_tc.cu -- training of the learned smoother with its hidden
// layer (16 -> 16 channels, 84 % of the network's multiply-adds) on the
// tensor cores (tcgen05, BF16 operands, FP32 accumulation in tensor memory),
// and the first and last layers on the CUDA cores, all on BF16 channels-last
// activations (32 bytes per cell).
//
// Patches are cubes: the input x has side S = P + 8, the activations h1 side
// S1 = S - 2, h2 side S2 = S - 4, the output y side S3 = S - 6 (valid 3x3x3
// convolutions; tap d = (dx, dy, dz) in {0,1,2}^3, index dx + 3 dy + 9 dz).
//
// The hidden layer's three GEMMs:
//   forward        out[q][co] = sum_{t,ci} h1[q + d][ci] W[t][ci][co]
//   backward-data  gin[c][ci] = sum_e gout[c - 2 + e][co] W[26 - e][ci][co],
//                  the forward's form with the source gout, shift -2, taps
//                  flipped and W transposed; the ReLU mask of the layer's
//                  input applied in the epilogue
// run brick-staged (brick_tc_kernel): a brick of output cells with its
// source region in shared memory, each tap's A operand the same rows
// shifted (K-major, M = 128 cells, K = 16 channels, N = 16), 27 MMAs per
// 128-row tile.
//   weight grad    gW[t][ci][co] = sum_q h1[q + d][ci] gout[q][co]
// runs on bricks too, with the cells as K (wgrad_tc_kernel): both operands
// MN-major, A = (dz, channel) of the source region against the brick's gout
// rows shifted by dx, one accumulator per dy, added to gW with atomics once per
// CTA.
// Every wait in both kernels is bounded (an error word is set and the CTA
// stops issuing).
#include "cn_fastdiv.h"
#include "cn_internal.h"
#include "cn_tc.cuh"
#include "cn_tma.cuh"
#include "learned_tc.h"

#include <cuda_bf16.h>

#include <algorithm>

namespace cn {
namespace nntr {

constexpr uint32_t WBYTES = 27 * 512;            // packed weights of one layer
constexpr uint32_t IDESC_K = tc::idesc_bf16_f32(128, 16);
// M = 64, N = 48, both operands MN-major (bits 15 and 16)
constexpr uint32_t IDESC_MN = tc::idesc_bf16_f32(64, 48) | (1u << 15) | (1u << 16);

enum { FWD = 0, BWD = 1 };

struct Args {
    const uint16_t *src;  // gathered activations [B][Sin^3][16] BF16
    const uint16_t *gout; // weight gradient: [B][Sout^3][16] gradient at the layer's output
    const uint16_t *act;  // backward-data: the layer's input at the output cells (ReLU mask)
    const uint16_t *w;    // forward / backward-data: packed B tiles [27][2][16][8]
    uint16_t *out;        // forward / backward-data: [B][Sout^3][16]
    float *gw;            // weight gradient: [27][16][16] FP32, accumulated
    int Sin, Sout, shift;
    int relu;
    int *err;
};

__device__ __forceinline__ uint16_t bf16_bits(float v) { return __bfloat16_as_ushort(__float2bfloat16_rn(v)); }

// 16-byte asynchronous copy; src_bytes 0 writes zeros (nothing is read)
__device__ __forceinline__ void cp16(void *dst, const void *src, uint32_t src_bytes)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(src_bytes)
                 : "memory");
}

// ------------------------------------------------------ weight gradient
// gW[t][ci][co] = sum over cells q of h1[q + d(t)][ci] gout[q][co]: K = cells.
// A CTA takes bricks of BX x BY x BZ output cells and stages, per z plane and
// channel half, the rows (16 bytes: 8 channels of a cell) of the source region
// (row x + RX y, RX = BX + 2) and of gout in the same numbering, zero in rows
// that are no cell of the brick.  MN-major, a plane of rows is 8 rows of A^T,
// and the planes (z, half) are evenly spaced: 8 of them from plane z on are the
// M = 64 of the three dz taps (the last 16 rows, a plane too far, are dropped),
// and dy is a start address RX dy rows on.  gout is staged three times, shifted
// by dx rows: its planes (dx, half) are the N = 48.  3 MMAs per 16 cells (K) into
// 3 accumulators of 48 columns, kept over all bricks of the CTA.  Against a
// gather of every tap's rows (27 copies of 32 bytes a cell) a cell is staged 1.5
// and its gradient 3 times; B200, 32 patches of 32^3: 384 -> 116 us (with dx as
// start addresses too, 9 MMAs of N = 16 at 37 cycles each: 155, of which the MMAs
// alone 122 and the staging alone 66).  Two CTAs per SM, one staging while the
// other's MMAs run.
constexpr int WGT_NT = 256;
constexpr int WGT_SMEM = 110 * 1024; // two CTAs per SM
constexpr uint32_t WGT_COLS = 256;   // 3 x 48, a power of two

struct WgGeo {
    int BX, BY, BZ;  // brick of output cells
    int RX;          // BX + 2
    int H, KP;       // rows per staged plane: source region, gout (a multiple of 16)
    int bricks[3];   // per patch
    int total;       // in all
};

__global__ void __launch_bounds__(WGT_NT, 2) wgrad_tc_kernel(const __grid_constant__ Args a,
                                                             const __grid_constant__ WgGeo g)
{
    extern __shared__ __align__(128) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar;
    __shared__ uint32_t slot;
    __shared__ int flag;
    const uint32_t aplane = (uint32_t)g.H * 16u, gplane = (uint32_t)g.KP * 16u;
    unsigned char *A = smem;                              // [BZ + 3][2][H][16 B], the last z plane never written
    unsigned char *G = smem + 2 * (g.BZ + 3) * aplane;    // [BZ][3 shifts][2][KP][16 B]
    const int r = threadIdx.x, warp = r >> 5;
    if (r == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(&slot, WGT_COLS);
        tc::tmem_relinquish();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = slot;

    const int Si = a.Sin, So = a.Sout, per = g.bricks[0] * g.bricks[1] * g.bricks[2];
    const int64_t si2 = (int64_t)Si * Si, so2 = (int64_t)So * So;
    bool ok = true;
    int it = 0;
    for (int brick = blockIdx.x; brick < g.total; brick += gridDim.x, ++it) {
        const int b = brick / per;
        int br = brick - b * per;
        const int ox = (br % g.bricks[0]) * g.BX;
        br /= g.bricks[0];
        const int oy = (br % g.bricks[1]) * g.BY, oz = (br / g.bricks[1]) * g.BZ;
        const int nx = min(g.BX, So - ox), ny = min(g.BY, So - oy), nz = min(g.BZ, So - oz);
        const int ks = (g.RX * ny + 15) / 16; // K steps per z plane
        if (it > 0) {                         // the previous brick's MMAs have read the buffers
            if (r == 0) flag = mbar_wait_bounded(&bar, (it - 1) & 1) ? 1 : 0;
            __syncthreads();
            if (!flag) {
                ok = false;
                break;
            }
        }
        // source region: all rows the shifted K steps read, zero past the region
        const int arows = 16 * ks + 2 + 2 * g.RX;
        for (int t = r; t < 2 * arows; t += WGT_NT) {
            const int u = t >> 1, hh = t & 1, y = u / g.RX, x = u - y * g.RX;
            const bool in = x < nx + 2 && y < ny + 2;
            const uint16_t *src = in ? a.src + (((int64_t)b * Si + oz) * si2 + (int64_t)(oy + y) * Si + ox + x) * 16 + 8 * hh
                                     : a.src;
            unsigned char *dst = A + hh * aplane + u * 16;
            for (int z = 0; z < nz + 2; ++z) {
                cp16(dst + 2 * z * aplane, src, in ? 16u : 0u);
                if (in) src += si2 * 16;
            }
        }
        for (int t = r; t < 32 * ks; t += WGT_NT) {
            const int u = t >> 1, hh = t & 1, y = u / g.RX, x = u - y * g.RX;
            const int64_t e = (((int64_t)b * So + oz) * so2 + (int64_t)(oy + y) * So + ox + x) * 16 + 8 * hh;
            unsigned char *dst = G + hh * gplane + u * 16;
            for (int z = 0; z < nz; ++z)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const bool in = (unsigned)(x - c) < (unsigned)nx && y < ny;
                    cp16(dst + (6 * z + 2 * c) * gplane, in ? a.gout + e + (z * so2 - c) * 16 : a.gout, in ? 16u : 0u);
                }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        fence_proxy_async_smem(); // generic-proxy smem writes -> visible to the tensor cores
        tc::fence_before_sync();
        __syncthreads();
        if (r == 0) {
            tc::fence_after_sync();
            // descriptors: K cores 128 bytes apart, planes H or KP rows; the
            // address field counts rows (16 bytes)
            const uint64_t da = tc::smem_desc(smem_u32(A), 128u, aplane), db = tc::smem_desc(smem_u32(G), 128u, gplane);
            for (int z = 0; z < nz; ++z) {
#pragma unroll 1
                for (int k = 0; k < ks; ++k) {
                    const uint64_t ak = da + (uint32_t)(2 * z * g.H + 16 * k), bk = db + (uint32_t)(6 * z * g.KP + 16 * k);
                    const uint32_t acc = it + z + k > 0 ? 1u : 0u;
#pragma unroll
                    for (int dy = 0; dy < 3; ++dy)
                        tc::mma_bf16(tbase + 48u * dy, ak + (uint32_t)(g.RX * dy), bk, IDESC_MN, acc);
                }
            }
            tc::mma_commit(&bar);
        }
    }
    if (ok && it > 0) { // the last brick's MMAs, then gW
        if (r == 0) flag = mbar_wait_bounded(&bar, (it - 1) & 1) ? 1 : 0;
        __syncthreads();
        ok = flag != 0;
        // row 16 dz + ci of an M = 64 accumulator lies in lane 32 dz + ci; warp w
        // reads dz = w % 4 (3: the dropped rows), columns 8 (w / 4) .. + 7
        if (ok && (warp & 3) < 3) {
            tc::fence_after_sync();
            const int dz = warp & 3, ci = r & 31, co = 8 * (warp >> 2);
#pragma unroll 1
            for (int t = 0; t < 9; ++t) {
                float v[8];
                tc::tmem_ld8(tbase + ((uint32_t)(32 * dz) << 16) + 16u * t + (uint32_t)co, v);
                if (ci < 16) { // gw rows are 64-byte aligned
                    float4 *dst = reinterpret_cast<float4 *>(a.gw + ((t + 9 * dz) * 16 + ci) * 16 + co);
                    atomicAdd(dst, make_float4(v[0], v[1], v[2], v[3]));
                    atomicAdd(dst + 1, make_float4(v[4], v[5], v[6], v[7]));
                }
            }
        }
    }
    if (!ok && r == 0 && a.err) atomicExch(a.err, kDevErrTimeout);
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tbase, WGT_COLS);
}

// Brick shape of the weight gradient for B output cubes of side So: of the
// splits that fit the shared memory of half an SM, the least of (bricks per
// CTA) x (a brick's MMAs at 40 cycles each, its staging at 40 bytes a cycle and
// 2500 cycles of latency) + 16 cycles of atomics per CTA.
static WgGeo wgrad_geo(int B, int So, int ctas, size_t *smem)
{
    WgGeo best = {};
    double least = 0;
    for (int nx = (So + 63) / 64, last = nx + 2; nx <= last && nx <= So; ++nx) {
        WgGeo g;
        g.BX = (So + nx - 1) / nx;
        g.RX = g.BX + 2;
        g.bricks[0] = (So + g.BX - 1) / g.BX;
        for (g.BZ = 1; g.BZ <= 8 && g.BZ <= So; ++g.BZ)
            for (g.BY = 1; g.BY <= So; ++g.BY) {
                g.KP = (g.RX * g.BY + 15) / 16 * 16;
                g.H = (g.KP + 2 + 2 * g.RX + 7) / 8 * 8;
                const int64_t bytes = 32LL * ((g.BZ + 3) * g.H + 3 * g.BZ * g.KP);
                if (bytes > WGT_SMEM) break;
                g.bricks[1] = (So + g.BY - 1) / g.BY;
                g.bricks[2] = (So + g.BZ - 1) / g.BZ;
                g.total = B * g.bricks[0] * g.bricks[1] * g.bricks[2];
                const double cost = (double)((g.total + ctas - 1) / ctas) *
                                        (7.5 * g.BZ * g.KP + bytes / 40.0 + 2500.0) +
                                    16.0 * (g.total < ctas ? g.total : ctas);
                if (best.total == 0 || cost < least) {
                    least = cost;
                    best = g;
                    *smem = (size_t)bytes;
                }
            }
    }
    return best;
}

// backward-data B tiles: tap e, K = the layer's output channel co, N = its
// input channel ci: B[e][kc][ci][8] = W[26 - e][ci][kc * 8 + j]
__global__ void pack_bwd_kernel(const float *W, uint16_t *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 27 * 256) return;
    const int e = i / 256, rr = i % 256;
    const int kc = rr / 128, ci = (rr / 8) % 16, j = rr % 8;
    out[i] = bf16_bits(W[((26 - e) * 16 + ci) * 16 + kc * 8 + j]);
}

// ------------------------------------------------ brick-staged forward
// The forward and data-gradient GEMMs without im2col, as the grid inference
// kernel does it: a CTA owns a brick of BX x BY x BZ output cells of one
// patch (BX the whole row) and stages the source region around it, (BX+2) x
// (BY+2) x (BZ+2) cells starting at the brick origin + shift, zero outside
// the source cube, one row of 16 channels per region cell (two K planes of
// 16-byte rows).  Output cell (x, y, z) sits at row m = x + RX y + RX RY z
// and its tap e source at row m + e_x + RX e_y + RX RY e_z, so a tap's A
// operand for a 128-row tile is the same run of rows shifted: 27 MMAs (M =
// 128, N = 16, K = 16) per tile into one TMEM accumulator.  Rows whose (x,
// y, z) fall outside the brick or the output cube are computed and dropped.
// One brick per CTA; the wait for the MMAs is bounded (error word, skipped
// epilogue).
struct BrickGeo {
    int BX, BY, BZ;        // brick of output cells
    int RX, RY, RZ;        // source region = brick + 2
    int MT;                // 128-row M tiles covering the brick's rows
    int SROWS;             // staged rows: 128 MT + the largest tap offset (zero past the region)
    int bricks[3];         // bricks per patch along x, y, z
    FastDiv dRX, dRXY;     // divisions by RX, RX RY
};

constexpr int BRICK_NT = 256;
// A brick's copies, MMAs and epilogue follow one another, so small bricks and
// four CTAs per SM, which overlap; B200, the batch of 32 patches of 32^3: two
// CTAs (2880 rows, 16 tiles) 955 us, three 921, four 924; 5 patches of 13^3 184,
// 172, 169.
constexpr int BRICK_CTAS = 4;
constexpr int BRICK_MAX_ROWS = 1352;    // 2 planes x 1352 x 16 B and the weights: a quarter of the SM's shared memory
constexpr int BRICK_MAX_MT = 8;         // 128 TMEM columns

template <int MODE>
__global__ void __launch_bounds__(BRICK_NT, BRICK_CTAS) brick_tc_kernel(const __grid_constant__ Args a,
                                                                const __grid_constant__ BrickGeo g)
{
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t plane = (uint32_t)g.SROWS * 16u;
    unsigned char *A = smem;                          // [2][SROWS][16 B]
    unsigned char *Wb = smem + 2 * plane;             // [27][2][16][16 B]
    uint64_t *bar = reinterpret_cast<uint64_t *>(Wb + WBYTES);
    uint32_t *slot = reinterpret_cast<uint32_t *>(bar + 1);
    int *okf = reinterpret_cast<int *>(slot + 1);
    const int r = threadIdx.x, warp = r >> 5;
    constexpr uint32_t TCOLS = 16 * BRICK_MAX_MT;

    const int per = g.bricks[0] * g.bricks[1] * g.bricks[2];
    const int b = blockIdx.x / per;
    int br = blockIdx.x - b * per;
    const int ox = (br % g.bricks[0]) * g.BX;
    br /= g.bricks[0];
    const int oy = (br % g.bricks[1]) * g.BY;
    const int oz = (br / g.bricks[1]) * g.BZ;

    if (r == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    if (warp == 0) {
        tc::tmem_alloc(slot, TCOLS);
        tc::tmem_relinquish();
    }
    for (int i = r; i < (int)(WBYTES / 16); i += BRICK_NT)
        reinterpret_cast<uint4 *>(Wb)[i] = __ldg(reinterpret_cast<const uint4 *>(a.w) + i);
    // ---- source region: lanes 2i, 2i+1 copy the two channel halves of a row,
    // one column along z after the other
    const int rxy = g.RX * g.RY;
    const int64_t si2 = (int64_t)a.Sin * a.Sin;
    for (int t = r; t < 2 * rxy; t += BRICK_NT) {
        const int u = t >> 1, hh = t & 1, j = g.dRX.div(u), i = u - j * g.RX;
        const int sx = ox + i + a.shift, sy = oy + j + a.shift, sz0 = oz + a.shift;
        const bool xy = (unsigned)sx < (unsigned)a.Sin && (unsigned)sy < (unsigned)a.Sin;
        const uint16_t *col = a.src + (((int64_t)b * a.Sin + sz0) * si2 + (int64_t)a.Sin * sy + sx) * 16 + 8 * hh;
        unsigned char *dst = A + hh * plane + u * 16;
        for (int k = 0; k < g.RZ; ++k) {
            const bool in = xy && (unsigned)(sz0 + k) < (unsigned)a.Sin;
            cp16(dst + k * rxy * 16, in ? col + k * si2 * 16 : a.src, in ? 16u : 0u);
        }
    }
    for (int t = r; t < 2 * (g.SROWS - rxy * g.RZ); t += BRICK_NT) // the rows past it
        *reinterpret_cast<uint4 *>(A + (t & 1) * plane + (rxy * g.RZ + (t >> 1)) * 16) = make_uint4(0, 0, 0, 0);
    asm volatile("cp.async.wait_all;" ::: "memory");
    fence_proxy_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tbase = *slot;

    if (r == 0) {
        const uint32_t a0 = smem_u32(A), b0 = smem_u32(Wb);
        const int sy = g.RX, sz = g.RX * g.RY;
#pragma unroll 1
        for (int t = 0; t < g.MT; ++t) {
#pragma unroll
            for (int q = 0; q < 27; ++q) {
                const int off = q % 3 + sy * ((q / 3) % 3) + sz * (q / 9);
                const uint64_t da = tc::smem_desc(a0 + 16u * (uint32_t)(128 * t + off), plane, 128u);
                const uint64_t db = tc::smem_desc(b0 + 512u * q, 256u, 128u);
                tc::mma_bf16(tbase + 16u * t, da, db, IDESC_K, q > 0 ? 1u : 0u);
            }
        }
        tc::mma_commit(bar);
        *okf = mbar_wait_bounded(bar, 0) ? 1 : 0;
    }
    __syncthreads();
    const int ok = *okf;
    tc::fence_after_sync();
    if (ok) {
        // warp w: TMEM lanes 32 (w % 4) .. + 31 of tiles w / 4, w / 4 + 2, ...
        const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;
        const int64_t so3 = (int64_t)a.Sout * a.Sout * a.Sout;
#pragma unroll 1
        for (int t = warp >> 2; t < g.MT; t += 2) {
            float v[16];
            tc::tmem_ld16(tbase + lanes + 16u * t, v);
            const int m = 128 * t + 32 * (warp & 3) + (r & 31);
            const int z = g.dRXY.div(m), rem = m - z * rxy;
            const int y = g.dRX.div(rem), x = rem - y * g.RX;
            const int X = ox + x, Y = oy + y, Z = oz + z;
            if (x >= g.BX || y >= g.BY || z >= g.BZ || X >= a.Sout || Y >= a.Sout || Z >= a.Sout) continue;
            const int64_t L = (int64_t)b * so3 + X + (int64_t)a.Sout * (Y + (int64_t)a.Sout * Z);
            uint32_t h[8];
            if (MODE == BWD) {
                const uint4 *mk = reinterpret_cast<const uint4 *>(a.act + L * 16);
                const uint4 m0 = mk[0], m1 = mk[1];
                const uint32_t mw[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const float lo = __uint_as_float(mw[q] << 16), hi = __uint_as_float(mw[q] & 0xFFFF0000u);
                    h[q] = (uint32_t)bf16_bits(lo > 0.f ? v[2 * q] : 0.f) |
                           ((uint32_t)bf16_bits(hi > 0.f ? v[2 * q + 1] : 0.f) << 16);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    float p = v[2 * q], u = v[2 * q + 1];
                    if (a.relu) {
                        p = fmaxf(p, 0.f);
                        u = fmaxf(u, 0.f);
                    }
                    h[q] = (uint32_t)bf16_bits(p) | ((uint32_t)bf16_bits(u) << 16);
                }
            }
            uint4 *dst = reinterpret_cast<uint4 *>(a.out + L * 16);
            dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
            dst[1] = make_uint4(h[4], h[5], h[6], h[7]);
        }
    } else if (r == 0 && a.err) {
        atomicExch(a.err, kDevErrTimeout);
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tbase, TCOLS);
}

// Brick shape for an output cube of side So: whole rows (BX = So, at most
// 64), and the (BY, BZ), BZ <= 4, of least cost while the staged rows fit
// BRICK_MAX_ROWS and the tiles BRICK_MAX_MT; cost = bricks x (tiles + 3),
// a brick's set-up (weights, barrier, TMEM, staging latency) counted as
// three tiles of MMAs.  False if none fits.
static bool brick_geo(int So, BrickGeo &g)
{
    g.BX = So < 64 ? So : 64;
    g.RX = g.BX + 2;
    const int64_t bx = (So + g.BX - 1) / g.BX;
    int64_t best = -1;
    for (int bz = 1; bz <= 4 && bz <= So; ++bz)
        for (int by = 1; by <= So; ++by) {
            const int ry = by + 2, rz = bz + 2;
            const int span = (g.BX - 1) + g.RX * (by - 1) + g.RX * ry * (bz - 1) + 1;
            const int mt = (span + 127) / 128;
            const int offmax = 2 + 2 * g.RX + 2 * g.RX * ry;
            const int srows = ((128 * mt + offmax + 7) / 8) * 8;
            if (mt > BRICK_MAX_MT || srows > BRICK_MAX_ROWS || srows < g.RX * ry * rz) continue;
            const int64_t cost = bx * ((So + by - 1) / by) * ((So + bz - 1) / bz) * (mt + 3);
            if (best < 0 || cost < best) {
                best = cost;
                g.BY = by;
                g.BZ = bz;
                g.RY = ry;
                g.RZ = rz;
                g.MT = mt;
                g.SROWS = srows;
            }
        }
    if (best < 0) return false;
    g.bricks[0] = (int)bx;
    g.bricks[1] = (So + g.BY - 1) / g.BY;
    g.bricks[2] = (So + g.BZ - 1) / g.BZ;
    g.dRX = FastDiv((uint32_t)g.RX);
    g.dRXY = FastDiv((uint32_t)(g.RX * g.RY));
    return true;
}

// ---------------------------------------------------- CUDA-core layers
// The first and last layers and their gradients: FP32 arithmetic on pairs of
// channels (two multiply-adds per instruction), bound by instruction issue.
// Every kernel tiles its cells so that an operand unpacked from BF16, or a
// tap's weights read from shared memory, serves several cells or taps; B200,
// batch of 32 patches of 32^3 cells, against one cell and tap at a time:
// l1_fwd_cl 163 -> 83 us, l3_fwd_cl 114 -> 70, l3_bwd_data_cl 107 -> 45,
// l3_wgrad_cl 161 -> 57, l1_wgrad_cl 280 -> 146.
__device__ __forceinline__ float2 fma2(float a, float2 b, float2 c) { return __ffma2_rn(make_float2(a, a), b, c); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

// 16 channels of a cell as pairs
struct Raw16 { // as they are in memory
    uint4 a, b;
};
__device__ __forceinline__ Raw16 load_raw(const uint16_t *p)
{
    const uint4 *s = reinterpret_cast<const uint4 *>(p);
    return {__ldg(s), __ldg(s + 1)};
}
__device__ __forceinline__ void unpack_raw(const Raw16 &r, float2 (&v)[8])
{
    const uint32_t w[8] = {r.a.x, r.a.y, r.a.z, r.a.w, r.b.x, r.b.y, r.b.z, r.b.w};
#pragma unroll
    for (int j = 0; j < 8; ++j)
        v[j] = make_float2(__uint_as_float(w[j] << 16), __uint_as_float(w[j] & 0xFFFF0000u));
}
__device__ __forceinline__ void unpack16(const uint16_t *p, float2 (&v)[8]) { unpack_raw(load_raw(p), v); }
// 16 weights of a tap from shared memory, as pairs
__device__ __forceinline__ void weights16(const float *w, float2 (&v)[8])
{
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float4 q = *reinterpret_cast<const float4 *>(w + 4 * j);
        v[2 * j] = make_float2(q.x, q.y);
        v[2 * j + 1] = make_float2(q.z, q.w);
    }
}
__device__ __forceinline__ void store16(uint16_t *p, const uint32_t (&h)[8])
{
    uint4 *dst = reinterpret_cast<uint4 *>(p);
    dst[0] = make_uint4(h[0], h[1], h[2], h[3]);
    dst[1] = make_uint4(h[4], h[5], h[6], h[7]);
}

// layer 1 forward: x [B][2][S^3] FP32 -> h1 [B][(S-2)^3][16] BF16, ReLU.  A
// thread computes 4 cells of a row: per (dy, dz) it holds the row's 6 inputs of
// both channels and takes the three taps in order (the same order of
// summation as cell by cell).
__global__ void __launch_bounds__(128) l1_fwd_cl(const float *__restrict__ x, const float *__restrict__ W1,
                                                  uint16_t *__restrict__ h1, int B, int S)
{
    __shared__ __align__(16) float sw[27 * 2 * 16];
    for (int i = threadIdx.x; i < 27 * 32; i += blockDim.x) sw[i] = W1[i];
    __syncthreads();
    const int So = S - 2, quads = (So + 3) / 4;
    const int64_t per = (int64_t)So * So * So, s3 = (int64_t)S * S * S;
    const uint32_t rows = (uint32_t)(B * So * So), total = rows * (uint32_t)quads;
    const bool vec = S % 4 == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0; // rows of x are 16-byte aligned
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const uint32_t row = t / (uint32_t)quads, xx = 4 * (t - row * quads), zb = row / (uint32_t)So, yy = row - zb * So,
                       b = zb / (uint32_t)So, zz = zb - b * So;
        const float *x0 = x + (int64_t)b * 2 * s3 + xx + (int64_t)S * (yy + (int64_t)S * zz);
        float2 acc[4][8];
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int o = 0; o < 8; ++o) acc[c][o] = make_float2(0.f, 0.f);
#pragma unroll 1
        for (int r = 0; r < 9; ++r) {
            const float *p = x0 + (int64_t)S * (r % 3 + (int64_t)S * (r / 3));
            float v[2][6];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const float *q = p + i * s3;
                if (vec) {
                    // positions 4 and 5 belong to no valid cell at a row's end
                    const float4 a = __ldg(reinterpret_cast<const float4 *>(q));
                    const float2 e = __ldg(reinterpret_cast<const float2 *>((int)xx + 5 < S ? q + 4 : q));
                    v[i][0] = a.x;
                    v[i][1] = a.y;
                    v[i][2] = a.z;
                    v[i][3] = a.w;
                    v[i][4] = e.x;
                    v[i][5] = e.y;
                } else {
#pragma unroll
                    for (int k = 0; k < 6; ++k) v[i][k] = (int)xx + k < S ? __ldg(q + k) : 0.f;
                }
            }
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                float2 w0[8], w1[8];
                weights16(sw + (3 * r + dx) * 32, w0);
                weights16(sw + (3 * r + dx) * 32 + 16, w1);
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int o = 0; o < 8; ++o) acc[c][o] = fma2(v[0][c + dx], w0[o], fma2(v[1][c + dx], w1[o], acc[c][o]));
            }
        }
        uint16_t *dst = h1 + ((int64_t)b * per + xx + (int64_t)So * (yy + (int64_t)So * zz)) * 16;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            if ((int)xx + c >= So) break;
            uint32_t h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                h[j] = (uint32_t)bf16_bits(fmaxf(acc[c][j].x, 0.f)) | ((uint32_t)bf16_bits(fmaxf(acc[c][j].y, 0.f)) << 16);
            store16(dst + 16 * c, h);
        }
    }
}

// A thread's run of ZT cells along z of a cube of side So (lanes along x):
// item t -> patch b, (x, y), first z.
constexpr int ZT = 4;
struct ZRun {
    int b, x, y, z;
};
__device__ __forceinline__ ZRun z_run(uint32_t t, uint32_t So)
{
    const uint32_t nz = (So + ZT - 1) / ZT, xy = t / So, q = xy / So, b = q / nz;
    return {(int)b, (int)(t - xy * So), (int)(xy - q * So), (int)((q - b * nz) * ZT)};
}
__host__ __device__ inline uint32_t z_runs(int B, int So) { return (uint32_t)B * So * So * ((So + ZT - 1) / ZT); }

// The sums of the last layer's forward and of its data gradient come before
// a BF16 rounding (of gh2, and of what follows from it), where another order of
// summation moves a value by a whole BF16 step and the gradients by more than
// FP32 rounding.  Both keep the order of one cell at a time: taps dx, dy, dz,
// then channels, one chain of fused multiply-adds per result.

// layer 3 forward: h2 [B][S^3][16] BF16 -> y [B][(S-2)^3] FP32.  A CTA takes qx
// x yb threads' cells of one output plane, 4 cells of a row each, from a copy
// of the rows around them in shared memory: a cell is unpacked once per (dy,
// dz) for its three taps, a tap's weights serve 4 cells.  (Straight from global
// memory the threads' 128-byte steps along x cost a cache line per lane and
// load.)  16-byte chunks of a row lie 9 apart every 8, so that 8 lanes read from
// distinct banks.  The planes arrive one after the other (all at once: 73 us
// instead of 70).
constexpr int L3_NT = 128, L3_QX = 16; // threads; most quads of cells along x
struct L3Geo {
    int qx, yb;        // quads along x and rows of a CTA
    int bx, by;        // CTAs along x and y of a plane
    int pitch;         // 16-byte units of a staged row
    FastDiv dqx, drow; // qx, chunks of a full row
};
static L3Geo l3_geo(int So, size_t *smem)
{
    L3Geo g;
    const int quads = (So + 3) / 4;
    g.bx = (quads + L3_QX - 1) / L3_QX;
    g.qx = (quads + g.bx - 1) / g.bx;
    g.yb = std::min(So, L3_NT / g.qx);
    g.by = (So + g.yb - 1) / g.yb;
    g.yb = (So + g.by - 1) / g.by;
    g.pitch = 9 * g.qx + 8; // 9 qx + 4 used; the rest keeps the lanes' steps across rows
    g.dqx = FastDiv((uint32_t)g.qx);
    g.drow = FastDiv((uint32_t)(8 * g.qx + 4));
    *smem = (size_t)3 * (g.yb + 2) * g.pitch * 16;
    return g;
}
constexpr size_t L3_SMEM = (size_t)3 * (L3_NT / L3_QX + 2) * (9 * L3_QX + 8) * 16; // the largest: qx = L3_QX

__global__ void __launch_bounds__(L3_NT, 3) l3_fwd_cl(const uint16_t *__restrict__ h2, const float *__restrict__ W3,
                                                      float *__restrict__ y, int S, const __grid_constant__ L3Geo g)
{
    extern __shared__ __align__(16) uint4 rows[]; // [3 planes][yb + 2][pitch]
    __shared__ __align__(16) float sw[27 * 16];
    for (int i = threadIdx.x; i < 27 * 16; i += L3_NT) sw[i] = W3[i];
    const int So = S - 2;
    int u = blockIdx.x;
    const int x0 = 4 * g.qx * (u % g.bx);
    u /= g.bx;
    const int y0 = g.yb * (u % g.by);
    u /= g.by;
    const int b = u / So, z = u - b * So;
    const int nx = min(4 * g.qx + 2, S - x0), ny = min(g.yb, So - y0), sr = g.yb + 2;
    const uint4 *src = reinterpret_cast<const uint4 *>(h2) +
                       2 * (((int64_t)b * S + z) * S * S + (int64_t)S * y0 + x0);
    const int chunks = 8 * g.qx + 4;
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) {
        for (int t = threadIdx.x; t < (ny + 2) * chunks; t += L3_NT) {
            const int j = g.drow.div(t), ch = t - j * chunks;
            if (ch < 2 * nx) // past the cube's end: read by cells that are no output only
                cp16(rows + (pl * sr + j) * g.pitch + ch + (ch >> 3), src + 2 * (int64_t)S * (j + (int64_t)S * pl) + ch, 16u);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const int j = g.dqx.div(threadIdx.x), q = threadIdx.x - j * g.qx, xx = x0 + 4 * q;
    const bool ok = j < ny && xx < So;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int dz = 0; dz < 3; ++dz) {
        if (dz == 0) asm volatile("cp.async.wait_group 2;" ::: "memory");
        if (dz == 1) asm volatile("cp.async.wait_group 1;" ::: "memory");
        if (dz == 2) asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        if (!ok) continue;
#pragma unroll 1
        for (int dy = 0; dy < 3; ++dy) {
            const uint4 *p = rows + (dz * sr + j + dy) * g.pitch + 9 * q;
            float2 v[6][8];
#pragma unroll
            for (int k = 0; k < 6; ++k)
                unpack_raw({p[2 * k + (k >= 4)], p[2 * k + 1 + (k >= 4)]}, v[k]);
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) {
                float2 w[8];
                weights16(sw + (9 * dz + 3 * dy + dx) * 16, w);
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        acc[c] = fmaf(v[c + dx][i].y, w[i].y, fmaf(v[c + dx][i].x, w[i].x, acc[c]));
            }
        }
    }
    if (!ok) return;
    float *dst = y + (((int64_t)b * So + z) * So + y0 + j) * So + xx;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        if (xx + c < So) dst[c] = acc[c];
}

// layer 3 backward-data: gh2[c][ci] = (h2[c][ci] > 0) sum_e gc[c - 2 + e] W3[26 - e][ci]
// for c in S^3 (gc on (S-2)^3, zero outside); ZT cells along z per thread, which
// share a tap's weights
__global__ void __launch_bounds__(128) l3_bwd_data_cl(const float *__restrict__ gc, const float *__restrict__ W3,
                                                       const uint16_t *__restrict__ h2, uint16_t *__restrict__ gh2,
                                                       int B, int S)
{
    __shared__ __align__(16) float sw[27 * 16];
    for (int i = threadIdx.x; i < 27 * 16; i += blockDim.x) sw[i] = W3[i];
    __syncthreads();
    const int So = S - 2;
    const int64_t o2 = (int64_t)So * So, s2 = (int64_t)S * S;
    const uint32_t total = z_runs(B, S);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
        const ZRun q = z_run(t, (uint32_t)S);
        float2 acc[ZT][8];
#pragma unroll
        for (int c = 0; c < ZT; ++c)
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[c][i] = make_float2(0.f, 0.f);
        const int ox = q.x - 2, oy = q.y - 2;
        const bool okx[3] = {ox >= 0, (unsigned)(ox + 1) < (unsigned)So, ox + 2 < So};
#pragma unroll 1
        for (int ez = 0; ez < 3; ++ez) {
            const int oz = q.z - 2 + ez;
            bool okz[ZT];
#pragma unroll
            for (int c = 0; c < ZT; ++c) okz[c] = (unsigned)(oz + c) < (unsigned)So;
            const float *pz = gc + q.b * (o2 * So) + ox + (int64_t)So * oy + o2 * oz, *wz = sw + (26 - 9 * ez) * 16;
#pragma unroll 1
            for (int ey = 0; ey < 3; ++ey, pz += So, wz -= 3 * 16) {
                if ((unsigned)(oy + ey) >= (unsigned)So) continue;
                float g[3][ZT];
#pragma unroll
                for (int ex = 0; ex < 3; ++ex)
#pragma unroll
                    for (int c = 0; c < ZT; ++c) g[ex][c] = okx[ex] && okz[c] ? __ldg(pz + ex + c * o2) : 0.f;
#pragma unroll
                for (int ex = 0; ex < 3; ++ex) {
                    float2 w[8];
                    weights16(wz - ex * 16, w);
#pragma unroll
                    for (int c = 0; c < ZT; ++c)
#pragma unroll
                        for (int i = 0; i < 8; ++i) acc[c][i] = fma2(g[ex][c], w[i], acc[c][i]);
                }
            }
        }
        const int64_t e = (q.b * (s2 * S) + q.x + (int64_t)S * q.y + s2 * q.z) * 16;
#pragma unroll
        for (int c = 0; c < ZT; ++c) {
            if (q.z + c >= S) break;
            float2 m[8];
            unpack16(h2 + e + c * s2 * 16, m);
            uint32_t h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j)
                h[j] = (uint32_t)bf16_bits(m[j].x > 0.f ? acc[c][j].x : 0.f) |
                       ((uint32_t)bf16_bits(m[j].y > 0.f ? acc[c][j].y : 0.f) << 16);
            store16(gh2 + e + c * s2 * 16, h);
        }
    }
}

// Warp sums of v[0..16): the lanes halve the values they carry at each step
// (16 shuffles, not 80), and lane l ends with the sum of value l / 2.
__device__ __forceinline__ float warp_sum16(float (&v)[16])
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int n = 8; n > 0; n >>= 1) {
        const bool up = lane & (2 * n);
#pragma unroll
        for (int i = 0; i < n; ++i) {
            const float keep = up ? v[n + i] : v[i], send = up ? v[i] : v[n + i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * n);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

// The weight gradients of the first and last layers: blocks of 9 warps, warp w
// = taps (dx, dy) = (w % 3, w / 3) with all three dz.  The lanes of all 9 warps
// take the same 32 columns (patch b, x, y) of output cells and walk up runs of
// them, with the BF16 operand unpacked once per cell (the next planes in
// flight) and the other one in a window of three planes.  The shifted reads of
// the 9 warps hit L1.  Layer 1's two input channels are two blocks (its 96
// accumulators in one thread left one block per SM: 318 us).  The warps' sums
// go to FP32 atomics, 16 neighbouring words each: one word per lane and 5
// shuffles per value made them the end of every small batch (8 patches of
// 16^3, the whole step: 299 us, this way 252).
constexpr int WG_THREADS = 9 * 32;
// Resident per SM, planes in flight: the batch of 32 patches of 32^3 in all, us:
// 3 and 1 1011, 2 and 2 986, 2 and 3 1112 (spills); 3 with 4 planes in shared
// memory 991.
constexpr int WG_CTAS = 2;
constexpr int WG_AHEAD = 2;

struct WgItem {
    int b, x, y, z0, z1;
    bool ok;
};
// item k of `runs` runs of a column group: 32 consecutive columns of patch-major (b, y, x)
__device__ __forceinline__ WgItem wg_item(int item, int runs, int run, int columns, int So)
{
    const int group = item / runs, k = item - group * runs, col = group * 32 + (threadIdx.x & 31);
    WgItem w;
    w.ok = col < columns;
    const int c = w.ok ? col : 0, yb = c / So;
    w.x = c - yb * So;
    w.b = yb / So;
    w.y = yb - w.b * So;
    w.z0 = k * run;
    w.z1 = min(So, w.z0 + run);
    return w;
}
// the block's sums of the three dz taps' 16 values into dst[tap stride][16]
__device__ __forceinline__ void wg_add(float2 (&acc)[3][8], float *dst, int tap_stride)
{
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        float a[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            a[2 * i] = acc[d][i].x;
            a[2 * i + 1] = acc[d][i].y;
        }
        const float sum = warp_sum16(a);
        if ((threadIdx.x & 1) == 0) atomicAdd(dst + 9 * d * tap_stride + ((threadIdx.x & 31) >> 1), sum);
    }
}

// layer 3: gW3[t][ci] += sum_q h2[q + d(t)][ci] gc[q], q in (S-2)^3, h2 side S
__global__ void __launch_bounds__(WG_THREADS, WG_CTAS)
    l3_wgrad_cl(const uint16_t *__restrict__ h2, const float *__restrict__ gc, float *__restrict__ gW3, int B, int S,
                int run)
{
    const int w = threadIdx.x >> 5, dx = w % 3, dy = w / 3;
    const int So = S - 2, columns = B * So * So, runs = (So + run - 1) / run, items = (columns + 31) / 32 * runs;
    const int64_t s2 = (int64_t)S * S, s3 = s2 * S, o2 = (int64_t)So * So;
    float2 acc[3][8];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[d][i] = make_float2(0.f, 0.f);
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const WgItem q = wg_item(item, runs, run, columns, So);
        const uint16_t *hp = h2 + (q.b * s3 + q.x + dx + (int64_t)S * (q.y + dy) + s2 * q.z0) * 16;
        const float *gp = gc + q.b * (o2 * So) + q.x + (int64_t)So * q.y + o2 * q.z0;
        const int nz = q.z1 - q.z0, planes = nz + 2;
        Raw16 hb[WG_AHEAD]; // the next planes of h2 and of gc (0 past the run and for lanes without a column)
        float gb[WG_AHEAD];
#pragma unroll
        for (int k = 0; k < WG_AHEAD; ++k) {
            if (k < planes) hb[k] = load_raw(hp + k * s2 * 16);
            gb[k] = q.ok && k < nz ? __ldg(gp + k * o2) : 0.f;
        }
        hp += WG_AHEAD * s2 * 16;
        gp += WG_AHEAD * o2;
        float g1 = 0.f, g2 = 0.f; // gc at planes z - 1, z - 2
        for (int z = 0; z < planes; z += WG_AHEAD) {
#pragma unroll
            for (int k = 0; k < WG_AHEAD; ++k) {
                if (z + k >= planes) break;
                float2 v[8];
                unpack_raw(hb[k], v); // plane z of h2: dz 0 of cell z, 1 of z - 1, 2 of z - 2
                const float g0 = gb[k];
                if (z + k + WG_AHEAD < planes) hb[k] = load_raw(hp);
                gb[k] = q.ok && z + k + WG_AHEAD < nz ? __ldg(gp) : 0.f;
                hp += s2 * 16;
                gp += o2;
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    acc[0][i] = fma2(g0, v[i], acc[0][i]);
                    acc[1][i] = fma2(g1, v[i], acc[1][i]);
                    acc[2][i] = fma2(g2, v[i], acc[2][i]);
                }
                g2 = g1;
                g1 = g0;
            }
        }
    }
    wg_add(acc, gW3 + w * 16, 16);
}

// layer 1, input channel blockIdx.y: gW1[t][i][o] += sum_q x[i][q + d(t)] gh1[q][o],
// q in (S-2)^3, x side S
__global__ void __launch_bounds__(WG_THREADS, WG_CTAS)
    l1_wgrad_cl(const float *__restrict__ x, const uint16_t *__restrict__ gh1, float *__restrict__ gW1, int B, int S,
                int run)
{
    const int w = threadIdx.x >> 5, dx = w % 3, dy = w / 3, i = blockIdx.y;
    const int So = S - 2, columns = B * So * So, runs = (So + run - 1) / run, items = (columns + 31) / 32 * runs;
    const int64_t s2 = (int64_t)S * S, s3 = s2 * S, o2 = (int64_t)So * So;
    float2 acc[3][8];
#pragma unroll
    for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int o = 0; o < 8; ++o) acc[d][o] = make_float2(0.f, 0.f);
    for (int item = blockIdx.x; item < items; item += gridDim.x) {
        const WgItem q = wg_item(item, runs, run, columns, So);
        const float *xp = x + (2 * q.b + i) * s3 + q.x + dx + (int64_t)S * (q.y + dy) + s2 * q.z0;
        const uint16_t *gp = gh1 + (q.b * (o2 * So) + q.x + (int64_t)So * q.y + o2 * q.z0) * 16;
        const int nz = q.z1 - q.z0;
        // x at planes z, z + 1 (0 for lanes without a column), and the next planes of gh1 and x
        float v0 = q.ok ? __ldg(xp) : 0.f, v1 = q.ok ? __ldg(xp + s2) : 0.f;
        Raw16 gb[WG_AHEAD];
        float vb[WG_AHEAD];
        xp += 2 * s2;
#pragma unroll
        for (int k = 0; k < WG_AHEAD; ++k) {
            if (k >= nz) break;
            gb[k] = load_raw(gp + k * o2 * 16);
            vb[k] = q.ok ? __ldg(xp + k * s2) : 0.f;
        }
        gp += WG_AHEAD * o2 * 16;
        xp += WG_AHEAD * s2;
        for (int z = 0; z < nz; z += WG_AHEAD) {
#pragma unroll
            for (int k = 0; k < WG_AHEAD; ++k) {
                if (z + k >= nz) break;
                float2 g[8];
                unpack_raw(gb[k], g);
                const float v2 = vb[k];
                if (z + k + WG_AHEAD < nz) {
                    gb[k] = load_raw(gp);
                    vb[k] = q.ok ? __ldg(xp) : 0.f;
                }
                gp += o2 * 16;
                xp += s2;
#pragma unroll
                for (int o = 0; o < 8; ++o) {
                    acc[0][o] = fma2(v0, g[o], acc[0][o]);
                    acc[1][o] = fma2(v1, g[o], acc[1][o]);
                    acc[2][o] = fma2(v2, g[o], acc[2][o]);
                }
                v0 = v1;
                v1 = v2;
            }
        }
    }
    wg_add(acc, gW1 + w * 32 + 16 * i, 32);
}

static unsigned grid_of(int64_t n, int threads, int64_t cap)
{
    int64_t b = (n + threads - 1) / threads;
    if (b > cap) b = cap;
    return (unsigned)(b < 1 ? 1 : b);
}

// Run length and CTAs of a first/last-layer weight gradient over output cubes
// of side So: whole columns where there is a group of 32 for every CTA, else
// runs short enough for that, of 4 cells at least (a run re-reads two planes).
static unsigned wg_launch(int B, int So, int ctas, int &run)
{
    const int64_t groups = ((int64_t)B * So * So + 31) / 32;
    const int64_t runs = (ctas + groups - 1) / groups;
    run = (int)((So + runs - 1) / runs);
    if (run < 4) run = 4;
    const int64_t items = groups * ((So + run - 1) / run);
    return (unsigned)(items < ctas ? items : ctas);
}

static DeviceOnce wgrad_once, brick_once[2], l3_once;

// weight gradient: persistent CTAs, two per SM
static cn_status launch_wgrad(Args &a, int B, int sms, cudaStream_t st)
{
    cn_status s = smem_opt_in(wgrad_once, wgrad_tc_kernel, WGT_SMEM);
    if (s != CN_OK) return s;
    size_t smem = 0;
    const WgGeo g = wgrad_geo(B, a.Sout, 2 * sms, &smem);
    wgrad_tc_kernel<<<(unsigned)std::min(g.total, 2 * sms), WGT_NT, smem, st>>>(a, g);
    CN_CUDA_TRY(cudaGetLastError());
    return CN_OK;
}

// forward / backward-data: one CTA per brick
template <int MODE>
static cn_status launch_conv(Args &a, int B, cudaStream_t st)
{
    BrickGeo g;
    if (!brick_geo(a.Sout, g)) return fail(CN_ERR_INVALID_ARGUMENT, "learned smoother training: empty patch");
    const size_t smem = 2 * (size_t)g.SROWS * 16 + WBYTES + 16;
    // one opt-in per device, at the largest brick any patch size can take
    constexpr size_t smem_max = 2 * (size_t)BRICK_MAX_ROWS * 16 + WBYTES + 16;
    cn_status s = smem_opt_in(brick_once[MODE], brick_tc_kernel<MODE>, smem_max);
    if (s != CN_OK) return s;
    const int64_t ctas = (int64_t)B * g.bricks[0] * g.bricks[1] * g.bricks[2];
    brick_tc_kernel<MODE><<<(unsigned)ctas, BRICK_NT, smem, st>>>(a, g);
    CN_CUDA_TRY(cudaGetLastError());
    return CN_OK;
}

} // namespace nntr

namespace nntc {

cn_status train_forward_tc(const TrainBufs &T, const float *x, const float *W, int B, int P, cudaStream_t st)
{
    using namespace nntr;
    const int S = P + 8, S1 = S - 2, S2 = S - 4, S3 = S - 6;
    const float *W1 = W, *W2 = W + 27 * 2 * 16, *W3 = W + 27 * 2 * 16 + 27 * 16 * 16;
    if ((int64_t)B * S * S * S >= (int64_t)1 << 31)
        return fail(CN_ERR_UNSUPPORTED, "learned smoother training: batch too large for 32-bit cell indices");
    cn_status s;
    // packed B tiles of the hidden layer: forward, backward-data
    if ((s = pack_weights(W2, 16, 16, T.wfwd, st)) != CN_OK) return s;
    pack_bwd_kernel<<<27, 256, 0, st>>>(W2, T.wbwd);
    l1_fwd_cl<<<grid_of((int64_t)B * S1 * S1 * ((S1 + 3) / 4), 128, 148 * 64), 128, 0, st>>>(x, W1, T.h1, B, S);
    CN_CUDA_TRY(cudaGetLastError());
    Args a = {};
    a.src = T.h1;
    a.w = T.wfwd;
    a.out = T.h2;
    a.Sin = S1;
    a.Sout = S2;
    a.shift = 0;
    a.relu = 1;
    a.err = T.err;
    if ((s = launch_conv<FWD>(a, B, st)) != CN_OK) return s;
    size_t smem = 0;
    const L3Geo g = l3_geo(S3, &smem);
    if ((s = smem_opt_in(l3_once, l3_fwd_cl, L3_SMEM)) != CN_OK) return s;
    l3_fwd_cl<<<(unsigned)((int64_t)B * S3 * g.by * g.bx), L3_NT, smem, st>>>(T.h2, W3, T.y, S2, g);
    CN_CUDA_TRY(cudaGetLastError());
    return CN_OK;
}

cn_status train_backward_tc(const TrainBufs &T, const float *x, const float *W, float *gW, int B, int P,
                            cudaStream_t st)
{
    using namespace nntr;
    const int S = P + 8, S1 = S - 2, S2 = S - 4, S3 = S - 6;
    const float *W3 = W + 27 * 2 * 16 + 27 * 16 * 16;
    float *gW1 = gW, *gW2 = gW + 27 * 2 * 16, *gW3 = gW + 27 * 2 * 16 + 27 * 16 * 16;
    cn_status s;
    CN_CUDA_TRY(cudaMemsetAsync(gW, 0, sizeof(float) * (27 * 2 * 16 + 27 * 16 * 16 + 27 * 16), st));
    int dev = 0, sms = 148;
    CN_CUDA_TRY(cudaGetDevice(&dev));
    CN_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    int run = 0;
    unsigned ctas = wg_launch(B, S3, WG_CTAS * sms, run);
    l3_wgrad_cl<<<ctas, WG_THREADS, 0, st>>>(T.h2, T.gc, gW3, B, S2, run);
    l3_bwd_data_cl<<<grid_of(z_runs(B, S2), 128, 148 * 64), 128, 0, st>>>(T.gc, W3, T.h2, T.gh2, B, S2);
    CN_CUDA_TRY(cudaGetLastError());
    Args w = {};
    w.src = T.h1;
    w.gout = T.gh2;
    w.gw = gW2;
    w.Sin = S1;
    w.Sout = S2;
    w.shift = 0;
    w.err = T.err;
    if ((s = launch_wgrad(w, B, sms, st)) != CN_OK) return s;
    Args d = {};
    d.src = T.gh2;
    d.act = T.h1;
    d.w = T.wbwd;
    d.out = T.gh1;
    d.Sin = S2;
    d.Sout = S1;
    d.shift = -2;
    d.err = T.err;
    if ((s = launch_conv<BWD>(d, B, st)) != CN_OK) return s;
    ctas = wg_launch(B, S1, WG_CTAS * sms / 2, run);
    l1_wgrad_cl<<<dim3(ctas, 2), WG_THREADS, 0, st>>>(x, T.gh1, gW1, B, S, run);
    CN_CUDA_TRY(cudaGetLastError());
    return CN_OK;
}

} // namespace nntc
} // namespace cn
