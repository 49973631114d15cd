// euler_stage.cuh -- the fused lab + WENO5-JS + Rusanov + flux-divergence +
// SSP-RK3 stage computation of one 8x8x8 tile, shared by the uniform-grid
// kernel (euler.cu) and the AMR block kernel (amr.cu).  Where the tile comes
// from and how its halo cells arrive differs: a uniform grid's tile (CartSrc)
// takes them as TMA boxes, and by a rule per face where the face carries a BC or
// a skipped neighbour (what FieldLab's lab holds there); an AMR block's by
// asynchronous copies and its own interface ghost fill (the policy `Src`).
#pragma once

#include "cn_fastdiv.h"
#include "cn_internal.h"
#include "cn_tma.cuh"
#include "euler_math.cuh"

#include <cuda.h>

namespace cn {
namespace euler {

constexpr int TB = 8;                 // tile edge
constexpr int G = 3;                  // ghost width
constexpr int NCORE = TB * TB * TB;   // tile cells: 512
constexpr int NLINE = TB * TB;        // lines along one direction: 64
constexpr int NHALO = 2 * G * NLINE;  // one direction's halo slabs: 384
constexpr int NSIDES = 24;            // quarters (4 x 4 cells) of a tile's six sides
// Shared-memory entry of core cell (x, y, z): a permutation of the dense
// index without padding, e = (x ^ y) + 8 (y ^ z) + 64 z.  For lines along
// any direction the 16 (FP64, FP32 pairs) or 32 (FP32) lines that one
// wavefront touches at the same position fall in distinct banks.  Along a
// line the entry of its cell a is the entry of cell 0 XOR a * m with
// m = 1, 9, 72 for x, y, z.
__device__ __forceinline__ int core_sm(int x, int y, int z) { return (x ^ y) + 8 * (y ^ z) + 64 * z; }
__device__ __forceinline__ int core_sm(int i) { return i ^ ((i >> 3) & 7) ^ ((i >> 3) & 56); }
// Halo slot of a direction, slab coordinate h = 0..5 (cells -3..-1 and 8..10)
// of line l: x and z at 64 h + l, y at 192 (h / 3) + 8 (h % 3) + x + 24 z,
// the order in which a TMA box [z][y][x] of a side lands.  Both are free of
// bank conflicts.
//
// FP64 keeps two slots (three CTAs per SM): while the sweep of one direction
// runs, the next direction's halo cells arrive in the other slot by
// asynchronous copies.  FP32 has room for all three and loads them at once.
template <typename T> struct Stg {
    static constexpr bool all = sizeof(T) == 4;
    static constexpr int SV = NCORE + (all ? 3 : 2) * NHALO; // shared entries per variable
    // first entry of direction D's halo slot
    static __device__ __forceinline__ int slot(int D) { return NCORE + (all ? D : (D & 1)) * NHALO; }
};
// Where primitive variable c of shared entry e (core cell or halo-slot cell)
// lives.  FP64: one array per variable, [5][SV].  FP32: variables (0, 1) and
// (2, 3) interleaved as pairs, so that one 64-bit shared access and one
// packed FP32x2 instruction serve two variables, and variable 4 alone:
// [pairs (0,1): 2 SV][pairs (2,3): 2 SV][variable 4: SV].
__device__ __forceinline__ double &prim(double *W, int c, int e) { return W[c * Stg<double>::SV + e]; }
__device__ __forceinline__ float &prim(float *W, int c, int e)
{
    constexpr int SV = Stg<float>::SV;
    return c < 2 ? W[2 * e + c] : (c < 4 ? W[2 * SV + 2 * e + (c - 2)] : W[4 * SV + e]);
}
constexpr int NCELL = TB * TB * TB;   // 512
constexpr int NACC = NCORE;           // the cells' flux-difference accumulators, per variable
constexpr int NT = 192;               // threads per CTA: 64 lines x 3 runs of 3 faces
constexpr int CPT = (NCELL + NT - 1) / NT; // cells per thread: 3

template <typename T> struct StageParams {
    const T *U[5];   // state whose lab is loaded (component bases)
    const T *Un[5];  // U^n (stages 2 and 3)
    T *out[5];
    T dt;
    T gamma, gm1, igm1;
    // out = cn Un + cs (ku U + dt L(U)): SSP-RK3 stage 1 (cn 0, cs 1), 2 (3/4,
    // 1/4), 3 (1/3, 2/3), or L(U) itself (ku 0, dt 1); Un is read if use_un
    T cn, cs;
    int use_u, use_un;
    double *partials; // per-tile FP64 sums of the 5 outputs (may be null)
    int *err;
};

// One tile of work: its block, tile origin, block extents and storage.
template <typename T> struct TileInfo {
    int block;
    int x0, y0, z0;
    int N0, N1, N2;
    int64_t boff;     // element offset of the block in each component
    T ih[3];          // 1/h of the block
    int bx, by, bz;   // block coordinates (uniform grid)
};

// Tensor maps of a state as [component][block][z][y][x]: boxes of a tile's
// cells (8 x 8 x 8, all components) and of its sides (x: 4 x 8 x 8, y: 8 x 3 x 8,
// z: 8 x 8 x 3; one component in FP64, all five in FP32).
struct TileMaps {
    CUtensorMap core, hx, hy, hz;
};

// Uniform Cartesian grid: tiles in block order; which sides of a tile are boxes
// of one block's cells, from each component's BC tables.
struct CartSrc {
    LabGeom L;
    BcView bc[5];
    double ih[3];
    FastDiv tiles, tx, ty, nbx, nby; // tiles per block and along x, y; blocks along x, y
    template <typename T> __device__ __forceinline__ void tile(int item, TileInfo<T> &t) const
    {
        t.block = tiles.div(item);
        const int r = item - t.block * (int)tiles.d, q = tx.div(r), z = ty.div(q);
        t.x0 = (r - q * (int)tx.d) * 8;
        t.y0 = (q - z * (int)ty.d) * 8;
        t.z0 = z * 8;
        t.N0 = L.n[0];
        t.N1 = L.n[1];
        t.N2 = L.n[2];
        t.boff = (int64_t)t.block * L.bstride;
        t.ih[0] = (T)ih[0];
        t.ih[1] = (T)ih[1];
        t.ih[2] = (T)ih[2];
        const int b = nbx.div(t.block);
        t.bx = t.block - b * (int)nbx.d;
        t.bz = nby.div(b);
        t.by = b - t.bz * (int)nby.d;
    }
    // By the lanes of one warp: bit 2 d + s of the result is set when side
    // (d, s) of the tile lies outside its block and is not a plain copy of the
    // neighbour block's cells in all five components, as in a lab: no
    // component's block carries a BC or skip flag (mode byte 0), or the face
    // carries no BC other than Base and no skip flag in any component
    // (BcView::faces).
    template <typename T> __device__ __forceinline__ unsigned slow_sides(const TileInfo<T> &t) const
    {
        const int lane = threadIdx.x & 31, c = lane < 5 ? lane : 0;
        const unsigned mode = __ldg(bc[c].mode + t.block);
        const unsigned faces = __reduce_or_sync(0xffffffffu, (unsigned)__ldg(bc[c].faces + t.block));
        const unsigned any = __reduce_or_sync(0xffffffffu, mode);
        const unsigned outside = (t.x0 == 0 ? 1u : 0u) | (t.x0 + TB == t.N0 ? 2u : 0u) | (t.y0 == 0 ? 4u : 0u) |
                                 (t.y0 + TB == t.N1 ? 8u : 0u) | (t.z0 == 0 ? 16u : 0u) |
                                 (t.z0 + TB == t.N2 ? 32u : 0u);
        return any ? (outside & faces) : 0u;
    }
    // block that holds side (d, s) of the tile when it is plain
    template <typename T> __device__ __forceinline__ int side_block(const TileInfo<T> &t, int d, int s) const
    {
        const int n = d == 0 ? t.N0 : (d == 1 ? t.N1 : t.N2), o = d == 0 ? t.x0 : (d == 1 ? t.y0 : t.z0);
        if (s ? o + TB < n : o > 0) return t.block;
        const int b = d == 0 ? t.bx : (d == 1 ? t.by : t.bz), m = L.nb[d];
        const int q = s ? (b + 1 < m ? b + 1 : 0) : (b > 0 ? b - 1 : m - 1);
        return t.block + (q - b) * (d == 0 ? 1 : (d == 1 ? L.nb[0] : L.nb[0] * L.nb[1]));
    }
};

// The direction is a runtime (warp-uniform) value: one copy of the face code
// serves all three sweeps, which keeps the kernel's hot code small enough for
// the instruction caches.

// Halo cell i (0..383) of direction D: tile-local coordinates and entry in the
// direction's slot.  Lanes walk x first, so that the global accesses of a
// warp cover whole rows.
__device__ __forceinline__ void halo_cell(int D, int i, int &x, int &y, int &z, int &e)
{
    int h;
    if (D == 0) {
        h = i % (2 * G);
        y = (i / (2 * G)) % TB;
        z = i / (2 * G * TB);
        x = h < G ? h - G : h - G + TB;
        e = 64 * h + y + 8 * z;
    } else if (D == 1) {
        x = i % TB;
        h = (i / TB) % G;
        z = (i / (TB * G)) % TB;
        const int side = i / (TB * G * TB);
        y = h - G + side * (TB + G);
        e = i;
    } else {
        x = i % TB;
        y = (i / TB) % TB;
        h = i / (TB * TB);
        z = h < G ? h - G : h - G + TB;
        e = i;
    }
}

__device__ __forceinline__ void cp_async(double *dst, const double *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async(float *dst, const float *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits until at most N of the thread's newest copy groups are in flight
template <int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// Left- and right-biased states of the run's three faces, all five variables;
// at[0..7]: shared entries of the run's 8 cells.  FP32 takes the variables
// (0, 1) and (2, 3) as pairs and variable 4 alone.
template <typename V>
__device__ __forceinline__ void load_run(const V *P, const int (&at)[8], V (&u)[8])
{
#pragma unroll
    for (int k = 0; k < 8; ++k)
        u[k] = P[at[k]];
}
template <bool SCALED>
__device__ __forceinline__ void run_states(const double *W, const int (&at)[8], double (&WL)[3][5],
                                           double (&WR)[3][5])
{
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        double u[8], l[3], r[3];
        load_run(W + c * Stg<double>::SV, at, u);
        weno5_run<SCALED>(u, l, r);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            WL[i][c] = l[i];
            WR[i][c] = r[i];
        }
    }
}
template <bool SCALED>
__device__ __forceinline__ void run_states(const float *W, const int (&at)[8], float (&WL)[3][5], float (&WR)[3][5])
{
    constexpr int SV = Stg<float>::SV;
#pragma unroll
    for (int c = 0; c < 4; c += 2) {
        float2 u[8], l[3], r[3];
        load_run(reinterpret_cast<const float2 *>(W + c * SV), at, u);
        weno5_run<SCALED>(u, l, r);
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            WL[i][c] = l[i].x;
            WL[i][c + 1] = l[i].y;
            WR[i][c] = r[i].x;
            WR[i][c + 1] = r[i].y;
        }
    }
    float u[8], l[3], r[3];
    load_run(W + 4 * SV, at, u);
    weno5_run<SCALED>(u, l, r);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        WL[i][4] = l[i];
        WR[i][4] = r[i];
    }
}

// Face fluxes of direction D for the whole tile, differenced into the
// per-cell accumulators A (shared memory, [5][NACC], entries core_sm).  Each
// of the tile's 64 lines along D has 9 faces (face a between cells a-1 and
// a); thread t takes the run of faces 3r .. 3r+2, r = t / 64, of line t % 64:
// it loads the run's 8 cells of one variable after the other, forms the
// states of the three faces (weno5_run) and then the fluxes.  Run r completes
// cells 3r and 3r+1 by itself.  Cells 2 and 5 lie between runs: run 0 leaves
// its last flux and run 2 its first one in halo-slot entries that only they
// themselves read (cells -3 and 10 of the line), and after a barrier run 1,
// which has kept its own first and last flux, completes both cells.  The
// caller synchronises before A or the slot is used again.
template <typename T, bool SCALED>
__device__ __forceinline__ void sweep(int D, T *__restrict__ W, T *__restrict__ A, T gamma, T igm1, T ihd)
{
    const int run = threadIdx.x >> 6, line = threadIdx.x & 63;
    const int l0 = line & 7, l1 = line >> 3;
    const int x = D == 0 ? 0 : l0, y = D == 1 ? 0 : (D == 0 ? l0 : l1), z = D == 2 ? 0 : l1;
    const int c0 = core_sm(x, y, z);                      // the line's cell 0
    const int m = D == 0 ? 1 : (D == 1 ? 9 : 72);
    // the line's slab cell h = 0 and the stride along h within a side
    const int h0 = Stg<T>::slot(D) + (D == 1 ? l0 + 24 * l1 : line), hs = D == 1 ? 8 : 64;
    constexpr int HSIDE = G * NLINE;                      // entries of one side
    const int f0 = 3 * run;
    int at[8]; // shared entries of the run's cells f0-3 .. f0+4
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int a = f0 - 3 + k;
        at[k] = (unsigned)a < (unsigned)TB ? (c0 ^ (a * m)) : (a < 0 ? h0 + hs * (a + G) : h0 + HSIDE + hs * (a - TB));
    }
    T WL[3][5], WR[3][5];
    run_states<SCALED>(W, at, WL, WR);
    T Ff[5], Fq[5]; // the run's first flux and the previous face's
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        T Fl[5];
        rusanov<T>(WL[i], WR[i], D, gamma, igm1, Fl);
        if (i == 0) {
#pragma unroll
            for (int c = 0; c < 5; ++c)
                Ff[c] = Fl[c];
            if (run == 2) {
#pragma unroll
                for (int c = 0; c < 5; ++c)
                    prim(W, c, h0 + HSIDE + 2 * hs) = Fl[c];
            }
        } else {
            // cell f0+i-1 is complete: its faces' fluxes are Fq and Fl
            const int e = at[i + 2];
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const T df = Fl[c] - Fq[c];
                A[c * NACC + e] = D == 0 ? df * ihd : dfma(df, ihd, A[c * NACC + e]);
            }
        }
#pragma unroll
        for (int c = 0; c < 5; ++c)
            Fq[c] = Fl[c];
    }
    if (run == 0) {
#pragma unroll
        for (int c = 0; c < 5; ++c)
            prim(W, c, h0) = Fq[c];
    }
    __syncthreads(); // the exchanged fluxes
    if (run == 1) {
        const int e2 = at[2], e5 = at[5]; // cells 2 and 5
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const T d2 = Ff[c] - prim(W, c, h0), d5 = prim(W, c, h0 + HSIDE + 2 * hs) - Fq[c];
            A[c * NACC + e2] = D == 0 ? d2 * ihd : dfma(d2, ihd, A[c * NACC + e2]);
            A[c * NACC + e5] = D == 0 ? d5 * ihd : dfma(d5, ihd, A[c * NACC + e5]);
        }
    }
}

// Starts the copies of direction D's two 3-cell halo slabs into its slot as
// conservative values, cell by cell: plain copies of a cell asynchronously, the
// others resolved by the source policy, all five components at once, and
// stored.  The caller commits the group.
template <typename T, typename Src>
__device__ __forceinline__ void issue_halo(int D, const StageParams<T> &p, const Src &src, const TileInfo<T> &t,
                                           const typename Src::Side *sides, T *W)
{
    static_assert(NHALO % NT == 0, "whole halo cells per thread");
#pragma unroll
    for (int j = 0; j < NHALO / NT; ++j) {
        int x, y, z, e;
        halo_cell(D, threadIdx.x + j * NT, x, y, z, e);
        e += Stg<T>::slot(D);
        // the quarter of the side the cell lies in: the other two axes, in order
        const int q = D == 0 ? x : (D == 1 ? y : z), a = D == 0 ? y : x, b = D == 2 ? y : z;
        const typename Src::Side &S = sides[8 * D + 4 * (q > 0) + (a >> 2) + 2 * (b >> 2)];
        const int gx = t.x0 + x, gy = t.y0 + y, gz = t.z0 + z;
        if (S.plain()) {
            const int64_t o = S.offset(gx, gy, gz);
#pragma unroll
            for (int c = 0; c < 5; ++c)
                cp_async(&prim(W, c, e), p.U[c] + o);
        } else {
            T v[5];
            src.halo5(p.U, S, gx, gy, gz, v);
#pragma unroll
            for (int c = 0; c < 5; ++c)
                prim(W, c, e) = v[c];
        }
    }
}

// Conversion to primitives, in place, of the thread's halo cells of
// direction D (those it brought itself, or by TMA).
template <typename T> __device__ __forceinline__ void convert_halo(int D, T gm1, T *W, T &vmax)
{
#pragma unroll
    for (int j = 0; j < NHALO / NT; ++j) {
        int x, y, z, e;
        halo_cell(D, threadIdx.x + j * NT, x, y, z, e);
        e += Stg<T>::slot(D);
        T u[5], w[5];
#pragma unroll
        for (int c = 0; c < 5; ++c)
            u[c] = prim(W, c, e);
        to_primitive<T>(u[0], u[1], u[2], u[3], u[4], gm1, w);
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            prim(W, c, e) = w[c];
            if constexpr (sizeof(T) == 4) vmax = fmaxf(vmax, fabsf(w[c]));
        }
    }
}
// ... and of conservative values in registers, into the core or a slot
template <typename T> __device__ __forceinline__ void store_primitive(const T (&u)[5], T gm1, T *W, int e, T &vmax)
{
    T w[5];
    to_primitive<T>(u[0], u[1], u[2], u[3], u[4], gm1, w);
#pragma unroll
    for (int c = 0; c < 5; ++c) {
        prim(W, c, e) = w[c];
        if constexpr (sizeof(T) == 4) vmax = fmaxf(vmax, fabsf(w[c]));
    }
}

// Sweep of direction D; the Rusanov fluxes are twice the flux: 1/(2h) (exact).
template <typename T, bool SCALED>
__device__ __forceinline__ void sweep_dir(int D, const StageParams<T> &p, const TileInfo<T> &t, T *W, T *A)
{
    const T ihd = T(0.5) * (D == 0 ? t.ih[0] : (D == 1 ? t.ih[1] : t.ih[2]));
    sweep<T, SCALED>(D, W, A, p.gamma, p.igm1, ihd);
}

// Core cells from A (dense, conservative) into W.
template <typename T> __device__ __forceinline__ void convert_core(const T *A, T gm1, T *W, T &vmax)
{
#pragma unroll
    for (int k = 0; k < CPT; ++k) {
        const int i = threadIdx.x + k * NT;
        if (i < NCORE) {
            T u[5];
#pragma unroll
            for (int c = 0; c < 5; ++c)
                u[c] = A[c * NCORE + i];
            store_primitive<T>(u, gm1, W, core_sm(i), vmax);
        }
    }
}

// FP32, everything staged: the three sweeps.  The tile's WENO5 weights skip the
// range rescaling when every staged primitive is within kUnscaledMax (same
// values, fewer instructions: see euler_math.cuh); vmax: the largest primitive
// magnitude the thread staged (NaN data gives NaN states on either form).
template <typename T>
__device__ __forceinline__ void sweeps_at_once(const StageParams<T> &p, const TileInfo<T> &t, T *W, T *A, T vmax)
{
    const bool scaled = __syncthreads_or(!(vmax <= T(kUnscaledMax))) != 0;
#pragma unroll 1
    for (int D = 0; D < 3; ++D) {
        if (scaled)
            sweep_dir<T, true>(D, p, t, W, A);
        else
            sweep_dir<T, false>(D, p, t, W, A);
        if (D < 2) __syncthreads();
    }
}

// Epilogue: RHS or SSP-RK3 stage, coalesced along x of the tile rows.  All of
// the thread's U_s and U^n are loaded before the barrier that completes A, so
// a tile waits for one memory latency: `out` may alias U^n (stage 3 updates
// U in place), but each (component, cell) is loaded and stored by the same
// thread.
template <typename T> struct Epilogue {
    T us[5][CPT], un[5][CPT];
    int64_t eo[CPT];
    __device__ __forceinline__ void load(const StageParams<T> &p, const TileInfo<T> &t)
    {
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int i = threadIdx.x + k * NT;
            const int x = i % TB, y = (i / TB) % TB, z = i / (TB * TB);
            eo[k] = t.boff + (t.x0 + x) + (int64_t)t.N0 * ((t.y0 + y) + (int64_t)t.N1 * (t.z0 + z));
            const bool ok = i < NCELL;
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                us[c][k] = (p.use_u && ok) ? p.U[c][eo[k]] : T(0);
                un[c][k] = (p.use_un && ok) ? p.Un[c][eo[k]] : T(0);
            }
        }
    }
    // the new values, and the FP64 sums of the tile to p.partials[slot] if
    // requested (red: [NT/32][5], shared)
    __device__ __forceinline__ void store(const StageParams<T> &p, const T *A, double (*red)[5], int slot)
    {
        double sums[5] = {0, 0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < CPT; ++k) {
            const int i = threadIdx.x + k * NT;
            if (i < NCELL) {
                const int e = core_sm(i);
#pragma unroll
                for (int c = 0; c < 5; ++c) {
                    const T v = dfma(p.cn, un[c][k], p.cs * dfma(p.dt, -A[c * NACC + e], us[c][k]));
                    p.out[c][eo[k]] = v;
                    sums[c] += (double)v;
                }
            }
        }
        if (p.partials) {
            const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                double s = sums[c];
#pragma unroll
                for (int off = 16; off > 0; off >>= 1)
                    s += __shfl_down_sync(0xffffffffu, s, off);
                if (lane == 0)
                    red[warp][c] = s;
            }
            __syncthreads();
            if (threadIdx.x < 5) {
                double s = 0;
                for (int w = 0; w < NT / 32; ++w)
                    s += red[w][threadIdx.x];
                p.partials[(int64_t)slot * 5 + threadIdx.x] = s;
            }
        }
    }
};

// The whole stage for one tile whose cells the threads copy themselves (rows
// of 8 cells, 16-byte aligned: block offsets and extents are multiples of 8
// cells): staging, three sweeps, epilogue.  Uses W [5][Stg<T>::SV], A [5][NACC]
// (16-byte aligned), red [NT/32][5], ts and sides [NSIDES] in shared memory.
template <typename T, typename Src>
__device__ __forceinline__ void stage_tile(const StageParams<T> &p, const Src &src, int item, T *W, T *A,
                                           double (*red)[5], TileInfo<T> *ts, typename Src::Side *sides)
{
    // the tile's geometry is kept in shared memory (ts, and the sources of the
    // quarters of its six sides) and re-read after each barrier, so it does not
    // occupy registers across the three sweeps
    {
        TileInfo<T> w;
        src.template tile<T>(item, w);
        if (threadIdx.x == 0) *ts = w;
        if (threadIdx.x < NSIDES) sides[threadIdx.x] = src.side(w, threadIdx.x);
    }
    __syncthreads();
    const TileInfo<T> &t = *ts;
    // the tile's cells by 16-byte copies into A (free until the sweeps), dense
    // [5][8][8][8], the halo cells one by one into their slots
    constexpr int V = 16 / (int)sizeof(T), CH = NCORE / V; // cells of a chunk, chunks of a component
    for (int q = threadIdx.x; q < CH; q += NT) {
        const int i = q * V, x = i % TB, y = (i / TB) % TB, z = i / (TB * TB);
        const int64_t o = t.boff + (t.x0 + x) + (int64_t)t.N0 * ((t.y0 + y) + (int64_t)t.N1 * (t.z0 + z));
#pragma unroll
        for (int c = 0; c < 5; ++c)
            cp_async16(A + c * NCORE + i, p.U[c] + o);
    }
    cp_commit();
    constexpr int first = Stg<T>::all ? 3 : 2; // directions whose slots are free now
#pragma unroll 1
    for (int D = 0; D < first; ++D) {
        issue_halo<T>(D, p, src, t, sides, W);
        cp_commit();
    }
    cp_wait<first>();
    __syncthreads(); // other threads' chunks
    T vmax = T(0);
    convert_core<T>(A, p.gm1, W, vmax);
    if constexpr (Stg<T>::all) {
        cp_wait<0>();
#pragma unroll 1
        for (int D = 0; D < 3; ++D)
            convert_halo<T>(D, p.gm1, W, vmax);
        sweeps_at_once<T>(p, t, W, A, vmax);
    } else {
#pragma unroll 1
        for (int D = 0; D < 3; ++D) {
            if (D == 0)
                cp_wait<1>();
            else
                cp_wait<0>();
            convert_halo<T>(D, p.gm1, W, vmax);
            // W, this slot; every thread is done with the previous sweep
            __syncthreads();
            if (D == 1) {
                issue_halo<T>(2, p, src, t, sides, W);
                cp_commit();
            }
            sweep_dir<T, false>(D, p, t, W, A);
        }
    }
    Epilogue<T> E;
    E.load(p, t);
    __syncthreads(); // A
    E.store(p, A, red, item);
    __syncthreads(); // shared memory is reused by the next tile
}

// ---------------------------------------------------------------------------
// Tiles of a uniform grid, staged by TMA.  A side of a tile lies in one block
// (tiles are aligned), so a side whose cells are all plain copies is one box
// of 3 planes (x: 4 cells, the 16-byte granularity of the copy's start) per
// component; the other sides (faces with BCs) are resolved cell by cell.
// Against per-thread copies of the halo cells this removes most address
// arithmetic and L1 traffic of the staging.
//
// One CTA per tile.  (Persistent CTAs that start the next tile's copies during
// the epilogue measured slower: FP64 20.3 against 18.7 ms a step of 256 x 512 x
// 512 cells, FP32 9.5 against 9.0 ms on 384^3, with tiles handed out by cluster
// launch control; 22.7 and 10.9 ms with a grid stride.)
// ---------------------------------------------------------------------------
// Where the copies land.  The tile's cells: in A (free until the sweeps),
// dense [5][8][8][8].  FP64 sides: y and z in their slots, converted in place,
// x in slot 0 and the entries behind it as [side][z][y][4].  FP32 cannot
// convert in place (its pairs are interleaved): its sides land as
// [side][component][...] arrays from the start of W and pass through registers.
template <typename T> struct Land {
    static constexpr int X = 4 * NLINE, YZ = G * NLINE; // entries of a side
    static constexpr int NC = Stg<T>::all ? 5 : 1;      // components of a side's copy
    static __device__ __forceinline__ int size(int D) { return D == 0 ? X : YZ; }
    static __device__ __forceinline__ int side(int D, int s) // first entry of a side, component 0
    {
        if constexpr (Stg<T>::all)
            return 5 * ((D == 0 ? 0 : 2 * X + (D - 1) * 2 * YZ) + s * size(D));
        else
            return Stg<T>::slot(D) + s * size(D);
    }
    static __device__ __forceinline__ int cstride(int D) { return Stg<T>::all ? size(D) : Stg<T>::SV; }
    static __device__ __forceinline__ uint32_t bytes(int D) { return 5u * (uint32_t)size(D) * (uint32_t)sizeof(T); }
    // entry of halo cell i of direction D, component 0
    static __device__ __forceinline__ int cell(int D, int i)
    {
        if (D == 0) {
            const int h = i % (2 * G), yz = i / (2 * G);
            return (h < G ? side(0, 0) + h + 1 : side(0, 1) + h - G) + 4 * yz;
        }
        const int s = i >= YZ;
        return side(D, s) + i - s * YZ;
    }
};

// issues side s of direction D of the tile (component c; FP32: all)
template <typename T>
__device__ __forceinline__ void tma_side(int D, int s, int c, const TileMaps &maps, const CartSrc &src,
                                         const TileInfo<T> &t, T *W, uint64_t *bar)
{
    const int n = D == 0 ? t.N0 : (D == 1 ? t.N1 : t.N2), o = D == 0 ? t.x0 : (D == 1 ? t.y0 : t.z0);
    int a = s ? o + TB : o - (D == 0 ? 4 : G); // first plane of the box, in the block that holds it
    if (a < 0) a += n;
    if (a >= n) a -= n;
    const void *map = D == 0 ? &maps.hx : (D == 1 ? &maps.hy : &maps.hz);
    tma_load_5d(W + Land<T>::side(D, s) + c * Land<T>::cstride(D), map, D == 0 ? a : t.x0, D == 1 ? a : t.y0,
                D == 2 ? a : t.z0, src.template side_block<T>(t, D, s), c, bar);
}

// Warp 0: starts the copies of the tile: its cells and the sides whose landing
// area is free (FP64: x, FP32: all), on bar[0]; FP64 announces the y and z
// sides' bytes on bar[1] and bar[2].  Returns the sides that are not plain.
template <typename T>
__device__ __forceinline__ unsigned start_tile(const TileInfo<T> &t, const TileMaps &maps, const CartSrc &src, T *W,
                                               T *A, uint64_t *bar)
{
    const int q = threadIdx.x;
    constexpr uint32_t cells = 5u * NCORE * (uint32_t)sizeof(T);
    if (q == 0) {
        mbar_arrive_expect_tx(bar, cells);
        tma_load_5d(A, &maps.core, t.x0, t.y0, t.z0, t.block, 0, bar);
    }
    const unsigned slow = src.template slow_sides<T>(t);
    constexpr int NS = Stg<T>::all ? 6 : 2, CC = 5 / Land<T>::NC; // sides that start now, copies per side
    if (q == 0) {
        uint32_t bytes = 0;
        for (int k = 0; k < NS; ++k)
            bytes += ((slow >> k) & 1u) ? 0u : Land<T>::bytes(k >> 1);
        mbar_arrive_expect_tx(bar, bytes);
        if constexpr (!Stg<T>::all)
            for (int D = 1; D < 3; ++D)
                mbar_arrive_expect_tx(bar + D, Land<T>::bytes(D) * (2u - __popc((slow >> (2 * D)) & 3u)));
    }
    __syncwarp();
    if (q < CC * NS) {
        const int k = q / CC, c = q % CC;
        if (!((slow >> k) & 1u)) tma_side<T>(k >> 1, k & 1, c, maps, src, t, W, bar);
    }
    return slow;
}

// halo cells of direction D on the sides in `slow`, by the face rules, into
// the landing area
template <typename T>
__device__ __forceinline__ void resolve_sides(int D, unsigned slow, const StageParams<T> &p, const CartSrc &src,
                                              const TileInfo<T> &t, T *W, const FaceRule<T> (*rules)[5])
{
    if (!((slow >> (2 * D)) & 3u)) return;
#pragma unroll 1
    for (int j = 0; j < NHALO / NT; ++j) {
        const int i = threadIdx.x + j * NT;
        int x, y, z, e;
        halo_cell(D, i, x, y, z, e);
        const int s = (D == 0 ? x : (D == 1 ? y : z)) > 0;
        if (!((slow >> (2 * D + s)) & 1u)) continue;
        const int l = Land<T>::cell(D, i), n = D == 0 ? t.N0 : (D == 1 ? t.N1 : t.N2);
        const int g[3] = {t.x0 + x, t.y0 + y, t.z0 + z};
        const int gd = D == 0 ? g[0] : (D == 1 ? g[1] : g[2]);
        const int64_t st = D == 0 ? 1 : (D == 1 ? t.N0 : (int64_t)t.N0 * t.N1);
        // the cell's offset without its coordinate along D, and the shift to the neighbour
        const int64_t o = t.boff + g[0] + (int64_t)t.N0 * (g[1] + (int64_t)t.N1 * g[2]) - gd * st;
        const int64_t nbr = (int64_t)(src.template side_block<T>(t, D, s) - t.block) * src.L.bstride;
        T v[5];
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            const FaceRule<T> r = rules[2 * D + s][c];
            v[c] = r.value;
            if (r.kind != kRuleValue) {
                const int q = r.kind == kRuleEdge     ? (s ? n - 1 : 0)
                              : r.kind == kRuleMirror ? (s ? 2 * n - 1 : -1) - gd
                                                      : (s ? gd - n : gd + n);
                v[c] *= p.U[c][o + q * st + (r.kind == kRuleCopy ? nbr : 0)];
            }
        }
#pragma unroll
        for (int c = 0; c < 5; ++c)
            W[l + c * Land<T>::cstride(D)] = v[c];
    }
}

// FP64: starts the sides of direction D (1 or 2) once their slot is free;
// five warps issue one component each
template <typename T>
__device__ __forceinline__ void start_sides(int D, unsigned slow, const StageParams<T> &p, const CartSrc &src,
                                            const TileInfo<T> &t, T *W, const FaceRule<T> (*rules)[5],
                                            const TileMaps &maps, uint64_t *bar)
{
    const int c = threadIdx.x >> 5, s = threadIdx.x & 31;
    if (c < 5 && s < 2 && !((slow >> (2 * D + s)) & 1u)) tma_side<T>(D, s, c, maps, src, t, W, bar + D);
    resolve_sides<T>(D, slow, p, src, t, W, rules);
}

// waits for a copy barrier's only phase; records a timeout and gives the
// copies a second bounded wait, so that they are not left writing into this
// CTA's shared memory
__device__ __forceinline__ void wait_copies(uint64_t *bar, int *err)
{
    if (!mbar_wait_bounded_sleep(bar, 0, 100)) {
        if (err) atomicExch(err, kDevErrTimeout);
        mbar_wait_bounded_sleep(bar, 0, 100);
    }
}

// What the TMA form keeps in shared memory beside W and A.
template <typename T> struct TileShared {
    uint64_t bar[3];
    TileInfo<T> t;
    unsigned slow;
    FaceRule<T> rules[6][5];
    double red[NT / 32][5];
};

// The whole stage for one tile of a uniform grid.  W [5][Stg<T>::SV] and A
// [5][NACC] in shared memory, 128-byte aligned.
template <typename T>
__device__ __forceinline__ void stage_tile_tma(const StageParams<T> &p, const CartSrc &src, const TileMaps &maps, T *W,
                                               T *A, TileShared<T> &sh)
{
    const TileInfo<T> &t = sh.t;
    if (threadIdx.x < 32) {
        if (threadIdx.x == 0) {
            mbar_init(sh.bar, 2); // the cells' arrival and the sides'
            mbar_init(sh.bar + 1, 1);
            mbar_init(sh.bar + 2, 1);
            fence_mbar_init();
            src.template tile<T>(blockIdx.x, sh.t);
        }
        __syncwarp();
        const unsigned slow = start_tile<T>(t, maps, src, W, A, sh.bar);
        if (threadIdx.x == 0) sh.slow = slow;
    } else if (sizeof(T) == 8 && p.use_un) {
        // meanwhile the other warps fetch the tile's U^n, which the epilogue
        // reads, into L2 (rows of 8 cells)
        TileInfo<T> w;
        src.template tile<T>(blockIdx.x, w);
        for (int r = threadIdx.x - 32; r < 5 * NLINE; r += NT - 32) {
            const int c = r / NLINE, y = r % TB, z = (r / TB) % TB;
            const T *row = p.Un[c] + w.boff + w.x0 + (int64_t)w.N0 * (w.y0 + y + (int64_t)w.N1 * (w.z0 + z));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(row));
        }
    }
    __syncthreads(); // sh
    constexpr int LD = Stg<T>::all ? 3 : 1; // directions that pass through registers
    if (sh.slow) {
        if (threadIdx.x < 30) {
            const int k = threadIdx.x / 5, c = threadIdx.x % 5;
            if ((sh.slow >> k) & 1u) sh.rules[k][c] = face_rule<T>(src.L, src.bc[c], t.block, k >> 1, k & 1);
        }
        __syncthreads();
#pragma unroll 1
        for (int D = 0; D < LD; ++D)
            resolve_sides<T>(D, sh.slow, p, src, t, W, sh.rules);
    }
    wait_copies(sh.bar, p.err);
    T vmax = T(0);
    {
        T v[LD][NHALO / NT][5];
#pragma unroll
        for (int D = 0; D < LD; ++D)
#pragma unroll
            for (int j = 0; j < NHALO / NT; ++j) {
                const int l = Land<T>::cell(D, threadIdx.x + j * NT);
#pragma unroll
                for (int c = 0; c < 5; ++c)
                    v[D][j][c] = W[l + c * Land<T>::cstride(D)];
            }
        fence_proxy_async_smem(); // FP64: the y sides land behind the x sides next
        __syncthreads();
        if constexpr (!Stg<T>::all) start_sides<T>(1, sh.slow, p, src, t, W, sh.rules, maps, sh.bar);
#pragma unroll
        for (int D = 0; D < LD; ++D)
#pragma unroll
            for (int j = 0; j < NHALO / NT; ++j) {
                int x, y, z, e;
                halo_cell(D, threadIdx.x + j * NT, x, y, z, e);
                store_primitive<T>(v[D][j], p.gm1, W, Stg<T>::slot(D) + e, vmax);
            }
    }
    convert_core<T>(A, p.gm1, W, vmax);
    if constexpr (Stg<T>::all) {
        sweeps_at_once<T>(p, t, W, A, vmax);
    } else {
#pragma unroll 1
        for (int D = 0; D < 3; ++D) {
            if (D > 0) {
                wait_copies(sh.bar + D, p.err);
                convert_halo<T>(D, p.gm1, W, vmax);
            }
            fence_proxy_async_smem(); // before the z sides land in slot 0
            // W, this slot; every thread is done with the previous sweep
            __syncthreads();
            if (D == 1) start_sides<T>(2, sh.slow, p, src, t, W, sh.rules, maps, sh.bar);
            sweep_dir<T, false>(D, p, t, W, A);
        }
    }
    Epilogue<T> E;
    E.load(p, t);
    __syncthreads(); // A
    E.store(p, A, sh.red, blockIdx.x);
}

} // namespace euler
} // namespace cn
