// labfill.cu -- K0: explicit lab fill (Cartesian::loadLab into lab buffers).
//
// One CTA per (block, slab of lab planes along z).  The slab's lab cells are
// the block's own cells, the x ghosts, the y-ghost rows of the inside planes
// and the z-ghost planes (non-tensorial labs: edges and corners stay
// undefined, as in the reference).  The block's own planes are one contiguous
// run of memory, brought by one bulk copy into shared memory; meanwhile the
// threads walk the ghosts, those behind faces without a BC or a skipped
// neighbour in closed form (the periodic neighbour's cell), several loads in
// flight per thread; ghost rows are resolved once per row (x passes through
// the FieldLab resolution unchanged), other BC-chain cells one by one
// (cn::lab_resolve: skip rule, BC chain).  lab_fill_rows_kernel is the one-pass
// form of labs without edges and corners, lab_fill_kernel walks row by row
// (tensorial labs, and labs with more ghost rows than the former's table);
// node and face grids (lab_fill_grow_kernel) take per-cell resolution.  Stores
// are coalesced along the lab's rows.  The stencil kernels read what their labs
// would hold without making them; these kernels give the reference's FieldLab
// contents for user stencils and the bit-exact comparison with it.
#include "cn_fastdiv.h"
#include "cn_internal.h"
#include "cn_tma.cuh"

#include <algorithm>
#include <type_traits>

namespace cn {

constexpr int KL = 4;              // cells per thread resolved before their loads
constexpr int KLM = 8;             // cells per thread in flight in the one-pass form
constexpr int KLO = 8;             // own cells in flight per thread of the row form without the copy
constexpr int KLR = 3;             // rows in flight per thread of the row form
constexpr int KLX = 3;             // x ghosts in flight per thread of the row form
constexpr int kBulkBytes = 24576;  // largest bulk copy of a slab's block planes
constexpr int kGhostBytes = 24576; // largest x ghosts beside them (whole runs)
constexpr int kRunCtas = 4096;     // least CTAs of a launch with whole runs
// target cells of a CTA's slab: three planes of the 38^2 lab of 32^3 blocks
// with three ghosts.  Thinner slabs leave more of the SM's on-chip memory
// to the L1 cache (the shared-memory carve-out follows the resident CTAs'
// needs), which measured faster than thicker slabs
constexpr int kCellsPerCta = 4332;
constexpr int kRowsCtas = 4;       // resident CTAs per SM of the one-pass form
constexpr int kWarpRowCtas = 6;    // of the row form

// a cell's source, collected from lab_resolve
template <typename T> struct LabSource {
    int kind = 0; // 0 undefined, 1 the value v, 2 comp[idx] times the signs
    int nsign = 0;
    int64_t idx = 0;
    T v = T(0), s0 = T(1), s1 = T(1), s2 = T(1);
    __device__ __forceinline__ void value(T x)
    {
        kind = 1;
        v = x;
    }
    __device__ __forceinline__ void load(int64_t i, int n, T a, T b, T c)
    {
        kind = 2;
        idx = i;
        nsign = n;
        s0 = a;
        s1 = b;
        s2 = c;
    }
};

// Loads the sources of up to KL cells, then stores them: src[k] for cell
// dst[k] (offsets in the CTA's output, -1: no cell).
template <typename T>
__device__ __forceinline__ void lab_store(const T *__restrict__ comp, const LabSource<T> (&src)[KL],
                                          const int (&dst)[KL], T *__restrict__ o)
{
    T v[KL];
#pragma unroll
    for (int k = 0; k < KL; ++k)
        v[k] = src[k].kind == 2 ? comp[src[k].idx] : src[k].v;
#pragma unroll
    for (int k = 0; k < KL; ++k) {
        if (dst[k] < 0 || src[k].kind == 0) continue;
        T x = v[k];
        if (src[k].kind == 2) {
            if (src[k].nsign > 2) x = src[k].s2 * x;
            if (src[k].nsign > 1) x = src[k].s1 * x;
            if (src[k].nsign > 0) x = src[k].s0 * x;
        }
        o[dst[k]] = x;
    }
}

// Node and face grids (per-block extents): every cell of the CTA's slab
// resolved on its own.
template <typename T>
__global__ void __launch_bounds__(256)
    lab_fill_grow_kernel(const T *__restrict__ comp, LabGeom L, BcView bc, int block_begin, int pz, FastDiv dE0,
                         FastDiv dPlane, int apply_bc, T *__restrict__ out)
{
    const int E0 = L.n[0] + L.lo[0] + L.hi[0];
    const int E1 = L.n[1] + L.lo[1] + L.hi[1];
    const int E2 = L.n[2] + L.lo[2] + L.hi[2];
    const int plane = E0 * E1;
    const int bl = blockIdx.y, z0 = blockIdx.x * pz; // block-major, as lab_fill_rows_kernel
    const int nz = min(pz, E2 - z0);
    const int block = block_begin + bl;
    const int bx = block % L.nb[0];
    const int by = (block / L.nb[0]) % L.nb[1];
    const int bz = block / (L.nb[0] * L.nb[1]);
    const uint8_t mode = bc.mode[block];
    const int cells = nz * plane;
    T *o = out + ((int64_t)bl * E2 + z0) * plane;
    for (int t0 = threadIdx.x; t0 < cells; t0 += KL * blockDim.x) {
        LabSource<T> src[KL];
        int dst[KL];
#pragma unroll
        for (int k = 0; k < KL; ++k) {
            const int t = t0 + k * blockDim.x;
            dst[k] = -1;
            if (t < cells) {
                const int zz = dPlane.div(t), r = t - zz * plane;
                const int y = dE0.div(r), x = r - y * E0;
                dst[k] = t;
                lab_resolve<T, true>(L, bc, mode, block, bx, by, bz, x - L.lo[0], y - L.lo[1], z0 + zz - L.lo[2],
                                     apply_bc != 0, src[k]);
            }
        }
        lab_store<T>(comp, src, dst, o);
    }
}

// a y- or z-ghost row: the source of its first cell and its first cell's
// offset in the lab
template <typename T> struct alignas(16) RowSrc {
    int64_t idx; // of the first cell in the component
    int dst;     // the first cell's offset in the lab
    int kind;    // 0 undefined, 1 the value v, 2 + n: the cells times n signs
    T v, s0, s1, s2;
};
constexpr int kRows = 96; // rows resolved per round

// Divisors of the row form (fixed per launch).
struct LabDivs {
    FastDiv n0, n1; // block extents along x, y
    FastDiv e0;     // lab extent along x
    FastDiv gx, gy; // ghosts per row along x: lo0 + hi0, along y: lo1 + hi1
    FastDiv wpl;    // rows per z-ghost plane, and rows with x ghosts per plane: n1, or E1 if tensorial
};

// lab coordinates of x ghost u of the inside rows
__device__ __forceinline__ void x_ghost_cell(const LabDivs &dv, int u, int gx, int n0, int n1, int lo0, int lo1, int zi0,
                                            int &x, int &y, int &z)
{
    const int r = dv.gx.div(u), zp = dv.n1.div(r);
    const int g = u - r * gx;
    x = g < lo0 ? g : g + n0;
    y = r - zp * n1 + lo1;
    z = zi0 + zp;
}

// Ghost row `row` of a slab: rows [0, ny) are the y-ghost rows of its inside
// planes, then come the rows of its z-ghost planes (tensorial: the y-ghost rows
// among them); the source of its first cell (x = 0 of the block) and that
// cell's offset in the lab.  x passes through every step of the resolution
// unchanged, so cell x of the row is the source shifted by x (or the same
// value).
template <typename T>
__device__ __forceinline__ RowSrc<T> lab_row(const LabGeom &L, const BcView &bc, uint8_t mode, uint8_t faces,
                                             int block, int bx, int by, int bz, bool abc, const LabDivs &dv, int row,
                                             int ny, int gy, bool tens, int zi0, int nlo, int zhi, int z0, int E0,
                                             int E1)
{
    const int n0 = L.n[0], n1 = L.n[1], n2 = L.n[2];
    int y, z; // lab coordinates of the row
    if (row < ny) {
        const int zp = dv.gy.div(row), g = row - zp * gy;
        y = g < L.lo[1] ? g : g + n1;
        z = zi0 + zp;
    } else {
        const int rr = row - ny, zp = dv.wpl.div(rr);
        y = rr - zp * (tens ? E1 : n1) + (tens ? 0 : L.lo[1]);
        z = zp < nlo ? z0 + zp : zhi + (zp - nlo);
    }
    const int q1 = y - L.lo[1], q2 = z - L.lo[2];
    const int r1 = q1 < 0 ? -1 : (q1 >= n1 ? 1 : 0), r2 = q2 < 0 ? -1 : (q2 >= n2 ? 1 : 0);
    const int crossed = (r1 ? (r1 < 0 ? 4 : 8) : 0) | (r2 ? (r2 < 0 ? 16 : 32) : 0);
    RowSrc<T> R;
    if (faces & crossed) {
        LabSource<T> s;
        lab_resolve<T, false>(L, bc, mode, block, bx, by, bz, 0, q1, q2, abc, s);
        R.idx = s.idx;
        R.kind = s.kind == 2 ? 2 + s.nsign : s.kind;
        R.v = s.v;
        R.s0 = s.s0;
        R.s1 = s.s1;
        R.s2 = s.s2;
    } else {
        int nby = by + r1, nbz = bz + r2;
        nby = nby < 0 ? nby + L.nb[1] : (nby >= L.nb[1] ? nby - L.nb[1] : nby);
        nbz = nbz < 0 ? nbz + L.nb[2] : (nbz >= L.nb[2] ? nbz - L.nb[2] : nbz);
        R.kind = 2;
        R.idx = (int64_t)(bx + L.nb[0] * (nby + L.nb[1] * nbz)) * L.bstride + n0 * ((q1 - r1 * n1) + n1 * (q2 - r2 * n2));
    }
    R.dst = L.lo[0] + E0 * (y + E1 * z);
    return R;
}

// Lab planes [z0, z1) of a CTA's slab: the planes inside the block
// [zi0, zi0 + nin), nlo z-ghost planes below them and the z-ghost planes
// from zhi up (nghost in all).
struct SlabPlanes {
    int zi0, nin, nlo, zhi, nghost;
};
__host__ __device__ __forceinline__ int imax(int a, int b) { return a > b ? a : b; }
__host__ __device__ __forceinline__ int imin(int a, int b) { return a < b ? a : b; }
__host__ __device__ __forceinline__ SlabPlanes slab_planes(const LabGeom &L, int z0, int z1)
{
    SlabPlanes P;
    P.zi0 = imax(z0, L.lo[2]);
    P.nin = imax(0, imin(z1, L.lo[2] + L.n[2]) - P.zi0);
    P.nlo = imax(0, imin(z1, L.lo[2]) - z0);
    P.zhi = imax(z0, L.lo[2] + L.n[2]);
    P.nghost = P.nlo + imax(0, z1 - P.zhi);
    return P;
}

// one cell's source stored (kind 0: nothing)
template <typename T>
__device__ __forceinline__ void lab_store1(const T *__restrict__ comp, const LabSource<T> &s, int dst, T *__restrict__ o)
{
    if (dst < 0 || s.kind == 0) return;
    T x = s.kind == 2 ? comp[s.idx] : s.v;
    if (s.kind == 2) {
        if (s.nsign > 2) x = s.s2 * x;
        if (s.nsign > 1) x = s.s1 * x;
        if (s.nsign > 0) x = s.s0 * x;
    }
    o[dst] = x;
}

// Cell grids with non-tensorial labs whose y- and z-ghost rows fit in shared
// memory (kRows per slab), the common case: the one-pass form, at kRowsCtas
// CTAs per SM.
template <typename T, bool RUNS>
__global__ void __launch_bounds__(256, kRowsCtas)
    lab_fill_rows_kernel(const T *__restrict__ comp, LabGeom L, BcView bc, int block_begin, int pz, LabDivs dv,
                         int apply_bc, int bulk, int *err, T *__restrict__ out)
{
    const int n0 = L.n[0], n1 = L.n[1];
    const int E0 = n0 + L.lo[0] + L.hi[0];
    const int E1 = n1 + L.lo[1] + L.hi[1];
    const int E2 = L.n[2] + L.lo[2] + L.hi[2];
    // one CTA per (slab, block): x the slab, so that a block's slabs run
    // together (CTAs start in the order of their linear index) and the ghost
    // planes read from a block's z neighbours are read close in time to the
    // neighbours' own CTAs, while they are in L2
    const int bl = blockIdx.y, z0 = blockIdx.x * pz;
    const int block = block_begin + bl;
    const int bx = block % L.nb[0];
    const int by = (block / L.nb[0]) % L.nb[1];
    const int bz = block / (L.nb[0] * L.nb[1]);
    const uint8_t mode = bc.mode[block];
    const uint8_t faces = bc.faces[block];
    const bool abc = apply_bc != 0;
    const SlabPlanes P = slab_planes(L, z0, min(z0 + pz, E2));
    const int zi0 = P.zi0, nin = P.nin, nlo = P.nlo, zhi = P.zhi;
    const int gx = L.lo[0] + L.hi[0], gy = L.lo[1] + L.hi[1];
    T *o = out + (int64_t)bl * E0 * E1 * E2;
    const int ny = nin * gy, nrows = ny + P.nghost * n1;
    __shared__ RowSrc<T> rows[kRows];
    // One pass over all three kinds of plain copies, KLM loads in flight
    // per thread: the block's own cells, the x ghosts behind clear faces
    // and the ghost rows whose source is a plain cell run.  The
    // rows are resolved first; cells that need BC chains or skips are
    // left to a second pass.
    const int A = nin * n1 * n0, B = nin * n1 * gx, tot = A + B + nrows * n0;
    const int64_t bbase = (int64_t)block * L.bstride + (int64_t)n0 * n1 * (zi0 - L.lo[2]);
    // The block's own planes of the slab are one contiguous run of
    // memory: with room in the dynamic shared memory (`bulk` bytes) one
    // bulk copy brings them while the threads work on the ghosts.
    extern __shared__ __align__(128) unsigned char lab_bulk[];
    __shared__ __align__(8) uint64_t bulk_bar;
    const uint32_t bytes0 = (uint32_t)A * (uint32_t)sizeof(T);
    const bool use_bulk = A > 0 && bytes0 <= (uint32_t)bulk && ((uint32_t)(n0 * n1) * sizeof(T)) % 16 == 0;
    if (use_bulk && threadIdx.x == 0) {
        mbar_init(&bulk_bar, 1);
        fence_mbar_init();
        mbar_arrive_expect_tx(&bulk_bar, bytes0);
        bulk_g2s(lab_bulk, comp + bbase, bytes0, &bulk_bar);
    }
    // With both x faces clear, the own rows of a plane and their x ghosts are
    // one contiguous run of the lab, all of it plain copies.  RUNS: the ghosts
    // wait in shared memory behind the planes and the run is stored in order,
    // so that no sector is written in two parts.
    const bool runs = RUNS && use_bulk && !(faces & 3);
    T *xg = reinterpret_cast<T *>(lab_bulk + bulk);
    for (int j = threadIdx.x; j < nrows; j += blockDim.x)
        rows[j] = lab_row<T>(L, bc, mode, faces, block, bx, by, bz, abc, dv, j, ny, gy, false, zi0, nlo, zhi, z0, E0,
                             E1);
    __syncthreads(); // the rows, and the barrier's initialisation
    bool deferred = false;
    const int base = use_bulk ? A : 0; // the first item of the pass
    for (int t0 = base + threadIdx.x; t0 < tot; t0 += KLM * blockDim.x) {
        int64_t idx[KLM];
        int dst[KLM];
#pragma unroll
        for (int k = 0; k < KLM; ++k) {
            const int t = t0 + k * blockDim.x;
            dst[k] = -1;
            idx[k] = 0;
            if (t < A) {
                const int r = dv.n0.div(t), zp = dv.n1.div(r);
                dst[k] = (t - r * n0 + L.lo[0]) + E0 * ((r - zp * n1 + L.lo[1]) + E1 * (zi0 + zp));
                idx[k] = bbase + t;
            } else if (t < A + B) {
                int x, y, z;
                x_ghost_cell(dv, t - A, gx, n0, n1, L.lo[0], L.lo[1], zi0, x, y, z);
                const int q0 = x - L.lo[0], r0 = q0 < 0 ? -1 : 1;
                if (faces & (r0 < 0 ? 1 : 2)) {
                    deferred = true;
                } else {
                    const int nbx = bx + r0 < 0 ? bx + r0 + L.nb[0] : (bx + r0 >= L.nb[0] ? bx + r0 - L.nb[0] : bx + r0);
                    dst[k] = runs ? -2 - (t - A) : x + E0 * (y + E1 * z);
                    idx[k] = (int64_t)(nbx + L.nb[0] * (by + L.nb[1] * bz)) * L.bstride + (q0 - r0 * n0) +
                             n0 * ((y - L.lo[1]) + n1 * (z - L.lo[2]));
                }
            } else if (t < tot) {
                const int u = t - A - B, j = dv.n0.div(u), x = u - j * n0;
                const RowSrc<T> &R = rows[j];
                if (R.kind == 2) {
                    dst[k] = R.dst + x;
                    idx[k] = R.idx + x;
                } else {
                    deferred = true;
                }
            }
        }
        T v[KLM];
#pragma unroll
        for (int k = 0; k < KLM; ++k)
            if (RUNS ? dst[k] != -1 : dst[k] >= 0) v[k] = comp[idx[k]];
#pragma unroll
        for (int k = 0; k < KLM; ++k)
            if (dst[k] >= 0) o[dst[k]] = v[k];
            else if (RUNS && dst[k] != -1) xg[-2 - dst[k]] = v[k];
    }
    if (use_bulk) {
        if (RUNS && runs) __syncthreads(); // the x ghosts
        // the block's cells from shared memory
        if (!mbar_wait_bounded_sleep(&bulk_bar, 0, 200)) {
            // record the error; a second bounded wait keeps the copy from
            // landing in a later CTA's shared memory
            if (threadIdx.x == 0 && err) atomicExch(err, kDevErrTimeout);
            mbar_wait_bounded_sleep(&bulk_bar, 0, 200);
        } else {
            const T *sb = reinterpret_cast<const T *>(lab_bulk);
            if (RUNS && runs) {
                T *ob = o + E0 * (L.lo[1] + E1 * zi0);
                const int run = n1 * E0, skip = E0 * (E1 - n1);
#pragma unroll 4
                for (int t = threadIdx.x; t < nin * run; t += blockDim.x) {
                    const int r = dv.e0.div(t), zp = dv.n1.div(r), x = t - r * E0 - L.lo[0];
                    const T *s = (unsigned)x < (unsigned)n0 ? sb + r * n0 + x
                                                            : xg + r * gx + L.lo[0] + (x < 0 ? x : x - n0);
                    ob[t + zp * skip] = *s;
                }
            } else {
                for (int t0 = threadIdx.x; t0 < A; t0 += KLM * blockDim.x) {
#pragma unroll
                    for (int k = 0; k < KLM; ++k) {
                        const int t = t0 + k * blockDim.x;
                        if (t < A) {
                            const int r = dv.n0.div(t), zp = dv.n1.div(r);
                            o[(t - r * n0 + L.lo[0]) + E0 * ((r - zp * n1 + L.lo[1]) + E1 * (zi0 + zp))] = sb[t];
                        }
                    }
                }
            }
        }
    }
    if (deferred) {
        // the second pass: the same items of this thread
        const int nt = (int)blockDim.x;
        for (int t = A + ((((int)threadIdx.x + base - A) % nt) + nt) % nt; t < tot; t += nt) {
            LabSource<T> src[1];
            int dst[1] = {-1};
            if (t < A + B) {
                int x, y, z;
                x_ghost_cell(dv, t - A, gx, n0, n1, L.lo[0], L.lo[1], zi0, x, y, z);
                if (!(faces & (x < L.lo[0] ? 1 : 2))) continue;
                lab_resolve<T, false>(L, bc, mode, block, bx, by, bz, x - L.lo[0], y - L.lo[1], z - L.lo[2], abc,
                                      src[0]);
                dst[0] = x + E0 * (y + E1 * z);
            } else {
                const int u = t - A - B, j = dv.n0.div(u), x = u - j * n0;
                const RowSrc<T> &R = rows[j];
                if (R.kind == 2) continue;
                src[0].kind = min(R.kind, 2);
                src[0].nsign = R.kind - 2;
                src[0].idx = R.idx + x;
                src[0].v = R.v;
                src[0].s0 = R.s0;
                src[0].s1 = R.s1;
                src[0].s2 = R.s2;
                dst[0] = R.dst + x;
            }
            lab_store1<T>(comp, src[0], dst[0], o);
        }
    }
}

// Cell grids by rows: 2^wl threads (the least power of two that holds a row,
// at most a warp) walk the cells of a row, so that a row's place and source are
// found once for all its cells.  Tensorial labs, whose x ghosts cross other
// faces too, and labs with more ghost rows than lab_fill_rows_kernel's table.
// Tensorial labs are bound by instruction issue when each ghost is located by
// itself: B200, all tensorial labs of 512^3 FP64 with three ghosts 873 -> 598
// us, of 256^3 FP32 115 -> 81.  Labs without edges and corners are not (596 us by
// the one-pass form, 615 by this one): their bound is the memory's latency.
template <typename T, bool TENS>
__global__ void __launch_bounds__(256, kWarpRowCtas)
    lab_fill_kernel(const T *__restrict__ comp, LabGeom L, BcView bc, int block_begin, int pz, LabDivs dv, int wl,
                         int apply_bc, int bulk, int *err, T *__restrict__ out)
{
    const int n0 = L.n[0], n1 = L.n[1];
    const int E0 = n0 + L.lo[0] + L.hi[0];
    const int E1 = n1 + L.lo[1] + L.hi[1];
    const int E2 = L.n[2] + L.lo[2] + L.hi[2];
    // one CTA per (slab, block): x the slab, so that a block's slabs run
    // together (CTAs start in the order of their linear index) and the ghost
    // planes read from a block's z neighbours are read close in time to the
    // neighbours' own CTAs, while they are in L2
    const int bl = blockIdx.y, z0 = blockIdx.x * pz;
    const int block = block_begin + bl;
    const int bx = block % L.nb[0];
    const int by = (block / L.nb[0]) % L.nb[1];
    const int bz = block / (L.nb[0] * L.nb[1]);
    const uint8_t mode = bc.mode[block];
    const uint8_t faces = bc.faces[block];
    const bool abc = apply_bc != 0;
    const SlabPlanes P = slab_planes(L, z0, min(z0 + pz, E2));
    const int zi0 = P.zi0, nin = P.nin;
    const int gx = L.lo[0] + L.hi[0], gy = L.lo[1] + L.hi[1];
    T *o = out + (int64_t)bl * E0 * E1 * E2;
    const int own = nin * n1, ny = nin * gy, nrows = ny + P.nghost * (TENS ? E1 : n1);
    const int lx = threadIdx.x & ((1 << wl) - 1), grp = threadIdx.x >> wl, ngrp = blockDim.x >> wl;
    __shared__ RowSrc<T> rows[kRows];
    // The block's own planes of the slab are one contiguous run of
    // memory: with room in the dynamic shared memory (`bulk` bytes) one
    // bulk copy brings them while the threads work on the ghosts.
    extern __shared__ __align__(128) unsigned char lab_bulk[];
    __shared__ __align__(8) uint64_t bulk_bar;
    const T *src0 = comp + (int64_t)block * L.bstride + (int64_t)n0 * n1 * (zi0 - L.lo[2]);
    const uint32_t bytes0 = (uint32_t)(own * n0) * (uint32_t)sizeof(T);
    const bool use_bulk = own > 0 && bytes0 <= (uint32_t)bulk && ((uint32_t)(n0 * n1) * sizeof(T)) % 16 == 0;
    if (use_bulk && threadIdx.x == 0) {
        mbar_init(&bulk_bar, 1);
        fence_mbar_init();
        mbar_arrive_expect_tx(&bulk_bar, bytes0);
        bulk_g2s(lab_bulk, src0, bytes0, &bulk_bar);
    }
    // The y-ghost rows of the inside planes and the rows of the z-ghost
    // planes: kRows at a time resolved by a thread each, then copied, KLR rows
    // in flight per thread.
    for (int rb = 0; rb < nrows; rb += kRows) {
        const int nr = min(kRows, nrows - rb);
        if (rb > 0) __syncthreads(); // the previous rows are copied
        for (int j = threadIdx.x; j < nr; j += blockDim.x)
            rows[j] = lab_row<T>(L, bc, mode, faces, block, bx, by, bz, abc, dv, rb + j, ny, gy, TENS, zi0, P.nlo, P.zhi,
                                 z0, E0, E1);
        __syncthreads();
        for (int x = lx; x < n0; x += 1 << wl)
            for (int j0 = grp; j0 < nr; j0 += KLR * ngrp) {
                T v[KLR];
                int dst[KLR], kind[KLR];
#pragma unroll
                for (int k = 0; k < KLR; ++k) {
                    const int j = j0 + k * ngrp;
                    kind[k] = 0;
                    if (j < nr) {
                        const int4 h = *reinterpret_cast<const int4 *>(&rows[j]); // idx, dst, kind
                        kind[k] = h.w;
                        dst[k] = h.z + x;
                        if (h.w == 1) v[k] = rows[j].v;
                        else if (h.w) v[k] = comp[(((int64_t)h.y << 32) | (uint32_t)h.x) + x];
                    }
                }
#pragma unroll
                for (int k = 0; k < KLR; ++k) {
                    if (kind[k] == 0) continue;
                    const RowSrc<T> &R = rows[j0 + k * ngrp];
                    T q = v[k];
                    if (kind[k] > 4) q = R.s2 * q;
                    if (kind[k] > 3) q = R.s1 * q;
                    if (kind[k] > 2) q = R.s0 * q;
                    o[dst[k]] = q;
                }
            }
    }
    if (nrows == 0) __syncthreads(); // the barrier's initialisation
    // The x ghosts of the own rows (tensorial: of all rows), KLX at a time: the
    // periodic neighbour's cell where only clear faces lie between (as
    // lab_resolve gives it), the others in a second pass.
    const int xrows = TENS ? (min(z0 + pz, E2) - z0) * E1 : own, B = xrows * gx;
    bool deferred = false;
    auto ghost = [&](int t, int &x, int &y, int &z) { // lab coordinates of x ghost t
        const int r = dv.gx.div(t), zp = dv.wpl.div(r), g = t - r * gx;
        x = g < L.lo[0] ? g : g + n0;
        y = TENS ? r - zp * E1 : r - zp * n1 + L.lo[1];
        z = (TENS ? z0 : zi0) + zp;
    };
    auto beyond = [](int q, int n) { return q < 0 ? -1 : (q >= n ? 1 : 0); };
    auto crossed = [](int r, int lo) { return r ? (r < 0 ? lo : 2 * lo) : 0; };
    auto wrap = [](int b, int nb) { return b < 0 ? b + nb : (b >= nb ? b - nb : b); };
    for (int t0 = threadIdx.x; t0 < B; t0 += KLX * blockDim.x) {
        T v[KLX];
        int dst[KLX];
#pragma unroll
        for (int k = 0; k < KLX; ++k) {
            const int t = t0 + k * blockDim.x;
            dst[k] = -1;
            if (t >= B) continue;
            int x, y, z;
            ghost(t, x, y, z);
            const int q0 = x - L.lo[0], q1 = y - L.lo[1], q2 = z - L.lo[2];
            const int r0 = q0 < 0 ? -1 : 1, r1 = TENS ? beyond(q1, n1) : 0, r2 = TENS ? beyond(q2, L.n[2]) : 0;
            if (faces & (crossed(r0, 1) | crossed(r1, 4) | crossed(r2, 16))) {
                deferred = true;
            } else {
                const int nbx = wrap(bx + r0, L.nb[0]), nby = wrap(by + r1, L.nb[1]), nbz = wrap(bz + r2, L.nb[2]);
                dst[k] = x + E0 * (y + E1 * z);
                v[k] = comp[(int64_t)(nbx + L.nb[0] * (nby + L.nb[1] * nbz)) * L.bstride + (q0 - r0 * n0) +
                            n0 * ((q1 - r1 * n1) + n1 * (q2 - r2 * L.n[2]))];
            }
        }
#pragma unroll
        for (int k = 0; k < KLX; ++k)
            if (dst[k] >= 0) o[dst[k]] = v[k];
    }
    // the block's own rows
    if (use_bulk) {
        if (!mbar_wait_bounded_sleep(&bulk_bar, 0, 200)) {
            // record the error; a second bounded wait keeps the copy from
            // landing in a later CTA's shared memory
            if (threadIdx.x == 0 && err) atomicExch(err, kDevErrTimeout);
            mbar_wait_bounded_sleep(&bulk_bar, 0, 200);
        } else {
            const T *sb = reinterpret_cast<const T *>(lab_bulk);
#pragma unroll 4
            for (int r = grp; r < own; r += ngrp) {
                const int zp = dv.n1.div(r), d = L.lo[0] + E0 * ((r - zp * n1 + L.lo[1]) + E1 * (zi0 + zp));
                for (int x = lx; x < n0; x += 1 << wl) o[d + x] = sb[r * n0 + x];
            }
        }
    } else {
        // planes too large for the copy: their rows as one run, in pairs of
        // cells where rows hold whole pairs.  Row by row, KLR loads in flight
        // and a part of the lanes idle at each row's end, took up to 1.4 times
        // as long: B200, tensorial labs of 64 blocks of 96 x 96 x 40, one ghost,
        // FP64 111 -> 91 us, FP32 71 -> 58; non-tensorial ones of 128 blocks of
        // 100 x 100 x 30, FP64, 186 -> 143.
        auto copy = [&](auto pair) {
            constexpr int V = decltype(pair)::value, N = KLO / V;
            struct alignas(sizeof(T) * V) Cells {
                T v[V];
            };
            const Cells *src = reinterpret_cast<const Cells *>(src0);
            const int cnt = own * n0 / V;
            for (int p0 = threadIdx.x; p0 < cnt; p0 += N * blockDim.x) {
                Cells v[N];
#pragma unroll
                for (int k = 0; k < N; ++k)
                    if (p0 + k * blockDim.x < cnt) v[k] = src[p0 + k * blockDim.x];
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const int p = p0 + k * blockDim.x, t = V * p, r = dv.n0.div(t), zp = dv.n1.div(r);
                    T *d = o + (t - r * n0 + L.lo[0]) + E0 * ((r - zp * n1 + L.lo[1]) + E1 * (zi0 + zp));
                    if (p < cnt)
#pragma unroll
                        for (int i = 0; i < V; ++i) d[i] = v[k].v[i];
                }
            }
        };
        if (n0 % 2 == 0)
            copy(std::integral_constant<int, 2>{});
        else
            copy(std::integral_constant<int, 1>{});
    }
    if (deferred) { // this thread's x ghosts beyond faces with BCs or skips, one by one
        for (int t = threadIdx.x; t < B; t += blockDim.x) {
            int x, y, z;
            ghost(t, x, y, z);
            const int q0 = x - L.lo[0], q1 = y - L.lo[1], q2 = z - L.lo[2];
            if (!(faces & (crossed(beyond(q0, n0), 1) | crossed(beyond(q1, n1), 4) | crossed(beyond(q2, L.n[2]), 16))))
                continue;
            LabSource<T> src;
            lab_resolve<T, false>(L, bc, mode, block, bx, by, bz, q0, q1, q2, abc, src);
            lab_store1<T>(comp, src, x + E0 * (y + E1 * z), o);
        }
    }
}

template <typename T>
static cn_status launch_fill(cn_grid *g, int comp, const cn_stencil *s, int b0, int cnt,
                             int apply_bc, void *d_labs, cudaStream_t st)
{
    const LabGeom L = make_geom(g, s);
    const T *src = reinterpret_cast<const T *>(g->d_data) + (size_t)comp * g->comp_stride;
    const int64_t E0 = L.n[0] + L.lo[0] + L.hi[0], E1 = L.n[1] + L.lo[1] + L.hi[1], E2 = L.n[2] + L.lo[2] + L.hi[2];
    const int64_t plane = E0 * E1;
    if (plane * E2 >= (int64_t(1) << 31))
        return fail(CN_ERR_UNSUPPORTED, "cn_lab_fill: labs of 2^31 cells or more");
    // planes per CTA: about kCellsPerCta cells
    int pz = (int)std::max<int64_t>(1, std::min<int64_t>(E2, kCellsPerCta / plane));
    const bool grow = L.grow[0] || L.grow[1] || L.grow[2];
    // Both forms resolve kRows ghost rows of a slab at a time: slabs of fewer
    // planes until every slab's rows fit.  The one-pass form needs that.
    auto rows_fit = [&](int p) {
        for (int z0 = 0; z0 < E2; z0 += p) {
            const SlabPlanes P = slab_planes(L, z0, (int)std::min<int64_t>(z0 + p, E2));
            if (P.nin * (L.lo[1] + L.hi[1]) + P.nghost * (L.tensorial ? E1 : L.n[1]) > kRows) return false;
        }
        return true;
    };
    bool one_pass = !grow && !L.tensorial;
    if (one_pass) {
        while (pz > 1 && !rows_fit(pz)) --pz;
        one_pass = rows_fit(pz);
    }
    const int64_t slabs = (E2 + pz - 1) / pz;
    if (slabs > 65535) return fail(CN_ERR_UNSUPPORTED, "cn_lab_fill: more than 65535 lab slabs per block");
    const int threads = plane * pz >= 1024 ? 256 : 128;
    LabDivs dv;
    dv.n0 = FastDiv((uint32_t)L.n[0]);
    dv.n1 = FastDiv((uint32_t)L.n[1]);
    dv.e0 = FastDiv((uint32_t)E0);
    dv.gx = FastDiv((uint32_t)(L.lo[0] + L.hi[0]));
    dv.gy = FastDiv((uint32_t)(L.lo[1] + L.hi[1]));
    dv.wpl = FastDiv((uint32_t)(L.tensorial ? E1 : L.n[1]));
    int wl = 2;
    while (wl < 5 && (1 << wl) < L.n[0]) ++wl;
    // dynamic shared memory for the bulk copy of a slab's block planes
    const int64_t bulk = (int64_t)pz * L.n[0] * L.n[1] * (int64_t)sizeof(T);
    const int nbulk = !grow && bulk <= kBulkBytes ? (int)bulk : 0;
    const int64_t ghosts = (int64_t)pz * L.n[1] * (L.lo[0] + L.hi[0]) * (int64_t)sizeof(T);
    // Whole runs pay where x ghosts are a good part of a row (FP64, a sixth of
    // it and more), planes and runs are whole sectors, and many CTAs of some
    // size hide the barrier between the ghosts' loads and their stores.  B200,
    // FP64, ghosts as they come -> in runs, without BCs: 4096 blocks of 32^3,
    // three ghosts a side 597 -> 570 us; 4096 of 16^3, two 103 -> 90, three 131
    // -> 125; 1728 of 24^3, two 114 -> 103, three 135 -> 130.  Walls along y and z
    // (their ghosts take a second pass): 601 -> 579, 106 -> 96, 133 -> 131, 115 ->
    // 107, 139 -> 136, but 512 of 32^3, three 81 -> 84: twice as many CTAs there.
    // With walls along x, whose blocks store as they come, it loses (4096 of
    // 32^3, three 612 -> 622; 1728 of 24^3, three 147 -> 152), without whole
    // sectors too (8000 of 18 x 17 x 19, two 222 -> 228), with smaller ghosts
    // (4096 of 16^3, one 84.7 -> 88.1; 1728 of 32^3, two 220 -> 223), in FP32
    // (32^3, three 204 -> 230) and with few CTAs (512 of 16^3, three, 1536 CTAs
    // 19.1 -> 21.1).  Not under capture: BCs may be pushed later.
    const bool bulk_planes = nbulk && (int64_t)L.n[0] * L.n[1] * (int64_t)sizeof(T) % 16 == 0;
    bool runs = one_pass && g->bc_count_x == 0 && bulk_planes && sizeof(T) == 8 && L.n[0] >= 16 &&
                6 * (L.lo[0] + L.hi[0]) >= L.n[0] && E0 * L.n[1] % 4 == 0 && plane % 4 == 0 && ghosts <= kGhostBytes &&
                slabs * std::min(cnt, 65535) >= (g->bc_count ? 2 * kRunCtas : kRunCtas);
    if (runs && st) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        CN_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
        runs = cap == cudaStreamCaptureStatusNone;
    }
    if (!grow) {
        static DeviceOnce once[4];
        cn_status r = runs           ? smem_opt_in(once[3], lab_fill_rows_kernel<T, true>, (size_t)kBulkBytes + kGhostBytes)
                      : one_pass    ? smem_opt_in(once[0], lab_fill_rows_kernel<T, false>, (size_t)kBulkBytes)
                      : L.tensorial ? smem_opt_in(once[1], lab_fill_kernel<T, true>, (size_t)kBulkBytes)
                                    : smem_opt_in(once[2], lab_fill_kernel<T, false>, (size_t)kBulkBytes);
        if (r != CN_OK) return r;
    }
    // CTAs in block-major order: the slab along x, the block along y (a
    // block's slabs run together), at most 65535 blocks per launch
    for (int c0 = 0; c0 < cnt; c0 += 65535) {
        const dim3 grid((unsigned)slabs, (unsigned)std::min(65535, cnt - c0));
        T *out = reinterpret_cast<T *>(d_labs) + (int64_t)c0 * plane * E2;
        if (grow) {
            lab_fill_grow_kernel<T><<<grid, threads, 0, st>>>(src, L, bc_view(g, comp), b0 + c0, pz,
                                                              FastDiv((uint32_t)E0), FastDiv((uint32_t)plane),
                                                              apply_bc, out);
        } else if (one_pass) {
            auto kernel = runs ? lab_fill_rows_kernel<T, true> : lab_fill_rows_kernel<T, false>;
            kernel<<<grid, threads, nbulk + (runs ? (int)ghosts : 0), st>>>(src, L, bc_view(g, comp), b0 + c0, pz, dv,
                                                                            apply_bc, nbulk, g->d_err, out);
        } else {
            auto kernel = L.tensorial ? lab_fill_kernel<T, true> : lab_fill_kernel<T, false>;
            kernel<<<grid, threads, nbulk, st>>>(src, L, bc_view(g, comp), b0 + c0, pz, dv, wl, apply_bc, nbulk,
                                                 g->d_err, out);
        }
    }
    CN_CUDA_TRY(cudaGetLastError());
    return CN_OK;
}

} // namespace cn

using namespace cn;

extern "C" cn_status cn_lab_fill(cn_grid *g, int comp, const cn_stencil *s, int block_begin,
                                 int block_count, int apply_bc, void *d_labs, void *stream)
{
    if (!g) {
        return fail(CN_ERR_NOT_ALLOCATED, "FieldLab: can not load lab data when not allocated first");
    }
    if (comp < 0 || comp >= g->ncomp) {
        return fail(CN_ERR_INVALID_ARGUMENT, "cn_lab_fill: bad component");
    }
    if (!d_labs) {
        return fail(CN_ERR_NOT_ALLOCATED, "FieldLab: can not load lab data when not allocated first");
    }
    cn_status st = check_lab(g, s);
    if (st != CN_OK) return st;
    if (block_begin < 0 || block_count < 0 || block_begin + (int64_t)block_count > g->nblocks) {
        return fail(CN_ERR_INVALID_ARGUMENT, "cn_lab_fill: block range outside the grid");
    }
    if (block_count == 0) return CN_OK;
    cudaStream_t cs = as_stream(stream);
    st = sync_bc(g, cs);
    if (st != CN_OK) return st;
    switch (g->dtype) {
    case CN_FLOAT64:
        return launch_fill<double>(g, comp, s, block_begin, block_count, apply_bc, d_labs, cs);
    case CN_FLOAT32:
        return launch_fill<float>(g, comp, s, block_begin, block_count, apply_bc, d_labs, cs);
    case CN_INT32:
        return launch_fill<int32_t>(g, comp, s, block_begin, block_count, apply_bc, d_labs, cs);
    }
    return fail(CN_ERR_UNSUPPORTED, "cn_lab_fill: dtype");
}
