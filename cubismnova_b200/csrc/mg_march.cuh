// mg_march.cuh -- the multigrid level operators as marching kernels, for fields
// without BCs (periodic neighbours are cells at a constant offset).
//
// A thread owns V cells of a row (16 bytes where rows allow it) over a run of
// planes and marches up it: p of planes z - 1 and z and the z face means stay
// in registers, everything else is a cached load issued before anything waits.
// Fields with BCs take the tile kernels of mg.cu.  Operations and their order
// are those of the tile kernels (op7_tile), uncontracted, so results are bit
// for bit the same.
//
// The operator is stored as one harmonic mean per face: per cell the means
// across its lower x, y, z faces, and per block those across its upper
// boundary faces (harm is symmetric to the bit, so a face has one value from
// either side), 12 B per cell in FP32.  Sweeps that only need the right-hand side
// (the first one, from a zero guess) ride on the kernel that makes it, and the
// FP64 accumulation on the last sweep.
//
// Bound by DRAM at the fine levels: on 256^3 cells (B200) a sweep takes 73 us
// (24 B per cell, 85 % of the copy bandwidth; 156 with the tile kernel), the
// restricted residual 69 (150), the prolongation 25 (99), the last sweep with
// the accumulation 103 (156 + 60), the FP64 residual with the next cycle's
// first sweep 166 (243 + 156 + 16).  A solve to 1e-8 went from 23.0 to 10.2
// ms, of 64^3 cells from 2.41 to 1.43 ms.
#pragma once

#include "cn_fastdiv.h"
#include "cn_internal.h"
#include "mg_internal.h"

#include <cstring>

namespace cn {
namespace mg {

// Geometry and thread layout of a marching launch over a level (indices are
// 32-bit: a level has fewer than 2^32 stored elements; differences wrap).
struct Layer {
    int n[3], nb[3];
    uint32_t bs, bs64;        // block strides of the FP32 fields and of p64
    int TZ, total;            // planes per thread, threads
    FastDiv per_block, plane, row, nb0, nb1;
};

// V consecutive values loaded and stored as one
template <typename T, int V> struct alignas(sizeof(T) * V) Vec {
    T v[V];
};
template <typename T, int V> __device__ __forceinline__ Vec<T, V> ldv(const T *p)
{
    Vec<T, V> r;
    if constexpr (sizeof(T) * V == 16) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(p));
        memcpy(&r, &q, 16);
    } else if constexpr (sizeof(T) * V == 8) {
        const uint2 q = __ldg(reinterpret_cast<const uint2 *>(p));
        memcpy(&r, &q, 8);
    } else {
        static_assert(V == 1, "16, 8 or one value");
        r.v[0] = __ldg(p);
    }
    return r;
}
// the same of data that other CTAs of a running kernel have written (from L2)
template <typename T, int V> __device__ __forceinline__ Vec<T, V> ldv_l2(const T *p)
{
    Vec<T, V> r;
    if constexpr (sizeof(T) * V == 16) {
        const uint4 q = __ldcg(reinterpret_cast<const uint4 *>(p));
        memcpy(&r, &q, 16);
    } else if constexpr (sizeof(T) * V == 8) {
        const uint2 q = __ldcg(reinterpret_cast<const uint2 *>(p));
        memcpy(&r, &q, 8);
    } else {
        static_assert(V == 1, "16, 8 or one value");
        r.v[0] = __ldcg(p);
    }
    return r;
}
// L2: the field may have been written by other CTAs of this kernel
template <bool L2, typename T, int V> __device__ __forceinline__ Vec<T, V> ldf(const T *p)
{
    if constexpr (L2) return ldv_l2<T, V>(p);
    return ldv<T, V>(p);
}
template <typename T, int V> __device__ __forceinline__ void stv(T *p, const Vec<T, V> &r)
{
    *reinterpret_cast<Vec<T, V> *>(p) = r;
}

struct Column {
    int block, x, y, z0, z1;
    int b[3];
};
// the thread's cells: V along x, R rows
template <int V, int R> __device__ __forceinline__ bool column(const Layer &g, Column &c, int t)
{
    if (t >= g.total) return false;
    c.block = g.per_block.div(t);
    const int r = t - c.block * (int)g.per_block.d, zc = g.plane.div(r), q = r - zc * (int)g.plane.d, y = g.row.div(q);
    c.x = V * (q - y * (int)g.row.d);
    c.y = R * y;
    c.z0 = zc * g.TZ;
    c.z1 = min(c.z0 + g.TZ, g.n[2]);
    const int b12 = g.nb0.div(c.block);
    c.b[0] = c.block - b12 * (int)g.nb0.d;
    c.b[2] = g.nb1.div(b12);
    c.b[1] = b12 - c.b[2] * (int)g.nb1.d;
    return true;
}
// index distance to the neighbour on side s of direction d for a cell at
// coordinate q (stride st; n cells a block, block stride bs)
__device__ __forceinline__ uint32_t step_to(const Layer &g, const Column &c, int d, int s, int q, int n, uint32_t st,
                                            uint32_t bs)
{
    const uint32_t one = s ? st : 0u - st;
    if (s ? q + 1 < n : q > 0) return one;
    const int m = g.nb[d], b = c.b[d], nbr = s ? (b + 1 < m ? b + 1 : 0) : (b > 0 ? b - 1 : m - 1);
    const uint32_t bd = (uint32_t)(nbr - b) * (d == 0 ? 1u : (d == 1 ? (uint32_t)g.nb[0] : (uint32_t)(g.nb[0] * g.nb[1])));
    return one + bd * bs + (s ? 0u - (uint32_t)n * st : (uint32_t)n * st);
}

// L p and D of one cell from its neighbours and face means
template <typename T>
__device__ __forceinline__ void op7_faces(T pc, T xm, T xp, T ym, T yp, T zm, T zp, T kxm, T kxp, T kym, T kyp, T kzm, T kzp,
                                          T ih2, T &Lp, T &D)
{
    const T f0 = kxp * (xp - pc) - kxm * (pc - xm);
    const T f1 = kyp * (yp - pc) - kym * (pc - ym);
    const T f2 = kzp * (zp - pc) - kzm * (pc - zm);
    Lp = ih2 * ((f0 + f1) + f2);
    const T s0 = kxp + kxm, s1 = kyp + kym, s2 = kzp + kzm;
    D = ih2 * ((s0 + s1) + s2);
}

// What one plane of a column of R rows reads beside planes z - 1 and z.
template <typename T, int V, int R> struct Plane7 {
    Vec<T, V> vz[R], ym, yp, kx[R], ky[R + 1], kz[R];
    T xm[R], xp[R], kxe[R];
};
// Where a column stands: indices of its first row in the field and in the
// dense face arrays, and the offsets to its neighbours.
template <typename T, int V, int R, bool L2 = false> struct Walk {
    uint32_t o, q;                 // field, dense
    uint32_t n0, s2;               // row and plane strides
    uint32_t xm, xp, ym, yp, zp;   // neighbour distances (zp: of the block's last plane)
    const T *kxe, *kye, *kze;      // upper means: x of the last cell, y of the last row, z of the last plane
    uint32_t sxe, rxe, sye;        // their strides per plane (and per row)
    Vec<T, V> a[R], b[R], kzm[R];  // planes z - 1 and z, lower z means

    __device__ __forceinline__ void start(const Layer &g, const Column &c, const Faces<T> &F, const T *p, uint32_t bs)
    {
        const uint32_t n1 = g.n[1], n2 = g.n[2], cells = (uint32_t)g.n[0] * n1 * n2, blk = (uint32_t)c.block;
        n0 = (uint32_t)g.n[0];
        s2 = n0 * n1;
        const uint32_t in = c.x + n0 * (c.y + n1 * (uint32_t)c.z0);
        o = blk * bs + in;
        q = blk * cells + in;
        xm = step_to(g, c, 0, 0, c.x, g.n[0], 1, bs);
        xp = step_to(g, c, 0, 1, c.x + V - 1, g.n[0], 1, bs);
        ym = step_to(g, c, 1, 0, c.y, g.n[1], n0, bs);
        yp = step_to(g, c, 1, 1, c.y + R - 1, g.n[1], n0, bs);
        zp = step_to(g, c, 2, 1, g.n[2] - 1, g.n[2], s2, bs);
        if (c.x + V < g.n[0]) {
            kxe = F.k[0] + q + V;
            sxe = s2;
            rxe = n0;
        } else {
            kxe = F.u[0] + blk * (n1 * n2) + c.y + n1 * (uint32_t)c.z0;
            sxe = n1;
            rxe = 1;
        }
        if (c.y + R < g.n[1]) {
            kye = F.k[1] + q + R * n0;
            sye = s2;
        } else {
            kye = F.u[1] + blk * (n0 * n2) + c.x + n0 * (uint32_t)c.z0;
            sye = n0;
        }
        kze = F.u[2] + blk * s2 + c.x + n0 * (uint32_t)c.y;
        const uint32_t zm = step_to(g, c, 2, 0, c.z0, g.n[2], s2, bs);
#pragma unroll
        for (int r = 0; r < R; ++r) {
            a[r] = ldf<L2, T, V>(p + (uint32_t)(o + r * n0 + zm));
            b[r] = ldf<L2, T, V>(p + (uint32_t)(o + r * n0));
            kzm[r] = ldv<T, V>(F.k[2] + (uint32_t)(q + r * n0));
        }
    }
    // loads of the plane at (o + k s2); last: the block's last plane
    __device__ __forceinline__ void fetch(const Faces<T> &F, const T *p, uint32_t k, bool last, Plane7<T, V, R> &f) const
    {
        const uint32_t oo = o + k * s2, qq = q + k * s2;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const uint32_t orow = oo + r * n0, qrow = qq + r * n0;
            f.vz[r] = ldf<L2, T, V>(p + (uint32_t)(orow + (last ? zp : s2)));
            f.kz[r] = ldv<T, V>(last ? kze + r * n0 : F.k[2] + (uint32_t)(qrow + s2));
            f.kx[r] = ldv<T, V>(F.k[0] + qrow);
            f.kxe[r] = __ldg(kxe + (uint32_t)(k * sxe + r * rxe));
            f.xm[r] = ldf<L2, T, 1>(p + (uint32_t)(orow + xm)).v[0];
            f.xp[r] = ldf<L2, T, 1>(p + (uint32_t)(orow + (V - 1) + xp)).v[0];
            f.ky[r] = ldv<T, V>(F.k[1] + qrow);
        }
        f.ky[R] = ldv<T, V>(kye + (uint32_t)(k * sye));
        f.ym = ldf<L2, T, V>(p + (uint32_t)(oo + ym));
        f.yp = ldf<L2, T, V>(p + (uint32_t)(oo + (R - 1) * n0 + yp));
    }
    // L p and D of the plane's cell (row r, i); advance() goes to the next plane
    __device__ __forceinline__ void eval(const Plane7<T, V, R> &f, int r, int i, T ih2, T &Lp, T &D) const
    {
        const T xl = i > 0 ? b[r].v[i > 0 ? i - 1 : 0] : f.xm[r];
        const T xr = i + 1 < V ? b[r].v[i + 1 < V ? i + 1 : 0] : f.xp[r];
        const T kr = i + 1 < V ? f.kx[r].v[i + 1 < V ? i + 1 : 0] : f.kxe[r];
        const T yl = r > 0 ? b[r > 0 ? r - 1 : 0].v[i] : f.ym.v[i];
        const T yr = r + 1 < R ? b[r + 1 < R ? r + 1 : 0].v[i] : f.yp.v[i];
        op7_faces<T>(b[r].v[i], xl, xr, yl, yr, a[r].v[i], f.vz[r].v[i], f.kx[r].v[i], kr, f.ky[r].v[i], f.ky[r + 1].v[i],
                     kzm[r].v[i], f.kz[r].v[i], ih2, Lp, D);
    }
    __device__ __forceinline__ void advance(const Plane7<T, V, R> &f)
    {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            a[r] = b[r];
            b[r] = f.vz[r];
            kzm[r] = f.kz[r];
        }
    }
};

// Weighted Jacobi sweep pout = pin + omega (L pin - f) / D; ADD: also p64 += pout.
// Two planes' loads in flight (one: 84 us on 256^3 instead of 73).
template <int V, int U, bool ADD>
__global__ void __launch_bounds__(256)
    jacobi_march(const __grid_constant__ Layer g, const __grid_constant__ Faces<float> F, float ih2, float omega,
                 const float *__restrict__ pin, const float *__restrict__ fin, float *__restrict__ pout,
                 double *__restrict__ p64)
{
    Column c;
    if (!column<V, 1>(g, c, blockIdx.x * 256 + threadIdx.x)) return;
    Walk<float, V, 1> w;
    w.start(g, c, F, pin, g.bs);
    const int planes = c.z1 - c.z0;
    const bool top = c.z1 == g.n[2];
    uint32_t o64 = (uint32_t)c.block * g.bs64 + (w.o - (uint32_t)c.block * g.bs);
    for (int z = 0; z < planes; z += U) {
        Plane7<float, V, 1> f[U];
        Vec<float, V> rhs[U];
        constexpr int W = V >= 2 ? 2 : 1;
        Vec<double, W> acc[U][V / W];
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (U == 1 || z + k < planes) {
                if (ADD) {
#pragma unroll
                    for (int j = 0; j < V / W; ++j)
                        acc[k][j] = *reinterpret_cast<const Vec<double, W> *>(p64 + (uint32_t)(o64 + k * w.s2 + W * j));
                }
                w.fetch(F, pin, k, top && z + k + 1 == planes, f[k]);
                rhs[k] = ldv<float, V>(fin + (uint32_t)(w.o + k * w.s2));
            }
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (U == 1 || z + k < planes) {
                Vec<float, V> r;
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    float Lp, D;
                    w.eval(f[k], 0, i, ih2, Lp, D);
                    r.v[i] = w.b[0].v[i] + omega * ((Lp - rhs[k].v[i]) / D);
                }
                stv<float, V>(pout + (uint32_t)(w.o + k * w.s2), r);
                if (ADD) {
#pragma unroll
                    for (int j = 0; j < V / W; ++j) {
#pragma unroll
                        for (int i = 0; i < W; ++i)
                            acc[k][j].v[i] += (double)r.v[W * j + i];
                        stv<double, W>(p64 + (uint32_t)(o64 + k * w.s2 + W * j), acc[k][j]);
                    }
                }
                w.advance(f[k]);
            }
        w.o += U * w.s2;
        w.q += U * w.s2;
        w.kxe += U * w.sxe;
        w.kye += U * w.sye;
        o64 += U * w.s2;
    }
}

// First Jacobi sweep from a zero guess: p = omega (0 - f) / D, one cell each.
__device__ __forceinline__ float first_sweep(float f, float D, float omega) { return 0.0f + omega * ((0.0f - f) / D); }

__global__ void __launch_bounds__(256) jacobi_first(int64_t total, FastDiv cells, uint32_t bs, const float *__restrict__ D,
                                                    const float *__restrict__ f, float *__restrict__ p, float omega)
{
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < total; i += (int64_t)gridDim.x * 256) {
        const uint32_t b = (uint32_t)cells.div((int)i), o = b * bs + ((uint32_t)i - b * cells.d);
        p[o] = first_sweep(f[o], D[i], omega);
    }
}

// Residual restricted onto the coarse right-hand side, fc = (sum of the 8
// children's f - L p) / 8, children summed in the order
// ((r0+r1)+(r2+r3))+((r4+r5)+(r6+r7)), child c = dx | dy<<1 | dz<<2; a thread
// owns 2 rows and pairs of planes (4 cells a row: 73 us on 256^3, 2 cells: 136).  With pc, also the coarse level's first
// Jacobi sweep from zero (Dc: its dense diagonal).
template <int V, bool L2>
__device__ __forceinline__ void restrict_column(const Layer &g, const Column &c, const Faces<float> &F, float ih2, float omega,
                                                const float *__restrict__ p, const float *__restrict__ fin,
                                                float *__restrict__ fc, float *__restrict__ pc, const float *__restrict__ Dc,
                                                uint32_t bsc)
{
    Walk<float, V, 2, L2> w;
    w.start(g, c, F, p, g.bs);
    const uint32_t m0 = w.n0 / 2, m1 = (uint32_t)g.n[1] / 2, in = c.x / 2 + m0 * (c.y / 2 + m1 * (uint32_t)(c.z0 / 2));
    uint32_t oc = (uint32_t)c.block * bsc + in, qc = (uint32_t)c.block * (m0 * m1 * ((uint32_t)g.n[2] / 2)) + in;
    for (int z = c.z0; z < c.z1; z += 2) {
        float sum[2][V / 2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            Plane7<float, V, 2> f;
            w.fetch(F, p, 0, z + k + 1 == g.n[2], f);
            Vec<float, V> rhs[2];
#pragma unroll
            for (int r = 0; r < 2; ++r)
                rhs[r] = ldf<L2, float, V>(fin + (uint32_t)(w.o + r * w.n0));
            float res[2][V];
#pragma unroll
            for (int r = 0; r < 2; ++r)
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    float Lp, D;
                    w.eval(f, r, i, ih2, Lp, D);
                    res[r][i] = rhs[r].v[i] - Lp;
                }
#pragma unroll
            for (int i = 0; i < V / 2; ++i)
                sum[k][i] = (res[0][2 * i] + res[0][2 * i + 1]) + (res[1][2 * i] + res[1][2 * i + 1]);
            w.advance(f);
            w.o += w.s2;
            w.q += w.s2;
            w.kxe += w.sxe;
            w.kye += w.sye;
        }
        Vec<float, V / 2> s;
#pragma unroll
        for (int i = 0; i < V / 2; ++i)
            s.v[i] = (sum[0][i] + sum[1][i]) * 0.125f;
        stv<float, V / 2>(fc + oc, s);
        if (pc) {
            const Vec<float, V / 2> D = ldv<float, V / 2>(Dc + qc);
            Vec<float, V / 2> e;
#pragma unroll
            for (int i = 0; i < V / 2; ++i)
                e.v[i] = first_sweep(s.v[i], D.v[i], omega);
            stv<float, V / 2>(pc + oc, e);
        }
        oc += m0 * m1;
        qc += m0 * m1;
    }
}

template <int V>
__global__ void __launch_bounds__(256)
    resid_restrict_march(const __grid_constant__ Layer g, const __grid_constant__ Faces<float> F, float ih2, float omega,
                         const float *__restrict__ p, const float *__restrict__ fin, float *__restrict__ fc,
                         float *__restrict__ pc, const float *__restrict__ Dc, uint32_t bsc)
{
    Column c;
    if (column<V, 2>(g, c, blockIdx.x * 256 + threadIdx.x))
        restrict_column<V, false>(g, c, F, ih2, omega, p, fin, fc, pc, Dc, bsc);
}

// p += trilinear interpolation of the coarse correction e (weights 3/4, 1/4
// along x, then y, then z); bsc: e's block stride.
template <int V, bool L2>
__device__ __forceinline__ void prolong_column(const Layer &g, const Column &c, float *__restrict__ p,
                                               const float *__restrict__ e, uint32_t bsc)
{
    constexpr int H = V / 2; // coarse cells under the thread's
    const int m0 = g.n[0] / 2, m1 = g.n[1] / 2, m2 = g.n[2] / 2, X = c.x / 2, Y = c.y / 2;
    const uint32_t t1 = (uint32_t)m0, t2 = (uint32_t)(m0 * m1);
    const uint32_t xl = step_to(g, c, 0, 0, X, m0, 1, bsc), xr = step_to(g, c, 0, 1, X + H - 1, m0, 1, bsc);
    const uint32_t dy = step_to(g, c, 1, c.y & 1, Y, m1, t1, bsc);
    // x and y interpolated values of the thread's cells in the coarse plane
    // whose cell (X, Y) is at index u
    auto plane = [&](uint32_t u) {
        Vec<float, V> r;
        float a[2][V];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const uint32_t w = u + (k ? dy : 0u);
            const float l = ldf<L2, float, 1>(e + (uint32_t)(w + xl)).v[0], h = ldf<L2, float, 1>(e + (uint32_t)(w + (H - 1) + xr)).v[0];
            const Vec<float, H> m = ldf<L2, float, H>(e + w);
#pragma unroll
            for (int i = 0; i < V; ++i) {
                const int j = i >> 1;
                const float v0 = m.v[j];
                const float v1 = (i & 1) ? (j + 1 < H ? m.v[j + 1 < H ? j + 1 : 0] : h) : (j > 0 ? m.v[j > 0 ? j - 1 : 0] : l);
                a[k][i] = 0.75f * v0 + 0.25f * v1;
            }
        }
#pragma unroll
        for (int i = 0; i < V; ++i)
            r.v[i] = 0.75f * a[0][i] + 0.25f * a[1][i];
        return r;
    };
    const int Z0 = c.z0 / 2;
    uint32_t u = (uint32_t)c.block * bsc + X + t1 * Y + t2 * Z0;
    const uint32_t top = step_to(g, c, 2, 1, m2 - 1, m2, t2, bsc);
    uint32_t o = (uint32_t)c.block * g.bs + c.x + (uint32_t)g.n[0] * (c.y + (uint32_t)g.n[1] * (uint32_t)c.z0);
    const uint32_t s2 = (uint32_t)(g.n[0] * g.n[1]);
    Vec<float, V> bm = plane(u + step_to(g, c, 2, 0, Z0, m2, t2, bsc)), bc = plane(u);
    for (int z = c.z0; z < c.z1; z += 2) {
        const Vec<float, V> bn = plane(u + (z / 2 + 1 < m2 ? t2 : top));
        Vec<float, V> q0 = ldv_l2<float, V>(p + o), q1 = ldv_l2<float, V>(p + (uint32_t)(o + s2));
#pragma unroll
        for (int i = 0; i < V; ++i) {
            q0.v[i] = q0.v[i] + (0.75f * bc.v[i] + 0.25f * bm.v[i]);
            q1.v[i] = q1.v[i] + (0.75f * bc.v[i] + 0.25f * bn.v[i]);
        }
        stv<float, V>(p + o, q0);
        stv<float, V>(p + (uint32_t)(o + s2), q1);
        bm = bc;
        bc = bn;
        u += t2;
        o += 2 * s2;
    }
}

template <int V>
__global__ void __launch_bounds__(256)
    prolong_march(const __grid_constant__ Layer g, float *__restrict__ p, const float *__restrict__ e, uint32_t bsc)
{
    Column c;
    if (column<V, 1>(g, c, blockIdx.x * 256 + threadIdx.x)) prolong_column<V, false>(g, c, p, e, bsc);
}

// Sum of the CTA's (a, b) in thread 0 (256 threads), fixed order.
__device__ __forceinline__ void cta_sum2(double &a, double &b, double (*sh)[8])
{
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, off);
        b += __shfl_down_sync(0xffffffffu, b, off);
    }
    const int w = threadIdx.x >> 5;
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        sh[0][w] = a;
        sh[1][w] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        a = b = 0;
        for (int i = 0; i < 8; ++i) {
            a += sh[0][i];
            b += sh[1][i];
        }
    }
}

// FP64 residual of the outer iteration: r = f - L p64, r32 = (float) r, the
// first Jacobi sweep on it from zero (p0, optional), and the sums of r^2 and
// f^2: per-CTA partials that the last CTA to finish adds in order into out
// (`done` counts CTAs and is left at 0).  Compiled for three CTAs per SM (82
// registers without, two CTAs: 198 us on 256^3 instead of 166).
template <int V, int U>
__global__ void __launch_bounds__(256, 3)
    resid64_march(const __grid_constant__ Layer g, const __grid_constant__ Faces<double> F, double ih2, float omega,
                  const double *__restrict__ p64, const float *__restrict__ fin, float *__restrict__ r32,
                  float *__restrict__ p0, const float *__restrict__ D, double *partials, unsigned *done, double *out)
{
    __shared__ double sh[2][8];
    __shared__ bool last;
    double rr = 0, ff = 0;
    Column c;
    if (column<V, 1>(g, c, blockIdx.x * 256 + threadIdx.x)) {
        Walk<double, V, 1> w;
        w.start(g, c, F, p64, g.bs64);
        const int planes = c.z1 - c.z0;
        const bool top = c.z1 == g.n[2];
        uint32_t o32 = (uint32_t)c.block * g.bs + (w.o - (uint32_t)c.block * g.bs64);
        for (int z = 0; z < planes; z += U) {
            Plane7<double, V, 1> f[U];
            Vec<float, V> rhs[U], d[U];
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (U == 1 || z + k < planes) {
                    w.fetch(F, p64, k, top && z + k + 1 == planes, f[k]);
                    rhs[k] = ldv<float, V>(fin + (uint32_t)(o32 + k * w.s2));
                    if (p0) d[k] = ldv<float, V>(D + (uint32_t)(w.q + k * w.s2));
                }
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (U == 1 || z + k < planes) {
                    Vec<float, V> r, e;
#pragma unroll
                    for (int i = 0; i < V; ++i) {
                        double Lp, unused;
                        w.eval(f[k], 0, i, ih2, Lp, unused);
                        const double fc = (double)rhs[k].v[i], q = fc - Lp;
                        r.v[i] = (float)q;
                        rr += q * q;
                        ff += fc * fc;
                        if (p0) e.v[i] = first_sweep(r.v[i], d[k].v[i], omega);
                    }
                    if (r32) stv<float, V>(r32 + (uint32_t)(o32 + k * w.s2), r);
                    if (p0) stv<float, V>(p0 + (uint32_t)(o32 + k * w.s2), e);
                    w.advance(f[k]);
                }
            w.o += U * w.s2;
            w.q += U * w.s2;
            w.kxe += U * w.sxe;
            w.kye += U * w.sye;
            o32 += U * w.s2;
        }
    }
    cta_sum2(rr, ff, sh);
    if (threadIdx.x == 0) {
        partials[2 * blockIdx.x] = rr;
        partials[2 * blockIdx.x + 1] = ff;
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    rr = ff = 0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += 256) {
        rr += __ldcg(partials + 2 * i);
        ff += __ldcg(partials + 2 * i + 1);
    }
    cta_sum2(rr, ff, sh);
    if (threadIdx.x == 0) {
        out[0] = rr;
        out[1] = ff;
        *done = 0;
        __threadfence_system();
    }
}

// ---------------------------------------------------------------------------
// The coarse levels of a V-cycle in one launch.  From the first level of at
// most kTailCells cells down to the coarsest (solved by its dense inverse) the
// operators are a few hundred nanoseconds of work each, so launches dominate:
// a cluster of kTailCtas CTAs walks through all of them with a cluster barrier
// between one operator and the next (about 2 us an operator, all latency,
// against 4 for a launch; with the 32^3 level in it the two break even).  The
// fields stay in L2 (read past L1, since other CTAs write them); results are
// those of the separate kernels.
// ---------------------------------------------------------------------------
constexpr int kTailCells = 4096, kTailLevels = 8, kTailCtas = 8, kTailThreads = 512;

struct TailLevel {
    Layer one, two, pro; // layouts of the sweeps (V = 2), the restriction (2 x 2 rows), the prolongation
    Faces<float> F;
    const float *D;
    float *p, *pt, *f;
    float ih2;
};
struct Tail {
    TailLevel lev[kTailLevels];
    int levels;      // the last one is the coarsest
    int nu1, nu2;
    float omega;
    int first_done;  // the first sweep of the top level is in pt
    const double *inv; // dense inverse of the coarsest operator
    int N;
};

__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// coarsest_dense_kernel's solve, 32 rows per group of 8 warps
__device__ __forceinline__ void tail_coarsest(const Tail &t, double *b, double (*red)[8][32], double *wsum)
{
    const TailLevel &c = t.lev[t.levels - 1];
    const Layer &g = c.one;
    const int N = t.N, GX = g.nb[0] * g.n[0], GY = g.nb[1] * g.n[1];
    auto offset = [&](int i) {
        const int gx = i % GX, gy = (i / GX) % GY, gz = i / (GX * GY);
        const int blk = gx / g.n[0] + g.nb[0] * (gy / g.n[1] + g.nb[1] * (gz / g.n[2]));
        return (uint32_t)blk * g.bs + (gx % g.n[0]) + g.n[0] * ((gy % g.n[1]) + g.n[1] * (gz % g.n[2]));
    };
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < 8) {
        double s = 0;
        for (int i = threadIdx.x; i < N; i += 256) {
            b[i] = -(double)__ldcg(c.f + offset(i));
            s += b[i];
        }
        for (int off = 16; off > 0; off >>= 1) s += __shfl_down_sync(0xffffffffu, s, off);
        if (lane == 0) wsum[warp] = s;
    }
    __syncthreads();
    double tot = 0;
    for (int w = 0; w < 8; ++w) tot += wsum[w];
    const double mean = tot / N;
    for (int i = threadIdx.x; i < N; i += kTailThreads) b[i] -= mean;
    __syncthreads();
    const int group = warp >> 3, w8 = warp & 7, per = (N + 7) / 8, j0 = w8 * per, j1 = min(N, j0 + per);
    for (int r0 = (int)(blockIdx.x * (kTailThreads / 256)) * 32; r0 < N; r0 += kTailCtas * (kTailThreads / 256) * 32) {
        const int row = r0 + group * 32 + lane;
        double acc = 0;
        if (row < N)
            for (int j = j0; j < j1; ++j) acc += __ldg(t.inv + (int64_t)j * N + row) * b[j];
        red[group][w8][lane] = acc;
        __syncthreads();
        if (w8 == 0 && row < N) {
            double x = 0;
            for (int w = 0; w < 8; ++w) x += red[group][w][lane];
            c.p[offset(row)] = (float)x;
        }
        __syncthreads();
    }
}

__global__ void __cluster_dims__(kTailCtas, 1, 1) __launch_bounds__(kTailThreads)
    tail_kernel(const __grid_constant__ Tail t)
{
    __shared__ double b[512];
    __shared__ double red[kTailThreads / 256][8][32];
    __shared__ double wsum[8];
    const int tid = blockIdx.x * kTailThreads + threadIdx.x, all = kTailCtas * kTailThreads;
    auto sweep = [&](const TailLevel &L, const float *src, float *dst) {
        for (int i = tid; i < L.one.total; i += all) {
            Column c;
            column<2, 1>(L.one, c, i);
            Walk<float, 2, 1, true> w;
            w.start(L.one, c, L.F, src, L.one.bs);
            for (int z = c.z0; z < c.z1; ++z) {
                Plane7<float, 2, 1> f;
                w.fetch(L.F, src, 0, z + 1 == L.one.n[2], f);
                const Vec<float, 2> rhs = ldv_l2<float, 2>(L.f + w.o);
                Vec<float, 2> r;
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    float Lp, D;
                    w.eval(f, 0, k, L.ih2, Lp, D);
                    r.v[k] = w.b[0].v[k] + t.omega * ((Lp - rhs.v[k]) / D);
                }
                stv<float, 2>(dst + w.o, r);
                w.advance(f);
                w.o += w.s2;
                w.q += w.s2;
                w.kxe += w.sxe;
                w.kye += w.sye;
            }
        }
        cluster_sync();
    };
    const int last = t.levels - 1;
#pragma unroll 1
    for (int l = 0; l < last; ++l) {
        const TailLevel &L = t.lev[l];
        float *p = L.p, *q = L.pt;
        if (t.nu1 == 0 || (l == 0 && !t.first_done)) {
            // zero, or the first sweep from zero
            const int cells = L.one.n[0] * L.one.n[1] * L.one.n[2];
            float *dst = t.nu1 ? q : p;
            for (int i = tid; i < (int)(L.one.nb[0] * L.one.nb[1] * L.one.nb[2]) * cells; i += all) {
                const int bl = i / cells;
                const uint32_t o = (uint32_t)bl * L.one.bs + (i - bl * cells);
                dst[o] = t.nu1 ? first_sweep(__ldcg(L.f + o), __ldg(L.D + i), t.omega) : 0.0f;
            }
            cluster_sync();
        }
#pragma unroll 1
        for (int s = 0; s < t.nu1; ++s) {
            float *src = p;
            p = q;
            q = src;
            if (s > 0) sweep(L, src, p);
        }
        const TailLevel &C = t.lev[l + 1];
        const bool first = l + 1 < last && t.nu1 > 0;
        for (int i = tid; i < L.two.total; i += all) {
            Column c;
            column<2, 2>(L.two, c, i);
            restrict_column<2, true>(L.two, c, L.F, L.ih2, t.omega, p, L.f, C.f, first ? C.pt : nullptr, C.D, C.one.bs);
        }
        cluster_sync();
    }
    tail_coarsest(t, b, red, wsum);
    cluster_sync();
#pragma unroll 1
    for (int l = last - 1; l >= 0; --l) {
        const TailLevel &L = t.lev[l], &C = t.lev[l + 1];
        // where this level's and the coarser one's solutions are after their sweeps
        float *p = (t.nu1 & 1) ? L.pt : L.p, *q = (t.nu1 & 1) ? L.p : L.pt;
        const float *e = l + 1 < last && ((t.nu1 + t.nu2) & 1) ? C.pt : C.p;
        for (int i = tid; i < L.pro.total; i += all) {
            Column c;
            column<2, 1>(L.pro, c, i);
            prolong_column<2, true>(L.pro, c, p, e, C.one.bs);
        }
        cluster_sync();
#pragma unroll 1
        for (int s = 0; s < t.nu2; ++s) {
            float *src = p;
            p = q;
            q = src;
            sweep(L, src, p);
        }
    }
}

} // namespace mg
} // namespace cn
