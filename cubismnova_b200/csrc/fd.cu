// fd.cu -- K1: lab fill fused with the 2nd-order finite-difference stencils
// (7-point Laplacian, central gradient, divergence) and the ddx kernel ABI.
//
// Design.  A thread owns V cells of a row (16 bytes where rows allow it) over a
// run of TZ planes and marches up it: the z neighbours stay in registers, the
// x and y neighbours are cached loads, across a face of the block at a
// constant offset in the neighbour block.  Threads run over all columns of all
// blocks, x fastest, so that blocks of any extent fill the warps.  Cells beside
// faces that carry a BC or a skipped neighbour are left to other CTAs of the
// same launch, which find what lies behind each face once (Absorbing and
// Symmetry lead to the own cell at ghost width 1, Dirichlet and undefined cells
// to a constant): together the lab of a stencil (-1,2) non-tensorial
// (Block/FieldLab.h:180-224).
//
// Bound by DRAM at large sizes and by latency and the launch at small ones.
// Against tiles staged in shared memory (one bulk copy per z slab, faces cell
// by cell), B200: Laplacian + gradient FP64 128^3 22.3 -> 18.5 us, 512^3 1003
// -> 891 us (94 % of the copy bandwidth); divergence FP64 512^3 2161 -> 705
// us, FP32 on 30 x 33 x 27 blocks with walls (25.7 M cells) 406 -> 81 us;
// Laplacian FP32 512^3 793 -> 199 us.  BC code inlined into the march cost the
// registers of a third of the warps (84 -> 107 us on the ragged case).
//
// Faces with BCs: a few CTAs that walked their cells one face after the other,
// each cell with its own chain of BC loads, set the time of small grids and of
// large faces.  FP64 Laplacian with walls, that -> now: 128^3 25 -> 15 us, 36 x
// 36 x 200 blocks (2.1 M cells) 95 -> 15, one block of 32^3 24 -> 7; a BC on every
// face of every 8^3 block of 128^3 179 -> 48.
//
// Arithmetic uses __d*_rn / __f*_rn intrinsics so nothing is contracted into
// an FMA: results are bit-identical to the reference loops compiled without
// contraction (Kernel/Laplacian/Laplacian.cpp:123-130,
// Kernel/Divergence/nova/nova.cpp:113-126, ISPC .../ddxGold.cpp:9-33).
#include <algorithm>
#include <cstring>

#include "cn_fastdiv.h"
#include "cn_internal.h"

namespace cn {

template <typename T> struct Arith;
template <> struct Arith<double> {
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
};
template <> struct Arith<float> {
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
};

// Largest block plane the operators take, a limit of the interface that the
// kernel does not need: a plane with the planes and rows around it, each array
// padded to 4 elements, within 100 KB (square planes up to 36 cells for the
// FP64 divergence, 64 for an FP64 Laplacian).
constexpr size_t kMaxPlaneBytes = 100 * 1024 - 128;
static size_t plane_bytes(int n0, int n1, size_t es, int nc)
{
    auto pad4 = [](size_t n) { return (n + 3) & ~(size_t)3; };
    return (3 * pad4((size_t)n0 * n1) + 2 * (pad4(n0) + pad4(n1))) * es * nc;
}

enum FdOp { kLap = 0, kGrad = 1, kLapGrad = 2, kDiv = 3 };

template <typename T> struct FdParams {
    const T *in[3];  // component read along x, y, z (kDiv: 3 components, else the same)
    BcView bc[3];
    LabGeom L;
    T *lap;          // kLap / kLapGrad / kDiv output component base
    T *grad;         // kGrad / kLapGrad: first of 3 components
    int64_t out_cstride;
    T ih[3], ih2[3];
    int TZ, block0, total;       // planes per thread, first block and threads of this launch
    uint32_t face_share;          // share of CTAs that look at faces, / 2^32
    FastDiv per_block, plane, n0; // threads per block, N0 * N1, N0
    FastDiv nb0, nb1, f0, f1;     // blocks along x, y; N0, N1
    int xw;                       // cells of a row beside x faces that bc_faces takes
    FastDiv fxw;
    int faces, faces_per_cta, parts; // faces of this launch's blocks; see bc_faces
};

// Outputs of one cell from its six neighbours (kDiv: x neighbours of the
// first component, y of the second, z of the third; c0 unused).
template <typename T, int OP>
__device__ __forceinline__ void cell_eval(const FdParams<T> &p, T c0, T xp, T xm, T yp, T ym, T zp, T zm,
                                          T &lap, T &g0, T &g1, T &g2)
{
    using A = Arith<T>;
    if (OP == kDiv) {
        const T t0 = A::mul(A::sub(xp, xm), p.ih[0]);
        const T t1 = A::mul(A::sub(yp, ym), p.ih[1]);
        const T t2 = A::mul(A::sub(zp, zm), p.ih[2]);
        lap = A::mul(T(0.5), A::add(A::add(t0, t1), t2));
        return;
    }
    if (OP == kLap || OP == kLapGrad) {
        const T c2 = A::mul(T(2), c0);
        const T ddx = A::mul(p.ih2[0], A::add(A::sub(xp, c2), xm));
        const T ddy = A::mul(p.ih2[1], A::add(A::sub(yp, c2), ym));
        const T ddz = A::mul(p.ih2[2], A::add(A::sub(zp, c2), zm));
        lap = A::add(A::add(ddx, ddy), ddz);
    }
    if (OP == kGrad || OP == kLapGrad) {
        g0 = A::mul(T(0.5), A::mul(A::sub(xp, xm), p.ih[0]));
        g1 = A::mul(T(0.5), A::mul(A::sub(yp, ym), p.ih[1]));
        g2 = A::mul(T(0.5), A::mul(A::sub(zp, zm), p.ih[2]));
    }
}

// V consecutive cells of a row, loaded and stored as one (V * sizeof(T) <= 16
// bytes, aligned: row lengths are multiples of V then).
template <typename T, int V> struct alignas(sizeof(T) * V) Pack {
    T v[V];
};
template <typename T, int V> __device__ __forceinline__ Pack<T, V> load(const T *p)
{
    Pack<T, V> r;
    if constexpr (sizeof(T) * V == 16) {
        const uint4 q = __ldg(reinterpret_cast<const uint4 *>(p));
        memcpy(&r, &q, 16);
    } else if constexpr (sizeof(T) * V == 8) {
        const uint2 q = __ldg(reinterpret_cast<const uint2 *>(p));
        memcpy(&r, &q, 8);
    } else {
        r.v[0] = __ldg(p);
    }
    return r;
}
template <typename T, int V> __device__ __forceinline__ void store(T *p, const Pack<T, V> &r)
{
    *reinterpret_cast<Pack<T, V> *>(p) = r;
}

// One thread's run of planes from cell o, all neighbours plain cells: U planes
// at a time, their loads before their stores.  zm, zp: offsets of the lower
// neighbour of the first plane and of the upper one of the last.
template <typename T, int OP, int V, int U>
__device__ __forceinline__ void march(const FdParams<T> &p, int64_t o, int64_t s2, int planes, int64_t xm, int64_t xp,
                                      int64_t ym, int64_t yp, int64_t zm, int64_t zp)
{
    using P = Pack<T, V>;
    const T *px = p.in[0] + o, *py = p.in[1] + o, *pz = p.in[2] + o;
    T *lap = p.lap + o, *grad = p.grad + o;
    P a = load<T, V>(pz + zm), b = load<T, V>(pz); // planes z - 1 and z
    for (int z = 0; z < planes; z += U) {
        P vz[U], vym[U], vyp[U], vx[U];
        Pack<T, 1> vxm[U], vxp[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (U == 1 || z + k < planes) {
                vz[k] = load<T, V>(pz + (z + k + 1 == planes ? zp : s2));
                vym[k] = load<T, V>(py + ym);
                vyp[k] = load<T, V>(py + yp);
                if (OP == kDiv && V > 1) vx[k] = load<T, V>(px);
                vxm[k] = load<T, 1>(px + xm);
                vxp[k] = load<T, 1>(px + (V - 1) + xp);
                px += s2;
                py += s2;
                pz += s2;
            }
        }
#pragma unroll
        for (int k = 0; k < U; ++k) {
            if (U == 1 || z + k < planes) {
                P l, g0, g1, g2;
                const P &c = OP == kDiv ? vx[k] : b;
#pragma unroll
                for (int i = 0; i < V; ++i) {
                    const T m = i > 0 ? c.v[i > 0 ? i - 1 : 0] : vxm[k].v[0];
                    const T q = i + 1 < V ? c.v[i + 1 < V ? i + 1 : 0] : vxp[k].v[0];
                    cell_eval<T, OP>(p, b.v[i], q, m, vyp[k].v[i], vym[k].v[i], vz[k].v[i], a.v[i], l.v[i], g0.v[i],
                                     g1.v[i], g2.v[i]);
                }
                if (OP == kLap || OP == kLapGrad || OP == kDiv) {
                    store<T, V>(lap, l);
                    lap += s2;
                }
                if (OP == kGrad || OP == kLapGrad) {
                    store<T, V>(grad, g0);
                    store<T, V>(grad + p.out_cstride, g1);
                    store<T, V>(grad + 2 * p.out_cstride, g2);
                    grad += s2;
                }
                a = b;
                b = vz[k];
            }
        }
    }
}

// offset to a neighbour across a side without BCs: side s of direction d
// (stride st) at coordinate q of block coordinate b
__device__ __forceinline__ int64_t side_offset(const LabGeom &L, int b, int d, int s, int q, int64_t st)
{
    const int n = L.n[d];
    if (s ? q + 1 < n : q > 0) return s ? st : -st;
    const int m = L.nb[d], nbr = s ? (b + 1 < m ? b + 1 : 0) : (b > 0 ? b - 1 : m - 1);
    const int bs = d == 0 ? 1 : (d == 1 ? L.nb[0] : L.nb[0] * L.nb[1]);
    return (s ? st : -st) + (int64_t)(nbr - b) * bs * L.bstride + (s ? -n : n) * st;
}

// What lies behind a face of a block for a cell beside it: the cell at distance
// off (kind 0), times `value` behind Absorbing or Symmetry (kind 2; they lead to
// the own cell), or `value` itself (kind 1).
template <typename T> struct Side {
    int64_t off;
    T value;
    int kind;
};

// The cells beside block faces that carry a BC or a skipped neighbour, which
// the marching threads leave out: `parts` CTAs look at the same few of the
// nblocks * 6 faces and walk the cells of those one after the other, 256 parts
// apart (x faces: the V cells of the columns there).  The BCs are a chain of
// dependent loads, so one thread each finds what lies behind the faces of
// these blocks, for all cells.  Out of line, so that its registers stay its own.
constexpr int kFacesPerCta = 32;                     // at most
constexpr int kFaceBlocks = (kFacesPerCta + 10) / 6; // blocks they belong to, at most
template <typename T, int OP, int V> __device__ __noinline__ void bc_faces(const FdParams<T> &p, int cta)
{
    const LabGeom &L = p.L;
    const int lane = threadIdx.x & 31, group = cta / p.parts, first = group * p.faces_per_cta;
    bool set = false;
    if (lane < p.faces_per_cta && first + lane < p.faces) {
        const int f = (first + lane) % 6;
        const BcView &bc = f < 2 ? p.bc[0] : (f < 4 ? p.bc[1] : p.bc[2]);
        set = (__ldg(bc.faces + p.block0 + (first + lane) / 6) >> f) & 1;
    }
    unsigned m = __ballot_sync(0xffffffffu, set); // the same in all warps
    if (!m) return;
    __shared__ Side<T> sides[kFaceBlocks][6];
    const int64_t s1 = L.n[0], s2 = (int64_t)L.n[0] * L.n[1];
    const int b6 = first / 6;
    if (threadIdx.x < 6 * kFaceBlocks && 6 * b6 + (int)threadIdx.x < p.faces) {
        const int f = threadIdx.x % 6, d = f >> 1, block = p.block0 + b6 + threadIdx.x / 6;
        const int b12 = p.nb0.div(block), b0 = block - b12 * (int)p.nb0.d, b2 = p.nb1.div(b12),
                  b1 = b12 - b2 * (int)p.nb1.d;
        const FaceRule<T> r = face_rule<T>(L, f < 2 ? p.bc[0] : (f < 4 ? p.bc[1] : p.bc[2]), block, d, f & 1);
        Side<T> e = {0, r.value, r.kind == kRuleValue ? 1 : 2};
        if (r.kind == kRuleCopy)
            e = {side_offset(L, pick3(d, b0, b1, b2), d, f & 1, f & 1 ? L.n[d] - 1 : 0, d == 0 ? 1 : (d == 1 ? s1 : s2)), T(1), 0};
        sides[threadIdx.x / 6][f] = e;
    }
    __syncthreads();
    int i = (cta - group * p.parts) * 256 + threadIdx.x; // in the current face
    while (m) {
        const int item = first + __ffs(m) - 1, blk = item / 6, f = item - 6 * blk, d = f >> 1;
        const int n = d == 0 ? p.xw * L.n[1] * L.n[2] : L.n[0] * pick3(d, 0, L.n[2], L.n[1]);
        if (i >= n) {
            i -= n;
            m &= m - 1;
            continue;
        }
        int q[3];
        if (d == 0) {
            const int r = p.fxw.div(i);
            q[2] = p.f1.div(r);
            q[1] = r - q[2] * L.n[1];
            q[0] = i - r * p.xw + (f & 1 ? L.n[0] - p.xw : 0);
        } else {
            const int r = p.f0.div(i);
            q[0] = i - r * L.n[0];
            q[1] = d == 1 ? (f & 1 ? L.n[1] - 1 : 0) : r;
            q[2] = d == 2 ? (f & 1 ? L.n[2] - 1 : 0) : r;
        }
        i += 256 * p.parts;
        const int64_t o = (int64_t)(p.block0 + blk) * L.bstride + q[0] + s1 * q[1] + s2 * q[2];
        const Side<T> *e = sides[blk - b6];
        T v[6]; // lower and upper neighbour along x, y, z
        bool at[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const int64_t st = k < 2 ? 1 : (k < 4 ? s1 : s2);
            at[k] = k & 1 ? q[k >> 1] + 1 == L.n[k >> 1] : q[k >> 1] == 0;
            v[k] = __ldg(p.in[k >> 1] + o + (at[k] ? e[k].off : (k & 1 ? st : -st)));
        }
        const T c = __ldg(p.in[0] + o);
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (at[k] && e[k].kind) v[k] = e[k].kind == 1 ? e[k].value : Arith<T>::mul(e[k].value, v[k]);
        T l, g0, g1, g2;
        cell_eval<T, OP>(p, c, v[1], v[0], v[3], v[2], v[5], v[4], l, g0, g1, g2);
        if (OP == kLap || OP == kLapGrad || OP == kDiv) p.lap[o] = l;
        if (OP == kGrad || OP == kLapGrad) {
            p.grad[o] = g0;
            p.grad[o + p.out_cstride] = g1;
            p.grad[o + 2 * p.out_cstride] = g2;
        }
    }
}

// Resident CTAs per SM: three for the FP64 divergence (78 registers; of 512^3
// cells 705 us, with the four that its 62 registers would allow 816).
// BCS: the grid carries BCs.
template <typename T, int OP> constexpr int min_ctas() { return OP == kDiv && sizeof(T) == 8 ? 3 : 0; }
template <typename T, int OP, int V, int U, bool BCS>
__global__ void __launch_bounds__(256, min_ctas<T, OP>()) fd_kernel(const __grid_constant__ FdParams<T> p)
{
    int cta = blockIdx.x;
    if constexpr (BCS) {
        const int fc = __umulhi(cta, p.face_share); // face CTAs before this one
        if (__umulhi(cta + 1, p.face_share) != fc) {
            bc_faces<T, OP, V>(p, fc);
            return;
        }
        cta -= fc;
    }
    const int t = cta * 256 + threadIdx.x;
    if (t >= p.total) return;
    const LabGeom &L = p.L;
    const int bl = p.per_block.div(t), r = t - bl * (int)p.per_block.d;
    const int zc = p.plane.div(r), c = r - zc * (int)p.plane.d;
    const int y = p.n0.div(c), x = V * (c - y * (int)p.n0.d);
    const int block = p.block0 + bl;
    int z0 = zc * p.TZ, z1 = min(z0 + p.TZ, L.n[2]);
    if constexpr (BCS) {
        // faces of the block that this run touches; those with BCs are bc_faces'
        const unsigned fx = (x < p.xw ? 1u : 0u) | (x + V > L.n[0] - p.xw ? 2u : 0u),
                       fy = (y == 0 ? 4u : 0u) | (y + 1 == L.n[1] ? 8u : 0u),
                       fz = (z0 == 0 ? 16u : 0u) | (z1 == L.n[2] ? 32u : 0u);
        if (fx && (__ldg(p.bc[0].faces + block) & fx)) return;
        if (fy && (__ldg(p.bc[1].faces + block) & fy)) return;
        if (fz) {
            const unsigned f = __ldg(p.bc[2].faces + block) & fz;
            z0 += (f & 16u) ? 1 : 0;
            z1 -= (f & 32u) ? 1 : 0;
        }
        if (z0 >= z1) return;
    }
    const int b12 = p.nb0.div(block), b0 = block - b12 * (int)p.nb0.d;
    const int b2 = p.nb1.div(b12), b1 = b12 - b2 * (int)p.nb1.d;
    const int64_t s1 = L.n[0], s2 = (int64_t)L.n[0] * L.n[1];
    march<T, OP, V, U>(p, (int64_t)block * L.bstride + x + s1 * y + s2 * z0, s2, z1 - z0, side_offset(L, b0, 0, 0, x, 1),
                       side_offset(L, b0, 0, 1, x + V - 1, 1), side_offset(L, b1, 1, 0, y, s1),
                       side_offset(L, b1, 1, 1, y, s1), side_offset(L, b2, 2, 0, z0, s2),
                       side_offset(L, b2, 2, 1, z1 - 1, s2));
}

static cn_status check_out(const cn_grid *in, const cn_grid *out, int out_comp, int ncomp_out)
{
    if (!out) return fail(CN_ERR_INVALID_ARGUMENT, "output grid is NULL");
    if (out->nblocks != in->nblocks || out->n[0] != in->n[0] || out->n[1] != in->n[1] ||
        out->n[2] != in->n[2] || out->dtype != in->dtype)
        return fail(CN_ERR_SIZE_MISMATCH, "Cartesian: Can not assign two grids of unequal size.");
    if (out_comp < 0 || out_comp + ncomp_out > out->ncomp)
        return fail(CN_ERR_INVALID_ARGUMENT, "output component out of range");
    return CN_OK;
}

// Threads that fill the GPU (148 SMs, four CTAs): blocks with fewer columns in
// all are cut into shorter runs of planes; up to twice as many threads, eight
// CTAs, where the runs keep four planes.  B200, lap_grad of 128^3 FP64 from
// memory 22.6 -> 20.5 us with the latter, of 256^3 129 -> 120, divergence of
// 256^3 FP32 51.5 -> 47.5; runs of two planes lose (Laplacian of 128^3 FP32 6.4
// -> 8.2).
constexpr int64_t kFillThreads = 148 * 1024;
constexpr int kLongRun = 4;

template <typename T, int OP, int V> static cn_status launch_march(const cn_grid *u, FdParams<T> &p, cudaStream_t st)
{
    // planes whose loads are in flight together (FP64 divergence: its three
    // fields' loads fill the registers with one, 695 against 837 us on 512^3)
    constexpr int U = OP == kDiv && sizeof(T) == 8 ? 1 : 2;
    const int N2 = u->n[2], cols = u->n[0] / V * u->n[1]; // columns of a block
    const int64_t all = (int64_t)u->nblocks * cols;
    auto run = [&](int64_t threads) { // planes of a run that make `threads` threads
        const int nzc = (int)std::min<int64_t>((N2 + U - 1) / U, std::max<int64_t>(1, (threads + all - 1) / all));
        return ((N2 + nzc - 1) / nzc + U - 1) / U * U;
    };
    p.TZ = std::min(run(kFillThreads), std::max(kLongRun, run(2 * kFillThreads)));
    const int nzc = (N2 + p.TZ - 1) / p.TZ;
    const int per_block = cols * nzc;
    p.per_block = FastDiv((uint32_t)per_block);
    p.plane = FastDiv((uint32_t)cols);
    p.n0 = FastDiv((uint32_t)(u->n[0] / V));
    p.nb0 = FastDiv((uint32_t)u->nb[0]);
    p.nb1 = FastDiv((uint32_t)u->nb[1]);
    p.f0 = FastDiv((uint32_t)u->n[0]);
    p.f1 = FastDiv((uint32_t)u->n[1]);
    // Without BCs nothing is skipped either, and no CTA looks at faces.  A
    // captured call may meet BCs that are pushed later.
    bool bcs = u->bc_count != 0;
    if (!bcs && st) {
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        CN_CUDA_TRY(cudaStreamIsCapturing(st, &cap));
        bcs = cap != cudaStreamCaptureStatusNone;
    }
    // one launch; beyond 2^30 threads or 2^28 blocks, several over block ranges
    const int most = std::min((1 << 30) / per_block, 1 << 28);
    for (p.block0 = 0; p.block0 < u->nblocks; p.block0 += most) {
        p.total = std::min(most, u->nblocks - p.block0) * per_block;
        const int march = (p.total + 255) / 256;
        if (!bcs) {
            fd_kernel<T, OP, V, U, false><<<(unsigned)march, 256, 0, st>>>(p);
        } else {
            // A CTA takes few faces where these are large or few in all, and
            // several CTAs share large ones as long as there are few: at most
            // four per SM.  Face CTAs are spread over the launch, so that the
            // cells beside x faces, parts of sectors, are written when the
            // march writes the rest (the same blocks in order).
            p.faces = p.total / per_block * 6;
            // Cells beside x faces are written apart from the rest of their
            // sector.  For several outputs that do not fit L2 (126 MB) they are
            // taken by whole sectors: Laplacian + gradient of 512^3 FP64 cells
            // with walls 1105 -> 900 us; the Laplacian alone 581 -> 591, and
            // of 128^3 with the gradient 21 -> 25.
            constexpr int sector = 32 / sizeof(T);
            const bool wide = (OP == kGrad || OP == kLapGrad) && V > 1 && u->n[0] % sector == 0 &&
                              (int64_t)u->nblocks * u->block_stride * (int64_t)sizeof(T) * 3 > (126 << 20);
            p.xw = wide ? sector : V;
            p.fxw = FastDiv((uint32_t)p.xw);
            const int large = std::max({p.xw * u->n[1] * N2, u->n[0] * N2, u->n[0] * u->n[1]}); // cells of the largest face
            p.faces_per_cta = std::max(1, std::min({kFacesPerCta, p.faces / (148 * 2) + 1, 8192 / large}));
            const int groups = (p.faces + p.faces_per_cta - 1) / p.faces_per_cta;
            p.parts = std::max(1, std::min((large + 255) / 256, 148 * 4 / groups));
            const int faces = groups * p.parts, ctas = faces + march;
            p.face_share = (uint32_t)((((uint64_t)faces << 32) + ctas - 1) / ctas); // exact: faces of them in all
            fd_kernel<T, OP, V, U, true><<<(unsigned)ctas, 256, 0, st>>>(p);
        }
        CN_CUDA_TRY(cudaGetLastError());
    }
    return CN_OK;
}

template <typename T, int OP>
static cn_status launch_fd(cn_grid *u, int comp, cn_grid *o1, int c1, cn_grid *o2, int c2,
                           cudaStream_t st)
{
    cn_stencil s = {{-1, -1, -1}, {2, 2, 2}, 0};
    cn_status stt = check_lab(u, &s);
    if (stt != CN_OK) return stt;
    stt = sync_bc(u, st);
    if (stt != CN_OK) return stt;
    FdParams<T> p = {};
    p.L = make_geom(u, &s);
    for (int c = 0; c < 3; ++c) {
        const int k = comp + (OP == kDiv ? c : 0);
        p.in[c] = reinterpret_cast<const T *>(u->d_data) + (size_t)k * u->comp_stride;
        p.bc[c] = bc_view(u, k);
    }
    if (o1) p.lap = reinterpret_cast<T *>(o1->d_data) + (size_t)c1 * o1->comp_stride;
    if (o2) {
        p.grad = reinterpret_cast<T *>(o2->d_data) + (size_t)c2 * o2->comp_stride;
        p.out_cstride = o2->comp_stride;
    }
    for (int d = 0; d < 3; ++d) {
        p.ih[d] = (T)(1. / u->h[d]);
        p.ih2[d] = (T)(1. / (u->h[d] * u->h[d]));
    }
    const int N0 = u->n[0], N1 = u->n[1];
    if (plane_bytes(N0, N1, sizeof(T), OP == kDiv ? 3 : 1) > kMaxPlaneBytes)
        return fail(CN_ERR_UNSUPPORTED, "block too large for the fused stencil tile");
    // An output on top of an input would be written while it is read: the march
    // then reads a copy of the inputs.
    const int nin = OP == kDiv ? 3 : 1;
    auto on_input = [&](const cn_grid *o, int c, int n) { return o == u && c < comp + nin && comp < c + n; };
    T *copy = nullptr;
    if (on_input(o1, c1, 1) || on_input(o2, c2, 3)) {
        const size_t bytes = (size_t)nin * u->comp_stride * sizeof(T);
        CN_CUDA_TRY(cudaMallocAsync(&copy, bytes, st));
        CN_CUDA_TRY(cudaMemcpyAsync(copy, p.in[0], bytes, cudaMemcpyDeviceToDevice, st));
        for (int c = 0; c < 3; ++c) p.in[c] = copy + (OP == kDiv ? c * u->comp_stride : 0);
    }
    // cells per thread along x: 16 bytes where rows are multiples of them
    if (sizeof(T) == 4 && N0 % 4 == 0) stt = launch_march<T, OP, 16 / sizeof(T)>(u, p, st);
    else if (N0 % 2 == 0) stt = launch_march<T, OP, 2>(u, p, st);
    else stt = launch_march<T, OP, 1>(u, p, st);
    if (copy) CN_CUDA_TRY(cudaFreeAsync(copy, st));
    return stt;
}

template <int OP>
static cn_status dispatch_fd(cn_grid *u, int comp, int ncin, cn_grid *o1, int c1, cn_grid *o2,
                             int c2, void *stream)
{
    if (!u) return fail(CN_ERR_INVALID_ARGUMENT, "input grid is NULL");
    if (u->entity != CN_ENTITY_CELL)
        return fail(CN_ERR_UNSUPPORTED, "finite-difference stencils need cell-centred grids");
    if (comp < 0 || comp + ncin > u->ncomp)
        return fail(CN_ERR_INVALID_ARGUMENT, "input component out of range");
    cn_status s;
    if (o1 && (s = check_out(u, o1, c1, 1)) != CN_OK) return s;
    if (o2 && (s = check_out(u, o2, c2, 3)) != CN_OK) return s;
    cudaStream_t st = as_stream(stream);
    if (u->dtype == CN_FLOAT64) return launch_fd<double, OP>(u, comp, o1, c1, o2, c2, st);
    if (u->dtype == CN_FLOAT32) return launch_fd<float, OP>(u, comp, o1, c1, o2, c2, st);
    return fail(CN_ERR_UNSUPPORTED, "finite-difference stencils need FLOAT32 or FLOAT64 grids");
}

// ---------------------------------------------------------------- ddx ABI
// One thread per (x, y) column of 32 x 8 tiles, looping over z: no index
// divisions, coalesced rows along x.
template <typename T>
__global__ void __launch_bounds__(256)
    ddx_kernel(int nx, int ny, int nz, const T *__restrict__ src, int xps, int xyps,
               T *__restrict__ dst, int xpd, int xypd, T fac)
{
    using A = Arith<T>;
    const int x = blockIdx.x * 32 + (threadIdx.x & 31);
    if (x >= nx) return;
    for (int y = blockIdx.y * 8 + (threadIdx.x >> 5); y < ny; y += gridDim.y * 8) {
        for (int z = blockIdx.z; z < nz; z += gridDim.z) {
            const T *s = src + x + (int64_t)xps * y + (int64_t)xyps * z;
            T acc = A::add(s[-1], s[1]);
            acc = A::add(acc, s[-xps]);
            acc = A::add(acc, s[xps]);
            acc = A::add(acc, s[-xyps]);
            acc = A::add(acc, s[xyps]);
            acc = A::sub(acc, A::mul(T(6), s[0]));
            dst[x + (int64_t)xpd * y + (int64_t)xypd * z] = A::mul(fac, acc);
        }
    }
}

template <typename T>
static cn_status launch_ddx(int nx, int ny, int nz, const T *src, int xps, int xyps, T *dst,
                            int xpd, int xypd, T fac, cudaStream_t st)
{
    if (nx < 1 || ny < 1 || nz < 1 || !src || !dst)
        return fail(CN_ERR_INVALID_ARGUMENT, "ddx: bad extent or pointer");
    const int gx = (nx + 31) / 32;
    const dim3 grid((unsigned)gx, (unsigned)std::min((ny + 7) / 8, 65535), (unsigned)std::min(nz, 65535));
    ddx_kernel<T><<<grid, 256, 0, st>>>(nx, ny, nz, src, xps, xyps, dst, xpd, xypd, fac);
    CN_CUDA_TRY(cudaGetLastError());
    return CN_OK;
}

} // namespace cn

using namespace cn;

extern "C" {

cn_status cn_laplacian(cn_grid *u, int comp, cn_grid *out, int out_comp, void *stream)
{
    if (!out) return fail(CN_ERR_INVALID_ARGUMENT, "output grid is NULL");
    return dispatch_fd<kLap>(u, comp, 1, out, out_comp, nullptr, 0, stream);
}

cn_status cn_gradient(cn_grid *u, int comp, cn_grid *out, int out_comp, void *stream)
{
    if (!out) return fail(CN_ERR_INVALID_ARGUMENT, "output grid is NULL");
    return dispatch_fd<kGrad>(u, comp, 1, nullptr, 0, out, out_comp, stream);
}

cn_status cn_lap_grad(cn_grid *u, int comp, cn_grid *lap, int lap_comp, cn_grid *grad,
                      int grad_comp, void *stream)
{
    if (!lap || !grad) return fail(CN_ERR_INVALID_ARGUMENT, "output grid is NULL");
    return dispatch_fd<kLapGrad>(u, comp, 1, lap, lap_comp, grad, grad_comp, stream);
}

cn_status cn_divergence(cn_grid *v, int comp, cn_grid *out, int out_comp, void *stream)
{
    if (!out) return fail(CN_ERR_INVALID_ARGUMENT, "output grid is NULL");
    return dispatch_fd<kDiv>(v, comp, 3, out, out_comp, nullptr, 0, stream);
}

void cn_ddx_f64(int Nx, int Ny, int Nz, const double *src, int xps, int xyps, double *dst,
                int xpd, int xypd, double factor)
{
    // ddxGold.cpp:49: fac = 1.0 / (factor * factor)
    (void)launch_ddx<double>(Nx, Ny, Nz, src, xps, xyps, dst, xpd, xypd,
                             1.0 / (factor * factor), nullptr);
}

void cn_ddx_f32(int Nx, int Ny, int Nz, const float *src, int xps, int xyps, float *dst,
                int xpd, int xypd, float factor)
{
    // computed in double, stored as float, as `const Real fac = 1.0 / (f*f)`
    const float fac = (float)(1.0 / (double)(factor * factor));
    (void)launch_ddx<float>(Nx, Ny, Nz, src, xps, xyps, dst, xpd, xypd, fac, nullptr);
}

cn_status cn_ddx_async(cn_dtype dtype, int Nx, int Ny, int Nz, const void *src, int xps,
                       int xyps, void *dst, int xpd, int xypd, double factor, void *stream)
{
    cudaStream_t st = as_stream(stream);
    if (dtype == CN_FLOAT64)
        return launch_ddx<double>(Nx, Ny, Nz, (const double *)src, xps, xyps, (double *)dst, xpd,
                                  xypd, 1.0 / (factor * factor), st);
    if (dtype == CN_FLOAT32) {
        const float f = (float)factor;
        return launch_ddx<float>(Nx, Ny, Nz, (const float *)src, xps, xyps, (float *)dst, xpd,
                                 xypd, (float)(1.0 / (double)(f * f)), st);
    }
    return fail(CN_ERR_UNSUPPORTED, "ddx: dtype must be FLOAT32 or FLOAT64");
}

} // extern "C"
