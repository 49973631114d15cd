// aos.cu -- grid <-> array-of-structures (AoS) file buffer on the device.
//
// The reference writes a grid to a file by copying every block field into
// one AoS buffer in a host loop over blocks (IO/CartesianHDF.h:76-80, OpenMP
// over blocks) with Field2AOS (IO/FieldAOS.h:37-57 scalar, :79-101 tensor,
// :136-141 face container -> the face field of one direction), and reads it
// back with AOS2Field (:59-77, :103-124).  For a file index range r (global
// entity indices, the HDF dataset's hyperslab) and every point p of r that
// lies in the grid:
//     buf[c + ncomp * flat_r(p)] = (FileT) field_c[p]       (Field2AOS)
//     field_c[p] = (T) buf[c + ncomp * flat_r(p)]           (AOS2Field)
// with flat_r the x-fastest flat index over r's extent; points of r outside
// the grid are not touched.  Here one launch covers the whole grid: a CTA
// takes an item of up to pts() points, consecutive in the file (of all the
// intersection's points in x-fastest order where it covers whole planes of the
// file range, else of one x-row), reads each component with coalesced loads
// (consecutive x are consecutive in a block), converts, interleaves the
// components in shared memory and writes the item's ncomp * len contiguous file
// values with coalesced stores (the reverse for the read).  HBM-bound: ncomp *
// (sizeof(T) + sizeof(FileT)) bytes per point.  Items cut from all points are
// full whatever the row length, and one CTA per item keeps loads and stores of
// different items in flight together; against rows of at most 512 points taken
// in turn by resident CTAs, B200, both directions: 3 FP64 components and an
// FP32 file, 384^3 919 -> 692 us (5.9 TB/s), 192^3 177 -> 95, 64^3 the launches.
#include "cn_fastdiv.h"
#include "cn_internal.h"

namespace cn {
namespace aos {

constexpr int kThreads = 256;             // threads per CTA
// points per thread, for up to maxc components: 12 or more loads in flight
// (3 FP64 components and an FP32 file, 384^3, both directions: 2 points 872 us,
// 4 points 730; 5 components: 4 points 1872, 2 points 1255)
constexpr int per(int maxc) { return maxc > 4 ? 2 : 4; }
constexpr int pts(int maxc) { return kThreads * per(maxc); } // points per work item
constexpr int kMaxComp = 16;              // components per call
constexpr size_t kSmemDefault = 48 << 10; // above this the kernel opts in

struct Geo {
    int nb[3];       // blocks
    int cells[3];    // block cells
    int grow[3];     // 1: the last block along d holds cells + 1 entities
    int ib[3];       // intersection begin (global entity index)
    int ie[3];       // intersection extent
    int sb[3];       // file range begin
    int se[3];       // file range extent
    int comp0, ncomp;
    int flat;        // 1: the intersection is contiguous in the file, items are cut from all its points
    int points;      // points of the intersection (flat)
    int chunks;      // item chunks per x-row of the intersection, or of all points
    FastDiv dv_chunks, dv_ie0, dv_ie1, dv_c0, dv_c1, dv_c2;
    int64_t bstride; // elements
    int64_t cstride; // elements
};

template <typename D, typename S> __device__ __forceinline__ D conv(S v) { return static_cast<D>(v); }

// A thread takes points t, t + kThreads, ... of the CTA's item.  All divisions
// are multiply-high forms of divisors fixed at launch (cn_fastdiv.h).  MAXC >=
// ncomp bounds the component loops at compile time so that a thread issues
// every load of its points before converting any.

// The item's file values dst[0, n) <-> shared st[0, n): 16-byte accesses
// when dst is 16-byte aligned and n * sizeof(F) a multiple of 16 (whole-grid
// files with 4-byte values and 4 | x-extent * ncomp, or 8-byte values and
// 2 | it), else element by element.
template <typename F, bool OUT>
__device__ __forceinline__ void stage_copy(F *dst, F *st, int n, int t)
{
    const size_t bytes = (size_t)n * sizeof(F);
    if ((reinterpret_cast<uintptr_t>(dst) & 15) == 0 && (bytes & 15) == 0) {
        int4 *d4 = reinterpret_cast<int4 *>(dst);
        int4 *s4 = reinterpret_cast<int4 *>(st);
        const int n4 = (int)(bytes >> 4);
        for (int k = t; k < n4; k += kThreads) {
            if (OUT) d4[k] = s4[k];
            else s4[k] = __ldg(d4 + k);
        }
    } else {
        for (int k = t; k < n; k += kThreads) {
            if (OUT) dst[k] = st[k];
            else st[k] = __ldg(dst + k);
        }
    }
}

// Resident CTAs per SM that the register budget is set for (every
// instantiation compiles without spills at these bounds).
constexpr int min_ctas(int maxc) { return maxc > 8 ? 2 : (maxc > 4 ? 3 : (maxc > 1 ? 4 : 6)); }

template <typename T, typename F, bool TO_AOS, int MAXC>
__global__ void __launch_bounds__(kThreads, min_ctas(MAXC))
    aos_kernel(const __grid_constant__ Geo G, T *__restrict__ grid, F *__restrict__ buf)
{
    extern __shared__ __align__(16) unsigned char aos_smem[];
    F *st = reinterpret_cast<F *>(aos_smem);
    const int t = threadIdx.x;
    constexpr int kPer = per(MAXC), kPts = pts(MAXC);
    const int nc = G.ncomp;
    T *const gbase = grid + (int64_t)G.comp0 * G.cstride;
    const int w = blockIdx.x;
    const int row0 = G.flat ? 0 : G.dv_chunks.div(w);
    const int xs = (w - row0 * G.chunks) * kPts;             // item start, relative to the row's begin
    const int len = min(kPts, (G.flat ? G.points : G.ie[0]) - xs);
    const int iz0 = G.dv_ie1.div(row0);
    F *dst = buf + ((int64_t)(G.ib[0] + xs - G.sb[0]) +
                    (int64_t)G.se[0] * ((G.ib[1] + row0 - iz0 * G.ie[1] - G.sb[1]) +
                                        (int64_t)G.se[1] * (G.ib[2] + iz0 - G.sb[2]))) * nc;
    // in-grid offset of point p of the item
    auto offset = [&](int p) -> int64_t {
        int x = xs + p, row = row0;
        if (G.flat) {
            row = G.dv_ie0.div(x);
            x -= row * G.ie[0];
        }
        x += G.ib[0];
        const int iz = G.dv_ie1.div(row);
        const int gy = G.ib[1] + (row - iz * G.ie[1]), gz = G.ib[2] + iz;
        const int bx = min(G.dv_c0.div(x), G.nb[0] - 1), lx = x - bx * G.cells[0];
        const int by = min(G.dv_c1.div(gy), G.nb[1] - 1), ly = gy - by * G.cells[1];
        const int bz = min(G.dv_c2.div(gz), G.nb[2] - 1), lz = gz - bz * G.cells[2];
        const int ex = G.cells[0] + ((G.grow[0] && bx == G.nb[0] - 1) ? 1 : 0);
        const int ey = G.cells[1] + ((G.grow[1] && by == G.nb[1] - 1) ? 1 : 0);
        return (int64_t)(bx + G.nb[0] * (by + G.nb[1] * bz)) * G.bstride + lx + (int64_t)ex * (ly + ey * lz);
    };
    if (TO_AOS) {
        T v[kPer][MAXC];
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            if (t + j * kThreads < len) {
                const int64_t off = offset(t + j * kThreads);
#pragma unroll
                for (int c = 0; c < MAXC; ++c)
                    if (c < nc) v[j][c] = __ldg(gbase + off + c * G.cstride);
            }
        }
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int p = t + j * kThreads;
            if (p < len) {
#pragma unroll
                for (int c = 0; c < MAXC; ++c)
                    if (c < nc) st[p * nc + c] = conv<F>(v[j][c]);
            }
        }
        __syncthreads();
        stage_copy<F, true>(dst, st, len * nc, t);
    } else {
        stage_copy<F, false>(dst, st, len * nc, t);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            const int p = t + j * kThreads;
            if (p < len) {
                const int64_t off = offset(p);
#pragma unroll
                for (int c = 0; c < MAXC; ++c)
                    if (c < nc) gbase[off + c * G.cstride] = conv<T>(st[p * nc + c]);
            }
        }
    }
}

template <typename T, typename F, bool TO_AOS, int MAXC>
cn_status launch_one(Geo G, int64_t rows, T *data, F *buf, cudaStream_t s)
{
    constexpr int kPts = pts(MAXC);
    G.chunks = ((G.flat ? G.points : G.ie[0]) + kPts - 1) / kPts;
    G.dv_chunks = FastDiv((uint32_t)G.chunks);
    const size_t smem = (size_t)kPts * G.ncomp * sizeof(F);
    // the opt-in is a property of the current device's context: set it on every large launch
    if (smem > kSmemDefault) {
        CN_CUDA_TRY(cudaFuncSetAttribute(aos_kernel<T, F, TO_AOS, MAXC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)(kPts * MAXC * sizeof(F))));
    }
    aos_kernel<T, F, TO_AOS, MAXC><<<(unsigned)(rows * G.chunks), kThreads, smem, s>>>(G, data, buf);
    CN_CUDA_TRY(cudaGetLastError());
    return CN_OK;
}

template <typename T, typename F>
cn_status launch(const Geo &G, int64_t rows, cn_grid *g, void *buf, bool to_aos, cudaStream_t s)
{
    T *data = reinterpret_cast<T *>(g->d_data);
    F *b = reinterpret_cast<F *>(buf);
    const int nc = G.ncomp;
    if (to_aos) {
        if (nc == 1) return launch_one<T, F, true, 1>(G, rows, data, b, s);
        if (nc <= 4) return launch_one<T, F, true, 4>(G, rows, data, b, s);
        if (nc <= 8) return launch_one<T, F, true, 8>(G, rows, data, b, s);
        return launch_one<T, F, true, kMaxComp>(G, rows, data, b, s);
    }
    if (nc == 1) return launch_one<T, F, false, 1>(G, rows, data, b, s);
    if (nc <= 4) return launch_one<T, F, false, 4>(G, rows, data, b, s);
    if (nc <= 8) return launch_one<T, F, false, 8>(G, rows, data, b, s);
    return launch_one<T, F, false, kMaxComp>(G, rows, data, b, s);
}

template <typename T>
cn_status dispatch_file(const Geo &G, int64_t rows, cn_grid *g, cn_dtype file_dtype, void *buf, bool to_aos, cudaStream_t s)
{
    switch (file_dtype) {
    case CN_FLOAT64:
        return launch<T, double>(G, rows, g, buf, to_aos, s);
    case CN_FLOAT32:
        return launch<T, float>(G, rows, g, buf, to_aos, s);
    case CN_INT32:
        return launch<T, int32_t>(G, rows, g, buf, to_aos, s);
    }
    return fail(CN_ERR_UNSUPPORTED, "cn_grid_aos: file dtype");
}

cn_status run(cn_grid *g, int comp0, int ncomp, const int span_begin[3], const int span_end[3],
              cn_dtype file_dtype, void *buf, void *stream, bool to_aos)
{
    const char *who = to_aos ? "cn_grid_to_aos" : "cn_grid_from_aos";
    if (!g || !span_begin || !span_end) {
        return fail(CN_ERR_INVALID_ARGUMENT, std::string(who) + ": grid or file range is NULL");
    }
    if (comp0 < 0 || ncomp < 1 || comp0 + ncomp > g->ncomp) {
        return fail(CN_ERR_INVALID_ARGUMENT, std::string(who) + ": components outside the grid");
    }
    if (ncomp > kMaxComp) {
        return fail(CN_ERR_UNSUPPORTED, std::string(who) + ": more than 16 components per call");
    }
    if (file_dtype < CN_FLOAT32 || file_dtype > CN_INT32) {
        return fail(CN_ERR_INVALID_ARGUMENT, std::string(who) + ": bad file dtype");
    }
    // a floating-point value converted to int32 is undefined out of range in
    // the reference's implicit conversion; only int32 <-> int32 is allowed
    const cn_dtype dst_type = to_aos ? file_dtype : g->dtype;
    const cn_dtype src_type = to_aos ? g->dtype : file_dtype;
    if (dst_type == CN_INT32 && src_type != CN_INT32) {
        return fail(CN_ERR_UNSUPPORTED, std::string(who) + ": floating-point to int32 conversion");
    }
    Geo G;
    int64_t rows = 1;
    for (int d = 0; d < 3; ++d) {
        if (span_end[d] < span_begin[d]) {
            return fail(CN_ERR_INVALID_ARGUMENT, std::string(who) + ": file range end before begin");
        }
        G.nb[d] = g->nb[d];
        G.cells[d] = g->cells[d];
        G.grow[d] = (g->entity == CN_ENTITY_NODE || g->entity == CN_ENTITY_FACE_X + d) ? 1 : 0;
        G.sb[d] = span_begin[d];
        G.se[d] = span_end[d] - span_begin[d];
        // grid index range [0, nb * cells + grow)
        const int gend = g->nb[d] * g->cells[d] + G.grow[d];
        const int b = span_begin[d] > 0 ? span_begin[d] : 0;
        const int e = span_end[d] < gend ? span_end[d] : gend;
        G.ib[d] = b;
        G.ie[d] = e > b ? e - b : 0;
        if (d > 0) rows *= G.ie[d];
    }
    if ((int64_t)G.se[0] * G.se[1] * G.se[2] > 0 && !buf) {
        return fail(CN_ERR_INVALID_ARGUMENT, std::string(who) + ": buffer is NULL");
    }
    if (G.ie[0] == 0 || rows == 0) return CN_OK; // empty intersection
    // the kernel dereferences buf: device, managed or pinned host memory only
    cudaPointerAttributes pa;
    if (cudaPointerGetAttributes(&pa, buf) != cudaSuccess || pa.type == cudaMemoryTypeUnregistered) {
        cudaGetLastError();
        return fail(CN_ERR_INVALID_ARGUMENT, std::string(who) + ": buffer is not device-accessible memory");
    }
    G.comp0 = comp0;
    G.ncomp = ncomp;
    // row chunks, at the fewest points per item
    if (rows * ((G.ie[0] + pts(kMaxComp) - 1) / pts(kMaxComp)) >= (int64_t(1) << 31)) {
        return fail(CN_ERR_UNSUPPORTED, std::string(who) + ": more than 2^31 row chunks in the file range");
    }
    // whole planes of the file: items across rows, all of them full
    const int64_t points = rows * G.ie[0];
    G.flat = G.ie[0] == G.se[0] && G.ie[1] == G.se[1] && points < (int64_t(1) << 31) - pts(1);
    G.points = G.flat ? (int)points : 0;
    if (G.flat) rows = 1;
    G.dv_ie0 = FastDiv((uint32_t)G.ie[0]);
    G.dv_ie1 = FastDiv((uint32_t)G.ie[1]);
    G.dv_c0 = FastDiv((uint32_t)G.cells[0]);
    G.dv_c1 = FastDiv((uint32_t)G.cells[1]);
    G.dv_c2 = FastDiv((uint32_t)G.cells[2]);
    G.bstride = g->block_stride;
    G.cstride = g->comp_stride;
    cudaStream_t s = as_stream(stream);
    switch (g->dtype) {
    case CN_FLOAT64:
        return dispatch_file<double>(G, rows, g, file_dtype, buf, to_aos, s);
    case CN_FLOAT32:
        return dispatch_file<float>(G, rows, g, file_dtype, buf, to_aos, s);
    case CN_INT32:
        return dispatch_file<int32_t>(G, rows, g, file_dtype, buf, to_aos, s);
    }
    return fail(CN_ERR_UNSUPPORTED, std::string(who) + ": grid dtype");
}

} // namespace aos
} // namespace cn

extern "C" cn_status cn_grid_to_aos(cn_grid *g, int comp0, int ncomp, const int span_begin[3],
                                    const int span_end[3], cn_dtype file_dtype, void *d_buf, void *stream)
{
    return cn::aos::run(g, comp0, ncomp, span_begin, span_end, file_dtype, d_buf, stream, true);
}

extern "C" cn_status cn_grid_from_aos(cn_grid *g, int comp0, int ncomp, const int span_begin[3],
                                      const int span_end[3], cn_dtype file_dtype, const void *d_buf, void *stream)
{
    return cn::aos::run(g, comp0, ncomp, span_begin, span_end, file_dtype, const_cast<void *>(d_buf), stream,
                        false);
}
