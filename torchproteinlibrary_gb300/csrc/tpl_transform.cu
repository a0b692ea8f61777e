// CoordsTransform on the GPU (sm_103a): translate, rotate, centre and bounding box
// of batched coordinate rows [B, 3 * atoms_stride]; atoms at and past num_atoms[b]
// are written as zeros, as the reference's zero-initialised outputs leave them.
//
// Reference: Layers/FullAtomModel/TransformCUDAKernels.cu:4-107 launches one block
// per atom index with one thread per chain (<<<atoms_stride, batch_size>>>, so
// batch_size <= 1024) and sums each centroid serially in one thread; the bounding
// box runs on the CPU (Layers/FullAtomModel/CoordsTransform/
// coordsTransform_interface.cpp:175-200, Math/nUtil.cpp:27-57).  Here the
// elementwise transforms are coalesced, 16-byte-vectorised passes over the batch
// (HBM-bound: 2 x 12 B per atom in FP32; padding atoms are written, not read), and
// centroid and box are block reductions, one CTA per chain.
//
// A row starts at any place of a 16-byte block (3 * atoms_stride is a multiple of four
// for one stride in four), so every kernel takes the few elements or atoms before the
// row's first boundary and after its last one by themselves and moves the rest as
// vectors.  Scalar passes over such rows had been issue-bound: 4096 rows of 1000..3471
// atoms, stride 3471 (41 us of HBM traffic each): translate 70 -> 39 us, rotate 54 -> 46 us,
// box 26 -> 21 us.
#include <cfloat>
#include <cmath>
#include <cstring>

#include "tpl_internal.h"
#include "tpl_rows.cuh"

namespace tpl {
namespace {

constexpr int kUnroll = 4;  // vectors in flight per thread in the elementwise passes

// 16-byte streaming load / store (data touched once).
template <typename T>
__device__ __forceinline__ void load16(const T *p, T (&v)[Vec16<T>::n]) {
    const typename Vec16<T>::type x = __ldcs(reinterpret_cast<const typename Vec16<T>::type *>(p));
    memcpy(v, &x, sizeof(x));
}
template <typename T>
__device__ __forceinline__ void store16(T *p, const T (&v)[Vec16<T>::n]) {
    typename Vec16<T>::type x;
    memcpy(&x, v, sizeof(x));
    __stcs(reinterpret_cast<typename Vec16<T>::type *>(p), x);
}

// out[b, e] = (in ? in[b, e] : 0) + (add ? add[b, e % 3] * (scale_by_count ? 1 / n_b : 1) : 0)
// for e < 3 n_b, 0 after.  Covers translate (add = T), its backward (add = null),
// and the centre's backward (in = null, add = dL/dcentre, scaled by 1 / n_b).
// Grid: y over rows (strided), x over pieces of a row, so no thread divides by the
// row length.  Between the row's first and last 16-byte boundary elements move as
// vectors when `in` and `out` have the same alignment; the others one by one.
struct ShiftArgs {
    const void *in;
    void *out;
    const void *add;
    const int *num_atoms;
    int B;
    int row;  // 3 * atoms_stride
    int scale_by_count;
};

template <typename T>
__global__ void __launch_bounds__(256) shift_kernel(ShiftArgs a) {
    constexpr int N = Vec16<T>::n;
    const T *add = static_cast<const T *>(a.add);
    const int step = gridDim.x * blockDim.x, first = blockIdx.x * blockDim.x + threadIdx.x;
    for (int b = blockIdx.y; b < a.B; b += gridDim.y) {
        const T *in = a.in ? static_cast<const T *>(a.in) + (size_t)b * a.row : nullptr;
        T *out = static_cast<T *>(a.out) + (size_t)b * a.row;
        const int n = max(0, min(a.num_atoms[b], a.row / 3)), n3 = 3 * n;
        T t[3] = {T(0), T(0), T(0)};
        if (add)
            for (int k = 0; k < 3; k++) {
                t[k] = add[3 * (size_t)b + k];
                if (a.scale_by_count && n > 0) t[k] = t[k] / T(n);
            }
        auto pick = [&](int r) { return r == 0 ? t[0] : (r == 1 ? t[1] : t[2]); };
        const int off = row_head(out);  // elements of `out` since a 16-byte boundary
        const int head = in && row_head(in) != off ? a.row : min((N - off) & (N - 1), a.row);
        const int nv = (a.row - head) / N;
        // kUnroll independent vectors per thread and step: loads issued before use
        for (int v0 = first; v0 < nv; v0 += kUnroll * step) {
            T x[kUnroll][N];
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int v = v0 + u * step, e = head + v * N;
                if (in && v < nv && e < n3) load16(in + e, x[u]);
                else
                    for (int k = 0; k < N; k++) x[u][k] = T(0);
            }
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int v = v0 + u * step;
                if (v >= nv) continue;
                const int e = head + v * N, r = e % 3;
                const T te[3] = {pick(r), pick(r == 2 ? 0 : r + 1), pick(r == 0 ? 2 : r - 1)};
#pragma unroll
                for (int k = 0; k < N; k++) x[u][k] = e + k < n3 ? x[u][k] + te[k % 3] : T(0);
                store16(out + e, x[u]);
            }
        }
        // the elements outside the vectors
        const int rest = a.row - nv * N;
        for (int i0 = first; i0 < rest; i0 += kUnroll * step) {
            T x[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int i = i0 + u * step, e = i < head ? i : i + nv * N;
                x[u] = in && i < rest && e < n3 ? __ldcs(in + e) : T(0);
            }
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int i = i0 + u * step, e = i < head ? i : i + nv * N;
                if (i < rest) __stcs(out + e, e < n3 ? x[u] + pick(e % 3) : T(0));
            }
        }
    }
}

// out[b, atom] = R_b x (or R_b^T x) for atom < n_b, 0 after; R row-major [B, 3, 3].
// Grid: y over rows (strided), x over pieces of 512 aligned groups of N atoms
// (tpl_rows.cuh), two tiles of 32 groups per warp whose loads are in flight together (one
// tile: 54 us; the launch is then bound by the latency of its many short blocks).  A warp loads and stores its tile as 96 vectors in
// memory order and turns it to one group per lane and back through shared memory: with a
// group per lane straight from memory every 32-byte sector is written in two pieces
// (strides of 48 bytes), with an atom per lane in three.  48-byte lane strides are free of
// bank conflicts.  Atoms outside the groups, and rows whose input and output differ in
// alignment, are taken one by one.
template <typename T>
__global__ void __launch_bounds__(256) rotate_kernel(const T *in, T *out, const T *R, const int *num_atoms, int B,
                                                     int stride, int transpose) {
    constexpr int N = Vec16<T>::n;
    using V = typename Vec16<T>::type;
    __shared__ V s_tile[8][96];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    V *tile = s_tile[w];
    for (int b = blockIdx.y; b < B; b += gridDim.y) {
        const int n = min(num_atoms[b], stride);
        T m[9];
        for (int k = 0; k < 9; k++) m[k] = R[9 * (size_t)b + (transpose ? 3 * (k % 3) + k / 3 : k)];
        const T *x = in + (size_t)b * 3 * stride;
        T *y = out + (size_t)b * 3 * stride;
        auto turn = [&](const T *v, T *r) {
            const T x0 = v[0], x1 = v[1], x2 = v[2];
            r[0] = m[0] * x0 + m[1] * x1 + m[2] * x2;
            r[1] = m[3] * x0 + m[4] * x1 + m[5] * x2;
            r[2] = m[6] * x0 + m[7] * x1 + m[8] * x2;
        };
        const int off = row_head(y);
        const int head = row_head(x) != off ? stride : min(off, stride);
        const int ng = (stride - head) / N;
        const V *src = reinterpret_cast<const V *>(x + 3 * head);  // vector k of group g is 3 g + k
        V *dst = reinterpret_cast<V *>(y + 3 * head);
        const int nvec = 3 * ng, live = 3 * (n - head);  // vectors of the groups; values that hold atoms
        for (int g0 = blockIdx.x * 512 + 32 * w; g0 < ng; g0 += gridDim.x * 512) {
            V v[2][3];
#pragma unroll
            for (int u = 0; u < 2; u++)
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const int k = 3 * (g0 + 256 * u) + lane + 32 * q;
                    if (k < nvec && k * N < live) v[u][q] = __ldcs(src + k);
                    else memset(&v[u][q], 0, sizeof(V));
                }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int g = g0 + 256 * u;
                if (3 * g * N < live) {  // the same for the whole warp
#pragma unroll
                    for (int q = 0; q < 3; q++) tile[lane + 32 * q] = v[u][q];
                    __syncwarp();
                    T p[3 * N];
                    load_group(reinterpret_cast<const T *>(tile + 3 * lane), p);
                    const int left = n - head - N * (g + lane);  // atoms from this lane's group on
#pragma unroll
                    for (int q = 0; q < N; q++) {
                        if (q < left) turn(p + 3 * q, p + 3 * q);
                        else p[3 * q] = p[3 * q + 1] = p[3 * q + 2] = T(0);
                    }
                    store_group(reinterpret_cast<T *>(tile + 3 * lane), p);
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 3; q++) v[u][q] = tile[lane + 32 * q];
                    __syncwarp();  // the next tile rewrites it
                }
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    const int k = 3 * g + lane + 32 * q;
                    if (k < nvec) __stcs(dst + k, v[u][q]);
                }
            }
        }
        const int rest = stride - N * ng;
        for (int i0 = blockIdx.x * 256 + threadIdx.x; i0 < rest; i0 += gridDim.x * 256) {
            const int i = i0 < head ? i0 : i0 + N * ng;
            T r[3] = {T(0), T(0), T(0)};
            if (i < n) turn(x + 3 * i, r);
            for (int k = 0; k < 3; k++) y[3 * i + k] = r[k];
        }
    }
}

// Threads per chain of the two reductions: a thread's loads are what is waited for, and more
// small CTAs keep more of them in flight (4096 rows of 1157..3471 atoms, 256 / 128 threads:
// centre 24.7 / 22.1 us, box 22.4 / 21.1; a launch of 4000 atoms each 35.3 / 33.9 and 33.1 / 32.4).
constexpr int kReduceThreads = 128;

// Centroid of the first n_b atoms of chain b = blockIdx.x (FP64 accumulation);
// 0 for an empty chain.
template <typename T>
__global__ void __launch_bounds__(kReduceThreads) center_kernel(const T *in, T *center, const int *num_atoms,
                                                                int stride) {
    constexpr int ROWS = kReduceThreads / 8;
    __shared__ T s_sum[ROWS][3];
    const int b = blockIdx.x, lane = threadIdx.x & 31;
    const int n = min(num_atoms[b], stride);  // a count past the row is clamped to it
    const T *x = in + (size_t)b * 3 * stride;
    // offsets from the chain's first atom, summed in the coordinate type per thread and over
    // eight lanes and in FP64 across those: the offsets stay of the chain's own extent
    // wherever the chain sits, and GB300's FP64 rate is a small fraction of its FP32 rate
    const T p0 = n > 0 ? x[0] : T(0), p1 = n > 0 ? x[1] : T(0), p2 = n > 0 ? x[2] : T(0);
    T s[3] = {T(0), T(0), T(0)};
    // aligned groups of N atoms as three vectors per thread (tpl_rows.cuh), two groups in
    // flight; then the atoms before and after them
    constexpr int N = Vec16<T>::n;
    const int head = max(0, min(row_head(x), n)), ng = max(0, n - head) / N;
    const T *xg = x + 3 * head;
#pragma unroll 2
    for (int g = threadIdx.x; g < ng; g += kReduceThreads) {
        T v[3 * N];
        load_group(xg + 3 * N * g, v);
        if constexpr (N == 4) {
            s[0] += ((v[0] - p0) + (v[3] - p0)) + ((v[6] - p0) + (v[9] - p0));
            s[1] += ((v[1] - p1) + (v[4] - p1)) + ((v[7] - p1) + (v[10] - p1));
            s[2] += ((v[2] - p2) + (v[5] - p2)) + ((v[8] - p2) + (v[11] - p2));
        } else {
            s[0] += (v[0] - p0) + (v[3] - p0);
            s[1] += (v[1] - p1) + (v[4] - p1);
            s[2] += (v[2] - p2) + (v[5] - p2);
        }
    }
    for (int q = threadIdx.x; q < n - N * ng; q += kReduceThreads) {
        const int i = q < head ? q : q + N * ng;
        s[0] += x[3 * i] - p0;
        s[1] += x[3 * i + 1] - p1;
        s[2] += x[3 * i + 2] - p2;
    }
#pragma unroll
    for (int off = 4; off > 0; off >>= 1)
#pragma unroll
        for (int c = 0; c < 3; c++) s[c] += __shfl_xor_sync(0xffffffffu, s[c], off);
    if ((lane & 7) == 0)
#pragma unroll
        for (int c = 0; c < 3; c++) s_sum[threadIdx.x >> 3][c] = s[c];
    __syncthreads();
    if (threadIdx.x >= 32) return;
    static_assert(ROWS <= 32, "one sum per lane");
    double t[3];
#pragma unroll
    for (int c = 0; c < 3; c++) t[c] = lane < ROWS ? (double)s_sum[lane][c] : 0.0;
#pragma unroll
    for (int off = ROWS / 2; off > 0; off >>= 1)
#pragma unroll
        for (int c = 0; c < 3; c++) t[c] += __shfl_xor_sync(0xffffffffu, t[c], off);
    if (lane < 3) {
        const double v = lane == 0 ? t[0] : (lane == 1 ? t[1] : t[2]);
        const double p = lane == 0 ? (double)p0 : (lane == 1 ? (double)p1 : (double)p2);
        center[3 * b + lane] = n > 0 ? (T)(p + v / n) : T(0);
    }
}

// Axis-aligned bounding box of the first n_b atoms of chain b: lo = min, hi = max
// per coordinate (+inf / -inf for an empty chain, as Math/nUtil.cpp:27-57).
template <typename T>
__global__ void __launch_bounds__(kReduceThreads) bbox_kernel(const T *in, T *lo, T *hi, const int *num_atoms,
                                                              int stride) {
    constexpr int NW = kReduceThreads / 32, N = Vec16<T>::n;
    __shared__ T s_warp[NW][6];
    const int b = blockIdx.x, lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int n = min(num_atoms[b], stride);
    const T *x = in + (size_t)b * 3 * stride;
    const T inf = (T)INFINITY;
    T m[6] = {inf, inf, inf, -inf, -inf, -inf};  // min, max
    auto add = [&](const T *v) {
#pragma unroll
        for (int c = 0; c < 3; c++) {
            m[c] = v[c] < m[c] ? v[c] : m[c];
            m[3 + c] = v[c] > m[3 + c] ? v[c] : m[3 + c];
        }
    };
    const int head = max(0, min(row_head(x), n)), ng = max(0, n - head) / N;
    const T *xg = x + 3 * head;
#pragma unroll 2
    for (int g = threadIdx.x; g < ng; g += kReduceThreads) {
        T v[3 * N];
        load_group(xg + 3 * N * g, v);
#pragma unroll
        for (int q = 0; q < N; q++) add(v + 3 * q);
    }
    for (int q = threadIdx.x; q < n - N * ng; q += kReduceThreads) add(x + 3 * (q < head ? q : q + N * ng));
    auto lower = [](T p, T q) { return q < p ? q : p; };
    auto upper = [](T p, T q) { return q > p ? q : p; };
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int c = 0; c < 6; c++) {
            const T o = __shfl_xor_sync(0xffffffffu, m[c], off);
            m[c] = c < 3 ? lower(m[c], o) : upper(m[c], o);
        }
    if (lane == 0)
#pragma unroll
        for (int c = 0; c < 6; c++) s_warp[w][c] = m[c];
    __syncthreads();
    if (threadIdx.x < 6) {
        const int c = threadIdx.x;
        T r = s_warp[0][c];
        for (int k = 1; k < NW; k++) r = c < 3 ? lower(r, s_warp[k][c]) : upper(r, s_warp[k][c]);
        if (c < 3) lo[3 * b + c] = r;
        else hi[3 * b + c - 3] = r;
    }
}

// Row-major 2-D grid: x covers one row's items in 256-thread blocks, y the rows
// (capped; the kernels stride over the remaining rows).
dim3 grid_rows(int B, long long items_per_row) {
    long long gx = (items_per_row + 255) / 256;
    if (gx < 1) gx = 1;
    if (gx > 65535) gx = 65535;
    int gy = B < 1 ? 1 : B;
    if (gy > 65535) gy = 65535;
    return dim3((unsigned)gx, (unsigned)gy, 1);
}

}  // namespace

template <typename T>
int coords_shift(const T *in, T *out, const T *add, int scale_by_count, const int *num_atoms, int B, int stride,
                 cudaStream_t st) {
    if (B == 0 || stride == 0) return TPL_OK;
    ShiftArgs a{in, out, add, num_atoms, B, 3 * stride, scale_by_count};
    const long long nv = (a.row + Vec16<T>::n - 1) / Vec16<T>::n;
    shift_kernel<T><<<grid_rows(B, (nv + kUnroll - 1) / kUnroll), 256, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <typename T>
int coords_rotate(const T *in, T *out, const T *R, int transpose, const int *num_atoms, int B, int stride,
                  cudaStream_t st) {
    if (B == 0 || stride == 0) return TPL_OK;
    const long long groups = (stride + Vec16<T>::n - 1) / Vec16<T>::n;
    rotate_kernel<T><<<grid_rows(B, (groups + 1) / 2), 256, 0, st>>>(in, out, R, num_atoms, B, stride, transpose);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <typename T>
int coords_center(const T *in, T *center, const int *num_atoms, int B, int stride, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    center_kernel<T><<<B, kReduceThreads, 0, st>>>(in, center, num_atoms, stride);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <typename T>
int coords_bbox(const T *in, T *lo, T *hi, const int *num_atoms, int B, int stride, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    bbox_kernel<T><<<B, kReduceThreads, 0, st>>>(in, lo, hi, num_atoms, stride);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template int coords_shift<float>(const float *, float *, const float *, int, const int *, int, int, cudaStream_t);
template int coords_shift<double>(const double *, double *, const double *, int, const int *, int, int, cudaStream_t);
template int coords_rotate<float>(const float *, float *, const float *, int, const int *, int, int, cudaStream_t);
template int coords_rotate<double>(const double *, double *, const double *, int, const int *, int, int, cudaStream_t);
template int coords_center<float>(const float *, float *, const int *, int, int, cudaStream_t);
template int coords_center<double>(const double *, double *, const int *, int, int, cudaStream_t);
template int coords_bbox<float>(const float *, float *, float *, const int *, int, int, cudaStream_t);
template int coords_bbox<double>(const double *, double *, double *, const int *, int, int, cudaStream_t);

}  // namespace tpl
