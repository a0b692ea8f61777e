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
// for one stride in four), so kernels that have enough to move take the few elements or
// atoms before the row's first boundary and after its last one by themselves and move the
// rest as vectors.  Scalar passes over such rows had been issue-bound: 4096 rows of
// 1000..3471 atoms, stride 3471 (41 us of HBM traffic each): translate 70 -> 39 us, rotate 54
// -> 46 us, box 26 -> 21 us.
#include <cfloat>
#include <cmath>
#include <cstring>
#include <type_traits>

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
// row length; VEC: 16-byte vectors inside a row (rows that start on a 16-byte boundary and
// hold whole vectors), else element by element.  In float64 SCALE says whether there is
// anything to scale: a translation that shares the code computes the division too (GB300, 4096
// rows of 4000 atoms: 284 -> 98 us).
struct ShiftArgs {
    const void *in;
    void *out;
    const void *add;
    const int *num_atoms;
    int B;
    int row;  // 3 * atoms_stride
    int scale_by_count;
};

// Whether the addend is divided by the count is a template parameter in float64 alone, where the
// division's instructions cost the calls without one; float32 has one kernel for both.
template <typename T, bool VEC, bool SCALE>
__global__ void __launch_bounds__(256) shift_kernel(ShiftArgs a) {
    constexpr int N = VEC ? Vec16<T>::n : 1;
    const T *in = static_cast<const T *>(a.in);
    T *out = static_cast<T *>(a.out);
    const T *add = static_cast<const T *>(a.add);
    const int nv = a.row / N;  // vectors per row
    for (int b = blockIdx.y; b < a.B; b += gridDim.y) {
        const int n = max(0, min(a.num_atoms[b], a.row / 3)), n3 = 3 * n;
        T t[3] = {T(0), T(0), T(0)};
        if (add)
            for (int k = 0; k < 3; k++) {
                t[k] = add[3 * (size_t)b + k];
                if ((sizeof(T) == 8 ? SCALE : a.scale_by_count != 0) && n > 0) t[k] = t[k] / T(n);
            }
        const size_t base = (size_t)b * a.row;
        // kUnroll independent vectors per thread and step: loads issued before use
        const int step = gridDim.x * blockDim.x;
        for (int v0 = blockIdx.x * blockDim.x + threadIdx.x; v0 < nv; v0 += kUnroll * step) {
            T x[kUnroll][Vec16<T>::n];
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int v = v0 + u * step;
                if (v >= nv) continue;
                if (VEC) {
                    if (in && v * N < n3) load16(in + base + (size_t)v * N, x[u]);
                    else
                        for (int k = 0; k < N; k++) x[u][k] = T(0);
                } else {
                    x[u][0] = in && v < n3 ? __ldcs(in + base + v) : T(0);
                }
            }
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int v = v0 + u * step;
                if (v >= nv) continue;
#pragma unroll
                for (int k = 0; k < N; k++) {
                    const int e = v * N + k;
                    x[u][k] = e < n3 ? x[u][k] + t[e % 3] : T(0);
                }
                if (VEC) store16(out + base + (size_t)v * N, x[u]);
                else __stcs(out + base + v, x[u][0]);
            }
        }
    }
}

// The same for rows that start anywhere: vectors between the row's first and last 16-byte
// boundary where `in` and `out` have the same phase, the elements outside them by themselves.
// Eight blocks per SM in float32: short rows leave most of a block idle (16000 rows of 20
// atoms: 17 us, at 38 registers 20).
template <typename T, bool SCALE>
__global__ void __launch_bounds__(256, sizeof(T) == 4 ? 8 : 6) shift_rows_kernel(ShiftArgs a) {
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
                if (SCALE && n > 0) t[k] = t[k] / T(n);
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
                if (v >= nv) continue;
                if (in && e < n3) load16(in + e, x[u]);
                else
                    for (int k = 0; k < N; k++) x[u][k] = T(0);
            }
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int v = v0 + u * step;
                if (v >= nv) continue;
                const int e = head + v * N;
#pragma unroll
                for (int k = 0; k < N; k++) x[u][k] = e + k < n3 ? x[u][k] + t[(e + k) % 3] : T(0);
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
// Grid: y over rows (strided), x over atoms of a row.
template <typename T>
__global__ void __launch_bounds__(256) rotate_kernel(const T *in, T *out, const T *R, const int *num_atoms, int B,
                                                     int stride, int transpose) {
    for (int b = blockIdx.y; b < B; b += gridDim.y) {
        const int n = num_atoms[b];
        T m[9];
        for (int k = 0; k < 9; k++) m[k] = R[9 * (size_t)b + (transpose ? 3 * (k % 3) + k / 3 : k)];
        const T *x = in + (size_t)b * 3 * stride;
        T *y = out + (size_t)b * 3 * stride;
        const int step = gridDim.x * blockDim.x;
        for (int i0 = blockIdx.x * blockDim.x + threadIdx.x; i0 < stride; i0 += kUnroll * step) {
            T v[kUnroll][3];
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {  // loads of kUnroll atoms in flight
                const int i = i0 + u * step;
                if (i < min(n, stride))
                    for (int k = 0; k < 3; k++) v[u][k] = __ldcs(x + 3 * i + k);
            }
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int i = i0 + u * step;
                if (i >= stride) continue;
                T r0 = T(0), r1 = T(0), r2 = T(0);
                if (i < n) {
                    const T x0 = v[u][0], x1 = v[u][1], x2 = v[u][2];
                    r0 = m[0] * x0 + m[1] * x1 + m[2] * x2;
                    r1 = m[3] * x0 + m[4] * x1 + m[5] * x2;
                    r2 = m[6] * x0 + m[7] * x1 + m[8] * x2;
                }
                __stcs(y + 3 * i, r0);
                __stcs(y + 3 * i + 1, r1);
                __stcs(y + 3 * i + 2, r2);
            }
        }
    }
}

// The same for float32 batches that pass through more memory than L2 holds (129 MB), on rows
// of three quarters of a block's atoms at least: there the partial sectors cost, and the
// tiles' latency does not (one atom per thread / tiles, us: 4096 rows of 3471 atoms 56.9 / 52.7,
// ragged 51.2 / 44.2; 1000 rows, 83 MB, 12.0 / 12.7; 16000 of 1001 62.7 / 67.5; float64, bound by
// its arithmetic, 4096 of 3471 226 / 236).
// Grid: y over rows (strided), x over pieces of 512 aligned groups of N atoms
// (tpl_rows.cuh), two tiles of 32 groups per warp whose loads are in flight together (one
// tile: 54 us; the launch is then bound by the latency of its many short blocks).  A warp
// loads and stores its tile as 96 vectors in memory order and turns it to one group per lane and back through shared memory: with a
// group per lane straight from memory every 32-byte sector is written in two pieces
// (strides of 48 bytes), with an atom per lane in three.  48-byte lane strides are free of
// bank conflicts.  Atoms outside the groups, and rows whose input and output differ in
// alignment, are taken one by one.
__global__ void __launch_bounds__(256) rotate_tiles_kernel(const float *in, float *out, const float *R,
                                                           const int *num_atoms, int B, int stride, int transpose) {
    using T = float;
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

// Threads per chain NT of the two reductions: a thread's loads are what is waited for.  Where
// the batch fills the GPU more small CTAs keep more of them in flight, 128 threads each; a
// smaller batch waits for its longest chain, and long rows for themselves: 256.  256 / 128
// threads, us: float32 4096 rows of 1157..3471 atoms centre 24.7 / 22.1, box 22.4 / 21.1; 450 of
// 20001 15.4 / 26.9, 19.3 / 29.1; 800 of 20001 centre 27.0 / 30.7.  In float64 the reduction's
// own additions weigh more: box of 150 rows of 20001 45 / 66, of 300 84 / 90, of 450 121 / 118,
// of 300 of 4000 22.6 / 20.7; centre of 150 of 20001 40.4 / 44.6, of 600 6.2 / 5.4.
template <typename T>
static bool wide_reduction(int B, int stride, bool box) {
    const int sms = device_sm_count();
    const bool lng = stride > 12000;
    if (sizeof(T) == 4) return lng || B <= 4 * sms;
    return lng ? !box || B <= 2 * sms : B <= sms && (box || stride > 2000);
}

// Centroid of the first n_b atoms of chain b = blockIdx.x (FP64 accumulation);
// 0 for an empty chain.
// (32 registers in float32: 2000 chains of 4000 atoms are one wave of CTAs of 128 threads then,
// 10.4 us, and two with 40, 15.0)
template <typename T, int NT>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 2048 : 1536) / NT) center_kernel(const T *in, T *center, const int *num_atoms, int stride) {
    // lanes summed in the coordinate type: fewer where a thread has more atoms
    constexpr int LR = NT == 128 ? 8 : 32, ROWS = NT / LR;
    // (float64 sums where few rows are left: the conversions are then those of many warps)
    using Sum = std::conditional_t<ROWS <= 8, double, T>;
    __shared__ Sum s_sum[ROWS][3];
    const int b = blockIdx.x, lane = threadIdx.x & 31;
    const int n = min(num_atoms[b], stride);  // a count past the row is clamped to it
    const T *x = in + (size_t)b * 3 * stride;
    // offsets from the chain's first atom, summed in the coordinate type per thread and over
    // LR lanes and in FP64 across those: the offsets stay of the chain's own extent
    // wherever the chain sits, and GB300's FP64 rate is a small fraction of its FP32 rate
    const T p0 = n > 0 ? x[0] : T(0), p1 = n > 0 ? x[1] : T(0), p2 = n > 0 ? x[2] : T(0);
    T s[3] = {T(0), T(0), T(0)};
    // aligned groups of N atoms as three vectors per thread (tpl_rows.cuh), two groups in
    // flight; the few atoms before and after them, loaded first, are added last
    constexpr int N = Vec16<T>::n;
    const int head = max(0, min(row_head(x), n)), ng = max(0, n - head) / N;
    const T *xg = x + 3 * head;
    const int q = threadIdx.x;
    const bool outside = q < n - N * ng;  // at most 2 (N - 1)
    T o[3] = {p0, p1, p2};
    if (outside) {
        const T *xo = x + 3 * (q < head ? q : q + N * ng);
        o[0] = xo[0];
        o[1] = xo[1];
        o[2] = xo[2];
    }
#pragma unroll 2
    for (int g = threadIdx.x; g < ng; g += NT) {
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
    if (outside) {
        s[0] += o[0] - p0;
        s[1] += o[1] - p1;
        s[2] += o[2] - p2;
    }
#pragma unroll
    for (int off = LR / 2; off > 0; off >>= 1)
#pragma unroll
        for (int c = 0; c < 3; c++) s[c] += __shfl_xor_sync(0xffffffffu, s[c], off);
    if (lane % LR == 0)
#pragma unroll
        for (int c = 0; c < 3; c++) s_sum[threadIdx.x / LR][c] = (Sum)s[c];
    __syncthreads();
    if (threadIdx.x >= 32) return;
    if constexpr (ROWS <= 8) {  // a sum a lane
        if (lane < 3) {
            double t = 0.0;
#pragma unroll
            for (int q = 0; q < ROWS; q++) t += s_sum[q][lane];
            const double p = lane == 0 ? (double)p0 : (lane == 1 ? (double)p1 : (double)p2);
            center[3 * b + lane] = n > 0 ? (T)(p + t / n) : T(0);
        }
        return;
    }
    static_assert(ROWS <= 32, "a row a lane");
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
template <typename T, int NT>
__global__ void __launch_bounds__(NT, (sizeof(T) == 4 ? 2048 : 1536) / NT) bbox_kernel(const T *in, T *lo, T *hi, const int *num_atoms, int stride) {
    constexpr int NW = NT / 32, N = Vec16<T>::n;
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
    const int q = threadIdx.x;
    const bool outside = q < n - N * ng;  // the atoms before and after the groups, at most 2 (N - 1)
    T o[3];
    if (outside) {
        const T *xo = x + 3 * (q < head ? q : q + N * ng);
        o[0] = xo[0];
        o[1] = xo[1];
        o[2] = xo[2];
    }
#pragma unroll 2
    for (int g = threadIdx.x; g < ng; g += NT) {
        T v[3 * N];
        load_group(xg + 3 * N * g, v);
#pragma unroll
        for (int i = 0; i < N; i++) add(v + 3 * i);
    }
    if (outside) add(o);
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

// Rows that cannot move as vectors throughout: the vectors between the boundaries cost a
// second round of loads for the elements outside them, which only pays where there is enough
// to move. Elements / vectors, us: float32 4096 rows of 101 atoms 6.0 / 6.4, of 401 11.4 / 8.8;
// 64 of 2001 2.8 / 3.0, 150 3.5 / 3.1; float64 1000 of 1001 8.6 / 8.9, 4096 34.9 / 32.9.
template <typename T, bool SCALE>
static void launch_shift(const ShiftArgs &a, cudaStream_t st) {
    constexpr int N = Vec16<T>::n;
    auto grid = [&](int per_item) { return grid_rows(a.B, ((a.row + per_item - 1) / per_item + kUnroll - 1) / kUnroll); };
    auto aligned16 = [](const void *p) { return ((uintptr_t)p & 15u) == 0; };
    if (a.row % N == 0 && aligned16(a.out) && aligned16(a.in))
        shift_kernel<T, true, SCALE && sizeof(T) == 8><<<grid(N), 256, 0, st>>>(a);
    else if (a.row < 900 || (long long)a.B * a.row < (sizeof(T) == 4 ? 600000 : 6000000))
        shift_kernel<T, false, SCALE && sizeof(T) == 8><<<grid(1), 256, 0, st>>>(a);
    else
        shift_rows_kernel<T, SCALE><<<grid(N), 256, 0, st>>>(a);
}

template <typename T>
int coords_shift(const T *in, T *out, const T *add, int scale_by_count, const int *num_atoms, int B, int stride,
                 cudaStream_t st) {
    if (B == 0 || stride == 0) return TPL_OK;
    const ShiftArgs a{in, out, add, num_atoms, B, 3 * stride, scale_by_count};
    if (scale_by_count) launch_shift<T, true>(a, st);
    else launch_shift<T, false>(a, st);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <typename T>
int coords_rotate(const T *in, T *out, const T *R, int transpose, const int *num_atoms, int B, int stride,
                  cudaStream_t st) {
    if (B == 0 || stride == 0) return TPL_OK;
    if constexpr (sizeof(T) == 4) {
        if (stride >= 1500 && (long long)B * stride >= 5000000) {
            const long long groups = (stride + Vec16<T>::n - 1) / Vec16<T>::n;
            rotate_tiles_kernel<<<grid_rows(B, (groups + 1) / 2), 256, 0, st>>>(in, out, R, num_atoms, B, stride,
                                                                               transpose);
            return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
        }
    }
    rotate_kernel<T><<<grid_rows(B, (stride + kUnroll - 1) / kUnroll), 256, 0, st>>>(in, out, R, num_atoms, B, stride,
                                                                                   transpose);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <typename T>
int coords_center(const T *in, T *center, const int *num_atoms, int B, int stride, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    if (wide_reduction<T>(B, stride, false)) center_kernel<T, 256><<<B, 256, 0, st>>>(in, center, num_atoms, stride);
    else center_kernel<T, 128><<<B, 128, 0, st>>>(in, center, num_atoms, stride);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <typename T>
int coords_bbox(const T *in, T *lo, T *hi, const int *num_atoms, int B, int stride, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    if (wide_reduction<T>(B, stride, true)) bbox_kernel<T, 256><<<B, 256, 0, st>>>(in, lo, hi, num_atoms, stride);
    else bbox_kernel<T, 128><<<B, 128, 0, st>>>(in, lo, hi, num_atoms, stride);
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
