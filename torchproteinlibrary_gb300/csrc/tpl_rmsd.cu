// Coords2RMSD on the GPU: least RMSD after optimal superposition, with its
// gradient.  The reference (Layers/RMSD/Coords2RMSD/coords2rmsd_interface.cpp:52-111,
// RMSDKernels.cu:5-57) builds the 3x3 correlation on the GPU with one thread per
// matrix entry, copies the 4x4 quaternion matrix to the CPU for an eigen solve per
// chain, computes sum |x|^2 with single-thread kernels, and backpropagates with a
// Python loop of .item() calls (TorchProteinLibrary/RMSD/Coords2RMSD/Coords2RMSD.py:40-62).
//
// Here one CTA per chain does everything in one launch: optional centring, the
// correlation R_ab = sum x_a y_b and R2 = sum |x|^2 + |y|^2 (float32: FP32 per thread and
// over four or eight lanes, two-float sums from there, FP64 from the moments on; float64:
// FP64 throughout), the 4x4 matrix T (same
// layout as the reference), its largest eigenpair by the characteristic-polynomial
// method on one warp (key_eigen_halves), U from the unit quaternion, UT = U^T and
// rmsd = sqrt((R2 - 2 |lambda_max| + 1e-10) / N).  The backward is one launch with
// one thread per atom (chains on x, blocks of atoms on y):
// dL/dx_i = g (x_i - UT y_i) / (rmsd N) on the centred coordinates.
//
// What bounds the float32 forward is the FP64 pipe: GB300 issues two FP64 lanes per
// cycle and SM, conversions included, so an FP64 instruction of any warp holds the pipe
// for 16 cycles whether one lane or 32 take part.  A form with every warp's partial sums
// converted and the solve written for one lane spent about 280 of them per chain (ncu:
// FP64 pipe 73 % busy; 4096 chains of 400..2303 atoms, 20 us of HBM traffic: 90 us per
// layer call); this one, which solves two chains with the same instructions and reads the
// coordinates once, about 45 (FP64 pipe 26 % busy): 37 us.
#include <cmath>
#include <cstring>

#include "tpl_common.cuh"
#include "tpl_internal.h"
#include "tpl_rows.cuh"

namespace tpl {

constexpr int kRmsdThreads = 256;

template <typename T>
struct RmsdArgs {
    const T *src;
    const T *dst;
    const int *num_atoms;
    int atoms_stride;
    int center;
    T *rmsd;
    T *ut;              // [B, 9]
    double *centroids;  // [B, 6] (src, dst), may be null
    const T *grad_rmsd;
    T *grad_src;
    WsHeader *hdr;
};

constexpr int kRmsdWarps = kRmsdThreads / 32;

// Block sums of NV per-thread values (the float64 forward): a shuffle tree within each warp,
// then across the warps on one lane per value.  Every thread returns with the sums in s_out.
template <int NV>
__device__ __forceinline__ void block_sums(double (&v)[NV], double *s_red, double *s_out) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int k = 0; k < NV; k++) v[k] += __shfl_xor_sync(0xffffffffu, v[k], off);
    if (lane == 0)
#pragma unroll
        for (int k = 0; k < NV; k++) s_red[w * NV + k] = v[k];
    __syncthreads();
    if (threadIdx.x < NV) {
        double r = 0.0;
#pragma unroll
        for (int i = 0; i < kRmsdWarps; i++) r += s_red[i * NV + threadIdx.x];
        s_out[threadIdx.x] = r;
    }
    __syncthreads();
}

__device__ __forceinline__ double det3(double a, double b, double c, double d, double e, double f, double g, double h,
                                       double k) {
    return a * (e * k - f * h) - b * (d * k - f * g) + c * (d * h - e * g);
}

// Largest eigenpair of the symmetric 4x4 K by cyclic Jacobi rotations in FP64, on one
// thread: the fallback of key_eigen_halves for a near-multiple largest root (collinear
// or otherwise degenerate structures, two-atom chains), where Newton on the quartic
// converges only linearly and stalls at about the square root of the rounding error.
// Rotation (p, r) with t = sgn(theta) / (|theta| + sqrt(theta^2 + 1)),
// theta = (a_rr - a_pp) / (2 a_pr), zeroes a_pr (A' = J^T A J, V' = V J).  a and v
// are 16 doubles of shared scratch each, so that the rare path adds no registers to
// the kernel.
__device__ __forceinline__ void jacobi_top_eigenpair(const double *K, double *a, double *v, double &lam,
                                                  double (&q)[4]) {
    for (int i = 0; i < 16; i++) {
        a[i] = K[i];
        v[i] = (i % 5 == 0) ? 1.0 : 0.0;
    }
    for (int sweep = 0; sweep < 16; sweep++) {
        double off = 0.0, dg = 0.0;
        for (int i = 0; i < 4; i++) {
            dg += a[5 * i] * a[5 * i];
            for (int j = i + 1; j < 4; j++) off += a[4 * i + j] * a[4 * i + j];
        }
        if (!(off > 1e-30 * (dg + off))) break;
        for (int p = 0; p < 3; p++)
            for (int r = p + 1; r < 4; r++) {
                const double apr = a[4 * p + r];
                if (!(fabs(apr) > 1e-300)) continue;
                const double theta = (a[5 * r] - a[5 * p]) / (2.0 * apr);
                const double t = (theta >= 0.0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
                const double c = 1.0 / sqrt(t * t + 1.0), sn = t * c;
                for (int k = 0; k < 4; k++) {  // A J
                    const double akp = a[4 * k + p], akr = a[4 * k + r];
                    a[4 * k + p] = c * akp - sn * akr;
                    a[4 * k + r] = sn * akp + c * akr;
                }
                for (int k = 0; k < 4; k++) {  // J^T (A J)
                    const double apk = a[4 * p + k], ark = a[4 * r + k];
                    a[4 * p + k] = c * apk - sn * ark;
                    a[4 * r + k] = sn * apk + c * ark;
                }
                for (int k = 0; k < 4; k++) {  // V J
                    const double vkp = v[4 * k + p], vkr = v[4 * k + r];
                    v[4 * k + p] = c * vkp - sn * vkr;
                    v[4 * k + r] = sn * vkp + c * vkr;
                }
            }
    }
    int best = 0;
    for (int i = 1; i < 4; i++)
        if (a[5 * i] > a[5 * best]) best = i;
    lam = a[5 * best];
#pragma unroll
    for (int k = 0; k < 4; k++) q[k] = v[4 * k + best];
}

// The eigenvector of key_eigen_halves<true>, in FP32: the largest row of the cofactor
// matrix of M = K - l I (entries of order one, in shared memory), one cofactor per
// lane of each half warp.  The root itself stays FP64: when the top two eigenvalues nearly
// meet it is ill-conditioned, and an all-FP32 solve moved it by up to 3e-5 relative (a 2.4e-4
// gradient error on one of 256 training-step chains), where this form matches the
// FP64 solve to 1e-5 of the largest gradient.
__device__ void eigvec_f32(const float *sM, double (&q)[4]) {
    float cf;
    {
        const int i = (threadIdx.x & 15) >> 2, j = threadIdx.x & 3;
        float m[9];  // rows but i, columns but j
#pragma unroll
        for (int t = 0; t < 9; t++) m[t] = sM[4 * (t / 3 + (t / 3 >= i)) + t % 3 + (t % 3 >= j)];
        cf = fmaf(m[0], fmaf(m[4], m[8], -m[5] * m[7]),
                  fmaf(-m[1], fmaf(m[3], m[8], -m[5] * m[6]), m[2] * fmaf(m[3], m[7], -m[4] * m[6])));
        if ((i + j) & 1) cf = -cf;
    }
    float nrm = cf * cf;
    nrm += __shfl_xor_sync(0xffffffffu, nrm, 1);
    nrm += __shfl_xor_sync(0xffffffffu, nrm, 2);
    int best = 0;
    float bn = __shfl_sync(0xffffffffu, nrm, 0, 16);
    for (int i = 1; i < 4; i++) {
        const float v = __shfl_sync(0xffffffffu, nrm, 4 * i, 16);
        if (v > bn) {
            bn = v;
            best = i;
        }
    }
    const bool ok = bn > 1e-30f;
    const float inv = ok ? rsqrtf(bn) : 0.f;
#pragma unroll
    for (int k = 0; k < 4; k++) q[k] = (double)(__shfl_sync(0xffffffffu, cf, 4 * best + k, 16) * inv);
    if (!ok) {
        q[0] = 1.0;
        q[1] = q[2] = q[3] = 0.0;
    }
}

// Power of two that scales e0 into [0.5, 1), and its inverse (1 for e0 = 0, clamped well
// inside the exponent range): the key matrix of a scaled correlation has coefficients
// and eigenvalues of order one, and scaling back is exact.
__device__ __forceinline__ void unit_scale(double e0, double &scale, double &inv) {
    int e = ((__double2hiint(e0) >> 20) & 0x7ff) - 1022;
    e = e0 != 0.0 ? max(-900, min(900, e)) : 0;
    scale = __hiloint2double((1023 - e) << 20, 0);
    inv = __hiloint2double((1023 + e) << 20, 0);
}

// The key matrix entry by entry (row-major, reference layout,
// coords2rmsd_interface.cpp:146-149): K_e = +-R[a] +- R[b], and +- R[8] on the diagonal.
constexpr int kKeyA[16] = {0, 5, 6, 1, 5, 0, 1, 2, 6, 1, 0, 5, 1, 2, 5, 0};
constexpr int kKeyB[16] = {4, 7, 2, 3, 7, 4, 3, 6, 2, 3, 4, 7, 3, 6, 7, 4};
constexpr unsigned kKeyNegA = 0x8400u, kKeyNegB = 0x913eu, kKeyNegC = 0x0420u;  // entries with a minus sign
constexpr uint64_t pack_nibbles(const int (&v)[16]) {
    uint64_t w = 0;
    for (int i = 0; i < 16; i++) w |= (uint64_t)v[i] << (4 * i);
    return w;
}
__device__ __forceinline__ double negate_if(double v, bool neg) {  // on the sign bit: no FP64 instruction
    return __hiloint2double(__double2hiint(v) ^ (neg ? 0x80000000 : 0), __double2loint(v));
}

// Largest eigenpair of the 4x4 key matrix K (symmetric and traceless) of the
// correlation R by its characteristic polynomial, as in Theobald's
// quaternion-characteristic-polynomial method (Acta Cryst. A61, 478, 2005):
// det(K - l I) = l^4 + c2 l^2 + c1 l + c0, c2 = -2 |R|^2, c1 = -8 det R, c0 = det K.
//   * R (nine doubles, shared memory) and e0 = (sum |x|^2 + |y|^2) / 2 >= l_max come
//     scaled by unit_scale(), so nothing is divided to bring them to order one.
//   * FP64 instructions are few: one entry of K per lane (two additions), |R|^2 as a
//     shuffle sum, the cofactor expansion of det K along row 0 on four lanes and det R on
//     four others in the same instructions.
//   * Newton's method from e0 descends monotonically to the largest root.  It runs in
//     FP32 and is then polished by three FP64 Newton steps whose quotient uses an FP32
//     reciprocal (each step gains about seven digits).
//   * The eigenvector is the largest row of the cofactor matrix of K - l I (rank one
//     for a simple root), one cofactor per lane.
//   * F32_VEC (float32 inputs): the eigenvector in FP32 instead (eigvec_f32).
// Executed by a full warp whose halves of 16 lanes each solve a problem of their own (an
// FP64 instruction costs the same for both): sR, e0 and the scratch sK (16 doubles), sM
// (16 floats) and s_jac (32 doubles) are the half's; every lane of it returns its l
// (scaled) and unit q (q = 1, 0, 0, 0 when every cofactor vanishes).
template <bool F32_VEC>
__device__ void key_eigen_halves(const double *sR, double e0, double *sK, float *sM, double *s_jac, double &l,
                                 double (&q)[4]) {
    const int e = threadIdx.x & 15;
    constexpr uint64_t kA = pack_nibbles(kKeyA), kB = pack_nibbles(kKeyB);
    const bool diag = (e >> 2) == (e & 3);
    double k = negate_if(sR[(kA >> (4 * e)) & 15], (kKeyNegA >> e) & 1u) +
               negate_if(sR[(kB >> (4 * e)) & 15], (kKeyNegB >> e) & 1u);
    if (diag) k += negate_if(sR[8], (kKeyNegC >> e) & 1u);
    sK[e] = k;
    double t2 = e < 9 ? sR[e] : 0.0;
    t2 *= t2;
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) t2 += __shfl_xor_sync(0xffffffffu, t2, off);
    const double c2 = -2.0 * t2;
    __syncwarp();
    double c0, c1;
    {
        const int j = e & 3;  // lanes 0..3: the minor of K without row 0 and column j; 4..7: R
        double m[9];
#pragma unroll
        for (int t = 0; t < 9; t++)
            m[t] = *((e & 4) ? sR + t : sK + 4 * (1 + t / 3) + t % 3 + (t % 3 >= j));
        const double d = det3(m[0], m[1], m[2], m[3], m[4], m[5], m[6], m[7], m[8]);
        double s = negate_if(sK[j], j & 1) * d;
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        c0 = __shfl_sync(0xffffffffu, s, 0, 16);
        c1 = -8.0 * __shfl_sync(0xffffffffu, d, 4, 16);
    }
    l = 0.0;
    bool simple = true;
    if (e0 > 0.0) {
        const float e0f = (float)e0, a2 = (float)c2, a1 = (float)c1, a0 = (float)c0;
        float s = e0f * 1.0000002f;  // not below e0
        for (int it = 0; it < 64; it++) {
            const float P = fmaf(fmaf(fmaf(s, s, a2), s, a1), s, a0);
            const float dP = fmaf(fmaf(4.f * s, s, 2.f * a2), s, a1);
            if (!(dP != 0.f)) break;
            const float d = P / dP;
            s -= d;
            if (fabsf(d) <= 1e-6f * e0f) break;
        }
        l = (double)s;
        float corr = INFINITY;  // the last polish step
        for (int it = 0; it < 3; it++) {
            const double l2 = l * l;
            const double P = fma(fma(l2 + c2, l, c1), l, c0);
            const double dP = fma(fma(4.0, l2, 2.0 * c2), l, c1);
            const float dPf = (float)dP;
            if (!(dPf != 0.f) || !isfinite(dPf)) {
                corr = INFINITY;
                break;
            }
            const double d = P * (double)(1.f / dPf);
            l -= d;
            corr = (float)d;
        }
        // a simple root has converged by the third polish step (each gains about
        // seven digits); a near-multiple one (the top eigenvalues of K nearly or
        // exactly equal) converges only linearly: a last step above 1e-10 of e0 sends
        // the chain to the Jacobi solve (the same decision on every lane of the half)
        simple = fabsf(corr) <= 1e-10f * e0f;
    }
    __syncwarp();
    if (F32_VEC) {
        if (diag) k -= l;
        sM[e] = (float)k;
        __syncwarp();
        eigvec_f32(sM, q);
    } else {
        // cofactor (i, j) of M = K - l I on lane 4 i + j
        const int i = e >> 2, j = e & 3;
        double m[9];  // rows but i, columns but j
#pragma unroll
        for (int t = 0; t < 9; t++) {
            const int r = t / 3 + (t / 3 >= i), c = t % 3 + (t % 3 >= j);
            m[t] = sK[4 * r + c] - (r == c ? l : 0.0);
        }
        double cof = det3(m[0], m[1], m[2], m[3], m[4], m[5], m[6], m[7], m[8]);
        if ((i + j) & 1) cof = -cof;
        // squared norm of the row of this lane (lanes 4 i .. 4 i + 3)
        double nrm = cof * cof;
        nrm += __shfl_xor_sync(0xffffffffu, nrm, 1);
        nrm += __shfl_xor_sync(0xffffffffu, nrm, 2);
        int best = 0;
        double bn = __shfl_sync(0xffffffffu, nrm, 0, 16);
        for (int r = 1; r < 4; r++) {
            const double v = __shfl_sync(0xffffffffu, nrm, 4 * r, 16);
            if (v > bn) {
                bn = v;
                best = r;
            }
        }
        const double inv = bn > 1e-300 ? 1.0 / sqrt(bn) : 0.0;
#pragma unroll
        for (int r = 0; r < 4; r++) q[r] = __shfl_sync(0xffffffffu, cof, 4 * best + r, 16) * inv;
        if (!(bn > 1e-300)) {
            q[0] = 1.0;
            q[1] = q[2] = q[3] = 0.0;
        }
    }
    if (__any_sync(0xffffffffu, !simple)) {
        double lj = 0.0, qj[4] = {1.0, 0.0, 0.0, 0.0};
        if (!simple && e == 0) jacobi_top_eigenpair(sK, s_jac, s_jac + 16, lj, qj);
        __syncwarp();
        lj = __shfl_sync(0xffffffffu, lj, 0, 16);
#pragma unroll
        for (int i = 0; i < 4; i++) qj[i] = __shfl_sync(0xffffffffu, qj[i], 0, 16);
        if (!simple) {
            l = lj;
#pragma unroll
            for (int i = 0; i < 4; i++) q[i] = qj[i];
        }
    }
}

// Rotation of the unit quaternion q, transposed (coords2rmsd_interface.cpp:36-46).
template <typename T>
__device__ __forceinline__ void store_ut(T *ut, T q0, T q1, T q2, T q3) {
    ut[0] = q0 * q0 + q1 * q1 - q2 * q2 - q3 * q3;
    ut[3] = T(2) * (q1 * q2 - q0 * q3);
    ut[6] = T(2) * (q1 * q3 + q0 * q2);
    ut[1] = T(2) * (q1 * q2 + q0 * q3);
    ut[4] = q0 * q0 - q1 * q1 + q2 * q2 - q3 * q3;
    ut[7] = T(2) * (q2 * q3 - q0 * q1);
    ut[2] = T(2) * (q1 * q3 - q0 * q2);
    ut[5] = T(2) * (q2 * q3 + q0 * q1);
    ut[8] = q0 * q0 - q1 * q1 - q2 * q2 + q3 * q3;
}

template <typename T>
__device__ __forceinline__ int checked_atoms(const RmsdArgs<T> &a, int b, bool reports) {
    const int n = a.num_atoms[b];
    if (n >= 0 && n <= a.atoms_stride) return n;
    if (reports && a.hdr) atomicCAS(&a.hdr->status, 0u, (unsigned)TPL_ERR_ATOMS);
    return max(0, min(n, a.atoms_stride));
}

constexpr int kRmsdSums = 16;  // R (row-major), R2, sum x, sum y

// Value k of the 16 sums of a chain of n atoms again, from the centres c: one lane a value,
// four atoms in FP32 at a time.  Rare, and so out of the way of the kernel's registers.
__device__ __forceinline__ double sum_again(const float *x, const float *y, int n, const float *c, int k) {
    // what the value is a sum of: components p and r (3..5: y) multiplied, or p alone
    const int p = k < 9 ? k / 3 : k - 10, r = k < 9 ? 3 + k % 3 : -1;
    auto at = [&](int i, int q) { return (q < 3 ? x[3 * i + q] : y[3 * i + q - 3]) - c[q]; };
    double d = 0.0;
#pragma unroll 1
    for (int i0 = 0; i0 < n; i0 += 4) {
        float s = 0.f;
#pragma unroll 1
        for (int i = i0; i < min(i0 + 4, n); i++) {
            if (k == 9) {
#pragma unroll 1
                for (int q = 0; q < 6; q++) s = fmaf(at(i, q), at(i, q), s);
            } else {
                s = fmaf(at(i, p), r < 0 ? 1.f : at(i, r), s);
            }
        }
        d += (double)s;
    }
    return d;
}

// float32 forward: one pass over the chain.  Both sets are taken relative to a
// provisional centre, the mean of 16 atoms spread over the chain, and the sums are
// moved to the true centroids afterwards in FP64 (R - n cx cy^T and so on): the
// provisional centre is off by a quarter of the radius of gyration where the 16 atoms are
// drawn like the others (a twentieth along a coil), so the sums keep the size, and the
// rounding, of centred ones, and the second read of every coordinate goes.  Where they are
// not, and the shift makes up more than a third of sum |x|^2 + |y|^2 (of independent points
// one chain in 1e8), the sums are taken again from the centroids found (sum_again; a coil of
// 2300 atoms whose sampled ones are 300 A off: 8e-4 relative without, 7e-6 with).  Atoms are
// read as float4 groups (tpl_rows.cuh) where both rows
// have the same alignment.
//
// NC = 1 or 2 chains per CTA, NT threads each; the first warp then solves for both, one per
// half, as an FP64 instruction costs the same for 16 lanes or 32.
template <int NT, int NC>
__global__ void __launch_bounds__(NT * NC) rmsd_fwd_f32_kernel(RmsdArgs<float> a, int nb) {
    constexpr int LR = NT > 64 ? 8 : 4;  // lanes summed in FP32
    constexpr int ROWS = NT / LR;
    __shared__ __align__(16) float s_red[NC][ROWS][kRmsdSums];
    __shared__ double s_R[2][9], s_K[2][16], s_jac[2][32];
    __shared__ float s_M[2][16], s_c[NC][6];
    __shared__ int s_n[NC];
    const int ch = NC == 1 ? 0 : threadIdx.x / NT, tid = threadIdx.x - ch * NT, lane = tid & 31, w = tid >> 5;
    const int b = min(NC * (int)blockIdx.x + ch, nb - 1);
    const bool own = NC * (int)blockIdx.x + ch < nb;  // false: the last CTA's half without a chain
    const int n = own ? checked_atoms(a, b, tid == 0) : 0;
    const float *x = a.src + (size_t)b * 3 * a.atoms_stride;
    const float *y = a.dst + (size_t)b * 3 * a.atoms_stride;
    // The thread's first group is asked for before the centres are known: a small batch
    // then waits for memory once less.  (Not in the form for large batches, where it takes
    // 16 more registers.)
    constexpr bool kAhead = NC == 1;
    const int head = row_head(x), ng = head == row_head(y) ? max(0, n - head) >> 2 : 0;
    const float *xg = x + 3 * head, *yg = y + 3 * head;
    float xv[12], yv[12];
    if (kAhead && tid < ng) {
        load_group(xg + 12 * tid, xv);
        load_group(yg + 12 * tid, yv);
    }
    float c[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};  // provisional centres, the same on every thread
    if (a.center && n > 0) {
        const size_t i = (size_t)n * (2 * (lane & 15) + 1) / 32;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            c[k] = x[3 * i + k];
            c[3 + k] = y[3 * i + k];
        }
#pragma unroll
        for (int off = 8; off > 0; off >>= 1)
#pragma unroll
            for (int k = 0; k < 6; k++) c[k] += __shfl_xor_sync(0xffffffffu, c[k], off);
#pragma unroll
        for (int k = 0; k < 6; k++) c[k] *= 1.f / 16.f;
    }
    float v[kRmsdSums];
#pragma unroll
    for (int k = 0; k < kRmsdSums; k++) v[k] = 0.f;
    auto add = [&](float (&s)[kRmsdSums], const float *xa, const float *ya) {
        const float xi[3] = {xa[0] - c[0], xa[1] - c[1], xa[2] - c[2]}, yi[3] = {ya[0] - c[3], ya[1] - c[4], ya[2] - c[5]};
#pragma unroll
        for (int p = 0; p < 3; p++) {
#pragma unroll
            for (int r = 0; r < 3; r++) s[3 * p + r] = fmaf(xi[p], yi[r], s[3 * p + r]);
            s[10 + p] += xi[p];
            s[13 + p] += yi[p];
        }
        s[9] += xi[0] * xi[0] + xi[1] * xi[1] + xi[2] * xi[2] + yi[0] * yi[0] + yi[1] * yi[1] + yi[2] * yi[2];
    };
    auto add_group = [&]() {
        float s[kRmsdSums];  // the group's own sums first: fewer roundings at the size of the running sums
#pragma unroll
        for (int k = 0; k < kRmsdSums; k++) s[k] = 0.f;
#pragma unroll
        for (int q = 0; q < 4; q++) add(s, xv + 3 * q, yv + 3 * q);
#pragma unroll
        for (int k = 0; k < kRmsdSums; k++) v[k] += s[k];
    };
    if (kAhead && tid < ng) add_group();
#pragma unroll 2
    for (int g = kAhead ? tid + NT : tid; g < ng; g += NT) {
        load_group(xg + 12 * g, xv);
        load_group(yg + 12 * g, yv);
        add_group();
    }
    // the atoms before the groups come after the last group's
    const int i0 = ng > 0 ? head + 4 * ng : 0, nhead = ng > 0 ? head : 0;
    for (int i = i0 + tid - nhead; i < n; i += NT) {
        const int at = i < i0 ? i - i0 + nhead : i;  // the nhead atoms before the groups, then the rest
        add(v, x + 3 * at, y + 3 * at);
    }
    // Sums over LR lanes: a lane hands half of its values to its partner and keeps the sums
    // of the other half, so that 16 values take 14 shuffles (12 for four lanes).  The sums of
    // a warp's groups and the warps are then added in more than FP32: FP32 additions of ever
    // larger sums up to the whole warp were most of the rounding error (rmsd against FP64,
    // 4096 chains of 400..2303 atoms: 1.4e-6 with all five levels in FP32; the fewer threads
    // a chain has, the larger its threads' sums, hence four lanes for 64).
    constexpr int LEFT = kRmsdSums / LR;  // values a lane is left with
    static_assert((LR == 8 || LR == 4) && LEFT * LR == kRmsdSums && ROWS * LR == NT, "rows of s_red");
#pragma unroll
    for (int off = 16, h = kRmsdSums / 2; h >= LEFT; off >>= 1, h >>= 1) {
        const bool up = (lane & off) != 0;
#pragma unroll
        for (int k = 0; k < h; k++) {
            const float give = up ? v[k] : v[k + h], keep = up ? v[k + h] : v[k];
            v[k] = keep + __shfl_xor_sync(0xffffffffu, give, off);
        }
    }
    // values LEFT (lane / LR) and the next ones, summed over the lanes with this lane's low bits
    if constexpr (LEFT == 2)
        *reinterpret_cast<float2 *>(&s_red[ch][4 * w + (lane & 3)][2 * (lane >> 2)]) = make_float2(v[0], v[1]);
    else
        *reinterpret_cast<float4 *>(&s_red[ch][8 * w + (lane & 7)][4 * (lane >> 3)]) =
            make_float4(v[0], v[1], v[2], v[3]);
    if (tid == 0) {
        s_n[ch] = n;
#pragma unroll
        for (int k = 0; k < 6; k++) s_c[ch][k] = c[k];
    }
    __syncthreads();
    if (threadIdx.x >= 32) return;

    // The first warp: value k of chain h on lane 16 h + k (one chain: half the rows on each
    // half).  The rows are added exactly but for the last bits of a two-float sum (Knuth's
    // two-sum; 47 bits), which costs three FP64 instructions instead of two a row, then moved
    // to the true centroids in FP64.
    const int half = lane >> 4, h = NC == 1 ? 0 : half, k = lane & 15;
    const int bh = NC * (int)blockIdx.x + h, nh = s_n[h];
    const bool writes = NC == 1 ? half == 0 : bh < nb;
    constexpr int R = NC == 1 ? ROWS / 2 : ROWS;
    float hi = 0.f, lo = 0.f;
#pragma unroll
    for (int i = 0; i < R; i++) {
        const float u = s_red[h][(NC == 1 ? R * half : 0) + i][k], t = hi + u, z = t - hi;
        lo += (hi - (t - z)) + (u - z);
        hi = t;
    }
    double d = (double)hi + (fabsf(hi) <= 3.402823466e38f ? (double)lo : 0.0);  // an infinite sum stays one
    if (NC == 1) d += __shfl_xor_sync(0xffffffffu, d, 16);
    if (a.center) {
        double rn = 0.0;  // 1 / n: an FP32 reciprocal and one Newton step
        if (nh > 0) {
            rn = (double)(1.f / (float)nh);
            rn = fma(rn, fma(-(double)nh, rn, 1.0), rn);
        }
#pragma unroll 1
        for (bool first = true;; first = false) {
            const double m = d * rn;  // lanes 10 .. 15: the centroids from the provisional centres
            if (k >= 10 && writes && a.centroids) a.centroids[6 * bh + k - 10] = (double)s_c[h][k - 10] + m;
            const double sx = __shfl_sync(0xffffffffu, d, 10 + (k < 9 ? k / 3 : 0), 16);
            const double my = __shfl_sync(0xffffffffu, m, 13 + (k < 9 ? k % 3 : 0), 16);
            double sq = k >= 10 ? d * m : 0.0;
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, off);
            if (!first || !__any_sync(0xffffffffu, k == 9 && 3.0 * sq > d)) {
                d -= k < 9 ? sx * my : sq;
                break;
            }
            if (k >= 10 && writes) s_c[h][k - 10] = (float)((double)s_c[h][k - 10] + m);
            __syncwarp();
            const size_t row = (size_t)min(bh, nb - 1) * 3 * a.atoms_stride;
            d = sum_again(a.src + row, a.dst + row, nh, s_c[h], k);
        }
    } else if (k < 6 && writes && a.centroids) {
        a.centroids[6 * bh + k] = 0.0;
    }
    const double r2 = __shfl_sync(0xffffffffu, d, 9, 16);
    double scale, inv;
    unit_scale(0.5 * r2, scale, inv);
    if (k < 9) s_R[half][k] = d * scale;
    __syncwarp();
    double l, q[4];
    key_eigen_halves<true>(s_R[half], 0.5 * r2 * scale, s_K[half], s_M[half], s_jac[half], l, q);
    if (k != 0 || !writes) return;
    store_ut(a.ut + (size_t)9 * bh, (float)q[0], (float)q[1], (float)q[2], (float)q[3]);
    const float msd = nh > 0 ? (float)(r2 - 2.0 * fabs(l * inv) + 1e-10) * (1.f / (float)nh) : 0.f;
    a.rmsd[bh] = sqrtf(msd > 0.f ? msd : 0.f);
}

// float64 forward: two passes (centroids, then the correlation), everything in FP64.
__global__ void __launch_bounds__(kRmsdThreads) rmsd_fwd_f64_kernel(RmsdArgs<double> a) {
    __shared__ double s_red[kRmsdWarps * 10];
    __shared__ double s_out[10];
    __shared__ double s_R[9], s_K[2][16];
    __shared__ double s_jac[2][32];  // scratch of the Jacobi fallback
    __shared__ double s_c[6];     // centroids (src, dst)
    const int b = blockIdx.x, tid = threadIdx.x;
    const int n = checked_atoms(a, b, tid == 0);
    const double *x = a.src + (size_t)b * 3 * a.atoms_stride;
    const double *y = a.dst + (size_t)b * 3 * a.atoms_stride;
    if (a.center) {
        double sx[6] = {0, 0, 0, 0, 0, 0};
#pragma unroll 4
        for (int i = tid; i < n; i += kRmsdThreads)
            for (int k = 0; k < 3; k++) {
                sx[k] += x[3 * i + k];
                sx[3 + k] += y[3 * i + k];
            }
        block_sums<6>(sx, s_red, s_out);
        if (tid < 6) s_c[tid] = n > 0 ? s_out[tid] / n : 0.0;
    } else if (tid < 6) {
        s_c[tid] = 0.0;
    }
    __syncthreads();
    double ct[6];
    for (int k = 0; k < 6; k++) ct[k] = s_c[k];
    double acc[10] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};  // R (row-major) and R2
#pragma unroll 4
    for (int i = tid; i < n; i += kRmsdThreads) {
        double xi[3], yi[3];
        for (int k = 0; k < 3; k++) {
            xi[k] = x[3 * i + k] - ct[k];
            yi[k] = y[3 * i + k] - ct[3 + k];
        }
        for (int p = 0; p < 3; p++)
            for (int q = 0; q < 3; q++) acc[3 * p + q] = fma(xi[p], yi[q], acc[3 * p + q]);
        acc[9] += xi[0] * xi[0] + xi[1] * xi[1] + xi[2] * xi[2] + yi[0] * yi[0] + yi[1] * yi[1] + yi[2] * yi[2];
    }
    block_sums<10>(acc, s_red, s_out);
    if (tid >= 32) return;
    const double r2 = s_out[9];
    double scale, inv;
    unit_scale(0.5 * r2, scale, inv);
    if (tid < 9) s_R[tid] = s_out[tid] * scale;
    __syncwarp();
    double l, q[4];
    const int half = tid >> 4;  // both halves solve the same chain
    key_eigen_halves<false>(s_R, 0.5 * r2 * scale, s_K[half], nullptr, s_jac[half], l, q);
    if (tid != 0) return;
    store_ut(a.ut + (size_t)9 * b, q[0], q[1], q[2], q[3]);
    const double msd = n > 0 ? (r2 - 2.0 * fabs(l * inv) + 1e-10) / (double)n : 0.0;
    a.rmsd[b] = sqrt(msd > 0.0 ? msd : 0.0);
    if (a.centroids)
        for (int k = 0; k < 6; k++) a.centroids[6 * b + k] = s_c[k];
}

// One atom per thread: a block's life is two memory latencies, and small blocks of few
// registers overlap them best.  (Groups of four atoms as 16-byte vectors, a thread each:
// 20000 chains of 1000 atoms 210 -> 151 us, but 4096 of 2300 71 -> 81, of 200 8 -> 14, 256 of
// 2300 5.4 -> 6.9, float64 4096 of 20 14 -> 24.)
template <typename T>
__global__ void __launch_bounds__(kRmsdThreads) rmsd_bwd_kernel(RmsdArgs<T> a) {
    const int b = blockIdx.x, tid = threadIdx.x;
    const int n = max(0, min(a.num_atoms[b], a.atoms_stride));
    const T *x = a.src + (size_t)b * 3 * a.atoms_stride;
    const T *y = a.dst + (size_t)b * 3 * a.atoms_stride;
    T *gx = a.grad_src + (size_t)b * 3 * a.atoms_stride;
    // per-chain constants once per block: converting the FP64 centroids on every
    // thread would keep GB300's slow FP64 pipe busy
    __shared__ T s_c[6], s_U[9], s_scale;
    if (tid < 6) s_c[tid] = (a.center && a.centroids) ? (T)a.centroids[6 * b + tid] : T(0);
    if (tid < 9) s_U[tid] = a.ut[(size_t)9 * b + tid];
    if (tid == 0) {
        const T r = a.rmsd[b];
        s_scale = (n > 0 && r > T(0)) ? a.grad_rmsd[b] / (r * (T)n) : T(0);
    }
    __syncthreads();
    T c[6], U[9];
    for (int k = 0; k < 6; k++) c[k] = s_c[k];
    for (int k = 0; k < 9; k++) U[k] = s_U[k];
    const T scale = s_scale;
    // one atom per thread: chains on x, blocks of atoms on y
    const int i = blockIdx.y * kRmsdThreads + tid;
    if (i < a.atoms_stride) {
        if (i < n) {
            T xi[3], yi[3];
            for (int k = 0; k < 3; k++) {
                xi[k] = x[3 * i + k] - c[k];
                yi[k] = y[3 * i + k] - c[3 + k];
            }
            for (int k = 0; k < 3; k++)
                gx[3 * i + k] = scale * (xi[k] - (U[3 * k] * yi[0] + U[3 * k + 1] * yi[1] + U[3 * k + 2] * yi[2]));
        } else {
            gx[3 * i] = gx[3 * i + 1] = gx[3 * i + 2] = T(0);
        }
    }
}

template <typename T>
static int rmsd_fwd_launch(const T *src, const T *dst, const int *num_atoms, int B, int stride, int center, T *rmsd,
                           T *ut, double *centroids, void *ws, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    RmsdArgs<T> a{src, dst, num_atoms, stride, center, rmsd, ut, centroids, nullptr, nullptr, (WsHeader *)ws};
    if constexpr (sizeof(T) == 4) {
        // Threads per chain: with few chains per SM the longest chain's loads bound the
        // launch (256 chains of 50..500 residues, training step as a graph: 65.7 / 66.6 /
        // 68.9 us at 512 / 256 / 128 threads); with many, a CTA holds its registers while
        // its first warp solves, so small CTAs keep more chains' loads in flight, and two
        // chains share a solve (forward of 4096 chains of up to 2303 atoms, threads x chains:
        // 128 x 1 42.9 us, 128 x 2 45.2, 64 x 1 40.3, 64 x 2 32.9, 32 x 2 31.7; of 1200
        // chains 20.0 / 12.9 / 14.3 / 12.8 / 15.4; of 620 chains 11.8 with 64 x 2 and 11.3
        // with 256 x 1).
        const int sms = device_sm_count();
        if (B <= 2 * sms) rmsd_fwd_f32_kernel<512, 1><<<B, 512, 0, st>>>(a, B);
        else if (B <= 4 * sms) rmsd_fwd_f32_kernel<256, 1><<<B, 256, 0, st>>>(a, B);
        else rmsd_fwd_f32_kernel<64, 2><<<B / 2 + B % 2, 128, 0, st>>>(a, B);
    } else {
        rmsd_fwd_f64_kernel<<<B, kRmsdThreads, 0, st>>>(a);
    }
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <typename T>
static int rmsd_bwd_launch(const T *grad_rmsd, const T *src, const T *dst, const int *num_atoms, const T *rmsd,
                           const T *ut, const double *centroids, int B, int stride, int center, T *grad_src,
                           cudaStream_t st) {
    if (B == 0) return TPL_OK;
    RmsdArgs<T> a{src, dst, num_atoms, stride, center, const_cast<T *>(rmsd), const_cast<T *>(ut),
                  const_cast<double *>(centroids), grad_rmsd, grad_src, nullptr};
    const int ablocks = (max(stride, 1) + kRmsdThreads - 1) / kRmsdThreads;
    if (ablocks > 65535) return TPL_ERR_UNSUPPORTED;
    rmsd_bwd_kernel<T><<<dim3((unsigned)B, (unsigned)ablocks), kRmsdThreads, 0, st>>>(a);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

int rmsd_forward(bool f64, const void *src, const void *dst, const int *num_atoms, int B, int stride, int center,
                 void *rmsd, void *ut, double *centroids, void *ws, cudaStream_t st) {
    if (f64)
        return rmsd_fwd_launch<double>((const double *)src, (const double *)dst, num_atoms, B, stride, center,
                                       (double *)rmsd, (double *)ut, centroids, ws, st);
    return rmsd_fwd_launch<float>((const float *)src, (const float *)dst, num_atoms, B, stride, center, (float *)rmsd,
                                  (float *)ut, centroids, ws, st);
}

int rmsd_backward(bool f64, const void *grad_rmsd, const void *src, const void *dst, const int *num_atoms,
                  const void *rmsd, const void *ut, const double *centroids, int B, int stride, int center,
                  void *grad_src, cudaStream_t st) {
    if (f64)
        return rmsd_bwd_launch<double>((const double *)grad_rmsd, (const double *)src, (const double *)dst, num_atoms,
                                       (const double *)rmsd, (const double *)ut, centroids, B, stride, center,
                                       (double *)grad_src, st);
    return rmsd_bwd_launch<float>((const float *)grad_rmsd, (const float *)src, (const float *)dst, num_atoms,
                                  (const float *)rmsd, (const float *)ut, centroids, B, stride, center,
                                  (float *)grad_src, st);
}

}  // namespace tpl
