// float64 Angles2Backbone and Angles2Coords (reference: the CPU layers,
// Layers/ReducedModel/cBackboneProteinCPUKernels.cpp:14-145 and
// Layers/FullAtomModel/cConformation.cpp:30-211), one thread-block cluster per chain.
//
// FP64 instructions bound these kernels: GB300 issues two FP64 lanes per cycle and SM, so
// one warp instruction holds an SM's FP64 pipe for 16 cycles however many lanes take
// part.  Hence
//   * few FP64 instructions: sines from a 29-instruction polynomial (sincos_f64), one scan
//     over a warp (18 instructions a level, scan_inclusive) instead of one over a block,
//     and joints walked once (the backbone's local positions stay in registers);
//   * full warps: R residues per lane share one scan, frames of earlier chunks are composed
//     one matrix entry per lane (three instructions a chunk), lanes that a scan has no work
//     for take half of their neighbours', and warps whose chunk holds no residue of the chain
//     only pass the barriers; four CTAs of the backbone kernels per SM, whose spills cost
//     nothing beside the FP64 pipe (backward, three: 256 chains 96.3 against 86.6 us);
//   * every SM: a chain's chunks of 32 R residues are spread over the CTAs of a cluster of
//     1 to 8, which exchange one frame (and, backward, six sums) per chunk through
//     distributed shared memory.  A chain longer than the cluster's capacity is taken in
//     passes.
// Positions are kept relative to the pass's first joint, in world orientation.
//
// GB300, against one CTA per chain with block-wide scans (forward, backward): Angles2Backbone
// 256 chains of 60..350 residues 124 -> 54 us, 268 -> 87 us; Angles2Coords 64 chains of 150
// residues 132 -> 49 us, 293 -> 70 us, where a warp's own FP64 instructions are what is
// waited for.  Errors against 64-bit plain torch are no larger than before (6.4e-15 and
// 4.2e-15 relative).
#include <cooperative_groups.h>

#include <algorithm>

#include "tpl_a2c.cuh"
#include "tpl_common.cuh"
#include "tpl_internal.h"
#include "tpl_topology.cuh"

namespace cg = cooperative_groups;

namespace tpl {
namespace {

using FrameD = Frame<double>;

__device__ __noinline__ double2 sincos_any(double a) {
    double2 v;
    sincos(a, &v.x, &v.y);
    return v;
}

// sin and cos without the library's branches: Cody-Waite reduction by pi/2 (rounded by
// adding 1.5 * 2^52, whose sum's low bits are the quadrant; pi/2 as three doubles, the
// rounding of the reduced argument kept as rl), then the Taylor series of sin to r^17 and
// of cos to r^16 (truncation below 1e-17 on |r| <= pi/4), with rl taken into what is added
// last to r and to 1.  Against 113-bit sines (five million arguments, those next to
// multiples of pi/2 among them) within 0.97 ulp of the result for |a| <= 1e4, 9.4e-17
// absolute.  (Two terms of pi/2, and rl added to r and to 1 before the series: one
// instruction less, 1.47 ulp and 1.3e-16, but 296 ulp next to multiples of pi/2.)  Larger
// arguments, infinities and NaN go to sincos.
__device__ __forceinline__ void sincos_f64(double a, double *s, double *c) {
    if (!(fabs(a) <= 1.0e4)) {
        const double2 v = sincos_any(a);
        *s = v.x;
        *c = v.y;
        return;
    }
    constexpr double kShift = 6755399441055744.0;
    constexpr double kHi = 1.5707963267948966, kMid = 6.123233995736766e-17, kLo = -1.4973849048591833e-33;
    const double t = fma(a, 0.63661977236758134, kShift), k = t - kShift;
    // rh is exact; below 2^-40 (by the exponent bits) rh - r no longer is, and r's rounding
    // is half an ulp of the result
    const double rh = fma(-k, kHi, a), r = fma(-k, kMid, rh);
    const bool tiny = (unsigned)(__double2hiint(r) & 0x7fffffff) < 0x3d700000u;
    const double rl = fma(-k, kLo, tiny ? 0.0 : fma(-k, kMid, rh - r));
    const double r2 = r * r;
    double ps = fma(r2, 1.0 / 355687428096000.0, -1.0 / 1307674368000.0);
    ps = fma(ps, r2, 1.0 / 6227020800.0);
    ps = fma(ps, r2, -1.0 / 39916800.0);
    ps = fma(ps, r2, 1.0 / 362880.0);
    ps = fma(ps, r2, -1.0 / 5040.0);
    ps = fma(ps, r2, 1.0 / 120.0);
    ps = fma(ps, r2, -1.0 / 6.0);
    double pc = fma(r2, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);
    pc = fma(pc, r2, 1.0 / 479001600.0);
    pc = fma(pc, r2, -1.0 / 3628800.0);
    pc = fma(pc, r2, 1.0 / 40320.0);
    pc = fma(pc, r2, -1.0 / 720.0);
    pc = fma(pc, r2, 1.0 / 24.0);
    pc = fma(pc, r2, -0.5);
    const double cr = fma(fma(pc, r, -rl), r, 1.0), sr = r + fma(ps * r2, r, rl * cr);
    const unsigned q = (unsigned)__double2loint(t);
    const double ss = (q & 1u) ? cr : sr, cc = (q & 1u) ? sr : cr;
    *s = __hiloint2double(__double2hiint(ss) ^ (int)((q << 30) & 0x80000000u), __double2loint(ss));
    *c = __hiloint2double(__double2hiint(cc) ^ (int)(((q + 1u) << 30) & 0x80000000u), __double2loint(cc));
}

// Inclusive prefix of the lane transforms.  At level off the lanes with that bit compose the
// prefix of the block before them onto their own; the lanes without it have nothing to do,
// so each works for the lane off above it: a composition's four columns (three of the
// rotation, and the translation) are two each, 18 FP64 instructions a level for the warp
// where a lane on its own would take 36.
__device__ __forceinline__ FrameD scan_inclusive(FrameD t, int lane) {
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const bool owner = (lane & off) != 0;
        const int src = (lane & ~(2 * off - 1)) | (off - 1);  // last lane of the block before
        double a[9], ap[3], x[6];                             // the prefix; this lane's two columns of t
#pragma unroll
        for (int i = 0; i < 9; i++) a[i] = __shfl_sync(0xffffffffu, t.r[i], src);
#pragma unroll
        for (int i = 0; i < 3; i++) ap[i] = __shfl_sync(0xffffffffu, t.p[i], src);
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const double c2 = __shfl_xor_sync(0xffffffffu, t.r[3 * i + 2], off);
            const double cp = __shfl_xor_sync(0xffffffffu, t.p[i], off);
            x[i] = owner ? t.r[3 * i] : c2;
            x[3 + i] = owner ? t.r[3 * i + 1] : cp;
        }
        double y[6];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            y[i] = fma(a[3 * i], x[0], fma(a[3 * i + 1], x[1], a[3 * i + 2] * x[2]));
            y[3 + i] = fma(a[3 * i], x[3], fma(a[3 * i + 1], x[4], fma(a[3 * i + 2], x[5], owner ? 0.0 : ap[i])));
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const double c2 = __shfl_xor_sync(0xffffffffu, y[i], off);
            const double cp = __shfl_xor_sync(0xffffffffu, y[3 + i], off);
            if (owner) {
                t.r[3 * i] = y[i];
                t.r[3 * i + 1] = y[3 + i];
                t.r[3 * i + 2] = c2;
                t.p[i] = cp;
            }
        }
    }
    return t;
}

// Exclusive prefix of the lane transforms; lane 31's inclusive one is left in t.
__device__ __forceinline__ FrameD scan_exclusive(FrameD &t, int lane) {
    t = scan_inclusive(t, lane);
    FrameD e = shfl_up_frame(t, 1);
    if (lane == 0) frame_identity(e);
    return e;
}

// apply_joint on the identity, without the products by its zeros and ones.
__device__ __forceinline__ void first_joint(FrameD &f, double cb, double sb, double d, double ca, double sa) {
    f.r[0] = cb;
    f.r[1] = sb * sa;
    f.r[2] = sb * ca;
    f.r[3] = 0.0;
    f.r[4] = ca;
    f.r[5] = -sa;
    f.r[6] = -sb;
    f.r[7] = cb * sa;
    f.r[8] = cb * ca;
    f.p[0] = d * cb;
    f.p[1] = 0.0;
    f.p[2] = -(d * sb);
}

// What the chunks of a pass tell one another: the chunk's transform, its atoms, and its
// sums (G, S) of the adjoint.  One slot per warp of the CTA.
template <int NW>
struct ChunkSlots {
    FrameD frame[NW];
    int atoms[NW];
    double sums[NW][6];
};

// The CTAs of a chain as one group of CS * NW warps.  Each quarter of an SM has its own
// FP64 pipe, and a chain shorter than the pass leaves the last chunks without work, so
// the chunks go round the CTAs (chunk c on rank c % CS) and the warp that takes a CTA's
// first chunk differs from CTA to CTA.
template <int NW>
struct Chain {
    cg::cluster_group cluster;
    ChunkSlots<NW> *slots;
    int rank, cs, w, lane, c, nc;
    __device__ __forceinline__ Chain(ChunkSlots<NW> *s) : cluster(cg::this_cluster()), slots(s) {
        rank = (int)cluster.block_rank();
        cs = (int)cluster.num_blocks();
        w = ((threadIdx.x >> 5) + blockIdx.x) % NW;  // slot in the CTA
        lane = threadIdx.x & 31;
        c = w * cs + rank;
        nc = cs * NW;
    }
    __device__ __forceinline__ int chain() const { return (int)blockIdx.x / cs; }
    // every thread of the cluster: what was written to the slots before is visible after
    __device__ __forceinline__ void sync() {
        if (cs > 1) cluster.sync();
        else __syncthreads();
    }
    __device__ __forceinline__ const ChunkSlots<NW> *of(int chunk) const {
        return cs > 1 ? cluster.map_shared_rank(slots, chunk % cs) : slots;
    }
    // Publish the chunk's total (lane 31's t) and atoms; every thread of the cluster calls it.
    __device__ __forceinline__ void publish(const FrameD &t, int atoms) {
        if (lane == 31) {
            slots->frame[w] = t;
            slots->atoms[w] = atoms;
        }
        sync();
    }
    // F o (transforms of chunks 0 .. count - 1), and their atoms added to n.  Lanes 0..8 hold
    // one rotation entry each (row-major), 9..11 the translation: a composition is three
    // FP64 instructions for all of them.
    __device__ __forceinline__ FrameD prefix(const FrameD &F, int count, int &n) const {
        const int e = lane < 12 ? lane : 0, row = e < 9 ? e / 3 : e - 9, col = e < 9 ? e % 3 : 3;
        double acc = F.r[0];
#pragma unroll
        for (int i = 1; i < 12; i++)
            if (e == i) acc = i < 9 ? F.r[i] : F.p[i - 9];
        for (int q = 0; q < count; q++) {
            const ChunkSlots<NW> *s = of(q);
            const FrameD &t = s->frame[q / cs];
            double m[3];
#pragma unroll
            for (int k = 0; k < 3; k++) m[k] = col < 3 ? t.r[3 * k + col] : t.p[k];
            const double a0 = __shfl_sync(0xffffffffu, acc, 3 * row), a1 = __shfl_sync(0xffffffffu, acc, 3 * row + 1),
                         a2 = __shfl_sync(0xffffffffu, acc, 3 * row + 2);
            acc = fma(a0, m[0], fma(a1, m[1], fma(a2, m[2], col < 3 ? 0.0 : acc)));
            n += s->atoms[q / cs];
        }
        FrameD o;
#pragma unroll
        for (int i = 0; i < 9; i++) o.r[i] = __shfl_sync(0xffffffffu, acc, i);
#pragma unroll
        for (int i = 0; i < 3; i++) o.p[i] = __shfl_sync(0xffffffffu, acc, 9 + i);
        return o;
    }
    // Publish the chunk's sums (v: the same on every lane); every thread of the cluster calls
    // it.
    __device__ __forceinline__ void publish_sums(const double (&v)[6]) {
        if (lane == 0)
#pragma unroll
            for (int i = 0; i < 6; i++) slots->sums[w][i] = v[i];
        sync();
    }
    // Lane i < 6: component i of the sums over the chunks after this one, and of all of them.
    // last: the pass's last chunk that holds residues.
    __device__ __forceinline__ void sums_after(int last, double &after, double &all) const {
        after = all = 0.0;
#pragma unroll 4
        for (int q = last; q >= 0; q--) {
            all += lane < 6 ? of(q)->sums[q / cs][lane] : 0.0;
            if (q == c + 1) after = all;
        }
    }
};

// Sums of six values over the lanes above this one, and over the warp, with the halves of
// the lanes working for one another as in scan_inclusive: at level off a lane without that
// bit adds the sum of the block after it, three values itself and three on the lane off
// above it.
__device__ __forceinline__ void suffix_excl(const double (&v)[6], int lane, double (&suf)[6], double (&total)[6]) {
    double t[6];
#pragma unroll
    for (int i = 0; i < 6; i++) t[i] = v[i];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const bool owner = (lane & off) == 0;
        const int src = (lane & ~(2 * off - 1)) | off;  // first lane of the block after
#pragma unroll
        for (int i = 0; i < 3; i++) {
            const double b0 = __shfl_sync(0xffffffffu, t[i], src), b1 = __shfl_sync(0xffffffffu, t[3 + i], src);
            const double x = __shfl_xor_sync(0xffffffffu, t[3 + i], off);
            const double y = (owner ? t[i] : x) + (owner ? b0 : b1);
            const double z = __shfl_xor_sync(0xffffffffu, y, off);
            if (owner) {
                t[i] = y;
                t[3 + i] = z;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 6; i++) {
        total[i] = __shfl_sync(0xffffffffu, t[i], 0);
        const double e = __shfl_down_sync(0xffffffffu, t[i], 1);
        suf[i] = lane == 31 ? 0.0 : e;
    }
}

// R v of a frame's rotation.
__device__ __forceinline__ void rot(const FrameD &f, const double *v, double *o) {
#pragma unroll
    for (int i = 0; i < 3; i++) o[i] = fma(f.r[3 * i], v[0], fma(f.r[3 * i + 1], v[1], f.r[3 * i + 2] * v[2]));
}

// dL/dalpha of a joint: u . (S - o x G) over its subtree.
__device__ __forceinline__ double joint_gradient(const double *u, const double *o, const double *G, const double *S) {
    double x[3];
    cross3(o, G, x);
    return fma(u[0], S[0] - x[0], fma(u[1], S[1] - x[1], u[2] * (S[2] - x[2])));
}

// S' = S + d x G: the torque about an origin that lies d before the old one.
__device__ __forceinline__ void move_origin(const double *d, const double *G, double *S) {
    double x[3];
    cross3(d, G, x);
#pragma unroll
    for (int i = 0; i < 3; i++) S[i] += x[i];
}

__device__ __forceinline__ void add_moment(const double *x, const double *g, double *G, double *S) {
    double m[3];
    cross3(x, g, m);
#pragma unroll
    for (int i = 0; i < 3; i++) {
        G[i] += g[i];
        S[i] += m[i];
    }
}

__device__ __forceinline__ void load3(const double *p, double *v) {
#pragma unroll
    for (int i = 0; i < 3; i++) v[i] = __ldg(p + i);
}

// ------------------------------------------------------------ Angles2Backbone
struct BackboneArgs {
    const double *angles;
    const int *lengths;
    double *coords;
    double *grad_angles;
    const double *grad_coords;
    WsHeader *hdr;
    TileRecord *rec;  // backward: nrec records per chain, one per pass but the first is used
    int L, nrec;
    BondConsts bc;
    double inv_d[3];  // 1 / bond length
};

__device__ __forceinline__ int backbone_length(const BackboneArgs &a, int b) {
    const int len = a.lengths[b];
    if (len >= 0 && len <= a.L) return len;
    if (threadIdx.x == 0 && a.hdr) atomicCAS(&a.hdr->status, 0u, (unsigned)TPL_ERR_LENGTH);
    return max(0, min(len, a.L));
}

// The lane's R residues from j0, walked from identity: N, CA, C positions (when POS) and
// the lane transform.  Residues past the chain, and omega of its last one, move nothing.
template <int R, bool POS>
__device__ __forceinline__ FrameD walk(const BackboneArgs &a, const double *ang, int j0, int len, double (*pos)[9]) {
    FrameD f;
    frame_identity(f);
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int j = j0 + r;
        if (j >= len) break;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            if (POS)
#pragma unroll
                for (int i = 0; i < 3; i++) pos[r][3 * k + i] = f.p[i];
            if (k == 2 && j == len - 1) break;
            double s, c;
            sincos_f64(ang[(size_t)k * a.L + j], &s, &c);
            if (r == 0 && k == 0) first_joint(f, a.bc.cbd[k], a.bc.sbd[k], a.bc.dd[k], c, s);
            else apply_joint(f, a.bc.cbd[k], a.bc.sbd[k], a.bc.dd[k], c, s);
        }
    }
    return f;
}

template <int R, int NW>
__global__ void __launch_bounds__(32 * NW, 4) a2b_fwd_f64_kernel(BackboneArgs a) {
    __shared__ ChunkSlots<NW> s_slots;
    Chain<NW> ch(&s_slots);
    const int b = ch.chain(), len = backbone_length(a, b), cap = ch.nc * 32 * R;
    const double *ang = a.angles + (size_t)b * 3 * a.L;
    double *out = a.coords + (size_t)b * 9 * a.L;
    FrameD F;  // chain frame at the pass start
    frame_identity(F);
    int n = 0;
    for (int p0 = 0; p0 < a.L; p0 += cap) {
        const int c0 = p0 + 32 * ch.c * R, j0 = c0 + ch.lane * R;
        if (p0 < len) {  // the same for every thread of the cluster
            double pos[R][9];
            FrameD t, E;
            if (c0 < len) {  // the same for every lane of the warp
                t = walk<R, true>(a, ang, j0, len, pos);
                E = scan_exclusive(t, ch.lane);
            }
            ch.publish(t, 0);
            if (c0 < len) {
                const FrameD P = compose(ch.prefix(F, ch.c, n), E);
#pragma unroll
                for (int r = 0; r < R; r++)
                    if (j0 + r < len)
#pragma unroll
                        for (int k = 0; k < 3; k++) {
                            double *o = out + (size_t)9 * (j0 + r) + 3 * k;
                            if (r == 0 && k == 0) {  // the lane's origin
#pragma unroll
                                for (int i = 0; i < 3; i++) o[i] = P.p[i];
                            } else {
                                frame_point(P, pos[r][3 * k], pos[r][3 * k + 1], pos[r][3 * k + 2], o);
                            }
                        }
            }
            if (p0 + cap < len) F = ch.prefix(F, ch.nc, n);
            ch.sync();  // every CTA has read the slots: the next pass, or a CTA's exit, may follow
        }
#pragma unroll
        for (int r = 0; r < R; r++)
            if (j0 + r >= len && j0 + r < a.L)
#pragma unroll
                for (int k = 0; k < 9; k++) out[(size_t)9 * (j0 + r) + k] = 0.0;
    }
}

template <int R, int NW>
__global__ void __launch_bounds__(32 * NW, 4) a2b_bwd_f64_kernel(BackboneArgs a) {
    __shared__ ChunkSlots<NW> s_slots;
    Chain<NW> ch(&s_slots);
    const int b = ch.chain(), len = backbone_length(a, b), cap = ch.nc * 32 * R;
    const double *ang = a.angles + (size_t)b * 3 * a.L;
    const double *gin = a.grad_coords + (size_t)b * 9 * a.L;
    double *gout = a.grad_angles + (size_t)b * 3 * a.L;
    TileRecord *rec = a.rec + (size_t)b * a.nrec;
    const int npass = (len + cap - 1) / cap;
    int n = 0;
    {  // sweep 1: the chain frame at every pass but the first
        FrameD F;
        frame_identity(F);
        for (int p = 0; p + 1 < npass; p++) {
            FrameD t = walk<R, false>(a, ang, p * cap + (32 * ch.c + ch.lane) * R, len, nullptr);
            ch.publish(scan_inclusive(t, ch.lane), 0);
            F = ch.prefix(F, ch.nc, n);
            if (ch.c == 0 && ch.lane == 0) frame_store(rec[p + 1].fexc, F);
            ch.sync();
        }
    }
    // sweep 2: passes last to first; G and S of every atom of the later passes, S about the
    // start of the pass after
    double Gc[3] = {0, 0, 0}, Sc[3] = {0, 0, 0}, oc[3] = {0, 0, 0};
    for (int p = npass - 1; p >= 0; p--) {
        const int p0 = p * cap, c0 = p0 + 32 * ch.c * R, j0 = c0 + ch.lane * R;
        FrameD F;
        frame_identity(F);
        if (p > 0) frame_load(F, rec[p].fexc);
        double d[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            d[i] = oc[i] - F.p[i];
            oc[i] = F.p[i];
            F.p[i] = 0.0;
        }
        move_origin(d, Gc, Sc);
        // positions: first in the lane's frame, then turned to world orientation, still
        // relative to the lane's first N, where bonds and moments keep their digits
        double pos[R][9], nxt[3] = {0, 0, 0};
        FrameD t, E;
        if (c0 < len) {  // the same for every lane of the warp
            t = walk<R, true>(a, ang, j0, len, pos);
#pragma unroll
            for (int i = 0; i < 3; i++) nxt[i] = t.p[i];
            E = scan_exclusive(t, ch.lane);
        }
        ch.publish(t, 0);
        double v6[6] = {0, 0, 0, 0, 0, 0}, tot[6] = {0, 0, 0, 0, 0, 0}, suf[6];
        double P[3] = {0, 0, 0};  // the lane's first N from the pass start
        if (c0 < len) {
            const FrameD W = compose(ch.prefix(F, ch.c, n), E);
            double y[3];
            rot(W, nxt, y);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                nxt[i] = y[i];
                P[i] = W.p[i];
            }
#pragma unroll
            for (int r = 0; r < R; r++)
                if (j0 + r < len)
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        double g[3];
                        load3(gin + (size_t)9 * (j0 + r) + 3 * k, g);
                        if (r == 0 && k == 0) {  // the lane's origin: zero, and no moment
#pragma unroll
                            for (int i = 0; i < 3; i++) v6[i] += g[i];
                            continue;
                        }
                        rot(W, pos[r] + 3 * k, y);
#pragma unroll
                        for (int i = 0; i < 3; i++) pos[r][3 * k + i] = y[i];
                        add_moment(y, g, v6, v6 + 3);
                    }
            // about the pass start; a lane past the chain has nothing, and its P may be NaN (psi
            // of the last residue moves no atom, but the frame after it)
            if (j0 < len) move_origin(P, v6, v6 + 3);
            suffix_excl(v6, ch.lane, suf, tot);
        }
        ch.publish_sums(tot);
        double after, whole;
        ch.sums_after(min(ch.nc, (len - p0 + 32 * R - 1) / (32 * R)) - 1, after, whole);
        if (c0 < len) {
            double G[3], S[3];
#pragma unroll
            for (int i = 0; i < 3; i++) {
                G[i] = suf[i] + __shfl_sync(0xffffffffu, after, i) + Gc[i];
                S[i] = suf[3 + i] + __shfl_sync(0xffffffffu, after, 3 + i) + Sc[i];
                P[i] = -P[i];
            }
            move_origin(P, G, S);  // back about the lane's first N
#pragma unroll
            for (int r = R - 1; r >= 0; r--) {
                const int j = j0 + r;
                if (j < len) {
                    const double *xN = pos[r], *xA = pos[r] + 3, *xC = pos[r] + 6;
                    const bool end = j == len - 1;
                    const double *gj = gin + (size_t)9 * j;  // read again: kept, it would cost a CTA per SM
                    double u[3], g[3];
#pragma unroll
                    for (int i = 0; i < 3; i++) u[i] = nxt[i] - xC[i];
                    const double om = end ? 0.0 : a.inv_d[2] * joint_gradient(u, nxt, G, S);
#pragma unroll
                    for (int i = 0; i < 3; i++) u[i] = xC[i] - xA[i];
                    const double ps = end ? 0.0 : a.inv_d[1] * joint_gradient(u, xC, G, S);
                    load3(gj + 6, g);
                    add_moment(xC, g, G, S);
#pragma unroll
                    for (int i = 0; i < 3; i++) u[i] = xA[i] - xN[i];
                    const double ph = a.inv_d[0] * joint_gradient(u, xA, G, S);
                    load3(gj + 3, g);
                    add_moment(xA, g, G, S);
                    load3(gj, g);
                    add_moment(xN, g, G, S);
                    gout[j] = ph;
                    gout[(size_t)a.L + j] = ps;
                    gout[(size_t)2 * a.L + j] = om;
#pragma unroll
                    for (int i = 0; i < 3; i++) nxt[i] = xN[i];
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
            Gc[i] += __shfl_sync(0xffffffffu, whole, i);
            Sc[i] += __shfl_sync(0xffffffffu, whole, 3 + i);
        }
        ch.sync();  // every CTA has read the slots
    }
    for (int j = len + (int)threadIdx.x + 32 * NW * ch.rank; j < a.L; j += 32 * NW * ch.cs)
#pragma unroll
        for (int k = 0; k < 3; k++) gout[(size_t)k * a.L + j] = 0.0;
}

// ------------------------------------------------------------ Angles2Coords
__device__ const Topology<double> g_topo = make_topology<double>();
constexpr Topology<double> kTopo = make_topology<double>();

struct LetterTable {
    uint32_t v[256];  // type | atoms << 8; 0 for what is no residue letter
};
constexpr LetterTable make_letters() {
    LetterTable t{};
    for (int i = 0; i < kResTypes; i++)
        t.v[(unsigned char)kResLetters[i]] = (uint32_t)(i | kTopo.natoms[i] << 8);
    return t;
}
__device__ const LetterTable g_letters = make_letters();

template <int K>
__device__ __forceinline__ void backbone_joint(FrameD &f, double c, double s) {
    constexpr double cb = kTopo.bb_cb[K], sb = kTopo.bb_sb[K], d = kTopo.bb_d[K];
    apply_joint(f, cb, sb, d, c, s);
}

// A lane's residue: type word (0 past the chain), the sines of its angles, the transform
// from its N to the next, and its atoms before it in the chunk.
struct Residue {
    uint32_t info;
    double cs[8], sn[8];
};

template <int ROWS>
__device__ __forceinline__ FrameD load_residue(const A2cArgs<double> &a, int b, int j, int len, bool renorm, Residue &q) {
    FrameD t;
    frame_identity(t);
    q.info = 0u;
    if (j < len) {
        q.info = g_letters.v[a.seq[(size_t)b * a.seq_stride + j]];
        const double *ang = a.angles + (size_t)b * 8 * a.L + j;
#pragma unroll
        for (int k = 0; k < ROWS; k++) {
            // omega of the chain's last residue moves no atom
            const double v = k == 2 && j == len - 1 ? 0.0 : ang[(size_t)k * a.L];
            sincos_f64(v, &q.sn[k], &q.cs[k]);
        }
        constexpr double cb = kTopo.bb_cb[0], sb = kTopo.bb_sb[0], d = kTopo.bb_d[0];
        first_joint(t, cb, sb, d, q.cs[0], q.sn[0]);
        backbone_joint<1>(t, q.cs[1], q.sn[1]);
        backbone_joint<2>(t, q.cs[2], q.sn[2]);
    }
    if (renorm) renormalize(t);
    return t;
}

// The first atom of a side-chain group: the group's origin, but with the product by its zero
// local position, so that a NaN angle makes it NaN as it does the group's other atoms (it is
// the only one of Lys' fifth).
__device__ __forceinline__ void group_origin(const FrameD &f, double *x) {
#pragma unroll
    for (int i = 0; i < 3; i++) x[i] = fma(f.r[3 * i + 1], 0.0, f.p[i]);
}

// Atoms of the lanes before this one, and of the warp.
__device__ __forceinline__ int atoms_exclusive(int na, int lane, int &total) {
    int inc = na;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += o;
    }
    total = __shfl_sync(0xffffffffu, inc, 31);
    return inc - na;
}

template <int NW>
__global__ void __launch_bounds__(32 * NW) a2c_fwd_f64_kernel(A2cArgs<double> a, bool renorm) {
    __shared__ ChunkSlots<NW> s_slots;
    Chain<NW> ch(&s_slots);
    const int b = ch.chain(), cap = ch.nc * 32;
    const int len = ring_chain_length(a, b, g_letters.v, ch.lane, [](int, int) {});
    double *out = a.coords + (size_t)b * 3 * a.maxA;
    const bool names = a.res_names && a.atom_names;
    uint32_t *rn = names ? a.res_names + (size_t)b * a.maxA : nullptr;
    uint32_t *an = names ? a.atom_names + (size_t)b * a.maxA : nullptr;
    FrameD F;  // chain frame at the pass start
    frame_identity(F);
    int total = 0;  // atoms before the pass
    for (int p0 = 0; p0 < len; p0 += cap) {
        const int c0 = p0 + 32 * ch.c, j = c0 + ch.lane;
        Residue q;
        FrameD t, E;
        int aoff = 0, chunk_atoms = 0;
        q.info = 0u;
        if (c0 < len) {  // the same for every lane of the warp
            t = load_residue<8>(a, b, j, len, renorm, q);
            aoff = atoms_exclusive((int)(q.info >> 8), ch.lane, chunk_atoms);
            E = scan_exclusive(t, ch.lane);
        }
        ch.publish(t, chunk_atoms);
        FrameD X;  // at N, relative to the pass's first N
        const double org[3] = {F.p[0], F.p[1], F.p[2]};
        int a0 = total + aoff;
        if (c0 < len) {
            FrameD Fr = F;
            Fr.p[0] = Fr.p[1] = Fr.p[2] = 0.0;
            X = compose(ch.prefix(Fr, ch.c, a0), E);
        }
        if (j < len) {
            const int ty = (int)(q.info & 0xffu), na = (int)(q.info >> 8);
            auto emit = [&](int slot, const double *x) {
                if (a0 + slot < a.maxA)
#pragma unroll
                    for (int i = 0; i < 3; i++) out[3 * (size_t)(a0 + slot) + i] = x[i] + org[i];
            };
            auto local = [&](const FrameD &f, double x, double y, double z, int slot) {
                double v[3];
                frame_point(f, x, y, z, v);
                emit(slot, v);
            };
            emit(0, X.p);
            backbone_joint<0>(X, q.cs[0], q.sn[0]);
            emit(1, X.p);
            if (g_topo.pro[ty])
#pragma unroll
                for (int k = 0; k < 3; k++)
                    local(X, g_topo.pro_local[k][0], g_topo.pro_local[k][1], g_topo.pro_local[k][2], 2 + k);
            FrameD S = X;
            apply_rx(S, g_topo.dummy_c, g_topo.dummy_s);
            const int nj = g_topo.njoints[ty];
#pragma unroll
            for (int k = 0; k < kMaxScJoints; k++) {
                if (k >= nj) break;
                const bool fixed = g_topo.jchi[ty][k] < 0;  // joint k turns by chi k or not at all (topology_layout_ok)
                apply_joint(S, g_topo.jcb[ty][k], g_topo.jsb[ty][k], g_topo.jd[ty][k], fixed ? 1.0 : q.cs[3 + k],
                            fixed ? 0.0 : q.sn[3 + k]);
                const int f0 = g_topo.jfirst[ty][k];
                double first[3];
                group_origin(S, first);
                emit(2 + f0, first);
                for (int m = 1; m < g_topo.jna[ty][k]; m++) {
                    const double *v = g_topo.sc[ty][f0 + m];
                    local(S, v[0], v[1], v[2], 2 + f0 + m);
                }
            }
            backbone_joint<1>(X, q.cs[1], q.sn[1]);
            emit(na - 2, X.p);
            local(X, g_topo.o_local[0], g_topo.o_local[1], g_topo.o_local[2], na - 1);
            if (names)
                for (int k = 0; k < na && a0 + k < a.maxA; k++) {
                    rn[a0 + k] = g_topo.res_name[ty];
                    an[a0 + k] = g_topo.atom_name[ty][k];
                }
        }
        const int chunks = min(ch.nc, (len - p0 + 31) / 32);
        if (p0 + cap < len) F = ch.prefix(F, chunks, total);
        else
            for (int k = 0; k < chunks; k++) total += ch.of(k)->atoms[k / ch.cs];
        ch.sync();  // every CTA has read the slots
    }
    if (total > a.maxA) {
        if (threadIdx.x == 0) a2c_error(a.hdr, TPL_ERR_ATOMS);
        total = a.maxA;
    }
    const int first = (int)threadIdx.x + 32 * NW * ch.rank, step = 32 * NW * ch.cs;
    for (int i = 3 * total + first; i < 3 * a.maxA; i += step) out[i] = 0.0;
    if (names)
        for (int i = total + first; i < a.maxA; i += step) rn[i] = an[i] = 0u;
}

// The adjoint over the rebuilt tree.  A lane takes its residue's atoms in order, once: the
// subtree of side-chain joint k is the side chain from its group on, so its gradient
// u_k . (S - o_k x G) over the whole side chain less the atoms before the group, both
// linear in (G, S), needs only u_k, u_k x o_k and one number kept from the walk.
template <int NW>
__global__ void __launch_bounds__(32 * NW) a2c_bwd_f64_kernel(A2cArgs<double> a, bool renorm, int max_pass) {
    __shared__ ChunkSlots<NW> s_slots;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    FrameD *s_frame = reinterpret_cast<FrameD *>(s_dyn);  // chain frame and first atom of every pass
    int *s_atom = reinterpret_cast<int *>(s_frame + max_pass);
    Chain<NW> ch(&s_slots);
    const int b = ch.chain(), cap = ch.nc * 32;
    const int len = ring_chain_length(a, b, g_letters.v, ch.lane, [](int, int) {});
    const double *gin = a.grad_coords + (size_t)b * 3 * a.maxA;
    double *gout = a.grad_angles + (size_t)b * 8 * a.L;
    const int npass = (len + cap - 1) / cap;
    if (threadIdx.x == 0) {
        frame_identity(s_frame[0]);
        s_atom[0] = 0;
    }
    {  // sweep 1: chain frame and first atom of every pass
        FrameD F;
        frame_identity(F);
        int total = 0;
        for (int p = 0; p + 1 < npass; p++) {
            Residue q;
            FrameD t = load_residue<3>(a, b, p * cap + 32 * ch.c + ch.lane, len, renorm, q);
            int chunk_atoms;
            atoms_exclusive((int)(q.info >> 8), ch.lane, chunk_atoms);
            ch.publish(scan_inclusive(t, ch.lane), chunk_atoms);
            F = ch.prefix(F, ch.nc, total);
            if (threadIdx.x == 0) {
                s_frame[p + 1] = F;
                s_atom[p + 1] = total;
            }
            ch.sync();
        }
    }
    __syncthreads();
    // sweep 2: passes last to first; sums over the later passes, S about the start of the
    // pass after
    double Gc[3] = {0, 0, 0}, Sc[3] = {0, 0, 0}, oc[3] = {0, 0, 0};
    for (int p = npass - 1; p >= 0; p--) {
        const int p0 = p * cap, c0 = p0 + 32 * ch.c, j = c0 + ch.lane;
        FrameD F = s_frame[p];
        double d[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            d[i] = oc[i] - F.p[i];
            oc[i] = F.p[i];
            F.p[i] = 0.0;
        }
        move_origin(d, Gc, Sc);
        Residue q;
        FrameD t, X;
        q.info = 0u;
        int aoff = 0, chunk_atoms = 0;
        if (c0 < len) {  // the same for every lane of the warp
            t = load_residue<8>(a, b, j, len, renorm, q);
            aoff = atoms_exclusive((int)(q.info >> 8), ch.lane, chunk_atoms);
            X = scan_exclusive(t, ch.lane);
        }
        const int na = (int)(q.info >> 8), ty = (int)(q.info & 0xffu);
        ch.publish(t, chunk_atoms);
        int a0 = s_atom[p] + aoff;
        // the residue's frame at N, taken as the origin: moments and axes keep their digits
        double P[3] = {0, 0, 0};  // N from the pass start
        if (c0 < len) {
            X = compose(ch.prefix(F, ch.c, a0), X);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                P[i] = X.p[i];
                X.p[i] = 0.0;
            }
        }
        double v6[6] = {0, 0, 0, 0, 0, 0};  // the residue's own sums
        double Gco[3] = {0, 0, 0}, Sco[3] = {0, 0, 0}, Gsc[3] = {0, 0, 0}, Ssc[3] = {0, 0, 0};
        double u[3][3], o[3][3], chi[5] = {0, 0, 0, 0, 0};  // axes and origins of phi, psi, omega
        if (j < len) {
            auto take = [&](int slot, const double *x, double *G, double *S) {
                double g[3] = {0, 0, 0};
                if (a0 + slot < a.maxA)
#pragma unroll
                    for (int i = 0; i < 3; i++) g[i] = gin[3 * (size_t)(a0 + slot) + i];
                add_moment(x, g, G, S);
            };
            auto joint = [&](const FrameD &f, int k) {
#pragma unroll
                for (int i = 0; i < 3; i++) {
                    u[k][i] = f.r[3 * i];
                    o[k][i] = f.p[i];
                }
            };
            take(0, X.p, v6, v6 + 3);
            backbone_joint<0>(X, q.cs[0], q.sn[0]);
            joint(X, 0);
            take(1, X.p, v6, v6 + 3);
            if (g_topo.pro[ty])
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    double v[3];
                    frame_point(X, g_topo.pro_local[k][0], g_topo.pro_local[k][1], g_topo.pro_local[k][2], v);
                    take(2 + k, v, Gsc, Ssc);
                }
            FrameD S = X;
            apply_rx(S, g_topo.dummy_c, g_topo.dummy_s);
            const int nj = g_topo.njoints[ty];
            double ju[5][3], jm[5][3];
            int turning = 0;  // joints that a chi angle turns: the first ones, or none
#pragma unroll
            for (int k = 0; k < kMaxScJoints; k++) {
#pragma unroll
                for (int i = 0; i < 3; i++) ju[k][i] = jm[k][i] = 0.0;
                if (k >= nj) continue;
                const bool fixed = g_topo.jchi[ty][k] < 0;
                if (!fixed) turning = k + 1;
                apply_joint(S, g_topo.jcb[ty][k], g_topo.jsb[ty][k], g_topo.jd[ty][k], fixed ? 1.0 : q.cs[3 + k],
                            fixed ? 0.0 : q.sn[3 + k]);
                if (!fixed) {
#pragma unroll
                    for (int i = 0; i < 3; i++) ju[k][i] = S.r[3 * i];
                    cross3(ju[k], S.p, jm[k]);
                    chi[k] = -joint_gradient(ju[k], S.p, Gsc, Ssc);  // less the atoms before the group
                }
                const int f0 = g_topo.jfirst[ty][k];
                double first[3];
                group_origin(S, first);
                take(2 + f0, first, Gsc, Ssc);
                for (int m = 1; m < g_topo.jna[ty][k]; m++) {
                    const double *v = g_topo.sc[ty][f0 + m];
                    double x[3];
                    frame_point(S, v[0], v[1], v[2], x);
                    take(2 + f0 + m, x, Gsc, Ssc);
                }
            }
#pragma unroll
            for (int k = 0; k < kMaxScJoints; k++)  // u . (S - o x G) = u . S - (u x o) . G
                if (k < turning)                    // an angle without a joint gets 0, whatever the sums
#pragma unroll
                    for (int i = 0; i < 3; i++) chi[k] += fma(ju[k][i], Ssc[i], -jm[k][i] * Gsc[i]);
            backbone_joint<1>(X, q.cs[1], q.sn[1]);
            joint(X, 1);
            take(na - 2, X.p, Gco, Sco);
            double v[3];
            frame_point(X, g_topo.o_local[0], g_topo.o_local[1], g_topo.o_local[2], v);
            take(na - 1, v, Gco, Sco);
            backbone_joint<2>(X, q.cs[2], q.sn[2]);
            joint(X, 2);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                v6[i] += Gsc[i] + Gco[i];
                v6[3 + i] += Ssc[i] + Sco[i];
            }
        }
        double suf[6] = {0, 0, 0, 0, 0, 0}, tot[6] = {0, 0, 0, 0, 0, 0}, after, whole;
        if (c0 < len) {
            if (j < len) move_origin(P, v6, v6 + 3);  // about the pass start
            suffix_excl(v6, ch.lane, suf, tot);
        }
        ch.publish_sums(tot);
        ch.sums_after(min(ch.nc, (len - p0 + 31) / 32) - 1, after, whole);
        double G[3], S[3];
#pragma unroll
        for (int i = 0; i < 3; i++) {
            G[i] = suf[i] + __shfl_sync(0xffffffffu, after, i) + Gc[i];
            S[i] = suf[3 + i] + __shfl_sync(0xffffffffu, after, 3 + i) + Sc[i];
            P[i] = -P[i];
        }
        if (j < len) move_origin(P, G, S);  // back about this residue's N
        if (j < len) {
            const double om = j == len - 1 ? 0.0 : joint_gradient(u[2], o[2], G, S);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                G[i] += Gco[i];
                S[i] += Sco[i];
            }
            const double ps = joint_gradient(u[1], o[1], G, S);
#pragma unroll
            for (int i = 0; i < 3; i++) {
                G[i] += Gsc[i];
                S[i] += Ssc[i];
            }
            const double ph = joint_gradient(u[0], o[0], G, S);  // CA sits on the axis
            double *o8 = gout + j;
            o8[0] = ph;
            o8[(size_t)a.L] = ps;
            o8[(size_t)2 * a.L] = om;
#pragma unroll
            for (int k = 0; k < 5; k++) o8[(size_t)(3 + k) * a.L] = chi[k];
        }
#pragma unroll
        for (int i = 0; i < 3; i++) {
            Gc[i] += __shfl_sync(0xffffffffu, whole, i);
            Sc[i] += __shfl_sync(0xffffffffu, whole, 3 + i);
        }
        ch.sync();  // every CTA has read the slots
    }
    for (int i = len + (int)threadIdx.x + 32 * NW * ch.rank; i < a.L; i += 32 * NW * ch.cs)
#pragma unroll
        for (int k = 0; k < 8; k++) gout[(size_t)k * a.L + i] = 0.0;
}

// sincos_f64 as the kernels above evaluate it, for the tests.
__global__ void sincos_f64_kernel(const double *a, double *s, double *c, int n) {
    const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
    if (i < n) sincos_f64(a[i], s + i, c + i);
}

// ------------------------------------------------------------------ host side
constexpr int kMaxCluster = 8;  // the portable cluster size

// CTAs per chain: enough for the longest chain's chunks in one pass, at most kMaxCluster.
int cluster_size(int L, int residues_per_cta) {
    int cs = 1;
    while (cs < kMaxCluster && cs * residues_per_cta < L) cs *= 2;
    return cs;
}

template <typename... Params, typename... Args>
int launch_cluster(void (*kernel)(Params...), int B, int cs, int threads, size_t smem, cudaStream_t st, Args... args) {
    if ((long long)B * cs > 0x7fffffffll) return TPL_ERR_UNSUPPORTED;
    if (smem > 0 && !set_max_dynamic_smem(reinterpret_cast<const void *>(kernel), (int)smem)) return TPL_ERR_LAUNCH;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)cs;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(B * cs));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

constexpr int kBackboneWarps = 4, kAtomWarps = 2;

// Residues per lane of the backbone kernels: two share a scan; one where the batch leaves
// FP64 pipes idle and the walk's length is what is waited for (forward + backward, one
// against two: 32 x 64 residues 34 / 52 us, 64 x 128 38 / 53, 64 x 300 54 / 57, 128 x 200
// 57 / 57, 256 x 350 149 / 143, 1024 x 1000 1254 / 981).
bool one_per_lane(int B, int L) {
    return (long long)B * L <= 128ll * device_sm_count() && L <= kMaxCluster * 32 * kBackboneWarps;
}

}  // namespace

int a2b_forward_f64_plain(const double *angles, const int32_t *lengths, double *coords, int B, int L,
                          cudaStream_t st) {
    if (B == 0 || L == 0) return TPL_OK;
    BackboneArgs a{};
    a.angles = angles;
    a.lengths = lengths;
    a.coords = coords;
    a.L = L;
    a.bc = bond_constants();
    constexpr int NW = kBackboneWarps;
    if (one_per_lane(B, L))
        return launch_cluster(a2b_fwd_f64_kernel<1, NW>, B, cluster_size(L, 32 * NW), 32 * NW, 0, st, a);
    return launch_cluster(a2b_fwd_f64_kernel<2, NW>, B, cluster_size(L, 64 * NW), 32 * NW, 0, st, a);
}

int a2b_backward_f64_plain(double *grad_angles, const double *grad_coords, const double *angles,
                           const int32_t *lengths, void *ws, int B, int L, cudaStream_t st) {
    if (B == 0 || L == 0) return TPL_OK;
    BackboneArgs a{};
    a.angles = angles;
    a.lengths = lengths;
    a.grad_angles = grad_angles;
    a.grad_coords = grad_coords;
    a.hdr = reinterpret_cast<WsHeader *>(ws);
    a.rec = reinterpret_cast<TileRecord *>(reinterpret_cast<char *>(ws) + sizeof(WsHeader));
    a.L = L;
    a.nrec = (L + 255) / 256;  // the workspace holds a record per 256 residues; a pass holds more
    a.bc = bond_constants();
    for (int k = 0; k < 3; k++) a.inv_d[k] = 1.0 / a.bc.dd[k];
    constexpr int NW = kBackboneWarps;
    if (one_per_lane(B, L))
        return launch_cluster(a2b_bwd_f64_kernel<1, NW>, B, cluster_size(L, 32 * NW), 32 * NW, 0, st, a);
    return launch_cluster(a2b_bwd_f64_kernel<2, NW>, B, cluster_size(L, 64 * NW), 32 * NW, 0, st, a);
}

int sincos_poly_f64(const double *a, double *s, double *c, int n, cudaStream_t st) {
    if (n <= 0) return TPL_OK;
    sincos_f64_kernel<<<(unsigned)((n + 255ll) / 256), 256, 0, st>>>(a, s, c, n);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

int a2c_forward_f64(const A2cArgs<double> &a, int B, bool renorm, cudaStream_t st) {
    constexpr int NW = kAtomWarps;
    return launch_cluster(a2c_fwd_f64_kernel<NW>, B, cluster_size(a.L, 32 * NW), 32 * NW, 0, st, a, renorm);
}

int a2c_backward_f64(const A2cArgs<double> &a, int B, bool renorm, cudaStream_t st) {
    constexpr int NW = kAtomWarps;
    const int cs = cluster_size(a.L, 32 * NW), max_pass = std::max(1, (a.L + cs * 32 * NW - 1) / (cs * 32 * NW));
    const size_t smem = (sizeof(FrameD) + sizeof(int)) * (size_t)max_pass;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (smem + sizeof(ChunkSlots<NW>) > (size_t)optin) return TPL_ERR_UNSUPPORTED;
    return launch_cluster(a2c_bwd_f64_kernel<NW>, B, cs, 32 * NW, smem, st, a, renorm, max_pass);
}

}  // namespace tpl
