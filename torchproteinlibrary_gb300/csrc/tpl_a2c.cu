// Angles2Coords kernels for sm_103a (the reference has no GPU path here: it
// builds one heap-allocated node graph per chain on the CPU,
// Layers/FullAtomModel/cConformation.cpp:30-211, OpenMP over chains in
// Angles2Coords/angles2coords_interface.cpp:27,92).
//
// float32 runs the chunked kernels further down by default (a2c_fwd_ring_kernel,
// a2c_bwd_coords_ring_kernel: four or eight warps per chain on chunks of 32
// residues, the carry handed between warps).  The CTA kernels described here serve
// the tree-rebuilding backward and the threads_per_cta options 128, 256 and 512;
// float64 is in tpl_f64.cu.
//
// One CTA per chain, looping over tiles of R*NT residues with the carry (frame
// and atom offset) kept in shared memory.  Inside a tile the backbone is the
// same parallel scan as Angles2Backbone (per-thread joint products, warp
// shuffles, shared-memory warp totals); the atom offsets of the residues are an
// integer scan of per-residue atom counts carried alongside.  Each thread then
// walks its residues from its world frame and places every atom of each residue
// (backbone, Pro ring, side-chain joints below the dummy transform, carbonyl),
// stages them in shared memory and the tile's contiguous atom range is written
// with coalesced stores.
//
// The backward is the adjoint of the same tree: for a joint with axis u and
// origin o, dL/dalpha = u . sum over its subtree of (x - o) x g.  Subtrees of the
// backbone joints are "everything after" in atom order (plus the residue's own
// side chain for phi), so the kernel scans (G, S) = (sum g, sum x x g) backwards
// over tiles, threads and residues; side-chain joints use prefix sums over the
// side-chain path of their residue.  Complexity O(atoms) per chain instead of
// the reference's O(nodes x subtree).
#include <cstddef>
#include <cstdio>

#include "tpl_a2c.cuh"
#include "tpl_async.cuh"
#include "tpl_common.cuh"
#include "tpl_internal.h"
#include "tpl_pair.cuh"
#include "tpl_sincos.cuh"
#include "tpl_topology.cuh"

namespace tpl {

__device__ const Topology<float> g_topo_f32 = make_topology<float>();

// The register polynomial of the Angles2Backbone kernels (about one ulp, no special-function
// unit; sincosf beyond |a| = 1e4).
__device__ __forceinline__ void sc(float a, float *s, float *c) { sincos_poly(a, s, c); }

__device__ __forceinline__ void renorm_if(Frame<float> &f, bool on) {
    if (on) renormalize(f);
}

// Shared-memory layout of the tile buffers (dynamic).
template <int TILE>
struct A2cSmem {
    Topology<float> topo;
    float ang[8][TILE];
    float xyz[TILE * kMaxResAtoms * 3];
    signed char type[TILE];
    signed char lut[256];
};

// The forward also stages the tile's residue and atom names, so that they leave
// with the coordinates' coalesced store instead of per-residue scattered writes.
template <int TILE>
struct A2cSmemFwd {
    A2cSmem<TILE> f;
    uint32_t res_name[TILE * kMaxResAtoms];
    uint32_t atom_name[TILE * kMaxResAtoms];
};

template <int TILE>
struct A2cSmemBwd {
    A2cSmem<TILE> f;
    float g[TILE * kMaxResAtoms * 3];
};

// Copy the topology to shared memory and build the letter -> type table.
template <int NT>
__device__ __forceinline__ void load_topology(Topology<float> &dst, signed char *lut) {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(&g_topo_f32);
    uint32_t *d = reinterpret_cast<uint32_t *>(&dst);
    constexpr int n = sizeof(Topology<float>) / 4;
    static_assert(sizeof(Topology<float>) % 4 == 0, "topology size");
    for (int i = threadIdx.x; i < n; i += NT) d[i] = src[i];
    for (int i = threadIdx.x; i < 256; i += NT) lut[i] = (signed char)residue_type((unsigned char)i);
}

// Chain length = index of the first NUL of the sequence row (at most the row
// stride); every letter before it must be one of the 20 residues.
template <int NT>
__device__ __forceinline__ int chain_length(const unsigned char *row, int stride, const signed char *lut, int *s_len,
                                            int *s_bad) {
    if (threadIdx.x == 0) {
        *s_len = stride;
        *s_bad = 0;
    }
    __syncthreads();
    for (int j = threadIdx.x; j < stride; j += NT)
        if (row[j] == 0) atomicMin(s_len, j);
    __syncthreads();
    const int len = *s_len;
    for (int j = threadIdx.x; j < len; j += NT)
        if (lut[row[j]] < 0) *s_bad = 1;
    __syncthreads();
    return len;
}

// Per-thread scan state for one tile: backbone aggregate of the thread's
// residues, its exclusive prefix inside the warp, atom counts.
template <int R, int NT>
struct TileScan {
    float cs[R][3], sn[R][3];
    Frame<float> exc;     // exclusive prefix inside the warp
    int cnt_exc;      // atoms before this thread inside the warp
    int cnt_own;      // atoms of this thread
};

template <int R, int NT>
__device__ __forceinline__ void a2c_tile_scan(const Topology<float> &tp, const float (*ang)[R * NT],
                                              const signed char *type, int n, bool chain_end, bool renorm,
                                              TileScan<R, NT> &ts, Frame<float> *s_wtot, int *s_wcnt) {
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    Frame<float> agg;
    frame_identity(agg);
    int cnt = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        const int j = tid * R + r;
#pragma unroll
        for (int k = 0; k < 3; k++) {
            ts.cs[r][k] = 1.f;
            ts.sn[r][k] = 0.f;
        }
        if (j < n) {
            cnt += tp.natoms[type[j]];
#pragma unroll
            for (int k = 0; k < 3; k++) {
                if (k == 2 && chain_end && j == n - 1) break;
                sc(ang[k][j], &ts.sn[r][k], &ts.cs[r][k]);
                apply_joint(agg, tp.bb_cb[k], tp.bb_sb[k], tp.bb_d[k], ts.cs[r][k], ts.sn[r][k]);
            }
        }
    }
    renorm_if(agg, renorm);
    Frame<float> inc = warp_scan_frames(agg, lane);
    ts.exc = shfl_up_frame(inc, 1);
    if (lane == 0) frame_identity(ts.exc);
    int ci = cnt;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        int o = __shfl_up_sync(0xffffffffu, ci, off);
        if (lane >= off) ci += o;
    }
    ts.cnt_exc = ci - cnt;
    ts.cnt_own = cnt;
    if (lane == 31) {
        s_wtot[w] = inc;
        s_wcnt[w] = ci;
    }
}

// Thread 0: warp prefixes with the tile carry folded in (rotation only: positions
// are relative to the tile origin), the tile aggregate and the tile atom count.
template <int NW>
__device__ __forceinline__ void a2c_tile_prefix(const Frame<float> &carry, const Frame<float> *s_wtot, const int *s_wcnt,
                                                bool renorm, Frame<float> *s_wpre, int *s_wcpre, Frame<float> &tile_agg,
                                                int &tile_cnt) {
    Frame<float> run;
    frame_identity(run);
    Frame<float> c0 = carry;
    c0.p[0] = c0.p[1] = c0.p[2] = 0.f;
    int cr = 0;
    for (int w = 0; w < NW; w++) {
        s_wpre[w] = compose(c0, run);
        s_wcpre[w] = cr;
        run = compose(run, s_wtot[w]);
        renorm_if(run, renorm);
        cr += s_wcnt[w];
    }
    tile_agg = run;
    tile_cnt = cr;
}

// All atoms of residue j (type ty) from the frame P at its N atom.  chi_angle(q)
// returns the residue's chi_(q+1); emit(slot, xyz) receives positions in P's
// coordinates; returns the frame at the next N.
template <typename Chi, typename Emit>
__device__ __forceinline__ void residue_atoms(const Topology<float> &tp, int ty, Frame<float> &P, const float cs[3],
                                              const float sn[3], Chi chi_angle, Emit emit) {
    emit(0, P.p);
    Frame<float> F = P;
    apply_joint(F, tp.bb_cb[0], tp.bb_sb[0], tp.bb_d[0], cs[0], sn[0]);
    emit(1, F.p);
    const int na = tp.natoms[ty];
    if (tp.pro[ty]) {
        for (int a = 0; a < 3; a++) {
            float x[3];
            frame_point(F, tp.pro_local[a][0], tp.pro_local[a][1], tp.pro_local[a][2], x);
            emit(2 + a, x);
        }
    }
    const int nj = tp.njoints[ty];
    if (nj > 0) {
        Frame<float> S = F;
        apply_rx(S, tp.dummy_c, tp.dummy_s);
        for (int k = 0; k < nj; k++) {
            const int chi = tp.jchi[ty][k];
            float c = 1.f, s = 0.f;
            if (chi >= 0) sc(chi_angle(chi), &s, &c);
            apply_joint(S, tp.jcb[ty][k], tp.jsb[ty][k], tp.jd[ty][k], c, s);
            const int f0 = tp.jfirst[ty][k];
            for (int a = 0; a < tp.jna[ty][k]; a++) {
                float x[3];
                frame_point(S, tp.sc[ty][f0 + a][0], tp.sc[ty][f0 + a][1], tp.sc[ty][f0 + a][2], x);
                emit(2 + f0 + a, x);
            }
        }
    }
    Frame<float> C = F;
    apply_joint(C, tp.bb_cb[1], tp.bb_sb[1], tp.bb_d[1], cs[1], sn[1]);
    emit(na - 2, C.p);
    {
        float x[3];
        frame_point(C, tp.o_local[0], tp.o_local[1], tp.o_local[2], x);
        emit(na - 1, x);
    }
    P = C;
    apply_joint(P, tp.bb_cb[2], tp.bb_sb[2], tp.bb_d[2], cs[2], sn[2]);
}

// apply_rx and frame_point (tpl_common.cuh) on a PairFrame: the same chain of fused
// multiply-adds per output, so the same rounding.
__device__ __forceinline__ void apply_rx_pair(PairFrame &f, float ca, float sa) {
    const float2 c1 = f.c[1], c2 = f.c[2];
    f.c[1] = __ffma2_rn(c1, f2(ca), __fmul2_rn(c2, f2(sa)));
    f.c[2] = __ffma2_rn(c2, f2(ca), __fmul2_rn(c1, f2(-sa)));
    const float e1 = f.r2[1], e2 = f.r2[2];
    f.r2[1] = fmaf(e1, ca, e2 * sa);
    f.r2[2] = fmaf(e2, ca, -e1 * sa);
}

// frame_point on a PairFrame: x and y of the point, and its z.
__device__ __forceinline__ float2 pair_point(const PairFrame &P, float x, float y, float z, float &oz) {
    oz = fmaf(P.r2[0], x, fmaf(P.r2[1], y, fmaf(P.r2[2], z, P.p2)));
    return __ffma2_rn(P.c[0], f2(x), __ffma2_rn(P.c[1], f2(y), __ffma2_rn(P.c[2], f2(z), P.p)));
}

// The topology as the chunked float32 kernels read it: one 16-byte shared-memory load
// per side-chain joint and per atom position, one word per residue letter.
struct alignas(16) RingJoint {
    float cb, sb, d;
    int bits;  // atoms of the joint's group | index of its first side-chain atom << 8 | alpha fixed at 0 << 16
};
struct alignas(16) RingPoint {
    float x, y, z, pad;
};
struct RingTopology {
    RingJoint joint[kResTypes][kMaxScJoints];
    RingPoint point[kResTypes][kMaxScAtoms];
    uint32_t res_name[kResTypes];
    uint32_t atom_name[kResTypes][16];
    uint32_t letter[256];  // type | atoms << 8 | side-chain joints << 16 | Pro << 24; 0 for what is no residue letter
};
constexpr Topology<float> kTopoF32 = make_topology<float>();

constexpr RingTopology make_ring_topology() {
    const Topology<float> tp = make_topology<float>();
    RingTopology r{};
    for (int t = 0; t < kResTypes; t++) {
        for (int k = 0; k < kMaxScJoints; k++)
            r.joint[t][k] = {tp.jcb[t][k], tp.jsb[t][k], tp.jd[t][k],
                             tp.jna[t][k] | tp.jfirst[t][k] << 8 | (tp.jchi[t][k] < 0 ? 1 << 16 : 0)};
        for (int q = 0; q < kMaxScAtoms; q++) r.point[t][q] = {tp.sc[t][q][0], tp.sc[t][q][1], tp.sc[t][q][2], 0.f};
        r.res_name[t] = tp.res_name[t];
        for (int q = 0; q < kMaxResAtoms; q++) r.atom_name[t][q] = tp.atom_name[t][q];
        r.letter[(unsigned char)kResLetters[t]] =
            (uint32_t)(t | tp.natoms[t] << 8 | tp.njoints[t] << 16 | tp.pro[t] << 24);  // never 0: natoms >= 4
    }
    return r;
}
__device__ const RingTopology g_ring_topo = make_ring_topology();

template <int NT>
__device__ __forceinline__ void load_ring_topology(RingTopology &dst) {
    const uint4 *src = reinterpret_cast<const uint4 *>(&g_ring_topo);
    static_assert(sizeof(RingTopology) % 16 == 0, "topology size");
    for (int i = threadIdx.x; i < (int)(sizeof(RingTopology) / 16); i += NT) reinterpret_cast<uint4 *>(&dst)[i] = src[i];
}

// The three backbone joints' constants as literals.
template <int K>
__device__ __forceinline__ void apply_backbone(PairFrame &f, float c, float s) {
    constexpr float cb = kTopoF32.bb_cb[K], sb = kTopoF32.bb_sb[K], d = kTopoF32.bb_d[K];
    apply_joint_pair(f, cb, sb, d, c, s);
}

// residue_atoms for float32 on paired frames, with the chi angles' cos and sin
// computed beforehand (chi_c[q], chi_s[q] for chi_(q+1)): the same atoms in the
// same slots, without the frame at the next N.
template <typename Emit>
__device__ __forceinline__ void residue_atoms_pair(const RingTopology &tp, uint32_t info, const PairFrame &P,
                                                   const float cs[2], const float sn[2], const float chi_c[5],
                                                   const float chi_s[5], Emit emit) {
    const int ty = info & 0xff, na = (info >> 8) & 0xff, nj = (info >> 16) & 0xff;
    emit(0, P.p, P.p2);
    PairFrame F = P;
    apply_backbone<0>(F, cs[0], sn[0]);
    emit(1, F.p, F.p2);
    if (info >> 24) {  // Pro
        constexpr float p[9] = {kTopoF32.pro_local[0][0], kTopoF32.pro_local[0][1], kTopoF32.pro_local[0][2],
                                kTopoF32.pro_local[1][0], kTopoF32.pro_local[1][1], kTopoF32.pro_local[1][2],
                                kTopoF32.pro_local[2][0], kTopoF32.pro_local[2][1], kTopoF32.pro_local[2][2]};
#pragma unroll
        for (int a = 0; a < 3; a++) {
            float z;
            const float2 xy = pair_point(F, p[3 * a], p[3 * a + 1], p[3 * a + 2], z);
            emit(2 + a, xy, z);
        }
    }
    if (nj > 0) {
        PairFrame S = F;
        constexpr float dc = kTopoF32.dummy_c, ds = kTopoF32.dummy_s;
        apply_rx_pair(S, dc, ds);
        // unrolled over the joints: joint k reads chi angle k or none (Ala's fixed
        // alpha; topology_layout_ok), so the angle is a register, not a select
#pragma unroll
        for (int k = 0; k < kMaxScJoints; k++) {
            if (k >= nj) break;
            const RingJoint j = tp.joint[ty][k];
            const bool fixed = (j.bits >> 16) != 0;
            apply_joint_pair(S, j.cb, j.sb, j.d, k == 0 && fixed ? 1.f : chi_c[k], k == 0 && fixed ? 0.f : chi_s[k]);
            const int f0 = (j.bits >> 8) & 0xff, n = j.bits & 0xff;
            emit(2 + f0, S.p, S.p2);  // the group's first atom sits at the joint's origin
            for (int a = 1; a < n; a++) {
                const RingPoint v = tp.point[ty][f0 + a];
                float z;
                const float2 xy = pair_point(S, v.x, v.y, v.z, z);
                emit(2 + f0 + a, xy, z);
            }
        }
    }
    PairFrame C = F;
    apply_backbone<1>(C, cs[1], sn[1]);
    emit(na - 2, C.p, C.p2);
    constexpr float ox = kTopoF32.o_local[0], oy = kTopoF32.o_local[1], oz = kTopoF32.o_local[2];
    float z;
    const float2 xy = pair_point(C, ox, oy, oz, z);
    emit(na - 1, xy, z);
}

// Copy n staged values (world coordinates, xyz interleaved) to dst, coalesced.
template <int NT>
__device__ __forceinline__ void store_tile_atoms(float *dst, const float *src, int n) {
    for (int i = threadIdx.x; i < n; i += NT) dst[i] = src[i];
}

template <int R, int NT>
__global__ void __launch_bounds__(NT) a2c_fwd_kernel(A2cArgs<float> a, int renorm) {
    constexpr int TILE = R * NT, NW = NT / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    A2cSmemFwd<TILE> &smf = *reinterpret_cast<A2cSmemFwd<TILE> *>(smem_raw);
    A2cSmem<TILE> &sm = smf.f;
    __shared__ Frame<float> s_wtot[NW], s_wpre[NW];
    __shared__ int s_wcnt[NW], s_wcpre[NW];
    __shared__ Frame<float> s_carry;
    __shared__ float s_org[3];
    __shared__ int s_len, s_bad, s_abase, s_tcnt;

    const int b = blockIdx.x, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    load_topology<NT>(sm.topo, sm.lut);
    const unsigned char *row = a.seq + (size_t)b * a.seq_stride;
    int len = chain_length<NT>(row, a.seq_stride, sm.lut, &s_len, &s_bad);
    float *out = a.coords + (size_t)b * 3 * a.maxA;
    uint32_t *rn = a.res_names ? a.res_names + (size_t)b * a.maxA : nullptr;
    uint32_t *an = a.atom_names ? a.atom_names + (size_t)b * a.maxA : nullptr;
    bool ok = true;
    if (s_bad) {
        if (tid == 0) a2c_error(a.hdr, TPL_ERR_SEQUENCE);
        ok = false;
    }
    if (len > a.L) {
        if (tid == 0) a2c_error(a.hdr, TPL_ERR_LENGTH);
        ok = false;
    }
    if (tid == 0) {
        frame_identity(s_carry);
        s_abase = 0;
    }
    __syncthreads();
    const float *ang_b = a.angles + (size_t)b * 8 * a.L;
    for (int s0 = 0; ok && s0 < len; s0 += TILE) {
        const int n = min(TILE, len - s0);
        for (int k = 0; k < 8; k++)
            for (int i = tid; i < n; i += NT) sm.ang[k][i] = ang_b[(size_t)k * a.L + s0 + i];
        for (int i = tid; i < n; i += NT) sm.type[i] = sm.lut[row[s0 + i]];
        __syncthreads();
        const bool chain_end = (s0 + n == len);
        TileScan<R, NT> ts;
        a2c_tile_scan<R, NT>(sm.topo, sm.ang, sm.type, n, chain_end, renorm, ts, s_wtot, s_wcnt);
        __syncthreads();
        if (tid == 0) {
            Frame<float> agg;
            int tcnt;
            a2c_tile_prefix<NW>(s_carry, s_wtot, s_wcnt, renorm, s_wpre, s_wcpre, agg, tcnt);
            s_org[0] = s_carry.p[0]; s_org[1] = s_carry.p[1]; s_org[2] = s_carry.p[2];
            s_tcnt = tcnt;
            Frame<float> nc = compose(s_carry, agg);
            renorm_if(nc, renorm);
            s_carry = nc;
        }
        __syncthreads();
        Frame<float> P = compose(s_wpre[w], ts.exc);
        renorm_if(P, renorm);
        int aoff = s_wcpre[w] + ts.cnt_exc;  // first atom of this thread inside the tile
        const int abase = s_abase;
        // positions are built relative to the tile origin and moved to it as they are
        // staged (the same FP32 addition as at store time, without a per-value modulo)
        const float org[3] = {s_org[0], s_org[1], s_org[2]};
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int j = tid * R + r;
            if (j < n) {
                const int ty = sm.type[j];
                float *dst = sm.xyz + 3 * aoff;
                residue_atoms(sm.topo, ty, P, ts.cs[r], ts.sn[r], [&](int q) { return sm.ang[3 + q][j]; },
                                 [&](int slot, const float *x) {
                                     dst[3 * slot] = x[0] + org[0];
                                     dst[3 * slot + 1] = x[1] + org[1];
                                     dst[3 * slot + 2] = x[2] + org[2];
                                 });
                if (rn && an) {
                    const int na = sm.topo.natoms[ty];
                    for (int k = 0; k < na; k++) {
                        smf.res_name[aoff + k] = sm.topo.res_name[ty];
                        smf.atom_name[aoff + k] = sm.topo.atom_name[ty][k];
                    }
                }
                aoff += sm.topo.natoms[ty];
            }
        }
        __syncthreads();
        const int tcnt = s_tcnt;
        const int nstore = max(0, min(tcnt, a.maxA - abase));
        store_tile_atoms<NT>(out + (size_t)3 * abase, sm.xyz, 3 * nstore);
        if (rn && an)
            for (int i = tid; i < nstore; i += NT) {
                rn[abase + i] = smf.res_name[i];
                an[abase + i] = smf.atom_name[i];
            }
        __syncthreads();
        if (tid == 0) s_abase = abase + tcnt;
        __syncthreads();
    }
    int total = ok ? s_abase : 0;
    if (total > a.maxA) {
        if (tid == 0) a2c_error(a.hdr, TPL_ERR_ATOMS);
        total = a.maxA;
    }
    for (int i = 3 * total + tid; i < 3 * a.maxA; i += NT) out[i] = 0.f;
    if (rn && an)
        for (int i = total + tid; i < a.maxA; i += NT) rn[i] = an[i] = 0u;
    (void)lane;
}

// ---------------------------------------------------------- handoffs of a chain
// What a backward hands on (G, S and an origin) as three 16-byte accesses.
__device__ __forceinline__ void store_sums(float *slot, float g0, float g1, float g2, float s0, float s1, float s2,
                                           const float *o) {
    float4 *d = reinterpret_cast<float4 *>(slot);
    d[0] = make_float4(g0, g1, g2, s0);
    d[1] = make_float4(s1, s2, o[0], o[1]);
    d[2] = make_float4(o[2], 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void load_sums(const float *slot, float (&v)[9]) {
    const float4 *s = reinterpret_cast<const float4 *>(slot);
    const float4 a = s[0], b = s[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    v[8] = slot[8];
}

// ------------------------------------------ forward, four or eight warps per chain
// Chunks of 32 residues, one per lane, dealt round the NW = 4 or 8 warps of a CTA.  A
// CTA takes chains b, b + grid, ... (persistent: the topology loads once) and their
// chunks form one stream: chunk g of the stream is on warp g % NW, chain after chain,
// with no CTA barrier anywhere, so that a short chain or a chain's last chunk leaves no
// warp waiting.  Per chunk a warp composes each residue's three backbone joints
// (N -> CA -> C -> next N), scans the lane transforms and the atom counts over the warp,
// receives the chain frame and first atom index of its chunk from the warp of the chunk
// before (the named-barrier handoff of tpl_pair.cuh; at a chain's first chunk the
// handoff only keeps the order of the stream), and places every atom of its residue in a
// per-warp buffer.  Positions are built relative to the chunk's first N atom and moved
// to it as they are staged.
//
// Instruction issue and latency bound it (4096 x 500 random residues: issue active 46 %
// with the CTA-synchronised form).  What is out of the way of the arithmetic:
//   * the next chunk's angles come by cp.async while this one is worked on (a lane copies
//     and reads only its own), and its letters one chunk ahead;
//   * the coordinates leave as one bulk copy of the chunk's whole 16-byte blocks, issued
//     by one lane; the values are staged at their global 16-byte phase;
//   * names are staged as one 16-bit code per atom (type, slot) and looked up as they are
//     stored, 0.9 instead of 3.6 KB per warp, which keeps six CTAs of four warps per SM.
constexpr int kA2cChunk = 32;
constexpr int kA2cStageAtoms = kA2cChunk * kMaxResAtoms;

// Per warp: the chunk's coordinates (4 words of slack for the 16-byte phase of their
// destination), the next chunk's angles, the name codes (when names are written).
struct alignas(16) A2cRingWarp {
    float xyz[kA2cStageAtoms * 3 + 4];
    float ang[8 * kA2cChunk];
};
template <int NW, bool NAMES>
struct A2cRingSmem {
    RingTopology topo;
    A2cRingWarp warp[NW];
    uint16_t code[NAMES ? NW : 1][NAMES ? kA2cStageAtoms : 8];
};

template <int NW, bool NAMES>
__global__ void __launch_bounds__(32 * NW, NW == 4 ? 6 : 3) a2c_fwd_ring_kernel(A2cArgs<float> a, int renorm, int nb) {
    constexpr int NT = 32 * NW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    A2cRingSmem<NW, NAMES> &sm = *reinterpret_cast<A2cRingSmem<NW, NAMES> *>(smem_raw);
    __shared__ __align__(16) float s_ring[NW][16];  // chain frame (12, pair_store_vec) and first atom index

    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const RingTopology &tp = sm.topo;
    float *stage = sm.warp[w].xyz, *abuf = sm.warp[w].ang + lane;

    // the warp's next chunk: chunk k of chain b (length len, nch chunks; an empty or
    // refused chain has one, which writes its zeros)
    int b = blockIdx.x, k = w, len = 0, nch = 0;
    unsigned char letter = 0;
    auto enter = [&]() {
        len = ring_chain_length(a, b, tp.letter, lane, [](int, int) {});
        nch = max(1, (len + kA2cChunk - 1) / kA2cChunk);
    };
    auto settle = [&]() {  // chunk numbers past the chain's belong to the chains after it
        while (k >= nch) {
            k -= nch;
            b += gridDim.x;
            if (b >= nb) break;
            enter();
        }
    };
    auto fetch = [&](int end) {
        const int j = k * kA2cChunk + lane;
        if (b < nb && j < end) {
            letter = j < a.seq_stride ? a.seq[(size_t)b * a.seq_stride + j] : (unsigned char)0;
            const float *src = a.angles + (size_t)b * 8 * a.L + j;
#pragma unroll
            for (int q = 0; q < 8; q++) cp_async4(abuf + q * kA2cChunk, src + (size_t)q * a.L);
        }
    };
    // The first chunk's data are asked for before its chain's length is known (the row is
    // padded to L), together with the letters and the topology: a small batch waits for
    // memory once (32 residues 6.7 -> 6.2 us, 256 x 50..500 15.9 -> 15.4 us with names).
    {
        unsigned char c[kFirstLetters][4];
        if (b < nb) {
            load_letters(a, b, 0, lane, c);
            fetch(a.L);
        }
        load_ring_topology<NT>(sm.topo);
        __syncthreads();
        if (b < nb) {
            len = ring_chain_length(a, b, tp.letter, lane, c, [](int, int) {});
            nch = max(1, (len + kA2cChunk - 1) / kA2cChunk);
            if (k >= nch) {
                cp_async_wait_all();  // the copies into the same buffer are not ordered
                settle();
                fetch(len);
            }
        }
    }
#pragma unroll 1
    while (b < nb) {
        const int cb = b, ck = k, cnch = nch;
        const int j = ck * kA2cChunk + lane;
        const bool live = j < len, last = j + 1 >= len;
        const uint32_t info = live ? tp.letter[letter] : 0u;
        const int na = (info >> 8) & 0xff;
        float ang[8];
        cp_async_wait_all();
#pragma unroll
        for (int q = 0; q < 8; q++) ang[q] = live ? abuf[q * kA2cChunk] : 0.f;
        if (last) ang[2] = 0.f;  // omega of the chain's last residue moves no atom
        k += NW;
        settle();
        fetch(len);

        // cos and sin of the eight angles, in pairs and for every lane at once (the chi
        // angles' outside the divergent side-chain walk)
        float cs[3], sn[3], chc[5], chs[5];
        float m = 0.f;
#pragma unroll
        for (int q = 0; q < 8; q++) m = fmaxf(m, fabsf(ang[q]));
        if (m <= 1.0e4f) {  // NaN passes: sincos_fast2 returns NaN for it
            sincos_fast2(ang[0], ang[1], &sn[0], &cs[0], &sn[1], &cs[1]);
            sincos_fast2(ang[2], ang[3], &sn[2], &cs[2], &chs[0], &chc[0]);
            sincos_fast2(ang[4], ang[5], &chs[1], &chc[1], &chs[2], &chc[2]);
            sincos_fast2(ang[6], ang[7], &chs[3], &chc[3], &chs[4], &chc[4]);
        } else {
#pragma unroll
            for (int q = 0; q < 3; q++) sincos_poly(ang[q], &sn[q], &cs[q]);
#pragma unroll
            for (int q = 0; q < 5; q++) sincos_poly(ang[3 + q], &chs[q], &chc[q]);
        }
        PairFrame t = pair_identity();
        if (live) {
            apply_backbone<0>(t, cs[0], sn[0]);
            apply_backbone<1>(t, cs[1], sn[1]);
            apply_backbone<2>(t, cs[2], sn[2]);
        }
        if (renorm) renormalize_pair(t);
        t = warp_inclusive_pair(t, lane);
        int ci = na;  // atoms of the lanes up to this one
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, ci, off);
            if (lane >= off) ci += o;
        }
        const int cnt = __shfl_sync(0xffffffffu, ci, 31), aoff = ci - na;

        PairFrame F = pair_identity();  // chain frame at the chunk start
        int abase = 0;                  // first atom of the chunk
        if (cb != (int)blockIdx.x || ck > 0) ring_wait<NW>(w);
        if (ck > 0) {
            F = pair_load_vec(s_ring[w]);
            abase = __float_as_int(s_ring[w][12]);
        }
        const float2 org = F.p;  // the chunk's origin; positions are relative to it
        const float org2 = F.p2;
        F.p = make_float2(0.f, 0.f);
        F.p2 = 0.f;
        const PairFrame Q = compose_pair(F, t);
        // Lane 31's Q is the frame the next chunk starts from.  It is the frame handed on that
        // is pulled back to a rotation, at every handoff, so that a chain's rounding does not
        // add up to a scale however many chunks it has.  (Only the chunk's own transform
        // renormalised, before the wait: 61.0 -> 60.1 us a training step of 256 chains, but the
        // scale drifts: distances within a chunk 3.2e-6 off after 64 chunks of a ring
        // conformation and 2.3e-5 after 512, where they are 4e-7 off with it.)
        if (ck + 1 < cnch) {
            PairFrame Fn = Q;
            if (renorm) renormalize_pair(Fn);
            Fn.p = __fadd2_rn(Fn.p, org);
            Fn.p2 += org2;
            if (lane == 31) {
                pair_store_vec(s_ring[(w + 1) % NW], Fn);
                s_ring[(w + 1) % NW][12] = __int_as_float(abase + cnt);
            }
        }
        if (ck + 1 < cnch || cb + (int)gridDim.x < nb) ring_signal<NW>((w + 1) % NW);

        const PairFrame P = frame_before(Q, F, lane);  // at this lane's N
        float *out = a.coords + (size_t)cb * 3 * a.maxA;
        float *gdst = out + (size_t)3 * abase;
        float *stg = stage + block_offset(gdst);  // the chunk's values keep their global 16-byte phase
        if (lane == 0) bulk_reads_done();
        __syncwarp();  // the previous chunk has left the staging buffers
        if (live) {
            float *dst = stg + 3 * aoff;
            residue_atoms_pair(tp, info, P, cs, sn, chc, chs, [&](int slot, float2 xy, float z) {
                xy = __fadd2_rn(xy, org);
                dst[3 * slot] = xy.x;
                dst[3 * slot + 1] = xy.y;
                dst[3 * slot + 2] = z + org2;
            });
            if (NAMES) {
                uint16_t *code = sm.code[NAMES ? w : 0] + aoff;
                const int c0 = (int)(info & 0xff) << 4;
#pragma unroll
                for (int q = 0; q < kMaxResAtoms; q++)
                    if (q < na) code[q] = (uint16_t)(c0 + q);
            }
        }
        async_proxy_fence();
        __syncwarp();
        const int nstore = max(0, min(cnt, a.maxA - abase));
        bulk_store_span(gdst, stg, 3 * nstore, lane);
        uint32_t *rn = NAMES ? a.res_names + (size_t)cb * a.maxA : nullptr;
        uint32_t *an = NAMES ? a.atom_names + (size_t)cb * a.maxA : nullptr;
        if (NAMES) {
            const uint16_t *code = sm.code[NAMES ? w : 0];
            const uint32_t *atom_name = tp.atom_name[0];
#pragma unroll 2
            for (int i = lane; i < nstore; i += 32) {
                const int c = code[i];
                rn[abase + i] = tp.res_name[c >> 4];
                an[abase + i] = atom_name[c];
            }
        }
        if (ck + 1 == cnch) {  // the chain's last chunk also writes the zeros past its atoms
            int total = abase + cnt;
            if (total > a.maxA) {
                if (lane == 0) a2c_error(a.hdr, TPL_ERR_ATOMS);
                total = a.maxA;
            }
            zero_span(out + (size_t)3 * total, 3 * (a.maxA - total), lane);
            if (NAMES) {
                zero_span(rn + total, a.maxA - total, lane);
                zero_span(an + total, a.maxA - total, lane);
            }
        }
    }
    if (lane == 0) bulk_reads_done();  // shared memory outlives the copies' reads
}

// ------------------------------------------------------------------ backward
template <int R, int NT>
__global__ void __launch_bounds__(NT) a2c_bwd_kernel(A2cArgs<float> a, int renorm, int max_tiles) {
    constexpr int TILE = R * NT, NW = NT / 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    A2cSmemBwd<TILE> &sm = *reinterpret_cast<A2cSmemBwd<TILE> *>(smem_raw);
    Frame<float> *s_carries = reinterpret_cast<Frame<float> *>(smem_raw + sizeof(A2cSmemBwd<TILE>));
    int *s_tbase = reinterpret_cast<int *>(s_carries + max_tiles);
    __shared__ Frame<float> s_wtot[NW], s_wpre[NW];
    __shared__ int s_wcnt[NW], s_wcpre[NW];
    __shared__ float s_wsum[NW][6], s_wsuf[NW][6];
    __shared__ double s_tail[6];
    __shared__ int s_len, s_bad;

    const int b = blockIdx.x, tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    load_topology<NT>(sm.f.topo, sm.f.lut);
    const Topology<float> &tp = sm.f.topo;
    const unsigned char *row = a.seq + (size_t)b * a.seq_stride;
    int len = chain_length<NT>(row, a.seq_stride, sm.f.lut, &s_len, &s_bad);
    float *gout = a.grad_angles + (size_t)b * 8 * a.L;
    const float *gin = a.grad_coords + (size_t)b * 3 * a.maxA;
    const float *ang_b = a.angles + (size_t)b * 8 * a.L;
    bool ok = !s_bad && len <= a.L;
    if (tid == 0) {
        if (s_bad) a2c_error(a.hdr, TPL_ERR_SEQUENCE);
        if (len > a.L) a2c_error(a.hdr, TPL_ERR_LENGTH);
    }
    const int ntiles = ok ? (len + TILE - 1) / TILE : 0;
    if (ntiles > max_tiles) {
        if (tid == 0) a2c_error(a.hdr, TPL_ERR_ARGUMENT);
        ok = false;
    }
    // sweep 1: tile carries and atom bases
    if (tid == 0) {
        frame_identity(s_carries[0]);
        s_tbase[0] = 0;
    }
    __syncthreads();
    for (int t = 0; ok && t < ntiles; t++) {
        const int s0 = t * TILE, n = min(TILE, len - s0);
        for (int k = 0; k < 3; k++)
            for (int i = tid; i < n; i += NT) sm.f.ang[k][i] = ang_b[(size_t)k * a.L + s0 + i];
        for (int i = tid; i < n; i += NT) sm.f.type[i] = sm.f.lut[row[s0 + i]];
        __syncthreads();
        TileScan<R, NT> ts;
        a2c_tile_scan<R, NT>(tp, sm.f.ang, sm.f.type, n, s0 + n == len, renorm, ts, s_wtot, s_wcnt);
        __syncthreads();
        if (tid == 0) {
            Frame<float> agg;
            int tcnt;
            a2c_tile_prefix<NW>(s_carries[t], s_wtot, s_wcnt, renorm, s_wpre, s_wcpre, agg, tcnt);
            if (t + 1 < max_tiles) {
                Frame<float> nc = compose(s_carries[t], agg);
                renorm_if(nc, renorm);
                s_carries[t + 1] = nc;
                s_tbase[t + 1] = s_tbase[t] + tcnt;
            }
        }
        __syncthreads();
    }
    if (tid == 0)
        for (int i = 0; i < 6; i++) s_tail[i] = 0.0;
    __syncthreads();
    // sweep 2: tiles last-first
    for (int t = ntiles - 1; ok && t >= 0; t--) {
        const int s0 = t * TILE, n = min(TILE, len - s0);
        const int abase = s_tbase[t];
        for (int k = 0; k < 8; k++)
            for (int i = tid; i < n; i += NT) sm.f.ang[k][i] = ang_b[(size_t)k * a.L + s0 + i];
        for (int i = tid; i < n; i += NT) sm.f.type[i] = sm.f.lut[row[s0 + i]];
        __syncthreads();
        TileScan<R, NT> ts;
        a2c_tile_scan<R, NT>(tp, sm.f.ang, sm.f.type, n, s0 + n == len, renorm, ts, s_wtot, s_wcnt);
        __syncthreads();
        if (tid == 0) {
            Frame<float> agg;
            int tcnt;
            a2c_tile_prefix<NW>(s_carries[t], s_wtot, s_wcnt, renorm, s_wpre, s_wcpre, agg, tcnt);
            s_wcnt[0] = tcnt;  // reuse: tile atom count
        }
        __syncthreads();
        const int tcnt = s_wcnt[0];
        const int nload = max(0, min(tcnt, a.maxA - abase));
        for (int i = tid; i < 3 * tcnt; i += NT) sm.g[i] = i < 3 * nload ? gin[(size_t)3 * abase + i] : 0.f;
        Frame<float> P = compose(s_wpre[w], ts.exc);
        renorm_if(P, renorm);
        Frame<float> start[R];
        int roff[R];
        int aoff = s_wcpre[w] + ts.cnt_exc;
        __syncthreads();  // sm.g complete
        float G[3] = {0, 0, 0}, S[3] = {0, 0, 0};
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int j = tid * R + r;
            start[r] = P;
            roff[r] = aoff;
            if (j < n) {
                const int ty = sm.f.type[j];
                float *dst = sm.f.xyz + 3 * aoff;
                const float *gg = sm.g + 3 * aoff;
                residue_atoms(tp, ty, P, ts.cs[r], ts.sn[r], [&](int q) { return sm.f.ang[3 + q][j]; },
                                 [&](int slot, const float *x) {
                    dst[3 * slot] = x[0];
                    dst[3 * slot + 1] = x[1];
                    dst[3 * slot + 2] = x[2];
                    float xg[3];
                    cross3(x, gg + 3 * slot, xg);
                    for (int c = 0; c < 3; c++) {
                        G[c] += gg[3 * slot + c];
                        S[c] += xg[c];
                    }
                });
                aoff += tp.natoms[ty];
            }
        }
        // block-exclusive suffix over threads, plus the carry from later tiles
        float suf[6];
        const float v[6] = {G[0], G[1], G[2], S[0], S[1], S[2]};
        for (int i = 0; i < 6; i++) {
            float inc = v[i];
            for (int off = 1; off < 32; off <<= 1) {
                float o = __shfl_down_sync(0xffffffffu, inc, off);
                if (lane + off < 32) inc += o;
            }
            float tot = __shfl_sync(0xffffffffu, inc, 0);
            suf[i] = inc - v[i];
            if (lane == 0) s_wsum[w][i] = tot;
        }
        __syncthreads();
        if (tid == 0) {
            // later tiles' (G, S) are kept about the world origin in FP64; move them
            // to this tile's origin o: S_o = S_world - o x G
            const double o[3] = {(double)s_carries[t].p[0], (double)s_carries[t].p[1], (double)s_carries[t].p[2]};
            double ox[3];
            cross3(o, s_tail, ox);
            double run[6];
            for (int i = 0; i < 3; i++) {
                run[i] = s_tail[i];
                run[3 + i] = s_tail[3 + i] - ox[i];
            }
            double tot[6] = {0, 0, 0, 0, 0, 0};
            for (int ww = NW - 1; ww >= 0; ww--)
                for (int i = 0; i < 6; i++) {
                    s_wsuf[ww][i] = (float)run[i];
                    run[i] += (double)s_wsum[ww][i];
                    tot[i] += (double)s_wsum[ww][i];
                }
            double ot[3];
            cross3(o, tot, ot);
            for (int i = 0; i < 3; i++) {
                s_tail[i] += tot[i];
                s_tail[3 + i] += tot[3 + i] + ot[i];
            }
        }
        __syncthreads();
        float Gn[3], Sn[3];
        for (int c = 0; c < 3; c++) {
            Gn[c] = suf[c] + s_wsuf[w][c];
            Sn[c] = suf[3 + c] + s_wsuf[w][3 + c];
        }
        float(*s_gr)[TILE] = sm.f.ang;  // angles of this tile stay in registers (ts) / are re-read below
#pragma unroll
        for (int r = R - 1; r >= 0; r--) {
            const int j = tid * R + r;
            if (j >= n) continue;
            const int ty = sm.f.type[j];
            const int na = tp.natoms[ty], nj = tp.njoints[ty];
            const float *X = sm.f.xyz + 3 * roff[r];
            const float *Gg = sm.g + 3 * roff[r];
            // per-group sums of this residue
            auto acc = [&](int lo, int hi, float *gs, float *ss) {
                for (int c = 0; c < 3; c++) gs[c] = ss[c] = 0.f;
                for (int q = lo; q < hi; q++) {
                    float xg[3];
                    cross3(X + 3 * q, Gg + 3 * q, xg);
                    for (int c = 0; c < 3; c++) {
                        gs[c] += Gg[3 * q + c];
                        ss[c] += xg[c];
                    }
                }
            };
            float Gco[3], Sco[3], Gmid[3], Smid[3], Gn0[3], Sn0[3];
            acc(na - 2, na, Gco, Sco);
            acc(1, na - 2, Gmid, Smid);   // CA, Pro ring / side chain
            acc(0, 1, Gn0, Sn0);          // N
            // frames of the residue
            Frame<float> F = start[r];
            apply_joint(F, tp.bb_cb[0], tp.bb_sb[0], tp.bb_d[0], ts.cs[r][0], ts.sn[r][0]);
            Frame<float> C = F;
            apply_joint(C, tp.bb_cb[1], tp.bb_sb[1], tp.bb_d[1], ts.cs[r][1], ts.sn[r][1]);
            Frame<float> Nn = C;
            apply_joint(Nn, tp.bb_cb[2], tp.bb_sb[2], tp.bb_d[2], ts.cs[r][2], ts.sn[r][2]);
            float tmp[3], cr[3];
            auto gradient = [&](const Frame<float> &J, const float *Gs, const float *Ss) {
                cross3(J.p, Gs, cr);
                for (int c = 0; c < 3; c++) tmp[c] = Ss[c] - cr[c];
                return J.r[0] * tmp[0] + J.r[3] * tmp[1] + J.r[6] * tmp[2];
            };
            const bool last = (s0 + j == len - 1);
            const float g_om = last ? 0.f : gradient(Nn, Gn, Sn);
            float Gc[3], Sc[3];
            for (int c = 0; c < 3; c++) {
                Gc[c] = Gn[c] + Gco[c];
                Sc[c] = Sn[c] + Sco[c];
            }
            const float g_ps = gradient(C, Gc, Sc);
            for (int c = 0; c < 3; c++) {
                Gc[c] += Gmid[c];
                Sc[c] += Smid[c];
            }
            const float g_ph = gradient(F, Gc, Sc);
            // side-chain joints: subtree of joint k = its group and all later groups
            float g_chi[5] = {0, 0, 0, 0, 0};
            if (nj > 0) {
                float Gsc[3], Ssc[3];
                acc(2, na - 2, Gsc, Ssc);
                Frame<float> Sf = F;
                apply_rx(Sf, tp.dummy_c, tp.dummy_s);
                for (int k = 0; k < nj; k++) {
                    const int chi = tp.jchi[ty][k];
                    float c = 1.f, s = 0.f;
                    if (chi >= 0) sc(sm.f.ang[3 + chi][j], &s, &c);
                    apply_joint(Sf, tp.jcb[ty][k], tp.jsb[ty][k], tp.jd[ty][k], c, s);
                    if (chi >= 0) g_chi[chi] = gradient(Sf, Gsc, Ssc);
                    const int f0 = 2 + tp.jfirst[ty][k];
                    float Gk[3], Sk[3];
                    acc(f0, f0 + tp.jna[ty][k], Gk, Sk);
                    for (int q = 0; q < 3; q++) {
                        Gsc[q] -= Gk[q];
                        Ssc[q] -= Sk[q];
                    }
                }
            }
            // suffix for the previous residue: this residue's atoms join it
            for (int c = 0; c < 3; c++) {
                Gn[c] = Gc[c] + Gn0[c];
                Sn[c] = Sc[c] + Sn0[c];
            }
            // chi angles are read from shared memory above, so stage gradients in
            // registers until every thread has finished with the angle rows
            start[r].r[0] = g_ph; start[r].r[1] = g_ps; start[r].r[2] = g_om;
            for (int q = 0; q < 5; q++) start[r].r[3 + q] = g_chi[q];
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < R; r++) {
            const int j = tid * R + r;
            if (j < n)
                for (int q = 0; q < 8; q++) s_gr[q][j] = start[r].r[q];
        }
        __syncthreads();
        for (int k = 0; k < 8; k++)
            for (int i = tid; i < n; i += NT) gout[(size_t)k * a.L + s0 + i] = s_gr[k][i];
        __syncthreads();
    }
    // zeros past the chain (and everywhere when the chain was rejected)
    const int from = ok ? len : 0;
    for (int k = 0; k < 8; k++)
        for (int i = from + tid; i < a.L; i += NT) gout[(size_t)k * a.L + i] = 0.f;
}

// ------------------------------------------------- backward from the coordinates
// The forward's output holds the origin of every joint: N, CA and C for the
// backbone, and for each side-chain joint the first atom of its group, which sits
// at the joint's origin (every group of the table starts at its local origin).
// Each rotation axis is a bond of known length: u = (origin - parent origin) / d,
// with CA as the parent of the first side-chain joint (the dummy joint has no
// length).  So dL/dalpha = u . (S - o x G) over the joint's subtree needs only the
// coordinates and dL/dx, and this backward never rebuilds the tree.  Each lane owns
// one residue: it sums G and S over the residue's atoms, a warp suffix scan adds the
// later residues of its chunk and a carry the later chunks, and the lane visits its
// residue's atoms last to first:
//   omega_j  subtree: every later residue        axis C_j -> N_j+1, origin N_j+1
//   psi_j    + O_j                                axis CA_j -> C_j,  origin C_j
//   chi_k    side-chain groups k.. only           axis o_k-1 -> o_k, origin o_k
//   phi_j    + side chain + C_j                   axis N_j -> CA_j,  origin CA_j
// Positions are taken relative to the chunk's first N atom to keep the sums small.
// G and S with their additions in paired FP32: (G0, G1), (S0, S1), (G2, S2).  The backward is
// bound by instruction issue: the layer at 4096 x 500 283.4 -> 280.9 us, the same results.
struct PairSums {
    float2 g, s, z;
};
__device__ __forceinline__ PairSums zero_sums() {
    return {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
}
__device__ __forceinline__ PairSums operator+(const PairSums &a, const PairSums &b) {
    return {__fadd2_rn(a.g, b.g), __fadd2_rn(a.s, b.s), __fadd2_rn(a.z, b.z)};
}

__device__ __forceinline__ float joint_grad(const float *o, const float *p_prev, float inv_d, const PairSums &t) {
    const float G[3] = {t.g.x, t.g.y, t.z.x};
    float cr[3];
    cross3(o, G, cr);
    return ((o[0] - p_prev[0]) * (t.s.x - cr[0]) + (o[1] - p_prev[1]) * (t.s.y - cr[1]) +
            (o[2] - p_prev[2]) * (t.z.y - cr[2])) *
           inv_d;
}

// Sums over the lanes above this one (exclusive suffix), and the warp's.
__device__ __forceinline__ PairSums suffix_excl(const PairSums &v, int lane, PairSums &total) {
    PairSums inc = v;
    auto from = [](float2 x, int off) {
        return make_float2(__shfl_down_sync(0xffffffffu, x.x, off), __shfl_down_sync(0xffffffffu, x.y, off));
    };
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const PairSums o = {from(inc.g, off), from(inc.s, off), from(inc.z, off)};
        if (lane + off < 32) inc = inc + o;
    }
    auto first = [](float2 x) {
        return make_float2(__shfl_sync(0xffffffffu, x.x, 0), __shfl_sync(0xffffffffu, x.y, 0));
    };
    total = {first(inc.g), first(inc.s), first(inc.z)};
    auto less = [](float2 x, float2 y) { return __fadd2_rn(x, make_float2(-y.x, -y.y)); };
    return {less(inc.g, v.g), less(inc.s, v.s), less(inc.z, v.z)};
}

// The cross product on its own, then added: accumulated straight into S it would save three
// additions but chain two FMAs per atom (4096 x 500: 144 -> 157 us).
__device__ __forceinline__ void add_atom(const float *xs, const float *gs, const float *o, PairSums &t) {
    const float2 xy = __fadd2_rn(make_float2(xs[0], xs[1]), make_float2(-o[0], -o[1]));
    const float xr[3] = {xy.x, xy.y, xs[2] - o[2]}, g[3] = {gs[0], gs[1], gs[2]};
    float xg[3];
    cross3(xr, g, xg);
    t = t + PairSums{make_float2(g[0], g[1]), make_float2(xg[0], xg[1]), make_float2(g[2], xg[2])};
}

// The kernel: chunks of 32 residues, one per lane, last chunk first, dealt round NW = 4 or
// 8 warps as one stream over the CTA's chains, as in a2c_fwd_ring_kernel (chains last to
// first: the first CTAs read the rows the forward wrote last, which may still be in L2).
// A warp finds the first atom of every chunk itself as it reads a chain's sequence (4 bytes a
// chunk and warp; where that does not fit the shared memory, past 140 000 residues with eight
// warps, a CTA takes one chain and its warps share one table).  Per
// chunk it receives the atom range of coordinates and dL/dx in shared memory (one bulk
// copy each of their whole 16-byte blocks, word copies of the ragged ends), walks each
// lane's residue, suffix-scans the sums over the warp and takes the sums over later chunks
// from the warp of chunk k + 1 (G, S and that chunk's first N atom, through the
// named-barrier handoff of tpl_pair.cuh).  The buffers are free after the walk, so the
// next chunk's copies run under the scan, the handoff and the stores.
struct RingBwdJoint {
    float inv_d;
    int bits;  // atoms of the joint's group | index of its first side-chain atom << 8 | turned by a chi angle << 16
};
struct RingBwdTopology {
    RingBwdJoint joint[kResTypes][kMaxScJoints];
    uint16_t letter[256];  // type | atoms << 8; 0 for what is no residue letter
};
constexpr RingBwdTopology make_ring_bwd_topology() {
    const Topology<float> tp = make_topology<float>();
    RingBwdTopology r{};
    for (int t = 0; t < kResTypes; t++) {
        for (int k = 0; k < tp.njoints[t]; k++)
            r.joint[t][k] = {1.f / tp.jd[t][k],
                             tp.jna[t][k] | tp.jfirst[t][k] << 8 | (tp.jchi[t][k] < 0 ? 0 : 1 << 16)};
        r.letter[(unsigned char)kResLetters[t]] = (uint16_t)(t | tp.natoms[t] << 8);
    }
    return r;
}
__device__ const RingBwdTopology g_ring_bwd_topo = make_ring_bwd_topology();

template <int NW>
struct A2cBwdRingSmem {
    alignas(16) float x[NW][kA2cStageAtoms * 3 + 4];  // 4 words of slack for the 16-byte phase of the source
    alignas(16) float g[NW][kA2cStageAtoms * 3 + 4];
    RingBwdTopology topo;
    int base[1];  // first atom of each chunk, max_chunks + 1 entries per warp, or for all of them (dynamic)
};

// shared_bases: one table for the CTA; the grid is then the batch.
template <int NW>
__global__ void __launch_bounds__(32 * NW) a2c_bwd_coords_ring_kernel(A2cArgs<float> a, int nb, int max_chunks,
                                                                      bool shared_bases) {
    constexpr int NT = 32 * NW;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    A2cBwdRingSmem<NW> &sm = *reinterpret_cast<A2cBwdRingSmem<NW> *>(smem_raw);
    __shared__ __align__(16) float s_ring[NW][12];  // G, S, the chunk's first N
    __shared__ __align__(8) uint64_t s_bar[NW];

    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int b_first = nb - 1 - (int)blockIdx.x;
    unsigned char c_first[kFirstLetters][4];  // of the first chain, asked for together with the topology
    if (b_first >= 0) load_letters(a, b_first, 0, lane, c_first);
    {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(&g_ring_bwd_topo);
        for (int i = threadIdx.x; i < (int)(sizeof(RingBwdTopology) / 4); i += NT)
            reinterpret_cast<uint32_t *>(&sm.topo)[i] = src[i];
    }
    if (lane == 0) mbar_init(&s_bar[w]);
    __syncthreads();
    int *base = sm.base + (shared_bases ? 0 : w * (max_chunks + 1));
    constexpr float inv_dphi = 1.f / kTopoF32.bb_d[0], inv_dpsi = 1.f / kTopoF32.bb_d[1],
                    inv_dom = 1.f / kTopoF32.bb_d[2];

    // the warp's next chunk: the i-th of chain b counted from its last (length len, nch
    // chunks; an empty or refused chain has one, which writes its zeros)
    int b = b_first, i = w, len = 0, nch = 0;
    unsigned char letter = 0;
    auto enter = [&](auto &letters) {
        int run = 0;
        __syncwarp();  // every lane has read the bases of the chain before
        len = ring_chain_length(a, b, sm.topo.letter, lane, letters, [&](int c, int n) {
#pragma unroll
            for (int off = 1; off < 8; off <<= 1) n += __shfl_xor_sync(0xffffffffu, n, off);
            int inc = n;  // atoms of the chunks up to this lane's
#pragma unroll
            for (int off = 8; off < 32; off <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, inc, off);
                if (lane >= off) inc += v;
            }
            c += lane >> 3;
            if ((lane & 7) == 0 && c <= max_chunks) base[c] = run + inc - n;
            run += __shfl_sync(0xffffffffu, inc, 31);
        });
        __syncwarp();  // what follows writes some of the same entries
        if (len > 0 && run > a.maxA) {  // a chain whose atoms overflow the rows gets zeros
            if (lane == 0) a2c_error(a.hdr, TPL_ERR_ATOMS);
            len = 0;
        }
        nch = max(1, (len + kA2cChunk - 1) / kA2cChunk);
        if (lane == 0) {
            if (len == 0) base[0] = run = 0;
            base[nch] = run;
        }
        __syncwarp();
    };
    auto settle = [&]() {
        while (i >= nch) {
            i -= nch;
            b -= (int)gridDim.x;
            if (b < 0) break;
            unsigned char c[1][4];
            load_letters(a, b, 0, lane, c);
            enter(c);
        }
    };
    bool failed = false;  // a bulk copy timed out: the remaining chunks only pass the carry on
    auto fetch = [&]() {  // start the next chunk's copies
        if (b < 0 || failed) return;
        const int k = nch - 1 - i, j = k * kA2cChunk + lane, a0 = base[k], n3 = 3 * (base[k + 1] - a0);
        if (j < len) letter = a.seq[(size_t)b * a.seq_stride + j];
        const size_t at = (size_t)b * 3 * a.maxA + (size_t)3 * a0;
        const float *x = a.coords + at, *g = a.grad_coords + at;
        stage_spans(StageSpan(x, sm.x[w] + block_offset(x), n3), StageSpan(g, sm.g[w] + block_offset(g), n3), &s_bar[w],
                    lane);
    };
    if (b >= 0) {
        enter(c_first);
        if (shared_bases) __syncthreads();  // the warps write the same entries, in their own time
        settle();
        fetch();
    }
    unsigned parity = 0;
#pragma unroll 1
    while (b >= 0) {
        const int cb = b, clen = len, k = nch - 1 - i, j = k * kA2cChunk + lane;
        const bool live = j < clen;
        const unsigned info = live ? sm.topo.letter[letter] : 0u;
        const int ty = info & 0xff, na = info >> 8;
        int inc = na;  // the residue's first atom inside the chunk: warp exclusive scan
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += v;
        }
        const int aoff = inc - na;
        const size_t at = (size_t)cb * 3 * a.maxA + (size_t)3 * base[k];
        const float *sx = sm.x[w] + block_offset(a.coords + at), *sg = sm.g[w] + block_offset(a.grad_coords + at);
        if (!failed) {
            cp_async_wait_all();
            const bool ok = mbar_wait(&s_bar[w], parity);
            if (!__all_sync(0xffffffffu, ok)) {
                if (lane == 0) a2c_error(a.hdr, TPL_ERR_LOOKBACK_TIMEOUT);
                (void)mbar_wait(&s_bar[w], parity);  // bounded: let the copies in flight land
                failed = true;
            }
            parity ^= 1u;
        }
        __syncwarp();  // every lane's word copies have landed
        // One walk over the residue's atoms, last to first, from G = S = 0.  Every
        // joint gradient u . (S - o x G) is linear in (G, S), so each joint's share of
        // its own residue is taken here and the share of the later residues is added
        // after the scan: complete for the chi joints (side-chain atoms only), and
        // the own parts of psi and phi.  The walk ends with the residue's totals.
        float o[3] = {0.f, 0.f, 0.f};  // chunk origin: its first N atom
        PairSums v = zero_sums();
        float gr[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float xN[3] = {0.f, 0.f, 0.f}, xA[3] = {0.f, 0.f, 0.f}, xC[3] = {0.f, 0.f, 0.f};
        if (live && !failed) {
#pragma unroll
            for (int c = 0; c < 3; c++) o[c] = sx[c];
            const float *X = sx + 3 * aoff, *Gg = sg + 3 * aoff;
#pragma unroll
            for (int c = 0; c < 3; c++) {
                xN[c] = X[c] - o[c];
                xA[c] = X[3 + c] - o[c];
                xC[c] = X[3 * (na - 2) + c] - o[c];
            }
            add_atom(X + 3 * (na - 1), Gg + 3 * (na - 1), o, v);  // O
            gr[1] = joint_grad(xC, xA, inv_dpsi, v);
            add_atom(X + 3 * (na - 2), Gg + 3 * (na - 2), o, v);  // C
            // side chain, groups last to first; chi subtrees hold side-chain atoms only
            PairSums side = zero_sums();
            RingBwdJoint jt[kMaxScJoints];
#pragma unroll
            for (int kk = 0; kk < kMaxScJoints; kk++) jt[kk] = sm.topo.joint[ty][kk];
            if (jt[0].bits == 0)  // no side-chain joint: the Pro ring (nothing for Gly)
                for (int q = 2; q < na - 2; q++) add_atom(X + 3 * q, Gg + 3 * q, o, side);
            // unrolled over the joints: joint kk reads chi angle kk or none (Ala;
            // topology_layout_ok), so its gradient goes to a register, not a select
#pragma unroll
            for (int kk = kMaxScJoints - 1; kk >= 0; kk--) {
                if (jt[kk].bits == 0) continue;
                const int f0 = 2 + ((jt[kk].bits >> 8) & 0xff), f1 = f0 + (jt[kk].bits & 0xff);
                for (int q = f1 - 1; q >= f0; q--) add_atom(X + 3 * q, Gg + 3 * q, o, side);
                if (jt[kk].bits >> 16) {
                    const float *pk = X + 3 * f0;
                    const float *pp = kk == 0 ? X + 3 : X + 3 * (2 + ((jt[kk > 0 ? kk - 1 : 0].bits >> 8) & 0xff));
                    const float ok_[3] = {pk[0] - o[0], pk[1] - o[1], pk[2] - o[2]};
                    const float op_[3] = {pp[0] - o[0], pp[1] - o[1], pp[2] - o[2]};
                    gr[3 + kk] = joint_grad(ok_, op_, jt[kk].inv_d, side);
                }
            }
            v = v + side;
            gr[0] = joint_grad(xA, xN, inv_dphi, v);
            add_atom(X + 3, Gg + 3, o, v);  // CA
            add_atom(X, Gg, o, v);          // N
        }
#pragma unroll
        for (int c = 0; c < 3; c++) o[c] = __shfl_sync(0xffffffffu, o[c], 0);  // lane 0 is live in every chunk but an empty one
        // the walk was the last to read the buffers: the next chunk's copies may start
        const bool more = i + 1 < nch || b - (int)gridDim.x >= 0;  // the stream goes on after this chunk
        const bool first = cb == b_first && i == 0, top = i == 0;   // first of the stream, last chunk of its chain
        __syncwarp();
        i += NW;
        settle();
        fetch();

        PairSums ctot;
        const PairSums later = suffix_excl(v, lane, ctot);
        float xn[3];  // the next residue's N: the next lane's
#pragma unroll
        for (int c = 0; c < 3; c++) xn[c] = __shfl_down_sync(0xffffffffu, xN[c], 1);
        // the sums over later chunks, moved to this chunk's origin: S_o = S_on + (on - o) x G
        float Gc[3] = {0.f, 0.f, 0.f}, Sc[3] = {0.f, 0.f, 0.f};
        if (!first) ring_wait<NW>(w);
        if (!top) {
            float c9[9];
            load_sums(s_ring[w], c9);
            float d[3], dx[3];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                Gc[c] = c9[c];
                Sc[c] = c9[3 + c];
                d[c] = c9[6 + c] - o[c];
                if (lane == 31) xn[c] = d[c];  // the next chunk's first N
            }
            cross3(d, Gc, dx);
#pragma unroll
            for (int c = 0; c < 3; c++) Sc[c] += dx[c];
        }
        if (k > 0 && lane == 0)
            store_sums(s_ring[(w + 1) % NW], Gc[0] + ctot.g.x, Gc[1] + ctot.g.y, Gc[2] + ctot.z.x, Sc[0] + ctot.s.x,
                       Sc[1] + ctot.s.y, Sc[2] + ctot.z.y, o);
        if (more) ring_signal<NW>((w + 1) % NW);
        float *gout = a.grad_angles + (size_t)cb * 8 * a.L;
        if (live && !failed) {
            // the later residues' share: sums over every atom after this residue
            const PairSums t = later + PairSums{make_float2(Gc[0], Gc[1]), make_float2(Sc[0], Sc[1]), make_float2(Gc[2], Sc[2])};
            if (j + 1 < clen) gr[2] = joint_grad(xn, xC, inv_dom, t);  // omega_j
            gr[1] += joint_grad(xC, xA, inv_dpsi, t);
            gr[0] += joint_grad(xA, xN, inv_dphi, t);
#pragma unroll
            for (int q = 0; q < 8; q++) gout[(size_t)q * a.L + j] = gr[q];
        }
        if (top)  // zeros past the chain (and everywhere when it was refused)
#pragma unroll 1
            for (int q = 0; q < 8; q++)
                zero_span(gout + (size_t)q * a.L + clen, a.L - clen, lane);
    }
}

// ------------------------------------------------------------------ host side
template <int R, int NT>
static int launch_a2c_fwd(const A2cArgs<float> &a, int B, int renorm, cudaStream_t st) {
    constexpr int TILE = R * NT;
    const size_t smem = sizeof(A2cSmemFwd<TILE>);
    auto k = a2c_fwd_kernel<R, NT>;
    if (!set_max_dynamic_smem(reinterpret_cast<const void *>(k), (int)smem))
        return TPL_ERR_LAUNCH;
    k<<<B, NT, smem, st>>>(a, renorm);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <int R, int NT>
static int launch_a2c_bwd(const A2cArgs<float> &a, int B, int renorm, cudaStream_t st) {
    constexpr int TILE = R * NT;
    const int max_tiles = (a.L + TILE - 1) / TILE + 1;
    const size_t smem = sizeof(A2cSmemBwd<TILE>) + (sizeof(Frame<float>) + sizeof(int)) * max_tiles;
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if ((int)smem > optin) return TPL_ERR_UNSUPPORTED;
    auto k = a2c_bwd_kernel<R, NT>;
    if (!set_max_dynamic_smem(reinterpret_cast<const void *>(k), (int)smem))
        return TPL_ERR_LAUNCH;
    k<<<B, NT, smem, st>>>(a, renorm, max_tiles);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

// Warps per chain of the float32 kernels: eight while the batch leaves SMs short of chains,
// four once every SM has several.  GB300, eight / four warps, us, chains of U{50..500}
// residues: forward with names 700 chains 25.9 / 28.0, 1024 37.2 / 38.9, 1500 49.0 / 48.6
// (without names the same line); backward, of whose CTAs of eight warps two fit an SM, 256
// chains 14.9 / 17.9, 400 22.0 / 20.5, 512 24.1 / 21.5.
static int a2c_ring_warps(int B, int chains_per_sm) { return B <= chains_per_sm * device_sm_count() ? 8 : 4; }

// The resident CTAs, at most one per chain (a batch of one per SM need not ask).
template <typename K>
static int ring_grid(K kernel, int threads, size_t smem, int B) {
    const int sms = device_sm_count();
    if (B <= sms) return B;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    return std::min(B, per_sm * sms);
}

template <int NW>
static int launch_a2c_fwd_ring(const A2cArgs<float> &a, int B, int renorm, cudaStream_t st) {
    const bool names = a.res_names && a.atom_names;
    const size_t smem = names ? sizeof(A2cRingSmem<NW, true>) : sizeof(A2cRingSmem<NW, false>);
    auto k = names ? a2c_fwd_ring_kernel<NW, true> : a2c_fwd_ring_kernel<NW, false>;
    if (!set_max_dynamic_smem(reinterpret_cast<const void *>(k), (int)smem))
        return TPL_ERR_LAUNCH;
    const int grid = ring_grid(k, 32 * NW, smem, B);
    k<<<grid, 32 * NW, smem, st>>>(a, renorm, B);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

template <int NW>
static int launch_a2c_bwd_coords_ring(const A2cArgs<float> &a, int B, int L, cudaStream_t st) {
    const int max_chunks = std::max(1, (L + kA2cChunk - 1) / kA2cChunk);
    auto k = a2c_bwd_coords_ring_kernel<NW>;
    size_t smem = 0;
    auto fits = [&](int tables) {
        smem = offsetof(A2cBwdRingSmem<NW>, base) + sizeof(int) * (size_t)tables * (size_t)(max_chunks + 1);
        if (smem <= (1u << 30) && set_max_dynamic_smem(reinterpret_cast<const void *>(k), (int)smem)) return true;
        (void)cudaGetLastError();  // a size past the limit is no failure yet
        return false;
    };
    const bool shared_bases = !fits(NW);
    if (shared_bases && !fits(1)) return TPL_ERR_UNSUPPORTED;
    const int grid = shared_bases ? B : ring_grid(k, 32 * NW, smem, B);
    k<<<grid, 32 * NW, smem, st>>>(a, B, max_chunks, shared_bases);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

int a2c_forward(bool f64, const unsigned char *seq, int seq_stride, const void *angles, void *coords,
                uint32_t *res_names, uint32_t *atom_names, void *ws, int B, int L, int maxA,
                const tpl_options &opt, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    const int renorm = opt.renormalize >= 0 ? 1 : 0;
    if (f64) {
        A2cArgs<double> a{seq, seq_stride, (const double *)angles, (double *)coords, res_names, atom_names,
                          nullptr, nullptr, (WsHeader *)ws, L, maxA};
        return a2c_forward_f64(a, B, renorm != 0, st);
    }
    A2cArgs<float> a{seq, seq_stride, (const float *)angles, (float *)coords, res_names, atom_names,
                     nullptr, nullptr, (WsHeader *)ws, L, maxA};
    // threads_per_cta: 4 or 8 = that many warps on chunks of 32 residues (0: by the batch);
    // 128 = 128 threads x 2 residues; 256 or 512 = one residue per thread
    switch (opt.threads_per_cta) {
        case 4: return launch_a2c_fwd_ring<4>(a, B, renorm, st);
        case 8: return launch_a2c_fwd_ring<8>(a, B, renorm, st);
        case 128: return launch_a2c_fwd<2, 128>(a, B, renorm, st);
        case 256: return launch_a2c_fwd<1, 256>(a, B, renorm, st);
        case 512: return launch_a2c_fwd<1, 512>(a, B, renorm, st);
    }
    return a2c_ring_warps(B, 8) == 8 ? launch_a2c_fwd_ring<8>(a, B, renorm, st)
                                     : launch_a2c_fwd_ring<4>(a, B, renorm, st);
}

int a2c_backward(bool f64, void *grad_angles, const void *grad_coords, const unsigned char *seq, int seq_stride,
                 const void *angles, void *ws, int B, int L, int maxA, const tpl_options &opt, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    const int renorm = opt.renormalize >= 0 ? 1 : 0;
    if (f64) {
        A2cArgs<double> a{seq, seq_stride, (const double *)angles, nullptr, nullptr, nullptr,
                          (double *)grad_angles, (const double *)grad_coords, (WsHeader *)ws, L, maxA};
        return a2c_backward_f64(a, B, renorm != 0, st);
    }
    A2cArgs<float> a{seq, seq_stride, (const float *)angles, nullptr, nullptr, nullptr, (float *)grad_angles,
                     (const float *)grad_coords, (WsHeader *)ws, L, maxA};
    switch (opt.threads_per_cta) {
        case 128: return launch_a2c_bwd<2, 128>(a, B, renorm, st);
        case 512: return launch_a2c_bwd<1, 512>(a, B, renorm, st);
    }
    return launch_a2c_bwd<1, 256>(a, B, renorm, st);
}

int a2c_backward_coords(float *grad_angles, const float *grad_coords, const float *coords, const unsigned char *seq,
                        int seq_stride, void *ws, int B, int L, int maxA, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    A2cArgs<float> a{seq, seq_stride, nullptr, const_cast<float *>(coords), nullptr, nullptr, grad_angles, grad_coords,
                     (WsHeader *)ws, L, maxA};
    return a2c_ring_warps(B, 2) == 8 ? launch_a2c_bwd_coords_ring<8>(a, B, L, st)
                                     : launch_a2c_bwd_coords_ring<4>(a, B, L, st);
}

int num_atoms_host(const char *seq) {
    static constexpr Topology<double> tp = make_topology<double>();
    int n = 0;
    for (const char *p = seq; *p; p++) {
        int t = residue_type((unsigned char)*p);
        if (t < 0) return -1;
        n += tp.natoms[t];
    }
    return n;
}

}  // namespace tpl
