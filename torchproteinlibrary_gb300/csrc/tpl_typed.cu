// Coords2TypedCoords on the GPU (sm_103a): atoms regrouped by the 11 atom types of
// ProtUtil::get11AtomType (Math/nUtil.cpp:567-703), stable within a type.
//
// Reference: Layers/FullAtomModel/Coords2TypedCoords/coords2typedcoords_interface.cpp
// runs on the CPU, one OpenMP task per chain, with string compares per atom.  Here
// one CTA per chain classifies its atoms from the packed 4-byte name words that
// Angles2Coords writes, one probe of a perfect hash each, ranks every atom among those of
// its type, and moves the coordinates in input order within each type, groups of 128 atoms
// ordered in shared memory first so that a type's run is written by consecutive lanes
// (typed_fwd_group_kernel; short rows in large batches take typed_fwd_scatter_kernel, rows
// past 32 768 atoms typed_fwd_kernel).  The backward is
// the inverse gather.  Integer and byte work only; coordinates are copied unchanged.
#include <cstddef>
#include <cstdint>
#include <type_traits>

#include "tpl_async.cuh"
#include "tpl_internal.h"

namespace tpl {
namespace {

constexpr int kTypes = 11;
constexpr int kTypedThreads = 256;

// Name word: the bytes of a NUL-padded 4-byte name slot, little-endian.
constexpr uint32_t nm(const char *s) {
    uint32_t w = 0;
    for (int i = 0; i < 4 && s[i]; i++) w |= (uint32_t)(unsigned char)s[i] << (8 * i);
    return w;
}

struct TypedName {
    uint32_t res, atom;
    int type;
};

// Residue-specific types (0-based, as get11AtomType returns them); the
// residue-agnostic backbone names are handled first in atom_type().
constexpr TypedName kTypedNames[] = {
    // 0: sulfur / selenium
    {nm("CYS"), nm("SG"), 0}, {nm("MET"), nm("SD"), 0}, {nm("MSE"), nm("SE"), 0},
    // 1: amide N
    {nm("ASN"), nm("ND2"), 1}, {nm("GLN"), nm("NE2"), 1},
    // 2: aromatic N
    {nm("HIS"), nm("ND1"), 2}, {nm("HIS"), nm("NE2"), 2}, {nm("TRP"), nm("NE1"), 2},
    // 3: guanidine N
    {nm("ARG"), nm("NH1"), 3}, {nm("ARG"), nm("NH2"), 3}, {nm("ARG"), nm("NE"), 3},
    // 4: N with three hydrogens
    {nm("LYS"), nm("NZ"), 4},
    // 5: carbonyl / amide O
    {nm("ACE"), nm("O"), 5}, {nm("ASN"), nm("OD1"), 5}, {nm("GLN"), nm("OE1"), 5},
    // 6: hydroxyl O
    {nm("SER"), nm("OG"), 6}, {nm("THR"), nm("OG1"), 6}, {nm("TYR"), nm("OH"), 6},
    // 7: carboxyl O
    {nm("ASP"), nm("OD1"), 7}, {nm("ASP"), nm("OD2"), 7}, {nm("GLU"), nm("OE1"), 7}, {nm("GLU"), nm("OE2"), 7},
    // 8: sp2 C
    {nm("ARG"), nm("CZ"), 8}, {nm("ASP"), nm("CG"), 8}, {nm("GLU"), nm("CD"), 8}, {nm("ACE"), nm("C"), 8},
    {nm("ASN"), nm("CG"), 8}, {nm("GLN"), nm("CD"), 8},
    // 9: aromatic C
    {nm("HIS"), nm("CD2"), 9}, {nm("HIS"), nm("CE1"), 9}, {nm("HIS"), nm("CG"), 9},
    {nm("PHE"), nm("CD1"), 9}, {nm("PHE"), nm("CD2"), 9}, {nm("PHE"), nm("CE1"), 9}, {nm("PHE"), nm("CE2"), 9},
    {nm("PHE"), nm("CG"), 9}, {nm("PHE"), nm("CZ"), 9},
    {nm("TRP"), nm("CD1"), 9}, {nm("TRP"), nm("CD2"), 9}, {nm("TRP"), nm("CE2"), 9}, {nm("TRP"), nm("CE3"), 9},
    {nm("TRP"), nm("CG"), 9}, {nm("TRP"), nm("CH2"), 9}, {nm("TRP"), nm("CZ2"), 9}, {nm("TRP"), nm("CZ3"), 9},
    {nm("TYR"), nm("CD1"), 9}, {nm("TYR"), nm("CD2"), 9}, {nm("TYR"), nm("CE1"), 9}, {nm("TYR"), nm("CE2"), 9},
    {nm("TYR"), nm("CG"), 9}, {nm("TYR"), nm("CZ"), 9},
    // 10: sp3 C
    {nm("ALA"), nm("CB"), 10}, {nm("ARG"), nm("CB"), 10}, {nm("ARG"), nm("CG"), 10}, {nm("ARG"), nm("CD"), 10},
    {nm("ASN"), nm("CB"), 10}, {nm("ASP"), nm("CB"), 10}, {nm("GLN"), nm("CB"), 10}, {nm("GLN"), nm("CG"), 10},
    {nm("GLU"), nm("CB"), 10}, {nm("GLU"), nm("CG"), 10}, {nm("HIS"), nm("CB"), 10},
    {nm("ILE"), nm("CB"), 10}, {nm("ILE"), nm("CD1"), 10}, {nm("ILE"), nm("CG1"), 10}, {nm("ILE"), nm("CG2"), 10},
    {nm("LEU"), nm("CB"), 10}, {nm("LEU"), nm("CD1"), 10}, {nm("LEU"), nm("CD2"), 10}, {nm("LEU"), nm("CG"), 10},
    {nm("LYS"), nm("CB"), 10}, {nm("LYS"), nm("CD"), 10}, {nm("LYS"), nm("CG"), 10}, {nm("LYS"), nm("CE"), 10},
    {nm("MET"), nm("CB"), 10}, {nm("MET"), nm("CE"), 10}, {nm("MET"), nm("CG"), 10},
    {nm("MSE"), nm("CB"), 10}, {nm("MSE"), nm("CE"), 10}, {nm("MSE"), nm("CG"), 10}, {nm("PHE"), nm("CB"), 10},
    {nm("PRO"), nm("CB"), 10}, {nm("PRO"), nm("CG"), 10}, {nm("PRO"), nm("CD"), 10}, {nm("SER"), nm("CB"), 10},
    {nm("THR"), nm("CG2"), 10}, {nm("TRP"), nm("CB"), 10}, {nm("TYR"), nm("CB"), 10},
    {nm("VAL"), nm("CB"), 10}, {nm("VAL"), nm("CG1"), 10}, {nm("VAL"), nm("CG2"), 10},
    {nm("ACE"), nm("CH3"), 10}, {nm("THR"), nm("CB"), 10}, {nm("CYS"), nm("CB"), 10},
};
constexpr int kTypedNameCount = sizeof(kTypedNames) / sizeof(TypedName);

// The names as two tables in which every one has a place of its own (multipliers found by
// trial; checked at compile time), so that a lookup is one probe of each and no branch:
// the residue-agnostic names by their atom word, the pairs by both words.
constexpr int kPairSlots = 512, kPlainSlots = 16;
struct alignas(8) TypedTables {  // an entry is read as one 8-byte word
    uint32_t pair[kPairSlots][2];   // residue word | type << 24, atom word; type 0xff in an empty slot
    uint32_t plain[kPlainSlots][2];  // atom word, type; type 0xffffffff in an empty slot
    int clashes;
};
__host__ __device__ constexpr uint32_t pair_slot(uint32_t res, uint32_t atom) {
    return ((res * 0x6d30140du) ^ (atom * 0x75d7323u)) >> 23;
}
__host__ __device__ constexpr uint32_t plain_slot(uint32_t atom) { return (atom * 0xed753c7bu) >> 28; }
constexpr TypedTables build_typed_tables() {
    TypedTables t{};
    for (int i = 0; i < kPairSlots; i++) t.pair[i][0] = 0xff000000u;
    for (int i = 0; i < kPlainSlots; i++) t.plain[i][1] = 0xffffffffu;
    for (int i = 0; i < kTypedNameCount; i++) {
        const uint32_t k = pair_slot(kTypedNames[i].res, kTypedNames[i].atom);
        if (t.pair[k][0] != 0xff000000u) t.clashes++;
        t.pair[k][0] = kTypedNames[i].res | (uint32_t)kTypedNames[i].type << 24;
        t.pair[k][1] = kTypedNames[i].atom;
    }
    // O is not a terminal oxygen (the reference's call passes false)
    const TypedName plain[6] = {{0, nm("O"), 5}, {0, nm("OXT"), 7}, {0, nm("OT2"), 7},
                                {0, nm("N"), 1}, {0, nm("C"), 8},   {0, nm("CA"), 10}};
    for (int i = 0; i < 6; i++) {
        const uint32_t k = plain_slot(plain[i].atom);
        if (t.plain[k][1] != 0xffffffffu) t.clashes++;
        t.plain[k][0] = plain[i].atom;
        t.plain[k][1] = (uint32_t)plain[i].type;
    }
    return t;
}
static_assert(build_typed_tables().clashes == 0, "every name has its own slot");
static_assert(alignof(TypedTables) >= sizeof(uint2) && offsetof(TypedTables, plain) % sizeof(uint2) == 0,
              "entries on 8-byte boundaries, in global memory too");
__device__ const TypedTables g_typed_tables = build_typed_tables();

// Drop the space bytes of a name word (the reference erases whitespace from the
// atom name before comparing) and stop at the first NUL.
__device__ __forceinline__ uint32_t squeeze(uint32_t w) {
    uint32_t out = 0;
    int k = 0;
    for (int i = 0; i < 4; i++) {
        const uint32_t c = (w >> (8 * i)) & 0xffu;
        if (c == 0) break;
        if (c == ' ' || (c >= 9 && c <= 13)) continue;
        out |= c << (8 * k++);
    }
    return out;
}

// squeeze() without the byte loop when the name has no byte below '!' before its
// first NUL (the names Angles2Coords writes): the word up to that NUL.  Per byte,
// (w - 0x01) & ~w & 0x80 flags a NUL and (w - 0x21) & ~w & 0x80 a byte below 0x21;
// borrows only make false flags above a true one, so the lowest flag is exact.
__device__ __forceinline__ uint32_t squeeze_fast(uint32_t w) {
    const uint32_t nul = (w - 0x01010101u) & ~w & 0x80808080u;
    const uint32_t valid = nul ? (((nul & (0u - nul)) >> 7) - 1u) : 0xffffffffu;  // bytes before the first NUL
    const uint32_t low = (w - 0x21212121u) & ~w & 0x80808080u;
    if ((low & valid) == 0u) return w & valid;
    return squeeze(w);
}

// The 0-based type of an atom, or -1 for a name pair the reference rejects; tables in
// global memory, or a copy in shared memory.
__device__ __forceinline__ int atom_type(uint32_t res, uint32_t atom, const TypedTables &t) {
    atom = squeeze_fast(atom);
    res = res & 0x00ffffffu;  // the residue is its 3-letter code
    const uint2 p = *reinterpret_cast<const uint2 *>(t.pair[pair_slot(res, atom)]);
    const uint2 q = *reinterpret_cast<const uint2 *>(t.plain[plain_slot(atom)]);
    const int by_pair = p.y == atom && (p.x & 0x00ffffffu) == res ? (int)p.x >> 24 : -1;
    const int by_atom = q.x == atom ? (int)q.y : -1;
    return by_atom >= 0 ? by_atom : by_pair;
}
__device__ __forceinline__ int atom_type(uint32_t res, uint32_t atom) { return atom_type(res, atom, g_typed_tables); }

// Input rows hold in_stride atoms (coordinates and names); typed rows and atom
// indexes hold out_stride slots.  One CTA per chain, for chains too long for
// typed_fwd_group_kernel's codes: the scatter pass looks the types up again.
template <typename T>
__global__ void __launch_bounds__(kTypedThreads) typed_fwd_kernel(const T *coords, const uint32_t *res_names,
                                                                  const uint32_t *atom_names, const int *num_atoms,
                                                                  int in_stride, int out_stride, T *out,
                                                                  int *n_of_type, int *offsets, int *atom_index,
                                                                  WsHeader *hdr) {
    constexpr int NW = kTypedThreads / 32;
    __shared__ int s_count[kTypes], s_off[kTypes], s_base[kTypes];
    __shared__ int s_wc[kTypes][NW];
    const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int n = max(0, min(num_atoms[b], min(in_stride, out_stride)));
    const size_t row = (size_t)b * in_stride, orow = (size_t)b * out_stride;
    if (tid < kTypes) {
        s_count[tid] = 0;
        s_base[tid] = 0;
    }
    __syncthreads();
    for (int j = tid; j < n; j += kTypedThreads) {
        const int t = atom_type(res_names[row + j], atom_names[row + j]);
        if (t >= 0) atomicAdd(&s_count[t], 1);
        else atomicCAS(&hdr->status, 0u, (unsigned)TPL_ERR_ATOM_TYPE);
    }
    __syncthreads();
    if (tid == 0) {
        int o = 0;
        for (int k = 0; k < kTypes; k++) {
            s_off[k] = o;
            o += s_count[k];
        }
    }
    __syncthreads();
    if (tid < kTypes) {
        n_of_type[(size_t)b * kTypes + tid] = s_count[tid];
        offsets[(size_t)b * kTypes + tid] = s_off[tid];
    }
    const int ntyped = s_off[kTypes - 1] + s_count[kTypes - 1];
    // stable scatter, one tile of kTypedThreads atoms at a time
    for (int j0 = 0; j0 < n; j0 += kTypedThreads) {
        const int j = j0 + tid;
        // the atom's coordinates, loaded before the ranking so that the load overlaps it
        T x0 = T(0), x1 = T(0), x2 = T(0);
        if (j < n) {
            const T *src = coords + 3 * (row + j);
            x0 = src[0];
            x1 = src[1];
            x2 = src[2];
        }
        const int t = j < n ? atom_type(res_names[row + j], atom_names[row + j]) : -1;
        int rank = 0;
        const unsigned below = (1u << lane) - 1u;
#pragma unroll
        for (int k = 0; k < kTypes; k++) {
            const unsigned m = __ballot_sync(0xffffffffu, t == k);
            if (t == k) rank = __popc(m & below);
            if (lane == 0) s_wc[k][w] = __popc(m);
        }
        __syncthreads();
        if (t >= 0) {
            int before = s_base[t];
            for (int v = 0; v < w; v++) before += s_wc[t][v];
            const int slot = s_off[t] + before + rank;
            T *dst = out + 3 * (orow + slot);
            dst[0] = x0;
            dst[1] = x1;
            dst[2] = x2;
            atom_index[orow + slot] = j;
        }
        __syncthreads();
        if (tid < kTypes)
            for (int v = 0; v < NW; v++) s_base[tid] += s_wc[tid][v];
        __syncthreads();
    }
    // slots past the typed atoms are zero, as in the reference's zero-filled outputs
    for (int s = ntyped + tid; s < out_stride; s += kTypedThreads) {
        T *dst = out + 3 * (orow + s);
        dst[0] = dst[1] = dst[2] = T(0);
        atom_index[orow + s] = 0;
    }
}

// The same regrouping by NW = 4 or 8 warps per chain with two CTA barriers, for chains whose
// per-atom codes fit in shared memory.  Each warp takes an equal run of the chain's 32-atom
// tiles.  Pass 1 types the atoms and ranks each among the warp's atoms of its type (per
// tile, __match_any_sync groups the lanes of each type); type and rank stay in shared
// memory, and with them how many atoms of each type came before every group of 128.  After
// a barrier every warp knows where its atoms of each type start (the type's offset plus
// the earlier warps' counts): an atom's slot is that plus its rank, so the order within a
// type is the input order.  Pass 2 takes the groups in turn: the atoms' places when the
// group is ordered by type, and its slots, go to shared memory, the coordinates come there
// by cp.async one group ahead, and consecutive lanes write consecutive words of a type's
// run.
//
// What bounds it is instruction issue and the sectors written: an atom scattered straight
// to its slot costs three partial sectors of coordinates and one of index.  GB300, 4096
// chains of U{50..500} residues (72 us of HBM traffic): 142 us with scattered stores, a
// probed name hash and ranks found twice (73 M warp instructions, 21.7 M sector writes);
// 102 us with four warps per chain (63 M, 17.0 M), 98 with eight.  Ordering the groups without keeping the ranks was slower than
// scattering (160 us, 101 M).
constexpr int kTypedUnroll = 4;
constexpr int kTypedGroup = 32 * kTypedUnroll;  // atoms ordered and written together
constexpr int kTypedMaxAtoms = 32768;           // 16-bit codes: ranks below 4096 with NW = 4 up to 16384 atoms, 8 past that

// Groups of one warp's share of a row, and the dynamic shared memory: per warp two groups'
// coordinates, codes (16 bits per atom), and per warp the counts before each group and
// after the last.
constexpr int typed_groups(int in_stride, int nw) {
    return (((in_stride + 31) / 32 + nw - 1) / nw + kTypedUnroll - 1) / kTypedUnroll;
}
template <typename T>
constexpr int kRawWords = 3 * kTypedGroup * (int)sizeof(T) / 4 + 4;  // 4 words for the 16-byte phase
template <typename T>
constexpr size_t typed_smem(int in_stride, int nw) {
    return 8 * (size_t)nw * kRawWords<T> +
           2 * ((size_t)in_stride + (size_t)nw * (typed_groups(in_stride, nw) + 1) * kTypes);
}

// Copy the n words at src to dst, shared memory of the same 16-byte phase, by the warp
// with cp.async (not committed).
__device__ __forceinline__ void stage_words(float *dst, const float *src, int n, int lane) {
    const StageSpan sp(src, dst, n);
    sp.ends(lane);
    for (int i = 4 * lane; i < sp.body; i += 128) cp_async16(dst + sp.head + i, src + sp.head + i);
}

template <typename T, int NW>
__global__ void __launch_bounds__(32 * NW) typed_fwd_group_kernel(
    const T *__restrict__ coords, const uint32_t *__restrict__ res_names, const uint32_t *__restrict__ atom_names,
    const int *__restrict__ num_atoms, int in_stride, int out_stride, T *__restrict__ out,
    int *__restrict__ n_of_type, int *__restrict__ offsets, int *__restrict__ atom_index, WsHeader *hdr) {
    constexpr int kWords = sizeof(T) / 4;
    extern __shared__ __align__(16) unsigned char s_dyn[];
    uint16_t *s_code = reinterpret_cast<uint16_t *>(s_dyn + 8 * NW * kRawWords<T>);  // by atom: rank << 4 | type (15: none)
    __shared__ int s_cnt[NW][kTypes];
    __shared__ __align__(16) TypedTables s_tab;
    __shared__ uint32_t s_perm[NW][kTypedGroup];  // by place in the group: 3 * slot << 9 | 3 * atom of the group
    __shared__ int2 s_at[NW][16];                 // per type: place and slot of rank 0
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, b = blockIdx.x;
    {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(&g_typed_tables);
        uint32_t *dst = reinterpret_cast<uint32_t *>(&s_tab);
        for (int i = threadIdx.x; i < (int)(sizeof(TypedTables) / 4); i += 32 * NW) dst[i] = src[i];
    }
    const int n = max(0, min(num_atoms[b], min(in_stride, out_stride)));
    const size_t row = (size_t)b * in_stride, orow = (size_t)b * out_stride;
    const uint32_t *rn = res_names + row, *an = atom_names + row;
    const unsigned below = (1u << lane) - 1u;
    const int ntiles = (n + 31) >> 5, per = (ntiles + NW - 1) / NW;
    const int a0 = min(n, 32 * w * per), a1 = min(n, a0 + 32 * per);  // this warp's atoms
    uint16_t *s_before = s_code + in_stride + w * (typed_groups(in_stride, NW) + 1) * kTypes;
    int *cnt = s_cnt[w];
    if (lane < kTypes) cnt[lane] = 0;

    const float *src = reinterpret_cast<const float *>(coords + 3 * row);
    float *s_raw = reinterpret_cast<float *>(s_dyn) + 2 * w * kRawWords<T>;  // two groups' coordinates
    auto fetch = [&](int j0, int q) {
        if (j0 < a1) {
            const float *from = src + (size_t)3 * kWords * j0;
            stage_words(s_raw + q * kRawWords<T> + block_offset(from), from, 3 * kWords * min(kTypedGroup, a1 - j0), lane);
        }
        cp_async_commit();
    };
    fetch(a0, 0);  // the first group's coordinates arrive during pass 1
    __syncthreads();  // the tables and the zeroed counts
    bool bad = false;
    uint16_t *before = s_before;
    uint32_t r[kTypedUnroll], a[kTypedUnroll];  // the next group's names, loaded one group ahead (115 -> 102 us)
    auto names = [&](int j0) {
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            const int j = j0 + 32 * u + lane;
            r[u] = j < a1 ? rn[j] : 0u;
            a[u] = j < a1 ? an[j] : 0u;
        }
    };
    names(a0);
    for (int j0 = a0; j0 < a1; j0 += kTypedGroup, before += kTypes) {
        uint32_t res[kTypedUnroll], atom[kTypedUnroll];
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            res[u] = r[u];
            atom[u] = a[u];
        }
        names(j0 + kTypedGroup);
        if (lane < kTypes) before[lane] = (uint16_t)cnt[lane];
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            const int j = j0 + 32 * u + lane;
            const int t = j < a1 ? atom_type(res[u], atom[u], s_tab) : -2;  // -1: a name pair the reference rejects
            bad |= t == -1;
            const unsigned m = __match_any_sync(0xffffffffu, t);
            const int c = t >= 0 ? cnt[t] : 0;
            __syncwarp();
            if (t >= 0 && (m & below) == 0u) cnt[t] = c + __popc(m);
            if (j < a1) s_code[j] = (uint16_t)(t >= 0 ? (c + __popc(m & below)) << 4 | t : 15);
            __syncwarp();
        }
    }
    if (lane < kTypes) before[lane] = (uint16_t)cnt[lane];
    if (bad) atomicCAS(&hdr->status, 0u, (unsigned)TPL_ERR_ATOM_TYPE);
    __syncthreads();
    // lane k < kTypes: the type's total, its offset, and this warp's first slot of it
    int tot = 0, earlier = 0;
    if (lane < kTypes)
#pragma unroll
        for (int v = 0; v < NW; v++) {
            const int c = s_cnt[v][lane];
            tot += c;
            earlier += v < w ? c : 0;
        }
    auto scan = [&](int v) {  // inclusive over lanes 0 .. 15
#pragma unroll
        for (int off = 1; off < 16; off <<= 1) {
            const int o = __shfl_up_sync(0xffffffffu, v, off);
            if (lane >= off) v += o;
        }
        return v;
    };
    const int inc = scan(tot), type_off = inc - tot, slot0 = type_off + earlier;
    const int ntyped = __shfl_sync(0xffffffffu, inc, kTypes - 1);
    if (w == 0 && lane < kTypes) {
        n_of_type[(size_t)b * kTypes + lane] = tot;
        offsets[(size_t)b * kTypes + lane] = type_off;
    }

    uint32_t *perm = s_perm[w];
    T *o = out + 3 * orow;
    before = s_before;
    // word e = lane + 32 i of a group's coordinates belongs to place e / 3: 32 (i / 3) plus
    // one of three values per lane
    int at[3], x[3];
#pragma unroll
    for (int k = 0; k < 3; k++) {
        at[k] = (lane + 32 * k) / 3;
        x[k] = (lane + 32 * k) % 3;
    }
    for (int j0 = a0, q = 0; j0 < a1; j0 += kTypedGroup, q ^= 1, before += kTypes) {
        __syncwarp();  // every lane is done with the group before
        fetch(j0 + kTypedGroup, q ^ 1);
        // lane k < kTypes: the type's run in the group ordered by type
        const int b0 = lane < kTypes ? before[lane] : 0, c = lane < kTypes ? before[kTypes + lane] - b0 : 0;
        const int run = scan(c), in_group = __shfl_sync(0xffffffffu, run, kTypes - 1);
        if (lane < kTypes) s_at[w][lane] = make_int2(run - c - b0, slot0);
        __syncwarp();
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            const int j = j0 + 32 * u + lane;
            const int code = j < a1 ? s_code[j] : 15, t = code & 15, rank = code >> 4;
            if (t != 15) {
                const int2 p = s_at[w][t];
                perm[p.x + rank] = (uint32_t)(3 * (p.y + rank)) << 9 | (uint32_t)(3 * (32 * u + lane));
            }
        }
        cp_async_wait1();  // this group's coordinates
        __syncwarp();
        const T *raw = reinterpret_cast<const T *>(s_raw + q * kRawWords<T> + block_offset(src + (size_t)3 * kWords * j0));
#pragma unroll
        for (int i = 0; i < 3 * kTypedUnroll; i++) {
            if (lane + 32 * i < 3 * in_group) {
                const uint32_t p = perm[32 * (i / 3) + at[i % 3]];
                o[(p >> 9) + x[i % 3]] = raw[(p & 511u) + x[i % 3]];
            }
        }
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            if (32 * u + lane < in_group) {
                const uint32_t p = perm[32 * u + lane];
                // thirds of multiples of three below 2^17 and 2^9
                atom_index[orow + ((p >> 9) * 43691u >> 17)] = j0 + (int)((p & 511u) * 171u >> 9);
            }
        }
    }
    // slots past the typed atoms are zero, as in the reference's zero-filled outputs; a
    // share of each span per warp
    auto zeros = [&](void *p, int words) {
        const int share = (words + NW - 1) / NW;
        zero_span(static_cast<uint32_t *>(p) + w * share, min(share, words - w * share), lane);
    };
    zeros(out + 3 * (orow + ntyped), 3 * kWords * (out_stride - ntyped));
    zeros(atom_index + orow + ntyped, out_stride - ntyped);
}

// Short rows in batches that fill the GPU: the same two passes, but the types are found again
// tile by tile and the coordinates go straight to their slots.  A warp has a tile or a few
// there, so ordering and staging them costs more than the partial sectors of scattered
// stores, and this form's small shared memory keeps twice the chains on an SM.  GB300,
// scattered / ordered, us: float32 16000 chains of up to 100 atoms 31 / 48, of up to 400
// 51 / 66, 4096 of 600 each 30 / 34, of 800 each 41 / 38; 300 of 400 5.1 / 4.7; float64 16000 of
// up to 100 36 / 63.
constexpr int kTypedScatterWarps = 4;
constexpr int kTypedScatterAtoms = 600;

template <typename T>
__global__ void __launch_bounds__(32 * kTypedScatterWarps) typed_fwd_scatter_kernel(
    const T *__restrict__ coords, const uint32_t *__restrict__ res_names, const uint32_t *__restrict__ atom_names,
    const int *__restrict__ num_atoms, int in_stride, int out_stride, T *__restrict__ out,
    int *__restrict__ n_of_type, int *__restrict__ offsets, int *__restrict__ atom_index, WsHeader *hdr) {
    extern __shared__ signed char s_ty[];
    __shared__ int s_cnt[kTypedScatterWarps][kTypes];
    __shared__ int s_ntyped;
    __shared__ TypedTables s_tab;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, b = blockIdx.x;
    {
        const uint32_t *src = reinterpret_cast<const uint32_t *>(&g_typed_tables);
        uint32_t *dst = reinterpret_cast<uint32_t *>(&s_tab);
        for (int i = threadIdx.x; i < (int)(sizeof(TypedTables) / 4); i += 32 * kTypedScatterWarps) dst[i] = src[i];
    }
    const int n = max(0, min(num_atoms[b], min(in_stride, out_stride)));
    const size_t row = (size_t)b * in_stride, orow = (size_t)b * out_stride;
    const uint32_t *rn = res_names + row, *an = atom_names + row;
    const unsigned below = (1u << lane) - 1u;
    const int ntiles = (n + 31) >> 5, per = (ntiles + kTypedScatterWarps - 1) / kTypedScatterWarps;
    const int t0 = min(ntiles, w * per), t1 = min(ntiles, t0 + per);

    if (lane < kTypes) s_cnt[w][lane] = 0;
    __syncthreads();  // the tables' copy and the zeroed counts
    bool bad = false;
    for (int tb = t0; tb < t1; tb += kTypedUnroll) {
        uint32_t r[kTypedUnroll], a[kTypedUnroll];
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            const int j = 32 * (tb + u) + lane;
            const bool in = tb + u < t1 && j < n;
            r[u] = in ? rn[j] : 0u;
            a[u] = in ? an[j] : 0u;
        }
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            const int j = 32 * (tb + u) + lane;
            const bool in = tb + u < t1 && j < n;
            const int t = in ? atom_type(r[u], a[u], s_tab) : -2;  // -1: a name pair the reference rejects
            if (in) s_ty[j] = (signed char)t;
            bad |= t == -1;
            // the lanes of each type: the lowest of them adds their number
            const unsigned m = __match_any_sync(0xffffffffu, t);
            if (t >= 0 && (m & below) == 0u) s_cnt[w][t] += __popc(m);
            __syncwarp();
        }
    }
    if (bad) atomicCAS(&hdr->status, 0u, (unsigned)TPL_ERR_ATOM_TYPE);
    __syncthreads();
    // lane k < kTypes: the type's total, its offset, and this warp's first slot of it
    int tot = 0, before = 0;
    if (lane < kTypes)
#pragma unroll
        for (int v = 0; v < kTypedScatterWarps; v++) {
            const int c = s_cnt[v][lane];
            tot += c;
            before += v < w ? c : 0;
        }
    int inc = tot;
#pragma unroll
    for (int off = 1; off < 16; off <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += v;
    }
    const int type_off = inc - tot;
    if (w == 0 && lane < kTypes) {
        n_of_type[(size_t)b * kTypes + lane] = tot;
        offsets[(size_t)b * kTypes + lane] = type_off;
    }
    if (w == 0 && lane == kTypes - 1) s_ntyped = inc;
    __syncthreads();  // every warp has read the counts
    int *s_next = s_cnt[w];  // reused: this warp's next free slot of each type
    if (lane < kTypes) s_next[lane] = type_off + before;
    __syncwarp();

    for (int tb = t0; tb < t1; tb += kTypedUnroll) {
        T x[kTypedUnroll][3];
        int ty[kTypedUnroll];
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            const int j = 32 * (tb + u) + lane;
            const bool in = tb + u < t1 && j < n;
            const T *src = coords + 3 * (row + j);
#pragma unroll
            for (int c = 0; c < 3; c++) x[u][c] = in ? src[c] : T(0);
            ty[u] = in ? (int)s_ty[j] : -2;
        }
#pragma unroll
        for (int u = 0; u < kTypedUnroll; u++) {
            const int j = 32 * (tb + u) + lane, t = ty[u];
            const unsigned m = __match_any_sync(0xffffffffu, t);
            if (t >= 0) {
                const int slot = s_next[t] + __popc(m & below);
                T *dst = out + 3 * (orow + slot);
                dst[0] = x[u][0];
                dst[1] = x[u][1];
                dst[2] = x[u][2];
                atom_index[orow + slot] = j;
            }
            __syncwarp();
            if (t >= 0 && (m & below) == 0u) s_next[t] += __popc(m);
            __syncwarp();
        }
    }
    __syncthreads();
    // slots past the typed atoms are zero, as in the reference's zero-filled outputs
    const int ntyped = s_ntyped;
    T *o = out + 3 * orow;
    for (int e = 3 * ntyped + threadIdx.x; e < 3 * out_stride; e += 32 * kTypedScatterWarps) o[e] = T(0);
    for (int q = ntyped + threadIdx.x; q < out_stride; q += 32 * kTypedScatterWarps) atom_index[orow + q] = 0;
}

// grad_flat[atom_index[s]] = grad_typed[s] for the typed slots, zero elsewhere;
// grad_flat rows hold in_stride atoms, grad_typed rows out_stride slots.
template <typename T>
__global__ void __launch_bounds__(kTypedThreads) typed_bwd_kernel(const T *grad_typed, T *grad_flat,
                                                                  const int *n_of_type, const int *atom_index,
                                                                  int in_stride, int out_stride) {
    const int b = blockIdx.x, tid = threadIdx.x;
    const size_t row = (size_t)b * in_stride, orow = (size_t)b * out_stride;
    int ntyped = 0;
    for (int k = 0; k < kTypes; k++) ntyped += n_of_type[(size_t)b * kTypes + k];
    ntyped = max(0, min(ntyped, out_stride));
    for (int e = tid; e < 3 * in_stride; e += kTypedThreads) grad_flat[3 * row + e] = T(0);
    __syncthreads();
    for (int s = tid; s < ntyped; s += kTypedThreads) {
        const int j = atom_index[orow + s];
        if (j < 0 || j >= in_stride) continue;
        const T *src = grad_typed + 3 * (orow + s);
        T *dst = grad_flat + 3 * (row + j);
        dst[0] = src[0];
        dst[1] = src[1];
        dst[2] = src[2];
    }
}

// The same with every flat row written once, in order: the slot of each atom is
// first inverted into shared memory (in_stride ints), then grad_flat[j] is gathered
// from grad_typed[slot(j)] with coalesced stores (zero for atoms without a slot).
template <typename T>
__global__ void __launch_bounds__(kTypedThreads) typed_bwd_gather_kernel(const T *__restrict__ grad_typed,
                                                                         T *__restrict__ grad_flat,
                                                                         const int *__restrict__ n_of_type,
                                                                         const int *__restrict__ atom_index,
                                                                         int in_stride, int out_stride) {
    extern __shared__ int s_slot[];
    const int b = blockIdx.x, tid = threadIdx.x;
    const size_t row = (size_t)b * in_stride, orow = (size_t)b * out_stride;
    int ntyped = 0;
    for (int k = 0; k < kTypes; k++) ntyped += n_of_type[(size_t)b * kTypes + k];
    ntyped = max(0, min(ntyped, out_stride));
    for (int j = tid; j < in_stride; j += kTypedThreads) s_slot[j] = -1;
    __syncthreads();
    for (int s = tid; s < ntyped; s += kTypedThreads) {
        const int j = atom_index[orow + s];
        if (j >= 0 && j < in_stride) s_slot[j] = s;
    }
    __syncthreads();
    const T *src = grad_typed + 3 * orow;
    T *dst = grad_flat + 3 * row;
    // eight gathers per thread in flight before their stores (GB300, 4096 chains of
    // 2300 atoms: 0.086 / 0.074 / 0.070 / 0.075 ms with 2 / 4 / 8 / 16)
    constexpr int U = 8;
    const int ne = 3 * in_stride;
    for (int e0 = tid; e0 < ne; e0 += U * kTypedThreads) {
        T v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = e0 + u * kTypedThreads;
            v[u] = T(0);
            if (e < ne) {
                const int j = e / 3, c = e - 3 * j;
                const int s = s_slot[j];
                if (s >= 0) v[u] = src[3 * s + c];
            }
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = e0 + u * kTypedThreads;
            if (e < ne) dst[e] = v[u];
        }
    }
}

constexpr int kGatherMaxAtoms = 16384;  // 64 KB of slots per CTA

}  // namespace

int typed_forward(bool f64, const void *coords, const uint32_t *res_names, const uint32_t *atom_names,
                  const int *num_atoms, int B, int in_stride, int out_stride, void *out, int *n_of_type, int *offsets,
                  int *atom_index, void *ws, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    WsHeader *hdr = reinterpret_cast<WsHeader *>(ws);
    if (in_stride <= kTypedMaxAtoms) {
        auto launch = [&](auto nw, auto *out_t, auto *coords_t) -> int {
            constexpr int NW = decltype(nw)::value;
            using T = std::remove_pointer_t<decltype(out_t)>;
            auto kernel = typed_fwd_group_kernel<T, NW>;
            const size_t smem = typed_smem<T>(in_stride, NW);
            if (!set_max_dynamic_smem(reinterpret_cast<const void *>(kernel), (int)smem)) return TPL_ERR_LAUNCH;
            kernel<<<B, 32 * NW, smem, st>>>(coords_t, res_names, atom_names, num_atoms, in_stride, out_stride, out_t,
                                             n_of_type, offsets, atom_index, hdr);
            return cudaGetLastError() == cudaSuccess ? (int)TPL_OK : (int)TPL_ERR_LAUNCH;
        };
        auto pick = [&](auto *out_t, auto *coords_t) -> int {
            if (in_stride <= kTypedScatterAtoms && B >= 3 * device_sm_count()) {
                using T = std::remove_pointer_t<decltype(out_t)>;
                typed_fwd_scatter_kernel<T><<<B, 32 * kTypedScatterWarps, in_stride, st>>>(
                    coords_t, res_names, atom_names, num_atoms, in_stride, out_stride, out_t, n_of_type, offsets,
                    atom_index, hdr);
                return cudaGetLastError() == cudaSuccess ? (int)TPL_OK : (int)TPL_ERR_LAUNCH;
            }
            // Eight warps per chain for rows past 3500 atoms, where a chain's codes are most of
            // the shared memory and more warps share them, and for batches below four chains per
            // SM; past 16384 atoms four warps' ranks would not fit the codes either.  Eight /
            // four, us: 4096 chains of 2745 atoms 68.4 / 66.2, of 4465 98.2 / 102.7; 256 of 2250
            // 11.7 / 15.3; 512 of 4465 23.8 / 25.6.
            const bool eight = in_stride > 3500 || B < 4 * device_sm_count();
            return eight ? launch(std::integral_constant<int, 8>{}, out_t, coords_t)
                         : launch(std::integral_constant<int, 4>{}, out_t, coords_t);
        };
        return f64 ? pick(static_cast<double *>(out), static_cast<const double *>(coords))
                   : pick(static_cast<float *>(out), static_cast<const float *>(coords));
    }
    // longer chains: one CTA per chain, the types looked up again in the scatter pass
    if (f64)
        typed_fwd_kernel<double><<<B, kTypedThreads, 0, st>>>(
            static_cast<const double *>(coords), res_names, atom_names, num_atoms, in_stride, out_stride,
            static_cast<double *>(out), n_of_type, offsets, atom_index, hdr);
    else
        typed_fwd_kernel<float><<<B, kTypedThreads, 0, st>>>(
            static_cast<const float *>(coords), res_names, atom_names, num_atoms, in_stride, out_stride,
            static_cast<float *>(out), n_of_type, offsets, atom_index, hdr);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

int typed_backward(bool f64, const void *grad_typed, void *grad_flat, const int *n_of_type, const int *atom_index,
                   int B, int in_stride, int out_stride, cudaStream_t st) {
    if (B == 0) return TPL_OK;
    if (in_stride <= kGatherMaxAtoms) {
        const int smem = in_stride * (int)sizeof(int);
        if (f64) {
            auto k = typed_bwd_gather_kernel<double>;
            if (!set_max_dynamic_smem(reinterpret_cast<const void *>(k), smem))
                return TPL_ERR_LAUNCH;
            k<<<B, kTypedThreads, smem, st>>>(static_cast<const double *>(grad_typed), static_cast<double *>(grad_flat),
                                              n_of_type, atom_index, in_stride, out_stride);
        } else {
            auto k = typed_bwd_gather_kernel<float>;
            if (!set_max_dynamic_smem(reinterpret_cast<const void *>(k), smem))
                return TPL_ERR_LAUNCH;
            k<<<B, kTypedThreads, smem, st>>>(static_cast<const float *>(grad_typed), static_cast<float *>(grad_flat),
                                              n_of_type, atom_index, in_stride, out_stride);
        }
        return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
    }
    if (f64)
        typed_bwd_kernel<double><<<B, kTypedThreads, 0, st>>>(static_cast<const double *>(grad_typed),
                                                             static_cast<double *>(grad_flat), n_of_type, atom_index,
                                                             in_stride, out_stride);
    else
        typed_bwd_kernel<float><<<B, kTypedThreads, 0, st>>>(static_cast<const float *>(grad_typed),
                                                            static_cast<float *>(grad_flat), n_of_type, atom_index,
                                                            in_stride, out_stride);
    return cudaGetLastError() == cudaSuccess ? TPL_OK : TPL_ERR_LAUNCH;
}

}  // namespace tpl
