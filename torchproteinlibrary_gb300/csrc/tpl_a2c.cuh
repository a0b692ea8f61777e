// Arguments and chain lengths of the Angles2Coords kernels (tpl_a2c.cu, tpl_f64.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "tpl_internal.h"

namespace tpl {

template <typename T>
struct A2cArgs {
    const unsigned char *seq;
    int seq_stride;
    const T *angles;
    T *coords;
    uint32_t *res_names;
    uint32_t *atom_names;
    T *grad_angles;
    const T *grad_coords;
    WsHeader *hdr;
    int L, maxA;
};

__device__ __forceinline__ void a2c_error(WsHeader *h, int code) {
    if (h) atomicCAS(&h->status, 0u, (unsigned)code);
}

// A lane's letters of U blocks of 128 of chain b's row, from letter j0 on: four of each, all
// loads in flight at once; 0 past the row.
template <int U, typename T>
__device__ __forceinline__ void load_letters(const A2cArgs<T> &a, int b, int j0, int lane, unsigned char (&c)[U][4]) {
    const unsigned char *row = a.seq + (size_t)b * a.seq_stride;
#pragma unroll
    for (int v = 0; v < U; v++)
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int j = j0 + 128 * v + 4 * lane + u;
            c[v][u] = j < a.seq_stride ? row[j] : (unsigned char)0;
        }
}

// Length of chain b for the kernels whose warps find it each for itself: the index of
// the row's first NUL (at most the row stride), or 0, with the error recorded, when a
// letter before it is no residue or the chain is longer than L.  A lane looks at four
// letters of every 128, so that a chain costs few instructions; atoms(chunk, n) is called
// by the whole warp for every 128 letters in order, with the number of the first of their
// four chunks of 32 and the atoms of this lane's four residues (lanes 8 g .. 8 g + 7: chunk
// + g).  table: letter -> word with the atom count in bits 8..15, 0 for what is no residue.
// c: the row's first U blocks (load_letters).
template <int U, typename T, typename Table, typename Atoms>
__device__ __forceinline__ int ring_chain_length(const A2cArgs<T> &a, int b, const Table *table, int lane,
                                                 unsigned char (&c)[U][4], Atoms atoms) {
    int len = a.seq_stride;
    bool bad = false;
#pragma unroll 1
    for (int j0 = 0;;) {
#pragma unroll
        for (int v = 0; v < U; v++, j0 += 128) {
            if (j0 >= len) break;
            const int j = j0 + 4 * lane;
            unsigned nul = 0;
#pragma unroll
            for (int u = 0; u < 4; u++) nul |= c[v][u] == 0 ? 1u << u : 0u;
            const unsigned lanes = __ballot_sync(0xffffffffu, nul != 0);
            if (lanes != 0u) {
                const int l = __ffs(lanes) - 1;
                len = min(len, j0 + 4 * l + __ffs(__shfl_sync(0xffffffffu, nul, l)) - 1);
            }
            int n = 0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const unsigned info = j + u < len ? table[c[v][u]] : 0x100u;
                bad |= info == 0u;
                n += j + u < len ? (int)((info >> 8) & 0xffu) : 0;
            }
            atoms(j0 >> 5, n);
        }
        if (j0 >= len) break;
        load_letters(a, b, j0, lane, c);
    }
    bad = __any_sync(0xffffffffu, bad);
    if (bad || len > a.L) {
        if (lane == 0) a2c_error(a.hdr, bad ? TPL_ERR_SEQUENCE : TPL_ERR_LENGTH);
        return 0;
    }
    return len;
}
template <typename T, typename Table, typename Atoms>
__device__ __forceinline__ int ring_chain_length(const A2cArgs<T> &a, int b, const Table *table, int lane,
                                                 Atoms atoms) {
    unsigned char c[1][4];
    load_letters(a, b, 0, lane, c);
    return ring_chain_length(a, b, table, lane, c, atoms);
}
// Blocks a kernel asks for before it does anything else: its first chain's length then
// waits for memory once, not once every 128 letters.
constexpr int kFirstLetters = 4;

// float64 launchers (tpl_f64.cu).
int a2c_forward_f64(const A2cArgs<double> &a, int B, bool renorm, cudaStream_t st);
int a2c_backward_f64(const A2cArgs<double> &a, int B, bool renorm, cudaStream_t st);

}  // namespace tpl
