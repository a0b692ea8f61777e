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

// U pieces of 32 letters of chain b's row from letter j0 on, all loads in flight at once;
// 0 past the row.
template <int U, typename T>
__device__ __forceinline__ void load_letters(const A2cArgs<T> &a, int b, int j0, int lane, unsigned char (&c)[U]) {
    const unsigned char *row = a.seq + (size_t)b * a.seq_stride;
#pragma unroll
    for (int u = 0; u < U; u++) {
        const int j = j0 + 32 * u + lane;
        c[u] = j < a.seq_stride ? row[j] : (unsigned char)0;
    }
}

// Length of chain b for the kernels whose warps find it each for itself: the index of
// the row's first NUL (at most the row stride), or 0, with the error recorded, when a
// letter before it is no residue or the chain is longer than L.  atoms(chunk, n) is
// called by the whole warp for every chunk of 32 letters in order, with the atom count of
// this lane's residue.  table: letter -> word with the atom count in bits 8..15, 0 for
// what is no residue.  c: the row's first U pieces (load_letters).
template <int U, typename T, typename Table, typename Atoms>
__device__ __forceinline__ int ring_chain_length(const A2cArgs<T> &a, int b, const Table *table, int lane,
                                                 unsigned char (&c)[U], Atoms atoms) {
    int len = a.seq_stride;
    bool bad = false;
    for (int j0 = 0;;) {
        // votes and lookups of all pieces side by side: none waits for the one before
        uint32_t info[U];
#pragma unroll
        for (int u = U - 1; u >= 0; u--) {
            const unsigned nul = __ballot_sync(0xffffffffu, c[u] == 0);
            info[u] = table[c[u]];
            if (nul != 0u) len = min(a.seq_stride, j0 + 32 * u + __ffs(nul) - 1);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int j1 = j0 + 32 * u;
            const bool in = j1 + lane < len;
            bad |= in && info[u] == 0u;
            if (j1 < len) atoms(j1 >> 5, in ? (int)((info[u] >> 8) & 0xffu) : 0);
        }
        j0 += 32 * U;
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
    unsigned char c[4];
    load_letters(a, b, 0, lane, c);
    return ring_chain_length(a, b, table, lane, c, atoms);
}
// Pieces a kernel asks for before it does anything else: its first chain's length then
// waits for memory once, not once every 128 letters.
constexpr int kFirstLetters = 16;

// float64 launchers (tpl_f64.cu).
int a2c_forward_f64(const A2cArgs<double> &a, int B, bool renorm, cudaStream_t st);
int a2c_backward_f64(const A2cArgs<double> &a, int B, bool renorm, cudaStream_t st);

}  // namespace tpl
