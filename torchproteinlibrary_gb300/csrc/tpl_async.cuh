// Asynchronous copies between global and shared memory for spans of 4-byte words at any
// alignment, shared by the Angles2Backbone and Angles2Coords kernels: whole 16-byte blocks
// move as bulk copies (one instruction of one lane), the words outside them one by one.
// A span is staged at its global 16-byte phase, so both sides of a block are aligned.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace tpl {

__device__ __forceinline__ unsigned smem_addr(const void *p) {
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// Word offset of p inside its 16-byte block.
__device__ __forceinline__ int block_offset(const void *p) { return (int)((reinterpret_cast<uintptr_t>(p) >> 2) & 3u); }

__device__ __forceinline__ void cp_async4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
}

// Orders the generic accesses of the executing thread before later bulk copies.
__device__ __forceinline__ void async_proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

constexpr unsigned kMbarPolls = 1u << 22;  // bounded mbarrier wait (about 0.5 s with the back-off)

__device__ __forceinline__ void mbar_init(uint64_t *bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// Wait for the phase with the given parity to complete; false after kMbarPolls polls.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
    for (unsigned i = 0; i < kMbarPolls; i++) {
        unsigned done;
        asm volatile(
            "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
            : "=r"(done)
            : "r"(smem_addr(bar)), "r"(parity)
            : "memory");
        if (done) return true;
        if (i >= 8) __nanosleep(100);
    }
    return false;
}

// The n words at src and their staging place dst (which has src's 16-byte phase): `head`
// words before the whole blocks, `body` words in them, `tail` words after.
struct StageSpan {
    const float *src;
    float *dst;
    int head, body, tail;
    __device__ __forceinline__ StageSpan(const float *s, float *d, int n) : src(s), dst(d) {
        head = min((4 - block_offset(s)) & 3, n);
        body = (n - head) & ~3;
        tail = n - head - body;
    }
    __device__ __forceinline__ void ends(int lane) const {  // by the warp: cp.async, not committed
        if (lane < head) cp_async4(dst + lane, src + lane);
        if (lane < tail) cp_async4(dst + head + body + lane, src + head + body + lane);
    }
    __device__ __forceinline__ void blocks(uint64_t *bar) const {  // by one lane, counted on *bar
        if (body > 0)
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                             smem_addr(dst + head)),
                         "l"(src + head), "r"(4 * body), "r"(smem_addr(bar))
                         : "memory");
    }
};

// Two spans into shared memory, by the warp; *bar completes a phase when their blocks have
// landed, the words outside them are this lane's cp.async copies.  The buffers' earlier
// readers are done (a __syncwarp before).
__device__ __forceinline__ void stage_spans(const StageSpan &x, const StageSpan &g, uint64_t *bar, int lane) {
    x.ends(lane);
    g.ends(lane);
    if (lane == 0) {
        async_proxy_fence();  // the buffers were last read through the generic proxy
        mbar_expect(bar, 4 * (x.body + g.body));
        x.blocks(bar);
        g.blocks(bar);
    }
}

// Store n words to dst from stg, shared memory at dst's 16-byte phase, written by the whole
// warp before an async_proxy_fence() and a __syncwarp: the whole blocks as one bulk copy by
// lane 0, the words outside them by the first lanes.  The caller waits for the copy's reads
// (bulk_reads_done, lane 0) before the buffer is rewritten or given up.
__device__ __forceinline__ void bulk_store_span(float *dst, const float *stg, int n, int lane) {
    const int head = min((4 - block_offset(dst)) & 3, n), body = (n - head) & ~3, tail = n - head - body;
    if (lane < head) dst[lane] = stg[lane];
    if (lane < tail) dst[head + body + lane] = stg[head + body + lane];
    if (lane == 0 && body > 0)
        asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n"
                     "cp.async.bulk.commit_group;" ::"l"(dst + head),
                     "r"(smem_addr(stg + head)), "r"(4 * body)
                     : "memory");
}
__device__ __forceinline__ void bulk_reads_done() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }

// Zeros to n words from dst, by the warp.
__device__ __forceinline__ void zero_span(void *p, int n, int lane) {
    uint32_t *dst = static_cast<uint32_t *>(p);
    if (n <= 0) return;
    const int head = min((4 - block_offset(dst)) & 3, n), nb = (n - head) >> 2;
    if (lane < head) dst[lane] = 0u;
    for (int i = lane; i < nb; i += 32) __stcs(reinterpret_cast<uint4 *>(dst + head) + i, make_uint4(0u, 0u, 0u, 0u));
    if (lane < n - head - 4 * nb) dst[head + 4 * nb + lane] = 0u;
}

}  // namespace tpl
