// Inline-PTX helpers shared by the staged kernels: mbarriers, bulk copies, explicit shared-memory
// loads, the rANS decode step and the bf16 packing of decoded weights.
#pragma once
#include "common.cuh"

namespace ci {

constexpr uint32_t kWaitPolls = 1u << 22;   // mbarrier polls before a wait gives up
constexpr uint32_t kLutBytes = kProbScale * 4;

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok;
}
// 1-D bulk copy global -> this CTA's own shared memory, 16-byte aligned, size % 16 == 0.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
// All cp.async issued so far by this thread have landed (for the other lanes of the warp behind a __syncwarp).
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// The mbarrier gets one arrival when all cp.async issued so far by this thread have landed.
__device__ __forceinline__ void cp_async_arrive(uint32_t bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_async_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void ldmatrix_x4(uint32_t addr, uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
                 : "r"(addr));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&x)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(x[0]), "r"(x[1]), "r"(x[2]), "r"(x[3]), "r"(b0), "r"(b1));
}

// bf16 bits of one weight from its table entry (symbol in bits 19..12) and sign+mantissa byte.
__device__ __forceinline__ uint32_t weight_bits(uint32_t entry, uint32_t man) {
    return ((entry >> 5) & 0x7F80u) | ((man & 0x80u) << 8) | (man & 0x7Fu);
}
// Two weights (rows k, k+1 of one column) as a packed bf16 pair, five instructions:
// both symbols are brought to bits 14..7 / 30..23 with one byte permute, both
// sign+mantissa bytes are doubled into their halves with another, one bit-select merges.
__device__ __forceinline__ uint32_t weight_pair(uint32_t e_lo, uint32_t e_hi, uint32_t m_lo, uint32_t m_hi) {
    const uint32_t ee = __byte_perm(e_lo >> 5, e_hi << 11, 0x7610);
    const uint32_t vv = __byte_perm(m_lo, m_hi, 0x4400);
    return (ee & 0x7F807F80u) | (vv & 0x807F807Fu);
}

// Exponent bits of a packed bf16 pair from ee, the rest from vv: a bit-select, which the compiler makes two instructions of.
__device__ __forceinline__ uint32_t exp_or_man(uint32_t ee, uint32_t vv) {
    uint32_t w;
    asm("lop3.b32 %0, %1, %2, %3, 0xE4;" : "=r"(w) : "r"(ee), "r"(vv), "n"(0x7F807F80));
    return w;
}

__device__ __forceinline__ uint32_t lds_u32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds_u8(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}

// One symbol with the table at shared address lut_s.
__device__ __forceinline__ uint32_t decode_fast(uint32_t &state, uint32_t lut_s) {
    const uint32_t e = lds_u32(lut_s + ((state & kProbMask) << 2));
    state = (e >> 20) * (state >> kProbBits) + (e & 0xFFFu);
    return e;
}
// The same with the table on a 16 KB boundary of the shared window: the entry's address needs no addition.
__device__ __forceinline__ uint32_t decode_aligned(uint32_t &state, uint32_t lut_s) {
    const uint32_t e = lds_u32(((state << 2) & ((kProbScale - 1) << 2)) | lut_s);
    state = (e >> 20) * (state >> kProbBits) + (e & 0xFFFu);
    return e;
}
// Renormalisation, STRIDE bytes between the rows of a stream.
//
// No lower-bound test anywhere in this family: a well-formed stream always has a byte left when its
// state is below 2^16, and the launchers guarantee enough mapped shared memory below every window
// that a malformed stream reads garbage instead of faulting.
//
// renorm_spec: exact.  The first byte is loaded by the caller before the state update is known to
// need it (its address does not depend on the new state, and some lane of the warp needs it on
// nearly every step anyway), which takes one shared-memory latency off the decode chain.  A second
// byte is needed exactly when the state before renormalisation is below 2^8, so its test and load
// do not wait for the first byte either.
template <uint32_t STRIDE>
__device__ __forceinline__ void renorm_spec(uint32_t &state, uint32_t &pos, uint32_t first) {
    asm volatile(
        "{\n\t.reg .pred p1, p2;\n\t.reg .u32 b;\n\t"
        "setp.lt.u32 p1, %0, 65536;\n\t"
        "setp.lt.u32 p2, %0, 256;\n\t"
        "@p2 ld.shared.u8 b, [%1+-%3];\n\t"
        "@p1 mad.lo.u32 %0, %0, 256, %2;\n\t"
        "@p1 sub.u32 %1, %1, %3;\n\t"
        "@p2 mad.lo.u32 %0, %0, 256, b;\n\t"
        "@p2 sub.u32 %1, %1, %3;\n\t}"
        : "+r"(state), "+r"(pos)
        : "r"(first), "n"(STRIDE));
}
template <uint32_t STRIDE>
__device__ __forceinline__ void renorm_fast(uint32_t &state, uint32_t &pos) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .u32 b;\n\t"
        "setp.lt.u32 p, %0, 65536;\n\t"
        "@p ld.shared.u8 b, [%1];\n\t"
        "@p mad.lo.u32 %0, %0, 256, b;\n\t"
        "@p sub.u32 %1, %1, %2;\n\t}"
        : "+r"(state), "+r"(pos)
        : "n"(STRIDE));
}

// Four streams of one lane whose bytes are the four byte columns of one word column (rows 128 bytes apart).
//
// step() decodes one symbol of each stream and returns the table entries.  The next byte of every stream is loaded
// before it is known to be needed (its address does not depend on the new state, and some lane needs it on nearly
// every step), which takes one shared-memory latency off the decode chain; about one symbol in three merges it, under
// a predicate.  A second byte is needed only after a symbol of frequency below 16: one test for the four streams, one
// branch.  The whole renormalisation is one asm block so that the rare branch updates the registers in place; with the
// branch in C++ the compiler copies all eight of them on the common path (2 of 22 instructions per symbol).
//
// step_together(): the whole warp takes that branch or does not, by a vote on a test that does not wait for the first bytes
// (the state before them is below 2^8).  Where tensor instructions follow, lanes that part in every step have to be brought
// together again: in a loop of steps, packing and mma alone one warp a scheduler took 211 cycles a step and takes 166,
// 16 warps 378 and 359.  Without such instructions there is little in it: the decoders take 0.5 to 1.6 % longer with it, the
// gather between 2 % less (few ids, or entry points) and 1 % more (tile height 16).  Second bytes under predicates instead of a
// branch: 403 at 16 warps.
//
// step_ahead(): both bytes are loaded before they are known to be needed and merged under predicates: the shortest chain, for
// launches of so few warps that nothing else happens meanwhile.  In that loop one warp a scheduler takes 131 cycles a step, but
// 16 warps 403.
struct Quad {
    uint32_t s[4], p[4];                                        // states, shared addresses of the next bytes

    __device__ __forceinline__ void start(uint32_t states_s, uint32_t first) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            s[j] = lds_u32(states_s + 4 * j);
            p[j] = first + j;
        }
    }
    __device__ __forceinline__ void step(uint32_t lut_s, uint32_t (&e)[4]) {
        uint32_t y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = lds_u8(p[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = decode_aligned(s[j], lut_s);
        asm volatile(
            "{\n\t.reg .pred p0, p1, p2, p3, r;\n\t.reg .u32 m0, m1;\n\t"
            "setp.lt.u32 p0, %0, 65536;\n\t"
            "setp.lt.u32 p1, %1, 65536;\n\t"
            "setp.lt.u32 p2, %2, 65536;\n\t"
            "setp.lt.u32 p3, %3, 65536;\n\t"
            "@p0 mad.lo.u32 %0, %0, 256, %8;\n\t"
            "@p1 mad.lo.u32 %1, %1, 256, %9;\n\t"
            "@p2 mad.lo.u32 %2, %2, 256, %10;\n\t"
            "@p3 mad.lo.u32 %3, %3, 256, %11;\n\t"
            "@p0 sub.u32 %4, %4, 128;\n\t"
            "@p1 sub.u32 %5, %5, 128;\n\t"
            "@p2 sub.u32 %6, %6, 128;\n\t"
            "@p3 sub.u32 %7, %7, 128;\n\t"
            "min.u32 m0, %0, %1;\n\t"
            "min.u32 m1, %2, %3;\n\t"
            "min.u32 m0, m0, m1;\n\t"
            "setp.lt.u32 r, m0, 65536;\n\t"
            "@!r bra DONE;\n\t"
            "setp.lt.u32 p0, %0, 65536;\n\t"
            "setp.lt.u32 p1, %1, 65536;\n\t"
            "setp.lt.u32 p2, %2, 65536;\n\t"
            "setp.lt.u32 p3, %3, 65536;\n\t"
            "@p0 ld.shared.u8 m0, [%4];\n\t"
            "@p0 mad.lo.u32 %0, %0, 256, m0;\n\t"
            "@p0 sub.u32 %4, %4, 128;\n\t"
            "@p1 ld.shared.u8 m0, [%5];\n\t"
            "@p1 mad.lo.u32 %1, %1, 256, m0;\n\t"
            "@p1 sub.u32 %5, %5, 128;\n\t"
            "@p2 ld.shared.u8 m0, [%6];\n\t"
            "@p2 mad.lo.u32 %2, %2, 256, m0;\n\t"
            "@p2 sub.u32 %6, %6, 128;\n\t"
            "@p3 ld.shared.u8 m0, [%7];\n\t"
            "@p3 mad.lo.u32 %3, %3, 256, m0;\n\t"
            "@p3 sub.u32 %7, %7, 128;\n\t"
            "DONE:\n\t}"
            : "+r"(s[0]), "+r"(s[1]), "+r"(s[2]), "+r"(s[3]), "+r"(p[0]), "+r"(p[1]), "+r"(p[2]), "+r"(p[3])
            : "r"(y[0]), "r"(y[1]), "r"(y[2]), "r"(y[3]));
    }
    __device__ __forceinline__ void step_together(uint32_t lut_s, uint32_t (&e)[4]) {
        uint32_t y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = lds_u8(p[j]);
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = decode_aligned(s[j], lut_s);
        const uint32_t low = min(min(s[0], s[1]), min(s[2], s[3]));
#pragma unroll
        for (int j = 0; j < 4; ++j)
            asm("{\n\t.reg .pred p;\n\t"
                "setp.lt.u32 p, %0, 65536;\n\t"
                "@p mad.lo.u32 %0, %0, 256, %2;\n\t"
                "@p sub.u32 %1, %1, 128;\n\t}"
                : "+r"(s[j]), "+r"(p[j])
                : "r"(y[j]));
        if (__any_sync(kFull, low < 256u)) {
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = lds_u8(p[j]);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                asm volatile("{\n\t.reg .pred p;\n\t"
                             "setp.lt.u32 p, %0, 65536;\n\t"
                             "@p mad.lo.u32 %0, %0, 256, %2;\n\t"
                             "@p sub.u32 %1, %1, 128;\n\t}"
                             : "+r"(s[j]), "+r"(p[j])
                             : "r"(y[j]));
        }
    }
    __device__ __forceinline__ void step_ahead(uint32_t lut_s, uint32_t (&e)[4]) {
        uint32_t y[4], v[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            y[j] = lds_u8(p[j]);
            v[j] = lds_u8(p[j] - 128);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) e[j] = decode_aligned(s[j], lut_s);
#pragma unroll
        for (int j = 0; j < 4; ++j)
            asm("{\n\t.reg .pred p, q;\n\t"
                "setp.lt.u32 p, %0, 65536;\n\t"
                "setp.lt.u32 q, %0, 256;\n\t"
                "@p mad.lo.u32 %0, %0, 256, %2;\n\t"
                "@p sub.u32 %1, %1, 128;\n\t"
                "@q mad.lo.u32 %0, %0, 256, %3;\n\t"
                "@q sub.u32 %1, %1, 128;\n\t}"
                : "+r"(s[j]), "+r"(p[j])
                : "r"(y[j]), "r"(v[j]));
    }
    // Streams of columns that do not exist (`cols` of the four do) run along with the first one.  Their own would start at
    // 2^16 over zero bytes: a symbol of frequency 1 at every step, and with it the branch for a second byte.
    __device__ __forceinline__ void keep(uint32_t cols) {
#pragma unroll
        for (uint32_t j = 1; j < 4; ++j)
            if (j >= cols) {
                s[j] = s[0];
                p[j] = p[0];
            }
    }
    // Keeps a malformed stream's cursors within reach of the window at `low`: call it at least every 32 symbols.
    __device__ __forceinline__ void clamp(uint32_t low) {
#pragma unroll
        for (int j = 0; j < 4; ++j) p[j] = max(p[j], low);
    }
};

__device__ __forceinline__ void sts_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// Every lane polls an mbarrier phase itself, bounded.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok = 0;
    for (uint32_t it = 0; it < kWaitPolls && !ok; ++it) ok = mbar_try_wait(bar, parity);
    return ok != 0;
}

// The decode table into shared memory at lut_s: a prepared one by one bulk copy that nobody waits for until the first
// look-up (start_lut by thread 0 before the CTA's first barrier, wait_lut by every thread behind it), otherwise built on
// the spot.
__device__ __forceinline__ void start_lut(uint32_t lut_s, uint32_t bar, const uint32_t *lut) {
    if (threadIdx.x == 0 && lut != nullptr) {
        mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        fence_async_proxy();
        mbar_expect_tx(bar, kLutBytes);
        bulk_load(lut_s, lut, kLutBytes, bar);
    }
}
__device__ __forceinline__ bool wait_lut(uint32_t bar, const uint32_t *lut) { return lut == nullptr || mbar_wait(bar, 0); }

// A span of an entry point (first row | rows << 16): moves `off` from the tile's byte block to the span and returns its rows, or
// more than any window holds where it reaches beyond the tile's `depth` rows -- entry points made of other arrays than these --
// so that the copy is refused like that of any wrong depth.
__device__ __forceinline__ uint32_t enter_span(uint32_t span, uint32_t depth, uint32_t &off) {
    const uint32_t first = span & 0xFFFFu, rows = span >> 16;
    off += first * 64;
    return first + rows <= depth ? rows : 0xFFFFFFFFu;
}

// Sign+mantissa bytes on their way through a warp that decodes four segments (two tiles, both halves) at once: chunks of
// kChunkRows rows of 32 bytes per segment, double buffered.  The segments of a chunk start 8 banks apart, so a row of
// the warp's 128 columns is one conflict-free wavefront.
constexpr uint32_t kChunkRows = 16;
constexpr uint32_t kSegPitch = kChunkRows * 32 + 32;
constexpr uint32_t kManBytes = 2 * 4 * kSegPitch;
// Cost model of the persistent kernels' launches, in us at 64 symbols per stream.  A round of units -- every one of w warps
// takes one -- lasts 2.6 + 0.7 x warps, where a scheduler with a warp more than the others counts half (measured in full
// rounds of the fused linear: 12 warps 11.2, 14 13.1, 16 13.7, 19 16.4; two warps a scheduler 9, one 7.4).
// `extra` is what a round of more than 16 warps costs on top, where they have fewer registers or a pipe is full already.
inline double round_cost(uint32_t w, double extra) {
    if (w <= 4) return 7.4;
    if (w <= 8) return 9.0;
    return 2.6 + 0.35 * (w + (w + 3) / 4 * 4) + (w > 16 ? extra : 0.0);
}
// `units` units on a multiprocessor with w warps: full rounds, then what is left on fewer warps.
inline double run_cost(uint32_t units, uint32_t w, double extra) {
    const double tail = units % w ? round_cost(units % w, extra) : 0.0;
    return (units / w) * round_cost(w, extra) + tail;
}

// Lane 0 polls an mbarrier phase, bounded; the verdict is broadcast to the warp.
__device__ __forceinline__ bool mbar_wait_warp(uint32_t bar, uint32_t parity) {
    uint32_t ok = 0;
    if (lane_id() == 0)
        for (uint32_t it = 0; it < kWaitPolls && !ok; ++it) ok = mbar_try_wait(bar, parity);
    return __shfl_sync(kFull, ok, 0) != 0;
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

}  // namespace ci
