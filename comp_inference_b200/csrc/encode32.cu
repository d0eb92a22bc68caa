// GPU rANS encoder for 32-wide tiles: bf16 weight (or exponent plane) -> packed tiled stream, one encoding pass.
//
// Replaces, for the format's own tile width, the two counting / writing passes of encode.cu and everything around them
// (split into planes, two device-to-host waits, table uploads; the reference: src/cuda/rans_kernels.cuh:76-188,
// src/cuda/rans_ops.cu:328-370).  Steps, all queued before the one wait:
//   1. k_exp_histogram     exponent (and optionally sign+mantissa) histogram of the bf16 weight
//   2. k_make_tables       the 12-bit frequency rule, cumulative table, slot map and the encoder's own table, on the GPU
//   3. k_encode32          one lane = one or two columns: reads the weight, writes the tiled sign+mantissa bytes and
//                          encodes; bytes are collected four at a time and stored as [tile][word][64 streams] words
//   4. k_scan_tiles        tile offsets from the deepest stream of every tile
//   -- wait: stream length, frequencies --
//   5. k_pack32            shifts every stream to the bottom of its tile and interleaves the bytes into the stream
//
// Encoding reads 2 bytes and writes 1 + 0.35 bytes per weight; what bounds it is the chain of each stream and the
// instructions around it (about 25 per symbol), not memory.  Division by the frequency is a multiplication by
// m = ceil(2^(32+s) / f), s = ceil(log2 f) - 1, and a shift: exact for states below 2^24 because
// m f - 2^(32+s) < f <= 2^(s+1) (Granlund and Montgomery, "Division by Invariant Integers using Multiplication").
//
// Measured, 4096 x 11008 at tile height 128 through compress_weight_cuda on a B200: 1650 us (and up to 6000 when the
// stream-ordered allocator returned its memory) -> 162, of which the encoder itself 78, the histogram 20, packing 11; with pointers that
// step from row to row instead of a 64-bit product for each, the encoder 64; with the kernels launched ahead of the end of the
// one before and the depths cleared beside the tables, 141 in all, and 2048 x 2048 84 -> 68.
#include <type_traits>

#include "common.cuh"

namespace ci {

constexpr uint32_t kEncHead = 16384;         // scratch: histograms, encoder table, results; then the stream words
constexpr uint32_t kOffManHist = 2048, kOffEncTab = 4096, kOffResult = 8192;

struct EncResult {                           // copied to the host in one piece
    unsigned long long total;
    uint16_t freqs[256], cdf[256];
    unsigned long long man_hist[256];
};

// Words of one stream's slot: a symbol costs at most 12 bits plus log2(1 + 1/16) of rounding.
__host__ __device__ inline uint32_t stream_words(uint32_t half) { return (half * 3 / 2 + half / 32 + 8 + 3) / 4; }

// Every kernel behind the first is launched with programmatic dependent launch: it waits here until the one before has finished,
// and lets the next one be scheduled.
__device__ __forceinline__ void behind_previous() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
template <class... Params, class... Args>
static int launch_behind(void (*kernel)(Params...), uint32_t blocks, uint32_t threads, cudaStream_t s, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CI_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
    return CI_OK;
}

// ---------------------------------------------------------------- 1. histogram

// Counters [bin][lane]: a warp's increments never meet in a bank, however few different symbols there are.
template <bool MAN>
__global__ void __launch_bounds__(512) k_exp_histogram(const uint16_t *__restrict__ w, uint64_t n, unsigned long long *hist,
                                                       unsigned long long *man_hist) {
    extern __shared__ uint32_t s_cnt[];                         // [256][32], with MAN twice
    behind_previous();
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t i = threadIdx.x; i < 8192 * (MAN ? 2 : 1); i += blockDim.x) s_cnt[i] = 0;
    __syncthreads();
    auto count = [&](uint32_t raw) {
        atomicAdd(&s_cnt[((raw >> 7) & 0xFFu) * 32 + lane], 1u);
        if (MAN) atomicAdd(&s_cnt[8192 + (((raw >> 8) & 0x80u) | (raw & 0x7Fu)) * 32 + lane], 1u);
    };
    const uint64_t vec = (reinterpret_cast<uintptr_t>(w) & 15u) ? 0 : n / 8, step = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint4 *src = reinterpret_cast<const uint4 *>(w);
    for (uint64_t i = first; i < vec; i += step) {
        const uint4 v = src[i];
        const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            count(u[j] & 0xFFFFu);
            count(u[j] >> 16);
        }
    }
    for (uint64_t i = vec * 8 + first; i < n; i += step) count(w[i]);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < (MAN ? 512u : 256u); b += blockDim.x) {
        uint32_t sum = 0;
        for (uint32_t l = 0; l < 32; ++l) sum += s_cnt[b * 32 + ((l + b) & 31)];
        if (sum) atomicAdd(b < 256 ? &hist[b] : &man_hist[b - 256], (unsigned long long)sum);
    }
}

// ---------------------------------------------------------------- 2. tables

__device__ __forceinline__ uint4 encoder_entry(uint32_t f, uint32_t start) {
    // {m, start (+ 4095 where m stands for a division by one: it yields x - 1), (4096 - f) << 5 | s, first state too large}
    if (f == 1) return make_uint4(0xFFFFFFFFu, start + 4095u, 4095u << 5, 1u << 12);
    const uint32_t s = 31 - __clz(f - 1);
    const uint32_t m = (uint32_t)(((1ull << (32 + s)) + f - 1) / f);
    return make_uint4(m, start, (4096u - f) << 5 | s, f << 12);
}

// Block 0: tables.  hist != null: the frequency rule of ci_normalize_freqs; null: frequencies are in res already.  The other blocks
// clear the tiles' depths, which the encoder takes the maximum into: block 0 alone would take 100000 x 1024 at tile height 16
// (200000 tiles) from 402 us to 414.
__global__ void __launch_bounds__(256) k_make_tables(const unsigned long long *hist, const unsigned long long *man_hist,
                                                     EncResult *res, uint4 *enc, uint32_t *tables, uint8_t *slot_map,
                                                     uint32_t *max_lens, uint32_t tiles) {
    __shared__ uint32_t s_f[256], s_c[256];
    __shared__ unsigned long long s_tot[8];
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    behind_previous();
    if (blockIdx.x != 0) {
        for (uint32_t i = (blockIdx.x - 1) * 256 + t; i < tiles; i += (gridDim.x - 1) * 256) max_lens[i] = 0;
        return;
    }
    if (hist != nullptr) {
        unsigned long long h = hist[t], sum = h;
        for (int d = 16; d; d >>= 1) sum += __shfl_xor_sync(kFull, sum, d);
        if (lane == 0) s_tot[warp] = sum;
        __syncthreads();
        sum = 0;
        for (int i = 0; i < 8; ++i) sum += s_tot[i];
        // floor(h / total * 4096) in double precision, zeros -> 1 (comp_inference/comp_inference.py:197-198)
        uint32_t f = (uint32_t)floor(__dmul_rn(__ddiv_rn((double)h, (double)sum), 4096.0));
        s_f[t] = f ? f : 1;
        if (man_hist) res->man_hist[t] = man_hist[t];
        __syncthreads();
        if (warp == 0) {
            // A surplus goes to the largest frequency (ties: the lowest symbol).  A deficit is taken one unit at a time from
            // whichever is largest then (comp_inference/comp_inference.py:204-227): that levels everything above some v
            // down to v, and the units that are left come off the first symbols at that level.
            uint32_t v[8], total = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                v[j] = s_f[lane * 8 + j];
                total += v[j];
            }
            total = __reduce_add_sync(kFull, total);
            if (total < 4096u) {
                uint32_t top = 0;                               // value << 8 | 255 - symbol
#pragma unroll
                for (int j = 0; j < 8; ++j) top = max(top, v[j] << 8 | (255 - (lane * 8 + j)));
                top = __reduce_max_sync(kFull, top);
                if (lane == 0) s_f[255 - (top & 255u)] += 4096u - total;
            } else if (total > 4096u) {
                const uint32_t need = total - 4096u;
                auto above = [&](uint32_t level) {
                    uint32_t sum = 0;
#pragma unroll
                    for (int j = 0; j < 8; ++j) sum += v[j] > level ? v[j] - level : 0u;
                    return __reduce_add_sync(kFull, sum);
                };
                uint32_t level = 0;                             // the smallest with above(level) <= need
                for (uint32_t d = 4096; d; d >>= 1)
                    if (above(level + d - 1) > need) level += d;
                uint32_t left = need - above(level), at = 0;
#pragma unroll
                for (int j = 0; j < 8; ++j) at += v[j] >= level;
                uint32_t rank = at;                             // symbols at the level in lower lanes
                for (int d = 1; d < 32; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(kFull, rank, d);
                    if (lane >= d) rank += o;
                }
                rank -= at;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    uint32_t f = min(v[j], level);
                    if (v[j] >= level && rank++ < left) --f;
                    s_f[lane * 8 + j] = f;
                }
            }
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t v[8], sum8 = 0;
#pragma unroll
            for (int j = 0; j < 8; ++j) { v[j] = s_f[lane * 8 + j]; sum8 += v[j]; }
            uint32_t run = sum8;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(kFull, run, d);
                if (lane >= d) run += o;
            }
            run -= sum8;
#pragma unroll
            for (int j = 0; j < 8; ++j) { s_c[lane * 8 + j] = run; run += v[j]; }
        }
        __syncthreads();
        res->freqs[t] = (uint16_t)s_f[t];
        res->cdf[t] = (uint16_t)s_c[t];
    } else {
        s_f[t] = res->freqs[t];
        s_c[t] = res->cdf[t];
    }
    __syncthreads();
    enc[t] = encoder_entry(s_f[t], s_c[t]);
    if (tables) tables[t] = s_f[t] | (s_c[t] << 16);
    if (slot_map)
        for (uint32_t s = t; s < kProbScale; s += 256) {        // last symbol whose range starts at or below the slot
            uint32_t a = 0;
            for (uint32_t d = 128; d; d >>= 1)
                if (s_c[a + d] <= s) a += d;
            slot_map[s] = (uint8_t)a;
        }
}

// ---------------------------------------------------------------- 3. encoder

struct Enc32Args {
    const void *src;                         // bf16 [K][N], or the exponent plane u8 [K][N]
    uint32_t K, N, th, half, tiles_n, tiles_k;
    uint8_t *mantissa;                       // tiled, or null
    uint32_t *states, *sizes, *max_lens;     // max_lens zeroed before
    uint32_t *words;                         // [tiles][stream_words][64]
    uint32_t cap_words;
    const uint4 *table;
};

// One stream: state, the last bytes emitted (newest in the low byte), their number, and its first word.
struct Chain {
    uint32_t x, acc, n;
    uint32_t *base;

    // Encodes one symbol.  Written with predicates: as branches the emission costs 20 of 44 instructions per symbol in
    // reconvergence and 64-bit pointers.  A byte leaves about one symbol in three; a second one only before symbols of
    // frequency below 16.  The slot of stream_words() words always suffices: every symbol multiplies the state by at
    // most 4096 (1 + 1/16) and every byte divides it by 256.
    __device__ __forceinline__ void put(const uint4 e) {
        asm volatile(
            "{\n\t.reg .pred p, q, r;\n\t.reg .u32 t;\n\t.reg .u64 a;\n\t"
            "setp.ge.u32 p, %0, %4;\n\t"
            "@p prmt.b32 %1, %1, %0, 0x2104;\n\t"             // acc << 8 | x & 0xFF
            "@p shr.u32 %0, %0, 8;\n\t"
            "@p add.u32 %2, %2, 1;\n\t"
            "and.b32 t, %2, 3;\n\t"
            "setp.eq.and.u32 q, t, 0, p;\n\t"
            "@q mad.wide.u32 a, %2, 64, %3;\n\t"
            "@q st.global.u32 [a+-256], %1;\n\t"
            "setp.ge.u32 r, %0, %4;\n\t"
            "@!r bra DONE;\n\t"
            "prmt.b32 %1, %1, %0, 0x2104;\n\t"
            "shr.u32 %0, %0, 8;\n\t"
            "add.u32 %2, %2, 1;\n\t"
            "and.b32 t, %2, 3;\n\t"
            "setp.eq.u32 q, t, 0;\n\t"
            "@q mad.wide.u32 a, %2, 64, %3;\n\t"
            "@q st.global.u32 [a+-256], %1;\n\t"
            "DONE:\n\t}"
            : "+r"(x), "+r"(acc), "+r"(n)
            : "l"(base), "r"(e.w)
            : "memory");
        const uint32_t q = __funnelshift_r(__umulhi(x, e.x), 0u, e.z);   // the shift is e.z mod 32
        x = q * (e.z >> 5) + (x + e.y);                         // x / f * 4096 + x % f + start
    }
    __device__ __forceinline__ void finish() {
        if (n & 3u) base[(n >> 2) * 64] = acc << (8 * (4 - (n & 3u)));
    }
};

// One warp takes one half (top or bottom streams) of COLS neighbouring tiles, a lane one or two columns.  Rows are taken
// last first, four at a time, loaded one batch ahead of the chains.  (Both halves in one lane, twice the independent
// chains and half the warps, was slower: 95 to 141 us against 80 for 4096 x 11008.)
// Warps of a block: 4096 x 11008 65 us with eight, 64 with four; one column a lane, 2048 x 2048, 9.7 and 10.2.
template <int COLS>
constexpr uint32_t kEncWarps = COLS == 2 ? 4 : 8;

template <int COLS, bool PLANE>
__global__ void __launch_bounds__(kEncWarps<COLS> * 32, 32 / kEncWarps<COLS>) k_encode32(const __grid_constant__ Enc32Args a) {
    __shared__ uint4 s_tab[256];
    behind_previous();
    for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) s_tab[i] = a.table[i];
    __syncthreads();
    const uint32_t lane = lane_id(), per_row = (a.tiles_n + COLS - 1) / COLS * 2;
    const uint32_t gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (gw >= per_row * a.tiles_k) return;
    const uint32_t tk = gw / per_row, rem = gw - tk * per_row, strip = rem >> 1, h = rem & 1;
    const uint32_t col = strip * (32 * COLS) + lane * COLS;     // first column of this lane
    const uint32_t tn = strip * COLS + (COLS == 2 ? lane >> 4 : 0), c = col & 31;
    const bool live = col < a.N, in_tile = tn < a.tiles_n;
    const size_t t = (size_t)tk * a.tiles_n + tn;

    Chain z[COLS];
#pragma unroll
    for (int j = 0; j < COLS; ++j) {
        z[j].x = kRansL;
        z[j].acc = z[j].n = 0;
        z[j].base = a.words + t * a.cap_words * 64 + h * 32 + c + j;
    }
    const uint32_t row0 = tk * a.th + h * a.half;
    if (live && row0 < a.K) {
        constexpr int kBatch = 4;
        using Src = std::conditional_t<PLANE, uint8_t, uint16_t>;
        uint32_t i = min(a.half, a.K - row0);                   // rows left
        const Src *src = static_cast<const Src *>(a.src) + (size_t)(row0 + i) * a.N + col;      // one row behind the next
        uint8_t *man = a.mantissa + t * a.th * 32 + ((size_t)h * a.half + i) * 32 + c;
        const size_t pitch = a.N;
        auto fetch = [&]() -> uint32_t {                        // the symbols of the lane's columns, a row further up
            src -= pitch;
            if constexpr (COLS == 2) {
                if constexpr (PLANE) return *reinterpret_cast<const uint16_t *>(src);
                else return *reinterpret_cast<const uint32_t *>(src);
            } else {
                return *src;
            }
        };
        auto code = [&](int up, uint32_t w) {                   // `up` rows above man
            if constexpr (PLANE) {
                z[0].put(s_tab[w & 0xFFu]);
                if constexpr (COLS == 2) z[1].put(s_tab[w >> 8]);
            } else {
                const uint32_t m = ((w >> 8) & 0x00800080u) | (w & 0x007F007Fu);
                uint8_t *dst = man - up * 32;
                if constexpr (COLS == 2) *reinterpret_cast<uint16_t *>(dst) = (uint16_t)__byte_perm(m, 0u, 0x4420);
                else *dst = (uint8_t)m;
                z[0].put(s_tab[(w >> 7) & 0xFFu]);
                if constexpr (COLS == 2) z[1].put(s_tab[(w >> 23) & 0xFFu]);
            }
        };
        for (; i % kBatch; --i) {
            code(1, fetch());
            man -= 32;
        }
        if (i) {
            uint32_t w[kBatch], nx[kBatch];
#pragma unroll
            for (int r = 0; r < kBatch; ++r) w[r] = fetch();
            for (; i; i -= kBatch) {
                if (i > kBatch) {
#pragma unroll
                    for (int r = 0; r < kBatch; ++r) nx[r] = fetch();
                }
#pragma unroll
                for (int r = 0; r < kBatch; ++r) code(r + 1, w[r]);
                man -= 32 * kBatch;
#pragma unroll
                for (int r = 0; r < kBatch; ++r) w[r] = nx[r];
            }
        }
    }
    uint32_t deepest = 0;
#pragma unroll
    for (int j = 0; j < COLS; ++j) {
        if (in_tile) {
            z[j].finish();
            const size_t sid = t * 64 + h * 32 + c + j;
            a.states[sid] = z[j].x;
            a.sizes[sid] = z[j].n;
        }
        deepest = max(deepest, z[j].n);
    }
#pragma unroll
    for (int d = COLS == 2 ? 8 : 16; d; d >>= 1) deepest = max(deepest, __shfl_xor_sync(kFull, deepest, d));
    if ((lane & (COLS == 2 ? 15 : 31)) == 0 && in_tile) atomicMax(a.max_lens + t, deepest);
}

// ---------------------------------------------------------------- 4. offsets

// Exclusive scan of 64 x max_lens by one block, 16384 tiles a pass; the 64-bit total goes to the overflow check.
__global__ void __launch_bounds__(1024) k_scan_tiles(const uint32_t *__restrict__ max_lens, uint32_t tiles,
                                                     uint32_t *__restrict__ offsets, EncResult *res) {
    __shared__ unsigned long long s_warp[33];
    behind_previous();
    const uint32_t t = threadIdx.x, lane = t & 31, warp = t >> 5;
    unsigned long long base = 0;
    for (uint32_t first = 0; first < tiles; first += 16384) {
        uint32_t v[4][4];                                       // tile first + 4096 k + 4 t + j
        unsigned long long run, mine;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t at = first + 4096 * k + 4 * t;
#pragma unroll
            for (int j = 0; j < 4; ++j) v[k][j] = at + j < tiles ? max_lens[at + j] * 64u : 0u;
        }
        for (int k = 0; k < 4 && first + 4096 * k < tiles; ++k) {
            mine = (unsigned long long)v[k][0] + v[k][1] + v[k][2] + v[k][3];
            run = mine;
            for (int d = 1; d < 32; d <<= 1) {
                const unsigned long long o = __shfl_up_sync(kFull, run, d);
                if (lane >= d) run += o;
            }
            if (lane == 31) s_warp[warp] = run;
            __syncthreads();
            if (warp == 0) {
                const unsigned long long own = s_warp[lane];
                unsigned long long w = own;
                for (int d = 1; d < 32; d <<= 1) {
                    const unsigned long long o = __shfl_up_sync(kFull, w, d);
                    if (lane >= d) w += o;
                }
                s_warp[lane] = w - own;
                if (lane == 31) s_warp[32] = w;
            }
            __syncthreads();
            unsigned long long o = base + s_warp[warp] + run - mine;
            const uint32_t at = first + 4096 * k + 4 * t;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                if (at + j < tiles) offsets[at + j] = (uint32_t)o;
                o += v[k][j];
            }
            base += s_warp[32];
            __syncthreads();
        }
    }
    if (t == 0) res->total = base;
}

// ---------------------------------------------------------------- 5. pack

// One warp per tile.  Output row r of a stream with n bytes in a tile of depth ml is its byte r - (ml - n); a lane makes
// four rows of four neighbouring streams: per stream two words and a funnel shift, then a 4 x 4 byte transpose.
__global__ void __launch_bounds__(256) k_pack32(const uint32_t *__restrict__ words, uint32_t cap_words,
                                                const uint32_t *__restrict__ sizes, const uint32_t *__restrict__ offsets,
                                                const uint32_t *__restrict__ max_lens, uint32_t tiles,
                                                uint8_t *__restrict__ stream) {
    const uint32_t t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = lane_id();
    if (t >= tiles) return;
    const uint32_t ml = max_lens[t], j = lane & 15;
    const uint4 n = *reinterpret_cast<const uint4 *>(sizes + (size_t)t * 64 + 4 * j);
    const uint32_t skip[4] = {ml - n.x, ml - n.y, ml - n.z, ml - n.w};
    const uint32_t *src = words + (size_t)t * cap_words * 64 + 4 * j;
    uint32_t *dst = reinterpret_cast<uint32_t *>(stream + offsets[t]) + j;
    for (uint32_t r = (lane >> 4) * 4; r < ml; r += 8) {
        uint32_t v[4];
#pragma unroll
        for (int s = 0; s < 4; ++s) {
            const int b = (int)r - (int)skip[s], w = b >> 2;    // arithmetic: rows above the stream are zero
            const uint32_t hi = w >= 0 ? src[(size_t)w * 64 + s] : 0u;
            const uint32_t lo = w + 1 >= 0 && w + 1 < (int)cap_words ? src[(size_t)(w + 1) * 64 + s] : 0u;
            v[s] = __funnelshift_l(lo, hi, 8 * (b & 3));        // bytes b .. b + 3, the first in the high byte
        }
        // rows of four streams: byte 3 - i of every v
        const uint32_t a = __byte_perm(v[0], v[1], 0x6273), b = __byte_perm(v[2], v[3], 0x6273);   // {v0.3, v1.3, v0.2, v1.2}
        const uint32_t c = __byte_perm(v[0], v[1], 0x4051), d = __byte_perm(v[2], v[3], 0x4051);   // {v0.1, v1.1, v0.0, v1.0}
        const uint32_t o[4] = {__byte_perm(a, b, 0x5410), __byte_perm(a, b, 0x7632), __byte_perm(c, d, 0x5410),
                               __byte_perm(c, d, 0x7632)};
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (r + i < ml) dst[(size_t)(r + i) * 16] = o[i];
    }
}

// ------------------------------------------------------------------------ host

// Page-locked landing place of the results, one per host thread: a pageable copy would be staged by the driver.
struct PinnedResult {
    EncResult *p = nullptr;
    ~PinnedResult() {
        if (p != nullptr) (void)cudaFreeHost(p);                // idle: every call that used it has waited
    }
};
static EncResult *pinned_result() {
    static thread_local PinnedResult r;
    if (r.p == nullptr && cudaHostAlloc((void **)&r.p, sizeof *r.p, cudaHostAllocPortable) != cudaSuccess) r.p = nullptr;
    return r.p;
}

static bool encode32_takes(const Geom &g) { return g.tw == 32 && g.th >= 16 && g.th % 16 == 0; }

static uint32_t table_blocks(const Enc32Args &a) { return 2 + a.tiles_k * a.tiles_n / 16384; }

template <int COLS, bool PLANE>
static int launch_encode32(const Enc32Args &a, cudaStream_t s) {
    const uint32_t warps = (a.tiles_n + COLS - 1) / COLS * 2 * a.tiles_k;
    return launch_behind(k_encode32<COLS, PLANE>, (warps + kEncWarps<COLS> - 1) / kEncWarps<COLS>, kEncWarps<COLS> * 32, s, a);
}

template <bool PLANE>
static int encode32(Enc32Args a, uint32_t *d_offsets, EncResult *d_res, uint64_t *stream_len, cudaStream_t s) {
    // Two columns a lane halve the loads, stores and address arithmetic per symbol, but also the warps: only where a
    // multiprocessor keeps 16 of them.
    const bool aligned = a.N % 2 == 0 && (reinterpret_cast<uintptr_t>(a.src) & (PLANE ? 1u : 3u)) == 0 &&
                         (reinterpret_cast<uintptr_t>(a.mantissa) & 1u) == 0;
    const uint64_t warps2 = (uint64_t)(a.tiles_n + 1) / 2 * 2 * a.tiles_k;
    int rc = aligned && warps2 >= 16ull * sm_count() ? launch_encode32<2, PLANE>(a, s) : launch_encode32<1, PLANE>(a, s);
    if (rc) return rc;
    if ((rc = launch_behind(k_scan_tiles, 1, 1024, s, a.max_lens, a.tiles_k * a.tiles_n, d_offsets, d_res))) return rc;
    EncResult *h = pinned_result();
    CI_REQUIRE(h != nullptr, "no page-locked memory for the encoder's results");
    CI_CUDA(cudaMemcpyAsync(h, d_res, sizeof *h, cudaMemcpyDeviceToHost, s));
    CI_CUDA(cudaStreamSynchronize(s));
    *stream_len = h->total;
    if (h->total > 0xFFFFFFFFull) {
        set_error("compressed stream of %llu bytes exceeds the format's 32-bit offsets", h->total);
        return CI_E_OVERFLOW;
    }
    return CI_OK;
}

static int fill_args(Enc32Args &a, const void *src, uint32_t K, uint32_t N, uint32_t th, uint32_t tw, uint32_t *d_states,
                     uint32_t *d_sizes, uint32_t *d_offsets, uint32_t *d_max_lens, void *d_scratch, size_t scratch_bytes) {
    CI_REQUIRE(src && d_states && d_sizes && d_offsets && d_max_lens && d_scratch, "null pointer");
    int rc = check_tile(K, N, th, tw);
    if (rc) return rc;
    const Geom g = make_geom(K, N, th, tw);
    CI_REQUIRE(encode32_takes(g), "the one-pass encoder takes 32-wide tiles, got %u", tw);
    CI_REQUIRE((reinterpret_cast<uintptr_t>(d_scratch) & 15u) == 0 && (reinterpret_cast<uintptr_t>(d_sizes) & 15u) == 0,
               "scratch and sizes must be 16-byte aligned");
    if (scratch_bytes < ci_compress_scratch_bytes(K, N, th, tw)) {
        set_error("scratch of %zu bytes, %zu needed", scratch_bytes, ci_compress_scratch_bytes(K, N, th, tw));
        return CI_E_WORKSPACE;
    }
    uint8_t *base = static_cast<uint8_t *>(d_scratch);
    a.src = src;
    a.K = K; a.N = N; a.th = th; a.half = g.half; a.tiles_n = g.tiles_n; a.tiles_k = g.tiles_k;
    a.mantissa = nullptr;
    a.states = d_states; a.sizes = d_sizes; a.max_lens = d_max_lens;
    a.words = reinterpret_cast<uint32_t *>(base + kEncHead);
    a.cap_words = stream_words(g.half);
    a.table = reinterpret_cast<const uint4 *>(base + kOffEncTab);
    return CI_OK;
}

}  // namespace ci

using namespace ci;

extern "C" {

size_t ci_compress_scratch_bytes(uint32_t K, uint32_t N, uint32_t th, uint32_t tw) {
    if (check_tile(K, N, th, tw)) return 0;
    const Geom g = make_geom(K, N, th, tw);
    if (!encode32_takes(g)) return 0;
    return kEncHead + (size_t)g.tiles_k * g.tiles_n * stream_words(g.half) * 64 * sizeof(uint32_t);
}

int ci_compress_bf16(const uint16_t *d_w, uint32_t K, uint32_t N, uint32_t th, uint32_t tw, uint8_t *d_man_tiled,
                     uint32_t *d_states, uint32_t *d_sizes, uint32_t *d_tile_offsets, uint32_t *d_tile_max_lens,
                     uint32_t *d_tables, uint8_t *d_slot_map, void *d_scratch, size_t scratch_bytes, uint16_t *freqs,
                     uint16_t *cdf, uint64_t *man_hist, uint64_t *stream_len, ci_stream_t stream) {
    CI_REQUIRE(d_man_tiled && freqs && cdf && stream_len, "null pointer");
    Enc32Args a;
    int rc = fill_args(a, d_w, K, N, th, tw, d_states, d_sizes, d_tile_offsets, d_tile_max_lens, d_scratch, scratch_bytes);
    if (rc) return rc;
    a.mantissa = d_man_tiled;
    cudaStream_t s = (cudaStream_t)stream;
    uint8_t *base = static_cast<uint8_t *>(d_scratch);
    unsigned long long *hist = reinterpret_cast<unsigned long long *>(base);
    unsigned long long *mh = reinterpret_cast<unsigned long long *>(base + kOffManHist);
    EncResult *res = reinterpret_cast<EncResult *>(base + kOffResult);
    const uint64_t n = (uint64_t)K * N;
    CI_CUDA(cudaMemsetAsync(base, 0, kOffEncTab, s));
    if (K % th || N % 32) CI_CUDA(cudaMemsetAsync(d_man_tiled, 0, (size_t)a.tiles_k * a.tiles_n * th * 32, s));
    uint64_t blocks = (n / 8 + 511) / 512 + 1, cap = (uint64_t)sm_count() * (man_hist ? 3 : 4);
    if (blocks > cap) blocks = cap;
    static SmemLimit lim[2] = {};
    const size_t smem = man_hist ? 65536 : 32768;
    const void *kernel = man_hist ? (const void *)k_exp_histogram<true> : (const void *)k_exp_histogram<false>;
    if ((rc = ensure_smem_limit(lim[man_hist != nullptr], kernel, smem))) return rc;
    if (man_hist) k_exp_histogram<true><<<(uint32_t)blocks, 512, smem, s>>>(d_w, n, hist, mh);
    else k_exp_histogram<false><<<(uint32_t)blocks, 512, smem, s>>>(d_w, n, hist, nullptr);
    CI_LAUNCH_CHECK(k_exp_histogram);
    if ((rc = launch_behind(k_make_tables, table_blocks(a), 256, s, hist, man_hist ? mh : nullptr, res, reinterpret_cast<uint4 *>(base + kOffEncTab),
                            d_tables, d_slot_map, a.max_lens, a.tiles_k * a.tiles_n)))
        return rc;
    rc = encode32<false>(a, d_tile_offsets, res, stream_len, s);
    const EncResult *h = pinned_result();
    if (rc == CI_OK) {
        memcpy(freqs, h->freqs, sizeof h->freqs);
        memcpy(cdf, h->cdf, sizeof h->cdf);
        if (man_hist) memcpy(man_hist, h->man_hist, sizeof h->man_hist);
    }
    return rc;
}

int ci_compress_plane(const uint8_t *d_plane, uint32_t K, uint32_t N, const uint16_t *freqs, const uint16_t *cdf, uint32_t th,
                      uint32_t tw, uint32_t *d_states, uint32_t *d_sizes, uint32_t *d_tile_offsets, uint32_t *d_tile_max_lens,
                      uint32_t *d_tables, uint8_t *d_slot_map, void *d_scratch, size_t scratch_bytes, uint64_t *stream_len,
                      ci_stream_t stream) {
    CI_REQUIRE(freqs && cdf && stream_len, "null pointer");
    uint32_t sum = 0;
    for (int i = 0; i < 256; ++i) {
        CI_REQUIRE(freqs[i] >= 1, "symbol %d has zero frequency; every symbol needs at least 1", i);
        CI_REQUIRE(cdf[i] == sum, "cdf[%d] is %u, the frequencies before it sum to %u", i, cdf[i], sum);
        sum += freqs[i];
    }
    CI_REQUIRE(sum == kProbScale, "frequencies sum to %u, expected 4096", sum);
    Enc32Args a;
    int rc = fill_args(a, d_plane, K, N, th, tw, d_states, d_sizes, d_tile_offsets, d_tile_max_lens, d_scratch, scratch_bytes);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    uint8_t *base = static_cast<uint8_t *>(d_scratch);
    EncResult *res = reinterpret_cast<EncResult *>(base + kOffResult), *h = pinned_result();
    CI_REQUIRE(h != nullptr, "no page-locked memory for the encoder's results");
    memcpy(h->freqs, freqs, sizeof h->freqs);                   // idle: every call that used it has waited
    memcpy(h->cdf, cdf, sizeof h->cdf);
    CI_CUDA(cudaMemcpyAsync(res, h, sizeof *res, cudaMemcpyHostToDevice, s));
    if ((rc = launch_behind(k_make_tables, table_blocks(a), 256, s, nullptr, nullptr, res, reinterpret_cast<uint4 *>(base + kOffEncTab), d_tables,
                            d_slot_map, a.max_lens, a.tiles_k * a.tiles_n)))
        return rc;
    return encode32<true>(a, d_tile_offsets, res, stream_len, s);
}

int ci_compress_pack(uint32_t K, uint32_t N, uint32_t th, uint32_t tw, const uint32_t *d_sizes, const uint32_t *d_tile_offsets,
                     const uint32_t *d_tile_max_lens, const void *d_scratch, size_t scratch_bytes, uint8_t *d_stream,
                     uint64_t stream_len, ci_stream_t stream) {
    Enc32Args a;
    int rc = fill_args(a, d_scratch, K, N, th, tw, const_cast<uint32_t *>(d_sizes), const_cast<uint32_t *>(d_sizes),
                       const_cast<uint32_t *>(d_tile_offsets), const_cast<uint32_t *>(d_tile_max_lens),
                       const_cast<void *>(d_scratch), scratch_bytes);
    if (rc) return rc;
    CI_REQUIRE(d_stream || stream_len == 0, "null stream buffer");
    CI_REQUIRE((reinterpret_cast<uintptr_t>(d_stream) & 3u) == 0, "stream buffer must be 4-byte aligned");
    if (stream_len == 0) return CI_OK;
    const uint32_t tiles = a.tiles_k * a.tiles_n;
    k_pack32<<<(tiles + 7) / 8, 256, 0, (cudaStream_t)stream>>>(a.words, a.cap_words, d_sizes, d_tile_offsets, d_tile_max_lens,
                                                                tiles, d_stream);
    CI_LAUNCH_CHECK(k_pack32);
    return CI_OK;
}

}  // extern "C"
