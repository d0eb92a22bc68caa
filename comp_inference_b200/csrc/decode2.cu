// Stand-alone decoder for 32-wide tiles, two streams per lane: the exponent plane (u8) or the bf16 weight [K,N] of weights
// with few streams for their size -- tall tiles, small matrices -- which leave the four-streams decoder (decode4.cu) too few
// warps: a warp of it decodes two tiles at 260 cycles a row, whatever the rest of the multiprocessor does.
//
// Work unit: one warp decodes one tile = 64 streams.  Lane l owns columns 2 (l % 16) and 2 (l % 16) + 1 of the top
// (l < 16) or bottom half, so a row's two weights are one 4-byte store and its two sign+mantissa bytes one load.  Byte block
// and initial states arrive by bulk copy, sign+mantissa bytes in double-buffered chunks of 16 rows.  A unit is the whole
// chain of a stream, usually one a warp: nothing is fetched for the next one ahead.
//
// Measured on a B200 (graph replays over more than L2), four streams per lane -> two: 4096 x 11008 at tile height 1024 59.8 ->
// 51.9 us (1376 tiles: nine or ten warps a multiprocessor, so three on some scheduler and 2.3 on average; the waits that are left are
// the chain's own, arithmetic and table look-ups), 1000 x 1000 at 512 34 -> 17, 777 x 1001 at 128 13.3 -> 7.3.
#include "decode.cuh"
#include "ptx.cuh"

namespace ci {

constexpr uint32_t kDec2Warps = 20;
constexpr uint32_t kDec2BarBytes = 512;      // per warp the window's barrier and two chunk barriers; the table's
constexpr uint32_t kDec2Seg = kChunkRows * 32 + 32;             // one half's rows of a chunk, the halves 8 banks apart
constexpr uint32_t kDec2Man = 2 * 2 * kDec2Seg;

struct Dec2Args {
    DecArgs a;
    uint32_t cap_rows;     // rows of the byte window (>= every tile_max_len)
    uint32_t win_bytes;    // window + 64 initial states
    uint32_t total;        // tiles
    uint32_t vec;          // output rows can be written as aligned pairs
};

// Two streams of one lane whose bytes are neighbours (rows 64 bytes apart).  As Quad, but the second byte is handled under
// predicates: it is needed exactly where the state is below 2^8 before the first one, so nothing waits, and where the chain
// of one warp is what counts, a branch per symbol costs more than the four instructions (1024 x 4096 at tile height 1024:
// 45.8 us with it, 35.9 without).
struct Pair {
    uint32_t s[2], p[2];

    __device__ __forceinline__ void start(uint32_t states_s, uint32_t first) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            s[j] = lds_u32(states_s + 4 * j);
            p[j] = first + j;
        }
    }
    __device__ __forceinline__ void step(uint32_t lut_s, uint32_t (&e)[2]) {
        const uint32_t y0 = lds_u8(p[0]), y1 = lds_u8(p[1]);
        e[0] = decode_aligned(s[0], lut_s);
        e[1] = decode_aligned(s[1], lut_s);
        asm volatile(
            "{\n\t.reg .pred p0, p1, r0, r1;\n\t.reg .u32 m0, m1;\n\t"
            "setp.lt.u32 p0, %0, 65536;\n\t"
            "setp.lt.u32 p1, %1, 65536;\n\t"
            "setp.lt.u32 r0, %0, 256;\n\t"
            "setp.lt.u32 r1, %1, 256;\n\t"
            "@r0 ld.shared.u8 m0, [%2+-64];\n\t"
            "@r1 ld.shared.u8 m1, [%3+-64];\n\t"
            "@p0 mad.lo.u32 %0, %0, 256, %4;\n\t"
            "@p1 mad.lo.u32 %1, %1, 256, %5;\n\t"
            "@p0 sub.u32 %2, %2, 64;\n\t"
            "@p1 sub.u32 %3, %3, 64;\n\t"
            "@r0 mad.lo.u32 %0, %0, 256, m0;\n\t"
            "@r1 mad.lo.u32 %1, %1, 256, m1;\n\t"
            "@r0 sub.u32 %2, %2, 64;\n\t"
            "@r1 sub.u32 %3, %3, 64;\n\t}"
            : "+r"(s[0]), "+r"(s[1]), "+r"(p[0]), "+r"(p[1])
            : "r"(y0), "r"(y1));
    }
    // The same with the second bytes loaded ahead too, see Quad::step_ahead.
    __device__ __forceinline__ void step_ahead(uint32_t lut_s, uint32_t (&e)[2]) {
        uint32_t y[2], v[2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            y[j] = lds_u8(p[j]);
            v[j] = lds_u8(p[j] - 64);
        }
        e[0] = decode_aligned(s[0], lut_s);
        e[1] = decode_aligned(s[1], lut_s);
#pragma unroll
        for (int j = 0; j < 2; ++j)
            asm("{\n\t.reg .pred p, q;\n\t"
                "setp.lt.u32 p, %0, 65536;\n\t"
                "setp.lt.u32 q, %0, 256;\n\t"
                "@p mad.lo.u32 %0, %0, 256, %2;\n\t"
                "@p sub.u32 %1, %1, 64;\n\t"
                "@q mad.lo.u32 %0, %0, 256, %3;\n\t"
                "@q sub.u32 %1, %1, 64;\n\t}"
                : "+r"(s[j]), "+r"(p[j])
                : "r"(y[j]), "r"(v[j]));
    }
    __device__ __forceinline__ void clamp(uint32_t low) {
        p[0] = max(p[0], low);
        p[1] = max(p[1], low);
    }
};

// EDGE: the last tile row is not whole, or output rows cannot be written as aligned pairs.
// AHEAD: at most a warp a scheduler, so the chain alone counts.  4096 x 2048 at tile height 1024 (1.7 warps a multiprocessor) 36.5 us ->
// 30.7; with nine or ten warps it costs 6 %.
template <bool BF16, bool EDGE, bool AHEAD>
__global__ void __launch_bounds__(kDec2Warps * 32, 1) k_decode2(const __grid_constant__ Dec2Args p, void *out) {
    extern __shared__ __align__(128) uint8_t smem[];
    const DecArgs &a = p.a;
    const Geom &g = a.g;
    const uint32_t W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = lane_id();
    const uint32_t smem_s = smem_u32(smem);
    const uint32_t lut_s = (smem_s + kLutBytes - 1) & ~(kLutBytes - 1);
    const uint32_t lut_bar = lut_s + kLutBytes + kDec2BarBytes - 16;
    start_lut(lut_s, lut_bar, a.lut);
    const uint32_t man_s = lut_s + kLutBytes + kDec2BarBytes + warp * (BF16 ? kDec2Man : 0);
    const uint32_t win_s = lut_s + kLutBytes + kDec2BarBytes + W * (BF16 ? kDec2Man : 0) + warp * p.win_bytes;
    const uint32_t bar = lut_s + kLutBytes + warp * 24, man_bar = bar + 8;
    const uint32_t h = lane >> 4, c2 = 2 * (lane & 15);         // stream half, first column inside the tile
    // Rank in the grid, the CTA running fastest: the warps of a multiprocessor are as many as on any other.
    const uint32_t gw = warp * gridDim.x + blockIdx.x, n_warps = gridDim.x * W;

    // Rows [kChunkRows * c, + kChunkRows) of both halves into chunk buffer `buf`; src: the lane's piece of chunk 0.
    auto issue_man = [&](const uint8_t *src, uint32_t c, uint32_t buf) {
        if (c * kChunkRows + (lane >> 1) < g.half) {
            const uint32_t dst = man_s + buf * (2 * kDec2Seg) + lane * 16;
            cp_async16(dst, src + c * (kChunkRows * 32));
            cp_async16(dst + kDec2Seg, src + c * (kChunkRows * 32) + g.half * 32);
        }
        cp_async_arrive(man_bar + buf * 8);
    };
    // Starts the copies of tile t (whole warp).
    // The sign+mantissa bytes do not wait for the byte range.  Where many warps start at once asking for them first spreads their copies
    // (1500 x 4000 at tile height 128 8.8 us -> 8.5, 3000 x 1500 at 64 6.7 -> 6.4); where few do, it is 0.5 % slower.
    const bool man_first = W > 8;
    auto issue = [&](uint32_t t, uint32_t &ml) {
        ml = __ldg(a.tile_max_lens + t);
        const uint32_t off = __ldg(a.tile_offsets + t);
        const uint8_t *man = a.mantissa + (size_t)t * g.th * 32 + lane * 16;
        if (BF16 && man_first) issue_man(man, 0, 0);
        if (ml > p.cap_rows) ml = 0;                            // metadata disagrees with the declared maximum
        if (lane == 0) {
            fence_async_proxy();
            mbar_expect_tx(bar, ml * 64 + 256);
            if (ml) bulk_load(win_s, a.stream + off, ml * 64, bar);
            bulk_load(win_s + p.cap_rows * 64, a.states + (size_t)t * 64, 256, bar);
        }
        if (BF16 && !man_first) issue_man(man, 0, 0);
    };

    if (lane == 0) {
        mbar_init(bar, 1);
        mbar_init(man_bar, 32);
        mbar_init(man_bar + 8, 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    uint32_t ml = 0;
    if (gw < p.total) issue(gw, ml);
    if (a.lut == nullptr) load_lut(reinterpret_cast<uint32_t *>(smem + (lut_s - smem_s)), nullptr, a.tables, a.slot_map);
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");          // the output may be in use by the kernel before
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    (void)wait_lut(lut_bar, a.lut);

    const uint32_t n_chunks = (g.half + kChunkRows - 1) / kChunkRows;
    uint32_t parity = 0, chunk0 = 0, chunk1 = 0;                // phases of the window's and the chunks' barriers
    for (uint32_t t = gw; t < p.total; t += n_warps) {
        if (t != gw) {
            __syncwarp();                                       // every lane is done with the window
            issue(t, ml);
        }
        const uint32_t tk = t / g.tiles_n, tn = t - tk * g.tiles_n, col = tn * 32 + c2;
        const uint32_t row = tk * g.th + h * g.half;            // first row of this lane's streams
        uint32_t rows = 0xFFFFFFFFu, h_d = h, c_d = c2, len = 0xFFFFFFFFu;
        if constexpr (EDGE) {
            // A lane without rows or columns decodes the top half's first columns, and a stream that is used up starts over:
            // past the end of a stream the symbols are rare ones, and every step would take the branch for a second byte.
            rows = row < g.K ? min(g.half, g.K - row) : 0u;
            if (col >= g.N) {
                rows = 0;
                c_d = 0;
            }
            if (rows == 0) h_d = 0;
            const uint32_t first = tk * g.th + h_d * g.half;    // < K: only tiles with rows exist
            len = (min(g.half, g.K - first) + kChunkRows - 1) / kChunkRows;
        } else if (col >= g.N) {
            rows = 0;
            c_d = 0;
        }
        uint32_t left = len;
        const uint32_t st_s = win_s + p.cap_rows * 64 + (h_d * 32 + c_d) * 4;
        const uint32_t first = win_s + h_d * 32 + c_d + (ml - 1) * 64;   // last byte row; an empty tile starts one row below
        (void)mbar_wait(bar, parity);
        parity ^= 1;
        Pair z;
        auto start_streams = [&]() {
            z.start(st_s, first);
            if (EDGE && tn * 32 + c_d + 1 >= g.N) {             // as Quad::keep
                z.s[1] = z.s[0];
                z.p[1] = z.p[0];
            }
        };
        start_streams();

        uint8_t *o = reinterpret_cast<uint8_t *>(out) + ((size_t)row * a.ld + col) * (BF16 ? 2 : 1);
        const size_t pitch = (size_t)a.ld * (BF16 ? 2 : 1);
        const uint8_t *man = a.mantissa + (size_t)t * g.th * 32 + lane * 16;
#pragma unroll 1
        for (uint32_t c = 0; c < n_chunks; ++c) {
            uint32_t ms = 0;
            if constexpr (BF16) {
                const uint32_t buf = c & 1;
                __syncwarp();                                   // every lane is done with the other chunk buffer
                if (c + 1 < n_chunks) issue_man(man, c + 1, buf ^ 1);
                (void)mbar_wait(man_bar + buf * 8, buf ? chunk1 : chunk0);
                if (buf) chunk1 ^= 1; else chunk0 ^= 1;
                ms = man_s + buf * (2 * kDec2Seg) + h * kDec2Seg + c2;
            }
            z.clamp(win_s);
            const uint32_t n = min(kChunkRows, g.half - c * kChunkRows);
            auto decode_rows = [&](auto store) {
#pragma unroll 1
                for (uint32_t r = 0; r < n; r += 8) {           // half a tile is a multiple of eight rows
#pragma unroll
                    for (uint32_t i = 0; i < 8; ++i) {
                        const uint32_t m = BF16 ? lds_u16(ms + i * 32) : 0u;
                        uint32_t e[2];
                        if constexpr (AHEAD) z.step_ahead(lut_s, e);
                        else z.step(lut_s, e);
                        store(r + i, BF16 ? exp_or_man(__byte_perm(e[0], e[1], 0x6521) << 3, __byte_perm(m, 0u, 0x1100))
                                          : (e[0] >> 12 & 0xFFu) | (e[1] >> 4 & 0xFF00u));
                        o += pitch;
                    }
                    ms += 256;
                }
            };
            auto store_pair = [&](uint32_t v) {
                if constexpr (BF16) *reinterpret_cast<uint32_t *>(o) = v;
                else *reinterpret_cast<uint16_t *>(o) = (uint16_t)v;
            };
            const uint32_t done = c * kChunkRows;
            const bool mine = rows > done;
            if (!EDGE || __all_sync(kFull, p.vec && (!mine || rows >= done + n))) {
                decode_rows([&](uint32_t, uint32_t v) {
                    if (mine) store_pair(v);
                });
            } else {
                decode_rows([&](uint32_t r, uint32_t v) {
                    if (done + r >= rows) return;
                    if (p.vec) {
                        store_pair(v);
                    } else if constexpr (BF16) {
                        reinterpret_cast<uint16_t *>(o)[0] = (uint16_t)v;
                        if (col + 1 < g.N) reinterpret_cast<uint16_t *>(o)[1] = (uint16_t)(v >> 16);
                    } else {
                        o[0] = (uint8_t)v;
                        if (col + 1 < g.N) o[1] = (uint8_t)(v >> 8);
                    }
                });
            }
            if (EDGE && --left == 0) {
                left = len;
                start_streams();
            }
        }
    }
}

template <bool BF16, bool EDGE, bool AHEAD>
static int launch_dec2_as(const Dec2Args &p, uint32_t blocks, uint32_t warps, size_t smem, int max_smem, void *out, cudaStream_t s) {
    static SmemLimit lim = {};
    if (int rc = ensure_smem_limit(lim, (const void *)k_decode2<BF16, EDGE, AHEAD>, (size_t)max_smem)) return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    CI_CUDA(cudaLaunchKernelEx(&cfg, k_decode2<BF16, EDGE, AHEAD>, p, out));
    return CI_OK;
}

template <bool BF16, bool EDGE>
static int launch_dec2(const Dec2Args &p, uint32_t blocks, uint32_t warps, size_t smem, int max_smem, void *out, cudaStream_t s) {
    return warps <= 4 ? launch_dec2_as<BF16, EDGE, true>(p, blocks, warps, smem, max_smem, out, s)
                      : launch_dec2_as<BF16, EDGE, false>(p, blocks, warps, smem, max_smem, out, s);
}

int launch_decode2(const DecArgs &a, uint32_t max_tile_len, bool bf16, void *out, cudaStream_t s) {
    const Geom &g = a.g;
    if (g.tw != 32 || g.th % 16 != 0 || max_tile_len == 0) return 1;
    if (!a.stream_aligned || (reinterpret_cast<uintptr_t>(a.states) & 15u)) return 1;
    if (bf16 && (reinterpret_cast<uintptr_t>(a.mantissa) & 15u)) return 1;
    int dev = 0, max_smem = 0;
    CI_CUDA(cudaGetDevice(&dev));
    CI_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    Dec2Args p;
    p.a = a;
    p.cap_rows = max_tile_len;
    p.win_bytes = (max_tile_len * 64u + 256u + 127u) & ~127u;
    p.total = g.tiles_k * g.tiles_n;
    const uint32_t fixed = 2 * kLutBytes + kDec2BarBytes, P = (uint32_t)sm_count();
    const uint32_t warp_bytes = p.win_bytes + (bf16 ? kDec2Man : 0u), units = (p.total + P - 1) / P;
    uint32_t w_max = ((uint32_t)max_smem - fixed) / warp_bytes;
    if (w_max > kDec2Warps) w_max = kDec2Warps;
    // us at 64 symbols per stream, as run_cost: a round of one warp per scheduler is the chain (3.5), with n it is n warps'
    // instructions.  512 symbols a stream took 31 us with up to 4 warps, 46 with 8, 54 with 10, 60 with 12, 256 symbols 42.5 with 17;
    // the 2 us or so that every launch has are left out, as they are in run_cost.
    auto round2 = [](uint32_t w) { return w <= 4 ? 3.5 : w <= 8 ? 5.3 : w <= 12 ? 7.2 : w <= 16 ? 8.8 : 10.0; };
    uint32_t warps = 0;
    double best = 0.0;
    for (uint32_t w = 1; w <= w_max; ++w) {
        const double cost = (units / w) * round2(w) + (units % w ? round2(units % w) : 0.0);
        if (warps == 0 || cost < best) { best = cost; warps = w; }
    }
    if (warps == 0) return 1;
    const double four = decode4_cost(a, max_tile_len, bf16);   // 0: not a weight for it
    if (four > 0.0 && four <= best) return 1;
    const uint32_t blocks = p.total < P ? p.total : P;
    p.vec = a.ld % 2 == 0 && g.N % 2 == 0 && (reinterpret_cast<uintptr_t>(out) & (bf16 ? 3u : 1u)) == 0;
    const bool edge = g.K % g.th != 0 || !p.vec;
    const size_t smem = fixed + (size_t)warps * warp_bytes;
    if (bf16) return edge ? launch_dec2<true, true>(p, blocks, warps, smem, max_smem, out, s)
                          : launch_dec2<true, false>(p, blocks, warps, smem, max_smem, out, s);
    return edge ? launch_dec2<false, true>(p, blocks, warps, smem, max_smem, out, s)
                : launch_dec2<false, false>(p, blocks, warps, smem, max_smem, out, s);
}

}  // namespace ci
