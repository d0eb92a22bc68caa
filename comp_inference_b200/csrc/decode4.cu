// Stand-alone decoder for 32-wide tiles, four streams per lane: exponent plane (u8) or the full bf16
// weight [K,N].  Replaces rans_decompress_tiled_kernel_triton_ilp2 (comp_inference/rans_triton.py:34-119)
// and the decode + uninterleave + reconstruct chain of rans_decompress_module_weight_bf16
// (comp_inference/comp_inference.py:633-711).
//
// Work unit: one warp decodes two horizontally adjacent tiles of one tile row = 128 streams.  Lane l
// (quad = l / 2, half = l % 2) owns the four adjacent columns 4 quad .. 4 quad + 3 of the 64-column
// strip, top-half streams on even lanes and bottom-half streams on odd lanes, so
//  * the two tiles' byte blocks, copied by cp.async into one window of 128-byte rows (left tile in
//    bytes 0..63, right tile in 64..127), give every lane a word column -- a shared-memory bank -- of its
//    own: the per-symbol renormalisation byte loads never conflict, whatever row each cursor is on;
//  * the sign+mantissa bytes come through shared memory in chunks of 16 rows (ptx.cuh): read with global loads they
//    were the kernel's largest stall (1.9 of 6 cycles per instruction) and four wavefronts a row;
//  * a decoded row of the lane is four adjacent weights: one 8-byte store (4 bytes for the plane), and the
//    sixteen lanes of a half write 128 contiguous bytes of an output row.
// Initial states arrive with the unit's bytes, byte ranges of later units are loaded ahead by all
// lanes in parallel, windows are double buffered per warp where they fit (tall tiles: one window), and the kernel is
// launched with programmatic dependent launch (its preamble overlaps the previous kernel of the stream).
#include "decode.cuh"
#include "ptx.cuh"

namespace ci {

constexpr uint32_t kDec4Warps = 21;          // six on one scheduler: 80 registers a thread, which it needs (none spilled)
constexpr uint32_t kDec4AheadWarps = 8;      // up to here the chain is what counts: Quad::step_ahead
constexpr uint32_t kDec4BarBytes = 128;      // the table's barrier

struct Dec4Args {
    DecArgs a;
    uint32_t cap_rows;     // rows of a byte window (>= every tile_max_len)
    uint32_t stage_bytes;  // window + 128 initial states
    uint32_t stages;       // windows per warp
    uint32_t pairs_n;      // tile pairs per tile row = ceil(tiles_n / 2)
    uint32_t total;        // units
    uint32_t vec;          // output rows can be written as aligned quads
    uint32_t step, subs;   // INDEX, ENTRY: rows between entry points, entry points per half tile
    uint32_t *entry_states;
    uint16_t *entry_rows;
    const uint32_t *entry_spans;
};

// ENTRY: units are the rows between two entry points of a tile pair, as in linear_mma4.cu.
// INDEX: nothing is stored but the decoder's state every `step` symbols, and for every stream the rows of its byte block
// that are left then.
// EDGE: the last tile row is not whole (rows beyond K are decoded to garbage and not stored), or output rows cannot be
// written as aligned quads (N or the address is odd).
template <bool BF16, bool EDGE, bool INDEX, bool ENTRY, bool AHEAD>
__global__ void __launch_bounds__((AHEAD ? kDec4AheadWarps : kDec4Warps) * 32, 1) k_decode4(const __grid_constant__ Dec4Args p, void *out) {
    extern __shared__ __align__(128) uint8_t smem[];
    const DecArgs &a = p.a;
    const Geom &g = a.g;
    const uint32_t W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = lane_id();
    const uint32_t smem_s = smem_u32(smem);
    // The table sits on a 16 KB boundary of the shared window: an entry's address is then
    // (state << 2 & 0x3FFC) | base, without an addition.
    const uint32_t lut_s = (smem_s + kLutBytes - 1) & ~(kLutBytes - 1);
    uint32_t *s_lut = reinterpret_cast<uint32_t *>(smem + (lut_s - smem_s));
    const uint32_t lut_bar = lut_s + kLutBytes + kDec4BarBytes - 16;
    start_lut(lut_s, lut_bar, a.lut);
    const uint32_t man_s = lut_s + kLutBytes + kDec4BarBytes + (BF16 ? warp * kManBytes : 0);
    const uint32_t wbase_s = lut_s + kLutBytes + kDec4BarBytes + (BF16 ? W * kManBytes : 0) + warp * p.stages * p.stage_bytes;
    const uint32_t st_off = p.cap_rows * 128;
    const uint32_t seg_bytes = g.th * 16;                       // half a tile of sign+mantissa bytes

    const uint32_t quad = lane >> 1, hsel = lane & 1;           // column quad of the 64-column strip, stream half
    const uint32_t tsel = quad >> 3;                            // left / right tile
    // Rank in the grid, the CTA running fastest: what the last round lacks, it lacks on every multiprocessor alike.
    const uint32_t gw = warp * gridDim.x + blockIdx.x, n_warps = gridDim.x * W;

    const uint32_t subs = ENTRY ? p.subs : 1u, step = ENTRY ? p.step : g.half;

    // Unit u = (tile row, entry point, tile pair), the pair running fastest: warps that run at the same time write
    // neighbouring pieces of the same output rows.
    auto unit_tiles = [&](uint32_t u, uint32_t &tk, uint32_t &sub, uint32_t &tp, uint32_t &t0, bool &two) {
        tk = u / p.pairs_n;
        tp = u - tk * p.pairs_n;
        sub = 0;
        if constexpr (ENTRY) {
            sub = tk % subs;
            tk /= subs;
        }
        t0 = tk * g.tiles_n + 2 * tp;
        two = 2 * tp + 1 < g.tiles_n;
    };

    // Byte ranges of the units this warp will decode, 32 at a time: lane j holds its (dbase + j)-th unit.
    uint32_t d_off0 = 0, d_ml0 = 0, d_off1 = 0, d_ml1 = 0, dbase = 0;
    auto load_desc = [&]() {
        const uint64_t u = (uint64_t)gw + (uint64_t)(dbase + lane) * n_warps;
        d_off0 = d_ml0 = d_off1 = d_ml1 = 0;
        if (u >= p.total) return;
        uint32_t tk, sub, tp, t0;
        bool two;
        unit_tiles((uint32_t)u, tk, sub, tp, t0, two);
        auto range = [&](uint32_t t, uint32_t &off, uint32_t &ml) {
            off = __ldg(a.tile_offsets + t);
            if constexpr (ENTRY) {
                ml = enter_span(__ldg(p.entry_spans + (size_t)t * subs + sub), __ldg(a.tile_max_lens + t), off);
            } else {
                ml = __ldg(a.tile_max_lens + t);
            }
        };
        range(t0, d_off0, d_ml0);
        if (two) range(t0 + 1, d_off1, d_ml1);
    };

    auto issue = [&](uint32_t t0, uint32_t sub, bool two, uint32_t stage, uint32_t off0, uint32_t ml0, uint32_t off1, uint32_t ml1) {
        const uint32_t dst = wbase_s + stage * p.stage_bytes;
        if (ml0 > p.cap_rows || ml1 > p.cap_rows) ml0 = ml1 = 0;   // metadata disagrees with the declared maximum
        // states, 16 lanes a tile, and for entry points the rows of the next bytes, 8 lanes a tile
        if constexpr (ENTRY) {
            const size_t e = ((size_t)t0 * subs + sub) * 64, d = (size_t)subs * 64;
            if (lane < 16 || two) cp_async16(dst + st_off + lane * 16, p.entry_states + e + (lane < 16 ? 0 : d) + (lane & 15) * 4);
            if (lane < 8 || (two && lane < 16))
                cp_async16(dst + st_off + 512 + lane * 16, p.entry_rows + e + (lane < 8 ? 0 : d) + (lane & 7) * 8);
        } else {
            if (lane < 16 || two) cp_async16(dst + st_off + lane * 16, a.states + (size_t)t0 * 64 + lane * 4);   // the tiles are neighbours
        }
        // byte blocks: eight lanes a row of the window, four for each tile
        const bool right = lane & 4;
        const uint8_t *src = a.stream + (right ? off1 : off0) + (lane & 3) * 16 + (lane >> 3) * 64;
        const uint32_t rows = right ? ml1 : ml0;
        uint32_t to = dst + lane * 16;
        for (uint32_t r = lane >> 3; r < rows; r += 4, to += 512, src += 256) cp_async16(to, src);
    };
    // Sign+mantissa bytes of the segments (left A, left B, right A, right B) of the unit whose first tile is t0: this lane's
    // piece of the first chunk.
    auto man_of = [&](uint32_t t0, uint32_t sub) {
        return a.mantissa + (size_t)t0 * (2 * seg_bytes) + (ENTRY ? sub * step * 32 : 0u) + lane * 16;
    };
    // Rows [row, + kChunkRows) of the four segments into chunk buffer `buf`; src: this lane's piece of them.
    auto issue_man = [&](const uint8_t *src, bool two, uint32_t row, uint32_t buf) {
        const uint32_t dst = man_s + buf * (4 * kSegPitch) + lane * 16;
        if (row + (lane >> 1) < step) {
            cp_async16(dst, src);
            cp_async16(dst + kSegPitch, src + seg_bytes);
            if (two) {
                cp_async16(dst + 2 * kSegPitch, src + 2 * seg_bytes);
                cp_async16(dst + 3 * kSegPitch, src + 3 * seg_bytes);
            }
        }
    };

    load_desc();
    uint32_t tk = 0, sub = 0, tp = 0, t0 = 0;                   // of unit t
    bool two = false;
    if (gw < p.total) {
        unit_tiles(gw, tk, sub, tp, t0, two);
        if (BF16) issue_man(man_of(t0, sub), two, 0, 0);        // does not wait for the byte ranges
    }
    uint32_t nx_off0 = __shfl_sync(kFull, d_off0, 0), nx_ml0 = __shfl_sync(kFull, d_ml0, 0);
    uint32_t nx_off1 = __shfl_sync(kFull, d_off1, 0), nx_ml1 = __shfl_sync(kFull, d_ml1, 0);
    if (gw < p.total) issue(t0, sub, two, 0, nx_off0, nx_ml0, nx_off1, nx_ml1);
    if (a.lut == nullptr) load_lut(s_lut, nullptr, a.tables, a.slot_map);
    __syncthreads();
    // Only the weight was touched so far.  With programmatic dependent launch the output buffer may still
    // be in use by the previous kernel of the stream: wait for it, then let the next launch begin.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    (void)wait_lut(lut_bar, a.lut);
    const uint32_t n_chunks = (step + kChunkRows - 1) / kChunkRows;
    uint32_t stage = 0, li = 0, chunk = 0;
    const uint8_t *man = BF16 ? man_of(t0, sub) : nullptr;      // the sign+mantissa chunk that was asked for last
    Quad z;

    for (uint32_t t = gw; t < p.total; t += n_warps, ++li) {
        const bool tile_live = tsel == 0 || two;
        const uint32_t col0 = 64 * tp + 4 * quad;               // first of this lane's four columns
        const uint32_t cols = tile_live && col0 < g.N ? min(4u, g.N - col0) : 0u;
        const uint32_t row = tk * g.th + hsel * g.half + (ENTRY ? sub * step : 0u);   // first row of this lane's streams
        uint32_t rows_left = cols == 0 ? 0u : !EDGE ? 0xFFFFFFFFu : row < g.K ? min(step, g.K - row) : 0u;
        // A lane without rows decodes the left tile's top half, and a stream that is used up before the unit's last row starts
        // over: any real symbols will do, but past the end of a stream the symbols are rare ones, and every step would
        // take the branch for a second byte.
        uint32_t tsel_d = two ? tsel : 0u, hsel_d = hsel, len = 0xFFFFFFFFu;   // len: blocks of four rows, where short
        bool empty = false;                                     // an entry point's unit may lie beyond K altogether
        if (EDGE && (tk + 1) * g.th > g.K) {
            const uint32_t top = row - hsel * g.half, top_rows = top < g.K ? min(step, g.K - top) : 0u;
            const uint32_t own = row < g.K ? min(step, g.K - row) : 0u;
            empty = top_rows == 0;
            if (own == 0) hsel_d = 0;
            len = ((own ? own : top_rows) + 3) >> 2;
        }
        uint32_t left = len;
        const uint32_t ml = tsel_d ? nx_ml1 : nx_ml0;
        const bool more = (uint64_t)t + n_warps < p.total;
        uint32_t n_tk = 0, n_sub = 0, n_tp = 0, n_t0 = 0;       // of unit t + n_warps
        bool n_two = false;
        if (more) unit_tiles(t + n_warps, n_tk, n_sub, n_tp, n_t0, n_two);
        auto next_unit = [&]() {
            if (!more) return;
            if (li + 1 - dbase == 32) {
                dbase = li + 1;
                load_desc();
            }
            const uint32_t j = li + 1 - dbase;
            nx_off0 = __shfl_sync(kFull, d_off0, j);
            nx_ml0 = __shfl_sync(kFull, d_ml0, j);
            nx_off1 = __shfl_sync(kFull, d_off1, j);
            nx_ml1 = __shfl_sync(kFull, d_ml1, j);
            issue(n_t0, n_sub, n_two, p.stages == 2 ? stage ^ 1 : 0u, nx_off0, nx_ml0, nx_off1, nx_ml1);
        };

        const uint32_t win_s = wbase_s + stage * p.stage_bytes;
        // Columns beyond N: see Quad::keep; a lane without any takes the first ones of its tile.  (An index keeps the rows
        // that its own streams have left, so there every stream is its own.)
        const uint32_t quad_d = INDEX || cols != 0 ? quad & 7 : 0u;
        const uint32_t cols_d = INDEX ? 4u : min(4u, g.N - (64 * tp + 32 * tsel_d + 4 * quad_d));
        const uint32_t st_s = win_s + st_off + tsel_d * 256 + (hsel_d * 32 + quad_d * 4) * 4;
        uint32_t first = win_s + tsel_d * 64 + hsel_d * 32 + quad_d * 4;
        if (!ENTRY && ml <= p.cap_rows) first += (ml - 1) * 128;  // last byte row; an empty tile starts one row below
        cp_async_wait();                                        // this unit's bytes and states, its first sign+mantissa chunk
        __syncwarp();
        auto start_streams = [&]() {
            z.start(st_s, first);
            if constexpr (ENTRY) {                              // every stream has its own row of the window
                const uint32_t rows_s = win_s + st_off + 512 + tsel_d * 128 + (hsel_d * 32 + quad_d * 4) * 2;
                const uint32_t r01 = lds_u32(rows_s), r23 = lds_u32(rows_s + 4), top = p.cap_rows - 1;
                z.p[0] += min(r01 & 0xFFFFu, top) * 128;
                z.p[1] += min(r01 >> 16, top) * 128;
                z.p[2] += min(r23 & 0xFFFFu, top) * 128;
                z.p[3] += min(r23 >> 16, top) * 128;
            }
            if (EDGE && cols_d < 4) z.keep(cols_d);             // without EDGE N is a multiple of four
        };
        start_streams();

        uint8_t *o8 = reinterpret_cast<uint8_t *>(out) + ((size_t)row * a.ld + col0) * (BF16 ? 2 : 1);
        const size_t o_pitch = (size_t)a.ld * (BF16 ? 2 : 1);
#pragma unroll 1
        for (uint32_t c = 0; c < n_chunks; ++c, ++chunk) {
            const uint32_t buf = chunk & 1;
            if (BF16 && c != 0) {
                cp_async_wait();                                // this chunk is here
                __syncwarp();                                   // for every lane, and all are done with the other buffer
            }
            if constexpr (BF16) {
                const bool last = c + 1 == n_chunks;
                man = last ? man_of(n_t0, n_sub) : man + kChunkRows * 32;
                if (!last || more) issue_man(man, last ? n_two : two, last ? 0u : (c + 1) * kChunkRows, buf ^ 1);
            }
            if (c == 0 && p.stages == 2) next_unit();
            if constexpr (INDEX) {
                if (c * kChunkRows % p.step == 0 && tile_live) {
                    const size_t at = (((size_t)t0 + tsel) * p.subs + c * kChunkRows / p.step) * 64 + hsel * 32 + (quad & 7) * 4;
                    const uint32_t below = win_s + tsel * 64 + hsel * 32 + (quad & 7) * 4 - 128;
                    *reinterpret_cast<uint4 *>(p.entry_states + at) = make_uint4(z.s[0], z.s[1], z.s[2], z.s[3]);
                    // A used-up stream's cursor was clamped to the window: none or one, but none in a tile without bytes.
                    uint32_t left[4];
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) left[j] = z.p[j] > below + j ? min((z.p[j] - below - j) >> 7, ml) : 0u;
                    *reinterpret_cast<uint2 *>(p.entry_rows + at) = make_uint2(left[0] | left[1] << 16, left[2] | left[3] << 16);
                }
            }
            z.clamp(win_s);
            uint32_t ms = man_s + (buf * 4 + tsel * 2 + hsel) * kSegPitch + (quad & 7) * 4;
            const uint32_t n = EDGE && empty ? 0u : min(kChunkRows, step - c * kChunkRows);
#pragma unroll 1
            for (uint32_t r = 0; r < n; r += 4) {
#pragma unroll
                for (uint32_t i = 0; i < 4; ++i) {
                    uint32_t e[4];
                    if constexpr (AHEAD) z.step_ahead(lut_s, e);
                    else z.step(lut_s, e);
                    // bits 8..23 of two entries side by side: the symbols sit at bits 4..11 / 20..27
                    const uint32_t a01 = __byte_perm(e[0], e[1], 0x6521), a23 = __byte_perm(e[2], e[3], 0x6521);
                    if constexpr (INDEX) continue;
                    const bool store = EDGE ? i < rows_left : rows_left != 0;
                    if (BF16) {
                        const uint32_t m = lds_u32(ms + i * 32);
                        const uint32_t w01 = exp_or_man(a01 << 3, __byte_perm(m, 0u, 0x1100));
                        const uint32_t w23 = exp_or_man(a23 << 3, __byte_perm(m, 0u, 0x3322));
                        if (store) {
                            if (!EDGE || (p.vec && cols == 4)) {
                                *reinterpret_cast<uint2 *>(o8) = make_uint2(w01, w23);
                            } else {
                                uint16_t *o = reinterpret_cast<uint16_t *>(o8);
                                o[0] = (uint16_t)w01;
                                if (cols > 1) o[1] = (uint16_t)(w01 >> 16);
                                if (cols > 2) o[2] = (uint16_t)w23;
                                if (cols > 3) o[3] = (uint16_t)(w23 >> 16);
                            }
                        }
                    } else {
                        const uint32_t w = __byte_perm(a01 >> 4, a23 >> 4, 0x6420);
                        if (store) {
                            if (!EDGE || (p.vec && cols == 4)) {
                                *reinterpret_cast<uint32_t *>(o8) = w;
                            } else {
                                o8[0] = (uint8_t)w;
                                if (cols > 1) o8[1] = (uint8_t)(w >> 8);
                                if (cols > 2) o8[2] = (uint8_t)(w >> 16);
                                if (cols > 3) o8[3] = (uint8_t)(w >> 24);
                            }
                        }
                    }
                    o8 += o_pitch;
                }
                ms += 128;
                if (EDGE) {
                    rows_left = rows_left > 4 ? rows_left - 4 : 0u;
                    if (--left == 0) {
                        left = len;
                        start_streams();
                    }
                }
            }
        }
        if (p.stages == 2) {
            stage ^= 1;
        } else {
            __syncwarp();                                       // every lane is done with the only window
            next_unit();
        }
        tk = n_tk;
        sub = n_sub;
        tp = n_tp;
        t0 = n_t0;
        two = n_two;
    }
}

// One warp per tile: rows [lowest, lowest + depth) of the byte block that the symbols from an entry point to the next touch,
// and every stream's next byte relative to that.  rows: in, bytes left; out, the index of the next byte in the span.
__global__ void __launch_bounds__(256) k_entry_spans(uint16_t *rows, uint32_t *spans, uint32_t tiles, uint32_t subs, uint32_t *cap) {
    const uint32_t t = blockIdx.x * 8 + (threadIdx.x >> 5), lane = lane_id();
    if (t >= tiles) return;
    uint32_t *r = reinterpret_cast<uint32_t *>(rows + (size_t)t * subs * 64) + lane;     // two streams a lane
    uint32_t cur = r[0], deepest = 0;
    for (uint32_t s = 0; s < subs; ++s) {
        const uint32_t nxt = s + 1 < subs ? r[(s + 1) * 32] : 0u;
        const uint32_t hi = __reduce_max_sync(kFull, max(cur & 0xFFFFu, cur >> 16));
        const uint32_t lo = min(hi, __reduce_min_sync(kFull, min(nxt & 0xFFFFu, nxt >> 16)));
        auto rel = [&](uint32_t left) { return left > lo + 1 ? left - 1 - lo : 0u; };
        r[s * 32] = rel(cur & 0xFFFFu) | rel(cur >> 16) << 16;
        if (lane == 0) spans[(size_t)t * subs + s] = lo | (hi - lo) << 16;
        deepest = max(deepest, hi - lo);
        cur = nxt;
    }
    if (lane == 0) atomicMax(cap, deepest);
}

// ------------------------------------------------------------------------ host

template <bool BF16, bool EDGE, bool INDEX, bool ENTRY, bool AHEAD>
static int launch_dec4_as(const Dec4Args &p, uint32_t blocks, uint32_t warps, size_t smem, int max_smem, void *out,
                       cudaStream_t s) {
    static SmemLimit lim = {};
    if (int rc = ensure_smem_limit(lim, (const void *)k_decode4<BF16, EDGE, INDEX, ENTRY, AHEAD>, (size_t)max_smem)) return rc;
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
    CI_CUDA(cudaLaunchKernelEx(&cfg, k_decode4<BF16, EDGE, INDEX, ENTRY, AHEAD>, p, out));
    return CI_OK;
}

template <bool BF16, bool EDGE, bool INDEX, bool ENTRY>
static int launch_dec4(const Dec4Args &p, uint32_t blocks, uint32_t warps, size_t smem, int max_smem, void *out,
                       cudaStream_t s) {
    return warps <= kDec4AheadWarps ? launch_dec4_as<BF16, EDGE, INDEX, ENTRY, true>(p, blocks, warps, smem, max_smem, out, s)
                                    : launch_dec4_as<BF16, EDGE, INDEX, ENTRY, false>(p, blocks, warps, smem, max_smem, out, s);
}

static int decode4(const DecArgs &a, uint32_t max_tile_len, bool bf16, void *out, uint32_t step,
                   uint32_t *entry_states, uint16_t *entry_rows, cudaStream_t s);

int build_entry_points(const DecArgs &a, uint32_t max_tile_len, uint32_t step, uint32_t *d_states, uint16_t *d_rows,
                       uint32_t *d_spans, uint32_t *d_cap, cudaStream_t s) {
    const int rc = decode4(a, max_tile_len, false, nullptr, step, d_states, d_rows, s);
    if (rc) return rc;
    CI_CUDA(cudaMemsetAsync(d_cap, 0, sizeof(uint32_t), s));
    const uint32_t tiles = a.g.tiles_k * a.g.tiles_n;
    k_entry_spans<<<(tiles + 7) / 8, 256, 0, s>>>(d_rows, d_spans, tiles, a.g.half / step, d_cap);
    CI_LAUNCH_CHECK(k_entry_spans);
    return CI_OK;
}

// Returns CI_OK when it launched, 1 when the tensor does not qualify, < 0 on error.
int launch_decode4(const DecArgs &a, uint32_t max_tile_len, bool bf16, void *out, cudaStream_t s) {
    return decode4(a, max_tile_len, bf16, out, 0, nullptr, nullptr, s);
}

constexpr uint32_t kDec4Fixed = 2 * kLutBytes + kDec4BarBytes;  // up to one table size is lost to the table's alignment

// A round of w warps, as round_cost: up to a warp a scheduler it is the chain of Quad::step_ahead (512 symbols a stream took 39 us
// with one to four warps, 60 with five, 62 with six; with step() 61, 72 and 74).
static double round4(uint32_t w) { return w <= 4 ? 4.6 : w <= kDec4AheadWarps ? 8.2 : round_cost(w, 0.9); }

// The warp count with the cheapest rounds; a second window where it costs no warp that pays.
static double plan_rounds(Dec4Args &p, uint32_t man_bytes, int max_smem, uint32_t &warps) {
    const uint32_t P = (uint32_t)sm_count(), room = (uint32_t)max_smem - kDec4Fixed;
    double best = 0.0;
    warps = 0;
    for (uint32_t stages = 2; stages >= 1; --stages) {
        uint32_t w_max = room / (stages * p.stage_bytes + man_bytes);
        if (w_max > kDec4Warps) w_max = kDec4Warps;
        for (uint32_t w = 1; w <= w_max; ++w) {
            const uint32_t units = (p.total + P - 1) / P;
            // The last round of fewer warps overlaps the ends of full ones and costs more than its own: 7944 x 4328 at tile height
            // 64 (58 units) takes 3.6 rounds of 16 warps 33.9 us, 2.9 of 20 31.0; 4096 x 22016 4.7 of 16 72.5, 5 of 15 70.2.
            const double tail = units % w ? 0.5 * (round4(w) + round4(units % w)) + 0.5 : 0.0;
            const double cost = ((units / w) * round4(w) + tail) * (stages == 1 ? 1.02 : 1.0);
            if (warps == 0 || cost < best) { best = cost; warps = w; p.stages = stages; }
        }
    }
    return best;
}

static bool has_entries(const DecArgs &a, bool bf16) {
    const Geom &g = a.g;
    return bf16 && a.entry_step != 0 && a.entry_cap != 0 && g.half > a.entry_step && g.half % a.entry_step == 0 &&
           a.entry_step % kChunkRows == 0 &&
           ((reinterpret_cast<uintptr_t>(a.entry_states) | reinterpret_cast<uintptr_t>(a.entry_rows)) & 15u) == 0;
}

// Bytes of one window and the initial states (with entry points also the rows of the next bytes).
static uint32_t stage_bytes4(uint32_t cap_rows, bool entry) { return (cap_rows * 128u + (entry ? 768u : 512u) + 127u) & ~127u; }

double decode4_cost(const DecArgs &a, uint32_t max_tile_len, bool bf16) {
    const Geom &g = a.g;
    int dev = 0, max_smem = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess)
        return 0.0;
    const bool entry = has_entries(a, bf16);
    Dec4Args p;
    p.stage_bytes = stage_bytes4(entry ? a.entry_cap : max_tile_len, entry);
    p.total = g.tiles_k * ((g.tiles_n + 1) / 2) * (entry ? g.half / a.entry_step : 1u);
    uint32_t warps;
    double cost = plan_rounds(p, bf16 ? kManBytes : 0u, max_smem, warps);
    if (warps == 0) return 0.0;                                 // too deep for a window of four streams a lane
    if (warps <= kDec4AheadWarps && (g.K % g.th != 0 || g.N % 4 != 0)) cost *= 1.3;     // the chain of EDGE is longer
    // A launch takes 1 us longer to its first symbol than one of decode2.cu: 2048 x 2048 at tile height 128 6.6 us there, 8.2 here.
    if (warps <= kDec4AheadWarps && !entry) cost += 64.0 / g.half;
    return entry ? cost * a.entry_step / g.half : cost;         // per 64 symbols of the whole stream
}

static int decode4(const DecArgs &a, uint32_t max_tile_len, bool bf16, void *out, uint32_t step,
                   uint32_t *entry_states, uint16_t *entry_rows, cudaStream_t s) {
    const Geom &g = a.g;
    if (g.tw != 32 || g.th % 16 != 0 || max_tile_len == 0) return 1;
    if (!a.stream_aligned || (reinterpret_cast<uintptr_t>(a.states) & 15u)) return 1;
    if (bf16 && (reinterpret_cast<uintptr_t>(a.mantissa) & 15u)) return 1;
    int dev = 0, max_smem = 0;
    CI_CUDA(cudaGetDevice(&dev));
    CI_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    Dec4Args p;
    p.a = a;
    const bool entry = has_entries(a, bf16);
    p.cap_rows = entry ? a.entry_cap : max_tile_len;
    p.stage_bytes = stage_bytes4(p.cap_rows, entry);
    p.pairs_n = (g.tiles_n + 1) / 2;
    p.step = entry ? a.entry_step : step;
    p.subs = p.step ? g.half / p.step : 0;
    p.total = g.tiles_k * p.pairs_n * (entry ? p.subs : 1u);
    p.entry_states = entry ? const_cast<uint32_t *>(a.entry_states) : entry_states;
    p.entry_rows = entry ? const_cast<uint16_t *>(a.entry_rows) : entry_rows;
    p.entry_spans = a.entry_spans;
    const uint32_t P = (uint32_t)sm_count(), man_bytes = bf16 ? kManBytes : 0u;
    uint32_t warps = 0;
    plan_rounds(p, man_bytes, max_smem, warps);
    if (warps == 0) return 1;
    uint32_t blocks = (p.total + warps - 1) / warps;
    if (blocks > P) blocks = P;
    const size_t smem = kDec4Fixed + (size_t)warps * (p.stages * p.stage_bytes + man_bytes);
    p.vec = a.ld % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & (bf16 ? 7u : 3u)) == 0;
    const bool edge = g.K % g.th != 0 || g.N % 4 != 0 || !p.vec;
    if (step) return launch_dec4<false, false, true, false>(p, blocks, warps, smem, max_smem, nullptr, s);
    if (entry) return edge ? launch_dec4<true, true, false, true>(p, blocks, warps, smem, max_smem, out, s)
                           : launch_dec4<true, false, false, true>(p, blocks, warps, smem, max_smem, out, s);
    if (bf16) return edge ? launch_dec4<true, true, false, false>(p, blocks, warps, smem, max_smem, out, s)
                          : launch_dec4<true, false, false, false>(p, blocks, warps, smem, max_smem, out, s);
    return edge ? launch_dec4<false, true, false, false>(p, blocks, warps, smem, max_smem, out, s)
                : launch_dec4<false, false, false, false>(p, blocks, warps, smem, max_smem, out, s);
}

}  // namespace ci
