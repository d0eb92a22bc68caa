// Fused decode + row gather for 32-wide tiles, four streams per lane: out[i,:] = W[ids[i],:].
// Replaces fused_rans_embedding_kernel_ilp2 (comp_inference/embedding_triton.py:170-275); ids outside
// [0,K) produce a zero row (embedding_triton.py:203-210).
//
// A stream cannot be entered in the middle: to emit row r of a tile the (r mod tile_h/2) symbols above it
// in its half-tile stream are decoded and dropped.  Work unit: one warp takes (token, 128 columns) = the
// token's half (top or bottom) of four neighbouring tiles = 128 streams; lane l owns the four adjacent
// columns 4l .. 4l+3 of the strip.  The four 32-byte-wide half slices of the tiles' byte blocks are
// copied by cp.async side by side into a window of 128-byte rows, which gives every lane a word column
// (a shared-memory bank) of its own, so the renormalisation byte loads never conflict; the row's four
// weights leave as one 8-byte store.  Only the rows a stream can reach are copied: two bytes a symbol at most.
//
// At the tile heights that suit gathers only a few symbols are decoded per task, so what bounds the kernel is the work
// around them.  A warp therefore takes many tasks: eight at a time their ids are read and their tiles'
// offsets and depths fetched, one tile per lane, while the eight before them are worked off; a task then costs two
// shuffles for its lane's own tile, and no division.  Byte windows, initial states and the row's sign+mantissa bytes are
// fetched one task ahead.  Tall tiles are entered at the entry point before the row where the caller has them.  Measured on
// a B200, 4096 ids of 32000 x 4096 at tile height 16: 148 us with one task at a time, divisions in 64 bits and eight
// shuffles per task -> 71.
#include "embedding.cuh"
#include "ptx.cuh"

namespace ci {

constexpr uint32_t kEmb4Warps = 24;          // x 32 threads x 80 registers
constexpr uint32_t kEmb4BarBytes = 512;      // up to 24 warps x 2 stages x 8 B, the table's barrier

struct Emb4Args {
    EmbArgs a;
    uint32_t cap_rows;     // rows of a byte window (>= every tile_max_len)
    uint32_t stage_bytes;
    uint32_t stages;       // windows per warp: 2, or 1 for tall tiles
    uint32_t blocks_n;     // 128-column blocks per row = ceil(tiles_n / 4)
    uint32_t total;        // tasks, the column block running fastest
    uint32_t out_vec;      // rows of the output can be written as 8-byte quads
    uint32_t subs;         // ENTRY: entry points per half tile
};

// ENTRY: streams are entered at the entry point before the row (tall tiles), not at their start.
// RAGGED: the last block of 128 columns lacks tiles.  A lane without one decodes the block's first tile along: real symbols,
// where random ones would take the branch for a second byte at every step.  (An instantiation of its own: in all of them it cost
// 2 %, 87.4 us to 89.3 at 4096 ids of 32000 x 4096.)
template <bool ENTRY, bool RAGGED>
__global__ void __launch_bounds__(kEmb4Warps * 32, 1) k_embedding4(const __grid_constant__ Emb4Args p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const EmbArgs &a = p.a;
    const Geom &g = a.g;
    const uint32_t W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = lane_id();
    const uint32_t smem_s = smem_u32(smem);
    // The table sits on a 16 KB boundary of the shared window: an entry's address is then
    // (state << 2 & 0x3FFC) | base, without an addition.
    const uint32_t lut_s = (smem_s + kLutBytes - 1) & ~(kLutBytes - 1);
    uint32_t *s_lut = reinterpret_cast<uint32_t *>(smem + (lut_s - smem_s));
    const uint32_t lut_bar = lut_s + kLutBytes + kEmb4BarBytes - 16;
    start_lut(lut_s, lut_bar, a.lut);
    const uint32_t wbase_s = lut_s + kLutBytes + kEmb4BarBytes + warp * p.stages * p.stage_bytes;
    const uint32_t bar_base = lut_s + kLutBytes + warp * 16;
    // Task n of this warp is gw + n * n_warps, the CTA running fastest in gw: the symbols to drop are a matter of the id, and a
    // run of consecutive tasks has one or two ids.  4096 ids of 32000 x 4096, runs -> this: tile height 16 86 us -> 72, 128
    // 460 -> 336, 1024 (2048 ids) 292 -> 209.
    const uint32_t n_warps = gridDim.x * W;
    const uint32_t gw = warp * gridDim.x + blockIdx.x, lo = 0, hi = gw < p.total ? (p.total - gw + n_warps - 1) / n_warps : 0u;
    const uint32_t tsel = lane >> 3, quad = lane & 7;           // tile of the block, column quad inside it

    if (lane == 0) {
        mbar_init(bar_base, 32);                                // one arrival per lane when its copies have landed
        mbar_init(bar_base + 8, 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (a.lut == nullptr) load_lut(s_lut, nullptr, a.tables, a.slot_map);
    __syncthreads();
    // The ids (and the output buffer) may be products of the previous kernel of the stream: with
    // programmatic dependent launch wait for it here, after the table load that does not depend on it.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    (void)wait_lut(lut_bar, a.lut);
    if (lo >= hi) return;

    // A batch of eight tasks from `first` on: lane l holds what tile l % 4 of task first + l / 4 needs.
    struct Batch {
        uint32_t ti, cb;       // token and column block of the lane's task
        uint32_t row;          // its row of the table; ~0 when the id is outside
        uint32_t off, ml;      // the lane's tile: byte offset, depth (0 for a tile that is not read)
    };
    auto load_ids = [&](uint32_t first, Batch &b) {
        const uint32_t t = gw + min(first + (lane >> 2), hi - 1) * n_warps;
        b.ti = t / p.blocks_n;
        b.cb = t - b.ti * p.blocks_n;
        const int64_t id = __ldg(a.ids + b.ti);
        b.row = id >= 0 && id < (int64_t)g.K ? (uint32_t)id : 0xFFFFFFFFu;
    };
    auto load_tiles = [&](Batch &b) {
        const uint32_t tn = b.cb * 4 + (lane & 3);
        b.off = b.ml = 0;
        if (b.row != 0xFFFFFFFFu && tn < g.tiles_n) {
            const uint32_t tk = b.row / g.th;
            const size_t tile = (size_t)tk * g.tiles_n + tn;
            b.off = __ldg(a.tile_offsets + tile);
            if constexpr (ENTRY) {
                const uint32_t rel = b.row - tk * g.th, inner = rel >= g.half ? rel - g.half : rel;
                b.ml = enter_span(__ldg(a.entry_spans + tile * p.subs + inner / a.entry_step), __ldg(a.tile_max_lens + tile), b.off);
            } else {
                b.ml = __ldg(a.tile_max_lens + tile);
            }
        }
        if (b.ml > p.cap_rows) b.ml = 0;                        // metadata disagrees with the declared maximum
    };

    // What the lane knows about one task.
    struct Task {
        uint32_t ti, cb, inner, ml;
        bool live;             // the id is inside the table
        uint4 states;
        uint32_t man;
        uint2 rows;            // ENTRY: next byte's row of every stream
    };
    // The tile of the column block whose streams this lane decodes.
    auto tile_of = [&](uint32_t cb) { return !RAGGED || cb * 4 + tsel < g.tiles_n ? tsel : 0u; };
    // Task k of the batch: its copies into `stage`, its states and sign+mantissa bytes.
    auto open = [&](const Batch &b, uint32_t k, uint32_t stage, Task &t) {
        t.ti = __shfl_sync(kFull, b.ti, 4 * k);
        t.cb = __shfl_sync(kFull, b.cb, 4 * k);
        const uint32_t tsel_d = tile_of(t.cb), src_lane = 4 * k + tsel_d;
        const uint32_t row = __shfl_sync(kFull, b.row, 4 * k), off = __shfl_sync(kFull, b.off, src_lane);
        t.ml = __shfl_sync(kFull, b.ml, src_lane);
        const uint32_t tn = t.cb * 4 + tsel_d;
        t.live = row != 0xFFFFFFFFu;
        const uint32_t tk = row / g.th, rel = row - tk * g.th, h = rel >= g.half ? 1u : 0u;
        t.inner = t.live ? rel - h * g.half : 0u;
        t.states = make_uint4(kRansL, kRansL, kRansL, kRansL);
        t.man = 0;
        if (t.live) {
            const size_t tile = (size_t)tk * g.tiles_n + tn;
            uint32_t rows;
            if constexpr (ENTRY) {
                const size_t e = (tile * p.subs + t.inner / a.entry_step) * 64 + h * 32 + quad * 4;
                t.inner %= a.entry_step;
                t.states = __ldg(reinterpret_cast<const uint4 *>(a.entry_states + e));
                t.rows = __ldg(reinterpret_cast<const uint2 *>(a.entry_rows + e));
                rows = t.ml;
            } else {
                t.states = __ldg(reinterpret_cast<const uint4 *>(a.states + tile * 64 + h * 32 + quad * 4));
                rows = min(t.ml, 2 * t.inner + 2);
            }
            t.man = __ldg(reinterpret_cast<const uint32_t *>(a.mantissa + tile * (g.th * 32) + rel * 32 + quad * 4));
            // eight lanes a tile: pieces of 16 bytes, two a row, from the last row upwards
            const uint32_t skip = t.ml - rows;
            const uint8_t *src = a.stream + off + h * 32 + (size_t)(skip + (quad >> 1)) * 64 + (quad & 1) * 16;
            const uint32_t dst = wbase_s + stage * p.stage_bytes + (skip + (quad >> 1)) * 128 + tsel * 32 + (quad & 1) * 16;
            for (uint32_t i = tsel_d == tsel ? quad >> 1 : rows; i < rows; i += 4)
                cp_async16(dst + (i - (quad >> 1)) * 128, src + (size_t)(i - (quad >> 1)) * 64);
        }
        cp_async_arrive(bar_base + stage * 8);
    };

    Batch cur, nxt;
    load_ids(lo, cur);
    load_tiles(cur);
    Task t, n;
    open(cur, 0, 0, t);
    uint32_t parity0 = 0, parity1 = 0, stage = 0;
    for (uint32_t first = lo; first < hi; first += 8) {
        const bool more = first + 8 < hi;
        const uint32_t count = min(8u, hi - first);
        if (more) load_ids(first + 8, nxt);
#pragma unroll 1
        for (uint32_t k = 0; k < count; ++k) {
            if (k == 2 && more) load_tiles(nxt);                // two tasks after its ids were asked for
            const bool last = k + 1 == count;
            __syncwarp();                                       // every lane is done with the other window
            if (p.stages == 2) {
                if (!last) open(cur, k + 1, stage ^ 1, n);
                else if (more) open(nxt, 0, stage ^ 1, n);
            }
            const uint32_t win_s = wbase_s + stage * p.stage_bytes;
            const bool ok = mbar_wait(bar_base + stage * 8, stage ? parity1 : parity0);
            if (stage) parity1 ^= 1; else parity0 ^= 1;
            Quad z;
            z.s[0] = t.states.x;
            z.s[1] = t.states.y;
            z.s[2] = t.states.z;
            z.s[3] = t.states.w;
            const uint32_t start = win_s + tile_of(t.cb) * 32 + quad * 4 + (!ENTRY && t.ml ? (t.ml - 1) * 128 : 0u);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) z.p[j] = start + j;
            if constexpr (ENTRY) {
                const uint32_t top = p.cap_rows - 1;
                if (t.live) {
                    z.p[0] += min(t.rows.x & 0xFFFFu, top) * 128;
                    z.p[1] += min(t.rows.x >> 16, top) * 128;
                    z.p[2] += min(t.rows.y & 0xFFFFu, top) * 128;
                    z.p[3] += min(t.rows.y >> 16, top) * 128;
                }
            }
            // The rows above the wanted one, four at a time: the loop around one costs 5 % (tile height 128: 336 us -> 321).
            const uint32_t drop = __shfl_sync(kFull, t.inner, 0);
            uint32_t i = 0;
#pragma unroll 1
            for (; i + 4 <= drop; i += 4) {
                uint32_t e[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) z.step(lut_s, e);
                if ((i & 12) == 12) z.clamp(win_s);
            }
#pragma unroll 1
            for (; i < drop; ++i) {
                uint32_t e[4];
                z.step(lut_s, e);
            }
            uint32_t w01 = 0, w23 = 0;
            if (ok && t.live) {
                const uint32_t mask = (kProbScale - 1) << 2;
                const uint32_t e0 = lds_u32(((z.s[0] << 2) & mask) | lut_s), e1 = lds_u32(((z.s[1] << 2) & mask) | lut_s);
                const uint32_t e2 = lds_u32(((z.s[2] << 2) & mask) | lut_s), e3 = lds_u32(((z.s[3] << 2) & mask) | lut_s);
                const uint32_t a01 = __byte_perm(e0, e1, 0x6521), a23 = __byte_perm(e2, e3, 0x6521);
                w01 = exp_or_man(a01 << 3, __byte_perm(t.man, 0u, 0x1100));
                w23 = exp_or_man(a23 << 3, __byte_perm(t.man, 0u, 0x3322));
            }
            const uint32_t col0 = t.cb * 128 + tsel * 32 + quad * 4;
            if (col0 < g.N) {
                uint16_t *dst = a.out + (size_t)t.ti * a.ldo + col0;
                if (p.out_vec && col0 + 4 <= g.N) {
                    *reinterpret_cast<uint2 *>(dst) = make_uint2(w01, w23);
                } else {
                    const uint32_t v[4] = {w01 & 0xFFFFu, w01 >> 16, w23 & 0xFFFFu, w23 >> 16};
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (col0 + c < g.N) dst[c] = (uint16_t)v[c];
                }
            }
            if (p.stages == 2) {
                stage ^= 1;
            } else {
                __syncwarp();                                   // every lane is done with the only window
                if (!last) open(cur, k + 1, 0, n);
                else if (more) open(nxt, 0, 0, n);
            }
            t = n;
        }
        cur = nxt;
    }
}

// ------------------------------------------------------------------------ host

int launch_embedding4(const EmbArgs &a, uint32_t max_tile_len, cudaStream_t s) {
    const Geom &g = a.g;
    if (g.tw != 32 || g.th % 2 != 0 || max_tile_len == 0) return 1;
    if ((reinterpret_cast<uintptr_t>(a.stream) & 15u) || (reinterpret_cast<uintptr_t>(a.states) & 15u) ||
        (reinterpret_cast<uintptr_t>(a.mantissa) & 3u))
        return 1;
    int dev = 0, max_smem = 0;
    CI_CUDA(cudaGetDevice(&dev));
    CI_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    Emb4Args p;
    p.a = a;
    const bool entry = a.entry_step != 0 && a.entry_cap != 0 && g.half > a.entry_step && g.half % a.entry_step == 0 &&
                       ((reinterpret_cast<uintptr_t>(a.entry_states) | reinterpret_cast<uintptr_t>(a.entry_rows)) & 15u) == 0;
    p.cap_rows = entry ? a.entry_cap : max_tile_len;
    p.subs = entry ? g.half / a.entry_step : 1u;
    p.stage_bytes = (p.cap_rows * 128u + 127u) & ~127u;
    p.blocks_n = (g.tiles_n + 3) / 4;
    p.out_vec = ((reinterpret_cast<uintptr_t>(a.out) & 7u) == 0 && (a.ldo & 3) == 0) ? 1u : 0u;
    const uint32_t fixed = 2 * kLutBytes + kEmb4BarBytes;           // up to one table size is lost to the table's alignment
    const uint32_t room = (uint32_t)max_smem - fixed;
    if (room < p.stage_bytes) return 1;
    p.stages = room / (2 * p.stage_bytes) >= 12 ? 2 : 1;        // a deep window is worth doubling while 12 warps still fit
    uint32_t w_max = room / (p.stages * p.stage_bytes);
    if (w_max > kEmb4Warps) w_max = kEmb4Warps;
    const bool ragged = g.tiles_n % 4 != 0;
    static SmemLimit lim[4] = {};
    void (*const kernel)(Emb4Args) = entry ? (ragged ? k_embedding4<true, true> : k_embedding4<true, false>)
                                           : (ragged ? k_embedding4<false, true> : k_embedding4<false, false>);
    if (int rc = ensure_smem_limit(lim[entry + 2 * ragged], (const void *)kernel, (size_t)max_smem)) return rc;
    const uint32_t P = (uint32_t)sm_count();
    const uint64_t ids_per_launch = 0x40000000ull / p.blocks_n;     // task numbers fit 32 bits
    for (uint64_t i0 = 0; i0 < a.n_ids; i0 += ids_per_launch) {
        const uint64_t n = a.n_ids - i0 < ids_per_launch ? a.n_ids - i0 : ids_per_launch;
        p.a.ids = a.ids + i0;
        p.a.out = a.out + i0 * a.ldo;
        p.total = (uint32_t)(n * p.blocks_n);
        uint32_t blocks = p.total < P ? p.total : P, warps = (p.total + blocks - 1) / blocks;
        if (warps > w_max) warps = w_max;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(warps * 32);
        cfg.dynamicSmemBytes = fixed + (size_t)warps * p.stages * p.stage_bytes;
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        CI_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    }
    return CI_OK;
}

}  // namespace ci
