// Fused decode + row gather for 32-wide tiles where many ids share streams: out[i,:] = W[ids[i],:].
// Replaces fused_rans_embedding_kernel_ilp2 (comp_inference/embedding_triton.py:170-275) as embedding4.cu does, whose layout of
// lanes, windows and columns this is; ids outside [0,K) produce a zero row (embedding_triton.py:203-210).
//
// To emit row r of a tile the symbols above it in its half-tile stream have to be decoded (from the entry point before, where
// there is one).  embedding4.cu does that for every id; here up to eight ids of one half tile, or of one span between entry
// points, a "bin", are one group: the streams are decoded once, down to the group's last row, and every row that an id asks for
// leaves on the way.  Work unit: (group, 128 columns), one warp.
//
// The groups are made by every CTA for itself, in shared memory: a counting sort of the ids by bin.  It costs 3 us and 148
// reads of the ids from L2, and no launch, no workspace and no second pass over memory; groups come in the order of their bins, so
// that all CTAs mean the same ones.  Bins of more than 128 ids -- padding, tokens that repeat -- are ordered by the ids' ranks: with a
// sort of such a bin by the whole CTA, a barrier a step, 4096 ids of which half are one token took 16000 x 2048 at tile height
// 16 49.3 us and now 33.3, all of them one 57.4 -> 22.8, in Zipf's distribution 44.0 -> 35.4; 32000 x 4096 there 74.1 -> 58.1,
// 63.5 -> 29.2, 66.1 -> 58.5.
//
// Bound by instructions (76 % of the issue slots at tile height 16, where a group is 1.6 ids and 5 rows), 680 a task there, of
// which the decode step 300.
#include <math.h>

#include "embedding.cuh"
#include "ptx.cuh"

namespace ci {

constexpr uint32_t kEmbGWarps = 24;          // x 32 threads x 80 registers
constexpr uint32_t kEmbGBarBytes = 256;      // the table's barrier, the number of groups, the warps' sums of the scan
constexpr uint32_t kEmbGIds = 4096;          // ids of one launch
constexpr uint32_t kEmbGroup = 8;            // ids of a group
constexpr uint32_t kEmbGRanked = 128;        // ids of a bin that a warp sorts
constexpr uint32_t kEmbGSorts = 512;         // at least kEmbGIds / (kEmbGroup + 1)
constexpr uint32_t kEmbGBins = 16384;        // counters of the sort

struct EmbGArgs {
    EmbArgs a;
    uint32_t cap_rows;     // rows of a byte window (>= every tile_max_len)
    uint32_t stage_bytes;  // window and sign+mantissa bytes of a group
    uint32_t stages;       // windows per warp
    uint32_t blocks_n;     // 128-column blocks per row
    uint32_t n;            // ids
    uint32_t seg, bins;    // rows of a bin, bins of the table
    uint32_t subs;         // ENTRY: bins per half tile, else 1
    uint32_t out_vec;      // rows of the output can be written as 8-byte quads
};

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All copies of this thread but those of the last group have landed.
__device__ __forceinline__ void cp_async_wait_but_last() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// ENTRY, RAGGED: see embedding4.cu.
template <bool ENTRY, bool RAGGED>
__global__ void __launch_bounds__(kEmbGWarps * 32, 1) k_embedding_group(const __grid_constant__ EmbGArgs p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const EmbArgs &a = p.a;
    const Geom &g = a.g;
    const uint32_t W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = lane_id();
    const uint32_t smem_s = smem_u32(smem);
    const uint32_t lut_s = (smem_s + kLutBytes - 1) & ~(kLutBytes - 1);
    const uint32_t lut_bar = lut_s + kLutBytes;
    start_lut(lut_s, lut_bar, a.lut);
    uint32_t *const head = reinterpret_cast<uint32_t *>(smem + (lut_bar - smem_s));   // [4]: groups, [5]: sorts, [6]: bins of very many ids, [8..]: the scan's sums
    uint32_t *const tokens = head + kEmbGBarBytes / 4;          // [n]: row in the bin << 16 | id
    uint32_t *const groups = tokens + p.n;                      // [<= n]: bin << 16 | first token << 3 | ids - 1
    uint32_t *const sorts = groups + p.n;                       // tokens to sort: first one << 16 | in order of ids << 15 | their number
    uint32_t *const count = sorts + kEmbGSorts;                 // [bins + 1]: ids of a bin, later where the next bin's begin (low half)
    const uint32_t windows_s = (smem_u32(count) + (p.bins + 1) * 4 + 127) & ~127u;
    const uint32_t wbase_s = windows_s + warp * p.stages * p.stage_bytes;
    const uint32_t man_off = p.cap_rows * 128;

    for (uint32_t i = threadIdx.x; i <= p.bins; i += blockDim.x) count[i] = 0;
    if (threadIdx.x < 2) head[5 + threadIdx.x] = 0;
    if (a.lut == nullptr) load_lut(reinterpret_cast<uint32_t *>(smem + (lut_s - smem_s)), nullptr, a.tables, a.slot_map);
    __syncthreads();
    // The ids (and the output buffer) may be products of the previous kernel of the stream.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // ---- groups: count, scan, place; ids outside the table are the bin behind the last one --------------------
    auto row_of = [&](uint32_t i) {
        const int64_t id = __ldg(a.ids + i);
        return id >= 0 && id < (int64_t)g.K ? (uint32_t)id : 0xFFFFFFFFu;
    };
    auto bin_of = [&](uint32_t row) { return row != 0xFFFFFFFFu ? row / p.seg : p.bins; };
#pragma unroll 4
    for (uint32_t i = threadIdx.x; i < p.n; i += blockDim.x) atomicAdd(count + bin_of(row_of(i)), 1u);
    __syncthreads();
    {
        const uint32_t per = p.bins / blockDim.x + 1, b0 = min(threadIdx.x * per, p.bins + 1), b1 = min(b0 + per, p.bins + 1);
        uint32_t mine = 0;                                      // groups << 16 | ids
        for (uint32_t b = b0; b < b1; ++b) mine += count[b] + ((count[b] + kEmbGroup - 1) / kEmbGroup << 16);
        uint32_t run = mine;
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t o = __shfl_up_sync(kFull, run, d);
            if (lane >= d) run += o;
        }
        if (lane == 31) head[8 + warp] = run;
        __syncthreads();
        for (uint32_t w = 0; w < warp; ++w) run += head[8 + w];
        run -= mine;
        uint32_t at = run & 0xFFFFu, grp = run >> 16;
        for (uint32_t b = b0; b < b1; ++b) {
            const uint32_t k = count[b];
            count[b] = at;
            for (uint32_t j = 0; j < k; j += kEmbGroup) groups[grp++] = b << 16 | (at + j) << 3 | (min(k - j, kEmbGroup) - 1);
            at += k;
            if (k > kEmbGRanked) {                              // its number, and behind it where it ends
                count[b] = (atomicAdd(head + 6, 1u) + 1) << 16 | at;
                for (uint32_t j = 0; j < k; j += kEmbGRanked)
                    sorts[atomicAdd(head + 5, 1u)] = (at - k + j) << 16 | 0x8000u | min(k - j, kEmbGRanked);
            } else if (k > kEmbGroup) {
                sorts[atomicAdd(head + 5, 1u)] = (at - k) << 16 | k;
            }
        }
        if (threadIdx.x == blockDim.x - 1) head[4] = grp;
    }
    __syncthreads();
    auto token_of = [&](uint32_t i, uint32_t row, uint32_t bin) { return (row != 0xFFFFFFFFu ? row - bin * p.seg : 0u) << 16 | i; };
    const uint32_t heavy = head[6];                             // bins of more ids than a warp sorts
    if (heavy == 0) {
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < p.n; i += blockDim.x) {
            const uint32_t row = row_of(i), bin = bin_of(row);
            tokens[atomicAdd(count + bin, 1u)] = token_of(i, row, bin);
        }
    } else {
        // Tokens that repeat, padding, ids outside the table.  In such a bin an id's place is its rank among the bin's ids: from a
        // bit for every id of the launch, in the windows' memory, which nobody uses yet, and the number of bits before each word.
        const uint32_t words = (p.n + 31) / 32;
        uint32_t *const bits = reinterpret_cast<uint32_t *>(smem + (windows_s - smem_s));      // [heavy][words]
        uint16_t *const before = reinterpret_cast<uint16_t *>(bits + heavy * words);
        for (uint32_t i = threadIdx.x; i < heavy * words; i += blockDim.x) bits[i] = 0;
        __syncthreads();
#pragma unroll 4
        for (uint32_t i0 = warp * 32; i0 < p.n; i0 += blockDim.x) {
            const uint32_t i = i0 + lane, row = i < p.n ? row_of(i) : 0xFFFFFFFFu, bin = bin_of(row);
            const uint32_t l = i < p.n ? count[bin] >> 16 : 0u;
            if (l == 0 && i < p.n) tokens[atomicAdd(count + bin, 1u)] = token_of(i, row, bin);
            const uint32_t same = __match_any_sync(kFull, l);
            if (l != 0 && lane == __ffs(same) - 1) bits[(l - 1) * words + i0 / 32] = same;     // a word is one warp's
        }
        __syncthreads();
        for (uint32_t l = warp; l < heavy; l += W) {
            uint32_t sum = 0;
            for (uint32_t w0 = 0; w0 < words; w0 += 32) {
                const uint32_t mine = w0 + lane < words ? __popc(bits[l * words + w0 + lane]) : 0u;
                uint32_t run = mine;
                for (uint32_t d = 1; d < 32; d <<= 1) {
                    const uint32_t o = __shfl_up_sync(kFull, run, d);
                    if (lane >= d) run += o;
                }
                if (w0 + lane < words) before[l * words + w0 + lane] = (uint16_t)(sum + run - mine);
                sum += __shfl_sync(kFull, run, 31);
            }
        }
        __syncthreads();
#pragma unroll 4
        for (uint32_t i = threadIdx.x; i < p.n; i += blockDim.x) {
            const uint32_t row = row_of(i), bin = bin_of(row), l = count[bin] >> 16;
            if (l == 0) continue;
            const uint32_t first = bin ? count[bin - 1] & 0xFFFFu : 0u, at = (l - 1) * words + i / 32;
            tokens[first + before[at] + __popc(bits[at] & ((1u << (i & 31)) - 1))] = token_of(i, row, bin);
        }
    }
    __syncthreads();
    // A bin of more than one group in order of rows (and ids), so that every CTA splits it alike and a group's rows are near one
    // another: by rank, a warp a bin; one whose tokens are in order of ids by runs of 128.
    for (uint32_t l = warp; l < head[5]; l += W) {
        const uint32_t first = sorts[l] >> 16, k = sorts[l] & 0x7FFFu;
        if (k <= 32) {
            const uint32_t mine = lane < k ? tokens[first + lane] : 0xFFFFFFFFu;
            uint32_t rank = 0;
            for (uint32_t i = 0; i < k; ++i) rank += __shfl_sync(kFull, mine, i) < mine;
            if (lane < k) tokens[first + rank] = mine;
            continue;
        }
        uint32_t mine[kEmbGRanked / 32], rank[kEmbGRanked / 32];
#pragma unroll
        for (uint32_t j = 0; j < kEmbGRanked / 32; ++j) {
            mine[j] = lane + 32 * j < k ? tokens[first + lane + 32 * j] : 0xFFFFFFFFu;
            rank[j] = 0;
        }
        if (sorts[l] & 0x8000u) {                               // all of one row: they are in order
            const uint32_t row = tokens[first] >> 16;
            bool same = true;
#pragma unroll
            for (uint32_t j = 0; j < kEmbGRanked / 32; ++j) same &= lane + 32 * j >= k || mine[j] >> 16 == row;
            if (__all_sync(kFull, same)) continue;
        }
        for (uint32_t i = 0; i < k; ++i) {
            const uint32_t v = tokens[first + i];
#pragma unroll
            for (uint32_t j = 0; j < kEmbGRanked / 32; ++j) rank[j] += v < mine[j];
        }
        __syncwarp();
#pragma unroll
        for (uint32_t j = 0; j < kEmbGRanked / 32; ++j)
            if (lane + 32 * j < k) tokens[first + rank[j]] = mine[j];
    }
    __syncthreads();
    const uint32_t total = head[4] * p.blocks_n, n_warps = gridDim.x * W, gw = warp * gridDim.x + blockIdx.x;
    (void)wait_lut(lut_bar, a.lut);
    if (gw >= total) return;

    const uint32_t tsel = lane >> 3, quad = lane & 7;           // tile of the block, column quad inside it

    struct Desc {
        uint32_t rec, cb;      // the group, the column block
        uint32_t off, ml;      // lane j < 4: tile j of the block, byte offset and depth
    };
    // A group's bin as tile row, half, entry point.
    auto place = [&](uint32_t rec, uint32_t &tk, uint32_t &h, uint32_t &sub) {
        const uint32_t half = ENTRY ? (rec >> 16) / p.subs : rec >> 16;
        sub = ENTRY ? (rec >> 16) - half * p.subs : 0u;
        tk = half >> 1;
        h = half & 1;
    };
    const uint32_t step_grp = n_warps / p.blocks_n, step_cb = n_warps - step_grp * p.blocks_n;
    uint32_t grp = gw / p.blocks_n, cb = gw - grp * p.blocks_n; // of the task that is described next
    auto load_desc = [&](Desc &d) {
        d.cb = cb;
        d.rec = groups[grp];
        grp += step_grp;
        cb += step_cb;
        if (cb >= p.blocks_n) {
            cb -= p.blocks_n;
            ++grp;
        }
        d.off = d.ml = 0;
        const uint32_t tn = d.cb * 4 + lane;
        if (lane >= 4 || tn >= g.tiles_n || (d.rec >> 16) >= p.bins) return;
        uint32_t tk, h, sub;
        place(d.rec, tk, h, sub);
        const size_t tile = (size_t)tk * g.tiles_n + tn;
        d.off = __ldg(a.tile_offsets + tile);
        if constexpr (ENTRY) {
            d.ml = enter_span(__ldg(a.entry_spans + tile * p.subs + sub), __ldg(a.tile_max_lens + tile), d.off);
        } else {
            d.ml = __ldg(a.tile_max_lens + tile);
        }
        if (d.ml > p.cap_rows) d.ml = 0;                        // metadata disagrees with the declared maximum
    };
    struct Task {
        uint32_t cb, ml, ids;
        uint32_t tok;          // lane j < ids: row in the bin << 16 | id; else ~0
        bool live;             // ids inside the table
        uint4 states;
        uint2 rows;            // ENTRY: next byte's row of every stream
    };
    // The tile of the column block whose streams this lane decodes.
    auto tile_of = [&](uint32_t cb) { return !RAGGED || cb * 4 + tsel < g.tiles_n ? tsel : 0u; };
    auto open = [&](const Desc &d, uint32_t stage, Task &t) {
        t.cb = d.cb;
        t.ids = (d.rec & 7u) + 1;
        t.tok = lane < t.ids ? tokens[(d.rec >> 3 & 0x1FFFu) + lane] : 0xFFFFFFFFu;
        t.live = (d.rec >> 16) < p.bins;
        const uint32_t tsel_d = tile_of(t.cb), off = __shfl_sync(kFull, d.off, tsel_d);
        t.ml = __shfl_sync(kFull, d.ml, tsel_d);
        t.states = make_uint4(kRansL, kRansL, kRansL, kRansL);
        if (t.live) {
            const uint32_t last = __reduce_max_sync(kFull, lane < t.ids ? t.tok >> 16 : 0u);
            uint32_t tk, h, sub;
            place(d.rec, tk, h, sub);
            const size_t tile0 = (size_t)tk * g.tiles_n + t.cb * 4, tile = tile0 + tsel_d;
            uint32_t rows;
            if constexpr (ENTRY) {
                const size_t e = (tile * p.subs + sub) * 64 + h * 32 + quad * 4;
                t.states = __ldg(reinterpret_cast<const uint4 *>(a.entry_states + e));
                t.rows = __ldg(reinterpret_cast<const uint2 *>(a.entry_rows + e));
                rows = t.ml;
            } else {
                t.states = __ldg(reinterpret_cast<const uint4 *>(a.states + tile * 64 + h * 32 + quad * 4));
                rows = min(t.ml, 2 * last + 2);                 // two bytes a symbol at most
            }
            // eight lanes a tile: pieces of 16 bytes, two a row, from the last row upwards
            const uint32_t skip = t.ml - rows, base_s = wbase_s + stage * p.stage_bytes;
            const uint8_t *src = a.stream + off + h * 32 + (size_t)(skip + (quad >> 1)) * 64 + (quad & 1) * 16;
            uint32_t dst = base_s + (skip + (quad >> 1)) * 128 + tsel * 32 + (quad & 1) * 16;
            for (uint32_t i = tsel_d == tsel ? quad >> 1 : rows; i < rows; i += 4, dst += 512, src += 256) cp_async16(dst, src);
            // sign+mantissa bytes of the rows: eight lanes an id, two a tile
            const bool exists = !RAGGED || t.cb * 4 + (quad >> 1) < g.tiles_n;
            const uint8_t *man = a.mantissa + (tile0 + (quad >> 1)) * (g.th * 32) + (h * g.half + sub * p.seg) * 32 + (quad & 1) * 16;
#pragma unroll
            for (uint32_t s = 0; s < kEmbGroup; s += 4) {
                const uint32_t tok = __shfl_sync(kFull, t.tok, s + tsel);
                if (s + tsel < t.ids && exists) cp_async16(base_s + man_off + (s + tsel) * 128 + quad * 16, man + (tok >> 16) * 32);
            }
        }
    };

    Desc d;
    Task cur, nxt;
    load_desc(d);
    open(d, 0, cur);
    cp_async_commit();
    if (gw + n_warps < total) load_desc(d);
    uint32_t stage = 0;
    for (uint32_t t = gw; t < total; t += n_warps) {
        const bool more = t + n_warps < total;
        if (p.stages == 2) {
            __syncwarp();                                       // every lane is done with the other window
            if (more) open(d, stage ^ 1, nxt);
            cp_async_commit();
            cp_async_wait_but_last();
        } else {
            cp_async_wait();
        }
        __syncwarp();
        Desc after = d;
        if (t + 2ull * n_warps < total) load_desc(after);
        const uint32_t win_s = wbase_s + stage * p.stage_bytes, man_s = win_s + man_off + lane * 4;
        const uint32_t col0 = cur.cb * 128 + lane * 4;
        auto store = [&](uint32_t id, uint32_t w01, uint32_t w23) {
            if (col0 >= g.N) return;
            uint16_t *dst = a.out + (size_t)id * a.ldo + col0;
            if (p.out_vec && col0 + 4 <= g.N) {
                *reinterpret_cast<uint2 *>(dst) = make_uint2(w01, w23);
            } else {
                const uint32_t v[4] = {w01 & 0xFFFFu, w01 >> 16, w23 & 0xFFFFu, w23 >> 16};
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (col0 + c < g.N) dst[c] = (uint16_t)v[c];
            }
        };
        if (cur.live) {
            Quad z;
            z.s[0] = cur.states.x;
            z.s[1] = cur.states.y;
            z.s[2] = cur.states.z;
            z.s[3] = cur.states.w;
            const uint32_t start = win_s + tile_of(cur.cb) * 32 + quad * 4 + (!ENTRY && cur.ml ? (cur.ml - 1) * 128 : 0u);
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) z.p[j] = start + j;
            if constexpr (ENTRY) {
                const uint32_t top = p.cap_rows - 1;
                z.p[0] += min(cur.rows.x & 0xFFFFu, top) * 128;
                z.p[1] += min(cur.rows.x >> 16, top) * 128;
                z.p[2] += min(cur.rows.y & 0xFFFFu, top) * 128;
                z.p[3] += min(cur.rows.y >> 16, top) * 128;
            }
            // The rows that are wanted, from the first on; those between them four at a time (see embedding4.cu).
            uint32_t at = 0, row = cur.tok >> 16;               // rows decoded; the lane's row, 0xFFFF when none or done
            for (uint32_t left = cur.ids; left != 0;) {
                const uint32_t next = __reduce_min_sync(kFull, row);
                uint32_t e[4];
#pragma unroll 1
                for (; at + 4 <= next; at += 4) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) z.step(lut_s, e);
                    if ((at & 12) == 12) z.clamp(win_s);
                }
#pragma unroll 1
                for (; at < next; ++at) z.step(lut_s, e);
                z.step(lut_s, e);
                ++at;
                const uint32_t a01 = __byte_perm(e[0], e[1], 0x6521) << 3, a23 = __byte_perm(e[2], e[3], 0x6521) << 3;
                uint32_t who = __ballot_sync(kFull, row == next);
                if (row == next) row = 0xFFFFu;
                left -= __popc(who);
                for (; who != 0; who &= who - 1) {
                    const uint32_t s = __ffs(who) - 1, m = lds_u32(man_s + s * 128);
                    store(__shfl_sync(kFull, cur.tok, s) & 0xFFFFu, exp_or_man(a01, __byte_perm(m, 0u, 0x1100)),
                          exp_or_man(a23, __byte_perm(m, 0u, 0x3322)));
                }
            }
        } else {
            for (uint32_t s = 0; s < cur.ids; ++s) store(__shfl_sync(kFull, cur.tok, s) & 0xFFFFu, 0u, 0u);
        }
        if (p.stages == 2) {
            stage ^= 1;
        } else {
            __syncwarp();                                       // every lane is done with the only window
            if (more) open(d, 0, nxt);
        }
        d = after;
        cur = nxt;
    }
}

// ------------------------------------------------------------------------ host

// What groups gain in us, for ids spread evenly over the table.  Rows to decode, 128 columns each, for one id
// at a time and for groups (a bin is decoded to the last of its rows); 7.2e-5 us a row, about as much on top for a group,
// 3.5 us for the sort.  us, embedding4.cu -> groups: 32000 x 4096 at tile height 16, 2048 ids 39 -> 44, 4096 71 -> 70; at 64,
// 256 ids 18 -> 19, 1024 50 -> 41, 4096 180 -> 84; at 128, 128 ids 20 -> 20, 512 47 -> 39, 4096 327 -> 132; at 1024 with entry
// points, 4096 376 -> 148; 16000 x 2048 at 16, 2048 ids 20.6 -> 20.8, 4096 37.6 -> 29.9; 8000 x 1000 at 128, 256 ids 13.1 -> 13.3,
// 1024 34.5 -> 17.8.  (A table of a few bins would spend its time on sorting them.)  How the ids are spread is not known here.
// 4096 ids in Zipf's distribution gain too (32000 x 4096 at 16 71 -> 59, at 128 338 -> 128; 16000 x 2048 at 16 38 -> 35, 37 -> 37 where
// frequent tokens are neighbours).  Where groups pay little, a batch padded with token 0, the first of its streams, which
// embedding4.cu has at once, loses up to 3 us: half of them padding, 16000 x 2048 at 16, 4096 ids 31.0 -> 33.3, 32000 x 1024 at 64,
// 2048 ids 19.5 -> 21.9, 8000 x 1000 at 128, 512 ids 12.9 -> 16.1; 32000 x 4096 at 64, 4096 ids 113 -> 77.
static double one_by_one(uint32_t seg, double ids, uint32_t blocks_n) { return ids * (seg + 1) / 2 * blocks_n * 7.2e-5; }
static double groups_gain(uint32_t bins, uint32_t seg, double ids, uint32_t blocks_n) {
    const double each = ids / bins, hit = 1.0 - exp(-each);
    if (each > 64.0) return -1e9;
    const double full = ids / kEmbGroup, bins_hit = bins * hit;
    const double groups = bins_hit > full ? bins_hit : full;
    const double deep = bins * seg * (1.0 - hit / each), split = full * seg * 0.55;
    const double rows = deep > split ? deep : split;
    return one_by_one(seg, ids, blocks_n) - (rows + groups) * blocks_n * 7.2e-5 - 3.5;
}
// More ids than one launch takes, in which embedding4.cu does not have to stop: a launch behind the first costs 6 us, and where
// groups gain less than a fifth the ids behind the first 4096 lose it again, since embedding4.cu takes those in less time than the
// first ones.  What is left behind the whole launches goes to embedding4.cu unless it is enough for groups of its own.  us, embedding4.cu
// -> groups throughout -> this rule: 32000 x 4096 at tile height 16, 4097 ids 71.0 -> 85.6 -> 71.0, 6144 104 -> 113 -> 104, 8200 137 ->
// 155 -> 137, 12288 200 -> 207 -> 200; at 64, 4100 ids 179 -> 88.3 -> 86.2; 16000 x 2048 at 16, 4097 ids 38.5 -> 40.2 -> 38.4,
// 8192 71.3 -> 64.8 -> 64.6; 8000 x 1000 at 128, 4100 ids 108 -> 52.6 -> 50.9.  Returns how many ids groups take.
static uint64_t grouped_ids(uint32_t bins, uint32_t seg, uint64_t ids, uint32_t blocks_n) {
    if (ids <= kEmbGIds) return groups_gain(bins, seg, (double)ids, blocks_n) > 0.0 ? ids : 0;
    const uint64_t rest = ids % kEmbGIds, whole = ids - rest;
    const double gain = groups_gain(bins, seg, (double)kEmbGIds, blocks_n);
    const double rest_gain = rest ? groups_gain(bins, seg, (double)rest, blocks_n) : 0.0;
    if (gain < 0.2 * one_by_one(seg, (double)kEmbGIds, blocks_n)) return 0;
    if (whole / kEmbGIds * gain + (rest_gain > 0.0 ? rest_gain : 0.0) <= (ids - 1) / kEmbGIds * 6.0) return 0;
    return rest_gain > 0.0 ? ids : whole;
}

int launch_embedding_group(const EmbArgs &a, uint32_t max_tile_len, cudaStream_t s) {
    const Geom &g = a.g;
    if (g.tw != 32 || g.th % 2 != 0 || max_tile_len == 0) return 1;
    if ((reinterpret_cast<uintptr_t>(a.stream) & 15u) || (reinterpret_cast<uintptr_t>(a.states) & 15u) ||
        (reinterpret_cast<uintptr_t>(a.mantissa) & 15u))
        return 1;
    const bool entry = a.entry_step != 0 && a.entry_cap != 0 && g.half > a.entry_step && g.half % a.entry_step == 0 &&
                       ((reinterpret_cast<uintptr_t>(a.entry_states) | reinterpret_cast<uintptr_t>(a.entry_rows)) & 15u) == 0;
    EmbGArgs p;
    p.a = a;
    p.seg = entry ? a.entry_step : g.half;
    p.bins = (g.K + p.seg - 1) / p.seg;
    if (p.seg > 0xFFFFu || p.bins > kEmbGBins) return 1;        // rows in a bin and bins are 16-bit numbers below 0xFFFF
    const uint64_t ids = a.n_ids < kEmbGIds ? a.n_ids : kEmbGIds;
    p.blocks_n = (g.tiles_n + 3) / 4;
    const uint64_t grouped = grouped_ids(p.bins, p.seg, a.n_ids, p.blocks_n);
    if (grouped == 0) return 1;
    int dev = 0, max_smem = 0;
    CI_CUDA(cudaGetDevice(&dev));
    CI_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    p.cap_rows = entry ? a.entry_cap : max_tile_len;
    p.subs = entry ? g.half / a.entry_step : 1u;
    p.stage_bytes = p.cap_rows * 128u + kEmbGroup * 128u;
    p.out_vec = ((reinterpret_cast<uintptr_t>(a.out) & 7u) == 0 && (a.ldo & 3) == 0) ? 1u : 0u;
    // up to one table size is lost to the table's alignment
    const uint32_t fixed = 2 * kLutBytes + kEmbGBarBytes + (uint32_t)(ids * 8) + kEmbGSorts * 4 + (p.bins + 1) * 4 + 128;
    if (fixed + p.stage_bytes > (uint32_t)max_smem) return 1;   // the ranks of 4096 ids, 24 KB, fit in any case
    const uint32_t room = (uint32_t)max_smem - fixed;
    p.stages = room / (2 * p.stage_bytes) >= 12 ? 2 : 1;        // as in embedding4.cu
    uint32_t w_max = room / (p.stages * p.stage_bytes);
    if (w_max > kEmbGWarps) w_max = kEmbGWarps;
    const bool ragged = g.tiles_n % 4 != 0;
    static SmemLimit lim[4] = {};
    void (*const kernel)(EmbGArgs) = entry ? (ragged ? k_embedding_group<true, true> : k_embedding_group<true, false>)
                                           : (ragged ? k_embedding_group<false, true> : k_embedding_group<false, false>);
    if (int rc = ensure_smem_limit(lim[entry + 2 * ragged], (const void *)kernel, (size_t)max_smem)) return rc;
    const uint32_t P = (uint32_t)sm_count();
    for (uint64_t i0 = 0; i0 < grouped; i0 += kEmbGIds) {
        p.n = (uint32_t)(grouped - i0 < kEmbGIds ? grouped - i0 : kEmbGIds);
        p.a.ids = a.ids + i0;
        p.a.out = a.out + i0 * a.ldo;
        const uint64_t most = (uint64_t)p.n * p.blocks_n;       // units, if no two ids shared a bin
        const uint32_t blocks = most < P ? (uint32_t)most : P;
        uint32_t warps = (uint32_t)((most + blocks - 1) / blocks < w_max ? (most + blocks - 1) / blocks : w_max);
        if (warps < 4) warps = w_max < 4 ? w_max : 4;           // the sort is all warps' work
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(blocks);
        cfg.blockDim = dim3(warps * 32);
        const size_t ranks = (size_t)p.n / (kEmbGRanked + 1) * ((p.n + 31) / 32) * 6, windows = (size_t)warps * p.stages * p.stage_bytes;
        cfg.dynamicSmemBytes = fixed + (ranks > windows ? ranks : windows);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        at[0].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        CI_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    }
    if (grouped == a.n_ids) return CI_OK;
    EmbArgs rest = a;
    rest.ids += grouped;
    rest.out += grouped * a.ldo;
    rest.n_ids -= grouped;
    return launch_embedding4(rest, max_tile_len, s);
}

}  // namespace ci
