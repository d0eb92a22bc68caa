// Fused decode + linear on a weight stored transposed, for 32-wide tiles: y[M,V] = x[M,H] . W[V,H]^T, the LM head on the
// embedding's own layout.  Replaces fused_rans_matmul_transposed (comp_inference/transposed_linear_triton.py:187-358).
//
// Streams run down the rows of W, which are the outputs here, and the contraction runs along a row.  Work unit: one warp
// decodes sixteen columns of four vertically adjacent tiles = 128 streams, four per lane.  Lane T (g = T / 4, q = T % 4)
// owns columns 4q .. 4q + 3 of row segment g, the segments being the top / bottom halves of the four tiles.  That is the A
// fragment of mma.sync m16n8k16 if its rows g and g + 8 are two consecutive rows of segment g and its sixteen k are the
// unit's columns: two symbols of each of the lane's streams are one fragment, no transpose, and the B fragment -- the
// activations of the sixteen columns -- stays in registers for the whole unit.  (The kernel for forced cases in linear.cu
// reduces every row over the lanes with 31 shuffles per 32 rows instead.)
//
// A unit yields a sum for every row.  For one or two activation rows and up to 64 rows a segment they stay in registers from
// one column block to the next (REG); otherwise they live in shared memory, private to the warp: read as the mma's C operand
// and written back, two 8-byte loads and stores per two rows.  The warps of a CTA take column blocks of the same four
// tiles ("group"); at the end of its run in a group the CTA adds its warps' sums, writes an fp32 partial and draws a
// ticket; the CTA that draws the last one adds the partials in a fixed order and writes bf16.  Where there is room for two
// sets of sums a CTA deals the units of two groups out as one sequence before it does so.
//
// Bytes are staged as in linear_mma4.cu: one window of 128-byte rows per unit (a shared-memory bank per lane), sign and
// mantissa in 16-row chunks, initial states with the window, all waited for with cp.async.wait_all.  Bound by the instructions
// of the decode step like that kernel: 21 per 32 symbols, 75 % of the issue slots in long runs (32000 x 4096, one row).
//
// Measured on a B200, us, before -> with sums in registers, two sets, states among the copies and the chunks of three warps
// in front of the table: 32000 x 4096 at tile height 128, one row 139 -> 118, two 145 -> 129, eight 215 -> 194; at 64 155 -> 129; at
// 1024 with entry points 273 -> 194; 16000 x 4096 at 1024, four rows 208 -> 187; 8000 x 1024 at 128 31.5 -> 21.2.  The shuffle kernel takes 1000 and 3590
// for the first and for eight rows at 1024.
#include "linear.cuh"
#include "ptx.cuh"

namespace ci {

constexpr uint32_t kT4Warps = 16;
constexpr uint32_t kT4BarBytes = 128;        // the table's barrier, the flag of the last arrival
constexpr uint32_t kT4SegPitch = kChunkRows * 16 + 16;       // eight segments of a chunk, 4 banks apart
constexpr uint32_t kT4ManBuf = 8 * kT4SegPitch;              // one of the two chunk buffers of a warp
constexpr uint32_t kT4ManBytes = 2 * kT4ManBuf;
constexpr uint32_t kT4RegChunks = 4;         // chunks of a segment whose sums a lane holds in registers

// The table's alignment leaves up to a table's size unused in front of the table, where the chunks of three warps have room; the
// rest of it is left at the end of the window.  Wherever the window begins, their buffers have room in the two together, one by one.
// (Whole chunks would need 1 KB more: 30000 x 3000 at tile height 1024, eight rows, then has room for a warp less, 237 us -> 255.)
constexpr uint32_t kT4Front = 3;
constexpr bool front_fits() {
    for (uint32_t gap = 0; gap < kLutBytes; gap += 16)
        if (gap / kT4ManBuf + (kLutBytes - gap) / kT4ManBuf < 2 * kT4Front) return false;
    return true;
}
static_assert(front_fits(), "no room for the chunk buffers beside the table");

struct T4Args {
    LinArgs a;
    uint32_t cap_rows;     // rows of a byte window (>= every tile_max_len)
    uint32_t stage_bytes;  // window + initial states (with entry points also the rows of the next bytes)
    uint32_t stages;       // windows per warp
    uint32_t front;        // warps whose sign+mantissa chunks lie in front of the table, as far as there is room
    uint32_t acc_bytes;    // sums of a warp in one group
    uint32_t sets;         // groups that a CTA works on between two barriers
    uint32_t cblocks;      // 16-column blocks per group
    uint32_t subs, step;   // ENTRY: groups per four tiles, the rows of a segment in each; else 1, half a tile
    uint32_t total;        // units
    uint32_t x_wide;       // four activations are one aligned 8-byte load
    uint32_t wide;         // states (and rows) can be copied 16 bytes at a time
    uint32_t *status;
};

__device__ __forceinline__ void cp_async4(uint32_t dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
// d = w . x with nothing added: the sums of two rows of each segment over the unit's columns.
__device__ __forceinline__ void mma_bf16_zero(float (&d)[4], const uint32_t (&w)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(b0), "r"(b1), "f"(0.f));
}

// MT: activation rows that a pass takes (1, 2 or 8).
// REG: the sums of up to 64 rows a segment stay in registers (one or two activation rows).  Every column of D is made a row of
// activations -- column n is row n % MT -- so that all four lanes of a segment hold the sums of its two rows, and lane q adds
// those of rows 4q .. 4q + 3 of a 16-row chunk to its own: 16 MT registers, turned by one chunk at a time because a loop cannot
// index them.  (One activation column per row pair in one D instead would let an infinite weight reach its neighbours' sums.)
// ENTRY: a group is the rows of four tiles between two entry points (see linear_mma4.cu), so its sums are those of a short
// tile; without, a tall tile's sums and window leave room for three warps.
// RAGGED: the matrix ends inside a column block.  Zero activations alone would not do for the columns that are missing: the
// symbols they repeat may be those of an infinite weight, and zero times that is not a number.  Their exponents are masked to
// zero.  An instantiation of its own (32000 x 4090, one row 116.8 us -> 118.5): in all of them the masks cost 32000 x 4096 2.6 %,
// a second loop for the last block 2.8 %.
template <int MT, bool ENTRY, bool REG, bool RAGGED>
__global__ void __launch_bounds__(kT4Warps * 32, 1) k_linear_t4(const __grid_constant__ T4Args p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const LinArgs &a = p.a;
    const Geom &g = a.g;
    const uint32_t W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = lane_id();
    const uint32_t smem_s = smem_u32(smem);
    const uint32_t lut_s = (smem_s + kLutBytes - 1) & ~(kLutBytes - 1);    // see linear_mma4.cu
    uint32_t *s_lut = reinterpret_cast<uint32_t *>(smem + (lut_s - smem_s));
    const uint32_t lut_bar = lut_s + kLutBytes + kT4BarBytes - 16;
    start_lut(lut_s, lut_bar, a.lut);
    const uint32_t behind_s = lut_s + kLutBytes + kT4BarBytes;
    uint32_t man_s = warp < p.front ? smem_s + warp * kT4ManBytes : behind_s + (warp - p.front) * kT4ManBytes;
    const uint32_t acc0_s = behind_s + (W - p.front) * kT4ManBytes, set_bytes = W * p.acc_bytes;
    uint32_t man_step = kT4ManBuf;                              // from the warp's first chunk buffer to its second
    if (lut_s - smem_s < p.front * kT4ManBytes && warp < p.front) {
        const uint32_t front = (lut_s - smem_s) / kT4ManBuf, end_s = acc0_s + p.sets * set_bytes + W * p.stages * p.stage_bytes;
        auto buffer = [&](uint32_t i) { return i < front ? smem_s + i * kT4ManBuf : end_s + (i - front) * kT4ManBuf; };
        man_s = buffer(2 * warp);
        man_step = buffer(2 * warp + 1) - man_s;
    }
    const uint32_t acc_s = acc0_s + warp * p.acc_bytes;         // of the first set; the others set_bytes further each
    const uint32_t wbase_s = acc0_s + p.sets * set_bytes + warp * p.stages * p.stage_bytes;
    const uint32_t st_off = p.cap_rows * 128;
    const uint32_t subs = ENTRY ? p.subs : 1u, step = ENTRY ? p.step : g.half;
    const uint32_t seg_acc = step * (MT * 4) + (MT == 8 ? 32 : MT * 4);  // bytes between the sums of two segments
    uint32_t *const s_flag = reinterpret_cast<uint32_t *>(smem + (lut_bar + 8 - smem_s));

    const uint32_t sg = lane >> 2, q = lane & 3;                // row segment and column quad of this lane
    // Units of this CTA: [lo, hi), column block running fastest.  Those of `sets` groups, a span, are dealt to the warps in
    // turn; a span ends with a barrier.
    const uint32_t lo = (uint32_t)((uint64_t)blockIdx.x * p.total / gridDim.x);
    const uint32_t hi = (uint32_t)((uint64_t)(blockIdx.x + 1) * p.total / gridDim.x);

    struct Unit {
        uint32_t u, grp, cb;   // unit, its group and column block; u = hi: none
        uint32_t span;         // first group of its span
    };
    auto span_end = [&](uint32_t grp0) { return (uint32_t)min((uint64_t)hi, (uint64_t)(grp0 + p.sets) * p.cblocks); };
    auto settle = [&](Unit &x) {                                // after x.u and x.cb have moved
        for (uint32_t end = span_end(x.span); x.u >= end; end = span_end(x.span)) {
            if (end >= hi) {
                x.u = hi;
                return;
            }
            x.span += p.sets;
            x.u = end + warp;
            x.grp = x.span;
            x.cb = warp;
        }
        for (; x.cb >= p.cblocks; x.cb -= p.cblocks) ++x.grp;
    };
    auto advance = [&](Unit &x) {
        if (x.u >= hi) return;
        x.u += W;
        x.cb += W;
        settle(x);
    };

    // Lanes 0..3: byte offset and depth of the group's four tiles in a unit's tile column.
    auto load_desc = [&](const Unit &x, uint32_t &off, uint32_t &ml) {
        off = ml = 0;
        if (x.u >= hi || lane >= 4) return;
        const uint32_t tk = 4 * (x.grp / subs) + lane;
        if (tk >= g.tiles_k) return;
        const size_t tile = (size_t)tk * g.tiles_n + (x.cb >> 1);
        off = __ldg(a.tile_offsets + tile);
        if constexpr (ENTRY) {
            ml = enter_span(__ldg(a.entry_spans + tile * subs + x.grp % subs), __ldg(a.tile_max_lens + tile), off);
        } else {
            ml = __ldg(a.tile_max_lens + tile);
        }
    };
    auto issue = [&](const Unit &x, uint32_t stage, uint32_t off, uint32_t ml) {
        const uint32_t hb = x.cb & 1, dst = wbase_s + stage * p.stage_bytes;
        if (ml > p.cap_rows) {                                  // metadata disagrees with the declared maximum
            atomicExch(p.status, 2u);
            ml = 0;
        }
        // byte blocks: eight lanes a row of the window, two (one a half) for every tile
        const uint32_t n = __shfl_sync(kFull, ml, lane >> 1 & 3), from = __shfl_sync(kFull, off, lane >> 1 & 3);
        const uint8_t *bytes = a.stream + from + hb * 16 + (lane & 1) * 32 + (lane >> 3) * 64;
        uint32_t to = dst + lane * 16;
        for (uint32_t r = lane >> 3; r < n; r += 4, to += 512, bytes += 256) cp_async16(to, bytes);
        // States of the unit's 16 columns, segment by segment: four columns a lane.
        const uint32_t grp4 = x.grp / subs, tk = 4 * grp4 + (lane >> 3);
        if (tk < g.tiles_k) {
            const size_t at = (((size_t)tk * g.tiles_n + (x.cb >> 1)) * subs + (ENTRY ? x.grp - grp4 * subs : 0u)) * 64 +
                              (lane >> 2 & 1) * 32 + hb * 16 + (lane & 3) * 4;
            const uint32_t *src = (ENTRY ? a.entry_states : a.states) + at, d = dst + st_off + lane * 16;
            if (p.wide) {
                cp_async16(d, src);
            } else {
                for (uint32_t j = 0; j < 4; ++j) cp_async4(d + 4 * j, src + j);
            }
            if constexpr (ENTRY) {                              // two lanes' rows are 16 bytes
                const uint16_t *rows = a.entry_rows + at;
                if (p.wide) {
                    if ((lane & 1) == 0) cp_async16(dst + st_off + 512 + lane * 8, rows);
                } else {
                    for (uint32_t j = 0; j < 2; ++j) cp_async4(dst + st_off + 512 + lane * 8 + 4 * j, rows + 2 * j);
                }
            }
        }
    };
    // Sign+mantissa bytes: a lane copies one row of one half of every tile, 16 columns.
    const uint32_t man_row = lane & 15, man_half = lane >> 4;
    auto man_of = [&](const Unit &x) {
        const uint32_t grp4 = x.grp / subs, sub_row = ENTRY ? (x.grp - grp4 * subs) * step : 0u;
        return a.mantissa + (((size_t)4 * grp4 * g.tiles_n + (x.cb >> 1)) * g.th + man_half * g.half + sub_row + man_row) * 32 +
               (x.cb & 1) * 16;
    };
    const size_t tile_step = (size_t)g.tiles_n * g.th * 32;
    // Rows [row, + kChunkRows) into chunk buffer `buf`; src: this lane's piece of them, `tiles` of the group exist.
    auto issue_man = [&](const uint8_t *src, uint32_t tiles, uint32_t row, uint32_t buf) {
        if (row + man_row >= step) return;
        const uint32_t dst = man_s + buf * man_step + man_half * kT4SegPitch + man_row * 16;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            if (j < tiles) cp_async16(dst + 2 * j * kT4SegPitch, src + j * tile_step);
    };
    auto tiles_of = [&](const Unit &x) { return g.tiles_k - 4 * (x.grp / subs); };
    // Activations of the lane's column of D, columns col .. col + 3 of the weight.
    const uint32_t x_row = REG ? sg % MT : sg;
    auto load_x = [&](const Unit &x, uint32_t (&xb)[2]) {
        xb[0] = xb[1] = 0;
        if (x.u >= hi || x_row >= a.M) return;
        const uint32_t col = x.cb * 16 + 4 * q;
        const uint16_t *src = a.x + (size_t)x_row * a.ldx + col;
        if (p.x_wide) {
            if (col < g.N) {
                const uint2 v = __ldg(reinterpret_cast<const uint2 *>(src));
                xb[0] = v.x;
                xb[1] = v.y;
            }
            return;
        }
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
            if (col + j < g.N) xb[j >> 1] |= (uint32_t)__ldg(src + j) << (16 * (j & 1));
    };

    Unit cur{lo + warp, lo / p.cblocks, 0, lo / p.cblocks};
    cur.cb = lo - cur.grp * p.cblocks + warp;
    settle(cur);
    Unit nxt = cur;
    advance(nxt);
    uint32_t off, ml, noff, nml;
    load_desc(cur, off, ml);
    load_desc(nxt, noff, nml);
    const uint8_t *man = man_of(cur);                           // the sign+mantissa chunk that was asked for last
    uint32_t man_tiles = tiles_of(cur);
    if (cur.u < hi) {
        issue(cur, 0, off, ml);
        issue_man(man, man_tiles, 0, 0);
    }
    if (a.lut == nullptr) load_lut(s_lut, nullptr, a.tables, a.slot_map);
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");          // everything above touched only the weight
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (!wait_lut(lut_bar, a.lut)) atomicExch(p.status, 1u);
    const bool live_m = MT == 8 ? 2 * q < a.M : q == 0;         // !REG: lanes whose two D columns are activation rows
    const uint32_t n_chunks = (step + kChunkRows - 1) / kChunkRows;
    uint32_t stage = 0, chunk = 0;
    uint32_t xb[2], nxb[2];
    load_x(cur, xb);
    Quad z;
    float sum[kT4RegChunks][4 * MT];                            // REG: [chunk][row 4q + 0..3][activation row]
    auto zero_sums = [&]() {
#pragma unroll
        for (uint32_t f = 0; f < kT4RegChunks; ++f)
#pragma unroll
            for (int i = 0; i < 4 * MT; ++i) sum[f][i] = 0.f;
    };
    auto turn_sums = [&]() {
#pragma unroll
        for (int i = 0; i < 4 * MT; ++i) {
            const float t = sum[0][i];
#pragma unroll
            for (uint32_t f = 0; f + 1 < kT4RegChunks; ++f) sum[f][i] = sum[f + 1][i];
            sum[kT4RegChunks - 1][i] = t;
        }
    };
    auto store_sums = [&](uint32_t set) {
#pragma unroll
        for (uint32_t f = 0; f < kT4RegChunks; ++f)
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t r = f * kChunkRows + 4 * q + i;
                if (r < step) {
#pragma unroll
                    for (uint32_t m = 0; m < MT; ++m)
                        asm volatile("st.shared.f32 [%0], %1;" ::"r"(acc_s + set * set_bytes + sg * seg_acc + (r * MT + m) * 4),
                                     "f"(sum[f][i * MT + m]) : "memory");
                }
            }
    };
    for (uint32_t run = lo; run < hi;) {                        // the CTA's spans
        const uint32_t grp0 = run / p.cblocks, end = span_end(grp0), n_sets = (end - 1) / p.cblocks - grp0 + 1;
        uint32_t set = 0;                                       // REG: whose sums the registers hold
        if constexpr (REG) {
            zero_sums();
        } else {
            for (uint32_t k = 0; k < n_sets; ++k)
                for (uint32_t i = lane * 4; i < p.acc_bytes; i += 128)
                    asm volatile("st.shared.u32 [%0], %1;" ::"r"(acc_s + k * set_bytes + i), "r"(0u) : "memory");
            __syncwarp();
        }
        while (cur.u < end) {
            if constexpr (REG) {
                for (; set < cur.grp - grp0; ++set) {
                    store_sums(set);
                    zero_sums();
                }
            }
            load_x(nxt, nxb);
            // The segment whose streams this lane decodes: its own, or, where the group has no such tile, the same half of the
            // first one (real symbols; random ones would take the branch for a second byte at every step).
            const uint32_t sd = 4 * (cur.grp / subs) + (sg >> 1) < g.tiles_k ? sg : sg & 1;
            const uint32_t my_ml = __shfl_sync(kFull, ml, sd >> 1), col = cur.cb * 16 + 4 * q;
            const uint32_t win_s = wbase_s + stage * p.stage_bytes;
            const uint32_t first = win_s + (!ENTRY && my_ml <= p.cap_rows ? my_ml - 1 : 0u) * 128 + sd * 16;
            cp_async_wait();                                    // this unit's bytes and states, its first sign+mantissa chunk
            __syncwarp();
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) {
                // a column beyond the matrix repeats the symbols of the block's first one
                const uint32_t c = col + j < g.N ? 4 * q + j : 0u;
                z.s[j] = lds_u32(win_s + st_off + sd * 64 + c * 4);
                z.p[j] = first + c;
                if constexpr (ENTRY) z.p[j] += min(lds_u16(win_s + st_off + 512 + sd * 32 + c * 2), p.cap_rows - 1) * 128;
            }
            // RAGGED: exponent bits of the columns that exist
            const uint32_t exp01 = (col < g.N ? 0x7F80u : 0u) | (col + 1 < g.N ? 0x7F800000u : 0u);
            const uint32_t exp23 = (col + 2 < g.N ? 0x7F80u : 0u) | (col + 3 < g.N ? 0x7F800000u : 0u);
            auto next_unit = [&]() {
                off = noff;
                ml = nml;
                if (nxt.u >= hi) return;
                issue(nxt, p.stages == 2 ? stage ^ 1 : 0u, off, ml);
                Unit after = nxt;
                advance(after);
                load_desc(after, noff, nml);
            };
            uint32_t ac = acc_s + (REG ? 0u : (cur.grp - grp0) * set_bytes) + sg * seg_acc + (MT == 8 ? q * 8 : 0u);
#pragma unroll 1
            for (uint32_t c = 0; c < n_chunks; ++c, ++chunk) {
                const uint32_t buf = chunk & 1;
                if (c != 0) {
                    cp_async_wait();                            // this chunk is here
                    __syncwarp();                               // for every lane, and all are done with the other buffer
                }
                const bool last = c + 1 == n_chunks;
                if (last) {                                     // the next unit's first chunk
                    man = man_of(nxt);
                    man_tiles = tiles_of(nxt);
                } else {
                    man += kChunkRows * 32;
                }
                if (!last || nxt.u < hi) issue_man(man, man_tiles, last ? 0u : (c + 1) * kChunkRows, buf ^ 1);
                if (c == 0 && p.stages == 2) next_unit();
                z.clamp(win_s);
                uint32_t ms = man_s + buf * man_step + sg * kT4SegPitch + q * 4;
                const uint32_t n = min(kChunkRows, step - c * kChunkRows);
#pragma unroll 1
                for (uint32_t r = 0; r < n; r += 4) {
                    const bool mine = q == r >> 2;              // REG
#pragma unroll
                    for (uint32_t i = 0; i < 4; i += 2) {
                        float d[4] = {0.f, 0.f, 0.f, 0.f};
                        const uint32_t ad = ac + i * (MT * 4);
                        if (!REG && live_m) {
                            if constexpr (MT == 1) {
                                d[0] = __uint_as_float(lds_u32(ad));
                                d[2] = __uint_as_float(lds_u32(ad + 4));
                            } else {
                                asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(d[0]), "=f"(d[1]) : "r"(ad));
                                asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(d[2]), "=f"(d[3]) : "r"(ad + MT * 4));
                            }
                        }
                        uint32_t w[4];
#pragma unroll
                        for (uint32_t k = 0; k < 2; ++k) {      // rows i, i + 1: columns 0, 1 and 2, 3 of the lane
                            uint32_t e[4];
                            z.step_together(lut_s, e);
                            const uint32_t m = lds_u32(ms + (i + k) * 16);
                            const uint32_t e01 = __byte_perm(e[0], e[1], 0x6521) << 3, e23 = __byte_perm(e[2], e[3], 0x6521) << 3;
                            const uint32_t m01 = __byte_perm(m, 0u, 0x1100), m23 = __byte_perm(m, 0u, 0x3322);
                            w[k] = RAGGED ? (e01 & exp01) | (m01 & 0x807F807Fu) : exp_or_man(e01, m01);
                            w[2 + k] = RAGGED ? (e23 & exp23) | (m23 & 0x807F807Fu) : exp_or_man(e23, m23);
                        }
                        if constexpr (REG) {
                            mma_bf16_zero(d, w, xb[0], xb[1]);
                            if (mine) {
#pragma unroll
                                for (int m = 0; m < MT; ++m) {
                                    sum[0][i * MT + m] += d[m];
                                    sum[0][(i + 1) * MT + m] += d[2 + m];
                                }
                            }
                        } else {
                            mma_bf16(d, w, xb[0], xb[1]);
                            if (live_m) {
                                if constexpr (MT == 1) {
                                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(ad), "f"(d[0]) : "memory");
                                    asm volatile("st.shared.f32 [%0], %1;" ::"r"(ad + 4), "f"(d[2]) : "memory");
                                } else {
                                    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(ad), "f"(d[0]), "f"(d[1]) : "memory");
                                    asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(ad + MT * 4), "f"(d[2]), "f"(d[3]) : "memory");
                                }
                            }
                        }
                    }
                    ac += 4 * (MT * 4);
                    ms += 64;
                }
                if constexpr (REG) turn_sums();
            }
            if constexpr (REG) {
                for (uint32_t c = n_chunks; c < kT4RegChunks; ++c) turn_sums();
            }
            if (p.stages == 2) {
                stage ^= 1;
            } else {
                __syncwarp();                                   // every lane is done with the only window
                next_unit();
            }
            cur = nxt;
            advance(nxt);
            xb[0] = nxb[0];
            xb[1] = nxb[1];
        }
        if constexpr (REG) {
            for (; set < n_sets; ++set) {
                store_sums(set);
                zero_sums();
            }
        }
        // ---- the span's sums of this CTA, group by group -----------------------------------------------------
        __syncthreads();
        for (uint32_t k = 0; k < n_sets; ++k) {
            const uint32_t grp = grp0 + k, rows = 8 * step;
            const uint32_t first_cta = (uint32_t)(((uint64_t)(grp * p.cblocks + 1) * gridDim.x - 1) / p.total);
            const uint32_t last_cta = (uint32_t)(((uint64_t)min((grp + 1) * p.cblocks, p.total) * gridDim.x - 1) / p.total);
            const uint32_t count = last_cta - first_cta + 1;
            // row r of the group = row r % step of its segment r / step
            auto out_row = [&](uint32_t r) {
                const uint32_t seg = r / step;
                return (4 * (grp / subs) * 2 + seg) * g.half + (ENTRY ? grp % subs * step : 0u) + r - seg * step;
            };
            float *mine = a.partial + (size_t)(blockIdx.x + grp) * rows * a.M;
            for (uint32_t i = threadIdx.x; i < rows * a.M; i += blockDim.x) {
                const uint32_t m = i / rows, r = i - m * rows, seg = r / step, v = out_row(r);
                const uint32_t at = acc0_s + k * set_bytes + seg * seg_acc + (r - seg * step) * (MT * 4) + m * 4;
                float total = 0.f;
                for (uint32_t w = 0; w < W; ++w) total += __uint_as_float(lds_u32(at + w * p.acc_bytes));
                if (count > 1) {
                    mine[i] = total;
                } else if (v < g.K) {
                    if (a.bias) total += load_bf16(a.bias + v);
                    a.y[(size_t)m * a.ldy + v] = float_to_bf16_bits(total);
                }
            }
            if (count > 1) {
                if (last_arrival(a.tickets + grp, count, s_flag)) {
                    for (uint32_t i = threadIdx.x; i < rows * a.M; i += blockDim.x) {
                        const uint32_t m = i / rows, v = out_row(i - m * rows);
                        if (v >= g.K) continue;
                        float total = 0.f;
                        for (uint32_t c = first_cta; c <= last_cta; ++c) total += __ldcg(a.partial + (size_t)(c + grp) * rows * a.M + i);
                        if (a.bias) total += load_bf16(a.bias + v);
                        a.y[(size_t)m * a.ldy + v] = float_to_bf16_bits(total);
                    }
                    if (threadIdx.x == 0) a.tickets[grp] = 0;   // ready for the next call
                }
            }
        }
        __syncthreads();                                        // the sums may be cleared
        run = end;
    }
}

// ------------------------------------------------------------------------ host

template <int MT, bool ENTRY, bool REG, bool RAGGED>
static int launch_t4_pass(T4Args p, uint32_t blocks, uint32_t warps, size_t smem, int max_smem, cudaStream_t s) {
    static SmemLimit lim = {};
    if (int rc = ensure_smem_limit(lim, (const void *)k_linear_t4<MT, ENTRY, REG, RAGGED>, (size_t)max_smem)) return rc;
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
    CI_CUDA(cudaLaunchKernelEx(&cfg, k_linear_t4<MT, ENTRY, REG, RAGGED>, p));
    return CI_OK;
}

size_t linear_t4_workspace_bytes(uint32_t M, uint32_t V, uint32_t th) {
    const uint32_t groups = (V + 4 * th - 1) / (4 * th);
    return ((size_t)sm_count() + groups + 1) * 4 * th * (M < 8 ? M : 8) * sizeof(float);
}

int launch_linear_t4(const LinArgs &a, uint32_t max_tile_len, size_t partial_capacity, cudaStream_t s) {
    const Geom &g = a.g;
    if (g.tw != 32 || g.th % 16 != 0 || max_tile_len == 0) return 1;
    if ((reinterpret_cast<uintptr_t>(a.stream) & 15u) || (reinterpret_cast<uintptr_t>(a.mantissa) & 15u)) return 1;
    if (partial_capacity < linear_t4_workspace_bytes(a.M, g.K, g.th)) return 1;
    const bool entry = a.entry_step != 0 && a.entry_cap != 0 && g.half > a.entry_step && g.half % a.entry_step == 0 &&
                       a.entry_step % kChunkRows == 0 && (reinterpret_cast<uintptr_t>(a.entry_rows) & 3u) == 0;
    const uint32_t step = entry ? a.entry_step : g.half, subs = g.half / step, groups = (g.tiles_k + 3) / 4 * subs;
    if (groups >= kTicketBytes - 1) return 1;
    int dev = 0, max_smem = 0;
    CI_CUDA(cudaGetDevice(&dev));
    CI_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    T4Args p;
    p.cap_rows = entry ? a.entry_cap : max_tile_len;
    p.step = step;
    p.subs = subs;
    p.stage_bytes = p.cap_rows * 128u + (entry ? 768u : 512u);
    p.cblocks = (g.N + 15) / 16;
    p.total = groups * p.cblocks;
    p.status = a.tickets + (kTicketBytes - 1);
    p.wide = ((entry ? reinterpret_cast<uintptr_t>(a.entry_states) | reinterpret_cast<uintptr_t>(a.entry_rows)
                     : reinterpret_cast<uintptr_t>(a.states)) & 15u) == 0;
    const uint32_t P = (uint32_t)sm_count(), fixed = 2 * kLutBytes + kT4BarBytes, room = (uint32_t)max_smem - fixed;
    const uint32_t blocks = p.total < P ? p.total : P;
    // Passes over the weight x rounds of units: sums for eight activation rows take eight times the shared memory of one,
    // which a tall tile cannot afford at a useful number of warps.  Two sets of sums where there is room: a CTA with the units
    // of two groups then deals them out as one sequence, and without a second one rounds its units up in each.
    const uint32_t units = (p.total + blocks - 1) / blocks;
    uint32_t warps = 0, rows_per_pass = 0;
    double best = 0.0;
    for (uint32_t mt = 1; mt <= 8; mt = mt == 2 ? 8 : mt * 2)
        for (uint32_t stages = 1; stages <= 2; ++stages)
            for (uint32_t sets = 1; sets <= (mt == 8 ? 1u : 2u); ++sets) {
                const uint32_t acc = (8 * (step * (mt * 4) + (mt == 8 ? 32 : mt * 4)) + 15) & ~15u;
                const uint32_t own = stages * p.stage_bytes + sets * acc;
                uint32_t w_max = (room + kT4Front * kT4ManBytes) / (own + kT4ManBytes);
                if (w_max < kT4Front) w_max = room / own;
                if (w_max > kT4Warps) w_max = kT4Warps;
                for (uint32_t w = 1; w <= w_max; ++w) {
                    const bool split = groups > 1 && (sets == 1 || units > p.cblocks);   // some CTA's units end in two rounds
                    const double cost = (double)((a.M + mt - 1) / mt) *
                                        (run_cost(units, w, 0.0) + (split ? 0.5 * round_cost(w, 0.0) : 0.0)) * (stages == 1 ? 1.02 : 1.0);
                    if (warps == 0 || cost < best) {
                        best = cost;
                        warps = w;
                        rows_per_pass = mt;
                        p.stages = stages;
                        p.sets = sets;
                        p.front = w < kT4Front ? w : kT4Front;
                        p.acc_bytes = acc;
                    }
                }
            }
    if (warps == 0) return 1;
    const size_t smem = fixed + (size_t)warps * (p.stages * p.stage_bytes + p.sets * p.acc_bytes) + (size_t)(warps - p.front) * kT4ManBytes;
    for (uint32_t m0 = 0; m0 < a.M; m0 += rows_per_pass) {
        p.a = a;
        p.a.x = a.x + (size_t)m0 * a.ldx;
        p.a.y = a.y + (size_t)m0 * a.ldy;
        p.x_wide = ((reinterpret_cast<uintptr_t>(p.a.x) & 7u) == 0 && (a.ldx & 3) == 0 && g.N % 4 == 0) ? 1u : 0u;
        p.a.M = a.M - m0 < rows_per_pass ? a.M - m0 : rows_per_pass;
        using Pass = int (*)(T4Args, uint32_t, uint32_t, size_t, int, cudaStream_t);
#define CI_T4_SET(E, R)                                                                                      \
    {launch_t4_pass<1, E, true, R>, launch_t4_pass<2, E, true, R>, launch_t4_pass<1, E, false, R>,           \
     launch_t4_pass<2, E, false, R>, launch_t4_pass<8, E, false, R>}
        static const Pass pass[4][5] = {CI_T4_SET(false, false), CI_T4_SET(true, false), CI_T4_SET(false, true), CI_T4_SET(true, true)};
#undef CI_T4_SET
        const bool reg = step <= kT4RegChunks * kChunkRows;
        const int rc = pass[entry + 2 * (g.N % 16 != 0)][rows_per_pass == 8 ? 4 : rows_per_pass - 1 + (reg ? 0 : 2)](p, blocks, warps, smem,
                                                                                                                  max_smem, s);
        if (rc) return rc;
    }
    return CI_OK;
}

}  // namespace ci
