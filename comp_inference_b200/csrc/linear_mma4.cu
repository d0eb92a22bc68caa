// Fused decode + linear for 32-wide tiles, register-direct tensor-core path (activation batches of
// up to 16 rows): y[M,N] = x[M,K] . W[K,N] with W decoded from its rANS streams inside the kernel.
// Replaces fused_rans_matmul_kernel_ilp2_splitk (comp_inference/linear_triton.py:317-552).
//
// Work unit: one warp decodes a pair of vertically adjacent tiles of one 32-column group = 128
// streams, four per lane.  Lane T (g = T / 4, q = T % 4) owns the four adjacent columns 4g .. 4g+3 of
// row segment q, the segments being the top / bottom halves of the upper and of the lower tile.  That
// is exactly the fragment ownership of mma.sync m16n8k16 -- the four threads that share g hold
// different k -- once the k index of the instruction is read as "segment q, rows r..r+3": four
// consecutive symbols of a stream are one packed pair of registers, the matching activations
// x[m][those rows] are one 8-byte load per activation row.  The weights are the A operand (two columns
// of the lane = mma rows g and g + 8, two mma per four rows) and activation row g the B operand; an
// instantiation for 9..16 activation rows issues a second pair of mma for row g + 8.  No shared-memory
// transpose, no ldmatrix.
//
// Bound by the on-chip units, not by HBM (15 to 20 %): in full rounds of 16 warps, 19.4 instructions and 5.4 load / shared-memory
// wavefronts per 32 symbols, which take 6.7 cycles: issue slots 72 % busy, that pipe 80 %; the decode step alone, without its
// surroundings, 16.5, 5.1 and 5.6.  So the data movement around the step is arranged to cost as few instructions and
// wavefronts as possible:
//  * compressed bytes: the two tiles' byte blocks ([row][64 B] each) are copied by cp.async into one
//    window of 128-byte rows (upper tile in bytes 0..63, lower tile in 64..127).  The four streams of a
//    lane are the four bytes of one word column, so every lane reads its own bank whatever row each of
//    its cursors is on;
//  * sign+mantissa bytes: chunks of 16 rows of the four segments, double buffered per warp by cp.async, the segments
//    8 banks apart so that a row of the warp's 128 columns is one conflict-free wavefront (read straight from
//    global memory a row took four, one per 32-byte sector: a quarter of the pipe's load);
//  * all copies of a warp are its own, so it waits for them by cp.async.wait_all and a __syncwarp; an mbarrier per
//    buffer cost 0.5 instructions per 32 symbols more, bulk copies issued by one lane more than that;
//  * activations: the load of four rows of a unit touches four segments, a wavefront for each of them, activation row and half
//    warp.  Lanes without an activation row take no part (half of the wavefronts at up to four rows), and from a certain size on
//    the activations are put in the order of the loads first (k_interleave_x).  A copy in shared memory for one or two rows
//    saved another 1.5 % of a long launch and cost 1 us at the start of every one.
// The byte windows are double buffered per warp where they fit; byte ranges of the next units are loaded one unit ahead by
// all lanes in parallel.
//
// Scheduling: warp-level stream-K as in linear_mma.cu (units ordered by column group then tile-row
// pair, equal contiguous runs per warp, fp32 partials + ticket, fixed summation order).
//
// Measured (graph replays over more than L2 of weights) before -> with Quad::step_together, the waits and
// activations as above and 96 registers for 17 to 20 warps: 4096 x 22016 at tile height 128, 1 row 76.3 -> 67.1 us, 16 rows
// 84.7 -> 74.7; 11008 x 4096, 1 row 40.3 -> 36.9; 4096 x 12288 46.3 -> 42.6; 4096 x 4096 18.0 -> 17.1, at tile height 1024 with
// entry points (ENTRY) 18.7 -> 17.8.
#include <type_traits>

#include "linear.cuh"
#include "ptx.cuh"

namespace ci {

constexpr uint32_t kBar4Bytes = 128;         // the table's barrier
constexpr uint32_t kMma4Warps = 16;          // x 32 threads x 128 registers = the register file
// Where it saves a round of units: 96 registers a thread, without spills (one instantiation spills 16 bytes).  Bounded for 21
// warps it would be 80, with up to 160 bytes spilled: 4096 x 22016 on 20 warps, one row 67.2 us -> 72.6, 16 rows 74.7 -> 77.3.
constexpr uint32_t kMma4ManyWarps = 20;

struct Mma4Args {
    LinArgs a;
    uint32_t cap_rows;     // rows of a byte window (>= every tile_max_len)
    uint32_t stage_bytes;  // window + 128 initial states
    uint32_t slots;        // warps of the grid: warp i takes units [i * total / slots, (i + 1) * total / slots)
    uint32_t total;        // units in the matrix
    uint32_t pairs_k;      // tile-row pairs = ceil(tiles_k / 2)
    uint32_t subs;         // units per pair: 1, or the entry points per half tile
    uint32_t step;         // rows of a segment in a unit: half a tile, or the rows between entry points
    uint32_t per_group;    // units of a column group = pairs_k * subs
    uint32_t stages;       // byte windows per warp: 2, or 1 where tall tiles leave no room for two
    uint32_t y_vec;        // outputs can be written as 16-byte rows of eight
    uint32_t x_order;      // activations are in the order of k_interleave_x
    uint32_t *status;      // set non-zero if a wait ran out
};

// Packed bf16 pair (rows k, k+1) of column c of the lane from two table entries and the two
// 4-column sign+mantissa words of those rows.
template <int C>
__device__ __forceinline__ uint32_t weight_pair4(uint32_t e_lo, uint32_t e_hi, uint32_t m_lo, uint32_t m_hi) {
    // Bits 8..23 of each entry side by side: the symbols sit at bits 4..11 / 20..27, three below their
    // place in a bf16 pair; whatever else the shift drags along is masked out by the bit-select.
    const uint32_t ee = __byte_perm(e_lo, e_hi, 0x6521) << 3;
    const uint32_t vv = __byte_perm(m_lo, m_hi, 0x4400 + 0x1111 * C);
    return exp_or_man(ee, vv);
}

// Four symbols of each of the lane's streams -> four packed weight pairs per column -> tensor core.
// m = sign+mantissa words of the four rows, xf = the activations of those rows.
// The weights are the A operand -- columns c and c + 1 of the lane are mma rows g and g + 8, so one mma takes
// two columns -- and activation row g is the B operand (xf[0], xf[1]); with more than 8 activation rows (HI)
// a second pair of mma takes activation row g + 8 (xf[2], xf[3]).  Compared with the weights as the B
// operand (one mma per column) this halves the mma count and the accumulators for up to 8 rows and needs
// no interleaving of the activation registers.
template <bool HI>
__device__ __forceinline__ void mma4(float (&acc)[4][4], const uint32_t (&b)[4][2], const uint32_t (&xf)[4]) {
    const uint32_t w01[4] = {b[0][0], b[1][0], b[0][1], b[1][1]};
    const uint32_t w23[4] = {b[2][0], b[3][0], b[2][1], b[3][1]};
    mma_bf16(acc[0], w01, xf[0], xf[1]);
    mma_bf16(acc[1], w23, xf[0], xf[1]);
    if constexpr (HI) {
        mma_bf16(acc[2], w01, xf[2], xf[3]);
        mma_bf16(acc[3], w23, xf[2], xf[3]);
    }
}
// Four activations into the registers that the mma before has just read, where the lane has a row.
__device__ __forceinline__ void load_x(uint32_t &lo, uint32_t &hi, const uint16_t *src, bool has) {
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "setp.ne.u32 p, %3, 0;\n\t"
                 "@p ld.global.nc.v2.u32 {%0, %1}, [%2];\n\t}"
                 : "+r"(lo), "+r"(hi)
                 : "l"(src), "r"((uint32_t)has));
}
// Two symbols of each stream -> one packed pair per column.
__device__ __forceinline__ void rows2(uint32_t (&b)[4][2], int h, Quad &z, uint32_t lut_s, uint32_t m0, uint32_t m1) {
    uint32_t e[4], f[4];
    z.step_together(lut_s, e);
    z.step_together(lut_s, f);
    b[0][h] = weight_pair4<0>(e[0], f[0], m0, m1);
    b[1][h] = weight_pair4<1>(e[1], f[1], m0, m1);
    b[2][h] = weight_pair4<2>(e[2], f[2], m0, m1);
    b[3][h] = weight_pair4<3>(e[3], f[3], m0, m1);
}

// RAGGED: K is not a whole number of tile pairs, so the last units of a column group lack their lower tile or end
// inside a tile (an instantiation of its own: the common case carries none of the bookkeeping in its registers).
// Every lane still runs the full warp-wide loop.  A lane whose segment has n_my < n_blocks 4-row groups reads zeros instead
// of activations from group n_my on, and what it decodes past the end of its stream is masked to zero.  It starts its stream
// over whenever that is used up, and a lane without a segment decodes the upper tile's top half: any real symbols will do,
// but past the end of a stream the symbols are rare ones, and every step would take the branch for a second byte.
//
// ENTRY: a unit is not a pair of whole tiles but the rows between two entry points of it (tall tiles: 512 symbols are one
// serial chain).  The states and cursors of its streams come from the index, its window holds just the rows of the byte
// blocks that those symbols touch.  4096 x 4096 at tile height 1024, one row: 63 us -> 17.8.
__device__ __align__(16) uint16_t g_zero_activations[256];

// The order of k_interleave_x in 8-byte pieces of four activations: piece q of row m of the four rows r4 of a unit's segments is at
// ((pair * half4 + r4) * M + m) * 4 + q, so that what the 32 lanes read for four rows of a unit are neighbours.
struct XOrder {
    uint32_t half4;        // k4 per row segment (half a tile)
    uint32_t M;
    // Which four activations stand there, and of which row.
    __device__ __forceinline__ uint32_t k4(uint32_t place, uint32_t &m) const {
        const uint32_t row = place / (4 * M), in = place - row * 4 * M, pk = row / half4;
        m = in >> 2;
        return (4 * pk + (in & 3)) * half4 + row - pk * half4;
    }
};

template <bool HI, bool RAGGED, bool ENTRY, uint32_t MAX_WARPS>
__global__ void __launch_bounds__(MAX_WARPS * 32, 1) k_linear_mma4(const __grid_constant__ Mma4Args p) {
    extern __shared__ __align__(128) uint8_t smem[];
    const LinArgs &a = p.a;
    const Geom &g = a.g;
    const uint32_t W = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = lane_id();
    const uint32_t smem_s = smem_u32(smem);
    // The table sits on a 16 KB boundary of the shared window, so that an entry's address is
    // (state << 2 & 0x3FFC) | base: one shift and one three-input logic operation, no addition.
    const uint32_t lut_s = (smem_s + kLutBytes - 1) & ~(kLutBytes - 1);
    uint32_t *s_lut = reinterpret_cast<uint32_t *>(smem + (lut_s - smem_s));
    const uint32_t lut_bar = lut_s + kLutBytes + kBar4Bytes - 16;
    start_lut(lut_s, lut_bar, a.lut);
    const uint32_t wbase_s = lut_s + kLutBytes + kBar4Bytes + W * kManBytes + warp * p.stages * p.stage_bytes;
    const uint32_t man_s = lut_s + kLutBytes + kBar4Bytes + warp * kManBytes;
    const uint32_t seg_bytes = g.th * 16;                       // half a tile of sign+mantissa bytes
    const uint32_t st_off = p.cap_rows * 128;

    const uint32_t gq = lane >> 2, q = lane & 3;                // column quad and row segment of this lane
    const uint32_t tsel = q >> 1, hsel = q & 1;                 // upper / lower tile, top / bottom half

    // This warp's rank in the grid.  Runs differ by one unit in a regular pattern along the ranks: counted through one
    // scheduler's warps (warp % 4) after the other, so that the longer runs do not all meet on the same ones.
    const uint32_t gw = blockIdx.x * W + (warp & 3) * (W >> 2) + min(warp & 3, W & 3) + (warp >> 2);
    const uint32_t lo = gw < p.slots ? gw * p.total / p.slots : p.total;       // slots * total fits 32 bits
    const uint32_t hi = gw < p.slots ? (gw + 1) * p.total / p.slots : p.total;

    const uint32_t subs = ENTRY ? p.subs : 1u, step = ENTRY ? p.step : g.half;

    // Byte ranges of this warp's units, 32 at a time: lane j holds unit dbase + j.
    uint32_t d_off0 = 0, d_ml0 = 0, d_off1 = 0, d_ml1 = 0, dbase = lo;
    auto load_desc = [&]() {
        const uint32_t u = dbase + lane;
        if (u >= hi) return;
        const uint32_t grp = u / p.per_group, v = u - grp * p.per_group, pk = v / subs, sub = v - pk * subs;
        const uint32_t t0 = (2 * pk) * g.tiles_n + grp;
        auto range = [&](uint32_t t, uint32_t &off, uint32_t &ml) {
            off = __ldg(a.tile_offsets + t);
            if constexpr (ENTRY) {
                ml = enter_span(__ldg(a.entry_spans + (size_t)t * subs + sub), __ldg(a.tile_max_lens + t), off);
            } else {
                ml = __ldg(a.tile_max_lens + t);
            }
        };
        range(t0, d_off0, d_ml0);
        d_off1 = 0;
        d_ml1 = 0;
        if (2 * pk + 1 < g.tiles_k) range(t0 + g.tiles_n, d_off1, d_ml1);
    };

    // Starts every copy of the unit (grp, pk, sub) into `stage` (whole warp).
    auto issue = [&](uint32_t grp, uint32_t pk, uint32_t sub, uint32_t stage, uint32_t off0, uint32_t ml0, uint32_t off1, uint32_t ml1) {
        const uint32_t t0 = (2 * pk) * g.tiles_n + grp;
        const bool two = 2 * pk + 1 < g.tiles_k;
        const uint32_t dst = wbase_s + stage * p.stage_bytes;
        if (ml0 > p.cap_rows || ml1 > p.cap_rows) {             // metadata disagrees with the declared maximum
            if (lane == 0) atomicExch(p.status, 2u);
            ml0 = ml1 = 0;
        }
        // states, 16 lanes a tile, and for entry points the rows of their next bytes, 8 lanes a tile
        const bool lower = lane >= 16;
        if constexpr (ENTRY) {
            const size_t e = ((size_t)t0 * subs + sub) * 64, d = (size_t)g.tiles_n * subs * 64;
            if (!lower || two) cp_async16(dst + st_off + lane * 16, a.entry_states + e + (lower ? d : 0) + (lane & 15) * 4);
            if (lane < 8 || (two && lane < 16))
                cp_async16(dst + st_off + 512 + lane * 16, a.entry_rows + e + (lane < 8 ? 0 : d) + (lane & 7) * 8);
        } else {
            if (!lower || two) cp_async16(dst + st_off + lane * 16, a.states + (size_t)(t0 + (lower ? g.tiles_n : 0u)) * 64 + (lane & 15) * 4);
        }
        // byte blocks: eight lanes a row of the window, four for each tile
        const bool low_tile = lane & 4;
        const uint8_t *src = a.stream + (low_tile ? off1 : off0) + (lane & 3) * 16 + (lane >> 3) * 64;
        const uint32_t rows = low_tile ? ml1 : ml0;
        uint32_t to = dst + lane * 16;
        for (uint32_t r = lane >> 3; r < rows; r += 4, to += 512, src += 256) cp_async16(to, src);
    };

    // Sign+mantissa bytes of a unit's upper tile, this lane's 16-byte piece of every chunk row pair.
    auto man_of = [&](uint32_t grp, uint32_t pk, uint32_t sub) {
        return a.mantissa + ((size_t)2 * pk * g.tiles_n + grp) * (2 * seg_bytes) + (ENTRY ? sub * step * 32 : 0u) + lane * 16;
    };
    // Rows [row, + kChunkRows) of the four segments of a unit into chunk buffer `buf`; src: this lane's piece of them.
    const size_t tile_step = (size_t)g.tiles_n * (2 * seg_bytes);
    auto issue_man = [&](const uint8_t *src, bool two, uint32_t row, uint32_t buf) {
        const uint32_t dst = man_s + buf * (4 * kSegPitch) + lane * 16;
        if (row + (lane >> 1) < step) {
            cp_async16(dst, src);
            cp_async16(dst + kSegPitch, src + seg_bytes);
            if (two) {
                src += tile_step;
                cp_async16(dst + 2 * kSegPitch, src);
                cp_async16(dst + 3 * kSegPitch, src + seg_bytes);
            }
        }
    };

    load_desc();
    uint32_t grp = lo / p.per_group, pk = lo - grp * p.per_group, sub = 0;   // of unit t
    if constexpr (ENTRY) {
        sub = pk % subs;
        pk /= subs;
    }
    // The sign+mantissa bytes do not wait for the byte ranges: they are asked for while those are on their way.
    if (lo < hi) issue_man(man_of(grp, pk, sub), 2 * pk + 1 < g.tiles_k, 0, 0);
    uint32_t nx_off0 = __shfl_sync(kFull, d_off0, 0), nx_ml0 = __shfl_sync(kFull, d_ml0, 0);
    uint32_t nx_off1 = __shfl_sync(kFull, d_off1, 0), nx_ml1 = __shfl_sync(kFull, d_ml1, 0);
    if (lo < hi) issue(grp, pk, sub, 0, nx_off0, nx_ml0, nx_off1, nx_ml1);
    if (a.lut == nullptr) load_lut(s_lut, nullptr, a.tables, a.slot_map);
    __syncthreads();
    // Everything above touches only the weight, which the previous kernel has not written (ci_weight_written).  When
    // this launch was allowed to start before its predecessor in the stream has finished (programmatic dependent launch), wait here
    // for it -- activations, workspace and output may be its products -- and let the next launch start
    // its own preamble while this grid works.  Both are no-ops in an ordinary launch.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (!wait_lut(lut_bar, a.lut)) atomicExch(p.status, 1u);
    if (lo >= hi) return;                                       // no CTA-wide synchronisation below this line
    const bool fused_ar = a.ar.world > 1;                       // row-parallel: exchange the sums with the peers here
    const uint32_t ar_seq = fused_ar ? fuse_seq(a.ar) : 0u;

    float acc[4][4];
    auto zero_acc = [&]() {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    };

    // Writes the finished (or partial) sums of column group grp.  After a lane exchange (below) a lane
    // works on rows gq and gq + 8 of the activation batch, columns 8q .. 8q+7 of the group.
    auto flush = [&](uint32_t grp) {
        auto warp_of = [&](uint32_t u) { return ((u + 1) * p.slots - 1) / p.total; };
        const uint32_t first_w = warp_of(grp * p.per_group), last_w = warp_of((grp + 1) * p.per_group - 1);
        const uint32_t count = last_w - first_w + 1;
        const uint32_t n0 = grp * 32 + 8 * q;
        auto store_row = [&](uint32_t m, const float (&v)[8]) {
            if (m >= a.M) return;
            uint16_t h[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                float f = v[j];
                if (a.bias && n0 + j < g.N) f += load_bf16(a.bias + n0 + j);
                h[j] = float_to_bf16_bits(f);
            }
            uint16_t *dst = a.y + (size_t)m * a.ldy + n0;
            if (p.y_vec && n0 + 8 <= g.N) {
                uint4 o;
                o.x = h[0] | ((uint32_t)h[1] << 16);
                o.y = h[2] | ((uint32_t)h[3] << 16);
                o.z = h[4] | ((uint32_t)h[5] << 16);
                o.w = h[6] | ((uint32_t)h[7] << 16);
                *reinterpret_cast<uint4 *>(dst) = o;
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j)
                    if (n0 + j < g.N) dst[j] = h[j];
            }
        };
        float v0[8], v1[8];
        {
            // The D fragments hold columns 4 gq .. 4 gq + 3 of activation rows 2q and 2q + 1 (acc[c / 2], and
            // acc[2 + c / 2] for rows 8 + 2q, 9 + 2q; element 2 (c % 2) + row parity).  Everything below works on
            // "row gq (v0) and gq + 8 (v1), columns 8q .. 8q + 7": fetch those from lanes (2q, gq / 2) and
            // (2q + 1, gq / 2).
            const uint32_t srcA = (2 * q) * 4 + (gq >> 1), srcB = srcA + 4;
            const bool odd = gq & 1;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float e0 = acc[c >> 1][2 * (c & 1)], e1 = acc[c >> 1][2 * (c & 1) + 1];
                const float a0 = __shfl_sync(kFull, e0, srcA), a1 = __shfl_sync(kFull, e1, srcA);
                const float b0 = __shfl_sync(kFull, e0, srcB), b1 = __shfl_sync(kFull, e1, srcB);
                v0[c] = odd ? a1 : a0;
                v0[4 + c] = odd ? b1 : b0;
                v1[c] = v1[4 + c] = 0.f;
                if constexpr (HI) {
                    const float h0 = acc[2 + (c >> 1)][2 * (c & 1)], h1 = acc[2 + (c >> 1)][2 * (c & 1) + 1];
                    const float c0 = __shfl_sync(kFull, h0, srcA), c1 = __shfl_sync(kFull, h1, srcA);
                    const float d0 = __shfl_sync(kFull, h0, srcB), d1 = __shfl_sync(kFull, h1, srcB);
                    v1[c] = odd ? c1 : c0;
                    v1[4 + c] = odd ? d1 : d0;
                }
            }
        }
        if (count == 1) {
            if (fused_ar) {                                     // M <= 2: rows 0 / 1 live in the lanes with gq < M
                if (gq < a.M && n0 < g.N) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        if (n0 + 2 * j >= g.N) break;           // N need only be even: the last quad may be short
                        const float2 r = fuse_exchange_pair(a.ar, ar_seq, (gq * g.N + n0) / 2 + j, v0[2 * j], v0[2 * j + 1]);
                        v0[2 * j] = r.x;
                        v0[2 * j + 1] = r.y;
                    }
                }
                __syncwarp();
                if (lane == 0) fuse_group_done(a.ar, ar_seq, g.groups);
            }
            store_row(gq, v0);
            store_row(gq + 8, v1);
            return;
        }
        // Slot gw + grp is unique: along the unit order both the warp rank and the group only grow.
        float *mine = a.partial + (size_t)(gw + grp) * a.M * 32 + 8 * q;
        if (gq < a.M) {
            *reinterpret_cast<float4 *>(mine + gq * 32) = make_float4(v0[0], v0[1], v0[2], v0[3]);
            *reinterpret_cast<float4 *>(mine + gq * 32 + 4) = make_float4(v0[4], v0[5], v0[6], v0[7]);
        }
        if (gq + 8 < a.M) {
            *reinterpret_cast<float4 *>(mine + (gq + 8) * 32) = make_float4(v1[0], v1[1], v1[2], v1[3]);
            *reinterpret_cast<float4 *>(mine + (gq + 8) * 32 + 4) = make_float4(v1[4], v1[5], v1[6], v1[7]);
        }
        // One acquire-release ticket instead of fence + relaxed ticket + fence: the warp barrier orders the
        // lanes' partial stores before lane 0's release, and the last arriver's acquire before the lanes' loads.
        __syncwarp();
        uint32_t last = 0;
        if (lane == 0) {
            uint32_t seen;
            asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(seen) : "l"(a.tickets + grp) : "memory");
            last = seen == count - 1;
        }
        last = __shfl_sync(kFull, last, 0);
        __syncwarp();                                           // lane 0's acquire is ordered before every lane's loads
        if (!last) return;
        if (a.M <= 2) {
            // One or two activation rows: lane = column, up to sixteen partials of both rows in flight at
            // once, so the reduction costs one L2 round trip.  Fixed order: partial first_w, first_w + 1, ...
            float s0 = 0.f, s1 = 0.f;
            const bool two = a.M == 2;
            for (uint32_t w0 = first_w; w0 <= last_w; w0 += 16) {
                float t0[16], t1[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const bool in = w0 + i <= last_w;
                    const float *src = a.partial + (size_t)(w0 + i + grp) * a.M * 32 + lane;
                    t0[i] = in ? __ldcg(src) : 0.f;
                    t1[i] = (in && two) ? __ldcg(src + 32) : 0.f;
                }
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    s0 += t0[i];
                    s1 += t1[i];
                }
            }
            const uint32_t n = grp * 32 + lane;
            if (fused_ar) {                                     // even lanes exchange (n, n + 1) of both rows
                const float o0 = __shfl_down_sync(kFull, s0, 1), o1 = __shfl_down_sync(kFull, s1, 1);
                float2 r0 = make_float2(s0, o0), r1 = make_float2(s1, o1);
                if ((lane & 1) == 0 && n < g.N) {
                    r0 = fuse_exchange_pair(a.ar, ar_seq, n / 2, s0, o0);
                    if (two) r1 = fuse_exchange_pair(a.ar, ar_seq, (g.N + n) / 2, s1, o1);
                }
                const float u0 = __shfl_up_sync(kFull, r0.y, 1), u1 = __shfl_up_sync(kFull, r1.y, 1);
                s0 = (lane & 1) ? u0 : r0.x;
                s1 = (lane & 1) ? u1 : r1.x;
                if (lane == 0) fuse_group_done(a.ar, ar_seq, g.groups);
            }
            if (n < g.N) {
                const float b = a.bias ? load_bf16(a.bias + n) : 0.f;
                a.y[n] = float_to_bf16_bits(s0 + b);
                if (two) a.y[(size_t)a.ldy + n] = float_to_bf16_bits(s1 + b);
            }
        } else {
            // Four partials in flight at a time, each two rows of eight floats per lane.
            const bool has0 = gq < a.M, has1 = gq + 8 < a.M;
#pragma unroll
            for (int j = 0; j < 8; ++j) v0[j] = v1[j] = 0.f;
            const float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
            for (uint32_t w0 = first_w; w0 <= last_w; w0 += 4) {
                float4 t[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool in = w0 + i <= last_w;
                    const float *src = a.partial + (size_t)(w0 + i + grp) * a.M * 32 + 8 * q;
                    t[i][0] = (in && has0) ? __ldcg(reinterpret_cast<const float4 *>(src + gq * 32)) : z;
                    t[i][1] = (in && has0) ? __ldcg(reinterpret_cast<const float4 *>(src + gq * 32 + 4)) : z;
                    t[i][2] = (in && has1) ? __ldcg(reinterpret_cast<const float4 *>(src + (gq + 8) * 32)) : z;
                    t[i][3] = (in && has1) ? __ldcg(reinterpret_cast<const float4 *>(src + (gq + 8) * 32 + 4)) : z;
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    v0[0] += t[i][0].x; v0[1] += t[i][0].y; v0[2] += t[i][0].z; v0[3] += t[i][0].w;
                    v0[4] += t[i][1].x; v0[5] += t[i][1].y; v0[6] += t[i][1].z; v0[7] += t[i][1].w;
                    v1[0] += t[i][2].x; v1[1] += t[i][2].y; v1[2] += t[i][2].z; v1[3] += t[i][2].w;
                    v1[4] += t[i][3].x; v1[5] += t[i][3].y; v1[6] += t[i][3].z; v1[7] += t[i][3].w;
                }
            }
            store_row(gq, v0);
            store_row(gq + 8, v1);
        }
        __syncwarp();
        if (lane == 0) a.tickets[grp] = 0;                      // ready for the next call
    };

    // Activations of rows gq and gq + 8, four consecutive k of the lane's segment at a time.  Lanes without a row load nothing
    // (from rows that lie apart a load is a wavefront per segment and half warp).
    const bool has0 = gq < a.M, has1 = gq + 8 < a.M;
    const uint16_t *x0 = a.x + (p.x_order ? lane * 4 : (size_t)(has0 ? gq : 0) * a.ldx);
    const uint16_t *x1 = a.x + (p.x_order ? 128 + lane * 4 : (size_t)(has1 ? gq + 8 : 0) * a.ldx);
    const uint32_t x_step = p.x_order ? 16 * a.M : 4;
    uint32_t stage = 0;
    uint32_t cur_grp = grp;
    zero_acc();
    const uint32_t n_blocks = step / 4;                         // blocks of four symbols per stream
    const uint32_t n_chunks = (step + kChunkRows - 1) / kChunkRows;
    const uint32_t ragged_pk = (g.K % (2 * g.th)) ? p.pairs_k - 1 : 0xFFFFFFFFu;   // the unit index with rows beyond K
    uint32_t chunk = 0;                                         // sign+mantissa chunks consumed: buffer and phase parity

    Quad z;
    const uint8_t *man = man_of(grp, pk, sub);                  // the sign+mantissa chunk that was asked for last
    bool two = 2 * pk + 1 < g.tiles_k;
    for (uint32_t t = lo; t < hi; ++t) {
        const bool last_sub = !ENTRY || sub + 1 == subs, wrap = last_sub && pk + 1 == p.pairs_k;
        const uint32_t n_grp = grp + wrap, n_pk = wrap ? 0u : pk + last_sub, n_sub = last_sub ? 0u : sub + 1;   // of unit t + 1
        if (grp != cur_grp) {
            flush(cur_grp);
            zero_acc();
            cur_grp = grp;
        }
        const uint32_t krow = (2 * pk + tsel) * g.th + hsel * g.half + (ENTRY ? sub * step : 0u);
        // Blocks of this lane's segment that exist, and the rows of the last one (0 = all four); see the kernel's header.
        uint32_t n_my = n_blocks, len = n_blocks, cut = 0;
        uint32_t tsel_d = tsel, hsel_d = hsel;                  // the segment whose stream this lane decodes, its blocks: len
        bool empty = false;                                     // an entry point's unit may lie beyond K altogether
        const bool rag = RAGGED && pk == ragged_pk;             // the same for every lane: other units skip the bookkeeping
        if (rag) {
            const uint32_t seg = krow < g.K ? min(step, g.K - krow) : 0u;
            n_my = len = (seg + 3) >> 2;
            cut = seg & 3;
            const uint32_t top = 2 * pk * g.th + (ENTRY ? sub * step : 0u), top_rows = top < g.K ? min(step, g.K - top) : 0u;
            empty = top_rows == 0;
            if (seg == 0) {
                tsel_d = hsel_d = 0;
                len = (top_rows + 3) >> 2;
            }
        }
        const uint32_t r4 = pk * (g.half / 4) + (ENTRY ? sub * step / 4 : 0u);
        uint32_t xs = x_step;
        const size_t x_at = p.x_order ? (size_t)r4 * x_step : krow;
        const uint16_t *xp0 = x0 + x_at, *xp1 = x1 + x_at;
        if (RAGGED && n_my == 0 && !p.x_order) {
            xp0 = xp1 = g_zero_activations;
            xs = 0;
        }
        // Columns beyond N: see Quad::keep; a lane without any takes the first ones of its group.
        const uint32_t left_n = g.N - grp * 32, gq_d = 4 * gq < left_n ? gq : 0u;
        const uint32_t cols = min(4u, left_n - 4 * gq_d);
        const uint32_t ml = tsel_d ? nx_ml1 : nx_ml0;
        auto next_unit = [&]() {                                // every lane is done with the window it goes to
            if (t + 1 >= hi) return;
            if (t + 1 - dbase == 32) {
                dbase = t + 1;
                load_desc();
            }
            const uint32_t j = t + 1 - dbase;
            nx_off0 = __shfl_sync(kFull, d_off0, j);
            nx_ml0 = __shfl_sync(kFull, d_ml0, j);
            nx_off1 = __shfl_sync(kFull, d_off1, j);
            nx_ml1 = __shfl_sync(kFull, d_ml1, j);
            issue(n_grp, n_pk, n_sub, p.stages == 1 ? 0u : stage ^ 1, nx_off0, nx_ml0, nx_off1, nx_ml1);
        };
        // ---- this lane's four streams --------------------------------------
        const uint32_t win_s = wbase_s + stage * p.stage_bytes;
        const uint32_t st_s = win_s + st_off + tsel_d * 256 + (hsel_d * 32 + gq_d * 4) * 4;
        uint32_t first = win_s + tsel_d * 64 + hsel_d * 32 + gq_d * 4;
        if (!ENTRY && ml <= p.cap_rows) first += (ml - 1) * 128;   // last byte row; an empty tile starts one row below

        cp_async_wait();                                        // this unit's bytes and states, the first sign+mantissa chunk
        __syncwarp();
        auto start_streams = [&]() {
            z.start(st_s, first);
            if constexpr (ENTRY) {                              // every stream has its own row of the window
                const uint32_t rows_s = win_s + st_off + 512 + tsel_d * 128 + (hsel_d * 32 + gq_d * 4) * 2;
                const uint32_t r01 = lds_u32(rows_s), r23 = lds_u32(rows_s + 4);
                const uint32_t top = p.cap_rows - 1;
                z.p[0] += min(r01 & 0xFFFFu, top) * 128;
                z.p[1] += min(r01 >> 16, top) * 128;
                z.p[2] += min(r23 & 0xFFFFu, top) * 128;
                z.p[3] += min(r23 >> 16, top) * 128;
            }
            if (cols < 4) z.keep(cols);
        };
        start_streams();

        uint32_t wb[4][2] = {};
        uint32_t xf[4] = {};                                     // the group before: its weights, its activations
        uint32_t blk = 0, left = len;                           // left: blocks until this lane's stream is used up
        // Compiled for whole units and, in RAGGED, once more for the one of a column group that is not: with the tests in
        // one loop for both, all units paid for them.
        auto decode_unit = [&](auto rag_tag) {
            constexpr bool RAG = decltype(rag_tag)::value;
#pragma unroll 1
            for (uint32_t c = 0; c < n_chunks; ++c, ++chunk) {
                const uint32_t buf = chunk & 1;
                if (c != 0) {
                    cp_async_wait();                                // this chunk is here
                    __syncwarp();                                   // for every lane, and all are done with the other buffer
                }
                const bool last = c + 1 == n_chunks;
                if (last) {                                         // the next unit's first chunk
                    man = man_of(n_grp, n_pk, n_sub);
                    two = 2 * n_pk + 1 < g.tiles_k;
                } else {
                    man += kChunkRows * 32;
                }
                if (!last || t + 1 < hi) issue_man(man, two, last ? 0u : (c + 1) * kChunkRows, buf ^ 1);
                if (c == 0 && p.stages == 2) next_unit();
                z.clamp(win_s);
                uint32_t ms = man_s + (buf * 4 + q) * kSegPitch + gq * 4;
                const uint32_t end = RAG && empty ? 0u : min(blk + kChunkRows / 4, n_blocks);
#pragma unroll 1
                for (; blk < end; ++blk) {
                    const uint32_t m[4] = {lds_u32(ms), lds_u32(ms + 32), lds_u32(ms + 64), lds_u32(ms + 96)};
                    // The tensor instruction of the group before comes first: behind it the compiler knows that the warp is
                    // converged, and the register copies that its checks of that need go.
                    mma4<HI>(acc, wb, xf);
                    load_x(xf[0], xf[1], xp0, has0);                // used by the mma at the end
                    if constexpr (HI) load_x(xf[2], xf[3], xp1, has1);
                    rows2(wb, 0, z, lut_s, m[0], m[1]);
                    rows2(wb, 1, z, lut_s, m[2], m[3]);
                    if constexpr (RAG) {
                        const uint32_t n = blk + 1 < n_my ? 4u : blk >= n_my ? 0u : cut ? cut : 4u;   // rows of the block that exist
                        if (n < 4) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                wb[i][0] &= n == 0 ? 0u : n == 1 ? 0xFFFFu : 0xFFFFFFFFu;
                                wb[i][1] &= n == 3 ? 0xFFFFu : 0u;
                            }
                        }
                    }
                    ms += 128;
                    xp0 += xs;
                    if constexpr (HI) xp1 += xs;
                    if constexpr (RAG) {
                        if (blk + 1 == n_my && !p.x_order) { // rows beyond K from the next block on
                            xp0 = xp1 = g_zero_activations;
                            xs = 0;
                        }
                        if (--left == 0) {
                            left = len;
                            start_streams();
                        }
                    }
                }
            }
        };
        if constexpr (RAGGED) {
            if (rag) decode_unit(std::true_type{});
            else decode_unit(std::false_type{});
        } else {
            decode_unit(std::false_type{});
        }
        mma4<HI>(acc, wb, xf);
        if (p.stages == 1) {
            __syncwarp();                                       // every lane is done with the only window
            next_unit();
        } else {
            stage ^= 1;
        }
        grp = n_grp;
        pk = n_pk;
        sub = n_sub;
    }
    flush(cur_grp);
}

// The activations in the order in which the kernel's warps read them, [tile pair][four rows][M][segment][4], zeros beyond K: a
// warp's load of four rows is then one run of 32 M bytes (of 256 where M is larger than eight).  From rows K elements apart it is
// a cache line, and a wavefront of the load pipe, per row and segment.
__global__ void __launch_bounds__(256) k_interleave_x(const uint16_t *__restrict__ x, int64_t ldx, uint32_t K, XOrder order,
                                                      uint32_t pieces, uint32_t aligned, uint2 *__restrict__ out) {
    asm volatile("griddepcontrol.wait;" ::: "memory");          // the activations may be the previous kernel's product
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t i = blockIdx.x * 256 + threadIdx.x;
    if (i >= pieces) return;
    uint32_t m;
    const uint32_t k = 4 * order.k4(i, m);
    uint2 v = make_uint2(0u, 0u);
    if (k < K) {
        const uint16_t *src = x + (size_t)m * ldx + k;
        if (aligned) {
            v = __ldg(reinterpret_cast<const uint2 *>(src));
        } else {
            const uint32_t n = K - k;
            v.x = __ldg(src) | (n > 1 ? (uint32_t)__ldg(src + 1) << 16 : 0u);
            v.y = (n > 2 ? (uint32_t)__ldg(src + 2) : 0u) | (n > 3 ? (uint32_t)__ldg(src + 3) << 16 : 0u);
        }
    }
    out[i] = v;
}

// ------------------------------------------------------------------------ host

int launch_linear_mma4(const LinArgs &a, uint32_t max_tile_len, cudaStream_t s) {
    const Geom &g = a.g;
    // 16-symbol-aligned streams; the last pair of tile rows may lack its lower tile and either tile may be short
    if (g.tw != 32 || g.th % 16 != 0 || a.M > 16 || max_tile_len == 0) return 1;
    if ((reinterpret_cast<uintptr_t>(a.stream) & 15u) || (reinterpret_cast<uintptr_t>(a.mantissa) & 15u) ||
        (reinterpret_cast<uintptr_t>(a.states) & 15u))
        return 1;
    // activations are read as 8-byte quads: where they are not that, the reordering kernel makes them so
    const bool quads_ok = (reinterpret_cast<uintptr_t>(a.x) & 7u) == 0 && (a.ldx & 3) == 0 && g.K % 4 == 0;
    if (!quads_ok && a.x_scratch == nullptr && !a.dry_run) return 1;
    if (!quads_ok && a.ar.world > 1) return 1;                  // every rank has to take the same kernel: only plain cases
    int dev = 0, max_smem = 0;
    CI_CUDA(cudaGetDevice(&dev));
    CI_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    Mma4Args p;
    p.a = a;
    const bool entry = a.entry_step != 0 && a.entry_cap != 0 && g.half > a.entry_step && g.half % a.entry_step == 0 &&
                       a.entry_step % kChunkRows == 0 &&
                       ((reinterpret_cast<uintptr_t>(a.entry_states) | reinterpret_cast<uintptr_t>(a.entry_rows)) & 15u) == 0;
    p.cap_rows = entry ? a.entry_cap : max_tile_len;
    p.stage_bytes = (p.cap_rows * 128u + (entry ? 768u : 512u) + 127u) & ~127u;
    const uint32_t fixed = 2 * kLutBytes + kBar4Bytes;         // up to one table size is lost to the table's alignment
    const uint32_t room = (uint32_t)max_smem - fixed;
    const uint32_t P = (uint32_t)sm_count();
    p.pairs_k = (g.tiles_k + 1) / 2;
    p.step = entry ? a.entry_step : g.half;
    p.subs = g.half / p.step;
    p.per_group = p.pairs_k * p.subs;
    p.total = g.groups * p.per_group;
#ifndef CI_MMA4_MIN_UNITS
#define CI_MMA4_MIN_UNITS 6
#endif
    // A unit here is a serial chain twice as long as in the two-streams kernel (two tiles instead of one).
    // That pays once the multiprocessors are saturated (about eight warps each); a small matrix -- a
    // tensor-parallel shard, say -- is latency bound and finishes sooner with the shorter units
    // (measured cross-over: 4096 x 2048 at tile height 128).  The two-streams kernel takes tiles of up to 256 rows.
    if (g.th <= 256 && !entry && p.total < P * CI_MMA4_MIN_UNITS) return 1;
    // One CTA per multiprocessor, the units dealt out in equal runs (they differ by one at most).  The warp count decides
    // how well the last round is filled.  One row, us: 11008 x 4096 takes two rounds of 19 warps 36.9, 2.7 of 14 41.1;
    // 4096 x 22016 takes 3.7 rounds of 20 warps 67.2, 4.7 of 16 70.1, 5.4 of 14 78.1; 4096 x 12288 2.6 of 16 42.6, 2.1 of
    // 20 45.7.  A second window per warp, which hides the copies of the next unit, is worth 2 %: less than a warp that would
    // not fit beside it.
    const uint32_t x_rows = p.pairs_k * 2 * g.th;               // K, rounded up to whole tile pairs
    uint32_t warps = 0;
    bool many = false;
    double best = 0.0;
    const uint32_t units = (p.total + P - 1) / P;
    for (uint32_t stages = 2; stages >= 1; --stages) {
        uint32_t w_max = room / (stages * p.stage_bytes + kManBytes);
        if (w_max > kMma4ManyWarps) w_max = kMma4ManyWarps;
        for (uint32_t w = 1; w <= w_max; ++w) {
            const double cost = run_cost(units, w, 0.3) * (stages == 1 ? 1.02 : 1.0);
            if (warps == 0 || cost < best) { best = cost; warps = w; many = w > kMma4Warps; p.stages = stages; }
        }
    }
    if (warps == 0 || (g.th <= 256 && !entry && warps < 4)) return 1;
    const uint32_t warp_bytes = p.stages * p.stage_bytes + kManBytes;
    uint32_t blocks = (p.total + warps - 1) / warps;
    if (blocks > P) blocks = P;
    p.slots = blocks * warps < p.total ? blocks * warps : p.total;
    if ((uint64_t)p.slots * (p.total + 1) >> 32) return 1;      // 1.8 million units
    p.y_vec = ((reinterpret_cast<uintptr_t>(a.y) & 15u) == 0 && (a.ldy & 7) == 0) ? 1u : 0u;
    p.x_order = 0;
    p.status = a.tickets + (kTicketBytes - 1);
    if (a.dry_run) return CI_OK;                                // qualification only

    const bool ragged = g.K % (2 * g.th) != 0;
#define CI_MMA4_SET(E, W)                                                                                            \
    k_linear_mma4<false, false, E, W>, k_linear_mma4<true, false, E, W>, k_linear_mma4<false, true, E, W>,           \
        k_linear_mma4<true, true, E, W>
    static void (*const kernels[16])(Mma4Args) = {CI_MMA4_SET(false, kMma4Warps), CI_MMA4_SET(false, kMma4ManyWarps),
                                                  CI_MMA4_SET(true, kMma4Warps), CI_MMA4_SET(true, kMma4ManyWarps)};
#undef CI_MMA4_SET
    static SmemLimit lim[16] = {};
    const int which = (a.M > 8) + 2 * ragged + 4 * many + 8 * entry;
    void (*kernel)(Mma4Args) = kernels[which];
    if (int rc = ensure_smem_limit(lim[which], (const void *)kernel, (size_t)max_smem)) return rc;
    // Programmatic dependent launch: the grid may be scheduled while the previous kernel of the stream
    // drains; the kernel itself waits for that kernel before it reads activations or touches the workspace.
    cudaLaunchConfig_t cfg = {};
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    // The launch in front costs about 2 us and takes a wavefront per row beyond the first, segment and four rows of a unit out of
    // the load pipe.  us without -> with: 4096 x 4096 at 6 rows 20.1 -> 20.9, 8 21.3 -> 20.9, 16 27.7 -> 22.2; 5504 x 4100 at
    // 2 rows 22.3 -> 24.1, 5 26.7 -> 25.9; 4096 x 22016 at 2 rows 70.9 -> 71.5, 3 74.0 -> 72.0, 16 121.2 -> 75.8; at tile
    // height 64, where the steps of a short unit wait for less, 6784 x 5168 at 4 rows 32.9 -> 33.7, 8 34.9 -> 34.1; with so few units
    // that the pipe is not busy, 4936 x 2120 at tile height 1024 and 13 rows 27.6 -> 28.9.  The lines lie so that none of these
    // loses; the number of products alone does not tell gain from loss to the last 2 %, so that 4096 x 4096 at 8 and 9 rows, for
    // one, goes without.
    const uint64_t x_lines = (uint64_t)(a.M - 1) * g.K * g.N;
    const bool reorder = a.x_scratch != nullptr && a.M >= 3 && x_lines >= (p.step < 64 ? 200000000ull : units >= 16 ? 90000000ull : 150000000ull);
    if (!quads_ok || reorder) {
        const uint32_t pieces = x_rows / 4 * a.M;
        cfg.gridDim = dim3((pieces + 255) / 256);
        cfg.blockDim = dim3(256);
        CI_CUDA(cudaLaunchKernelEx(&cfg, k_interleave_x, a.x, a.ldx, g.K, XOrder{g.half / 4, a.M}, pieces, (uint32_t)quads_ok,
                                   reinterpret_cast<uint2 *>(a.x_scratch)));
        p.a.x = a.x_scratch;
        p.x_order = 1;
    }
    cfg.gridDim = dim3(blocks);
    cfg.blockDim = dim3(warps * 32);
    cfg.dynamicSmemBytes = fixed + (size_t)warps * warp_bytes;
    CI_CUDA(cudaLaunchKernelEx(&cfg, kernel, p));
    return CI_OK;
}

}  // namespace ci
