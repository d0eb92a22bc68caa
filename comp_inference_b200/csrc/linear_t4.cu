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
// A unit yields a sum for every row, so the sums live in shared memory, private to the warp: read as the mma's C operand
// and written back, two 8-byte loads and stores per two rows.  The warps of a CTA take column blocks of the same four
// tiles ("group"); at the end of its run in a group the CTA adds its warps' sums, writes an fp32 partial and draws a
// ticket; the CTA that draws the last one adds the partials in a fixed order and writes bf16.
//
// Bytes are staged as in linear_mma4.cu: one window of 128-byte rows per unit (a shared-memory bank per lane), sign and
// mantissa in 16-row chunks.  Bound by the decode step like that kernel.  Measured on a B200, 32000 x 4096, one row, tile
// height 128: 1000 us (the shuffle kernel) -> 139; 32000 x 5120 at tile height 1024: 516 us without entry points -> 274 with
// them, eight rows 3590 -> 444.
#include "linear.cuh"
#include "ptx.cuh"

namespace ci {

constexpr uint32_t kT4Warps = 16;
constexpr uint32_t kT4BarBytes = 640;        // up to 16 warps x (2 window stages + 2 chunks) x 8 B
constexpr uint32_t kT4SegPitch = kChunkRows * 16 + 16;       // eight segments of a chunk, 4 banks apart
constexpr uint32_t kT4ManBytes = 2 * 8 * kT4SegPitch;

struct T4Args {
    LinArgs a;
    uint32_t cap_rows;     // rows of a byte window (>= every tile_max_len)
    uint32_t stage_bytes;
    uint32_t stages;       // windows per warp
    uint32_t acc_bytes;    // sums of a warp
    uint32_t cblocks;      // 16-column blocks per group
    uint32_t subs, step;   // ENTRY: groups per four tiles, the rows of a segment in each; else 1, half a tile
    uint32_t total;        // units
    uint32_t *status;
};

// MT: sums per row in shared memory (1, 2 or 8 activation rows).
// ENTRY: a group is the rows of four tiles between two entry points (see linear_mma4.cu), so its sums are those of a short
// tile; without, a tall tile's sums and window leave room for three warps.
template <int MT, bool ENTRY>
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
    const uint32_t bar_base = lut_s + kLutBytes + warp * 32, man_bar = bar_base + 16;
    const uint32_t man_s = lut_s + kLutBytes + kT4BarBytes + warp * kT4ManBytes;
    const uint32_t acc0_s = lut_s + kLutBytes + kT4BarBytes + W * kT4ManBytes, acc_s = acc0_s + warp * p.acc_bytes;
    const uint32_t wbase_s = acc0_s + W * p.acc_bytes + warp * p.stages * p.stage_bytes;
    const uint32_t subs = ENTRY ? p.subs : 1u, step = ENTRY ? p.step : g.half;
    const uint32_t seg_acc = step * (MT * 4) + (MT == 8 ? 32 : MT * 4);  // bytes between the sums of two segments
    __shared__ uint32_t s_flag;

    const uint32_t sg = lane >> 2, q = lane & 3;                // row segment and column quad of this lane
    // Units of this CTA: [lo, hi), column block running fastest; those of a group are dealt to the warps in turn.
    const uint32_t lo = (uint32_t)((uint64_t)blockIdx.x * p.total / gridDim.x);
    const uint32_t hi = (uint32_t)((uint64_t)(blockIdx.x + 1) * p.total / gridDim.x);

    auto group_end = [&](uint32_t u) { return min(hi, (u / p.cblocks + 1) * p.cblocks); };
    // u: a unit of this warp in the run that began at base -> the next one, base updated; hi when there is none
    auto advance = [&](uint32_t u, uint32_t &base) {
        uint32_t n = u + W;
        while (n >= group_end(base)) {
            base = group_end(base);
            if (base >= hi) return hi;
            n = base + warp;
        }
        return n;
    };

    // Lanes 0..3: byte offset and depth of the group's four tiles in unit u's tile column.
    auto load_desc = [&](uint32_t u, uint32_t &off, uint32_t &ml) {
        off = ml = 0;
        if (u >= hi || lane >= 4) return;
        const uint32_t grp = u / p.cblocks, ct = (u - grp * p.cblocks) >> 1, tk = 4 * (grp / subs) + lane;
        if (tk >= g.tiles_k) return;
        const size_t tile = (size_t)tk * g.tiles_n + ct;
        off = __ldg(a.tile_offsets + tile);
        if constexpr (ENTRY) {
            ml = enter_span(__ldg(a.entry_spans + tile * subs + grp % subs), __ldg(a.tile_max_lens + tile), off);
        } else {
            ml = __ldg(a.tile_max_lens + tile);
        }
    };
    auto issue = [&](uint32_t u, uint32_t stage, uint32_t off, uint32_t ml) {
        const uint32_t hb = u % p.cblocks & 1, dst = wbase_s + stage * p.stage_bytes;
        if (ml > p.cap_rows) {                                  // metadata disagrees with the declared maximum
            atomicExch(p.status, 2u);
            ml = 0;
        }
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t n = __shfl_sync(kFull, ml, j) * 2;
            const uint8_t *src = a.stream + __shfl_sync(kFull, off, j) + hb * 16;
            for (uint32_t i = lane; i < n; i += 32)             // (row i / 2, half i % 2)
                cp_async16(dst + (i >> 1) * 128 + j * 32 + (i & 1) * 16, src + (size_t)(i >> 1) * 64 + (i & 1) * 32);
        }
        cp_async_arrive(bar_base + stage * 8);
    };
    auto issue_man = [&](uint32_t u, uint32_t c, uint32_t buf) {
        const uint32_t grp = u / p.cblocks, cb = u - grp * p.cblocks;
        const uint32_t row = lane & 15, h = lane >> 4;          // a lane copies one row of one half of every tile
        if (c * kChunkRows + row < step) {
            const uint32_t tk0 = 4 * (grp / subs), sub_row = ENTRY ? grp % subs * step : 0u;
            const uint8_t *src = a.mantissa + (((size_t)tk0 * g.tiles_n + (cb >> 1)) * g.th + h * g.half + sub_row + c * kChunkRows + row) * 32 +
                                 (cb & 1) * 16;
            const uint32_t dst = man_s + (buf * 8 + h) * kT4SegPitch + row * 16;
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j)
                if (tk0 + j < g.tiles_k) cp_async16(dst + 2 * j * kT4SegPitch, src + (size_t)j * g.tiles_n * g.th * 32);
        }
        cp_async_arrive(man_bar + buf * 8);
    };
    // The segment whose streams this lane decodes: its own, or, where the group has no such tile, the same half of the
    // first one (real symbols; random ones would take the branch for a second byte at every step).
    auto seg_of = [&](uint32_t grp) { return 4 * (grp / subs) + (sg >> 1) < g.tiles_k ? sg : sg & 1; };
    // Initial states of this lane's streams in unit u; a column beyond the matrix repeats the block's first one (its
    // weights are finite and meet zero activations).
    auto load_states = [&](uint32_t u, uint32_t (&s)[4], uint32_t (&rows)[4]) {
        const uint32_t grp = u / p.cblocks, cb = u - grp * p.cblocks, tk = 4 * (grp / subs) + (seg_of(grp) >> 1);
        rows[0] = rows[1] = rows[2] = rows[3] = 0;
        const size_t at = (((size_t)tk * g.tiles_n + (cb >> 1)) * subs + (ENTRY ? grp % subs : 0u)) * 64 + (sg & 1) * 32 + (cb & 1) * 16;
        const uint32_t *src = (ENTRY ? a.entry_states : a.states) + at;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) {
            const uint32_t c = cb * 16 + 4 * q + j < g.N ? 4 * q + j : 0u;
            s[j] = __ldg(src + c);
            if constexpr (ENTRY) rows[j] = min((uint32_t)__ldg(a.entry_rows + at + c), p.cap_rows - 1);
        }
    };

    if (lane == 0) {
        for (uint32_t i = 0; i < 4; ++i) mbar_init(bar_base + 8 * i, 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    uint32_t base = lo;
    uint32_t u = lo + warp < group_end(lo) ? lo + warp : advance(lo + warp - W, base);
    uint32_t nbase = base, nu = u < hi ? advance(u, nbase) : hi;
    uint32_t off, ml, noff, nml;
    load_desc(u, off, ml);
    load_desc(nu, noff, nml);
    if (u < hi) {
        issue(u, 0, off, ml);
        issue_man(u, 0, 0);
    }
    if (a.lut == nullptr) load_lut(s_lut, nullptr, a.tables, a.slot_map);
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");          // everything above touched only the weight
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (!wait_lut(lut_bar, a.lut)) atomicExch(p.status, 1u);
    const bool live_m = MT == 8 ? 2 * q < a.M : q == 0;         // lanes whose two D columns are activation rows
    const uint32_t n_chunks = (step + kChunkRows - 1) / kChunkRows;
    uint32_t parity0 = 0, parity1 = 0, stage = 0, chunk = 0;
    Quad z;
    for (uint32_t run = lo; run < hi; run = group_end(run)) {   // the CTA's runs: one per group it touches
        const uint32_t end = group_end(run), grp = run / p.cblocks;
        for (uint32_t i = lane * 4; i < p.acc_bytes; i += 128) asm volatile("st.shared.u32 [%0], %1;" ::"r"(acc_s + i), "r"(0u) : "memory");
        __syncwarp();
        for (; u < end; u = nu, base = nbase, nu = u < hi ? advance(u, nbase) : hi) {
            const uint32_t cb = u - grp * p.cblocks, col = cb * 16 + 4 * q;
            uint32_t next_row[4];
            load_states(u, z.s, next_row);
            uint32_t xb[2] = {0u, 0u};                          // activations of row sg, columns col .. col + 3
            if (sg < a.M) {
                const uint16_t *x = a.x + (size_t)sg * a.ldx + col;
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j)
                    if (col + j < g.N) xb[j >> 1] |= (uint32_t)__ldg(x + j) << (16 * (j & 1));
            }
            const uint32_t sd = seg_of(grp), my_ml = __shfl_sync(kFull, ml, sd >> 1);
            const uint32_t win_s = wbase_s + stage * p.stage_bytes;
            const uint32_t first = win_s + (!ENTRY && my_ml <= p.cap_rows ? my_ml - 1 : 0u) * 128 + sd * 16;
#pragma unroll
            for (uint32_t j = 0; j < 4; ++j) z.p[j] = first + next_row[j] * 128 + (col + j < g.N ? 4 * q + j : 0u);
            if (!mbar_wait(bar_base + stage * 8, stage ? parity1 : parity0)) atomicExch(p.status, 1u);
            if (stage) parity1 ^= 1; else parity0 ^= 1;
            auto next_unit = [&]() {
                off = noff;
                ml = nml;
                if (nu >= hi) return;
                issue(nu, p.stages == 2 ? stage ^ 1 : 0u, off, ml);
                uint32_t b2 = nbase;
                load_desc(advance(nu, b2), noff, nml);
            };
            uint32_t ac = acc_s + sg * seg_acc + (MT == 8 ? q * 8 : 0u);
#pragma unroll 1
            for (uint32_t c = 0; c < n_chunks; ++c, ++chunk) {
                const uint32_t buf = chunk & 1;
                __syncwarp();                                   // every lane is done with the other buffers
                if (c + 1 < n_chunks) issue_man(u, c + 1, buf ^ 1);
                else if (nu < hi) issue_man(nu, 0, buf ^ 1);
                if (c == 0 && p.stages == 2) next_unit();       // behind it: a chunk's arrival waits for older copies
                if (!mbar_wait(man_bar + buf * 8, (chunk >> 1) & 1)) atomicExch(p.status, 1u);
                z.clamp(win_s);
                uint32_t ms = man_s + (buf * 8 + sg) * kT4SegPitch + q * 4;
                const uint32_t n = min(kChunkRows, step - c * kChunkRows);
#pragma unroll 1
                for (uint32_t r = 0; r < n; r += 4) {
#pragma unroll
                    for (uint32_t i = 0; i < 4; i += 2) {
                        float d[4] = {0.f, 0.f, 0.f, 0.f};
                        const uint32_t ad = ac + i * (MT * 4);
                        if (live_m) {
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
                            z.step(lut_s, e);
                            const uint32_t m = lds_u32(ms + (i + k) * 16);
                            const uint32_t e01 = __byte_perm(e[0], e[1], 0x6521) << 3, e23 = __byte_perm(e[2], e[3], 0x6521) << 3;
                            w[k] = exp_or_man(e01, __byte_perm(m, 0u, 0x1100));
                            w[2 + k] = exp_or_man(e23, __byte_perm(m, 0u, 0x3322));
                        }
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
                    ac += 4 * (MT * 4);
                    ms += 64;
                }
            }
            if (p.stages == 2) {
                stage ^= 1;
            } else {
                __syncwarp();                                   // every lane is done with the only window
                next_unit();
            }
        }
        // ---- the group's sums of this CTA ------------------------------------------------------------------
        __syncthreads();
        const uint32_t rows = 8 * step, first_cta = (uint32_t)(((uint64_t)(grp * p.cblocks + 1) * gridDim.x - 1) / p.total);
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
            const uint32_t at = acc0_s + seg * seg_acc + (r - seg * step) * (MT * 4) + m * 4;
            float sum = 0.f;
            for (uint32_t w = 0; w < W; ++w) sum += __uint_as_float(lds_u32(at + w * p.acc_bytes));
            if (count > 1) {
                mine[i] = sum;
            } else if (v < g.K) {
                if (a.bias) sum += load_bf16(a.bias + v);
                a.y[(size_t)m * a.ldy + v] = float_to_bf16_bits(sum);
            }
        }
        if (count > 1) {
            if (last_arrival(a.tickets + grp, count, &s_flag)) {
                for (uint32_t i = threadIdx.x; i < rows * a.M; i += blockDim.x) {
                    const uint32_t m = i / rows, v = out_row(i - m * rows);
                    if (v >= g.K) continue;
                    float sum = 0.f;
                    for (uint32_t c = first_cta; c <= last_cta; ++c) sum += __ldcg(a.partial + (size_t)(c + grp) * rows * a.M + i);
                    if (a.bias) sum += load_bf16(a.bias + v);
                    a.y[(size_t)m * a.ldy + v] = float_to_bf16_bits(sum);
                }
                if (threadIdx.x == 0) a.tickets[grp] = 0;       // ready for the next call
            }
        }
        __syncthreads();                                        // the sums may be cleared
    }
}

// ------------------------------------------------------------------------ host

template <int MT, bool ENTRY>
static int launch_t4_pass(T4Args p, uint32_t blocks, uint32_t warps, size_t smem, int max_smem, cudaStream_t s) {
    static SmemLimit lim = {};
    if (int rc = ensure_smem_limit(lim, (const void *)k_linear_t4<MT, ENTRY>, (size_t)max_smem - 1024)) return rc;
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
    CI_CUDA(cudaLaunchKernelEx(&cfg, k_linear_t4<MT, ENTRY>, p));
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
                       a.entry_step % kChunkRows == 0;
    const uint32_t step = entry ? a.entry_step : g.half, subs = g.half / step, groups = (g.tiles_k + 3) / 4 * subs;
    if (groups >= kTicketBytes - 1) return 1;
    int dev = 0, max_smem = 0;
    CI_CUDA(cudaGetDevice(&dev));
    CI_CUDA(cudaDeviceGetAttribute(&max_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    T4Args p;
    p.cap_rows = entry ? a.entry_cap : max_tile_len;
    p.step = step;
    p.subs = subs;
    p.stage_bytes = p.cap_rows * 128u;
    p.cblocks = (g.N + 15) / 16;
    p.total = groups * p.cblocks;
    p.status = a.tickets + (kTicketBytes - 1);
    const uint32_t P = (uint32_t)sm_count(), fixed = 2 * kLutBytes + kT4BarBytes + 1024, room = (uint32_t)max_smem - fixed;
    const uint32_t blocks = p.total < P ? p.total : P;
    // Passes over the weight x rounds of units: sums for eight activation rows take eight times the shared memory of one,
    // which a tall tile cannot afford at a useful number of warps.  The units of a CTA count as one sequence here, without the
    // barrier that ends each of its groups: at 32000 x 4096 and tile height 128, 47 of 148 CTAs take 8 rounds for 6.8 rounds of work.
    uint32_t warps = 0, rows_per_pass = 0;
    double best = 0.0;
    for (uint32_t mt = 1; mt <= 8; mt = mt == 2 ? 8 : mt * 2)
        for (uint32_t stages = 1; stages <= 2; ++stages) {
            const uint32_t acc = (8 * (step * (mt * 4) + (mt == 8 ? 32 : mt * 4)) + 15) & ~15u;
            const uint32_t warp_bytes = stages * p.stage_bytes + kT4ManBytes + acc;
            uint32_t w_max = room / warp_bytes;
            if (w_max > kT4Warps) w_max = kT4Warps;
            for (uint32_t w = 1; w <= w_max; ++w) {
                const double cost = (double)((a.M + mt - 1) / mt) * run_cost((p.total + blocks - 1) / blocks, w, 0.0) *
                                    (stages == 1 ? 1.02 : 1.0);
                if (warps == 0 || cost < best) {
                    best = cost;
                    warps = w;
                    rows_per_pass = mt;
                    p.stages = stages;
                    p.acc_bytes = acc;
                }
            }
        }
    if (warps == 0) return 1;
    const size_t smem = fixed - 1024 + (size_t)warps * (p.stages * p.stage_bytes + kT4ManBytes + p.acc_bytes);
    for (uint32_t m0 = 0; m0 < a.M; m0 += rows_per_pass) {
        p.a = a;
        p.a.x = a.x + (size_t)m0 * a.ldx;
        p.a.y = a.y + (size_t)m0 * a.ldy;
        p.a.M = a.M - m0 < rows_per_pass ? a.M - m0 : rows_per_pass;
        int rc;
        if (entry)
            rc = rows_per_pass == 1   ? launch_t4_pass<1, true>(p, blocks, warps, smem, max_smem, s)
                 : rows_per_pass == 2 ? launch_t4_pass<2, true>(p, blocks, warps, smem, max_smem, s)
                                      : launch_t4_pass<8, true>(p, blocks, warps, smem, max_smem, s);
        else
            rc = rows_per_pass == 1   ? launch_t4_pass<1, false>(p, blocks, warps, smem, max_smem, s)
                 : rows_per_pass == 2 ? launch_t4_pass<2, false>(p, blocks, warps, smem, max_smem, s)
                                      : launch_t4_pass<8, false>(p, blocks, warps, smem, max_smem, s);
        if (rc) return rc;
    }
    return CI_OK;
}

}  // namespace ci
