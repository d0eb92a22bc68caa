// Shared declarations of the stand-alone decoders.
#pragma once
#include "common.cuh"

namespace ci {

struct DecArgs {
    const uint8_t *stream;
    const uint32_t *states, *tables, *tile_offsets, *tile_max_lens, *lut;
    const uint8_t *slot_map, *mantissa;
    Geom g;
    uint32_t stream_aligned;   // stream pointer is 16-byte aligned
    uint32_t ld;               // elements from one output row to the next
    // entry points into the streams of tall tiles (ci_build_entry_points), step 0: none
    uint32_t entry_step, entry_cap;
    const uint32_t *entry_states, *entry_spans;
    const uint16_t *entry_rows;
};

// Every launcher: CI_OK when launched, 1 when the tensor does not qualify (the caller then tries the next one), < 0 on error.
// Four-streams-per-lane decoder for 32-wide tiles (decode4.cu).
int launch_decode4(const DecArgs &a, uint32_t max_tile_len, bool bf16, void *out, cudaStream_t s);
// Two streams per lane (decode2.cu), where few streams leave that one too few warps.
double decode4_cost(const DecArgs &a, uint32_t max_tile_len, bool bf16);   // run_cost of launch_decode4, 0: it does not qualify
int launch_decode2(const DecArgs &a, uint32_t max_tile_len, bool bf16, void *out, cudaStream_t s);
int build_entry_points(const DecArgs &a, uint32_t max_tile_len, uint32_t step, uint32_t *d_states, uint16_t *d_rows,
                       uint32_t *d_spans, uint32_t *d_cap, cudaStream_t s);
// Other tile widths, unaligned states (decode_staged.cu).
int launch_decode_staged(const DecArgs &a, uint32_t max_tile_len, bool bf16, void *out, cudaStream_t s);

}  // namespace ci
