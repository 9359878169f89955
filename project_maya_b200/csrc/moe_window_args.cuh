// moe_window_args.cuh - the argument block of the streamed window kernels (moe_window.cuh) and their launchers.
#pragma once

#include "maya_internal.cuh"

namespace maya {

constexpr int kWMaxGroups = 128;     // T <= 16 tokens x 8 routes

// What a launch works on.
struct WArgs {
    const unsigned long long* ptr;   // [groups] blob addresses (0: skipped)
    const int* start;                // [groups + 1] entry ranges
    int* n_groups;                   // device count; set to -1 when a wait ran out
    const int* ent_slot;             // [entries] an entry's h / partial slot: 8 token + route
    unsigned* error;                 // optional: set to 1 when a wait ran out
    unsigned polls;                  // looks at a row's copy before a warp gives up
    int cap;                         // most groups (<= kWMaxGroups)
    int ncm;                         // columns of a job, <= kWNC
    int plain;                       // the rows do not start and end on 16-byte boundaries inside a blob: no bulk copies
    int n_embd, n_ff;
    size_t row_off;                  // byte offset of the rows in a blob: gate/up 0, down: the down rows
    size_t up_off;                   // gate/up: byte offset of the up rows
    float limit;
    const uint8_t* xq;               // gate/up: token columns, xq_stride apart; down: h images [slot]
    size_t xq_stride;
    uint8_t* hq;                     // gate/up out: [slot][n_ff / 32] q8_1
    float* part;                     // down out: [slot][n_embd]
    const uint8_t* sh;               // the shared expert's rows (NULL: none): gate rows then up rows, or down rows
    int n_ff_sh, n_tok;              // its width; every one of n_tok tokens uses it
    uint8_t* sh_hq;                  // [n_tok][n_ff_sh / 32] q8_1: gate/up out, down in
    float* sh_out;                   // down out: [n_tok][n_embd]
};

// By type (GROUP 0: Q8_0, the K-quants and IQ4_XS, 1: the codebook types); SH: with A.sh.  kWindowTooWide: the rows are
// longer than a column has room for, nothing launched.
template<bool SH, bool UP, int GROUP> int launch_window_group(int type, const WArgs& A, cudaStream_t s);

}  // namespace maya
