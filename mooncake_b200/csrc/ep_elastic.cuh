// Kernels of the elastic-style calls (flat receive layout, one copy of a token
// per destination rank). The exchange itself is the group dispatch / combine of
// ep_kernels.cu with every rank standing for one "expert"; the kernels here
// prepare its routing input and turn its outputs into the tensors the elastic
// interface returns.
//
// Reference (paths inside the Mooncake tree): the interface is
// mooncake-wheel/mooncake/mooncake_elastic_buffer.py:437-774, the device code
// mooncake-ep/include/elastic/mooncake_ep_elastic_dispatch_official.cuh,
// ..._dispatch_copy_epilogue.cuh, ..._combine_official.cuh and
// ..._combine_reduce_epilogue.cuh.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "ep_kernels.cuh"

namespace mcep {

// A record per row a rank is about to receive, stored by the source in the
// receiver's memory at [source rank][position among the source's rows]:
// [K] int32 expert choices, [K] fp32 weights, int32 token index at the source.
// `record_stride` bytes apart; one set per parity.
struct ElasticRouteParams {
    const int64_t* topk_idx;     // [T][K]
    const float* topk_weights;   // [T][K] or null
    int T, K, E, R, M, rank;
    int64_t* rank_topk;          // [T][K] destination rank at its last listing inside the token, else -1
    int32_t* dst_slot;           // [T][K] rank * M + position among this rank's tokens for that destination, else -1
    int64_t* copied_topk_idx;    // [T][K] copy of topk_idx kept with the handle, or null
    void* const* record_base;    // [R] every rank's record area of this call's parity (null: not mapped)
    int record_stride;
    char fill[16];
};
static_assert(cheap_to_launch<ElasticRouteParams>);
cudaError_t launch_elastic_route(const ElasticRouteParams& p, cudaStream_t stream);

struct ElasticEpilogueParams {
    const int64_t* layout_range;  // [R] (begin << 32) | count, as the exchange left it
    const char* records;          // this rank's record area of this call's parity
    int record_stride;
    int R, M, K, L, rank;
    int alignment;                // expert_alignment
    int expand;
    int64_t* recv_topk_idx;       // [n][K] local expert or -1
    float* recv_topk_weights;     // [n][K] or null (expand: scratch, scattered later)
    int32_t* recv_src_metadata;   // [n][K+2]
    int32_t* psum_rank;           // [R] inclusive
    int32_t* psum_expert;         // [L+1] exclusive, aligned counts
    int32_t* psum_start;          // expand: [L+1] copy kept while psum_expert becomes the segment ends
    int32_t* hist;                // [L] scratch, zero between calls
    unsigned* ticket;             // scratch word, zero between calls
    int32_t* status;
    char fill[40];
};
static_assert(cheap_to_launch<ElasticEpilogueParams>);
cudaError_t launch_elastic_epilogue(const ElasticEpilogueParams& p, int num_sms, cudaStream_t stream,
                                    bool pdl);

// Expanded layout: one row per (received token, local expert it chose), experts'
// segments starting at psum_start[e], rows of one expert in receive order.
struct ElasticExpandParams {
    const int64_t* layout_range;  // [R]
    const int64_t* recv_topk_idx; // [n][K]
    const float* flat_weights;    // [n][K] or null
    const void* flat_x;           // [n][row_bytes]
    int R, K, L, row_bytes;
    const int32_t* psum_start;    // [L+1]
    int32_t* psum_expert;         // [L+1]: entries < L become the ends of the segments
    int32_t* recv_src_metadata;   // [n][K+2], columns 2.. written here
    void* recv_x;                 // [max_rows][row_bytes]
    float* recv_topk_weights;     // [max_rows] or null
    int max_rows;                 // rows that aligned segments push beyond are dropped (metadata -1, status)
    int32_t* status;
    char fill[56];
};
static_assert(cheap_to_launch<ElasticExpandParams>);
cudaError_t launch_elastic_expand_scan(const ElasticExpandParams& p, cudaStream_t stream);
cudaError_t launch_elastic_expand_copy(const ElasticExpandParams& p, int num_sms, cudaStream_t stream);

// Expanded layout, combine side: the rows of one received token are summed into
// one row before they travel (1 row: copied; more: fp32 accumulation in listing
// order, rounded to bf16 once; none, all dropped by the dispatch call: zeros).
struct ElasticLocalReduceParams {
    const int64_t* layout_range;      // [R]
    const int32_t* recv_src_metadata; // [n][K+2]
    const void* x;                    // [x_rows][H] bf16
    int R, K, H, x_rows;
    void* y;                          // [n][H] bf16
    char fill[48];
};
static_assert(cheap_to_launch<ElasticLocalReduceParams>);
cudaError_t launch_elastic_local_reduce(const ElasticLocalReduceParams& p, int num_sms,
                                        cudaStream_t stream);

// ---- a single rank ----------------------------------------------------------------------
// Nothing is exchanged: a received row is the token itself, its position the number
// of earlier tokens that name any expert, its expanded rows follow from the routing
// alone. One launch (small batches) or two (layout, copy) write all outputs, the
// rows go straight to where they end up, and combine gathers from there.
struct ElasticSingleParams {
    const void* x;               // [T][H] bf16
    const int64_t* topk_idx;     // [T][K]
    const float* topk_weights;   // [T][K] or null
    int T, K, E, H, alignment;
    int C;                       // tokens per block of the copy kernel, and behind a layout kernel
    int warps_per_row, parts;    // the warps and the blocks that share a row (set by the launcher)
    bool x_last;                 // see input_beyond_l2 (set by the launcher)
    bool own_segments;
    int max_rows;                // expanded: rows recv_x has room for
    int32_t* status;
    int32_t* rows;               // kept for combine: [T] received row of the token, or (expanded) [T][K] row
                                 // of the entry; -1: none
    int32_t* token_pos;          // expanded: [T] scratch, received row of the token (else == rows)
    void* recv_x;
    int64_t* recv_topk_idx;      // [n][K]
    float* recv_topk_weights;    // [n][K], expanded: [rows]; or null
    int32_t* recv_src_metadata;  // [n][K+2]
    int32_t* dst_slot;           // [T][K]
    int64_t* copied_topk_idx;    // [T][K] or null
    int32_t* psum_rank;          // [1]
    int32_t* psum_expert;        // [E+1]
    // a caller that waits for the counts: host memory the device can write,
    // [0] flag (host_seq once the rest is there), [1] received rows, [2..] psum_expert
    int32_t* host_counts;
    int32_t host_seq;
    RouteBits bits;              // behind a layout kernel: row 0 all tokens that name an expert, 1 + e (expanded)
                                 // those that name e
    unsigned long long* totals;  // [E] listings and rows of the experts, zero between calls
    union {                      // expanded
        int32_t* starts;         // [E + 1] where the experts' segments start, or (own_segments)
        uint16_t* listings;      // [E][chunks, padded] of every chunk, segments made of them in the copy kernel
    };
    unsigned* ticket;            // expanded: chunks that are done
};
static_assert(cheap_to_launch<ElasticSingleParams>);
// The tables of the layout kernel; bits.words null: no launch of its own, the copy kernel counts.
struct SingleTables {
    RouteBits bits = {};
    int32_t* starts = nullptr;
    uint16_t* listings = nullptr;
    unsigned* ticket = nullptr;
};
// What the host does meanwhile: goes on, waits for the counts, or captures the call.
enum class HostIs { kFree, kWaiting, kCapturing };
// Whether the kernels below take this problem (else the general path does), and its tables,
// in `bytes` bytes at `scratch` (256-byte aligned).
bool elastic_single_tables(int T, int K, int E, int H, bool expand, HostIs host, int num_sms, void* scratch,
                           size_t bytes, unsigned* ticket, SingleTables* tables);
cudaError_t launch_elastic_single_dispatch(ElasticSingleParams p, bool expand, const SingleTables& tables,
                                           const LaunchCtx& ctx);

// float ones of a given length (the weights of the exchange's reduction)
cudaError_t launch_elastic_fill_ones(float* w, size_t n, cudaStream_t stream);

}  // namespace mcep
