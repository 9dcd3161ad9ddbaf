// Parameter blocks and launchers of the EP kernels. Host code fills a block,
// the launcher picks the grid and starts the kernel on the given stream.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include <string>

namespace mcep {

constexpr int kMaxTopk = 16;       // MCEP_MAX_TOPK
constexpr int kMaxRanks = 64;      // ranks of one group (one NVLink domain)
constexpr int kMaxExperts = 4096;  // MCEP_MAX_EXPERTS
constexpr int kTileChannels = 512; // one warp pass: 32 lanes x 16 channels
constexpr int kMetaHeaderBytes = 16;  // per-row side message: token index + padding, then scales

// Status bits the kernels may raise instead of trapping.
constexpr int kStatusSlotRange = 1;
constexpr int kStatusHardTimeout = 2;
constexpr int kStatusBadSource = 4;
constexpr int kStatusNoPeer = 8;  // a rank marked active has no mapped buffer

// What a launch costs the host depends on the size of the kernel's parameters: 1.67 us where it is
// 32 bytes beyond a multiple of 64 (32, 96, 160, 224, 288, 352), 2.0 - 2.1 for any other from 16 to
// 1024 (with programmatic serialisation; without 2.0 and 2.5). So parameter blocks are filled up to
// such a size (us per layer: one token in FP8 10.1 -> 9.8, 128 of 4 KB in bf16 9.9 -> 9.6, elastic decode
// call of 128 14.2 -> 13.8, expanded, waiting, 1024 30.1 -> 29.4). The layout kernel's are not (128 bytes): a
// synchronous layer that the host bounds would gain 0.3 us (not filled | filled: 300 tokens of 8 KB in FP8
// to 8 11.7 | 11.3, 1000 in bf16 to 2 11.5 | 11.1, from 400 to 8 on none), but the host of an asynchronous one gets
// ahead of the device and then waits for every event between the streams (300 14.9 | 18.2, 900 to 2 15.7 |
// 18.3; whoever is ahead anyway has 18.2 and 18.3 with either).
template <typename P>
constexpr bool cheap_to_launch = sizeof(P) % 64 == 32;

struct LaunchCtx {
    cudaStream_t stream;
    int num_sms;
    bool pdl;            // launch with programmatic stream serialisation
    bool chain = false;  // the same for what follows the first kernel of a call made of several
};

// ---- routing layout ---------------------------------------------------------
// The routing as bits: which tokens of a chunk chose an expert, and how many. A token's
// position among the tokens of its expert is the sum of the counts of the chunks ahead
// and of the lower bits of its own (bits_before, ep_routing.cuh).
constexpr int kChunkTokens = 128;
struct RouteBits {
    uint4* words;     // [chunks][experts], bit t % 128 of chunk t / 128; null: not there
    uint8_t* counts;  // [experts][stride], padding undefined
    int experts, chunks, stride;
};
// Such bits in `capacity` bytes at `memory` (16-byte aligned); words null where they do
// not fit or where the batch has more than 128 chunks.
RouteBits route_bits(void* memory, size_t capacity, int T, int E);

struct LayoutParams {
    const int64_t* topk_idx;  // [T][K]
    int T, K, E, R;
    RouteBits bits;           // words not null: these are written, and nothing below
    int32_t* count;           // [E]
    int32_t* slot;            // [T*K]
    int32_t* rank_count;      // [R] or null
    int32_t* expert_prefix;   // [E] or null
    unsigned* ticket;         // scratch word, required with rank_count/expert_prefix
    // single-rank groups: the layout already is the receive layout
    int32_t* recv_count;      // [E] or null
    int64_t* layout_range;    // [E] or null
    // optional scratch for the two-pass (chunked) variant: per-chunk histograms
    int32_t* chunk_hist;      // [chunk_hist_entries] or null
    size_t chunk_hist_entries;
};
cudaError_t launch_layout(const LayoutParams& p, const LaunchCtx& ctx);

// ---- single rank: packed outputs written directly ------------------------------
struct DirectDispatchParams {
    const void* x;              // [T][H] bf16
    const int64_t* topk_idx;    // [T][K]
    int T, K, E, M, H;
    int use_fp8;
    int C;                      // counting: tokens per batch (set by the launcher)
    int32_t* status;
    void* recv_x;
    float* recv_scales;
    int32_t* recv_src_info;
    int32_t* recv_count;        // [E], written without `slot`
    int64_t* layout_range;      // [E], written without `slot`
    int32_t* rowmap;            // [T*K] row of (token, k) inside its expert, kept for combine
    // Positions from the layout kernel (words null: none), or from another one; neither: they
    // are counted in the send kernel. (Last, so that what a counting kernel reads lies together.)
    RouteBits bits;
    const int32_t* slot;        // [T*K]
    bool x_last;                // see input_beyond_l2 (set by the launcher)
    int warps_per_row, tokens_per_block, parts;  // with positions: how a block's warps are dealt out, blocks that
                                                 // share a row (set by the launcher)
    bool counting() const { return slot == nullptr && bits.words == nullptr; }
};
static_assert(cheap_to_launch<DirectDispatchParams>);
// whether the send kernels count the slots themselves for this many tokens
bool counts_in_send_kernel(int T, int K, int H, int num_sms, bool group);
// Whether the input of a layer, `copies` rows of each token and the result are so many bytes that the
// last use of the experts' outputs is worth telling L2 (ld32_readonly with `last`). Of less, all of it
// stays there anyway, and what a caller uses again is not to be the first that goes (us per layer on
// three sets of inputs in turn, no mark | marked: to 1, 1500 rows of 8 KB, 37 MB, 11.3 | 11.7, 2000, 49 MB,
// 12.7 | 12.2; to 2, 1200, 39 MB, 11.9 | 12.1, 1600, 52 MB, 14.6 | 14.2).
bool layer_beyond_l2(long long T, int copies, int H);
// The same for the input. A shared expert reads it again behind dispatch: in bf16 it is marked only where
// input and rows are more than L2's 120 MiB, and it would not be found there anyway. us of a program with
// such a reader, only the outputs marked | the input too: 2096 rows of 10 KB to 2 74.1 | 75.5, 6368 of 2 KB
// to 4 67.6 | 69.1, flat elastic 3496 of 12 KB 95.8 | 97.6; beyond the line 3488 of 14 KB to 3 144.0 | 144.1,
// 4592 of 8 KB to 4 122.8 | 122.2 (without the reader 101.2 | 100.5 and 89.7 | 88.4). FP8 rows are half as
// long and the reader loses next to nothing: 2684 of 12 KB to 1 125.9 | 125.4, 1032 of 14 KB to 3 110.8 |
// 109.5, 2320 to 2 177.8 | 178.0 (with outputs made long before 2096 of 10 KB to 8 91.7 | 93.0, no mark 95.4).
bool input_beyond_l2(long long T, int copies, int H, bool fp8);
cudaError_t launch_direct_dispatch(DirectDispatchParams p, const LaunchCtx& ctx);

struct SendShape {
    int tokens, threads;  // tokens per batch, threads per block
};

// Single rank: (token, k) -> packed row, inverted from the handle.
struct CombineInvertParams {
    const int32_t* src_info;    // [L][R*M]
    const int64_t* layout_range;// [L][R]
    const int64_t* topk_idx;    // [T][K]
    int L, R, M, T, K, rank;
    int32_t* rowmap;            // scratch [T*K]
    int32_t* status;
    char fill[32];
};
static_assert(cheap_to_launch<CombineInvertParams>);
cudaError_t launch_combine_invert(const CombineInvertParams& p, const LaunchCtx& ctx);

struct DirectCombineParams {
    const int64_t* topk_idx;    // [T][K]
    const float* topk_weights;  // [T][K]
    const int32_t* active_ranks;
    int T, K, E, M, H;
    const void* x;              // rows at x + (expert * M + rowmap[t*K+k]) * 2H
    const int32_t* rowmap;
    int absolute;               // rowmap names rows of the whole tensor, which has M of them (-1: none), every
                                // weight is 1; topk_idx and topk_weights are not read
    int tokens_per_block, tiles_per_block, span;  // set by the launcher (span: tokens a block works through, < 0:
                                                  // the last ones of the batch first)
    // search: no rowmap; rows are looked up in the handle by the kernel
    int search;
    const int32_t* src_info;
    const int64_t* layout_range;
    void* combined_x;           // [T][H] bf16
    char fill[48];
};
static_assert(cheap_to_launch<DirectCombineParams>);
cudaError_t launch_direct_combine(DirectCombineParams p, const LaunchCtx& ctx);

// ---- groups: words exchanged through symmetric memory -----------------------------
// All words are 64-bit: (sequence number of the call << 32) | value, value >= 1.
// A word that does not carry the current sequence number has not arrived.
struct Words {
    // byte offsets inside every rank's symmetric allocation, for this call's parity
    size_t cnt_off;    // at the owner of an expert: [R src][L] tokens src sends to local expert
    size_t beg_off;    // at a sender: [E] first row of its segment in expert e, written by e's owner
    size_t dflag_off;  // at a receiver: [R src] all of src's dispatch rows have landed
    size_t cflag_off;  // at a token owner: [R owner] owner's expert outputs can be read
};

struct WaitCfg {
    int32_t* active_ranks;     // read and written (timeout -> 0)
    int64_t timeout_ns;        // < 0: only the hard bound applies
    int64_t hard_timeout_ns;
    int32_t* status;
};

// Dispatch in a group. Block 0 is the control block: it publishes this rank's
// per-expert counts to the experts' owners, collects the counts all sources
// announce for its own experts, fixes the receive layout and answers every
// source with the first row of its segment. The other blocks send token rows
// straight to their final place in the owners' packed receive area.
struct GroupDispatchParams {
    const void* x;              // [T][H] bf16
    const int64_t* topk_idx;    // [T][K]
    const int32_t* slot;        // [T*K] and
    const int32_t* count;       // [E] from a layout kernel, or null: `bits`, or counted in the send kernel
    void* const* peer_base;     // [R] base of every rank's symmetric buffer
    char* local_base;           // this rank's
    int T, K, E, R, M, H, rank;
    int use_fp8;
    int C;                      // tokens per batch (set by the launcher)
    Words w;
    size_t rx_off;              // packed receive rows [L][R*M][row_bytes] of this parity
    size_t meta_off;            // side messages [L][R*M][meta_stride] of this parity
    int row_bytes, meta_stride;
    uint32_t seq;
    const uint32_t* seq_ptr;    // graph mode: the call's sequence number lives in device memory (else null)
    WaitCfg wait;
    // scratch in the local workspace (per parity)
    uint64_t* res_cnt;          // [L*R] the control block's verdict per (expert, source)
    uint64_t* res_dflag;        // [R] verdict words of the payload flags
    unsigned* ticket;           // sender blocks that have finished
    int32_t* rowmap;            // [T*K] row of (token, k) at its expert's owner, kept for combine
    // outputs (caller's tensors)
    void* recv_x;               // == local_base + rx_off when the caller took the in-place tensor
    float* recv_scales;
    int32_t* recv_src_info;
    int32_t* recv_count;        // [L]
    int64_t* layout_range;      // [L][R]
    int copy_rows;              // recv_x is a tensor of the caller's: copy the rows out
    RouteBits bits;             // from the layout kernel (words null: none)
    bool x_last;                // see input_beyond_l2 (set by the launcher)
    bool counting() const { return slot == nullptr && bits.words == nullptr; }
    char fill[40];
};
static_assert(cheap_to_launch<GroupDispatchParams>);
bool group_call_can_be_one_kernel(int T, int K, int E, int num_sms);
// one launch: control + send + receive duties
cudaError_t launch_group_dispatch(GroupDispatchParams p, const LaunchCtx& ctx);
// two launches (hook mode, large batches, caller-owned recv_x)
cudaError_t launch_group_dispatch_send(GroupDispatchParams p, const LaunchCtx& ctx);
cudaError_t launch_group_dispatch_recv(const GroupDispatchParams& p, const LaunchCtx& ctx);

// Combine in a group: expert outputs are made readable in symmetric memory
// (copied there, or written there by the caller: zero copy), every peer is told
// so with one word, and token owners read their rows straight from the experts'
// owners and reduce them.
struct GroupCombineParams {
    const void* x;              // [L][R*M][H] bf16 expert outputs (ignored with zero_copy)
    const int64_t* layout_range;// [L][R] from the handle
    const int64_t* topk_idx;    // [T][K]
    const float* topk_weights;  // [T][K]
    const int32_t* rowmap;      // [T*K] left by the dispatch call of this handle
    void* const* peer_base;
    char* local_base;
    int T, K, E, R, M, H, rank;
    int zero_copy;
    Words w;
    size_t cin_off;             // combine input [L][R*M][H] bf16 of this parity
    uint32_t seq;
    const uint32_t* seq_ptr;    // graph mode (see GroupDispatchParams)
    WaitCfg wait;
    uint64_t* res_cflag;        // [R]
    unsigned* ticket;
    void* combined_x;           // [T][H] bf16
    int behind_publish;         // the reduce phase directly follows the publish phase of its call (no hook)
    int tokens_per_block, tiles_per_block, span;  // set by the launcher (reduce phase of large batches)
    char fill[8];
};
static_assert(cheap_to_launch<GroupCombineParams>);
cudaError_t launch_group_combine(const GroupCombineParams& p, const LaunchCtx& ctx);
cudaError_t launch_group_combine_publish(const GroupCombineParams& p, const LaunchCtx& ctx);
cudaError_t launch_group_combine_reduce(GroupCombineParams p, const LaunchCtx& ctx);

// In-process groups (several logical ranks on one GPU, tests): the send phase
// (phases = 1) or the whole call (phases = 3) of `n` ranks as ONE cooperative
// launch, because kernels that wait for one another must not be separate
// launches on one GPU. `dev_params` is device memory for `n` parameter blocks.
// All ranks must agree on payload type and hidden size.
cudaError_t launch_group_dispatch_multi(GroupDispatchParams* params, int n,
                                        GroupDispatchParams* dev_params, int phases,
                                        const LaunchCtx& ctx);
cudaError_t launch_group_combine_multi(const GroupCombineParams* params, int n,
                                       GroupCombineParams* dev_params, const LaunchCtx& ctx);

// A barrier of the group on the device: every rank writes one word to every
// active peer and waits for theirs; the ranks leave within about one NVLink
// latency of each other. `bar_off` = [R] u64 words in symmetric memory,
// `epoch` = the number of this barrier (all ranks count alike).
struct BarrierParams {
    void* const* peer_base;
    char* local_base;
    const int32_t* active_ranks;  // [R] or null (all active)
    size_t bar_off;
    int rank, R;
    uint32_t epoch;
    int64_t hard_timeout_ns;
    int32_t* status;
    char fill[32];
};
static_assert(cheap_to_launch<BarrierParams>);
cudaError_t launch_barrier(const BarrierParams& p, const LaunchCtx& ctx);

// Graph mode: after the last kernel of a call, the word that holds the next
// sequence number of that call's parity moves on by two.
cudaError_t launch_advance_seq(uint32_t* word, const LaunchCtx& ctx);

uint64_t kernel_launch_count();
// Brackets a launch made outside ep_kernels.cu so that it is counted - and, when
// per-kernel timing is on, timed - like the launches made there.
class LaunchScope {
public:
    LaunchScope(const char* name, cudaStream_t stream);
    cudaError_t done(cudaError_t err);  // pass cudaGetLastError() of the launch

private:
    const char* name_;
    cudaStream_t stream_;
    cudaEvent_t a_ = nullptr, b_ = nullptr;
};
// Per-kernel device times: switch on, run, then drain "name launches total_ms" lines.
void set_kernel_timing(bool on);
std::string drain_kernel_times();

}  // namespace mcep
