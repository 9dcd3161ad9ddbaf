// Kernels of the elastic-style calls: see ep_elastic.cuh. None of them waits for
// another GPU; the exchange between the ranks is the group dispatch / combine.
#include "ep_elastic.cuh"

#include <type_traits>

#include "ep_device.cuh"
#include "ep_kernels.cuh"
#include "ep_launch.cuh"
#include "ep_routing.cuh"

namespace mcep {
namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

__device__ __forceinline__ int rows_received(const int64_t* layout_range, int R, int* s_begin,
                                             int* s_end) {
    // (begin << 32) | count per source rank; the rows of all sources are [0, n)
    __shared__ int s_n;
    for (int r = threadIdx.x; r < R; r += blockDim.x) {
        const int64_t v = layout_range[r];
        const int begin = (int)(v >> 32), cnt = (int)(v & 0xffffffffll);
        if (s_begin) s_begin[r] = begin;
        if (s_end) s_end[r] = begin + cnt;
    }
    if (threadIdx.x < 32) {
        int n = 0;
        for (int r = threadIdx.x; r < R; r += 32) {
            const int64_t v = layout_range[r];
            n = max(n, (int)(v >> 32) + (int)(v & 0xffffffffll));
        }
        for (int d = 16; d > 0; d >>= 1) n = max(n, __shfl_xor_sync(kAll, n, d));
        if (threadIdx.x == 0) s_n = n;
    }
    __syncthreads();
    return s_n;
}

// Block-wide exclusive position of the threads whose `flag` is set, continuing
// from the positions earlier rounds handed out. All threads of the block call it.
__device__ __forceinline__ int block_position(bool flag, int* s_warp, int* s_base) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned bal = __ballot_sync(kAll, flag);
    if (lane == 0) s_warp[warp] = __popc(bal);
    __syncthreads();
    int before = *s_base;
    for (int i = 0; i < warp; ++i) before += s_warp[i];
    const int pos = before + __popc(bal & ((1u << lane) - 1u));
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int i = 0; i < kWarps; ++i) s += s_warp[i];
        *s_base += s;
    }
    __syncthreads();
    return pos;
}

// One block per destination rank r and 256 tokens: which tokens go to r, at which lane of their
// top-k list (the last one that names an expert of r, as `deduplicate` of
// mooncake_ep_elastic_ptx.cuh:690-693 elects), and in which position (token
// order, as the deterministic prologue of the reference assigns them:
// mooncake_ep_elastic_dispatch_deterministic_prologue.cuh:134-166). The block
// also stores, in rank r's memory, the record of every row r is about to get.
__global__ void __launch_bounds__(kThreads) ep_elastic_route_kernel(ElasticRouteParams p) {
    const int r = blockIdx.x;                 // destination rank
    const int first = blockIdx.y * kThreads;  // this block's 256 tokens
    const int L = p.E / p.R;
    pdl_launch_dependents();  // the exchange's first kernel may take its place; it waits for this one at its top
    __shared__ int s_warp[kWarps];
    __shared__ int s_base;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    {
        // tokens of the earlier blocks that go to rank r: counted again here (the index matrix
        // sits in L2) rather than waited for, so no block of this kernel depends on another
        int before = 0;
        for (int t = threadIdx.x; t < first; t += kThreads) {
            bool hit = false;
#pragma unroll
            for (int k = 0; k < kMaxTopk; ++k) {
                if (k >= p.K) break;
                const int64_t e = ld_ro(p.topk_idx + (size_t)t * p.K + k);
                hit = hit || (e >= 0 && e < p.E && (int)e / L == r);
            }
            before += hit ? 1 : 0;
        }
        for (int d = 16; d > 0; d >>= 1) before += __shfl_xor_sync(kAll, before, d);
        if (lane == 0) s_warp[warp] = before;
        __syncthreads();
        if (threadIdx.x == 0) {
            int sum = 0;
            for (int i = 0; i < kWarps; ++i) sum += s_warp[i];
            s_base = sum;
        }
        __syncthreads();
    }
    {
        const int t = first + threadIdx.x;
        // the token's choices, all loaded before anything is stored
        int64_t raw[kMaxTopk];
        int rk[kMaxTopk];
        int master = -1;
        if (t < p.T) {
#pragma unroll
            for (int k = 0; k < kMaxTopk; ++k) raw[k] = k < p.K ? ld_ro(p.topk_idx + (size_t)t * p.K + k) : -1;
#pragma unroll
            for (int k = 0; k < kMaxTopk; ++k) {
                rk[k] = (raw[k] >= 0 && raw[k] < p.E) ? (int)raw[k] / L : -1;
                if (rk[k] == r) master = k;
            }
        }
        const int slot = block_position(master >= 0, s_warp, &s_base);
        if (t >= p.T) return;
#pragma unroll
        for (int k = 0; k < kMaxTopk; ++k) {
            if (k >= p.K) break;
            const size_t at = (size_t)t * p.K + k;
            if (rk[k] == r) {
                p.rank_topk[at] = (k == master) ? r : -1;
                p.dst_slot[at] = (k == master) ? p.rank * p.M + slot : -1;
            } else if (rk[k] < 0 && r == 0) {
                p.rank_topk[at] = -1;
                p.dst_slot[at] = -1;
            }
        }
        // what the receiver needs to know about the row, stored where it will look for it:
        // in rank r's memory, at this rank's region, at the row's position
        char* base = static_cast<char*>(p.record_base[r]);
        if (master >= 0 && base != nullptr) {
            char* rec = base + ((size_t)p.rank * p.M + slot) * p.record_stride;
#pragma unroll
            for (int k = 0; k < kMaxTopk; ++k) {
                if (k >= p.K) break;
                reinterpret_cast<int32_t*>(rec)[k] = rk[k] >= 0 ? (int32_t)raw[k] : -1;
                reinterpret_cast<float*>(rec)[p.K + k] =
                    p.topk_weights ? ld_ro(p.topk_weights + (size_t)t * p.K + k) : 0.f;
            }
            reinterpret_cast<int32_t*>(rec)[2 * p.K] = t;
        }
        if (r != 0 || p.copied_topk_idx == nullptr) return;
#pragma unroll
        for (int k = 0; k < kMaxTopk; ++k) {
            if (k >= p.K) break;
            p.copied_topk_idx[(size_t)t * p.K + k] = raw[k];
        }
    }
}

// Receiver side, after the exchange: per received row the record its source
// stored here is turned into the row's local expert choices,
// weights and source metadata (mooncake_ep_elastic_dispatch_copy_epilogue.cuh:
// 114-132, 212-248); the last block to finish turns the per-expert hit counts
// into the aligned exclusive prefix sum of
// mooncake_ep_elastic_dispatch_official.cuh:255-310.
__global__ void __launch_bounds__(kThreads) ep_elastic_epilogue_kernel(ElasticEpilogueParams p) {
    __shared__ int s_begin[kMaxRanks], s_end[kMaxRanks];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    pdl_wait();  // the exchange's kernels wrote the layout
    const int n = rows_received(p.layout_range, p.R, s_begin, s_end);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        int run = 0;
        for (int r = 0; r < p.R; ++r) {
            run += s_end[r] - s_begin[r];
            p.psum_rank[r] = run;
        }
    }
    const int lo = p.rank * p.L;
    const int md_stride = p.K + 2;
    for (int i = blockIdx.x * kWarps + warp; i < n; i += gridDim.x * kWarps) {
        int src = -1;
        for (int r0 = 0; r0 < p.R && src < 0; r0 += 32) {
            const int r = r0 + lane;
            const unsigned b = __ballot_sync(kAll, r < p.R && i >= s_begin[r] && i < s_end[r]);
            if (b) src = r0 + __ffs(b) - 1;
        }
        if (src < 0) continue;
        // the record the source stored for its (i - begin)-th row, in this rank's memory
        const char* rec = p.records + ((size_t)src * p.M + (i - s_begin[src])) * p.record_stride;
        int e = -1;
        float w = 0.f;
        if (lane < p.K) {
            e = ld_s32_coherent(rec + 4 * lane);
            w = ld_f32_coherent(rec + 4 * (p.K + lane));
        }
        const int tok = ld_s32_coherent(rec + 8 * p.K);
        if (tok < 0 || tok >= p.M) {
            if (lane == 0) atomicOr(p.status, kStatusBadSource);
            continue;
        }
        const int local = (e >= lo && e < lo + p.L) ? e - lo : -1;
        const unsigned hit = __ballot_sync(kAll, local >= 0);
        const int master = hit ? 31 - __clz(hit) : 0;
        if (lane < p.K) {
            p.recv_topk_idx[(size_t)i * p.K + lane] = local;
            if (p.recv_topk_weights) p.recv_topk_weights[(size_t)i * p.K + lane] = w;
            if (local >= 0) atomicAdd(p.hist + local, 1);
            if (p.expand) p.recv_src_metadata[(size_t)i * md_stride + 2 + lane] = -1;
        }
        if (lane == 0) {
            p.recv_src_metadata[(size_t)i * md_stride] = src * p.M + tok;
            p.recv_src_metadata[(size_t)i * md_stride + 1] = src * p.K + master;
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(p.ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (warp == 0) {
        int run = 0;
        for (int e0 = 0; e0 < p.L + 1; e0 += 32) {
            const int e = e0 + lane;
            // entry e of the exclusive sum adds the aligned count of expert e - 1
            int c = 0;
            if (e >= 1 && e <= p.L) {
                c = ld_l2(p.hist + e - 1);
                c = (c + p.alignment - 1) / p.alignment * p.alignment;
            }
            int v = c;
            for (int d = 1; d < 32; d <<= 1) {
                const int u = __shfl_up_sync(kAll, v, d);
                if (lane >= d) v += u;
            }
            if (e <= p.L) {
                p.psum_expert[e] = run + v;
                if (p.psum_start) p.psum_start[e] = run + v;
            }
            run += __shfl_sync(kAll, v, 31);
        }
        __syncwarp();
        for (int e = lane; e < p.L; e += 32) p.hist[e] = 0;
        if (lane == 0) *p.ticket = 0;
    }
}

// Expanded layout: one block per local expert numbers the rows that chose it, in
// receive order (the reference hands the positions out with an atomic, in
// arrival order: mooncake_ep_elastic_dispatch_copy_epilogue.cuh:138-141).
__global__ void __launch_bounds__(kThreads) ep_elastic_expand_scan_kernel(ElasticExpandParams p) {
    const int e = blockIdx.x;
    __shared__ int s_warp[kWarps];
    __shared__ int s_base;
    const int n = rows_received(p.layout_range, p.R, nullptr, nullptr);
    if (threadIdx.x == 0) s_base = 0;
    __syncthreads();
    const int start = p.psum_start[e];
    const int md_stride = p.K + 2;
    for (int i0 = 0; i0 < n; i0 += kThreads) {
        const int i = i0 + threadIdx.x;
        int k_hit = -1;
        if (i < n)
            for (int k = 0; k < p.K; ++k)
                if (p.recv_topk_idx[(size_t)i * p.K + k] == e) k_hit = k;
        const int pos = block_position(k_hit >= 0, s_warp, &s_base);
        if (k_hit >= 0 && start + pos < p.max_rows)
            p.recv_src_metadata[(size_t)i * md_stride + 2 + k_hit] = start + pos;
        else if (k_hit >= 0)  // (the entry stays -1: dropped)
            atomicOr(p.status, kStatusSlotRange);
    }
    if (threadIdx.x == 0) p.psum_expert[e] = start + s_base;
}

__device__ __forceinline__ void copy_row(void* dst, const void* src, int row_bytes, int lane) {
    for (int c = lane * 32; c < row_bytes; c += 32 * 32)
        st32(static_cast<char*>(dst) + c, ld32_coherent(static_cast<const char*>(src) + c));
}

__global__ void __launch_bounds__(kThreads) ep_elastic_expand_copy_kernel(ElasticExpandParams p) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = rows_received(p.layout_range, p.R, nullptr, nullptr);
    const int md_stride = p.K + 2;
    for (int i = blockIdx.x * kWarps + warp; i < n; i += gridDim.x * kWarps) {
        const int slot = lane < p.K ? p.recv_src_metadata[(size_t)i * md_stride + 2 + lane] : -1;
        unsigned todo = __ballot_sync(kAll, slot >= 0);
        const char* src = static_cast<const char*>(p.flat_x) + (size_t)i * p.row_bytes;
        while (todo) {
            const int k = __ffs(todo) - 1;
            todo &= todo - 1;
            const int dst = __shfl_sync(kAll, slot, k);
            copy_row(static_cast<char*>(p.recv_x) + (size_t)dst * p.row_bytes, src, p.row_bytes, lane);
            if (p.recv_topk_weights && lane == 0)
                p.recv_topk_weights[dst] = p.flat_weights[(size_t)i * p.K + k];
        }
    }
}

// mooncake_ep_elastic_combine_official.cuh:146-216 with multiple reduction: one
// row is copied; two rows are added as the reference's bf16 add does (the exact
// sum rounded once, which an fp32 add followed by the bf16 rounding also gives);
// more are accumulated in fp32 from zero in listing order and rounded once.
__global__ void __launch_bounds__(kThreads) ep_elastic_local_reduce_kernel(ElasticLocalReduceParams p) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n = rows_received(p.layout_range, p.R, nullptr, nullptr);
    const int md_stride = p.K + 2;
    const int row_bytes = p.H * 2;
    for (int i = blockIdx.x * kWarps + warp; i < n; i += gridDim.x * kWarps) {
        const int slot = lane < p.K ? p.recv_src_metadata[(size_t)i * md_stride + 2 + lane] : -1;
        const unsigned valid = __ballot_sync(kAll, slot >= 0 && slot < p.x_rows);
        const int cnt = __popc(valid);
        char* dst = static_cast<char*>(p.y) + (size_t)i * row_bytes;
        if (cnt == 0) {
            for (int c = lane * 32; c < row_bytes; c += 32 * 32) st32(dst + c, V32{});
            continue;
        }
        if (cnt == 1) {
            const int s = __shfl_sync(kAll, slot, __ffs(valid) - 1);
            for (int c = lane * 32; c < row_bytes; c += 32 * 32)
                st32(dst + c, ld32_readonly(static_cast<const char*>(p.x) + (size_t)s * row_bytes + c));
            continue;
        }
        // the rows to add, in listing order (gathered before the lanes' loops part ways)
        int rows[kMaxTopk];
        {
            unsigned todo = valid;
#pragma unroll
            for (int j = 0; j < kMaxTopk; ++j) {
                const int k = todo ? __ffs(todo) - 1 : 0;
                const int s = __shfl_sync(kAll, slot, k);
                rows[j] = todo ? s : -1;
                todo &= todo - 1;
            }
        }
        for (int c = lane * 32; c < row_bytes; c += 32 * 32) {
            float acc[16];
#pragma unroll
            for (int j = 0; j < 16; ++j) acc[j] = 0.f;
#pragma unroll
            for (int m = 0; m < kMaxTopk; ++m) {
                if (m >= cnt) break;
                const V32 v = ld32_readonly(static_cast<const char*>(p.x) + (size_t)rows[m] * row_bytes + c);
                // two rows: a + b, not 0 + a + b (the sign of a zero sum differs)
                const bool first = m == 0 && cnt == 2;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    acc[2 * j] = first ? bf16lo(v.w[j]) : __fadd_rn(acc[2 * j], bf16lo(v.w[j]));
                    acc[2 * j + 1] = first ? bf16hi(v.w[j]) : __fadd_rn(acc[2 * j + 1], bf16hi(v.w[j]));
                }
            }
            st32(dst + c, pack_bf16x16(acc));
        }
    }
}

// ---- a single rank ----------------------------------------------------------------------
__device__ __forceinline__ int aligned_count(int c, int a) { return (c + a - 1) / a * a; }

// An expanded row, or -1 where aligned segments reach beyond the caller's tensors: the row
// is dropped, in the copy, in the metadata and in the rows that combine gathers.
__device__ __forceinline__ int row_with_room(const ElasticSingleParams& p, int row) {
    if (row < p.max_rows) return row;
    atomicOr(p.status, kStatusSlotRange);
    return -1;
}

// In-place exclusive sums of a[0..n), the total in a[n] (shared memory, whole block).
__device__ void exclusive_sums(int* a, int n) {
    __shared__ int s_sum[32];
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int per = n <= nthr ? 1 : (n + nthr - 1) / nthr, b = min(tid * per, n), e = min(b + per, n);
    int sum = 0;
    for (int i = b; i < e; ++i) sum += a[i];
    auto scan = [&](int v) {
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(kAll, v, d);
            if (lane >= d) v += u;
        }
        return v;
    };
    const int incl = scan(sum);
    if (lane == 31) s_sum[warp] = incl;
    __syncthreads();
    // every warp scans the warps' sums for itself: no further barrier for them
    const int mine = lane < nwarps ? s_sum[lane] : 0, warps = scan(mine);
    int run = __shfl_sync(kAll, warps - mine, warp) + incl - sum;
    for (int i = b; i < e; ++i) {
        const int c = a[i];
        a[i] = run;
        run += c;
    }
    if (tid == nthr - 1) a[n] = run;
    __syncthreads();
}

// What a caller may be waiting for on the host, then the flag that says so. One block
// of the copy kernel does it, so that no kernel's completion waits for the bus.
__device__ void tell_host(const ElasticSingleParams& p) {
    if (p.host_counts == nullptr) return;
    volatile int32_t* h = p.host_counts;
    for (int i0 = threadIdx.x; i0 <= p.E; i0 += 4 * blockDim.x) {
        int v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = __ldcg(p.psum_expert + min(i0 + u * (int)blockDim.x, p.E));
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (i0 + u * (int)blockDim.x <= p.E) h[2 + i0 + u * blockDim.x] = v[u];
    }
    if (threadIdx.x == 0) h[1] = ld_l2(p.psum_rank);
    __threadfence_system();
    __syncthreads();
    if (threadIdx.x == 0) h[0] = p.host_seq;
}

// The layout as bits (RouteBits), a block per 128 tokens, as ep_layout_bits_kernel. Row 0 of
// the table stands for "the token goes anywhere", from which its received row is found; rows
// 1 + e (kExpand) are the experts'. The experts' hits are listings: an expert listed twice
// counts twice in them and has its row at the last listing
// (mooncake_ep_elastic_dispatch_copy_epilogue.cuh:114-141). Every block adds its own to the
// totals, so that whoever needs them reads one word per expert, however many chunks there
// are. (One block that reads every chunk's hits, a load after the other, is what the call waits
// for: the layer, 4826 rows of 11 KB expanded to 1 of 128 experts 44.7 us, now 43.0; 4364 of 5 KB
// to 1 of 2048 63.1, now 33.8; flat, 10904 of 9 KB to 2 of 1024 81.2, now 66.9.)
// An expanded row's place depends on the hits of all experts below its own: the block that
// finishes last makes the segments of them (kExpand). For flat rows they are results only, and
// a block of the copy kernel does it, so that no row waits.
constexpr int kBitsThreads = 256;

template <bool kExpand, int KB>
__device__ __forceinline__ void single_bits(const ElasticSingleParams& p, uint32_t* mask, int* extra) {
    const int t = blockIdx.x * kChunkTokens + threadIdx.x, lane = threadIdx.x & 31, word = threadIdx.x >> 5;
    if (threadIdx.x >= kChunkTokens) return;
    int e[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) e[k] = -1;
    if (t < p.T) load_choices<KB, true>(p.topk_idx, t, p.K, p.E, choices_in_pairs(p.topk_idx, p.K), e);
    bool any = false;
#pragma unroll
    for (int k = 0; k < KB; ++k) any |= e[k] >= 0;
    const unsigned sent = __ballot_sync(kAll, any);
    if (lane == 0) mask[word] = sent;
    int all[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) all[k] = e[k];
    if (kExpand) drop_repeats<KB, true>(e);
#pragma unroll
    for (int k = 0; k < KB; ++k) {
        if (kExpand && e[k] >= 0) atomicOr(&mask[(1 + e[k]) * 4 + word], 1u << lane);
        if (all[k] >= 0 && (!kExpand || e[k] < 0)) atomicAdd(&extra[all[k]], 1);
    }
}

// The totals: listings in the low half of a word, rows (tokens, repeats left out) in the high.
__device__ __forceinline__ void add_hits(const ElasticSingleParams& p, int e, int listings, int rows) {
    if (listings) atomicAdd(p.totals + e, (unsigned long long)(unsigned)rows << 32 | (unsigned)listings);
}

// use(expert, listings, rows) for every expert's total, which is zero afterwards; whole block,
// four words per thread requested together.
template <typename Use>
__device__ __forceinline__ void take_totals(const ElasticSingleParams& p, Use use) {
    const int nthr = blockDim.x;
    for (int x0 = threadIdx.x; x0 < p.E; x0 += 4 * nthr) {
        unsigned long long v[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) v[u] = x0 + u * nthr < p.E ? __ldcg(p.totals + x0 + u * nthr) : 0ull;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int x = x0 + u * nthr;
            if (x >= p.E) break;
            p.totals[x] = 0ull;
            use(x, (int)(unsigned)v[u], (int)(v[u] >> 32));
        }
    }
}

// ---- segments made by every block of the copy kernel -----------------------------------
// Up to 16 chunks and 256 experts the layout kernel leaves its listings as they are, a word per
// expert and chunk, and every block of the copy kernel sums up those of all experts. What the block
// that finishes last does else - a fence, the ticket, the totals, the sums and the segments, five
// round trips to L2 one after the other - stands ahead of every row; here one load and a scan do, with
// 4 KB more for a block to read, which on larger tables costs what it saves. Device us per layer, that
// block's segments | their own: 1024 rows of 8 KB to 8 of 128 27.0 | 25.0, to 2 of 64 14.7 | 12.6; 2048 of 14 KB to 8
// of 256 83.8 | 82.1, to 1 of 8 24.2 | 22.6.
// It must not spill: with the first listings asked for ahead of the bits in registers, 50 bytes
// a thread, 1024 of 8 KB to 8 25.7, 2048 of 14 KB 84.3; by cp.async 25.1 and 91.0.
constexpr int kOwnChunks = 16, kOwnExperts = 256;
constexpr int kElasticWarps = 4, kElasticTiles = 2;  // of the copy kernel: see there

// [E][chunks, a multiple of 8] words, the ones of chunks that there are not are zero.
__host__ __device__ constexpr int listings_stride_of(int chunks) { return (chunks + 7) / 8 * 8; }
__device__ __forceinline__ void leave_listings(const ElasticSingleParams& p, int e, int listings) {
    const int stride = listings_stride_of(gridDim.x);
    uint16_t* row = p.listings + (size_t)e * stride;
    row[blockIdx.x] = (uint16_t)listings;
    if (blockIdx.x == gridDim.x - 1)
        for (int c = gridDim.x; c < stride; ++c) row[c] = 0;
}
__device__ __forceinline__ int sum_words(const uint4& v) {
    const uint32_t s = (v.x & 0xffffu) + (v.y & 0xffffu) + (v.z & 0xffffu) + (v.w & 0xffffu);
    return (int)(s + (v.x >> 16) + (v.y >> 16) + (v.z >> 16) + (v.w >> 16));
}
// Where the segments start: a thread has `per` experts, whose sums lie in three parts (inside a
// thread's experts, a warp's threads, the block's warps). The block
// meets once, in `make`.
struct OwnSegments {
    struct Shared {
        int expert[kOwnExperts], thread[kElasticWarps * 32], warp[kElasticWarps];
    };
    Shared& s;
    const int per, first;

    __device__ __forceinline__ static const uint4* row(const ElasticSingleParams& p, int e) {
        return reinterpret_cast<const uint4*>(p.listings + e * listings_stride_of(p.bits.chunks));
    }
    __device__ __forceinline__ OwnSegments(const ElasticSingleParams& p, Shared& shared)
        : s(shared), per((p.E + blockDim.x - 1) / blockDim.x), first(threadIdx.x * per) {}
    __device__ __forceinline__ void make(const ElasticSingleParams& p) {
        const int lane = threadIdx.x & 31;
        int sum = 0;
        for (int x = first; x < min(first + per, p.E); ++x) {
            int n = sum_words(ld_ro(row(p, x)));
            if (p.bits.chunks > 8) n += sum_words(ld_ro(row(p, x) + 1));
            s.expert[x] = sum;
            sum += p.alignment == 1 ? n : aligned_count(n, p.alignment);
        }
        int incl = sum;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int u = __shfl_up_sync(kAll, incl, d);
            if (lane >= d) incl += u;
        }
        s.thread[threadIdx.x] = incl - sum;
        if (lane == 31) s.warp[threadIdx.x >> 5] = incl;
        __syncthreads();
    }
    __device__ __forceinline__ static int start(const Shared& s, int per, int e) {
        const int thread = per == 1 ? e : e / per;
        int n = s.expert[e] + s.thread[thread];
        for (int w = 0; w < thread >> 5; ++w) n += s.warp[w];
        return n;
    }
};

// The segments' ends; whole block. Not inlined: its registers are not taken from the rows' warps.
__device__ __noinline__ void write_segments(const OwnSegments::Shared& s, int per, RouteBits bits, int E,
                                            int32_t* psum_expert, int32_t* psum_rank) {
    for (int x = threadIdx.x; x < E; x += blockDim.x)
        psum_expert[x] = OwnSegments::start(s, per, x) + bits_total(bits, 1 + x);
    if (threadIdx.x != 0) return;
    int n = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) n += s.warp[w];
    psum_expert[E] = n;
    psum_rank[0] = bits_total(bits, 0);
}


template <bool kExpand>
__global__ void __launch_bounds__(kBitsThreads) ep_elastic_bits_kernel(ElasticSingleParams p) {
    extern __shared__ uint4 smem_u128[];  // [1 or 1 + E] bits of this chunk, then [E + 1] listings beyond them
    __shared__ bool s_last;
    const int tid = threadIdx.x, rows = kExpand ? 1 + p.E : 1;
    int* extra = reinterpret_cast<int*>(smem_u128 + rows);
    for (int i = tid; i < rows; i += kBitsThreads) smem_u128[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int i = tid; i <= p.E; i += kBitsThreads) extra[i] = 0;
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    uint32_t* mask = reinterpret_cast<uint32_t*>(smem_u128);
    if (p.K <= 4)
        single_bits<kExpand, 4>(p, mask, extra);
    else if (p.K <= 8)
        single_bits<kExpand, 8>(p, mask, extra);
    else
        single_bits<kExpand, 16>(p, mask, extra);
    __syncthreads();
    for (int x = tid; x < rows; x += kBitsThreads) {
        const uint4 m = smem_u128[x];
        const int n = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
        p.bits.words[(size_t)blockIdx.x * p.bits.experts + x] = m;
        p.bits.counts[(size_t)x * p.bits.stride + blockIdx.x] = (uint8_t)n;
        if (!kExpand || x == 0) continue;
        if (p.own_segments)
            leave_listings(p, x - 1, n + extra[x - 1]);
        else
            add_hits(p, x - 1, n + extra[x - 1], n);
    }
    if (!kExpand) {
        for (int x = tid; x < p.E; x += kBitsThreads) add_hits(p, x, extra[x], 0);
        return;
    }
    if (p.own_segments) return;  // the copy kernel makes the segments
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicInc(p.ticket, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    int* with_row = reinterpret_cast<int*>(smem_u128);  // [E] (the bits are not needed any more)
    take_totals(p, [&](int x, int listings, int rows) {
        extra[x] = aligned_count(listings, p.alignment);
        with_row[x] = rows;
    });
    __syncthreads();
    exclusive_sums(extra, p.E);  // where every expert's segment starts
    for (int x = tid; x <= p.E; x += kBitsThreads) {
        p.starts[x] = extra[x];
        p.psum_expert[x] = extra[x] + (x < p.E ? with_row[x] : 0);  // where it ends
    }
    if (tid == 0) p.psum_rank[0] = bits_total<true>(p.bits, 0);
}

// Whether any of the `n` entries from `q` on names an expert; n <= 8, requested together.
__device__ __forceinline__ bool names_any(const int64_t* q, int n, int E, bool vec) {
    bool any = false;
    if (vec) {
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
            longlong2 v = make_longlong2(-1, -1);
            if (k < n) v = ld_ro(reinterpret_cast<const longlong2*>(q + k));
            any |= (uint64_t)v.x < (uint64_t)E || (uint64_t)v.y < (uint64_t)E;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int64_t v = k < n ? ld_ro(q + k) : -1;
            any |= (uint64_t)v < (uint64_t)E;
        }
    }
    return any;
}

// Tokens of [0, upto) that name any expert; whole block, once per kernel, with a barrier.
__device__ __forceinline__ int sent_before(const ElasticSingleParams& p, int upto) {
    __shared__ int s_sent[32];
    const bool vec = choices_in_pairs(p.topk_idx, p.K);
    int n = 0;
    for (int t = threadIdx.x; t < upto; t += blockDim.x) {
        const int64_t* q = p.topk_idx + (size_t)t * p.K;
        n += names_any(q, min(p.K, 8), p.E, vec) || (p.K > 8 && names_any(q + 8, p.K - 8, p.E, vec));
    }
    if (upto <= (int)blockDim.x) return __syncthreads_count(n);  // one pass (128 tokens: 0.3 us less)
    n = __reduce_add_sync(kAll, n);
    if ((threadIdx.x & 31) == 0) s_sent[threadIdx.x >> 5] = n;
    __syncthreads();
    n = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) n += s_sent[w];
    return n;
}

// Every listing of tokens [0, T), repeats included, into hits[E] (whole block, no barrier).
__device__ __forceinline__ void count_hits(const ElasticSingleParams& p, int* hits) {
    for (int i = threadIdx.x; i < p.T * p.K; i += blockDim.x) {
        const int e = all_bits(ld_ro(p.topk_idx + i));
        if (e >= 0 && e < p.E) atomicAdd(&hits[e], 1);
    }
}

// Small batches, without a layout kernel: rows and per-entry outputs. A block takes C
// tokens (kExpand: one), finds their places itself and copies the rows, up to four of a
// batch per warp requested before the first is stored; block 0 writes the counts.
template <bool kExpand>
__global__ void __launch_bounds__(512, 2) ep_elastic_single_copy_kernel(ElasticSingleParams p) {
    extern __shared__ int smem_i32[];  // [E + 1] hits / starts, [E] earlier tokens (kExpand)
    constexpr int kEntries = 128;
    __shared__ int s_exp[kEntries];  // expert of the entry or -1
    __shared__ int s_row[kEntries];  // expanded row of the entry or -1 (kExpand)
    __shared__ int s_pos[kEntries];  // received row of token c
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int K = p.K, nchunks = p.H / 16, ntiles = (p.H + kTileChannels - 1) / kTileChannels;
    // (only where something is counted, and sent_before has a barrier ahead of that; cleared in every
    // block and with a barrier of their own, a dispatch of 3 to 54 tokens in a captured graph, where
    // nothing hides it, took 3.1 us instead of 2.9)
    if (kExpand || blockIdx.x == 0)
        for (int i = tid; i < (kExpand ? 2 * p.E + 1 : p.E + 1); i += nthr) smem_i32[i] = 0;
    pdl_wait();
    pdl_launch_dependents();
    if (blockIdx.x == 0) {  // the counts
        int* rows = smem_i32 + p.E + 1;
        const int n = sent_before(p, p.T);
        count_hits(p, smem_i32);
        if (kExpand) count_tokens<1, true>(p.topk_idx, 0, p.T, K, p.E, choices_in_pairs(p.topk_idx, K), rows);
        __syncthreads();
        for (int i = tid; i < p.E; i += nthr) smem_i32[i] = aligned_count(smem_i32[i], p.alignment);
        __syncthreads();
        exclusive_sums(smem_i32, p.E);
        for (int i = tid; i <= p.E; i += nthr)
            p.psum_expert[i] = smem_i32[i] + (kExpand && i < p.E ? rows[i] : 0);
        if (tid == 0) p.psum_rank[0] = n;
        __syncthreads();
        tell_host(p);
        return;
    }
    const int bid = blockIdx.x - 1;
    const int t0 = bid * p.C;
    if (t0 >= p.T) return;
    const int nt = min(p.C, p.T - t0), ne = nt * K, items = nt * ntiles;
    auto load_item = [&](int item) {
        V32 r = {};
        const int tok = item / ntiles, c = (item - tok * ntiles) * 32 + lane;
        if (item < items && c < nchunks)
            r = ld32_readonly(static_cast<const char*>(p.x) + ((size_t)(t0 + tok) * p.H + (size_t)c * 16) * 2);
        return r;
    };
    constexpr int kAhead = kExpand ? 1 : 4;
    V32 v[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) v[u] = load_item(warp + u * nwarps);
    int64_t raw = -1;
    float w = 0.f;
    if (tid < ne) {
        raw = ld_ro(p.topk_idx + (size_t)t0 * K + tid);
        if (p.topk_weights) w = ld_ro(p.topk_weights + (size_t)t0 * K + tid);
    }
    const int e = (uint64_t)raw < (uint64_t)p.E ? (int)raw : -1;
    if (tid < ne) s_exp[tid] = e;
    __syncthreads();
    int pos = sent_before(p, t0);
    for (int tok = 0; tok < nt; ++tok) {
        bool any = false;
        for (int k = 0; k < K; ++k) any |= s_exp[tok * K + k] >= 0;
        if (tid == 0) s_pos[tok] = any ? pos : -1, p.token_pos[t0 + tok] = any ? pos : -1;
        pos += any ? 1 : 0;
    }
    if (kExpand) {
        int* before = smem_i32 + p.E + 1;
        count_hits(p, smem_i32);
        count_tokens<1, true>(p.topk_idx, 0, t0, K, p.E, choices_in_pairs(p.topk_idx, K), before);
        __syncthreads();
        for (int i = tid; i < p.E; i += nthr) smem_i32[i] = aligned_count(smem_i32[i], p.alignment);
        __syncthreads();
        exclusive_sums(smem_i32, p.E);
        if (tid < ne) {
            bool last = e >= 0;
            for (int k = tid + 1; k < K; ++k) last = last && s_exp[k] != e;
            const int row = last ? row_with_room(p, smem_i32[e] + before[e]) : -1;
            s_row[tid] = row;
            p.rows[(size_t)t0 * K + tid] = row;
        }
    }
    __syncthreads();
    if (tid < ne) {
        const int tok = tid / K, k = tid - tok * K, pos = s_pos[tok];
        int master = 0;
        for (int j = 0; j < K; ++j)
            if (s_exp[tok * K + j] >= 0) master = j;
        const size_t at = (size_t)t0 * K + tid;
        p.dst_slot[at] = pos >= 0 && k == master ? pos : -1;
        if (p.copied_topk_idx) p.copied_topk_idx[at] = raw;
        if (pos >= 0) {
            p.recv_topk_idx[(size_t)pos * K + k] = e;
            int32_t* md = p.recv_src_metadata + (size_t)pos * (K + 2);
            if (k == 0) md[0] = t0 + tok;
            if (k == 1 % K) md[1] = master;
            if (kExpand) {
                const int row = s_row[tid];
                md[2 + k] = row;
                if (p.recv_topk_weights && row >= 0) p.recv_topk_weights[row] = w;
            } else if (p.recv_topk_weights) {
                p.recv_topk_weights[(size_t)pos * K + k] = w;
            }
        }
    }
    char* out = static_cast<char*>(p.recv_x);
    for (int i0 = warp; i0 < items; i0 += nwarps * kAhead) {
        if (i0 != warp) {
#pragma unroll
            for (int u = 0; u < kAhead; ++u) v[u] = load_item(i0 + u * nwarps);
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int item = i0 + u * nwarps;
            if (item >= items) break;
            const int tok = item / ntiles, c = (item - tok * ntiles) * 32 + lane;
            if (c >= nchunks) continue;
            if (kExpand) {
                for (int k = tok * K; k < (tok + 1) * K; ++k)
                    if (s_row[k] >= 0) st32(out + ((size_t)s_row[k] * p.H + (size_t)c * 16) * 2, v[u]);
            } else if (s_pos[tok] >= 0) {
                st32(out + ((size_t)s_pos[tok] * p.H + (size_t)c * 16) * 2, v[u]);
            }
        }
    }
}

// Behind ep_elastic_bits_kernel: as ep_dispatch_rows_kernel, a warp owns tiles of one token,
// finds the token's place itself and needs no other warp; the warp of a token's first tile
// writes what there is per entry. Block 0 writes and passes on the counts.
// Two tiles per warp and 40 warps per SM: a row is stored once (or K times, few in general),
// so it is the bytes requested at a time that matter. Flat, 4096 rows of 14 KB, dispatch
// alone: 20.3 us, one tile and 32 warps 29.0, 48 warps 25.6, four tiles and 32 warps 20.8 (a
// block per eight tokens and a layout kernel of one cluster before: 23.5). Expanded, the
// layer, 4096 rows of 14 KB to 2 and to 8: 64.8 and 176.9 us, one tile and 40 warps 74.9 and
// 178.3, 42 warps in blocks of seven 71.7 and 176.4, four tiles and 32 warps 67.5 and 182.1
// (a block per token before: 65.1 and 179.2; with what the layout kernel has lost since 63.2
// and 172.2).

template <bool kExpand, bool kOwn>
__global__ void __launch_bounds__(kElasticWarps * 32, 10) ep_elastic_rows_kernel(ElasticSingleParams p) {
    extern __shared__ int smem_i32[];  // flat: [E + 1] hits / sums (block 0)
    __shared__ typename std::conditional<kOwn, OwnSegments::Shared, char>::type s_own;
    constexpr int kTiles = kElasticTiles;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    pdl_launch_dependents();
    if (blockIdx.x == 0) {
        pdl_wait();
        if (!kExpand) {
            take_totals(p, [&](int x, int listings, int) { smem_i32[x] = aligned_count(listings, p.alignment); });
            __syncthreads();
            exclusive_sums(smem_i32, p.E);
            for (int x = tid; x <= p.E; x += blockDim.x) p.psum_expert[x] = smem_i32[x];
            if (tid == 0) p.psum_rank[0] = bits_total<false>(p.bits, 0);
            __syncthreads();
        }
        if constexpr (kOwn) {
            OwnSegments segments(p, s_own);
            segments.make(p);
            write_segments(s_own, segments.per, p.bits, p.E, p.psum_expert, p.psum_rank);
            __syncthreads();
        }
        tell_host(p);
        return;
    }
    const int sub = warp / p.warps_per_row;
    const int group = (blockIdx.x - 1) / p.parts, part = (blockIdx.x - 1) - group * p.parts;
    const int first = (part * p.warps_per_row + warp - sub * p.warps_per_row) * kTiles;  // tile
    const int t = group * p.C + sub, K = p.K;
    const bool mine = t < p.T && lane < K;
    const int nchunks = p.H / 16;  // (asked of the parameters each time, 8 bytes spill)
    V32 v[kTiles];
#pragma unroll
    for (int u = 0; u < kTiles; ++u) {
        const int c = (first + u) * 32 + lane;
        if (t < p.T && c < nchunks)
            v[u] = ld32_readonly(static_cast<const char*>(p.x) + ((size_t)t * p.H + (size_t)c * 16) * 2, p.x_last);
    }
    int64_t raw = -1;
    float w = 0.f;
    if (mine) {
        raw = ld_ro(p.topk_idx + (size_t)t * K + lane);
        if (first == 0 && p.topk_weights) w = ld_ro(p.topk_weights + (size_t)t * K + lane);
    }
    const int e = (uint64_t)raw < (uint64_t)p.E ? (int)raw : -1;
    const unsigned named = __ballot_sync(kAll, e >= 0);
    pdl_wait();
    int row = -1, pos = -1;
    // (a repeat's earlier listings find the last one's row and store the same bytes)
    if constexpr (kOwn) {
        OwnSegments segments(p, s_own);
        if (named) pos = bits_before(p.bits, 0, t);
        int before = 0;
        if (e >= 0) before = bits_before(p.bits, 1 + e, t);
        segments.make(p);
        if (e >= 0) row = row_with_room(p, OwnSegments::start(s_own, segments.per, e) + before);
    } else {
        if (named) pos = bits_before(p.bits, 0, t);
        if (kExpand && e >= 0) row = row_with_room(p, ld_ro(p.starts + e) + bits_before(p.bits, 1 + e, t));
    }
    if (first == 0 && t < p.T) {
        const int master = 31 - __clz(named);
        const unsigned same = __match_any_sync(kAll, e);
        const int kept = 31 - __clz(same) == lane ? row : -1;  // the entry's row: at its last listing
        const size_t at = (size_t)t * K + lane;
        if (mine) {
            p.dst_slot[at] = named && lane == master ? pos : -1;
            if (p.copied_topk_idx) p.copied_topk_idx[at] = raw;
            if (kExpand) p.rows[at] = kept;
            if (named) {
                p.recv_topk_idx[(size_t)pos * K + lane] = e;
                int32_t* md = p.recv_src_metadata + (size_t)pos * (K + 2);
                if (lane == 0) md[0] = t;
                if (lane == 1 % K) md[1] = master;
                if (kExpand) {
                    md[2 + lane] = kept;
                    if (p.recv_topk_weights && kept >= 0) p.recv_topk_weights[kept] = w;
                } else if (p.recv_topk_weights) {
                    p.recv_topk_weights[(size_t)pos * K + lane] = w;
                }
            }
        }
        if (!kExpand && lane == 0) p.token_pos[t] = pos;
    }
    char* out = static_cast<char*>(p.recv_x);
    const size_t row_bytes = (size_t)p.H * 2;
    if (kExpand) {
#pragma unroll 4
        for (int k = 0; k < K; ++k) {
            const int r = __shfl_sync(kAll, row, k);
            if (r < 0) continue;
#pragma unroll
            for (int u = 0; u < kTiles; ++u) {
                const int c = (first + u) * 32 + lane;
                if (c < nchunks) st32(out + (size_t)r * row_bytes + (size_t)c * 32, v[u]);
            }
        }
    } else if (named) {
#pragma unroll
        for (int u = 0; u < kTiles; ++u) {
            const int c = (first + u) * 32 + lane;
            if (c < nchunks) st32(out + (size_t)pos * row_bytes + (size_t)c * 32, v[u]);
        }
    }
}

__global__ void ep_elastic_fill_ones_kernel(float* w, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        w[i] = 1.0f;
}

}  // namespace

cudaError_t launch_elastic_route(const ElasticRouteParams& p, cudaStream_t stream) {
    LaunchScope scope("ep_elastic_route", stream);
    const int chunks = p.T > 0 ? (p.T + kThreads - 1) / kThreads : 1;
    ep_elastic_route_kernel<<<dim3(p.R, chunks), kThreads, 0, stream>>>(p);
    return scope.done(cudaGetLastError());
}

cudaError_t launch_elastic_epilogue(const ElasticEpilogueParams& p, int num_sms, cudaStream_t stream,
                                    bool pdl) {
    const int cap_blocks = (p.R * p.M + kWarps - 1) / kWarps;
    const int grid = max(1, min(2 * num_sms, cap_blocks));
    // with `pdl` the blocks may become resident while the exchange's last kernel drains;
    // they wait for its completion before they read anything
    return launch_kernel("ep_elastic_epilogue", ep_elastic_epilogue_kernel, dim3(grid), dim3(kThreads), 0, 1,
                         LaunchCtx{stream, num_sms, pdl}, p);
}

cudaError_t launch_elastic_expand_scan(const ElasticExpandParams& p, cudaStream_t stream) {
    LaunchScope scope("ep_elastic_expand_scan", stream);
    ep_elastic_expand_scan_kernel<<<p.L, kThreads, 0, stream>>>(p);
    return scope.done(cudaGetLastError());
}

cudaError_t launch_elastic_expand_copy(const ElasticExpandParams& p, int num_sms, cudaStream_t stream) {
    LaunchScope scope("ep_elastic_expand_copy", stream);
    ep_elastic_expand_copy_kernel<<<4 * num_sms, kThreads, 0, stream>>>(p);
    return scope.done(cudaGetLastError());
}

cudaError_t launch_elastic_local_reduce(const ElasticLocalReduceParams& p, int num_sms,
                                        cudaStream_t stream) {
    LaunchScope scope("ep_elastic_local_reduce", stream);
    ep_elastic_local_reduce_kernel<<<4 * num_sms, kThreads, 0, stream>>>(p);
    return scope.done(cudaGetLastError());
}

namespace {
// One launch saves the host 2 us of 11 - 16, which most of these calls are bound by, and costs the
// device up to 2 (the layer, wall | device, counting and behind a layout kernel).
// Flat rows, up to seven tokens per SM in one resident wave: 520 tokens of 8 KB to 8 11.5 | 8.4 and
// 13.5 | 7.7, 1036 11.5 | 11.3 and 13.5 | 8.9, of 14 KB 13.2 | 13.2 and 13.7 | 11.3. Above 4096
// choices only where the host's time counts: a call whose host waits for the counts gets them
// later (1000 to 8: 30.4 - 32.0 and 28.8 - 29.7), a captured one has paid for its launches (the
// layers in a graph, 520 of 8 KB 8.2 and 7.9, 1036 10.9 and 9.3, of 1 KB 8.6 and 6.4), and with
// more than eight choices a block counts longer than the launch takes (518 of 1 KB to 16 12.8 | 12.4
// and 13.7 | 7.1).
// Expanded rows, where every block counts all choices: two tokens per SM; four while they are 16
// choices (444 of 4 KB to 4 11.4 | 10.2 and 13.7 | 11.2, 394 of 8 KB to 6 15.1 | 14.9 and 15.0 | 14.9)
// and the rows have up to eight tiles, a warp each: above, the blocks are two to an SM and more than
// one wave (444 of 14 KB to 4 17.9 | 17.8 and 16.4 | 16.2), which a host that waits does not notice
// (a call that waits, 444 to 4 21.5 and 24.3, 394 to 6 22.7 and 24.7).
bool counts_in_copy_kernel(int T, int K, int H, int num_sms, bool expand, HostIs host) {
    if (expand)
        return T <= 2 * num_sms || (T <= 4 * num_sms && T * K <= 16 * num_sms &&
                                    (host == HostIs::kWaiting || H <= 8 * kTileChannels));
    return T <= 7 * num_sms && T * K <= (host == HostIs::kFree && K <= 8 ? 8 * 7 * num_sms : 4096);
}

// Expanded rows whose segments every block of the copy kernel makes (the figures: OwnSegments). With
// 256 experts and two loads for each, long rows, whose blocks move least for what they read, lose
// (1100 tokens of 14 KB to 2 20.8 | 21.2, of 5 KB 13.4 | 12.8; of 14 KB to 2 of 160 20.2 | 20.0).
bool makes_own_segments(int T, int E, int H) {
    if (T > kOwnChunks * kChunkTokens || E > kOwnExperts) return false;
    return E * listings_stride_of((T + kChunkTokens - 1) / kChunkTokens) <= 160 * kOwnChunks || H <= 8 * kTileChannels;
}
}  // namespace

bool elastic_single_tables(int T, int K, int E, int H, bool expand, HostIs host, int num_sms, void* scratch,
                           size_t bytes, unsigned* ticket, SingleTables* tables) {
    *tables = SingleTables();
    if (K > kMaxTopk || E > kMaxExperts) return false;
    if (counts_in_copy_kernel(T, K, H, num_sms, expand, host)) return true;
    const bool own = expand && makes_own_segments(T, E, H);
    const size_t starts =
        own ? (size_t)E * kOwnChunks * sizeof(uint16_t) : ((size_t)(E + 1) * sizeof(int32_t) + 15) / 16 * 16;
    if (starts > bytes) return false;
    if (own)
        tables->listings = static_cast<uint16_t*>(scratch);
    else
        tables->starts = static_cast<int32_t*>(scratch);
    tables->bits = route_bits(static_cast<char*>(scratch) + starts, bytes - starts, T, expand ? 1 + E : 1);
    tables->ticket = ticket;
    return tables->bits.words != nullptr;
}

cudaError_t launch_elastic_single_dispatch(ElasticSingleParams p, bool expand, const SingleTables& tables,
                                           const LaunchCtx& ctx) {
    const int ntiles = (p.H + kTileChannels - 1) / kTileChannels;
    if (tables.bits.words == nullptr) {
        // one launch: the block of the counts, and a block per token or (flat) per as many
        // tokens as make one resident wave
        p.C = expand ? 1 : (p.T + 2 * ctx.num_sms - 1) / (2 * ctx.num_sms);
        if (p.C > 128 / p.K) p.C = 128 / p.K;
        if (p.C < 1) p.C = 1;
        const int items = p.C * ntiles;
        const int warps = items < 8 ? 8 : items < 16 ? items : 16;
        auto k = expand ? ep_elastic_single_copy_kernel<true> : ep_elastic_single_copy_kernel<false>;
        return launch_kernel("ep_elastic_single_copy", k, dim3(1 + (p.T + p.C - 1) / p.C), dim3(warps * 32),
                             (size_t)(2 * p.E + 1) * sizeof(int), 1, ctx, p);
    }
    p.bits = tables.bits, p.ticket = tables.ticket, p.own_segments = tables.listings != nullptr;
    if (p.own_segments)
        p.listings = tables.listings;
    else
        p.starts = tables.starts;
    p.x_last = input_beyond_l2(p.T, expand ? p.K : 1, p.H, false);
    auto layout = expand ? ep_elastic_bits_kernel<true> : ep_elastic_bits_kernel<false>;
    const size_t smem = (expand ? 1 + (size_t)p.E : 1) * sizeof(uint4) + ((size_t)p.E + 1) * sizeof(int);
    if (cudaError_t e = allow_shared_memory(reinterpret_cast<const void*>(layout), smem)) return e;
    if (cudaError_t e = launch_kernel("ep_elastic_layout_bits", layout, dim3(p.bits.chunks), dim3(kBitsThreads), smem,
                                      1, ctx, p))
        return e;
    LaunchCtx chained = ctx;
    chained.pdl = ctx.chain;
    const int warps = (ntiles + kElasticTiles - 1) / kElasticTiles;  // of a row
    p.parts = (warps + kElasticWarps - 1) / kElasticWarps;
    p.warps_per_row = (warps + p.parts - 1) / p.parts;
    p.C = kElasticWarps / p.warps_per_row;
    auto k = p.own_segments ? ep_elastic_rows_kernel<true, true>
             : expand           ? ep_elastic_rows_kernel<true, false>
                                : ep_elastic_rows_kernel<false, false>;
    return launch_kernel("ep_elastic_rows", k, dim3(1 + (p.T + p.C - 1) / p.C * p.parts),
                         dim3(p.C * p.warps_per_row * 32), expand ? 0 : ((size_t)p.E + 1) * sizeof(int), 1, chained, p);
}

cudaError_t launch_elastic_fill_ones(float* w, size_t n, cudaStream_t stream) {
    LaunchScope scope("ep_elastic_fill_ones", stream);
    ep_elastic_fill_ones_kernel<<<64, 256, 0, stream>>>(w, n);
    return scope.done(cudaGetLastError());
}

}  // namespace mcep
