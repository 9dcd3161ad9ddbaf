// Hand-written sm_100a kernels of the EP hot path: routing layout, dispatch and
// combine, for a single rank and for a group of ranks on one NVLink domain.
//
// What they replace in the reference (paths inside the Mooncake tree):
//   mooncake-ep/src/mooncake_ep_kernel.cu:138-470  `dispatch`
//   mooncake-ep/src/mooncake_ep_kernel.cu:550-754  `combine`
// Design differences, all deliberate:
//   * receive order is deterministic (source rank, then token index): a token's
//     row inside its expert is (first row of the source's segment) + (earlier
//     tokens of the same source for that expert), never an atomic in arrival
//     order;
//   * dispatch has ONE data pass: the owner of an expert collects the counts
//     every source announces, answers each source with the first row of its
//     segment, and the source then stores the row - read once, quantised in
//     registers - straight into its final place in the owner's packed receive
//     area over NVLink (the reference stages the row locally, copies it to the
//     owner's staging and copies it again into the packed output);
//   * combine has ONE data pass over NVLink: expert outputs are made readable in
//     symmetric memory, and the token owner reads its K rows from the experts'
//     owners and reduces them in registers (the reference pushes every row into
//     staging at the token owner first);
//   * no cooperative launch, no grid-wide barrier; sender blocks depend on the
//     control block (block 0, resident first) and on other GPUs only;
//   * work is split by token and by row, not by expert, so the grid fills 148
//     SMs for 8 experts as well as for 256;
//   * the words ranks exchange are 64-bit (call sequence number << 32 | value)
//     and are never cleaned.
#include "ep_kernels.cuh"

#include <algorithm>
#include <climits>
#include <atomic>
#include <map>
#include <mutex>
#include <string>
#include <tuple>
#include <vector>

#include "ep_device.cuh"
#include "ep_launch.cuh"
#include "ep_routing.cuh"

namespace mcep {

static std::atomic<uint64_t> g_launches{0};
uint64_t kernel_launch_count() { return g_launches.load(); }

// Optional per-kernel timing: every launch is bracketed by two events on its own
// stream (which also serialises kernels that would otherwise overlap through
// programmatic dependent launch), so a caller can read each kernel's device time.
namespace {
struct TimingRec {
    const char* name;
    cudaEvent_t a, b;
};
std::atomic<bool> g_timing{false};
std::mutex g_timing_mu;
std::vector<TimingRec> g_recs;
}  // namespace

void set_kernel_timing(bool on) { g_timing.store(on); }

std::string drain_kernel_times() {
    std::lock_guard<std::mutex> lk(g_timing_mu);
    std::map<std::string, std::pair<int, double>> agg;
    for (auto& r : g_recs) {
        float ms = 0.f;
        if (cudaEventSynchronize(r.b) == cudaSuccess &&
            cudaEventElapsedTime(&ms, r.a, r.b) == cudaSuccess) {
            auto& e = agg[r.name];
            e.first += 1;
            e.second += ms;
        }
        cudaEventDestroy(r.a);
        cudaEventDestroy(r.b);
    }
    g_recs.clear();
    std::string out;
    for (auto& kv : agg) {
        char line[256];
        snprintf(line, sizeof(line), "%s %d %.6f\n", kv.first.c_str(), kv.second.first,
                 kv.second.second);
        out += line;
    }
    return out;
}

LaunchScope::LaunchScope(const char* name, cudaStream_t stream) : name_(name), stream_(stream) {
    if (g_timing.load()) {
        cudaEventCreate(&a_);
        cudaEventCreate(&b_);
        cudaEventRecord(a_, stream_);
    }
}

cudaError_t LaunchScope::done(cudaError_t err) {
    if (a_ != nullptr) {
        cudaEventRecord(b_, stream_);
        std::lock_guard<std::mutex> lk(g_timing_mu);
        g_recs.push_back(TimingRec{name_, a_, b_});
    }
    if (err == cudaSuccess) g_launches.fetch_add(1);
    return err;
}

bool kernel_timing_on() { return g_timing.load(); }

cudaError_t allow_shared_memory(const void* kernel, size_t smem) {
    if (smem <= 40 * 1024) return cudaSuccess;
    static std::mutex mu;
    static std::map<std::pair<const void*, int>, size_t> allowed;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    size_t& have = allowed[std::make_pair(kernel, dev)];
    if (smem <= have) return cudaSuccess;
    e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess) have = smem;
    return e;
}

cudaError_t cluster_fits(const void* kernel, int blocks, int threads, size_t smem, bool* fits) {
    *fits = false;
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, int, int, size_t>, bool> known;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    const auto key = std::make_tuple(kernel, dev, blocks, threads, smem);
    const auto it = known.find(key);
    if (it != known.end()) {
        *fits = it->second;
        return cudaSuccess;
    }
    if ((e = allow_shared_memory(kernel, smem))) return e;
    if (blocks > 8 && (e = cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(blocks), cfg.blockDim = dim3(threads), cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = blocks;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr, cfg.numAttrs = 1;
    int clusters = 0;
    e = cudaOccupancyMaxActiveClusters(&clusters, kernel, &cfg);
    if (e != cudaSuccess && e != cudaErrorInvalidClusterSize) return e;
    if (e != cudaSuccess) cudaGetLastError();
    *fits = known[key] = e == cudaSuccess && clusters > 0;
    return cudaSuccess;
}

namespace kernels {

constexpr unsigned kFull = 0xffffffffu;

template <typename... KArgs, typename... Args>
cudaError_t launch(const char* name, void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem,
                   const LaunchCtx& ctx, Args&&... args) {
    return launch_kernel(name, kernel, grid, block, smem, 1, ctx, std::forward<Args>(args)...);
}

__device__ __forceinline__ int warp_inclusive_scan(int v, int lane) {
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        int u = __shfl_up_sync(kFull, v, d);
        if (lane >= d) v += u;
    }
    return v;
}

// In-place exclusive scan of a[0..n) in shared memory; a[n] receives the total.
// Every thread of the block must call it.
__device__ void block_exclusive_scan(int* a, int n, int* warp_totals /*[32]*/) {
    const int nthr = blockDim.x, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int per = (n + nthr - 1) / nthr;
    const int b = min(tid * per, n), e = min(b + per, n);
    int sum = 0;
    for (int i = b; i < e; ++i) sum += a[i];
    int incl = warp_inclusive_scan(sum, lane);
    if (lane == 31) warp_totals[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        int w = lane < nwarps ? warp_totals[lane] : 0;
        int wi = warp_inclusive_scan(w, lane);
        warp_totals[lane] = wi - w;
        if (lane == 31) a[n] = wi;
    }
    __syncthreads();
    int run = warp_totals[warp] + incl - sum;
    for (int i = b; i < e; ++i) {
        int v = a[i];
        a[i] = run;
        run += v;
    }
    __syncthreads();
}

// Last index i in [0, n) with pre[i] <= g (pre is a non-decreasing exclusive
// prefix, pre[0] == 0): the non-empty segment that holds row g.
__device__ __forceinline__ int find_segment(const int* pre, int n, int g) {
    int lo = 0, hi = n;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (pre[mid] <= g)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// =============================================================================
// waiting for words of other ranks
// =============================================================================
// The timeout rule of mooncake-ep/src/mooncake_ep_kernel.cu:417-429 and :685-699:
// after `timeout` the waiter clears active_ranks[src]; whoever sees the entry
// cleared stops waiting. Every wait is also bounded by the hard limit.

//
// Waits of one dispatch call form a chain: an owner waits for the sources'
// counts; a sender waits for the owner's answer, which a live owner may hold
// back until it has given up on a dead source; a receiver waits for the senders'
// payload words, which may be late for the same reason. So the answer is given
// twice, and the payload word three times, the bound of the count - otherwise
// one dead rank would make every live rank give up on every other. The dead
// rank itself is still given up on after ONE timeout: whoever times out clears
// its entry of the mask, and every waiter looks at the mask.
__device__ __forceinline__ WaitCfg scaled(const WaitCfg& w, int times) {
    WaitCfg r = w;
    if (r.timeout_ns >= 0) r.timeout_ns *= times;
    r.hard_timeout_ns *= times;
    return r;
}

// One waiter per word (or waiters that may disagree harmlessly). Returns the
// word's value (>= 1) or 0 when given up.
__device__ __forceinline__ uint32_t wait_word(const uint64_t* word, uint32_t seq, const WaitCfg& w,
                                              int src) {
    uint64_t start = 0;
    while (true) {
        const uint64_t v = ld_acquire_sys(word);
        if ((uint32_t)(v >> 32) == seq) return (uint32_t)v;
        const uint64_t now = globaltimer_ns();
        if (start == 0) start = now;
        const int64_t waited = (int64_t)(now - start);
        if (w.timeout_ns >= 0 && waited > w.timeout_ns) st_volatile_s32(w.active_ranks + src, 0);
        if (waited > w.hard_timeout_ns) {
            st_volatile_s32(w.active_ranks + src, 0);
            atomicOr(w.status, kStatusHardTimeout);
        }
        if (!ld_volatile_s32(w.active_ranks + src)) return 0;
    }
}

// Many waiters per word that must agree (or one token of a result would count a
// rank in and the next would not): the first block to reach a verdict publishes
// it with a compare-and-swap into a local word, and every block - that one
// included - takes the verdict from that word:
//   resolved = seq << 32 | value     arrived
//   resolved = seq << 32 | 0         given up
// No block waits for another block: each keeps polling the peer's word itself
// until some verdict exists. Returns the value, or 0.
__device__ __forceinline__ uint32_t resolve_flag(const uint64_t* flags, uint64_t* resolved, int i,
                                                 uint32_t seq, const WaitCfg& w, int src,
                                                 bool primary = true) {
    unsigned long long* res = reinterpret_cast<unsigned long long*>(resolved + i);
    uint64_t start = 0;
    if (!primary) {
        // Many blocks want the same verdict. One of them (the "primary" for this
        // flag) goes for the flag at once; the others look at the verdict word
        // alone for a short while, which keeps hundreds of blocks from hammering
        // one address with compare-and-swaps, and then fall back to doing the
        // work themselves - they never depend on the primary making progress.
        start = globaltimer_ns();
        while (globaltimer_ns() - start < 4000) {
            const uint64_t r = ld_acquire_gpu(resolved + i);
            if ((uint32_t)(r >> 32) == seq) {
                const uint32_t v = (uint32_t)r;
                if (v) (void)ld_acquire_sys(flags + i);
                return v;
            }
        }
    }
    while (true) {
        // both words are requested together: one round trip in the common case
        const uint64_t r = ld_acquire_gpu(resolved + i);
        const uint64_t f = ld_acquire_sys(flags + i);
        if ((uint32_t)(r >> 32) == seq) {
            // decided already (possibly by another block). If it is an arrival,
            // the flag load above was our own acquire of the sender's release -
            // unless it raced ahead of the flag, then take it again.
            const uint32_t v = (uint32_t)r;
            if (v && (uint32_t)(f >> 32) != seq) (void)ld_acquire_sys(flags + i);
            return v;
        }
        unsigned long long mine;
        if ((uint32_t)(f >> 32) == seq) {
            mine = (unsigned long long)f;  // arrived
        } else {
            const uint64_t now = globaltimer_ns();
            if (start == 0) start = now;
            const int64_t waited = (int64_t)(now - start);
            if (w.timeout_ns >= 0 && waited > w.timeout_ns) st_volatile_s32(w.active_ranks + src, 0);
            if (waited > w.hard_timeout_ns) {
                st_volatile_s32(w.active_ranks + src, 0);
                atomicOr(w.status, kStatusHardTimeout);
            }
            if (ld_volatile_s32(w.active_ranks + src)) continue;  // keep waiting
            mine = (unsigned long long)seq << 32;                 // given up
        }
        // first verdict wins; the value the swap returns is the winner's
        const unsigned long long old = atomicCAS(res, (unsigned long long)r, mine);
        const unsigned long long verdict = (old == (unsigned long long)r) ? mine : old;
        if ((uint32_t)(verdict >> 32) != seq) continue;  // lost to a stale word: look again
        const uint32_t v = (uint32_t)verdict;
        if (v && (uint32_t)(f >> 32) != seq) (void)ld_acquire_sys(flags + i);
        return v;
    }
}

// A word another block of this GPU writes (the control block's verdicts). The
// writer is resident before any reader and never waits for a reader.
__device__ __forceinline__ uint32_t wait_local_word(const uint64_t* word, uint32_t seq,
                                                    const WaitCfg& w) {
    uint64_t start = 0;
    while (true) {
        const uint64_t v = ld_acquire_gpu(word);
        if ((uint32_t)(v >> 32) == seq) return (uint32_t)v;
        const uint64_t now = globaltimer_ns();
        if (start == 0) start = now;
        if ((int64_t)(now - start) > w.hard_timeout_ns) {
            atomicOr(w.status, kStatusHardTimeout);
            return 0;
        }
    }
}

// The same from a kernel that may have started beside the writer's, which is ahead of it in the
// stream: looked at for a while only, then that kernel's end is waited for, which has the word.
__device__ __forceinline__ uint32_t local_word_of_kernel_ahead(const uint64_t* word, uint32_t seq, const WaitCfg& w) {
    const uint64_t start = globaltimer_ns();
    do {
        const uint64_t v = ld_acquire_gpu(word);
        if ((uint32_t)(v >> 32) == seq) return (uint32_t)v;
    } while (globaltimer_ns() - start < 50000);
    pdl_wait();
    return wait_local_word(word, seq, w);
}

// =============================================================================
// phase trace (diagnostic builds only: -DMCEP_PHASE_TRACE)
// =============================================================================
// Thread 0 of every block stamps the global nanosecond timer at phase
// boundaries, so blocks - and kernels - can be lined up against each other.
// Compiled out of the normal library.
#ifdef MCEP_PHASE_TRACE
constexpr int kTraceBodies = 4, kTraceBlocks = 1024, kTraceSlots = 8;
__device__ unsigned long long g_phase_trace[kTraceBodies][kTraceBlocks][kTraceSlots];
#define MCEP_TRACE(body, slot)                                              \
    do {                                                                    \
        if (threadIdx.x == 0 && blockIdx.x < kTraceBlocks)                  \
            g_phase_trace[body][blockIdx.x][slot] = globaltimer_ns();       \
    } while (0)
#else
#define MCEP_TRACE(body, slot) \
    do {                       \
    } while (0)
#endif

// =============================================================================
// routing layout
// =============================================================================
// One block owns `epc` consecutive experts. It builds, in shared memory, one
// bit per (expert, token) and a popcount prefix per 32-token word; a slot is
// then prefix + popcount of the lower bits. Token order is the only order.
__global__ void __launch_bounds__(1024)
    ep_routing_layout_kernel(LayoutParams p, int epc, int words) {
    extern __shared__ uint32_t smem_u32[];
    uint32_t* mask = smem_u32;
    uint32_t* wpre = smem_u32 + (size_t)epc * words;
    __shared__ bool s_last;

    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int e0 = blockIdx.x * epc;
    const int e1 = min(p.E, e0 + epc);
    const int ne = e1 - e0;
    const int n = p.T * p.K;

    for (int i = tid; i < ne * words; i += nthr) mask[i] = 0;
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    // Every block reads the whole index matrix; the loads are issued eight at a
    // time so a pass costs a few memory round trips, not one per entry.
    constexpr int kU = 8;
    for (int i0 = tid; i0 < n; i0 += nthr * kU) {
        int ev[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = i0 + u * nthr;
            ev[u] = i < n ? (int)ld_ro(p.topk_idx + i) : -1;
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int e = ev[u];
            if (e >= e0 && e < e1) {
                const int t = (i0 + u * nthr) / p.K;
                atomicOr(&mask[(e - e0) * words + (t >> 5)], 1u << (t & 31));
            }
        }
    }
    __syncthreads();
    for (int le = warp; le < ne; le += nwarps) {
        int carry = 0;
        for (int w0 = 0; w0 < words; w0 += 32) {
            const int w = w0 + lane;
            const int c = w < words ? __popc(mask[le * words + w]) : 0;
            const int incl = warp_inclusive_scan(c, lane);
            if (w < words) wpre[le * words + w] = carry + incl - c;
            carry += __shfl_sync(kFull, incl, 31);
        }
        if (lane == 0) {
            const int e = e0 + le;
            p.count[e] = carry;
            if (p.recv_count) p.recv_count[e] = carry;
            if (p.layout_range) p.layout_range[e] = carry;  // begin 0 | count
        }
    }
    __syncthreads();
    for (int i0 = tid; i0 < n; i0 += nthr * kU) {
        int ev[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = i0 + u * nthr;
            ev[u] = i < n ? (int)ld_ro(p.topk_idx + i) : -2;
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int i = i0 + u * nthr;
            const int e = ev[u];
            if (e >= e0 && e < e1) {
                const int t = i / p.K, k = i - t * p.K;
                bool dup = false;
                for (int kk = 0; kk < k; ++kk) dup |= ((int)ld_ro(p.topk_idx + t * p.K + kk) == e);
                const int o = (e - e0) * words + (t >> 5);
                p.slot[i] = dup ? -1 : (int)(wpre[o] + __popc(mask[o] & ((1u << (t & 31)) - 1u)));
            } else if (e < 0 && i < n && blockIdx.x == 0) {
                p.slot[i] = -1;
            }
        }
    }
    if (p.rank_count == nullptr && p.expert_prefix == nullptr) return;

    // The block that finishes last turns the per-expert counts into per-rank
    // counts and prefix offsets inside each rank's block of experts.
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = (atomicInc(p.ticket, gridDim.x - 1) == gridDim.x - 1);
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const int L = p.E / p.R;
    for (int r = warp; r < p.R; r += nwarps) {
        int carry = 0;
        for (int b = 0; b < L; b += 32) {
            const int le = b + lane;
            const int c = le < L ? ld_l2(p.count + r * L + le) : 0;
            const int incl = warp_inclusive_scan(c, lane);
            if (le < L && p.expert_prefix) p.expert_prefix[r * L + le] = carry + incl - c;
            carry += __shfl_sync(kFull, incl, 31);
        }
        if (lane == 0 && p.rank_count) p.rank_count[r] = carry;
    }
}

// ---- the same layout in two passes over token chunks ------------------------------
// The kernel above lets every block read the whole index matrix (each block owns
// some experts). For large batches that costs more than the work itself, so the
// usual route is two small kernels in which a block owns a CHUNK of tokens and
// reads only that chunk:
//   pass 1  per-chunk histogram of the (de-duplicated) expert choices;
//   pass 2  per expert, the count of all earlier chunks (a short column sum) plus
//           the position inside the chunk (bitmap + popcount, as above) = slot;
//           the block of the last chunk also writes the totals.
// A repeated expert inside a token counts once; token order is the only order.
// One lane per token: the token's K choices are requested together (one memory
// round trip) and de-duplicated in registers; e[k] = -1 for masked, out-of-range
// and repeated entries.
__device__ __forceinline__ void request_token_choices(const int64_t* topk_idx, int t, int T, int K,
                                                      int E, int (&e)[kMaxTopk]) {
#pragma unroll
    for (int k = 0; k < kMaxTopk; ++k) {
        e[k] = -1;
        if (t < T && k < K) {
            const int v = (int)ld_ro(topk_idx + (size_t)t * K + k);
            e[k] = (v >= 0 && v < E) ? v : -1;
        }
    }
}
__device__ __forceinline__ void drop_repeated_choices(int (&e)[kMaxTopk]) {
#pragma unroll
    for (int k = 1; k < kMaxTopk; ++k) {
        bool dup = false;
#pragma unroll
        for (int kk = 0; kk < k; ++kk) dup |= (e[kk] == e[k]);
        if (dup) e[k] = -1;
    }
}
__device__ __forceinline__ void load_token_choices(const int64_t* topk_idx, int t, int T, int K, int E,
                                                   int (&e)[kMaxTopk]) {
    request_token_choices(topk_idx, t, T, K, E, e);
    drop_repeated_choices(e);
}

// a chunk is `warps` x 32 tokens: warp w of the block takes tokens [32w, 32w + 32)
__global__ void __launch_bounds__(256) ep_layout_hist_kernel(LayoutParams p) {
    extern __shared__ int smem_i32[];
    int* hist = smem_i32;  // [E]
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int t = blockIdx.x * nthr + tid;
    // The first kernel of a call may be chained to the kernel that WRITES the index
    // matrix (the elastic calls' route kernel): nothing is read before the wait.
    for (int i = tid; i < p.E; i += nthr) hist[i] = 0;
    pdl_wait();
    pdl_launch_dependents();
    int e[kMaxTopk];
    load_token_choices(p.topk_idx, t, p.T, p.K, p.E, e);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kMaxTopk; ++k)
        if (e[k] >= 0) atomicAdd(&hist[e[k]], 1);
    __syncthreads();
    for (int i = tid; i < p.E; i += nthr) p.chunk_hist[(size_t)blockIdx.x * p.E + i] = hist[i];
}

__global__ void __launch_bounds__(256) ep_layout_slot_kernel(LayoutParams p) {
    extern __shared__ int smem_i32[];
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, words = nthr >> 5;
    int* base = smem_i32;                                          // [E] tokens of earlier chunks
    uint32_t* mask = reinterpret_cast<uint32_t*>(smem_i32 + p.E);  // [E][words], word w written by warp w only
    const int t = blockIdx.x * nthr + tid;
    int e[kMaxTopk];
    load_token_choices(p.topk_idx, t, p.T, p.K, p.E, e);
    for (int i = tid; i < p.E * words; i += nthr) mask[i] = 0;
    __syncthreads();
    // bit (expert, token): lanes of a warp that chose the same expert in the same
    // position k form a group; its lowest lane ORs the group into the warp's word
    for (int k = 0; k < p.K; ++k) {
        const unsigned key = e[k] >= 0 ? (unsigned)e[k] : (0x80000000u | lane);
        const unsigned grp = __match_any_sync(kFull, key);
        if (e[k] >= 0 && (int)(__ffs(grp) - 1) == lane) mask[e[k] * words + warp] |= grp;
        __syncwarp();
    }
    pdl_wait();
    pdl_launch_dependents();
    for (int i = tid; i < p.E; i += nthr) {
        // column sum over the earlier chunks, eight loads in flight at a time
        int sum = 0;
        for (int c0 = 0; c0 < (int)blockIdx.x; c0 += 8) {
            int v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u)
                v[u] = c0 + u < (int)blockIdx.x ? ld_l2(p.chunk_hist + (size_t)(c0 + u) * p.E + i) : 0;
#pragma unroll
            for (int u = 0; u < 8; ++u) sum += v[u];
        }
        base[i] = sum;
    }
    __syncthreads();
    if (t < p.T) {
        const unsigned lower = (1u << lane) - 1u;
#pragma unroll
        for (int k = 0; k < kMaxTopk; ++k) {
            if (k >= p.K) break;
            int slot = -1;
            if (e[k] >= 0) {
                const uint32_t* m = mask + e[k] * words;
                slot = base[e[k]] + __popc(m[warp] & lower);
                for (int w = 0; w < warp; ++w) slot += __popc(m[w]);
            }
            p.slot[(size_t)t * p.K + k] = slot;
        }
    }
    if (blockIdx.x != gridDim.x - 1) return;
    // the block of the last chunk knows every total
    __syncthreads();
    for (int i = tid; i < p.E; i += nthr) {
        int c = base[i];
        for (int w = 0; w < words; ++w) c += __popc(mask[i * words + w]);
        base[i] = c;
        p.count[i] = c;
        if (p.recv_count) p.recv_count[i] = c;
        if (p.layout_range) p.layout_range[i] = c;  // begin 0 | count
    }
    if (p.rank_count == nullptr && p.expert_prefix == nullptr) return;
    __syncthreads();
    const int L = p.E / p.R;
    for (int r = warp; r < p.R; r += words) {
        int carry = 0;
        for (int b = 0; b < L; b += 32) {
            const int le = b + lane;
            const int c = le < L ? base[r * L + le] : 0;
            const int incl = warp_inclusive_scan(c, lane);
            if (le < L && p.expert_prefix) p.expert_prefix[r * L + le] = carry + incl - c;
            carry += __shfl_sync(kFull, incl, 31);
        }
        if (lane == 0 && p.rank_count) p.rank_count[r] = carry;
    }
}

// ---- the same layout in one launch of one cluster -----------------------------------
// For callers that want finished positions and up to 16384 tokens. The blocks of one
// cluster share the tokens, one lane per token:
//   bit (expert, token) in the block's shared bitmap, word-major [word][E];
//   per expert: popcounts of the words -> exclusive prefix over the words, total;
//   cluster barrier; totals of the lower blocks through distributed shared memory;
//   slot = lower blocks + lower words + lower bits of the own word.
// 4096 tokens x 8 of 256: one launch in place of the two above (4 + 10 us).
constexpr int kLayoutCluster = 8, kLayoutClusterLarge = 16;

template <int KB>
__device__ __forceinline__ void cluster_layout(const LayoutParams& p, uint32_t* mask, int* pre, int* total) {
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, words = nthr >> 5;
    const int rank = blockIdx.x, blocks = gridDim.x;
    const int t = rank * nthr + tid;
    for (int i = tid; i < p.E * words; i += nthr) mask[i] = 0;
    int e[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) e[k] = -1;
    if (t < p.T) load_choices<KB, false>(p.topk_idx, t, p.K, p.E, choices_in_pairs(p.topk_idx, p.K), e);
    drop_repeats<KB, false>(e);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < KB; ++k)
        if (e[k] >= 0) atomicOr(&mask[warp * p.E + e[k]], 1u << lane);
    __syncthreads();
    for (int x = tid; x < p.E; x += nthr) {
        int run = 0;
        for (int w = 0; w < words; ++w) {
            const int c = __popc(mask[w * p.E + x]);
            pre[w * p.E + x] = run;
            run += c;
        }
        total[x] = run;
    }
    cluster_sync();  // (a block barrier as well)
    for (int x = tid; x < p.E; x += nthr) {
        int base;
        const int c = blocks > kLayoutCluster ? cluster_sum<kLayoutClusterLarge>(total + x, rank, blocks, &base)
                                              : cluster_sum<kLayoutCluster>(total + x, rank, blocks, &base);
        total[p.E + x] = base;
        if (rank == blocks - 1) {
            p.count[x] = c;
            if (p.recv_count) p.recv_count[x] = c;
            if (p.layout_range) p.layout_range[x] = c;  // begin 0 | count
        }
    }
    __syncthreads();
    if (t < p.T) {
        const unsigned lower = (1u << lane) - 1u;
        int32_t* out = p.slot + (size_t)t * p.K;
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            if (k >= p.K) break;
            int s = -1;
            if (e[k] >= 0) {
                const int at = warp * p.E + e[k];
                s = total[p.E + e[k]] + pre[at] + __popc(mask[at] & lower);
            }
            out[k] = s;
        }
    }
    cluster_sync();  // no block leaves while its totals may still be read
}

__global__ void __launch_bounds__(1024) ep_layout_cluster_kernel(LayoutParams p) {
    extern __shared__ int smem_i32[];
    const int words = blockDim.x >> 5;
    uint32_t* mask = reinterpret_cast<uint32_t*>(smem_i32);  // [words][E]
    int* pre = smem_i32 + words * p.E;                       // [words][E]
    int* total = smem_i32 + 2 * words * p.E;                 // [E] this block, [E] lower blocks
    pdl_wait();
    pdl_launch_dependents();
    if (p.K <= 4)
        cluster_layout<4>(p, mask, pre, total);
    else if (p.K <= 8)
        cluster_layout<8>(p, mask, pre, total);
    else
        cluster_layout<16>(p, mask, pre, total);
}

// ---- the layout as bits, for kernels that look positions up themselves -------------
// What dispatch uses between the smallest and the largest batches. Every chunk of 128
// tokens is a block of its own and nothing is summed here: per expert the chunk's bits
// (RouteBits) and their number, one load, one store. A block's words lie together: what a warp
// stores is four lines, as [expert][chunk] it was 32 (elastic calls, the layer: 4096 rows of
// 4 KB expanded to 8 of 512 55.9 us, now 54.5, to 2 of 2048 34.8, now 30.5). A sender finds
// its position from them in one round trip more than it would read a finished one
// (bits_before), but a finished one costs a cluster barrier, remote totals and a prefix over
// all experts before it exists: from the kernel's start to its end 5.7 us for 2001 tokens to 8
// of 128, 9.3 for 4096 to 8 of 256; here 2.4 and 2.
constexpr int kBitsThreads = 256;

template <int KB>
__device__ __forceinline__ void set_bits(const LayoutParams& p, uint32_t* mask) {
    const int t = blockIdx.x * kChunkTokens + threadIdx.x;
    int e[KB];
#pragma unroll
    for (int k = 0; k < KB; ++k) e[k] = -1;
    if (threadIdx.x < kChunkTokens && t < p.T)
        load_choices<KB, false>(p.topk_idx, t, p.K, p.E, choices_in_pairs(p.topk_idx, p.K), e);
#pragma unroll
    for (int k = 0; k < KB; ++k)  // (a repeated expert sets its bit twice)
        if (e[k] >= 0) atomicOr(&mask[e[k] * 4 + (threadIdx.x >> 5)], 1u << (threadIdx.x & 31));
}

__global__ void __launch_bounds__(kBitsThreads) ep_layout_bits_kernel(LayoutParams p) {
    extern __shared__ uint4 smem_u128[];  // [E] bits of this chunk
    const int tid = threadIdx.x;
    for (int i = tid; i < p.E; i += kBitsThreads) smem_u128[i] = make_uint4(0u, 0u, 0u, 0u);
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    uint32_t* mask = reinterpret_cast<uint32_t*>(smem_u128);
    if (p.K <= 4)
        set_bits<4>(p, mask);
    else if (p.K <= 8)
        set_bits<8>(p, mask);
    else
        set_bits<16>(p, mask);
    __syncthreads();
    for (int e = tid; e < p.E; e += kBitsThreads) {
        const uint4 m = smem_u128[e];
        p.bits.words[(size_t)blockIdx.x * p.bits.experts + e] = m;
        p.bits.counts[(size_t)e * p.bits.stride + blockIdx.x] =
            (uint8_t)(__popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w));
    }
}

// =============================================================================
// sending token rows (single rank and groups)
// =============================================================================
// A block takes a batch of `C` consecutive tokens, reads each bf16 row once (32
// bytes per lane, one warp per 512-channel tile), quantises it in registers when
// FP8 is on, and stores it to the row of every selected expert's packed receive
// area: this GPU's (single rank, or an expert this rank owns) or a peer's, over
// NVLink.
//
// A group's launch is one resident wave that strides over the batches; so is a single
// rank's, which sends small batches this way (larger ones: ep_dispatch_rows_kernel).
//
// What goes where for entry (t, k) with expert e, owner rank o, local expert le,
// row r = first row of this rank's segment in e + earlier tokens of this rank:
//   payload    -> o's receive rows   [le][r][H e4m3 | H bf16]
//   o == this rank: token index and scales go straight into the caller's
//                   src_info / transposed scales tensors;
//   o is a peer:    a side message [16 B: token index | 16 B of scales per 512
//                   channels] goes to o's side area [le][r]; o's receive duty
//                   moves it into its src_info / scales tensors.
struct SendView {
    const char* x;
    const int64_t* topk_idx;
    int T, K, E, R, M, H, rank;
    int L, RM;
    int C;                    // tokens per batch
    bool x_last;              // see input_beyond_l2
    RouteBits bits;           // the layout kernel's bits (words null: none), or
    const int32_t* slot;      // [T*K] position among this rank's tokens for the expert (layout kernel),
                              // or null: counted here (small batches, one per block)
    int32_t* status;
    // rows this rank owns
    char* recv_x;
    float* recv_scales;
    int32_t* recv_src_info;
    int row_bytes;
    int32_t* rowmap;
    // single rank, counted here: the receive layout, written by the block that takes the last batch
    int32_t* recv_count;
    int64_t* layout_range;
    // groups only
    const uint64_t* beg;      // local words: first row of this rank's segment per expert
    uint32_t seq;
    WaitCfg wait;
    size_t rx_off, meta_off;
    int meta_stride;
    char* const* s_peer;      // shared-memory copies of the peer table and the mask
    const int* s_active;
};

constexpr int kBatchEntries = 128;  // (token, k) entries of a batch

// Returns whether one of this thread's entries went to a peer.
// kCount: the positions are counted here, hist: [E] zeros in shared memory; else `bits` or `slot`
// have them. All threads of the block call it.
template <bool kFP8, bool kGroup, bool kCount>
__device__ __forceinline__ bool send_tokens(const SendView& v, int sid, int nsend, int* hist) {
    __shared__ char* s_dst[kBatchEntries];
    __shared__ char* s_meta[kGroup ? kBatchEntries : 1];
    __shared__ int s_raw[kBatchEntries];   // expert of the entry, -1: none
    __shared__ int s_exp[kBatchEntries];   // the same without repeats inside a token
    __shared__ int s_row[kBatchEntries];
    __shared__ int s_le[kBatchEntries];

    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int nchunks = v.H / 16;
    const int ntiles = (v.H + kTileChannels - 1) / kTileChannels;
    const int S = v.H / 128;
    const int K = v.K;

    // one warp item = one tile of one row of the batch that starts at token t
    auto load_item = [&](int t, int item) {
        V32 r = {};
        const int tok = item / ntiles, c = (item - tok * ntiles) * 32 + lane;
        if (tok < v.C && t + tok < v.T && c < nchunks)
            r = ld32_readonly(v.x + ((size_t)(t + tok) * v.H + (size_t)c * 16) * 2, !kCount && v.x_last);
        return r;
    };
    int t0 = sid * v.C;
    V32 ahead = load_item(t0, warp);
    if (kGroup && !kCount) pdl_wait();  // (the layout kernel has waited for the rows; it is its tables that come now)
    if (kCount && !kGroup && v.T == 0 && sid == 0)
        for (int e = tid; e < v.E; e += nthr) v.recv_count[e] = 0, v.layout_range[e] = 0;
    int counted = 0;  // tokens that are in hist
    bool remote = false;  // (of this thread's entries) something was stored in a peer's memory
    for (; t0 < v.T;) {
        const int nt = min(v.C, v.T - t0), ne = nt * K, items = nt * ntiles;
        const int t1 = t0 + nsend * v.C;
        int raw = -1, slot = 0;
        if (tid < ne) raw = (int)ld_ro(v.topk_idx + (size_t)t0 * K + tid);
        if (kCount) {
            count_tokens<1>(v.topk_idx, counted, t0, K, v.E, choices_in_pairs(v.topk_idx, K), hist);
        } else if (v.bits.words != nullptr) {
            if (raw >= 0 && raw < v.E) slot = bits_before(v.bits, raw, t0 + tid / K);
        } else if (tid < ne) {
            slot = ld_ro(v.slot + (size_t)t0 * K + tid);
        }
        if (raw >= v.E) raw = -1;
        if (tid < ne) s_raw[tid] = raw;
        __syncthreads();  // hist holds every token before t0
        const int tok0 = tid / K * K;  // first entry of this entry's token
        int e = raw;
        if (tid < ne) {
            for (int j = tok0; j < tid; ++j)
                if (s_raw[j] == raw) e = -1;  // a repeat of an earlier entry of this token
            s_exp[tid] = e;
        }
        if (nt > 1) __syncthreads();
        if (tid < ne) {
            char* dst = nullptr;
            char* meta = nullptr;
            int row = -1, le = 0;
            if (e >= 0) {
                int s = slot;
                if (kCount) {
                    s = hist[e];
                    for (int j = 0; j < tok0; ++j) s += (s_exp[j] == e);  // earlier tokens of the batch
                }
                if (s >= v.M) {
                    atomicOr(v.status, kStatusSlotRange);
                } else if (!kGroup) {
                    le = e;
                    row = s;
                    dst = v.recv_x + ((size_t)e * v.RM + s) * (size_t)v.row_bytes;
                } else {
                    const int dr = e / v.L;
                    le = e - dr * v.L;
                    if (v.s_active[dr]) {
                        // the owner's answer: first row of this rank's segment
                        const uint32_t b = wait_word(v.beg + e, v.seq, v.wait, dr);
                        if (b) {
                            row = (int)(b - 1) + s;
                            if (row >= v.RM) {
                                atomicOr(v.status, kStatusSlotRange);
                                row = -1;
                            } else if (dr == v.rank) {
                                dst = v.recv_x + ((size_t)le * v.RM + row) * (size_t)v.row_bytes;
                            } else {
                                const size_t r = (size_t)le * v.RM + row;
                                dst = v.s_peer[dr] + v.rx_off + r * (size_t)v.row_bytes;
                                meta = v.s_peer[dr] + v.meta_off + r * (size_t)v.meta_stride;
                            }
                        }
                    }
                }
            }
            v.rowmap[(size_t)t0 * K + tid] = row;
            s_dst[tid] = dst;
            if (kGroup) s_meta[tid] = meta, remote |= meta != nullptr;
            s_le[tid] = le;
            s_row[tid] = row;
        }
        __syncthreads();  // the destinations are in place, hist has been read
        if (kGroup) MCEP_TRACE(0, 7);  // the owners' answers are in, rows can go
        if (kCount && tid < ne && e >= 0) atomicAdd(&hist[e], 1);
        // A repeated expert in a token's list was sent once; combine still adds
        // that row once per listing (mooncake_ep_kernel.cu:734-742 reads the
        // (expert, token) slot for every k), so the repeat records the same row.
        if (tid < ne && e < 0 && raw >= 0)
            for (int j = tok0; j < tid; ++j)
                if (s_exp[j] == raw) v.rowmap[(size_t)t0 * K + tid] = s_row[j];

        if (warp >= items && t1 < v.T) ahead = load_item(t1, warp);
        for (int item = warp; item < items; item += nwarps) {
            const V32 cur = ahead;
            ahead = item + nwarps < items ? load_item(t0, item + nwarps) : load_item(t1, warp);
            const int tok = item / ntiles, tile = item - tok * ntiles;
            const int c = tile * 32 + lane, k0 = tok * K;
            const bool act = c < nchunks;
            if (kFP8) {
                float sinv;
                const uint4 q = quantize16(cur, sinv);
                float4 sc;
                if (kGroup) {
                    sc.x = __shfl_sync(kFull, sinv, 0);
                    sc.y = __shfl_sync(kFull, sinv, 8);
                    sc.z = __shfl_sync(kFull, sinv, 16);
                    sc.w = __shfl_sync(kFull, sinv, 24);
                }
#pragma unroll 4
                for (int k = k0; k < k0 + K; ++k) {
                    char* d = s_dst[k];
                    if (d == nullptr) continue;
                    if (act) st16(d + (size_t)c * 16, q);
                    char* m = kGroup ? s_meta[k] : nullptr;
                    if (m != nullptr) {
                        if (lane == 0)
                            st16(m + kMetaHeaderBytes + (size_t)tile * 16, *reinterpret_cast<uint4*>(&sc));
                    } else if (act && (lane & 7) == 0) {
                        v.recv_scales[((size_t)s_le[k] * S + (c >> 3)) * v.RM + s_row[k]] = sinv;
                    }
                }
            } else {
#pragma unroll 4
                for (int k = k0; k < k0 + K; ++k) {
                    char* d = s_dst[k];
                    if (d == nullptr || !act) continue;
                    st32(d + (size_t)c * 32, cur);
                }
            }
        }
        if (tid < ne && s_dst[tid] != nullptr) {
            const int t = t0 + tid / K;
            if (kGroup && s_meta[tid] != nullptr)
                st16(s_meta[tid], make_uint4((uint32_t)t, 0u, 0u, 0u));
            else
                v.recv_src_info[(size_t)s_le[tid] * v.RM + s_row[tid]] = t;
        }
        counted = t0 + nt;
        if (kCount || t1 < v.T) __syncthreads();  // done with the tables of this batch; hist is complete
        if (!kGroup && kCount && counted == v.T)
            for (int x = tid; x < v.E; x += nthr) {
                const int n = hist[x];
                v.recv_count[x] = n;
                v.layout_range[x] = n;  // begin 0 | count
            }
        t0 = t1;
    }
    return remote;
}

// =============================================================================
// single rank: dispatch writes the packed outputs directly
// =============================================================================
// Small batches (counts_in_send_kernel) of several tokens per block, in one launch: bound by latency,
// index load -> count -> row stores, one batch per block.
template <bool kFP8>
__global__ void __launch_bounds__(512, 2) ep_dispatch_send_direct_kernel(DirectDispatchParams p) {
    extern __shared__ int smem_i32[];  // [E]
    for (int i = threadIdx.x; i < p.E; i += blockDim.x) smem_i32[i] = 0;
    __syncthreads();
    pdl_wait();
    pdl_launch_dependents();
    SendView v = {};
    v.x = reinterpret_cast<const char*>(p.x), v.topk_idx = p.topk_idx;
    v.T = p.T, v.K = p.K, v.E = p.E, v.R = 1, v.M = p.M, v.H = p.H, v.rank = 0;
    v.L = p.E, v.RM = p.M, v.C = p.C, v.status = p.status;
    v.recv_x = reinterpret_cast<char*>(p.recv_x), v.recv_scales = p.recv_scales;
    v.recv_src_info = p.recv_src_info, v.row_bytes = p.H * (kFP8 ? 1 : 2);
    v.rowmap = p.rowmap, v.recv_count = p.recv_count, v.layout_range = p.layout_range;
    send_tokens<kFP8, false, true>(v, blockIdx.x, gridDim.x, smem_i32);
}

// The same with a token per block (one_token_per_block): what the kernel above spends between its
// three barriers - a table of all experts, atomics into it, the entries of the batch compared with
// one another - is here a comparison of every earlier token's choices with this token's own, a
// thread per token, and one barrier. The last block counts for the outputs. Device time per layer,
// table | comparison: 1 token of 14 KB in FP8 to 8 7.3 us | 6.0, 128 10.4 | 9.4, 256 of 8 KB 10.0 | 9.4; 128 of 4 KB in
// bf16 to 4 6.0 | 4.9.
template <bool kFP8, int KB>
__device__ __forceinline__ void send_one_token(const DirectDispatchParams& p, int (*s_part)[KB]) {
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int t = blockIdx.x, K = p.K, M = p.M, nchunks = p.H / 16, ntiles = (p.H + kTileChannels - 1) / kTileChannels;
    const bool vec = choices_in_pairs(p.topk_idx, K);
    auto load_tile = [&](int tile) {
        V32 r = {};
        const int c = tile * 32 + lane;
        if (c < nchunks) r = ld32_readonly(static_cast<const char*>(p.x) + ((size_t)t * p.H + (size_t)c * 16) * 2);
        return r;
    };
    V32 row = load_tile(warp);
    int e = -1, own[KB];
    if (lane < K) e = (int)ld_ro(p.topk_idx + (size_t)t * K + lane);
    load_choices<KB, false>(p.topk_idx, t, K, p.E, vec, own);
    int n = 0;  // lane k: earlier tokens of this warp's that chose the k-th expert
    for (int j0 = warp * 32; j0 < t; j0 += nthr) {
        unsigned same = 0;
        if (j0 + lane < t) {
            int other[KB];
            load_choices<KB, false>(p.topk_idx, j0 + lane, K, p.E, vec, other);
#pragma unroll
            for (int k = 0; k < KB; ++k) {
                bool hit = false;
#pragma unroll
                for (int a = 0; a < KB; ++a) hit |= other[a] == own[k];
                if (hit) same |= 1u << k;
            }
        }
#pragma unroll
        for (int k = 0; k < KB; ++k) {
            const unsigned hits = __ballot_sync(kFull, (same >> k) & 1u);
            if (lane == k) n += __popc(hits);
        }
    }
    const int counting = min(nwarps, (t + 31) / 32);  // warps that have counted
    if (t > 0) {
        if (lane < KB && warp < counting) s_part[warp][lane] = n;
        __syncthreads();
    }
    // (a repeated expert has the same row and gets the same bytes twice)
    int s = -1;
    if (lane < K && e >= 0 && e < p.E) {
        s = 0;
        for (int w = 0; w < counting; ++w) s += s_part[w][lane];
        if (s >= M) {
            atomicOr(p.status, kStatusSlotRange);
            s = -1;
        }
    }
    const int to = s >= 0 ? e * M + s : -1;  // (31 bits: the launcher)
    if (warp == 0 && lane < K) {
        p.rowmap[(size_t)t * K + lane] = s;
        if (s >= 0) p.recv_src_info[to] = t;
    }
    char* out = static_cast<char*>(p.recv_x);
    const int S = p.H / 128, at = s >= 0 ? e * S * M + s : 0;
    for (int tile = warp; tile < ntiles; tile += nwarps) {
        if (tile != warp) row = load_tile(tile);
        const int c = tile * 32 + lane;
        if (kFP8) {
            float sinv;
            const uint4 q = quantize16(row, sinv);
#pragma unroll 4
            for (int k = 0; k < K; ++k) {
                const int r = __shfl_sync(kFull, to, k), sr = __shfl_sync(kFull, at, k);
                if (r < 0 || c >= nchunks) continue;
                st16(out + (size_t)r * p.H + (size_t)c * 16, q);
                if ((lane & 7) == 0) p.recv_scales[(size_t)sr + (size_t)(c >> 3) * M] = sinv;
            }
        } else {
#pragma unroll 4
            for (int k = 0; k < K; ++k) {
                const int r = __shfl_sync(kFull, to, k);
                if (r >= 0 && c < nchunks) st32(out + (size_t)r * p.H * 2 + (size_t)c * 32, row);
            }
        }
    }
}

template <bool kFP8, int KB>
__global__ void __launch_bounds__(512, 2) ep_dispatch_one_token_kernel(DirectDispatchParams p) {
    extern __shared__ int smem_i32[];  // [E]
    __shared__ int s_part[16][KB];
    const bool counts = (int)blockIdx.x == p.T;
    if (counts) {
        for (int i = threadIdx.x; i < p.E; i += blockDim.x) smem_i32[i] = 0;
        __syncthreads();
    }
    pdl_wait();
    pdl_launch_dependents();
    if (!counts) return send_one_token<kFP8, KB>(p, s_part);
    count_tokens_of<KB, 1, false>(p.topk_idx, 0, p.T, p.K, p.E, choices_in_pairs(p.topk_idx, p.K), smem_i32);
    __syncthreads();
    for (int x = threadIdx.x; x < p.E; x += blockDim.x) {
        const int n = smem_i32[x];
        p.recv_count[x] = n;
        p.layout_range[x] = n;  // begin 0 | count
    }
}

// The counts of a batch whose layout is there as bits; whole block. The first block does it once
// its own rows are out and the others hide it; the last one, an expert per thread ahead of its
// rows, was waited for (the layer: 885 rows of 11 KB to 2 of 512 14.6 us, now 13.4; 3539 of 256
// bytes in FP8 to 8 of 2048 28.8, now 23.7; a block of its own ahead of the rows costs 0.4 at few
// choices, 1000 rows of 14 KB to 2 15.4 against 14.7). Not inlined: what it keeps in registers is
// not taken from the rows' warps (inlined, 16 bytes are spilled: 1000 rows to 4 22.4, now 21.6).
__device__ __noinline__ void write_counts(RouteBits bits, int E, int32_t* recv_count, int64_t* layout_range) {
    bits_totals<4>(bits, E, [&](int x, int n) {
        recv_count[x] = n;
        layout_range[x] = n;  // begin 0 | count
    });
}

// Single rank, behind a layout kernel: a warp owns one tile of one token and needs no
// other: lane k finds the token's k-th row, the tile goes to each. Nothing is shared and
// nobody waits at a barrier. The hardware hands the blocks out in ascending order as SMs come
// free, which keeps an expert's rows together in time and in HBM pages (4096 rows of 14 KB to 8
// with a block per token: 85 us, with one resident wave striding over the tokens, where the
// slowest SM decides, 98). Blocks are small because it is the turnover of independent
// warps that hides the chain index -> bits -> stores: with a block per token that met at
// three barriers a block lived 6 us, 2001 of them behind one another were bound by that
// and not by HBM (2001 rows of 8 KB to 8 in FP8, the layer 49.5 us, now 45.5; 2000 of 4 KB
// in bf16 25.6, now 22.6; 4000 of 1 KB 19.8, now 14.9).
// How many warps and tiles of each (us per layer; launch_direct_dispatch chooses): many warps per SM where the
// time is that of the loads and of quantising (FP8 to 4, 2048 rows of 14 KB: 46.1 with 42
// warps, 48.1 with 32; bf16 to 8, 1500 rows of 8 KB: 42.0 | 42.9); with few copies per row
// and long rows in FP8 two tiles per warp (4096 rows of 14 KB to 3: 68.5, one tile 73.0;
// before 72.7); fewer warps for large bf16 outputs, as the rows that are written at a time
// then lie closer together in HBM (4096 rows of 14 KB to 8: 172.9 with 32 warps, 174.7 with
// 42, 176.1 with 48; 174.6 before). The blocks of a row are neighbours in the grid (parts of
// a row one after the other over all rows: 175.9).
template <bool kFP8, int kTiles, int kWarps, int kBlocks>
__global__ void __launch_bounds__(kWarps * 32, kBlocks)
    ep_dispatch_rows_kernel(DirectDispatchParams p) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = warp / p.warps_per_row;  // which token of the block
    const int group = blockIdx.x / p.parts, part = blockIdx.x - group * p.parts;
    const int tile = (warp - sub * p.warps_per_row + part * p.warps_per_row) * kTiles;  // the first
    const int t = group * p.tokens_per_block + sub, nchunks = p.H / 16;
    const int K = p.K, M = p.M;
    const bool mine = t < p.T && lane < K;
    pdl_launch_dependents();
    // (the rows and the index matrix are complete: the layout kernel has waited for them)
    V32 row[kTiles];
    int e = -1;
#pragma unroll
    for (int u = 0; u < kTiles; ++u) {
        const int c = (tile + u) * 32 + lane;
        row[u] = V32{};
        if (t < p.T && c < nchunks)
            row[u] = ld32_readonly(static_cast<const char*>(p.x) + ((size_t)t * p.H + (size_t)c * 16) * 2, p.x_last);
    }
    if (mine) e = (int)ld_ro(p.topk_idx + (size_t)t * K + lane);
    pdl_wait();
    // (a repeated expert has the same row and gets the same bytes twice)
    int s = -1;
    if (p.bits.words != nullptr) {
        if (e >= 0 && e < p.E) s = bits_before(p.bits, e, t);
    } else {
        if (mine) s = ld_ro(p.slot + (size_t)t * K + lane);
        for (int k = 0; k < K; ++k) {  // (that layout kernel leaves a repeat without a position)
            const int ek = __shfl_sync(kFull, e, k), sk = __shfl_sync(kFull, s, k);
            if (s < 0 && e >= 0 && ek == e) s = sk;
        }
    }
    if (s >= M) {
        atomicOr(p.status, kStatusSlotRange);
        s = -1;
    }
    // (31 bits: mcep_dispatch has larger tensors filled by the kernel that counts. 64 bits in the
    // shuffles: 2756 rows of 256 bytes in FP8 to 8 11.5 us, 11.0 so)
    const int to = s >= 0 ? e * M + s : -1;
    if (tile == 0 && mine) {
        p.rowmap[(size_t)t * K + lane] = s;
        if (s >= 0) p.recv_src_info[to] = t;
    }
    char* out = static_cast<char*>(p.recv_x);
    if (kFP8) {
        const int S = p.H / 128, at = s >= 0 ? e * S * M + s : 0;
        float sinv[kTiles];
        uint4 q[kTiles];
#pragma unroll
        for (int u = 0; u < kTiles; ++u) q[u] = quantize16(row[u], sinv[u]);
#pragma unroll 4
        for (int k = 0; k < K; ++k) {
            const int r = __shfl_sync(kFull, to, k), sr = __shfl_sync(kFull, at, k);
            if (r < 0) continue;
#pragma unroll
            for (int u = 0; u < kTiles; ++u) {
                const int c = (tile + u) * 32 + lane;
                if (c >= nchunks) continue;
                st16(out + (size_t)r * p.H + (size_t)c * 16, q[u]);
                if ((lane & 7) == 0) p.recv_scales[(size_t)sr + (size_t)(c >> 3) * M] = sinv[u];
            }
        }
    } else {
#pragma unroll 4
        for (int k = 0; k < K; ++k) {
            const int r = __shfl_sync(kFull, to, k);
            if (r < 0) continue;
#pragma unroll
            for (int u = 0; u < kTiles; ++u) {
                const int c = (tile + u) * 32 + lane;
                if (c < nchunks) st32(out + (size_t)r * p.H * 2 + (size_t)c * 32, row[u]);
            }
        }
    }
    if (p.bits.words != nullptr && blockIdx.x == 0) write_counts(p.bits, p.E, p.recv_count, p.layout_range);
}

// Single rank: rowmap[t][k] = packed row of (token t, expert topk[t][k]) as the
// handle records it.
__global__ void __launch_bounds__(256) ep_combine_invert_kernel(CombineInvertParams p) {
    const int RM = p.R * p.M;
    const long long total = (long long)p.L * p.M;
    pdl_wait();
    pdl_launch_dependents();
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        const int le = (int)(i / p.M), j = (int)(i - (long long)le * p.M);
        const long long lr = ld_ro(p.layout_range + le * p.R + p.rank);
        const int cnt = (int)(lr & 0xffffffffll);
        if (j >= cnt) continue;
        const int row = (int)(lr >> 32) + j;
        if (row >= RM) {
            atomicOr(p.status, kStatusSlotRange);
            continue;
        }
        const int t = ld_ro(p.src_info + (size_t)le * RM + row);
        if (t < 0 || t >= p.T) {
            atomicOr(p.status, kStatusBadSource);
            continue;
        }
        const int e = p.rank * p.L + le;
        for (int k = 0; k < p.K; ++k)
            if ((int)ld_ro(p.topk_idx + (size_t)t * p.K + k) == e) p.rowmap[(size_t)t * p.K + k] = row;
    }
}

// =============================================================================
// weighted top-k reduction
// =============================================================================
// One block per token, one warp per 512-channel tile; each lane owns 16
// channels: up to K 32-byte loads in flight, fp32 FMA accumulation in k order,
// one bf16 rounding, one 32-byte store (mooncake_ep_kernel.cu:715-752).
// kDepth rows are requested before the first of them is used. s_ptr has kMaxTopk
// entries, null where nothing is to be added. hold: the kernel ahead is waited for before a store.
template <int kDepth, bool kReadOnly, bool kLast>
__device__ __forceinline__ void reduce_rows(const char* const* s_ptr, const float* s_w, int K,
                                            int H, void* out_row, bool hold = false) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int nchunks = H / 16;
    const int ntiles = (H + kTileChannels - 1) / kTileChannels;
    for (int tile = warp; tile < ntiles; tile += nwarps) {
        const int c = tile * 32 + lane;
        if (c >= nchunks) continue;
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        for (int k0 = 0; k0 < K; k0 += kDepth) {
            V32 v[kDepth];
#pragma unroll
            for (int b = 0; b < kDepth; ++b) {
                const char* rp = s_ptr[k0 + b];
                if (rp != nullptr)
                    v[b] = kReadOnly ? ld32_readonly(rp + (size_t)c * 32)
                                     : ld32_coherent(rp + (size_t)c * 32, kLast);
            }
#pragma unroll
            for (int b = 0; b < kDepth; ++b) {
                if (s_ptr[k0 + b] == nullptr) continue;
                const float wk = s_w[k0 + b];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    acc[2 * i] = fmaf(bf16lo(v[b].w[i]), wk, acc[2 * i]);
                    acc[2 * i + 1] = fmaf(bf16hi(v[b].w[i]), wk, acc[2 * i + 1]);
                }
            }
        }
        if (hold) pdl_wait();
        st32(reinterpret_cast<char*>(out_row) + (size_t)c * 32, pack_bf16x16(acc));
    }
}

// Single rank, rows known (p.rowmap). No barrier and no shared memory: a warp owns
// one 512-channel tile of one row of every block's group of tokens, so its loads
// overlap the sums of the others; the next row's place and weights are requested
// before this row's data is used. Bound by HBM reads (4096 tokens, hidden 7168,
// top-8: 470 MB of rows in 90 us, with the last dirty lines of whatever wrote them
// still leaving L2; 80 us on rows that have been in HBM for a while). The loop runs
// over groups, alike for all warps of a block: with a loop that the compiler has to
// take for divergent (a token index that depends on the warp, a loop over tiles) the
// shuffles cost so many registers that loaded rows spilled, 108 us - so tiles beyond
// a block's warps are the grid's y. A barrier per token (tokens handed out by a
// counter) took 111 us.
// kAbs: rowmap holds rows of the whole tensor and every weight is 1 (elastic calls).
constexpr int kReduceWarps = 16;  // 64 registers a thread with two blocks per SM: nothing spills in the kernel below

template <int kDepth, bool kAbs, int kBlocks, bool kLast>
__global__ void __launch_bounds__(kReduceWarps * 32, kBlocks) ep_combine_rows_kernel(DirectCombineParams p) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = warp / p.tiles_per_block;  // which token of the group
    const int c = ((warp - sub * p.tiles_per_block + blockIdx.y * p.tiles_per_block) * 32) + lane;
    const bool act = c < p.H / 16;
    pdl_wait();
    pdl_launch_dependents();
    const size_t row_bytes = (size_t)p.H * 2;
    const char* x = reinterpret_cast<const char*>(p.x) + (size_t)c * 32;
    char* out = reinterpret_cast<char*>(p.combined_x) + (size_t)c * 32;
    // a block's groups: every grid-th one, or (p.span) a run of tokens, the last run first
    // where the runs are many (p.span < 0)
    const int run = p.span < 0 ? -p.span : p.span;
    const int step = (run ? 1 : gridDim.x) * p.tokens_per_block;
    const int first = (p.span < 0 ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * (run ? run : p.tokens_per_block);
    const int end = run ? min(p.T, first + run) : p.T;

    // rows that there are (kAbs: a dispatch may have kept some beyond the caller's tensor)
    const unsigned rows = kAbs ? (unsigned)p.M : 1u << 31;
    int next_row = -1, next_e = -1;
    float next_w = 1.f;
    bool on = lane < p.K;
    auto request = [&](int tok) {
        if (on && tok < end) {
            const size_t at = (size_t)tok * p.K + lane;
            next_row = ld_ro(p.rowmap + at);
            if (!kAbs) next_e = (int)ld_ro(p.topk_idx + at), next_w = ld_ro(p.topk_weights + at);
        } else {
            next_row = -1;
        }
    };
    request(first + sub);
    // (the mask is asked for together with the first rows' places, not ahead of them: 128 tokens
    // of 14 KB 3.9 -> 3.7 us)
    if (ld_volatile_s32(p.active_ranks) == 0) on = false, next_row = -1;
    for (int t0 = first; t0 < end; t0 += step) {
        int row = next_row;
        if (!kAbs) row = (next_e >= 0 && next_e < p.E && row >= 0 && row < p.M) ? next_e * p.M + row : -1;
        const float w = next_w;
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        for (int k0 = 0; k0 < p.K; k0 += kDepth) {
            V32 v[kDepth];
#pragma unroll
            for (int b = 0; b < kDepth; ++b) {
                const int r = __shfl_sync(kFull, row, k0 + b);
                if ((unsigned)r < rows && act) v[b] = ld32_readonly(x + (size_t)r * row_bytes, kLast);
            }
            if (k0 == 0) request(t0 + step + sub);
#pragma unroll
            for (int b = 0; b < kDepth; ++b) {
                const int r = __shfl_sync(kFull, row, k0 + b);
                const float wk = kAbs ? 1.f : __shfl_sync(kFull, w, k0 + b);
                if ((unsigned)r < rows) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        acc[2 * i] = fmaf(bf16lo(v[b].w[i]), wk, acc[2 * i]);
                        acc[2 * i + 1] = fmaf(bf16hi(v[b].w[i]), wk, acc[2 * i + 1]);
                    }
                }
            }
        }
        if (act && t0 + sub < end) st32(out + (size_t)(t0 + sub) * row_bytes, pack_bf16x16(acc));
    }
}

// One row per token (top-1, and every flat elastic combine of a single rank): a gather.
// The kernel above would have a single load per lane in flight; here a warp requests
// up to four tiles of its block's `tokens_per_block` rows before it uses the first.
template <bool kAbs, bool kLast>
__global__ void __launch_bounds__(512, 2) ep_combine_one_row_kernel(DirectCombineParams p) {
    constexpr int kAhead = 4, kMost = 16;
    __shared__ int s_row[kMost];
    __shared__ float s_w[kMost];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    const int nchunks = p.H / 16, ntiles = (p.H + kTileChannels - 1) / kTileChannels;
    const int t0 = blockIdx.x * p.tokens_per_block, nt = min(p.tokens_per_block, p.T - t0), items = nt * ntiles;
    pdl_wait();
    pdl_launch_dependents();
    if (tid < nt) {
        const bool on = ld_volatile_s32(p.active_ranks) != 0;
        int row = ld_ro(p.rowmap + t0 + tid);
        float w = 1.f;
        if (!kAbs) {
            const int e = (int)ld_ro(p.topk_idx + t0 + tid);
            w = ld_ro(p.topk_weights + t0 + tid);
            row = (e >= 0 && e < p.E && row >= 0 && row < p.M) ? e * p.M + row : -1;
        } else if (row >= p.M) {
            row = -1;
        }
        s_row[tid] = on ? row : -1;
        s_w[tid] = w;
    }
    __syncthreads();
    const size_t row_bytes = (size_t)p.H * 2;
    for (int i0 = warp; i0 < items; i0 += nwarps * kAhead) {
        V32 v[kAhead];
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int item = i0 + u * nwarps, tok = item / ntiles, c = (item - tok * ntiles) * 32 + lane;
            const int r = item < items && c < nchunks ? s_row[tok] : -1;
            const char* x = reinterpret_cast<const char*>(p.x) + (size_t)c * 32;
            if (r >= 0) v[u] = ld32_readonly(x + (size_t)r * row_bytes, kLast);
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int item = i0 + u * nwarps, tok = item / ntiles, c = (item - tok * ntiles) * 32 + lane;
            if (item >= items || c >= nchunks) continue;
            float acc[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = 0.f;
            if (s_row[tok] >= 0) {
                const float w = kAbs ? 1.f : s_w[tok];
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    acc[2 * i] = fmaf(bf16lo(v[u].w[i]), w, 0.f);
                    acc[2 * i + 1] = fmaf(bf16hi(v[u].w[i]), w, 0.f);
                }
            }
            st32(reinterpret_cast<char*>(p.combined_x) + (size_t)(t0 + tok) * row_bytes + (size_t)c * 32, pack_bf16x16(acc));
        }
    }
}

// Small batches whose rows are not recorded (a handle older than the last two
// calls, or a copy of one): no separate inversion pass. Warp k looks the token up
// in the handle itself - the segment of expert topk[t][k] - 32 entries of src_info
// at a time.
__global__ void __launch_bounds__(512) ep_combine_search_kernel(DirectCombineParams p) {
    __shared__ const char* s_ptr[kMaxTopk];
    __shared__ float s_w[kMaxTopk];
    __shared__ int s_row[kMaxTopk];
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    pdl_wait();
    pdl_launch_dependents();
    for (int t = blockIdx.x; t < p.T; t += gridDim.x) {
        int e = -1;
        float w = 0.f;
        if (tid < p.K) {
            e = (int)ld_ro(p.topk_idx + (size_t)t * p.K + tid);
            w = ld_ro(p.topk_weights + (size_t)t * p.K + tid);
        }
        for (int k = warp; k < p.K; k += nwarps) {
            const int ek = (int)ld_ro(p.topk_idx + (size_t)t * p.K + k);
            int row = -1;
            if (ek >= 0 && ek < p.E) {
                const long long lr = ld_ro(p.layout_range + ek);
                const int cnt = (int)(lr & 0xffffffffll), begin = (int)(lr >> 32);
                for (int j0 = 0; j0 < cnt; j0 += 32) {
                    const int j = begin + j0 + lane;
                    const bool hit = j0 + lane < cnt && j < p.M &&
                                     ld_ro(p.src_info + (size_t)ek * p.M + j) == t;
                    const unsigned m = __ballot_sync(kFull, hit);
                    if (m) {
                        row = begin + j0 + __ffs(m) - 1;
                        break;
                    }
                }
            }
            if (lane == 0) s_row[k] = row;
        }
        __syncthreads();  // s_row is in place; the previous token's rows are done with s_ptr
        if (tid < kMaxTopk) {
            const char* ptr = nullptr;
            const int r = tid < p.K ? s_row[tid] : -1;
            if (e >= 0 && e < p.E && ld_volatile_s32(p.active_ranks) && r >= 0 && r < p.M)
                ptr = reinterpret_cast<const char*>(p.x) + ((size_t)e * p.M + r) * p.H * 2;
            s_ptr[tid] = ptr;
            s_w[tid] = w;
        }
        __syncthreads();
        reduce_rows<8, true, false>(s_ptr, s_w, p.K, p.H,
                             reinterpret_cast<char*>(p.combined_x) + (size_t)t * p.H * 2);
    }
}

// =============================================================================
// groups: dispatch
// =============================================================================
__device__ __forceinline__ void load_peer_tables(void* const* peer_base, const int32_t* active_ranks,
                                                 int R, int32_t* status, char** s_peer,
                                                 int* s_active) {
    // (the last threads of the block: in a small batch's control block the others count)
    for (int r = blockDim.x - 1 - threadIdx.x; r < R; r += blockDim.x) {
        char* pb = reinterpret_cast<char*>(peer_base[r]);
        int a = ld_volatile_s32(active_ranks + r);
        if (a && pb == nullptr) {  // marked active but never mapped: leave it alone
            atomicOr(status, kStatusNoPeer);
            a = 0;
        }
        s_peer[r] = pb;
        s_active[r] = a;
    }
}

// The control block (block 0 of the send kernel).
//  1. announce: count of this rank's tokens per expert -> the expert's owner;
//  2. collect: for this rank's own experts, the counts of every active source
//     (bounded wait; a source that does not answer is marked inactive and
//     counts as zero);
//  3. fix the receive layout (source-rank order), write `layout_range` and
//     `recv_count`, leave the verdicts for the receive duty, and answer every
//     source with the first row of its segment in each of this rank's experts.
__device__ __forceinline__ void dispatch_control(const GroupDispatchParams& p, int* smem_i32,
                                                 char* const* s_peer, const int* s_active) {
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int L = p.E / p.R, n = L * p.R;
    const int* hist = smem_i32;   // [E] counts of this rank's tokens
    int* s_cnt = smem_i32 + p.E;  // [L*R]
    MCEP_TRACE(0, 1);
    for (int x = tid; x < p.E; x += nthr) {
        const int dr = x / L;
        if (!s_active[dr] || dr == p.rank) continue;
        const int c = hist[x];
        uint64_t* wd = reinterpret_cast<uint64_t*>(s_peer[dr] + p.w.cnt_off) + (p.rank * L + (x - dr * L));
        st_relaxed_sys(wd, ((uint64_t)p.seq << 32) | (uint32_t)(c + 1));
    }
    MCEP_TRACE(0, 2);  // counts announced
    const uint64_t* my_cnt = reinterpret_cast<const uint64_t*>(p.local_base + p.w.cnt_off);
    for (int i = tid; i < n; i += nthr) {
        const int le = i / p.R, src = i - le * p.R;
        int c = -1;  // -1: nothing will come from this source (inactive, or given up on)
        if (s_active[src]) {
            if (src == p.rank) {
                c = hist[src * L + le];
            } else {
                const uint32_t v = wait_word(my_cnt + src * L + le, p.seq, p.wait, src);
                c = v ? (int)v - 1 : -1;
            }
            if (c > p.M) {
                atomicOr(p.wait.status, kStatusSlotRange);
                c = 0;
            }
        }
        s_cnt[i] = c;
    }
    __syncthreads();
    MCEP_TRACE(0, 3);  // every source's counts are in
    // Every thread fixes its own (expert, source) entry: the rows of the lower
    // sources come first. The answer goes out at once; the outputs follow.
    for (int i = tid; i < n; i += nthr) {
        const int le = i / p.R, src = i - le * p.R;
        int begin = 0;
        for (int s2 = 0; s2 < src; ++s2) begin += max(s_cnt[le * p.R + s2], 0);
        // a source that is inactive, or went silent while its counts were
        // awaited, counts as zero and gets no answer
        const bool answered = s_cnt[i] >= 0;
        const int c = max(s_cnt[i], 0);
        if (answered) {
            uint64_t* wd = reinterpret_cast<uint64_t*>(s_peer[src] + p.w.beg_off) + (p.rank * L + le);
            st_relaxed_sys(wd, ((uint64_t)p.seq << 32) | (uint32_t)(begin + 1));
        }
        *reinterpret_cast<volatile uint64_t*>(p.res_cnt + i) = ((uint64_t)p.seq << 32) | (uint32_t)(c + 1);
        p.layout_range[i] = c ? (((int64_t)begin << 32) | (int64_t)c) : 0;
        if (src == p.R - 1) p.recv_count[le] = begin + c;
    }
    MCEP_TRACE(0, 4);  // answers are out
}

// Receive duty of dispatch, shared by `np` participants (blocks): rows that
// peers stored into this rank's receive area are complete once the source's
// payload word has arrived; their side messages are then moved into the
// caller's `src_info` and transposed `scales`, and - when the caller's recv_x
// is not the in-place tensor - the rows themselves are copied out.
// (Rows of experts this rank sent to itself need nothing: the sender wrote the
// final tensors.)
constexpr int kRowWarps = 8;

// kAlone: in a kernel of its own, behind the control block's.
template <bool kFP8, bool kAlone>
__device__ __forceinline__ void dispatch_recv_duty(const GroupDispatchParams& p, int j, int np,
                                                   int* smem_i32) {
    const int L = p.E / p.R, n = L * p.R;
    int* pre = smem_i32;          // [n + 1] rows to process per (expert, source), then prefix
    int* beg = smem_i32 + n + 1;  // [n] first row of each (expert, source)
    __shared__ int s_wt[32];
    __shared__ int s_ok[kMaxRanks];
    __shared__ int s_tot[kMaxRanks];
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int RM = p.R * p.M;
    const int nchunks = p.H / 16;
    const int ntiles = (p.H + kTileChannels - 1) / kTileChannels;
    const int S = p.H / 128;
    for (int r = tid; r < p.R; r += nthr) s_tot[r] = 0;
    __syncthreads();
    // the control block's verdicts: what every source sends to every local expert
    bool from_peers = false;
    for (int i = tid; i < n; i += nthr) {
        const uint32_t v = kAlone ? local_word_of_kernel_ahead(p.res_cnt + i, p.seq, scaled(p.wait, 2))
                                  : wait_local_word(p.res_cnt + i, p.seq, scaled(p.wait, 2));
        const int c = v ? (int)v - 1 : 0;
        pre[i] = c;
        if (c) atomicAdd(&s_tot[i % p.R], c);
        from_peers |= c != 0 && i % p.R != p.rank;
    }
    if (!__syncthreads_or(from_peers ? 1 : 0)) return;  // only rows this rank sent to itself
    for (int le = tid; le < L; le += nthr) {
        int run = 0;
        for (int src = 0; src < p.R; ++src) {
            beg[le * p.R + src] = run;
            run += pre[le * p.R + src];
        }
    }
    __syncthreads();
    // rows this rank sent to itself need nothing; all of the above, and the
    // prefix below, is ready before the payload words are even looked at
    for (int i = tid; i < n; i += nthr)
        if (i % p.R == p.rank) pre[i] = 0;
    __syncthreads();
    block_exclusive_scan(pre, n, s_wt);
    // a peer's rows count once its payload word is here (one verdict per source
    // for all participants)
    for (int r = tid; r < p.R; r += nthr) {
        int ok = 0;
        if (r != p.rank && s_tot[r] > 0) {
            const uint64_t* flags = reinterpret_cast<const uint64_t*>(p.local_base + p.w.dflag_off);
            ok = resolve_flag(flags, p.res_dflag, r, p.seq, scaled(p.wait, 3), r,
                              np <= 80 || (j & 7) == (r & 7)) != 0;
        }
        s_ok[r] = ok;
    }
    __syncthreads();
    MCEP_TRACE(1, 1);  // every payload word has a verdict
    const int total = pre[n];
    const char* rx = p.local_base + p.rx_off;
    const char* mt = p.local_base + p.meta_off;
    // rows are dealt to the participants one at a time (warp w of participant j
    // takes row w * np + j, ...): a batch with fewer rows than there are warps
    // still spreads over all of them
    for (int g = warp * np + j; g < total; g += np * nwarps) {
        const int i = find_segment(pre, n, g);
        const int le = i / p.R;
        if (!s_ok[i - le * p.R]) continue;  // a source that was given up on
        const int row = beg[i] + (g - pre[i]);
        if (row >= RM) {
            if (lane == 0) atomicOr(p.wait.status, kStatusSlotRange);
            continue;
        }
        const size_t r = (size_t)le * RM + row;
        const char* meta = mt + r * (size_t)p.meta_stride;
        // one round trip: the token index and 16 bytes (four scales) per lane are
        // requested together, then scattered into the transposed scales
        const int tok = lane == 31 ? ld_s32_coherent(meta) : 0;
        if (kFP8) {
            for (int q0 = 0; q0 < ntiles; q0 += 32) {
                const int q = q0 + lane;
                if (q >= ntiles) continue;
                const uint4 sc = ld16_coherent(meta + kMetaHeaderBytes + (size_t)q * 16);
                const uint32_t w4[4] = {sc.x, sc.y, sc.z, sc.w};
#pragma unroll
                for (int u = 0; u < 4; ++u)
                    if (4 * q + u < S)
                        p.recv_scales[((size_t)le * S + 4 * q + u) * RM + row] = __uint_as_float(w4[u]);
            }
        }
        if (lane == 31) p.recv_src_info[r] = tok;
        if (!p.copy_rows) continue;
        const char* src = rx + r * (size_t)p.row_bytes;
        char* out = reinterpret_cast<char*>(p.recv_x) + r * (size_t)p.row_bytes;
        if (kFP8) {
            constexpr int kB = 8;  // 8 x 16 B per lane in flight
            for (int t0 = 0; t0 < ntiles; t0 += kB) {
                uint4 v[kB];
#pragma unroll
                for (int b = 0; b < kB; ++b) {
                    const int c = (t0 + b) * 32 + lane;
                    if (t0 + b < ntiles && c < nchunks) v[b] = ld16_coherent(src + (size_t)c * 16);
                }
#pragma unroll
                for (int b = 0; b < kB; ++b) {
                    const int c = (t0 + b) * 32 + lane;
                    if (t0 + b < ntiles && c < nchunks) st16(out + (size_t)c * 16, v[b]);
                }
            }
        } else {
            constexpr int kB = 4;  // 4 x 32 B per lane in flight
            for (int t0 = 0; t0 < ntiles; t0 += kB) {
                V32 v[kB];
#pragma unroll
                for (int b = 0; b < kB; ++b) {
                    const int c = (t0 + b) * 32 + lane;
                    if (t0 + b < ntiles && c < nchunks) v[b] = ld32_coherent(src + (size_t)c * 32);
                }
#pragma unroll
                for (int b = 0; b < kB; ++b) {
                    const int c = (t0 + b) * 32 + lane;
                    if (t0 + b < ntiles && c < nchunks) st32(out + (size_t)c * 32, v[b]);
                }
            }
        }
    }
    MCEP_TRACE(1, 2);
}

// Participants of the receive duty inside the one-launch kernel: the control
// block and the last sender blocks to finish (at most this many).
constexpr int kRecvHelpers = 64;

// kPhases: 1 = control + send; 3 = control + send + receive duty (one launch).
// kCount: smem_i32 begins with E zeros.
// `bid` of `nblocks`: the block's place in its rank's share of the grid (the
// whole grid, except for in-process groups where one launch carries all ranks).
template <bool kFP8, bool kCount, int kPhases>
__device__ __forceinline__ void dispatch_body(const GroupDispatchParams& p, int bid, int nblocks,
                                              int* smem_i32) {
    __shared__ char* s_peer[kMaxRanks];
    __shared__ int s_active[kMaxRanks];
    __shared__ int s_ticket;
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int nsend = nblocks - 1;
    const int nh = nsend < kRecvHelpers ? nsend : kRecvHelpers;
    MCEP_TRACE(0, 0);
    if (bid == 0) {  // the counts do not wait for the peer tables (0.8 us)
        if (!kCount) pdl_wait();
        if (kCount) {
            count_tokens<2>(p.topk_idx, 0, p.T, p.K, p.E, choices_in_pairs(p.topk_idx, p.K), smem_i32);
        } else if (p.bits.words != nullptr) {
            bits_totals<4>(p.bits, p.E, [&](int i, int n) { smem_i32[i] = n; });
        } else {
            for (int i = tid; i < p.E; i += nthr) smem_i32[i] = ld_ro(p.count + i);
        }
    }
    load_peer_tables(p.peer_base, p.wait.active_ranks, p.R, p.wait.status, s_peer, s_active);

    if (bid == 0) {
        __syncthreads();
        dispatch_control(p, smem_i32, s_peer, s_active);
        if (kPhases == 3) {
            __syncthreads();
            dispatch_recv_duty<kFP8, false>(p, nh, nh + 1, smem_i32);
        }
        return;
    }

    const int sid = bid - 1;
    __syncthreads();  // the tables above are in place
    SendView v = {};
    v.x = reinterpret_cast<const char*>(p.x), v.topk_idx = p.topk_idx, v.slot = p.slot, v.bits = p.bits;
    v.T = p.T, v.K = p.K, v.E = p.E, v.R = p.R, v.M = p.M, v.H = p.H, v.rank = p.rank;
    v.L = p.E / p.R, v.RM = p.R * p.M, v.C = p.C, v.status = p.wait.status;
    v.recv_x = reinterpret_cast<char*>(p.recv_x), v.recv_scales = p.recv_scales;
    v.recv_src_info = p.recv_src_info, v.row_bytes = p.row_bytes;
    v.beg = reinterpret_cast<const uint64_t*>(p.local_base + p.w.beg_off);
    v.seq = p.seq, v.wait = scaled(p.wait, 2), v.rx_off = p.rx_off, v.meta_off = p.meta_off;
    v.meta_stride = p.meta_stride, v.rowmap = p.rowmap, v.s_peer = s_peer, v.s_active = s_active;
    v.x_last = p.x_last;
    const bool remote = send_tokens<kFP8, true, kCount>(v, sid, nsend, smem_i32);
    MCEP_TRACE(0, 5);  // all rows of this block are issued

    // Completion. Rows are not fenced one by one: a block that stored something in a
    // peer's memory issues ONE system-scope fence for all of it (2 - 4 us, even when
    // idle), then takes a ticket. Whoever takes the last ticket has, through the
    // counter, observed every such fence - all of this rank's rows are performed
    // system-wide - and tells every peer with one word. Rows of experts this rank
    // owns are nobody else's to read: the kernel's end orders them.
    const bool any_remote = __syncthreads_or(remote ? 1 : 0) != 0;
    if (tid == 0) {
        if (any_remote) __threadfence_system();
        s_ticket = (int)atomicAdd(p.ticket, 1u);
    }
    __syncthreads();
    MCEP_TRACE(0, 6);  // the fence has returned
    const int ticket = s_ticket;
    if (ticket == nsend - 1) {
        if (tid == 0) *p.ticket = 0;
        __threadfence();
        for (int r = tid; r < p.R; r += nthr) {
            if (r == p.rank || !s_active[r] || !ld_volatile_s32(p.wait.active_ranks + r)) continue;
            uint64_t* f = reinterpret_cast<uint64_t*>(s_peer[r] + p.w.dflag_off) + p.rank;
            st_relaxed_sys(f, ((uint64_t)p.seq << 32) | 1u);
        }
    }
    if (kPhases == 3 && ticket >= nsend - nh) {
        __syncthreads();
        dispatch_recv_duty<kFP8, false>(p, ticket - (nsend - nh), nh + 1, smem_i32);
    }
}

// Graph mode: a captured launch is replayed with the arguments it was captured
// with, so the call's sequence number cannot be one of them; it is read from the
// device word the host named (stable until the call's last kernel has finished:
// the word of the other parity belongs to the other call that may be in flight).
template <typename Params>
__device__ __forceinline__ void resolve_seq(Params& p) {
    if (p.seq_ptr != nullptr) p.seq = *reinterpret_cast<const volatile uint32_t*>(p.seq_ptr);
}

__global__ void ep_advance_seq_kernel(uint32_t* word) { *word += 2; }

// One thread per rank: tell that rank "I am here", then wait until it has said
// the same. Bounded: a rank that never comes raises the hard-timeout status bit
// and the others go on.
__global__ void __launch_bounds__(kMaxRanks) ep_barrier_kernel(BarrierParams p) {
    const int r = threadIdx.x;
    if (r >= p.R || r == p.rank) return;
    if (p.active_ranks != nullptr && !ld_volatile_s32(p.active_ranks + r)) return;
    char* peer = reinterpret_cast<char*>(p.peer_base[r]);
    if (peer == nullptr) return;
    st_release_sys(reinterpret_cast<uint64_t*>(peer + p.bar_off) + p.rank, (uint64_t)p.epoch);
    const uint64_t* mine = reinterpret_cast<const uint64_t*>(p.local_base + p.bar_off) + r;
    const uint64_t start = globaltimer_ns();
    // (a peer that has left this barrier may already have announced the next one)
    while ((int32_t)((uint32_t)ld_acquire_sys(mine) - p.epoch) < 0) {
        if ((int64_t)(globaltimer_ns() - start) > p.hard_timeout_ns) {
            atomicOr(p.status, kStatusHardTimeout);
            return;
        }
    }
}

template <bool kFP8, bool kCount, int kPhases>
__global__ void __launch_bounds__(512, 2) ep_dispatch_kernel(GroupDispatchParams p) {
    extern __shared__ int smem_i32[];
    if (kCount) {
        for (int i = threadIdx.x; i < p.E; i += blockDim.x) smem_i32[i] = 0;
        __syncthreads();
        pdl_wait();  // (behind a layout kernel: in the body)
    }
    pdl_launch_dependents();
    resolve_seq(p);
    dispatch_body<kFP8, kCount, kPhases>(p, blockIdx.x, gridDim.x, smem_i32);
}

// In-process groups (several logical ranks on one GPU): the ranks' kernels wait
// for one another, so they cannot be separate launches - nothing would
// guarantee that they run at the same time. ONE cooperative launch carries all
// ranks: consecutive runs of `per_rank` blocks do the work of one rank each.
template <bool kFP8, bool kCount, int kPhases>
__global__ void __launch_bounds__(512)
    ep_dispatch_multi_kernel(const GroupDispatchParams* ps, int per_rank) {
    extern __shared__ int smem_i32[];
    __shared__ GroupDispatchParams s_p;
    const int which = blockIdx.x / per_rank;
    if (threadIdx.x == 0) s_p = ps[which];
    __syncthreads();
    if (kCount) {
        for (int i = threadIdx.x; i < s_p.E; i += blockDim.x) smem_i32[i] = 0;
        __syncthreads();
    }
    dispatch_body<kFP8, kCount, kPhases>(s_p, blockIdx.x - which * per_rank, per_rank, smem_i32);
}

// Everything that the receive duty reads arrives with words of this call (the control block's verdicts,
// the peers' payload words), so it starts beside the send kernel and only ends behind it: what the
// stream sees as done is done. One rank on this path, us per layer with this, the reduce phase's like
// (ep_combine_kernel), the own counts taken directly and the first tiles ahead of the layout's end:
// 400 tokens of 14 KB to 8 29.3 -> 26.5, 1024 of 4 KB 24.7 -> 22.1, 2048 of 14 KB 95.3 -> 92.1; in hook mode 1024
// of 8 KB 36.9 -> 33.4, where the host has queued the phases ahead. Rows of peers have not been moved by it
// beside a send kernel: that takes several GPUs.
template <bool kFP8>
__global__ void __launch_bounds__(kRowWarps * 32, 4) ep_dispatch_recv_kernel(GroupDispatchParams p) {
    extern __shared__ int smem_i32[];
    pdl_launch_dependents();
    resolve_seq(p);
    MCEP_TRACE(1, 0);
    dispatch_recv_duty<kFP8, true>(p, blockIdx.x, gridDim.x, smem_i32);
    pdl_wait();
}

// =============================================================================
// groups: combine
// =============================================================================
// Publish duty, shared by `np` participants: rows of expert outputs that peers
// will ask for (every segment of the handle whose source is another rank) are
// copied into this rank's combine input in symmetric memory, same [expert][row]
// position; one system fence per block, a ticket, and whoever finishes last
// tells every peer. With zero copy the caller's kernels wrote the rows there
// already and only the word is sent.
// `first_lr`: layout_range[tid], requested by the caller ahead of its peer tables.
__device__ __forceinline__ void combine_publish_duty(const GroupCombineParams& p, int j, int np,
                                                     int* smem_i32, char* const* s_peer,
                                                     const int* s_active, long long first_lr) {
    const int L = p.E / p.R, n = L * p.R;
    int* pre = smem_i32;  // [n + 1]
    __shared__ int s_wt[32];
    const int tid = threadIdx.x, nthr = blockDim.x;
    const int lane = tid & 31, warp = tid >> 5, nwarps = nthr >> 5;
    const int RM = p.R * p.M;
    const int nchunks = p.H / 16;
    const int ntiles = (p.H + kTileChannels - 1) / kTileChannels;
    bool stored = false;
    if (!p.zero_copy) {
        int* beg = smem_i32 + n + 1;  // [n] first row of each (expert, source) segment
        bool mine = false;
        for (int i = tid; i < n; i += nthr) {
            const int src = i % p.R;
            const long long lr = i == tid ? first_lr : ld_ro(p.layout_range + i);
            int c = (int)(lr & 0xffffffffll);
            if (src == p.rank || !s_active[src]) c = 0;
            pre[i] = c;
            beg[i] = (int)(lr >> 32);
            mine = mine || c > 0;
        }
        int total = 0;
        if (__syncthreads_or(mine ? 1 : 0)) {
            block_exclusive_scan(pre, n, s_wt);
            total = pre[n];
        }
        const char* xb = reinterpret_cast<const char*>(p.x);
        char* cin = p.local_base + p.cin_off;
        // A work item is a run of tiles of one row, sized so that the rows spread
        // over every warp of the participants and an item's loads are all in
        // flight at once (8 x 32 B per lane): the copy costs one memory round trip.
        constexpr int kB = 8;
        const int warps_total = np * nwarps;
        int parts = total > 0 ? warps_total / total : 1;
        if (parts < 1) parts = 1;
        if (parts > ntiles) parts = ntiles;
        int tpp = (ntiles + parts - 1) / parts;  // tiles per item
        if (tpp > kB && parts < ntiles) tpp = kB;
        parts = (ntiles + tpp - 1) / tpp;
        const long long items = (long long)total * parts;
        for (long long g = (long long)warp * np + j; g < items; g += (long long)np * nwarps) {
            const int rg = (int)(g / parts), part = (int)(g - (long long)rg * parts);
            const int i = find_segment(pre, n, rg);
            const int le = i / p.R;
            const int row = beg[i] + (rg - pre[i]);
            if (row >= RM) {
                if (lane == 0) atomicOr(p.wait.status, kStatusSlotRange);
                continue;
            }
            const size_t off = ((size_t)le * RM + row) * (size_t)p.H * 2;
            const int t_end = min(ntiles, (part + 1) * tpp);
            for (int t0 = part * tpp; t0 < t_end; t0 += kB) {
                V32 v[kB];
#pragma unroll
                for (int b = 0; b < kB; ++b) {
                    const int c = (t0 + b) * 32 + lane;
                    if (t0 + b < t_end && c < nchunks) v[b] = ld32_readonly(xb + off + (size_t)c * 32);
                }
#pragma unroll
                for (int b = 0; b < kB; ++b) {
                    const int c = (t0 + b) * 32 + lane;
                    if (t0 + b < t_end && c < nchunks) st32(cin + off + (size_t)c * 32, v[b]);
                }
            }
            stored = true;
        }
    }
    // One fence for the block's rows, then the ticket (see the dispatch kernel).
    // The rows were stored to THIS GPU's memory and peers read them through this
    // GPU's L2, so a device-scope fence (about 1 us) is enough to order them
    // before the word that goes out to the peers; the system-scope one (4 us and
    // more) is for stores that cross NVLink.
    const int any = __syncthreads_or(stored ? 1 : 0);
    MCEP_TRACE(2, 3);  // this block's rows are copied
    // One thread, of the last warp: the others go on to the reduce duty, whose first loads
    // are warp 0's, while the ticket is on its way (128 tokens of 7 KB on one rank, the layer:
    // 16.5 us with a barrier behind the ticket, 15.8 without).
    if (tid == nthr - 32) {
        if (any || (p.zero_copy && j == 0)) __threadfence();
        if (atomicAdd(p.ticket, 1u) == (unsigned)(np - 1)) {
            *p.ticket = 0;
            __threadfence();
            for (int r = 0; r < p.R; ++r) {
                if (r == p.rank || !s_active[r]) continue;
                uint64_t* f = reinterpret_cast<uint64_t*>(s_peer[r] + p.w.cflag_off) + p.rank;
                st_relaxed_sys(f, ((uint64_t)p.seq << 32) | 1u);
            }
        }
    }
}

// Reduce duty: one block per token. Row k of token t lives at the owner of
// expert topk[t][k], at the row the dispatch call recorded; it is read from
// there (a peer's combine input over NVLink once that peer's word has arrived,
// or this rank's own expert output) and the K rows are reduced in registers.
// An owner that is inactive, or whose word does not arrive in time (it is then
// marked inactive), contributes nothing (mooncake_ep_kernel.cu:685-699, 728-732).
template <bool kLast>
__device__ __forceinline__ void combine_reduce_duty(const GroupCombineParams& p, int first_token, int token_stride,
                                                    char* const* s_peer, const int* s_active, bool hold) {
    __shared__ const char* s_ptr[kMaxTopk];
    __shared__ float s_w[kMaxTopk];
    const int tid = threadIdx.x;
    const int L = p.E / p.R, RM = p.R * p.M;
    const uint64_t* flags = reinterpret_cast<const uint64_t*>(p.local_base + p.w.cflag_off);
    const char* own = p.zero_copy ? p.local_base + p.cin_off : reinterpret_cast<const char*>(p.x);
    for (int t = first_token; t < p.T; t += token_stride) {
        if (tid < kMaxTopk) {
            const char* ptr = nullptr;
            float w = 0.f;
            if (tid < p.K) {
                const int e = (int)ld_ro(p.topk_idx + (size_t)t * p.K + tid);
                w = ld_ro(p.topk_weights + (size_t)t * p.K + tid);
                const int row = ld_l2(p.rowmap + (size_t)t * p.K + tid);
                if (e >= 0 && e < p.E && row >= 0 && row < RM) {
                    const int o = e / L, le = e - o * L;
                    const size_t off = ((size_t)le * RM + row) * (size_t)p.H * 2;
                    if (o == p.rank) {
                        if (s_active[o]) ptr = own + off;  // (as of the kernel's start)
                    } else if (ld_volatile_s32(p.wait.active_ranks + o) && s_peer[o] != nullptr) {
                        const uint32_t v = resolve_flag(flags, p.res_cflag, o, p.seq, p.wait, o,
                                                        ((first_token + o) & 7) == 0);
                        if (v && ld_volatile_s32(p.wait.active_ranks + o))
                            ptr = s_peer[o] + p.cin_off + off;
                    }
                }
            }
            s_ptr[tid] = ptr;
            s_w[tid] = w;
        }
        __syncthreads();
        if (t == first_token) MCEP_TRACE(2, 4);  // the owners' words are in, rows can be read
        reduce_rows<8, false, kLast>(s_ptr, s_w, p.K, p.H,
                                     reinterpret_cast<char*>(p.combined_x) + (size_t)t * p.H * 2, hold);
        __syncthreads();  // the rows are done with s_ptr
    }
}

// kPhases: 1 = publish, 2 = reduce, 3 = both in one launch.
template <int kPhases, bool kLast>
__device__ __forceinline__ void combine_body(const GroupCombineParams& p, int bid, int nblocks,
                                             int* smem_i32) {
    __shared__ char* s_peer[kMaxRanks];
    __shared__ int s_active[kMaxRanks];
    MCEP_TRACE(2, 0);
    long long first_lr = 0;
    if ((kPhases & 1) && !p.zero_copy && (int)threadIdx.x < p.E) first_lr = ld_ro(p.layout_range + threadIdx.x);
    load_peer_tables(p.peer_base, p.wait.active_ranks, p.R, p.wait.status, s_peer, s_active);
    __syncthreads();
    if (kPhases & 1) combine_publish_duty(p, bid, nblocks, smem_i32, s_peer, s_active, first_lr);
    MCEP_TRACE(2, 1);
    if (kPhases & 2) {
        combine_reduce_duty<kLast>(p, bid, nblocks, s_peer, s_active, kPhases == 2 && !p.behind_publish);
    }
    MCEP_TRACE(2, 2);
}

// What the reduce phase reads was complete when the publish phase began - that kernel lets the next
// one start only once it has waited for all before it - and a peer's rows come with the peer's word.
// So it starts beside the publish phase (or what the caller has put between), and only ends behind
// it. With a hook (not behind_publish) that work may still read the result's memory: nothing is
// stored there before it has finished. Waiting at the top, hook mode, one rank on this path, us per layer:
// 1024 tokens of 8 KB to 8 34.8, so 33.4; 400 of 4 KB in FP8 17.3 and 15.9; 250 of 14 KB 22.3 and 20.9.
template <int kPhases, bool kLast = false>
__global__ void __launch_bounds__(512) ep_combine_kernel(GroupCombineParams p) {
    extern __shared__ int smem_i32[];
    if (kPhases != 2) pdl_wait();
    pdl_launch_dependents();
    resolve_seq(p);
    combine_body<kPhases, kLast>(p, blockIdx.x, gridDim.x, smem_i32);
    if (kPhases == 2) pdl_wait();
}

// The reduce duty of batches with more tokens than SMs, in a launch of its own: as
// ep_combine_rows_kernel, no barrier per token, a warp owns one tile of one row of every
// group of tokens. What a group adds: a row lies in its owner's memory, readable once
// the owner's word is here. A warp asks for an owner's word once - when a token of it
// first needs that owner - and keeps the verdict. One rank on this path, 2048 tokens of
// 14 KB to 8: 47 us, with a barrier per token and the words looked at for every one 59
// (512 tokens 16.7 and 18.9).
template <int kDepth, bool kLast>
__global__ void __launch_bounds__(kReduceWarps * 32, 2) ep_combine_gather_kernel(GroupCombineParams p) {
    __shared__ char* s_peer[kMaxRanks];
    __shared__ int s_active[kMaxRanks];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sub = warp / p.tiles_per_block;
    const int c = ((warp - sub * p.tiles_per_block + blockIdx.y * p.tiles_per_block) * 32) + lane;
    const bool act = c < p.H / 16;
    pdl_launch_dependents();
    resolve_seq(p);
    const int L = p.E / p.R, RM = p.R * p.M;
    const size_t row_bytes = (size_t)p.H * 2;
    const int run = p.span < 0 ? -p.span : p.span;
    const int step = (run ? 1 : gridDim.x) * p.tokens_per_block;
    const int first = (p.span < 0 ? gridDim.x - 1 - blockIdx.x : blockIdx.x) * (run ? run : p.tokens_per_block);
    const int end = run ? min(p.T, first + run) : p.T;

    int next_row = -1, next_e = -1;
    float next_w = 0.f;
    auto request = [&](int tok) {
        if (lane < p.K && tok < end) {
            const size_t at = (size_t)tok * p.K + lane;
            next_row = ld_l2(p.rowmap + at);
            next_e = (int)ld_ro(p.topk_idx + at), next_w = ld_ro(p.topk_weights + at);
        } else {
            next_row = -1;
        }
    };
    request(first + sub);
    load_peer_tables(p.peer_base, p.wait.active_ranks, p.R, p.wait.status, s_peer, s_active);
    __syncthreads();
    const char* own = p.zero_copy ? p.local_base + p.cin_off : reinterpret_cast<const char*>(p.x);
    const uint64_t* flags = reinterpret_cast<const uint64_t*>(p.local_base + p.w.cflag_off);
    unsigned known[2] = {0, 0}, good[2] = {0, 0};  // owners whose word has been asked for / whose rows count
    for (int t0 = first; t0 < end; t0 += step) {
        int owner = -1;
        const char* row = nullptr;
        if (next_e >= 0 && next_e < p.E && next_row >= 0 && next_row < RM) {
            owner = next_e / L;
            const size_t off = ((size_t)(next_e - owner * L) * RM + next_row) * row_bytes;
            row = (owner == p.rank ? own : s_peer[owner] + p.cin_off) + off;
        }
        const float w = next_w;
        const bool ask = owner >= 0 && !((known[owner >> 5] >> (owner & 31)) & 1u);
        if (__any_sync(kFull, ask)) {
            bool ok = false;
            if (ask && owner == p.rank) {
                ok = s_active[owner] != 0;  // (as of the kernel's start: nobody waits for this rank here)
            } else if (ask && ld_volatile_s32(p.wait.active_ranks + owner)) {
                if (s_peer[owner] != nullptr)
                    ok = resolve_flag(flags, p.res_cflag, owner, p.seq, p.wait, owner,
                                      ((blockIdx.x + owner) & 7) == 0 && warp == 0) != 0 &&
                         ld_volatile_s32(p.wait.active_ranks + owner) != 0;
            }
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const unsigned bit = ask && (owner >> 5) == h ? 1u << (owner & 31) : 0u;
                known[h] |= __reduce_or_sync(kFull, bit);
                good[h] |= __reduce_or_sync(kFull, ok ? bit : 0u);
            }
            __syncwarp();  // the acquire of one lane orders the loads of all
        }
        if (owner < 0 || !((good[owner >> 5] >> (owner & 31)) & 1u)) row = nullptr;
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        for (int k0 = 0; k0 < p.K; k0 += kDepth) {
            V32 v[kDepth];
            unsigned there = 0;
#pragma unroll
            for (int b = 0; b < kDepth; ++b) {
                const char* r = reinterpret_cast<const char*>(
                    __shfl_sync(kFull, (unsigned long long)reinterpret_cast<uintptr_t>(row), k0 + b));
                if (r != nullptr) {
                    there |= 1u << b;
                    if (act) v[b] = ld32_coherent(r + (size_t)c * 32, kLast);
                }
            }
            if (k0 == 0) request(t0 + step + sub);
#pragma unroll
            for (int b = 0; b < kDepth; ++b) {
                const float wk = __shfl_sync(kFull, w, k0 + b);
                if (there & (1u << b)) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        acc[2 * i] = fmaf(bf16lo(v[b].w[i]), wk, acc[2 * i]);
                        acc[2 * i + 1] = fmaf(bf16hi(v[b].w[i]), wk, acc[2 * i + 1]);
                    }
                }
            }
        }
        if (!p.behind_publish && t0 == first) pdl_wait();
        if (act && t0 + sub < end)
            st32(reinterpret_cast<char*>(p.combined_x) + (size_t)(t0 + sub) * row_bytes + (size_t)c * 32,
                 pack_bf16x16(acc));
    }
    pdl_wait();
}

// All logical ranks of an in-process group in one cooperative launch (see
// ep_dispatch_multi_kernel).
__global__ void __launch_bounds__(512)
    ep_combine_multi_kernel(const GroupCombineParams* ps, int per_rank) {
    extern __shared__ int smem_i32[];
    __shared__ GroupCombineParams s_p;
    const int which = blockIdx.x / per_rank;
    if (threadIdx.x == 0) s_p = ps[which];
    __syncthreads();
    combine_body<3, false>(s_p, blockIdx.x - which * per_rank, per_rank, smem_i32);
}

// threads per block: one warp per tile, at most 16 warps
inline int block_threads(int H, int at_least = 32) {
    int ntiles = (H + kTileChannels - 1) / kTileChannels;
    if (ntiles > 16) ntiles = 16;
    if (ntiles < 1) ntiles = 1;
    int t = ntiles * 32;
    return t < at_least ? at_least : t;
}
// how many blocks of this kernel are resident at a time on the whole device
template <typename K>
inline long long resident_blocks(K kernel, int threads, size_t smem, const LaunchCtx& ctx) {
    // the occupancy query is not free: remember the answer per (kernel, block, smem)
    static std::mutex mu;
    static std::map<std::tuple<const void*, int, size_t>, int> cache;
    int per_sm = 0;
    {
        std::lock_guard<std::mutex> lk(mu);
        auto key = std::make_tuple(reinterpret_cast<const void*>(kernel), threads, smem);
        auto it = cache.find(key);
        if (it != cache.end()) {
            per_sm = it->second;
        } else {
            if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) !=
                    cudaSuccess ||
                per_sm < 1) {
                cudaGetLastError();
                per_sm = 1;
            }
            cache[key] = per_sm;
        }
    }
    return (long long)ctx.num_sms * per_sm;
}
// a grid that fills the machine once (blocks stride over the work items)
template <typename K>
inline int persistent_grid(long long items, K kernel, int threads, size_t smem, const LaunchCtx& ctx) {
    const long long cap = resident_blocks(kernel, threads, smem, ctx);
    long long g = items < cap ? items : cap;
    return (int)(g < 1 ? 1 : g);
}

}  // namespace kernels
using namespace kernels;

// =============================================================================
// launchers
// =============================================================================
// The chunked route: chunks of up to 256 tokens (fewer when the per-chunk bitmap
// of all experts would not fit 48 KB of shared memory), at most 128 chunks, and
// per-chunk histograms that fit the scratch the caller gave.
static bool layout_chunking(const LayoutParams& p, int* chunk_tokens, int* words, int* chunks) {
    if (p.chunk_hist == nullptr || p.T < 512) return false;
    int w = (int)(12288 / p.E) - 1;  // (1 + w) * E ints of shared memory, 48 KB at most
    if (w > 8) w = 8;
    if (w < 1) return false;
    const int ct = w * 32;
    const int c = (p.T + ct - 1) / ct;
    if (c > 128 || (size_t)c * p.E > p.chunk_hist_entries) return false;
    *chunk_tokens = ct, *words = w, *chunks = c;
    return true;
}

// Threads per block of the cluster route with clusters of `blocks`: a multiple of
// 32, one lane per token; 0 when the tables of E experts do not fit shared memory
// or the batch is too large.
static int layout_cluster_threads(const LayoutParams& p, int blocks) {
    if (p.rank_count != nullptr || p.expert_prefix != nullptr) return 0;
    const int threads = ((p.T + blocks - 1) / blocks + 31) / 32 * 32;
    if (threads < 32 || threads > 1024) return 0;
    return (size_t)p.E * (threads / 16 + 2) * sizeof(int) <= 160 * 1024 ? threads : 0;
}

RouteBits route_bits(void* memory, size_t capacity, int T, int E) {
    RouteBits b = {};
    const int chunks = (T + kChunkTokens - 1) / kChunkTokens;
    const int stride = (chunks + 15) / 16 * 16;
    if (chunks < 1 || chunks > 128 || (size_t)E * (chunks * sizeof(uint4) + stride) > capacity) return b;
    b.words = static_cast<uint4*>(memory);
    b.counts = reinterpret_cast<uint8_t*>(b.words + (size_t)E * chunks);
    b.experts = E, b.chunks = chunks, b.stride = stride;
    return b;
}

cudaError_t launch_layout(const LayoutParams& p, const LaunchCtx& ctx) {
    if (p.bits.words != nullptr) {
        const size_t smem = (size_t)p.E * sizeof(uint4);
        if (cudaError_t e = allow_shared_memory(reinterpret_cast<const void*>(ep_layout_bits_kernel), smem)) return e;
        return launch("ep_layout_bits", ep_layout_bits_kernel, dim3(p.bits.chunks), dim3(kBitsThreads), smem, ctx, p);
    }
    // Sixteen blocks (opt-in cluster size) once eight would have more than 8 warps
    // each: setting the bits is bound by the shared-memory atomics of a block.
    const void* k = reinterpret_cast<const void*>(ep_layout_cluster_kernel);
    for (int blocks : {kLayoutClusterLarge, kLayoutCluster}) {
        if (blocks == kLayoutClusterLarge && p.T <= kLayoutCluster * 256) continue;
        const int threads = layout_cluster_threads(p, blocks);
        if (threads == 0) continue;
        const size_t smem = (size_t)p.E * (threads / 16 + 2) * sizeof(int);
        bool fits = false;
        if (cudaError_t e = cluster_fits(k, blocks, threads, smem, &fits)) return e;
        if (fits)
            return launch_kernel("ep_layout_cluster", ep_layout_cluster_kernel, dim3(blocks), dim3(threads), smem,
                                 blocks, ctx, p);
    }
    int chunk_tokens = 0, cwords = 0, chunks = 0;
    if (layout_chunking(p, &chunk_tokens, &cwords, &chunks)) {
        cudaError_t e = launch("ep_layout_hist", ep_layout_hist_kernel, dim3(chunks),
                               dim3(chunk_tokens), (size_t)p.E * sizeof(int), ctx, p);
        if (e != cudaSuccess) return e;
        LaunchCtx chained = ctx;
        chained.pdl = true;
        return launch("ep_layout_slot", ep_layout_slot_kernel, dim3(chunks), dim3(chunk_tokens),
                      (size_t)p.E * (1 + cwords) * sizeof(int), chained, p);
    }
    const int words = (p.T + 31) / 32 > 0 ? (p.T + 31) / 32 : 1;
    const long long n = (long long)p.T * p.K;
    // Every block reads the whole index matrix, so the number of blocks trades
    // parallelism against L2 traffic: keep blocks * n * 8 bytes around 8 MB.
    long long max_blocks = n > 0 ? (1ll << 20) / n : ctx.num_sms;
    if (max_blocks < 8) max_blocks = 8;
    if (max_blocks > ctx.num_sms) max_blocks = ctx.num_sms;
    int epc = (int)((p.E + max_blocks - 1) / max_blocks);
    if (epc < 1) epc = 1;
    const size_t budget = 200 * 1024;
    while (epc > 1 && (size_t)epc * words * 8 > budget) --epc;
    const size_t smem = (size_t)epc * words * 8;
    if (smem > budget) return cudaErrorInvalidValue;  // > 819k tokens per rank
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(ep_routing_layout_kernel,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
        if (e != cudaSuccess) return e;
    }
    int threads = 128;
    while (threads < 1024 && threads * 4 < n) threads <<= 1;
    const int grid = (p.E + epc - 1) / epc;
    return launch("ep_routing_layout", ep_routing_layout_kernel, dim3(grid), dim3(threads), smem,
                  ctx, p, epc, words);
}

bool counts_in_send_kernel(int T, int K, int H, int num_sms, bool group) {
    // A group's sender blocks are one resident wave, a token each, and up to here a dispatch without a
    // hook is one launch for all ranks of a process alike (group_call_can_be_one_kernel), whatever
    // their tokens. One rank on this path, us per layer to 8, counting | layout kernel: rows of 4 KB
    // in bf16 150 tokens 11.4 | 12.6, 292 14.4 | 13.8; of 14 KB 150 18.3 | 18.4, 292 20.3 | 21.4. Rows of
    // 8 KB would take the layout kernel from 200 on (16.4 | 15.3, 292 18.2 | 16.4, in FP8 17.8 | 16.8), but
    // three launches in place of one are not measured where peers have rows to move.
    if (group) return T <= 2 * num_sms;
    // A single rank counts in one resident wave of blocks with as many tokens each as that
    // takes. The layout kernel is the faster one on the device at nearly every size, but a
    // layer of three launches takes the host 12.4 us and one of two 10: it is used where the
    // rows, in either type, are more than the device moves in that time. Up to two choices per
    // token (us per layer, counting | layout kernel): rows of 8 KB to 2, 600 tokens (10 MB) 10.6 |
    // 12.4, 1000 (16 MB) 14.3 | 14.2, in FP8 13.9 | 12.7, 4000 38.9 | 37.1; of 2 KB 2000 (8 MB) 10.3 |
    // 12.3, 4000 16.3 | 14.3; of 14 KB to 1, 600 (9 MB) 11.3 | 12.4, 1000 16.1 | 15.5, 4000 44.2 |
    // 41.7, 8000 in FP8 76.6 | 71.1. Just below the line some lose: of 8 KB to 1, 1500 (12 MB) 11.0 | 11.7,
    // in FP8 12.2 | 11.8, and a stream that is ahead of the device has 12.4 | 10.7; of 2 KB to 2, 3000
    // 12.4 | 11.8.
    const long long bytes = (long long)T * K * H * 2;
    if (K <= 2) return bytes < 12 << 20 && T <= 8192 / K;
    // From three on counting is slower by block: rows of 8 KB to 8 in FP8, 200 tokens (13 MB)
    // 10.0 | 12.4, 300 (20 MB) 13.5 | 12.4, 400 16.3 | 14.9; of 14 KB in bf16, 160 (18 MB) 15.2 |
    // 13.8, 300 24.8 | 21.1, 590 32.6 | 31.7; of 4 KB to 4, 590 (10 MB) 10.0 | 12.4. Around the line, wall
    // and a stream that is ahead: of 8 KB to 8 in FP8, 240 (15 MB) 9.9 | 11.4 and 9.4 | 9.5, 270 (17 MB)
    // 10.5 | 11.7 and 9.5 | 9.6; in bf16 240 11.1 | 11.3 and 10.0 | 10.5, 270 11.7 | 11.5 and 10.3 | 10.4; of 5 KB
    // 400 (16 MB) in FP8 11.1 | 11.9 and 10.3 | 9.4, in bf16 11.9 | 11.5 and 11.2 | 10.1; of 3 KB 590 (14 MB) in
    // FP8 11.4 | 11.6 and 10.7 | 9.2.
    return T <= num_sms || (T <= 4 * num_sms && bytes < 17 << 20);
}

// Tokens per batch and threads per block of the kernels that work through batches.
// A single rank that counts: one resident wave of up to 16 warps, each with a tile at a
// time (1000 rows of 8 KB to 2: 11.9 us per layer, two waves 14.0).
// A group's sender blocks are one resident wave that strides: batches of 16 warp tiles,
// 8 warps once there are more tokens than blocks (2000 rows of 8 KB to 8: 64.0 us per
// layer, 16 warps 67.3; one token per batch 64.6, rows of 2 KB 30.7 against 27.0), a warp
// per tile before (256 tokens of 14 KB to 8: 20.9 us, 8 warps 23.4).
static SendShape send_shape(int T, int K, int H, int num_sms, bool group) {
    const int ntiles = (H + kTileChannels - 1) / kTileChannels;
    SendShape s;
    s.tokens = (T + 2 * num_sms - 1) / (2 * num_sms);  // two blocks per SM
    if (group && s.tokens > 16 / ntiles) s.tokens = 16 / ntiles;
    if (group && s.tokens > 8) s.tokens = 8;
    if (s.tokens > kBatchEntries / K) s.tokens = kBatchEntries / K;
    if (s.tokens < 1) s.tokens = 1;
    const int most = group && T > 2 * num_sms ? 8 : 16, least = group ? 8 : 4;
    int warps = s.tokens * ntiles;
    if (warps > most) warps = most;
    if (warps < least) warps = least;
    s.threads = 32 * warps;
    return s;
}

// Batches that count for themselves, a token per block instead of several: as many as are resident at
// a time, at two blocks of 16 warps, and three per SM, as each compares itself with all earlier ones.
// Device us per layer, several | one: 300 tokens of 1 KB in FP8 to 8 8.5 | 7.6, of 8 KB to 2 7.6 | 6.3; 400 9.3 | 8.9
// and 7.8 | 7.4; 500 of 8 KB to 1 7.0 | 7.1, of 4 KB to 8 10.8 | 11.1; 1100 of 4 KB to 1 8.1 | 11.5.
static bool one_token_per_block(int T, int warps, int num_sms) {
    return T > 0 && T <= 3 * num_sms && T < 2 * num_sms * (16 / warps);
}

bool layer_beyond_l2(long long T, int copies, int H) { return T * (copies + 2) * H * 2 > 40ll << 20; }
bool input_beyond_l2(long long T, int copies, int H, bool fp8) {
    return fp8 ? layer_beyond_l2(T, copies, H) : T * (copies + 1) * H * 2 > 120ll << 20;
}

cudaError_t launch_direct_dispatch(DirectDispatchParams p, const LaunchCtx& ctx) {
    if (!p.counting()) {
        p.x_last = input_beyond_l2(p.T, p.K, p.H, p.use_fp8);
        const int ntiles = (p.H + kTileChannels - 1) / kTileChannels;
        void (*k)(DirectDispatchParams) = ep_dispatch_rows_kernel<true, 1, 7, 6>;
        int tiles = 1, most = 7;
        if (p.use_fp8) {
            // four tiles | two: 8192 rows of 14 KB to 1 72.0 | 78.8, 4000 of 4 KB 11.3 | 12.2, 2000 of
            // 14 KB 19.2 | 20.4; to 2, 2000 of 14 KB 31.1 | 30.3
            // two tiles | one: 4096 rows of 14 KB to 3 68.5 | 73.0, to 4 82.4 | 85.5, to 8 145.9 |
            // 145.8; 4000 of 4 KB to 4 29.2 | 29.8; 1500 of 8 KB to 8 37.6 | 36.5
            if (p.K == 1 && ntiles >= 4)
                k = ep_dispatch_rows_kernel<true, 4, 4, 8>, tiles = 4, most = 4;
            else if (p.K <= 4 && ntiles >= 4)
                k = ep_dispatch_rows_kernel<true, 2, 4, 10>, tiles = 2, most = 4;
        } else if (p.K == 1 ? ntiles >= 4 : p.K == 2 && ntiles > 8) {
            // two tiles | one: 8000 rows of 14 KB to 1 76.3 | 86.1, 1000 of 8 KB 10.1 | 11.0; 4000 of
            // 14 KB to 2 59.0 | 60.0, 2000 of 8 KB 22.5 | 22.1; to 3 1500 of 8 KB 22.2 | 21.8
            k = ep_dispatch_rows_kernel<false, 2, 4, 10>, tiles = 2, most = 4;
        } else if ((long long)p.T * p.K * p.H * 2 < 256 << 20) {
            // 42 warps per SM | 32: to 3, 4096 rows of 14 KB (168 MB) 78.4 | 79.8; to 4 (224 MB) 97.4 |
            // 97.2, to 6 135.8 | 135.5, to 8 174.7 | 173.7
            k = ep_dispatch_rows_kernel<false, 1, 7, 6>;
        } else {
            k = ep_dispatch_rows_kernel<false, 1, 4, 8>, most = 4;
        }
        const int warps = (ntiles + tiles - 1) / tiles;  // of a row
        p.parts = (warps + most - 1) / most;
        p.warps_per_row = (warps + p.parts - 1) / p.parts;
        p.tokens_per_block = most / p.warps_per_row;
        const int groups = (p.T + p.tokens_per_block - 1) / p.tokens_per_block;
        return launch("ep_dispatch_rows", k, dim3(groups * p.parts), dim3(32 * p.warps_per_row * p.tokens_per_block), 0,
                      ctx, p);
    }
    const int ntiles = (p.H + kTileChannels - 1) / kTileChannels, warps = ntiles < 4 ? 4 : ntiles < 16 ? ntiles : 16;
    if (one_token_per_block(p.T, warps, ctx.num_sms) && (long long)p.E * p.M * (p.H / 128) <= INT_MAX) {
        void (*one)(DirectDispatchParams) = nullptr;
        if (p.K <= 4)
            one = p.use_fp8 ? ep_dispatch_one_token_kernel<true, 4> : ep_dispatch_one_token_kernel<false, 4>;
        else if (p.K <= 8)
            one = p.use_fp8 ? ep_dispatch_one_token_kernel<true, 8> : ep_dispatch_one_token_kernel<false, 8>;
        else
            one = p.use_fp8 ? ep_dispatch_one_token_kernel<true, 16> : ep_dispatch_one_token_kernel<false, 16>;
        return launch("ep_dispatch_send_direct", one, dim3(p.T + 1), dim3(32 * warps), (size_t)p.E * sizeof(int), ctx,
                      p);
    }
    const SendShape s = send_shape(p.T, p.K, p.H, ctx.num_sms, false);
    p.C = s.tokens;
    auto k = p.use_fp8 ? ep_dispatch_send_direct_kernel<true> : ep_dispatch_send_direct_kernel<false>;
    const int grid = p.T > 0 ? (p.T + p.C - 1) / p.C : 1;
    return launch("ep_dispatch_send_direct", k, dim3(grid), dim3(s.threads), (size_t)p.E * sizeof(int), ctx, p);
}

cudaError_t launch_combine_invert(const CombineInvertParams& p, const LaunchCtx& ctx) {
    const long long total = (long long)p.L * p.M;
    long long blocks = (total + 255) / 256;
    const long long cap = (long long)ctx.num_sms * 8;
    if (blocks > cap) blocks = cap;
    if (blocks < 1) blocks = 1;
    return launch("ep_combine_invert", ep_combine_invert_kernel, dim3((int)blocks), dim3(256), 0,
                  ctx, p);
}

// How the kernels that give a warp one tile of a row per token are laid out.
struct ReduceShape {
    int tiles_per_block, tokens_per_block, span, threads;  // span < 0: the last run first
    dim3 grid;
};
static ReduceShape reduce_shape(int T, int K, int H, int num_sms) {
    ReduceShape s;
    // Blocks of up to 8 warps (whole rows, or part of one) once there are more tokens than
    // SMs (400 tokens of 14 KB to 8: 20.7 us per layer, 16 warps 22.0; 4096: 173.6 and
    // 175.1); up to one block per SM, registers are spent on loads in flight.
    const int ntiles = (H + kTileChannels - 1) / kTileChannels;
    const int most_warps = T > num_sms ? 8 : kReduceWarps;
    const int parts = (ntiles + most_warps - 1) / most_warps;  // blocks that share a row
    s.tiles_per_block = (ntiles + parts - 1) / parts;
    s.tokens_per_block = 1;
    if (T > num_sms) {
        const int fit = most_warps / s.tiles_per_block, most = (T + 2 * num_sms - 1) / (2 * num_sms);
        s.tokens_per_block = fit < most ? fit : most;
    }
    s.threads = 32 * s.tiles_per_block * s.tokens_per_block;
    const int groups = T > 0 ? (T + s.tokens_per_block - 1) / s.tokens_per_block : 1;
    // How the groups are dealt out, in waves of the blocks that are resident at a time
    // (two of 16 warps per SM, more of smaller ones). Fewer than 8 rows per token, or
    // fewer than 4 waves: a full wave striding (4096 tokens of 14 KB to 4: 45.7 us, runs
    // 47.5; 600 to 8: 10.6, equal runs, which leave blocks out, 12.4). Else, 4 to 8 waves:
    // every block an equal run of consecutive groups (1024 tokens to 8: 20.5 us, strided
    // 22.5). More: runs of two, handed out as blocks finish, so that no SM falls behind
    // (4096 tokens to 8 after a write of 512 MB, whose last lines are still leaving L2:
    // 96 us, equal runs and strided 100; 8192 tokens 168 against 184 and 181). Those are rows
    // beyond L2: the last tokens' are taken first, as what was written last is still there
    // where the rows were made in token order (combine of the rows just received, first | last
    // tokens first: 4096 x 14 KB 94.2 us | 90.1, 3000 73 | 67.6, 8000 x 8 KB 102.4 | 97.5). Rows that are
    // written expert by expert just before, as a grouped GEMM does, gain less or nothing (90.1 |
    // 88.2, 69.6 | 69.6, 98.3 | 96.3), rows made long before nothing (96.3 | 96.3, 74.4 | 75.8, 102.4 |
    // 104.4). The group's kernel has the order too (one rank on that path, 4096 x 14 KB 101.4 | 97.2,
    // written by expert 99.4 | 97.3, long before 101.4 | 101.4; rows of peers have not been measured).
    // With fewer waves it gains and loses 1 %.
    const int resident = std::max(1, num_sms * (2 * kReduceWarps * 32 / s.threads) / parts);
    const int waves = (groups + resident - 1) / resident;
    const int run = K < 8 || waves < 4 ? 0 : waves <= 8 ? waves : 2;
    s.span = (run == 2 ? -run : run) * s.tokens_per_block;
    s.grid = dim3(run ? (groups + run - 1) / run : groups < resident ? groups : resident, parts);
    return s;
}

cudaError_t launch_direct_combine(DirectCombineParams p, const LaunchCtx& ctx) {
    if (p.search) {
        const int threads = block_threads(p.H);
        const int grid = persistent_grid(p.T, ep_combine_search_kernel, threads, 0, ctx);
        return launch("ep_combine_search", ep_combine_search_kernel, dim3(grid), dim3(threads), 0, ctx, p);
    }
    const bool last = layer_beyond_l2(p.T, p.K, p.H);
    const int row_tiles = (p.H + kTileChannels - 1) / kTileChannels;
    if (p.K == 1) {
        // two rounds of four tiles per warp (4096 rows of 14 KB: 21.0 us, 29 - 32 with the
        // kernel for more rows; four rows per block 21.5, two 25.6)
        int c = 112 / row_tiles;
        if (c > 16) c = 16;
        const int most = (p.T + 2 * ctx.num_sms - 1) / (2 * ctx.num_sms);
        p.tokens_per_block = c < 1 ? 1 : c < most ? c : most < 1 ? 1 : most;
        const int warps = p.tokens_per_block * row_tiles;
        void (*k)(DirectCombineParams) = nullptr;
        if (p.absolute)
            k = last ? ep_combine_one_row_kernel<true, true> : ep_combine_one_row_kernel<true, false>;
        else
            k = last ? ep_combine_one_row_kernel<false, true> : ep_combine_one_row_kernel<false, false>;
        const int grid = p.T > 0 ? (p.T + p.tokens_per_block - 1) / p.tokens_per_block : 1;
        return launch("ep_combine_reduce_direct", k, dim3(grid), dim3(32 * (warps < 16 ? warps : 16)), 0, ctx, p);
    }
    const ReduceShape shape = reduce_shape(p.T, p.K, p.H, ctx.num_sms);
    p.tiles_per_block = shape.tiles_per_block, p.tokens_per_block = shape.tokens_per_block, p.span = shape.span;
    void (*k)(DirectCombineParams) = nullptr;
    if (p.T <= ctx.num_sms)
        k = p.absolute ? ep_combine_rows_kernel<8, true, 1, false> : ep_combine_rows_kernel<8, false, 1, false>;
    else if (p.absolute)
        k = last ? ep_combine_rows_kernel<4, true, 2, true> : ep_combine_rows_kernel<4, true, 2, false>;
    else
        k = last ? ep_combine_rows_kernel<4, false, 2, true> : ep_combine_rows_kernel<4, false, 2, false>;
    return launch("ep_combine_reduce_direct", k, shape.grid, dim3(shape.threads), 0, ctx, p);
}

// ---- groups -----------------------------------------------------------------------
namespace {

using DispatchKernel = void (*)(GroupDispatchParams);

template <int kPhases>
DispatchKernel pick_dispatch(bool fp8, bool counting) {
    if (counting) return fp8 ? ep_dispatch_kernel<true, true, kPhases> : ep_dispatch_kernel<false, true, kPhases>;
    return fp8 ? ep_dispatch_kernel<true, false, kPhases> : ep_dispatch_kernel<false, false, kPhases>;
}

// the control block keeps two tables of E entries, a sender one, the receive duty two and a total
size_t dispatch_smem(const GroupDispatchParams& p) { return (size_t)(2 * p.E + 1) * sizeof(int); }

}  // namespace

bool group_call_can_be_one_kernel(int T, int K, int E, int num_sms) {
    // a small batch: one block per token plus the control block (the launcher
    // falls back to two launches when that many blocks are not resident at once)
    return (long long)T * K <= 4096 && E <= 2048 && T + 1 <= 2 * num_sms;
}

cudaError_t launch_group_dispatch(GroupDispatchParams p, const LaunchCtx& ctx) {
    const SendShape s = send_shape(p.T, p.K, p.H, ctx.num_sms, true);
    p.C = s.tokens;
    const size_t smem = dispatch_smem(p);
    auto k = pick_dispatch<3>(p.use_fp8 != 0, p.counting());
    const int grid = 1 + (p.T > 0 ? p.T : 1);
    if (p.C != 1 || grid > resident_blocks(k, s.threads, smem, ctx)) return cudaErrorInvalidConfiguration;
    return launch("ep_dispatch", k, dim3(grid), dim3(s.threads), smem, ctx, p);
}

cudaError_t launch_group_dispatch_send(GroupDispatchParams p, const LaunchCtx& ctx) {
    const SendShape s = send_shape(p.T, p.K, p.H, ctx.num_sms, true);
    p.C = s.tokens;
    const size_t smem = dispatch_smem(p);
    p.x_last = input_beyond_l2(p.T, p.K, p.H, p.use_fp8);
    auto k = pick_dispatch<1>(p.use_fp8 != 0, p.counting());
    // the control block, then one block per token (small batches) or a resident wave
    // (a wave, not a block per batch: a block that stored rows in a peer's memory, nearly
    // every one in a group of several GPUs, ends with a system-scope fence)
    long long cap = resident_blocks(k, s.threads, smem, ctx) - 1;
    if (cap < 1) cap = 1;
    const int batches = p.T > 0 ? (p.T + p.C - 1) / p.C : 1;
    const int senders = (int)(batches < cap ? batches : cap);
    return launch("ep_dispatch_send", k, dim3(1 + senders), dim3(s.threads), smem, ctx, p);
}

cudaError_t launch_group_dispatch_recv(const GroupDispatchParams& p, const LaunchCtx& ctx) {
    const int threads = kRowWarps * 32;
    const size_t smem = (size_t)(2 * p.E + 1) * sizeof(int);
    auto k = p.use_fp8 ? ep_dispatch_recv_kernel<true> : ep_dispatch_recv_kernel<false>;
    // The row count is only known on the device. Under even routing a rank
    // receives about what it sends; the grid is sized for twice that - blocks
    // stride, so a skewed or larger load is still covered - and never beyond
    // one resident wave. Without a row copy the duty is light: fewer blocks.
    long long rows = 2ll * (p.T * p.K > 64 ? p.T * p.K : 64);
    const long long worst = (long long)p.E * p.M;
    if (rows > worst) rows = worst;
    long long blocks = (rows + kRowWarps - 1) / kRowWarps;
    if (!p.copy_rows && blocks > 2ll * ctx.num_sms) blocks = 2ll * ctx.num_sms;
    const int grid = persistent_grid(blocks, k, threads, smem, ctx);
    return launch("ep_dispatch_recv", k, dim3(grid), dim3(threads), smem, ctx, p);
}

cudaError_t launch_group_combine(const GroupCombineParams& p, const LaunchCtx& ctx) {
    const int threads = block_threads(p.H, 256);
    const size_t smem = (size_t)(2 * p.E + 1) * sizeof(int);
    auto k = ep_combine_kernel<3>;
    // one block per token for the reduce duty, and enough blocks for this rank's
    // share of the publish duty when it has few tokens of its own
    long long want = p.T > 64 ? p.T : 64;
    const int grid = persistent_grid(want, k, threads, smem, ctx);
    return launch("ep_combine", k, dim3(grid), dim3(threads), smem, ctx, p);
}

cudaError_t launch_group_combine_publish(const GroupCombineParams& p, const LaunchCtx& ctx) {
    const int threads = kRowWarps * 32;
    const size_t smem = (size_t)(2 * p.E + 1) * sizeof(int);
    auto k = ep_combine_kernel<1>;
    long long blocks = 1;
    if (!p.zero_copy) {
        const long long rows = (long long)p.E * p.M;  // L * R * M
        blocks = (rows + kRowWarps - 1) / kRowWarps;
    }
    const int grid = persistent_grid(blocks, k, threads, smem, ctx);
    return launch("ep_combine_publish", k, dim3(grid), dim3(threads), smem, ctx, p);
}

cudaError_t launch_group_combine_reduce(GroupCombineParams p, const LaunchCtx& ctx) {
    // Rows of 6 tiles and more, once a block would have several tokens; the other kernel's block
    // has a row of up to 8 tiles in one pass, beyond that it has two and loses earlier (one rank on
    // this path, us per layer with it | without). 5 tiles: 2000 tokens to 2 26.1 | 25.7, to 8 43.8 |
    // 42.2. 6 tiles: to 1 800 tokens 18.2 | 18.5, 1200 21.2 | 22.7; to 4 800 21.9 | 21.5, 1200 26.4 | 27.4;
    // to 8 1200 35.5 | 35.2, 1600 42.5 | 42.4, 2000 49.5 | 54.2. 8 tiles: to 2 800 20.8 | 20.2, 1200 25.0 |
    // 25.5; to 4 1200 30.4 | 30.2, 1600 33.6 | 34.4; to 8 1200 42.0 | 41.1, 1600 51.1 | 54.6. 9 tiles: to 2
    // 300 17.4 | 18.0; to 8 300 22.8 | 22.5, 450 25.7 | 25.9, 600 32.3 | 30.7, 800 35.0 | 36.7. 14 tiles: to
    // 8 300 26.3 | 26.2, 600 37.7 | 39.4, 2000 100 | 111.
    const int tiles = (p.H + kTileChannels - 1) / kTileChannels;
    const bool last = layer_beyond_l2(p.T, p.K, p.H);
    if (tiles >= 6 && 2 * p.T > (tiles > 8 ? 6 : 12 + p.K) * ctx.num_sms) {
        const ReduceShape shape = reduce_shape(p.T, p.K, p.H, ctx.num_sms);
        p.tiles_per_block = shape.tiles_per_block, p.tokens_per_block = shape.tokens_per_block, p.span = shape.span;
        auto k = last ? ep_combine_gather_kernel<4, true> : ep_combine_gather_kernel<4, false>;
        return launch("ep_combine_reduce", k, shape.grid, dim3(shape.threads), 0, ctx, p);
    }
    const int threads = block_threads(p.H);
    auto k = last ? ep_combine_kernel<2, true> : ep_combine_kernel<2>;
    const int grid = persistent_grid(p.T, k, threads, 0, ctx);
    return launch("ep_combine_reduce", k, dim3(grid), dim3(threads), 0, ctx, p);
}

cudaError_t launch_barrier(const BarrierParams& p, const LaunchCtx& ctx) {
    LaunchCtx plain = ctx;
    plain.pdl = false;
    return launch("ep_barrier", ep_barrier_kernel, dim3(1), dim3(kMaxRanks), 0, plain, p);
}

cudaError_t launch_advance_seq(uint32_t* word, const LaunchCtx& ctx) {
    LaunchCtx plain = ctx;
    plain.pdl = false;  // ordinary stream order: after everything the call launched
    return launch("ep_advance_seq", ep_advance_seq_kernel, dim3(1), dim3(1), 0, plain, word);
}

// ---- in-process groups: all ranks in one cooperative launch ------------------------
namespace {

template <typename... KArgs, typename... Args>
cudaError_t launch_cooperative(const char* name, void (*kernel)(KArgs...), int grid, int threads,
                               size_t smem, const LaunchCtx& ctx, Args... args) {
    (void)name;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = ctx.stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t err = cudaLaunchKernelEx(&cfg, kernel, args...);
    if (err == cudaSuccess) g_launches.fetch_add(1);
    return err;
}

using DispatchMultiKernel = void (*)(const GroupDispatchParams*, int);

template <int kPhases>
DispatchMultiKernel pick_dispatch_multi(bool fp8, bool counting) {
    if (counting)
        return fp8 ? ep_dispatch_multi_kernel<true, true, kPhases> : ep_dispatch_multi_kernel<false, true, kPhases>;
    return fp8 ? ep_dispatch_multi_kernel<true, false, kPhases> : ep_dispatch_multi_kernel<false, false, kPhases>;
}

}  // namespace

cudaError_t launch_group_dispatch_multi(GroupDispatchParams* params, int n,
                                        GroupDispatchParams* dev_params, int phases,
                                        const LaunchCtx& ctx) {
    if (n < 1) return cudaSuccess;
    int want = 2;
    size_t smem = 0;
    bool counting = false;  // one rank that has no layout: all count (a layout is then left unused)
    for (int i = 0; i < n; ++i) {
        if (params[i].use_fp8 != params[0].use_fp8 || params[i].H != params[0].H) return cudaErrorInvalidValue;
        params[i].C = 1;
        counting = counting || params[i].counting();
        const int blocks = 1 + (params[i].T > 0 ? params[i].T : 1);
        if (blocks > want) want = blocks;
        const size_t sm = (size_t)(2 * params[i].E + 4) * sizeof(int);
        if (sm > smem) smem = sm;
    }
    const int threads = block_threads(params[0].H, 256);
    const bool fp8 = params[0].use_fp8 != 0;
    auto k = phases == 3 ? pick_dispatch_multi<3>(fp8, counting) : pick_dispatch_multi<1>(fp8, counting);
    const long long cap = resident_blocks(k, threads, smem, ctx) / n;
    if (cap < 2) return cudaErrorInvalidConfiguration;
    const int per_rank = (int)(want < cap ? want : cap);
    cudaError_t e = cudaMemcpyAsync(dev_params, params, sizeof(GroupDispatchParams) * n,
                                    cudaMemcpyHostToDevice, ctx.stream);
    if (e != cudaSuccess) return e;
    // (the copy reads pageable host memory: it has been staged when the call returns)
    return launch_cooperative("ep_dispatch_multi", k, per_rank * n, threads, smem, ctx,
                              (const GroupDispatchParams*)dev_params, per_rank);
}

cudaError_t launch_group_combine_multi(const GroupCombineParams* params, int n,
                                       GroupCombineParams* dev_params, const LaunchCtx& ctx) {
    if (n < 1) return cudaSuccess;
    int want = 64;
    size_t smem = 0;
    for (int i = 0; i < n; ++i) {
        if (params[i].H != params[0].H) return cudaErrorInvalidValue;
        if (params[i].T > want) want = params[i].T;
        const size_t sm = (size_t)(2 * params[i].E + 1) * sizeof(int);
        if (sm > smem) smem = sm;
    }
    const int threads = block_threads(params[0].H, 256);
    const long long cap = resident_blocks(ep_combine_multi_kernel, threads, smem, ctx) / n;
    if (cap < 1) return cudaErrorInvalidConfiguration;
    const int per_rank = (int)(want < cap ? want : cap);
    cudaError_t e = cudaMemcpyAsync(dev_params, params, sizeof(GroupCombineParams) * n,
                                    cudaMemcpyHostToDevice, ctx.stream);
    if (e != cudaSuccess) return e;
    return launch_cooperative("ep_combine_multi", ep_combine_multi_kernel, per_rank * n, threads,
                              smem, ctx, (const GroupCombineParams*)dev_params, per_rank);
}

}  // namespace mcep

#ifdef MCEP_PHASE_TRACE
// Diagnostic builds only: copies the trace of the calling thread's device out
// ([body 4][block 1024][slot 8] u64) after waiting for the device to go idle.
extern "C" int mcep_debug_read_phase_trace(unsigned long long* out, size_t bytes) {
    if (cudaDeviceSynchronize() != cudaSuccess) return -1;
    if (bytes > sizeof(mcep::kernels::g_phase_trace)) bytes = sizeof(mcep::kernels::g_phase_trace);
    return cudaMemcpyFromSymbol(out, mcep::kernels::g_phase_trace, bytes) == cudaSuccess ? 0 : -1;
}
#endif
