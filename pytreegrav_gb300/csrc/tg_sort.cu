// Device-wide exclusive scans and a stable LSD radix sort of (uint64 key, uint32 value) pairs.
//
// The sort replaces pytreegrav's _radix_argsort (octree.py:101-132). Any stable sort of the keys
// yields the same permutation, which is what makes the GPU order bit-identical to the reference.
// radix_sort_pairs is a one-sweep sort: digits of up to nine bits, one kernel per digit over tiles of 4096 or
// 6144 pairs, each tile's offsets by decoupled look-back (k_onesweep). The two-kernel passes with 8-bit digits and
// tiles of 4096 keys (radix_hist, radix_scatter; lanes of equal digits found by ballots, offsets from a digit-major
// scan) remain for the Morton order that allocates nothing (tg_noalloc.cu).
#include <algorithm>
#include <cstdio>
#include <mutex>
#include <vector>

#include "tg_common.cuh"

namespace tg {

static thread_local char g_err[512] = "";

void set_last_error(const char *where, cudaError_t e) {
    snprintf(g_err, sizeof(g_err), "%s: %s", where, cudaGetErrorString(e));
}
void set_last_error_msg(const char *msg) { snprintf(g_err, sizeof(g_err), "%s", msg); }
const char *last_error() { return g_err; }

int num_sms() {
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0) sms = 1;
    }
    return sms;
}

unsigned long long current_cuda_context_id() {
    using CtxGetCurrent = int (*)(void **);
    using CtxGetId = int (*)(void *, unsigned long long *);
    static CtxGetCurrent get = nullptr;
    static CtxGetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get = (CtxGetCurrent)p;
        p = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetId", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = (CtxGetId)p;
    });
    if (!get || !get_id) return 0;
    void *ctx = nullptr;
    if (get(&ctx) != 0) ctx = nullptr;
    if (!ctx) {  // none bound to this thread yet (or just reset): let the runtime bind its context
        cudaFree(nullptr);
        if (get(&ctx) != 0) ctx = nullptr;
    }
    unsigned long long id = 0;
    if (!ctx || get_id(ctx, &id) != 0) return 0;
    return id;
}

namespace {
constexpr int POOL_DEVICES = 64;
std::mutex g_res_mu;
// Per device: the context the pooled streams, events and page-locked words belong to, and the pools. After a
// device reset (a new context) the old handles are dropped, not reused.
struct ResPool {
    unsigned long long ctx = 0;  // context id
    std::vector<cudaStream_t> streams;
    std::vector<cudaEvent_t> events[2];  // [timing]
    std::vector<void *> words;           // HOST_WORDS_BYTES each
};
ResPool g_res[POOL_DEVICES];
int current_device() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= POOL_DEVICES) return -1;
    return dev;
}
// The pool of device dev for the current context (g_res_mu held).
ResPool &res_pool(int dev) {
    ResPool &r = g_res[dev];
    const unsigned long long ctx = current_cuda_context_id();
    if (ctx && !r.ctx) r.ctx = ctx;  // filled before the context could be identified
    if (ctx && r.ctx != ctx) {
        r.streams.clear();
        r.events[0].clear();
        r.events[1].clear();
        r.words.clear();
        r.ctx = ctx;
    }
    return r;
}
}  // namespace

int current_device_or(int fallback) {
    int dev = 0;
    return cudaGetDevice(&dev) == cudaSuccess ? dev : fallback;
}

cudaError_t pool_stream(cudaStream_t *s) {
    const int dev = current_device();
    if (dev >= 0) {
        std::lock_guard<std::mutex> lock(g_res_mu);
        ResPool &r = res_pool(dev);
        if (!r.streams.empty()) {
            *s = r.streams.back();
            r.streams.pop_back();
            return cudaSuccess;
        }
    }
    return cudaStreamCreateWithFlags(s, cudaStreamNonBlocking);
}

void release_stream(cudaStream_t s) {
    if (!s) return;
    int dev = -1;
    // pooled only on the current device, whose context the pool's key is checked against
    if (cudaStreamGetDevice(s, &dev) != cudaSuccess || dev < 0 || dev >= POOL_DEVICES || dev != current_device()) {
        cudaStreamDestroy(s);
        return;
    }
    std::lock_guard<std::mutex> lock(g_res_mu);
    res_pool(dev).streams.push_back(s);
}

cudaError_t pool_event(cudaEvent_t *e, bool timing) {
    const int dev = current_device();
    if (dev >= 0) {
        std::lock_guard<std::mutex> lock(g_res_mu);
        auto &v = res_pool(dev).events[timing ? 1 : 0];
        if (!v.empty()) {
            *e = v.back();
            v.pop_back();
            return cudaSuccess;
        }
    }
    return cudaEventCreateWithFlags(e, timing ? cudaEventDefault : cudaEventDisableTiming);
}

void release_event(cudaEvent_t e, bool timing, int dev) {
    if (!e) return;
    const int cur = current_device();
    if (dev < 0) dev = cur;
    if (dev < 0 || dev >= POOL_DEVICES || dev != cur) {  // pooled only on the current device (as streams)
        cudaEventDestroy(e);
        return;
    }
    std::lock_guard<std::mutex> lock(g_res_mu);
    res_pool(dev).events[timing ? 1 : 0].push_back(e);
}

tg_status HostWords::take() {
    if (p) return TG_OK;
    dev = current_device();
    if (dev >= 0) {
        std::lock_guard<std::mutex> lock(g_res_mu);
        auto &v = res_pool(dev).words;
        if (!v.empty()) {
            p = v.back();
            v.pop_back();
            return TG_OK;
        }
    }
    TG_CUDA(cudaHostAlloc(&p, HOST_WORDS_BYTES, cudaHostAllocDefault));
    return TG_OK;
}

HostWords::~HostWords() {
    if (!p) return;
    if (dev < 0 || dev != current_device()) {  // pooled only on the current device (as streams)
        cudaFreeHost(p);
        return;
    }
    std::lock_guard<std::mutex> lock(g_res_mu);
    res_pool(dev).words.push_back(p);
}

// The library's memory pool of the current device, made on first use.
static cudaError_t current_pool(cudaMemPool_t *pool) {
    constexpr int MAX_DEVICES = 64;
    static std::mutex mu;
    static cudaMemPool_t pools[MAX_DEVICES] = {};
    static unsigned long long pool_ctx[MAX_DEVICES] = {};  // context ids: a device reset makes a new context
    *pool = nullptr;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return e;
    std::lock_guard<std::mutex> lock(mu);
    const unsigned long long ctx = current_cuda_context_id();
    if (pools[dev] && ctx && !pool_ctx[dev]) pool_ctx[dev] = ctx;          // made before a context was bound
    if (pools[dev] && ctx && pool_ctx[dev] != ctx) pools[dev] = nullptr;  // the old pool died with its context
    if (!pools[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        e = cudaMemPoolCreate(&pools[dev], &props);
        if (e != cudaSuccess) {
            pools[dev] = nullptr;
            return e;
        }
        pool_ctx[dev] = current_cuda_context_id();
        size_t free_b = 0, total_b = 0;
        unsigned long long keep = TG_POOL_KEEP_BYTES;
        if (cudaMemGetInfo(&free_b, &total_b) == cudaSuccess && total_b / 4 > keep) keep = total_b / 4;
        e = cudaMemPoolSetAttribute(pools[dev], cudaMemPoolAttrReleaseThreshold, &keep);
        if (e != cudaSuccess) return e;
    }
    *pool = pools[dev];
    return cudaSuccess;
}

cudaError_t dev_malloc(void **p, size_t bytes, cudaStream_t s) {
    cudaMemPool_t pool;
    const cudaError_t e = current_pool(&pool);
    if (e != cudaSuccess) return e;
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, s) : cudaMallocAsync(p, bytes, s);
}

cudaError_t pool_bytes(int64_t *reserved, int64_t *used_high, bool reset) {
    *reserved = *used_high = 0;
    cudaMemPool_t pool;
    cudaError_t e = current_pool(&pool);
    if (e != cudaSuccess || !pool) return e;
    unsigned long long r = 0, h = 0, zero = 0;
    if ((e = cudaMemPoolGetAttribute(pool, cudaMemPoolAttrReservedMemCurrent, &r)) != cudaSuccess) return e;
    if ((e = cudaMemPoolGetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &h)) != cudaSuccess) return e;
    *reserved = (int64_t)r;
    *used_high = (int64_t)h;
    return reset ? cudaMemPoolSetAttribute(pool, cudaMemPoolAttrUsedMemHigh, &zero) : cudaSuccess;
}

// ---------------------------------------------------------------------------------------------
// Exclusive scan in one pass (decoupled look-back over tiles of 2048).
constexpr int SCAN_THREADS = 256;
constexpr int SCAN_ITEMS = 8;
constexpr int SCAN_TILE = SCAN_THREADS * SCAN_ITEMS;

template <typename T>
__device__ T block_exclusive_scan(T v, T *total) {
    __shared__ T warp_sums[SCAN_THREADS / 32];
    T inc = warp_inclusive_scan(v);
    int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    if (l == 31) warp_sums[w] = inc;
    __syncthreads();
    if (w == 0) {
        T s = (l < SCAN_THREADS / 32) ? warp_sums[l] : T(0);
        T si = warp_inclusive_scan(s);
        if (l < SCAN_THREADS / 32) warp_sums[l] = si - s;
        if (l == SCAN_THREADS / 32 - 1) *total = si;
    }
    __syncthreads();
    T r = warp_sums[w] + inc - v;
    __syncthreads();
    return r;
}

template <typename T>
__global__ void __launch_bounds__(SCAN_THREADS) k_scan(const T *in, T *out, int64_t n, T *total,
                                                       unsigned long long *status, int *counter, long long spins) {
    __shared__ T tot;
    __shared__ long long before_s;
    __shared__ int tile_s;
    if (threadIdx.x == 0) tile_s = atomicAdd(counter, 1);
    __syncthreads();
    const int tile = tile_s;
    const int64_t base = (int64_t)tile * SCAN_TILE + (int64_t)threadIdx.x * SCAN_ITEMS;
    T vals[SCAN_ITEMS];
    T v = 0;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        vals[i] = (base + i < n) ? in[base + i] : T(0);
        v += vals[i];
    }
    T ex = block_exclusive_scan(v, &tot);
    if (threadIdx.x < 32) {
        const long long before = scan_look_back((long long)tot, tile, status, spins, [&]() {
            long long sum = 0;
            for (int64_t i = threadIdx.x; i < (int64_t)tile * SCAN_TILE; i += 32) sum += in[i];
            for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(FULL, sum, o);
            return sum;
        });
        if (threadIdx.x == 0) {
            before_s = before;
            if (total && (int64_t)(tile + 1) * SCAN_TILE >= n) *total = (T)(before + (long long)tot);
        }
    }
    __syncthreads();
    ex += (T)before_s;
#pragma unroll
    for (int i = 0; i < SCAN_ITEMS; i++) {
        if (base + i < n) out[base + i] = ex;
        ex += vals[i];
    }
}

template <typename T>
static tg_status exclusive_scan(const T *in, T *out, int64_t n, T *total_dev, cudaStream_t s) {
    if (n <= 0) {
        if (total_dev) TG_CUDA(cudaMemsetAsync(total_dev, 0, sizeof(T), s));
        return TG_OK;
    }
    const int64_t nb = (n + SCAN_TILE - 1) / SCAN_TILE;
    unsigned long long *status = nullptr;  // then the tile counter
    TG_CUDA(tg::dev_malloc((void **)&status, sizeof(unsigned long long) * (nb + 1), s));
    TG_CUDA(cudaMemsetAsync(status, 0, sizeof(unsigned long long) * (nb + 1), s));
    { k_scan<T><<<(unsigned)nb, SCAN_THREADS, 0, s>>>(in, out, n, total_dev, status, (int *)(status + nb), scan_spins()); tg::note_launch(); }
    TG_CUDA(cudaGetLastError());
    TG_CUDA(cudaFreeAsync(status, s));
    return TG_OK;
}

tg_status exclusive_scan_i64(const int64_t *in, int64_t *out, int64_t n, int64_t *total_dev, cudaStream_t s) {
    return exclusive_scan<long long>((const long long *)in, (long long *)out, n, (long long *)total_dev, s);
}
tg_status exclusive_scan_i32(const int32_t *in, int32_t *out, int64_t n, cudaStream_t s) {
    return exclusive_scan<int>(in, out, n, nullptr, s);
}

// ---------------------------------------------------------------------------------------------
// Radix sort.
// RS_* (tile geometry of the two-kernel passes) are defined in tg_common.cuh.

// Per-warp stable ranking of the warp's ROUNDS * 32 keys; leaves per-warp digit counts in wcount.
// kv: the slice's keys, one per round, loaded here up front (one memory round trip per slice) and
// left to the caller.
template <int ROUNDS>
__device__ __forceinline__ void rank_loaded_slice(const uint64_t *kv, int64_t n, int64_t wbase, int shift,
                                                  int *wcount, int *digit, int *rank);

template <int ROUNDS = RS_ROUNDS>
__device__ __forceinline__ void rank_warp_slice(const uint64_t *keys, int64_t n, int64_t wbase, int shift,
                                                int *wcount, int *digit, int *rank, uint64_t *kv) {
    const int lane = lane_id();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int64_t i = wbase + r * 32 + lane;
        kv[r] = i < n ? __ldg(keys + i) : 0ull;
    }
    rank_loaded_slice<ROUNDS>(kv, n, wbase, shift, wcount, digit, rank);
}

template <int ROUNDS>
__device__ __forceinline__ void rank_loaded_slice(const uint64_t *kv, int64_t n, int64_t wbase, int shift,
                                                  int *wcount, int *digit, int *rank) {
    const int lane = lane_id();
    const unsigned lt = lanemask_lt();
    // every round's lanes with the same digit first, from nine ballots (the eight digit bits and
    // "in range"); independent of the counters, so the rounds overlap
    unsigned peers[ROUNDS];
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int64_t i = wbase + r * 32 + lane;
        const bool in = i < n;
        const int d = in ? (int)((kv[r] >> shift) & (RS_BINS - 1)) : RS_BINS;  // RS_BINS: past the end
        unsigned m = __ballot_sync(FULL, in);
        m = in ? m : ~m;
#pragma unroll
        for (int b = 0; b < 8; b++) {
            const bool bit = (d >> b) & 1;
            const unsigned v = __ballot_sync(FULL, bit);
            m &= bit ? v : ~v;
        }
        peers[r] = m;
        digit[r] = d;
    }
    // then the per-warp digit counters, round by round
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int d = digit[r];
        const int base = (d < RS_BINS) ? wcount[d] : 0;
        __syncwarp();
        if (d < RS_BINS && (31 - __clz(peers[r])) == lane) wcount[d] = base + __popc(peers[r]);
        __syncwarp();
        rank[r] = base + __popc(peers[r] & lt);
    }
}

__global__ void __launch_bounds__(RS_THREADS) radix_hist(const uint64_t *keys, int64_t n, int shift, int ntiles,
                                                         int *hist) {
    __shared__ int wcount[RS_WARPS][RS_BINS];
    for (int i = threadIdx.x; i < RS_WARPS * RS_BINS; i += RS_THREADS) (&wcount[0][0])[i] = 0;
    __syncthreads();
    int w = threadIdx.x >> 5;
    int64_t wbase = (int64_t)blockIdx.x * RS_TILE + (int64_t)w * RS_WARP_KEYS;
    int digit[RS_ROUNDS], rank[RS_ROUNDS];
    uint64_t kv[RS_ROUNDS];
    rank_warp_slice(keys, n, wbase, shift, wcount[w], digit, rank, kv);
    __syncthreads();
    for (int d = threadIdx.x; d < RS_BINS; d += RS_THREADS) {
        int s = 0;
#pragma unroll
        for (int ww = 0; ww < RS_WARPS; ww++) s += wcount[ww][d];
        hist[(int64_t)d * ntiles + blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(RS_THREADS) radix_scatter(const uint64_t *keys, const uint32_t *vals, int64_t n,
                                                            int shift, int ntiles, const int *offs,
                                                            uint64_t *keys_out, uint32_t *vals_out) {
    __shared__ int wcount[RS_WARPS][RS_BINS];
    for (int i = threadIdx.x; i < RS_WARPS * RS_BINS; i += RS_THREADS) (&wcount[0][0])[i] = 0;
    __syncthreads();
    int w = threadIdx.x >> 5;
    int64_t wbase = (int64_t)blockIdx.x * RS_TILE + (int64_t)w * RS_WARP_KEYS;
    int digit[RS_ROUNDS], rank[RS_ROUNDS];
    uint64_t kv[RS_ROUNDS];
    rank_warp_slice(keys, n, wbase, shift, wcount[w], digit, rank, kv);
    __syncthreads();
    // warp offsets within the tile, then the tile's global offset per digit
    for (int d = threadIdx.x; d < RS_BINS; d += RS_THREADS) {
        int run = offs[(int64_t)d * ntiles + blockIdx.x];
#pragma unroll
        for (int ww = 0; ww < RS_WARPS; ww++) {
            int c = wcount[ww][d];
            wcount[ww][d] = run;
            run += c;
        }
    }
    __syncthreads();
    const int lane = lane_id();
#pragma unroll
    for (int r = 0; r < RS_ROUNDS; r++) {
        int64_t i = wbase + r * 32 + lane;
        if (i < n) {
            int pos = wcount[w][digit[r]] + rank[r];
            keys_out[pos] = kv[r];
            vals_out[pos] = vals[i];
        }
    }
}

// ---------------------------------------------------------------------------------------------
// One-sweep passes (decoupled look-back). All digit histograms come from one read of the keys;
// then each pass is one kernel: a CTA takes the next tile from an atomic counter (so every earlier
// tile belongs to a CTA that is already running), ranks its keys stably as above, publishes its
// per-digit count, orders its tile by digit in shared memory, looks back over earlier tiles' published words for
// its exclusive prefix, and writes the tile out. A look-back spin is bounded; running out sets the sort's own
// error word instead of hanging, and the sort then leaves the identity permutation (k_sort_fallback).
// Digits have up to nine bits (63 key bits: seven passes; a sort's bits are shared out evenly over its passes).
// The passes follow the published one-sweep method (Adinets and Merrill, "Onesweep: A Faster Least Significant Digit
// Radix Sort for GPUs", 2022); that a warp finds its lanes of equal digits by an OR of lane masks into a word per digit
// is likewise a known way of GPU radix ranking, in place of a match instruction.
// A pass is bound by the chain of one tile (load, rank, publish, look back, write) with the ~300 tiles that fit the
// SMs, a third of the copy bandwidth: hence few instructions per key (lanes of equal digits find one another by
// an OR into a word per digit, ~12 instructions where ballots over the digit's bits took ~45) and the tile's own
// reordering before the look-back, which then finds its predecessors further on. Tiles of 512 threads x 8
// keys: Morton order of 1e6 points 264 us, 8e6 940 us (ballots, 8-bit digits, 256 threads x 8: 298 and 1136;
// this kernel with 8-bit digits 256 and 963, but slower builds below 1e6). From LONG_SORT pairs 12 keys per thread:
// longer runs of a digit to write (8e6 points 879 us; 1e6 266).

constexpr int OS_BITS = 9, OS_BINS = 1 << OS_BITS;
constexpr int MAX_PASSES = (64 + OS_BITS - 1) / OS_BITS;
constexpr int OS_WARPS = 16, OS_THREADS = OS_WARPS * 32;
static_assert(OS_THREADS == OS_BINS, "a thread per digit");
constexpr int64_t LONG_SORT = 3 << 20;
template <int ROUNDS>  // keys per thread
struct OsTile {
    static constexpr int WARP_KEYS = ROUNDS * 32, KEYS = OS_WARPS * WARP_KEYS;
};
// A status word: flag (bits 62-63: aggregate or inclusive), the pass it belongs to (bits 56-61, pass + 1),
// value (bits 0-55). Words of an earlier pass read as not yet published, so the status array is
// cleared once per sort rather than once per pass.
constexpr unsigned long long ST_AGG = 1ull << 62, ST_INC = 2ull << 62, ST_FLAGS = 3ull << 62;
constexpr unsigned long long ST_TAGS = 63ull << 56, ST_VAL = (1ull << 56) - 1;
constexpr long long SPIN_LIMIT = 1ll << 22;
constexpr int LB = 4;  // predecessors read per look-back round trip

// Every pass's digit histogram from one read of the keys; the last block to finish scans each pass's counts
// in place (exclusive), which took a launch of its own.
constexpr int HIST_THREADS = OS_BINS / 2;
__global__ void __launch_bounds__(HIST_THREADS) k_sort_hist(const uint64_t *keys, int64_t n, int npass, int width,
                                                            int *hist, int *done) {
    __shared__ int h[MAX_PASSES * OS_BINS];
    __shared__ int tot[MAX_PASSES * HIST_THREADS / 32];
    __shared__ bool last;
    chain_wait();
    chain_next();
    for (int i = threadIdx.x; i < npass * OS_BINS; i += HIST_THREADS) h[i] = 0;
    __syncthreads();
    const unsigned mask = (1u << width) - 1;
    for (int64_t i = (int64_t)blockIdx.x * HIST_THREADS + threadIdx.x; i < n; i += (int64_t)gridDim.x * HIST_THREADS) {
        const uint64_t k = keys[i];
        for (int p = 0; p < npass; p++) atomicAdd(&h[p * OS_BINS + ((unsigned)(k >> (width * p)) & mask)], 1);
    }
    __syncthreads();
    for (int i = threadIdx.x; i < npass * OS_BINS; i += HIST_THREADS)
        if (h[i]) atomicAdd(&hist[i], h[i]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(done, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int lane = lane_id(), w = threadIdx.x >> 5;
    int2 v[MAX_PASSES];
    int inc[MAX_PASSES];
#pragma unroll
    for (int p = 0; p < MAX_PASSES; p++) {
        if (p >= npass) break;
        v[p] = __ldcg(reinterpret_cast<const int2 *>(hist + p * OS_BINS) + threadIdx.x);
        inc[p] = warp_inclusive_scan(v[p].x + v[p].y);
        if (lane == 31) tot[p * (HIST_THREADS / 32) + w] = inc[p];
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < MAX_PASSES; p++) {
        if (p >= npass) break;
        int below = inc[p] - v[p].x - v[p].y;
        for (int k = 0; k < w; k++) below += tot[p * (HIST_THREADS / 32) + k];
        reinterpret_cast<int2 *>(hist + p * OS_BINS)[threadIdx.x] = make_int2(below, below + v[p].x);
    }
}

template <int ROUNDS>
struct alignas(16) OsSmem {
    unsigned short wcount[OS_WARPS][OS_BINS];  // a warp's digit counts, then its first positions within the tile
    int prefix[OS_BINS];                       // the digit's place in the output, less lstart
    int warp_sum[OS_WARPS];
    int tile;
    union alignas(16) {  // cleared 16 bytes at a time
        unsigned peers[OS_WARPS][OS_BINS];  // while ranking: a warp's lanes with the digit
        struct {
            uint64_t key[OsTile<ROUNDS>::KEYS];  // the tile in digit order
            uint32_t val[OsTile<ROUNDS>::KEYS];
        };
    };
};
template <int ROUNDS>
__global__ void __launch_bounds__(OS_THREADS, 2)
    k_onesweep(const uint64_t *keys, const uint32_t *vals, int64_t n, int shift, int width, int pass, const int *digit_off,
               unsigned long long *status, int *tile_counter, uint64_t *keys_out, uint32_t *vals_out, int *err,
               long long spin_limit) {
    const unsigned long long tag = (unsigned long long)(pass + 1) << 56;
    extern __shared__ __align__(16) unsigned char os_raw[];
    OsSmem<ROUNDS> &sm = *reinterpret_cast<OsSmem<ROUNDS> *>(os_raw);
    constexpr int TILE = OsTile<ROUNDS>::KEYS;
    chain_wait();
    chain_next();
    if (threadIdx.x == 0) sm.tile = atomicAdd(tile_counter, 1);
    const int w = threadIdx.x >> 5, lane = lane_id();
    const unsigned lt = lanemask_lt(), mask = (1u << width) - 1;
    unsigned short *wc = sm.wcount[w];
    unsigned *peers = sm.peers[w];
    for (int i = lane; i < OS_BINS / 8; i += 32) reinterpret_cast<uint4 *>(wc)[i] = make_uint4(0, 0, 0, 0);
    for (int i = lane; i < OS_BINS / 4; i += 32) reinterpret_cast<uint4 *>(peers)[i] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const int t = sm.tile;
    const int64_t tbase = (int64_t)t * TILE;
    const int cnt = n - tbase < TILE ? (int)(n - tbase) : TILE;
    const int wofs = w * OsTile<ROUNDS>::WARP_KEYS + lane;
    const uint64_t *kp = keys + tbase;
    const uint32_t *vp = vals + tbase;
    int place[ROUNDS];  // rank within the warp's keys of the digit (low half), the digit (high half)
    uint64_t kv[ROUNDS];
    uint32_t vv[ROUNDS];  // values loaded with the keys, so the scatter reads nothing from memory
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int i = wofs + r * 32;
        kv[r] = i < cnt ? kp[i] : 0ull;  // coherent loads: the pass before may still write when this kernel starts
        vv[r] = i < cnt ? vp[i] : 0u;
    }
    // ranks round by round: the lanes of one digit find one another through a word per digit
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const bool in = wofs + r * 32 < cnt;
        const int d = (int)((unsigned)(kv[r] >> shift) & mask);
        if (in) atomicOr(&peers[d], 1u << lane);
        __syncwarp();
        unsigned m = 0;
        int base = 0;
        if (in) {
            m = peers[d];
            base = wc[d];
        }
        __syncwarp();
        if (in && (31 - __clz(m)) == lane) {
            peers[d] = 0;
            wc[d] = (unsigned short)(base + __popc(m));
        }
        __syncwarp();
        place[r] = d << 16 | (base + __popc(m & lt));
    }
    __syncthreads();
    // a thread per digit: its counts per warp become the warps' first places within the tile
    const int d = threadIdx.x;
    int run = 0;
#pragma unroll
    for (int ww = 0; ww < OS_WARPS; ww++) run += sm.wcount[ww][d];
    volatile unsigned long long *st = status + (int64_t)t * OS_BINS + d;
    *st = (t == 0 ? ST_INC : ST_AGG) | tag | (unsigned long long)run;
    const int inc = warp_inclusive_scan(run);
    if (lane == 31) sm.warp_sum[w] = inc;
    __syncthreads();
    int start = inc - run;
#pragma unroll
    for (int ww = 0; ww < OS_WARPS; ww++) start += ww < w ? sm.warp_sum[ww] : 0;
    int first = start;
#pragma unroll
    for (int ww = 0; ww < OS_WARPS; ww++) {
        const int c = sm.wcount[ww][d];
        sm.wcount[ww][d] = (unsigned short)first;
        first += c;
    }
    __syncthreads();
    // the tile in digit order in shared memory, then written out: keys of one digit go to consecutive
    // places, so consecutive threads write consecutive words instead of one scattered sector each
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        if (wofs + r * 32 < cnt) {
            const int loc = wc[place[r] >> 16] + (place[r] & 0xffff);
            sm.key[loc] = kv[r];
            sm.val[loc] = vv[r];
        }
    }
    // earlier tiles publish their counts without waiting on anyone, so each wait ends once that tile's CTA
    // (already running: it took its tile before this one) has ranked. The words of LB predecessors are read
    // together (independent loads, one round trip), then summed in order up to the first inclusive one.
    long long acc = 0;
    bool done = false;
    for (int64_t j = t - 1; j >= 0 && !done; j -= LB) {
        unsigned long long word[LB];
#pragma unroll
        for (int k = 0; k < LB; k++)
            word[k] = j - k >= 0 ? ((const volatile unsigned long long *)status)[(j - k) * OS_BINS + d] : 0ull;
#pragma unroll
        for (int k = 0; k < LB; k++) {
            if (done || j - k < 0) break;
            unsigned long long wd = word[k];
            const volatile unsigned long long *src = status + (j - k) * OS_BINS + d;
            auto ready = [tag](unsigned long long x) { return (x & ST_FLAGS) && (x & ST_TAGS) == tag; };
            for (long long spins = 0; !ready(wd) && spins < spin_limit; spins++) wd = *src;
            if (!ready(wd)) {
                atomicExch(err, 1);
                done = true;
                break;
            }
            acc += (long long)(wd & ST_VAL);
            if ((wd & ST_FLAGS) == ST_INC) done = true;
        }
    }
    if (t > 0) *st = ST_INC | tag | (unsigned long long)(acc + run);
    sm.prefix[d] = digit_off[d] + (int)acc - start;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ROUNDS; r++) {
        const int i = r * OS_THREADS + threadIdx.x;
        if (i >= cnt) break;
        const uint64_t k = sm.key[i];
        const unsigned pos = (unsigned)(sm.prefix[(unsigned)(k >> shift) & mask] + i);
        if (pos >= (unsigned)n) continue;  // only after a look-back that gave up (garbage keys)
        keys_out[pos] = k;
        vals_out[pos] = sm.val[i];
    }
}

// After the passes: if a look-back gave up (some keys went to wrong places, some places were never
// written), every value becomes its own index and every key its own position -- sorted pairs and a
// valid permutation, so every later kernel sees well-formed input -- and the caller's flag is set.
__global__ void k_sort_fallback(uint64_t *keys, uint32_t *vals, int64_t n, const int *local_err, int *err) {
    chain_wait();
    chain_next();
    if (!*local_err) return;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i0 == 0) atomicExch(err, 1);
    for (int64_t i = i0; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        keys[i] = (uint64_t)i;
        vals[i] = (uint32_t)i;
    }
}

long long scan_spins() { return loop_limits().sort_spin > 0 ? loop_limits().sort_spin : SPIN_LIMIT; }

tg_status radix_sort_pairs(uint64_t *keys, uint32_t *vals, int64_t n, int bits, cudaStream_t s, int *err,
                           bool caller_falls_back, SortedPairs *left) {
    if (left) {
        left->keys = keys;
        left->vals = vals;
    }
    if (n <= 1 || bits <= 0) return TG_OK;
    if (n > (int64_t)0x7fffffff || !err) return TG_ERR_BAD_ARG;
    const long long spin_limit = loop_limits().sort_spin > 0 ? loop_limits().sort_spin : SPIN_LIMIT;
    const bool lng = n >= LONG_SORT;
    const int ntiles = div_up(n, lng ? OsTile<12>::KEYS : OsTile<8>::KEYS);
    const int npass = (bits + OS_BITS - 1) / OS_BITS, width = (bits + npass - 1) / npass;
    // one allocation: status words, histograms, tile counters, the histogram's and the error word (zeroed), then
    // the other halves of the key and value buffers
    const size_t st_bytes = sizeof(unsigned long long) * (size_t)ntiles * OS_BINS;
    const size_t hist_bytes = sizeof(int) * MAX_PASSES * OS_BINS;
    const size_t head = (st_bytes + hist_bytes + sizeof(int) * (MAX_PASSES + 2) + 255) / 256 * 256;
    const size_t key_bytes = (sizeof(uint64_t) * (size_t)n + 255) / 256 * 256;
    DevArray<unsigned char> own(s), &mem = left ? left->mem : own;
    mem.reset();
    TG_CUDA(mem.alloc((int64_t)(head + key_bytes + sizeof(uint32_t) * (size_t)n)));
    unsigned char *scr = mem.p;
    unsigned long long *status = (unsigned long long *)scr;
    int *hist = (int *)(scr + st_bytes);
    int *counters = hist + MAX_PASSES * OS_BINS;
    int *done = counters + MAX_PASSES;
    int *local_err = caller_falls_back ? err : done + 1;
    uint64_t *k2 = (uint64_t *)(scr + head);
    uint32_t *v2 = (uint32_t *)(scr + head + key_bytes);
    TG_CUDA(cudaMemsetAsync(scr, 0, head, s));
    const int hblocks = (int)std::min<int64_t>(div_up(n, HIST_THREADS * 4), (int64_t)num_sms() * 4);
    TG_CHAIN(k_sort_hist, hblocks, HIST_THREADS, 0, s, keys, n, npass, width, hist, done);
    auto pass = lng ? k_onesweep<12> : k_onesweep<8>;
    const int smem = lng ? (int)sizeof(OsSmem<12>) : (int)sizeof(OsSmem<8>);
    TG_CUDA(cudaFuncSetAttribute(pass, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    uint64_t *kin = keys, *kout = k2;
    uint32_t *vin = vals, *vout = v2;
    for (int p = 0; p < npass; p++) {
        TG_CHAIN(pass, ntiles, OS_THREADS, smem, s, kin, vin, n, width * p, width, p, hist + p * OS_BINS, status,
                 counters + p, kout, vout, local_err, spin_limit);
        uint64_t *tk = kin; kin = kout; kout = tk;
        uint32_t *tv = vin; vin = vout; vout = tv;
    }
    TG_CUDA(cudaGetLastError());
    if (left) {
        left->keys = kin;
        left->vals = vin;
    } else if (kin != keys) {
        TG_CUDA(cudaMemcpyAsync(keys, kin, sizeof(uint64_t) * n, cudaMemcpyDeviceToDevice, s));
        TG_CUDA(cudaMemcpyAsync(vals, vin, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, s));
        kin = keys;
        vin = vals;
    }
    if (!caller_falls_back) TG_CHAIN(k_sort_fallback, std::min(div_up(n, 256), 4 * num_sms()), 256, 0, s, kin, vin, n,
                                     local_err, err);
    TG_CUDA(cudaGetLastError());
    return TG_OK;
}

}  // namespace tg
