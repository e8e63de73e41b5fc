// sort.cu -- stable LSD radix sort of (cell hash, particle index) pairs.
//
// Replaces thrust::sort_by_key in sortParticles (DamBreak.Core/fluidSystem.cu:94-99,
// Poiseuille.Core/poiseuilleFlowSystem.cu:103-108, PeristalsisSystem.cu:116-121).
// One kernel launch per 8-bit digit, following the single-pass "onesweep" scheme
// of Adinets & Merrill (2022):
//   * the digit histograms of every pass come from one read of the keys;
//   * each CTA takes the next tile from an atomic counter, ranks its keys with a
//     warp-level multisplit, publishes its per-digit counts and resolves its global
//     offsets by decoupled look-back over earlier tiles, in two levels;
//   * ranks follow input order inside a warp, warps follow each other inside a
//     tile and tiles follow tile order, so the sort is stable and equals a stable
//     sort by key -- bit-identical to the reference's thrust result.
// Every look-back wait is bounded: after g_spin_limit polls (kSpinLimit unless a
// test lowered it) the CTA records CMAG_DEVERR_LOOKBACK_TIMEOUT, treats the
// missing counts as zero and finishes; its scatter then writes only positions
// below n (underestimated offsets stay in range) and flags any other as
// CMAG_DEVERR_RANGE.
#include <cuda_runtime.h>

#include <cstdio>
#include <cstring>
#include <mutex>

#include "kernels.h"

namespace cmag {

namespace {

constexpr uint32_t kFlagAgg = 1u << 30;     // tile aggregate published
constexpr uint32_t kFlagPrefix = 2u << 30;  // inclusive prefix published
constexpr uint32_t kCountMask = (1u << 30) - 1u;
constexpr int kSpinLimit = 1 << 22;
// polls before a look-back wait gives up (cmag_testing_set_sort_spin_limit)
__device__ int g_spin_limit = kSpinLimit;
constexpr int kWarps = kSortThreads / 32;
constexpr uint32_t kInvalidDigit = 256;
constexpr int kGroup = 16;  // tiles of a look-back group
constexpr int kReads = 16;  // group words a lane reads per look-back round (two lanes a digit)

__device__ __forceinline__ uint32_t lanemask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Lanes of the warp whose digit (9 bits with the invalid one) equals this lane's: nine
// ballots take half the time of __match_any_sync here.
__device__ __forceinline__ uint32_t same_digit(uint32_t d)
{
    uint32_t peers = 0xffffffffu;
#pragma unroll
    for (int b = 0; b < 9; ++b) {
        const bool bit = (d >> b) & 1u;
        const uint32_t set = __ballot_sync(0xffffffffu, bit);
        peers &= bit ? set : ~set;
    }
    return peers;
}

// exclusive scan of one value per thread over the block
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t *s_warp)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t wbase = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) wbase += (w < warp) ? s_warp[w] : 0u;
    __syncthreads();
    return wbase + x - v;
}

// Digit histograms of every pass; the same blocks clear the look-back status of the
// passes and, where ckeys is given, copy the pairs (a sort of an odd number of passes
// starts from the copy, so that its result lands in the caller's arrays).
__global__ void __launch_bounds__(256) k_digit_hist(const uint32_t *__restrict__ keys, uint32_t n,
                                                    int passes, uint32_t *__restrict__ hist,
                                                    uint4 *__restrict__ status, uint32_t status_words4,
                                                    const uint32_t *__restrict__ vals, uint32_t *__restrict__ ckeys,
                                                    uint32_t *__restrict__ cvals)
{
    __shared__ uint32_t s_hist[kMaxPasses * kRadix];
    for (int b = threadIdx.x; b < passes * kRadix; b += blockDim.x) s_hist[b] = 0;
    __syncthreads();
    const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, step = gridDim.x * blockDim.x;
    for (uint32_t i = tid; i < status_words4; i += step) status[i] = make_uint4(0, 0, 0, 0);
    for (uint32_t i0 = tid; i0 < n; i0 += 4 * step) {  // four loads in flight
        uint32_t k[4], v[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t i = i0 + u * step;
            k[u] = i < n ? keys[i] : 0u;
            v[u] = i < n && ckeys ? vals[i] : 0u;
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t i = i0 + u * step;
            if (i >= n) break;
            if (ckeys) {
                ckeys[i] = k[u];
                cvals[i] = v[u];
            }
            for (int ps = 0; ps < passes; ++ps) atomicAdd(&s_hist[ps * kRadix + ((k[u] >> (8 * ps)) & 255u)], 1u);
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < passes * kRadix; b += blockDim.x)
        if (s_hist[b]) atomicAdd(&hist[b], s_hist[b]);
}

// Published words of one lane pair's digit: reads `mine` of the up to kReads words
// st[first - half * kReads - k] (k < kReads, none below `low`), nearest first, and adds
// up both lanes' published counts up to the first inclusive prefix or the first word not
// yet published.
struct LookBack {
    uint32_t add;
    int used;   // words consumed by the pair
    bool done;  // reached a prefix (or the words below `low`, which count as one)
};
__device__ __forceinline__ LookBack look_back(const volatile uint32_t *st, uint32_t d, int first, int low)
{
    const int lane = threadIdx.x & 31, half = lane & 1;
    uint32_t v[kReads];
#pragma unroll
    for (int k = 0; k < kReads; ++k) {
        const int q = first - half * kReads - k;
        v[k] = q >= low ? (uint32_t)st[(size_t)q * kRadix + d] : (uint32_t)kFlagPrefix;
    }
    uint32_t add = 0;
    int used = 0;
    bool stop = false, done = false;
#pragma unroll
    for (int k = 0; k < kReads; ++k) {
        if (!stop) {
            if (v[k] & (kFlagAgg | kFlagPrefix)) {
                add += v[k] & kCountMask;
                ++used;
                if (v[k] & kFlagPrefix) stop = done = true;
            } else {
                stop = true;
            }
        }
    }
    // the farther lane's words count when the nearer lane consumed all of its own
    const uint32_t pair = 3u << (lane & ~1);
    const uint32_t o_add = __shfl_xor_sync(pair, add, 1);
    const int o_used = __shfl_xor_sync(pair, used, 1);
    const int flags = (stop ? 1 : 0) | (done ? 2 : 0);
    const int o_flags = __shfl_xor_sync(pair, flags, 1);
    const int near_flags = half ? o_flags : flags, far_flags = half ? flags : o_flags;
    if (near_flags & 1) return {half ? o_add : add, half ? o_used : used, (near_flags & 2) != 0};
    return {add + o_add, used + o_used, (far_flags & 2) != 0};
}

// The counts of digit d in the words low .. first, waiting for those not yet published.
__device__ __forceinline__ uint32_t sum_back(const volatile uint32_t *st, uint32_t d, int first, int low,
                                             int spin_limit, uint32_t *err)
{
    uint32_t sum = 0;
    for (int spins = 0; first >= low;) {  // the same trips for both lanes of a digit
        const LookBack b = look_back(st, d, first, low);
        sum += b.add;
        if (b.done) break;
        first -= b.used;
        if (b.used == 0) {
            if (++spins > spin_limit) {
                set_error(err, CMAG_DEVERR_LOOKBACK_TIMEOUT);
                break;  // give up: the rest counts as zero
            }
            if (spins > 8) __nanosleep(64);
        }
    }
    return sum;
}

// One digit's pass.  Bound by latency: a tile's loads, the chain of its ranking steps,
// and the look-back, whose every round trip to other tiles' words takes about 1.2 us.
//   * Tiles as large as leave every SM one (up to 8 pairs a thread; sort_items): two
//     blocks on an SM cost each other far more than the second hides, because the one
//     that waits polls (ranking 12 us beside a waiting block, 2 us alone).
//   * The look-back has two levels: a tile adds the words of its group of 16 tiles, and
//     the groups' words before it (the group's last tile publishes its sum, then its
//     inclusive prefix): two or three round trips, where looking back tile by tile took
//     ten to twelve.
//   * The pairs are put in digit order in shared memory and written as runs.
// 954,860 pairs of 23 bits: 25.7 -> 17-20 us a pass (ncu), the whole call 144-153 ->
// 97-105 us (boxes differ); 4 million of 30 bits 392 -> 288 us, 2,000 of 12 bits 62 -> 56 us.
template <int kItems>
__global__ void __launch_bounds__(kSortThreads, 1)
    k_onesweep(const uint32_t *__restrict__ kin, const uint32_t *__restrict__ vin,
               uint32_t *__restrict__ kout, uint32_t *__restrict__ vout, uint32_t n, int shift,
               const uint32_t *__restrict__ hist, uint32_t *tile_ctr, uint32_t *status,
               uint32_t *group_status, uint32_t *err)
{
    constexpr uint32_t kTile = kSortThreads * kItems;  // pairs of a tile
    extern __shared__ uint32_t s_pairs[];  // keys, then values, of the tile in digit order
    uint32_t *const s_key = s_pairs, *const s_val = s_pairs + kTile;
    __shared__ uint32_t s_whist[kWarps][kRadix];  // per-warp digit counts -> offsets
    __shared__ uint32_t s_base[kRadix];           // global start of each digit in this tile
    __shared__ uint32_t s_run[kRadix];            // the tile's count of each digit
    __shared__ uint32_t s_first[kRadix];          // first place of each digit in the tile
    __shared__ uint32_t s_quarter[4][kRadix];     // counts of a quarter of the warps
    __shared__ uint32_t s_scan[kWarps];
    __shared__ uint32_t s_tile;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr, 1u);
    const uint32_t count = threadIdx.x < kRadix ? hist[threadIdx.x] : 0u;
    for (int b = threadIdx.x; b < kWarps * kRadix; b += kSortThreads) (&s_whist[0][0])[b] = 0;
    __syncthreads();
    const uint32_t tile = s_tile;

    const uint32_t chunk = tile * kTile + (uint32_t)warp * (32u * kItems);
    uint32_t key[kItems], val[kItems], off[kItems];
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        uint32_t i = chunk + (uint32_t)it * 32u + (uint32_t)lane;
        if (i < n) {
            key[it] = kin[i];
            val[it] = vin[i];
        } else {
            key[it] = 0xffffffffu;
            val[it] = 0;
        }
    }
    // digit offsets of this pass, while the pairs load: exclusive scan of the histogram
    const uint32_t digit_start = block_exclusive_scan(count, s_scan);
    const uint32_t lt = lanemask_lt();
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        uint32_t i = chunk + (uint32_t)it * 32u + (uint32_t)lane;
        uint32_t d = (i < n) ? ((key[it] >> shift) & 255u) : kInvalidDigit;
        const uint32_t peers = same_digit(d);
        uint32_t before = 0;
        if (d != kInvalidDigit) before = s_whist[warp][d];
        __syncwarp();
        if (d != kInvalidDigit && lane == __ffs(peers) - 1) s_whist[warp][d] = before + __popc(peers);
        __syncwarp();
        off[it] = before + __popc(peers & lt);
    }
    __syncthreads();

    // four threads own a digit, a quarter of the warps each: warp-exclusive offsets and
    // the tile total, published
    volatile uint32_t *st = status, *gst = group_status;
    {
        constexpr int kQuarter = kWarps / 4;
        const uint32_t d = threadIdx.x % kRadix, q = threadIdx.x / kRadix;
        uint32_t c[kQuarter], run = 0;
#pragma unroll
        for (int w = 0; w < kQuarter; ++w) {
            const uint32_t v = s_whist[q * kQuarter + w][d];
            c[w] = run;
            run += v;
        }
        s_quarter[q][d] = run;
        __syncthreads();
        uint32_t before = 0;
        for (uint32_t k = 0; k < q; ++k) before += s_quarter[k][d];
        if (q == 3) {
            st[(size_t)tile * kRadix + d] = kFlagAgg | (before + run);
            s_run[d] = before + run;
        }
#pragma unroll
        for (int w = 0; w < kQuarter; ++w) s_whist[q * kQuarter + w][d] = before + c[w];
    }
    if (threadIdx.x < kRadix) s_base[threadIdx.x] = digit_start;
    __syncthreads();
    const uint32_t place = block_exclusive_scan(threadIdx.x < kRadix ? s_run[threadIdx.x] : 0u, s_scan);
    if (threadIdx.x < kRadix) s_first[threadIdx.x] = place;
    __syncthreads();
    // the pairs in digit order
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        if (chunk + (uint32_t)it * 32u + (uint32_t)lane >= n) continue;
        const uint32_t d = (key[it] >> shift) & 255u;
        const uint32_t at = s_first[d] + s_whist[warp][d] + off[it];
        s_key[at] = key[it];
        s_val[at] = val[it];
    }
    // threads 2d and 2d + 1 look back for digit d
    if (threadIdx.x < 2 * kRadix) {
        const uint32_t d = threadIdx.x >> 1;
        const int spin_limit = g_spin_limit;
        const int group = (int)tile / kGroup, begin = group * kGroup;
        uint32_t exclusive = 0;
        if ((int)tile > begin) exclusive = sum_back(st, d, (int)tile - 1, begin, spin_limit, err);
        const bool last = (int)tile == begin + kGroup - 1;  // the group's (an unfinished group has no reader)
        const uint32_t total = exclusive + s_run[d];
        if (last && !(threadIdx.x & 1)) gst[(size_t)group * kRadix + d] = (group ? kFlagAgg : kFlagPrefix) | total;
        if (group > 0) {
            const uint32_t before = sum_back(gst, d, group - 1, 0, spin_limit, err);
            if (last && !(threadIdx.x & 1)) gst[(size_t)group * kRadix + d] = kFlagPrefix | (before + total);
            exclusive += before;
        }
        if (!(threadIdx.x & 1)) s_base[d] += exclusive;
    }
    __syncthreads();

    const uint32_t in_tile = min(kTile, n - tile * kTile);
#pragma unroll
    for (int it = 0; it < kItems; ++it) {
        const uint32_t at = (uint32_t)it * kSortThreads + threadIdx.x;
        if (at >= in_tile) continue;
        const uint32_t k = s_key[at], d = (k >> shift) & 255u;
        const uint32_t o = s_base[d] + (at - s_first[d]);
        if (o < n) {  // always true unless a look-back gave up
            kout[o] = k;
            vout[o] = s_val[at];
        } else {
            set_error(err, CMAG_DEVERR_RANGE);
        }
    }
}

}  // namespace

namespace {
// look-back words of one pass: every tile's, then every group's
size_t status_words(uint32_t n)
{
    const size_t tiles = sort_tiles(n);
    return (tiles + (tiles + kGroup - 1) / kGroup) * kRadix;
}
}  // namespace

size_t sort_head_words() { return (size_t)kMaxPasses * kRadix + kMaxPasses; }

size_t sort_workspace_words(uint32_t n, int passes)
{
    return sort_head_words() + (size_t)(passes > 0 ? passes : 1) * status_words(n);
}

SortWorkspace sort_workspace_view(uint32_t *base, uint32_t n)
{
    SortWorkspace ws;
    ws.hist = base;
    ws.tile_ctr = base + kMaxPasses * kRadix;
    ws.status = ws.tile_ctr + kMaxPasses;
    (void)n;
    return ws;
}

namespace {

// A plain launch that returns its own error (not one that the caller left pending).
template <typename... KArgs, typename... Args>
cudaError_t launch(void (*kernel)(KArgs...), uint32_t blocks, uint32_t threads, size_t smem, cudaStream_t st,
                   Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = blocks;
    cfg.blockDim = threads;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

cudaError_t launch_digit_hist(const uint32_t *keys, uint32_t n, int passes, const SortWorkspace &ws,
                              const uint32_t *vals, uint32_t *ckeys, uint32_t *cvals, cudaStream_t st)
{
    uint32_t blocks = (n + 2047) / 2048;
    const uint32_t cap = 8u * (uint32_t)device_sm_count();  // 8 blocks per SM
    if (blocks > cap) blocks = cap;
    const uint32_t status_words4 = (uint32_t)((size_t)passes * status_words(n) / 4);
    return launch(k_digit_hist, blocks, 256, 0, st, keys, n, passes, ws.hist, reinterpret_cast<uint4 *>(ws.status),
                  status_words4, vals, ckeys, cvals);
}

template <int kItems>
cudaError_t launch_pass(const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout, uint32_t n, int pass,
                        const SortWorkspace &ws, uint32_t *err, cudaStream_t st)
{
    constexpr int bytes = 2 * kSortThreads * kItems * (int)sizeof(uint32_t);  // a tile's pairs
    if (pass == 0) {
        const cudaError_t e =
            cudaFuncSetAttribute(k_onesweep<kItems>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        if (e != cudaSuccess) return e;
    }
    const uint32_t tiles = sort_tiles(n);
    uint32_t *status = ws.status + (size_t)pass * status_words(n);
    return launch(k_onesweep<kItems>, tiles, kSortThreads, bytes, st, kin, vin, kout, vout, n, 8 * pass,
                  ws.hist + pass * kRadix, ws.tile_ctr + pass, status, status + (size_t)tiles * kRadix, err);
}

cudaError_t launch_onesweep_pass(const uint32_t *kin, const uint32_t *vin, uint32_t *kout, uint32_t *vout,
                                 uint32_t n, int pass, const SortWorkspace &ws, uint32_t *err, cudaStream_t st)
{
    switch (sort_items(n)) {
    case 1: return launch_pass<1>(kin, vin, kout, vout, n, pass, ws, err, st);
    case 2: return launch_pass<2>(kin, vin, kout, vout, n, pass, ws, err, st);
    case 3: return launch_pass<3>(kin, vin, kout, vout, n, pass, ws, err, st);
    case 4: return launch_pass<4>(kin, vin, kout, vout, n, pass, ws, err, st);
    case 5: return launch_pass<5>(kin, vin, kout, vout, n, pass, ws, err, st);
    case 6: return launch_pass<6>(kin, vin, kout, vout, n, pass, ws, err, st);
    case 7: return launch_pass<7>(kin, vin, kout, vout, n, pass, ws, err, st);
    default: return launch_pass<8>(kin, vin, kout, vout, n, pass, ws, err, st);
    }
}

}  // namespace

// The sort of n pairs on a zeroed head of the workspace (sort_head_words() words): the
// result is in keys / vals; alt_*: n words of scratch each.  A launch that fails ends it.
cudaError_t launch_sort(uint32_t *keys, uint32_t *vals, uint32_t *alt_keys, uint32_t *alt_vals, uint32_t n,
                        int passes, const SortWorkspace &ws, uint32_t *err, cudaStream_t st)
{
    const bool odd = passes & 1;
    cudaError_t e = launch_digit_hist(keys, n, passes, ws, vals, odd ? alt_keys : nullptr, odd ? alt_vals : nullptr, st);
    uint32_t *kb[2] = {keys, alt_keys}, *vb[2] = {vals, alt_vals};
    for (int k = 0; k < passes && e == cudaSuccess; ++k) {
        const int src = (k & 1) ^ (odd ? 1 : 0), dst = src ^ 1;
        e = launch_onesweep_pass(kb[src], vb[src], kb[dst], vb[dst], n, k, ws, err, st);
    }
    return e;
}

}  // namespace cmag

// ---------------------------------------------------------------------------
// Sort without any allocation: fixed scratch in device memory of this library.
//
// Some callers cannot call cudaMalloc at the moment they need the sort:
// latency-critical loops where an allocation would stall the device, and hosts
// whose device memory all comes from their own pool (a framework's caching
// allocator, an embedded runtime with a fixed budget).  For them the sort's
// workspace lives in one file-scope device array, sized for at most
// kNoAllocMaxKeys keys and held by every GPU that loads this library until the
// process exits.
// ---------------------------------------------------------------------------
namespace {

constexpr uint32_t kNoAllocMaxKeys = 1u << 20;  // 1,048,576 (hash, index) pairs
// (sort_items(): at most this many tiles for n up to kNoAllocMaxKeys)
constexpr uint32_t kNoAllocMaxTiles = cmag::kSortTiles;
static_assert(kNoAllocMaxKeys <= cmag::kSortTiles * cmag::kSortThreads * 8, "tiles of the largest size");
constexpr size_t kNoAllocMaxStatus =
    (size_t)(kNoAllocMaxTiles + (kNoAllocMaxTiles + cmag::kGroup - 1) / cmag::kGroup) * cmag::kRadix;
// histograms + tile counters + look-back status of up to four passes
constexpr size_t kNoAllocWsWords = (size_t)cmag::kMaxPasses * cmag::kRadix + cmag::kMaxPasses +
                                   (size_t)cmag::kMaxPasses * kNoAllocMaxStatus;
// + error word, then the alternate key and value buffers
constexpr size_t kNoAllocWords = kNoAllocWsWords + 1 + 2 * (size_t)kNoAllocMaxKeys;

__device__ __align__(256) uint32_t g_noalloc_scratch[kNoAllocWords];

// The array's device address belongs to the CUDA context the module was loaded
// in (normally the device's primary context).  It is looked up once per context,
// with that context current, and cached under the context handle, so a host that
// makes its own context current gets that context's copy.  The driver's
// cuCtxGetCurrent is reached through the runtime (no link to the driver library).
typedef int (*CtxGetCurrentFn)(void **ctx);
CtxGetCurrentFn ctx_get_current()
{
    static CtxGetCurrentFn fn = [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f, 12000, cudaEnableDefault, &q) !=
                cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            return (CtxGetCurrentFn) nullptr;
        return reinterpret_cast<CtxGetCurrentFn>(f);
    }();
    return fn;
}

constexpr int kMaxContexts = 64;
struct ScratchAddr {
    void *ctx;
    uint32_t *ptr;
};
std::mutex g_noalloc_mu;
ScratchAddr g_noalloc_addr[kMaxContexts] = {};
int g_noalloc_used = 0;

thread_local char g_noalloc_msg[256];

int noalloc_fail(int code, const char *msg, cudaError_t e = cudaSuccess)
{
    if (e != cudaSuccess)
        std::snprintf(g_noalloc_msg, sizeof(g_noalloc_msg), "%s: %s", msg, cudaGetErrorString(e));
    else
        std::snprintf(g_noalloc_msg, sizeof(g_noalloc_msg), "%s", msg);
    return code;
}

// Device address of the scratch array in the current context (set-up on the first
// call in each context; later calls read the cache).
int noalloc_scratch(uint32_t **out)
{
    void *ctx = nullptr;
    CtxGetCurrentFn get = ctx_get_current();
    // no context current yet (the runtime creates the primary one on the lookup
    // below): nothing to key the cache on this time
    if (get && get(&ctx) != 0) ctx = nullptr;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (ctx)
        for (int k = 0; k < g_noalloc_used; ++k)
            if (g_noalloc_addr[k].ctx == ctx) {
                *out = g_noalloc_addr[k].ptr;
                return CMAG_OK;
            }
    void *ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || !ptr)
        return noalloc_fail(CMAG_ERR_CUDA, "cudaGetSymbolAddress(scratch)", e);
    // without a context handle (driver entry point unavailable) nothing is cached
    if (ctx && g_noalloc_used < kMaxContexts) g_noalloc_addr[g_noalloc_used++] = {ctx, static_cast<uint32_t *>(ptr)};
    *out = static_cast<uint32_t *>(ptr);
    return CMAG_OK;
}

int device_error_fail(uint32_t bits)
{
    char msg[160];
    std::snprintf(msg, sizeof(msg), "sort: device-side check failed (bits 0x%x:%s%s)", bits,
                  (bits & CMAG_DEVERR_LOOKBACK_TIMEOUT) ? " look-back spin limit reached" : "",
                  (bits & CMAG_DEVERR_RANGE) ? " scatter index out of range" : "");
    return noalloc_fail(CMAG_ERR_DEVICE, msg);
}

}  // namespace

extern "C" {

const char *cmag_sort_particles_noalloc_error(void) { return g_noalloc_msg; }

int cmag_sort_particles_noalloc(uint32_t *d_hash, uint32_t *d_index, uint32_t n, uint32_t key_bits,
                                void *cuda_stream)
{
    using namespace cmag;
    if (n == 0) return CMAG_OK;
    if (!d_hash || !d_index) return noalloc_fail(CMAG_ERR_INVALID, "null argument");
    if (n > kNoAllocMaxKeys)
        return noalloc_fail(CMAG_ERR_INVALID,
                            "cmag_sort_particles_noalloc sorts at most 1048576 pairs; use "
                            "cmag_sort_particles for more");
    if (key_bits > 32) return noalloc_fail(CMAG_ERR_INVALID, "key_bits must be at most 32");
    uint32_t *base = nullptr;
    if (int rc = noalloc_scratch(&base)) return rc;
    cudaStream_t st = (cudaStream_t)cuda_stream;
    int passes = sort_passes(key_bits);
    if (passes < 1) passes = 1;
    // the scratch keeps the previous call's contents: clear the counters this call reads
    // (the histogram pass clears the look-back status) and the error word
    uint32_t *err = base + kNoAllocWsWords;
    uint32_t *alt_keys = err + 1, *alt_vals = alt_keys + kNoAllocMaxKeys;
    cudaError_t e = cudaMemsetAsync(base, 0, sort_head_words() * sizeof(uint32_t), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(err, 0, sizeof(uint32_t), st);
    if (e != cudaSuccess) return noalloc_fail(CMAG_ERR_CUDA, "cudaMemsetAsync", e);
    e = launch_sort(d_hash, d_index, alt_keys, alt_vals, n, passes, sort_workspace_view(base, n), err, st);
    // a launch that failed leaves its error pending; it is reported but not
    // cleared (an error left by the caller's earlier work stays the caller's)
    if (e == cudaSuccess) e = cudaPeekAtLastError();
    if (e != cudaSuccess) return noalloc_fail(CMAG_ERR_CUDA, "sort launch (or an earlier pending error)", e);
    // wait for the sort and read its device-side check word
    uint32_t bits = 0;
    e = cudaMemcpyAsync(&bits, err, sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return noalloc_fail(CMAG_ERR_CUDA, "sort", e);
    if (bits) return device_error_fail(bits);
    return CMAG_OK;
}

int cmag_testing_set_sort_spin_limit(int32_t polls)
{
    using namespace cmag;
    const int v = polls < 0 ? kSpinLimit : polls;
    cudaError_t e = cudaMemcpyToSymbol(g_spin_limit, &v, sizeof(int));
    if (e != cudaSuccess) return noalloc_fail(CMAG_ERR_CUDA, "cudaMemcpyToSymbol(spin limit)", e);
    return CMAG_OK;
}

}  // extern "C"
