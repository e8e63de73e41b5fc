// small_step.cu -- the step of a small planar scene in three launches.
//
// A scene of a few thousand particles leaves the GPU idle in the staged step: each
// of its nine dependent launches (hash, three scan launches, scatter, order, density,
// force, integrate) runs a few blocks for 3-4 us, the neighbour loops take 14-38 us
// because one thread a particle waits on a serial chain of loads, and replaying the
// captured step costs the host about 15 us.  Here
//   * one thread-block cluster (16 blocks on 16 SMs) hashes, counts, scans and sorts:
//     stages separated by the hardware cluster barrier (about 0.5 us, mostly the wait
//     for the block's writes) instead of launches, the scan's block totals through
//     distributed shared memory.  Bound by the latency of its five stages (10-17 us).
//     512 threads a block: at 1024 the cluster waits for 16 SMs that are nearly empty
//     when other solvers run beside it (16,384 particles, 8 lanes: 20.5 against 25 us a step);
//   * the density and the force give each particle 8 lanes (4 in the larger scenes),
//     one per row of its cell box, so a particle's cell lookups and loads are in
//     flight together.  Bound by that latency up to about 10,000 particles, then by
//     instruction issue;
//   * the force launch integrates its particles too.
// One solver alone, us per step, staged -> here: Poiseuille 4,480 particles 43 -> 20, dam
// break 8,702 61 -> 31, Peristalsis 16,384 60 -> 41; three solvers in turn, where the
// host's 15 us a step counts: 15.6 -> 8.5, 22.8 -> 15.2, 24.1 -> 19.1.
//
// Same bits as the staged step with one lane per particle: the lanes leave their
// candidates' terms in shared memory, and one lane per sum adds them in the order of
// the one-lane walk, NaN of particles at no finite place included.  (The staged step's
// lanes add partial sums of their rows, which rounds differently.)
#include <cuda_runtime.h>

#include "kernels.h"
#include "neighbor_walk.cuh"
#include "pair_terms.cuh"
#include "particle_motion.cuh"

namespace cmag {

namespace {

constexpr int kSortBlock = 512;  // threads per block of the sort's cluster
constexpr uint32_t kMaxCluster = 16;

__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// All threads of the cluster: memory written before is visible after.
__device__ __forceinline__ void cluster_sync()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// The word at shared address `local` of block `rank` of the cluster.
__device__ __forceinline__ uint32_t load_peer(const uint32_t *local, uint32_t rank)
{
    uint32_t addr = (uint32_t)__cvta_generic_to_shared(local), v;
    asm volatile("mapa.shared::cluster.u32 %0, %0, %2;\n\tld.shared::cluster.u32 %1, [%0];"
                 : "+r"(addr), "=r"(v)
                 : "r"(rank)
                 : "memory");
    return v;
}

// Sum over the block, in every thread.
__device__ __forceinline__ uint32_t block_sum(uint32_t x, uint32_t *s_warp)
{
    x = __reduce_add_sync(0xffffffffu, x);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = x;
    __syncthreads();
    uint32_t t = 0;
    for (uint32_t w = 0; w < (blockDim.x >> 5); ++w) t += s_warp[w];
    __syncthreads();
    return t;
}

// Phase, hash, per-cell counts, dense offsets and the stable counting sort with the
// gather: the kernels of cells.cu in one cluster.  Data written by other blocks of
// the cluster is read with ordinary loads after the barriers.
template <int SYS>
__global__ void __launch_bounds__(kSortBlock, 1) k_small_sort(DevParams p, SmallStep a)
{
    pdl_entry();
    __shared__ uint32_t s_warp[kSortBlock / 32];
    __shared__ uint32_t s_total;
    const uint32_t rank = cluster_rank(), blocks = gridDim.x;
    const uint32_t tid = rank * blockDim.x + threadIdx.x, threads = blocks * blockDim.x;
    const uint32_t cells = p.scan_cells + 1;
    const uint32_t per = (cells + threads - 1) / threads;  // cells a thread scans
    // ---- phase and hash: per-cell counts and arrival ranks (k_hash)
    PhaseState ph{};
    if (SYS == CMAG_PERISTALSIS) ph = next_phase(p, *a.phase, a.k_milli);
    for (uint32_t i = tid; i < p.n; i += threads) {
        float4 q = a.pos[i];
        if (SYS == CMAG_PERISTALSIS && ph.configure && configure_wall(p, ph.configure_height, q)) a.pos[i] = q;
        const int3 g = grid_pos(p, q.x, q.y, q.z);
        uint32_t rel = grid_hash(p, g.x, g.y, g.z) - p.scan_base;
        if (rel >= p.scan_cells) {
            set_error(a.err, CMAG_DEVERR_RANGE);
            rel = p.scan_cells - 1;
        }
        a.hash[i] = p.scan_base + rel;
        a.rank[i] = atomicAdd(a.cnt + rel, 1u);
        if (SYS == CMAG_DAMBREAK && p.wc_mark) wall_cache_note(p, i, q, g, p.wc_state[kWcStamp] + 1u);
    }
    cluster_sync();
    // ---- cell scan: counts -> dense offsets, counters cleared (k_tile_sum,
    // k_tile_prefix, k_cell_offsets); the blocks' totals through shared memory
    if (tid == 0) {
        if (SYS == CMAG_PERISTALSIS) *a.phase = ph;
        if (SYS == CMAG_DAMBREAK && p.wc_state) {
            p.wc_state[kWcStamp] += 1u;
            if (p.wc_state[kWcMoved]) {
                p.wc_state[kWcEpoch] += 1u;
                p.wc_state[kWcMoved] = 0u;
            }
        }
    }
    const uint32_t c0 = min(cells, tid * per), c1 = min(cells, c0 + per);
    uint32_t sum = 0;
    for (uint32_t c = c0; c < c1; ++c) sum += a.cnt[c];
    uint32_t x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if ((threadIdx.x & 31) >= (uint32_t)o) x += y;
    }
    const uint32_t total = block_sum(sum, s_warp);
    if (threadIdx.x == 0) s_total = total;
    if ((threadIdx.x & 31) == 31) s_warp[threadIdx.x >> 5] = x;
    cluster_sync();
    uint32_t run = x - sum;
    for (uint32_t r = 0; r < rank; ++r) run += load_peer(&s_total, r);
    for (uint32_t w = 0; w < (threadIdx.x >> 5); ++w) run += s_warp[w];
    for (uint32_t c = c0; c < c1; ++c) {
        const uint32_t v = a.cnt[c];
        a.off[c] = run;
        run += v;
        if (v) a.cnt[c] = 0;
    }
    cluster_sync();
    // ---- counting sort: scatter, then order and gather (k_cell_scatter, k_cell_order)
    for (uint32_t i = tid; i < p.n; i += threads) {
        const uint32_t h = a.hash[i], q = a.off[h - p.scan_base] + a.rank[i];
        if (q < p.n) {
            a.shash[q] = h;
            a.tmp[q] = i;
        } else {
            set_error(a.err, CMAG_DEVERR_RANGE);
        }
    }
    cluster_sync();
    for (uint32_t q = tid; q < p.n; q += threads) {
        const uint32_t c = a.shash[q] - p.scan_base, b = a.off[c], e = a.off[c + 1], own = a.tmp[q];
        uint32_t dst = q;
        if (!(b <= q && q < e && e <= p.n)) {  // counts and offsets disagree
            set_error(a.err, CMAG_DEVERR_RANGE);
        } else if (e - b > 1u) {
            uint32_t r = 0;
#pragma unroll 8
            for (uint32_t k = b; k < e; ++k) r += a.tmp[k] < own ? 1u : 0u;
            dst = b + r;
        }
        a.idx[dst] = own;
        const uint32_t j = own < p.n ? own : dst;  // own >= n only after a failed sort
        a.spos[dst] = a.pos[j];
        a.svel[dst] = a.vlf[j];
    }
}

// ---- neighbour loops: L lanes per particle, lane r on row r of a batch of L rows ------

// 8 lanes take a box of 7 rows at once: the shortest chain, and the form of scenes up to
// kWideParticles.  4 lanes take it in two batches with half the warps: above that line,
// where solvers that share the GPU compete for issue slots (us per step, 8 lanes / 4, three
// solvers in turn; one alone: Poiseuille 4480 particles 8.5 / 10.0; 19.3 / 29.2, dam break
// 8702 15.2 / 16.3; 31.5 / 38.8, Poiseuille 10,800 14.5 / 12.8; 30.2 / 31.2, dam break 12,158
// 19.0 / 19.3; 40.7 / 42.6, Peristalsis 16,384 21.0 / 19.1; 39.4 / 40.6, Poiseuille 16,960
// 21.0 / 17.9; 34.8 / 33.4).
constexpr uint32_t kWideParticles = 12000;
constexpr int kSlots = 8;            // terms of a row held at once
constexpr uint32_t kRowMost = 32;    // candidates of a row that one lane takes
constexpr int kLoopThreads = 256;    // per block
// Words between the slots of neighbouring rows: `words` for each of the warp's
// particles and as many of padding, so that the lanes that write a slot, and those
// that read one, fall into different banks.
template <int L>
__host__ __device__ constexpr int slot_stride(int words)
{
    return words * (32 / L + 1);
}

// The candidates of one row: sorted particles b0, b0 + 1, ... (n0 of them) and, when
// the row wraps in x, n1 more from b1; with their image shifts.
struct Row {
    uint32_t b0, n0, b1, n1;
    float sx0, sx1, sy;
};

template <int SYS, bool TRIM>
__device__ __forceinline__ Row find_row(const DevParams &p, const uint32_t *off, int dy, int3 g, float3 f)
{
    Row r{0, 0, 0, 0, 0.0f, 0.0f, 0.0f};
    walk::RowRuns rr;
    const walk::Slab sl{};
    if (dy <= p.cell_count && walk::row_runs<SYS, true, TRIM>(p, off, dy, sl, g, f.x, f.y, rr)) {
        r.b0 = rr.b0;
        r.n0 = rr.e0 - rr.b0;
        r.b1 = rr.b1;
        r.n1 = rr.e1 > rr.b1 ? rr.e1 - rr.b1 : 0u;
        r.sx0 = rr.sx0;
        r.sx1 = rr.sx1;
        r.sy = rr.sy;
    }
    return r;
}

// Lanes of one particle.
template <int L>
struct Group {
    uint32_t mask;
    int lane, index;
    __device__ __forceinline__ Group()
    {
        const int l = threadIdx.x & 31;
        lane = l % L;
        index = l / L;
        mask = ((1u << L) - 1u) << (l - lane);
    }
    template <class T>
    __device__ __forceinline__ T get(T v, int from) const
    {
        return __shfl_sync(mask, v, from, L);
    }
    __device__ __forceinline__ Row get(const Row &v, int from) const
    {
        return Row{get(v.b0, from), get(v.n0, from), get(v.b1, from), get(v.n1, from),
                   get(v.sx0, from), get(v.sx1, from), get(v.sy, from)};
    }
    __device__ __forceinline__ bool all(bool b) const { return __all_sync(mask, b) != 0; }
    __device__ __forceinline__ uint32_t largest(uint32_t v) const { return __reduce_max_sync(mask, v); }
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }
    // first of the particle's `words` words of slot k of row r
    __device__ __forceinline__ int slot(int k, int r, int words) const
    {
        return (k * L + r) * slot_stride<L>(words) + index * words;
    }
};

// The factors (1 - q/2)^4 and 2q + 1 of the pair step (density.cu, wendland_run) of
// candidates at a and c (two: there are two).
template <int SYS>
__device__ __forceinline__ float4 pair_weights(const DevParams &p, float4 pi, float4 a, float4 c, bool two,
                                               float sx, float sy)
{
    float2 ax = make_float2(a.x, c.x), ay = make_float2(a.y, c.y);
    if (SYS != CMAG_DAMBREAK) ax = __fadd2_rn(ax, make_float2(sx, sx));
    if (SYS == CMAG_PERISTALSIS) ay = __fadd2_rn(ay, make_float2(sy, sy));
    const float2 m1 = make_float2(-1.0f, -1.0f), one = make_float2(1.0f, 1.0f);
    const float2 rx = __ffma2_rn(ax, m1, make_float2(pi.x, pi.x)), ry = __ffma2_rn(ay, m1, make_float2(pi.y, pi.y));
    const float2 d2 = __ffma2_rn(ry, ry, __fmul2_rn(rx, rx));
    const float2 dt = __fadd2_rn(d2, make_float2(1e-30f, 1e-30f));
    const float2 d = __fmul2_rn(d2, make_float2(rsqrtf(dt.x), rsqrtf(dt.y)));
    float2 t = __ffma2_rn(d, make_float2(-0.5f * p.inv_h, -0.5f * p.inv_h), one);
    t = make_float2(fmaxf(t.x, 0.0f), fmaxf(t.y, 0.0f));
    const float2 t2 = __fmul2_rn(t, t), t4 = __fmul2_rn(t2, t2);
    const float2 lin = __ffma2_rn(d, make_float2(2.0f * p.inv_h, 2.0f * p.inv_h), one);
    // a run's odd last candidate: its weight is rounded before the sum
    return two ? make_float4(t4.x, lin.x, t4.y, lin.y)
               : make_float4(__fmul_rn(t4.x, lin.x), 1.0f, 0.0f, 0.0f);
}

// Whether a term (w.x w.y, w.z w.w) changes a sum: a factor (1 - q/2)^4 is not zero, or the
// other one is NaN, of a candidate that is not at a finite place (0 * NaN is NaN).
__device__ __forceinline__ bool counts(float4 w)
{
    return w.x != 0.0f || w.z != 0.0f || isnan(w.y + w.w);
}

// A cubic-spline candidate's weight (density.cu).
template <int SYS>
__device__ __forceinline__ float spline_weight(const DevParams &p, float4 pi, float4 pj, float sx, float sy)
{
    const float3 r = walk::rel<SYS>(pi, pj, sx, sy, 0.0f);
    const float d2 = __fmaf_rn(r.y, r.y, __fmul_rn(r.x, r.x));
    const float v = kernel_w(p, fminf(d2 * rsqrtf(fmaxf(d2, 1e-30f)) * p.inv_h, 2.0f));
    return (d2 < p.support2) ? v : 0.0f;
}

// Lanes 0 .. lanes - 1 add the rows' slots in order, K slots a row (the row's `at`
// terms and exact zeros).
template <int K, int L>
__device__ __forceinline__ void sum_slots(const Group<L> &gr, float *s, uint32_t at, int lanes, float &sum)
{
#pragma unroll
    for (int k = 0; k < K; ++k)
        if (k >= (int)at) *reinterpret_cast<float4 *>(s + gr.slot(k, gr.lane, 4)) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    gr.sync();
    if (gr.lane < lanes) {
#pragma unroll
        for (int r = 0; r < L; ++r)
#pragma unroll
            for (int k = 0; k < K; ++k) {
                const float2 v = *reinterpret_cast<const float2 *>(s + gr.slot(k, r, 4) + 2 * gr.lane);
                sum = __fmaf_rn(v.x, v.y, sum);
            }
    }
    gr.sync();
}

// Density sum over the rows of one batch (lane r holds row r), added to `sum` in the
// walk's order.  Wendland: lane 0 adds the even candidates of each run, lane 1 the odd
// ones; cubic spline: lane 0 adds all.  Each lane leaves its row's non-zero terms in
// its slots, then they are added row by row.  For rows of at most kRowMost candidates;
// false (and nothing added) when a row has more terms than slots.
template <int SYS, int L>
__device__ __forceinline__ bool add_rows(const DevParams &p, const float4 *spos, const Group<L> &gr, const Row &row,
                                         float4 pi, float *s, float &sum)
{
    // a term is stored behind the row's earlier ones and counted when it changes the sum
    // (no branch); the slot after the last is scratch
    uint32_t at = 0;
    auto put = [&](float4 w) {
        *reinterpret_cast<float4 *>(s + gr.slot(min(at, (uint32_t)kSlots), gr.lane, 4)) = w;
        at += counts(w) ? 1u : 0u;
    };
    const bool wendland = p.kernel == CMAG_KERNEL_WENDLAND;
    if (wendland) {
        constexpr uint32_t U = 2;  // pair steps loaded together
        const uint32_t h0 = (row.n0 + 1) / 2, h = h0 + (row.n1 + 1) / 2, most = gr.largest(h);
        for (uint32_t m0 = 0; m0 < most; m0 += U) {
            float4 q0[U], q1[U];
            bool two[U];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t m = m0 + u;
                const bool first = m < h0;
                const uint32_t k = 2 * (first ? m : m - h0), n = first ? row.n0 : row.n1;
                const uint32_t j = m < h ? (first ? row.b0 : row.b1) + k : 0u;
                two[u] = m < h && k + 1 < n;
                q0[u] = __ldg(spos + j);
                q1[u] = __ldg(spos + j + (two[u] ? 1 : 0));
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                float4 w = pair_weights<SYS>(p, pi, q0[u], q1[u], two[u], m0 + u < h0 ? row.sx0 : row.sx1, row.sy);
                if (m0 + u >= h) w = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                put(w);
            }
        }
    } else {
        constexpr uint32_t U = 4;
        const uint32_t n = row.n0 + row.n1, most = gr.largest(n);
        for (uint32_t k0 = 0; k0 < most; k0 += U) {
            float4 q[U];
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const uint32_t k = k0 + u;
                q[u] = __ldg(spos + (k < n ? (k < row.n0 ? row.b0 + k : row.b1 + (k - row.n0)) : 0u));
            }
#pragma unroll
            for (uint32_t u = 0; u < U; ++u) {
                const float w = spline_weight<SYS>(p, pi, q[u], k0 + u < row.n0 ? row.sx0 : row.sx1, row.sy);
                put(make_float4(k0 + u < n ? w : 0.0f, 1.0f, 0.0f, 0.0f));
            }
        }
    }
    const uint32_t most = gr.largest(at);
    if (most > (uint32_t)kSlots) return false;
    if (most <= 4) sum_slots<4>(gr, s, at, wendland ? 2 : 1, sum);
    else if (most <= 6) sum_slots<6>(gr, s, at, wendland ? 2 : 1, sum);
    else sum_slots<kSlots>(gr, s, at, wendland ? 2 : 1, sum);
    return true;
}

// The same with rows of any length, one after another, every lane on the row's next
// candidates (pair steps).
template <int SYS, int L>
__device__ __noinline__ float add_long_rows(const DevParams &p, const float4 *spos, const Group<L> &gr, const Row &mine,
                                            float4 pi, float *s, float sum)
{
    const bool wendland = p.kernel == CMAG_KERNEL_WENDLAND;
    const uint32_t per = wendland ? 2u : 1u;  // candidates a lane takes
    for (int r = 0; r < L; ++r) {
        const Row row = gr.get(mine, r);
        for (int part = 0; part < 2; ++part) {
            const uint32_t b = part ? row.b1 : row.b0, e = b + (part ? row.n1 : row.n0);
            const float sx = part ? row.sx1 : row.sx0;
            for (uint32_t base = b; base < e; base += per * L) {
                const uint32_t j = base + per * gr.lane;
                float4 w = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (j < e) {
                    const float4 q = __ldg(spos + j);
                    if (wendland) {
                        const bool two = j + 1 < e;
                        w = pair_weights<SYS>(p, pi, q, __ldg(spos + j + (two ? 1 : 0)), two, sx, row.sy);
                    } else {
                        w = make_float4(spline_weight<SYS>(p, pi, q, sx, row.sy), 1.0f, 0.0f, 0.0f);
                    }
                }
                if (gr.all(!counts(w))) continue;  // out of reach: nothing to add
                *reinterpret_cast<float4 *>(s + gr.slot(0, gr.lane, 4)) = w;
                gr.sync();
                if (gr.lane < (int)per) {
                    for (int l = 0; l < L; ++l) {
                        const float2 v = *reinterpret_cast<const float2 *>(s + gr.slot(0, l, 4) + 2 * gr.lane);
                        sum = __fmaf_rn(v.x, v.y, sum);
                    }
                }
                gr.sync();
            }
        }
    }
    return sum;
}

// Density (k_density).
template <int SYS, bool TRIM, int L>
__global__ void __launch_bounds__(kLoopThreads, 4) k_small_density(DevParams p, SmallStep a)
{
    pdl_entry();
    __shared__ float4 s_all[kLoopThreads / 32][(kSlots + 1) * L * slot_stride<L>(4) / 4];
    float *const s = reinterpret_cast<float *>(s_all[threadIdx.x >> 5]);
    const Group<L> gr;
    const uint32_t i = (blockIdx.x * kLoopThreads + threadIdx.x) / L;
    if (i >= p.n) return;  // whole groups
    const float4 pi = __ldg(a.spos + i);
    const bool pinned = SYS == CMAG_POISEUILLE && pi.w == 1.0f;
    uint32_t wc = 0;  // kept wall density: 0 none, 1 keep this result, 2 take the kept one
    float4 kept = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const int3 g = grid_pos(p, pi.x, pi.y, pi.z);
    if (SYS == CMAG_DAMBREAK && p.wc_entry && pi.w != (float)CMAG_FLUID && !walk::fluid_near(p, g)) {
        kept = p.wc_entry[a.idx[i]];
        wc = __float_as_uint(kept.z) == p.wc_state[kWcEpoch] ? 2u : 1u;
    }
    float sum = 0.0f;
    if (!pinned && wc != 2u) {
        const float3 f = walk::frac_cell(p, pi);
        const bool wendland = p.kernel == CMAG_KERNEL_WENDLAND;
        for (int dy0 = -p.cell_count; dy0 <= p.cell_count; dy0 += L) {
            const Row row = find_row<SYS, TRIM>(p, a.off, dy0 + gr.lane, g, f);
            if (!gr.all(row.n0 + row.n1 <= kRowMost) || !add_rows<SYS>(p, a.spos, gr, row, pi, s, sum))
                sum = add_long_rows<SYS>(p, a.spos, gr, row, pi, s, sum);
        }
        sum = wendland ? p.w_norm * (gr.get(sum, 0) + gr.get(sum, 1)) : gr.get(sum, 0);
    }
    if (gr.lane != 0) return;
    float rho, pr;
    if (pinned) {
        rho = p.rho0;
        pr = p.p_wall;
    } else if (wc == 2u) {
        rho = kept.x;
        pr = kept.y;
    } else {
        rho = sum * p.mass;
        pr = eos_pressure(p, rho);
    }
    a.meas[i] = make_float4(rho, pr, 0.0f, SYS == CMAG_PERISTALSIS ? pi.w : 0.0f);
    const float inv_rho = 1.0f / rho;
    a.aux[i] = make_float2(pr * inv_rho * inv_rho, SYS == CMAG_DAMBREAK ? rho : inv_rho);
    if (wc == 1u) p.wc_entry[a.idx[i]] = make_float4(rho, pr, __uint_as_float(p.wc_state[kWcEpoch]), 0.0f);
}

// A candidate's terms in its slot, and out of it into the sum of lane c: x and y of
// a r (DamBreak: words a, rx, a, ry), of a r then b v (Poiseuille: a, rx, b, vx and
// a, ry, b, vy), or of a r (lanes 0, 1) and b v (lanes 2, 3; Peristalsis: a, rx, a, ry,
// b, vx, b, vy).
template <int SYS>
struct Slot {
    static constexpr int words = SYS == CMAG_DAMBREAK ? 4 : 8;
    // terms of a row held at once: a collapsing column presses up to 11 particles into
    // the 6 cells in reach
    static constexpr int count = SYS == CMAG_DAMBREAK ? 16 : 8;
    static constexpr int lanes = SYS == CMAG_PERISTALSIS ? 4 : 2;  // that add
    static __device__ __forceinline__ void put(float *s, const PairTerms &t)
    {
        float4 *d = reinterpret_cast<float4 *>(s);
        if (SYS == CMAG_POISEUILLE) {
            d[0] = make_float4(t.a, t.rx, t.b, t.vx);
            d[1] = make_float4(t.a, t.ry, t.b, t.vy);
        } else {
            d[0] = make_float4(t.a, t.rx, t.a, t.ry);
            if (SYS == CMAG_PERISTALSIS) d[1] = make_float4(t.b, t.vx, t.b, t.vy);
        }
    }
    static __device__ __forceinline__ void take(const float *s, int c, float &sum)
    {
        if (SYS == CMAG_POISEUILLE) {
            const float4 f = reinterpret_cast<const float4 *>(s)[c];
            sum = __fmaf_rn(f.z, f.w, __fmaf_rn(f.x, f.y, sum));
        } else {
            const float2 f = reinterpret_cast<const float2 *>(s)[c];
            sum = __fmaf_rn(f.x, f.y, sum);
        }
    }
    // like sum_slots
    template <int K, int L>
    static __device__ __forceinline__ void add(const Group<L> &gr, float *s, uint32_t at, float &sum)
    {
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (k >= (int)at) put(s + gr.slot(k, gr.lane, words), PairTerms{});
        gr.sync();
        if (gr.lane < lanes) {
#pragma unroll
            for (int r = 0; r < L; ++r)
#pragma unroll
                for (int k = 0; k < K; ++k) take(s + gr.slot(k, r, words), gr.lane, sum);
        }
        gr.sync();
    }
};

// The force sums over the rows of one batch, like add_rows and add_long_rows.
template <int SYS, bool TRIM, int L>
__device__ __forceinline__ bool add_row_forces(const DevParams &p, const SmallStep &a, const Group<L> &gr,
                                               const Row &row, const PairSelf &self, float *s, float &sum)
{
    constexpr uint32_t U = 4;  // candidates loaded together
    const uint32_t n = row.n0 + row.n1, longest = gr.largest(n);
    uint32_t at = 0;
    for (uint32_t k0 = 0; k0 < longest; k0 += U) {
        float4 q[U], v[U];
        float2 x[U];
        uint32_t j[U];
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            const uint32_t k = k0 + u;
            // (the particle itself stands in for a missing candidate: no terms)
            j[u] = k < n ? (k < row.n0 ? row.b0 + k : row.b1 + (k - row.n0)) : self.i;
            q[u] = __ldg(a.spos + j[u]);
            v[u] = __ldg(a.svel + j[u]);
            x[u] = __ldg(a.aux + j[u]);
        }
#pragma unroll
        for (uint32_t u = 0; u < U; ++u) {
            PairTerms t;
            const bool hit = pair_terms<SYS, TRIM>(p, self, j[u], q[u], v[u], x[u],
                                                   k0 + u < row.n0 ? row.sx0 : row.sx1, row.sy, t);
            Slot<SYS>::put(s + gr.slot(min(at, (uint32_t)Slot<SYS>::count), gr.lane, Slot<SYS>::words), t);
            at += hit ? 1u : 0u;
        }
    }
    const uint32_t most = gr.largest(at);
    if (most > (uint32_t)Slot<SYS>::count) return false;
    if (most <= 6) Slot<SYS>::template add<6>(gr, s, at, sum);
    else if (most <= 8) Slot<SYS>::template add<8>(gr, s, at, sum);
    else if (most <= 12) Slot<SYS>::template add<12>(gr, s, at, sum);
    else Slot<SYS>::template add<Slot<SYS>::count>(gr, s, at, sum);
    return true;
}

template <int SYS, bool TRIM, int L>
__device__ __noinline__ float add_long_row_forces(const DevParams &p, const SmallStep &a, const Group<L> &gr,
                                                  const Row &mine, const PairSelf &self, float *s, float sum)
{
    for (int r = 0; r < L; ++r) {
        const Row row = gr.get(mine, r);
        for (int part = 0; part < 2; ++part) {
            const uint32_t b = part ? row.b1 : row.b0, e = b + (part ? row.n1 : row.n0);
            const float sx = part ? row.sx1 : row.sx0;
            for (uint32_t base = b; base < e; base += L) {
                const uint32_t j = base + gr.lane < e ? base + gr.lane : self.i;
                PairTerms t{};
                const float4 q = __ldg(a.spos + j);
                const float d2 = pair_distance<SYS>(self, q, sx, row.sy, t);
                const bool out = !(d2 < p.support2) && (SYS != CMAG_DAMBREAK || TRIM || q.w == (float)CMAG_FLUID);
                if (gr.all(out || j == self.i)) continue;  // out of reach: nothing to add
                pair_terms<SYS, TRIM>(p, self, j, q, __ldg(a.svel + j), __ldg(a.aux + j), sx, row.sy, t);
                Slot<SYS>::put(s + gr.slot(0, gr.lane, Slot<SYS>::words), t);
                gr.sync();
                if (gr.lane < Slot<SYS>::lanes)
                    for (int l = 0; l < L; ++l)
                        Slot<SYS>::take(s + gr.slot(0, l, Slot<SYS>::words), gr.lane, sum);
                gr.sync();
            }
        }
    }
    return sum;
}

// Force (k_force) and integration (k_integrate) of the same particle.
template <int SYS, bool TRIM, int L>
__global__ void __launch_bounds__(kLoopThreads, 2) k_small_force(DevParams p, SmallStep a)
{
    pdl_entry();
    extern __shared__ float4 smem[];
    constexpr int kWords = (Slot<SYS>::count + 1) * L * slot_stride<L>(Slot<SYS>::words);  // of a warp
    float *const s = reinterpret_cast<float *>(smem) + (threadIdx.x >> 5) * kWords;
    const Group<L> gr;
    const uint32_t i = (blockIdx.x * kLoopThreads + threadIdx.x) / L;
    if (i >= p.n) return;  // whole groups
    float4 pi = __ldg(a.spos + i);
    if (SYS == CMAG_DAMBREAK && pi.w != (float)CMAG_FLUID) return;
    const float4 vi = __ldg(a.svel + i);
    const float2 ai = __ldg(a.aux + i);
    const PairSelf self{i, pi, vi, ai, -p.mass, p.visc_coeff * ai.y, a.lists};
    const int3 g = grid_pos(p, pi.x, pi.y, pi.z);
    const float3 f = walk::frac_cell(p, pi);
    float sum = 0.0f;
    for (int dy0 = -p.cell_count; dy0 <= p.cell_count; dy0 += L) {
        const Row row = find_row<SYS, TRIM>(p, a.off, dy0 + gr.lane, g, f);
        if (!gr.all(row.n0 + row.n1 <= kRowMost) || !add_row_forces<SYS, TRIM>(p, a, gr, row, self, s, sum))
            sum = add_long_row_forces<SYS, TRIM>(p, a, gr, row, self, s, sum);
    }
    float ax = gr.get(sum, 0), ay = gr.get(sum, 1);
    const float bx = gr.get(sum, 2), by = gr.get(sum, 3);  // Peristalsis: viscous force
    if (gr.lane != 0) return;
    const uint32_t o = a.idx[i];
    if (o >= p.n) return;  // only after a failed sort (reported by the sort itself)
    if (SYS == CMAG_PERISTALSIS) {
        a.out_a[o] = make_float4(bx, by, 0.0f, 0.0f);  // viscous
        a.out_b[o] = make_float4(ax, ay, 0.0f, 0.0f);  // pressure
        ax = bx + ax;
        ay = by + ay;
        if (pi.w != 0.0f) {
            if (move_wall(p, a.phase->is_bc, a.phase->t, pi)) a.pos[o] = pi;
            return;
        }
    } else {
        a.out_a[o] = make_float4(ax, ay, 0.0f, 0.0f);
        if (SYS == CMAG_POISEUILLE && pi.w == 1.0f) return;  // walls stay fixed
    }
    // pi and vi are this particle's position and leap-frog velocity
    float4 v = a.vel[o], lf = vi;
    integrate_fluid(p, ax, ay, 0.0f, pi, v, lf);
    a.pos[o] = pi;
    a.vel[o] = v;
    a.vlf[o] = lf;
}

using SmallKernel = void (*)(DevParams, SmallStep);

struct Kernels {
    SmallKernel sort, density, force;
    uint32_t force_smem, lanes;
};

template <int SYS, bool TRIM, int L>
Kernels kernels_for()
{
    return {k_small_sort<SYS>, k_small_density<SYS, TRIM, L>, k_small_force<SYS, TRIM, L>,
            (uint32_t)((kLoopThreads / 32) * (Slot<SYS>::count + 1) * L * slot_stride<L>(Slot<SYS>::words) * sizeof(float)),
            (uint32_t)L};
}

template <int L>
Kernels kernels_of_lanes(const DevParams &p)
{
    if (p.system == CMAG_DAMBREAK)
        return p.trim ? kernels_for<CMAG_DAMBREAK, true, L>() : kernels_for<CMAG_DAMBREAK, false, L>();
    return p.system == CMAG_POISEUILLE ? kernels_for<CMAG_POISEUILLE, true, L>()
                                       : kernels_for<CMAG_PERISTALSIS, true, L>();
}

Kernels kernels_of(const DevParams &p)
{
    return p.n <= kWideParticles ? kernels_of_lanes<8>(p) : kernels_of_lanes<4>(p);
}

cudaLaunchConfig_t sort_config(const DevParams &p, uint32_t cluster, cudaStream_t st, cudaLaunchAttribute (&attr)[2])
{
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    const uint32_t most = p.n > p.scan_cells ? p.n : p.scan_cells;
    uint32_t threads = ((most + cluster - 1) / cluster + 31u) & ~31u;
    threads = threads < 128u ? 128u : (threads > (uint32_t)kSortBlock ? (uint32_t)kSortBlock : threads);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = cluster;
    cfg.blockDim = threads;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return cfg;
}

}  // namespace

bool small_step_fits(const DevParams &p)
{
    return p.planar && p.n <= kSmallParticles && p.scan_cells < kSmallCells && p.table_base == 0 && !p.wall_noslip &&
           (p.trim || p.system == CMAG_DAMBREAK);
}

uint32_t small_step_cluster(const DevParams &p)
{
    const Kernels k = kernels_of(p);
    if (cudaFuncSetAttribute(k.force, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.force_smem) == cudaSuccess &&
        cudaFuncSetAttribute(k.sort, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        for (uint32_t cluster = kMaxCluster; cluster >= 8; cluster /= 2) {
            int found = 0;
            cudaLaunchAttribute attr[2];
            cudaLaunchConfig_t cfg = sort_config(p, cluster, nullptr, attr);
            if (cudaOccupancyMaxActiveClusters(&found, k.sort, &cfg) == cudaSuccess && found > 0) return cluster;
        }
    }
    (void)cudaGetLastError();
    return 0;
}

cudaError_t launch_small_step(const DevParams &p, const SmallStep &a, uint32_t cluster, cudaStream_t st)
{
    const Kernels k = kernels_of(p);
    cudaLaunchAttribute attr[2];
    cudaLaunchConfig_t cfg = sort_config(p, cluster, st, attr);
    cudaError_t e = cudaLaunchKernelEx(&cfg, k.sort, p, a);
    cfg.attrs = attr + 1;  // programmatic dependent launch, no cluster
    cfg.numAttrs = 1;
    cfg.gridDim = (uint32_t)(((uint64_t)p.n * k.lanes + kLoopThreads - 1) / kLoopThreads);
    cfg.blockDim = kLoopThreads;
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k.density, p, a);
    cfg.dynamicSmemBytes = k.force_smem;
    if (e == cudaSuccess) e = cudaLaunchKernelEx(&cfg, k.force, p, a);
    return e;
}

}  // namespace cmag
