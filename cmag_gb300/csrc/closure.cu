// closure.cu -- the learned closure's kernels (the C ABI is in closure_api.cu).
//
// A coarse DamBreak run misses the sub-grid part of the pressure, viscous and
// wall accelerations that a run at half its spacing resolves.  The closure
// predicts that part per fluid particle from 16 features of the particle and its
// neighbours and adds it to the acceleration before integration.  No reference
// counterpart; the features reuse the neighbour walk of the density and force
// loops.
//
// Features of fluid particle i (V_j = m / rho_j, W_ij = W(|x_i - x_j| / h), the
// sums over every particle j, i included, inside the support):
//   0      rho_i / rho0 - 1            1      p_i / B
//   2..4   sum V_j W_ij (x_j - x_i) / h
//   5..7   sum V_j W_ij (v_j - v_i) / c0
//   8      sum V_j W_ij                 9      sum V_j W_ij |x_j - x_i|^2 / h^2
//   10     sum over wall particles of V_j W_ij
//   11..13 the uncorrected acceleration a_i / |g|
//   14     sum V_j (v_j - v_i) . grad_i W_ij * h / c0
//   15     |v_i| / c0
// (v: the leap-frog velocity the force loop uses; rho, p: this step's density.)
//
// Network: x = bf16((f - mean) * inv_std); h1 = bf16(silu(W1 x + b1));
// h2 = bf16(silu(W2 h1 + b2)); h3 = bf16(silu(W3 h2 + b3)); y = W4 h3 + b4;
// correction = out_scale * clamp(y, +-out_limit) (the limit guards a coarse run
// against outputs far outside the training data; none by default).  BF16
// parameters and activations, FP32 dot products
// on the tensor cores (the products of two BF16 values are exact in FP32).
// Training: the loss 0.5/n sum |y - t|^2, gradients through the same forward (its dot
// products on the FP32 pipes)
// (rounding treated as identity), Adam on an FP32 master copy.
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "closure.h"
#include "host_common.h"
#include "neighbor_walk.cuh"

namespace cmag {

namespace {

constexpr int kWalkThreads = 128;  // per block of the feature and interpolation walks
constexpr int kInterpLanes = 4;    // lanes that share an interpolation point
constexpr uint32_t kInterpPoints = kWalkThreads / kInterpLanes;  // points of a block

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ float sigmoid(float z) { return 1.0f / (1.0f + expf(-z)); }

template <int N>
__device__ __forceinline__ void load_row(const float *src, float (&v)[N])
{
    const float4 *s = reinterpret_cast<const float4 *>(src);
#pragma unroll
    for (int q = 0; q < N / 4; ++q) {
        const float4 t = s[q];
        v[4 * q] = t.x; v[4 * q + 1] = t.y; v[4 * q + 2] = t.z; v[4 * q + 3] = t.w;
    }
}

__device__ __forceinline__ void normalise(const float *mean, const float *inv_std,
                                          const float (&f)[kFeat], float (&x)[kFeat])
{
#pragma unroll
    for (int k = 0; k < kFeat; ++k) x[k] = bf16r((f[k] - mean[k]) * inv_std[k]);
}

// What the neighbour sums below read of candidate j besides its position, in one load:
// a vector (xyz) and its volume m / rho_j (w).  v: in original order through idx
// (ORIGINAL), or in sorted order.
template <bool ORIGINAL>
__global__ void __launch_bounds__(256)
    k_neighbor_values(float mass, const float4 *__restrict__ v, const float2 *__restrict__ aux,
                      const uint32_t *__restrict__ idx, uint32_t n, float4 *__restrict__ out)
{
    pdl_entry();
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const uint32_t o = ORIGINAL ? idx[j] : j;
    float4 a = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (o < n) {  // o >= n only after a failed sort: no volume
        a = __ldg(v + o);
        a.w = mass / aux[j].y;
    }
    out[j] = a;
}

// Calls visit(j, a, b, two) for the candidates of the cell box around q in the walk's
// order, two of a run at a time: positions a of j and, with `two`, b of j + 1.
// G lanes share a point: each takes every G-th row of the box.
template <bool PLANAR, bool TRIM, int G, class Visit>
__device__ __forceinline__ void for_each_two(const DevParams &p, const float4 *__restrict__ spos,
                                             const uint32_t *__restrict__ off, int lane, float4 q, Visit &&visit)
{
    walk::for_each_run<CMAG_DAMBREAK, PLANAR, TRIM, G>(
        p, off, lane, grid_pos(p, q.x, q.y, q.z), walk::frac_cell(p, q),
        [&](uint32_t b, uint32_t e, float, float, float) {
            for (uint32_t j = b; j < e; j += 2) {
                const bool two = j + 1 < e;
                const float4 a = __ldg(spos + j);
                visit(j, a, __ldg(spos + (two ? j + 1 : j)), two);
            }
        });
}

__device__ __forceinline__ float2 both(float v) { return make_float2(v, v); }

// Distances of candidates a, b from q and their kernel weights: the operations of
// kernel_w on each half (Wendland in paired FP32; cubic spline one by one).
struct TwoWeights {
    float2 rx, ry, rz, d2, inv_d, q, w;
    bool in0, in1;
};
__device__ __forceinline__ bool two_distances(const DevParams &p, float4 q, const float4 &a, const float4 &b,
                                              bool two, TwoWeights &t)
{
    t.rx = __fadd2_rn(make_float2(a.x, b.x), both(-q.x));  // x_j - x_i
    t.ry = __fadd2_rn(make_float2(a.y, b.y), both(-q.y));
    t.rz = __fadd2_rn(make_float2(a.z, b.z), both(-q.z));
    t.d2 = __ffma2_rn(t.rz, t.rz, __ffma2_rn(t.ry, t.ry, __fmul2_rn(t.rx, t.rx)));
    t.in0 = t.d2.x < p.support2;
    t.in1 = two && t.d2.y < p.support2;
    return t.in0 || t.in1;
}
__device__ __forceinline__ void two_weights(const DevParams &p, TwoWeights &t)
{
    t.inv_d = make_float2(t.d2.x > 0.0f ? rsqrtf(t.d2.x) : 0.0f, t.d2.y > 0.0f ? rsqrtf(t.d2.y) : 0.0f);
    t.q = __fmul2_rn(__fmul2_rn(t.d2, t.inv_d), both(p.inv_h));
    if (p.kernel == CMAG_KERNEL_WENDLAND) {
        const float2 u = __ffma2_rn(t.q, both(-0.5f), both(1.0f)), u2 = __fmul2_rn(u, u);
        t.w = __fmul2_rn(__fmul2_rn(both(p.w_norm), __fmul2_rn(u2, u2)), __ffma2_rn(t.q, both(2.0f), both(1.0f)));
    } else {
        t.w = make_float2(kernel_w(p, t.q.x), kernel_w(p, t.q.y));
    }
}

// The 16 features of a fluid particle at pi with velocity vi (acc_i: its uncorrected
// acceleration): sums over every candidate in the walk's order, which is kept (the
// correction steers the flow, so another order would change a whole run).  65,536 fluid
// particles are 13 warps an SM, and each walks one dependent chain: bound by its
// latency.  Two candidates at a time put two loads in flight and share paired FP32
// operations; volume and velocity come in one load instead of a load, a division and a
// load behind the support test; a candidate outside the support adds nothing, whatever
// it holds.  81 us one at a time, 61 us so (plus 3.5 us for the values) at 65,536 fluid
// particles among 176,000; four lanes to a particle that hand their terms on in order
// took 197 us (a row holds four candidates, too few for the exchange).
template <bool PLANAR, bool TRIM>
__device__ __forceinline__ void features(const DevParams &p, const float4 *__restrict__ spos,
                                         const float4 *__restrict__ nval, float4 mi,
                                         const uint32_t *__restrict__ off, float4 pi, float4 vi,
                                         float4 acc_i, float (&f)[kFeat])
{
    const float ih = p.inv_h, ic = 1.0f / p.c0;
    float s1x = 0.f, s1y = 0.f, s1z = 0.f, svx = 0.f, svy = 0.f, svz = 0.f;
    float shep = 0.f, s2 = 0.f, wall = 0.f, div = 0.f;
    for_each_two<PLANAR, TRIM, 1>(p, spos, off, 0, pi, [&](uint32_t j, const float4 &a, const float4 &b, bool two) {
        TwoWeights t;
        if (!two_distances(p, pi, a, b, two, t)) return;
        const float4 va = __ldg(nval + j), vb = __ldg(nval + (two ? j + 1 : j));
        two_weights(p, t);
        const float2 vol = make_float2(va.w, vb.w);
        const float2 vw = __fmul2_rn(vol, t.w);
        const float2 dvx = __fadd2_rn(make_float2(va.x, vb.x), both(-vi.x)),
                     dvy = __fadd2_rn(make_float2(va.y, vb.y), both(-vi.y)),
                     dvz = __fadd2_rn(make_float2(va.z, vb.z), both(-vi.z));
        // grad_i W_ij = dW/dr (x_i - x_j) / |x_i - x_j|
        float2 dw;
        if (p.kernel == CMAG_KERNEL_WENDLAND) {
            const float2 u = __ffma2_rn(t.q, both(-0.5f), both(1.0f));
            dw = __fmul2_rn(__fmul2_rn(both(-2.5f * p.dw_norm), t.q), __fmul2_rn(__fmul2_rn(u, u), u));
        } else {
            dw = make_float2(kernel_dw(p, t.q.x), kernel_dw(p, t.q.y));
        }
        const float2 gw = __fmul2_rn(dw, t.inv_d);
        const float2 dot = __ffma2_rn(dvz, t.rz, __ffma2_rn(dvy, t.ry, __fmul2_rn(dvx, t.rx)));
        const float2 g = __fmul2_rn(make_float2(-vol.x, -vol.y), gw);
        auto add = [&](float w, float rx, float ry, float rz, float d2, float vx, float vy, float vz, float type,
                       float gj, float dj) {
            s1x = __fmaf_rn(w, rx, s1x); s1y = __fmaf_rn(w, ry, s1y); s1z = __fmaf_rn(w, rz, s1z);
            svx = __fmaf_rn(w, vx, svx); svy = __fmaf_rn(w, vy, svy); svz = __fmaf_rn(w, vz, svz);
            shep += w;
            s2 = __fmaf_rn(w, d2, s2);
            if (type != (float)CMAG_FLUID) wall += w;
            if (d2 > 0.0f) div = __fmaf_rn(gj, dj, div);
        };
        if (t.in0) add(vw.x, t.rx.x, t.ry.x, t.rz.x, t.d2.x, dvx.x, dvy.x, dvz.x, a.w, g.x, dot.x);
        if (t.in1) add(vw.y, t.rx.y, t.ry.y, t.rz.y, t.d2.y, dvx.y, dvy.y, dvz.y, b.w, g.y, dot.y);
    });
    const float ig = rsqrtf(p.gvx * p.gvx + p.gvy * p.gvy + p.gvz * p.gvz);
    f[0] = mi.x / p.rho0 - 1.0f;
    f[1] = mi.y / p.B;
    f[2] = s1x * ih; f[3] = s1y * ih; f[4] = s1z * ih;
    f[5] = svx * ic; f[6] = svy * ic; f[7] = svz * ic;
    f[8] = shep;
    f[9] = s2 * ih * ih;
    f[10] = wall;
    f[11] = acc_i.x * ig; f[12] = acc_i.y * ig; f[13] = acc_i.z * ig;
    f[14] = div * p.h * ic;
    f[15] = sqrtf(vi.x * vi.x + vi.y * vi.y + vi.z * vi.z) * ic;
}

// NORM false: the raw features of every fluid particle to feat[o * 16] (original
// order o); NORM true: the normalised BF16 network input of every sorted particle
// to xb[i * 16] (zeros for walls).
template <bool PLANAR, bool TRIM, bool NORM>
__global__ void __launch_bounds__(kWalkThreads)
    k_closure_features(DevParams p, ClosureView c, const float4 *__restrict__ spos,
                       const float4 *__restrict__ nval, const float4 *__restrict__ meas, const uint32_t *__restrict__ idx,
                       const uint32_t *__restrict__ off, const float4 *__restrict__ acc,
                       float *feat, __nv_bfloat16 *xb)
{
    pdl_entry();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= p.n) return;
    const float4 pi = spos[i];
    const uint32_t o = idx[i];
    const bool fluid = pi.w == (float)CMAG_FLUID && o < p.n;  // o < n unless the sort failed
    if (NORM && !fluid) {
        uint4 *dst = reinterpret_cast<uint4 *>(xb + (size_t)i * kFeat);
        dst[0] = dst[1] = make_uint4(0, 0, 0, 0);
    }
    if (!fluid) return;
    float f[kFeat];
    features<PLANAR, TRIM>(p, spos, nval, meas[i], off, pi, nval[i], acc[o], f);
    if (!NORM) {
        float4 *dst = reinterpret_cast<float4 *>(feat + (size_t)o * kFeat);
#pragma unroll
        for (int q = 0; q < kFeat / 4; ++q) dst[q] = make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
        return;
    }
    float x[kFeat];
    normalise(c.mean, c.inv_std, f, x);
    uint32_t w[kFeat / 2];
#pragma unroll
    for (int k = 0; k < kFeat / 2; ++k) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(x[2 * k], x[2 * k + 1]);
        w[k] = *reinterpret_cast<const uint32_t *>(&v);
    }
    uint4 *dst = reinterpret_cast<uint4 *>(xb + (size_t)i * kFeat);
    dst[0] = make_uint4(w[0], w[1], w[2], w[3]);
    dst[1] = make_uint4(w[4], w[5], w[6], w[7]);
}

// raw FP32 feature rows -> normalised BF16 network input rows
__global__ void k_normalise(ClosureView c, const float *__restrict__ feat, uint32_t n,
                            __nv_bfloat16 *__restrict__ xb)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    float f[kFeat], x[kFeat];
    load_row(feat + (size_t)s * kFeat, f);
    normalise(c.mean, c.inv_std, f, x);
#pragma unroll
    for (int k = 0; k < kFeat / 2; ++k)
        reinterpret_cast<__nv_bfloat162 *>(xb + (size_t)s * kFeat)[k] = __floats2bfloat162_rn(x[2 * k], x[2 * k + 1]);
}

// ---- the network on the tensor cores: mma.sync m16n8k16, BF16 in, FP32 accumulate.
// A warp evaluates 16 rows at a time; a layer's FP32 accumulator fragments become
// the next layer's BF16 A fragments in registers (the C layout of n-tiles 2j and
// 2j+1 is the A layout of k-tile j), so activations never leave the registers.

constexpr int kW1Stride = 24;   // BF16 per shared row of W1 (16 + 8: conflict-free fragment loads)
constexpr int kWStride = 72;    // BF16 per shared row of W2, W3, W4 (64 + 8)
constexpr int kSW1 = 0, kSW2 = kSW1 + kHidden * kW1Stride, kSW3 = kSW2 + kHidden * kWStride,
              kSW4 = kSW3 + kHidden * kWStride, kSWEnd = kSW4 + 8 * kWStride;
constexpr int kSB1 = 0, kSB2 = kSB1 + kHidden, kSB3 = kSB2 + kHidden, kSB4 = kSB3 + kHidden,
              kSBEnd = kSB4 + 8;

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ uint32_t pack_silu(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo * sigmoid(lo), hi * sigmoid(hi));
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ uint32_t lds32(const __nv_bfloat16 *p)
{
    return *reinterpret_cast<const uint32_t *>(p);
}

// one hidden layer: c[nt] = bias + A x W^T over KT k-tiles; W rows of `stride` BF16
template <int KT>
__device__ __forceinline__ void hidden_layer(const __nv_bfloat16 *W, int stride, const float *b,
                                             const uint32_t (&a)[KT][4], float (&c)[8][4], int g, int t)
{
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        c[nt][0] = c[nt][2] = b[nt * 8 + 2 * t];
        c[nt][1] = c[nt][3] = b[nt * 8 + 2 * t + 1];
    }
#pragma unroll
    for (int kt = 0; kt < KT; ++kt)
#pragma unroll
        for (int nt = 0; nt < 8; ++nt) {
            const __nv_bfloat16 *row = W + (nt * 8 + g) * stride + kt * 16 + 2 * t;
            mma16816(c[nt], a[kt], lds32(row), lds32(row + 8));
        }
}

__device__ __forceinline__ void to_a(const float (&c)[8][4], uint32_t (&a)[4][4])
{
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
        a[kt][0] = pack_silu(c[2 * kt][0], c[2 * kt][1]);
        a[kt][1] = pack_silu(c[2 * kt][2], c[2 * kt][3]);
        a[kt][2] = pack_silu(c[2 * kt + 1][0], c[2 * kt + 1][1]);
        a[kt][3] = pack_silu(c[2 * kt + 1][2], c[2 * kt + 1][3]);
    }
}

// APPLY false: out[r * 3 ..] = network(xb row r) for r < n.
// APPLY true: rows are sorted particles; acc[idx[r]] += out_scale * clamp(y) for
// fluid rows.
// Byte layout of the staged weights: padded BF16 rows of W1..W4, then FP32 biases.
constexpr int kImageBytes = kSWEnd * 2 + kSBEnd * 4;
constexpr int kImageWords = kImageBytes / 16;
static_assert(kSWEnd * 2 % 16 == 0 && kImageBytes % 16 == 0, "image rows must stay 16-byte aligned");

// Builds the image once per parameter change (one thread per 32-bit image word),
// so each network block stages it with plain 16-byte copies.
__global__ void k_pack(const __nv_bfloat16 *__restrict__ w, uint32_t *__restrict__ image)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < kSWEnd / 2) {  // two BF16 weights per word
        __nv_bfloat16 h[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int q = 2 * k + e;
            __nv_bfloat16 v = __float2bfloat16_rn(0.0f);
            if (q < kSW2) {
                const int o = q / kW1Stride, i = q % kW1Stride;
                if (i < kFeat) v = w[kOffW1 + o * kFeat + i];
            } else {
                const int base = q < kSW3 ? kSW2 : (q < kSW4 ? kSW3 : kSW4);
                const int off = q < kSW3 ? kOffW2 : (q < kSW4 ? kOffW3 : kOffW4);
                const int o = (q - base) / kWStride, i = (q - base) % kWStride;
                if (i < kHidden && (base != kSW4 || o < kOut)) v = w[off + o * kHidden + i];
            }
            h[e] = v;
        }
        const __nv_bfloat162 v2 = __halves2bfloat162(h[0], h[1]);
        image[k] = *reinterpret_cast<const uint32_t *>(&v2);
    } else if (k < kImageBytes / 4) {
        const int b = k - kSWEnd / 2;
        float v = 0.0f;
        if (b < kSB2) v = __bfloat162float(w[kOffB1 + b]);
        else if (b < kSB3) v = __bfloat162float(w[kOffB2 + b - kSB2]);
        else if (b < kSB4) v = __bfloat162float(w[kOffB3 + b - kSB3]);
        else if (b - kSB4 < kOut) v = __bfloat162float(w[kOffB4 + b - kSB4]);
        image[k] = __float_as_uint(v);
    }
}

// APPLY false: out[r * 3 ..] = network(xb row r) for r < n.
// APPLY true: rows are sorted particles; acc[idx[r]] += out_scale * clamp(y) for
// fluid rows.
template <bool APPLY>
__global__ void __launch_bounds__(128)
    k_mlp(ClosureView c, const __nv_bfloat16 *__restrict__ xb, uint32_t n,
          const float4 *__restrict__ spos, const uint32_t *__restrict__ idx, float4 *acc,
          float *__restrict__ out)
{
    pdl_entry();
    __shared__ uint4 simage[kImageWords];
    for (int k = threadIdx.x; k < kImageWords; k += blockDim.x) simage[k] = __ldg(c.image + k);
    const __nv_bfloat16 *sw = reinterpret_cast<const __nv_bfloat16 *>(simage);
    const float *sb = reinterpret_cast<const float *>(simage) + kSWEnd / 2;
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const uint32_t warps = gridDim.x * (blockDim.x >> 5);
    const uint32_t tiles = (n + 15) / 16;
    const float scale = APPLY ? *c.out_scale : 0.0f, lim = APPLY ? *c.out_limit : 0.0f;
    for (uint32_t tile = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); tile < tiles; tile += warps) {
        const uint32_t r0 = tile * 16 + g, r1 = r0 + 8;
        if (APPLY) {  // sorted order keeps wall cells together: skip tiles without fluid
            const bool f = (r0 < n && spos[r0].w == (float)CMAG_FLUID) ||
                           (r1 < n && spos[r1].w == (float)CMAG_FLUID);
            if (!__any_sync(0xffffffffu, f)) continue;
        }
        uint32_t a1[1][4];
        {
            const uint32_t *x0 = reinterpret_cast<const uint32_t *>(xb + (size_t)r0 * kFeat);
            const uint32_t *x1 = reinterpret_cast<const uint32_t *>(xb + (size_t)r1 * kFeat);
            a1[0][0] = r0 < n ? x0[t] : 0u;
            a1[0][1] = r1 < n ? x1[t] : 0u;
            a1[0][2] = r0 < n ? x0[t + 4] : 0u;
            a1[0][3] = r1 < n ? x1[t + 4] : 0u;
        }
        float cc[8][4];
        uint32_t a[4][4];
        hidden_layer<1>(sw + kSW1, kW1Stride, sb + kSB1, a1, cc, g, t);
        to_a(cc, a);
        hidden_layer<4>(sw + kSW2, kWStride, sb + kSB2, a, cc, g, t);
        to_a(cc, a);
        hidden_layer<4>(sw + kSW3, kWStride, sb + kSB3, a, cc, g, t);
        to_a(cc, a);
        // output layer (3 of 8 columns used)
        float y[4] = {sb[kSB4 + 2 * t], sb[kSB4 + 2 * t + 1], sb[kSB4 + 2 * t], sb[kSB4 + 2 * t + 1]};
#pragma unroll
        for (int kt = 0; kt < 4; ++kt) {
            const __nv_bfloat16 *row = sw + kSW4 + g * kWStride + kt * 16 + 2 * t;
            mma16816(y, a[kt], lds32(row), lds32(row + 8));
        }
        // lane (g, 0) holds columns 0, 1 of rows r0 (y[0..1]) and r1 (y[2..3]);
        // column 2 sits in lane (g, 1)
        const float y2r0 = __shfl_down_sync(0xffffffffu, y[0], 1);
        const float y2r1 = __shfl_down_sync(0xffffffffu, y[2], 1);
        if (t == 0) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t r = h ? r1 : r0;
                const float o0 = h ? y[2] : y[0], o1 = h ? y[3] : y[1], o2 = h ? y2r1 : y2r0;
                if (r < n && !APPLY) {
                    out[(size_t)r * kOut + 0] = o0;
                    out[(size_t)r * kOut + 1] = o1;
                    out[(size_t)r * kOut + 2] = o2;
                }
                if (r < n && APPLY && spos[r].w == (float)CMAG_FLUID) {
                    const uint32_t o = idx[r];
                    if (o < n) {  // o >= n only after a failed sort
                        float4 av = acc[o];
                        av.x += scale * fminf(fmaxf(o0, -lim), lim);
                        av.y += scale * fminf(fmaxf(o1, -lim), lim);
                        av.z += scale * fminf(fmaxf(o2, -lim), lim);
                        acc[o] = av;
                    }
                }
            }
        }
        __syncwarp();
    }
}

// ---- training: forward and backward on the tensor cores ----------------------------
// A block of 8 warps takes tiles of 64 samples; two warps share 16 samples, each with
// half of a layer's columns.  The forward pass runs on the FP32 pipes in a fixed order
// (forward_layer); each layer's slope of the activation stays in registers, its BF16
// activations go to shared memory.  The backward products run on the tensor cores: they
// need FP32 deltas against BF16 weights or activations, so a delta is split into three
// BF16 parts (8 + 8 + 8 bits hold its 24), whose products are exact; their sums round
// as FP32 ones do (mma_add).  Weight gradients (16 rows and half the columns of each
// matrix to a warp) accumulate in registers over all of the block's tiles and are added
// to global memory once.  Error against 64 bits on the same activations (norm of W1's
// gradient, median of 12 seeds; FP32 pipes before / here): 64 rows 2.8e-7 / 1.7e-7,
// 2048 2.1e-7 / 1.3e-7, 5003 1.8e-7 / 1.2e-7, 65,536 3.4e-7 / 1.1e-7; with the sums in
// one chain on the tensor cores and one copy of the gradient 2.9e-7, -, 2.8e-7, 3.4e-7,
// most of it a gradient shrunk by 2.3e-7 of itself.
// 65,536 samples: 88 us; 423 us in the form before, 128 samples a block on the FP32 pipes
// with one 190 KB block an SM (59 us with the forward pass on the tensor cores too, whose
// activations round the other way now and then: not kept).  Bound by the forward pass's
// instructions and the chain of layers, at four warps a scheduler.
constexpr int kTile = 64;        // samples of a block's tile
constexpr int kBackThreads = 256;  // two warps to 16 samples, 32 of 64 columns each
constexpr int kXStride = 24;     // BF16 per row of inputs and output deltas (conflict-free)
constexpr int kHStride = 72;     // BF16 per row of activations and deltas
constexpr int kPlane = kTile * kHStride;    // one part of a delta
constexpr int kPlane4 = kTile * kXStride;   // one part of the output delta (16 columns, 3 used)
constexpr int kSmemBackward = kImageBytes + 2 * (kTile * kXStride + 3 * kPlane + 3 * kPlane + 3 * kPlane4);

__device__ __forceinline__ uint32_t shared_of(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Four 8x8 BF16 matrices; lane l gives the address of row l % 8 of matrix l / 8.
__device__ __forceinline__ void load_matrices(uint32_t (&r)[4], const __nv_bfloat16 *row)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(shared_of(row))
                 : "memory");
}
__device__ __forceinline__ void load_matrices_trans(uint32_t (&r)[4], const __nv_bfloat16 *row)
{
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(shared_of(row))
                 : "memory");
}

__device__ __forceinline__ uint32_t pack2(float lo, float hi)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ __forceinline__ float2 unpack2(uint32_t v)
{
    return make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}

// What is left of x after its BF16 part (0 where that part is infinite).
__device__ __forceinline__ float rest_of(float x, float part)
{
    return fabsf(part) <= 3.4e38f ? x - part : 0.0f;
}

// The three BF16 parts of (x, y) into the planes at `at`.
__device__ __forceinline__ void store_parts(__nv_bfloat16 *at, int plane, float x, float y)
{
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const uint32_t w = pack2(x, y);
        *reinterpret_cast<uint32_t *>(at + q * plane) = w;
        const float2 v = unpack2(w);
        x = rest_of(x, v.x);
        y = rest_of(y, v.y);
    }
}

// c = activations of a layer (pre-activations in c): BF16 activations of the warp's 16
// rows to h (its row 0 and first column), slopes to c.
__device__ __forceinline__ void activate(float (&c)[4][4], __nv_bfloat16 *h, int g, int t)
{
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        float a[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const float z = c[nt][k], s = sigmoid(z);
            a[k] = z * s;
            c[nt][k] = s * (1.0f + z * (1.0f - s));
        }
        *reinterpret_cast<uint32_t *>(h + g * kHStride + nt * 8 + 2 * t) = pack2(a[0], a[1]);
        *reinterpret_cast<uint32_t *>(h + (g + 8) * kHStride + nt * 8 + 2 * t) = pack2(a[2], a[3]);
    }
}

// c = b + h W^T for the warp's 16 rows and 32 outputs (h in shared memory, K inputs a row;
// W, b: the first output), each sum in FP32 from its bias over ascending inputs: the order
// fixes every pre-activation's bits, and with them which activations round up to the next
// BF16 value.  (On the tensor cores, whose sums round otherwise, about one activation in
// 10,000 went the other way; a gradient moved by up to 4e-5 of itself.)
template <int K, int WSTRIDE, int HSTRIDE>
__device__ __forceinline__ void forward_layer(const __nv_bfloat16 *W, const float *b, const __nv_bfloat16 *h,
                                              float (&c)[4][4], int g, int t)
{
    float2 s0[4], s1[4];  // rows g and g + 8, outputs nt * 8 + 2 t and the next
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) s0[nt] = s1[nt] = make_float2(b[nt * 8 + 2 * t], b[nt * 8 + 2 * t + 1]);
    auto four = [](const __nv_bfloat16 *p, float (&v)[4]) {
        const uint2 u = *reinterpret_cast<const uint2 *>(p);
        const float2 a = unpack2(u.x), e = unpack2(u.y);
        v[0] = a.x, v[1] = a.y, v[2] = e.x, v[3] = e.y;
    };
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float h0[4], h1[4];
        four(h + g * HSTRIDE + k, h0);
        four(h + (g + 8) * HSTRIDE + k, h1);
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            const __nv_bfloat16 *row = W + (nt * 8 + 2 * t) * WSTRIDE + k;
            float w0[4], w1[4];
            four(row, w0);
            four(row + WSTRIDE, w1);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float2 w = make_float2(w0[q], w1[q]);
                s0[nt] = __ffma2_rn(w, make_float2(h0[q], h0[q]), s0[nt]);
                s1[nt] = __ffma2_rn(w, make_float2(h1[q], h1[q]), s1[nt]);
            }
        }
    }
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        c[nt][0] = s0[nt].x;
        c[nt][1] = s0[nt].y;
        c[nt][2] = s1[nt].x;
        c[nt][3] = s1[nt].y;
    }
}

// d = A B: sums of 16 products from zero.
__device__ __forceinline__ void mma16816_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
        "{%8,%9}, {%10,%10,%10,%10};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}

// c += A B, MAIN: for the main part of a delta.  The tensor cores truncate a running sum
// at every addition, always towards zero; over a chain of products that shrinks the sum
// by about 1e-7 of it.  So the main part's products are summed from zero, 16 at a time
// (their 16 bits each mostly fit), and added here in FP32, rounded to nearest.  The small
// parts (2^-8 and 2^-16 of the main one) lose nothing that counts in a chain.
template <bool MAIN>
__device__ __forceinline__ void mma_add(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    if (!MAIN) {
        mma16816(c, a, b0, b1);
        return;
    }
    float m[4];
    mma16816_zero(m, a, b0, b1);
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += m[i];
}

// c = d W for the warp's 16 rows (W: its first column): the deltas of the layer below
// before its slopes; the small parts first.
template <bool MAIN>
__device__ __forceinline__ void backward_part(const __nv_bfloat16 *W, const __nv_bfloat16 *d, float (&c)[4][4],
                                              int lane)
{
    const int r = lane & 7, q = lane >> 3;
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
        uint32_t a[4];
        load_matrices(a, d + (r + (q & 1) * 8) * kHStride + kt * 16 + (q >> 1) * 8);
#pragma unroll
        for (int nt = 0; nt < 4; nt += 2) {
            uint32_t w[4];
            load_matrices_trans(w, W + (kt * 16 + (q & 1) * 8 + r) * kWStride + nt * 8 + (q >> 1) * 8);
            mma_add<MAIN>(c[nt], a, w[0], w[1]);
            mma_add<MAIN>(c[nt + 1], a, w[2], w[3]);
        }
    }
}
__device__ __forceinline__ void backward_layer(const __nv_bfloat16 *W, const __nv_bfloat16 *d, float (&c)[4][4],
                                               int lane)
{
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) c[nt][0] = c[nt][1] = c[nt][2] = c[nt][3] = 0.0f;
#pragma unroll 1
    for (int part = 2; part >= 1; --part) backward_part<false>(W, d + part * kPlane, c, lane);
    backward_part<true>(W, d, c, lane);
}

// g[nt] += sum over the tile's samples of d[s][m0 ..] h[s][nt * 8 ..], and the same
// against ones into gb (bias: in one warp of those that share m0).  A tile's products are
// summed from zero, the small parts first, and then added.
template <bool MAIN, int NT, int DSTRIDE, int HSTRIDE>
__device__ __forceinline__ void grad_part(float (&a0)[NT][4], float (&ab)[4], const __nv_bfloat16 *d, int m0,
                                          const __nv_bfloat16 *h, bool bias, int lane)
{
    constexpr uint32_t kOnes = 0x3f803f80u;
    const int r = lane & 7, q = lane >> 3;
#pragma unroll
    for (int s0 = 0; s0 < kTile; s0 += 16) {
        uint32_t a[4];
        load_matrices_trans(a, d + (s0 + (q >> 1) * 8 + r) * DSTRIDE + m0 + (q & 1) * 8);
#pragma unroll
        for (int k = 0; k < NT / 2; ++k) {
            uint32_t b[4];
            load_matrices_trans(b, h + (s0 + (q & 1) * 8 + r) * HSTRIDE + k * 16 + (q >> 1) * 8);
            mma_add<MAIN>(a0[2 * k], a, b[0], b[1]);
            mma_add<MAIN>(a0[2 * k + 1], a, b[2], b[3]);
        }
        if (bias) mma_add<MAIN>(ab, a, kOnes, kOnes);
    }
}
template <int NT, int DSTRIDE, int HSTRIDE>
__device__ __forceinline__ void weight_grad(float (&g)[NT][4], float (&gb)[4], const __nv_bfloat16 *d, int plane,
                                            int m0, const __nv_bfloat16 *h, bool bias, int lane)
{
    float a0[NT][4] = {}, ab[4] = {};
#pragma unroll 1
    for (int part = 2; part >= 1; --part)
        grad_part<false, NT, DSTRIDE, HSTRIDE>(a0, ab, d + part * plane, m0, h, bias, lane);
    grad_part<true, NT, DSTRIDE, HSTRIDE>(a0, ab, d, m0, h, bias, lane);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        gb[i] += ab[i];
#pragma unroll
        for (int nt = 0; nt < NT; ++nt) g[nt][i] += a0[nt][i];
    }
}

// (x, y) added to p[0], p[1] (8-byte aligned).
__device__ __forceinline__ void add_pair(float *p, float x, float y)
{
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};" : : "l"(p), "f"(x), "f"(y) : "memory");
}

template <int NT>
__device__ __forceinline__ void add_gradient(float *grad, int columns, const float (&g)[NT][4], int row, int rows,
                                             int col, int t)
{
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        if (row < rows) add_pair(grad + row * columns + col + nt * 8 + 2 * t, g[nt][0], g[nt][1]);
        if (row + 8 < rows) add_pair(grad + (row + 8) * columns + col + nt * 8 + 2 * t, g[nt][2], g[nt][3]);
    }
}

__device__ __forceinline__ void multiply_store(float (&c)[4][4], const float (&slope)[4][4], __nv_bfloat16 *d, int g,
                                               int t)
{
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) {
        store_parts(d + g * kHStride + nt * 8 + 2 * t, kPlane, c[nt][0] * slope[nt][0], c[nt][1] * slope[nt][1]);
        store_parts(d + (g + 8) * kHStride + nt * 8 + 2 * t, kPlane, c[nt][2] * slope[nt][2], c[nt][3] * slope[nt][3]);
    }
}

// Loss and gradient over n samples; both are added to global FP32 accumulators, the
// gradient to one of kGradCopies of them (closure.h).
__global__ void __launch_bounds__(kBackThreads, 2)
    k_backward(ClosureView cv, const float *__restrict__ feat, const float *__restrict__ target, uint32_t n,
               float *__restrict__ grad, float *__restrict__ loss)
{
    extern __shared__ uint4 smem[];
    const __nv_bfloat16 *sw = reinterpret_cast<const __nv_bfloat16 *>(smem);
    const float *sb = reinterpret_cast<const float *>(smem) + kSWEnd / 2;
    __nv_bfloat16 *X = reinterpret_cast<__nv_bfloat16 *>(reinterpret_cast<char *>(smem) + kImageBytes);
    __nv_bfloat16 *H1 = X + kTile * kXStride, *H2 = H1 + kPlane, *H3 = H2 + kPlane;
    __nv_bfloat16 *D = H3 + kPlane;       // three parts of one layer's deltas
    __nv_bfloat16 *D4 = D + 3 * kPlane;   // three parts of the output deltas
    for (int k = threadIdx.x; k < kImageWords; k += kBackThreads) smem[k] = __ldg(cv.image + k);
    for (int k = threadIdx.x; k < 3 * kPlane4 / 2; k += kBackThreads) reinterpret_cast<uint32_t *>(D4)[k] = 0u;
    __syncthreads();

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
    const int w0 = (warp & 3) * 16;  // the warp's first row in the tile, and its first row of the gradients
    const int n0 = (warp >> 2) * 32;  // its first column of a layer, and of the gradients
    const bool left = n0 == 0;
    auto pair_sync = [&] { asm volatile("bar.sync %0, 64;" : : "r"(1 + (warp & 3)) : "memory"); };
    const float inv_n = 1.0f / (float)n;
    // ge: W1's gradient in the left warps, W4's in the right ones
    float g2[4][4] = {}, g3[4][4] = {}, ge[2][4] = {};
    float gb2[4] = {}, gb3[4] = {}, gbe[4] = {};
    double l = 0.0;
    const uint32_t tiles = (n + kTile - 1) / kTile;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t r0 = tile * kTile + w0 + g, r1 = r0 + 8;
        // inputs
        if (left) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int k = 2 * t + 8 * half;
                const float m0 = cv.mean[k], m1 = cv.mean[k + 1], i0 = cv.inv_std[k], i1 = cv.inv_std[k + 1];
                float2 f0 = make_float2(0.0f, 0.0f), f1 = f0;
                if (r0 < n) f0 = __ldg(reinterpret_cast<const float2 *>(feat + (size_t)r0 * kFeat + k));
                if (r1 < n) f1 = __ldg(reinterpret_cast<const float2 *>(feat + (size_t)r1 * kFeat + k));
                *reinterpret_cast<uint32_t *>(X + (w0 + g) * kXStride + k) = pack2((f0.x - m0) * i0, (f0.y - m1) * i1);
                *reinterpret_cast<uint32_t *>(X + (w0 + g + 8) * kXStride + k) = pack2((f1.x - m0) * i0, (f1.y - m1) * i1);
            }
        }
        pair_sync();
        // forward
        float s1[4][4], s2[4][4], c[4][4];
        forward_layer<kFeat, kW1Stride, kXStride>(sw + kSW1 + n0 * kW1Stride, sb + kSB1 + n0, X + w0 * kXStride, s1, g, t);
        activate(s1, H1 + w0 * kHStride + n0, g, t);
        pair_sync();
        forward_layer<kHidden, kWStride, kHStride>(sw + kSW2 + n0 * kWStride, sb + kSB2 + n0, H1 + w0 * kHStride, s2, g, t);
        activate(s2, H2 + w0 * kHStride + n0, g, t);
        pair_sync();
        forward_layer<kHidden, kWStride, kHStride>(sw + kSW3 + n0 * kWStride, sb + kSB3 + n0, H2 + w0 * kHStride, c, g, t);
        activate(c, H3 + w0 * kHStride + n0, g, t);
        pair_sync();
        // outputs, in FP32 (three columns: a lane's 16 activations of each row, then the
        // four lanes of the row), and the output deltas
        float d0[kOut], d1[kOut];
#pragma unroll
        for (int o = 0; o < kOut; ++o) {
            float y0 = 0.0f, y1 = 0.0f;
#pragma unroll
            for (int nt = 0; nt < 8; ++nt) {
                const float2 w = unpack2(lds32(sw + kSW4 + o * kWStride + nt * 8 + 2 * t));
                const float2 h0 = unpack2(lds32(H3 + (w0 + g) * kHStride + nt * 8 + 2 * t)),
                             h1 = unpack2(lds32(H3 + (w0 + g + 8) * kHStride + nt * 8 + 2 * t));
                y0 = __fmaf_rn(w.y, h0.y, __fmaf_rn(w.x, h0.x, y0));
                y1 = __fmaf_rn(w.y, h1.y, __fmaf_rn(w.x, h1.x, y1));
            }
            y0 += __shfl_xor_sync(0xffffffffu, y0, 1);
            y1 += __shfl_xor_sync(0xffffffffu, y1, 1);
            y0 += __shfl_xor_sync(0xffffffffu, y0, 2);
            y1 += __shfl_xor_sync(0xffffffffu, y1, 2);
            const float b = sb[kSB4 + o];
            d0[o] = r0 < n ? y0 + b - __ldg(target + (size_t)r0 * kOut + o) : 0.0f;
            d1[o] = r1 < n ? y1 + b - __ldg(target + (size_t)r1 * kOut + o) : 0.0f;
            if (left && t == 0) l += (double)d0[o] * d0[o] + (double)d1[o] * d1[o];
            d0[o] *= inv_n;
            d1[o] *= inv_n;
        }
        if (left && t == 0) {
            store_parts(D4 + (w0 + g) * kXStride, kPlane4, d0[0], d0[1]);
            store_parts(D4 + (w0 + g + 8) * kXStride, kPlane4, d1[0], d1[1]);
        } else if (left && t == 1) {
            store_parts(D4 + (w0 + g) * kXStride + 2, kPlane4, d0[2], 0.0f);
            store_parts(D4 + (w0 + g + 8) * kXStride + 2, kPlane4, d1[2], 0.0f);
        }
        // layer 3's deltas (W4 has three rows: FP32)
        float d[4][4];
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
            d[nt][0] = d[nt][1] = d[nt][2] = d[nt][3] = 0.0f;
#pragma unroll
            for (int o = 0; o < kOut; ++o) {
                const float2 w = unpack2(lds32(sw + kSW4 + o * kWStride + n0 + nt * 8 + 2 * t));
                d[nt][0] = __fmaf_rn(w.x, d0[o], d[nt][0]);
                d[nt][1] = __fmaf_rn(w.y, d0[o], d[nt][1]);
                d[nt][2] = __fmaf_rn(w.x, d1[o], d[nt][2]);
                d[nt][3] = __fmaf_rn(w.y, d1[o], d[nt][3]);
            }
        }
        multiply_store(d, c, D + w0 * kHStride + n0, g, t);
        __syncthreads();
        if (!left) weight_grad<2, kXStride, kHStride>(ge, gbe, D4, kPlane4, 0, H3 + w0, true, lane);
        weight_grad<4, kHStride, kHStride>(g3, gb3, D, kPlane, w0, H2 + n0, left, lane);
        backward_layer(sw + kSW3 + n0, D + w0 * kHStride, c, lane);
        __syncthreads();
        multiply_store(c, s2, D + w0 * kHStride + n0, g, t);
        __syncthreads();
        weight_grad<4, kHStride, kHStride>(g2, gb2, D, kPlane, w0, H1 + n0, left, lane);
        backward_layer(sw + kSW2 + n0, D + w0 * kHStride, c, lane);
        __syncthreads();
        multiply_store(c, s1, D + w0 * kHStride + n0, g, t);
        __syncthreads();
        if (left) weight_grad<2, kHStride, kXStride>(ge, gbe, D, kPlane, w0, X, true, lane);
        __syncthreads();
    }
    grad += (blockIdx.x % kGradCopies) * kGradStride;
    add_gradient(grad + kOffW2, kHidden, g2, w0 + g, kHidden, n0, t);
    add_gradient(grad + kOffW3, kHidden, g3, w0 + g, kHidden, n0, t);
    if (left) add_gradient(grad + kOffW1, kFeat, ge, w0 + g, kHidden, 0, t);
    else add_gradient(grad + kOffW4, kHidden, ge, g, kOut, w0, t);
    if (t == 0 && left) {  // every column of a bias product holds the sum
        const int o = w0 + g;
        atomicAdd(grad + kOffB1 + o, gbe[0]);
        atomicAdd(grad + kOffB1 + o + 8, gbe[2]);
        atomicAdd(grad + kOffB2 + o, gb2[0]);
        atomicAdd(grad + kOffB2 + o + 8, gb2[2]);
        atomicAdd(grad + kOffB3 + o, gb3[0]);
        atomicAdd(grad + kOffB3 + o + 8, gb3[2]);
    }
    if (t == 0 && warp == 4 && g < kOut) atomicAdd(grad + kOffB4 + g, gbe[0]);
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) l += __shfl_xor_sync(0xffffffffu, l, w);
    // FP64: few operations, and the sum of many small squares keeps its digits
    __shared__ double s_loss[kBackThreads / 32];
    if (lane == 0) s_loss[warp] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kBackThreads / 32; ++w) l += s_loss[w];
        atomicAdd(loss, (float)(0.5 * l * inv_n));
    }
}

// Where parameter k lies in the network image (k_pack).
__device__ __forceinline__ void update_image(uint32_t *image, int k, float v)
{
    int row, col, base, stride, bias = -1;
    if (k < kOffB1) base = kSW1, stride = kW1Stride, row = k / kFeat, col = k % kFeat;
    else if (k < kOffW2) bias = kSB1 + k - kOffB1;
    else if (k < kOffB2) base = kSW2, stride = kWStride, row = (k - kOffW2) / kHidden, col = (k - kOffW2) % kHidden;
    else if (k < kOffW3) bias = kSB2 + k - kOffB2;
    else if (k < kOffB3) base = kSW3, stride = kWStride, row = (k - kOffW3) / kHidden, col = (k - kOffW3) % kHidden;
    else if (k < kOffW4) bias = kSB3 + k - kOffB3;
    else if (k < kOffB4) base = kSW4, stride = kWStride, row = (k - kOffW4) / kHidden, col = (k - kOffW4) % kHidden;
    else bias = kSB4 + k - kOffB4;
    if (bias >= 0) image[kSWEnd / 2 + bias] = __float_as_uint(bf16r(v));
    else reinterpret_cast<__nv_bfloat16 *>(image)[base + row * stride + col] = __float2bfloat16_rn(v);
}

// The gradient of parameter k: the sum of its copies.
__device__ __forceinline__ float gradient_of(const float *grad, int k)
{
    static_assert(kGradCopies == 4, "added in pairs");
    grad += k;
    return (grad[0] + grad[kGradStride]) + (grad[2 * kGradStride] + grad[3 * kGradStride]);
}

// Leaves the gradient in its first copy.
__global__ void k_fold_gradient(float *grad)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < kClosureParams) grad[k] = gradient_of(grad, k);
}

__global__ void k_adam(float *master, float *m, float *v, float *grad, __nv_bfloat16 *w, uint32_t *image,
                       float lr, float beta1, float beta2, float eps, float bias1, float bias2)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kClosureParams) return;
    const float g = gradient_of(grad, k);
    const float mk = beta1 * m[k] + (1.0f - beta1) * g;
    const float vk = beta2 * v[k] + (1.0f - beta2) * g * g;
    m[k] = mk;
    v[k] = vk;
    const float step = lr * (mk / bias1) / (sqrtf(vk / bias2) + eps);
    const float nw = master[k] - step;
    master[k] = nw;
    w[k] = __float2bfloat16_rn(nw);
    update_image(image, k, nw);
#pragma unroll
    for (int c = 0; c < kGradCopies; ++c) grad[c * kGradStride + k] = 0.0f;
}

__global__ void k_round(const float *master, __nv_bfloat16 *w)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < kClosureParams) w[k] = __float2bfloat16_rn(master[k]);
}

// Shepard-normalised SPH interpolation of a float4 array (original order) of
// the system's fluid particles at arbitrary points: out.xyz = sum_j V_j W a_j /
// sum_j V_j W, out.w = sum_j V_j W (0 where no fluid particle is in reach).
// Bound by the latency of the walk and by lanes of a warp whose rows differ in length:
// four lanes share a point's rows (the sums meet at the end).  At 65,536 points in a
// scene of 176,000 particles: 124 us one candidate at a time, 74 us two at a time, 52 us
// with four lanes (plus 4 us for the values).
template <bool PLANAR, bool TRIM>
__global__ void __launch_bounds__(kWalkThreads)
    k_interp(DevParams p, const float4 *__restrict__ spos, const float4 *__restrict__ nval,
             const uint32_t *__restrict__ off, const float4 *__restrict__ pts, uint32_t n,
             float4 *__restrict__ out)
{
    pdl_entry();
    // (from the block's points: four threads a point pass 2^32 at 2^30 points)
    const uint32_t t = blockIdx.x * kInterpPoints + threadIdx.x / kInterpLanes;
    const float4 q = pts[min(t, n - 1)];
    float sx = 0.f, sy = 0.f, sz = 0.f, sw = 0.f;
    for_each_two<PLANAR, TRIM, kInterpLanes>(p, spos, off, threadIdx.x % kInterpLanes, q, [&](uint32_t j, const float4 &a, const float4 &b, bool two) {
        TwoWeights w;
        if (!two_distances(p, q, a, b, two, w)) return;
        w.in0 = w.in0 && a.w == (float)CMAG_FLUID;
        w.in1 = w.in1 && b.w == (float)CMAG_FLUID;
        if (!(w.in0 || w.in1)) return;
        const float4 va = __ldg(nval + j), vb = __ldg(nval + (two ? j + 1 : j));
        two_weights(p, w);
        const float2 vw = __fmul2_rn(make_float2(va.w, vb.w), w.w);
        if (w.in0) {
            sx = __fmaf_rn(vw.x, va.x, sx); sy = __fmaf_rn(vw.x, va.y, sy); sz = __fmaf_rn(vw.x, va.z, sz);
            sw += vw.x;
        }
        if (w.in1) {
            sx = __fmaf_rn(vw.y, vb.x, sx); sy = __fmaf_rn(vw.y, vb.y, sy); sz = __fmaf_rn(vw.y, vb.z, sz);
            sw += vw.y;
        }
    });
    sx = walk::group_sum<kInterpLanes>(sx);
    sy = walk::group_sum<kInterpLanes>(sy);
    sz = walk::group_sum<kInterpLanes>(sz);
    sw = walk::group_sum<kInterpLanes>(sw);
    if (t >= n || threadIdx.x % kInterpLanes != 0) return;
    const float inv = sw > 0.0f ? 1.0f / sw : 0.0f;
    out[t] = make_float4(sx * inv, sy * inv, sz * inv, sw);
}

template <class K>
void allow_smem(K kernel, size_t bytes)
{
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

template <bool NORM>
void dispatch_features(const DevParams &p, const ClosureView &c, const float4 *spos,
                       const float4 *svel, const float2 *aux, const float4 *meas,
                       const uint32_t *idx, const uint32_t *off, const float4 *acc, float4 *nval,
                       float *feat, __nv_bfloat16 *xb, cudaStream_t st)
{
    if (p.n == 0) return;
    launch_pdl(k_neighbor_values<false>, (p.n + 255) / 256, 256, 0, st, p.mass, svel, aux, idx, p.n, nval);
    const uint32_t blocks = (p.n + kWalkThreads - 1) / kWalkThreads;
#define CMAG_FEAT(PL, TR) \
    launch_pdl(k_closure_features<PL, TR, NORM>, blocks, kWalkThreads, 0, st, p, c, spos, nval, meas, idx, off, acc, feat, xb)
    if (p.planar) {
        if (p.trim) CMAG_FEAT(true, true);
        else CMAG_FEAT(true, false);
    } else {
        if (p.trim) CMAG_FEAT(false, true);
        else CMAG_FEAT(false, false);
    }
#undef CMAG_FEAT
}

// Each block stages the weight image once (23 KB) and its 4 warps loop over
// 16-row tiles, so the grid stays at a few blocks per SM (8 per SM at most)
// however many rows there are.
uint32_t mlp_blocks(uint32_t n)
{
    const uint32_t tiles = (n + 15) / 16;
    const uint32_t cap = 8u * (uint32_t)device_sm_count();
    uint32_t b = (tiles + 3) / 4;
    return b < 1 ? 1 : (b > cap ? cap : b);
}

}  // namespace

void launch_closure_features(const DevParams &p, const float4 *spos, const float4 *svel,
                             const float2 *aux, const float4 *meas, const uint32_t *idx,
                             const uint32_t *off, const float4 *acc, float4 *nval, float *feat, cudaStream_t st)
{
    dispatch_features<false>(p, ClosureView{}, spos, svel, aux, meas, idx, off, acc, nval, feat, nullptr, st);
}

void launch_closure_apply(const DevParams &p, const ClosureView &c, const float4 *spos,
                          const float4 *svel, const float2 *aux, const float4 *meas,
                          const uint32_t *idx, const uint32_t *off, float4 *acc, float4 *nval,
                          __nv_bfloat16 *xb, cudaStream_t st)
{
    if (p.n == 0) return;
    dispatch_features<true>(p, c, spos, svel, aux, meas, idx, off, acc, nval, nullptr, xb, st);
    launch_pdl(k_mlp<true>, mlp_blocks(p.n), 128, 0, st, c, xb, p.n, spos, idx, acc, (float *)nullptr);
}

void launch_closure_forward(const ClosureView &c, const float *feat, uint32_t n,
                            __nv_bfloat16 *xb, float *out, cudaStream_t st)
{
    if (n == 0) return;
    k_normalise<<<(n + 255) / 256, 256, 0, st>>>(c, feat, n, xb);
    k_mlp<false><<<mlp_blocks(n), 128, 0, st>>>(c, xb, n, nullptr, nullptr, nullptr, out);
}

void launch_interpolate(const DevParams &p, const float4 *spos, const float2 *aux,
                        const uint32_t *idx, const uint32_t *off, const float4 *arr, float4 *nval,
                        const float4 *pts, uint32_t n, float4 *out, cudaStream_t st)
{
    if (n == 0) return;
    launch_pdl(k_neighbor_values<true>, (p.n + 255) / 256, 256, 0, st, p.mass, arr, aux, idx, p.n, nval);
    const uint32_t blocks = (n - 1) / kInterpPoints + 1;
#define CMAG_INTERP(PL, TR) launch_pdl(k_interp<PL, TR>, blocks, kWalkThreads, 0, st, p, spos, nval, off, pts, n, out)
    if (p.planar) {
        if (p.trim) CMAG_INTERP(true, true);
        else CMAG_INTERP(true, false);
    } else {
        if (p.trim) CMAG_INTERP(false, true);
        else CMAG_INTERP(false, false);
    }
#undef CMAG_INTERP
}

void launch_closure_backward(const ClosureView &c, const float *feat, const float *target,
                             uint32_t n, float *grad, float *loss, cudaStream_t st)
{
    if (n == 0) return;
    allow_smem(k_backward, kSmemBackward);
    const uint32_t tiles = (n + kTile - 1) / kTile, most = 2u * (uint32_t)device_sm_count();  // 2 blocks an SM
    k_backward<<<tiles < most ? tiles : most, kBackThreads, kSmemBackward, st>>>(c, feat, target, n, grad, loss);
}

void launch_closure_fold(float *grad, cudaStream_t st)
{
    k_fold_gradient<<<(kClosureParams + 255) / 256, 256, 0, st>>>(grad);
}

uint32_t closure_image_words() { return (uint32_t)kImageWords; }

void launch_closure_adam(float *master, float *m, float *v, float *grad, __nv_bfloat16 *w,
                         uint4 *image, float lr, float beta1, float beta2, float eps, float bias1,
                         float bias2, cudaStream_t st)
{
    k_adam<<<(kClosureParams + 255) / 256, 256, 0, st>>>(master, m, v, grad, w, reinterpret_cast<uint32_t *>(image),
                                                        lr, beta1, beta2, eps, bias1, bias2);
}

void launch_closure_round(const float *master, __nv_bfloat16 *w, uint4 *image, cudaStream_t st)
{
    k_round<<<(kClosureParams + 255) / 256, 256, 0, st>>>(master, w);
    k_pack<<<(kImageBytes / 4 + 255) / 256, 256, 0, st>>>(w, reinterpret_cast<uint32_t *>(image));
}

}  // namespace cmag
