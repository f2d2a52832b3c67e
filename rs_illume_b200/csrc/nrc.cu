// Neural radiance cache: input encoding, a 5 x 64 ReLU MLP on the BF16
// tensor cores (tcgen05.mma, FP32 accumulators in TMEM), relative-L2 loss
// and Adam.
// No counterpart in the reference (a learned component added on top of the
// path tracer); the method follows published neural radiance caching:
//   inputs: position (12-frequency sin/cos per axis, 72), outgoing direction
//   and normal (one-blob, 32 bins on each of theta/pi and phi/2pi, 128),
//   albedo (3) = 203, padded to 208;
//   layers 208->64, 4 x (64->64), 64->16 (first 3 outputs = RGB radiance),
//   ReLU between, no biases;
//   loss = mean over samples and channels of (p - y)^2 / (sg(p)^2 + 0.01).
//
// Kernels
//   k_mlp_infer_tc inference: per 128-row tile a warpgroup encodes its rows
//                  into TMEM as layer 0's A operand, one thread issues the
//                  MMAs, each layer's accumulator becomes the next A
//   k_mlp_train_tc training: the same forward, then the loss gradient and the
//                  way back through the layers (transposed weights); stores
//                  the encoding, the bf16 activations and dOut
//   k_wgrad_tc     dW_l = dOut_l^T * in_l for all six layers on tcgen05
//                  (M = outputs, N = inputs, K = batch rows, both operands
//                  MN-major as the rows are stored, staged by bulk copies);
//                  split-K over the rows, one FP32 partial per chunk, no atomics
//   k_reduce_adam  sums the CTA partials, Adam on the FP32 master weights,
//                  bf16 weight packs and the inference moving average
//   k_nrc_encode   the encoding alone (for inspection)
// Row counts may live in device memory (NrcCount), so the path tracer enqueues
// inference and training without reading its queue sizes on the host.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <vector>

#include "context.h"
#include "illume_gpu.h"
#include "nrc.h"
#include "pcg32.h"

namespace ilm {
namespace nrc {

constexpr int kIn = 208, kInReal = 203, kHid = 64, kOut = 16, kLayers = 6;
__host__ __device__ constexpr int in_dim(int l) { return l == 0 ? kIn : kHid; }
__host__ __device__ constexpr int out_dim(int l) { return l == 5 ? kOut : kHid; }
// FP32 parameter offsets, row-major [out][in]
__host__ __device__ constexpr int param_off(int l) {
    return l == 0 ? 0 : kHid * kIn + (l - 1) * kHid * kHid;
}
constexpr int kParams = kHid * kIn + 4 * kHid * kHid + kOut * kHid;   // 30720
// bf16 inference pack in the tensor cores' canonical K-major layout without
// swizzle: layer l's [out][in] matrix as 8x8 core matrices of 128 contiguous
// bytes, core matrix (o/8, i/8) at (o/8 * in/8 + i/8) * 64 elements from the
// layer's start (param_off(l)), row o%8 at 8 elements, column i%8.
__host__ __device__ constexpr int tc_index(int l, int o, int i) {
    return param_off(l) + ((o >> 3) * (in_dim(l) >> 3) + (i >> 3)) * 64 + (o & 7) * 8 + (i & 7);
}
// Transposed bf16 pack for the backward pass, the same canonical layout:
// layer l >= 1 as W_l^T ([in][out], N = in, K = out), core matrix (i/8, o/8)
// at (i/8 * out/8 + o/8) * 64 elements from tcb_off(l).
__host__ __device__ constexpr int tcb_off(int l) { return (l - 1) * kHid * kHid; }   // l = 1..5
__host__ __device__ constexpr int tcb_index(int l, int o, int i) {
    return tcb_off(l) + ((i >> 3) * (out_dim(l) >> 3) + (o >> 3)) * 64 + (i & 7) * 8 + (o & 7);
}
constexpr int kTcbElems = 4 * kHid * kHid + kHid * kOut;   // 17408
constexpr float kLossEps = 0.01f;

struct Enc {   // position normalisation: q = (p - origin) * scale
    float x0, y0, z0, sx, sy, sz;
};

struct AdamArgs {
    float lr, b1, b2, eps;
    float ema_a;   // moving-average decay (0 = off)
    float wd;      // decoupled weight decay (AdamW; 0 = none)
};

// Optimiser counters in device memory, so that a captured training step
// replays with the right bias corrections.
struct StepState {
    int step;        // Adam steps taken
    int ema_steps;   // Adam steps since the inference weights restarted
};

__device__ __forceinline__ uint32_t rows_of(const NrcCount& c) {
    uint32_t n = c.cap;
    if (c.dev) {
        unsigned long long d = *c.dev;
        n = d < (unsigned long long)c.cap ? (uint32_t)d : c.cap;
    }
    if (c.batches > 1) n = n > c.batch ? (n - c.batch + c.batches - 1) / c.batches : 0u;
    return n;
}

__device__ __forceinline__ uint32_t pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// ---------------------------------------------------------------- encoding
// What the encoder needs of one input row.
struct RowIn {
    float q[3];     // normalised position
    float u[4];     // theta/pi, phi/2pi of the direction, then of the normal
    float alb[3];
    float ps[3], pc[3];   // encoding state: the last octave's (sin, cos) per axis
};

// theta / pi of a unit vector's z, phi / 2 pi of its x and y.
__device__ __forceinline__ float row_theta(float z) {
    return acosf(fminf(fmaxf(z, -1.0f), 1.0f)) * (1.0f / 3.14159265358979f);
}
__device__ __forceinline__ float row_phi(float x, float y) {
    return atan2f(y, x) * (0.5f / 3.14159265358979f) + 0.5f;
}

__device__ __forceinline__ RowIn load_row(const float* __restrict__ raw, uint32_t r, const Enc& e) {
    const float* p = raw + 12 * (size_t)r;
    RowIn v;
    v.q[0] = (p[0] - e.x0) * e.sx;
    v.q[1] = (p[1] - e.y0) * e.sy;
    v.q[2] = (p[2] - e.z0) * e.sz;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        v.u[2 * k] = row_theta(p[5 + 3 * k]);
        v.u[2 * k + 1] = row_phi(p[3 + 3 * k], p[4 + 3 * k]);
    }
    v.alb[0] = p[9];
    v.alb[1] = p[10];
    v.alb[2] = p[11];
    return v;
}

// The eight features 8 KC .. 8 KC + 7 of a row as four bf16 pairs (pair t =
// features 8 KC + 2t, 8 KC + 2t + 1).  The layout:
//   [0, 72)    axis f / 24, octave k = (f % 24) / 2: (sin, cos)(2^k pi q)
//   [72, 200)  one-blob of u[(f - 72) / 32], bin j = (f - 72) % 32:
//              exp(-((u - (j + 1/2)/32) * 32)^2 / 2)
//   200..202   albedo, then zeros
// Groups are evaluated in order (KC = 0, 1, ... 25), and two recurrences cut
// the special-function work:
//   * octaves: one sincospi per axis at octave 0, then the double angle,
//     sin 2x = 2 sin x cos x, cos 2x = (cos x - sin x)(cos x + sin x); the
//     error doubles per octave, about 2^11 float ulps at octave 11, far below
//     a bf16 ulp; the last octave of a group is kept in the row state;
//   * one-blob bins: two exps per group of 8 bins, g_j = exp(-d_j^2 / 2) and
//     the ratio r_j = g_{j+1} / g_j = exp(d_j - 1/2) (d_{j+1} = d_j - 1), then
//     g_{j+1} = g_j r_j and r_{j+1} = r_j / e; relative error grows by a few
//     ulps per step.
template <int KC>
__device__ __forceinline__ uint4 feature_group(RowIn& v) {
    constexpr int F = 8 * KC;
    uint4 q;
    if constexpr (F < 72) {
        constexpr int a = F / 24, o0 = (F % 24) >> 1;
        float s, c;
        if constexpr (o0 == 0) {
            sincospif(v.q[a], &s, &c);
        } else {
            s = 2.0f * v.ps[a] * v.pc[a];
            c = (v.pc[a] - v.ps[a]) * (v.pc[a] + v.ps[a]);
        }
        uint32_t w[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            w[t] = pack(s, c);
            if (t < 3) {
                const float s2 = 2.0f * s * c, c2 = (c - s) * (c + s);
                s = s2;
                c = c2;
            }
        }
        v.ps[a] = s;
        v.pc[a] = c;
        q = make_uint4(w[0], w[1], w[2], w[3]);
    } else if constexpr (F < 200) {
        constexpr int ui = (F - 72) >> 5, j0 = (F - 72) & 31;
        constexpr float kInvE = 0.36787944117144233f;   // e^-1
        const float d = (v.u[ui] - (j0 + 0.5f) * (1.0f / 32.0f)) * 32.0f;
        float g = __expf(-0.5f * d * d), r = __expf(d - 0.5f);
        float gv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            gv[k] = g;
            g *= r;
            r *= kInvE;
        }
        q = make_uint4(pack(gv[0], gv[1]), pack(gv[2], gv[3]), pack(gv[4], gv[5]), pack(gv[6], gv[7]));
    } else {
        q = make_uint4(pack(v.alb[0], v.alb[1]), pack(v.alb[2], 0.0f), 0u, 0u);
    }
    return q;
}

// Whole-row encoder (104 words) for k_nrc_encode.
template <int B>
__device__ __forceinline__ void encode_row(RowIn& v, uint32_t* out) {
    const uint4 q = feature_group<B>(v);
    out[4 * B] = q.x;
    out[4 * B + 1] = q.y;
    out[4 * B + 2] = q.z;
    out[4 * B + 3] = q.w;
    if constexpr (B + 1 < kIn / 8) encode_row<B + 1>(v, out);
}

__global__ void k_nrc_encode(const float* __restrict__ raw, uint32_t n, Enc ec, __nv_bfloat16* __restrict__ enc) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    RowIn v = load_row(raw, i, ec);
    encode_row<0>(v, reinterpret_cast<uint32_t*>(enc + (size_t)i * kIn));
}

// ---------------------------------------------------------------- tcgen05
// The network's layers are D = A * W^T on the 5th-generation tensor cores: A
// 128 rows of bf16 operands in TMEM, W in shared memory, FP32 D in TMEM.  The
// weight packs use the canonical K-major layout without swizzle: 8x8 core
// matrices of 128 contiguous bytes; LBO = 128 bytes (next core matrix along
// K), SBO = the stride between 8-row groups.  Every mbarrier wait is bounded;
// a timeout sets kErrMlpTimeout in *err.  Waits that gave up are followed by
// a drain, up to kTcDrainCap more polls on the last commit's phase, so that
// tcgen05.dealloc does not free columns an MMA may still write.  If the drain
// runs out too, the columns are freed all the same -- a CTA that kept them
// would leave the tcgen05.alloc of later CTAs on its SM waiting -- and the
// error word marks the launch's results as invalid.
constexpr int kTcWBytes = kParams * 2;                         // 61,440: all layers' forward weights
constexpr int kTcbWBytes = kTcbElems * 2;                      // 34,816: the transposed ones, layers 1-5
constexpr uint32_t kErrMlpTimeout = 4u;
constexpr uint32_t kTcWaitCap = 1u << 22;   // try_wait polls before a wait gives up
constexpr uint32_t kTcDrainCap = 1u << 26;  // further polls for a batch whose wait gave up

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor: start, LBO, SBO (bytes), version 1, no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor, kind::f16: D f32, A and B bf16, both K-major.
__host__ __device__ constexpr uint32_t idesc_bf16(int m, int n) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}
__device__ __forceinline__ void umma(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
        :
        : "r"(tmem_d), "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}
__device__ __forceinline__ void umma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(uint32_t mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}
// Contiguous bytes from global to shared memory (16-byte aligned, a multiple
// of 16), counted on an mbarrier.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t mbar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(mbar)
                 : "memory");
}

// ---------------------------------------------------------------- inference on tcgen05
// k_mlp_infer_tc: the inference forward.  What it spends its time on is the
// threads' work on the MMAs' A operands (encoding, accumulator -> bf16 ->
// ReLU), so everything else is kept off that path:
//  * A lives in TMEM (tcgen05.st; 32 columns hold a row's 64 bf16 features).
//    From shared memory an MMA of N = 64 took about 100 cycles to issue, its
//    A tile being four fifths of what it fetches; eight tiles in flight waited
//    700 cycles and more for each batch of four.
//  * Up to five 128-row tiles are in flight per SM, one per warpgroup, each
//    with 64 accumulator and 32 operand columns (480 of the 512); thread t of
//    a warpgroup owns row t.
//  * No barriers: the last of a tile's four warps to finish its share of an
//    operand (an acquire-release counter in shared memory) issues the batch
//    and commits it to the tile's mbarrier, and each warp waits there by itself.
// Layer 0 is issued in four parts of K = 64, 64, 64 and 16 features, so a tile
// takes nine MMA batches.  727,329 rows: 136.5 us with two tiles per
// warpgroup from shared memory and two barriers a batch, 77.8 us now (553 TFLOP/s,
// 0.34 of the measured bf16 peak).
// Waits are bounded; a warp whose wait gave up sets `fail`, which ends the
// others' waits, and every tile's last commit is drained before the TMEM is
// freed.
constexpr int kInfGroups = 5;                   // warpgroups per CTA, at most
constexpr uint32_t kInfCols = 96;               // TMEM columns per warpgroup: 64 accumulator, 32 operand

// Row r's 12 inputs; by 16-byte loads where the array allows.
__device__ __forceinline__ void load_raw(const float* __restrict__ raw, uint32_t r, bool vec, float (&p)[12]) {
    const float* src = raw + 12 * (size_t)r;
    if (vec) {
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(src) + k);
            p[4 * k] = v.x; p[4 * k + 1] = v.y; p[4 * k + 2] = v.z; p[4 * k + 3] = v.w;
        }
    } else {
#pragma unroll
        for (int k = 0; k < 12; ++k) p[k] = __ldg(src + k);
    }
}

// Octaves O0 .. O0 + 3 of an axis as four bf16 pairs, from octave O0 - 1 in
// (s, c) (octave 0: from q); (s, c) becomes the last one.  The doubling is
// feature_group's, each operation rounded by itself, except that c - s and
// c + s of octave kFuse round once with the product that s is (kFuse < 0:
// none).  Which octaves those are is the rounding that this kernel has had since
// it worked on tiles in pairs, and it differs between even and odd tiles: about
// one row in 7,000 gets answers a bf16 rounding apart in the two (4e-5 to 6e-5
// of the answers' norm in all).  It is kept because one rule for all tiles, which
// is no nearer to 64 bits (0.0072 either way), changes answers by as much
// (4.5e-5).  The training kernel and k_nrc_encode round every row by
// feature_group.
template <int O0, int kFuse>
__device__ __forceinline__ void octaves(float q, float& s, float& c, uint32_t (&w)[4]) {
    float s1 = s, c1 = c;   // the octave before (s, c)
    if constexpr (O0 == 0) {
        sincospif(q, &s, &c);
    } else {
        const float s2 = __fmul_rn(__fmul_rn(2.0f, s), c), c2 = __fmul_rn(__fsub_rn(c, s), __fadd_rn(c, s));
        s = s2;
        c = c2;
    }
#pragma unroll
    for (int t = 0; t < 4; ++t) {
        w[t] = pack(s, c);
        if (t == 3) break;
        const float s2 = __fmul_rn(__fmul_rn(2.0f, s), c);
        float lo, hi;
        if (O0 + t == kFuse) {
            lo = __fmaf_rn(__fmul_rn(-2.0f, s1), c1, c);
            hi = __fmaf_rn(__fmul_rn(2.0f, s1), c1, c);
        } else {
            lo = __fsub_rn(c, s);
            hi = __fadd_rn(c, s);
        }
        s1 = s;
        c1 = c;
        s = s2;
        c = __fmul_rn(lo, hi);
    }
}

__device__ __forceinline__ void tmem_st4(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c),
                 "r"(d)
                 : "memory");
}

// Feature group KC >= 9 of a row into its operand columns.
template <int KC>
__device__ __forceinline__ void put_group(uint32_t tmem_a, RowIn& v) {
    const uint4 q = feature_group<KC>(v);
    tmem_st4(tmem_a + 4 * (KC & 7), q.x, q.y, q.z, q.w);
}
template <int KC, int KEND>
__device__ __forceinline__ void put_groups(uint32_t tmem_a, RowIn& v) {
    put_group<KC>(tmem_a, v);
    if constexpr (KC + 1 < KEND) put_groups<KC + 1, KEND>(tmem_a, v);
}

// Part 0 of layer 0 (groups 0-7): axes 0 and 1 and the first 8 octaves of axis
// 2, whose last one stays in the row state.
template <bool kOdd>
__device__ __forceinline__ void put_positions(uint32_t tmem_a, RowIn& v) {
    uint32_t w[4];
    float s = 0.0f, c = 0.0f;
    octaves<0, -1>(v.q[0], s, c, w);
    tmem_st4(tmem_a, w[0], w[1], w[2], w[3]);
    octaves<4, -1>(0.0f, s, c, w);
    tmem_st4(tmem_a + 4, w[0], w[1], w[2], w[3]);
    octaves<8, kOdd ? 9 : -1>(0.0f, s, c, w);
    tmem_st4(tmem_a + 8, w[0], w[1], w[2], w[3]);
    octaves<0, -1>(v.q[1], s, c, w);
    tmem_st4(tmem_a + 12, w[0], w[1], w[2], w[3]);
    octaves<4, -1>(0.0f, s, c, w);
    tmem_st4(tmem_a + 16, w[0], w[1], w[2], w[3]);
    octaves<8, kOdd ? 9 : 8>(0.0f, s, c, w);
    tmem_st4(tmem_a + 20, w[0], w[1], w[2], w[3]);
    octaves<0, -1>(v.q[2], s, c, w);
    tmem_st4(tmem_a + 24, w[0], w[1], w[2], w[3]);
    octaves<4, -1>(0.0f, s, c, w);
    tmem_st4(tmem_a + 28, w[0], w[1], w[2], w[3]);
    v.ps[2] = s;
    v.pc[2] = c;
}

// A row's share of layer-0 part `part` (groups 8 part .. 8 part + 7, at most 25).
__device__ __forceinline__ void encode_part(int part, bool odd, uint32_t tmem_a, const float* __restrict__ raw,
                                            uint32_t r, bool in_range, bool vec, const Enc& e, RowIn& v) {
    if (part == 0) {
        v = RowIn{};
        if (in_range) {
            float p[12];
            load_raw(raw, r, vec, p);
            v.q[0] = (p[0] - e.x0) * e.sx;
            v.q[1] = (p[1] - e.y0) * e.sy;
            v.q[2] = (p[2] - e.z0) * e.sz;
#pragma unroll
            for (int k = 0; k < 2; ++k) {
                v.u[2 * k] = row_theta(p[5 + 3 * k]);
                v.u[2 * k + 1] = row_phi(p[3 + 3 * k], p[4 + 3 * k]);
            }
            v.alb[0] = p[9];
            v.alb[1] = p[10];
            v.alb[2] = p[11];
        }
        if (odd) put_positions<true>(tmem_a, v);
        else put_positions<false>(tmem_a, v);
    } else if (part == 1) {
        uint32_t w[4];
        octaves<8, -1>(0.0f, v.ps[2], v.pc[2], w);
        tmem_st4(tmem_a, w[0], w[1], w[2], w[3]);
        put_groups<9, 16>(tmem_a, v);
    } else if (part == 2) {
        put_groups<16, 24>(tmem_a, v);
    } else {
        put_groups<24, 26>(tmem_a, v);
    }
}

// Accumulator row (64 columns) -> bf16 -> ReLU -> its operand columns.
// Rounding is monotone, so the packed maximum with zero gives what the ReLU
// before it gives, in half the instructions.
__device__ __forceinline__ void acc_to_operand(uint32_t tmem_d, uint32_t tmem_a) {
    const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t r[32];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,"
            "%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(tmem_d + 32u * h));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        uint32_t w[16];
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const __nv_bfloat162 b =
                __hmax2(__floats2bfloat162_rn(__uint_as_float(r[2 * k]), __uint_as_float(r[2 * k + 1])), zero);
            w[k] = *reinterpret_cast<const uint32_t*>(&b);
        }
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
                tmem_a + 16u * h),
            "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
            "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
            : "memory");
    }
}

// One MMA with A in TMEM; B's descriptor by its low word (start address, LBO)
// and high word (SBO, version).
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint32_t b_lo, uint32_t b_hi, uint32_t idesc,
                                        uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\tmov.b64 db, {%2, %3};\n\tsetp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %4, p;\n\t}\n"
        :
        : "r"(tmem_d), "r"(tmem_a), "r"(b_lo), "r"(b_hi), "r"(idesc), "r"(acc)
        : "memory");
}

// Issues batch k (0-3: the parts of layer 0, 4-8: layers 1-5) of a tile and
// commits it to the tile's mbarrier; called by a whole warp, whose lane 0
// issues.  A K-step is 8 operand columns and 256 bytes of weights.
__device__ __forceinline__ void inf_issue(int k, uint32_t tmem_d, uint32_t tmem_a, uint32_t w_base, uint32_t mbar,
                                          uint32_t lane) {
    constexpr uint32_t kLbo = (128u >> 4) << 16;
    constexpr uint32_t kHi8 = (8u * 128u >> 4) | (1u << 14), kHi26 = (26u * 128u >> 4) | (1u << 14);
    const int l = k < 4 ? 0 : k - 3;
    const uint32_t w_at = w_base + 2u * (l == 0 ? 0u : (uint32_t)(kHid * kIn + (l - 1) * kHid * kHid)) +
                          (k < 4 ? (uint32_t)k * 1024u : 0u);
    const uint32_t b_lo = (w_at >> 4) | kLbo, b_hi = l == 0 ? kHi26 : kHi8;
    const uint32_t idesc = k == 8 ? idesc_bf16(128, 16) : idesc_bf16(128, 64);
    tc_fence_after();
    if (lane == 0) {
        umma_ts(tmem_d, tmem_a, b_lo, b_hi, idesc, k > 0 && k < 4 ? 1u : 0u);
        if (k != 3) {
            umma_ts(tmem_d, tmem_a + 8u, b_lo + 16u, b_hi, idesc, 1u);
            umma_ts(tmem_d, tmem_a + 16u, b_lo + 32u, b_hi, idesc, 1u);
            umma_ts(tmem_d, tmem_a + 24u, b_lo + 48u, b_hi, idesc, 1u);
        }
        umma_commit(mbar);
    }
}

// A warp's bounded wait for a phase; false (for the whole warp) when it or
// another warp gave up.
__device__ __forceinline__ bool warp_wait(uint32_t mbar, uint32_t parity, volatile int* fail) {
    bool ok = true;
    uint32_t it = 0;
    while (!mbar_try_wait(mbar, parity)) {
        if (++it >= kTcWaitCap || *fail) {
            *fail = 1;
            ok = false;
            break;
        }
    }
    ok = __all_sync(0xFFFFFFFFu, ok);
    tc_fence_after();
    return ok;
}

__global__ void __launch_bounds__(128 * kInfGroups, 1) k_mlp_infer_tc(const float* __restrict__ raw, NrcCount cnt, Enc ec,
                                                                      const __nv_bfloat16* __restrict__ wtc,
                                                                      float* __restrict__ out, uint32_t* err,
                                                                      uint32_t tmem_cols) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    __shared__ __align__(8) uint64_t mbar[kInfGroups];   // a warpgroup's last batch is done
    __shared__ __align__(8) uint64_t wbar;               // the weights are here
    __shared__ uint32_t arrived[kInfGroups];             // warps that finished their share, ever
    __shared__ uint32_t issued[kInfGroups];              // batches issued, ever
    __shared__ int fail;
    __shared__ uint32_t tmem_base;
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);   // uniform, and known to be
    const int g = warp >> 2;
    const uint32_t lane = threadIdx.x & 31u, t = threadIdx.x & 127u;
    const uint32_t groups = blockDim.x >> 7;
    if (threadIdx.x < groups) {
        mbar_init(smem_u32(&mbar[threadIdx.x]));
        arrived[threadIdx.x] = 0;
        issued[threadIdx.x] = 0;
    }
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&wbar));
        fail = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(tmem_cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) {   // the weights, while the first tiles are encoded
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&wbar)), "r"(kTcWBytes)
                     : "memory");
        bulk_load(smem_u32(tc_smem), wtc, kTcWBytes, smem_u32(&wbar));
    }
    const uint32_t n = rows_of(cnt);
    const bool vec = ((uintptr_t)raw & 15u) == 0;
    const uint32_t tmem_d = tmem_base + kInfCols * g, tmem_a = tmem_d + 64u;   // the MMAs' addresses
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;                  // this warp's rows of them
    const uint32_t mb = smem_u32(&mbar[g]);
    const uint32_t tiles = (n + 127) / 128;
    uint32_t parity = 0;
    bool ok = true, weights_here = false;
    for (uint32_t tile = blockIdx.x * groups + g; tile < tiles && ok; tile += gridDim.x * groups) {
        const uint32_t r = tile * 128u + t;
        RowIn v;
        for (int k = 0; k < 9; ++k) {
            if (k > 0) {
                ok = warp_wait(mb, parity, &fail);
                parity ^= 1u;
                if (!ok) break;
            }
            if (k < 4) encode_part(k, (tile & 1u) != 0, tmem_a + lanes, raw, r, r < n, vec, ec, v);
            else acc_to_operand(tmem_d + lanes, tmem_a + lanes);
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();     // accumulator reads and operand writes, ordered before the MMAs
            __syncwarp();
            uint32_t before = 0;
            if (lane == 0)
                asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                             : "=r"(before)
                             : "r"(smem_u32(&arrived[g]))
                             : "memory");
            before = __shfl_sync(0xFFFFFFFFu, before, 0);
            if ((before & 3u) == 3u) {   // the operand is complete
                if (!weights_here) {
                    uint32_t it = 0;
                    while (!mbar_try_wait(smem_u32(&wbar), 0u) && ++it < kTcWaitCap) {}
                    if (it >= kTcWaitCap) fail = 1;
                    weights_here = true;
                }
                if (lane == 0) issued[g] += 1;
                inf_issue(k, tmem_d, tmem_a, smem_u32(tc_smem), mb, lane);
            }
            __syncwarp();
        }
        if (!ok) break;
        ok = warp_wait(mb, parity, &fail);
        parity ^= 1u;
        if (!ok) break;
        float o[16];
        tmem_ld16(tmem_d + lanes, o);
        tc_fence_before();   // the next tile's batches overwrite the columns
        if (r < n) {
            out[3 * (size_t)r] = o[0];
            out[3 * (size_t)r + 1] = o[1];
            out[3 * (size_t)r + 2] = o[2];
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) {
        tc_fence_after();
        // the weights' copy and every warpgroup's last batch, before shared
        // memory and TMEM are given back
        uint32_t it = 0;
        while (!mbar_try_wait(smem_u32(&wbar), 0u) && ++it < kTcDrainCap) {}
        if (fail) {
            for (uint32_t q = 0; q < groups; ++q) {
                if (issued[q] == 0) continue;
                it = 0;
                while (!mbar_try_wait(smem_u32(&mbar[q]), (issued[q] - 1u) & 1u) && ++it < kTcDrainCap) {}
            }
            atomicOr(err, kErrMlpTimeout);
        }
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(tmem_cols));
    }
}

// ---------------------------------------------------------------- training forward and backward on tcgen05
// k_mlp_train_tc: encoding, forward, loss gradient (mean over the n rows and 3
// channels) and the way back through the layers, one 128-row tile at a time
// per CTA of 256 threads, two CTAs per SM.  A training batch is a tile or two
// per SM, so the kernel is one chain of 14 MMA batches and bound by its
// latency: two threads share a row (warps w and w + 4 reach the same TMEM
// lanes; the first half's warps write some columns of each operand, the second
// half's the others), operands go straight to TMEM, the last of the eight
// warps to finish its share issues the batch, both weight packs arrive by bulk
// copies while the first rows are encoded, and each row's ReLU masks stay in
// its threads' registers on the way back.  32,768 rows: 45 us as a
// forward and a backward kernel with A in shared memory, 20 us now.
// The weight gradients need the encoding ([n][208]), the five activations and
// the six dOuts ([n][64], layer 5 [n][16]); they are stored in blocks of 8
// rows x 8 features (128 bytes), which is how k_wgrad_tc's operands lie in
// shared memory: feature block c of rows 8 b .. 8 b + 7 at block b * (features
// / 8) + c.  Rows n .. up to the tile's end are stored too, with dOut = 0.
constexpr int kTrThreads = 256, kTrWarps = kTrThreads / 32;
constexpr int kTrSmem = kTcWBytes + kTcbWBytes;                // 96,256
constexpr int kTrGrid = 296;                                   // CTAs, at most
constexpr uint32_t kTrCols = 128;                              // TMEM columns: 64 accumulator, 32 operand

// What a thread keeps of its row between the parts of layer 0: the first half
// the direction's and the normal's theta and the albedo, the second half
// their phi and the last octave of axis 2.
struct HalfRow {
    float u0, u1, c0, c1, c2;
};

// Feature group KC of a row into its operand columns and its stored encoding.
template <int KC>
__device__ __forceinline__ void train_group(uint32_t tmem_a, uint4* genc, RowIn& v) {
    const uint4 q = feature_group<KC>(v);
    tmem_st4(tmem_a + 4 * (KC & 7), q.x, q.y, q.z, q.w);
    genc[8 * KC] = q;
}

// A thread's share of layer-0 part `part` (groups 8 part .. 8 part + 7, at
// most 25): axis 0 and the first octaves of axis 2 against axis 1 and the
// rest of axis 2; the thetas' groups (9-12, 17-20) and the albedo against the
// phis' (13-16, 21-24).
__device__ __forceinline__ void encode_share(int part, int half, uint32_t tmem_a, uint4* genc,
                                             const float* __restrict__ raw, uint32_t r, bool in_range, bool vec,
                                             const Enc& e, HalfRow& k) {
    RowIn v = {};
    if (part == 0) {
        float p[12] = {};
        if (in_range) load_raw(raw, r, vec, p);
        if (half == 0) {
            k.u0 = row_theta(p[5]);
            k.u1 = row_theta(p[8]);
            k.c0 = p[9]; k.c1 = p[10]; k.c2 = p[11];
            if (in_range) {
                v.q[0] = (p[0] - e.x0) * e.sx;
                v.q[2] = (p[2] - e.z0) * e.sz;
            }
            train_group<0>(tmem_a, genc, v);
            train_group<1>(tmem_a, genc, v);
            train_group<2>(tmem_a, genc, v);
            train_group<6>(tmem_a, genc, v);
        } else {
            k.u0 = row_phi(p[3], p[4]);
            k.u1 = row_phi(p[6], p[7]);
            if (in_range) {
                v.q[1] = (p[1] - e.y0) * e.sy;
                v.q[2] = (p[2] - e.z0) * e.sz;
            }
            train_group<3>(tmem_a, genc, v);
            train_group<4>(tmem_a, genc, v);
            train_group<5>(tmem_a, genc, v);
            feature_group<6>(v);        // octaves 0-3 of axis 2, for the chain
            train_group<7>(tmem_a, genc, v);
            k.c0 = v.ps[2];
            k.c1 = v.pc[2];
        }
    } else if (half == 0) {
        v.u[0] = k.u0;
        v.u[2] = k.u1;
        v.alb[0] = k.c0; v.alb[1] = k.c1; v.alb[2] = k.c2;
        if (part == 1) {
            train_group<9>(tmem_a, genc, v);
            train_group<10>(tmem_a, genc, v);
            train_group<11>(tmem_a, genc, v);
            train_group<12>(tmem_a, genc, v);
        } else if (part == 2) {
            train_group<17>(tmem_a, genc, v);
            train_group<18>(tmem_a, genc, v);
            train_group<19>(tmem_a, genc, v);
            train_group<20>(tmem_a, genc, v);
        } else {
            train_group<25>(tmem_a, genc, v);
        }
    } else {
        v.u[1] = k.u0;
        v.u[3] = k.u1;
        if (part == 1) {
            v.ps[2] = k.c0;
            v.pc[2] = k.c1;
            train_group<8>(tmem_a, genc, v);
            train_group<13>(tmem_a, genc, v);
            train_group<14>(tmem_a, genc, v);
            train_group<15>(tmem_a, genc, v);
        } else if (part == 2) {
            train_group<16>(tmem_a, genc, v);
            train_group<21>(tmem_a, genc, v);
            train_group<22>(tmem_a, genc, v);
            train_group<23>(tmem_a, genc, v);
        } else {
            train_group<24>(tmem_a, genc, v);
        }
    }
}

// 32 accumulator columns of a row.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
        "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]);
}

// Half a row's operand (32 features, 16 words): into its TMEM columns and, as
// four 16-byte feature blocks, into memory.
__device__ __forceinline__ void put_half(const uint32_t (&w)[16], uint32_t tmem_a, uint4* dst, bool operand) {
    if (operand)
        asm volatile(
            "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(
                tmem_a),
            "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
            "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
            : "memory");
#pragma unroll
    for (int c = 0; c < 4; ++c) dst[8 * c] = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
}

// Issues batch k of a tile: 0-8 the forward's (inf_issue), 9 dAct4 = dOut5 *
// W5 (K = 16), 9 + i the same of layer 5 - i; then commits it.
__device__ __forceinline__ void train_issue(int k, uint32_t tmem_d, uint32_t tmem_a, uint32_t w_base, uint32_t wb_base,
                                            uint32_t mbar, uint32_t lane) {
    if (k < 9) {
        inf_issue(k, tmem_d, tmem_a, w_base, mbar, lane);
        return;
    }
    constexpr uint32_t kLbo = (128u >> 4) << 16;
    constexpr uint32_t kHi2 = (2u * 128u >> 4) | (1u << 14), kHi8 = (8u * 128u >> 4) | (1u << 14);
    const int l = 14 - k;
    const uint32_t b_lo = ((wb_base + 2u * (uint32_t)tcb_off(l)) >> 4) | kLbo;
    constexpr uint32_t idesc = idesc_bf16(128, 64);
    tc_fence_after();
    if (lane == 0) {
        if (l == 5) {
            umma_ts(tmem_d, tmem_a, b_lo, kHi2, idesc, 0u);
        } else {
            umma_ts(tmem_d, tmem_a, b_lo, kHi8, idesc, 0u);
            umma_ts(tmem_d, tmem_a + 8u, b_lo + 16u, kHi8, idesc, 1u);
            umma_ts(tmem_d, tmem_a + 16u, b_lo + 32u, kHi8, idesc, 1u);
            umma_ts(tmem_d, tmem_a + 24u, b_lo + 48u, kHi8, idesc, 1u);
        }
        umma_commit(mbar);
    }
}

__global__ void __launch_bounds__(kTrThreads, 2) k_mlp_train_tc(const float* __restrict__ raw,
                                                                const float* __restrict__ target, NrcCount cnt, Enc ec,
                                                                const __nv_bfloat16* __restrict__ wtc,
                                                                const __nv_bfloat16* __restrict__ wtcb, uint32_t ld,
                                                                __nv_bfloat16* __restrict__ enc,
                                                                __nv_bfloat16* __restrict__ acts,
                                                                __nv_bfloat16* __restrict__ douts,
                                                                float* __restrict__ loss_part, uint32_t* err) {
    extern __shared__ __align__(1024) uint8_t tc_smem[];
    __shared__ __align__(8) uint64_t mbar, wbar;   // the last batch is done; the weights are here
    __shared__ uint32_t arrived, issued, tmem_base;
    __shared__ int fail;
    __shared__ float warp_loss[kTrWarps];
    const int warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0);   // uniform, and known to be
    const int half = warp >> 2;
    const uint32_t lane = threadIdx.x & 31u, t = 32u * (warp & 3) + lane;    // t: row of the tile
    if (threadIdx.x == 0) {
        mbar_init(smem_u32(&mbar));
        mbar_init(smem_u32(&wbar));
        arrived = issued = 0;
        fail = 0;
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(kTrCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&wbar)), "r"(kTrSmem)
                     : "memory");
        bulk_load(smem_u32(tc_smem), wtc, kTcWBytes, smem_u32(&wbar));
        bulk_load(smem_u32(tc_smem + kTcWBytes), wtcb, kTcbWBytes, smem_u32(&wbar));
    }
    const uint32_t n = rows_of(cnt);
    const float scale = n > 0 ? 1.0f / (3.0f * (float)n) : 0.0f;
    const bool vec = ((uintptr_t)raw & 15u) == 0;
    const uint32_t tmem_d = tmem_base, tmem_a = tmem_base + 64u;
    const uint32_t lanes = (uint32_t)(32 * (warp & 3)) << 16;   // this warp's rows of them
    const uint32_t mb = smem_u32(&mbar), w_base = smem_u32(tc_smem);
    const uint32_t tiles = (n + 127) / 128;
    uint32_t parity = 0;
    bool ok = true, weights_here = false;
    float loss = 0.0f;
    for (uint32_t tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x) {
        const uint32_t r = tile * 128u + t;
        const bool in_range = r < n;
        // 16-byte block of feature group 0 of this row, in arrays of F groups
        auto block = [&](__nv_bfloat16* base, uint32_t F) {
            return reinterpret_cast<uint4*>(base) + (size_t)(r >> 3) * F * 8u + (r & 7u);
        };
        HalfRow keep;
        uint32_t mask[5];   // bit k: the low half of word k of this thread's activations is positive; k + 16: the high
        for (int k = 0; k <= 14; ++k) {
            if (k > 0) {
                ok = warp_wait(mb, parity, &fail);
                parity ^= 1u;
                if (!ok) break;
            }
            if (k < 4) {
                encode_share(k, half, tmem_a + lanes, block(enc, kIn / 8), raw, r, in_range, vec, ec, keep);
            } else if (k < 9) {
                // layer k - 4's activation: accumulator -> bf16 -> ReLU (rounding is monotone)
                float v[32];
                tmem_ld32(tmem_d + lanes + 32u * half, v);
                const __nv_bfloat162 zero = __floats2bfloat162_rn(0.0f, 0.0f);
                uint32_t w[16], m = 0;
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    const __nv_bfloat162 b = __hmax2(__floats2bfloat162_rn(v[2 * q], v[2 * q + 1]), zero);
                    w[q] = *reinterpret_cast<const uint32_t*>(&b);
                    m |= (((w[q] & 0x7FFF7FFFu) + 0x7FFF7FFFu) & 0x80008000u) >> (15 - q);
                }
#pragma unroll
                for (int l = 0; l < 5; ++l)
                    if (l == k - 4) mask[l] = m;
                put_half(w, tmem_a + lanes + 16u * half, block(acts + (size_t)(k - 4) * ld * kHid, 8) + 32 * half, true);
            } else if (k == 9) {
                // prediction, loss and dL/dpred -> dOut5
                if (half == 0) {
                    float o[16];
                    tmem_ld16(tmem_d + lanes, o);
                    float d[3] = {0.0f, 0.0f, 0.0f};
                    if (in_range) {
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            const float p = o[c], y = target[3 * (size_t)r + c];
                            const float den = p * p + kLossEps, e = p - y;
                            loss += e * e / den;
                            d[c] = 2.0f * e / den * scale;
                        }
                    }
                    const uint32_t w0 = pack(d[0], d[1]), w1 = pack(d[2], 0.0f);
                    tmem_st4(tmem_a + lanes, w0, w1, 0u, 0u);
                    tmem_st4(tmem_a + lanes + 4u, 0u, 0u, 0u, 0u);
                    uint4* g5 = block(douts + (size_t)5 * ld * kHid, kOut / 8);
                    g5[0] = make_uint4(w0, w1, 0u, 0u);
                    g5[8] = make_uint4(0u, 0u, 0u, 0u);
                }
            } else {
                // dOut_l = dAct_l where layer l's activation is positive
                const int l = 14 - k;
                float v[32];
                tmem_ld32(tmem_d + lanes + 32u * half, v);
                uint32_t w[16], m = 0;
#pragma unroll
                for (int q = 0; q < 5; ++q)
                    if (q == l) m = mask[q];
#pragma unroll
                for (int q = 0; q < 16; ++q)
                    w[q] = pack(v[2 * q], v[2 * q + 1]) & (((m >> q) & 0x00010001u) * 0xFFFFu);
                put_half(w, tmem_a + lanes + 16u * half, block(douts + (size_t)l * ld * kHid, 8) + 32 * half, l > 0);
                if (l == 0) {
                    tc_fence_before();   // the next tile's batches overwrite the accumulator
                    break;
                }
            }
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            tc_fence_before();     // accumulator reads and operand writes, ordered before the MMAs
            __syncwarp();
            uint32_t before = 0;
            if (lane == 0)
                asm volatile("atom.acq_rel.cta.shared::cta.add.u32 %0, [%1], 1;"
                             : "=r"(before)
                             : "r"(smem_u32(&arrived))
                             : "memory");
            before = __shfl_sync(0xFFFFFFFFu, before, 0);
            if (before % kTrWarps == kTrWarps - 1) {   // the operand is complete
                if (!weights_here) {
                    uint32_t it = 0;
                    while (!mbar_try_wait(smem_u32(&wbar), 0u) && ++it < kTcWaitCap) {}
                    if (it >= kTcWaitCap) fail = 1;
                    weights_here = true;
                }
                if (lane == 0) issued += 1;
                train_issue(k, tmem_d, tmem_a, w_base, w_base + kTcWBytes, mb, lane);
            }
            __syncwarp();
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFu, loss, o);
    if (lane == 0) warp_loss[warp] = loss;
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0) {
        tc_fence_after();
        float sum = 0.0f;
        for (int w = 0; w < kTrWarps; ++w) sum += warp_loss[w];
        loss_part[blockIdx.x] = sum;
        // the weights' copies and the last batch, before shared memory and
        // TMEM are given back
        uint32_t it = 0;
        while (!mbar_try_wait(smem_u32(&wbar), 0u) && ++it < kTcDrainCap) {}
        if (fail) {
            it = 0;
            while (issued && !mbar_try_wait(mb, (issued - 1u) & 1u) && ++it < kTcDrainCap) {}
            atomicOr(err, kErrMlpTimeout);
        }
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(kTrCols));
    }
}

// ---------------------------------------------------------------- weight gradient on tcgen05
// k_wgrad_tc: dW_l[o][i] = sum over rows r of dOut_l[r][o] * in_l[r][i], split
// over the batch rows and the six layers: CTA (c, l) takes layer l's rows
// [c * R, (c + 1) * R) and writes layer l's slice of partial c (k_reduce_adam
// sums the partials, in the order of the chunks; chunks past the last row
// write nothing).  D = A * B with
// M = o, N = i (208 or 64), K = rows, FP32 D in TMEM (256 or 64 columns).
// Both operands are MN-major without swizzle: a core matrix is 8 consecutive
// rows (K) x 8 features (MN), 128 contiguous bytes, which is how
// k_mlp_train_tc stores them:
//   A (dOut_l^T): core matrix (o/8, r/8) at (r/8) * LBO_A + (o/8) * 128,
//                 LBO_A = O * 16 (an 8-row group of all O outputs), SBO = 128;
//   B (in_l):     core matrix (i/8, r/8) at (r/8) * LBO_B + (i/8) * 128,
//                 LBO_B = I * 16, SBO = 128.
// So 64 rows of an operand are one contiguous block, and a step is staged by
// two bulk copies into a ring of kWgStages (A, then B behind it); one thread
// keeps the ring full and issues the MMAs.  The MMA has M = 128 and the layer O
// = 64 or 16 real rows: the descriptor's MN groups past O/8 read the bytes
// that follow (the next 8-row groups, then B), and the D rows they give are
// never read.  32,768 rows (60 MB of operands, 16 MB of partials): 28 us with
// 16-byte copies by every thread from row-major arrays, 15.7 us now.  (Chunks of
// 704 rows instead of 256, 47 partials instead of 128, took 12.6 us, but sum in
// another order: after four Adam steps on the same batch the weights were 1e-4
// from these.)  Waits are bounded as in the other kernels.
constexpr int kWgRows = 64;                                   // rows per staging step (4 MMAs of K = 16)
constexpr int kWgStages = 2;
constexpr int kWgStage = kWgRows * (kHid + kIn) * 2;          // 34,816
constexpr int kWgSmem = kWgStages * kWgStage;                 // 69,632: three CTAs per SM
constexpr int kWgMinRows = 256;                               // rows per CTA, at least
constexpr int kMaxPartials = 148;                             // row chunks (one FP32 partial each), at most

__device__ __forceinline__ uint32_t idesc_bf16_mn(int m, int n) {
    return idesc_bf16(m, n) | (1u << 15) | (1u << 16);        // A and B MN-major
}

// Also advances the step counters (read by k_reduce_adam, which follows).
__global__ void __launch_bounds__(128, 3) k_wgrad_tc(NrcCount cnt, uint32_t ld, uint32_t rows_per_cta,
                                                     const __nv_bfloat16* __restrict__ enc,
                                                     const __nv_bfloat16* __restrict__ acts,
                                                     const __nv_bfloat16* __restrict__ douts,
                                                     float* __restrict__ partial, StepState* st, int do_step,
                                                     uint32_t* err) {
    extern __shared__ __align__(1024) uint8_t wg_smem[];
    __shared__ __align__(8) uint64_t full[kWgStages], done[kWgStages];
    __shared__ int fail;
    __shared__ uint32_t tmem_base;
    const uint32_t n = rows_of(cnt);
    if (do_step && n > 0 && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {   // an empty batch takes no step
        st->step += 1;
        st->ema_steps += 1;
    }
    const uint32_t row0 = blockIdx.x * rows_per_cta;
    if (row0 >= n) return;
    const int t = threadIdx.x, warp = t >> 5;
    const int l = blockIdx.y;                        // this CTA's layer
    const int O = out_dim(l), I = in_dim(l);
    const uint32_t cols = l == 0 ? 256u : 64u;       // TMEM columns: N = 208 or 64, a power of two
    const int steps = (int)((min(rows_per_cta, n - row0) + kWgRows - 1) / kWgRows);
    if (t < kWgStages) {
        mbar_init(smem_u32(&full[t]));
        mbar_init(smem_u32(&done[t]));
    }
    if (t == 0) fail = 0;
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                     "r"(cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = tmem_base;
    if (t == 0) {
        const uint8_t* a_src = reinterpret_cast<const uint8_t*>(douts + (size_t)l * ld * kHid) + (size_t)row0 * O * 2;
        const uint8_t* b_src = reinterpret_cast<const uint8_t*>(l == 0 ? enc : acts + (size_t)(l - 1) * ld * kHid) +
                               (size_t)row0 * I * 2;
        const uint32_t a_bytes = kWgRows * O * 2, b_bytes = kWgRows * I * 2;
        auto load = [&](int s) {
            const int b = s % kWgStages;
            const uint32_t dst = smem_u32(wg_smem + b * kWgStage), bar = smem_u32(&full[b]);
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(a_bytes + b_bytes)
                         : "memory");
            bulk_load(dst, a_src + (size_t)s * a_bytes, a_bytes, bar);
            bulk_load(dst + a_bytes, b_src + (size_t)s * b_bytes, b_bytes, bar);
        };
        auto wait = [&](uint64_t* bar, int s) {   // for step s's phase of its ring slot
            uint32_t it = 0;
            while (!mbar_try_wait(smem_u32(&bar[s % kWgStages]), (uint32_t)(s / kWgStages) & 1u) && ++it < kTcWaitCap) {}
            return it < kTcWaitCap;
        };
        const uint32_t idesc = idesc_bf16_mn(128, I);
        int loaded = 0, issued = 0;   // steps
        bool ok = true;
        for (; loaded < min(steps, kWgStages); ++loaded) load(loaded);
        for (int s = 0; s < steps; ++s) {
            if (!(ok = wait(full, s))) break;
            tc_fence_after();
            const uint32_t a0 = smem_u32(wg_smem + (s % kWgStages) * kWgStage), b0 = a0 + a_bytes;
#pragma unroll
            for (int ks = 0; ks < kWgRows / 16; ++ks)
                umma(tmem_d, umma_desc(a0 + (uint32_t)(ks * 2 * O * 16), (uint32_t)(O * 16), 128u),
                     umma_desc(b0 + (uint32_t)(ks * 2 * I * 16), (uint32_t)(I * 16), 128u), idesc,
                     (s > 0 || ks > 0) ? 1u : 0u);
            umma_commit(smem_u32(&done[s % kWgStages]));
            issued = s + 1;
            // the slot of step s - 1 takes step s - 1 + kWgStages once its MMAs are done
            if (s >= 1 && loaded < steps) {
                if (!(ok = wait(done, s - 1))) break;
                load(loaded++);
            }
        }
        if (ok) ok = wait(done, steps - 1);   // a commit covers every earlier MMA of the thread
        if (!ok) {
            // copies in flight and the last commit, before shared memory and TMEM are given back
            uint32_t it = 0;
            for (int s = max(0, loaded - kWgStages); s < loaded; ++s)
                while (!mbar_try_wait(smem_u32(&full[s % kWgStages]), (uint32_t)(s / kWgStages) & 1u) && ++it < kTcDrainCap) {}
            it = 0;
            while (issued && !mbar_try_wait(smem_u32(&done[(issued - 1) % kWgStages]),
                                            (uint32_t)((issued - 1) / kWgStages) & 1u) && ++it < kTcDrainCap) {}
            fail = 1;
            atomicOr(err, kErrMlpTimeout);
        }
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    // D rows o < O to this chunk's partial
    if (!fail && warp * 32 < O) {
        float* dst = partial + (size_t)blockIdx.x * kParams + param_off(l) + (size_t)(warp * 32 + (t & 31)) * I;
        const bool real = warp * 32 + (t & 31) < O;
        for (int c0 = 0; c0 < I; c0 += 16) {
            float v[16];
            tmem_ld16(tmem_d + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
            if (real) {
                float4* d4 = reinterpret_cast<float4*>(dst + c0);
                d4[0] = make_float4(v[0], v[1], v[2], v[3]);
                d4[1] = make_float4(v[4], v[5], v[6], v[7]);
                d4[2] = make_float4(v[8], v[9], v[10], v[11]);
                d4[3] = make_float4(v[12], v[13], v[14], v[15]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(cols));
    }
}

// ---------------------------------------------------------------- optimiser
__device__ __forceinline__ void param_coords(int p, int& l, int& o, int& i) {
    l = 0;
    while (l < 5 && p >= param_off(l + 1)) ++l;
    int local = p - param_off(l), in = in_dim(l);
    o = local / in;
    i = local - o * in;
}

// grad = sum of the CTA partials; with do_step, Adam on the FP32 master
// weights (bias corrections 1 - beta^step; rows 3..15 of the output layer and
// the padded inputs stay zero), the bf16 training packs (forward and
// transposed, both in the tensor cores' canonical layout), and the inference
// pack: with ema_a > 0, ema = ema_a * ema + (1 - ema_a) * w (ema
// starts at 0) and the pack holds ema / (1 - ema_a^ema_steps), else w.
// A block takes kAdamParams parameters; its threads bring all their partials to
// shared memory at once (one load at a time by the summing thread took 7.5 us
// for 128 partials, 7.0 us now), and one thread each adds them in their
// order.  One more block sums the loss.
constexpr int kAdamParams = 64, kAdamThreads = 256;
static_assert(kParams % kAdamParams == 0, "whole blocks");
__global__ void __launch_bounds__(kAdamThreads)
    k_reduce_adam(const float* __restrict__ partial, uint32_t rows_per_part, const float* __restrict__ loss_part,
                  int n_loss, float* __restrict__ loss, NrcCount cnt, float* __restrict__ grad, float* __restrict__ w,
                  float* __restrict__ m, float* __restrict__ v, AdamArgs ar, const StepState* __restrict__ st,
                  int do_step, __nv_bfloat16* __restrict__ wtc, __nv_bfloat16* __restrict__ wtcb,
                  float* __restrict__ ema, __nv_bfloat16* __restrict__ winf) {
    __shared__ float s_part[kMaxPartials][kAdamParams];
    if (blockIdx.x == kParams / kAdamParams) {
        float sum = 0.0f;
        for (int k = threadIdx.x; k < n_loss; k += kAdamThreads) sum += loss_part[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
        if ((threadIdx.x & 31) == 0) s_part[0][threadIdx.x >> 5] = sum;
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int k = 1; k < kAdamThreads / 32; ++k) sum += s_part[0][k];
            *loss = sum;
        }
        return;
    }
    const int q = threadIdx.x % kAdamParams, p = blockIdx.x * kAdamParams + q;
    const uint32_t n = rows_of(cnt);
    const int n_part = (int)((n + rows_per_part - 1) / rows_per_part);   // the chunks that hold rows
#pragma unroll 16
    for (int k = threadIdx.x / kAdamParams; k < n_part; k += kAdamThreads / kAdamParams)
        s_part[k][q] = __ldg(partial + (size_t)k * kParams + p);
    __syncthreads();
    if (threadIdx.x >= kAdamParams) return;
    float gsum = 0.0f;
#pragma unroll 8
    for (int k = 0; k < n_part; ++k) gsum += s_part[k][q];
    grad[p] = gsum;
    if (!do_step || n == 0) return;
    const float step = (float)st->step;
    const float c1 = 1.0f - powf(ar.b1, step), c2 = 1.0f - powf(ar.b2, step);
    int l, o, i;
    param_coords(p, l, o, i);
    float x = w[p];
    bool frozen = (l == 5 && o >= 3) || (l == 0 && i >= kInReal);
    if (!frozen) {
        float mm = ar.b1 * m[p] + (1.0f - ar.b1) * gsum;
        float vv = ar.b2 * v[p] + (1.0f - ar.b2) * gsum * gsum;
        m[p] = mm;
        v[p] = vv;
        x -= ar.lr * ((mm / c1) / (sqrtf(vv / c2) + ar.eps) + ar.wd * x);
        w[p] = x;
    }
    __nv_bfloat16 h = __float2bfloat16_rn(x);
    wtc[tc_index(l, o, i)] = h;
    if (l >= 1) wtcb[tcb_index(l, o, i)] = h;
    float xi = x;
    if (ar.ema_a > 0.0f) {
        float e = ar.ema_a * ema[p] + (1.0f - ar.ema_a) * x;
        ema[p] = e;
        xi = e / (1.0f - powf(ar.ema_a, (float)st->ema_steps));
    }
    winf[tc_index(l, o, i)] = __float2bfloat16_rn(xi);
}

// Packs the master weights (after creation or replacement) and restarts the
// moving average: the inference pack holds w.
__global__ void k_pack(const float* __restrict__ w, __nv_bfloat16* __restrict__ wtc,
                       __nv_bfloat16* __restrict__ wtcb, float* __restrict__ ema, __nv_bfloat16* __restrict__ winf,
                       StepState* st) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p == 0) st->ema_steps = 0;
    if (p >= kParams) return;
    int l, o, i;
    param_coords(p, l, o, i);
    __nv_bfloat16 h = __float2bfloat16_rn(w[p]);
    wtc[tc_index(l, o, i)] = h;
    winf[tc_index(l, o, i)] = h;
    if (l >= 1) wtcb[tcb_index(l, o, i)] = h;
    ema[p] = 0.0f;
}

}  // namespace nrc
}  // namespace ilm

using namespace ilm;
using namespace ilm::nrc;

struct ilm_nrc {
    ilm_nrc_config cfg;
    DeviceBuffer state;                          // StepState
    DeviceBuffer w, m, v, grad, wtc, wtcb;       // params and their training packs
    DeviceBuffer ema, winf;                      // moving average and its inference pack
    DeviceBuffer partial;                        // k_wgrad_tc partial sums
    DeviceBuffer err;                            // device error word (kErrMlpTimeout)
    DeviceBuffer raw, enc, out, target, acts, douts, loss, loss_part;
    cudaStream_t stream = nullptr;
    ~ilm_nrc() {
        if (stream) cudaStreamDestroy(stream);
    }
};

namespace {

Enc enc_params(const ilm_nrc* h) {
    const float* b = h->cfg.bound;
    return Enc{b[0], b[1], b[2], 1.0f / fmaxf(b[3] - b[0], 1e-12f), 1.0f / fmaxf(b[4] - b[1], 1e-12f),
               1.0f / fmaxf(b[5] - b[2], 1e-12f)};
}

cudaError_t pack(ilm_nrc* h, cudaStream_t s) {
    k_pack<<<(kParams + 255) / 256, 256, 0, s>>>(
        static_cast<const float*>(h->w.ptr), static_cast<__nv_bfloat16*>(h->wtc.ptr),
        static_cast<__nv_bfloat16*>(h->wtcb.ptr), static_cast<float*>(h->ema.ptr),
        static_cast<__nv_bfloat16*>(h->winf.ptr), static_cast<StepState*>(h->state.ptr));
    return cudaGetLastError();
}

// Rows per batch that a count can give (the batch's share of the cap).
uint32_t batch_cap(const NrcCount& c) { return c.batches > 1 ? (c.cap + c.batches - 1) / c.batches : c.cap; }

cudaError_t reserve_train(ilm_nrc* h, uint32_t rows) {
    const size_t ld = ((size_t)rows + 127) / 128 * 128;   // whole tiles
    cudaError_t e;
    if ((e = h->enc.reserve(ld * kIn * 2)) != cudaSuccess) return e;
    if ((e = h->acts.reserve(ld * 5 * kHid * 2)) != cudaSuccess) return e;
    return h->douts.reserve(ld * 6 * kHid * 2);
}

// Network output with the inference weights (the moving-average pack).
cudaError_t infer_rows(ilm_nrc* h, const float* raw, NrcCount cnt, float* out, cudaStream_t s) {
    // one CTA per SM, a warpgroup for every tile as long as there are SMs and
    // warpgroups; TMEM columns are allocated in powers of two
    const uint32_t tiles = std::max<uint32_t>(1, (batch_cap(cnt) + 127) / 128);
    const uint32_t groups = std::min<uint32_t>(kInfGroups, (tiles + 147) / 148);
    const uint32_t grid = std::min<uint32_t>(148, (tiles + groups - 1) / groups);
    const uint32_t cols = groups == 1 ? 128u : (groups == 2 ? 256u : 512u);
    k_mlp_infer_tc<<<grid, 128 * groups, kTcWBytes, s>>>(raw, cnt, enc_params(h),
                                                         static_cast<const __nv_bfloat16*>(h->winf.ptr), out,
                                                         static_cast<uint32_t*>(h->err.ptr), cols);
    return cudaGetLastError();
}

// Loss gradient of the current weights into h->grad and the loss sum into
// h->loss; with do_step, one Adam step.
cudaError_t train_rows(ilm_nrc* h, const float* raw, const float* target, NrcCount cnt, int do_step,
                       cudaStream_t s) {
    cudaError_t e;
    const uint32_t cap = batch_cap(cnt);
    if ((e = reserve_train(h, cap)) != cudaSuccess) return e;
    const uint32_t tiles = (cap + 127) / 128, ld = tiles * 128;   // ld: layer stride of acts / douts
    const uint32_t grid = std::max<uint32_t>(1, std::min<uint32_t>(kTrGrid, tiles));
    __nv_bfloat16* enc = static_cast<__nv_bfloat16*>(h->enc.ptr);
    __nv_bfloat16* acts = static_cast<__nv_bfloat16*>(h->acts.ptr);
    __nv_bfloat16* douts = static_cast<__nv_bfloat16*>(h->douts.ptr);
    float* loss_part = static_cast<float*>(h->loss_part.ptr);
    uint32_t* err = static_cast<uint32_t*>(h->err.ptr);
    k_mlp_train_tc<<<grid, kTrThreads, kTrSmem, s>>>(raw, target, cnt, enc_params(h),
                                                     static_cast<const __nv_bfloat16*>(h->wtc.ptr),
                                                     static_cast<const __nv_bfloat16*>(h->wtcb.ptr), ld, enc, acts, douts,
                                                     loss_part, err);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    // row chunks of kWgMinRows or more (a multiple of kWgRows), at most kMaxPartials
    uint32_t per_cta = (cap + kMaxPartials - 1) / kMaxPartials;
    per_cta = std::max<uint32_t>(kWgMinRows, (per_cta + kWgRows - 1) / kWgRows * kWgRows);
    const uint32_t chunks = std::max<uint32_t>(1, (cap + per_cta - 1) / per_cta);
    StepState* st = static_cast<StepState*>(h->state.ptr);
    k_wgrad_tc<<<dim3(chunks, kLayers), 128, kWgSmem, s>>>(cnt, ld, per_cta, enc, acts, douts,
                                                           static_cast<float*>(h->partial.ptr), st, do_step, err);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    AdamArgs ar{h->cfg.lr, h->cfg.beta1, h->cfg.beta2, h->cfg.eps,
                h->cfg.ema > 0.0f && h->cfg.ema < 1.0f ? h->cfg.ema : 0.0f, h->cfg.weight_decay};
    k_reduce_adam<<<kParams / kAdamParams + 1, kAdamThreads, 0, s>>>(
        static_cast<const float*>(h->partial.ptr), per_cta, loss_part, (int)grid, static_cast<float*>(h->loss.ptr), cnt,
        static_cast<float*>(h->grad.ptr), static_cast<float*>(h->w.ptr), static_cast<float*>(h->m.ptr),
        static_cast<float*>(h->v.ptr), ar, st, do_step, static_cast<__nv_bfloat16*>(h->wtc.ptr),
        static_cast<__nv_bfloat16*>(h->wtcb.ptr), static_cast<float*>(h->ema.ptr),
        static_cast<__nv_bfloat16*>(h->winf.ptr));
    return cudaGetLastError();
}

// Device copy of host-or-device input into dst (grown as needed).
cudaError_t take(DeviceBuffer& dst, const float* src, size_t bytes, cudaStream_t s) {
    cudaError_t e = dst.reserve(bytes);
    if (e != cudaSuccess) return e;
    return cudaMemcpyAsync(dst.ptr, src, bytes, cudaMemcpyDefault, s);
}

}  // namespace

namespace ilm {

cudaError_t nrc_infer_async(ilm_nrc* h, const float* raw, NrcCount n, float* out, cudaStream_t s) {
    return infer_rows(h, raw, n, out, s);
}

cudaError_t nrc_train_async(ilm_nrc* h, const float* raw, const float* target, NrcCount n, cudaStream_t s) {
    return train_rows(h, raw, target, n, 1, s);
}

cudaError_t nrc_reserve(ilm_nrc* h, uint32_t rows) { return reserve_train(h, rows); }

uint32_t* nrc_error_word(ilm_nrc* h) { return static_cast<uint32_t*>(h->err.ptr); }

}  // namespace ilm

extern "C" {

int32_t ilm_nrc_create(ilm_context* ctx, const ilm_nrc_config* cfg, ilm_nrc** out) {
    if (!ctx || !cfg || !out) return ILM_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    if (!(cfg->weight_decay >= 0.0f) || !std::isfinite(cfg->weight_decay) || !(cfg->weight_decay * cfg->lr < 1.0f)) {
        set_error(ctx, "ilm_nrc_create: weight_decay must be finite, >= 0 and below 1 / lr");
        return ILM_ERR_INVALID_ARGUMENT;
    }
    if (cudaSetDevice(ctx->device) != cudaSuccess) return ILM_ERR_CUDA;
    auto h = std::make_unique<ilm_nrc>();
    h->cfg = *cfg;
    cudaError_t e;
    if ((e = cudaStreamCreateWithFlags(&h->stream, cudaStreamNonBlocking)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    for (DeviceBuffer* b : {&h->w, &h->m, &h->v, &h->grad, &h->ema})
        if ((e = b->reserve(kParams * 4)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    if ((e = h->partial.reserve((size_t)kMaxPartials * kParams * 4)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    if ((e = h->wtc.reserve(kParams * 2)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    if ((e = h->winf.reserve(kParams * 2)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    if ((e = h->wtcb.reserve(kTcbElems * 2)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    if ((e = h->loss.reserve(4)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    if ((e = h->loss_part.reserve(kTrGrid * 4)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    if ((e = h->err.reserve(4)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    cudaMemset(h->err.ptr, 0, 4);
    if ((e = h->state.reserve(sizeof(StepState))) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    cudaMemset(h->state.ptr, 0, sizeof(StepState));
    // He-uniform initialisation from PCG32; padded inputs and output rows 3..15 zero
    std::vector<float> w(kParams, 0.0f);
    Pcg32 rng(cfg->seed);
    for (int l = 0; l < kLayers; ++l) {
        int in = in_dim(l), fan = l == 0 ? kInReal : in;
        float s = std::sqrt(6.0f / (float)fan);
        for (int o = 0; o < out_dim(l); ++o)
            for (int i = 0; i < in; ++i) {
                float u = rng.uniform_float();
                bool zero = (l == 0 && i >= kInReal) || (l == 5 && o >= 3);
                w[param_off(l) + o * in + i] = zero ? 0.0f : (2.0f * u - 1.0f) * s;
            }
    }
    cudaMemcpy(h->w.ptr, w.data(), kParams * 4, cudaMemcpyHostToDevice);
    cudaMemset(h->m.ptr, 0, kParams * 4);
    cudaMemset(h->v.ptr, 0, kParams * 4);
    cudaMemset(h->wtc.ptr, 0, kParams * 2);
    cudaMemset(h->winf.ptr, 0, kParams * 2);
    cudaMemset(h->wtcb.ptr, 0, kTcbElems * 2);
    cudaFuncSetAttribute(k_mlp_train_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrSmem);
    cudaFuncSetAttribute(k_wgrad_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kWgSmem);
    cudaFuncSetAttribute(k_mlp_infer_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcWBytes);
    if ((e = pack(h.get(), h->stream)) != cudaSuccess) return cuda_fail(ctx, e, "nrc pack");
    if ((e = cudaStreamSynchronize(h->stream)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    *out = h.release();
    return ILM_OK;
}

int32_t ilm_nrc_destroy(ilm_context* ctx, ilm_nrc* h) {
    if (!ctx || !h) return ILM_ERR_INVALID_ARGUMENT;
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(h->stream);
    delete h;
    return ILM_OK;
}

int32_t ilm_nrc_params(ilm_context* ctx, ilm_nrc* h, float* get, const float* set) {
    if (!ctx || !h) return ILM_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return ILM_ERR_CUDA;
    cudaStreamSynchronize(h->stream);
    cudaError_t e;
    if (set) {
        if ((e = cudaMemcpy(h->w.ptr, set, kParams * 4, cudaMemcpyDefault)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
        if ((e = pack(h, h->stream)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
        cudaStreamSynchronize(h->stream);
    }
    if (get && (e = cudaMemcpy(get, h->w.ptr, kParams * 4, cudaMemcpyDefault)) != cudaSuccess)
        return cuda_fail(ctx, e, "nrc");
    return ILM_OK;
}

int32_t ilm_nrc_infer(ilm_context* ctx, ilm_nrc* h, const float* inputs, uint64_t n, float* out, void* stream) {
    if (!ctx || !h || (n && (!inputs || !out))) return ILM_ERR_INVALID_ARGUMENT;
    if (n == 0) return ILM_OK;
    if (n > (1ull << 28)) return ILM_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return ILM_ERR_CUDA;
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : h->stream;
    cudaError_t e;
    bool dev_in = classify(inputs) == PtrKind::kDevice, dev_out = classify(out) == PtrKind::kDevice;
    const float* raw = inputs;
    if (!dev_in) {
        if ((e = take(h->raw, inputs, n * 12 * 4, s)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
        raw = static_cast<const float*>(h->raw.ptr);
    }
    float* dst = out;
    if (!dev_out) {
        if ((e = h->out.reserve(n * 12)) != cudaSuccess) return cuda_fail(ctx, e, "nrc buffers");
        dst = static_cast<float*>(h->out.ptr);
    }
    if ((e = infer_rows(h, raw, NrcCount{nullptr, (uint32_t)n, 1, 0}, dst, s)) != cudaSuccess)
        return cuda_fail(ctx, e, "nrc forward");
    if (!dev_out) {
        cudaMemcpyAsync(out, dst, n * 12, cudaMemcpyDeviceToHost, s);
        uint32_t flags = 0;
        cudaMemcpyAsync(&flags, h->err.ptr, 4, cudaMemcpyDeviceToHost, s);
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
        if (flags) {
            set_error(ctx, "ilm_nrc_infer: a tensor-core wait ran out of time");
            return ILM_ERR_TIMEOUT;
        }
    }
    return ILM_OK;
}

static int32_t train_impl(ilm_context* ctx, ilm_nrc* h, const float* inputs, const float* targets, uint64_t n,
                          float* loss, float* grad_out, int step, void* stream) {
    if (!ctx || !h || !inputs || !targets || n == 0 || n > (1ull << 24)) return ILM_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return ILM_ERR_CUDA;
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : h->stream;
    cudaError_t e;
    const float* raw = inputs;
    if (classify(inputs) != PtrKind::kDevice) {
        if ((e = take(h->raw, inputs, n * 12 * 4, s)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
        raw = static_cast<const float*>(h->raw.ptr);
    }
    const float* tg = targets;
    if (classify(targets) != PtrKind::kDevice) {
        if ((e = take(h->target, targets, n * 3 * 4, s)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
        tg = static_cast<const float*>(h->target.ptr);
    }
    if ((e = train_rows(h, raw, tg, NrcCount{nullptr, (uint32_t)n, 1, 0}, step, s)) != cudaSuccess)
        return cuda_fail(ctx, e, "nrc training");
    if (grad_out) cudaMemcpyAsync(grad_out, h->grad.ptr, kParams * 4, cudaMemcpyDefault, s);
    if (loss) {
        float ls = 0.0f;
        cudaMemcpyAsync(&ls, h->loss.ptr, 4, cudaMemcpyDeviceToHost, s);
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
        *loss = ls / (3.0f * (float)n);
    } else if (grad_out) {
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    }
    return ILM_OK;
}

int32_t ilm_nrc_train_step(ilm_context* ctx, ilm_nrc* h, const float* inputs, const float* targets, uint64_t n,
                           float* loss, void* stream) {
    return train_impl(ctx, h, inputs, targets, n, loss, nullptr, 1, stream);
}

int32_t ilm_nrc_gradients(ilm_context* ctx, ilm_nrc* h, const float* inputs, const float* targets, uint64_t n,
                          float* grad_out, float* loss) {
    return train_impl(ctx, h, inputs, targets, n, loss, grad_out, 0, nullptr);
}

int32_t ilm_nrc_encode(ilm_context* ctx, ilm_nrc* h, const float* inputs, uint64_t n, void* enc_out) {
    if (!ctx || !h || !inputs || !enc_out || n == 0 || n > (1ull << 28)) return ILM_ERR_INVALID_ARGUMENT;
    if (cudaSetDevice(ctx->device) != cudaSuccess) return ILM_ERR_CUDA;
    cudaError_t e;
    if ((e = take(h->raw, inputs, n * 12 * 4, h->stream)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    if ((e = h->enc.reserve(n * kIn * 2)) != cudaSuccess) return cuda_fail(ctx, e, "nrc buffers");
    k_nrc_encode<<<(unsigned)((n + 127) / 128), 128, 0, h->stream>>>(static_cast<const float*>(h->raw.ptr),
                                                                     (uint32_t)n, enc_params(h),
                                                                     static_cast<__nv_bfloat16*>(h->enc.ptr));
    if ((e = cudaGetLastError()) != cudaSuccess) return cuda_fail(ctx, e, "nrc encode");
    cudaMemcpyAsync(enc_out, h->enc.ptr, n * kIn * 2, cudaMemcpyDefault, h->stream);
    if ((e = cudaStreamSynchronize(h->stream)) != cudaSuccess) return cuda_fail(ctx, e, "nrc");
    return ILM_OK;
}

}  // extern "C"
