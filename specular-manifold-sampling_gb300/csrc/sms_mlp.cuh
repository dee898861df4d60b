// sms_mlp.cuh -- device side of the learned seed proposal: the warp-level
// BF16 tensor-core forward pass, the mixture transform and seed sampling.
//
// A warp carries 16 samples (one m16 tile) through all layers in registers:
// the FP32 accumulator fragment of n-tiles (2k, 2k+1) of mma.m16n8k16 is, once
// rounded to BF16 and paired, exactly the A fragment of k-tile k of the next
// layer, so hidden activations never leave the register file.
#pragma once
#include <cuda_bf16.h>

#include "sms_device.cuh"
#include "sms_mlp.h"

namespace sms {
namespace mlp {

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}

// D += A (16x16 bf16, row-major) * B (16x8 bf16, column-major), FP32 accumulate.
__device__ __forceinline__ void mma16816(float d[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ float sigmoid(float z) { return 1.f / (1.f + __expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigmoid(z); }
__device__ __forceinline__ float dsilu(float z) {
    float s = sigmoid(z);
    return s * (1.f + z * (1.f - s));
}

// Copy bf16 weights (first `elems` elements) to shared memory: 16-byte
// asynchronous copies, all in flight at once; stage_wait before their use.
__device__ __forceinline__ void stage_weights(const __nv_bfloat16 *__restrict__ src, __nv_bfloat16 *dst, int elems) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    for (int i = threadIdx.x; i < elems / 8; i += blockDim.x)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + 16u * (uint32_t)i), "l"(src + 8 * i)
                     : "memory");
}
__device__ __forceinline__ void stage_wait() {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
}

// An 8x8 block of bf16 accumulator pairs (lane 4 g + t: row g, columns 2 t and
// 2 t + 1) to its transpose in memory: columns c0 .. c0 + 7 are rows of `ld`
// elements, its rows their elements r0 .. r0 + 7.
__device__ __forceinline__ void store_transposed(__nv_bfloat16 *dst, size_t ld, int c0, int r0, uint32_t frag) {
    const int lane = threadIdx.x & 31;
    uint32_t tr;
    asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(tr) : "r"(frag));
    *reinterpret_cast<uint32_t *>(dst + (size_t)(c0 + (lane >> 2)) * ld + r0 + 2 * (lane & 3)) = tr;
}
__device__ __forceinline__ void store_transposed_tile(__nv_bfloat16 *dst, size_t ld, int c0, const uint32_t a[4]) {
    store_transposed(dst, ld, c0, 0, a[0]);
    store_transposed(dst, ld, c0, 8, a[1]);
    store_transposed(dst, ld, c0 + 8, 0, a[2]);
    store_transposed(dst, ld, c0 + 8, 8, a[3]);
}

// Feature f = x of a row of the staged input tile: columns xn[0..8], then per
// feature sin (pi 2^j xn), j < kEncFreq, and cos (pi 2^j xn), then zeros.
__device__ __forceinline__ void stage_feature(__nv_bfloat16 *row, int f, float x) {
    row[f] = __float2bfloat16(x);
    #pragma unroll 1
    for (int j = 0; j < kEncFreq; ++j) {
        float sn, cs;
        sincospif(x * (float)(1 << j), &sn, &cs);
        row[kIn + f * 2 * kEncFreq + j] = __float2bfloat16(sn);
        row[kIn + f * 2 * kEncFreq + kEncFreq + j] = __float2bfloat16(cs);
    }
}
__device__ __forceinline__ void stage_padding(__nv_bfloat16 *row) {
    #pragma unroll
    for (int c = kInEnc; c < kInPad; ++c) row[c] = __float2bfloat16(0.f);
}

// Stage the encoded inputs of a 16-row tile as bf16 rows of kXLd elements:
// lanes l and l + 16 write row l, from the row's normalised features xn on
// both; half of the features each.
__device__ __forceinline__ void stage_inputs(const float xn[kIn], __nv_bfloat16 *sx) {
    const int lane = threadIdx.x & 31;
    __nv_bfloat16 *row = sx + (lane & 15) * kXLd;
    constexpr int kHalf = (kIn + 1) / 2;
    #pragma unroll
    for (int k = 0; k < kHalf; ++k) {
        const bool high = lane >= 16;
        const float x = high ? (k + kHalf < kIn ? xn[k + kHalf < kIn ? k + kHalf : 0] : 0.f) : xn[k];
        if (high && k + kHalf >= kIn) stage_padding(row);
        else stage_feature(row, high ? k + kHalf : k, x);
    }
    __syncwarp();
}
static_assert(2 * ((kIn + 1) / 2) == kIn + 1, "stage_inputs: the odd slot writes the padding");

// A fragment kt of the staged input rows.
__device__ __forceinline__ void input_fragment(const __nv_bfloat16 *sx, int kt, uint32_t a[4]) {
    const int lane = threadIdx.x & 31;
    const __nv_bfloat16 *xp = sx + (lane >> 2) * kXLd + kt * 16 + 2 * (lane & 3);
    a[0] = *reinterpret_cast<const uint32_t *>(xp);
    a[1] = *reinterpret_cast<const uint32_t *>(xp + 8 * kXLd);
    a[2] = *reinterpret_cast<const uint32_t *>(xp + 8);
    a[3] = *reinterpret_cast<const uint32_t *>(xp + 8 * kXLd + 8);
}

// Accumulators of NT n-tiles, started from the bias.
template <int NT>
__device__ __forceinline__ void start_bias(const float *bias, float acc[][4]) {
    const int t = threadIdx.x & 3;
    #pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const float b0 = bias[nt * 8 + 2 * t], b1 = bias[nt * 8 + 2 * t + 1];
        acc[nt][0] = b0; acc[nt][1] = b1; acc[nt][2] = b0; acc[nt][3] = b1;
    }
}

// acc += A (one k-tile) x B, B rows of ld elements from W.
template <int NT>
__device__ __forceinline__ void mma_row(const __nv_bfloat16 *W, int ld, int kt, const uint32_t a[4], float acc[][4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    #pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const __nv_bfloat16 *wp = W + (nt * 8 + g) * ld + kt * 16 + 2 * t;
        mma16816(acc[nt], a, *reinterpret_cast<const uint32_t *>(wp), *reinterpret_cast<const uint32_t *>(wp + 8));
    }
}

// The accumulators of 2 KT n-tiles as KT bf16 A fragments.
template <int KT>
__device__ __forceinline__ void pack_tiles(const float acc[][4], uint32_t a[][4]) {
    #pragma unroll
    for (int kt = 0; kt < KT; ++kt) {
        a[kt][0] = pack_bf16(acc[2 * kt][0], acc[2 * kt][1]);
        a[kt][1] = pack_bf16(acc[2 * kt][2], acc[2 * kt][3]);
        a[kt][2] = pack_bf16(acc[2 * kt + 1][0], acc[2 * kt + 1][1]);
        a[kt][3] = pack_bf16(acc[2 * kt + 1][2], acc[2 * kt + 1][3]);
    }
}

// Forward pass of one warp's 16 samples.  sw: forward weight copy in shared
// memory; sx: the staged input tile.  out: accumulators of the output layer
// (6 n-tiles).  The layers are a loop (see mlp_train_fb_kernel).
__device__ __forceinline__ void forward(const MlpDev &m, const __nv_bfloat16 *sw, const __nv_bfloat16 *sx,
                                        float out[6][4]) {
    float acc[8][4];
    uint32_t a[4][4];
    start_bias<8>(m.bias, acc);
    #pragma unroll 1
    for (int kt = 0; kt < kInPad / 16; ++kt) {
        uint32_t a0[4];
        input_fragment(sx, kt, a0);
        mma_row<8>(sw, kInPad + kPadK, kt, a0, acc);
    }
    #pragma unroll 1
    for (int l = 1;; ++l) {
        // acc: pre-activations of layer l - 1
        #pragma unroll
        for (int nt = 0; nt < 8; ++nt)
            #pragma unroll
            for (int i = 0; i < 4; ++i) acc[nt][i] = silu(acc[nt][i]);
        pack_tiles<4>(acc, a);
        if (l == kLayers - 1) break;
        start_bias<8>(m.bias + l * 64, acc);
        #pragma unroll
        for (int kt = 0; kt < 4; ++kt)
            mma_row<8>(sw + smf_off(1) + (l - 1) * kHidden * (kHidden + kPadK), kHidden + kPadK, kt, a[kt], acc);
    }
    start_bias<6>(m.bias + (kLayers - 1) * 64, out);
    #pragma unroll
    for (int kt = 0; kt < 4; ++kt) mma_row<6>(sw + smf_off(kLayers - 1), kHidden + kPadK, kt, a[kt], out);
}
static_assert(smf_off(kLayers - 1) == smf_off(1) + (kLayers - 2) * kHidden * (kHidden + kPadK),
              "hidden layers are evenly spaced");

// Write the accumulators of NT n-tiles of the output layer from column c0 on as
// rows of `stage` ([16][kOutPad] floats).
template <int NT = 6>
__device__ __forceinline__ void stage_outputs(const float o[][4], float *stage, int c0 = 0) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    #pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int c = c0 + nt * 8 + 2 * t;
        stage[g * kOutPad + c] = o[nt][0];
        stage[g * kOutPad + c + 1] = o[nt][1];
        stage[(g + 8) * kOutPad + c] = o[nt][2];
        stage[(g + 8) * kOutPad + c + 1] = o[nt][3];
    }
}

__device__ __forceinline__ float log_sigma(float raw) { return kLsMin + (kLsMax - kLsMin) * sigmoid(raw); }

// Raw outputs o[0..39] -> mixture (cdf[8], mean[16], sigma[16]) written with
// stride `stride` (SoA of a query batch); means are anchor + offset, sigmas
// are scaled by sigma_scale (seeding sharpness).
__device__ __forceinline__ void mixture_from_raw(const float *o, float *dst, size_t stride, float au, float av,
                                                 float sigma_scale) {
    float mx = o[0];
    #pragma unroll
    for (int k = 1; k < kComp; ++k) mx = fmaxf(mx, o[k]);
    float w[kComp], s = 0.f;
    #pragma unroll
    for (int k = 0; k < kComp; ++k) { w[k] = __expf(o[k] - mx); s += w[k]; }
    const float inv = 1.f / s;
    float c = 0.f;
    #pragma unroll
    for (int k = 0; k < kComp; ++k) {
        c += w[k] * inv;
        dst[(size_t)k * stride] = k == kComp - 1 ? 1.f : c;
    }
    #pragma unroll
    for (int k = 0; k < 2 * kComp; ++k) {
        dst[(size_t)(8 + k) * stride] = o[8 + k] + ((k & 1) ? av : au);
        dst[(size_t)(24 + k) * stride] = sigma_scale * __expf(log_sigma(o[24 + k]));
    }
}

// uv -> seed point on the frame.
__device__ __forceinline__ f3 frame_point(const SeedFrame &fr, float u, float v) {
    const f3 o = mk(fr.org[0], fr.org[1], fr.org[2]);
    if (fr.kind == 1) {
        float st, ct, sp, cp;
        sincospif(u, &st, &ct);
        sincospif(2.f * v, &sp, &cp);
        return o + mk(st * cp, st * sp, ct) * fr.ax_u[0];
    }
    return o + mk(fr.ax_u[0], fr.ax_u[1], fr.ax_u[2]) * u + mk(fr.ax_v[0], fr.ax_v[1], fr.ax_v[2]) * v;
}

// point on the shape -> uv (inverse of frame_point).
__device__ __forceinline__ void frame_uv(const SeedFrame &fr, f3 p, float &u, float &v) {
    const f3 d = p - mk(fr.org[0], fr.org[1], fr.org[2]);
    if (fr.kind == 1) {
        const float r = fr.ax_u[0];
        const float z = fminf(1.f, fmaxf(-1.f, d.z / r));
        u = acosf(z) * kInvPi;
        float ph = atan2f(d.y, d.x);
        if (ph < 0.f) ph += 2.f * kPi;
        v = ph * (0.5f * kInvPi);
        return;
    }
    const f3 au = mk(fr.ax_u[0], fr.ax_u[1], fr.ax_u[2]), av = mk(fr.ax_v[0], fr.ax_v[1], fr.ax_v[2]);
    u = dot(d, au) / dot(au, au);
    v = dot(d, av) / dot(av, av);
}

// Anchor of the mixture means for shading point x and light sample lp: the
// uv where the straight segment x -> lp meets the frame's plane (box frames;
// clamped to [-1, 2]^2), or the uv of the sphere point along the bisector of
// the directions from the centre to x and to lp (sphere frames).
__device__ __forceinline__ void anchor_uv(const SeedFrame &fr, f3 x, f3 lp, float &u, float &v) {
    const f3 o = mk(fr.org[0], fr.org[1], fr.org[2]);
    if (fr.kind == 1) {
        const f3 a = normalize(x - o), b = normalize(lp - o), h = a + b;
        const float l2 = dot(h, h);
        const f3 d = l2 > 1e-12f ? h * (1.f / sqrtf(l2)) : a;
        frame_uv(fr, o + d * fr.ax_u[0], u, v);
        return;
    }
    const f3 au = mk(fr.ax_u[0], fr.ax_u[1], fr.ax_u[2]), av = mk(fr.ax_v[0], fr.ax_v[1], fr.ax_v[2]);
    const f3 nrm = cross(au, av), d = lp - x;
    const float den = dot(d, nrm);
    const float t = fabsf(den) > 1e-12f * sqrtf(dot(d, d) * dot(nrm, nrm)) ? dot(o - x, nrm) / den : 0.5f;
    frame_uv(fr, x + d * t, u, v);
    u = fminf(2.f, fmaxf(-1.f, u));
    v = fminf(2.f, fmaxf(-1.f, v));
}

// Seed of one walk under the proposal: three uniform draws (component or
// defensive choice, then a 2D sample).  With probability `defensive` the
// shape's uniform seeding (the reference's sample_position); otherwise a
// Gaussian draw (Box-Muller) from the chosen component of the query's
// mixture (gmm: kGmmParams rows with row stride n).
__device__ __forceinline__ f3 proposal_seed(const DevScene &sc, const SeedProposal &pr, const DevShape &shape, const float *gmm,
                       size_t n, float u_sel, float u1, float u2) {
    if (u_sel < pr.defensive) return sample_position(sc, shape, u1, u2);
    const float us = (u_sel - pr.defensive) / (1.f - pr.defensive);
    int k = 0;
    while (k < kComp - 1 && us >= sms_ldg(gmm + (size_t)k * n)) ++k;
    const float r = sqrtf(-2.f * logf(1.f - u1));
    float sn, cs;
    sincospif(2.f * u2, &sn, &cs);
    const float u = sms_ldg(gmm + (size_t)(8 + 2 * k) * n) + sms_ldg(gmm + (size_t)(24 + 2 * k) * n) * (r * cs);
    const float v = sms_ldg(gmm + (size_t)(9 + 2 * k) * n) + sms_ldg(gmm + (size_t)(25 + 2 * k) * n) * (r * sn);
    return frame_point(pr.frame, u, v);
}

}  // namespace mlp
}  // namespace sms
