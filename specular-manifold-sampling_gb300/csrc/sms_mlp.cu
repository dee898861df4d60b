// sms_mlp.cu -- training and inference kernels of the learned seed proposal.
//
// No counterpart in the reference, which seeds Newton walks uniformly on the
// specular shape (manifold_ss.cpp:223, Shape::sample_position).  The network
// maps a query's features (shading point, light sample, shading normal) to an
// 8-component diagonal Gaussian mixture over the caster's uv frame; the
// estimator mixes it with the uniform seeding (sms_mlp.cuh, proposal_seed).
//
// Network: 9 (padded to 16) -> 64 -> 64 -> 64 -> 64 -> 48 (40 used), SiLU
// between layers, BF16 weights and activations, FP32 accumulation on the
// tensor cores (mma.m16n8k16), FP32 master weights and Adam moments.
//
// One optimizer step is four launches:
//   mlp_train_fb_kernel  forward, mixture NLL and its gradient, backward
//                        through all layers (two warps per 16 samples);
//                        writes the transposed layer inputs h^T and
//                        pre-activation gradients dz^T, accumulates bias
//                        gradients and the batch loss
//   mlp_wgrad_kernel     dW_l = dz_l^T h_l on the tensor cores, one warp per
//                        (16x8 tile, batch chunk)
//   mlp_adam_kernel      Adam on the master copy, refreshes both BF16 copies
//   mlp_step_kernel      advances the device step counter
#include <algorithm>

#include "sms_mlp.cuh"

namespace sms {
namespace mlp {

constexpr int kZsFloats = 4 * 8 * 4 * 32;   // per 16 samples: hidden pre-activations
// per 16 samples: the staged input tile (16 x kXLd bf16), reused for the output
// rows (16 x kOutPad floats)
constexpr int kStageFloats = 16 * kXLd / 2;
static_assert(kStageFloats >= 16 * kOutPad, "stage holds the output rows");
// training, per 16 samples: the A fragments its two warps pass each other,
// [buffer][k-tile][register][lane]
constexpr int kPassWords = 2 * 4 * 4 * 32;
constexpr int kTrainTiles = 4;   // 16-sample tiles of a training block

// lowbias32 integer hash (C. Wellons, "Prospecting for hash functions").
__device__ __forceinline__ uint32_t hash32(uint32_t x) {
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    return x;
}

// Negative log-likelihood of (u, v) (relative to the anchor) under the
// mixture of raw outputs row[40]; row becomes `scale` times its gradient with
// respect to them (padded columns zero).
__device__ float mixture_nll(float *row, float u, float v, float scale) {
    float mx = row[0];
    #pragma unroll
    for (int k = 1; k < kComp; ++k) mx = fmaxf(mx, row[k]);
    float se = 0.f;
    #pragma unroll
    for (int k = 0; k < kComp; ++k) se += __expf(row[k] - mx);
    const float logz = mx + __logf(se);
    float *lp = row + kGmmParams;   // log densities, in the padding
    static_assert(kOutPad - kGmmParams >= kComp, "the padding holds the log densities");
    float lmax = -INFINITY;
    #pragma unroll 2
    for (int k = 0; k < kComp; ++k) {
        const float lsx = log_sigma(row[24 + 2 * k]), lsy = log_sigma(row[25 + 2 * k]);
        const float dx = (u - row[8 + 2 * k]) * __expf(-lsx), dy = (v - row[9 + 2 * k]) * __expf(-lsy);
        lp[k] = (row[k] - logz) - 1.8378770664093453f - lsx - lsy - 0.5f * (dx * dx + dy * dy);
        lmax = fmaxf(lmax, lp[k]);
    }
    float s = 0.f;
    #pragma unroll
    for (int k = 0; k < kComp; ++k) s += __expf(lp[k] - lmax);
    const float logp = lmax + __logf(s);
    #pragma unroll 2
    for (int k = 0; k < kComp; ++k) {
        const float r = __expf(lp[k] - logp);   // responsibility
        row[k] = (__expf(row[k] - logz) - r) * scale;
        #pragma unroll
        for (int d = 0; d < 2; ++d) {
            const float raw = row[24 + 2 * k + d];
            const float sg = sigmoid(raw);
            const float ls = kLsMin + (kLsMax - kLsMin) * sg;
            const float iv = __expf(-2.f * ls);
            const float e = (d == 0 ? u : v) - row[8 + 2 * k + d];
            row[8 + 2 * k + d] = (-r * e * iv) * scale;
            row[24 + 2 * k + d] = (r * (1.f - e * e * iv) * (kLsMax - kLsMin) * sg * (1.f - sg)) * scale;
        }
        lp[k] = 0.f;
    }
    return -logp;
}

// ------------------------------------------------------------------ inference
__global__ void __launch_bounds__(128) mlp_forward_kernel(MlpDev m, const float *__restrict__ feat, uint32_t n,
                                                          float *__restrict__ out, int mixture) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __nv_bfloat16 *sw = reinterpret_cast<__nv_bfloat16 *>(smem_raw);
    float *stage = reinterpret_cast<float *>(smem_raw + (size_t)kWeightsFwd * 2) + (threadIdx.x / 32) * kStageFloats;
    stage_weights(m.wbf, sw, kWeightsFwd);
    stage_wait();
    const int lane = threadIdx.x & 31;
    const uint32_t wpb = blockDim.x / 32;
    for (uint32_t w = blockIdx.x * wpb + threadIdx.x / 32; (size_t)w * 16 < n; w += gridDim.x * wpb) {
        const uint32_t b0 = w * 16;
        float xn[kIn];
        #pragma unroll
        for (int k = 0; k < kIn; ++k) {
            const uint32_t row = b0 + (uint32_t)(lane & 15);
            xn[k] = row < n ? (__ldg(feat + (size_t)k * n + row) - m.shift[k]) * m.scale[k] : 0.f;
        }
        __nv_bfloat16 *sx = reinterpret_cast<__nv_bfloat16 *>(stage);
        stage_inputs(xn, sx);
        float o[6][4];
        forward(m, sw, sx, o);
        __syncwarp();
        stage_outputs(o, stage);
        __syncwarp();
        if (lane < 16 && b0 + lane < n) {
            const float *row = stage + lane * kOutPad;
            if (mixture) {
                const uint32_t r = b0 + lane;
                auto F = [&](int k) { return __ldg(feat + (size_t)k * n + r); };
                float au, av;
                anchor_uv(m.frame, mk(F(0), F(1), F(2)), mk(F(3), F(4), F(5)), au, av);
                mixture_from_raw(row, out + r, n, au, av, m.sigma_scale);
            } else {
                for (int c = 0; c < kGmmParams; ++c) out[(size_t)c * n + b0 + lane] = row[c];
            }
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ training
// A serial chain per 16 samples, one block per SM (shared memory): bound by the
// latency of its instructions.  Two warps share the 16 samples, each with half
// of every layer's outputs, and pass each other their halves as bf16 A
// fragments (8,192 samples: 42 us with one warp, 33 with two).  The layers are a
// loop: the code is run through once, and unrolled (10,000 instructions) its warps
// waited more for instructions than for anything else (from a cold cache 7.5 of 13
// cycles an instruction; now 0.1 of 7).  The weights come asynchronously while the
// inputs are encoded.
struct TrainTile {
    uint32_t *pass;   // kPassWords
    int tile, half;   // of the block; this warp's half of the outputs
    int turn = 0;     // buffer of the next exchange

    __device__ __forceinline__ void sync() const {
        asm volatile("bar.sync %0, 64;" ::"r"(1 + tile) : "memory");
    }
    // own: this warp's k-tiles 2 half and 2 half + 1; a: all four.  The buffers
    // alternate, so that a warp may write the next before the other has read
    // this one, and only that.
    __device__ __forceinline__ void exchange(const uint32_t own[2][4], uint32_t a[4][4]) {
        const int lane = threadIdx.x & 31;
        uint32_t *buf = pass + turn * (kPassWords / 2) + lane;
        turn ^= 1;
        #pragma unroll
        for (int k = 0; k < 2; ++k)
            #pragma unroll
            for (int i = 0; i < 4; ++i) buf[((2 * half + k) * 4 + i) * 32] = own[k][i];
        sync();
        #pragma unroll
        for (int k = 0; k < 4; ++k)
            #pragma unroll
            for (int i = 0; i < 4; ++i) a[k][i] = buf[(k * 4 + i) * 32];
    }
};

// Bias gradient of NT n-tiles of dz, gb the first one's.
template <int NT>
__device__ __forceinline__ void bias_grad(const float dz[][4], float *gb) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    #pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
        const int c = nt * 8 + 2 * t;
        float s0 = dz[nt][0] + dz[nt][2], s1 = dz[nt][1] + dz[nt][3];
        #pragma unroll
        for (int off = 4; off < 32; off <<= 1) {
            s0 += __shfl_xor_sync(0xffffffffu, s0, off);
            s1 += __shfl_xor_sync(0xffffffffu, s1, off);
        }
        if (g == 0) {
            atomicAdd(gb + c, s0);
            atomicAdd(gb + c + 1, s1);
        }
    }
}

// This warp's half of the dz of the layer below: (dZ W) dsilu(z), W its rows of
// the [in][out] copy (ldb elements each), z its pre-activations.
template <int KT>
__device__ __forceinline__ void dz_back(const __nv_bfloat16 *Wb, int ldb, const uint32_t da[4][4], const float *z,
                                        float dz[4][4]) {
    const int lane = threadIdx.x & 31;
    #pragma unroll
    for (int nt = 0; nt < 4; ++nt)
        #pragma unroll
        for (int i = 0; i < 4; ++i) dz[nt][i] = 0.f;
    #pragma unroll
    for (int kt = 0; kt < KT; ++kt) mma_row<4>(Wb, ldb, kt, da[kt], dz);
    #pragma unroll
    for (int nt = 0; nt < 4; ++nt)
        #pragma unroll
        for (int i = 0; i < 4; ++i) dz[nt][i] *= dsilu(z[(nt * 4 + i) * 32 + lane]);
}

__global__ void __launch_bounds__(64 * kTrainTiles) mlp_train_fb_kernel(MlpDev m, const float *__restrict__ feat,
                                                                        const float *__restrict__ uv, size_t ld,
                                                                        uint32_t n_data, int batch, int shuffle) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __nv_bfloat16 *sw = reinterpret_cast<__nv_bfloat16 *>(smem_raw);
    float *fsm = reinterpret_cast<float *>(smem_raw + (size_t)kWeightsAll * 2);
    TrainTile T;
    T.tile = (int)(threadIdx.x / 64);
    T.half = (int)(threadIdx.x / 32) & 1;
    float *zs = fsm + T.tile * kZsFloats;
    float *stage = fsm + kTrainTiles * kZsFloats + T.tile * kStageFloats;
    T.pass = reinterpret_cast<uint32_t *>(fsm + kTrainTiles * (kZsFloats + kStageFloats)) + T.tile * kPassWords;
    stage_weights(m.wbf, sw, kWeightsAll);
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, half = T.half;
    const int b0 = ((int)blockIdx.x * kTrainTiles + T.tile) * 16;
    const uint32_t step = *m.step;
    auto row_of = [&](int r) -> uint32_t {
        const uint32_t b = (uint32_t)(b0 + r);
        return shuffle ? hash32(step * 0x9E3779B9u ^ hash32(b)) % n_data : b % n_data;
    };
    __nv_bfloat16 *sx = reinterpret_cast<__nv_bfloat16 *>(stage);
    if (b0 < batch) {
        // while the weights come: a quarter of the features per 16 lanes
        const uint32_t r = row_of(lane & 15);
        __nv_bfloat16 *row = sx + (lane & 15) * kXLd;
        const int q = 2 * half + (lane >> 4);
        #pragma unroll
        for (int k = 0; k < (kIn + 3) / 4; ++k) {
            const int f = q + 4 * k;
            if (f < kIn) stage_feature(row, f, (__ldg(feat + (size_t)f * ld + r) - m.shift[f]) * m.scale[f]);
        }
        if (q == 3) stage_padding(row);
    }
    stage_wait();
    if (b0 >= batch) return;   // whole tiles only (batch is a multiple of 16)

    // ---- forward
    float acc[4][4];
    uint32_t own[2][4], a[4][4];
    const int n0 = 32 * half;   // first output of this warp
    start_bias<4>(m.bias + n0, acc);
    #pragma unroll 1
    for (int kt = 0; kt < kInPad / 16; ++kt) {
        uint32_t a0[4];
        input_fragment(sx, kt, a0);
        if ((kt & 1) == half) store_transposed_tile(m.hT + b0, batch, kt * 16, a0);
        mma_row<4>(sw + n0 * (kInPad + kPadK), kInPad + kPadK, kt, a0, acc);
    }
    #pragma unroll 1
    for (int l = 1;; ++l) {
        // acc: pre-activations of layer l - 1
        float *zp = zs + (((l - 1) * 8 + 4 * half) * 4) * 32 + lane;
        #pragma unroll
        for (int nt = 0; nt < 4; ++nt)
            #pragma unroll
            for (int i = 0; i < 4; ++i) {
                zp[(nt * 4 + i) * 32] = acc[nt][i];
                acc[nt][i] = silu(acc[nt][i]);
            }
        pack_tiles<2>(acc, own);
        __nv_bfloat16 *dst = m.hT + (size_t)h_row(l) * batch + b0;
        store_transposed_tile(dst, batch, n0, own[0]);
        store_transposed_tile(dst, batch, n0 + 16, own[1]);
        T.exchange(own, a);
        if (l == kLayers - 1) break;
        const __nv_bfloat16 *W = sw + smf_off(1) + ((l - 1) * kHidden + n0) * (kHidden + kPadK);
        start_bias<4>(m.bias + l * 64 + n0, acc);
        #pragma unroll
        for (int kt = 0; kt < 4; ++kt) mma_row<4>(W, kHidden + kPadK, kt, a[kt], acc);
    }
    {
        float o[3][4];
        start_bias<3>(m.bias + (kLayers - 1) * 64 + 24 * half, o);
        #pragma unroll
        for (int kt = 0; kt < 4; ++kt)
            mma_row<3>(sw + smf_off(kLayers - 1) + 24 * half * (kHidden + kPadK), kHidden + kPadK, kt, a[kt], o);
        // the inputs under the output rows were last read before the exchanges
        stage_outputs<3>(o, stage, 24 * half);
    }
    T.sync();

    // ---- loss, 8 rows a warp
    float loss = 0.f;
    if (lane < 8) {
        const int i = 8 * half + lane;
        const uint32_t r = row_of(i);
        auto F = [&](int k) { return __ldg(feat + (size_t)k * ld + r); };
        float au, av;
        anchor_uv(m.frame, mk(F(0), F(1), F(2)), mk(F(3), F(4), F(5)), au, av);
        // the loss is the batch mean of (weighted) NLLs
        const float inv_b = (m.weighted ? __ldg(uv + 2 * ld + r) : 1.f) / (float)batch;
        loss = mixture_nll(stage + i * kOutPad, __ldg(uv + r) - au, __ldg(uv + ld + r) - av, inv_b) * inv_b;
    }
    #pragma unroll
    for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
    if (lane == 0) atomicAdd(m.loss + step % kLossHist, loss);
    T.sync();

    // ---- backward: dz of the output layer whole on both warps, then halves
    {
        float dz[6][4];
        #pragma unroll
        for (int nt = 0; nt < 6; ++nt) {
            const int c = nt * 8 + 2 * t;
            dz[nt][0] = stage[g * kOutPad + c];
            dz[nt][1] = stage[g * kOutPad + c + 1];
            dz[nt][2] = stage[(g + 8) * kOutPad + c];
            dz[nt][3] = stage[(g + 8) * kOutPad + c + 1];
        }
        pack_tiles<3>(dz, a);
        __nv_bfloat16 *dst = m.dzT + (size_t)dz_row(kLayers - 1) * batch + b0;
        float *gb = m.grad + b_off(kLayers - 1);
        if (half == 0) {
            store_transposed_tile(dst, batch, 0, a[0]);
            store_transposed_tile(dst, batch, 16, a[1]);
            bias_grad<2>(dz, gb);
        } else {
            store_transposed_tile(dst, batch, 32, a[2]);
            bias_grad<4>(dz + 2, gb + 16);
        }
    }
    dz_back<3>(sw + smb_off(kLayers - 1) + n0 * (kOutPad + kPadK), kOutPad + kPadK, a,
               zs + ((kLayers - 2) * 8 + 4 * half) * 4 * 32, acc);
    #pragma unroll 1
    for (int l = kLayers - 2;; --l) {
        pack_tiles<2>(acc, own);
        __nv_bfloat16 *dst = m.dzT + (size_t)dz_row(l) * batch + b0;
        store_transposed_tile(dst, batch, n0, own[0]);
        store_transposed_tile(dst, batch, n0 + 16, own[1]);
        if (l == 0) break;
        T.exchange(own, a);
        bias_grad<4>(acc, m.grad + b_off(l) + n0);
        dz_back<4>(sw + smb_off(1) + ((l - 1) * kHidden + n0) * (kHidden + kPadK), kHidden + kPadK, a,
                   zs + ((l - 1) * 8 + 4 * half) * 4 * 32, acc);
    }
    bias_grad<4>(acc, m.grad + b_off(0) + n0);
}
static_assert(smb_off(kLayers - 1) == smb_off(1) + (kLayers - 2) * kHidden * (kHidden + kPadK),
              "hidden layers are evenly spaced");

// Samples a warp of mlp_wgrad_kernel sums up (the last one of a tile fewer).
// 8,192 samples at 128 / 256 / 512 / 1024: 88.6 / 86.5 / 88.6 / 89.9 us a
// gradient, 31,712 samples 201 / 183 / 175 / 173: longer chunks leave warps idle
// in small batches, shorter ones add more atomics.  A chunk that had to divide
// the batch was 32 samples at 31,712 (529 us).
constexpr int kWgradChunk = 256;

// dW_l[o][i] += sum_b dz_l[b][o] h_l[b][i] over one batch chunk; one warp per
// (layer, 16x8 output tile, chunk).  A = dz^T rows, B = h^T rows, both
// contiguous along the batch.  Bound by the latency of its loads, which are
// 16 bytes a lane (4 bytes before: 23 -> 8 us at 8,192 samples).
__global__ void __launch_bounds__(128) mlp_wgrad_kernel(MlpDev m, int batch) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int wid = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32;
    const int chunks = (batch + kWgradChunk - 1) / kWgradChunk;
    int tile = wid / chunks;
    const int ch = wid % chunks;
    int l = 0;
    for (; l < kLayers; ++l) {
        const int tl = (layer_out(l) / 16) * (layer_in(l) / 8);
        if (tile < tl) break;
        tile -= tl;
    }
    if (l >= kLayers) return;
    const int K = layer_in(l);
    const int mt = tile / (K / 8), nt = tile % (K / 8);
    const int b0 = ch * kWgradChunk, len = min(kWgradChunk, batch - b0);   // a multiple of 16
    const __nv_bfloat16 *ar = m.dzT + (size_t)(dz_row(l) + mt * 16 + g) * batch + b0;
    const __nv_bfloat16 *ar8 = ar + (size_t)8 * batch;
    const __nv_bfloat16 *br = m.hT + (size_t)(h_row(l) + nt * 8 + g) * batch + b0;
    float acc[4] = {0.f, 0.f, 0.f, 0.f};
    // The order of the samples within the sum is free as long as A and B agree:
    // lane t of a row takes 8 consecutive ones in one load, four pairs that
    // serve as the k pairs of two products.  Rows start on 16 bytes (the batch
    // is a multiple of 16 samples).
    const int wide = len & ~31;
    #pragma unroll 8
    for (int bb = 8 * t; bb < wide; bb += 32) {
        const uint4 a = *reinterpret_cast<const uint4 *>(ar + bb), a8 = *reinterpret_cast<const uint4 *>(ar8 + bb),
                    bv = *reinterpret_cast<const uint4 *>(br + bb);
        const uint32_t a0[4] = {a.x, a8.x, a.y, a8.y}, a1[4] = {a.z, a8.z, a.w, a8.w};
        mma16816(acc, a0, bv.x, bv.y);
        mma16816(acc, a1, bv.z, bv.w);
    }
    if (wide < len) {
        const int bb = wide + 2 * t;
        const uint32_t a[4] = {*reinterpret_cast<const uint32_t *>(ar + bb), *reinterpret_cast<const uint32_t *>(ar8 + bb),
                               *reinterpret_cast<const uint32_t *>(ar + bb + 8),
                               *reinterpret_cast<const uint32_t *>(ar8 + bb + 8)};
        mma16816(acc, a, *reinterpret_cast<const uint32_t *>(br + bb), *reinterpret_cast<const uint32_t *>(br + bb + 8));
    }
    float *gw = m.grad + w_off(l);
    const int r0 = mt * 16 + g, c0 = nt * 8 + 2 * t;
    atomicAdd(gw + r0 * K + c0, acc[0]);
    atomicAdd(gw + r0 * K + c0 + 1, acc[1]);
    atomicAdd(gw + (r0 + 8) * K + c0, acc[2]);
    atomicAdd(gw + (r0 + 8) * K + c0 + 1, acc[3]);
}

// Store parameter i (FP32) into the BF16 copies / bias table.  Padded input
// columns (>= kInEnc) of the first layer stay zero.
__device__ __forceinline__ float publish(const MlpDev &m, int i, float p) {
    int l = 0;
    while (l + 1 < kLayers && i >= w_off(l + 1)) ++l;
    const int j = i - w_off(l), K = layer_in(l), N = layer_out(l);
    if (j < N * K) {
        const int r = j / K, c = j % K;
        if (l == 0 && c >= kInEnc) p = 0.f;
        m.wbf[smf_off(l) + r * (K + kPadK) + c] = __float2bfloat16(p);
        m.wbf[smb_off(l) + c * (N + kPadK) + r] = __float2bfloat16(p);
    } else {
        m.bias[l * 64 + (j - N * K)] = p;
    }
    return p;
}

__global__ void mlp_adam_kernel(MlpDev m, float lr) {
    constexpr float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float tstep = (float)(*m.step + 1u);
    const float c1 = 1.f - powf(b1, tstep), c2 = 1.f - powf(b2, tstep);
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x) {
        const float gv = m.grad[i];
        const float mo = b1 * m.adam_m[i] + (1.f - b1) * gv;
        const float vo = b2 * m.adam_v[i] + (1.f - b2) * gv * gv;
        m.adam_m[i] = mo;
        m.adam_v[i] = vo;
        m.params[i] = publish(m, i, m.params[i] - lr * (mo / c1) / (sqrtf(vo / c2) + eps));
        m.grad[i] = 0.f;
    }
}

__global__ void mlp_step_kernel(MlpDev m) {
    const uint32_t s = *m.step + 1u;
    m.loss[s % kLossHist] = 0.f;
    *m.step = s;
}

__global__ void mlp_sync_kernel(MlpDev m) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kParams; i += gridDim.x * blockDim.x)
        m.params[i] = publish(m, i, m.params[i]);
}

__global__ void feature_moments_kernel(const float *__restrict__ feat, size_t ld, uint32_t n, double *out) {
    __shared__ double part[2 * kIn];
    if (threadIdx.x < 2 * kIn) part[threadIdx.x] = 0.0;
    __syncthreads();
    double s[kIn], q[kIn];
    #pragma unroll
    for (int k = 0; k < kIn; ++k) { s[k] = 0.0; q[k] = 0.0; }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        #pragma unroll
        for (int k = 0; k < kIn; ++k) {
            const double f = feat[(size_t)k * ld + i];
            s[k] += f;
            q[k] += f * f;
        }
    }
    #pragma unroll
    for (int k = 0; k < kIn; ++k) {
        atomicAdd(&part[k], s[k]);
        atomicAdd(&part[kIn + k], q[k]);
    }
    __syncthreads();
    if (threadIdx.x < 2 * kIn) atomicAdd(out + threadIdx.x, part[threadIdx.x]);
}

// ---------------------------------------------------------------- launchers
size_t smem_forward() { return (size_t)kWeightsFwd * 2 + (size_t)4 * kStageFloats * 4; }
size_t smem_train() {
    return (size_t)kWeightsAll * 2 + (size_t)kTrainTiles * (kZsFloats + kStageFloats + kPassWords) * 4;
}
size_t smem_seed_fused() { return (size_t)kWeightsFwd * 2 + (size_t)4 * (32 * kIn + kStageFloats) * 4; }

cudaError_t configure_kernels() {
    cudaError_t e = cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem_forward());
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(mlp_train_fb_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_train());
}

cudaError_t launch_sync(const MlpDev &m, cudaStream_t s) {
    mlp_sync_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(m);
    return cudaGetLastError();
}

cudaError_t launch_forward(const MlpDev &m, const float *feat, uint32_t n, float *out, bool mixture, int num_sms,
                           cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint32_t warps = (n + 15) / 16;
    const uint32_t blocks = std::min<uint32_t>((warps + 3) / 4, (uint32_t)num_sms * 4);
    mlp_forward_kernel<<<blocks, 128, smem_forward(), s>>>(m, feat, n, out, mixture ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_train_step(const MlpDev &m, const float *feat, const float *uv, size_t ld, uint32_t n_data,
                              int batch, float lr, bool shuffle, bool update, cudaStream_t s) {
    mlp_train_fb_kernel<<<(batch / 16 + kTrainTiles - 1) / kTrainTiles, 64 * kTrainTiles, smem_train(), s>>>(
        m, feat, uv, ld, n_data, batch, shuffle ? 1 : 0);
    int tiles = 0;
    for (int l = 0; l < kLayers; ++l) tiles += (layer_out(l) / 16) * (layer_in(l) / 8);
    const int wg_warps = tiles * ((batch + kWgradChunk - 1) / kWgradChunk);
    mlp_wgrad_kernel<<<(wg_warps + 3) / 4, 128, 0, s>>>(m, batch);
    if (update) {
        mlp_adam_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(m, lr);
        mlp_step_kernel<<<1, 1, 0, s>>>(m);
    }
    return cudaGetLastError();
}

cudaError_t launch_feature_moments(const float *feat, size_t ld, uint32_t n, double *out, cudaStream_t s) {
    if (n == 0) return cudaSuccess;
    const uint32_t blocks = std::min<uint32_t>((n + 255) / 256, 512u);
    feature_moments_kernel<<<blocks, 256, 0, s>>>(feat, ld, n, out);
    return cudaGetLastError();
}

}  // namespace mlp
}  // namespace sms
