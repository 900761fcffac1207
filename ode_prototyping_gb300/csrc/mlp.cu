// mlp.cu -- training and inference kernels of the learned step-size proposer
// (16 -> 64 -> 64 -> 1, SiLU).  No counterpart in the reference.
//
// Training keeps FP32 master weights in a gb_mlp struct in device memory.
// The single passes (gb_mlp_forward_f32, _backward_f32, _adam_step):
//   forward  : one thread per sample, weights staged in shared memory, the
//              pre-activations z1, z2 saved for the backward pass;
//   backward : per-sample deltas (dz1, dz2, h1, h2) in one pass, then one
//              thread per parameter sums its gradient over the batch in
//              sample order (deterministic, no atomics);
//   adam     : one thread per parameter.
// A training epoch (gb_mlp_train) is two kernels, deterministic as well: epoch
// (forward, loss, deltas and gradient sums of a slice of the samples) and update
// (the slices' sums in order, then Adam).
// Inference in the controller uses BF16-rounded weights with FP32
// accumulation (mlp.cuh); gb_mlp_infer_bf16 exposes the same arithmetic.
#include <algorithm>
#include <cstring>

#include "mlp.cuh"

namespace gb {

namespace {

constexpr int kParamsW1 = kHid * kIn;
constexpr int kParamsW2 = kHid * kHid;
// trainable parameters in gb_mlp order: w1, b1, w2, b2, w3, b3
constexpr int kTrainable = kParamsW1 + kHid + kParamsW2 + kHid + kHid + 1;
constexpr int kActPerSample = 2 * kHid;         // z1, z2
constexpr int kDeltaPerSample = 4 * kHid;       // h1, dz1, h2, dz2

static_assert(offsetof(gb_mlp, b1) == sizeof(float) * kParamsW1, "layout");
static_assert(offsetof(gb_mlp, w2) == sizeof(float) * (kParamsW1 + kHid), "layout");

__device__ __forceinline__ float dsilu(float z) {
  const float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

__device__ __forceinline__ float* param_ptr(gb_mlp* m, int p) {
  return reinterpret_cast<float*>(m) + p;  // w1..b3 are contiguous floats
}

__global__ void forward_kernel(const gb_mlp* __restrict__ W, const float* __restrict__ x,
                               float* __restrict__ y, long long B, float* __restrict__ act,
                               int bf16) {
  __shared__ float w1[kHid * kIn];
  __shared__ float w2[kHid * kHid];
  __shared__ float w3[kHid], b1[kHid], b2[kHid];
  __shared__ float mean[kIn], scl[kIn];
  for (int k = threadIdx.x; k < kHid * kIn; k += blockDim.x) {
    float v = (&W->w1[0][0])[k];
    w1[k] = bf16 ? __bfloat162float(__float2bfloat16_rn(v)) : v;
  }
  for (int k = threadIdx.x; k < kHid * kHid; k += blockDim.x) {
    float v = (&W->w2[0][0])[k];
    w2[k] = bf16 ? __bfloat162float(__float2bfloat16_rn(v)) : v;
  }
  for (int k = threadIdx.x; k < kHid; k += blockDim.x) {
    float v = W->w3[k];
    w3[k] = bf16 ? __bfloat162float(__float2bfloat16_rn(v)) : v;
    b1[k] = W->b1[k];
    b2[k] = W->b2[k];
  }
  for (int k = threadIdx.x; k < kIn; k += blockDim.x) {
    mean[k] = W->in_mean[k];
    scl[k] = W->in_scale[k];
  }
  __syncthreads();
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s >= B) return;
  float xin[kIn];
#pragma unroll
  for (int k = 0; k < kIn; ++k) xin[k] = (x[s * kIn + k] - mean[k]) * scl[k];
  float h1[kHid];
  for (int o = 0; o < kHid; ++o) {
    float acc = b1[o];
#pragma unroll
    for (int k = 0; k < kIn; ++k) acc = fmaf(w1[o * kIn + k], xin[k], acc);
    if (act) act[s * kActPerSample + o] = acc;
    h1[o] = silu(acc);
  }
  float out = W->b3;
  for (int o = 0; o < kHid; ++o) {
    float acc = b2[o];
    for (int k = 0; k < kHid; ++k) acc = fmaf(w2[o * kHid + k], h1[k], acc);
    if (act) act[s * kActPerSample + kHid + o] = acc;
    out = fmaf(w3[o], silu(acc), out);
  }
  y[s] = W->out_scale * out + W->out_bias;
}

// Per-sample deltas: h1, dz1, h2, dz2.
__global__ void delta_kernel(const gb_mlp* __restrict__ W, const float* __restrict__ act,
                             const float* __restrict__ dy, long long B,
                             float* __restrict__ delta) {
  __shared__ float w2[kHid * kHid];
  __shared__ float w3[kHid];
  for (int k = threadIdx.x; k < kHid * kHid; k += blockDim.x) w2[k] = (&W->w2[0][0])[k];
  for (int k = threadIdx.x; k < kHid; k += blockDim.x) w3[k] = W->w3[k];
  __syncthreads();
  const long long s = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (s >= B) return;
  const float g = dy[s] * W->out_scale;
  const float* z1 = act + s * kActPerSample;
  const float* z2 = z1 + kHid;
  float* d = delta + s * kDeltaPerSample;
  float dz2[kHid];
  for (int o = 0; o < kHid; ++o) {
    dz2[o] = g * w3[o] * dsilu(z2[o]);
    d[2 * kHid + o] = silu(z2[o]);
    d[3 * kHid + o] = dz2[o];
  }
  for (int k = 0; k < kHid; ++k) {
    float acc = 0.f;
    for (int o = 0; o < kHid; ++o) acc = fmaf(w2[o * kHid + k], dz2[o], acc);
    d[k] = silu(z1[k]);
    d[kHid + k] = acc * dsilu(z1[k]);
  }
}

// One thread per trainable parameter; sums over samples in order.
__global__ void grad_kernel(const gb_mlp* __restrict__ W, const float* __restrict__ x,
                            const float* __restrict__ delta, const float* __restrict__ dy,
                            long long B, gb_mlp* __restrict__ G) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= kTrainable) return;
  double acc = 0.0;  // FP64 accumulation keeps the batch sum order-stable
  if (p < kParamsW1) {
    const int o = p / kIn, k = p % kIn;
    const float mean = W->in_mean[k], scl = W->in_scale[k];
    for (long long s = 0; s < B; ++s)
      acc += (double)delta[s * kDeltaPerSample + kHid + o] * ((x[s * kIn + k] - mean) * scl);
  } else if (p < kParamsW1 + kHid) {
    const int o = p - kParamsW1;
    for (long long s = 0; s < B; ++s) acc += delta[s * kDeltaPerSample + kHid + o];
  } else if (p < kParamsW1 + kHid + kParamsW2) {
    const int q = p - kParamsW1 - kHid;
    const int o = q / kHid, k = q % kHid;
    for (long long s = 0; s < B; ++s)
      acc += (double)delta[s * kDeltaPerSample + 3 * kHid + o] * delta[s * kDeltaPerSample + k];
  } else if (p < kParamsW1 + 2 * kHid + kParamsW2) {
    const int o = p - kParamsW1 - kHid - kParamsW2;
    for (long long s = 0; s < B; ++s) acc += delta[s * kDeltaPerSample + 3 * kHid + o];
  } else if (p < kTrainable - 1) {
    const int o = p - kParamsW1 - 2 * kHid - kParamsW2;
    const float os = W->out_scale;
    for (long long s = 0; s < B; ++s)
      acc += (double)(dy[s] * os) * delta[s * kDeltaPerSample + 2 * kHid + o];
  } else {
    const float os = W->out_scale;
    for (long long s = 0; s < B; ++s) acc += (double)(dy[s] * os);
  }
  *param_ptr(G, p) = (float)acc;
}

__global__ void zero_nontrainable_kernel(gb_mlp* G) {
  const int k = threadIdx.x;
  if (k < kIn) {
    G->in_mean[k] = 0.f;
    G->in_scale[k] = 0.f;
  }
  if (k == 0) {
    G->out_scale = 0.f;
    G->out_bias = 0.f;
  }
}

__device__ __forceinline__ void adam_param(float g, float& w, float& m, float& v, float lr,
                                           float b1, float b2, float eps, float c1, float c2) {
  m = b1 * m + (1.f - b1) * g;
  v = b2 * v + (1.f - b2) * g * g;
  const float mh = m / c1, vh = v / c2;
  w -= lr * mh / (sqrtf(vh) + eps);
}

__global__ void adam_kernel(gb_mlp* W, const gb_mlp* G, gb_mlp* M, gb_mlp* V, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= kTrainable) return;
  adam_param(*param_ptr(const_cast<gb_mlp*>(G), p), *param_ptr(W, p), *param_ptr(M, p),
             *param_ptr(V, p), lr, b1, b2, eps, c1, c2);
}

// ---------------------------------------------------------------------------
// The two kernels of a training epoch.
// ---------------------------------------------------------------------------
// acc + w0 v0 + w1 v1 + ..., one multiply-add after the other
__device__ __forceinline__ float chain4(float4 w, float4 v, float acc) {
  return fmaf(w.w, v.w, fmaf(w.z, v.z, fmaf(w.y, v.y, fmaf(w.x, v.x, acc))));
}

// An unevaluated sum of three floats, about 72 bits: exact products and sums of
// FP32 values to more than FP64's precision on the FP32 pipe, where a product
// and its sum take 22 cycles of a sub-partition and an FP64 multiply-add 76
// (with two conversions of 64 before it).  A product's error term is exact down
// to 2^-149 (products above 2^-102); what is lost below that is nothing beside
// Adam's 1e-8.
struct Sum3 {
  float h = 0.f, m = 0.f, l = 0.f;
};

// t += h + m + l
__device__ __forceinline__ void add3(Sum3& t, float h, float m, float l) {
  float e1, e2, e3, s;
  two_sum(t.h, h, s, e1);
  t.h = s;
  two_sum(t.m, m, s, e2);
  two_sum(s, e1, t.m, e3);
  t.l = __fadd_rn(t.l, __fadd_rn(l, __fadd_rn(e2, e3)));
}
// t += a b
__device__ __forceinline__ void add_product(Sum3& t, float a, float b) {
  const float p = __fmul_rn(a, b);
  add3(t, p, __fmaf_rn(a, b, -p), 0.f);
}
__device__ __forceinline__ void add_value(Sum3& t, float a) {
  float e, s;
  two_sum(t.h, a, s, e);
  t.h = s;
  two_sum(t.m, e, s, e);
  t.m = s;
  t.l = __fadd_rn(t.l, e);
}

// t rounded to FP32: the parts made disjoint first, as the sums above may leave
// the middle one as large as the first after a cancellation.
__device__ __forceinline__ float round3(const Sum3& t) {
  float h, m, l;
  two_sum(t.h, t.m, h, m);
  two_sum(m, t.l, m, l);
  two_sum(h, m, h, m);
  return __fadd_rn(h, __fadd_rn(m, l));
}

// Forward pass, loss (the asymmetric squared error w (y - t)^2 with w = over_w
// where y > t), deltas and gradient sums of a slice of the samples, 16 samples
// at a time.  GRAD false: the forward pass and each sample's loss alone.
//
// Forward and deltas: a thread per (output, two samples); every output is the
// same chain of multiply-adds as in forward_kernel and delta_kernel, so the
// values are theirs bit for bit.  The weights' rows are padded by 4 floats:
// 16-byte reads along them and single reads across them without bank conflicts.
// Gradient: every thread keeps a 2 x 4 block of w2's sums, a 1 x 2 block of w1's
// and one of the vectors', as sums of three floats of exact products (29 us at
// 2000 samples with FP64 multiply-adds: 5313 a sample, the FP64 pipe's rate).
// partial: [slice][3][parameter].
//
// The chip's SMs have one slice each, so what bounds an epoch is the chain
// within a CTA: the deltas stay in shared memory (as a kernel of their own the
// forward pass took 8 us and the gradient sums 14.5: an epoch 30.2 -> 26.8 us).
constexpr int kBatch = 16;  // samples staged at a time
constexpr int kEpochThreads = 512;
constexpr int kPartial = (kTrainable + 3) / 4 * 4;  // parameters, for 16-byte stores
template <bool GRAD>
__global__ void __launch_bounds__(kEpochThreads)
    epoch_kernel(const gb_mlp* __restrict__ W, const float* __restrict__ x,
                 const float* __restrict__ target, long long B, long long per, float over_w,
                 float* __restrict__ partial, float* __restrict__ lsample) {
  constexpr int T = kEpochThreads, G = T / kHid, R = kBatch / G, kPad = kHid + 4;
  __shared__ __align__(16) float w1[kHid][kIn + 4], w2[kHid][kPad];
  __shared__ __align__(16) float xs[kBatch][kIn], h1[kBatch][kPad], h2[kBatch][kPad],
      dz1[GRAD ? kBatch : 1][kPad], dz2[GRAD ? kBatch : 1][kPad], w3[kHid];
  __shared__ float sg[kBatch];
  after_previous(W, x, target, partial, lsample);
  let_next_in();
  const int t = threadIdx.x, o = t % kHid, g = t / kHid;
  const long long s0 = blockIdx.x * per, s1 = min(B, s0 + per);
#pragma unroll
  for (int k = t; k < kHid * kIn; k += T) w1[k / kIn][k % kIn] = (&W->w1[0][0])[k];
#pragma unroll
  for (int k = t; k < kHid * kHid; k += T) w2[k / kHid][k % kHid] = (&W->w2[0][0])[k];
  if (t < kHid) w3[t] = W->w3[t];
  const float mean = W->in_mean[t % kIn], scale = W->in_scale[t % kIn];
  const float b1 = W->b1[o], b2 = W->b2[o], b3 = W->b3, os = W->out_scale, ob = W->out_bias;
  const int o2 = t / 16, k4 = t % 16;  // w2's block: rows 2 o2, 2 o2 + 1, columns 4 k4 ...
  const int o1 = t / 8, k2 = t % 8;    // w1's: columns 2 k2, 2 k2 + 1
  Sum3 a2[2][4], a1[2], av;
  for (long long b = s0; b < s1; b += kBatch) {
    const int m = (int)min((long long)kBatch, s1 - b);
    if (t < m * kIn) xs[t / kIn][t % kIn] = (x[b * kIn + t] - mean) * scale;
    __syncthreads();
    float z1[R], z2[R];
#pragma unroll
    for (int r = 0; r < R; ++r) z1[r] = b1;
#pragma unroll
    for (int k = 0; k < kIn; k += 4) {
      const float4 w = *reinterpret_cast<const float4*>(&w1[o][k]);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (g + G * r < m)
          z1[r] = chain4(w, *reinterpret_cast<const float4*>(&xs[g + G * r][k]), z1[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) h1[g + G * r][o] = silu(z1[r]);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) z2[r] = b2;
#pragma unroll 4
    for (int k = 0; k < kHid; k += 4) {
      const float4 w = *reinterpret_cast<const float4*>(&w2[o][k]);
#pragma unroll
      for (int r = 0; r < R; ++r)
        z2[r] = chain4(w, *reinterpret_cast<const float4*>(&h1[g + G * r][k]), z2[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) h2[g + G * r][o] = silu(z2[r]);
    __syncthreads();
    if (t < m) {
      float out = b3;
#pragma unroll
      for (int k = 0; k < kHid; k += 4)
        out = chain4(*reinterpret_cast<const float4*>(&w3[k]),
                     *reinterpret_cast<const float4*>(&h2[t][k]), out);
      const float y = os * out + ob;
      const float res = y - target[b + t];
      const float w = res > 0.f ? over_w : 1.f;
      if (GRAD)
        sg[t] = 2.f * w * res / (float)B * os;
      else
        lsample[b + t] = w * res * res;
    }
    __syncthreads();
    if constexpr (GRAD) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (g + G * r < m) dz2[g + G * r][o] = sg[g + G * r] * w3[o] * dsilu(z2[r]);
      __syncthreads();
      float acc[R];
#pragma unroll
      for (int r = 0; r < R; ++r) acc[r] = 0.f;
#pragma unroll 4
      for (int k = 0; k < kHid; k += 4) {
        const float4 w = make_float4(w2[k][o], w2[k + 1][o], w2[k + 2][o], w2[k + 3][o]);
#pragma unroll
        for (int r = 0; r < R; ++r)
          acc[r] = chain4(w, *reinterpret_cast<const float4*>(&dz2[g + G * r][k]), acc[r]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) dz1[g + G * r][o] = acc[r] * dsilu(z1[r]);
      __syncthreads();
#pragma unroll 1
      for (int r = 0; r < m; ++r) {
        const float2 go = reinterpret_cast<const float2*>(dz2[r])[o2];
        const float4 gk = reinterpret_cast<const float4*>(h1[r])[k4];
        const float2 gx = reinterpret_cast<const float2*>(xs[r])[k2];
        const float ao[2] = {go.x, go.y}, ak[4] = {gk.x, gk.y, gk.z, gk.w};
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) add_product(a2[i][j], ao[i], ak[j]);
        add_product(a1[0], dz1[r][o1], gx.x);
        add_product(a1[1], dz1[r][o1], gx.y);
        if (t < kHid)
          add_value(av, dz1[r][t]);
        else if (t < 2 * kHid)
          add_value(av, dz2[r][t - kHid]);
        else if (t < 3 * kHid)
          add_product(av, sg[r], h2[r][t - 2 * kHid]);
        else if (t == 3 * kHid)
          add_value(av, sg[r]);
      }
      __syncthreads();
    }
  }
  if constexpr (GRAD) {
    float* out = partial + (long long)blockIdx.x * 3 * kPartial;
    constexpr int pw2 = kParamsW1 + kHid;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int q = (pw2 + (2 * o2 + i) * kHid) / 4 + k4;
      const Sum3* v = a2[i];
      reinterpret_cast<float4*>(out)[q] = make_float4(v[0].h, v[1].h, v[2].h, v[3].h);
      reinterpret_cast<float4*>(out + kPartial)[q] = make_float4(v[0].m, v[1].m, v[2].m, v[3].m);
      reinterpret_cast<float4*>(out + 2 * kPartial)[q] = make_float4(v[0].l, v[1].l, v[2].l, v[3].l);
    }
    const auto put = [&](int p, const Sum3& v) {
      out[p] = v.h;
      out[kPartial + p] = v.m;
      out[2 * kPartial + p] = v.l;
    };
#pragma unroll
    for (int j = 0; j < 2; ++j) put(o1 * kIn + 2 * k2 + j, a1[j]);
    if (t < kHid)
      put(kParamsW1 + t, av);
    else if (t <= 3 * kHid)  // b2, w3, b3 follow w2
      put(pw2 + kParamsW2 + t - kHid, av);
  }
}

// The slices' sums of 32 parameters (warp g adds slices g, g + 16, ... in order,
// then the warps' sums are added in order), rounded to FP32, and the Adam step.
// Bound by the latency of the loads: all of a warp's in flight at once up to 160
// slices (8 warps and 5 slices at a time: 9.4 us, so 6.0; the epoch 26.8 -> 25.0).
constexpr int kUpdateWarps = 16;
constexpr int kUpdateLoads = 10;  // slices of a warp loaded together: 160 cover the SMs
__global__ void __launch_bounds__(32 * kUpdateWarps)
    update_kernel(gb_mlp* W, const float* __restrict__ partial, int slices, gb_mlp* M, gb_mlp* V,
                  float lr, float b1, float b2, float eps, float c1, float c2) {
  __shared__ Sum3 sums[kUpdateWarps][32];
  after_previous(W, partial, M, V);
  let_next_in();
  const int lane = threadIdx.x % 32, g = threadIdx.x / 32;
  const int p = blockIdx.x * 32 + lane;
  const bool mine = g == 0 && p < kTrainable;
  float w = 0.f, m = 0.f, u = 0.f;
  if (mine) {
    w = *param_ptr(W, p);
    m = *param_ptr(M, p);
    u = *param_ptr(V, p);
  }
  Sum3 v;
  if (p < kTrainable) {
    constexpr int K = kUpdateLoads;
    for (int c = g; c < slices; c += K * kUpdateWarps) {
      float h[K], d[K], l[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const bool on = c + k * kUpdateWarps < slices;
        const float* q = partial + (long long)(c + k * kUpdateWarps) * 3 * kPartial + p;
        h[k] = on ? q[0] : 0.f;
        d[k] = on ? q[kPartial] : 0.f;
        l[k] = on ? q[2 * kPartial] : 0.f;
      }
#pragma unroll
      for (int k = 0; k < K; ++k) add3(v, h[k], d[k], l[k]);
    }
  }
  sums[g][lane] = v;
  __syncthreads();
  if (mine) {
#pragma unroll
    for (int r = 1; r < kUpdateWarps; ++r)
      add3(v, sums[r][lane].h, sums[r][lane].m, sums[r][lane].l);
    adam_param(round3(v), w, m, u, lr, b1, b2, eps, c1, c2);
    *param_ptr(W, p) = w;
    *param_ptr(M, p) = m;
    *param_ptr(V, p) = u;
  }
}

__global__ void mean_kernel(const float* __restrict__ v, long long B, float* out) {
  __shared__ double sh[256];
  double acc = 0.0;
  for (long long s = threadIdx.x; s < B; s += 256) acc += v[s];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int st = 128; st > 0; st /= 2) {
    if ((int)threadIdx.x < st) sh[threadIdx.x] += sh[threadIdx.x + st];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = (float)(sh[0] / (double)B);
}

unsigned nblk(long long n, int b) { return (unsigned)((n + b - 1) / b); }

uint64_t splitmix64(uint64_t& s) {
  uint64_t z = (s += 0x9e3779b97f4a7c15ULL);
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
  return z ^ (z >> 31);
}

}  // namespace

void* mlp_upload(const void* host_mlp, int* rc) {
  *rc = GB_OK;
  if (!host_mlp) {
    *rc = GB_ERR_INVALID_ARGUMENT;
    return nullptr;
  }
  const gb_mlp& m = *reinterpret_cast<const gb_mlp*>(host_mlp);
  MlpDev d;
  for (int o = 0; o < kHid; ++o) {
    for (int k = 0; k < kIn; ++k) d.w1[o * kIn + k] = __float2bfloat16_rn(m.w1[o][k]);
    for (int k = 0; k < kHid; ++k) d.w2[o * kHid + k] = __float2bfloat16_rn(m.w2[o][k]);
    d.w3[o] = __float2bfloat16_rn(m.w3[o]);
    d.b1[o] = m.b1[o];
    d.b2[o] = m.b2[o];
  }
  d.b3 = m.b3;
  for (int k = 0; k < kIn; ++k) {
    d.in_mean[k] = m.in_mean[k];
    d.in_scale[k] = m.in_scale[k];
  }
  d.out_scale = m.out_scale;
  d.out_bias = m.out_bias;
  void* p = nullptr;
  cudaError_t e = cudaMalloc(&p, sizeof(MlpDev));
  if (e == cudaSuccess) e = cudaMemcpy(p, &d, sizeof(MlpDev), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) {
    note_cuda_error(e);
    if (p) cudaFree(p);
    *rc = GB_ERR_CUDA;
    return nullptr;
  }
  return p;
}

}  // namespace gb

using namespace gb;

extern "C" int gb_mlp_init(gb_mlp* m, uint64_t seed) {
  if (!m) return GB_ERR_INVALID_ARGUMENT;
  std::memset(m, 0, sizeof *m);
  uint64_t s = seed;
  auto uni = [&s](float lim) {
    const double u = (double)(splitmix64(s) >> 11) * (1.0 / 9007199254740992.0);
    return (float)((2.0 * u - 1.0) * lim);
  };
  const float l1 = std::sqrt(6.0f / (kIn + kHid));
  const float l2 = std::sqrt(6.0f / (kHid + kHid));
  const float l3 = std::sqrt(6.0f / (kHid + 1));
  for (int o = 0; o < kHid; ++o)
    for (int k = 0; k < kIn; ++k) m->w1[o][k] = uni(l1);
  for (int o = 0; o < kHid; ++o)
    for (int k = 0; k < kHid; ++k) m->w2[o][k] = uni(l2);
  for (int o = 0; o < kHid; ++o) m->w3[o] = uni(l3);
  for (int k = 0; k < kIn; ++k) m->in_scale[k] = 1.f;
  m->out_scale = 1.f;
  return GB_OK;
}

extern "C" int64_t gb_mlp_act_floats(int64_t B) { return B < 0 ? 0 : B * kActPerSample; }

extern "C" int gb_mlp_forward_f32(const gb_mlp* W, const float* x, float* y, int64_t B,
                                  float* act, gb_stream_t stream) {
  if (!W || !x || !y || B < 1) return GB_ERR_INVALID_ARGUMENT;
  forward_kernel<<<nblk(B, 128), 128, 0, as_cuda(stream)>>>(W, x, y, B, act, 0);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

extern "C" int gb_mlp_infer_bf16(const gb_mlp* W, const float* x, float* y, int64_t B,
                                 gb_stream_t stream) {
  if (!W || !x || !y || B < 1) return GB_ERR_INVALID_ARGUMENT;
  forward_kernel<<<nblk(B, 128), 128, 0, as_cuda(stream)>>>(W, x, y, B, nullptr, 1);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

extern "C" size_t gb_mlp_backward_workspace_bytes(int64_t B) {
  return B < 1 ? 0 : (size_t)B * kDeltaPerSample * sizeof(float);
}

extern "C" int gb_mlp_backward_f32(const gb_mlp* W, const float* x, const float* act,
                                   const float* dy, gb_mlp* G, int64_t B, void* work,
                                   gb_stream_t stream) {
  if (!W || !x || !act || !dy || !G || !work || B < 1) return GB_ERR_INVALID_ARGUMENT;
  cudaStream_t s = as_cuda(stream);
  float* delta = reinterpret_cast<float*>(work);
  delta_kernel<<<nblk(B, 128), 128, 0, s>>>(W, act, dy, B, delta);
  GB_CUDA_TRY(cudaGetLastError());
  grad_kernel<<<nblk(kTrainable, 128), 128, 0, s>>>(W, x, delta, dy, B, G);
  GB_CUDA_TRY(cudaGetLastError());
  zero_nontrainable_kernel<<<1, 32, 0, s>>>(G);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

extern "C" int gb_mlp_adam_step(gb_mlp* W, const gb_mlp* G, gb_mlp* M, gb_mlp* V, float lr,
                                float b1, float b2, float eps, int32_t step, gb_stream_t stream) {
  if (!W || !G || !M || !V || step < 1) return GB_ERR_INVALID_ARGUMENT;
  const float c1 = 1.f - std::pow(b1, (float)step);
  const float c2 = 1.f - std::pow(b2, (float)step);
  adam_kernel<<<nblk(kTrainable, 256), 256, 0, as_cuda(stream)>>>(W, G, M, V, lr, b1, b2, eps,
                                                                   c1, c2);
  GB_CUDA_TRY(cudaGetLastError());
  return GB_OK;
}

extern "C" int gb_mlp_train(gb_mlp* W, const float* x, const float* target, int64_t B,
                            int32_t epochs, float lr, float over_w, float* loss_host,
                            gb_stream_t stream) {
  if (!W || !x || !target || B < 1 || epochs < 0) return GB_ERR_INVALID_ARGUMENT;
  cudaStream_t s = as_cuda(stream);
  // slices of the gradient sums: one per SM, at least 4 samples each
  const long long per = std::max(4LL, ((long long)B + num_sms() - 1) / num_sms());
  const int slices = (int)((B + per - 1) / per);
  // one allocation: partial sums, losses, moments
  const size_t n_partial = (size_t)slices * 3 * kPartial * sizeof(float);
  const size_t n_sample = (size_t)B * sizeof(float);
  unsigned char* base = nullptr;
  int rc = GB_OK;
  cudaError_t e = cudaMalloc((void**)&base, n_partial + n_sample + 2 * sizeof(gb_mlp) +
                                                sizeof(float));
  if (e != cudaSuccess) {
    note_cuda_error(e);
    return GB_ERR_CUDA;
  }
  float* partial = reinterpret_cast<float*>(base);
  float* ls = reinterpret_cast<float*>(base + n_partial);
  gb_mlp* M = reinterpret_cast<gb_mlp*>(ls + B);
  gb_mlp* V = M + 1;
  float* loss = reinterpret_cast<float*>(V + 1);
  e = cudaMemsetAsync(M, 0, 2 * sizeof(gb_mlp), s);
  for (int ep = 1; ep <= epochs && e == cudaSuccess; ++ep) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)ep), c2 = 1.f - std::pow(b2, (float)ep);
    e = launch_after(epoch_kernel<true>, (unsigned)slices, kEpochThreads, s, W, x, target, B, per,
                     over_w, partial, nullptr);
    if (e == cudaSuccess)
      e = launch_after(update_kernel, nblk(kTrainable, 32), 32 * kUpdateWarps, s, W, partial,
                       slices, M, V, lr, b1, b2, 1e-8f, c1, c2);
  }
  if (e != cudaSuccess) {
    note_cuda_error(e);
    rc = GB_ERR_CUDA;
  }
  if (rc == GB_OK) {
    // the loss of the trained network
    epoch_kernel<false><<<(unsigned)slices, kEpochThreads, 0, s>>>(W, x, target, B, per, over_w,
                                                                   nullptr, ls);
    mean_kernel<<<1, 256, 0, s>>>(ls, B, loss);
    float hl = 0.f;
    e = cudaMemcpyAsync(&hl, loss, sizeof(float), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    if (e != cudaSuccess) {
      note_cuda_error(e);
      rc = GB_ERR_CUDA;
    } else if (loss_host) {
      *loss_host = hl;
    }
  }
  cudaStreamSynchronize(s);
  cudaFree(base);
  return rc;
}
