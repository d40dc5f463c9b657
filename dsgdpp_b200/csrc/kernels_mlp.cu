// kernels_mlp.cu -- the step-size controller network: 16 -> 64 -> 64 -> 1, GELU.
//
// No reference counterpart: the reference's only adaptive step rule is
// BoldDriver (mf/sgd/decay/decay_bolddriver.h:59-67).  The controller maps 16
// features of the run's recent history to a log step multiplier clipped to
// [-1, 1]; BoldDriver stays the fallback.  Everything is FP32 and tiny (5,313
// parameters), so a call is bound by launches, copies and the latency of its
// chain.  A CTA of 256 threads takes four samples at a time (one, when there
// are few): four threads share a hidden unit, hold its weights in registers
// -- loaded once, with wide loads, before the inputs are needed -- and add
// their shares with two shuffles.  Gradients are summed in registers over a
// CTA's samples, so few rows of partial gradients reach memory; a second
// launch adds them in a fixed order (training is deterministic) and applies
// Adam.  Inputs and results live in pinned host memory that the kernels read
// and write, so no copy is enqueued.  Measured against one CTA of 64 threads
// per sample, a row of gradients per sample and copies through the stream:
// one forward pass of a sample 29.0 -> 19.5 us, gradient of 256 samples 70.4
// -> 32.8 us (host time of the call).
#include <type_traits>

#include "kernels.cuh"

namespace dsgdpp {
namespace {

constexpr int kIn = 16, kHid = 64;
// parameter layout
constexpr int kW1 = 0;                      // [kHid][kIn]
constexpr int kB1 = kW1 + kHid * kIn;       // [kHid]
constexpr int kW2 = kB1 + kHid;             // [kHid][kHid]
constexpr int kB2 = kW2 + kHid * kHid;      // [kHid]
constexpr int kW3 = kB2 + kHid;             // [kHid]
constexpr int kB3 = kW3 + kHid;             // [1]
constexpr int kParams = kB3 + 1;            // 5313

struct MlpGrid {
  int samples, per_cta, ctas;  // at a time, per CTA
};

__device__ __forceinline__ float gelu(float x) {
  return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}
// d/dx [x Phi(x)] = Phi(x) + x phi(x)
__device__ __forceinline__ float gelu_grad(float x) {
  const float cdf = 0.5f * (1.0f + erff(x * 0.70710678118654752f));
  const float pdf = 0.39894228040143268f * expf(-0.5f * x * x);
  return cdf + x * pdf;
}

constexpr int kThreads = 256;
constexpr int kStride = (kParams + 1 + 3) / 4 * 4;  // a row of partials: gradients, then the loss

__device__ __forceinline__ double gelu(double x) {
  return 0.5 * x * (1.0 + erf(x * 0.70710678118654752));
}
template <typename A>
__device__ __forceinline__ A quad_sum(A v) {  // over the four threads of a unit
  v += __shfl_xor_sync(kFullMask, v, 1);
  return v + __shfl_xor_sync(kFullMask, v, 2);
}

// Samples [blockIdx.x * per_cta, ...) of the batch, S at a time.  out[b] =
// clip(net(x_b), -1, 1).  GRAD: this CTA's sums of the gradient of (net(x_b) -
// y)^2 / batch (unclipped output) and of that loss into row blockIdx.x of
// partials.  Outputs, and gradients of few samples, take sums and activations
// in FP64: one output is one sum of 64 terms that may cancel, and FP32 sums err
// by 1e-6 of it now and then (FP64 by 5e-8, for 2 us more).  Thread (j, q) works on hidden unit j: on a quarter of its inputs
// for every sample, then on the unit itself for sample q.
template <int S, bool GRAD>
__global__ void __launch_bounds__(kThreads) mlp_kernel(const float* __restrict__ P, const float* X,
                                                       const float* Y, int batch, int per_cta,
                                                       float* out, float* partials) {
  using A = std::conditional_t<GRAD && S != 1, float, double>;
  const int t = threadIdx.x, j = t >> 2, q = t & 3, warp = t >> 5;
  __shared__ float xs[S][kIn];
  __shared__ A h1s[S][kHid], red[kThreads / 32][S];
  __shared__ float d2s[GRAD ? S : 1][kHid], d1s[GRAD ? S : 1][kHid];
  __shared__ float w2s[GRAD ? kHid : 1][kHid + 1];
  float w1[4], w2[16];
  {
    const float4 a = *reinterpret_cast<const float4*>(P + kW1 + j * kIn + q * 4);
    w1[0] = a.x; w1[1] = a.y; w1[2] = a.z; w1[3] = a.w;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float4 v = *reinterpret_cast<const float4*>(P + kW2 + j * kHid + q * 16 + 4 * c);
      w2[4 * c] = v.x; w2[4 * c + 1] = v.y; w2[4 * c + 2] = v.z; w2[4 * c + 3] = v.w;
    }
  }
  const float b1 = P[kB1 + j], b2 = P[kB2 + j], w3 = P[kW3 + j], b3 = P[kB3];
  if constexpr (GRAD) {
#pragma unroll
    for (int c = 0; c < 16; ++c) w2s[j][q * 16 + c] = w2[c];
  }
  float g1[4] = {}, g2[16] = {}, gb1 = 0, gb2 = 0, g3 = 0, gb3 = 0, loss = 0;
  const int begin = blockIdx.x * per_cta, end = min(batch, begin + per_cta);
  for (int s0 = begin; s0 < end; s0 += S) {
    for (int k = t; k < S * kIn; k += kThreads) {
      const int b = s0 + k / kIn;
      xs[k / kIn][k % kIn] = b < end ? X[(size_t)b * kIn + k % kIn] : 0.0f;
    }
    const bool mine = q < S && s0 + q < end;  // this thread's sample exists
    const float y = GRAD && mine ? Y[s0 + q] : 0.0f;
    __syncthreads();
    A z1 = 0, z2 = 0;  // of sample q
#pragma unroll
    for (int s = 0; s < S; ++s) {
      A a = 0;
#pragma unroll
      for (int c = 0; c < 4; ++c) a += (A)w1[c] * (A)xs[s][q * 4 + c];
      a = quad_sum(a) + b1;
      if (s == q) z1 = a;
    }
    if (q < S) h1s[q][j] = gelu(z1);
    __syncthreads();
#pragma unroll
    for (int s = 0; s < S; ++s) {
      A a = 0;
#pragma unroll
      for (int c = 0; c < 16; ++c) a += (A)w2[c] * h1s[s][q * 16 + c];
      a = quad_sum(a) + b2;
      if (s == q) z2 = a;
    }
    const A h2 = gelu(z2);
    A o = (A)w3 * h2;  // summed over the units: in the warp, then over the warps
#pragma unroll
    for (int off = 4; off < 32; off <<= 1) o += __shfl_xor_sync(kFullMask, o, off);
    if ((t & 31) < S) red[warp][q] = o;
    __syncthreads();
    A raw = b3;
    if (q < S) {
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) raw += red[w][q];
    }
    if (j == 0 && mine && out) out[s0 + q] = fminf(1.0f, fmaxf(-1.0f, (float)raw));
    if constexpr (GRAD) {
      // the loss is taken on the unclipped output (the clip applies to the
      // proposed multiplier only), so a saturated output still gets a gradient
      const A miss = raw - (A)y;
      const float dout = mine ? (float)((A)2 * miss / (A)batch) : 0.0f;
      if (mine) loss += (float)(miss * miss / (A)batch);
      gb3 += dout;
      g3 += dout * (float)h2;
      const float d2 = dout * w3 * gelu_grad((float)z2);
      gb2 += d2;
      if (q < S) d2s[q][j] = d2;
      __syncthreads();
      float dh1 = 0;  // sum_i W2[i][j] d2[i] of sample q
#pragma unroll
      for (int s = 0; s < S; ++s) {
        const float dj = d2s[s][j];
        float a = 0;
#pragma unroll
        for (int c = 0; c < 16; ++c) {
          g2[c] += dj * (float)h1s[s][q * 16 + c];
          a += w2s[q * 16 + c][j] * d2s[s][q * 16 + c];
        }
        a = quad_sum(a);
        if (s == q) dh1 = a;
      }
      const float d1 = dh1 * gelu_grad((float)z1);
      if (q < S) {
        gb1 += d1;
        d1s[q][j] = d1;
      }
      __syncthreads();
#pragma unroll
      for (int s = 0; s < S; ++s)
#pragma unroll
        for (int c = 0; c < 4; ++c) g1[c] += d1s[s][j] * xs[s][q * 4 + c];
    }
    __syncthreads();  // xs, h1s and red are free again
  }
  if constexpr (GRAD) {
    float* g = partials + (size_t)blockIdx.x * kStride;
    *reinterpret_cast<float4*>(g + kW1 + j * kIn + q * 4) = make_float4(g1[0], g1[1], g1[2], g1[3]);
#pragma unroll
    for (int c = 0; c < 4; ++c)
      *reinterpret_cast<float4*>(g + kW2 + j * kHid + q * 16 + 4 * c) =
          make_float4(g2[4 * c], g2[4 * c + 1], g2[4 * c + 2], g2[4 * c + 3]);
    gb1 = quad_sum(gb1);
    gb2 = quad_sum(gb2);
    g3 = quad_sum(g3);
    gb3 = quad_sum(gb3);
    loss = quad_sum(loss);
    if (q == 0) {
      g[kB1 + j] = gb1;
      g[kB2 + j] = gb2;
      g[kW3 + j] = g3;
      if (j == 0) {
        g[kB3] = gb3;
        g[kParams] = loss;
      }
    }
  }
}

// Column sums of the partials in a fixed order, 64 columns per CTA: the
// gradient to `grad` (pinned host memory; may be null) and the loss to `loss`;
// with P the gradient is applied by Adam (Kingma & Ba, ICLR 2015, with bias
// correction) instead.
__global__ void __launch_bounds__(256) mlp_reduce_kernel(const float* partials, int rows,
                                                         float* grad, float* loss, float* P,
                                                         float* m, float* v, float lr, float b1,
                                                         float b2, float eps, float c1, float c2) {
  __shared__ float sh[4][64];
  const int p = blockIdx.x * 64 + (threadIdx.x & 63), g = threadIdx.x >> 6;
  float s = 0;
  if (p <= kParams) {
#pragma unroll 8
    for (int r = g; r < rows; r += 4) s += partials[(size_t)r * kStride + p];
  }
  sh[g][threadIdx.x & 63] = s;
  __syncthreads();
  if (g != 0 || p > kParams) return;
  const int k = threadIdx.x;
  const float gp = (sh[0][k] + sh[1][k]) + (sh[2][k] + sh[3][k]);
  if (p == kParams) {
    if (loss) *loss = gp;
    return;
  }
  if (grad) grad[p] = gp;
  if (!P) return;
  const float mp = b1 * m[p] + (1 - b1) * gp;
  const float vp = b2 * v[p] + (1 - b2) * gp * gp;
  m[p] = mp;
  v[p] = vp;
  P[p] -= lr * (mp / c1) / (sqrtf(vp / c2) + eps);
}

}  // namespace

int mlp_param_count() { return kParams; }
int mlp_input_count() { return kIn; }

namespace {

// Samples per CTA: one each while they fit the GPU at a time, then four at a
// time on at most one CTA per SM (of a B200: the split also says which sums are
// FP64, so it does not depend on the device).
MlpGrid mlp_grid(int batch) {
  constexpr int kSMs = 148;
  if (batch <= kSMs) return MlpGrid{1, 1, batch};
  const int per = 4 * ((batch + 4 * kSMs - 1) / (4 * kSMs));
  return MlpGrid{4, per, (batch + per - 1) / per};
}

}  // namespace

size_t mlp_partials(int batch) { return (size_t)mlp_grid(batch).ctas * kStride; }

cudaError_t launch_mlp(const float* P, const float* X, const float* Y, int batch, float* out,
                       float* partials, cudaStream_t st) {
  if (batch <= 0) return cudaSuccess;
  const MlpGrid g = mlp_grid(batch);
  if (partials && g.samples == 1)
    mlp_kernel<1, true><<<g.ctas, kThreads, 0, st>>>(P, X, Y, batch, g.per_cta, out, partials);
  else if (partials)
    mlp_kernel<4, true><<<g.ctas, kThreads, 0, st>>>(P, X, Y, batch, g.per_cta, out, partials);
  else if (g.samples == 1)
    mlp_kernel<1, false><<<g.ctas, kThreads, 0, st>>>(P, X, Y, batch, g.per_cta, out, partials);
  else
    mlp_kernel<4, false><<<g.ctas, kThreads, 0, st>>>(P, X, Y, batch, g.per_cta, out, partials);
  return cudaGetLastError();
}

cudaError_t launch_mlp_reduce(const float* partials, int batch, float* grad, float* loss,
                              cudaStream_t st) {
  mlp_reduce_kernel<<<(kParams + 64) / 64, 256, 0, st>>>(partials, mlp_grid(batch).ctas, grad,
                                                         loss, nullptr, nullptr, nullptr, 0, 0, 0,
                                                         0, 1, 1);
  return cudaGetLastError();
}

cudaError_t launch_mlp_adam(const float* partials, int batch, float* loss, float* P, float* m,
                            float* v, float lr, float b1, float b2, float eps, int step,
                            cudaStream_t st) {
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  mlp_reduce_kernel<<<(kParams + 64) / 64, 256, 0, st>>>(partials, mlp_grid(batch).ctas, nullptr,
                                                         loss, P, m, v, lr, b1, b2, eps, c1, c2);
  return cudaGetLastError();
}

}  // namespace dsgdpp
