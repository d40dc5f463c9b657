// kernels_loss.cu -- FP64 loss reductions of DSGD++ on sm_100a.
//
// Reference: nzsl (mf/loss/nzsl.h:29-52), l2 (mf/loss/l2.h:39-48) and nzl2
// (mf/loss/nzl2.h:29-87), summed over blocks (mf/matrix/op/sum.h:27-30).
// With FP64 factors every term is formed exactly as the reference forms it
// (the inner product summed in z order, no FMA contraction).  With FP32/BF16
// factors a group of lanes shares an entry (coalesced row loads); products of
// floats are exact in FP64 and only the order of the inner product's additions
// differs.  Terms are reduced by a fixed two-level tree (per-CTA partials,
// then one CTA), so every result is deterministic run to run.
#include "loss_rows.cuh"

namespace dsgdpp {
namespace {

// FP64 factors: one thread per entry, the inner product in z order (as the
// reference forms it, no contraction) over entries first, first + stride, ...
// Bound by the lookups of 32 rows per load instruction, so a load takes 16
// bytes of a row: with the second element of a vector under a condition each
// load became two of 8 bytes (2M entries, rank 10: 62 -> 51 us, 32: 267 -> 152,
// 256: 1982 -> 1061 us per loss).
__device__ __forceinline__ double nzsl_exact(const uint32_t* row, const uint32_t* col,
                                             const double* val, const double* W, const double* H,
                                             uint32_t r, uint32_t rp, uint64_t first,
                                             uint64_t end, uint64_t stride) {
  double acc = 0;
  for (uint64_t k = first; k < end; k += stride) {
    const double* w = W + (size_t)row[k] * rp;
    const double* h = H + (size_t)col[k] * rp;
    double ip = 0;
    uint32_t z = 0;
    for (; z + 1 < r; z += 2) {
      const double2 a = *reinterpret_cast<const double2*>(w + z);
      const double2 b = *reinterpret_cast<const double2*>(h + z);
      ip = __dadd_rn(ip, __dmul_rn(a.x, b.x));
      ip = __dadd_rn(ip, __dmul_rn(a.y, b.y));
    }
    if (z < r) ip = __dadd_rn(ip, __dmul_rn(w[z], h[z]));
    const double diff = __dsub_rn(val[k], ip);
    acc = __dadd_rn(acc, __dmul_rn(diff, diff));
  }
  return acc;
}

// ---- per-problem (segmented) reductions of the batched form ----------------------
// One CTA per chunk of a problem's range; owner_sums then adds each problem's
// chunk partials in chunk order, so every per-problem sum is deterministic.
// Sums of squares of ranges of W (the first nw) and of H.
template <typename T>
__global__ void __launch_bounds__(256) sumsq_chunks_kernel(const RangeChunk* chunks, uint32_t nw,
                                                           const T* W, const T* H,
                                                           double* partials) {
  __shared__ double sh[32];
  const RangeChunk c = chunks[blockIdx.x];  // whole rows or pieces of 2^14 elements: whole vectors
  const double acc = sum_squares<T>((blockIdx.x < nw ? W : H) + c.begin, c.end - c.begin,
                                    threadIdx.x, blockDim.x);
  const double t = block_reduce(acc, sh);
  if (threadIdx.x == 0) partials[blockIdx.x] = t;
}
// out[o.out] = the sum of partials [o.begin, o.end), in a fixed order
__global__ void __launch_bounds__(256) owner_sums_kernel(const double* partials,
                                                         const OwnerRange* owners, double* out) {
  __shared__ double sh[32];
  const OwnerRange o = owners[blockIdx.x];
  double acc = 0;
  for (uint32_t k = o.begin + threadIdx.x; k < o.end; k += blockDim.x)
    acc = __dadd_rn(acc, partials[k]);
  const double t = block_reduce(acc, sh);
  if (threadIdx.x == 0) out[o.out] = t;
}

__global__ void __launch_bounds__(256) loss_exact_kernel(const __grid_constant__ LossArgs a) {
  uint64_t first = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x, end = a.nnz;
  uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  if (a.chunks) {
    const RangeChunk c = a.chunks[blockIdx.x];
    first = c.begin + threadIdx.x;
    end = c.end;
    stride = blockDim.x;
  }
  loss_finish<double>(a, nzsl_exact(a.row, a.col, static_cast<const double*>(a.val),
                                    static_cast<const double*>(a.W),
                                    static_cast<const double*>(a.H), a.r, a.rp, first, end,
                                    stride));
}

LossShape loss_shape(int precision, uint32_t r, uint32_t rp, const void* W, const void* H) {
  const uint32_t es = precision == kFp32 ? 4 : 2;
  const bool wide = rp * es % 32 == 0 &&
                    ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(H)) & 31u) == 0;
  LossShape s;
  s.words = wide ? 8 : 4;
  const uint32_t nv = (r * es + 4 * s.words - 1) / (4 * s.words);  // vectors up to the rank
  s.lanes = nv == 1 ? 1 : nv == 2 && wide ? 2 : 4;
  while (nv > 4u * s.lanes) s.lanes *= 2;
  s.vecs = (nv + s.lanes - 1) / s.lanes;
  return s;
}

void* loss_fn(int precision, uint32_t r, uint32_t rp, const void* W, const void* H) {
  if (precision == kFp64) return reinterpret_cast<void*>(&loss_exact_kernel);
  const LossShape s = loss_shape(precision, r, rp, W, H);
  const bool mask = r * (precision == kFp32 ? 4u : 2u) % (4u * s.words) != 0;
  const bool longer = s.lanes > 4;
  if (precision == kFp32) return longer ? loss_kernel_fp32_long(s, mask) : loss_kernel_fp32(s, mask);
  return longer ? loss_kernel_bf16_long(s, mask) : loss_kernel_bf16(s, mask);
}

// Sum over rows of |X_i - Xold_i| (v[0]) and their maximum (v[1]): groups of
// lanes read a row coalesced, two rows in flight.
template <typename T>
__device__ __forceinline__ void row_moves(const T* X, const T* Xold, uint64_t rows, uint32_t rp,
                                          double (&out)[2]) {
  using C = typename Elem<T>::C;
  constexpr int VW = Elem<T>::VW;
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint32_t vpr = rp / VW, lanes = row_lanes(vpr), gl = (uint32_t)tid & (lanes - 1);
  const uint64_t groups = (uint64_t)gridDim.x * blockDim.x / lanes;
  const uint4* A = reinterpret_cast<const uint4*>(X);
  const uint4* B = reinterpret_cast<const uint4*>(Xold);
  for (uint64_t k0 = 0; k0 < rows; k0 += 2 * groups) {
    double s[2] = {0, 0};
    for (uint32_t v = gl; v < vpr; v += lanes) {
      uint4 x[2], y[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const uint64_t i = k0 + u * groups + tid / lanes;
        x[u] = y[u] = make_uint4(0, 0, 0, 0);
        if (i < rows) {
          x[u] = A[i * vpr + v];
          y[u] = B[i * vpr + v];
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        C a[VW], b[VW];
        Elem<T>::unpack(x[u], a);
        Elem<T>::unpack(y[u], b);
#pragma unroll
        for (int e = 0; e < VW; ++e) {
          const double d = (double)a[e] - (double)b[e];
          s[u] += d * d;
        }
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      for (uint32_t off = lanes / 2; off > 0; off >>= 1)
        s[u] += __shfl_xor_sync(kFullMask, s[u], off);
      if (gl == 0) {
        const double nrm = sqrt(s[u]);  // rows past the end add 0
        out[0] += nrm;
        out[1] = fmax(out[1], nrm);
      }
    }
  }
}

template <typename T>
__global__ void __launch_bounds__(256) update_norms_kernel(const T* W, const T* W0, uint64_t m,
                                                           const T* H, const T* H0, uint64_t n,
                                                           uint32_t rp, double* partials,
                                                           uint32_t* ticket, double* out) {
  double v[2] = {0, 0};
  row_moves<T>(W, W0, m, rp, v);
  row_moves<T>(H, H0, n, rp, v);
  grid_sums<2, 1>(v, partials, ticket, out);
}

__global__ void __launch_bounds__(1024) sum_partials_kernel(const double* partials, uint32_t count,
                                                            double* out) {
  __shared__ double sh[32];
  double acc = 0;
  for (uint32_t k = threadIdx.x; k < count; k += blockDim.x) acc = __dadd_rn(acc, partials[k]);
  const double t = block_reduce(acc, sh);
  if (threadIdx.x == 0) out[0] = t;
}

}  // namespace

cudaError_t load_fp32_loss_kernels() {
  cudaFuncAttributes at;
  const cudaError_t e = cudaFuncGetAttributes(&at, loss_kernel_fp32(LossShape{1, 1, 8}, false));
  if (e != cudaSuccess) return e;
  return cudaFuncGetAttributes(&at, loss_kernel_fp32_long(LossShape{8, 4, 8}, false));
}

cudaError_t launch_loss(int precision, const LossArgs& a, uint32_t grid, cudaStream_t st) {
  void* fn = loss_fn(precision, a.r, a.rp, a.W, a.H);
  if (!fn) return cudaErrorInvalidValue;
  LossArgs args = a;
  void* params[] = {&args};
  return cudaLaunchKernel(fn, dim3(grid), dim3(256), params, 0, st);
}

int loss_ctas_per_sm(int precision, uint32_t r, uint32_t rp) {
  void* fn = loss_fn(precision, r, rp, nullptr, nullptr);
  int n = 0;
  if (!fn || cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, 256, 0) != cudaSuccess) return 0;
  return n;
}

cudaError_t launch_sumsq_chunks(int precision, const RangeChunk* chunks, uint32_t nw, uint32_t nh,
                                const void* W, const void* H, double* partials, cudaStream_t st) {
  if (nw + nh == 0) return cudaSuccess;
  if (precision == kFp64)
    sumsq_chunks_kernel<double><<<nw + nh, 256, 0, st>>>(chunks, nw, (const double*)W,
                                                         (const double*)H, partials);
  else if (precision == kFp32)
    sumsq_chunks_kernel<float><<<nw + nh, 256, 0, st>>>(chunks, nw, (const float*)W,
                                                        (const float*)H, partials);
  else
    sumsq_chunks_kernel<__nv_bfloat16><<<nw + nh, 256, 0, st>>>(
        chunks, nw, (const __nv_bfloat16*)W, (const __nv_bfloat16*)H, partials);
  return cudaGetLastError();
}

cudaError_t launch_owner_sums(const double* partials, const OwnerRange* owners, uint32_t count,
                              double* out, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  owner_sums_kernel<<<count, 256, 0, st>>>(partials, owners, out);
  return cudaGetLastError();
}

cudaError_t launch_sum_partials(const double* partials, uint32_t count, double* out,
                                cudaStream_t st) {
  sum_partials_kernel<<<1, 1024, 0, st>>>(partials, count, out);
  return cudaGetLastError();
}

cudaError_t launch_update_norms(int precision, const void* W, const void* W0, uint64_t m,
                                const void* H, const void* H0, uint64_t n, uint32_t rp,
                                double* partials, uint32_t grid, uint32_t* ticket, double* out,
                                cudaStream_t st) {
  if (precision == kFp64)
    update_norms_kernel<double><<<grid, 256, 0, st>>>(
        (const double*)W, (const double*)W0, m, (const double*)H, (const double*)H0, n, rp,
        partials, ticket, out);
  else if (precision == kFp32)
    update_norms_kernel<float><<<grid, 256, 0, st>>>((const float*)W, (const float*)W0, m,
                                                     (const float*)H, (const float*)H0, n, rp,
                                                     partials, ticket, out);
  else
    update_norms_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(
        (const __nv_bfloat16*)W, (const __nv_bfloat16*)W0, m, (const __nv_bfloat16*)H,
        (const __nv_bfloat16*)H0, n, rp, partials, ticket, out);
  return cudaGetLastError();
}

}  // namespace dsgdpp
