// loss_rows.cuh -- the loss kernel of FP32 and BF16 factors (squared errors of
// entries, many lanes per row) and the sums that all loss kernels share.  See
// kernels_loss.cu.
#pragma once

#include "kernels.cuh"

namespace dsgdpp {

// Lanes, vectors per lane and words per vector of the FP32 / BF16 kernels.
// Rows of whole 32-byte vectors (and bases on 32 bytes) are read with 32-byte
// loads, others with 16-byte ones; in both, up to 128 bytes of a row per
// instruction and up to four vectors per lane before more lanes share a row.
struct LossShape {
  int lanes, vecs, words;
};
// The loss kernel of a mapping, for rows whose rank is a whole number of vectors
// or (mask) not; null where there is none.
void* loss_kernel_fp32(LossShape s, bool mask);
void* loss_kernel_fp32_long(LossShape s, bool mask);
void* loss_kernel_bf16(LossShape s, bool mask);
void* loss_kernel_bf16_long(LossShape s, bool mask);

namespace {

__device__ __forceinline__ double block_reduce(double v, double* sh) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(kFullMask, v, off);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  double t = 0;
  if (warp == 0) {
    t = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t += __shfl_xor_sync(kFullMask, t, off);
  }
  return t;  // valid in thread 0
}

__device__ __forceinline__ double block_max(double v, double* sh) {
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = fmax(v, __shfl_xor_sync(kFullMask, v, off));
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) sh[warp] = v;
  __syncthreads();
  double t = 0;
  if (warp == 0) {
    t = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.0;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) t = fmax(t, __shfl_xor_sync(kFullMask, t, off));
  }
  return t;  // valid in thread 0
}

// f * 2^-896 as a double, exactly for finite f, built from the float's bits with integer
// operations: the 8-bit exponent field and 23-bit fraction move into the low
// bits of the double's exponent field and the top of its fraction, so an
// exponent field e reads as 2^(e-1023) where the float meant 2^(e-127) --
// for normal and subnormal floats alike.  The conversion unit (16 values per
// clock and SM), which bounds the loss kernels, then converts only W.  (The
// arithmetic shift brings the sign along; the mask clears its copies.)  An
// infinity or NaN, exponent field 255, reads as a number of 2^128 to 2^129: the
// loss of factors whose H alone is not finite is.  Finding such elements takes
// one more operation per element of H; tried as an FP32 multiply-add by zero it
// cost 6% at rank 32 and 42% at rank 256.
__device__ __forceinline__ double f32_scaled(uint32_t b) {
  return __hiloint2double(((int)b >> 3) & (int)0x8fffffffu, (int)(b << 29));
}

// ---- squared errors, FP32 / BF16 factors ------------------------------------------
// A warp takes 32 consecutive entries (one index load per lane, the next 32
// loaded while these are summed) and walks them in L rounds of 32 / L, L lanes
// per entry with V vectors of the W row and of the H column each.  Products of
// two floats are exact in FP64; each lane sums its elements in z order.  The
// lane sums of the L rounds are then added by a transposing butterfly -- each
// step halves the values a lane holds -- that leaves every lane with the inner
// product of one entry, so the difference and its square are formed once per
// 32 entries on all lanes.
//
// L is chosen so that one load instruction covers 128 contiguous bytes of a
// row (4 lanes of 32 bytes where rows are whole 32-byte vectors): an L1 lookup
// handles one line at a time, and 16 rows of 32 bytes per instruction cost
// four times the lookups.
//
// Bound: no single unit -- on 20M Zipf(1.1) entries at rank 32 the L1 data
// path is 69% busy, instruction issue 51%, the conversion unit 48% and the
// integer pipe 47%.  Measured there against 2 lanes with four 16-byte vectors, a full
// butterfly per round and zero-filled, predicated loads (ms per loss without
// factor terms): FP32 rank 10 0.40 -> 0.22, 16 0.33 -> 0.20, 32 0.45 -> 0.31,
// 50 0.75 -> 0.61, 64 0.73 -> 0.55, 128 1.47 -> 1.05; BF16 rank 32 0.39 ->
// 0.27, 64 0.57 -> 0.48, 128 1.05 -> 0.83.  100M entries at rank 32: 2.21 ->
// 1.54 ms.
template <int N>
struct Words {
  uint32_t w[N];
};
template <int N>
__device__ __forceinline__ Words<N> load_words(const void* p) {
  Words<N> r;
  if constexpr (N == 8) {
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r.w[0]), "=r"(r.w[1]), "=r"(r.w[2]), "=r"(r.w[3]), "=r"(r.w[4]), "=r"(r.w[5]),
          "=r"(r.w[6]), "=r"(r.w[7])
        : "l"(p));
  } else {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    r.w[0] = v.x; r.w[1] = v.y; r.w[2] = v.z; r.w[3] = v.w;
  }
  return r;
}
// element e of a vector, as the bits of a float
template <typename T, int N>
__device__ __forceinline__ uint32_t elem_bits(const Words<N>& v, int e) {
  if constexpr (sizeof(T) == 4) return v.w[e];
  else return (e & 1) ? v.w[e / 2] & 0xffff0000u : v.w[e / 2] << 16;
}

// vector words of each side that a lane has in flight (8: 0.27 against 0.26 ms
// at BF16 rank 32; 32 spill, or halve the warps)
constexpr int kLossWords = 16;
// BF16 rows of 32 lanes with four vectors (ranks from 769 that fill no 32-byte
// vector) take 8, and test for a ragged rank at run time (below) whether it is
// or not: the sums of 32 lanes leave no registers for more.  2M entries, 16
// words / 8 / 8 and the test: rank 776 1063 / - / 971 us, 1000 1110 / 1144 / 975
// (16-byte loads, a butterfly per round: 997).  FP32 is slower so (rank 508: 473
// -> 709).
template <typename T, int L, int V>
constexpr bool kTight = sizeof(T) == 2 && L == 32 && V == 4;
// From 8 lanes on the masked instances test for a ragged rank at run time too.
// It always is, but the branch keeps the unpacking and masking of a row's last
// vector behind that of the others, out of the registers that the sums need.
// 2M entries, us, masked at once / behind the test: FP32 rank 130 225 / 197, 250
// 390 / 246, 258 470 / 393, 450 816 / 500, 511 597 / 490; BF16 rank 599 707 / 633,
// 740 735 / 642 (260 306 / 320).
template <typename T, int L, int V, bool MASK>
constexpr bool kLateMask = kTight<T, L, V> || (MASK && L >= 8);

// The squared error of 32 entries (nrec of them exist; the others name rows
// that an entry names: no other row of W or H need be memory of the caller's),
// one entry per lane in the end.  A lane whose vector starts past
// the rank reads the row's first one and drops it; with MASK (the rank is no
// whole number of vectors) a vector that reaches past the rank is masked there:
// a caller's padding may hold anything, and a context's holds NaN once an
// update was infinite.
template <typename T, int L, int V, int N, bool MASK>
__device__ __forceinline__ double squares32(uint32_t my_row, uint32_t my_col, float my_val,
                                            uint32_t nrec, const T* W, const T* H, uint32_t r,
                                            uint32_t rp) {
  constexpr int NG = 32 / L;                   // entries per round
  constexpr int EPV = N * 4 / (int)sizeof(T);  // elements per vector
  // vectors of each side that a lane has in flight: U rounds of a row's V, or
  // C of one round's
  constexpr int F = (kTight<T, L, V> ? 8 : kLossWords) / N;
  constexpr int C = V < F ? V : F;
  constexpr int U = F / V < 1 ? 1 : F / V < L ? F / V : L;
  const uint32_t lane = threadIdx.x & 31u, grp = lane / L, gl = lane % L;
  // this lane's last vector: only it may start past the rank, or reach past it
  const uint32_t z_last = (uint32_t)((V - 1) * L + gl) * EPV;
  const bool last_in = z_last < r;
  const uint32_t last_at = last_in ? z_last : 0;
  double ip[L];
#pragma unroll
  for (int t0 = 0; t0 < L; t0 += U) {
#pragma unroll
    for (int u = 0; u < U; ++u) ip[t0 + u] = 0;
#pragma unroll
    for (int v0 = 0; v0 < V; v0 += C) {
      Words<N> wv[U][C], hv[U][C];
      if (t0 + v0) asm volatile("" ::: "memory");  // no more loads ahead than planned
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const uint32_t ri = (t0 + u) * NG + grp;
        const T* w = W + (size_t)__shfl_sync(kFullMask, my_row, ri) * rp;
        const T* h = H + (size_t)__shfl_sync(kFullMask, my_col, ri) * rp;
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (v0 + c >= V) continue;
          const uint32_t at = v0 + c == V - 1 ? last_at : (uint32_t)((v0 + c) * L + gl) * EPV;
          wv[u][c] = load_words<N>(w + at);
          hv[u][c] = load_words<N>(h + at);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        double s = ip[t0 + u];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          if (v0 + c >= V) continue;
          if ((kLateMask<T, L, V, MASK> ? r % EPV != 0 : MASK) && v0 + c == V - 1) {
#pragma unroll
            for (int k = 0; k < N; ++k) {
              // whole words past the rank, and the upper half of one that ends it
              const uint32_t z = z_last + k * (4 / (uint32_t)sizeof(T));
              const uint32_t keep = z >= r ? 0u : z + 4 / (uint32_t)sizeof(T) > r ? 0xffffu : ~0u;
              wv[u][c].w[k] &= keep;  // H's part reads as finite whatever it holds
            }
          }
          const double before = s;
          // The product of two floats is exact in FP64, so the fused
          // multiply-add rounds exactly like the separate add.  The sum is
          // formed with H scaled by 2^-896 and scaled back once: a power of
          // two, so it rounds exactly as unscaled wherever the scaled terms
          // stay normal doubles (magnitudes of 2^-126 and up; below that the
          // absolute error stays under 2^-178).
#pragma unroll
          for (int e = 0; e < EPV; ++e)
            s = fma((double)__uint_as_float(elem_bits<T>(wv[u][c], e)),
                    f32_scaled(elem_bits<T>(hv[u][c], e)), s);
          if (v0 + c == V - 1 && !last_in) s = before;
        }
        ip[t0 + u] = s;
      }
    }
  }
#pragma unroll
  for (int off = L / 2; off > 0; off >>= 1) {
    const bool up = (gl & off) != 0;
#pragma unroll
    for (int k = 0; k < off; ++k) {
      const double keep = up ? ip[k + off] : ip[k], send = up ? ip[k] : ip[k + off];
      ip[k] = __dadd_rn(keep, __shfl_xor_sync(kFullMask, send, off));
    }
  }
  // this lane's entry: round gl of its group
  const uint32_t ri = gl * NG + grp;
  const float x = __shfl_sync(kFullMask, my_val, ri);
  const double diff = __dsub_rn((double)x, __dmul_rn(ip[0], 0x1p896));
  return ri < nrec ? __dmul_rn(diff, diff) : 0.0;
}

// Entries [begin, end) dealt to warps warp, warp + nwarps, ... 32 at a time.
template <typename T, int L, int V, int N, bool MASK>
__device__ __forceinline__ double nzsl_lanes(const LossArgs& a, uint64_t begin, uint64_t end,
                                             uint64_t warp, uint64_t nwarps) {
  const uint32_t lane = threadIdx.x & 31u;
  const T* W = static_cast<const T*>(a.W);
  const T* H = static_cast<const T*>(a.H);
  const float* val = static_cast<const float*>(a.val);
  double acc = 0;
  uint64_t base = begin + warp * 32;
  uint32_t n_row = 0, n_col = 0;  // of a lane without an entry: those of an earlier one
  float n_val = 0;
  if (base < end) {
    const uint64_t k = min(base + lane, end - 1);
    n_row = a.row[k];
    n_col = a.col[k];
    n_val = val[k];
  }
  for (; base < end; base += nwarps * 32) {
    const uint32_t my_row = n_row, my_col = n_col;
    const float my_val = n_val;
    // the next 32 entries travel while these are summed
    const uint64_t nk = base + nwarps * 32 + lane;
    if (nk < end) {
      n_row = a.row[nk];
      n_col = a.col[nk];
      n_val = val[nk];
    }
    const uint32_t nrec = (uint32_t)min((uint64_t)32, end - base);
    acc = __dadd_rn(acc, squares32<T, L, V, N, MASK>(my_row, my_col, my_val, nrec, W, H, a.r,
                                                     a.rp));
  }
  return acc;
}

// Squares of the elements of one 16-byte vector, added in element order.
// The square of a float is exact in FP64, so the fused multiply-add rounds as
// the separate add does; FP64 elements keep the separate multiply and add.
template <typename T>
__device__ __forceinline__ double add_squares(double acc, const uint4& v) {
  typename Elem<T>::C f[Elem<T>::VW];
  Elem<T>::unpack(v, f);
#pragma unroll
  for (int e = 0; e < Elem<T>::VW; ++e) {
    if constexpr (sizeof(T) == 8) {
      acc = __dadd_rn(acc, __dmul_rn(f[e], f[e]));
    } else {
      const double x = (double)f[e];
      acc = fma(x, x, acc);
    }
  }
  return acc;
}

// Sum of squares of `count` factor elements (L2Loss, mf/loss/l2.h) dealt to
// threads tid, tid + stride, ...: 16-byte loads, four in flight per thread; the
// elements past the last whole vector (none when rows are padded to a vector)
// go to the first threads.
template <typename T>
__device__ __forceinline__ double sum_squares(const T* X, uint64_t count, uint64_t tid,
                                              uint64_t stride) {
  constexpr int VW = Elem<T>::VW;
  const uint4* V = reinterpret_cast<const uint4*>(X);
  const uint64_t nvec = count / VW;
  double acc = 0;
  uint64_t k = tid;
  for (; k + 3 * stride < nvec; k += 4 * stride) {
    uint4 v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) v[u] = __ldcs(V + k + u * stride);
#pragma unroll
    for (int u = 0; u < 4; ++u) acc = add_squares<T>(acc, v[u]);
  }
  for (; k < nvec; k += stride) acc = add_squares<T>(acc, __ldcs(V + k));
  for (uint64_t j = nvec * VW + tid; j < count; j += stride) {
    const double x = (double)(typename Elem<T>::C)X[j];
    acc = __dadd_rn(acc, __dmul_rn(x, x));
  }
  return acc;
}

// Lanes that share a row of `vpr` 16-byte vectors in the row-wise sums: the
// power of two that covers it (at most 32), so rows are read coalesced.
// The row-wise sums below read with the default cache policy: they run between
// epochs, and evict-first loads would take the factors out of L2 that the next
// epoch starts on -- which is how stale its first reads are, and moved the loss
// trace (3M entries, rank 50, ten epochs with this loss after each: by 1.4
// times what one run differs by from another).
__device__ __forceinline__ uint32_t row_lanes(uint32_t vpr) {
  uint32_t l = 1;
  while (l < vpr && l < 32) l <<= 1;
  return l;
}

// sum_i cnt[i] |X_i|^2 (Nzl2Loss, mf/loss/nzl2.h).  FP64 rows are summed by a
// thread each, in z order, and then weighed, as the reference does.  FP32 and
// BF16 rows are dealt to groups of lanes; each lane weighs its own share of a
// row, four rows in flight.
template <typename T>
__device__ __forceinline__ double weighted_squares(const T* X, uint64_t rows, uint32_t rp,
                                                   const uint32_t* cnt, uint64_t tid,
                                                   uint64_t stride) {
  const uint32_t vpr = rp / Elem<T>::VW, lanes = row_lanes(vpr), gl = (uint32_t)tid & (lanes - 1);
  const uint4* V = reinterpret_cast<const uint4*>(X);
  const uint64_t groups = stride / lanes;
  double acc = 0;
  if constexpr (sizeof(T) == 8) {
    for (uint64_t i = tid; i < rows; i += stride) {
      double row = 0;
#pragma unroll 4
      for (uint32_t v = 0; v < vpr; ++v) row = add_squares<T>(row, V[i * vpr + v]);
      acc = __dadd_rn(acc, __dmul_rn((double)cnt[i], row));
    }
    return acc;
  }
  for (uint64_t i0 = tid / lanes; i0 < rows; i0 += 4 * groups) {
    for (uint32_t v = gl; v < vpr; v += lanes) {
      uint4 x[4];
      double c[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint64_t i = i0 + u * groups;
        x[u] = make_uint4(0, 0, 0, 0);
        c[u] = 0;
        if (i < rows) {
          x[u] = V[i * vpr + v];
          c[u] = (double)cnt[i];
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) acc = fma(c[u], add_squares<T>(0.0, x[u]), acc);
    }
  }
  return acc;
}

// CTAs of 256 threads per SM that the loss kernels' registers are bounded for,
// by the vector registers a lane holds (N words, V vectors of each side): three
// at rank 64 or 128 spill (0.58 and 1.12 against 0.55 and 1.05 ms), two at rank
// 32 leave the SM idle (0.33 against 0.31 ms).  The sums of 16 or 32 lanes
// spill at three, and are faster so all the same: with two and 8 words in
// flight, which need no spills, 2M entries take 578 instead of 396 us at FP32
// rank 300 and 810 instead of 680 at BF16 rank 600.
constexpr int loss_ctas(int N, int V) { return N * V < 16 ? 3 : 2; }

// ---- one launch per loss --------------------------------------------------------
// Sums of up to K values per thread over the grid: each CTA writes its sums,
// and the CTA that finishes last adds all CTAs' in a fixed order -- every
// result is deterministic -- and writes them to `out`, which may be pinned host
// memory, so a loss is one launch and needs no copy.  MAXK: that value is a
// maximum instead of a sum.
template <int K, int MAXK = -1>
__device__ void grid_sums(double (&v)[K], double* partials, uint32_t* ticket, double* out) {
  __shared__ double sh[32];
  __shared__ bool last;
  auto reduce = [&](double x, bool is_max) {
    const double t = is_max ? block_max(x, sh) : block_reduce(x, sh);
    __syncthreads();
    return t;
  };
#pragma unroll
  for (int k = 0; k < K; ++k) {
    const double t = reduce(v[k], k == MAXK);
    if (threadIdx.x == 0) partials[(size_t)k * gridDim.x + blockIdx.x] = t;
  }
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
#pragma unroll
  for (int k = 0; k < K; ++k) {
    double x = 0;
    for (uint32_t i = threadIdx.x; i < gridDim.x; i += blockDim.x) {
      const double p = __ldcg(partials + (size_t)k * gridDim.x + i);
      x = k == MAXK ? fmax(x, p) : __dadd_rn(x, p);
    }
    const double t = reduce(x, k == MAXK);
    if (threadIdx.x == 0) out[k] = t;
  }
  if (threadIdx.x == 0) {
    *ticket = 0;  // for the next launch
    __threadfence_system();
  }
}

// This CTA's share of the terms of the L2 (1) or nonzero-weighted L2 (2) loss
// of W and of H as v[1], v[2].
template <typename T>
__device__ __forceinline__ void loss_terms(const LossArgs& a, double (&v)[3]) {
  const uint64_t tid = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const T* W = static_cast<const T*>(a.W);
  const T* H = static_cast<const T*>(a.H);
  v[1] = a.reg == 1 ? sum_squares<T>(W, a.m * a.rp, tid, stride)
                    : weighted_squares<T>(W, a.m, a.rp, a.cnt1, tid, stride);
  v[2] = a.reg == 1 ? sum_squares<T>(H, a.n * a.rp, tid, stride)
                    : weighted_squares<T>(H, a.n, a.rp, a.cnt2, tid, stride);
}

// The factor terms beside a CTA's squared errors `e`, and their sums over the
// grid: a function of its own, one per type.  Inlined into every mapping it made
// those of ranks up to 128 spill.
template <typename T>
__device__ __noinline__ void loss_with_terms(const LossArgs& a, double e) {
  double v[3] = {e, 0, 0};
  loss_terms<T>(a, v);
  grid_sums<3>(v, a.partials, a.ticket, a.out);
}

template <typename T>
__device__ __forceinline__ void loss_finish(const LossArgs& a, double e) {
  if (a.ticket && a.reg) {
    loss_with_terms<T>(a, e);
  } else if (a.ticket) {
    double v[1] = {e};
    grid_sums<1>(v, a.partials, a.ticket, a.out);
  } else {
    __shared__ double sh[32];
    const double t = block_reduce(e, sh);
    if (threadIdx.x == 0) a.partials[blockIdx.x] = t;
  }
}

template <typename T, int L, int V, int N, bool MASK>
__global__ void __launch_bounds__(256, loss_ctas(N, V))
    loss_kernel(const __grid_constant__ LossArgs a) {
  const uint32_t per = blockDim.x >> 5, w = threadIdx.x >> 5;
  // entries [begin, end): of the whole grid, or of CTA k in range k
  uint64_t begin = 0, end = a.nnz, warp = (uint64_t)blockIdx.x * per + w;
  uint64_t nwarps = (uint64_t)gridDim.x * per;
  if (a.chunks) {
    begin = a.chunks[blockIdx.x].begin;
    end = a.chunks[blockIdx.x].end;
    warp = w;
    nwarps = per;
  }
  loss_finish<T>(a, nzsl_lanes<T, L, V, N, MASK>(a, begin, end, warp, nwarps));
}

}  // namespace
}  // namespace dsgdpp
