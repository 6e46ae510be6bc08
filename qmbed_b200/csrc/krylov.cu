// Dense vector kernels for Lanczos / thick restart, reductions and the small
// FP64 Hermitian eigensolver. All reductions accumulate in FP64 through a
// fixed two-stage tree (per-block partials, then an ordered sum), so results
// do not depend on scheduling.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>

#include "device_util.cuh"
#include <cstdlib>
#include <string>

#include "krylov.cuh"

namespace qmbed {

bool dense_on_tensor_cores() {
  static const bool on = [] {
    const char* env = std::getenv("QMBED_DENSE");
    return !(env && std::string(env) == "scalar");
  }();
  return on;
}


namespace {

constexpr int kThreads = 256;
constexpr int kChunk = 8;    // columns per pass of the multi-dot
constexpr int kCombine = 4;  // outputs per pass of the combination kernel

template <typename T, bool CPLX>
__device__ inline void load(const T* __restrict__ p, uint64_t i, double& re, double& im) {
  if (CPLX) {
    re = static_cast<double>(p[2 * i]);
    im = static_cast<double>(p[2 * i + 1]);
  } else {
    re = static_cast<double>(p[i]);
    im = 0.0;
  }
}

template <typename T, bool CPLX>
__device__ inline void store(T* __restrict__ p, uint64_t i, double re, double im) {
  if (CPLX) {
    p[2 * i] = static_cast<T>(re);
    p[2 * i + 1] = static_cast<T>(im);
  } else {
    p[i] = static_cast<T>(re);
  }
}

__device__ inline double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Overlaps of a tall FP64 panel with one vector, one warp per column: each
// block stages a slab of `slab` rows of w in shared memory and its warps
// sweep the columns; every lane keeps eight independent loads in flight.
// partials[(j * G + block) * 2 + {0,1}] as for multi_dot_kernel. Bound by the
// panel's read (kept_columns: the last `keep` columns stay in the L2): 44.7 us
// on average for 1 to 100 columns of 718,146 rows, 42 with the kept columns.
constexpr int kMaxSlab = 2048;
template <bool CPLX>
__global__ void __launch_bounds__(kThreads) panel_dot_kernel(const double* __restrict__ A, uint64_t ld, int m,
                                                             const double* w, uint64_t n, int slab, int keep,
                                                             double* __restrict__ partials) {
  constexpr int W = CPLX ? 2 : 1;
  extern __shared__ __align__(16) double ws[];
  const uint64_t r0 = static_cast<uint64_t>(blockIdx.x) * slab;
  const int rows = static_cast<int>(min(static_cast<uint64_t>(slab), n - r0));
  await_previous();
  for (int t = threadIdx.x; t < rows * W; t += blockDim.x) ws[t] = __ldcg(w + r0 * W + t);
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const uint64_t G = gridDim.x;
  for (int j = threadIdx.x >> 5; j < m; j += kThreads / 32) {
    const double* q = A + static_cast<uint64_t>(j) * ld * W + r0 * W;
    double sr = 0.0, si = 0.0;
    auto sweep = [&](auto stream) {
      constexpr bool STREAM = decltype(stream)::value;
      for (int r = lane; r < rows; r += 32 * 8) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int k = r + 32 * u;
          if (k < rows) {
            if (CPLX) {
              const double2* at = reinterpret_cast<const double2*>(q) + k;
              const double2 x = STREAM ? __ldcs(at) : __ldg(at);
              const double2 y = reinterpret_cast<const double2*>(ws)[k];
              sr += x.x * y.x + x.y * y.y;
              si += x.x * y.y - x.y * y.x;
            } else {
              sr += (STREAM ? __ldcs(q + k) : __ldg(q + k)) * ws[k];
            }
          }
        }
      }
    };
    if (j < m - keep) sweep(std::true_type{});
    else sweep(std::false_type{});
    sr = warp_sum(sr);
    if (CPLX) si = warp_sum(si);
    if (lane == 0) {
      partials[(static_cast<uint64_t>(j) * G + blockIdx.x) * 2] = sr;
      partials[(static_cast<uint64_t>(j) * G + blockIdx.x) * 2 + 1] = si;
    }
  }
}

// partials[(j * G + block) * 2 + {0,1}] = sum over this block's rows of conj(A_j) w.
// With `with_self`, column m receives sum |w|^2 (computed in the first pass).
template <typename T, bool CPLX>
__global__ void __launch_bounds__(kThreads) multi_dot_kernel(const T* __restrict__ A, uint64_t ld, int m,
                                                              const T* __restrict__ w, uint64_t n,
                                                              double* __restrict__ partials, int with_self) {
  __shared__ double red[kThreads / 32][2 * kChunk];
  const int G = gridDim.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t stride = static_cast<uint64_t>(G) * blockDim.x;
  double self = 0.0;
  for (int j0 = 0; j0 < m; j0 += kChunk) {
    const int cnt = min(kChunk, m - j0);
    double ar[kChunk], ai[kChunk];
#pragma unroll
    for (int jj = 0; jj < kChunk; ++jj) ar[jj] = ai[jj] = 0.0;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
      double wr, wi;
      load<T, CPLX>(w, i, wr, wi);
      if (j0 == 0) self += wr * wr + wi * wi;
#pragma unroll
      for (int jj = 0; jj < kChunk; ++jj) {
        if (jj < cnt) {
          double xr, xi;
          load<T, CPLX>(A + (j0 + jj) * ld * (CPLX ? 2 : 1), i, xr, xi);
          ar[jj] += xr * wr + xi * wi;
          ai[jj] += xr * wi - xi * wr;
        }
      }
    }
#pragma unroll
    for (int jj = 0; jj < kChunk; ++jj) {
      double a = warp_sum(ar[jj]);
      double b = warp_sum(ai[jj]);
      if (lane == 0) {
        red[warp][2 * jj] = a;
        red[warp][2 * jj + 1] = b;
      }
    }
    __syncthreads();
    if (threadIdx.x < 2 * cnt) {
      double total = 0.0;
      for (int wv = 0; wv < kThreads / 32; ++wv) total += red[wv][threadIdx.x];
      const int j = j0 + threadIdx.x / 2;
      partials[(static_cast<uint64_t>(j) * G + blockIdx.x) * 2 + (threadIdx.x & 1)] = total;
    }
    __syncthreads();
  }
  if (with_self) {
    const double s = warp_sum(self);
    if (lane == 0) red[warp][0] = s;
    __syncthreads();
    if (threadIdx.x < 2) {
      double total = 0.0;
      if (threadIdx.x == 0)
        for (int wv = 0; wv < kThreads / 32; ++wv) total += red[wv][0];
      partials[(static_cast<uint64_t>(m) * G + blockIdx.x) * 2 + threadIdx.x] = total;
    }
  }
}

// out[t] = sum_b partials[(t/2 * G + b) * 2 + t%2]: one block per output,
// strided per-thread sums then a shared-memory tree, both in a fixed order.
constexpr int kFinishThreads = 128;
__global__ void __launch_bounds__(kFinishThreads) finish_kernel(const double* partials, int G, int count,
                                                                double* __restrict__ out) {
  const int t = blockIdx.x;
  await_previous();
  if (t >= count) return;
  const int j = t / 2, c = t & 1;
  double total = 0.0;
  for (int b = threadIdx.x; b < G; b += kFinishThreads) total += __ldcg(partials + (static_cast<uint64_t>(j) * G + b) * 2 + c);
  __shared__ double tree[kFinishThreads];
  tree[threadIdx.x] = total;
  __syncthreads();
  for (int width = kFinishThreads / 2; width > 0; width >>= 1) {
    if (threadIdx.x < width) tree[threadIdx.x] += tree[threadIdx.x + width];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[t] = tree[0];
}

// w = src - sum_j h_j A_j (src may be w); per-block partial of ||w||^2 when
// `partials` is set.
template <typename T, bool CPLX>
__global__ void __launch_bounds__(kThreads) subtract_kernel(const T* __restrict__ A, uint64_t ld, int m,
                                                             const double* __restrict__ h, const T* src, T* w,
                                                             uint64_t n, double* __restrict__ partials) {
  extern __shared__ double hs[];
  for (int t = threadIdx.x; t < 2 * m; t += blockDim.x) hs[t] = h[t];
  __syncthreads();
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  const uint64_t col = ld * (CPLX ? 2 : 1);
  double sq = 0.0;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    double wr, wi;
    load<T, CPLX>(src, i, wr, wi);
    double sr = 0.0, si = 0.0;
    // batches of kChunk independent loads keep several requests in flight per thread
    for (int j0 = 0; j0 < m; j0 += kChunk) {
      double xr[kChunk], xi[kChunk];
#pragma unroll
      for (int jj = 0; jj < kChunk; ++jj) {
        if (j0 + jj < m) load<T, CPLX>(A + (j0 + jj) * col, i, xr[jj], xi[jj]);
        else xr[jj] = xi[jj] = 0.0;
      }
#pragma unroll
      for (int jj = 0; jj < kChunk; ++jj) {
        if (j0 + jj < m) {
          const double hr = hs[2 * (j0 + jj)], hi = hs[2 * (j0 + jj) + 1];
          sr += hr * xr[jj] - hi * xi[jj];
          si += hr * xi[jj] + hi * xr[jj];
        }
      }
    }
    // norm of the value as stored (rounded to T)
    const T rr = static_cast<T>(wr - sr), ri = static_cast<T>(wi - si);
    store<T, CPLX>(w, i, static_cast<double>(rr), static_cast<double>(ri));
    if (partials) sq += static_cast<double>(rr) * static_cast<double>(rr) + (CPLX ? static_cast<double>(ri) * static_cast<double>(ri) : 0.0);
  }
  if (partials) {
    __shared__ double red[kThreads / 32];
    sq = warp_sum(sq);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
      double total = 0.0;
      for (int wv = 0; wv < kThreads / 32; ++wv) total += red[wv];
      partials[2 * blockIdx.x] = total;
      partials[2 * blockIdx.x + 1] = 0.0;
    }
  }
}

// out_k = sum_j Y[j + m k] A_j for k in [k0, k0 + kCombine).
template <typename T, bool CPLX>
__global__ void __launch_bounds__(kThreads) combine_kernel(const T* __restrict__ A, uint64_t ld, int m,
                                                            const double* __restrict__ Y, int K, int k0,
                                                            T* __restrict__ out, uint64_t ld_out, uint64_t n) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  const int cnt = min(kCombine, K - k0);
  const uint64_t col = ld * (CPLX ? 2 : 1);
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    double ar[kCombine], ai[kCombine];
#pragma unroll
    for (int kk = 0; kk < kCombine; ++kk) ar[kk] = ai[kk] = 0.0;
    for (int j0 = 0; j0 < m; j0 += kChunk) {
      double xr[kChunk], xi[kChunk];
#pragma unroll
      for (int jj = 0; jj < kChunk; ++jj) {
        if (j0 + jj < m) load<T, CPLX>(A + (j0 + jj) * col, i, xr[jj], xi[jj]);
        else xr[jj] = xi[jj] = 0.0;
      }
#pragma unroll
      for (int jj = 0; jj < kChunk; ++jj) {
        if (j0 + jj >= m) continue;
#pragma unroll
        for (int kk = 0; kk < kCombine; ++kk) {
          if (kk < cnt) {
            const uint64_t y = (static_cast<uint64_t>(k0 + kk) * m + j0 + jj) * 2;
            const double yr = __ldg(Y + y), yi = __ldg(Y + y + 1);
            ar[kk] += yr * xr[jj] - yi * xi[jj];
            ai[kk] += yr * xi[jj] + yi * xr[jj];
          }
        }
      }
    }
#pragma unroll
    for (int kk = 0; kk < kCombine; ++kk)
      if (kk < cnt) store<T, CPLX>(out + (k0 + kk) * ld_out * (CPLX ? 2 : 1), i, ar[kk], ai[kk]);
  }
}

// Real combinations on the FP64 tensor cores: out[:, k0 + q] = sum_j Re(Y[j, k0 + q]) A[:, j] for
// q < 8, one m8n8k4 DMMA per 8 rows x 4 basis columns. A warp takes tiles of
// 8 consecutive rows; lane l holds A[row 8t + l / 4][column j0 + l % 4] (four
// 64-byte column segments per MMA) and the block's Y columns come from shared
// memory (y[j][q]); D[l / 4][2 (l % 4) + h] is row 8t + l / 4 of output
// column k0 + 2 (l % 4) + h.
template <typename T>
__global__ void __launch_bounds__(kThreads) combine_mma_kernel(const T* __restrict__ A, uint64_t ld, int m,
                                                                const double* __restrict__ Y, int K, int k0,
                                                                T* __restrict__ out, uint64_t ld_out, uint64_t n) {
  extern __shared__ double ys[];  // ys[j * 8 + q] = Re Y[j, k0 + q], zero-padded to a multiple of 4 rows
  const int m4 = (m + 3) & ~3;
  for (int t = threadIdx.x; t < m4 * 8; t += blockDim.x) {
    const int j = t / 8, q = t % 8;
    ys[t] = (j < m && k0 + q < K) ? Y[(static_cast<uint64_t>(k0 + q) * m + j) * 2] : 0.0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int r = lane >> 2, kq = lane & 3;
  const uint64_t tiles = (n + 7) / 8;
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (blockDim.x >> 5);
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); t < tiles; t += warps) {
    const uint64_t row = t * 8 + r;
    const bool in = row < n;
    double c0 = 0.0, c1 = 0.0;
    for (int j0 = 0; j0 < m4; j0 += 16) {
      double a[4], b[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = j0 + 4 * u + kq;
        a[u] = (in && j < m) ? static_cast<double>(A[static_cast<uint64_t>(j) * ld + row]) : 0.0;
        b[u] = j < m4 ? ys[j * 8 + r] : 0.0;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                     : "+d"(c0), "+d"(c1)
                     : "d"(a[u]), "d"(b[u]));
    }
    const int q0 = k0 + 2 * kq;
    if (in && q0 < K) out[static_cast<uint64_t>(q0) * ld_out + row] = static_cast<T>(c0);
    if (in && q0 + 1 < K) out[static_cast<uint64_t>(q0 + 1) * ld_out + row] = static_cast<T>(c1);
  }
}

template <typename T>
__global__ void scale_kernel(T* __restrict__ w, uint64_t count, double divisor) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride)
    w[i] = static_cast<T>(static_cast<double>(w[i]) / divisor);
}

// Ritz candidates of a restart, one block each: the candidate and its action are
// divided by the candidate's norm; out[4 k ..]: |c|^2 before, Re <c, H c>,
// |H c - lambda c|^2 and |c|^2 after. A candidate whose norm is not above eps, or
// not finite, is left as it is (its norm says so).
//
// Bound by one block's reads of two columns, three times over, and by launch
// and read-back: one launch and one host synchronisation for all candidates,
// where the norm, the two scalings, the Ritz value and the residual were eight
// launches and three synchronisations for each. Measured (B200): 13.5 us at 9252
// rows; the 20-site solve of 4 pairs 8.8 -> 7.4 ms, 12,870 rows 50 -> 38 us a step.
constexpr int kCandidateThreads = 1024;
// Doubles of a column up to which one block per candidate is the faster form:
// four candidates of 92,378 gain (58 -> 50 us a step), a single one is even there
// (4.6 ms a solve either way), and its time grows with the column from then on.
constexpr uint64_t kCandidateDoubles = 1u << 17;
template <bool CPLX>
__global__ void __launch_bounds__(kCandidateThreads) ritz_candidate_kernel(double* C, double* CA, uint64_t n,
                                                                           double* __restrict__ out) {
  constexpr int W = CPLX ? 2 : 1;
  __shared__ double red[2][kCandidateThreads / 32];
  double* c = C + blockIdx.x * n * W;
  double* a = CA + blockIdx.x * n * W;
  const uint64_t count = n * W;
  // both sums over the block, in a fixed order, on every thread
  auto total = [&](double& u, double& v) {
    u = warp_sum(u);
    v = warp_sum(v);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
      red[0][threadIdx.x >> 5] = u;
      red[1][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    u = v = 0.0;
    for (int q = 0; q < kCandidateThreads / 32; ++q) {
      u += red[0][q];
      v += red[1][q];
    }
  };
  double sq = 0.0, none = 0.0;
#pragma unroll 4
  for (uint64_t i = threadIdx.x; i < count; i += kCandidateThreads) sq += c[i] * c[i];
  total(sq, none);
  const double norm = sqrt(fmax(sq, 0.0));
  double lambda = 0.0, after = 0.0, residual = 0.0;
  if (isfinite(norm) && norm > 2.220446049250313e-16) {
    // Re(conj(c) a) is the sum over both parts
#pragma unroll 4
    for (uint64_t i = threadIdx.x; i < count; i += kCandidateThreads) {
      const double x = c[i] / norm, y = a[i] / norm;
      c[i] = x;
      a[i] = y;
      lambda += x * y;
      after += x * x;
    }
    total(lambda, after);
#pragma unroll 4
    for (uint64_t i = threadIdx.x; i < count; i += kCandidateThreads) {
      const double r = a[i] - lambda * c[i];
      residual += r * r;
    }
    total(residual, none);
  }
  if (threadIdx.x == 0) {
    out[4 * blockIdx.x] = sq;
    out[4 * blockIdx.x + 1] = lambda;
    out[4 * blockIdx.x + 2] = residual;
    out[4 * blockIdx.x + 3] = after;
  }
}

template <typename T>
__global__ void scale_into_kernel(const T* __restrict__ src, T* __restrict__ dst, uint64_t count, double divisor) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride)
    dst[i] = static_cast<T>(static_cast<double>(src[i]) / divisor);
}

__global__ void widen_real_kernel(const double* __restrict__ src, double* __restrict__ dst, uint64_t n) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    dst[2 * i] = src[i];
    dst[2 * i + 1] = 0.0;
  }
}

template <typename D>
__global__ void real_part_strided_kernel(const double* __restrict__ src, D* __restrict__ dst, uint64_t n) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    dst[i] = static_cast<D>(src[2 * i]);
}

template <typename S, typename D>
__global__ void convert_kernel(const S* __restrict__ src, D* __restrict__ dst, uint64_t count) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride)
    dst[i] = static_cast<D>(src[i]);
}

// Affine LCG state after k steps: x -> a x + c (mod 2^64), by squaring.
__device__ inline uint64_t lcg_jump(uint64_t x, uint64_t k) {
  uint64_t A = 1, C = 0;                                       // accumulated map
  uint64_t a = 6364136223846793005ULL, c = 1442695040888963407ULL;  // current power
  while (k) {
    if (k & 1) {
      A = a * A;
      C = a * C + c;
    }
    c = a * c + c;
    a = a * a;
    k >>= 1;
  }
  return A * x + C;
}

// Element i takes the (i+1)-th LCG state. A block covers blockDim * per_thread
// consecutive elements; thread t takes base + t, base + t + blockDim, ...,
// advancing its state by the blockDim-step map (A, C) between them, so every
// warp store is contiguous.
template <typename T, bool CPLX>
__global__ void lcg_start_kernel(T* __restrict__ out, uint64_t n, uint64_t seed, uint64_t per_thread) {
  const uint64_t stride = blockDim.x;
  const uint64_t base = static_cast<uint64_t>(blockIdx.x) * stride * per_thread;
  const uint64_t i0 = base + threadIdx.x;
  if (i0 >= n) return;
  const uint64_t C = lcg_jump(0, stride);
  const uint64_t A = lcg_jump(1, stride) - C;  // the jump is affine: jump(x) = A x + C
  uint64_t state = lcg_jump(seed | 1ULL, i0 + 1);
  const uint64_t end = min(base + stride * per_thread, n);
  for (uint64_t i = i0; i < end; i += stride) {
    const uint64_t mantissa = state >> 11;
    const double value = static_cast<double>(mantissa) / 9007199254740992.0 - 0.5;
    store<T, CPLX>(out, i, value, 0.0);
    state = A * state + C;
  }
}

template <typename T, bool CPLX>
__global__ void __launch_bounds__(kThreads) residual_kernel(const T* __restrict__ y, const T* __restrict__ x,
                                                             double lambda, uint64_t n,
                                                             double* __restrict__ partials) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  double sq = 0.0;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    double yr, yi, xr, xi;
    load<T, CPLX>(y, i, yr, yi);
    load<T, CPLX>(x, i, xr, xi);
    const double dr = yr - lambda * xr, di = yi - lambda * xi;
    sq += dr * dr + di * di;
  }
  __shared__ double red[kThreads / 32];
  sq = warp_sum(sq);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sq;
  __syncthreads();
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int wv = 0; wv < kThreads / 32; ++wv) total += red[wv];
    partials[2 * blockIdx.x] = total;
    partials[2 * blockIdx.x + 1] = 0.0;
  }
}

// --- scans and reductions used by assembly -------------------------------------------
constexpr int kScanItems = 4;

__global__ void scan_block_totals_kernel(const uint32_t* __restrict__ counts, uint64_t n,
                                         uint64_t* __restrict__ totals) {
  const uint64_t base = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * kScanItems;
  uint32_t local = 0;
  for (int k = 0; k < kScanItems; ++k)
    if (base + k < n) local += counts[base + k];
  uint32_t total = block_reduce_sum_u32(local);
  if (threadIdx.x == 0) totals[blockIdx.x] = total;
}

template <typename IDX>
__global__ void scan_write_kernel(const uint32_t* __restrict__ counts, uint64_t n,
                                  const uint64_t* __restrict__ block_offsets, IDX* __restrict__ out) {
  const uint64_t base = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) * kScanItems;
  uint32_t local[kScanItems];
  uint32_t sum = 0;
  for (int k = 0; k < kScanItems; ++k) {
    local[k] = base + k < n ? counts[base + k] : 0u;
    sum += local[k];
  }
  uint64_t running = block_offsets[blockIdx.x] + block_exclusive_scan_u32(sum);
  for (int k = 0; k < kScanItems; ++k) {
    if (base + k <= n) out[base + k] = static_cast<IDX>(running);
    running += local[k];
  }
}

__global__ void __launch_bounds__(kThreads) sum_complex_kernel(const double* __restrict__ v, uint64_t n,
                                                                double* __restrict__ partials) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  double re = 0.0, im = 0.0;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride) {
    re += v[2 * i];
    im += v[2 * i + 1];
  }
  __shared__ double red[kThreads / 32][2];
  re = warp_sum(re);
  im = warp_sum(im);
  if ((threadIdx.x & 31) == 0) {
    red[threadIdx.x >> 5][0] = re;
    red[threadIdx.x >> 5][1] = im;
  }
  __syncthreads();
  if (threadIdx.x < 2) {
    double total = 0.0;
    for (int wv = 0; wv < kThreads / 32; ++wv) total += red[wv][threadIdx.x];
    partials[2 * blockIdx.x + threadIdx.x] = total;
  }
}

__global__ void __launch_bounds__(kThreads) max_shifted_kernel(const double* __restrict__ diag,
                                                                const double* __restrict__ offsum, uint64_t n,
                                                                double sr, double si, double* __restrict__ partials) {
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  double m = 0.0;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += stride)
    m = fmax(m, offsum[i] + hypot(diag[2 * i] - sr, diag[2 * i + 1] - si));
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  __shared__ double red[kThreads / 32];
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    double total = 0.0;
    for (int wv = 0; wv < kThreads / 32; ++wv) total = fmax(total, red[wv]);
    partials[blockIdx.x] = total;
  }
}

// --- parallel cyclic Jacobi (one CTA) ---------------------------------------------------
// A: np x np row-major complex (interleaved), V: np x np column-major complex.
// Round-robin ordering pairs np/2 disjoint (p,q) per round; each rotation
// zeroes |a_pq| after removing its phase (complex Jacobi rotation).
__global__ void __launch_bounds__(1024) jacobi_kernel(int np, double* __restrict__ A, double* __restrict__ V,
                                                      int max_sweeps) {
  extern __shared__ int order[];
  __shared__ double c_s[512], s_s[512], pr_s[512], pi_s[512];
  __shared__ int p_s[512], q_s[512];
  __shared__ double red[32][2];
  __shared__ int done;
  __shared__ double previous_off;
  const int half = np / 2;
  // Converged when the off-diagonal mass is at rounding level for this size,
  // or when a sweep no longer reduces it (rounding floor reached).
  const double floor_rel = (2.220446049250313e-16 * np) * (2.220446049250313e-16 * np) * 1e-2;
  if (threadIdx.x == 0) previous_off = -1.0;
  for (int i = threadIdx.x; i < np; i += blockDim.x) order[i] = i;
  for (int idx = threadIdx.x; idx < np * np; idx += blockDim.x) {
    V[2 * idx] = (idx / np == idx % np) ? 1.0 : 0.0;
    V[2 * idx + 1] = 0.0;
  }
  __syncthreads();
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    double off = 0.0, total = 0.0;
    for (int idx = threadIdx.x; idx < np * np; idx += blockDim.x) {
      const double v = A[2 * idx] * A[2 * idx] + A[2 * idx + 1] * A[2 * idx + 1];
      total += v;
      if (idx / np != idx % np) off += v;
    }
    off = warp_sum(off);
    total = warp_sum(total);
    if ((threadIdx.x & 31) == 0) {
      red[threadIdx.x >> 5][0] = off;
      red[threadIdx.x >> 5][1] = total;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double o = 0.0, t = 0.0;
      for (int wv = 0; wv < static_cast<int>(blockDim.x >> 5); ++wv) {
        o += red[wv][0];
        t += red[wv][1];
      }
      // stagnation counts only once the off-diagonal mass is near rounding level
      const bool stalled = sweep > 4 && previous_off >= 0.0 && o >= 0.5 * previous_off && o <= 1e-24 * t;
      done = (o <= floor_rel * t || o == 0.0 || stalled) ? 1 : 0;
      previous_off = o;
    }
    __syncthreads();
    if (done) break;
    for (int round = 0; round < np - 1; ++round) {
      for (int t = threadIdx.x; t < half; t += blockDim.x) {
        int p = order[t], q = order[np - 1 - t];
        if (p > q) {
          const int tmp = p;
          p = q;
          q = tmp;
        }
        p_s[t] = p;
        q_s[t] = q;
        const double br = A[2 * (p * np + q)], bi = A[2 * (p * np + q) + 1];
        const double mag = hypot(br, bi);
        if (mag == 0.0) {
          c_s[t] = 1.0;
          s_s[t] = 0.0;
          pr_s[t] = 1.0;
          pi_s[t] = 0.0;
        } else {
          const double app = A[2 * (p * np + p)], aqq = A[2 * (q * np + q)];
          const double theta = (aqq - app) / (2.0 * mag);
          const double tt = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
          const double c = 1.0 / sqrt(tt * tt + 1.0);
          c_s[t] = c;
          s_s[t] = tt * c;
          pr_s[t] = br / mag;
          pi_s[t] = bi / mag;
        }
      }
      __syncthreads();
      // rows: A <- J^H A
      for (int idx = threadIdx.x; idx < half * np; idx += blockDim.x) {
        const int t = idx / np, k = idx % np;
        const int p = p_s[t], q = q_s[t];
        const double c = c_s[t], s = s_s[t], fr = pr_s[t], fi = pi_s[t];
        const double apr = A[2 * (p * np + k)], api = A[2 * (p * np + k) + 1];
        const double aqr = A[2 * (q * np + k)], aqi = A[2 * (q * np + k) + 1];
        // p: c a_p - s phase a_q ; q: s conj(phase) a_p + c a_q
        A[2 * (p * np + k)] = c * apr - s * (fr * aqr - fi * aqi);
        A[2 * (p * np + k) + 1] = c * api - s * (fr * aqi + fi * aqr);
        A[2 * (q * np + k)] = s * (fr * apr + fi * api) + c * aqr;
        A[2 * (q * np + k) + 1] = s * (fr * api - fi * apr) + c * aqi;
      }
      __syncthreads();
      // columns: A <- A J, V <- V J
      for (int idx = threadIdx.x; idx < half * np; idx += blockDim.x) {
        const int t = idx / np, k = idx % np;
        const int p = p_s[t], q = q_s[t];
        const double c = c_s[t], s = s_s[t], fr = pr_s[t], fi = pi_s[t];
        {
          const double apr = A[2 * (k * np + p)], api = A[2 * (k * np + p) + 1];
          const double aqr = A[2 * (k * np + q)], aqi = A[2 * (k * np + q) + 1];
          // p: c a_p - s conj(phase) a_q ; q: s phase a_p + c a_q
          A[2 * (k * np + p)] = c * apr - s * (fr * aqr + fi * aqi);
          A[2 * (k * np + p) + 1] = c * api - s * (fr * aqi - fi * aqr);
          A[2 * (k * np + q)] = s * (fr * apr - fi * api) + c * aqr;
          A[2 * (k * np + q) + 1] = s * (fr * api + fi * apr) + c * aqi;
        }
        {
          const double vpr = V[2 * (p * np + k)], vpi = V[2 * (p * np + k) + 1];
          const double vqr = V[2 * (q * np + k)], vqi = V[2 * (q * np + k) + 1];
          V[2 * (p * np + k)] = c * vpr - s * (fr * vqr + fi * vqi);
          V[2 * (p * np + k) + 1] = c * vpi - s * (fr * vqi - fi * vqr);
          V[2 * (q * np + k)] = s * (fr * vpr - fi * vpi) + c * vqr;
          V[2 * (q * np + k) + 1] = s * (fr * vpi + fi * vpr) + c * vqi;
        }
      }
      __syncthreads();
      for (int t = threadIdx.x; t < half; t += blockDim.x) {
        const int p = p_s[t], q = q_s[t];
        if (c_s[t] != 1.0 || s_s[t] != 0.0) {
          A[2 * (p * np + q)] = A[2 * (p * np + q) + 1] = 0.0;
          A[2 * (q * np + p)] = A[2 * (q * np + p) + 1] = 0.0;
          A[2 * (p * np + p) + 1] = 0.0;
          A[2 * (q * np + q) + 1] = 0.0;
        }
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        const int last = order[np - 1];
        for (int i = np - 1; i > 1; --i) order[i] = order[i - 1];
        order[1] = last;
      }
      __syncthreads();
    }
  }
}

// Parallel cyclic Jacobi with the matrix and its eigenvectors in shared
// memory (one CTA, real symmetric or complex Hermitian, row-major a of the
// lower part's size n padded to even np). A round rotates np/2 disjoint pairs
// at once; J^H A J splits into the (np/2)^2 independent 2 x 2 blocks (pair s
// rows, pair t columns), so rows and columns are rotated by one thread per
// block in one pass. What bounds it is the round's latency chain (shared reads,
// two reciprocal square roots per angle, two barriers), not arithmetic:
// the projected matrices are 8 to 44 wide. So the warps behind the first one or
// two rotate the vectors while those compute the next round's angles, and the
// angles lie as (c, s) pairs, which a warp reads without bank conflicts.
// Measured (B200): 16 x 16 real 39 us and 44 x 44 real 215 us; 44 and 234 with
// a square root, a division and a reciprocal square root per angle, 46 and 310
// with angles, then blocks and vectors; 210 us and (40 x 40) 2268 us for
// jacobi_kernel, which keeps both matrices in global memory as complex numbers;
// that kernel remains for matrices beyond the shared memory.
constexpr int kJacobiBlockItems = 512;       // 2 x 2 blocks of a trip
constexpr int kJacobiMaxThreads = 512 + 64;  // and up to two warps for the next round's angles
constexpr size_t kJacobiMaxSmem = 200 * 1024;  // real n <= 112, complex n <= 78
constexpr int kEigenWorkspace = 10;             // workspace slot of the handle (0-9: the filtered solver's)

template <bool CPLX>
struct JacobiElem;
template <>
struct JacobiElem<false> {
  using type = double;
};
template <>
struct JacobiElem<true> {
  using type = double2;
};

__device__ __forceinline__ double jacobi_sq(double v) { return v * v; }
__device__ __forceinline__ double jacobi_sq(double2 v) { return v.x * v.x + v.y * v.y; }
// |v| to the last bits whatever its size: b / |b| is the phase of a unitary rotation
__device__ __forceinline__ double jacobi_abs(double v) { return fabs(v); }
__device__ __forceinline__ double jacobi_abs(double2 v) { return hypot(v.x, v.y); }
// x c - y s f and x s conj(f) + y c: the two rows (or, with f conjugated,
// columns) of a rotated pair; real data has the phase's sign inside s.
__device__ __forceinline__ void jacobi_rotate(double& x, double& y, double c, double s, double, double) {
  const double u = c * x - s * y, v = s * x + c * y;
  x = u;
  y = v;
}
__device__ __forceinline__ void jacobi_rotate(double2& x, double2& y, double c, double s, double fr, double fi) {
  const double2 u = make_double2(c * x.x - s * (fr * y.x - fi * y.y), c * x.y - s * (fr * y.y + fi * y.x));
  const double2 v = make_double2(s * (fr * x.x + fi * x.y) + c * y.x, s * (fr * x.y - fi * x.x) + c * y.y);
  x = u;
  y = v;
}
__device__ __forceinline__ void jacobi_drop_imag(double&) {}
__device__ __forceinline__ void jacobi_drop_imag(double2& v) { v.y = 0.0; }
__device__ __forceinline__ double jacobi_re(double v) { return v; }
__device__ __forceinline__ double jacobi_re(double2 v) { return v.x; }
__device__ __forceinline__ void jacobi_set(double& v, double re) { v = re; }
__device__ __forceinline__ void jacobi_set(double2& v, double re) { v = make_double2(re, 0.0); }

size_t jacobi_smem_bytes(int n, bool cplx) {
  const size_t np = static_cast<size_t>(n + (n & 1));
  return 2 * np * (np + 1) * (cplx ? 16 : 8) + 2 * (np / 2) * ((cplx ? 2 : 1) * sizeof(double2) + sizeof(int));
}

// in: n x n row-major; values: n; vectors: column-major n x n.
template <bool CPLX>
__global__ void __launch_bounds__(kJacobiMaxThreads)
    jacobi_smem_kernel(int n, const double* __restrict__ in, double* __restrict__ values,
                       double* __restrict__ vectors, int max_sweeps) {
  using E = typename JacobiElem<CPLX>::type;
  extern __shared__ __align__(16) unsigned char jacobi_raw[];
  __shared__ double red[kJacobiMaxThreads / 32][2];
  __shared__ int done;
  __shared__ double previous_off;
  const int np = n + (n & 1), half = np / 2, ld = np + 1;
  E* A = reinterpret_cast<E*>(jacobi_raw);
  E* V = A + np * ld;  // V[k * ld + j]: component k of vector j
  // of this round and the next, per pair: (c, s), phase, (p, q)
  constexpr int RW = CPLX ? 2 : 1;
  double2* rot = reinterpret_cast<double2*>(V + np * ld);
  int* pairs = reinterpret_cast<int*>(rot + 2 * RW * half);
  const double floor_rel = (2.220446049250313e-16 * np) * (2.220446049250313e-16 * np) * 1e-2;
  if (threadIdx.x == 0) previous_off = -1.0;
  for (int idx = threadIdx.x; idx < np * np; idx += blockDim.x) {
    const int i = idx / np, j = idx % np;
    E v;
    jacobi_set(v, 0.0);
    if (i < n && j < n) v = reinterpret_cast<const E*>(in)[i * n + j];
    A[i * ld + j] = v;
    jacobi_set(V[i * ld + j], i == j ? 1.0 : 0.0);
  }
  __syncthreads();
  // this thread's first block (s0, t0) of A and the step to its next one; the
  // same for V, which the warps behind the angles' have
  const int chain = (half + 31) / 32 * 32;
  const int va = static_cast<int>(threadIdx.x) - chain, vn = static_cast<int>(blockDim.x) - chain;
  const int s0 = threadIdx.x / half, t0 = threadIdx.x % half, ds = blockDim.x / half, dt = blockDim.x % half;
  const int i0 = va >= 0 ? va / half : half, j0 = va >= 0 ? va % half : 0, di = vn / half, dj = vn % half;
  // The rotations of a round, from A as the round before left it.
  auto angles = [&](int round) {
    const int t = threadIdx.x;
    if (t >= half) return;
    // round-robin pairing: position 0 is fixed, the others move by one place per round
    int p = t == 0 ? 0 : t - round, q = np - 1 - t - round;
    if (t != 0 && p < 1) p += np - 1;
    if (q < 1) q += np - 1;
    if (p > q) {
      const int swap = p;
      p = q;
      q = swap;
    }
    const E b = A[p * ld + q];
    const double mag = jacobi_abs(b);
    double c = 1.0, s = 0.0, fr = 1.0, fi = 0.0;
    if (mag != 0.0) {
      // cos 2 theta = |d| / sqrt(d^2 + 4 |b|^2), d = a_qq - a_pp: c^2 = (1 + cos 2 theta) / 2
      // and s = sin 2 theta / (2 c), two reciprocal square roots in the round's dependent chain
      double d = jacobi_re(A[q * ld + q]) - jacobi_re(A[p * ld + p]), b2 = 2.0 * mag;
      double x = d * d + b2 * b2;
      if (!(x > 1e-280 && x < 1e280)) {  // squares out of range: the same ratio from scaled entries
        const double top = fmax(fabs(d), b2);
        d /= top;
        b2 /= top;
        x = d * d + b2 * b2;
      }
      const double u = rsqrt(x), c2 = fma(0.5 * fabs(d), u, 0.5), v = rsqrt(c2);
      c = c2 * v;
      s = copysign(0.5 * b2 * u * v, d);
      if constexpr (CPLX) {
        fr = b.x / mag;
        fi = b.y / mag;
      } else if (b < 0.0) {
        s = -s;
      }
    }
    const int at = (round & 1) * half + t;
    rot[at] = make_double2(c, s);
    if constexpr (CPLX) rot[2 * half + at] = make_double2(fr, fi);
    pairs[at] = p | q << 16;
  };
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    double off = 0.0, total = 0.0;
    for (int idx = threadIdx.x; idx < np * np; idx += blockDim.x) {
      const int i = idx / np, j = idx % np;
      const double v = jacobi_sq(A[i * ld + j]);
      total += v;
      if (i != j) off += v;
    }
    off = warp_sum(off);
    total = warp_sum(total);
    if ((threadIdx.x & 31) == 0) {
      red[threadIdx.x >> 5][0] = off;
      red[threadIdx.x >> 5][1] = total;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      double o = 0.0, t = 0.0;
      for (int wv = 0; wv < static_cast<int>(blockDim.x >> 5); ++wv) {
        o += red[wv][0];
        t += red[wv][1];
      }
      // stagnation counts only once the off-diagonal mass is near rounding level
      const bool stalled = sweep > 4 && previous_off >= 0.0 && o >= 0.5 * previous_off && o <= 1e-24 * t;
      done = (o <= floor_rel * t || o == 0.0 || stalled) ? 1 : 0;
      previous_off = o;
    }
    __syncthreads();
    if (done) break;
    angles(0);
    __syncthreads();
    for (int round = 0; round < np - 1; ++round) {
      const double2* cs = rot + (round & 1) * half;
      const int* pq_of = pairs + (round & 1) * half;
      auto phase = [&](int t) { return CPLX ? cs[2 * half + t] : make_double2(1.0, 0.0); };
      for (int s = s0, t = t0; s < half;) {
        const double2 ct = cs[t], ft = phase(t), cr = cs[s], fs = phase(s);
        const int tp = pq_of[t] & 0xffff, tq = pq_of[t] >> 16, p = pq_of[s] & 0xffff, q = pq_of[s] >> 16;
        E pp = A[p * ld + tp], pq = A[p * ld + tq], qp = A[q * ld + tp], qq = A[q * ld + tq];
        jacobi_rotate(pp, qp, cr.x, cr.y, fs.x, fs.y);
        jacobi_rotate(pq, qq, cr.x, cr.y, fs.x, fs.y);
        jacobi_rotate(pp, pq, ct.x, ct.y, ft.x, -ft.y);
        jacobi_rotate(qp, qq, ct.x, ct.y, ft.x, -ft.y);
        if (s == t && (ct.x != 1.0 || ct.y != 0.0)) {
          jacobi_set(pq, 0.0);
          jacobi_set(qp, 0.0);
          jacobi_drop_imag(pp);
          jacobi_drop_imag(qq);
        }
        A[p * ld + tp] = pp;
        A[p * ld + tq] = pq;
        A[q * ld + tp] = qp;
        A[q * ld + tq] = qq;
        s += ds;
        t += dt;
        if (t >= half) {
          t -= half;
          ++s;
        }
      }
      __syncthreads();
      // the next round's angles beside rows 2i, 2i + 1 of V
      if (va < 0 && round + 2 < np) angles(round + 1);
      for (int i = i0, t = j0; i < half;) {
        const double2 ct = cs[t], ft = phase(t);
        const int tp = pq_of[t] & 0xffff, tq = pq_of[t] >> 16;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          E* row = V + (2 * i + h) * ld;
          E vp = row[tp], vq = row[tq];
          jacobi_rotate(vp, vq, ct.x, ct.y, ft.x, -ft.y);
          row[tp] = vp;
          row[tq] = vq;
        }
        i += di;
        t += dj;
        if (t >= half) {
          t -= half;
          ++i;
        }
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) values[i] = jacobi_re(A[i * ld + i]);
  for (int idx = threadIdx.x; idx < n * n; idx += blockDim.x)
    reinterpret_cast<E*>(vectors)[idx] = V[(idx % n) * ld + idx / n];
}

int sm_count(int device) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  return sms;
}

int reduction_grid(uint64_t n, int sms) {
  uint64_t blocks = (n + kThreads - 1) / kThreads;
  return static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>(blocks, static_cast<uint64_t>(4) * sms)));
}

int stream_grid(uint64_t n, int sms) {
  uint64_t blocks = (n + kThreads - 1) / kThreads;
  return static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>(blocks, static_cast<uint64_t>(8) * sms)));
}

// Columns that stay in the L2 between the sweeps of a panel: the overlaps go up
// the columns, the subtraction down, so each sweep begins with the columns that
// the other one ended with. Those are read as usual, the others evict-first (a
// sweep over a panel beyond the L2 drives out the columns it is about to need
// otherwise). Two Lanczos runs of 100 steps at 718,146 rows (28 sites): 26.5 ms
// without, 25.4 at 30 MB, 25.3 at 40 to 50, 25.5 at 70, 26.6 with none kept.
// Other sizes, none / 24 / 48 / 96 MB: 200,474 rows, 100 steps 9.7 / 9.6 / 9.6 / 9.9
// ms; 400,023 complex rows, 60 steps 12.0 / 11.6 / 11.7 / 12.1; 718,146 rows, 30
// steps 4.06 / 3.92 / 3.95 / 4.07; 2,587,018 rows, 60 steps 39.0 / 39.2 / 39.2 /
// 39.6; 9,398,520 rows, 40 steps 71 each.
int kept_columns(uint64_t n, bool cplx) {
  constexpr uint64_t kKeptPanelBytes = 48ull << 20;
  return static_cast<int>(std::min<uint64_t>(kKeptPanelBytes / (n * (cplx ? 16 : 8)), 1u << 20));
}

// Rows of a panel_dot_kernel block: 256..2048, for about eight blocks per SM.
int panel_slab(uint64_t n, int sms) {
  const uint64_t target = (n + 8ull * sms - 1) / (8ull * sms);
  return static_cast<int>(std::min<uint64_t>(kMaxSlab, std::max<uint64_t>(256, (target + 255) / 256 * 256)));
}

// Doubles of partial sums that the overlaps with m columns take.
size_t panel_partials(uint64_t n, int m, int sms) {
  const int slab = panel_slab(n, sms);
  return static_cast<size_t>(m) * ((n + slab - 1) / slab) * 2 + 2 * static_cast<size_t>(m) + 64;
}

constexpr int kOrthoThreads = 256;
constexpr int kOrthoChunk = 8;

__device__ __forceinline__ double block_sum(double v, double* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double total = 0.0;
  if (threadIdx.x == 0)
    for (int k = 0; k < kOrthoThreads / 32; ++k) total += red[k];
  __syncthreads();
  return total;
}

// One Gram-Schmidt pass of the Lanczos step over the basis panel Q (m
// columns, leading dimension n, FP64): w -= sum_k h_k q_k with the overlaps
// h (device, interleaved complex), reading src (which may be w) and writing
// w. Per-block partial sums, in a fixed order: partials[2b] = |w'|^2 for the
// three-term residual w' = src - Re(h_{m-1}) q_{m-1} - beta q_{m-2}
// (before_mode 1) or |src|^2 (before_mode 2), partials[2b+1] =
// |src - sum_k h_k q_k|^2. Elements are complex values
// (kComplex), pairs of real rows loaded as one 16-byte word (kRealPair, n
// even), or single real rows (kReal).
//
// Bound by the panel's read. The columns are taken from the last down, `keep`
// of them from what the overlaps' sweep left in the L2 (kept_columns), and a
// thread takes ROWS elements along, so that the grid sweeps the columns once
// instead of once per grid stride: 718,146 rows by 1 to 100 columns (28 sites)
// 48.9 -> 46.6 us on average, 6.2 TB/s, and 44 with the kept columns.
enum { kReal = 0, kRealPair = 1, kComplex = 2 };
template <int MODE, int ROWS>
__global__ void __launch_bounds__(kOrthoThreads, 4) orthogonalize_kernel(const double* __restrict__ Q, uint64_t n, int m,
                                                                      const double* h, double beta_value,
                                                                      const double* beta_device,
                                                                      int before_mode, int keep, const double* src,
                                                                      double* w, double* __restrict__ partials) {
  extern __shared__ double hs[];
  __shared__ double red[kOrthoThreads / 32];
  await_previous();
  for (int t = threadIdx.x; t < 2 * m; t += blockDim.x) hs[t] = __ldcg(h + t);
  __syncthreads();
  const double alpha = hs[2 * (m - 1)];
  const double beta = beta_device ? __ldcg(beta_device) : beta_value;
  // element count and the stride between columns, in elements
  const uint64_t elems = MODE == kRealPair ? n / 2 : n;
  const uint64_t col = MODE == kReal ? n : n / (MODE == kRealPair ? 2 : 1);
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  // columns loaded ahead per element: eight 8-byte or four 16-byte words in all
  constexpr int CH = (MODE == kReal ? kOrthoChunk : kOrthoChunk / 2) / (ROWS > 1 ? 2 : 1);
  double before = 0.0, after = 0.0;
  for (uint64_t i0 = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i0 < elems; i0 += ROWS * stride) {
    // (a, b): real and imaginary parts, or the two rows of a pair
    double sa[ROWS], sb[ROWS], ta[ROWS], tb[ROWS];  // the pass's sum, the three-term one
#pragma unroll
    for (int u = 0; u < ROWS; ++u) sa[u] = sb[u] = ta[u] = tb[u] = 0.0;
    for (int j0 = (m - 1) / CH * CH; j0 >= 0; j0 -= CH) {
      double xa[CH][ROWS], xb[CH][ROWS];
      auto read = [&](auto stream) {
        constexpr bool STREAM = decltype(stream)::value;
#pragma unroll
        for (int jj = 0; jj < CH; ++jj)
#pragma unroll
          for (int u = 0; u < ROWS; ++u) {
            const uint64_t i = i0 + u * stride;
            xa[jj][u] = xb[jj][u] = 0.0;
            if (j0 + jj < m && (ROWS == 1 || i < elems)) {
              if (MODE == kReal) {
                const double* q = Q + static_cast<uint64_t>(j0 + jj) * col + i;
                xa[jj][u] = STREAM ? __ldcs(q) : __ldg(q);
              } else {
                const double2* q = reinterpret_cast<const double2*>(Q) + static_cast<uint64_t>(j0 + jj) * col + i;
                const double2 v = STREAM ? __ldcs(q) : __ldg(q);
                xa[jj][u] = v.x;
                xb[jj][u] = v.y;
              }
            }
          }
      };
      if (j0 >= keep) read(std::true_type{});
      else read(std::false_type{});
#pragma unroll
      for (int jj = 0; jj < CH; ++jj) {
        const int k = j0 + jj;
        if (k < m) {
          const double hr = hs[2 * k], hi = hs[2 * k + 1];
#pragma unroll
          for (int u = 0; u < ROWS; ++u) {
            if (MODE == kComplex) {
              sa[u] += hr * xa[jj][u] - hi * xb[jj][u];
              sb[u] += hr * xb[jj][u] + hi * xa[jj][u];
            } else {  // real basis: the overlaps are real
              sa[u] += hr * xa[jj][u];
              sb[u] += hr * xb[jj][u];
            }
            if (k >= m - 2) {
              const double t = k == m - 1 ? alpha : beta;
              ta[u] += t * xa[jj][u];
              tb[u] += t * xb[jj][u];
            }
          }
        }
      }
    }
#pragma unroll
    for (int u = 0; u < ROWS; ++u) {
      const uint64_t i = i0 + u * stride;
      if (ROWS > 1 && i >= elems) break;
      double wa, wb = 0.0;
      if (MODE == kReal) {
        wa = src[i];
      } else {
        const double2 v = reinterpret_cast<const double2*>(src)[i];
        wa = v.x;
        wb = v.y;
      }
      if (before_mode == 1) {
        const double ba = wa - ta[u], bb = wb - tb[u];
        before += ba * ba + bb * bb;
      } else if (before_mode == 2) {
        before += wa * wa + wb * wb;
      }
      const double ra = wa - sa[u], rb = wb - sb[u];
      if (MODE == kReal) w[i] = ra;
      else reinterpret_cast<double2*>(w)[i] = make_double2(ra, rb);
      after += ra * ra + rb * rb;
    }
  }
  before = block_sum(before, red);
  after = block_sum(after, red);
  if (threadIdx.x == 0) {
    partials[2 * blockIdx.x] = before;
    partials[2 * blockIdx.x + 1] = after;
  }
}

// Launches orthogonalize_kernel and returns its grid (partials: two per block).
// Elements a thread takes along: as many as one resident grid (four blocks an
// SM) needs for one sweep, three at most.
int launch_orthogonalize(const double* A, uint64_t n, int m, const double* h, double beta, const double* beta_device,
                         int before_mode, const double* src, double* w, double* partials, bool cplx, int sms,
                         cudaStream_t stream) {
  // pairs of real rows move as 16-byte words when every column starts 16-byte aligned
  const int mode = cplx ? kComplex : (n % 2 == 0 ? kRealPair : kReal);
  const uint64_t elems = mode == kRealPair ? n / 2 : n, resident = 4ull * sms * kOrthoThreads;
  const int rows = static_cast<int>(std::min<uint64_t>(3, (elems + resident - 1) / resident));
  const uint64_t per_block = static_cast<uint64_t>(rows) * kOrthoThreads;
  const int G = static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>((elems + per_block - 1) / per_block, 4ull * sms)));
  const size_t smem = static_cast<size_t>(m) * 16;
  auto launch = [&](auto kernel) {
    if (smem > 48 * 1024)
      QMBED_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    launch_dependent(kernel, G, kOrthoThreads, smem, stream, A, n, m, h, beta, beta_device, before_mode,
                     kept_columns(n, cplx), src, w, partials);
  };
  auto by_rows = [&](auto mode_tag) {
    constexpr int MODE = decltype(mode_tag)::value;
    if (rows == 1) launch(orthogonalize_kernel<MODE, 1>);
    else if (rows == 2) launch(orthogonalize_kernel<MODE, 2>);
    else launch(orthogonalize_kernel<MODE, 3>);
  };
  if (mode == kComplex) by_rows(std::integral_constant<int, kComplex>{});
  else if (mode == kRealPair) by_rows(std::integral_constant<int, kRealPair>{});
  else by_rows(std::integral_constant<int, kReal>{});
  QMBED_LAUNCH_CHECK();
  return G;
}

// out[0..1] = sums of the two partial columns over G blocks (fixed order);
// out[2..3] = alpha (the last overlap) for the host's Hermiticity check.
__global__ void __launch_bounds__(128) orthogonalize_finish_kernel(const double* __restrict__ partials, int G,
                                                                   const double* __restrict__ alpha,
                                                                   double* __restrict__ out) {
  __shared__ double tree[2][128];
  double b = 0.0, a = 0.0;
  for (int k = threadIdx.x; k < G; k += 128) {
    b += partials[2 * k];
    a += partials[2 * k + 1];
  }
  tree[0][threadIdx.x] = b;
  tree[1][threadIdx.x] = a;
  __syncthreads();
  for (int width = 64; width > 0; width >>= 1) {
    if (threadIdx.x < width) {
      tree[0][threadIdx.x] += tree[0][threadIdx.x + width];
      tree[1][threadIdx.x] += tree[1][threadIdx.x + width];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    out[0] = tree[0][0];
    out[1] = tree[1][0];
    out[2] = alpha[0];
    out[3] = alpha[1];
  }
}

// End of a queued step: every block sums the norms' partials in the same order,
// the first writes the record (norms before and after, the DGKS verdict and the
// last overlap), all scale the vector into the next column. One launch; a
// record kernel of its own took 3.2 us and a gap in front of the scaling.
__global__ void __launch_bounds__(kThreads) scale_and_record_kernel(const double* partials, int G, int m,
                                                                    const double* h, double* __restrict__ record,
                                                                    const double* src,
                                                                    double* __restrict__ dst, uint64_t count) {
  __shared__ double tree[2][128];
  await_previous();
  if (threadIdx.x < 128) {
    double b = 0.0, a = 0.0;
    for (int k = threadIdx.x; k < G; k += 128) {
      b += __ldcg(partials + 2 * k);
      a += __ldcg(partials + 2 * k + 1);
    }
    tree[0][threadIdx.x] = b;
    tree[1][threadIdx.x] = a;
  }
  __syncthreads();
  for (int width = 64; width > 0; width >>= 1) {
    if (threadIdx.x < width) {
      tree[0][threadIdx.x] += tree[0][threadIdx.x + width];
      tree[1][threadIdx.x] += tree[1][threadIdx.x + width];
    }
    __syncthreads();
  }
  const double before = sqrt(fmax(tree[0][0], 0.0)), after = sqrt(fmax(tree[1][0], 0.0));
  const bool ok = isfinite(after) && after > 1.0e-14;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    record[0] = before;
    record[1] = after;
    record[2] = before > 2.220446049250313e-16 && after <= 0.70710678118654752440 * before ? 1.0 : 0.0;
    record[3] = ok ? 1.0 : 0.0;
    record[FusedOrtho::kRecordHead + 2 * (m - 1)] = __ldcg(h);
    record[FusedOrtho::kRecordHead + 2 * (m - 1) + 1] = __ldcg(h + 1);
  }
  if (!ok) return;
  const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
  for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride)
    dst[i] = __ldcg(src + i) / after;
}

}  // namespace

uint64_t exclusive_scan_counts(const uint32_t* counts, uint64_t n, DeviceBuffer& row_ptr, bool* is64) {
  const uint64_t per_block = static_cast<uint64_t>(kThreads) * kScanItems;
  const uint64_t blocks = std::max<uint64_t>(1, (n + 1 + per_block - 1) / per_block);
  DeviceBuffer totals(blocks * sizeof(uint64_t));
  scan_block_totals_kernel<<<static_cast<unsigned>(blocks), kThreads>>>(counts, n, totals.as<uint64_t>());
  QMBED_LAUNCH_CHECK();
  std::vector<uint64_t> host(blocks);
  QMBED_CUDA(cudaMemcpy(host.data(), totals.get(), blocks * 8, cudaMemcpyDeviceToHost));
  uint64_t running = 0;
  for (uint64_t b = 0; b < blocks; ++b) {
    const uint64_t t = host[b];
    host[b] = running;
    running += t;
  }
  QMBED_CUDA(cudaMemcpy(totals.get(), host.data(), blocks * 8, cudaMemcpyHostToDevice));
  *is64 = running >= (1ULL << 32);
  if (*is64) {
    row_ptr.allocate((n + 1) * sizeof(uint64_t));
    scan_write_kernel<uint64_t><<<static_cast<unsigned>(blocks), kThreads>>>(counts, n, totals.as<uint64_t>(),
                                                                            row_ptr.as<uint64_t>());
  } else {
    row_ptr.allocate((n + 1) * sizeof(uint32_t));
    scan_write_kernel<uint32_t><<<static_cast<unsigned>(blocks), kThreads>>>(counts, n, totals.as<uint64_t>(),
                                                                            row_ptr.as<uint32_t>());
  }
  QMBED_LAUNCH_CHECK();
  return running;
}

C64 device_sum_complex(const double* v, uint64_t n) {
  int device = 0;
  cudaGetDevice(&device);
  const int G = reduction_grid(n, sm_count(device));
  DeviceBuffer partials(2 * G * sizeof(double));
  sum_complex_kernel<<<G, kThreads>>>(v, n, partials.as<double>());
  QMBED_LAUNCH_CHECK();
  std::vector<double> host(2 * G);
  QMBED_CUDA(cudaMemcpy(host.data(), partials.get(), host.size() * 8, cudaMemcpyDeviceToHost));
  double re = 0.0, im = 0.0;
  for (int b = 0; b < G; ++b) {
    re += host[2 * b];
    im += host[2 * b + 1];
  }
  return C64(re, im);
}

double device_max_shifted_column(const double* diag, const double* offsum, uint64_t n, C64 shift) {
  int device = 0;
  cudaGetDevice(&device);
  const int G = reduction_grid(n, sm_count(device));
  DeviceBuffer partials(G * sizeof(double));
  max_shifted_kernel<<<G, kThreads>>>(diag, offsum, n, shift.real(), shift.imag(), partials.as<double>());
  QMBED_LAUNCH_CHECK();
  std::vector<double> host(G);
  QMBED_CUDA(cudaMemcpy(host.data(), partials.get(), host.size() * 8, cudaMemcpyDeviceToHost));
  double m = 0.0;
  for (double v : host) m = std::max(m, v);
  return m;
}

BlockOps::BlockOps(int device, cudaStream_t stream)
    : device_(device), stream_(stream), sms_(sm_count(device)), fused_(device, sms_) {
  QMBED_CUDA(cudaSetDevice(device_));
  BlockPool::attach(device_);
}

BlockOps::~BlockOps() {
  if (host_results_) cudaFreeHost(host_results_);
  BlockPool::detach(device_);
}

void Scratch::take(BlockOps& ops, size_t bytes) {
  release();
  QMBED_CUDA(cudaSetDevice(ops.device()));
  device_ = ops.device();
  stream_ = ops.stream();
  bytes = bytes > 0 ? bytes : 1;
  ptr_ = BlockPool::take(bytes, &bytes_);
  if (ptr_) return;
  DeviceBuffer fresh(bytes);
  bytes_ = bytes;
  ptr_ = fresh.detach();
}

void Scratch::release() {
  if (!ptr_) return;
  cudaStreamSynchronize(stream_);
  BlockPool::give(ptr_, bytes_, device_);
  ptr_ = nullptr;
}

void* BlockOps::workspace(int slot, size_t bytes) {
  if (slot < 0 || slot > 64) raise(QMBED_INTERNAL_STATE, "workspace slot out of range");
  if (workspace_.size() <= static_cast<size_t>(slot)) workspace_.resize(slot + 1);
  DeviceBuffer& b = workspace_[slot];
  if (b.bytes() < bytes) {
    QMBED_CUDA(cudaStreamSynchronize(stream_));  // the old buffer may still be read by queued work
    b.release();
    b.allocate(bytes);
  }
  return b.get();
}

void BlockOps::ensure_partials(size_t doubles) {
  if (partials_doubles_ < doubles) {
    partials_.allocate(doubles * sizeof(double));
    partials_doubles_ = doubles;
  }
  if (host_results_doubles_ < doubles) {
    if (host_results_) cudaFreeHost(host_results_);
    host_results_ = nullptr;
    QMBED_CUDA(cudaMallocHost(&host_results_, doubles * sizeof(double)));
    host_results_doubles_ = doubles;
    results_.allocate(doubles * sizeof(double));
  }
}

void BlockOps::ensure_coeffs(size_t bytes) {
  if (coeffs_bytes_ < bytes) {
    coeffs_.allocate(bytes);
    coeffs_bytes_ = bytes;
  }
}

void BlockOps::sync() { QMBED_CUDA(cudaStreamSynchronize(stream_)); }

#define QMBED_DISPATCH(precision, cplx, KERNEL_CALL)          \
  do {                                                        \
    if ((precision) == 64) {                                  \
      using T = double;                                       \
      if (cplx) { constexpr bool C = true; KERNEL_CALL; }     \
      else { constexpr bool C = false; KERNEL_CALL; }         \
    } else {                                                  \
      using T = float;                                        \
      if (cplx) { constexpr bool C = true; KERNEL_CALL; }     \
      else { constexpr bool C = false; KERNEL_CALL; }         \
    }                                                         \
  } while (0)

void BlockOps::dots(const void* A, uint64_t ld, int m, const void* w, uint64_t n, int precision, bool cplx,
                    C64* out, double* self_sq) {
  if (m <= 0) {
    if (self_sq) *self_sq = std::pow(norm(w, n, precision, cplx), 2);
    return;
  }
  const int G = reduction_grid(n, sms_);
  const int columns = m + (self_sq ? 1 : 0);
  ensure_partials(static_cast<size_t>(columns) * G * 2 + 2 * static_cast<size_t>(columns) + 64);
  QMBED_DISPATCH(precision, cplx,
                 (multi_dot_kernel<T, C><<<G, kThreads, 0, stream_>>>(static_cast<const T*>(A), ld, m,
                                                                      static_cast<const T*>(w), n,
                                                                      partials_.as<double>(), self_sq ? 1 : 0)));
  QMBED_LAUNCH_CHECK();
  const int count = 2 * columns;
  finish_kernel<<<count, kFinishThreads, 0, stream_>>>(partials_.as<double>(), G, count, results_.as<double>());
  QMBED_LAUNCH_CHECK();
  QMBED_CUDA(cudaMemcpyAsync(host_results_, results_.get(), count * sizeof(double), cudaMemcpyDeviceToHost, stream_));
  sync();
  for (int j = 0; j < m; ++j) out[j] = C64(host_results_[2 * j], host_results_[2 * j + 1]);
  if (self_sq) *self_sq = host_results_[2 * m];
}

void BlockOps::dots_device(const void* A, uint64_t ld, int m, const void* w, uint64_t n, int precision, bool cplx,
                           double* out) {
  if (m <= 0 || n == 0) return;
  int G;
  if (precision == 64) {
    const int slab = panel_slab(n, sms_);
    G = static_cast<int>((n + slab - 1) / slab);
    ensure_partials(panel_partials(n, m, sms_));
    const size_t smem = static_cast<size_t>(slab) * (cplx ? 16 : 8);
    if (cplx)
      launch_dependent(panel_dot_kernel<true>, G, kThreads, smem, stream_, static_cast<const double*>(A), ld, m,
                       static_cast<const double*>(w), n, slab, kept_columns(n, cplx), partials_.as<double>());
    else
      launch_dependent(panel_dot_kernel<false>, G, kThreads, smem, stream_, static_cast<const double*>(A), ld, m,
                       static_cast<const double*>(w), n, slab, kept_columns(n, cplx), partials_.as<double>());
  } else {
    G = reduction_grid(n, sms_);
    ensure_partials(static_cast<size_t>(m) * G * 2 + 2 * static_cast<size_t>(m) + 64);
    QMBED_DISPATCH(precision, cplx,
                   (multi_dot_kernel<T, C><<<G, kThreads, 0, stream_>>>(static_cast<const T*>(A), ld, m,
                                                                        static_cast<const T*>(w), n,
                                                                        partials_.as<double>(), 0)));
  }
  QMBED_LAUNCH_CHECK();
  launch_dependent(finish_kernel, 2 * m, kFinishThreads, 0, stream_, partials_.as<double>(), G, 2 * m, out);
  QMBED_LAUNCH_CHECK();
}

void BlockOps::scale_into(const void* src, void* dst, uint64_t n, double divisor, int precision, bool cplx) {
  const uint64_t count = n * (cplx ? 2 : 1);
  const int G = stream_grid(count, sms_);
  if (precision == 64)
    scale_into_kernel<double><<<G, kThreads, 0, stream_>>>(static_cast<const double*>(src), static_cast<double*>(dst),
                                                           count, divisor);
  else
    scale_into_kernel<float><<<G, kThreads, 0, stream_>>>(static_cast<const float*>(src), static_cast<float*>(dst),
                                                          count, divisor);
  QMBED_LAUNCH_CHECK();
}

double BlockOps::norm(const void* w, uint64_t n, int precision, bool cplx) {
  C64 v;
  dots(w, n, 1, w, n, precision, cplx, &v);
  return std::sqrt(std::max(v.real(), 0.0));
}

double BlockOps::subtract(const void* A, uint64_t ld, int m, const C64* h, void* w, uint64_t n, int precision,
                          bool cplx, bool want_norm, const void* src) {
  if (m <= 0 && src && src != w) copy(src, w, n * (cplx ? 2 : 1) * (precision == 64 ? 8 : 4));
  if (m <= 0 && !want_norm) return 0.0;
  if (m <= 0) return norm(w, n, precision, cplx);
  ensure_coeffs(static_cast<size_t>(m) * 16);
  QMBED_CUDA(cudaMemcpyAsync(coeffs_.get(), h, static_cast<size_t>(m) * 16, cudaMemcpyHostToDevice, stream_));
  const int G = reduction_grid(n, sms_);
  ensure_partials(2 * static_cast<size_t>(G) + 64);
  const size_t smem = static_cast<size_t>(m) * 16;
  double* partials = want_norm ? partials_.as<double>() : nullptr;
  QMBED_DISPATCH(precision, cplx, ({
                   auto kernel = subtract_kernel<T, C>;
                   if (smem > 48 * 1024)
                     QMBED_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     static_cast<int>(smem)));
                   kernel<<<G, kThreads, smem, stream_>>>(static_cast<const T*>(A), ld, m, coeffs_.as<double>(),
                                                          static_cast<const T*>(src ? src : w), static_cast<T*>(w), n,
                                                          partials);
                 }));
  QMBED_LAUNCH_CHECK();
  if (!want_norm) return 0.0;
  QMBED_CUDA(cudaMemcpyAsync(host_results_, partials_.get(), 2 * G * sizeof(double), cudaMemcpyDeviceToHost, stream_));
  sync();
  double total = 0.0;
  for (int b = 0; b < G; ++b) total += host_results_[2 * b];
  return std::sqrt(total);
}

void BlockOps::combine(const void* A, uint64_t ld, int m, const C64* Y, int K, void* out, uint64_t ld_out, uint64_t n,
                       int precision, bool cplx) {
  if (K <= 0) return;
  ensure_coeffs(static_cast<size_t>(m) * K * 16);
  QMBED_CUDA(cudaMemcpyAsync(coeffs_.get(), Y, static_cast<size_t>(m) * K * 16, cudaMemcpyHostToDevice, stream_));
  const int G = stream_grid(n, sms_);
  // real data with real coefficients: the tensor-core kernel, 8 columns per launch
  bool real_y = !cplx;
  for (int i = 0; i < m * K && real_y; ++i) real_y = Y[i].imag() == 0.0;
  const size_t ys_bytes = static_cast<size_t>((m + 3) & ~3) * 8 * sizeof(double);
  if (real_y && dense_on_tensor_cores() && ys_bytes <= 48 * 1024) {
    for (int k0 = 0; k0 < K; k0 += 8) {
      if (precision == 64)
        combine_mma_kernel<double><<<G, kThreads, ys_bytes, stream_>>>(static_cast<const double*>(A), ld, m,
                                                                       coeffs_.as<double>(), K, k0,
                                                                       static_cast<double*>(out), ld_out, n);
      else
        combine_mma_kernel<float><<<G, kThreads, ys_bytes, stream_>>>(static_cast<const float*>(A), ld, m,
                                                                      coeffs_.as<double>(), K, k0,
                                                                      static_cast<float*>(out), ld_out, n);
      QMBED_LAUNCH_CHECK();
    }
    sync();
    return;
  }
  for (int k0 = 0; k0 < K; k0 += kCombine) {
    QMBED_DISPATCH(precision, cplx,
                   (combine_kernel<T, C><<<G, kThreads, 0, stream_>>>(static_cast<const T*>(A), ld, m,
                                                                      coeffs_.as<double>(), K, k0,
                                                                      static_cast<T*>(out), ld_out, n)));
    QMBED_LAUNCH_CHECK();
  }
  sync();  // Y lives in caller memory reused on the next call
}

void BlockOps::scale(void* w, uint64_t n, double divisor, int precision, bool cplx) {
  const uint64_t count = n * (cplx ? 2 : 1);
  const int G = stream_grid(count, sms_);
  if (precision == 64) scale_kernel<double><<<G, kThreads, 0, stream_>>>(static_cast<double*>(w), count, divisor);
  else scale_kernel<float><<<G, kThreads, 0, stream_>>>(static_cast<float*>(w), count, divisor);
  QMBED_LAUNCH_CHECK();
}

void BlockOps::convert(const void* src, int src_precision, void* dst, int dst_precision, uint64_t elements) {
  const int G = stream_grid(elements, sms_);
  if (src_precision == dst_precision) {
    copy(src, dst, elements * (src_precision == 64 ? 8 : 4));
    return;
  }
  if (src_precision == 64)
    convert_kernel<double, float><<<G, kThreads, 0, stream_>>>(static_cast<const double*>(src),
                                                               static_cast<float*>(dst), elements);
  else
    convert_kernel<float, double><<<G, kThreads, 0, stream_>>>(static_cast<const float*>(src),
                                                               static_cast<double*>(dst), elements);
  QMBED_LAUNCH_CHECK();
}

void BlockOps::widen_real(const double* src, double* dst, uint64_t n) {
  const int G = stream_grid(n, sms_);
  widen_real_kernel<<<G, kThreads, 0, stream_>>>(src, dst, n);
  QMBED_LAUNCH_CHECK();
}

void BlockOps::import_complex(const double* src, void* dst, uint64_t n, int precision, bool cplx) {
  if (cplx) {
    convert(src, 64, dst, precision, 2 * n);
    return;
  }
  const int G = stream_grid(n, sms_);
  if (precision == 64) real_part_strided_kernel<double><<<G, kThreads, 0, stream_>>>(src, static_cast<double*>(dst), n);
  else real_part_strided_kernel<float><<<G, kThreads, 0, stream_>>>(src, static_cast<float*>(dst), n);
  QMBED_LAUNCH_CHECK();
}

void BlockOps::copy(const void* src, void* dst, uint64_t bytes) {
  if (bytes == 0 || src == dst) return;
  QMBED_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, stream_));
}

void BlockOps::lcg_start(void* out, uint64_t n, uint64_t seed, int precision, bool cplx) {
  const uint64_t per_thread = 64;
  const uint64_t threads = (n + per_thread - 1) / per_thread;
  const unsigned blocks = static_cast<unsigned>(std::max<uint64_t>(1, (threads + kThreads - 1) / kThreads));
  QMBED_DISPATCH(precision, cplx,
                 (lcg_start_kernel<T, C><<<blocks, kThreads, 0, stream_>>>(static_cast<T*>(out), n, seed,
                                                                           per_thread)));
  QMBED_LAUNCH_CHECK();
}

bool BlockOps::ritz_candidates(double* C, double* CA, uint64_t n, int count, bool cplx,
                               std::vector<RitzCandidate>& out) {
  if (count < 1 || n == 0 || n * (cplx ? 2 : 1) > kCandidateDoubles) return false;
  ensure_partials(4 * static_cast<size_t>(count) + 64);
  auto kernel = cplx ? ritz_candidate_kernel<true> : ritz_candidate_kernel<false>;
  kernel<<<count, kCandidateThreads, 0, stream_>>>(C, CA, n, results_.as<double>());
  QMBED_LAUNCH_CHECK();
  QMBED_CUDA(cudaMemcpyAsync(host_results_, results_.get(), 4 * static_cast<size_t>(count) * sizeof(double),
                             cudaMemcpyDeviceToHost, stream_));
  sync();
  out.resize(static_cast<size_t>(count));
  for (int k = 0; k < count; ++k) {
    const double* r = host_results_ + 4 * k;
    out[k] = {std::sqrt(std::max(r[0], 0.0)), r[1], std::sqrt(r[2]), std::sqrt(std::max(r[3], 0.0))};
  }
  return true;
}

double BlockOps::residual_norm(const void* y, const void* x, double lambda, uint64_t n, int precision, bool cplx) {
  const int G = reduction_grid(n, sms_);
  ensure_partials(2 * static_cast<size_t>(G) + 64);
  QMBED_DISPATCH(precision, cplx,
                 (residual_kernel<T, C><<<G, kThreads, 0, stream_>>>(static_cast<const T*>(y),
                                                                     static_cast<const T*>(x), lambda, n,
                                                                     partials_.as<double>())));
  QMBED_LAUNCH_CHECK();
  QMBED_CUDA(cudaMemcpyAsync(host_results_, partials_.get(), 2 * G * sizeof(double), cudaMemcpyDeviceToHost, stream_));
  sync();
  double total = 0.0;
  for (int b = 0; b < G; ++b) total += host_results_[2 * b];
  return std::sqrt(total);
}

void device_hermitian_eigen(int n, const std::vector<C64>& a, std::vector<double>& values, std::vector<C64>& vectors,
                            BlockOps& ops) {
  const cudaStream_t stream = ops.stream();
  values.assign(n, 0.0);
  vectors.assign(static_cast<size_t>(n) * n, C64(0.0, 0.0));
  if (n == 0) return;
  if (n == 1) {
    values[0] = a[0].real();
    vectors[0] = C64(1.0, 0.0);
    return;
  }
  if (n > 1024) raise(QMBED_UNSUPPORTED_BACKEND, "projected eigenproblems above 1024 are not supported");
  bool real = true;
  for (size_t i = 0; i < static_cast<size_t>(n) * n && real; ++i) real = a[i].imag() == 0.0;
  const size_t smem = jacobi_smem_bytes(n, !real);
  if (smem <= kJacobiMaxSmem) {
    // [matrix][values][vectors] in one buffer of the handle, the vectors 16-byte aligned
    const size_t w = real ? 1 : 2, nn = static_cast<size_t>(n) * n, nv = static_cast<size_t>(n + (n & 1));
    const size_t first = nn * w + ((nn * w) & 1);
    double* buf = static_cast<double*>(ops.workspace(kEigenWorkspace, (first + nv + nn * w) * sizeof(double)));
    std::vector<double> host(nn * w + nv);
    for (size_t i = 0; i < nn; ++i) {
      if (real) {
        host[i] = a[i].real();
      } else {
        host[2 * i] = a[i].real();
        host[2 * i + 1] = a[i].imag();
      }
    }
    QMBED_CUDA(cudaMemcpyAsync(buf, host.data(), nn * w * sizeof(double), cudaMemcpyHostToDevice, stream));
    const int half = (n + 1) / 2;
    const int items = half * half, trips = (items + kJacobiBlockItems - 1) / kJacobiBlockItems;
    const int threads = ((items + trips - 1) / trips + 31) / 32 * 32 + (half + 31) / 32 * 32;
    auto kernel = real ? jacobi_smem_kernel<false> : jacobi_smem_kernel<true>;
    // one limit for every size: handles are solved on several threads
    QMBED_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kJacobiMaxSmem)));
    kernel<<<1, threads, smem, stream>>>(n, buf, buf + first, buf + first + nv, 100);
    QMBED_LAUNCH_CHECK();
    QMBED_CUDA(cudaMemcpyAsync(host.data(), buf + first, (nn * w + nv) * sizeof(double), cudaMemcpyDeviceToHost, stream));
    QMBED_CUDA(cudaStreamSynchronize(stream));
    for (int i = 0; i < n; ++i) values[i] = host[i];
    for (size_t i = 0; i < nn; ++i)
      vectors[i] = real ? C64(host[nv + i], 0.0) : C64(host[nv + 2 * i], host[nv + 2 * i + 1]);
    return;
  }
  const int np = n + (n & 1);
  std::vector<double> host(2 * static_cast<size_t>(np) * np, 0.0);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      host[2 * (static_cast<size_t>(i) * np + j)] = a[static_cast<size_t>(i) * n + j].real();
      host[2 * (static_cast<size_t>(i) * np + j) + 1] = a[static_cast<size_t>(i) * n + j].imag();
    }
  DeviceBuffer dA(host.size() * 8), dV(host.size() * 8);
  QMBED_CUDA(cudaMemcpyAsync(dA.get(), host.data(), host.size() * 8, cudaMemcpyHostToDevice, stream));
  const int threads = std::min(1024, std::max(32, ((np / 2 * np) + 31) / 32 * 32));
  jacobi_kernel<<<1, threads, np * sizeof(int), stream>>>(np, dA.as<double>(), dV.as<double>(), 100);
  QMBED_LAUNCH_CHECK();
  std::vector<double> hv(host.size());
  QMBED_CUDA(cudaMemcpyAsync(host.data(), dA.get(), host.size() * 8, cudaMemcpyDeviceToHost, stream));
  QMBED_CUDA(cudaMemcpyAsync(hv.data(), dV.get(), hv.size() * 8, cudaMemcpyDeviceToHost, stream));
  QMBED_CUDA(cudaStreamSynchronize(stream));
  for (int i = 0; i < n; ++i) values[i] = host[2 * (static_cast<size_t>(i) * np + i)];
  for (int col = 0; col < n; ++col)
    for (int row = 0; row < n; ++row)
      vectors[static_cast<size_t>(col) * n + row] =
          C64(hv[2 * (static_cast<size_t>(col) * np + row)], hv[2 * (static_cast<size_t>(col) * np + row) + 1]);
}

// Ascending eigenpairs of a real symmetric m x m matrix (row-major, symmetrised
// here) on the device; V row-major with eigenvectors as columns.
void device_symmetric_eigen(int m, const std::vector<double>& a, std::vector<double>& values, std::vector<double>& V,
                            BlockOps& ops) {
  std::vector<C64> ac(static_cast<size_t>(m) * m);
  for (int i = 0; i < m; ++i)
    for (int j = 0; j < m; ++j) ac[static_cast<size_t>(i) * m + j] = C64(0.5 * (a[i * m + j] + a[j * m + i]), 0.0);
  std::vector<double> vals;
  std::vector<C64> vecs;
  device_hermitian_eigen(m, ac, vals, vecs, ops);
  std::vector<int> order(m);
  std::iota(order.begin(), order.end(), 0);
  std::stable_sort(order.begin(), order.end(), [&](int l, int r) { return vals[l] < vals[r]; });
  values.assign(m, 0.0);
  V.assign(static_cast<size_t>(m) * m, 0.0);
  for (int q = 0; q < m; ++q) {
    const int col = order[q];
    values[q] = vals[col];
    // eigenvectors of a real matrix are real up to one phase: remove it
    C64 big(0.0, 0.0);
    for (int i = 0; i < m; ++i)
      if (std::abs(vecs[static_cast<size_t>(col) * m + i]) > std::abs(big)) big = vecs[static_cast<size_t>(col) * m + i];
    const C64 phase = std::abs(big) > 0.0 ? std::conj(big) / std::abs(big) : C64(1.0, 0.0);
    for (int i = 0; i < m; ++i) V[static_cast<size_t>(i) * m + q] = (vecs[static_cast<size_t>(col) * m + i] * phase).real();
  }
}


void BlockOps::gram_schmidt_pass(const double* A, uint64_t n, int m, double beta, bool three_term, double* w,
                                 bool cplx, double* before_sq, double* after_sq, C64* last_overlap) {
  if (m <= 0 || n == 0) raise(QMBED_INTERNAL_STATE, "empty Gram-Schmidt pass");
  ensure_coeffs(static_cast<size_t>(m) * 16);
  double* h = coeffs_.as<double>();
  dots_device(A, n, m, w, n, 64, cplx, h);
  ensure_partials(8 * static_cast<size_t>(sms_) + 64);
  const int G = launch_orthogonalize(A, n, m, h, beta, nullptr, three_term ? 1 : 0, w, w, partials_.as<double>(), cplx, sms_, stream_);
  orthogonalize_finish_kernel<<<1, 128, 0, stream_>>>(partials_.as<double>(), G, h + 2 * (m - 1),
                                                      results_.as<double>());
  QMBED_LAUNCH_CHECK();
  QMBED_CUDA(cudaMemcpyAsync(host_results_, results_.get(), 4 * sizeof(double), cudaMemcpyDeviceToHost, stream_));
  sync();
  *before_sq = host_results_[0];
  *after_sq = host_results_[1];
  if (last_overlap) *last_overlap = C64(host_results_[2], host_results_[3]);
}

void BlockOps::lanczos_step(const double* A, uint64_t n, int m, double* w, double* slot, bool cplx) {
  if (fused_.applies(n, m)) {
    fused_.step(A, n, m, w, w, slot, cplx, true, stream_);
    return;
  }
  const double* beta = nullptr;
  double* record = fused_.next_record(m, &beta);
  ensure_coeffs(static_cast<size_t>(m) * 16);
  double* h = coeffs_.as<double>();
  dots_device(A, n, m, w, n, 64, cplx, h);
  ensure_partials(8 * static_cast<size_t>(sms_) + 64);
  const int G = launch_orthogonalize(A, n, m, h, 0.0, beta, 1, w, w, partials_.as<double>(), cplx, sms_, stream_);
  const uint64_t count = slot ? n * (cplx ? 2 : 1) : 0;
  launch_dependent(scale_and_record_kernel, slot ? stream_grid(count, sms_) : 1, kThreads, 0, stream_,
                   partials_.as<double>(), G, m, h + 2 * (m - 1), record, w, slot, count);
  QMBED_LAUNCH_CHECK();
}

// Steps queue up, 8 at first and twice as many each time up to 32, so that a run
// that ends early throws away no more steps than it has used, or seven. A step
// that the queue leaves short (a second pass is due, or the norm is below the
// kernels' 1e-14 or not finite and the next column was not written) is finished
// here if it is the queue's last, whose vector is still in w; else it is made
// again as a queue of one. After such a step queues start over from one, so a
// run of them costs what it would step by step (with queues of 32 throughout,
// each of them threw away up to 31 products).
constexpr int kFirstQueue = 8, kLongestQueue = 32;

void BlockOps::lanczos_run(double* A, uint64_t n, int capacity, double* w, bool cplx,
                           const std::function<void(int)>& product,
                           const std::function<bool(const OrthoRecord&)>& take) {
  auto col = [&](int j) { return A + static_cast<uint64_t>(j) * n * (cplx ? 2 : 1); };
  // every step's buffers before the first: an allocation between them waits for the device
  fused_.reserve(std::min(capacity, kLongestQueue), capacity, stream_);
  if (!fused_.applies(n, capacity)) {
    ensure_coeffs(static_cast<size_t>(capacity) * 16);
    ensure_partials(std::max(panel_partials(n, capacity, sms_), 8 * static_cast<size_t>(sms_) + 64));
  }
  std::vector<OrthoRecord> records;
  double beta = 0.0;
  bool on = true;
  int queue = kFirstQueue;
  for (int index = 0; on && index < capacity;) {
    const int end = std::min(capacity, index + queue);
    fused_.begin(end - index, end, beta, stream_);
    for (int i = index; i < end; ++i) {
      product(i);
      lanczos_step(A, n, i + 1, w, i + 1 < capacity ? col(i + 1) : nullptr, cplx);
    }
    fused_.finish(records, stream_);
    int i = index;
    bool stepwise = false;
    for (; on && i < end; ++i) {
      OrthoRecord& r = records[static_cast<size_t>(i - index)];
      const bool second_due = r.second && !fused_.applies(n, i + 1);
      const bool left_short = second_due || !r.ok;
      stepwise = stepwise || left_short;
      if (left_short && i + 1 < end) break;
      if (second_due) {
        double unused_sq = 0.0, after_sq = 0.0;
        gram_schmidt_pass(A, n, i + 1, 0.0, false, w, cplx, &unused_sq, &after_sq, nullptr);
        r.norm = std::sqrt(std::max(after_sq, 0.0));
      }
      on = take(r);
      beta = r.norm;
      if (on && left_short && i + 1 < capacity) scale_into(w, col(i + 1), n, beta, 64, cplx);
    }
    queue = stepwise ? 1 : std::min(2 * queue, kLongestQueue);
    index = i;
  }
}

void BlockOps::project_out(const double* A, uint64_t n, int m, const double* src, double* w, bool cplx, C64* h,
                           double* src_norm_sq, double* out_norm_sq) {
  if (m <= 0 || n == 0) raise(QMBED_INTERNAL_STATE, "empty projection");
  ensure_coeffs(static_cast<size_t>(m) * 16);
  double* hd = coeffs_.as<double>();
  dots_device(A, n, m, src, n, 64, cplx, hd);
  ensure_partials(8 * static_cast<size_t>(sms_) + 2 * static_cast<size_t>(m) + 64);
  const int G = launch_orthogonalize(A, n, m, hd, 0.0, nullptr, 2, src, w, partials_.as<double>(), cplx, sms_, stream_);
  orthogonalize_finish_kernel<<<1, 128, 0, stream_>>>(partials_.as<double>(), G, hd, results_.as<double>());
  QMBED_LAUNCH_CHECK();
  QMBED_CUDA(cudaMemcpyAsync(host_results_, results_.get(), 2 * sizeof(double), cudaMemcpyDeviceToHost, stream_));
  QMBED_CUDA(cudaMemcpyAsync(host_results_ + 2, hd, static_cast<size_t>(m) * 16, cudaMemcpyDeviceToHost, stream_));
  sync();
  *src_norm_sq = host_results_[0];
  *out_norm_sq = host_results_[1];
  for (int j = 0; j < m; ++j) h[j] = C64(host_results_[2 + 2 * j], host_results_[3 + 2 * j]);
}

// Symmetric tridiagonal eigenproblem (diagonal d, off-diagonal e) by the
// implicit QL method with Wilkinson shifts (Bowdler, Martin, Reinsch and
// Wilkinson, Numer. Math. 11 (1968) 293-306). Rotations are accumulated into
// Z (row-major n x n, Z[k * n + c]) or, with `first_row`, into its first
// row only (all that Boltzmann weights and spectral measures need). Returns ascending values
// with the columns permuted alike.
void tridiagonal_eigen(std::vector<double> d, std::vector<double> e, bool first_row, std::vector<double>& values,
                       std::vector<double>& V) {
  const int n = static_cast<int>(d.size());
  const int rows = first_row ? 1 : n;
  std::vector<double> Z(static_cast<size_t>(rows) * n, 0.0);
  for (int k = 0; k < rows; ++k) Z[static_cast<size_t>(k) * n + k] = 1.0;
  e.resize(static_cast<size_t>(n), 0.0);
  for (int l = 0; l < n; ++l) {
    for (int sweep = 0;; ++sweep) {
      int m = l;
      for (; m + 1 < n; ++m)
        if (std::fabs(e[m]) <= 2.220446049250313e-16 * (std::fabs(d[m]) + std::fabs(d[m + 1]))) break;
      if (m == l) break;
      if (sweep == 60) raise(QMBED_INTERNAL_STATE, "tridiagonal eigensolver did not converge");
      double g = (d[l + 1] - d[l]) / (2.0 * e[l]);
      double r = std::hypot(g, 1.0);
      g = d[m] - d[l] + e[l] / (g + std::copysign(r, g));
      double s = 1.0, c = 1.0, p = 0.0;
      bool deflated = false;
      for (int i = m - 1; i >= l; --i) {
        const double f = s * e[i], b = c * e[i];
        r = std::hypot(f, g);
        e[i + 1] = r;
        if (r == 0.0) {  // underflow: split the matrix here and restart
          d[i + 1] -= p;
          e[m] = 0.0;
          deflated = true;
          break;
        }
        s = f / r;
        c = g / r;
        g = d[i + 1] - p;
        r = (d[i] - g) * s + 2.0 * c * b;
        p = s * r;
        d[i + 1] = g + p;
        g = c * r - b;
        for (int k = 0; k < rows; ++k) {
          double* z = Z.data() + static_cast<size_t>(k) * n;
          const double t = z[i + 1];
          z[i + 1] = s * z[i] + c * t;
          z[i] = c * z[i] - s * t;
        }
      }
      if (deflated) continue;
      d[l] -= p;
      e[l] = g;
      e[m] = 0.0;
    }
  }
  std::vector<int> order(static_cast<size_t>(n));
  for (int i = 0; i < n; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return d[a] < d[b]; });
  values.resize(static_cast<size_t>(n));
  V.assign(static_cast<size_t>(rows) * n, 0.0);
  for (int c = 0; c < n; ++c) {
    values[c] = d[order[c]];
    for (int k = 0; k < rows; ++k) V[static_cast<size_t>(k) * n + c] = Z[static_cast<size_t>(k) * n + order[c]];
  }
}


}  // namespace qmbed
