// Fused Gram-Schmidt step (see gram_schmidt.cuh). Reference behaviour
// (matrixlab-research/QMBED, src/solve/mod.rs): dgks_reorthogonalize
// 1050-1099, orthonormalize_*_with_projection 1520-1642, LanczosIter::next
// 2694-2813, in the classical (block) form of a pass.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "gram_schmidt.cuh"

namespace qmbed {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kMinRows = 128, kMaxRows = 1024;  // rows of a block's slab
constexpr int kMaxColumns = 512;
constexpr unsigned kSpinLimit = 1u << 22;
constexpr double kEps = 2.220446049250313e-16;
constexpr double kDgks = 0.70710678118654752440;  // 1/sqrt(2)
constexpr int kRecordHead = FusedOrtho::kRecordHead;  // before, norm, second, ok, four barrier counters; then 2 m overlaps

struct GridState {
  int status, pad;
  double first[kRecordHead];  // what a record before the first would hold
};

struct OrthoArgs {
  const double* A;
  uint64_t n;
  int m, rows;
  const double* src;
  double* w;
  double* slot;
  int three_term;
  const double* beta;  // previous record's norm, followed by its `second`
  double* record;
  double* partials;    // for each pass [m][G][1 or 2], then [G][2]
  int* status;
};

__device__ __forceinline__ double warp_total(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Barrier of the whole (cooperative) grid on a counter of its own, with a
// bounded wait; false when a block gave up, after which every block leaves.
__device__ bool grid_barrier(unsigned* counter, int* status, unsigned blocks) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    unsigned polls = 0, seen;
    do {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(counter) : "memory");
      if (seen < blocks && ++polls > kSpinLimit) {
        atomicExch(status, 1);
        ok = 0;
      }
    } while (seen < blocks && ok);
  }
  __syncthreads();
  return ok != 0;
}

// Overlaps of the slab's vector with the panel's columns, one warp per column
// (two at once: their reads are in flight together), to this block's partials.
template <bool CPLX>
__device__ __forceinline__ void slab_overlaps(const OrthoArgs& a, const double* ws, uint64_t r0, int rows,
                                              double* partials) {
  constexpr int W = CPLX ? 2 : 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int j = warp; j < a.m; j += 2 * kWarps) {
    const bool pair = j + kWarps < a.m;
    const double* q = a.A + (static_cast<uint64_t>(j) * a.n + r0) * W;
    const double* p = q + (pair ? static_cast<uint64_t>(kWarps) * a.n * W : 0);
    double sum[2][2] = {};
#pragma unroll 4
    for (int r = lane; r < rows; r += 32) {
      if (CPLX) {
        const double2 y = reinterpret_cast<const double2*>(ws)[r];
        const double2 x = reinterpret_cast<const double2*>(q)[r], z = reinterpret_cast<const double2*>(p)[r];
        sum[0][0] += x.x * y.x + x.y * y.y;
        sum[0][1] += x.x * y.y - x.y * y.x;
        sum[1][0] += z.x * y.x + z.y * y.y;
        sum[1][1] += z.x * y.y - z.y * y.x;
      } else {
        sum[0][0] += q[r] * ws[r];
        sum[1][0] += p[r] * ws[r];
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const double sr = warp_total(sum[h][0]), si = CPLX ? warp_total(sum[h][1]) : 0.0;
      if (lane == 0 && (h == 0 || pair)) {
        double* to = partials + (static_cast<size_t>(j + h * kWarps) * gridDim.x + blockIdx.x) * W;
        to[0] = sr;
        if (CPLX) to[1] = si;
      }
    }
  }
}

// A block owns `rows` consecutive rows; its part of the vector stays in shared
// memory through both passes. Overlaps: one warp per column over the slab,
// partial sums to global memory, and after the barrier every block adds the
// partials of all columns in the same fixed order (so all blocks hold the
// same overlaps without a second launch). Subtraction: thread groups share a
// row's columns when the slab has fewer rows than the block threads.
//
// When the step before made a second pass, this one most likely does: the
// second pass's overlaps are then taken along with the first one's norms, in
// front of the same barrier (and left unused if the test says otherwise; the
// results do not depend on it).
//
// Latency-bound by the barriers, the panel reads between them and the sums of
// the partials (the panels it serves fit the L2; keeping a block's slab of the
// panel in shared memory changed nothing). Measured (B200) at 9252 rows and up
// to 44 columns with the second pass: 15.5 us on
// the device's own time, 19.9 us with the second pass behind barriers of its
// own, an arrival count that the last block resets and one column at a time; as
// nine launches (16 us of kernels) and two host round trips about 100 us a step.
// Slabs of 64 rows 17.2 us, of 256 15.6; 1024 threads 17.2.
template <bool CPLX>
__global__ void __launch_bounds__(kThreads, 1) ortho_fused_kernel(const __grid_constant__ OrthoArgs a) {
  constexpr int W = CPLX ? 2 : 1;
  extern __shared__ __align__(16) double smem[];
  double* ws = smem;                     // rows x W
  double* hs = ws + a.rows * W;          // m x W
  double* part = hs + a.m * W;           // kThreads x W
  __shared__ double red[kWarps][2];
  __shared__ double total[2];
  const unsigned G = gridDim.x;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t r0 = static_cast<uint64_t>(blockIdx.x) * a.rows;
  const int rows = static_cast<int>(min(static_cast<uint64_t>(a.rows), a.n - r0));
  const size_t pass_size = static_cast<size_t>(a.m) * G * W + 2 * static_cast<size_t>(G);
  unsigned* counters = reinterpret_cast<unsigned*>(a.record + 4);
  const bool ahead = __ldcg(a.beta + 1) != 0.0;
  if (__ldcg(a.status) != 0) return;  // a step before this one gave up
  for (int t = threadIdx.x; t < rows * W; t += kThreads) ws[t] = a.src[r0 * W + t];
  __syncthreads();
  double before = 0.0, after = 0.0;
  bool second = false;
  for (int pass = 0; pass < 2; ++pass) {
    double* partials = a.partials + pass * pass_size;
    double* norms = partials + pass_size - 2 * static_cast<size_t>(G);
    if (pass == 0 || !ahead) {
      slab_overlaps<CPLX>(a, ws, r0, rows, partials);
      if (!grid_barrier(counters + 2 * pass, a.status, G)) return;
    }
    // four columns of a warp at once
    for (int j0 = warp; j0 < a.m; j0 += 4 * kWarps) {
      double sum[4][W] = {};
#pragma unroll 2
      for (unsigned b = lane; b < G; b += 32) {
#pragma unroll
        for (int h = 0; h < 4; ++h) {
          if (j0 + h * kWarps < a.m) {
            const double* p = partials + (static_cast<size_t>(j0 + h * kWarps) * G + b) * W;
#pragma unroll
            for (int c = 0; c < W; ++c) sum[h][c] += __ldcg(p + c);
          }
        }
      }
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        const int j = j0 + h * kWarps;
#pragma unroll
        for (int c = 0; c < W; ++c) {
          const double v = warp_total(sum[h][c]);
          if (lane == 0 && j < a.m) {
            hs[j * W + c] = v;
            if (pass == 0 && blockIdx.x == 0) a.record[kRecordHead + 2 * j + c] = v;
          }
        }
      }
    }
    __syncthreads();
    const int groups = a.rows >= kThreads ? 1 : kThreads / a.rows;  // a.rows is a power of two
    const int group = groups > 1 ? static_cast<int>(threadIdx.x) / a.rows : 0;
    const double alpha = hs[(a.m - 1) * W];
    const double beta = a.three_term ? __ldcg(a.beta) : 0.0;
    double bs = 0.0, as = 0.0;
    for (int base = 0; base < rows; base += kThreads) {
      const int r = groups > 1 ? static_cast<int>(threadIdx.x) % a.rows : base + static_cast<int>(threadIdx.x);
      double sa = 0.0, sb = 0.0;
      if (r < rows) {
        const int from = a.m * group / groups, to = a.m * (group + 1) / groups;
        const double* q = a.A + (r0 + r) * W;
#pragma unroll 8
        for (int j = from; j < to; ++j) {
          if (CPLX) {
            const double2 x = *reinterpret_cast<const double2*>(q + static_cast<uint64_t>(j) * a.n * 2);
            const double hr = hs[2 * j], hi = hs[2 * j + 1];
            sa += hr * x.x - hi * x.y;
            sb += hr * x.y + hi * x.x;
          } else {
            sa += hs[j] * q[static_cast<uint64_t>(j) * a.n];
          }
        }
      }
      if (groups > 1) {
        part[threadIdx.x * W] = sa;
        if (CPLX) part[threadIdx.x * W + 1] = sb;
        __syncthreads();
        if (group == 0) {
          for (int g = 1; g < groups; ++g) {
            sa += part[(g * a.rows + threadIdx.x) * W];
            if (CPLX) sb += part[(g * a.rows + threadIdx.x) * W + 1];
          }
        }
      }
      if (r < rows && group == 0) {
        double wa = ws[r * W], wb = CPLX ? ws[r * W + 1] : 0.0;
        if (pass == 0) {
          double ba = wa, bb = wb;
          if (a.three_term) {
            const double* last = a.A + (static_cast<uint64_t>(a.m - 1) * a.n + r0 + r) * W;
            ba -= alpha * last[0];
            if (CPLX) bb -= alpha * last[1];
            if (a.m > 1) {
              const double* prev = last - a.n * W;
              ba -= beta * prev[0];
              if (CPLX) bb -= beta * prev[1];
            }
          }
          bs += ba * ba + bb * bb;
        }
        wa -= sa;
        wb -= sb;
        as += wa * wa + wb * wb;
        ws[r * W] = wa;
        if (CPLX) ws[r * W + 1] = wb;
      }
      if (groups > 1) break;
    }
    bs = warp_total(bs);
    as = warp_total(as);
    if (lane == 0) {
      red[warp][0] = bs;
      red[warp][1] = as;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
      double s = 0.0;
      for (int q = 0; q < kWarps; ++q) s += red[q][threadIdx.x];
      norms[2 * blockIdx.x + threadIdx.x] = s;
    }
    if (pass == 0 && ahead) slab_overlaps<CPLX>(a, ws, r0, rows, partials + pass_size);
    if (!grid_barrier(counters + 2 * pass + 1, a.status, G)) return;
    if (warp < 2) {
      double s = 0.0;
#pragma unroll 4
      for (unsigned b = lane; b < G; b += 32) s += __ldcg(norms + 2 * b + warp);
      s = warp_total(s);
      if (lane == 0) total[warp] = s;
    }
    __syncthreads();
    after = sqrt(fmax(total[1], 0.0));
    if (pass == 0) {
      before = sqrt(fmax(total[0], 0.0));
      second = before > kEps && after <= kDgks * before;
      if (!second) break;
    }
  }
  const bool ok = isfinite(after) && after > 1.0e-14;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    a.record[0] = before;
    a.record[1] = after;
    a.record[2] = second ? 1.0 : 0.0;
    a.record[3] = ok ? 1.0 : 0.0;
  }
  double* out = a.slot && ok ? a.slot : a.w;
  const double divisor = ok ? after : 1.0;
  for (int t = threadIdx.x; t < rows * W; t += kThreads) out[r0 * W + t] = ws[t] / divisor;
}

size_t smem_bytes(int rows, int m, bool cplx) {
  return static_cast<size_t>(rows + m + kThreads) * (cplx ? 16 : 8);
}

int slab_rows(uint64_t n, int sms) {
  int rows = kMinRows;
  while (rows < kMaxRows && static_cast<uint64_t>(rows) * sms < n) rows *= 2;
  return rows;
}

}  // namespace

FusedOrtho::~FusedOrtho() {
  if (host_) cudaFreeHost(host_);
}

bool FusedOrtho::applies(uint64_t n, int m) const {
  return n > 0 && m >= 1 && m <= kMaxColumns && n <= static_cast<uint64_t>(kMaxRows) * sms_;
}

void FusedOrtho::reserve(int steps, int m, cudaStream_t stream) {
  const size_t bytes = sizeof(GridState) + static_cast<size_t>(steps) * (kRecordHead + 2 * m) * sizeof(double);
  // the fused kernel's partial sums; wider panels take other kernels, which have their own
  const size_t part = 2 * (static_cast<size_t>(std::min(m, kMaxColumns)) * 2 + 2) * sms_ * sizeof(double);
  if (state_.bytes() < bytes || partials_.bytes() < part) {
    QMBED_CUDA(cudaStreamSynchronize(stream));
    if (state_.bytes() < bytes) state_.allocate(bytes);
    if (partials_.bytes() < part) partials_.allocate(part);
  }
  if (host_bytes_ < bytes) {
    if (host_) cudaFreeHost(host_);
    host_ = nullptr;
    QMBED_CUDA(cudaMallocHost(&host_, bytes));
    host_bytes_ = bytes;
  }
}

void FusedOrtho::begin(int steps, int m, double beta, cudaStream_t stream) {
  reserve(steps, m, stream);
  steps_ = steps;
  cap_ = kRecordHead + 2 * m;
  count_ = 0;
  columns_.clear();
  const size_t bytes = sizeof(GridState) + static_cast<size_t>(steps) * cap_ * sizeof(double);
  GridState head{};
  head.first[1] = beta;
  std::memcpy(host_, &head, sizeof head);
  QMBED_CUDA(cudaMemcpyAsync(state_.get(), host_, sizeof head, cudaMemcpyHostToDevice, stream));
  QMBED_CUDA(cudaMemsetAsync(state_.as<GridState>() + 1, 0, bytes - sizeof head, stream));  // the barriers' counters
}

double* FusedOrtho::next_record(int m, const double** previous_norm) {
  if (count_ >= steps_ || kRecordHead + 2 * m > cap_)
    raise(QMBED_INTERNAL_STATE, "Gram-Schmidt step outside its run");
  GridState* head = state_.as<GridState>();
  double* record = reinterpret_cast<double*>(head + 1) + static_cast<size_t>(count_) * cap_;
  *previous_norm = count_ > 0 ? record - cap_ + 1 : head->first + 1;
  columns_.push_back(m);
  ++count_;
  return record;
}

void FusedOrtho::step(const double* A, uint64_t n, int m, const double* src, double* w, double* slot, bool cplx,
                     bool three_term, cudaStream_t stream) {
  if (!applies(n, m)) raise(QMBED_INTERNAL_STATE, "fused Gram-Schmidt step outside its sizes");
  OrthoArgs a{};
  a.A = A;
  a.n = n;
  a.m = m;
  a.rows = slab_rows(n, sms_);
  a.src = src;
  a.w = w;
  a.slot = slot;
  a.three_term = three_term ? 1 : 0;
  a.record = next_record(m, &a.beta);
  a.partials = partials_.as<double>();
  a.status = &state_.as<GridState>()->status;
  const unsigned grid = static_cast<unsigned>((n + a.rows - 1) / a.rows);
  const size_t smem = smem_bytes(a.rows, m, cplx);
  const void* kernel = cplx ? reinterpret_cast<const void*>(ortho_fused_kernel<true>)
                            : reinterpret_cast<const void*>(ortho_fused_kernel<false>);
  if (smem > 40 * 1024)
    QMBED_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  void* args[] = {&a};
  QMBED_CUDA(cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(kThreads), args, smem, stream));
  QMBED_LAUNCH_CHECK();
}

void FusedOrtho::finish(std::vector<OrthoRecord>& records, cudaStream_t stream) {
  const size_t bytes = sizeof(GridState) + static_cast<size_t>(count_) * cap_ * sizeof(double);
  QMBED_CUDA(cudaMemcpyAsync(host_, state_.get(), bytes, cudaMemcpyDeviceToHost, stream));
  QMBED_CUDA(cudaStreamSynchronize(stream));
  if (reinterpret_cast<const GridState*>(host_)->status != 0)
    raise(QMBED_DEVICE_TIMEOUT, "a Gram-Schmidt step's grid barrier timed out");
  records.resize(static_cast<size_t>(count_));
  const double* base = reinterpret_cast<const double*>(reinterpret_cast<const unsigned char*>(host_) + sizeof(GridState));
  for (int i = 0; i < count_; ++i) {
    const double* r = base + static_cast<size_t>(i) * cap_;
    OrthoRecord& out = records[static_cast<size_t>(i)];
    out.before = r[0];
    out.norm = r[1];
    out.second = r[2] != 0.0;
    out.ok = r[3] != 0.0;
    out.h.resize(static_cast<size_t>(columns_[i]));
    for (int j = 0; j < columns_[i]; ++j) out.h[j] = {r[kRecordHead + 2 * j], r[kRecordHead + 2 * j + 1]};
  }
  count_ = 0;
  columns_.clear();
}

}  // namespace qmbed
