// Structured full-space chain action (diagonal z products + single bit flips).
//
// The action is y[s] = D(s) x[s] + sum_i c_i x[s ^ (1 << i)], with the fused
// epilogue out = alpha y + beta x + gamma p + kappa q of the Chebyshev
// (Clenshaw) step. Vectors move through boxes of 16-byte words in shared
// memory: the flips inside a box read the box (or the thread's own
// registers), the other flips read their partner from global memory, or take
// a pass of their own over boxes that span those bits (flip_box_kernel).
// Chains too short for a box, vectors that start off a 16-byte boundary and
// calls that write over x or q take flip_chain_kernel, one tile per block.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <string>

#include "device_util.cuh"
#include "flipchain.cuh"

namespace qmbed {

namespace {

constexpr int kTileBytes = 64 * 1024;
constexpr int kFlipThreads = 512;
constexpr int kMaxDiagTerms = 256;

template <typename T, bool CPLX>
struct Elem;
template <typename T>
struct Elem<T, false> {
  using type = T;
};
template <>
struct Elem<float, true> {
  using type = float2;
};
template <>
struct Elem<double, true> {
  using type = double2;
};

template <typename T>
__device__ __forceinline__ T scale_add(T acc, T c, T v) { return acc + c * v; }
__device__ __forceinline__ float2 scale_add(float2 acc, float c, float2 v) {
  return make_float2(acc.x + c * v.x, acc.y + c * v.y);
}
__device__ __forceinline__ double2 scale_add(double2 acc, double c, double2 v) {
  return make_double2(acc.x + c * v.x, acc.y + c * v.y);
}
template <typename T>
__device__ __forceinline__ T scaled(T c, T v) { return c * v; }
__device__ __forceinline__ float2 scaled(float c, float2 v) { return make_float2(c * v.x, c * v.y); }
__device__ __forceinline__ double2 scaled(double c, double2 v) { return make_double2(c * v.x, c * v.y); }
template <typename T>
__device__ __forceinline__ T zero_elem() { return T(0); }
template <>
__device__ __forceinline__ float2 zero_elem<float2>() { return make_float2(0.f, 0.f); }
template <>
__device__ __forceinline__ double2 zero_elem<double2>() { return make_double2(0.0, 0.0); }
// kappa * q with complex kappa (real vectors use its real part)
template <typename T>
__device__ __forceinline__ T kappa_times(T kr, T, T q) { return kr * q; }
__device__ __forceinline__ float2 kappa_times(float kr, float ki, float2 q) {
  return make_float2(kr * q.x - ki * q.y, kr * q.y + ki * q.x);
}
__device__ __forceinline__ double2 kappa_times(double kr, double ki, double2 q) {
  return make_double2(kr * q.x - ki * q.y, kr * q.y + ki * q.x);
}
template <typename T>
__device__ __forceinline__ T add(T a, T b) { return a + b; }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }

template <typename E, typename T>
__device__ __forceinline__ E epilogue(E hx, E x, const E* p, const E* q, uint64_t s, T alpha, T beta, T gamma, T kr,
                                      T ki) {
  E o = add(scaled(alpha, hx), scaled(beta, x));
  if (p) o = add(o, scaled(gamma, p[s]));
  if (q) o = add(o, kappa_times(kr, ki, q[s]));
  return o;
}

// D_low[j] = sum over terms with mask inside the low tb bits of c (-1)^popcount(~j & mask)
template <typename T>
__global__ void diag_low_table_kernel(int tb, int nd, const uint64_t* __restrict__ masks,
                                      const double* __restrict__ coefs, T* __restrict__ table) {
  const uint64_t low = (1ull << tb) - 1ull;
  for (uint64_t j = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < (1ull << tb);
       j += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    double d = 0.0;
    for (int k = 0; k < nd; ++k)
      if ((masks[k] & ~low) == 0) d += (__popcll(~j & masks[k]) & 1) ? -coefs[k] : coefs[k];
    table[j] = static_cast<T>(d);
  }
}

// D_high[t] = sum over terms with mask inside the bits >= tb of c (-1)^popcount(~(t << tb) & mask)
__global__ void diag_high_table_kernel(int tb, int sites, int nd, const uint64_t* __restrict__ masks,
                                       const double* __restrict__ coefs, double* __restrict__ table) {
  const uint64_t low = (1ull << tb) - 1ull;
  const uint64_t count = 1ull << (sites - tb);
  for (uint64_t t = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; t < count;
       t += static_cast<uint64_t>(gridDim.x) * blockDim.x) {
    const uint64_t base = t << tb;
    double d = 0.0;
    for (int k = 0; k < nd; ++k)
      if (masks[k] != 0 && (masks[k] & low) == 0) d += (__popcll(~base & masks[k]) & 1) ? -coefs[k] : coefs[k];
    table[t] = d;
  }
}

// One pass over tiles of 2^tb consecutive elements (64 KB): flips of the low tb
// bits read the tile, flips of the higher bits their partner element in global memory.
// D(s) = D_low(j) + D_high(t) + D_cross(s): terms inside the low bits come from
// a 2^tb table computed once, terms inside the high bits once per tile, and
// only the terms spanning both are evaluated per element.
// TB > 0 fixes the tile bits at compile time (the tile loop unrolls); TB = 0
// takes them from `tb` (chains shorter than a tile).
template <typename T, bool CPLX, int TB>
__global__ void __launch_bounds__(kFlipThreads) flip_chain_kernel(int sites, int tb, int nd,
                                                                const uint64_t* __restrict__ masks,
                                                                const double* __restrict__ coefs,
                                                                const T* __restrict__ low_table,
                                                                const double* __restrict__ xcoef,
                                                                const typename Elem<T, CPLX>::type* __restrict__ x,
                                                                typename Elem<T, CPLX>::type* out,
                                                                const typename Elem<T, CPLX>::type* p,
                                                                const typename Elem<T, CPLX>::type* q, T alpha, T beta,
                                                                T gamma, T kr, T ki) {
  using E = typename Elem<T, CPLX>::type;
  extern __shared__ unsigned char smem_raw[];
  E* tile = reinterpret_cast<E*>(smem_raw);
  __shared__ T cx[64];
  __shared__ uint64_t cross_mask[kMaxDiagTerms];
  __shared__ T cross_coef[kMaxDiagTerms];
  __shared__ int n_cross;
  __shared__ T d_high;
  const uint64_t low = (1ull << tb) - 1ull;
  if (threadIdx.x < sites) cx[threadIdx.x] = static_cast<T>(xcoef[threadIdx.x]);
  if (threadIdx.x == 0) {
    int c = 0;
    for (int k = 0; k < nd; ++k)
      if ((masks[k] & low) != 0 && (masks[k] & ~low) != 0) {
        cross_mask[c] = masks[k];
        cross_coef[c] = static_cast<T>(coefs[k]);
        ++c;
      }
    n_cross = c;
  }
  const uint64_t tiles = 1ull << (sites - tb);
  const int count = 1 << tb;
  for (uint64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    const uint64_t base = t << tb;
    __syncthreads();  // previous tile consumed; cross terms ready
    if (threadIdx.x == 0) {
      double d = 0.0;
      for (int k = 0; k < nd; ++k)  // constant terms (mask 0) are in the low table
        if (masks[k] != 0 && (masks[k] & low) == 0) d += (__popcll(~base & masks[k]) & 1) ? -coefs[k] : coefs[k];
      d_high = static_cast<T>(d);
    }
    for (int j = threadIdx.x; j < count; j += blockDim.x) tile[j] = x[base + j];
    __syncthreads();
    const T dh = d_high;
    const int nc = n_cross;
    for (int j = threadIdx.x; j < count; j += blockDim.x) {
      const uint64_t s = base + j;
      T d = dh + __ldg(low_table + j);
      for (int k = 0; k < nc; ++k) d += (__popcll(~s & cross_mask[k]) & 1) ? -cross_coef[k] : cross_coef[k];
      const E xs = tile[j];
      E acc = scaled(d, xs);
      if (TB > 0) {
#pragma unroll
        for (int i = 0; i < TB; ++i) acc = scale_add(acc, cx[i], tile[j ^ (1 << i)]);
      } else {
        for (int i = 0; i < tb; ++i) acc = scale_add(acc, cx[i], tile[j ^ (1 << i)]);
      }
      // high bits: partner elements from global memory, four loads in flight per thread
      int i = TB > 0 ? TB : tb;
      for (; i + 4 <= sites; i += 4) {
        const E y0 = x[s ^ (1ull << i)], y1 = x[s ^ (1ull << (i + 1))];
        const E y2 = x[s ^ (1ull << (i + 2))], y3 = x[s ^ (1ull << (i + 3))];
        acc = scale_add(acc, cx[i], y0);
        acc = scale_add(acc, cx[i + 1], y1);
        acc = scale_add(acc, cx[i + 2], y2);
        acc = scale_add(acc, cx[i + 3], y3);
      }
      for (; i < sites; ++i) acc = scale_add(acc, cx[i], x[s ^ (1ull << i)]);
      out[s] = epilogue(acc, xs, p, q, s, alpha, beta, gamma, kr, ki);
    }
  }
}

int log2_int(int v) {
  int r = 0;
  while ((1 << (r + 1)) <= v) ++r;
  return r;
}

// ---------------------------------------------------------------------------
// Box action (TMA-staged boxes)
// ---------------------------------------------------------------------------
//
// A box holds 2^VB words of 16 bytes in shared memory. The first launch takes
// contiguous boxes (cp.async.bulk): diagonal, the flips of the bits inside the
// word and the box, the flips of `extra` bits above the box by direct reads of
// the partner words, and the whole epilogue. For vectors far beyond the L2 a
// group pass takes the top bits [b0, b0 + G): its box (cp.async.bulk.tensor) is
// a 64-byte run, a batch of the bits above the run and all values of the
// group's bits, so every flip of the group stays inside the box; it adds
// alpha sum c_i x[s ^ 2^i] to out.
//
// What bounds it: every flip of a word costs one 16-byte read per thread,
// from shared memory or from the L2, except those between words that one
// thread owns, so the load pipe is the limit (21 reads and writes per word at
// 22 sites; 62% of its rate) and the L2 serves the direct reads at 13 TB/s. A
// thread owns eight words that differ in the top three bits of the box; each
// serves its diagonal and the flips along those bits as it is read, and is not
// kept, so that many small boxes (16 KB, 128 threads) stay resident. Larger
// boxes with fewer direct reads were slower (64 KB boxes with a group pass at
// 22 sites in complex128: 86 us), persistent blocks with a box pipeline slower
// still (109 us). Measured against the earlier kernels (64 KB tiles with one
// element per thread and step; three passes from 256 MB on): complex128 H.v of
// 22 sites 105 -> 63 to 72 us, 24 sites 440 -> 280 us, complex64 of 24 sites
// 284 -> 122 us, 25 sites 522 -> 286 us, 28 sites 4.1 -> 2.7 ms; with p and q
// 125 -> 84 us at 22 sites in complex128.

constexpr int kBoxMaxWords = 12;  // word bits of a group pass's box (64 KB)
constexpr int kBoxMaxExtra = 16;  // flips above the box by direct reads
constexpr int kBoxLaneBits = 5;
constexpr unsigned kWaitPolls = 1u << 22;

__device__ __forceinline__ uint32_t smem_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(done)
      : "r"(smem_addr(bar)), "r"(parity)
      : "memory");
  return done != 0;
}
// Bounded wait for the phase `parity` of a stage barrier; false on time-out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, unsigned limit = kWaitPolls) {
  for (unsigned polls = 0; polls < limit; ++polls)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}
__device__ __forceinline__ void tensor_load5(void* dst, const CUtensorMap* map, int c1, int c3, int c4, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
      "%6}], [%7];" ::"r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(c1), "r"(0), "r"(c3), "r"(c4), "r"(smem_addr(bar))
      : "memory");
}

// A 16-byte word as the kernels compute on it: four floats (two packed pairs)
// or two doubles.
template <typename T>
struct Word;
template <>
struct Word<float> {
  unsigned long long a, b;
};
template <>
struct Word<double> {
  double a, b;
};
template <typename T>
struct Coef;  // a real factor in the form axpy() takes
template <>
struct Coef<float> {
  using type = unsigned long long;
};
template <>
struct Coef<double> {
  using type = double;
};
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long x, unsigned long long y, unsigned long long z) {
  unsigned long long r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(x), "l"(y), "l"(z));
  return r;
}
__device__ __forceinline__ unsigned long long coef_of(float c) { return pack2(c, c); }
__device__ __forceinline__ double coef_of(double c) { return c; }
__device__ __forceinline__ void axpy(Word<float>& acc, unsigned long long c, const Word<float>& v) {
  acc.a = fma2(c, v.a, acc.a);
  acc.b = fma2(c, v.b, acc.b);
}
__device__ __forceinline__ void axpy(Word<double>& acc, double c, const Word<double>& v) {
  acc.a = fma(c, v.a, acc.a);
  acc.b = fma(c, v.b, acc.b);
}
// A box (or a part of it) whose copy did not arrive within the wait: the thread
// that gave up writes words `first` .. `first + count - 1` itself, from ordinary
// loads. The copy may still be under way; it brings the same bytes, and the
// second wait keeps the block from ending in front of it. Word v of the box is
// word base | (v below run_bits) | (v above them) << shift of x.
template <typename W>
__device__ __noinline__ void fill_words(W* box, const W* x, int first, int count, uint64_t base, int run_bits, int shift,
                                        uint64_t* bar) {
  for (int v = first; v < first + count; ++v)
    box[v] = x[base | static_cast<uint64_t>(v & ((1 << run_bits) - 1)) | (static_cast<uint64_t>(v >> run_bits) << shift)];
  mbar_wait(bar, 0);
}
__device__ __forceinline__ Word<float> load_word(const Word<float>* p) {
  const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(p);
  return Word<float>{v.x, v.y};
}
__device__ __forceinline__ Word<double> load_word(const Word<double>* p) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  return Word<double>{v.x, v.y};
}
__device__ __forceinline__ void store_word(Word<float>* p, const Word<float>& v) {
  *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(v.a, v.b);
}
__device__ __forceinline__ void store_word(Word<double>* p, const Word<double>& v) {
  *reinterpret_cast<double2*>(p) = make_double2(v.a, v.b);
}

// Element layout of a word: EV elements, VBITS = log2(EV) bits of the state
// index inside it.
template <typename T, bool CPLX>
struct WordShape {
  static constexpr int EV = 16 / (static_cast<int>(sizeof(T)) * (CPLX ? 2 : 1));
  static constexpr int VBITS = EV == 1 ? 0 : (EV == 2 ? 1 : 2);
};

// acc += diag(m_0 .. m_EV-1) v, one factor per element
template <bool CPLX>
__device__ __forceinline__ void axpy_diag(Word<float>& acc, const float* m, const Word<float>& v) {
  acc.a = fma2(CPLX ? pack2(m[0], m[0]) : pack2(m[0], m[1]), v.a, acc.a);
  acc.b = fma2(CPLX ? pack2(m[1], m[1]) : pack2(m[2], m[3]), v.b, acc.b);
}
template <bool CPLX>
__device__ __forceinline__ void axpy_diag(Word<double>& acc, const double* m, const Word<double>& v) {
  acc.a = fma(m[0], v.a, acc.a);
  acc.b = fma(CPLX ? m[0] : m[1], v.b, acc.b);
}
// the word with its elements exchanged along state bit `bit` < VBITS
template <bool CPLX>
__device__ __forceinline__ Word<float> flip_inside(const Word<float>& v, int bit) {
  if (CPLX || bit == 1) return Word<float>{v.b, v.a};
  const float2 x = unpack2(v.a), y = unpack2(v.b);
  return Word<float>{pack2(x.y, x.x), pack2(y.y, y.x)};
}
template <bool CPLX>
__device__ __forceinline__ Word<double> flip_inside(const Word<double>& v, int) {
  return Word<double>{v.b, v.a};
}
// kappa q (real vectors: its real part)
template <bool CPLX>
__device__ __forceinline__ Word<float> kappa_word(float kr, float ki, const Word<float>& q) {
  if (!CPLX) return Word<float>{fma2(pack2(kr, kr), q.a, 0ull), fma2(pack2(kr, kr), q.b, 0ull)};
  const float2 x = unpack2(q.a), y = unpack2(q.b);
  return Word<float>{pack2(kr * x.x - ki * x.y, kr * x.y + ki * x.x), pack2(kr * y.x - ki * y.y, kr * y.y + ki * y.x)};
}
template <bool CPLX>
__device__ __forceinline__ Word<double> kappa_word(double kr, double ki, const Word<double>& q) {
  if (!CPLX) return Word<double>{kr * q.a, kr * q.b};
  return Word<double>{kr * q.a - ki * q.b, kr * q.b + ki * q.a};
}

template <typename T>
struct BoxArgs {
  using C = typename Coef<T>::type;
  int sites;
  int extra;      // flips above the box by direct reads
  int b0, G, bb;  // group pass: bits [b0, b0 + G), bb batch bits above the 64-byte run
  int lo;         // group pass: lowest word bit of the box with a flip
  // alpha c of the flips, by value: the multiply-adds take them from constant memory
  C cbit[kBoxMaxWords];    // along a word bit of the box
  C cinside[2];            // inside the word
  C cextra[kBoxMaxExtra];  // above the box
  // Diagonal, split by the bits a term holds: inside the
  // lanes' bits (lane_table, per lane and element), inside the other bits of
  // the box (word_table), above the box (high_table, per box), spanning the
  // lanes' bits and others (terms 0 .. n_lane - 1) and spanning the other box
  // bits and those above (the next n_word terms).
  // Tables and sums in FP64: alpha D + beta is rounded to T once.
  const double* lane_table;
  const double* word_table;
  const double* high_table;
  const uint64_t* span_masks;
  const double* span_coefs;
  int n_lane, n_word;
  const Word<T>* x;
  Word<T>* out;
  const Word<T>* p;
  const Word<T>* q;
  double alpha, beta;
  T gamma, kr, ki;
  unsigned polls;  // limit of a wait on a copy
};

constexpr int kRegBits = 3;  // a thread's eight words differ in the top bits of the box
constexpr int kWordsPerThread = 1 << kRegBits;

// Loads that stay where they are written (before the wait on a box).
__device__ __forceinline__ Word<float> load_early(const Word<float>* p) {
  Word<float> v;
  asm volatile("ld.global.v2.b64 {%0, %1}, [%2];" : "=l"(v.a), "=l"(v.b) : "l"(p));
  return v;
}
__device__ __forceinline__ Word<double> load_early(const Word<double>* p) {
  Word<double> v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.a), "=d"(v.b) : "l"(p));
  return v;
}

// Diagonal of box `id` without the terms that touch the lanes' bits, for the
// words u << kBoxLaneBits.
template <typename T, int VB, int VBITS>
__device__ __forceinline__ double word_diagonal(const BoxArgs<T>& a, uint64_t id, int u) {
  const uint64_t s = (id << (VB + VBITS)) | (static_cast<uint64_t>(u) << (kBoxLaneBits + VBITS));
  double d = a.word_table[u] + a.high_table[id];
  for (int k = a.n_lane; k < a.n_lane + a.n_word; ++k) {
    const double c = a.span_coefs[k];
    d += (__popcll(~s & a.span_masks[k]) & 1) ? -c : c;
  }
  return d;
}

// The diagonal of the thread's words v0 | j << LOW (word v of a box).
template <typename T, bool CPLX, int VB>
struct BoxDiagonal {
  static constexpr int EV = WordShape<T, CPLX>::EV, VBITS = WordShape<T, CPLX>::VBITS;
  double lane[EV];
  uint64_t mask0 = 0;
  double coef0 = 0.0;
  __device__ __forceinline__ explicit BoxDiagonal(const BoxArgs<T>& a) {
#pragma unroll
    for (int e = 0; e < EV; ++e) lane[e] = __ldg(a.lane_table + (threadIdx.x & 31) * EV + e);
    if (a.n_lane > 0) {
      mask0 = __ldg(a.span_masks);
      coef0 = __ldg(a.span_coefs);
    }
  }
  // acc += (alpha D + beta) x of word v
  __device__ __forceinline__ void add(const BoxArgs<T>& a, uint64_t gbase, const double* dword, int v,
                                      const Word<T>& own, Word<T>& acc) const {
    const uint64_t s = (gbase | static_cast<uint64_t>(v)) << VBITS;
    const double du = dword[v >> kBoxLaneBits];
    double m[EV];
#pragma unroll
    for (int e = 0; e < EV; ++e) m[e] = lane[e] + du + ((__popcll(~(s | e) & mask0) & 1) ? -coef0 : coef0);
    for (int k = 1; k < a.n_lane; ++k) {
      const uint64_t mask = __ldg(a.span_masks + k);
      const double c = __ldg(a.span_coefs + k);
#pragma unroll
      for (int e = 0; e < EV; ++e) m[e] += (__popcll(~(s | e) & mask) & 1) ? -c : c;
    }
    T factor[EV];
#pragma unroll
    for (int e = 0; e < EV; ++e) factor[e] = static_cast<T>(a.alpha * m[e] + a.beta);
    axpy_diag<CPLX>(acc, factor, own);
  }
};

// Flips of the thread's words v0 | j << LOW, one eighth of the box after the
// other: wait(j) is called before the j-th eighth is read. A word gives the
// flips of its own bits to its sum (and whatever `own` adds), the flips along
// the register bits to the sums of the seven other eighths, and takes the
// flips along the lower bits from partners in its own eighth. So arithmetic
// starts with the first eighth that arrives, and sum j is complete after
// eighth max(j, j ^ 4). GROUP: only the flips along word bits >= a.lo.
template <typename T, bool CPLX, int VB, bool GROUP, typename Wait, typename Own>
__device__ __forceinline__ void box_flips(const BoxArgs<T>& a, const Word<T>* box, int v0, Wait&& wait, Own&& own_part,
                                          Word<T> (&acc)[kWordsPerThread]) {
  constexpr int VBITS = WordShape<T, CPLX>::VBITS;
  constexpr int LOW = VB - kRegBits;
#pragma unroll
  for (int j = 0; j < kWordsPerThread; ++j) {
    wait(j);
    const int v = v0 | (j << LOW);
    const Word<T> own = load_word(box + v);
    if (!GROUP) {
      own_part(v, own, acc[j]);
#pragma unroll
      for (int i = 0; i < VBITS; ++i) axpy(acc[j], a.cinside[i], flip_inside<CPLX>(own, i));
    }
#pragma unroll
    for (int k = 0; k < kRegBits; ++k)
      if (!GROUP || LOW + k >= a.lo) axpy(acc[j ^ (1 << k)], a.cbit[LOW + k], own);
#pragma unroll
    for (int i = 0; i < LOW; ++i)
      if (!GROUP || i >= a.lo) axpy(acc[j], a.cbit[i], load_word(box + (v ^ (1 << i))));
  }
}

// A block per contiguous box of 2^VB words (8 or 10), the flips of the `extra`
// bits above the box from their partners' words in global memory. They come
// after the box (which keeps the load pipe busier) or, with FAR_FIRST, before
// it: FP32 sums then stay small until the diagonal, usually the largest term,
// joins them, and their rounding error is a quarter smaller.
template <typename T, bool CPLX, int VB, bool FAR_FIRST>
__global__ void __launch_bounds__((1 << VB) / kWordsPerThread) flip_box_kernel(const __grid_constant__ BoxArgs<T> a) {
  using W = Word<T>;
  constexpr int VBITS = WordShape<T, CPLX>::VBITS;
  constexpr int LOW = VB - kRegBits;
  __shared__ __align__(128) W box[1 << VB];
  __shared__ __align__(8) uint64_t full;
  __shared__ double dword[1 << (VB - kBoxLaneBits)];
  const uint64_t id = blockIdx.x;
  await_previous();
  if (threadIdx.x == 0) {
    mbar_init(&full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    mbar_expect_tx(&full, 16u << VB);
    bulk_load(box, a.x + (id << VB), 16u << VB, &full);
  }
  for (int u = threadIdx.x; u < (1 << (VB - kBoxLaneBits)); u += blockDim.x)
    dword[u] = word_diagonal<T, VB, VBITS>(a, id, u);
  __syncthreads();
  const uint64_t gbase = id << VB;
  const uint64_t g0 = gbase | threadIdx.x;
  W acc[kWordsPerThread];
#pragma unroll
  for (int j = 0; j < kWordsPerThread; ++j) {
    if (a.q) acc[j] = kappa_word<CPLX>(a.kr, a.ki, load_word(a.q + g0 + (j << LOW)));
    else acc[j].a = acc[j].b = 0;
  }
  if (a.p) {
#pragma unroll
    for (int j = 0; j < kWordsPerThread; ++j) axpy(acc[j], coef_of(a.gamma), load_word(a.p + g0 + (j << LOW)));
  }
  auto far_flips = [&] {
#pragma unroll 1
    for (int i = 0; i < a.extra; ++i) {
      const W* partner = a.x + (g0 ^ (1ull << (VB + i)));
#pragma unroll
      for (int j = 0; j < kWordsPerThread; ++j) axpy(acc[j], a.cextra[i], load_word(partner + (j << LOW)));
    }
  };
  if (FAR_FIRST) far_flips();
  const BoxDiagonal<T, CPLX, VB> diagonal(a);
  box_flips<T, CPLX, VB, false>(
      a, box, static_cast<int>(threadIdx.x),
      [&](int j) {
        if (j == 0 && !mbar_wait(&full, 0, a.polls))
          fill_words(box, a.x, 0, 1 << VB, gbase, VB, 0, &full);
      },
      [&](int v, const W& own, W& sum) { diagonal.add(a, gbase, dword, v, own, sum); }, acc);
  if (!FAR_FIRST) far_flips();
#pragma unroll
  for (int j = 0; j < kWordsPerThread; ++j) {
    store_word(a.out + g0 + (j << LOW), acc[j]);
  }
}

// A group pass: a block per box of 64 KB (12 word bits), three resident per SM,
// in two trips of eight words per thread. The box arrives in eighths (the top
// three word bits), each on its own barrier, so that a block's arithmetic
// overlaps its own copy: blocks that started together would otherwise load,
// compute and store in step. out is requested before the first wait.
constexpr int kPassTrips = 2;
constexpr int kPassThreads = (1 << kBoxMaxWords) / (kWordsPerThread * kPassTrips);

template <typename T, bool CPLX>
__global__ void __launch_bounds__(kPassThreads, 3) flip_group_kernel(const __grid_constant__ CUtensorMap map,
                                                                     const __grid_constant__ BoxArgs<T> a) {
  using W = Word<T>;
  constexpr int VB = kBoxMaxWords;
  constexpr int VBITS = WordShape<T, CPLX>::VBITS;
  constexpr int LOW = VB - kRegBits;
  constexpr uint32_t kPart = 16u << LOW;  // bytes of an eighth
  extern __shared__ __align__(128) unsigned char smem_raw[];
  W* box = reinterpret_cast<W*>(smem_raw);
  __shared__ __align__(8) uint64_t full[kWordsPerThread];
  // box id = batch block (low bits) | index above the group
  const int run_bits = 2 + a.bb;
  const int batch_shift = a.b0 - VBITS - run_bits;
  const uint64_t blk = blockIdx.x & ((1ull << batch_shift) - 1), above = static_cast<uint64_t>(blockIdx.x) >> batch_shift;
  await_previous();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int j = 0; j < kWordsPerThread; ++j) mbar_init(&full[j], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
#pragma unroll
    for (int j = 0; j < kWordsPerThread; ++j) {
      mbar_expect_tx(&full[j], kPart);
      tensor_load5(box + (j << LOW), &map, static_cast<int>(blk << a.bb), j, static_cast<int>(above), &full[j]);
    }
  }
  __syncthreads();
  const uint64_t gbase = (blk << run_bits) | (above << (a.b0 + a.G - VBITS));
  // global word of box word v
  auto global_word = [&](int v) -> uint64_t {
    return gbase | static_cast<uint64_t>(v & ((1 << run_bits) - 1)) |
           (static_cast<uint64_t>(v >> run_bits) << (a.b0 - VBITS));
  };
#pragma unroll 1
  for (int trip = 0; trip < kPassTrips; ++trip) {
    const int v0 = static_cast<int>(threadIdx.x) | (trip * kPassThreads);
    W acc[kWordsPerThread], before[kWordsPerThread];
#pragma unroll
    for (int j = 0; j < kWordsPerThread; ++j) {
      before[j] = load_early(a.out + global_word(v0 | (j << LOW)));
      acc[j].a = acc[j].b = 0;
    }
    box_flips<T, CPLX, VB, true>(
        a, box, v0,
        [&](int j) {
          if (trip == 0 && !mbar_wait(&full[j], 0, a.polls))
            fill_words(box, a.x, j << LOW, 1 << LOW, gbase, run_bits, a.b0 - VBITS, &full[j]);
        },
        [](int, const W&, W&) {}, acc);
#pragma unroll
    for (int j = 0; j < kWordsPerThread; ++j) {
      axpy(acc[j], coef_of(static_cast<T>(1)), before[j]);
      store_word(a.out + global_word(v0 | (j << LOW)), acc[j]);
    }
  }
}

// Self-test of the bounded stage wait: one thread arms an mbarrier for bytes
// that no copy will deliver and waits `polls` times; status receives 1 when
// the wait gave up.
__global__ void stage_wait_selftest_kernel(unsigned polls, int* status) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x != 0) return;
  mbar_init(&bar, 1);
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  mbar_expect_tx(&bar, 16);
  bool done = false;
  for (unsigned i = 0; i < polls && !done; ++i) done = mbar_try_wait(&bar, 0);
  *status = done ? 0 : 1;
}

PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
  });
  if (!fn) raise(QMBED_CUDA_ERROR, "cuTensorMapEncodeTiled is not available");
  return fn;
}

// Tensor map of the group boxes over x (4-byte units): d0 the 64-byte run
// (R bits), d1 the bits between the run and the group (box: bb of them), d2
// the group's bits below its top three (at most 7), d3 the top three (one
// eighth of a box per copy), d4 the bits above.
CUtensorMap group_map(const void* x, int sites, int esize, int r, int b0, int G, int bb) {
  const int g1 = G - 3;
  const cuuint64_t dims[5] = {static_cast<cuuint64_t>((esize << r) / 4), 1ull << (b0 - r), 1ull << g1, 8ull,
                              1ull << (sites - b0 - G)};
  const cuuint64_t strides[4] = {static_cast<cuuint64_t>(esize) << r, static_cast<cuuint64_t>(esize) << b0,
                                 static_cast<cuuint64_t>(esize) << (b0 + g1), static_cast<cuuint64_t>(esize) << (b0 + G)};
  const cuuint32_t box[5] = {static_cast<cuuint32_t>((esize << r) / 4), 1u << bb, 1u << g1, 1u, 1u};
  const cuuint32_t elem[5] = {1, 1, 1, 1, 1};
  CUtensorMap map;
  const CUresult rc = tensor_map_encoder()(&map, CU_TENSOR_MAP_DATA_TYPE_UINT32, 5, const_cast<void*>(x), dims, strides,
                                           box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (rc != CUDA_SUCCESS) raise(QMBED_CUDA_ERROR, "cuTensorMapEncodeTiled failed with code " + std::to_string(rc));
  return map;
}

// One launch while the partners above the box come from the L2. Vectors from
// 512 MB on (256 MB when p or q stream beside them) take their top nine bits
// in a group pass instead: complex64 H.v of 25 sites (268 MB) 292 us in one
// launch against 307 with a group pass and 631 against 630 at 26 sites; with p
// and q 351 against 329 at 25 sites and 167 against 172 at 24.
constexpr uint64_t kGroupPassBytes = 512ull << 20, kGroupPassBytesPq = 256ull << 20;
// Bits of a group pass (of 7 to 10, 9 is fastest or within 3% of it from 24 to
// 28 sites: longer runs against fewer direct reads) and the most bits read
// directly beside one (a window of 2^10 boxes, 16 MB) before another pass.
constexpr int kGroupBits = 9, kDirectBits = 10;

// QMBED_FLIP_PASSES=single|multi forces flip_chain_kernel or group passes (tests).
BoxPlan box_plan(int sites, int vbits, uint64_t bytes, bool pq) {
  BoxPlan plan;
  const char* env = std::getenv("QMBED_FLIP_PASSES");
  const bool single = env && std::strcmp(env, "single") == 0, multi = env && std::strcmp(env, "multi") == 0;
  const int words = sites - vbits;  // word bits of the whole vector
  if (single || words < 8 || (multi && words <= kBoxMaxWords)) return plan;
  // 4 KB boxes while 16 KB boxes would leave SMs without work
  plan.vb = words >= 17 ? 10 : 8;
  plan.extra = words - plan.vb;
  if (multi) plan.vb = 10;
  // Separate passes used to sum the flips of FP32 vectors from 256 MB on:
  // complex64 of 25 sites has 0.94e-7 of relative error in that form, 0.89e-7
  // with the far flips first (286 us) and 1.19e-7 with them last (258 us).
  // Below, the order of the one-pass kernel had 1.19e-7 at 24 sites, now 1.16e-7.
  plan.far_first = bytes >= (256ull << 20);
  const bool passes = multi || bytes >= (pq ? kGroupPassBytesPq : kGroupPassBytes);
  if (!passes) return plan;
  plan.extra = words - plan.vb;
  do {
    const int g = std::min(plan.extra, kGroupBits);
    plan.groups.push_back(g);
    plan.extra -= g;
  } while (plan.extra > kDirectBits);
  return plan;
}

}  // namespace

FlipChain::FlipChain(const FlipChainDesc& d) : sites_(d.sites), n_diag_(static_cast<int>(d.z_masks.size())) {
  if (sites_ < 1 || sites_ > 40) raise(QMBED_UNSUPPORTED_BACKEND, "the flip-chain action covers 1 to 40 sites");
  if (n_diag_ > kMaxDiagTerms) raise(QMBED_UNSUPPORTED_BACKEND, "too many diagonal products for the flip-chain action");
  diag_masks_.allocate(std::max(n_diag_, 1) * sizeof(uint64_t));
  diag_coefs_.allocate(std::max(n_diag_, 1) * sizeof(double));
  x_coefs_.allocate(64 * sizeof(double));
  // low-bit diagonal tables of the tile kernel (2^tb values of the working
  // precision, at most kTileBytes each): FP64 table first, FP32 table second
  tables_.allocate(2 * static_cast<size_t>(kTileBytes));
  std::vector<double> x(64, 0.0);
  for (int i = 0; i < sites_; ++i) x[i] = d.x_coefs[i];
  if (n_diag_ > 0) {
    QMBED_CUDA(cudaMemcpy(diag_masks_.get(), d.z_masks.data(), n_diag_ * sizeof(uint64_t), cudaMemcpyHostToDevice));
    QMBED_CUDA(cudaMemcpy(diag_coefs_.get(), d.z_coefs.data(), n_diag_ * sizeof(double), cudaMemcpyHostToDevice));
  }
  QMBED_CUDA(cudaMemcpy(x_coefs_.get(), x.data(), 64 * sizeof(double), cudaMemcpyHostToDevice));
  host_diag_masks_ = d.z_masks;
  host_diag_coefs_ = d.z_coefs;
  host_x_ = x;
}

double FlipChain::norm_bound() const {
  double b = 0.0;
  for (double c : host_diag_coefs_) b += std::fabs(c);
  for (double c : host_x_) b += std::fabs(c);
  return b;
}

void FlipChain::apply(int precision, bool cplx, const void* x, void* out, const void* p, const void* q,
                      const FlipStep& step, cudaStream_t stream) const {
  const int esize = (precision == 64 ? 8 : 4) * (cplx ? 2 : 1);
  prepare_tables(stream);
  {
    const int vbits = log2_int(16 / esize);
    const BoxPlan plan = box_plan(sites_, vbits, dim() * static_cast<uint64_t>(esize), p || q);
    auto aligned = [](const void* ptr) { return ptr == nullptr || (reinterpret_cast<uintptr_t>(ptr) & 15) == 0; };
    if (plan.vb > 0 && aligned(x) && aligned(out) && aligned(p) && aligned(q)) {
      const bool over = x == out || (q && q == out);
      if (over && (!plan.groups.empty() || dim() * static_cast<uint64_t>(esize) >= (256ull << 20)))
        raise(QMBED_INVALID_OPTIONS, "the flip-chain action cannot write over x or q");
      if (!over) {
        apply_boxes(precision, cplx, x, out, p, q, step, stream, plan);
        return;
      }
    }
  }
  const int tbits = log2_int(kTileBytes / esize);
  const int tb = std::min(sites_, tbits);
  const uint64_t n = dim();
  int device = 0, sms = 148;
  QMBED_CUDA(cudaGetDevice(&device));
  QMBED_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  const int table_slot = precision == 64 ? 1 : 2;
  void* table = static_cast<unsigned char*>(tables_.get()) + (precision == 64 ? 0 : kTileBytes);
  if (!(tables_ready_ & table_slot) || table_tb_[table_slot - 1] != tb) {
    const int blocks = static_cast<int>(std::min<uint64_t>(((1ull << tb) + 255) / 256, 1024));
    if (precision == 64)
      diag_low_table_kernel<double><<<blocks, 256, 0, stream>>>(tb, n_diag_, diag_masks_.as<uint64_t>(),
                                                                diag_coefs_.as<double>(), static_cast<double*>(table));
    else
      diag_low_table_kernel<float><<<blocks, 256, 0, stream>>>(tb, n_diag_, diag_masks_.as<uint64_t>(),
                                                               diag_coefs_.as<double>(), static_cast<float*>(table));
    QMBED_LAUNCH_CHECK();
    tables_ready_ |= table_slot;
    table_tb_[table_slot - 1] = tb;
  }
  const size_t smem = static_cast<size_t>(esize) << tb;
  const int grid = static_cast<int>(std::max<uint64_t>(1, std::min<uint64_t>(n >> tb, 3ull * sms)));
  auto run = [&](auto ttag, auto ctag) {
    using T = decltype(ttag);
    constexpr bool C = decltype(ctag)::value;
    using E = typename Elem<T, C>::type;
    const T a = static_cast<T>(step.alpha), b = static_cast<T>(step.beta), g = static_cast<T>(step.gamma),
            kr = static_cast<T>(step.kappa_re), ki = static_cast<T>(step.kappa_im);
    // the full-tile width for this element size, known at compile time
    constexpr int kFull = (sizeof(E) == 4) ? 14 : (sizeof(E) == 8 ? 13 : 12);
    auto kernel = tb == kFull ? flip_chain_kernel<T, C, kFull> : flip_chain_kernel<T, C, 0>;
    QMBED_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    kernel<<<grid, kFlipThreads, smem, stream>>>(sites_, tb, n_diag_, diag_masks_.as<uint64_t>(),
                                                 diag_coefs_.as<double>(), static_cast<const T*>(table),
                                                 x_coefs_.as<double>(), static_cast<const E*>(x), static_cast<E*>(out),
                                                 static_cast<const E*>(p), static_cast<const E*>(q), a, b, g, kr, ki);
    QMBED_LAUNCH_CHECK();
  };
  if (precision == 64) cplx ? run(double{}, std::true_type{}) : run(double{}, std::false_type{});
  else cplx ? run(float{}, std::true_type{}) : run(float{}, std::false_type{});
}

}  // namespace qmbed

namespace qmbed {

namespace {

// QMBED_FLIP_WAIT_POLLS bounds the waits on box copies (tests: 0 gives every copy up at once).
unsigned wait_polls() {
  const char* env = std::getenv("QMBED_FLIP_WAIT_POLLS");
  return env ? static_cast<unsigned>(std::strtoul(env, nullptr, 10)) : kWaitPolls;
}

template <typename T>
typename Coef<T>::type host_coef(double c) {
  const T v = static_cast<T>(c);
  typename Coef<T>::type r;
  for (size_t i = 0; i < sizeof(r) / sizeof(T); ++i)
    std::memcpy(reinterpret_cast<unsigned char*>(&r) + i * sizeof(T), &v, sizeof(T));
  return r;
}

template <typename T, bool C>
void launch_box_plan(BoxArgs<T> base, const BoxPlan& plan, double alpha, const std::vector<double>& xc, int sites,
                     cudaStream_t stream) {
  constexpr int VBITS = WordShape<T, C>::VBITS;
  base.sites = sites;
  base.extra = plan.extra;
  for (int i = 0; i < plan.vb; ++i) base.cbit[i] = host_coef<T>(alpha * xc[VBITS + i]);
  for (int i = 0; i < VBITS; ++i) base.cinside[i] = host_coef<T>(alpha * xc[i]);
  for (int i = 0; i < plan.extra; ++i) base.cextra[i] = host_coef<T>(alpha * xc[VBITS + plan.vb + i]);
  const unsigned boxes = 1u << (sites - VBITS - plan.vb);
  if (plan.vb == 8) launch_dependent(flip_box_kernel<T, C, 8, false>, boxes, 32, 0, stream, base);
  else if (plan.far_first) launch_dependent(flip_box_kernel<T, C, 10, sizeof(T) == 4>, boxes, 128, 0, stream, base);
  else launch_dependent(flip_box_kernel<T, C, 10, false>, boxes, 128, 0, stream, base);
  QMBED_LAUNCH_CHECK();
  if (plan.groups.empty()) return;
  constexpr int kSmem = 16 << kBoxMaxWords;
  auto group = flip_group_kernel<T, C>;
  QMBED_CUDA(cudaFuncSetAttribute(group, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
  int b0 = VBITS + plan.vb + plan.extra;
  for (int G : plan.groups) {
    BoxArgs<T> g = base;
    // a box's eighths are its group's top three bits: a smaller group takes
    // the bits below it along, without their flips
    const int skip = std::max(0, 3 - G);
    g.b0 = b0 - skip;
    g.G = G + skip;
    g.bb = kBoxMaxWords - 2 - g.G;
    g.lo = kBoxMaxWords - G;
    for (int i = g.lo; i < kBoxMaxWords; ++i) g.cbit[i] = host_coef<T>(alpha * xc[b0 + i - g.lo]);
    const CUtensorMap map =
        group_map(base.x, sites, static_cast<int>(sizeof(T)) * (C ? 2 : 1), VBITS + 2, g.b0, g.G, g.bb);
    launch_dependent(group, 1u << (sites - VBITS - kBoxMaxWords), kPassThreads, kSmem, stream, map, g);
    QMBED_LAUNCH_CHECK();
    b0 += G;
  }
}

}  // namespace

// The diagonal's tables for boxes of 2^vb words with vbits state bits inside a
// word; complete before any stream can use them.
const FlipChain::BoxTables& FlipChain::box_tables(int vbits, int vb, cudaStream_t stream) const {
  std::lock_guard<std::mutex> lock(tables_mu_);
  BoxTables& t = box_tables_[vbits][vb == 10 ? 1 : 0];
  if (!t.ready) build_box_tables(vbits, vb, stream, t);
  return t;
}

// The tables of every element size, on the first call: a later one may be under
// capture, where nothing can be allocated.
void FlipChain::prepare_tables(cudaStream_t stream) const {
  std::lock_guard<std::mutex> lock(tables_mu_);
  if (tables_prepared_) return;
  for (int vbits = 0; vbits < 3; ++vbits) {
    const int vb = box_plan(sites_, vbits, 0, false).vb;
    BoxTables& t = box_tables_[vbits][vb == 10 ? 1 : 0];
    if (vb > 0 && !t.ready) build_box_tables(vbits, vb, stream, t);
  }
  tables_prepared_ = true;
}

void FlipChain::build_box_tables(int vbits, int vb, cudaStream_t stream, BoxTables& t) const {
  const uint64_t lanes = (1ull << (kBoxLaneBits + vbits)) - 1, in_box = (1ull << (vb + vbits)) - 1;
  const uint64_t words = in_box & ~lanes;
  const int n_lanes = 1 << (kBoxLaneBits + vbits), n_words = 1 << (vb - kBoxLaneBits);
  std::vector<double> table(static_cast<size_t>(n_lanes + n_words), 0.0);
  std::vector<uint64_t> masks[2];
  std::vector<double> coefs[2];
  for (size_t k = 0; k < host_diag_masks_.size(); ++k) {
    const uint64_t m = host_diag_masks_[k];
    const double c = host_diag_coefs_[k];
    auto sign = [&](uint64_t s) { return (__builtin_popcountll(~s & m) & 1) ? -c : c; };
    if ((m & ~lanes) == 0) {
      for (int i = 0; i < n_lanes; ++i) table[i] += sign(static_cast<uint64_t>(i));
    } else if ((m & ~words) == 0) {
      for (int u = 0; u < n_words; ++u) table[n_lanes + u] += sign(static_cast<uint64_t>(u) << (kBoxLaneBits + vbits));
    } else if ((m & in_box) != 0) {
      const int list = (m & lanes) != 0 ? 0 : 1;
      masks[list].push_back(m);
      coefs[list].push_back(c);
    }
  }
  t.n_lane = static_cast<int>(masks[0].size());
  t.n_word = static_cast<int>(masks[1].size());
  masks[0].insert(masks[0].end(), masks[1].begin(), masks[1].end());
  coefs[0].insert(coefs[0].end(), coefs[1].begin(), coefs[1].end());
  const uint64_t boxes = 1ull << (sites_ - vbits - vb);
  // [span masks][span coefs][lane table, word table][high table], FP64
  const size_t spans = std::max<size_t>(masks[0].size(), 1) * 8;
  t.at_coefs = spans;
  t.at_table = 2 * spans;
  t.at_words = t.at_table + static_cast<size_t>(n_lanes) * 8;
  t.at_high = t.at_words + static_cast<size_t>(n_words) * 8;
  std::vector<unsigned char> image(t.at_high, 0);
  if (!masks[0].empty()) {
    std::memcpy(image.data(), masks[0].data(), masks[0].size() * 8);
    std::memcpy(image.data() + t.at_coefs, coefs[0].data(), coefs[0].size() * 8);
  }
  std::memcpy(image.data() + t.at_table, table.data(), table.size() * 8);
  t.buf.allocate(t.at_high + boxes * 8);
  QMBED_CUDA(cudaMemcpyAsync(t.buf.get(), image.data(), image.size(), cudaMemcpyHostToDevice, stream));
  const int blocks = static_cast<int>(std::min<uint64_t>((boxes + 255) / 256, 4096));
  diag_high_table_kernel<<<blocks, 256, 0, stream>>>(vb + vbits, sites_, n_diag_, diag_masks_.as<uint64_t>(),
                                                     diag_coefs_.as<double>(),
                                                     reinterpret_cast<double*>(t.buf.as<unsigned char>() + t.at_high));
  QMBED_LAUNCH_CHECK();
  QMBED_CUDA(cudaStreamSynchronize(stream));
  t.ready = true;
}

void FlipChain::apply_boxes(int precision, bool cplx, const void* x, void* out, const void* p, const void* q,
                            const FlipStep& step, cudaStream_t stream, const BoxPlan& plan) const {
  const int esize = (precision == 64 ? 8 : 4) * (cplx ? 2 : 1);
  const BoxTables& t = box_tables(log2_int(16 / esize), plan.vb, stream);
  unsigned char* base = t.buf.as<unsigned char>();
  auto run = [&](auto ttag, auto ctag) {
    using T = decltype(ttag);
    BoxArgs<T> a{};
    a.lane_table = reinterpret_cast<const double*>(base + t.at_table);
    a.word_table = reinterpret_cast<const double*>(base + t.at_words);
    a.high_table = reinterpret_cast<const double*>(base + t.at_high);
    a.span_masks = reinterpret_cast<const uint64_t*>(base);
    a.span_coefs = reinterpret_cast<const double*>(base + t.at_coefs);
    a.n_lane = t.n_lane;
    a.n_word = t.n_word;
    a.x = static_cast<const Word<T>*>(x);
    a.out = static_cast<Word<T>*>(out);
    a.p = static_cast<const Word<T>*>(p);
    a.q = static_cast<const Word<T>*>(q);
    a.alpha = step.alpha;
    a.beta = step.beta;
    a.gamma = static_cast<T>(step.gamma);
    a.kr = static_cast<T>(step.kappa_re);
    a.ki = static_cast<T>(step.kappa_im);
    a.polls = wait_polls();
    launch_box_plan<T, decltype(ctag)::value>(a, plan, step.alpha, host_x_, sites_, stream);
  };
  if (precision == 64) cplx ? run(double{}, std::true_type{}) : run(double{}, std::false_type{});
  else cplx ? run(float{}, std::true_type{}) : run(float{}, std::false_type{});
}

}  // namespace qmbed

namespace qmbed {

int flip_stage_wait_selftest(int device) {
  QMBED_CUDA(cudaSetDevice(device));
  DeviceBuffer status(sizeof(int));
  QMBED_CUDA(cudaMemset(status.get(), 0xff, sizeof(int)));
  stage_wait_selftest_kernel<<<1, 32>>>(1u << 10, status.as<int>());
  QMBED_LAUNCH_CHECK();
  int host = -1;
  QMBED_CUDA(cudaMemcpy(&host, status.get(), sizeof(int), cudaMemcpyDeviceToHost));
  return host;
}

}  // namespace qmbed
