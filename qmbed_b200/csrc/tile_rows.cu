// Assembly and actions of stored rows in tiles of 32 (see tile_rows.cuh).
//
// Reference behaviour (matrixlab-research/QMBED):
//   OperatorBuilder::build (column streaming, coalesce, drop |v| <= eps) src/operator/mod.rs:2091-2216
//   index_transition (sqrt(R_src/R_tgt) conj(phase))                     src/basis/mod.rs:1561-1580
//   apply / apply_real                                                   src/operator/mod.rs:1401-1548
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <set>
#include <type_traits>
#include <vector>

#include "device_util.cuh"
#include "krylov.cuh"
#include "tile_rows.cuh"

namespace qmbed {

namespace {

constexpr double kEps = 2.220446049250313e-16;
constexpr uint32_t kNoEntry = 0xffffffffu;
constexpr int kMaxRowSlots = 64;
constexpr int kMaxTableCodes = 2048;
constexpr int kMaxStoredValues = 1024;  // distinct values of a packed real operator
constexpr int kFillThreads = 256;
constexpr int kMaxProgramSmem = 96 * 1024;  // products and fence keys in shared memory
constexpr int kSumSlots = 4096;  // dictionary of coalesced values (open addressing)

// One off-diagonal site pair on the device.
struct RowGroup {
  uint64_t flip;
  uint16_t amp[4];  // amplitude index per digit pattern d_i | d_j << 1
  uint8_t i, j, nz, pad[5];
};
struct RowPair {  // diagonal products of two sites
  double re[4], im[4];
  int i, j;
};

struct FillArgs {
  SectorParams p;
  uint64_t mask, dim;
  int direct;
  const uint64_t* states;
  const uint16_t* orbits;
  const uint64_t* binom;
  const uint8_t* class_of;  // R -> orbit class
  const uint64_t* fences;
  int n_fences;
  uint64_t fence_seg;
  int fence_levels;
  const RowGroup* groups;
  int n_groups;
  const RowPair* pairs;
  int n_pairs;
  const FlipTerm* terms;  // diagonal products of three or more sites
  int n_terms;
  int cplx;           // complex rows: interleaved diagonal
  int phases, classes, col_bits, codes;
  const double2* values;   // per code, without the orbit factor
  const double* inv_sqrt;  // [R] 1/sqrt(R), [257 + R] sqrt(R)
  int max_slots;
  const uint32_t* tile_ptr;
  uint32_t* entries;
  double* diag64;
  float* diag32;
  unsigned long long* nnz;
  unsigned int* used;         // per (amplitude, phase): an uncoalesced entry has this value
  unsigned long long* sums;   // dictionary of coalesced values (real rows)
  int* flags;
};

__device__ __forceinline__ int group_digits(const RowGroup& g, uint64_t s) {
  return static_cast<int>((s >> g.i) & 1) | (static_cast<int>((s >> g.j) & 1) << 1);
}

// Active groups g0 .. g0 + 63 of a row state.
__device__ __forceinline__ uint64_t active_groups(const RowGroup* groups, int n_groups, int g0, uint64_t s) {
  uint64_t active = 0;
  const int gn = min(64, n_groups - g0);
  for (int g = 0; g < gn; ++g) {
    const RowGroup& grp = groups[g0 + g];
    active |= static_cast<uint64_t>((grp.nz >> group_digits(grp, s)) & 1) << g;
  }
  return active;
}

// Slots of each tile: the most active groups of its 32 rows.
__global__ void __launch_bounds__(kFillThreads) tile_width_kernel(const FillArgs a, uint32_t* widths, int* max_width) {
  extern __shared__ __align__(16) unsigned char smem[];
  RowGroup* groups = reinterpret_cast<RowGroup*>(smem);
  for (int g = threadIdx.x; g < a.n_groups; g += blockDim.x) groups[g] = a.groups[g];
  __syncthreads();
  const uint64_t tiles = (a.dim + 31) / 32;
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (blockDim.x >> 5);
  const int lane = threadIdx.x & 31;
  int top = 0;
  for (uint64_t t = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; t < tiles; t += warps) {
    const uint64_t r = t * 32 + lane;
    int n = 0;
    if (r < a.dim) {
      const uint64_t s = a.direct ? r : a.states[r];
      for (int g0 = 0; g0 < a.n_groups; g0 += 64) n += __popcll(active_groups(groups, a.n_groups, g0, s));
    }
    n = __reduce_max_sync(0xffffffffu, n);
    if (lane == 0) widths[t] = static_cast<uint32_t>(n);
    top = max(top, n);
  }
  if (lane == 0 && top > 0) atomicMax(max_width, top);
}

// Orbit minimum of `t` with the group element that reaches it, on the narrow
// word S (u32 for chains of up to 32 sites: a rotation by one site is three
// instructions). The minimum over a sequence of rotations is taken first and
// the first shift that reaches it is tracked only when characters depend on
// it (SHIFT). Ties keep the earlier element, as canonicalize().
template <typename S, bool SHIFT>
__device__ __forceinline__ void orbit_minimum(S t, const SectorParams& p, S mask, S& rep, int& shift, bool& neg) {
  const int n = p.sites, translations = p.has_momentum ? n : 1;
  rep = t;
  shift = 0;
  neg = false;
  for (int inv = 0; inv < (p.inversion != 0 ? 2 : 1); ++inv) {
    const S base = inv ? static_cast<S>(~t & mask) : t;
    for (int refl = 0; refl < (p.parity != 0 ? 2 : 1); ++refl) {
      S r = refl ? static_cast<S>(reflect_state(static_cast<uint64_t>(base), n)) : base;
      S best = r;
      int at = 0;
#pragma unroll 4
      for (int s = 1; s < translations; ++s) {
        r = static_cast<S>(((r << 1) & mask) | (r >> (n - 1)));
        if (SHIFT) {
          const bool less = r < best;
          best = less ? r : best;
          at = less ? s : at;
        } else {
          best = min(best, r);
        }
      }
      if (best < rep) {
        rep = best;
        shift = at;
        neg = (refl && p.parity < 0) != (inv && p.inversion < 0);
      }
    }
  }
}

// One warp per tile, one lane per row: pops up to four active groups per lane
// and round, resolves their targets together (orbit minimum, then fence keys
// in shared memory and the last levels of the search in flight at once) and
// writes the entries straight to their slots, with the diagonal beside. A
// second look at the row's columns (kept in shared memory) counts the
// coalesced entries. One pass over the transitions: the previous assembly
// expanded every row three times (Hermiticity, count, fill) from one thread
// with its row list in local memory.
template <typename S, bool SHIFT>
__global__ void __launch_bounds__(kFillThreads) tile_fill_kernel(const __grid_constant__ FillArgs a) {
  constexpr int U = 4;
  extern __shared__ __align__(16) unsigned char smem[];
  RowGroup* groups = reinterpret_cast<RowGroup*>(smem);
  RowPair* pairs = reinterpret_cast<RowPair*>(groups + a.n_groups);
  uint64_t* fence = reinterpret_cast<uint64_t*>(pairs + a.n_pairs);
  uint32_t* stage_all = reinterpret_cast<uint32_t*>(fence + a.n_fences);
  for (int g = threadIdx.x; g < a.n_groups; g += blockDim.x) groups[g] = a.groups[g];
  for (int q = threadIdx.x; q < a.n_pairs; q += blockDim.x) pairs[q] = a.pairs[q];
  for (int i = threadIdx.x; i < a.n_fences; i += blockDim.x) fence[i] = a.fences[i];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  uint32_t* stage = stage_all + static_cast<size_t>(threadIdx.x >> 5) * a.max_slots * 32 + lane;
  const uint64_t tiles = (a.dim + 31) / 32;
  const uint64_t warps = static_cast<uint64_t>(gridDim.x) * (blockDim.x >> 5);
  const uint32_t col_mask = (1u << a.col_bits) - 1u;
  const bool symmetric = a.p.symmetric != 0;
  uint32_t counted = 0;
  for (uint64_t t = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5; t < tiles; t += warps) {
    const uint64_t r = t * 32 + lane;
    const bool valid = r < a.dim;
    const uint64_t s = valid ? (a.direct ? r : a.states[r]) : 0;
    const uint32_t base = a.tile_ptr[t], width = a.tile_ptr[t + 1] - base;
    double dr = 0.0, di = 0.0;
    if (valid) {
      for (int q = 0; q < a.n_pairs; ++q) {
        const RowPair& pr = pairs[q];
        const int v = static_cast<int>((s >> pr.i) & 1) | (static_cast<int>((s >> pr.j) & 1) << 1);
        dr += pr.re[v];
        di += pr.im[v];
      }
      for (int q = 0; q < a.n_terms; ++q) {
        const FlipTerm& ft = a.terms[q];
        if ((s & ft.req_mask) != ft.req_val) continue;
        const bool neg = __popcll(~s & ft.sign_mask) & 1;
        dr += neg ? -ft.kr : ft.kr;
        di += neg ? -ft.ki : ft.ki;
      }
    }
    uint32_t kept = 0;
    const int last_word = (a.n_groups - 1) / 64 * 64;
    for (int g0 = last_word; g0 >= 0; g0 -= 64) {
      uint64_t active = valid ? active_groups(groups, a.n_groups, g0, s) : 0;
      while (__any_sync(0xffffffffu, active != 0)) {
        S key[U];
        uint32_t code[U], fb[U];
        bool act[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
          act[u] = active != 0;
          key[u] = 0;
          code[u] = 0;
          fb[u] = 0;
          if (!act[u]) continue;
          const int g = 63 - __clzll(static_cast<long long>(active));
          active ^= 1ull << g;
          const RowGroup& grp = groups[g0 + g];
          const S target = static_cast<S>(s ^ grp.flip);
          uint32_t phase = 0;
          if (symmetric) {
            int shift;
            bool neg;
            orbit_minimum<S, SHIFT>(target, a.p, static_cast<S>(a.mask), key[u], shift, neg);
            if (a.cplx) phase = static_cast<uint32_t>(2 * shift + (neg ? 1 : 0));
            else phase = neg != (SHIFT && (shift & 1)) ? 1u : 0u;
          } else {
            key[u] = target;
          }
          code[u] = grp.amp[group_digits(grp, s)] * static_cast<uint32_t>(a.phases) + phase;
        }
        int64_t col[U];
        if (symmetric) {
          for (int len = a.n_fences; len > 1;) {
            const int half = len >> 1;
#pragma unroll
            for (int u = 0; u < U; ++u) fb[u] = (fence[fb[u] + half] <= key[u]) ? fb[u] + half : fb[u];
            len -= half;
          }
          uint64_t at[U], len[U];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            at[u] = static_cast<uint64_t>(fb[u]) * a.fence_seg;
            len[u] = min(a.fence_seg, a.dim - at[u]);
          }
          for (int it = 0; it < a.fence_levels; ++it) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
              if (len[u] <= 1) continue;
              const uint64_t half = len[u] >> 1;
              at[u] = (__ldg(a.states + at[u] + half) <= key[u]) ? at[u] + half : at[u];
              len[u] -= half;
            }
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
            col[u] = act[u] && __ldg(a.states + at[u]) == key[u] ? static_cast<int64_t>(at[u]) : -1;
        } else {
#pragma unroll
          for (int u = 0; u < U; ++u)
            col[u] = !act[u] ? -1
                     : a.direct ? (key[u] < a.dim ? static_cast<int64_t>(key[u]) : -1)
                                : colex_rank_checked(static_cast<uint64_t>(key[u]), a.p.sites, a.p.up, a.binom);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
          if (col[u] < 0) continue;
          if (static_cast<uint64_t>(col[u]) == r) {
            const double2 v = a.values[code[u] * a.classes];
            dr += v.x;
            di += v.y;
            continue;
          }
          const uint32_t cls = symmetric ? a.class_of[a.orbits[col[u]]] : 0u;
          const uint32_t e = static_cast<uint32_t>(col[u]) | ((code[u] * a.classes + cls) << a.col_bits);
          a.entries[(static_cast<uint64_t>(base) + kept) * 32 + lane] = e;
          stage[kept * 32] = e;
          ++kept;
        }
      }
    }
    for (uint32_t j = kept; j < width; ++j) a.entries[(static_cast<uint64_t>(base) + j) * 32 + lane] = kNoEntry;
    if (valid) {
      // |d| <= eps is not stored (src/operator/mod.rs:2162-2164)
      if (!(hypot(dr, di) > kEps)) dr = di = 0.0;
      if (a.cplx) {
        a.diag64[2 * r] = dr;
        a.diag64[2 * r + 1] = di;
        a.diag32[2 * r] = static_cast<float>(dr);
        a.diag32[2 * r + 1] = static_cast<float>(di);
      } else {
        a.diag64[r] = dr;
        a.diag32[r] = static_cast<float>(dr);
      }
    }
    // the row's nonzeros after coalescing, and the values they have
    for (uint32_t i = 0; i < kept; ++i) {
      const uint32_t e = stage[i * 32], c = e & col_mask;
      bool first = true;
      for (uint32_t j = 0; j < i && first; ++j) first = (stage[j * 32] & col_mask) != c;
      if (!first) continue;
      double2 sum = a.values[e >> a.col_bits];
      bool single = true;
      for (uint32_t j = i + 1; j < kept; ++j) {
        const uint32_t f = stage[j * 32];
        if ((f & col_mask) != c) continue;
        const double2 v = a.values[f >> a.col_bits];
        sum.x += v.x;
        sum.y += v.y;
        single = false;
      }
      if (single) {
        ++counted;
        const uint32_t v = (e >> a.col_bits) / static_cast<uint32_t>(a.classes);
        if (a.used[v] == 0) a.used[v] = 1;
        continue;
      }
      const double ratio = symmetric ? a.inv_sqrt[257 + a.orbits[r]] * a.inv_sqrt[a.orbits[c]] : 1.0;
      if (!(hypot(sum.x, sum.y) * ratio > kEps)) {
        // entries that cancel are none: the row does not read the column (which may hold an infinity)
        for (uint32_t j = i; j < kept; ++j)
          if ((stage[j * 32] & col_mask) == c) a.entries[(static_cast<uint64_t>(base) + j) * 32 + lane] = kNoEntry;
        continue;
      }
      ++counted;
      if (a.cplx) continue;
      const unsigned long long bits =
          sum.x == 0.0 ? 0ull : static_cast<unsigned long long>(__double_as_longlong(sum.x));
      uint32_t h = static_cast<uint32_t>((bits * 0x9E3779B97F4A7C15ull) >> 40) & (kSumSlots - 1);
      int probe = 0;
      for (; probe < kSumSlots; ++probe) {
        const unsigned long long have = *reinterpret_cast<volatile unsigned long long*>(a.sums + h);
        if (have == bits) break;
        if (have == ~0ull) {
          const unsigned long long prev = atomicCAS(a.sums + h, ~0ull, bits);
          if (prev == ~0ull || prev == bits) break;
        }
        h = (h + 1) & (kSumSlots - 1);
      }
      if (probe == kSumSlots) atomicOr(a.flags, 1);
    }
  }
  counted = warp_sum_u32(counted);
  if (lane == 0 && counted > 0) atomicAdd(a.nnz, static_cast<unsigned long long>(counted));
}

std::vector<int> orbit_sizes(const SectorParams& p) {
  std::set<int> sizes;
  for (int d = 1; d <= (p.has_momentum ? p.sites : 1); ++d)
    if (p.sites % d == 0 || !p.has_momentum)
      for (int f1 = 1; f1 <= (p.parity != 0 ? 2 : 1); ++f1)
        for (int f2 = 1; f2 <= (p.inversion != 0 ? 2 : 1); ++f2) sizes.insert(d * f1 * f2);
  return std::vector<int>(sizes.begin(), sizes.end());
}

int device_sms(int device) {
  int sms = 148;
  QMBED_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  return sms;
}

// Entries are read once per application: past the L1, which then keeps the
// gathered vector.
__device__ __forceinline__ uint32_t load_entry(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.global.nc.L1::no_allocate.b32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

template <typename T>
struct Pair2;
template <>
struct Pair2<float> {
  using type = float2;
};
template <>
struct Pair2<double> {
  using type = double2;
};

// Complex element i of a product's input (an ordinary load, see
// await_previous): 8 or 16 bytes at once when the vector allows it (VEC2).
template <typename T, bool VEC2>
__device__ __forceinline__ typename Pair2<T>::type load_complex(const T* x, uint64_t i) {
  using P = typename Pair2<T>::type;
  if (VEC2) return reinterpret_cast<const P*>(x)[i];
  P v;
  v.x = x[2 * i];
  v.y = x[2 * i + 1];
  return v;
}

// y[r] = sqrt(R_r) sum_e value[code_e] x[col_e] + d[r] x[r], one lane per row.
// VC: complex vectors; VALC: complex values. With SPLIT > 1 a block of SPLIT
// warps shares one tile's slots (small sectors), else every warp has a tile of its own.
//
// Bound by the gathers' way through the L2: a slot of 32 rows touches 15 (FP64)
// or 11 (FP32) sectors of 32, and DRAM carries little more than the entries
// (x stays in the L2). Small blocks and few registers win, because the rows'
// latency chain (tile pointer, entries, gathers) is hidden by warps in flight:
// blocks of 128 threads against 1024 were 20.8 against 24.2 us at 28 sites
// (718,146 rows, FP64) and 119 against 145 us at 31 (4,850,640 rows). Against
// row lists with a scaled copy of x (measured in the same call): 34.7 -> 20.8
// us and 212 -> 119 us; complex rows of 26 sites at k = 3 (400,023 rows, 20
// bytes per entry before, 4 now) 85.5 -> 40 us.
constexpr int kSpmvThreads = 128;
template <typename T, bool VC, bool VALC, bool VEC2, int SPLIT, int KB>
__global__ void __launch_bounds__(kSpmvThreads) tile_spmv_kernel(uint64_t n, const uint32_t* __restrict__ tile_ptr,
                                                         const uint32_t* __restrict__ entries, int col_bits,
                                                         const double2* __restrict__ values, int codes,
                                                         const T* __restrict__ diag,
                                                         const uint16_t* __restrict__ orbits,
                                                         const double* __restrict__ sqrt_table,
                                                         const T* x, T* y) {
  using P = typename Pair2<T>::type;
  using V = typename std::conditional<VALC, P, T>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  V* table = reinterpret_cast<V*>(smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint64_t tiles = (n + 31) / 32;
  const uint64_t t = SPLIT > 1 ? blockIdx.x : static_cast<uint64_t>(blockIdx.x) * (blockDim.x >> 5) + warp;
  const uint32_t col_mask = (1u << col_bits) - 1u;
  const uint64_t r = t * 32 + lane;
  const bool valid = t < tiles && r < n;
  int from = 0, to = 0;
  const uint32_t* row = entries + lane;
  uint32_t e[KB];
  if (t < tiles) {
    const uint32_t base = __ldg(tile_ptr + t);
    const int width = static_cast<int>(__ldg(tile_ptr + t + 1) - base);
    from = SPLIT > 1 ? width * warp / SPLIT : 0;
    to = SPLIT > 1 ? width * (warp + 1) / SPLIT : width;
    row += static_cast<uint64_t>(base) * 32;
  }
  // the first entries and the row's own operands are requested before the
  // code table is staged, the next entries before the current ones are used
#pragma unroll
  for (int u = 0; u < KB; ++u) e[u] = from + u < to ? load_entry(row + (from + u) * 32) : kNoEntry;
  T xr = 0, xi = 0, dr = 0, di = 0;
  uint32_t orbit = 0;
  const bool own = valid && (SPLIT == 1 || warp == 0);
  if (own) {
    if (VALC) {
      dr = __ldcs(diag + 2 * r);
      di = __ldcs(diag + 2 * r + 1);
    } else {
      dr = __ldcs(diag + r);
    }
    if (orbits) orbit = __ldcs(orbits + r);
  }
  for (int i = threadIdx.x; i < codes; i += blockDim.x) {
    const double2 v = values[i];
    if constexpr (VALC) {
      table[i].x = static_cast<T>(v.x);
      table[i].y = static_cast<T>(v.y);
    } else {
      table[i] = static_cast<T>(v.x);
    }
  }
  await_previous();
  if (own) {
    if (VC) {
      const P v = load_complex<T, VEC2>(x, r);
      xr = v.x;
      xi = v.y;
    } else {
      xr = x[r];
    }
  }
  __syncthreads();
  T ar = 0, ai = 0;
  for (int j0 = from; j0 < to; j0 += KB) {
    T gr[KB], gi[KB];
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      gr[u] = gi[u] = 0;
      if (e[u] == kNoEntry) continue;
      if (VC) {
        const P v = load_complex<T, VEC2>(x, e[u] & col_mask);
        gr[u] = v.x;
        gi[u] = v.y;
      } else {
        gr[u] = x[e[u] & col_mask];
      }
    }
    uint32_t f[KB];
#pragma unroll
    for (int u = 0; u < KB; ++u) f[u] = j0 + KB + u < to ? load_entry(row + (j0 + KB + u) * 32) : kNoEntry;
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      if (e[u] != kNoEntry) {
        const V c = table[e[u] >> col_bits];
        if constexpr (VALC) {
          ar += c.x * gr[u] - c.y * gi[u];
          ai += c.x * gi[u] + c.y * gr[u];
        } else {
          ar += c * gr[u];
          if (VC) ai += c * gi[u];
        }
      }
      e[u] = f[u];
    }
  }
  if (SPLIT > 1) {
    __shared__ T part[2][SPLIT][32];
    part[0][warp][lane] = ar;
    if (VC) part[1][warp][lane] = ai;
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int q = 1; q < SPLIT; ++q) {
      ar += part[0][q][lane];
      if (VC) ai += part[1][q][lane];
    }
  }
  if (!valid) return;
  const T scale = orbits ? static_cast<T>(__ldg(sqrt_table + 257 + orbit)) : static_cast<T>(1);
  if (VC) {
    P out;
    if (VALC) {
      out.x = scale * ar + dr * xr - di * xi;
      out.y = scale * ai + dr * xi + di * xr;
    } else {
      out.x = scale * ar + dr * xr;
      out.y = scale * ai + dr * xi;
    }
    if (VEC2) {
      __stcs(reinterpret_cast<P*>(y) + r, out);
    } else {
      __stcs(y + 2 * r, out.x);
      __stcs(y + 2 * r + 1, out.y);
    }
  } else {
    __stcs(y + r, scale * ar + dr * xr);
  }
}

// Block action on tiles: a row's NB values are LPR consecutive 16-byte
// vectors, one per lane, and a warp takes 32 / LPR rows of a tile (LPR
// neighbouring warps share one). Entries are read once per row and shared by
// its lanes. Bound by the L1's data path (75% at 28 sites, 16 columns FP32: each
// gathered column is 32 to 128 bytes of a line of its own) and by the L2: at 32
// sites (9,398,520 rows, FP32, 8 columns) the 589 us move 6.6 GB through it
// (11 TB/s); the row lists took 766 us. At 34 sites it is DRAM: 16.1 GB in 2.65 ms,
// where the row lists moved 24.5 GB in 4.24. At 28 sites (718,146 rows, 16 columns) 70
// against 75 us in FP32 and 136 against 139 us in FP64. Many small blocks in one
// moving window of rows are what is fast: blocks of 256 to 1024 threads with
// chunks of rows of their own, for reuse in the L1, took 1.2 to 1.9 times as long.
template <typename T, int NB, bool HAS_P, int KB>
__global__ void __launch_bounds__(256) tile_spmm_kernel(uint64_t n, const uint32_t* __restrict__ tile_ptr,
                                                         const uint32_t* __restrict__ entries, int col_bits,
                                                         const double2* __restrict__ values, int codes,
                                                         const T* __restrict__ diag, const T* z,
                                                         const T* p, T* out, T alpha, T beta, T gamma) {
  constexpr int VEC = 16 / sizeof(T);
  constexpr int LPR = NB / VEC;
  constexpr int RPW = 32 / LPR;
  extern __shared__ __align__(16) unsigned char smem[];
  T* table = reinterpret_cast<T*>(smem);
  const int lane = threadIdx.x & 31;
  const uint64_t w = (static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const uint64_t t = w / LPR;
  const int in_tile = static_cast<int>(w % LPR) * RPW + lane / LPR, part = lane % LPR;
  const uint64_t r = t * 32 + in_tile;
  const uint32_t col_mask = (1u << col_bits) - 1u;
  int width = 0;
  const uint32_t* row = entries + in_tile;
  uint32_t e[KB];
  if (r < n) {
    const uint32_t base = __ldg(tile_ptr + t);
    width = static_cast<int>(__ldg(tile_ptr + t + 1) - base);
    row += static_cast<uint64_t>(base) * 32;
  }
#pragma unroll
  for (int u = 0; u < KB; ++u) e[u] = u < width ? __ldg(row + u * 32) : kNoEntry;
  for (int i = threadIdx.x; i < codes; i += blockDim.x) table[i] = static_cast<T>(values[i].x);
  await_previous();
  __syncthreads();
  if (r >= n) return;
  T acc[VEC];
#pragma unroll
  for (int v = 0; v < VEC; ++v) acc[v] = 0;
  for (int j0 = 0; j0 < width; j0 += KB) {
    T g[KB][VEC];
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      if (e[u] != kNoEntry) {
        load16_rw(z + static_cast<uint64_t>(e[u] & col_mask) * NB + part * VEC, g[u]);
      } else {
#pragma unroll
        for (int v = 0; v < VEC; ++v) g[u][v] = 0;
      }
    }
#pragma unroll
    for (int u = 0; u < KB; ++u) {
      const T c = e[u] != kNoEntry ? table[e[u] >> col_bits] : static_cast<T>(0);
#pragma unroll
      for (int v = 0; v < VEC; ++v) acc[v] += c * g[u][v];
    }
#pragma unroll
    for (int u = 0; u < KB; ++u) e[u] = j0 + KB + u < width ? __ldg(row + (j0 + KB + u) * 32) : kNoEntry;
  }
  const T d = __ldcs(diag + r);
  T self[VEC], o[VEC];
  load16_rw(z + r * NB + part * VEC, self);
#pragma unroll
  for (int v = 0; v < VEC; ++v) o[v] = alpha * (acc[v] + d * self[v]) + beta * self[v];
  if (HAS_P) {
    T q[VEC];
    load16_rw(p + r * NB + part * VEC, q);
#pragma unroll
    for (int v = 0; v < VEC; ++v) o[v] += gamma * q[v];
  }
  store16(out + r * NB + part * VEC, o);
}

}  // namespace

bool assemble_tile_rows(const SpinBasis& basis, const FlipProgram& prog, bool real, TileRows& out) {
  const SectorParams& p = basis.params();
  const uint64_t n = basis.dim();
  if (!prog.ok || basis.words() != 1 || n == 0 || !prog.terms.empty()) return false;
  const bool symmetric = basis.symmetric();
  if (symmetric && basis.fence_count() == 0) return false;
  // amplitudes of the off-diagonal pairs
  std::map<std::pair<uint64_t, uint64_t>, int> ids;
  std::vector<C64> amps;
  std::vector<RowGroup> groups;
  auto bits = [](double v) {
    uint64_t b;
    v = v == 0.0 ? 0.0 : v;
    std::memcpy(&b, &v, 8);
    return b;
  };
  for (const FlipGroup& g : prog.groups) {
    if (g.kind != kGroupPair) return false;
    RowGroup rg{};
    rg.flip = g.flip;
    rg.i = g.site_i;
    rg.j = g.site_j;
    rg.nz = g.nz;
    for (int v = 0; v < 4; ++v) {
      if (!((g.nz >> v) & 1)) continue;
      const C64 a(prog.amp_re[4 * g.first + v], prog.amp_im[4 * g.first + v]);
      // entries at rounding level are dropped by the coalescing rules: the row lists handle them
      if (std::abs(a) < 1e-12) return false;
      if (real && a.imag() != 0.0) return false;
      auto [it, fresh] = ids.insert({{bits(a.real()), bits(a.imag())}, static_cast<int>(amps.size())});
      if (fresh) amps.push_back(a);
      rg.amp[v] = static_cast<uint16_t>(it->second);
    }
    groups.push_back(rg);
    if (amps.size() > static_cast<size_t>(kMaxTableCodes)) return false;
  }
  std::vector<int> sizes{1};
  if (symmetric) sizes = orbit_sizes(p);
  if (sizes.back() > 256) return false;
  const bool cplx = !real;
  const int phases = !symmetric ? 1 : (cplx ? 2 * (p.has_momentum ? p.sites : 1) : 2);
  const int classes = static_cast<int>(sizes.size());
  const uint64_t codes = std::max<uint64_t>(1, amps.size()) * phases * classes;
  int col_bits = 1;
  while (col_bits < 32 && (1ull << col_bits) < std::max<uint64_t>(n, 2)) ++col_bits;
  // one code stays free, so that no entry equals kNoEntry
  if (col_bits >= 32 || codes > static_cast<uint64_t>(kMaxTableCodes) || codes >= (1ull << (32 - col_bits))) return false;

  // values per code: amplitude x character, then the same over sqrt(R)
  const bool pi = p.has_momentum && p.momentum != 0 && 2 * p.momentum == p.sites;
  std::vector<double> values(4 * codes, 0.0);
  for (size_t a = 0; a < amps.size(); ++a)
    for (int ph = 0; ph < phases; ++ph) {
      C64 chi(1.0, 0.0);
      if (symmetric && cplx) {
        const int shift = ph / 2;
        if (p.has_momentum && p.momentum != 0) {
          const long long s = (p.sites - shift) % p.sites;
          const double angle = -(2.0 * M_PI) * static_cast<double>(static_cast<long long>(p.momentum) * s) /
                               static_cast<double>(p.sites);
          chi = pi ? C64((shift & 1) ? -1.0 : 1.0, 0.0) : C64(std::cos(angle), std::sin(angle));
        }
        if (ph & 1) chi = -chi;
      } else if (ph & 1) {
        chi = C64(-1.0, 0.0);
      }
      const C64 v(amps[a].real() * chi.real() - amps[a].imag() * chi.imag(),
                  amps[a].real() * chi.imag() + amps[a].imag() * chi.real());
      for (int c = 0; c < classes; ++c) {
        const size_t code = (a * phases + ph) * classes + c;
        const double inv = 1.0 / std::sqrt(static_cast<double>(sizes[c]));
        values[2 * code] = v.real();
        values[2 * code + 1] = v.imag();
        values[2 * (codes + code)] = symmetric ? v.real() * inv : v.real();
        values[2 * (codes + code) + 1] = symmetric ? v.imag() * inv : v.imag();
      }
    }
  std::vector<RowPair> pairs;
  for (size_t q = 0; q < prog.diag_pairs.size(); ++q) {
    RowPair rp{};
    rp.i = static_cast<int>(prog.diag_pairs[q] & 0xff);
    rp.j = static_cast<int>(prog.diag_pairs[q] >> 8);
    for (int v = 0; v < 4; ++v) {
      rp.re[v] = prog.amp_re[4 * q + v];
      rp.im[v] = prog.amp_im[4 * q + v];
    }
    pairs.push_back(rp);
  }
  std::vector<uint8_t> class_of(264, 0);
  for (int c = 0; c < classes; ++c) class_of[static_cast<size_t>(sizes[c])] = static_cast<uint8_t>(c);
  std::vector<double> inv_sqrt(2 * 257, 0.0);
  for (int q = 1; q <= 256; ++q) {
    inv_sqrt[q] = 1.0 / std::sqrt(static_cast<double>(q));
    inv_sqrt[257 + q] = std::sqrt(static_cast<double>(q));
  }
  const int n_used = static_cast<int>(codes) / classes;

  // one upload: [values][pairs][terms][inv_sqrt][groups][class_of], and one
  // scratch area: [nnz][max width, flags][sums][used]
  std::vector<unsigned char> image;
  auto put = [&](const void* src, size_t bytes) {
    const size_t at = (image.size() + 15) & ~static_cast<size_t>(15);
    image.resize(at + bytes);
    if (bytes) std::memcpy(image.data() + at, src, bytes);
    return at;
  };
  const size_t at_values = put(values.data(), values.size() * 8);
  const size_t at_pairs = put(pairs.data(), pairs.size() * sizeof(RowPair));
  const size_t at_terms = put(prog.diag_terms.data(), prog.diag_terms.size() * sizeof(FlipTerm));
  const size_t at_inv = put(inv_sqrt.data(), inv_sqrt.size() * 8);
  const size_t at_groups = put(groups.data(), groups.size() * sizeof(RowGroup));
  const size_t at_class = put(class_of.data(), class_of.size());
  const size_t scratch = (image.size() + 15) & ~static_cast<size_t>(15);
  const size_t scratch_bytes = 16 + kSumSlots * 8 + static_cast<size_t>(n_used) * 4;
  const uint64_t tiles = (n + 31) / 32;
  const size_t at_widths = (scratch + scratch_bytes + 15) & ~static_cast<size_t>(15);
  DeviceBuffer work(at_widths + tiles * 4);
  unsigned char* base = work.as<unsigned char>();
  QMBED_CUDA(cudaMemcpy(base, image.data(), image.size(), cudaMemcpyHostToDevice));
  QMBED_CUDA(cudaMemsetAsync(base + scratch, 0, 16, nullptr));
  QMBED_CUDA(cudaMemsetAsync(base + scratch + 16, 0xff, kSumSlots * 8, nullptr));
  QMBED_CUDA(cudaMemsetAsync(base + scratch + 16 + kSumSlots * 8, 0, static_cast<size_t>(n_used) * 4, nullptr));

  FillArgs a{};
  a.p = p;
  a.mask = low_mask<uint64_t>(p.sites);
  a.dim = n;
  a.direct = basis.direct() ? 1 : 0;
  a.states = static_cast<const uint64_t*>(basis.states());
  a.orbits = basis.orbits();
  a.binom = basis.binomials();
  a.class_of = base + at_class;
  a.fences = basis.fence_keys();
  a.n_fences = symmetric ? basis.fence_count() : 0;
  a.fence_seg = basis.fence_segment();
  a.fence_levels = basis.fence_levels();
  a.groups = reinterpret_cast<const RowGroup*>(base + at_groups);
  a.n_groups = static_cast<int>(groups.size());
  a.pairs = reinterpret_cast<const RowPair*>(base + at_pairs);
  a.n_pairs = static_cast<int>(pairs.size());
  a.terms = reinterpret_cast<const FlipTerm*>(base + at_terms);
  a.n_terms = static_cast<int>(prog.diag_terms.size());
  a.cplx = cplx ? 1 : 0;
  a.phases = phases;
  a.classes = classes;
  a.col_bits = col_bits;
  a.codes = static_cast<int>(codes);
  a.values = reinterpret_cast<const double2*>(base + at_values);
  a.inv_sqrt = reinterpret_cast<const double*>(base + at_inv);
  a.nnz = reinterpret_cast<unsigned long long*>(base + scratch);
  int* max_width = reinterpret_cast<int*>(base + scratch + 8);
  a.flags = max_width + 1;
  a.sums = reinterpret_cast<unsigned long long*>(base + scratch + 16);
  a.used = reinterpret_cast<unsigned int*>(base + scratch + 16 + kSumSlots * 8);
  const size_t program_smem = groups.size() * sizeof(RowGroup) + pairs.size() * sizeof(RowPair) +
                              static_cast<size_t>(a.n_fences) * 8;
  if (program_smem > static_cast<size_t>(kMaxProgramSmem)) return false;
  const int sms = device_sms(basis.device());
  const size_t group_smem = groups.size() * sizeof(RowGroup);
  const unsigned wgrid = static_cast<unsigned>(std::min<uint64_t>((tiles + 7) / 8, static_cast<uint64_t>(sms) * 8));
  if (group_smem > 48 * 1024) return false;
  tile_width_kernel<<<wgrid, kFillThreads, group_smem>>>(a, reinterpret_cast<uint32_t*>(base + at_widths), max_width);
  QMBED_LAUNCH_CHECK();
  bool wide = false;
  const uint64_t slots = exclusive_scan_counts(reinterpret_cast<uint32_t*>(base + at_widths), tiles, out.tile_ptr, &wide);
  int widest = 0;
  QMBED_CUDA(cudaMemcpy(&widest, max_width, sizeof(int), cudaMemcpyDeviceToHost));
  if (wide || widest > kMaxRowSlots) return false;

  const size_t smem = program_smem + static_cast<size_t>(kFillThreads / 32) * std::max(widest, 1) * 128;
  out.entries.allocate(std::max<uint64_t>(slots, 1) * 128);
  out.diag64.allocate(n * (cplx ? 16 : 8));
  out.diag32.allocate(n * (cplx ? 8 : 4));
  out.values.allocate(values.size() * 8);
  QMBED_CUDA(cudaMemcpyAsync(out.values.get(), base + at_values, values.size() * 8, cudaMemcpyDeviceToDevice, nullptr));
  a.max_slots = std::max(widest, 1);
  a.tile_ptr = out.tile_ptr.as<uint32_t>();
  a.entries = out.entries.as<uint32_t>();
  a.diag64 = out.diag64.as<double>();
  a.diag32 = out.diag32.as<float>();
  // characters depend on the shift except in k = 0 and parity-only sectors
  const bool shift = p.has_momentum && p.momentum != 0;
  auto kernel = p.sites <= 32 ? (shift ? tile_fill_kernel<uint32_t, true> : tile_fill_kernel<uint32_t, false>)
                              : (shift ? tile_fill_kernel<uint64_t, true> : tile_fill_kernel<uint64_t, false>);
  // one limit for every size: operators may be assembled on several threads
  QMBED_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  kMaxProgramSmem + kFillThreads / 32 * kMaxRowSlots * 128));
  int per_sm = 1;
  QMBED_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kFillThreads, smem));
  const unsigned grid = static_cast<unsigned>(
      std::min<uint64_t>((tiles + 7) / 8, static_cast<uint64_t>(sms) * std::max(per_sm, 1) * 4));
  kernel<<<grid, kFillThreads, smem>>>(a);
  QMBED_LAUNCH_CHECK();
  std::vector<unsigned char> host(scratch_bytes);
  QMBED_CUDA(cudaMemcpy(host.data(), base + scratch, scratch_bytes, cudaMemcpyDeviceToHost));
  uint64_t nnz = 0;
  std::memcpy(&nnz, host.data(), 8);
  int flags = 0;
  std::memcpy(&flags, host.data() + 12, 4);
  if (flags) return false;
  int distinct = 0;
  if (real) {
    std::set<uint64_t> seen;
    for (int v = 0; v < n_used; ++v) {
      uint32_t used = 0;
      std::memcpy(&used, host.data() + 16 + kSumSlots * 8 + 4 * v, 4);
      if (used) seen.insert(bits(values[2 * static_cast<size_t>(v) * classes]));
    }
    for (int q = 0; q < kSumSlots; ++q) {
      uint64_t b = 0;
      std::memcpy(&b, host.data() + 16 + 8 * q, 8);
      if (b != ~0ull) seen.insert(b);
    }
    distinct = static_cast<int>(seen.size());
    // the packed format's limits on distinct values (more of them: explicit values)
    if (distinct > kMaxStoredValues || static_cast<uint64_t>(distinct) > (1ull << (32 - col_bits))) return false;
  }
  out.n = n;
  out.sms = sms;
  out.complex_values = cplx;
  out.col_bits = col_bits;
  out.codes = static_cast<int>(codes);
  out.nnz = nnz;
  out.distinct_values = distinct;
  return true;
}

namespace {

// Sectors of up to this many tiles per SM take four warps per tile: with one warp each,
// fewer than eight warps would sit on an SM and a row's gathers run in series
// (complex rows of 22 sites, 1003 tiles: 6.8 against 8.4 us a call; at 1776
// tiles, 24 sites, 7.2 against 6.8).
constexpr uint64_t kSplitTilesPerSm = 8;
// Real FP64 rows keep eight gathers in flight per lane from here on: at 28
// sites (718,146 rows) four take 20.8 us and eight 21.8, at 30 (2,587,018) 75.0
// and 70.3, at 31 131.5 and 119.2. In FP32 and with complex vectors four are
// faster at every size (32 sites FP32 187 against 212 us).
constexpr uint64_t kDeepRows = 1ull << 21;

template <typename T, bool VC, bool VALC, bool VEC2>
void launch_spmv(const TileRows& rows, const SpinBasis& basis, const double* sqrt_table, const T* diag, const void* x,
                 void* y, cudaStream_t stream) {
  const uint64_t tiles = (rows.n + 31) / 32;
  const size_t smem = static_cast<size_t>(rows.codes) * sizeof(T) * (VALC ? 2 : 1);
  const double2* values = rows.values.as<double2>() + rows.codes;
  const uint16_t* orbits = basis.symmetric() ? basis.orbits() : nullptr;
  auto launch = [&](auto kernel, uint64_t blocks) {
    launch_dependent(kernel, static_cast<unsigned>(blocks), kSpmvThreads, smem, stream, rows.n,
                     rows.tile_ptr.as<uint32_t>(), rows.entries.as<uint32_t>(), rows.col_bits, values, rows.codes, diag,
                     orbits, sqrt_table, static_cast<const T*>(x), static_cast<T*>(y));
  };
  constexpr int kWarps = kSpmvThreads / 32;
  const uint64_t blocks = (tiles + kWarps - 1) / kWarps;
  constexpr int kDeep = !VC && sizeof(T) == 8 ? 8 : 4;
  if (tiles <= kSplitTilesPerSm * rows.sms) launch(tile_spmv_kernel<T, VC, VALC, VEC2, kWarps, 4>, tiles);
  else if (rows.n >= kDeepRows) launch(tile_spmv_kernel<T, VC, VALC, VEC2, 1, kDeep>, blocks);
  else launch(tile_spmv_kernel<T, VC, VALC, VEC2, 1, 4>, blocks);
  QMBED_LAUNCH_CHECK();
}

template <typename T>
void spmv_precision(const TileRows& rows, const SpinBasis& basis, const double* sqrt_table, const T* diag, bool vc,
                    const void* x, void* y, cudaStream_t stream) {
  const uintptr_t both = reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y);
  const bool vec2 = both % (2 * sizeof(T)) == 0;
  if (!vc) launch_spmv<T, false, false, true>(rows, basis, sqrt_table, diag, x, y, stream);
  else if (rows.complex_values)
    vec2 ? launch_spmv<T, true, true, true>(rows, basis, sqrt_table, diag, x, y, stream)
         : launch_spmv<T, true, true, false>(rows, basis, sqrt_table, diag, x, y, stream);
  else
    vec2 ? launch_spmv<T, true, false, true>(rows, basis, sqrt_table, diag, x, y, stream)
         : launch_spmv<T, true, false, false>(rows, basis, sqrt_table, diag, x, y, stream);
}

}  // namespace

void tile_spmv(const TileRows& rows, const SpinBasis& basis, const double* sqrt_table, int precision,
               bool complex_vectors, const void* x, void* y, cudaStream_t stream) {
  if (precision == 64)
    spmv_precision<double>(rows, basis, sqrt_table, rows.diag64.as<double>(), complex_vectors, x, y, stream);
  else
    spmv_precision<float>(rows, basis, sqrt_table, rows.diag32.as<float>(), complex_vectors, x, y, stream);
}

void tile_spmm(const TileRows& rows, int shape, int precision, int nb, const void* z, const void* p, void* out,
               double alpha, double beta, double gamma, cudaStream_t stream) {
  const uint64_t tiles = (rows.n + 31) / 32;
  static constexpr int kThreadsOf[kTileBlockShapes] = {64, 128, 64, 256};
  static constexpr int kBatchOf[kTileBlockShapes] = {4, 4, 2, 8};
  auto launch = [&](auto ttag, auto nbtag, auto ptag, auto kbtag) {
    using T = decltype(ttag);
    constexpr int NB = decltype(nbtag)::value;
    constexpr bool HP = decltype(ptag)::value;
    constexpr int LPR = NB * static_cast<int>(sizeof(T)) / 16;
    const int threads = kThreadsOf[shape];
    const uint64_t warps = tiles * LPR;
    const unsigned grid = static_cast<unsigned>((warps + threads / 32 - 1) / (threads / 32));
    const T* diag = precision == 64 ? reinterpret_cast<const T*>(rows.diag64.get())
                                    : reinterpret_cast<const T*>(rows.diag32.get());
    launch_dependent(tile_spmm_kernel<T, NB, HP, decltype(kbtag)::value>, grid, threads,
                     static_cast<size_t>(rows.codes) * sizeof(T), stream, rows.n, rows.tile_ptr.as<uint32_t>(),
                     rows.entries.as<uint32_t>(), rows.col_bits, rows.values.as<double2>(), rows.codes, diag,
                     static_cast<const T*>(z), static_cast<const T*>(p), static_cast<T*>(out),
                     static_cast<T>(alpha), static_cast<T>(beta), static_cast<T>(gamma));
  };
  auto by_kb = [&](auto ttag, auto nbtag, auto ptag) {
    if (kBatchOf[shape] == 8) launch(ttag, nbtag, ptag, std::integral_constant<int, 8>{});
    else if (kBatchOf[shape] == 2) launch(ttag, nbtag, ptag, std::integral_constant<int, 2>{});
    else launch(ttag, nbtag, ptag, std::integral_constant<int, 4>{});
  };
  auto by_p = [&](auto ttag, auto nbtag) {
    if (p) by_kb(ttag, nbtag, std::true_type{});
    else by_kb(ttag, nbtag, std::false_type{});
  };
  auto by_nb = [&](auto ttag) {
    if (nb == 8) by_p(ttag, std::integral_constant<int, 8>{});
    else by_p(ttag, std::integral_constant<int, 16>{});
  };
  if (precision == 64) by_nb(double{});
  else by_nb(float{});
  QMBED_LAUNCH_CHECK();
}

}  // namespace qmbed
