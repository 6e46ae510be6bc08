// Structured action of full-space spin-1/2 chains whose terms are products of
// z (diagonal) or a single x (one bit flip): transverse-field Ising chains and
// their relatives. No matrix is stored: the diagonal is evaluated from the bits
// of the state index and the flips are served from boxes of the vector in shared
// memory, in one pass or in one pass per group of bits.
#pragma once

#include <complex>
#include <memory>
#include <mutex>
#include <vector>

#include "common.cuh"

namespace qmbed {

struct FlipChainDesc {
  int sites = 0;
  std::vector<uint64_t> z_masks;   // diagonal products: sites of the z factors
  std::vector<double> z_coefs;     // coefficient x z1^|mask|, so D(s) = sum c (-1)^popcount(~s & mask)
  std::vector<double> x_coefs;     // per site: amplitude of the single flip of that bit
};

// out = alpha * (H x) + beta * x + gamma * p + kappa * q  on full-space
// vectors (real or interleaved complex, FP64 or FP32); p and q may be null;
// out may alias p (rows are read before they are written), never x or q.
// kappa is complex (applied to complex vectors; its real part for real ones).
struct FlipStep {
  double alpha = 1.0, beta = 0.0, gamma = 0.0;
  double kappa_re = 0.0, kappa_im = 0.0;
};

// Runs the box action's bounded wait on a barrier that no copy
// completes (1024 polls) on `device`; returns 1 when it gave up as designed.
int flip_stage_wait_selftest(int device);

// How an application runs: word bits of its boxes (0: one tile per block),
// flips above the box that read their partners directly, and the bits of the
// group passes, lowest first.
struct BoxPlan {
  int vb = 0;
  int extra = 0;
  std::vector<int> groups;
  bool far_first = false;  // FP32: the direct flips before the box's
};

class FlipChain {
 public:
  explicit FlipChain(const FlipChainDesc& d);
  uint64_t dim() const { return 1ull << sites_; }
  int sites() const { return sites_; }
  // y = H x (step = identity coefficients) or the fused three/four-term form.
  void apply(int precision, bool cplx, const void* x, void* out, const void* p, const void* q, const FlipStep& step,
             cudaStream_t stream) const;
  // Gershgorin-type bounds: |D| max over the diagonal terms plus sum |x|.
  double norm_bound() const;

 private:
  int sites_;
  int n_diag_;
  DeviceBuffer diag_masks_, diag_coefs_, x_coefs_;
  mutable DeviceBuffer tables_;  // low-bit diagonal tables (FP64, FP32)
  mutable int tables_ready_ = 0;  // bit 1: FP64 table, bit 2: FP32 table
  mutable int table_tb_[2] = {0, 0};
  // Box action and the diagonal's tables per box width.
  struct BoxTables {
    bool ready = false;
    DeviceBuffer buf;
    size_t at_coefs = 0, at_table = 0, at_words = 0, at_high = 0;
    int n_lane = 0, n_word = 0;
  };
  const BoxTables& box_tables(int vbits, int vb, cudaStream_t stream) const;
  void prepare_tables(cudaStream_t stream) const;
  void build_box_tables(int vbits, int vb, cudaStream_t stream, BoxTables& t) const;
  void apply_boxes(int precision, bool cplx, const void* x, void* out, const void* p, const void* q,
                   const FlipStep& step, cudaStream_t stream, const BoxPlan& plan) const;
  mutable std::mutex tables_mu_;
  mutable bool tables_prepared_ = false;
  mutable BoxTables box_tables_[3][2];  // [state bits inside a word][box width]
  std::vector<uint64_t> host_diag_masks_;
  std::vector<double> host_diag_coefs_, host_x_;
};

}  // namespace qmbed
