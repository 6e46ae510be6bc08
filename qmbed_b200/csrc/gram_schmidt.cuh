// Gram-Schmidt steps of the FP64 Krylov solvers without a host round trip per
// step: one cooperative launch orthogonalises a vector against a panel
// (overlaps, subtraction, the DGKS test and its second pass, the norm and the
// scaled result) and leaves a record on the device; the solver queues as many
// steps as it can and reads their records together.
#pragma once

#include <cuda_runtime.h>

#include <complex>
#include <cstdint>
#include <vector>

#include "common.cuh"

namespace qmbed {

struct OrthoRecord {
  double before = 0.0;  // norm before (of the three-term residual, or of src)
  double norm = 0.0;    // norm of the orthogonalised vector
  bool second = false;  // the DGKS test asked for a second pass (a fused step has made it)
  bool ok = false;      // norm finite and above 1e-14: the scaled result was written
  std::vector<std::complex<double>> h;  // overlaps of the first pass
};

class FusedOrtho {
 public:
  FusedOrtho(int device, int sms) : device_(device), sms_(sms) {}
  ~FusedOrtho();
  FusedOrtho(const FusedOrtho&) = delete;
  FusedOrtho& operator=(const FusedOrtho&) = delete;

  // Whether panels of n rows and up to m columns take the fused kernel.
  bool applies(uint64_t n, int m) const;
  // Buffers for runs of up to `steps` records on panels of up to m columns, so
  // that none of them allocates.
  void reserve(int steps, int m, cudaStream_t stream);
  // Starts a run of at most `steps` records for panels of up to `m` columns;
  // `beta` stands for the norm of the record before the first.
  void begin(int steps, int m, double beta, cudaStream_t stream);
  // Queues one step: w = src - A A^H src (A: m columns of n rows; a second pass
  // as the DGKS test has it), scaled by its norm into `slot` (into w when
  // null). `three_term`: the test compares with the norm of
  // src - Re(h_{m-1}) a_{m-1} - beta a_{m-2}, beta the previous record's norm.
  void step(const double* A, uint64_t n, int m, const double* src, double* w, double* slot, bool cplx, bool three_term,
           cudaStream_t stream);
  // Device record of a step that other kernels queue: before, norm, second,
  // ok at 0 .. 3, overlaps from kRecordHead on; previous_norm: the beta above.
  static constexpr int kRecordHead = 8;
  double* next_record(int m, const double** previous_norm);
  // Waits and reads the records queued since begin(). Raises when a step's
  // grid barrier timed out.
  void finish(std::vector<OrthoRecord>& records, cudaStream_t stream);

 private:
  int device_, sms_;
  int steps_ = 0, cap_ = 0, count_ = 0;
  std::vector<int> columns_;
  DeviceBuffer state_, partials_;
  double* host_ = nullptr;  // pinned
  size_t host_bytes_ = 0;
};

}  // namespace qmbed
