// FP64 GEMM on the tensor cores (tcgen05) from fixed-point slices, see gemm_fx.cu.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "gemm_simt.cuh"

namespace cphf {

// Plan of one fixed-point GEMM: operand orientation, K split and workspace layout.
struct FxPlan {
  GemmDesc d;              // possibly transposed (C^T = B^T A^T) so that the padded tiles are fewest
  int64_t ldk = 0;         // padded K of the planes
  int m_tiles = 0, n_tiles = 0;
  int splits = 1, kb_per_split = 0;
  int64_t m_chunk = 0;     // rows of A per pass (bounds the planes)
  double us = 0.0;         // expected time
  size_t key_bytes = 0;    // flag + row keys, cleared before each pass
  size_t off_ea = 0, off_eb = 0, off_a = 0, off_b = 0, off_ws = 0, total = 0;
};

// true when the kernels can run on the device (sm_103 / sm_100 family)
bool fx_available(int device);
// Fills the plan and returns true when the fixed-point GEMM is expected to be faster than the
// native kernel on this shape.
bool fx_plan(const GemmDesc& d, int num_sms, FxPlan& p);
// C = alpha A B + beta C.  `ws`: plan.total bytes; `err`: raised when a bounded wait expired.
// Non-finite operands are left to the native kernel, which runs only when one was met; with
// `nonfinite` (single-pass plans) they are left to the caller: it receives the device flag that is
// set when one was met, C is then untouched.
cudaError_t fx_gemm(const FxPlan& p, cudaStream_t stream, void* ws, int* err, int num_sms,
                    const int** nonfinite = nullptr);

}  // namespace cphf
