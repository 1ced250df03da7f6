// Tensor-core (tcgen05) engine: what it accepts, and dispatch to the forward / backward kernels.
#include "sa_common.cuh"
#include "sa_tc_host.cuh"

namespace sa {
namespace tc {
int forward(const Problem& p, float* out, float* lse2, float* carry, float* total, cudaStream_t s);
int backward(const Problem& p, const float* stats, const float* carry, const void* d_out, const RowLayout& d_out_rows,
             float* dq_acc, float* dq0, float* dk0, void* dk, void* dv, cudaStream_t s);
int backward_wide(const Problem& p, const float* stats, const float* carry, const void* d_out, const RowLayout& d_out_rows,
                  float* dq_acc, float* dq0, float* dk0, void* dk, void* dv, cudaStream_t s);
}  // namespace tc

int tc_available() { return 1; }

int tc_supported(const Problem& p) {
  if (p.dtype != SA_BF16) return SA_ERR_UNSUPPORTED;
  if (p.head_dim != 64 && p.head_dim != 128) return SA_ERR_UNSUPPORTED;
  if (p.damp != SA_DAMP_NONE) return SA_ERR_UNSUPPORTED;
  return SA_OK;
}

int tc_forward(const Problem& p, float* out, float* lse2, float* carry, float* total, cudaStream_t s) {
  return tc::forward(p, out, lse2, carry, total, s);
}

int tc_backward_supported(const Problem& p) {
  return tc_supported(p);
}

int tc_backward(const Problem& p, const float* stats, const float* carry, const void* d_out, const RowLayout& d_out_rows,
                float* dq_acc, float* dq0, float* dk0, void* dk, void* dv, cudaStream_t s) {
  auto run = p.head_dim == 128 ? tc::backward_wide : tc::backward;
  return run(p, stats, carry, d_out, d_out_rows, dq_acc, dq0, dk0, dk, dv, s);
}
}  // namespace sa
