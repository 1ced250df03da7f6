// Tensor-core engine, forward: what its translation units share.
#pragma once

#include "sa_tc_host.cuh"
#include "sa_tc_ptx.cuh"

namespace sa {
namespace tc {

constexpr int kMaxLiveTiles = 1024;   // key tiles of a sequence when dead tiles are left out (sa_tc_skip.cu)

struct ForwardMaps {                  // boxes of 128 rows x 64 columns
  CUtensorMap q, k, v, q0, k0;
};
// Two heads a CTA (sa_tc_fwd_pair.cu): head_dim 64, an even number of heads sharing a selector.
int forward_pair(const Problem& p, const ForwardMaps& m, const float* carry, float* out, float* lse2, const WaitCtx& status,
                 const uint8_t* alive, cudaStream_t s);

// Two rows a CTA (sa_tc_fwd_self.cu): head_dim 64, one head per selector, an even number of rows.
int forward_self(const Problem& p, const ForwardMaps& m, const float* carry, float* out, float* lse2, const WaitCtx& status,
                 const uint8_t* alive, cudaStream_t s);

}  // namespace tc
}  // namespace sa
