// rk_cand.cu -- the candidate kernel for Rockable's NEAR predicates, with fused
// multiply-adds (see rk_cand.cuh).
#include "rk_cand.cuh"

namespace rk {

void launch_candidates_float(const Scene& s, unsigned grid, size_t smem, const uint64_t* pairs, int64_t np, int mv, int me,
                             int mf, uint64_t* out, uint32_t* unc, int64_t cap, unsigned long long* counter,
                             cudaStream_t st) {
  k_candidates<false><<<grid, 32 * kCandWarps, smem, st>>>(s, pairs, np, mv, me, mf, out, unc, cap, counter);
}

}  // namespace rk
