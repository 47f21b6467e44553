// The sumcheck steps of the fold-round driver (zc_rounds.cu), launched by the
// sumcheck unit.
#pragma once
#include "common.cuh"

namespace zc {

// CTAs of a round's sumcheck pass, and so partial sums its hop adds up.
constexpr int kRoundPartials = 4 * 152;

// s0 partials of the first round: sum_j eq[j] mle[2j] over M pairs.
zc_status sc_first_partials(zc_field field, const uint32_t* mle, int64_t M, const uint32_t* eq,
                            uint32_t* partial, int* np, cudaStream_t st);
// A round's fold (M >= 2 pairs) and the next round's partials.
zc_status sc_fold_partials(zc_field field, const uint32_t* mle, int64_t M, const uint32_t* beta,
                           int beta_limbs, const uint32_t* msg, uint32_t* mle_out,
                           const uint32_t* eq, uint32_t* eq_out, uint32_t* claim,
                           uint32_t* partial, int* np, cudaStream_t st);

}  // namespace zc
