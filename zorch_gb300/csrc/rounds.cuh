// What the fold-round driver (zc_rounds.cu) launches from other units: the
// sumcheck steps, and commits that end in a round's hop.
#pragma once
#include "common.cuh"
#include "roundhop.cuh"

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

// zc_merkle_commit, zc_fri_fold_commit and zc_fri_fold_commit_bitrev with the
// committed layer's hop in the launch that computes its root.
zc_status merkle_commit_hop(const zc_poseidon2* p, const zc_leaves& lv, uint32_t* layers,
                            const RoundHop& hop, cudaStream_t st);
zc_status fold_commit_natural(const zc_poseidon2* p, const uint32_t* cw, int64_t n, int ef_in,
                              const uint32_t* beta, int ef_beta, uint32_t shift_mont,
                              uint32_t generator, uint32_t* out, uint32_t* layers, cudaStream_t st,
                              const RoundHop& hop);
zc_status fold_commit_bitrev(const zc_poseidon2* p, const uint32_t* cw, int64_t n, int ef_in,
                             const uint32_t* beta, int ef_beta, uint32_t shift_mont,
                             uint32_t generator, uint32_t* out, uint32_t* layers, cudaStream_t st,
                             const RoundHop& hop);

}  // namespace zc
