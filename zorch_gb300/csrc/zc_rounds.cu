// The commit-and-fold rounds of an open in one call: what FriProver's commit
// phase, the Basefold open and the SP1 stacked open share (zorch/pcs/fold.py:
// 90-115, zorch/pcs/basefold/prover.py:419-480, zorch/pcs/jagged/open.py:
// 237-330). A round as six to eight calls from Python is 60-80 us of host time
// where the GPU needs 60 for a small layer; here it is launches only,
// and its sumcheck message, root binding and transcript step run in the launch
// that computes the layer's root.
#include "internal.cuh"
#include "roundhop.cuh"
#include "rounds.cuh"

namespace zc {

// The hop of a layer whose tree stands already.
template <class K>
__global__ void __launch_bounds__(32) k_round_hop(const P2Params* rt, const RoundHop a,
                                                  const uint32_t* root) {
  __shared__ P2Params s_rt;
  __shared__ uint32_t vals[16];
  const P2Params* hp = rt;
  if constexpr (!K::kOwnTables) {
    KIn<K>::make(rt, &s_rt);
    hp = KIn<K>::half(rt, &s_rt);
  }
  pdl_wait();
  HopWarp<K> w;
  w.begin(a, vals, hp);
  w.end(a, vals, root, hp);
}

// Rows and sibling paths of the same q positions in up to kMaxOpen layers, one
// CTA per (position, layer); leaf = (idx >> shift) mod num_leaves as
// zc_merkle_open_reduced.
constexpr int kMaxOpen = 32;
struct OpenTable {
  zc_open_job job[kMaxOpen];
};

__global__ void __launch_bounds__(128) k_open_layers(const __grid_constant__ OpenTable T,
                                                     const int32_t* idx, int q) {
  pdl_wait();
  const zc_open_job& j = T.job[blockIdx.y];
  const zc_leaves& lv = j.leaves;
  const int qi = blockIdx.x;
  const int64_t L = lv.num_leaves;
  const int64_t i = (int64_t)(((uint64_t)(uint32_t)idx[qi] >> j.shift) & (uint64_t)(L - 1));
  const int w = lv.groups * lv.group_len;
  for (int e = threadIdx.x; e < w; e += blockDim.x) {
    const int gq = e / lv.group_len, r = e - gq * lv.group_len;
    j.rows[(int64_t)qi * w + e] = lv.base[gq * lv.group_stride + i * lv.group_len + r];
  }
  const int depth = ilog2_dev(L);
  for (int x = threadIdx.x; x < depth * 8; x += blockDim.x) {
    const int l = x >> 3, word = x & 7;
    const int64_t node = (i >> l) ^ 1;
    j.paths[((int64_t)l * q + qi) * 8 + word] = j.layers[8 * (level_offset(L, l) + node) + word];
  }
}

// Words of the sumcheck's workspace: the partials, two tables each for the mle
// (S/2 and S/4 entries) and the eq (S/4 and S/8) that the rounds swap.
struct RoundSpace {
  size_t partial, mle[2], eq[2], total;
};
inline RoundSpace round_space(int rounds) {
  RoundSpace w;
  const size_t S = (size_t)1 << rounds;
  const auto at_least1 = [](size_t n) { return n ? n : 1; };
  size_t o = 0;
  w.partial = o, o += 4 * (size_t)kRoundPartials;
  w.mle[0] = o, o += 4 * at_least1(S / 2);
  w.mle[1] = o, o += 4 * at_least1(S / 4);
  w.eq[0] = o, o += 4 * at_least1(S / 4);
  w.eq[1] = o, o += 4 * at_least1(S / 8);
  w.total = o;
  return w;
}

}  // namespace zc

using namespace zc;

extern "C" {

size_t zc_fold_rounds_workspace_bytes(int32_t rounds) {
  return rounds < 0 || rounds > 30 ? 0 : 4 * round_space(rounds).total;
}

zc_status zc_fold_rounds(const zc_poseidon2* p, const zc_fold_rounds_desc* d, void* stream) {
  if (!p || !d || d->rounds < 1 || d->log_n < d->rounds || d->log_n > 30) return ZC_BAD_ARG;
  if (!d->codeword || !d->first_tree || !d->final_layer || !d->state || !d->betas || !d->roots ||
      !d->shifts)
    return ZC_BAD_ARG;
  if (d->rounds > 1 && (!d->layers || !d->trees)) return ZC_BAD_ARG;
  if (d->beta_limbs != 1 && d->beta_limbs != 4) return ZC_BAD_ARG;
  if ((uintptr_t)d->first_tree % 16 || (uintptr_t)d->trees % 16 || (uintptr_t)d->layers % 16 ||
      (uintptr_t)d->final_layer % 16 || (uintptr_t)d->betas % 16)
    return ZC_BAD_ARG;
  const bool sc = d->mle != nullptr;
  const RoundSpace ws = round_space(d->rounds);
  uint32_t* const w = (uint32_t*)d->workspace;
  if (sc) {
    if (!d->eq || !d->claim || !d->zinv || !d->msgs || !w) return ZC_BAD_ARG;
    if ((uintptr_t)d->mle % 16 || (uintptr_t)d->eq % 16 || (uintptr_t)d->claim % 16 ||
        (uintptr_t)d->zinv % 16 || (uintptr_t)d->msgs % 16 || (uintptr_t)w % 16)
      return ZC_BAD_ARG;
    if (d->workspace_bytes < 4 * ws.total) return ZC_OOM;
  }
  const zc_field field = p->field;
  // Whatever the folds would refuse is refused here, before the first hop moves
  // the transcript.
  ZC_TRY(with_field(field, [&](auto f) -> zc_status {
    using F = decltype(f);
    if (d->log_n > F::TWO_ADICITY) {
      set_error("fold rounds: the codeword exceeds the field's two-adic range");
      return ZC_BAD_SHAPE;
    }
    if (d->generator != 0 && d->generator != F::GEN) {
      set_error("only the field's canonical generator is built");
      return ZC_UNSUPPORTED;
    }
    for (int r = 0; r < d->rounds; r++)
      if (d->shifts[r] >= F::P) {
        set_error("fold rounds: a coset shift is no field element");
        return ZC_BAD_ARG;
      }
    return ZC_OK;
  }));
  cudaStream_t st = (cudaStream_t)stream;
  const int ef_beta = d->beta_limbs == 4;
  const uint32_t *cw = d->codeword, *mle = d->mle, *eq = d->eq;
  uint32_t *layers = d->layers, *trees = d->trees;
  int ef = d->ef_in ? 1 : 0, np = 0;
  const auto hop_of = [&](int r, int layer_ef) {
    RoundHop h{};
    h.state = d->state;
    h.n = d->beta_limbs;
    h.chal = d->betas + (size_t)r * d->beta_limbs;
    if (sc) {
      h.partial = w + ws.partial;
      h.np = np;
      h.claim = d->claim;
      h.zinv = d->zinv + 4 * (size_t)(d->rounds - 1 - r);
      h.msg = d->msgs + 8 * (size_t)r;
    }
    h.bind = d->bind;
    h.log_height = (uint32_t)(d->log_n - r - 1);
    h.width = (uint32_t)(2 * (layer_ef ? 4 : 1));
    h.raw_out = d->raw_roots ? d->raw_roots + 8 * (size_t)r : nullptr;
    h.root_out = d->roots + 8 * (size_t)r;
    return h;
  };
  if (sc) ZC_TRY(sc_first_partials(field, mle, (int64_t)1 << (d->rounds - 1), eq, w + ws.partial,
                                   &np, st));
  {
    const int64_t L = (int64_t)1 << (d->log_n - 1);
    const RoundHop h = hop_of(0, ef);
    if (d->first_committed) {
      ZC_TRY(with_perm(p, [&](auto k, const P2Params* rt) {
        pdl_launch(k_round_hop<decltype(k)>, 1, 32, 0, st, rt, h,
                                                   d->first_tree + 8 * level_offset(L, d->log_n - 1));
        return launch_check();
      }));
    } else {
      const int limbs = ef ? 4 : 1;
      const zc_leaves lv = d->bit_reversed ? zc_leaves{cw, L, 1, 2 * limbs, 0}
                                           : zc_leaves{cw, L, 2, limbs, L * limbs};
      ZC_TRY(merkle_commit_hop(p, lv, d->first_tree, h, st));
    }
  }
  for (int r = 0; r < d->rounds; r++) {
    const int64_t n = (int64_t)1 << (d->log_n - r);
    const uint32_t* beta = d->betas + (size_t)r * d->beta_limbs;
    const bool last = r == d->rounds - 1;
    if (sc) {  // before the next layer's hop, which takes the partials
      const int64_t M = (int64_t)1 << (d->rounds - 1 - r);
      const uint32_t* msg = d->msgs + 8 * (size_t)r;
      uint32_t* mle_out = w + ws.mle[r & 1];
      if (M >= 2) {
        uint32_t* eq_out = w + ws.eq[r & 1];
        ZC_TRY(sc_fold_partials(field, mle, M, beta, d->beta_limbs, msg, mle_out, eq, eq_out,
                                d->claim, w + ws.partial, &np, st));
        eq = eq_out;
      } else {
        ZC_TRY(zc_sumcheck_fold(field, mle, M, beta, d->beta_limbs, msg, mle_out, nullptr, nullptr,
                                d->claim, stream));
      }
      mle = mle_out;
    }
    if (last) {
      ZC_TRY((d->bit_reversed ? zc_fri_fold_bitrev : zc_fri_fold)(
          field, cw, n, ef, beta, ef_beta, d->shifts[r], d->generator, d->final_layer, stream));
      break;
    }
    const int out_ef = ef | ef_beta;
    const RoundHop h = hop_of(r + 1, out_ef);
    ZC_TRY((d->bit_reversed ? fold_commit_bitrev : fold_commit_natural)(
        p, cw, n, ef, beta, ef_beta, d->shifts[r], d->generator, layers, trees, st, h));
    trees += 8 * (n / 2 - 1);  // 2 (n / 4) - 1 digests
    ef = out_ef;
    cw = layers;
    layers += (n / 2) * (ef ? 4 : 1);
  }
  return ZC_OK;
}

zc_status zc_open_layers(const zc_open_job* jobs, int32_t count, const int32_t* idx, int32_t q,
                         void* stream) {
  if (count < 0 || q < 0 || (count > 0 && !jobs) || (count > 0 && q > 0 && !idx))
    return ZC_BAD_ARG;
  for (int i = 0; i < count; i++) {
    const zc_open_job& j = jobs[i];
    if (!j.layers || (q > 0 && (!j.rows || !j.paths)) || j.shift < 0 || j.shift > 31)
      return ZC_BAD_ARG;
    if (!is_pow2(j.leaves.num_leaves) || j.leaves.num_leaves > (1ll << 32)) return ZC_NOT_POW2;
  }
  if (q == 0) return ZC_OK;
  for (int i = 0; i < count; i += kMaxOpen) {
    OpenTable T;
    const int n = count - i < kMaxOpen ? count - i : kMaxOpen;
    for (int k = 0; k < n; k++) T.job[k] = jobs[i + k];
    for (int k = n; k < kMaxOpen; k++) T.job[k] = zc_open_job{};
    pdl_launch(k_open_layers, dim3((unsigned)q, (unsigned)n), 128, 0, (cudaStream_t)stream, T, idx, q);
    ZC_TRY(launch_check());
  }
  return ZC_OK;
}

}  // extern "C"
