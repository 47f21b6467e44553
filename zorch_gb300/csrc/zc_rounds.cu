// The commit-and-fold rounds of an open in one call: what FriProver's commit
// phase, the Basefold open and the SP1 stacked open share (zorch/pcs/fold.py:
// 90-115, zorch/pcs/basefold/prover.py:419-480, zorch/pcs/jagged/open.py:
// 237-330). A round used to be six to eight calls from Python, 60-80 us of
// host time where the GPU needs 60 for a small layer; here it is launches only,
// and its transcript step, root binding and sumcheck message are one kernel.
#include "duplex.cuh"
#include "ef4.cuh"
#include "internal.cuh"
#include "rounds.cuh"

namespace zc {

struct RoundHop1 {
  uint32_t* state;
  // sumcheck message (msg == nullptr: none): np partial sums of s0
  const uint32_t* partial;
  int np;
  const uint32_t* claim;
  const uint32_t* zinv;
  uint32_t* msg;
  // the layer's root; bind: SP1's separator over [log_height, width]
  const uint32_t* root;
  int bind;
  uint32_t log_height, width;
  uint32_t* raw_out;
  uint32_t* root_out;
  int n_chal;
  uint32_t* chal;
};

// Threads of a round's hop: the CTA sums the message's partials (608 of them took
// one warp 20 us), then its first warp goes on alone.
constexpr int kHopT = 256;

// The round's message (s0 = the partials' sum, s1 = (claim - s0) /
// z_last + s0, zorch/pcs/basefold/kernel.py:52-66), observed; the layer's root,
// bound if asked (k_bind_root's two permutations), observed; n_chal challenge
// words squeezed. A chain of 1 to 5 permutations; as separate launches it was
// three to five of them with a launch gap between each.
template <class K>
__global__ void __launch_bounds__(kHopT) k_round_hop(const P2Params* rt, const RoundHop1 a) {
  using F = typename K::F;
  __shared__ P2Params s_rt;
  __shared__ uint32_t vals[16];
  const int lane = threadIdx.x & 31, l = lane & 15;
  LaneDuplex t;
  uint32_t raw = 0;
  if (threadIdx.x < 32) {
    t.load(a.state);
    raw = a.root[l & 7];
  }
  if constexpr (!K::kOwnTables) {
    KIn<K>::make(rt, &s_rt);  // staged by the whole CTA
    KIn<K>::half(rt, &s_rt);
  }
  if (a.msg) {
    ef4 s0{{0, 0, 0, 0}};
    for (int i = threadIdx.x; i < a.np; i += blockDim.x)
      s0 = ef_add<F>(s0, ld4(a.partial + 4 * i));
    s0 = block_sum<F>(s0);
    if (threadIdx.x == 0) {
      const ef4 s1 = ef_add<F>(ef_mul<F>(ef_sub<F>(ld4(a.claim), s0), ld4(a.zinv)), s0);
      st4(a.msg, s0);
      st4(a.msg + 4, s1);
#pragma unroll
      for (int e = 0; e < 4; e++) {
        vals[e] = s0.c[e];
        vals[4 + e] = s1.c[e];
      }
    }
    __syncthreads();
  }
  if (threadIdx.x >= 32) return;
  const auto body = [&](const auto& perm) {
    // SP1's separator: compress([root, sponge([log_height, width])]). Its first
    // permutation runs on the upper half while the lower one observes the
    // message, when that is one permutation (nothing pending).
    uint32_t sep = l == 0 ? to_mont<F>(a.log_height) : (l == 1 ? to_mont<F>(a.width) : 0u);
    bool sep_done = false;
    if (a.msg) {
      if (a.bind && (t.in_pos & 7) == 0) {
        uint32_t x = lane < 16 ? (l < 8 ? vals[l] : t.x) : sep;
        x = perm.half(x);
        sep = __shfl_sync(kFullMask, x, 16 | l);
        t.absorbed(__shfl_sync(kFullMask, x, l));
        sep_done = true;
      } else {
        t.observe(vals, 8, perm);
      }
    }
    uint32_t root = raw;
    if (a.bind) {
      if (!sep_done) sep = perm.half(sep);
      const uint32_t par = __shfl_sync(kFullMask, sep, (lane & 16) | (l & 7));
      root = perm.half(l < 8 ? raw : par);
    }
    if (lane < 8) {
      if (a.raw_out) a.raw_out[lane] = raw;
      a.root_out[lane] = root;
      vals[8 + lane] = root;
    }
    __syncwarp();
    t.observe(vals + 8, 8, perm);
    for (int i = 0; i < a.n_chal; i++) {
      const uint32_t w = t.sample(perm);
      if (lane == 0) a.chal[i] = w;
    }
  };
  body(CallPerm<K>{K::kOwnTables ? rt : &s_rt});
  t.store(a.state);
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
  cudaStream_t st = (cudaStream_t)stream;
  const zc_field field = p->field;
  const int ef_beta = d->beta_limbs == 4;
  const uint32_t *cw = d->codeword, *mle = d->mle, *eq = d->eq;
  uint32_t *tree = d->first_tree, *layers = d->layers, *trees = d->trees;
  int ef = d->ef_in ? 1 : 0, np = 0;
  if (!d->first_committed) {
    const int64_t L = (int64_t)1 << (d->log_n - 1);
    const int limbs = ef ? 4 : 1;
    const zc_leaves lv = d->bit_reversed ? zc_leaves{cw, L, 1, 2 * limbs, 0}
                                         : zc_leaves{cw, L, 2, limbs, L * limbs};
    ZC_TRY(zc_merkle_commit(p, lv, tree, stream));
  }
  if (sc) ZC_TRY(sc_first_partials(field, mle, (int64_t)1 << (d->rounds - 1), eq, w + ws.partial,
                                   &np, st));
  for (int r = 0; r < d->rounds; r++) {
    const int64_t n = (int64_t)1 << (d->log_n - r), L = n >> 1;
    uint32_t* beta = d->betas + (size_t)r * d->beta_limbs;
    RoundHop1 h{};
    h.state = d->state;
    if (sc) {
      h.partial = w + ws.partial;
      h.np = np;
      h.claim = d->claim;
      h.zinv = d->zinv + 4 * (size_t)(d->rounds - 1 - r);
      h.msg = d->msgs + 8 * (size_t)r;
    }
    h.root = tree + 8 * level_offset(L, d->log_n - r - 1);
    h.bind = d->bind;
    h.log_height = (uint32_t)(d->log_n - r - 1);
    h.width = (uint32_t)(2 * (ef ? 4 : 1));
    h.raw_out = d->raw_roots ? d->raw_roots + 8 * (size_t)r : nullptr;
    h.root_out = d->roots + 8 * (size_t)r;
    h.n_chal = d->beta_limbs;
    h.chal = beta;
    ZC_TRY(with_perm(p, [&](auto k, const P2Params* rt) {
      k_round_hop<decltype(k)><<<1, kHopT, 0, st>>>(rt, h);
      return launch_check();
    }));
    const bool last = r == d->rounds - 1;
    uint32_t* out = last ? d->final_layer : layers;
    if (last) {
      ZC_TRY((d->bit_reversed ? zc_fri_fold_bitrev : zc_fri_fold)(
          field, cw, n, ef, beta, ef_beta, d->shifts[r], d->generator, out, stream));
    } else {
      ZC_TRY((d->bit_reversed ? zc_fri_fold_commit_bitrev : zc_fri_fold_commit)(
          p, cw, n, ef, beta, ef_beta, d->shifts[r], d->generator, out, trees, stream));
      tree = trees;
      trees += 8 * (n / 2 - 1);  // 2 (n / 4) - 1 digests
    }
    ef |= ef_beta;
    cw = out;
    layers += last ? 0 : (n / 2) * (ef ? 4 : 1);
    if (sc) {
      const int64_t M = (int64_t)1 << (d->rounds - 1 - r);
      uint32_t* mle_out = w + ws.mle[r & 1];
      if (M >= 2) {
        uint32_t* eq_out = w + ws.eq[r & 1];
        ZC_TRY(sc_fold_partials(field, mle, M, beta, d->beta_limbs, h.msg, mle_out, eq, eq_out,
                                d->claim, w + ws.partial, &np, st));
        eq = eq_out;
      } else {
        ZC_TRY(zc_sumcheck_fold(field, mle, M, beta, d->beta_limbs, h.msg, mle_out, nullptr,
                                nullptr, d->claim, stream));
      }
      mle = mle_out;
    }
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
    k_open_layers<<<dim3((unsigned)q, (unsigned)n), 128, 0, (cudaStream_t)stream>>>(T, idx, q);
    ZC_TRY(launch_check());
  }
  return ZC_OK;
}

}  // extern "C"
