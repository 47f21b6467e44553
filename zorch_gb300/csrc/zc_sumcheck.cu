// The Basefold open's multilinear side on the GPU: eq tables, MLE
// evaluation of committed columns, staggered batching, and the interleaved
// sumcheck rounds (zorch/pcs/basefold/prover.py:419-547,
// zorch/pcs/basefold/kernel.py:52-78, zorch/poly/multilinear.py:92-109,
// zorch/poly/eq.py:55-130). EF4 values are 4 Montgomery limbs (c0..c3).
//
// Field sums are exact, so every reduction here is a deterministic tree of
// per-block partial sums whatever the order.
#include <algorithm>

#include "ef4.cuh"
#include "internal.cuh"
#include "rounds.cuh"

namespace zc {

// expand_eq_to_hypercube(z, 1) for m <= kEqSmall variables, one CTA a table
// (z[0] ends on the top bit): the tables of the upper and the lower half of the
// variables are doubled up side by side in shared memory (out[2i] = s - s z_j,
// out[2i+1] = s z_j), at most six dependent products, and the table is their
// outer product. Doubled through global memory, one step after another,
// twelve variables take 14.5 us.
constexpr int kEqSmall = 12;
struct EqTable {
  const uint32_t* z;
  int m;
  uint32_t* out;
};
template <class F>
__global__ void __launch_bounds__(512) k_eq_small(const EqTable t0, const EqTable t1) {
  pdl_wait();
  constexpr int H = kEqSmall / 2;
  __shared__ __align__(16) uint32_t tab[2][2][4 << H];  // [parity of the step][half][entry]
  const EqTable t = blockIdx.x ? t1 : t0;
  const int m1 = t.m / 2, m2 = t.m - m1;
  const int half = threadIdx.x >> H, i = threadIdx.x & ((1 << H) - 1);  // halves 0 and 1 work
  const int mh = half == 0 ? m1 : m2;
  const uint32_t* zh = half == 0 ? t.z : t.z + 4 * m1;
  if (half < 2 && i == 0) st4(tab[0][half], ef4{{F::ONE, 0, 0, 0}});
  for (int j = 0; j < H; j++) {
    __syncthreads();
    if (half < 2 && j < mh && i < (1 << j)) {
      const ef4 s = ld4(tab[j & 1][half] + 4 * i);
      const ef4 hi = ef_mul<F>(s, ld4(zh + 4 * j));
      st4(tab[(j & 1) ^ 1][half] + 8 * i, ef_sub<F>(s, hi));
      st4(tab[(j & 1) ^ 1][half] + 8 * i + 4, hi);
    }
  }
  __syncthreads();
  const uint32_t *hi = tab[m1 & 1][0], *lo = tab[m2 & 1][1];  // after m1 and m2 steps
  for (int k = threadIdx.x; k < (1 << t.m); k += blockDim.x)
    st4(t.out + 4 * k,
        ef_mul<F>(ld4(hi + 4 * (k >> m2)), ld4(lo + 4 * (k & ((1 << m2) - 1)))));
}

// out[i] = hi[i >> m2] * lo[i & (2^m2 - 1)]: the table of z = (z_hi, z_lo) as
// the outer product of the halves' tables (exact, so equal to the doubling).
template <class F>
__global__ void k_eq_outer(const uint32_t* hi, const uint32_t* lo, int m2, int64_t total,
                           uint32_t* out) {
  pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x)
    st4(out + 4 * i, ef_mul<F>(ld4(hi + 4 * (i >> m2)), ld4(lo + 4 * (i & ((1ll << m2) - 1)))));
}

inline int grid_for(int64_t n, int threads) {
  int64_t b = (n + threads - 1) / threads;
  if (b > 152 * 16) b = 152 * 16;
  return (int)(b > 0 ? b : 1);
}

// Workspace of zc_eq_expand: the two half tables for m > kEqSmall.
inline size_t eq_ws_bytes(int m) {
  if (m <= kEqSmall) return 0;
  const int m1 = m / 2, m2 = m - m1;
  return (size_t)16 * (((size_t)1 << m1) + ((size_t)1 << m2));
}

template <class F>
zc_status eq_expand(const uint32_t* z, int m, uint32_t* out, uint32_t* ws, cudaStream_t st) {
  if (m <= kEqSmall) {
    pdl_launch(k_eq_small<F>, 1, 512, 0, st, EqTable{z, m, out}, EqTable{});
    return launch_check();
  }
  const int m1 = m / 2, m2 = m - m1;
  uint32_t* th = ws;
  uint32_t* tl = ws + ((size_t)4 << m1);
  pdl_launch(k_eq_small<F>, 2, 512, 0, st, EqTable{z, m1, th}, EqTable{z + 4 * m1, m2, tl});
  ZC_TRY(launch_check());
  const int64_t total = (int64_t)1 << m;
  pdl_launch(k_eq_outer<F>, grid_for(total, 256), 256, 0, st, th, tl, m2, total, out);
  return launch_check();
}

// acc[c] += w[c] x for EF4 weights w and base words x, two terms to a reduction:
// |w_e x| <= p * p/2 with x of least magnitude, so two products sum to at most
// p^2, which sredc takes.
template <class F>
__device__ __forceinline__ void ef_dot2(ef4& acc, const ef4& w0, uint32_t x0, const ef4& w1,
                                        uint32_t x1) {
  const int32_t a = centred<F>(x0), b = centred<F>(x1);
#pragma unroll
  for (int e = 0; e < 4; e++)
    acc.c[e] = madd<F>(acc.c[e], snorm<F>(sredc<F>((int64_t)(int32_t)w0.c[e] * a +
                                                   (int64_t)(int32_t)w1.c[e] * b)));
}

// eval_mle of base columns with eq = hi (x) lo: partial[c][h] =
// sum_l lo[l] cols[c][h 2^m2 + l], one CTA per h and kEvalCols columns: a table
// entry (16 bytes) is read once for four column words (4 bytes each), where
// reading it for every word made the table the larger traffic (24 us for 2^20 x
// 8; the columns are 5 us of HBM).
constexpr int kEvalCols = 4;
template <class F>
__global__ void __launch_bounds__(256) k_eval_inner(const uint32_t* cols, int w, int64_t S, int m2,
                                                    const uint32_t* lo, uint32_t* partial,
                                                    int64_t H) {
  pdl_wait();
  const int64_t h = blockIdx.x;
  const int c0 = blockIdx.y * kEvalCols;
  const int64_t L = (int64_t)1 << m2;
  ef4 acc[kEvalCols];
#pragma unroll
  for (int c = 0; c < kEvalCols; c++) acc[c] = ef4{{0, 0, 0, 0}};
  for (int64_t l = threadIdx.x; l < L; l += 2 * blockDim.x) {
    const bool two = l + blockDim.x < L;
    const ef4 w0 = ld4(lo + 4 * l);
    const ef4 w1 = two ? ld4(lo + 4 * (l + blockDim.x)) : ef4{{0, 0, 0, 0}};
#pragma unroll
    for (int c = 0; c < kEvalCols; c++) {
      if (c0 + c >= w) break;
      const uint32_t* col = cols + (c0 + c) * S + h * L + l;
      ef_dot2<F>(acc[c], w0, gld(col), w1, two ? gld(col + blockDim.x) : 0u);
    }
  }
#pragma unroll
  for (int c = 0; c < kEvalCols; c++) {
    if (c0 + c >= w) break;  // the same for the whole CTA
    const ef4 r = block_sum<F>(acc[c]);
    if (threadIdx.x == 0) st4(partial + 4 * ((c0 + c) * H + h), r);
  }
}

// out[c] = sum_h hi[h] partial[c][h], one block per column.
template <class F>
__global__ void __launch_bounds__(256) k_eval_outer(const uint32_t* partial, const uint32_t* hi,
                                                    int64_t H, uint32_t* out) {
  pdl_wait();
  const int64_t c = blockIdx.x;
  ef4 acc{{0, 0, 0, 0}};
  for (int64_t h = threadIdx.x; h < H; h += blockDim.x)
    acc = ef_add<F>(acc, ef_mul<F>(ld4(hi + 4 * h), ld4(partial + 4 * (c * H + h))));
  acc = block_sum<F>(acc);
  if (threadIdx.x == 0) st4(out + 4 * c, acc);
}

// eval_mle workspace: half tables + partial sums.
inline void eval_split(int m, int* m1, int* m2) {
  *m2 = m < kEqSmall ? m : kEqSmall;
  *m1 = m - *m2;
}
inline size_t eval_ws_bytes(int w, int m) {
  int m1, m2;
  eval_split(m, &m1, &m2);
  const size_t H = (size_t)1 << m1;
  return (size_t)16 * (H + ((size_t)1 << m2) + (size_t)w * H) + eq_ws_bytes(m1);
}

template <class F>
zc_status eval_mle(const uint32_t* cols, int w, int m, const uint32_t* z, uint32_t* out,
                   uint32_t* ws, cudaStream_t st) {
  int m1, m2;
  eval_split(m, &m1, &m2);
  const int64_t H = (int64_t)1 << m1, S = (int64_t)1 << m;
  uint32_t* hi = ws;
  uint32_t* lo = hi + 4 * H;
  uint32_t* partial = lo + ((size_t)4 << m2);
  uint32_t* eqws = partial + 4 * (size_t)w * H;
  // z[0 .. m1): high index bits, z[m1 .. m): low ones (m2 <= kEqSmall)
  if (m1 <= kEqSmall) {
    pdl_launch(k_eq_small<F>, 2, 512, 0, st, EqTable{z, m1, hi}, EqTable{z + 4 * m1, m2, lo});
    ZC_TRY(launch_check());
  } else {
    ZC_TRY(eq_expand<F>(z, m1, hi, eqws, st));
    ZC_TRY(eq_expand<F>(z + 4 * m1, m2, lo, eqws, st));
  }
  pdl_launch(k_eval_inner<F>, dim3((unsigned)H, (unsigned)((w + kEvalCols - 1) / kEvalCols)), 256, 0, st, 
      cols, w, S, m2, lo, partial, H);
  ZC_TRY(launch_check());
  pdl_launch(k_eval_outer<F>, (unsigned)w, 256, 0, st, partial, hi, H, out);
  return launch_check();
}

// ---------------------------------------------------------------- rounds --
// s0 partials: sum_j eq[j] mle[2j] over M pairs (mle has 2M EF4 entries).
template <class F>
__global__ void __launch_bounds__(256) k_sc_reduce(const uint32_t* mle, const uint32_t* eq,
                                                   int64_t M, uint32_t* partial) {
  pdl_wait();
  ef4 acc{{0, 0, 0, 0}};
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < M;
       j += (int64_t)gridDim.x * blockDim.x)
    acc = ef_add<F>(acc, ef_mul<F>(ld4(eq + 4 * j), ld4(mle + 8 * j)));
  acc = block_sum<F>(acc);
  if (threadIdx.x == 0) st4(partial + 4 * blockIdx.x, acc);
}

// msg = (s0, s1): s0 = sum of partials, s1 = (claim - s0) / z_last + s0
// (zorch/pcs/basefold/kernel.py:52-66).
template <class F>
__global__ void __launch_bounds__(256) k_sc_message(const uint32_t* partial, int np,
                                                    const uint32_t* claim, const uint32_t* zinv,
                                                    uint32_t* msg) {
  pdl_wait();
  ef4 acc{{0, 0, 0, 0}};
  for (int i = threadIdx.x; i < np; i += blockDim.x) acc = ef_add<F>(acc, ld4(partial + 4 * i));
  acc = block_sum<F>(acc);
  if (threadIdx.x == 0) {
    const ef4 s1 = ef_add<F>(ef_mul<F>(ef_sub<F>(ld4(claim), acc), ld4(zinv)), acc);
    st4(msg, acc);
    st4(msg + 4, s1);
  }
}

// The round's fold (zorch/pcs/basefold/kernel.py:68-74, mle_fold
// zorch/poly/multilinear.py:101-109, contract_hypercube_step zorch/poly/eq.py:65-77):
// mle_out[j] = mle[2j] + beta mle[2j+1] (j < M), eq_out[k] = eq[2k] + eq[2k+1]
// (k < M/2, when eq_out), claim = s0 + beta s1 (block 0).
template <class F>
__global__ void k_sc_fold(const uint32_t* mle, int64_t M, const uint32_t* beta, int beta_limbs,
                          const uint32_t* msg, uint32_t* mle_out, const uint32_t* eq,
                          uint32_t* eq_out, uint32_t* claim) {
  pdl_wait();
  ef4 b{{gld(beta), 0, 0, 0}};
  if (beta_limbs == 4) b = ld4(beta);
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < M;
       j += (int64_t)gridDim.x * blockDim.x) {
    const ef4 e0 = ld4(mle + 8 * j), e1 = ld4(mle + 8 * j + 4);
    st4(mle_out + 4 * j, ef_add<F>(e0, beta_limbs == 4 ? ef_mul<F>(b, e1) : ef_base<F>(e1, b.c[0])));
    if (eq_out && j < M / 2)
      st4(eq_out + 4 * j, ef_add<F>(ld4(eq + 8 * j), ld4(eq + 8 * j + 4)));
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const ef4 s0 = ld4(msg), s1 = ld4(msg + 4);
    st4(claim, ef_add<F>(s0, beta_limbs == 4 ? ef_mul<F>(b, s1) : ef_base<F>(s1, b.c[0])));
  }
}

// The fold of a round and the next round's s0 partials in one pass: thread k <
// M/2 folds outputs 2k and 2k+1 and contracts eq entry k, which are the terms
// eq'[k] mle'[2k] of the next message (k_sc_reduce's sum), so the folded table
// is not read back and the round has one launch fewer.
template <class F>
__global__ void __launch_bounds__(256) k_sc_fold_reduce(const uint32_t* mle, int64_t M,
                                                        const uint32_t* beta, int beta_limbs,
                                                        const uint32_t* msg, uint32_t* mle_out,
                                                        const uint32_t* eq, uint32_t* eq_out,
                                                        uint32_t* claim, uint32_t* partial) {
  pdl_wait();
  ef4 b{{gld(beta), 0, 0, 0}};
  if (beta_limbs == 4) b = ld4(beta);
  const auto mul = [&](const ef4& x) { return beta_limbs == 4 ? ef_mul<F>(b, x) : ef_base<F>(x, b.c[0]); };
  ef4 acc{{0, 0, 0, 0}};
  for (int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < M / 2;
       k += (int64_t)gridDim.x * blockDim.x) {
    const ef4 f0 = ef_add<F>(ld4(mle + 16 * k), mul(ld4(mle + 16 * k + 4)));
    const ef4 f1 = ef_add<F>(ld4(mle + 16 * k + 8), mul(ld4(mle + 16 * k + 12)));
    const ef4 e = ef_add<F>(ld4(eq + 8 * k), ld4(eq + 8 * k + 4));
    st4(mle_out + 8 * k, f0);
    st4(mle_out + 8 * k + 4, f1);
    st4(eq_out + 4 * k, e);
    acc = ef_add<F>(acc, ef_mul<F>(e, f0));
  }
  acc = block_sum<F>(acc);
  if (threadIdx.x == 0) st4(partial + 4 * blockIdx.x, acc);
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    const ef4 s0 = ld4(msg), s1 = ld4(msg + 4);
    st4(claim, ef_add<F>(s0, mul(s1)));
  }
}

// The partial-Lagrange weight of entry `idx` over nbv EF4 challenges: the product
// over the bits of idx, from the top, of r_j or 1 - r_j (zorch/poly/eq.py:55-62).
template <class F>
__device__ __forceinline__ ef4 rlc_weight(const uint32_t* chal, int nbv, int idx) {
  ef4 w{{F::ONE, 0, 0, 0}};
  for (int j = 0; j < nbv; j++) {
    const ef4 wr = ef_mul<F>(w, ef4{{gld(chal + 4 * j), gld(chal + 4 * j + 1),
                                     gld(chal + 4 * j + 2), gld(chal + 4 * j + 3)}});
    w = (idx >> (nbv - 1 - j)) & 1 ? wr : ef_sub<F>(w, wr);
  }
  return w;
}

// Staggered batching with an offset into the weight table and accumulation
// (batch_staggered, zorch/pcs/basefold/batching.py:66-80): out[j] (+)= sum_c
// weights[offset + c] cw[c][j]. A CTA forms its w weights one per thread, then
// two columns go to a reduction (ef_dot2). 2^21 x 8 words from HBM take 31 us, of
// which the bytes 15; 52 with the whole table doubled up by one thread, 10 us and
// more before the first word, and a reduction a column.
template <class F>
__global__ void __launch_bounds__(256) k_rlc_ex(const uint32_t* cw, int64_t n, int w,
                                                const uint32_t* chal, int nbv, int offset,
                                                int accumulate, uint32_t* out) {
  pdl_wait();
  extern __shared__ __align__(16) uint32_t wt[];  // w x 4
  for (int c = threadIdx.x; c < w; c += blockDim.x)
    st4(wt + 4 * c, rlc_weight<F>(chal, nbv, offset + c));
  __syncthreads();
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n;
       j += (int64_t)gridDim.x * blockDim.x) {
    ef4 r{{0, 0, 0, 0}};
    if (accumulate) r = ld4(out + 4 * j);
    const uint32_t* x = cw + j;
    int c = 0;
    for (; c + 4 <= w; c += 4) {
      const uint32_t x0 = gld(x + c * n), x1 = gld(x + (c + 1) * n),
                     x2 = gld(x + (c + 2) * n), x3 = gld(x + (c + 3) * n);
      ef_dot2<F>(r, ld4(wt + 4 * c), x0, ld4(wt + 4 * c + 4), x1);
      ef_dot2<F>(r, ld4(wt + 4 * c + 8), x2, ld4(wt + 4 * c + 12), x3);
    }
    for (; c < w; c += 2) {
      const bool two = c + 1 < w;
      ef_dot2<F>(r, ld4(wt + 4 * c), gld(x + c * n),
                 two ? ld4(wt + 4 * c + 4) : ef4{{0, 0, 0, 0}}, two ? gld(x + (c + 1) * n) : 0u);
    }
    st4(out + 4 * j, r);
  }
}

// out (+)= sum_c weights[offset + c] values[c] (EF4 x EF4): the claim of the
// batch, one column a thread.
template <class F>
__global__ void __launch_bounds__(256) k_rlc_values(const uint32_t* values, int w,
                                                    const uint32_t* chal, int nbv, int offset,
                                                    int accumulate, uint32_t* out) {
  pdl_wait();
  ef4 acc{{0, 0, 0, 0}};
  for (int c = threadIdx.x; c < w; c += blockDim.x)
    acc = ef_add<F>(acc, ef_mul<F>(rlc_weight<F>(chal, nbv, offset + c), ld4(values + 4 * c)));
  acc = block_sum<F>(acc);
  if (threadIdx.x == 0) st4(out, accumulate ? ef_add<F>(acc, ld4(out)) : acc);
}

// [4][n] limbs <-> [n] EF4 words, for a transform that acts limb by limb.
__global__ void __launch_bounds__(256) k_ef4_limbs(const uint32_t* in, int64_t n, int to_limbs,
                                                   uint32_t* out) {
  pdl_wait();
  for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n;
       j += (int64_t)gridDim.x * blockDim.x) {
    if (to_limbs) {
      const ef4 v = ld4(in + 4 * j);
#pragma unroll
      for (int e = 0; e < 4; e++) out[e * n + j] = v.c[e];
    } else {
      st4(out + 4 * j, ef4{{in[j], in[n + j], in[2 * n + j], in[3 * n + j]}});
    }
  }
}

// Up to eight CTAs per SM (each forms the weights once). w <= 4096: 64 KB of them.
template <class F>
zc_status rlc_launch(const uint32_t* cw, int64_t n, int w, const uint32_t* chal, int nbv,
                     int offset, int accumulate, uint32_t* out, cudaStream_t st) {
  const size_t smem = (size_t)16 * w;
  ZC_TRY(allow_smem(k_rlc_ex<F>, smem));
  int64_t blocks = (n + 255) / 256;
  if (blocks > 152 * 8) blocks = 152 * 8;
  pdl_launch(k_rlc_ex<F>, (unsigned)blocks, 256, smem, st, cw, n, w, chal, nbv, offset, accumulate, out);
  return launch_check();
}

constexpr int kReduceBlocks = 256;

template <class F>
__global__ void k_ef4_inv(const uint32_t* in, uint32_t* out, int64_t count) {
  pdl_wait();
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count;
       i += (int64_t)gridDim.x * blockDim.x)
    st4(out + 4 * i, ef_inv<F>(ld4(in + 4 * i)));
}

// ------------------------------------------------- rounds.cuh's two steps --
// One CTA of 256 per 256 items, at most four per SM (the partials are summed by
// one warp, the round's hop).
static int sc_blocks(int64_t items) {
  const int64_t b = (items + 255) / 256;
  return (int)(b < kRoundPartials ? b : kRoundPartials);
}

zc_status sc_first_partials(zc_field field, const uint32_t* mle, int64_t M, const uint32_t* eq,
                            uint32_t* partial, int* np, cudaStream_t st) {
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    *np = sc_blocks(M);
    pdl_launch(k_sc_reduce<F>, *np, 256, 0, st, mle, eq, M, partial);
    return launch_check();
  });
}

zc_status sc_fold_partials(zc_field field, const uint32_t* mle, int64_t M, const uint32_t* beta,
                           int beta_limbs, const uint32_t* msg, uint32_t* mle_out,
                           const uint32_t* eq, uint32_t* eq_out, uint32_t* claim,
                           uint32_t* partial, int* np, cudaStream_t st) {
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    *np = sc_blocks(M / 2);
    pdl_launch(k_sc_fold_reduce<F>, *np, 256, 0, st, mle, M, beta, beta_limbs, msg, mle_out, eq, eq_out,
                                             claim, partial);
    return launch_check();
  });
}

}  // namespace zc

using namespace zc;

extern "C" {

size_t zc_eq_expand_workspace_bytes(int32_t m) { return m < 0 ? 0 : eq_ws_bytes(m); }

zc_status zc_eq_expand(zc_field field, const uint32_t* z, int32_t m, uint32_t* out, void* ws,
                       size_t ws_bytes, void* stream) {
  if (m < 0 || !out || (m > 0 && !z)) return ZC_BAD_ARG;
  if (m > 2 * kEqSmall) return ZC_BAD_SHAPE;
  if ((uintptr_t)out % 16 || (uintptr_t)ws % 16) return ZC_BAD_ARG;
  if (ws_bytes < eq_ws_bytes(m) || (eq_ws_bytes(m) && !ws)) return ZC_OOM;
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    return eq_expand<F>(z, m, out, (uint32_t*)ws, (cudaStream_t)stream);
  });
}

size_t zc_eval_mle_workspace_bytes(int32_t w, int32_t m) {
  return (w <= 0 || m < 0) ? 0 : eval_ws_bytes(w, m);
}

zc_status zc_eval_mle(zc_field field, const uint32_t* cols, int32_t w, int32_t m,
                      const uint32_t* z, uint32_t* out, void* ws, size_t ws_bytes, void* stream) {
  if (w <= 0 || m < 0 || m > 30 || !cols || !out || (m > 0 && !z)) return ZC_BAD_ARG;
  if ((uintptr_t)out % 16 || (uintptr_t)ws % 16) return ZC_BAD_ARG;
  if (!ws || ws_bytes < eval_ws_bytes(w, m)) return ZC_OOM;
  int m1, m2;
  eval_split(m, &m1, &m2);
  if (((int64_t)1 << m1) > 65535 || w > 65535) return ZC_BAD_SHAPE;
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    return eval_mle<F>(cols, w, m, z, out, (uint32_t*)ws, (cudaStream_t)stream);
  });
}

zc_status zc_rlc_columns_ex(zc_field field, const uint32_t* cw, int64_t n, int32_t w,
                            const uint32_t* challenges, int32_t nbv, int32_t offset,
                            int32_t accumulate, uint32_t* out, void* stream) {
  if (!cw || !out || n < 0 || w < 1 || nbv < 0 || nbv > 12 || offset < 0 ||
      offset + w > (1 << nbv) || (nbv > 0 && !challenges))
    return ZC_BAD_ARG;
  if ((uintptr_t)out % 16) return ZC_BAD_ARG;
  if (n == 0) return ZC_OK;
  cudaStream_t st = (cudaStream_t)stream;
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    return rlc_launch<F>(cw, n, w, challenges, nbv, offset, accumulate, out, st);
  });
}

zc_status zc_rlc_columns(zc_field field, const uint32_t* cw, int64_t n, int32_t w,
                         const uint32_t* challenges, uint32_t* out, void* stream) {
  if (!cw || !out || n < 0 || w < 1 || w > 4096) return ZC_BAD_ARG;
  const int nbv = ilog2(w);
  if (nbv > 0 && !challenges) return ZC_BAD_ARG;
  if ((uintptr_t)out % 16) return ZC_BAD_ARG;
  if (n == 0) return ZC_OK;
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    return rlc_launch<F>(cw, n, w, challenges, nbv, 0, 0, out, (cudaStream_t)stream);
  });
}

zc_status zc_ef4_limbs(const uint32_t* in, int64_t n, int32_t to_limbs, uint32_t* out,
                       void* stream) {
  if (n < 0 || (n > 0 && (!in || !out))) return ZC_BAD_ARG;
  if ((uintptr_t)(to_limbs ? in : out) % 16) return ZC_BAD_ARG;
  if (n == 0) return ZC_OK;
  pdl_launch(k_ef4_limbs, grid_for(n, 256), 256, 0, (cudaStream_t)stream, in, n, to_limbs, out);
  return launch_check();
}

zc_status zc_rlc_values(zc_field field, const uint32_t* values, int32_t w,
                        const uint32_t* challenges, int32_t nbv, int32_t offset,
                        int32_t accumulate, uint32_t* out, void* stream) {
  if (!values || !out || w < 1 || nbv < 0 || nbv > 30 || offset < 0 ||
      (nbv < 30 && offset + w > (1 << nbv)) || (nbv > 0 && !challenges))
    return ZC_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    pdl_launch(k_rlc_values<F>, 1, 256, 0, st, values, w, challenges, nbv, offset, accumulate, out);
    return launch_check();
  });
}

zc_status zc_ef4_inv(zc_field field, const uint32_t* in, uint32_t* out, int64_t count,
                     void* stream) {
  if (count < 0 || (count > 0 && (!in || !out))) return ZC_BAD_ARG;
  if ((uintptr_t)in % 16 || (uintptr_t)out % 16) {
    set_error("EF4 operands must be 16-byte aligned");
    return ZC_BAD_ARG;
  }
  if (count == 0) return ZC_OK;
  cudaStream_t st = (cudaStream_t)stream;
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    const int64_t blocks = std::min<int64_t>((count + 127) / 128, 152 * 4);
    pdl_launch(k_ef4_inv<F>, (unsigned)blocks, 128, 0, st, in, out, count);
    return launch_check();
  });
}

size_t zc_sumcheck_workspace_bytes(void) { return (size_t)16 * kReduceBlocks; }

zc_status zc_sumcheck_message(zc_field field, const uint32_t* mle, int64_t M, const uint32_t* eq,
                              const uint32_t* claim, const uint32_t* zinv, uint32_t* msg,
                              void* ws, size_t ws_bytes, void* stream) {
  if (!mle || !eq || !claim || !zinv || !msg || M < 1) return ZC_BAD_ARG;
  if (!ws || ws_bytes < (size_t)16 * kReduceBlocks || (uintptr_t)ws % 16) return ZC_OOM;
  if ((uintptr_t)mle % 16 || (uintptr_t)eq % 16 || (uintptr_t)claim % 16 ||
      (uintptr_t)zinv % 16 || (uintptr_t)msg % 16)
    return ZC_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  return with_field(field, [&](auto f) -> zc_status {
    using F = decltype(f);
    const int blocks = (int)((M + 255) / 256 < kReduceBlocks ? (M + 255) / 256 : kReduceBlocks);
    pdl_launch(k_sc_reduce<F>, blocks, 256, 0, st, mle, eq, M, (uint32_t*)ws);
    ZC_TRY(launch_check());
    pdl_launch(k_sc_message<F>, 1, 256, 0, st, (const uint32_t*)ws, blocks, claim, zinv, msg);
    return launch_check();
  });
}

zc_status zc_sumcheck_fold(zc_field field, const uint32_t* mle, int64_t M, const uint32_t* beta,
                           int32_t beta_limbs, const uint32_t* msg, uint32_t* mle_out,
                           const uint32_t* eq, uint32_t* eq_out, uint32_t* claim, void* stream) {
  if (!mle || !beta || !msg || !mle_out || !claim || M < 1 || (beta_limbs != 1 && beta_limbs != 4))
    return ZC_BAD_ARG;
  if (eq_out && (!eq || M < 2)) return ZC_BAD_ARG;
  if ((uintptr_t)mle % 16 || (uintptr_t)mle_out % 16 || (uintptr_t)claim % 16 ||
      (uintptr_t)msg % 16 || (eq && (uintptr_t)eq % 16) || (eq_out && (uintptr_t)eq_out % 16))
    return ZC_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  return with_field(field, [&](auto f) {
    using F = decltype(f);
    pdl_launch(k_sc_fold<F>, grid_for(M, 256), 256, 0, st, mle, M, beta, beta_limbs, msg, mle_out, eq,
                                                   eq_out, claim);
    return launch_check();
  });
}

}  // extern "C"
