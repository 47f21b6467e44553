// The Merkle tree machinery shared by the commit and the fused fold-and-commit
// translation units: leaf layouts, the per-level and fused-subtree kernels,
// the tree driver, and the transcript hop run by a tree's root launch.
//
// Large trees: one thread per leaf (k_leaf, no barriers, full occupancy) writes
// the leaf digests; each level wider than tree_shape().levelwise_min nodes is
// one launch of one thread per parent. The small top of a tree, and whole
// small trees, run as fused CTA subtrees (k_subtree): the first level by one
// thread per leaf (or a quarter-warp per parent), every level above by
// quarter- or half-warps out of shared memory, writing every level (the tree
// keeps all layers for openings, zorch/commit/merkle.py:187-202) without
// reading a level back.
#pragma once
#include <stdlib.h>
#include <string.h>

#include <type_traits>

#include "internal.cuh"
#include "roundhop.cuh"

namespace zc {

// Leaf p = concat over q < G of base[q*gs + p*g .. +g] (zc_leaves).
struct LayoutLeaf {
  const uint32_t* base;
  int G, g;
  int64_t gs;
  template <class K>
  __device__ __forceinline__ void digest(int64_t p, uint32_t* d, const K& k) const {
    // PaddingFreeSponge<16, 8, 8> (overwrite mode, no padding)
    uint32_t s[16];
#pragma unroll
    for (int j = 0; j < 16; j++) s[j] = 0;
    const int w = G * g;
    const uint32_t* src = base + p * (int64_t)g;
    int q = 0, r = 0;
    for (int e = 0; e < w; e += 8) {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        if (e + j < w) {
          s[j] = gld(src + (int64_t)q * gs + r);
          if (++r == g) {
            r = 0;
            q++;
          }
        }
      }
      p2_permute(s, k);
    }
#pragma unroll
    for (int j = 0; j < 8; j++) d[j] = s[j];
  }
  // The same on a quarter-warp (lane q holds state words 4q .. 4q+3): lanes 0
  // and 1 end with the digest. Every lane of the warp makes the call; `on`: the
  // quarter has a leaf.
  template <class Perm>
  __device__ __forceinline__ void quarter_digest(int64_t p, bool on, uint32_t (&x)[4],
                                                 const Perm& perm) const {
    const int q4 = 4 * (threadIdx.x & 3);
    const int w = G * g;
    const uint32_t* src = base + p * (int64_t)g;
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = 0;
    for (int e = 0; e < w; e += 8) {
      if (on && q4 < 8) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
          const int i = e + q4 + k;
          if (i < w) {
            const int gi = i / g;
            x[k] = gld(src + (int64_t)gi * gs + (i - gi * g));
          }
        }
      }
      perm(x);
    }
  }
};

// Node p of level l0 from children 2p, 2p+1 of the stored level l0-1.
struct NodeLeaf {
  const uint32_t* in;
  template <class K>
  __device__ __forceinline__ void digest(int64_t p, uint32_t* d, const K& k) const {
    uint32_t a[8], b[8];
    load_digest(in + 16 * p, a);
    load_digest(in + 16 * p + 8, b);
    p2_compress(a, b, d, k);
  }
};

// fri_fold_values on one element j of a natural-order layer of n elements:
// g = (f[j] + f[j+n/2])/2 + beta * (f[j] - f[j+n/2]) * xinv, xinv = 1/(2 x_j)
// (zorch/coding/reed_solomon.py:543-548).
template <class F, int LI, int LB>
struct FoldMath {
  static constexpr int LO = (LI == 4 || LB == 4) ? 4 : 1;
  __device__ __forceinline__ static void fold(const uint32_t* f, int64_t half, int64_t j,
                                              uint32_t xinv, const uint32_t* beta,
                                              uint32_t* out) {
    uint32_t a[4] = {0, 0, 0, 0}, b[4] = {0, 0, 0, 0};
#pragma unroll
    for (int e = 0; e < LI; e++) {
      a[e] = gld(f + j * LI + e);
      b[e] = gld(f + (j + half) * LI + e);
    }
    uint32_t sum[4], d[4];
#pragma unroll
    for (int e = 0; e < LI; e++) {
      sum[e] = mmul<F>(madd<F>(a[e], b[e]), F::INV2);
      d[e] = mmul<F>(msub<F>(a[e], b[e]), xinv);
    }
    if (LO == 1) {
      out[0] = madd<F>(sum[0], mmul<F>(beta[0], d[0]));
    } else if (LB == 1) {  // EF4 layer, base challenge
#pragma unroll
      for (int e = 0; e < 4; e++) out[e] = madd<F>(sum[e], mmul<F>(beta[0], d[e]));
    } else if (LI == 1) {  // base layer, EF4 challenge: beta * d is a scalar multiple
#pragma unroll
      for (int e = 0; e < 4; e++) {
        uint32_t t = mmul<F>(beta[e], d[0]);
        out[e] = e == 0 ? madd<F>(sum[0], t) : t;
      }
    } else {
      ef4 B{{beta[0], beta[1], beta[2], beta[3]}}, D{{d[0], d[1], d[2], d[3]}};
      ef4 r = ef_mul<F>(B, D);
#pragma unroll
      for (int e = 0; e < 4; e++) out[e] = madd<F>(sum[e], r.c[e]);
    }
  }
};

__device__ __forceinline__ int64_t brev64(int64_t i, int bits) {
  return bits ? (int64_t)(__brevll((unsigned long long)i) >> (64 - bits)) : 0;
}

// Leaf p of the next layer's pair tree, computed from the current layer f (n
// elements) and written to g on the way. Natural order (BR = false): the leaf
// is (g[p], g[p + n/4]), g[j] folded from (f[j], f[j + n/2]) at x_j = shift w^j.
// Bit-reversed order (BR = true, BitReversedReedSolomon.fold,
// zorch/coding/reed_solomon.py:484-492, 532-540): the leaf is (g[2p], g[2p+1]),
// g[i] folded from (f[2i], f[2i+1]) at x_i = shift w^brev(i) (i read over
// log2(n/2) bits); brev(2p+1) = brev(2p) + n/4, so x_{2p+1} = x_{2p} w^(n/4).
template <class F, int LI, int LB, bool BR = false>
struct FoldLeaf {
  using M = FoldMath<F, LI, LB>;
  static constexpr int LO = M::LO;
  const uint32_t* f;
  uint32_t* g;
  const uint32_t* beta;
  int64_t n;
  uint32_t inv2s;  // 1 / (2 shift)
  uint32_t winv;   // w_n^-1
  uint32_t w4inv;  // w_n^(-n/4)
  template <class K>
  __device__ __forceinline__ void digest(int64_t p, uint32_t* d, const K& k) const {
    const int64_t quarter = n >> 2, half = n >> 1;
    uint32_t bt[4];
#pragma unroll
    for (int e = 0; e < LB; e++) bt[e] = gld(beta + e);
    uint32_t o0[4], o1[4];
    int64_t i0, i1;
    if (BR) {
      const uint32_t x0 = mmul<F>(inv2s, mpow<F>(winv, (uint64_t)brev64(2 * p, ilog2_dev(half))));
      M::fold(f + 4 * p * LI, 1, 0, x0, bt, o0);
      M::fold(f + (4 * p + 2) * LI, 1, 0, mmul<F>(x0, w4inv), bt, o1);
      i0 = 2 * p;
      i1 = 2 * p + 1;
    } else {
      const uint32_t x0 = mmul<F>(inv2s, mpow<F>(winv, (uint64_t)p));
      M::fold(f, half, p, x0, bt, o0);
      M::fold(f, half, p + quarter, mmul<F>(x0, w4inv), bt, o1);
      i0 = p;
      i1 = p + quarter;
    }
    uint32_t s[16];
#pragma unroll
    for (int j = 0; j < 16; j++) s[j] = 0;
#pragma unroll
    for (int e = 0; e < LO; e++) {
      g[i0 * LO + e] = o0[e];
      g[i1 * LO + e] = o1[e];
      s[e] = o0[e];
      s[LO + e] = o1[e];
    }
    p2_permute(s, k);  // 2*LO <= 8 elements: one absorb block
#pragma unroll
    for (int j = 0; j < 8; j++) d[j] = s[j];
  }
  // On a quarter-warp: lanes 0 and 1 fold one element each.
  template <class Perm>
  __device__ __forceinline__ void quarter_digest(int64_t p, bool on, uint32_t (&x)[4],
                                                 const Perm& perm) const {
    const int q = threadIdx.x & 3;
#pragma unroll
    for (int e = 0; e < 4; e++) x[e] = 0;
    if (on && q < 2) {
      const int64_t quarter = n >> 2, half = n >> 1;
      uint32_t bt[4];
#pragma unroll
      for (int e = 0; e < LB; e++) bt[e] = gld(beta + e);
      uint32_t o[4];
      int64_t i;
      if (BR) {
        uint32_t xi = mmul<F>(inv2s, mpow<F>(winv, (uint64_t)brev64(2 * p, ilog2_dev(half))));
        if (q) xi = mmul<F>(xi, w4inv);
        i = 2 * p + q;
        M::fold(f + 2 * i * LI, 1, 0, xi, bt, o);
      } else {
        uint32_t xi = mmul<F>(inv2s, mpow<F>(winv, (uint64_t)p));
        if (q) xi = mmul<F>(xi, w4inv);
        i = p + q * quarter;
        M::fold(f, half, i, xi, bt, o);
      }
#pragma unroll
      for (int e = 0; e < LO; e++) {
        g[i * LO + e] = o[e];
        x[e] = o[e];
      }
    }
    if (LO == 1) {  // both elements are words of lane 0's block
      const uint32_t second = __shfl_down_sync(kFullMask, x[0], 1);
      if (q == 0) x[1] = second;
      if (q == 1) x[0] = 0;
    }
    perm(x);
  }
};

// Nodes per tree-top CTA of the batched commit (k_tree_top) at its first
// level; its threads: 4 per node, so every level above is one round
// (subtree_level: quarter-warps while a level has more than 16 parents,
// half-warps above).
constexpr int kSubT = 128;
// Largest number of nodes per fused-subtree CTA (k_subtree) at its first
// level.
constexpr int kSubCap = 256;

// The tree driver's shape: levels with more than `levelwise_min` nodes run one
// thread per node; the top runs as fused subtrees of `subtree_t` first-level
// nodes per CTA. Defaults 2^14 and 128 (the 2^22 FRI commit phase, event-timed
// call by call: 4.82 ms against 4.84 at 2^13, 4.99 at 2^15, 5.00 with 256-node
// subtrees; 64-node ones 4.78 there, but 2.15 against 2.13 ms for the Basefold
// open of 2^20 x 8).
// The environment variables ZC_LEVELWISE_MIN_LOG (8..20) and ZC_SUBTREE_T (a
// power of two in 2..256) override them for tuning (read once; no byte of any
// result depends on them).
struct TreeShape {
  int64_t levelwise_min;
  int subtree_t;
};
inline const TreeShape& tree_shape() {
  static const TreeShape shape = [] {
    TreeShape t{(int64_t)1 << 14, 128};
    if (const char* e = getenv("ZC_LEVELWISE_MIN_LOG")) {
      const int v = atoi(e);
      if (v >= 8 && v <= 20) t.levelwise_min = (int64_t)1 << v;
    }
    if (const char* e = getenv("ZC_SUBTREE_T")) {
      const int v = atoi(e);
      if (v >= 2 && v <= kSubCap && (v & (v - 1)) == 0) t.subtree_t = v;
    }
    return t;
  }();
  return shape;
}

// Threads of a subtree CTA of T first-level nodes: a quarter-warp each, at least
// a warp and at most kSubThreads (so the permutations keep their registers: at
// most 128 CTAs are launched at the default shape, so one per SM does). A hop's
// warp comes on top.
constexpr int kSubThreads = 512;
inline int subtree_threads(int T) {
  const int t = 4 * T < kSubThreads ? 4 * T : kSubThreads;
  return t > 32 ? t : 32;
}

// The tree kernels' permutations for the provider K, inlined (out of line, as
// the hop's, measured 1 to 5 % slower on the opens: the constants are loaded per
// call).
template <class K>
__device__ __forceinline__ uint32_t half_perm_k(uint32_t x, const P2Params* hp) {
  if constexpr (K::kOwnTables)
    return HalfBb16(hp).permute(x);
  else
    return p2_permute_half<typename K::F>(x, hp);
}
template <class K>
__device__ __forceinline__ void quarter_perm_k(uint32_t (&x)[4], const P2Params* hp) {
  if constexpr (K::kOwnTables)
    quarter_permute_bb16(x, hp);
  else
    p2_permute_quarter<typename K::F>(x, hp);
}

// Levels of at most this many parents run on half-warps, wider ones on
// quarter-warps (the table at the quarters in poseidon2.cuh: 4,617 against 5,500
// cycles for 16, 7,240 against 5,930 for 32).
constexpr int kHalfMaxWidth = 16;

// One level of a subtree: parent i (< width) = compress(children 2i, 2i+1)
// read from the digest slots `src` ([node][8 words], 16-byte aligned),
// written to the `dst` slots and to the tree's level at `lay`. Wider levels run
// on quarter-warps, Q = W/4 parents a round; narrow ones on half-warps,
// whose permutation has the shorter dependency chain. A warp with no parent in
// a round skips it (a warp-uniform branch: the shuffles need every lane of a
// running warp). W: the threads (whole warps) that work on the tree.
template <class K>
__device__ __forceinline__ void subtree_level(const uint32_t* src, uint32_t* dst, uint32_t* lay,
                                              int width, int W, const P2Params* hp) {
  const int t = threadIdx.x;
  if (width > kHalfMaxWidth || width > (W >> 4)) {
    const int q = t & 3, Q = W >> 2;  // lane q holds words 4q .. 4q+3
    for (int r = 0; r < width; r += Q) {
      if (r + 8 * (t >> 5) >= width) continue;
      const int node = r + (t >> 2);
      const bool on = node < width;
      uint4 v = on ? reinterpret_cast<const uint4*>(src)[4 * node + q] : make_uint4(0, 0, 0, 0);
      uint32_t x[4] = {v.x, v.y, v.z, v.w};
      quarter_perm_k<K>(x, hp);
      if (on && q < 2) {
        const uint4 o = make_uint4(x[0], x[1], x[2], x[3]);
        reinterpret_cast<uint4*>(lay)[2 * node + q] = o;
        reinterpret_cast<uint4*>(dst)[2 * node + q] = o;
      }
    }
    return;
  }
  // half-warps (one round: width <= W/16): lane l holds word l
  const int l = t & 15, node = t >> 4;
  if (2 * (t >> 5) >= width) return;
  const bool on = node < width;
  uint32_t x = on ? src[16 * node + l] : 0u;
  x = half_perm_k<K>(x, hp);
  if (on && l < 8) {
    lay[8 * node + l] = x;
    dst[8 * node + l] = x;
  }
}

// One subtree of T first-level nodes per CTA:
// the first level is T leaf digests (a quarter-warp each: the chain of a
// thread's permutation is 3x as long; for NodeLeaf, stored children
// compressed), then every level up to the subtree root is compressed out of
// ping-pong shared-memory slots (subtree_level), each level written to
// `layers`. A launch that ends at the root can run the layer's transcript step
// as well (hop): one warp more than the tree's W threads does what does not
// need the root -- the sumcheck message, its observe, SP1's separator -- beside
// the levels, and the rest once the root stands. As a launch of its own the step
// came 2 us after the root and took 4 to 8 (Basefold open of 2^20 x 8 with it:
// 2.19 ms, without 2.08). Without a hop the kernel is built without its code (a
// commit of 2^16: 111 us against 115). Barrier 1 is the tree's, 2 the root's;
// every warp of the tree reaches both.
template <class K, class Leaf, bool HOP>
__global__ void __launch_bounds__(kSubThreads + 32, 1)
    k_subtree(Leaf leaf, uint32_t* layers, int64_t L, int l0, int T, const P2Params* rt,
              const RoundHop hop) {
  __shared__ P2Params s_rt;
  __shared__ __align__(16) uint32_t sm[2][8 * kSubCap];  // [node][word] digest slots
  KIn<K>::make(rt, &s_rt);
  const P2Params* hp = KIn<K>::half(rt, &s_rt);
  pdl_wait();
  const int t = threadIdx.x;
  const int W = blockDim.x - (HOP ? 32 : 0);
  if constexpr (HOP) {
    if (t >= W) {  // the hop's warp
      __shared__ uint32_t vals[16];
      HopWarp<K> side;
      side.begin(hop, vals, hp);
      asm volatile("bar.sync 2, %0;" ::"r"((int)blockDim.x) : "memory");
      side.end(hop, vals, sm[(31 - __clz(T)) & 1], hp);
      return;
    }
  }
  const int64_t base = (int64_t)blockIdx.x * T;
  uint32_t* lay0 = layers + 8 * (level_offset(L, l0) + base);
  if constexpr (std::is_same<Leaf, NodeLeaf>::value) {
    subtree_level<K>(leaf.in + 16 * base, sm[0], lay0, T, W, hp);
  } else {
    const int q = t & 3, Q = W >> 2;
    const auto perm = [&](uint32_t (&x)[4]) { quarter_perm_k<K>(x, hp); };
    for (int r = 0; r < T; r += Q) {
      if (r + 8 * (t >> 5) >= T) continue;  // warp-uniform
      const int node = r + (t >> 2);
      const bool on = node < T;
      uint32_t x[4];
      leaf.quarter_digest(base + node, on, x, perm);
      if (on && q < 2) {
        const uint4 o = make_uint4(x[0], x[1], x[2], x[3]);
        reinterpret_cast<uint4*>(lay0)[2 * node + q] = o;
        reinterpret_cast<uint4*>(sm[0])[2 * node + q] = o;
      }
    }
  }
  int cur = 0, lvl = l0, width = T;
  while (width > 1) {
    if constexpr (HOP)
      asm volatile("bar.sync 1, %0;" ::"r"(W) : "memory");  // the tree's warps
    else
      __syncthreads();
    width >>= 1;
    lvl++;
    subtree_level<K>(sm[cur], sm[cur ^ 1],
                     layers + 8 * (level_offset(L, lvl) + (int64_t)blockIdx.x * width), width, W,
                     hp);
    cur ^= 1;
  }
  if constexpr (HOP)  // the root, in sm[cur], for the hop's warp
    asm volatile("bar.sync 2, %0;" ::"r"((int)blockDim.x) : "memory");
}

// Threads of a k_leaf CTA, and the CTAs per SM it is compiled for: eight for the
// built-in instance (54 registers; the register file then holds nine, and 128
// threads measured 1.74 ms where 256 took 1.76-1.79 for 2^20 x 8 permutations);
// no bound for run-time parameter sets, whose constants come from shared memory
// and which would spill under it. Small CTAs also spread a narrow level over
// every SM: 2^15 parents are 256 CTAs, not 128.
constexpr int kLeafT = 128;
template <class K>
struct HashOcc {
  static constexpr int v = 1;
};
template <>
struct HashOcc<Bb16Builtin> {
  static constexpr int v = 8;
};

// One thread per leaf (or per parent for NodeLeaf): no shared memory, no
// barriers, so every warp stays busy for the whole launch.
template <class K, class Leaf>
__global__ void __launch_bounds__(kLeafT, HashOcc<K>::v) k_leaf(Leaf leaf, uint32_t* out, int64_t count,
                                                const P2Params* rt) {
  __shared__ P2Params s_rt;
  K k = KIn<K>::make(rt, &s_rt);
  pdl_wait();
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= count) return;
  uint32_t d[8];
  leaf.digest(p, d, k);
  store_digest(out + 8 * p, d);
}

// The query layer of a query-strided tree (StridedMerkleTree,
// zorch/commit/strided_merkle.py:100-152): node y is the root of the binary
// tree, adjacent pairs in coset order, over the sponge-hashed rows y, y + s, ...,
// y + (rpq-1) s -- what the reference's strided levels compute for residue y.
// A CTA takes `np` nodes, one thread per row, then one per compression of each
// level out of shared memory (row r of node y in slot r * np + y). Against one
// thread folding a whole coset, rpq times the threads: 2^20 rows in cosets of
// 16 are 2^16 threads of 31 permutations each, 3.4 warps where a
// sub-partition needs ten, or 2^20 of one and 2^19, 2^18, ... of the others.
constexpr int kMaxStridedLog = 8;
constexpr int kStridedT = 256;
template <class K>
__global__ void __launch_bounds__(kStridedT, 4) k_strided(LayoutLeaf rows, int64_t s, int log_rpq,
                                                         int np, uint32_t* out,
                                                         const P2Params* rt) {
  __shared__ P2Params s_rt;
  __shared__ __align__(16) uint32_t sm[8 * kStridedT];
  K k = KIn<K>::make(rt, &s_rt);
  pdl_wait();
  const int t = threadIdx.x;
  const int64_t y0 = (int64_t)blockIdx.x * np;
  int width = np << log_rpq;  // digests of the current level
  const int r = t / np, y = t - r * np;
  uint32_t d[8];
  if (t < width) {
    rows.digest(y0 + y + (int64_t)r * s, d, k);
    if (log_rpq) store_digest(sm + 8 * t, d);
  }
  for (int l = 0; l < log_rpq; l++) {
    __syncthreads();
    width >>= 1;
    uint32_t a[8], b[8];
    if (t < width) {  // children (2r, y), (2r + 1, y)
      load_digest(sm + 8 * (2 * r * np + y), a);
      load_digest(sm + 8 * ((2 * r + 1) * np + y), b);
    }
    __syncthreads();  // read before anyone overwrites
    if (t < width) {
      p2_compress(a, b, d, k);
      store_digest(sm + 8 * t, d);
    }
  }
  if (t < width) store_digest(out + 8 * (y0 + t), d);
}

// `ctas` subtrees of T nodes at level l0; a hop only with ctas == 1.
template <class K, class Leaf>
zc_status subtree_launch(const Leaf& leaf, uint32_t* layers, int64_t L, int l0, int T, int64_t ctas,
                         const P2Params* rt, cudaStream_t st, const RoundHop& hop) {
  const int threads = subtree_threads(T);
  if (hop.state)
    pdl_launch(k_subtree<K, Leaf, true>, (unsigned)ctas, threads + 32, 0, st, leaf, layers, L, l0, T, rt,
                                                                      hop);
  else
    pdl_launch(k_subtree<K, Leaf, false>, (unsigned)ctas, threads, 0, st, leaf, layers, L, l0, T, rt, hop);
  return launch_check();
}

// Levels with more than tree_shape().levelwise_min nodes run one thread per
// node (k_leaf with NodeLeaf, throughput-bound: a level this wide fills the
// GPU); the narrower top of the tree is latency-bound and runs as fused CTA
// subtrees (k_subtree with NodeLeaf), log2(T)+1 levels per launch.
// Launches the levels above `l_done` (all levels <= l_done already stored).
template <class K>
zc_status finish_tree(uint32_t* layers, int64_t L, int l_done, const P2Params* rt,
                      cudaStream_t st, const RoundHop& hop = RoundHop{}) {
  const int depth = ilog2(L);
  const int sub_t = tree_shape().subtree_t;
  int l = l_done;
  while (l < depth) {
    const int64_t parents = (L >> l) >> 1;
    NodeLeaf nl{layers + 8 * level_offset(L, l)};
    if (parents > tree_shape().levelwise_min) {
      pdl_launch(k_leaf<K, NodeLeaf>, (unsigned)((parents + kLeafT - 1) / kLeafT), kLeafT, 0, st, 
          nl, layers + 8 * level_offset(L, l + 1), parents, rt);
      ZC_TRY(launch_check());
      l += 1;
      continue;
    }
    const int T = parents < sub_t ? (int)parents : sub_t;
    const bool top = parents == T;  // this launch's single CTA makes the root
    ZC_TRY(subtree_launch<K>(nl, layers, L, l + 1, T, parents / T, rt, st, top ? hop : RoundHop{}));
    l += 1 + ilog2(T);
  }
  return ZC_OK;
}

template <class K, class Leaf>
zc_status commit_tree(const Leaf& leaf, uint32_t* layers, int64_t L, const P2Params* rt,
                      cudaStream_t st, const RoundHop& hop = RoundHop{}) {
  if (L > tree_shape().levelwise_min) {
    pdl_launch(k_leaf<K, Leaf>, (unsigned)((L + kLeafT - 1) / kLeafT), kLeafT, 0, st, leaf, layers, L, rt);
    ZC_TRY(launch_check());
    return finish_tree<K>(layers, L, 0, rt, st, hop);
  }
  const int sub_t = tree_shape().subtree_t;
  const int T0 = L < sub_t ? (int)L : sub_t;
  const bool top = L == T0;
  ZC_TRY(subtree_launch<K>(leaf, layers, L, 0, T0, L / T0, rt, st, top ? hop : RoundHop{}));
  return finish_tree<K>(layers, L, ilog2(T0), rt, st, hop);
}

constexpr int kMaxHopChallenges = 64;

inline zc_status check_hop(const uint32_t* state, int32_t n_chal, const uint32_t* chal) {
  if (!state || n_chal < 0 || n_chal > kMaxHopChallenges || (n_chal > 0 && !chal)) {
    set_error("a root hop needs the 34-word state and 0..64 challenge words");
    return ZC_BAD_ARG;
  }
  return ZC_OK;
}

}  // namespace zc
