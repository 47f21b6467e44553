// Width-16 Poseidon2 permutation, sponge and 2-to-1 compression on one thread's
// registers. Semantics follow hash-frx / Plonky3 as pinned by the reference's
// KoalaBear-16 golden root (zorch/commit/testing/merkle_test.py:51-63):
// initial external layer, R_F/2 full rounds, R_P partial rounds, R_F/2 full
// rounds; external layer = M4 = circ(2,3,1,1) per 4-lane block plus the
// lane-class sums; internal layer s_i <- j*sum(s) + diag_i * s_i.
//
// Two constant providers:
//  - Bb16Builtin: the built-in BabyBear-16 instance (x^7, 4+4+13), constants in
//    __constant__ memory, compile-time shape;
//  - RtParams:    any width-16 instance passed at run time (the reference's
//    Poseidon2Params), staged into shared memory by the kernel.
#pragma once
#include <stddef.h>

#include "field.cuh"
#include "poseidon2_babybear16.h"

namespace zc {

// Run-time Poseidon2 parameters (all Montgomery). Mirrors hash-frx's
// Poseidon2Params fields as used at zorch/testkit/koalabear16.py:253-263.
struct P2Params {
  uint32_t field_id;
  uint32_t alpha;
  uint32_t rounds_f_half;
  uint32_t rounds_p;
  uint32_t ext_init[8][16];
  uint32_t ext_term[8][16];
  uint32_t int_rc[64];
  uint32_t diag[16];
  uint32_t j_scale;
  uint32_t j_is_one;
  // diag and j_scale as int32 of least magnitude (RtParams' partial rounds).
  int32_t j_c;
  // Partial rounds of their own (KoalaBear, x^3): kP2Plonky3Kb for Plonky3's
  // diagonal with j = 1, kP2Sp1Kb for SP1's with any j; 0: none.
  int32_t kind;
  alignas(16) int32_t diag_c[16];
  // Derived tables of the half-warp partial rounds (half_partials), for runs of
  // up to `chain` rounds: chain_m[k][i] = j d_i^k as an int32 of least
  // magnitude (0 for word 0), chain_t[k] = j sum_{i>=1} d_i^k, chain_e = j + d_0,
  // chain_mode: 1 where d_0 = -2 j, 2 where j = 1 as well.
  uint32_t chain;
  uint32_t chain_mode;
  uint32_t chain_e;
  uint32_t chain_t[16];
  alignas(16) int32_t chain_m[16][20];  // rows of 16, padded to spread 16-byte reads over the banks
  // kP2Sp1Kb: round r's constant times mu^-r and its S-box's factor mu^2r, and
  // mu^rounds_p, mu = 2^24 j (kb_sp1_partials).
  uint32_t sp1_rc[64];
  uint32_t sp1_mul[64];
  uint32_t sp1_out;
};
constexpr int kChainMax = 16;

// The representative of least magnitude of a word in [0, p).
template <class F>
ZC_HD int32_t centred(uint32_t x) {
  return x > F::P / 2 ? (int32_t)(x - F::P) : (int32_t)x;
}

constexpr int kP2Plonky3Kb = 1, kP2Sp1Kb = 2;

// Which of the two KoalaBear-16 internal diagonals (over j) this is:
// [-2, 1, 2, 1/2, 3, 4, -1/2, -3, -4, 2^-8, 2^-3, 2^-24, -2^-8, -2^-3, -2^-4,
// -2^-24] (Plonky3) or [-2, 1, 2, 4, 8, ..., 2^13, 2^15] (SP1).
template <class F>
inline int p2_kind(const P2Params* p) {
  if (F::ID != KoalaBear::ID || p->alpha != 3) return 0;
  const auto mul = [&](uint32_t c) { return mmul<F>(p->j_scale, c); };
  const auto inv2k = [&](int k) { return mpow<F>(F::INV2, (uint64_t)k); };
  uint32_t plonky3[16], sp1[16];
  const uint32_t three = madd<F>(F::TWO, F::ONE), four = madd<F>(F::TWO, F::TWO);
  const uint32_t d[16] = {mneg<F>(F::TWO), F::ONE,         F::TWO,          F::INV2,
                          three,           four,           mneg<F>(F::INV2), mneg<F>(three),
                          mneg<F>(four),   inv2k(8),       inv2k(3),        inv2k(24),
                          mneg<F>(inv2k(8)), mneg<F>(inv2k(3)), mneg<F>(inv2k(4)),
                          mneg<F>(inv2k(24))};
  for (int i = 0; i < 16; i++) {
    plonky3[i] = d[i];
    sp1[i] = i == 0 ? d[0] : mpow<F>(F::TWO, (uint64_t)(i == 15 ? 15 : i - 1));
  }
  int kind = kP2Plonky3Kb;
  for (int i = 0; i < 16; i++)
    if (p->j_scale != F::ONE || p->diag[i] != plonky3[i]) kind = 0;
  if (kind) return kind;
  kind = kP2Sp1Kb;
  for (int i = 0; i < 16; i++)
    if (p->j_scale == 0 || p->diag[i] != mul(sp1[i])) kind = 0;
  return kind;
}

// Fills the derived constants from diag, j_scale and rounds_p.
template <class F>
inline void p2_chain_tables(P2Params* p) {
  p->j_c = centred<F>(p->j_scale);
  for (int i = 0; i < 16; i++) p->diag_c[i] = centred<F>(p->diag[i]);
  p->kind = p2_kind<F>(p);
  if (p->kind == kP2Sp1Kb) {
    const uint32_t mu = mmul<F>(p->j_scale, mpow<F>(F::TWO, 24)), mu_inv = minv<F>(mu);
    uint32_t up = F::ONE, down = F::ONE;
    for (uint32_t r = 0; r < p->rounds_p; r++) {
      p->sp1_rc[r] = mmul<F>(p->int_rc[r], down);
      p->sp1_mul[r] = mmul<F>(up, up);
      up = mmul<F>(up, mu);
      down = mmul<F>(down, mu_inv);
    }
    p->sp1_out = up;
  }
  const uint32_t runs = (p->rounds_p + kChainMax - 1) / kChainMax;
  p->chain = runs ? (p->rounds_p + runs - 1) / runs : 0;
  p->chain_e = madd<F>(p->j_scale, p->diag[0]);
  p->chain_mode = madd<F>(p->chain_e, p->j_scale) ? 0 : (p->j_is_one ? 2 : 1);
  uint32_t pw[16];
  for (int i = 0; i < 16; i++) pw[i] = F::ONE;
  for (int k = 0; k < kChainMax; k++) {
    uint32_t t = 0;
    for (int i = 0; i < 20; i++) p->chain_m[k][i] = 0;
    for (int i = 1; i < 16; i++) {
      t = madd<F>(t, pw[i]);
      p->chain_m[k][i] = centred<F>(mmul<F>(p->j_scale, pw[i]));
      pw[i] = mmul<F>(pw[i], p->diag[i]);
    }
    p->chain_t[k] = mmul<F>(p->j_scale, t);
  }
}

static __constant__ uint32_t c_bb16_int_rc[ZC_BB16_ROUNDS_P] = ZC_BB16_INT_RC_MONT_INIT;

// Round-constant addition and S-box x -> (x + c)^alpha for x, c in [0, p):
// x + c - p lies in [-p, p) and is one three-operand add, and the power chain
// runs on signed Montgomery products (smul) with a single normalisation at
// the end. Exponents other than 3, 5, 7 take the generic square-and-multiply.
template <class F, int ALPHA>
ZC_HD uint32_t ark_sbox_a(uint32_t x, uint32_t c, uint32_t alpha) {
  const int32_t a = (int32_t)(x + c - F::P);
  if (ALPHA == 3) return snorm<F>(smul<F>(smul<F>(a, a), a));
  if (ALPHA == 5) {
    const int32_t a2 = smul<F>(a, a);
    return snorm<F>(smul<F>(smul<F>(a2, a2), a));
  }
  if (ALPHA == 7) {
    const int32_t a2 = smul<F>(a, a);
    return snorm<F>(smul<F>(smul<F>(a2, a), smul<F>(a2, a2)));
  }
  if (alpha == 3) return ark_sbox_a<F, 3>(x, c, alpha);
  if (alpha == 5) return ark_sbox_a<F, 5>(x, c, alpha);
  if (alpha == 7) return ark_sbox_a<F, 7>(x, c, alpha);
  return mpow<F>(madd<F>(x, c), alpha);
}

// Constants of the built-in instance less p, so that the round-constant addition
// into (-p, p) is a plain two-operand add (ark_sbox_bb16).
struct Bb16Ext {
  uint32_t v[64];
};
constexpr Bb16Ext bb16_less_p(const uint32_t (&c)[64]) {
  Bb16Ext t{};
  for (int i = 0; i < 64; i++) t.v[i] = c[i] - BabyBear::P;
  return t;
}
constexpr uint32_t kBb16ExtInit[64] = ZC_BB16_EXT_INIT_MONT_INIT;
constexpr uint32_t kBb16ExtTerm[64] = ZC_BB16_EXT_TERM_MONT_INIT;
static __constant__ Bb16Ext c_bb16_init_lp = bb16_less_p(kBb16ExtInit);
static __constant__ Bb16Ext c_bb16_term_lp = bb16_less_p(kBb16ExtTerm);
// Zero, but not to the compiler: see smul3.
static __constant__ uint32_t c_zero = 0;

// smul with its subtraction as a three-operand add. The S-boxes of a
// permutation keep the FMA pipe's integer multiplier busy (a 32 x 32 -> 64 or
// high product takes it 4 cycles of a warp, a low product 2, 10 in all per
// Montgomery product; measured), and the compiler likes to spread two-operand
// adds onto that pipe as multiply-adds. A third operand it cannot see to be
// zero keeps the subtraction on the ALU pipe: 5 % less time for the whole
// permutation (1.74 against 1.83 ms for 2^20 threads x 8 permutations).
template <class F>
__device__ __forceinline__ int32_t smul3(int32_t a, int32_t b) {
  const int64_t c = (int64_t)a * b;
  const uint32_t m = (uint32_t)c * F::MU;
  const int32_t mp = __mulhi((int32_t)m, (int32_t)F::P);
  return (int32_t)((uint32_t)(c >> 32) - (uint32_t)mp + c_zero);
}

// Montgomery reduction of c, |c| <= p^2, into (-p, p).
template <class F>
__device__ __forceinline__ int32_t sredc(int64_t c) {
  const uint32_t m = (uint32_t)c * F::MU;
  return (int32_t)(c >> 32) - __mulhi((int32_t)m, (int32_t)F::P);
}

// Products by small constants and powers of two in a field p = A 2^T + 1 with
// 2^31 = p + 2^T - 1 (BabyBear: 15, 27; KoalaBear: 127, 24).
template <class F>
struct Pow2 {
  static constexpr uint32_t P = F::P;
  static constexpr int T = F::TWO_ADICITY;
  static constexpr uint32_t A = (P - 1) >> T;
  static_assert((A << T) + 1 == P && P + (1u << T) - 1 == 0x80000000u, "p = A 2^T + 1");
  __device__ __forceinline__ static uint32_t add(uint32_t a, uint32_t b) { return madd<F>(a, b); }
  __device__ __forceinline__ static uint32_t dbl(uint32_t x) { return madd<F>(x, x); }
  __device__ __forceinline__ static uint32_t half(uint32_t x) {
    return (x >> 1) + (x & 1u) * ((P + 1) >> 1);
  }
  // x 2^-K in (-p, p / 2^K] for x in [0, p).
  template <int K>
  __device__ __forceinline__ static int32_t shr(uint32_t x) {
    static_assert(K >= 1 && K <= T, "k out of range");
    return (int32_t)((x >> K) - (x & ((1u << K) - 1u)) * (A << (T - K)));
  }
  template <int K>
  __device__ __forceinline__ static uint32_t div2exp(uint32_t x) {
    return snorm<F>(shr<K>(x));
  }
  // sum + x 2^-K in [0, p): the sum of the three terms lies in (-p, p + p/2^K],
  // so one correction from below and one from above (an instruction less than
  // normalising x 2^-K first). The first takes its largest value plus p in 32
  // bits: K >= 3 for BabyBear, 6 for KoalaBear.
  template <int K>
  __device__ __forceinline__ static uint32_t add_div2exp(uint32_t sum, uint32_t x) {
    static_assert(K <= T && 2 * (uint64_t)P + (P >> K) < (1ull << 32), "k out of range");
    const uint32_t r =
        snorm<F>((int32_t)((sum + (x >> K)) - (x & ((1u << K) - 1u)) * (A << (T - K))));
    const uint32_t t = r - P;
    return t < r ? t : r;
  }
  // 2^K x: the bits above 2^31 come back as 2^31 = 2^T - 1 (mod p); below 2p
  // for x in [0, p) and K <= 4.
  template <int K>
  __device__ __forceinline__ static uint32_t mul2exp(uint32_t x) {
    static_assert(K >= 1 && K <= 4, "k out of range");
    const uint32_t r = ((x << K) & 0x7fffffffu) + (x >> (31 - K)) * ((1u << T) - 1u);
    const uint32_t t = r - P;
    return t < r ? t : r;
  }
  // The pair of d = 2^-T, carried as h and g = 2^-T h_{r-1} in (-p, 2^(31-T)):
  // h' = sum + 2^-T g, g' = 2^-T h. g > -p, so its shift is in [-A, 0] and the
  // sum of the terms in (-p, p): one correction.
  __device__ __forceinline__ static void lowest_pair(uint32_t sum, uint32_t& h, uint32_t& g) {
    const uint32_t hn = snorm<F>((int32_t)((sum + (uint32_t)((int32_t)g >> T)) -
                                           (g & ((1u << T) - 1u)) * A));
    g = (uint32_t)shr<T>(h);
    h = hn;
  }
};

// The built-in BabyBear-16 instance (x^7, 4 + 4 full and 13 partial rounds),
// one state per thread.
//
// What bounds it: the FMA pipe's multiplier (564 Montgomery products, 5,640
// cycles of a warp) and the ALU pipe, which every high or wide product also
// holds for 2 cycles and each of the 3,498 other instructions for 2. Were both
// always busy, that is (5,640 + 2,256 + 6,996) / 2 = 7,446 cycles; 8,100 measured
// with eight warps a sub-partition, 92 % of it. So an instruction saved is about a cycle saved, and
// the partial rounds, 13 x 118 instructions as written in the definition, are
// rearranged to need fewer:
//  - The diagonal [-2, 1, 2, 1/2, 3, 4, -1/2, -3, -4, 2^-8, 1/4, 1/8, 2^-27,
//    -2^-8, -1/16, -2^-27] holds five pairs (d, -d), at words (3, 6), (4, 7),
//    (5, 8), (9, 13), (12, 15). A pair (a, b) is carried as h = (a + b)/2 and
//    g = (a - b)/2: then h' = sum + d g and g' = d h, so the sum over the
//    words needs one addition per pair, the update one addition per pair, and
//    over two rounds h'' = sum' + d^2 h with no g at all.
//  - Multiplications by 2^-k need no product: p = 15 * 2^27 + 1, so with q the
//    low k bits of x, x 2^-k = (x >> k) - q * 15 * 2^(27-k), in (-p, p).
// 87 instructions per partial round and 5,190 per permutation, where the rounds as
// written in the definition make 5,880: 1.654 against 1.911 ms for 2^20 threads x
// 8 permutations at the same clock.
struct Bb16Builtin {
  using F = BabyBear;
  static constexpr bool kOwnPermute = true;
  static constexpr bool kOwnTables = true;  // the compile-time instance
  // x + c in (-p, p), c_lp = c - p; the power chain is unnormalised.
  __device__ __forceinline__ static uint32_t sbox(uint32_t x, uint32_t c_lp) {
    const int32_t a = (int32_t)(x + c_lp);
    const int32_t a2 = smul3<F>(a, a);
    return snorm<F>(smul3<F>(smul3<F>(a2, a), smul3<F>(a2, a2)));
  }
  // One full round, M4 block by block: the next block's S-boxes (FMA pipe) are
  // independent of this block's additions (ALU pipe).
  __device__ __forceinline__ static void full_round(uint32_t* s, const uint32_t* c_lp);

  // One partial round. For each pair h = h_r and hp = h_{r-1}; for the last one
  // (d = 2^-27, whose square is no power of two that shr takes) hp = g_r =
  // d h_{r-1}, in (-p, 16). FIRST: hp = a - b of the words as they came in.
  template <bool FIRST>
  __device__ __forceinline__ static void partial_round(uint32_t* s, uint32_t (&h)[5],
                                                       uint32_t (&hp)[5], uint32_t c) {
    using B = Pow2<F>;
    const uint32_t y = sbox(s[0], c - F::P);
    const uint32_t H = B::add(B::add(B::add(h[0], h[1]), B::add(h[2], h[3])), h[4]);
    const uint32_t part = B::add(B::add(B::add(s[1], s[2]), B::add(s[10], s[11])),
                                 B::add(s[14], B::dbl(H)));  // words 1..15
    const uint32_t sum = B::add(part, y);
    s[0] = msub<F>(part, y);  // sum - 2 y
    s[1] = B::add(sum, s[1]);
    s[2] = B::add(sum, B::dbl(s[2]));
    s[10] = B::add(sum, B::div2exp<2>(s[10]));
    s[11] = B::add(sum, B::div2exp<3>(s[11]));
    s[14] = msub<F>(sum, B::div2exp<4>(s[14]));
    // h_{r+1} takes hp's place: sum + d^2 h_{r-1}, or sum + d (a - b) / 2
    if (FIRST) {
      hp[0] = B::add(sum, B::div2exp<2>(hp[0]));
      hp[1] = B::add(B::add(sum, hp[1]), B::half(hp[1]));
      hp[2] = B::add(sum, B::dbl(hp[2]));
      hp[3] = B::add_div2exp<9>(sum, hp[3]);
      const uint32_t hn = B::add_div2exp<27>(sum, B::half(hp[4]));
      hp[4] = (uint32_t)B::shr<27>(h[4]);
      h[4] = hn;
    } else {
      hp[0] = B::add(sum, B::div2exp<2>(hp[0]));
      hp[1] = B::add(B::add(sum, hp[1]), B::mul2exp<3>(hp[1]));
      hp[2] = B::add(sum, B::mul2exp<4>(hp[2]));
      hp[3] = B::add_div2exp<16>(sum, hp[3]);
      B::lowest_pair(sum, h[4], hp[4]);
    }
  }
  __device__ __forceinline__ static void partial_rounds(uint32_t* s) {
    using B = Pow2<F>;
    constexpr int ia[5] = {3, 4, 5, 9, 12}, ib[5] = {6, 7, 8, 13, 15};
    uint32_t h[5], hp[5];
#pragma unroll
    for (int i = 0; i < 5; i++) {
      h[i] = B::half(B::add(s[ia[i]], s[ib[i]]));
      hp[i] = msub<F>(s[ia[i]], s[ib[i]]);
    }
    partial_round<true>(s, h, hp, c_bb16_int_rc[0]);
    static_assert(ZC_BB16_ROUNDS_P % 2 == 1, "the remaining rounds run in twos");
    // two rounds per turn: h and hp of the first four pairs change places
#pragma unroll 1
    for (int r = 1; r < ZC_BB16_ROUNDS_P; r += 2) {
      uint32_t cur[5] = {hp[0], hp[1], hp[2], hp[3], h[4]};
      uint32_t old[5] = {h[0], h[1], h[2], h[3], hp[4]};
      partial_round<false>(s, cur, old, c_bb16_int_rc[r]);
      uint32_t cur2[5] = {old[0], old[1], old[2], old[3], cur[4]};
      uint32_t old2[5] = {cur[0], cur[1], cur[2], cur[3], old[4]};
      partial_round<false>(s, cur2, old2, c_bb16_int_rc[r + 1]);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        h[i] = cur2[i];
        hp[i] = old2[i];
      }
      h[4] = cur2[4];
      hp[4] = old2[4];
    }
    // hp[0..3] = h_13 and h[0..3] = h_12 (g_13 = d h_12); h[4], hp[4] = h_13, g_13
    const uint32_t g[5] = {B::half(h[0]), B::add(B::dbl(h[1]), h[1]), B::dbl(B::dbl(h[2])),
                           B::div2exp<8>(h[3]), snorm<F>((int32_t)hp[4])};
    const uint32_t hh[5] = {hp[0], hp[1], hp[2], hp[3], h[4]};
#pragma unroll
    for (int i = 0; i < 5; i++) {
      s[ia[i]] = B::add(hh[i], g[i]);
      s[ib[i]] = msub<F>(hh[i], g[i]);
    }
  }
  __device__ __forceinline__ void permute(uint32_t* s) const;
};

template <class F_>
struct RtParams {
  using F = F_;
  static constexpr bool kOwnTables = false;
#ifdef __CUDA_ARCH__
  static constexpr bool kOwnPermute = true;
#else
  static constexpr bool kOwnPermute = false;
#endif
  const P2Params* p;  // shared memory on the device, plain memory on the host
  ZC_HD int rf_half() const { return (int)p->rounds_f_half; }
  ZC_HD int rp() const { return (int)p->rounds_p; }
  ZC_HD uint32_t ei(int r, int i) const { return p->ext_init[r][i]; }
  ZC_HD uint32_t et(int r, int i) const { return p->ext_term[r][i]; }
  ZC_HD uint32_t ir(int r) const { return p->int_rc[r]; }
  ZC_HD uint32_t dg(int i) const { return p->diag[i]; }
  ZC_HD uint32_t ark_sbox(uint32_t x, uint32_t c) const {
    switch (p->alpha) {
      case 3: return ark_sbox_a<F, 3>(x, c, 3);
      case 5: return ark_sbox_a<F, 5>(x, c, 5);
      case 7: return ark_sbox_a<F, 7>(x, c, 7);
      default: return ark_sbox_a<F, 0>(x, c, p->alpha);
    }
  }
  ZC_HD uint32_t jsum(uint32_t s) const { return p->j_is_one ? s : mmul<F>(s, p->j_scale); }
  // Generic internal layer s_i <- j*sum(s) + diag_i * s_i.
  ZC_HD void internal_layer(uint32_t* s) const {
    uint32_t a0 = madd<F>(madd<F>(s[0], s[1]), madd<F>(s[2], s[3]));
    uint32_t a1 = madd<F>(madd<F>(s[4], s[5]), madd<F>(s[6], s[7]));
    uint32_t a2 = madd<F>(madd<F>(s[8], s[9]), madd<F>(s[10], s[11]));
    uint32_t a3 = madd<F>(madd<F>(s[12], s[13]), madd<F>(s[14], s[15]));
    uint32_t sum = jsum(madd<F>(madd<F>(a0, a1), madd<F>(a2, a3)));
#pragma unroll
    for (int i = 0; i < 16; i++) s[i] = madd<F>(sum, mmul<F>(dg(i), s[i]));
  }
  // One thread's permutation on the device (below).
  __device__ __forceinline__ void permute(uint32_t* s) const;
};

// M4 = circ(2, 3, 1, 1) on one 4-word block.
template <class F>
ZC_HD void m4_block(uint32_t (&x)[4]) {
  const uint32_t t01 = madd<F>(x[0], x[1]), t23 = madd<F>(x[2], x[3]);
  const uint32_t t0123 = madd<F>(t01, t23);
  const uint32_t t01123 = madd<F>(t0123, x[1]), t01233 = madd<F>(t0123, x[3]);
  const uint32_t y3 = madd<F>(t01233, madd<F>(x[0], x[0]));
  const uint32_t y1 = madd<F>(t01123, madd<F>(x[2], x[2]));
  x[0] = madd<F>(t01123, t01);
  x[2] = madd<F>(t01233, t23);
  x[1] = y1;
  x[3] = y3;
}

// External (M4 block-circulant) linear layer.
template <class F>
ZC_HD void p2_ext_linear(uint32_t* s) {
#pragma unroll
  for (int c = 0; c < 16; c += 4) {
    uint32_t x[4] = {s[c], s[c + 1], s[c + 2], s[c + 3]};
    m4_block<F>(x);
#pragma unroll
    for (int k = 0; k < 4; k++) s[c + k] = x[k];
  }
  uint32_t sums[4];
#pragma unroll
  for (int k = 0; k < 4; k++)
    sums[k] = madd<F>(madd<F>(s[k], s[4 + k]), madd<F>(s[8 + k], s[12 + k]));
#pragma unroll
  for (int i = 0; i < 16; i++) s[i] = madd<F>(s[i], sums[i & 3]);
}

__device__ __forceinline__ void Bb16Builtin::full_round(uint32_t* s, const uint32_t* c_lp) {
  uint32_t col[4];
#pragma unroll
  for (int c = 0; c < 16; c += 4) {
    uint32_t x[4];
#pragma unroll
    for (int k = 0; k < 4; k++) x[k] = sbox(s[c + k], c_lp[c + k]);
    m4_block<F>(x);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      s[c + k] = x[k];
      col[k] = c ? madd<F>(col[k], x[k]) : x[k];
    }
  }
#pragma unroll
  for (int i = 0; i < 16; i++) s[i] = madd<F>(s[i], col[i & 3]);
}

__device__ __forceinline__ void Bb16Builtin::permute(uint32_t* s) const {
  p2_ext_linear<F>(s);
#pragma unroll 1
  for (int r = 0; r < ZC_BB16_ROUNDS_F_HALF; r++) full_round(s, c_bb16_init_lp.v + 16 * r);
  partial_rounds(s);
#pragma unroll 1
  for (int r = 0; r < ZC_BB16_ROUNDS_F_HALF; r++) full_round(s, c_bb16_term_lp.v + 16 * r);
}

// A run-time instance, one state per thread, constants from shared memory (rows of
// four words a load). The exponent is chosen once a permutation. A partial
// round's word is d_i s_i + j sum as one 64-bit value, j sum formed once, and
// one reduction: with d_i and j of least magnitude |d_i s_i + j sum| <= p^2,
// which sredc takes. 18 pipe cycles a word where a product, its correction and
// a modular addition take 24.
template <class F, int ALPHA>
__device__ __forceinline__ uint32_t rt_sbox(uint32_t x, uint32_t c, uint32_t alpha) {
  const int32_t a = (int32_t)(x + c - F::P);
  if (ALPHA == 3) return snorm<F>(smul3<F>(smul3<F>(a, a), a));
  if (ALPHA == 7) {
    const int32_t a2 = smul3<F>(a, a);
    return snorm<F>(smul3<F>(smul3<F>(a2, a), smul3<F>(a2, a2)));
  }
  return ark_sbox_a<F, 0>(x, c, alpha);
}

template <class F, int ALPHA>
__device__ __forceinline__ void rt_full_round(uint32_t* s, const uint32_t* c, uint32_t alpha) {
  uint32_t col[4];
#pragma unroll
  for (int b = 0; b < 16; b += 4) {
    const uint4 v = *reinterpret_cast<const uint4*>(c + b);
    uint32_t x[4] = {rt_sbox<F, ALPHA>(s[b], v.x, alpha), rt_sbox<F, ALPHA>(s[b + 1], v.y, alpha),
                     rt_sbox<F, ALPHA>(s[b + 2], v.z, alpha),
                     rt_sbox<F, ALPHA>(s[b + 3], v.w, alpha)};
    m4_block<F>(x);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      s[b + k] = x[k];
      col[k] = b ? madd<F>(col[k], x[k]) : x[k];
    }
  }
#pragma unroll
  for (int i = 0; i < 16; i++) s[i] = madd<F>(s[i], col[i & 3]);
}

// Partial rounds of the KoalaBear-16 instance of Plonky3: its diagonal holds six
// pairs (d, -d), at words (3, 6), (4, 7), (5, 8), (9, 12), (10, 13), (11, 15),
// carried as sums and differences as the built-in BabyBear instance carries its
// five. 70 instructions a round, against 16 products of the general form.
template <bool FIRST>
__device__ __forceinline__ void kb_plonky3_round(uint32_t* s, uint32_t (&h)[6], uint32_t (&hp)[6],
                                                 uint32_t c) {
  using F = KoalaBear;
  using B = Pow2<F>;
  const uint32_t y = rt_sbox<F, 3>(s[0], c, 3);
  const uint32_t H = B::add(B::add(B::add(h[0], h[1]), B::add(h[2], h[3])), B::add(h[4], h[5]));
  const uint32_t part = B::add(B::add(s[1], s[2]), B::add(s[14], B::dbl(H)));
  const uint32_t sum = B::add(part, y);
  s[0] = msub<F>(part, y);  // sum - 2 y
  s[1] = B::add(sum, s[1]);
  s[2] = B::add(sum, B::dbl(s[2]));
  s[14] = msub<F>(sum, B::div2exp<4>(s[14]));
  if (FIRST) {  // hp = a - b: times d / 2
    hp[0] = B::add(sum, B::div2exp<2>(hp[0]));
    hp[1] = B::add(B::add(sum, hp[1]), B::half(hp[1]));
    hp[2] = B::add(sum, B::dbl(hp[2]));
    hp[3] = B::add_div2exp<9>(sum, hp[3]);
    hp[4] = B::add(sum, B::div2exp<4>(hp[4]));
    const uint32_t hn = B::add_div2exp<24>(sum, B::half(hp[5]));
    hp[5] = (uint32_t)B::shr<24>(h[5]);
    h[5] = hn;
  } else {  // hp = h_{r-1}: times d^2
    hp[0] = B::add(sum, B::div2exp<2>(hp[0]));
    hp[1] = B::add(B::add(sum, hp[1]), B::mul2exp<3>(hp[1]));
    hp[2] = B::add(sum, B::mul2exp<4>(hp[2]));
    hp[3] = B::add_div2exp<16>(sum, hp[3]);
    hp[4] = B::add_div2exp<6>(sum, hp[4]);
    B::lowest_pair(sum, h[5], hp[5]);
  }
}

__device__ __forceinline__ void kb_plonky3_partials(uint32_t* s, const P2Params* p) {
  using F = KoalaBear;
  using B = Pow2<F>;
  constexpr int ia[6] = {3, 4, 5, 9, 10, 11}, ib[6] = {6, 7, 8, 12, 13, 15};
  const int rp = (int)p->rounds_p;
  if (rp == 0) return;
  uint32_t h[6], hp[6];
#pragma unroll
  for (int i = 0; i < 6; i++) {
    h[i] = B::half(B::add(s[ia[i]], s[ib[i]]));
    hp[i] = msub<F>(s[ia[i]], s[ib[i]]);
  }
  kb_plonky3_round<true>(s, h, hp, p->int_rc[0]);
  // hp = h_{r+1} and h = h_r of the first five pairs after a round: they change
  // places, two rounds a turn
  int r = 1;
#pragma unroll 1
  for (; r + 1 < rp; r += 2) {
    uint32_t cur[6] = {hp[0], hp[1], hp[2], hp[3], hp[4], h[5]};
    uint32_t old[6] = {h[0], h[1], h[2], h[3], h[4], hp[5]};
    kb_plonky3_round<false>(s, cur, old, p->int_rc[r]);
    uint32_t cur2[6] = {old[0], old[1], old[2], old[3], old[4], cur[5]};
    uint32_t old2[6] = {cur[0], cur[1], cur[2], cur[3], cur[4], old[5]};
    kb_plonky3_round<false>(s, cur2, old2, p->int_rc[r + 1]);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      h[i] = cur2[i];
      hp[i] = old2[i];
    }
    h[5] = cur2[5];
    hp[5] = old2[5];
  }
  if (r < rp) {
    uint32_t cur[6] = {hp[0], hp[1], hp[2], hp[3], hp[4], h[5]};
    uint32_t old[6] = {h[0], h[1], h[2], h[3], h[4], hp[5]};
    kb_plonky3_round<false>(s, cur, old, p->int_rc[r]);
#pragma unroll
    for (int i = 0; i < 5; i++) {
      h[i] = cur[i];
      hp[i] = old[i];
    }
    h[5] = cur[5];
    hp[5] = old[5];
  }
  const uint32_t g[6] = {B::half(h[0]),       B::add(B::dbl(h[1]), h[1]), B::dbl(B::dbl(h[2])),
                         B::div2exp<8>(h[3]), B::div2exp<3>(h[4]),        snorm<F>((int32_t)hp[5])};
  const uint32_t hh[6] = {hp[0], hp[1], hp[2], hp[3], hp[4], h[5]};
#pragma unroll
  for (int i = 0; i < 6; i++) {
    s[ia[i]] = B::add(hh[i], g[i]);
    s[ib[i]] = msub<F>(hh[i], g[i]);
  }
}

// Partial rounds of SP1's KoalaBear-16 instance, s_i' = j (sum + 2^k_i s_i) with
// k = 0, 1, 2, ..., 13, 15 (and -2 for word 0). With t = s / mu^r, mu = 2^24 j,
// they are t_i' = 2^-24 (sum + 2^k_i t_i): every factor 2^(k_i - 24) is a shift
// and one low product. Word 0's S-box takes (t_0 mu^r + c)^3 = mu^3r (t_0 +
// c mu^-r)^3, so a round costs one product more (mu^2r), and the sixteen words
// are scaled by mu^rounds_p at the end.
// Words may exceed p here: t_i' = sum + 2^-e t_i, e = 24 - k_i >= 9, is corrected
// from below only and stays below p + (p + p/512) 2^-e. The excesses of the
// fifteen words sum to less than 0.003 p, so every partial sum of two stays
// below 2.004 p < 2^32 = 2.015 p, and the sum itself is reduced below p (its
// factor 2^-24) before it is used: the bounds hold from round to round.
template <int I>
__device__ __forceinline__ void kb_sp1_words(uint32_t* s, uint32_t sum) {
  if constexpr (I < 16) {
    using F = KoalaBear;
    constexpr int e = 24 - (I == 15 ? 15 : I - 1);
    s[I] = snorm<F>((int32_t)((sum + (s[I] >> e)) - (s[I] & ((1u << e) - 1u)) * (127u << (24 - e))));
    kb_sp1_words<I + 1>(s, sum);
  }
}

__device__ __forceinline__ void kb_sp1_partials(uint32_t* s, const P2Params* p) {
  using F = KoalaBear;
  using B = Pow2<F>;
  const int rp = (int)p->rounds_p;
#pragma unroll 1
  for (int r = 0; r < rp; r++) {
    const int32_t a = (int32_t)(s[0] + p->sp1_rc[r] - F::P);
    const uint32_t y =
        snorm<F>(smul3<F>(smul3<F>(smul3<F>(a, a), a), (int32_t)p->sp1_mul[r]));
    uint32_t q[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      q[k] = B::add(k ? B::add(s[4 * k], s[4 * k + 1]) : s[1], B::add(s[4 * k + 2], s[4 * k + 3]));
    const uint32_t part = B::add(B::add(q[0], q[1]), B::add(q[2], q[3]));
    const uint32_t sum = B::div2exp<24>(B::add(part, y));
    s[0] = B::div2exp<24>(msub<F>(part, y));  // 2^-24 (sum - 2 y)
    kb_sp1_words<1>(s, sum);
  }
  const int32_t out = (int32_t)p->sp1_out;
#pragma unroll
  for (int i = 0; i < 16; i++) s[i] = snorm<F>(smul3<F>((int32_t)s[i], out));
}

template <class F, int ALPHA>
__device__ __forceinline__ void rt_permute_a(uint32_t* s, const P2Params* p) {
  const int rfh = (int)p->rounds_f_half, rp = (int)p->rounds_p;
  const uint32_t alpha = p->alpha;
  p2_ext_linear<F>(s);
#pragma unroll 1
  for (int r = 0; r < rfh; r++) rt_full_round<F, ALPHA>(s, p->ext_init[r], alpha);
  const int kind = F::ID == KoalaBear::ID && ALPHA == 3 ? p->kind : 0;
  if (kind == kP2Plonky3Kb) kb_plonky3_partials(s, p);
  if (kind == kP2Sp1Kb) kb_sp1_partials(s, p);
#pragma unroll 1
  for (int r = 0; r < (kind ? 0 : rp); r++) {
    s[0] = rt_sbox<F, ALPHA>(s[0], p->int_rc[r], alpha);
    uint32_t a[4];
#pragma unroll
    for (int k = 0; k < 4; k++)
      a[k] = madd<F>(madd<F>(s[4 * k], s[4 * k + 1]), madd<F>(s[4 * k + 2], s[4 * k + 3]));
    const uint32_t sum = madd<F>(madd<F>(a[0], a[1]), madd<F>(a[2], a[3]));
    const int64_t js = (int64_t)p->j_c * (int32_t)sum;
#pragma unroll
    for (int b = 0; b < 16; b += 4) {
      const int4 d = *reinterpret_cast<const int4*>(p->diag_c + b);
      s[b] = snorm<F>(sredc<F>(js + (int64_t)d.x * (int32_t)s[b]));
      s[b + 1] = snorm<F>(sredc<F>(js + (int64_t)d.y * (int32_t)s[b + 1]));
      s[b + 2] = snorm<F>(sredc<F>(js + (int64_t)d.z * (int32_t)s[b + 2]));
      s[b + 3] = snorm<F>(sredc<F>(js + (int64_t)d.w * (int32_t)s[b + 3]));
    }
  }
#pragma unroll 1
  for (int r = 0; r < rfh; r++) rt_full_round<F, ALPHA>(s, p->ext_term[r], alpha);
}

template <class F>
__device__ __forceinline__ void RtParams<F>::permute(uint32_t* s) const {
  if (p->alpha == 3)
    rt_permute_a<F, 3>(s, p);
  else if (p->alpha == 7)
    rt_permute_a<F, 7>(s, p);
  else
    rt_permute_a<F, 0>(s, p);
}

#pragma nv_exec_check_disable
template <class K>
ZC_HD void p2_permute(uint32_t* s, const K& k) {
  if constexpr (K::kOwnPermute) {
    k.permute(s);
  } else {
    using F = typename K::F;
    p2_ext_linear<F>(s);
#pragma unroll 1
    for (int r = 0; r < k.rf_half(); r++) {
#pragma unroll
      for (int i = 0; i < 16; i++) s[i] = k.ark_sbox(s[i], k.ei(r, i));
      p2_ext_linear<F>(s);
    }
#pragma unroll 1
    for (int r = 0; r < k.rp(); r++) {
      s[0] = k.ark_sbox(s[0], k.ir(r));
      k.internal_layer(s);
    }
#pragma unroll 1
    for (int r = 0; r < k.rf_half(); r++) {
#pragma unroll
      for (int i = 0; i < 16; i++) s[i] = k.ark_sbox(s[i], k.et(r, i));
      p2_ext_linear<F>(s);
    }
  }
}

// TruncatedPermutation<2, 8, 16>: permute(l || r)[0:8].
#pragma nv_exec_check_disable
template <class K>
ZC_HD void p2_compress(const uint32_t* l, const uint32_t* r, uint32_t* out,
                                            const K& k) {
  uint32_t s[16];
#pragma unroll
  for (int i = 0; i < 8; i++) {
    s[i] = l[i];
    s[8 + i] = r[i];
  }
  p2_permute(s, k);
#pragma unroll
  for (int i = 0; i < 8; i++) out[i] = s[i];
}

// ------------------------------------------------------------- halves ---
// The same permutation on a half-warp (lanes 16h .. 16h+15): lane l of the
// half holds state word l. One thread's permutation is a dependency chain of
// ~5,200 instructions (~9 us at 2.07 GHz); on a half-warp each lane runs one
// S-box per round. The latency-bound parts of a commit -- the narrow top
// levels of a tree and the transcript -- use halves, and what bounds them is
// the dependency chain, so each step is arranged for the fewest dependent
// operations (latencies measured: add 4.5 cycles, add and minimum 9, low
// product 4.5, high or wide product 9.4, shuffle 24):
//  - external layer: y_j = s_b + x_j + 2 x_{j+1} is M4 = circ(2,3,1,1) on the
//    4-word block b (s_b = block sum, j + 1 mod 4), then y += the sum of y over
//    the lane class (l mod 4). The block's and the class's other three words
//    come by three independent shuffles each: two shuffle latencies per layer,
//    not four (a butterfly's);
//  - partial rounds: half_partials.
// 3,720 to 3,930 cycles for the built-in instance by the code around it; 4,900 with
// butterfly sums throughout. Its parts, each repeated by itself: an external layer
// 122 (nine of them), an S-box 108 (eight), the partial rounds 1,837; 3,800 in all.
// Constants come from a P2Params in shared memory. Every lane of the warp must
// make the call (full-warp shuffles), active half or not.
constexpr unsigned kFullMask = 0xffffffffu;

template <class F>
__device__ __forceinline__ uint32_t half_ext_linear(uint32_t x) {
  const uint32_t a = __shfl_xor_sync(kFullMask, x, 1), b = __shfl_xor_sync(kFullMask, x, 2),
                 c = __shfl_xor_sync(kFullMask, x, 3);
  // x_{j+1}: lane j ^ 1 for an even j, j ^ 3 for an odd one
  const uint32_t nxt = (threadIdx.x & 1) ? c : a;
  const uint32_t u = madd<F>(x, madd<F>(nxt, nxt));
  const uint32_t y = madd<F>(madd<F>(madd<F>(x, a), madd<F>(b, c)), u);
  const uint32_t y2 = madd<F>(y, y);
  const uint32_t d = __shfl_xor_sync(kFullMask, y, 4), e = __shfl_xor_sync(kFullMask, y, 8),
                 f = __shfl_xor_sync(kFullMask, y, 12);
  return madd<F>(madd<F>(y2, d), madd<F>(e, f));
}

// f (x + c)^alpha, the factor's product off the dependency chain: it multiplies
// the first power, beside the square. FACTOR = false: f = 1.
template <class F, int ALPHA, bool FACTOR>
__device__ __forceinline__ uint32_t ark_sbox_times(uint32_t x, uint32_t c, uint32_t alpha,
                                                   uint32_t f) {
  if (!FACTOR) return ark_sbox_a<F, ALPHA>(x, c, alpha);
  const int32_t a = (int32_t)(x + c - F::P);
  if (ALPHA == 3) return snorm<F>(smul<F>(smul<F>(a, a), smul<F>(a, (int32_t)f)));
  if (ALPHA == 7) {
    const int32_t a2 = smul<F>(a, a);
    return snorm<F>(smul<F>(smul<F>(a2, smul<F>(a, (int32_t)f)), smul<F>(a2, a2)));
  }
  return mmul<F>(ark_sbox_a<F, ALPHA>(x, c, alpha), f);
}

// n <= 16 partial rounds. Words 1..15 evolve linearly given the rounds' sums, so
// with s_i the words at the start, y_r round r's S-box output and
//   B_r = j * (sum of words 1..15 before round r)
//       = sum_i j d_i^r s_i + sum_{m < r} j T_{r-1-m} sigma_m,  T_k = sum_{i>=1} d_i^k,
// a round is sigma_r = j y_r + B_r and word 0 becomes (j + d_0) y_r + B_r: the chain
// from one S-box to the next is one addition (two products more for a general
// d_0), where summing the fifteen words takes four shuffles and additions. Lane k
// holds B_k: its first sum is a 15-term dot product (15 independent shuffles,
// four terms to a reduction), and each round adds j T_{k-1-r} sigma_r to it
// while the next S-box runs. Each lane l > 0 keeps its own word, x_l = sigma_r
// + d_l x_l, off the chain too. Every lane runs the S-box of word 0. (Keeping x_l
// as one wide accumulation, or B and x on the two halves of a warp in one
// product, measured 10 % and 30 % slower: 2,107 and 2,504 cycles.)
// MODE: 0: any j and d_0; 1: d_0 = -2 j, so word 0 becomes B_r - j y_r; 2: j = 1 too.
// step(r, s0) = the S-box of round r on s0, times j for MODE 1. Returns this
// lane's word.
template <class F, int MODE, bool UNROLL, class Step>
__device__ __forceinline__ uint32_t half_partials(uint32_t x, int n, uint32_t dg, uint32_t j,
                                                  uint32_t e, uint32_t w, const int32_t (&m)[16],
                                                  const Step& step) {
  const int base = threadIdx.x & 16;
  const int32_t xc = centred<F>(x);  // |xc| <= p/2
  int32_t part[4];
#pragma unroll
  for (int g = 0; g < 4; g++) {
    int64_t acc = 0;
#pragma unroll
    for (int i = 4 * g; i < 4 * g + 4; i++)
      if (i) acc += (int64_t)m[i] * __shfl_sync(kFullMask, xc, base + i);  // |term| <= p^2 / 4
    part[g] = sredc<F>(acc);
  }
  uint32_t B = madd<F>(madd<F>(snorm<F>(part[0]), snorm<F>(part[1])),
                       madd<F>(snorm<F>(part[2]), snorm<F>(part[3])));
  uint32_t s0 = __shfl_sync(kFullMask, x, base), b = __shfl_sync(kFullMask, B, base);
  auto round = [&](int r) {
    const uint32_t y = step(r, s0);
    const uint32_t jy = MODE > 0 ? y : mmul<F>(y, j);
    const uint32_t sigma = madd<F>(jy, b);
    s0 = MODE > 0 ? msub<F>(b, jy) : madd<F>(mmul<F>(y, e), b);
    x = madd<F>(sigma, mmul<F>(dg, x));
    B = madd<F>(B, mmul<F>(w, sigma));
    b = __shfl_sync(kFullMask, B, base + ((r + 1) & 15));
    w = __shfl_up_sync(kFullMask, w, 1, 16);  // T_{k-1-r} for the next round
  };
  if constexpr (UNROLL) {
#pragma unroll
    for (int r = 0; r < ZC_BB16_ROUNDS_P; r++) round(r);
  } else {
#pragma unroll 5  // 1: 1,850 cycles for ten rounds of x^3, 5: 1,690
    for (int r = 0; r < n; r++) round(r);
  }
  return (threadIdx.x & 15) == 0 ? s0 : x;
}

// Constants are read from shared memory one round ahead.
template <class F, int ALPHA>
__device__ __forceinline__ uint32_t half_permute_a(uint32_t x, const P2Params* p) {
  const int l = threadIdx.x & 15;
  const int rfh = (int)p->rounds_f_half, rp = (int)p->rounds_p;
  const uint32_t alpha = p->alpha, dg = p->diag[l], js = p->j_scale, e = p->chain_e;
  x = half_ext_linear<F>(x);
  uint32_t c = rfh > 0 ? p->ext_init[0][l] : 0u;
#pragma unroll 1
  for (int r = 0; r < rfh; r++) {
    const uint32_t c_next = r + 1 < rfh ? p->ext_init[r + 1][l] : 0u;
    x = half_ext_linear<F>(ark_sbox_a<F, ALPHA>(x, c, alpha));
    c = c_next;
  }
  if (rp > 0) {
    int32_t m[16];
    const int4* row = reinterpret_cast<const int4*>(p->chain_m[l]);
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const int4 v = row[g];
      m[4 * g] = v.x, m[4 * g + 1] = v.y, m[4 * g + 2] = v.z, m[4 * g + 3] = v.w;
    }
    const uint32_t w = l ? p->chain_t[l - 1] : 0u;
    const int run = (int)p->chain;
#pragma unroll 1
    for (int r0 = 0; r0 < rp; r0 += run) {
      const int n = rp - r0 < run ? rp - r0 : run;
      uint32_t rc = p->int_rc[r0];
      const auto next_rc = [&](int r) {
        const uint32_t cur = rc;
        rc = p->int_rc[r0 + r + 1 < rp ? r0 + r + 1 : 0];
        return cur;
      };
      const auto step = [&](int r, uint32_t s0) {
        return ark_sbox_a<F, ALPHA>(s0, next_rc(r), alpha);
      };
      const auto step_j = [&](int r, uint32_t s0) {
        return ark_sbox_times<F, ALPHA, true>(s0, next_rc(r), alpha, js);
      };
      switch (p->chain_mode) {
        case 2: x = half_partials<F, 2, false>(x, n, dg, js, e, w, m, step); break;
        case 1: x = half_partials<F, 1, false>(x, n, dg, js, e, w, m, step_j); break;
        default: x = half_partials<F, 0, false>(x, n, dg, js, e, w, m, step); break;
      }
    }
  }
  c = rfh > 0 ? p->ext_term[0][l] : 0u;
#pragma unroll 1
  for (int r = 0; r < rfh; r++) {
    const uint32_t c_next = p->ext_term[r + 1 < rfh ? r + 1 : r][l];
    x = half_ext_linear<F>(ark_sbox_a<F, ALPHA>(x, c, alpha));
    c = c_next;
  }
  return x;
}

// Lane l (of the caller's half-warp) passes state word l and gets word l of
// the permuted state back. `p` points to shared memory. Only KoalaBear's
// exponent is inlined; one copy of the rest in a translation unit.
template <class F>
__device__ __noinline__ uint32_t p2_permute_half_any(uint32_t x, const P2Params* p) {
  switch (p->alpha) {
    case 3: return half_permute_a<F, 3>(x, p);
    case 7: return half_permute_a<F, 7>(x, p);
    default: return half_permute_a<F, 0>(x, p);
  }
}
template <class F>
__device__ __forceinline__ uint32_t p2_permute_half(uint32_t x, const P2Params* p) {
  if (F::ID == KoalaBear::ID && p->alpha == 3) return half_permute_a<F, 3>(x, p);
  return p2_permute_half_any<F>(x, p);
}

// ----------------------------------------------------------- quarters ---
// The same permutation on a quarter-warp (lanes 4g .. 4g+3): lane q of the
// quarter holds the M4 block q (state words 4q .. 4q+3) in registers. The
// block matrix M4 is then local arithmetic, and only the sums over the four
// blocks need shuffles (xor 1, xor 2). In the partial rounds every lane keeps
// word 0 itself and runs its S-box redundantly, so the round needs no
// broadcast: the sum over words 1..15 (local, then two shuffle levels) runs
// while the S-box does, and every lane derives the new word 0 from the sum.
// The form for widths between the other two. Cycles of one SM by the number
// of permutations it runs at once (built-in instance; the multiplier pipe binds
// from 64 up, the dependency chain below):
//   permutations      8      16      32      64     128
//   half-warps     3,718   4,617   7,240  13,230
//   quarter-warps          5,500   5,930   7,950  13,130
//   threads                                       18,100
// Every lane of the warp must make the call (full-warp shuffles).
template <class F>
__device__ __forceinline__ void quarter_ext_linear(uint32_t (&x)[4]) {
  m4_block<F>(x);
  uint32_t s[4];
#pragma unroll
  for (int k = 0; k < 4; k++) s[k] = madd<F>(x[k], __shfl_xor_sync(kFullMask, x[k], 1));
#pragma unroll
  for (int k = 0; k < 4; k++) s[k] = madd<F>(s[k], __shfl_xor_sync(kFullMask, s[k], 2));
#pragma unroll
  for (int k = 0; k < 4; k++) x[k] = madd<F>(x[k], s[k]);
}

// One full round; c: the round's sixteen constants (16-byte aligned).
template <class F, int ALPHA>
__device__ __forceinline__ void quarter_full_round(uint32_t (&x)[4], const uint32_t* c,
                                                   uint32_t alpha) {
  const uint4 v = *reinterpret_cast<const uint4*>(c + 4 * (threadIdx.x & 3));
  x[0] = ark_sbox_a<F, ALPHA>(x[0], v.x, alpha);
  x[1] = ark_sbox_a<F, ALPHA>(x[1], v.y, alpha);
  x[2] = ark_sbox_a<F, ALPHA>(x[2], v.z, alpha);
  x[3] = ark_sbox_a<F, ALPHA>(x[3], v.w, alpha);
  quarter_ext_linear<F>(x);
}

// One partial round; w0: word 0, on every lane (lane 0's x[0] is not kept).
// MODE as in half_partials (chain_mode): for 1, y below is j times the S-box.
template <class F, int ALPHA, int MODE>
__device__ __forceinline__ void quarter_partial_round(uint32_t (&x)[4], uint32_t& w0, uint32_t c,
                                                      uint32_t alpha, const uint32_t (&dg)[4],
                                                      uint32_t j, uint32_t d0) {
  const uint32_t y = ark_sbox_times<F, ALPHA, MODE == 1>(w0, c, alpha, j);
  // words 1..15 of this round's input
  uint32_t part = madd<F>(madd<F>((threadIdx.x & 3) ? x[0] : 0u, x[1]), madd<F>(x[2], x[3]));
  part = madd<F>(part, __shfl_xor_sync(kFullMask, part, 1));
  part = madd<F>(part, __shfl_xor_sync(kFullMask, part, 2));
  uint32_t dx[4];
#pragma unroll
  for (int k = 0; k < 4; k++) dx[k] = snorm<F>(smul3<F>((int32_t)x[k], (int32_t)dg[k]));
  if (MODE != 2) part = mmul<F>(part, j);
  const uint32_t sum = madd<F>(part, MODE == 0 ? mmul<F>(y, j) : y);
  // word 0: sum + d_0 y, j part - j y for d_0 = -2 j
  w0 = MODE == 0 ? madd<F>(sum, mmul<F>(d0, y)) : msub<F>(part, y);
#pragma unroll
  for (int k = 0; k < 4; k++) x[k] = madd<F>(sum, dx[k]);
}

template <class F, int ALPHA, int MODE>
__device__ __forceinline__ void quarter_permute_a(uint32_t (&x)[4], const P2Params* p) {
  const int q = threadIdx.x & 3;
  const int rfh = (int)p->rounds_f_half, rp = (int)p->rounds_p;
  const uint32_t alpha = p->alpha;
  const uint4 d = *reinterpret_cast<const uint4*>(p->diag + 4 * q);
  const uint32_t dg[4] = {d.x, d.y, d.z, d.w};
  quarter_ext_linear<F>(x);
#pragma unroll 1
  for (int r = 0; r < rfh; r++) quarter_full_round<F, ALPHA>(x, p->ext_init[r], alpha);
  uint32_t w0 = __shfl_sync(kFullMask, x[0], threadIdx.x & ~3);
#pragma unroll 4  // 1: 6,570 cycles a permutation of x^3 (9,060 for j != 1), 4: 5,900 (6,990)
  for (int r = 0; r < rp; r++)
    quarter_partial_round<F, ALPHA, MODE>(x, w0, p->int_rc[r], alpha, dg, p->j_scale, p->diag[0]);
  if (q == 0) x[0] = w0;
#pragma unroll 1
  for (int r = 0; r < rfh; r++) quarter_full_round<F, ALPHA>(x, p->ext_term[r], alpha);
}

// Lane q (of the caller's quarter-warp) passes state words 4q .. 4q+3 and gets
// them back permuted. `p` points to shared memory.
template <class F>
__device__ __forceinline__ void p2_permute_quarter(uint32_t (&x)[4], const P2Params* p) {
  if (p->alpha == 3 && p->chain_mode == 2) return quarter_permute_a<F, 3, 2>(x, p);
  if (p->alpha == 3 && p->chain_mode == 1) return quarter_permute_a<F, 3, 1>(x, p);
  if (p->alpha == 7 && p->chain_mode == 2) return quarter_permute_a<F, 7, 2>(x, p);
  quarter_permute_a<F, 0, 0>(x, p);
}

// The built-in instance on a quarter-warp: the partial rounds unrolled, their
// constants constant-bank operands (fully unrolled saves 7 % more of a lone
// permutation and 2 % of 128, for 1.5x the code).
__device__ __forceinline__ void quarter_permute_bb16(uint32_t (&x)[4], const P2Params* p) {
  using F = BabyBear;
  const uint4 d = *reinterpret_cast<const uint4*>(p->diag + 4 * (threadIdx.x & 3));
  const uint32_t dg[4] = {d.x, d.y, d.z, d.w};
  quarter_ext_linear<F>(x);
#pragma unroll 1
  for (int r = 0; r < ZC_BB16_ROUNDS_F_HALF; r++) quarter_full_round<F, 7>(x, p->ext_init[r], 7);
  uint32_t w0 = __shfl_sync(kFullMask, x[0], threadIdx.x & ~3);
#pragma unroll
  for (int r = 0; r < ZC_BB16_ROUNDS_P; r++)
    quarter_partial_round<F, 7, 2>(x, w0, c_bb16_int_rc[r], 7, dg, 0u, 0u);
  if ((threadIdx.x & 3) == 0) x[0] = w0;
#pragma unroll 1
  for (int r = 0; r < ZC_BB16_ROUNDS_F_HALF; r++) quarter_full_round<F, 7>(x, p->ext_term[r], 7);
}

// The built-in BabyBear-16 instance on a half-warp: the same rounds as
// half_permute_a, unrolled, this lane's constants in registers (loaded once per
// kernel where permutations follow one another) and the partial-round
// constants read as constant-bank operands, so no round loads a constant or
// runs loop control.
static_assert(ZC_BB16_ROUNDS_F_HALF == 4, "built-in instance: 4 + 4 full rounds");
static_assert(ZC_BB16_ROUNDS_P <= kChainMax, "built-in instance: one run of partial rounds");
struct HalfBb16 {
  uint32_t ei[4], et[4], dg, w;
  int32_t m[16];
  // p: the instance's parameters, in shared or global memory
  __device__ __forceinline__ explicit HalfBb16(const P2Params* p) {
    const int l = threadIdx.x & 15;
#pragma unroll
    for (int r = 0; r < 4; r++) {
      ei[r] = p->ext_init[r][l];
      et[r] = p->ext_term[r][l];
    }
    dg = p->diag[l];
    w = l ? p->chain_t[l - 1] : 0u;
    const int4* row = reinterpret_cast<const int4*>(p->chain_m[l]);
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const int4 v = row[g];
      m[4 * g] = v.x, m[4 * g + 1] = v.y, m[4 * g + 2] = v.z, m[4 * g + 3] = v.w;
    }
  }
  __device__ __forceinline__ uint32_t permute(uint32_t x) const {
    using F = BabyBear;
    x = half_ext_linear<F>(x);
#pragma unroll
    for (int r = 0; r < 4; r++) x = half_ext_linear<F>(ark_sbox_a<F, 7>(x, ei[r], 7));
    x = half_partials<F, 2, true>(x, ZC_BB16_ROUNDS_P, dg, 0u, 0u, w, m, [](int r, uint32_t s0) {
      return ark_sbox_a<F, 7>(s0, c_bb16_int_rc[r], 7);
    });
#pragma unroll
    for (int r = 0; r < 4; r++) x = half_ext_linear<F>(ark_sbox_a<F, 7>(x, et[r], 7));
    return x;
  }
};

// The half-warp permutation out of line, for a round's hop, which has it at five
// places and runs once between large kernels: its code comes from L2 (or, after
// a layer of hundreds of MB, from HBM) each time, 15 KB instead of 75 (5.7 us a
// hop inlined, 4.3 out of line).
template <class K>
__device__ __noinline__ uint32_t half_perm_call(uint32_t x, const P2Params* p) {
  if constexpr (K::kOwnTables)
    return HalfBb16(p).permute(x);
  else
    return p2_permute_half<typename K::F>(x, p);
}

// Stage run-time params into shared memory (whole block participates), the
// words [FROM, TO) of the block: what one thread's permutation reads lies in
// front of the half-warp tables and, for one instance, behind them.
constexpr int kP2Words = (int)(sizeof(P2Params) / 4);
constexpr int kP2ChainAt = (int)(offsetof(P2Params, chain) / 4);
constexpr int kP2Sp1At = (int)(offsetof(P2Params, sp1_rc) / 4);
template <int FROM, int TO>
__device__ __forceinline__ void stage_words(P2Params* dst, const P2Params* src) {
  const uint32_t* s = reinterpret_cast<const uint32_t*>(src);
  uint32_t* d = reinterpret_cast<uint32_t*>(dst);
  for (int i = FROM + threadIdx.x; i < TO; i += blockDim.x) d[i] = s[i];
}

}  // namespace zc
