// A fold round's transcript step (zorch/pcs/fold.py:106-113, zorch/pcs/basefold/
// kernel.py:52-66, zorch/pcs/jagged/open.py:262-296): the sumcheck message,
// observed; the layer's root, bound to its shape if asked, observed; the
// challenge squeezed. Run by one warp, of a launch of its own (zc_rounds.cu) or
// of the launch that computes the root (tree.cuh).
#pragma once
#include "duplex.cuh"
#include "ef4.cuh"

namespace zc {

struct RoundHop {
  uint32_t* state;  // the 34-word duplex state, advanced in place; nullptr: no hop
  int n;            // challenge words to squeeze into chal
  uint32_t* chal;
  // sumcheck message (msg == nullptr: none): np partial sums of s0
  const uint32_t* partial;
  int np;
  const uint32_t* claim;
  const uint32_t* zinv;
  uint32_t* msg;
  // bind: SP1's separator over [log_height, width]; the raw and the observed
  // root are written where asked
  int bind;
  uint32_t log_height, width;
  uint32_t* raw_out;
  uint32_t* root_out;
};

template <class K>
struct HopWarp {
  using F = typename K::F;
  LaneDuplex t;
  uint32_t sep;  // sponge([log_height, width]), word l of each half

  // What does not need the root: the message s0 = the partials' sum, s1 =
  // (claim - s0) / z_last + s0; its observe; the separator's first permutation,
  // on the upper half beside that observe when that is one permutation (nothing
  // pending). vals: 16 words of shared memory.
  __device__ __forceinline__ void begin(const RoundHop& a, uint32_t* vals, const P2Params* hp) {
    const CallPerm<K> perm{hp};
    const int lane = threadIdx.x & 31, l = lane & 15;
    t.load(a.state);
    sep = l == 0 ? to_mont<F>(a.log_height) : (l == 1 ? to_mont<F>(a.width) : 0u);
    bool sep_done = false;
    if (a.msg) {
      ef4 s0{{0, 0, 0, 0}};
      // ten loads in flight: one at a time, 608 partials took a warp 20 us
      for (int i = lane; i < a.np; i += 320) {
        ef4 v[10];
#pragma unroll
        for (int j = 0; j < 10; j++)
          v[j] = i + 32 * j < a.np ? ld4(a.partial + 4 * (i + 32 * j)) : ef4{{0, 0, 0, 0}};
#pragma unroll
        for (int j = 0; j < 10; j++) s0 = ef_add<F>(s0, v[j]);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int e = 0; e < 4; e++)
          s0.c[e] = madd<F>(s0.c[e], __shfl_xor_sync(kFullMask, s0.c[e], o));
      const ef4 s1 = ef_add<F>(ef_mul<F>(ef_sub<F>(ld4(a.claim), s0), ld4(a.zinv)), s0);
      if (lane == 0) {
        st4(a.msg, s0);
        st4(a.msg + 4, s1);
#pragma unroll
        for (int e = 0; e < 4; e++) {
          vals[e] = s0.c[e];
          vals[4 + e] = s1.c[e];
        }
      }
      __syncwarp();
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
    if (a.bind && !sep_done) sep = perm.half(sep);
  }

  // The rest; root: 8 words in shared or global memory.
  __device__ __forceinline__ void end(const RoundHop& a, uint32_t* vals, const uint32_t* root,
                                      const P2Params* hp) {
    const CallPerm<K> perm{hp};
    const int lane = threadIdx.x & 31, l = lane & 15;
    const uint32_t raw = root[l & 7];
    uint32_t bound = raw;
    if (a.bind) {  // compress([root, separator])
      const uint32_t par = __shfl_sync(kFullMask, sep, (lane & 16) | (l & 7));
      bound = perm.half(l < 8 ? raw : par);
    }
    if (lane < 8) {
      if (a.raw_out) a.raw_out[lane] = raw;
      if (a.root_out) a.root_out[lane] = bound;
      vals[8 + lane] = bound;
    }
    __syncwarp();
    t.observe(vals + 8, 8, perm);
    for (int i = 0; i < a.n; i++) {
      const uint32_t w = t.sample(perm);
      if (lane == 0) a.chal[i] = w;
    }
    t.store(a.state);
  }
};

}  // namespace zc
