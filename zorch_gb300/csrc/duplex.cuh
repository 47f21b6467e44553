// The Fiat-Shamir duplex state machine (DuplexTranscript,
// zorch/transcript.py:239-481) shared by the transcript kernels and the
// tree-top kernels that run a round's transcript hop in the same launch.
#pragma once
#include <type_traits>

#include "internal.cuh"

namespace zc {

// ------------------------------------------------------------ duplex ------
// The DuplexTranscript state machine (zorch/transcript.py:239-481) on one
// thread. Packed state: in_buf[8] out_buf[8] sponge[16] in_pos out_pos.
struct Duplex {
  uint32_t in_buf[8];
  uint32_t out_buf[8];
  uint32_t sponge[16];
  int32_t in_pos;
  int32_t out_pos;
};

// _observe_body (zorch/transcript.py:637-748): the stream in_buf[0:in_pos] ++
// values is absorbed a full rate block at a time (overwrite sponge[0:8],
// permute); the tail stays pending; a fresh output iff no tail remains.
// `perm(s)` permutes the 16-word sponge in place. The host's form; the device's is
// LaneDuplex.
#pragma nv_exec_check_disable
template <class Perm>
ZC_HD void duplex_observe(Duplex& t, const uint32_t* v, int64_t m, const Perm& perm) {
  if (m <= 0) return;
  int pos = t.in_pos & 7;  // a corrupt caller state cannot index past the buffer
  for (int64_t i = 0; i < m; i++) {
    t.in_buf[pos++] = v[i];
    if (pos == 8) {
      for (int j = 0; j < 8; j++) t.sponge[j] = t.in_buf[j];
      perm(t.sponge);
      pos = 0;
    }
  }
  for (int j = pos; j < 8; j++) t.in_buf[j] = 0;
  t.in_pos = pos;
  if (pos == 0) {
    for (int j = 0; j < 8; j++) t.out_buf[j] = t.sponge[j];
    t.out_pos = 8;
  } else {
    for (int j = 0; j < 8; j++) t.out_buf[j] = 0;
    t.out_pos = 0;
  }
}

// _sample_one (zorch/transcript.py:370-387) n times; _duplexing (:299-313)
// merges the pending prefix over sponge[0:in_pos] (:154-163) and permutes.
#pragma nv_exec_check_disable
template <class Perm>
ZC_HD void duplex_sample(Duplex& t, int n, uint32_t* out, const Perm& perm) {
  t.in_pos &= 7;
  if (t.out_pos < 0 || t.out_pos > 8) t.out_pos = 0;
  for (int i = 0; i < n; i++) {
    if (t.in_pos > 0 || t.out_pos == 0) {
      for (int j = 0; j < t.in_pos; j++) t.sponge[j] = t.in_buf[j];
      perm(t.sponge);
      for (int j = 0; j < 8; j++) {
        t.in_buf[j] = 0;
        t.out_buf[j] = t.sponge[j];
      }
      t.in_pos = 0;
      t.out_pos = 8;
    }
    t.out_pos -= 1;
    out[i] = t.out_buf[t.out_pos];
  }
}

template <class K>
struct HostPerm {
  const K& k;
  void operator()(uint32_t* s) const { p2_permute(s, k); }
};

// The half-warp permutation of a transcript kernel: run-time instances
// (constants in shared memory) and the built-in one (this lane's constants in
// registers, loaded once when the kernel starts).
template <class F>
struct HalfPerm {
  const P2Params* p;  // shared memory
  __device__ uint32_t half(uint32_t x) const { return p2_permute_half<F>(x, p); }
};
struct HalfPermBb16 {
  HalfBb16 h;
  __device__ explicit HalfPermBb16(const P2Params* p) : h(p) {}
  __device__ uint32_t half(uint32_t x) const { return h.permute(x); }
};

// Calls fn(perm) with the transcript's half-warp permutation: the unrolled
// built-in form for the built-in instance, the run-time form (constants
// staged to shared memory) otherwise.
template <class K, class Fn>
__device__ __forceinline__ void with_half_perm(const P2Params* rt, P2Params* s_rt, Fn&& fn) {
  if constexpr (std::is_same<K, Bb16Builtin>::value) {
    const HalfPermBb16 perm(rt);
    fn(perm);
  } else {
    KIn<K>::make(rt, s_rt);
    const HalfPerm<typename K::F> perm{KIn<K>::half(rt, s_rt)};
    fn(perm);
  }
}

// The same out of line; p: the parameters, in shared memory or, for the built-in
// instance, anywhere.
template <class K>
struct CallPerm {
  const P2Params* p;
  __device__ __forceinline__ uint32_t half(uint32_t x) const { return half_perm_call<K>(x, p); }
};

// The duplex on one warp: lane l of each half (both run the same) holds sponge
// word l and, for l < 8, words l of the input and output buffers. The same
// steps as duplex_observe and duplex_sample with no word-by-word state in
// memory: a step costs its permutations and a few shuffles (a hop of one
// absorbed block and four squeezed words took 8 us with the state in local
// arrays, of which the permutation 2.5).
struct LaneDuplex {
  uint32_t in, out, x;
  int in_pos, out_pos;

  // buffers of the wire layout: in_buf[8], out_buf[8], sponge[16]
  __device__ __forceinline__ void load(const uint32_t* in_buf, const uint32_t* out_buf,
                                       const uint32_t* sponge, const uint32_t* in_p,
                                       const uint32_t* out_p) {
    const int l = threadIdx.x & 15;
    in = l < 8 ? in_buf[l] : 0u;
    out = l < 8 ? out_buf[l] : 0u;
    x = sponge[l];
    in_pos = (int)in_p[0];
    out_pos = (int)out_p[0];
  }
  // Inputs may alias outputs: every lane has read them by now.
  __device__ __forceinline__ void store(uint32_t* in_buf, uint32_t* out_buf, uint32_t* sponge,
                                        uint32_t* in_p, uint32_t* out_p) const {
    __syncwarp();
    const int lane = threadIdx.x & 31;
    if (lane < 8) {
      in_buf[lane] = in;
      out_buf[lane] = out;
    }
    if (lane < 16) sponge[lane] = x;
    if (lane == 0) {
      in_p[0] = (uint32_t)in_pos;
      out_p[0] = (uint32_t)out_pos;
    }
  }
  __device__ __forceinline__ void load(const uint32_t* st) {
    load(st, st + 8, st + 16, st + 32, st + 33);
  }
  __device__ __forceinline__ void store(uint32_t* st) const {
    store(st, st + 8, st + 16, st + 32, st + 33);
  }

  template <class HP>
  __device__ __forceinline__ void observe(const uint32_t* v, int64_t m, const HP& perm) {
    if (m <= 0) return;
    const int l = threadIdx.x & 15;
    int pos = in_pos & 7;  // a corrupt caller state cannot index past the buffer
    int64_t i = 0;
    // a pending block is completed first; then whole blocks, each one's words
    // loaded before the permutation that precedes them; the tail stays pending
    uint32_t nxt = 0;
    if (pos != 0) {
      const int take = m < 8 - pos ? (int)m : 8 - pos;
      if (l >= pos && l < pos + take) in = v[l - pos];
      pos += take;
      i = take;
      if (pos == 8) nxt = in;
    } else if (m >= 8) {
      nxt = l < 8 ? v[l] : 0u;
      pos = 8;
      i = 8;
    }
    while (pos == 8) {
      if (l < 8) x = nxt;
      pos = 0;
      if (m - i >= 8) {
        if (l < 8) nxt = v[i + l];
        pos = 8;
        i += 8;
      }
      x = perm.half(x);
    }
    if (pos == 0 && i < m) {
      pos = (int)(m - i);
      if (l < pos) in = v[i + l];
    }
    if (l >= pos) in = 0u;
    in_pos = pos;
    out = pos == 0 && l < 8 ? x : 0u;
    out_pos = pos == 0 ? 8 : 0;
  }

  // After a whole block has been absorbed with nothing pending: y, the permuted
  // sponge's word of this lane.
  __device__ __forceinline__ void absorbed(uint32_t y) {
    x = y;
    in = 0u;
    in_pos = 0;
    out = (threadIdx.x & 15) < 8 ? y : 0u;
    out_pos = 8;
  }

  // The next challenge word, on every lane.
  template <class HP>
  __device__ __forceinline__ uint32_t sample(const HP& perm) {
    const int l = threadIdx.x & 15;
    in_pos &= 7;
    if (out_pos < 0 || out_pos > 8) out_pos = 0;
    if (in_pos > 0 || out_pos == 0) {
      if (l < in_pos) x = in;
      x = perm.half(x);
      in = 0u;
      out = l < 8 ? x : 0u;
      in_pos = 0;
      out_pos = 8;
    }
    out_pos -= 1;
    return __shfl_sync(kFullMask, out, out_pos);
  }
};

}  // namespace zc
