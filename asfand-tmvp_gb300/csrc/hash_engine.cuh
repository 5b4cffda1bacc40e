// hash_engine.cuh — the three forms of a sponge behind one interface: one
// thread (keccak.cuh), two threads (keccak_pair.cuh) or one warp
// (keccak_warp.cuh) per sponge.  The Keccak stages (hash_kernels.cu) are
// written once against it.
//
// A Msg is a message of up to eight 64-bit words in the form's own layout:
// all words in one thread, their 32-bit halves in two, or word k in lane k.
// Every thread of a warp calls an engine's functions together (the pair and
// warp forms exchange by shuffles); `live` is false in threads that only
// repeat another sponge's work, and they store nothing.  The 16 sponges of a
// pair-form warp may have different lengths (a mixed pass's groups): all its
// threads permute as often as the longest of them needs.
#pragma once
#include <cstddef>
#include <cstdint>

#include "keccak.cuh"
#include "keccak_pair.cuh"
#include "keccak_warp.cuh"

namespace tmvp {

struct ThreadSponge {
  struct Msg {
    uint64_t w[8];
  };
  __device__ __forceinline__ Msg load(const uint8_t *p, int nw) const {
    Msg m;
    const uint64_t *s = reinterpret_cast<const uint64_t *>(p);
#pragma unroll
    for (int i = 0; i < 8; i++) m.w[i] = i < nw ? s[i] : 0ull;
    return m;
  }
  __device__ __forceinline__ void store(uint8_t *p, const Msg &m, int nw) const {
    uint64_t *d = reinterpret_cast<uint64_t *>(p);
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (i < nw) d[i] = m.w[i];
  }
  // words 0..3 of a, then words 0..3 of b
  __device__ __forceinline__ Msg cat4(const Msg &a, const Msg &b) const {
    Msg m;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      m.w[i] = a.w[i];
      m.w[4 + i] = b.w[i];
    }
    return m;
  }
  // words 4..7 as 0..3
  __device__ __forceinline__ Msg hi4(const Msg &a) const { return cat4(Msg{{a.w[4], a.w[5], a.w[6], a.w[7]}}, a); }
  // b's words 0..3 where pick, else a's, by mask (no branch on pick)
  __device__ __forceinline__ Msg sel4(const Msg &a, const Msg &b, bool pick) const {
    Msg m = a;
    const uint64_t mask = 0ull - (uint64_t)pick;
#pragma unroll
    for (int i = 0; i < 4; i++) m.w[i] ^= mask & (a.w[i] ^ b.w[i]);
    return m;
  }
  __device__ __forceinline__ Msg sha3_256_mem(const uint8_t *p, int nbytes) const {
    Msg m;
    uint64_t h[4];
    sha3_256_words(h, reinterpret_cast<const uint64_t *>(p), nbytes);
#pragma unroll
    for (int i = 0; i < 8; i++) m.w[i] = i < 4 ? h[i] : 0ull;
    return m;
  }
  template <int NW>  // 4 or 8 words
  __device__ __forceinline__ Msg sha3_256(const Msg &a) const {
    Msg m;
    uint64_t h[4];
    if constexpr (NW == 4) {
      const uint64_t in[4] = {a.w[0], a.w[1], a.w[2], a.w[3]};
      sha3_256_32(h, in);
    } else {
      sha3_256_64(h, a.w);
    }
#pragma unroll
    for (int i = 0; i < 8; i++) m.w[i] = i < 4 ? h[i] : 0ull;
    return m;
  }
  __device__ __forceinline__ Msg sha3_512_64(const Msg &a) const {
    Msg m;
    tmvp::sha3_512_64(m.w, a.w);
    return m;
  }
  // SHAKE-128 of the 32-byte message a, nbytes (a multiple of 8) to out
  __device__ __forceinline__ void shake128(const Msg &a, uint8_t *out, int nbytes) const {
    const uint64_t seed[4] = {a.w[0], a.w[1], a.w[2], a.w[3]};
    shake128_32(reinterpret_cast<uint64_t *>(out), nbytes, seed);
  }
  // its first 32 bytes
  __device__ __forceinline__ Msg shake128_first(const Msg &a) const {
    Msg m;
    uint64_t h[4];
    const uint64_t seed[4] = {a.w[0], a.w[1], a.w[2], a.w[3]};
    shake128_32(h, 32, seed);
#pragma unroll
    for (int i = 0; i < 8; i++) m.w[i] = i < 4 ? h[i] : 0ull;
    return m;
  }
};

// Thread `me` of a pair holds the low (0) or high (1) halves.
struct PairSponge {
  int me;
  bool live;
  struct Msg {
    uint32_t w[8];
  };
  __device__ __forceinline__ Msg load(const uint8_t *p, int nw) const {
    Msg m;
    const uint32_t *s = reinterpret_cast<const uint32_t *>(p) + me;
#pragma unroll
    for (int i = 0; i < 8; i++) m.w[i] = i < nw ? s[2 * i] : 0u;
    return m;
  }
  __device__ __forceinline__ void store(uint8_t *p, const Msg &m, int nw) const {
    if (!live) return;
    uint32_t *d = reinterpret_cast<uint32_t *>(p) + me;
#pragma unroll
    for (int i = 0; i < 8; i++)
      if (i < nw) d[2 * i] = m.w[i];
  }
  __device__ __forceinline__ Msg cat4(const Msg &a, const Msg &b) const {
    Msg m;
#pragma unroll
    for (int i = 0; i < 4; i++) {
      m.w[i] = a.w[i];
      m.w[4 + i] = b.w[i];
    }
    return m;
  }
  __device__ __forceinline__ Msg hi4(const Msg &a) const { return cat4(Msg{{a.w[4], a.w[5], a.w[6], a.w[7]}}, a); }
  __device__ __forceinline__ Msg sel4(const Msg &a, const Msg &b, bool pick) const {
    Msg m = a;
    const uint32_t mask = 0u - (uint32_t)pick;
#pragma unroll
    for (int i = 0; i < 4; i++) m.w[i] ^= mask & (a.w[i] ^ b.w[i]);
    return m;
  }
  __device__ __forceinline__ Msg sha3_256_mem(const uint8_t *p, int nbytes) const {
    Msg m;
    uint32_t h[4];
    pair_sha3_256_mem(me, p, nbytes, h);
#pragma unroll
    for (int i = 0; i < 8; i++) m.w[i] = i < 4 ? h[i] : 0u;
    return m;
  }
  template <int NW>
  __device__ __forceinline__ Msg sha3_256(const Msg &a) const {
    Msg m;
    pair_sha3_lanes<17>(me, a.w, NW, m.w, 4);
#pragma unroll
    for (int i = 4; i < 8; i++) m.w[i] = 0u;
    return m;
  }
  __device__ __forceinline__ Msg sha3_512_64(const Msg &a) const {
    Msg m;
    pair_sha3_lanes<9>(me, a.w, 8, m.w, 8);
    return m;
  }
  __device__ __forceinline__ void absorb_seed(uint32_t (&w)[25], const Msg &a) const {
    pair_zero(w);
#pragma unroll
    for (int k = 0; k < 4; k++) w[k] = a.w[k];
    w[4] ^= pair_half(0x1Full, me);
    w[20] ^= pair_half(0x8000000000000000ull, me);
  }
  __device__ __forceinline__ void shake128(const Msg &a, uint8_t *out, int nbytes) const {
    uint32_t w[25];
    absorb_seed(w, a);
    uint32_t *o32 = reinterpret_cast<uint32_t *>(out) + me;
    const int nw = nbytes >> 3;
    const int most = __reduce_max_sync(0xFFFFFFFFu, nw);  // (a warp may hold sponges of several parameter sets)
    for (int at = 0; at < most; at += 21) {
      pair_keccak_f1600(w, me);
      if (live) {
#pragma unroll
        for (int q = 0; q < 21; q++)
          if (q < nw - at) o32[2 * q] = w[q];
      }
      o32 += 2 * 21;
    }
  }
  __device__ __forceinline__ Msg shake128_first(const Msg &a) const {
    uint32_t w[25];
    absorb_seed(w, a);
    pair_keccak_f1600(w, me);
    Msg m;
#pragma unroll
    for (int i = 0; i < 8; i++) m.w[i] = i < 4 ? w[i] : 0u;
    return m;
  }
};

// Lane k < 25 holds state lane k.
struct WarpSponge {
  int lane;
  bool live;
  WarpKeccakLane L;
  typedef uint64_t Msg;  // word k in lane k
  // lane k takes the word of lane (k + from) mod 32
  __device__ __forceinline__ Msg down(Msg v, int from) const {
    const uint32_t lo = __shfl_sync(0xFFFFFFFFu, (uint32_t)v, (lane + from) & 31);
    const uint32_t hi = __shfl_sync(0xFFFFFFFFu, (uint32_t)(v >> 32), (lane + from) & 31);
    return ((uint64_t)hi << 32) | lo;
  }
  __device__ __forceinline__ Msg load(const uint8_t *p, int nw) const {
    return lane < nw ? reinterpret_cast<const uint64_t *>(p)[lane] : 0ull;
  }
  __device__ __forceinline__ void store(uint8_t *p, Msg m, int nw) const {
    if (live && lane < nw) reinterpret_cast<uint64_t *>(p)[lane] = m;
  }
  __device__ __forceinline__ Msg cat4(Msg a, Msg b) const {
    const Msg up = down(b, 28);  // lane k takes lane k - 4
    return lane < 4 ? a : up;
  }
  __device__ __forceinline__ Msg hi4(Msg a) const { return down(a, 4); }
  __device__ __forceinline__ Msg sel4(Msg a, Msg b, bool pick) const {
    return a ^ ((0ull - (uint64_t)pick) & (a ^ b));
  }
  __device__ __forceinline__ Msg sha3_256_mem(const uint8_t *p, int nbytes) const {
    uint32_t lo, hi;
    warp_hash_words<17>(lo, hi, L, lane, reinterpret_cast<const uint64_t *>(p), nbytes, 0x06);
    return warp_lane_word(lo, hi);
  }
  template <int NW>
  __device__ __forceinline__ Msg sha3_256(Msg a) const {
    uint32_t lo, hi;
    warp_absorb_lanes<17>(lo, hi, lane, a, NW, 0x06);
    warp_keccak_f1600<8>(lo, hi, L);
    return warp_lane_word(lo, hi);
  }
  __device__ __forceinline__ Msg sha3_512_64(Msg a) const {
    uint32_t lo, hi;
    warp_absorb_lanes<9>(lo, hi, lane, a, 8, 0x06);
    warp_keccak_f1600<8>(lo, hi, L);
    return warp_lane_word(lo, hi);
  }
  __device__ __forceinline__ void shake128(Msg a, uint8_t *out, int nbytes) const {
    uint32_t lo, hi;
    warp_absorb_lanes<21>(lo, hi, lane, a, 4, 0x1F);
    uint64_t *o = reinterpret_cast<uint64_t *>(out);
    int nw = nbytes >> 3;
    while (nw > 0) {
      warp_keccak_f1600<24>(lo, hi, L);
      const int k = nw < 21 ? nw : 21;
      if (live && lane < k) o[lane] = warp_lane_word(lo, hi);
      o += 21;
      nw -= k;
    }
  }
  __device__ __forceinline__ Msg shake128_first(Msg a) const {
    uint32_t lo, hi;
    warp_absorb_lanes<21>(lo, hi, lane, a, 4, 0x1F);
    warp_keccak_f1600<8>(lo, hi, L);
    return warp_lane_word(lo, hi);
  }
};

}  // namespace tmvp
