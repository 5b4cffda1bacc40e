// cpa_onekey.cuh — re-encryption of many ciphertexts under one key as one
// matrix product on the tcgen05 tensor cores.
//
// With one key, the public polynomials (A, b) are the same for every
// ciphertext and only the secrets differ, so the products are
//   out[ciphertext][(p, n)] = sum_(j, k) s_j[ciphertext][k] M[(j, k)][(p, n)]
// with M the negacyclic Toeplitz matrices of the public polynomials.  The
// per-instance kernel (cpa5i.cuh) spends 12 MMAs of N = 48, its Hankel and
// digit stagings and its phase barriers on each ciphertext (262 us for 65536
// Saber ones); here 264 MMAs of N = 256 serve 128 ciphertexts.
//
//   * A (M side): the CBD secrets of 128 ciphertexts as raw e4m3 bytes (worth
//     s * 2^-9), one row of K bytes a ciphertext, K reversed.
//   * B (N side): the Hankel core matrices of each public polynomial's digit
//     planes (SBO = 128, LBO = 256 as in cpa_umma.cuh), made once per key
//     (k_onekey_prep) in global memory and streamed through shared memory.  A
//     coefficient is written in balanced base 32 (digits -16 .. 15); digit i is
//     the e4m3 number d * 32^i * 2^-9, exact for every i < 3, so all digit
//     planes of a product add up in one accumulator along K and nothing is
//     combined afterwards.
//   * Accumulators: x * 2^-18 for an exact integer |x| <= 4624 * |s| * 256 l
//     < 2^24 (static_assert below), so every partial sum is exact in f32.
//
// The ciphertexts are the rows so that a thread reads its own ciphertext's
// consecutive coefficients: the fields it compares with are at fixed bits of a
// few 64-bit loads.  (With the ciphertexts as columns, 112 of them an MMA, each
// element took two loads, and operand reads of 7.5 KB for 56 cycles of products
// shared the shared-memory port with them: 133 us.)
//
// A CTA takes a run of consecutive (block, output polynomial) units, so that
// the runs of all SMs differ by one polynomial at most and a few blocks still
// reach every SM.  One CTA per SM: one warp issues the MMAs, one copies the planes, 16 warps
// write the next block's secrets while the MMAs of this one run, then round
// and compare each output polynomial's accumulators (two buffers, 512 tensor-
// memory columns).  Every wait is bounded; a thread that gives up reports and
// goes to the end, and no barrier of threads lies in between.
#pragma once
#include <cstdint>

#include "cpa5i.cuh"

namespace tmvp {

constexpr int kOkWorkers = 16;        // warps; after them one that issues the MMAs and one that copies A
constexpr int kOkThreads = 32 * (kOkWorkers + 2);
constexpr int kOkHankel = 62 * 128;   // core matrices of one digit plane
constexpr int kOkRows = 128;          // ciphertexts per block
constexpr int digits32(int w) { return (w + 4) / 5; }

template <int SET>
struct OneKeyC {
  using C = SetC<SET>;
  static constexpr int L = C::L, PA = digits32(C::EQ), PB = digits32(C::EP);
  static constexpr int planes(int p) { return p < L ? PA : PB; }
  static constexpr int PLANES = L * (L * PA + PB);  // digit planes of all products, (p, j, digit) in order
  static constexpr int OPS = PLANES * kOkHankel;
  static constexpr int BR = 16 * kOkRows, BJ = 16 * BR;  // secret bytes of one 16-byte K chunk, and of one j
  // secret buffers, and planes in shared memory, that fit 227 KB
  static constexpr int NBUF = L < 4 ? 2 : 1;
  static constexpr int FIT = (227 * 1024 - 512 - NBUF * L * BJ) / kOkHankel, RING = FIT < 8 ? FIT : 8;
  static constexpr int A = 0, P = NBUF * L * BJ, BAR = P + RING * kOkHankel, TOTAL = BAR + 256;
  static_assert(RING >= 4, "planes on their way while one is read");
  static_assert((4 * 1024 + 16 * 32 + 16) * (C::MU / 2) * 256 * L < (1 << 24), "exact in the f32 accumulators");
};

// e4m3 byte of d * 2^(5 i - 9), |d| <= 16 (exact).
__device__ __forceinline__ uint32_t e4m3_scaled(int d, int i) {
  const uint32_t m = (uint32_t)(d < 0 ? -d : d), sg = d < 0 ? 0x80u : 0u;
  if (m == 0) return 0;
  const int f = 31 - __clz((int)m), e = f + 5 * i - 9;  // the number is 1.x * 2^e
  if (e < -6) return sg | (m << (5 * i));               // subnormal (i = 0, m < 8): units of 2^-9
  return sg | (uint32_t)((e + 7) << 3) | (((m << 3) >> f) & 7u);
}

// Block (p, j, plane): the core matrices of that digit plane.
template <int SET>
__global__ void __launch_bounds__(256) k_onekey_prep(const uint8_t *a_stream, const uint8_t *b_stream, uint8_t *ops) {
  using C = SetC<SET>;
  using K = OneKeyC<SET>;
  constexpr int L = C::L;
  __shared__ uint8_t ext[512];
  int b = blockIdx.x, p, j, d;
  if (b < L * L * K::PA) {
    p = b / (L * K::PA);
    j = b / K::PA % L;
    d = b % K::PA;
  } else {
    b -= L * L * K::PA;
    p = L;
    j = b / K::PB;
    d = b % K::PB;
  }
  const int k = threadIdx.x, W = p < L ? C::EQ : C::EP;
  chain_wait();
  const uint8_t *src = p < L ? a_stream + 32 * (p * L + j) * C::EQ : b_stream + 32 * j * C::EP;
  // the W-bit coefficient k (byte reads inside the polynomial only)
  uint32_t x = 0;
  for (int q = (k * W) >> 3; q <= (k * W + W - 1) >> 3; q++) x |= (uint32_t)src[q] << (8 * (q - ((k * W) >> 3)));
  int v = (int)((x >> ((k * W) & 7)) & ((1u << W) - 1u));
  if (v >= 1 << (W - 1)) v -= 1 << W;
  // balanced base-32 digit d (the last one is what is left; |it| <= 16)
  int dig = 0;
  for (int i = 0; i <= d; i++) {
    dig = i + 1 < digits32(W) ? ((v + 16) & 31) - 16 : v;
    v = (v - dig) / 32;
  }
  const uint32_t e = e4m3_scaled(dig, d);
  ext[255 + k] = (uint8_t)e;                          // a_ext[m] = a[m - 255], m >= 255
  if (k > 0) ext[k - 1] = (uint8_t)(e ^ 0x80u);       // -a[m + 1], m < 255
  __syncthreads();
  uint8_t *out = ops + (size_t)blockIdx.x * kOkHankel;
  for (int i = k; i < kOkHankel / 4; i += 256) {
    const int byte = 4 * i, at = 8 * (byte >> 7) + ((byte >> 4) & 7) + (byte & 15);
    reinterpret_cast<uint32_t *>(out)[i] =
        (uint32_t)ext[at] | (uint32_t)ext[at + 1] << 8 | (uint32_t)ext[at + 2] << 16 | (uint32_t)ext[at + 3] << 24;
  }
}

// Sixteen CBD coefficients from MU / 2 words of the GenSecret stream, as raw
// e4m3 bytes in reversed order (coefficient 15 in the first byte).
template <int MU>
__device__ __forceinline__ void cbd16_reversed(const uint32_t *w, uint32_t (&o)[4]) {
#pragma unroll
  for (int h = 0; h < 4; h++) {
    uint32_t v = 0;
    if constexpr (MU == 8) {
      // popcounts of the nibbles of four bytes; a + 16 - b has bit 4 where a >= b
      uint32_t n = w[h] - ((w[h] >> 1) & 0x55555555u);
      n = (n & 0x33333333u) + ((n >> 2) & 0x33333333u);
      v = __vsub4(n & 0x0f0f0f0fu, (n >> 4) & 0x0f0f0f0fu);
    } else if constexpr (MU == 2) {
      const uint32_t x = (w[0] >> (8 * h)) & 0xffu;
      const uint32_t spread = (x & 3u) | ((x & 0xcu) << 6) | ((x & 0x30u) << 12) | ((x & 0xc0u) << 18);
      v = __vsub4(spread & 0x01010101u, (spread >> 1) & 0x01010101u);
    } else {
#pragma unroll
      for (int b = 0; b < 4; b++) {
        const int bit = (4 * h + b) * MU, i = bit >> 5, sh = bit & 31;
        const uint32_t x = sh + MU <= 32 ? w[i] >> sh : __funnelshift_r(w[i], w[i + 1], sh);
        constexpr uint32_t m = (1u << (MU / 2)) - 1u;
        v |= ((uint32_t)(__popc(x & m) - __popc((x >> (MU / 2)) & m)) & 0xffu) << (8 * b);
      }
    }
    o[3 - h] = __byte_perm(raw_secrets4(v), 0u, 0x0123);
  }
}

struct OneKeyArgs {
  const uint8_t *ops;       // k_onekey_prep
  const uint8_t *s_stream;  // [n][gs_bytes]
  const uint8_t *ct;        // [n][ct_bytes]
  const uint8_t *msg;       // [n][64]: m' in the first 32 bytes
  uint8_t *fail;            // zeroed by the caller; 1 where the re-encryption differs
  int *err;
  int n, units;             // ciphertexts; output polynomials of blocks of kOkRows
};

template <int SET>
__global__ void __launch_bounds__(kOkThreads, 1) k_onekey_reenc(const __grid_constant__ OneKeyArgs a) {
  using C = SetC<SET>;
  using K = OneKeyC<SET>;
  constexpr int L = C::L, BR = K::BR, BJ = K::BJ, NB = K::NBUF, RING = K::RING;
  extern __shared__ __align__(128) uint8_t sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform)
  const uint32_t s0 = smem_u32(sm), bar = s0 + K::BAR;
  // barriers: secrets full, accumulators full / empty (two of each), planes full / empty
  const uint32_t s_full = bar, d_full = bar + 16, d_empty = bar + 32, p_full = bar + 48, p_empty = p_full + 8 * RING;
  uint32_t *slot = reinterpret_cast<uint32_t *>(sm + K::BAR + 48 + 16 * RING);
  if (warp == kOkWorkers) tmem_alloc(smem_u32(slot), 512);
  if (tid == 0) {
    for (int i = 0; i < 2; i++) {
      mbar_init(s_full + 8 * i, 32 * kOkWorkers);
      mbar_init(d_full + 8 * i, 1);
      mbar_init(d_empty + 8 * i, 32 * kOkWorkers);
    }
    for (int i = 0; i < RING; i++) {
      mbar_init(p_full + 8 * i, 1);
      mbar_init(p_empty + 8 * i, 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(slot);
  chain_wait();
  // units [u0, u1) of (block, output polynomial); `it` counts this CTA's blocks
  const int u0 = (int)((long long)a.units * blockIdx.x / gridDim.x),
            u1 = (int)((long long)a.units * (blockIdx.x + 1) / gridDim.x);
  bool ok = true;
  if (warp == kOkWorkers) {
    // the MMAs: the whole warp runs the loop, so that the descriptors stay in
    // uniform registers, and one lane issues
    const bool one = lane == 0;
    constexpr uint32_t idesc = umma_idesc_e4m3(256);
    int rb = 0, it = -1;
    uint32_t rp = 0, dn = 0;  // parity of ring buffer rb; accumulator buffers used so far
    for (int u = u0; ok && u < u1; u++, dn++) {
      const int p = u % (L + 1);
      if (u == u0 || p == 0) {
        it++;
        ok = mbar_spin_bounded(s_full + 8 * (it % NB), (it / NB) & 1);
      }
      const uint32_t d = tmem + 256 * (dn & 1);
      if (ok && dn >= 2) ok = mbar_spin_bounded(d_empty + 8 * (dn & 1), ((dn >> 1) - 1) & 1);
      const int np = L * K::planes(p);
      for (int q = 0; ok && q < np; q++) {
        ok = mbar_spin_bounded(p_full + 8 * rb, rp);
        if (!ok) break;
        tc_fence_after();
        const int j = q / K::planes(p);
        const uint64_t ad = umma_desc(s0 + K::A + (it % NB) * (L * BJ) + j * BJ, BR, 128);
        const uint64_t bd = umma_desc(s0 + K::P + rb * kOkHankel, 256, 128);
#pragma unroll
        for (int t = 0; t < 8; t++)
          umma_f8_if(one, d, ad + (uint64_t)((2 * t * BR) >> 4), bd + (uint64_t)((4 * t * 128) >> 4), idesc,
                     (q | t) != 0);
        if (one) umma_commit(p_empty + 8 * rb);
        if (++rb == RING) {
          rb = 0;
          rp ^= 1;
        }
      }
      if (ok && one) umma_commit(d_full + 8 * (dn & 1));
    }
    if (!ok && one && a.err) atomicOr(a.err, 2);
    // the last MMAs have completed when the workers have read their accumulators
  } else if (warp == kOkWorkers + 1) {
    // the planes of each unit, each into the ring's next buffer once the MMAs
    // that read it are over
    if (lane == 0) {
      int rb = 0, i = 0;
      uint32_t rp = 1;  // (the first round finds every buffer free)
      for (int u = u0; ok && u < u1; u++) {
        const int p = u % (L + 1), np = L * K::planes(p);
        const uint8_t *src = a.ops + (size_t)(p * L * K::PA) * kOkHankel;
        for (int q = 0; ok && q < np; q++, i++, src += kOkHankel) {
          ok = i < RING || mbar_wait_bounded(p_empty + 8 * rb, rp);
          if (!ok) break;
          mbar_expect_tx(p_full + 8 * rb, kOkHankel);
          bulk_g2s(s0 + K::P + rb * kOkHankel, src, kOkHankel, p_full + 8 * rb);
          if (++rb == RING) {
            rb = 0;
            rp ^= 1;
          }
        }
      }
      if (!ok && a.err) atomicOr(a.err, 2);
      // no copy outlives the CTA: the last ones have landed (bounded)
      for (int k = i < RING ? 0 : i - RING; k < i; k++) mbar_wait_bounded(p_full + 8 * (k % RING), (k / RING) & 1);
    }
    __syncwarp();
  } else {
    // Secrets of block blk into buffer b: 8 ciphertexts x 4 chunks of 16
    // coefficients a warp task (64-byte reads a ciphertext, conflict-free stores)
    auto stage = [&](int blk, int b) {
      const int base = blk * kOkRows, nv = min(kOkRows, a.n - base);
      const uint32_t dst = s0 + K::A + b * (L * BJ);
#pragma unroll 4
      for (int u = warp; u < (kOkRows / 8) * L * 4; u += kOkWorkers) {
        const int c = 8 * (u / (4 * L)) + (lane & 7), j = u / 4 % L, g = 4 * (u & 3) + (lane >> 3);
        if (c < nv) {
          uint32_t w[C::MU / 2], o[4];
          const uint8_t *src = a.s_stream + (size_t)(base + c) * C::GS + j * C::COIN + g * (2 * C::MU);
          if constexpr (C::MU == 8) {
            const uint4 v = *reinterpret_cast<const uint4 *>(src);
            w[0] = v.x; w[1] = v.y; w[2] = v.z; w[3] = v.w;
          } else {
#pragma unroll
            for (int i = 0; i < C::MU / 2; i++) w[i] = reinterpret_cast<const uint32_t *>(src)[i];
          }
          cbd16_reversed<C::MU>(w, o);
          sts128(dst + j * BJ + (15 - g) * BR + 16 * c, o[0], o[1], o[2], o[3]);
        }
      }
      fence_async_smem();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(s_full + 8 * b) : "memory");
    };
    // this thread's ciphertext of a block, and its 64 coefficients of a product
    const int q4 = warp & 3, g = warp >> 2, c = 32 * q4 + lane;
    uint32_t dn = 0;
    int it = 0;
    if (u0 < u1) stage(u0 / (L + 1), 0);
    for (int u = u0; ok && u < u1;) {
      const int blk = u / (L + 1), base = blk * kOkRows, ub = min((blk + 1) * (L + 1), u1);  // the block's units end here
      const bool valid = base + c < a.n, more = ub < u1;
      // the next block's secrets: with two buffers, the MMAs that read that one
      // were over when the previous block's last accumulators were complete
      if (NB == 2 && more) stage(blk + 1, (it + 1) & 1);
      // output polynomial p (the last one with the message bits)
      auto poly = [&](auto last_c, int p) {
        constexpr bool LAST = decltype(last_c)::value;
        constexpr int W = LAST ? C::ET : C::EP, TOP = LAST ? C::EP : C::EQ;  // the field: the W bits below bit TOP
        // the 64 fields, W 64-bit words, requested before the accumulators are waited for
        uint32_t w[2 * W + 1], m[2] = {0u, 0u};
        w[2 * W] = 0;
        const uint8_t *src = a.ct + (size_t)(base + c) * C::CT + p * C::POLYCOMP + 8 * W * g;
#pragma unroll
        for (int i = 0; i < W; i++) {
          uint2 v = make_uint2(0u, 0u);
          if (valid) v = __ldg(reinterpret_cast<const uint2 *>(src) + i);
          w[2 * i] = v.x;
          w[2 * i + 1] = v.y;
        }
        if (LAST && valid) {
          const uint2 v = __ldg(reinterpret_cast<const uint2 *>(a.msg + (size_t)(base + c) * 64 + 8 * g));
          m[0] = v.x;
          m[1] = v.y;
        }
        ok = mbar_wait_warp(d_full + 8 * (dn & 1), (dn >> 1) & 1);
        if (!ok) return;
        tc_fence_after();
        // one secret buffer: the block's MMAs are over now
        if (NB == 1 && LAST && more) stage(blk + 1, 0);
        const uint32_t tc = tmem + ((uint32_t)(32 * q4) << 16) + 256 * (dn & 1) + 64 * g;
        uint32_t diff = 0;
#pragma unroll
        for (int k0 = 0; k0 < 64; k0 += 16) {
          uint32_t f[16];
          tmem_ld16(tc + k0, f);
#pragma unroll
          for (int i = 0; i < 16; i++) {
            const int k = k0 + i, bit = W * k, b5 = bit & 31;
            // x + h1 (an integer below 2^24: exact in f32), less the message bit
            uint32_t x = (uint32_t)__float2int_rn(__fmaf_rn(__uint_as_float(f[i]), 262144.0f, (float)C::H1));
            if (LAST) x -= ((m[k >> 5] >> (k & 31)) & 1u) << (C::EP - 1);
            const uint32_t want = b5 + W <= 32 ? w[bit >> 5] >> b5 : __funnelshift_r(w[bit >> 5], w[(bit >> 5) + 1], b5);
            diff |= ((x >> (TOP - W)) ^ want) & ((1u << W) - 1u);
          }
        }
        tc_fence_before();
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(d_empty + 8 * (dn & 1)) : "memory");
        if (valid && diff) a.fail[base + c] = 1;
        dn++;
      };
#pragma unroll 1
      for (; ok && u < ub && u % (L + 1) < L; u++) poly(std::false_type{}, u % (L + 1));
      if (ok && u < ub) {
        poly(std::true_type{}, L);
        u++;
      }
      it++;
    }
    if (!ok && a.err) atomicOr(a.err, 2);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kOkWorkers) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------
// Decryption of many ciphertexts under one key, the same way: the key's secrets
// are the Hankel side, resident in shared memory, and a row is one ciphertext's
// b' in two balanced base-32 digit planes.  Digit 1 meets a copy of the secrets
// scaled by 32, so that both planes add up in one accumulator: x * 2^-18 with
// |x| <= 16 * 33 * 7 * 256 l < 2^24.
//
// What bounds it: the digits (about 6 instructions a coefficient and plane
// pair) of 16 warps, which fill two buffers of one j each ahead of the MMAs
// (48 of N = 256 for 128 Saber ciphertexts) and decode a block's accumulators
// while the next block's first digits are multiplied.  The n ciphertexts are
// spread evenly over whole rounds of one block per SM.  65536 Saber ciphertexts:
// 47 us (five to a CTA of the per-instance kernel, which shares the staged secret
// and the MMAs: 82).

template <int SET>
struct OneKeyD {
  using C = SetC<SET>;
  static constexpr int L = C::L, PLANES = 2 * L;
  static constexpr int BR = 16 * kOkRows, PL = 16 * BR, BJ = 2 * PL;  // digit bytes: a 16-byte K chunk, a plane, a j
  static constexpr int A = 0, B = 2 * BJ, BAR = B + PLANES * kOkHankel, TOTAL = BAR + 128;
  static_assert(TOTAL <= 227 * 1024, "fits an SM");
  static_assert(16 * 33 * 7 * 256 * L < (1 << 24), "exact in the f32 accumulators");
};
constexpr int kOkDecThreads = 32 * (kOkWorkers + 1);

// Block (j, digit): the core matrices of the secret polynomial j times 32^digit.
template <int SET>
__global__ void __launch_bounds__(256) k_onekey_sprep(const uint8_t *sk, uint8_t *planes, int *err) {
  using C = SetC<SET>;
  __shared__ uint8_t ext[512];
  const int k = threadIdx.x, j = blockIdx.x >> 1, d = blockIdx.x & 1;
  constexpr int W = C::SABLE ? 2 : C::EQ;
  chain_wait();
  const uint8_t *src = sk + 32 * j * W;
  uint32_t x = 0;
  for (int q = (k * W) >> 3; q <= (k * W + W - 1) >> 3; q++) x |= (uint32_t)src[q] << (8 * (q - ((k * W) >> 3)));
  int v = (int)((x >> ((k * W) & 7)) & ((1u << W) - 1u));
  if (v >= 1 << (W - 1)) v -= 1 << W;
  if (v < -7 || v > 7) {  // (as the per-instance kernel: reported, the result is not used)
    if (err) atomicOr(err, 1);
    v = 0;
  }
  const uint32_t e = e4m3_scaled(v, d);
  ext[255 + k] = (uint8_t)e;
  if (k > 0) ext[k - 1] = (uint8_t)(e ^ 0x80u);
  __syncthreads();
  uint8_t *out = planes + (size_t)blockIdx.x * kOkHankel;
  for (int i = k; i < kOkHankel / 4; i += 256) {
    const int byte = 4 * i, at = 8 * (byte >> 7) + ((byte >> 4) & 7) + (byte & 15);
    reinterpret_cast<uint32_t *>(out)[i] =
        (uint32_t)ext[at] | (uint32_t)ext[at + 1] << 8 | (uint32_t)ext[at + 2] << 16 | (uint32_t)ext[at + 3] << 24;
  }
}

struct OneKeyDecArgs {
  const uint8_t *planes;  // k_onekey_sprep
  const uint8_t *ct;      // [n][ct_bytes]
  const uint8_t *sk;      // the key: H(pk) is copied from it
  uint8_t *m_out;         // [n][64]: m' | H(pk)
  int *err;
  int n, rows, blocks;    // ciphertexts; of a block (<= kOkRows); blocks
};

template <int SET>
__global__ void __launch_bounds__(kOkDecThreads, 1) k_onekey_decrypt(const __grid_constant__ OneKeyDecArgs a) {
  using C = SetC<SET>;
  using K = OneKeyD<SET>;
  constexpr int L = C::L, BR = K::BR, W = C::EP;
  extern __shared__ __align__(128) uint8_t sm[];
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform)
  const uint32_t s0 = smem_u32(sm), bar = s0 + K::BAR;
  // barriers: digits full / empty, accumulators full / empty (two of each), planes
  const uint32_t a_full = bar, a_empty = bar + 16, d_full = bar + 32, d_empty = bar + 48, b_full = bar + 64;
  uint32_t *slot = reinterpret_cast<uint32_t *>(sm + K::BAR + 72);
  if (warp == kOkWorkers) tmem_alloc(smem_u32(slot), 512);
  if (tid == 0) {
    for (int i = 0; i < 2; i++) {
      mbar_init(a_full + 8 * i, 32 * kOkWorkers);
      mbar_init(a_empty + 8 * i, 1);
      mbar_init(d_full + 8 * i, 1);
      mbar_init(d_empty + 8 * i, 32 * kOkWorkers);
    }
    mbar_init(b_full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(slot);
  chain_wait();
  bool ok = true;
  if (warp == kOkWorkers) {
    // the planes, once, then the MMAs (the whole warp runs the loop, one lane issues)
    const bool one = lane == 0;
    if (one) {
      mbar_expect_tx(b_full, K::PLANES * kOkHankel);
      for (int q = 0; q < K::PLANES; q++)
        bulk_g2s(s0 + K::B + q * kOkHankel, a.planes + (size_t)q * kOkHankel, kOkHankel, b_full);
    }
    __syncwarp();
    ok = mbar_wait_bounded(b_full, 0);
    if (!ok) mbar_wait_bounded(b_full, 0);  // (no copy outlives the CTA)
    constexpr uint32_t idesc = umma_idesc_e4m3(256);
    uint32_t item = 0, dn = 0;  // digit buffers and accumulators used so far
    for (int blk = blockIdx.x; ok && blk < a.blocks; blk += gridDim.x, dn++) {
      const uint32_t d = tmem + 256 * (dn & 1);
      if (dn >= 2) ok = mbar_spin_bounded(d_empty + 8 * (dn & 1), ((dn >> 1) - 1) & 1);
      for (int j = 0; ok && j < L; j++, item++) {
        const uint32_t ab = item & 1;
        ok = mbar_spin_bounded(a_full + 8 * ab, (item >> 1) & 1);
        if (!ok) break;
        tc_fence_after();
#pragma unroll
        for (int p = 0; p < 2; p++) {
          const uint64_t ad = umma_desc(s0 + K::A + ab * K::BJ + p * K::PL, BR, 128);
          const uint64_t bd = umma_desc(s0 + K::B + (2 * j + p) * kOkHankel, 256, 128);
#pragma unroll
          for (int t = 0; t < 8; t++)
            umma_f8_if(one, d, ad + (uint64_t)((2 * t * BR) >> 4), bd + (uint64_t)((4 * t * 128) >> 4), idesc,
                       (j | p | t) != 0);
        }
        if (one) umma_commit(a_empty + 8 * ab);
      }
      if (ok && one) umma_commit(d_full + 8 * (dn & 1));
    }
    if (!ok && one && a.err) atomicOr(a.err, 2);
    // the last MMAs have completed when the workers have read their accumulators
  } else {
    uint32_t item = 0;
    // Digits of b'_j of a block's ciphertexts into the next buffer: 8 ciphertexts
    // x 4 chunks of 16 coefficients a warp task
    auto stage = [&](int blk, int j) {
      const uint32_t ab = item & 1;
      ok = item < 2 || mbar_wait_warp(a_empty + 8 * ab, ((item >> 1) - 1) & 1);
      item++;
      if (!ok) return;
      const int base = blk * a.rows, nv = min(a.rows, a.n - base);
      const uint32_t dst = s0 + K::A + ab * K::BJ;
#pragma unroll 4
      for (int u = warp; u < (kOkRows / 8) * 4; u += kOkWorkers) {
        const int c = 8 * (u >> 2) + (lane & 7), g = 4 * (u & 3) + (lane >> 3);
        if (c < nv) {
          const int off = 2 * W * g;
          const uint8_t *src = a.ct + (size_t)(base + c) * C::CT + j * C::POLYCOMP + (off & ~3);
          uint32_t w[5];
#pragma unroll
          for (int i = 0; i < 5; i++) w[i] = __ldg(reinterpret_cast<const uint32_t *>(src) + i);
          if (W & 1) {  // 18 bytes a chunk
#pragma unroll
            for (int i = 0; i < 5; i++) w[i] = __funnelshift_r(w[i], i < 4 ? w[i + 1] : 0u, 8 * (off & 2));
          }
          uint32_t lo[4], hi[4];
#pragma unroll
          for (int h = 0; h < 4; h++) {  // coefficients 4h .. 4h + 3, the last first
            constexpr uint32_t m = ((1u << W) - 1u) * 0x10001u;
            const uint32_t x0 = field_pair<W>(w, 5, 4 * W * h) & m, x1 = field_pair<W>(w, 5, 4 * W * h + 2 * W) & m;
            lo[3 - h] = raw_sdigits4(__byte_perm(x0, x1, 0x0246));
            hi[3 - h] = raw_sdigits4(__byte_perm((x0 + 0x00100010u) >> 5, (x1 + 0x00100010u) >> 5, 0x0246));
          }
          const uint32_t at = dst + (15 - g) * BR + 16 * c;
          sts128(at, lo[0], lo[1], lo[2], lo[3]);
          sts128(at + K::PL, hi[0], hi[1], hi[2], hi[3]);
        }
      }
      fence_async_smem();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a_full + 8 * ab) : "memory");
    };
    // this thread's ciphertext of a block, and its 64 coefficients
    const int q4 = warp & 3, g = warp >> 2, c = 32 * q4 + lane;
    const uint2 hpk = __ldg(reinterpret_cast<const uint2 *>(a.sk + C::SK - 64) + g);
    uint32_t dn = 0;
    auto decode = [&](int blk) {
      const int base = blk * a.rows;
      const bool valid = c < min(a.rows, a.n - base);
      uint32_t w[2 * C::ET + 1];
      w[2 * C::ET] = 0;
      const uint8_t *src = a.ct + (size_t)(base + c) * C::CT + L * C::POLYCOMP + 8 * C::ET * g;
#pragma unroll
      for (int i = 0; i < C::ET; i++) {
        uint2 v = make_uint2(0u, 0u);
        if (valid) v = __ldg(reinterpret_cast<const uint2 *>(src) + i);
        w[2 * i] = v.x;
        w[2 * i + 1] = v.y;
      }
      ok = mbar_wait_warp(d_full + 8 * (dn & 1), (dn >> 1) & 1);
      if (!ok) return;
      tc_fence_after();
      const uint32_t tc = tmem + ((uint32_t)(32 * q4) << 16) + 256 * (dn & 1) + 64 * g;
      uint32_t mw[2] = {0u, 0u};
#pragma unroll
      for (int k0 = 0; k0 < 64; k0 += 16) {
        uint32_t f[16];
        tmem_ld16(tc + k0, f);
#pragma unroll
        for (int i = 0; i < 16; i++) {
          const int k = k0 + i, bit = C::ET * k, b5 = bit & 31;
          // m'_k = ((x + h2 - (c_m,k << (ep - et))) mod p) >> (ep - 1)
          const int x = __float2int_rn(__fmaf_rn(__uint_as_float(f[i]), 262144.0f, (float)C::H2));
          const uint32_t cm =
              b5 + C::ET <= 32 ? w[bit >> 5] >> b5 : __funnelshift_r(w[bit >> 5], w[(bit >> 5) + 1], b5);
          const uint32_t v = (uint32_t)x - ((cm & ((1u << C::ET) - 1u)) << (C::EP - C::ET));
          mw[k >> 5] |= ((v >> (C::EP - 1)) & 1u) << (k & 31);
        }
      }
      tc_fence_before();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(d_empty + 8 * (dn & 1)) : "memory");
      dn++;
      if (valid) {
        uint2 *mo = reinterpret_cast<uint2 *>(a.m_out + (size_t)(base + c) * 64);
        mo[g] = make_uint2(mw[0], mw[1]);
        mo[4 + g] = hpk;
      }
    };
    // a block is decoded once two more buffers of digits are on their way
    int last = -1;
    for (int blk = blockIdx.x; ok && blk < a.blocks; blk += gridDim.x) {
#pragma unroll 1
      for (int j = 0; ok && j < L; j++) {
        stage(blk, j);
        if (ok && j == 1 && last >= 0) decode(last);
      }
      last = blk;
    }
    if (ok && last >= 0) decode(last);
    if (!ok && a.err) atomicOr(a.err, 2);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kOkWorkers) tmem_dealloc(tmem, 512);
}

}  // namespace tmvp
