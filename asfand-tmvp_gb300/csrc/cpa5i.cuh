// cpa5i.cuh — the tcgen05 IND-CPA kernel specialised per parameter set: one
// CTA of 256 threads per instance (a resident CTA takes further ones), with
// every width, count and offset a compile-time constant.
//
// Per instance:
//   1. the packed inputs arrive by TMA bulk copies (cp.async.bulk) issued by
//      one thread, counted on an mbarrier;
//   2. radix-16 digit columns (r16_digits, raw e4m3 bytes worth digit * 2^-9)
//      with K reversed, and the secrets (CBD or unpacked) in registers, from
//      there the Hankel core matrices (cpa_umma.cuh);
//   3. one thread issues the 4 l tcgen05.mma (M = 128, N = 16 .. 64, K = 32;
//      each even tile of the Hankel sequence serves four K steps through the
//      negacyclic wrap) into tensor memory and commits them to an mbarrier;
//   4. accumulators -> registers (tcgen05.ld: every digit column of one
//      coefficient per thread), the odd K steps' sums through shared memory to
//      the warp of their coefficients -> the compare / decode / output epilogue
//      (encryption and key generation: rounded 16-bit values, then packed
//      eight coefficients at a time).
// Same results as the runtime-shaped kernels (cpa_tc_kernel.cuh,
// cpa_persist.cuh); the arithmetic per instance is the same.
#pragma once
#include <cstdint>
#include <type_traits>

#include "chain.cuh"
#include "cpa_persist.cuh"
#include "hash_engine.cuh"

namespace tmvp {

// l, log2 q, log2 p, log2 T, mu, Sable (same table as make_params)
constexpr int kSetTab[6][6] = {{2, 13, 10, 3, 10, 0}, {3, 13, 10, 4, 8, 0}, {4, 13, 10, 6, 6, 0},
                               {2, 11, 9, 3, 2, 1},   {3, 11, 9, 5, 2, 1},  {4, 11, 10, 3, 2, 1}};

template <int SET>
struct SetC {
  static constexpr int L = kSetTab[SET][0], EQ = kSetTab[SET][1], EP = kSetTab[SET][2], ET = kSetTab[SET][3];
  static constexpr int MU = kSetTab[SET][4], SABLE = kSetTab[SET][5];
  static constexpr int POLYBYTES = EQ * 32, POLYCOMP = EP * 32, SCALE = ET * 32, COIN = MU * 32;
  static constexpr int PK = L * POLYCOMP + 32, INDCPA_SK = SABLE ? L * 64 : L * POLYBYTES;
  static constexpr int SK = INDCPA_SK + PK + 64, CT = L * POLYCOMP + SCALE;
  static constexpr int GM = L * L * POLYBYTES, GS = L * COIN;
  static constexpr int H1 = 1 << (EQ - EP - 1);
  static constexpr int H2 = (1 << (EP - 2)) - (1 << (EP - ET - 1)) + (1 << (EQ - EP - 1));
};

template <int OP, int SET>
struct ShapeC {
  using C = SetC<SET>;
  static constexpr int L = C::L;
  // kDecryptK: R ciphertexts per CTA, as many as fill 16 digit columns
  static constexpr int R = OP == kDecrypt    ? 1
                           : OP == kDecryptK ? 16 / r16_digits(C::EP)
                                             : (OP == kKeygen || OP == kMatvec ? L : L + 1);
  static constexpr int RA = (OP == kDecrypt || OP == kDecryptK) ? 0 : L;
  static constexpr int WA = C::EQ, WB = C::EP;
  static constexpr int DA = r16_digits(WA), DB = r16_digits(WB);
  static constexpr int NCOLS = RA * DA + (R - RA) * DB;
  static_assert(NCOLS <= 16, "at most two 8-column groups per K step");
  static constexpr int NC4 = (NCOLS + 3) & ~3;     // column slots of one K step
  static constexpr int PG = NC4 / 4;               // 8-column groups of two K steps
  static constexpr int NU = 4 * NC4;               // N of every MMA (four K steps' columns)
  static_assert(NU % 16 == 0, "an N that M = 128 admits");
  static constexpr int TMEM_COLS = NU <= 32 ? 32 : 64;
  // Largest |secret| (CBD: mu / 2; sk and matvec secrets: what small4 admits)
  // and the K rows that one accumulator sums, for combine()
  static constexpr int SMAX = (OP == kMatvec || OP == kDecrypt || OP == kDecryptK) ? 7 : C::MU / 2;
  static constexpr int ROWS = 128 * L;
  static constexpr int col_base(int p) { return p < RA ? p * DA : RA * DA + (p - RA) * DB; }
  static constexpr int digits(int p) { return p < RA ? DA : DB; }
};

constexpr int al16c(int x) { return (x + 15) & ~15; }

// Threads per CTA (one instance): eight warps shorten every staging phase of
// an instance; tensor memory is read by warps w and w + 4 (two M halves).
constexpr int kI5Threads = 256;

// Where a layout puts the packed GenMatrix and b streams, the sums that warps
// exchange and the packed outputs: outside the Hankel core matrices (kFree: the
// core matrices are written as soon as the secrets are read, and the next
// instance's copies start beside the MMAs), or over them (kLate: they wait until
// the streams are read).  kFree is the faster one at the same number of CTAs
// per SM (LightSaber 65536, us: re-encryption 238 -> 227, key generation 258 ->
// 238), but not at one less (Saber 276 -> 281, FireSaber 390 -> 436).
enum InputPlace { kFree, kLate };

// Shared-memory layout of one CTA (byte offsets): the Hankel core matrices H
// (l x HJ), the digit columns BM, the packed secrets (GenSecret stream, secret
// key or matvec secrets), streams and epilogue buffers (InputPlace), ciphertext
// and message.
//
// Digit columns of one j: K step t is 32 K rows (K reversed), two 16-byte K
// chunks, in blocks of two steps: column 2n + (t & 1) of a block, PG groups of
// 8 columns (SB bytes a group, the chunks LB apart), in two sequences,
// [4 5][0 1][-4 -5] and [6 7][2 3][-6 -7] (-t: the digits of step t negated),
// so that one descriptor at the start of a sequence reads steps (4, 5 | 0, 1)
// and one a block later (0, 1 | -4, -5).
// The strides put the 16-byte pieces that a store instruction writes at once
// into different banks.
template <int OP, int SET, InputPlace IP>
struct LayoutAt {
  using C = SetC<SET>;
  using S = ShapeC<OP, SET>;
  static constexpr bool HAS_AS = OP == kEncrypt || OP == kReenc || OP == kKeygen;
  static constexpr bool HAS_B = OP == kEncrypt || OP == kReenc;
  static constexpr bool HAS_CT = OP == kReenc || OP == kDecrypt || OP == kDecryptK;
  static constexpr bool HAS_SK = OP == kDecrypt || OP == kDecryptK;
  // ciphertexts per CTA and their stride in shared memory (16 bytes of
  // slack after each for the field readers)
  static constexpr int NCT = OP == kDecryptK ? S::R : 1;
  static constexpr int CTS = al16c(C::CT + 16);
  // matvec: A as 16-bit coefficients (l x l x 512 bytes) inside H, int8 secrets after it
  static constexpr bool HAS_MV = OP == kMatvec;
  static constexpr int MV_A = C::L * C::L * 512, MV_S = C::L * 256;
  // Hankel core matrices per secret polynomial: tiles start at block w of 32
  // rows (core 4w, w <= 6) and reach 15 row groups and two K chunks on
  static constexpr int CORES = 42;
  static constexpr int CS = 144, HJ = CORES * CS;  // (a core is 128 bytes; the stride spreads equal rows of 8 cores over the banks)
  static constexpr int LB = !HAS_AS || S::NC4 != 16 ? 160 : 128;
  static constexpr int SB = S::NC4 != 16 ? 288 : (HAS_AS ? 272 : 304);
  static constexpr int QB = 16 * (S::NC4 == 16 ? (HAS_AS ? 206 : 234) : (S::NC4 == 12 ? 164 : (S::NC4 == 8 ? 114 : 60)));  // one sequence, padded
  static_assert(QB >= 3 * S::PG * SB, "a sequence's three blocks");
  static constexpr int BJ = 2 * QB;  // digit columns of one j
  // byte offset of step t's columns within one j, and of their negated copy (t >= 4)
  __device__ static __forceinline__ uint32_t step_off(int t) {
    return (uint32_t)(((t >> 1) & 1) * QB + (t >= 4 ? 0 : S::PG * SB) + (t & 1) * 16);
  }
  __device__ static __forceinline__ uint32_t neg_off(int t) {
    return (uint32_t)(((t >> 1) & 1) * QB + 2 * S::PG * SB + (t & 1) * 16);
  }
  // byte offset of digit column n from there
  __host__ __device__ static constexpr int col_off(int n) { return (n >> 2) * SB + (n & 3) * 32; }
  // accumulator sums that another warp finishes: two 16-bit values a word, the last odd one by itself
  static constexpr int XWORDS = S::R / 2, XBYTES = al16c(S::R * 512);
  static constexpr int H = 0;
  static constexpr int BM = H + C::L * HJ;
  static constexpr int SS = BM + C::L * BJ, SKO = SS;  // packed secrets
  static constexpr int SS_BYTES = HAS_AS ? C::GS : (HAS_SK ? C::INDCPA_SK : MV_S);
  static constexpr InputPlace PLACE = IP;
  static constexpr int OUT_BYTES = OP == kEncrypt ? C::CT + 16
                                   : (OP == kKeygen ? C::L * C::POLYCOMP + C::INDCPA_SK + 16 : 0);
  static constexpr int A_BYTES = al16c(HAS_AS ? C::GM + 16 : (HAS_MV ? MV_A : 0));
  static constexpr int STREAMS = al16c(A_BYTES + (HAS_B ? C::L * C::POLYCOMP + 16 : 0));
  static constexpr int FREE0 = al16c(SS + SS_BYTES + 16);  // past the secrets
  static constexpr int A = IP == kFree ? FREE0 : H;
  static constexpr int B = A + A_BYTES;
  static constexpr int XCH = A + STREAMS, OUT = XCH + XBYTES;
  static_assert(IP != kLate || OUT + OUT_BYTES <= BM, "streams and epilogue buffers fit H");
  // the output ops' 16-bit values (R x 8 runs of 80 bytes), over the digit
  // columns (the next instance's inputs are landing in H)
  static constexpr int VALS = BM;
  static_assert(HAS_CT || HAS_MV || S::R * 640 <= C::L * BJ, "epilogue values fit the digit columns");
  // ciphertext and message, read until the end of an instance: two buffers of
  // CTB bytes, so that the next instance's copies land beside them
  static constexpr int CTO = IP == kLate ? FREE0 : al16c(OUT + OUT_BYTES);
  static constexpr int MSG = HAS_CT ? al16c(CTO + NCT * CTS) : CTO;
  static constexpr int CTB = (HAS_B ? al16c(MSG + 32 + 16) : MSG) - CTO;
  static constexpr int SEC8 = CTO + 2 * CTB;
  // mbarriers in, mma, clc; TMEM base; the next instance; two CLC responses
  static constexpr int BAR = al16c(SEC8 + (OP == kKeygen ? C::L * 256 : 0));
  static constexpr int TOTAL = BAR + 64;
  static constexpr int CTAS = (228 * 1024) / (TOTAL + 1024);  // that shared memory admits
  static constexpr int IN_BYTES = (HAS_AS ? C::GM + C::GS : 0) + (HAS_B ? C::L * C::POLYCOMP + 32 : 0) +
                                  (HAS_CT ? C::CT : 0) + (HAS_SK ? C::INDCPA_SK : 0) + (HAS_MV ? MV_A + MV_S : 0);
};

// CTAs per SM that the registers admit without spilling more than a few words:
// 8 of 32 registers (decryption), 6 of 40, and 5 of 48 where a thread loads 32
// accumulator columns.
template <int OP, int SET>
constexpr int reg_ctas() {
  return ShapeC<OP, SET>::NC4 == 16 ? 5 : (OP == kDecrypt ? 8 : 6);
}

// The layout of an operation: the first place that costs no resident CTA.
template <int OP, int SET>
constexpr InputPlace input_place() {
  if (OP == kDecrypt || OP == kDecryptK) return kFree;  // (no streams)
  constexpr int free = LayoutAt<OP, SET, kFree>::CTAS, late = LayoutAt<OP, SET, kLate>::CTAS,
                cap = reg_ctas<OP, SET>();
  return free >= (late < cap ? late : cap) ? kFree : kLate;
}
template <int OP, int SET>
using LayoutC = LayoutAt<OP, SET, input_place<OP, SET>()>;

// Eight W-bit little-endian fields from byte `byte0` (16 bytes of slack after
// the stream), as four words of two 16-bit lanes, two at a time and without
// clearing the bits above them in each lane (whoever uses them masks).
template <int W>
__device__ __forceinline__ uint32_t field_pair(const uint32_t *w, int nw, int bit) {
  const int i = bit >> 5, sh = bit & 31;
  const uint32_t y = (sh + 2 * W <= 32 || i + 1 >= nw) ? (w[i] >> sh) : __funnelshift_r(w[i], w[i + 1], sh);
  return __byte_perm(y, y << (16 - W), 0x7610);
}
template <int W>
__device__ __forceinline__ void unpack8d(const uint8_t *base, int byte0, uint32_t (&X)[4]) {
  const uint32_t wp = smem_u32(base) + (uint32_t)(byte0 & ~3);
  const int sh = 8 * (byte0 & 3);
  uint32_t q[5];
#pragma unroll
  for (int i = 0; i < 5; i++) q[i] = lds32(wp + 4 * i);
  uint32_t a[4];
#pragma unroll
  for (int i = 0; i < 4; i++) a[i] = __funnelshift_r(q[i], q[i + 1], sh);
#pragma unroll
  for (int k = 0; k < 4; k++) X[k] = field_pair<W>(a, 4, 2 * W * k);
}

// Signed 5-bit top digits t (the low five bits of each byte) as raw e4m3
// bytes: t for t < 16, else 0x80 | (32 - t), the number t - 32 (magnitudes up
// to 16): 32 - t = 15 - (t & 15) + 1.
__device__ __forceinline__ uint32_t raw_sdigits4(uint32_t t) {
  const uint32_t s = (t >> 4) & 0x01010101u;
  return ((t & 0x0F0F0F0Fu) ^ (s * 15u)) + s * 0x81u;
}

// Four secrets -7 .. 7 (int8) as raw e4m3 bytes, sign and magnitude: worth
// s * 2^-9 as the digits are, so that the accumulators hold x * 2^-18.
__device__ __forceinline__ uint32_t raw_secrets4(uint32_t v) {
  const uint32_t s = (v >> 7) & 0x01010101u;
  return ((v & 0x0F0F0F0Fu) ^ (s * 15u)) + s * 0x81u;
}

// Radix-16 digit d (r16_digits) of eight W-bit coefficients X (four words of
// two 16-bit lanes, coefficient 2i in the low lane of X[i]) as raw bytes in
// K-reversed order: .x = coefficients 7, 6, 5, 4 and .y = 3, 2, 1, 0.  The
// e4m3 byte b in 0..16 is the number b * 2^-9 (0..7 subnormal, 8..15 the
// lowest normal binade, 16 = 2^-5), so every digit is its own encoding and
// the accumulators carry the factor 2^-9.
template <int W>
__device__ __forceinline__ uint2 raw_digits8(const uint32_t (&X)[4], int d) {
  const int lo = 4 * d;
  const int wd = W - lo < 4 ? W - lo : (W - lo == 5 ? 5 : 4);
  const uint32_t mask = ((1u << wd) - 1u) * 0x01010101u;
  uint32_t a, b;
  if (lo + wd <= 8) {  // inside the low byte of each lane
    a = __byte_perm(X[2], X[3], 0x0246) >> lo;
    b = __byte_perm(X[0], X[1], 0x0246) >> lo;
  } else if (lo >= 8) {  // inside the high byte
    a = __byte_perm(X[2], X[3], 0x1357) >> (lo - 8);
    b = __byte_perm(X[0], X[1], 0x1357) >> (lo - 8);
  } else {  // across both
    a = __byte_perm(X[2] >> lo, X[3] >> lo, 0x0246);
    b = __byte_perm(X[0] >> lo, X[1] >> lo, 0x0246);
  }
  if (wd == 5) return make_uint2(raw_sdigits4(a), raw_sdigits4(b));
  return make_uint2(a & mask, b & mask);
}

// Words 2g .. 2g + 5 of one polynomial's s_ext (s_ext[d] = -s[d + 1] for
// d < 255, s[d - 255] from there on) in lane g, from its coefficients 8g .. 8g + 7
// (e0, e1: raw e4m3 bytes).
__device__ __forceinline__ void secret_windows(uint32_t e0, uint32_t e1, int g, uint32_t (&w)[6]) {
  constexpr uint32_t n = 0x80808080u;
  const uint32_t nx = __shfl_sync(0xffffffffu, e0, (g + 1) & 31);
  w[0] = __byte_perm(e0, e1, 0x4321) ^ n;
  w[1] = __byte_perm(e1, nx, 0x4321) ^ (g == 31 ? 0x00808080u : n);  // s_ext[255] = s[0] keeps its sign
#pragma unroll
  for (int i = 1; i <= 2; i++) {  // (past word 63: s_ext[256 + d] = -s_ext[d])
    const uint32_t f = g + i >= 32 ? n : 0u;
    w[2 * i] = __shfl_sync(0xffffffffu, w[0], (g + i) & 31) ^ f;
    w[2 * i + 1] = __shfl_sync(0xffffffffu, w[1], (g + i) & 31) ^ f;
  }
}

// The Hankel core matrices of one polynomial, by a warp (row i of core m,
// s_ext[8m + i .. 8m + i + 15], at byte CS m + 16i of h): lane g makes core g
// from its windows, and lanes 0 .. 9 also core 32 + g, which is minus core g.
// The windows by way of shared memory, eight threads to six cores, took 84 more
// wavefronts of loads for an instance of Saber, on a port that the MMAs' operand
// reads and these stores keep busy, one more barrier for the decryption, and
// 0.9 KB of shared memory a polynomial.  65536 instances, us: Saber's decryption
// 203 -> 169, re-encryption 281 -> 271, encryption 291 -> 285, key generation
// 303 -> 302; FireSaber's re-encryption 461 -> 380 (four CTAs per SM, not
// three), LightSaber's 236 -> 216.  (Cores 128 bytes apart, rows in a
// lane-dependent order against bank conflicts: decryption 179, encryption 294.)
template <class LO>
__device__ __forceinline__ void stage_hankel(uint32_t h, const uint32_t (&w)[6], int g) {
  const uint32_t core = h + (uint32_t)(LO::CS * g);
#pragma unroll
  for (int sh = 0; sh < 4; sh++) {
#pragma unroll
    for (int par = 0; par < 2; par++) {
      uint32_t o[4];
#pragma unroll
      for (int k = 0; k < 4; k++) o[k] = sh ? __funnelshift_r(w[par + k], w[par + k + 1], 8 * sh) : w[par + k];
      const uint32_t at = core + (uint32_t)(64 * par + 16 * sh);
      sts128(at, o[0], o[1], o[2], o[3]);
      if (g < LO::CORES - 32) {
        constexpr uint32_t n = 0x80808080u;
        sts128(at + 32 * LO::CS, o[0] ^ n, o[1] ^ n, o[2] ^ n, o[3] ^ n);
      }
    }
  }
}

// Digit columns of 32 coefficients of one W-bit packed polynomial: lane m
// (0..7) of an 8-lane group takes coefficients 32m .. 32m + 31, exactly W
// aligned words of the stream at src, so that four groups (a warp) reading
// four polynomials load conflict-free, one 32-bit word per lane per load.
// They are K step t = 7 - m: coefficient groups 4m, 4m + 1 of 8 fill the second
// 16-byte K chunk of each digit column and 4m + 2, 4m + 3 the first, one 128-bit
// store each (and one more for the negated copy of steps 4..7).  colbase: the
// digit columns of this j (LO::BM + j * LO::BJ as a shared-window address); cb:
// first column.
template <int W, class LO>
__device__ __forceinline__ void stage_digits32(const uint8_t *sm, int src, uint32_t colbase, int cb, int m) {
  const uint32_t wp = smem_u32(sm) + (uint32_t)(src + 4 * W * m);
  uint32_t w[W];
#pragma unroll
  for (int i = 0; i < W; i++) w[i] = lds32(wp + 4 * i);
  uint32_t X[16];  // coefficients 2k, 2k + 1 in the low / high 16-bit lanes of X[k]
#pragma unroll
  for (int k = 0; k < 16; k++) X[k] = field_pair<W>(w, W, 2 * W * k);
  const int t = 7 - m;
  const uint32_t c1 = colbase + LO::step_off(t), cn = colbase + LO::neg_off(t);
#pragma unroll
  for (int d = 0; d < r16_digits(W); d++) {
    uint2 v[4];
#pragma unroll
    for (int g = 0; g < 4; g++) {
      const uint32_t Xg[4] = {X[4 * g], X[4 * g + 1], X[4 * g + 2], X[4 * g + 3]};
      v[g] = raw_digits8<W>(Xg, d);
    }
    const uint32_t co = (uint32_t)LO::col_off(cb + d);
    sts128(c1 + co + LO::LB, v[1].x, v[1].y, v[0].x, v[0].y);
    sts128(c1 + co, v[3].x, v[3].y, v[2].x, v[2].y);
    if (t >= 4) {
      constexpr uint32_t n = 0x80808080u;
      sts128(cn + co + LO::LB, v[1].x ^ n, v[1].y ^ n, v[0].x ^ n, v[0].y ^ n);
      sts128(cn + co, v[3].x ^ n, v[3].y ^ n, v[2].x ^ n, v[2].y ^ n);
    }
  }
}

// 32 W-bit values (16-bit lanes of x, each below 2^W) as W words at dst.
template <int W>
__device__ __forceinline__ void pack32(uint32_t dst, const uint32_t (&x)[16]) {
  uint32_t o[W + 1] = {};
#pragma unroll
  for (int k = 0; k < 16; k++) {
    const uint32_t y = (x[k] & 0xFFFFu) + ((x[k] >> 16) << W);
    const int bit = 2 * W * k, i = bit >> 5, sh = bit & 31;
    o[i] |= y << sh;
    if (sh + 2 * W > 32) o[i + 1] |= y >> (32 - sh);
  }
#pragma unroll
  for (int i = 0; i < W; i++) sts32(dst + 4 * i, o[i]);
}

// 16-bit values of coefficients 32m .. 32m + 31 of polynomial p (epilogue
// values: 80 bytes a run of 32, so that eight lanes' 128-bit loads differ in
// banks).
__device__ __forceinline__ constexpr int vals_off(int p, int m) { return 80 * (8 * p + m); }
__device__ __forceinline__ void load_vals32(uint32_t src, uint32_t (&x)[16]) {
#pragma unroll
  for (int i = 0; i < 16; i += 4) lds128(src + 4 * i, x[i], x[i + 1], x[i + 2], x[i + 3]);
}

// Two int8 of v sign-extended to 16-bit lanes (SEL: per lane the byte and, with
// bit 3 set, its sign replicated).
template <int SEL>
__device__ __forceinline__ uint32_t sext2(uint32_t v) {
  uint32_t r;
  asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(v), "n"(SEL));
  return r;
}

// Cluster launch control: asks for a CTA of this grid that has not been
// launched yet, to run its work here instead.  The 16-byte answer lands at
// resp and counts on mbar.
__device__ __forceinline__ void clc_try_cancel(uint32_t resp, uint32_t mbar) {
  asm volatile(
      "clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(resp),
      "r"(mbar)
      : "memory");
}
// The answer: the taken CTA's blockIdx.x, or ~0u when none was left to take.
__device__ __forceinline__ uint32_t clc_answer(uint32_t resp) {
  uint32_t x;
  asm volatile(
      "{\n\t.reg .pred p;\n\t.reg .b128 h;\n\t"
      "ld.shared.b128 h, [%1];\n\t"
      "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, h;\n\t"
      "mov.u32 %0, 0xffffffff;\n\t"
      "@p clusterlaunchcontrol.query_cancel.get_first_ctaid::x.b32.b128 %0, h;\n\t}\n"
      : "=r"(x)
      : "r"(resp)
      : "memory");
  return x;
}

// The CTA's barrier, whether the predicate held in all threads: the threads may
// come to it from different branches.
__device__ __forceinline__ bool bar_and(bool p) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %1, 0;\n\t"
      "bar.red.and.pred q, 0, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)p)
      : "memory");
  return r != 0;
}

// The input copies of instance inst into ciphertext / message buffer cb
// (0 or CTB), counted on mbar (one thread).  kDecryptK: ciphertexts
// inst * NCT .. of the one key.
template <int OP, int SET>
__device__ __forceinline__ void cpa5i_load(const CpaArgs &a, const unsigned inst, uint32_t d, uint32_t cb,
                                           uint32_t mbar) {
  using C = SetC<SET>;
  using LO = LayoutC<OP, SET>;
  constexpr bool DECK = OP == kDecryptK;
  const size_t inst0 = DECK ? (size_t)inst * LO::NCT : (size_t)inst;
  const int nvalid = DECK ? min(LO::NCT, a.n - (int)inst0) : 1;
  const uint32_t in_bytes = DECK ? (uint32_t)(C::INDCPA_SK + nvalid * C::CT) : (uint32_t)LO::IN_BYTES;
  mbar_expect_tx(mbar, in_bytes + (a.stall_inputs ? 16 : 0));
  if (LO::HAS_AS) {
    bulk_g2s(d + LO::A, a.a_stream + (a.key_shared ? 0 : (size_t)inst * C::GM), C::GM, mbar);
    bulk_g2s(d + LO::SS, a.s_stream + (size_t)inst * C::GS, C::GS, mbar);
  }
  if (LO::HAS_B) {
    bulk_g2s(d + LO::B, a.pk + (size_t)inst * a.pk_stride + a.pk_off, C::L * C::POLYCOMP, mbar);
    bulk_g2s(d + LO::MSG + cb, a.msg + (size_t)inst * a.msg_stride, 32, mbar);
  }
  if (DECK) {
    for (int r = 0; r < nvalid; r++)
      bulk_g2s(d + LO::CTO + cb + r * LO::CTS, a.ct + (inst0 + r) * C::CT, C::CT, mbar);
  } else if (LO::HAS_CT) {
    bulk_g2s(d + LO::CTO + cb, a.ct + (size_t)inst * C::CT, C::CT, mbar);
  }
  if (LO::HAS_SK)
    bulk_g2s(d + LO::SKO, a.sk + ((a.key_shared || DECK) ? 0 : (size_t)inst * C::SK), C::INDCPA_SK, mbar);
  if (LO::HAS_MV) {
    bulk_g2s(d + LO::A, reinterpret_cast<const uint8_t *>(a.mv_A) + (size_t)inst * LO::MV_A, LO::MV_A, mbar);
    bulk_g2s(d + LO::SS, reinterpret_cast<const uint8_t *>(a.mv_s) + (size_t)inst * LO::MV_S, LO::MV_S, mbar);
  }
}

// Digit sums.  An accumulator holds x * 2^-18 for an exact integer x with
// |x| < 2^22, so adding 1.5 * 2^5 (48) leaves x in the low bits of the f32
// pattern; the pattern of 48.0 itself is 0 in its low 16 bits, which are all
// that the results (mod 2^13 or less) need.  sum_d 16^d x_d is formed in f32 by
// fused multiply-adds where it stays below 2^22 for every admissible secret
// (exact: an integer below 2^24 in units of 2^-18), else the digit of weight
// 256 joins as an integer.
constexpr int digit_bound(int w) { return w == 13 ? 17 * 256 : (w == 9 ? 17 * 16 : (1 << w) - 1); }

// Product p's share of the even (par 0) or odd (1) K steps of one coefficient
// from its accumulator columns f, plus `add` (a small integer), in the low 16
// bits.
template <int OP, int SET>
__device__ __forceinline__ uint32_t combine5(const uint32_t (&f)[2 * ShapeC<OP, SET>::NC4], int p, int par, int add) {
  using S = ShapeC<OP, SET>;
  const int c0 = S::col_base(p), D = S::digits(p), W = p < S::RA ? S::WA : S::WB;
  auto col = [&](int d) { return __uint_as_float(f[2 * (c0 + d) + par]); };
  static_assert(digit_bound(13) * 7 < (1 << 15) && S::ROWS <= 512, "255 * 7 * 512 + add < 2^22");
  float x = col(0) + (48.0f + (float)add / 262144.0f);
  if (D > 1) x = __fmaf_rn(16.0f, col(1), x);
  if (D < 3) return __float_as_uint(x);
  if (digit_bound(W) * S::SMAX * S::ROWS + (1 << 13) < (1 << 22))
    return __float_as_uint(__fmaf_rn(256.0f, col(2), x));
  return __float_as_uint(x) + 256u * __float_as_uint(col(2) + 48.0f);
}

// The decryptions are launched ordinarily (chain.cuh): they start a pass beside
// the Keccak front on another stream, so nothing is gained there, and the two
// instructions of the wait alone cost the decryption of 65536 Saber ciphertexts
// 10 us (registers: it has 32).
constexpr bool is_decryption(int op) { return op == kDecrypt || op == kDecryptK; }

// The instances of a launch, from the CTA of kI5Threads threads that runs
// blockIdx.x (sm: its dynamic shared memory).  at(gi) names the arguments and
// the instance of CTA gi: a pair-like struct {const CpaArgs &a; unsigned inst}.
//
// The grid has one CTA per instance, but a resident CTA goes on to the next
// one that has not started (cluster launch control) instead of exiting: tensor
// memory and barriers are set up once, and the next instance's input copies
// run beside the epilogue of this one.  Without that, an empty instance (no
// staging, no MMAs) took 0.207 of the decryption's 0.273 ms at 65536; with it
// 0.090 of 0.246 (re-encryption 0.353 -> 0.342).
//
// What bounds the kernel now: the shared-memory port and the instruction
// slots, each about 60 % busy, in phases that only other CTAs overlap (65536
// Saber, us, decryption / re-encryption: 203 / 281 before the core matrices came
// from registers; without the MMAs 153 / 240, without the core matrices 154 /
// 243, without the digits 185 / 209, inputs from L2 203 / 281).
//
// TAIL: warp 0 finishes the instance (CpaArgs::tail) while the others go on to
// the next one's first barrier.
template <int OP, int SET, bool TAIL = false, class AT>
__device__ __forceinline__ void cpa5i_run(const AT &at, uint8_t *sm) {
  using C = SetC<SET>;
  using S = ShapeC<OP, SET>;
  using LO = LayoutC<OP, SET>;
  constexpr int L = C::L, NU = S::NU, NT = kI5Threads;
  const uint32_t mbar_in = smem_u32(sm + LO::BAR), mbar_mma = mbar_in + 8, mbar_clc = mbar_in + 16;
  const uint32_t clc_resp = mbar_in + 32;
  uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(sm + LO::BAR + 24);
  volatile uint32_t *next_slot = reinterpret_cast<volatile uint32_t *>(sm + LO::BAR + 28);
  constexpr bool DECK = OP == kDecryptK, IS_DEC = OP == kDecrypt || DECK;

  // 0. tensor memory, barriers, and the first input copies (one thread)
  if (threadIdx.x < 32) tmem_alloc(smem_u32(tmem_slot), S::TMEM_COLS);
  if (threadIdx.x == 0) {
    mbar_init(mbar_in, 1);
    mbar_init(mbar_mma, 1);
    mbar_init(mbar_clc, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (!is_decryption(OP)) chain_wait();
    const auto w = at(blockIdx.x);
    cpa5i_load<OP, SET>(w.a, w.inst, smem_u32(sm), 0, mbar_in);
  }
  if (!is_decryption(OP)) chain_wait();  // (all threads)
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t *>(tmem_slot);
  uint32_t *sec8w = reinterpret_cast<uint32_t *>(sm + LO::SEC8);
  uint8_t *H = sm + LO::H, *Bm = sm + LO::BM;
  unsigned gi = blockIdx.x;
  for (uint32_t it = 0;; it++) {
  // per-thread values are made afresh for every instance (not kept across the
  // loop in registers, which bound the CTAs per SM)
  int tid = threadIdx.x;
  asm volatile("" : "+r"(tid));
  const int warp = tid >> 5, lane = tid & 31;
  const uint32_t par = it & 1u, cbuf = par ? (uint32_t)LO::CTB : 0u;
  const auto here = at(gi);
  const CpaArgs &a = here.a;
  const unsigned inst = here.inst;
  const size_t inst0 = DECK ? (size_t)inst * LO::NCT : (size_t)inst;
  const int nvalid = DECK ? min(LO::NCT, a.n - (int)inst0) : 1;
  if (tid == 0) {  // ask for the next instance; answer buffer par was read before this instance's predecessor's barriers
    mbar_expect_tx(mbar_clc, 16);
    clc_try_cancel(clc_resp + 16 * par, mbar_clc);
  }
  bool ready = __all_sync(0xffffffffu, mbar_wait_bounded(mbar_in, par)) != 0;  // (a warp's lanes agree: shuffles follow)
  if (ready) {
    // 1. digit columns (K reversed, core-matrix order): lane g converts
    // coefficients 8g..8g+7 (K rows k' = 8kq+7..8kq, kq = 31 - g) of one
    // polynomial per item.  Warp p < R makes polynomial p of every j (one
    // item per j); with R == 1 (decryption) warp j makes j.  The columns past
    // NCOLS of each stored group are left as they are: they only feed
    // accumulator columns that are never read.
    const int kq = 31 - lane;
    const uint32_t bh = smem_u32(Bm) + (uint32_t)(((kq >> 1) & 1) * LO::LB + 8 * (kq & 1));
    const uint32_t bl = bh + LO::step_off(kq >> 2), bn = bh + LO::neg_off(kq >> 2);
    auto put = [&](int j, int n, uint2 v) {
      sts64(bl + j * LO::BJ + LO::col_off(n), v.x, v.y);
      if (kq >= 16) sts64(bn + j * LO::BJ + LO::col_off(n), v.x ^ 0x80808080u, v.y ^ 0x80808080u);
    };
    auto item = [&](auto wc, uint32_t src, int cb, int j) {
      constexpr int W = decltype(wc)::value;
      uint32_t X[4];
      unpack8d<W>(sm + src, lane * W, X);
#pragma unroll
      for (int d = 0; d < r16_digits(W); d++) {
        put(j, cb + d, raw_digits8<W>(X, d));
      }
    };
    if constexpr (OP == kMatvec) {
      // coefficients already in 16-bit lanes: digit d of the low 13 bits
      // (the result is needed mod 2^eq, eq <= 13)
      // over the warps that have no secrets
      for (int t = warp; t < L * L && warp < NT / 32 - L; t += NT / 32 - L) {
        const int p = t / L, j = t % L;
        const int ij = a.mv_transpose ? (j * L + p) : (p * L + j);
        uint32_t X[4];
        lds128(smem_u32(sm + LO::A) + (uint32_t)(512 * ij + 16 * lane), X[0], X[1], X[2], X[3]);
#pragma unroll
        for (int d = 0; d < S::DA; d++) put(j, p * S::DA + d, raw_digits8<S::WA>(X, d));
      }
    } else if constexpr (DECK) {
      // warp r makes ciphertext r's b'_j for every j
      if (warp < nvalid) {
#pragma unroll
        for (int j = 0; j < L; j++)
          item(std::integral_constant<int, S::WB>{}, (int)cbuf + LO::CTO + warp * LO::CTS + 32 * j * S::WB, warp * S::DB,
               j);
      }
    } else if constexpr (S::R == 1) {
      if (warp < L) item(std::integral_constant<int, S::WB>{}, (int)cbuf + LO::CTO + 32 * warp * S::WB, 0, warp);
    } else {
      // public matrix A (RA x L polynomials), then b (encryption, re-encryption):
      // four polynomials per warp, eight lanes each; one that is left over (the
      // ninth for L = 3) by a whole warp, in a third of the instructions (65536
      // Saber, us: key generation 302 -> 297, encryption 285 -> 281,
      // re-encryption 271 -> 268)
      constexpr int NA = S::RA * L, NB = (S::R - S::RA) * L, NA8 = NA % 4 == 1 ? NA - 1 : NA;
      constexpr int WA_WARPS = (NA + 3) / 4, WB_WARPS = (NB + 3) / 4;
      static_assert(WA_WARPS + WB_WARPS <= 8, "digit polynomials fit the CTA's warps");
      const uint32_t bm32 = smem_u32(Bm);
      if (4 * warp < NA8) {
        const int t = 4 * warp + (lane >> 3);
        if (t < NA8) {
          const int p = t / L, j = t % L;
          const int ij = (OP == kKeygen) ? (j * L + p) : (p * L + j);
          stage_digits32<S::WA, LO>(sm, LO::A + 32 * ij * S::WA, bm32 + (uint32_t)(j * LO::BJ), p * S::DA, lane & 7);
        }
      } else if (warp < WA_WARPS) {
        item(std::integral_constant<int, S::WA>{}, LO::A + 32 * (L * L - 1) * S::WA, (S::RA - 1) * S::DA, L - 1);
      } else if (warp < WA_WARPS + WB_WARPS) {
        const int t = 4 * (warp - WA_WARPS) + (lane >> 3);
        if (t < NB) {
          const int pb = t / L, j = t % L;
          stage_digits32<S::WB, LO>(sm, LO::B + 32 * j * S::WB, bm32 + (uint32_t)(j * LO::BJ),
                                    S::RA * S::DA + pb * S::DB, lane & 7);
        }
      }
    }
  }
  // 2. secrets: a polynomial to a warp that makes no digit columns (the last L
  // warps, of which the one of b does for L = 4); lane g takes the words 2g,
  // 2g + 1 (coefficients 8g..8g+7).  Core matrices over the streams wait in a
  // barrier until those are read (in both branches, so that only these warps
  // hold their windows across it).
  const int sj = S::R == 1 ? warp - L : kI5Threads / 32 - 1 - warp;
  if (sj >= 0 && sj < L) {
    uint32_t win[6] = {};
    if (ready) {
      const int j = sj, g = lane;
      uint32_t sb[2], bad = 0;
      if (IS_DEC && !C::SABLE) {
        // 13-bit two's complement (SABER pack.cu:53-84); -8 .. 7 where bits 3 .. 12
        // agree (fields unmasked and one check for both words: 169 -> 166 us for
        // 65536 Saber decryptions)
        uint32_t X[4];
        unpack8d<C::EQ>(sm + LO::SKO, (32 * j + g) * C::EQ, X);
#pragma unroll
        for (int i = 0; i < 4; i++) bad |= X[i] ^ (X[i] >> 1);
        bad &= 0x0FF80FF8u;
        sb[0] = __byte_perm(X[0], X[1], 0x6420);
        sb[1] = __byte_perm(X[2], X[3], 0x6420);
      } else {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int w = 64 * j + 2 * g + h;
          if (OP == kMatvec) {
            sb[h] = lds32(smem_u32(sm + LO::SS) + 4 * w);  // four int8 coefficients
            bad |= (sb[h] ^ (sb[h] >> 1)) & 0x78787878u;
          } else if (IS_DEC) {
            // 2-bit two's complement (SABLE pack.cu:371-376): one byte = 4 coefficients
            const uint32_t x = sm[LO::SKO + w];
            const uint32_t spread = (x & 3u) | ((x & 0xcu) << 6) | ((x & 0x30u) << 12) | ((x & 0xc0u) << 18);
            sb[h] = spread | (((spread >> 1) & 0x01010101u) * 0xfcu);
          } else if (C::MU == 8) {
            // CBD mu = 8 (SABER poly.cu:864-887)
            const uint32_t x = lds32(smem_u32(sm + LO::SS) + 4 * w);
            uint32_t n = x - ((x >> 1) & 0x55555555u);
            n = (n & 0x33333333u) + ((n >> 2) & 0x33333333u);
            sb[h] = __vsub4(n & 0x0f0f0f0fu, (n >> 4) & 0x0f0f0f0fu);
          } else if (C::MU == 2) {
            // CBD mu = 2 (SABLE fips202.cu:625-651)
            const uint32_t x = sm[LO::SS + w];
            const uint32_t spread = (x & 3u) | ((x & 0xcu) << 6) | ((x & 0x30u) << 12) | ((x & 0xc0u) << 18);
            sb[h] = __vsub4(spread & 0x01010101u, (spread >> 1) & 0x01010101u);
          } else {
            // CBD mu = 6, 10: fields of mu bits, popcount halves
            uint32_t r = 0;
#pragma unroll
            for (int b = 0; b < 4; b++) {
              const uint32_t x = get_bits(sm + LO::SS, (4 * w + b) * C::MU, C::MU);
              const int v = __popc(x & ((1u << (C::MU / 2)) - 1u)) - __popc(x >> (C::MU / 2));
              r |= ((uint32_t)v & 0xffu) << (8 * b);
            }
            sb[h] = r;
          }
        }
      }
      if (OP == kKeygen) {
        sec8w[64 * j + 2 * g] = sb[0];
        sec8w[64 * j + 2 * g + 1] = sb[1];
      }
      const uint32_t e0 = raw_secrets4(sb[0]), e1 = raw_secrets4(sb[1]);
      // a magnitude of 8 is too large too (CBD secrets are at most mu / 2 <= 5, the 2-bit ones 2)
      if ((IS_DEC && !C::SABLE) || OP == kMatvec) {
        if ((bad | ((e0 | e1) & 0x08080808u)) != 0u && a.err) atomicOr(a.err, 1);
      }
      secret_windows(e0, e1, g, win);
    }
    if (LO::PLACE != kFree) ready = bar_and(ready);
    if (ready) stage_hankel<LO>(smem_u32(H) + (uint32_t)(sj * LO::HJ), win, lane);
  } else if (LO::PLACE != kFree) {
    ready = bar_and(ready);
  }
  fence_async_smem();  // generic-proxy writes -> visible to the tensor core
  ready = __syncthreads_and(ready) != 0;
  if (!ready) {  // the input copies did not complete in time: report, leave
    if (tid == 0 && a.err) atomicOr(a.err, 2);
    if (warp == 0) {
      mbar_wait_bounded(mbar_in, par);
      mbar_wait_bounded(mbar_clc, par);
    }
    break;
  }
  // 3. the MMAs (one thread).  Coefficients and K steps come in blocks of 32:
  // coefficient block o takes step t through the 32 x 32 Hankel block
  // B = o + t (rows 32B + r of s_ext[. + e]), where block B + 8 = -block B
  // (s_ext[d + 256] = -s_ext[d] for d < 255).  A tile w is the blocks
  // w .. w + 3, four lane quadrants rho, read from core 4w on.  An MMA costs
  // about (4 KB + 32 N bytes) / 128 cycles, the reads of its operands from
  // shared memory (N = 16: 39, 32: 40, 64: 48 cycles measured), so fewer MMAs of a
  // larger N do the same products in less time.
  // So only the even tiles are used, each against four steps: tile w against
  // step w gives blocks o = rho, against step w - 4 (w < 4: the negated step
  // w + 4) blocks o = rho + 4; against the odd steps w + 1 and w - 3 (-(w + 5))
  // blocks o = rho - 1 (block -1 = -block 7) and rho + 3, which other warps
  // finish.  Two sets of 2 NC4 columns, for rho and rho + 4, even and odd
  // steps in turn.  12 MMAs of N = 48 for Saber's re-encryption (24 of N = 32
  // with a tile per step): 342 -> 301 us at 65536 with the stagings above, the
  // decryption 246 -> 216.  (Two tiles against all eight steps, 6 MMAs of
  // N = 32 for the decryption, took 225: the sums of eight products of each
  // block then cross all warps.)
  if (tid == 0) {
    tc_fence_after();  // the previous instance's accumulator loads come before these MMAs
    constexpr uint32_t idesc = umma_idesc_e4m3(NU);
    const uint64_t ad0 = umma_desc(smem_u32(H), 2 * LO::CS, LO::CS);
    const uint64_t bd0 = umma_desc(smem_u32(Bm), LO::LB, LO::SB);
#pragma unroll
    for (int j = 0; j < L; j++) {
      const uint64_t hj = ad0 + (uint64_t)((j * LO::HJ) >> 4), bj = bd0 + (uint64_t)((j * LO::BJ) >> 4);
#pragma unroll
      for (int w = 0; w < 8; w += 2)
        umma_f8(tmem, hj + (uint64_t)((4 * w * LO::CS) >> 4),
                bj + (uint64_t)((((w >> 1) & 1) * LO::QB + (w < 4 ? S::PG * LO::SB : 0)) >> 4), idesc, (j | w) != 0);
    }
    umma_commit(mbar_mma);
  }
  // 4. accumulators: one warp polls the MMA barrier and the CLC answer, the
  // others wait in the CTA barrier.  The next instance's copies start as soon
  // as what they overwrite is read: beside the MMAs, or beside the epilogue
  // where they land in H (the other ciphertext buffer was last read before this
  // instance's barriers).
  bool done = true;
  if (warp == 0) {
    if (LO::PLACE != kFree) done = mbar_wait_bounded(mbar_mma, par);
    done = mbar_wait_bounded(mbar_clc, par) && done;
    done = __all_sync(0xffffffffu, done) != 0;
    if (tid == 0) {
      const uint32_t nx = done ? clc_answer(clc_resp + 16 * par) : ~0u;
      *next_slot = nx;
      if (nx != ~0u) {
        const auto wn = at(nx);
        cpa5i_load<OP, SET>(wn.a, wn.inst, smem_u32(sm), (uint32_t)LO::CTB - cbuf, mbar_in);
      }
      if (OP == kReenc && done) a.fail[inst] = 0;  // set below, after the barrier, by a warp that finds a difference
    }
    if (LO::PLACE == kFree) done = mbar_wait_bounded(mbar_mma, par) && done;
  }
  done = __syncthreads_and(done) != 0;
  if (!done) {
    // the tensor core or the CLC answer did not come in time: report, and
    // give what is still in flight a second bounded wait before releasing
    if (tid == 0 && a.err) atomicOr(a.err, 2);
    if (warp == 0) {
      mbar_wait_bounded(mbar_mma, par);
      mbar_wait_bounded(mbar_clc, par);
      if (*next_slot != ~0u) mbar_wait_bounded(mbar_in, par ^ 1u);
    }
    break;
  }
  const uint32_t next = *next_slot;
  tc_fence_after();
  // The thread's coefficient k (block o = 4 hsel + q4 of 32; its warp reads
  // tensor-memory lanes 32 q4 ..), and what the epilogue needs of the inputs:
  // the ciphertext's coefficient k, the message bit.  (Read here: beside the
  // MMAs, which read shared memory at full rate, the same loads made the
  // re-encryption 299 instead of 285 us at 65536, by shuffles from one load a
  // warp 303.)
  const int q4 = warp & 3, hsel = warp >> 2;
  const int k = 128 * hsel + 32 * q4 + lane;
  const uint32_t ctb = smem_u32(sm) + cbuf + (uint32_t)LO::CTO;
  constexpr int CMO = L * C::POLYCOMP;
  auto field = [&](uint32_t off, int W) -> uint32_t {  // coefficient k of the W-bit stream at ctb + off
    const uint32_t p = ctb + off + (uint32_t)(((W * k) >> 5) * 4);
    return __funnelshift_r(lds32(p), lds32(p + 4), (W * k) & 31) & ((1u << W) - 1u);
  };
  uint32_t cf[LO::HAS_CT ? S::R : 1], mk = 0;
  if constexpr (IS_DEC) {  // c_m of each ciphertext
#pragma unroll
    for (int r = 0; r < S::R; r++) cf[r] = field((uint32_t)(r * LO::CTS + CMO), C::ET);
  }
  if constexpr (LO::HAS_B) mk = (sm[LO::MSG + cbuf + (k >> 3)] >> (k & 7)) & 1u;
  if constexpr (OP == kReenc) {
#pragma unroll
    for (int p = 0; p < L; p++) cf[p] = field((uint32_t)(p * C::POLYCOMP), C::EP);
    cf[L] = field((uint32_t)CMO, C::ET);
  }
  const uint32_t xch = smem_u32(sm + LO::XCH);
  // coefficient k of every product, in the low 16 bits (a.. the sums of an
  // accumulator's digit columns, see combine5)
  uint32_t val[S::R];
  // the rounding constant that the op adds to every product
  constexpr int ROUND = IS_DEC ? C::H2 : (OP == kMatvec ? 0 : C::H1);
  {
    const uint32_t t0 = tmem + ((uint32_t)(32 * q4) << 16);
    // odd steps first: block o' = q4 - 1 (hsel 0; block 7 negated for
    // q4 = 0) or q4 + 3, for the warp of that block; two 16-bit values a word
    uint32_t f[2 * S::NC4];
    uint32_t odd[S::R];
    tmem_ld_cols(t0 + (uint32_t)(2 * S::NC4 * hsel), f);
    const int od = (warp + 7) & 7;  // the block the odd steps belong to
#pragma unroll
    for (int p = 0; p < S::R; p++) odd[p] = combine5<OP, SET>(f, p, 1, 0);
    if (warp == 0) {
#pragma unroll
      for (int p = 0; p < S::R; p++) odd[p] = 0u - odd[p];
    }
#pragma unroll
    for (int i = 0; i < LO::XWORDS; i++)
      sts32(xch + (uint32_t)((i * 256 + 32 * od + lane) * 4), __byte_perm(odd[2 * i], odd[2 * i + 1], 0x5410));
    if (S::R & 1) *reinterpret_cast<uint16_t *>(sm + LO::XCH + 1024 * LO::XWORDS + 2 * (32 * od + lane)) = (uint16_t)odd[S::R - 1];
#pragma unroll
    for (int p = 0; p < S::R; p++) val[p] = combine5<OP, SET>(f, p, 0, ROUND);
    tc_fence_before();  // the loads above come before the next instance's MMAs (its barriers lie between)
    __syncthreads();
#pragma unroll
    for (int i = 0; i < LO::XWORDS; i++) {
      const uint32_t x = lds32(xch + (uint32_t)((i * 256 + tid) * 4));
      val[2 * i] += x;
      val[2 * i + 1] += x >> 16;
    }
    if (S::R & 1) val[S::R - 1] += *reinterpret_cast<const uint16_t *>(sm + LO::XCH + 1024 * LO::XWORDS + 2 * tid);
  }
  if constexpr (OP == kEncrypt || OP == kKeygen) {
    // coefficient k of every output polynomial, rounded (b, b') or encoded
    // with the message bit (c_m), as 16-bit values for the packing pass;
    // the MMAs are done, so the digit columns are free
    constexpr uint32_t qm = (1u << C::EQ) - 1u, pm = (1u << C::EP) - 1u;
#pragma unroll
    for (int p = 0; p < S::R; p++) {
      const uint32_t v = val[p];
      uint16_t *at32 = reinterpret_cast<uint16_t *>(sm + LO::VALS + vals_off(p, warp)) + lane;
      if (p < L) {
        *at32 = (uint16_t)((v & qm) >> (C::EQ - C::EP));
      } else {
        *at32 = (uint16_t)(((v - (mk << (C::EP - 1))) & pm) >> (C::EP - C::ET));
      }
    }
    __syncthreads();  // the 16-bit values are complete
  }

  // 5. epilogues
  constexpr uint32_t pmask = (1u << C::EP) - 1u;
  if constexpr (OP == kDecrypt) {
    // m'_k = ((v_k + h2 - (c_m,k << (ep-et))) mod p) >> (ep-1): one bit per
    // thread, gathered into bytes by a ballot per warp
    const uint32_t v = val[0];
    const uint32_t t = (v - (cf[0] << (C::EP - C::ET))) & pmask;
    const uint32_t bits = __ballot_sync(0xffffffffu, ((t >> (C::EP - 1)) & 1u) != 0u);
    uint8_t *mo = a.m_out + (size_t)inst * a.m_out_stride;
    if (lane == 0) reinterpret_cast<uint32_t *>(mo)[4 * hsel + q4] = bits;  // (rows of 32 or 64 bytes)
    if (a.copy_hpk && warp == 0) mo[32 + lane] = a.sk[(a.key_shared ? 0 : (size_t)inst * C::SK) + C::SK - 64 + lane];
  } else if constexpr (DECK) {
    // ciphertext r of the CTA: decode as above from its own columns and c_m
#pragma unroll
    for (int r = 0; r < S::R; r++) {
      if (r >= nvalid) break;
      const uint32_t v = val[r];
      const uint32_t t = (v - (cf[r] << (C::EP - C::ET))) & pmask;
      const uint32_t bits = __ballot_sync(0xffffffffu, ((t >> (C::EP - 1)) & 1u) != 0u);
      uint8_t *mo = a.m_out + (inst0 + r) * a.m_out_stride;
      if (lane == 0) reinterpret_cast<uint32_t *>(mo)[4 * hsel + q4] = bits;
      if (a.copy_hpk && warp == 0) mo[32 + lane] = a.sk[C::SK - 64 + lane];
    }
  } else if constexpr (OP == kReenc) {
    // round coefficient k of b' and encode that of v', compare with the ciphertext
    uint32_t diff = 0, diffm = 0;
#pragma unroll
    for (int p = 0; p < S::R; p++) {
      const uint32_t v = val[p];
      if (p < L) diff |= (v >> (C::EQ - C::EP)) ^ cf[p];
      else diffm = ((v - (mk << (C::EP - 1))) >> (C::EP - C::ET)) ^ cf[L];
    }
    diff = (diff & pmask) | (diffm & ((1u << C::ET) - 1u));
    if constexpr (TAIL) {
      const bool bad = __syncthreads_or(diff != 0u) != 0;
      if (warp == 0) {
        const WarpSponge e{lane, true, warp_keccak_lane(lane)};
        const uint8_t *z = a.sk + (a.key_shared ? 0 : (size_t)inst * C::SK) + C::SK - 32;
        const auto kk = e.sel4(e.load(a.kr + (size_t)inst * 64, 4), e.load(z, 4), bad);
        e.store(a.ss + (size_t)inst * 32, e.template sha3_256<8>(e.cat4(kk, e.load(a.hc + (size_t)inst * 32, 4))), 4);
      }
    } else {
      if (__any_sync(0xffffffffu, diff != 0u) && lane == 0) a.fail[inst] = 1;
    }
  } else if constexpr (OP == kMatvec) {
    // coefficient k of every output polynomial, mod 2^eq
    const uint32_t m = (1u << a.mv_eq) - 1u;
    uint16_t *o = a.mv_out + (size_t)inst * (L * 256) + k;
#pragma unroll
    for (int p = 0; p < L; p++) o[256 * p] = (uint16_t)(val[p] & m);
  } else if (OP == kEncrypt) {
    // pack the 16-bit values, 32 to a lane: b' at EP bits (warp 0), c_m at ET
    // bits (warp 1)
    const uint32_t out = smem_u32(sm + LO::OUT), vals = smem_u32(sm + LO::VALS);
    uint32_t x[16];
    if (warp == 0 && lane < 8 * L) {
      load_vals32(vals + vals_off(0, lane), x);
      pack32<C::EP>(out + 4 * C::EP * lane, x);
    } else if (warp == 1 && lane < 8) {
      load_vals32(vals + vals_off(L, lane), x);
      pack32<C::ET>(out + L * C::POLYCOMP + 4 * C::ET * lane, x);
    }
    __syncthreads();
    copy16(a.ct_out + (size_t)inst * C::CT, sm + LO::OUT, C::CT);
    if (TAIL && warp == 0) {
      const WarpSponge e{lane, true, warp_keccak_lane(lane)};
      const auto h = e.sha3_256_mem(sm + LO::OUT, C::CT);
      e.store(a.ss + (size_t)inst * 32, e.template sha3_256<8>(e.cat4(e.load(a.kr + (size_t)inst * 64, 4), h)), 4);
    }
  } else if (OP == kKeygen) {
    constexpr int bbytes = L * C::POLYCOMP;
    uint8_t *outb = sm + LO::OUT;
    const uint32_t out = smem_u32(outb);
    uint32_t x[16];
    if (warp == 0 && lane < 8 * L) {
      load_vals32(smem_u32(sm + LO::VALS) + vals_off(0, lane), x);
      pack32<C::EP>(out + 4 * C::EP * lane, x);
    } else if (warp == 1 && lane < 8 * L) {
      // secret key: 13-bit two's complement (Saber) or 2-bit (Sable) of sec8,
      // two int8 at a time sign-extended to 16-bit lanes
      constexpr int sw = C::SABLE ? 2 : C::EQ;
      const uint32_t s8 = smem_u32(sm + LO::SEC8) + 32 * lane;
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const uint32_t v = lds32(s8 + 4 * i);
        x[2 * i] = sext2<0x9180>(v) & (((1u << sw) - 1u) * 0x10001u);
        x[2 * i + 1] = sext2<0xB3A2>(v) & (((1u << sw) - 1u) * 0x10001u);
      }
      pack32<sw>(out + bbytes + 4 * sw * lane, x);
    }
    __syncthreads();
    uint8_t *pko = a.pk_out + (size_t)inst * C::PK;
    uint8_t *sko = a.sk_out + (size_t)inst * a.sk_stride;
    if (tid < 32) sko[C::INDCPA_SK + bbytes + tid] = pko[bbytes + tid];  // seed_A
    copy16(pko, outb, bbytes);
    copy16(sko + C::INDCPA_SK, outb, bbytes);
    copy16(sko, outb + bbytes, C::INDCPA_SK);
    if constexpr (TAIL) {
      __syncthreads();  // pk is complete in global memory
      if (warp == 0) {
        const WarpSponge e{lane, true, warp_keccak_lane(lane)};
        const auto h = e.sha3_256_mem(pko, C::PK);
        e.store(sko + C::SK - 64, e.cat4(h, e.load(a.coins + (size_t)inst * 96 + 64, 4)), 8);
      }
    }
  }
  if (next == ~0u) break;
  gi = next;
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x < 32) tmem_dealloc(tmem, S::TMEM_COLS);
}

// CTAs per SM that shared memory (228 KB, 1 KB of it per CTA reserved), tensor
// memory (512 columns) and registers allow.  The speed comes from the CTAs that
// overlap each other's phases.
template <int OP, int SET>
constexpr int min_ctas() {
  constexpr int by_smem = LayoutC<OP, SET>::CTAS, by_tmem = 512 / ShapeC<OP, SET>::TMEM_COLS;
  constexpr int m = by_smem < by_tmem ? by_smem : by_tmem;
  constexpr int cap = reg_ctas<OP, SET>();
  return m < cap ? m : cap;
}

// The arguments and the instance that CTA gi of a launch stands for.
struct CpaAt {
  const CpaArgs &a;
  unsigned inst;
};

template <int OP, int SET>
__global__ void __launch_bounds__(kI5Threads, min_ctas<OP, SET>()) k_cpa5i(const __grid_constant__ CpaArgs a) {
  extern __shared__ __align__(16) uint8_t sm[];
  cpa5i_run<OP, SET>([&](unsigned gi) { return CpaAt{a, gi}; }, sm);
}

// The same with the instance's last Keccak stage in it (CpaArgs::tail).
template <int OP, int SET>
__global__ void __launch_bounds__(kI5Threads, 2) k_cpa5t(const __grid_constant__ CpaArgs a) {
  extern __shared__ __align__(16) uint8_t sm[];
  cpa5i_run<OP, SET, true>([&](unsigned gi) { return CpaAt{a, gi}; }, sm);
}

// Mixed launch whose groups all have parameter set SET (the per-set launches
// of a mixed pass): the group table travels as a kernel parameter (constant
// bank), so a CTA finds its group and reads its arguments without a global
// round trip; then the same body as k_cpa5i, with the same registers and
// occupancy.  CTA gi stands for instance gi of the table.
struct MixParam {
  int ngroups, total;
  int first[kMaxGroups + 1];
  CpaArgs g[kMaxGroups];
};
static_assert(sizeof(MixParam) < 32000, "the group table fits the kernel-parameter space");

template <int OP, int SET>
__global__ void __launch_bounds__(kI5Threads, min_ctas<OP, SET>()) k_cpa5ms(const __grid_constant__ MixParam T) {
  extern __shared__ __align__(16) uint8_t sm[];
  cpa5i_run<OP, SET>(
      [&](unsigned u) {
        const int gi = (int)u;
        int lo = 0, hi = T.ngroups - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (gi >= T.first[mid]) lo = mid;
          else hi = mid - 1;
        }
        return CpaAt{T.g[lo], (unsigned)(gi - T.first[lo])};
      },
      sm);
}

// Pads `smem` until at most 512 / cols CTAs of fn fit on an SM, so that every
// resident CTA's tensor-memory allocation succeeds at once.
template <class F>
inline int cap_tmem_residency(F fn, int &smem, int cols) {
  const int cap = 512 / cols;
  cudaError_t e;
  for (int it = 0; it < 64; it++) {
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess)
      return (int)e;
    int nb = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, kI5Threads, smem)) != cudaSuccess) return (int)e;
    if (nb <= cap) return 0;
    smem += 2048;
  }
  return 0;
}

template <int OP, int SET>
inline int launch_cpa5ms(const CpaArgs *groups, int ng, cudaStream_t s) {
  using LO = LayoutC<OP, SET>;
  using S = ShapeC<OP, SET>;
  if (ng < 1 || ng > kMaxGroups) return (int)cudaErrorInvalidValue;
  MixParam T;
  T.ngroups = ng;
  T.first[0] = 0;
  for (int g = 0; g < ng; g++) {
    T.g[g] = groups[g];
    T.first[g + 1] = T.first[g] + groups[g].n;
  }
  T.total = T.first[ng];
  for (int g = ng; g < kMaxGroups; g++) T.first[g + 1] = T.total;
  if (T.total <= 0) return 0;
  auto fn = k_cpa5ms<OP, SET>;
  int smem = LO::TOTAL;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return (int)e;
  int rc = cap_tmem_residency(fn, smem, S::TMEM_COLS);
  if (rc) return rc;
  return (int)launch_chained<!is_decryption(OP)>(fn, T.total, kI5Threads, smem, s, T);
}

// Groups of one parameter set (a mixed pass launches each set's groups by themselves).
template <int OP>
inline int launch_cpa5m(const CpaArgs *groups, int ng, cudaStream_t s) {
  for (int g = 1; g < ng; g++)
    if (groups[g].P.set != groups[0].P.set) return (int)cudaErrorInvalidValue;
  switch (groups[0].P.set) {
    case 0: return launch_cpa5ms<OP, 0>(groups, ng, s);
    case 1: return launch_cpa5ms<OP, 1>(groups, ng, s);
    case 2: return launch_cpa5ms<OP, 2>(groups, ng, s);
    case 3: return launch_cpa5ms<OP, 3>(groups, ng, s);
    case 4: return launch_cpa5ms<OP, 4>(groups, ng, s);
    case 5: return launch_cpa5ms<OP, 5>(groups, ng, s);
  }
  return (int)cudaErrorInvalidValue;
}

template <int OP, int SET>
inline int launch_cpa5i(const CpaArgs &a, cudaStream_t s) {
  using LO = LayoutC<OP, SET>;
  using S = ShapeC<OP, SET>;
  auto fn = k_cpa5i<OP, SET>;
  if constexpr (OP == kReenc || OP == kEncrypt || OP == kKeygen) {
    if (a.tail) fn = k_cpa5t<OP, SET>;
  }
  int smem = LO::TOTAL;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  if (e != cudaSuccess) return (int)e;
  // at most 512 / TMEM_COLS resident CTAs per SM, so every CTA's tensor
  // memory allocation succeeds at once: pad the shared memory until no more fit
  const int cap = 512 / S::TMEM_COLS;
  for (int it = 0; it < 64; it++) {
    if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess)
      return (int)e;
    int nb = 0;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fn, kI5Threads, smem)) != cudaSuccess) return (int)e;
    if (nb <= cap) break;
    smem += 2048;
  }
  return (int)launch_chained<!is_decryption(OP)>(fn, OP == kDecryptK ? (a.n + S::R - 1) / S::R : a.n, kI5Threads,
                                                 smem, s, a);
}

// Dispatch over the six parameter sets (matvec is not set-shaped).
template <int OP>
inline int launch_cpa5i_set(const CpaArgs &a, cudaStream_t s) {
  switch (a.P.set) {
    case 0: return launch_cpa5i<OP, 0>(a, s);
    case 1: return launch_cpa5i<OP, 1>(a, s);
    case 2: return launch_cpa5i<OP, 2>(a, s);
    case 3: return launch_cpa5i<OP, 3>(a, s);
    case 4: return launch_cpa5i<OP, 4>(a, s);
    case 5: return launch_cpa5i<OP, 5>(a, s);
  }
  return (int)cudaErrorInvalidValue;
}

}  // namespace tmvp
