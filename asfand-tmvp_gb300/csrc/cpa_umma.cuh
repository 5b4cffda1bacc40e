// cpa_umma.cuh — the tcgen05 (5th-generation tensor core) engine of the
// FP8 IND-CPA form.
//
// One CTA computes, for its instance, D[256][N] = sum_j H_j x B_j where
//   * H_j is the 256 x 256 matrix of the secret polynomial s_j with the K
//     index reversed: H_j[r][k'] = s_ext[r + k'] (a Hankel matrix), which is
//     the negacyclic Toeplitz matrix T(s_j)[r][c] = s_ext[r - c + 255] with
//     c = 255 - k';
//   * B_j holds N digit columns of the public polynomials of module index j,
//     coefficient c at row k' = 255 - c;
// with tcgen05.mma kind::f8f6f4 (e4m3 x e4m3 -> f32), M = 128, N = 16 .. 64,
// K = 32 per instruction, A and B read from shared memory and D
// accumulated in tensor memory (TMEM).
//
// Operand layout (K-major, no swizzle): the MMA reads "core matrices" of 8
// rows x 16 bytes, stored as 128 contiguous bytes; the shared-memory
// descriptor gives the byte distance between core matrices adjacent in K
// (leading byte offset, LBO) and in M/N (stride byte offset, SBO).
//   * H_j: the core matrix at 8-row group b and 16-byte K chunk a holds
//     s_ext[8b + 16a + i + e] (row i, byte e), which depends on m = b + 2a
//     only.  So H_j is stored as distinct core matrices at m * 128 bytes and
//     described with SBO = 128 and LBO = 256: the MMA's core matrix (b, a)
//     lands on m = b + 2a.  The per-instance kernel (cpa5i.cuh) reads even
//     tiles of the sequence and needs 42 of them (5.25 KB per secret
//     polynomial); the persistent kernel (cpa_persist.cuh) keeps the earlier
//     layout of 62 (7.75 KB, kHankelCores) -- either instead of the 64 KB of
//     the dense matrix.
//   * B_j, persistent kernel: dense, core (8-column group c, K chunk a) at
//     a * (16 N) + c * 128; per-instance kernel: LayoutC there.
//
// Every product of an e4m3 digit (0..15) and an e4m3 secret (|s| <= 7) is an
// integer of magnitude <= 105, and every sum the MMA forms is an integer of
// magnitude <= 4 * 256 * 105 < 2^17, exact in f32.
#pragma once
#include <cstdint>

#include "kem_common.cuh"

namespace tmvp {

constexpr int kHankelCores = 62;                  // distinct core matrices of H_j
constexpr int kHankelBytes = kHankelCores * 128;  // per secret polynomial (7936 bytes)
constexpr int kUmmaM = 128;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Shared-memory matrix descriptor (tcgen05): start address, LBO and SBO in
// 16-byte units, descriptor version 1 (bits 46-48 = 0b001), no swizzle.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor for kind::f8f6f4: D f32, A and B e4m3, both
// K-major, M = 128, N = n.
__host__ __device__ constexpr uint32_t umma_idesc_e4m3(int n) {
  return (1u << 4)                      // D format f32
         | (0u << 7) | (0u << 10)       // A, B format e4m3
         | ((uint32_t)(n >> 3) << 17)   // N / 8
         | ((uint32_t)(kUmmaM >> 4) << 24);  // M / 16
}

__device__ __forceinline__ void umma_f8(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc,
                                        uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// The same issued by the threads with `issue` set: one of a warp that computes
// the operands together, so that the descriptors stay in uniform registers.
__device__ __forceinline__ void umma_f8_if(bool issue, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"((uint32_t)issue)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}

__device__ __forceinline__ void tmem_alloc(uint32_t dst_smem, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(dst_smem),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}

__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t mbar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(mbar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(mbar), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// try_wait with a suspend-time hint: the thread sleeps until the phase
// completes or about `ns` nanoseconds pass, instead of spinning.
__device__ __forceinline__ bool mbar_try_wait_sleep(uint32_t mbar, uint32_t parity, uint32_t ns) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok)
      : "r"(mbar), "r"(parity), "r"(ns)
      : "memory");
  return ok != 0;
}

// Bounded wait for phase `parity` of an mbarrier: sleeps in 20 us slices and
// gives up after about two seconds (or 2^22 polls), returning false.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t mbar, uint32_t parity) {
  if (mbar_try_wait_sleep(mbar, parity, 20000u)) return true;
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0; it < (1u << 22); it++) {
    if (mbar_try_wait_sleep(mbar, parity, 20000u)) return true;
    if ((it & 15u) == 15u && global_ns() - t0 > 2000000000ull) return false;
  }
  return false;
}

// The same by a whole warp, true in all its lanes or in none: lanes reach the
// bound at different polls, and what follows the wait (shuffles, tensor-memory
// loads) needs all of them.  Polled together: a vote after each lane's own loop
// made the one-key re-encryption 107.0 instead of 105.4 us (65536 Saber); the
// per-instance kernel, whose loop is not worth its registers there, takes that
// vote (decapsulation of 65536 Saber 1000 us, with this 1011).
__device__ __forceinline__ bool mbar_wait_warp(uint32_t mbar, uint32_t parity) {
  constexpr unsigned F = 0xffffffffu;
  if (__all_sync(F, mbar_try_wait_sleep(mbar, parity, 20000u))) return true;
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0; it < (1u << 22); it++) {
    if (__all_sync(F, mbar_try_wait_sleep(mbar, parity, 20000u))) return true;
    if (__any_sync(F, global_ns() - t0 > 2000000000ull)) return false;
  }
  return false;
}

// The same bound, polling without sleeping: for one thread whose wait is short
// and on whose wake-up others depend.
__device__ __forceinline__ bool mbar_spin_bounded(uint32_t mbar, uint32_t parity) {
  auto test = [&] {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok != 0;
  };
  for (int i = 0; i < 64; i++)
    if (test()) return true;
  const uint64_t t0 = global_ns();
  for (uint32_t it = 0; it < (1u << 28); it++) {
    if (test()) return true;
    if ((it & 1023u) == 1023u && global_ns() - t0 > 2000000000ull) return false;
  }
  return false;
}

// 16 consecutive f32 columns of this warp's 32 TMEM lanes.  The load and its
// completion wait are one asm statement, so no use of r[] can be scheduled
// between them.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// 8 consecutive f32 columns of this warp's 32 TMEM lanes (load and wait in
// one asm statement, as tmem_ld16).
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}

// 8, 16, 24 or 32 columns, one wait
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[8]) { tmem_ld8(taddr, r); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[16]) { tmem_ld16(taddr, r); }
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[24]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%24];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%25];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15]), "=&r"(r[16]), "=&r"(r[17]), "=&r"(r[18]), "=&r"(r[19]), "=&r"(r[20]), "=&r"(r[21]), "=&r"(r[22]), "=&r"(r[23])
      : "r"(taddr), "r"(taddr + 16)
      : "memory");
}
__device__ __forceinline__ void tmem_ld_cols(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%32];\n\t"
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%33];\n\t"
      "tcgen05.wait::ld.sync.aligned;"
      : "=&r"(r[0]), "=&r"(r[1]), "=&r"(r[2]), "=&r"(r[3]), "=&r"(r[4]), "=&r"(r[5]), "=&r"(r[6]), "=&r"(r[7]), "=&r"(r[8]), "=&r"(r[9]), "=&r"(r[10]), "=&r"(r[11]), "=&r"(r[12]), "=&r"(r[13]), "=&r"(r[14]), "=&r"(r[15]), "=&r"(r[16]), "=&r"(r[17]), "=&r"(r[18]), "=&r"(r[19]), "=&r"(r[20]), "=&r"(r[21]), "=&r"(r[22]), "=&r"(r[23]), "=&r"(r[24]), "=&r"(r[25]), "=&r"(r[26]), "=&r"(r[27]), "=&r"(r[28]), "=&r"(r[29]), "=&r"(r[30]), "=&r"(r[31])
      : "r"(taddr), "r"(taddr + 16)
      : "memory");
}

// Byte-wise e4m3 encoding of four digits 0..15 (one per byte).
constexpr uint32_t kE4m3Lo8 = 0x44403800u;  // 3, 2, 1, 0
constexpr uint32_t kE4m3Hi8 = 0x4E4C4A48u;  // 7, 6, 5, 4
__device__ __forceinline__ uint32_t e4m3_digits4(uint32_t d) {
  const uint32_t lo7 = d & 0x07070707u;
  const uint32_t hi = (d >> 3) & 0x01010101u;  // 1 where the digit is 8..15
  // PRMT selector nibbles from the low three bits of each byte
  const uint32_t u = (lo7 | (lo7 >> 4)) & 0x00FF00FFu;
  const uint32_t sel = (u | (u >> 8)) & 0xFFFFu;
  const uint32_t lut = __byte_perm(kE4m3Lo8, kE4m3Hi8, sel);  // e4m3 of 0..7
  const uint32_t big = lo7 | 0x50505050u;                      // e4m3 of 8..15
  const uint32_t m = hi * 0xFFu;
  return (big & m) | (lut & ~m);
}

// Radix-16 digits of a w-bit public coefficient x (results are needed mod
// 2^w): unsigned nibbles, except that a 5-bit top digit t = x >> (w - 5) is
// used as t - 32 when t >= 16.  That changes the product by a multiple of
// 2^w only, and keeps every digit within e4m3's exact integers (|d| <= 16):
// 13-bit coefficients need 3 digits instead of 4, 9-bit ones 2 instead of 3.
__host__ __device__ constexpr int r16_digits(int w) { return w <= 5 ? 1 : 1 + (w - 5 + 3) / 4; }

// e4m3 of four 5-bit top digits t (one per byte), each as the signed value
// t (t < 16) or t - 32 (t >= 16); magnitude 16 encodes as 0x58.
__device__ __forceinline__ uint32_t e4m3_sdigits4(uint32_t t) {
  const uint32_t m = ((t >> 4) & 0x01010101u) * 0xFFu;           // bytes with t >= 16
  const uint32_t mag = (m & (0x20202020u - t)) | (~m & t);       // 32 - t there (1..16), else t
  const uint32_t is16 = (mag >> 4) & 0x01010101u;
  return e4m3_digits4(mag & 0x0F0F0F0Fu) | (is16 * 0x58u) | (m & 0x80808080u);
}

// The encoded sequence s_ext[0..511] of each secret polynomial j < L, from
// its encoded words S (64 per polynomial, byte e of word u = coefficient
// 4u + e): s_ext[d] = -s[d + 1] for d < 255, s[d - 255] for 255 <= d <= 510,
// 0 at 511.  ext: 128 words per polynomial.  NEG negates four encoded bytes.
template <class NEG>
__device__ __forceinline__ void stage_ext(uint32_t *ext, const uint32_t *S, int L, int tid,
                                          int nthreads, NEG neg4f) {
  for (int idx = tid; idx < L * 128; idx += nthreads) {
    const int j = idx >> 7, w = idx & 127;
    const uint32_t *s = S + 64 * j;
    uint32_t v;
    if (w < 63) {
      v = neg4f(__byte_perm(s[w], s[w + 1], 0x4321));
    } else if (w == 63) {
      v = (neg4f(s[63]) >> 8) | (s[0] << 24);
    } else if (w < 127) {
      v = __byte_perm(s[w - 64], s[w - 63], 0x4321);
    } else {
      v = s[63] >> 8;
    }
    ext[idx] = v;
  }
}

// Shared-memory accesses through 32-bit shared-window addresses.
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared.b32 %0, [%1];" : "=r"(v) : "r"(a));
  return v;
}
__device__ __forceinline__ void sts32(uint32_t a, uint32_t x) {
  asm volatile("st.shared.b32 [%0], %1;" ::"r"(a), "r"(x) : "memory");
}
__device__ __forceinline__ void lds128(uint32_t a, uint32_t &x, uint32_t &y, uint32_t &z, uint32_t &w) {
  asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x), "=r"(y), "=r"(z), "=r"(w) : "r"(a));
}
__device__ __forceinline__ void sts64(uint32_t a, uint32_t x, uint32_t y) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(a), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t a, uint32_t x, uint32_t y, uint32_t z, uint32_t w) {
  asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(a), "r"(x), "r"(y), "r"(z), "r"(w) : "memory");
}

// The first `cores` Hankel core matrices of every j < L (H: cores * 128 bytes
// per polynomial):
// row i of core m is s_ext[8m + i .. 8m + i + 15], so row x = 8m + i sits at
// byte 16x.  Rows x = 4q + sh (q < 2 cores) with the same byte shift sh are
// windows of consecutive words.  Thread group g (four threads, sh = 0..3)
// makes the rows q = 2u + (g & 1) for a run of u, from a window of ext words
// that slides by two words per row; the eight threads of two neighbouring
// groups store eight consecutive rows (128 contiguous bytes) at a time.
__device__ __forceinline__ void stage_hankel(uint8_t *H, const uint32_t *ext, int L, int tid,
                                             int nthreads, int cores = kHankelCores) {
  const int pairs = nthreads >> 3;                 // group pairs
  const int run = (cores + pairs - 1) / pairs;      // rows per thread and polynomial
  const int sh = tid & 3, par = (tid >> 2) & 1, u0 = (tid >> 3) * run;
  const uint32_t sel = (uint32_t)(sh | ((sh + 1) << 4) | ((sh + 2) << 8) | ((sh + 3) << 12));
  if (u0 >= cores) return;
  for (int j = 0; j < L; j++) {
    const uint32_t *e = ext + 128 * j;
    uint8_t *hj = H + (size_t)j * cores * 128;
    int q = 2 * u0 + par;
    uint32_t w0 = e[q], w1 = e[q + 1], w2 = e[q + 2], w3 = e[q + 3], w4 = e[q + 4];
    for (int u = u0; u < u0 + run && u < cores; u++, q += 2) {
      *reinterpret_cast<uint4 *>(hj + 16 * (4 * q + sh)) =
          make_uint4(__byte_perm(w0, w1, sel), __byte_perm(w1, w2, sel), __byte_perm(w2, w3, sel),
                     __byte_perm(w3, w4, sel));
      if (u + 1 < u0 + run && u + 1 < cores) {
        w0 = w2; w1 = w3; w2 = w4;
        w3 = e[q + 5];
        w4 = e[q + 6];
      }
    }
  }
}

}  // namespace tmvp
