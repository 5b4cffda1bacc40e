// hash_kernels.cuh — the Keccak stages of the batched KEM: how a launch's
// sponges are spread over the GPU, and the launches.
#pragma once
#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "kem_common.cuh"

namespace tmvp {

// One SHAKE-128 expansion per instance: 32-byte seed at
// src + i*src_stride + src_off (8-byte aligned), out_bytes (multiple of 8)
// written to out + i*out_stride.  prehash: the seed is first replaced by
// SHAKE-128(seed)[0:32] and, if seed_out is set, stored there.
struct ShakeJob {
  const uint8_t *src;
  size_t src_stride, src_off;
  uint8_t *out;
  size_t out_stride;
  int out_bytes;
  int prehash;
  uint8_t *seed_out;
  size_t seed_out_stride, seed_out_off;
};

// The forms of a sponge: one thread, one warp, or two threads (hash_engine.cuh).
enum HashForm { kHashThread, kHashWarp, kHashPair };

// What a launch may use.  sms: SMs of the GPU.  The defaults let the planner
// choose per role; with `limits`, the caller's own (tmvp_ctx_set_warp_hash /
// _pair_hash), a launch of at most warp_max sponges runs one warp per sponge,
// else of at most pair_max two threads per sponge, else one thread (short
// sponges counting four times against the first and twice against the second).
// cap: most 128-thread blocks per SM of a decapsulation front whose sponges take
// one thread each; they stride over the plan's blocks, without the planner's own
// limits (0: those).  A split front is not capped: its first launch has one block
// per SM already (decapsulation of 20000 Saber: 362 us, capped at any of 2 to 8 in
// one launch 384 to 451).
constexpr size_t kWarpHashDefault = 1024, kPairHashDefault = 32768;
struct HashCfg {
  int sms;
  bool limits = false;
  size_t warp_max = kWarpHashDefault, pair_max = kPairHashDefault;
  int cap = 0;
  bool beside = false;  // the launch shares the GPU with others of its pass
  bool even = false;  // one role: its blocks limited to an even share per SM in every form
  bool one = false;  // never two launches (sponges_split)
};

// A launch's sponges: role r's sponges [first, first + count) in `form`, from
// block block0 on.  Blocks start in order, so segments go longest role first.
struct SpongeSeg {
  int role, form;
  unsigned block0, first, count;
};
struct SpongePlan {
  int nseg;
  unsigned blocks, threads, smem;  // threads: 128, or 32 with only the warp form
  SpongeSeg seg[8];
};
struct SpongeRole {
  size_t n;
  int perms;   // Keccak-f per sponge
  int id = 0;  // the stage's name for the role
  bool brief = false;  // G, the final key, the key-generation tail: counted several times against the caller's limits
};
constexpr unsigned kHashBlock = 128;
constexpr int kSpongeSmemMax = 117000;  // the most shared memory a plan asks for (one block per SM)
// One or two roles over the GPU: S[0] and S[1] (empty unless sponges_split),
// two launches that run side by side.
void plan_sponges(const HashCfg &cfg, const SpongeRole *roles, int nroles, SpongePlan (&S)[2]);
// Whether a launch of two roles over n instances becomes two: the two-role
// launches below put the second on s2 (which the caller forks from and joins
// to s).
bool sponges_split(const HashCfg &cfg, size_t n);

// Decapsulation front: GenMatrix from the seed of the pk embedded in sk, and
// H(c) (saber_dec, cuda_kernel.cu:383-384 and :447); with_gm = false: H(c) only.
cudaError_t launch_dec_front(const HashCfg &cfg, const KemParams &P, const uint8_t *sk, const uint8_t *ct,
                             uint8_t *a_stream, uint8_t *hc, size_t n, bool with_gm, cudaStream_t s,
                             cudaStream_t s2);
// kr = G(m' || H(pk)) and the GenSecret stream (saber_dec, cuda_kernel.cu:378-385).
cudaError_t launch_dec_g(const HashCfg &cfg, const KemParams &P, const uint8_t *mbuf, uint8_t *kr, uint8_t *s_stream,
                         size_t n, cudaStream_t s);
// K = H((fail ? z : kr[0:32]) || H(c)) (cuda_kernel.cu:185-186, :445-450);
// hc null: H(c) is made from ct; fail null: no selection; sk of instance i at
// sk + i * sk_stride (0: one key).
cudaError_t launch_final_key(const HashCfg &cfg, const KemParams &P, const uint8_t *ct, const uint8_t *hc,
                             const uint8_t *kr, const uint8_t *fail, const uint8_t *sk, size_t sk_stride, uint8_t *ss,
                             size_t n, cudaStream_t s);
// Encapsulation front (saber_enc, cuda_kernel.cu:116-127): m = H(coins), H(pk),
// kr = G(m || H(pk)), the GenSecret stream; with_gm: GenMatrix from pk's seed.
cudaError_t launch_enc_front(const HashCfg &cfg, const KemParams &P, const uint8_t *pk, const uint8_t *coins,
                             uint8_t *mbuf, uint8_t *kr, uint8_t *s_stream, uint8_t *a_stream, size_t n, bool with_gm,
                             cudaStream_t s, cudaStream_t s2);
// GenMatrix streams of n keys, seed_A at the end of pk + i * pk_stride.
cudaError_t launch_genmatrix(const HashCfg &cfg, const KemParams &P, const uint8_t *pk, size_t pk_stride,
                             uint8_t *a_stream, size_t n, cudaStream_t s);
// Two SHAKE-128 jobs over n instances.
cudaError_t launch_shake_jobs(const HashCfg &cfg, const ShakeJob &j0, const ShakeJob &j1, size_t n, cudaStream_t s,
                              cudaStream_t s2);
// Key-generation tail: sk[SK-64 : SK-32] = H(pk), sk[SK-32 : SK] = z.
cudaError_t launch_kp_final(const HashCfg &cfg, const KemParams &P, const uint8_t *pk, uint8_t *sk,
                            const uint8_t *coins, size_t n, cudaStream_t s);

// Mixed-parameter decapsulation: group g covers global instances
// [first, first + n) with its own parameters and buffers (device table).
struct HashGroup {
  KemParams P;
  int first, n;
  const uint8_t *sk, *ct;
  uint8_t *a_stream, *s_stream, *mbuf, *kr, *fail, *hc, *ss;
};
// perms: the roles' longest sponge among the groups.
cudaError_t launch_mix_front(const HashCfg &cfg, const HashGroup *T, int ng, size_t total, int gm_perms, int h_perms,
                             cudaStream_t s, cudaStream_t s2);
cudaError_t launch_mix_g(const HashCfg &cfg, const HashGroup *T, int ng, size_t total, int perms, cudaStream_t s);
cudaError_t launch_mix_final(const HashCfg &cfg, const HashGroup *T, int ng, size_t total, cudaStream_t s);

// dst[i * words + w] = src[w] for i < n (16-byte words)
__global__ void k_replicate16(uint4 *dst, const uint4 *src, int words, size_t n);

// Keccak-f of one GenMatrix / GenSecret / H(c) / H(pk) sponge.
inline int gm_perms(const KemParams &P) { return (P.gm_bytes + 167) / 168; }
inline int gs_perms(const KemParams &P) { return (P.gs_bytes + 167) / 168; }
inline int sha3_256_perms(int nbytes) { return nbytes / 136 + 1; }

}  // namespace tmvp
