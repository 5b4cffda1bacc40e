// hash_kernels.cu — the Keccak stages of the batched KEM, each written once
// for the three forms of a sponge (hash_engine.cuh), and the planner that
// spreads a launch's sponges over the GPU.
//
// Replaces the reference's single-block hash kernels and its 25-lane
// shake128_gpu (TMVP-Saber/SABER-GPU/src/poly.cu:918-1114,
// TMVP_SABLE/src/fips202.cu:409-668), which cap the batch at 1024 and rely
// on implicit warp synchrony.
#include "hash_kernels.cuh"

#include <algorithm>

#include "chain.cuh"
#include "hash_engine.cuh"

namespace tmvp {

namespace {

// ---- the stages: run<E>(e, role, i) makes sponge i of a role ---------------

struct GenMatrix {
  KemParams P;
  const uint8_t *pk;
  size_t pk_stride;
  uint8_t *a_stream;
  template <class E>
  __device__ __forceinline__ void run(const E &e, int, size_t i) const {
    const auto seed = e.load(pk + i * pk_stride + (size_t)P.l * P.polycompbytes, 4);
    e.shake128(seed, a_stream + i * P.gm_bytes, P.gm_bytes);
  }
};

template <class E>
__device__ __forceinline__ void dec_hash_ct(const E &e, const KemParams &P, const uint8_t *ct, uint8_t *hc, size_t i) {
  e.store(hc + i * 32, e.sha3_256_mem(ct + i * P.ct_bytes, P.ct_bytes), 4);
}

template <class E>
__device__ __forceinline__ void dec_genmatrix(const E &e, const KemParams &P, const uint8_t *sk, uint8_t *a_stream,
                                              size_t i) {
  const auto seed = e.load(sk + i * P.sk_bytes + P.indcpa_sk_bytes + (size_t)P.l * P.polycompbytes, 4);
  e.shake128(seed, a_stream + i * P.gm_bytes, P.gm_bytes);
}

template <class E>
__device__ __forceinline__ void dec_g_one(const E &e, const KemParams &P, const uint8_t *mbuf, uint8_t *kr,
                                          uint8_t *s_stream, size_t i) {
  const auto g = e.sha3_512_64(e.load(mbuf + i * 64, 8));
  e.store(kr + i * 64, g, 8);
  e.shake128(e.hi4(g), s_stream + i * P.gs_bytes, P.gs_bytes);
}

template <class E>
__device__ __forceinline__ void final_key_one(const E &e, const KemParams &P, const uint8_t *ct, const uint8_t *hc,
                                              const uint8_t *kr, const uint8_t *fail, const uint8_t *sk,
                                              size_t sk_stride, uint8_t *ss, size_t i) {
  auto k = e.load(kr + i * 64, 4);
  if (fail) k = e.sel4(k, e.load(sk + i * sk_stride + P.sk_bytes - 32, 4), fail[i] != 0);
  const auto h = hc ? e.load(hc + i * 32, 4) : e.sha3_256_mem(ct + i * P.ct_bytes, P.ct_bytes);
  e.store(ss + i * 32, e.template sha3_256<8>(e.cat4(k, h)), 4);
}

struct DecFront {  // role 0: GenMatrix, role 1: H(c)
  KemParams P;
  const uint8_t *sk, *ct;
  uint8_t *a_stream, *hc;
  template <class E>
  __device__ __forceinline__ void run(const E &e, int role, size_t i) const {
    if (role == 0) dec_genmatrix(e, P, sk, a_stream, i);
    else dec_hash_ct(e, P, ct, hc, i);
  }
};

struct DecG {
  KemParams P;
  const uint8_t *mbuf;
  uint8_t *kr, *s_stream;
  template <class E>
  __device__ __forceinline__ void run(const E &e, int, size_t i) const {
    dec_g_one(e, P, mbuf, kr, s_stream, i);
  }
};

struct FinalKey {
  KemParams P;
  const uint8_t *ct, *hc, *kr, *fail, *sk;
  size_t sk_stride;
  uint8_t *ss;
  template <class E>
  __device__ __forceinline__ void run(const E &e, int, size_t i) const {
    final_key_one(e, P, ct, hc, kr, fail, sk, sk_stride, ss, i);
  }
};

struct EncFront {  // role 0: GenMatrix, role 1: the chain to the GenSecret stream
  KemParams P;
  const uint8_t *pk, *coins;
  uint8_t *mbuf, *kr, *s_stream, *a_stream;
  template <class E>
  __device__ __forceinline__ void run(const E &e, int role, size_t i) const {
    if (role == 0) {
      const auto seed = e.load(pk + i * P.pk_bytes + (size_t)P.l * P.polycompbytes, 4);
      e.shake128(seed, a_stream + i * P.gm_bytes, P.gm_bytes);
      return;
    }
    const auto m = e.template sha3_256<4>(e.load(coins + i * 32, 4));
    const auto buf = e.cat4(m, e.sha3_256_mem(pk + i * P.pk_bytes, P.pk_bytes));
    e.store(mbuf + i * 64, buf, 8);
    const auto g = e.sha3_512_64(buf);
    e.store(kr + i * 64, g, 8);
    e.shake128(e.hi4(g), s_stream + i * P.gs_bytes, P.gs_bytes);
  }
};

struct ShakeJobs {
  ShakeJob j[2];
  template <class E>
  __device__ __forceinline__ void run(const E &e, int role, size_t i) const {
    const ShakeJob &J = j[role];
    auto seed = e.load(J.src + i * J.src_stride + J.src_off, 4);
    if (J.prehash) {  // seed_A <- SHAKE-128(seed_A)[0:32] (Saber round-3 key generation)
      seed = e.shake128_first(seed);
      if (J.seed_out) e.store(J.seed_out + i * J.seed_out_stride + J.seed_out_off, seed, 4);
    }
    e.shake128(seed, J.out + i * J.out_stride, J.out_bytes);
  }
};

struct KpFinal {
  KemParams P;
  const uint8_t *pk;
  uint8_t *sk;
  const uint8_t *coins;
  template <class E>
  __device__ __forceinline__ void run(const E &e, int, size_t i) const {
    const auto h = e.sha3_256_mem(pk + i * P.pk_bytes, P.pk_bytes);
    e.store(sk + i * P.sk_bytes + P.sk_bytes - 64, e.cat4(h, e.load(coins + i * 96 + 64, 4)), 8);
  }
};

// Mixed-parameter stages: global sponge gi belongs to the group whose range
// holds it.
struct MixBase {
  const HashGroup *T;
  int ng;
  __device__ __forceinline__ const HashGroup &group(size_t gi) const {
    int lo = 0, hi = ng - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((int)gi >= T[mid].first) lo = mid;
      else hi = mid - 1;
    }
    return T[lo];
  }
};
struct MixFront : MixBase {
  template <class E>
  __device__ __forceinline__ void run(const E &e, int role, size_t gi) const {
    const HashGroup &G = group(gi);
    const size_t i = gi - (size_t)G.first;
    if (role == 0) dec_genmatrix(e, G.P, G.sk, G.a_stream, i);
    else dec_hash_ct(e, G.P, G.ct, G.hc, i);
  }
};
struct MixG : MixBase {
  template <class E>
  __device__ __forceinline__ void run(const E &e, int, size_t gi) const {
    const HashGroup &G = group(gi);
    dec_g_one(e, G.P, G.mbuf, G.kr, G.s_stream, gi - (size_t)G.first);
  }
};
struct MixFinal : MixBase {
  template <class E>
  __device__ __forceinline__ void run(const E &e, int, size_t gi) const {
    const HashGroup &G = group(gi);
    final_key_one(e, G.P, G.ct, G.hc, G.kr, G.fail, G.sk, (size_t)G.P.sk_bytes, G.ss, gi - (size_t)G.first);
  }
};

// Blocks of 128 threads, one warp on each of an SM's four sub-partitions; of
// one warp in a launch that has only the warp form (few sponges then spread
// over all SMs: four on one SM share its shuffle unit, 51.2 against 49.2 us
// for 17 LightSaber encapsulations).
// The segment, form and role depend on the block alone.  Past the end of a
// segment the pair and warp forms repeat its last sponge (their shuffles need
// every thread) and store nothing.
template <class R>
__device__ __forceinline__ void sponge_block(const SpongePlan &S, const R &r, const unsigned block) {
  int k = 0;
  while (k + 1 < S.nseg && block >= S.seg[k + 1].block0) k++;
  const unsigned b = block - S.seg[k].block0, count = S.seg[k].count, first = S.seg[k].first;
  const int role = S.seg[k].role;
  switch (S.seg[k].form) {
    case kHashThread: {
      const unsigned i = b * kHashBlock + threadIdx.x;
      if (i < count) r.run(ThreadSponge{}, role, first + i);
      break;
    }
    case kHashPair: {
      const unsigned i = b * (kHashBlock / 2) + (threadIdx.x >> 1);
      const bool live = i < count;
      r.run(PairSponge{(int)(threadIdx.x & 1), live}, role, first + (live ? i : count - 1));
      break;
    }
    default: {
      const int lane = (int)(threadIdx.x & 31);
      const unsigned i = b * (blockDim.x >> 5) + (threadIdx.x >> 5);
      const bool live = i < count;
      r.run(WarpSponge{lane, live, warp_keccak_lane(lane)}, role, first + (live ? i : count - 1));
    }
  }
}

template <class R>
__global__ void __launch_bounds__(kHashBlock) k_sponges(const __grid_constant__ SpongePlan S,
                                                        const __grid_constant__ R r) {
  chain_wait();
  sponge_block(S, r, blockIdx.x);
}

// The same by fewer blocks than the plan has, each taking every gridDim.x-th of
// them: a capped front holds neither threads nor shared memory beyond its blocks.
template <class R>
__global__ void __launch_bounds__(kHashBlock) k_sponges_strided(const __grid_constant__ SpongePlan S,
                                                                const __grid_constant__ R r) {
  chain_wait();
  for (unsigned b = blockIdx.x; b < S.blocks; b += gridDim.x) sponge_block(S, r, b);
}

unsigned per_block(int form) {
  return form == kHashThread ? kHashBlock : (form == kHashPair ? kHashBlock / 2 : kHashBlock / 32);
}

template <class R>
cudaError_t launch_sponges(const SpongePlan &S, const R &r, cudaStream_t s) {
  if (S.blocks == 0) return cudaSuccess;
  auto fn = k_sponges<R>;
  if (S.smem > 48 * 1024) {
    // always the largest limit: the attribute is the function's, so a smaller one set by
    // another thread's context would refuse a launch of this one
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, kSpongeSmemMax);
    if (e != cudaSuccess) return e;
  }
  return launch_chained(fn, S.blocks, S.threads, S.smem, s, S, r);
}

template <class R>
cudaError_t launch_sponges(const HashCfg &cfg, const SpongeRole *roles, int nroles, const R &r, cudaStream_t s,
                           cudaStream_t s2) {
  SpongePlan S[2];
  plan_sponges(cfg, roles, nroles, S);
  for (SpongePlan &T : S) {
    bool warp_only = true;
    for (int k = 0; k < T.nseg; k++) warp_only = warp_only && T.seg[k].form == kHashWarp;
    T.threads = warp_only ? 32 : kHashBlock;
    if (warp_only) {
      T.blocks = 0;
      for (int k = 0; k < T.nseg; k++) {
        T.seg[k].block0 = T.blocks;
        T.blocks += T.seg[k].count;
      }
    }
  }
  const cudaError_t e = launch_sponges(S[0], r, s);
  return e != cudaSuccess ? e : launch_sponges(S[1], r, s2);
}

}  // namespace

// Adds role r's sponges [first, first + count) in `form` to S.
static void add_seg(SpongePlan &S, int role, int form, size_t first, size_t count) {
  if (!count) return;
  S.seg[S.nseg++] = SpongeSeg{role, form, S.blocks, (unsigned)first, (unsigned)count};
  S.blocks += (unsigned)((count + per_block(form) - 1) / per_block(form));
}

// Shared memory that leaves room for at most `blocks` blocks per SM (228 KB,
// 1 KB of it per block reserved).
static unsigned smem_limit(int blocks) {
  return blocks <= 1 ? (unsigned)kSpongeSmemMax : (unsigned)(227 * 1024 / (blocks + 1));
}

// Two thread-form roles below one round, n1 sponges of p1 permutations and n2 of
// p2 <= p1, one block resident per SM: how many of the n2 run in the thread form.
// The SMs without a block of the first role make whole rounds of the second
// until those end; what is left then takes a whole block's time, or, two threads
// a sponge, half the sponges of a block in two thirds of it.  Times in
// permutations of a thread-form block (4.7 us; 5.2 where it absorbs, two threads
// 3.5 there): encapsulation of 9800 Saber 242 -> 221 us, of 14000 300 -> 279, key
// generation of 16384 263 -> 252.
static size_t thread_part(int sms, size_t n1, int p1, size_t n2, int p2) {
  const int b1 = (int)((n1 + kHashBlock - 1) / kHashBlock), b2 = (int)((n2 + kHashBlock - 1) / kHashBlock), f = sms - b1;
  if (f <= 0) return n2;
  const double t1 = p1, t2 = 1.1 * p2, tp = 0.74 * p2;
  const int d = (int)(t1 / t2), left = b2 - d * f;
  if (d < 1 || left <= 0) return n2;
  const double thread = left <= f ? std::max(t1, (d + 1) * t2) : t1 + t2;
  const int e = (int)((t1 - d * t2) / tp), p = 2 * left - e * f;
  const double pair = p <= f ? std::max(t1, d * t2 + (e + 1) * tp) : t1 + ((p + sms - 1) / sms) * tp;
  return pair < thread ? (size_t)(d * f) * kHashBlock : n2;
}

bool sponges_split(const HashCfg &cfg, size_t n) {
  return !cfg.limits && !cfg.one && n >= (size_t)128 * cfg.sms && n < (size_t)192 * cfg.sms;
}

// Why the lines lie where they do (152 SMs, 608 sub-partitions; a sponge of 23
// permutations):
//  * A permutation's 4300 integer instructions fill a sub-partition's integer
//    pipe from one thread-form warp on (92% of it; 99% from two), so a launch
//    takes as long as its fullest sub-partition: 109 us per thread-form warp
//    there.  128-thread blocks put one warp on each of an SM's four; with
//    64-thread blocks, 16384 x (23 + 9) permutations took 209 us, with 128 147.
//  * One warp a sponge takes 47 us up to about 2.75 sponges a sub-partition,
//    two threads a sponge 67 us up to 16, one thread 109 us up to 32: the
//    forms' lines.  Past whole rounds of 32, the rest goes the same way beside
//    them: 20011 sponges in 122 us instead of 206.
//    Beside one round of a single role the warp form pays below one sponge a
//    sub-partition, beside two up to two: GenMatrix of 19456 + 600 Saber keys 145
//    us (rest in pairs 167), + 700 240 (167), of 38912 + 1216 258 (265), + 1300 291
//    (264), of three rounds + 1300 363 (362).
//    A one-role launch that shares the GPU (G, H(c) alone) leaves the warp form,
//    which issues five times the instructions, at 1.5: decapsulation of 1000
//    Saber 83 -> 77 us, of 1600 107 -> 91, of 1200 FireSaber 144 -> 134, of 1600
//    with cached A 70 -> 54.  The shorter role of a front beside the decryption
//    does so at 2 in all: decapsulation of 800 Saber 87 -> 78 us, FireSaber 125
//    -> 113, LightSaber 54 -> 46.
//  * Two roles side by side: longest first, and few blocks resident, so that
//    an SM that finishes early takes the next block instead of all being
//    placed at the start: with one block per SM 16384 x (23 + 9) takes 135
//    us; with two per SM 32768 345 -> 266 and 65536 530 -> 502 (one: 272, 517).
//  * One role over several rounds: as many blocks resident per SM as rounds, so
//    that none gets one more while a neighbour has one less (a grid's first
//    152 blocks land on 148 SMs); the rest in a finer form then starts behind
//    them.  65536 x 10 permutations 185 -> 166 us, x 8 154 -> 136, x 6 113 ->
//    107, and a pass of two chains leaves room for the other one's kernels
//    (decapsulation of 65536 Saber 1037 -> 1015, of 38912 659 -> 634).  Not
//    with one round and a finer rest (20011 x 10: 70 -> 78) and not for a
//    single permutation (25 -> 27).
//  * Just above one round (up to 1.5) the longer role's thread-form blocks run
//    alone at one per SM and the rest as a second launch beside them: as one
//    launch, four SMs get two of those blocks (key generation of 20011: 386 us,
//    as two 324).
//  * cfg.even: beside a kernel whose blocks take most of an SM each, blocks that
//    fit anywhere pile up on the SMs it left or finished first; limited to an
//    even share each, the one-key pass of 8192 takes 96 instead of 157 us, of
//    20000 162 instead of 253.
void plan_sponges(const HashCfg &cfg, const SpongeRole *roles, int nroles, SpongePlan (&S)[2]) {
  S[0] = SpongePlan{};
  S[1] = SpongePlan{};
  int order[2] = {0, 1};
  if (nroles == 2 && roles[1].perms > roles[0].perms) std::swap(order[0], order[1]);  // longest first
  if (cfg.limits) {
    size_t total = 0;
    for (int r = 0; r < nroles; r++) total += roles[r].n;
    const bool short_sponges = roles[0].brief;
    const int form = (short_sponges ? 4 * total : total) <= cfg.warp_max   ? kHashWarp
                     : (short_sponges ? 2 * total : total) <= cfg.pair_max ? kHashPair
                                                                           : kHashThread;
    for (int k = 0; k < nroles; k++) add_seg(S[0], roles[order[k]].id, form, 0, roles[order[k]].n);
    return;
  }
  const size_t W = 4 * (size_t)cfg.sms;  // sub-partitions
  const bool split = nroles == 2 && sponges_split(cfg, roles[order[0]].n);
  size_t warps = 0;  // sponges in the warp form so far
  for (int k = 0; k < nroles; k++) {
    const SpongeRole &r = roles[order[k]];
    const size_t full = r.n / (32 * W) * (32 * W), rest = r.n - full;
    int form = kHashThread;
    const bool slack = cfg.beside && k == 1 && 5 * r.perms <= 3 * roles[order[0]].perms;  // ends first in either form
    const size_t rounds = full / (32 * W);
    const size_t above = nroles == 2 || rounds > 2 ? 9 * W / 4 : (rounds == 2 ? 2 * W : W - 1);
    const size_t line = full ? above : (slack ? 2 * W : (cfg.beside && nroles == 1 ? 3 * W / 2 : 11 * W / 4));
    if (warps + rest <= line) form = kHashWarp;
    else if (rest <= 16 * W) form = kHashPair;
    if (form == kHashWarp) warps += rest;
    add_seg(S[split && k == 1], r.id, kHashThread, 0, full);
    size_t fit = rest;
    if (k == 1 && form == kHashThread && !full && cfg.cap == 0 && roles[order[0]].n < 32 * W)
      fit = thread_part(cfg.sms, roles[order[0]].n, roles[order[0]].perms, rest, r.perms);
    add_seg(S[split && (k == 1 || form != kHashThread)], r.id, form, full, fit);
    add_seg(S[split && k == 1], r.id, kHashPair, full + fit, rest - fit);
    if (nroles == 1) {
      // blocks per SM when every SM has its share
      const int q = (int)rounds + (form == kHashThread && rest ? 1 : 0);
      if (r.perms >= 4 && q <= 5 && (form == kHashThread || rest == 0 || q >= 2)) S[0].smem = smem_limit(q);
      else if (cfg.even) S[0].smem = smem_limit((int)((S[0].blocks + cfg.sms - 1) / cfg.sms));
    }
    if (nroles == 2 && k == 0 && (cfg.cap == 0 || split) && (full || form == kHashThread))
      S[0].smem = smem_limit(full && !split ? 2 : 1);
  }
}

cudaError_t launch_dec_front(const HashCfg &cfg, const KemParams &P, const uint8_t *sk, const uint8_t *ct,
                             uint8_t *a_stream, uint8_t *hc, size_t n, bool with_gm, cudaStream_t s, cudaStream_t s2) {
  const SpongeRole roles[2] = {{n, gm_perms(P), 0}, {n, sha3_256_perms(P.ct_bytes), 1}};
  if (cfg.cap > 0 && with_gm && !sponges_split(cfg, n)) {  // one launch, no limit but the cap on its blocks
    SpongePlan S[2];
    plan_sponges(cfg, roles, 2, S);
    const unsigned most = (unsigned)(cfg.cap * cfg.sms);
    if (S[0].seg[0].form == kHashThread && S[0].blocks > most)
      return launch_chained(k_sponges_strided<DecFront>, most, kHashBlock, 0, s, S[0], DecFront{P, sk, ct, a_stream, hc});
  }
  return launch_sponges(cfg, with_gm ? roles : roles + 1, with_gm ? 2 : 1, DecFront{P, sk, ct, a_stream, hc}, s, s2);
}

cudaError_t launch_dec_g(const HashCfg &cfg, const KemParams &P, const uint8_t *mbuf, uint8_t *kr, uint8_t *s_stream,
                         size_t n, cudaStream_t s) {
  const SpongeRole role{n, 1 + gs_perms(P), 0, true};
  return launch_sponges(cfg, &role, 1, DecG{P, mbuf, kr, s_stream}, s, s);
}

cudaError_t launch_final_key(const HashCfg &cfg, const KemParams &P, const uint8_t *ct, const uint8_t *hc,
                             const uint8_t *kr, const uint8_t *fail, const uint8_t *sk, size_t sk_stride, uint8_t *ss,
                             size_t n, cudaStream_t s) {
  const SpongeRole role{n, 1 + (hc ? 0 : sha3_256_perms(P.ct_bytes)), 0, true};
  return launch_sponges(cfg, &role, 1, FinalKey{P, ct, hc, kr, fail, sk, sk_stride, ss}, s, s);
}

cudaError_t launch_enc_front(const HashCfg &cfg, const KemParams &P, const uint8_t *pk, const uint8_t *coins,
                             uint8_t *mbuf, uint8_t *kr, uint8_t *s_stream, uint8_t *a_stream, size_t n, bool with_gm,
                             cudaStream_t s, cudaStream_t s2) {
  const SpongeRole roles[2] = {{n, gm_perms(P), 0}, {n, 2 + sha3_256_perms(P.pk_bytes) + gs_perms(P), 1}};
  return launch_sponges(cfg, with_gm ? roles : roles + 1, with_gm ? 2 : 1, EncFront{P, pk, coins, mbuf, kr, s_stream, a_stream}, s, s2);
}

cudaError_t launch_genmatrix(const HashCfg &cfg, const KemParams &P, const uint8_t *pk, size_t pk_stride,
                             uint8_t *a_stream, size_t n, cudaStream_t s) {
  const SpongeRole role{n, gm_perms(P)};
  return launch_sponges(cfg, &role, 1, GenMatrix{P, pk, pk_stride, a_stream}, s, s);
}

cudaError_t launch_shake_jobs(const HashCfg &cfg, const ShakeJob &j0, const ShakeJob &j1, size_t n, cudaStream_t s,
                              cudaStream_t s2) {
  const SpongeRole roles[2] = {{n, (j0.out_bytes + 167) / 168 + j0.prehash, 0},
                               {n, (j1.out_bytes + 167) / 168 + j1.prehash, 1}};
  return launch_sponges(cfg, roles, 2, ShakeJobs{{j0, j1}}, s, s2);
}

cudaError_t launch_kp_final(const HashCfg &cfg, const KemParams &P, const uint8_t *pk, uint8_t *sk,
                            const uint8_t *coins, size_t n, cudaStream_t s) {
  const SpongeRole role{n, sha3_256_perms(P.pk_bytes), 0, true};
  return launch_sponges(cfg, &role, 1, KpFinal{P, pk, sk, coins}, s, s);
}

cudaError_t launch_mix_front(const HashCfg &cfg, const HashGroup *T, int ng, size_t total, int gm, int h,
                             cudaStream_t s, cudaStream_t s2) {
  const SpongeRole roles[2] = {{total, gm, 0}, {total, h, 1}};
  MixFront r;
  r.T = T;
  r.ng = ng;
  return launch_sponges(cfg, roles, 2, r, s, s2);
}

cudaError_t launch_mix_g(const HashCfg &cfg, const HashGroup *T, int ng, size_t total, int perms, cudaStream_t s) {
  const SpongeRole role{total, perms, 0, true};
  MixG r;
  r.T = T;
  r.ng = ng;
  return launch_sponges(cfg, &role, 1, r, s, s);
}

cudaError_t launch_mix_final(const HashCfg &cfg, const HashGroup *T, int ng, size_t total, cudaStream_t s) {
  const SpongeRole role{total, 1, 0, true};
  MixFinal r;
  r.T = T;
  r.ng = ng;
  return launch_sponges(cfg, &role, 1, r, s, s);
}

// dst[i * words + w] = src[w] for i < n (16-byte words): one key's bytes and
// its expanded A repeated per instance, for the one-key decapsulation.  Blocks
// take instances, threads the words of one (coalesced stores; the source
// stays in L1).
__global__ void __launch_bounds__(256) k_replicate16(uint4 *dst, const uint4 *src, int words, size_t n) {
  for (size_t i = blockIdx.x; i < n; i += gridDim.x) {
    uint4 *d = dst + i * (size_t)words;
    for (int w = threadIdx.x; w < words; w += blockDim.x) d[w] = src[w];
  }
}

}  // namespace tmvp
