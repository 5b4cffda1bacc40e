// cpa_f8u_onekey.cu — the one-key re-encryption as a matrix product
// (cpa_onekey.cuh): operand preparation and launches.
#include "cpa_onekey.cuh"

namespace tmvp {

namespace {

template <int SET>
int prep(const uint8_t *a_stream, const uint8_t *b_stream, uint8_t *ops, cudaStream_t s) {
  return (int)launch_chained(k_onekey_prep<SET>, OneKeyC<SET>::PLANES, 256, 0, s, a_stream, b_stream, ops);
}

template <int SET>
int reenc(OneKeyArgs a, int sms, cudaStream_t s) {
  using K = OneKeyC<SET>;
  a.units = (a.n + kOkRows - 1) / kOkRows * (K::C::L + 1);
  auto fn = k_onekey_reenc<SET>;
  const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, K::TOTAL);
  if (e != cudaSuccess) return (int)e;
  return (int)launch_chained(fn, a.units < sms ? a.units : sms, kOkThreads, K::TOTAL, s, a);
}

template <int SET>
int decrypt(OneKeyDecArgs a, uint8_t *planes, int sms, cudaStream_t s) {
  using K = OneKeyD<SET>;
  cudaError_t e = launch_chained(k_onekey_sprep<SET>, K::PLANES, 256, 0, s, a.sk, planes, a.err);
  if (e != cudaSuccess) return (int)e;
  const int rounds = (a.n + kOkRows * sms - 1) / (kOkRows * sms);
  a.rows = (a.n + sms * rounds - 1) / (sms * rounds);
  a.blocks = (a.n + a.rows - 1) / a.rows;
  a.planes = planes;
  auto fn = k_onekey_decrypt<SET>;
  if ((e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, K::TOTAL)) != cudaSuccess)
    return (int)e;
  return (int)launch_chained(fn, a.blocks < sms ? a.blocks : sms, kOkDecThreads, K::TOTAL, s, a);
}

}  // namespace

#define TMVP_OK_SETS(X) \
  switch (P.set) {      \
    case 0: return X(0); \
    case 1: return X(1); \
    case 2: return X(2); \
    case 3: return X(3); \
    case 4: return X(4); \
    case 5: return X(5); \
  }

size_t onekey_operand_bytes(const KemParams &P) {
#define TMVP_OK_BYTES(S) (size_t) OneKeyC<S>::OPS
  TMVP_OK_SETS(TMVP_OK_BYTES)
  return 0;
}

int onekey_prep(const KemParams &P, const uint8_t *a_stream, const uint8_t *b_stream, uint8_t *ops, void *s) {
#define TMVP_OK_PREP(S) prep<S>(a_stream, b_stream, ops, (cudaStream_t)s)
  TMVP_OK_SETS(TMVP_OK_PREP)
  return (int)cudaErrorInvalidValue;
}

int onekey_reenc(const CpaArgs &b, const uint8_t *ops, int sms, void *s) {
  const KemParams &P = b.P;
  OneKeyArgs a{};
  a.ops = ops;
  a.s_stream = b.s_stream;
  a.ct = b.ct;
  a.msg = b.msg;
  a.fail = b.fail;
  a.err = b.err;
  a.n = b.n;
#define TMVP_OK_REENC(S) reenc<S>(a, sms, (cudaStream_t)s)
  TMVP_OK_SETS(TMVP_OK_REENC)
  return (int)cudaErrorInvalidValue;
}

size_t onekey_secret_bytes(const KemParams &P) { return (size_t)(2 * P.l * kOkHankel); }

int onekey_decrypt(const CpaArgs &b, uint8_t *planes, int sms, void *s) {
  const KemParams &P = b.P;
  OneKeyDecArgs a{};
  a.ct = b.ct;
  a.sk = b.sk;
  a.m_out = b.m_out;
  a.err = b.err;
  a.n = b.n;
#define TMVP_OK_DEC(S) decrypt<S>(a, planes, sms, (cudaStream_t)s)
  TMVP_OK_SETS(TMVP_OK_DEC)
  return (int)cudaErrorInvalidValue;
}

}  // namespace tmvp
