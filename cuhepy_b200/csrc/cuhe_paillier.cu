// C ABI of the Paillier / Paillier-Lookup path (see include/cuhe_paillier.h).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/cuhe_paillier.h"
#include "host_bigint.h"
#include "paillier_kernels.cuh"
#include "split_kernels.cuh"

using cuhe::host::Limbs;

// Scratch of cuhe_paillier_decode_hamming_static: one popcount per ciphertext
// chunk.  Host code must not pass this name to a kernel (on the host it is a
// stand-in, not a device address); the device address is looked up per device.
static __device__ __align__(256) uint32_t g_static_decode_counts[CUHE_STATIC_DECODE_MAX_CHUNKS];

namespace {

std::string g_create_error;

struct Variant {
  int K, TPI, W;
};

// (K, TPI, W) combinations compiled into the library.
#define CUHE_VARIANTS(X) \
  X(64, 8, 3)            \
  X(64, 8, 4)            \
  X(64, 16, 4)           \
  X(128, 8, 4)           \
  X(128, 16, 3)          \
  X(128, 16, 4)          \
  X(128, 16, 5)          \
  X(128, 32, 3)          \
  X(128, 32, 4)          \
  X(256, 16, 4)          \
  X(256, 32, 3)          \
  X(256, 32, 4)          \
  X(256, 32, 5)

struct DeviceBuffer {
  void* ptr = nullptr;
  size_t bytes = 0;
  cudaError_t reserve(size_t need) {
    if (need <= bytes) return cudaSuccess;
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
    size_t grow = std::max(need, size_t(1) << 20);
    cudaError_t e = cudaMalloc(&ptr, grow);
    if (e == cudaSuccess) bytes = grow;
    return e;
  }
  void release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
  }
};

bool is_device_pointer(const void* p) {
  if (!p) return false;
  cudaPointerAttributes attr;
  if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return attr.type == cudaMemoryTypeDevice || attr.type == cudaMemoryTypeManaged;
}

}  // namespace

struct cuhe_paillier {
  int device = 0;
  int sms = 1;  // multiprocessors of the device
  int smem_limit = 48 << 10;  // dynamic shared memory a block may ask for beside 1 KB of static
  int K = 0;
  int n_words = 0;
  int tpi = 0, window = 0;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  uint32_t* d_consts = nullptr;
  int* d_status = nullptr;
  cuhe::KeyScalars ks{};
  Limbs n, n2;
  Limbs secret_exp;  // empty until set
  Limbs secret_mult;
  bool have_secret = false;
  int32_t* d_ops_n = nullptr;
  int nops_n = 0;
  int32_t* d_ops_sec = nullptr;
  int nops_sec = 0;
  int32_t* d_ops_sec52 = nullptr;  // the secret exponent's schedule for the FP64-pipe kernel's window
  int nops_sec52 = 0;
  uint32_t* d_crt = nullptr;  // CRT constant block, present once the factors are installed
  double* d_crt52 = nullptr;  // per side: the constants mod p, q of k_pair_crt (pair_const_doubles)
  double* d_pair = nullptr;   // the constants mod n of k_pair_modexp
  unsigned long long pair_ninv = 0;  // -n^-1 mod 2^52
  double* d_n52 = nullptr;    // n^2 as 52-bit limbs, then R52 R mod n^2 in words
  unsigned long long ninv52 = 0;  // -(n^2)^-1 mod 2^52
  int32_t* d_ops_n52 = nullptr;   // the schedule of n for k_pair_modexp's window
  int nops_n52 = 0;
  // each side's exponent in k_pair_crt: the secret's, or p - 1 and its cofactor
  struct SideExponent {
    int32_t* d_ops = nullptr;
    int32_t* d_fall = nullptr;
    int nops = 0, nfall = 0, halved = 0;
    size_t room = 0;  // ops that each array holds
    cuhe::PairExponent get() const { return {d_ops, d_fall, nops, nfall, halved}; }
  } side_exp[2];
  Limbs factor[2];  // p, q once installed
  cuhe::CrtScalars cs{};
  bool have_factors = false;
  bool fp64 = true;           // exponentiations, server products and table encryption on the FP64 pipe
  bool fp64_small = false;    // server products also for n^2 of 2048 bits (set_fp64(ctx, 2))
  uint32_t* d_gtab = nullptr;
  int message_chunks = 0;
  uint32_t* d_wide = nullptr;  // 16-bit-digit table W[j][D], built on demand (see cuhe_lookup_set_wide_table)
  // The tables as rows of limb pairs mod n (FP64-pipe encryption), built from
  // the installed ones when a call first needs them and dropped with them.
  struct PairTables {
    double2* digits = nullptr;  // [message_chunks][256]: the 8-bit table
    double2* embed = nullptr;   // [ceil(message_chunks / 2)][256]: 8 embedding bits (16 plaintext bits)
    double2* noise = nullptr;   // [noise_entries]
    double2* noise2 = nullptr;  // [noise_entries][noise_entries]: products of two
    double2* wide_digits = nullptr;  // [ceil(message_chunks / 2)][65536]: 16-bit digits
    // Rows of 65,536 entries by 16 embedding bits, as far as calls reached.
    // Rows are added and never moved, nor is the device array of their
    // addresses: calls captured in a graph read both at every replay.
    std::vector<double2*> wide_blocks;      // each growth's allocation
    const double2** embed_rows = nullptr;   // [ceil(message_chunks / 4)], wide_rows of them set
    int wide_rows = 0;
    void release() {
      for (double2** p : {&digits, &embed, &noise}) {
        cudaFree(*p);
        *p = nullptr;
      }
      release_wide();
    }
    void release_wide() {
      cudaFree(noise2);
      cudaFree(wide_digits);
      noise2 = wide_digits = nullptr;
      for (double2* block : wide_blocks) cudaFree(block);
      wide_blocks.clear();
      cudaFree(embed_rows);
      embed_rows = nullptr;
      wide_rows = 0;
    }
    bool wide() const { return wide_digits || wide_rows; }
  } pt;
  double2* d_entry = nullptr;  // k_pair_rows' constants
  int wide_mode = 1;           // 0 never, 1 for large batches when it fits, 2 always
  uint32_t* d_noise = nullptr;
  int noise_entries = 0;
  DeviceBuffer work;
  DeviceBuffer tmp_ops;
  cudaStream_t copy = nullptr;  // host-buffer pipelines: transfers beside the compute
  cudaStream_t side = nullptr;  // and a second compute stream (created on first use)
  std::string error;
  std::mutex mu;
};

namespace {

int fail(cuhe_paillier* ctx, int code, const std::string& msg) {
  if (ctx) ctx->error = msg; else g_create_error = msg;
  return code;
}

int cuda_fail(cuhe_paillier* ctx, cudaError_t e, const char* where) {
  return fail(ctx, CUHE_CUDA_ERROR, std::string(where) + ": " + cudaGetErrorName(e) + " (" +
                                         cudaGetErrorString(e) + ")");
}

#define CUHE_CUDA(ctx, call, where)                   \
  do {                                                \
    cudaError_t _e = (call);                          \
    if (_e != cudaSuccess) return cuda_fail(ctx, _e, where); \
  } while (0)

// ---- kernel launchers -----------------------------------------------------

template <int K, int TPI, int W>
size_t modexp_smem() {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  return size_t(5 * K + IPB * cuhe::inst_stride_words<K>((1 << (W - 1)) + 1)) * 4;
}

template <int K, int TPI, int W>
cudaError_t launch_modexp(cuhe_paillier* ctx, const uint32_t* base, const uint32_t* aux, uint32_t* out,
                          long long count, const int32_t* ops, int nops, int mode, int pop_words) {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  const size_t smem = modexp_smem<K, TPI, W>();
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_modexp<K, TPI, W>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(smem));
  if (e != cudaSuccess) return e;
  const long long blocks = (count + IPB - 1) / IPB;
  cuhe::k_modexp<K, TPI, W><<<dim3(unsigned(blocks)), cuhe::kBlockThreads, smem, ctx->stream>>>(
      base, aux, K, out, count, ctx->d_consts, ctx->ks, ops, nops, mode, pop_words, ctx->d_status);
  return cudaGetLastError();
}

template <int KH, int TPI, int W>
size_t modexp_crt_smem() {
  constexpr int IPB = cuhe::kBlockThreads / (2 * TPI);
  return size_t(7 * 2 * KH + IPB * 2 * (((1 << (W - 1)) + 1) * KH + 4)) * 4;
}

// CRT decrypt / decode: KH = K/2 words per side, TPI lanes per side.
template <int KH, int TPI, int W>
cudaError_t launch_modexp_crt(cuhe_paillier* ctx, const uint32_t* base, uint32_t* out, long long count,
                              int mode, int pop_words) {
  constexpr int IPB = cuhe::kBlockThreads / (2 * TPI);
  const size_t smem = modexp_crt_smem<KH, TPI, W>();
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_modexp_crt<KH, TPI, W>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  const long long blocks = (count + IPB - 1) / IPB;
  cuhe::k_modexp_crt<KH, TPI, W><<<dim3(unsigned(blocks)), cuhe::kBlockThreads, smem, ctx->stream>>>(
      base, out, count, ctx->d_consts, ctx->ks, ctx->d_crt, ctx->cs, ctx->d_ops_sec, ctx->nops_sec, mode,
      pop_words, ctx->d_status);
  return cudaGetLastError();
}

// Batches of at most one CTA of the five-limb kernels to an SM (half the ten-
// limb kernel's items10 a CTA; one warp to a scheduler) run with five limbs
// per lane: at key_len 1024 2,368 decodes take 1.21 ms against 2.19 with ten,
// as many decryptions 4.2 against 7.3, encryptions 13.3 against 22.7.  With
// two CTAs to an SM the ten-limb kernel, whose one warp per scheduler then
// holds the same items, is as fast or faster (decodes 2.15 and 2.19 ms,
// encryptions 25.5 and 22.7).
bool pair_small(const cuhe_paillier* ctx, long long count, int items10) {
  return count <= (long long)ctx->sms * items10 / 2;
}

// And batches of at most one CTA of the split kernels to an SM (a quarter of
// items10, again one warp to a scheduler) run with the components on
// different lanes: 1,184 decodes at key_len 1024 take 0.90 ms against 1.21
// with five limbs a lane, 592 encryptions at key_len 2048 37.1 against 52.9.
// One item more, two CTAs to an SM, 1.49 against 1.21 and 66.4 against 52.9
// (all with three-bit windows; the split kernels' own take another 5 and 6%).
bool pair_tiny(const cuhe_paillier* ctx, long long count, int items10) {
  return count <= (long long)ctx->sms * items10 / 4;
}

// How many of a batch's items run with ten limbs per lane: none of a small
// batch, and of a larger one all, or all but a small remainder after whole
// waves of two CTAs to an SM, which would hold the SMs for as long as a whole
// one-CTA wave (20,011 decryptions at key_len 512: 4.8 -> 4.3 ms).
long long pair_waves(const cuhe_paillier* ctx, long long count, int items10) {
  if (pair_small(ctx, count, items10)) return 0;
  const long long rest = count % (2ll * ctx->sms * items10);
  return rest < count && pair_small(ctx, rest, items10) ? count - rest : count;
}

// The same on pairs of residues mod p and mod q (k_pair_crt).
template <int KH, int kL>
cudaError_t launch_pair_crt_l(cuhe_paillier* ctx, const uint32_t* base, uint32_t* out, long long count, int mode,
                              int pop_words) {
  using Lay = cuhe::PairLayout<5 * KH / 16, kL, 4, 2>;
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_pair_crt<KH, kL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(Lay::kBytes));
  if (e != cudaSuccess) return e;
  const long long blocks = (count + Lay::kItems - 1) / Lay::kItems;
  cuhe::k_pair_crt<KH, kL><<<dim3(unsigned(blocks)), cuhe52::kPairThreads, Lay::kBytes, ctx->stream>>>(
      base, out, count, ctx->d_consts, ctx->ks, ctx->d_crt, ctx->cs, ctx->d_crt52, ctx->side_exp[0].get(),
      ctx->side_exp[1].get(), mode, pop_words, ctx->d_status);
  return cudaGetLastError();
}

template <int KH>
cudaError_t launch_pair_crt(cuhe_paillier* ctx, const uint32_t* base, uint32_t* out, long long count, int mode,
                            int pop_words) {
  const long long main = pair_waves(ctx, count, cuhe::PairLayout<5 * KH / 16, 10, 4, 2>::kItems);
  if (main) {
    if (cudaError_t e = launch_pair_crt_l<KH, 10>(ctx, base, out, main, mode, pop_words)) return e;
    if (main == count) return cudaSuccess;
    base += main * 2 * KH;
    out += mode == cuhe::EXP_DECODE ? main : main * 2 * KH;
  }
  if (pair_tiny(ctx, count - main, cuhe::PairLayout<5 * KH / 16, 10, 4, 2>::kItems))
    return launch_pair_crt_l<KH, cuhe::kSplit>(ctx, base, out, count - main, mode, pop_words);
  return launch_pair_crt_l<KH, 5>(ctx, base, out, count - main, mode, pop_words);
}

// The exponentiation mod n^2 on pairs of residues mod n (no factors needed).
template <int K, int kL>
cudaError_t launch_pair_modexp_l(cuhe_paillier* ctx, const uint32_t* base, const uint32_t* aux, uint32_t* out,
                                 long long count, const int32_t* ops, int nops, int mode, int pop_words) {
  using Lay = cuhe::PairLayout<5 * K / 16, kL, 2, 1>;
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_pair_modexp<K, kL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(Lay::kBytes));
  if (e != cudaSuccess) return e;
  const long long blocks = (count + Lay::kItems - 1) / Lay::kItems;
  cuhe::k_pair_modexp<K, kL><<<dim3(unsigned(blocks)), cuhe52::kPairThreads, Lay::kBytes, ctx->stream>>>(
      base, aux, out, count, ctx->d_consts, ctx->ks, ctx->d_pair, ctx->pair_ninv, ops, nops, mode, pop_words,
      ctx->d_status);
  return cudaGetLastError();
}

template <int K>
cudaError_t launch_pair_modexp(cuhe_paillier* ctx, const uint32_t* base, const uint32_t* aux, uint32_t* out,
                               long long count, const int32_t* ops, int nops, int mode, int pop_words) {
  const long long main = pair_waves(ctx, count, cuhe::PairLayout<5 * K / 16, 10, 2, 1>::kItems);
  if (main) {
    if (cudaError_t e = launch_pair_modexp_l<K, 10>(ctx, base, aux, out, main, ops, nops, mode, pop_words)) return e;
    if (main == count) return cudaSuccess;
    base += main * K;
    if (aux) aux += main * K;
    out += mode == cuhe::EXP_DECODE ? main : main * K;
  }
  if (pair_tiny(ctx, count - main, cuhe::PairLayout<5 * K / 16, 10, 2, 1>::kItems))
    return launch_pair_modexp_l<K, cuhe::kSplit>(ctx, base, aux, out, count - main, ops, nops, mode, pop_words);
  return launch_pair_modexp_l<K, 5>(ctx, base, aux, out, count - main, ops, nops, mode, pop_words);
}

// k_pair_modexp for this context's width when the FP64 pipe is selected, else null.
using PairModexp = cudaError_t (*)(cuhe_paillier*, const uint32_t*, const uint32_t*, uint32_t*, long long,
                                   const int32_t*, int, int, int);
PairModexp pair_modexp(const cuhe_paillier* ctx) {
  if (!ctx->fp64 || !ctx->d_pair) return nullptr;
  if (ctx->K == 64) return &launch_pair_modexp<64>;
  if (ctx->K == 128) return &launch_pair_modexp<128>;
  if (ctx->K == 256) return &launch_pair_modexp<256>;
  return nullptr;
}

// Whether the server's products take 52-bit limbs mod n^2 (n^2 of 4096 or
// 8192 bits; 2048 bits only with set_fp64(ctx, 2)).
bool limbs52(const cuhe_paillier* ctx) {
  return ctx->fp64 && ctx->d_n52 && (ctx->K >= 128 || ctx->fp64_small);
}

// encode_hamming_server on the FP64 pipe: queries to R52 Montgomery limbs,
// then one product per output.
template <int K>
cudaError_t launch_outer52(cuhe_paillier* ctx, const uint32_t* query, long long nq, double* q52,
                           const uint32_t* index, long long nx, uint32_t* out) {
  constexpr int TPI = K / 16, K52 = 5 * K / 8, IPB = cuhe::kBlockThreads / TPI;
  const size_t csmem = size_t(K + IPB * K) * 4;
  cuhe::k_to_mont52<K><<<dim3(unsigned((nq + IPB - 1) / IPB)), cuhe::kBlockThreads, csmem, ctx->stream>>>(
      query, nq, q52, ctx->d_consts, ctx->ks, reinterpret_cast<const uint32_t*>(ctx->d_n52 + K52),
      ctx->d_status);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  const size_t smem = size_t(K52 + IPB * K52) * 8;
  const long long bx = (nx + IPB - 1) / IPB;
  for (long long q0 = 0; q0 < nq; q0 += 65535) {
    const long long qn = std::min<long long>(65535, nq - q0);
    cuhe::k_mulmod_outer52<K><<<dim3(unsigned(bx), unsigned(qn)), cuhe::kBlockThreads, smem, ctx->stream>>>(
        q52 + q0 * K52, index, nx, out + q0 * nx * K, ctx->d_consts, ctx->d_n52, ctx->ninv52, ctx->d_status);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

using Outer52 = cudaError_t (*)(cuhe_paillier*, const uint32_t*, long long, double*, const uint32_t*, long long,
                                uint32_t*);
Outer52 outer52(const cuhe_paillier* ctx) {
  if (!limbs52(ctx)) return nullptr;
  if (ctx->K == 64) return &launch_outer52<64>;
  if (ctx->K == 128) return &launch_outer52<128>;
  if (ctx->K == 256) return &launch_outer52<256>;
  return nullptr;
}

// Rows of limb pairs for the lookup encryption (k_pair_rows, k_pair_products)
// and encryption from them (k_pair_lookup).
template <int K>
cudaError_t launch_pair_rows(cuhe_paillier* ctx, const uint32_t* in, long long count, bool digits, double2* out) {
  constexpr int KL = 5 * K / 16, IPB = cuhe52::kPairThreads / (KL / 10);
  const size_t smem = size_t(2 * KL + 1) * 16;
  cuhe::k_pair_rows<K><<<dim3(unsigned((count + IPB - 1) / IPB)), cuhe52::kPairThreads, smem, ctx->stream>>>(
      in, count, digits ? ctx->d_consts + size_t(cuhe::C_RM) * K : nullptr, out, ctx->d_entry, ctx->d_pair,
      ctx->pair_ninv);
  return cudaGetLastError();
}

template <int K>
cudaError_t launch_pair_products(cuhe_paillier* ctx, const double2* src, int rows, int kind, long long first,
                                 long long count, double2* out) {
  constexpr int KL = 5 * K / 16, IPB = cuhe52::kPairThreads / (KL / 10);
  const size_t smem = size_t(IPB) * (KL + 1) * 16;
  cuhe::k_pair_products<K><<<dim3(unsigned((count + IPB - 1) / IPB)), cuhe52::kPairThreads, smem, ctx->stream>>>(
      src, rows, kind, first, count, out, ctx->d_pair, ctx->pair_ninv);
  return cudaGetLastError();
}

template <int K, int kL>
cudaError_t launch_pair_lookup_l(cuhe_paillier* ctx, const cuhe::LookupDigits& dg, long long count,
                                 const double2* table, const double2* noise, bool pairs, const uint8_t* idx,
                                 uint32_t* out) {
  using Lay = cuhe::LookupLayout<K, kL>;
  const size_t smem = Lay::bytes(dg.rows);
  // the device's limit, not this call's size: a kernel has one setting, and
  // other contexts set it between this line and the launch
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_pair_lookup<K, kL>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       ctx->smem_limit);
  if (e != cudaSuccess) return e;
  const long long blocks = (count + Lay::kGroups - 1) / Lay::kGroups;
  cuhe::k_pair_lookup<K, kL><<<dim3(unsigned(blocks)), cuhe52::kPairThreads, smem, ctx->stream>>>(
      dg, count, table, noise, ctx->noise_entries, pairs ? 1 : 0, idx, out, ctx->d_consts, ctx->ks, ctx->d_pair,
      ctx->pair_ninv, ctx->d_status);
  return cudaGetLastError();
}

template <int K>
cudaError_t launch_pair_lookup(cuhe_paillier* ctx, const cuhe::LookupDigits& dg, long long count, const double2* table,
                               const double2* noise, bool pairs, const uint8_t* idx, uint32_t* out) {
  if (pair_small(ctx, count, cuhe::LookupLayout<K, 10>::kGroups))
    return launch_pair_lookup_l<K, 5>(ctx, dg, count, table, noise, pairs, idx, out);
  return launch_pair_lookup_l<K, 10>(ctx, dg, count, table, noise, pairs, idx, out);
}

struct PairLookup {
  cudaError_t (*rows)(cuhe_paillier*, const uint32_t*, long long, bool, double2*);
  cudaError_t (*products)(cuhe_paillier*, const double2*, int, int, long long, long long, double2*);
  cudaError_t (*launch)(cuhe_paillier*, const cuhe::LookupDigits&, long long, const double2*, const double2*, bool,
                        const uint8_t*, uint32_t*);
};
bool pair_lookup(const cuhe_paillier* ctx, PairLookup* l) {
  if (!ctx->fp64 || !ctx->d_pair) return false;
  if (ctx->K == 64) *l = {&launch_pair_rows<64>, &launch_pair_products<64>, &launch_pair_lookup<64>};
  else if (ctx->K == 128) *l = {&launch_pair_rows<128>, &launch_pair_products<128>, &launch_pair_lookup<128>};
  else if (ctx->K == 256) *l = {&launch_pair_rows<256>, &launch_pair_products<256>, &launch_pair_lookup<256>};
  else return false;
  return true;
}

template <int K>
cudaError_t prepare_pair_tasks(int device, int* grid) {
  constexpr size_t smem = cuhe::PairLayout<5 * K / 16, 10, 2, 1>::kBytes;
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_pair_modexp_tasks<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(smem));
  if (e != cudaSuccess) return e;
  int per_sm = 0, sms = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cuhe::k_pair_modexp_tasks<K>, cuhe52::kPairThreads, smem);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  *grid = std::max(1, per_sm) * sms;
  return cudaSuccess;
}

template <int K>
cudaError_t launch_pair_tasks(const cuhe::ModexpTask* tasks, int ntasks, long long units, unsigned long long* counter,
                              int* status, int grid, cudaStream_t stream) {
  cuhe::k_pair_modexp_tasks<K><<<grid, cuhe52::kPairThreads, cuhe::PairLayout<5 * K / 16, 10, 2, 1>::kBytes, stream>>>(
      tasks, ntasks, units, counter, status);
  return cudaGetLastError();
}

template <int K, int TPI>
cudaError_t launch_modexp_var(cuhe_paillier* ctx, const uint32_t* base, const uint32_t* exps, int exp_words,
                              int windows, uint32_t* out, long long count) {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  const size_t smem = size_t(2 * K + IPB * cuhe::inst_stride_words<K>(17)) * 4;
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_modexp_var<K, TPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(smem));
  if (e != cudaSuccess) return e;
  const long long blocks = (count + IPB - 1) / IPB;
  cuhe::k_modexp_var<K, TPI><<<dim3(unsigned(blocks)), cuhe::kBlockThreads, smem, ctx->stream>>>(
      base, exps, exp_words, windows, out, count, ctx->d_consts, ctx->ks, ctx->d_status);
  return cudaGetLastError();
}

template <int K, int TPI>
cudaError_t launch_mulmod(cuhe_paillier* ctx, const uint32_t* a, const uint32_t* b, uint32_t* out,
                          long long count) {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  const size_t smem = size_t(K + IPB * cuhe::inst_stride_words<K>(1)) * 4;
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_mulmod<K, TPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       int(smem));
  if (e != cudaSuccess) return e;
  const long long blocks = (count + IPB - 1) / IPB;
  cuhe::k_mulmod<K, TPI><<<dim3(unsigned(blocks)), cuhe::kBlockThreads, smem, ctx->stream>>>(
      a, b, out, count, ctx->d_consts, ctx->ks, ctx->d_status);
  return cudaGetLastError();
}

template <int K, int TPI>
cudaError_t launch_convert(cuhe_paillier* ctx, const uint32_t* in, uint32_t* out, long long count, int to_mont) {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  const size_t smem = size_t(K) * 4;
  const long long blocks = (count + IPB - 1) / IPB;
  cuhe::k_convert<K, TPI><<<dim3(unsigned(blocks)), cuhe::kBlockThreads, smem, ctx->stream>>>(
      in, out, count, ctx->d_consts, ctx->ks, to_mont, ctx->d_status);
  return cudaGetLastError();
}

template <int K, int TPI>
cudaError_t launch_outer(cuhe_paillier* ctx, const uint32_t* qmont, long long nq, const uint32_t* index,
                         long long nx, uint32_t* out) {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  const size_t smem = size_t(K) * 4;
  const long long bx = (nx + IPB - 1) / IPB;
  for (long long q0 = 0; q0 < nq; q0 += 65535) {
    const long long qn = std::min<long long>(65535, nq - q0);
    cuhe::k_mulmod_outer<K, TPI><<<dim3(unsigned(bx), unsigned(qn)), cuhe::kBlockThreads, smem, ctx->stream>>>(
        qmont + q0 * K, qn, index, nx, out + q0 * nx * K, ctx->d_consts, ctx->ks, ctx->d_status);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

template <int K, int TPI>
cudaError_t launch_lookup(cuhe_paillier* ctx, const uint8_t* bits, int embed_len, int chunk_len, int chunk_num,
                          const uint32_t* plain, long long count, const uint8_t* idx, uint32_t* out) {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  const size_t rows_bytes = size_t(IPB) * cuhe::lookup_rows_stride(ctx->message_chunks) * 2;
  const size_t smem = size_t(K + IPB * cuhe::inst_stride_words<K>(1)) * 4 + ((rows_bytes + 15) & ~size_t(15));
  const bool wide = ctx->d_wide != nullptr;
  auto kernel = wide ? cuhe::k_lookup_encrypt<K, TPI, true> : cuhe::k_lookup_encrypt<K, TPI, false>;
  // (the device's limit: as for k_pair_lookup)
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_limit);
  if (e != cudaSuccess) return e;
  const long long blocks = (count + IPB - 1) / IPB;
  kernel<<<dim3(unsigned(blocks)), cuhe::kBlockThreads, smem, ctx->stream>>>(
      bits, embed_len, chunk_len, chunk_num, plain, K, count, ctx->message_chunks, wide ? ctx->d_wide : ctx->d_gtab,
      ctx->d_noise, ctx->noise_entries, idx, out, ctx->d_consts, ctx->ks, ctx->d_status);
  return cudaGetLastError();
}

// W[j][D] = G[2j][D mod 256] * G[2j+1][D / 256] for every 16-bit D, entries of
// the digit zero taken as one.
template <int K, int TPI>
cudaError_t launch_wide_table(cuhe_paillier* ctx, uint32_t* wide) {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  const size_t smem = size_t(IPB * cuhe::inst_stride_words<K>(1)) * 4;
  const long long entries = (long long)((ctx->message_chunks + 1) / 2) * 65536;
  cuhe::k_wide_table<K, TPI><<<dim3(unsigned((entries + IPB - 1) / IPB)), cuhe::kBlockThreads, smem, ctx->stream>>>(
      ctx->d_gtab, ctx->message_chunks, wide, ctx->d_consts, ctx->ks);
  return cudaGetLastError();
}

template <int K, int TPI>
cudaError_t launch_table_rows(cuhe_paillier* ctx, const uint32_t* bases, int rows, uint32_t* gtab) {
  constexpr int IPB = cuhe::kBlockThreads / TPI;
  const size_t smem = size_t(IPB * cuhe::inst_stride_words<K>(2)) * 4;
  const long long blocks = ((long long)rows * 16 + IPB - 1) / IPB;
  cuhe::k_table_rows<K, TPI><<<dim3(unsigned(blocks)), cuhe::kBlockThreads, smem, ctx->stream>>>(
      bases, rows, gtab, ctx->d_consts, ctx->ks);
  return cudaGetLastError();
}

// Persistent mixed launch: shared memory attribute and a grid of one wave of
// resident CTAs (SMs x CTAs per SM).
template <int K, int TPI, int W>
cudaError_t prepare_tasks(int device, int* grid) {
  const size_t smem = modexp_smem<K, TPI, W>();
  cudaError_t e = cudaFuncSetAttribute(cuhe::k_modexp_tasks<K, TPI, W>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
  if (e != cudaSuccess) return e;
  int per_sm = 0, sms = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cuhe::k_modexp_tasks<K, TPI, W>, cuhe::kBlockThreads,
                                                    smem);
  if (e != cudaSuccess) return e;
  e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  if (e != cudaSuccess) return e;
  *grid = std::max(1, per_sm) * sms;
  return cudaSuccess;
}

template <int K, int TPI, int W>
cudaError_t launch_tasks(const cuhe::ModexpTask* tasks, int ntasks, long long units, unsigned long long* counter,
                         int* status, int grid, cudaStream_t stream) {
  cuhe::k_modexp_tasks<K, TPI, W><<<grid, cuhe::kBlockThreads, modexp_smem<K, TPI, W>(), stream>>>(
      tasks, ntasks, units, counter, status);
  return cudaGetLastError();
}

// Runtime dispatch over the compiled variants.
struct Dispatch {
  cudaError_t (*modexp)(cuhe_paillier*, const uint32_t*, const uint32_t*, uint32_t*, long long, const int32_t*,
                        int, int, int) = nullptr;
  cudaError_t (*modexp_var)(cuhe_paillier*, const uint32_t*, const uint32_t*, int, int, uint32_t*, long long) = nullptr;
  cudaError_t (*modexp_crt)(cuhe_paillier*, const uint32_t*, uint32_t*, long long, int, int) = nullptr;
  cudaError_t (*mulmod)(cuhe_paillier*, const uint32_t*, const uint32_t*, uint32_t*, long long) = nullptr;
  cudaError_t (*convert)(cuhe_paillier*, const uint32_t*, uint32_t*, long long, int) = nullptr;
  cudaError_t (*outer)(cuhe_paillier*, const uint32_t*, long long, const uint32_t*, long long, uint32_t*) = nullptr;
  cudaError_t (*lookup)(cuhe_paillier*, const uint8_t*, int, int, int, const uint32_t*, long long, const uint8_t*,
                        uint32_t*) = nullptr;
  cudaError_t (*table_rows)(cuhe_paillier*, const uint32_t*, int, uint32_t*) = nullptr;
  cudaError_t (*wide_table)(cuhe_paillier*, uint32_t*) = nullptr;
  cudaError_t (*prepare_tasks)(int, int*) = nullptr;
  cudaError_t (*launch_tasks)(const cuhe::ModexpTask*, int, long long, unsigned long long*, int*, int,
                              cudaStream_t) = nullptr;
};

bool find_dispatch(int K, int TPI, int W, Dispatch* d) {
#define CUHE_MATCH(k, t, w)                                        \
  if (K == k && TPI == t && W == w) {                              \
    d->modexp = &launch_modexp<k, t, w>;                           \
    d->modexp_var = &launch_modexp_var<k, t>;                      \
    d->modexp_crt = &launch_modexp_crt<k / 2, t / 2, w>;           \
    d->mulmod = &launch_mulmod<k, t>;                              \
    d->convert = &launch_convert<k, t>;                            \
    d->outer = &launch_outer<k, t>;                                \
    d->lookup = &launch_lookup<k, t>;                              \
    d->table_rows = &launch_table_rows<k, t>;                      \
    d->wide_table = &launch_wide_table<k, t>;                      \
    d->prepare_tasks = &prepare_tasks<k, t, w>;                    \
    d->launch_tasks = &launch_tasks<k, t, w>;                      \
    return true;                                                   \
  }
  CUHE_VARIANTS(CUHE_MATCH)
#undef CUHE_MATCH
  return false;
}

// Exponentiation by the secret exponent (decrypt / decode): the CRT kernel
// when the factorisation is installed, else the direct kernel mod n^2.
cudaError_t secret_modexp(cuhe_paillier* ctx, const Dispatch& d, const uint32_t* base, uint32_t* out,
                          long long count, int mode, int pop_words) {
  if (ctx->have_factors && ctx->fp64) {
    if (ctx->K == 64) return launch_pair_crt<32>(ctx, base, out, count, mode, pop_words);
    if (ctx->K == 128) return launch_pair_crt<64>(ctx, base, out, count, mode, pop_words);
    if (ctx->K == 256) return launch_pair_crt<128>(ctx, base, out, count, mode, pop_words);
  }
  if (ctx->have_factors) return d.modexp_crt(ctx, base, out, count, mode, pop_words);
  if (PairModexp f = pair_modexp(ctx)) return f(ctx, base, nullptr, out, count, ctx->d_ops_sec52, ctx->nops_sec52,
                                                mode, pop_words);
  return d.modexp(ctx, base, nullptr, out, count, ctx->d_ops_sec, ctx->nops_sec, mode, pop_words);
}

void default_tuning(int K, int* tpi, int* w) {
  *w = 4;
  *tpi = K / 8;  // eight limbs per lane
}

// ---- staging of host buffers ----------------------------------------------

struct Staged {
  const void* src;
  void* dev;
  size_t bytes;
  bool in;    // copy host->device before
  bool out;   // copy device->host after
  void* host_out;
};

class Stager {
 public:
  explicit Stager(cuhe_paillier* ctx) : ctx_(ctx) {}
  // Reserve space for all buffers first, then bind.
  void add(const void* host_or_dev, size_t bytes, bool in, bool out) {
    items_.push_back({host_or_dev, nullptr, bytes, in, out, const_cast<void*>(host_or_dev)});
  }
  // Device scratch that lives in the workspace for the duration of the call.
  void add_scratch(size_t bytes) { items_.push_back({nullptr, nullptr, bytes, false, false, nullptr}); }
  int bind() {
    size_t total = 0;
    for (auto& it : items_) {
      if ((!it.src || !is_device_pointer(it.src)) && it.bytes) total += (it.bytes + 255) & ~size_t(255);
    }
    if (total) {
      cudaError_t e = ctx_->work.reserve(total);
      if (e != cudaSuccess) return cuda_fail(ctx_, e, "workspace allocation");
    }
    size_t off = 0;
    for (auto& it : items_) {
      if (!it.bytes) { it.dev = nullptr; continue; }
      if (!it.src) {
        it.dev = static_cast<char*>(ctx_->work.ptr) + off;
        off += (it.bytes + 255) & ~size_t(255);
        continue;
      }
      if (is_device_pointer(it.src)) {
        it.dev = const_cast<void*>(it.src);
        it.in = it.out = false;
      } else {
        it.dev = static_cast<char*>(ctx_->work.ptr) + off;
        off += (it.bytes + 255) & ~size_t(255);
        staged_ = true;
        if (it.in) {
          cudaError_t e = cudaMemcpyAsync(it.dev, it.src, it.bytes, cudaMemcpyHostToDevice, ctx_->stream);
          if (e != cudaSuccess) return cuda_fail(ctx_, e, "host to device copy");
        }
      }
    }
    return CUHE_OK;
  }
  void* dev(size_t i) const { return items_[i].dev; }
  int finish() {
    for (auto& it : items_) {
      if (it.out) {
        cudaError_t e = cudaMemcpyAsync(it.host_out, it.dev, it.bytes, cudaMemcpyDeviceToHost, ctx_->stream);
        if (e != cudaSuccess) return cuda_fail(ctx_, e, "device to host copy");
      }
    }
    if (staged_) {
      cudaError_t e = cudaStreamSynchronize(ctx_->stream);
      if (e != cudaSuccess) return cuda_fail(ctx_, e, "stream synchronize");
    }
    return CUHE_OK;
  }
  bool staged() const { return staged_; }
  // item i lives in the workspace (its caller buffer is host memory)
  bool is_staged(size_t i) const { return items_[i].src && items_[i].dev != items_[i].src; }

 private:
  cuhe_paillier* ctx_;
  std::vector<Staged> items_;
  bool staged_ = false;
};

// Host buffers of at least this many bytes move piece by piece beside the
// compute instead of before or after it.
constexpr size_t kPipeBytes = size_t(64) << 20;

// The context's copy and side streams, created on first use; both start
// after the work already queued on the context's stream (which may still
// use the workspace the pipeline is about to fill).
int pipeline_streams(cuhe_paillier* ctx) {
  for (cudaStream_t* st : {&ctx->copy, &ctx->side})
    if (!*st) CUHE_CUDA(ctx, cudaStreamCreateWithFlags(st, cudaStreamNonBlocking), "pipeline stream");
  cudaEvent_t ready;
  CUHE_CUDA(ctx, cudaEventCreateWithFlags(&ready, cudaEventDisableTiming), "event");
  cudaError_t e = cudaEventRecord(ready, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->copy, ready, 0);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->side, ready, 0);
  cudaEventDestroy(ready);
  CUHE_CUDA(ctx, e, "pipeline order");
  return CUHE_OK;
}

// `waiter` waits for the work queued so far on `from`.
cudaError_t stream_after(cudaStream_t waiter, cudaStream_t from) {
  cudaEvent_t ev;
  cudaError_t e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
  if (e != cudaSuccess) return e;
  e = cudaEventRecord(ev, from);
  if (e == cudaSuccess) e = cudaStreamWaitEvent(waiter, ev, 0);
  cudaEventDestroy(ev);
  return e;
}

// The wide tables, rows of 65,536 entries that halve the table products per
// ciphertext: 16 embedding bits a row (32 plaintext bits, built as far as the
// calls reach, 42 MB a row at key_len 1024), 16-bit plaintext digits (128 rows
// there), and on the integer pipe 16-bit digits in words (32 MB a row); one
// product per entry to build.  Mode 1 builds what a call of at least
// kWideMinItems ciphertexts wants when all of them together take at most
// kWideMaxBytes and a quarter of the device memory they find free (else the
// 8-bit tables serve); mode 2 builds it for any call and fails without memory;
// mode 0 never.
constexpr long long kWideMinItems = 1 << 16;
constexpr size_t kWideMaxBytes = size_t(8) << 30;

int check_status(cuhe_paillier* ctx, bool synchronous) {
  // Range errors are reported by the kernels through d_status; reading it
  // needs a synchronisation, done only for calls that already synchronise.
  if (!synchronous) return CUHE_OK;
  int status = 0;
  cudaError_t e = cudaMemcpyAsync(&status, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "status read");
  if (status) {
    cudaMemsetAsync(ctx->d_status, 0, sizeof(int), ctx->stream);
    return fail(ctx, CUHE_RANGE, "input outside its valid range (ciphertext >= n^2, plaintext >= n, or noise index)");
  }
  return CUHE_OK;
}

int upload_schedule(cuhe_paillier* ctx, const Limbs& e, int32_t** dptr, int* nops, bool pairs = false) {
  std::vector<int32_t> ops = cuhe::host::window_schedule(e, ctx->window);
  *nops = int(ops.size());
  if (pairs) ops = cuhe::host::pair_schedule(e, cuhe::kPairWindow, cuhe::kSplitWindow, nops);
  if (*dptr) cudaFree(*dptr);
  *dptr = nullptr;
  if (ops.empty()) return CUHE_OK;
  CUHE_CUDA(ctx, cudaMalloc(dptr, ops.size() * sizeof(int32_t)), "schedule allocation");
  CUHE_CUDA(ctx, cudaMemcpy(*dptr, ops.data(), ops.size() * sizeof(int32_t), cudaMemcpyHostToDevice),
            "schedule upload");
  return CUHE_OK;
}

// One of a side's schedules into its array of side.room ops, which stays where
// it is: calls captured in a graph read it at every replay.
int upload_side_schedule(cuhe_paillier* ctx, const Limbs& e, int32_t* d_ops, int* nops) {
  const std::vector<int32_t> ops = cuhe::host::pair_schedule(e, cuhe::kPairWindow, cuhe::kSplitWindow, nops);
  CUHE_CUDA(ctx, cudaMemcpy(d_ops, ops.data(), ops.size() * sizeof(int32_t), cudaMemcpyHostToDevice),
            "schedule upload");
  return CUHE_OK;
}

// The 52-bit constants mod n^2: n^2 as K52 = 5K/8 limbs of 52 bits (doubles),
// then R52 R mod n^2 as K words; R52 = 2^(52 K52), R = 2^(32K).
int setup_direct52(cuhe_paillier* ctx) {
  const size_t k = size_t(ctx->K), k52 = 5 * k / 8;
  Limbs one(k, 0u);
  one[0] = 1u;
  std::vector<double> block(k52 + k / 2, 0.0);
  for (size_t i = 0; i < k52; ++i) {
    uint64_t limb = 0;
    for (int b = 0; b < 52; ++b) {
      const size_t bit = 52 * i + size_t(b);
      if (bit / 32 < ctx->n2.size() && ((ctx->n2[bit / 32] >> (bit % 32)) & 1u)) limb |= 1ull << b;
    }
    block[i] = double(limb);
  }
  const Limbs r52r = cuhe::host::shift_mod(one, 52 * k52 + 32 * k, ctx->n2);
  std::memcpy(block.data() + k52, r52r.data(), 4 * k);
  const uint64_t m0 = (uint64_t(ctx->n2[1]) << 32) | ctx->n2[0];
  uint64_t inv = m0;
  for (int it = 0; it < 6; ++it) inv *= 2 - m0 * inv;
  ctx->ninv52 = (0 - inv) & ((1ull << 52) - 1);
  CUHE_CUDA(ctx, cudaMalloc(&ctx->d_n52, block.size() * 8), "constants allocation");
  CUHE_CUDA(ctx, cudaMemcpy(ctx->d_n52, block.data(), block.size() * 8, cudaMemcpyHostToDevice), "constants upload");
  return CUHE_OK;
}

// v as k limbs of 52 bits, balanced (each but the top one in [-2^51, 2^51))
void balanced52(const Limbs& v, size_t k, double* out, size_t stride) {
  int64_t carry = 0;
  for (size_t i = 0; i < k; ++i) {
    int64_t limb = carry;
    for (int b = 0; b < 52; ++b) {
      const size_t bit = 52 * i + size_t(b);
      if (bit / 32 < v.size() && ((v[bit / 32] >> (bit % 32)) & 1u)) limb += int64_t(1) << b;
    }
    carry = i + 1 < k && limb >= (int64_t(1) << 51) ? 1 : 0;
    if (carry) limb -= int64_t(1) << 52;
    out[i * stride] = double(limb);
  }
}

// The constants of one modulus m (pair_const_doubles) for pair_power: k limbs
// per component, `entry` chunks of a value; scale: null, or the factor of the
// scale row.  m in its natural limb count w; m^2 in 2w limbs.
std::vector<double> pair_constants(const Limbs& m_in, size_t k, int entry, const Limbs* scale) {
  Limbs m = m_in;
  while (m.size() > 1 && m.back() == 0) m.pop_back();
  const size_t w = m.size(), bits = 52 * k;
  const Limbs mm = cuhe::host::mul(m, m, 2 * w);
  std::vector<double> block(size_t(cuhe::pair_const_doubles(int(k), entry)), 0.0);
  balanced52(m, k, block.data(), 1);
  double* rows = block.data() + k;
  auto put = [&](int row, const Limbs& v) {  // the pair (v mod m, floor(v / m))
    Limbs quotient;
    const Limbs rem = cuhe::host::mod_reduce(v, m, &quotient);
    balanced52(rem, k, rows + size_t(row) * 2 * k, 2);
    balanced52(quotient, k, rows + size_t(row) * 2 * k + 1, 2);
  };
  Limbs x(2 * w, 0u);
  x[0] = 1u;  // m >= 3
  rows[size_t(entry) * 2 * k] = 1.0;
  x = cuhe::host::shift_mod(x, bits, mm);
  put(entry + 2, x);
  for (int j = 0; j < entry; ++j) {
    x = cuhe::host::shift_mod(x, bits, mm);
    put(j, x);  // R^(j+2)
  }
  if (scale) {
    const Limbs u = cuhe::host::mod_reduce(*scale, m);
    balanced52(cuhe::host::shift_mod(u, bits, m), k, rows + size_t(entry + 1) * 2 * k, 2);
  }
  return block;
}

// -m^-1 mod 2^52 for odd m (Newton's iteration on the low 64 bits)
unsigned long long negative_inverse52(const Limbs& m) {
  const uint64_t m0 = (uint64_t(m.size() > 1 ? m[1] : 0u) << 32) | m[0];
  uint64_t inv = m0;
  for (int it = 0; it < 6; ++it) inv *= 2 - m0 * inv;
  return (0 - inv) & ((1ull << 52) - 1);
}

int upload_constants(cuhe_paillier* ctx, const std::vector<double>& block, double** dptr) {
  if (!*dptr) CUHE_CUDA(ctx, cudaMalloc(dptr, block.size() * 8), "constants allocation");
  CUHE_CUDA(ctx, cudaMemcpy(*dptr, block.data(), block.size() * 8, cudaMemcpyHostToDevice), "constants upload");
  return CUHE_OK;
}

// k_pair_crt's constants and schedules, from the factors and the secret
// exponent (whichever came last).  A multiple u (p - 1) of p - 1 with u > 1
// (a textbook key's phi) is raised as p - 1, half the exponent's length.
int setup_pair_crt(cuhe_paillier* ctx) {
  if (!ctx->have_factors) return CUHE_OK;
  const size_t k = 5 * size_t(ctx->K) / 32;
  std::vector<double> block;
  for (int s = 0; s < 2; ++s) {
    auto& side = ctx->side_exp[s];
    Limbs p = ctx->factor[s], other = ctx->factor[1 - s];
    ctx->cs.ninv52[s] = negative_inverse52(p);
    side.halved = 0;
    Limbs cofactor, main = ctx->secret_exp, scale;
    if (ctx->have_secret) {
      // (other factor)^-1 multiplier [cofactor] mod p
      while (p.size() > 1 && p.back() == 0) p.pop_back();
      const size_t w = p.size();
      Limbs inv;
      if (!cuhe::host::mod_inverse_odd(cuhe::host::mod_reduce(other, p), p, &inv))
        return fail(ctx, CUHE_INVALID_ARGUMENT, "factors are not coprime");
      scale = cuhe::host::mod_reduce(cuhe::host::mul(inv, cuhe::host::mod_reduce(ctx->secret_mult, p), 2 * w), p);
      Limbs pm1 = p;
      pm1[0] -= 1u;  // p is odd
      while (pm1.size() > 1 && pm1.back() == 0) pm1.pop_back();
      if (!cuhe::host::is_zero(ctx->secret_exp) &&
          cuhe::host::is_zero(cuhe::host::mod_reduce(ctx->secret_exp, pm1, &cofactor)) &&
          cuhe::host::bit_length(cofactor) > 1) {
        side.halved = 1;
        main = pm1;
        scale = cuhe::host::mod_reduce(cuhe::host::mul(scale, cuhe::host::mod_reduce(cofactor, p), 2 * w), p);
      }
    }
    const std::vector<double> one = pair_constants(p, k, 4, ctx->have_secret ? &scale : nullptr);
    block.insert(block.end(), one.begin(), one.end());
    if (!ctx->have_secret) continue;
    // both schedules are of divisors of the secret exponent: a context's
    // arrays are made anew for a longer secret only
    const size_t room = cuhe::host::pair_schedule_room(cuhe::host::bit_length(ctx->secret_exp), cuhe::kPairWindow);
    if (room > side.room) {
      for (int32_t** ops : {&side.d_ops, &side.d_fall}) {
        cudaFree(*ops);
        *ops = nullptr;
      }
      side.room = 0;
      for (int32_t** ops : {&side.d_ops, &side.d_fall})
        CUHE_CUDA(ctx, cudaMalloc(ops, room * sizeof(int32_t)), "schedule allocation");
      side.room = room;
    }
    if (int rc = upload_side_schedule(ctx, main, side.d_ops, &side.nops)) return rc;
    if (side.halved)
      if (int rc = upload_side_schedule(ctx, cofactor, side.d_fall, &side.nfall)) return rc;
  }
  return upload_constants(ctx, block, &ctx->d_crt52);
}

struct DeviceGuard {
  int prev = -1;
  explicit DeviceGuard(int dev) {
    cudaGetDevice(&prev);
    if (prev != dev) cudaSetDevice(dev);
  }
  ~DeviceGuard() {
    int cur = -1;
    cudaGetDevice(&cur);
    if (prev >= 0 && cur != prev) cudaSetDevice(prev);
  }
};

}  // namespace

extern "C" {

const char* cuhe_version(void) { return "cuhe_b200 paillier 1"; }

int cuhe_window_schedule(const uint32_t* exponent, int exponent_words, int window, int32_t* ops, int capacity) {
  if (!exponent || exponent_words <= 0 || window < 1 || window > 8 || capacity < 0) return CUHE_INVALID_ARGUMENT;
  Limbs e(exponent, exponent + exponent_words);
  std::vector<int32_t> sched = cuhe::host::window_schedule(e, window);
  for (int i = 0; i < capacity && i < int(sched.size()); ++i) ops[i] = sched[size_t(i)];
  return int(sched.size());
}

const char* cuhe_last_error(const cuhe_paillier* ctx) {
  return ctx ? ctx->error.c_str() : g_create_error.c_str();
}

int cuhe_paillier_words(const cuhe_paillier* ctx) { return ctx ? ctx->K : 0; }

int cuhe_paillier_create(const uint32_t* n_in, int n_words, int device, cuhe_paillier** out) {
  if (!out || !n_in || n_words <= 0) return fail(nullptr, CUHE_INVALID_ARGUMENT, "null argument");
  *out = nullptr;
  Limbs n(n_in, n_in + n_words);
  while (!n.empty() && n.back() == 0) n.pop_back();
  if (n.empty() || (n[0] & 1u) == 0) return fail(nullptr, CUHE_INVALID_ARGUMENT, "n must be odd and nonzero");
  const size_t nbits = cuhe::host::bit_length(n);
  int K = 0;
  for (int cand : {64, 128, 256}) {
    if (nbits <= size_t(cand) * 16) { K = cand; break; }
  }
  if (!K) return fail(nullptr, CUHE_INVALID_ARGUMENT, "n wider than 4096 bits is not supported");
  int count = 0;
  cudaError_t ce = cudaGetDeviceCount(&count);
  if (ce != cudaSuccess || count == 0) return fail(nullptr, CUHE_CUDA_ERROR, "no CUDA device available");
  if (device < 0 || device >= count) return fail(nullptr, CUHE_INVALID_ARGUMENT, "invalid device ordinal");
  DeviceGuard guard(device);

  auto* ctx = new (std::nothrow) cuhe_paillier();
  if (!ctx) return fail(nullptr, CUHE_OUT_OF_MEMORY, "context allocation");
  ctx->device = device;
  if (cudaDeviceGetAttribute(&ctx->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) ctx->sms = 148;
  cudaDeviceGetAttribute(&ctx->smem_limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  ctx->smem_limit -= 1 << 10;
  ctx->K = K;
  ctx->n_words = K / 2;
  default_tuning(K, &ctx->tpi, &ctx->window);

  const size_t k = size_t(K);
  Limbs nk = cuhe::host::resized(n.data(), n.size(), k);
  Limbs n2 = cuhe::host::mul(nk, nk, k);
  ctx->n = nk;
  ctx->n2 = n2;
  // R mod N = 2^(32K) mod N via doubling from 1; likewise R^2 = R * 2^(32K)
  Limbs one(k, 0u);
  one[0] = 1u;
  Limbs rm = cuhe::host::shift_mod(one, 32 * k, n2);
  Limbs r2 = cuhe::host::shift_mod(rm, 32 * k, n2);
  Limbs rmn = cuhe::host::shift_mod(one, 32 * k, nk);
  Limbs r2n = cuhe::host::shift_mod(rmn, 32 * k, nk);
  Limbs nneg(k, 0u);
  cuhe::host::sub_in_place(nneg, nk);  // 2^(32K) - n (mod 2^(32K))
  Limbs nr = cuhe::host::shift_mod(nk, 32 * k, n2);  // n < n^2
  Limbs multr(k, 0u);

  std::vector<uint32_t> block(size_t(cuhe::C_ROWS) * k, 0u);
  auto put = [&](int row, const Limbs& v) { std::memcpy(block.data() + size_t(row) * k, v.data(), 4 * k); };
  put(cuhe::C_N2, n2);
  put(cuhe::C_R2, r2);
  put(cuhe::C_ONE, one);
  put(cuhe::C_RM, rm);
  put(cuhe::C_N, nk);
  put(cuhe::C_R2N, r2n);
  put(cuhe::C_NNEG, nneg);
  put(cuhe::C_NR, nr);
  put(cuhe::C_MULTR, multr);
  ctx->ks.ninv2 = 0u - cuhe::host::inv32(n2[0]);
  ctx->ks.ninv1 = 0u - cuhe::host::inv32(nk[0]);
  ctx->ks.ndiv = cuhe::host::inv32(nk[0]);
  ctx->ks.mult_is_zero = 1u;

  cudaError_t e = cudaStreamCreateWithFlags(&ctx->own_stream, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaMalloc(&ctx->d_consts, block.size() * 4);
  if (e == cudaSuccess) e = cudaMemcpy(ctx->d_consts, block.data(), block.size() * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMalloc(&ctx->d_status, sizeof(int));
  if (e == cudaSuccess) e = cudaMemset(ctx->d_status, 0, sizeof(int));
  if (e != cudaSuccess) {
    int rc = cuda_fail(nullptr, e, "context setup");
    cuhe_paillier_destroy(ctx);
    return rc;
  }
  ctx->stream = ctx->own_stream;
  ctx->pair_ninv = negative_inverse52(nk);
  if (upload_schedule(ctx, nk, &ctx->d_ops_n, &ctx->nops_n) != CUHE_OK ||
      upload_schedule(ctx, nk, &ctx->d_ops_n52, &ctx->nops_n52, true) != CUHE_OK ||
      setup_direct52(ctx) != CUHE_OK ||
      upload_constants(ctx, pair_constants(nk, 5 * k / 16, 2, nullptr), &ctx->d_pair) != CUHE_OK) {
    g_create_error = ctx->error;
    cuhe_paillier_destroy(ctx);
    return CUHE_CUDA_ERROR;
  }
  *out = ctx;
  return CUHE_OK;
}

void cuhe_paillier_destroy(cuhe_paillier* ctx) {
  if (!ctx) return;
  DeviceGuard guard(ctx->device);
  if (ctx->own_stream) cudaStreamSynchronize(ctx->own_stream);
  if (ctx->stream && ctx->stream != ctx->own_stream) cudaStreamSynchronize(ctx->stream);
  cudaFree(ctx->d_consts);
  cudaFree(ctx->d_status);
  cudaFree(ctx->d_ops_n);
  cudaFree(ctx->d_ops_sec);
  cudaFree(ctx->d_ops_sec52);
  cudaFree(ctx->d_crt);
  cudaFree(ctx->d_crt52);
  cudaFree(ctx->d_pair);
  cudaFree(ctx->d_n52);
  for (auto& side : ctx->side_exp) {
    cudaFree(side.d_ops);
    cudaFree(side.d_fall);
  }
  cudaFree(ctx->d_ops_n52);
  cudaFree(ctx->d_gtab);
  cudaFree(ctx->d_wide);
  ctx->pt.release();
  cudaFree(ctx->d_entry);
  cudaFree(ctx->d_noise);
  for (cudaStream_t st : {ctx->copy, ctx->side})
    if (st) cudaStreamSynchronize(st);
  ctx->work.release();
  ctx->tmp_ops.release();
  for (cudaStream_t st : {ctx->copy, ctx->side})
    if (st) cudaStreamDestroy(st);
  if (ctx->own_stream) cudaStreamDestroy(ctx->own_stream);
  delete ctx;
}

int cuhe_paillier_set_stream(cuhe_paillier* ctx, void* stream) {
  if (!ctx) return CUHE_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mu);
  ctx->stream = stream ? static_cast<cudaStream_t>(stream) : ctx->own_stream;
  return CUHE_OK;
}

int cuhe_synchronize(cuhe_paillier* ctx) {
  if (!ctx) return CUHE_INVALID_ARGUMENT;
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "synchronize");
  return check_status(ctx, true);
}

int cuhe_paillier_set_tuning(cuhe_paillier* ctx, int tpi, int window) {
  if (!ctx) return CUHE_INVALID_ARGUMENT;
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  int dt, dw;
  default_tuning(ctx->K, &dt, &dw);
  if (!tpi) tpi = dt;
  if (!window) window = dw;
  Dispatch d;
  if (!find_dispatch(ctx->K, tpi, window, &d))
    return fail(ctx, CUHE_INVALID_ARGUMENT, "tuning (threads per instance, window) not compiled for this width");
  const bool changed = window != ctx->window;
  ctx->tpi = tpi;
  ctx->window = window;
  if (changed) {
    int rc = upload_schedule(ctx, ctx->n, &ctx->d_ops_n, &ctx->nops_n);
    if (rc) return rc;
    if (ctx->have_secret) {
      rc = upload_schedule(ctx, ctx->secret_exp, &ctx->d_ops_sec, &ctx->nops_sec);
      if (rc) return rc;
    }
  }
  return CUHE_OK;
}

int cuhe_paillier_get_tuning(const cuhe_paillier* ctx, int* tpi, int* window) {
  if (!ctx) return CUHE_INVALID_ARGUMENT;
  if (tpi) *tpi = ctx->tpi;
  if (window) *window = ctx->window;
  return CUHE_OK;
}

int cuhe_paillier_set_secret(cuhe_paillier* ctx, const uint32_t* exponent, int exponent_words,
                             const uint32_t* multiplier, int multiplier_words) {
  if (!ctx || !exponent || !multiplier || exponent_words <= 0 || multiplier_words <= 0)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "null secret");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  const size_t k = size_t(ctx->K);
  if (!cuhe::host::fits(exponent, size_t(exponent_words), k))
    return fail(ctx, CUHE_INVALID_ARGUMENT, "secret exponent wider than n^2");
  if (!cuhe::host::fits(multiplier, size_t(multiplier_words), k))
    return fail(ctx, CUHE_INVALID_ARGUMENT, "secret multiplier too wide");
  Limbs e = cuhe::host::resized(exponent, size_t(exponent_words), k);
  Limbs mult = cuhe::host::resized(multiplier, size_t(multiplier_words), k);
  if (cuhe::host::cmp(mult, ctx->n) >= 0) {
    // the reference reduces (x * mult) mod n; reduce the multiplier first
    while (cuhe::host::cmp(mult, ctx->n) >= 0) cuhe::host::sub_in_place(mult, ctx->n);
  }
  Limbs multr = cuhe::host::shift_mod(mult, 32 * k, ctx->n);
  // kernels already queued may still read the previous secret
  CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "synchronize before secret upload");
  CUHE_CUDA(ctx, cudaMemcpy(ctx->d_consts + size_t(cuhe::C_MULTR) * k, multr.data(), 4 * k, cudaMemcpyHostToDevice),
            "secret upload");
  ctx->ks.mult_is_zero = cuhe::host::is_zero(mult) ? 1u : 0u;
  ctx->secret_exp = e;
  ctx->secret_mult = mult;
  ctx->have_secret = true;
  int rc = upload_schedule(ctx, e, &ctx->d_ops_sec52, &ctx->nops_sec52, true);
  if (!rc) rc = setup_pair_crt(ctx);
  if (!rc) rc = upload_schedule(ctx, e, &ctx->d_ops_sec, &ctx->nops_sec);
  if (rc) ctx->have_secret = false;  // nothing reads what is half installed
  return rc;
}

int cuhe_paillier_set_factors(cuhe_paillier* ctx, const uint32_t* p_in, int p_words, const uint32_t* q_in,
                              int q_words) {
  if (!ctx) return CUHE_INVALID_ARGUMENT;
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  if (!p_in && !q_in) {
    ctx->have_factors = false;
    return CUHE_OK;
  }
  if (!p_in || !q_in || p_words <= 0 || q_words <= 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "null factor");
  const size_t k = size_t(ctx->K), kh = k / 2;
  if (!cuhe::host::fits(p_in, size_t(p_words), k) || !cuhe::host::fits(q_in, size_t(q_words), k))
    return fail(ctx, CUHE_INVALID_ARGUMENT, "factor wider than n");
  Limbs p = cuhe::host::resized(p_in, size_t(p_words), k), q = cuhe::host::resized(q_in, size_t(q_words), k);
  Limbs n2k = cuhe::host::resized(ctx->n.data(), ctx->n.size(), 2 * k);
  if (cuhe::host::cmp(cuhe::host::mul(p, q, 2 * k), n2k) != 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "p * q != n");
  if (!(p[0] & 1u) || !(q[0] & 1u) || cuhe::host::bit_length(p) < 2 || cuhe::host::bit_length(q) < 2)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "factors must be odd and greater than 1");
  if (cuhe::host::bit_length(p) > 16 * kh || cuhe::host::bit_length(q) > 16 * kh)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "unbalanced factors: p^2 or q^2 wider than half of n^2");
  Limbs one(kh, 0u);
  one[0] = 1u;
  Limbs side[2] = {cuhe::host::mul(p, p, kh), cuhe::host::mul(q, q, kh)};  // p^2, q^2
  Limbs qinv;
  if (!cuhe::host::mod_inverse_odd(cuhe::host::mod_reduce(side[1], side[0]), side[0], &qinv))
    return fail(ctx, CUHE_INVALID_ARGUMENT, "factors are not coprime");
  std::vector<uint32_t> block(size_t(cuhe::CR_ROWS) * k, 0u);
  auto put_half = [&](int row, int s, const Limbs& v) {
    std::memcpy(block.data() + size_t(row) * k + size_t(s) * kh, v.data(), 4 * kh);
  };
  for (int s = 0; s < 2; ++s) {
    Limbs rm = cuhe::host::shift_mod(one, 32 * kh, side[s]);
    put_half(cuhe::CR_M, s, side[s]);
    put_half(cuhe::CR_RM, s, rm);
    put_half(cuhe::CR_R3, s, cuhe::host::shift_mod(rm, 64 * kh, side[s]));
    put_half(cuhe::CR_PR, s, cuhe::host::shift_mod(cuhe::host::resized((s ? q : p).data(), kh, kh), 32 * kh, side[s]));
    ctx->cs.ninv[s] = 0u - cuhe::host::inv32(side[s][0]);
  }
  put_half(cuhe::CR_P, 0, cuhe::host::resized(p.data(), kh, kh));
  {
    const Limbs ph = cuhe::host::resized(p.data(), kh, kh), nh = cuhe::host::resized(ctx->n.data(), kh, kh);
    Limbs qp;
    if (!cuhe::host::mod_inverse_odd(cuhe::host::mod_reduce(q, ph), ph, &qp))
      return fail(ctx, CUHE_INVALID_ARGUMENT, "factors are not coprime");
    put_half(cuhe::CR_QI, 0, cuhe::host::shift_mod(qp, 32 * kh, ph));
    put_half(cuhe::CR_QR, 0, cuhe::host::shift_mod(cuhe::host::resized(q.data(), kh, kh), 32 * kh, nh));
    ctx->cs.pinv = 0u - cuhe::host::inv32(p[0]);
  }
  put_half(cuhe::CR_H, 0, cuhe::host::shift_mod(qinv, 32 * kh, side[0]));
  Limbs cq = cuhe::host::shift_mod(cuhe::host::resized(side[1].data(), kh, k), 32 * k, ctx->n2);
  std::memcpy(block.data() + size_t(cuhe::CR_CQ) * k, cq.data(), 4 * k);
  // kernels already queued may still read the previous constants
  CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "synchronize before CRT constants upload");
  if (!ctx->d_crt) CUHE_CUDA(ctx, cudaMalloc(&ctx->d_crt, block.size() * 4), "CRT constants allocation");
  CUHE_CUDA(ctx, cudaMemcpy(ctx->d_crt, block.data(), block.size() * 4, cudaMemcpyHostToDevice), "CRT constants upload");
  ctx->factor[0] = p;
  ctx->factor[1] = q;
  ctx->have_factors = true;
  const int rc = setup_pair_crt(ctx);
  if (rc) ctx->have_factors = false;  // decryption goes without what is half installed
  return rc;
}

int cuhe_paillier_has_factors(const cuhe_paillier* ctx) { return ctx && ctx->have_factors ? 1 : 0; }

int cuhe_paillier_set_fp64(cuhe_paillier* ctx, int enable) {
  if (!ctx) return CUHE_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lock(ctx->mu);
  ctx->fp64 = enable != 0;
  ctx->fp64_small = enable == 2;
  return CUHE_OK;
}

int cuhe_paillier_get_fp64(const cuhe_paillier* ctx) { return !ctx || !ctx->fp64 ? 0 : ctx->fp64_small ? 2 : 1; }

int cuhe_paillier_encrypt(cuhe_paillier* ctx, const uint32_t* m, const uint32_t* r, uint32_t* c, int64_t count) {
  if (!ctx || count < 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (count == 0) return CUHE_OK;
  if (!m || !r || !c) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const size_t bytes = size_t(count) * ctx->K * 4;
  Stager st(ctx);
  st.add(m, bytes, true, false);
  st.add(r, bytes, true, false);
  st.add(c, bytes, false, true);
  if (int rc = st.bind()) return rc;
  if (PairModexp f = pair_modexp(ctx)) {
    CUHE_CUDA(ctx, f(ctx, (const uint32_t*)st.dev(1), (const uint32_t*)st.dev(0), (uint32_t*)st.dev(2), count,
                     ctx->d_ops_n52, ctx->nops_n52, cuhe::EXP_ENCRYPT, 0),
              "encrypt launch");
  } else {
    CUHE_CUDA(ctx, d.modexp(ctx, (const uint32_t*)st.dev(1), (const uint32_t*)st.dev(0), (uint32_t*)st.dev(2), count,
                            ctx->d_ops_n, ctx->nops_n, cuhe::EXP_ENCRYPT, 0),
              "encrypt launch");
  }
  if (int rc = st.finish()) return rc;
  return check_status(ctx, st.staged());
}

int cuhe_paillier_decrypt(cuhe_paillier* ctx, const uint32_t* c, uint32_t* m, int64_t count) {
  if (!ctx || count < 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (!ctx->have_secret) return fail(ctx, CUHE_NOT_READY, "decrypt: secret key not installed");
  if (count == 0) return CUHE_OK;
  if (!c || !m) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const size_t bytes = size_t(count) * ctx->K * 4;
  Stager st(ctx);
  st.add(c, bytes, true, false);
  st.add(m, bytes, false, true);
  if (int rc = st.bind()) return rc;
  CUHE_CUDA(ctx, secret_modexp(ctx, d, (const uint32_t*)st.dev(0), (uint32_t*)st.dev(1), count, cuhe::EXP_DECRYPT, 0),
            "decrypt launch");
  if (int rc = st.finish()) return rc;
  return check_status(ctx, st.staged());
}

int cuhe_paillier_decode_hamming(cuhe_paillier* ctx, const uint32_t* c, int64_t vectors, int chunk_num,
                                 int chunk_len, int64_t* distance) {
  if (!ctx || vectors < 0 || chunk_num <= 0 || chunk_len <= 0 || chunk_len % 32)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid decode layout");
  if (!ctx->have_secret) return fail(ctx, CUHE_NOT_READY, "decode: secret key not installed");
  if (vectors == 0) return CUHE_OK;
  if (!c || !distance) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  if (chunk_len / 32 > ctx->K) return fail(ctx, CUHE_INVALID_ARGUMENT, "chunk_len wider than n^2");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const int64_t total = vectors * chunk_num;
  const size_t cbytes = size_t(total) * ctx->K * 4;
  // A large host input moves in two pieces on the copy stream: the first
  // sixteenth, decoded on the context's stream as soon as it has arrived,
  // and the rest, decoded on the side stream (so the first launch's last
  // wave overlaps the second) while only the first piece's copy is exposed.
  const bool pipe = cbytes >= kPipeBytes && vectors >= 32 && !is_device_pointer(c);
  Stager st(ctx);
  st.add(c, cbytes, !pipe, false);
  st.add_scratch(size_t(total) * 4);  // per-chunk popcounts
  st.add(distance, size_t(vectors) * 8, false, true);
  if (int rc = st.bind()) return rc;
  uint32_t* d_counts = static_cast<uint32_t*>(st.dev(1));
  const uint32_t* d_c = static_cast<const uint32_t*>(st.dev(0));
  if (pipe && st.is_staged(0)) {
    if (int rc = pipeline_streams(ctx)) return rc;
    const int64_t first = std::max<int64_t>(1, vectors / 16) * chunk_num;
    const size_t fbytes = size_t(first) * ctx->K * 4;
    cudaEvent_t arrived[2];
    for (auto& ev : arrived) CUHE_CUDA(ctx, cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "event");
    cudaError_t e = cudaMemcpyAsync(const_cast<uint32_t*>(d_c), c, fbytes, cudaMemcpyHostToDevice, ctx->copy);
    if (e == cudaSuccess) e = cudaEventRecord(arrived[0], ctx->copy);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(const_cast<uint32_t*>(d_c) + size_t(first) * ctx->K, c + size_t(first) * ctx->K,
                          cbytes - fbytes, cudaMemcpyHostToDevice, ctx->copy);
    if (e == cudaSuccess) e = cudaEventRecord(arrived[1], ctx->copy);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->stream, arrived[0], 0);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(ctx->side, arrived[1], 0);
    for (auto& ev : arrived) cudaEventDestroy(ev);
    CUHE_CUDA(ctx, e, "piecewise upload");
    CUHE_CUDA(ctx, secret_modexp(ctx, d, d_c, d_counts, first, cuhe::EXP_DECODE, chunk_len / 32), "decode launch");
    cudaStream_t own = ctx->stream;
    ctx->stream = ctx->side;  // the launchers queue on ctx->stream
    e = secret_modexp(ctx, d, d_c + size_t(first) * ctx->K, d_counts + first, total - first, cuhe::EXP_DECODE,
                      chunk_len / 32);
    ctx->stream = own;
    CUHE_CUDA(ctx, e, "decode launch");
    CUHE_CUDA(ctx, stream_after(ctx->stream, ctx->side), "decode join");
  } else {
    CUHE_CUDA(ctx, secret_modexp(ctx, d, d_c, d_counts, total, cuhe::EXP_DECODE, chunk_len / 32), "decode launch");
  }
  cuhe::k_sum_chunks<<<unsigned((vectors + 255) / 256), 256, 0, ctx->stream>>>(
      d_counts, vectors, chunk_num, reinterpret_cast<long long*>(st.dev(2)));
  CUHE_CUDA(ctx, cudaGetLastError(), "decode reduction");
  if (int rc = st.finish()) return rc;
  return check_status(ctx, st.staged());
}

}  // extern "C"

namespace {

constexpr int kMaxStaticDevices = 64;
std::mutex g_static_mu;
uint32_t* g_static_counts[kMaxStaticDevices] = {};

// Device address of g_static_decode_counts on `device` (which is current).
int static_counts(cuhe_paillier* ctx, int device, uint32_t** out) {
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (device < 0 || device >= kMaxStaticDevices) return fail(ctx, CUHE_INVALID_ARGUMENT, "device ordinal out of range");
  if (!g_static_counts[device]) {
    void* address = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&address, g_static_decode_counts);
    if (e != cudaSuccess) return cuda_fail(ctx, e, "static scratch address");
    g_static_counts[device] = static_cast<uint32_t*>(address);
  }
  *out = g_static_counts[device];
  return CUHE_OK;
}

}  // namespace

extern "C" {

int cuhe_paillier_decode_hamming_static(cuhe_paillier* ctx, const uint32_t* c, int64_t vectors, int chunk_num,
                                        int chunk_len, int64_t* distance) {
  if (!ctx || vectors < 0 || chunk_num <= 0 || chunk_len <= 0 || chunk_len % 32)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid decode layout");
  if (!ctx->have_secret) return fail(ctx, CUHE_NOT_READY, "decode: secret key not installed");
  if (vectors == 0) return CUHE_OK;
  if (!c || !distance) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  if (chunk_len / 32 > ctx->K) return fail(ctx, CUHE_INVALID_ARGUMENT, "chunk_len wider than n^2");
  if (vectors > CUHE_STATIC_DECODE_MAX_CHUNKS / chunk_num)
    return fail(ctx, CUHE_INVALID_ARGUMENT,
                "decode_hamming_static: vectors*chunk_num exceeds the static scratch of " +
                    std::to_string(CUHE_STATIC_DECODE_MAX_CHUNKS) + " ciphertext chunks");
  DeviceGuard guard(ctx->device);
  if (!is_device_pointer(c) || !is_device_pointer(distance))
    return fail(ctx, CUHE_INVALID_ARGUMENT, "decode_hamming_static needs device buffers for c and distance");
  std::lock_guard<std::mutex> lock(ctx->mu);
  uint32_t* counts = nullptr;
  if (int rc = static_counts(ctx, ctx->device, &counts)) return rc;
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const int64_t total = vectors * chunk_num;
  CUHE_CUDA(ctx, secret_modexp(ctx, d, c, counts, total, cuhe::EXP_DECODE, chunk_len / 32), "static decode launch");
  cuhe::k_sum_chunks<<<unsigned((vectors + 255) / 256), 256, 0, ctx->stream>>>(
      counts, vectors, chunk_num, reinterpret_cast<long long*>(distance));
  CUHE_CUDA(ctx, cudaGetLastError(), "static decode reduction");
  return CUHE_OK;
}

int cuhe_fp64_peak(int device, double* fp64_per_second) {
  if (!fp64_per_second) return fail(nullptr, CUHE_INVALID_ARGUMENT, "null output");
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
    return fail(nullptr, CUHE_CUDA_ERROR, "no such CUDA device");
  DeviceGuard guard(device);
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  double* sink = nullptr;
  cudaEvent_t a = nullptr, b = nullptr;
  cudaError_t e = cudaMalloc(&sink, 8);
  if (e == cudaSuccess) e = cudaEventCreate(&a);
  if (e == cudaSuccess) e = cudaEventCreate(&b);
  const int iters = 8192, blocks = sms * 8, threads = 256;
  float ms = 0.f;
  if (e == cudaSuccess) {
    cuhe::k_fp64_probe<<<blocks, threads>>>(sink, iters, 1.0);  // warm-up
    cudaEventRecord(a);
    for (int r = 0; r < 5; ++r) cuhe::k_fp64_probe<<<blocks, threads>>>(sink, iters, 2.0 + r);
    cudaEventRecord(b);
    e = cudaEventSynchronize(b);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms, a, b);
  }
  if (a) cudaEventDestroy(a);
  if (b) cudaEventDestroy(b);
  cudaFree(sink);
  if (e != cudaSuccess) return cuda_fail(nullptr, e, "fp64 probe");
  *fp64_per_second = 5.0 * blocks * threads * double(iters) * 8.0 / (double(ms) * 1e-3);
  return CUHE_OK;
}

int cuhe_imad_peak(int device, double* word_products_per_second) {
  if (!word_products_per_second) return fail(nullptr, CUHE_INVALID_ARGUMENT, "null output");
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count)
    return fail(nullptr, CUHE_CUDA_ERROR, "no such CUDA device");
  DeviceGuard guard(device);
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
  uint32_t* sink = nullptr;
  cudaEvent_t a = nullptr, b = nullptr;
  cudaError_t e = cudaMalloc(&sink, 4);
  if (e == cudaSuccess) e = cudaEventCreate(&a);
  if (e == cudaSuccess) e = cudaEventCreate(&b);
  const int iters = 4096, blocks = sms * 8, threads = 256;
  float ms_pairs = 0.f, ms_chain = 0.f;
  if (e == cudaSuccess) {
    cuhe::k_imad_probe<<<blocks, threads>>>(sink, iters, 1u);  // warm-up
    cudaEventRecord(a);
    for (int r = 0; r < 5; ++r) cuhe::k_imad_probe<<<blocks, threads>>>(sink, iters, 2u + r);
    cudaEventRecord(b);
    e = cudaEventSynchronize(b);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms_pairs, a, b);
  }
  if (e == cudaSuccess) {
    cuhe::k_imad_chain_probe<<<blocks, threads>>>(sink, iters, 1u);  // warm-up
    cudaEventRecord(a);
    for (int r = 0; r < 5; ++r) cuhe::k_imad_chain_probe<<<blocks, threads>>>(sink, iters, 2u + r);
    cudaEventRecord(b);
    e = cudaEventSynchronize(b);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms_chain, a, b);
  }
  float ms_wide = 0.f;
  if (e == cudaSuccess) {
    cuhe::k_imad_wide_probe<<<blocks, threads>>>(sink, iters, 1u);  // warm-up
    cudaEventRecord(a);
    for (int r = 0; r < 5; ++r) cuhe::k_imad_wide_probe<<<blocks, threads>>>(sink, iters, 2u + r);
    cudaEventRecord(b);
    e = cudaEventSynchronize(b);
    if (e == cudaSuccess) e = cudaEventElapsedTime(&ms_wide, a, b);
  }
  if (a) cudaEventDestroy(a);
  if (b) cudaEventDestroy(b);
  cudaFree(sink);
  if (e != cudaSuccess) return cuda_fail(nullptr, e, "imad probe");
  // word products per thread per iteration: 32 in the chain probe (4 rows of
  // 8 limbs), 8 in the lo/hi and wide probes
  const double products = 5.0 * blocks * threads * double(iters) * 32.0;
  const double pairs_rate = products / 4.0 / (double(ms_pairs) * 1e-3);
  const double chain_rate = products / (double(ms_chain) * 1e-3);
  const double wide_rate = products / 4.0 / (double(ms_wide) * 1e-3);
  *word_products_per_second = std::max(pairs_rate, std::max(chain_rate, wide_rate));
  return CUHE_OK;
}

int cuhe_paillier_modexp(cuhe_paillier* ctx, const uint32_t* base, const uint32_t* exponent, int exponent_words,
                         uint32_t* out, int64_t count) {
  if (!ctx || count < 0 || !exponent || exponent_words <= 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (count == 0) return CUHE_OK;
  if (!base || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  // exponent of any width: build its schedule
  Limbs e(exponent, exponent + exponent_words);
  while (e.size() > 1 && e.back() == 0) e.pop_back();
  const PairModexp f52 = pair_modexp(ctx);
  int nops = 0;
  std::vector<int32_t> ops = f52 ? cuhe::host::pair_schedule(e, cuhe::kPairWindow, cuhe::kSplitWindow, &nops)
                                 : cuhe::host::window_schedule(e, ctx->window);
  if (!f52) nops = int(ops.size());
  if (!ops.empty()) {
    if (cudaError_t ce = ctx->tmp_ops.reserve(ops.size() * 4)) return cuda_fail(ctx, ce, "schedule allocation");
    CUHE_CUDA(ctx, cudaMemcpyAsync(ctx->tmp_ops.ptr, ops.data(), ops.size() * 4, cudaMemcpyHostToDevice, ctx->stream),
              "schedule upload");
  }
  const size_t bytes = size_t(count) * ctx->K * 4;
  Stager st(ctx);
  st.add(base, bytes, true, false);
  st.add(out, bytes, false, true);
  if (int rc = st.bind()) return rc;
  if (f52) {
    CUHE_CUDA(ctx, f52(ctx, (const uint32_t*)st.dev(0), nullptr, (uint32_t*)st.dev(1), count,
                       (const int32_t*)ctx->tmp_ops.ptr, nops, cuhe::EXP_POW, 0),
              "modexp launch");
  } else {
    CUHE_CUDA(ctx, d.modexp(ctx, (const uint32_t*)st.dev(0), nullptr, (uint32_t*)st.dev(1), count,
                            (const int32_t*)ctx->tmp_ops.ptr, nops, cuhe::EXP_POW, 0),
              "modexp launch");
  }
  if (int rc = st.finish()) return rc;
  // the schedule buffer is reused by the next call: keep host order
  if (!st.staged()) CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "modexp synchronize");
  return check_status(ctx, true);
}

int cuhe_paillier_modexp_each(cuhe_paillier* ctx, const uint32_t* base, const uint32_t* exponents,
                              int exponent_words, uint32_t* out, int64_t count) {
  if (!ctx || count < 0 || exponent_words <= 0 || exponent_words > ctx->K)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (count == 0) return CUHE_OK;
  if (!base || !exponents || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const size_t bytes = size_t(count) * ctx->K * 4;
  Stager st(ctx);
  st.add(base, bytes, true, false);
  st.add(exponents, size_t(count) * exponent_words * 4, true, false);
  st.add(out, bytes, false, true);
  if (int rc = st.bind()) return rc;
  CUHE_CUDA(ctx, d.modexp_var(ctx, (const uint32_t*)st.dev(0), (const uint32_t*)st.dev(1), exponent_words,
                              exponent_words * 8, (uint32_t*)st.dev(2), count),
            "modexp_each launch");
  if (int rc = st.finish()) return rc;
  return check_status(ctx, st.staged());
}

int cuhe_paillier_mulmod(cuhe_paillier* ctx, const uint32_t* a, const uint32_t* b, uint32_t* out, int64_t count) {
  if (!ctx || count < 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (count == 0) return CUHE_OK;
  if (!a || !b || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const size_t bytes = size_t(count) * ctx->K * 4;
  Stager st(ctx);
  st.add(a, bytes, true, false);
  st.add(b, bytes, true, false);
  st.add(out, bytes, false, true);
  if (int rc = st.bind()) return rc;
  CUHE_CUDA(ctx, d.mulmod(ctx, (const uint32_t*)st.dev(0), (const uint32_t*)st.dev(1), (uint32_t*)st.dev(2), count),
            "mulmod launch");
  if (int rc = st.finish()) return rc;
  return check_status(ctx, st.staged());
}

int cuhe_paillier_from_hex(cuhe_paillier* ctx, const char* text, const int64_t* offsets, int64_t count, int reduce,
                           uint32_t* out) {
  if (!ctx || count < 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (count == 0) return CUHE_OK;
  if (!text || !offsets || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  if (offsets[0] != 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "offsets must start at 0");
  for (int64_t i = 0; i < count; ++i)
    if (offsets[i + 1] < offsets[i]) return fail(ctx, CUHE_INVALID_ARGUMENT, "offsets must not decrease");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const size_t text_bytes = size_t(offsets[count]);
  const size_t bytes = size_t(count) * ctx->K * 4;
  Stager st(ctx);
  st.add(text, text_bytes ? text_bytes : 1, true, false);
  st.add(offsets, size_t(count + 1) * 8, true, false);
  st.add(out, bytes, false, true);
  if (int rc = st.bind()) return rc;
  const long long threads = count * ctx->K;
  cuhe::k_hex_to_limbs<<<unsigned((threads + 255) / 256), 256, 0, ctx->stream>>>(
      (const char*)st.dev(0), (const long long*)st.dev(1), count, ctx->K, (uint32_t*)st.dev(2), ctx->d_status);
  CUHE_CUDA(ctx, cudaGetLastError(), "hex parse launch");
  if (reduce) {
    // x mod n^2 for any x < 2^(32K): (x R mod n^2) R^-1
    CUHE_CUDA(ctx, d.convert(ctx, (const uint32_t*)st.dev(2), (uint32_t*)st.dev(2), count, 2), "reduce launch");
    CUHE_CUDA(ctx, d.convert(ctx, (const uint32_t*)st.dev(2), (uint32_t*)st.dev(2), count, 0), "reduce launch");
  }
  if (int rc = st.finish()) return rc;
  int status = 0;
  CUHE_CUDA(ctx, cudaMemcpyAsync(&status, ctx->d_status, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream), "status");
  CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "hex parse");
  if (status) {
    cudaMemsetAsync(ctx->d_status, 0, sizeof(int), ctx->stream);
    if (status & cuhe::ST_HEX) return fail(ctx, CUHE_INVALID_ARGUMENT, "Invalid hex digit");
    return fail(ctx, CUHE_RANGE, "input outside its valid range");
  }
  return CUHE_OK;
}

int cuhe_paillier_to_hex(cuhe_paillier* ctx, const uint32_t* limbs, int64_t count, char* out) {
  if (!ctx || count < 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (count == 0) return CUHE_OK;
  if (!limbs || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  const size_t words = size_t(ctx->K);
  Stager st(ctx);
  st.add(limbs, size_t(count) * words * 4, true, false);
  st.add(out, size_t(count) * words * 8, false, true);
  if (int rc = st.bind()) return rc;
  const long long threads = count * ctx->K;
  cuhe::k_limbs_to_hex<<<unsigned((threads + 255) / 256), 256, 0, ctx->stream>>>(
      (const uint32_t*)st.dev(0), count, ctx->K, (char*)st.dev(1));
  CUHE_CUDA(ctx, cudaGetLastError(), "hex format launch");
  if (int rc = st.finish()) return rc;
  CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "hex format");
  return CUHE_OK;
}

int cuhe_paillier_mulmod_outer(cuhe_paillier* ctx, const uint32_t* query, int64_t nq, const uint32_t* index,
                               int64_t nx, uint32_t* out) {
  if (!ctx || nq < 0 || nx < 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (nq == 0 || nx == 0) return CUHE_OK;
  if (!query || !index || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const size_t kb = size_t(ctx->K) * 4;
  const size_t obytes = size_t(nq) * size_t(nx) * kb;
  // A large host output moves in query-row blocks on the copy stream, each
  // block's download beside the next block's products.
  const bool pipe = obytes >= kPipeBytes && nq >= 2 && !is_device_pointer(out);
  const Outer52 f52 = outer52(ctx);
  Stager st(ctx);
  st.add(query, size_t(nq) * kb, true, false);
  st.add(index, size_t(nx) * kb, true, false);
  st.add(out, obytes, false, !pipe);
  st.add_scratch(size_t(nq) * (f52 ? size_t(ctx->K) * 5 : kb));  // queries in Montgomery form (words or 52-bit limbs)
  if (int rc = st.bind()) return rc;
  uint32_t* qm = static_cast<uint32_t*>(st.dev(3));
  uint32_t* d_out = static_cast<uint32_t*>(st.dev(2));
  // the FP64 form converts each query block inside its launch
  auto outer = [&](int64_t q0, int64_t qn, uint32_t* o) -> cudaError_t {
    if (f52)
      return f52(ctx, (const uint32_t*)st.dev(0) + size_t(q0) * ctx->K, qn,
                 reinterpret_cast<double*>(qm) + size_t(q0) * (5 * size_t(ctx->K) / 8), (const uint32_t*)st.dev(1),
                 nx, o);
    return d.outer(ctx, qm + size_t(q0) * ctx->K, qn, (const uint32_t*)st.dev(1), nx, o);
  };
  if (!f52) CUHE_CUDA(ctx, d.convert(ctx, (const uint32_t*)st.dev(0), qm, nq, 1), "query conversion");
  if (pipe && st.is_staged(2)) {
    if (int rc = pipeline_streams(ctx)) return rc;
    const int64_t rows = std::max<int64_t>(1, nq / 8);
    const size_t row_words = size_t(nx) * ctx->K;
    for (int64_t q0 = 0; q0 < nq; q0 += rows) {
      const int64_t qn = std::min(rows, nq - q0);
      CUHE_CUDA(ctx, outer(q0, qn, d_out + size_t(q0) * row_words), "mulmod_outer launch");
      CUHE_CUDA(ctx, stream_after(ctx->copy, ctx->stream), "download order");
      CUHE_CUDA(ctx, cudaMemcpyAsync(out + size_t(q0) * row_words, d_out + size_t(q0) * row_words,
                                     size_t(qn) * row_words * 4, cudaMemcpyDeviceToHost, ctx->copy),
                "piecewise download");
    }
    CUHE_CUDA(ctx, stream_after(ctx->stream, ctx->copy), "download join");
  } else {
    CUHE_CUDA(ctx, outer(0, nq, d_out), "mulmod_outer launch");
  }
  if (int rc = st.finish()) return rc;
  // the scratch slice is reused by the next call: keep host order
  if (!st.staged()) CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "mulmod_outer synchronize");
  return check_status(ctx, true);
}

}  // extern "C"

namespace {

bool capturing(const cuhe_paillier* ctx) {
  cudaStreamCaptureStatus st = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(ctx->stream, &st) != cudaSuccess || st != cudaStreamCaptureStatusNone;
}

// One table of rows: allocate, then build on the context's stream and wait (a
// later call may use another stream).  A table that does not fit, or is first
// wanted under stream capture, leaves *out null (CUHE_OK: another one serves
// the call).
template <class Build>
int pair_table(cuhe_paillier* ctx, double2** out, long long rows, Build build) {
  if (*out || capturing(ctx)) return CUHE_OK;
  double2* t = nullptr;
  if (cudaMalloc(&t, size_t(rows) * size_t(5 * ctx->K / 16) * 16) != cudaSuccess) {
    cudaGetLastError();
    return CUHE_OK;
  }
  cudaError_t e = build(t);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) {
    cudaFree(t);
    return cuda_fail(ctx, e, "lookup table build");
  }
  *out = t;
  return CUHE_OK;
}

// The 8-bit digit, embedding and noise rows (65,536 + 32,768 + 256 rows at
// key_len 1024, 63 MB): made when tables are installed, or by the first call
// after the pipe was changed.
int pair_tables(cuhe_paillier* ctx, const PairLookup& pl) {
  auto& pt = ctx->pt;
  const int chunks = ctx->message_chunks, entries = ctx->noise_entries, rows8 = (chunks + 1) / 2;
  if (chunks == 0 || entries == 0 || (pt.digits && pt.noise && pt.embed)) return CUHE_OK;
  if (capturing(ctx)) return CUHE_OK;
  if (!ctx->d_entry) {  // R^(j+2) 2^(-32K) mod n^2 as pairs
    const size_t k = size_t(ctx->K), kl = 5 * k / 16;
    Limbs n = ctx->n;
    while (n.size() > 1 && n.back() == 0) n.pop_back();
    Limbs x(k, 0u);
    x[0] = 1u;
    x = cuhe::host::shift_mod(x, 52 * kl, ctx->n2);
    for (size_t i = 0; i < 32 * k; ++i) cuhe::host::half_mod(x, ctx->n2);
    std::vector<double> block(4 * kl, 0.0);
    for (int j = 0; j < 2; ++j) {
      x = cuhe::host::shift_mod(x, 52 * kl, ctx->n2);
      Limbs quotient;
      const Limbs rem = cuhe::host::mod_reduce(x, n, &quotient);
      balanced52(rem, kl, block.data() + size_t(j) * 2 * kl, 2);
      balanced52(quotient, kl, block.data() + size_t(j) * 2 * kl + 1, 2);
    }
    if (int rc = upload_constants(ctx, block, reinterpret_cast<double**>(&ctx->d_entry))) return rc;
  }
  if (int rc = pair_table(ctx, &pt.digits, (long long)chunks * 256, [&](double2* t) {
        return pl.rows(ctx, ctx->d_gtab, (long long)chunks * 256, true, t);
      }))
    return rc;
  if (int rc = pair_table(ctx, &pt.noise, entries,
                          [&](double2* t) { return pl.rows(ctx, ctx->d_noise, entries, false, t); }))
    return rc;
  if (!pt.digits) return CUHE_OK;
  return pair_table(ctx, &pt.embed, (long long)rows8 * 256, [&](double2* t) {
    return pl.products(ctx, pt.digits, chunks, cuhe::kEmbed, 0, (long long)rows8 * 256, t);
  });
}

}  // namespace

extern "C" {

int cuhe_lookup_set_tables(cuhe_paillier* ctx, const uint32_t* g_table, int message_chunks, const uint32_t* noise,
                           int noise_entries) {
  if (!ctx || !g_table || !noise || message_chunks <= 0 || noise_entries <= 0 || noise_entries > 256)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid tables");
  if (message_chunks * 256 > 65536) return fail(ctx, CUHE_INVALID_ARGUMENT, "too many message chunks");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const size_t kb = size_t(ctx->K) * 4;
  const size_t gbytes = size_t(message_chunks) * 256 * kb;
  cudaFree(ctx->d_gtab);
  cudaFree(ctx->d_noise);
  cudaFree(ctx->d_wide);
  ctx->pt.release();
  ctx->d_gtab = nullptr;
  ctx->d_noise = nullptr;
  ctx->d_wide = nullptr;
  ctx->message_chunks = 0;
  ctx->noise_entries = 0;
  CUHE_CUDA(ctx, cudaMalloc(&ctx->d_gtab, gbytes), "table allocation");
  CUHE_CUDA(ctx, cudaMalloc(&ctx->d_noise, size_t(noise_entries) * kb), "table allocation");
  Stager st(ctx);
  st.add(g_table, gbytes, true, false);
  st.add(noise, size_t(noise_entries) * kb, true, false);
  if (int rc = st.bind()) return rc;
  CUHE_CUDA(ctx, d.convert(ctx, (const uint32_t*)st.dev(0), ctx->d_gtab, (long long)message_chunks * 256, 1),
            "table conversion");
  CUHE_CUDA(ctx, d.convert(ctx, (const uint32_t*)st.dev(1), ctx->d_noise, noise_entries, 1), "table conversion");
  CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "table synchronize");
  if (int rc = check_status(ctx, true)) return rc;
  ctx->message_chunks = message_chunks;
  ctx->noise_entries = noise_entries;
  PairLookup pl{};
  return pair_lookup(ctx, &pl) ? pair_tables(ctx, pl) : CUHE_OK;
}

int cuhe_lookup_build_tables(cuhe_paillier* ctx, const uint32_t* g, int message_chunks, const uint32_t* noise,
                             int noise_entries) {
  if (!ctx || !g || message_chunks <= 0 || message_chunks * 256 > 65536)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid table request");
  if (noise && (noise_entries <= 0 || noise_entries > 256)) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid noise");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const size_t k = size_t(ctx->K), kb = k * 4;
  // base_i = g^(2^(8i)) for all rows: one batched modexp per row exponent is
  // wasteful; square on the device 8 times per row in one group instead.
  std::vector<uint32_t> gk(k, 0u);
  std::memcpy(gk.data(), g, kb);  // caller passes K words
  DeviceBuffer bases, gdev, pows;
  CUHE_CUDA(ctx, bases.reserve(size_t(message_chunks) * kb), "table scratch");
  CUHE_CUDA(ctx, gdev.reserve(kb), "table scratch");
  CUHE_CUDA(ctx, cudaMemcpyAsync(gdev.ptr, gk.data(), kb, cudaMemcpyHostToDevice, ctx->stream), "upload g");
  // bases: row i = g^(2^(8i)); computed as a batched modexp over rows with
  // per-row exponent 2^(8i) is not fixed-exponent, so use successive
  // fixed-exponent launches of 2^8 on the previous row (message_chunks launches).
  std::vector<int32_t> ops256 = cuhe::host::window_schedule(Limbs{256u}, ctx->window);
  CUHE_CUDA(ctx, pows.reserve(ops256.size() * 4), "table scratch");
  CUHE_CUDA(ctx, cudaMemcpyAsync(pows.ptr, ops256.data(), ops256.size() * 4, cudaMemcpyHostToDevice, ctx->stream),
            "upload schedule");
  uint32_t* b = static_cast<uint32_t*>(bases.ptr);
  CUHE_CUDA(ctx, cudaMemcpyAsync(b, gdev.ptr, kb, cudaMemcpyDeviceToDevice, ctx->stream), "row 0");
  for (int i = 1; i < message_chunks; ++i) {
    CUHE_CUDA(ctx, d.modexp(ctx, b + (i - 1) * k, nullptr, b + i * k, 1, (const int32_t*)pows.ptr, int(ops256.size()),
                            cuhe::EXP_POW, 0),
              "row base");
  }
  // to Montgomery form, then fill rows
  DeviceBuffer bm;
  CUHE_CUDA(ctx, bm.reserve(size_t(message_chunks) * kb), "table scratch");
  CUHE_CUDA(ctx, d.convert(ctx, b, (uint32_t*)bm.ptr, message_chunks, 1), "row conversion");
  cudaFree(ctx->d_gtab);
  cudaFree(ctx->d_wide);
  ctx->pt.release();
  ctx->d_gtab = nullptr;
  ctx->d_wide = nullptr;
  ctx->message_chunks = 0;
  CUHE_CUDA(ctx, cudaMalloc(&ctx->d_gtab, size_t(message_chunks) * 256 * kb), "table allocation");
  CUHE_CUDA(ctx, d.table_rows(ctx, (const uint32_t*)bm.ptr, message_chunks, ctx->d_gtab), "table rows");
  if (noise) {
    cudaFree(ctx->d_noise);
    ctx->d_noise = nullptr;
    ctx->noise_entries = 0;
    CUHE_CUDA(ctx, cudaMalloc(&ctx->d_noise, size_t(noise_entries) * kb), "noise allocation");
    Stager st(ctx);
    st.add(noise, size_t(noise_entries) * kb, true, false);
    if (int rc = st.bind()) return rc;
    CUHE_CUDA(ctx, d.convert(ctx, (const uint32_t*)st.dev(0), ctx->d_noise, noise_entries, 1), "noise conversion");
  }
  CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "table synchronize");
  bases.release();
  gdev.release();
  pows.release();
  bm.release();
  if (int rc = check_status(ctx, true)) return rc;
  ctx->message_chunks = message_chunks;
  if (noise) ctx->noise_entries = noise_entries;
  PairLookup pl{};
  return pair_lookup(ctx, &pl) ? pair_tables(ctx, pl) : CUHE_OK;
}

int cuhe_lookup_get_g_table(cuhe_paillier* ctx, uint32_t* out) {
  if (!ctx || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  if (!ctx->d_gtab) return fail(ctx, CUHE_NOT_READY, "tables not installed");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const long long entries = (long long)ctx->message_chunks * 256;
  Stager st(ctx);
  st.add(out, size_t(entries) * ctx->K * 4, false, true);
  if (int rc = st.bind()) return rc;
  CUHE_CUDA(ctx, d.convert(ctx, ctx->d_gtab, (uint32_t*)st.dev(0), entries, 0), "table export");
  if (int rc = st.finish()) return rc;
  CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "table export");
  return check_status(ctx, true);
}

}  // extern "C"

namespace {

// Device bytes of one 65,536-entry row of the wide tables: words, limb pairs.
size_t wide_word_row(const cuhe_paillier* ctx) { return size_t(65536) * size_t(ctx->K) * 4; }
size_t wide_pair_row(const cuhe_paillier* ctx) { return size_t(65536) * size_t(5 * ctx->K / 16) * 16; }

// Whether a wide table may take `bytes` more.  Under the default policy all of
// them together (the words', the digits' and the embeddings') stay within
// kWideMaxBytes and a quarter of the memory that would be free without them.
int wide_allowed(cuhe_paillier* ctx, long long items, size_t bytes, bool* allowed) {
  *allowed = ctx->wide_mode == 2;
  if (ctx->wide_mode != 1 || items < kWideMinItems) return CUHE_OK;
  const size_t digit_rows = size_t(ctx->message_chunks + 1) / 2;
  const size_t held = (ctx->d_wide ? digit_rows * wide_word_row(ctx) : 0) +
                      ((ctx->pt.wide_digits ? digit_rows : 0) + size_t(ctx->pt.wide_rows)) * wide_pair_row(ctx);
  if (held + bytes > kWideMaxBytes) return CUHE_OK;
  size_t free_bytes = 0, total_bytes = 0;
  CUHE_CUDA(ctx, cudaMemGetInfo(&free_bytes, &total_bytes), "free memory");
  *allowed = held + bytes <= (free_bytes + held) / 4;
  return CUHE_OK;
}

// The integer kernel's 16-bit-digit table; under stream capture, where nothing
// may be allocated, the 8-bit table serves.
int ensure_wide_table(cuhe_paillier* ctx, const Dispatch& d, long long items) {
  if (ctx->d_wide || !ctx->d_gtab || capturing(ctx)) return CUHE_OK;
  const size_t bytes = size_t((ctx->message_chunks + 1) / 2) * wide_word_row(ctx);
  bool allowed = false;
  if (int rc = wide_allowed(ctx, items, bytes, &allowed)) return rc;
  if (!allowed) return CUHE_OK;
  void* wide = nullptr;
  if (cudaMalloc(&wide, bytes) != cudaSuccess) {
    cudaGetLastError();
    if (ctx->wide_mode == 2) return fail(ctx, CUHE_OUT_OF_MEMORY, "wide table allocation");
    return CUHE_OK;
  }
  if (cudaError_t e = d.wide_table(ctx, static_cast<uint32_t*>(wide))) {
    cudaFree(wide);
    return cuda_fail(ctx, e, "wide table build");
  }
  ctx->d_wide = static_cast<uint32_t*>(wide);
  return CUHE_OK;
}

// Noise products of two repay their table (noise_entries^2 products, seven
// saved by a ciphertext) from this many ciphertexts in one call; mode 0, which
// asks for the small tables alone, does without.
constexpr long long kNoisePairItems = 8192;

// Rows [wide_rows, need) of the 16-bit embedding table (of the 8-bit table's
// rows8), in an allocation of their own.  Without memory for them the table
// stays as it is (CUHE_OUT_OF_MEMORY in mode 2).
int grow_embed_rows(cuhe_paillier* ctx, const PairLookup& pl, int rows8, int need) {
  auto& pt = ctx->pt;
  const int before = pt.wide_rows, added = need - before;
  const size_t entries = wide_pair_row(ctx) / sizeof(double2);  // pairs of a row
  double2* block = nullptr;
  cudaError_t e = pt.embed_rows ? cudaSuccess : cudaMalloc(&pt.embed_rows, size_t((rows8 + 1) / 2) * sizeof(double2*));
  if (e == cudaSuccess) e = cudaMalloc(&block, size_t(added) * entries * sizeof(double2));
  if (e != cudaSuccess) {
    cudaGetLastError();
    return ctx->wide_mode == 2 ? fail(ctx, CUHE_OUT_OF_MEMORY, "wide table allocation") : CUHE_OK;
  }
  std::vector<const double2*> rows;
  for (int r = 0; r < added; ++r) rows.push_back(block + size_t(r) * entries);
  e = pl.products(ctx, pt.embed, rows8, cuhe::kWide, (long long)before * 65536, (long long)added * 65536, block);
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(pt.embed_rows + before, rows.data(), rows.size() * sizeof(double2*), cudaMemcpyHostToDevice,
                        ctx->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(ctx->stream);
  if (e != cudaSuccess) {
    cudaFree(block);
    return cuda_fail(ctx, e, "wide table build");
  }
  pt.wide_blocks.push_back(block);
  pt.wide_rows = need;
  return CUHE_OK;
}

// Encryption from the limb-pair tables, building those the call needs; *done
// is false (nothing launched) when they do not fit in device memory.
int pair_lookup_encrypt(cuhe_paillier* ctx, const PairLookup& pl, cuhe::LookupDigits dg, long long count,
                        const uint8_t* idx, uint32_t* out, bool* done) {
  *done = false;
  auto& pt = ctx->pt;
  const int chunks = ctx->message_chunks, entries = ctx->noise_entries;
  if (int rc = pair_tables(ctx, pl)) return rc;
  if (!pt.digits || !pt.noise) return CUHE_OK;
  if (count >= kNoisePairItems && ctx->wide_mode != 0)
    if (int rc = pair_table(ctx, &pt.noise2, (long long)entries * entries, [&](double2* t) {
          return pl.products(ctx, pt.noise, entries, cuhe::kNoise, 0, (long long)entries * entries, t);
        }))
      return rc;
  const double2* table = pt.digits;
  dg.message_chunks = chunks;
  dg.rows = chunks;
  dg.wide = dg.embed_bits = 0;
  bool allowed = false;
  if (dg.bits && dg.chunk_len % 2 == 0 && pt.embed) {
    const int rows8 = (chunks + 1) / 2;
    // rows that this call's chunks reach (32 plaintext bits each)
    const int reach = std::min(2 * dg.embed_len, dg.chunk_len);
    const int need8 = std::min(rows8, (reach + 15) / 16), need = (need8 + 1) / 2;
    if (pt.wide_rows < need && !capturing(ctx)) {
      if (int rc = wide_allowed(ctx, count, size_t(need - pt.wide_rows) * wide_pair_row(ctx), &allowed)) return rc;
      if (allowed)
        if (int rc = grow_embed_rows(ctx, pl, rows8, need)) return rc;
    }
    const bool wide = pt.wide_rows >= need && pt.wide_rows;
    dg.embed_bits = wide ? 16 : 8;
    dg.rows = wide ? need : need8;
    dg.embed_rows = wide ? pt.embed_rows : nullptr;
    table = pt.embed;
  } else {
    const int rows = (chunks + 1) / 2;
    if (!pt.wide_digits && !capturing(ctx)) {
      if (int rc = wide_allowed(ctx, count, size_t(rows) * wide_pair_row(ctx), &allowed)) return rc;
      if (allowed) {
        if (int rc = pair_table(ctx, &pt.wide_digits, (long long)rows * 65536, [&](double2* t) {
              return pl.products(ctx, pt.digits, chunks, cuhe::kWide, 0, (long long)rows * 65536, t);
            }))
          return rc;
        if (!pt.wide_digits && ctx->wide_mode == 2) return fail(ctx, CUHE_OUT_OF_MEMORY, "wide table allocation");
      }
    }
    if (pt.wide_digits) {
      dg.wide = 1;
      dg.rows = rows;
      table = pt.wide_digits;
    }
  }
  // a short table's pairs are complete for every valid index; with any other
  // the call reports the range error
  const bool pairs = pt.noise2 != nullptr;
  cudaError_t e = pl.launch(ctx, dg, count, table, pairs ? pt.noise2 : pt.noise, pairs, idx, out);
  if (e != cudaSuccess) return cuda_fail(ctx, e, "lookup encrypt launch");
  *done = true;
  return CUHE_OK;
}

}  // namespace

extern "C" {

int cuhe_lookup_set_wide_table(cuhe_paillier* ctx, int mode) {
  if (!ctx || mode < 0 || mode > 2) return fail(ctx, CUHE_INVALID_ARGUMENT, "wide table mode must be 0, 1 or 2");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  ctx->wide_mode = mode;
  if (mode == 0 && (ctx->d_wide || ctx->pt.wide() || ctx->pt.noise2)) {
    CUHE_CUDA(ctx, cudaStreamSynchronize(ctx->stream), "wide table release");
    cudaFree(ctx->d_wide);
    ctx->d_wide = nullptr;
    ctx->pt.release_wide();
  }
  return CUHE_OK;
}

int cuhe_lookup_wide_table_ready(const cuhe_paillier* ctx) { return ctx && (ctx->d_wide || ctx->pt.wide()) ? 1 : 0; }

int cuhe_lookup_encrypt_bits(cuhe_paillier* ctx, const uint8_t* bits, int64_t vectors, int embed_len, int chunk_len,
                             int chunk_num, const uint8_t* noise_index, uint32_t* out) {
  if (!ctx || vectors < 0 || embed_len <= 0 || chunk_len <= 0 || chunk_num <= 0)
    return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid layout");
  if (!ctx->d_gtab || !ctx->d_noise) return fail(ctx, CUHE_NOT_READY, "lookup tables not installed");
  if (int64_t(chunk_num) * chunk_len < 2 * int64_t(embed_len))
    return fail(ctx, CUHE_INVALID_ARGUMENT, "chunks do not cover the padded embedding");
  if (vectors == 0) return CUHE_OK;
  if (!bits || !noise_index || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  const int64_t total = vectors * chunk_num;
  PairLookup pl{};
  const bool pairs = pair_lookup(ctx, &pl);
  Stager st(ctx);
  st.add(bits, size_t(vectors) * embed_len, true, false);
  st.add(noise_index, size_t(total) * cuhe::kNoiseMultiples, true, false);
  st.add(out, size_t(total) * ctx->K * 4, false, true);
  if (int rc = st.bind()) return rc;
  bool done = false;
  if (pairs) {
    cuhe::LookupDigits dg{};
    dg.bits = (const uint8_t*)st.dev(0);
    dg.embed_len = embed_len;
    dg.chunk_len = chunk_len;
    dg.chunk_num = chunk_num;
    if (int rc = pair_lookup_encrypt(ctx, pl, dg, total, (const uint8_t*)st.dev(1), (uint32_t*)st.dev(2), &done))
      return rc;
  }
  if (!done) {
    if (int rc = ensure_wide_table(ctx, d, total)) return rc;
    CUHE_CUDA(ctx, d.lookup(ctx, (const uint8_t*)st.dev(0), embed_len, chunk_len, chunk_num, nullptr, total,
                            (const uint8_t*)st.dev(1), (uint32_t*)st.dev(2)),
              "lookup encrypt launch");
  }
  if (int rc = st.finish()) return rc;
  return check_status(ctx, st.staged());
}

int cuhe_lookup_encrypt_ints(cuhe_paillier* ctx, const uint32_t* m, int64_t count, const uint8_t* noise_index,
                             uint32_t* out) {
  if (!ctx || count < 0) return fail(ctx, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (!ctx->d_gtab || !ctx->d_noise) return fail(ctx, CUHE_NOT_READY, "lookup tables not installed");
  if (count == 0) return CUHE_OK;
  if (!m || !noise_index || !out) return fail(ctx, CUHE_INVALID_ARGUMENT, "null buffer");
  DeviceGuard guard(ctx->device);
  std::lock_guard<std::mutex> lock(ctx->mu);
  Dispatch d;
  find_dispatch(ctx->K, ctx->tpi, ctx->window, &d);
  PairLookup pl{};
  const bool pairs = pair_lookup(ctx, &pl);
  Stager st(ctx);
  st.add(m, size_t(count) * ctx->K * 4, true, false);
  st.add(noise_index, size_t(count) * cuhe::kNoiseMultiples, true, false);
  st.add(out, size_t(count) * ctx->K * 4, false, true);
  if (int rc = st.bind()) return rc;
  bool done = false;
  if (pairs) {
    cuhe::LookupDigits dg{};
    dg.plain = (const uint32_t*)st.dev(0);
    dg.plain_words = ctx->K;
    dg.chunk_num = 1;
    if (int rc = pair_lookup_encrypt(ctx, pl, dg, count, (const uint8_t*)st.dev(1), (uint32_t*)st.dev(2), &done))
      return rc;
  }
  if (!done) {
    if (int rc = ensure_wide_table(ctx, d, count)) return rc;
    CUHE_CUDA(ctx, d.lookup(ctx, nullptr, 0, 0, 1, (const uint32_t*)st.dev(0), count, (const uint8_t*)st.dev(1),
                            (uint32_t*)st.dev(2)),
              "lookup encrypt launch");
  }
  if (int rc = st.finish()) return rc;
  return check_status(ctx, st.staged());
}

}  // extern "C"

// ---------------------------------------------------------------------------
// Mixed batches: many (key, exponent, bases) exponentiations of uneven sizes
// and widths in one persistent launch per width.
// ---------------------------------------------------------------------------
struct cuhe_mix {
  struct Entry {
    cuhe_paillier* ctx;
    const uint32_t* base;
    uint32_t* out;
    long long count;
    Limbs exponent;
  };
  struct Width {
    int K = 0, tpi = 0, window = 0, grid = 0, ntasks = 0;
    long long units = 0;
    cuhe::ModexpTask* d_tasks = nullptr;
    std::vector<int32_t*> d_ops;
    Dispatch d;
    bool fp52 = false;  // k_pair_modexp_tasks: every context of the width selects the FP64 pipe
    cudaError_t (*prepare)(int, int*) = nullptr;
    cudaError_t (*launch)(const cuhe::ModexpTask*, int, long long, unsigned long long*, int*, int,
                          cudaStream_t) = nullptr;
  };
  int device = 0;
  std::vector<Entry> entries;
  std::map<int, std::pair<int, int>> tuning;  // K -> (tpi, window)
  std::vector<Width> widths;
  unsigned long long* d_counters = nullptr;
  int* d_status = nullptr;
  bool planned = false;
  std::string error;
  // widths after the first run on their own streams, forked from and joined
  // back to the launch stream, so that one width's last wave overlaps the
  // next width's kernel (created by the plan: a launch allocates nothing)
  std::vector<cudaStream_t> side;
  std::vector<cudaEvent_t> done;
  cudaEvent_t fork = nullptr;

  void release_plan() {
    for (auto& w : widths) {
      cudaFree(w.d_tasks);
      for (int32_t* p : w.d_ops) cudaFree(p);
    }
    widths.clear();
    cudaFree(d_counters);
    d_counters = nullptr;
    for (cudaStream_t st : side) cudaStreamDestroy(st);
    for (cudaEvent_t ev : done) cudaEventDestroy(ev);
    side.clear();
    done.clear();
    if (fork) cudaEventDestroy(fork);
    fork = nullptr;
    planned = false;
  }
};

namespace {
int mix_fail(cuhe_mix* mix, int code, const std::string& msg) {
  if (mix) mix->error = msg; else g_create_error = msg;
  return code;
}
}  // namespace

extern "C" {

const char* cuhe_mix_last_error(const cuhe_mix* mix) { return mix ? mix->error.c_str() : g_create_error.c_str(); }

int cuhe_mix_create(int device, cuhe_mix** out) {
  if (!out) return mix_fail(nullptr, CUHE_INVALID_ARGUMENT, "null output");
  *out = nullptr;
  int count = 0;
  if (cudaGetDeviceCount(&count) != cudaSuccess || device < 0 || device >= count) {
    cudaGetLastError();
    return mix_fail(nullptr, CUHE_INVALID_ARGUMENT, "invalid device ordinal");
  }
  auto* mix = new (std::nothrow) cuhe_mix();
  if (!mix) return mix_fail(nullptr, CUHE_OUT_OF_MEMORY, "mix allocation");
  mix->device = device;
  DeviceGuard guard(device);
  if (cudaMalloc(&mix->d_status, sizeof(int)) != cudaSuccess || cudaMemset(mix->d_status, 0, sizeof(int)) != cudaSuccess) {
    cudaGetLastError();
    delete mix;
    return mix_fail(nullptr, CUHE_OUT_OF_MEMORY, "mix status allocation");
  }
  *out = mix;
  return CUHE_OK;
}

void cuhe_mix_destroy(cuhe_mix* mix) {
  if (!mix) return;
  DeviceGuard guard(mix->device);
  cudaDeviceSynchronize();
  mix->release_plan();
  cudaFree(mix->d_status);
  delete mix;
}

int cuhe_mix_add_modexp(cuhe_mix* mix, cuhe_paillier* ctx, const uint32_t* base, uint32_t* out, int64_t count,
                        const uint32_t* exponent, int exponent_words) {
  if (!mix || !ctx || !exponent || exponent_words <= 0 || count < 0)
    return mix_fail(mix, CUHE_INVALID_ARGUMENT, "invalid argument");
  if (ctx->device != mix->device) return mix_fail(mix, CUHE_INVALID_ARGUMENT, "context on another device");
  if (count == 0) return CUHE_OK;
  DeviceGuard guard(mix->device);
  if (!is_device_pointer(base) || !is_device_pointer(out))
    return mix_fail(mix, CUHE_INVALID_ARGUMENT, "mixed batches take device buffers");
  if (!cuhe::host::fits(exponent, size_t(exponent_words), size_t(ctx->K)))
    return mix_fail(mix, CUHE_INVALID_ARGUMENT, "exponent wider than n^2");
  mix->entries.push_back({ctx, base, out, count, cuhe::host::resized(exponent, size_t(exponent_words), size_t(ctx->K))});
  mix->planned = false;
  return CUHE_OK;
}

int cuhe_mix_set_tuning(cuhe_mix* mix, int words, int tpi, int window) {
  if (!mix) return CUHE_INVALID_ARGUMENT;
  Dispatch d;
  if (!find_dispatch(words, tpi, window, &d))
    return mix_fail(mix, CUHE_INVALID_ARGUMENT, "tuning (threads per instance, window) not compiled for this width");
  mix->tuning[words] = {tpi, window};
  mix->planned = false;
  return CUHE_OK;
}

int cuhe_mix_plan(cuhe_mix* mix) {
  if (!mix) return CUHE_INVALID_ARGUMENT;
  DeviceGuard guard(mix->device);
  cudaDeviceSynchronize();
  mix->release_plan();
  std::map<int, std::vector<size_t>> by_width;
  for (size_t i = 0; i < mix->entries.size(); ++i) by_width[mix->entries[i].ctx->K].push_back(i);
  for (auto& kv : by_width) {
    cuhe_mix::Width w;
    w.K = kv.first;
    auto it = mix->tuning.find(w.K);
    if (it != mix->tuning.end()) {
      w.tpi = it->second.first;
      w.window = it->second.second;
    } else {
      default_tuning(w.K, &w.tpi, &w.window);
    }
    if (!find_dispatch(w.K, w.tpi, w.window, &w.d)) return mix_fail(mix, CUHE_INVALID_ARGUMENT, "no compiled variant");
    // the pipe follows the contexts, as their one-launch-per-batch calls do
    w.fp52 = true;
    for (size_t i : kv.second) w.fp52 = w.fp52 && pair_modexp(mix->entries[i].ctx) != nullptr;
    w.prepare = w.d.prepare_tasks;
    w.launch = w.d.launch_tasks;
    if (w.fp52) {
      w.window = cuhe::kPairWindow;
      w.tpi = w.K / 32;
      if (w.K == 64) { w.prepare = &prepare_pair_tasks<64>; w.launch = &launch_pair_tasks<64>; }
      if (w.K == 128) { w.prepare = &prepare_pair_tasks<128>; w.launch = &launch_pair_tasks<128>; }
      if (w.K == 256) { w.prepare = &prepare_pair_tasks<256>; w.launch = &launch_pair_tasks<256>; }
    }
    const long long ipb = cuhe::kBlockThreads / w.tpi;
    std::vector<cuhe::ModexpTask> tasks;
    for (size_t i : kv.second) {
      const auto& e = mix->entries[i];
      std::vector<int32_t> ops = cuhe::host::window_schedule(e.exponent, w.window);
      int32_t* d_ops = nullptr;
      if (!ops.empty()) {
        if (cudaMalloc(&d_ops, ops.size() * 4) != cudaSuccess ||
            cudaMemcpy(d_ops, ops.data(), ops.size() * 4, cudaMemcpyHostToDevice) != cudaSuccess) {
          cudaGetLastError();
          cudaFree(d_ops);
          return mix_fail(mix, CUHE_OUT_OF_MEMORY, "schedule upload");
        }
        w.d_ops.push_back(d_ops);
      }
      cuhe::ModexpTask t{};
      t.base = e.base;
      t.out = e.out;
      t.count = e.count;
      t.consts = e.ctx->d_consts;
      t.ops = d_ops;
      t.first_unit = w.units;
      t.ks = e.ctx->ks;
      t.nops = int(ops.size());
      t.mode = cuhe::EXP_POW;
      t.n52 = e.ctx->d_pair;
      t.ninv52 = e.ctx->pair_ninv;
      tasks.push_back(t);
      w.units += (e.count + ipb - 1) / ipb;
    }
    w.ntasks = int(tasks.size());
    if (cudaMalloc(&w.d_tasks, tasks.size() * sizeof(cuhe::ModexpTask)) != cudaSuccess ||
        cudaMemcpy(w.d_tasks, tasks.data(), tasks.size() * sizeof(cuhe::ModexpTask), cudaMemcpyHostToDevice) !=
            cudaSuccess) {
      cudaGetLastError();
      return mix_fail(mix, CUHE_OUT_OF_MEMORY, "task table upload");
    }
    cudaError_t e = w.prepare(mix->device, &w.grid);
    if (e != cudaSuccess) return mix_fail(mix, CUHE_CUDA_ERROR, std::string("mixed launch setup: ") + cudaGetErrorString(e));
    mix->widths.push_back(std::move(w));
  }
  if (!mix->widths.empty() &&
      cudaMalloc(&mix->d_counters, mix->widths.size() * sizeof(unsigned long long)) != cudaSuccess) {
    cudaGetLastError();
    return mix_fail(mix, CUHE_OUT_OF_MEMORY, "counter allocation");
  }
  if (mix->widths.size() > 1) {
    if (cudaEventCreateWithFlags(&mix->fork, cudaEventDisableTiming) != cudaSuccess)
      return mix_fail(mix, CUHE_CUDA_ERROR, "mixed launch events");
    for (size_t i = 1; i < mix->widths.size(); ++i) {
      cudaStream_t st = nullptr;
      cudaEvent_t ev = nullptr;
      if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess)
        return mix_fail(mix, CUHE_CUDA_ERROR, "mixed launch streams");
      mix->side.push_back(st);
      if (cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) != cudaSuccess)
        return mix_fail(mix, CUHE_CUDA_ERROR, "mixed launch events");
      mix->done.push_back(ev);
    }
  }
  mix->planned = true;
  return CUHE_OK;
}

int cuhe_mix_launch(cuhe_mix* mix, void* stream) {
  if (!mix) return CUHE_INVALID_ARGUMENT;
  if (!mix->planned) return mix_fail(mix, CUHE_NOT_READY, "mixed batch not planned");
  if (mix->widths.empty()) return CUHE_OK;
  DeviceGuard guard(mix->device);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaError_t e = cudaMemsetAsync(mix->d_counters, 0, mix->widths.size() * sizeof(unsigned long long), s);
  if (e == cudaSuccess && mix->fork) e = cudaEventRecord(mix->fork, s);
  for (size_t i = 0; i < mix->widths.size() && e == cudaSuccess; ++i) {
    const auto& w = mix->widths[i];
    cudaStream_t ws = i == 0 ? s : mix->side[i - 1];
    if (i > 0) e = cudaStreamWaitEvent(ws, mix->fork, 0);
    if (e == cudaSuccess)
      e = w.launch(w.d_tasks, w.ntasks, w.units, mix->d_counters + i, mix->d_status, w.grid, ws);
    if (e == cudaSuccess && i > 0) e = cudaEventRecord(mix->done[i - 1], ws);
    if (e == cudaSuccess && i > 0) e = cudaStreamWaitEvent(s, mix->done[i - 1], 0);
  }
  if (e != cudaSuccess) return mix_fail(mix, CUHE_CUDA_ERROR, std::string("mixed launch: ") + cudaGetErrorString(e));
  return CUHE_OK;
}

int cuhe_mix_check(cuhe_mix* mix) {
  if (!mix) return CUHE_INVALID_ARGUMENT;
  DeviceGuard guard(mix->device);
  int status = 0;
  cudaError_t e = cudaDeviceSynchronize();
  if (e == cudaSuccess) e = cudaMemcpy(&status, mix->d_status, sizeof(int), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return mix_fail(mix, CUHE_CUDA_ERROR, std::string("mixed batch: ") + cudaGetErrorString(e));
  if (status) {
    cudaMemset(mix->d_status, 0, sizeof(int));
    return mix_fail(mix, CUHE_RANGE, "input outside its valid range (base >= n^2)");
  }
  return CUHE_OK;
}

int cuhe_mix_info(const cuhe_mix* mix, int index, int* words, int* tpi, int* window, int* grid, int64_t* units,
                  int* tasks) {
  if (!mix || index < 0 || size_t(index) >= mix->widths.size()) return CUHE_INVALID_ARGUMENT;
  const auto& w = mix->widths[size_t(index)];
  if (words) *words = w.K;
  if (tpi) *tpi = w.tpi;
  if (window) *window = w.window;
  if (grid) *grid = w.grid;
  if (units) *units = w.units;
  if (tasks) *tasks = w.ntasks;
  return CUHE_OK;
}

int cuhe_mix_widths(const cuhe_mix* mix) { return mix ? int(mix->widths.size()) : 0; }

}  // extern "C"
