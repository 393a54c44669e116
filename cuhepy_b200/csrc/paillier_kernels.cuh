// Paillier / Paillier-Lookup kernels for sm_100a.
//
// One instance (ciphertext) is owned by a TPI-lane group (see bigint_group.cuh);
// a 128-thread block holds 128/TPI instances.  All arithmetic mod n^2 is in the
// Montgomery domain with R = 2^(32K); arithmetic mod n uses the same K-limb
// routines with n zero-padded to K limbs.
#pragma once
#include <cstdint>
#include "bigint52.cuh"
#include "bigint_group.cuh"
#include "pair52.cuh"

namespace cuhe {

// Rows of the per-key constant block (each row K words).
enum ConstRow : int {
  C_N2 = 0,     // n^2
  C_R2 = 1,     // R^2 mod n^2
  C_ONE = 2,    // 1
  C_RM = 3,     // R mod n^2  (Montgomery form of 1)
  C_N = 4,      // n, zero-padded
  C_R2N = 5,    // R^2 mod n
  C_NNEG = 6,   // 2^(32K) - n
  C_NR = 7,     // n * R mod n^2
  C_MULTR = 8,  // (secret multiplier) * R mod n
  C_ROWS = 9
};

// Rows of the CRT constant block (each row K words).  Half rows hold the p^2
// value in words [0, K/2) and the q^2 value in words [K/2, K); R_h = 2^(16K).
enum CrtRow : int {
  CR_M = 0,    // p^2 | q^2
  CR_RM = 1,   // R_h mod p^2 | R_h mod q^2
  CR_R3 = 2,   // R_h^3 mod p^2 | R_h^3 mod q^2
  CR_H = 3,    // (q^2)^-1 R_h mod p^2 | 0
  CR_CQ = 4,   // q^2 R mod n^2 (full row)
  CR_PR = 5,   // p R_h mod p^2 | q R_h mod q^2
  CR_P = 6,    // p | 0
  CR_QI = 7,   // q^-1 R_h mod p | 0
  CR_QR = 8,   // q R_h mod n | 0
  CR_ROWS = 9
};

struct CrtScalars {
  uint32_t ninv[2];   // -(p^2)^-1, -(q^2)^-1 mod 2^32
  uint32_t pinv;      // -p^-1 mod 2^32
  unsigned long long ninv52[2];  // -p^-1, -q^-1 mod 2^52
};

struct KeyScalars {
  uint32_t ninv2;  // -(n^2)^-1 mod 2^32
  uint32_t ninv1;  // -n^-1 mod 2^32
  uint32_t ndiv;   // n^-1 mod 2^32 (exact division)
  uint32_t mult_is_zero;
};

// status bits written by kernels
enum StatusBits : int { ST_RANGE = 1 };

enum ExpMode : int { EXP_POW = 0, EXP_ENCRYPT = 1, EXP_DECRYPT = 2, EXP_DECODE = 3 };

constexpr int kBlockThreads = 128;

template <int K>
__host__ __device__ constexpr int inst_stride_words(int buffers) {
  return buffers * K + 4;  // +4 words shifts consecutive instances by 4 banks
}

// -- helpers shared by kernels ---------------------------------------------

template <int K, int TPI>
__device__ __forceinline__ void copy_rows_to_smem(uint32_t* dst, const uint32_t* consts, const int* rows,
                                                  int nrows) {
  for (int r = 0; r < nrows; ++r)
    for (int i = threadIdx.x; i < K; i += blockDim.x) dst[r * K + i] = consts[rows[r] * K + i];
}

// x + small (small < 2^32) over the group, with lookahead carry resolution.
template <int K, int TPI>
__device__ __forceinline__ void add_small(const Group<K, TPI>& g, uint32_t (&x)[K / TPI], uint32_t small) {
  constexpr int L = K / TPI;
  uint32_t add0 = (g.gl == 0) ? small : 0u;
  x[0] = add_cc(x[0], add0);
#pragma unroll
  for (int j = 1; j < L; ++j) x[j] = addc_cc(x[j], 0u);
  const uint32_t carry = addc(0u, 0u);
  uint32_t ones = x[0];
#pragma unroll
  for (int j = 1; j < L; ++j) ones &= x[j];
  const bool cin = g.lookahead(carry != 0u, ones == 0xffffffffu, nullptr);
  if (cin) {
    x[0] = add_cc(x[0], 1u);
#pragma unroll
    for (int j = 1; j < L; ++j) x[j] = addc_cc(x[j], 0u);
    (void)addc(0u, 0u);
  }
}

// x - y for x >= y over the group.
template <int K, int TPI>
__device__ __forceinline__ void sub_group(const Group<K, TPI>& g, uint32_t (&x)[K / TPI],
                                          const uint32_t (&y)[K / TPI]) {
  constexpr int L = K / TPI;
  x[0] = sub_cc(x[0], y[0]);
#pragma unroll
  for (int j = 1; j < L; ++j) x[j] = subc_cc(x[j], y[j]);
  const uint32_t borrow = subc(0u, 0u) & 1u;
  uint32_t zero = x[0];
#pragma unroll
  for (int j = 1; j < L; ++j) zero |= x[j];
  const bool bin = g.lookahead(borrow != 0u, zero == 0u, nullptr);
  if (bin) {
    x[0] = sub_cc(x[0], 1u);
#pragma unroll
    for (int j = 1; j < L; ++j) x[j] = subc_cc(x[j], 0u);
    (void)subc(0u, 0u);
  }
}

// x += y over the group; returns the carry out of the top lane.
template <int K, int TPI>
__device__ __forceinline__ bool add_group(const Group<K, TPI>& g, uint32_t (&x)[K / TPI],
                                          const uint32_t (&y)[K / TPI]) {
  constexpr int L = K / TPI;
  x[0] = add_cc(x[0], y[0]);
#pragma unroll
  for (int j = 1; j < L; ++j) x[j] = addc_cc(x[j], y[j]);
  const uint32_t carry = addc(0u, 0u);
  uint32_t ones = x[0];
#pragma unroll
  for (int j = 1; j < L; ++j) ones &= x[j];
  bool out = false;
  const bool cin = g.lookahead(carry != 0u, ones == 0xffffffffu, &out);
  if (cin) {
    x[0] = add_cc(x[0], 1u);
#pragma unroll
    for (int j = 1; j < L; ++j) x[j] = addc_cc(x[j], 0u);
    (void)addc(0u, 0u);
  }
  return out;
}

// x = (x - y) mod m for x, y < m over the group.
template <int K, int TPI>
__device__ __forceinline__ void sub_mod(const Group<K, TPI>& g, uint32_t (&x)[K / TPI],
                                        const uint32_t (&y)[K / TPI], const uint32_t (&m)[K / TPI]) {
  constexpr int L = K / TPI;
  x[0] = sub_cc(x[0], y[0]);
#pragma unroll
  for (int j = 1; j < L; ++j) x[j] = subc_cc(x[j], y[j]);
  const uint32_t borrow = subc(0u, 0u) & 1u;
  uint32_t zero = x[0];
#pragma unroll
  for (int j = 1; j < L; ++j) zero |= x[j];
  bool under = false;  // x < y: the group-wide borrow (same value in every lane)
  const bool bin = g.lookahead(borrow != 0u, zero == 0u, &under);
  if (bin) {
    x[0] = sub_cc(x[0], 1u);
#pragma unroll
    for (int j = 1; j < L; ++j) x[j] = subc_cc(x[j], 0u);
    (void)subc(0u, 0u);
  }
  if (under) (void)add_group<K, TPI>(g, x, m);
}

// Epilogue shared by the decrypt / decode kernels.  x = base^e mod n^2
// (canonical); writes floor((x - 1)/n) * mult mod n (EXP_DECRYPT) or the
// popcount of its even bits over pop_words words (EXP_DECODE).  Block rows:
// s_one = 1, s_r2n = R^2 mod n, s_multr = mult * R mod n.
template <int K, int TPI>
__device__ __forceinline__ void decrypt_epilogue(const Group<K, TPI>& g, uint32_t (&x)[K / TPI],
                                                 uint32_t* __restrict__ out, long long inst,
                                                 const uint32_t* __restrict__ consts, const KeyScalars& ks,
                                                 const uint32_t* s_one, const uint32_t* s_r2n,
                                                 const uint32_t* s_multr, int mode, int pop_words) {
  constexpr int L = K / TPI;
  uint32_t nn[L];
  g.load_ro(nn, consts + C_N * K);
  uint32_t res[L];
  if (g.is_zero(x)) {
    // floor(-1/n) = -1  ->  (-mult) mod n
    uint32_t multr[L], mult[L];
    g.load(multr, s_multr);
    g.mont_mul(mult, multr, s_one, nn, ks.ninv1);
#pragma unroll
    for (int j = 0; j < L; ++j) res[j] = nn[j];
    if (ks.mult_is_zero) {
#pragma unroll
      for (int j = 0; j < L; ++j) res[j] = 0u;
    } else {
      sub_group<K, TPI>(g, res, mult);
    }
  } else {
    uint32_t one[L];
#pragma unroll
    for (int j = 0; j < L; ++j) one[j] = (g.gl == 0 && j == 0) ? 1u : 0u;
    sub_group<K, TPI>(g, x, one);                 // y
    uint32_t t1[L];
    g.mont_mul(t1, x, s_one, nn, ks.ninv1);       // y R^-1 mod n
    uint32_t rem[L];
    g.mont_mul(rem, t1, s_r2n, nn, ks.ninv1);     // y mod n
    sub_group<K, TPI>(g, x, rem);                 // y - (y mod n) = q*n
    uint32_t q[L], mneg[L];
    g.load_ro(mneg, consts + C_NNEG * K);
    g.exact_div(q, x, mneg, ks.ndiv, K / 2);      // q = floor(y/n) < n
    g.mont_mul(res, q, s_multr, nn, ks.ninv1);    // q * mult mod n
  }
  if (mode == EXP_DECRYPT) {
    g.store(out + inst * K, res);
    return;
  }
  // EXP_DECODE
  int pc = 0;
#pragma unroll
  for (int j = 0; j < L; ++j)
    if (g.gl * L + j < pop_words) pc += __popc(res[j] & 0x55555555u);
#pragma unroll
  for (int off = TPI / 2; off > 0; off >>= 1) pc += __shfl_xor_sync(g.mask, pc, off, TPI);
  if (g.gl == 0) out[inst] = uint32_t(pc);
}

// ---------------------------------------------------------------------------
// Fixed-exponent modular exponentiation with per-instance bases.
//   EXP_POW     out = base^e mod n^2
//   EXP_ENCRYPT out = base^e * (1 + aux*n) mod n^2          (Paillier encrypt, g = n+1)
//   EXP_DECRYPT out = floor((base^e mod n^2 - 1)/n) * mult mod n
//   EXP_DECODE  out32 = popcount of the even bits of the EXP_DECRYPT value
// The exponent is a host-built sliding-window schedule (host_bigint.h).
// ---------------------------------------------------------------------------
// One CTA's share of a modexp launch: instances [block*IPB, block*IPB + IPB).
// Every thread of the CTA calls it (it synchronises the CTA once, after
// staging the key rows in shared memory).
template <int K, int TPI, int W>
__device__ __forceinline__ void modexp_unit(const uint32_t* __restrict__ base, const uint32_t* __restrict__ aux,
                                            int aux_words, uint32_t* __restrict__ out, long long count,
                                            const uint32_t* __restrict__ consts, const KeyScalars& ks,
                                            const int32_t* __restrict__ ops, int nops, int mode, int pop_words,
                                            int* status, long long block) {
  constexpr int L = K / TPI;
  constexpr int T = 1 << (W - 1);
  constexpr int IPB = kBlockThreads / TPI;
  constexpr int STRIDE = inst_stride_words<K>(T + 1);
  extern __shared__ __align__(16) uint32_t smem[];
  // block rows: ONE, R2, NR, R2N, MULTR
  uint32_t* s_one = smem;
  uint32_t* s_r2 = smem + K;
  uint32_t* s_nr = smem + 2 * K;
  uint32_t* s_r2n = smem + 3 * K;
  uint32_t* s_multr = smem + 4 * K;
  {
    const int rows[5] = {C_ONE, C_R2, C_NR, C_R2N, C_MULTR};
    copy_rows_to_smem<K, TPI>(smem, consts, rows, 5);
  }
  __syncthreads();

  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long inst = block * IPB + slot;
  if (inst >= count) return;  // whole groups leave together
  uint32_t* s_inst = smem + 5 * K + slot * STRIDE;
  uint32_t* s_x = s_inst;               // current value (b operand of squarings)
  uint32_t* s_tab = s_inst + K;         // T odd powers

  uint32_t n2[L];
  g.load_ro(n2, consts + C_N2 * K);
  uint32_t x[L], acc[L];
  g.load(x, base + inst * K);
  if (!g.less_than(x, n2)) {
    if (g.gl == 0) atomicOr(status, ST_RANGE);
    return;
  }
  // odd-power table in Montgomery form
  g.mont_mul(acc, x, s_r2, n2, ks.ninv2);  // x*R
  g.publish(s_tab, acc);
  if (T > 1) {
    uint32_t sq[L];
    g.mont_mul(sq, acc, s_tab, n2, ks.ninv2);  // x^2 R
    g.publish(s_x, sq);
#pragma unroll 1
    for (int t = 1; t < T; ++t) {
      g.mont_mul(acc, acc, s_x, n2, ks.ninv2);
      g.publish(s_tab + t * K, acc);
    }
  }
  // exponent schedule
  if (nops == 0) {
    g.load(acc, s_tab);  // unused value, replaced below by R mod n^2
    uint32_t rm[L];
    g.load_ro(rm, consts + C_RM * K);
#pragma unroll
    for (int j = 0; j < L; ++j) acc[j] = rm[j];
  } else {
    const int first = __ldg(ops) & 0xffff;
    g.load(acc, s_tab + (first - 1) * K);
  }
  g.publish(s_x, acc);
#pragma unroll 1
  for (int o = 1; o < nops; ++o) {
    const int op = __ldg(ops + o);
    const int sq = op >> 16;
    const int idx = op & 0xffff;
#pragma unroll 1
    for (int s = 0; s < sq; ++s) {
      g.mont_mul(acc, acc, s_x, n2, ks.ninv2);
      g.publish(s_x, acc);
    }
    if (idx) {
      g.mont_mul(acc, acc, s_tab + (idx - 1) * K, n2, ks.ninv2);
      g.publish(s_x, acc);
    }
  }

  if (mode == EXP_POW) {
    g.mont_mul(x, acc, s_one, n2, ks.ninv2);
    g.store(out + inst * K, x);
    return;
  }
  if (mode == EXP_ENCRYPT) {
    uint32_t m[L];
    g.load(m, aux + inst * aux_words);  // aux_words == K (zero-padded m < n)
    uint32_t nn[L];
    g.load_ro(nn, consts + C_N * K);
    if (!g.less_than(m, nn)) {
      if (g.gl == 0) atomicOr(status, ST_RANGE);
      return;
    }
    g.mont_mul(x, m, s_nr, n2, ks.ninv2);  // m*n (exact, < n^2)
    add_small<K, TPI>(g, x, 1u);           // 1 + m*n = g^m mod n^2
    g.publish(s_x, x);
    g.mont_mul(x, acc, s_x, n2, ks.ninv2);  // r^n * g^m
    g.store(out + inst * K, x);
    return;
  }
  // decrypt / decode
  g.mont_mul(x, acc, s_one, n2, ks.ninv2);
  decrypt_epilogue<K, TPI>(g, x, out, inst, consts, ks, s_one, s_r2n, s_multr, mode, pop_words);
}

template <int K, int TPI, int W>
__global__ void __launch_bounds__(kBlockThreads)
k_modexp(const uint32_t* __restrict__ base, const uint32_t* __restrict__ aux, int aux_words,
         uint32_t* __restrict__ out, long long count, const uint32_t* __restrict__ consts, KeyScalars ks,
         const int32_t* __restrict__ ops, int nops, int mode, int pop_words, int* status) {
  modexp_unit<K, TPI, W>(base, aux, aux_words, out, count, consts, ks, ops, nops, mode, pop_words, status,
                         (long long)blockIdx.x);
}

// One fixed-exponent exponentiation batch of a mixed launch: `count` bases of
// one key (its constant block and Montgomery scalars) raised to one exponent
// (its window schedule).  first_unit = CTA units of the tasks before it.
struct ModexpTask {
  const uint32_t* base;
  uint32_t* out;
  long long count;
  const uint32_t* consts;
  const int32_t* ops;
  long long first_unit;
  KeyScalars ks;
  int nops;
  int mode;
  const double* n52;            // k_pair_modexp_tasks: the key's constants mod n (pair_const_doubles)
  unsigned long long ninv52;    // -n^-1 mod 2^52
};

// Persistent mixed launch: CTAs take units (IPB instances of one task) from
// a global counter until every unit of every task is done, so batches of
// uneven sizes and different keys share one launch without tail waves per
// batch.  tasks[] is ordered by first_unit.
template <int K, int TPI, int W>
__global__ void __launch_bounds__(kBlockThreads)
k_modexp_tasks(const ModexpTask* __restrict__ tasks, int ntasks, long long total_units,
               unsigned long long* __restrict__ counter, int* status) {
  __shared__ long long s_unit;
  while (true) {
    if (threadIdx.x == 0) s_unit = (long long)atomicAdd(counter, 1ull);
    __syncthreads();
    const long long unit = s_unit;
    if (unit >= total_units) break;
    int lo = 0, hi = ntasks - 1;  // last task with first_unit <= unit
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tasks[mid].first_unit <= unit) lo = mid; else hi = mid - 1;
    }
    const ModexpTask& t = tasks[lo];
    modexp_unit<K, TPI, W>(t.base, nullptr, K, t.out, t.count, t.consts, t.ks, t.ops, t.nops, t.mode, 0, status,
                           unit - t.first_unit);
    __syncthreads();  // shared rows and tables are restaged by the next unit
  }
}

// ---------------------------------------------------------------------------
// Decrypt / decode exponentiation by the Chinese remainder theorem, for keys
// whose factorisation n = p q is known (EXP_DECRYPT / EXP_DECODE only).
//
// Each ciphertext is owned by 2*TPI consecutive lanes.  Its lower TPI lanes
// (side 0) compute x_p = c^e mod p^2 and its upper TPI lanes (side 1)
// x_q = c^e mod q^2, each a KH-word Montgomery exponentiation with
// R_h = 2^(32 KH) on its own half of the lanes, so one modular product costs
// a quarter of a K-word one.  Garner's recombination
//   h = (x_p - x_q) (q^2)^-1 mod p^2,   x = x_q + q^2 h   (< n^2, exact)
// runs on the two halves together as a K-word group, and the same epilogue
// as k_modexp follows, so the result equals the direct c^e mod n^2 path for
// every c < n^2.
// ---------------------------------------------------------------------------
template <int KH, int TPI, int W>
__global__ void __launch_bounds__(kBlockThreads)
k_modexp_crt(const uint32_t* __restrict__ base, uint32_t* __restrict__ out, long long count,
             const uint32_t* __restrict__ consts, KeyScalars ks, const uint32_t* __restrict__ crt, CrtScalars cs,
             const int32_t* __restrict__ ops, int nops, int mode, int pop_words, int* status) {
  constexpr int K = 2 * KH;
  constexpr int L = KH / TPI;
  constexpr int T = 1 << (W - 1);
  constexpr int IPB = kBlockThreads / (2 * TPI);
  constexpr int SIDE = (T + 1) * KH + 4;  // per side: x, then T odd powers; +4 words moves the banks
  extern __shared__ __align__(16) uint32_t smem[];
  // block rows: ONE, R2N, MULTR (K words each), RM, R3, H (two halves), CQ (K words)
  uint32_t* s_one = smem;
  uint32_t* s_r2n = smem + K;
  uint32_t* s_multr = smem + 2 * K;
  uint32_t* s_rm = smem + 3 * K;
  uint32_t* s_r3 = smem + 4 * K;
  uint32_t* s_h = smem + 5 * K;
  uint32_t* s_cq = smem + 6 * K;
  {
    const int rows[3] = {C_ONE, C_R2N, C_MULTR};
    copy_rows_to_smem<K, TPI>(smem, consts, rows, 3);
    const int crows[4] = {CR_RM, CR_R3, CR_H, CR_CQ};
    copy_rows_to_smem<K, TPI>(smem + 3 * K, crt, crows, 4);
  }
  __syncthreads();

  Group<K, 2 * TPI> g;   // the whole ciphertext
  Group<KH, TPI> h;      // this side's half
  const int side = (threadIdx.x / TPI) & 1;
  const int slot = threadIdx.x / (2 * TPI);
  const long long inst = (long long)blockIdx.x * IPB + slot;
  if (inst >= count) return;  // both halves leave together
  uint32_t* s_item = smem + 7 * K + slot * 2 * SIDE;
  uint32_t* s_x = s_item + side * SIDE;
  uint32_t* s_tab = s_x + KH;

  {
    uint32_t c[L], n2[L];
    g.load_ro(n2, consts + C_N2 * K);
    g.load(c, base + inst * K);
    if (!g.less_than(c, n2)) {
      if (g.gl == 0) atomicOr(status, ST_RANGE);
      return;
    }
  }
  const uint32_t ninv = cs.ninv[side];
  uint32_t m[L], lo[L], hi[L], acc[L];
  h.load_ro(m, crt + CR_M * K + side * KH);
  h.load(lo, base + inst * K);
  h.load(hi, base + inst * K + KH);
  // c = lo + hi R_h:  (lo + hi * (R_h mod M)) R_h^-1 = c R_h^-1, then * R_h^3 R_h^-1
  h.mont_mul_acc(acc, lo, hi, s_rm + side * KH, m, ninv);
  h.mont_mul(acc, acc, s_r3 + side * KH, m, ninv);  // c R_h mod M (Montgomery form)
  h.publish(s_tab, acc);
  if (T > 1) {
    uint32_t sq[L];
    h.mont_mul(sq, acc, s_tab, m, ninv);
    h.publish(s_x, sq);
#pragma unroll 1
    for (int t = 1; t < T; ++t) {
      h.mont_mul(acc, acc, s_x, m, ninv);
      h.publish(s_tab + t * KH, acc);
    }
  }
  if (nops == 0) {
    h.load(acc, s_rm + side * KH);  // e = 0: Montgomery form of 1
  } else {
    const int first = __ldg(ops) & 0xffff;
    h.load(acc, s_tab + (first - 1) * KH);
  }
  h.publish(s_x, acc);
#pragma unroll 1
  for (int o = 1; o < nops; ++o) {
    const int op = __ldg(ops + o);
    const int sq = op >> 16;
    const int idx = op & 0xffff;
#pragma unroll 1
    for (int s = 0; s < sq; ++s) {
      h.mont_mul(acc, acc, s_x, m, ninv);
      h.publish(s_x, acc);
    }
    if (idx) {
      h.mont_mul(acc, acc, s_tab + (idx - 1) * KH, m, ninv);
      h.publish(s_x, acc);
    }
  }
  uint32_t xs[L];
  h.mont_mul(xs, acc, s_one, m, ninv);  // x_side, canonical
  __syncwarp(g.mask);
  h.store(s_x, xs);
  __syncwarp(g.mask);
  uint32_t* s_xp = s_item;
  uint32_t* s_xq = s_item + SIDE;
  if (side == 0) {
    // h = x_p (q^2)^-1 - x_q (q^2)^-1 mod p^2   (x_q may exceed p^2; x_q < R_h)
    uint32_t xq[L], v[L], u[L];
    h.load(xq, s_xq);
    h.mont_mul(v, xs, s_h, m, ninv);
    h.mont_mul(u, xq, s_h, m, ninv);
    sub_mod<KH, TPI>(h, v, u, m);
    __syncwarp(h.mask);
    h.store(s_xp, v);
  }
  __syncwarp(g.mask);
  // x = x_q + q^2 h over the whole group: side 0 lanes hold the low words
  uint32_t hv[L], xq[L], x[L];
  if (side == 0) {
    h.load(hv, s_xp);
    h.load(xq, s_xq);
  } else {
#pragma unroll
    for (int j = 0; j < L; ++j) hv[j] = xq[j] = 0u;
  }
  uint32_t n2[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.mont_mul(x, hv, s_cq, n2, ks.ninv2);  // h q^2 mod n^2 = h q^2
  (void)add_group<K, 2 * TPI>(g, x, xq);
  decrypt_epilogue<K, 2 * TPI>(g, x, out, inst, consts, ks, s_one, s_r2n, s_multr, mode, pop_words);
}

// limb i (52 bits at 52 i) of a little-endian array of nwords 32-bit words
__device__ __forceinline__ uint64_t limb52_from_words(const uint32_t* w, int nwords, int i) {
  const int bit = 52 * i, j = bit >> 5, off = bit & 31;
  const uint64_t w0 = j < nwords ? w[j] : 0u;
  const uint64_t w1 = j + 1 < nwords ? w[j + 1] : 0u;
  const uint64_t w2 = j + 2 < nwords ? w[j + 2] : 0u;
  uint64_t v = (w0 | (w1 << 32)) >> off;
  if (off) v |= w2 << (64 - off);
  return v & cuhe52::kMask;
}

// word i (32 bits at 32 i) of an array of nlimbs 52-bit limbs
__device__ __forceinline__ uint32_t word_from_limbs52(const uint64_t* l, int nlimbs, int i) {
  const int bit = 32 * i, j = bit / 52, off = bit - 52 * j;
  const uint64_t l0 = j < nlimbs ? l[j] : 0u;
  const uint64_t l1 = j + 1 < nlimbs ? l[j + 1] : 0u;
  uint64_t v = l0 >> off;
  if (off > 20) v |= l1 << (52 - off);
  return uint32_t(v);
}

// ---------------------------------------------------------------------------
// Exponentiation mod m^2 on pairs of residues mod m (pair52.cuh): the
// decrypt / decode kernel by the Chinese remainder theorem (m = p and q), and
// the kernel mod n^2 (m = n) for encryption's r^n, public powers and
// decryption without the factors.  K limbs of 52 bits a component on TPI
// lanes, 128 threads.  kL = 10 limbs per lane with two CTAs per SM (about 250
// registers a thread, which let the compiler interleave the accumulations; a
// quarter fewer squarings a second with 168 registers and three CTAs) is the
// best rate, 2,210 M squarings a second at 2,048-bit m^2; kL = 5 spreads a
// value over twice the lanes for batches that leave SMs idle: 1,930 M a second
// when the GPU is full, but 2.6 us a squaring against 4.4 for a warp alone
// (the host's rule: pair_small).
//
// A value of 32-bit words enters as kEntry chunks u_j of 52 K bits,
// x R = sum_j u_j (R^(j+2) R^-1), one product with a constant pair each, and
// leaves by a product with the pair (1, 0), its components re-cut to 32-bit
// words in [0, m]; the recombination, the Paillier factor 1 + a n (the pair
// (1, a): it takes the place of (1, 0)) and the L() epilogue follow on words.
// ---------------------------------------------------------------------------
constexpr int kPairWindow = 3;                       // odd powers x, x^3, x^5, x^7
constexpr int kPairTable = 1 << (kPairWindow - 1);

// Constants of one modulus m as doubles: m as K limbs, then rows of K pairs:
// the entry chunks' R^(j+2) mod m^2, (1, 0), (w R mod m, 0) and R mod m^2.
__host__ __device__ constexpr int pair_const_doubles(int K, int entry) { return K + 2 * K * (entry + 3); }

// An exponent's window schedule.  halved: e = u (p - 1) and the schedule is
// that of p - 1; when x^(p-1) = 1 + p z1 (always, for x prime to a prime p),
// x^e = 1 + p (z1 u mod p).  Any other value in a CTA sends it through the
// schedule `fall` of u next, which holds for every x and every p.
struct PairExponent {
  const int32_t* ops;
  const int32_t* fall;
  int nops, nfall;
  int halved;
};

template <int K, int TPI>
__device__ __forceinline__ void pair_publish(const cuhe52::Pair52<K, TPI>& f, double2* s, const double (&x)[K / TPI],
                                             const double (&y)[K / TPI]) {
  __syncwarp();
#pragma unroll
  for (int k = 0; k < K / TPI; ++k) s[f.gl * (K / TPI) + k] = make_double2(x[k], y[k]);
  __syncwarp();
}

// x^e for this group's value (all lanes of the warp call it): words = the
// value, nwords of them; rows = the modulus' constant pairs in shared memory
// (kEntry entry rows, (1, 0), the scale row); one = R mod m^2 in global
// memory; s = this group's K pairs, tab = this thread's table column (stride
// kPairThreads).  aux: null, or the words a of the factor (1, a).  Leaves the
// canonical limbs (z0, z1), in [0, m] (z1 with aux up to m + 2 m^2 / R), as
// pairs of 64-bit integers in s.  kUnits (every thread of the CTA calls it):
// when z0 is 1 for every value of the CTA, leaves (1, y) instead, y = z1 w
// mod m in [0, m + m^2 / R] with w the scale row's factor, and returns true.
template <int K, int TPI, int kEntry, bool kUnits>
__device__ __forceinline__ bool pair_power(const cuhe52::Pair52<K, TPI>& f, const uint32_t* __restrict__ words,
                                           int nwords, const double2* rows, const double2* __restrict__ one,
                                           double2* s, double2* tab, const double (&m)[K / TPI], uint64_t ninv,
                                           const PairExponent& ex, const uint32_t* __restrict__ aux) {
  constexpr int L = K / TPI;
  constexpr int kStride = cuhe52::kPairThreads;
  const int32_t* ops = ex.ops;
  int nops = ex.nops;
  bool halved = kUnits && ex.halved != 0;
  double z0[L], z1[L], a0[L], a1[L];
  uint64_t A0[L], A1[L];
  const int at = f.gl * L;
  auto bits = [](double d) { return static_cast<uint64_t>(__double_as_longlong(d)); };
  auto raw = [](uint64_t v) { return __longlong_as_double(static_cast<long long>(v)); };

  bool voted = false;
  int j = 0;  // entry chunks, then the square of x; again from there with the schedule ex.fall
  while (true) {
#pragma unroll 1
    for (; j <= kEntry; ++j) {
      if (j < kEntry) {
#pragma unroll
        for (int k = 0; k < L; ++k) a0[k] = f.to_f64(limb52_from_words(words, nwords, j * K + at + k));
      } else {
        if (nops == 0) break;
#pragma unroll
        for (int k = 0; k < L; ++k) {
          tab[k * kStride] = make_double2(z0[k], z1[k]);
          a0[k] = z0[k];
        }
        f.twice_limbs(a1, z1);
        pair_publish<K, TPI>(f, s, z0, a1);
      }
      f.template product<false>(A0, A1, a0, a0, j < kEntry ? rows + j * K : s, m, ninv);
      if (j == kEntry) {  // x^2 stays in s for the odd powers, x in z
        f.template limbs<2>(a0, A0);
        f.template limbs<2>(a1, A1);
        pair_publish<K, TPI>(f, s, a0, a1);
        break;
      }
      // the chunks are summed as columns, kept in s between them
      f.template columns<2>(A0);
      f.template columns<2>(A1);
#pragma unroll
      for (int k = 0; k < L; ++k) {
        if (j > 0) {
          A0[k] += bits(s[at + k].x);
          A1[k] += bits(s[at + k].y);
        }
        s[at + k] = make_double2(raw(A0[k]), raw(A1[k]));
      }
      if (j == kEntry - 1) {
        f.from_columns(z0, A0);
        f.from_columns(z1, A1);
      }
    }
    if (nops == 0) {  // e = 0
#pragma unroll
      for (int k = 0; k < L; ++k) {
        const double2 t = __ldg(one + at + k);
        z0[k] = t.x;
        z1[k] = t.y;
      }
    } else {
#pragma unroll 1
      for (int t = 1; t < kPairTable; ++t) {  // x^(2t+1) = x^(2t-1) x^2
        f.template product<true>(A0, A1, z0, z1, s, m, ninv);
        f.template limbs<2>(z0, A0);
        f.template limbs<3>(z1, A1);
#pragma unroll
        for (int k = 0; k < L; ++k) tab[(t * L + k) * kStride] = make_double2(z0[k], z1[k]);
      }
      const int first = (__ldg(ops) & 0xffff) - 1;
#pragma unroll
      for (int k = 0; k < L; ++k) {
        const double2 t = tab[(first * L + k) * kStride];
        z0[k] = t.x;
        z1[k] = t.y;
      }
    }
    // Each op squares at least once and then multiplies by a table entry; the
    // last pass is the way out, the product with (1, 0) or (1, aux).
    f.twice_limbs(a1, z1);
    int op = nops > 1 ? __ldg(ops + 1) : 0;
#pragma unroll 1
    for (int o = 1;; ++o) {
      const bool out = o >= nops;
      const int sq = out ? 0 : op >> 16, idx = op & 0xffff;
      if (o + 1 < nops) op = __ldg(ops + o + 1);
#pragma unroll 1
      for (int i = 1; i <= sq; ++i) {
        pair_publish<K, TPI>(f, s, z0, a1);  // (z0, 2 z1)
        f.template product<false>(A0, A1, z0, z0, s, m, ninv);
        f.template limbs<2>(z0, A0);
        if (i < sq) f.template twice<2>(a1, A1);
        else f.template limbs<2>(z1, A1);
      }
      const double2* b = s;
      if (out) {
        if (aux) {
          double one0[L];
#pragma unroll
          for (int k = 0; k < L; ++k) {
            A1[k] = limb52_from_words(aux, nwords, at + k);
            one0[k] = at + k == 0 ? 1.0 : 0.0;
          }
          f.from_columns(a1, A1);
          pair_publish<K, TPI>(f, s, one0, a1);
        } else {
          b = rows + kEntry * K;
        }
#pragma unroll
        for (int k = 0; k < L; ++k) {
          a0[k] = z0[k];
          a1[k] = z1[k];
        }
      } else {
        if (idx == 0) continue;  // the schedule's last squarings
        pair_publish<K, TPI>(f, s, z0, z1);
#pragma unroll
        for (int k = 0; k < L; ++k) {
          const double2 t = tab[((idx - 1) * L + k) * kStride];
          a0[k] = t.x;
          a1[k] = t.y;
        }
      }
      f.template product<true>(A0, A1, a0, a1, b, m, ninv);
      if (out) break;
      f.template limbs<2>(z0, A0);
      f.template limbs<3>(z1, A1);
      f.template twice<3>(a1, A1);
    }
    f.template columns<2>(A0);
    f.template columns<3>(A1);
    f.canonical(A0);
    f.canonical(A1);
    bool isone = true;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < L; ++k) {
      s[at + k] = make_double2(raw(A0[k]), raw(A1[k]));
      isone = isone && A0[k] == (at + k == 0 ? 1ull : 0ull);
    }
    __syncwarp();
    if (!kUnits) return false;
    // (once per thread: a CTA whose values are not all units stays in the
    // general form from here on)
    if (!voted) {
      if (__syncthreads_and(isone)) break;
      voted = true;
    }
    if (!halved) return false;
    halved = false;  // raise x^(p-1) (still in z) to u
    ops = ex.fall;
    nops = ex.nfall;
    j = kEntry;
  }
  // (1, z1) -> (1, z1 w mod m)
#pragma unroll
  for (int k = 0; k < L; ++k) a0[k] = f.to_f64(A1[k]);
  f.template product<false>(A0, A1, a0, a0, rows + (kEntry + 1) * K, m, ninv);
  f.template columns<2>(A0);
  f.canonical(A0);
#pragma unroll
  for (int k = 0; k < L; ++k) s[at + k].y = raw(A0[k]);
  return true;
}

// word i (32 bits at 32 i) of component `second` of K pairs of 64-bit limbs
template <int K>
__device__ __forceinline__ uint32_t word_from_pairs(const double2* s, bool second, int i) {
  const int bit = 32 * i, j = bit / 52, off = bit - 52 * j;
  auto limb = [&](int k) -> uint64_t {
    if (k >= K) return 0;
    return static_cast<uint64_t>(__double_as_longlong(second ? s[k].y : s[k].x));
  };
  uint64_t v = limb(j) >> off;
  if (off > 20) v |= limb(j + 1) << (52 - off);
  return uint32_t(v);
}

// x = z1 m + z0 mod m^2 (canonical) over a group, from the pairs in s: mr =
// m R mod m^2 (R = 2^(32K)), mm = m^2.
template <int KL, int K, int TPI>
__device__ __forceinline__ void pair_words(const Group<K, TPI>& g, uint32_t (&x)[K / TPI], const double2* s,
                                           const uint32_t* mr, const uint32_t (&mm)[K / TPI], uint32_t ninv) {
  constexpr int L = K / TPI;
  uint32_t z[L];
#pragma unroll
  for (int j = 0; j < L; ++j) z[j] = word_from_pairs<KL>(s, true, g.gl * L + j);
  g.mont_mul(x, z, mr, mm, ninv);  // z1 m mod m^2, a multiple of m
#pragma unroll
  for (int j = 0; j < L; ++j) z[j] = word_from_pairs<KL>(s, false, g.gl * L + j);
  (void)add_group<K, TPI>(g, x, z);  // at most m^2
  if (!g.less_than(x, mm)) sub_group<K, TPI>(g, x, mm);
}

// kL of the split form (pair52_split.cuh), whose layout is a specialisation.
constexpr int kSplit = -5;
// Its table holds up to 16 odd powers (80 KB, one CTA per SM), as many as the
// exponent's wide schedule uses (host pair_schedule, behind the other's ops):
// at |e| = 279 four-bit windows, from some 500 bits on five.
constexpr int kSplitWindow = 5;

template <int K, int kL, int kEntry, int kSides>
struct PairLayout {  // K limbs per component (kL per lane), kSides moduli per item
  static constexpr int TPI = K / kL;
  static constexpr int kGroups = cuhe52::kPairThreads / TPI;   // values of a CTA
  static constexpr int kItems = kGroups / kSides;
  static constexpr int kRows = (kEntry + 2) * K;               // constant pairs per modulus
  static constexpr int kSlot = K + 1;                          // pairs per value; +1 moves the banks
  static constexpr size_t kTab = size_t(kPairTable) * kL * cuhe52::kPairThreads;
  static constexpr size_t kBytes = (size_t(kSides) * kRows + size_t(kGroups) * kSlot + kTab) * 16;
};

template <int KL, int kEntry, int kSides, bool kUnits>
__device__ __forceinline__ bool split_run(double* smem, const double* __restrict__ cm, int side, int group,
                                          const uint32_t* __restrict__ words, int nwords, uint64_t ninv52,
                                          const PairExponent& ex, const uint32_t* __restrict__ aux);

// Decrypt / decode with the factors installed: c^e mod p^2 and mod q^2 in the
// two halves of the CTA (whole warps per side, so each side follows its own
// schedule).  For ciphertexts c^e is 1 mod n and the plaintext comes from the
// second components alone; a CTA with any other value takes Garner's
// recombination and the epilogue of k_modexp_crt on words, 2 KH / 16 lanes
// per ciphertext.
template <int KH, int kL>
__global__ void __launch_bounds__(cuhe52::kPairThreads, 2)
k_pair_crt(const uint32_t* __restrict__ base, uint32_t* __restrict__ out, long long count,
           const uint32_t* __restrict__ consts, KeyScalars ks, const uint32_t* __restrict__ crt, CrtScalars cs,
           const double* __restrict__ crt52, PairExponent e0, PairExponent e1, int mode, int pop_words, int* status) {
  constexpr int K = 2 * KH, KL = 5 * KH / 16, kEntry = 4;
  using Lay = PairLayout<KL, kL, kEntry, 2>;
  constexpr int IPB = Lay::kItems, TPI = Lay::TPI;
  extern __shared__ __align__(16) uint32_t smem[];
  double2* s_rows = reinterpret_cast<double2*>(smem);
  double2* s_vals = s_rows + 2 * Lay::kRows;
  double2* s_tab = s_vals + Lay::kGroups * Lay::kSlot;
  constexpr int kConst = pair_const_doubles(KL, kEntry);
  if constexpr (kL != kSplit) {
    for (int i = threadIdx.x; i < 2 * Lay::kRows; i += blockDim.x) {
      const int sd = i / Lay::kRows;
      s_rows[i] = reinterpret_cast<const double2*>(crt52 + sd * kConst + KL)[i - sd * Lay::kRows];
    }
    __syncthreads();
  }
  const long long first = (long long)blockIdx.x * IPB;
  bool units;
  {
    const int side = threadIdx.x / (cuhe52::kPairThreads / 2);
    const int group = threadIdx.x / TPI;  // side * IPB + item
    const long long inst = min(first + group - side * IPB, count - 1);  // idle groups repeat the last item
    if constexpr (kL == kSplit) {
      units = split_run<KL, kEntry, 2, true>(reinterpret_cast<double*>(smem), crt52, side, group, base + inst * K, K,
                                             cs.ninv52[side], side ? e1 : e0, nullptr);
    } else {
      cuhe52::Pair52<KL, TPI> f;
      const double* cm = crt52 + side * kConst;
      double m[kL];
#pragma unroll
      for (int k = 0; k < kL; ++k) m[k] = __ldg(cm + f.gl * kL + k);
      units = pair_power<KL, TPI, kEntry, true>(f, base + inst * K, K, s_rows + side * Lay::kRows,
                                                reinterpret_cast<const double2*>(cm + KL) + (kEntry + 2) * KL,
                                                s_vals + group * Lay::kSlot, s_tab + threadIdx.x, m,
                                                f.gl == 0 ? cs.ninv52[side] : 0ull, side ? e1 : e0, nullptr);
    }
  }
  __syncthreads();
  if (units) {
    // x^e = 1 + n t with t mult = r_p mod p, r_q mod q (the scale rows hold
    // q^-1 mult and p^-1 mult, times the cofactor): the plaintext
    // t mult mod n = r_q + q ((r_p - r_q) q^-1 mod p), three products of KH
    // words an item where the general recombination below takes five of K
    // words and four of KH (key_len 1024: 0.40 of 3.94 ms a wave of decodes)
    constexpr int LT = KH / 16, L = 16, PER = cuhe52::kPairThreads / LT;
    uint32_t* s_qi = reinterpret_cast<uint32_t*>(s_tab);
    uint32_t* s_qr = s_qi + KH;
    for (int i = threadIdx.x; i < KH; i += blockDim.x) {
      s_qi[i] = crt[CR_QI * K + i];
      s_qr[i] = crt[CR_QR * K + i];
    }
    __syncthreads();
    Group<KH, LT> h;
#pragma unroll 1
    for (int item = threadIdx.x / LT; item < IPB; item += PER) {
      const long long inst = first + item;
      if (inst >= count) break;
      uint32_t x[L], y[L], u[L], m[L];
      {
        // c < n^2: the upper half decides unless it equals n^2's
        h.load(x, base + inst * K + KH);
        h.load_ro(y, consts + C_N2 * K + KH);
        bool less = h.less_than(x, y);
        if (!less) {
          sub_group<KH, LT>(h, x, y);  // zero when they are equal
          const bool equal = h.is_zero(x);
          h.load(x, base + inst * K);
          h.load_ro(y, consts + C_N2 * K);
          less = equal && h.less_than(x, y);
        }
        if (!less) {
          if (h.gl == 0) atomicOr(status, ST_RANGE);
          continue;
        }
      }
      const double2* sp = s_vals + item * Lay::kSlot;
      const double2* sq = s_vals + (IPB + item) * Lay::kSlot;
      h.load_ro(m, crt + CR_P * K);
#pragma unroll
      for (int t = 0; t < L; ++t) {
        x[t] = word_from_pairs<KL>(sp, true, h.gl * L + t);
        y[t] = word_from_pairs<KL>(sq, true, h.gl * L + t);
      }
      h.mont_mul(u, x, s_qi, m, cs.pinv);  // r_p q^-1 mod p
      h.mont_mul(x, y, s_qi, m, cs.pinv);  // r_q q^-1 mod p
      sub_mod<KH, LT>(h, u, x, m);
      h.load_ro(m, consts + C_N * K);
      h.mont_mul(x, u, s_qr, m, ks.ninv1);  // q times that, at most n - q
      (void)add_group<KH, LT>(h, x, y);     // r_q is at most q + q^2 / R: the sum is below 2 n
      if (!h.less_than(x, m)) sub_group<KH, LT>(h, x, m);
      if (mode == EXP_DECRYPT) {
        h.store(out + inst * K, x);
#pragma unroll
        for (int t = 0; t < L; ++t) x[t] = 0u;
        h.store(out + inst * K + KH, x);
      } else {
        int pc = 0;
#pragma unroll
        for (int t = 0; t < L; ++t)
          if (h.gl * L + t < pop_words) pc += __popc(x[t] & 0x55555555u);
#pragma unroll
        for (int off = LT / 2; off > 0; off >>= 1) pc += __shfl_xor_sync(h.mask, pc, off, LT);
        if (h.gl == 0) out[inst] = uint32_t(pc);
      }
    }
    return;
  }
  // words: ONE, R2N, MULTR (K words each), p R_h, H (two halves), CQ, then
  // per item of a pass x_p and x_q (KH words each), over the powers' table
  constexpr int LT = KH / 16, L = 16;  // lanes per side
  constexpr int PER = cuhe52::kPairThreads / (2 * LT);
  uint32_t* s_one = reinterpret_cast<uint32_t*>(s_tab);
  uint32_t* s_r2n = s_one + K;
  uint32_t* s_multr = s_one + 2 * K;
  uint32_t* s_pr = s_one + 3 * K;
  uint32_t* s_h = s_one + 4 * K;
  uint32_t* s_cq = s_one + 5 * K;
  {
    const int rows[3] = {C_ONE, C_R2N, C_MULTR};
    copy_rows_to_smem<K, LT>(s_one, consts, rows, 3);
    const int crows[3] = {CR_PR, CR_H, CR_CQ};
    copy_rows_to_smem<K, LT>(s_pr, crt, crows, 3);
  }
  __syncthreads();
  Group<K, 2 * LT> g;  // the whole ciphertext
  Group<KH, LT> h;     // this side's half
  const int side = (threadIdx.x / LT) & 1;
  const int slot = threadIdx.x / (2 * LT);
  uint32_t* s_xp = s_one + 6 * K + slot * (K + 4);
  uint32_t* s_xq = s_xp + KH;
#pragma unroll 1
  for (int item = slot; item < IPB; item += PER) {
    const long long inst = first + item;
    if (inst >= count) break;
    uint32_t n2[L], x[L], m[L], hv[L], xq[L];
    g.load_ro(n2, consts + C_N2 * K);
    g.load(x, base + inst * K);
    if (!g.less_than(x, n2)) {
      if (g.gl == 0) atomicOr(status, ST_RANGE);
      continue;
    }
    h.load_ro(m, crt + CR_M * K + side * KH);
    pair_words<KL, KH, LT>(h, x, s_vals + (side * IPB + item) * Lay::kSlot, s_pr + side * KH, m, cs.ninv[side]);
    __syncwarp(g.mask);
    h.store(side == 0 ? s_xp : s_xq, x);
    __syncwarp(g.mask);
    if (side == 0) {
      // h = x_p (q^2)^-1 - x_q (q^2)^-1 mod p^2   (x_q may exceed p^2; x_q < R_h)
      h.load(xq, s_xq);
      h.mont_mul(hv, x, s_h, m, cs.ninv[0]);
      h.mont_mul(x, xq, s_h, m, cs.ninv[0]);
      sub_mod<KH, LT>(h, hv, x, m);
      __syncwarp(h.mask);
      h.store(s_xp, hv);
    }
    __syncwarp(g.mask);
    // x = x_q + q^2 h over the whole group: side 0 lanes hold the low words
    if (side == 0) {
      h.load(hv, s_xp);
      h.load(xq, s_xq);
    } else {
#pragma unroll
      for (int j = 0; j < L; ++j) hv[j] = xq[j] = 0u;
    }
    g.mont_mul(x, hv, s_cq, n2, ks.ninv2);  // h q^2 mod n^2 = h q^2
    (void)add_group<K, 2 * LT>(g, x, xq);
    decrypt_epilogue<K, 2 * LT>(g, x, out, inst, consts, ks, s_one, s_r2n, s_multr, mode, pop_words);
    __syncwarp(g.mask);
  }
}

// The exponentiation mod n^2 (k_modexp's modes): items [block * kItems, ...)
// of a batch.
template <int K, int kL>
__device__ __forceinline__ void pair_modexp_unit(const uint32_t* __restrict__ base, const uint32_t* __restrict__ aux,
                                                 uint32_t* __restrict__ out, long long count,
                                                 const uint32_t* __restrict__ consts, const KeyScalars& ks,
                                                 const double* __restrict__ n52, unsigned long long ninv52,
                                                 const int32_t* __restrict__ ops, int nops, int mode, int pop_words,
                                                 int* status, long long block) {
  constexpr int KL = 5 * K / 16, kEntry = 2;
  using Lay = PairLayout<KL, kL, kEntry, 1>;
  constexpr int IPB = Lay::kItems, TPI = Lay::TPI;
  extern __shared__ __align__(16) uint32_t smem[];
  double2* s_rows = reinterpret_cast<double2*>(smem);
  double2* s_vals = s_rows + Lay::kRows;
  double2* s_tab = s_vals + Lay::kGroups * Lay::kSlot;
  if constexpr (kL != kSplit) {
    for (int i = threadIdx.x; i < Lay::kRows; i += blockDim.x)
      s_rows[i] = reinterpret_cast<const double2*>(n52 + KL)[i];
    __syncthreads();
  }
  const long long first = block * IPB;
  {
    const int group = threadIdx.x / TPI;
    const long long inst = min(first + group, count - 1);  // idle groups repeat the last item
    const PairExponent ex{ops, nullptr, nops, 0, 0};
    if constexpr (kL == kSplit) {
      (void)split_run<KL, kEntry, 1, false>(reinterpret_cast<double*>(smem), n52, 0, group, base + inst * K, K, ninv52,
                                            ex, mode == EXP_ENCRYPT ? aux + inst * K : nullptr);
    } else {
      cuhe52::Pair52<KL, TPI> f;
      double m[kL];
#pragma unroll
      for (int k = 0; k < kL; ++k) m[k] = __ldg(n52 + f.gl * kL + k);
      (void)pair_power<KL, TPI, kEntry, false>(f, base + inst * K, K, s_rows,
                                               reinterpret_cast<const double2*>(n52 + KL) + (kEntry + 2) * KL,
                                               s_vals + group * Lay::kSlot, s_tab + threadIdx.x, m,
                                               f.gl == 0 ? ninv52 : 0ull, ex,
                                               mode == EXP_ENCRYPT ? aux + inst * K : nullptr);
    }
  }
  __syncthreads();
  constexpr int LT = K / 16, L = 16, PER = cuhe52::kPairThreads / LT;
  uint32_t* s_one = reinterpret_cast<uint32_t*>(s_tab);
  uint32_t* s_nr = s_one + K;
  uint32_t* s_r2n = s_one + 2 * K;
  uint32_t* s_multr = s_one + 3 * K;
  {
    const int rows[4] = {C_ONE, C_NR, C_R2N, C_MULTR};
    copy_rows_to_smem<K, LT>(s_one, consts, rows, 4);
  }
  __syncthreads();
  Group<K, LT> g;
  uint32_t n2[L], x[L], y[L];
  g.load_ro(n2, consts + C_N2 * K);
#pragma unroll 1
  for (int item = threadIdx.x / LT; item < IPB; item += PER) {
    const long long inst = first + item;
    if (inst >= count) break;
    g.load(x, base + inst * K);
    bool valid = g.less_than(x, n2);
    if (mode == EXP_ENCRYPT) {
      g.load(x, aux + inst * K);
      g.load_ro(y, consts + C_N * K);
      valid = g.less_than(x, y) && valid;
    }
    if (!valid) {
      if (g.gl == 0) atomicOr(status, ST_RANGE);
      continue;
    }
    pair_words<KL, K, LT>(g, x, s_vals + item * Lay::kSlot, s_nr, n2, ks.ninv2);
    if (mode == EXP_POW || mode == EXP_ENCRYPT) g.store(out + inst * K, x);
    else decrypt_epilogue<K, LT>(g, x, out, inst, consts, ks, s_one, s_r2n, s_multr, mode, pop_words);
  }
}

template <int K, int kL>
__global__ void __launch_bounds__(cuhe52::kPairThreads, 2)
k_pair_modexp(const uint32_t* __restrict__ base, const uint32_t* __restrict__ aux, uint32_t* __restrict__ out,
              long long count, const uint32_t* __restrict__ consts, KeyScalars ks, const double* __restrict__ n52,
              unsigned long long ninv52, const int32_t* __restrict__ ops, int nops, int mode, int pop_words,
              int* status) {
  pair_modexp_unit<K, kL>(base, aux, out, count, consts, ks, n52, ninv52, ops, nops, mode, pop_words, status, blockIdx.x);
}

// The persistent mixed launch (k_modexp_tasks): units of PairLayout::kItems
// instances of one task.
template <int K>
__global__ void __launch_bounds__(cuhe52::kPairThreads, 2)
k_pair_modexp_tasks(const ModexpTask* __restrict__ tasks, int ntasks, long long total_units,
                    unsigned long long* __restrict__ counter, int* status) {
  __shared__ long long s_unit;
  while (true) {
    if (threadIdx.x == 0) s_unit = (long long)atomicAdd(counter, 1ull);
    __syncthreads();
    const long long unit = s_unit;
    if (unit >= total_units) break;
    int lo = 0, hi = ntasks - 1;  // last task with first_unit <= unit
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (tasks[mid].first_unit <= unit) lo = mid; else hi = mid - 1;
    }
    const ModexpTask& t = tasks[lo];
    pair_modexp_unit<K, 10>(t.base, nullptr, t.out, t.count, t.consts, t.ks, t.n52, t.ninv52, t.ops, t.nops, t.mode, 0,
                        status, unit - t.first_unit);
    __syncthreads();  // shared rows and tables are restaged by the next unit
  }
}

// ---------------------------------------------------------------------------
// encode_hamming_server on the FP64 pipe (n^2 of 4096 / 8192 bits):
// out[q][j] = index[j] * query[q] mod n^2 as one Montgomery product of 52-bit
// limbs, the query entering in the Montgomery domain of R52
// (k_to_mont52: query R52 mod n^2, once per query) and the index value and
// the result crossing between 32-bit words and 52-bit limbs by bit
// shuffling, so each output costs one product: mont52(index, query R52) =
// index * query mod n^2, canonical, as k_mulmod_outer's.
// ---------------------------------------------------------------------------
// row: R52 R mod n^2; out = x R52 mod n^2.
template <int K>
__global__ void __launch_bounds__(kBlockThreads)
k_to_mont52(const uint32_t* __restrict__ in, long long count, double* __restrict__ out,
            const uint32_t* __restrict__ consts, KeyScalars ks, const uint32_t* __restrict__ row, int* status) {
  constexpr int TPI = K / 16, L = 16, K52 = 5 * K / 8, L52 = K52 / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* s_r52r = smem;
  for (int i = threadIdx.x; i < K; i += blockDim.x) s_r52r[i] = row[i];
  __syncthreads();
  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long inst = (long long)blockIdx.x * IPB + slot;
  if (inst >= count) return;
  uint32_t n2[L], x[L], xr[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.load(x, in + inst * K);
  if (!g.less_than(x, n2)) {
    if (g.gl == 0) atomicOr(status, ST_RANGE);
    return;
  }
  g.mont_mul(xr, x, s_r52r, n2, ks.ninv2);  // x R52 mod n^2
  uint32_t* s_w = smem + K + slot * K;
  g.publish(s_w, xr);
#pragma unroll
  for (int k = 0; k < L52; ++k)
    out[inst * K52 + g.gl * L52 + k] = cuhe52::to_f64(limb52_from_words(s_w, K, g.gl * L52 + k));
}


template <int K>
__global__ void __launch_bounds__(kBlockThreads, 3)
k_mulmod_outer52(const double* __restrict__ q52, const uint32_t* __restrict__ index, long long nx,
                 uint32_t* __restrict__ out, const uint32_t* __restrict__ consts, const double* __restrict__ n52,
                 unsigned long long ninv52, int* status) {
  constexpr int TPI = K / 16, L = 16, K52 = 5 * K / 8, L52 = K52 / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  extern __shared__ __align__(16) double smd[];
  double* s_b = smd;          // the query, K52 limbs (Montgomery form)
  double* s_inst = smd + K52; // per instance K52 doubles: the index words in, the result limbs out
  const long long qi = blockIdx.y;
  for (int i = threadIdx.x; i < K52; i += blockDim.x) s_b[i] = q52[qi * K52 + i];
  __syncthreads();
  Group<K, TPI> g;
  cuhe52::Group52<K52, TPI> f;
  const int slot = threadIdx.x / TPI;
  const long long j = (long long)blockIdx.x * IPB + slot;
  if (j >= nx) return;
  uint32_t n2[L], x[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.load_ro(x, index + j * K);
  if (!g.less_than(x, n2)) {
    if (g.gl == 0) atomicOr(status, ST_RANGE);
    return;
  }
  uint32_t* s_w = reinterpret_cast<uint32_t*>(s_inst + slot * K52);
  g.publish(s_w, x);
  double a52[L52], m52[L52], r52[L52];
#pragma unroll
  for (int k = 0; k < L52; ++k) {
    a52[k] = cuhe52::to_f64(limb52_from_words(s_w, K, f.gl * L52 + k));
    m52[k] = __ldg(n52 + f.gl * L52 + k);
  }
  f.mont_mul(r52, a52, s_b, m52, ninv52);
  uint64_t* s_l = reinterpret_cast<uint64_t*>(s_inst + slot * K52);
  __syncwarp(f.mask);
#pragma unroll
  for (int k = 0; k < L52; ++k) s_l[f.gl * L52 + k] = cuhe52::to_u64(r52[k]);
  __syncwarp(f.mask);
  uint32_t w[L];
#pragma unroll
  for (int t = 0; t < L; ++t) w[t] = word_from_limbs52(s_l, K52, g.gl * L + t);
  g.store(out + (qi * nx + j) * K, w);
}

// ---------------------------------------------------------------------------
// Modular exponentiation with a per-instance exponent (fixed 4-bit windows, so
// every group of a warp follows the same schedule):
//   out[i] = base[i]^exps[i] mod n^2, exps[i] held in exp_words words.
// ---------------------------------------------------------------------------
template <int K, int TPI>
__global__ void __launch_bounds__(kBlockThreads)
k_modexp_var(const uint32_t* __restrict__ base, const uint32_t* __restrict__ exps, int exp_words, int windows,
             uint32_t* __restrict__ out, long long count, const uint32_t* __restrict__ consts, KeyScalars ks,
             int* status) {
  constexpr int L = K / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  constexpr int T = 16;
  constexpr int STRIDE = inst_stride_words<K>(T + 1);
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* s_one = smem;
  uint32_t* s_r2 = smem + K;
  {
    const int rows[2] = {C_ONE, C_R2};
    copy_rows_to_smem<K, TPI>(smem, consts, rows, 2);
  }
  __syncthreads();
  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long inst = (long long)blockIdx.x * IPB + slot;
  if (inst >= count) return;
  uint32_t* s_x = smem + 2 * K + slot * STRIDE;
  uint32_t* s_tab = s_x + K;
  uint32_t n2[L], x[L], acc[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.load(x, base + inst * K);
  if (!g.less_than(x, n2)) {
    if (g.gl == 0) atomicOr(status, ST_RANGE);
    return;
  }
  g.load_ro(acc, consts + C_RM * K);
  g.publish(s_tab, acc);                   // x^0
  g.mont_mul(acc, x, s_r2, n2, ks.ninv2);  // x^1
  g.publish(s_tab + K, acc);
  g.publish(s_x, acc);
#pragma unroll 1
  for (int t = 2; t < T; ++t) {
    g.mont_mul(acc, acc, s_x, n2, ks.ninv2);
    g.publish(s_tab + t * K, acc);
  }
  const uint32_t* e = exps + inst * exp_words;
  g.load_ro(acc, consts + C_RM * K);
  g.publish(s_x, acc);
  bool started = false;
#pragma unroll 1
  for (int w = windows - 1; w >= 0; --w) {
    const int bit = 4 * w;
    const int digit = (bit / 32 < exp_words) ? int((__ldg(e + bit / 32) >> (bit % 32)) & 15u) : 0;
    if (started) {
#pragma unroll 1
      for (int s = 0; s < 4; ++s) {
        g.mont_mul(acc, acc, s_x, n2, ks.ninv2);
        g.publish(s_x, acc);
      }
    }
    if (digit) {
      g.mont_mul(acc, acc, s_tab + digit * K, n2, ks.ninv2);
      g.publish(s_x, acc);
      started = true;
    }
  }
  g.mont_mul(x, acc, s_one, n2, ks.ninv2);
  g.store(out + inst * K, x);
}

// distance[v] = sum of the chunk_num per-chunk popcounts of vector v.
__global__ void k_sum_chunks(const uint32_t* __restrict__ counts, long long vectors, int chunk_num,
                             long long* __restrict__ distance) {
  const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= vectors) return;
  long long s = 0;
  for (int c = 0; c < chunk_num; ++c) s += counts[v * chunk_num + c];
  distance[v] = s;
}

// Integer multiply-add throughput probe in the Montgomery kernels' own
// instruction mix: four independent 8-limb accumulators, each updated per
// iteration by one mad.lo.cc/madc.hi.cc row (8 word products, the shape of
// Group::mac_row) with no shuffles or memory traffic, so the probe is bound
// only by the integer multiply pipe.  Each row is 8 word products.
// FP64-pipe probe: eight independent fused multiply-add chains per thread
// (round toward zero, the form of the limb products), FP64 instructions only.
__global__ void __launch_bounds__(256) k_fp64_probe(double* sink, int iters, double seed) {
  double x[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) x[j] = seed + 1e-3 * double(threadIdx.x) + double(j);
  const double y = 1.0000000001, z = 1e-9;
#pragma unroll 1
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = __fma_rz(x[j], y, z);
  }
  double folded = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) folded += x[j];
  if (folded == 1.2345678) sink[0] = folded;
}

__global__ void __launch_bounds__(256) k_imad_chain_probe(uint32_t* sink, int iters, uint32_t seed) {
  uint32_t acc[4][8], c0[4], c1[4], a[8];
  const uint32_t b = seed * 2654435761u + blockIdx.x;
#pragma unroll
  for (int j = 0; j < 8; ++j) a[j] = (seed ^ threadIdx.x) * (j + 3u) + 0x9e3779b9u;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    c0[s] = c1[s] = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[s][j] = a[j] ^ s;
  }
#pragma unroll 1
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int s = 0; s < 4; ++s) Group<128, 16>::mac_row(acc[s], c0[s], c1[s], a, b + s);
  }
  uint32_t folded = 0;
#pragma unroll
  for (int s = 0; s < 4; ++s) {
    folded ^= c0[s] ^ c1[s];
#pragma unroll
    for (int j = 0; j < 8; ++j) folded ^= acc[s][j];
  }
  if (folded == 0x12345678u) sink[0] = folded;
}

// Integer multiply-add throughput probe in 64-bit form: every iteration
// issues one mad.wide.u32 (a full 32x32->64 word product added to a 64-bit
// accumulator) on each of eight independent accumulators.
__global__ void __launch_bounds__(256) k_imad_wide_probe(uint32_t* sink, int iters, uint32_t seed) {
  unsigned long long acc[8];
  const uint32_t b = seed * 2654435761u + blockIdx.x;
#pragma unroll
  for (int j = 0; j < 8; ++j) acc[j] = ((unsigned long long)(seed ^ threadIdx.x) << 7) + 977u * j + 1u;
#pragma unroll 1
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const uint32_t lo = uint32_t(acc[j]);
      asm volatile("mad.wide.u32 %0, %1, %2, %0;" : "+l"(acc[j]) : "r"(lo), "r"(b));
    }
  }
  unsigned long long folded = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) folded ^= acc[j];
  if (folded == 0x9e3779b97f4a7c15ull) sink[0] = uint32_t(folded);
}

// Integer multiply-add throughput probe: every iteration issues one
// mad.lo.u32 and one mad.hi.u32 (one 32x32->64 word product) per operand
// pair into 16 accumulators that depend only on themselves.
__global__ void __launch_bounds__(256) k_imad_probe(uint32_t* sink, int iters, uint32_t seed) {
  uint32_t lo[8], hi[8], x[8];
  const uint32_t a = seed ^ threadIdx.x, b = seed * 2654435761u + blockIdx.x;
#pragma unroll
  for (int j = 0; j < 8; ++j) { lo[j] = a + j; hi[j] = b - j; x[j] = (a * 33u) ^ (b + 7u * j); }
#pragma unroll 1
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      asm volatile("mad.lo.u32 %0, %1, %2, %0;" : "+r"(lo[j]) : "r"(x[j]), "r"(b));
      asm volatile("mad.hi.u32 %0, %1, %2, %0;" : "+r"(hi[j]) : "r"(x[j]), "r"(b));
    }
  }
  uint32_t folded = 0;
#pragma unroll
  for (int j = 0; j < 8; ++j) folded ^= lo[j] ^ hi[j];
  if (folded == 0x9e3779b9u) sink[0] = folded;
}

// ---------------------------------------------------------------------------
// Pointwise modular multiplication: out[i] = a[i] * b[i] mod n^2.
// ---------------------------------------------------------------------------
template <int K, int TPI>
__global__ void __launch_bounds__(kBlockThreads)
k_mulmod(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b, uint32_t* __restrict__ out,
         long long count, const uint32_t* __restrict__ consts, KeyScalars ks, int* status) {
  constexpr int L = K / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  constexpr int STRIDE = inst_stride_words<K>(1);
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* s_r2 = smem;
  {
    const int rows[1] = {C_R2};
    copy_rows_to_smem<K, TPI>(smem, consts, rows, 1);
  }
  __syncthreads();
  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long inst = (long long)blockIdx.x * IPB + slot;
  if (inst >= count) return;
  uint32_t* s_b = smem + K + slot * STRIDE;
  uint32_t n2[L], x[L], y[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.load(x, a + inst * K);
  g.load(y, b + inst * K);
  if (!g.less_than(x, n2) || !g.less_than(y, n2)) {
    if (g.gl == 0) atomicOr(status, ST_RANGE);
    return;
  }
  g.publish(s_b, y);
  g.mont_mul(x, x, s_b, n2, ks.ninv2);   // a b R^-1
  g.mont_mul(x, x, s_r2, n2, ks.ninv2);  // a b
  g.store(out + inst * K, x);
}

// out[q][j] = query[q] * index[j] mod n^2 with queries given in Montgomery form
// (query * R mod n^2).  One Montgomery product per output.
template <int K, int TPI>
__global__ void __launch_bounds__(kBlockThreads)
k_mulmod_outer(const uint32_t* __restrict__ qmont, long long nq, const uint32_t* __restrict__ index,
               long long nx, uint32_t* __restrict__ out, const uint32_t* __restrict__ consts, KeyScalars ks,
               int* status) {
  constexpr int L = K / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  extern __shared__ __align__(16) uint32_t smem[];
  const long long qi = blockIdx.y;
  for (int i = threadIdx.x; i < K; i += blockDim.x) smem[i] = qmont[qi * K + i];
  __syncthreads();
  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long j = (long long)blockIdx.x * IPB + slot;
  if (j >= nx) return;
  uint32_t n2[L], x[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.load_ro(x, index + j * K);
  if (!g.less_than(x, n2)) {
    if (g.gl == 0) atomicOr(status, ST_RANGE);
    return;
  }
  g.mont_mul(x, x, smem, n2, ks.ninv2);
  g.store(out + (qi * nx + j) * K, x);
}

// out[i] = in[i] * R mod n^2 (to Montgomery form), or in[i] * R^-1 (from).
template <int K, int TPI>
__global__ void __launch_bounds__(kBlockThreads)
k_convert(const uint32_t* __restrict__ in, uint32_t* __restrict__ out, long long count,
          const uint32_t* __restrict__ consts, KeyScalars ks, int to_mont, int* status) {
  constexpr int L = K / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  extern __shared__ __align__(16) uint32_t smem[];
  {
    const int rows[1] = {to_mont ? (int)C_R2 : (int)C_ONE};
    copy_rows_to_smem<K, TPI>(smem, consts, rows, 1);
  }
  __syncthreads();
  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long inst = (long long)blockIdx.x * IPB + slot;
  if (inst >= count) return;
  uint32_t n2[L], x[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.load(x, in + inst * K);
  // to_mont == 2: any x < 2^(32K) (x R mod n^2: the CIOS bound holds for any
  // first operand below R), the first half of a reduction mod n^2
  if (to_mont != 2 && !g.less_than(x, n2)) {
    if (g.gl == 0) atomicOr(status, ST_RANGE);
    return;
  }
  g.mont_mul(x, x, smem, n2, ks.ninv2);
  g.store(out + inst * K, x);
}

// Hexadecimal text <-> little-endian 32-bit limbs, one thread per limb.
// Value i is text[offsets[i], offsets[i+1]) with an optional 0x / 0X
// prefix; limb w holds the digits 8w .. 8w+7 counted from the right, digits
// beyond the K-th limb are dropped (the reference's hex_to_le_words keeps
// the low limbs), and any character that is not a hex digit sets ST_HEX.
enum : int { ST_HEX = 2 };

__device__ __forceinline__ int hex_value(char c) {
  if (c >= '0' && c <= '9') return c - '0';
  if (c >= 'a' && c <= 'f') return c - 'a' + 10;
  if (c >= 'A' && c <= 'F') return c - 'A' + 10;
  return -1;
}

__global__ void k_hex_to_limbs(const char* __restrict__ text, const long long* __restrict__ offsets, long long count,
                               int words, uint32_t* __restrict__ out, int* status) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count * words) return;
  const long long i = t / words;
  const int w = int(t - i * words);
  long long s = offsets[i];
  const long long e = offsets[i + 1];
  if (e - s >= 2 && text[s] == '0' && (text[s + 1] == 'x' || text[s + 1] == 'X')) s += 2;
  uint32_t v = 0;
  bool bad = false;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const long long pos = e - 1 - 8ll * w - j;
    if (pos >= s) {
      const int d = hex_value(text[pos]);
      bad |= d < 0;
      v |= uint32_t(d < 0 ? 0 : d) << (4 * j);
    }
  }
  if (w == words - 1)
    for (long long pos = s; pos < e - 8ll * words; ++pos) bad |= hex_value(text[pos]) < 0;
  out[t] = v;
  if (bad) atomicOr(status, ST_HEX);
}

// out[i * 8 words ...]: value i as 8 * words lowercase digits, most significant first
__global__ void k_limbs_to_hex(const uint32_t* __restrict__ limbs, long long count, int words, char* __restrict__ out) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count * words) return;
  const long long i = t / words;
  const int w = int(t - i * words);
  const uint32_t v = limbs[t];
  char* o = out + i * 8ll * words + 8ll * (words - 1 - w);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const uint32_t d = (v >> (4 * (7 - j))) & 15u;
    o[j] = char(d < 10 ? '0' + d : 'a' + d - 10);
  }
}

// ---------------------------------------------------------------------------
// Paillier-Lookup encryption by fixed-base table product:
//   c = prod_i G[i][digit_i(m)] * prod_k NOISE[idx_k]  mod n^2
// G and NOISE are device-resident in Montgomery form.  The plaintext digits
// come either from binary embeddings (Hamming padding "0b" per bit, read as
// MSB-first chunks of chunk_len bits) or from little-endian plaintext words.
// kWide: G is the 16-bit-digit table W[j][D] = G[2j][D mod 256] *
// G[2j+1][D / 256] (k_wide_table), one product per pair of 8-bit digits; the
// product of the same powers of g, so the ciphertext is the same.  The next
// table row is loaded while the current product runs.
// ---------------------------------------------------------------------------
constexpr int kNoiseMultiples = 14;

// 16-bit entries of row list per instance: message_chunks rounded up to even
__host__ __device__ constexpr int lookup_rows_stride(int message_chunks) { return (message_chunks + 1) & ~1; }

// The table rows of an instance's nonzero digits (one lane): 8-bit digits as
// i * 256 + d into rows16, or with kWide 16-bit digits as j * 65536 + D into
// rows32 (the same storage); returns their count.  Digits come from a binary
// embedding (Hamming padding "0b" per bit, MSB-first chunks of chunk_len
// bits) or from little-endian plaintext words.
template <bool kWide>
__device__ __forceinline__ int lookup_digit_rows(const uint8_t* __restrict__ bits, int embed_len, int chunk_len,
                                                 int chunk_num, const uint32_t* __restrict__ plain, int plain_words,
                                                 long long inst, int message_chunks, uint16_t* s_rows16) {
  uint32_t* s_rows32 = reinterpret_cast<uint32_t*>(s_rows16);
  int cnt = 0;
  int pending = 0;  // kWide: the low byte of the current 16-bit digit
  auto push = [&](int i, int d) {
    if (kWide) {
      if ((i & 1) == 0) {
        pending = d;
        if (i + 1 == message_chunks && d) s_rows32[cnt++] = uint32_t(i / 2) * 65536u + uint32_t(d);
      } else if (pending | d) {
        s_rows32[cnt++] = uint32_t(i / 2) * 65536u + uint32_t(pending + 256 * d);
      }
    } else if (d) {
      s_rows16[cnt++] = uint16_t(i * 256 + d);
    }
  };
  if (bits) {
    const long long vec = inst / chunk_num;
    const int chunk = int(inst % chunk_num);
    const int padded_total = 2 * embed_len;
    const int cbase = chunk * chunk_len;
    int avail = padded_total - cbase;
    if (avail > chunk_len) avail = chunk_len;
    if (avail < 0) avail = 0;
    const uint8_t* vb = bits + vec * embed_len;
    for (int i = 0; i < message_chunks; ++i) {
      int d = 0;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const int e = 8 * i + b;  // exponent within the chunk value
        if (e < avail) {
          const int p = cbase + (avail - 1 - e);  // padded MSB-first position
          if (p & 1) d |= (vb[p >> 1] & 1) << b;
        }
      }
      push(i, d);
    }
  } else {
    const uint8_t* mb = reinterpret_cast<const uint8_t*>(plain + inst * plain_words);
    const int bytes = plain_words * 4 < message_chunks ? plain_words * 4 : message_chunks;
    for (int i = 0; i < message_chunks; ++i) push(i, i < bytes ? int(mb[i]) : 0);
  }
  return cnt;
}

template <int K, int TPI, bool kWide = false>
__global__ void __launch_bounds__(kBlockThreads)
k_lookup_encrypt(const uint8_t* __restrict__ bits, int embed_len, int chunk_len, int chunk_num,
                 const uint32_t* __restrict__ plain, int plain_words, long long count, int message_chunks,
                 const uint32_t* __restrict__ gtab, const uint32_t* __restrict__ noise, int noise_entries,
                 const uint8_t* __restrict__ noise_idx, uint32_t* __restrict__ out,
                 const uint32_t* __restrict__ consts, KeyScalars ks, int* status) {
  constexpr int L = K / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  constexpr int ACC_STRIDE = inst_stride_words<K>(1);
  extern __shared__ __align__(16) uint32_t smem[];
  uint32_t* s_one = smem;
  {
    const int rows[1] = {C_ONE};
    copy_rows_to_smem<K, TPI>(smem, consts, rows, 1);
  }
  __syncthreads();
  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long inst = (long long)blockIdx.x * IPB + slot;
  if (inst >= count) return;
  uint32_t* s_acc = smem + K + slot * ACC_STRIDE;
  // table rows of the nonzero digits: 8-bit digits as i * 256 + d (16 bits),
  // 16-bit digits as j * 65536 + D (32 bits); lookup_rows_stride(message_chunks)
  // 16-bit entries (a multiple of four bytes) a slot either way
  uint16_t* s_rows16 =
      reinterpret_cast<uint16_t*>(smem + K + IPB * ACC_STRIDE) + slot * lookup_rows_stride(message_chunks);
  uint32_t* s_rows32 = reinterpret_cast<uint32_t*>(s_rows16);
  __shared__ int s_count[IPB];

  // nonzero digits -> list of table rows (lane 0 of the group)
  if (g.gl == 0)
    s_count[slot] = lookup_digit_rows<kWide>(bits, embed_len, chunk_len, chunk_num, plain, plain_words, inst,
                                             message_chunks, s_rows16);
  __syncwarp(g.mask);
  const int cnt = s_count[slot];
  auto row_of = [&](int j) -> long long { return kWide ? (long long)s_rows32[j] : (long long)s_rows16[j]; };

  uint32_t n2[L], acc[L], a[L], nx[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.load_ro(acc, consts + C_RM * K);  // Montgomery one
  g.publish(s_acc, acc);
  if (cnt > 0) g.load_ro(a, gtab + row_of(0) * K);
#pragma unroll 1
  for (int j = 0; j < cnt; ++j) {
    if (j + 1 < cnt) g.load_ro(nx, gtab + row_of(j + 1) * K);
    g.mont_mul(acc, a, s_acc, n2, ks.ninv2);
    g.publish(s_acc, acc);
#pragma unroll
    for (int k = 0; k < L; ++k) a[k] = nx[k];
  }
  const uint8_t* idx = noise_idx + inst * kNoiseMultiples;
#pragma unroll 1
  for (int k = 0; k < kNoiseMultiples; ++k) {
    const int r = idx[k];
    if (r >= noise_entries) {
      if (g.gl == 0) atomicOr(status, ST_RANGE);
      return;
    }
    g.load_ro(a, noise + (long long)r * K);
    g.mont_mul(acc, a, s_acc, n2, ks.ninv2);
    g.publish(s_acc, acc);
  }
  g.mont_mul(a, acc, s_one, n2, ks.ninv2);
  g.store(out + inst * K, a);
}

// The 16-bit-digit table: W[j][D] = G[2j][D mod 256] * G[2j+1][D / 256]
// (Montgomery form in and out; the digit zero's factor, and for an odd
// message_chunks the last row's high factor, is 1).  One group per entry.
template <int K, int TPI>
__global__ void __launch_bounds__(kBlockThreads)
k_wide_table(const uint32_t* __restrict__ gtab, int message_chunks, uint32_t* __restrict__ wide,
             const uint32_t* __restrict__ consts, KeyScalars ks) {
  constexpr int L = K / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  constexpr int STRIDE = inst_stride_words<K>(1);
  extern __shared__ __align__(16) uint32_t smem[];
  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long inst = (long long)blockIdx.x * IPB + slot;  // j * 65536 + D
  const int wide_chunks = (message_chunks + 1) / 2;
  if (inst >= (long long)wide_chunks * 65536) return;
  const int j = int(inst >> 16), D = int(inst & 65535);
  uint32_t* s_b = smem + slot * STRIDE;
  uint32_t n2[L], lo[L], hi[L], r[L];
  g.load_ro(n2, consts + C_N2 * K);
  if (D & 255) g.load_ro(lo, gtab + ((long long)(2 * j) * 256 + (D & 255)) * K);
  else g.load_ro(lo, consts + C_RM * K);
  if (2 * j + 1 < message_chunks && D >> 8) g.load_ro(hi, gtab + ((long long)(2 * j + 1) * 256 + (D >> 8)) * K);
  else g.load_ro(hi, consts + C_RM * K);
  g.publish(s_b, hi);
  g.mont_mul(r, lo, s_b, n2, ks.ninv2);
  g.store(wide + inst * K, r);
}

// ---------------------------------------------------------------------------
// Paillier-Lookup encryption on pairs of residues mod n (pair52.cuh): tables
// and noise entries are rows of KL limb pairs in the R domain, a product is
// five n-wide limb products, and the ciphertext leaves as in k_pair_modexp.
//
// Digits.  Plaintext words are read as 8-bit digits (or 16-bit, with the wide
// table).  A binary embedding sets every second plaintext bit only, so the
// table of its digits is indexed by embedding bits: 8 of them (16 plaintext
// bits) by 256 rows, or 16 (32 plaintext bits) by 65,536, which halves the
// rows per ciphertext again and the wide table with them.  Noise entries
// come one by one or, for large calls, two at a time from a table of all
// their products.  At key_len 1024 an embedding of 512 bits takes 64 + 14,
// or wide 32 + 7, products instead of 120 + 14 and 64 + 14.
// ---------------------------------------------------------------------------

// A row's limb pairs stand in the order of the ten-limb kernels' loads: limb
// 10 g + k at k (KL / 10) + g, so that a group's lanes read neighbours.
template <int KL, int kL>
__device__ __forceinline__ int pair_row_slot(int gl, int k) {
  constexpr int T = KL / 10;
  if (kL == 10) return k * T + gl;
  return ((gl & 1) * 5 + k) * T + (gl >> 1);
}

// out[i] = in[i] as a row: in = K words in the 32-bit Montgomery form x 2^(32K)
// mod n^2, entry = R^(j+2) 2^(-32K) mod n^2 as pairs for the two chunks.  one:
// null, or that form of 1, which takes the place of every 256th row from the
// first: the digit zero, which the 8-bit kernel never looks up, is looked up
// here where another group of the warp has a digit.
template <int K>
__global__ void __launch_bounds__(cuhe52::kPairThreads, 2)
k_pair_rows(const uint32_t* __restrict__ in, long long count, const uint32_t* __restrict__ one,
            double2* __restrict__ out,
            const double2* __restrict__ entry, const double* __restrict__ n52, unsigned long long ninv52) {
  constexpr int KL = 5 * K / 16, TPI = KL / 10, L = 10;
  extern __shared__ __align__(16) uint32_t smem[];
  double2* s_rows = reinterpret_cast<double2*>(smem);
  for (int i = threadIdx.x; i < 2 * KL + 1; i += blockDim.x) s_rows[i] = i < 2 * KL ? entry[i] : make_double2(0.0, 0.0);
  __syncthreads();
  cuhe52::Pair52<KL, TPI> f;
  const long long item = (long long)blockIdx.x * (cuhe52::kPairThreads / TPI) + threadIdx.x / TPI;
  const long long inst = min(item, count - 1);
  const uint32_t* x = one && inst % 256 == 0 ? one : in + inst * K;
  const uint64_t ninv = f.gl == 0 ? ninv52 : 0ull;
  double m[L], a[L], r[L];
  uint64_t A0[L], A1[L], S0[L], S1[L];
#pragma unroll
  for (int k = 0; k < L; ++k) m[k] = __ldg(n52 + f.gl * L + k);
#pragma unroll 1
  for (int j = 0; j < 2; ++j) {
#pragma unroll
    for (int k = 0; k < L; ++k) a[k] = f.to_f64(limb52_from_words(x, K, j * KL + f.gl * L + k));
    f.template product<false>(A0, A1, a, a, s_rows + j * KL, m, ninv);
    f.template columns<2>(A0);
    f.template columns<2>(A1);
#pragma unroll
    for (int k = 0; k < L; ++k) {
      S0[k] = j ? S0[k] + A0[k] : A0[k];
      S1[k] = j ? S1[k] + A1[k] : A1[k];
    }
  }
  f.from_columns(a, S0);
  f.from_columns(r, S1);
  if (item >= count) return;
#pragma unroll
  for (int k = 0; k < L; ++k) out[item * KL + pair_row_slot<KL, L>(f.gl, k)] = make_double2(a[k], r[k]);
}

// Table of products of two rows of one source: entry i = x y, with
//   kEmbed  row j = i / 256 of 8 embedding bits b: digits 2j and 2j + 1 of the
//           8-bit table at the bits of b spread to the even places
//   kWide   row j = i / 65536 of 16 bits D: rows 2j and 2j + 1 at D's bytes
//   kNoise  i = a entries + b: noise entries a and b
// A factor past the source's last row is one.  Entries [first, first + count)
// of the whole table, from the start of out.
enum PairProducts : int { kEmbed = 0, kWide = 1, kNoise = 2 };

__device__ __forceinline__ int spread4(int b) { return (b & 1) | (b & 2) << 1 | (b & 4) << 2 | (b & 8) << 3; }

template <int K>
__global__ void __launch_bounds__(cuhe52::kPairThreads, 2)
k_pair_products(const double2* __restrict__ src, int rows, int kind, long long first, long long count,
                double2* __restrict__ out, const double* __restrict__ n52, unsigned long long ninv52) {
  constexpr int KL = 5 * K / 16, TPI = KL / 10, L = 10, kSlot = KL + 1;
  extern __shared__ __align__(16) uint32_t smem[];
  double2* s = reinterpret_cast<double2*>(smem) + (threadIdx.x / TPI) * kSlot;
  cuhe52::Pair52<KL, TPI> f;
  const long long item = first + (long long)blockIdx.x * (cuhe52::kPairThreads / TPI) + threadIdx.x / TPI;
  const long long i = min(item, first + count - 1);
  long long ia, ib;
  if (kind == kNoise) {
    ia = i / rows;
    ib = i % rows;
  } else {
    const int bits = kind == kWide ? 16 : 8;
    const int j = int(i >> bits), d = int(i & ((1 << bits) - 1));
    const int lo = kind == kWide ? d & 255 : spread4(d & 15), hi = kind == kWide ? d >> 8 : spread4(d >> 4);
    ia = (2ll * j) * 256 + lo;
    ib = 2 * j + 1 < rows ? (2ll * j + 1) * 256 + hi : -1;
  }
  // R mod n^2 stands in limb order, rows in their own
  const double2* one = reinterpret_cast<const double2*>(n52 + KL) + 4 * KL;
  double m[L], a0[L], a1[L], y0[L], y1[L];
  uint64_t A0[L], A1[L];
#pragma unroll
  for (int k = 0; k < L; ++k) {
    m[k] = __ldg(n52 + f.gl * L + k);
    const int slot = pair_row_slot<KL, L>(f.gl, k);
    const double2 x = __ldg(src + ia * KL + slot);
    const double2 y = ib >= 0 ? __ldg(src + ib * KL + slot) : __ldg(one + f.gl * L + k);
    a0[k] = x.x;
    a1[k] = x.y;
    y0[k] = y.x;
    y1[k] = y.y;
  }
  pair_publish<KL, TPI>(f, s, y0, y1);
  f.template product<true>(A0, A1, a0, a1, s, m, f.gl == 0 ? ninv52 : 0ull);
  f.template limbs<2>(a0, A0);
  f.template limbs<3>(a1, A1);
  if (item >= first + count) return;
#pragma unroll
  for (int k = 0; k < L; ++k) out[(item - first) * KL + pair_row_slot<KL, L>(f.gl, k)] = make_double2(a0[k], a1[k]);
}

// How a ciphertext's rows are found.
struct LookupDigits {
  const uint8_t* bits;    // embeddings, or null for plaintext words
  const uint32_t* plain;
  int embed_len, chunk_len, chunk_num, plain_words;
  int embed_bits;         // 8 or 16: digits of embedding bits; 0: of plaintext bits
  int wide;               // 16-bit digits
  int rows;               // rows of the table
  int message_chunks;     // 8-bit plaintext digits the tables cover
  const double2* const* embed_rows;  // 16 embedding bits: each row's 65,536 entries, in place of one table
};

__device__ __forceinline__ int lookup_digit(const LookupDigits& d, long long inst, int r) {
  int v = 0;
  if (d.bits) {
    const long long vec = inst / d.chunk_num;
    const int cbase = int(inst % d.chunk_num) * d.chunk_len;
    const int avail = min(max(2 * d.embed_len - cbase, 0), d.chunk_len);
    const uint8_t* vb = d.bits + vec * d.embed_len;
    if (d.embed_bits) {  // chunk_len is even: plaintext bit 2 i is embedding bit last - i
      const int last = (cbase + avail) / 2 - 1, n = d.embed_bits;
#pragma unroll 1
      for (int b = 0; b < n; ++b) {
        const int i = r * n + b;
        if (2 * i < avail) v |= (vb[last - i] & 1) << b;
      }
      return v;
    }
    const int n = d.wide ? 16 : 8;
#pragma unroll 1
    for (int b = 0; b < n; ++b) {
      const int e = n * r + b;  // exponent within the chunk value
      if (e >= avail || e >= 8 * d.message_chunks) break;
      const int p = cbase + (avail - 1 - e);  // padded MSB-first position
      if (p & 1) v |= (vb[p >> 1] & 1) << b;
    }
    return v;
  }
  const uint8_t* mb = reinterpret_cast<const uint8_t*>(d.plain + inst * d.plain_words);
  const int bytes = min(d.plain_words * 4, d.message_chunks);
  if (!d.wide) return r < bytes ? int(mb[r]) : 0;
  if (2 * r < bytes) v = mb[2 * r];
  if (2 * r + 1 < bytes) v |= int(mb[2 * r + 1]) << 8;
  return v;
}

template <int K, int kL>
struct LookupLayout {
  static constexpr int KL = 5 * K / 16, TPI = KL / kL;
  static constexpr int kGroups = cuhe52::kPairThreads / TPI, kSlot = KL + 1;
  static size_t bytes(int rows) {  // (1, 0), the values, n R in words, the digits
    return size_t(kSlot + kGroups * kSlot) * 16 + size_t(K) * 4 + size_t(kGroups) * ((rows + 1) & ~1) * 2;
  }
};

template <int K, int kL>
__global__ void __launch_bounds__(cuhe52::kPairThreads, 2)
k_pair_lookup(LookupDigits dg, long long count, const double2* __restrict__ table, const double2* __restrict__ noise,
              int noise_entries, int noise_pairs, const uint8_t* __restrict__ noise_idx, uint32_t* __restrict__ out,
              const uint32_t* __restrict__ consts, KeyScalars ks, const double* __restrict__ n52,
              unsigned long long ninv52, int* status) {
  using Lay = LookupLayout<K, kL>;
  constexpr int KL = Lay::KL, TPI = Lay::TPI, L = kL, IPB = Lay::kGroups;
  extern __shared__ __align__(16) uint32_t smem[];
  double2* s_unit = reinterpret_cast<double2*>(smem);
  double2* s_vals = s_unit + Lay::kSlot;
  uint32_t* s_nr = reinterpret_cast<uint32_t*>(s_vals + IPB * Lay::kSlot);
  uint16_t* s_digits = reinterpret_cast<uint16_t*>(s_nr + K);
  for (int i = threadIdx.x; i < Lay::kSlot; i += blockDim.x) s_unit[i] = make_double2(i == 0 ? 1.0 : 0.0, 0.0);
  for (int i = threadIdx.x; i < K; i += blockDim.x) s_nr[i] = consts[C_NR * K + i];
  __syncthreads();
  const long long first = (long long)blockIdx.x * IPB;
  bool valid = true;
  {
    cuhe52::Pair52<KL, TPI> f;
    const int group = threadIdx.x / TPI;
    const long long inst = min(first + group, count - 1);  // idle groups repeat the last item
    double2* s = s_vals + group * Lay::kSlot;
    uint16_t* digits = s_digits + group * ((dg.rows + 1) & ~1);
    for (int r = f.gl; r < dg.rows; r += TPI) digits[r] = uint16_t(lookup_digit(dg, inst, r));
    __syncwarp();
    const uint8_t* idx = noise_idx + inst * kNoiseMultiples;
    for (int k = 0; k < kNoiseMultiples; ++k) valid = valid && idx[k] < noise_entries;
    const int digit_bits = dg.embed_bits == 16 || dg.wide ? 16 : 8;
    const int noises = noise_pairs ? kNoiseMultiples / 2 : kNoiseMultiples;
    double m[L], a0[L], a1[L], z0[L], z1[L];
    uint64_t A0[L], A1[L];
#pragma unroll
    for (int k = 0; k < L; ++k) m[k] = __ldg(n52 + f.gl * L + k);
    const uint64_t ninv = f.gl == 0 ? ninv52 : 0ull;
    // the rows in order: digits that are not zero for every group of the
    // warp (a zero digit's row is one), then the noise
    auto next = [&](int t) {
      while (t < dg.rows && !__any_sync(0xffffffffu, digits[t] != 0)) ++t;
      return t;
    };
    auto row = [&](int t) -> const double2* {
      if (t < dg.rows) {
        if (dg.embed_rows) return dg.embed_rows[t] + static_cast<long long>(digits[t]) * KL;
        return table + ((static_cast<long long>(t) << digit_bits) + digits[t]) * KL;
      }
      const int k = t - dg.rows;
      if (!valid) return noise;
      if (noise_pairs) return noise + (static_cast<long long>(idx[2 * k]) * noise_entries + idx[2 * k + 1]) * KL;
      return noise + static_cast<long long>(idx[k]) * KL;
    };
    int t = next(0);
    const int end = dg.rows + noises;
    bool begun = false;
#pragma unroll 1
    while (true) {
      const bool out_now = t >= end;
      if (!out_now) {
        const double2* r = row(t);
#pragma unroll
        for (int k = 0; k < L; ++k) {
          const double2 v = __ldg(r + pair_row_slot<KL, L>(f.gl, k));
          a0[k] = v.x;
          a1[k] = v.y;
        }
        t = t < dg.rows ? next(t + 1) : t + 1;
        if (t < end) {  // bring the next row closer while this product runs
          const double2* ahead = row(t);
          for (int k = f.gl; k * 8 < KL; k += TPI) asm volatile("prefetch.global.L1 [%0];" ::"l"(ahead + k * 8));
        }
        if (!begun) {  // the first row is the value
          begun = true;
#pragma unroll
          for (int k = 0; k < L; ++k) {
            z0[k] = a0[k];
            z1[k] = a1[k];
          }
          continue;
        }
        pair_publish<KL, TPI>(f, s, z0, z1);
      } else {
#pragma unroll
        for (int k = 0; k < L; ++k) {
          a0[k] = z0[k];
          a1[k] = z1[k];
        }
      }
      f.template product<true>(A0, A1, a0, a1, out_now ? s_unit : s, m, ninv);
      if (out_now) break;
      f.template limbs<2>(z0, A0);
      f.template limbs<3>(z1, A1);
    }
    f.template columns<2>(A0);
    f.template columns<3>(A1);
    f.canonical(A0);
    f.canonical(A1);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < L; ++k)
      s[f.gl * L + k] = make_double2(__longlong_as_double(static_cast<long long>(A0[k])),
                                     __longlong_as_double(static_cast<long long>(A1[k])));
    // the validity of a group's noise indexes, for the lanes that store it
    if (f.gl == 0) s[KL].x = valid ? 1.0 : 0.0;
  }
  __syncthreads();
  constexpr int LT = K / 16, LW = 16, PER = cuhe52::kPairThreads / LT;
  Group<K, LT> g;
  uint32_t n2[LW], x[LW];
  g.load_ro(n2, consts + C_N2 * K);
#pragma unroll 1
  for (int item = threadIdx.x / LT; item < IPB; item += PER) {
    const long long inst = first + item;
    if (inst >= count) break;
    const double2* s = s_vals + item * Lay::kSlot;
    if (s[KL].x == 0.0) {
      if (g.gl == 0) atomicOr(status, ST_RANGE);
      continue;
    }
    pair_words<KL, K, LT>(g, x, s, s_nr, n2, ks.ninv2);
    g.store(out + inst * K, x);
  }
}

// ---------------------------------------------------------------------------
// Fixed-base table construction: rows i of G = base_i^j, j = 0..255, with
// base_i = g^(2^(8i)) (all in Montgomery form).  One group per (row, chunk of
// 16 consecutive j); thread-level work is 16 sequential products.
// ---------------------------------------------------------------------------
template <int K, int TPI>
__global__ void __launch_bounds__(kBlockThreads)
k_table_rows(const uint32_t* __restrict__ bases_mont, int rows, uint32_t* __restrict__ gtab,
             const uint32_t* __restrict__ consts, KeyScalars ks) {
  constexpr int L = K / TPI;
  constexpr int IPB = kBlockThreads / TPI;
  constexpr int STRIDE = inst_stride_words<K>(2);
  extern __shared__ __align__(16) uint32_t smem[];
  Group<K, TPI> g;
  const int slot = threadIdx.x / TPI;
  const long long inst = (long long)blockIdx.x * IPB + slot;  // row * 16 + block of j
  if (inst >= (long long)rows * 16) return;
  const int row = int(inst / 16);
  const int jb = int(inst % 16);
  uint32_t* s_base = smem + slot * STRIDE;
  uint32_t* s_pow = s_base + K;
  uint32_t n2[L], b[L], p[L];
  g.load_ro(n2, consts + C_N2 * K);
  g.load_ro(b, bases_mont + (long long)row * K);
  g.publish(s_base, b);
  // p = base^(16*jb) via square-and-multiply over the 8-bit exponent
  g.load_ro(p, consts + C_RM * K);
  const int e = 16 * jb;
#pragma unroll 1
  for (int bit = 7; bit >= 0; --bit) {
    g.publish(s_pow, p);
    g.mont_mul(p, p, s_pow, n2, ks.ninv2);
    if ((e >> bit) & 1) g.mont_mul(p, p, s_base, n2, ks.ninv2);
  }
#pragma unroll 1
  for (int t = 0; t < 16; ++t) {
    g.store(gtab + ((long long)row * 256 + e + t) * K, p);
    g.mont_mul(p, p, s_base, n2, ks.ninv2);
  }
}

}  // namespace cuhe
