// k_pair_crt and k_pair_modexp with a pair's components on different lanes
// (pair52_split.cuh): the layout and the exponentiation they call.
#pragma once
#include "paillier_kernels.cuh"
// after the limb constants
#include "pair52_split.cuh"

namespace cuhe {

template <int K, int kEntry, int kSides>
struct PairLayout<K, kSplit, kEntry, kSides> {
  static constexpr int L = 5, kHalf = K / L;                 // limbs and lanes per component
  static constexpr int TPI = 2 * kHalf;                      // lanes per value
  static constexpr int kGroups = cuhe52::kPairThreads / TPI;
  static constexpr int kItems = kGroups / kSides;
  static constexpr int kRows = (kEntry + 2) * (K + 4);       // constants per modulus, in pairs of doubles
  static constexpr int kSlot = K + 1;
  // doubles: the powers of one component per thread; the operands, and zeros
  static constexpr size_t kTab = size_t(1 << (kSplitWindow - 1)) * L * cuhe52::kPairThreads;
  static constexpr size_t kWork = size_t(3 * kGroups + 1) * (K + 4);
  static constexpr size_t kBytes = (size_t(kSides) * kRows + size_t(kGroups) * kSlot) * 16 + (kTab + kWork) * 8;
};

// pair_power with the components on different lanes (pair52_split.cuh): the
// same results, by the exponent's wide schedule.  rows: the constants' arrays in shared memory
// (split_rows: kEntry entry rows of two components, then (1, 0)'s component 0
// twice, then the scale row), zeros: kOperand zeros; work: this value's three
// operand arrays (z0, 2 z0, t0), whose two leading limbs are zero; s: its K
// result pairs; tab: this thread's column of its component's powers.
template <int K, int TPI, int kEntry, bool kUnits>
__device__ __forceinline__ bool split_power(const cuhe52::Split52<K, TPI>& f, const uint32_t* __restrict__ words,
                                            int nwords, const double* rows, const double* zeros,
                                            const double2* __restrict__ one, double* work, double2* s, double* tab,
                                            const double (&m)[K / TPI], const PairExponent& ex,
                                            const uint32_t* __restrict__ aux) {
  using Split = cuhe52::Split52<K, TPI>;
  constexpr int L = K / TPI, kStride = cuhe52::kPairThreads, kArr = Split::kOperand;
  const int32_t* ops = ex.ops;
  int nops = ex.nops;
  bool halved = kUnits && ex.halved != 0, voted = false;
  double z[L], t[L], w[L];
  uint64_t A[L];
  const int at = f.f.gl * L;
  double* zarr = work;
  double* warr = work + kArr;
  double* tarr = work + 2 * kArr;
  auto row = [&](int r) { return f.operand(rows + (2 * r + f.half) * kArr); };
  // half 0's limbs x into an operand array
  auto publish = [&](double* arr, const double (&x)[L]) {
    if (f.half == 0) {
#pragma unroll
      for (int k = 0; k < L; ++k) arr[2 + at + k] = x[k];
    }
  };
  auto result = [&](double2* p) -> double* { return f.half ? &p->y : &p->x; };

  // entry: chunks times constants, summed as columns
  uint64_t S[L];
#pragma unroll
  for (int k = 0; k < L; ++k) S[k] = 0;
#pragma unroll 1
  for (int j = 0; j < kEntry; ++j) {
#pragma unroll
    for (int k = 0; k < L; ++k) z[k] = f.f.to_f64(limb52_from_words(words, nwords, j * K + at + k));
    f.template product<false>(A, z, z, row(j), zeros, m);
    f.f.template columns<2>(A);
#pragma unroll
    for (int k = 0; k < L; ++k) S[k] += A[k];
  }
  f.f.from_columns(z, S);
  while (true) {
    if (nops == 0) {  // e = 0
#pragma unroll
      for (int k = 0; k < L; ++k) {
        const double2 v = __ldg(one + at + k);
        z[k] = f.half ? v.y : v.x;
      }
    } else {
      const int32_t* wide = ops + nops;  // op count, odd powers, ops
      const int odd = __ldg(wide + 1);
      nops = __ldg(wide);
      ops = wide + 2;
      // x to the table and x^2 to z, then x^(2i+1) = x^(2i-1) x^2 in t
#pragma unroll
      for (int k = 0; k < L; ++k) {
        tab[k * kStride] = z[k];
        t[k] = z[k];
      }
      f.f.twice_limbs(w, z);
      __syncwarp();
      publish(zarr, z);
      publish(warr, w);
      publish(tarr, t);
      __syncwarp();
      f.template product<false>(A, z, z, f.half ? warr : zarr + 2, zeros, m);
      f.f.template limbs<2>(z, A);
      __syncwarp();
      publish(zarr, z);
      __syncwarp();
#pragma unroll 1
      for (int i = 1; i < odd; ++i) {
        f.template product<true>(A, t, z, f.operand(zarr), f.half ? tarr : zeros, m);
        f.f.template limbs<3>(t, A);
        __syncwarp();
        publish(tarr, t);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < L; ++k) tab[(i * L + k) * kStride] = t[k];
      }
      const int first = (__ldg(ops) & 0xffff) - 1;
#pragma unroll
      for (int k = 0; k < L; ++k) z[k] = tab[(first * L + k) * kStride];
    }
    f.f.twice_limbs(w, z);
    int op = nops > 1 ? __ldg(ops + 1) : 0;
#pragma unroll 1
    for (int o = 1;; ++o) {
      const bool out = o >= nops;
      const int sq = out ? 0 : op >> 16, idx = op & 0xffff;
      if (o + 1 < nops) op = __ldg(ops + o + 1);
#pragma unroll 1
      for (int i = 0; i < sq; ++i) {
        __syncwarp();
        publish(zarr, z);
        publish(warr, w);
        __syncwarp();
        f.template product<false>(A, z, z, f.half ? warr : zarr + 2, zeros, m);
        f.f.template limbs<2>(z, A);
        f.f.template twice<2>(w, A);
      }
      if (!out && idx == 0) continue;  // the schedule's last squarings
      __syncwarp();
      publish(zarr, z);
      const double* b = f.operand(zarr);
      const double* c = f.half ? tarr : zeros;
      if (out) {
        // z times (1, 0), or (1, aux): half 1 adds aux z0
        b = f.operand(rows + 2 * kEntry * kArr);
        c = f.half && aux ? zarr : zeros;
#pragma unroll
        for (int k = 0; k < L; ++k) {
          t[k] = z[k];
          A[k] = aux ? limb52_from_words(aux, nwords, at + k) : 0ull;
        }
        f.f.from_columns(w, A);
      } else {
#pragma unroll
        for (int k = 0; k < L; ++k) {
          t[k] = tab[((idx - 1) * L + k) * kStride];
          w[k] = z[k];
        }
        publish(tarr, t);
      }
      __syncwarp();
      f.template product<true>(A, t, w, b, c, m);
      if (out) break;
      f.f.template limbs<3>(z, A);
      f.f.template twice<3>(w, A);
    }
    f.f.template columns<3>(A);
    f.f.canonical(A);
    bool isone = true;
    __syncwarp();
#pragma unroll
    for (int k = 0; k < L; ++k) {
      *result(s + at + k) = __longlong_as_double(static_cast<long long>(A[k]));
      isone = isone && (f.half == 1 || A[k] == (at + k == 0 ? 1ull : 0ull));
    }
    __syncwarp();
    if (!kUnits) return false;
    if (!voted) {
      if (__syncthreads_and(isone)) break;
      voted = true;
    }
    if (!halved) return false;
    halved = false;  // raise x^(p-1) (still in z) to the cofactor
    ops = ex.fall;
    nops = ex.nfall;
  }
  // (1, z1) -> (1, z1 w mod m); half 0 multiplies by nothing
#pragma unroll
  for (int k = 0; k < L; ++k) t[k] = f.half ? f.f.to_f64(A[k]) : 0.0;
  f.template product<false>(A, t, t, f.operand(rows + 2 * (kEntry + 1) * kArr), zeros, m);
  f.f.template columns<2>(A);
  f.f.canonical(A);
  if (f.half) {
#pragma unroll
    for (int k = 0; k < L; ++k) s[at + k].y = __longlong_as_double(static_cast<long long>(A[k]));
  }
  return true;
}

// The constants' arrays for split_power from the pairs at `pairs` (kEntry + 2
// rows of K pairs): array (2 r + component) of kOperand doubles; the unit and
// scale rows hold their component 0 in both.
template <int K, int kEntry>
__device__ __forceinline__ void split_rows(double* out, const double2* __restrict__ pairs) {
  constexpr int kArr = K + 4, kAll = 2 * (kEntry + 2) * kArr;
  for (int i = threadIdx.x; i < kAll; i += blockDim.x) {
    const int r = i / (2 * kArr), comp = (i / kArr) & 1, k = i % kArr - 2;
    double v = 0.0;
    if (k >= 0 && k < K) {
      const double2 p = __ldg(pairs + r * K + k);
      v = comp && r < kEntry ? p.y : p.x;
    }
    out[i] = v;
  }
}

// The split form of a kernel's exponentiation: stages the constants of
// kSides moduli (cm, kConst doubles each) and runs split_power for this
// thread's value.  smem: the kernel's; group: the value's place in the CTA.
template <int KL, int kEntry, int kSides, bool kUnits>
__device__ __forceinline__ bool split_run(double* smem, const double* __restrict__ cm, int side, int group,
                                          const uint32_t* __restrict__ words, int nwords, uint64_t ninv52,
                                          const PairExponent& ex, const uint32_t* __restrict__ aux) {
  using Lay = PairLayout<KL, kSplit, kEntry, kSides>;
  constexpr int L = Lay::L, kConst = pair_const_doubles(KL, kEntry), kArr = KL + 4;
  double* vals = smem + 2 * kSides * Lay::kRows;
  double* tab = vals + 2 * Lay::kGroups * Lay::kSlot;
  double* work = tab + Lay::kTab;  // one array of zeros, then three per value
#pragma unroll 1
  for (int sd = 0; sd < kSides; ++sd)
    split_rows<KL, kEntry>(smem + sd * (2 * Lay::kRows),
                           reinterpret_cast<const double2*>(cm + sd * kConst + KL));
  for (int i = threadIdx.x; i < int(Lay::kWork); i += blockDim.x) work[i] = 0.0;
  __syncthreads();
  cm += side * kConst;
  const int gl = threadIdx.x & (Lay::kHalf - 1);
  double m[L];
#pragma unroll
  for (int k = 0; k < L; ++k) m[k] = __ldg(cm + gl * L + k);
  cuhe52::Split52<KL, Lay::kHalf> f(ninv52, m);
  return split_power<KL, Lay::kHalf, kEntry, kUnits>(
      f, words, nwords, smem + side * (2 * Lay::kRows), work,
      reinterpret_cast<const double2*>(cm + KL) + (kEntry + 2) * KL, work + kArr * (1 + 3 * group),
      reinterpret_cast<double2*>(vals) + group * Lay::kSlot, tab + threadIdx.x, m, ex, aux);
}

}  // namespace cuhe
