// The pair arithmetic of pair52.cuh spread for latency: one component per
// lane group.  Lanes [0, TPI) of a value hold component 0, lanes [TPI, 2 TPI)
// component 1, five limbs a lane, so a value takes four times the lanes of
// the ten-limb kernels and a lane forms half the limb products of the
// five-limb ones.  For batches that leave most of the GPU idle, where what
// counts is one product's serial chain.
//
// Both halves run the same instructions on their own operands.  Component 1's
// columns need component 0's quotients (z1 = (x0 y1 + x1 y0 - mu + mu' m) / R),
// so half 1 runs one step behind: its first step is an empty one (operand
// limbs 0, columns 0), half 0 sits the last one out, and half 0's quotients
// reach half 1 in the step that needs them.
//
// A step takes two limbs: the quotient of the two lowest columns V,
// Q = -V m^-1 mod 2^104, is formed at once on the integer pipe, which halves
// the broadcasts and FP64 latencies in the chain.
//
// What bounds it: the issue of one warp per scheduler, 211 instructions in
// 345 cycles a step (60 FP64 instructions of two slots, 97 integer adds and
// logic, 23 multiplies, 12 shuffles), beside a chain of about 300.  A step of
// the five-limb kernels, one limb of both components, takes 256 for the same
// 20 limb products per lane, so a value of 20 limbs needs 11 x 345 cycles a
// squaring against 20 x 256: one decode at key_len 1024 0.83 against 1.19 ms,
// 0.80 with the wider windows that its table has room for.
#pragma once
#include "pair52.cuh"

namespace cuhe52 {

template <int K, int TPI>
struct Split52 {
  static_assert(K % TPI == 0 && K % 2 == 0 && 2 * TPI <= 32, "limbs divide over lanes and steps");
  using Pair = Pair52<K, TPI>;
  static constexpr int L = K / TPI;
  static_assert(L >= 3 && TPI >= 2, "two columns leave a lane per step");
  // doubles of a published operand: two zero limbs (half 1's empty step), K
  // limbs, two that half 0 reads and drops in the last step
  static constexpr int kOperand = K + 4;

  Pair f;           // the half's lanes; limbs, columns and carries as there
  int half;         // component
  int from;         // lane of the value that across() reads
  uint64_t n0, n1;  // the inverse on lane 0 of each half, 0 elsewhere

  // ninv: -m^-1 mod 2^52; one Newton step over m's two low limbs doubles it
  __device__ __forceinline__ Split52(uint64_t ninv, const double (&m)[L]) {
    using u128 = unsigned __int128;
    half = (int(threadIdx.x & 31) / TPI) & 1;
    from = half ? f.gl : 1;
    const u128 low = static_cast<u128>(__double2ll_rn(m[0])) + (static_cast<u128>(__double2ll_rn(m[1])) << 52);
    const u128 inv = u128(0) - ninv, twice = u128(0) - inv * (2 - low * inv);
    n0 = f.gl == 0 ? ninv : 0ull;
    n1 = f.gl == 0 ? static_cast<uint64_t>(twice >> 52) & kMask : 0ull;
  }

  // Limbs 2i, 2i + 1 for half 0 and 2i - 2, 2i - 1 for half 1 of an operand
  // are at its pointer + 2i.
  __device__ __forceinline__ const double* operand(const double* arr) const { return half ? arr : arr + 2; }

  // One step.  X: the columns as between the steps there (plus
  // Pair::bias<nb>(k); a step adds two limbs' patterns to every position but
  // the lowest, which keeps that level, and position 1 stands one limb's
  // patterns below position 0 and receives one limb's more), with the limb
  // products of this step's operands added and those of the next, b and c,
  // formed while this step's quotients travel.  drop: half 0's quotients.
  template <bool kBoth, bool kLast>
  __device__ __forceinline__ void step(uint64_t (&E)[L + 2], const double (&a)[L], const double (&a2)[L], double2 b,
                                       double2 c, const double (&m)[L], uint64_t drop0, uint64_t drop1, uint64_t& q0,
                                       uint64_t& q1) const {
    constexpr int nb = kBoth ? 3 : 2;
    uint64_t X[L + 4];
#pragma unroll
    for (int k = 0; k < L + 2; ++k) X[k] = E[k];
    X[L + 2] = X[L + 3] = kLast ? 0ull : kTop<nb>();
    X[0] -= drop0;
    X[1] -= drop1;
    // on lane 0: column 0 (its debt of kOffC repaid) and column 1 without
    // the biases they hold before the quotient's products
    const uint64_t v0 = X[0] - (Pair::template bias<nb>(0) + Pair::kOffC + (nb - 1) * kPairLo);
    const uint64_t v1 = X[1] - (Pair::template bias<nb>(1) + (nb - 1) * (2 * kPairLo + kPairHi)) +
                        static_cast<uint64_t>(static_cast<int64_t>(v0) >> 52);
    const uint64_t w0 = v0 & kMask, low = w0 * n0;
    q0 = low & kMask;
    q1 = (((__umul64hi(w0, n0) << 12) | (low >> 52)) + w0 * n1 + v1 * n0) & kMask;
    const uint64_t mu0 = Pair::bcast(q0), mu1 = Pair::bcast(q1);
    if (!kLast) products<kBoth>(X, a, a2, b, c, 2);
    mac(X, m, Pair::to_f64(mu0), 0);
    mac(X, m, Pair::to_f64(mu1), 1);
    // columns 0 and 1 of every lane go to the lane below; lane 0's are exact
    // multiples of 2^52 and pass their carries up
    const uint64_t up0 = down(X[0]), up1 = down(X[1]);
    uint32_t c0, c1;
    asm("shr.u32 %0, %1, %2;" : "=r"(c0) : "r"(static_cast<uint32_t>(X[0] >> 32)), "r"(f.csh));
    const uint64_t second = X[1] + c0;
    asm("shr.u32 %0, %1, %2;" : "=r"(c1) : "r"(static_cast<uint32_t>(second >> 32)), "r"(f.csh));
#pragma unroll
    for (int k = 0; k < L + 2; ++k) E[k] = X[k + 2];
    E[0] += c1;
    E[L - 2] += up0;
    E[L - 1] += up1;
  }

  // what the shift takes from the columns that enter at the top
  template <int nb>
  static __device__ __forceinline__ constexpr uint64_t kTop() {
    return 0ull - static_cast<uint64_t>(L) * nb * kPairStep;
  }

  template <bool kBoth, int N>
  static __device__ __forceinline__ void products(uint64_t (&X)[N], const double (&a)[L], const double (&a2)[L],
                                                  double2 b, double2 c, int at) {
    mac(X, a, b.x, at);
    if (kBoth) mac(X, a2, c.x, at);
    mac(X, a, b.y, at + 1);
    if (kBoth) mac(X, a2, c.y, at + 1);
  }

  template <int N>
  static __device__ __forceinline__ void mac(uint64_t (&ext)[N], const double (&x)[L], double y, int at) {
    uint64_t ph = 0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
      uint64_t h, l;
      Pair::mul52(x[k], y, h, l);
      if (k == 0) ext[at] += l;
      else ext[k + at] += l + ph;
      ph = h;
    }
    ext[L + at] += ph;
  }

  __device__ __forceinline__ uint64_t down(uint64_t v) const {
    uint32_t lo = __shfl_down_sync(0xffffffffu, static_cast<uint32_t>(v), 1, TPI);
    uint32_t hi = __shfl_down_sync(0xffffffffu, static_cast<uint32_t>(v >> 32), 1, TPI);
    if (f.gl == TPI - 1) {  // an empty column
      lo = static_cast<uint32_t>(Pair::kOff - Pair::kOffC);
      hi = static_cast<uint32_t>((Pair::kOff - Pair::kOffC) >> 32);
    }
    return (static_cast<uint64_t>(hi) << 32) | lo;
  }

  // half 0's quotients for half 1 (0 on every lane but lane 0), 0 for half 0,
  // whose lane 1 always holds one of 0
  __device__ __forceinline__ uint64_t across(uint64_t q) const {
    const uint32_t lo = __shfl_sync(0xffffffffu, static_cast<uint32_t>(q), from, 2 * TPI);
    const uint32_t hi = __shfl_sync(0xffffffffu, static_cast<uint32_t>(q >> 32), from, 2 * TPI);
    return (static_cast<uint64_t>(hi) << 32) | lo;
  }

  // The product a b [+ a2 c] R^-1 of each half into raw accumulators (nb = 2,
  // 3 with kBoth), b and c published operands through operand().
  template <bool kBoth>
  __device__ __forceinline__ void product(uint64_t (&acc)[L], const double (&a)[L], const double (&a2)[L],
                                          const double* b, const double* c, const double (&m)[L]) const {
    constexpr int nb = kBoth ? 3 : 2;
    const double2* b2 = reinterpret_cast<const double2*>(b);
    const double2* c2 = reinterpret_cast<const double2*>(c);
    constexpr int kU = 2;  // steps per block: 9% faster than 1, 4 and 5 crowd the instruction cache
    const double2 none = make_double2(0.0, 0.0);
    f.template init<nb>(acc);
    uint64_t E[L + 2], drop0 = 0, drop1 = 0, q0, q1;
#pragma unroll
    for (int k = 0; k < L; ++k) E[k] = acc[k];
    E[L] = E[L + 1] = kTop<nb>();
    products<kBoth>(E, a, a2, b2[0], kBoth ? c2[0] : none, 0);
#pragma unroll kU
    for (int i = 1; i <= K / 2; ++i) {
      step<kBoth, false>(E, a, a2, b2[i], kBoth ? c2[i] : none, m, drop0, drop1, q0, q1);
      drop0 = across(q0);
      drop1 = across(q1);
    }
    // half 0 is done, but for the patterns of the products with the last
    // operand limbs, which are zeros
#pragma unroll
    for (int k = 0; k < L; ++k)
      acc[k] = E[k] - (nb - 1) * (k == 0 ? kPairLo : k == 1 ? 2 * kPairLo + kPairHi : 2 * kPairStep);
    step<kBoth, true>(E, a, a2, none, none, m, drop0, drop1, q0, q1);
#pragma unroll
    for (int k = 0; k < L; ++k) acc[k] = half ? E[k] : acc[k];
  }
};

}  // namespace cuhe52
