// Arithmetic mod m^2 (m odd) on pairs of residues mod m, on the FP64 pipe.
//
// A value mod m^2 is held as (x0, x1) = x0 + x1 m.  With R = 2^(52K) > m and
// Montgomery's quotient mu = -x0 y0 m^-1 mod R (so x0 y0 + mu m = z0 R),
//
//   (x0 + x1 m)(y0 + y1 m) R^-1  =  z0 + z1 m  (mod m^2),
//   z0 = (x0 y0 + mu m) / R,   z1 = (x0 y1 + x1 y0 - mu + mu' m) / R,
//
// mu' again chosen to make the division exact.  A product costs five K x K
// limb products and a squaring (x0 y1 + x1 y0 = x0 (2 x1)) four, where the
// Montgomery product of 2K-limb values mod m^2 costs eight: the quotient of
// the first reduction is what the second component needs, and nothing wider
// than m is ever multiplied.  R is at least 2^8 m.  Operands with components
// below 8 m (sums of up to four entry products, each below 2 m) give
// z0 < m + 64 m^2 / R and z1 < m + 128 m^2 / R, below 2 m again, so no product
// ends with a subtraction.
//
// Limbs are 52 bits and balanced (in [-2^51, 2^51] up to a carry of 2^10),
// held exactly as doubles.  The
// 104-bit product of two limbs is three FP64 instructions:
//
//   h = fma_rz(x, y, C)      C = 1.5 2^104: bits(h) = bits(C) + floor(xy / 2^52)
//   s = (C + 2^52) - h       exact
//   l = fma_rz(x, y, s)      bits(l) = bits(2^52) + (xy mod 2^52)
//
// for |xy| < 2^103 (the double-precision technique of Emmart, Zheng and
// Weems, ARITH 2018, with a centred constant for signed limbs).  The raw
// patterns are summed in 64-bit integer accumulators whose initial values
// cancel the biases, whose counts the schedule fixes.  Because limbs are
// balanced, each column's carry moves one place up and operands are in range;
// carries never ripple through the value.
//
// What bounds it: the dispatch of FP64 instructions (two issue slots each)
// and integer adds.  A limb product with its accumulation takes 10.2-11.4
// cycles per warp in isolation in every form tried (high halves chained
// through the FMA addend, low halves by integer multiplies, 46- and 49-bit
// limbs with FP64 accumulators) and 10.5 in a loop of whole squarings, so the
// gain over the 2K-limb product is the number of limb products: 2,210 M
// squarings mod a 2,048-bit m^2 a second, ten limbs a lane and two CTAs on
// every SM, against 980 M.
#pragma once
#include <cstdint>

namespace cuhe52 {

constexpr double kPairC = 30423614405477505635920876929024.0;    // 1.5 * 2^104
constexpr double kPairC52 = 30423614405477510139520504299520.0;  // 1.5 * 2^104 + 2^52
constexpr double kBalance = 6755399441055744.0;                  // 2^52 + 2^51
constexpr uint64_t kPairHi = 0x4678000000000000ull;              // bits of kPairC
constexpr uint64_t kPairLo = 0x4330000000000000ull;              // bits of 2^52
constexpr uint64_t kPairStep = kPairHi + kPairLo;

constexpr int kPairThreads = 128;

// K limbs per component over TPI consecutive lanes, lane g owning limbs
// [gL, gL + L).  Every lane of a warp takes part in every call (shuffles use
// the full mask), so groups of a warp follow one schedule.  U: steps per
// unrolled block; 2 keeps the product small in the instruction cache (65,536
// decodes at key_len 1024 with U = 1, 2, 4, 5, 10: 26.8, 25.7, 28.4, 28.4 and
// 31.2 ms).
template <int K, int TPI, int U = 2>
struct Pair52 {
  static_assert(K % TPI == 0 && K % U == 0, "limbs divide over lanes and blocks");
  static constexpr int L = K / TPI;
  // A leaving column passes its carry unsigned: kOff is added to it, and
  // kOff >> 52 is taken from every column in advance.
  static constexpr uint64_t kOff = 1ull << 60, kOffC = 1ull << 8;

  int gl;        // lane of the group
  uint32_t csh;  // carry shift: 20 on lane 0, 32 (no carry) elsewhere

  __device__ __forceinline__ Pair52() {
    gl = int(threadIdx.x & 31) & (TPI - 1);
    csh = gl == 0 ? 20u : 32u;
  }

  __device__ __forceinline__ static void mul52(double x, double y, uint64_t& hi, uint64_t& lo) {
    const double h = __fma_rz(x, y, kPairC);
    const double s = __dsub_rn(kPairC52, h);
    const double l = __fma_rz(x, y, s);
    hi = static_cast<uint64_t>(__double_as_longlong(h));
    lo = static_cast<uint64_t>(__double_as_longlong(l));
  }
  // an integer in [0, 2^52) as a double
  __device__ __forceinline__ static double to_f64(uint64_t v) {
    return __dsub_rn(__longlong_as_double(static_cast<long long>(v | kPairLo)), 4503599627370496.0);
  }
  __device__ __forceinline__ static uint64_t bcast(uint64_t v) {
    if (TPI == 1) return v;
    const uint32_t lo = __shfl_sync(0xffffffffu, static_cast<uint32_t>(v), 0, TPI);
    const uint32_t hi = __shfl_sync(0xffffffffu, static_cast<uint32_t>(v >> 32), 0, TPI);
    return (static_cast<uint64_t>(hi) << 32) | lo;
  }

  // Accumulator k of nb products per column and step holds its column plus
  // bias(k) before every step, on every lane: a step adds nb of both halves'
  // patterns (the low halves alone at position 0, whose column then leaves
  // the lane as column + kOff - kOffC), and the shift takes L steps' patterns
  // from the column that enters at the top.  Column 0 of the group alone has
  // no column below it and lacks the - kOffC.
  template <int nb>
  __device__ __forceinline__ static constexpr uint64_t bias(int k) {
    return kOff - kOffC - nb * kPairLo - static_cast<uint64_t>(k) * nb * kPairStep;
  }
  template <int nb>
  __device__ __forceinline__ void init(uint64_t (&acc)[L]) const {
#pragma unroll
    for (int k = 0; k < L; ++k) acc[k] = bias<nb>(k);
    if (TPI == 1 || gl == 0) acc[0] = bias<nb>(0) + kOffC;
  }

  // acc += a b, logical position k in register (k + s) % L; the top limb's
  // high half belongs to the next lane and waits in pend until the shift
  __device__ __forceinline__ static void mac(uint64_t (&acc)[L], uint64_t& pend, const double (&a)[L], double b, int s) {
    uint64_t ph = 0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
      uint64_t h, l;
      mul52(a[k], b, h, l);
      if (k == 0) acc[s % L] += l;
      else acc[(k + s) % L] += l + ph;
      ph = h;
    }
    pend += ph;
  }

  // Column 0 of the group leaves, every other column moves down one position.
  template <int nb>
  __device__ __forceinline__ void shift(uint64_t (&acc)[L], uint64_t pend, int s) const {
    constexpr uint64_t kTop = 0ull - static_cast<uint64_t>(L) * nb * kPairStep;
    const uint64_t a0 = acc[s % L];
    if (TPI == 1) {
      acc[s % L] = pend + (kOff - kOffC + kTop);
      acc[(s + 1) % L] += static_cast<uint32_t>(a0 >> 32) >> 20;
    } else {
      uint32_t lo = __shfl_down_sync(0xffffffffu, static_cast<uint32_t>(a0), 1, TPI);
      uint32_t hi = __shfl_down_sync(0xffffffffu, static_cast<uint32_t>(a0 >> 32), 1, TPI);
      if (gl == TPI - 1) {  // an empty column
        lo = static_cast<uint32_t>(kOff - kOffC);
        hi = static_cast<uint32_t>((kOff - kOffC) >> 32);
      }
      uint32_t c;  // shr clamps at 32: no carry from any lane but 0
      asm("shr.u32 %0, %1, %2;" : "=r"(c) : "r"(static_cast<uint32_t>(a0 >> 32)), "r"(csh));
      acc[s % L] = ((static_cast<uint64_t>(hi) << 32) | lo) + pend + kTop;
      acc[(s + 1) % L] += c;
    }
  }

  // the same for k >= 1, given the high half of k = 0
  __device__ __forceinline__ static void mac_rest(uint64_t (&acc)[L], uint64_t& pend, const double (&a)[L], double b,
                                                  uint64_t ph, int s) {
#pragma unroll
    for (int k = 1; k < L; ++k) {
      uint64_t h, l;
      mul52(a[k], b, h, l);
      acc[(k + s) % L] += l + ph;
      ph = h;
    }
    pend += ph;
  }

  // The K steps of a product: A0 = a0 b.x + mu m, A1 = a0 b.y [+ a1 b.x, with
  // kBoth] - mu + mu' m, b.x and b.y the limbs of one array of pairs.  A
  // squaring passes b = (x0, 2 x1) and kBoth = false.  ninv = -m^-1 mod 2^52
  // on lane 0, 0 elsewhere (which makes mu's subtraction lane 0's alone).
  // The pair past b's end is read and not used.
  //
  // A step's serial chain is column 0 -> quotient (integer product) ->
  // shuffle -> product with m -> the next column 0, about 190 cycles for each
  // component.  Column 0 of both is formed first, from limb products made
  // during the step before, so both quotients travel while the other columns'
  // products run; and squarings and products are separate loops, with no
  // branch inside a step (one loop with the quotients in turn runs 17% fewer
  // squarings a second, and one warp alone takes 1.6 times as long).
  template <bool kBoth>
  __device__ __forceinline__ void steps(uint64_t (&A0)[L], uint64_t (&A1)[L], const double (&a0)[L],
                                        const double (&a1)[L], const double2* b, const double (&m)[L],
                                        uint64_t ninv) const {
    double2 bi = b[0];
    uint64_t h0, l0, h1, l1, h2 = 0, l2 = 0;
    mul52(a0[0], bi.x, h0, l0);
    mul52(a0[0], bi.y, h1, l1);
    if (kBoth) mul52(a1[0], bi.x, h2, l2);
#pragma unroll 1
    for (int i0 = 0; i0 < K; i0 += U) {
#pragma unroll
      for (int s = 0; s < U; ++s) {
        const double2 bn = b[i0 + s + 1];
        uint64_t pend0 = 0, pend1 = 0;
        A0[s % L] += l0;
        A1[s % L] += l1;
        if (kBoth) A1[s % L] += l2;
        const uint64_t q0 = (A0[s % L] * ninv) & kMask;
        A1[s % L] -= q0;
        const uint64_t q1 = (A1[s % L] * ninv) & kMask;
        const uint64_t mu0 = bcast(q0);
        const uint64_t mu1 = bcast(q1);
        mac_rest(A0, pend0, a0, bi.x, h0, s);
        mac_rest(A1, pend1, a0, bi.y, h1, s);
        if (kBoth) mac_rest(A1, pend1, a1, bi.x, h2, s);
        bi = bn;
        mul52(a0[0], bi.x, h0, l0);
        mul52(a0[0], bi.y, h1, l1);
        if (kBoth) mul52(a1[0], bi.x, h2, l2);
        mac(A0, pend0, m, to_f64(mu0), s);
        mac(A1, pend1, m, to_f64(mu1), s);
        shift<2>(A0, pend0, s);
        shift<kBoth ? 3 : 2>(A1, pend1, s);
      }
      if (U % L) {  // back to logical order
        uint64_t t0[L], t1[L];
#pragma unroll
        for (int k = 0; k < L; ++k) {
          t0[k] = A0[(k + U) % L];
          t1[k] = A1[(k + U) % L];
        }
#pragma unroll
        for (int k = 0; k < L; ++k) {
          A0[k] = t0[k];
          A1[k] = t1[k];
        }
      }
    }
  }

  // The whole product (arguments as for steps) into raw accumulators: A0 of 2
  // and A1 of 2 (3 with kBoth) products per column and step.
  template <bool kBoth>
  __device__ __forceinline__ void product(uint64_t (&A0)[L], uint64_t (&A1)[L], const double (&a0)[L],
                                          const double (&a1)[L], const double2* b, const double (&m)[L],
                                          uint64_t ninv) const {
    init<2>(A0);
    init<kBoth ? 3 : 2>(A1);
    steps<kBoth>(A0, A1, a0, a1, b, m, ninv);
  }

  // minus bias(k), and plus kOffC's repayment at the group's position 0
  template <int nb>
  __device__ __forceinline__ uint64_t column(const uint64_t (&acc)[L], int k, int times, uint64_t lift) const {
    uint64_t v = acc[k];
    if (times == 2) v += v;
    const uint64_t plain = lift - times * bias<nb>(k), first = plain - times * kOffC;
    return v + (k == 0 ? (TPI == 1 || gl == 0 ? first : plain) : plain);
  }
  template <int nb>
  __device__ __forceinline__ void columns(uint64_t (&acc)[L]) const {
#pragma unroll
    for (int k = 0; k < L; ++k) acc[k] = column<nb>(acc, k, 1, 0);
  }

  // Columns plus kLift to balanced limbs.  Every column's carry goes one
  // place up and no further: a limb then lies in [-2^51 - 2^10, 2^51 + 2^10],
  // which the products take, and nothing waits for a neighbour's carry (the
  // value itself is nonnegative and below R / 2).
  static constexpr uint64_t kLift = (1ull << 51) + (1ull << 61);
  __device__ __forceinline__ void split(double (&r)[L], const uint64_t (&t)[L]) const {
    uint32_t c[L];  // carry + 2^9
#pragma unroll
    for (int k = 0; k < L; ++k) c[k] = static_cast<uint32_t>(t[k] >> 32) >> 20;
    uint32_t in = 1u << 9;
    if (TPI > 1) {
      in = __shfl_up_sync(0xffffffffu, c[L - 1], 1, TPI);
      if (gl == 0) in = 1u << 9;
    }
#pragma unroll
    for (int k = 0; k < L; ++k) {
      // carry - 2^52 - 2^51, then + 2^52 + the column's low 52 bits
      const double g = __dsub_rn(__hiloint2double(0x43380000, static_cast<int>(k == 0 ? in : c[k - 1])),
                                 2.0 * kBalance + 512.0);
      r[k] = __dadd_rn(__longlong_as_double(static_cast<long long>((t[k] & kMask) | kPairLo)), g);
    }
  }
  // balanced limbs of an accumulator, of twice an accumulator, of columns
  template <int nb>
  __device__ __forceinline__ void limbs(double (&r)[L], const uint64_t (&acc)[L]) const {
    uint64_t t[L];
#pragma unroll
    for (int k = 0; k < L; ++k) t[k] = column<nb>(acc, k, 1, kLift);
    split(r, t);
  }
  template <int nb>
  __device__ __forceinline__ void twice(double (&r)[L], const uint64_t (&acc)[L]) const {
    uint64_t t[L];
#pragma unroll
    for (int k = 0; k < L; ++k) t[k] = column<nb>(acc, k, 2, kLift);
    split(r, t);
  }
  __device__ __forceinline__ void from_columns(double (&r)[L], const uint64_t (&v)[L]) const {
    uint64_t t[L];
#pragma unroll
    for (int k = 0; k < L; ++k) t[k] = v[k] + kLift;
    split(r, t);
  }
  // twice a value given as limbs
  __device__ __forceinline__ void twice_limbs(double (&r)[L], const double (&x)[L]) const {
    uint64_t t[L];
#pragma unroll
    for (int k = 0; k < L; ++k) t[k] = 2 * static_cast<uint64_t>(__double2ll_rn(x[k])) + kLift;
    split(r, t);
  }

  // Columns to canonical limbs in [0, 2^52) (carries rippled through the
  // group; the value is nonnegative and below R).
  __device__ __forceinline__ void canonical(uint64_t (&v)[L]) const {
    int64_t carry = 0;
#pragma unroll
    for (int k = 0; k < L; ++k) {
      const int64_t t = static_cast<int64_t>(v[k]) + carry;
      carry = t >> 52;
      v[k] = static_cast<uint64_t>(t) & kMask;
    }
    if constexpr (TPI > 1) {
      for (int guard = 0; guard < TPI; ++guard) {
        int c = __shfl_up_sync(0xffffffffu, static_cast<int>(carry), 1, TPI);
        if (gl == 0) c = 0;
        carry = c;
#pragma unroll
        for (int k = 0; k < L; ++k) {
          const int64_t t = static_cast<int64_t>(v[k]) + carry;
          carry = t >> 52;
          v[k] = static_cast<uint64_t>(t) & kMask;
        }
        if (!__any_sync(0xffffffffu, gl != TPI - 1 && carry != 0)) break;
      }
    }
  }
};

}  // namespace cuhe52
