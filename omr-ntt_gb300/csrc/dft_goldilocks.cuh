// dft_goldilocks.cuh -- in-register R-point DFTs (R = 2, 4, 8, 16) over
// Goldilocks on three-limb values.
//
// On canonical words the Goldilocks passes are bound by the integer ALU pipe,
// where a 64-bit modular add costs seven instructions and a subtract five: the
// borrow or carry of every butterfly is folded back at once.  With this DFT the
// ALU and the multiply pipe are equally busy.  A value of the DFT
// is x0 + x1 2^32 + x2 2^64 with a small signed x2, so an add or subtract is
// three instructions (one carry chain, no fold), and the fold 2^64 = 2^32 - 1
// happens once per output.  The roots are powers of two (omega_16 = -2^60),
// and p divides 2^96 + 1, so a twiddle is a shift by s < 32 bits and a
// rotation of whole limbs with 2^96 = -1; the sign is carried at compile time
// and turns the next add into a subtract.  A 16-point DFT is 4 x 4 radix-4
// butterflies: 41 clocks a warp element and scheduler on GB300, against 67.6
// for radix-2 butterflies on canonical words (44.6 with every limb term and
// fold as a wide multiply-add).
//
// Bounds, in units of 2^64 (eps = 2^-32): inputs lie in (-eps, 2) (64-bit
// words, or unreduced products, Goldilocks::mul3).  The a input of a radix-4
// butterfly is biased by a multiple C p of the modulus, so that
//   * the outputs that are shifted are non-negative and below 16
//     (|a - c| < 2, -eps < I (b - d) < 2, |(a + c) - (b + d)| < 4: C = 5 gives
//     values in (0, 13); a shift by s <= 28 bits then fits three limbs);
//   * the results are non-negative and below 2^7 (kBiasOut), as the unsigned
//     final fold needs: shifted values lie in (-1 - eps, 2), the unshifted
//     ones of the first layer in (0, 13).
#pragma once
#include "fields.cuh"

namespace omr {

#if defined(__CUDACC__)

OMR_D GlWide gl_wide(uint64_t x) { return GlWide{(uint32_t)x, (uint32_t)(x >> 32), 0u}; }

OMR_D GlWide gl_add3(GlWide a, GlWide b) {
  GlWide r;
  asm("add.cc.u32 %0, %3, %6;\n\t"
      "addc.cc.u32 %1, %4, %7;\n\t"
      "addc.u32 %2, %5, %8;"
      : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
      : "r"(a.x0), "r"(a.x1), "r"(a.x2), "r"(b.x0), "r"(b.x1), "r"(b.x2));
  return r;
}
OMR_D GlWide gl_sub3(GlWide a, GlWide b) {
  GlWide r;
  asm("sub.cc.u32 %0, %3, %6;\n\t"
      "subc.cc.u32 %1, %4, %7;\n\t"
      "subc.u32 %2, %5, %8;"
      : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
      : "r"(a.x0), "r"(a.x1), "r"(a.x2), "r"(b.x0), "r"(b.x1), "r"(b.x2));
  return r;
}
// a + s b for a compile-time sign s
template <bool NEG>
OMR_D GlWide gl_acc3(GlWide a, GlWide b) {
  if constexpr (NEG)
    return gl_sub3(a, b);
  else
    return gl_add3(a, b);
}
// a + C p, C p = C 2^64 - C 2^32 + C
template <uint32_t C>
OMR_D GlWide gl_bias(GlWide a) {
  return gl_add3(a, GlWide{C, 0u - C, C - 1u});
}

// (x - K 2^64) 2^S for 0 <= x < 2^(96 - S mod 32), 0 < S < 96 (K = 0 unless q = 1).
// K is a bias of the caller's that kept x non-negative; it comes off as a
// constant of the chain.  The limb terms are added up, not multiplied by
// 2^32 - 1, where that takes no more than one add above the multiply: the
// multiply pipe (a wide multiply holds it four clocks) is the busier one.
template <int S, uint32_t K>
OMR_D GlWide gl_shift3(GlWide x) {
  static_assert(S > 0 && S < 96 && (S / 32 == 1 || K == 0), "shift out of range");
  constexpr int q = S / 32, s = S % 32;
  uint32_t y0 = x.x0, y1 = x.x1, y2 = x.x2;
  if constexpr (s != 0) {
    y2 = __funnelshift_l(x.x1, x.x2, s);
    y1 = __funnelshift_l(x.x0, x.x1, s);
    y0 = x.x0 << s;
  }
  GlWide r;
  if constexpr (q == 0) {
    // y0 + y1 2^32 + y2 (2^32 - 1)
    asm("mad.lo.cc.u32 %0, %5, 0xffffffff, %3;\n\t"
        "madc.hi.cc.u32 %1, %5, 0xffffffff, %4;\n\t"
        "addc.u32 %2, 0, 0;"
        : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
        : "r"(y0), "r"(y1), "r"(y2));
  } else if constexpr (q == 1) {
    // (y0 + y1) 2^32 - (y1 + y2), and - K 2^(96 + s) = + K 2^s
    asm("{.reg .u32 a0, a1, b0, b1;\n\t"
        "add.cc.u32 a0, %3, %4;\n\t"
        "addc.u32 a1, 0, 0;\n\t"
        "add.cc.u32 b0, %4, %5;\n\t"
        "addc.u32 b1, 0, 0;\n\t"
        "sub.cc.u32 %0, %6, b0;\n\t"
        "subc.cc.u32 %1, a0, b1;\n\t"
        "subc.u32 %2, a1, 0;}"
        : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
        : "r"(y0), "r"(y1), "r"(y2), "r"(K << s));
  } else {
    // y0 2^32 - (y0 + y1 + y2 2^32)
    asm("{.reg .u32 b0, b1;\n\t"
        "add.cc.u32 b0, %3, %4;\n\t"
        "addc.u32 b1, %5, 0;\n\t"
        "sub.cc.u32 %0, 0, b0;\n\t"
        "subc.cc.u32 %1, %3, b1;\n\t"
        "subc.u32 %2, 0, 0;}"
        : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
        : "r"(y0), "r"(y1), "r"(y2));
  }
  return r;
}

// x (non-negative, x2 < 2^8) as a 64-bit word congruent mod p (any u64)
OMR_D uint64_t gl_fold(GlWide x) {
  // a carry c leaves a remainder below 2^40, so + c (2^32 - 1) cannot carry again
  uint32_t r0, r1;
  asm("{.reg .u32 t0, t1, c;\n\t"
      "mad.lo.cc.u32 t0, %4, 0xffffffff, %2;\n\t"
      "madc.hi.cc.u32 t1, %4, 0xffffffff, %3;\n\t"
      "addc.u32 c, 0, 0;\n\t"
      "sub.cc.u32 %0, t0, c;\n\t"
      "subc.u32 t1, t1, 0;\n\t"
      "add.u32 %1, t1, c;}"
      : "=&r"(r0), "=&r"(r1)
      : "r"(x.x0), "r"(x.x1), "r"(x.x2));
  return Goldilocks::pack(r0, r1);
}

// One radix-4 butterfly: a + b + c + d, a + I b - c - I d, ..., I = omega_4
// (2^48 forward, -2^48 inverse); b, c, d carry compile-time signs.
constexpr uint32_t kGlBiasMid = 5, kGlBiasOut = 28, kGlBiasI = 16;
template <bool INV, bool NB, bool NC, bool ND>
OMR_D void gl_radix4(GlWide a, GlWide b, GlWide c, GlWide d, GlWide& y0, GlWide& y1, GlWide& y2, GlWide& y3) {
  const GlWide s0 = gl_acc3<NC>(a, c), d0 = gl_acc3<!NC>(a, c);
  // s1 = |b + d|, d1 = |b - d| up to the sign of b
  const GlWide s1 = gl_acc3<NB != ND>(b, d);
  GlWide bb = b;
  bb.x2 += kGlBiasI;
  const GlWide d1 = gl_acc3<NB == ND>(bb, d);
  const GlWide i1 = gl_shift3<48, kGlBiasI>(d1);
  y0 = gl_acc3<NB>(s0, s1);
  y2 = gl_acc3<!NB>(s0, s1);
  y1 = gl_acc3<NB != INV>(d0, i1);
  y3 = gl_acc3<NB == INV>(d0, i1);
}

// exponent of omega_R^k as a power of two (mod 192)
constexpr int gl_root_pow(int logr, int k, bool inv) {
  const int e = (39 * (64 >> logr) * k) % 192;
  return inv ? (192 - e) % 192 : e;
}
template <int E>
OMR_D GlWide gl_twiddle3(GlWide x) {  // |omega|: the sign (E >= 96) is the caller's
  constexpr int S = E % 96;
  if constexpr (S == 0)
    return x;
  else
    return gl_shift3<S, 0>(x);
}

// In place, natural order in and out; results any u64 after gl_fold.
template <int LOGR, bool INV>
OMR_D void gl_dft3(GlWide (&v)[1 << LOGR]) {
  static_assert(LOGR >= 1 && LOGR <= 4, "2..16 points");
  if constexpr (LOGR == 1) {
    const GlWide a = gl_bias<kGlBiasMid>(v[0]), b = v[1];
    v[0] = gl_add3(a, b);
    v[1] = gl_sub3(a, b);
  } else if constexpr (LOGR == 2) {
    gl_radix4<INV, false, false, false>(gl_bias<kGlBiasMid>(v[0]), v[1], v[2], v[3], v[0], v[1], v[2], v[3]);
  } else if constexpr (LOGR == 3) {
    GlWide a[4], b[4];
    gl_radix4<INV, false, false, false>(gl_bias<kGlBiasOut>(v[0]), v[2], v[4], v[6], a[0], a[1], a[2], a[3]);
    gl_radix4<INV, false, false, false>(gl_bias<kGlBiasMid>(v[1]), v[3], v[5], v[7], b[0], b[1], b[2], b[3]);
    constexpr int E1 = gl_root_pow(3, 1, INV), E2 = gl_root_pow(3, 2, INV), E3 = gl_root_pow(3, 3, INV);
    b[1] = gl_twiddle3<E1>(b[1]);
    b[2] = gl_twiddle3<E2>(b[2]);
    b[3] = gl_twiddle3<E3>(b[3]);
    v[0] = gl_add3(a[0], b[0]);
    v[4] = gl_sub3(a[0], b[0]);
    v[1] = gl_acc3<(E1 >= 96)>(a[1], b[1]);
    v[5] = gl_acc3<(E1 < 96)>(a[1], b[1]);
    v[2] = gl_acc3<(E2 >= 96)>(a[2], b[2]);
    v[6] = gl_acc3<(E2 < 96)>(a[2], b[2]);
    v[3] = gl_acc3<(E3 >= 96)>(a[3], b[3]);
    v[7] = gl_acc3<(E3 < 96)>(a[3], b[3]);
  } else {
    GlWide u[4][4];  // u[j][k]
    gl_radix4<INV, false, false, false>(gl_bias<kGlBiasOut>(v[0]), v[4], v[8], v[12], u[0][0], u[0][1], u[0][2],
                                        u[0][3]);
    gl_radix4<INV, false, false, false>(gl_bias<kGlBiasMid>(v[1]), v[5], v[9], v[13], u[1][0], u[1][1], u[1][2],
                                        u[1][3]);
    gl_radix4<INV, false, false, false>(gl_bias<kGlBiasMid>(v[2]), v[6], v[10], v[14], u[2][0], u[2][1], u[2][2],
                                        u[2][3]);
    gl_radix4<INV, false, false, false>(gl_bias<kGlBiasMid>(v[3]), v[7], v[11], v[15], u[3][0], u[3][1], u[3][2],
                                        u[3][3]);
    constexpr int E1 = gl_root_pow(4, 1, INV), E2 = gl_root_pow(4, 2, INV), E3 = gl_root_pow(4, 3, INV),
                  E4 = gl_root_pow(4, 4, INV), E6 = gl_root_pow(4, 6, INV), E9 = gl_root_pow(4, 9, INV);
    u[1][1] = gl_twiddle3<E1>(u[1][1]);
    u[2][1] = gl_twiddle3<E2>(u[2][1]);
    u[3][1] = gl_twiddle3<E3>(u[3][1]);
    u[1][2] = gl_twiddle3<E2>(u[1][2]);
    u[2][2] = gl_twiddle3<E4>(u[2][2]);
    u[3][2] = gl_twiddle3<E6>(u[3][2]);
    u[1][3] = gl_twiddle3<E3>(u[1][3]);
    u[2][3] = gl_twiddle3<E6>(u[2][3]);
    u[3][3] = gl_twiddle3<E9>(u[3][3]);
    gl_radix4<INV, false, false, false>(u[0][0], u[1][0], u[2][0], u[3][0], v[0], v[4], v[8], v[12]);
    gl_radix4<INV, (E1 >= 96), (E2 >= 96), (E3 >= 96)>(u[0][1], u[1][1], u[2][1], u[3][1], v[1], v[5], v[9], v[13]);
    gl_radix4<INV, (E2 >= 96), (E4 >= 96), (E6 >= 96)>(u[0][2], u[1][2], u[2][2], u[3][2], v[2], v[6], v[10], v[14]);
    gl_radix4<INV, (E3 >= 96), (E6 >= 96), (E9 >= 96)>(u[0][3], u[1][3], u[2][3], u[3][3], v[3], v[7], v[11], v[15]);
  }
}

#endif  // __CUDACC__

}  // namespace omr
