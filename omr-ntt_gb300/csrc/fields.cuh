// fields.cuh -- prime-field arithmetic for the GB300 NTT engine (host + device).
//
// The four fields of the reference crate (src/fields.rs:4-17):
//   BabyBear   p = 2^31 - 2^27 + 1, generator 31, 2-adicity 27
//   KoalaBear  p = 2^31 - 2^24 + 1, generator 3,  2-adicity 24
//   TeddyBear  p = 2^32 - 2^30 + 1, generator 5,  2-adicity 30
//   Goldilocks p = 2^64 - 2^32 + 1, generator 7,  2-adicity 32
//
// Elements cross every boundary in canonical form ([0, p)), one u32 word (the
// 32-bit fields) or one u64 word (Goldilocks).  Inside the kernels:
//   * 31-bit fields (BabyBear, KoalaBear): data stays canonical; a multiply by
//     a precomputed twiddle is Shoup's method (w, w' = floor(w 2^32 / p)), three
//     integer multiplies plus one conditional subtract; a product of two
//     runtime values uses Montgomery reduction with one operand in Montgomery
//     form (x*2^32 mod p).
//   * TeddyBear (p > 2^31): Montgomery only (no 1-bit headroom for Shoup's
//     [0, 2p) intermediate), with carry checks on add/sub.
//   * Goldilocks: 64x64->128 product and the 2^64 = 2^32 - 1, 2^96 = -1 (mod p)
//     folding; twiddles are plain canonical words.  Between its first load and
//     its last store a transform's words are any u64 congruent to the value.
// Roots of unity follow ark-ff's convention used by NttDomain::new
// (src/encoder.rs:34): omega_N = GEN^((p - 1) / N) for N a power of two.
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define OMR_HD __host__ __device__ __forceinline__
#define OMR_D __device__ __forceinline__
#else
#define OMR_HD inline
#define OMR_D inline
#endif

namespace omr {

enum FieldId : int { BABYBEAR = 0, GOLDILOCKS = 1, KOALABEAR = 2, TEDDYBEAR = 3 };

// ---------------------------------------------------------------- host helpers
// Exact modular arithmetic for table construction (host side, constexpr).
constexpr uint64_t hmulmod(uint64_t a, uint64_t b, uint64_t p) {
  return (uint64_t)(((unsigned __int128)a * b) % p);
}
constexpr uint64_t hpowmod(uint64_t b, uint64_t e, uint64_t p) {
  uint64_t r = 1 % p;
  b %= p;
  while (e) {
    if (e & 1) r = hmulmod(r, b, p);
    b = hmulmod(b, b, p);
    e >>= 1;
  }
  return r;
}
constexpr uint32_t inv_mod_2_32(uint32_t p) {  // p odd; Newton iteration
  uint32_t x = p;                              // correct to 3 bits
  for (int i = 0; i < 5; i++) x *= 2u - p * x;
  return x;
}

// ---------------------------------------------------------------- 32-bit fields
template <uint32_t P_, uint32_t GEN_, int TA_, int ID_>
struct Field32 {
  using E = uint32_t;
  static constexpr int ID = ID_;
  static constexpr uint32_t P = P_;
  static constexpr uint32_t GEN = GEN_;
  static constexpr int TWO_ADICITY = TA_;
  static constexpr bool SMALL = P_ < 0x80000000u;  // 1 bit of headroom: Shoup + min tricks
  static constexpr uint32_t PINV = inv_mod_2_32(P_);  // p^-1 mod 2^32
  static constexpr int WORD = 4;

  // Twiddle operand as stored in device tables.
  struct Tw {
    uint32_t w;   // SMALL: canonical w ; otherwise w * 2^32 mod p (Montgomery form)
    uint32_t wq;  // SMALL: floor(w * 2^32 / p) ; otherwise unused
  };

  static constexpr uint64_t p64() { return P_; }

  // host: build the twiddle operand for a canonical constant
  static constexpr Tw make_tw(uint64_t w) {
    return SMALL ? Tw{(uint32_t)w, (uint32_t)((w << 32) / P_)}
                 : Tw{(uint32_t)((w << 32) % P_), 0u};
  }
  static constexpr uint32_t to_mont_host(uint64_t w) { return (uint32_t)((w << 32) % P_); }

#if defined(__CUDACC__)
  // s in [0, 2p) -> [0, p): the smaller of s and s - p (mod 2^32), as one
  // fused add-min (a plain min of two sums compiles to two instructions)
  OMR_D static E reduce_once(E s) { return __viaddmin_u32(s, 0u - P, s); }
  OMR_D static E add(E a, E b) {
    if constexpr (SMALL) {
      return reduce_once(a + b);
    } else {
      E s = a + b;
      return (s < a || s >= P) ? s - P : s;
    }
  }
  OMR_D static E sub(E a, E b) {
    if constexpr (SMALL) {
      const E d = a - b;  // a borrow leaves d > 2^32 - p, so d + p wraps below it
      return __viaddmin_u32(d, P, d);
    } else {
      E d = a - b;
      return a < b ? d + P : d;
    }
  }
  // a (canonical or any u32 for Montgomery) times b in Montgomery form -> canonical a*b
  OMR_D static E mont(E a, E bm) {
    uint32_t lo = a * bm;
    uint32_t hi = __umulhi(a, bm);
    uint32_t m = lo * PINV;
    uint32_t mh = __umulhi(m, P);
    uint32_t r = hi - mh;
    return hi < mh ? r + P : r;
  }
  // a * twiddle -> canonical
  OMR_D static E mul_tw(E a, Tw t) {
    if constexpr (SMALL) {
      uint32_t q = __umulhi(a, t.wq);
      return reduce_once(a * t.w - q * P);  // in [0, 2p)
    } else {
      return mont(a, t.w);
    }
  }
  // runtime twiddle product: both operands in "twiddle-Montgomery" form, result too.
  // (used for on-the-fly twiddle generation; for SMALL fields the Montgomery
  //  form is kept in Tw.w only by the generator helpers below)
  OMR_D static E mont_mul(E am, E bm) { return mont(am, bm); }
  // a t + b (Horner step); words are canonical already
  OMR_D static E mul_add(E a, Tw t, E b) { return add(mul_tw(a, t), b); }
  OMR_D static E canon(E a) { return a; }
#endif
};

using BabyBear = Field32<0x78000001u, 31u, 27, BABYBEAR>;
using KoalaBear = Field32<0x7f000001u, 3u, 24, KOALABEAR>;
using TeddyBear = Field32<0xc0000001u, 5u, 30, TEDDYBEAR>;

// ---------------------------------------------------------------- Goldilocks
// x0 + x1 2^32 + x2 2^64 with a small signed x2: an unreduced value
// (dft_goldilocks.cuh)
struct GlWide {
  uint32_t x0, x1, x2;
};

struct Goldilocks {
  using E = uint64_t;
  static constexpr int ID = GOLDILOCKS;
  static constexpr uint64_t P = 0xffffffff00000001ull;
  static constexpr uint64_t GEN = 7;
  static constexpr int TWO_ADICITY = 32;
  static constexpr bool SMALL = false;
  static constexpr int WORD = 8;
  struct Tw {
    uint64_t w;
  };
  static constexpr uint64_t p64() { return P; }
  static constexpr Tw make_tw(uint64_t w) { return Tw{w}; }

#if defined(__CUDACC__)
  // Inside a transform a word is any u64 congruent to its value ("lazy"):
  // products, DFT inputs and DFT outputs.  canon() brings it into [0, p) when
  // the last pass writes its results.  add and sub take and give canonical
  // words (sums of inputs).
  OMR_D static uint64_t pack(uint32_t lo, uint32_t hi) { return ((uint64_t)hi << 32) | lo; }
  // a - b (mod p), canonical: a borrow becomes the mask 0xffffffff, which is
  // 2^64 - p in the low word
  OMR_D static E sub(E a, E b) {
    uint32_t r0, r1;
    asm("{.reg .u32 m;\n\t"
        "sub.cc.u32 %0, %2, %4;\n\t"
        "subc.cc.u32 %1, %3, %5;\n\t"
        "subc.u32 m, 0, 0;\n\t"       // borrow mask
        "sub.cc.u32 %0, %0, m;\n\t"   // - (2^32 - 1) on borrow (= + p)
        "subc.u32 %1, %1, 0;}"
        : "=&r"(r0), "=&r"(r1)
        : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"((uint32_t)b), "r"((uint32_t)(b >> 32)));
    return pack(r0, r1);
  }
  // a + b = a - (p - b): one borrow-corrected subtraction
  OMR_D static E add(E a, E b) { return sub(a, P - b); }
  // any u64 -> [0, p): a + 2^32 - 1 carries iff a >= p, and is then a - p
  OMR_D static E canon(E a) {
    uint32_t r0, r1;
    asm("{.reg .u32 x, m;\n\t"
        "add.cc.u32 x, %2, 0xffffffff;\n\t"
        "addc.cc.u32 x, %3, 0;\n\t"
        "addc.u32 m, 0, 0;\n\t"
        "mad.lo.cc.u32 %0, m, 0xffffffff, %2;\n\t"
        "addc.u32 %1, %3, 0;}"
        : "=&r"(r0), "=&r"(r1)
        : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)));
    return pack(r0, r1);
  }
  // lo + 2^64 hi reduced to three limbs with 2^64 = 2^32 - 1 and 2^96 = -1:
  // lo + h0 (2^32 - 1) - h1, in (-2^32, 2^65).  h0 (2^32 - 1) is one
  // 32 x 32 -> 64 multiply-add (mad.lo/hi with carry).  A flag is read only by
  // the instruction family that set it (addc after additions, subc after
  // subtractions): a subtraction's borrow and an addition's carry are not
  // interchangeable in the compiled code.
  OMR_D static GlWide reduce3(uint64_t lo, uint64_t hi) {
    GlWide r;
    asm("{.reg .u32 t0, t1, c;\n\t"
        "mad.lo.cc.u32 t0, %5, 0xffffffff, %3;\n\t"
        "madc.hi.cc.u32 t1, %5, 0xffffffff, %4;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "sub.cc.u32 %0, t0, %6;\n\t"
        "subc.cc.u32 %1, t1, 0;\n\t"
        "subc.u32 %2, c, 0;}"
        : "=&r"(r.x0), "=&r"(r.x1), "=r"(r.x2)
        : "r"((uint32_t)lo), "r"((uint32_t)(lo >> 32)), "r"((uint32_t)hi), "r"((uint32_t)(hi >> 32)));
    return r;
  }
  // reduce3's result as one word: x2 is -1, 0 or 1, and lo + x2 (2^32 - 1)
  // neither borrows nor carries (x2 = -1 only with lo >= 2^64 - 2^32, x2 = 1
  // only with lo < 2^64 - 2^33)
  OMR_D static E fold_small(GlWide x) {
    uint32_t r0, r1;
    asm("{.reg .u32 s;\n\t"
        "shr.s32 s, %4, 31;\n\t"
        "sub.cc.u32 %0, %2, %4;\n\t"
        "subc.u32 %1, %3, s;\n\t"
        "add.u32 %1, %1, %4;}"
        : "=&r"(r0), "=&r"(r1)
        : "r"(x.x0), "r"(x.x1), "r"(x.x2));
    return pack(r0, r1);
  }
  // products of any two u64.  The 128-bit product through the compiler's own
  // 64-bit multiplies: 20 clocks a warp and scheduler on GB300 against 23 for a
  // mad.lo/hi.cc chain; the whole product with this reduction 30 against 47
  // for one that reduced to a canonical word.
  OMR_D static GlWide mul3(E a, E b) { return reduce3(a * b, __umul64hi(a, b)); }
  OMR_D static E mul(E a, E b) { return fold_small(mul3(a, b)); }
  OMR_D static E mul_tw(E a, Tw t) { return mul(a, t.w); }
  OMR_D static E mont_mul(E a, E b) { return mul(a, b); }
  // a t + b (Horner step), any u64: a t + b < 2^128
  OMR_D static E mul_add(E a, Tw t, E b) {
    const uint64_t lo = a * t.w, s = lo + b;
    return fold_small(reduce3(s, __umul64hi(a, t.w) + (s < lo ? 1u : 0u)));
  }
#endif
};

// Host-side root of unity (ark convention): omega_N = GEN^((p-1)/N).
template <class F>
constexpr uint64_t root_of_unity_host(int log_n) {
  return hpowmod(F::GEN, (F::p64() - 1) >> log_n, F::p64());
}

}  // namespace omr
