// BN254 Fr / Fq arithmetic for sm_103a: 8 x 32-bit little-endian limbs in
// Montgomery form with R = 2^256, byte-identical to the reference's in-memory
// 4 x 64-bit representation (crates/field/src/lib.rs:30-36, 321), so a
// caller's `&[Fr]` crosses the C ABI with no conversion.
//
// The multiply is bound by the integer multiply pipe: 136 partial products of
// 32x32->64 bits, each one wide multiply-add with carry, which the pipe takes
// at half the rate of a 32-bit one (measured on a GB300: 31 of 64 lanes a
// clock and SM; a wide multiply-add into a 64-bit sum without carries, the
// form limbs of 29 bits allow, 20, and 81 + 81 of those in nine limbs 48 G
// products/s). So a row's products are laid out as two carry chains of four
// (fe_mul below): 72 G products/s against 50 for rows of 64-bit sums with the
// carry added by separate instructions, 0.98 of what the pipe's rate allows,
// and 847 against 1187 clocks for one product alone.
#pragma once
#include <cstdint>

namespace apg {

struct FrConsts {
  static constexpr uint32_t P0 = 0xf0000001u, P1 = 0x43e1f593u, P2 = 0x79b97091u, P3 = 0x2833e848u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t INV = 0xefffffffu;  // -p^-1 mod 2^32
  __host__ __device__ static constexpr uint32_t R(int i) {
    return (const uint32_t[8]){0x4ffffffbu, 0xac96341cu, 0x9f60cd29u, 0x36fc7695u,
                               0x7879462eu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u}[i];
  }
  __host__ __device__ static constexpr uint32_t R2(int i) {
    return (const uint32_t[8]){0xae216da7u, 0x1bb8e645u, 0xe35c59e3u, 0x53fe3ab1u,
                               0x53bb8085u, 0x8c49833du, 0x7f4e44a5u, 0x0216d0b1u}[i];
  }
};

struct FqConsts {
  static constexpr uint32_t P0 = 0xd87cfd47u, P1 = 0x3c208c16u, P2 = 0x6871ca8du, P3 = 0x97816a91u,
                            P4 = 0x8181585du, P5 = 0xb85045b6u, P6 = 0xe131a029u, P7 = 0x30644e72u;
  static constexpr uint32_t INV = 0xe4866389u;  // -q^-1 mod 2^32
  __host__ __device__ static constexpr uint32_t R(int i) {
    return (const uint32_t[8]){0xc58f0d9du, 0xd35d438du, 0xf5c70b3du, 0x0a78eb28u,
                               0x7879462cu, 0x666ea36fu, 0x9a07df2fu, 0x0e0a77c1u}[i];
  }
  __host__ __device__ static constexpr uint32_t R2(int i) {
    return (const uint32_t[8]){0x538afa89u, 0xf32cfc5bu, 0xd44501fbu, 0xb5e71911u,
                               0x0a417ff6u, 0x47ab1effu, 0xcab8351fu, 0x06d89f71u}[i];
  }
};

template <class C>
struct Fe {
  uint32_t v[8];
};

typedef Fe<FrConsts> Fr;
typedef Fe<FqConsts> Fq;

template <class C>
__host__ __device__ __forceinline__ Fe<C> fe_zero() {
  Fe<C> r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = 0;
  return r;
}

template <class C>
__host__ __device__ __forceinline__ Fe<C> fe_one() {
  Fe<C> r;
#pragma unroll
  for (int i = 0; i < 8; ++i) r.v[i] = C::R(i);
  return r;
}

template <class C>
__device__ __forceinline__ bool fe_is_zero(const Fe<C>& a) {
  return (a.v[0] | a.v[1] | a.v[2] | a.v[3] | a.v[4] | a.v[5] | a.v[6] | a.v[7]) == 0;
}

template <class C>
__device__ __forceinline__ bool fe_eq(const Fe<C>& a, const Fe<C>& b) {
  uint32_t d = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) d |= a.v[i] ^ b.v[i];
  return d == 0;
}

// r = a - m if a >= m (a < 2m): subtract, keep the difference unless it borrowed.
template <class C>
__device__ __forceinline__ void fe_reduce_once(uint32_t r[8]) {
  uint32_t s0, s1, s2, s3, s4, s5, s6, s7, br;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(s0), "=r"(s1), "=r"(s2), "=r"(s3), "=r"(s4), "=r"(s5), "=r"(s6), "=r"(s7), "=r"(br)
      : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]),
        "n"(C::P0), "n"(C::P1), "n"(C::P2), "n"(C::P3), "n"(C::P4), "n"(C::P5), "n"(C::P6), "n"(C::P7));
  const bool keep = br != 0;
  r[0] = keep ? r[0] : s0;
  r[1] = keep ? r[1] : s1;
  r[2] = keep ? r[2] : s2;
  r[3] = keep ? r[3] : s3;
  r[4] = keep ? r[4] : s4;
  r[5] = keep ? r[5] : s5;
  r[6] = keep ? r[6] : s6;
  r[7] = keep ? r[7] : s7;
}

template <class C>
__device__ __forceinline__ Fe<C> fe_add(const Fe<C>& a, const Fe<C>& b) {
  Fe<C> r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
        "=r"(r.v[7])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  fe_reduce_once<C>(r.v);
  return r;
}

template <class C>
__device__ __forceinline__ Fe<C> fe_sub(const Fe<C>& a, const Fe<C>& b) {
  Fe<C> r;
  uint32_t br;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
        "=r"(r.v[7]), "=r"(br)
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]),
        "r"(b.v[0]), "r"(b.v[1]), "r"(b.v[2]), "r"(b.v[3]), "r"(b.v[4]), "r"(b.v[5]), "r"(b.v[6]), "r"(b.v[7]));
  // On borrow add the modulus back (masked add: br is 0 or all ones).
  asm("add.cc.u32  %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;"
      : "+r"(r.v[0]), "+r"(r.v[1]), "+r"(r.v[2]), "+r"(r.v[3]), "+r"(r.v[4]), "+r"(r.v[5]), "+r"(r.v[6]),
        "+r"(r.v[7])
      : "r"(br & C::P0), "r"(br & C::P1), "r"(br & C::P2), "r"(br & C::P3), "r"(br & C::P4), "r"(br & C::P5),
        "r"(br & C::P6), "r"(br & C::P7));
  return r;
}

template <class C>
__device__ __forceinline__ Fe<C> fe_neg(const Fe<C>& a) {
  return fe_is_zero(a) ? a : fe_sub(fe_zero<C>(), a);
}

template <class C>
__device__ __forceinline__ Fe<C> fe_dbl(const Fe<C>& a) {
  return fe_add(a, a);
}

// ---- products ------------------------------------------------------------------
//
// A value T is held as two arrays of eight words, T = E + 2^32 O: every
// partial product of limb j and a multiplier lands in words (j, j + 1), so
// the products of the even limbs fill E in one chain of four wide
// multiply-adds with carry, those of the odd limbs fill O, and neither chain
// needs a carry beyond its own words (T stays below 2^288 within a row). The
// low and the high half of a product are consecutive instructions on
// consecutive words, which is what lets them run as one wide instruction.
//
// A Montgomery row adds a b_i, then m p with m = -E_0 p^-1 mod 2^32, which
// clears E_0; dividing by 2^32 then makes O the next row's E (its words now
// stand at 0..7), moves E_2.. down to be the next O, and adds E_1 into the
// new E_0, the carry of which is the next row's carry into its odd chain.

// (E, O) <- T / 2^32 (word E_0 is zero or retired), returned with the roles
// as the asm blocks below leave them: the new E in o[], the new O in e[2..7]
// and two new top words.
__device__ __forceinline__ void eo_swap(uint32_t e[8], uint32_t o[8], uint32_t n6, uint32_t n7) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const uint32_t t = o[k];
    o[k] = k < 6 ? e[k + 2 < 8 ? k + 2 : 7] : k == 6 ? n6 : n7;
    e[k] = t;
  }
}

// E = even limbs of a times b, O = odd limbs (the first row).
__device__ __forceinline__ void eo_first(uint32_t e[8], uint32_t o[8], const uint32_t a[8], uint32_t b) {
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    const uint64_t x = (uint64_t)a[k] * b, y = (uint64_t)a[k + 1] * b;
    e[k] = (uint32_t)x;
    e[k + 1] = (uint32_t)(x >> 32);
    o[k] = (uint32_t)y;
    o[k + 1] = (uint32_t)(y >> 32);
  }
}

// T <- T / 2^32 + a b.
__device__ __forceinline__ void eo_mul_row(uint32_t e[8], uint32_t o[8], const uint32_t a[8], uint32_t b) {
  uint32_t n6, n7;
  asm("add.cc.u32     %0, %0, %8;\n\t"
      "madc.lo.cc.u32 %9, %18, %24, %9;\n\t"
      "madc.hi.cc.u32 %10, %18, %24, %10;\n\t"
      "madc.lo.cc.u32 %11, %20, %24, %11;\n\t"
      "madc.hi.cc.u32 %12, %20, %24, %12;\n\t"
      "madc.lo.cc.u32 %13, %22, %24, %13;\n\t"
      "madc.hi.cc.u32 %14, %22, %24, %14;\n\t"
      "madc.lo.cc.u32 %15, %25, %24, 0;\n\t"
      "madc.hi.u32    %16, %25, %24, 0;\n\t"
      "mad.lo.cc.u32  %0, %17, %24, %0;\n\t"
      "madc.hi.cc.u32 %1, %17, %24, %1;\n\t"
      "madc.lo.cc.u32 %2, %19, %24, %2;\n\t"
      "madc.hi.cc.u32 %3, %19, %24, %3;\n\t"
      "madc.lo.cc.u32 %4, %21, %24, %4;\n\t"
      "madc.hi.cc.u32 %5, %21, %24, %5;\n\t"
      "madc.lo.cc.u32 %6, %23, %24, %6;\n\t"
      "madc.hi.cc.u32 %7, %23, %24, %7;\n\t"
      "addc.u32       %16, %16, 0;"
      : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]),
        "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "=&r"(n6), "=&r"(n7)
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(a[4]), "r"(a[5]), "r"(a[6]), "r"(b), "r"(a[7]));
  eo_swap(e, o, n6, n7);
}

// T <- T + m p, m chosen to clear the low word.
template <class C>
__device__ __forceinline__ void eo_reduce_row(uint32_t e[8], uint32_t o[8]) {
  const uint32_t m = e[0] * C::INV;
  asm("mad.lo.cc.u32  %8, %16, %18, %8;\n\t"
      "madc.hi.cc.u32 %9, %16, %18, %9;\n\t"
      "madc.lo.cc.u32 %10, %16, %20, %10;\n\t"
      "madc.hi.cc.u32 %11, %16, %20, %11;\n\t"
      "madc.lo.cc.u32 %12, %16, %22, %12;\n\t"
      "madc.hi.cc.u32 %13, %16, %22, %13;\n\t"
      "madc.lo.cc.u32 %14, %16, %24, %14;\n\t"
      "madc.hi.u32    %15, %16, %24, %15;\n\t"
      "mad.lo.cc.u32  %0, %16, %17, %0;\n\t"
      "madc.hi.cc.u32 %1, %16, %17, %1;\n\t"
      "madc.lo.cc.u32 %2, %16, %19, %2;\n\t"
      "madc.hi.cc.u32 %3, %16, %19, %3;\n\t"
      "madc.lo.cc.u32 %4, %16, %21, %4;\n\t"
      "madc.hi.cc.u32 %5, %16, %21, %5;\n\t"
      "madc.lo.cc.u32 %6, %16, %23, %6;\n\t"
      "madc.hi.cc.u32 %7, %16, %23, %7;\n\t"
      "addc.u32       %15, %15, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]),
        "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7])
      : "r"(m), "n"(C::P0), "n"(C::P1), "n"(C::P2), "n"(C::P3), "n"(C::P4), "n"(C::P5), "n"(C::P6), "n"(C::P7));
}

// T <- T / 2^32 + m p, m chosen to clear the low word (a row with no product).
template <class C>
__device__ __forceinline__ void eo_shift_reduce_row(uint32_t e[8], uint32_t o[8]) {
  const uint32_t m = (o[0] + e[1]) * C::INV;
  uint32_t n6, n7;
  asm("add.cc.u32     %0, %0, %8;\n\t"
      "madc.lo.cc.u32 %9, %17, %19, %9;\n\t"
      "madc.hi.cc.u32 %10, %17, %19, %10;\n\t"
      "madc.lo.cc.u32 %11, %17, %21, %11;\n\t"
      "madc.hi.cc.u32 %12, %17, %21, %12;\n\t"
      "madc.lo.cc.u32 %13, %17, %23, %13;\n\t"
      "madc.hi.cc.u32 %14, %17, %23, %14;\n\t"
      "madc.lo.cc.u32 %15, %17, %25, 0;\n\t"
      "madc.hi.u32    %16, %17, %25, 0;\n\t"
      "mad.lo.cc.u32  %0, %17, %18, %0;\n\t"
      "madc.hi.cc.u32 %1, %17, %18, %1;\n\t"
      "madc.lo.cc.u32 %2, %17, %20, %2;\n\t"
      "madc.hi.cc.u32 %3, %17, %20, %3;\n\t"
      "madc.lo.cc.u32 %4, %17, %22, %4;\n\t"
      "madc.hi.cc.u32 %5, %17, %22, %5;\n\t"
      "madc.lo.cc.u32 %6, %17, %24, %6;\n\t"
      "madc.hi.cc.u32 %7, %17, %24, %7;\n\t"
      "addc.u32       %16, %16, 0;"
      : "+r"(o[0]), "+r"(o[1]), "+r"(o[2]), "+r"(o[3]), "+r"(o[4]), "+r"(o[5]), "+r"(o[6]), "+r"(o[7]),
        "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "=&r"(n6), "=&r"(n7)
      : "r"(m), "n"(C::P0), "n"(C::P1), "n"(C::P2), "n"(C::P3), "n"(C::P4), "n"(C::P5), "n"(C::P6), "n"(C::P7));
  eo_swap(e, o, n6, n7);
}

// r = T / 2^32 (the low word zero or retired): O plus E's words 1..7.
__device__ __forceinline__ void eo_merge(uint32_t r[8], const uint32_t e[8], const uint32_t o[8]) {
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, 0;"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(o[0]), "r"(o[1]), "r"(o[2]), "r"(o[3]), "r"(o[4]), "r"(o[5]), "r"(o[6]), "r"(o[7]), "r"(e[1]), "r"(e[2]),
        "r"(e[3]), "r"(e[4]), "r"(e[5]), "r"(e[6]), "r"(e[7]));
}

// a b / 2^256 mod p: eight product rows, each followed by its reduction row.
// With a, b < m < 2^254 T stays below 2m between rows, so the result needs
// one conditional subtraction.
template <class C>
__device__ __forceinline__ Fe<C> fe_mul(const Fe<C>& a, const Fe<C>& b) {
  uint32_t e[8], o[8];
  eo_first(e, o, a.v, b.v[0]);
  eo_reduce_row<C>(e, o);
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    eo_mul_row(e, o, a.v, b.v[i]);
    eo_reduce_row<C>(e, o);
  }
  Fe<C> r;
  eo_merge(r.v, e, o);
  fe_reduce_once<C>(r.v);
  return r;
}

// (t + M m) / 2^256 for the M below 2^256 that clears the low 256 bits of t
// (eight words): the reduction rows alone. At most m.
template <class C>
__device__ __forceinline__ void eo_redc(uint32_t r[8], const uint32_t t[8]) {
  const uint32_t p[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
  uint32_t e[8], o[8];
  const uint32_t m = t[0] * C::INV;
#pragma unroll
  for (int k = 0; k < 8; k += 2) {
    e[k] = t[k];
    e[k + 1] = t[k + 1];
    const uint64_t y = (uint64_t)p[k + 1] * m;
    o[k] = (uint32_t)y;
    o[k + 1] = (uint32_t)(y >> 32);
  }
  asm("mad.lo.cc.u32  %0, %9, %10, %0;\n\t"
      "madc.hi.cc.u32 %1, %9, %10, %1;\n\t"
      "madc.lo.cc.u32 %2, %9, %11, %2;\n\t"
      "madc.hi.cc.u32 %3, %9, %11, %3;\n\t"
      "madc.lo.cc.u32 %4, %9, %12, %4;\n\t"
      "madc.hi.cc.u32 %5, %9, %12, %5;\n\t"
      "madc.lo.cc.u32 %6, %9, %13, %6;\n\t"
      "madc.hi.cc.u32 %7, %9, %13, %7;\n\t"
      "addc.u32       %8, %8, 0;"
      : "+r"(e[0]), "+r"(e[1]), "+r"(e[2]), "+r"(e[3]), "+r"(e[4]), "+r"(e[5]), "+r"(e[6]), "+r"(e[7]), "+r"(o[7])
      : "r"(m), "n"(C::P0), "n"(C::P2), "n"(C::P4), "n"(C::P6));
#pragma unroll
  for (int i = 1; i < 8; ++i) eo_shift_reduce_row<C>(e, o);
  eo_merge(r, e, o);
}

// The cross products a_i a_j (i < j) of a square, each once, into words 1..14
// of two arrays by the parity of their position i + j. A row's chain ends
// either on words no earlier row of its parity has touched (a_7's product) or
// one short of them (a_6's), where its carry starts the next word.
__device__ __forceinline__ void eo_cross(uint32_t E[16], uint32_t O[16], const uint32_t a[8]) {
#pragma unroll
  for (int j = 1; j < 8; ++j) {
    const uint64_t x = (uint64_t)a[0] * a[j];
    uint32_t* w = (j & 1) ? O : E;
    w[j] = (uint32_t)x;
    w[j + 1] = (uint32_t)(x >> 32);
  }
  asm("mad.lo.cc.u32  %0, %7, %8, %0;\n\t"  // a_1: a_2, a_4, a_6
      "madc.hi.cc.u32 %1, %7, %8, %1;\n\t"
      "madc.lo.cc.u32 %2, %7, %9, %2;\n\t"
      "madc.hi.cc.u32 %3, %7, %9, %3;\n\t"
      "madc.lo.cc.u32 %4, %7, %10, %4;\n\t"
      "madc.hi.cc.u32 %5, %7, %10, %5;\n\t"
      "addc.u32       %6, 0, 0;"
      : "+r"(O[3]), "+r"(O[4]), "+r"(O[5]), "+r"(O[6]), "+r"(O[7]), "+r"(O[8]), "=r"(O[9])
      : "r"(a[1]), "r"(a[2]), "r"(a[4]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %6, %7, %0;\n\t"  // a_1: a_3, a_5, a_7
      "madc.hi.cc.u32 %1, %6, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %8, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %8, %3;\n\t"
      "madc.lo.cc.u32 %4, %6, %9, 0;\n\t"
      "madc.hi.u32    %5, %6, %9, 0;"
      : "+r"(E[4]), "+r"(E[5]), "+r"(E[6]), "+r"(E[7]), "=&r"(E[8]), "=&r"(E[9])
      : "r"(a[1]), "r"(a[3]), "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %6, %7, %0;\n\t"  // a_2: a_3, a_5, a_7
      "madc.hi.cc.u32 %1, %6, %7, %1;\n\t"
      "madc.lo.cc.u32 %2, %6, %8, %2;\n\t"
      "madc.hi.cc.u32 %3, %6, %8, %3;\n\t"
      "madc.lo.cc.u32 %4, %6, %9, %4;\n\t"
      "madc.hi.u32    %5, %6, %9, 0;"
      : "+r"(O[5]), "+r"(O[6]), "+r"(O[7]), "+r"(O[8]), "+r"(O[9]), "=&r"(O[10])
      : "r"(a[2]), "r"(a[3]), "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"  // a_2: a_4, a_6
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;"
      : "+r"(E[6]), "+r"(E[7]), "+r"(E[8]), "+r"(E[9]), "=r"(E[10])
      : "r"(a[2]), "r"(a[4]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %5, %6, %0;\n\t"  // a_3: a_4, a_6
      "madc.hi.cc.u32 %1, %5, %6, %1;\n\t"
      "madc.lo.cc.u32 %2, %5, %7, %2;\n\t"
      "madc.hi.cc.u32 %3, %5, %7, %3;\n\t"
      "addc.u32       %4, 0, 0;"
      : "+r"(O[7]), "+r"(O[8]), "+r"(O[9]), "+r"(O[10]), "=r"(O[11])
      : "r"(a[3]), "r"(a[4]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"  // a_3: a_5, a_7
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, %2;\n\t"
      "madc.hi.u32    %3, %4, %6, 0;"
      : "+r"(E[8]), "+r"(E[9]), "+r"(E[10]), "=&r"(E[11])
      : "r"(a[3]), "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %4, %5, %0;\n\t"  // a_4: a_5, a_7
      "madc.hi.cc.u32 %1, %4, %5, %1;\n\t"
      "madc.lo.cc.u32 %2, %4, %6, %2;\n\t"
      "madc.hi.u32    %3, %4, %6, 0;"
      : "+r"(O[9]), "+r"(O[10]), "+r"(O[11]), "=&r"(O[12])
      : "r"(a[4]), "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"  // a_4: a_6
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32       %2, 0, 0;"
      : "+r"(E[10]), "+r"(E[11]), "=r"(E[12])
      : "r"(a[4]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %3, %4, %0;\n\t"  // a_5: a_6
      "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
      "addc.u32       %2, 0, 0;"
      : "+r"(O[11]), "+r"(O[12]), "=r"(O[13])
      : "r"(a[5]), "r"(a[6]));
  asm("mad.lo.cc.u32  %0, %2, %3, %0;\n\t"  // a_5: a_7
      "madc.hi.u32    %1, %2, %3, 0;"
      : "+r"(E[12]), "=&r"(E[13])
      : "r"(a[5]), "r"(a[7]));
  asm("mad.lo.cc.u32  %0, %2, %3, %0;\n\t"  // a_6: a_7
      "madc.hi.u32    %1, %2, %3, 0;"
      : "+r"(O[13]), "=&r"(O[14])
      : "r"(a[6]), "r"(a[7]));
}

// a^2 / 2^256 mod p: the 28 cross products once, doubled, the eight squares
// added, then the reduction rows: 100 wide products against 128 in a multiply
// (measured on GB300: 85 G squares/s against 72 G products/s, 728 clocks
// alone against 847). a^2 < 2^508, so the doubling never carries out of 16
// words, and the reduced low half (at most m) plus the high half is below 2m.
template <class C>
__device__ __forceinline__ Fe<C> fe_sqr(const Fe<C>& a) {
  uint32_t E[16], O[16], T[16], cy;
  eo_cross(E, O, a.v);
  T[0] = 0;
  T[1] = O[1];
  asm("add.cc.u32  %0, %7, %13;\n\t"
      "addc.cc.u32 %1, %8, %14;\n\t"
      "addc.cc.u32 %2, %9, %15;\n\t"
      "addc.cc.u32 %3, %10, %16;\n\t"
      "addc.cc.u32 %4, %11, %17;\n\t"
      "addc.cc.u32 %5, %12, %18;\n\t"
      "addc.u32    %6, 0, 0;"
      : "=&r"(T[2]), "=&r"(T[3]), "=&r"(T[4]), "=&r"(T[5]), "=&r"(T[6]), "=&r"(T[7]), "=&r"(cy)
      : "r"(E[2]), "r"(E[3]), "r"(E[4]), "r"(E[5]), "r"(E[6]), "r"(E[7]), "r"(O[2]), "r"(O[3]), "r"(O[4]), "r"(O[5]),
        "r"(O[6]), "r"(O[7]));
  asm("{\n\t"
      ".reg .u32 t;\n\t"
      "add.cc.u32  t, %20, 0xffffffff;\n\t"  // the carry back into the flag
      "addc.cc.u32 %0, %7, %13;\n\t"
      "addc.cc.u32 %1, %8, %14;\n\t"
      "addc.cc.u32 %2, %9, %15;\n\t"
      "addc.cc.u32 %3, %10, %16;\n\t"
      "addc.cc.u32 %4, %11, %17;\n\t"
      "addc.cc.u32 %5, %12, %18;\n\t"
      "addc.u32    %6, %19, 0;\n\t"
      "}"
      : "=&r"(T[8]), "=&r"(T[9]), "=&r"(T[10]), "=&r"(T[11]), "=&r"(T[12]), "=&r"(T[13]), "=&r"(T[14])
      : "r"(E[8]), "r"(E[9]), "r"(E[10]), "r"(E[11]), "r"(E[12]), "r"(E[13]), "r"(O[8]), "r"(O[9]), "r"(O[10]),
        "r"(O[11]), "r"(O[12]), "r"(O[13]), "r"(O[14]), "r"(cy));
  T[15] = T[14] >> 31;
#pragma unroll
  for (int k = 14; k > 1; --k) T[k] = __funnelshift_l(T[k - 1], T[k], 1);
  T[1] <<= 1;
  asm("mad.lo.cc.u32  %0, %16, %16, 0;\n\t"
      "madc.hi.cc.u32 %1, %16, %16, %1;\n\t"
      "madc.lo.cc.u32 %2, %17, %17, %2;\n\t"
      "madc.hi.cc.u32 %3, %17, %17, %3;\n\t"
      "madc.lo.cc.u32 %4, %18, %18, %4;\n\t"
      "madc.hi.cc.u32 %5, %18, %18, %5;\n\t"
      "madc.lo.cc.u32 %6, %19, %19, %6;\n\t"
      "madc.hi.cc.u32 %7, %19, %19, %7;\n\t"
      "madc.lo.cc.u32 %8, %20, %20, %8;\n\t"
      "madc.hi.cc.u32 %9, %20, %20, %9;\n\t"
      "madc.lo.cc.u32 %10, %21, %21, %10;\n\t"
      "madc.hi.cc.u32 %11, %21, %21, %11;\n\t"
      "madc.lo.cc.u32 %12, %22, %22, %12;\n\t"
      "madc.hi.cc.u32 %13, %22, %22, %13;\n\t"
      "madc.lo.cc.u32 %14, %23, %23, %14;\n\t"
      "madc.hi.u32    %15, %23, %23, %15;"
      : "+r"(T[0]), "+r"(T[1]), "+r"(T[2]), "+r"(T[3]), "+r"(T[4]), "+r"(T[5]), "+r"(T[6]), "+r"(T[7]), "+r"(T[8]),
        "+r"(T[9]), "+r"(T[10]), "+r"(T[11]), "+r"(T[12]), "+r"(T[13]), "+r"(T[14]), "+r"(T[15])
      : "r"(a.v[0]), "r"(a.v[1]), "r"(a.v[2]), "r"(a.v[3]), "r"(a.v[4]), "r"(a.v[5]), "r"(a.v[6]), "r"(a.v[7]));
  uint32_t lo[8];
  eo_redc<C>(lo, T);
  Fe<C> r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]), "r"(lo[4]), "r"(lo[5]), "r"(lo[6]), "r"(lo[7]), "r"(T[8]),
        "r"(T[9]), "r"(T[10]), "r"(T[11]), "r"(T[12]), "r"(T[13]), "r"(T[14]), "r"(T[15]));
  fe_reduce_once<C>(r.v);
  return r;
}

// Sums of up to fifteen products, reduced once: each product costs its 64 wide
// products and an addition of 16 words, and the sum one set of reduction rows.
// Fifteen products of values below m stay below 2^512 (m^2 < 2^507.2), and
// their reduced value below 15 * 0.19 m + m < 4 m.
constexpr int kWideProducts = 15;

template <class C>
struct FeWide {
  uint32_t w[16];
};

template <class C>
__device__ __forceinline__ FeWide<C> wide_zero() {
  FeWide<C> r;
#pragma unroll
  for (int k = 0; k < 16; ++k) r.w[k] = 0;
  return r;
}

// acc += a b.
template <class C>
__device__ __forceinline__ void wide_mac(FeWide<C>& acc, const Fe<C>& a, const Fe<C>& b) {
  uint32_t e[8], o[8], t[16], cy;
  eo_first(e, o, a.v, b.v[0]);
  t[0] = e[0];
#pragma unroll
  for (int i = 1; i < 8; ++i) {
    eo_mul_row(e, o, a.v, b.v[i]);
    t[i] = e[0];
  }
  eo_merge(t + 8, e, o);
  asm("add.cc.u32  %0, %0, %9;\n\t"
      "addc.cc.u32 %1, %1, %10;\n\t"
      "addc.cc.u32 %2, %2, %11;\n\t"
      "addc.cc.u32 %3, %3, %12;\n\t"
      "addc.cc.u32 %4, %4, %13;\n\t"
      "addc.cc.u32 %5, %5, %14;\n\t"
      "addc.cc.u32 %6, %6, %15;\n\t"
      "addc.cc.u32 %7, %7, %16;\n\t"
      "addc.u32    %8, 0, 0;"
      : "+r"(acc.w[0]), "+r"(acc.w[1]), "+r"(acc.w[2]), "+r"(acc.w[3]), "+r"(acc.w[4]), "+r"(acc.w[5]), "+r"(acc.w[6]),
        "+r"(acc.w[7]), "=&r"(cy)
      : "r"(t[0]), "r"(t[1]), "r"(t[2]), "r"(t[3]), "r"(t[4]), "r"(t[5]), "r"(t[6]), "r"(t[7]));
  asm("{\n\t"
      ".reg .u32 x;\n\t"
      "add.cc.u32  x, %16, 0xffffffff;\n\t"  // the carry back into the flag
      "addc.cc.u32 %0, %0, %8;\n\t"
      "addc.cc.u32 %1, %1, %9;\n\t"
      "addc.cc.u32 %2, %2, %10;\n\t"
      "addc.cc.u32 %3, %3, %11;\n\t"
      "addc.cc.u32 %4, %4, %12;\n\t"
      "addc.cc.u32 %5, %5, %13;\n\t"
      "addc.cc.u32 %6, %6, %14;\n\t"
      "addc.u32    %7, %7, %15;\n\t"
      "}"
      : "+r"(acc.w[8]), "+r"(acc.w[9]), "+r"(acc.w[10]), "+r"(acc.w[11]), "+r"(acc.w[12]), "+r"(acc.w[13]),
        "+r"(acc.w[14]), "+r"(acc.w[15])
      : "r"(t[8]), "r"(t[9]), "r"(t[10]), "r"(t[11]), "r"(t[12]), "r"(t[13]), "r"(t[14]), "r"(t[15]), "r"(cy));
}

// r = a - 2m if a >= 2m.
template <class C>
__device__ __forceinline__ void fe_sub_twice_if(uint32_t r[8]) {
  constexpr uint32_t q[8] = {C::P0 << 1,
                             (C::P1 << 1) | (C::P0 >> 31),
                             (C::P2 << 1) | (C::P1 >> 31),
                             (C::P3 << 1) | (C::P2 >> 31),
                             (C::P4 << 1) | (C::P3 >> 31),
                             (C::P5 << 1) | (C::P4 >> 31),
                             (C::P6 << 1) | (C::P5 >> 31),
                             (C::P7 << 1) | (C::P6 >> 31)};
  uint32_t s0, s1, s2, s3, s4, s5, s6, s7, br;
  asm("sub.cc.u32  %0, %9, %17;\n\t"
      "subc.cc.u32 %1, %10, %18;\n\t"
      "subc.cc.u32 %2, %11, %19;\n\t"
      "subc.cc.u32 %3, %12, %20;\n\t"
      "subc.cc.u32 %4, %13, %21;\n\t"
      "subc.cc.u32 %5, %14, %22;\n\t"
      "subc.cc.u32 %6, %15, %23;\n\t"
      "subc.cc.u32 %7, %16, %24;\n\t"
      "subc.u32    %8, 0, 0;"
      : "=r"(s0), "=r"(s1), "=r"(s2), "=r"(s3), "=r"(s4), "=r"(s5), "=r"(s6), "=r"(s7), "=r"(br)
      : "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "n"(q[0]), "n"(q[1]),
        "n"(q[2]), "n"(q[3]), "n"(q[4]), "n"(q[5]), "n"(q[6]), "n"(q[7]));
  const bool keep = br != 0;
  r[0] = keep ? r[0] : s0;
  r[1] = keep ? r[1] : s1;
  r[2] = keep ? r[2] : s2;
  r[3] = keep ? r[3] : s3;
  r[4] = keep ? r[4] : s4;
  r[5] = keep ? r[5] : s5;
  r[6] = keep ? r[6] : s6;
  r[7] = keep ? r[7] : s7;
}

// The sum's value times 2^-256 mod m.
template <class C>
__device__ __forceinline__ Fe<C> fe_from_wide(const FeWide<C>& a) {
  uint32_t lo[8];
  eo_redc<C>(lo, a.w);
  Fe<C> r;
  asm("add.cc.u32  %0, %8, %16;\n\t"
      "addc.cc.u32 %1, %9, %17;\n\t"
      "addc.cc.u32 %2, %10, %18;\n\t"
      "addc.cc.u32 %3, %11, %19;\n\t"
      "addc.cc.u32 %4, %12, %20;\n\t"
      "addc.cc.u32 %5, %13, %21;\n\t"
      "addc.cc.u32 %6, %14, %22;\n\t"
      "addc.u32    %7, %15, %23;"
      : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
      : "r"(lo[0]), "r"(lo[1]), "r"(lo[2]), "r"(lo[3]), "r"(lo[4]), "r"(lo[5]), "r"(lo[6]), "r"(lo[7]), "r"(a.w[8]),
        "r"(a.w[9]), "r"(a.w[10]), "r"(a.w[11]), "r"(a.w[12]), "r"(a.w[13]), "r"(a.w[14]), "r"(a.w[15]));
  fe_sub_twice_if<C>(r.v);
  fe_reduce_once<C>(r.v);
  return r;
}

// Montgomery form -> canonical limbs (multiply by 1), and back (multiply by R^2).
template <class C>
__device__ __forceinline__ Fe<C> fe_from_mont(const Fe<C>& a) {
  Fe<C> r;
  eo_redc<C>(r.v, a.v);
  fe_reduce_once<C>(r.v);
  return r;
}

template <class C>
__device__ __forceinline__ Fe<C> fe_to_mont(const Fe<C>& a) {
  Fe<C> r2;
#pragma unroll
  for (int i = 0; i < 8; ++i) r2.v[i] = C::R2(i);
  return fe_mul(a, r2);
}

template <class C>
__device__ __forceinline__ Fe<C> fe_from_u64(uint64_t x) {
  Fe<C> a = fe_zero<C>();
  a.v[0] = (uint32_t)x;
  a.v[1] = (uint32_t)(x >> 32);
  return fe_to_mont(a);
}

// Canonical value < m? (used to validate inputs arriving in canonical form)
template <class C>
__device__ __forceinline__ bool fe_lt_mod(const uint32_t a[8]) {
  const uint32_t p[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
#pragma unroll
  for (int i = 7; i >= 0; --i) {
    if (a[i] != p[i]) return a[i] < p[i];
  }
  return false;
}

// 1/a by Bernstein and Yang's divsteps ("Fast constant-time gcd computation
// and modular inversion", 2019), in the half-delta form, on the Montgomery
// value A = aR. State: delta (starts at 1/2), f = m (odd), g = A, and
// d, e with f = d A and g = e A (mod m), starting at d = 0, e = 1. One divstep:
// if delta > 0 and g is odd, (delta, f, g) <- (1 - delta, g, (g - f) / 2);
// otherwise (1 + delta, f, (g + (g mod 2) f) / 2). g reaches 0 with f = +-1,
// and then 1/A = +-d. Thirty divsteps depend only on the low 32 bits of f and
// g, so they run on those bits alone and yield an integer matrix T with
// 2^30 (f', g') = T (f, g) (entries at most 2^30); T is then applied once to
// the full f, g and (mod m) to d, e. Big values are nine signed 30-bit limbs
// (value = sum l_i 2^(30 i), limbs 0..7 in [0, 2^30), limb 8 signed), so a
// limb of T (f, g) is one 64-bit sum of 32x32 products. For d, e the multiple
// k m that clears the low 30 bits (k = -(T (d, e))_0 m^-1 mod 2^30, taken in
// [-2^29, 2^29)) is added before the division: each batch grows |d|, |e| by
// less than m / 2, so they stay below 2^269 for the batches a 254-bit modulus
// needs (the half-delta form needs at most 590 divsteps for 256-bit inputs:
// 20 batches; measured at most 18 over 400,000 random inputs of both fields),
// and one reduction at the end brings d into [0, m). Variable time (the
// inputs are public values). Written as __host__ __device__ plain C++ so the
// same code is checked on the host.
struct Signed30 {
  int32_t l[9];
};

__host__ __device__ __forceinline__ Signed30 s30_from_words(const uint32_t w[8]) {
  Signed30 s;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    const int bit = 30 * i, wi = bit >> 5, sh = bit & 31;
    uint64_t v = wi < 8 ? (uint64_t)(w[wi] >> sh) : 0;
    if (wi + 1 < 8 && sh) v |= (uint64_t)w[wi + 1] << (32 - sh);
    s.l[i] = (int32_t)(v & 0x3fffffffu);
  }
  return s;
}

// (f, g) <- (u f + v g, q f + r g) / 2^30 (exact: the low 30 bits cancel).
__host__ __device__ __forceinline__ void s30_update_fg(Signed30& f, Signed30& g, int32_t u, int32_t v, int32_t q,
                                                       int32_t r) {
  int64_t cf = ((int64_t)u * f.l[0] + (int64_t)v * g.l[0]) >> 30;
  int64_t cg = ((int64_t)q * f.l[0] + (int64_t)r * g.l[0]) >> 30;
#pragma unroll
  for (int i = 1; i < 9; ++i) {
    cf += (int64_t)u * f.l[i] + (int64_t)v * g.l[i];
    cg += (int64_t)q * f.l[i] + (int64_t)r * g.l[i];
    f.l[i - 1] = (int32_t)(cf & 0x3fffffff);
    g.l[i - 1] = (int32_t)(cg & 0x3fffffff);
    cf >>= 30;
    cg >>= 30;
  }
  f.l[8] = (int32_t)cf;
  g.l[8] = (int32_t)cg;
}

// (d, e) <- (u d + v e + k_d m, q d + r e + k_e m) / 2^30, each k chosen to
// clear the low 30 bits, so the results are d / 2^30-style values mod m.
__host__ __device__ __forceinline__ void s30_update_de(Signed30& d, Signed30& e, int32_t u, int32_t v, int32_t q,
                                                       int32_t r, const Signed30& m, uint32_t minv30) {
  const int64_t d0 = (int64_t)u * d.l[0] + (int64_t)v * e.l[0];
  const int64_t e0 = (int64_t)q * d.l[0] + (int64_t)r * e.l[0];
  int32_t kd = (int32_t)(((uint32_t)(0u - (uint32_t)d0) * minv30) & 0x3fffffffu);
  int32_t ke = (int32_t)(((uint32_t)(0u - (uint32_t)e0) * minv30) & 0x3fffffffu);
  kd -= (kd >> 29) << 30;  // into [-2^29, 2^29)
  ke -= (ke >> 29) << 30;
  int64_t cd = (d0 + (int64_t)kd * m.l[0]) >> 30;
  int64_t ce = (e0 + (int64_t)ke * m.l[0]) >> 30;
#pragma unroll
  for (int i = 1; i < 9; ++i) {
    cd += (int64_t)u * d.l[i] + (int64_t)v * e.l[i] + (int64_t)kd * m.l[i];
    ce += (int64_t)q * d.l[i] + (int64_t)r * e.l[i] + (int64_t)ke * m.l[i];
    d.l[i - 1] = (int32_t)(cd & 0x3fffffff);
    e.l[i - 1] = (int32_t)(ce & 0x3fffffff);
    cd >>= 30;
    ce >>= 30;
  }
  d.l[8] = (int32_t)cd;
  e.l[8] = (int32_t)ce;
}

// Nine-limb signed value -> nine 32-bit words, two's complement.
__host__ __device__ __forceinline__ void s30_to_words(const Signed30& s, uint32_t w[9]) {
  uint64_t acc = 0;
  int nb = 0, j = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    acc |= (uint64_t)(uint32_t)s.l[i] << nb;
    nb += 30;
    if (nb >= 32) {
      w[j++] = (uint32_t)acc;
      acc >>= 32;
      nb -= 32;
    }
  }
  const int64_t top = (int64_t)s.l[8] * ((int64_t)1 << nb) + (int64_t)acc;  // nb = 16 here
  w[7] = (uint32_t)top;
  w[8] = (uint32_t)(top >> 32);
}

// w += a on nine words.
__host__ __device__ __forceinline__ void words9_add(uint32_t w[9], const uint32_t a[9]) {
  uint64_t c = 0;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    c += (uint64_t)w[i] + a[i];
    w[i] = (uint32_t)c;
    c >>= 32;
  }
}

// w -= a when w >= a (both nonnegative nine-word values).
__host__ __device__ __forceinline__ void words9_csub(uint32_t w[9], const uint32_t a[9]) {
  uint32_t t[9];
  int64_t b = 0;
#pragma unroll
  for (int i = 0; i < 9; ++i) {
    b += (int64_t)w[i] - a[i];
    t[i] = (uint32_t)b;
    b >>= 32;
  }
  if (b == 0) {
#pragma unroll
    for (int i = 0; i < 9; ++i) w[i] = t[i];
  }
}

// Trailing zeros of a nonzero word.
__host__ __device__ __forceinline__ int ctz32(uint32_t x) {
#ifdef __CUDA_ARCH__
  return __ffs((int)x) - 1;
#else
  return __builtin_ctz(x);
#endif
}

// Thirty divsteps on the low words of f and g, with the matrix they amount to
// (times 2^30), zeta = -(delta + 1/2) in and out. In variable time (an inversion
// of one warp on a GB300: 42,100 -> 27,700 clocks; spreading the two updates over
// the lanes of a quad, 32,900): a run of
// even g's is one shift, and while zeta >= 0 the next zeta + 1 steps exchange
// nothing, so up to six of them are one addition of w f, w = -g / f mod 2^6 (for
// odd f, f (f^2 - 2) f = (f^2 - 1)^2 - 1 = -1 mod 64). The form of the divsteps
// is that of P. Wuille's "The safegcd implementation in libsecp256k1 explained".
__host__ __device__ __forceinline__ void divsteps30(uint32_t f, uint32_t g, int32_t& zeta, int32_t& u, int32_t& v,
                                                    int32_t& q, int32_t& r) {
  u = 1, v = 0, q = 0, r = 1;
  int left = 30;
  for (;;) {
    const int z = ctz32(g | (1u << left));
    g >>= z;
    u = (int32_t)((uint32_t)u << z);
    v = (int32_t)((uint32_t)v << z);
    zeta -= z;
    left -= z;
    if (left == 0) return;
    if (zeta < 0) {  // delta > 0 and g odd: (f, g) <- (g, -f)
      zeta = -zeta - 1;
      uint32_t t = f;
      f = g;
      g = 0u - t;
      int32_t s = u;
      u = q;
      q = -s;
      s = v;
      v = r;
      r = -s;
    }
    const int steps = zeta + 1 < left ? zeta + 1 : left;
    const uint32_t w = (g * f * (f * f - 2u)) & (steps < 6 ? (1u << steps) - 1u : 63u);
    g += f * w;
    q += u * (int32_t)w;
    r += v * (int32_t)w;
  }
}

// x = d mod m, or -d (when f ended at -1).
__host__ __device__ __forceinline__ void s30_finish(const Signed30& d, bool neg, const uint32_t mw[8], uint32_t x[8]) {
  // d in (-12 m, 12 m): lift by 16 m, reduce by 16 m, 8 m, 4 m, 2 m, m.
  uint32_t w[9], km[5][9];
  s30_to_words(d, w);
#pragma unroll
  for (int k = 0; k < 5; ++k) {  // km[k] = 2^(4-k) m
    const int sh = 4 - k;
#pragma unroll
    for (int i = 0; i < 9; ++i) {
      const uint32_t hi = i < 8 ? mw[i] : 0u, lo = i > 0 ? mw[i - 1] : 0u;
      km[k][i] = sh ? (hi << sh) | (lo >> (32 - sh)) : hi;
    }
  }
  words9_add(w, km[0]);
#pragma unroll
  for (int k = 0; k < 5; ++k) words9_csub(w, km[k]);
  uint32_t z = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) z |= w[i];
  if (neg && z) {
    int64_t b = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      b += (int64_t)mw[i] - w[i];
      w[i] = (uint32_t)b;
      b >>= 32;
    }
  }
#pragma unroll
  for (int i = 0; i < 8; ++i) x[i] = w[i];
}

// x = A^-1 mod m for 0 < A < m (m odd, below 2^254); false if g did not reach
// 0 within the batch guard (unreachable for such inputs).
__host__ __device__ inline bool inverse_divsteps(const uint32_t A[8], const uint32_t mw[8], uint32_t x[8]) {
  uint32_t minv30 = 1;  // m^-1 mod 2^32 by Newton's iteration (each step doubles the correct bits)
#pragma unroll
  for (int i = 0; i < 5; ++i) minv30 *= 2u - mw[0] * minv30;
  minv30 &= 0x3fffffffu;
  const Signed30 m = s30_from_words(mw);
  Signed30 f = m, g = s30_from_words(A), d, e;
#pragma unroll
  for (int i = 0; i < 9; ++i) d.l[i] = e.l[i] = 0;
  e.l[0] = 1;
  int32_t zeta = -1;
  bool done = false;
  for (int batch = 0; batch < 24; ++batch) {
    int32_t any = 0;
#pragma unroll
    for (int i = 0; i < 9; ++i) any |= g.l[i];
    if (!any) {
      done = true;
      break;
    }
    const uint32_t fl = (uint32_t)f.l[0] | ((uint32_t)f.l[1] << 30), gl = (uint32_t)g.l[0] | ((uint32_t)g.l[1] << 30);
    int32_t u, v, q, r;
    divsteps30(fl, gl, zeta, u, v, q, r);
    s30_update_fg(f, g, u, v, q, r);
    s30_update_de(d, e, u, v, q, r, m, minv30);
  }
  s30_finish(d, f.l[8] < 0, mw, x);
  return done;
}

// Bit a kernel raises in its context's device flags when an inversion did not
// converge (the divsteps above end in fewer batches than their guard for
// every nonzero input below the modulus; the flag makes a broken invariant an
// error instead of a wrong value). The host reads it as DEV_INVERSE.
constexpr uint32_t kFlagInverse = 32u;

// 1/a for a in Montgomery form (0 for 0): the divsteps give A^-1 = a^-1 R^-1,
// and a^-1 R = A^-1 * R^3 (one Montgomery product with R^3 = R2 * R2 reduced
// once). `flags` (nullable) receives kFlagInverse if the batch guard ends it.
template <class C>
__device__ __noinline__ Fe<C> fe_inverse(const Fe<C>& a, uint32_t* flags = nullptr) {
  if (fe_is_zero(a)) return a;
  const uint32_t p[8] = {C::P0, C::P1, C::P2, C::P3, C::P4, C::P5, C::P6, C::P7};
  Fe<C> x;
  if (!inverse_divsteps(a.v, p, x.v) && flags) atomicOr(flags, kFlagInverse);
  Fe<C> r2;
#pragma unroll
  for (int i = 0; i < 8; ++i) r2.v[i] = C::R2(i);
  return fe_mul(x, fe_mul(r2, r2));
}

template <class C>
__device__ __forceinline__ Fe<C> ld_fe(const Fe<C>* p) {
  const uint4* q = reinterpret_cast<const uint4*>(p);
  uint4 x = q[0], y = q[1];
  Fe<C> r;
  r.v[0] = x.x; r.v[1] = x.y; r.v[2] = x.z; r.v[3] = x.w;
  r.v[4] = y.x; r.v[5] = y.y; r.v[6] = y.z; r.v[7] = y.w;
  return r;
}

template <class C>
__device__ __forceinline__ void st_fe(Fe<C>* p, const Fe<C>& a) {
  uint4* q = reinterpret_cast<uint4*>(p);
  q[0] = make_uint4(a.v[0], a.v[1], a.v[2], a.v[3]);
  q[1] = make_uint4(a.v[4], a.v[5], a.v[6], a.v[7]);
}

}  // namespace apg
