// Fixed-point arithmetic of the FS_FP64 element kernels.
//
// GB300 does 2 double operations per clock and SM but 64 multiply-adds of
// 32-bit integers into 64 bits, so the bilinear part of the element matrices
// (the expansion of the strain rows to the global dofs and the Gram product)
// runs on integers that hold more bits than a double's significand.
//
// A number is X 2^(E-58), X an integer of about 58 bits and sign, E an exponent
// shared by a group of numbers and above the largest of them: it is kept to
// 2^-58 of the group's largest, whose last bit in double is 2^-53 of it.  Numbers
// below 2^-5 of the largest thus keep fewer bits than in double; the groups are
// chosen so that this does not matter to their products (fs_elem_fixed.cuh).  X is
// split in two limbs, X = h 2^29 + l with |l| <= 2^28; a product keeps h h' (into
// one 64-bit sum) and h l' + l h' (into another), three multiply-adds, and drops
// l l' (below 2^-60 of the largest product).  A sum becomes an X again by one
// rounding, a double by another.
//
// The sums are exact while they fit 63 bits: products of X up to c 2^58 and c' 2^58
// may be up to 32 / (c c') of them.  Entries and products (triangle; quadrilateral,
// whose groups M, R and of layered dofs have a bit to spare): M below 2 and 3, 1 and
// 12; T 1.2 and 5, 20; R 1.42 and 5, 0.71 and 20; T R 8.6 and 17.1 in sum; layered
// 1 and 13, 0.5 and 33.  Largest: T of a quadrilateral, 28.8 of 32.
//
// Group exponents are far from a double's limits and all numbers finite: the
// kernels check this (fx_usable) and take their double path otherwise.
#pragma once

#include <math.h>
#include <stdint.h>
#include <string.h>

#ifndef FS_HD
#if defined(__CUDACC__)
#define FS_HD __host__ __device__ __forceinline__
#else
#define FS_HD inline
#endif
#endif

namespace fs {

constexpr int FX_LIMB = 29, FX_BITS = 2 * FX_LIMB;

struct fx {
    int32_t h, l;
};
struct FxSum {
    int64_t hh, c;
};

FS_HD uint32_t fx_hi(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2hiint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return (uint32_t)(u >> 32);
#endif
}
FS_HD uint32_t fx_lo(double x)
{
#if defined(__CUDA_ARCH__)
    return (uint32_t)__double2loint(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return (uint32_t)u;
#endif
}
FS_HD double fx_bits(uint64_t u)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((long long)u);
#else
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
FS_HD int fx_clz(uint32_t u)
{
#if defined(__CUDA_ARCH__)
    return __clz((int)u);
#else
    return u ? __builtin_clz(u) : 32;
#endif
}

// running maximum of magnitudes, as high words
FS_HD void fx_max(uint32_t &mx, double x)
{
    const uint32_t u = fx_hi(x) & 0x7fffffffu;
    mx = u > mx ? u : mx;
}
// the exponent of numbers that are not all zero: every |x| of them is below 2^E
FS_HD int fx_exp(uint32_t mx) { return (int)(mx >> 20) - 1022; }
// the group's exponent; of a group of zeros (a thickness or a material stiffness
// that vanishes) one at which they stay zeros
FS_HD int fx_group(uint32_t mx) { return mx ? fx_exp(mx) : 0; }
// finite, and products of four such groups are normal doubles to their last
// bit (a group of zeros counts as usable)
FS_HD bool fx_usable(uint32_t mx) { return mx < (uint32_t)(1023 + 200) << 20 && (mx == 0 || mx > (uint32_t)(1023 - 200) << 20); }

// X of x in a group of exponent E (towards zero); |x| = 2^E exactly (a unit
// vector's 1.0 in exponent 0) is taken too.  A zero is shifted out where E is
// above -960, as every group's exponent is
FS_HD int64_t fx_int(double x, int E)
{
    const uint32_t hi = fx_hi(x);
    const uint64_t m = ((uint64_t)((hi & 0xfffffu) | 0x100000u) << 32 | fx_lo(x)) << (FX_BITS - 52);
    int s = E + 1023 - (int)((hi >> 20) & 0x7ffu);
    s = s < 63 ? s : 63;
    const int64_t X = (int64_t)(m >> s);
    return (int32_t)hi < 0 ? -X : X;
}
FS_HD fx fx_split(int64_t X)
{
    fx r;
    r.h = (int32_t)((X + (1 << (FX_LIMB - 1))) >> FX_LIMB);
    r.l = (int32_t)((uint32_t)X - ((uint32_t)r.h << FX_LIMB));
#if defined(__CUDA_ARCH__)
    // a limb is 32 bits to the compiler, not a shifted 64-bit number whose
    // products it would widen (a 64-bit product is five instructions, not one)
    asm("" : "+r"(r.h), "+r"(r.l));
#endif
    return r;
}
FS_HD fx fx_make(double x, int E) { return fx_split(fx_int(x, E)); }
FS_HD fx fx_neg(fx a) { return fx{-a.h, -a.l}; }

FS_HD void fx_mac(FxSum &s, fx a, fx b)
{
    s.hh += (int64_t)a.h * b.h;
    s.c += (int64_t)a.h * b.l;
    s.c += (int64_t)a.l * b.h;
}
FS_HD FxSum fx_mul(fx a, fx b)
{
    FxSum s;
    s.hh = (int64_t)a.h * b.h;
    s.c = (int64_t)a.h * b.l;
    s.c += (int64_t)a.l * b.h;
    return s;
}
// X of a sum of products, in the product of their groups' exponents (downwards)
FS_HD int64_t fx_round(FxSum s) { return s.hh + (s.c >> FX_LIMB); }
FS_HD fx fx_done(FxSum s) { return fx_split(fx_round(s)); }

// X in an exponent larger by s >= 0
FS_HD int64_t fx_shift(int64_t X, int s) { return X >> (s < 63 ? s : 63); }

// the double nearest (ties away) to X 2^(E-58), E the products' exponent
FS_HD double fx_double(FxSum s, int E)
{
    const int64_t X = fx_round(s), sg = X >> 63;
    const uint64_t u = (uint64_t)((X ^ sg) - sg);
    const bool low = (u >> 32) == 0;
    const uint32_t uh = low ? (uint32_t)u : (uint32_t)(u >> 32), ul = low ? 0u : (uint32_t)u;
    // exponent field of a leading bit 63, less one for that bit
    const int lead = E - FX_BITS + 63 + 1022 - (low ? 32 : 0);
    const int sh = fx_clz(uh) & 31;
    const uint64_t m = ((uint64_t)uh << 32 | ul) << sh;
    // 53 bits and the next one as a carry; the leading bit adds one to the exponent
    const uint64_t r = (m >> 11) + ((uint32_t)m >> 10 & 1u) + ((uint64_t)(uint32_t)(lead - sh) << 52);
    return fx_bits(uh == 0 ? 0ull : r | ((uint64_t)sg & 0x8000000000000000ull));
}

}  // namespace fs
