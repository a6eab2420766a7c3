// 32-bit numbers on the 16-bit tensor cores: a float as the sum of three bfloat16 numbers, high to low.
#pragma once

#include "common.cuh"

// Two floats -> (h, m, l) pairs of bfloat16, each part rounded: what the three leave of a float is below 2^-26 of it, and a
// product of two numbers taken apart this way lacks less than a float's rounding when h h', h m', m h', m m', h l' and l h' are
// summed. (The high part of a float above bfloat16's largest number is infinite.)
__device__ __forceinline__ void take_apart(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    const __nv_bfloat162 hh = __floats2bfloat162_rn(a, b);
    h = *reinterpret_cast<const uint32_t*>(&hh);
    const float ra = a - __uint_as_float(h << 16), rb = b - __uint_as_float(h & 0xffff0000u);
    const __nv_bfloat162 mm = __floats2bfloat162_rn(ra, rb);
    m = *reinterpret_cast<const uint32_t*>(&mm);
    const __nv_bfloat162 ll = __floats2bfloat162_rn(ra - __uint_as_float(m << 16), rb - __uint_as_float(m & 0xffff0000u));
    l = *reinterpret_cast<const uint32_t*>(&ll);
}

// The same cut off instead of rounded: the three parts are exactly the float, the largest ones included (what is not finite
// stays so in their sum). For products with 16-bit numbers, which take all three, and beside a number taken apart by rounding.
__device__ __forceinline__ void cut_apart(float a, float b, uint32_t& h, uint32_t& m, uint32_t& l) {
    h = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
    const float ra = a - __uint_as_float(h << 16), rb = b - __uint_as_float(h & 0xffff0000u);
    m = __byte_perm(__float_as_uint(ra), __float_as_uint(rb), 0x7632);
    const float sa = ra - __uint_as_float(m << 16), sb = rb - __uint_as_float(m & 0xffff0000u);
    l = __byte_perm(__float_as_uint(sa), __float_as_uint(sb), 0x7632);
}
