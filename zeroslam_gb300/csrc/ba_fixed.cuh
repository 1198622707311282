// Fixed-point numbers for products on the integer pipe: a value v scaled by a
// power of two is q = round(v 2^sh), q = a1 2^kFxLow + a0 with a0 in
// [-2^(kFxLow-1), 2^(kFxLow-1)), held as (a0, a1). A product is then four
// 32-bit multiply-adds: a1 b1, a1 b0 + a0 b1, and the upper half of a0 b0.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace zs {
namespace fixed {

using ll = long long;

constexpr int kLow = 30;  // bits of a0

// 2^p as a double, p in [-1022, 1023].
__device__ __forceinline__ double pow2(int p) { return __longlong_as_double((ll)(p + 1023) << 52); }

// e with |v| < 2^e (and >= 2^(e - 1) where v is normal): -4096 for 0, 1025 for
// values that are not finite.
__device__ __forceinline__ int exponent(double v) {
    const ll bits = __double_as_longlong(v) & 0x7fffffffffffffffll;
    return bits ? (int)(bits >> 52) - 1022 : -4096;
}

// round(v 2^sh) to nearest; where that is above most or not finite, bad is set.
__device__ __forceinline__ ll quantize(double v, int sh, ll most, int& bad) {
    const ll bits = __double_as_longlong(v);
    const int ex = (int)((bits >> 52) & 0x7ff);
    const ll m = (bits & ((1ll << 52) - 1)) | (ex ? 1ll << 52 : 0);
    const int s = (ex ? ex : 1) - 1075 + sh;  // v 2^sh = m 2^s
    ll q;
    if (s >= 0) {
        q = m << min(s, 10);
    } else {
        q = s > -55 ? (m + (1ll << (-s - 1))) >> -s : 0;
    }
    if (ex == 0x7ff || q > most) bad = 1;
    return bits < 0 ? -q : q;
}

__device__ __forceinline__ int2 split(ll q) {
    const ll a1 = (q + (1ll << (kLow - 1))) >> kLow;
    return make_int2((int)(q - (a1 << kLow)), (int)a1);
}

// x 2^s, s of either sign (to nearest below zero).
__device__ __forceinline__ ll shift(ll x, int s) {
    if (s >= 0) return x << min(s, 63);
    return s > -63 ? (x + (1ll << (-s - 1))) >> -s : 0;
}

}  // namespace fixed
}  // namespace zs
