// fixed.cuh -- complex arithmetic in 64-bit fixed point (gebrd.cu, bdapply.cu).
//
// One FP64 instruction of a warp takes 17 cycles of its SM (0.5 lanes per clock and
// scheduler), one 32 x 32 + 64 bit integer multiply-add 1.1.  A product of two 62-bit
// numbers is three of the latter: high x high, and the two cross terms with 28 bits of
// the low halves; what is left out is below 2^-58 of the factors' ranges, of either sign.
#pragma once
#include <cuda_runtime.h>

namespace tebd {
namespace {

// A fixed-point number x in memory: x + 8 as hi 2^32 + lo with lo signed, so that hi and
// lo >> 4 are x rounded to 28 bits below hi.  A complex one is (re lo, re hi, im lo, im hi).
__device__ __forceinline__ int2 enc(long long x) {
  const long long y = x + 8;
  return make_int2((int)y, (int)((y + 0x80000000ll) >> 32));
}
__device__ __forceinline__ long long dec(int lo, int hi) { return (((long long)hi << 32) + lo) - 8; }
__device__ __forceinline__ int4 enc2(long long re, long long im) {
  const int2 a = enc(re), b = enc(im);
  return make_int4(a.x, a.y, b.x, b.y);
}
// a vector entry for the products: (re hi, re lo >> 4, im hi, im lo >> 4)
__device__ __forceinline__ int4 vec_entry(long long re, long long im) {
  const int4 e = enc2(re, im);
  return make_int4(e.y, e.x >> 4, e.w, e.z >> 4);
}

// x 2^sh rounded to an integer, |x| 2^sh < 2^63, in integer instructions (the FP64
// pipe, at 16 cycles per warp instruction, is what the kernel must spare)
__device__ __forceinline__ long long to_fix(double x, int sh) {
  const long long b = __double_as_longlong(x);
  const int e = (int)((b >> 52) & 0x7ff);
  const long long m = (b & 0xfffffffffffffll) | 0x10000000000000ll;
  const int s = e - 1075 + sh;
  long long r = s >= 0 ? m << min(s, 10) : (s > -54 ? (m + (1ll << (-s - 1))) >> (-s) : 0ll);
  if (e == 0) r = 0;
  return b < 0 ? -r : r;
}

// 2^k as a double, -1022 <= k <= 1023
__device__ __forceinline__ double pow2(int k) { return __longlong_as_double((long long)(k + 1023) << 52); }

__device__ __forceinline__ void mw(long long &acc, int a, int b) { acc += (long long)a * b; }  // one IMAD.WIDE

// A sum in halves: h of the high x high products, x of the cross terms
struct Acc {
  long long hr = 0, hi = 0, xr = 0, xi = 0;
  // += a v: `a` as stored, v a vector entry, nh, nl the negatives of v.z, v.w
  __device__ __forceinline__ void add(const int4 &a, const int4 &v, int nh, int nl) {
    const int arl = a.x >> 4, ail = a.z >> 4;
    mw(hr, a.y, v.x);
    mw(hr, a.w, nh);
    mw(hi, a.y, v.z);
    mw(hi, a.w, v.x);
    mw(xr, a.y, v.y);
    mw(xr, arl, v.x);
    mw(xr, a.w, nl);
    mw(xr, ail, nh);
    mw(xi, a.y, v.w);
    mw(xi, arl, v.z);
    mw(xi, a.w, v.y);
    mw(xi, ail, v.x);
  }
  // += conj(a) v: nh, nl the negatives of v.x, v.y
  __device__ __forceinline__ void add_conj(const int4 &a, const int4 &v, int nh, int nl) {
    const int arl = a.x >> 4, ail = a.z >> 4;
    mw(hr, a.y, v.x);
    mw(hr, a.w, v.z);
    mw(hi, a.y, v.z);
    mw(hi, a.w, nh);
    mw(xr, a.y, v.y);
    mw(xr, arl, v.x);
    mw(xr, a.w, v.w);
    mw(xr, ail, v.z);
    mw(xi, a.y, v.w);
    mw(xi, arl, v.z);
    mw(xi, a.w, nl);
    mw(xi, ail, nh);
  }
  // in units of 2^(64 - kUp) times the factors' own (h has 2^64, x 2^36)
  template <int kUp>
  __device__ __forceinline__ longlong2 value() const {
    constexpr int dn = 28 - kUp;
    constexpr long long half = 1ll << (dn - 1);
    return make_longlong2((long long)((unsigned long long)hr << kUp) + ((xr + half) >> dn),
                          (long long)((unsigned long long)hi << kUp) + ((xi + half) >> dn));
  }
};

}  // namespace
}  // namespace tebd
