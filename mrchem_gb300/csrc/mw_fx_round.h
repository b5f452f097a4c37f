// mw_fx_round.h -- shifts of the 62-bit fixed-point numbers of mw_apply_fx.cu, for the GPU and for host tests
#pragma once

#if defined(__CUDACC__)
#define FX_HD __host__ __device__ __forceinline__
#else
#define FX_HD inline
#endif

namespace mwg {

// v 2^-s, rounded to nearest (halves up), |v| <= 2^62, s >= 0.  A truncation would be a bias that adds up over the
// items.  The count stops at 62, where the rounding term 2^61 still makes zero of every |v| < 2^61: with
// (1 << 63) >> 1 = -2^62 a zero came out as -1.
FX_HD long long fx_round(long long v, int s) {
    s = s < 62 ? s : 62;
    return (v + ((1ll << s) >> 1)) >> s;
}

}  // namespace mwg
