// Spectral step of the power-of-two column pass (column DCT-II spectrum -> scaling by
// -1/(4 H W lambda) -> DCT-III pre-twiddle).  The spectrum of the column pair sits in `sms`
// (natural order, padded addresses) and is overwritten in place by the pre-twiddled input of
// the inverse FFT.
#pragma once
#include "unw_regfft.cuh"
#include "unw_rowops.cuh"

template <int N>
__device__ __forceinline__ void col_spectral_k(float2* __restrict__ sms, int k, const float2* __restrict__ dw,
                                               const float* __restrict__ sH, float ca, float cb, bool ja0,
                                               bool hasb, float negs) {
    const int km = (N - k) & (N - 1);
    const float2 C = sms[pad16(k)], Cm = sms[pad16(km)];
    const float2 wk = __ldg(&dw[k]), wm = __ldg(&dw[km]);
    const float ck = __ldg(&sH[k]), cm = __ldg(&sH[km]);
    float2 ok, om;
    col_spectral_pair(C, Cm, k, km, wk, wm, ck, cm, ca, cb, ja0, hasb, negs, ok, om);
    if (km != k) sms[pad16(km)] = om;
    sms[pad16(k)] = ok;
}

// thread t owns the frequencies k = t + T i with their mirrors N - k: i < 8 for every thread
// (k < N/2) and k = N/2 for thread 0 alone.  The fixed trip count lets the table loads of the
// next frequencies issue before the current ones are used.
template <int N>
__device__ __forceinline__ void col_spectral_p2(float2* __restrict__ sms, int t, const float2* __restrict__ dw,
                                                const float* __restrict__ sH, float ca, float cb, bool ja0,
                                                bool hasb, float negs) {
    constexpr int T = N / 16;
#pragma unroll 2
    for (int i = 0; i < 8; i++) col_spectral_k<N>(sms, t + T * i, dw, sH, ca, cb, ja0, hasb, negs);
    if (t == 0) col_spectral_k<N>(sms, N / 2, dw, sH, ca, cb, ja0, hasb, negs);
}
