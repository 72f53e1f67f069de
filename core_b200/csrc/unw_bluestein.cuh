// Length-N DFT for lengths that are not powers of two, by Bluestein's chirp-z
// algorithm (L. Bluestein, IEEE Trans. Audio Electroacoust. 18(4), 1970) on the
// register radix-16 FFT of a power-of-two length M >= 2N - 1:
//   X_k = conj(c_k) * sum_m (x_m conj(c_m)) c_{k-m},  c_m = exp(i pi m^2 / N),
// the convolution done as FFT_M, a product with the precomputed spectrum of the
// chirp filter (scaled by 1/M), and a second forward FFT of the conjugate.
// Every DCT pass of a non-power-of-two axis runs on this, so those axes use
// the same conflict-free register/shared-memory FFT as the power-of-two ones.
#pragma once
#include "unw_regfft.cuh"

// Both transforms run with their ends in registers: the zero-padded input goes from shared memory
// straight into the first pass, the filter spectrum multiplies the last pass's registers, which are
// the second transform's input as they stand, and the chirp of the result is applied on the way
// out.  (The caller applies the input's chirp as it writes x.)  Against separate loops over shared
// memory for the two chirps and the filter: 40% fewer shared-memory accesses and a third
// fewer barriers.  What bounds the passes now is latency at about 24 warps per SM (issue slots 50% busy,
// 88 instructions per point of which half are the transforms' arithmetic).

// x_m conj(c_m) in sm[pad16(m)], m < N (written and synchronised by the caller) ->
// X_k in sm[pad16(k)], k < N, synchronised on return.  M / 16 threads per
// sequence, t = this thread's index within its sequence; every thread of the
// CTA must call (the FFT passes synchronise the CTA).  N <= M / 2.
//
// From M = 8192 on the registers that this needs cost a resident CTA, or spill at 1024 threads: there
// the transforms run from and to shared memory with loops for the padding, the filter and the
// chirp.  Row-forward / row-inverse pass, us per launch, fused and not: 200 x 180 (M = 512)
// 15.0 / 11.7 and 16.9 / 13.1; 560 x 700 (1536) 17.6 / 15.1 and 19.1 / 15.4; 1500 x 2001 (4096)
// 42.4 / 32.7 and 43.4 / 34.2; 1838 x 2750 (6144) 82.9 / 67.2 and 83.7 / 69.4; 2000 x 5500 (12288)
// 174 / 153 and 183 / 164; but 1500 x 3900 (8192) 90.6 / 78.0 and 86.3 / 71.4, 500 x 8000 (16384)
// 72.4 / 58.6 and 65.9 / 56.1.  Times three a power of two is always fused.
template <int M>
constexpr bool blue_fused() { return M < 8192; }

template <int M>
__device__ __forceinline__ void blue_fft(float2* __restrict__ sm, int t, int N, const DctPlanDev& P) {
    constexpr int T = M / 16;
    const float2* __restrict__ ch = P.chirp;
    const float2* __restrict__ hs = P.hspec;
    if constexpr (!blue_fused<M>()) {
        for (int m = t; m < M; m += T)
            if (m >= N) sm[pad16(m)] = make_float2(0.f, 0.f);
        __syncthreads();
        smem_fft<M>(sm, t, P.fft.tw);
        for (int m = t; m < M; m += T) {
            const int a = pad16(m);
            sm[a] = cconj(cmul(sm[a], __ldg(&hs[m])));
        }
        __syncthreads();
        smem_fft<M>(sm, t, P.fft.tw);
        for (int k = t; k < N; k += T) {
            const int a = pad16(k);
            sm[a] = cmul(cconj(sm[a]), cconj(__ldg(&ch[k])));
        }
    } else {
        float2 v[16];
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const int m = t + T * q;
            v[q] = make_float2(0.f, 0.f);
            if (q < 8 && m < N) v[q] = sm[pad16(m)];
        }
        __syncthreads();  // every input read before the first pass writes
        io_fft<M, true, true>(v, sm, t, P.fft.tw);
#pragma unroll
        for (int q = 0; q < 16; q++) v[q] = cconj(cmul(v[q], __ldg(&hs[t + T * q])));
        io_fft<M, true, true>(v, sm, t, P.fft.tw);
#pragma unroll
        for (int q = 0; q < 8; q++) {
            const int k = t + T * q;
            if (k < N) sm[pad16(k)] = cmul(cconj(v[q]), cconj(__ldg(&ch[k])));
        }
    }
    __syncthreads();
}

// Bluestein length M = 3 * M3 (M3 a power of two >= 256, N <= 3 M3 / 2).  The two length-M FFTs
// are split into a radix-3 stage and three register FFTs of length M3, one per third of the
// CTA, so that no permutation pass is needed:
//   FFT 1, decimation in frequency: radix-3 butterflies across the thirds of the input (the last one is
//     zero) with twiddles W_M^{s m}, formed by each third as it loads -> third s holds
//     X_{3k+s} at index k;
//   the filter spectrum is applied in that order (its table is stored [s][k]);
//   FFT 2, decimation in time: third r holds the sub-sequence x_{3m+r}, the same registers ->
//     three FFTs of length M3, twiddles W_M^{r k}, radix-3 butterflies through shared memory ->
//     natural order.
template <int M3>
__device__ __forceinline__ void blue_fft3(float2* __restrict__ sm, int t, int N, const DctPlanDev& P) {
    constexpr int T3 = M3 / 16, T = 3 * T3;
    constexpr int R = RegFft<M3>::SEQ_STRIDE;      // slots per third
    const float2* __restrict__ ch = P.chirp;
    const float2* __restrict__ tw = P.fft.tw;       // exp(-2 pi i m / M), m < M
    const int grp = t / T3, tt = t - grp * T3;
    const float2* __restrict__ hs = P.hspec + grp * M3;
    float2* const smg = sm + grp * R;
    const float h = 0.86602540378443865f;           // sqrt(3)/2
    const float2 wg = grp == 0 ? make_float2(1.f, 0.f) : make_float2(-0.5f, grp == 1 ? -h : h);
    float2 v[16];
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const int m = tt + T3 * q;
        float2 a = m < N ? sm[pad16(m)] : make_float2(0.f, 0.f);
        if (m + M3 < N) {
            const float2 b = cmul(sm[R + pad16(m)], wg);
            a = make_float2(a.x + b.x, a.y + b.y);
        }
        v[q] = grp ? cmul(a, __ldg(&tw[grp * m])) : a;
    }
    __syncthreads();  // every input read before the first pass writes
    io_fft<M3, true, true, 3>(v, smg, tt, tw);
#pragma unroll
    for (int q = 0; q < 16; q++) v[q] = cconj(cmul(v[q], __ldg(&hs[tt + T3 * q])));
    io_fft<M3, true, true, 3>(v, smg, tt, tw);
#pragma unroll
    for (int q = 0; q < 16; q++) {
        const int k = tt + T3 * q;
        smg[pad16(k)] = grp ? cmul(v[q], __ldg(&tw[grp * k])) : v[q];
    }
    __syncthreads();
    for (int k = t; k < M3; k += T) {
        const int a = pad16(k);
        const float2 y0 = sm[a], y1 = sm[R + a], y2 = sm[2 * R + a];
        const float2 s = make_float2(y1.x + y2.x, y1.y + y2.y);
        if (k < N) sm[a] = cmul(make_float2(y0.x + s.x, -(y0.y + s.y)), cconj(__ldg(&ch[k])));
        if (k + M3 < N) {
            // y0 - s/2 - i sqrt(3)/2 (y1 - y2), conjugated
            const float re = (y0.x - 0.5f * s.x) + h * (y1.y - y2.y);
            const float im = (y0.y - 0.5f * s.y) - h * (y1.x - y2.x);
            sm[R + a] = cmul(make_float2(re, -im), cconj(__ldg(&ch[k + M3])));
        }
    }
    __syncthreads();
}

// The two Bluestein FFT shapes as one interface for the DCT kernels:
// threads per sequence, shared-memory slots per sequence (with the bank offset
// between sequences), the slot of natural index m, and the length-N DFT of the
// chirped input.
template <int M>
struct BlP2 {
    static constexpr int LEN = M;
    static constexpr bool FUSED = blue_fused<M>();
    static constexpr int T = M / 16;
    static constexpr int SLOTS = RegFft<M>::SEQ_STRIDE;
    static __device__ __forceinline__ int pos(int m) { return pad16(m); }
    static __device__ __forceinline__ void dft(float2* sm, int t, int N, const DctPlanDev& P) {
        blue_fft<M>(sm, t, N, P);
    }
};

template <int M3>
struct BlMix3 {
    static constexpr int LEN = 3 * M3;
    static constexpr bool FUSED = true;
    static constexpr int T = 3 * (M3 / 16);
    static constexpr int R = RegFft<M3>::SEQ_STRIDE;
    static constexpr int SLOTS = 3 * R;
    static constexpr int L3 = ilog2c(M3);
    static __device__ __forceinline__ int pos(int m) { return (m >> L3) * R + pad16(m & (M3 - 1)); }
    static __device__ __forceinline__ void dft(float2* sm, int t, int N, const DctPlanDev& P) {
        blue_fft3<M3>(sm, t, N, P);
    }
};
