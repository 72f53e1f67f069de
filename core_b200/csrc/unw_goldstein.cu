// Goldstein adaptive phase filter, the code path insardev runs on CUDA devices
// (goldstein_pytorch, insardev/insardev/utils_goldstein.py:157-330):
// overlapping psize_y x psize_x patches at half-patch steps, each patch's 2-D
// spectrum weighted by max(|F|, 1e-10)^alpha with alpha = 1 - weighted mean
// coherence, inverse transform, triangular taper, overlap-add, division by the
// number of valid patches covering a pixel.
//
// A group of px threads owns one column of patches and walks down it: thread c holds column c of
// the current patch in registers, so loads and stores are whole rows of the group.  Transforms
// are in registers, along y with a thread per column and along x with a thread per row, with one
// exchange through shared memory each way; forward transforms leave bit-reversed order and inverse ones
// take it (the spectrum weight does not depend on position), so nothing is reordered.
// A pixel is covered by 2 x 2 patches: the lower half of a patch stays in registers for the next
// patch of the walk, the right half goes to the neighbouring group through shared memory, and
// each finished half-patch cell is normalised and written once.  No accumulator in global memory,
// one launch, deterministic.
//
// What bounds it (B200): instruction issue at two CTAs per SM (128 registers a thread): 3700 warp
// instructions per 32 x 32 patch at 2.3 per cycle, DRAM at 5%.  2048 x 2048 with 32 x 32 patches takes 154 us
// (traffic alone 13 us); the earlier form, radix-2 passes through shared memory with a sincospi per
// butterfly, four launches and an accumulator in global memory, 765 us.  1001 x 1203 with 16 x 16:
// 39 us, before 280.  Butterflies as packed additions: 154 us against 166 with scalar ones.
#include <cuda_runtime.h>
#include <stdint.h>
#include <math.h>
#include <algorithm>

#include "../../include/unwrap_b200.h"
#include "unw_kernels.h"

namespace {

struct GsArgs {
    const float2* phase; long long pp;
    const float* corr; long long cp;
    int ny, nx;             // input grid
    int npy, npx;           // patches per axis
    int seg;                // cell rows per CTA
    int min_valid;
    float2* out; long long op;
};

// Taper (utils_goldstein.py:198-203): separable tent over half a patch, built in
// float64 and rounded once.
template <int PY, int PX>
__device__ __forceinline__ float gs_taper(int y, int x) {
    const int qy = y < PY / 2 ? y : PY - 1 - y;   // mirrored quadrant index
    const int qx = x < PX / 2 ? x : PX - 1 - x;
    constexpr double cy = PY / 2.0 - 1.0, cx = PX / 2.0 - 1.0;
    const double wy = 1.0 - fabs((double)qy - cy) / cy;
    const double wx = 1.0 - fabs((double)qx - cx) / cx;
    return (float)(wy * wx);
}

// exp(-2 pi i k / n) for n <= 64
constexpr float gs_quarter(int k) {  // cos(2 pi k / 64), k <= 16
    constexpr float t[17] = {
    1.f, 0.99518472667219693f, 0.98078528040323045f, 0.95694033573220887f, 0.92387953251128676f,
    0.88192126434835503f, 0.83146961230254524f, 0.77301045336273697f, 0.70710678118654752f,
    0.63439328416364550f, 0.55557023301960222f, 0.47139673682599765f, 0.38268343236508977f,
    0.29028467725446236f, 0.19509032201612827f, 0.09801714032956060f, 0.f};
    return t[k];
}
constexpr float gs_cos(int k64) {  // cos(2 pi k / 64)
    k64 &= 63;
    if (k64 > 32) k64 = 64 - k64;
    return k64 <= 16 ? gs_quarter(k64) : -gs_quarter(32 - k64);
}
constexpr float gs_sin(int k64) { return gs_cos(k64 - 16); }

// a * exp(-+2 pi i K / N) (INV: +)
template <int N, int K, bool INV>
__device__ __forceinline__ float2 gs_tw(float2 a) {
    constexpr int k = K * (64 / N);
    if constexpr (k == 0) return a;
    else if constexpr (k == 16) return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
    else {
        constexpr float c = gs_cos(k), s = INV ? gs_sin(k) : -gs_sin(k);
        return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
    }
}

// Forward transform, natural order in, bit-reversed out (decimation in frequency).
template <int N, int K>
__device__ __forceinline__ void gs_dif_bf(float2* v) {
    if constexpr (K < N / 2) {
        const float2 a = v[K], b = v[K + N / 2];
        v[K] = add2(a, b);
        v[K + N / 2] = gs_tw<N, K, false>(sub2(a, b));
        gs_dif_bf<N, K + 1>(v);
    }
}
template <int N>
__device__ __forceinline__ void gs_dif(float2* v) {
    if constexpr (N > 1) {
        gs_dif_bf<N, 0>(v);
        gs_dif<N / 2>(v);
        gs_dif<N / 2>(v + N / 2);
    }
}
// Inverse transform (not scaled), bit-reversed in, natural order out (decimation in time).
template <int N, int K>
__device__ __forceinline__ void gs_dit_bf(float2* v) {
    if constexpr (K < N / 2) {
        const float2 a = v[K], b = gs_tw<N, K, true>(v[K + N / 2]);
        v[K] = add2(a, b);
        v[K + N / 2] = sub2(a, b);
        gs_dit_bf<N, K + 1>(v);
    }
}
template <int N>
__device__ __forceinline__ void gs_dit(float2* v) {
    if constexpr (N > 1) {
        gs_dit<N / 2>(v);
        gs_dit<N / 2>(v + N / 2);
        gs_dit_bf<N, 0>(v);
    }
}

// F * max(|F|, 1e-10)^alpha, t = alpha / 2, as 2^(t log2 |F|^2) with the argument split into an integer and a
// rest (W. J. Cody and W. Waite, Software Manual for the Elementary Functions, 1980, the chapter on x**y;
// rounding to the nearest integer by adding 1.5 * 2^23): |F|^2 = 2^e f with sqrt(1/2) <= f < sqrt(2), t e =
// n + rest, the rest exact by the fma.  The units' log2 and exp2 only see |log2 f| <= 1/2 and a power within
// [-1, 1], so their error (2^-22.6 absolute of log2 f, times |t| <= 1; 2^-22 of exp2) does not grow with
// |F|.  Measured against 64 bits over a filtered grid: 1.7e-7, with powf(sqrtf) 1.8e-7.
// For |t| <= 1 and |F.x|, |F.y| < 2^62: |F|^2 <= 2^125, so that 2^n is a normal number.
__device__ __forceinline__ float2 gs_weight(float2 F, float t) {
    constexpr float magic = 12582912.f;                     // 1.5 * 2^23: integers in the low bits
    const float m2 = fmaxf(fmaf(F.x, F.x, F.y * F.y), 1e-20f);
    const int e = (__float_as_int(m2) - 0x3f3504f3) >> 23;  // mantissa in [0.707, 1.414)
    const float f = __int_as_float(__float_as_int(m2) - (e << 23));
    const float fe = __int_as_float(0x4b400000 + e) - magic;
    const float nm = fmaf(t, fe, magic), n = nm - magic;
    float l, x;
    asm("lg2.approx.f32 %0, %1;" : "=f"(l) : "f"(f));
    asm("ex2.approx.f32 %0, %1;" : "=f"(x) : "f"(fmaf(t, l, fmaf(t, fe, -n))));
    const float s = x * __int_as_float((__float_as_int(nm) << 23) + 0x3f800000);
    return mul2(F, make_float2(s, s));
}
// The same for any alpha (coherence outside [-1, 3]) and any |F| (scaled by a power of two where its square
// would overflow).
constexpr float GS_BIG = 4611686018427387904.f;             // 2^62
__device__ __noinline__ float gs_pow(float2 F, float alpha) {
    const bool big = fmaxf(fabsf(F.x), fabsf(F.y)) >= GS_BIG;
    if (big) F = make_float2(F.x * 0x1p-66f, F.y * 0x1p-66f);
    const float m = sqrtf(F.x * F.x + F.y * F.y);
    return powf(fmaxf(big ? m * 0x1p66f : m, 1e-10f), alpha);
}

__device__ __noinline__ float2 gs_third(float2 s) { return make_float2(s.x / 3.f, s.y / 3.f); }

__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// PX threads per patch.  Patches of at most 32 columns lie inside a warp.
template <int PX>
__device__ __forceinline__ void gs_sync() {
    if (PX <= 32) __syncwarp();
    else __syncthreads();
}

template <int PY, int PX>
struct GsShape {
    static constexpr int NT = 256, NS = NT / PX;           // threads, patch columns per CTA
    static constexpr int SY = PY / 2, SX = PX / 2;
    static constexpr int TILE = PY * (PX + 1);             // one padding slot per row
    static constexpr size_t SMEM = sizeof(float2) * ((size_t)NS * TILE + 2 * (size_t)NS * SY * SX) +
                                   sizeof(float) * (size_t)PY * PX;
    static constexpr int CTAS = PY <= 32 ? 2 : 1;          // per SM, by registers
};

template <int PY, int PX>
__global__ void __launch_bounds__(256, (GsShape<PY, PX>::CTAS)) k_gs_walk(GsArgs a) {
    using S = GsShape<PY, PX>;
    constexpr int NS = S::NS, SY = S::SY, SX = S::SX;
    extern __shared__ float2 gs_sm[];
    float2* const tile = gs_sm + (size_t)(threadIdx.x / PX) * S::TILE;
    float2* const exch = gs_sm + (size_t)NS * S::TILE;               // [2][NS][SY][SX]
    float* const wgt = reinterpret_cast<float*>(exch + 2 * NS * SY * SX);
    __shared__ int cover[2][NS];          // valid patches of a slot over the current cell row
    __shared__ float rw[8];
    __shared__ int rv[8];
    const int slot = threadIdx.x / PX, c = threadIdx.x % PX;
    // taper, and its sum in float64 rounded once
    __shared__ double red[32];
    double ws[1] = {0.0};
    for (int e = threadIdx.x; e < PY * PX; e += 256) {
        wgt[e] = gs_taper<PY, PX>(e / PX, e % PX);
        ws[0] += (double)wgt[e];
    }
    block_sum<1>(ws, red);
    if (threadIdx.x == 0) red[0] = ws[0];
    __syncthreads();
    const float wsum = (float)red[0];
    constexpr float inv_n = 1.0f / (float)(PY * PX);
    // slot s walks patch column pj; it finishes the cells below its left half with the slot before it
    const int pj = blockIdx.x * (NS - 1) + slot - 1;
    const int x = pj * SX + c;
    const int i0 = blockIdx.y * a.seg, i1 = min(i0 + a.seg, (a.ny + SY - 1) / SY);
    const bool col = pj >= 0 && pj < a.npx;
    float2 carry[SY];
#pragma unroll
    for (int r = 0; r < SY; r++) carry[r] = make_float2(0.f, 0.f);
    int before = 0, buf = 0;
    for (int pi = i0 - 1; pi < i1; pi++) {
        const int y0 = pi * SY;
        // load (outside the grid and NaN -> 0; utils_goldstein.py:214-230), coherence, valid pixels
        float2 v[PY];
        unsigned nan = 0u;                 // NaN pixels of the upper half
        float wc = 0.f;
        int vc = 0;
        const int rows = col && pi >= 0 && x < a.nx ? a.ny - y0 : 0;   // of this column, from y0 on
        const float2* ph = a.phase + (long long)y0 * a.pp + x;
        const float* co = a.corr + (long long)y0 * a.cp + x;
        // all loads of a kind together: the coherence is reduced before the phase takes its registers
        {
            float k[PY];
#pragma unroll
            for (int r = 0; r < PY; r++) k[r] = r < rows ? co[(long long)r * a.cp] : 0.f;
#pragma unroll
            for (int r = 0; r < PY; r++) wc = fmaf(wgt[r * PX + c], isnan(k[r]) ? 0.f : k[r], wc);
        }
#pragma unroll
        for (int r = 0; r < PY; r++) v[r] = r < rows ? ph[(long long)r * a.pp] : make_float2(0.f, 0.f);
        // the rows that the next patch adds start towards L2
        if (PY + SY <= rows) {
            for (int q = c; q < SY; q += PX) {
                const int x0 = pj * SX;
                prefetch_l2(a.phase + (long long)(y0 + PY + q) * a.pp + x0);
                prefetch_l2(a.corr + (long long)(y0 + PY + q) * a.cp + x0);
            }
        }
        vc = max(0, min(rows, PY));
#pragma unroll
        for (int r = 0; r < PY; r++) {
            const bool bad = isnan(v[r].x) || isnan(v[r].y);
            if (bad) {
                v[r] = make_float2(0.f, 0.f);
                vc--;
                if (r < SY) nan |= 1u << r;
            }
        }
        // sums over the patch's threads
#pragma unroll
        for (int o = (PX < 32 ? PX : 32) / 2; o > 0; o >>= 1) {
            wc += __shfl_xor_sync(0xffffffffu, wc, o);
            vc += __shfl_xor_sync(0xffffffffu, vc, o);
        }
        if (PX > 32) {
            const int w = threadIdx.x >> 5;
            if ((threadIdx.x & 31) == 0) { rw[w] = wc; rv[w] = vc; }
            __syncthreads();
            wc = rw[w & ~1] + rw[w | 1];
            vc = rv[w & ~1] + rv[w | 1];
        }
        const float alpha = 1.0f - wc / wsum;                          // utils_goldstein.py:259-262
        const bool valid = col && pi >= 0 && pi < a.npy && vc >= a.min_valid;  // :264-267
        const bool work = PX <= 32 ? __any_sync(0xffffffffu, valid) : __syncthreads_or(valid);
        if (work) {
            gs_dif<PY>(v);
#pragma unroll
            for (int r = 0; r < PY; r++) tile[r * (PX + 1) + c] = v[r];
            gs_sync<PX>();
            for (int r = c; r < PY; r += PX) {
                float2 u[PX];
#pragma unroll
                for (int k = 0; k < PX; k++) u[k] = tile[r * (PX + 1) + k];
                gs_dif<PX>(u);
                // spectrum weight (:270-276)
                float top = 0.f;
#pragma unroll
                for (int k = 0; k < PX; k++) top = fmaxf(top, fmaxf(fabsf(u[k].x), fabsf(u[k].y)));
                if (fabsf(alpha) <= 2.f && top < GS_BIG) {
#pragma unroll
                    for (int k = 0; k < PX; k++) u[k] = gs_weight(u[k], 0.5f * alpha);
                } else {
#pragma unroll
                    for (int k = 0; k < PX; k++) {
                        const float q = gs_pow(u[k], alpha);
                        u[k] = make_float2(u[k].x * q, u[k].y * q);
                    }
                }
                gs_dit<PX>(u);
#pragma unroll
                for (int k = 0; k < PX; k++) tile[r * (PX + 1) + k] = u[k];
            }
            gs_sync<PX>();
#pragma unroll
            for (int r = 0; r < PY; r++) v[r] = tile[r * (PX + 1) + c];
            gs_sync<PX>();  // read before the next patch overwrites it
            gs_dit<PY>(v);
        }
        // taper and overlap-add (:283-307): the upper half is complete along y
        float2 tot[SY];
        if (valid) {
#pragma unroll
            for (int r = 0; r < SY; r++) {
                const float w0 = wgt[r * PX + c] * inv_n, w1 = wgt[(r + SY) * PX + c] * inv_n;
                tot[r] = fma2(make_float2(w0, w0), v[r], carry[r]);
                carry[r] = mul2(make_float2(w1, w1), v[r + SY]);
            }
        } else {
#pragma unroll
            for (int r = 0; r < SY; r++) {
                tot[r] = carry[r];
                carry[r] = make_float2(0.f, 0.f);
            }
        }
        if (c >= SX) {
#pragma unroll
            for (int r = 0; r < SY; r++) exch[((buf * NS + slot) * SY + r) * SX + c - SX] = tot[r];
        }
        const int own = before + (valid ? 1 : 0);
        before = valid ? 1 : 0;
        if (c == 0) cover[buf][slot] = own;
        __syncthreads();
        // normalisation and NaN restore (:308-320)
        if (pi >= i0 && slot > 0 && c < SX && x < a.nx) {
            const int n = own + cover[buf][slot - 1];
            // s / n, n = 1 to 4: by a power of two it is the product with the exact reciprocal, and by three a
            // division (cells with one invalid patch).  2048 x 2048, 32 x 32: 154 us, with a division throughout 232
            const float rn = n == 4 ? 0.25f : n == 2 ? 0.5f : 1.f;
            float2* o = a.out + (long long)y0 * a.op + x;
            auto write = [&](auto quotient) {
#pragma unroll
                for (int r = 0; r < SY; r++) {
                    if (y0 + r < a.ny) {
                        const float2 s = add2(tot[r], exch[((buf * NS + slot - 1) * SY + r) * SX + c]);
                        const bool bad = n == 0 || ((nan >> r) & 1u);
                        const float q = __int_as_float(0x7fc00000);
                        o[(long long)r * a.op] = bad ? make_float2(q, q) : quotient(s);
                    }
                }
            };
            if (n != 3) write([&](float2 s) { return mul2(s, make_float2(rn, rn)); });
            else write([](float2 s) { return gs_third(s); });
        }
        buf ^= 1;
    }
}

template <int PY, int PX>
cudaError_t gs_launch(GsArgs a, cudaStream_t s) {
    using S = GsShape<PY, PX>;
    const int cells_y = (a.ny + S::SY - 1) / S::SY, cells_x = (a.nx + S::SX - 1) / S::SX;
    const int strips = (cells_x + S::NS - 2) / (S::NS - 1);
    // one wave of CTAs: as few walks as fill the SMs, since each starts with one patch row more
    const int segs = std::max(1, std::min(cells_y, 148 * S::CTAS / strips));
    a.seg = (cells_y + segs - 1) / segs;
    const cudaError_t e = unw_smem_limit((const void*)k_gs_walk<PY, PX>);
    if (e != cudaSuccess) return e;
    k_gs_walk<PY, PX><<<dim3(strips, (cells_y + a.seg - 1) / a.seg), 256, S::SMEM, s>>>(a);
    return cudaGetLastError();
}

template <int PY>
cudaError_t gs_launch_y(int px, const GsArgs& a, cudaStream_t s) {
    switch (px) {
        case 4: return gs_launch<PY, 4>(a, s);
        case 8: return gs_launch<PY, 8>(a, s);
        case 16: return gs_launch<PY, 16>(a, s);
        case 32: return gs_launch<PY, 32>(a, s);
        default: return gs_launch<PY, 64>(a, s);
    }
}

struct GsLayout {
    int H, W;               // padded grid (utils_goldstein.py:214-226)
    size_t total;           // workspace: room for the result of a call in place
};

GsLayout gs_layout(long long ny, long long nx, int py, int px) {
    GsLayout L{};
    const int sy = py / 2, sx = px / 2;
    const long long pad_y = py - sy, pad_x = px - sx;
    const long long ey = (sy - ((ny + pad_y - py) % sy)) % sy;
    const long long ex = (sx - ((nx + pad_x - px) % sx)) % sx;
    L.H = (int)(ny + pad_y + ey);
    L.W = (int)(nx + pad_x + ex);
    auto up = [](size_t v) { return (v + 255) / 256 * 256; };
    // the size that the entry point has always asked for (callers may keep one buffer)
    L.total = up(sizeof(float) * ((size_t)py * px + 1)) + up(sizeof(float2) * (size_t)L.H * L.W) + up(sizeof(float) * (size_t)L.H * L.W) + 256;
    return L;
}

bool gs_psize_ok(int p) { return p >= 4 && p <= 64 && (p & (p - 1)) == 0; }

}  // namespace

extern "C" {

size_t unw_goldstein_workspace_bytes(int64_t H, int64_t W, int32_t psize_y, int32_t psize_x) {
    if (H <= 0 || W <= 0 || !gs_psize_ok(psize_y) || !gs_psize_ok(psize_x)) return 0;
    return gs_layout(H, W, psize_y, psize_x).total;
}

int unw_goldstein_c64(const float* phase, int64_t phase_pitch, const float* corr, int64_t corr_pitch, int64_t H,
                      int64_t W, int32_t psize_y, int32_t psize_x, float threshold, float* out, int64_t out_pitch,
                      void* workspace, size_t workspace_bytes, void* cuda_stream) {
    if (!phase || !corr || !out) return unw_set_error(UNW_E_ARG, "goldstein: null pointer");
    if (H <= 0 || W <= 0) return unw_set_error(UNW_E_ARG, "goldstein: bad shape");
    if (phase_pitch < W || corr_pitch < W || out_pitch < W)
        return unw_set_error(UNW_E_ARG, "goldstein: pitch smaller than width");
    if (!gs_psize_ok(psize_y) || !gs_psize_ok(psize_x))
        return unw_set_error(UNW_E_UNSUPPORTED, "goldstein: patch sizes must be powers of two in [4, 64]");
    if (!(threshold >= 0.f) || !(threshold <= 1.f)) return unw_set_error(UNW_E_ARG, "goldstein: threshold in [0, 1]");
    if (!workspace) return unw_set_error(UNW_E_ARG, "goldstein: workspace is NULL");
    const GsLayout L = gs_layout(H, W, psize_y, psize_x);
    char* base = (char*)(((size_t)workspace + 255) / 256 * 256);
    if ((size_t)(base - (char*)workspace) + L.total - 256 > workspace_bytes)
        return unw_set_error(UNW_E_WORKSPACE, "goldstein: workspace too small");
    cudaStream_t s = (cudaStream_t)cuda_stream;
    GsArgs a{};
    a.phase = (const float2*)phase; a.pp = phase_pitch;
    a.corr = corr; a.cp = corr_pitch;
    a.ny = (int)H; a.nx = (int)W;
    a.npy = (L.H - psize_y) / (psize_y / 2) + 1;
    a.npx = (L.W - psize_x) / (psize_x / 2) + 1;
    a.min_valid = (int)((double)psize_y * (double)psize_x * (double)threshold);
    a.out = (float2*)out; a.op = out_pitch;
    // a result over an input goes through the workspace: patches read pixels of finished cells
    auto overlaps = [&](const void* p, size_t bytes) {
        const size_t o = (size_t)out, ob = sizeof(float2) * ((size_t)(H - 1) * out_pitch + W), q = (size_t)p;
        return o < q + bytes && q < o + ob;
    };
    const bool staged = overlaps(phase, sizeof(float2) * ((size_t)(H - 1) * phase_pitch + W)) ||
                        overlaps(corr, sizeof(float) * ((size_t)(H - 1) * corr_pitch + W));
    if (staged) { a.out = (float2*)base; a.op = W; }
    cudaError_t e = cudaErrorInvalidValue;
    switch (psize_y) {
        case 4: e = gs_launch_y<4>(psize_x, a, s); break;
        case 8: e = gs_launch_y<8>(psize_x, a, s); break;
        case 16: e = gs_launch_y<16>(psize_x, a, s); break;
        case 32: e = gs_launch_y<32>(psize_x, a, s); break;
        case 64: e = gs_launch_y<64>(psize_x, a, s); break;
    }
    if (e == cudaSuccess && staged)
        e = cudaMemcpy2DAsync(out, sizeof(float2) * out_pitch, a.out, sizeof(float2) * W, sizeof(float2) * W, H,
                              cudaMemcpyDeviceToDevice, s);
    if (e != cudaSuccess) return unw_set_error(UNW_E_CUDA, cudaGetErrorString(e));
    return UNW_OK;
}

}  // extern "C"
