// Column half of the DCT preconditioner as a direct tridiagonal solve.
//
// After the row DCT-II the Neumann Laplacian couples only the rows of one column l:
//   (T_H + s_l) z = x,   T_H = second difference with reflecting ends,  s_l = 4 sin^2(pi l / 2W),
// which is what column DCT-II, division by the eigenvalue and column DCT-III
// (utils_unwrap2d.py:1390-1403, the column half of dct_2d / idct_2d at :1316-1365) solve in
// exact arithmetic.  With rho = exp(-theta), rho + 1/rho = 2 + s_l, the operator on the evenly
// reflected, infinitely extended column factors into a causal and an anti-causal first-order
// recurrence,
//   y_i = rho y_{i-1} + x_i,      z_i = rho (y_i + z_{i+1}),
// so a column costs a few multiply-adds per row instead of two transforms, for any H.
//
// A segment of consecutive rows is summarised by two states,
//   f = sum_j rho^(n-1-j) x_j  (causal, at its end),   b = sum_j rho^j x_j  (at its start),
// from which the recurrences' start values of every segment follow; then each segment runs the
// two recurrences over its own rows.  T is read, the result goes to a second array (Tz).
//
// Two kinds of CTA in one launch, by column:
//  * fast, theta >= 0.278 (91% of the columns): a recurrence forgets its past within 64 rows (32
//    from theta = 0.557 on) to 2e-8, so a CTA takes 16 segments of L rows of 64 adjacent columns,
//    of which the first and last 64 (32) rows are halo that neighbouring CTAs also read.
//    Float32, two columns per lane as packed operations; no exchange between CTAs.
//  * wide, the columns below: the 1/theta^2 amplification of the lowest modes and the long
//    memory take float64 and the whole column: a CTA holds 4 columns x 128 chunks of rows, joins
//    the chunks' states by a scan and closes the reflecting ends exactly (the geometric series
//    of the images, 1 / (1 - rho^2H)).
//    Column l = 0 (s = 0, rho = 1) is singular: its mean is removed (the zeroed DC term), the
//    recurrences are prefix sums, and the additive constant that makes the solution's mean zero
//    follows from the moments sum x, sum j x, sum j^2 x.
//
// r.z of the PCG by Parseval's identity along the rows only:
//   r.z = sum_i sum_l e_l X_l(i) Z_l(i),  e_0 = 1/2, e_l = 1,  Z_l = z_l / 2W as written.
//
// What bounds it (B200): 8 bytes per pixel of T and Tz, at 4096 x 4096 134 MB or 20.5 us at the
// measured copy rate; it takes 41 us there in the solver (kernel trace; 42 us from cold L2) and 32 us in mode 0,
// without r.z (682 CTAs, two per SM at 64 registers; the latency of the four batches of row loads of a
// segment is most of a CTA's 10.7 us).  Up to 1024 x 1024 it is
// the chain of one CTA, 5 us, of which the wide CTAs are the longest.  In the solver, CUDA-event
// times per launch against the column FFTs (two transforms and the spectral step) that it
// replaced: 4096 x 4096 45.5 us / 89.9, 2048 x 2048 15.6 / 22.9, 1838 x 2750 (Bluestein) 22.9 / 110.6,
// 1024 x 1024 12.9 / 18.8, 200 x 180 11.4 / 25.1 (about 8 us of each is the event pair).
// Tried and not kept, at 4096 x 4096: all columns in float64 in clusters that exchange the chunk states
// through distributed shared memory (69 us: start-up, barrier and folding took two thirds of a
// CTA's time), one column per lane (64 us), an L2 prefetch of the segment's rows (47 us).
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <mutex>

#include "unw_kernels.h"
#include "unw_rowops.cuh"

namespace {

constexpr unsigned long long TRI_WAIT_NS = 2000000000ull;  // 2 s at most for the tile's copies
constexpr int TRI_STATUS_TIMEOUT = 16;                      // UNW_S_TC_TIMEOUT
constexpr int TRI_NW = 16;                                  // warps per CTA
constexpr int TRI_WCOLS = 4, TRI_CHUNKS = 128;              // columns and row chunks of a wide CTA
constexpr int TRI_SUBMAX = 28;                              // 8-row pieces of the longest chunk (28672 / 128 / 8)
constexpr int TRI_COLS = 64;                                // columns of a fast CTA
constexpr int TRI_HALO_A = 64, TRI_HALO_B = 32;             // halo rows of the fast CTAs

// Per-column constants, one array of W entries each (k_tri_tables): float64, then rho and the
// Green factor 1 / (1 - rho^2) again in float32 for the fast CTAs.
enum { TQ_RHO = 0, TQ_SEG, TQ_SEGLAST, TQ_ALL, TQ_IMG, TQ_GREEN, TQ_N };
__host__ __device__ __forceinline__ float* tri_tab32(double* tab, int W) { return reinterpret_cast<float*>(tab + (size_t)TQ_N * W); }

__device__ __forceinline__ uint32_t tri_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool tri_wait(uint64_t* bar, uint32_t parity) {
    unsigned long long t0, t1;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
    while (true) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(tri_smem(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t1));
        if (t1 - t0 > TRI_WAIT_NS) return false;
    }
}

// Row r of the evenly reflected column, -H <= r < 2H: the row of [0, H) that it repeats.
__device__ __forceinline__ int tri_mirror1(int r, int H) {
    const int s = r < 0 ? -1 - r : r;
    return s < H ? s : 2 * H - 1 - s;
}
__device__ __noinline__ int tri_mirror(int r, int H) {  // any r
    r %= 2 * H;
    if (r < 0) r += 2 * H;
    return tri_mirror1(r, H);
}

// Chunk states of a wide CTA, [column][chunk]; p, f, b: the chunk's power rho^rows and states, then
// (after the scan) y, u in f, b: the causal state before the chunk and z / rho after it.
struct TriWideShared {
    double p[TRI_WCOLS][TRI_CHUNKS], f[TRI_WCOLS][TRI_CHUNKS], b[TRI_WCOLS][TRI_CHUNKS];
    double m1[TRI_CHUNKS], m2[TRI_CHUNKS];  // moments of column 0
    double mean;
};

// Scan of a wide column by one warp: four consecutive chunks per lane.
__device__ __forceinline__ void tri_wide_scan(const GridDev& G, int c, int v, TriWideShared& sh) {
    const int lane = threadIdx.x & 31, W = G.W, H = G.H;
    const unsigned all = 0xffffffffu;
    const double* __restrict__ tab = G.tri + c;
    const double rho = tab[(size_t)TQ_RHO * W], pall = tab[(size_t)TQ_ALL * W];
    const double img = tab[(size_t)TQ_IMG * W], green = tab[(size_t)TQ_GREEN * W];
    double p[4], f[4], b[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        p[t] = sh.p[v][4 * lane + t];
        f[t] = sh.f[v][4 * lane + t];
        b[t] = sh.b[v][4 * lane + t];
    }
    double P = 1.0, F = 0.0, B = 0.0;  // the lane's four chunks as one
#pragma unroll
    for (int t = 0; t < 4; t++) { F = fma(p[t], F, f[t]); P *= p[t]; }
#pragma unroll
    for (int t = 3; t >= 0; t--) B = fma(p[t], B, b[t]);
    double Pl = P, Pr = P, Fl = F, Br = B;  // inclusive over lanes <= this / >= this
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double pu = __shfl_up_sync(all, Pl, o), fu = __shfl_up_sync(all, Fl, o);
        const double pd = __shfl_down_sync(all, Pr, o), bd = __shfl_down_sync(all, Br, o);
        if (lane >= o) { Fl = fma(Pl, fu, Fl); Pl *= pu; }
        if (lane + o < 32) { Br = fma(Pr, bd, Br); Pr *= pd; }
    }
    const double ft = __shfl_sync(all, Fl, 31), bt = __shfl_sync(all, Br, 0);
    double pe = __shfl_up_sync(all, Pl, 1), fe = __shfl_up_sync(all, Fl, 1);    // exclusive
    double qe = __shfl_down_sync(all, Pr, 1), be = __shfl_down_sync(all, Br, 1);
    if (lane == 0) { pe = 1.0; fe = 0.0; }
    if (lane == 31) { qe = 1.0; be = 0.0; }
    if (c == 0) {
        // rho = 1: prefix sums of x - mean, and z from the moments (mean of z = 0)
        const int Lc = (H + TRI_CHUNKS - 1) / TRI_CHUNKS;
        const double N = (double)H;
        double a1[4], s1 = 0.0, s2 = 0.0;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            a1[t] = sh.m1[4 * lane + t];
            s1 += a1[t];
            s2 += sh.m2[4 * lane + t];
        }
        double i1 = s1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double x = __shfl_up_sync(all, i1, o);
            if (lane >= o) i1 += x;
            s2 += __shfl_xor_sync(all, s2, o);
        }
        const double t1 = __shfl_sync(all, i1, 31), mean = ft / N;
        const double c1 = t1 - ft * (N - 1.0) * 0.5;
        const double c2 = s2 - ft * (N - 1.0) * (2.0 * N - 1.0) / 6.0;
        const double z0 = (c2 - (2.0 * N - 1.0) * c1) / (2.0 * N);
        double p0 = fe, p1 = i1 - s1;
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const int chunk = 4 * lane + t, r0 = min(chunk * Lc, H), r1 = min(r0 + Lc, H);
            sh.f[v][chunk] = p0 - mean * (double)r0;
            p0 += f[t];
            p1 += a1[t];
            const double j1 = (double)r1;
            sh.b[v][chunk] = z0 - (j1 * p0 - p1 - mean * (j1 * (j1 + 1.0) * 0.5));
        }
        if (lane == 0) sh.mean = mean;
        return;
    }
    double y = fma(pe, fma(pall, ft, bt) * img, fe);    // with the left images before row 0
    double br = fma(qe, fma(pall, bt, ft) * img, be);   // with the right images after row H - 1
    double ye[4];
#pragma unroll
    for (int t = 0; t < 4; t++) {
        sh.f[v][4 * lane + t] = y;
        ye[t] = y = fma(p[t], y, f[t]);
    }
#pragma unroll
    for (int t = 3; t >= 0; t--) {
        sh.b[v][4 * lane + t] = fma(rho, ye[t], br) * green;  // z / rho at the row after the chunk
        br = fma(p[t], br, b[t]);
    }
}

// Four columns from c0 in float64, all rows.  Lane: column (lane & 3), chunk 8 w + (lane >> 2).
template <int MODE>
__device__ __forceinline__ double tri_wide(const GridDev& G, int c0, TriWideShared& sh) {
    constexpr int K = 8;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, cl = lane & 3;
    const int H = G.H, W = G.W, P = G.P, Lc = (H + TRI_CHUNKS - 1) / TRI_CHUNKS;
    const int c = c0 + cl;
    const bool on = c < W;
    const int chunk = 8 * w + (lane >> 2), r0 = chunk * Lc;
    const int nr = on ? max(0, min(Lc, H - r0)) : 0;
    const float* __restrict__ x0 = G.T + (size_t)r0 * P + c;
    const double* __restrict__ tab = G.tri + c;
    const double rho = on ? tab[(size_t)TQ_RHO * W] : 0.0;
    const double pc = nr == Lc ? tab[(size_t)TQ_SEG * W] : (nr > 0 ? tab[(size_t)TQ_SEGLAST * W] : 1.0);
    double rK = rho * rho;
    rK *= rK;
    rK *= rK;  // rho^8
    const int ns = (nr + K - 1) / K;
    // 1. states of the chunk
    double fm[TRI_SUBMAX];
    double fs = 0.0, bs = 0.0, pw = 1.0, m1 = 0.0, m2 = 0.0;
    float x[K];
    for (int m = 0; m < ns; m++) {
#pragma unroll
        for (int k = 0; k < K; k++) x[k] = m * K + k < nr ? __ldg(x0 + (ptrdiff_t)((m * K + k) * P)) : 0.f;
        double f = 0.0, b = 0.0, pk = rK;
        if ((m + 1) * K <= nr) {
#pragma unroll
            for (int k = 0; k < K; k++) f = fma(rho, f, (double)x[k]);
        } else {
            pk = 1.0;
#pragma unroll
            for (int k = 0; k < K; k++)
                if (m * K + k < nr) { f = fma(rho, f, (double)x[k]); pk *= rho; }
        }
#pragma unroll
        for (int k = K - 1; k >= 0; k--) b = fma(rho, b, (double)x[k]);
        fm[m] = f;
        fs = fma(pk, fs, f);
        bs = fma(pw, b, bs);
        pw *= rK;
        if (c == 0) {
            double j = (double)(r0 + m * K);
            for (int k = 0; k < K; k++, j += 1.0) {
                m1 = fma(j, (double)x[k], m1);
                m2 = fma(j * j, (double)x[k], m2);
            }
        }
    }
    sh.p[cl][chunk] = pc;
    sh.f[cl][chunk] = fs;
    sh.b[cl][chunk] = bs;
    if (c == 0) {
        sh.m1[chunk] = m1;
        sh.m2[chunk] = m2;
    }
    __syncthreads();
    // 2. start values of every chunk
    if (w < TRI_WCOLS && c0 + w < W) tri_wide_scan(G, c0 + w, w, sh);
    __syncthreads();
    // 3. the recurrences
    if (nr == 0) return 0.0;
    double y = sh.f[cl][chunk], u = sh.b[cl][chunk];
    const double mean = c == 0 ? sh.mean : 0.0;
    for (int m = 0; m < ns; m++) {  // causal state at the start of every piece
        const double t = fm[m];
        fm[m] = y;
        y = fma(rK, y, t - mean * (double)K);
    }
    const double osc = rho * (0.5 / (double)W);
    float* __restrict__ z0p = G.Tz + (size_t)r0 * P + c;
    double acc = 0.0;
    for (int m = ns - 1; m >= 0; m--) {
        double yk[K];
        if (m < ns - 1) {
#pragma unroll
            for (int k = 0; k < K; k++) x[k] = __ldg(x0 + (ptrdiff_t)((m * K + k) * P));
        }
        double t = fm[m];
#pragma unroll
        for (int k = 0; k < K; k++) yk[k] = t = fma(rho, t, (double)x[k] - mean);
#pragma unroll
        for (int k = K - 1; k >= 0; k--) {
            if (m * K + k < nr) {
                u = fma(rho, u, yk[k]);
                const double o = u * osc;
                if (MODE >= 1) acc = fma((double)x[k], o, acc);
                z0p[(ptrdiff_t)((m * K + k) * P)] = (float)o;
            }
        }
    }
    return c == 0 ? 0.5 * acc : acc;
}

// Rows [tile * SC * L, (tile + 1) * SC * L) of the 64 columns from c0, in float32; SC = 16 - 2 HS
// segments of L rows with HS = halo / L segments on either side.  `tile_s` (TMA): the 16 L rows from
// row (tile * SC - HS) * L on.
// PAIRS: rows are 8-byte aligned and a lane's two columns move as 8 bytes (columns between W and the
// pitch are padding: read as zero, written as zero).
template <int L, int MODE, bool TMA, bool PAIRS>
__device__ __forceinline__ double tri_fast(const GridDev& G, int c0, int tile, int halo, const float* tile_s,
                                           float2 (*sf)[32], float2 (*sb)[32]) {
    constexpr int K = 8, NS = L / K;
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int H = G.H, W = G.W;
    int P = G.P;
    const int HS = halo / L, SC = TRI_NW - 2 * HS;
    const int c = c0 + 2 * lane;
    const bool on0 = c < W, on1 = c + 1 < W;
    const bool in = PAIRS ? c < P : on0;
    const bool edge = c0 + TRI_COLS > W;          // columns beyond W in this strip
    const int r0 = (tile * SC - HS + w) * L;      // first row of this warp's segment
    const int base = (tile * SC - HS) * L;        // first row of the staged tile
    const float* __restrict__ T = G.T + c;
    float2 rho = make_float2(0.f, 0.f), green = rho;
    {
        const float* t = tri_tab32(const_cast<double*>(G.tri), W) + c;
        if (on0) { rho.x = __ldg(t); green.x = __ldg(t + W); }
        if (on1) { rho.y = __ldg(t + 1); green.y = __ldg(t + 1 + W); }
    }
    auto ld = [&](ptrdiff_t o) {  // the lane's two columns at row offset o
        float2 v = make_float2(0.f, 0.f);
        if (PAIRS) {
            if (in) v = __ldg(reinterpret_cast<const float2*>(T + o));
        } else {
            if (on0) v.x = __ldg(T + o);
            if (on1) v.y = __ldg(T + o + 1);
        }
        return v;
    };
    // Eight rows of the segment from row r.  Rows outside [0, H) repeat the reflected ones; rows
    // beyond the halo after the last row are left out (their weight is below 2e-8).
    auto get = [&](int m, float2 (&x)[K]) {
        const int r = r0 + m * K;
        if (r >= 0 && r + K <= H) {
            if (TMA) {
                const float* t = tile_s + (w * L + m * K) * TRI_COLS + 2 * lane;
#pragma unroll
                for (int k = 0; k < K; k++) x[k] = *reinterpret_cast<const float2*>(t + k * TRI_COLS);
            } else {
                const ptrdiff_t o = (ptrdiff_t)r * P;
#pragma unroll
                for (int k = 0; k < K; k++) x[k] = ld(o + (ptrdiff_t)(k * P));
            }
        } else {
            const bool near = H >= halo;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const int rr = min(r + k, H + halo - 1);
                const int q = near ? tri_mirror1(rr, H) : tri_mirror(rr, H);
                x[k] = TMA ? *reinterpret_cast<const float2*>(tile_s + (q - base) * TRI_COLS + 2 * lane)
                           : ld((ptrdiff_t)q * P);
            }
#pragma unroll
            for (int k = 0; k < K; k++)
                if (r + k >= H + halo) x[k] = make_float2(0.f, 0.f);
        }
        if (PAIRS && edge) {
#pragma unroll
            for (int k = 0; k < K; k++) {
                if (!on1) x[k].y = 0.f;
                if (!on0) x[k].x = 0.f;
            }
        }
    };
    const float2 zero = make_float2(0.f, 0.f);
    float2 rK = mul2(rho, rho);
    rK = mul2(rK, rK);
    rK = mul2(rK, rK);  // rho^8
    float2 pseg = rK;
#pragma unroll
    for (int t = 1; t < NS; t *= 2) pseg = mul2(pseg, pseg);

    // 1. states of the segment
    float2 x[K], fm[NS], fs = zero, bs = zero, pw = make_float2(1.f, 1.f);
#pragma unroll
    for (int m = 0; m < NS; m++) {
        get(m, x);
        float2 f = zero, b = zero;
#pragma unroll
        for (int k = 0; k < K; k++) f = fma2(rho, f, x[k]);
#pragma unroll
        for (int k = K - 1; k >= 0; k--) b = fma2(rho, b, x[k]);
        fm[m] = f;
        fs = fma2(rK, fs, f);
        bs = fma2(pw, b, bs);
        pw = mul2(pw, rK);
    }
    sf[w][lane] = fs;
    sb[w][lane] = bs;
    __syncthreads();
    if (w < HS || w >= TRI_NW - HS || r0 >= H) return 0.0;

    // 2. start values
    float2 y = zero, br = zero;
#pragma unroll
    for (int v = 0; v < TRI_NW - 1; v++) {
        const float2 t = fma2(pseg, y, sf[v][lane]);
        if (v < w) y = t;
    }
#pragma unroll
    for (int v = TRI_NW - 1; v > 0; v--) {
        const float2 t = fma2(pseg, br, sb[v][lane]);
        if (v > w) br = t;
    }
    float2 u = mul2(fma2(rho, fma2(pseg, y, fs), br), green);  // z / rho at the row after the segment
#pragma unroll
    for (int m = 0; m < NS; m++) {
        const float2 t = fm[m];
        fm[m] = y;
        y = fma2(rK, y, t);
    }
    // 3. the recurrences
    asm volatile("" : "+r"(P));  // row offsets are formed again, not kept across the exchange
    const float scale = (float)(0.5 / (double)W);
    const float2 osc = mul2(rho, make_float2(scale, scale));
    float* __restrict__ Z = G.Tz + (ptrdiff_t)r0 * P + c;
    double acc = 0.0;
#pragma unroll
    for (int m = NS - 1; m >= 0; m--) {
        if (m < NS - 1) get(m, x);
        float2 yk[K], t = fm[m];
#pragma unroll
        for (int k = 0; k < K; k++) yk[k] = t = fma2(rho, t, x[k]);
        auto row = [&](int k) {
            u = fma2(rho, u, yk[k]);
            const float2 o = mul2(u, osc);
            // the float32 products of r.z are joined in pairs and summed in float64
            if (MODE >= 1) acc += (double)fmaf(x[k].x, o.x, x[k].y * o.y);
            float* z = Z + (ptrdiff_t)((m * K + k) * P);
            if (PAIRS) {
                if (in) *reinterpret_cast<float2*>(z) = o;
            } else {
                if (on0) z[0] = o.x;
                if (on1) z[1] = o.y;
            }
        };
        if (r0 + (m + 1) * K <= H) {
#pragma unroll
            for (int k = K - 1; k >= 0; k--) row(k);
        } else {
#pragma unroll
            for (int k = K - 1; k >= 0; k--) {
                if (r0 + m * K + k < H) row(k);
                else u = fma2(rho, u, yk[k]);
            }
        }
    }
    return acc;
}

// MODE 0: DCT initial solve and operator entry point (always runs); MODE 1 / 2: PCG (gated), also
// r.z and its scalar step (col_finalize).  TMA: the fast CTAs' tiles come into shared memory by 2-D
// bulk copies, otherwise each thread loads its own rows; both give the same bits.
template <int L, int MODE, bool TMA>
__global__ void __launch_bounds__(TRI_NW * 32, 2) k_col_tri(const GridDev* __restrict__ grids,
                                                            const int* __restrict__ starts, int n,
                                                            const CUtensorMap* __restrict__ maps) {
    constexpr int TR = TRI_NW * L, BOX = 256;
    extern __shared__ unsigned char tri_raw[];
    __shared__ union {
        TriWideShared wide;
        struct { float2 f[TRI_NW][32], b[TRI_NW][32]; } fast;
    } sh;
    __shared__ double red[32];
    __shared__ __align__(8) uint64_t bar;
    const int g = find_grid(starts, n, blockIdx.x);
    const GridDev& G = grids[g];
    InstState* st = G.st;
    if (MODE >= 1 && !(st->irls_active && st->cg_active)) return;
    const int local = blockIdx.x - starts[g];
    const int nct = starts[g + 1] - starts[g];
    const int nwide = G.tri_ws * (32 / TRI_WCOLS);
    double acc[1];
    if (local < nwide) {
        acc[0] = tri_wide<MODE>(G, TRI_WCOLS * local, sh.wide);
    } else {
        // tiles outermost, so that CTAs running together read whole rows
        int f = local - nwide, c0, tile, halo;
        const int na = G.tri_as;
        if (f < na * G.tri_nta) {
            tile = f / na;
            c0 = 32 * G.tri_ws + TRI_COLS * (f - tile * na);
            halo = TRI_HALO_A;
        } else {
            f -= na * G.tri_nta;
            const int first = 32 * G.tri_ws + TRI_COLS * na, nb = (G.W - first + TRI_COLS - 1) / TRI_COLS;
            tile = f / nb;
            c0 = first + TRI_COLS * (f - tile * nb);
            halo = TRI_HALO_B;
        }
        float* const tile_s = reinterpret_cast<float*>((unsigned char*)(((size_t)tri_raw + 127) & ~(size_t)127));
        bool ok = true;
        if (TMA) {
            const CUtensorMap* mt = maps + UNW_MAPS_PER_GRID * g + UNW_MAP_COL;
            if (threadIdx.x == 0) {
                const int base = (tile * (TR - 2 * halo)) - halo;
                asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tri_smem(&bar)) : "memory");
                asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
                asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"((unsigned long long)mt) : "memory");
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tri_smem(&bar)),
                             "r"((uint32_t)(TR * TRI_COLS * 4))
                             : "memory");
                for (int b = 0; b < TR / BOX; b++)
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
                        ::"r"(tri_smem(tile_s + (size_t)b * BOX * TRI_COLS)), "l"((unsigned long long)mt),
                        "r"(tri_smem(&bar)), "r"(c0), "r"(base + b * BOX)
                        : "memory");
            }
            __syncthreads();  // the barrier is initialised
            ok = tri_wait(&bar, 0);
            if (__syncthreads_or(!ok)) {
                if (threadIdx.x == 0) {
                    tri_wait(&bar, 0);  // the copies that were late may still land: once more (bounded)
                    atomicOr(&st->status, TRI_STATUS_TIMEOUT);
                }
                ok = false;
            }
        }
        if (!ok) acc[0] = 0.0;
        else if (TMA || (!(G.P & 1) && !(((size_t)G.T | (size_t)G.Tz) & 7)))
            acc[0] = tri_fast<L, MODE, TMA, true>(G, c0, tile, halo, tile_s, sh.fast.f, sh.fast.b);
        else acc[0] = tri_fast<L, MODE, TMA, false>(G, c0, tile, halo, tile_s, sh.fast.f, sh.fast.b);
    }
    if (MODE == 0) return;
    if (arrive<1>(G, local, nct, acc, red)) {
        finish_sum<1>(G, nct, acc, red);
        if (threadIdx.x == 0) col_finalize<MODE>(st, acc[0]);
    }
}

// theta = -ln rho from 2 sinh(theta / 2) = sqrt(s) = 2 sin(pi l / 2W); every power as an exponential,
// so that none is formed by cancellation.
__global__ void k_tri_tables(double* __restrict__ tab, int W, int H) {
    const int l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l >= W) return;
    double* t = tab + l;
    const size_t S = (size_t)W;
    float* t32 = tri_tab32(tab, W) + l;
    const int Lc = (H + TRI_CHUNKS - 1) / TRI_CHUNKS;
    if (l == 0) {
        for (int q = TQ_RHO; q <= TQ_ALL; q++) t[q * S] = 1.0;
        t[TQ_IMG * S] = 0.0;
        t[TQ_GREEN * S] = 0.0;
        t32[0] = 1.f;
        t32[S] = 0.f;
        return;
    }
    const double th = 2.0 * asinh(sinpi((double)l / (2.0 * (double)W)));
    t[TQ_RHO * S] = exp(-th);
    t[TQ_SEG * S] = exp(-th * (double)Lc);
    t[TQ_SEGLAST * S] = exp(-th * (double)((H - 1) % Lc + 1));
    t[TQ_ALL * S] = exp(-th * (double)H);
    t[TQ_IMG * S] = -1.0 / expm1(-2.0 * th * (double)H);
    const double green = -1.0 / expm1(-2.0 * th);
    t[TQ_GREEN * S] = green;
    t32[0] = (float)exp(-th);
    t32[S] = (float)green;
}

template <int L, bool TMA>
cudaError_t tri_launch(int mode, int nblk, cudaStream_t s, const GridDev* gd, const int* st, int n,
                       const CUtensorMap* maps) {
    const size_t smem = TMA ? (size_t)TRI_NW * L * TRI_COLS * 4 + 128 : 0;
    auto go = [&](auto kfn) {
        if (TMA) {
            const cudaError_t e = unw_smem_limit((const void*)kfn);
            if (e != cudaSuccess) return e;
        }
        kfn<<<nblk, TRI_NW * 32, smem, s>>>(gd, st, n, maps);
        return cudaGetLastError();
    };
    switch (mode) {
        case 0: return go(k_col_tri<L, 0, TMA>);
        case 1: return go(k_col_tri<L, 1, TMA>);
        default: return go(k_col_tri<L, 2, TMA>);
    }
}

PFN_cuTensorMapEncodeTiled_v12000 tri_encode_fn() {
    static std::once_flag once;
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = (PFN_cuTensorMapEncodeTiled_v12000)p;
    });
    return fn;
}

}  // namespace

// Rows per segment of the fast CTAs: 32 (fewer halo rows read twice) once that still gives every SM
// two CTAs, else 16 (more and shorter CTAs).  Measured per launch: 4096 x 4096 45.5 us with 32,
// 53.1 us with 16; 1024 x 1024 5 us with 16 (118 CTAs).
int unw_tri_rows(int H, int W) {
    const int tile = TRI_NW * 32 - 2 * TRI_HALO_B;
    return (long long)((W + TRI_COLS - 1) / TRI_COLS) * ((H + tile - 1) / tile) >= 2 * 148 ? 32 : 16;
}

// Groups of 32 wide columns (l / W < 0.0892, theta < 0.278), then strips of 64 columns with the long halo
// (starting at l / W < 0.1821, theta < 0.557), tiles per strip with either halo; returns the CTAs.
int unw_tri_shape(int H, int W, int L, int* ws, int* as, int* nta, int* ntb) {
    const int a = TRI_NW * L - 2 * TRI_HALO_A, b = TRI_NW * L - 2 * TRI_HALO_B;
    *ws = (int)std::min<long long>((W + 31) / 32, ((long long)W * 892 + 319999) / 320000);
    const int rest = std::max(0, W - 32 * *ws);
    const int lim = (int)(((long long)W * 1821 + 9999) / 10000);  // first column of the short halo
    *as = std::min((rest + TRI_COLS - 1) / TRI_COLS, std::max(0, (lim - 32 * *ws + TRI_COLS - 1) / TRI_COLS));
    *nta = (H + a - 1) / a;
    *ntb = (H + b - 1) / b;
    const int nb = (std::max(0, rest - TRI_COLS * *as) + TRI_COLS - 1) / TRI_COLS;
    return *ws * (32 / TRI_WCOLS) + *as * *nta + nb * *ntb;
}

size_t unw_tri_table_bytes(long long W) { return (sizeof(double) * TQ_N + sizeof(float) * 2) * (size_t)W; }

cudaError_t unw_tri_tables(double* tab, int H, int W, cudaStream_t s) {
    k_tri_tables<<<(W + 127) / 128, 128, 0, s>>>(tab, W, H);
    return cudaGetLastError();
}

bool unw_tri_map(const float* T, int H, int W, int P, void* out) {
    auto fn = tri_encode_fn();
    if (!fn || (P & 3) || ((size_t)T & 15)) return false;
    cuuint64_t dims[2] = {(cuuint64_t)W, (cuuint64_t)H};
    cuuint64_t strides[1] = {(cuuint64_t)P * 4};
    cuuint32_t box[2] = {TRI_COLS, 256};
    cuuint32_t estr[2] = {1, 1};
    return fn((CUtensorMap*)out, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(T), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

cudaError_t unw_launch_col_tri(int L, bool tma, int mode, int nblk, cudaStream_t s, const GridDev* gd,
                               const int* starts, int n, const void* maps) {
    if (nblk <= 0) return cudaSuccess;
    const CUtensorMap* m = (const CUtensorMap*)maps;
    if (L == 16)
        return tma ? tri_launch<16, true>(mode, nblk, s, gd, starts, n, m)
                   : tri_launch<16, false>(mode, nblk, s, gd, starts, n, m);
    return tma ? tri_launch<32, true>(mode, nblk, s, gd, starts, n, m)
               : tri_launch<32, false>(mode, nblk, s, gd, starts, n, m);
}
