// filter.cu -- row filtering for filtered backprojection (FBP).
//
// The reference's FBP (examples/fbp.py:27-56) multiplies each sinogram row's
// length-N DFT by a real frequency response w (|linspace(-1,1,N)|, optionally
// apodised), fftshifted, and keeps the real part of the inverse DFT.  For a
// real row that is exactly the circular convolution of the row with
// h = Re(IDFT(fftshift(w))).  This kernel evaluates that convolution
// directly, out[r][k] = scale * sum_j pre[j] in[r][j] h[(k - j) mod N], with
// the optional per-cell pre-weight (e.g. fan-beam cosine weighting) fused in.
//
// CURADON_GB300_FILTER=scalar selects the one-row kernel wherever rows are
// summed directly (the packed one computes the same bits; see
// k_filter_rows_pk).  Long rows of ramp-like taps go by FFT (k_filter_fft).
//
// Block = 256 threads x 4 consecutive outputs each = 1024 outputs of RB rows;
// the RB input rows and h live in shared memory; as j advances, the four h
// values a thread needs shift by one, so each step loads one new h value and
// RB row values (broadcast) for 4 * RB fused multiply-adds.
#include <algorithm>

#include "common.cuh"

namespace cg {
namespace {

constexpr int kFiltThreads = 256;
constexpr int kFiltOut = 4;  // outputs per thread

// Whether the taps have (almost) no response at zero frequency, as every ramp
// filter's: |sum h| <= 5 % of sum |h|.  Called by every thread of a block of
// at least 128 threads; the same sums whatever the block.
__device__ bool ramp_taps(const float *__restrict__ h, int N) {
    __shared__ float2 part[4];
    const int t = threadIdx.x;
    if (t < 128) {
        float2 a = make_float2(0.f, 0.f);
#pragma unroll 8
        for (int i = t; i < N; i += 128) a.x += h[i], a.y += fabsf(h[i]);
#pragma unroll
        for (int o = 16; o; o >>= 1) {
            a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
            a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
        }
        if (t % 32 == 0) part[t / 32] = a;
    }
    __syncthreads();
    const float sum = (part[0].x + part[1].x) + (part[2].x + part[3].x);
    const float mag = (part[0].y + part[1].y) + (part[2].y + part[3].y);
    __syncthreads();
    return fabsf(sum) <= 0.05f * mag;  // false for NaN
}

template <int RB>
__global__ void __launch_bounds__(kFiltThreads)
    k_filter_rows(const float *__restrict__ in, float *__restrict__ out,
                  const float *__restrict__ h, const float *__restrict__ pre, int nrows, int N,
                  float scale, bool skip_ramp) {
    wait_previous();
    if (skip_ramp && ramp_taps(h, N)) return;
    extern __shared__ float smem[];
    float *sh = smem;            // N
    float *srow = smem + N;      // RB x N
    const int r0 = blockIdx.y * RB;
    for (int i = threadIdx.x; i < N; i += kFiltThreads) sh[i] = h[i];
    for (int r = 0; r < RB; ++r) {
        const bool ok = r0 + r < nrows;
        const float *row = in + (size_t)(r0 + r) * N;
        for (int i = threadIdx.x; i < N; i += kFiltThreads)
            srow[r * N + i] = ok ? (pre ? row[i] * pre[i] : row[i]) : 0.f;
    }
    __syncthreads();
    const int k0 = (blockIdx.x * kFiltThreads + threadIdx.x) * kFiltOut;
    if (k0 >= N) return;
    float acc[RB][kFiltOut];
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
        for (int i = 0; i < kFiltOut; ++i) acc[r][i] = 0.f;
    // hw[i] = h[(k0 + i - j) mod N] for the current j (indices clamped to the
    // row for outputs past its end, which are not stored)
    float hw[kFiltOut];
#pragma unroll
    for (int i = 0; i < kFiltOut; ++i) hw[i] = sh[(k0 + i) % N];
    int hidx = k0;  // (k0 - j) mod N
    for (int j = 0; j < N; ++j) {
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            const float s = srow[r * N + j];
#pragma unroll
            for (int i = 0; i < kFiltOut; ++i) acc[r][i] = fmaf(s, hw[i], acc[r][i]);
        }
        // advance to j + 1: shift the window, load h[(k0 - j - 1) mod N]
        hidx = hidx == 0 ? N - 1 : hidx - 1;
#pragma unroll
        for (int i = kFiltOut - 1; i > 0; --i) hw[i] = hw[i - 1];
        hw[0] = sh[hidx];
    }
#pragma unroll
    for (int r = 0; r < RB; ++r) {
        if (r0 + r >= nrows) break;
        float *o = out + (size_t)(r0 + r) * N;
#pragma unroll
        for (int i = 0; i < kFiltOut; ++i)
            if (k0 + i < N) o[k0 + i] = acc[r][i] * scale;
    }
}

// The same convolution on pairs of rows: the rows 2p and 2p + 1 of the block
// are interleaved in shared memory and h is stored duplicated, so one packed
// FP32 FMA (`__ffma2_rn`) advances one output of two rows; the accumulation
// order of every output is that of k_filter_rows.
template <int RB>
__global__ void __launch_bounds__(kFiltThreads)
    k_filter_rows_pk(const float *__restrict__ in, float *__restrict__ out,
                     const float *__restrict__ h, const float *__restrict__ pre, int nrows, int N,
                     float scale, bool skip_ramp) {
    wait_previous();
    if (skip_ramp && ramp_taps(h, N)) return;
    static_assert(RB % 2 == 0, "row pairs");
    extern __shared__ float2 smem2[];
    float2 *sh = smem2;         // N: (h, h)
    float2 *srow = smem2 + N;   // RB / 2 x N: (row 2p, row 2p + 1)
    const int r0 = blockIdx.y * RB;
    for (int i = threadIdx.x; i < N; i += kFiltThreads) sh[i] = make_float2(h[i], h[i]);
    for (int rp = 0; rp < RB / 2; ++rp) {
        const int ra = r0 + 2 * rp, rb = ra + 1;
        const float *rowa = in + (size_t)ra * N, *rowb = in + (size_t)rb * N;
        for (int i = threadIdx.x; i < N; i += kFiltThreads) {
            const float w = pre ? pre[i] : 1.f;
            srow[rp * N + i] = make_float2(ra < nrows ? rowa[i] * w : 0.f,
                                           rb < nrows ? rowb[i] * w : 0.f);
        }
    }
    __syncthreads();
    const int k0 = (blockIdx.x * kFiltThreads + threadIdx.x) * kFiltOut;
    if (k0 >= N) return;
    float2 acc[RB / 2][kFiltOut];
#pragma unroll
    for (int rp = 0; rp < RB / 2; ++rp)
#pragma unroll
        for (int i = 0; i < kFiltOut; ++i) acc[rp][i] = make_float2(0.f, 0.f);
    float2 hw[kFiltOut];
#pragma unroll
    for (int i = 0; i < kFiltOut; ++i) hw[i] = sh[(k0 + i) % N];
    int hidx = k0;
#pragma unroll 4
    for (int j = 0; j < N; ++j) {
#pragma unroll
        for (int rp = 0; rp < RB / 2; ++rp) {
            const float2 sv = srow[rp * N + j];
#pragma unroll
            for (int i = 0; i < kFiltOut; ++i) acc[rp][i] = __ffma2_rn(sv, hw[i], acc[rp][i]);
        }
        hidx = hidx == 0 ? N - 1 : hidx - 1;
#pragma unroll
        for (int i = kFiltOut - 1; i > 0; --i) hw[i] = hw[i - 1];
        hw[0] = sh[hidx];
    }
#pragma unroll
    for (int rp = 0; rp < RB / 2; ++rp) {
        const int ra = r0 + 2 * rp;
#pragma unroll
        for (int i = 0; i < kFiltOut; ++i) {
            if (k0 + i >= N) continue;
            if (ra < nrows) out[(size_t)ra * N + k0 + i] = acc[rp][i].x * scale;
            if (ra + 1 < nrows) out[(size_t)(ra + 1) * N + k0 + i] = acc[rp][i].y * scale;
        }
    }
}

template <int RB>
int launch_rb_pk(const float *in, float *out, const float *h, const float *pre, int nrows, int N,
                 float scale, bool skip_ramp, cudaStream_t s) {
    const size_t smem = sizeof(float2) * (size_t)N * (RB / 2 + 1);
    if (int rc = ensure_smem_attr((const void *)k_filter_rows_pk<RB>, (int)smem)) return rc;
    dim3 grid(ceil_div(N, kFiltThreads * kFiltOut), ceil_div(nrows, RB));
    CG_TRY(launch_after(k_filter_rows_pk<RB>, grid, kFiltThreads, smem, s, 1, in, out, h, pre,
                        nrows, N, scale, skip_ramp));
    return CG_OK;
}

template <int RB>
int launch_rb(const float *in, float *out, const float *h, const float *pre, int nrows, int N,
              float scale, bool skip_ramp, cudaStream_t s) {
    const size_t smem = sizeof(float) * (size_t)N * (RB + 1);
    if (int rc = ensure_smem_attr((const void *)k_filter_rows<RB>, (int)smem)) return rc;
    dim3 grid(ceil_div(N, kFiltThreads * kFiltOut), ceil_div(nrows, RB));
    CG_TRY(launch_after(k_filter_rows<RB>, grid, kFiltThreads, smem, s, 1, in, out, h, pre, nrows,
                        N, scale, skip_ramp));
    return CG_OK;
}

// ------------------------------------------------------------ by FFT

// The same circular convolution in O(N log N) for ramp-like taps.  These
// filters remove a row's large smooth part, so the rounding errors of its
// transform, which are relative to that part, would stand out in the result
// (7e-6 of it at 1449 cells).  The row's circular differences d[i] = s[i] -
// s[i - 1] are transformed instead and multiplied by the spectrum of g, the
// taps' circular running sums after their mean is taken off, themselves of
// mean zero (summed in pairs of floats, rounded once): sum_j s[j] h[k - j] = sum_n d[n]
// g[k - n] + mean(h) sum(s).
// The differences, packed as C >= N complex numbers z[n] = (d[2n], d[2n + 1])
// with zeros behind, give the spectrum of the zero-extended real row of M = 2C
// values (two real halves in one complex transform); g goes in at the lags
// -(N - 1) .. N - 1.  T = C / 16 threads hold a row, 16 values each:
// Cooley-Tukey passes of radix 16, 16 and C / 256 in registers with two
// exchanges through shared memory per transform (Stockham order, a pad after
// every 16 values: no bank conflicts).  Every block transforms the taps once
// (its threads keep the spectrum in registers) and tabulates the twiddle
// factors, then walks over its rows.  Rows never meet, so a row's error is
// relative to that row; a row with a value of 1e30 and more, an infinity or a
// NaN (or such taps) is summed directly, in k_filter_rows' order.
// Bound by shared-memory latency at 12 warps per SM (146 registers, 44 KB at
// 2048 values) and, for few rows, by the taps' transform (about 8 us of the
// whole).  Direct / FFT, us in a CUDA graph, rows x cells: 512 x 725 47.6 /
// 15.2, 1024 x 1449 159 / 26.5, 2048 x 2897 1030 / 69, 5000 x 512 79.5 / 30.7;
// relative error of a noisy fan-beam sinogram against 64 bits with the same
// taps 1.2e-6 / 1.6e-7 at 1449 cells, 1.5e-6 / 1.8e-7 at 2897.

// a + b of unevaluated sums of two floats (Knuth's two-sum; the low parts' own
// rounding is 2^-48 of the sum).
__device__ __forceinline__ float2 add_pair(float2 a, float2 b) {
    const float s = __fadd_rn(a.x, b.x), v = __fadd_rn(s, -a.x);
    const float e = __fadd_rn(__fadd_rn(a.x, -__fadd_rn(s, -v)), __fadd_rn(b.x, -v));
    const float lo = __fadd_rn(e, __fadd_rn(a.y, b.y));
    const float hi = __fadd_rn(s, lo);
    return make_float2(hi, __fadd_rn(lo, -__fadd_rn(hi, -s)));
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -(a.y * b.y)), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 conj2(float2 a) { return make_float2(a.x, -a.y); }

// Transforms of 2, 4, 8 and 16 values v[0], v[S], v[2 S], ... in place.
template <int S>
__device__ __forceinline__ void fft2(float2 *v) {
    const float2 a = v[0];
    v[0] = cadd(a, v[S]), v[S] = csub(a, v[S]);
}
template <int S>
__device__ __forceinline__ void fft4(float2 *v) {
    const float2 a = cadd(v[0], v[2 * S]), b = csub(v[0], v[2 * S]);
    const float2 c = cadd(v[S], v[3 * S]), d = csub(v[S], v[3 * S]);
    v[0] = cadd(a, c), v[2 * S] = csub(a, c);
    v[S] = make_float2(b.x + d.y, b.y - d.x), v[3 * S] = make_float2(b.x - d.y, b.y + d.x);
}
template <int S>
__device__ __forceinline__ void fft8(float2 *v) {
    constexpr float r = 0.70710678118654752f;
    fft4<2 * S>(v), fft4<2 * S>(v + S);
    // odd half times W8^k; outputs k, k + 4 from (even k, odd k)
    float2 o[4], e[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) e[k] = v[2 * S * k], o[k] = v[2 * S * k + S];
    o[1] = make_float2(r * (o[1].x + o[1].y), r * (o[1].y - o[1].x));
    o[2] = make_float2(o[2].y, -o[2].x);
    o[3] = make_float2(r * (o[3].y - o[3].x), -r * (o[3].x + o[3].y));
#pragma unroll
    for (int k = 0; k < 4; ++k) v[S * k] = cadd(e[k], o[k]), v[S * (k + 4)] = csub(e[k], o[k]);
}
template <int S>
__device__ __forceinline__ void fft16(float2 *v) {
    // columns n1, n1 + 4, ...; times W16^(n1 k2); rows
    constexpr float c1 = 0.92387953251128676f, s1 = 0.38268343236508977f, r = 0.70710678118654752f;
    const float2 w[10] = {{1.f, 0.f}, {c1, -s1}, {r, -r}, {s1, -c1}, {0.f, -1.f},
                          {-s1, -c1}, {-r, -r}, {-c1, -s1}, {-1.f, 0.f}, {-c1, s1}};
#pragma unroll
    for (int n = 0; n < 4; ++n) fft4<4 * S>(v + n * S);
#pragma unroll
    for (int n = 1; n < 4; ++n)
#pragma unroll
        for (int k = 1; k < 4; ++k) v[(n + 4 * k) * S] = cmul(v[(n + 4 * k) * S], w[n * k]);
    float2 t[16];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        fft4<S>(v + 4 * k * S);
#pragma unroll
        for (int m = 0; m < 4; ++m) t[k + 4 * m] = v[(4 * k + m) * S];
    }
#pragma unroll
    for (int k = 0; k < 16; ++k) v[k * S] = t[k];
}

template <int C>
struct RowFft {
    static constexpr int T = C / 16, R3 = C / 256, NB = 16 / R3;
    static constexpr int G = T < 128 ? 128 / T : 1;  // rows at a time per block
    static constexpr int kTables = 256 + C + C / 2 + 1;
    static constexpr int kRow = C + C / 16;
    static constexpr size_t smem = sizeof(float2) * (kTables + 1 + (size_t)G * kRow);
    static __device__ __forceinline__ int at(int i) { return i + (i >> 4); }

    // v[q] = value t + T q, in and out; d: the row's kRow values of shared memory
    static __device__ __forceinline__ void forward(float2 (&v)[16], float2 *d, const float2 *tb,
                                                   const float2 *tc, int t) {
        fft16<1>(v);
        __syncthreads();  // earlier reads of d
#pragma unroll
        for (int i = 0; i < 16; ++i) d[at(16 * t + i)] = v[i];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = d[at(t + T * q)];
#pragma unroll
        for (int i = 1; i < 16; ++i) v[i] = cmul(v[i], tb[i * 16 + (t & 15)]);
        fft16<1>(v);
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 16; ++i) d[at((t >> 4) * 256 + (t & 15) + 16 * i)] = v[i];
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = d[at(t + T * q)];
#pragma unroll
        for (int b = 0; b < NB; ++b) {
#pragma unroll
            for (int i = 1; i < R3; ++i) v[b + i * NB] = cmul(v[b + i * NB], tc[i * 256 + t + T * b]);
            if constexpr (R3 == 2) fft2<NB>(v + b);
            else if constexpr (R3 == 4) fft4<NB>(v + b);
            else if constexpr (R3 == 8) fft8<NB>(v + b);
            else fft16<NB>(v + b);
        }
    }
};

template <int C>
__global__ void __launch_bounds__(RowFft<C>::T *RowFft<C>::G)
    k_filter_fft(const float *__restrict__ in, float *__restrict__ out,
                 const float *__restrict__ h, const float *__restrict__ pre, int nrows, int N,
                 float scale) {
    wait_previous();
    using F = RowFft<C>;
    constexpr int T = F::T, G = F::G, M = 2 * C;
    extern __shared__ float2 fsm[];
    float2 *tb = fsm, *tc = tb + 256, *tu = tc + C;
    __shared__ int sbad[G];
    __shared__ float ssum[G][T / 32];
    const int t = threadIdx.x % T, g = threadIdx.x / T;
    float2 *d = fsm + F::kTables + 1 + g * F::kRow;
    auto twiddle = [](int e, int n) {  // exp(-2 pi i e / n), 0 <= e < n a power of two
        float sn, cs;
        sincospif(2.0f * (float)e / (float)n, &sn, &cs);
        return make_float2(cs, -sn);
    };
    if (!ramp_taps(h, N)) return;  // (the direct kernel's)
    // g as floats in d: chunks of L taps per thread, the chunks' sums scanned,
    // sums kept as unevaluated pairs of floats (64-bit units are scarce)
    auto bad = [](float x) { return !(fabsf(x) < 1e30f); };
    bool odd_taps = false;
    float *run = reinterpret_cast<float *>(d);
    float2 *chunk = tc + g * T;
    float mean_tap;
    {
        const int L = (N + T - 1) / T, l0 = min(t * L, N), l1 = min(l0 + L, N);
        float2 a = make_float2(0.f, 0.f);
        for (int l = l0; l < l1; ++l) {
            const float x = h[l];
            odd_taps = odd_taps || bad(x);
            a = add_pair(a, make_float2(x, 0.f));
        }
        chunk[t] = a;
        __syncthreads();
        for (int o = 1; o < T; o *= 2) {
            const float2 before = t >= o ? chunk[t - o] : make_float2(0.f, 0.f);
            __syncthreads();
            if (t >= o) chunk[t] = add_pair(chunk[t], before);
            __syncthreads();
        }
        const float mean = (chunk[T - 1].x + chunk[T - 1].y) / (float)N;
        const float2 first = t > 0 ? chunk[t - 1] : make_float2(0.f, 0.f);
        // the running sums' mean (about: a constant in g meets differences
        // that sum to zero), then the sums about it, rounded at their own size
        float off = 0.f;
        float2 sum = first;
        for (int l = l0; l < l1; ++l) {
            sum = add_pair(sum, make_float2(h[l], 0.f));
            off += sum.x;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) off += __shfl_xor_sync(0xffffffffu, off, o);
        if (t % 32 == 0) ssum[g][t / 32] = off;
        __syncthreads();
        off = 0.f;
#pragma unroll
        for (int w = 0; w < T / 32; ++w) off += ssum[g][w];
        off = off / (float)N - 0.5f * (float)(N + 1) * mean;
        sum = add_pair(first, make_float2(-off, 0.f));
        for (int l = l0; l < l1; ++l) {
            sum = add_pair(sum, make_float2(h[l], 0.f));
            run[l] = add_pair(sum, make_float2(-(float)(l + 1) * mean, 0.f)).x;
        }
        mean_tap = mean * scale;
    }
    const bool direct_all = __syncthreads_or(odd_taps);
    for (int e = threadIdx.x; e < 256; e += T * G) tb[e] = twiddle(((e >> 4) * (e & 15)) & 255, 256);
    for (int e = threadIdx.x; e < C; e += T * G) tc[e] = twiddle(((e >> 8) * (e & 255)) & (C - 1), C);
    for (int e = threadIdx.x; e <= C / 2; e += T * G) tu[e] = twiddle(e, M);

    // their spectrum at k = t + T m and C - k (and at C / 2), with the
    // transform's 1 / C and the scale
    float2 v[16];
    auto sum_at = [&](int m) { return m < N ? run[m] : M - m < N ? run[N - (M - m)] : 0.f; };
#pragma unroll
    for (int q = 0; q < 16; ++q)
        v[q] = make_float2(sum_at(2 * (t + T * q)), sum_at(2 * (t + T * q) + 1));
    F::forward(v, d, tb, tc, t);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) d[F::at(t + T * q)] = v[q];
    __syncthreads();
    // spectrum values X[k], X[C - k] of the real row from Z[k], Z[C - k]
    auto unpack = [&](int k, float2 &x0, float2 &x1) {
        const float2 a = d[F::at(k)], b = conj2(d[F::at((C - k) & (C - 1))]);
        const float2 e = make_float2(0.5f * (a.x + b.x), 0.5f * (a.y + b.y));
        const float2 o = cmul(tu[k], make_float2(0.5f * (a.y - b.y), -0.5f * (a.x - b.x)));
        x0 = cadd(e, o), x1 = conj2(csub(e, o));
    };
    float2 h0[9], h1[9];
    const float norm = scale / (float)C;
#pragma unroll
    for (int m = 0; m < 9; ++m) {
        unpack(m < 8 ? t + T * m : C / 2, h0[m], h1[m]);
        h0[m] = make_float2(norm * h0[m].x, norm * h0[m].y);
        h1[m] = make_float2(norm * h1[m].x, norm * h1[m].y);
    }
    for (int r0 = blockIdx.x * G; r0 < nrows; r0 += gridDim.x * G) {
        const int r = r0 + g;
        const float *row = in + (size_t)r * N;
        float *o = out + (size_t)r * N;
        bool direct = direct_all;
        float row_sum = 0.f;
        auto cell = [&](int i) {
            const float x = pre ? row[i] * pre[i] : row[i];
            direct = direct || bad(x);
            return x;
        };
        if (t == 0) sbad[g] = 0;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            v[q] = make_float2(0.f, 0.f);
            const int i = 2 * (t + T * q);
            if (q >= 8 || r >= nrows || i >= N) continue;  // N <= C: the upper half is zero
            const float s0 = cell(i > 0 ? i - 1 : N - 1), s1 = cell(i);
            v[q].x = s1 - s0, row_sum += s1;
            if (i + 1 < N) {
                const float s2 = cell(i + 1);
                v[q].y = s2 - s1, row_sum += s2;
            }
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) row_sum += __shfl_xor_sync(0xffffffffu, row_sum, o);
        if (t % 32 == 0) ssum[g][t / 32] = row_sum;
        __syncthreads();
        if (direct) sbad[g] = 1;
        F::forward(v, d, tb, tc, t);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; ++q) d[F::at(t + T * q)] = v[q];
        __syncthreads();
        // each thread its pairs (k, C - k) in place, real and imaginary parts
        // exchanged so that the forward transform goes back
        auto filter = [&](int k, float2 s0, float2 s1) {
            float2 x0, x1;
            unpack(k, x0, x1);
            const float2 p = cmul(x0, s0), q = conj2(cmul(x1, s1));
            const float2 e = make_float2(0.5f * (p.x + q.x), 0.5f * (p.y + q.y));
            const float2 f = cmul(conj2(tu[k]), make_float2(0.5f * (p.x - q.x), 0.5f * (p.y - q.y)));
            // e + i f and, at C - k, conj(e - i f)
            d[F::at((C - k) & (C - 1))] = make_float2(f.x - e.y, e.x + f.y);
            d[F::at(k)] = make_float2(e.y + f.x, e.x - f.y);
        };
#pragma unroll
        for (int m = 0; m < 8; ++m) filter(t + T * m, h0[m], h1[m]);
        if (t == 0) filter(C / 2, h0[8], h1[8]);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = d[F::at(t + T * q)];
        F::forward(v, d, tb, tc, t);
        if (r < nrows && !sbad[g]) {
            float constant = 0.f;
#pragma unroll
            for (int w = 0; w < T / 32; ++w) constant += ssum[g][w];
            constant *= mean_tap;
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int i = 2 * (t + T * q);
                if (i < N) o[i] = v[q].y + constant;
                if (i + 1 < N) o[i + 1] = v[q].x + constant;
            }
        } else if (r < nrows) {
            for (int k = t; k < N; k += T) {
                float acc = 0.f;
                for (int j = 0; j < N; ++j)
                    acc = fmaf(pre ? row[j] * pre[j] : row[j], h[k >= j ? k - j : k - j + N], acc);
                o[k] = acc * scale;
            }
        }
        __syncthreads();  // sbad, ssum
    }
}

template <int C>
int launch_fft(const float *in, float *out, const float *h, const float *pre, int nrows, int N,
               float scale, cudaStream_t s) {
    using F = RowFft<C>;
    if (int rc = ensure_smem_attr((const void *)k_filter_fft<C>, (int)F::smem)) return rc;
    // rows per block so that the resident blocks take all rows in one round
    int resident = 0;
    CG_TRY_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, k_filter_fft<C>,
                                                              F::T * F::G, F::smem));
    const int slots = std::max(1, resident * sm_count()), groups = ceil_div(nrows, F::G);
    const int blocks = ceil_div(groups, ceil_div(groups, slots));
    CG_TRY(launch_after(k_filter_fft<C>, blocks, F::T * F::G, F::smem, s, 1, in, out, h, pre,
                        nrows, N, scale));
    return CG_OK;
}

// Rows that are filtered by FFT: from 160 cells to 4096, whose tables and
// spectrum still fit a block; however many rows, so that a row's result is the
// same alone and in a stack.  Direct / FFT, us in a CUDA graph: 90 rows of 128
// cells 9.1 / 9.3; one row of 160 10.1 / 8.7, of 256 15.2 / 9.6, of 1449 92 /
// 13.3, of 4096 268 / 18.3; 47 rows 10.8 / 9.2, 15.6 / 9.6, 95 / 13.3, 272 / 18.7.
bool fft_rows(int N) { return N >= 160 && N <= 4096; }

}  // namespace

int launch_filter_rows(const float *in, float *out, const float *h, const float *pre, int nrows,
                       int N, float scale, cudaStream_t s) {
    constexpr size_t kMaxSmem = 227 * 1024;
    static const bool packed = [] {
        const char *v = getenv("CURADON_GB300_FILTER");
        return !(v && std::string(v) == "scalar");
    }();
    // ramp-like taps of long rows by FFT; the direct kernel launched after it
    // returns at once for them and does the others (the taps are known on the
    // device only)
    const bool fft = fft_rows(N);
    if (fft) {
        const int rc = N <= 512    ? launch_fft<512>(in, out, h, pre, nrows, N, scale, s)
                       : N <= 1024 ? launch_fft<1024>(in, out, h, pre, nrows, N, scale, s)
                       : N <= 2048 ? launch_fft<2048>(in, out, h, pre, nrows, N, scale, s)
                                   : launch_fft<4096>(in, out, h, pre, nrows, N, scale, s);
        if (rc) return rc;
    }
    // packed row pairs while two blocks of them fit an SM (measured: -11 % at
    // 1449 cells, -8 % at 725; at 2897 cells only one block fits, +6 %)
    if (packed && 2 * (sizeof(float) * (size_t)N * 10 + 1024) <= 228 * 1024)
        return launch_rb_pk<8>(in, out, h, pre, nrows, N, scale, fft, s);
    if (sizeof(float) * (size_t)N * 9 <= kMaxSmem)
        return launch_rb<8>(in, out, h, pre, nrows, N, scale, fft, s);
    if (sizeof(float) * (size_t)N * 5 <= kMaxSmem)
        return launch_rb<4>(in, out, h, pre, nrows, N, scale, fft, s);
    if (sizeof(float) * (size_t)N * 2 <= kMaxSmem)
        return launch_rb<1>(in, out, h, pre, nrows, N, scale, fft, s);
    return set_error(CG_ERR_INVALID, "row too long for the shared-memory filter (max 29056)");
}

}  // namespace cg
