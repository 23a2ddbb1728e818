// fwi_fft.cuh -- batched circular convolution of real sequences by FFT, in shared memory.
//
// The residual filters of compute_adjoint_source2d (apply_traces_lowpass / _bandpass,
// common.c:584-794: forward FFT, a real cosine-tapered window on the non-negative
// frequencies, inverse FFT, / n) and interpolate_traces (common.c:482-582: zero-stuffing by
// r, a rectangular band window, inverse FFT, real part / N) are, for real input, circular
// convolutions with a fixed real kernel h of the sequence length n:
//     y[i] = sum_j h[(i - j) mod n] x[j]        (interpolation: x zero-stuffed first).
// n is the trace length or the trace count (4001 and 601 on the benchmark survey: primes),
// so the kernel computes it as an M-point circular convolution, M the power of two >= 2n - 1:
// the zero-padded sequence times the spectrum G of the kernel wrapped onto M points (built
// once on the host in FP64, G = FFT_M(h wrapped) / M), which equals the n-point result on
// [0, n).  Two real sequences share one complex transform (x1 + i x2, the kernel is real).
//
// One block holds P such pairs in shared memory (P * M complex floats): the sequences are
// loaded bit-reversed, transformed by radix-2 decimation in time (natural order out),
// multiplied by G, transformed back by decimation in frequency with conjugate twiddles
// (bit-reversed order out) and written from the bit-reversed positions.  FP64 transforms where
// a block holds them (M <= 8192), FP32 above; agreement with the reference is to floating-point
// tolerance, not bitwise (its result carries its own FFT's rounding).
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace fwi {

struct ConvDesc {
    const float *in;            // input sequences: element e of sequence s at in[s * in_ss + e * in_es]
    long long in_es, in_ss;
    int n_in;                   // input samples per sequence
    int stuff;                  // zero-stuffing factor: input sample j lands on position j * stuff
    float *out;                 // output: position i of sequence s at out[s * out_ss + i * out_es]
    long long out_es, out_ss;
    int n_out;                  // positions written per sequence; positions >= N are written as 0
    int N;                      // convolution length
    int nseq;                   // sequences
    int M, logM;                // FFT size, a power of two >= 2N - 1
    int P;                      // sequence pairs per block
    int dbl;                    // 1: transforms in FP64 (G and tw double2), 0: FP32 (float2)
    const void *G;              // FFT_M of the wrapped kernel, / M
    const void *tw;             // exp(-2 pi i k / M), k < M / 2
};

template <class R> struct Cplx;
template <> struct Cplx<float> {
    typedef float2 T;
    static __device__ __forceinline__ T make(float a, float b) { return make_float2(a, b); }
};
template <> struct Cplx<double> {
    typedef double2 T;
    static __device__ __forceinline__ T make(double a, double b) { return make_double2(a, b); }
};

template <class T>
__device__ __forceinline__ T cmulc(T a, T b)
{
    T r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}

// The core of an M-point circular convolution of the P sequences in fbuf (each loaded at its
// bit-reversed positions): radix-2 decimation in time (natural order out), multiplication by the
// spectrum G (which carries the 1 / M), and the inverse by decimation in frequency with conjugate
// twiddles (bit-reversed order out).  Every thread of the block takes part.
template <class R>
__device__ __forceinline__ void fft_conv_core(typename Cplx<R>::T *fbuf, int P, int M, int logM,
                                              const typename Cplx<R>::T *G, const typename Cplx<R>::T *tw)
{
    typedef typename Cplx<R>::T C;
    const int tid = threadIdx.x, nth = blockDim.x, half_M = M >> 1;
    for (int len = 2, lg = 1; len <= M; len <<= 1, ++lg) {
        const int half = len >> 1, tstep = M >> lg;
        for (int b = tid; b < P * half_M; b += nth) {
            const int q = b / half_M, bb = b - q * half_M;
            const int p = bb & (half - 1), i = ((bb >> (lg - 1)) << lg) + p, j = i + half;
            C *f = fbuf + q * M;
            const C t = cmulc(tw[p * tstep], f[j]), a = f[i];
            f[i] = Cplx<R>::make(a.x + t.x, a.y + t.y);
            f[j] = Cplx<R>::make(a.x - t.x, a.y - t.y);
        }
        __syncthreads();
    }
    for (int i = tid; i < P * M; i += nth) fbuf[i] = cmulc(fbuf[i], G[i & (M - 1)]);
    __syncthreads();
    for (int len = M, lg = logM; len >= 2; len >>= 1, --lg) {
        const int half = len >> 1, tstep = M >> lg;
        for (int b = tid; b < P * half_M; b += nth) {
            const int q = b / half_M, bb = b - q * half_M;
            const int p = bb & (half - 1), i = ((bb >> (lg - 1)) << lg) + p, j = i + half;
            C *f = fbuf + q * M;
            const C w = tw[p * tstep], a = f[i], c = f[j];
            f[i] = Cplx<R>::make(a.x + c.x, a.y + c.y);
            f[j] = cmulc(Cplx<R>::make(a.x - c.x, a.y - c.y), Cplx<R>::make(w.x, -w.y));
        }
        __syncthreads();
    }
}

// grid: ceil(nseq / (2 P)) blocks; dynamic shared memory P * M complex values of type R
template <class R>
static __global__ void __launch_bounds__(512) k_fft_conv(const ConvDesc d)
{
    typedef typename Cplx<R>::T C;
    extern __shared__ __align__(16) unsigned char fsm[];
    C *fbuf = reinterpret_cast<C *>(fsm);
    const C *G = static_cast<const C *>(d.G), *tw = static_cast<const C *>(d.tw);
    const int M = d.M, P = d.P;
    const int s0 = blockIdx.x * 2 * P;  // first sequence of the block
    const int tid = threadIdx.x, nth = blockDim.x;
    for (int i = tid; i < P * M; i += nth) fbuf[i] = Cplx<R>::make(0, 0);
    __syncthreads();
    // load: pair q holds sequences s0 + 2q (real part) and s0 + 2q + 1 (imaginary part); the
    // sequence index runs fastest so that neighbouring threads read neighbouring addresses when
    // the sequences interleave (in_ss == 1)
    const int nsb = min(2 * P, d.nseq - s0);
    for (int t = tid; t < d.n_in * nsb; t += nth) {
        const int j = t / nsb, sl = t % nsb;
        const float v = d.in[(long long)(s0 + sl) * d.in_ss + (long long)j * d.in_es];
        const unsigned pos = __brev((unsigned)(j * d.stuff)) >> (32 - d.logM);
        R *c = reinterpret_cast<R *>(&fbuf[(sl >> 1) * M + pos]);
        c[sl & 1] = (R)v;
    }
    __syncthreads();
    fft_conv_core<R>(fbuf, P, M, d.logM, G, tw);
    for (int t = tid; t < d.n_out * nsb; t += nth) {
        const int i = t / nsb, sl = t % nsb;
        float v = 0.f;
        if (i < d.N) {
            const unsigned pos = __brev((unsigned)i) >> (32 - d.logM);
            const R *c = reinterpret_cast<const R *>(&fbuf[(sl >> 1) * M + pos]);
            v = (float)c[sl & 1];
        }
        d.out[(long long)(s0 + sl) * d.out_ss + (long long)i * d.out_es] = v;
    }
}

// ---------------------------------------------------------------- block transforms in radix-8 passes
// The wavenumber filter's convolutions, one sequence to a block: decimation in frequency with radix-8
// butterflies in registers (natural order in, digit-reversed out), multiplication by a spectrum kept in
// that order (fft_order), and back by decimation in time with conjugate twiddles.  What takes the time
// is shared-memory passes and the FP64 pipe, so passes are merged: the first, of radix 2^LR (logM = LR +
// 3 q), runs from the loads, whose upper half is zero; the last forward pass, the multiplication and the
// first inverse pass keep their eight values in registers; the last pass runs into the stores, of which
// only the lower half exists.  Per convolution that is 2 q - 1 passes over shared memory where radix 2
// takes 2 logM + 3 (7 against 29 for 8192 points).  One element in nine is padding against bank
// conflicts.  Where the block's memory holds the points only in FP32 (M > 8192) they are FP32 there and FP64
// in the passes: the points are then rounded once per pass.  With FP32 passes the error against 64
// bits of a transform and its inverse, 5001 points padded to 16384, was 4.6e-7 of the norm and with
// every factor read from the table 2.0e-7; radix-2 FP32 transforms of all z wavenumbers, whose independent
// errors the real part halves in energy, had 1.7e-7, and this has 6.2e-8.
// (The residual filters above keep the radix-2 order: a filtered residual far below the
// source's band is so small a difference that another order of the same FP64 operations moves the
// gradient by 6e-5, as much as FP32 rounding does.)
template <class T>
__device__ __forceinline__ T cadd(T a, T b)
{
    a.x += b.x;
    a.y += b.y;
    return a;
}
template <class T>
__device__ __forceinline__ T csub(T a, T b)
{
    a.x -= b.x;
    a.y -= b.y;
    return a;
}
// a * (S i)
template <int S, class T>
__device__ __forceinline__ T cmuli(T a)
{
    T r;
    r.x = S < 0 ? a.y : -a.y;
    r.y = S < 0 ? -a.x : a.x;
    return r;
}
template <class T>
__device__ __forceinline__ T conjc(T a)
{
    a.y = -a.y;
    return a;
}

// DFT of 2^LR values in registers, sign S (-1 forward)
template <int LR, int S, class T>
__device__ __forceinline__ void dft(T *x)
{
    if constexpr (LR == 1) {
        const T a = x[0], b = x[1];
        x[0] = cadd(a, b);
        x[1] = csub(a, b);
    } else if constexpr (LR == 2) {
        const T t0 = cadd(x[0], x[2]), t1 = csub(x[0], x[2]), t2 = cadd(x[1], x[3]);
        const T t3 = cmuli<S>(csub(x[1], x[3]));
        x[0] = cadd(t0, t2);
        x[2] = csub(t0, t2);
        x[1] = cadd(t1, t3);
        x[3] = csub(t1, t3);
    } else {
        T e[4] = {x[0], x[2], x[4], x[6]}, o[4] = {x[1], x[3], x[5], x[7]};
        dft<2, S>(e);
        dft<2, S>(o);
        const auto c = (decltype(x[0].x))0.70710678118654752440;
        const T o1 = o[1], o3 = o[3];
        // e^{S i pi / 4} and e^{S 3 i pi / 4}
        o[1].x = c * (o1.x - S * o1.y);
        o[1].y = c * (o1.y + S * o1.x);
        o[2] = cmuli<S>(o[2]);
        o[3].x = c * (-o3.x - S * o3.y);
        o[3].y = c * (S * o3.x - o3.y);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            x[k] = cadd(e[k], o[k]);
            x[k + 4] = csub(e[k], o[k]);
        }
    }
}
// x[k] *= w^k
template <int LR, class T>
__device__ __forceinline__ void twiddle(T *x, T w)
{
    if constexpr (LR >= 2) {
        const T w2 = cmulc(w, w);
        if constexpr (LR == 3) {
            const T w4 = cmulc(w2, w2);
            x[7] = cmulc(x[7], cmulc(w4, cmulc(w2, w)));
            x[6] = cmulc(x[6], cmulc(w4, w2));
            x[5] = cmulc(x[5], cmulc(w4, w));
            x[4] = cmulc(x[4], w4);
        }
        x[3] = cmulc(x[3], cmulc(w2, w));
        x[2] = cmulc(x[2], w2);
    }
    x[1] = cmulc(x[1], w);
}

// a block's transform: M points in shared memory as complex ST, passes and tables in FP64
template <class ST, int LR>
struct FftBlock {
    typedef double2 C;
    typename Cplx<ST>::T *f;
    int M, logM;
    const C *tw;
    __device__ __forceinline__ C get(int e) const
    {
        const auto v = f[e + (e >> 3)];
        return make_double2(v.x, v.y);
    }
    __device__ __forceinline__ void put(int e, C v) { f[e + (e >> 3)] = Cplx<ST>::make((ST)v.x, (ST)v.y); }

    // first pass from load(e), e < M / 2 (the rest is zero)
    template <class Load>
    __device__ __forceinline__ void first(Load load)
    {
        const int s = M >> LR;
        for (int i = threadIdx.x; i < s; i += blockDim.x) {
            C x[1 << LR];
#pragma unroll
            for (int k = 0; k < 1 << LR; ++k) x[k] = 2 * k < (1 << LR) ? load(i + k * s) : make_double2(0, 0);
            dft<LR, -1>(x);
            twiddle<LR>(x, tw[i]);
#pragma unroll
            for (int k = 0; k < 1 << LR; ++k) put(i + k * s, x[k]);
        }
        __syncthreads();
    }
    // last pass into store(e, value), e < M / 2
    template <class Store>
    __device__ __forceinline__ void last(Store store)
    {
        const int s = M >> LR;
        for (int i = threadIdx.x; i < s; i += blockDim.x) {
            C x[1 << LR];
#pragma unroll
            for (int k = 0; k < 1 << LR; ++k) x[k] = get(i + k * s);
            twiddle<LR>(x, conjc(tw[i]));
            dft<LR, 1>(x);
#pragma unroll
            for (int k = 0; 2 * k < 1 << LR; ++k) store(i + k * s, x[k]);
        }
    }
    // the last pass of one convolution and the first of the next on the same thread's elements:
    // map(e, value) in between, e < M / 2
    template <class Map>
    __device__ __forceinline__ void last_first(Map map)
    {
        const int s = M >> LR;
        for (int i = threadIdx.x; i < s; i += blockDim.x) {
            C x[1 << LR];
#pragma unroll
            for (int k = 0; k < 1 << LR; ++k) x[k] = get(i + k * s);
            const C w = tw[i];
            twiddle<LR>(x, conjc(w));
            dft<LR, 1>(x);
#pragma unroll
            for (int k = 0; k < 1 << LR; ++k) x[k] = 2 * k < (1 << LR) ? map(i + k * s, x[k]) : make_double2(0, 0);
            dft<LR, -1>(x);
            twiddle<LR>(x, w);
#pragma unroll
            for (int k = 0; k < 1 << LR; ++k) put(i + k * s, x[k]);
        }
        __syncthreads();
    }
    // between the first and the last pass: the remaining transforms and the multiplication by G
    __device__ __forceinline__ void inner(const C *__restrict__ G)
    {
        const int top = logM - LR;  // log2 of the transforms left, a multiple of three
        if (top == 0) {
            for (int e = threadIdx.x; e < M; e += blockDim.x) put(e, cmulc(get(e), G[e]));
            __syncthreads();
            return;
        }
        for (int lg = top; lg > 3; lg -= 3) pass<-1>(lg);
        for (int b = threadIdx.x; b < M >> 3; b += blockDim.x) {
            const int e = b << 3;
            C x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = get(e + k);
            dft<3, -1>(x);
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = cmulc(x[k], G[e + k]);
            dft<3, 1>(x);
#pragma unroll
            for (int k = 0; k < 8; ++k) put(e + k, x[k]);
        }
        __syncthreads();
        for (int lg = 6; lg <= top; lg += 3) pass<1>(lg);
    }
    // one radix-8 pass of the 2^lg-point transforms: forward butterflies then twiddles, or back
    template <int S>
    __device__ __forceinline__ void pass(int lg)
    {
        const int s = 1 << (lg - 3);
        for (int b = threadIdx.x; b < M >> 3; b += blockDim.x) {
            const int j = b & (s - 1);
            const int e = ((b >> (lg - 3)) << lg) + j;
            const C w = tw[j << (logM - lg)];
            C x[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) x[k] = get(e + k * s);
            if (S > 0) twiddle<3>(x, conjc(w));
            dft<3, S>(x);
            if (S < 0) twiddle<3>(x, w);
#pragma unroll
            for (int k = 0; k < 8; ++k) put(e + k * s, x[k]);
        }
        __syncthreads();
    }
};

// ---------------------------------------------------------------- 2-D wavenumber filter (Bluestein)
// An N-point DFT X_k = sum_j x_j e^{-2 pi i jk / N} is conj(b_k) times the convolution of
// u_j = x_j conj(b_j) with b, b_m = e^{i pi m^2 / N} (jk = (j^2 + k^2 - (k - j)^2) / 2); the inverse
// direction (e^{+2 pi i jk / N}) uses the conjugate chirps.  The convolution runs as the M-point
// one above (M the power of two >= 2N - 1) with the spectrum of b wrapped onto M points.
// The filter of a real nz x nx field, padded by `pad` replicated samples on every side to Nz x Nx, in
// three launches (WaveDesc::stage):
//   0  z transforms of the model's nx columns -- a padded column's is that of the edge column it
//      replicates -- two real columns to a transform, kept for wavenumbers 0 .. Nz/2
//   1  for each of these z wavenumbers (the others' result is the conjugate): the x transform of the
//      padded row, the window, and the inverse x transform in the same block, kept at the model's
//      columns; the chirp that ends the first and the one that starts the second multiply to 1
//   2  inverse z transforms, two columns to a transform (their real and imaginary parts), kept at the
//      model's rows, / (Nz Nx)
// Measured, 221 x 601 padded to 1821 x 2201 (B200): 33, 279 and 29 us, bound by the FP64 pipe and
// shared memory; with radix-2 passes, all padded columns and all z wavenumbers the call took 3.3 ms, 0.6
// now.
struct WaveDesc {
    const float *x;         // [nx][nz] model field (tapered)
    float2 *A, *Gc;         // [Nz/2 + 1][nx] spectra along z; [nx][Nz/2 + 1] filtered
    const float *win;       // [Nz/2 + 1][Nx] window
    float *y;               // [nx][nz] filtered field
    int nz, nx, pad;
    float divisor;          // Nz * Nx
    int N, M, logM;         // DFT length (Nz, Nx, Nz) and convolution size of the stage
    const void *tables;     // fwi_bluestein_tables: chirp (N), spectrum of b (M), of conj(b) (M) in fft_order
    const void *tw;         // exp(-2 pi i k / M), k < M / 2
};

// one transform per block
template <class ST, int LR, int STAGE>
static __global__ void __launch_bounds__(512) k_wavenumber(const WaveDesc d)
{
    typedef double R;
    typedef double2 C;
    extern __shared__ __align__(16) unsigned char fsm[];
    FftBlock<ST, LR> B{reinterpret_cast<typename Cplx<ST>::T *>(fsm), d.M, d.logM, static_cast<const C *>(d.tw)};
    const C *chirp = static_cast<const C *>(d.tables), *Bf = chirp + d.N, *Bi = Bf + d.M;
    const C zero = Cplx<R>::make(0, 0);
    const int N = d.N, b = blockIdx.x, c0 = 2 * b;
    if (STAGE == 0) {
        const bool two = c0 + 1 < d.nx;
        const float *p = d.x + (long long)c0 * d.nz;
        B.first([&](int e) {
            if (e >= N) return zero;
            const int z = min(max(e - d.pad, 0), d.nz - 1);
            return cmulc(Cplx<R>::make((R)p[z], two ? (R)p[d.nz + z] : (R)0), conjc(chirp[e]));
        });
        B.inner(Bf);
        B.last([&](int e, C v) {
            if (e < N) B.put(e, cmulc(v, conjc(chirp[e])));  // the thread's own elements
        });
        __syncthreads();
        for (int k = threadIdx.x; k <= N / 2; k += blockDim.x) {
            const C u = B.get(k), v = conjc(B.get(k ? N - k : 0));
            d.A[(long long)k * d.nx + c0] = make_float2((float)((R)0.5 * (u.x + v.x)), (float)((R)0.5 * (u.y + v.y)));
            if (two)
                d.A[(long long)k * d.nx + c0 + 1] =
                    make_float2((float)((R)0.5 * (u.y - v.y)), (float)((R)-0.5 * (u.x - v.x)));
        }
    } else if (STAGE == 1) {
        const float2 *p = d.A + (long long)b * d.nx;
        const float *w = d.win + (long long)b * N;
        B.first([&](int e) {
            if (e >= N) return zero;
            const float2 v = p[min(max(e - d.pad, 0), d.nx - 1)];
            return cmulc(Cplx<R>::make(v.x, v.y), conjc(chirp[e]));
        });
        B.inner(Bf);
        B.last_first([&](int e, C v) {
            const R g = e < N ? (R)w[e] : (R)0;
            return Cplx<R>::make(v.x * g, v.y * g);
        });
        B.inner(Bi);
        B.last([&](int e, C v) {
            const int c = e - d.pad;
            if (c < 0 || c >= d.nx) return;
            v = cmulc(v, chirp[e]);
            d.Gc[(long long)c * gridDim.x + b] = make_float2((float)v.x, (float)v.y);
        });
    } else {
        const bool two = c0 + 1 < d.nx;
        const int nk = N / 2 + 1;
        const float2 *p = d.Gc + (long long)c0 * nk;
        B.first([&](int e) {
            if (e >= N) return zero;
            const int k = e <= N / 2 ? e : N - e;
            const R sg = e <= N / 2 ? 1 : -1;
            const float2 g = p[k], h = two ? p[nk + k] : make_float2(0.f, 0.f);
            // g + i h of the full spectra
            return cmulc(Cplx<R>::make((R)g.x - sg * (R)h.y, sg * (R)g.y + (R)h.x), chirp[e]);
        });
        B.inner(Bi);
        B.last([&](int e, C v) {
            const int z = e - d.pad;
            if (z < 0 || z >= d.nz) return;
            v = cmulc(v, chirp[e]);
            float *o = d.y + (long long)c0 * d.nz + z;
            o[0] = (float)v.x / d.divisor;
            if (two) o[d.nz] = (float)v.y / d.divisor;
        });
    }
}

constexpr int FFT_CONV_MAX = 16384;      // largest M one block holds in FP32 (144 KB of shared memory)
constexpr int FFT_CONV_MAX_F64 = 8192;   // largest M one block holds in FP64 (144 KB)

// The transforms run in FP64 where the block holds them (M <= 8192): the filtered residual can
// be much smaller than the residual (a low-pass far below the source's band), and an FP32
// transform's rounding, relative to the input, then shows in the output.
static inline bool conv_in_f64(int M) { return M <= FFT_CONV_MAX_F64; }

static inline int fft_log2(int M)
{
    int lg = 0;
    while ((1 << lg) < M) lg++;
    return lg;
}
// radix 2^fft_lead of the first and last pass
static inline int fft_lead(int logM) { return logM % 3 ? logM % 3 : 3; }
static inline size_t fft_smem(int M, bool dbl) { return (size_t)(M + M / 8 + 1) * (dbl ? 16 : 8); }
static inline int fft_threads(int M)
{
    const int t = (M >> 4) / 32 * 32;  // two butterflies per thread and pass
    return t < 64 ? 64 : t > 512 ? 512 : t;
}

// M values from frequency order into the order the forward passes leave them in: position
// k1 (M >> LR) + k2 (M >> LR >> 3) + .. holds frequency k1 + 2^LR (k2 + 8 (k3 + ..))
template <class T>
static inline void fft_order(T *g, int M)
{
    const int logM = fft_log2(M);
    std::vector<T> a(g, g + M);
    for (int pos = 0; pos < M; pos++) {
        int f = 0, sh = 0, left = logM;
        for (int r = fft_lead(logM); left > 0; r = 3) {
            left -= r;
            f |= ((pos >> left) & ((1 << r) - 1)) << sh;
            sh += r;
        }
        g[pos] = a[f];
    }
}

template <class F>
static inline cudaError_t fft_launch(F fn, const void *attr_fn, size_t smem)
{
    cudaError_t e = cudaFuncSetAttribute(attr_fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    fn();
    return cudaGetLastError();
}

// fills M, logM and P of d (M from d.N, as fwi_conv_size) and launches; cudaErrorInvalidValue when
// M > FFT_CONV_MAX, the sizes do not fit, or d.dbl does not match conv_in_f64(M)
static inline cudaError_t launch_fft_conv(ConvDesc d, cudaStream_t st)
{
    int M = 2, lg = 1;  // the size fwi_conv_size gives, for which G and tw were built
    while (M < 2 * d.N - 1) M <<= 1, ++lg;
    if (M > FFT_CONV_MAX || d.N < 1 || d.nseq < 1 || d.n_in < 1 || (d.n_in - 1) * d.stuff >= d.N ||
        (d.dbl != 0) != conv_in_f64(M))
        return cudaErrorInvalidValue;
    d.M = M;
    d.logM = lg;
    const size_t csize = d.dbl ? 16 : 8;
    d.P = M >= 8192 ? 1 : 8192 / M;  // up to 64 KB (FP32) / 128 KB (FP64) of pairs per block
    d.P = d.P < (d.nseq + 1) / 2 ? d.P : (d.nseq + 1) / 2;
    const size_t smem = (size_t)d.P * M * csize;
    const void *fn = d.dbl ? (const void *)k_fft_conv<double> : (const void *)k_fft_conv<float>;
    cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const int blocks = (d.nseq + 2 * d.P - 1) / (2 * d.P);
    if (d.dbl) k_fft_conv<double><<<blocks, 512, smem, st>>>(d);
    else k_fft_conv<float><<<blocks, 512, smem, st>>>(d);
    return cudaGetLastError();
}

// one stage of the wavenumber filter; d.N and its tables are set, blocks transforms are launched
template <int STAGE>
static inline cudaError_t launch_wavenumber(WaveDesc d, int blocks, cudaStream_t st)
{
    int M = 2, lg = 1;
    while (M < 2 * d.N - 1) M <<= 1, ++lg;
    if (M > FFT_CONV_MAX || d.N < 1 || blocks < 1) return cudaErrorInvalidValue;
    d.M = M;
    d.logM = lg;
    const bool dbl = conv_in_f64(M);
    const size_t smem = fft_smem(M, dbl);
    const int threads = fft_threads(M);
    auto go = [&](auto kernel) {
        return fft_launch([&] { kernel<<<blocks, threads, smem, st>>>(d); }, (const void *)kernel, smem);
    };
    static_assert(FFT_CONV_MAX == 2 * FFT_CONV_MAX_F64, "one size, 2^14 points, in FP32");
    if (!dbl) return go(k_wavenumber<float, 2, STAGE>);
    switch (fft_lead(lg)) {
    case 1: return go(k_wavenumber<double, 1, STAGE>);
    case 2: return go(k_wavenumber<double, 2, STAGE>);
    default: return go(k_wavenumber<double, 3, STAGE>);
    }
}

}  // namespace fwi
