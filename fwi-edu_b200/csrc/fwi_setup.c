/*
 * fwi_setup.c -- host-side set-up of the B200 engine: what the reference evaluates with the C library's
 * expf, logf, powf and cosf.
 *
 * The absorbing layers' weights and reflection coefficient (mealCoefs2d, propagation.c:192-354; the
 * coefficient fields themselves are formed on the device from them, fwi_coef.cuh), the model
 * operations of the FWI loop (Gardner's relation), taper and filter windows, and the FP64 tables of
 * the FFT kernels.  Keeping the reference's operation order with the same libm gives identical bits.
 * The file is compiled with -O2 -fno-fast-math -ffp-contract=off.
 */
#include <math.h>
#include <stdlib.h>
#include <string.h>
#include "fwi_setup.h"

int fwi_ck_interval(int nt)
{
    float r = roundf(sqrtf(2.0f * (nt - 1)));
    return (int)(r > 3.0f ? r : 3.0f);
}

int fwi_ck_count(int nt)
{
    int d = fwi_ck_interval(nt), n = 0;
    for (int it = 0; it < nt; it++) n += (it % d == 0 || (it + 1) % d == 0);
    return n;
}

void fwi_taper_coefs(int L, float *out)
{
    for (int i = 0; i <= L; i++) {
        float x = (float)3.141592653589793 * i / L;
        out[i] = 0.5f * (1.0f + cosf(x));
    }
}

/* the absorbing-layer weight of layer l of n: 2^(d^alpha) - 1, d = l/n (propagation.c:173-190) */
static float layer_weight(float alpha, int l, int n)
{
    float d = (0.1f * l) / (0.1f * n);
    return expf(logf(2.0f) * powf(d, alpha)) - 1.0f;
}

float fwi_layer_weights(int pml, float *out)
{
    const float pd = 2.0f, alpha = 2.5f;
    const float Rcoef = powf(10.0f, -1.0f * ((log10f(pml) - 1.0f) / (log10f(2.0f))) - 3.0f - 0.5f * pd);
    for (int l = 1; l <= pml; l++) out[l - 1] = layer_weight(alpha, l, pml);
    return logf(Rcoef);
}

/* set_waterlayer_value, clip_model, v2slow/slow2v, vp2density (common.c:218-330, 898-924) */
static void water_layer(float *m, float v, int wd, int nx, int nz)
{
    for (int ix = 0; ix < nx; ix++)
        for (int iz = 0; iz < wd; iz++) m[(size_t)ix * nz + iz] = v;
}
static void clip(float *m, size_t n, float lo, float hi)
{
    for (size_t i = 0; i < n; i++) {
        if (m[i] > hi) m[i] = hi;
        else if (m[i] < lo) m[i] = lo;
    }
}
static void reciprocal(const float *a, float *b, size_t n)
{
    for (size_t i = 0; i < n; i++) b[i] = a[i] != 0.0f ? 1.0f / a[i] : 0.0f;
}
static void gardner(const float *vp, float *rho, size_t n)
{
    for (size_t i = 0; i < n; i++) rho[i] = 310.0f * powf(vp[i], 0.25f);
}

void fwi_model_trial(const float *slow, const float *perturb, float *vp, float *rho, int nx, int nz, int waterdepth,
                     float vp_water, float rho_water, float vpmin, float vpmax, float rhomin, float rhomax, int g)
{
    size_t n = (size_t)nx * nz;
    for (size_t i = 0; i < n; i++) vp[i] = slow[i] + perturb[i];
    reciprocal(vp, vp, n);
    water_layer(vp, vp_water, waterdepth, nx, nz);
    clip(vp, n, vpmin, vpmax);
    if (g == 1) {
        gardner(vp, rho, n);
        water_layer(rho, rho_water, waterdepth, nx, nz);
        clip(rho, n, rhomin, rhomax);
    }
}

void fwi_model_update(float *slow, float *vp, float *rho, const float *perturb, float steplen, int nx, int nz,
                      int waterdepth, float vp_water, float rho_water, float vpmin, float vpmax, float rhomin,
                      float rhomax, int g)
{
    size_t n = (size_t)nx * nz;
    for (size_t i = 0; i < n; i++) slow[i] = slow[i] + steplen * perturb[i];
    reciprocal(slow, vp, n);
    water_layer(vp, vp_water, waterdepth, nx, nz);
    clip(vp, n, vpmin, vpmax);
    if (g == 1) {
        gardner(vp, rho, n);
        water_layer(rho, rho_water, waterdepth, nx, nz);
        clip(rho, n, rhomin, rhomax);
    }
    reciprocal(vp, slow, n);
}

/* ------------------------------------------------------------ residual filters, interpolation */
/* The window values come from the reference's own float expressions (apply_traces_lowpass and
 * apply_traces_bandpass; the bandpass forms its cosine argument in double because PI is a double
 * constant there).  Only entries 0..n/2 are used (the non-negative frequencies of an r2c FFT). */
void fwi_filter_window(int filter, int n, float fpass, float fcut, float dt, float *win)
{
    const float df = 1.0f / (n * dt);
    for (int it = 0; it < n; it++) {
        const float f = it * df;
        if (filter == 0) {
            const float taperLen = fcut - fpass;
            if (f < fpass) win[it] = 1.0f;
            else if (f >= fpass && f <= fcut)
                win[it] = 0.5f * (1.0f + cosf((float)3.141592653589793 * (f - fpass) / taperLen));
            else win[it] = 0.0f;
        } else {
            const float lo = fpass, hi = fcut - fpass;
            if (f < fpass) win[it] = 0.5f * (1.0f + cosf(3.141592653589793 * (fpass - f) / lo));
            else if (f >= fpass && f <= fcut) win[it] = 0.5f * (1.0f + cosf(3.141592653589793 * (f - fpass) / hi));
            else win[it] = 0.0f;
        }
    }
}

/* h[m] = (1/n) sum_k W(k) cos(2 pi k m / n) with W(k) = win[min(k, n - k)] (the real window seen
 * by a real signal's full spectrum), in double; k m mod n is stepped incrementally */
static void circular_kernel(const float *win, int n, double *h)
{
    double *cs = (double *)malloc(sizeof(double) * (size_t)n);
    for (int m = 0; m < n; m++) cs[m] = cos(2.0 * 3.141592653589793 * m / n);
    for (int m = 0; m < n; m++) {
        double a = 0.0;
        int idx = 0;
        for (int k = 0; k < n; k++) {
            a += (double)win[k <= n / 2 ? k : n - k] * cs[idx];
            idx += m;
            if (idx >= n) idx -= n;
        }
        h[m] = a / n;
    }
    free(cs);
}

void fwi_filter_operator(int filter, int n, float fpass, float fcut, float dt, float *C)
{
    float *win = (float *)malloc(sizeof(float) * (size_t)n);
    double *h = (double *)malloc(sizeof(double) * (size_t)n);
    fwi_filter_window(filter, n, fpass, fcut, dt, win);
    circular_kernel(win, n, h);
    for (int j = 0; j < n; j++)
        for (int i = 0; i < n; i++) C[(size_t)j * n + i] = (float)h[(i - j + n) % n];
    free(win);
    free(h);
}

/* ------------------------------------------------------------ FFT convolution spectra */
/* in-place radix-2 FFT of n = 2^k complex doubles (sign -1: forward, +1: inverse, unscaled) */
static void fft_pow2(double *re, double *im, int n, int sign)
{
    for (int i = 1, j = 0; i < n; i++) { /* bit reversal */
        int bit = n >> 1;
        for (; j & bit; bit >>= 1) j ^= bit;
        j ^= bit;
        if (i < j) {
            double t = re[i]; re[i] = re[j]; re[j] = t;
            t = im[i]; im[i] = im[j]; im[j] = t;
        }
    }
    for (int len = 2; len <= n; len <<= 1) {
        const double ang = sign * 2.0 * 3.141592653589793 / len;
        for (int k = 0; k < len / 2; k++) {
            const double wr = cos(ang * k), wi = sin(ang * k);
            for (int i = k; i < n; i += len) {
                const int j = i + len / 2;
                const double xr = re[j] * wr - im[j] * wi, xi = re[j] * wi + im[j] * wr;
                re[j] = re[i] - xr; im[j] = im[i] - xi;
                re[i] += xr; im[i] += xi;
            }
        }
    }
}

int fwi_conv_size(int n)
{
    int M = 2;
    while (M < 2 * n - 1) M <<= 1;
    return M;
}

void fwi_conv_spectrum(const double *h, int n, int M, float *G)
{
    double *re = (double *)calloc((size_t)M, sizeof(double)), *im = (double *)calloc((size_t)M, sizeof(double));
    for (int m = 0; m < n; m++) re[m] = h[m];
    for (int m = 1; m < n; m++) re[M - m] = h[n - m];
    fft_pow2(re, im, M, -1);
    for (int k = 0; k < M; k++) {
        G[2 * k] = (float)(re[k] / M);
        G[2 * k + 1] = (float)(im[k] / M);
    }
    free(re);
    free(im);
}

void fwi_conv_spectrum_f64(const double *h, int n, int M, double *G)
{
    double *re = (double *)calloc((size_t)M, sizeof(double)), *im = (double *)calloc((size_t)M, sizeof(double));
    for (int m = 0; m < n; m++) re[m] = h[m];
    for (int m = 1; m < n; m++) re[M - m] = h[n - m];
    fft_pow2(re, im, M, -1);
    for (int k = 0; k < M; k++) {
        G[2 * k] = re[k] / M;
        G[2 * k + 1] = im[k] / M;
    }
    free(re);
    free(im);
}

void fwi_bluestein_tables(int N, int M, double *out)
{
    double *br = (double *)malloc(sizeof(double) * (size_t)N), *bi = (double *)malloc(sizeof(double) * (size_t)N);
    for (int m = 0; m < N; m++) {
        /* m^2 mod 2N keeps the angle small (the chirp has period 2N in m^2) */
        const long long q = ((long long)m * m) % (2LL * N);
        const double a = 3.141592653589793 * (double)q / N;
        br[m] = cos(a);
        bi[m] = sin(a);
    }
    double *re = (double *)calloc((size_t)M, sizeof(double)), *im = (double *)calloc((size_t)M, sizeof(double));
    double *spec = (double *)malloc(sizeof(double) * 4 * (size_t)M);
    for (int c = 0; c < 2; c++) {  /* c = 0: b, c = 1: conj(b) */
        memset(re, 0, sizeof(double) * (size_t)M);
        memset(im, 0, sizeof(double) * (size_t)M);
        const double sg = c ? -1.0 : 1.0;
        for (int m = 0; m < N; m++) {
            re[m] = br[m];
            im[m] = sg * bi[m];
            if (m > 0) {
                re[M - m] = br[m];
                im[M - m] = sg * bi[m];
            }
        }
        fft_pow2(re, im, M, -1);
        for (int k = 0; k < M; k++) {
            spec[(size_t)c * 2 * M + 2 * k] = re[k] / M;
            spec[(size_t)c * 2 * M + 2 * k + 1] = im[k] / M;
        }
    }
    for (int m = 0; m < N; m++) out[2 * m] = br[m], out[2 * m + 1] = bi[m];
    memcpy(out + 2 * (size_t)N, spec, sizeof(double) * 4 * (size_t)M);
    free(br);
    free(bi);
    free(re);
    free(im);
    free(spec);
}

void fwi_fft_twiddles_f64(int M, double *tw)
{
    for (int k = 0; k < M / 2; k++) {
        const double a = 2.0 * 3.141592653589793 * k / M;
        tw[2 * k] = cos(a);
        tw[2 * k + 1] = -sin(a);
    }
}

void fwi_fft_twiddles(int M, float *tw)
{
    for (int k = 0; k < M / 2; k++) {
        const double a = 2.0 * 3.141592653589793 * k / M;
        tw[2 * k] = (float)cos(a);
        tw[2 * k + 1] = (float)-sin(a);
    }
}

void fwi_filter_kernel(int filter, int n, float fpass, float fcut, float dt, double *h)
{
    float *win = (float *)malloc(sizeof(float) * (size_t)n);
    fwi_filter_window(filter, n, fpass, fcut, dt, win);
    circular_kernel(win, n, h);
    free(win);
}

void fwi_interp_kernel(int ns, int r, double *g)
{
    const int N = (ns - 1) * r + 1, nkeep = N / (2 * r);
    float *win = (float *)calloc((size_t)N, sizeof(float));
    for (int k = 0; k < nkeep; k++) win[k] = (float)r;
    for (int k = N - nkeep + 1; k < N; k++) win[k] = (float)r;
    double *cs = (double *)malloc(sizeof(double) * (size_t)N);
    for (int m = 0; m < N; m++) cs[m] = cos(2.0 * 3.141592653589793 * m / N);
    for (int m = 0; m < N; m++) {
        double a = 0.0;
        int idx = 0;
        for (int k = 0; k < N; k++) {
            a += (double)win[k] * cs[idx];
            idx += m;
            if (idx >= N) idx -= N;
        }
        g[m] = a / N;
    }
    free(win);
    free(cs);
}

/* zero-stuffing by r, a rectangular window of height r on |k| < N / (2r) of the length-N
 * spectrum (N = (ns - 1) r + 1), inverse FFT, real part / N:  y[i] = sum_j x[j] g[(i - j r) mod N] */
void fwi_interp_operator(int ns, int r, int nt, float *M)
{
    const int N = (ns - 1) * r + 1, nkeep = N / (2 * r);
    float *win = (float *)calloc((size_t)N, sizeof(float));
    for (int k = 0; k < nkeep; k++) win[k] = (float)r;
    for (int k = N - nkeep + 1; k < N; k++) win[k] = (float)r;
    /* win is symmetric (win[k] = win[N - k]), so g is the cosine sum of the full window */
    double *g = (double *)malloc(sizeof(double) * (size_t)N), *cs = (double *)malloc(sizeof(double) * (size_t)N);
    for (int m = 0; m < N; m++) cs[m] = cos(2.0 * 3.141592653589793 * m / N);
    for (int m = 0; m < N; m++) {
        double a = 0.0;
        int idx = 0;
        for (int k = 0; k < N; k++) {
            a += (double)win[k] * cs[idx];
            idx += m;
            if (idx >= N) idx -= N;
        }
        g[m] = a / N;
    }
    for (int j = 0; j < ns; j++)
        for (int i = 0; i < nt; i++)
            M[(size_t)j * nt + i] = i < N ? (float)g[(((long long)i - (long long)j * r) % N + N) % N] : 0.0f;
    free(win);
    free(g);
    free(cs);
}

/* ------------------------------------------------------------ 2-D wavenumber filters */
/* generate_frequency (common.c:333-361): angular frequencies of an n-point FFT, float */
static void angular_frequency(float *f, float d, int n)
{
    const float df = 2.0f * (float)3.141592653589793 / (n * d);
    const int nf = n / 2 + 1;
    f[0] = 0.0f;
    for (int it = 1; it < nf; it++) {
        f[it] = it * df;
        if (n - it >= nf) f[n - it] = -f[it];
    }
}

void fwi_wavenumber_window(int filter, int Nx, int Nz, float dx, float dz, float kpass, float kcut, float *W)
{
    float *kx = (float *)malloc(sizeof(float) * (size_t)Nx), *kz = (float *)malloc(sizeof(float) * (size_t)Nz);
    angular_frequency(kx, dx, Nx);
    angular_frequency(kz, dz, Nz);
    const float pi = (float)3.141592653589793;
    for (int ix = 0; ix < Nx; ix++)
        for (int iz = 0; iz < Nz; iz++) {
            /* the reference evaluates iz <= Nz/2 and lets c2r mirror the rest; |KX|, |KZ| of the
             * mirrored entries are the same floats, so evaluating every entry is identical */
            const float KX = kx[ix] / (2.0f * pi), KZ = kz[iz] / (2.0f * pi);
            const float k = sqrtf(KX * KX + KZ * KZ);
            float w;
            if (filter == 0) {
                const float taperLen = kcut - kpass;
                if (k < kpass) w = 1.0f;
                else if (k >= kpass && k <= kcut) w = 0.5f * (1.0f + cosf(pi * (k - kpass) / taperLen));
                else w = 0.0f;
            } else {
                const float lo = kpass, hi = kcut - kpass;
                if (k < kpass) w = 0.5f * (1.0f + cosf(pi * (kpass - k) / lo));
                else if (k >= kpass && k <= kcut) w = 0.5f * (1.0f + cosf(pi * (k - kpass) / hi));
                else w = 0.0f;
            }
            W[(size_t)ix * Nz + iz] = w;
        }
    free(kx);
    free(kz);
}

