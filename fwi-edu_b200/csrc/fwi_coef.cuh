// fwi_coef.cuh -- the per-model set-up of a padded window on the device: the coefficient fields the
// stencil streams, and per shot the source terms and receiver weights that depend on the model.
//
// What the reference's engine does before its time loop (propagation.c:443-537): edge-replicating pad
// (pad_model2d, common.c:110-176), MEAL damping D and scale Beta (mealCoefs2d, propagation.c:192-354),
// both folded into the model and the time coefficients (:513-529), then K, 1/rho and its derivatives
// (acoustic_iso2d_rgfd_parameter, :103-171, with the two-point edge derivative of
// calculate_gradient2d, common.c:416-479).  Every operation is the reference's own, in its order and
// precision, rounded to nearest (the _rn intrinsics; its powf(x, 2) is x * x), so the fields are the
// strict IEEE build's bit for bit.  The layer weights and the reflection coefficient, the only values
// that take the C library's expf, logf and powf, come from the host (fwi_layer_weights).
//
// The six planes are written in the layout the window's runs read, plain or folded (fwi_fold.cuh); the
// bulk modulus is kept nowhere: the few cells that sources and receivers need are formed again.  With both
// layouts and K a window of 1201 x 4001 held 270 MB, 126 in one layout.
//
// Two launches of one thread per cell (or folded pair); bound by launch latency on small windows and by the
// written planes on large ones.  On the host, one core, the same fields took 5 ms for 221 x 601 and 35
// ms for 601 x 2001, once per window and model: a quarter of a one-shot modelling call on the one, and
// of a 6-shot gradient of 1001 steps on the other.
#pragma once
#include <cuda_runtime.h>

#include "fwi_kernels.cuh"

namespace fwi {

struct CoefDesc {
    const float *vp, *rho;  // the window [nxx][nz] of the model
    const float *weight;    // layer weights 1 .. pml (entry l - 1)
    float logR;             // logarithm of the reflection coefficient
    float dx, dz, dt, fpeak, invdx, invdz;
    int nz, nxx, pml, Nz, Nx, ld;
    int W;                  // columns per half of folded planes, 0: plain ones
    float *planes;          // c1, c2, ck, irx, irz, ir: [Nx][ld] or [W + 6][ld][2] each, zero outside the grid
};

// damping and scale of one axis: d0 * w and 1 + (beta - 1) * w (propagation.c:233-340)
__device__ __forceinline__ void layer_terms(float v, float w, float logR, float thick, float h, float fpeak, float &D,
                                            float &B)
{
    const float d0 = __fdiv_rn(fm(fm(-3.0f, v), logR), fm(2.0f, thick));
    const float ppw = __fdiv_rn(__fdiv_rn(v, __fsqrt_rn(3.0f)), fm(h, fpeak));
    const float beta = __fdiv_rn(fm(2.0f, ppw), 10.0f);
    D = fm(d0, w);
    B = fa(1.0f, fm(fs_(beta, 1.0f), w));
}

struct CoefCell {
    float c1, c2, c3, K, ir;
};
// time coefficients, bulk modulus and 1/rho of the padded cell (ix, iz)
__device__ __forceinline__ CoefCell coef_cell(const CoefDesc &D, int ix, int iz)
{
    CoefCell q;
    const int mx = min(max(ix - D.pml, 0), D.nxx - 1), mz = min(max(iz - D.pml, 0), D.nz - 1);
    float v = D.vp[(long long)mx * D.nz + mz], r = D.rho[(long long)mx * D.nz + mz];
    const int lx = ix < D.pml ? D.pml - ix : ix >= D.Nx - D.pml ? ix - (D.Nx - D.pml - 1) : 0;
    const int lz = iz < D.pml ? D.pml - iz : iz >= D.Nz - D.pml ? iz - (D.Nz - D.pml - 1) : 0;
    const float dtdt = fm(D.dt, D.dt);
    if (lx || lz) {
        float Dx = 0.f, Dz = 0.f, Bx = 1.f, Bz = 1.f;
        if (lx) layer_terms(v, D.weight[lx - 1], D.logR, fm((float)D.pml, D.dx), D.dx, D.fpeak, Dx, Bx);
        if (lz) layer_terms(v, D.weight[lz - 1], D.logR, fm((float)D.pml, D.dz), D.dz, D.fpeak, Dz, Bz);
        float d = __fsqrt_rn(fa(fm(Dx, Dx), fm(Dz, Dz)));
        const float bx = fs_(Bx, 1.0f), bz = fs_(Bz, 1.0f);
        const float B = fa(__fsqrt_rn(fa(fm(bx, bx), fm(bz, bz))), 1.0f);
        d = __fdiv_rn(d, B);
        v = __fdiv_rn(v, B);
        r = fm(r, B);
        // formed in double and rounded to float
        const double dtd = (double)fm(D.dt, d), den = __dadd_rn(1.0, dtd);
        q.c1 = (float)__ddiv_rn(__dsub_rn(2.0, (double)fm(fm(dtdt, d), d)), den);
        q.c2 = (float)__ddiv_rn(-__dsub_rn(1.0, dtd), den);
        q.c3 = (float)__ddiv_rn((double)dtdt, den);
    } else {
        q.c1 = 2.0f;
        q.c2 = -1.0f;
        q.c3 = dtdt;
    }
    q.K = fm(fm(r, v), v);
    q.ir = __fdiv_rn(1.0f, r);
    return q;
}

// calls cell(element, ix, iz) for every element of a plane that holds a cell of the grid, and
// none(element) for the others
template <class Cell, class None>
__device__ __forceinline__ void coef_elements(const CoefDesc &D, Cell cell, None none)
{
    const long long i0 = blockIdx.x * (long long)blockDim.x + threadIdx.x, st = (long long)gridDim.x * blockDim.x;
    const long long n = (long long)(D.W ? D.W + 6 : D.Nx) * D.ld;
    for (long long i = i0; i < n; i += st) {
        const int f = (int)(i / D.ld), iz = (int)(i - (long long)f * D.ld);
        if (!D.W) {
            if (iz < D.Nz) cell(i, f, iz);
            else none(i);
            continue;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int ix = f - 3 + h * D.W;
            if (iz < D.Nz && ix >= 0 && ix < D.Nx) cell(2 * i + h, ix, iz);
            else none(2 * i + h);
        }
    }
}
__device__ __forceinline__ long long coef_plane(const CoefDesc &D)
{
    return D.W ? 2ll * (D.W + 6) * D.ld : (long long)D.Nx * D.ld;
}

// c1, c2, coef3 * K and 1/rho
static __global__ void k_coef_model(const CoefDesc D)
{
    const long long n = coef_plane(D);
    float *p = D.planes;
    coef_elements(
        D,
        [&](long long e, int ix, int iz) {
            const CoefCell q = coef_cell(D, ix, iz);
            p[e] = q.c1;
            p[n + e] = q.c2;
            p[2 * n + e] = fm(q.c3, q.K);
            p[5 * n + e] = q.ir;
        },
        [&](long long e) { p[e] = p[n + e] = p[2 * n + e] = p[5 * n + e] = 0.f; });
}

// the derivatives of 1/rho (two-point at the edges, 12-point optimised inside)
static __global__ void k_coef_derivatives(const CoefDesc D)
{
    const float G1 = 0.91067892f, G2 = -0.34187892f, G3 = 0.13833962f;
    const float G4 = -0.04880710f, G5 = 0.01302148f, G6 = -0.00199047f;
    const long long n = coef_plane(D);
    const float *plane = D.planes + 5 * n;
    float *px = D.planes + 3 * n, *pz = D.planes + 4 * n;
    auto ir = [&](int ix, int iz) {
        const int h = D.W && ix >= D.W;
        return D.W ? plane[((long long)(ix - h * D.W + 3) * D.ld + iz) * 2 + h] : plane[(long long)ix * D.ld + iz];
    };
    coef_elements(
        D,
        [&](long long e, int ix, int iz) {
            float gx, gz;
            auto sum = [&](int sx, int sz) {
                auto d = [&](int k) { return fs_(ir(ix + k * sx, iz + k * sz), ir(ix - k * sx, iz - k * sz)); };
                const float a = fa(fm(G1, d(1)), fm(G2, d(2))), b = fa(fa(a, fm(G3, d(3))), fm(G4, d(4)));
                return fa(fa(b, fm(G5, d(5))), fm(G6, d(6)));
            };
            if (ix >= 6 && ix < D.Nx - 6 && iz >= 6 && iz < D.Nz - 6) {
                gx = fm(sum(1, 0), D.invdx);
                gz = fm(sum(0, 1), D.invdz);
            } else {
                if (ix == 0) gx = __fdiv_rn(fs_(ir(1, iz), ir(0, iz)), D.dx);
                else if (ix == D.Nx - 1) gx = __fdiv_rn(fs_(ir(ix, iz), ir(ix - 1, iz)), D.dx);
                else gx = __fdiv_rn(fs_(ir(ix + 1, iz), ir(ix - 1, iz)), fm(2.0f, D.dx));
                if (iz == 0) gz = __fdiv_rn(fs_(ir(ix, 1), ir(ix, 0)), D.dz);
                else if (iz == D.Nz - 1) gz = __fdiv_rn(fs_(ir(ix, iz), ir(ix, iz - 1)), D.dz);
                else gz = __fdiv_rn(fs_(ir(ix, iz + 1), ir(ix, iz - 1)), fm(2.0f, D.dz));
            }
            px[e] = gx;
            pz[e] = gz;
        },
        [&](long long e) { px[e] = pz[e] = 0.f; });
}

// Per shot (blockIdx.x): the source terms of every step in the reference's precisions (forward
// 1.0*src*K*dt*dt*invdx*invdz in double, propagation.c:558; replay in float, :662), and the receivers'
// K, in the receiver list's order and per column
static __global__ void k_shot_terms(const ShotDesc *__restrict__ shots)
{
    const ShotDesc &S = shots[blockIdx.x];
    const int i0 = blockIdx.y * blockDim.x + threadIdx.x, st = gridDim.y * blockDim.x;
    const CoefDesc D = *S.model;
    __shared__ float source_K;
    if (threadIdx.x == 0) source_K = coef_cell(D, S.isx, S.isz).K;
    __syncthreads();
    const float Ks = source_K;
    double *sd = const_cast<double *>(S.srcd);
    float *sf = const_cast<float *>(S.srcf), *rk = const_cast<float *>(S.recK);
    int4 *rc = const_cast<int4 *>(S.rcol);
    for (int i = i0; i < S.nt; i += st) {
        const double a = __dmul_rn(__dmul_rn((double)S.src[i], (double)Ks), (double)S.dt);
        sd[i] = __dmul_rn(__dmul_rn(__dmul_rn(a, (double)S.dt), (double)S.invdx), (double)S.invdz);
        sf[i] = fm(fm(fm(fm(fm(S.src[i], Ks), S.dt), S.dt), S.invdx), S.invdz);
    }
    for (int x = i0; x < S.Nx; x += st) {
        const int e0 = S.colptr[x], e1 = S.colptr[x + 1];
        for (int e = e0; e < e1; ++e) rk[e] = coef_cell(D, x, S.rec[e].x).K;
        rc[x] = e1 == e0       ? make_int4(-1, 0, 0, 0)
                : e1 == e0 + 1 ? make_int4(S.rec[e0].x, S.rec[e0].y, __float_as_int(rk[e0]), 0)
                               : make_int4(-2, 0, 0, 0);
    }
}

}  // namespace fwi
