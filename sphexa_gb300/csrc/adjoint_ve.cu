// Adjoint (reverse mode) of the volume-element SPH chain over the frozen neighbour lists of the
// last search, in FP64:
//   xmass -> kx/gradh -> EOS -> IAD + divv/curlv (+dV) -> AV switches -> momentum-energy<avClean>
// The arithmetic of one pair or one particle lives in adjoint_ve.cuh; this file holds the passes.
//
// Pass order (reverse of the forward):
//   quotients            1/h, rho = kx m/xm, xm/kx, ln xm
//   forward sums         en_i, avE_i (momentum-energy), G_i, vsig_i (AV), P_i (divv), S_om, S_r0 (gradh)
//   momentum-energy      pair partials -> x, v, h, prho, c, alpha, rho, xm, C, dV
//   AV switch            per particle (alpha -> G, vsig seeds), then pair partials
//   IAD + divv           per particle (C, divv, dV -> tau, P seeds), then pair partials
//   EOS                  per particle -> kx, xm, gradh, u
//   kx / gradh           per particle (-> sum seeds), then pair partials
//   xmass                per particle, then pair partials
// Every pair pass runs in one of two forms: scatter (each pair evaluated once by its list owner,
// the neighbour's partials added with FP64 atomics) or two-sided (each particle evaluates its own
// list for its partials and walks its incoming list, a CSR built once per list set, for the
// neighbour-side partials; each thread writes only its particle: bit-reproducible).
#include "adjoint_ve.cuh"
#include "pairs.cuh"

namespace sphgb {

namespace {

using namespace vead;

constexpr int kVeAdjBlock = 128;

struct VeAdjArgs {
    // forward state
    const double *x, *y, *z, *vx, *vy, *vz, *h, *m, *u, *alpha0, *alpha, *xm, *kx, *gradh, *prho, *c, *divv;
    const double* C[6];
    const double* dV[6];
    const double2 *wh, *whd;  // W and dW/dv in the context's form (the kernels' Smooth argument tells which)
    double K, gamma;
    AvPrm av;
    DevBox box;
    int avClean;
    ListView lv;
    const uint32_t* tOff;
    const uint32_t* tIdx;
    int64_t n;
    // seeds
    const double *sRho, *sAx, *sAy, *sAz, *sDu;
    // outputs
    double *bx, *by, *bz, *bvx, *bvy, *bvz, *bh, *bu;
    // per-particle quotients
    double *hInv, *rho, *rhoInv, *vol, *kxInv, *xmInv, *lnxm;
    // 1/(h dx), K h^-3, K h^-4 and vol / kx
    double *hDx, *hk3, *hk4, *kxv;
    const double4* expTab;
    CoordFp64 cf;
    // forward sums
    double *en, *avE, *G, *vsig, *P, *wom, *wr0;
    uint32_t* vsigArg;
    // FP32 copies {x y z c} and {vx vy vz 0} for the signal-velocity filter, and the bound on the
    // FP32 error of a position difference per component
    float4 *xc32, *v32;
    float ePos;
    // adjoints of the intermediate fields
    double *prhoB, *cB, *alphaB, *rhoB, *xmB, *kxB, *CB, *gB, *divvB, *gradhB;
    double* Rav;  // 3 x n: R_i = sum_j fac_j W_j r_j of the AV pair terms (i's C partials, avCbar)
    // seeds of the pair terms
    double *GB, *CGB, *vsigB, *tauB, *PB, *Skx, *Som, *Sr0, *R0b;
};

constexpr uint32_t kNoPair = 0xffffffffu;

// interpolant value and slope (dw/dv) on the interval holding v (as the forward passes select it)
template<bool Smooth>
__device__ __forceinline__ double lookupVS(const KTab<Smooth>& tab, double v, double& slope)
{
    return lookupVSlope(tab, v, slope);
}

// r = x_i - x_j with the legacy periodic fold at 2 h_i (box.hpp:216-238), d = |r|
__device__ __forceinline__ void geom(const VeAdjArgs& a, int64_t i, int64_t j, double r[3], double& d, double& rinv)
{
    const long long twoHBits = __double_as_longlong(2.0 * a.h[i]);
    const double dd[3] = {a.x[i] - a.x[j], a.y[i] - a.y[j], a.z[i] - a.z[j]};
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = a.box.pbc[k] ? CoordFp64::wrapLegacy(dd[k], twoHBits, a.box.L[k]) : dd[k];
    const double r2 = r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
    rinv = rsqrt(r2);
    d = r2 * rinv;
}

__device__ __forceinline__ void vdiff(const VeAdjArgs& a, int64_t i, int64_t j, double v[3])
{
    v[0] = a.vx[i] - a.vx[j];
    v[1] = a.vy[i] - a.vy[j];
    v[2] = a.vz[i] - a.vz[j];
}

__device__ __forceinline__ MeSide meSide(const VeAdjArgs& a, int64_t i)
{
    MeSide s;
    s.hInv = a.hInv[i];
    s.c = a.c[i];
    s.alpha = a.alpha[i];
    s.m = a.m[i];
    s.rho = a.rho[i];
    s.rhoInv = a.rhoInv[i];
    s.xm = a.xm[i];
    s.xmInv = a.xmInv[i];
    s.lnxm = a.lnxm[i];
    s.prho = a.prho[i];
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        s.C[q] = a.C[q][i];
        s.g[q] = a.avClean ? a.dV[q][i] : 0.0;
    }
    return s;
}

__device__ __forceinline__ void loadC(const VeAdjArgs& a, int64_t i, double C[6])
{
#pragma unroll
    for (int q = 0; q < 6; ++q) C[q] = a.C[q][i];
}

__device__ __forceinline__ double etaCritOf(unsigned cnt) { return cbrt(32.0 * M_PI / 3.0 / double(cnt + 1)); }

// add v to p[i]: atomically where other threads add to the same particle (scatter form)
__device__ __forceinline__ void put(double* p, int64_t i, double v, bool atomic)
{
    if (atomic) atomicAdd(p + i, v);
    else p[i] += v;
}

__global__ void veQuotKernel(VeAdjArgs a)
{
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= a.n) return;
    const double xm = a.xm[i], kx = a.kx[i];
    const double rho = kx * a.m[i] / xm;
    const double hInv = 1.0 / a.h[i], hk3 = a.K * (hInv * hInv * hInv), vol = xm / kx, kxInv = 1.0 / kx;
    a.hInv[i] = hInv;
    a.hDx[i] = hInv * kTabInvDx;
    a.hk3[i] = hk3;
    a.hk4[i] = hk3 * hInv;
    a.rho[i] = rho;
    a.rhoInv[i] = 1.0 / rho;
    a.vol[i] = vol;
    a.kxInv[i] = kxInv;
    a.kxv[i] = vol * kxInv;
    a.xmInv[i] = 1.0 / xm;
    a.lnxm[i] = log(xm);
    a.xc32[i] = make_float4(float(a.x[i]), float(a.y[i]), float(a.z[i]), float(a.c[i]));
    a.v32[i] = make_float4(float(a.vx[i]), float(a.vy[i]), float(a.vz[i]), 0.f);
}

// forward sums of the momentum-energy pass: en_i, avE_i (before max(0, .))
template<bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) vePreMeKernel(VeAdjArgs a)
{
    const KTab<Smooth> tw{a.wh};
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= a.n) return;
    const MeSide I = meSide(a, i);
    const unsigned nc = a.lv.capped(i);
    const double etaCrit = etaCritOf(nc);
    double en = 0.0, avE = 0.0;
    for (unsigned q = 0; q < nc; ++q) {
        const int64_t j = a.lv.at(i, q);
        double r[3], d, rinv, v[3];
        geom(a, i, j, r, d, rinv);
        vdiff(a, i, j, v);
        const MeSide J = meSide(a, j);
        double s;
        const double wi = lookupVS(tw, d * I.hInv, s), wj = lookupVS(tw, d * J.hInv, s);
        MeFwd f;
        meFwd(r, d, rinv, v, I, J, wi, wj, a.avClean != 0, etaCrit, f);
        meSums(v, J, f, en, avE);
    }
    a.en[i] = en;
    a.avE[i] = avE;
}

// the signal velocity of the AV switch (av_switches_kern.hpp:66-86): the first of i's approaching
// pairs, in list order, with the largest c_i + c_j - 3 (r.v)/|r| sets vsig_i (1e-40 c_i when none)
__device__ __forceinline__ void vsigStep(const VeAdjArgs& a, int64_t j, const double r[3], double rinv,
                                         const double v[3], double ci, double& vsig, uint32_t& arg)
{
    const double rv = r[0] * v[0] + r[1] * v[1] + r[2] * v[2];
    if (rv < 0.0) {
        const double vs = ci + a.c[j] - 3.0 * rv * rinv;
        if (vs > vsig) {
            vsig = vs;
            arg = uint32_t(j);
        }
    }
}

// vsig_i and its pair alone, when the forward passes kept the other sums of vePreKernel.  An FP32
// walk over i's list finds a lower bound L on vsig_i from the pairs that surely approach; a second one
// picks the pairs whose FP32 signal velocity plus the error bound reaches L, which every pair able to
// set vsig_i does, and only those (one or two) are evaluated in FP64 (vsigStep, in list order), so vsig_i
// and its pair come out as in vePreKernel.  In one walk each new maximum ran the FP64 step, for some lane
// of the warp in nearly every step (1M particles: 3.5 -> 0.78 ms).  Particles whose 2h exceeds a quarter of a periodic box edge (where
// the threshold-2h image rule of the FP64 geometry need not be the minimum image) walk in FP64.
__global__ void __launch_bounds__(kVeAdjBlock) veArgKernel(VeAdjArgs a)
{
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= a.n) return;
    const double ci = a.c[i];
    double vsig = 1e-40 * ci;
    uint32_t arg = kNoPair;
    const unsigned nc = a.lv.capped(i);
    auto exact = [&](uint32_t j) {
        double r[3], d, rinv, v[3];
        geom(a, i, j, r, d, rinv);
        vdiff(a, i, j, v);
        vsigStep(a, j, r, rinv, v, ci, vsig, arg);
    };
    const double twoH = 2.0 * a.h[i];
    bool fp64Walk = false;
#pragma unroll
    for (int k = 0; k < 3; ++k) fp64Walk |= a.box.pbc[k] && twoH > 0.25 * a.box.L[k];
    if (fp64Walk) {
        for (unsigned q = 0; q < nc; ++q) exact(a.lv.at(i, q));
    } else {
        const float4 Xi = a.xc32[i], Vi = a.v32[i];
        const float viMax = fmaxf(fabsf(Vi.x), fmaxf(fabsf(Vi.y), fabsf(Vi.z)));
        const float dr = 2.f * a.ePos;  // >= |r_f - r| (three components)
        // FP32 signal velocity of pair j with its error bound; rv: r.v with its own
        auto filter = [&](uint32_t j, float& rv, float& erv, float& vs, float& ev) {
            const float4 Xj = a.xc32[j], Vj = a.v32[j];
            float r[3] = {Xi.x - Xj.x, Xi.y - Xj.y, Xi.z - Xj.z};
#pragma unroll
            for (int k = 0; k < 3; ++k)
                if (a.box.pbc[k]) {  // minimum image: |r| <= 2h < L/4 for every listed pair
                    if (r[k] > 0.5f * a.box.Lf[k]) r[k] -= a.box.Lf[k];
                    else if (r[k] < -0.5f * a.box.Lf[k]) r[k] += a.box.Lf[k];
                }
            const float v[3] = {Vi.x - Vj.x, Vi.y - Vj.y, Vi.z - Vj.z};
            const float d2 = fmaf(r[0], r[0], fmaf(r[1], r[1], r[2] * r[2])), di = rsqrtf(d2), d = d2 * di;
            rv = fmaf(r[0], v[0], fmaf(r[1], v[1], r[2] * v[2]));
            // bounds: |v_f - v| <= dv, |r.v error| <= erv, |signal velocity error| <= ev
            const float vn = 1.8f * (viMax + fmaxf(fabsf(Vj.x), fmaxf(fabsf(Vj.y), fabsf(Vj.z))));
            const float dv = 1e-6f * vn;
            erv = dr * vn + d * (dv + 1e-6f * vn);
            const float rd = 3.f * rv * di;  // within 4 ulp of 3 rv / d, inside the 1e-6 below
            vs = Xi.w + Xj.w - rd;
            ev = 3.f * (4.f * dr * vn * di + 2.f * dv + 1e-6f * vn) + 1e-6f * (Xi.w + Xj.w + fabsf(rd));
        };
        float L = 0.f, rv, erv, vs, ev;  // vsig_i > 0
        for (unsigned q = 0; q < nc; ++q) {
            filter(a.lv.at(i, q), rv, erv, vs, ev);
            if (rv < -erv) L = fmaxf(L, vs - ev);  // surely approaches
        }
        uint32_t c0 = 0, c1 = 0;
        int held = 0;
        for (unsigned q = 0; q < nc; ++q) {
            const uint32_t j = a.lv.at(i, q);
            filter(j, rv, erv, vs, ev);
            if (!(rv >= erv) && !(vs + ev < L)) {  // may approach and may reach L (NaN: evaluate)
                if (held == 2) {
                    exact(c0);
                    exact(c1);
                    held = 0;
                }
                if (held == 0) c0 = j;
                else c1 = j;
                ++held;
            }
        }
        if (held > 0) exact(c0);
        if (held > 1) exact(c1);
    }
    a.vsig[i] = vsig;
    a.vsigArg[i] = arg;
}

// forward sums of the AV switch (G_i, vsig_i and the pair that set it), of divv (P_i) and of
// gradh (whomega0 = K h^-4 S_om, wrho0 = K h^-4 S_r0)
template<bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) vePreKernel(VeAdjArgs a)
{
    const KTab<Smooth> tw{a.wh};
    const KTab<Smooth> tdw{a.whd};
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= a.n) return;
    double Ci[6];
    loadC(a, i, Ci);
    const double hInv = a.hInv[i], ci = a.c[i], divvi = a.divv[i];
    const double Wk0 = a.K * hInv * hInv * hInv;
    double S[3] = {0.0, 0.0, 0.0}, P[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    double vsig = 1e-40 * ci, so = -3.0 * a.xm[i], sr = -3.0 * a.m[i];
    uint32_t arg = kNoPair;
    const unsigned nc = a.lv.capped(i);
    for (unsigned q = 0; q < nc; ++q) {
        const uint32_t j = a.lv.at(i, q);
        double r[3], d, rinv, v[3];
        geom(a, i, j, r, d, rinv);
        vdiff(a, i, j, v);
        const double v1 = d * hInv;
        double dw, dwd;
        const double w = lookupVS(tw, v1, dw);
        const double wd = lookupVS(tdw, v1, dwd);
        vsigStep(a, j, r, rinv, v, ci, vsig, arg);
        const double fac = a.vol[j] * (divvi - a.divv[j]) * w;
        const double xw = a.xm[j] * w;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            S[k] += fac * r[k];
#pragma unroll
            for (int t = 0; t < 3; ++t) P[3 * k + t] -= xw * v[k] * r[t];
        }
        const double dterh = -(3.0 * w + v1 * wd);
        so += a.xm[j] * dterh;
        sr += a.m[j] * dterh;
    }
    // G = -K h^-3 C_i S, S = sum_j vol_j (divv_i - divv_j) w r
    double G[3];
    symv(Ci, S, G);
#pragma unroll
    for (int k = 0; k < 3; ++k) a.G[k * a.n + i] = -Wk0 * G[k];
#pragma unroll
    for (int k = 0; k < 9; ++k) a.P[k * a.n + i] = P[k];
    a.vsig[i] = vsig;
    a.vsigArg[i] = arg;
    const double h4 = a.K * hInv * hInv * hInv * hInv;
    a.wom[i] = h4 * so;
    a.wr0[i] = h4 * sr;
}

// ---------------------------------------------------------------- momentum-energy
struct MeSeed {
    double mb[3], enb, avEb;
    bool any;
};

template<bool WithDu>
__device__ __forceinline__ MeSeed meSeed(const VeAdjArgs& a, int64_t i)
{
    MeSeed s;
    s.mb[0] = a.sAx ? -a.K * a.sAx[i] : 0.0;
    s.mb[1] = a.sAy ? -a.K * a.sAy[i] : 0.0;
    s.mb[2] = a.sAz ? -a.K * a.sAz[i] : 0.0;
    s.any = s.mb[0] != 0.0 || s.mb[1] != 0.0 || s.mb[2] != 0.0;
    s.enb = s.avEb = 0.0;
    if (WithDu) {
        const double du = a.sDu[i];
        s.enb = a.K * a.prho[i] * du;
        s.avEb = a.avE[i] >= 0.0 ? 0.5 * a.K * du : 0.0;
        s.any = s.any || du != 0.0;
    }
    return s;
}

struct MeAcc {
    double x[3], v[3], h, prho, c, alpha, rho, xm, C[6], g[6];
};

__device__ __forceinline__ void meAddI(MeAcc& s, const MeGrad& o)
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s.x[k] += o.r[k];
        s.v[k] += o.v[k];
    }
    s.h += o.hI;
    s.prho += o.prhoI;
    s.c += o.c;
    s.alpha += o.alpha;
    s.rho += o.rhoI;
    s.xm += o.xmI;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        s.C[q] += o.CI[q];
        s.g[q] += o.gI[q];
    }
}

__device__ __forceinline__ void meAddJ(MeAcc& s, const MeGrad& o)
{
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        s.x[k] -= o.r[k];
        s.v[k] -= o.v[k];
    }
    s.h += o.hJ;
    s.prho += o.prhoJ;
    s.c += o.c;
    s.alpha += o.alpha;
    s.rho += o.rhoJ;
    s.xm += o.xmJ;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        s.C[q] += o.CJ[q];
        s.g[q] += o.gJ[q];
    }
}

template<bool AvClean>
__device__ __forceinline__ void meFlush(const VeAdjArgs& a, int64_t k, const MeAcc& s, bool atomic)
{
    put(a.bx, k, s.x[0], atomic);
    put(a.by, k, s.x[1], atomic);
    put(a.bz, k, s.x[2], atomic);
    put(a.bvx, k, s.v[0], atomic);
    put(a.bvy, k, s.v[1], atomic);
    put(a.bvz, k, s.v[2], atomic);
    put(a.bh, k, s.h, atomic);
    put(a.prhoB, k, s.prho, atomic);
    put(a.cB, k, s.c, atomic);
    put(a.alphaB, k, s.alpha, atomic);
    put(a.rhoB, k, s.rho, atomic);
    put(a.xmB, k, s.xm, atomic);
#pragma unroll
    for (int q = 0; q < 6; ++q) put(a.CB + q * a.n, k, s.C[q], atomic);
    if (AvClean)
#pragma unroll
        for (int q = 0; q < 6; ++q) put(a.gB + q * a.n, k, s.g[q], atomic);
}

template<bool AvClean, bool WithDu, bool Smooth>
__device__ __forceinline__ void mePair(const VeAdjArgs& a, int64_t i, int64_t j, const MeSide& I, const MeSide& J,
                                       double etaCrit, const MeSeed& sd, MeGrad& o)
{
    const KTab<Smooth> tw{a.wh};
    double r[3], d, rinv, v[3];
    geom(a, i, j, r, d, rinv);
    vdiff(a, i, j, v);
    double dwi, dwj;
    const double wi = lookupVS(tw, d * I.hInv, dwi), wj = lookupVS(tw, d * J.hInv, dwj);
    meAdj<AvClean, WithDu>(r, d, rinv, v, I, J, wi, dwi, wj, dwj, etaCrit, sd.mb, sd.enb, sd.avEb, o);
}

// WithDu: a du seed is given (the energy sums en, avE of the forward are then needed)
template<bool TwoSided, bool AvClean, bool WithDu, bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) meVeAdjKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    MeAcc s{};
    const MeSide S = meSide(a, k);
    const MeSeed sd = meSeed<WithDu>(a, k);
    // own terms outside the pairs: du = K (prho en + avE / 2) and the rho seed
    s.prho = WithDu ? a.K * a.en[k] * a.sDu[k] : 0.0;
    s.rho = a.sRho ? a.sRho[k] : 0.0;
    if (sd.any) {
        const unsigned nc = a.lv.capped(k);
        const double etaCrit = etaCritOf(nc);
        for (unsigned q = 0; q < nc; ++q) {
            const int64_t j = a.lv.at(k, q);
            const MeSide J = meSide(a, j);
            MeGrad o;
            mePair<AvClean, WithDu, Smooth>(a, k, j, S, J, etaCrit, sd, o);
            meAddI(s, o);
            if (!TwoSided) {
                atomicAdd(a.bx + j, -o.r[0]);
                atomicAdd(a.by + j, -o.r[1]);
                atomicAdd(a.bz + j, -o.r[2]);
                atomicAdd(a.bvx + j, -o.v[0]);
                atomicAdd(a.bvy + j, -o.v[1]);
                atomicAdd(a.bvz + j, -o.v[2]);
                atomicAdd(a.bh + j, o.hJ);
                atomicAdd(a.prhoB + j, o.prhoJ);
                atomicAdd(a.cB + j, o.c);
                atomicAdd(a.alphaB + j, o.alpha);
                atomicAdd(a.rhoB + j, o.rhoJ);
                atomicAdd(a.xmB + j, o.xmJ);
#pragma unroll
                for (int t = 0; t < 6; ++t) atomicAdd(a.CB + t * a.n + j, o.CJ[t]);
                if (AvClean)
#pragma unroll
                    for (int t = 0; t < 6; ++t) atomicAdd(a.gB + t * a.n + j, o.gJ[t]);
            }
        }
    }
    if (TwoSided) {
        for (uint32_t e = a.tOff[k]; e < a.tOff[k + 1]; ++e) {
            const int64_t i = a.tIdx[e];
            const MeSeed si = meSeed<WithDu>(a, i);
            if (!si.any) continue;
            const MeSide I = meSide(a, i);
            MeGrad o;
            mePair<AvClean, WithDu, Smooth>(a, i, k, I, S, etaCritOf(a.lv.capped(i)), si, o);
            meAddJ(s, o);
        }
    }
    meFlush<AvClean>(a, k, s, !TwoSided);
}

// the geometry of an owned pair, in the forward passes' arithmetic
struct OwnGeom {
    CoordFp64::Target t;
    CoordFp64::Fold fold;
    double vx, vy, vz;
    __device__ __forceinline__ OwnGeom(const VeAdjArgs& a, int64_t k)
        : t(a.cf.target(k)), fold(a.cf.fold(t, 2.0 * a.h[k])), vx(a.vx[k]), vy(a.vy[k]), vz(a.vz[k])
    {
    }
    __device__ __forceinline__ void r(const VeAdjArgs& a, int64_t j, bool mutual, double o[3], double& d, double& rinv) const
    {
        a.cf.diffOwned(t, j, mutual, fold, o[0], o[1], o[2]);
        const double r2 = dist2(o[0], o[1], o[2]);
        rinv = invDist(r2);
        d = r2 * rinv;
    }
    __device__ __forceinline__ void v(const VeAdjArgs& a, int64_t j, double o[3]) const
    {
        o[0] = vx - __ldg(a.vx + j);
        o[1] = vy - __ldg(a.vy + j);
        o[2] = vz - __ldg(a.vz + j);
    }
};

// one evaluation per owned entry of the owned lists built with the neighbour lists: a mutual pair
// gives both particles' terms (meAdjMutual), a one-sided entry its owner's (the same function with
// the neighbour's seeds zero); the neighbour's partials are added with FP64 atomics.  No avClean.
// With a du seed.
template<bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) meVeAdjOnceKernel(VeAdjArgs a, OwnedView ov)
{
    constexpr bool WithDu = true;
    const KTab<Smooth> tw{a.wh};
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    MeAcc s{};
    const MeSide S = meSide(a, k);
    const MeSeed sd = meSeed<WithDu>(a, k);
    s.prho = WithDu ? a.K * a.en[k] * a.sDu[k] : 0.0;
    s.rho = a.sRho ? a.sRho[k] : 0.0;
    const OwnGeom og(a, k);
    const unsigned cnt = ov.size(k);
    for (unsigned q = 0; q < cnt; ++q) {
        bool mutual;
        const uint32_t j = ov.at(k, q, mutual);
        MeSeed sj{};
        if (mutual) sj = meSeed<WithDu>(a, j);
        if (!sd.any && !sj.any) continue;
        const MeSide J = meSide(a, j);
        double r[3], d, rinv, v[3];
        og.r(a, j, mutual, r, d, rinv);
        og.v(a, j, v);
        double dwi, dwj;
        const double wi = lookupVS(tw, d * S.hInv, dwi), wj = lookupVS(tw, d * J.hInv, dwj);
        MeGrad o;
        meAdjMutual<WithDu>(r, d, rinv, v, S, J, wi, dwi, wj, dwj, sd.mb, sd.enb, sd.avEb, sj.mb, sj.enb, sj.avEb, o);
        meAddI(s, o);
        atomicAdd(a.bx + j, -o.r[0]);
        atomicAdd(a.by + j, -o.r[1]);
        atomicAdd(a.bz + j, -o.r[2]);
        atomicAdd(a.bvx + j, -o.v[0]);
        atomicAdd(a.bvy + j, -o.v[1]);
        atomicAdd(a.bvz + j, -o.v[2]);
        atomicAdd(a.bh + j, o.hJ);
        atomicAdd(a.prhoB + j, o.prhoJ);
        atomicAdd(a.cB + j, o.c);
        atomicAdd(a.alphaB + j, o.alpha);
        atomicAdd(a.rhoB + j, o.rhoJ);
        atomicAdd(a.xmB + j, o.xmJ);
#pragma unroll
        for (int t = 0; t < 6; ++t) atomicAdd(a.CB + t * a.n + j, o.CJ[t]);
    }
    meFlush<false>(a, k, s, true);
}

// The same without a du seed (meAdjMutual<false>), arranged for few FP64 instructions: the kernel is
// bound by the FP64 pipe.  With s = m_j abar_i - m_i abar_j both ends' Abar are multiples of s, so with
// e = C s per end every projection follows from z = r . e, the position partial from e, and both C
// partials from one symmetric s r^T; K h^-3 and K h^-4 come per particle, table slopes stay in table
// units, the ramp's exp and quotient as in the forward pass.  About 218 FP64 instructions per warp step
// against 379 (1M particles: 40.2 -> 20.9 ms).
template<bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) meVeAdjOnceAKernel(VeAdjArgs a, OwnedView ov)
{
    const KTab<Smooth> tw{a.wh};
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    MeAcc s{};
    double xmOwn = 0.0;  // to be divided by xm_k
    const double ax = a.sAx ? a.sAx[k] : 0.0, ay = a.sAy ? a.sAy[k] : 0.0, az = a.sAz ? a.sAz[k] : 0.0;
    const bool any = ax != 0.0 || ay != 0.0 || az != 0.0;
    double CI[6];
    loadC(a, k, CI);
    const double hDxI = a.hDx[k], hk3I = a.hk3[k], hk4I = a.hk4[k], cI = a.c[k], alI = a.alpha[k], mI = a.m[k],
                 rhoI = a.rho[k], rhoInvI = a.rhoInv[k], xmI = a.xm[k], lnxmI = a.lnxm[k], prhoI = a.prho[k];
    const OwnGeom og(a, k);
    if (blockIdx.y == 0) s.rho = a.sRho ? a.sRho[k] : 0.0;
    const unsigned cnt = ov.size(k);
    for (unsigned q = blockIdx.y; q < cnt; q += gridDim.y) {
        bool mutual;
        const uint32_t j = ov.at(k, q, mutual);
        double bx = 0.0, by = 0.0, bz = 0.0;
        if (mutual) {
            bx = a.sAx ? __ldg(a.sAx + j) : 0.0;
            by = a.sAy ? __ldg(a.sAy + j) : 0.0;
            bz = a.sAz ? __ldg(a.sAz + j) : 0.0;
        }
        if (!any && bx == 0.0 && by == 0.0 && bz == 0.0) continue;
        const double mJ = __ldg(a.m + j);
        const double sv[3] = {fma(mJ, ax, -mI * bx), fma(mJ, ay, -mI * by), fma(mJ, az, -mI * bz)};
        double r[3], d, rinv, v[3];
        og.r(a, j, mutual, r, d, rinv);
        og.v(a, j, v);
        const double xi = d * hDxI, xj = d * __ldg(a.hDx + j);
        double tyi, tyj;
        const double wi = lookupXSlope(tw, xi, tyi), wj = lookupXSlope(tw, xj, tyj);
        double CJ[6], ei[3], ej[3];
#pragma unroll
        for (int t = 0; t < 6; ++t) CJ[t] = __ldg(a.C[t] + j);
        symv(CI, sv, ei);
        symv(CJ, sv, ej);
        const double zi = r[0] * ei[0] + r[1] * ei[1] + r[2] * ei[2], zj = r[0] * ej[0] + r[1] * ej[1] + r[2] * ej[2];
        const double Wi = hk3I * wi, Wj = __ldg(a.hk3 + j) * wj;
        const double Zi = Wi * zi, Zj = Wj * zj;  // s . A_i and s . A_j of the seeds -K abar
        const double rhoJ = __ldg(a.rho + j), rhoInvJ = __ldg(a.rhoInv + j), lnxmJ = __ldg(a.lnxm + j),
                     prhoJ = __ldg(a.prho + j);
        const AtwoodRamp w8 = atwoodRamp(a.expTab, rhoI, rhoJ, lnxmI, lnxmJ, xmI, __ldg(a.xm + j));
        const double wij = fma(r[2], v[2], fma(r[1], v[1], r[0] * v[0])) * rinv;
        const double vb2 = fma(Zi, rhoInvI, Zj * rhoInvJ);  // twice the viscosity's adjoint
        double hvi = 0.0, hvj = 0.0, rvb = 0.0, cb = 0.0, ab = 0.0;
        if (negative(wij)) {
            const double a8 = 0.125 * (alI + __ldg(a.alpha + j)), csum = cI + __ldg(a.c + j), ac = a8 * csum;
            const double hv = (ac - wij) * -wij, t1 = -vb2 * wij;
            hvi = hv * rhoInvI;
            hvj = hv * rhoInvJ;
            rvb = vb2 * fma(2.0, wij, -ac) * rinv;
            cb = t1 * a8;
            ab = t1 * (0.125 * csum);
        }
        const double pi = fma(w8.am, prhoI, hvi), pj = fma(w8.bm, prhoJ, hvj);
        const double gpi = w8.am * Zi, gpj = w8.bm * Zj;
        const double pa = prhoI * gpi, pb = prhoJ * gpj, D = pb - pa, sD = w8.s * D;
        double rI = -hvi * Zi * rhoInvI, rJ = -hvj * Zj * rhoInvJ;
        if (w8.ramp) {
            const double T = -10.0 * D * (lnxmJ - lnxmI) * w8.srInv;
            const double sgn = rhoI > rhoJ ? 1.0 : (rhoI < rhoJ ? -1.0 : 0.0);
            rI = fma(T, sgn - w8.At, rI);
            rJ = fma(T, -sgn - w8.At, rJ);
        }
        const double qi = Wi * pi, qj = Wj * pj;
        const double bi4 = pi * zi * hk4I, bj4 = pj * zj * __ldg(a.hk4 + j);
        const double hJ = -bj4 * fma(xj, tyj, 3.0 * wj);
        s.h = fma(-bi4, fma(xi, tyi, 3.0 * wi), s.h);
        const double db = fma(-rvb, wij, kTabInvDx * fma(bi4, tyi, bj4 * tyj)), dr = db * rinv;
        double g[3], vb[3];
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            g[t] = fma(dr, r[t], fma(rvb, v[t], fma(qi, ei[t], qj * ej[t])));
            vb[t] = rvb * r[t];
            s.x[t] += g[t];
            s.v[t] += vb[t];
        }
        s.prho += gpi;
        s.c += cb;
        s.alpha += ab;
        s.rho += rI;
        xmOwn += fma(2.0, pa, sD);
        const double S[6] = {sv[0] * r[0], fma(sv[0], r[1], sv[1] * r[0]), fma(sv[0], r[2], sv[2] * r[0]),
                             sv[1] * r[1], fma(sv[1], r[2], sv[2] * r[1]), sv[2] * r[2]};
#pragma unroll
        for (int t = 0; t < 6; ++t) {
            s.C[t] = fma(qi, S[t], s.C[t]);
            atomicAdd(a.CB + t * a.n + j, qj * S[t]);
        }
        atomicAdd(a.bx + j, -g[0]);
        atomicAdd(a.by + j, -g[1]);
        atomicAdd(a.bz + j, -g[2]);
        if (negative(wij)) {
            atomicAdd(a.bvx + j, -vb[0]);
            atomicAdd(a.bvy + j, -vb[1]);
            atomicAdd(a.bvz + j, -vb[2]);
            atomicAdd(a.cB + j, cb);
            atomicAdd(a.alphaB + j, ab);
        }
        atomicAdd(a.bh + j, hJ);
        atomicAdd(a.prhoB + j, gpj);
        atomicAdd(a.rhoB + j, rJ);
        atomicAdd(a.xmB + j, fma(2.0, pb, -sD) * __ldg(a.xmInv + j));
    }
    s.xm = xmOwn * a.xmInv[k];
    meFlush<false>(a, k, s, true);
}

// *any = 1 when a seed value is not zero (NaN counts)
__global__ void anySeedKernel(const double* __restrict__ x, int64_t n, int* __restrict__ any)
{
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (__any_sync(0xffffffffu, i < n && x[i] != 0.0) && (threadIdx.x & 31) == 0) *any = 1;
}

// ---------------------------------------------------------------- AV switch
__global__ void veAvSeedKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    const double G[3] = {a.G[k], a.G[a.n + k], a.G[2 * a.n + k]};
    double Gb[3], vsigb, hb, divvb, cb;
    avSeed(a.av, a.alphaB[k], a.alpha0[k], a.h[k], a.c[k], a.divv[k], G, a.vsig[k], Gb, vsigb, hb, divvb, cb);
    if (a.vsigArg[k] == kNoPair) cb += 1e-40 * vsigb;  // vsig = 1e-40 c_i when no pair approaches
    double C[6], CGb[3];
    loadC(a, k, C);
    symv(C, Gb, CGb);
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        a.GB[t * a.n + k] = Gb[t];
        a.CGB[t * a.n + k] = CGb[t];
    }
    a.vsigB[k] = vsigb;
    a.bh[k] += hb;
    a.divvB[k] += divvb;
    a.cB[k] += cb;
}

struct AvSeedV {
    double Gb[3], CGb[3], vsigb;
    uint32_t arg;
    bool any, gAny;  // gAny: a G seed; without one only the pair that set vsig has partials
};

__device__ __forceinline__ AvSeedV avSeedOf(const VeAdjArgs& a, int64_t i)
{
    AvSeedV s;
    s.Gb[0] = a.GB[i];
    s.Gb[1] = a.GB[a.n + i];
    s.Gb[2] = a.GB[2 * a.n + i];
#pragma unroll
    for (int t = 0; t < 3; ++t) s.CGb[t] = a.CGB[t * a.n + i];
    s.vsigb = a.vsigB[i];
    s.arg = a.vsigArg[i];
    s.gAny = s.Gb[0] != 0.0 || s.Gb[1] != 0.0 || s.Gb[2] != 0.0;
    s.any = s.gAny || s.vsigb != 0.0;
    return s;
}

template<bool Smooth>
__device__ __forceinline__ void avPair(const VeAdjArgs& a, int64_t i, int64_t j, const AvSeedV& sd, AvGrad& o)
{
    const KTab<Smooth> tw{a.wh};
    double r[3], d, rinv, v[3];
    geom(a, i, j, r, d, rinv);
    vdiff(a, i, j, v);
    const double hInv = a.hInv[i];
    double dw;
    const double w = lookupVS(tw, d * hInv, dw);
    avAdj(r, d, rinv, v, hInv, w, dw, a.K, a.vol[j], a.kxInv[j], a.divv[i], a.divv[j], sd.CGb, sd.vsigb,
          uint32_t(j) == sd.arg, o);
}

template<bool TwoSided, bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) veAvAdjKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double x[3] = {0, 0, 0}, v[3] = {0, 0, 0}, c = 0, h = 0, divv = 0, xm = 0, kx = 0;
    const AvSeedV sd = avSeedOf(a, k);
    if (sd.any) {
        double R[3] = {0.0, 0.0, 0.0};
        const unsigned nc = a.lv.capped(k);
        for (unsigned q = 0; q < nc; ++q) {
            const int64_t j = a.lv.at(k, q);
            if (!sd.gAny && uint32_t(j) != sd.arg) continue;
            AvGrad o;
            avPair<Smooth>(a, k, j, sd, o);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                x[t] += o.r[t];
                v[t] += o.v[t];
                R[t] += o.R[t];
            }
            c += o.cI;
            h += o.hI;
            divv += o.divvI;
            if (!TwoSided) {
                atomicAdd(a.bx + j, -o.r[0]);
                atomicAdd(a.by + j, -o.r[1]);
                atomicAdd(a.bz + j, -o.r[2]);
                if (uint32_t(j) == sd.arg) {
                    atomicAdd(a.bvx + j, -o.v[0]);
                    atomicAdd(a.bvy + j, -o.v[1]);
                    atomicAdd(a.bvz + j, -o.v[2]);
                    atomicAdd(a.cB + j, o.cJ);
                }
                atomicAdd(a.divvB + j, o.divvJ);
                atomicAdd(a.xmB + j, o.xmJ);
                atomicAdd(a.kxB + j, o.kxJ);
            }
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) put(a.Rav + t * a.n, k, R[t], !TwoSided);
    }
    if (TwoSided) {
        for (uint32_t e = a.tOff[k]; e < a.tOff[k + 1]; ++e) {
            const int64_t i = a.tIdx[e];
            const AvSeedV si = avSeedOf(a, i);
            if (!si.any || (!si.gAny && uint32_t(k) != si.arg)) continue;
            AvGrad o;
            avPair<Smooth>(a, i, k, si, o);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                x[t] -= o.r[t];
                v[t] -= o.v[t];
            }
            c += o.cJ;
            divv += o.divvJ;
            xm += o.xmJ;
            kx += o.kxJ;
        }
    }
    const bool at = !TwoSided;
    put(a.bx, k, x[0], at);
    put(a.by, k, x[1], at);
    put(a.bz, k, x[2], at);
    put(a.bvx, k, v[0], at);
    put(a.bvy, k, v[1], at);
    put(a.bvz, k, v[2], at);
    put(a.cB, k, c, at);
    put(a.bh, k, h, at);
    put(a.divvB, k, divv, at);
    put(a.xmB, k, xm, at);
    put(a.kxB, k, kx, at);
}

// scatter form over the owned lists: a mutual pair gives both directed terms (avAdj) from one geometry.
// With r and v of i's side, i's term of G_i enters through rc = r . C_i Gbar_i; j's is the same with
// the roles swapped, -r and the opposite divv difference.  Position partials along r are summed for
// both ends before the one division by |r|; the pair that set a signal velocity is the rare branch.
// FP64-pipe bound: about 80 instructions per pair with both terms (157 when each term was formed by
// itself; 1M particles: 15.4 -> 8.5 ms).
template<bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) veAvAdjOnceKernel(VeAdjArgs a, OwnedView ov)
{
    const KTab<Smooth> tw{a.wh};
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double x[3] = {0, 0, 0}, v[3] = {0, 0, 0}, R[3] = {0, 0, 0}, c = 0, h = 0, divv = 0, xm = 0, kx = 0;
    const AvSeedV sk = avSeedOf(a, k);
    const double hDxK = a.hDx[k], hk3K = a.hk3[k], hk4K = a.hk4[k], divvK = a.divv[k], volK = a.vol[k],
                 kxInvK = a.kxInv[k], kxvK = a.kxv[k];
    const OwnGeom og(a, k);
    const unsigned cnt = ov.size(k);
    for (unsigned q = blockIdx.y; q < cnt; q += gridDim.y) {
        bool mutual;
        const uint32_t j = ov.at(k, q, mutual);
        AvSeedV sj{};
        if (mutual) sj = avSeedOf(a, j);
        double vsigb = 0.0;  // of the ends whose signal velocity this pair set
        if (sk.any && j == sk.arg) vsigb += sk.vsigb;
        if (mutual && sj.any && uint32_t(k) == sj.arg) vsigb += sj.vsigb;
        if (!sk.gAny && !sj.gAny && vsigb == 0.0) continue;
        double r[3], d, rinv, g[3] = {0.0, 0.0, 0.0}, db = 0.0, divvb = 0.0;
        og.r(a, j, mutual, r, d, rinv);
        const double ddiv = divvK - __ldg(a.divv + j);
        if (sk.gAny) {
            const double xi = d * hDxK;
            double ty;
            const double w = lookupXSlope(tw, xi, ty);
            const double rc = r[0] * sk.CGb[0] + r[1] * sk.CGb[1] + r[2] * sk.CGb[2];
            const double W = hk3K * w, fac = __ldg(a.vol + j) * ddiv, gw = W * rc, fw = fac * W, u = gw * ddiv;
            const double b4 = -fac * rc * hk4K;
            divvb = gw * __ldg(a.vol + j);
            h = fma(-b4, fma(xi, ty, 3.0 * w), h);
            db = b4 * ty;
            atomicAdd(a.xmB + j, -u * __ldg(a.kxInv + j));
            atomicAdd(a.kxB + j, u * __ldg(a.kxv + j));
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                g[t] = -fw * sk.CGb[t];
                R[t] = fma(fw, r[t], R[t]);
            }
        }
        if (sj.gAny) {
            const double xj = d * __ldg(a.hDx + j);
            double ty;
            const double w = lookupXSlope(tw, xj, ty);
            const double rc = r[0] * sj.CGb[0] + r[1] * sj.CGb[1] + r[2] * sj.CGb[2];  // -(r_ji . C_j Gbar_j)
            const double W = __ldg(a.hk3 + j) * w, fac = volK * ddiv, gw = W * rc, fw = fac * W, u = gw * ddiv;
            const double b4 = -fac * rc * __ldg(a.hk4 + j);
            divvb = fma(gw, volK, divvb);
            xm = fma(-u, kxInvK, xm);
            kx = fma(u, kxvK, kx);
            db = fma(b4, ty, db);
            atomicAdd(a.bh + j, -b4 * fma(xj, ty, 3.0 * w));
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                g[t] = fma(-fw, sj.CGb[t], g[t]);
                atomicAdd(a.Rav + t * a.n + j, fw * r[t]);
            }
        }
        divv -= divvb;
        double dr = kTabInvDx * db * rinv;
        if (vsigb != 0.0) {  // c_i + c_j - 3 (r.v) / |r|
            double vv[3];
            og.v(a, j, vv);
            const double rv = r[0] * vv[0] + r[1] * vv[1] + r[2] * vv[2], rvb = -3.0 * vsigb * rinv;
            dr -= rvb * rv * rinv * rinv;
            c += vsigb;
            atomicAdd(a.cB + j, vsigb);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                g[t] = fma(rvb, vv[t], g[t]);
                v[t] = fma(rvb, r[t], v[t]);
            }
            atomicAdd(a.bvx + j, -rvb * r[0]);
            atomicAdd(a.bvy + j, -rvb * r[1]);
            atomicAdd(a.bvz + j, -rvb * r[2]);
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            g[t] = fma(dr, r[t], g[t]);
            x[t] += g[t];
        }
        atomicAdd(a.bx + j, -g[0]);
        atomicAdd(a.by + j, -g[1]);
        atomicAdd(a.bz + j, -g[2]);
        atomicAdd(a.divvB + j, divvb);
    }
    atomicAdd(a.bx + k, x[0]);
    atomicAdd(a.by + k, x[1]);
    atomicAdd(a.bz + k, x[2]);
    atomicAdd(a.bvx + k, v[0]);
    atomicAdd(a.bvy + k, v[1]);
    atomicAdd(a.bvz + k, v[2]);
    atomicAdd(a.cB + k, c);
    atomicAdd(a.bh + k, h);
    atomicAdd(a.divvB + k, divv);
    atomicAdd(a.xmB + k, xm);
    atomicAdd(a.kxB + k, kx);
#pragma unroll
    for (int t = 0; t < 3; ++t) atomicAdd(a.Rav + t * a.n + k, R[t]);
}

// ---------------------------------------------------------------- IAD + divv
__global__ void veIadSeedKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double C[6], Cb[6], gb[6], P[9], tauB[6], PB[9];
    loadC(a, k, C);
#pragma unroll
    for (int t = 0; t < 6; ++t) {
        Cb[t] = a.CB[t * a.n + k];
        gb[t] = a.avClean ? a.gB[t * a.n + k] : 0.0;
    }
    {  // C partials of the AV pair terms
        const double Gb[3] = {a.GB[k], a.GB[a.n + k], a.GB[2 * a.n + k]};
        const double R[3] = {a.Rav[k], a.Rav[a.n + k], a.Rav[2 * a.n + k]};
        avCbar(Gb, R, Cb);
    }
#pragma unroll
    for (int t = 0; t < 9; ++t) P[t] = a.P[t * a.n + k];
    double hb = 0.0, kxb = 0.0;
    iadDivvSeed(a.K, a.h[k], a.kx[k], C, Cb, a.divvB[k], gb, P, tauB, PB, hb, kxb);
#pragma unroll
    for (int t = 0; t < 6; ++t) a.tauB[t * a.n + k] = tauB[t];
#pragma unroll
    for (int t = 0; t < 9; ++t) a.PB[t * a.n + k] = PB[t];
    a.bh[k] += hb;
    a.kxB[k] += kxb;
}

template<bool Smooth>
__device__ __forceinline__ void iadPair(const VeAdjArgs& a, int64_t i, int64_t j, const double tauB[6],
                                        const double PB[9], IadGrad& o)
{
    const KTab<Smooth> tw{a.wh};
    double r[3], d, rinv, v[3];
    geom(a, i, j, r, d, rinv);
    vdiff(a, i, j, v);
    const double hInv = a.hInv[i];
    double dw;
    const double w = lookupVS(tw, d * hInv, dw);
    iadDivvAdj(r, d, rinv, v, hInv, w, dw, a.vol[j], a.kxInv[j], a.xm[j], tauB, PB, o);
}

__device__ __forceinline__ void iadSeedOf(const VeAdjArgs& a, int64_t i, double tauB[6], double PB[9])
{
#pragma unroll
    for (int t = 0; t < 6; ++t) tauB[t] = a.tauB[t * a.n + i];
#pragma unroll
    for (int t = 0; t < 9; ++t) PB[t] = a.PB[t * a.n + i];
}

template<bool TwoSided, bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) veIadAdjKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double x[3] = {0, 0, 0}, v[3] = {0, 0, 0}, h = 0, xm = 0, kx = 0;
    {
        double tauB[6], PB[9];
        iadSeedOf(a, k, tauB, PB);
        const unsigned nc = a.lv.capped(k);
        for (unsigned q = 0; q < nc; ++q) {
            const int64_t j = a.lv.at(k, q);
            IadGrad o;
            iadPair<Smooth>(a, k, j, tauB, PB, o);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                x[t] += o.r[t];
                v[t] += o.v[t];
            }
            h += o.hI;
            if (!TwoSided) {
                atomicAdd(a.bx + j, -o.r[0]);
                atomicAdd(a.by + j, -o.r[1]);
                atomicAdd(a.bz + j, -o.r[2]);
                atomicAdd(a.bvx + j, -o.v[0]);
                atomicAdd(a.bvy + j, -o.v[1]);
                atomicAdd(a.bvz + j, -o.v[2]);
                atomicAdd(a.xmB + j, o.xmJ);
                atomicAdd(a.kxB + j, o.kxJ);
            }
        }
    }
    if (TwoSided) {
        for (uint32_t e = a.tOff[k]; e < a.tOff[k + 1]; ++e) {
            const int64_t i = a.tIdx[e];
            double tauB[6], PB[9];
            iadSeedOf(a, i, tauB, PB);
            IadGrad o;
            iadPair<Smooth>(a, i, k, tauB, PB, o);
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                x[t] -= o.r[t];
                v[t] -= o.v[t];
            }
            xm += o.xmJ;
            kx += o.kxJ;
        }
    }
    const bool at = !TwoSided;
    put(a.bx, k, x[0], at);
    put(a.by, k, x[1], at);
    put(a.bz, k, x[2], at);
    put(a.bvx, k, v[0], at);
    put(a.bvy, k, v[1], at);
    put(a.bvz, k, v[2], at);
    put(a.bh, k, h, at);
    put(a.xmB, k, xm, at);
    put(a.kxB, k, kx, at);
}

// scatter form over the owned lists: a mutual pair gives both directed terms (iadDivvAdj) from one
// geometry.  In r and v of i's side both have one form: with T = tauB r, Q = r . T, p = PB r and
// e = v . p, the term of an end with weights (vol, xm) of the other is 2 vol w T - xm w PB^T v in r,
// -xm w p in v, and (vol Q - xm e) dw/d|r| along r.  FP64-pipe bound: about 140 instructions per pair
// (201 when each term was formed by itself; 1M particles: 19.7 -> 13.3 ms).
template<bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) veIadAdjOnceKernel(VeAdjArgs a, OwnedView ov)
{
    const KTab<Smooth> tw{a.wh};
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double x[3] = {0, 0, 0}, v[3] = {0, 0, 0}, h = 0, xm = 0, kx = 0;
    double tauK[6], PK[9];
    iadSeedOf(a, k, tauK, PK);
    const double hDxK = a.hDx[k], volK = a.vol[k], xmK = a.xm[k], kxInvK = a.kxInv[k], kxvK = a.kxv[k];
    const OwnGeom og(a, k);
    const unsigned cnt = ov.size(k);
    for (unsigned q = blockIdx.y; q < cnt; q += gridDim.y) {
        bool mutual;
        const uint32_t j = ov.at(k, q, mutual);
        double r[3], d, rinv, vv[3], g[3], vb[3], db;
        og.r(a, j, mutual, r, d, rinv);
        og.v(a, j, vv);
        // one end's term: weights of the other end, table coordinate x = |r| / (h dx) of this end
        auto term = [&](const double tau[6], const double PB[9], double vol, double xmo, double kxInv, double kxv, double xt,
                        double hDx, bool add, double& wQ, double& kxb, double& hb) {
            double ty, T[3];
            const double w = lookupXSlope(tw, xt, ty);
            symv(tau, r, T);
            const double Q = r[0] * T[0] + r[1] * T[1] + r[2] * T[2];
            double e = 0.0, p[3];
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                p[t] = PB[3 * t] * r[0] + PB[3 * t + 1] * r[1] + PB[3 * t + 2] * r[2];
                e = fma(vv[t], p[t], e);
            }
            const double a2 = 2.0 * vol * w, bw = xmo * w;
#pragma unroll
            for (int t = 0; t < 3; ++t) {
                const double pt = vv[0] * PB[t] + vv[1] * PB[3 + t] + vv[2] * PB[6 + t];
                g[t] = add ? fma(a2, T[t], fma(-bw, pt, g[t])) : fma(a2, T[t], -bw * pt);
                vb[t] = add ? fma(-bw, p[t], vb[t]) : -bw * p[t];
            }
            const double wb = fma(vol, Q, -xmo * e) * ty;
            wQ = w * fma(Q, kxInv, -e);
            kxb = -w * Q * kxv;
            hb = -wb * xt;
            db = add ? fma(wb, hDx, db) : wb * hDx;
        };
        double xb, kb, hb;
        term(tauK, PK, __ldg(a.vol + j), __ldg(a.xm + j), __ldg(a.kxInv + j), __ldg(a.kxv + j), d * hDxK, hDxK, false, xb,
             kb, hb);
        h += hb;
        atomicAdd(a.xmB + j, xb);
        atomicAdd(a.kxB + j, kb);
        if (mutual) {
            double tauJ[6], PJ[9];
            iadSeedOf(a, j, tauJ, PJ);
            const double hDxJ = __ldg(a.hDx + j);
            term(tauJ, PJ, volK, xmK, kxInvK, kxvK, d * hDxJ, hDxJ, true, xb, kb, hb);
            xm += xb;
            kx += kb;
            atomicAdd(a.bh + j, hb * __ldg(a.hInv + j));
        }
        const double dr = db * rinv;
#pragma unroll
        for (int t = 0; t < 3; ++t) {
            g[t] = fma(dr, r[t], g[t]);
            x[t] += g[t];
            v[t] += vb[t];
        }
        atomicAdd(a.bx + j, -g[0]);
        atomicAdd(a.by + j, -g[1]);
        atomicAdd(a.bz + j, -g[2]);
        atomicAdd(a.bvx + j, -vb[0]);
        atomicAdd(a.bvy + j, -vb[1]);
        atomicAdd(a.bvz + j, -vb[2]);
    }
    atomicAdd(a.bx + k, x[0]);
    atomicAdd(a.by + k, x[1]);
    atomicAdd(a.bz + k, x[2]);
    atomicAdd(a.bvx + k, v[0]);
    atomicAdd(a.bvy + k, v[1]);
    atomicAdd(a.bvz + k, v[2]);
    atomicAdd(a.bh + k, h * a.hInv[k]);
    atomicAdd(a.xmB + k, xm);
    atomicAdd(a.kxB + k, kx);
}

// ---------------------------------------------------------------- EOS, gradh, xmass
__global__ void veEosAdjKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double kxb = a.kxB[k], xmb = a.xmB[k], gradhb = 0.0, ub = 0.0;
    eosAdj(a.gamma, a.u[k], a.m[k], a.kx[k], a.xm[k], a.gradh[k], a.c[k], a.prhoB[k], a.cB[k], a.rhoB[k], kxb, xmb,
           gradhb, ub);
    a.kxB[k] = kxb;
    a.xmB[k] = xmb;
    a.gradhB[k] = gradhb;
    a.bu[k] = ub;
}

__global__ void veGradhSeedKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double skx, som, sr0, hb = 0.0, xmb = 0.0;
    gradhSeed(a.K, a.h[k], a.m[k], a.xm[k], a.kx[k], a.wom[k], a.wr0[k], a.kxB[k], a.gradhB[k], skx, som, sr0, hb, xmb);
    a.Skx[k] = skx;
    a.Som[k] = som;
    a.Sr0[k] = sr0;
    a.bh[k] += hb;
    a.xmB[k] += xmb;
}

template<bool Smooth>
__device__ __forceinline__ void gradhPair(const VeAdjArgs& a, int64_t i, int64_t j, GradhGrad& o)
{
    const KTab<Smooth> tw{a.wh};
    const KTab<Smooth> tdw{a.whd};
    double r[3], d, rinv;
    geom(a, i, j, r, d, rinv);
    const double hInv = a.hInv[i];
    double dw, dwd;
    const double w = lookupVS(tw, d * hInv, dw);
    const double wd = lookupVS(tdw, d * hInv, dwd);
    gradhAdj(r, d, rinv, hInv, w, dw, wd, dwd, a.xm[j], a.m[j], a.Skx[i], a.Som[i], a.Sr0[i], o);
}

template<bool TwoSided, bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) veGradhAdjKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double x[3] = {0, 0, 0}, h = 0, xm = 0;
    const unsigned nc = a.lv.capped(k);
    for (unsigned q = 0; q < nc; ++q) {
        const int64_t j = a.lv.at(k, q);
        GradhGrad o;
        gradhPair<Smooth>(a, k, j, o);
#pragma unroll
        for (int t = 0; t < 3; ++t) x[t] += o.r[t];
        h += o.hI;
        if (!TwoSided) {
            atomicAdd(a.bx + j, -o.r[0]);
            atomicAdd(a.by + j, -o.r[1]);
            atomicAdd(a.bz + j, -o.r[2]);
            atomicAdd(a.xmB + j, o.xmJ);
        }
    }
    if (TwoSided) {
        for (uint32_t e = a.tOff[k]; e < a.tOff[k + 1]; ++e) {
            const int64_t i = a.tIdx[e];
            GradhGrad o;
            gradhPair<Smooth>(a, i, k, o);
#pragma unroll
            for (int t = 0; t < 3; ++t) x[t] -= o.r[t];
            xm += o.xmJ;
        }
    }
    const bool at = !TwoSided;
    put(a.bx, k, x[0], at);
    put(a.by, k, x[1], at);
    put(a.bz, k, x[2], at);
    put(a.bh, k, h, at);
    put(a.xmB, k, xm, at);
}

// scatter form over the owned lists (gradhAdj at both ends of a mutual pair).  In table units, x = v / dx
// and slopes d/dx, an end's radial partial is B / (h dx) and its h partial -B x / h with
// B = wb w' - dx q (wd + x wd'), q = S_om xm + S_r0 m of the other end, wb = S_kx xm - 3 q.  FP64-pipe
// bound (1M particles: 8.2 -> 5.7 ms; xmass below 5.2 -> 3.2).
template<bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) veGradhAdjOnceKernel(VeAdjArgs a, OwnedView ov)
{
    constexpr double dx = 1.0 / kTabInvDx;
    const KTab<Smooth> tw{a.wh};
    const KTab<Smooth> tdw{a.whd};
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double x[3] = {0, 0, 0}, h = 0, xm = 0;
    const double hDxK = a.hDx[k], skx = a.Skx[k], som = a.Som[k], sr0 = a.Sr0[k], xmK = a.xm[k], mK = a.m[k];
    const OwnGeom og(a, k);
    const unsigned cnt = ov.size(k);
    // B of one end at table coordinate xt, with that end's seeds and the other end's xm and m; xmb: the
    // other end's xm partial
    auto term = [&](double xt, double sk, double so, double s0, double xmo, double mo, double& xmb) {
        const TabSlot sl = tabSlot(xt);
        double ty = 0.0, tyd = 0.0, w = 0.0, wd = 0.0;
        if (sl.k >= 0) {
            w = lookupXSlope(tw, sl, ty);
            wd = lookupXSlope(tdw, sl, tyd);
        }
        const double q = fma(so, xmo, s0 * mo), wb = fma(-3.0, q, sk * xmo);
        xmb = fma(sk, w, -so * fma(xt * dx, wd, 3.0 * w));
        return fma(wb, ty, -(dx * q) * fma(xt, tyd, wd));
    };
    for (unsigned q = blockIdx.y; q < cnt; q += gridDim.y) {
        bool mutual;
        const uint32_t j = ov.at(k, q, mutual);
        double r[3], d, rinv, xmb;
        og.r(a, j, mutual, r, d, rinv);
        const double xk = d * hDxK;
        const double bk = term(xk, skx, som, sr0, __ldg(a.xm + j), __ldg(a.m + j), xmb);
        h = fma(-bk, xk, h);
        double db = bk * hDxK;
        atomicAdd(a.xmB + j, xmb);
        if (mutual) {
            const double hDxJ = __ldg(a.hDx + j), xj = d * hDxJ;
            const double bj = term(xj, __ldg(a.Skx + j), __ldg(a.Som + j), __ldg(a.Sr0 + j), xmK, mK, xmb);
            db = fma(bj, hDxJ, db);
            xm += xmb;
            atomicAdd(a.bh + j, -bj * xj * __ldg(a.hInv + j));
        }
        const double dr = db * rinv;
#pragma unroll
        for (int t = 0; t < 3; ++t) x[t] = fma(dr, r[t], x[t]);
        atomicAdd(a.bx + j, -dr * r[0]);
        atomicAdd(a.by + j, -dr * r[1]);
        atomicAdd(a.bz + j, -dr * r[2]);
    }
    atomicAdd(a.bx + k, x[0]);
    atomicAdd(a.by + k, x[1]);
    atomicAdd(a.bz + k, x[2]);
    atomicAdd(a.bh + k, h * a.hInv[k]);
    atomicAdd(a.xmB + k, xm);
}

__global__ void veXmassSeedKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double r0b, hb = 0.0;
    xmassSeed(a.K, a.h[k], a.m[k], a.xm[k], a.xmB[k], r0b, hb);
    a.R0b[k] = r0b;
    a.bh[k] += hb;
}

template<bool Smooth>
__device__ __forceinline__ void xmassPair(const VeAdjArgs& a, int64_t i, int64_t j, double rb[3], double& hIb)
{
    const KTab<Smooth> tw{a.wh};
    double r[3], d, rinv;
    geom(a, i, j, r, d, rinv);
    const double hInv = a.hInv[i];
    double dw;
    lookupVS(tw, d * hInv, dw);
    xmassAdj(r, d, rinv, hInv, dw, a.m[j], a.R0b[i], rb, hIb);
}

template<bool TwoSided, bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) veXmassAdjKernel(VeAdjArgs a)
{
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double x[3] = {0, 0, 0}, h = 0;
    const unsigned nc = a.lv.capped(k);
    for (unsigned q = 0; q < nc; ++q) {
        const int64_t j = a.lv.at(k, q);
        double rb[3], hIb;
        xmassPair<Smooth>(a, k, j, rb, hIb);
#pragma unroll
        for (int t = 0; t < 3; ++t) x[t] += rb[t];
        h += hIb;
        if (!TwoSided) {
            atomicAdd(a.bx + j, -rb[0]);
            atomicAdd(a.by + j, -rb[1]);
            atomicAdd(a.bz + j, -rb[2]);
        }
    }
    if (TwoSided) {
        for (uint32_t e = a.tOff[k]; e < a.tOff[k + 1]; ++e) {
            const int64_t i = a.tIdx[e];
            double rb[3], hIb;
            xmassPair<Smooth>(a, i, k, rb, hIb);
#pragma unroll
            for (int t = 0; t < 3; ++t) x[t] -= rb[t];
        }
    }
    const bool at = !TwoSided;
    put(a.bx, k, x[0], at);
    put(a.by, k, x[1], at);
    put(a.bz, k, x[2], at);
    put(a.bh, k, h, at);
}

template<bool Smooth>
__global__ void __launch_bounds__(kVeAdjBlock) veXmassAdjOnceKernel(VeAdjArgs a, OwnedView ov)
{
    const KTab<Smooth> tw{a.wh};
    const int64_t k = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (k >= a.n) return;
    double x[3] = {0, 0, 0}, h = 0;
    const double hDxK = a.hDx[k], r0b = a.R0b[k], mK = a.m[k];
    const OwnGeom og(a, k);
    const unsigned cnt = ov.size(k);
    for (unsigned q = blockIdx.y; q < cnt; q += gridDim.y) {
        bool mutual;
        const uint32_t j = ov.at(k, q, mutual);
        double r[3], d, rinv, ty;
        og.r(a, j, mutual, r, d, rinv);
        const double xk = d * hDxK;
        lookupXSlope(tw, xk, ty);
        const double bk = r0b * __ldg(a.m + j) * ty;
        h = fma(-bk, xk, h);
        double db = bk * hDxK;
        if (mutual) {
            const double hDxJ = __ldg(a.hDx + j), xj = d * hDxJ;
            lookupXSlope(tw, xj, ty);
            const double bj = __ldg(a.R0b + j) * mK * ty;
            db = fma(bj, hDxJ, db);
            atomicAdd(a.bh + j, -bj * xj * __ldg(a.hInv + j));
        }
        const double dr = db * rinv;
#pragma unroll
        for (int t = 0; t < 3; ++t) x[t] = fma(dr, r[t], x[t]);
        atomicAdd(a.bx + j, -dr * r[0]);
        atomicAdd(a.by + j, -dr * r[1]);
        atomicAdd(a.bz + j, -dr * r[2]);
    }
    atomicAdd(a.bx + k, x[0]);
    atomicAdd(a.by + k, x[1]);
    atomicAdd(a.bz + k, x[2]);
    atomicAdd(a.bh + k, h * a.hInv[k]);
}

}  // namespace

// number of n-sized double sections of the VE adjoint state
constexpr int kVeAdjSections = 82;

int anySeed(sphgb_ctx* c, const double* seed, int64_t n, bool& any)
{
    SPHGB_TRY(c->reduceScratch.ensure(sizeof(unsigned long long) * 4));
    int* dev = c->reduceScratch.as<int>();
    int got = 0;
    SPHGB_CUDA(cudaMemsetAsync(dev, 0, sizeof(int), c->stream));
    anySeedKernel<<<gridFor(n, 256), 256, 0, c->stream>>>(seed, n, dev);
    SPHGB_TRY(launched(c, "anySeedKernel"));
    SPHGB_CUDA(cudaMemcpyAsync(&got, dev, sizeof(int), cudaMemcpyDeviceToHost, c->stream));
    SPHGB_CUDA(cudaStreamSynchronize(c->stream));
    any = got != 0;
    return SPHGB_OK;
}

int adjointVe(sphgb_ctx* c, sphgb_particles* p, const double* alphaPrev, int avClean, const sphgb_seeds* s,
              sphgb_grads* g, int deterministic)
{
    if (!c->haveNbr) return SPHGB_ERR_STATE;
    if (p->precision != SPHGB_FP64) return SPHGB_ERR_ARG;
    if (c->nbrFirst != 0 || c->nbrLast != p->n) return SPHGB_ERR_ARG;
    if (!alphaPrev || !p->x || !p->y || !p->z || !p->vx || !p->vy || !p->vz || !p->h || !p->m || !p->u || !p->alpha ||
        !p->xm || !p->kx || !p->gradh || !p->prho || !p->c || !p->divv || !p->c11 || !p->c12 || !p->c13 || !p->c22 ||
        !p->c23 || !p->c33)
        return SPHGB_ERR_ARG;
    if (avClean && (!p->dV11 || !p->dV12 || !p->dV13 || !p->dV22 || !p->dV23 || !p->dV33)) return SPHGB_ERR_ARG;
    if (!g || !g->x || !g->y || !g->z || !g->vx || !g->vy || !g->vz || !g->h || !g->u) return SPHGB_ERR_ARG;
    const int64_t n = p->n;
    if (deterministic) SPHGB_TRY(buildTranspose(c));
    SPHGB_TRY(c->adjState.ensure(sizeof(double) * kVeAdjSections * n));
    double* st = c->adjState.as<double>();

    VeAdjArgs a{};
    auto d = [](const void* q) { return static_cast<const double*>(q); };
    a.x = p->x;
    a.y = p->y;
    a.z = p->z;
    a.vx = d(p->vx);
    a.vy = d(p->vy);
    a.vz = d(p->vz);
    a.h = d(p->h);
    a.m = d(p->m);
    a.u = p->u;
    a.alpha0 = alphaPrev;
    a.alpha = d(p->alpha);
    a.xm = d(p->xm);
    a.kx = d(p->kx);
    a.gradh = d(p->gradh);
    a.prho = d(p->prho);
    a.c = d(p->c);
    a.divv = d(p->divv);
    const void* Cs[6] = {p->c11, p->c12, p->c13, p->c22, p->c23, p->c33};
    const void* dVs[6] = {p->dV11, p->dV12, p->dV13, p->dV22, p->dV23, p->dV33};
    for (int q = 0; q < 6; ++q) {
        a.C[q] = d(Cs[q]);
        a.dV[q] = avClean ? d(dVs[q]) : nullptr;
    }
    a.wh = tabW64(c);
    a.whd = tabDW64(c);
    a.K = c->K;
    a.gamma = c->prm.gamma;
    a.av = AvPrm{c->K, c->prm.minDt, c->prm.alphamin, c->prm.alphamax, c->prm.decay_constant};
    a.box = c->box;
    a.cf = coordFp64(c, p);
    a.expTab = c->expTab.as<double4>();
    {  // FP32 error of a position difference: a few ulp of the largest coordinate plus a box edge
        double xmax = 0.0, lmax = 0.0;
        for (int k = 0; k < 3; ++k) {
            xmax = fmax(xmax, fmax(fabs(c->box.lo[k]), fabs(c->box.hi[k])));
            lmax = fmax(lmax, c->box.L[k]);
        }
        a.ePos = float(4.0 * 0x1p-24 * (xmax + lmax) * 1.001);
    }
    a.avClean = avClean ? 1 : 0;
    a.lv = listView(c);
    a.tOff = c->tOff.as<uint32_t>();
    a.tIdx = c->tIdx.as<uint32_t>();
    a.n = n;
    if (s) {
        a.sRho = d(s->rho);
        a.sAx = d(s->ax);
        a.sAy = d(s->ay);
        a.sAz = d(s->az);
        a.sDu = s->du;
    }
    a.bx = g->x;
    a.by = g->y;
    a.bz = g->z;
    a.bvx = g->vx;
    a.bvy = g->vy;
    a.bvz = g->vz;
    a.bh = g->h;
    a.bu = g->u;
    double* q = st;
    auto take = [&](int sections) {
        double* r = q;
        q += int64_t(sections) * n;
        return r;
    };
    // accumulators first: one memset clears them
    a.prhoB = take(1);
    a.cB = take(1);
    a.alphaB = take(1);
    a.rhoB = take(1);
    a.xmB = take(1);
    a.kxB = take(1);
    a.CB = take(6);
    a.gB = take(6);
    a.divvB = take(1);
    a.gradhB = take(1);
    a.Rav = take(3);
    const int64_t accSections = 23;
    a.hInv = take(1);
    a.rho = take(1);
    a.rhoInv = take(1);
    a.vol = take(1);
    a.kxInv = take(1);
    a.xmInv = take(1);
    a.lnxm = take(1);
    a.hDx = take(1);
    a.hk3 = take(1);
    a.hk4 = take(1);
    a.kxv = take(1);
    a.en = take(1);
    a.avE = take(1);
    a.G = take(3);
    a.vsig = take(1);
    a.P = take(9);
    a.wom = take(1);
    a.wr0 = take(1);
    a.vsigArg = reinterpret_cast<uint32_t*>(take(1));
    a.GB = take(3);
    a.CGB = take(3);
    a.vsigB = take(1);
    a.tauB = take(6);
    a.PB = take(9);
    a.Skx = take(1);
    a.Som = take(1);
    a.Sr0 = take(1);
    a.R0b = take(1);
    a.xc32 = reinterpret_cast<float4*>(take(2));
    a.v32 = reinterpret_cast<float4*>(take(2));
    if ((reinterpret_cast<uintptr_t>(a.xc32) | reinterpret_cast<uintptr_t>(a.v32)) & 15) return SPHGB_ERR_STATE;
    if (q - st > int64_t(kVeAdjSections) * n) return SPHGB_ERR_TOO_LARGE;  // layout and size disagree

    for (double* z : {g->x, g->y, g->z, g->vx, g->vy, g->vz, g->h, g->u})
        SPHGB_CUDA(cudaMemsetAsync(z, 0, sizeof(double) * n, c->stream));
    SPHGB_CUDA(cudaMemsetAsync(st, 0, sizeof(double) * accSections * n, c->stream));

    const unsigned pb = gridFor(n, kVeAdjBlock), eb = gridFor(n, 256);
    const bool two = deterministic != 0;
    veQuotKernel<<<eb, 256, 0, c->stream>>>(a);
    SPHGB_TRY(launched(c, "veQuotKernel"));
    bool withDu = a.sDu != nullptr;
    if (withDu) {  // a du seed that is zero everywhere (autograd's for an unused output) is none
        SPHGB_TRY(anySeed(c, a.sDu, n, withDu));
        if (!withDu) a.sDu = nullptr;
    }
    // forward sums kept by the forward passes on these lists (sphgb_set_adjoint_tape) are read from
    // the tape instead of being summed again; vsig_i and its pair are always found here
    constexpr unsigned kTapeNeeded = kTapeGradh | kTapeIad | kTapeAv;
    const bool taped = c->tapeEpoch == c->nbrEpoch && c->tapeN == n && (c->tapeMask & kTapeNeeded) == kTapeNeeded;
    const bool tapedMe = taped && (c->tapeMask & kTapeMe) != 0;
    if (taped) {
        double* tp = c->veTape.as<double>();
        a.G = tp + int64_t(kTapeG) * n;
        a.P = tp + int64_t(kTapeP) * n;
        a.wom = tp + int64_t(kTapeWom) * n;
        a.wr0 = tp + int64_t(kTapeWr0) * n;
        if (tapedMe) {
            a.en = tp + int64_t(kTapeEn) * n;
            a.avE = tp + int64_t(kTapeAvE) * n;
        }
    }
    return withKernelForm(c, [&](auto smooth) -> int {
        constexpr bool S = decltype(smooth)::value;
        if (withDu && !tapedMe) {  // en and avE enter only through the du seed
            vePreMeKernel<S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
            SPHGB_TRY(launched(c, "vePreMeKernel"));
        }
        if (taped) {
            veArgKernel<<<pb, kVeAdjBlock, 0, c->stream>>>(a);
            SPHGB_TRY(launched(c, "veArgKernel"));
        } else {
            vePreKernel<S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
            SPHGB_TRY(launched(c, "vePreKernel"));
        }
        {
            using K = void (*)(VeAdjArgs);
            // [two-sided][avClean][du seed]
            const K me[2][2][2] = {{{meVeAdjKernel<false, false, false, S>, meVeAdjKernel<false, false, true, S>},
                                    {meVeAdjKernel<false, true, false, S>, meVeAdjKernel<false, true, true, S>}},
                                   {{meVeAdjKernel<true, false, false, S>, meVeAdjKernel<true, false, true, S>},
                                    {meVeAdjKernel<true, true, false, S>, meVeAdjKernel<true, true, true, S>}}};
            // one evaluation per mutual pair: owned lists of the current lists, order-free sums allowed
            if (!two && !c->deterministic && !a.avClean && c->ownedEpoch == c->nbrEpoch && !c->ownedFromLists) {
                if (withDu) meVeAdjOnceKernel<S><<<pb, kVeAdjBlock, 0, c->stream>>>(a, ownedView(c));
                else meVeAdjOnceAKernel<S><<<ownedGrid(n), kVeAdjBlock, 0, c->stream>>>(a, ownedView(c));
            } else
                me[two][a.avClean][withDu]<<<pb, kVeAdjBlock, 0, c->stream>>>(a);
            SPHGB_TRY(launched(c, "meVeAdjKernel"));
        }
        veAvSeedKernel<<<eb, 256, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veAvSeedKernel"));
        const bool once = !two && !c->deterministic && c->ownedEpoch == c->nbrEpoch && !c->ownedFromLists;
        if (two) veAvAdjKernel<true, S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
        else if (once) veAvAdjOnceKernel<S><<<ownedGrid(n), kVeAdjBlock, 0, c->stream>>>(a, ownedView(c));
        else veAvAdjKernel<false, S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veAvAdjKernel"));
        veIadSeedKernel<<<eb, 256, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veIadSeedKernel"));
        if (two) veIadAdjKernel<true, S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
        else if (once) veIadAdjOnceKernel<S><<<ownedGrid(n), kVeAdjBlock, 0, c->stream>>>(a, ownedView(c));
        else veIadAdjKernel<false, S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veIadAdjKernel"));
        veEosAdjKernel<<<eb, 256, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veEosAdjKernel"));
        veGradhSeedKernel<<<eb, 256, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veGradhSeedKernel"));
        if (two) veGradhAdjKernel<true, S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
        else if (once) veGradhAdjOnceKernel<S><<<ownedGrid(n), kVeAdjBlock, 0, c->stream>>>(a, ownedView(c));
        else veGradhAdjKernel<false, S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veGradhAdjKernel"));
        veXmassSeedKernel<<<eb, 256, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veXmassSeedKernel"));
        if (two) veXmassAdjKernel<true, S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
        else if (once) veXmassAdjOnceKernel<S><<<ownedGrid(n), kVeAdjBlock, 0, c->stream>>>(a, ownedView(c));
        else veXmassAdjKernel<false, S><<<pb, kVeAdjBlock, 0, c->stream>>>(a);
        SPHGB_TRY(launched(c, "veXmassAdjKernel"));
        SPHGB_CUDA(cudaStreamSynchronize(c->stream));
        return SPHGB_OK;
    });
}

}  // namespace sphgb
