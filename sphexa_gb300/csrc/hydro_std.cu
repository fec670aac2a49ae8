// Standard-SPH pair passes: density, ideal-gas EOS, IAD, momentum and energy.
//
// Reference j-loops restated:
//   density  -> xmassJLoop with rho<->xm swapped, then rho = m / xm
//               (sph/include/sph/hydro_std/density.hpp:41-60, hydro_ve/xmass_kern.hpp:50-79)
//   EOS      -> idealGasEOS_u (hydro_std/eos.hpp:54-80, sph/eos.hpp:34-44)
//   IAD      -> IADJLoopSTD (hydro_std/iad_kern.hpp:12-77)
//   ME       -> momentumAndEnergyJLoop + tsKCourant (hydro_std/momentum_energy_kern.hpp:12-134,
//               momentum_energy.hpp:41-101)
// FP64 form: per-particle quotients (m/rho, p/rho, p/rho^2, 1/h, 1/h^3) are formed once per
// particle, 1/|r| comes from rsqrt, periodic wrap tests run only where they can fire; where the lists
// cover every particle a mutual pair is evaluated once, its other end's share passing through a record that
// is gathered in a fixed order (PairRec: the same bits in every run; set_deterministic selects the walks over
// whole lists), and IAD and momentum-energy read the pair geometry that the density pass stored.  Results
// agree with the reference to rounding.  Mixed form: FP32 pair arithmetic on grid-local offsets, Kahan sums, per-particle epilogues (normalisation, 3x3 inverse factor) in FP64.
#include "pairs.cuh"

namespace sphgb {

namespace {

// ---------------------------------------------------------------- density / xmass
// neighbour-side fields of the mixed density / xmass pass: grid position and m in one 32-byte block
// per particle (one 256-bit load)
__global__ void packXmassKernel(int64_t n, const void* m, const u64* __restrict__ cell, const float4* __restrict__ loc,
                                float4* __restrict__ rec)
{
    const int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (j >= n) return;
    packGridBlock(rec + 2 * j, cell[j], loc[j], ld<float>(m, j), 0.f, 0.f);
}

// the same for the mixed IAD pass: grid position and m/rho
__global__ void packIadStdKernel(int64_t n, const void* m, const void* rho, const u64* __restrict__ cell,
                                 const float4* __restrict__ loc, float4* __restrict__ rec)
{
    const int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (j >= n) return;
    packGridBlock(rec + 2 * j, cell[j], loc[j], ld<float>(m, j) / ld<float>(rho, j), 0.f, 0.f);
}

template<class P, bool StoreRho, bool Smooth = false>
__global__ void __launch_bounds__(kPairBlock) xmassKernel(ListView lv, CoordFp64 cf, CoordMixed cm, const void* h,
                                                          const void* m, const void* wh, const double2* w64,
                                                          double K, void* out, const Rec8* rec = nullptr)
{
    const int64_t i = lv.first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= lv.last) return;
    const int64_t ii = i - lv.first;
    const unsigned nc = lv.capped(ii);
    if constexpr (std::is_same_v<P, Fp64Tag>) {
        const KTab<Smooth> tab{w64};
        auto t = cf.target(i);
        double hi = ld<double>(h, i), mi = ld<double>(m, i);
        double hInv = 1.0 / hi, h3Inv = hInv * hInv * hInv, twoH = 2.0 * hi, hInvDx = hInv * kTabInvDx;
        const bool wrap = cf.needsWrap(t, twoH);
        double rho0 = mi;
        for (unsigned k = 0; k < nc; ++k) {
            uint32_t j = lv.at(ii, k);
            double rx, ry, rz;
            cf.diffFast(t, j, twoH, wrap, rx, ry, rz);
            double r2 = dist2(rx, ry, rz);
            rho0 += lookupX(tab, r2 * invDist(r2) * hInvDx) * ld<double>(m, j);
        }
        double xm = mi / (rho0 * K * h3Inv);
        st<double>(out, i, StoreRho ? mi / xm : xm);
    } else {
        auto t = cm.target(i);
        float mi = ld<float>(m, i);
        KSum rho0;
        rho0.add(mi);
        // the list is read a granule (four entries) per load, the next granule one ahead, and the
        // next neighbour's block is loaded while the current pair is evaluated
        uint4 G = nc > 0 ? lv.granule(ii, 0) : make_uint4(uint32_t(i), 0u, 0u, 0u);
        uint4 Gn = nc > 4 ? lv.granule(ii, 1) : G;
        Rec8 Bn = ldRec8(rec + G.x);
        for (unsigned k = 0; k < nc; ++k) {
            const Rec8 B = Bn;  // cell xl yl zl m
            if (k + 1 < nc) {
                const unsigned s = (k + 1) & 3u;
                if (s == 0) {
                    G = Gn;
                    if (k + 5 < nc) Gn = lv.granule(ii, (k + 5) >> 2);
                }
                Bn = ldRec8(rec + pick(G, s));
            }
            float rx, ry, rz;
            cm.diffBlock(t, B, rx, ry, rz);
            float dist = sqrtf(fmaf(rx, rx, fmaf(ry, ry, rz * rz)));
            rho0.add(lookupH32(static_cast<const float4*>(wh), dist * t.hInv) * B.v[5]);
        }
        double hi = double(ld<float>(h, i));
        double rho = rho0.value64() * K / (hi * hi * hi);
        st<float>(out, i, StoreRho ? float(rho) : float(double(mi) / rho));
    }
}

// FP64 xmass / density with one evaluation per mutual pair over the owned lists: i adds
// W(d / h_i) m_j, and for a mutual pair j receives W(d / h_j) m_i.  It also fills the pair-geometry cache
// (geo) that the later pair-once passes read.  Mode: j's share by FP64 atomics, with the rounding errors of the
// sums in acc + n (exactSums) or without (xmass), or by the pair's record (PairRec, std density).
enum XmassMode { kXmassSum, kXmassExact, kXmassRecords };

template<bool Smooth, XmassMode Mode>
__global__ void __launch_bounds__(kPairBlock) xmassOnceKernel(ListView lv, OwnedView ov, CoordFp64 cf,
                                                               const double* h, const double* m, KTab<Smooth> tab,
                                                               const double* hInvDx, double* acc, PairGeo geo,
                                                               const double* vx, const double* vy, const double* vz,
                                                               int64_t n, PairRec pr)
{
    constexpr bool Exact = Mode == kXmassExact;
    const int64_t i = lv.first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= lv.last) return;
    const int64_t ii = i - lv.first;
    const unsigned no = ov.size(ii);
    auto t = cf.target(i);
    const double hi = h[i], mi = m[i], twoH = 2.0 * hi, hiInvDx = hInvDx[i];
    const auto fold = cf.fold(t, twoH);
    const int64_t gb = geo.g ? geo.base(ii) : 0, rb = Mode == kXmassRecords ? pr.base(ii) : 0;
    const double vxi = geo.g ? vx[i] : 0.0, vyi = geo.g ? vy[i] : 0.0, vzi = geo.g ? vz[i] : 0.0;
    double rho0 = 0.0;
    auto give = [&](uint32_t j, unsigned k, double v) {
        if constexpr (Mode == kXmassRecords) reinterpret_cast<double*>(pr.rec)[rb + 32 * int64_t(k)] = v;
        else sumAdd<Exact>(acc + j, acc + n + j, v);
    };
    for (unsigned k = blockIdx.y; k < no; k += gridDim.y) {
        bool mutual;
        const uint32_t j = ov.at(ii, k, mutual);
        double rx, ry, rz;
        cf.diffOwned(t, j, mutual, fold, rx, ry, rz);
        const double r2 = dist2(rx, ry, rz);
        const double rinv = invDist(r2);
        const double dist = r2 * rinv;
        const double wi = lookupX(tab, dist * hiInvDx);
        rho0 += wi * __ldg(m + j);
        if (geo.g) {  // the sweep's later pair-once passes load the geometry and both kernel values
            const double wj = lookupX(tab, dist * __ldg(hInvDx + j));
            const int64_t e = gb + 32 * int64_t(k);
            const double dvx = __ldg(vx + j) - vxi, dvy = __ldg(vy + j) - vyi, dvz = __ldg(vz + j) - vzi;
            // w_ij = (r . v_ij) / |r| with v_ij = -dv, in the order of every FP64 pass
            geo.g[e] = make_double2(dist, -fma(rz, dvz, fma(ry, dvy, rx * dvx)) * rinv);
            geo.w[e] = make_double2(wi, wj);
            if (geo.x) {
                geo.x[e] = make_double2(rx, ry);
                geo.x[geo.plane + e] = make_double2(rz, dvx);
                geo.x[2 * geo.plane + e] = make_double2(dvy, dvz);
            }
            if (mutual) give(j, k, wj * mi);
        } else if (mutual) {
            give(j, k, lookupX(tab, dist * __ldg(hInvDx + j)) * mi);
        }
    }
    if constexpr (Mode == kXmassRecords) pr.part[blockIdx.y * n + i] = rho0;
    else sumAdd<Exact>(acc + i, acc + n + i, rho0);
}

// snap: where it keeps the inputs of the cache (outside a sweep), or null
template<bool StoreRho>
__global__ void xmassOnceFinish(int64_t first, int64_t last, const double* h, const double* m, double K,
                                const double* acc, const double* lo, double* out, GeoInputs in, double* snap,
                                int64_t n)
{
    const int64_t i = first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= last) return;
    const double hi = h[i], mi = m[i];
    const double hInv = 1.0 / hi, h3Inv = hInv * hInv * hInv;
    const double xm = mi / ((mi + (lo ? acc[i] + lo[i] : acc[i])) * K * h3Inv);
    if (snap) {
#pragma unroll
        for (int q = 0; q < kGeoInputs; ++q) snap[q * n + i] = in.f[q][i];
    }
    out[i] = StoreRho ? mi / xm : xm;
}

// ---------------------------------------------------------------- EOS
template<class P>
__global__ void eosStdKernel(int64_t first, int64_t last, const double* u, const void* rho, double gamma, void* p,
                             void* c)
{
    using T = typename P::T;
    int64_t i = first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= last) return;
    double tmp = u[i] * (gamma - 1.0);
    double pi = double(ld<T>(rho, i)) * tmp;
    st<T>(p, i, T(pi));
    st<T>(c, i, T(sqrt(gamma * tmp)));
}

// ---------------------------------------------------------------- per-particle quotients
// aux[0,n) m/rho, [n,2n) p/rho, [2n,3n) p/rho^2
// (FP64; the mixed passes have them in their records)
__global__ void stdAuxKernel(int64_t n, const void* m, const void* rho, const void* p, double* aux)
{
    int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    const double ri = ld<double>(rho, i);
    aux[i] = ld<double>(m, i) / ri;
    if (p) {
        const double pi = ld<double>(p, i);
        aux[n + i] = pi / ri;
        aux[2 * n + i] = pi / (ri * ri);
    }
}

int launchStdAux(sphgb_ctx* c, const sphgb_particles* p, bool withPressure)
{
    const int64_t n = p->n;
    SPHGB_TRY(c->aux.ensure(sizeof(double) * 3 * n));
    stdAuxKernel<<<gridFor(n, 256), 256, 0, c->stream>>>(n, p->m, p->rho, withPressure ? p->p : nullptr,
                                                         c->aux.as<double>());
    return launched(c, "stdAuxKernel");
}

// ---------------------------------------------------------------- IAD
struct IadOut {
    void *c11, *c12, *c13, *c22, *c23, *c33;
};

// vol[j] = m[j] / rho[j], formed once per particle (the reference divides per pair)
template<class P, bool Smooth = false>
__global__ void __launch_bounds__(kPairBlock) iadKernel(ListView lv, CoordFp64 cf, CoordMixed cm, const void* h,
                                                        const void* vol, const void* wh, const double2* w64,
                                                        double K, IadOut o, const Rec8* rec = nullptr)
{
    const int64_t i = lv.first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= lv.last) return;
    const int64_t ii = i - lv.first;
    const unsigned nc = lv.capped(ii);
    if constexpr (std::is_same_v<P, Fp64Tag>) {
        const KTab<Smooth> tab{w64};
        auto t = cf.target(i);
        double hi = ld<double>(h, i), hiInv = 1.0 / hi, twoH = 2.0 * hi, hInvDx = hiInv * kTabInvDx;
        const bool wrap = cf.needsWrap(t, twoH);
        double t11 = 0, t12 = 0, t13 = 0, t22 = 0, t23 = 0, t33 = 0;
        for (unsigned k = 0; k < nc; ++k) {
            uint32_t j = lv.at(ii, k);
            double rx, ry, rz;
            cf.diffFast(t, j, twoH, wrap, rx, ry, rz);
            double r2 = dist2(rx, ry, rz);
            double w = lookupX(tab, r2 * invDist(r2) * hInvDx);
            double vw = ld<double>(vol, j) * w;
            t11 += rx * rx * vw;
            t12 += rx * ry * vw;
            t13 += rx * rz * vw;
            t22 += ry * ry * vw;
            t23 += ry * rz * vw;
            t33 += rz * rz * vw;
        }
        double cc[6];
        iadInvert<double>(t11, t12, t13, t22, t23, t33, hi, K, cc);
        st<double>(o.c11, i, cc[0]);
        st<double>(o.c12, i, cc[1]);
        st<double>(o.c13, i, cc[2]);
        st<double>(o.c22, i, cc[3]);
        st<double>(o.c23, i, cc[4]);
        st<double>(o.c33, i, cc[5]);
    } else {
        const float4* tab = static_cast<const float4*>(wh);
        auto t = cm.target(i);
        KSum t11, t12, t13, t22, t23, t33;
        // granules and blocks one ahead, as in the density pass
        uint4 G = nc > 0 ? lv.granule(ii, 0) : make_uint4(uint32_t(i), 0u, 0u, 0u);
        uint4 Gn = nc > 4 ? lv.granule(ii, 1) : G;
        Rec8 Bn = ldRec8(rec + G.x);
        for (unsigned k = 0; k < nc; ++k) {
            const Rec8 B = Bn;  // cell xl yl zl vol
            if (k + 1 < nc) {
                const unsigned s = (k + 1) & 3u;
                if (s == 0) {
                    G = Gn;
                    if (k + 5 < nc) Gn = lv.granule(ii, (k + 5) >> 2);
                }
                Bn = ldRec8(rec + pick(G, s));
            }
            float rx, ry, rz;
            cm.diffBlock<true>(t, B, rx, ry, rz);
            float dist = sqrtf(fmaf(rx, rx, fmaf(ry, ry, rz * rz)));
            float w = lookupH32(tab, dist * t.hInv);
            float vw = B.v[5] * w;
            t11.add(rx * rx * vw);
            t12.add(rx * ry * vw);
            t13.add(rx * rz * vw);
            t22.add(ry * ry * vw);
            t23.add(ry * rz * vw);
            t33.add(rz * rz * vw);
        }
        float cc[6];
        iadInvert<float>(t11.value(), t12.value(), t13.value(), t22.value(), t23.value(), t33.value(),
                         double(ld<float>(h, i)), K, cc);
        st<float>(o.c11, i, cc[0]);
        st<float>(o.c12, i, cc[1]);
        st<float>(o.c13, i, cc[2]);
        st<float>(o.c22, i, cc[3]);
        st<float>(o.c23, i, cc[4]);
        st<float>(o.c33, i, cc[5]);
    }
}

// FP64 IAD with one evaluation per mutual pair over the owned lists: i adds vol_j W_i r r^T, and a mutual
// pair gives j vol_i W_j r r^T by its record (r and the factor).  Geo: arrays of the pair-geometry cache (5, 2),
// or 0.
template<bool Smooth, int Geo>
__device__ __forceinline__ void iadStdOnceBody(ListView lv, OwnedView ov, CoordFp64 cf,
                                                               const double* h, const double* vol,
                                                               KTab<Smooth> tab, const double* hInv64, int64_t n,
                                                               PairRec pr, PairGeo geo)
{
    const int64_t i = lv.first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= lv.last) return;
    const int64_t ii = i - lv.first;
    const unsigned no = ov.size(ii);
    const double* hInvDx = hInv64 + 2 * n;
    const double voli = vol[i];
    typename CoordFp64::Target t{};
    double twoH = 0, hiInvDx = 0;
    CoordFp64::Fold fold{};
    int64_t g = 0;
    if constexpr (Geo != 0) g = geo.base(ii) + 32 * blockIdx.y;
    if constexpr (Geo != 5) {
        t = cf.target(i);
        twoH = 2.0 * h[i];
        fold = cf.fold(t, twoH);
        hiInvDx = hInvDx[i];
    }
    const int64_t rb = pr.base(ii);
    double tau[6] = {0, 0, 0, 0, 0, 0};
    for (unsigned k = blockIdx.y; k < no; k += gridDim.y, g += 32 * gridDim.y) {
        bool mutual;
        const uint32_t j = ov.at(ii, k, mutual);
        double rx, ry, rz;
        double2 wv;
        if constexpr (Geo != 0) wv = __ldg(geo.w + g);
        if constexpr (Geo == 5) {
            const double2 a0 = __ldg(geo.x + g);
            rx = a0.x, ry = a0.y, rz = __ldg(geo.x + geo.plane + g).x;
        } else {
            cf.diffOwned(t, j, mutual, fold, rx, ry, rz);
        }
        if constexpr (Geo == 0) {
            const double r2 = dist2(rx, ry, rz);
            const double dist = r2 * invDist(r2);
            wv.x = lookupX(tab, dist * hiInvDx);
            wv.y = lookupX(tab, dist * __ldg(hInvDx + j));
        }
        const double s[6] = {rx * rx, rx * ry, rx * rz, ry * ry, ry * rz, rz * rz};
        const double vw = __ldg(vol + j) * wv.x;
#pragma unroll
        for (int q = 0; q < 6; ++q) tau[q] = fma(vw, s[q], tau[q]);
        if (mutual) pr.rec[rb + 32 * int64_t(k)] = {rx, ry, rz, voli * wv.y};
    }
#pragma unroll
    for (int q = 0; q < 6; ++q) pr.part[(blockIdx.y * int64_t(6) + q) * n + i] = tau[q];
}

template<bool Smooth, int Geo>
__global__ void __launch_bounds__(kPairBlock) iadStdOnceKernel(ListView lv, OwnedView ov, CoordFp64 cf,
                                                               const double* h, const double* vol,
                                                               KTab<Smooth> tab, const double* hInv64, int64_t n,
                                                               PairRec pr, PairGeo geo)
{
    if constexpr (Geo >= 0) iadStdOnceBody<Smooth, Geo>(lv, ov, cf, h, vol, tab, hInv64, n, pr, geo);
    else if (*geo.stale) iadStdOnceBody<Smooth, 0>(lv, ov, cf, h, vol, tab, hInv64, n, pr, geo);
    else iadStdOnceBody<Smooth, -Geo>(lv, ov, cf, h, vol, tab, hInv64, n, pr, geo);
}

__global__ void iadStdOnceFinish(int64_t n, const double* h, double K, const double* acc, IadOut o)
{
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= n) return;
    double cc[6];
    iadInvert<double>(acc[i], acc[n + i], acc[2 * n + i], acc[3 * n + i], acc[4 * n + i], acc[5 * n + i], h[i], K, cc);
    st<double>(o.c11, i, cc[0]);
    st<double>(o.c12, i, cc[1]);
    st<double>(o.c13, i, cc[2]);
    st<double>(o.c22, i, cc[3]);
    st<double>(o.c23, i, cc[4]);
    st<double>(o.c33, i, cc[5]);
}

// ---------------------------------------------------------------- momentum and energy (std)
struct MeStdArgs {
    const void *vx, *vy, *vz, *h, *m, *rho, *p, *c;
    const void *c11, *c12, *c13, *c22, *c23, *c33;
    const void* wh;        // mixed: cubic pieces of W
    const double2* w64;    // FP64: W in the context's form
    const double* hInv64;  // [0,n) 1/h, [n,2n) 1/h^3, [2n,3n) 1/(h dx)
    const void* aux;       // m/rho, p/rho, p/rho^2
    int64_t n;
    double K;
    float Kcour;
    void *ax, *ay, *az;
    double* du;
    unsigned long long* minDt;
    const Rec8* pack;  // mixed: three blocks per particle (meStdPackKernel)
};

// neighbour-side fields of the mixed momentum-energy pass as three 32-byte blocks per particle, each read
// by one 256-bit load: {cell (2 words) xl yl zl 1/h vx vy} {vz c c11 c12 c13 c22 c23 c33} {m m/rho p/rho};
// aux (m/rho at 0, p/rho^2 at 2 n) is filled for the targets.  Fifteen gathers per pair before: 298k particles
// 0.42 -> 0.35 ms, and IAD, with one block, 0.17 -> 0.14.
__global__ void meStdPackKernel(int64_t n, MeStdArgs a, const u64* __restrict__ cell, const float4* __restrict__ loc,
                                float* __restrict__ aux, float4* __restrict__ pack)
{
    const int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (j >= n) return;
    const float rho = ld<float>(a.rho, j), m = ld<float>(a.m, j), p = ld<float>(a.p, j);
    const float moR = m / rho, poR = p / (rho * 1.f);
    aux[j] = moR;
    aux[2 * n + j] = p / (1.f * rho * rho);
    const u64 cj = cell[j];
    const float4 l = loc[j];
    float4* q = pack + 6 * j;
    q[0] = make_float4(__uint_as_float(unsigned(cj)), __uint_as_float(unsigned(cj >> 32)), l.x, l.y);
    q[1] = make_float4(l.z, l.w, ld<float>(a.vx, j), ld<float>(a.vy, j));
    q[2] = make_float4(ld<float>(a.vz, j), ld<float>(a.c, j), ld<float>(a.c11, j), ld<float>(a.c12, j));
    q[3] = make_float4(ld<float>(a.c13, j), ld<float>(a.c22, j), ld<float>(a.c23, j), ld<float>(a.c33, j));
    q[4] = make_float4(m, moR, poR, 0.f);  // the block's second half is not read
}

template<class P, bool Smooth = false>
__global__ void __launch_bounds__(kPairBlock) meStdKernel(ListView lv, CoordFp64 cf, CoordMixed cm, MeStdArgs a)
{
    using T = typename P::T;
    const int64_t i0 = lv.first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    const bool valid = i0 < lv.last;
    const int64_t i = valid ? i0 : lv.first;
    const int64_t ii = i - lv.first;
    const unsigned nc = valid ? lv.capped(ii) : 0u;
    const T* aux = static_cast<const T*>(a.aux);
    const T *auxMoR = aux, *auxPoR = aux + a.n, *auxPoR2 = aux + 2 * a.n;
    double dt = INFINITY;

    T hi = ld<T>(a.h, i), ci = ld<T>(a.c, i);
    T vxi = ld<T>(a.vx, i), vyi = ld<T>(a.vy, i), vzi = ld<T>(a.vz, i);
    T mi_roi = auxMoR[i], proi2 = auxPoR2[i];
    T c11i = ld<T>(a.c11, i), c12i = ld<T>(a.c12, i), c13i = ld<T>(a.c13, i);
    T c22i = ld<T>(a.c22, i), c23i = ld<T>(a.c23, i), c33i = ld<T>(a.c33, i);
    T maxv = 0;

    if constexpr (std::is_same_v<P, Fp64Tag>) {
        auto t = cf.target(i);
        const KTab<Smooth> tabX{a.w64};
        const double* hInv3 = a.hInv64 + a.n;
        const double* hInvDx = a.hInv64 + 2 * a.n;
        T hiInv3 = hInv3[i], hiInvDx = hInvDx[i], twoH = 2.0 * hi;
        const bool wrap = cf.needsWrap(t, twoH);
        T mx = 0, my = 0, mz = 0, en = 0;
        long long maxvBits = 0;
        for (unsigned k = 0; k < nc; ++k) {
            uint32_t j = lv.at(ii, k);
            T rx, ry, rz;
            cf.diffFast(t, j, twoH, wrap, rx, ry, rz);
            T r2 = dist2(rx, ry, rz);
            T rinv = invDist(r2);
            T dist = r2 * rinv;
            T vxij = vxi - ld<T>(a.vx, j), vyij = vyi - ld<T>(a.vy, j), vzij = vzi - ld<T>(a.vz, j);
            T rv = rx * vxij + ry * vyij + rz * vzij;
            T Wi = hiInv3 * lookupX(tabX, dist * hiInvDx);
            T Wj = __ldg(hInv3 + j) * lookupX(tabX, dist * __ldg(hInvDx + j));
            T a1i = c11i * rx + c12i * ry + c13i * rz;
            T a2i = c12i * rx + c22i * ry + c23i * rz;
            T a3i = c13i * rx + c23i * ry + c33i * rz;
            T c11j = ld<T>(a.c11, j), c12j = ld<T>(a.c12, j), c13j = ld<T>(a.c13, j);
            T c22j = ld<T>(a.c22, j), c23j = ld<T>(a.c23, j), c33j = ld<T>(a.c33, j);
            T a1j = c11j * rx + c12j * ry + c13j * rz;
            T a2j = c12j * rx + c22j * ry + c23j * rz;
            T a3j = c13j * rx + c23j * ry + c33j * rz;
            T cj = ld<T>(a.c, j);
            T wij = rv * rinv;
            T visc = T(0.5) * artificialViscosity<T>(1.0, 1.0, ci, cj, wij);
            maxvBits = maxBitsNonNeg(maxvBits, ci + cj - T(3) * wij);
            T mj = ld<T>(a.m, j);
            T mjrojWj = __ldg(auxMoR + j) * Wj;
            T mjproi = mj * proi2;
            {
                T aa = Wi * (mjproi + visc * mi_roi);
                T bb = mjrojWj * (__ldg(auxPoR + j) + visc);
                mx += aa * a1i + bb * a1j;
                my += aa * a2i + bb * a2j;
                mz += aa * a3i + bb * a3j;
            }
            {
                T aa = Wi * (T(2) * mjproi + visc * mi_roi);
                T bb = visc * mjrojWj;
                en += vxij * (aa * a1i + bb * a1j) + vyij * (aa * a2i + bb * a2j) + vzij * (aa * a3i + bb * a3j);
            }
        }
        if (valid) {
            a.du[i] = -a.K * 0.5 * en;
            st<T>(a.ax, i, a.K * mx);
            st<T>(a.ay, i, a.K * my);
            st<T>(a.az, i, a.K * mz);
            dt = courantDt(__longlong_as_double(maxvBits), hi, ci, a.Kcour);
        }
    } else {
        auto t = cm.target(i);
        const float4* tab2 = reinterpret_cast<const float4*>(a.wh);
        T hiInv = t.hInv, hiInv3 = hiInv * hiInv * hiInv;
        KSum mx, my, mz, en;
        // the list entry two pairs ahead and the next neighbour's blocks are loaded while the current
        // pair is evaluated
        uint32_t jn = nc > 0 ? lv.at(ii, 0) : uint32_t(i);
        uint32_t jnn = nc > 1 ? lv.at(ii, 1) : uint32_t(i);
        Rec8 n0 = ldRec8(a.pack + 3 * int64_t(jn)), n1 = ldRec8(a.pack + 3 * int64_t(jn) + 1);
        float4 n2 = __ldg(reinterpret_cast<const float4*>(a.pack + 3 * int64_t(jn) + 2));
        for (unsigned k = 0; k < nc; ++k) {
            const Rec8 b0 = n0;    // cell xl yl zl 1/h vx vy
            const Rec8 b1 = n1;    // vz c c11 c12 c13 c22 c23 c33
            const float4 b2 = n2;  // m m/rho p/rho
            if (k + 1 < nc) {
                jn = jnn;
                if (k + 2 < nc) jnn = lv.at(ii, k + 2);
                n0 = ldRec8(a.pack + 3 * int64_t(jn));
                n1 = ldRec8(a.pack + 3 * int64_t(jn) + 1);
                n2 = __ldg(reinterpret_cast<const float4*>(a.pack + 3 * int64_t(jn) + 2));
            }
            T rx, ry, rz;
            cm.diffBlock<true>(t, b0, rx, ry, rz);
            const T hjInv = b0.v[5];
            T r2 = fmaf(rx, rx, fmaf(ry, ry, rz * rz));
            T rinv = rsqrtf(r2);
            T dist = r2 * rinv;
            T vxij = vxi - b0.v[6], vyij = vyi - b0.v[7], vzij = vzi - b1.v[0];
            T v1 = dist * hiInv, v2 = dist * hjInv;
            T rv = rx * vxij + ry * vyij + rz * vzij;
            T Wi = hiInv3 * lookupH32(tab2, v1);
            T Wj = (hjInv * hjInv * hjInv) * lookupH32(tab2, v2);
            T a1i = c11i * rx + c12i * ry + c13i * rz;
            T a2i = c12i * rx + c22i * ry + c23i * rz;
            T a3i = c13i * rx + c23i * ry + c33i * rz;
            T c11j = b1.v[2], c12j = b1.v[3], c13j = b1.v[4];
            T c22j = b1.v[5], c23j = b1.v[6], c33j = b1.v[7];
            // sums of two products written out: which product is fused is part of the result
            T a1j = fmaf(c13j, rz, fmaf(c11j, rx, c12j * ry));
            T a2j = fmaf(c23j, rz, fmaf(c12j, rx, c22j * ry));
            T a3j = fmaf(c33j, rz, fmaf(c13j, rx, c23j * ry));
            T cj = b1.v[1];
            T wij = rv * rinv;
            T visc = T(0.5) * artificialViscosity<T>(1.f, 1.f, ci, cj, wij);
            T vsig = ci + cj - T(3) * wij;
            maxv = (vsig > maxv) ? vsig : maxv;
            T mj = b2.x;
            T mjrojWj = b2.y * Wj;
            T mjproi = mj * proi2;
            T aa = Wi * fmaf(visc, mi_roi, mjproi);
            T bb = mjrojWj * (b2.z + visc);
            mx.add(fmaf(aa, a1i, bb * a1j));
            my.add(fmaf(aa, a2i, bb * a2j));
            mz.add(fmaf(aa, a3i, bb * a3j));
            T ae = Wi * fmaf(visc, mi_roi, T(2) * mjproi);
            T be = visc * mjrojWj;
            en.add(fmaf(vzij, fmaf(be, a3j, ae * a3i),
                        fmaf(vxij, fmaf(be, a1j, ae * a1i), vyij * fmaf(be, a2j, ae * a2i))));
        }
        if (valid) {
            a.du[i] = -a.K * 0.5 * en.value64();
            st<T>(a.ax, i, float(a.K * mx.value64()));
            st<T>(a.ay, i, float(a.K * my.value64()));
            st<T>(a.az, i, float(a.K * mz.value64()));
            dt = courantDt(double(maxv), double(hi), double(ci), a.Kcour);
        }
    }
    if (a.minDt) blockMinDt(dt, a.minDt);
}

// neighbour-side fields of the pair-once momentum-energy pass in three 32-byte loads: A = h^-3 c_ab (six
// entries), c, m, q = p / rho^2 and s = m / rho
__global__ void meStdRec64Kernel(int64_t n, MeStdArgs a, Rec4d* __restrict__ rec)
{
    const int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (j >= n) return;
    const double f = a.hInv64[n + j], rho = ld<double>(a.rho, j), m = ld<double>(a.m, j);
    rec[3 * j] = {f * ld<double>(a.c11, j), f * ld<double>(a.c12, j), f * ld<double>(a.c13, j), f * ld<double>(a.c22, j)};
    rec[3 * j + 1] = {f * ld<double>(a.c23, j), f * ld<double>(a.c33, j), ld<double>(a.c, j), m};
    rec[3 * j + 2] = {ld<double>(a.p, j) / (rho * rho), m / rho, 0.0, 0.0};
}

// FP64 std momentum-energy with one evaluation per mutual pair over the owned lists.  With W A r = w A r
// at each end (A = h^-3 c) and t = visc s, i's directed term of momentum_energy_kern.hpp:60-134 is
// V_i = w_i (m_j q_i + t_i) A_i r + w_j (m_j q_j + t_j) A_j r, since m_j / rho_j (p_j / rho_j) = m_j q_j;
// j's is -V_j with m_i in place of m_j (the same where the masses are equal).  Energy: 2 m_j q_i w_i s_i +
// Q with s = v_ij . A r and Q = t_i w_i s_i + t_j w_j s_j; j's is 2 m_i q_j w_j s_j + Q.  Bound by the
// FP64 pipe: 1M particles 15.3 ms with every directed pair evaluated, now 5.3 ms and 0.6 for the gather of
// the records (IAD 5.7 -> 1.3 + 0.9, density 3.5 -> 2.6 + 0.2, which also fills the geometry cache; the inbox
// 1.2 ms once per neighbour search).  With atomics in place of the records the sweep took 12.5 ms and its bits
// differed from run to run; with them 14.5.
// Geo: arrays of the pair-geometry cache (5, 2), or 0 to form the geometry here.
template<bool Smooth, int Geo>
__device__ __forceinline__ void meStdOnceBody(ListView lv, OwnedView ov, CoordFp64 cf, MeStdArgs a,
                                                              const Rec4d* __restrict__ rec, PairRec pr,
                                              long long* __restrict__ accS, PairGeo geo)
{
    using T = double;
    const int64_t i = lv.first + blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    if (i >= lv.last) return;
    const int64_t ii = i - lv.first, n = a.n;
    const unsigned no = ov.size(ii);
    const KTab<Smooth> tabX{a.w64};
    const double* hInvDx = a.hInv64 + 2 * n;
    const T *vxA = static_cast<const T*>(a.vx), *vyA = static_cast<const T*>(a.vy), *vzA = static_cast<const T*>(a.vz);
    const Rec4d i0 = rec[3 * i], i1 = rec[3 * i + 1], i2 = rec[3 * i + 2];
    const T mi = i1.v[3];
    typename CoordFp64::Target t{};
    T vxi = 0, vyi = 0, vzi = 0, twoH = 0, hiInvDx = 0;
    CoordFp64::Fold fold{};
    int64_t g = 0;
    if constexpr (Geo != 0) g = geo.base(ii) + 32 * blockIdx.y;
    if constexpr (Geo != 5) {
        t = cf.target(i);
        twoH = 2.0 * ld<T>(a.h, i);
        fold = cf.fold(t, twoH);
        vxi = vxA[i], vyi = vyA[i], vzi = vzA[i];
        hiInvDx = hInvDx[i];
    }
    T mx = 0, my = 0, mz = 0, en = 0;
    long long maxvBits = 0;
    const int64_t rb = pr.base(ii);
    for (unsigned k = blockIdx.y; k < no; k += gridDim.y, g += 32 * gridDim.y) {
        bool mutual;
        const uint32_t j = ov.at(ii, k, mutual);
        const Rec4d j0 = ldRec4d(rec + 3 * int64_t(j)), j1 = ldRec4d(rec + 3 * int64_t(j) + 1),
                    j2 = ldRec4d(rec + 3 * int64_t(j) + 2);
        T rx, ry, rz, wij, vxij, vyij, vzij;
        double2 wv;
        if constexpr (Geo != 0) {
            wij = __ldg(geo.g + g).y;
            wv = __ldg(geo.w + g);
        }
        if constexpr (Geo == 5) {  // v_ij = v_i - v_j = -dv exactly
            const double2 a0 = __ldg(geo.x + g), a1 = __ldg(geo.x + geo.plane + g), a2 = __ldg(geo.x + 2 * geo.plane + g);
            rx = a0.x, ry = a0.y, rz = a1.x;
            vxij = -a1.y, vyij = -a2.x, vzij = -a2.y;
        } else {
            cf.diffOwned(t, j, mutual, fold, rx, ry, rz);
            vxij = vxi - vxA[j], vyij = vyi - vyA[j], vzij = vzi - vzA[j];
        }
        if constexpr (Geo == 0) {
            const T r2 = dist2(rx, ry, rz);
            const T rinv = invDist(r2), dist = r2 * rinv;
            wij = fma(rz, vzij, fma(ry, vyij, rx * vxij)) * rinv;
            wv.x = lookupX(tabX, dist * hiInvDx);
            wv.y = lookupX(tabX, dist * __ldg(hInvDx + j));
        }
        // sums of products written out: every form of the cache gives the same bits
        const T gix = fma(i0.v[2], rz, fma(i0.v[1], ry, i0.v[0] * rx));
        const T giy = fma(i1.v[0], rz, fma(i0.v[3], ry, i0.v[1] * rx));
        const T giz = fma(i1.v[1], rz, fma(i1.v[0], ry, i0.v[2] * rx));
        const T gjx = fma(j0.v[2], rz, fma(j0.v[1], ry, j0.v[0] * rx));
        const T gjy = fma(j1.v[0], rz, fma(j0.v[3], ry, j0.v[1] * rx));
        const T gjz = fma(j1.v[1], rz, fma(j1.v[0], ry, j0.v[2] * rx));
        const T cs = i1.v[2] + j1.v[2], mj = j1.v[3];
        const T vsig = fma(T(-3), wij, cs);
        maxvBits = maxBitsNonNeg(maxvBits, vsig);
        const T wsi = wv.x * fma(vzij, giz, fma(vyij, giy, vxij * gix));
        const T wsj = wv.y * fma(vzij, gjz, fma(vyij, gjy, vxij * gjx));
        T visc = 0;  // its products are formed for receding pairs too: 0 times an undefined density is NaN, as in
                     // the reference
        if (negative(wij)) visc = fma(T(0.25), cs, -wij) * -wij;  // half of artificial_viscosity(1, 1, ...)
        const T ti = i2.v[1] * visc, tj = j2.v[1] * visc, Q = fma(ti, wsi, tj * wsj);
        T Pi = wv.x * fma(mj, i2.v[0], ti), Pj = wv.y * fma(mj, j2.v[0], tj);
        T Vx = fma(Pi, gix, Pj * gjx), Vy = fma(Pi, giy, Pj * gjy), Vz = fma(Pi, giz, Pj * gjz);
        mx += Vx;
        my += Vy;
        mz += Vz;
        en += fma(mj * (2.0 * i2.v[0]), wsi, Q);
        if (mutual) {
            if (__double_as_longlong(mi) != __double_as_longlong(mj)) {
                Pi = wv.x * fma(mi, i2.v[0], ti), Pj = wv.y * fma(mi, j2.v[0], tj);
                Vx = fma(Pi, gix, Pj * gjx), Vy = fma(Pi, giy, Pj * gjy), Vz = fma(Pi, giz, Pj * gjz);
            }
            pr.rec[rb + 32 * int64_t(k)] = {-Vx, -Vy, -Vz, fma(mi * (2.0 * j2.v[0]), wsj, Q)};
            atomicMax(accS + j, __double_as_longlong(vsig));
        }
    }
    double* part = pr.part + blockIdx.y * int64_t(4) * n + i;
    part[0] = mx;
    part[n] = my;
    part[2 * n] = mz;
    part[3 * n] = en;
    atomicMax(accS + i, maxvBits);
}

template<bool Smooth, int Geo>
__global__ void __launch_bounds__(kPairBlock) meStdOnceKernel(ListView lv, OwnedView ov, CoordFp64 cf, MeStdArgs a,
                                                              const Rec4d* __restrict__ rec, PairRec pr,
                                                              long long* __restrict__ accS, PairGeo geo)
{
    if constexpr (Geo >= 0) meStdOnceBody<Smooth, Geo>(lv, ov, cf, a, rec, pr, accS, geo);
    else if (*geo.stale) meStdOnceBody<Smooth, 0>(lv, ov, cf, a, rec, pr, accS, geo);
    else meStdOnceBody<Smooth, -Geo>(lv, ov, cf, a, rec, pr, accS, geo);
}

__global__ void __launch_bounds__(kPairBlock) meStdOnceFinish(MeStdArgs a, const double* __restrict__ acc)
{
    const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
    double dt = INFINITY;
    if (i < a.n) {
        a.du[i] = -a.K * 0.5 * acc[3 * a.n + i];
        st<double>(a.ax, i, a.K * acc[i]);
        st<double>(a.ay, i, a.K * acc[a.n + i]);
        st<double>(a.az, i, a.K * acc[2 * a.n + i]);
        const long long mb = reinterpret_cast<const long long*>(acc + 4 * a.n)[i];
        dt = courantDt(__longlong_as_double(mb), ld<double>(a.h, i), ld<double>(a.c, i), a.Kcour);
    }
    if (a.minDt) blockMinDt(dt, a.minDt);
}

template<class P>
int launchXmass(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last, void* out, bool storeRho)
{
    SPHGB_TRY(checkPass(c, p, first, last));
    ListView lv = listView(c);
    lv.first = first;
    lv.last = last;
    CoordFp64 cf = coordFp64(c, p);
    CoordMixed cm = coordMixed(c);
    const void* wh = std::is_same_v<P, Fp64Tag> ? c->whx64.p : c->whH32.p;
    unsigned blocks = gridFor(last - first, kPairBlock);
    bool once = std::is_same_v<P, Fp64Tag> && pairOnce(c, p, first, last);
    const bool exact = once && !storeRho && exactSums(p->n);
    const int slices = int(ownedGrid(p->n).y);
    PairRec pr{};
    if (once) {  // sums, then their rounding errors or the own partial sums
        const size_t doubles = size_t(storeRho ? 1 + slices : exact ? 2 : 1) * size_t(p->n);
        SPHGB_TRY(c->pairAcc.ensure(sizeof(double) * doubles));
        if (storeRho) {
            SPHGB_TRY(pairRecords(c, c->pairAcc.as<double>() + p->n, &pr));
            once = pr.rec != nullptr;
        } else
            SPHGB_CUDA(cudaMemsetAsync(c->pairAcc.p, 0, sizeof(double) * doubles, c->stream));
    }
    if (once) {
        const int64_t n = p->n;
        const double* lo = exact ? c->pairAcc.as<double>() + n : nullptr;
        PairGeo geo{};
        SPHGB_TRY(pairGeoStore(c, p, &geo));
        double* snap = geo.g && !c->inSweep ? c->geoSnap.as<double>() : nullptr;
        SPHGB_TRY(withKernelForm(c, [&](auto smooth) {
            constexpr bool S = decltype(smooth)::value;
            auto run = [&](auto kernel) {
                kernel<<<ownedGrid(n), kPairBlock, 0, c->stream>>>(
                lv, ownedView(c), cf, static_cast<const double*>(p->h), static_cast<const double*>(p->m),
                KTab<S>{tabW64(c)}, c->hInv64.as<double>() + 2 * n, c->pairAcc.as<double>(), geo,
                static_cast<const double*>(p->vx), static_cast<const double*>(p->vy),
                static_cast<const double*>(p->vz), n, pr);
            };
            if (storeRho) run(xmassOnceKernel<S, kXmassRecords>);
            else if (exact) run(xmassOnceKernel<S, kXmassExact>);
            else run(xmassOnceKernel<S, kXmassSum>);
            return launched(c, "xmassOnceKernel");
        }));
        if (storeRho) SPHGB_TRY(gatherRecords(c, pr, n, 1, slices, c->pairAcc.as<double>()));
        const unsigned eb = gridFor(last - first, 256);
        if (storeRho)
            xmassOnceFinish<true><<<eb, 256, 0, c->stream>>>(first, last, static_cast<const double*>(p->h),
                                                              static_cast<const double*>(p->m), c->K,
                                                              c->pairAcc.as<double>(), lo, static_cast<double*>(out),
                                                              geoInputs(p), snap, n);
        else
            xmassOnceFinish<false><<<eb, 256, 0, c->stream>>>(first, last, static_cast<const double*>(p->h),
                                                               static_cast<const double*>(p->m), c->K,
                                                               c->pairAcc.as<double>(), lo, static_cast<double*>(out),
                                                               geoInputs(p), snap, n);
        return launched(c, "xmassOnceFinish");
    }
    const Rec8* rec = nullptr;
    if constexpr (std::is_same_v<P, MixedTag>) {
        SPHGB_TRY(c->pack.ensure(sizeof(Rec8) * 3 * size_t(p->n)));  // the ME blocks' space, free here
        packXmassKernel<<<gridFor(p->n, 256), 256, 0, c->stream>>>(p->n, p->m, c->gridKey.as<u64>(),
                                                                    c->gridLoc.as<float4>(), c->pack.as<float4>());
        SPHGB_TRY(launched(c, "packXmassKernel"));
        rec = c->pack.as<Rec8>();
    }
    return withKernelForm(c, [&](auto smooth) {
        constexpr bool S = std::is_same_v<P, Fp64Tag> && decltype(smooth)::value;
        if (storeRho)
            xmassKernel<P, true, S><<<blocks, kPairBlock, 0, c->stream>>>(lv, cf, cm, p->h, p->m, wh, tabW64(c),
                                                                           c->K, out, rec);
        else
            xmassKernel<P, false, S><<<blocks, kPairBlock, 0, c->stream>>>(lv, cf, cm, p->h, p->m, wh, tabW64(c),
                                                                            c->K, out, rec);
        return launched(c, "xmassKernel");
    });
}

template<class P>
int launchIad(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last)
{
    const Rec8* rec = nullptr;
    if constexpr (std::is_same_v<P, MixedTag>) {
        SPHGB_TRY(c->pack.ensure(sizeof(Rec8) * 3 * size_t(p->n)));  // the ME blocks' space, free here
        packIadStdKernel<<<gridFor(p->n, 256), 256, 0, c->stream>>>(p->n, p->m, p->rho, c->gridKey.as<u64>(),
                                                                    c->gridLoc.as<float4>(), c->pack.as<float4>());
        SPHGB_TRY(launched(c, "packIadStdKernel"));
        rec = c->pack.as<Rec8>();
    } else SPHGB_TRY(launchStdAux(c, p, false));
    ListView lv = listView(c);
    lv.first = first;
    lv.last = last;
    const void* wh = std::is_same_v<P, Fp64Tag> ? c->whx64.p : c->whH32.p;
    PairRec pr{};
    const int slices = int(ownedGrid(p->n).y);
    if (std::is_same_v<P, Fp64Tag> && pairOnce(c, p, first, last)) {
        SPHGB_TRY(c->pairAcc.ensure(sizeof(double) * 6 * size_t(1 + slices) * size_t(p->n)));
        SPHGB_TRY(pairRecords(c, c->pairAcc.as<double>() + 6 * p->n, &pr));
    }
    if (pr.rec) {
        const int64_t n = p->n;
        const PairGeo geo = pairGeoRead(c);
        const double* h = static_cast<const double*>(p->h);
        SPHGB_TRY(withKernelForm(c, [&](auto smooth) {
            constexpr bool S = decltype(smooth)::value;
            auto run = [&](auto kernel) {
                kernel<<<ownedGrid(n), kPairBlock, 0, c->stream>>>(
                    lv, ownedView(c), coordFp64(c, p), h, c->aux.as<double>(), KTab<S>{tabW64(c)},
                    c->hInv64.as<double>(), n, pr, geo);
            };
            withPairGeo(geo, [&](auto g) { run(iadStdOnceKernel<S, decltype(g)::value>); });
            return launched(c, "iadStdOnceKernel");
        }));
        SPHGB_TRY(gatherRecords(c, pr, n, 6, slices, c->pairAcc.as<double>()));
        iadStdOnceFinish<<<gridFor(n, 256), 256, 0, c->stream>>>(n, h, c->K, c->pairAcc.as<double>(),
                                                                 IadOut{p->c11, p->c12, p->c13, p->c22, p->c23, p->c33});
        return launched(c, "iadStdOnceFinish");
    }
    return withKernelForm(c, [&](auto smooth) {
        constexpr bool S = std::is_same_v<P, Fp64Tag> && decltype(smooth)::value;
        iadKernel<P, S><<<gridFor(last - first, kPairBlock), kPairBlock, 0, c->stream>>>(
            lv, coordFp64(c, p), coordMixed(c), p->h, c->aux.p, wh, tabW64(c), c->K,
            IadOut{p->c11, p->c12, p->c13, p->c22, p->c23, p->c33}, rec);
        return launched(c, "iadKernel");
    });
}

template<class P>
int launchMeStd(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last, double* minDt)
{
    unsigned long long* minDtWord = nullptr;
    SPHGB_TRY(beginDtReduction(c, &minDtWord));
    PairRec pr{};
    const int slices = int(ownedGrid(p->n).y);
    if (std::is_same_v<P, Fp64Tag> && pairOnce(c, p, first, last)) {
        const size_t n = size_t(p->n);  // four sums and the signal velocity, then the own partial sums
        SPHGB_TRY(c->pack.ensure(sizeof(Rec4d) * 3 * n));
        SPHGB_TRY(c->pairAcc.ensure(sizeof(double) * (5 + 4 * size_t(slices)) * n));
        SPHGB_TRY(pairRecords(c, c->pairAcc.as<double>() + 5 * n, &pr));
    }
    const bool once = pr.rec != nullptr;
    if (std::is_same_v<P, Fp64Tag> && !once) SPHGB_TRY(launchStdAux(c, p, true));
    if (std::is_same_v<P, MixedTag>) SPHGB_TRY(c->aux.ensure(sizeof(float) * 3 * size_t(p->n)));
    ListView lv = listView(c);
    lv.first = first;
    lv.last = last;
    MeStdArgs a{};
    a.vx = p->vx;
    a.vy = p->vy;
    a.vz = p->vz;
    a.h = p->h;
    a.m = p->m;
    a.rho = p->rho;
    a.p = p->p;
    a.c = p->c;
    a.c11 = p->c11;
    a.c12 = p->c12;
    a.c13 = p->c13;
    a.c22 = p->c22;
    a.c23 = p->c23;
    a.c33 = p->c33;
    a.wh = std::is_same_v<P, Fp64Tag> ? c->whx64.p : c->whH32.p;
    a.w64 = tabW64(c);
    a.hInv64 = c->hInv64.as<double>();
    a.aux = c->aux.p;
    a.n = p->n;
    a.K = c->K;
    a.Kcour = float(c->prm.Kcour);
    a.ax = p->ax;
    a.ay = p->ay;
    a.az = p->az;
    a.du = p->du;
    a.minDt = minDtWord;
    if (once) {
        const int64_t n = p->n;
        long long* accS = c->pairAcc.as<long long>() + 4 * n;
        SPHGB_CUDA(cudaMemsetAsync(accS, 0, sizeof(long long) * size_t(n), c->stream));
        meStdRec64Kernel<<<gridFor(n, 256), 256, 0, c->stream>>>(n, a, c->pack.as<Rec4d>());
        SPHGB_TRY(launched(c, "meStdRec64Kernel"));
        const PairGeo geo = pairGeoRead(c);
        const unsigned blocks = gridFor(n, kPairBlock);
        SPHGB_TRY(withKernelForm(c, [&](auto smooth) {
            constexpr bool S = decltype(smooth)::value;
            auto run = [&](auto kernel) {
                kernel<<<ownedGrid(n), kPairBlock, 0, c->stream>>>(lv, ownedView(c), coordFp64(c, p), a, c->pack.as<Rec4d>(),
                                                             pr, accS, geo);
            };
            withPairGeo(geo, [&](auto g) { run(meStdOnceKernel<S, decltype(g)::value>); });
            return launched(c, "meStdOnceKernel");
        }));
        SPHGB_TRY(gatherRecords(c, pr, n, 4, slices, c->pairAcc.as<double>()));
        meStdOnceFinish<<<blocks, kPairBlock, 0, c->stream>>>(a, c->pairAcc.as<double>());
        SPHGB_TRY(launched(c, "meStdOnceFinish"));
        return endDtReduction(c, a.minDt, minDt);
    }
    if constexpr (std::is_same_v<P, MixedTag>) {
        SPHGB_TRY(c->pack.ensure(sizeof(Rec8) * 3 * size_t(p->n)));
        meStdPackKernel<<<gridFor(p->n, 256), 256, 0, c->stream>>>(p->n, a, c->gridKey.as<u64>(), c->gridLoc.as<float4>(),
                                                                   c->aux.as<float>(), c->pack.as<float4>());
        SPHGB_TRY(launched(c, "meStdPackKernel"));
        a.pack = c->pack.as<Rec8>();
    }
    SPHGB_TRY(withKernelForm(c, [&](auto smooth) {
        constexpr bool S = std::is_same_v<P, Fp64Tag> && decltype(smooth)::value;
        meStdKernel<P, S><<<gridFor(last - first, kPairBlock), kPairBlock, 0, c->stream>>>(lv, coordFp64(c, p),
                                                                                            coordMixed(c), a);
        return launched(c, "meStdKernel");
    }));
    return endDtReduction(c, a.minDt, minDt);
}

}  // namespace

int passDensity(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last)
{
    if (!p->rho || !p->m || !p->h) return SPHGB_ERR_ARG;
    if (p->precision == SPHGB_MIXED) return launchXmass<MixedTag>(c, p, first, last, p->rho, true);
    return launchXmass<Fp64Tag>(c, p, first, last, p->rho, true);
}

int passXMass(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last)
{
    if (!p->xm || !p->m || !p->h) return SPHGB_ERR_ARG;
    if (p->precision == SPHGB_MIXED) return launchXmass<MixedTag>(c, p, first, last, p->xm, false);
    return launchXmass<Fp64Tag>(c, p, first, last, p->xm, false);
}

int passEosStd(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last)
{
    if (!p->u || !p->rho || !p->p || !p->c || first < 0 || last > p->n || first >= last) return SPHGB_ERR_ARG;
    unsigned blocks = gridFor(last - first, 256);
    if (p->precision == SPHGB_MIXED)
        eosStdKernel<MixedTag><<<blocks, 256, 0, c->stream>>>(first, last, p->u, p->rho, c->prm.gamma, p->p, p->c);
    else
        eosStdKernel<Fp64Tag><<<blocks, 256, 0, c->stream>>>(first, last, p->u, p->rho, c->prm.gamma, p->p, p->c);
    return launched(c, "eosStdKernel");
}

int passIadStd(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last)
{
    if (!p->m || !p->rho || !p->c11 || !p->c12 || !p->c13 || !p->c22 || !p->c23 || !p->c33) return SPHGB_ERR_ARG;
    SPHGB_TRY(checkPass(c, p, first, last));
    if (p->precision == SPHGB_MIXED) return launchIad<MixedTag>(c, p, first, last);
    return launchIad<Fp64Tag>(c, p, first, last);
}

int passMomentumEnergyStd(sphgb_ctx* c, sphgb_particles* p, int64_t first, int64_t last, double* minDt)
{
    if (!p->vx || !p->vy || !p->vz || !p->rho || !p->p || !p->c || !p->ax || !p->ay || !p->az || !p->du ||
        !p->c11 || !p->m)
        return SPHGB_ERR_ARG;
    SPHGB_TRY(checkPass(c, p, first, last));
    if (p->precision == SPHGB_MIXED) return launchMeStd<MixedTag>(c, p, first, last, minDt);
    return launchMeStd<Fp64Tag>(c, p, first, last, minDt);
}

}  // namespace sphgb
