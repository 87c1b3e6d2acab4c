// The grid-point step of gridpointa (plasim.f90:2441-2455): the kernel,
// shared by gridpoint.cu (FP32) and gridpoint_fp64.cu (FP64, compiled
// without FMA contraction so that every product and sum is rounded as the
// reference's 8-byte build rounds it).
#pragma once
#include "exotx_internal.cuh"

namespace exotx {

constexpr int GP_THREADS = 128;

template <typename T>
struct GpArgs {
    const T *gin;
    T *gout, *dw;
    const double *sid;      // per latitude (rcsq = 1/(1 - sid^2))
    const double *k;        // constants block
    const T *dq;            // nqspec == 0: grid humidity [inst][L][nhor]
    long long ncol;         // instances x nhor
    int L, nhor, nlon, nqspec;
    int g_lower;            // g(i, k) = 0 for every i < k
    double akap, rdbrv, adv, psurf, ww;
};

// the constants block in the step's precision: in shared memory (SK, staged
// once per block) or read from global memory and rounded at each use
template <typename T, bool SK>
struct GpConsts {
    const T *s;
    const double *g;
    __device__ __forceinline__ T operator()(int i) const {
        if constexpr (SK) return s[i];
        else return (T)g[i];
    }
};
template <typename T>
__host__ __device__ inline size_t gp_smem(int L, bool sk) {
    return sizeof(T) * (3 * (size_t)L * GP_THREADS + (sk ? 6 * (size_t)L + 2 * (size_t)L * L : 0));
}

// Any level count and any g: the profiles in shared memory.  LC > 0: the level
// count fixed at compile time, so the index arithmetic of the profiles and
// constants folds (the arithmetic, and its order, is the same).
template <typename T, bool SK, int LC>
__global__ void __launch_bounds__(GP_THREADS) k_gridpoint(const GpArgs<T> A) {
    extern __shared__ __align__(16) unsigned char gsm[];
    T *sv = reinterpret_cast<T *>(gsm);                 // zvgpg      [L][GP_THREADS]
    T *sb = sv + (size_t)A.L * GP_THREADS;              // zvgpg + gd [L][GP_THREADS]
    T *s1 = sb + (size_t)A.L * GP_THREADS;              // ztv1 - gt  [L][GP_THREADS]
    T *sk = s1 + (size_t)A.L * GP_THREADS;              // constants (SK)
    if constexpr (SK) {
        for (int i = threadIdx.x; i < 6 * A.L + 2 * A.L * A.L; i += GP_THREADS) sk[i] = (T)A.k[i];
        __syncthreads();
    }
    const GpConsts<T, SK> K{sk, A.k};
    const long long col = blockIdx.x * (long long)GP_THREADS + threadIdx.x;
    if (col >= A.ncol) return;
    const int L = LC > 0 ? LC : A.L, tx = threadIdx.x;
    const long long inst = col / A.nhor;
    const int h = (int)(col - inst * A.nhor);
    const size_t n = (size_t)A.nhor;
    const T *gin = A.gin + (size_t)inst * (6 * L + 3) * n;
    T *gout = A.gout + (size_t)inst * (9 * L + 1) * n;
#define IN(f, k) gin[((size_t)(f) * L + (k)) * n + h]
#define OUT(f, k) gout[((size_t)(f) * L + (k)) * n + h]
#define SH(a, k) a[(size_t)(k) * GP_THREADS + tx]
    const T gpj = gin[(size_t)6 * L * n + h], gpm = gin[((size_t)6 * L + 1) * n + h];
    const T gp = exp(gin[((size_t)6 * L + 2) * n + h]);   // gp = exp(gp), plasim.f90:2441
    const double s = A.sid[h / A.nlon];
    const T rc = (T)(1.0 / (1.0 - s * s));
    const T rdbrv1 = (T)1. / (T)A.rdbrv - (T)1.;
    // pass 1: profiles and the column totals of the divergence and of zvgpg
    T zsumd = 0, gvp = 0;
    for (int k = 0; k < L; k++) {
        const T gu = IN(0, k), gv = IN(1, k), gt = IN(2, k), gd = IN(3, k), gq = IN(5, k);
        const T zv = rc * (gu * gpm + gv * gpj);
        T zq;
        if (A.nqspec == 1) zq = fmax(gq / gp, (T)0.);
        else zq = A.dq ? fmax(A.dq[((size_t)inst * L + k) * n + h], (T)0.) : (T)0.;
        const T tv1 = (gt + K(3 * L + k)) * ((T)1. + rdbrv1 * zq) - K(3 * L + k);
        SH(sv, k) = zv;
        SH(sb, k) = zv + gd;
        SH(s1, k) = tv1 - gt;
        if (k == 0) { zsumd = K(0) * gd; gvp = K(0) * zv; }
        else { zsumd = zsumd + K(k) * gd; gvp = gvp + K(k) * zv; }
    }
    const T tot = zsumd + gvp;
    // pass 2, level by level: sigma-dot, vertical advection terms and tendencies
    T psd = 0, psv = 0;                 // running sums of dsigma * gd and of dsigma * zvgpg
    T gtd_m = 0, gqm_m = 0, gud_m = 0, gvd_m = 0;   // the level above's products
    T zs = 0;                           // zsumd of the tendency loop (plasim.f90:2661, :2692)
    // the next level's fields are loaded one iteration ahead (n* = level k + 1)
    T nu = IN(0, 0), nv = IN(1, 0), nt = IN(2, 0), nd = IN(3, 0), nz = IN(4, 0), nq = IN(5, 0);
    for (int k = 0; k < L; k++) {
        const T gu = nu, gv = nv, gt = nt, gd = nd, gz = nz, gq = nq;
        if (k + 1 < L) {
            nu = IN(0, k + 1); nv = IN(1, k + 1); nt = IN(2, k + 1);
            nd = IN(3, k + 1); nz = IN(4, k + 1); nq = IN(5, k + 1);
        }
        const T zv = SH(sv, k);
        T zq;
        if (A.nqspec == 1) zq = fmax(gq / gp, (T)0.);
        else zq = A.dq ? fmax(A.dq[((size_t)inst * L + k) * n + h], (T)0.) : (T)0.;
        const T tv1 = (gt + K(3 * L + k)) * ((T)1. + rdbrv1 * zq) - K(3 * L + k);
        const T tv2 = (gt + K(3 * L + k)) * ((T)1. + rdbrv1 * zq) / ((T)1. + (T)A.adv * zq) - K(3 * L + k);
        // this level's products of the sigma-dot flux with the layer differences
        T gtd = 0, gqm = 0, gud = 0, gvd = 0;
        if (k < L - 1) {
            if (k == 0) { psd = K(0) * gd; psv = K(0) * zv; }
            else { psd = psd + K(k) * gd; psv = psv + K(k) * zv; }
            const T zsdotp = (K(L + k) * tot - (psd + psv));
            gtd = zsdotp * (nt - gt);
            gqm = zsdotp * (nq + gq);
            gud = zsdotp * (nu - gu);
            gvd = zsdotp * (nv - gv);
        }
        T gtn, gqn, guz, gvz, dwv;
        if (k == 0) {
            zs = zv * K(0);
            gtn = gt * gd - (T)A.akap * tv2 * gd - K(2 * L + 0) * (gtd + K(4 * L + 0) * (K(L + 0) * gvp - zs));
            gqn = -K(2 * L + 0) * gqm;
            guz = -gu * gz - gpj * tv1 - K(2 * L + 0) * gvd;
            gvz = gv * gz - gpm * tv1 - K(2 * L + 0) * gud;
            dwv = gd * gp * (T)A.psurf * (T)A.ww;
        } else {
            T ztpta = K(6 * L + L * L + 0 + L * k) * SH(sv, 0);
            T ztptb = K(6 * L + L * L + 0 + L * k) * SH(sb, 0);
#pragma unroll 4
            for (int j = 1; j <= k; j++) {
                ztpta = ztpta + K(6 * L + L * L + j + L * k) * SH(sv, j);
                ztptb = ztptb + K(6 * L + L * L + j + L * k) * SH(sb, j);
            }
            if (k < L - 1) {
                zs = zs + zv * K(k);
                gtn = gt * gd + (T)A.akap * tv2 * (zv - ztptb) + K(5 * L + k) * (zv - ztpta) -
                      K(2 * L + k) * (gtd + gtd_m + gvp * (K(4 * L + k) * K(L + k) + K(4 * L + k - 1) * K(L + k - 1)) -
                                     zs * (K(4 * L + k - 1) + K(4 * L + k)) + zv * K(k) * K(4 * L + k - 1));
                gqn = -K(2 * L + k) * (gqm - gqm_m);
                guz = -gu * gz - gpj * tv1 - K(2 * L + k) * (gvd + gvd_m);
                gvz = gv * gz - gpm * tv1 - K(2 * L + k) * (gud + gud_m);
            } else {
                gtn = gt * gd + (T)A.akap * tv2 * (zv - ztptb) + K(5 * L + k) * (zv - ztpta) -
                      K(2 * L + k) * (gtd_m + K(4 * L + k - 1) * (K(L + k - 1) * gvp - zs));
                gqn = K(2 * L + k) * gqm_m;
                guz = -gu * gz - gpj * tv1 - K(2 * L + k) * gvd_m;
                gvz = gv * gz - gpm * tv1 - K(2 * L + k) * gud_m;
            }
            dwv = (zv - ztptb) * gp * (T)A.psurf * (T)A.ww;
        }
        // non-linear geopotential, summed over every level as dot_product does;
        // initsi's g is lower triangular (g(i, k) = 0 for i < k), and those
        // exact zero terms leave the partial sum at +0, so they are skipped
        T dot = 0;
        if (A.g_lower) {
#pragma unroll 4
            for (int i = k; i < L; i++) dot = dot + K(6 * L + i + L * k) * SH(s1, i);
        } else {
#pragma unroll 4
            for (int i = 0; i < L; i++) dot = dot + K(6 * L + i + L * k) * SH(s1, i);
        }
        const T gphi = dot * (T)2. / rc;
        T ke = gu * gu + gv * gv;
        ke = ke + gphi;
        OUT(0, k) = gtn;                 // gtn
        OUT(1, k) = gqn;                 // gqn
        OUT(2, k) = gu * gt;             // gut
        OUT(3, k) = gv * gt;             // gvt
        OUT(4, k) = guz;                 // guz
        OUT(5, k) = gvz;                 // gvz
        OUT(6, k) = ke;                  // gke
        gout[((size_t)7 * L + 1 + k) * n + h] = gu * gq;       // guq
        gout[((size_t)8 * L + 1 + k) * n + h] = gv * gq;       // gvq
        if (A.dw) A.dw[((size_t)inst * L + k) * n + h] = dwv;
        gtd_m = gtd; gqm_m = gqm; gud_m = gud; gvd_m = gvd;
    }
    gout[(size_t)7 * L * n + h] = gvp;   // gvpp
#undef IN
#undef OUT
#undef SH
}

// Up to LM levels and initsi's lower triangular g.  A thread copies its column's
// inputs to its own slots of shared memory asynchronously, all at once (nothing
// is shared, so the block never synchronises); the first pass adds each level,
// as it arrives, to the partial vertical sums of every level that holds it, in
// registers, which are independent chains; the second reads the inputs again
// from shared memory.  The constants are in the kernel's parameters.  The general
// form above loads each level when it needs it and waits: T127 L20 x8 FP32
// 285 -> 189 us, x3 FP64 224 -> 160 us; T85 L13 x8 FP32 97 -> 54.  HBM would take
// 110 us for the first (15L + 4 values per column); what is left is instruction
// issue and fetch, so the code is kept short: 32-bit offsets from the block's
// bases, one division where two would do.
template <typename T, int LM>
struct GpLevels {
    T ds[LM], sh[LM], rd[LM], t0[LM], t01[LM], tkp[LM];
    T g[LM * (LM + 1) / 2];   // g(i, k), i >= k, k by k
    T c[LM * (LM + 1) / 2];   // c(j, k), j <= k, k by k
    static __host__ __device__ constexpr int gi(int i, int k) { return k * LM - k * (k - 1) / 2 + i - k; }
    static __host__ __device__ constexpr int ci(int j, int k) { return k * (k + 1) / 2 + j; }
    void fill(const exotx_gp_params &h) {
        const int L = h.nlev;
        for (int k = 0; k < LM; k++) {
            const bool in = k < L;
            ds[k] = in ? (T)h.dsigma[k] : 0; sh[k] = in ? (T)h.sigmah[k] : 0; rd[k] = in ? (T)h.rdsig[k] : 0;
            t0[k] = in ? (T)h.t0[k] : 0; t01[k] = in ? (T)h.t01s2[k] : 0; tkp[k] = in ? (T)h.tkp[k] : 0;
            for (int i = k; i < LM; i++) g[gi(i, k)] = i < L ? (T)h.g[i + L * k] : 0;
            for (int j = 0; j <= k; j++) c[ci(j, k)] = in ? (T)h.c[j + L * k] : 0;
        }
    }
};

constexpr int GP_COLS = 64;   // columns, threads, of a block
template <typename T, int LM>
__host__ __device__ constexpr size_t gp_slots() { return sizeof(T) * (size_t)GP_COLS * (6 * LM + 3); }
// blocks per SM: what the shared memory holds, five at most
template <typename T, int LM>
__host__ __device__ constexpr int gp_blocks() {
    const int b = (int)(227 * 1024 / (gp_slots<T, LM>() + 1024));
    return b > 5 ? 5 : b;
}
// whether the specific humidities are kept between the passes too (else divided out again)
template <typename T>
__host__ __device__ constexpr bool gp_keepq(int LM) { return sizeof(T) == 4 && LM <= 20; }

template <typename T>
__device__ __forceinline__ void gp_copy(T *s, const T *g) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(s)), "l"(g),
                 "n"((int)sizeof(T))
                 : "memory");
}

// x / d from r = 1 / d rounded: one correction by the exact residual gives the
// correctly rounded quotient (Markstein, IBM J. Res. Dev. 34, 1990); where the
// residual is not finite the product stands, as the quotient itself would for a zero
// or infinite operand (1 / d overflows for d below 2^-128, surface pressures of e^-88)
__device__ __forceinline__ float gp_div(float x, float d, float r) {
    const float q = x * r, e = fmaf(-q, d, x);
    return fabsf(e) <= 3.402823466e38f ? fmaf(e, r, q) : q;
}
__device__ __forceinline__ double gp_div(double x, double d, double r) {
    const double q = x * r, e = fma(-q, d, x);
    return fabs(e) <= 1.7976931348623157e308 ? fma(e, r, q) : q;
}

template <typename T, int LM>
__global__ void __launch_bounds__(GP_COLS, gp_blocks<T, LM>())
    k_gridpoint_async(const __grid_constant__ GpArgs<T> A, const __grid_constant__ GpLevels<T, LM> K) {
    extern __shared__ __align__(16) unsigned char gsm[];
    using G = GpLevels<T, LM>;
    constexpr bool KEEPQ = gp_keepq<T>(LM);
    constexpr int NG = 4, GL = (LM + NG - 1) / NG;           // the copies in NG groups of GL levels
    T *sl = reinterpret_cast<T *>(gsm) + threadIdx.x;        // slot i at sl[i * GP_COLS]
    // the instance is the block's; a thread adds a 32-bit offset to its bases
    const int nb = (A.nhor + GP_COLS - 1) / GP_COLS, inst = blockIdx.x / nb;
    const int h = (blockIdx.x - inst * nb) * GP_COLS + threadIdx.x, L = A.L;
    if (h >= A.nhor) return;
    const uint32_t lev = (uint32_t)A.nhor * sizeof(T), off0 = h * sizeof(T);   // stride of a level; this column
    const size_t f = (size_t)L * lev;                        // stride of a field
    const char *in = (const char *)A.gin + (size_t)inst * (6 * f + 3 * lev);
    const auto at = [](const char *base, uint32_t o) { return reinterpret_cast<const T *>(base + o); };
#define SL(x, k) sl[(6 * (k) + (x)) * GP_COLS]
    for (int i = 0; i < 3; i++) gp_copy(sl + (6 * LM + i) * GP_COLS, at(in + 6 * f, off0 + i * lev));
    {
        uint32_t o = off0;
#pragma unroll 1
        for (int g = 0; g < NG; g++) {
#pragma unroll 1
            for (int k = g * GL; k < min((g + 1) * GL, L); k++, o += lev) {
#pragma unroll
                for (int x = 0; x < 6; x++) gp_copy(&SL(x, k), at(in + x * f, o));
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    }
    const char *dq = A.dq ? (const char *)A.dq + (size_t)inst * f : nullptr;
    const double s = A.sid[h / A.nlon];
    const T rc = (T)(1.0 / (1.0 - s * s));
    const T rdbrv1 = (T)1. / (T)A.rdbrv - (T)1.;
    const bool spec = A.nqspec == 1;
    const T rrc = (T)1. / rc;
    T gpj, gpm, gp, rgp;
    auto humidity = [&](T gq, int k) {
        if (spec) return fmax(gp_div(gq, gp, rgp), (T)0.);
        return dq ? fmax(*at(dq, off0 + k * lev), (T)0.) : (T)0.;
    };
    // pass 1: the column totals of the divergence and of zvgpg, the sums over c of
    // zvgpg (sa) and of zvgpg + gd (sb), over g of ztv1 - gt (sg)
    T sa[LM], sb[LM], sg[LM], sq[KEEPQ ? LM : 1];
    T zsumd = 0, gvp = 0;
#pragma unroll
    for (int k = 0; k < LM; k++) {
        if (k % GL == 0) {
            constexpr int last = NG - 1;
            if (k / GL == 0) asm volatile("cp.async.wait_group %0;" ::"n"(last) : "memory");
            else if (k / GL == 1) asm volatile("cp.async.wait_group %0;" ::"n"(last - 1) : "memory");
            else if (k / GL == 2) asm volatile("cp.async.wait_group %0;" ::"n"(last - 2) : "memory");
            else asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        if (k == 0) {
            gpj = sl[6 * LM * GP_COLS];
            gpm = sl[(6 * LM + 1) * GP_COLS];
            gp = exp(sl[(6 * LM + 2) * GP_COLS]);            // gp = exp(gp), plasim.f90:2441
            rgp = (T)1. / gp;
        }
        if (KEEPQ) sq[KEEPQ ? k : 0] = 0;
        if (k < L) {
            const T gu = SL(0, k), gv = SL(1, k), gt = SL(2, k), gd = SL(3, k), gq = SL(5, k);
            const T zv = rc * (gu * gpm + gv * gpj);
            const T zq = humidity(gq, k);
            const T tv1 = (gt + K.t0[k]) * ((T)1. + rdbrv1 * zq) - K.t0[k];
            const T zb = zv + gd, z1 = tv1 - gt;
            if (KEEPQ) sq[KEEPQ ? k : 0] = zq;
            if (k == 0) { zsumd = K.ds[0] * gd; gvp = K.ds[0] * zv; }
            else { zsumd = zsumd + K.ds[k] * gd; gvp = gvp + K.ds[k] * zv; }
#pragma unroll
            for (int m = k; m < LM; m++) {
                sa[m] = k == 0 ? K.c[G::ci(0, m)] * zv : sa[m] + K.c[G::ci(k, m)] * zv;
                sb[m] = k == 0 ? K.c[G::ci(0, m)] * zb : sb[m] + K.c[G::ci(k, m)] * zb;
            }
#pragma unroll
            for (int m = 0; m <= k; m++) sg[m] = (m == k ? (T)0 : sg[m]) + K.g[G::gi(k, m)] * z1;
        }
    }
    const T tot = zsumd + gvp;
    // pass 2, level by level: sigma-dot, vertical advection terms and tendencies
    T psd = 0, psv = 0;                 // running sums of dsigma * gd and of dsigma * zvgpg
    T gtd_m = 0, gqm_m = 0, gud_m = 0, gvd_m = 0;   // the level above's products
    T zs = 0;                           // zsumd of the tendency loop (plasim.f90:2661, :2692)
    char *out = (char *)A.gout + (size_t)inst * (9 * f + lev), *dw = A.dw ? (char *)A.dw + (size_t)inst * f : nullptr;
    uint32_t o = off0;
    const auto put = [&](char *base, T v) { *reinterpret_cast<T *>(base + o) = v; };
    T nu = SL(0, 0), nv = SL(1, 0), nt = SL(2, 0), nq = SL(5, 0);
#pragma unroll
    for (int k = 0; k < LM; k++) {
        if (k < L) {
            const bool last = k == L - 1;
            const T gu = nu, gv = nv, gt = nt, gq = nq, gd = SL(3, k), gz = SL(4, k);
            if (k + 1 < LM && !last) { nu = SL(0, k + 1); nv = SL(1, k + 1); nt = SL(2, k + 1); nq = SL(5, k + 1); }
            const T zv = rc * (gu * gpm + gv * gpj);
            const T zq = KEEPQ ? sq[KEEPQ ? k : 0] : humidity(gq, k);
            const T tv1 = (gt + K.t0[k]) * ((T)1. + rdbrv1 * zq) - K.t0[k];
            const T tv2 = (gt + K.t0[k]) * ((T)1. + rdbrv1 * zq) / ((T)1. + (T)A.adv * zq) - K.t0[k];
            // this level's products of the sigma-dot flux with the layer differences
            T gtd = 0, gqm = 0, gud = 0, gvd = 0;
            if (!last) {
                if (k == 0) { psd = K.ds[0] * gd; psv = K.ds[0] * zv; }
                else { psd = psd + K.ds[k] * gd; psv = psv + K.ds[k] * zv; }
                const T zsdotp = (K.sh[k] * tot - (psd + psv));
                gtd = zsdotp * (nt - gt);
                gqm = zsdotp * (nq + gq);
                gud = zsdotp * (nu - gu);
                gvd = zsdotp * (nv - gv);
            }
            T gtn, gqn, guz, gvz, dwv;
            if (k == 0) {
                zs = zv * K.ds[0];
                gtn = gt * gd - (T)A.akap * tv2 * gd - K.rd[0] * (gtd + K.t01[0] * (K.sh[0] * gvp - zs));
                gqn = -K.rd[0] * gqm;
                guz = -gu * gz - gpj * tv1 - K.rd[0] * gvd;
                gvz = gv * gz - gpm * tv1 - K.rd[0] * gud;
                dwv = gd * gp * (T)A.psurf * (T)A.ww;
            } else {
                const T ztpta = sa[k], ztptb = sb[k];
                const int m = k > 0 ? k - 1 : 0;             // the level above
                // the lowest level has no flux below it: its own products are zero
                T adv;
                if (last) adv = gtd_m + K.t01[m] * (K.sh[m] * gvp - zs);
                else {
                    zs = zs + zv * K.ds[k];
                    adv = gtd + gtd_m + gvp * (K.t01[k] * K.sh[k] + K.t01[m] * K.sh[m]) - zs * (K.t01[m] + K.t01[k]) +
                          zv * K.ds[k] * K.t01[m];
                }
                gtn = gt * gd + (T)A.akap * tv2 * (zv - ztptb) + K.tkp[k] * (zv - ztpta) - K.rd[k] * adv;
                gqn = -K.rd[k] * (gqm - gqm_m);
                guz = -gu * gz - gpj * tv1 - K.rd[k] * (gvd + gvd_m);
                gvz = gv * gz - gpm * tv1 - K.rd[k] * (gud + gud_m);
                dwv = (zv - ztptb) * gp * (T)A.psurf * (T)A.ww;
            }
            const T gphi = gp_div(sg[k] * (T)2., rc, rrc);   // non-linear geopotential
            T ke = gu * gu + gv * gv;
            ke = ke + gphi;
            put(out, gtn);
            put(out + f, gqn);
            put(out + 2 * f, gu * gt);      // gut
            put(out + 3 * f, gv * gt);      // gvt
            put(out + 4 * f, guz);
            put(out + 5 * f, gvz);
            put(out + 6 * f, ke);           // gke
            put(out + 7 * f + lev, gu * gq);   // guq, past gvpp
            put(out + 8 * f + lev, gv * gq);   // gvq
            if (dw) put(dw, dwv);
            o += lev;
            gtd_m = gtd; gqm_m = gqm; gud_m = gud; gvd_m = gvd;
        }
    }
    o = off0;
    put(out + 7 * f, gvp);                  // gvpp
#undef SL
}

template <typename T, int LM>
inline exotx_status gp_launch_async(const GpArgs<T> &A, const exotx_gp_params &h, cudaStream_t s) {
    GpLevels<T, LM> K;
    K.fill(h);
    constexpr size_t smem = gp_slots<T, LM>();
    if (smem > 48 * 1024)
        EXOTX_CUDA(cudaFuncSetAttribute(k_gridpoint_async<T, LM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const long long nb = (A.ncol / A.nhor) * ((A.nhor + GP_COLS - 1) / GP_COLS);
    k_gridpoint_async<T, LM><<<(unsigned)nb, GP_COLS, smem, s>>>(A, K);
    EXOTX_CHECK_LAUNCH();
    return EXOTX_OK;
}
template <typename T, bool SK, int LC>
inline exotx_status gp_launch_k(const GpArgs<T> &A, size_t smem, cudaStream_t s) {
    const long long nb = (A.ncol + GP_THREADS - 1) / GP_THREADS;
    EXOTX_CUDA(allow_smem(k_gridpoint<T, SK, LC>, smem));
    k_gridpoint<T, SK, LC><<<(unsigned)nb, GP_THREADS, smem, s>>>(A);
    EXOTX_CHECK_LAUNCH();
    return EXOTX_OK;
}
// The asynchronous form takes initsi's triangular g up to 25 levels in FP32 and 20
// in FP64: its code is unrolled over the levels, and beyond 128 KB of it the
// instruction cache no longer holds it (FP64, asynchronous / general form: T127 x3
// with 20 levels 160 / 224 us, T85 x5 with 25 levels 376 / 290).  The rest runs in the
// general form, its constants in shared memory where they fit beside the profiles.
template <typename T>
inline exotx_status gp_launch(const GpArgs<T> &A, const exotx_gp_params &h, cudaStream_t s) {
    const int L = A.L;
    if (A.g_lower && L <= (sizeof(T) == 4 ? 25 : 20)) {
        if (L <= 7) return gp_launch_async<T, 7>(A, h, s);
        if (L <= 10) return gp_launch_async<T, 10>(A, h, s);
        if (L <= 13) return gp_launch_async<T, 13>(A, h, s);
        if (L <= 16) return gp_launch_async<T, 16>(A, h, s);
        if (L <= 20) return gp_launch_async<T, 20>(A, h, s);
        if constexpr (sizeof(T) == 4) return gp_launch_async<T, 25>(A, h, s);
    }
    const bool sk = gp_smem<T>(L, true) <= 227 * 1024;
    const size_t smem = gp_smem<T>(L, sk);
    if (!sk) return gp_launch_k<T, false, 0>(A, smem, s);
    // the level counts of the standard configurations, for other than initsi's g and for
    // FP64's 25 (T85 x3, any count / its own: FP32 L10 31 / 23 us, L20 90 / 55; FP64 alike)
    switch (L) {
        case 10: return gp_launch_k<T, true, 10>(A, smem, s);
        case 20: return gp_launch_k<T, true, 20>(A, smem, s);
        case 25: return gp_launch_k<T, true, 25>(A, smem, s);
        default: return gp_launch_k<T, true, 0>(A, smem, s);
    }
}

}  // namespace exotx
