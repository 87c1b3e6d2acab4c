// radmod.f90 radiation column pass on the GPU (device code).
//
// The reference evaluates radstep (:927-1110) with array statements over all
// NHOR columns.  Here a block owns COLS = 16 columns (fewer where a column's
// scratch is large), held in shared memory level by level with the columns
// fastest.  A thread works one column c = tid % COLS and takes the levels, or
// the (jlev, jlev2) pairs of lwr, i = tid / COLS, + rad_items, ...:
// the transcendental work (cloud optics, ozone and water-vapour
// transmissivities, the O(NLEV^2) longwave absorptivities) is spread over all
// threads.  What is serial in height -- mko3's sums, the absorber paths, the
// adding method of swr -- runs on one lane per column, the two bands of swr on
// lanes of their own, while the block's other warps already take lwr's pairs.
// Every expression and summation order is the reference's.
//
// Bound by the FP64 (FP32: FP32 and special-function) instructions of pow, log
// and exp.  One warp per column, the form before, left the serial parts to one
// lane of 32: they were two thirds of its instructions.  8192 T42 L20 columns:
// FP64 401 -> 176 us, FP32 265 -> 75 us.
#pragma once
#include <cmath>
#include "exotx_internal.cuh"

namespace exotx {

constexpr int RAD_MAXLEV = 64;

// Items (levels, pairs) in flight per column, and so threads per block: 32 in
// FP64, 16 in FP32 (half the registers per thread, so more blocks per SM).
template <typename T> constexpr int rad_items() { return sizeof(T) == 8 ? 32 : 16; }
template <typename T> constexpr int rad_threads(int cols) { return cols * rad_items<T>(); }
// threads per SM that the registers are shared out among
template <typename T> constexpr int RAD_SM_THREADS = sizeof(T) == 8 ? 512 : 768;

struct RadDev {
    exotx_rad_params p;
    const void *sid, *cola, *dt, *dq, *dcc, *dql, *dqco2, *dp, *dls, *dicec;
    void *dqo3, *gmu0, *dalb, *dsalb;
    void *dfu, *dfd, *dftu, *dftd, *dswfl, *dlwfl, *dflux, *dtdt, *dtdtswr, *dtdtlwr, *dconv;
    const void *zsol;       // optional (NHOR,3): per-column zsolar1, zsolar2, rcoeff
    const int *cols;        // optional list of the columns to compute ...
    const int *ncols;       // ... and its length (device memory)
};

template <typename T> __device__ __forceinline__ T P_(T x, T y);
template <> __device__ __forceinline__ double P_(double x, double y) { return pow(x, y); }
template <> __device__ __forceinline__ float P_(float x, float y) { return powf(x, y); }

// ozone and water-vapour broadband absorption fits (radmod.f90:1907-1913, :1992-1993)
template <typename T> __device__ T ao3_(T x) {
    return (T)0.02118 * x / ((T)1 + (T)0.042 * x + (T)0.000323 * (x * x)) +
           (T)1.082 * x / P_((T)1 + (T)138.6 * x, (T)0.805) +
           (T)0.0658 * x / ((T)1 + ((T)103.6 * x) * ((T)103.6 * x) * ((T)103.6 * x));
}
template <typename T> __device__ T awv_(T x) {
    return (T)2.9 * x / (P_((T)1 + (T)141.5 * x, (T)0.635) + (T)5.925 * x);
}

// cos zenith of column (jlat, jlon) clipped at dawn (solang, radmod.f90:1380-1436)
template <typename T>
__device__ __forceinline__ T solang_mu(const exotx_rad_params &P, const T *sid, const T *cola, int jlat, int jlon,
                                       int nlon) {
    const T PI = (T)3.14159265359, TWOPI = PI + PI;
    T zdawn = sin((T)P.dawn * PI / (T)180.0), zmuz;
    if (P.ncstsol == 0) {
        T zrlon = TWOPI / nlon;
        T zhangle = (T)P.zmins * (T)P.zrtim + jlon * zrlon - PI;
        if (P.ngenkeplerian == 1) zhangle = zhangle - (T)P.rasc;
        if (zhangle < -PI) zhangle = zhangle + TWOPI;
        if (zhangle > PI) zhangle = zhangle - TWOPI;
        if (P.nfixed == 1) zhangle = zhangle + PI;
        zmuz = sin((T)P.zdecl) * sid[jlat] + cola[jlat] * cos((T)P.zdecl) * cos(zhangle);
    } else {
        T solclatcdec = (T)P.solclat * (T)P.solcdec;
        T solslat = sqrt((T)1 - (T)P.solclat * (T)P.solclat);
        T solsdec = sqrt((T)1 - (T)P.solcdec * (T)P.solcdec);
        if (P.ndcycle == 1) zmuz = solslat * solsdec + solclatcdec * cos((T)P.zmins * (T)P.zrtim - PI);
        else zmuz = solslat * solsdec + solclatcdec / PI;
    }
    return (zmuz > zdawn) ? zmuz : (T)0.0;
}

// Per-column scratch in shared memory: slot k of an array at [k*COLS + column].
// Several arrays take another's place once that is read: see the phases below.
struct RadScratch {
    int dt, dq, dcc, dql, o3, co2;                     // inputs
    int rcl1, rcl1s, rcl2, rcl2s, tcl2, tcl2s;         // cloud optics -> rb1 rb1s rb2 rb2s tb2 tb2u -> rl1 rl1s rl2 rl2s
    int nd1, nu1, nd2, nu2;                            // absorbers, then 1 - absorption -> tb1 tb1u
    int o3l, xo3l, wvl, ywvl;                          // absorber paths -> t1 r1s t2 r2s -> fu fd
    int q, qo3, qco2, tcc, st4, st4h, bu, bd, tau0, ftu, ftd, tau;   // lwr
    int sc;                                            // scalars
    int size;
};
enum { SC_MU0 = 0, SC_MU1, SC_ZA, SC_ZCS, SC_O3T, SC_XO3T, SC_WVT, SC_YWVT, SC_RL1, SC_RL1S, SC_RL2, SC_RL2S, SC_N };
__host__ __device__ inline RadScratch rad_scratch(int L) {
    const int E = L + 1;
    RadScratch s;
    int p = 0;
    auto take = [&](int n) { const int r = p; p += n; return r; };
    s.dt = take(E); s.dq = take(E); s.dcc = take(E); s.dql = take(E); s.o3 = take(L); s.co2 = take(L);
    s.rcl1 = take(L); s.rcl1s = take(L); s.rcl2 = take(L); s.rcl2s = take(L); s.tcl2 = take(L); s.tcl2s = take(L);
    s.nd1 = take(L); s.nu1 = take(L); s.nd2 = take(L); s.nu2 = take(L);
    s.o3l = take(E); s.xo3l = take(E); s.wvl = take(E); s.ywvl = take(E);
    s.q = take(L); s.qo3 = take(L); s.qco2 = take(L); s.tcc = take(L);
    s.st4 = take(E); s.st4h = take(E); s.bu = take(E + 1); s.bd = take(E + 1);
    s.tau0 = take(L); s.ftu = take(E); s.ftd = take(E);
    s.tau = take(L * (L + 1) / 2);
    s.sc = take(SC_N);
    s.size = p;
    return s;
}
// lwr's fit constants (:2207-2218) and mko3's, formed once per block
enum { RK_AO30 = 0, RK_CO20, RK_H2O0A, RK_H2O0, RK_AO3C, RK_ACO2C, RK_AH2OC, RK_TH2OC, RK_ZCONST, RK_N };
template <typename T>
__device__ T rad_const(const exotx_rad_params &P, int i) {
    const T zao30 = (T)0.209 * P_((T)7.e-5, (T)0.436);
    const T zco20 = (T)0.0676 * P_((T)0.01022, (T)0.421);
    const T zh2o0a = (T)0.846 * P_((T)3.59e-5, (T)0.243);
    const T zh2o0 = (T)0.832 * P_((T)0.0286, (T)0.26);
    switch (i) {
        case RK_AO30: return zao30;
        case RK_CO20: return zco20;
        case RK_H2O0A: return zh2o0a;
        case RK_H2O0: return zh2o0;
        case RK_AO3C: return (T)0.209 * P_((T)0.01 + (T)7.e-5, (T)0.436) - zao30 - (T)0.0212 * log10((T)0.01);
        case RK_ACO2C: return (T)0.0676 * P_((T)1.01022, (T)0.421) - zco20;
        case RK_AH2OC: return (T)0.846 * P_((T)0.01 + (T)3.59e-5, (T)0.243) - zh2o0a - (T)0.24 * log10((T)0.02);
        case RK_TH2OC: return (T)1. - ((T)0.832 * P_((T)2. + (T)0.0286, (T)0.26) - zh2o0) + (T)0.1196 * log((T)2. - (T)0.6931);
        default: return exp(-(T)P.bo3 / (T)P.co3);
    }
}
// byte offset of the warps' argument buffers, after the scratch of COLS columns,
// the log(sigmah) ratios, the constants and the pair list; and the total
template <typename T>
__host__ __device__ inline size_t rad_args(int L, int cols) {
    const size_t b = ((size_t)rad_scratch(L).size * cols + L + RK_N) * sizeof(T) + 8 + (size_t)(L * (L + 1) / 2) * 2;
    return (b + 15) & ~(size_t)15;
}
template <typename T>
__host__ __device__ inline size_t rad_smem(int L, int cols) {
    return rad_args<T>(L, cols) + (sizeof(T) == 8 ? (size_t)(rad_threads<T>(cols) / 32) * 128 * sizeof(T) : 0);
}

template <typename T, int COLS>
__global__ void __launch_bounds__(rad_threads<T>(COLS), RAD_SM_THREADS<T> / rad_threads<T>(COLS))
    k_radstep(const __grid_constant__ RadDev D) {
    extern __shared__ __align__(16) unsigned char smraw[];
    const exotx_rad_params &P = D.p;
    const int L = P.nlev, E = L + 1, nhor = P.nhor, nlon = P.nlon, npair = L * (L + 1) / 2;
    const RadScratch S = rad_scratch(L);
    constexpr int NI = rad_items<T>(), NTHR = rad_threads<T>(COLS);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, c = tid % COLS, it0 = tid / COLS;
    T *sm = reinterpret_cast<T *>(smraw) + c;
    T *lg = reinterpret_cast<T *>(smraw) + (size_t)S.size * COLS;        // log(sigmah(j-1)/sigmah(j))
    T *kc = lg + L;                                                      // rad_const
    int *next = reinterpret_cast<int *>(kc + RK_N);                      // pair chunks handed out
    unsigned short *pairs = reinterpret_cast<unsigned short *>(next + 2);
#define V(a, k) sm[(S.a + (k)) * COLS]
    const int count = D.cols ? *D.ncols : nhor;
    if (blockIdx.x * COLS >= count) return;                              // an empty column list costs no more than this
    const T PI = (T)3.14159265359, TWOPI = PI + PI;
    const T ga = (T)P.ga, gascon = (T)P.gascon;
    const int nclouds = P.nclouds, newrsc = P.newrsc, nrscat = P.nrscat;
    const T *dt = (const T *)D.dt, *dq = (const T *)D.dq, *dcc = (const T *)D.dcc, *dql = (const T *)D.dql;
    const T *dqco2 = (const T *)D.dqco2, *dpv = (const T *)D.dp, *dlsv = (const T *)D.dls,
            *dicv = (const T *)D.dicec, *sid = (const T *)D.sid, *cola = (const T *)D.cola;
    T *dqo3 = (T *)D.dqo3, *gmu0 = (T *)D.gmu0, *dalbv = (T *)D.dalb, *dsalbv = (T *)D.dsalb;
    // shortwave constants
    const T zero = (T)1e-6, zbetta = (T)1.66, zmbar = (T)1.9, zro3 = (T)2.14, zfo3 = (T)100. / zro3;
    const T aa = (T)0.2542857142857143, bb = (T)0.8229693877551021, c0 = (T)0.14997959183673468;
    const T zmu00 = (T)0.5;
    const T zb3 = (T)P.tswr1 * sqrt(zmu00) / zmu00;
    const T zb4 = (T)P.tswr2 * sqrt(zmu00);
    const T zb5 = (T)P.tswr3 * zmu00 * zmu00;
    // the pair list and the level constants, once per block
    for (int jl = tid; jl < L; jl += NTHR) {
        const int p0 = jl * L - jl * (jl - 1) / 2;       // row jl has L - jl entries
        for (int jl2 = jl; jl2 < L; jl2++) pairs[p0 + jl2 - jl] = (unsigned short)(jl << 8 | jl2);
        if (jl >= 1) lg[jl] = log((T)P.sigmah[jl - 1] / (T)P.sigmah[jl]);
    }
    if (lane == 0)
        for (int i = warp; i < RK_N; i += NTHR / 32) kc[i] = rad_const<T>(P, i);
    for (int base = blockIdx.x * COLS; base < count; base += gridDim.x * COLS) {
        const bool valid = base + c < count;
        const int w = valid ? base + c : count - 1;      // spare lanes repeat the last column and store nothing
        const int col = D.cols ? D.cols[w] : w;
        const int jlat = col / nlon, jlon = col - jlat * nlon;
        T csol1 = (T)P.zsolar1, csol2 = (T)P.zsolar2, crco = (T)P.rcoeff;
        if (D.zsol) {
            const T *z = (const T *)D.zsol;
            csol1 = z[col];
            csol2 = z[(size_t)nhor + col];
            crco = z[2 * (size_t)nhor + col];
        }
        for (int k = it0; k < E; k += NI) {
            V(dt, k) = dt[(size_t)k * nhor + col];
            V(dq, k) = dq[(size_t)k * nhor + col];
            V(dcc, k) = dcc[(size_t)k * nhor + col];
            V(dql, k) = dql[(size_t)k * nhor + col];
            if (k < L) V(co2, k) = dqco2[(size_t)k * nhor + col];
            if (k < L && P.no3 != 1) V(o3, k) = dqo3[(size_t)k * nhor + col];
            // mko3's layer thickness factor, beside its o3 slot until the ozone is formed
            if (k < L && P.no3 == 1) V(q, k) = dt[(size_t)k * nhor + col] * gascon / ga;
        }
        const T dp = dpv[col], dls = dlsv[col], dicec = dicv[col];
        // solang (radmod.f90:1380-1436)
        if (it0 == 0) {
            T m;
            if (P.nsol == 1) {
                m = solang_mu<T>(P, sid, cola, jlat, jlon, nlon);
                if (valid) gmu0[col] = m;
            } else {
                m = gmu0[col];
            }
            V(sc, SC_MU0) = m;
            V(sc, SC_MU1) = m;
        }
        // insolation and cloud zenith factors (radmod.f90:1650-1669): the
        // column's own cos zenith, or with ndcycle = 0 the means over its
        // latitude row -- over the sunlit columns (clouds) and over all
        // (insolation).  A warp forms each column's sums, reading the row's
        // gmu0 or, when this launch computes gmu0, evaluating solang for each
        // column of the row itself.
        if (P.ndcycle == 0) {
            __syncthreads();
            for (int cc = warp; cc < COLS; cc += NTHR / 32) {
                const int ww = min(base + cc, count - 1), cl = D.cols ? D.cols[ww] : ww, jr = cl / nlon;
                T zsum = 0;
                int icnt = 0;
                for (int j = lane; j < nlon; j += 32) {
                    T g = P.nsol == 1 ? solang_mu<T>(P, sid, cola, jr, j, nlon) : gmu0[(size_t)jr * nlon + j];
                    zsum += g;
                    icnt += g > (T)0.0 ? 1 : 0;
                }
                for (int o = 16; o > 0; o >>= 1) {
                    zsum += __shfl_xor_sync(0xffffffffu, zsum, o);
                    icnt += __shfl_xor_sync(0xffffffffu, icnt, o);
                }
                if (lane == 0) {
                    T *sl = reinterpret_cast<T *>(smraw) + cc;
                    sl[(S.sc + SC_MU0) * COLS] = icnt > 0 ? zsum / (T)icnt : (T)0.0;
                    sl[(S.sc + SC_MU1) * COLS] = icnt > 0 ? zsum / (T)nlon : (T)0.0;
                }
            }
        }
        // mko3 (radmod.f90:1489-1522): the sums in height on one lane per column
        if (P.no3 == 1) {
            __syncthreads();
            const T zconst = kc[RK_ZCONST];
            if (it0 == 0) {
                T sd = sid[jlat];
                V(sc, SC_ZA) = (T)P.a0o3 + (T)P.a1o3 * fabs(sd) + (T)P.aco3 * sd * cos(TWOPI * ((T)P.zcday - (T)P.toffo3));
                T zh = 0;
                for (int jl = L - 1; jl >= 1; jl--) {
                    zh = zh - V(q, jl) * lg[jl];
                    V(qo3, jl) = zh;
                }
            }
            __syncthreads();
            const T za = V(sc, SC_ZA);
            for (int jl = it0; jl < L; jl += NI)
                if (jl >= 1) V(qco2, jl) = -(za + za * zconst) / ((T)1. + exp((V(qo3, jl) - (T)P.bo3) / (T)P.co3));
            __syncthreads();
            if (it0 == 0) {
                T zo3t = za;
                for (int jl = L - 1; jl >= 1; jl--) {
                    T zo3 = V(qco2, jl) + zo3t;
                    V(o3, jl) = zo3;
                    zo3t = zo3t - zo3;
                }
                V(o3, 0) = zo3t;
            }
            __syncthreads();
            for (int jl = it0; jl < L; jl += NI) {
                T o = V(o3, jl) * ga / (zfo3 * (T)P.dsigma[jl] * dp);
                if (P.o3scale != 1.0) o = o * (T)P.o3scale;
                V(o3, jl) = o;
                if (valid) dqo3[(size_t)jl * nhor + col] = o;
            }
        }
        if (tid == 0) *next = 0;
        __syncthreads();
        const T zmu0 = V(sc, SC_MU0), zmu1 = V(sc, SC_MU1);
        const T zftop1 = csol1 * (T)P.gsol0 * (T)P.gdist2 * zmu1;
        const T zftop2 = csol2 * (T)P.gsol0 * (T)P.gdist2 * zmu1;
        const bool lit = P.nswr == 1 && zftop1 + zftop2 > zero;
        // ---- per level: cloud optics and layer absorbers of swr, absorbers and clouds of lwr
        const T SBK = (T)5.67e-8;
        const T zmmair = (T)0.0289644, zmmco2 = (T)0.0440098, zpv2pm = zmmco2 / zmmair;
        const T zrco2 = (T)1.9635;
        const T zfh2o = (T)0.1, zfco2 = (T)100. / zrco2;
        const T zps2 = (P.npbroaden > 0.5) ? dp * dp : (T)101100.0 * (T)101100.0;
        if (lit)
            for (int jl = it0; jl < L; jl += NI) {
                // clear-sky fraction above the level (cloud block, :1681-1768)
                T zcs = 1;
                for (int i = 0; i < jl; i++) zcs = zcs * ((T)1 - V(dcc, i));
                const T cl = V(dcc, jl);
                T rcl1 = 0, rcl2 = 0, tcl2 = 1, rcl1s = 0, rcl2s = 0, tcl2s = 1;
                if (nclouds == 1) {
                    if (P.nswrcl == 0) {
                        T sg = (T)P.sigma[jl];
                        int r = (sg <= (T)(1. / 3.)) ? 0 : ((sg > (T)(1. / 3.) && sg <= (T)(2. / 3.)) ? 1 : 2);
                        T c1 = (T)P.rcl1[r], c2 = (T)P.rcl2[r], a2 = (T)P.acl2[r];
                        rcl1s = c1 / (c1 + zmu00);
                        rcl1 = zcs * c1 / (c1 + zmu0) + ((T)1 - zcs) * rcl1s;
                        rcl2s = fmin((T)1 - a2, c2 / (c2 + zmu00));
                        rcl2 = fmin((T)1 - a2, zcs * c2 / (c2 + zmu0) + ((T)1 - zcs) * rcl2s);
                        tcl2s = (T)1 - rcl2s - a2;
                        tcl2 = (T)1 - rcl2 - a2;
                    } else if (cl > (T)0) {
                        T zlwp = fmin((T)1000.0, (T)1000. * V(dql, jl) * dp / ga * (T)P.dsigma[jl]);
                        T ztau = (T)2.0 * P_(log10(zlwp + (T)1.5), (T)3.9);
                        T zlog = log((T)1000.0 / ztau);
                        T zb2 = zb4 / log((T)3. + (T)0.1 * ztau);
                        T zom0 = fmin((T)0.9999, (T)1.0 - zb5 * zlog);
                        T zun = (T)1.0 - zom0;
                        T zuz = zun + (T)2.0 * zb2 * zom0;
                        T zu = sqrt(zuz / zun);
                        T zexp = exp(fmin((T)25.0, ztau * sqrt(zuz * zun) / zmu00));
                        T zr = (zu + (T)1.) * (zu + (T)1.) * zexp - (zu - (T)1.) * (zu - (T)1.) / zexp;
                        rcl1s = (T)1. - (T)1. / ((T)1. + zb3 * ztau);
                        tcl2s = (T)4. * zu / zr;
                        rcl2s = (zu * zu - (T)1.) / zr * (zexp - (T)1. / zexp);
                        T zb1 = (T)P.tswr1 * sqrt(zmu0);
                        zb2 = (T)P.tswr2 * sqrt(zmu0) / log((T)3. + (T)0.1 * ztau);
                        zom0 = fmin((T)0.9999, (T)1. - (T)P.tswr3 * zmu0 * zmu0 * zlog);
                        zun = (T)1.0 - zom0;
                        zuz = zun + (T)2.0 * zb2 * zom0;
                        zu = sqrt(zuz / zun);
                        zexp = exp(fmin((T)25.0, ztau * sqrt(zuz * zun) / zmu0));
                        zr = (zu + (T)1.) * (zu + (T)1.) * zexp - (zu - (T)1.) * (zu - (T)1.) / zexp;
                        rcl1 = (T)1. - (T)1. / ((T)1. + zb1 * ztau / zmu0);
                        tcl2 = (T)4. * zu / zr;
                        rcl2 = (zu * zu - (T)1.) / zr * (zexp - (T)1. / zexp);
                        rcl1 = zcs * rcl1 + ((T)1. - zcs) * rcl1s;
                        tcl2 = zcs * tcl2 + ((T)1. - zcs) * tcl2s;
                        rcl2 = zcs * rcl2 + ((T)1. - zcs) * rcl2s;
                    }
                }
                V(rcl1, jl) = rcl1; V(rcl2, jl) = rcl2; V(tcl2, jl) = tcl2;
                V(rcl1s, jl) = rcl1s; V(rcl2s, jl) = rcl2s; V(tcl2s, jl) = tcl2s;
                // absorber amounts of this layer (:1785-1789)
                V(nd1, jl) = zfo3 * (T)P.dsigma[jl] * dp * V(o3, jl) / ga;
                V(nd2, jl) = (T)0.1 * (T)P.dsigma[jl] * V(dq, jl) * dp / ga * sqrt((T)273. / V(dt, jl)) * (T)P.sigma[jl] *
                             dp / (T)100000.;
            }
        if (P.nlwr == 1) {
            // sigma T^4 on full levels and the surface, absorbers and cloud transmissivities
            for (int k = it0; k < E; k += NI) { T t2 = V(dt, k) * V(dt, k); V(st4, k) = SBK * (t2 * t2); }
            for (int jl = it0; jl < L; jl += NI) {
                T zzf1 = (T)P.sigma[jl] * (T)P.dsigma[jl] / ga / (T)100000.;
                T zzf2 = zpv2pm * (T)1.e-6;
                T zzf3 = (T)-1.66 * (T)P.acllwr * (T)1000. * (T)P.dsigma[jl] / ga;
                T zsfac = zzf1 * zps2;
                V(q, jl) = zfh2o * zsfac * V(dq, jl);
                V(qo3, jl) = zfo3 * zsfac * V(o3, jl);
                V(qco2, jl) = zfco2 * zzf2 * zsfac * V(co2, jl);
                if (P.clgray > 0) V(tcc, jl) = (T)1. - V(dcc, jl) * (T)P.clgray;
                else V(tcc, jl) = (T)1. - V(dcc, jl) * ((T)1. - exp(zzf3 * V(dql, jl) * dp));
            }
        }
        __syncthreads();
        // ---- accumulated absorber paths with the clear-sky mixing (:1779-1802), serial in height
        if (lit && it0 == 0) {
            const T zm = (T)35. / sqrt((T)1. + (T)1224. * zmu0 * zmu0);
            T zcs = 1, zo3t = 0, zxo3t = 0, zwvt = 0, zywvt = 0;
            for (int jl = 0; jl < L; jl++) {
                T zo3 = V(nd1, jl);
                zo3t = zo3t + zo3;
                zxo3t = zcs * (zxo3t + zm * zo3) + ((T)1. - zcs) * (zxo3t + zmbar * zo3);
                V(o3l, jl) = zo3t;
                V(xo3l, jl) = zxo3t;
                T zwv = V(nd2, jl);
                zwvt = zwvt + zwv;
                zywvt = zcs * (zywvt + zm * zwv) + ((T)1. - zcs) * (zywvt + zbetta * zwv);
                V(wvl, jl) = zwvt;
                V(ywvl, jl) = zywvt;
                zcs = zcs * ((T)1. - V(dcc, jl) * nclouds);
                V(nu1, jl) = zcs;
            }
            V(sc, SC_ZCS) = zcs; V(sc, SC_O3T) = zo3t; V(sc, SC_XO3T) = zxo3t; V(sc, SC_WVT) = zwvt; V(sc, SC_YWVT) = zywvt;
        }
        // half levels (:2230-2249)
        if (P.nlwr == 1)
            for (int k = it0; k < E; k += NI) {
                T v;
                if (k == 0) {
                    v = V(st4, 0) - (V(st4, 0) - V(st4, 1)) * (T)P.sigma[0] / ((T)P.sigma[0] - (T)P.sigma[1]);
                } else if (k < L) {
                    v = (V(st4, k) * ((T)P.sigma[k - 1] - (T)P.sigmah[k - 1]) + V(st4, k - 1) * ((T)P.sigmah[k - 1] - (T)P.sigma[k])) /
                        ((T)P.sigma[k - 1] - (T)P.sigma[k]);
                } else {
                    v = V(st4, L);
                    T h_L = (V(st4, L - 1) * ((T)P.sigma[L - 2] - (T)P.sigmah[L - 2]) +
                             V(st4, L - 2) * ((T)P.sigmah[L - 2] - (T)P.sigma[L - 1])) /
                            ((T)P.sigma[L - 2] - (T)P.sigma[L - 1]);
                    if (!((V(st4, L - 1) - h_L) * (V(st4, L - 1) - V(st4, L)) > (T)0.))
                        v = V(st4, L - 1) + (V(st4, L - 1) - V(st4, L - 2)) * ((T)1. - (T)P.sigma[L - 1]) /
                                               ((T)P.sigma[L - 1] - (T)P.sigma[L - 2]);
                }
                V(st4h, k) = v;
            }
        __syncthreads();
        // ---- transmissivity fits per level, and each layer's own reflectivities
        if (lit) {
            const T zcsf = V(sc, SC_ZCS), zo3t = V(sc, SC_O3T), zxo3t = V(sc, SC_XO3T), zwvt = V(sc, SC_WVT),
                    zywvt = V(sc, SC_YWVT);
            const T zs1 = csol1, zs2 = csol2;
            const T dccL = V(dcc, L - 1);
            const T zscf = crco * dp / (T)101100.0 * (T)9.80665 / ga;
            for (int i = it0; i < 2 * L; i += NI) {
                const int jl = i < L ? i : i - L;
                if (i < L) {
                    // Rayleigh scattering in the lowest layer only (newrsc = 0 default, :1928-1939)
                    const T zcs_run = V(nu1, jl);
                    T zrcs = (aa / ((T)1. + bb * zmu0) * zcs_run + c0 * ((T)1. - zcs_run - dccL * nclouds)) *
                             (T)P.dsigma[jl] * (dp / (T)101100.0) * ((T)9.80665 / ga) * nrscat * newrsc;
                    T zrcsu = c0 * ((T)1. - dccL) * (T)P.dsigma[jl] * (dp / (T)101100.0) * ((T)9.80665 / ga) * nrscat *
                              newrsc;
                    if (jl == L - 1) {
                        zrcs = zrcs * newrsc;
                        zrcsu = zrcsu * newrsc;
                        zrcsu = zrcsu + ((T)1.0 - exp(zscf * log((T)1.0 - (T)0.144))) * (1 - newrsc) * nrscat *
                                            ((T)1 - dccL * nclouds);
                        zrcs = zrcs + ((T)1.0 - exp(zscf * log((T)1.0 - ((T)0.219 / ((T)1. + (T)0.816 * zmu0))))) * zcsf *
                                          (1 - newrsc) * nrscat +
                               ((T)1.0 - exp(zscf * log((T)1.0 - (T)0.144))) * ((T)1. - zcsf - dccL) * nrscat *
                                   (1 - newrsc);
                    }
                    const T cl = V(dcc, jl);
                    V(rcl1, jl) = zrcs + V(rcl1, jl) * cl * nclouds;     // rb1
                    V(rcl1s, jl) = zrcsu + V(rcl1s, jl) * cl * nclouds;  // rb1s
                    V(nd1, jl) = (T)1. - ao3_<T>(V(xo3l, jl)) / zs1;
                    V(nu1, jl) = (T)1. - ao3_<T>(zxo3t + zmbar * (zo3t - V(o3l, jl))) / zs1;
                } else {
                    V(nd2, jl) = (T)1. - awv_<T>(V(ywvl, jl)) / zs2;
                    V(nu2, jl) = (T)1. - awv_<T>(zywvt + zbetta * (zwvt - V(wvl, jl))) / zs2;
                }
            }
        }
        __syncthreads();
        // ---- the adding method, one lane per column and band on warp 0
        const bool adds = tid < 2 * COLS && lit;
        const unsigned adding = warp == 0 ? __ballot_sync(0xffffffffu, adds) : 0u;
        if (adds) {
            const bool b1 = tid < COLS;
            const T zs1 = csol1, zs2 = csol2;
            T zta = 1, ztas = 1, zra = 0, zras = 0, ztt = 1, zttu;
            if (b1) zttu = (T)1. - ao3_<T>(V(sc, SC_XO3T) + zmbar * V(sc, SC_O3T)) / zs1;
            else zttu = (T)1. - awv_<T>(V(sc, SC_YWVT) + zbetta * V(sc, SC_WVT)) / zs2;
            // the absorber paths are read: their slots take t and rs of this band
            T *tt = sm + (b1 ? S.o3l : S.wvl) * COLS, *rr = sm + (b1 ? S.xo3l : S.ywvl) * COLS;
            T *rb = sm + (b1 ? S.rcl1 : S.rcl2) * COLS, *rbs = sm + (b1 ? S.rcl1s : S.rcl2s) * COLS;
            T *tb = sm + (b1 ? S.nd1 : S.tcl2) * COLS, *tbu = sm + (b1 ? S.nu1 : S.tcl2s) * COLS;
            const T *nd = sm + (b1 ? S.nd1 : S.nd2) * COLS, *nu = sm + (b1 ? S.nu1 : S.nu2) * COLS;
            for (int jl = 0; jl < L; jl++) {
                const int o = jl * COLS;
                const T cl = V(dcc, jl);
                T b, bs, t, tu;
                const T ztr = nd[o] / ztt;
                ztt = ztt * ztr;
                const T ztru = zttu / nu[o];
                zttu = zttu / ztru;
                if (b1) {
                    b = rb[o];
                    bs = rbs[o];
                    t = (T)1. - ((T)1. - ztr) * ((T)1. - cl) - b;
                    tu = (T)1. - ((T)1. - ztru) * ((T)1. - cl) - bs;
                } else {
                    b = rb[o] * cl * nclouds;
                    bs = rbs[o] * cl * nclouds;
                    t = (T)1. - ((T)1. - ztr) * ((T)1. - cl * nclouds) - ((T)1. - tb[o]) * cl * nclouds;
                    tu = (T)1. - ((T)1. - ztru) * ((T)1. - cl * nclouds) - ((T)1. - tbu[o]) * cl * nclouds;
                }
                tt[o] = zta;
                rr[o] = zras;
                const T z1mrabr = (T)1. / ((T)1. - zras * bs);
                zra = zra + zta * b * ztas * z1mrabr;
                zta = zta * t * z1mrabr;
                zras = bs + tu * zras * t * z1mrabr;
                ztas = tu * ztas * z1mrabr;
                rb[o] = b; rbs[o] = bs; tb[o] = t; tbu[o] = tu;
            }
            tt[L * COLS] = zta;
            rr[L * COLS] = zras;
            // surface albedo for the direct beam (:2046-2071)
            const int nst = P.nstartemp, ne = P.necham, ne6 = P.necham6;
            T dalb = dalbv[col];
            T dsalb[2] = {dsalbv[2 * col], dsalbv[2 * col + 1]};
            zras = dalb * (1 - nst) + dsalb[b1 ? 0 : 1] * nst;
            T ocean3 = fmin((T)0.05 / (zmu0 + (T)0.15), (T)0.15);
            T ocean6 = ((T)0.026 / (P_(zmu0, (T)1.7) + (T)0.065) +
                        (T)0.15 * (zmu0 - (T)1) * (zmu0 - (T)0.5) * (zmu0 - (T)0.1) + (T)0.0082);
            for (int i = 0; i < 2; i++) {
                dsalb[i] = dls * dsalb[i] + ((T)1. - dls) * dicec * dsalb[i] +
                           ((T)1. - dls) * ((T)1. - dicec) * ocean3 * ne * (1 - ne6) +
                           ((T)1. - dls) * ((T)1. - dicec) * (1 - ne) * ne6 * ocean6 +
                           ((T)1. - dls) * ((T)1. - dicec) * ((T)1. - ne) * (1 - ne6) * dsalb[i];
            }
            dalb = (csol1 * dsalb[0] + csol2 * dsalb[1]) * nst +
                   (dls * dalb + ((T)1. - dls) * dicec * dalb + ((T)1. - dls) * ((T)1. - dicec) * ocean3 * ne * (1 - ne6) +
                    ((T)1. - dls) * ((T)1. - dicec) * (1 - ne) * ne6 * ocean6 +
                    ((T)1. - dls) * ((T)1. - dicec) * ((T)1. - ne) * (1 - ne6) * dalb) *
                       (1 - nst);
            zra = dsalb[b1 ? 0 : 1] * nst + dalb * (1 - nst);
            __syncwarp(adding);   // both bands have read the albedos
            if (b1 && valid) {
                dalbv[col] = dalb;
                dsalbv[2 * col] = dsalb[0];
                dsalbv[2 * col + 1] = dsalb[1];
            }
            // upwards; level jl's rb and rbs slots take rl and rls of its upper interface
            V(sc, b1 ? SC_RL1 : SC_RL2) = zra;
            V(sc, b1 ? SC_RL1S : SC_RL2S) = zras;
            for (int jl = L - 1; jl >= 0; jl--) {
                const int o = jl * COLS;
                const T b = rb[o], bs = rbs[o], t = tb[o], tu = tbu[o];
                zra = b + t * zra * tu / ((T)1. - zras * bs);
                zras = bs + tu * zras * tu / ((T)1. - zras * bs);
                rb[o] = zra;
                rbs[o] = zras;
            }
        }
        // ---- lwr: clear-sky transmissivities for every (jlev, jlev2 >= jlev) pair (:2297-2346),
        // handed out 32/COLS at a time; each sums its absorbers, and multiplies the
        // layers' cloud transmissivities (random overlap), from jlev upward
        if (P.nlwr == 1) {
            const T zao30 = kc[RK_AO30], zco20 = kc[RK_CO20], zh2o0a = kc[RK_H2O0A], zh2o0 = kc[RK_H2O0];
            const T zao3c = kc[RK_AO3C], zaco2c = kc[RK_ACO2C], zah2oc = kc[RK_AH2OC], zth2oc = kc[RK_TH2OC];
            const T th2oc = (T)P.th2oc;
            constexpr int PW = 32 / COLS;
            // The fits' two branches (a power of a small path, a logarithm of a large
            // one) mix within a warp.  In FP64 its 4 x 32 arguments are sorted into the
            // powers (from the front of arg) and the logarithms (from the back), so each
            // is evaluated once by full warps (13 levels: 89 -> 80 us for 4608 columns);
            // in FP32 both branches cost less than the sorting (88 against 99 us)
            constexpr bool SORT = sizeof(T) == 8;
            __syncwarp();
            while (true) {
                int ch = lane == 0 ? atomicAdd(next, 1) : 0;
                ch = __shfl_sync(0xffffffffu, ch, 0);
                if (ch * PW >= npair) break;
                const int pi = ch * PW + lane / COLS;
                const bool live = pi < npair;
                const int jl = live ? pairs[pi] >> 8 : 0, jl2 = live ? pairs[pi] & 255 : 0;
                T zsumwv = 0, zsumo3 = 0, zsumco2 = 0, ztaucc = 1;
                for (int k = jl; k <= jl2; k++) {
                    zsumwv = zsumwv + V(q, k); zsumo3 = zsumo3 + V(qo3, k); zsumco2 = zsumco2 + V(qco2, k);
                    ztaucc = ztaucc * V(tcc, k);
                }
                T zah2o = 0, zaco2 = 0, zth2o = 0, zao3 = 0;
                if constexpr (SORT) {
                    T *arg = reinterpret_cast<T *>(smraw + rad_args<T>(L, COLS)) + warp * 128;
                    const T expo[4] = {(T)0.243, (T)0.421, (T)0.26, (T)0.436};
                    const unsigned below = (1u << lane) - 1u;
                    // evaluations 0 h2o, 1 co2, 2 h2o in the co2 overlap, 3 o3
                    const bool pw[4] = {zsumwv <= (T)0.01, zsumco2 <= (T)1.0, zsumwv <= (T)2., zsumo3 <= (T)0.01};
                    const T x[4] = {pw[0] ? zsumwv + (T)3.59e-5 : zsumwv + (T)0.01, pw[1] ? zsumco2 + (T)0.01022 : zsumco2,
                                    pw[2] ? zsumwv + (T)0.0286 : zsumwv - (T)0.6931, pw[3] ? zsumo3 + (T)7.e-5 : zsumo3};
                    int pos[4], np = 0, nl = 0, pend[4], l2a = 0, l2b = 0;
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const unsigned mp = __ballot_sync(0xffffffffu, live && pw[e]), ml = __ballot_sync(0xffffffffu, live && !pw[e]);
                        pos[e] = pw[e] ? np + __popc(mp & below) : 127 - (nl + __popc(ml & below));
                        if (e == 2) l2a = nl;
                        np += __popc(mp);
                        nl += __popc(ml);
                        if (e == 2) l2b = nl;
                        pend[e] = np;
                        if (live) arg[pos[e]] = x[e];
                    }
                    __syncwarp();
                    for (int i = lane; i < np; i += 32)
                        arg[i] = P_(arg[i], i < pend[0] ? expo[0] : i < pend[1] ? expo[1] : i < pend[2] ? expo[2] : expo[3]);
                    for (int i = lane; i < nl; i += 32) {
                        const T v = arg[127 - i];
                        arg[127 - i] = i >= l2a && i < l2b ? log(v) : log10(v);
                    }
                    __syncwarp();
                    if (live) {
                        T r[4];
#pragma unroll
                        for (int e = 0; e < 4; e++) r[e] = arg[pos[e]];
                        if (pw[0]) zah2o = (T)0.846 * r[0] - zh2o0a;
                        else zah2o = (T)0.24 * r[0] + zah2oc;
                        if (th2oc > (T)0.) zah2o = fmin(zah2o + ((T)1. - exp(-th2oc * zsumwv)), (T)1.);
                        if (pw[1]) zaco2 = (T)0.0676 * r[1] - zco20;
                        else zaco2 = (T)0.0546 * r[1] + zaco2c;
                        if (pw[2]) zth2o = (T)1. - ((T)0.832 * r[2] - zh2o0);
                        else zth2o = fmax((T)0., zth2oc - (T)0.1196 * r[2]);
                        if (pw[3]) zao3 = (T)0.209 * r[3] - zao30;
                        else zao3 = (T)0.0212 * r[3] + zao3c;
                    }
                    __syncwarp();   // arg is free for the next pairs
                } else if (live) {
                    if (zsumwv <= (T)0.01) zah2o = (T)0.846 * P_(zsumwv + (T)3.59e-5, (T)0.243) - zh2o0a;
                    else zah2o = (T)0.24 * log10(zsumwv + (T)0.01) + zah2oc;
                    if (th2oc > (T)0.) zah2o = fmin(zah2o + ((T)1. - exp(-th2oc * zsumwv)), (T)1.);
                    if (zsumco2 <= (T)1.0) zaco2 = (T)0.0676 * P_(zsumco2 + (T)0.01022, (T)0.421) - zco20;
                    else zaco2 = (T)0.0546 * log10(zsumco2) + zaco2c;
                    if (zsumwv <= (T)2.) zth2o = (T)1. - ((T)0.832 * P_(zsumwv + (T)0.0286, (T)0.26) - zh2o0);
                    else zth2o = fmax((T)0., zth2oc - (T)0.1196 * log(zsumwv - (T)0.6931));
                    if (zsumo3 <= (T)0.01) zao3 = (T)0.209 * P_(zsumo3 + (T)7.e-5, (T)0.436) - zao30;
                    else zao3 = (T)0.0212 * log10(zsumo3) + zao3c;
                }
                if (live) {
                    T tcs = (T)1. - zah2o - zao3 - zaco2 * zth2o;
                    tcs = fmin((T)1. - zero, fmax(zero, tcs));
                    if (jl == 0) V(tau0, jl2) = tcs;
                    V(tau, pi) = tcs * ztaucc;
                }
            }
        }
        __syncthreads();
        // ---- shortwave interface fluxes (in the slots of t1 and r1s)
        for (int jl = it0; jl < E; jl += NI) {
            T u = 0, d = 0;
            if (lit) {
                const T l1 = jl < L ? V(rcl1, jl) : V(sc, SC_RL1), l1s = jl < L ? V(rcl1s, jl) : V(sc, SC_RL1S);
                const T l2 = jl < L ? V(rcl2, jl) : V(sc, SC_RL2), l2s = jl < L ? V(rcl2s, jl) : V(sc, SC_RL2S);
                const T t1 = V(o3l, jl), t2 = V(wvl, jl);
                T z1mrabr = (T)1. / ((T)1. - V(xo3l, jl) * l1s);
                T zfd1 = t1 * z1mrabr;
                T zfu1 = -t1 * l1 * z1mrabr;
                z1mrabr = (T)1. / ((T)1. - V(ywvl, jl) * l2s);
                T zfd2 = t2 * z1mrabr;
                T zfu2 = -t2 * l2 * z1mrabr;
                u = zfu1 * zftop1 + zfu2 * zftop2;
                d = zfd1 * zftop1 + zfd2 * zftop2;
            }
            V(o3l, jl) = u;
            V(xo3l, jl) = d;
        }
        // ---- effective emission of each layer from the jlev = 1 transmissivities (:2376-2400)
        if (P.nlwr == 1) {
            for (int jl2 = it0; jl2 < L; jl2 += NI) {
                T prev = (jl2 == 0) ? (T)1. - zero : V(tau0, jl2 - 1);
                T ztau0 = V(tau0, jl2) / prev * V(tcc, jl2) * (T)P.tpofmt;
                ztau0 = fmin((T)1. - zero, fmax(zero, ztau0));
                T a = V(st4, jl2), h0 = V(st4h, jl2), h1 = V(st4h, jl2 + 1);
                T bd, bu;
                if ((a - h0) * (a - h1) > (T)0.) {
                    bd = (T)0.5 * a + (T)0.25 * (h0 + h1);
                    bu = bd;
                } else {
                    bd = (h1 - ztau0 * h0) / ((T)1. - ztau0) - (h0 - h1) / log(ztau0);
                    bu = h0 + h1 - bd;
                }
                V(bd, jl2 + 1) = bd;
                V(bu, jl2 + 1) = bu;
            }
            if (it0 == 0) {
                V(bd, 0) = 0;   // SBK * zttop**4 with zttop = 0
                V(bu, E) = (dls + (T)0.98 * ((T)1. - dls)) * V(st4, L);
            }
            __syncthreads();
            // fluxes (:2401-2415), each sum in the reference's order.
            // upward dftu(jlev): -zbu(jlev) then the terms of jlev2 = jlev..NLEV;
            // downward dftd(k): rows jlev < k contribute zbdl(jlev)*ztau(jlev,k-1) in
            // order, then iteration jlev = k (or the surface step) adds zbd(k-1).
            for (int i = it0; i < L + E; i += NI) {
                if (i < L) {
                    const int k = i, p0 = k * L - k * (k - 1) / 2 - k;   // row k's entry of jlev2 at p0 + jlev2
                    T u = (T)0 - V(bu, k + 1);
                    for (int jl2 = k; jl2 < L; jl2++) u = u - (V(bu, jl2 + 2) - V(bu, jl2 + 1)) * V(tau, p0 + jl2);
                    V(ftu, k) = u;
                } else {
                    const int k = i - L;
                    T d = 0;
                    for (int jl = 0; jl < k; jl++)
                        d = d + (V(bd, jl) - V(bd, jl + 1)) * V(tau, jl * L - jl * (jl - 1) / 2 - jl + (k - 1));
                    V(ftd, k) = d + V(bd, k);
                }
            }
            __syncthreads();
            const T zeps = dls + (T)0.98 * ((T)1. - dls);
            const T zepsd = ((T)1. - zeps) * V(ftd, L);
            for (int k = it0; k < E; k += NI) {
                if (k < L) V(ftu, k) = V(ftu, k) - V(tau, k * L - k * (k - 1) / 2 - k + (L - 1)) * zepsd;
                else V(ftu, L) = (T)0 - V(bu, E);
            }
        } else {
            for (int k = it0; k < E; k += NI) V(ftu, k) = V(ftd, k) = 0;
        }
        __syncthreads();
        // ---- outputs and heating rates (radstep :1084-1110)
        for (int k = it0; k < E; k += NI) {
            const T fu = V(o3l, k), fd = V(xo3l, k), ftu = V(ftu, k), ftd = V(ftd, k);
            const T sw0 = fu + fd, lw0 = ftu + ftd;
            if (!valid) continue;
            size_t o = (size_t)k * nhor + col;
            ((T *)D.dfu)[o] = fu;
            ((T *)D.dfd)[o] = fd;
            ((T *)D.dswfl)[o] = sw0;
            ((T *)D.dftu)[o] = ftu;
            ((T *)D.dftd)[o] = ftd;
            ((T *)D.dlwfl)[o] = lw0;
            ((T *)D.dflux)[o] = lw0 + sw0;
            if (k == L) continue;
            const int jl = k;
            const T sw1 = V(o3l, k + 1) + V(xo3l, k + 1), lw1 = V(ftu, k + 1) + V(ftd, k + 1);
            T fl0 = lw0 + sw0, fl1 = lw1 + sw1;
            T zdh;
            if (jl >= 1) zdh = -V(dt, jl) * gascon / ga * lg[jl];
            else zdh = -V(dt, 0) * gascon / ga * log((T)P.sigma[0] / (T)P.sigmah[0]) * (T)0.5;
            T den = (T)P.dsigma[jl] * dp * (T)P.acpd * ((T)1. + (T)P.adv * V(dq, jl));
            T zdtdt = -(ga * (fl1 - fl0) / den);
            ((T *)D.dtdt)[o] = ((T *)D.dtdt)[o] + zdtdt;
            ((T *)D.dtdtswr)[o] = -(ga * (sw1 - sw0) / den);
            ((T *)D.dtdtlwr)[o] = -(ga * (lw1 - lw0) / den);
            ((T *)D.dconv)[o] = (fl0 - fl1) / (zdh + (T)1.0e-9);
        }
        __syncthreads();   // the scratch is reused by the next columns
    }
#undef V
}

// Columns per block: 16, or fewer where the scratch of one block per SM in FP64,
// of two in FP32, does not fit.  (The registers allow one of 512 threads and three
// of 256, but two blocks of 16 columns, from 27 levels on, beat the blocks of eight
// that fit as many columns: L30 160 us against 173.)  8192 columns, L20: 16 columns
// 176 / 76 us, eight 183 / 81 (FP64 / FP32); eight columns by 512 threads 238, 16 by
// 256 in FP64 247.
template <typename T>
inline int rad_cols(int L) {
    const size_t room = 220 * 1024 / (sizeof(T) == 8 ? 1 : 2);
    return rad_smem<T>(L, 16) <= room ? 16 : rad_smem<T>(L, 8) <= room ? 8 : 4;
}

template <typename T>
inline exotx_status launch_radstep(const RadDev &D, int maxcols, bool list, cudaStream_t st) {
    const int L = D.p.nlev, cols = rad_cols<T>(L);
    const size_t smem = rad_smem<T>(L, cols);
    auto kern = cols == 16 ? k_radstep<T, 16> : cols == 8 ? k_radstep<T, 8> : k_radstep<T, 4>;
    EXOTX_CUDA(allow_smem(kern, smem));
    int blocks = (maxcols + cols - 1) / cols;
    // a column list is usually short (often empty): one wave of resident blocks
    // strides over it instead of one block per possible entry (FP32, 32768 columns all
    // listed: 549 us with one block per SM, 311 with the three that fit)
    if (list) {
        static int nsm = 0;
        if (!nsm) {
            int dev = 0;
            if (cudaGetDevice(&dev) != cudaSuccess ||
                cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || nsm < 1)
                nsm = 148;
        }
        const int regs = RAD_SM_THREADS<T> / rad_threads<T>(cols), fit = (int)((SMEM_MAX + 1024) / (smem + 1024));
        const int wave = nsm * (regs < fit ? regs : fit);
        blocks = blocks < wave ? blocks : wave;
    }
    cudaEvent_t ev = ktimer_start(EXOTX_K_RADSTEP, st);
    kern<<<blocks, rad_threads<T>(cols), smem, st>>>(D);
    EXOTX_CHECK_LAUNCH();
    ktimer_stop(EXOTX_K_RADSTEP, st, ev);
    return EXOTX_OK;
}

}  // namespace exotx
