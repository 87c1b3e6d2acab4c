// Folded SIMT Legendre transforms (FP64 parity path and FP32 path).
//
// Every spectral->Fourier operation of legmod.f90 is, per zonal wavenumber m,
//     F(lat, m) = sum_n c * T(m,n,lat) * X(m,n)      c in {1,-1,i,-i}
// and every Fourier->spectral operation is
//     X(m,n)    = sum_lat c * T(m,n,lat) * F(lat, m).
// The tables are exactly symmetric (P-type: qi,qc,qm,qq,qu) or antisymmetric
// (Q-type: qj,qe,qv) under lat -> -lat when n-m is even, and the reverse when
// n-m is odd, so both directions run over northern latitudes only:
//   inverse:  north = sym + anti, south = sym - anti
//   forward:  P-type terms see N+S for n-m even and N-S for odd; Q-type the reverse.
// The forward direction is the reference's own single-CPU branch
// (legmod.f90:191-220, :391-424, :466-497, :555-602); the inverse direction
// halves the work of the reference's unfolded loops (:240-254).
//
// A transform set is one launch per direction: the blocks of one launch cover
// every field, level and state of the set, so a small set fills the GPU and
// pays one launch.  Each thread keeps a register tile of the contraction
// (inverse: latitudes x columns, forward: modes x the outputs of a level) and
// reads its table entries straight from global memory (coalesced, shared by
// the block's warps through L1) one step ahead of their use; the other operand
// is staged in shared memory and read as broadcasts.
//
// Fourier-side addressing of the single operations is general: complex
// element (field f, latitude l, wavenumber m) lives at base + f*fs + l*ls +
// m*ms (complex units).  The sets work on the plan's m-major intermediate,
// complex (field, l, m) at m*nrows + field*nlat + l.
#include <algorithm>
#include "exotx_internal.cuh"

namespace exotx {

template <typename T> struct __align__(2 * sizeof(T)) C2 { T x, y; };
// a caller's array is aligned to its reals only
template <typename T> __device__ __forceinline__ C2<T> ld2(const T *p) { return C2<T>{p[0], p[1]}; }
__device__ __forceinline__ double mad(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float mad(float a, float b, float c) { return fmaf(a, b, c); }

constexpr int LEG_MAXSMEM = 200 * 1024;

// ------------------------------------------------------------------ inverse
// One launch covers up to three groups of units:
//   0  qi (P-type), a unit is one field
//   1  qj (Q-type), a unit is one field
//   2  qu and qv: a unit is a (divergence, vorticity) pair -> (u, v)
template <typename T>
struct LegInv {
    const T *tab;        // 4 inverse tables [t][w][j]
    const int *woff;
    const T *filt;       // skspgp(n)
    const T *a, *b;      // spectral inputs (re, im pairs); single op: fields a (and b) at stride a_fs (b_fs)
    long long a_fs, b_fs;
    T *oa, *ob;          // Fourier outputs (set: oa is the intermediate)
    long long fs, ls, ms, nrows;
    int nu[3], nt[3];    // units and column tiles of each group
    int ntiles, ty, tx;  // tiles per wavenumber; threads along columns and latitudes
    int L, nlat, nlath, ntp1, ncsp, nrsp, dset, mz;  // single op: wavenumbers ntp1 <= m < mz are zeroed
    T plavor;
};

// field maps of the sets: gridpointa takes sd[L] st[L] sz[L] sq[L] sp to
// gu gv gt gd gz gq gpj gpmt gp (6L+3 fields), gridpointd the same state to
// gu gv gt gq gp (4L+1).  Unit u of group 0 -> instance, input and output field
__device__ __forceinline__ void inv_field(int L, int dset, int u, int *inst, int *fin, int *fout) {
    const int nf = dset ? 2 * L + 1 : 4 * L + 1;
    *inst = u / nf;
    const int f = u - *inst * nf;
    if (dset) {
        *fin = f < L ? L + f : 2 * L + f;    // st, sq, sp
        *fout = 2 * L + f;
    } else {
        *fin = f;
        *fout = f < L ? 3 * L + f : f < 2 * L ? f + L : f < 4 * L ? f + 2 * L : 6 * L + 2;
    }
}

// Tile: JT latitudes x CC complex columns per thread (a column pair's two
// parities in separate sums).  Bound by the FP64 / FP32 pipe once the tile is
// 4 x 4 and by latency at the small resolutions, where 1 x 1 tiles spread the
// outputs over more threads (see inv_tile).
template <typename T, int JT, int CC, bool SET>
__global__ void __launch_bounds__(256) k_leg_inv(const __grid_constant__ LegInv<T> A) {
    extern __shared__ __align__(16) unsigned char smraw[];
    constexpr int LT = CC > 1 ? CC / 2 : 1;            // (D, Z) pairs per thread in group 2
    constexpr int U = JT * CC >= 8 ? 2 : 4;            // modes whose table entries are fetched together (even)
    C2<T> *xs = reinterpret_cast<C2<T> *>(smraw);
    const int m = blockIdx.x / A.ntiles;
    int ti = blockIdx.x - m * A.ntiles, g = 0;
    while (ti >= A.nt[g]) ti -= A.nt[g++];
    const int cpt = g == 2 ? LT : CC, cb = A.ty * cpt, u0 = ti * cb, n = min(cb, A.nu[g] - u0);
    const int nlat = A.nlat, nlath = A.nlath;
    pdl_trigger();
    pdl_wait();
    if (!SET && m >= A.ntp1) {   // the zero tail of the Fourier rows, wavenumbers fastest
        const int nz = A.mz - A.ntp1;
        for (int i = threadIdx.x; i < n * nlat * nz; i += blockDim.x) {
            const int z = i % nz, r = i / nz, lat = r % nlat, c = r / nlat;
            const size_t o = 2 * ((u0 + c) * A.fs + lat * A.ls + (long long)(A.ntp1 + z) * A.ms);
            A.oa[o] = 0; A.oa[o + 1] = 0;
            if (g == 2) { A.ob[o] = 0; A.ob[o + 1] = 0; }
        }
        return;
    }
    const int K = A.ntp1 - m, w0 = A.woff[m], Kp = (K + U - 1) / U * U;
    const int cs = cb + 1;       // odd row stride in complex units: staging writes spread over the banks
    C2<T> *xz = xs + (size_t)Kp * cs;
    // stage the filtered coefficients as [k][column], zeros past the last mode and column
    for (int i = threadIdx.x; i < cb * Kp; i += blockDim.x) {
        const int c = i / Kp, k = i - c * Kp;
        C2<T> va{0, 0}, vb{0, 0};
        if (c < n && k < K) {
            const T f = A.filt[m + k];
            const T *pa, *pb = nullptr;
            if constexpr (SET) {
                int inst, fin, fout;
                if (g == 0) inv_field(A.L, A.dset, u0 + c, &inst, &fin, &fout);
                else if (g == 1) { inst = u0 + c; fin = 4 * A.L; }
                else { inst = (u0 + c) / A.L; fin = (u0 + c) - inst * A.L; }
                pa = A.a + ((size_t)inst * (4 * A.L + 1) + fin) * A.nrsp;
                pb = pa + (size_t)2 * A.L * A.nrsp;
            } else {
                pa = A.a + (u0 + c) * A.a_fs;
                if (g == 2) pb = A.b + (u0 + c) * A.b_fs;
            }
            va = ld2(pa + 2 * (w0 + k));
            va.x *= f; va.y *= f;
            if (g == 2) {
                // vorticity; plavor leaves mode (0,1) (legmod.f90:332)
                vb = ld2(pb + 2 * (w0 + k));
                if (m == 0 && k == 1) vb.x -= A.plavor;
                vb.x *= f; vb.y *= f;
            }
        }
        xs[(size_t)k * cs + c] = va;
        if (g == 2) xz[(size_t)k * cs + c] = vb;
    }
    __syncthreads();
    const int ty = threadIdx.x / A.tx, tx = threadIdx.x - ty * A.tx;
    if (ty >= A.ty) return;
    const size_t tsz = (size_t)A.ncsp * nlath;
    int jc[JT];
#pragma unroll
    for (int i = 0; i < JT; i++) jc[i] = min(tx + i * A.tx, nlath - 1);
    const C2<T> *xr = xs + ty * cpt;
    auto put = [&](T *o, long long f, int lat, C2<T> v) {
        if constexpr (SET) reinterpret_cast<C2<T> *>(o)[(size_t)m * A.nrows + f * nlat + lat] = v;
        else {
            const size_t e = 2 * (f * A.fs + lat * A.ls + (long long)m * A.ms);
            o[e] = v.x; o[e + 1] = v.y;
        }
    };
    if (g < 2) {
        // qi is P-type (even n-m symmetric), qj Q-type: its two sums swap roles
        const T *tp = A.tab + (g == 0 ? INV_QI : INV_QJ) * tsz + (size_t)w0 * nlath;
        C2<T> s[JT][CC], a[JT][CC];
        T t0[U][JT], t1[U][JT];
#pragma unroll
        for (int i = 0; i < JT; i++)
#pragma unroll
            for (int c = 0; c < CC; c++) s[i][c] = a[i][c] = C2<T>{0, 0};
        auto fetch = [&](T (&t)[U][JT], int k) {
#pragma unroll
            for (int e = 0; e < U; e++)
#pragma unroll
                for (int i = 0; i < JT; i++) t[e][i] = k + e < K ? tp[(size_t)(k + e) * nlath + jc[i]] : (T)0;
        };
        auto step = [&](const T (&t)[U][JT], int k) {
#pragma unroll
            for (int e = 0; e < U; e++) {
                C2<T> x[CC];
#pragma unroll
                for (int c = 0; c < CC; c++) x[c] = xr[(size_t)(k + e) * cs + c];
#pragma unroll
                for (int i = 0; i < JT; i++)
#pragma unroll
                    for (int c = 0; c < CC; c++) {
                        C2<T> &o = (e & 1) ? a[i][c] : s[i][c];
                        o.x = mad(t[e][i], x[c].x, o.x);
                        o.y = mad(t[e][i], x[c].y, o.y);
                    }
            }
        };
        fetch(t0, 0);
        for (int k = 0; k < Kp; k += 2 * U) {
            fetch(t1, k + U);
            step(t0, k);
            if (k + U >= Kp) break;
            fetch(t0, k + 2 * U);
            step(t1, k + U);
        }
#pragma unroll
        for (int c = 0; c < CC; c++) {
            const int u = u0 + ty * CC + c;
            if (ty * CC + c >= n) continue;
            long long f = u;
            bool gpmt = false;
            if constexpr (SET) {
                int inst, fin, fout = 6 * A.L;
                if (g == 0) inv_field(A.L, A.dset, u, &inst, &fin, &fout);
                else inst = u;
                f = (long long)inst * (A.dset ? 4 * A.L + 1 : 6 * A.L + 3) + fout;
                gpmt = g == 0 && !A.dset && fout == 6 * A.L + 2;
            }
#pragma unroll
            for (int i = 0; i < JT; i++) {
                const int j = tx + i * A.tx;
                if (j >= nlath) continue;
                const C2<T> e = s[i][c], o = a[i][c];
                const C2<T> vn{e.x + o.x, e.y + o.y};
                const C2<T> vs = g == 0 ? C2<T>{e.x - o.x, e.y - o.y} : C2<T>{o.x - e.x, o.y - e.y};
                put(A.oa, f, j, vn);
                put(A.oa, f, nlat - 1 - j, vs);
                if (gpmt) {   // gpmt = i*m*gp (plasim.f90:2425-2430), the field before gp
                    const T mm = (T)m;
                    put(A.oa, f - 1, j, C2<T>{-vn.y * mm, vn.x * mm});
                    put(A.oa, f - 1, nlat - 1 - j, C2<T>{-vs.y * mm, vs.x * mm});
                }
            }
        }
    } else {
        // u = sum qv*Z - i*qu*D ; v = sum -i*qu*Z - qv*D  (legmod.f90:338-341)
        const T *tu = A.tab + INV_QU * tsz + (size_t)w0 * nlath, *tv = A.tab + INV_QV * tsz + (size_t)w0 * nlath;
        const C2<T> *zr = xz + ty * cpt;
        C2<T> us[JT][LT], ua[JT][LT], vs[JT][LT], va[JT][LT];   // symmetric and antisymmetric sums of u and v
        T p0[U][JT], q0[U][JT], p1[U][JT], q1[U][JT];
#pragma unroll
        for (int i = 0; i < JT; i++)
#pragma unroll
            for (int c = 0; c < LT; c++) us[i][c] = ua[i][c] = vs[i][c] = va[i][c] = C2<T>{0, 0};
        auto fetch = [&](T (&p)[U][JT], T (&q)[U][JT], int k) {
#pragma unroll
            for (int e = 0; e < U; e++)
#pragma unroll
                for (int i = 0; i < JT; i++) {
                    const size_t o = (size_t)(k + e) * nlath + jc[i];
                    p[e][i] = k + e < K ? tu[o] : (T)0;
                    q[e][i] = k + e < K ? tv[o] : (T)0;
                }
        };
        auto step = [&](const T (&p)[U][JT], const T (&q)[U][JT], int k) {
#pragma unroll
            for (int e = 0; e < U; e++)
#pragma unroll
                for (int c = 0; c < LT; c++) {
                    const C2<T> D = xr[(size_t)(k + e) * cs + c], Z = zr[(size_t)(k + e) * cs + c];
#pragma unroll
                    for (int i = 0; i < JT; i++) {
                        // qu terms (P-type) and qv terms (Q-type) fall on opposite parities
                        C2<T> &uP = (e & 1) ? ua[i][c] : us[i][c], &uQ = (e & 1) ? us[i][c] : ua[i][c];
                        C2<T> &vP = (e & 1) ? va[i][c] : vs[i][c], &vQ = (e & 1) ? vs[i][c] : va[i][c];
                        uP.x = mad(p[e][i], D.y, uP.x);
                        uP.y = mad(-p[e][i], D.x, uP.y);
                        uQ.x = mad(q[e][i], Z.x, uQ.x);
                        uQ.y = mad(q[e][i], Z.y, uQ.y);
                        vP.x = mad(p[e][i], Z.y, vP.x);
                        vP.y = mad(-p[e][i], Z.x, vP.y);
                        vQ.x = mad(-q[e][i], D.x, vQ.x);
                        vQ.y = mad(-q[e][i], D.y, vQ.y);
                    }
                }
        };
        fetch(p0, q0, 0);
        for (int k = 0; k < Kp; k += 2 * U) {
            fetch(p1, q1, k + U);
            step(p0, q0, k);
            if (k + U >= Kp) break;
            fetch(p0, q0, k + 2 * U);
            step(p1, q1, k + U);
        }
#pragma unroll
        for (int c = 0; c < LT; c++) {
            const int u = u0 + ty * LT + c;
            if (ty * LT + c >= n) continue;
            long long fu = u, fv = u;
            T *ov = A.ob;
            if constexpr (SET) {
                const int inst = u / A.L;
                fu = (long long)inst * (A.dset ? 4 * A.L + 1 : 6 * A.L + 3) + (u - inst * A.L);
                fv = fu + A.L;
                ov = A.oa;
            }
#pragma unroll
            for (int i = 0; i < JT; i++) {
                const int j = tx + i * A.tx;
                if (j >= nlath) continue;
                put(A.oa, fu, j, C2<T>{us[i][c].x + ua[i][c].x, us[i][c].y + ua[i][c].y});
                put(A.oa, fu, nlat - 1 - j, C2<T>{us[i][c].x - ua[i][c].x, us[i][c].y - ua[i][c].y});
                put(ov, fv, j, C2<T>{vs[i][c].x + va[i][c].x, vs[i][c].y + va[i][c].y});
                put(ov, fv, nlat - 1 - j, C2<T>{vs[i][c].x - va[i][c].x, vs[i][c].y - va[i][c].y});
            }
        }
    }
}

// ------------------------------------------------------------------ forward
// the sets' operations on one level: gridpointa's mktend and qtend together,
// gridpointd's fc2sp of the temperature and humidity tendencies and uv2dv
enum { OP_LEVEL_A = 4, OP_LEVEL_D = 5 };

template <typename T>
struct LegFwd {
    const T *tab;        // 4 forward tables, per-m blocks [t][woff*nlath + j*K + k]
    const int *woff;
    const T *filt;       // skgpsp(n)
    const T *in[6];      // single op: Fourier inputs; set: in[0] is the intermediate
    long long fs, ls, ms, nrows;
    T *out[3];           // single op: spectral outputs; set: out[0] is the set's output
    long long o_fs;      // spectral field stride (reals)
    int nu, nt;          // units (levels x states) and unit tiles per wavenumber
    int nu1, nt1;        // gridpointa: ln ps tendencies (fc2sp) and their tiles
    int lb, jc;          // units per block, latitude pairs per staged chunk
    int L, nlat, nlath, ntp1, ncsp;
};

template <int OP> struct FwdShape;
template <> struct FwdShape<OP_FC2SP> { static constexpr int nin = 1, nout = 1; static constexpr bool c = 1, e = 0, m = 0, q = 0; };
template <> struct FwdShape<OP_UV2DV> { static constexpr int nin = 2, nout = 2; static constexpr bool c = 0, e = 1, m = 1, q = 0; };
template <> struct FwdShape<OP_QTEND> { static constexpr int nin = 3, nout = 1; static constexpr bool c = 1, e = 1, m = 1, q = 0; };
template <> struct FwdShape<OP_MKTEND> { static constexpr int nin = 6, nout = 3; static constexpr bool c = 1, e = 1, m = 1, q = 1; };
template <> struct FwdShape<OP_LEVEL_A> { static constexpr int nin = 9, nout = 4; static constexpr bool c = 1, e = 1, m = 1, q = 1; };
template <> struct FwdShape<OP_LEVEL_D> { static constexpr int nin = 4, nout = 4; static constexpr bool c = 1, e = 1, m = 1, q = 0; };

// o += t * x, o += i * t * x, o -= i * t * x
template <typename T> __device__ __forceinline__ void acc(C2<T> &o, T t, C2<T> x) { o.x = mad(t, x.x, o.x); o.y = mad(t, x.y, o.y); }
template <typename T> __device__ __forceinline__ void acc_i(C2<T> &o, T t, C2<T> x) { o.x = mad(-t, x.y, o.x); o.y = mad(t, x.x, o.y); }
template <typename T> __device__ __forceinline__ void acc_mi(C2<T> &o, T t, C2<T> x) { o.x = mad(t, x.y, o.x); o.y = mad(-t, x.x, o.y); }

// One latitude pair's terms of one mode; P(i), Q(i) are input i's folded value
// of the parity that P- and Q-type tables pair with.  In FP32 a latitude
// pair's terms are summed before they join the running sum: one rounding of the
// long sum per latitude pair instead of three (relative error against FP64 at
// T85 2.2e-7 instead of 3.2e-7); in FP64 the tables' own rounding dominates.
template <typename T, int OP, typename FP, typename FQ>
__device__ __forceinline__ void fwd_terms(C2<T> *sum, T c, T e, T mm, T qq, FP P, FQ Q) {
    constexpr int NOUT = FwdShape<OP>::nout;
    constexpr bool GROUP = sizeof(T) == 4;
    C2<T> part[NOUT];
    C2<T> *o = GROUP ? part : sum;
    if constexpr (GROUP) {
#pragma unroll
        for (int x = 0; x < NOUT; x++) part[x] = C2<T>{0, 0};
    }
    if constexpr (OP == OP_FC2SP) {          // sp = sum qc*f  (legmod.f90:203-220)
        acc(o[0], c, P(0));
    } else if constexpr (OP == OP_UV2DV) {   // d = -qe*v + i*qm*u, z = qe*u + i*qm*v  (:391-424)
        acc(o[0], -e, Q(1)); acc_i(o[0], mm, P(0));
        acc(o[1], e, Q(0));  acc_i(o[1], mm, P(1));
    } else if constexpr (OP == OP_QTEND) {   // q = qe*vq + qc*qn - i*qm*uq; in qn, uq, vq  (:466-497)
        acc(o[0], e, Q(2)); acc(o[0], c, P(0)); acc_mi(o[0], mm, P(1));
    } else if constexpr (OP == OP_MKTEND || OP == OP_LEVEL_A) {
        // mktend (:555-602): d = qq*ke - qe*fv + i*qm*fu, t = qe*vt + qc*tn - i*qm*ut, z = qe*fu + i*qm*fv.
        // Inputs: mktend tn, fu, fv, ke, ut, vt; the level's tn, qn, ut, vt, fv (guz), fu (gvz), ke, uq, vq
        constexpr bool A = OP == OP_LEVEL_A;
        constexpr int TN = 0, FU = A ? 5 : 1, FV = A ? 4 : 2, KE = A ? 6 : 3, UT = A ? 2 : 4, VT = A ? 3 : 5;
        acc(o[0], qq, P(KE)); acc(o[0], -e, Q(FV)); acc_i(o[0], mm, P(FU));
        acc(o[1], e, Q(VT)); acc(o[1], c, P(TN)); acc_mi(o[1], mm, P(UT));
        acc(o[2], e, Q(FU)); acc_i(o[2], mm, P(FV));
        if constexpr (A) { acc(o[3], e, Q(8)); acc(o[3], c, P(1)); acc_mi(o[3], mm, P(7)); }   // qtend
    } else {                                 // gridpointd: in t, u, v, q
        acc(o[0], -e, Q(2)); acc_i(o[0], mm, P(1));
        acc(o[1], c, P(0));
        acc(o[2], e, Q(1)); acc_i(o[2], mm, P(2));
        acc(o[3], c, P(3));
    }
    if constexpr (GROUP) {
#pragma unroll
        for (int x = 0; x < NOUT; x++) { sum[x].x += part[x].x; sum[x].y += part[x].y; }
    }
}

// Tile: KT modes of one parity x every output of one unit per thread; the
// lanes of a warp take consecutive modes of both parities.  The units' folded
// values (N+S, N-S) are staged jc latitude pairs at a time and read as
// broadcasts, eleven complex values for the 22 products of a gridpointa level,
// so with KT = 4 the kernel is near the FP64 / FP32 pipe's rate; small sets
// take KT = 1 for more threads (see fwd_tile).
template <typename T, int OP, int KT, bool SET>
__device__ __forceinline__ void leg_fwd_block(const LegFwd<T> &A, C2<T> *sm, int m, int u0, int n, int lb) {
    using S = FwdShape<OP>;
    constexpr int NIN = S::nin, NOUT = S::nout;
    const int nlath = A.nlath, nlat = A.nlat, L = A.L;
    const int K = A.ntp1 - m, w0 = A.woff[m];
    const int K0 = (K + 1) >> 1, K1 = K >> 1, q0 = (K0 + KT - 1) / KT, q1 = (K1 + KT - 1) / KT, qn = q0 + q1;
    const int us = 2 * A.jc + 1;          // a unit's staged values of one input: {sum, difference} per latitude pair
    // this thread's unit and modes
    const int l = threadIdx.x / qn, r = threadIdx.x - l * qn;
    const bool odd = r >= q0, active = l < n;
    const int kq = odd ? r - q0 : r, kst = odd ? q1 : q0, kcnt = odd ? K1 : K0;
    int k[KT];
#pragma unroll
    for (int i = 0; i < KT; i++) k[i] = 2 * min(kq + i * kst, kcnt - 1) + odd;
    const size_t tsz = (size_t)A.ncsp * nlath;
    const T *tb = A.tab + (size_t)w0 * nlath;
    C2<T> o[KT][NOUT];
#pragma unroll
    for (int i = 0; i < KT; i++)
#pragma unroll
        for (int x = 0; x < NOUT; x++) o[i][x] = C2<T>{0, 0};
    const C2<T> *sp = sm + (size_t)l * us + (odd ? 1 : 0), *sq = sm + (size_t)l * us + (odd ? 0 : 1);
    struct Tab { T c, e, m, q; };
    auto fetch = [&](Tab (&t)[KT], int j) {
        const size_t jo = (size_t)j * K;
#pragma unroll
        for (int i = 0; i < KT; i++) {
            if constexpr (S::c) t[i].c = tb[FWD_QC * tsz + jo + k[i]];
            if constexpr (S::e) t[i].e = tb[FWD_QE * tsz + jo + k[i]];
            if constexpr (S::m) t[i].m = tb[FWD_QM * tsz + jo + k[i]];
            if constexpr (S::q) t[i].q = tb[FWD_QQ * tsz + jo + k[i]];
        }
    };
    Tab ta[KT], tn[KT];
    if (active) fetch(ta, 0);
    for (int j0 = 0; j0 < nlath; j0 += A.jc) {
        const int nj = min(A.jc, nlath - j0);
        if (j0) __syncthreads();
        for (int idx = threadIdx.x; idx < NIN * n * nj; idx += blockDim.x) {
            const int jj = idx % nj, rr = idx / nj, ul = rr % n, i = rr / n, u = u0 + ul, j = j0 + jj;
            C2<T> vn, vs;
            if constexpr (SET) {
                long long f;
                if constexpr (OP == OP_FC2SP) f = (long long)u * (9 * L + 1) + 7 * L;   // gvpp of state u
                else {
                    const int inst = u / L, lev = u - inst * L;
                    // gridpointa: tn qn ut vt uz vz ke [vpp] uq vq; gridpointd: t u v q
                    f = (long long)inst * (OP == OP_LEVEL_A ? 9 * L + 1 : 4 * L) + i * L + lev + (OP == OP_LEVEL_A && i >= 7);
                }
                const C2<T> *w = reinterpret_cast<const C2<T> *>(A.in[0]) + (size_t)m * A.nrows + f * nlat;
                vn = w[j];
                vs = w[nlat - 1 - j];
            } else {
                const T *w = A.in[i] + 2 * (u * A.fs + (long long)m * A.ms);
                vn = ld2(w + 2 * (j * A.ls));
                vs = ld2(w + 2 * ((nlat - 1 - j) * A.ls));
            }
            C2<T> *d = sm + ((size_t)i * lb + ul) * us + 2 * jj;
            d[0] = C2<T>{vn.x + vs.x, vn.y + vs.y};
            d[1] = C2<T>{vn.x - vs.x, vn.y - vs.y};
        }
        __syncthreads();
        if (!active) continue;
        const size_t is = (size_t)lb * us;
        for (int jj = 0; jj < nj; jj++) {
            fetch(tn, min(j0 + jj + 1, nlath - 1));
#pragma unroll
            for (int i = 0; i < KT; i++)
                fwd_terms<T, OP>(o[i], ta[i].c, ta[i].e, ta[i].m, ta[i].q,
                                 [&](int f) { return sp[f * is + 2 * jj]; }, [&](int f) { return sq[f * is + 2 * jj]; });
#pragma unroll
            for (int i = 0; i < KT; i++) ta[i] = tn[i];
        }
    }
    if (!active) return;
    const int u = u0 + l;
#pragma unroll
    for (int i = 0; i < KT; i++) {
        if (kq + i * kst >= kcnt) continue;
        const T f = A.filt[m + k[i]];
#pragma unroll
        for (int x = 0; x < NOUT; x++) {
            T *d;
            if constexpr (SET) {
                // sdf[L] stf[L] szf[L] sqf[L] (gridpointa: spf)
                if constexpr (OP == OP_FC2SP) d = A.out[0] + ((size_t)u * (4 * L + 1) + 4 * L) * A.o_fs;
                else {
                    const int inst = u / L, lev = u - inst * L;
                    d = A.out[0] + ((size_t)inst * (OP == OP_LEVEL_A ? 4 * L + 1 : 4 * L) + x * L + lev) * A.o_fs;
                }
            } else d = A.out[x] + (size_t)u * A.o_fs;
            d[2 * (w0 + k[i])] = o[i][x].x * f;
            d[2 * (w0 + k[i]) + 1] = o[i][x].y * f;
        }
    }
}

template <typename T, int OP, int KT, bool SET>
__global__ void __launch_bounds__(KT == 4 ? 384 : 512) k_leg_fwd(const __grid_constant__ LegFwd<T> A) {
    extern __shared__ __align__(16) unsigned char smraw[];
    C2<T> *sm = reinterpret_cast<C2<T> *>(smraw);
    const int nt = A.nt + A.nt1, m = blockIdx.x / nt, ti = blockIdx.x - m * nt;
    pdl_trigger();
    pdl_wait();
    if (ti < A.nt) {
        const int u0 = ti * A.lb;
        leg_fwd_block<T, OP, KT, SET>(A, sm, m, u0, min(A.lb, A.nu - u0), A.lb);
    } else if constexpr (OP == OP_LEVEL_A) {
        const int u0 = (ti - A.nt) * A.lb;
        leg_fwd_block<T, OP_FC2SP, KT, SET>(A, sm, m, u0, min(A.lb, A.nu1 - u0), A.lb);
    }
}

template <typename T> static const T *inv_tab(exotx_plan p);
template <> const double *inv_tab<double>(exotx_plan p) { return p->d_inv64; }
template <> const float *inv_tab<float>(exotx_plan p) { return p->d_inv32; }
template <typename T> static const T *fwd_tab(exotx_plan p);
template <> const double *fwd_tab<double>(exotx_plan p) { return p->d_fwd64; }
template <> const float *fwd_tab<float>(exotx_plan p) { return p->d_fwd32; }
template <typename T> static const T *filt_s(exotx_plan p);
template <> const double *filt_s<double>(exotx_plan p) { return p->d_fs64; }
template <> const float *filt_s<float>(exotx_plan p) { return p->d_fs32; }
template <typename T> static const T *filt_g(exotx_plan p);
template <> const double *filt_g<double>(exotx_plan p) { return p->d_fg64; }
template <> const float *filt_g<float>(exotx_plan p) { return p->d_fg32; }

// ------------------------------------------------------------ host launchers
// the inverse tile (0: 1 x 1, 1: 2 x 2, 2: 4 x 4 outputs per thread): the
// largest that still leaves LEG_THREADS threads.  cols: complex columns, a
// (D, Z) pair counting as two
constexpr long long LEG_THREADS = 40000;   // about 270 per SM
static int inv_tile(exotx_plan p, long long cols) {
    const long long outs = (long long)p->ntp1 * p->nlath * cols;
    return outs / 16 >= LEG_THREADS || p->nlath > 512 ? 2 : outs / 4 >= LEG_THREADS || p->nlath > 256 ? 1 : 0;
}
// modes per thread of the forward kernels, by the same rule
static int fwd_tile(exotx_plan p, long long units) {
    const long long outs = units * p->ncsp;
    return outs / 4 >= LEG_THREADS || p->ntp1 > 512 ? 4 : outs / 2 >= LEG_THREADS ? 2 : 1;
}

template <typename T, int JT, int CC, bool SET>
static exotx_status inv_launch_t(exotx_plan p, LegInv<T> &A, cudaStream_t s) {
    constexpr int LT = CC > 1 ? CC / 2 : 1;
    A.tx = (p->nlath + JT - 1) / JT;
    const int want = JT == 4 ? 192 : 128;
    A.ty = std::max(1, want / A.tx);
    // the staged columns of a block (modes x columns, twice for (D, Z) pairs) within the budget
    auto smem_of = [&](int ty) {
        const size_t Kp = (p->ntp1 + 3) & ~3;
        const size_t one = Kp * (ty * CC + 1), two = A.nu[2] ? 2 * Kp * (ty * LT + 1) : 0;
        return std::max(one, two) * 2 * sizeof(T);
    };
    while (A.ty > 1 && smem_of(A.ty) > 72 * 1024) A.ty--;
    const size_t smem = smem_of(A.ty);
    if (smem > LEG_MAXSMEM) return EXOTX_BAD_DIM;
    const int cb[3] = {A.ty * CC, A.ty * CC, A.ty * LT};
    A.ntiles = 0;
    for (int g = 0; g < 3; g++) A.ntiles += A.nt[g] = (A.nu[g] + cb[g] - 1) / cb[g];
    const int nm = p->ntp1 + (!SET && A.mz > p->ntp1 ? 1 : 0);
    const long long blocks = (long long)nm * A.ntiles;
    if (blocks > 0x7fffffffLL) return EXOTX_BAD_DIM;
    const int threads = (A.tx * A.ty + 31) / 32 * 32;
    auto kern = k_leg_inv<T, JT, CC, SET>;
    if (smem > 48 * 1024) EXOTX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LEG_MAXSMEM));
    cudaEvent_t ev = ktimer_start(EXOTX_K_LEG_INVERSE, s);
    EXOTX_CUDA(launch_pdl(kern, dim3((unsigned)blocks), dim3(threads), smem, s, A));
    EXOTX_CHECK_LAUNCH();
    ktimer_stop(EXOTX_K_LEG_INVERSE, s, ev);
    return EXOTX_OK;
}
template <typename T, bool SET>
static exotx_status inv_launch(exotx_plan p, LegInv<T> &A, cudaStream_t s) {
    A.tab = inv_tab<T>(p); A.woff = p->d_woff; A.filt = filt_s<T>(p);
    A.nlat = p->nlat; A.nlath = p->nlath; A.ntp1 = p->ntp1; A.ncsp = p->ncsp; A.nrsp = 2 * p->ncsp;
    A.plavor = (T)p->desc.plavor;
    switch (inv_tile(p, (long long)A.nu[0] + A.nu[1] + 2LL * A.nu[2])) {
        case 0: return inv_launch_t<T, 1, 1, SET>(p, A, s);
        case 1: return inv_launch_t<T, 2, 2, SET>(p, A, s);
        default: return inv_launch_t<T, 4, 4, SET>(p, A, s);
    }
}

template <typename T>
exotx_status leg_inverse_l(exotx_plan p, int op, const T *a, const T *b, T *oa, T *ob, int nlev,
                           long long a_fs, long long b_fs, FourierLayout L, cudaStream_t s) {
    if (nlev <= 0) return EXOTX_OK;
    if (op != OP_SP2FC && op != OP_SP2FCDMU && op != OP_DV2UV) return EXOTX_BAD_ARG;
    LegInv<T> A = {};
    A.a = a; A.b = b; A.a_fs = a_fs; A.b_fs = b_fs;
    A.oa = oa; A.ob = ob; A.fs = L.fs; A.ls = L.ls; A.ms = L.ms; A.mz = L.mz;
    A.nu[op == OP_SP2FC ? 0 : op == OP_SP2FCDMU ? 1 : 2] = nlev;
    return inv_launch<T, false>(p, A, s);
}

template <typename T>
exotx_status leg_inverse_set(exotx_plan p, int dset, const T *spin, T *W, int L, int ninst, cudaStream_t s) {
    LegInv<T> A = {};
    A.a = spin;
    A.oa = W;
    A.L = L; A.dset = dset;
    A.nrows = (long long)ninst * (dset ? 4 * L + 1 : 6 * L + 3) * p->nlat;
    A.nu[0] = ninst * (dset ? 2 * L + 1 : 4 * L + 1);
    A.nu[1] = dset ? 0 : ninst;
    A.nu[2] = ninst * L;
    return inv_launch<T, true>(p, A, s);
}

template <typename T, int OP, int KT, bool SET>
static exotx_status fwd_launch_t(exotx_plan p, LegFwd<T> &A, cudaStream_t s) {
    const int K0 = (p->ntp1 + 1) / 2, K1 = p->ntp1 / 2;
    const int qn = (K0 + KT - 1) / KT + (K1 + KT - 1) / KT;   // threads per unit at m = 0
    A.lb = std::min(std::max(1, 160 / qn), std::max(A.nu, 1));
    A.jc = std::min(p->nlath, 32);
    auto smem_of = [&] { return (size_t)FwdShape<OP>::nin * A.lb * (2 * A.jc + 1) * 2 * sizeof(T); };
    while (A.jc > 8 && smem_of() > 48 * 1024) A.jc = (A.jc + 1) / 2;
    const size_t smem = smem_of();
    const int threads = (qn * A.lb + 31) / 32 * 32;
    if (smem > LEG_MAXSMEM || threads > (KT == 4 ? 384 : 512)) return EXOTX_BAD_DIM;
    A.nt = (A.nu + A.lb - 1) / A.lb;
    A.nt1 = (A.nu1 + A.lb - 1) / A.lb;
    const long long blocks = (long long)p->ntp1 * (A.nt + A.nt1);
    if (blocks > 0x7fffffffLL) return EXOTX_BAD_DIM;
    auto kern = k_leg_fwd<T, OP, KT, SET>;
    if (smem > 48 * 1024) EXOTX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LEG_MAXSMEM));
    cudaEvent_t ev = ktimer_start(EXOTX_K_LEG_FORWARD, s);
    EXOTX_CUDA(launch_pdl(kern, dim3((unsigned)blocks), dim3(threads), smem, s, A));
    EXOTX_CHECK_LAUNCH();
    ktimer_stop(EXOTX_K_LEG_FORWARD, s, ev);
    return EXOTX_OK;
}
template <typename T, int OP, bool SET>
static exotx_status fwd_launch(exotx_plan p, LegFwd<T> &A, cudaStream_t s) {
    A.tab = fwd_tab<T>(p); A.woff = p->d_woff; A.filt = filt_g<T>(p);
    A.nlat = p->nlat; A.nlath = p->nlath; A.ntp1 = p->ntp1; A.ncsp = p->ncsp;
    switch (fwd_tile(p, A.nu)) {
        case 1: return fwd_launch_t<T, OP, 1, SET>(p, A, s);
        case 2: return fwd_launch_t<T, OP, 2, SET>(p, A, s);
        default: return fwd_launch_t<T, OP, 4, SET>(p, A, s);
    }
}

template <typename T>
exotx_status leg_forward_l(exotx_plan p, int op, const T *const *in, T *const *out, int nlev,
                           FourierLayout L, long long o_fs, cudaStream_t s) {
    if (nlev <= 0) return EXOTX_OK;
    LegFwd<T> A = {};
    const int nin = op == OP_FC2SP ? 1 : op == OP_UV2DV ? 2 : op == OP_QTEND ? 3 : 6;
    const int nout = op == OP_MKTEND ? 3 : op == OP_UV2DV ? 2 : 1;
    for (int i = 0; i < nin; i++) A.in[i] = in[i];
    for (int i = 0; i < nout; i++) A.out[i] = out[i];
    A.fs = L.fs; A.ls = L.ls; A.ms = L.ms; A.o_fs = o_fs;
    A.nu = nlev;
    switch (op) {
        case OP_FC2SP: return fwd_launch<T, OP_FC2SP, false>(p, A, s);
        case OP_UV2DV: return fwd_launch<T, OP_UV2DV, false>(p, A, s);
        case OP_QTEND: return fwd_launch<T, OP_QTEND, false>(p, A, s);
        case OP_MKTEND: return fwd_launch<T, OP_MKTEND, false>(p, A, s);
    }
    return EXOTX_BAD_ARG;
}

template <typename T>
exotx_status leg_forward_set(exotx_plan p, int dset, const T *W, T *spout, int L, int ninst, cudaStream_t s) {
    LegFwd<T> A = {};
    A.in[0] = W;
    A.out[0] = spout;
    A.o_fs = 2LL * p->ncsp;
    A.L = L;
    A.nrows = (long long)ninst * (dset ? 4 * L : 9 * L + 1) * p->nlat;
    A.nu = ninst * L;
    A.nu1 = dset ? 0 : ninst;
    return dset ? fwd_launch<T, OP_LEVEL_D, true>(p, A, s) : fwd_launch<T, OP_LEVEL_A, true>(p, A, s);
}

#define LEG_INSTANCES(T)                                                                                            \
    template exotx_status leg_inverse_l<T>(exotx_plan, int, const T *, const T *, T *, T *, int, long long,         \
                                           long long, FourierLayout, cudaStream_t);                                 \
    template exotx_status leg_forward_l<T>(exotx_plan, int, const T *const *, T *const *, int, FourierLayout,       \
                                           long long, cudaStream_t);                                                \
    template exotx_status leg_inverse_set<T>(exotx_plan, int, const T *, T *, int, int, cudaStream_t);              \
    template exotx_status leg_forward_set<T>(exotx_plan, int, const T *, T *, int, int, cudaStream_t);
LEG_INSTANCES(double)
LEG_INSTANCES(float)

}  // namespace exotx
