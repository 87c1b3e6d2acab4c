// Folded Legendre transforms of the FP64 and FP32 paths on the FP64 tensor
// cores (mma.sync m8n8k4.f64: fused multiply-adds in FP64, no split or rounding
// of the operands; tcgen05 has no FP64 form).
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
// pays one launch.  A warp owns 8-row tiles of the table (latitudes inverse,
// modes forward) by groups of 8 real columns (4 complex fields or levels).  Its
// table fragments come straight from global memory (64-byte runs, shared by the
// block's warps through L1), one step ahead of their use; the other operand is
// staged in shared memory as FP64, also for the FP32 path, whose arrays are
// float but whose sums run in FP64 with the FP64 tables and are rounded once.
// Factors i and -i read the partner column (re <-> im) and flip its sign.
//
// One T127 L20 state, FP64: 52 us inverse and 62 forward against 147 and 180 for
// register-tiled FP64 FMA kernels (4 x 4 tiles: 240 registers,
// 6 warps per SM, the FP64 pipe 16% busy: two of three instructions were loads
// and addresses).  Eight DMMAs need six loads here, and the FP64 tensor cores
// were measured at 36.7 TFLOP/s (FMA: 30.8).
//
// Fourier-side addressing of the single operations is general: complex
// element (field f, latitude l, wavenumber m) lives at base + f*fs + l*ls +
// m*ms (complex units).  The sets work on the plan's m-major intermediate,
// complex (field, l, m) at m*nrows + field*nlat + l.
#include <algorithm>
#include <type_traits>
#include "exotx_internal.cuh"

namespace exotx {

template <typename T> struct __align__(2 * sizeof(T)) C2 { T x, y; };
using Z2 = C2<double>;
// a caller's array is aligned to its reals only
template <typename T> __device__ __forceinline__ Z2 ld2(const T *p) { return Z2{(double)p[0], (double)p[1]}; }

// d (8x8, lane: row lane/4, columns 2(lane%4) and +1) += a (8x4, lane: row
// lane/4, column lane%4) * b (4x8, lane: row lane%4, column lane/4)
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d[0]), "+d"(d[1])
                 : "d"(a), "d"(b));
}
// asynchronous copy of one complex value to shared memory (zeros where !ok);
// WIDE: source aligned to its size, otherwise to its reals only
template <bool WIDE, typename T>
__device__ __forceinline__ void cp_complex(C2<T> *dst, const T *src, bool ok) {
    constexpr int B = sizeof(T);
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (WIDE) {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(2 * B), "r"(ok ? 2 * B : 0) : "memory");
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d), "l"(src), "n"(B), "r"(ok ? B : 0) : "memory");
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(d + B), "l"(src + 1), "n"(B), "r"(ok ? B : 0) : "memory");
    }
}
// row stride (doubles) of staged operands of nc real columns (a multiple of 8):
// 4 or 12 mod 16, so the four rows of a fragment fall on distinct banks
__host__ __device__ constexpr int leg_stride(int nc) { return nc + 4; }

constexpr int LEG_MAXSMEM = 200 * 1024;

// ------------------------------------------------------------------ inverse
// One launch covers up to three groups of units:
//   0  qi (P-type), a unit is one field
//   1  qj (Q-type), a unit is one field
//   2  qu and qv: a unit is a (divergence, vorticity) pair -> (u, v)
template <typename T>
struct LegInv {
    const double2 *tab;  // 4 inverse tables of tsz fragment pairs (plan.cu k_layout_inv)
    const int *ioff;     // first step of each wavenumber
    size_t tsz;
    const int *woff;
    const double *filt;  // skspgp(n)
    const T *a;          // spectral inputs (re, im pairs); single op: fields at stride a_fs,
    long long a_fs, b_off;   // the second input b_off bytes from the first
    T *oa, *ob;          // Fourier outputs (set: oa is the intermediate)
    long long fs, ls, ms, nrows;
    int nu[3], nt[3];    // units and column tiles of each group
    int ntiles, nlb;     // tiles per wavenumber; latitude blocks
    int wm, wn, kc;      // warps along latitudes and columns; modes staged at a time
    int L, nlat, nlath, ntl, ntp1, nrsp, dset, mz;  // ntl: tiles of 8 latitudes; single op: wavenumbers ntp1 <= m < mz are zeroed
    double plavor;
    const double *rscale;  // single op: factor of each latitude's coefficients (null: 1) ...
    double scale;          // ... times this,
    int roll;              // and (-1)^m: the grid row turned by half its length
};

// One launch covers up to NSEG segments (a resolution, a level count and a run
// of states each); segment i's blocks start at blk0[i]
template <typename A, int NSEG>
struct LegLaunch {
    A seg[NSEG];
    int blk0[NSEG];
    int nseg;
    __device__ __forceinline__ int find(int b) const {
        int i = 0;
        if constexpr (NSEG > 1)
            while (i + 1 < nseg && b >= blk0[i + 1]) i++;
        return i;
    }
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

// A warp: MT tiles of 8 latitudes x NT groups of 4 complex columns (group 2:
// x 4 (D, Z) pairs), both parities of n-m in separate accumulators.  A step is
// 8 modes: a tile's fragments of both parities are one 16-byte load per lane.
template <typename T, int MT, int NT, bool SET, int NSEG>
__global__ void __launch_bounds__(192, NT == 1 ? 2 : 4) k_leg_inv(const __grid_constant__ LegLaunch<LegInv<T>, NSEG> P) {
    const int seg = P.find(blockIdx.x), blk = blockIdx.x - P.blk0[seg];
    const LegInv<T> &A = P.seg[seg];
    constexpr bool PF = NT == 1;   // fetch a step ahead: few warps to hide the latency
    extern __shared__ __align__(16) unsigned char smraw[];
    double *xs = reinterpret_cast<double *>(smraw);
    int ti = blk % A.ntiles, g = 0;
    const int mb = blk / A.ntiles, m = mb / A.nlb, lb = mb - m * A.nlb;
    while (ti >= A.nt[g]) ti -= A.nt[g++];
    const int cb = (g == 2 ? 4 : 4 * NT) * A.wn, u0 = ti * cb, n = min(cb, A.nu[g] - u0);
    const int nlat = A.nlat, nlath = A.nlath;
    pdl_trigger();
    pdl_wait();
    if (!SET && m >= A.ntp1) {   // the zero tail of the Fourier rows, wavenumbers fastest
        const int nz = A.mz - A.ntp1;
        for (int i = threadIdx.x + lb * blockDim.x; i < n * nlat * nz; i += A.nlb * blockDim.x) {
            const int z = i % nz, r = i / nz, lat = r % nlat, c = r / nlat;
            const size_t o = 2 * ((u0 + c) * A.fs + lat * A.ls + (long long)(A.ntp1 + z) * A.ms);
            A.oa[o] = 0; A.oa[o + 1] = 0;
            if (g == 2) { A.ob[o] = 0; A.ob[o + 1] = 0; }
        }
        return;
    }
    const int K = A.ntp1 - m, w0 = A.woff[m];
    const int rs = leg_stride(2 * cb);
    double *xz = xs + (size_t)A.kc * rs;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int wn = warp / A.wm, wm = warp - wn * A.wm;
    const int cw = wn * (g == 2 ? 4 : 4 * NT);                       // the warp's first column of the block
    const int j0 = (lb * A.wm + wm) * 8 * MT;
    const bool active = wn < A.wn && cw < n && j0 < nlath;
    // fragment pairs of the warp's tiles, step by step (tiles past the last repeat it)
    const size_t sstr = (size_t)A.ntl * 32;
    const double2 *t0 = A.tab + (g == 0 ? INV_QI : g == 1 ? INV_QJ : INV_QU) * A.tsz + A.ioff[m] * sstr + lane;
    int to[MT];
#pragma unroll
    for (int i = 0; i < MT; i++) to[i] = min((j0 >> 3) + i, A.ntl - 1) * 32;
    // accumulators by parity: [p][tile][column group] (group 2: symmetric and
    // antisymmetric sums of u, then of v)
    double acc[2][MT][NT < 2 ? 2 : NT][2];
#pragma unroll
    for (int p = 0; p < 2; p++)
#pragma unroll
        for (int i = 0; i < MT; i++)
#pragma unroll
            for (int c = 0; c < (NT < 2 ? 2 : NT); c++) acc[p][i][c][0] = acc[p][i][c][1] = 0.0;
    for (int kb = 0; kb < K; kb += A.kc) {
        const int kn = min(A.kc, K - kb), kp = (kn + 7) & ~7, kh = kp >> 1;
        if (kb) __syncthreads();
        // stage the filtered coefficients, even modes then odd ones, zeros past the
        // last mode and column; a warp takes a column, lanes along its modes
        // two columns at a time, their loads together
        const int nw = blockDim.x >> 5;
        const long long bo = SET ? (long long)sizeof(T) * 2 * A.L * A.nrsp : A.b_off;   // bytes from a's field to b's
        for (int cc = warp; cc < cb; cc += 2 * nw) {
            const T *pa[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int c = cc + h * nw, u = u0 + min(c, n - 1);
                if constexpr (SET) {
                    int inst, fin, fout;
                    if (g == 0) inv_field(A.L, A.dset, u, &inst, &fin, &fout);
                    else if (g == 1) { inst = u; fin = 4 * A.L; }
                    else { inst = u / A.L; fin = u - inst * A.L; }
                    pa[h] = A.a + ((size_t)inst * (4 * A.L + 1) + fin) * A.nrsp;
                } else {
                    pa[h] = A.a + u * A.a_fs;
                }
                pa[h] += 2 * (w0 + kb);
            }
            const double *fl = A.filt + m + kb;
            for (int k = lane; k < kp; k += 32) {
                Z2 va[2], vb[2];
                const double f = k < kn ? fl[k] : 0.0;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const bool in = cc + h * nw < n && k < kn;
                    va[h] = vb[h] = Z2{0, 0};
                    if (in) va[h] = ld2(pa[h] + 2 * k);
                    if (in && g == 2) vb[h] = ld2(reinterpret_cast<const T *>(reinterpret_cast<const char *>(pa[h] + 2 * k) + bo));
                }
                const int o = ((k & 1) * kh + (k >> 1)) * rs;
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const int c = cc + h * nw;
                    if (c >= cb) break;
                    *reinterpret_cast<Z2 *>(xs + o + 2 * c) = Z2{va[h].x * f, va[h].y * f};
                    if (g == 2) {
                        // vorticity; plavor leaves mode (0,1) (legmod.f90:332)
                        if (m == 0 && kb + k == 1 && c < n) vb[h].x -= A.plavor;
                        *reinterpret_cast<Z2 *>(xz + o + 2 * c) = Z2{vb[h].x * f, vb[h].y * f};
                    }
                }
            }
        }
        __syncthreads();
        if (!active) continue;
        const int nst = kp >> 3;
        const double2 *tk = t0 + (kb >> 3) * sstr;
        const double *x0 = xs + q * rs + 2 * cw + r, *x1 = x0 + kh * rs;   // the two parities' rows
        const int dx = 4 * rs;
        if (g < 2) {
            double2 fa[MT], fb[MT];
            auto fetch = [&](double2 (&t)[MT]) {
#pragma unroll
                for (int i = 0; i < MT; i++) t[i] = tk[to[i]];
                tk += sstr;
            };
            auto step = [&](const double2 (&t)[MT], auto nc) {
#pragma unroll
                for (int c = 0; c < decltype(nc)::value; c++) {
                    const double b0 = x0[8 * c], b1 = x1[8 * c];
#pragma unroll
                    for (int i = 0; i < MT; i++) {
                        dmma(acc[0][i][c], t[i].x, b0);
                        dmma(acc[1][i][c], t[i].y, b1);
                    }
                }
                x0 += dx;
                x1 += dx;
            };
            if constexpr (PF) {
                fetch(fa);
                for (int st = 0; st < nst; st += 2) {
                    if (st + 1 < nst) fetch(fb);
                    step(fa, std::integral_constant<int, NT>{});
                    if (st + 1 >= nst) break;
                    if (st + 2 < nst) fetch(fa);
                    step(fb, std::integral_constant<int, NT>{});
                }
            } else if (cw + 4 < n) {
                for (int st = 0; st < nst; st++) { fetch(fa); step(fa, std::integral_constant<int, NT>{}); }
            } else {   // the block's last columns: one group
                for (int st = 0; st < nst; st++) { fetch(fa); step(fa, std::integral_constant<int, 1>{}); }
            }
        } else {
            // u = sum qv*Z - i*qu*D ; v = sum -i*qu*Z - qv*D  (legmod.f90:338-341)
            const int sw = (r ^ 1) - r, dz = A.kc * rs;   // the partner column, and Z behind D
            const double sg = (r & 1) ? -1.0 : 1.0;       // -i*x: re <- im, im <- -re
            const double2 *uk = tk + (INV_QV - INV_QU) * A.tsz;
            double2 pa[MT], qa[MT], pb[MT], qb[MT];
            auto fetch = [&](double2 (&t)[MT], double2 (&u)[MT]) {
#pragma unroll
                for (int i = 0; i < MT; i++) { t[i] = tk[to[i]]; u[i] = uk[to[i]]; }
                tk += sstr;
                uk += sstr;
            };
            auto step = [&](const double2 (&t)[MT], const double2 (&u)[MT]) {
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    const double *x = p ? x1 : x0;
                    const double d = -x[0], z = x[dz], di = sg * x[sw], zi = sg * x[dz + sw];
                    // qu terms (P-type) and qv terms (Q-type) fall on opposite parities
#pragma unroll
                    for (int i = 0; i < MT; i++) {
                        const double tu = p ? t[i].y : t[i].x, tv = p ? u[i].y : u[i].x;
                        dmma(acc[p][i][0], tu, di);
                        dmma(acc[1 - p][i][0], tv, z);
                        dmma(acc[p][i][1], tu, zi);
                        dmma(acc[1 - p][i][1], tv, d);
                    }
                }
                x0 += dx;
                x1 += dx;
            };
            if constexpr (PF) {
                fetch(pa, qa);
                for (int st = 0; st < nst; st += 2) {
                    if (st + 1 < nst) fetch(pb, qb);
                    step(pa, qa);
                    if (st + 1 >= nst) break;
                    if (st + 2 < nst) fetch(pa, qa);
                    step(pb, qb);
                }
            } else {
                for (int st = 0; st < nst; st++) { fetch(pa, qa); step(pa, qa); }
            }
        }
    }
    if (!active) return;
    auto put = [&](T *o, long long f, int lat, double x, double y) {
        if constexpr (SET) {
            reinterpret_cast<C2<T> *>(o)[(size_t)m * A.nrows + f * nlat + lat] = C2<T>{(T)x, (T)y};
        } else {
            const size_t e = 2 * (f * A.fs + lat * A.ls + (long long)m * A.ms);
            const double sc = (A.roll && (m & 1) ? -A.scale : A.scale) * (A.rscale ? A.rscale[lat] : 1.0);
            o[e] = (T)(x * sc); o[e + 1] = (T)(y * sc);
        }
    };
    if (g < 2) {
        // qi is P-type (even n-m symmetric); qj is Q-type: its two sums swap roles
#pragma unroll
        for (int c = 0; c < NT; c++) {
            const int u = u0 + cw + 4 * c + q;
            if (cw + 4 * c + q >= n) continue;
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
            for (int i = 0; i < MT; i++) {
                const int j = j0 + 8 * i + r;
                if (j >= nlath) continue;
                const double *e = acc[0][i][c], *o = acc[1][i][c];
                const double nx = e[0] + o[0], ny = e[1] + o[1];
                const double sx = g == 0 ? e[0] - o[0] : o[0] - e[0], sy = g == 0 ? e[1] - o[1] : o[1] - e[1];
                put(A.oa, f, j, nx, ny);
                put(A.oa, f, nlat - 1 - j, sx, sy);
                if (gpmt) {   // gpmt = i*m*gp (plasim.f90:2425-2430), the field before gp
                    const double mm = (double)m;
                    put(A.oa, f - 1, j, -ny * mm, nx * mm);
                    put(A.oa, f - 1, nlat - 1 - j, -sy * mm, sx * mm);
                }
            }
        }
    } else if (cw + q < n) {
        const int u = u0 + cw + q;
        long long fu = u, fv = u;
        T *ov = A.ob;
        if constexpr (SET) {
            const int inst = u / A.L;
            fu = (long long)inst * (A.dset ? 4 * A.L + 1 : 6 * A.L + 3) + (u - inst * A.L);
            fv = fu + A.L;
            ov = A.oa;
        }
#pragma unroll
        for (int i = 0; i < MT; i++) {
            const int j = j0 + 8 * i + r;
            if (j >= nlath) continue;
#pragma unroll
            for (int x = 0; x < 2; x++) {
                const double *s = acc[0][i][x], *a = acc[1][i][x];
                put(x ? ov : A.oa, x ? fv : fu, j, s[0] + a[0], s[1] + a[1]);
                put(x ? ov : A.oa, x ? fv : fu, nlat - 1 - j, s[0] - a[0], s[1] - a[1]);
            }
        }
    }
}

// ------------------------------------------------------------------ forward
// the sets' operations on one level: gridpointa's mktend and qtend together,
// gridpointd's fc2sp of the temperature and humidity tendencies and uv2dv
enum { OP_LEVEL_A = 4, OP_LEVEL_D = 5 };

constexpr int FWD_THREADS = 192;   // least threads of a block
// latitude pairs per staged chunk (of esize-byte values).  Few inputs leave room for
// longer chunks, fewer waits for the slowest warp: gridpointd T127 L20 x8 238 -> 222 us;
// in FP64 the copies on their way would take a block per SM with them (T63: 31 -> 34 us)
__host__ __device__ constexpr int fwd_jc(int nin, size_t esize) { return nin <= 4 && esize == 4 ? 32 : 16; }
// staged (north, south) values per thread and chunk: 9 inputs x 4 units x 16 pairs over 192 threads
constexpr int FWD_ITEMS = 3;

template <typename T>
struct LegFwd {
    const double4 *tab;      // forward fragments, the four tables side by side (plan.cu k_layout_fwd)
    const int *foff;         // first fragment of each (m, parity)
    const int *woff;
    const double *filt;      // skgpsp(n)
    const T *in[6];          // single op: Fourier inputs; set: in[0] is the intermediate
    long long fs, ls, ms, nrows;
    T *out[3];               // single op: spectral outputs; set: out[0] is the set's output
    long long o_fs;          // spectral field stride (reals)
    double scale;            // single op: factor of the outputs
    int folded;              // the intermediate holds N+S, then N-S per field (rr_fwd_body)
    int nu, nt;              // units (levels x states) and unit tiles per wavenumber
    int nu1, nt1;            // gridpointa: ln ps tendencies (fc2sp) and their tiles
    int wb, nmb;             // warps along the modes of a block; mode blocks per wavenumber
    int L, nlat, nlath, ntp1;
    // float sets: the FP64 sums of the grid rows (null: none), whose zonal means give
    // the n = 0 coefficients of n0 fields, a warp each in the launch's last blocks
    const double *rowsum, *qc00;   // qc(0, lat) at stride qstride
    int qstride, nlon, n0;
};

template <int OP> struct FwdShape;
template <> struct FwdShape<OP_FC2SP> { static constexpr int nin = 1, nout = 1; static constexpr bool m = 0, q = 0; };
template <> struct FwdShape<OP_UV2DV> { static constexpr int nin = 2, nout = 2; static constexpr bool m = 1, q = 0; };
template <> struct FwdShape<OP_QTEND> { static constexpr int nin = 3, nout = 1; static constexpr bool m = 1, q = 0; };
template <> struct FwdShape<OP_MKTEND> { static constexpr int nin = 6, nout = 3; static constexpr bool m = 1, q = 1; };
template <> struct FwdShape<OP_LEVEL_A> { static constexpr int nin = 9, nout = 4; static constexpr bool m = 1, q = 1; };
template <> struct FwdShape<OP_LEVEL_D> { static constexpr int nin = 4, nout = 4; static constexpr bool m = 1, q = 0; };

// The four tables' fragments (qc, qe, qm, qq) of one tile
struct __align__(32) FwdFrag { double c, e, m, q; };

// Four latitude pairs' terms.  V(i, type, rot) is input i's fragment of the
// parity that P-type (0) or Q-type (1) tables pair with, or (rot) i times it
template <int OP, int NTILE, int MT, typename Val>
__device__ __forceinline__ void fwd_terms(double (*o)[FwdShape<OP>::nout][2], const FwdFrag (&t)[MT], Val V) {
    auto add = [&](int x, double FwdFrag::*a, double b) {
#pragma unroll
        for (int i = 0; i < NTILE; i++) dmma(o[i][x], t[i].*a, b);
    };
    if constexpr (OP == OP_FC2SP) {          // sp = sum qc*f  (legmod.f90:203-220)
        add(0, &FwdFrag::c, V(0, 0, 0));
    } else if constexpr (OP == OP_UV2DV) {   // d = -qe*v + i*qm*u, z = qe*u + i*qm*v  (:391-424)
        add(0, &FwdFrag::e, -V(1, 1, 0)); add(0, &FwdFrag::m, V(0, 0, 1));
        add(1, &FwdFrag::e, V(0, 1, 0));  add(1, &FwdFrag::m, V(1, 0, 1));
    } else if constexpr (OP == OP_QTEND) {   // q = qe*vq + qc*qn - i*qm*uq; in qn, uq, vq  (:466-497)
        add(0, &FwdFrag::e, V(2, 1, 0)); add(0, &FwdFrag::c, V(0, 0, 0)); add(0, &FwdFrag::m, -V(1, 0, 1));
    } else if constexpr (OP == OP_MKTEND || OP == OP_LEVEL_A) {
        // mktend (:555-602): d = qq*ke - qe*fv + i*qm*fu, t = qe*vt + qc*tn - i*qm*ut, z = qe*fu + i*qm*fv.
        // Inputs: mktend tn, fu, fv, ke, ut, vt; the level's tn, qn, ut, vt, fv (guz), fu (gvz), ke, uq, vq
        constexpr bool A = OP == OP_LEVEL_A;
        constexpr int TN = 0, FU = A ? 5 : 1, FV = A ? 4 : 2, KE = A ? 6 : 3, UT = A ? 2 : 4, VT = A ? 3 : 5;
        add(0, &FwdFrag::q, V(KE, 0, 0)); add(1, &FwdFrag::e, V(VT, 1, 0)); add(2, &FwdFrag::e, V(FU, 1, 0));
        if constexpr (A) add(3, &FwdFrag::e, V(8, 1, 0));                                        // qtend
        add(0, &FwdFrag::e, -V(FV, 1, 0)); add(1, &FwdFrag::c, V(TN, 0, 0)); add(2, &FwdFrag::m, V(FV, 0, 1));
        if constexpr (A) add(3, &FwdFrag::c, V(1, 0, 0));
        add(0, &FwdFrag::m, V(FU, 0, 1)); add(1, &FwdFrag::m, -V(UT, 0, 1));
        if constexpr (A) add(3, &FwdFrag::m, -V(7, 0, 1));
    } else {                                 // gridpointd: in t, u, v, q
        add(0, &FwdFrag::e, -V(2, 1, 0)); add(2, &FwdFrag::e, V(1, 1, 0));
        add(1, &FwdFrag::c, V(0, 0, 0)); add(3, &FwdFrag::c, V(3, 0, 0));
        add(0, &FwdFrag::m, V(1, 0, 1)); add(2, &FwdFrag::m, V(2, 0, 1));
    }
}

// A warp: MT tiles of 8 modes of one parity x the block's group of 4 units,
// every output.  The units' folded values (N+S, N-S) are staged jc latitude
// pairs at a time into one of two buffers while the other is read.
template <typename T, int OP, int MT, bool SET>
__device__ __forceinline__ void leg_fwd_block(const LegFwd<T> &A, double *sm, int m, int mblk, int u0, int n) {
    using S = FwdShape<OP>;
    constexpr int NIN = S::nin, NOUT = S::nout, rs = leg_stride(8);
    constexpr int FWD_JC = fwd_jc(NIN, sizeof(T)), SEL = FWD_JC * rs, BUF = NIN * 2 * SEL;
    static_assert(NIN * 4 * FWD_JC <= FWD_ITEMS * FWD_THREADS, "a chunk's values fit the threads' items");
    const int nlath = A.nlath, nlat = A.nlat, L = A.L;
    const int K = A.ntp1 - m, K0 = (K + 1) >> 1, K1 = K >> 1;
    const int n0 = (K0 + 8 * MT - 1) / (8 * MT), n1 = (K1 + 8 * MT - 1) / (8 * MT);   // warps per parity
    if (mblk * A.wb >= n0 + n1) return;   // block-uniform
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int wl = mblk * A.wb + warp;
    const bool active = warp < A.wb && wl < n0 + n1;
    const int p = wl >= n0 ? 1 : 0, kq = p ? K1 : K0, kt = (kq + 7) >> 3;   // tiles of this parity
    const int kt0 = (p ? wl - n0 : wl) * MT;
    double o[MT][NOUT][2];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int x = 0; x < NOUT; x++) o[i][x][0] = o[i][x][1] = 0.0;
    // this warp's table fragments, four latitude pairs a step (tiles past the last repeat it)
    const FwdFrag *tb = reinterpret_cast<const FwdFrag *>(A.tab);
    int to[MT];
#pragma unroll
    for (int i = 0; i < MT; i++) to[i] = active ? min(kt0 + i, kt - 1) * 32 : 0;
    if (active) tb += (size_t)A.foff[2 * m + p] * 32 + lane;
    const int tstr = kt * 32;
    auto fetch = [&](FwdFrag (&t)[MT], int ntile) {
#pragma unroll
        for (int i = 0; i < MT; i++) {
            if (i >= ntile) break;
            if constexpr (S::m || S::q)
                asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];"
                    : "=d"(t[i].c), "=d"(t[i].e), "=d"(t[i].m), "=d"(t[i].q) : "l"(tb + to[i]));
            else t[i].c = tb[to[i]].c;
        }
        tb += tstr;
    };
    // this thread's staged items (latitude pair jj of a chunk, unit, input i):
    // the chunk's northern and southern values arrive in `raw` by asynchronous
    // copies and the same thread folds them into the operand buffer
    C2<T> *raw = reinterpret_cast<C2<T> *>(sm + BUF) + threadIdx.x;
    const T *pn[FWD_ITEMS];
    int so[FWD_ITEMS], je[FWD_ITEMS];
    const long long ls = SET ? 1 : A.ls;
    const bool folded = SET && A.folded;
#pragma unroll
    for (int e = 0; e < FWD_ITEMS; e++) {
        const int idx = threadIdx.x + e * blockDim.x, jj = idx % FWD_JC, rr = idx / FWD_JC, ul = rr & 3, i = rr >> 2, u = u0 + ul;
        so[e] = i < NIN ? 2 * i * SEL + jj * rs + 2 * ul : -1;
        je[e] = i < NIN && ul < n ? jj : nlath;   // the chunk from j0 holds this pair while j0 + je < nlath
        pn[e] = A.in[0];
        if (je[e] >= nlath) continue;
        if constexpr (SET) {
            long long f;
            if constexpr (OP == OP_FC2SP) f = (long long)u * (9 * L + 1) + 7 * L;   // gvpp of state u
            else {
                const int inst = u / L, lev = u - inst * L;
                // gridpointa: tn qn ut vt uz vz ke [vpp] uq vq; gridpointd: t u v q
                f = (long long)inst * (OP == OP_LEVEL_A ? 9 * L + 1 : 4 * L) + i * L + lev + (OP == OP_LEVEL_A && i >= 7);
            }
            pn[e] = A.in[0] + 2 * ((size_t)m * A.nrows + f * nlat);
        } else {
            pn[e] = A.in[i] + 2 * (u * A.fs + (long long)m * A.ms);
        }
    }
    auto load = [&](int j0, int ring) {
#pragma unroll
        for (int e = 0; e < FWD_ITEMS; e++) {
            if (so[e] < 0 || j0 >= nlath) continue;
            const int j = j0 + je[e];
            C2<T> *d = raw + 2 * (ring * FWD_ITEMS + e) * blockDim.x;
            const bool ok = j < nlath;   // zeros otherwise
            cp_complex<SET>(d, pn[e] + (ok ? 2 * (j * ls) : 0), ok);
            cp_complex<SET>(d + blockDim.x, pn[e] + (ok ? 2 * ((folded ? nlath + j : nlat - 1 - j) * ls) : 0), ok);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto fold = [&](int ring) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
#pragma unroll
        for (int e = 0; e < FWD_ITEMS; e++) {
            if (so[e] < 0) continue;
            const C2<T> *v = raw + 2 * (ring * FWD_ITEMS + e) * blockDim.x;
            const C2<T> vn = v[0], vs = v[blockDim.x];
            const double nx = vn.x, ny = vn.y, sx = vs.x, sy = vs.y;
            *reinterpret_cast<Z2 *>(sm + so[e]) = folded ? Z2{nx, ny} : Z2{nx + sx, ny + sy};
            *reinterpret_cast<Z2 *>(sm + so[e] + SEL) = folded ? Z2{sx, sy} : Z2{nx - sx, ny - sy};
        }
    };
    const int nl4 = (nlath + 3) & ~3;
    constexpr bool PF = MT == 1;   // fetch a step ahead: few warps to hide the latency
    FwdFrag ta[MT], tn[MT];
    load(0, 0);
    load(FWD_JC, 1);
    if (PF && active) fetch(tn, 1);
    // P-type tables see the sum on even n-m and the difference on odd, Q-type
    // the reverse; the partner column (re <-> im) for i*x: re <- -im, im <- re
    const double *bp = sm + q * rs + r + (p ? SEL : 0), *bq = sm + q * rs + r + (p ? 0 : SEL);
    const int sw = (r ^ 1) - r;
    const double sg = (r & 1) ? 1.0 : -1.0;
    for (int j0 = 0, ring = 0; j0 < nlath; j0 += FWD_JC, ring ^= 1) {
        fold(ring);
        __syncthreads();
        load(j0 + 2 * FWD_JC, ring);   // two chunks ahead
        // the chunk's steps over the warp's tiles (the last warp of a parity may hold one of MT = 2)
        auto steps = [&](auto nt) {
            constexpr int NTILE = decltype(nt)::value;
            const double *xp = bp, *xq = bq;
            const int jn = min(FWD_JC, nl4 - j0);
#pragma unroll 1
            for (int jj = 0; jj < jn; jj += 4) {
                if constexpr (PF) {
#pragma unroll
                    for (int i = 0; i < MT; i++) ta[i] = tn[i];
                    if (j0 + jj + 4 < nl4) fetch(tn, NTILE);
                } else {
                    fetch(ta, NTILE);
                }
                fwd_terms<OP, NTILE>(o, ta, [&](int i, int type, int rot) {
                    const double *x = (type ? xq : xp) + 2 * i * SEL;
                    return rot ? sg * x[sw] : x[0];
                });
                xp += 4 * rs;
                xq += 4 * rs;
            }
        };
        if (active) {
            if (MT == 1 || kt0 + 1 >= kt) steps(std::integral_constant<int, 1>{});
            else steps(std::integral_constant<int, MT>{});
        }
        __syncthreads();
    }
    if (!active || q >= n) return;
    const int u = u0 + q, w0 = A.woff[m];
#pragma unroll
    for (int i = 0; i < MT; i++) {
        const int kk = (kt0 + i) * 8 + r, k = 2 * kk + p;
        if (kk >= kq) continue;
        const double f = SET ? A.filt[m + k] : A.filt[m + k] * A.scale;
#pragma unroll
        for (int x = 0; x < NOUT; x++) {
            if (SET && sizeof(T) == 4 && m + k == 0 && (OP == OP_FC2SP || (x & 1)) && A.rowsum) continue;   // leg_fwd_n0
            T *d;
            if constexpr (SET) {
                // sdf[L] stf[L] szf[L] sqf[L] (gridpointa: spf)
                if constexpr (OP == OP_FC2SP) d = A.out[0] + ((size_t)u * (4 * L + 1) + 4 * L) * A.o_fs;
                else {
                    const int inst = u / L, lev = u - inst * L;
                    d = A.out[0] + ((size_t)inst * (OP == OP_LEVEL_A ? 4 * L + 1 : 4 * L) + x * L + lev) * A.o_fs;
                }
            } else d = A.out[x] + (size_t)u * A.o_fs;
            d[2 * (w0 + k)] = (T)(o[i][x][0] * f);
            d[2 * (w0 + k) + 1] = (T)(o[i][x][1] * f);
        }
    }
}

// The global means of a mixed set (k_n0_fp64, whose order of sums this is, does the
// same where the rows' sums come from elsewhere).  As warps of the forward launch
// they cost nothing; the launch of their own took 5 us of the 57 of T42 L20.
template <int OP>
__device__ __forceinline__ void leg_fwd_n0(const LegFwd<float> &A, int w) {
    constexpr bool D = OP == OP_LEVEL_D;
    const int L = A.L, nf = D ? 2 * L : 2 * L + 1, lane = threadIdx.x & 31;
    if (w >= A.n0) return;
    const int inst = w / nf, f = w - inst * nf;
    const int fin = f < L ? f : f < 2 * L ? (D ? 2 * L + f : f) : 7 * L, fout = f < L ? L + f : f < 2 * L ? 2 * L + f : 4 * L;
    const double *rs = A.rowsum + ((long long)inst * (D ? 4 * L : 9 * L + 1) + fin) * A.nlat;
    double acc = 0.0;
    for (int lat = lane; lat < A.nlat; lat += 32) acc += A.qc00[(size_t)lat * A.qstride] * (rs[lat] / (double)A.nlon);
    for (int o = 1; o < 32; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    if (lane == 0) {
        float *o = A.out[0] + ((size_t)inst * (D ? 4 * L : 4 * L + 1) + fout) * A.o_fs;
        o[0] = (float)(acc * A.filt[0]);
        o[1] = 0.0f;
    }
}

template <typename T, int OP, int MT, bool SET, int NSEG>
__global__ void __launch_bounds__(384, MT == 1 ? 1 : 2) k_leg_fwd(const __grid_constant__ LegLaunch<LegFwd<T>, NSEG> P) {
    const int seg = P.find(blockIdx.x), blk = blockIdx.x - P.blk0[seg];
    const LegFwd<T> &A = P.seg[seg];
    extern __shared__ __align__(16) unsigned char smraw[];
    double *sm = reinterpret_cast<double *>(smraw);
    const int nt = A.nt + A.nt1, mb = blk / nt, ti = blk - mb * nt;
    const int m = mb / A.nmb, mblk = mb - m * A.nmb;
    pdl_trigger();
    pdl_wait();
    if constexpr (SET && sizeof(T) == 4) {
        if (m >= A.ntp1) {
            leg_fwd_n0<OP>(A, (blk - A.ntp1 * A.nmb * nt) * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5));
            return;
        }
    }
    if (ti < A.nt) {
        // where one tile per warp suffices (the larger half of the wavenumbers) every warp of the block works
        const int K = A.ntp1 - m, tiles = (((K + 1) >> 1) + 7) / 8 + ((K >> 1) + 7) / 8;
        if (MT > 1 && tiles <= A.wb) leg_fwd_block<T, OP, 1, SET>(A, sm, m, mblk, 4 * ti, min(4, A.nu - 4 * ti));
        else leg_fwd_block<T, OP, MT, SET>(A, sm, m, mblk, 4 * ti, min(4, A.nu - 4 * ti));
    } else if constexpr (OP == OP_LEVEL_A) {
        const int u0 = 4 * (ti - A.nt);
        leg_fwd_block<T, OP_FC2SP, MT, SET>(A, sm, m, mblk, u0, min(4, A.nu1 - u0));
    }
}

// ------------------------------------------------------------ host launchers
// Both directions take the larger warp tile where that still leaves LEG_WARPS
// warps (about 8 per SM; twice that for the inverse, whose larger tile does not
// fetch ahead), and the smaller one otherwise.  T42 L20, one state: inverse
// 13 us with the smaller tile, 16 with the larger; T85 L13 x3: 33 and 29.
constexpr long long LEG_WARPS = 1200;

// one segment to launch: its plan and its arguments, completed by the launcher
template <typename A> struct LegItem { exotx_plan p; A a; };

template <typename T, int MT, int NT, bool SET, int NSEG>
static exotx_status inv_launch_t(LegItem<LegInv<T>> *it, int n, cudaStream_t s) {
    LegLaunch<LegInv<T>, NSEG> P;
    P.nseg = n;
    size_t smem = 0;
    int threads = 0;
    long long blocks = 0;
    for (int i = 0; i < n; i++) {
        exotx_plan p = it[i].p;
        LegInv<T> &A = P.seg[i] = it[i].a;
        A.tab = reinterpret_cast<const double2 *>(p->d_inv64); A.ioff = p->d_ioff; A.tsz = p->inv_tsz;
        A.woff = p->d_woff; A.filt = p->d_fs64;
        A.nlat = p->nlat; A.nlath = p->nlath; A.ntl = (p->nlath + 7) / 8; A.ntp1 = p->ntp1; A.nrsp = 2 * p->ncsp;
        A.plavor = p->desc.plavor;
        const int lt = (p->nlath + 8 * MT - 1) / (8 * MT);   // latitude warps
        A.nlb = (lt + 3) / 4;
        A.wm = (lt + A.nlb - 1) / A.nlb;
        A.wn = 6 / A.wm;
        // the staged columns of a block: all modes at once where they fit the budget
        auto smem_of = [&](int kc, int wn) {
            const size_t one = (size_t)kc * leg_stride(8 * NT * wn), two = A.nu[2] ? 2 * (size_t)kc * leg_stride(8 * wn) : 0;
            return std::max(one, two) * sizeof(double);
        };
        A.kc = (p->ntp1 + 7) & ~7;
        while (A.wn > 1 && smem_of(A.kc, A.wn) > 72 * 1024) A.wn--;
        if (smem_of(A.kc, A.wn) > 96 * 1024) A.kc = 256;
        smem = std::max(smem, smem_of(A.kc, A.wn));
        threads = std::max(threads, 32 * A.wm * A.wn);
        const int cb[3] = {4 * NT * A.wn, 4 * NT * A.wn, 4 * A.wn};
        A.ntiles = 0;
        for (int g = 0; g < 3; g++) A.ntiles += A.nt[g] = (A.nu[g] + cb[g] - 1) / cb[g];
        P.blk0[i] = (int)blocks;
        blocks += (long long)(p->ntp1 + (!SET && A.mz > p->ntp1 ? 1 : 0)) * A.nlb * A.ntiles;
        if (blocks > 0x7fffffffLL) return EXOTX_BAD_DIM;
    }
    if (smem > LEG_MAXSMEM) return EXOTX_BAD_DIM;
    auto kern = k_leg_inv<T, MT, NT, SET, NSEG>;
    if (smem > 48 * 1024) EXOTX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LEG_MAXSMEM));
    cudaEvent_t ev = ktimer_start(EXOTX_K_LEG_INVERSE, s);
    EXOTX_CUDA(launch_pdl(kern, dim3((unsigned)blocks), dim3(threads), smem, s, P));
    EXOTX_CHECK_LAUNCH();
    ktimer_stop(EXOTX_K_LEG_INVERSE, s, ev);
    return EXOTX_OK;
}
template <typename T, bool SET, int NSEG>
static exotx_status inv_launch(LegItem<LegInv<T>> *it, int n, cudaStream_t s) {
    long long tiles = 0;
    for (int i = 0; i < n; i++)
        tiles += (long long)it[i].p->ntp1 * ((it[i].p->nlath + 7) / 8) *
                 ((it[i].a.nu[0] + it[i].a.nu[1]) / 4 + it[i].a.nu[2] / 2 + 1);
    return tiles / 4 >= 2 * LEG_WARPS ? inv_launch_t<T, 2, 2, SET, NSEG>(it, n, s) : inv_launch_t<T, 2, 1, SET, NSEG>(it, n, s);
}

template <typename T>
exotx_status leg_inverse_l(exotx_plan p, int op, const T *a, const T *b, T *oa, T *ob, int nlev,
                           long long fs, FourierLayout L, cudaStream_t s, double scale,
                           const double *rscale, bool roll) {
    if (nlev <= 0) return EXOTX_OK;
    if (op != OP_SP2FC && op != OP_SP2FCDMU && op != OP_DV2UV) return EXOTX_BAD_ARG;
    LegItem<LegInv<T>> it = {p, {}};
    LegInv<T> &A = it.a;
    A.a = a; A.a_fs = fs; A.b_off = b ? reinterpret_cast<const char *>(b) - reinterpret_cast<const char *>(a) : 0;
    A.oa = oa; A.ob = ob; A.fs = L.fs; A.ls = L.ls; A.ms = L.ms; A.mz = L.mz;
    A.scale = scale; A.rscale = rscale; A.roll = roll;
    A.nu[op == OP_SP2FC ? 0 : op == OP_SP2FCDMU ? 1 : 2] = nlev;
    return inv_launch<T, false, 1>(&it, 1, s);
}

template <typename T>
exotx_status leg_inverse_set(const LegSeg<T> *segs, int n, int dset, cudaStream_t s) {
    if (n < 1 || n > TC_MAXSEG) return EXOTX_BAD_ARG;
    LegItem<LegInv<T>> it[TC_MAXSEG];
    for (int i = 0; i < n; i++) {
        const LegSeg<T> &g = segs[i];
        it[i] = {g.p, {}};
        LegInv<T> &A = it[i].a;
        A.a = g.in;
        A.oa = g.out;
        A.L = g.L; A.dset = dset;
        A.nrows = (long long)g.ninst * (dset ? 4 * g.L + 1 : 6 * g.L + 3) * g.p->nlat;
        A.nu[0] = g.ninst * (dset ? 2 * g.L + 1 : 4 * g.L + 1);
        A.nu[1] = dset ? 0 : g.ninst;
        A.nu[2] = g.ninst * g.L;
    }
    if (n == 1) return inv_launch<T, true, 1>(it, n, s);
    if constexpr (sizeof(T) == 4) return inv_launch<T, true, TC_MAXSEG>(it, n, s);   // ensembles are float
    return EXOTX_BAD_ARG;
}

template <typename T, int OP, int MT, bool SET, int NSEG>
static exotx_status fwd_launch_t(LegItem<LegFwd<T>> *it, int n, cudaStream_t s) {
    LegLaunch<LegFwd<T>, NSEG> P;
    P.nseg = n;
    int threads = FWD_THREADS;
    long long blocks = 0;
    for (int i = 0; i < n; i++) {
        exotx_plan p = it[i].p;
        LegFwd<T> &A = P.seg[i] = it[i].a;
        A.tab = reinterpret_cast<const double4 *>(p->d_fwd64); A.foff = p->d_foff; A.woff = p->d_woff; A.filt = p->d_fg64;
        A.nlat = p->nlat; A.nlath = p->nlath; A.ntp1 = p->ntp1;
        const int K0 = (p->ntp1 + 1) / 2, K1 = p->ntp1 / 2;
        const int nw = (K0 + 8 * MT - 1) / (8 * MT) + (K1 + 8 * MT - 1) / (8 * MT);   // mode warps at m = 0
        A.nmb = (nw + 11) / 12;
        A.wb = (nw + A.nmb - 1) / A.nmb;
        threads = std::max(threads, 32 * A.wb);
        A.nt = (A.nu + 3) / 4;
        A.nt1 = (A.nu1 + 3) / 4;
        P.blk0[i] = (int)blocks;
        blocks += (long long)p->ntp1 * A.nmb * (A.nt + A.nt1);
        if (A.rowsum) {   // one segment, so threads is its own
            A.qc00 = p->d_qref + (size_t)2 * p->nlat * p->ncsp;   // qc(w = 0, lat) of the reference tables [t][lat][w]
            A.qstride = p->ncsp; A.nlon = p->nlon;
            blocks += (A.n0 + threads / 32 - 1) / (threads / 32);
        }
        if (blocks > 0x7fffffffLL) return EXOTX_BAD_DIM;
    }
    // one operand chunk and two chunks of copies on their way
    const size_t smem = (size_t)FwdShape<OP>::nin * 2 * fwd_jc(FwdShape<OP>::nin, sizeof(T)) * leg_stride(8) * sizeof(double) +
                        (size_t)FWD_ITEMS * 4 * threads * sizeof(C2<T>);
    if (smem > LEG_MAXSMEM) return EXOTX_BAD_DIM;
    auto kern = k_leg_fwd<T, OP, MT, SET, NSEG>;
    if (smem > 48 * 1024) EXOTX_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, LEG_MAXSMEM));
    cudaEvent_t ev = ktimer_start(EXOTX_K_LEG_FORWARD, s);
    EXOTX_CUDA(launch_pdl(kern, dim3((unsigned)blocks), dim3(threads), smem, s, P));
    EXOTX_CHECK_LAUNCH();
    ktimer_stop(EXOTX_K_LEG_FORWARD, s, ev);
    return EXOTX_OK;
}
template <typename T, int OP, bool SET, int NSEG>
static exotx_status fwd_launch(LegItem<LegFwd<T>> *it, int n, cudaStream_t s) {
    long long tiles = 0;
    for (int i = 0; i < n; i++) tiles += (long long)(it[i].p->ncsp / 8 + it[i].p->ntp1) * ((it[i].a.nu + 3) / 4);
    return tiles / 2 >= LEG_WARPS ? fwd_launch_t<T, OP, 2, SET, NSEG>(it, n, s) : fwd_launch_t<T, OP, 1, SET, NSEG>(it, n, s);
}

template <typename T>
exotx_status leg_forward_l(exotx_plan p, int op, const T *const *in, T *const *out, int nlev,
                           FourierLayout L, long long o_fs, cudaStream_t s, double scale) {
    if (nlev <= 0) return EXOTX_OK;
    LegItem<LegFwd<T>> it = {p, {}};
    LegFwd<T> &A = it.a;
    const int nin = op == OP_FC2SP ? 1 : op == OP_UV2DV ? 2 : op == OP_QTEND ? 3 : 6;
    const int nout = op == OP_MKTEND ? 3 : op == OP_UV2DV ? 2 : 1;
    for (int i = 0; i < nin; i++) A.in[i] = in[i];
    for (int i = 0; i < nout; i++) A.out[i] = out[i];
    A.fs = L.fs; A.ls = L.ls; A.ms = L.ms; A.o_fs = o_fs; A.scale = scale;
    A.nu = nlev;
    switch (op) {
        case OP_FC2SP: return fwd_launch<T, OP_FC2SP, false, 1>(&it, 1, s);
        case OP_UV2DV: return fwd_launch<T, OP_UV2DV, false, 1>(&it, 1, s);
        case OP_QTEND: return fwd_launch<T, OP_QTEND, false, 1>(&it, 1, s);
        case OP_MKTEND: return fwd_launch<T, OP_MKTEND, false, 1>(&it, 1, s);
    }
    return EXOTX_BAD_ARG;
}

template <typename T>
exotx_status leg_forward_set(const LegSeg<T> *segs, int n, int dset, cudaStream_t s) {
    if (n < 1 || n > TC_MAXSEG) return EXOTX_BAD_ARG;
    LegItem<LegFwd<T>> it[TC_MAXSEG];
    for (int i = 0; i < n; i++) {
        const LegSeg<T> &g = segs[i];
        it[i] = {g.p, {}};
        LegFwd<T> &A = it[i].a;
        A.in[0] = g.in;
        A.out[0] = g.out;
        A.o_fs = 2LL * g.p->ncsp;
        A.L = g.L;
        A.folded = g.folded;
        A.nrows = (long long)g.ninst * (dset ? 4 * g.L : 9 * g.L + 1) * g.p->nlat;
        A.nu = g.ninst * g.L;
        A.nu1 = dset ? 0 : g.ninst;
        A.rowsum = n == 1 ? g.rowsum : nullptr;
        A.n0 = g.ninst * (dset ? 2 * g.L : 2 * g.L + 1);
    }
    if (n > 1) {
        if constexpr (sizeof(T) == 4)
            if (!dset) return fwd_launch<T, OP_LEVEL_A, true, TC_MAXSEG>(it, n, s);
        return EXOTX_BAD_ARG;
    }
    return dset ? fwd_launch<T, OP_LEVEL_D, true, 1>(it, n, s) : fwd_launch<T, OP_LEVEL_A, true, 1>(it, n, s);
}

#define LEG_INSTANCES(T)                                                                                            \
    template exotx_status leg_inverse_l<T>(exotx_plan, int, const T *, const T *, T *, T *, int, long long,         \
                                           FourierLayout, cudaStream_t, double, const double *, bool);              \
    template exotx_status leg_forward_l<T>(exotx_plan, int, const T *const *, T *const *, int, FourierLayout,       \
                                           long long, cudaStream_t, double);                                        \
    template exotx_status leg_inverse_set<T>(const LegSeg<T> *, int, int, cudaStream_t);                            \
    template exotx_status leg_forward_set<T>(const LegSeg<T> *, int, int, cudaStream_t);
LEG_INSTANCES(double)
LEG_INSTANCES(float)

}  // namespace exotx
