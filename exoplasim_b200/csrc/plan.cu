// Plan construction: Gaussian grid and associated-Legendre tables built on
// the GPU in FP64, then laid out for the folded transform kernels.
//
// This file is compiled with -fmad=false so every product and sum is rounded
// separately, in the order the reference's 8-byte build evaluates them.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>
#include "exotx_internal.cuh"

namespace exotx {

static std::atomic<unsigned long long> g_launches{0};
void note_launch(unsigned n) { g_launches += n; }

// ---------------------------------------------------------------- inigau
// ql / qld follow gaussmod.f90:46-86; the Newton loop follows :23-37.
__device__ double ql_dev(int k, double p) {
    double z0 = acos(p), z1 = 1.0, z2 = 0.0, z3 = 0.0, z4;
    for (int j = k; j >= 0; j -= 2) {
        z3 = z1 * cos(z0 * j);
        z2 = z2 + z3;
        z4 = (double)((k - j + 1) * (k + j)) * 0.5;
        z1 = z1 * z4 / (z4 + (j - 1));
    }
    if (k % 2 == 0) z2 = z2 - 0.5 * z3;
    z0 = sqrt(2.0);
    for (int j = 1; j <= k; j++) z0 = z0 * sqrt(1.0 - 0.25 / (double)(j * j));
    return z0 * z2;
}

__device__ double qld_dev(int k, double p) {
    double z = p * ql_dev(k, p) - sqrt((k + k + 1.0) / (k + k - 1.0)) * ql_dev(k - 1, p);
    return (p * p - 1.0) / (k * z);
}

// one thread per northern latitude; writes both hemispheres
__global__ void k_inigau(int klat, double *pz0, double *pzw) {
    int jlat = 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (jlat > klat / 2) return;
    const double PI = 3.14159265358979;
    const double ZEPS = 1.0e-16;
    double z0 = PI / (2 * klat + 1);
    double z1 = 1.0 / (double)(klat * klat * 8);
    double z4 = 2.0 / (double)(klat * klat);
    double z2 = z0 * (2 * jlat - 0.5);
    z2 = cos(z2 + z1 / tan(z2));
    for (int jiter = 1; jiter <= 50; jiter++) {
        double z3 = ql_dev(klat, z2) * qld_dev(klat, z2);
        z2 = z2 - z3;
        if (fabs(z3) < ZEPS) break;
    }
    double z5 = ql_dev(klat - 1, z2) / sqrt(klat - 0.5);
    pz0[jlat - 1] = z2;
    pzw[jlat - 1] = z4 * (1.0 - z2 * z2) / (z5 * z5);
    pz0[klat - jlat] = -z2;
    pzw[klat - jlat] = pzw[jlat - 1];
}

// ---------------------------------------------------------------- legini
// One block per latitude.  Thread 0 runs the sectoral chain f1m/f2m over m
// (legmod.f90:68-72, sequential by construction); then each thread runs the
// n-recurrence of its own m columns (:82-88) and writes the eight derived
// tables (:99-116) in the reference layout q(NCSP,NLAT).
__global__ void k_legini(int nlat, int ntru, int ncsp, const int *woff, const double *sid,
                         const double *gwd, double *qref) {
    extern __shared__ __align__(16) double sh[];
    double *f1 = sh, *f2 = sh + (ntru + 1);
    int jlat = blockIdx.x;
    double zsin = sid[jlat], zgwd = gwd[jlat];
    double zcsq = 1.0 - zsin * zsin;
    double zgwdcsq = zgwd / zcsq;
    if (threadIdx.x == 0) {
        double f1m = sqrt(1.5), f2m = 0.0;
        f1[0] = f1m;
        f2[0] = 0.0;
        for (int m = 1; m <= ntru; m++) {
            f2m = -f1m * sqrt(zcsq / (double)(m + m));
            f1m = f2m * sqrt(m + m + 3.0);
            f1[m] = f1m;
            f2[m] = f2m;
        }
    }
    __syncthreads();
    size_t tsz = (size_t)ncsp * nlat;
    double *qi = qref, *qj = qref + tsz, *qc = qref + 2 * tsz, *qe = qref + 3 * tsz;
    double *qm = qref + 4 * tsz, *qq = qref + 5 * tsz, *qu = qref + 6 * tsz, *qv = qref + 7 * tsz;
    size_t row = (size_t)jlat * ncsp;
    for (int m = threadIdx.x; m <= ntru; m += blockDim.x) {
        int w0 = woff[m];
        double amsq = (double)(m * m);
        // P(m,m), P(m,m+1), Q(m,m)
        double pm2 = (m == 0) ? sqrt(0.5) : f2[m];
        double pzd_prev = (m == 0) ? 0.0 : -m * f2[m] * zsin;
        double pm1 = 0.0;
        bool has2 = (m < ntru);
        if (has2) pm1 = ((m == 0) ? sqrt(1.5) : f1[m]) * zsin;
        // store helper
        auto store = [&](int n, double zpli, double zpld) {
            size_t o = row + w0 + (n - m);
            double znn1 = 0.0;
            if (n > 0) znn1 = 1.0 / (double)(n * (n + 1));
            qi[o] = zpli;
            qj[o] = zpld;
            qc[o] = zpli * zgwd;
            qu[o] = zpli * znn1 * m;
            qv[o] = zpld * znn1;
            qe[o] = zpld * zgwdcsq;
            qq[o] = zpli * zgwdcsq * n * (n + 1) * 0.5;
            qm[o] = zpli * zgwdcsq * m;
        };
        if (!has2) {  // mode (NTRU,NTRU)
            double zpld = -ntru * zsin * pm2;
            store(m, pm2, zpld);
            continue;
        }
        // pm2 = P(n-2), pm1 = P(n-1); Q(n-2) pending in pzd_prev
        for (int n = m + 2; n <= ntru; n++) {
            double z1 = sqrt(((n - 1) * (n - 1) - amsq) / (double)(4 * (n - 1) * (n - 1) - 1));
            double z2 = zsin * pm1 - z1 * pm2;
            double p = z2 * sqrt((4 * n * n - 1) / (n * n - amsq));
            double qd = (1 - n) * z2 + n * z1 * pm2;   // Q(n-1)
            store(n - 2, pm2, pzd_prev);
            pzd_prev = qd;
            pm2 = pm1;
            pm1 = p;
        }
        // now pm2 = P(NTRU-1), pm1 = P(NTRU), pzd_prev = Q(NTRU-1)
        double z3 = sqrt((ntru * ntru - amsq) / (double)(4 * ntru * ntru - 1));
        double qlast = -ntru * zsin * pm1 + (ntru + ntru + 1) * pm2 * z3;
        store(ntru - 1, pm2, pzd_prev);
        store(ntru, pm1, qlast);
    }
}

// Both layouts hold the tables as the 8x4 operand fragments that the Legendre
// kernels' FP64 tensor-core instructions read (legendre_fp64mma.cu): 32 lanes,
// lane = 4 r + q for row r and column q, zeros past the last latitude or mode.
// One block per wavenumber (and parity).

// inverse, qi,qj,qu,qv (reference tables 0,1,6,7): table t, step s of 8 modes,
// latitude tile b: lane (r, q) holds latitude 8b + r of the modes n-m = 8s + 2q
// and 8s + 2q + 1 side by side; ioff[m] steps precede wavenumber m
__global__ void k_layout_inv(int nlat, int ntru, int ncsp, int nlath, const int *woff, const int *ioff, size_t tsz,
                             const double *qref, double2 *inv64) {
    const int m = blockIdx.x, K = ntru + 1 - m, ns = (K + 7) >> 3, ntl = (nlath + 7) >> 3;
    const size_t rsz = (size_t)ncsp * nlat;
    const int src[4] = {0, 1, 6, 7};
    for (int i = threadIdx.x; i < ns * ntl * 32; i += blockDim.x) {
        const int lane = i & 31, b = (i >> 5) % ntl, s = (i >> 5) / ntl;
        const int j = 8 * b + (lane >> 2), k = 8 * s + 2 * (lane & 3);
        for (int t = 0; t < 4; t++) {
            const double *q = qref + src[t] * rsz + (size_t)j * ncsp + woff[m];
            inv64[t * tsz + (size_t)ioff[m] * ntl * 32 + i] =
                make_double2(j < nlath && k < K ? q[k] : 0.0, j < nlath && k + 1 < K ? q[k + 1] : 0.0);
        }
    }
}

// forward, qc,qe,qm,qq (2,3,4,5) side by side: block (m, parity p of n-m), step
// s of 4 latitude pairs, tile b of 8 modes: lane (r, q) holds mode
// n-m = 2 (8b + r) + p at latitude 4s + q; foff[2m + p] fragments precede a block
__global__ void k_layout_fwd(int nlat, int ntru, int ncsp, int nlath, const int *woff, const int *foff,
                             const double *qref, double4 *fwd64) {
    const int m = blockIdx.x >> 1, p = blockIdx.x & 1, K = ntru + 1 - m, kq = (K + 1 - p) >> 1, kt = (kq + 7) >> 3;
    const size_t rsz = (size_t)ncsp * nlat;
    for (int i = threadIdx.x; i < ((nlath + 3) >> 2) * kt * 32; i += blockDim.x) {
        const int lane = i & 31, b = (i >> 5) % kt, s = (i >> 5) / kt;
        const int j = 4 * s + (lane & 3), kk = 8 * b + (lane >> 2);
        double4 v = make_double4(0.0, 0.0, 0.0, 0.0);
        if (j < nlath && kk < kq) {
            const double *q = qref + 2 * rsz + (size_t)j * ncsp + woff[m] + 2 * kk + p;
            v = make_double4(q[0], q[rsz], q[2 * rsz], q[3 * rsz]);
        }
        fwd64[(size_t)foff[blockIdx.x] * 32 + i] = v;
    }
}

// Filter coefficients (legmod.f90:124-155, pyfft.f90:152-156); index n-1.
static void host_filters(const exotx_grid_desc &d, int ntru, std::vector<double> &g,
                         std::vector<double> &s) {
    int ntp1 = ntru + 1;
    g.assign(ntp1, 1.0);
    s.assign(ntp1, 1.0);
    for (int n = 1; n <= ntp1; n++) {
        double gv = 1.0, sv = 1.0, rn = (double)n;
        if (d.pyfft_nfs >= 0) {
            // pyfft is compiled without -fdefault-real-8: 4-byte arithmetic
            float x = (float)n / (float)ntru;
            float x2 = x * x, x4 = x2 * x2, x8 = x4 * x4;
            float f = expf(-8.0f * x8);
            gv = sv = (double)(1 - d.pyfft_nfs) * 1.0 + (double)d.pyfft_nfs * (double)f;
        } else if (d.nfilter == 1) {
            gv = (1 - d.ngptfilter) * gv + d.ngptfilter * (1.0 - rn / ntp1);
            sv = (1 - d.nspvfilter) * sv + d.nspvfilter * (1.0 - rn / ntp1);
        } else if (d.nfilter == 2) {
            double e = exp(-d.filterkappa * pow(rn / ntru, d.nfilterexp));
            gv = (1 - d.ngptfilter) * gv + d.ngptfilter * e;
            sv = (1 - d.nspvfilter) * sv + d.nspvfilter * e;
        } else if (d.nfilter == 3) {
            double r = rn * (double)(n + 1) / (d.landhoskn0 * (d.landhoskn0 + 1));
            gv = (1 - d.ngptfilter) * gv + d.ngptfilter * exp(-(r * r));
            sv = (1 - d.nspvfilter) * sv + d.nspvfilter * exp(-(r * r));
        } else if (d.nfilter == 4) {
            double r = 1.0 - rn / ntp1;
            gv = (1 - d.ngptfilter) * gv + d.ngptfilter * (r * r);
            sv = (1 - d.nspvfilter) * sv + d.nspvfilter * (r * r);
        }
        g[n - 1] = gv;
        s[n - 1] = sv;
    }
}

// A buffer of at least `bytes` for a call on stream s.  One that no longer
// suffices goes back first, unless a captured graph uses it: that one stays until
// the plan goes, and the next is at least half as large again, where memory allows,
// so that such buffers together take at most twice the last one's bytes.
exotx_status ensure_work(exotx_plan p, size_t bytes, cudaStream_t s) {
    const bool cap = capturing(s);
    if (p->work_bytes < bytes) {
        const bool keep = p->d_work && (cap || p->work_held);
        if (p->d_work && !keep) {
            cudaDeviceSynchronize();
            cudaFree(p->d_work);
            p->d_work = nullptr;
            p->work_bytes = 0;
        }
        void *q = nullptr;
        size_t size = std::max(bytes, p->work_bytes + p->work_bytes / 2);
        cudaError_t e = cudaMalloc(&q, size);
        if (e == cudaErrorMemoryAllocation && size > bytes) {
            cudaGetLastError();
            e = cudaMalloc(&q, size = bytes);
        }
        if (e == cudaErrorMemoryAllocation) cudaGetLastError();   // reported by the status alone
        EXOTX_CUDA(e);
        if (keep) p->old_work.push_back(p->d_work);
        p->d_work = q;
        p->work_bytes = size;
        p->work_held = false;
    }
    p->work_held = p->work_held || cap;
    return EXOTX_OK;
}

static void plan_free(exotx_plan p) {
    if (!p) return;
    host_pipe_free(p);
    tc_free(p);
    cudaFree(p->d_woff);
    cudaFree(p->d_sid);
    cudaFree(p->d_gwd);
    cudaFree(p->d_qref);
    cudaFree(p->d_inv64);
    cudaFree(p->d_fwd64);
    cudaFree(p->d_ioff);
    cudaFree(p->d_foff);
    cudaFree(p->d_fs64);
    cudaFree(p->d_fg64);
    cudaFree(p->d_fs32);
    cudaFree(p->d_fg32);
    cudaFree(p->d_work);
    for (void *w : p->old_work) cudaFree(w);
    delete p;
}

}  // namespace exotx

using namespace exotx;

EXOTX_API unsigned long long exotx_launch_count(void) { return g_launches.load(); }

EXOTX_API const char *exotx_status_string(exotx_status st) {
    switch (st) {
        case EXOTX_OK: return "ok";
        case EXOTX_BAD_DIM: return "unsupported dimension";
        case EXOTX_UNSUPPORTED_N: return "FFT length not supported";
        case EXOTX_BAD_ARG: return "bad argument";
        case EXOTX_CUDA_ERR: return "CUDA error";
        case EXOTX_NO_MEM: return "out of device memory";
        case EXOTX_TIMEOUT: return "device wait timed out";
        case EXOTX_NOT_BUILT: return "path not available in this build";
    }
    return "unknown status";
}

EXOTX_API exotx_status exotx_grid_desc_default(int nlat, exotx_grid_desc *d) {
    if (!d) return EXOTX_BAD_ARG;
    memset(d, 0, sizeof(*d));
    d->nlat = nlat;
    d->nfilter = 0;
    d->ngptfilter = 0;
    d->nspvfilter = 0;
    d->landhoskn0 = 15.0;
    d->filterkappa = 8.0;
    d->nfilterexp = 8;
    d->pyfft_nfs = -1;
    d->plavor = 1.63299310207;  // EZ = 1/sqrt(3/8), plasimmod.f90:118,227
    return EXOTX_OK;
}

EXOTX_API exotx_status exotx_inigau(int nlat, double *sid, double *gwd, exotx_stream s) {
    if (nlat < 2 || nlat % 2 || !sid || !gwd) return EXOTX_BAD_ARG;
    int nh = nlat / 2;
    k_inigau<<<(nh + 63) / 64, 64, 0, (cudaStream_t)s>>>(nlat, sid, gwd);
    EXOTX_CHECK_LAUNCH();
    return EXOTX_OK;
}

EXOTX_API exotx_status exotx_plan_create(const exotx_grid_desc *d, exotx_plan *out) {
    if (!d || !out) return EXOTX_BAD_ARG;
    *out = nullptr;
    int nlat = d->nlat;
    // NLAT even, NLON = 2 NLAT a supported FFT length, NTRU >= 1
    if (nlat < 4 || nlat % 2 || nlat > 2048) return EXOTX_BAD_DIM;
    if (!exotx_fft_supported(2 * nlat)) return EXOTX_UNSUPPORTED_N;
    if (d->nfilter < 0 || d->nfilter > 4 || d->pyfft_nfs > 1) return EXOTX_BAD_ARG;
    exotx_plan p = new exotx_plan_s();
    p->desc = *d;
    p->nlat = nlat;
    p->nlon = 2 * nlat;
    p->ntru = (p->nlon - 1) / 3;
    p->ntp1 = p->ntru + 1;
    p->ncsp = p->ntp1 * (p->ntru + 2) / 2;
    p->nlath = nlat / 2;
    p->kmax = p->ntp1;
    int ntp1 = p->ntp1, ncsp = p->ncsp, nlath = p->nlath;
    std::vector<int> woff(ntp1 + 1);
    woff[0] = 0;
    for (int m = 0; m < ntp1; m++) woff[m + 1] = woff[m] + (ntp1 - m);
    std::vector<double> g, sv;
    host_filters(*d, p->ntru, g, sv);
    std::vector<float> g32(g.begin(), g.end()), s32(sv.begin(), sv.end());
    size_t tsz = (size_t)ncsp * nlat;
    std::vector<int> ioff(ntp1), foff(2 * ntp1);
    int nstep = 0, nfrag = 0;
    for (int m = 0; m < ntp1; m++) {
        ioff[m] = nstep;
        nstep += (ntp1 - m + 7) / 8;
        for (int q = 0; q < 2; q++) {
            foff[2 * m + q] = nfrag;
            nfrag += (nlath + 3) / 4 * (((ntp1 - m + 1 - q) / 2 + 7) / 8);
        }
    }
    p->inv_tsz = (size_t)nstep * ((nlath + 7) / 8) * 32;
    exotx_status st = EXOTX_OK;
#define PALLOC(ptr, bytes)                                           \
    do {                                                             \
        if (cudaMalloc(&(ptr), (bytes)) != cudaSuccess) {            \
            st = EXOTX_NO_MEM;                                       \
            goto fail;                                               \
        }                                                            \
    } while (0)
    PALLOC(p->d_woff, sizeof(int) * (ntp1 + 1));
    PALLOC(p->d_sid, sizeof(double) * nlat);
    PALLOC(p->d_gwd, sizeof(double) * nlat);
    PALLOC(p->d_qref, sizeof(double) * 8 * tsz);
    PALLOC(p->d_inv64, sizeof(double2) * 4 * p->inv_tsz);
    PALLOC(p->d_fwd64, sizeof(double4) * 32 * (size_t)nfrag);
    PALLOC(p->d_ioff, sizeof(int) * ntp1);
    PALLOC(p->d_foff, sizeof(int) * 2 * ntp1);
    PALLOC(p->d_fs64, sizeof(double) * ntp1);
    PALLOC(p->d_fg64, sizeof(double) * ntp1);
    PALLOC(p->d_fs32, sizeof(float) * ntp1);
    PALLOC(p->d_fg32, sizeof(float) * ntp1);
#undef PALLOC
    {
        cudaStream_t s = 0;
        if (cudaMemcpy(p->d_ioff, ioff.data(), sizeof(int) * ntp1, cudaMemcpyHostToDevice) ||
            cudaMemcpy(p->d_foff, foff.data(), sizeof(int) * 2 * ntp1, cudaMemcpyHostToDevice) ||
            cudaMemcpy(p->d_woff, woff.data(), sizeof(int) * (ntp1 + 1), cudaMemcpyHostToDevice) ||
            cudaMemcpy(p->d_fg64, g.data(), sizeof(double) * ntp1, cudaMemcpyHostToDevice) ||
            cudaMemcpy(p->d_fs64, sv.data(), sizeof(double) * ntp1, cudaMemcpyHostToDevice) ||
            cudaMemcpy(p->d_fg32, g32.data(), sizeof(float) * ntp1, cudaMemcpyHostToDevice) ||
            cudaMemcpy(p->d_fs32, s32.data(), sizeof(float) * ntp1, cudaMemcpyHostToDevice)) {
            st = EXOTX_CUDA_ERR;
            goto fail;
        }
        k_inigau<<<(nlath + 63) / 64, 64, 0, s>>>(nlat, p->d_sid, p->d_gwd);
        note_launch();
        k_legini<<<nlat, 128, sizeof(double) * 2 * ntp1, s>>>(nlat, p->ntru, ncsp, p->d_woff, p->d_sid,
                                                              p->d_gwd, p->d_qref);
        note_launch();
        k_layout_inv<<<ntp1, 256, 0, s>>>(nlat, p->ntru, ncsp, nlath, p->d_woff, p->d_ioff, p->inv_tsz, p->d_qref,
                                          reinterpret_cast<double2 *>(p->d_inv64));
        note_launch();
        k_layout_fwd<<<2 * ntp1, 256, 0, s>>>(nlat, p->ntru, ncsp, nlath, p->d_woff, p->d_foff, p->d_qref,
                                              reinterpret_cast<double4 *>(p->d_fwd64));
        note_launch();
        if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess) {
            st = EXOTX_CUDA_ERR;
            goto fail;
        }
    }
    *out = p;
    return EXOTX_OK;
fail:
    plan_free(p);
    return st;
}

EXOTX_API exotx_status exotx_plan_destroy(exotx_plan p) {
    if (!p) return EXOTX_BAD_ARG;
    cudaDeviceSynchronize();
    plan_free(p);
    return EXOTX_OK;
}

EXOTX_API exotx_status exotx_plan_dims(exotx_plan p, int *nlat, int *nlon, int *ntru, int *ncsp) {
    if (!p) return EXOTX_BAD_ARG;
    if (nlat) *nlat = p->nlat;
    if (nlon) *nlon = p->nlon;
    if (ntru) *ntru = p->ntru;
    if (ncsp) *ncsp = p->ncsp;
    return EXOTX_OK;
}

EXOTX_API exotx_status exotx_plan_gauss(exotx_plan p, double *sid, double *gwd) {
    if (!p || !sid || !gwd) return EXOTX_BAD_ARG;
    EXOTX_CUDA(cudaMemcpy(sid, p->d_sid, sizeof(double) * p->nlat, cudaMemcpyDeviceToHost));
    EXOTX_CUDA(cudaMemcpy(gwd, p->d_gwd, sizeof(double) * p->nlat, cudaMemcpyDeviceToHost));
    return EXOTX_OK;
}

EXOTX_API exotx_status exotx_plan_table(exotx_plan p, int which, double *out) {
    if (!p || !out || which < 0 || which > 7) return EXOTX_BAD_ARG;
    size_t tsz = (size_t)p->ncsp * p->nlat;
    EXOTX_CUDA(cudaMemcpy(out, p->d_qref + which * tsz, sizeof(double) * tsz, cudaMemcpyDeviceToHost));
    return EXOTX_OK;
}

EXOTX_API exotx_status exotx_plan_tune(exotx_plan p, int key, long long value) {
    if (!p || value < 0) return EXOTX_BAD_ARG;
    switch (key) {
        case EXOTX_TUNE_CHUNK_INV: p->chunk_inv = (size_t)value; return EXOTX_OK;
        case EXOTX_TUNE_CHUNK_FWD: p->chunk_fwd = (size_t)value; return EXOTX_OK;
        case EXOTX_TUNE_INV_HALF:
            if (value > 1) return EXOTX_BAD_ARG;
            if (p->inv_half_ok != (int)value) {
                // the cached inverse job lists follow the mode: rebuild them
                // (after the work that may still read them)
                EXOTX_CUDA(cudaDeviceSynchronize());
                tc_free(p);
                p->inv_half_ok = (int)value;
            }
            return EXOTX_OK;
    }
    return EXOTX_BAD_ARG;
}
