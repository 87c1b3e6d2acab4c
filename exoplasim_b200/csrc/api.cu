// C-ABI entry points of the transform core (see include/exotx.h).
#include <algorithm>
#include <cstring>
#include "exotx_internal.cuh"

namespace exotx {

// reference layout fc(2,NLON/2,NLAT,nlev)
static FourierLayout ref_layout(exotx_plan p) {
    return FourierLayout{(long long)p->nlat * (p->nlon / 2), p->nlon / 2, 1, p->nlon / 2};
}
static bool prec_ok(int prec) { return prec == EXOTX_FP64 || prec == EXOTX_FP32 || prec == EXOTX_MIXED; }

// The FP64 and FP32 sets over ninst states: one Legendre and one FFT launch per
// chunk of states.  A chunk's m-major intermediate is held to PLAIN_CHUNK bytes
// (at least one state), so that it is still in L2 when the next kernel reads it
// and the plan's work buffer stays small.
constexpr size_t PLAIN_CHUNK = (size_t)96 << 20;
// Under capture, where nothing can be allocated, a chunk is what the buffer at
// hand takes; where memory is short it is one state.
static exotx_status plain_work(exotx_plan p, size_t per_inst, int ninst, cudaStream_t s, int *chunk) {
    int c = (int)std::min<size_t>((size_t)ninst, std::max<size_t>(1, PLAIN_CHUNK / per_inst));
    if (p->work_bytes < per_inst * c && capturing(s)) c = (int)std::max<size_t>(1, p->work_bytes / per_inst);
    exotx_status st = ensure_work(p, per_inst * c, s);
    if (st == EXOTX_NO_MEM && c > 1) st = ensure_work(p, per_inst * (c = 1), s);
    *chunk = c;
    return st;
}

// invlega / invlegd (legmod.f90:635-677) and fc2gp of every field: gridpointa
// (dset = 0, plasim.f90:2396-2440) spin (4L+1 fields) -> gpout (6L+3),
// gridpointd (dset = 1, :3142-3149) -> 4L+1
template <typename T>
static exotx_status inverse_set_plain(exotx_plan p, const T *spin, T *gpout, int L, int ninst, int dset,
                                     cudaStream_t s) {
    const size_t nrsp = 2 * (size_t)p->ncsp, nhor = (size_t)p->nlat * p->nlon;
    const int nfo = dset ? 4 * L + 1 : 6 * L + 3;
    const size_t per_inst = sizeof(T) * 2 * (size_t)nfo * p->nlat * p->ntp1;
    int chunk;
    EXOTX_TRY(plain_work(p, per_inst, ninst, s, &chunk));
    T *w = (T *)p->d_work;
    for (int i0 = 0; i0 < ninst; i0 += chunk) {
        const int ni = std::min(chunk, ninst - i0);
        const long long nrows = (long long)ni * nfo * p->nlat;
        const LegSeg<T> g = {p, L, ni, spin + i0 * (4 * L + 1) * nrsp, w, false};
        EXOTX_TRY(leg_inverse_set<T>(&g, 1, dset, s));
        EXOTX_TRY(fft_inverse_l<T>(w, gpout + i0 * nfo * nhor, p->nlon, nrows, p->ntp1, 1, nrows, s));
    }
    return EXOTX_OK;
}

// gp2fc of every field, then mktend, qtend and fc2sp(gvpp) (gridpointa,
// plasim.f90:2462-2486) or fc2sp and uv2dv (gridpointd, :3415-3428)
template <typename T>
static exotx_status forward_set_plain(exotx_plan p, const T *gpin, T *spout, int L, int ninst, int dset,
                                     cudaStream_t s) {
    const size_t nrsp = 2 * (size_t)p->ncsp, nhor = (size_t)p->nlat * p->nlon;
    const int nfi = dset ? 4 * L : 9 * L + 1, nfo = dset ? 4 * L : 4 * L + 1;
    const size_t per_inst = sizeof(T) * 2 * (size_t)nfi * p->nlat * p->ntp1;
    int chunk;
    EXOTX_TRY(plain_work(p, per_inst, ninst, s, &chunk));
    T *w = (T *)p->d_work;
    for (int i0 = 0; i0 < ninst; i0 += chunk) {
        const int ni = std::min(chunk, ninst - i0);
        const long long nrows = (long long)ni * nfi * p->nlat;
        EXOTX_TRY(fft_forward_l<T>(gpin + i0 * nfi * nhor, w, p->nlon, nrows, p->ntp1, 1, nrows, s));
        const LegSeg<T> g = {p, L, ni, w, spout + i0 * nfo * nrsp, false};
        EXOTX_TRY(leg_forward_set<T>(&g, 1, dset, s));
    }
    return EXOTX_OK;
}

}  // namespace exotx

using namespace exotx;

#define PLAN_PREC_CHECK(p, prec)                      \
    do {                                              \
        if (!(p) || !prec_ok(prec)) return EXOTX_BAD_ARG; \
    } while (0)

template <typename Fn>
static exotx_status by_prec(int prec, Fn fn) {
    if (prec == EXOTX_FP64) return fn((double *)nullptr);
    return fn((float *)nullptr);
}

static exotx_status inv_api(exotx_plan p, int prec, int op, const void *a, const void *b, void *oa, void *ob,
                            int nlev, exotx_stream s) {
    PLAN_PREC_CHECK(p, prec);
    if (nlev == 0) return EXOTX_OK;
    if (!a || !oa || nlev < 0 || ((op == OP_DV2UV) && (!b || !ob))) return EXOTX_BAD_ARG;
    const long long nrsp = 2LL * p->ncsp;
    FourierLayout F = ref_layout(p);
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        return leg_inverse_l<T>(p, op, (const T *)a, (const T *)b, (T *)oa, (T *)ob, nlev, nrsp, F,
                                (cudaStream_t)s);
    });
}

EXOTX_API exotx_status exotx_sp2fc(exotx_plan p, int prec, const void *sp, void *fc, int nlev, exotx_stream s) {
    return inv_api(p, prec, OP_SP2FC, sp, nullptr, fc, nullptr, nlev, s);
}
EXOTX_API exotx_status exotx_sp2fcdmu(exotx_plan p, int prec, const void *sp, void *fc, int nlev,
                                      exotx_stream s) {
    return inv_api(p, prec, OP_SP2FCDMU, sp, nullptr, fc, nullptr, nlev, s);
}
EXOTX_API exotx_status exotx_dv2uv(exotx_plan p, int prec, const void *pd, const void *pz, void *pu, void *pv,
                                   int nlev, exotx_stream s) {
    return inv_api(p, prec, OP_DV2UV, pd, pz, pu, pv, nlev, s);
}

static exotx_status fwd_api(exotx_plan p, int prec, int op, const void *const *in, int nin, void *const *out,
                            int nout, int nlev, exotx_stream s) {
    PLAN_PREC_CHECK(p, prec);
    if (nlev < 0) return EXOTX_BAD_ARG;
    if (nlev == 0) return EXOTX_OK;
    for (int i = 0; i < nin; i++) if (!in[i]) return EXOTX_BAD_ARG;
    for (int i = 0; i < nout; i++) if (!out[i]) return EXOTX_BAD_ARG;
    const long long nrsp = 2LL * p->ncsp;
    FourierLayout F = ref_layout(p);
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        const T *ii[6] = {};
        T *oo[3] = {};
        for (int i = 0; i < nin; i++) ii[i] = (const T *)in[i];
        for (int i = 0; i < nout; i++) oo[i] = (T *)out[i];
        return leg_forward_l<T>(p, op, ii, oo, nlev, F, nrsp, (cudaStream_t)s);
    });
}

EXOTX_API exotx_status exotx_fc2sp(exotx_plan p, int prec, const void *fc, void *sp, int nlev, exotx_stream s) {
    const void *in[1] = {fc};
    void *out[1] = {sp};
    return fwd_api(p, prec, OP_FC2SP, in, 1, out, 1, nlev, s);
}
EXOTX_API exotx_status exotx_uv2dv(exotx_plan p, int prec, const void *pu, const void *pv, void *pd, void *pz,
                                   int nlev, exotx_stream s) {
    const void *in[2] = {pu, pv};
    void *out[2] = {pd, pz};
    return fwd_api(p, prec, OP_UV2DV, in, 2, out, 2, nlev, s);
}
EXOTX_API exotx_status exotx_mktend(exotx_plan p, int prec, void *d, void *t, void *z, const void *tn,
                                    const void *fu, const void *fv, const void *ke, const void *ut,
                                    const void *vt, int nlev, exotx_stream s) {
    const void *in[6] = {tn, fu, fv, ke, ut, vt};
    void *out[3] = {d, t, z};
    return fwd_api(p, prec, OP_MKTEND, in, 6, out, 3, nlev, s);
}
EXOTX_API exotx_status exotx_qtend(exotx_plan p, int prec, void *q, const void *qn, const void *uq,
                                   const void *vq, int nlev, exotx_stream s) {
    const void *in[3] = {qn, uq, vq};
    void *out[1] = {q};
    return fwd_api(p, prec, OP_QTEND, in, 3, out, 1, nlev, s);
}

EXOTX_API exotx_status exotx_gp2fc(int prec, void *a, int n, int lot, exotx_stream s) {
    if (lot == 0 && prec_ok(prec) && exotx_fft_supported(n)) return EXOTX_OK;
    if (!a || lot < 0 || !prec_ok(prec)) return EXOTX_BAD_ARG;
    if (!exotx_fft_supported(n)) return EXOTX_UNSUPPORTED_N;
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        return fft_forward_l<T>((const T *)a, (T *)a, n, lot, n / 2, n / 2, 1, (cudaStream_t)s);
    });
}
EXOTX_API exotx_status exotx_fc2gp(int prec, void *a, int n, int lot, exotx_stream s) {
    if (lot == 0 && prec_ok(prec) && exotx_fft_supported(n)) return EXOTX_OK;
    if (!a || lot < 0 || !prec_ok(prec)) return EXOTX_BAD_ARG;
    if (!exotx_fft_supported(n)) return EXOTX_UNSUPPORTED_N;
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        return fft_inverse_l<T>((const T *)a, (T *)a, n, lot, n / 2, n / 2, 1, (cudaStream_t)s);
    });
}

// An output file's transforms: Legendre and FFT through an m-major intermediate
// in the caller's work array.  The scaling and the half-turn of the longitudes
// are factors of the Fourier coefficients (sqrt(2), (-1)^m), where separate calls
// made the reference's row-major Fourier layout with its zero tails and passed
// over the grid for each: a T42 L10 file's temperature, wind and cloud cover took
// 25 launches and 280 us, now 7 and 118, bound by the calls on the host.
EXOTX_API exotx_status exotx_sp2gp_scaled(exotx_plan p, int prec, const void *sp, void *gp, int nlev, double scale,
                                          int roll, void *work, exotx_stream s) {
    if (!p || (prec != EXOTX_FP64 && prec != EXOTX_FP32) || nlev < 0) return EXOTX_BAD_ARG;
    if (nlev == 0) return EXOTX_OK;
    if (!sp || !gp || !work) return EXOTX_BAD_ARG;
    if (!exotx_fft_supported(p->nlon)) return EXOTX_UNSUPPORTED_N;
    const long long nrsp = 2LL * p->ncsp, rows = (long long)nlev * p->nlat;
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        EXOTX_TRY(leg_inverse_l<T>(p, OP_SP2FC, (const T *)sp, nullptr, (T *)work, nullptr, nlev, nrsp,
                                   FourierLayout{p->nlat, 1, rows, p->ntp1}, (cudaStream_t)s, scale, nullptr, roll != 0));
        return fft_inverse_l<T>((const T *)work, (T *)gp, p->nlon, rows, p->ntp1, 1, rows, (cudaStream_t)s);
    });
}
EXOTX_API exotx_status exotx_dv2gp_scaled(exotx_plan p, int prec, const void *pd, const void *pz, void *gu, void *gv,
                                          int nlev, const double *rscale, double scale, int roll, void *work,
                                          exotx_stream s) {
    if (!p || (prec != EXOTX_FP64 && prec != EXOTX_FP32) || nlev < 0) return EXOTX_BAD_ARG;
    if (nlev == 0) return EXOTX_OK;
    if (!pd || !pz || !gu || !gv || !work) return EXOTX_BAD_ARG;
    if (!exotx_fft_supported(p->nlon)) return EXOTX_UNSUPPORTED_N;
    const long long nrsp = 2LL * p->ncsp, rows = (long long)nlev * p->nlat;
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        T *wu = (T *)work, *wv = wu + 2 * rows * p->ntp1;
        EXOTX_TRY(leg_inverse_l<T>(p, OP_DV2UV, (const T *)pd, (const T *)pz, wu, wv, nlev, nrsp,
                                   FourierLayout{p->nlat, 1, rows, p->ntp1}, (cudaStream_t)s, scale, rscale, roll != 0));
        EXOTX_TRY(fft_inverse_l<T>(wu, (T *)gu, p->nlon, rows, p->ntp1, 1, rows, (cudaStream_t)s));
        return fft_inverse_l<T>(wv, (T *)gv, p->nlon, rows, p->ntp1, 1, rows, (cudaStream_t)s);
    });
}
EXOTX_API exotx_status exotx_gp2sp_scaled(exotx_plan p, int prec, const void *gp, void *sp, int nlev, double scale,
                                          void *work, exotx_stream s) {
    if (!p || (prec != EXOTX_FP64 && prec != EXOTX_FP32) || nlev < 0) return EXOTX_BAD_ARG;
    if (nlev == 0) return EXOTX_OK;
    if (!sp || !gp || !work) return EXOTX_BAD_ARG;
    if (!exotx_fft_supported(p->nlon)) return EXOTX_UNSUPPORTED_N;
    const long long rows = (long long)nlev * p->nlat;
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        EXOTX_TRY(fft_forward_l<T>((const T *)gp, (T *)work, p->nlon, rows, p->ntp1, 1, rows, (cudaStream_t)s));
        const T *in[1] = {(const T *)work};
        T *out[1] = {(T *)sp};
        return leg_forward_l<T>(p, OP_FC2SP, in, out, nlev, FourierLayout{p->nlat, 1, rows, p->ntp1}, 2LL * p->ncsp,
                                (cudaStream_t)s, scale);
    });
}

// both forms of the inverse (forward) set: dset = 0 gridpointa, 1 gridpointd
static exotx_status inverse_set_api(exotx_plan p, int prec, const void *spin, void *gpout, int nlev, int ninst,
                                    int dset, exotx_stream s) {
    PLAN_PREC_CHECK(p, prec);
    if (ninst == 0) return EXOTX_OK;
    if (!spin || !gpout || nlev < 1 || ninst < 0) return EXOTX_BAD_ARG;
    if (prec == EXOTX_MIXED)
        return (dset ? tc_inverse_batch_d : tc_inverse_batch)(p, (const float *)spin, (float *)gpout, nlev, ninst,
                                                               (cudaStream_t)s);
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        return inverse_set_plain<T>(p, (const T *)spin, (T *)gpout, nlev, ninst, dset, (cudaStream_t)s);
    });
}
static exotx_status forward_set_api(exotx_plan p, int prec, const void *gpin, void *spout, int nlev, int ninst,
                                    int dset, exotx_stream s) {
    PLAN_PREC_CHECK(p, prec);
    if (ninst == 0) return EXOTX_OK;
    if (!gpin || !spout || nlev < 1 || ninst < 0) return EXOTX_BAD_ARG;
    if (prec == EXOTX_MIXED)
        return (dset ? tc_forward_batch_d : tc_forward_batch)(p, (const float *)gpin, (float *)spout, nlev, ninst,
                                                               (cudaStream_t)s);
    return by_prec(prec, [&](auto tag) {
        using T = std::remove_pointer_t<decltype(tag)>;
        return forward_set_plain<T>(p, (const T *)gpin, (T *)spout, nlev, ninst, dset, (cudaStream_t)s);
    });
}

EXOTX_API exotx_status exotx_inverse_set(exotx_plan p, int prec, const void *spin, void *gpout, int nlev,
                                         exotx_stream s) {
    return inverse_set_api(p, prec, spin, gpout, nlev, 1, 0, s);
}
EXOTX_API exotx_status exotx_forward_set(exotx_plan p, int prec, const void *gpin, void *spout, int nlev,
                                         exotx_stream s) {
    return forward_set_api(p, prec, gpin, spout, nlev, 1, 0, s);
}
EXOTX_API exotx_status exotx_inverse_set_batch(exotx_plan p, int prec, const void *spin, void *gpout, int nlev,
                                               int ninst, exotx_stream s) {
    return inverse_set_api(p, prec, spin, gpout, nlev, ninst, 0, s);
}
EXOTX_API exotx_status exotx_forward_set_batch(exotx_plan p, int prec, const void *gpin, void *spout, int nlev,
                                               int ninst, exotx_stream s) {
    return forward_set_api(p, prec, gpin, spout, nlev, ninst, 0, s);
}
EXOTX_API exotx_status exotx_inverse_set_d(exotx_plan p, int prec, const void *spin, void *gpout, int nlev,
                                           exotx_stream s) {
    return inverse_set_api(p, prec, spin, gpout, nlev, 1, 1, s);
}
EXOTX_API exotx_status exotx_forward_set_d(exotx_plan p, int prec, const void *gpin, void *spout, int nlev,
                                           exotx_stream s) {
    return forward_set_api(p, prec, gpin, spout, nlev, 1, 1, s);
}
EXOTX_API exotx_status exotx_inverse_set_d_batch(exotx_plan p, int prec, const void *spin, void *gpout, int nlev,
                                                 int ninst, exotx_stream s) {
    return inverse_set_api(p, prec, spin, gpout, nlev, ninst, 1, s);
}
EXOTX_API exotx_status exotx_forward_set_d_batch(exotx_plan p, int prec, const void *gpin, void *spout, int nlev,
                                                 int ninst, exotx_stream s) {
    return forward_set_api(p, prec, gpin, spout, nlev, ninst, 1, s);
}

EXOTX_API exotx_status exotx_tc_error(int *code, exotx_stream s) {
    if (!code) return EXOTX_BAD_ARG;
    int fe = 0;
    EXOTX_TRY(tc_error_read(code, (cudaStream_t)s));
    EXOTX_TRY(fft_error_read(&fe, (cudaStream_t)s));
    *code |= fe;
    EXOTX_TRY(fft_error_reset((cudaStream_t)s));
    return tc_error_reset((cudaStream_t)s);
}
