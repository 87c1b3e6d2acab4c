// FP32-accurate GEMMs on the tensor cores, for the radiation surrogate's
// training (surrogate.cu).  The three products of a layer and what follows
// each in the same kernel:
//   forward      Z = H W^T + b          then H' = silu(Z)
//   activation   dH = dZ W              then dZ' = dH silu'(Z), over Z
//   weights      dW = dZ^T H, db = column sums of dZ, every layer in one
//                launch, the sum over the batch in ranges of TG_KSPLIT rows
//                whose partials k_tg_reduce adds in a fixed order.
//
// Both operands are split into three BF16 terms (x ~= h + m + l to 2^-24
// relative) as they are staged in shared memory, and the six split products
// of order <= 2 accumulate in FP32 in tensor memory: the hi*hi product in one
// accumulator, the five corrections in another (the tensor-core adder
// truncates; keeping the large term's chain apart bounds that error), summed
// in the epilogue.  The result agrees with an FP32 SIMT GEMM to about 1e-6.
//
// A CTA (16 warps) computes a 128 x 64 tile: at the usual batch of 4096 rows and
// width 256 that is 128 CTAs, one wave (128 x 128 tiles gave 64).  Per K-chunk
// of 32 every thread splits the 12 values it loaded two chunks earlier into one
// of two buffers and issues the loads of the next but one; thread 0 issues the chunk's MMAs
// (tcgen05.mma, kind::f16, M = 128), whose commit frees the buffer.  Bound by
// the latency of that chain (eight chunks at width 256), not by the MMAs or by
// memory: the operands are in L2.  Two CTAs share an SM.  One step at batch
// 4096, six hidden layers: 1427 -> 228 us (before: scalar loads without a
// prefetch, 50 us per product, separate activation, column-sum and reduction
// passes).  Every wait is bounded and reports through an error word that
// exotx_mlp_check reads.
#include <algorithm>
#include "exotx_internal.cuh"
#include "tc_prims.cuh"

namespace exotx {

constexpr int TG_M = 128, TG_N = 64, TG_KC = 32, TG_THREADS = 512;
// K-adjacent core matrices 160 bytes apart, row groups 656: the stores then touch
// every bank once in both staging orders below (8-byte, 2 rows x 8 float4s a half
// warp: 160 = 32 mod 128; 4-byte, 8 row sets x 4 K pairs a warp: 656 = 16 mod 128)
constexpr uint32_t TG_LBO = 160, TG_SBO = TG_KC / 8 * TG_LBO + 16;
constexpr uint32_t TG_TA = TG_M / 8 * TG_SBO, TG_TB = TG_N / 8 * TG_SBO;   // bytes of one split term
constexpr uint32_t TG_STAGE = 3 * (TG_TA + TG_TB);
constexpr int TG_CLD = TG_N + 4;                                            // row of the epilogue's FP32 tile
constexpr size_t TG_SMEM = 2 * (size_t)TG_STAGE + 64;                       // 2 stages + barriers
constexpr int TG_KSPLIT = 256;                                              // batch rows per CTA of a weight gradient
static_assert(TG_M * TG_CLD * 4 <= 2 * TG_STAGE && TG_STAGE % 16 == 0 && TG_TA % 16 == 0 && TG_TB % 16 == 0, "");

__device__ int g_tg_error;   // nonzero: a bounded wait gave up

enum { TG_BIAS = 0, TG_SILU, TG_SILU_BWD, TG_WEIGHTS };

__device__ __forceinline__ float tg_silu(float z) { return z / (1.f + expf(-z)); }
__device__ __forceinline__ float tg_silu_grad(float z) {
    const float sg = 1.f / (1.f + expf(-z));
    return sg * (1.f + z * (1.f - sg));
}

// An operand tile of ROWS rows x 32 K, ROWS / 16 floats a thread.  KC: element
// (r, k) at p[r * ld + k]; float4s along K, eight threads to a row.  Otherwise it
// is at p[k * ld + r]; a float4 (float2 for 64 rows) along the rows for each of
// two consecutive K, eight row sets and four K pairs to a warp.
template <int ROWS, bool KC>
struct TgTile {
    static constexpr int VW = KC ? 4 : ROWS / 32, NV = ROWS / 16 / VW;
    __align__(16) float v[NV][VW];
    static __device__ __forceinline__ int row() {
        return KC ? (int)threadIdx.x >> 3 : VW * ((threadIdx.x & 7) + 8 * ((threadIdx.x >> 5) & 3));
    }
    static __device__ __forceinline__ int kof() {
        return KC ? 4 * (threadIdx.x & 7) : 2 * (((threadIdx.x & 31) >> 3) + 4 * (threadIdx.x >> 7));
    }
    // p: this thread's first element of the chunk; a whole and 16-byte aligned tile
    __device__ __forceinline__ void load(const float *p, long long ld) {
#pragma unroll
        for (int i = 0; i < NV; i++, p += KC ? TG_THREADS / 8 * ld : ld) {
            if constexpr (VW == 4) *reinterpret_cast<float4 *>(v[i]) = *reinterpret_cast<const float4 *>(p);
            else *reinterpret_cast<float2 *>(v[i]) = *reinterpret_cast<const float2 *>(p);
        }
    }
    // nr and nk: rows and K from that element on, beyond which the values are zero
    __device__ __forceinline__ void load(const float *p, long long ld, int nr, int nk) {
#pragma unroll
        for (int i = 0; i < NV; i++)
#pragma unroll
            for (int j = 0; j < VW; j++) {
                const int r = KC ? i * (TG_THREADS / 8) : j, k = KC ? j : i;
                v[i][j] = r < nr && k < nk ? p[KC ? r * ld + k : k * ld + r] : 0.f;
            }
    }
    // byte offset of this thread's first element in a stage
    static __device__ __forceinline__ uint32_t off() {
        const int r = row(), k = kof();
        return (r >> 3) * TG_SBO + (k >> 3) * TG_LBO + (r & 7) * 16 + (k & 7) * 2;
    }
    __device__ __forceinline__ void store(unsigned char *o, uint32_t term) const {
        if constexpr (KC) {
            uint32_t h[2], m[2], l[2];
#pragma unroll
            for (int i = 0; i < NV; i++, o += TG_THREADS / 64 * TG_SBO) {
                tc::split3x2(v[i][0], v[i][1], h[0], m[0], l[0]);
                tc::split3x2(v[i][2], v[i][3], h[1], m[1], l[1]);
                *reinterpret_cast<uint2 *>(o) = make_uint2(h[0], h[1]);
                *reinterpret_cast<uint2 *>(o + term) = make_uint2(m[0], m[1]);
                *reinterpret_cast<uint2 *>(o + 2 * term) = make_uint2(l[0], l[1]);
            }
        } else {
            uint32_t h, m, l;
#pragma unroll
            for (int j = 0; j < VW; j++, o += 16) {
                tc::split3x2(v[0][j], v[1][j], h, m, l);
                *reinterpret_cast<uint32_t *>(o) = h;
                *reinterpret_cast<uint32_t *>(o + term) = m;
                *reinterpret_cast<uint32_t *>(o + 2 * term) = l;
            }
        }
    }
};

// both operands' tiles of one chunk
template <bool AKC, bool BKC>
struct TgChunk {
    TgTile<TG_M, AKC> a;
    TgTile<TG_N, BKC> b;
};

struct TgArgs {
    int M, N, K;
    const float *A, *B;       // TG_WEIGHTS: A(m,k) = A[k * lda + m], else A[m * lda + k];
    long long lda, ldb;       // forward: B(k,n) = B[n * ldb + k], else B[k * ldb + n]
    const float *bias;
    float *C, *H;             // M x N, contiguous; H: TG_SILU
    // TG_WEIGHTS: one entry per layer, its first tile in grid x
    int nl, tile0[TG_MAXL + 1];
    int lM[TG_MAXL], lN[TG_MAXL];
    const float *lA[TG_MAXL], *lB[TG_MAXL];
    long long woff[TG_MAXL], boff[TG_MAXL], nparams;
    float *part;              // [K range][nparams]
};

template <int EPI>
__global__ void __launch_bounds__(TG_THREADS, 2) k_tc_gemm(const __grid_constant__ TgArgs g) {
    extern __shared__ __align__(128) unsigned char sm[];
    constexpr bool AKC = EPI != TG_WEIGHTS, BKC = EPI == TG_BIAS || EPI == TG_SILU;
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + 2 * (size_t)TG_STAGE);
    uint32_t *slot = reinterpret_cast<uint32_t *>(bar + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    pdl_trigger();
    int M = g.M, N = g.N, mt = blockIdx.x, nt = blockIdx.y, kbeg = 0, kend = g.K, layer = 0;
    const float *A = g.A, *B = g.B;
    long long lda = g.lda, ldb = g.ldb;
    if constexpr (EPI == TG_WEIGHTS) {
        while (layer + 1 < g.nl && (int)blockIdx.x >= g.tile0[layer + 1]) layer++;
        M = g.lM[layer]; N = g.lN[layer]; A = g.lA[layer]; B = g.lB[layer];
        lda = M; ldb = N;
        const int ntn = (N + TG_N - 1) / TG_N, t = blockIdx.x - g.tile0[layer];
        mt = t / ntn; nt = t % ntn;
        kbeg = blockIdx.y * TG_KSPLIT; kend = min(g.K, kbeg + TG_KSPLIT);
    }
    const int m0 = mt * TG_M, n0 = nt * TG_N;
    const int NT = min(TG_N, (N - n0 + 15) & ~15);   // MMA N
    const int nchunk = (kend - kbeg + TG_KC - 1) / TG_KC;
    const bool va = ((reinterpret_cast<uintptr_t>(A) | (uintptr_t)(lda * 4)) & 15) == 0;
    const bool vb = ((reinterpret_cast<uintptr_t>(B) | (uintptr_t)(ldb * 4)) & 15) == 0;
    if (warp == 0) tc::tmem_alloc(slot, 2 * TG_N);   // accumulators: hi*hi at column 0, corrections at TG_N
    if (tid == 0) {
        tc::mbar_init(bar, 1);
        tc::mbar_init(bar + 1, 1);
        tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = *slot;
    pdl_wait();
    using TA = TgTile<TG_M, AKC>;
    using TB = TgTile<TG_N, BKC>;
    TgChunk<AKC, BKC> cur, nxt;
    const float *pa = A + (AKC ? (m0 + TA::row()) * lda + kbeg + TA::kof() : (kbeg + TA::kof()) * lda + m0 + TA::row());
    const float *pb = B + (BKC ? (n0 + TB::row()) * ldb + kbeg + TB::kof() : (kbeg + TB::kof()) * ldb + n0 + TB::row());
    const long long sa = AKC ? TG_KC : TG_KC * lda, sb = BKC ? TG_KC : TG_KC * ldb;
    const bool whole = va && m0 + TG_M <= M && vb && n0 + TG_N <= N;
    const uint32_t oa = TA::off(), ob = 3 * TG_TA + TB::off();
    auto load = [&](TgChunk<AKC, BKC> &t, int c) {
        const int k0 = kbeg + c * TG_KC;
        if (whole && k0 + TG_KC <= kend) {
            t.a.load(pa, lda);
            t.b.load(pb, ldb);
        } else {
            t.a.load(pa, lda, M - m0 - TA::row(), kend - k0 - TA::kof());
            t.b.load(pb, ldb, N - n0 - TB::row(), kend - k0 - TB::kof());
        }
        pa += sa;
        pb += sb;
    };
    float cs[4] = {0.f, 0.f, 0.f, 0.f};              // TG_WEIGHTS: this thread's share of db
    const uint32_t idesc = tc::idesc_bf16(TG_M, NT);
    int issued = 0;                                  // chunks whose MMAs are on their way
    // stage chunk c, issue the loads of chunk c + 2 in its place, then the MMAs
    auto step = [&](TgChunk<AKC, BKC> &t, int c) {
        const int b = c & 1;
        unsigned char *st = sm + (size_t)b * TG_STAGE;
        bool ok = true;
        // the buffer's previous chunk must have been read by its MMAs
        if (c >= 2) ok = tc::mbar_wait(bar + b, ((c - 2) >> 1) & 1);
        if (ok) {
            t.a.store(st + oa, TG_TA);
            t.b.store(st + ob, TG_TB);
        }
        if constexpr (EPI == TG_WEIGHTS) {
#pragma unroll
            for (int j = 0; j < 4; j++) cs[j] += t.a.v[0][j] + t.a.v[1][j];
        }
        tc::fence_proxy_async();
        if (c + 2 < nchunk) load(t, c + 2);
        if (!__syncthreads_and(ok)) return false;
        if (tid == 0) {
            tc::fence_after_sync();
            const uint64_t da = tc::smem_desc(st, TG_LBO, TG_SBO);
            const uint64_t db = tc::smem_desc(st + 3 * TG_TA, TG_LBO, TG_SBO);
#pragma unroll
            for (int ks = 0; ks < TG_KC / 16; ks++) {
#pragma unroll
                for (int pr = 0; pr < 6; pr++) {
                    const bool first = c == 0 && ks == 0 && pr <= 1;
                    tc::mma_bf16(tmem + (pr == 0 ? 0u : (uint32_t)TG_N),
                                 tc::desc_add(da, tc::pair_a(pr) * TG_TA + ks * 2 * TG_LBO),
                                 tc::desc_add(db, tc::pair_b(pr) * TG_TB + ks * 2 * TG_LBO), idesc, !first);
                }
            }
            tc::mma_commit(bar + b);
        }
        issued = c + 1;
        return true;
    };
    load(cur, 0);
    if (nchunk > 1) load(nxt, 1);
    bool ok = true;
    for (int c = 0; c < nchunk && ok; c += 2) {
        ok = step(cur, c);
        if (ok && c + 1 < nchunk) ok = step(nxt, c + 1);
    }
    // every MMA has completed once the last issued chunk's commit has arrived; waited
    // for after a timeout too, before the accumulators are given back
    if (issued && !tc::mbar_wait(bar + ((issued - 1) & 1), ((issued - 1) >> 1) & 1)) ok = false;
    ok = __syncthreads_and(ok) != 0;
    if (!ok && tid == 0) atomicExch(&g_tg_error, 1);
    tc::fence_after_sync();
    float *ct = reinterpret_cast<float *>(sm);       // the tile, over the stages
    if (ok) {
        // warp w drains TMEM lane quarter w % 4 (32 rows), column quarter w / 4
        const int q = warp & 3, cc = (warp >> 2) * (TG_N / 4);
        const uint32_t lane_addr = (uint32_t)(32 * q) << 16;
        if (cc < NT) {                               // whole warp
            uint32_t ra[16], rb[16];
            tc::tmem_ld16_nw(tmem + lane_addr + (uint32_t)cc, ra);
            tc::tmem_ld16_nw(tmem + lane_addr + (uint32_t)(TG_N + cc), rb);
            tc::tmem_wait_ld();
            float *o = ct + (32 * q + lane) * TG_CLD + cc;
#pragma unroll
            for (int i = 0; i < 16; i += 4)
                *reinterpret_cast<float4 *>(o + i) =
                    make_float4(__uint_as_float(ra[i]) + __uint_as_float(rb[i]),
                                __uint_as_float(ra[i + 1]) + __uint_as_float(rb[i + 1]),
                                __uint_as_float(ra[i + 2]) + __uint_as_float(rb[i + 2]),
                                __uint_as_float(ra[i + 3]) + __uint_as_float(rb[i + 3]));
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == 0) tc::tmem_dealloc(tmem, 2 * TG_N);
    if (!ok) return;
    // 16 lanes to a row, four columns each
    float *C = g.C;
    if constexpr (EPI == TG_WEIGHTS) C = g.part + blockIdx.y * g.nparams + g.woff[layer];
    const int nv = N - n0 - 4 * (lane & 15);         // columns from this thread's first
    const bool vc = nv >= 4 && ((reinterpret_cast<uintptr_t>(C) | (uintptr_t)((long long)N * 4)) & 15) == 0 &&
                    (EPI != TG_SILU || (reinterpret_cast<uintptr_t>(g.H) & 15) == 0);
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
    if constexpr (EPI == TG_BIAS || EPI == TG_SILU) {
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (i < nv) bias[i] = g.bias[n0 + 4 * (lane & 15) + i];
    }
    for (int r = 2 * warp + (lane >> 4); r < TG_M && m0 + r < M; r += TG_THREADS / 16) {
        const float4 t = *reinterpret_cast<const float4 *>(ct + r * TG_CLD + 4 * (lane & 15));
        float z[4] = {t.x + bias[0], t.y + bias[1], t.z + bias[2], t.w + bias[3]};
        const size_t o = (size_t)(m0 + r) * N + n0 + 4 * (lane & 15);
        if constexpr (EPI == TG_SILU_BWD) {
            float zp[4] = {0.f, 0.f, 0.f, 0.f};
            if (vc) {
                const float4 y = *reinterpret_cast<const float4 *>(C + o);
                zp[0] = y.x; zp[1] = y.y; zp[2] = y.z; zp[3] = y.w;
            } else {
#pragma unroll
                for (int i = 0; i < 4; i++)
                    if (i < nv) zp[i] = C[o + i];
            }
#pragma unroll
            for (int i = 0; i < 4; i++) z[i] *= tg_silu_grad(zp[i]);
        }
        if (vc) {
            *reinterpret_cast<float4 *>(C + o) = make_float4(z[0], z[1], z[2], z[3]);
            if constexpr (EPI == TG_SILU)
                *reinterpret_cast<float4 *>(g.H + o) =
                    make_float4(tg_silu(z[0]), tg_silu(z[1]), tg_silu(z[2]), tg_silu(z[3]));
        } else {
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (i < nv) {
                    C[o + i] = z[i];
                    if constexpr (EPI == TG_SILU) g.H[o + i] = tg_silu(z[i]);
                }
        }
    }
    if constexpr (EPI == TG_WEIGHTS) {
        if (nt != 0) return;                         // whole block
        // db: the four K pairs of a warp, then the four warps of a row block
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; j++) {
            cs[j] += __shfl_xor_sync(0xffffffffu, cs[j], 8);
            cs[j] += __shfl_xor_sync(0xffffffffu, cs[j], 16);
        }
        if (lane < 8)
            *reinterpret_cast<float4 *>(ct + (warp >> 2) * TG_M + TgTile<TG_M, AKC>::row()) = make_float4(cs[0], cs[1], cs[2], cs[3]);
        __syncthreads();
        if (tid < TG_M && m0 + tid < M)
            g.part[blockIdx.y * g.nparams + g.boff[layer] + m0 + tid] =
                (ct[tid] + ct[TG_M + tid]) + (ct[2 * TG_M + tid] + ct[3 * TG_M + tid]);
    }
}

// G[i] = sum over the ranges, in order, of part[z][i]
__global__ void k_tg_reduce(const float *part, int nz, long long n, float *G) {
    pdl_wait();
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        float v = 0.f;
#pragma unroll 8
        for (int z = 0; z < nz; z++) v += part[z * n + i];
        G[i] = v;
    }
}

template <int EPI>
static exotx_status tg_launch(const TgArgs &g, dim3 grid, cudaStream_t s) {
    EXOTX_CUDA(cudaFuncSetAttribute(k_tc_gemm<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TG_SMEM));
    EXOTX_CUDA(launch_pdl(k_tc_gemm<EPI>, grid, dim3(TG_THREADS), TG_SMEM, s, g));
    EXOTX_CHECK_LAUNCH();
    return EXOTX_OK;
}
static dim3 tg_grid(const TgArgs &g) {
    return dim3((unsigned)((g.M + TG_M - 1) / TG_M), (unsigned)((g.N + TG_N - 1) / TG_N));
}

exotx_status tc_mlp_forward(int n, int din, int dout, const float *X, const float *W, const float *bias, float *Z, float *H,
                            cudaStream_t s) {
    TgArgs g = {};
    g.M = n; g.N = dout; g.K = din;
    g.A = X; g.lda = din; g.B = W; g.ldb = din; g.bias = bias; g.C = Z; g.H = H;
    return H ? tg_launch<TG_SILU>(g, tg_grid(g), s) : tg_launch<TG_BIAS>(g, tg_grid(g), s);
}

exotx_status tc_mlp_activation(int n, int din, int dout, const float *dZ, const float *W, float *Z, cudaStream_t s) {
    TgArgs g = {};
    g.M = n; g.N = din; g.K = dout;
    g.A = dZ; g.lda = dout; g.B = W; g.ldb = din; g.C = Z;
    return tg_launch<TG_SILU_BWD>(g, tg_grid(g), s);
}

size_t tc_mlp_weights_work(long long nparams, int n) { return (size_t)((n + TG_KSPLIT - 1) / TG_KSPLIT) * nparams; }

exotx_status tc_mlp_weights(int nl, const int *din, const int *dout, const float *const *dZ, const float *const *H,
                            const long long *woff, const long long *boff, long long nparams, int n, float *work, float *G,
                            cudaStream_t s) {
    TgArgs g = {};
    if (nl < 1 || nl > TG_MAXL) return EXOTX_BAD_ARG;
    g.K = n; g.nl = nl; g.nparams = nparams; g.part = work;
    for (int l = 0; l < nl; l++) {
        g.lM[l] = dout[l]; g.lN[l] = din[l]; g.lA[l] = dZ[l]; g.lB[l] = H[l];
        g.woff[l] = woff[l]; g.boff[l] = boff[l];
        g.tile0[l + 1] = g.tile0[l] + (dout[l] + TG_M - 1) / TG_M * ((din[l] + TG_N - 1) / TG_N);
    }
    const int nz = (n + TG_KSPLIT - 1) / TG_KSPLIT;
    EXOTX_TRY(tg_launch<TG_WEIGHTS>(g, dim3((unsigned)g.tile0[nl], (unsigned)nz), s));
    EXOTX_CUDA(launch_pdl(k_tg_reduce, dim3((unsigned)std::min<long long>((nparams + 255) / 256, 1184)), dim3(256), 0, s,
                          (const float *)work, nz, nparams, G));
    EXOTX_CHECK_LAUNCH();
    return EXOTX_OK;
}

exotx_status tc_sgemm_error(int *err, cudaStream_t s) {
    EXOTX_CUDA(cudaMemcpyFromSymbolAsync(err, g_tg_error, sizeof(int), 0, cudaMemcpyDeviceToHost, s));
    EXOTX_CUDA(cudaStreamSynchronize(s));
    return EXOTX_OK;
}

}  // namespace exotx
