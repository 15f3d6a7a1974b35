// Gated delta rule: a [d, dv] state per head, S <- g S, u = beta (v - S^T k), S <- S + k u^T, o = S^T q, with one decay g per head
// or one per head and key channel.  q and k arrive after convolution and SiLU and are made unit vectors here (q also scaled by
// d^(-1/2)); head h reads q / k head h / (H / G).  beta = sigmoid(b), log g = nA_h softplus(a + dt_bias) with nA = -exp(A_log).
//
// delta_scan_kernel   any storage type, heads up to 256: token by token, float32 (bfloat16 prompts: delta_tc, tensor cores)
// delta_step_kernel   one token with the low-rank second products of decays and gates, head norm and gate, a cluster per head
#include <cooperative_groups.h>
#include "mix_delta.cuh"

namespace cg = cooperative_groups;

namespace scmx {

constexpr int DS_T = 16;      // tokens staged together
constexpr int DS_COLS = 8;    // columns of the state per CTA
template <int NR, bool CH> constexpr size_t ds_smem() { return (size_t)2 * DS_T * (64 * NR * (CH ? 3 : 2) + DS_COLS + 3) * 4; }

// Grid (heads, column slices of 8).  Threads 0 .. 127 run the recurrence: 16 lanes share a column of the state, lane l holds rows 4 l + 64 r ..
// 4 l + 64 r + 3 in registers.  With o = (g S)^T q + (q . k) u both sums over the old state are taken in one pass.  Threads 128 .. 255 stage the
// next 16 tokens (unit vectors, decays) while the present ones run, their loads one tile ahead.
// A chain per token (two sums over the column, one correction) bounds it, so the chain is cut short: 300 float32 tokens of 8 heads of 128 took
// 320 us with a column on four lanes, 8 tokens staged in the open and 32 CTAs of 128 threads.
template <typename T, int NR, bool CH>
__global__ void __launch_bounds__(256) delta_scan_kernel(const DeltaArgs a) {
    constexpr int D = 64 * NR, E = D / 32, TW = DS_T / 4;      // elements per staging lane, tokens per staging warp
    extern __shared__ __align__(16) float sm[];
    float* sq = sm;                              // [2][DS_T][D], zero above d
    float* sk = sq + 2 * DS_T * D;
    float* sg = sk + 2 * DS_T * D;               // CH: decays per channel
    float* sv = sg + (CH ? 2 * DS_T * D : 0);    // [2][DS_T][DS_COLS]
    float* sb = sv + 2 * DS_T * DS_COLS;         // [2][DS_T]: beta, q . k, decay of the head
    float *sqk = sb + 2 * DS_T, *sgs = sqk + 2 * DS_T;
    pdl_launch_dependents();
    pdl_wait();
    const int h = blockIdx.x, e0 = blockIdx.y * DS_COLS, tid = threadIdx.x;
    const int n = (int)a.n, tiles = (n + DS_T - 1) / DS_T;
    if (tid >= 128) {
        const int lane = tid & 31, w = (tid - 128) >> 5, kh = h / (a.H / a.G), col = tid & (DS_COLS - 1), row = (tid - 128) / DS_COLS;
        const T *q = static_cast<const T*>(a.q) + (int64_t)kh * a.d, *k = static_cast<const T*>(a.k) + (int64_t)kh * a.d;
        const T *v = static_cast<const T*>(a.v) + (int64_t)h * a.dv + e0 + col, *b = static_cast<const T*>(a.b) + h;
        const float nA = a.nA[h], qs = rsqrtf((float)a.d);
        float dtb[CH ? E : 1];
        if (CH) {
#pragma unroll
            for (int j = 0; j < E; ++j) dtb[CH ? j : 0] = lane + 32 * j < a.d ? a.dtb[(int64_t)h * a.d + lane + 32 * j] : 0.0f;
        } else {
            dtb[0] = a.dtb[h];
        }
        float x[TW][E], y[TW][E], g[TW][CH ? E : 1], bt[TW], vv;
        auto fetch = [&](int t0) {
#pragma unroll
            for (int i = 0; i < TW; ++i) {
                const int t = t0 + w + 4 * i;
                const bool ok = t < n;
#pragma unroll
                for (int j = 0; j < E; ++j) {
                    const int e = lane + 32 * j;
                    const bool in = ok && e < a.d;
                    x[i][j] = in ? ldf(q + (int64_t)t * a.ldq + e) : 0.0f;
                    y[i][j] = in ? ldf(k + (int64_t)t * a.ldk + e) : 0.0f;
                    if (CH) g[i][CH ? j : 0] = in ? static_cast<const float*>(a.a)[(int64_t)t * a.lda + (int64_t)h * a.d + e] : 0.0f;
                }
                if (!CH) g[i][0] = ok ? ldf(static_cast<const T*>(a.a) + (int64_t)t * a.lda + h) : 0.0f;
                bt[i] = ok ? ldf(b + (int64_t)t * a.ldb) : 0.0f;
            }
            vv = t0 + row < n && e0 + col < a.dv ? ldf(v + (int64_t)(t0 + row) * a.ldv) : 0.0f;
        };
        auto put = [&](int buf) {
#pragma unroll
            for (int i = 0; i < TW; ++i) {
                const int r = buf * DS_T + w + 4 * i;
                float qq = 0.0f, kk = 0.0f, qk = 0.0f;
#pragma unroll
                for (int j = 0; j < E; ++j) {
                    qq += x[i][j] * x[i][j];
                    kk += y[i][j] * y[i][j];
                    qk += x[i][j] * y[i][j];
                }
                const float iq = qs / sqrtf(warp_sumf(qq) + 1e-6f), ik = 1.0f / sqrtf(warp_sumf(kk) + 1e-6f);
                qk = warp_sumf(qk);
#pragma unroll
                for (int j = 0; j < E; ++j) {
                    const int e = lane + 32 * j;
                    sq[r * D + e] = x[i][j] * iq;
                    sk[r * D + e] = y[i][j] * ik;
                    if (CH) sg[r * D + e] = e < a.d ? expf(nA * softplus_f32(g[i][CH ? j : 0] + dtb[CH ? j : 0])) : 0.0f;
                }
                if (lane == 0) {
                    sqk[r] = qk * iq * ik;
                    sb[r] = 1.0f / (1.0f + expf(-bt[i]));
                    if (!CH) sgs[r] = expf(nA * softplus_f32(g[i][0] + dtb[0]));
                }
            }
            sv[buf * DS_T * DS_COLS + tid - 128] = vv;
        };
        fetch(0);
        put(0);
        if (tiles > 1) fetch(DS_T);
        __syncthreads();
        for (int t = 0; t < tiles; ++t) {
            if (t + 1 < tiles) put((t + 1) & 1);
            if (t + 2 < tiles) fetch((t + 2) * DS_T);
            __syncthreads();
        }
        return;
    }
    const int l = tid & 15, col = tid >> 4;
    const bool ok = e0 + col < a.dv;
    float* gS = a.state + (int64_t)h * a.d * a.dv + e0 + col;
    float4 S[NR];
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int i = 64 * r + 4 * l;
        S[r].x = ok && i < a.d ? gS[(int64_t)i * a.dv] : 0.0f;
        S[r].y = ok && i + 1 < a.d ? gS[(int64_t)(i + 1) * a.dv] : 0.0f;
        S[r].z = ok && i + 2 < a.d ? gS[(int64_t)(i + 2) * a.dv] : 0.0f;
        S[r].w = ok && i + 3 < a.d ? gS[(int64_t)(i + 3) * a.dv] : 0.0f;
    }
    __syncthreads();
    for (int tile = 0; tile < tiles; ++tile) {
        const int r0 = (tile & 1) * DS_T, nt = min(DS_T, n - tile * DS_T);
#pragma unroll 2
        for (int t = 0; t < nt; ++t) {
            const float4 *k4 = reinterpret_cast<const float4*>(sk + (r0 + t) * D), *q4 = reinterpret_cast<const float4*>(sq + (r0 + t) * D);
            const float4* g4 = reinterpret_cast<const float4*>(sg + (CH ? (r0 + t) * D : 0));
            const float gs = CH ? 0.0f : sgs[r0 + t];
            float4 kk[NR];
            float pk[NR], pq[NR];
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                kk[r] = k4[16 * r + l];
                const float4 qq = q4[16 * r + l], gg = CH ? g4[16 * r + l] : make_float4(gs, gs, gs, gs);
                S[r].x *= gg.x; S[r].y *= gg.y; S[r].z *= gg.z; S[r].w *= gg.w;
                pk[r] = S[r].x * kk[r].x; pk[r] = fmaf(S[r].y, kk[r].y, pk[r]); pk[r] = fmaf(S[r].z, kk[r].z, pk[r]); pk[r] = fmaf(S[r].w, kk[r].w, pk[r]);
                pq[r] = S[r].x * qq.x; pq[r] = fmaf(S[r].y, qq.y, pq[r]); pq[r] = fmaf(S[r].z, qq.z, pq[r]); pq[r] = fmaf(S[r].w, qq.w, pq[r]);
            }
            float sumk = pk[0], sumq = pq[0];
#pragma unroll
            for (int r = 1; r < NR; ++r) {
                sumk += pk[r];
                sumq += pq[r];
            }
#pragma unroll
            for (int o = 1; o < 16; o *= 2) sumk += __shfl_xor_sync(0xffffffffu, sumk, o);
            const float u = sb[r0 + t] * (sv[(r0 + t) * DS_COLS + col] - sumk);
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                S[r].x = fmaf(kk[r].x, u, S[r].x); S[r].y = fmaf(kk[r].y, u, S[r].y); S[r].z = fmaf(kk[r].z, u, S[r].z); S[r].w = fmaf(kk[r].w, u, S[r].w);
            }
#pragma unroll
            for (int o = 1; o < 16; o *= 2) sumq += __shfl_xor_sync(0xffffffffu, sumq, o);
            if (l == 0 && ok) a.o[((int64_t)(tile * DS_T + t) * a.H + h) * a.dv + e0 + col] = fmaf(sqk[r0 + t], u, sumq);
        }
        __syncthreads();
    }
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        const int i = 64 * r + 4 * l;
        if (ok && i < a.d) gS[(int64_t)i * a.dv] = S[r].x;
        if (ok && i + 1 < a.d) gS[(int64_t)(i + 1) * a.dv] = S[r].y;
        if (ok && i + 2 < a.d) gS[(int64_t)(i + 2) * a.dv] = S[r].z;
        if (ok && i + 3 < a.d) gS[(int64_t)(i + 3) * a.dv] = S[r].w;
    }
}

template <typename T, int NR, bool CH>
static int run_delta_rows(const DeltaArgs& a, cudaStream_t st) {
    constexpr size_t smem = ds_smem<NR, CH>();
    if (smem > 48 * 1024) SCMX_CUDA_OK(cudaFuncSetAttribute(delta_scan_kernel<T, NR, CH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    SCMX_PDL_OK("delta_scan_kernel",
                launch_pdl(delta_scan_kernel<T, NR, CH>, dim3(a.H, (a.dv + DS_COLS - 1) / DS_COLS), dim3(256), smem, st, a));
    return SCMX_OK;
}

template <typename T, bool CH>
static int run_delta_scan(const DeltaArgs& a, cudaStream_t st) {
    SCMX_REQUIRE(a.n < (1ll << 30), SCMX_ELIMIT, "delta: %lld tokens", (long long)a.n);
    if (a.d <= 64) return run_delta_rows<T, 1, CH>(a, st);
    if (a.d <= 128) return run_delta_rows<T, 2, CH>(a, st);
    return run_delta_rows<T, 4, CH>(a, st);
}

// ---- one token ------------------------------------------------------------------------------------------------------------
struct DeltaStepArgs {
    const float *q, *k, *v, *b;      // one row each, after convolution and SiLU (b: logits)
    const float *a, *g;              // decay logits [H] and gates [H dv], or the low-rank vectors [ra], [rg]
    const void *wa, *wg;             // second low-rank products [H d, lwa], [H dv, lwg], rows zero padded to a multiple of 8
    const float *nA, *dtb, *w;       // -exp(A_log) [H], dt_bias, head norm weight [dv]
    float* state;                    // [H, d, dv]
    float* y;                        // [H dv]
    int H, G, d, dv, ra, rg, lwa, lwg, cw;      // cw: state columns per CTA (<= 256)
    float eps;
};

// Products of stored rows (multiples of 8 columns) with a vector in shared memory, a group of lanes per row.  The first vector of the
// first PASS rows per group is requested by `request`, which may run before the vector is known.
template <typename T>
struct RowDots {
    static constexpr int PASS = 2;
    Raw8<T> pre[PASS];
    int lpr, sub, first, step;
    __device__ __forceinline__ void setup(int n, int lane, int warp) {
        lpr = 1;
        while (lpr < 32 && 8 * lpr < n) lpr *= 2;
        sub = lane & (lpr - 1);
        step = 256 / lpr;
        first = (32 * warp + lane) / lpr;
    }
    __device__ __forceinline__ void request(const T* w, int n, int rows) {
#pragma unroll
        for (int k = 0; k < PASS; ++k)
            if (first + k * step < rows && 8 * sub < n) pre[k].load(w + (int64_t)(first + k * step) * n + 8 * sub);
    }
    // done(row, product) for every row, on the lanes of its group; the warps of the CTA call it together
    template <typename F>
    __device__ __forceinline__ void run(const T* w, const float* x, int n, int rows, F done) {
        auto dot = [&](const Raw8<T>& u, int e, float s) -> float {
            float v[8];
            u.get(v);
#pragma unroll
            for (int i = 0; i < 8; ++i) s = fmaf(v[i], x[e + i], s);
            return s;
        };
        auto finish = [&](int row, float s) {
            for (int e = 8 * (sub + lpr); e < n; e += 8 * lpr)
                if (row < rows) {
                    Raw8<T> u;
                    u.load(w + (int64_t)row * n + e);
                    s = dot(u, e, s);
                }
            for (int o = lpr / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (row < rows) done(row, s);
        };
#pragma unroll
        for (int k = 0; k < PASS; ++k) {
            const int row = first + k * step;
            finish(row, row < rows && 8 * sub < n ? dot(pre[k], 8 * sub, 0.0f) : 0.0f);
        }
        for (int r0 = PASS * step; r0 < rows; r0 += step) {
            const int row = first + r0;
            float s = 0.0f;
            if (row < rows && 8 * sub < n) {
                Raw8<T> u;
                u.load(w + (int64_t)row * n + 8 * sub);
                s = dot(u, 8 * sub, 0.0f);
            }
            finish(row, s);
        }
    }
};

template <typename T, bool CH>
__global__ void __launch_bounds__(256) delta_step_kernel(const DeltaStepArgs a) {
    extern __shared__ __align__(16) float sm[];
    float *sa = sm, *sg1 = sa + a.lwa, *sq = sg1 + a.lwg, *sk = sq + a.d, *sg = sk + a.d, *so = sg + a.d, *su = so + 512, *sgate = su + 256;
    __shared__ float red[33];
    __shared__ float ssq[8];         // the cluster's sums of squares, each written by its CTA
    pdl_launch_dependents();
    cg::cluster_group cl = cg::this_cluster();
    const int h = blockIdx.y, rank = (int)cl.block_rank(), nc = (int)cl.num_blocks(), tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int kh = h / (a.H / a.G);
    const int e0 = rank * a.cw, cw = min(a.cw, a.dv - e0);      // cw may be <= 0 on a trailing rank
    const int groups = cw > 0 ? 256 / cw : 0, grp = cw > 0 ? tid / cw : 0, col = cw > 0 ? tid - grp * cw : 0;
    const bool work = grp < groups;
    // low-rank weights of this CTA's channels and values never change: requested before the previous kernel ends
    const int per = (a.d + nc - 1) / nc, ch0 = min(a.d, rank * per), nch = min(per, a.d - ch0);
    const T *wa = static_cast<const T*>(a.wa) + ((int64_t)h * a.d + ch0) * a.lwa, *wg = static_cast<const T*>(a.wg) + ((int64_t)h * a.dv + e0) * a.lwg;
    RowDots<T> da, dg;
    if (CH) {
        da.setup(a.lwa, lane, warp);
        dg.setup(a.lwg, lane, warp);
        da.request(wa, a.lwa, nch);
        dg.request(wg, a.lwg, cw);
    }
    if (CH || nc > 1) cl.sync();     // every CTA of the cluster runs: its shared memory may be written
    pdl_wait();
    constexpr int PRE = 16;          // the first rows of this thread's column are requested before anything else
    float* S = a.state + (int64_t)h * a.d * a.dv + e0 + col;
    float pre[PRE];
#pragma unroll
    for (int j = 0; j < PRE; ++j) {
        const int i = grp + j * groups;
        pre[j] = work && i < a.d ? S[(int64_t)i * a.dv] : 0.0f;
    }
    const float v = tid < cw ? a.v[(int64_t)h * a.dv + e0 + tid] : 0.0f;
    const float beta = 1.0f / (1.0f + expf(-a.b[h])), nA = a.nA[h];
    if (CH) {
        for (int i = tid; i < a.lwa; i += 256) sa[i] = i < a.ra ? a.a[i] : 0.0f;
        for (int i = tid; i < a.lwg; i += 256) sg1[i] = i < a.rg ? a.g[i] : 0.0f;
    }
    // unit vectors: every warp takes the three sums for itself
    float qq = 0.0f, kk = 0.0f, qk = 0.0f;
    for (int i = lane; i < a.d; i += 32) {
        const float x = a.q[(int64_t)kh * a.d + i], y = a.k[(int64_t)kh * a.d + i];
        qq += x * x;
        kk += y * y;
        qk += x * y;
    }
    const float iq = rsqrtf((float)a.d) / sqrtf(warp_sumf(qq) + 1e-6f), ik = 1.0f / sqrtf(warp_sumf(kk) + 1e-6f);
    qk = warp_sumf(qk) * iq * ik;
    for (int i = tid; i < a.d; i += 256) {
        sq[i] = a.q[(int64_t)kh * a.d + i] * iq;
        sk[i] = a.k[(int64_t)kh * a.d + i] * ik;
        if (!CH) sg[i] = expf(nA * softplus_f32(a.a[h] + a.dtb[h]));
    }
    float gate = 0.0f;
    if (CH) {
        __syncthreads();
        da.run(wa, sa, a.lwa, nch, [&](int c, float z) {
            if (da.sub >= nc) return;
            const float g = expf(nA * softplus_f32(z + a.dtb[(int64_t)h * a.d + ch0 + c]));
            for (int r = da.sub; r < nc; r += da.lpr) *cl.map_shared_rank(sg + ch0 + c, r) = g;
        });
        dg.run(wg, sg1, a.lwg, cw, [&](int c, float z) {
            if (dg.sub == 0) sgate[c] = 1.0f / (1.0f + expf(-z));
        });
        cl.sync();
        if (tid < cw) gate = sgate[tid];
    } else {
        if (tid < cw) gate = silu_f32(a.g[(int64_t)h * a.dv + e0 + tid]);
        __syncthreads();
    }
    float pk = 0.0f, pq = 0.0f;
    if (work) {
#pragma unroll
        for (int j = 0; j < PRE; ++j) {
            const int i = grp + j * groups;
            if (i < a.d) {
                pre[j] *= sg[i];
                pk = fmaf(pre[j], sk[i], pk);
                pq = fmaf(pre[j], sq[i], pq);
            }
        }
#pragma unroll 8
        for (int i = grp + PRE * groups; i < a.d; i += groups) {
            const float s = S[(int64_t)i * a.dv] * sg[i];
            pk = fmaf(s, sk[i], pk);
            pq = fmaf(s, sq[i], pq);
        }
    }
    so[tid] = pk;
    so[256 + tid] = pq;
    __syncthreads();
    float o = 0.0f;
    if (tid < cw) {
        float k0 = 0.0f, q0 = 0.0f;
        for (int r = 0; r < groups; ++r) {
            k0 += so[r * cw + tid];
            q0 += so[256 + r * cw + tid];
        }
        const float u = beta * (v - k0);
        su[tid] = u;
        o = fmaf(qk, u, q0);
    }
    const float ss = block_sumf(o * o, red);      // (its barriers also publish su)
    // The sums are handed round before the rows in registers are stored, since a cluster barrier waits for the stores before it; rows that are read again go first.
    // One token of 8 heads of 128 takes 7.8 us with decays per channel, 5.4 per head (8.2 and 5.6 with all stores first and the sums fetched between two barriers).
    const float u = work ? su[col] : 0.0f;
    if (work)
#pragma unroll 8
        for (int i = grp + PRE * groups; i < a.d; i += groups) S[(int64_t)i * a.dv] = fmaf(sk[i], u, S[(int64_t)i * a.dv] * sg[i]);
    float total = ss;
    if (nc > 1) {
        if (tid < nc) *cl.map_shared_rank(ssq + rank, tid) = ss;
        cl.sync();
        total = 0.0f;
        for (int r = 0; r < nc; ++r) total += ssq[r];
    }
    if (tid < cw) a.y[(int64_t)h * a.dv + e0 + tid] = o * rms_inv_f32(total, a.dv, a.eps) * a.w[e0 + tid] * gate;
    if (work)
#pragma unroll
        for (int j = 0; j < PRE; ++j) {
            const int i = grp + j * groups;
            if (i < a.d) S[(int64_t)i * a.dv] = fmaf(sk[i], u, pre[j]);
        }
}

template <typename T, bool CH>
static int run_delta_step(DeltaStepArgs a, cudaStream_t st) {
    int nc = 1;                                   // CTAs per head: slices of at least 32 columns, 256 at most
    while (nc < 8 && (a.dv + nc - 1) / nc > 32) nc *= 2;
    a.cw = (a.dv + nc - 1) / nc;
    SCMX_REQUIRE(a.cw <= 256, SCMX_ELIMIT, "delta_step: %d values per head (2048 at most)", a.dv);
    const size_t smem = (size_t)(a.lwa + a.lwg + 3 * a.d + 512 + 256 + 256) * 4;
    SCMX_REQUIRE(smem <= 48 * 1024, SCMX_ELIMIT, "delta_step: head size %d, inner sizes %d and %d", a.d, a.ra, a.rg);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(nc, a.H);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = g_use_pdl ? 2 : 1;
    SCMX_PDL_OK("delta_step_kernel", cudaLaunchKernelEx(&cfg, delta_step_kernel<T, CH>, a));
    return SCMX_OK;
}

}  // namespace scmx

using namespace scmx;

extern "C" int64_t scmx_delta_scratch(int64_t n, int H, int d, int dv, int64_t ldv) {
    return n > 0 && H > 0 && d > 0 && dv > 0 && delta_tc_supported(n, H, d, dv, ldv) ? delta_tc_scratch(n, H, d, dv) : 0;
}

extern "C" int scmx_delta(const void* q, int64_t ldq, const void* k, int64_t ldk, const void* v, int64_t ldv, const void* b, int64_t ldb,
                          const void* a_, int64_t lda, int dt, int channel, int64_t n, int H, int G, int d, int dv, const float* nA,
                          const float* dt_bias, float* state, float* o, void* scratch, int64_t scratch_bytes, int32_t* status, void* stream) {
    SCMX_DT_OK("delta", dt);
    SCMX_REQUIRE(q && k && v && b && a_ && nA && dt_bias && state && o, SCMX_EINVAL, "delta: null buffer");
    SCMX_REQUIRE(n >= 0 && H > 0 && G > 0 && H % G == 0 && d > 0 && dv > 0, SCMX_EINVAL, "delta: n=%lld heads=%d over %d, sizes %d / %d", (long long)n, H, G, d, dv);
    SCMX_REQUIRE(d <= 256, SCMX_ELIMIT, "delta: head size %d (256 at most)", d);
    if (n == 0) return SCMX_OK;
    DeltaArgs a;
    a.q = q; a.k = k; a.v = v; a.b = b; a.a = a_; a.nA = nA; a.dtb = dt_bias; a.state = state; a.o = o;
    a.n = n; a.ldq = ldq; a.ldk = ldk; a.ldv = ldv; a.ldb = ldb; a.lda = lda; a.H = H; a.G = G; a.d = d; a.dv = dv;
    const cudaStream_t st = (cudaStream_t)stream;
    if (scratch != nullptr) {
        SCMX_REQUIRE(dt == 0 && status && delta_tc_supported(n, H, d, dv, ldv), SCMX_ELIMIT, "delta: no tensor-core form for head sizes %d / %d", d, dv);
        SCMX_REQUIRE(((uintptr_t)v & 15) == 0 && ((uintptr_t)scratch & 255) == 0 && scratch_bytes >= delta_tc_scratch(n, H, d, dv), SCMX_EINVAL,
                     "delta: scratch of %lld bytes or an unaligned pointer", (long long)scratch_bytes);
        return delta_tc(a, channel != 0, scratch, status, st);
    }
    if (dt == 0) return channel ? run_delta_scan<bf16_t, true>(a, st) : run_delta_scan<bf16_t, false>(a, st);
    return channel ? run_delta_scan<float, true>(a, st) : run_delta_scan<float, false>(a, st);
}

extern "C" int scmx_delta_step(const float* q, const float* k, const float* v, const float* b, const float* a_, const float* g, const void* wa,
                               int64_t lwa, int ra, const void* wg, int64_t lwg, int rg, int dt, int H, int G, int d, int dv, const float* nA,
                               const float* dt_bias, const float* w, float eps, float* state, float* y, void* stream) {
    SCMX_DT_OK("delta_step", dt);
    SCMX_REQUIRE(q && k && v && b && a_ && g && nA && dt_bias && w && state && y, SCMX_EINVAL, "delta_step: null buffer");
    SCMX_REQUIRE(H > 0 && G > 0 && H % G == 0 && d > 0 && dv > 0, SCMX_EINVAL, "delta_step: heads=%d over %d, sizes %d / %d", H, G, d, dv);
    SCMX_REQUIRE((wa != nullptr) == (wg != nullptr), SCMX_EINVAL, "delta_step: low-rank products of decays and gates come together");
    SCMX_REQUIRE(wa == nullptr || (ra > 0 && rg > 0 && lwa % 8 == 0 && lwg % 8 == 0 && lwa >= ra && lwg >= rg && lwa < (1 << 16) && lwg < (1 << 16) &&
                                   (((uintptr_t)wa | (uintptr_t)wg) & 15) == 0), SCMX_EINVAL, "delta_step: pitches %lld, %lld of inner sizes %d, %d",
                 (long long)lwa, (long long)lwg, ra, rg);
    DeltaStepArgs s;
    s.q = q; s.k = k; s.v = v; s.b = b; s.a = a_; s.g = g; s.wa = wa; s.wg = wg; s.nA = nA; s.dtb = dt_bias; s.w = w; s.state = state; s.y = y;
    s.H = H; s.G = G; s.d = d; s.dv = dv; s.ra = wa ? ra : 0; s.rg = wa ? rg : 0; s.lwa = wa ? (int)lwa : 0; s.lwg = wa ? (int)lwg : 0; s.cw = 0; s.eps = eps;
    const cudaStream_t st = (cudaStream_t)stream;
    if (wa == nullptr) return run_delta_step<float, false>(s, st);
    return dt == 0 ? run_delta_step<bf16_t, true>(s, st) : run_delta_step<float, true>(s, st);
}
