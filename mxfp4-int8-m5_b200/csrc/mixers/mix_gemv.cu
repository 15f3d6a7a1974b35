// Matrix-vector product of the decode step: out [N] = W [N, K] x, weights bfloat16 or float, x and out float32, float32
// accumulation.  Each warp sums two rows at a time (or a slice of their columns) and keeps two sets of 8 weight loads of 16 bytes per lane
// in flight across its rows; the first are issued before the previous kernel of the chain has finished (weights never change).
// Epilogues: none; xIELU; the causal convolution + SiLU of the first C rows, whose carried inputs are shifted in place; gelu(gate) up
// of rows that alternate 16 gate and 16 up rows (a warp owns one of each); a bfloat16 row in and out (the output head of the W4A8 decoders;
// this file is part of both libraries).
#include "mix_common.cuh"

namespace scmx {

struct GvArgs {
    const void* W;          // [N, ldw], zero padded to a multiple of 8 columns
    const float* x;         // [K]
    float* out;             // [N]
    int64_t ldw;
    int N, K, ks;           // ks: warps that share a row (1, 2, 4 or 8)
    float a_pos, a_neg;     // xIELU
    const float *cw, *cb;   // convolution weights [C, taps] and bias [C]
    float* tail;            // [C, taps - 1]
    int C, taps;
    const bf16_t* xh;       // EPI 4: the input row in bfloat16, and the outputs if outh is given
    bf16_t* outh;
    // The input row may be one that the sublayers before leave in parts (pro): 1: r = x + mult y, input r / rms(r) nw;
    // 2: r = x + nw y / rms(y), then with n > 0 the weighted sum of n - 1 stored rows and r, input r, or r / rms(r) fw.
    int pro, n, keep;       // keep: r goes to row n - 1 of the store before it is averaged
    float mult, eps;
    const float *y, *nw, *dwa, *fw;
    float *store, *x_out;   // x_out: r (not normalized), written by the first CTA, or null
    int64_t store_stride;
};

constexpr int GV_ROWS = 2;
constexpr int GV_PRO_MAXK = 2048;      // two 16-byte pieces per thread; wider rows are joined by the row kernels

// Weights are read once a token and are more than L2 holds in a model of some size: they leave it first, so that what a step comes back to (kernel
// code, states, caches, activations) stays.  Without it kernels that run once a token began with a cold start of several us: generation of 8
// tokens 1589 -> 1482 us (hybrid, width 2048), 1559 -> 1415 us (fabezen, width 1024).
__device__ __forceinline__ uint64_t first_out() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint4 load_w(const void* p, uint64_t policy) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p), "l"(policy));
    return v;
}

template <typename T> struct Vec8;
template <> struct Vec8<bf16_t> {
    uint4 w;
    __device__ __forceinline__ void load(const bf16_t* p, uint64_t policy) { w = load_w(p, policy); }
    __device__ __forceinline__ void zero() { w = make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ float dot(float4 lo, float4 hi, float s) const {
        s = fmaf(bf16_lo(w.x), lo.x, s); s = fmaf(bf16_hi(w.x), lo.y, s); s = fmaf(bf16_lo(w.y), lo.z, s); s = fmaf(bf16_hi(w.y), lo.w, s);
        s = fmaf(bf16_lo(w.z), hi.x, s); s = fmaf(bf16_hi(w.z), hi.y, s); s = fmaf(bf16_lo(w.w), hi.z, s); s = fmaf(bf16_hi(w.w), hi.w, s);
        return s;
    }
};
template <> struct Vec8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p, uint64_t policy) {
        const uint4 u = load_w(p, policy), v = load_w(p + 4, policy);
        a = make_float4(__uint_as_float(u.x), __uint_as_float(u.y), __uint_as_float(u.z), __uint_as_float(u.w));
        b = make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
    }
    __device__ __forceinline__ void zero() { a = b = make_float4(0, 0, 0, 0); }
    __device__ __forceinline__ float dot(float4 lo, float4 hi, float s) const {
        s = fmaf(a.x, lo.x, s); s = fmaf(a.y, lo.y, s); s = fmaf(a.z, lo.z, s); s = fmaf(a.w, lo.w, s);
        s = fmaf(b.x, hi.x, s); s = fmaf(b.y, hi.y, s); s = fmaf(b.z, hi.z, s); s = fmaf(b.w, hi.w, s);
        return s;
    }
};

// The residual and norm kernels between two products cost 2 - 5 us each in a chain of single rows, nearly all of it latency.  Every CTA computes
// the whole row itself while its first weights arrive: a few reads from L2 and one or two sums over the CTA.
__device__ __forceinline__ void gv_prologue(const GvArgs& a, float4* xs, int nv, float* red) {
    const int tid = threadIdx.x, quads = a.K >> 2;
    const bool first = blockIdx.x == 0;
    float4 r[2], w[2], s[2];
    float ss = 0.0f;
    const float self = a.pro == 2 && a.n > 0 ? a.dwa[a.n - 1] : 1.0f;
    auto sq = [](const float4& v) { return v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; };
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int i = tid + 256 * k;
        r[k] = w[k] = s[k] = make_float4(0, 0, 0, 0);
        if (i >= quads) continue;
        w[k] = ld4(a.nw + 4 * i);
        const float4 x = ld4(a.x + 4 * i), y = a.y != nullptr ? ld4(a.y + 4 * i) : make_float4(0, 0, 0, 0);
        if (a.pro == 1) {
            r[k] = a.y != nullptr ? make_float4(fmaf(a.mult, y.x, x.x), fmaf(a.mult, y.y, x.y), fmaf(a.mult, y.z, x.z), fmaf(a.mult, y.w, x.w)) : x;
            ss += sq(r[k]);
        } else {
            r[k] = y;
            ss += sq(y);
            s[k] = x;      // joined with the norm below
        }
    }
    const float inv = rms_inv_f32(block_sumf(ss, red), a.K, a.eps);
    if (a.pro == 2) {
        ss = 0.0f;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int i = tid + 256 * k;
            if (i >= quads) continue;
            r[k] = make_float4(s[k].x + r[k].x * inv * w[k].x, s[k].y + r[k].y * inv * w[k].y, s[k].z + r[k].z * inv * w[k].z, s[k].w + r[k].w * inv * w[k].w);
            if (a.n > 0) {
                float4 m = make_float4(0, 0, 0, 0);
#pragma unroll 4
                for (int j = 0; j < a.n - 1; ++j) {
                    const float c = a.dwa[j];
                    const float4 q = ld4(a.store + j * a.store_stride + 4 * i);
                    m.x += c * q.x; m.y += c * q.y; m.z += c * q.z; m.w += c * q.w;
                }
                if (a.keep && first) *reinterpret_cast<float4*>(a.store + (a.n - 1) * a.store_stride + 4 * i) = r[k];
                r[k] = make_float4(m.x + self * r[k].x, m.y + self * r[k].y, m.z + self * r[k].z, m.w + self * r[k].w);
            }
            if (a.fw != nullptr) {
                w[k] = ld4(a.fw + 4 * i);
                ss += sq(r[k]);
            }
        }
    }
    const float scale = a.pro == 1 ? inv : a.fw != nullptr ? rms_inv_f32(block_sumf(ss, red), a.K, a.eps) : 1.0f;
    const bool norm = a.pro == 1 || a.fw != nullptr;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int i = tid + 256 * k;
        if (i < 2 * nv) {
            float4 h = r[k];
            if (norm) h = make_float4(h.x * scale * w[k].x, h.y * scale * w[k].y, h.z * scale * w[k].z, h.w * scale * w[k].w);
            xs[(i & 1) * nv + (i >> 1)] = h;      // zero above K
            if (first && a.x_out != nullptr && i < quads) *reinterpret_cast<float4*>(a.x_out + 4 * i) = r[k];
        }
    }
}

template <typename T, int EPI>
__global__ void __launch_bounds__(256, 2) gemv_x_kernel(const GvArgs a) {
    constexpr int U = sizeof(T) == 2 ? 4 : 2;          // vectors per lane and row in a set
    extern __shared__ __align__(16) float4 xs[];       // [2][nv]: elements 0..3 and 4..7 of every vector of 8
    __shared__ float part[2][8][GV_ROWS], red[33];
    float* ys = reinterpret_cast<float*>(xs + 2 * ((a.K + 7) >> 3));      // EPI 2: products of this CTA's rows
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nv = (a.K + 7) >> 3, ks = a.ks, team = warp / ks, slice = warp - team * ks, teams = 8 / ks;
    const int first = slice * 32 + lane, step = 32 * ks;
    const int sets = (nv + U * step - 1) / (U * step);                 // of a row pair
    // row pairs of this CTA: equal shares, dealt to its teams in turn
    const int all = (a.N + GV_ROWS - 1) / GV_ROWS;
    const int base = (int)((int64_t)all * blockIdx.x / gridDim.x), pairs = (int)((int64_t)all * (blockIdx.x + 1) / gridDim.x);
    const int p0 = base + team, pstep = teams;
    const T* W = static_cast<const T*>(a.W);
    auto row_of = [&](int r0, int r) { return EPI == 3 ? 32 * (r0 >> 5) + ((r0 >> 1) & 15) + 16 * r : r0 + r; };
    using Set = Vec8<T>[GV_ROWS][U];
    const uint64_t policy = first_out();
    Set wa, wb;
    // the next set to load: of pair lp (done at pairs), from vector lv on
    int lp = p0, lv = first;
    auto fetch = [&](Set& w) {
        const bool on = lp < pairs;
        const int r0 = lp * GV_ROWS;
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int r = 0; r < GV_ROWS; ++r) {
                const int v = lv + u * step;
                if (on && v < nv && r0 + r < a.N) w[r][u].load(W + (int64_t)row_of(r0, r) * a.ldw + 8 * (int64_t)v, policy);
                else w[r][u].zero();
            }
        lv += U * step;
        if (lv - first >= sets * U * step) {
            lv = first;
            lp += pstep;
        }
    };
    fetch(wa);
    fetch(wb);
    pdl_wait();
    if (EPI == 4) {
        for (int v = tid; v < nv; v += 256) {
            float x[8];
            ld8(a.xh + 8 * v, x);
            xs[v] = make_float4(x[0], x[1], x[2], x[3]);
            xs[nv + v] = make_float4(x[4], x[5], x[6], x[7]);
        }
    } else if (a.pro != 0) {
        gv_prologue(a, xs, nv, red);
    } else if ((a.K & 3) == 0 && ((uintptr_t)a.x & 15) == 0) {
#pragma unroll 8
        for (int i = tid; i < 2 * nv; i += 256)
            xs[(i & 1) * nv + (i >> 1)] = 4 * i < a.K ? *reinterpret_cast<const float4*>(a.x + 4 * i) : make_float4(0, 0, 0, 0);
    } else {
        for (int i = tid; i < nv * 8; i += 256) {
            const float x = i < a.K ? a.x[i] : 0.0f;
            reinterpret_cast<float*>(xs + ((i >> 2) & 1) * nv + (i >> 3))[i & 3] = x;
        }
    }
    __syncthreads();
    float s[GV_ROWS] = {};
    int cp = p0, cv = first, turn = 0;
    auto finish = [&]() {                               // row pair cp is summed
        const int r0 = cp * GV_ROWS;
#pragma unroll
        for (int r = 0; r < GV_ROWS; ++r) s[r] = warp_sumf(s[r]);
        if (ks > 1) {
            if (lane == 0)
#pragma unroll
                for (int r = 0; r < GV_ROWS; ++r) part[turn][warp][r] = s[r];
            // the team's warps meet once per pair; two sets of sums, so that the next pair's are not written over these
            asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "r"(32 * ks) : "memory");
            if (slice == 0)
#pragma unroll
                for (int r = 0; r < GV_ROWS; ++r) {
                    s[r] = 0.0f;
                    for (int i = 0; i < ks; ++i) s[r] += part[turn][warp + i][r];
                }
            turn ^= 1;
        }
        if (slice == 0) {
            if (EPI == 3) {
                if (lane == 0) a.out[r0 >> 1] = gelu_tanh_f32(s[0]) * s[1];
            } else {
                const int row = r0 + lane;
                if (lane < GV_ROWS && row < a.N) {
                    float y = lane == 0 ? s[0] : s[1];
                    if (EPI == 1) y = xielu_f32(y, a.a_pos, a.a_neg);
                    if (EPI == 4 && a.outh != nullptr) a.outh[row] = f32_to_bf16(y);
                    else if (EPI == 2 && row < a.C) ys[row - GV_ROWS * base] = y;
                    else a.out[row] = y;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < GV_ROWS; ++r) s[r] = 0.0f;
    };
    auto consume = [&](Set& w) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int v = cv + u * step;
            if (v < nv) {
                const float4 lo = xs[v], hi = xs[nv + v];
#pragma unroll
                for (int r = 0; r < GV_ROWS; ++r) s[r] = w[r][u].dot(lo, hi, s[r]);
            }
        }
        if (lp < pairs) fetch(w);
        cv += U * step;
        if (cv - first >= sets * U * step) {
            finish();
            cv = first;
            cp += pstep;
        }
    };
    while (cp < pairs) {
        consume(wa);
        if (cp >= pairs) break;
        consume(wb);
    }
    if (EPI == 2) {
        // the convolution of all rows at once: its loads would otherwise be a chain in every row pair (33 MB of weights: 14 us, then 9)
        __syncthreads();
        const int row = GV_ROWS * base + tid;
        for (int r = row; r < min(GV_ROWS * pairs, a.C); r += 256) {
            const float y = ys[r - GV_ROWS * base];
            const float* cw = a.cw + (int64_t)r * a.taps;
            float* tl = a.tail + (int64_t)r * (a.taps - 1);
            float c = fmaf(cw[a.taps - 1], y, a.cb == nullptr ? 0.0f : a.cb[r]);
            for (int j = 0; j < a.taps - 1; ++j) {
                c = fmaf(cw[j], tl[j], c);
                tl[j] = j + 1 < a.taps - 1 ? tl[j + 1] : y;
            }
            a.out[r] = silu_f32(c);
        }
    }
}

template <typename T>
static int run_gemv(GvArgs a, int epi, cudaStream_t st) {
    constexpr int U = sizeof(T) == 2 ? 4 : 2;
    const int nv = (a.K + 7) / 8;
    SCMX_REQUIRE(nv * 32 <= 200 * 1024, SCMX_ELIMIT, "gemv_x: K=%d", a.K);
    // Persistent CTAs: x is staged once per CTA, and as many as stay resident (registers: two per SM) leave no wave of new ones that starts
    // with nothing in flight.  Rows are shared by as many warps as still fill a set of loads each.
    const int resident = (nv * 32 + 4096) * 2 <= 220 * 1024 ? 2 : 1;
    int ks = 1;
    while (ks < 8 && nv >= 2 * ks * 32 * U) ks *= 2;
    a.ks = ks;
    const int rows = 8 / ks * GV_ROWS, groups = (a.N + rows - 1) / rows, most = resident * sm_count();
    const dim3 grid((unsigned)(groups < most ? groups : most)), block(256);
    const size_t smem = (size_t)nv * 32 + (epi == 2 ? (size_t)4 * GV_ROWS * ((a.N / GV_ROWS + 1) / grid.x + 2) : 0);
    SCMX_REQUIRE(smem <= 220 * 1024, SCMX_ELIMIT, "gemv_x: N=%d K=%d", a.N, a.K);
    auto kernel = epi == 0 ? gemv_x_kernel<T, 0> : epi == 1 ? gemv_x_kernel<T, 1> : epi == 2 ? gemv_x_kernel<T, 2> : epi == 3 ? gemv_x_kernel<T, 3> : gemv_x_kernel<bf16_t, 4>;
    if (smem > 40 * 1024) SCMX_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    SCMX_PDL_OK("gemv_x_kernel", launch_pdl(kernel, grid, block, smem, st, a));
    return SCMX_OK;
}

}  // namespace scmx

using namespace scmx;

static int gemv_x(const void* W, int64_t ldw, int dt, const float* x, int64_t N, int64_t K, int epi, float a_pos, float a_neg, const float* conv_w,
                  const float* conv_b, float* tail, int C, int taps, float* out, GvArgs a, void* stream) {
    SCMX_DT_OK("gemv_x", dt);
    SCMX_REQUIRE(W && x && out && N > 0 && K > 0 && N < (1ll << 30) && K < (1ll << 30), SCMX_EINVAL, "gemv_x: N=%lld K=%lld", (long long)N, (long long)K);
    SCMX_REQUIRE(ldw % 8 == 0 && ldw >= K && ((uintptr_t)W & 15) == 0, SCMX_EINVAL, "gemv_x: row pitch %lld", (long long)ldw);
    SCMX_REQUIRE(epi >= 0 && epi <= 3 && (epi != 3 || N % 32 == 0), SCMX_EINVAL, "gemv_x: epi=%d on %lld rows", epi, (long long)N);
    SCMX_REQUIRE(epi != 2 || (conv_w && C > 0 && C <= N && taps >= 1 && (taps == 1 || tail)), SCMX_EINVAL, "gemv_x: convolution epilogue");
    a.W = W; a.x = x; a.out = out; a.ldw = ldw; a.N = (int)N; a.K = (int)K; a.ks = 1; a.a_pos = a_pos; a.a_neg = a_neg;
    a.cw = conv_w; a.cb = conv_b; a.tail = tail; a.C = C; a.taps = taps;
    return dt == 0 ? run_gemv<bf16_t>(a, epi, (cudaStream_t)stream) : run_gemv<float>(a, epi, (cudaStream_t)stream);
}

extern "C" int scmx_gemv_x(const void* W, int64_t ldw, int dt, const float* x, int64_t N, int64_t K, int epi, float a_pos, float a_neg,
                           const float* conv_w, const float* conv_b, float* tail, int C, int taps, float* out, void* stream) {
    return gemv_x(W, ldw, dt, x, N, K, epi, a_pos, a_neg, conv_w, conv_b, tail, C, taps, out, GvArgs{}, stream);
}

extern "C" int scmx_gemv_x_row(const void* W, int64_t ldw, int dt, const float* x, const float* y, const float* nw, int pro, float mult, float eps,
                               float* store, int64_t store_stride, const float* dwa, int n, int keep, const float* fw, float* x_out, int64_t N,
                               int64_t K, int epi, float a_pos, float a_neg, const float* conv_w, const float* conv_b, float* tail, int C, int taps,
                               float* out, void* stream) {
    SCMX_REQUIRE((pro == 1 || (pro == 2 && y)) && nw && K <= GV_PRO_MAXK && K % 4 == 0, SCMX_EINVAL, "gemv_x_row: pro=%d K=%lld", pro, (long long)K);
    SCMX_REQUIRE(n >= 0 && (n == 0 || (pro == 2 && store && dwa && store_stride >= K && store_stride % 4 == 0)), SCMX_EINVAL,
                 "gemv_x_row: average over %d results without a store", n);
    SCMX_REQUIRE(x_out == nullptr || (x_out != x && x_out != y && x_out != out), SCMX_EINVAL, "gemv_x_row: the new row needs a place of its own");
    SCMX_REQUIRE((((uintptr_t)x | (uintptr_t)y | (uintptr_t)nw | (uintptr_t)store | (uintptr_t)fw | (uintptr_t)x_out) & 15) == 0, SCMX_EINVAL,
                 "gemv_x_row: rows must be 16-byte aligned");
    GvArgs a = {};
    a.pro = pro; a.n = n; a.keep = keep; a.mult = mult; a.eps = eps; a.y = y; a.nw = nw; a.dwa = dwa; a.fw = pro == 2 ? fw : nullptr;
    a.store = store; a.x_out = x_out; a.store_stride = store_stride;
    return gemv_x(W, ldw, dt, x, N, K, epi, a_pos, a_neg, conv_w, conv_b, tail, C, taps, out, a, stream);
}

// Rows of up to 6400 values.  Callers send wider ones to the products they used before, although a stream is ahead there too (4096 x 12288: 22 us, 31 us as a tile of 128 rows).
static int row_product(const uint16_t* W, int64_t ldw, const uint16_t* x, int64_t N, int64_t K, void* out, int out_f32, void* stream) {
    SCMX_REQUIRE(W && x && out && N > 0 && K > 0 && N < (1ll << 30) && K % 8 == 0 && ldw % 8 == 0 && ldw >= K, SCMX_EINVAL, "row product: N=%lld K=%lld pitch %lld",
                 (long long)N, (long long)K, (long long)ldw);
    SCMX_REQUIRE((((uintptr_t)W | (uintptr_t)x) & 15) == 0 && K <= 6400, SCMX_ELIMIT, "row product: 16-byte aligned rows of at most 6400 (K=%lld)", (long long)K);
    GvArgs a = {};
    a.W = W; a.ldw = ldw; a.N = (int)N; a.K = (int)K; a.ks = 1; a.xh = x;
    if (out_f32) a.out = static_cast<float*>(out);
    else a.outh = static_cast<bf16_t*>(out);
    return run_gemv<bf16_t>(a, 4, (cudaStream_t)stream);
}

// One product under two names: scmx.h declares scmx_head_bf16, scmx_mixers.h declares scmx_gemv_bf16.
extern "C" int scmx_head_bf16(const uint16_t* W, int64_t ldw, const uint16_t* x, int64_t N, int64_t K, uint16_t* out, void* stream) {
    return row_product(W, ldw, x, N, K, out, 0, stream);
}

extern "C" int scmx_gemv_bf16(const void* W, int64_t ldw, const void* x, int64_t N, int64_t K, void* out, int out_f32, void* stream) {
    return row_product((const uint16_t*)W, ldw, (const uint16_t*)x, N, K, out, out_f32, stream);
}
