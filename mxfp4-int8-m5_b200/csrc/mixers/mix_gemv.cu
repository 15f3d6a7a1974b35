// Matrix-vector product of the decode step: out [N] = W [N, K] x, weights bfloat16 or float, x and out float32, float32
// accumulation.  Epilogues: none; xIELU; the causal convolution + SiLU of the first C rows, whose carried inputs are shifted in place;
// gelu(gate) up of rows that alternate 16 gate and 16 up rows (a warp owns one of each); a bfloat16 row in and out (the output head of
// the W4A8 decoders; this file is part of both libraries).
//
// Bound by the weights' bytes and by the latency of a link of the chain.  Every lane streams its pieces of the row pairs of its warp through a ring
// of its own in shared memory (16-byte asynchronous copies, nothing shared and no barrier), filled before the kernel waits for its predecessor:
// weights never change.  A CTA holds half of an SM's shared memory and few registers, so two products of a chain are resident together and the
// next one's first 14 MB arrive while this one waits for its input, joins its row or reduces.  16 warps and two products an instruction: with 8 warps
// a chunk's chain of dependent instructions, not memory, set the rate (131 MB 26 us; 33 us with one product an instruction).  Bulk copies of 2 KB, one
// thread issuing for a warp, took a quarter longer than these copies.  With the weights in registers (two CTAs that filled the register file) memory stood still
// between kernels: generation of 8 tokens 1486 -> 1280 us (hybrid, width 2048), 1445 -> 1229 us (fabezen, width 1024); the output head of 32000 x 2048
// 27 -> 19.8 us in a chain of its own, 6.6 TB/s.
#include "mix_common.cuh"

namespace scmx {

struct GvArgs {
    const void* W;          // [N, ldw], zero padded to a multiple of 8 columns
    const float* x;         // [K]
    float* out;             // [N]
    int64_t ldw;
    int N, K, ks;           // ks: warps that share a row (1, 2, 4, 8 or 16)
    int warps, slots;       // warps that stream weights, slots of a warp's ring
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
constexpr int GV_U = 2, GV_CP = 32 * GV_U, GV_SLOT = GV_ROWS * 16 * GV_CP;      // 16-byte pieces of a row per lane and per slot, bytes of a slot
constexpr int GV_MAX_SLOTS = 3;
constexpr int GV_THREADS = 512, GV_WARPS = GV_THREADS / 32;
constexpr int GV_PRO_MAXK = 2048;      // a 16-byte piece per thread; wider rows are joined by the row kernels

// Weights are read once a token and are more than L2 holds in a model of some size: they leave it first, so that what a step comes back to (kernel
// code, states, caches, activations) stays.  Without it kernels that run once a token began with a cold start of several us: generation of 8
// tokens 1589 -> 1482 us (hybrid, width 2048), 1559 -> 1415 us (fabezen, width 1024).
__device__ __forceinline__ uint64_t first_out() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ void copy_w(uint32_t dst, const void* src, uint64_t policy) {
    asm volatile("cp.async.cg.shared.global.L2::cache_hint [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "l"(policy) : "memory");
}
__device__ __forceinline__ void copies_end() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// At most n - 1 of the thread's groups of copies are still on their way.
__device__ __forceinline__ void copies_wait(int n) {
    if (n == 3) asm volatile("cp.async.wait_group 2;" ::: "memory");
    else if (n == 2) asm volatile("cp.async.wait_group 1;" ::: "memory");
    else asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The row in shared memory, in float4: with bfloat16 weights a 16-byte piece meets two of them, kept nv apart so that the lanes of a load are neighbours.
template <typename T> __device__ __forceinline__ int x_place(int i, int nv);
template <> __device__ __forceinline__ int x_place<bf16_t>(int i, int nv) { return (i & 1) * nv + (i >> 1); }
template <> __device__ __forceinline__ int x_place<float>(int i, int) { return i; }
// s += piece i of a row times x, two products per instruction (even and odd elements in the halves of s).
template <typename T> __device__ __forceinline__ uint64_t dot_piece(const uint4& w, const ulonglong2* x, int nv, int i, uint64_t s);
__device__ __forceinline__ uint64_t bf16_pair(uint32_t w) { return pack2(bf16_lo(w), bf16_hi(w)); }
template <> __device__ __forceinline__ uint64_t dot_piece<bf16_t>(const uint4& w, const ulonglong2* x, int nv, int i, uint64_t s) {
    const ulonglong2 lo = x[i], hi = x[nv + i];
    s = fma2(bf16_pair(w.x), lo.x, s); s = fma2(bf16_pair(w.y), lo.y, s);
    s = fma2(bf16_pair(w.z), hi.x, s); return fma2(bf16_pair(w.w), hi.y, s);
}
template <> __device__ __forceinline__ uint64_t dot_piece<float>(const uint4& w, const ulonglong2* x, int, int i, uint64_t s) {
    const ulonglong2 v = x[i];
    s = fma2(pack2(__uint_as_float(w.x), __uint_as_float(w.y)), v.x, s);
    return fma2(pack2(__uint_as_float(w.z), __uint_as_float(w.w)), v.y, s);
}

// The residual and norm kernels between two products cost 2 - 5 us each in a chain of single rows, nearly all of it latency.  Every CTA computes
// the whole row itself while its first weights arrive: a few reads from L2 and one or two sums over the CTA.
template <typename T>
__device__ __forceinline__ void gv_prologue(const GvArgs& a, float4* xs, int nv, float* red) {
    const int tid = threadIdx.x, quads = a.K >> 2;
    const bool first = blockIdx.x == 0;
    constexpr int PIECES = GV_PRO_MAXK / 4 / GV_THREADS;
    float4 r[PIECES], w[PIECES], s[PIECES];
    float ss = 0.0f;
    const float self = a.pro == 2 && a.n > 0 ? a.dwa[a.n - 1] : 1.0f;
    auto sq = [](const float4& v) { return v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w; };
#pragma unroll
    for (int k = 0; k < PIECES; ++k) {
        const int i = tid + GV_THREADS * k;
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
        for (int k = 0; k < PIECES; ++k) {
            const int i = tid + GV_THREADS * k;
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
    for (int k = 0; k < PIECES; ++k) {
        const int i = tid + GV_THREADS * k;
        if (i < 2 * nv) {
            float4 h = r[k];
            if (norm) h = make_float4(h.x * scale * w[k].x, h.y * scale * w[k].y, h.z * scale * w[k].z, h.w * scale * w[k].w);
            xs[x_place<T>(i, nv)] = h;      // zero above K
            if (first && a.x_out != nullptr && i < quads) *reinterpret_cast<float4*>(a.x_out + 4 * i) = r[k];
        }
    }
}

template <typename T, int EPI>
__global__ void __launch_bounds__(GV_THREADS, 2) gemv_x_kernel(const GvArgs a) {
    constexpr int PER = 16 / sizeof(T);                // values of a 16-byte piece
    // x: 2 nv float4 | partial sums of every (pair, slice) | the warps' rings (128-byte aligned)
    extern __shared__ __align__(128) float4 xs[];
    __shared__ float red[33];
    pdl_launch_dependents();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nv = (a.K + 7) >> 3, np = nv * (8 / PER), ks = a.ks, team = warp / ks, slice = warp - team * ks, teams = a.warps / ks;
    const int slots = a.slots, chunks = (np + GV_CP - 1) / GV_CP;
    // row pairs of this CTA: equal shares, dealt to its teams in turn; a team's warps share the chunks of a row
    const int all = (a.N + GV_ROWS - 1) / GV_ROWS;
    const int base = (int)((int64_t)all * blockIdx.x / gridDim.x), pairs = (int)((int64_t)all * (blockIdx.x + 1) / gridDim.x);
    const int c_lo = chunks * slice / ks, c_hi = chunks * (slice + 1) / ks;
    float* part = reinterpret_cast<float*>(xs + 2 * nv);      // [pairs - base][ks][GV_ROWS]
    const int part_bytes = ((int)((all + gridDim.x - 1) / gridDim.x) * ks * GV_ROWS * 4 + 127) & ~127;
    const uint8_t* ring = reinterpret_cast<uint8_t*>(xs) + ((32 * nv + 127) & ~127) + part_bytes + (size_t)warp * slots * GV_SLOT + 16 * lane;
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring), ring_end = ring_s + slots * GV_SLOT;
    const uint64_t policy = first_out();
    auto row_of = [&](int p, int r) {                  // past the end (N odd): the last row again, its sum is not used
        const int r0 = p * GV_ROWS;
        return EPI == 3 ? 32 * (r0 >> 5) + ((r0 >> 1) & 15) + 16 * r : min(r0 + r, a.N - 1);
    };
    // the next chunk to request: of pair ip, number ic; every request is one group of copies, empty ones past the end
    const int p_first = warp < a.warps ? base + team : pairs;
    int ip = p_first, ic = c_lo;
    const uint8_t *g0 = nullptr, *g1 = nullptr;
    auto row_start = [&]() {
        const int64_t pitch = a.ldw * (int64_t)sizeof(T);
        const uint8_t* w = static_cast<const uint8_t*>(a.W) + (int64_t)c_lo * (16 * GV_CP) + 16 * lane;
        g0 = w + row_of(ip, 0) * pitch;
        g1 = w + row_of(ip, 1) * pitch;
    };
    auto request = [&](uint32_t dst) {
        if (ip < pairs) {
            const int left = np - ic * GV_CP - lane;
#pragma unroll
            for (int u = 0; u < GV_U; ++u)
                if (32 * u < left) {
                    copy_w(dst + 512 * u, g0 + 512 * u, policy);
                    copy_w(dst + 512 * (GV_U + u), g1 + 512 * u, policy);
                }
            g0 += 16 * GV_CP;
            g1 += 16 * GV_CP;
            if (++ic == c_hi) {
                ic = c_lo;
                ip += teams;
                if (ip < pairs) row_start();
            }
        }
        copies_end();
    };
    if (ip < pairs) row_start();
    for (int i = 0; i < slots; ++i) request(ring_s + i * GV_SLOT);
    // the convolution's weights of row `tid` of this CTA (EPI 2)
    const int crow = GV_ROWS * base + tid, rows_end = min(GV_ROWS * pairs, a.N);
    constexpr int RT = 4;                              // taps that a thread keeps in registers
    const bool conv_early = EPI == 2 && a.taps <= RT && crow < min(rows_end, a.C);
    float cw[RT], tl[RT], cb = 0.0f;
    if (conv_early) {
#pragma unroll
        for (int j = 0; j < RT; ++j) cw[j] = j < a.taps ? a.cw[(int64_t)crow * a.taps + j] : 0.0f;
        cb = a.cb == nullptr ? 0.0f : a.cb[crow];
    }
    pdl_wait();
    if (conv_early) {
#pragma unroll
        for (int j = 0; j < RT; ++j) tl[j] = j < a.taps - 1 ? a.tail[(int64_t)crow * (a.taps - 1) + j] : 0.0f;
    }
    if (EPI == 4) {
        for (int v = tid; v < nv; v += GV_THREADS) {
            float x[8];
            ld8(a.xh + 8 * v, x);
            xs[x_place<T>(2 * v, nv)] = make_float4(x[0], x[1], x[2], x[3]);
            xs[x_place<T>(2 * v + 1, nv)] = make_float4(x[4], x[5], x[6], x[7]);
        }
    } else if (a.pro != 0) {
        gv_prologue<T>(a, xs, nv, red);
    } else if ((a.K & 3) == 0 && ((uintptr_t)a.x & 15) == 0) {
#pragma unroll 8
        for (int i = tid; i < 2 * nv; i += GV_THREADS)
            xs[x_place<T>(i, nv)] = 4 * i < a.K ? *reinterpret_cast<const float4*>(a.x + 4 * i) : make_float4(0, 0, 0, 0);
    } else {
        for (int i = tid; i < nv * 8; i += GV_THREADS) {
            const float x = i < a.K ? a.x[i] : 0.0f;
            reinterpret_cast<float*>(xs + x_place<T>(i >> 2, nv))[i & 3] = x;
        }
    }
    __syncthreads();
    const ulonglong2* x2 = reinterpret_cast<const ulonglong2*>(xs);
    uint32_t at = ring_s;
    const uint8_t* w_at = ring;
    for (int p = p_first; p < pairs; p += teams) {
        uint64_t s0 = 0, s1 = 0;                       // two float32 sums each
        for (int c = c_lo; c < c_hi; ++c) {
            copies_wait(slots);
            const int i = c * GV_CP + lane;
#pragma unroll
            for (int u = 0; u < GV_U; ++u)
                if (i + 32 * u < np) {
                    s0 = dot_piece<T>(*reinterpret_cast<const uint4*>(w_at + 512 * u), x2, nv, i + 32 * u, s0);
                    s1 = dot_piece<T>(*reinterpret_cast<const uint4*>(w_at + 512 * (GV_U + u)), x2, nv, i + 32 * u, s1);
                }
            request(at);
            at += GV_SLOT;
            w_at += GV_SLOT;
            if (at == ring_end) {
                at = ring_s;
                w_at = ring;
            }
        }
        const float2 a0 = unpack2(s0), a1 = unpack2(s1);
        const float t0 = warp_sumf(a0.x + a0.y), t1 = warp_sumf(a1.x + a1.y);
        if (lane < GV_ROWS) part[((p - base) * ks + slice) * GV_ROWS + lane] = lane == 0 ? t0 : t1;
    }
    __syncthreads();
    auto total = [&](int i) {                          // row i of this CTA, in the order of its pairs
        float y = 0.0f;
        for (int k = 0; k < ks; ++k) y += part[((i >> 1) * ks + k) * GV_ROWS + (i & 1)];
        return y;
    };
    if (EPI == 3) {
        for (int i = tid; i < pairs - base; i += GV_THREADS) a.out[base + i] = gelu_tanh_f32(total(2 * i)) * total(2 * i + 1);
        return;
    }
    for (int row = crow; row < rows_end; row += GV_THREADS) {
        float y = total(row - GV_ROWS * base);
        if (EPI == 1) y = xielu_f32(y, a.a_pos, a.a_neg);
        if (EPI == 4 && a.outh != nullptr) {
            a.outh[row] = f32_to_bf16(y);
        } else if (EPI == 2 && row < a.C) {
            float* t = a.tail + (int64_t)row * (a.taps - 1);
            if (conv_early && row == crow) {
                float c = cb;
#pragma unroll
                for (int j = 0; j < RT; ++j) c = j == a.taps - 1 ? fmaf(cw[j], y, c) : c;
#pragma unroll
                for (int j = 0; j < RT; ++j)
                    if (j < a.taps - 1) {
                        c = fmaf(cw[j], tl[j], c);
                        t[j] = j + 1 < a.taps - 1 ? tl[j + 1 < RT ? j + 1 : 0] : y;
                    }
                a.out[row] = silu_f32(c);
            } else {
                const float* w = a.cw + (int64_t)row * a.taps;
                float c = fmaf(w[a.taps - 1], y, a.cb == nullptr ? 0.0f : a.cb[row]);
                for (int j = 0; j < a.taps - 1; ++j) {
                    c = fmaf(w[j], t[j], c);
                    t[j] = j + 1 < a.taps - 1 ? t[j + 1] : y;
                }
                a.out[row] = silu_f32(c);
            }
        } else {
            a.out[row] = y;
        }
    }
}

template <typename T>
static int run_gemv(GvArgs a, int epi, cudaStream_t st) {
    const int nv = (a.K + 7) / 8, np = nv * (int)sizeof(T) / 2, x_bytes = (nv * 32 + 127) & ~127;
    SCMX_REQUIRE(nv * 32 <= 200 * 1024, SCMX_ELIMIT, "gemv_x: K=%d", a.K);
    // One persistent CTA per SM, more where a CTA would have over 512 row pairs (its sums are kept in shared memory to the end).
    const int all = (a.N + GV_ROWS - 1) / GV_ROWS, sms = sm_count();
    const int by_rows = (all + 511) / 512, grid = by_rows > sms ? by_rows : all < sms ? all : sms;
    const int ppc = (all + grid - 1) / grid;
    // Rows are shared by the warps where that shortens the longest queue of chunks.
    a.warps = x_bytes <= 184 * 1024 ? GV_WARPS : 4;                // very long rows leave room for few rings
    const int chunks = (np + GV_CP - 1) / GV_CP;
    int best = 1 << 30;
    for (int k = 1; k <= a.warps && k <= chunks && ppc * k <= 1024; k *= 2) {
        const int per = a.warps / k, cost = ((ppc + per - 1) / per) * ((chunks + k - 1) / k);
        if (cost < best) {
            best = cost;
            a.ks = k;
        }
    }
    // Three slots a warp, 96 KB a CTA: with the row and the sums half of an SM, so that the next product of a chain is resident beside this one.  Long rows leave
    // fewer.
    const int part = (ppc * a.ks * GV_ROWS * 4 + 127) & ~127;
    auto ring = [&](int budget) { return (budget - x_bytes - part) / (a.warps * GV_SLOT); };
    a.slots = ring(113 * 1024) >= 2 ? ring(113 * 1024) : ring(226 * 1024);
    a.slots = a.slots > GV_MAX_SLOTS ? GV_MAX_SLOTS : a.slots < 1 ? 1 : a.slots;
    if (a.slots > best) a.slots = best;
    const size_t smem = (size_t)x_bytes + part + (size_t)a.slots * a.warps * GV_SLOT;
    SCMX_REQUIRE(smem <= 226 * 1024, SCMX_ELIMIT, "gemv_x: N=%d K=%d", a.N, a.K);
    auto kernel = epi == 0 ? gemv_x_kernel<T, 0> : epi == 1 ? gemv_x_kernel<T, 1> : epi == 2 ? gemv_x_kernel<T, 2> : epi == 3 ? gemv_x_kernel<T, 3> : gemv_x_kernel<bf16_t, 4>;
    static bool configured[64][5] = {};
    const int dev = current_device();
    SCMX_REQUIRE(dev >= 0, SCMX_ECUDA, "no current CUDA device (ordinal 0..63)");
    if (!configured[dev][epi]) {
        SCMX_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024));
        configured[dev][epi] = true;
    }
    SCMX_PDL_OK("gemv_x_kernel", launch_pdl(kernel, dim3((unsigned)grid), dim3(GV_THREADS), smem, st, a));
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
