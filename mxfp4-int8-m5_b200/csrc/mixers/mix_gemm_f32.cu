// float32 GEMM, out = A [M, K] . W [N, K]^T, on tcgen05.mma kind::f16: every operand value is the sum of three bfloat16 parts (8 bits of mantissa
// each), and the six part products above 2^-24 of the whole are summed.  Rows of both operands are taken times a power of two that brings their largest
// value into [1, 2), so the parts are exact down to 2^-110 of it (bfloat16 has no more exponents; unscaled, values below 2^-110 would lose bits) and
// nothing overflows on the way; the epilogue scales back.
// The tensor core's float32 accumulator cuts bits off instead of rounding: an error with a sign, which grows with the number of instructions that
// add to it and which a scan over hundreds of tokens adds up.  Therefore the products of the leading parts have an accumulator of their own (the other
// five are 2^-8 of it), an accumulator takes 64 values of K, and the epilogue warps add both to float32 registers, rounded to nearest.
// Error against 64-bit sums (2-norm, normal operands), K = 1024 / 2048 / 6144: 1.2e-7 / 1.6e-7 / 2.6e-7, mean -5e-8; with accumulators of 256 values
// 2.4e-7 / 2.4e-7 / 2.6e-7, mean -1.9e-7; sums of CUDA-core multiply-adds 5.7e-7 / 8.1e-7 / 1.4e-6, mean 0; accumulators over the whole of K 1.0e-6 / 2.1e-6 /
// 6.7e-6.  State of the first scan after a prompt of 700 float32 tokens: 8.1e-7, with accumulators of 256 values 1.28e-6, with multiply-adds 1.0e-6.
//
// Structure of gemm_bf16 (TMA producer warp, one MMA-issuing thread, 8 epilogue warps, two accumulators, persistent tiles; CTA pairs with
// tile 256).  A stage holds the three parts of 64 values of both operands: six products use every part loaded twice.  The parts are
// written by a kernel before.
// Infinities and not-a-number values make a sum not a number here.  That is the answer where a row of either operand has a not-a-number value; the
// others are computed once more by plain multiply-adds on the float32 operands, 32 outputs of a row together.
#include "mix_tc.cuh"

namespace scmx {

int gemm_reduce(const float* part, int splits, int64_t stride, int64_t rows, int64_t ldp, int out_f32, void* out, int64_t ldo, cudaStream_t st);

struct GfArgs {
    int M, N, K;
    int part_bytes;              // bytes of one part of a row: K rounded up to 64, times 2
    int act;                     // 0: none, 1: xIELU, 2: gelu(gate) up, columns alternate 16 gate and 16 up
    float a_pos, a_neg;
    const float *A, *W;          // the operands themselves
    int64_t lda, ldw;
    const int32_t *ea, *ew;      // exponents of their rows
    int vec;                     // their rows start on 16 bytes
    float* out;
    int64_t ldo;
    int splits;                  // > 1: range s of K goes to out + s * split_stride (no activation)
    int64_t split_stride;
    int32_t* status;
    uint64_t wait_ns;
};

constexpr int GF_CHUNK = 1;                            // blocks of 64 values per accumulator (300 x 6144 x 1024: 1 us more than with 4)
constexpr int GF_PITCH = 80;                           // staged row of 16 outputs; conflict-free 16-byte stores
constexpr int GF_STAGE_WARP = 32 * GF_PITCH;

// Rows of an operand to be split: 2^-e x = p0 + p1 + p2, out [rows][3][kp], zero above K.
struct SplitRows {
    const float* x;
    int64_t ldx, rows;
    bf16_t* out;
    int32_t* e;
    int vec;                     // 16-byte loads
};

// Activations and a band of the weights in one launch; `team` warps (1, 2, 4 or 8) share a row, so that four loads a lane are a row of up to 4096.
// The weights' parts live for one call: kept ones would not follow a weight that is changed in place, and would hold 6 bytes beside every 4.
template <int V>
__device__ __forceinline__ void load_row(const float* x, int K, int c, float (&v)[V]) {
    if (V == 4) {
        const float4 q = c < K ? __ldg(reinterpret_cast<const float4*>(x + c)) : make_float4(0, 0, 0, 0);
        v[0] = q.x; v[1 % V] = q.y; v[2 % V] = q.z; v[3 % V] = q.w;
    } else {
#pragma unroll
        for (int e = 0; e < V; ++e) v[e] = c + e < K ? __ldg(x + c + e) : 0.0f;
    }
}
template <int V>
__device__ __forceinline__ void store_parts(float (&v)[V], bf16_t* o, int kp) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        uint32_t w[V / 2];
#pragma unroll
        for (int e = 0; e < V; e += 2) {
            w[e / 2] = pack_bf16x2(v[e], v[e + 1]);
            v[e] -= bf16_lo(w[e / 2]);
            v[e + 1] -= bf16_hi(w[e / 2]);
        }
        if (V == 4) *reinterpret_cast<uint2*>(o + p * kp) = make_uint2(w[0], w[(V / 2) - 1]);
        else *reinterpret_cast<uint32_t*>(o + p * kp) = w[0];
    }
}
// Largest magnitude (bits) of this thread's share of a row.
template <int V>
__device__ __forceinline__ uint32_t row_top(const float* x, int K, int at, int step) {
    uint32_t m = 0;
    for (int c0 = V * at; c0 < K; c0 += 4 * V * step) {
        float v[4][V];
#pragma unroll
        for (int i = 0; i < 4; ++i) load_row<V>(x, K, c0 + i * V * step, v[i]);
#pragma unroll
        for (int i = 0; i < 4 * V; ++i) m = max(m, __float_as_uint(v[i / V][i % V]) & 0x7FFFFFFFu);
    }
    return m;
}
// Its exponent, of subnormal numbers too; 0 for zero, infinities and not-a-number values.  GF_NAN stands for the last in a row's entry.
constexpr int GF_NAN = 1 << 16;
__device__ __forceinline__ int top_exponent(uint32_t m) {
    if (m == 0 || m >= 0x7F800000u) return 0;
    return m >= 0x00800000u ? (int)(m >> 23) - 127 : 31 - __clz((int)m) - 149;
}
template <int V>
__device__ __forceinline__ void split_row(const float* x, int K, int kp, bf16_t* o, int at, int step, int exp) {
    const int half = exp >> 1;      // -149 .. 127: 2^-exp in two factors
    const float f1 = __int_as_float((127 - half) << 23), f2 = __int_as_float((127 - (exp - half)) << 23);
    for (int c0 = V * at; c0 < kp; c0 += 4 * V * step) {
        float v[4][V];
#pragma unroll
        for (int i = 0; i < 4; ++i) load_row<V>(x, K, c0 + i * V * step, v[i]);
#pragma unroll
        for (int i = 0; i < 4 * V; ++i) v[i / V][i % V] *= f1;
#pragma unroll
        for (int i = 0; i < 4 * V; ++i) v[i / V][i % V] *= f2;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if (c0 + i * V * step < kp) store_parts<V>(v[i], o + c0 + i * V * step, kp);
    }
}
__global__ void __launch_bounds__(256) split3_kernel(const SplitRows a, const SplitRows b, int K, int kp, int team) {
    __shared__ uint32_t top[8];
    pdl_launch_dependents();
    pdl_wait();
    const int warp = threadIdx.x >> 5, at = (warp & (team - 1)) * 32 + (threadIdx.x & 31);
    const int64_t g = ((int64_t)blockIdx.x * 8 + warp) / team, r = g < a.rows ? g : g - a.rows;
    const SplitRows& s = g < a.rows ? a : b;
    const bool on = r < s.rows;
    const float* x = s.x + r * s.ldx;
    uint32_t m = !on ? 0 : s.vec ? row_top<4>(x, K, at, 32 * team) : row_top<2>(x, K, at, 32 * team);
    m = __reduce_max_sync(0xffffffffu, m);
    if (team > 1) {
        if ((threadIdx.x & 31) == 0) top[warp] = m;
        __syncthreads();
        for (int i = 0; i < team; ++i) m = max(m, top[(warp & ~(team - 1)) + i]);
    }
    if (!on) return;
    const int exp = top_exponent(m);
    if (at == 0) s.e[r] = m > 0x7F800000u ? GF_NAN : exp;
    bf16_t* o = s.out + r * 3 * kp;
    if (s.vec) split_row<4>(x, K, kp, o, at, 32 * team, exp);      // the row once more, from L1 or L2
    else split_row<2>(x, K, kp, o, at, 32 * team, exp);
}

static int run_split3(SplitRows a, SplitRows b, int K, int kp, cudaStream_t st) {
    auto vec = [&](const SplitRows& s) { return K % 4 == 0 && s.ldx % 4 == 0 && ((uintptr_t)s.x & 15) == 0; };
    a.vec = vec(a);
    b.vec = vec(b);
    int team = 1;
    while (team < 8 && kp > 512 * team) team *= 2;
    SCMX_PDL_OK("split3_kernel", launch_pdl(split3_kernel, dim3((unsigned)(((a.rows + b.rows) * team + 7) / 8)), dim3(256), 0, st, a, b, K, kp, team));
    return SCMX_OK;
}

// Sums of 32 columns times the powers of two of this lane's row (ea) and of the columns (ew: of column `lane`).  Powers up to 2^60 by multiplications, which
// are exact; the others with one rounding at the ends of the number range.
__device__ __noinline__ void gf_scale_far(float* s, int ea, int ew) {
#pragma unroll 1
    for (int j = 0; j < 32; ++j) s[j] = ldexpf(s[j], ea + __shfl_sync(0xffffffffu, ew, j));
}
__device__ __forceinline__ float gf_power(int e) { return __int_as_float((e + 127) << 23); }
__device__ __forceinline__ void gf_scale(float* s, int ea, int ew) {
    if (__all_sync(0xffffffffu, abs(ea) <= 60 && abs(ew) <= 60)) {
        const float fa = gf_power(ea), fw = gf_power(ew);
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] = s[j] * fa * __shfl_sync(0xffffffffu, fw, j);
    } else {
        float t[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) t[j] = s[j];
        gf_scale_far(t, ea, ew);
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] = t[j];
    }
}

// Four values of a row from k on, zero from k1 on.
__device__ __forceinline__ float4 gf_four(const float* x, int k, int k1, int vec) {
    if (vec && k + 4 <= k1) return *reinterpret_cast<const float4*>(x + k);
    return make_float4(k < k1 ? x[k] : 0.0f, k + 1 < k1 ? x[k + 1] : 0.0f, k + 2 < k1 ? x[k + 2] : 0.0f, k + 3 < k1 ? x[k + 3] : 0.0f);
}
// Outputs col0 .. col0 + 31 of this lane's row by multiply-adds over values [k0, k1), run by whole warps that hold a sum which is not a number.  16 values of the 32
// weight rows at a time in the warp's staging area (ws); a chain of scalar loads for every output took a hundred times as long.
__device__ __noinline__ void gf_dots(const GfArgs& a, int row, int col0, int k0, int k1, float4* ws, float* out) {
    const int lane = threadIdx.x & 31, piece = 4 * (lane & 3);
    const float* x = a.A + (int64_t)min(row, a.M - 1) * a.lda;
    float s[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) s[j] = 0.0f;
#pragma unroll 1
    for (int k = k0; k < k1; k += 16) {
        float4 q[4], w[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w[i] = gf_four(a.W + (int64_t)min(col0 + 8 * i + (lane >> 2), a.N - 1) * a.ldw, k + piece, k1, a.vec);
            q[i] = gf_four(x, k + 4 * i, k1, a.vec);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i) ws[32 * i + lane] = w[i];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 32; ++j) {
                const float4 u = ws[4 * j + i];
                s[j] = fmaf(q[i].x, u.x, s[j]); s[j] = fmaf(q[i].y, u.y, s[j]); s[j] = fmaf(q[i].z, u.z, s[j]); s[j] = fmaf(q[i].w, u.w, s[j]);
            }
    }
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 32; ++j) out[j] = s[j];
}

template <int BN_, bool PAIR>
struct GfSmem {
    static constexpr int BN = BN_, STAGES = 2;
    static constexpr int ACCS = BN == 256 ? 1 : 2;          // pairs of accumulators in tensor memory
    static constexpr int A_BYTES = BM * BK;
    static constexpr int B_BYTES = (PAIR ? BN / 2 : BN) * BK;
    static constexpr int STAGE_BYTES = 3 * (A_BYTES + B_BYTES);
    static constexpr int BAR_OFF = STAGES * STAGE_BYTES;
    static constexpr int MISC_OFF = BAR_OFF + 8 * (2 * STAGES + 4);
    static constexpr int EPI_OFF = (MISC_OFF + 16 + 127) & ~127;
    static constexpr int TOTAL = EPI_OFF + EPI_WARPS * GF_STAGE_WARP + 1024;
};

template <int BN, bool PAIR>
__device__ __forceinline__ void gemm_f32_body(const CUtensorMap& tmA, const CUtensorMap& tmB, const GfArgs& a) {
    using L = GfSmem<BN, PAIR>;
    constexpr int STAGES = L::STAGES;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar_full = sbase + L::BAR_OFF, bar_empty = bar_full + 8 * STAGES;
    const uint32_t bar_tfull = bar_empty + 8 * STAGES, bar_tempty = bar_tfull + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::MISC_OFF);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::MISC_OFF + 4);
    constexpr uint32_t TMEM_COLS = 2 * BN * L::ACCS;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = PAIR ? cluster_ctarank() : 0;
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        prefetch_map(&tmA);
        prefetch_map(&tmB);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (int i = 0; i < L::ACCS; ++i) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, PAIR ? 2 * EPI_WARPS : EPI_WARPS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        if (PAIR) {
            tmem_alloc2(smem_u32(tmem_slot), TMEM_COLS);
            tmem_relinquish2();
        } else {
            tmem_alloc(smem_u32(tmem_slot), TMEM_COLS);
            tmem_relinquish();
        }
    }
    pdl_launch_dependents();
    tc_fence_before();
    __syncthreads();
    if (PAIR) cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_wait();

    const uint32_t full_leader = PAIR ? mapa_u32(bar_full, 0) : bar_full;
    const uint32_t tempty_leader = PAIR ? mapa_u32(bar_tempty, 0) : bar_tempty;
    constexpr int TM_ROWS = PAIR ? 2 * BM : BM;
    const int worker = PAIR ? blockIdx.x >> 1 : blockIdx.x, nworkers = PAIR ? gridDim.x >> 1 : gridDim.x;
    const int tiles_m = (a.M + TM_ROWS - 1) / TM_ROWS, tiles_n = (a.N + BN - 1) / BN;
    const int per_split = tiles_m * tiles_n, total = per_split * a.splits;
    const int all_kb = a.part_bytes / BK, chunks = (all_kb + GF_CHUNK - 1) / GF_CHUNK;
    // blocks of 64 values of range sp: whole chunks
    auto first_kb = [&](int sp) { return min(all_kb, GF_CHUNK * (int)((int64_t)chunks * sp / a.splits)); };
    int fail = 0;

    if (warp == 0) {
        if (lane == 0) {
            int stage = 0;
            uint32_t phase = 0;
            for (int t = worker; t < total && fail == 0; t += nworkers) {
                const int sp = t / per_split, tt = t - sp * per_split, nt = tt / tiles_m, mt = tt - nt * tiles_m;
                const int kb0 = first_kb(sp), kb1 = first_kb(sp + 1);
                const int row0 = mt * TM_ROWS + (int)rank * BM, brow = nt * BN + (PAIR ? (int)rank * (BN / 2) : 0);
                for (int kb = kb0; kb < kb1; ++kb) {
                    if (int w = mbar_wait(bar_empty + 8 * stage, phase ^ 1, abort_flag, a.wait_ns)) { fail = w == 1 ? 1 : -1; break; }
                    const uint32_t sa = sbase + stage * L::STAGE_BYTES, sb = sa + 3 * L::A_BYTES;
                    if (!PAIR) mbar_expect_tx(bar_full + 8 * stage, L::STAGE_BYTES);
                    else if (leader) mbar_expect_tx(bar_full + 8 * stage, 2 * L::STAGE_BYTES);
#pragma unroll
                    for (int p = 0; p < 3; ++p) {
                        const int x = p * a.part_bytes + kb * BK;
                        if (PAIR) {
                            tma_load_2d_pair(sa + p * L::A_BYTES, &tmA, x, row0, full_leader + 8 * stage);
                            tma_load_2d_pair(sb + p * L::B_BYTES, &tmB, x, brow, full_leader + 8 * stage);
                        } else {
                            tma_load_2d(sa + p * L::A_BYTES, &tmA, x, row0, bar_full + 8 * stage);
                            tma_load_2d(sb + p * L::B_BYTES, &tmB, x, brow, bar_full + 8 * stage);
                        }
                    }
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                }
            }
        }
    } else if (warp == 1) {
        if (leader) {          // the whole warp; `on` is the lane that issues
            const uint32_t on = elect_lane();
            bool ok = true;
            constexpr uint32_t idesc = umma_idesc_bf16(TM_ROWS, BN);
            int stage = 0;
            uint32_t phase = 0, acc = 0, acc_phase = 0;
            for (int t = worker; t < total && ok; t += nworkers) {
                const int sp = t / per_split, kb0 = first_kb(sp), kb1 = first_kb(sp + 1);
                uint32_t d_tmem = 0;
                for (int kb = kb0; kb < kb1; ++kb) {
                    const bool fresh = (kb - kb0) % GF_CHUNK == 0;
                    if (fresh) {
                        if (!(ok = wait_warp<PAIR>(bar_tempty + 8 * acc, acc_phase ^ 1, abort_flag, a.wait_ns, 2, fail))) break;
                        tc_fence_after();
                        d_tmem = tmem_base + acc * 2 * BN;
                    }
                    if (!(ok = wait_warp(bar_full + 8 * stage, phase, abort_flag, a.wait_ns, 3, fail))) break;
                    tc_fence_after();
                    const uint32_t sa = sbase + stage * L::STAGE_BYTES, sb = sa + 3 * L::A_BYTES;
#pragma unroll
                    for (int i = 0; i < 6; ++i) {
                        constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};
                        const uint64_t da = umma_desc(sa + PA[i] * L::A_BYTES), db = umma_desc(sb + PB[i] * L::B_BYTES);
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; ++k) {
                            const uint64_t o = (uint64_t)(k * (UMMA_K >> 4));
                            const uint32_t add = fresh && k == 0 && (i == 0 || i == 5) ? 0u : 1u, d = d_tmem + (i == 5 ? 0 : BN);
                            if (PAIR) umma_bf16_pair(on, d, da + o, db + o, idesc, add);
                            else umma_bf16(on, d, da + o, db + o, idesc, add);
                        }
                    }
                    if (PAIR) umma_commit_pair(on, bar_empty + 8 * stage);
                    else umma_commit(on, bar_empty + 8 * stage);
                    if (++stage == STAGES) { stage = 0; phase ^= 1; }
                    if (kb + 1 == kb1 || (kb + 1 - kb0) % GF_CHUNK == 0) {
                        if (PAIR) umma_commit_pair(on, bar_tfull + 8 * acc);
                        else umma_commit(on, bar_tfull + 8 * acc);
                        if (++acc == L::ACCS) { acc = 0; acc_phase ^= 1; }
                    }
                }
            }
        }
    } else {
        constexpr int COLS = BN / 2;              // of this warp
        const int q = warp & 3, chalf = (warp - 2) >> 2;
        uint8_t* stg = smem + L::EPI_OFF + (warp - 2) * GF_STAGE_WARP;
        uint32_t acc = 0, acc_phase = 0;
        for (int t = worker; t < total && fail == 0; t += nworkers) {
            const int sp = t / per_split, tt = t - sp * per_split, nt = tt / tiles_m, mt = tt - nt * tiles_m;
            const int kb0 = first_kb(sp), kb1 = first_kb(sp + 1);
            const int n0 = nt * BN + chalf * COLS, row0 = mt * TM_ROWS + (int)rank * BM + 32 * q;
            const int ea = row0 + lane < a.M ? a.ea[row0 + lane] : GF_NAN;      // rows and columns that do not exist need no repair
            int ew[COLS / 32];
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) ew[c] = n0 + 32 * c + lane < a.N ? a.ew[n0 + 32 * c + lane] : GF_NAN;
            float sum[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) sum[j] = 0.0f;
            for (int kb = kb0; kb < kb1; kb += GF_CHUNK) {
                if (int w = mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag, a.wait_ns)) fail = w == 1 ? 4 : -1;
                epilogue_bar();         // the epilogue threads agree on giving up before anyone touches TMEM
                if (*abort_flag) { if (!fail) fail = -1; break; }
                tc_fence_after();
                const uint32_t taddr = tmem_base + acc * 2 * BN + chalf * COLS + ((uint32_t)(32 * q) << 16);
#pragma unroll
                for (int c = 0; c < COLS / 32; ++c) {
                    uint32_t r[32];
                    tmem_ld32(taddr + BN + 32 * c, r);
                    tmem_ld_fence(r);
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[32 * c + j] += __uint_as_float(r[j]);
                    tmem_ld32(taddr + 32 * c, r);
                    tmem_ld_fence(r);
#pragma unroll
                    for (int j = 0; j < 32; ++j) sum[32 * c + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (!PAIR || leader) mbar_arrive(bar_tempty + 8 * acc);
                    else mbar_arrive_cluster(tempty_leader + 8 * acc);
                }
                if (++acc == L::ACCS) { acc = 0; acc_phase ^= 1; }
            }
            if (fail) break;
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) {
                const uint32_t cols = __ballot_sync(0xffffffffu, ew[c] != GF_NAN);
                bool bad = false;      // not a number although neither row has such a value
#pragma unroll
                for (int j = 0; j < 32; ++j) bad |= (cols >> j & 1) && sum[32 * c + j] != sum[32 * c + j];
                gf_scale(sum + 32 * c, ea == GF_NAN ? 0 : ea, ew[c] == GF_NAN ? 0 : ew[c]);
                if (__any_sync(0xffffffffu, bad && ea != GF_NAN)) {
                    float t[32];
                    gf_dots(a, row0 + lane, n0 + 32 * c, 64 * kb0, min(a.K, 64 * kb1), reinterpret_cast<float4*>(stg), t);
#pragma unroll
                    for (int j = 0; j < 32; ++j)
                        if (sum[32 * c + j] != sum[32 * c + j]) sum[32 * c + j] = t[j];
                }
            }
            __syncwarp();
            float* out = a.out + (int64_t)sp * a.split_stride;
            const int npad = ((a.act == 2 ? a.N / 2 : a.N) + 3) & ~3, piece = lane & 3, rsub = lane >> 2;
            // units of 16 outputs: staged a row per lane, stored as 64-byte row pieces
            auto unit = [&](const float (&v)[16], int col) {
                float4* o = reinterpret_cast<float4*>(stg + lane * GF_PITCH);
#pragma unroll
                for (int j = 0; j < 4; ++j) o[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int rl = 8 * i + rsub, row = row0 + rl;
                    const float4 x = *reinterpret_cast<const float4*>(stg + rl * GF_PITCH + piece * 16);
                    if (row < a.M && col + 4 * piece < npad) *reinterpret_cast<float4*>(out + (int64_t)row * a.ldo + col + 4 * piece) = x;
                }
                __syncwarp();
            };
#pragma unroll
            for (int c = 0; c < COLS / 32; ++c) {
                float v[16];
                if (a.act == 2) {
#pragma unroll
                    for (int j = 0; j < 16; ++j) v[j] = gelu_tanh_f32(sum[32 * c + j]) * sum[32 * c + 16 + j];
                    unit(v, n0 / 2 + 16 * c);
                } else {
#pragma unroll
                    for (int u = 0; u < 2; ++u) {
#pragma unroll
                        for (int j = 0; j < 16; ++j) {
                            const float x = sum[32 * c + 16 * u + j];
                            v[j] = a.act == 1 ? xielu_f32(x, a.a_pos, a.a_neg) : x;
                        }
                        unit(v, n0 + 32 * c + 16 * u);
                    }
                }
            }
        }
    }

    if (fail > 0) {
        if (atomicCAS(a.status, 0, fail) == 0) {
            a.status[1] = blockIdx.x;
            a.status[2] = threadIdx.x;
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*abort_flag) {
        const uint64_t t0 = globaltimer_ns();
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);   // 0.2 ms for outstanding TMA writes
        __syncthreads();
    }
    if (PAIR) cluster_sync_all();
    tc_fence_after();
    if (warp == 1) {
        if (PAIR) tmem_dealloc2(tmem_base, TMEM_COLS);
        else tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

template <int BN>
__global__ void __launch_bounds__(CTA_THREADS, 1) gemm_f32_kernel(const __grid_constant__ CUtensorMap tmA,
                                                            const __grid_constant__ CUtensorMap tmB, const GfArgs a) {
    gemm_f32_body<BN, false>(tmA, tmB, a);
}
template <int BN>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(CTA_THREADS, 1)
    gemm_f32_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, const GfArgs a) {
    gemm_f32_body<BN, true>(tmA, tmB, a);
}

template <int BN, bool PAIR>
static int launch_gf(const void* A3, const void* W3, const GfArgs& a, cudaStream_t st) {
    using L = GfSmem<BN, PAIR>;
    static bool configured[64] = {};
    const int dev = current_device();
    SCMX_REQUIRE(dev >= 0, SCMX_ECUDA, "no current CUDA device (ordinal 0..63)");
    void (*kernel)(CUtensorMap, CUtensorMap, GfArgs);
    if constexpr (PAIR) kernel = gemm_f32_pair_kernel<BN>;
    else kernel = gemm_f32_kernel<BN>;
    if (!configured[dev]) {
        SCMX_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, L::TOTAL));
        configured[dev] = true;
    }
    CUtensorMap tmA, tmB;
    int rc = make_map_u8(&tmA, A3, a.M, 3 * (int64_t)a.part_bytes, BK, BM, 128, 3 * (int64_t)a.part_bytes);
    if (rc) return rc;
    rc = make_map_u8(&tmB, W3, a.N, 3 * (int64_t)a.part_bytes, BK, PAIR ? BN / 2 : BN, 128, 3 * (int64_t)a.part_bytes);
    if (rc) return rc;
    constexpr int rows = PAIR ? 2 * BM : BM;
    const int64_t tiles = ((a.M + rows - 1) / rows) * (int64_t)((a.N + BN - 1) / BN) * a.splits;
    int workers = PAIR ? sm_count() / 2 : sm_count();
    if (tiles < workers) workers = (int)tiles;
    SCMX_PDL_OK("gemm_f32", launch_pdl(kernel, dim3(PAIR ? 2 * workers : workers), dim3(CTA_THREADS), (size_t)L::TOTAL, st, tmA, tmB, a));
    return SCMX_OK;
}

}  // namespace scmx

using namespace scmx;

extern "C" int scmx_gemm_f32(const float* A, int64_t lda, const float* W, int64_t ldw, int64_t M, int64_t N, int64_t K, int act, float a_pos,
                             float a_neg, float* out, int64_t ldo, int tile, int splits, int64_t band, float* part, void* scratch, int32_t* status,
                             void* stream) {
    SCMX_REQUIRE(A && W && out && scratch && status, SCMX_EINVAL, "gemm_f32: null buffer");
    SCMX_REQUIRE(M >= 0 && N > 0 && K > 0 && M < (1ll << 30) && N < (1ll << 30) && K < (1ll << 28), SCMX_EINVAL, "gemm_f32: M=%lld N=%lld K=%lld",
                 (long long)M, (long long)N, (long long)K);
    SCMX_REQUIRE(lda >= K && ldw >= K, SCMX_EINVAL, "gemm_f32: the row pitches %lld, %lld must hold K=%lld", (long long)lda, (long long)ldw, (long long)K);
    SCMX_REQUIRE(act >= 0 && act <= 2 && (act != 2 || N % 32 == 0), SCMX_EINVAL, "gemm_f32: act=%d on %lld columns", act, (long long)N);
    const int64_t nout = act == 2 ? N / 2 : N;
    SCMX_REQUIRE(ldo % 4 == 0 && ldo >= (nout + 3) / 4 * 4, SCMX_EINVAL, "gemm_f32: output pitch %lld for %lld columns", (long long)ldo, (long long)N);
    SCMX_REQUIRE(((uintptr_t)scratch & 15) == 0 && ((uintptr_t)out & 15) == 0, SCMX_EINVAL, "gemm_f32: pointer not 16-byte aligned");
    SCMX_REQUIRE(tile == 64 || tile == 128 || tile == 256, SCMX_EINVAL, "gemm_f32: tile=%d", tile);
    SCMX_REQUIRE(band >= N || (band > 0 && band % 256 == 0), SCMX_EINVAL, "gemm_f32: bands of %lld rows", (long long)band);
    if (M == 0) return SCMX_OK;
    GfArgs a;
    a.M = (int)M; a.K = (int)K; a.part_bytes = (int)((K + 63) / 64 * 128); a.act = act; a.a_pos = a_pos; a.a_neg = a_neg;
    a.A = A; a.lda = lda; a.ldw = ldw; a.splits = splits > 1 ? splits : 1; a.status = status; a.wait_ns = g_wait_limit_ns;
    if (splits > 1)
        SCMX_REQUIRE(part && ((uintptr_t)part & 15) == 0 && act == 0 && splits <= (a.part_bytes / BK + GF_CHUNK - 1) / GF_CHUNK, SCMX_EINVAL,
                     "gemm_f32: %d ranges of K=%lld need a buffer and no activation", splits, (long long)K);
    const cudaStream_t st = (cudaStream_t)stream;
    const int kp = a.part_bytes / 2;
    bf16_t *a3 = (bf16_t*)scratch, *w3 = a3 + M * 3 * kp;
    int32_t* e = (int32_t*)(w3 + (N < band ? N : band) * 3 * kp);
    a.ea = e; a.ew = e + M;
    a.vec = lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    for (int64_t n0 = 0; n0 < N; n0 += band) {
        const int64_t n = N - n0 < band ? N - n0 : band, ldp = (n + 3) / 4 * 4;
        float* o = out + (act == 2 ? n0 / 2 : n0);
        a.N = (int)n; a.W = W + n0 * ldw;
        a.out = splits > 1 ? part : o; a.ldo = splits > 1 ? ldp : ldo; a.split_stride = splits > 1 ? M * ldp : 0;
        int rc = run_split3(SplitRows{A, lda, n0 == 0 ? M : 0, a3, e, 0}, SplitRows{a.W, ldw, n, w3, e + M, 0}, (int)K, kp, st);
        if (rc) return rc;
        rc = tile == 256 ? launch_gf<256, true>(a3, w3, a, st) : tile == 128 ? launch_gf<128, false>(a3, w3, a, st) : launch_gf<64, false>(a3, w3, a, st);
        if (rc) return rc;
        if (splits > 1 && (rc = gemm_reduce(part, splits, a.split_stride, M, ldp, 1, o, ldo, st))) return rc;
    }
    return SCMX_OK;
}
