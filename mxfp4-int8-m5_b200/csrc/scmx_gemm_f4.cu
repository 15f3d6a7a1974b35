// W4A8 GEMM on the tensor cores' 4-bit path: the packed codes are the operand as they lie in memory.  A code is an e2m1 number (sign << 3 |
// index, twice its value the integer magnitude) and a block code c multiplies 32 of them by 2^c, so a weight row is a matrix of
// tcgen05.mma kind::mxf4 with block factors 2^c; nothing is expanded, in memory or in shared memory.  An INT8 activation is three digits to base
// eight, x = d0 + 8 d1 + 64 d2 with |d| <= 4, every digit an e2m1 number too: three digit planes [3][rows][K / 2] of 4-bit codes (digits8).
// All products and sums are integers, |sum| <= 4 * 96 * K < 2^22 for K <= 10240, so the float32 accumulators hold them exactly, and
// total = s0 + 8 s1 + 64 s2 is the INT32 total of the INT8 product bit for bit.
//
// Three digits cost 1.5 times the tensor work of the INT8 product (4-bit products run at twice its rate) but weights cost half a byte a value on
// their whole way and no integer instructions.  It takes the place of the expanding kernel (scmx_gemm_w4.cu), whose permutes bound it, and of
// decode-then-GEMM for prompts of few rows.
//
// A pair of CTAs owns 256 weight rows (the M of the instruction, 128 per CTA) x up to 80 tokens: N = 3 planes x tokens, the first half of the
// tokens (all three planes) from one CTA, the second half from the other.  Tokens per tile follow the segment (a multiple of 16): an expert of 128
// rows takes two tiles of 64.  A stage is 256 values of K: 16 KB of codes, 3 x 40 x 128 bytes of digits and 1 KB of block factors per CTA, four
// MMAs.  Accumulators 2 x 240 columns of tensor memory, 8 columns of token factors (all 2, written once), 3 x 8 columns of weight factors.
// Factors are bytes 2^(1 + c) in the order that scale_vec::2X reads them from tensor memory (per 128 rows x 128 values 512 bytes: lane = row % 32, column =
// row / 32, one byte per block), written by factors_kernel before; the MMA thread copies them from a stage's shared memory with tcgen05.cp in
// front of the MMAs that read them.  (Warps that wrote them to tensor memory from the block codes, a step behind two barriers between the CTAs, held every
// stage up: 1300 - 1800 cycles against 480 of MMAs.)
// Grouped gate|up product of 64 experts with 128 rows each (2048 x 2048): 90 us by the expanding kernel, 61 us here; 16 rows each 88 and 31 us (134 MB of codes: 4.4
// TB/s).  A tile of 8 stages takes 6500 cycles against 3100 of products: the issuing warp (447 cycles a stage alone, 650 beside the epilogue warps) bounds it.
// Roles per CTA (576 threads): warp 0 TMA, warp 1 MMA (leader), warps 2..17 epilogue.  All waits are bounded.
#include "scmx_gemm_core.cuh"

namespace scmx {

constexpr int F4_STAGES = 6;
constexpr int F4_SLOTS = 3;                        // weight factors of that many stages in tensor memory
constexpr int F4_KV = 256;                         // values of K per stage
constexpr int F4_TNH = 40;                         // tokens per CTA of a pair at most
constexpr int F4_EPI_WARPS = 16;
constexpr int F4_THREADS = 64 + 32 * F4_EPI_WARPS;
constexpr int F4_MAX_E = 512;
constexpr int F4_A_BYTES = 128 * 128, F4_B_BYTES = 3 * F4_TNH * 128, F4_SF_BYTES = 1024;
constexpr int F4_SF_OFF = F4_A_BYTES + F4_B_BYTES, F4_STAGE_BYTES = F4_SF_OFF + F4_SF_BYTES;
constexpr int F4_ACC = 6 * F4_TNH;                 // columns of an accumulator set
constexpr int F4_SFB = 2 * F4_ACC, F4_SFA = F4_SFB + 8;
static_assert(F4_SFA + 8 * F4_SLOTS <= 512 && F4_STAGE_BYTES % 1024 == 0, "tensor memory / swizzle alignment");

struct F4Smem {
    static constexpr int BAR_OFF = F4_STAGES * F4_STAGE_BYTES;       // full[S], empty[S], tfull[2], tempty[2]
    static constexpr int MISC_OFF = BAR_OFF + 8 * (2 * F4_STAGES + 4);
    static constexpr int EPI_OFF = MISC_OFF + 16;                    // per epilogue warp 8 tokens x 64 bytes
    static constexpr int PT_OFF = EPI_OFF + F4_EPI_WARPS * 512;       // first tile of every expert
    static constexpr int OFF_OFF = PT_OFF + 4 * (F4_MAX_E + 4);      // expert offsets
    static constexpr int TN_OFF = OFF_OFF + 4 * (F4_MAX_E + 4);      // tokens per CTA of an expert's tiles
    static constexpr int XS_OFF = TN_OFF + 4 * (F4_MAX_E + 4);       // per epilogue warp the scales of 24 tokens
    static constexpr int TOTAL = XS_OFF + F4_EPI_WARPS * 24 * 4 + 1024;
};
static_assert(F4Smem::EPI_OFF % 16 == 0 && F4Smem::TOTAL <= 232448, "shared memory");

struct F4Maps {
    CUtensorMap w;                   // codes, 128 bytes x 128 rows
    CUtensorMap f;                   // factors, 8 x 128 bytes of one tile of 128 rows
    CUtensorMap x[F4_TNH / 8];       // digit planes, 128 bytes x 8 (i + 1) rows x 3 planes
};

struct F4Args {
    GemmArgs g;                      // M / R, N, K, epilogue, scales, output, expert segments (off), status
    int ftiles;                      // tiles of 128 rows per matrix: ceil(N / 128)
    int tiles_m, tnh;                // dense: token tiles, tokens per CTA
};

struct F4Tile {
    int row0, rows;      // first token of the tile, tokens of its segment from there on (may exceed the tile)
    int tnh;             // tokens per CTA of the pair, a multiple of 8
    int n0, wbase;       // first weight row inside the matrix / expert, and in the stack of all experts
    int f0;              // first tile of factors
};

// Tokens per CTA for a segment of `rows` tokens cut into equal tiles.
__host__ __device__ __forceinline__ int f4_tnh(int rows, int tiles) {
    const int per = (rows + tiles - 1) / tiles;
    return max(8, (per + 15) / 16 * 8);
}

// Whether a phase of a barrier has completed, without waiting.
__device__ __forceinline__ bool mbar_test_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// TMA loads of a CTA pair issued by the lane with `on` of a warp that stays together (a thread alone takes ~100 cycles to issue one); the bytes count on a
// barrier that may live in the other CTA.
__device__ __forceinline__ void load_2d_pair(uint32_t on, uint32_t dst, const CUtensorMap* map, int c0, int c1, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];\n\t}"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(on)
        : "memory");
}
__device__ __forceinline__ void load_3d_pair(uint32_t on, uint32_t dst, const CUtensorMap* map, int c0, int c1, int c2, uint32_t bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %6, 0;\n\t"
        "@q cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n\t}"
        ::"r"(dst), "l"(map), "r"(bar), "r"(c0), "r"(c1), "r"(c2), "r"(on)
        : "memory");
}
__device__ __forceinline__ void expect_bytes(uint32_t on, uint32_t bar, uint32_t bytes) {
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t@q mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n\t}" ::"r"(bar), "r"(bytes), "r"(on)
                 : "memory");
}
// The four products of a stage (64 values of K each: 32 bytes further in both operands), the first of a tile without what the accumulators held.  One block, so that
// the issuing warp spends few instructions on it beside 16 epilogue warps.
__device__ __forceinline__ void umma_mxf4_stage(uint32_t on, uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t id0, uint32_t id2, uint32_t sfa, uint32_t sfb,
                                                uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q, t;\n\t"
        "setp.ne.b32 p, %12, 0;\n\t"
        "setp.ne.b32 q, %13, 0;\n\t"
        "setp.eq.b32 t, 0, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %5, %9, [%11], [%15], p;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %2, %6, %10, [%11], [%15], t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %3, %7, %9, [%14], [%15], t;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::mxf4.block_scale.scale_vec::2X [%0], %4, %8, %10, [%14], [%15], t;\n\t}"
        ::"r"(d_tmem), "l"(a), "l"(a + 2), "l"(a + 4), "l"(a + 6), "l"(b), "l"(b + 2), "l"(b + 4), "l"(b + 6), "r"(id0), "r"(id2), "r"(sfa), "r"(accumulate), "r"(on),
        "r"(sfa + 4), "r"(sfb)
        : "memory");
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};" ::"r"(taddr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// The factors of a stage: twice 512 bytes of shared memory in both CTAs -> 32 lanes x 4 columns of tensor memory, the same in all four lane quarters.  In order with the MMAs of this
// thread.  The descriptor: 8 rows x 16 bytes are contiguous, groups of 8 rows 128 bytes apart, no swizzle.
__device__ __forceinline__ void tmem_cp_pair(uint32_t on, uint32_t taddr, uint32_t smem_addr) {
    const uint64_t desc = (uint64_t)((smem_addr >> 4) & 0x3FFFu) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %2, 0;\n\t"
        "@q tcgen05.cp.cta_group::2.32x128b.warpx4 [%0], %1;\n\t"
        "@q tcgen05.cp.cta_group::2.32x128b.warpx4 [%4], %3;\n\t}"
        ::"r"(taddr), "l"(desc), "r"(on), "l"(desc + (512 >> 4)), "r"(taddr + 4) : "memory");
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

// Instruction descriptor of kind::mxf4: A and B e2m1 (1 at [7,10) and [10,12)), both K-major, N >> 3 at [17,23), factors of type ue8m0 (bit 23),
// M >> 7 at [27,29), factor bytes of A inside its column at [29,31): 0 or 2 (of B at [4,6): 0).
__host__ __device__ constexpr uint32_t f4_idesc(int n, int sf) {
    return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | (2u << 27) | ((uint32_t)sf << 29);
}

// The factors 2^(1 + c) of four blocks from their codes of two bits: biased exponents 128 + c, a byte each.
__device__ __forceinline__ uint32_t f4_factors(uint32_t b) {
    return ((b & 3u) | ((b & 0xCu) << 6) | ((b & 0x30u) << 12) | ((b & 0xC0u) << 18)) + 0x80808080u;
}

// SiLU(g) u of two values, the steps and roundings of swiglu_bf16 taken in pairs (a conversion instruction rounds two).  The reciprocal of a
// bfloat16 number is at least 7e-6 (relative) away from the middle of two bfloat16 numbers or exact, so the approximate one (2^-23) rounds alike.
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ uint32_t swiglu2(float g0, float g1, float u0, float u1) {
    const uint32_t e = pack_bf16x2(expf(fabsf(g0)), expf(fabsf(g1)));
    const uint32_t x = pack_bf16x2(__fadd_rn(1.0f, bf16_lo(e)), __fadd_rn(1.0f, bf16_hi(e)));
    const uint32_t y = pack_bf16x2(rcp_approx(bf16_lo(x)), rcp_approx(bf16_hi(x)));
    const uint32_t z = pack_bf16x2(__fsub_rn(1.0f, bf16_lo(y)), __fsub_rn(1.0f, bf16_hi(y)));
    const uint32_t s = pack_bf16x2(__fmul_rn(g0, g0 < 0.0f ? bf16_lo(y) : bf16_lo(z)), __fmul_rn(g1, g1 < 0.0f ? bf16_hi(y) : bf16_hi(z)));
    return pack_bf16x2(__fmul_rn(bf16_lo(s), u0), __fmul_rn(bf16_hi(s), u1));
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(F4_THREADS, 1)
    gemm_f4_kernel(const __grid_constant__ F4Maps maps, const F4Args fa) {
    using L = F4Smem;
    const GemmArgs& a = fa.g;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar_full = sbase + L::BAR_OFF, bar_empty = bar_full + 8 * F4_STAGES;
    const uint32_t bar_tfull = bar_empty + 8 * F4_STAGES, bar_tempty = bar_tfull + 16;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L::MISC_OFF);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L::MISC_OFF + 4);
    int* ptile = reinterpret_cast<int*>(smem + L::PT_OFF);
    int* soff = reinterpret_cast<int*>(smem + L::OFF_OFF);
    int* stnh = reinterpret_cast<int*>(smem + L::TN_OFF);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();
    const bool leader = rank == 0;

    if (threadIdx.x == 0) {
        for (int s = 0; s < F4_STAGES; ++s) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(bar_tfull + 8 * i, 1);
            mbar_init(bar_tempty + 8 * i, 2 * F4_EPI_WARPS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        tmem_alloc2(smem_u32(tmem_slot), 512);
        tmem_relinquish2();
    }
    pdl_launch_dependents();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    if (warp >= 14) {       // factor 2 of every token, for all lanes
        const uint32_t two = 0x80808080u, at = tmem_base + F4_SFB + ((uint32_t)(32 * (warp & 3)) << 16);
        tmem_st4(at, two, two, two, two);
        tmem_st4(at + 4, two, two, two, two);
        tmem_st_wait();
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    tc_fence_after();
    pdl_wait();

    // ---- tiles: a segment (the whole problem, or an expert's rows) is cut into ceil(rows / 80) equal tiles
    constexpr int TN = 2 * F4_TNH;
    const int tiles_n = (a.N + 255) / 256;
    int tiles_m = fa.tiles_m;
    if (a.E > 0) {
        for (int i = threadIdx.x; i <= a.E; i += F4_THREADS) soff[i] = a.off[i];
        __syncthreads();
        if (warp == 2) {
            int run = 0;
            for (int b0 = 0; b0 < a.E; b0 += 32) {
                const int e = b0 + lane, rows = e < a.E ? soff[e + 1] - soff[e] : 0;
                const int c = (rows + TN - 1) / TN;
                int sc = c;
#pragma unroll
                for (int d = 1; d < 32; d <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, sc, d);
                    if (lane >= d) sc += v;
                }
                if (e < a.E) {
                    ptile[e] = run + sc - c;
                    stnh[e] = c > 0 ? f4_tnh(rows, c) : 8;
                }
                run += __shfl_sync(0xffffffffu, sc, 31);
            }
            if (lane == 0) ptile[a.E] = run;
        }
        __syncthreads();
        tiles_m = ptile[a.E];
    }
    const int num_kb = (a.K + F4_KV - 1) / F4_KV;
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    // Column tiles run fastest, so that CTAs that run together share tokens and the next token tiles find the weights in L2.  A role walks through the tiles of
    // its pair in steps: no division, no search from the start (both cost the MMA warp 1200 cycles a tile).
    struct Walk {
        int mt, nt, e;
    };
    const int step_m = npairs / tiles_n, step_n = npairs - step_m * tiles_n;
    auto settle = [&](Walk& w) {
        if (a.E > 0 && w.mt < tiles_m)                 // whole warps: 32 experts are looked at together
            for (int n = 32; n == 32; w.e += n) {
                const int e = w.e + 1 + lane;
                n = __popc(__ballot_sync(0xffffffffu, e <= a.E && ptile[e] <= w.mt));
            }
    };
    auto begin = [&]() {
        Walk w;
        w.mt = pair / tiles_n; w.nt = pair - w.mt * tiles_n; w.e = 0;
        settle(w);
        return w;
    };
    auto advance = [&](Walk& w) {
        w.mt += step_m;
        w.nt += step_n;
        if (w.nt >= tiles_n) {
            w.nt -= tiles_n;
            ++w.mt;
        }
        settle(w);
    };
    auto get_tile = [&](const Walk& w) {
        F4Tile tl;
        tl.n0 = w.nt * 256;
        int first = 0, rows = a.M, i = w.mt;
        tl.tnh = fa.tnh;
        if (a.E > 0) {
            first = soff[w.e];
            rows = soff[w.e + 1] - first;
            i = w.mt - ptile[w.e];
            tl.tnh = stnh[w.e];
        }
        tl.wbase = w.e * a.N + tl.n0;
        tl.f0 = w.e * fa.ftiles + (tl.n0 >> 7);
        tl.row0 = first + i * 2 * tl.tnh;
        tl.rows = rows - i * 2 * tl.tnh;          // may be <= 0: rounding can leave the last tile empty
        return tl;
    };
    const uint32_t full_leader = mapa_u32(bar_full, 0), tempty_leader = mapa_u32(bar_tempty, 0);
    int fail = 0;

    if (warp == 0) {
        // ------------------------------------------------ TMA producer: this CTA's weight rows and tokens
        const uint32_t on = elect_lane();
        bool ok = true;
        int stage = 0;
        uint32_t phase = 0;
        for (Walk wk = begin(); wk.mt < tiles_m && ok; advance(wk)) {
            const F4Tile tl = get_tile(wk);
            const CUtensorMap* mx = &maps.x[tl.tnh / 8 - 1];
            const int wrow = tl.wbase + (int)rank * 128, xrow = tl.row0 + (int)rank * tl.tnh;
            const uint32_t bytes = 2 * (F4_A_BYTES + 3 * 128 * tl.tnh + F4_SF_BYTES);
            for (int kb = 0; kb < num_kb; ++kb) {
                if (!(ok = wait_warp(bar_empty + 8 * stage, phase ^ 1, abort_flag, a.wait_ns, 1, fail))) break;
                const uint32_t sa = sbase + stage * F4_STAGE_BYTES, bar = full_leader + 8 * stage;
                if (leader) expect_bytes(on, bar_full + 8 * stage, bytes);
                load_2d_pair(on, sa, &maps.w, kb * 128, wrow, bar);
                load_3d_pair(on, sa + F4_A_BYTES, mx, kb * 128, xrow, 0, bar);
                load_3d_pair(on, sa + F4_SF_OFF, &maps.f, 0, 8 * kb, tl.f0 + (int)rank, bar);
                if (++stage == F4_STAGES) { stage = 0; phase ^= 1; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------ MMA issuer (leader CTA)
        if (leader) {          // the whole warp; `on` is the lane that issues
            const uint32_t on = elect_lane();
            bool ok = true;
            int stage = 0, slot = 0;
            uint32_t phase = 0, acc = 0, acc_phase = 0;
            bool copied = false;          // the factors of the current stage are in tensor memory
            auto copy_factors = [&](int st, int sl) {
                tmem_cp_pair(on, tmem_base + F4_SFA + 8 * sl, sbase + st * F4_STAGE_BYTES + F4_SF_OFF);
            };
            for (Walk wk = begin(); wk.mt < tiles_m && ok; advance(wk)) {
                const int n = 6 * (a.E > 0 ? stnh[wk.e] : fa.tnh);
                const uint32_t id0 = f4_idesc(n, 0), id2 = f4_idesc(n, 2);
                if (!(ok = wait_warp<true>(bar_tempty + 8 * acc, acc_phase ^ 1, abort_flag, a.wait_ns, 2, fail))) break;
                tc_fence_after();
                const uint32_t d_tmem = tmem_base + acc * F4_ACC;
                for (int kb = 0; kb < num_kb; ++kb) {
                    if (!copied) {
                        if (!(ok = wait_warp(bar_full + 8 * stage, phase, abort_flag, a.wait_ns, 3, fail))) break;
                        tc_fence_after();
                        copy_factors(stage, slot);
                    }
                    // the next stage's factors go in front of this stage's MMAs where they have arrived: the copy then runs under MMAs
                    const int stage1 = stage + 1 == F4_STAGES ? 0 : stage + 1, slot1 = slot + 1 == F4_SLOTS ? 0 : slot + 1;
                    const uint32_t phase1 = stage1 == 0 ? phase ^ 1 : phase;
                    copied = __all_sync(0xffffffffu, mbar_test_wait(bar_full + 8 * stage1, phase1));
                    if (copied) {
                        tc_fence_after();
                        copy_factors(stage1, slot1);
                    }
                    const uint32_t sa = sbase + stage * F4_STAGE_BYTES, sf = tmem_base + F4_SFA + 8 * slot;
                    const uint64_t da = umma_desc(sa), db = umma_desc(sa + F4_A_BYTES);
                    umma_mxf4_stage(on, d_tmem, da, db, id0, id2, sf, tmem_base + F4_SFB, kb != 0 ? 1u : 0u);
                    umma_commit_pair(on, bar_empty + 8 * stage);
                    stage = stage1; phase = phase1; slot = slot1;
                }
                if (!ok) break;
                umma_commit_pair(on, bar_tfull + 8 * acc);
                acc ^= 1;
                if (acc == 0) acc_phase ^= 1;
            }
        }
    } else {
        // ------------------------------------------------ epilogue: four warps share 32 weight rows (lanes) of the tile's tokens: two halves (the tokens of a
        // CTA), of which a warp takes every other group of 8
        const int q = warp & 3, half = ((warp - 2) >> 2) & 1, sub = (warp - 2) >> 3;
        uint8_t* stg = smem + L::EPI_OFF + (warp - 2) * 512;
        uint32_t acc = 0, acc_phase = 0;
        // what a tile's conversion needs is requested a tile ahead: the row's weight scale, and in lane 8 k + j the scale of token j of the warp's group k
        auto scales = [&](const F4Tile& t, float& w, float& x) {
            const int n = t.n0 + (int)rank * 128 + 32 * q, tk = 8 * (2 * (lane >> 3) + sub) + (lane & 7);
            w = x = 0.0f;
            if (a.epi == 0 || n >= a.N) return;
            w = a.wscale[t.wbase + (int)rank * 128 + 32 * q + lane];
            if (tk < min(t.tnh, t.rows - half * t.tnh)) x = a.xscale[t.row0 + half * t.tnh + tk];
        };
        float* xw = reinterpret_cast<float*>(smem + L::XS_OFF) + 24 * (warp - 2);
        const bool wide = a.K > 4854;             // 36 * 96 * K may reach 2^24
        Walk wk = begin();
        F4Tile next = {};
        float ws_next = 0.0f, xs_next = 0.0f;
        if (wk.mt < tiles_m) {
            next = get_tile(wk);
            scales(next, ws_next, xs_next);
        }
        while (wk.mt < tiles_m && fail == 0) {
            const F4Tile tl = next;
            const float ws = ws_next, xs_mine = xs_next;
            advance(wk);
            if (wk.mt < tiles_m) {
                next = get_tile(wk);
                scales(next, ws_next, xs_next);
            }
            const int n = tl.n0 + (int)rank * 128 + 32 * q;              // first output column of the warp (N is a multiple of 32)
            const bool on = n < a.N;
            const int t0 = tl.row0 + half * tl.tnh, nt = on ? max(0, min(tl.tnh, tl.rows - half * tl.tnh)) : 0;
            if (lane < 24) xw[lane] = xs_mine;
            __syncwarp();
            uint4 rp[3];
            if (a.epi == 2) {
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    const int j = 8 * (2 * k + sub) + (lane >> 2);
                    rp[k] = j < nt ? *reinterpret_cast<const uint4*>(a.res + (size_t)(t0 + j) * a.N + n + 8 * (lane & 3)) : make_uint4(0, 0, 0, 0);
                }
            }
            if (int w = mbar_wait(bar_tfull + 8 * acc, acc_phase, abort_flag, a.wait_ns)) fail = w == 1 ? 4 : -1;
            asm volatile("bar.sync 1, %0;" ::"n"(32 * F4_EPI_WARPS) : "memory");       // agree on giving up
            if (*abort_flag) { if (!fail) fail = -1; break; }
            tc_fence_after();
            const uint32_t col = tmem_base + acc * F4_ACC + half * 3 * tl.tnh + ((uint32_t)(32 * q) << 16);
            uint32_t r0[8], r1[8], r2[8];
            auto fetch = [&](int c) {
                tmem_ld8(col + c, r0);
                tmem_ld8(col + tl.tnh + c, r1);
                tmem_ld8(col + 2 * tl.tnh + c, r2);
            };
            // the accumulators are read: given back before the values are converted and stored (an arrive on the other CTA's barrier waits for what the thread stored)
            auto give_back = [&]() {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    if (leader) mbar_arrive(bar_tempty + 8 * acc);
                    else mbar_arrive_cluster(tempty_leader + 8 * acc);
                }
            };
            if (8 * sub < nt) fetch(8 * sub);
            else give_back();
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const int c = 8 * (2 * k + sub);
                if (c >= nt) break;
                tmem_ld_wait();
                if (c + 16 >= nt) give_back();
                // total = s0 + 8 s1 + 64 s2, rounded once where s0 + 8 s1 is below 2^24 and so exact (always for K <= 4854); else through integers, which float32
                // adds of 1.5 * 2^23 leave in the low bits of values below 2^22
                float f[8];
                uint32_t tot[8];
#pragma unroll
                for (int j = 0; j < 8; ++j) f[j] = fmaf(8.0f, __uint_as_float(r1[j]), __uint_as_float(r0[j]));
                bool ints = a.epi == 0;
                if (wide) {
                    float big = 0.0f;
#pragma unroll
                    for (int j = 0; j < 8; ++j) big = fmaxf(big, fabsf(f[j]));
                    ints |= big >= 16777216.0f;
                }
                if (ints) {
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        constexpr float MAGIC = 12582912.0f;
                        const uint32_t b0 = __float_as_uint(__fadd_rn(__uint_as_float(r0[j]), MAGIC)), b1 = __float_as_uint(__fadd_rn(__uint_as_float(r1[j]), MAGIC)),
                                       b2 = __float_as_uint(__fadd_rn(__uint_as_float(r2[j]), MAGIC));
                        tot[j] = b0 + 8u * b1 + 64u * b2 - 73u * 0x4B400000u;
                        f[j] = (float)(int)tot[j];
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) f[j] = fmaf(64.0f, __uint_as_float(r2[j]), f[j]);
                }
                __syncwarp();
                if (c + 16 < nt) fetch(c + 16);
                if (a.epi == 0) {
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        if (c + j < nt) reinterpret_cast<int32_t*>(a.out)[(size_t)(t0 + c + j) * a.N + n + lane] = (int32_t)tot[j];
                    continue;
                }
                uint32_t y[4];            // two tokens each
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float2 x = *reinterpret_cast<const float2*>(xw + 8 * k + 2 * j);
                    y[j] = pack_bf16x2(__fmul_rn(__fmul_rn(f[2 * j], x.x), ws), __fmul_rn(__fmul_rn(f[2 * j + 1], x.y), ws));
                }
                if (a.epi == 3) {
                    // rows alternate two gate and two up rows: where lane % 4 < 2 a lane holds gates and lane + 2 their up rows.  Of two tokens the gate lane
                    // finishes the first and the up lane the second.
                    const bool up = lane & 2;
#pragma unroll
                    for (int j = 0; j < 4; j += 2) {
                        float g[2], u[2];
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const uint32_t v = y[j + i], other = __shfl_xor_sync(0xffffffffu, up ? v : v >> 16, 2);      // low half counts
                            g[i] = up ? bf16_lo(other) : bf16_lo(v);
                            u[i] = up ? bf16_hi(v) : bf16_lo(other);
                        }
                        const uint32_t o = swiglu2(g[0], g[1], u[0], u[1]);
                        uint16_t* at = reinterpret_cast<uint16_t*>(stg + (2 * j + (up ? 1 : 0)) * 32) + (lane >> 2) * 2 + (lane & 1);
                        at[0] = (uint16_t)o;
                        at[32] = (uint16_t)(o >> 16);           // two tokens on
                    }
                } else {
#pragma unroll
                    for (int j = 0; j < 4; ++j) reinterpret_cast<uint32_t*>(stg)[32 * j + lane] = y[j];      // rows of words of two tokens
                }
                __syncwarp();
                if (a.epi == 3) {
                    const int j = c + (lane >> 1);
                    if (lane < 16 && j < nt)
                        *reinterpret_cast<uint4*>(static_cast<uint16_t*>(a.out) + (size_t)(t0 + j) * (a.N / 2) + n / 2 + 8 * (lane & 1)) =
                            *reinterpret_cast<const uint4*>(stg + 16 * lane);
                } else {
                    const int j = c + (lane >> 2);
                    // token lane / 4, weight rows 8 (lane % 4) ..: its halves of eight words
                    const uint4* w8 = reinterpret_cast<const uint4*>(stg) + 8 * (lane >> 3) + 2 * (lane & 3);
                    const uint4 wl = w8[0], wh = w8[1];
                    const uint32_t sel = (lane & 4) ? 0x7632u : 0x5410u;
                    uint4 v = make_uint4(__byte_perm(wl.x, wl.y, sel), __byte_perm(wl.z, wl.w, sel), __byte_perm(wh.x, wh.y, sel), __byte_perm(wh.z, wh.w, sel));
                    if (a.epi == 2) {
                        uint32_t o[4] = {v.x, v.y, v.z, v.w};
                        const uint32_t r[4] = {rp[k].x, rp[k].y, rp[k].z, rp[k].w};
#pragma unroll
                        for (int i = 0; i < 4; ++i) o[i] = pack_bf16x2(__fadd_rn(bf16_lo(r[i]), bf16_lo(o[i])), __fadd_rn(bf16_hi(r[i]), bf16_hi(o[i])));
                        v = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                    if (j < nt) *reinterpret_cast<uint4*>(static_cast<uint16_t*>(a.out) + (size_t)(t0 + j) * a.N + n + 8 * (lane & 3)) = v;
                }
                __syncwarp();
            }
            acc ^= 1;
            if (acc == 0) acc_phase ^= 1;
        }
    }

    // status[0]: 1 producer / free stage, 2 MMA / free accumulator, 3 MMA / operands, 4 epilogue / accumulator; status[1] CTA, status[2] thread
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
        while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
        __syncthreads();
    }
    cluster_sync_all();
    tc_fence_after();
    if (warp == 1) tmem_dealloc2(tmem_base, 512);
}

// ---- digits ----------------------------------------------------------------------------------------------------------------------
// INT8 rows (row r, or row tok[r] if tok is given) -> three planes of 4-bit digits [3][rows][K / 2], and their scales.  A thread turns 16 values.
__global__ void __launch_bounds__(256) digits_kernel(const int8_t* __restrict__ xq, const float* __restrict__ xs, const int32_t* __restrict__ tok,
                                                     int64_t rows, int64_t R, int K, uint32_t* __restrict__ dig, float* __restrict__ ds) {
    pdl_launch_dependents();
    pdl_wait();
    const int per = K / 16;
    const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x, r = i / per;
    if (r >= rows) return;
    const int v = (int)(i - r * per);
    const int64_t src = tok != nullptr ? tok[r] : r;
    const uint4 x = *reinterpret_cast<const uint4*>(xq + src * K + 16 * v);
    uint32_t lo[3], hi[3];
    digits8(x.x, x.y, lo);
    digits8(x.z, x.w, hi);
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint2*>(dig + (p * rows + r) * (K / 8) + 2 * v) = make_uint2(lo[p], hi[p]);
    if (v == 0 && ds != nullptr && r < R) ds[r] = xs[src];
}

// Block codes [E][N][K / 128] -> block factors [E][ceil(N / 128)][K / 128][512]: word 4 (row % 32) + row / 32 of a tile holds the four
// factors of a row.  A warp turns 16 blocks of 128 values of one tile; rows past N get the factor 2.  Several stacks of matrices in one launch.
struct FactorJob {
    const uint8_t* bcodes;
    uint4* out;
    int64_t warp0;           // first warp of the job
    int ftiles, N, kb128;
};
struct FactorJobs {
    FactorJob j[SCMX_F4_JOBS];
    int n;
    int64_t warps;
};

__global__ void __launch_bounds__(256) factors_kernel(const FactorJobs jobs) {
    pdl_launch_dependents();
    const int lane = threadIdx.x & 31;
    int64_t w = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    pdl_wait();
    if (w >= jobs.warps) return;
    int i0 = 0;
    while (i0 + 1 < jobs.n && w >= jobs.j[i0 + 1].warp0) ++i0;
    const FactorJob& job = jobs.j[i0];
    const int ftiles = job.ftiles, N = job.N, kb128 = job.kb128, chunks = (kb128 + 15) / 16;
    w -= job.warp0;
    const int64_t tile = w / chunks;
    const int k0 = (int)(w - tile * chunks) * 16, e = (int)(tile / ftiles), r0 = (int)(tile - (int64_t)e * ftiles) * 128 + lane;
    const bool wide = (kb128 & 15) == 0 && (reinterpret_cast<uintptr_t>(job.bcodes) & 15) == 0;
    uint32_t b[4][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int r = r0 + 32 * j;
        const uint8_t* p = job.bcodes + ((int64_t)e * N + r) * kb128 + k0;
        b[j][0] = b[j][1] = b[j][2] = b[j][3] = 0;
        if (r >= N) continue;
        if (wide) {
            const uint4 v = *reinterpret_cast<const uint4*>(p);
            b[j][0] = v.x; b[j][1] = v.y; b[j][2] = v.z; b[j][3] = v.w;
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (k0 + i < kb128) b[j][i >> 2] |= (uint32_t)p[i] << (8 * (i & 3));
        }
    }
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if (k0 + i < kb128)
            job.out[(tile * kb128 + k0 + i) * 32 + lane] = make_uint4(f4_factors((b[0][i >> 2] >> (8 * (i & 3))) & 255u), f4_factors((b[1][i >> 2] >> (8 * (i & 3))) & 255u),
                                                                      f4_factors((b[2][i >> 2] >> (8 * (i & 3))) & 255u), f4_factors((b[3][i >> 2] >> (8 * (i & 3))) & 255u));
}

static int run_f4(const uint32_t* dig, int64_t drows, const uint32_t* codes, const uint8_t* factors, int64_t rows_w, GemmArgs& g, cudaStream_t st) {
    F4Args fa = {};
    fa.ftiles = (g.N + 127) / 128;
    g.wait_ns = g_wait_limit_ns;
    fa.g = g;
    F4Maps maps;
    int rc = make_map_u8(&maps.w, codes, rows_w, g.K / 2, 128, 128, 128);
    if (rc) return rc;
    const int64_t kb128 = g.K / 128;
    rc = make_map_planes(&maps.f, factors, (int64_t)(g.E > 0 ? g.E : 1) * fa.ftiles, 4 * kb128, 128, 128, 512 * kb128, 8, 1, false);
    if (rc) return rc;
    for (int i = 0; i < F4_TNH / 8; ++i) {
        rc = make_map_planes(&maps.x[i], dig, 3, drows, g.K / 2, g.K / 2, drows * (g.K / 2), 8 * (i + 1), 3);
        if (rc) return rc;
    }
    int pairs = sm_count() / 2;
    if (g.E == 0) {
        // Token tiles: as few rounds of the pairs as possible, each a step of fixed cost (the operands' way, ~450 cycles a stage) and one per token.
        const int tiles_n = (g.N + 255) / 256;
        int best = 0x7fffffff;
        for (int n = (g.M + 2 * F4_TNH - 1) / (2 * F4_TNH), last = 2 * n + 1; n <= last; ++n) {
            const int tnh = f4_tnh(g.M, n), cost = ((n * tiles_n + pairs - 1) / pairs) * (56 + 2 * tnh);
            if (cost < best) {
                best = cost;
                fa.tnh = tnh;
            }
        }
        fa.tiles_m = (g.M + 2 * fa.tnh - 1) / (2 * fa.tnh);
        const int64_t tiles = fa.tiles_m * (int64_t)tiles_n;
        if (tiles < pairs) pairs = (int)tiles;
    }
    static bool configured[64] = {};
    const int dev = current_device();
    SCMX_REQUIRE(dev >= 0, SCMX_ECUDA, "no current CUDA device (ordinal 0..63)");
    if (!configured[dev]) {
        SCMX_CUDA_OK(cudaFuncSetAttribute(gemm_f4_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, F4Smem::TOTAL));
        configured[dev] = true;
    }
    SCMX_PDL_OK("gemm_f4_kernel", launch_pdl(gemm_f4_kernel, dim3(2 * pairs), dim3(F4_THREADS), (size_t)F4Smem::TOTAL, st, maps, fa));
    return SCMX_OK;
}

}  // namespace scmx

using namespace scmx;

extern "C" int scmx_f4_supported(const scmx_format* fmt, int64_t K) {
    DevFormat f;
    if (make_dev_format(fmt, &f)) return 0;
    // the default format: e2m1 magnitudes, blocks of 32 times 1, 2, 4, 8; integers below 2^22 in the accumulators
    return f.mag_lo == 0x03020100u && f.mag_hi == 0x0C080604u && f.block == 32 && f.bc_bits == 2 && f.pow2 && K % 128 == 0 && K <= 10240;
}

extern "C" int scmx_digits(const int8_t* xq, const float* xs, const int32_t* tok, int64_t rows, int64_t R, int64_t K, uint32_t* dig, float* ds,
                           void* stream) {
    SCMX_REQUIRE(xq && dig && rows >= 0 && K > 0 && K % 32 == 0 && K < (1ll << 30) && (!ds || xs), SCMX_EINVAL, "digits: rows=%lld K=%lld", (long long)rows, (long long)K);
    SCMX_REQUIRE(((reinterpret_cast<uintptr_t>(xq) | reinterpret_cast<uintptr_t>(dig)) & 15) == 0, SCMX_EINVAL, "digits: rows must be 16-byte aligned");
    if (rows == 0) return SCMX_OK;
    const int64_t blocks = (rows * (K / 16) + 255) / 256;
    SCMX_REQUIRE(blocks < (1ll << 31), SCMX_ELIMIT, "digits: rows=%lld K=%lld", (long long)rows, (long long)K);
    SCMX_PDL_OK("digits_kernel", launch_pdl(digits_kernel, dim3((unsigned)blocks), dim3(256), 0, (cudaStream_t)stream, xq, xs, tok, rows, R, (int)K, dig, ds));
    return SCMX_OK;
}

static int f4_common(const char* who, const uint32_t* dig, int64_t drows, const uint32_t* codes, const uint8_t* factors, int64_t N, int64_t K,
                     const scmx_format* fmt, const void* res, const void* out) {
    SCMX_REQUIRE(scmx_f4_supported(fmt, K), SCMX_EFORMAT, "%s: needs the default format, K %% 128 == 0 and K <= 10240", who);
    SCMX_REQUIRE(dig && codes && factors && N % 32 == 0 && drows >= 0 && drows < (1ll << 30) &&
                     ((reinterpret_cast<uintptr_t>(dig) | reinterpret_cast<uintptr_t>(codes) | reinterpret_cast<uintptr_t>(factors) | reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(res)) & 15) == 0,
                 SCMX_EINVAL, "%s: N must be a multiple of 32; digits, codes, factors, res and out 16-byte aligned", who);
    return SCMX_OK;
}

extern "C" int scmx_f4_factors(const scmx_f4_job* jobs, int n, void* stream) {
    SCMX_REQUIRE(jobs && n >= 0 && n <= SCMX_F4_JOBS, SCMX_EINVAL, "f4_factors: %d jobs (at most %d)", n, SCMX_F4_JOBS);
    FactorJobs f = {};
    for (int i = 0; i < n; ++i) {
        const scmx_f4_job& j = jobs[i];
        SCMX_REQUIRE(j.bcodes && j.factors && j.E >= 0 && j.N > 0 && j.K > 0 && j.K % 128 == 0 && j.K < (1ll << 30) && j.N < (1ll << 30) &&
                         (reinterpret_cast<uintptr_t>(j.factors) & 15) == 0, SCMX_EINVAL, "f4_factors: E=%lld N=%lld K=%lld", (long long)j.E, (long long)j.N, (long long)j.K);
        f.j[f.n++] = {j.bcodes, reinterpret_cast<uint4*>(j.factors), f.warps, (int)((j.N + 127) / 128), (int)j.N, (int)(j.K / 128)};
        f.warps += j.E * ((j.N + 127) / 128) * ((j.K / 128 + 15) / 16);
        SCMX_REQUIRE(f.warps < (1ll << 33), SCMX_ELIMIT, "f4_factors: too many blocks");
    }
    if (f.warps == 0) return SCMX_OK;
    SCMX_PDL_OK("factors_kernel", launch_pdl(factors_kernel, dim3((unsigned)((f.warps + 7) / 8)), dim3(256), 0, (cudaStream_t)stream, f));
    return SCMX_OK;
}

extern "C" int scmx_mm_f4(const uint32_t* dig, int64_t drows, const uint32_t* codes, const uint8_t* factors, int64_t M, int64_t N, int64_t K,
                          const scmx_format* fmt, int epi, const float* xscale, const float* wscale, const uint16_t* res, void* out,
                          int32_t* status, void* stream) {
    int rc = check_common("mm_f4", N, K, epi, xscale, wscale, out, status);
    if (rc) return rc;
    rc = f4_common("mm_f4", dig, drows, codes, factors, N, K, fmt, res, out);
    if (rc) return rc;
    SCMX_REQUIRE(M >= 0 && M <= drows && (epi != 2 || res), SCMX_EINVAL, "mm_f4: M=%lld of %lld rows", (long long)M, (long long)drows);
    if (M == 0) return SCMX_OK;
    GemmArgs g = {};
    g.M = (int)M; g.N = (int)N; g.K = (int)K; g.epi = epi; g.xscale = xscale; g.wscale = wscale; g.res = res; g.out = out; g.status = status;
    return run_f4(dig, drows, codes, factors, N, g, (cudaStream_t)stream);
}

extern "C" int scmx_moe_mm_f4(const uint32_t* dig, int64_t drows, int64_t R, const uint32_t* codes, const uint8_t* factors, const float* wscale,
                              const int32_t* off, int E, int64_t N, int64_t K, const scmx_format* fmt, int epi, const float* xscale, void* out,
                              int32_t* status, void* stream) {
    int rc = check_common("moe_mm_f4", N, K, epi, xscale, wscale, out, status);
    if (rc) return rc;
    rc = f4_common("moe_mm_f4", dig, drows, codes, factors, N, K, fmt, nullptr, out);
    if (rc) return rc;
    SCMX_REQUIRE(epi != 2 && E >= 1 && E <= F4_MAX_E && R >= 0 && R <= drows && off && (int64_t)E * N < (1ll << 31), SCMX_EINVAL,
                 "moe_mm_f4: epi 0, 1 or 3; 1..%d experts; R=%lld of %lld rows", F4_MAX_E, (long long)R, (long long)drows);
    if (R == 0) return SCMX_OK;
    GemmArgs g = {};
    g.M = (int)R; g.N = (int)N; g.K = (int)K; g.epi = epi; g.xscale = xscale; g.wscale = wscale; g.out = out;
    g.off = off; g.E = E; g.e_begin = 0; g.e_end = E; g.status = status;
    return run_f4(dig, drows, codes, factors, (int64_t)E * N, g, (cudaStream_t)stream);
}
