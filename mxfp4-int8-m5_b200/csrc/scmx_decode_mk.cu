// One decode step of a dense (Qwen3-style) stack as ONE persistent kernel: every SM keeps a CTA resident for the whole step and the CTAs move
// through the phases of each layer together.  A batch-1 step is a chain of ~10 tiny dependent kernels per layer; launched separately each link
// costs a grid drain and a launch, about 5 us, while the weights it reads would take 1 us at HBM speed.
//
// Per layer:
//   P1  RMSNorm + INT8 of h (each CTA, shared memory) -> q|k|v rows -> y (bf16)
//   P3  per (kv head, split) CTA: q/k RMSNorm + rotary embedding of the new token, cache append, attention over its positions -> partial
//       softmax states; one CTA per query head combines its splits -> o
//   P4  INT8 of o -> o-projection + residual -> h
//   P5  RMSNorm + INT8 of h -> gate|up with SwiGLU -> act
//   P6  INT8 of act -> down + residual -> h
//
// Bound by latency: what a link costs beyond its 4 us a layer of weights at HBM speed.  Two things keep it short.
// (1) Rows travel between CTAs as packets of 8 bytes, 4 of data and 4 of an epoch (launch and layer) written by one store: a reader polls the packets
//     themselves.  There is no barrier and no fence: a link is one store and one load through L2, about 1 us, where a grid barrier (fence, atomic,
//     poll) and the load after it took 2.5 - 4 us.  A buffer is not rewritten before its readers are done, because every CTA has rows in
//     every phase: who writes phase p of layer i + 1 has seen phase p - 1 complete, and so on back to phase p + 1 of layer i, whose rows were written after
//     their CTAs had read phase p of layer i.
// (2) Weights stream through rings in shared memory, one per warp, filled by asynchronous copies of the lanes that use them: the order of chunks is
//     known from the start, so the ring runs ahead through phases and layers (170 KB per SM, most of a layer) while the CTA waits, joins or reduces.
// Work item of a warp: 4 rows x 1024 columns; a row group's items are summed through shared memory (exact integers).
// 8 layers of width 2048 at 1500 positions with the head: 342 us with grid barriers and weights in registers, 312 us here.  A layer (32 us): rows of q|k|v 2.3 (and 2.0
// until the input row is there), attention 6.5, its combination and exchange 4.9, o 1.5, h 2.8, gate|up 5.4, act 1.7, down 3.7; two items at a time per warp changed
// nothing (321), polling without a pause slowed the writers (375).
// Arithmetic: the device functions of the stand-alone kernels (row kernels, GEMV, q/k/v epilogue, decode attention), so the step produces the
// same bits as the chain of those kernels.  Callers: e2e/decode.py:29-110 of the reference is the chain.
//
// Every wait is bounded (scmx_set_wait_limit_ns): a thread that gives up raises the abort word and writes the status word; the others see the abort word in their
// own waits; a CTA agrees on it at its next barrier and returns.  The launch is cooperative, so all CTAs are co-resident.
#include <algorithm>
#include "scmx_attn_core.cuh"
#include "scmx_common.cuh"
#include "scmx_gemv_core.cuh"
#include "scmx_ptx.cuh"

namespace scmx {

constexpr int MK_THREADS = 256;                       // the attention core wants 150 registers a thread: 384, 448 and 512 threads spill (357 - 375 us for the step below)
constexpr int MK_WARPS = MK_THREADS / 32;
constexpr int MK_MAXK = 6144;
constexpr int MK_MAXHQ = 32;
constexpr int MK_MAXROWS = 384;                      // output rows of a CTA in one phase at most: the widest phase, 12288 rows, on 32 SMs
constexpr int MK_CODES = 4 * 512, MK_CHUNK = MK_CODES + 32;      // bytes of an item: codes of 4 rows, their block codes
constexpr int MK_SLOTS = 9;
constexpr int MK_MAXLAYERS = 256;                     // of one launch: its table of weights lies in shared memory
constexpr unsigned MK_BACKOFF_NS = 40;
constexpr int MK_MARKS = 9;                          // diagnostic marks of a layer

struct MkArgs {
    const scmx_decode_layer* layers;
    int n_layers, D, F, hq, hk, nsplit;
    int first;            // number of the first layer, for the status word
    float eps, scale;
    const float* inv_freq;
    const float* rope_cs;
    int64_t rope_rows, cap;
    const int32_t* pos_dev;
    uint16_t* h;          // bf16 [D] residual stream, in and out
    uint32_t* head;       // [0] epoch of the last launch, [1] abort word (zero at launch)
    uint2 *xh[2], *xy, *xact, *xo, *xpart;      // packets: h after P6 / P4, y, act, o: {two bf16, epoch}; partial states [hq][nsplit][d + 2]: {float, epoch}
    int32_t* status;
    uint64_t wait_ns;
    unsigned long long* trace;   // diagnostic: null, or CTA 0 stores its cycle counter at every phase boundary
    int n_trace;
    unsigned long long* arrivals;      // diagnostic: null, or every CTA stores the global timer at its arrival at this link (1-based, five a layer)
    int link;
};

struct MkSmem {
    __align__(16) int8_t xq[MK_MAXK];       // INT8 input row; of every 32 values the first 16 in the first half, the others in the second
    int part[MK_MAXROWS * 6];               // [row group][step][4]
    float ws[MK_MAXROWS];
    float red[MK_WARPS];
    double dred[MK_WARPS];
    uint32_t res[MK_MAXROWS / 2];           // residual of the CTA's rows, two a word
};

__shared__ MkSmem sm;     // one instance per CTA

// ---- packets ------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void put(uint2* p, uint32_t data, uint32_t epoch) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((uint64_t)data | ((uint64_t)epoch << 32)) : "memory");
}
__device__ __forceinline__ uint2 get(const uint2* p) {
    uint64_t v;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return make_uint2((uint32_t)v, (uint32_t)(v >> 32));
}
// Two neighbouring packets; each is read whole.
__device__ __forceinline__ void get2(const uint2* p, uint2& a, uint2& b) {
    uint64_t x, y;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(x), "=l"(y) : "l"(p) : "memory");
    a = make_uint2((uint32_t)x, (uint32_t)(x >> 32));
    b = make_uint2((uint32_t)y, (uint32_t)(y >> 32));
}
// One turn of a wait: false once the limit has run out or another thread has given up.
struct MkWait {
    uint32_t turns = 0;
    uint64_t t0 = 0;
    __device__ __forceinline__ bool go_on(const MkArgs& a, int code) {
        __nanosleep(MK_BACKOFF_NS);              // a row's readers are all CTAs: polling without a pause crowds out the writers
        if ((++turns & 255u) != 0) return true;
        uint32_t ab;
        asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(ab) : "l"(a.head + 1) : "memory");
        if (ab) return false;
        const uint64_t now = globaltimer_ns();
        if (!t0) t0 = now;
        if (now - t0 <= a.wait_ns) return true;
        atomicExch(a.head + 1, 1u);
        atomicCAS(a.status, 0, code);
        return false;
    }
};
// Eight bf16 values, four packets; zero (and bad set) after a time-out.
__device__ __forceinline__ uint4 get8(const MkArgs& a, const uint2* p, uint32_t epoch, int code, bool& bad) {
    MkWait w;
    for (;;) {
        uint2 q[4];
        get2(p, q[0], q[1]);
        get2(p + 2, q[2], q[3]);
        if (q[0].y == epoch && q[1].y == epoch && q[2].y == epoch && q[3].y == epoch) return make_uint4(q[0].x, q[1].x, q[2].x, q[3].x);
        if (!w.go_on(a, code)) {
            bad = true;
            return make_uint4(0, 0, 0, 0);
        }
    }
}

__device__ __forceinline__ void mk_mark(const MkArgs& a, int& ti) {
    if (a.trace != nullptr && blockIdx.x == 0 && threadIdx.x == 0 && ti < a.n_trace) a.trace[ti] = (unsigned long long)clock64();
    ++ti;
}

__device__ __forceinline__ void mk_arrive(const MkArgs& a, int link) {
    if (a.arrivals != nullptr && threadIdx.x == 0 && link == a.link) a.arrivals[blockIdx.x] = globaltimer_ns();
}

// ---- input row of a phase: bf16 row -> INT8 row in shared memory, returns the scale ---------------------------------------------
__device__ __forceinline__ float amax8(const uint4& r) {
    const uint32_t w[4] = {r.x, r.y, r.z, r.w};
    float m = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) m = fmaxf(m, fmaxf(fabsf(__uint_as_float(w[j] << 16)), fabsf(__uint_as_float(w[j] & 0xFFFF0000u))));
    return m;
}

// Sums and maxima over the CTA behind one barrier: every thread adds the warps' parts (a sum of squares is exact in 64 bits, so its order is free).
__device__ __forceinline__ double mk_sum(double v) {
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) sm.dred[threadIdx.x >> 5] = v;
    __syncthreads();
    v = 0.0;
#pragma unroll
    for (int i = 0; i < MK_WARPS; ++i) v += sm.dred[i];
    return v;
}
__device__ __forceinline__ float mk_max(float v) {
    v = warp_max(v);
    if ((threadIdx.x & 31) == 0) sm.red[threadIdx.x >> 5] = v;
    __syncthreads();
    v = sm.red[0];
#pragma unroll
    for (int i = 1; i < MK_WARPS; ++i) v = fmaxf(v, sm.red[i]);
    return v;
}

// NORM: RMSNorm with weights nw first.  x: packets, or (x null) the plain row.  The arithmetic of act_quant / rmsnorm_quant.
template <bool NORM>
__device__ __forceinline__ float mk_input(const MkArgs& a, const uint2* x, const uint16_t* plain, uint32_t epoch, const uint16_t* nw, int K, int code, bool& bad) {
    constexpr int NV = (MK_MAXK / 8 + MK_THREADS - 1) / MK_THREADS;      // vectors of a thread
    const int nv = K / 8, tid = threadIdx.x;
    uint4 r[NV], wv[NV];
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int v = tid + MK_THREADS * i;
        r[i] = wv[i] = make_uint4(0, 0, 0, 0);
        if (NORM && v < nv) wv[i] = __ldg(reinterpret_cast<const uint4*>(nw) + v);
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int v = tid + MK_THREADS * i;
        if (v < nv) r[i] = x != nullptr ? get8(a, x + 4 * v, epoch, code, bad) : reinterpret_cast<const uint4*>(plain)[v];
    }
    float amax = 0.0f;
    if (NORM) {
        double ss = 0.0;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t w[4] = {r[i].x, r[i].y, r[i].z, r[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) ss += sq_f64(bf16_lo(w[j])) + sq_f64(bf16_hi(w[j]));
        }
        ss = mk_sum(ss);
        const float inv = rms_inverse(ss, K, a.eps);
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t x4[4] = {r[i].x, r[i].y, r[i].z, r[i].w}, w[4] = {wv[i].x, wv[i].y, wv[i].z, wv[i].w};
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t t = pack_bf16x2(__fmul_rn(bf16_lo(x4[j]), inv), __fmul_rn(bf16_hi(x4[j]), inv));
                o[j] = pack_bf16x2(__fmul_rn(bf16_lo(w[j]), bf16_lo(t)), __fmul_rn(bf16_hi(w[j]), bf16_hi(t)));
            }
            r[i] = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
#pragma unroll
    for (int i = 0; i < NV; ++i) amax = fmaxf(amax, amax8(r[i]));
    amax = mk_max(amax);
    float s, qi;
    quant_scale(amax, s, qi);
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int v = tid + MK_THREADS * i;
        if (v < nv) {
            const uint32_t x4[4] = {r[i].x, r[i].y, r[i].z, r[i].w};
            *reinterpret_cast<uint2*>(sm.xq + ((v >> 1) & 1) * (K / 2) + (v >> 2) * 16 + (v & 1) * 8) =
                make_uint2(quant4(bf16_lo(x4[0]), bf16_hi(x4[0]), bf16_lo(x4[1]), bf16_hi(x4[1]), qi),
                           quant4(bf16_lo(x4[2]), bf16_hi(x4[2]), bf16_lo(x4[3]), bf16_hi(x4[3]), qi));
        }
    }
    return s;
}

// ---- the warp's stream of weights -----------------------------------------------------------------------------------------------
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy4(uint32_t dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}

// At most n of the thread's groups of copies are still on their way.
__device__ __forceinline__ void mk_copies_wait(int n) {
    static_assert(MK_SLOTS == 9, "one case per slot");
    switch (n) {
        case 8: asm volatile("cp.async.wait_group 8;" ::: "memory"); break;
        case 7: asm volatile("cp.async.wait_group 7;" ::: "memory"); break;
        case 6: asm volatile("cp.async.wait_group 6;" ::: "memory"); break;
        case 5: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
        case 4: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
        case 3: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
        case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
        case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
        default: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    }
}

struct MkPhase {
    int groups, steps;       // row groups in all, items per group
    int base, count;         // the CTA's row groups: equal shares
    uint32_t inv;            // item / steps = item * inv >> 16 for the items of a CTA
    __device__ __forceinline__ int group_of(int item) const { return (int)(((uint32_t)item * inv) >> 16); }
};

// ---- the kernel's phases share this ------------------------------------------------------------------------------------------------
struct MkStream {
    const MkArgs& a;
    const MkPhase* ph;
    const unsigned long long* table;      // [layer][8]: codes and block codes of the four products
    uint32_t ring;           // shared address of the warp's ring
    int layer, phase, item;  // next item to request
    uint32_t dst;
    const uint32_t* codes;
    const uint8_t* bcodes;
    int lane, warp;

    __device__ __forceinline__ void load_layer() {
        codes = reinterpret_cast<const uint32_t*>(table[8 * layer + phase]);
        bcodes = reinterpret_cast<const uint8_t*>(table[8 * layer + 4 + phase]);
    }
    // to the next phase in which the warp has an item
    __device__ __forceinline__ void settle() {
        bool moved = false;
        while (layer < a.n_layers && item >= ph[phase].count * ph[phase].steps) {
            item = warp;
            moved = true;
            if (++phase == 4) {
                phase = 0;
                ++layer;
            }
        }
        if (moved && layer < a.n_layers) load_layer();
    }
    __device__ __forceinline__ void begin() {
        layer = phase = 0;
        item = warp;
        dst = ring;
        load_layer();
        settle();
    }
    __device__ __forceinline__ void request() {
        if (layer < a.n_layers) {
            const MkPhase& p = ph[phase];
            const int g = p.group_of(item), s = item - g * p.steps, row = 4 * (p.base + g);
            const uint32_t* c = codes + ((size_t)row * p.steps + s) * 128 + 4 * lane;      // K / 8 = 128 steps words a row
#pragma unroll
            for (int q = 0; q < 4; ++q) copy16(dst + 512 * q + 16 * lane, c + (size_t)q * p.steps * 128);
            // the 32 lanes x 32 codes of a step span 8 block-code bytes per row
            if (lane < 8) copy4(dst + MK_CODES + 4 * lane, bcodes + ((size_t)(row + (lane >> 1)) * p.steps + s) * 8 + 4 * (lane & 1));
            item += MK_WARPS;
            settle();
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        dst += MK_CHUNK;
        if (dst == ring + MK_SLOTS * MK_CHUNK) dst = ring;
    }
};

// Totals of an item: 4 rows x 1024 columns.
__device__ __forceinline__ void mk_item(const uint8_t* slot, const int8_t* xq, int half, int s, int lane, int (&tot)[4]) {
    const uint32_t mlo = 0x03020100u, mhi = 0x0C080604u;      // 2 x E2M1 magnitudes 0 1 2 3 | 4 6 8 12
    const int blk = s * 32 + lane;
    const uint4 xa = *reinterpret_cast<const uint4*>(xq + 16 * blk), xb = *reinterpret_cast<const uint4*>(xq + half + 16 * blk);
    const uint32_t x[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
    const int sh = 2 * (lane & 3);                            // the lane's 32-block inside its block-code byte
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint4 wv = *reinterpret_cast<const uint4*>(slot + 512 * q + 16 * lane);
        const uint32_t ww[4] = {wv.x, wv.y, wv.z, wv.w};
        const uint32_t code = (slot[MK_CODES + 8 * q + (lane >> 2)] >> sh) & 3u;
        // magnitudes of the positive and of the negative codes by sign-replicating byte permutes (a selector nibble with its top bit set yields the
        // replicated top bit of the selected byte, 0 for a magnitude), two DP4A chains
        int bp = 0, bn = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t w = ww[j], wx = w ^ 0x88888888u;
            bp = dp4a_ss(x[2 * j], prmt(mlo, mhi, w), bp);
            bn = dp4a_ss(x[2 * j], prmt(mlo, mhi, wx), bn);
            bp = dp4a_ss(x[2 * j + 1], prmt(mlo, mhi, w >> 16), bp);
            bn = dp4a_ss(x[2 * j + 1], prmt(mlo, mhi, wx >> 16), bn);
        }
        tot[q] = (bp - bn) << code;
    }
}

// Requests a range of the caches into L2 (whole 16-byte pieces).
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
    const uint64_t a = (uint64_t)p & ~15ull, n = (((uint64_t)p + bytes) & ~15ull) - a;
    if (n != 0) asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a), "r"((uint32_t)n) : "memory");
}

// ---- the new token's q (G heads), k, v of one key/value head: RMSNorm, rotary embedding (arithmetic of qkv_norm_kernel) ----
template <int G, int HD>
struct QkvSmem {
    float vals[(G + 2) * HD];
    float inv[G + 1];
    float cs[HD / 2], sn[HD / 2];
    uint16_t wq[HD], wk[HD];
    __align__(16) uint16_t q[G * HD];
    __align__(16) uint16_t k[HD];
    __align__(16) uint16_t v[HD];
};

template <int G, int HD>
__device__ __forceinline__ void qkv_prepare(QkvSmem<G, HD>& qs, const MkArgs& a, const uint16_t* q_norm, const uint16_t* k_norm, int kvh, int64_t pos, uint32_t epoch,
                                            int code, bool& bad) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int half = HD / 2, NE = (G + 2) * HD;
    for (int i = tid; i < HD; i += MK_THREADS) {
        qs.wq[i] = q_norm[i];
        qs.wk[i] = k_norm[i];
    }
    for (int i = tid; i < half; i += MK_THREADS) {
        if (a.rope_cs != nullptr && pos < a.rope_rows) {
            qs.cs[i] = a.rope_cs[pos * HD + i];
            qs.sn[i] = a.rope_cs[pos * HD + half + i];
        } else {
            const float ang = __fmul_rn((float)pos, a.inv_freq[i]);
            double s, c;
            sincos((double)ang, &s, &c);
            qs.cs[i] = (float)c;
            qs.sn[i] = (float)s;
        }
    }
    for (int e = 2 * tid; e < NE; e += 2 * MK_THREADS) {
        const int hh = e / HD, dd = e - hh * HD;
        const int src = hh < G ? (kvh * G + hh) * HD : (hh == G ? (a.hq + kvh) * HD : (a.hq + a.hk + kvh) * HD);
        uint2 p;
        MkWait w;
        while ((p = get(a.xy + (src + dd) / 2)).y != epoch)
            if (!w.go_on(a, code)) {
                bad = true;
                break;
            }
        qs.vals[e] = bf16_lo(p.x);
        qs.vals[e + 1] = bf16_hi(p.x);
    }
    __syncthreads();
    for (int hh = warp; hh < G + 1; hh += MK_WARPS) {
        double ss = 0.0;
        for (int i = lane; i < HD; i += 32) {
            const double x = (double)qs.vals[hh * HD + i];
            ss += x * x;
        }
        ss = warp_sum(ss);
        if (lane == 0) qs.inv[hh] = rms_inverse(ss, HD, a.eps);
    }
    __syncthreads();
    auto normed = [&](int hh, int dd) -> float {
        const uint16_t* w = hh < G ? qs.wq : qs.wk;
        return rbf(__fmul_rn(bf16_to_f32(w[dd]), rbf(__fmul_rn(qs.vals[hh * HD + dd], qs.inv[hh]))));
    };
    for (int e = tid; e < NE; e += MK_THREADS) {
        const int hh = e / HD, dd = e - hh * HD;
        if (hh > G) {
            qs.v[dd] = f32_to_bf16(qs.vals[e]);
            continue;
        }
        const bool lo = dd < half;
        const float self = normed(hh, dd), other = normed(hh, lo ? dd + half : dd - half);
        const int i = lo ? dd : dd - half;
        const float r = lo ? rbf(__fsub_rn(__fmul_rn(self, qs.cs[i]), __fmul_rn(other, qs.sn[i])))
                           : rbf(__fadd_rn(__fmul_rn(other, qs.sn[i]), __fmul_rn(self, qs.cs[i])));
        if (hh < G) qs.q[hh * HD + dd] = f32_to_bf16(r);
        else qs.k[dd] = f32_to_bf16(r);
    }
    __syncthreads();
}

// One (kv head, split) task of P3; out of line, so that its registers are its own.
template <int G, int HD>
__device__ __noinline__ bool mk_attention(const MkArgs& a, const scmx_decode_layer& L, int kvh, int split, int64_t t0, int64_t t1, int64_t pos, uint32_t epoch, int code) {
    __shared__ QkvSmem<G, HD> qs;
    __shared__ AttnSmem<G, HD> as;
    constexpr int stride = HD + 2;
    const int tid = threadIdx.x;
    const bool in_cache = pos < a.cap;
    bool bad = false;
    qkv_prepare<G, HD>(qs, a, L.q_norm, L.k_norm, kvh, pos, epoch, code, bad);
    uint16_t* kc = L.k_cache + (size_t)kvh * a.cap * HD;
    uint16_t* vc = L.v_cache + (size_t)kvh * a.cap * HD;
    if (split == 0 && in_cache && tid < HD / 8) {
        reinterpret_cast<uint4*>(kc + pos * HD)[tid] = reinterpret_cast<const uint4*>(qs.k)[tid];
        reinterpret_cast<uint4*>(vc + pos * HD)[tid] = reinterpret_cast<const uint4*>(qs.v)[tid];
    }
    uint2* part = a.xpart + ((size_t)kvh * G * a.nsplit + split) * stride;
    attn_split<G, HD>(qs.q, kc, vc, t0, t1, in_cache ? pos : -1, qs.k, qs.v, a.scale,
                      [&](int g, int e, float v) { put(part + (size_t)g * a.nsplit * stride + e, __float_as_uint(v), epoch); }, as);
    return bad;
}

// The splits of a query head (the arithmetic of attn_combine_cta): thread e owns output element e.
template <int HD>
__device__ __noinline__ bool mk_combine(const MkArgs& a, int head, int active, uint32_t epoch, int code) {
    __shared__ float ml[32][2], coef[33];
    constexpr int stride = HD + 2;
    const int tid = threadIdx.x;
    const uint2* p = a.xpart + (size_t)head * a.nsplit * stride;
    bool bad = false;
    __syncthreads();
    if (tid < 2 * active) {                               // a split's last packets; its other ones were stored before, mostly
        uint2 v;
        MkWait w;
        while ((v = get(p + (tid >> 1) * stride + HD + (tid & 1))).y != epoch)
            if (!w.go_on(a, code)) {
                bad = true;
                break;
            }
        ml[tid >> 1][tid & 1] = __uint_as_float(v.x);
    }
    __syncthreads();
    float v0[32];
    if (tid < HD && !bad) {
        MkWait w;
        for (bool late = true; late;) {                   // all splits' packets are requested together
            late = false;
#pragma unroll
            for (int s = 0; s < 32; ++s) {
                v0[s] = 0.0f;
                if (s < active) {
                    const uint2 v = get(p + s * stride + tid);
                    v0[s] = __uint_as_float(v.x);
                    late |= v.y != epoch;
                }
            }
            if (late && !w.go_on(a, code)) {
                bad = true;
                break;
            }
        }
    }
    if (tid >= HD && tid < HD + 32) {                     // the weights meanwhile, a split a lane
        const int s = tid - HD;
        const float ms = s < active ? ml[s][0] : -INFINITY, mm = warp_max(ms);
        if (s < active) coef[s] = ms == -INFINITY ? 0.0f : exp2f(ms - mm);
        __syncwarp();
        if (s == 0) {
            float ll = 0.0f;
            for (int i = 0; i < active; ++i) ll += ml[i][1] * coef[i];
            coef[32] = ll;
        }
    }
    __syncthreads();
    if (tid < HD) {
        float av = 0.0f;
#pragma unroll
        for (int s = 0; s < 32; ++s)
            if (s < active) av += v0[s] * coef[s];
        const uint32_t b = f32_to_bf16(av / coef[32]), other = __shfl_down_sync(0xffffffffu, b, 1);      // whole warps
        if ((tid & 1) == 0) put(a.xo + (head * HD + tid) / 2, b | (other << 16), epoch);
    }
    return bad;
}

// ---- the kernel ------------------------------------------------------------------------------------------------------------
// TRACE: the form that stores the diagnostic's times.  They cost the step of 8 layers 2 of 317 us, so the product's form has none of them.
template <int G, int HD, bool TRACE>
__global__ void __launch_bounds__(MK_THREADS, 1) decode_step_kernel(const __grid_constant__ MkArgs a) {
    extern __shared__ __align__(16) uint8_t rings[];
    __shared__ MkPhase ph[4];
    __shared__ scmx_decode_layer layer[2];        // this one and the next
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int D = a.D, F = a.F, QD = a.hq * HD, NQKV = (a.hq + 2 * a.hk) * HD;
    if (tid < 4) {
        const int rows = tid == 0 ? NQKV : tid == 2 ? 2 * F : D, K = tid == 1 ? QD : tid == 3 ? F : D, g = rows / 4;
        const int lo = (int)((int64_t)g * blockIdx.x / gridDim.x), hi = (int)((int64_t)g * (blockIdx.x + 1) / gridDim.x);
        ph[tid] = {g, K / 1024, lo, hi - lo, 65536u / (uint32_t)(K / 1024) + 1u};
    }
    constexpr int LWORDS = (int)(sizeof(scmx_decode_layer) / 8);
    if (tid < LWORDS) reinterpret_cast<unsigned long long*>(&layer[0])[tid] = reinterpret_cast<const unsigned long long*>(a.layers)[tid];
    unsigned long long* table = reinterpret_cast<unsigned long long*>(rings + MK_WARPS * MK_SLOTS * MK_CHUNK);
    for (int i = tid; i < 8 * a.n_layers; i += MK_THREADS)        // codes[4], bcodes[4] are the first words of a layer
        table[i] = reinterpret_cast<const unsigned long long*>(a.layers + (i >> 3))[i & 7];
    const uint32_t base_epoch = *reinterpret_cast<volatile const uint32_t*>(a.head);
    __syncthreads();
    MkStream st = {a, ph, table, (uint32_t)__cvta_generic_to_shared(rings) + warp * (MK_SLOTS * MK_CHUNK), 0, 0, 0, 0, nullptr, nullptr, lane, warp};
    const uint8_t* ring = rings + warp * (MK_SLOTS * MK_CHUNK);
    const uint8_t *slot = ring, *ring_end = ring + MK_SLOTS * MK_CHUNK;
    st.begin();
    for (int i = 0; i < MK_SLOTS; ++i) st.request();

    int64_t pos = a.pos_dev[0];
    pos = pos < 0 ? 0 : pos;
    const bool in_cache = pos < a.cap;
    int64_t T = in_cache ? pos + 1 : a.cap;
    int64_t chunk;
    int active;
    attn_chunking(T, a.nsplit, chunk, active);
    const int kvh = blockIdx.x % a.hk, split = blockIdx.x / a.hk;
    const bool attends = split < active;
    const int64_t t0 = (int64_t)split * chunk, t1 = t0 + chunk < T ? t0 + chunk : T;
    const int my_head = (int)gridDim.x - 1 - (int)blockIdx.x;      // query head whose splits this CTA combines
    bool bad = false;
    int ti = 0;

    auto gave_up = [&]() {                                         // the CTA agrees; copies in flight land before it leaves
        if (!__syncthreads_or(bad)) return false;
        asm volatile("cp.async.wait_all;" ::: "memory");
        return true;
    };
    // one product: the warp's items, summed per row group; the caller then finishes the rows.  Slots are refilled afterwards (refill), off the chain; in
    // between only where a phase has more items than the ring.
    int used = 0;
    auto refill = [&]() {
        for (; used > 0; --used) st.request();
    };
    auto items = [&](const MkPhase& p, int K) {
        for (int it = warp; it < p.count * p.steps; it += MK_WARPS) {
            const int g = p.group_of(it), s = it - g * p.steps;
            if (used == MK_SLOTS) refill();
            mk_copies_wait(MK_SLOTS - 1 - used);
            __syncwarp();                                          // block codes were copied by other lanes
            int tot[4];
            mk_item(slot, sm.xq, K / 2, s, lane, tot);
            __syncwarp();
            ++used;
            slot += MK_CHUNK;
            if (slot == ring_end) slot = ring;
#pragma unroll
            for (int q = 0; q < 4; ++q) tot[q] = __reduce_add_sync(0xffffffffu, tot[q]);
            if (lane < 4) sm.part[(g * p.steps + s) * 4 + lane] = lane < 2 ? (lane ? tot[1] : tot[0]) : (lane == 3 ? tot[3] : tot[2]);
        }
    };
    auto total = [&](const MkPhase& p, int r) {                    // row r of the CTA's
        int t = 0;
        for (int s = 0; s < p.steps; ++s) t += sm.part[((r >> 2) * p.steps + s) * 4 + (r & 3)];
        return t;
    };
    // rows of a plain product or one with a residual: T(acc xs ws) (+ res), two a thread, as packets, and as a plain row if `plain`
    auto finish = [&](const MkPhase& p, float xs, bool res, uint2* out, uint16_t* plain, uint32_t epoch) {
        for (int r = 2 * tid; r < 4 * p.count; r += 2 * MK_THREADS) {
            const int n = 4 * p.base + r;
            float y0 = scale_acc(total(p, r), xs, sm.ws[r]), y1 = scale_acc(total(p, r + 1), xs, sm.ws[r + 1]);
            if (res) {
                const uint32_t h = sm.res[r >> 1];
                y0 = __fadd_rn(bf16_lo(h), y0);
                y1 = __fadd_rn(bf16_hi(h), y1);
            }
            const uint32_t two = pack_bf16x2(y0, y1);
            put(out + (n >> 1), two, epoch);
            if (plain != nullptr) *reinterpret_cast<uint32_t*>(plain + n) = two;
        }
    };
    // scales and residual of the CTA's rows, requested before the input row is awaited (the residual's packets are complete long before)
    auto ahead = [&](const MkPhase& p, const float* wscale, const uint2* res, const uint16_t* res_plain) {
        for (int r = tid; r < 4 * p.count; r += MK_THREADS) {
            const int n = 4 * p.base + r;
            sm.ws[r] = __ldg(wscale + n);
            if ((r & 1) == 0 && res != nullptr) sm.res[r >> 1] = get(res + (n >> 1)).x;
            else if ((r & 1) == 0 && res_plain != nullptr) sm.res[r >> 1] = *reinterpret_cast<const uint32_t*>(res_plain + n);
        }
    };

    for (int li = 0; li < a.n_layers; ++li) {
        const scmx_decode_layer& L = layer[li & 1];
        if (li + 1 < a.n_layers && tid < LWORDS)              // read after several barriers
            reinterpret_cast<unsigned long long*>(&layer[(li + 1) & 1])[tid] = reinterpret_cast<const unsigned long long*>(a.layers + li + 1)[tid];
        const uint32_t epoch = base_epoch + 1 + li;
        const int code = 1000 + 5 * (a.first + li), link = code - 1000;
        if (TRACE) mk_mark(a, ti);
        if (attends && tid < 2 && t1 > t0) {                  // the positions that this CTA will attend to
            const int64_t te = t1 < T - 1 ? t1 : T - 1;
            if (te > t0) prefetch_l2((tid ? L.v_cache : L.k_cache) + ((size_t)kvh * a.cap + t0) * HD, (uint32_t)(te - t0) * HD * 2);
        }
        // P1: input RMSNorm + INT8, q|k|v projection
        ahead(ph[0], L.wscale[0], nullptr, nullptr);
        float xs = mk_input<true>(a, li > 0 ? a.xh[0] : nullptr, a.h, epoch - 1, L.ln_in, D, code, bad);
        if (gave_up()) return;
        if (TRACE) mk_mark(a, ti);
        items(ph[0], D);
        __syncthreads();
        finish(ph[0], xs, false, a.xy, nullptr, epoch);
        if (TRACE) mk_arrive(a, link + 1);
        refill();
        if (TRACE) mk_mark(a, ti);
        // P3: attention of one (kv head, split) per CTA
        if (attends) bad |= mk_attention<G, HD>(a, L, kvh, split, t0, t1, pos, epoch, code + 1);      // uniform over the CTA
        if (TRACE) mk_mark(a, ti);
        if (my_head < a.hq) bad |= mk_combine<HD>(a, my_head, active, epoch, code + 2);
        if (TRACE) mk_arrive(a, link + 2);
        __syncthreads();                                      // sm.ws and the products are free
        // P4: INT8 of o, o-projection + residual
        ahead(ph[1], L.wscale[1], li > 0 ? a.xh[0] : nullptr, a.h);
        xs = mk_input<false>(a, a.xo, nullptr, epoch, nullptr, QD, code + 2, bad);
        if (gave_up()) return;
        if (TRACE) mk_mark(a, ti);
        items(ph[1], QD);
        __syncthreads();
        finish(ph[1], xs, true, a.xh[1], nullptr, epoch);
        if (TRACE) mk_arrive(a, link + 3);
        refill();
        if (TRACE) mk_mark(a, ti);
        __syncthreads();
        // P5: post-attention RMSNorm + INT8, gate|up projection with SwiGLU
        ahead(ph[2], L.wscale[2], nullptr, nullptr);
        xs = mk_input<true>(a, a.xh[1], nullptr, epoch, L.ln_post, D, code + 3, bad);
        if (gave_up()) return;
        if (TRACE) mk_mark(a, ti);
        items(ph[2], D);
        __syncthreads();
        for (int g = tid; g < ph[2].count; g += MK_THREADS) {                  // a row group: two gate rows, two up rows
            float v[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) v[r] = scale_acc(total(ph[2], 4 * g + r), xs, sm.ws[4 * g + r]);
            put(a.xact + ph[2].base + g, pack_bf16x2(swiglu_bf16(v[0], v[2]), swiglu_bf16(v[1], v[3])), epoch);
        }
        if (TRACE) mk_arrive(a, link + 4);
        refill();
        if (TRACE) mk_mark(a, ti);
        __syncthreads();
        // P6: INT8 of act, down projection + residual
        ahead(ph[3], L.wscale[3], a.xh[1], nullptr);
        xs = mk_input<false>(a, a.xact, nullptr, epoch, nullptr, F, code + 4, bad);
        if (gave_up()) return;
        if (TRACE) mk_mark(a, ti);
        items(ph[3], F);
        __syncthreads();
        finish(ph[3], xs, true, a.xh[0], li + 1 == a.n_layers ? a.h : nullptr, epoch);
        if (TRACE) mk_arrive(a, link + 5);
        refill();
        __syncthreads();
    }
    // every CTA has read the epoch: the last rows need all of them
    if (blockIdx.x == 0 && tid == 0) a.head[0] = base_epoch + 1 + a.n_layers;
}

// Before a step: after one that gave up, its epochs must not come again.
__global__ void mk_begin_kernel(uint32_t* head) {
    if (head[1] != 0) {
        head[0] += 1u << 16;
        head[1] = 0;
    }
}

// Bytes of the packet buffers, each 16-byte aligned, after 16 bytes of header.
static size_t mk_scratch(int D, int F, int hq, int hk, int d, int nsplit, size_t (&off)[7]) {
    const size_t n[6] = {(size_t)D / 2, (size_t)D / 2, (size_t)(hq + 2 * hk) * d / 2, (size_t)F / 2, (size_t)hq * d / 2, (size_t)hq * nsplit * (d + 2)};
    size_t at = 16;
    for (int i = 0; i < 6; ++i) {
        off[i] = at;
        at += (8 * n[i] + 15) & ~(size_t)15;
    }
    return off[6] = at;
}

}  // namespace scmx

using namespace scmx;

static unsigned long long* g_trace = nullptr;
static int g_n_trace = 0;
extern "C" int scmx_set_decode_trace(unsigned long long* device_buf, int n) {
    g_trace = n > 0 ? device_buf : nullptr;
    g_n_trace = g_trace ? n : 0;
    return SCMX_OK;
}

extern "C" int64_t scmx_decode_step_scratch(int D, int F, int hq, int hk, int d, int nsplit) {
    size_t off[7];
    return D > 0 && F > 0 && hq > 0 && hk > 0 && d > 0 && nsplit > 0 ? (int64_t)mk_scratch(D, F, hq, hk, d, nsplit, off) : 0;
}

extern "C" int scmx_decode_step(const scmx_decode_layer* layers, int n_layers, int D, int F, int hq, int hk, int d, float eps,
                                float scale, const float* inv_freq, const float* rope_table, int64_t rope_rows,
                                int64_t capacity, const int32_t* pos_dev, uint16_t* h, void* scratch, int nsplit, int32_t* status, void* stream) {
    SCMX_REQUIRE(layers && pos_dev && h && scratch && status && inv_freq, SCMX_EINVAL, "decode_step: null buffer");
    SCMX_REQUIRE(n_layers > 0 && hq > 0 && hk > 0 && hq % hk == 0 && hq <= MK_MAXHQ, SCMX_EINVAL, "decode_step: hq=%d hk=%d", hq, hk);
    SCMX_REQUIRE(d == 128, SCMX_ELIMIT, "decode_step: head size %d (128)", d);
    const int G = hq / hk;
    SCMX_REQUIRE(G == 1 || G == 2 || G == 4, SCMX_ELIMIT, "decode_step: %d query heads per key/value head (1, 2 or 4)", G);
    SCMX_REQUIRE(D % 1024 == 0 && F % 1024 == 0 && (hq * d) % 1024 == 0 && D <= MK_MAXK && F <= MK_MAXK && hq * d <= MK_MAXK,
                 SCMX_ELIMIT, "decode_step: widths D=%d F=%d hq*d=%d must be multiples of 1024 up to %d", D, F, hq * d, MK_MAXK);
    SCMX_REQUIRE(capacity >= 1 && nsplit >= 1 && nsplit <= 32, SCMX_EINVAL, "decode_step: capacity=%lld nsplit=%d", (long long)capacity, nsplit);
    SCMX_REQUIRE((reinterpret_cast<uintptr_t>(scratch) & 15) == 0 && (reinterpret_cast<uintptr_t>(h) & 15) == 0, SCMX_EINVAL, "decode_step: unaligned buffer");
    static int coop_dev[64] = {};            // 0 unknown, 1 supported, -1 not: per device
    const int dev = current_device();
    SCMX_REQUIRE(dev >= 0, SCMX_ECUDA, "decode_step: no current CUDA device (ordinal 0..63)");
    constexpr int RINGS = MK_WARPS * MK_SLOTS * MK_CHUNK + 64 * MK_MAXLAYERS;
    if (!coop_dev[dev]) {
        int c = 0;
        SCMX_CUDA_OK(cudaDeviceGetAttribute(&c, cudaDevAttrCooperativeLaunch, dev));
        SCMX_CUDA_OK(cudaFuncSetAttribute(decode_step_kernel<1, 128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, RINGS));
        SCMX_CUDA_OK(cudaFuncSetAttribute(decode_step_kernel<1, 128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RINGS));
        SCMX_CUDA_OK(cudaFuncSetAttribute(decode_step_kernel<2, 128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, RINGS));
        SCMX_CUDA_OK(cudaFuncSetAttribute(decode_step_kernel<2, 128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RINGS));
        SCMX_CUDA_OK(cudaFuncSetAttribute(decode_step_kernel<4, 128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, RINGS));
        SCMX_CUDA_OK(cudaFuncSetAttribute(decode_step_kernel<4, 128, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, RINGS));
        coop_dev[dev] = c ? 1 : -1;
    }
    const int coop = coop_dev[dev] > 0, n_sm = sm_count();
    SCMX_REQUIRE(coop, SCMX_EDEVICE, "decode_step: the device does not support cooperative launches");
    // Every CTA has rows in every phase, which the reuse of the packet buffers rests on, and no more than its tables hold.
    const int qkv = (hq + 2 * hk) * d, most = std::max({qkv, 2 * F, D}) / 4, least = std::min({qkv, 2 * F, D}) / 4;
    SCMX_REQUIRE(hk * nsplit <= n_sm && hq <= n_sm && n_sm <= least && 4 * ((most + n_sm - 1) / n_sm) <= MK_MAXROWS, SCMX_EINVAL,
                 "decode_step: hk * nsplit = %d, hq = %d, phases of %d to %d rows on the %d CTAs of the grid", hk * nsplit, hq, 4 * least, 4 * most, n_sm);
    size_t off[7];
    mk_scratch(D, F, hq, hk, d, nsplit, off);
    uint8_t* sp = static_cast<uint8_t*>(scratch);
    auto at = [&](int i) { return reinterpret_cast<uint2*>(sp + off[i]); };
    MkArgs a;
    a.D = D; a.F = F; a.hq = hq; a.hk = hk; a.nsplit = nsplit; a.eps = eps; a.scale = scale;
    a.inv_freq = inv_freq; a.rope_cs = rope_table; a.rope_rows = rope_table ? rope_rows : 0; a.cap = capacity; a.pos_dev = pos_dev;
    a.h = h; a.head = reinterpret_cast<uint32_t*>(sp); a.xh[0] = at(0); a.xh[1] = at(1); a.xy = at(2); a.xact = at(3); a.xo = at(4); a.xpart = at(5); a.status = status;
    a.wait_ns = g_wait_limit_ns;
    cudaStream_t st = (cudaStream_t)stream;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)n_sm);
    cfg.blockDim = dim3(MK_THREADS);
    cfg.dynamicSmemBytes = RINGS;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    for (int first = 0; first < n_layers; first += MK_MAXLAYERS) {
        a.layers = layers + first; a.first = first; a.n_layers = std::min(n_layers - first, MK_MAXLAYERS);
        const int marks = (g_n_trace & 0xFFFF) - MK_MARKS * first;
        a.trace = g_trace && marks > 0 ? g_trace + MK_MARKS * first : nullptr; a.n_trace = marks;
        a.link = g_n_trace >> 16; a.arrivals = a.link > 0 ? g_trace + (g_n_trace & 0xFFFF) : nullptr;
        mk_begin_kernel<<<1, 1, 0, st>>>(a.head);
        SCMX_LAUNCH_OK("mk_begin_kernel");
        void (*kernel)(MkArgs) = G == 1   ? (g_trace ? decode_step_kernel<1, 128, true> : decode_step_kernel<1, 128, false>)
                                 : G == 2 ? (g_trace ? decode_step_kernel<2, 128, true> : decode_step_kernel<2, 128, false>)
                                          : (g_trace ? decode_step_kernel<4, 128, true> : decode_step_kernel<4, 128, false>);
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, a);
        SCMX_PDL_OK("decode_step_kernel", e);
    }
    return SCMX_OK;
}

// The step on scratch of its own, allocated and given back in the stream's order (a captured graph gets nodes for it).
extern "C" int scmx_decode_step_dense(const scmx_decode_layer* layers, int n_layers, int D, int F, int hq, int hk, int d, float eps,
                                      float scale, const float* inv_freq, const float* rope_table, int64_t rope_rows,
                                      int64_t capacity, const int32_t* pos_dev, uint16_t* h, uint16_t* y, uint16_t* act, uint16_t* o,
                                      float* partials, int nsplit, int32_t* counters, uint32_t* barrier, int32_t* status, void* stream) {
    SCMX_REQUIRE(y && act && o && partials && counters && barrier, SCMX_EINVAL, "decode_step: null buffer");
    const int64_t bytes = scmx_decode_step_scratch(D, F, hq, hk, d, nsplit);
    SCMX_REQUIRE(bytes > 0 && nsplit <= 32, SCMX_EINVAL, "decode_step: D=%d F=%d hq=%d hk=%d d=%d nsplit=%d", D, F, hq, hk, d, nsplit);
    cudaStream_t st = (cudaStream_t)stream;
    void* scratch = nullptr;
    SCMX_CUDA_OK(cudaMallocAsync(&scratch, (size_t)bytes, st));
    const cudaError_t zero = cudaMemsetAsync(scratch, 0, (size_t)bytes, st);
    const int rc = zero != cudaSuccess ? SCMX_OK
                                       : scmx_decode_step(layers, n_layers, D, F, hq, hk, d, eps, scale, inv_freq, rope_table, rope_rows, capacity, pos_dev, h,
                                                          scratch, nsplit, status, stream);
    SCMX_CUDA_OK(cudaFreeAsync(scratch, st));
    SCMX_CUDA_OK(zero);
    return rc;
}
