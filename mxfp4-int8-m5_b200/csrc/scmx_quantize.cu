// SC-MXFP4 quantizer + packer on the GPU, in float64, bit-compatible with the reference's NumPy pipeline
// (sim/mx_int8.py:39-109 via sim/make_testcase.py:26-44 and e2e/sc_format.py:93-111).
//
// One CTA per weight row, one thread per 32-wide block (looping when a row has more blocks than threads):
//   1. e0 = floor(log2 amax) - 2; candidates e0-1 then e0+1 replace the running best only when their squared error
//      is strictly smaller.  The 32 squared errors are summed in the order NumPy's pairwise reduction uses for a
//      contiguous axis of 32 doubles (eight strided partial sums, then a fixed tree) with no fused multiply-adds,
//      so near-ties resolve exactly as in the reference.
//   2. spread constraint: e = max(e, rowmax(e) - 3) (all-zero row: rowmax = 0); E_lo = rowmin(e); shift = e - E_lo.
//   3. E2M1 rounding with exact ties toward the smaller magnitude; nibble = sign << 3 | idx, eight per word;
//      2-bit shifts four per byte; wscale = 2^(E_lo - 1).
#include <limits.h>
#include "scmx_common.cuh"

namespace scmx {

__device__ __forceinline__ int e2m1_idx(double a) {
    // number of midpoints {.25,.75,1.25,1.75,2.5,3.5,5} strictly below a (np.searchsorted side='left')
    return (a > 0.25) + (a > 0.75) + (a > 1.25) + (a > 1.75) + (a > 2.5) + (a > 3.5) + (a > 5.0);
}
__device__ __forceinline__ int e2m1_x2(int idx) { return (int)((0xC8643210u >> (4 * idx)) & 0xFu); }

__device__ __forceinline__ double block_sq_err(const double (&b)[32], int e) {
    const double s = scalbn(1.0, e), si = scalbn(1.0, -e);
    double r[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double x = b[j + 8 * i];
            const double t = __dmul_rn(x, si);
            const double mag = 0.5 * (double)e2m1_x2(e2m1_idx(fabs(t)));
            const double v = t < 0.0 ? -mag : mag;
            const double d = __dsub_rn(__dmul_rn(v, s), x);
            const double sq = __dmul_rn(d, d);
            r[j] = (i == 0) ? sq : __dadd_rn(r[j], sq);
        }
    }
    return __dadd_rn(__dadd_rn(__dadd_rn(r[0], r[1]), __dadd_rn(r[2], r[3])),
                     __dadd_rn(__dadd_rn(r[4], r[5]), __dadd_rn(r[6], r[7])));
}

template <typename T> __device__ __forceinline__ double to_f64(T v);
template <> __device__ __forceinline__ double to_f64<float>(float v) { return (double)v; }
template <> __device__ __forceinline__ double to_f64<double>(double v) { return v; }
template <> __device__ __forceinline__ double to_f64<uint16_t>(uint16_t v) { return (double)bf16_to_f32(v); }

__device__ __forceinline__ int block_reduce_int(int v, int* red, bool take_max) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const int t = __shfl_xor_sync(0xffffffffu, v, o);
        v = take_max ? max(v, t) : min(v, t);
    }
    __syncthreads();
    if (lane == 0) red[w] = v;
    __syncthreads();
    if (w == 0) {
        int t = lane < nw ? red[lane] : (take_max ? INT_MIN : INT_MAX);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const int u = __shfl_xor_sync(0xffffffffu, t, o);
            t = take_max ? max(t, u) : min(t, u);
        }
        if (lane == 0) red[32] = t;
    }
    __syncthreads();
    return red[32];
}

template <typename T>
__global__ void __launch_bounds__(256) quantize_kernel(const T* __restrict__ w, int K, uint32_t* __restrict__ codes,
                                                       uint8_t* __restrict__ bcodes, float* __restrict__ wscale,
                                                       int8_t* __restrict__ qw, int32_t* __restrict__ row_exp) {
    extern __shared__ int s_e[];          // per-block exponent of this row (INT_MIN = all-zero block)
    __shared__ int red[33];
    const int64_t n = blockIdx.x;
    const int nb = K / 32;
    const T* wr = w + n * (int64_t)K;

    int hi = INT_MIN;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        double v[32];
        double amax = 0.0;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            v[i] = to_f64<T>(wr[b * 32 + i]);
            amax = fmax(amax, fabs(v[i]));
        }
        int e;
        if (amax == 0.0) {
            e = INT_MIN;
        } else {
            const int e0 = ilogb(amax) - 2;
            int best = e0;
            double err = block_sq_err(v, e0);
            const double em = block_sq_err(v, e0 - 1);
            if (em < err) { best = e0 - 1; err = em; }
            const double ep = block_sq_err(v, e0 + 1);
            if (ep < err) { best = e0 + 1; err = ep; }
            e = best;
        }
        s_e[b] = e;
        hi = max(hi, e);
    }
    hi = block_reduce_int(hi, red, true);
    if (hi == INT_MIN) hi = 0;            // all-zero row
    const int lo_c = hi - 3;
    int lo = INT_MAX;
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        const int e = max(s_e[b], lo_c);
        s_e[b] = e;
        lo = min(lo, e);
    }
    lo = block_reduce_int(lo, red, false);   // E_lo (also syncs s_e)
    if (threadIdx.x == 0) {
        wscale[n] = (float)scalbn(1.0, lo - 1);
        if (row_exp) row_exp[n] = lo;
    }
    for (int b = threadIdx.x; b < nb; b += blockDim.x) {
        const int e = s_e[b];
        const int shift = e - lo;
        const double si = scalbn(1.0, -e);
        uint32_t words[4];
        uint32_t qwords[8];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            uint32_t word = 0;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const double t = __dmul_rn(to_f64<T>(wr[b * 32 + 8 * j + i]), si);
                const int idx = e2m1_idx(fabs(t));
                const int neg = (t < 0.0) && idx > 0;
                word |= (uint32_t)(idx | (neg << 3)) << (4 * i);
                const int q = e2m1_x2(idx) << shift;
                const uint32_t qb = (uint32_t)(neg ? -q : q) & 0xFFu;
                if (i < 4) qwords[2 * j] = (i == 0 ? 0u : qwords[2 * j]) | (qb << (8 * i));
                else qwords[2 * j + 1] = (i == 4 ? 0u : qwords[2 * j + 1]) | (qb << (8 * (i - 4)));
            }
            words[j] = word;
        }
        reinterpret_cast<uint4*>(codes + n * (int64_t)(K / 8))[b] = make_uint4(words[0], words[1], words[2], words[3]);
        if (qw) {
            uint4* q4 = reinterpret_cast<uint4*>(qw + n * (int64_t)K + b * 32);
            q4[0] = make_uint4(qwords[0], qwords[1], qwords[2], qwords[3]);
            q4[1] = make_uint4(qwords[4], qwords[5], qwords[6], qwords[7]);
        }
        if ((b & 3) == 0) {
            const uint32_t byte = (uint32_t)(s_e[b] - lo) | ((uint32_t)(s_e[b + 1] - lo) << 2) |
                                  ((uint32_t)(s_e[b + 2] - lo) << 4) | ((uint32_t)(s_e[b + 3] - lo) << 6);
            bcodes[n * (int64_t)(nb / 4) + b / 4] = (uint8_t)byte;
        }
    }
}

// The same for float32 and bfloat16 rows on 16-byte boundaries, four lanes per block of 32 and eight elements per lane, so that loads,
// codes and INT8 values are coalesced and a row of up to 8192 elements stays in registers while the next one is on its way.  The
// squared errors of the candidates are taken in float32, where the scaled values and their distances to the grid are exact, so a sum is
// off by at most 10 roundings of 2^-24; only where two sums are closer than that (one block in 7000 of bfloat16 normal values) or the
// exponent leaves float32's range is the block decided in float64 as above, by the whole warp, so the packed bits are the same.
// Bound by instructions (against 6.6 us for the bytes), where the float64 form was bound by its compares and conversions.  Products and sums are taken two at
// a time; min, max and masks have no such form.  6144 x 2048 bfloat16 (44 MB in and out): 26.6 us (28.7 singly) against 107 us; with the float64 decision made by one lane 43 us, the
// codes by seven compares instead of the conversion instruction 50 us.
constexpr float QUANT_CLEAR = 4e-6f;      // relative distance of two float32 sums from which their order is certain (10 x 2^-24 each)
constexpr float QUANT_LEAST = 1e-30f;     // and that of two sums so small that squares may have lost bits below float32's range
constexpr int QUANT_EXP = 120;            // scales 2^-e and 2^e stay normal float32 numbers

// The float64 decision for the block at p by a whole warp, an element per lane; the sums in block_sq_err's order.
template <typename T>
__device__ __noinline__ int block_exponent_f64(const T* p) {
    const double x = to_f64<T>(p[threadIdx.x & 31]);
    double amax = fmax(0.0, fabs(x));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) amax = fmax(amax, __shfl_xor_sync(0xffffffffu, amax, o));
    if (amax == 0.0) return INT_MIN;
    const int e0 = ilogb(amax) - 2;
    double sum[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int e = e0 + (c == 1 ? -1 : c == 2 ? 1 : 0);
        const double s = scalbn(1.0, e), t = __dmul_rn(x, scalbn(1.0, -e));
        const double mag = 0.5 * (double)e2m1_x2(e2m1_idx(fabs(t)));
        const double d = __dsub_rn(__dmul_rn(t < 0.0 ? -mag : mag, s), x), sq = __dmul_rn(d, d);
        double r = sq;                        // lanes 0 .. 7: the strided partial sums
#pragma unroll
        for (int i = 8; i < 32; i += 8) r = __dadd_rn(r, __shfl_sync(0xffffffffu, sq, (threadIdx.x + i) & 31));
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) r = __dadd_rn(r, __shfl_xor_sync(0xffffffffu, r, o));
        sum[c] = __shfl_sync(0xffffffffu, r, 0);
    }
    int best = e0;
    double err = sum[0];
    if (sum[1] < err) { best = e0 - 1; err = sum[1]; }
    if (sum[2] < err) best = e0 + 1;
    return best;
}

// Packed float32 pairs: one instruction for two products or sums (min, max and masks stay single).
__device__ __forceinline__ uint64_t q_pack(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 q_unpack(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t q_mul(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ uint64_t q_fma(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Sum of the squared distances of the eight a = |t| (in pairs) times `scale` to the nearest E2M1 value: adding 2^22 times the power of two below
// max(a, 1) rounds to the grid's step there (which of two equally near values is taken does not matter here).  NaN gives NaN.
template <bool SATURATES>
__device__ __forceinline__ float grid_sq_err(const uint64_t (&t)[4], float scale) {
    const uint64_t big = q_pack(4194304.0f, 4194304.0f), small = q_pack(-4194304.0f, -4194304.0f), neg = q_pack(-1.0f, -1.0f), sc = q_pack(scale, scale);
    uint64_t s = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint64_t a = scale == 1.0f ? t[i] : q_mul(t[i], sc);
        const float2 v = q_unpack(a);
        const uint64_t p = q_pack(__int_as_float(__float_as_int(fmaxf(v.x, 1.0f)) & 0x7F800000), __int_as_float(__float_as_int(fmaxf(v.y, 1.0f)) & 0x7F800000));
        uint64_t r = q_fma(p, small, q_fma(p, big, a));
        if (SATURATES) {
            const float2 u = q_unpack(r);
            r = q_pack(fminf(u.x, 6.0f), fminf(u.y, 6.0f));
        }
        const uint64_t d = q_fma(a, neg, r);
        s = q_fma(d, d, s);
    }
    const float2 two = q_unpack(s);
    float e = two.x + two.y;
    e += __shfl_xor_sync(0xffffffffu, e, 1);
    e += __shfl_xor_sync(0xffffffffu, e, 2);
    return e;
}

// Eight codes of t = x si, si = 1 / 2^e.  The conversion instruction takes ties to the even code; here they go to the smaller magnitude, so a value
// whose low 16 bits are zero, which a tie is, first loses one unit in its last place (that reaches no other tie).  A negative value that
// becomes zero has no sign.
template <typename T>
__device__ __forceinline__ uint32_t e2m1_codes(const float (&x)[8], float si) {
    float u[8];
    if (sizeof(T) == 2) {                     // of a bfloat16 value the low 16 bits are always zero
        const uint64_t below = q_pack(si * 0.99999994f, si * 0.99999994f);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 v = q_unpack(q_mul(q_pack(x[2 * i], x[2 * i + 1]), below));
            u[2 * i] = v.x;
            u[2 * i + 1] = v.y;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float t = x[i] * si;
            u[i] = t * ((__float_as_uint(t) & 0xFFFFu) ? 1.0f : 0.99999994f);
        }
    }
    uint32_t w;
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b0, %2, %1;\n\tcvt.rn.satfinite.e2m1x2.f32 b1, %4, %3;\n\t"
        "cvt.rn.satfinite.e2m1x2.f32 b2, %6, %5;\n\tcvt.rn.satfinite.e2m1x2.f32 b3, %8, %7;\n\t"
        "mov.b32 %0, {b0, b1, b2, b3};\n\t}"
        : "=r"(w) : "f"(u[0]), "f"(u[1]), "f"(u[2]), "f"(u[3]), "f"(u[4]), "f"(u[5]), "f"(u[6]), "f"(u[7]));
    const uint32_t nz = ((w << 3) | (w << 2) | (w << 1)) & 0x88888888u;
    return w & (nz | 0x77777777u);
}

template <typename T> struct QuantRaw;      // eight elements as loaded
template <> struct QuantRaw<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p) {
        a = reinterpret_cast<const float4*>(p)[0];
        b = reinterpret_cast<const float4*>(p)[1];
    }
    __device__ __forceinline__ void zero() { a = b = make_float4(0, 0, 0, 0); }
    __device__ __forceinline__ void widen(float (&x)[8]) const {
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
    }
};
template <> struct QuantRaw<uint16_t> {
    uint4 w;
    __device__ __forceinline__ void load(const uint16_t* p) { w = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ void zero() { w = make_uint4(0, 0, 0, 0); }
    __device__ __forceinline__ void widen(float (&x)[8]) const {
        x[0] = bf16_lo(w.x); x[1] = bf16_hi(w.x); x[2] = bf16_lo(w.y); x[3] = bf16_hi(w.y);
        x[4] = bf16_lo(w.z); x[5] = bf16_hi(w.z); x[6] = bf16_lo(w.w); x[7] = bf16_hi(w.w);
    }
};

// Exponent of the block that this lane and its three neighbours hold, INT_MIN for a block of zeros; p: the warp's first element.
template <typename T>
__device__ __forceinline__ int block_exponent(const float (&x)[8], const T* p) {
    const int lane = threadIdx.x & 31;
    float amax = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; ++i) amax = fmaxf(amax, fabsf(x[i]));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
    amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
    const int e0 = (__float_as_int(amax) >> 23) - 127 - 2;       // of a normal number; others leave the range below
    const float si = __int_as_float((127 - min(max(e0, -QUANT_EXP), QUANT_EXP)) << 23);
    uint64_t t[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) t[i] = q_mul(q_pack(fabsf(x[2 * i]), fabsf(x[2 * i + 1])), q_pack(si, si));
    float err = grid_sq_err<true>(t, 1.0f);
    const float em = 0.25f * grid_sq_err<true>(t, 2.0f), ep = 4.0f * grid_sq_err<false>(t, 0.5f);
    auto clear = [](float a, float b) { return fabsf(a - b) > fmaxf(QUANT_CLEAR * fmaxf(a, b), QUANT_LEAST); };
    bool sure = clear(em, err);
    int e = e0;
    if (em < err) { e = e0 - 1; err = em; }
    sure = sure && clear(ep, err);
    if (ep < err) e = e0 + 1;
    sure = sure && e0 >= -QUANT_EXP && e0 <= QUANT_EXP;
    if (amax == 0.0f) e = INT_MIN;
    for (unsigned unsure = __ballot_sync(0xffffffffu, !sure && amax != 0.0f); unsure != 0;) {      // the same in every lane
        const int g = (__ffs(unsure) - 1) & ~3, decided = block_exponent_f64<T>(p + 8 * g);
        if ((lane & ~3) == g) e = decided;
        unsure &= ~(0xFu << g);
    }
    return e;
}

// Largest of `hi` and smallest of `low` over the CTA.
__device__ __forceinline__ void block_range(int& hi, int& low, int (&red)[2][32]) {
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    hi = __reduce_max_sync(0xffffffffu, hi);
    low = __reduce_min_sync(0xffffffffu, low);
    if (lane == 0) {
        red[0][threadIdx.x >> 5] = hi;
        red[1][threadIdx.x >> 5] = low;
    }
    __syncthreads();
    hi = __reduce_max_sync(0xffffffffu, lane < nw ? red[0][lane] : INT_MIN);
    low = __reduce_min_sync(0xffffffffu, lane < nw ? red[1][lane] : INT_MAX);
}

struct QuantOut {
    uint32_t* codes;
    uint8_t* bcodes;
    int8_t* qw;
};

// Codes of vector v of row n, whose block has exponent max(e, lo_c); the row's smallest exponent is lo.  Run by every lane of a warp.
template <typename T>
__device__ __forceinline__ void write_codes(const float (&x)[8], int e, int lo_c, int lo, int64_t n, int K, int v, const QuantOut& o) {
    const int nv = K / 8, eb = max(e, lo_c), shift = eb - lo;
    const bool in = v < nv;
    uint32_t word = 0, q[2] = {0, 0};
    const float sum = ((x[0] + x[1]) + (x[2] + x[3])) + ((x[4] + x[5]) + (x[6] + x[7]));      // finite: no element is NaN
    if (eb >= -QUANT_EXP && eb <= QUANT_EXP && fabsf(sum) < INFINITY) {
        const float si = __int_as_float((127 - eb) << 23);
        word = e2m1_codes<T>(x, si);
        if (o.qw) {
            const uint32_t plo = 0x03020100u << shift, phi = 0x0C080604u << shift;
            decode_word(word, plo, phi, lut_negate(plo), lut_negate(phi), q[0], q[1]);
        }
    } else {
        const double si = scalbn(1.0, -eb);
#pragma unroll 1
        for (int i = 0; i < 8; ++i) {
            float xi = 0.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) xi = j == i ? x[j] : xi;
            const double t = __dmul_rn((double)xi, si);
            const int idx = e2m1_idx(fabs(t));
            const int neg = t < 0.0 && idx > 0, m = e2m1_x2(idx) << shift;
            word |= (uint32_t)(idx | (neg << 3)) << (4 * i);
            const uint32_t qb = ((uint32_t)(neg ? -m : m) & 0xFFu) << (8 * (i & 3));
            if (i < 4) q[0] |= qb;
            else q[1] |= qb;
        }
    }
    uint32_t byte = in ? (uint32_t)shift << (2 * ((v >> 2) & 3)) : 0u;      // four blocks, 16 lanes, per byte
    byte |= __shfl_xor_sync(0xffffffffu, byte, 4);
    byte |= __shfl_xor_sync(0xffffffffu, byte, 8);
    if (!in) return;
    o.codes[n * nv + v] = word;
    if (o.qw) *reinterpret_cast<uint2*>(o.qw + n * K + 8 * (int64_t)v) = make_uint2(q[0], q[1]);
    if ((v & 15) == 0) o.bcodes[n * (K / 128) + (v >> 4)] = (uint8_t)byte;
}

__device__ __forceinline__ void write_row(int64_t n, int lo, float* wscale, int32_t* row_exp) {
    wscale[n] = (float)scalbn(1.0, lo - 1);
    if (row_exp) row_exp[n] = lo;
}

// Rows of at most eight elements per thread: a CTA takes row after row, the next one's elements on their way.
template <typename T>
__global__ void __launch_bounds__(1024) quantize_vec_kernel(const T* __restrict__ w, int64_t N, int K, const QuantOut out,
                                                            float* __restrict__ wscale, int32_t* __restrict__ row_exp) {
    __shared__ int red[2][2][32];
    const int tid = threadIdx.x;
    const bool in = tid < K / 8;
    QuantRaw<T> raw;
    raw.zero();
    if (in) raw.load(w + (int64_t)blockIdx.x * K + 8 * tid);
    int turn = 0;
    for (int64_t n = blockIdx.x; n < N; n += gridDim.x, turn ^= 1) {
        float x[8];
        raw.widen(x);
        if (in && n + gridDim.x < N) raw.load(w + (n + gridDim.x) * K + 8 * tid);
        const int e = block_exponent<T>(x, w + n * K + 8 * (tid & ~31));
        int hi = e, low = in ? e : INT_MAX;
        block_range(hi, low, red[turn]);      // the other buffer is read until every thread is past this barrier
        if (hi == INT_MIN) hi = 0;            // all-zero row
        const int lo_c = hi - 3, lo = max(low, lo_c);      // min over blocks of max(e, lo_c)
        if (tid == 0) write_row(n, lo, wscale, row_exp);
        write_codes<T>(x, e, lo_c, lo, n, K, tid, out);
    }
}

// Longer rows: the exponents wait in shared memory and the elements are read again.
template <typename T>
__global__ void __launch_bounds__(1024) quantize_long_kernel(const T* __restrict__ w, int64_t N, int K, const QuantOut out,
                                                             float* __restrict__ wscale, int32_t* __restrict__ row_exp) {
    extern __shared__ int s_e[];          // [K / 32]
    __shared__ int red[2][32];
    const int64_t n = blockIdx.x;
    const int tid = threadIdx.x, nv = K / 8;
    const T* wr = w + n * K;
    int hi = INT_MIN, low = INT_MAX;
    float x[8];
    QuantRaw<T> raw;
    for (int v = tid; v - tid < nv; v += 1024) {
        raw.zero();
        if (v < nv) raw.load(wr + 8 * (int64_t)v);
        raw.widen(x);
        const int e = block_exponent<T>(x, wr + 8 * (int64_t)(v & ~31));
        if (v >= nv) break;                   // the last pass: no shuffles follow
        hi = max(hi, e);
        low = min(low, e);
        if ((v & 3) == 0) s_e[v >> 2] = e;
    }
    block_range(hi, low, red);
    if (hi == INT_MIN) hi = 0;
    const int lo_c = hi - 3, lo = max(low, lo_c);
    if (tid == 0) write_row(n, lo, wscale, row_exp);
    for (int v = tid; v - tid < nv; v += 1024) {
        raw.zero();
        if (v < nv) raw.load(wr + 8 * (int64_t)v);
        raw.widen(x);
        write_codes<T>(x, v < nv ? s_e[v >> 2] : INT_MIN, lo_c, lo, n, K, v, out);
    }
}

template <typename T>
static int run_quantize_vec(const T* w, int64_t N, int K, const QuantOut& out, float* wscale, int32_t* row_exp, cudaStream_t st) {
    const int nv = K / 8;
    if (nv <= 1024) {
        const int threads = (nv + 31) / 32 * 32;
        int64_t grid = (int64_t)sm_count() * (threads < 64 ? 16 : 1024 / threads);      // 64 registers a thread: 1024 threads an SM
        if (grid > N) grid = N;
        quantize_vec_kernel<T><<<(unsigned)grid, threads, 0, st>>>(w, N, K, out, wscale, row_exp);
    } else {
        const size_t smem = (size_t)(K / 32) * sizeof(int);
        if (smem > 40 * 1024) SCMX_CUDA_OK(cudaFuncSetAttribute(quantize_long_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        quantize_long_kernel<T><<<(unsigned)N, 1024, smem, st>>>(w, N, K, out, wscale, row_exp);
    }
    SCMX_LAUNCH_OK("quantize_vec_kernel");
    return SCMX_OK;
}

}  // namespace scmx

using namespace scmx;

extern "C" int scmx_quantize_sc_mxfp4(const void* w, int w_dtype, int64_t N, int64_t K, uint32_t* codes, uint8_t* bcodes,
                                      float* wscale, int8_t* qw, int32_t* row_exp, void* stream) {
    SCMX_REQUIRE(N >= 0 && K > 0 && K % 128 == 0 && K <= (1 << 20), SCMX_EINVAL,
                 "quantize_sc_mxfp4: K=%lld must be a positive multiple of 128", (long long)K);
    SCMX_REQUIRE(w_dtype >= 0 && w_dtype <= 2, SCMX_EINVAL, "quantize_sc_mxfp4: w_dtype=%d (0 f32, 1 f64, 2 bf16)", w_dtype);
    SCMX_REQUIRE((reinterpret_cast<uintptr_t>(codes) & 15) == 0 && (!qw || (reinterpret_cast<uintptr_t>(qw) & 15) == 0),
                 SCMX_EINVAL, "quantize_sc_mxfp4: codes and qw must be 16-byte aligned");
    if (N == 0) return SCMX_OK;
    const int nb = (int)(K / 32);
    int threads = nb < 256 ? ((nb + 31) / 32) * 32 : 256;
    const size_t smem = (size_t)nb * sizeof(int);
    cudaStream_t st = (cudaStream_t)stream;
    if (w_dtype != 1 && ((uintptr_t)w & 15) == 0)      // every row starts on 16 bytes: K is a multiple of 128
        return w_dtype == 0 ? run_quantize_vec((const float*)w, N, (int)K, QuantOut{codes, bcodes, qw}, wscale, row_exp, st)
                            : run_quantize_vec((const uint16_t*)w, N, (int)K, QuantOut{codes, bcodes, qw}, wscale, row_exp, st);
    if (w_dtype == 0)
        quantize_kernel<float><<<(unsigned)N, threads, smem, st>>>((const float*)w, (int)K, codes, bcodes, wscale, qw, row_exp);
    else if (w_dtype == 1)
        quantize_kernel<double><<<(unsigned)N, threads, smem, st>>>((const double*)w, (int)K, codes, bcodes, wscale, qw, row_exp);
    else
        quantize_kernel<uint16_t><<<(unsigned)N, threads, smem, st>>>((const uint16_t*)w, (int)K, codes, bcodes, wscale, qw, row_exp);
    SCMX_LAUNCH_OK("quantize_kernel");
    return SCMX_OK;
}
