// epilogue.cuh -- the fused r^2 epilogue of the tensor-core kernels, applied
// to 32 accumulator columns (B rows) at a time as they leave TMEM.
//
// qLD's get_pairwise_ld_score (src/correlator/src/gemm_cpu.c:343-404):
// r^2 = 0 when a bit count is 0, values > 1.0001 become 123.456, 0/0 stays
// NaN.  Two evaluations (template MODE):
//   R2_EXACT      D = S*c - cA*cB is formed exactly in FP64 (every term is an
//                 integer below 2^53: the count enters FP64 through the 2^52
//                 bias trick and D is one fused multiply-add), then
//                 r^2 = (D*D) * (1/varA * 1/varB) with one rounding to FP32.
//                 No 64-bit integer arithmetic and one conversion per pair.
//   R2_REFERENCE  the reference's float/double operation sequence
//                 (qld_device.cuh: r2_reference), bit for bit, evaluated
//                 branch-free in FP32 (r2_reference_ff) with a rare
//                 fallback to the literal sequence.
// Per-column factors live in shared memory (filled once per tile); the
// per-row (A) factors in registers.
#pragma once

#include "qld_device.cuh"

namespace qld {
namespace epi {

// ------------------------------------------------- two columns at a time --
//
// Packed pairs of floats (Blackwell's f32x2 instructions): each half is
// rounded as the scalar instruction rounds it, one issue slot for both.
// The epilogue shares its SM's issue slots and shared-memory port with the
// unpack, and for tables of up to ~10,000 samples it, not the MMAs, sets a
// tile's time; in pairs of columns it takes half the arithmetic instructions
// and half the column-factor loads.  Exact mode, with the next tile's factors
// prefetched (ld_mxf4_pair.cu): band of 1,000 over 50,000 x 10,001 234 -> 199
// us, single region 2.12 -> 2.07 ms, 300-task batch 576 -> 566 us.
typedef unsigned long long f2;

__device__ __forceinline__ f2 pack2(float a, float b) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f2 splat2(float a) { return pack2(a, a); }
__device__ __forceinline__ void unpack2(f2 x, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x));
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 add2(f2 a, f2 b) {
    f2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// ------------------------------------------- R2_REFERENCE column factors --
//
// One float4 per column (and per A row, in registers): x = v = fl32(c/S) as
// the reference computes it; y + z = 1/(v(1-v)) as an unevaluated pair of
// floats (y = RN32 of the FP64 value, z = RN32 of the remainder: ~2^-48
// relative); w = RN32(1/v).  A zero row (c = 0) is all zeros, so every pair
// with it evaluates to 0 -- the reference's rule for an empty SNP -- without
// a test.  A row with v >= 1 (c = S, or a bit count above S) carries a NaN
// in y, which sends every pair with it to the literal sequence.
struct ColsR {
    static constexpr bool PAIRS = false;
    float4 *f;
    __device__ __forceinline__ ColsR(uint8_t *base, int) : f(reinterpret_cast<float4 *>(base)) {}
    __device__ __forceinline__ float4 col(int bl) const { return f[bl]; }
    __device__ __forceinline__ void put(int bl, float4 k) const { f[bl] = k; }
};
constexpr int COLR_BYTES = 16;

// The same factors by column pairs, each of the four as an f2: x, y, z, w.
struct ColsR2 {
    static constexpr bool PAIRS = true;
    float *f;
    __device__ __forceinline__ ColsR2(uint8_t *base, int) : f(reinterpret_cast<float *>(base)) {}
    __device__ __forceinline__ float4 col(int bl) const {
        const float *p = f + (bl >> 1) * 8 + (bl & 1);
        return make_float4(p[0], p[2], p[4], p[6]);
    }
    __device__ __forceinline__ void put(int bl, float4 k) const {
        float *p = f + (bl >> 1) * 8 + (bl & 1);
        p[0] = k.x;
        p[2] = k.y;
        p[4] = k.z;
        p[6] = k.w;
    }
    __device__ __forceinline__ void pair(int bl, f2 &x, f2 &y, f2 &z, f2 &w) const {   // bl even
        const ulonglong2 a = *reinterpret_cast<const ulonglong2 *>(f + bl * 4);
        const ulonglong2 b = *reinterpret_cast<const ulonglong2 *>(f + bl * 4 + 4);
        x = a.x;
        y = a.y;
        z = b.x;
        w = b.y;
    }
};

__device__ __forceinline__ float4 ref_factors(uint32_t c, int S) {
    if (c == 0u) return make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    const float v = __fdiv_rn((float)c, (float)S);
    if (!(v < 1.0f)) return make_float4(v, __uint_as_float(0x7FC00000u), 0.0f, 1.0f);
    const double om = __dsub_rn(1.0, (double)v);
    const double i = __ddiv_rn(1.0, __dmul_rn((double)v, om));
    const float hi = __double2float_rn(i);
    return make_float4(v, hi, __double2float_rn(__dsub_rn(i, (double)hi)), __frcp_rn(v));
}

// Returns whether the column has a NaN factor (v >= 1).
template <class C>
__device__ __forceinline__ bool store_col_ref(const C &f, int bl, uint32_t c, int S) {
    const float4 k = ref_factors(c, S);
    f.put(bl, k);
    return k.y != k.y;
}

// Per-thread A-row factors of the reference mode.
struct ARowR {
    float4 k;           // ref_factors of the row
    uint32_t c;
    float Sf, rSf;      // (float)S and its correctly rounded reciprocal
};

__device__ __forceinline__ ARowR make_arow_ref(uint32_t c, int S) {
    ARowR r;
    r.k = ref_factors(c, S);
    r.c = c;
    r.Sf = (float)S;
    r.rSf = __frcp_rn(r.Sf);
    return r;
}

// Columns t of a chunk (B rows b0 + t, t < CW <= 32) that A row a owes: inside
// the task (b < n) and the diagonal window dlo <= a - b <= dhi, as a bit mask.
template <int CW>
__device__ __forceinline__ uint32_t column_mask(int b0, int a, bool a_ok, int n, int dlo,
                                                int dhi) {
    int lo = 0, hi = n - b0 < CW ? n - b0 : CW;
    if (dlo > -2147483647 - 1 && a - b0 - dlo + 1 < hi) hi = a - b0 - dlo + 1;
    if (dhi < 2147483647 && a - b0 - dhi > 0) lo = a - b0 - dhi;
    if (!a_ok || lo >= hi) return 0u;
    return (0xFFFFFFFFu >> (32 - hi)) & (0xFFFFFFFFu << lo);
}

// *p = x if cond, as a predicated store: no branch, so the arithmetic around
// it is scheduled across it.
__device__ __forceinline__ void store_if(uint32_t *p, uint32_t x, bool cond) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.u32 q, %2, 0;\n\t"
        "@q st.global.u32 [%0], %1;\n\t}" ::"l"(p),
        "r"(x), "r"((uint32_t)cond));
}

// Shared-memory column factors of one tile for the integer-count kernels:
// BN entries each of d0 = 1/(c(S-c)) and d1 = c as double (R2_EXACT), or one
// ColsR float4 at the same address (R2_REFERENCE).  24 bytes per column.
struct Cols {
    uint8_t *base;
    double *d0, *d1;
    __device__ __forceinline__ Cols(uint8_t *b, int bn)
        : base(b), d0(reinterpret_cast<double *>(b)), d1(reinterpret_cast<double *>(b) + bn) {}
};
constexpr int COL_BYTES = 24;

template <int MODE>
__device__ __forceinline__ void store_col(const Cols &f, int bl, uint32_t c, int S) {
    if (MODE == R2_EXACT) {
        f.d0[bl] = row_exact(c, S).inv_var;
        f.d1[bl] = (double)c;
    } else {
        store_col_ref(ColsR(f.base, 0), bl, c, S);
    }
}

// Per-thread A-row factors.
struct ARow {
    uint32_t c;
    double inv, cd;     // exact
    ARowR rr;           // reference
};

template <int MODE>
__device__ __forceinline__ ARow make_arow(uint32_t c, int S) {
    ARow r;
    r.c = c;
    if (MODE == R2_EXACT) {
        r.inv = row_exact(c, S).inv_var;
        r.cd = (double)c;
    } else {
        r.rr = make_arow_ref(c, S);
    }
    return r;
}

__device__ __forceinline__ double u32_to_f64(uint32_t x) {
    // 2^52 + x has the integer x in its low mantissa bits; subtracting 2^52 is exact.
    return __hiloint2double(0x43300000, (int)x) - 4503599627370496.0;
}

// R2_EXACT from an integer count, in FP64.
__device__ __forceinline__ float pair_r2_exact(uint32_t cnt, const ARow &ra, const Cols &f,
                                               int bl, double S_d) {
    const double cbd = f.d1[bl];
    const double D = fma(S_d, u32_to_f64(cnt), -(ra.cd * cbd));
    const double r = (D * D) * (ra.inv * f.d0[bl]);
    if (ra.c == 0u || cbd == 0.0) return 0.0f;
    if (r > 1.0001) return 123.456f;
    return __double2float_rn(r);
}

// ------------------------------------------- R2_REFERENCE without branches --
//
// The reference's operation sequence (r2_reference) gives, per pair,
// fl32(RN64(x / den)) with x = fl32(d*d), d = fl32(v3 - p12),
// v3 = fl32(cab/S), p12 = fl32(vA*vB) and den = RN64(RN64(p12*(1-vA))*(1-vB)).
// r2_reference_ff evaluates it in FP32 alone (no FP64 instruction, no
// conversion, no MUFU), branch-free:
//  * v3 by Markstein's FMA correction: q = RN(cab * y) with y = RN(1/S),
//    then RN(q + (cab - q*S) * y), the residual exact in one FMA; with y the
//    correctly rounded reciprocal this is the correctly rounded quotient
//    (P. Markstein, IBM J. Res. Dev. 34(1), 1990); cab and S are integers
//    <= 2^24, exact in FP32.  p12, d and x as in the reference (__f*_rn: no
//    contraction).
//  * 1/den to ~2^-45: with e = vA*vB - p12 exact (the FMA TwoProduct),
//    p12*(1-vA)*(1-vB) = vA(1-vA) * vB(1-vB) * (1 - e/(vA vB)), so
//    1/den = IA * IB * (1 + t) up to 2^-48, where IA = 1/(vA(1-vA)) and IB
//    are the rows' float pairs (y + z) and t = e * (1/vA) * (1/vB); the
//    reference's two FP64 roundings of den move it by at most 2^-52.
//    q = x * IA * IB * (1 + t) is formed as an unevaluated float pair
//    (qh, ql) with FMA products (Dekker / Ogita-Rump-Oishi style error-free
//    transformations).
//  * The rounding test: RN32(qh + ql +- 2^-40 qh) are equal when no FP32
//    rounding midpoint lies within 2^-40 of the quotient, far beyond the
//    evaluation error, and then RN32(qh + ql) = fl32(RN64(x / den)).
//    Pairs failing it (~1e-5 at realistic S; more at S <= 100, whose simple
//    fractions meet midpoints more often), with a row whose v >= 1 (NaN
//    factors), or with 0 < x < 2^-100 (a subnormal-range quotient) are
//    flagged and recomputed by r2_flagged: a fixed SNP (v = 1) from x alone,
//    the rest with r2_reference.
//  * (double)r > 1.0001 is r > 1 + 838 * 2^-23, the largest float not above
//    1.0001.
// Exact zeros need no test: a zero row's factors are 0, so q = 0.
// The earlier FP64 form (Newton reciprocal of den from rcp.approx.f64 with a
// rounding test in FP64) spent its time in FP64 conversions and the MUFU.
// fl32(cab / S) for integer cab <= S <= 2^24 (exact in FP32), by Markstein's
// correction of RN(cab * RN(1/S)): the correctly rounded quotient.
__device__ __forceinline__ float ref_quotient_ff(float cab, const ARowR &A) {
    const float q0 = __fmul_rn(cab, A.rSf);
    return __fmaf_rn(__fmaf_rn(-q0, A.Sf, cab), A.rSf, q0);
}

__device__ __forceinline__ float r2_reference_ff(float cab, const ARowR &A, float4 B,
                                                 bool &redo) {
    const float v3 = ref_quotient_ff(cab, A);
    const float p12 = __fmul_rn(A.k.x, B.x);
    const float e = __fmaf_rn(A.k.x, B.x, -p12);
    const float d = __fsub_rn(v3, p12);
    const float x = __fmul_rn(d, d);
    const float Ph = __fmul_rn(A.k.y, B.y);
    float Pl = __fmaf_rn(A.k.y, B.y, -Ph);
    Pl = __fmaf_rn(A.k.y, B.z, Pl);
    Pl = __fmaf_rn(A.k.z, B.y, Pl);
    const float t = __fmul_rn(e, __fmul_rn(A.k.w, B.w));
    const float qh = __fmul_rn(x, Ph);
    float ql = __fmaf_rn(x, Ph, -qh);
    ql = __fmaf_rn(x, Pl, ql);
    ql = __fmaf_rn(qh, t, ql);
    const float rh = __fadd_rn(qh, __fmaf_rn(qh, 0x1p-40f, ql));
    const float rl = __fadd_rn(qh, __fmaf_rn(qh, -0x1p-40f, ql));
    const bool tiny = __float_as_uint(x) - 1u < __float_as_uint(0x1p-100f) - 1u;
    redo = !(rh == rl) || tiny;
    return rh > __uint_as_float(0x3F800000u + 838u) ? 123.456f : rh;
}

// r2_reference_ff for two columns (f2 halves): the same operations with the
// same roundings, a subtraction x - y written as an addition of -y computed
// as (-a) * b.  Leaves q (before the > 1.0001 rule) and x, and sets a flag
// per half as r2_reference_ff's `redo`.
struct ARowR2 {
    f2 rS, nS, v, nv, y, ny, z, w;
    __device__ __forceinline__ explicit ARowR2(const ARowR &a)
        : rS(splat2(a.rSf)), nS(splat2(-a.Sf)), v(splat2(a.k.x)), nv(splat2(-a.k.x)),
          y(splat2(a.k.y)), ny(splat2(-a.k.y)), z(splat2(a.k.z)), w(splat2(a.k.w)) {}
};

__device__ __forceinline__ void r2_reference_ff2(f2 cab, const ARowR2 &A, f2 bx, f2 by, f2 bz,
                                                 f2 bw, float &q0, float &q1, bool &redo0,
                                                 bool &redo1) {
    f2 v3 = mul2(cab, A.rS);
    v3 = fma2(fma2(v3, A.nS, cab), A.rS, v3);
    const f2 np12 = mul2(A.nv, bx);
    const f2 e = fma2(A.v, bx, np12);
    const f2 d = add2(v3, np12);
    const f2 x = mul2(d, d);
    const f2 nPh = mul2(A.ny, by), Ph = mul2(A.y, by);
    f2 Pl = fma2(A.y, by, nPh);
    Pl = fma2(A.y, bz, Pl);
    Pl = fma2(A.z, by, Pl);
    const f2 t = mul2(e, mul2(A.w, bw));
    const f2 qh = mul2(x, Ph);
    f2 ql = fma2(x, Ph, mul2(x, nPh));
    ql = fma2(x, Pl, ql);
    ql = fma2(qh, t, ql);
    const f2 rh = add2(qh, fma2(qh, splat2(0x1p-40f), ql));
    const f2 rl = add2(qh, fma2(qh, splat2(-0x1p-40f), ql));
    float l0, l1, x0, x1;
    unpack2(rh, q0, q1);
    unpack2(rl, l0, l1);
    unpack2(x, x0, x1);
    const uint32_t tiny = __float_as_uint(0x1p-100f) - 1u;
    redo0 = !(q0 == l0) || __float_as_uint(x0) - 1u < tiny;
    redo1 = !(q1 == l1) || __float_as_uint(x1) - 1u < tiny;
}

// A pair the fast path flagged.  A fixed SNP (v = 1: every sample carries
// the allele) makes the reference's denominator p12 (1 - vA)(1 - vB) exactly
// +0, so its quotient is x / +0 = +inf, hence 123.456, or 0 / 0, the x86
// default NaN 0xFFC00000 (gemm_cpu.c:363-389); that needs x alone, with the
// reference's float rounding, and no FP64 division.  Empty SNPs keep the
// zero rule; bit counts above S and the rare rounding cases run the literal
// sequence.  q = fl32((float)cab / S), the reference's v3.
__device__ __forceinline__ float r2_fixed(float q, float vA, float vB) {
    const float d = __fsub_rn(q, __fmul_rn(vA, vB));
    return __fmul_rn(d, d) == 0.0f ? __uint_as_float(0xFFC00000u) : 123.456f;
}

__device__ __forceinline__ float r2_flagged(uint32_t cab, const RowRef &A, const RowRef &B,
                                            int S, float q) {
    if (A.v == 0.0f || B.v == 0.0f) return 0.0f;
    if (A.v <= 1.0f && B.v <= 1.0f && (A.v == 1.0f || B.v == 1.0f)) return r2_fixed(q, A.v, B.v);
    return r2_reference(cab, A, B, S);
}

// The fast path over a reference-mode chunk: v becomes the results, a flagged
// pair keeps its accumulator word; returns the flagged columns.  put(t, c)
// takes every column's count: interleaved with the arithmetic, as its stores
// would otherwise queue up before it.
template <int SHIFT, bool FLOATCNT, int CW, class C, class Put>
__device__ __forceinline__ uint32_t ref_columns(uint32_t (&v)[CW], const ARowR &ra, const C &f,
                                                int bl0, int S, Put put) {
    auto count = [&](int t) {
        return FLOATCNT ? (uint32_t)__uint_as_float(v[t]) : v[t] >> SHIFT;
    };
    uint32_t redo = 0;
    if (S > (1 << 24)) {
#pragma unroll
        for (int t = 0; t < CW; ++t) put(t, count(t));
        redo = CW == 32 ? 0xFFFFFFFFu : (1u << CW) - 1u;
    } else if constexpr (C::PAIRS) {
        const ARowR2 A(ra);
        float rmax = 0.0f;
#pragma unroll
        for (int t = 0; t < CW; t += 2) {
            put(t, count(t));
            put(t + 1, count(t + 1));
            f2 bx, by, bz, bw;
            f.pair(bl0 + t, bx, by, bz, bw);
            float q0, q1;
            bool rd0, rd1;
            r2_reference_ff2(pack2(__uint_as_float(v[t]), __uint_as_float(v[t + 1])), A, bx, by,
                             bz, bw, q0, q1, rd0, rd1);
            rmax = max3(rmax, q0, q1);
            v[t] = rd0 ? v[t] : __float_as_uint(q0);
            v[t + 1] = rd1 ? v[t + 1] : __float_as_uint(q1);
            redo |= (uint32_t)rd0 << t | (uint32_t)rd1 << (t + 1);
        }
        const float limit = __uint_as_float(0x3F800000u + 838u);
        if (__any_sync(0xffffffffu, rmax > limit)) {
#pragma unroll
            for (int t = 0; t < CW; ++t)
                if (!((redo >> t) & 1u) && __uint_as_float(v[t]) > limit)
                    v[t] = __float_as_uint(123.456f);
        }
    } else {
#pragma unroll
        for (int t = 0; t < CW; ++t) {
            const uint32_t raw = v[t];
            put(t, count(t));
            bool rd;
            const float r = r2_reference_ff(FLOATCNT ? __uint_as_float(raw) : (float)(raw >> SHIFT),
                                            ra, f.col(bl0 + t), rd);
            v[t] = rd ? raw : __float_as_uint(r);
            redo |= (uint32_t)rd << t;
        }
    }
    return redo;
}

// The reference-mode chunk of CW (<= 32) columns: every pair on the fast
// path, the flagged ones (their accumulator word kept in v, a bit in `redo`)
// redone with r2_flagged.
// FLOATCNT: v holds each count as F32 bits (the 4-bit kernels' accumulators),
// else as an integer shifted left by SHIFT.  With ColsR2 the fast path runs on
// two columns at a time (FLOATCNT only).
template <int SHIFT, bool FLOATCNT, int CW = 32, class C>
__device__ __forceinline__ void chunk_ref(uint32_t (&v)[CW], const ARowR &ra, const C &f,
                                          int bl0, int b0, int a, bool a_ok, int n, int dlo,
                                          int dhi, float *r2, long long ldr, uint32_t *counts,
                                          long long ldc, int row0, int S) {
    static_assert(FLOATCNT || !C::PAIRS, "packed pairs take F32 counts");
    uint32_t redo = 0;
    if (counts) {
        uint32_t *oc = counts + (long long)(b0 - row0) * ldc + a;
        const uint32_t mask = column_mask<CW>(b0, a, a_ok, n, dlo, dhi);
        redo = ref_columns<SHIFT, FLOATCNT, CW>(v, ra, f, bl0, S, [&](int t, uint32_t c) {
            store_if(oc + (long long)t * ldc, c, (mask >> t) & 1u);
        });
    } else {
        redo = ref_columns<SHIFT, FLOATCNT, CW>(v, ra, f, bl0, S, [](int, uint32_t) {});
    }
    if (!a_ok) redo = 0;
    if (__any_sync(0xffffffffu, redo != 0)) {
        // A lane whose A row is a fixed SNP (v = 1) has all its pairs flagged:
        // they take r2_flagged's fixed-SNP rule here in one pass, with
        // r2_reference_ff's quotient, instead of one trip each through the
        // warp-wide loop below (columns with bit counts above S stay flagged).
        const bool a_fixed = S <= (1 << 24) && ra.k.x == 1.0f && redo != 0u;
        if (__any_sync(0xffffffffu, a_fixed) && a_fixed) {
#pragma unroll
            for (int t = 0; t < CW; ++t) {
                const float vb = f.col(bl0 + t).x;
                if (((redo >> t) & 1u) && vb <= 1.0f) {
                    const float cf = FLOATCNT ? __uint_as_float(v[t]) : (float)(v[t] >> SHIFT);
                    v[t] = __float_as_uint(
                        vb == 0.0f ? 0.0f : r2_fixed(ref_quotient_ff(cf, ra), 1.0f, vb));
                    redo &= ~(1u << t);
                }
            }
        }
        // one reduction for the flagged columns, not a vote for each (twelve 200-450-row
        // tasks of K = 3 with 5 % fixed and 5 % empty SNPs 30.6 -> 28.7 us, 300 tasks
        // 1,064 -> 1,050)
        const uint32_t columns = __reduce_or_sync(0xffffffffu, redo);
        if (columns != 0u) {
            RowRef rA;
            rA.c = ra.c;
            rA.v = ra.k.x;
            rA.one_minus = __dsub_rn(1.0, (double)ra.k.x);
#pragma unroll
            for (int t = 0; t < CW; ++t) {
                if (!((columns >> t) & 1u)) continue;
                if ((redo >> t) & 1u) {
                    const float4 cb = f.col(bl0 + t);
                    RowRef rb;
                    rb.c = cb.x != 0.0f;        // only the zero rule reads it
                    rb.v = cb.x;
                    rb.one_minus = __dsub_rn(1.0, (double)cb.x);
                    const uint32_t cnt =
                        FLOATCNT ? (uint32_t)__uint_as_float(v[t]) : v[t] >> SHIFT;
                    const float q = S <= (1 << 24) ? ref_quotient_ff((float)cnt, ra)
                                                   : __fdiv_rn((float)cnt, (float)S);
                    v[t] = __float_as_uint(r2_flagged(cnt, rA, rb, S, q));
                }
            }
        }
    }
    if (!a_ok) return;
    float *o = r2 + (long long)(b0 - row0) * ldr + a;
    const bool interior = (b0 + CW - 1 < n) && (a - (b0 + CW - 1) >= dlo) && (a - b0 <= dhi);
    if (interior) {
#pragma unroll
        for (int t = 0; t < CW; ++t) o[(long long)t * ldr] = __uint_as_float(v[t]);
    } else {
#pragma unroll
        for (int t = 0; t < CW; ++t) {
            const int b = b0 + t;
            if (b < n && a - b >= dlo && a - b <= dhi) o[(long long)t * ldr] = __uint_as_float(v[t]);
        }
    }
}

// chunk_ref for a warp whose row and columns have no NaN factor (no fixed SNP),
// without the counts: every pair on the fast path, in pairs of columns.  If
// one is flagged or meets the > 1.0001 rule, the chunk's counts are loaded
// again (reload(v)) and it goes through chunk_ref.  At S >= R2_PLAIN_S that is
// one chunk in some hundreds; smaller S meet rounding midpoints more often.
constexpr int R2_PLAIN_S = 256;
template <int CW, class Reload>
__device__ __forceinline__ void chunk_ref_plain(uint32_t (&v)[CW], const ARowR &ra,
                                                const ColsR2 &f, int bl0, int b0, int a, bool a_ok,
                                                int n, int dlo, int dhi, float *r2, float *o,
                                                long long ldr, int row0, int S, Reload reload) {
    const ARowR2 A(ra);
    float rmax = 0.0f;
    bool bad = false;
#pragma unroll
    for (int t = 0; t < CW; t += 2) {
        f2 bx, by, bz, bw;
        f.pair(bl0 + t, bx, by, bz, bw);
        float q0, q1;
        bool rd0, rd1;
        r2_reference_ff2(pack2(__uint_as_float(v[t]), __uint_as_float(v[t + 1])), A, bx, by, bz,
                         bw, q0, q1, rd0, rd1);
        rmax = max3(rmax, q0, q1);
        bad = bad || rd0 || rd1;
        v[t] = __float_as_uint(q0);
        v[t + 1] = __float_as_uint(q1);
    }
    bad = bad || rmax > __uint_as_float(0x3F800000u + 838u);
    if (__any_sync(0xffffffffu, a_ok && bad)) {
        reload(v);
        chunk_ref<0, true, CW>(v, ra, f, bl0, b0, a, a_ok, n, dlo, dhi, r2, ldr, nullptr, 0, row0,
                               S);
        return;
    }
    if (!a_ok) return;
    const bool interior = (b0 + CW - 1 < n) && (a - (b0 + CW - 1) >= dlo) && (a - b0 <= dhi);
    if (interior) {
#pragma unroll
        for (int t = 0; t < CW; ++t) o[(long long)t * ldr] = __uint_as_float(v[t]);
    } else {
#pragma unroll
        for (int t = 0; t < CW; ++t) {
            const int b = b0 + t;
            if (b < n && a - b >= dlo && a - b <= dhi) o[(long long)t * ldr] = __uint_as_float(v[t]);
        }
    }
}

// One 32-column chunk: accumulators v[t] (holding count << shift) of A row a
// against B rows b0 + t (local columns bl0 + t).  Output element (b, a) goes
// to r2[(b - row0) * ldr + a] (and counts likewise).  Only entries inside the
// task (b < n, a < m) and the diagonal window dlo <= a - b <= dhi are
// written (a single region: a >= b; a band: 1 <= a - b <= W).
template <int MODE, int SHIFT>
__device__ __forceinline__ void chunk(uint32_t (&v)[32], const ARow &ra, const Cols &f,
                                      int bl0, int b0, int a, bool a_ok, int n, int dlo,
                                      int dhi, float *r2, long long ldr, uint32_t *counts,
                                      long long ldc, int row0, int S) {
    if constexpr (MODE == R2_REFERENCE) {
        chunk_ref<SHIFT, false>(v, ra.rr, ColsR(f.base, 0), bl0, b0, a, a_ok, n, dlo, dhi, r2,
                                ldr, counts, ldc, row0, S);
    } else {
        if (!a_ok) return;
        const double S_d = (double)S;
        float *o = r2 + (long long)(b0 - row0) * ldr + a;
        uint32_t *oc = counts ? counts + (long long)(b0 - row0) * ldc + a : nullptr;
        const bool interior = (b0 + 31 < n) && (a - (b0 + 31) >= dlo) && (a - b0 <= dhi);
        if (interior) {
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                const uint32_t cnt = v[t] >> SHIFT;
                o[(long long)t * ldr] = pair_r2_exact(cnt, ra, f, bl0 + t, S_d);
                if (oc) oc[(long long)t * ldc] = cnt;
            }
        } else {
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                const int b = b0 + t;
                if (b < n && a - b >= dlo && a - b <= dhi) {
                    const uint32_t cnt = v[t] >> SHIFT;
                    o[(long long)t * ldr] = pair_r2_exact(cnt, ra, f, bl0 + t, S_d);
                    if (oc) oc[(long long)t * ldc] = cnt;
                }
            }
        }
    }
}

// ------------------------------------------------ 4-bit kernels, R2_EXACT --
//
// The 4-bit kernels' accumulators hold each count as an exact F32 integer
// (below 2^24, as are S, cA and cB), so D = S*c - cA*cB can be evaluated in
// FP32 with a tight bound: split cA*cB = hi + lo exactly (hi = fl(cA*cB),
// lo = fma(cA, cB, -hi), the FMA TwoProduct; lo is an integer, |lo| <= 2^23),
// then D = fl(fl(S*c - hi) - lo) with S*c - hi rounded once by an FMA.  If
// |S*c - hi| < 2^24 the FMA is exact and D is rounded once; otherwise
// |D| >= |S*c - hi| / 2 and D carries at most 3 * 2^-24 relative error.  Then r^2 = (D*D) * (invA*invB) with
// invA = fl(1/(cA(S-cA))) rounded from FP64: at most 11 * 2^-24 (6.6e-7)
// relative error against the FP64 value, a dozen FP32 instructions per pair
// instead of a chain of FP64 ones.  Exact zeros (D = 0), the 0 rule for
// empty SNPs and NaN for 0/0 match the FP64 evaluation; values above 1.00009
// (possible only when the bit counts do not match the data) are re-evaluated
// in FP64 so the 123.456 rule decides exactly as in the other kernels.
//
// Factors of a row or column: c and 1/(c(S-c)), the latter 0 for an empty SNP
// (c = 0), so that its pairs come out 0 without a test.  That fails only
// against a factor that is not a finite, non-negative number -- a fixed SNP
// (c = S: infinity) or a bit count above S -- which `special` reports: a warp
// that holds or meets one applies the zero rule explicitly.  Tables with fixed
// SNPs do that in nearly every tile, so the rule stands in the loop over the
// pairs; as a second pass that read the columns again it made them slower than
// a test in every launch had been (11,734 x 10,140 SNPs of K = 3 with 5 % fixed
// and 5 % empty SNPs: such a test 166 us, second pass 218, now 152; K = 80, 9,001 x
// 7,003 147 / 168 / 131; 300-row tasks in a batch 16.4 / 18.5 / 14.4).
struct FactorF {
    float c, inv;
    bool special;
};

__device__ __forceinline__ double inv_var64(double c, double S) { return 1.0 / (c * (S - c)); }

__device__ __forceinline__ FactorF factor_f32(uint32_t c, int S) {
    FactorF r;
    r.c = (float)c;
    r.inv = c == 0u ? 0.0f : __double2float_rn(inv_var64((double)c, (double)S));
    r.special = !(r.inv >= 0.0f && r.inv < __uint_as_float(0x7F800000u));
    return r;
}

// Column factors, a float4 per column pair: c, c, 1/(c(S-c)), 1/(c(S-c)).
struct ColsF {
    float *f;
    __device__ __forceinline__ ColsF(uint8_t *base, int) : f(reinterpret_cast<float *>(base)) {}
    __device__ __forceinline__ float c(int bl) const { return f[(bl >> 1) * 4 + (bl & 1)]; }
    __device__ __forceinline__ ulonglong2 pair(int bl) const {   // bl even: {c, c}, {inv, inv}
        return *reinterpret_cast<const ulonglong2 *>(f + bl * 2);
    }
};

// Returns the column's `special`.
__device__ __forceinline__ bool store_col_f32(const ColsF &f, int bl, uint32_t c, int S) {
    const FactorF x = factor_f32(c, S);
    f.f[(bl >> 1) * 4 + (bl & 1)] = x.c;
    f.f[(bl >> 1) * 4 + 2 + (bl & 1)] = x.inv;
    return x.special;
}

typedef FactorF ARowF;

__device__ __forceinline__ ARowF make_arow_f32(uint32_t c, int S) { return factor_f32(c, S); }

// The FP64 evaluation (pair_r2_exact) from the same exact inputs.
__device__ __forceinline__ float pair_r2_f64(float c, float ca, float cb, int S) {
    if (ca == 0.0f || cb == 0.0f) return 0.0f;
    const double Sd = (double)S, a = (double)ca, b = (double)cb;
    const double D = fma(Sd, (double)c, -(a * b));
    const double r = (D * D) * (inv_var64(a, Sd) * inv_var64(b, Sd));
    if (r > 1.0001) return 123.456f;
    return __double2float_rn(r);
}

// The FP32 values of a chunk's counts, in pairs of columns; their maximum folded
// into rmax.  ZERO: with the zero rule, a pair of an empty SNP is 0 whatever the
// other's factor (hi = cA cB is 0 there only).
template <int CW, bool ZERO>
__device__ __forceinline__ void chunk_values_f32(uint32_t (&v)[CW], const ARowF &ra,
                                                 const ColsF &f, int bl0, float S_f, float &rmax) {
    const f2 S2 = splat2(S_f), ca = splat2(ra.c), nca = splat2(-ra.c), ia = splat2(ra.inv);
#pragma unroll
    for (int t = 0; t < CW; t += 2) {
        const ulonglong2 col = f.pair(bl0 + t);
        const f2 cnt = pack2(__uint_as_float(v[t]), __uint_as_float(v[t + 1]));
        const f2 nhi = mul2(nca, col.x);                       // -hi
        const f2 lo = fma2(ca, col.x, nhi);
        const f2 D = sub2(fma2(S2, cnt, nhi), lo);
        float r0, r1;
        unpack2(mul2(mul2(D, D), mul2(ia, col.y)), r0, r1);
        if constexpr (ZERO) {
            float h0, h1;
            unpack2(nhi, h0, h1);
            r0 = h0 == 0.0f ? 0.0f : r0;
            r1 = h1 == 0.0f ? 0.0f : r1;
        }
        rmax = max3(rmax, r0, r1);
        v[t] = __float_as_uint(r0);
        v[t + 1] = __float_as_uint(r1);
    }
}

// One chunk of CW (<= 32) columns of F32 accumulators v[t] (count c as float bits), as
// chunk<R2_EXACT, 0> with the FP32 evaluation above.  taddr is the TMEM
// address the chunk was loaded from: the rare pairs whose FP32 value lies
// above 1.00009 are re-evaluated in FP64 from their count, reloaded one
// column at a time (warp-uniform loads, off the common path).
// cols_special: a column of the tile is `special`.  ONE: the loop with the zero
// rule for every warp, for callers whose time one loop less of code is worth more
// than the rule (65 tasks with counts in a batch 52.5 -> 49.4 us, with fixed SNPs
// 57.5 -> 51.7; the single-SM kernel is 2 % faster with both).
// The counts go out as plain or predicated stores: with a test and a branch per
// column the arithmetic waited for each (11,776 x 10,140 SNPs, K = 3 298 -> 183
// us, 9,001 x 7,003 of K = 130 249 -> 204).
template <int CW = 32, bool ONE = false>
__device__ __forceinline__ void chunk_f32(uint32_t (&v)[CW], uint32_t taddr, const ARowF &ra,
                                          const ColsF &f, bool cols_special, int bl0, int b0,
                                          int a, bool a_ok, int n, int dlo, int dhi, float *r2,
                                          long long ldr, uint32_t *counts, long long ldc, int row0,
                                          int S) {
    if (counts) {
        uint32_t *oc = counts + (long long)(b0 - row0) * ldc + a;
        const uint32_t mask = column_mask<CW>(b0, a, a_ok, n, dlo, dhi);
        if (mask == (CW == 32 ? 0xFFFFFFFFu : (1u << CW) - 1u)) {
#pragma unroll
            for (int t = 0; t < CW; ++t)
                oc[(long long)t * ldc] = (uint32_t)__uint_as_float(v[t]);
        } else {
#pragma unroll
            for (int t = 0; t < CW; ++t)
                store_if(oc + (long long)t * ldc, (uint32_t)__uint_as_float(v[t]),
                         (mask >> t) & 1u);
        }
    }
    float rmax = 0.0f;
    if (ONE || __any_sync(0xffffffffu, ra.special) || cols_special)
        chunk_values_f32<CW, true>(v, ra, f, bl0, (float)S, rmax);
    else
        chunk_values_f32<CW, false>(v, ra, f, bl0, (float)S, rmax);
    if (__any_sync(0xffffffffu, rmax > 1.00009f)) {
#pragma unroll
        for (int t = 0; t < CW; ++t) {
            const bool redo = __uint_as_float(v[t]) > 1.00009f;
            if (__any_sync(0xffffffffu, redo)) {
                uint32_t w;
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];"
                             : "=r"(w)
                             : "r"(taddr + (uint32_t)t));
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (redo)
                    v[t] = __float_as_uint(
                        pair_r2_f64(__uint_as_float(w), ra.c, f.c(bl0 + t), S));
            }
        }
    }
    if (!a_ok) return;
    float *o = r2 + (long long)(b0 - row0) * ldr + a;
    const bool interior = (b0 + CW - 1 < n) && (a - (b0 + CW - 1) >= dlo) && (a - b0 <= dhi);
    if (interior) {
#pragma unroll
        for (int t = 0; t < CW; ++t) o[(long long)t * ldr] = __uint_as_float(v[t]);
    } else {
#pragma unroll
        for (int t = 0; t < CW; ++t) {
            const int b = b0 + t;
            if (b < n && a - b >= dlo && a - b <= dhi) o[(long long)t * ldr] = __uint_as_float(v[t]);
        }
    }
}

// chunk_f32 for a warp whose row and columns are not `special`, without the
// counts and without its votes: the values as FP32 gives them, their maximum
// folded into rmax.  A caller that finds rmax above R2_RECHECK in any lane
// runs the tile's chunks again through chunk_f32, which overwrites them.
constexpr float R2_RECHECK = 1.00009f;
template <int CW>
__device__ __forceinline__ void chunk_f32_plain(uint32_t (&v)[CW], const ARowF &ra, const ColsF &f,
                                                int bl0, int b0, int a, bool a_ok, int n, int dlo,
                                                int dhi, float *o, long long ldr, float S_f,
                                                float &rmax) {
    chunk_values_f32<CW, false>(v, ra, f, bl0, S_f, rmax);
    if (!a_ok) return;
    const bool interior = (b0 + CW - 1 < n) && (a - (b0 + CW - 1) >= dlo) && (a - b0 <= dhi);
    if (interior) {
#pragma unroll
        for (int t = 0; t < CW; ++t) o[(long long)t * ldr] = __uint_as_float(v[t]);
    } else {
#pragma unroll
        for (int t = 0; t < CW; ++t) {
            const int b = b0 + t;
            if (b < n && a - b >= dlo && a - b <= dhi) o[(long long)t * ldr] = __uint_as_float(v[t]);
        }
    }
}

// A warp's share of a task summary (BatchSummary): fold() takes the r^2
// values chunk_f32 left in v (A row a against B rows b0 + t), flush() sums
// the warp's lanes and adds them to the task's summary with three atomics.
struct SumAcc {
    double sum = 0.0;
    unsigned long long cnt = 0;
    float mx = 0.0f;
    template <int CW>
    __device__ __forceinline__ void fold(const uint32_t (&v)[CW], int b0, int a, bool a_ok,
                                         int n, int symmetric, float threshold) {
        if (!a_ok) return;
#pragma unroll
        for (int t = 0; t < CW; ++t) {
            const int b = b0 + t;
            const float r = __uint_as_float(v[t]);
            // a pair of the task, and not NaN or the 123.456 sentinel
            if (b < n && (!symmetric || a > b) && r < 100.0f) {
                sum += (double)r;
                cnt += r >= threshold;
                mx = fmaxf(mx, r);
            }
        }
    }
    __device__ __forceinline__ void flush(BatchSummary *out) {
        for (int o = 16; o > 0; o >>= 1) {
            sum += __shfl_down_sync(0xffffffffu, sum, o);
            cnt += __shfl_down_sync(0xffffffffu, cnt, o);
            mx = fmaxf(mx, __shfl_down_sync(0xffffffffu, mx, o));
        }
        if ((threadIdx.x & 31) == 0) {
            atomicAdd(&out->sum, sum);
            atomicAdd(&out->n_above, cnt);
            atomicMax(&out->max_bits, __float_as_uint(mx));
        }
    }
};

}  // namespace epi
}  // namespace qld
