// Device code of the tile walks (idw_tile.cu): the recorded terms of 32 volume
// nodes taken 16 at a time, their weights as FP16 digits in tensor-core operand
// layout, and the sums over the terms as matrix products.
//
// A unit is a group of 32 volume nodes and one mirror image; a warp works on
// one unit.  Its list holds {term, node mask} entries in steps of 16, a term
// being a surface point or an approximated cluster.  In the fragment layout of
// mma.m16n8k16 lane (g, t) = (lane / 4, lane % 4) holds rows g and g + 8 of two
// 16-node tiles and four of the step's terms (entries 4t .. 4t+3), so it forms
// those 16 weights itself: no weight crosses a lane.
#pragma once
#include <cuda_fp16.h>

#include "idw_mixed.cuh"

namespace idw {

constexpr int kTileTerms = 16;  // list entries per step

// d += a b, FP16 operands, FP32 accumulators.
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint4 a, unsigned b0, unsigned b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}
// d = a b.
__device__ __forceinline__ void mma_f16_first(float (&d)[4], const uint4 a, unsigned b0, unsigned b1) {
    asm(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1), "f"(0.f));
}

// Two floats rounded to FP16, lo in the low half.
__device__ __forceinline__ unsigned pack_f16(float lo, float hi) {
    const __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<const unsigned *>(&h);
}

__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }
// a b - c, one rounding (the error of c = a b).
__device__ __forceinline__ float2 fms2(float2 a, float2 b, float2 c) { return fma2(a, b, neg2(c)); }
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2 &s, float2 &e) {
    s = add2(a, b);
    const float2 bp = sub2(s, a);
    e = add2(sub2(a, sub2(s, bp)), sub2(b, bp));
}

// Weight law of the tile walks, exponents (3, 5): w = A P y^3 (1 + kappa y^2),
// y = 1/d.  It is the reference's A ((L/d)^3 + alpha^5 (L/d)^5) times P / L^3,
// with kappa = alpha^5 L^2 in two floats and P the node's power-of-two scale.
struct TileLaw {
    float kh, kl;
};

// The weights of one term at a pair of nodes (the halves of each float2), in
// double-float: w + wl to about 2^-44.  h, l: the nodes' positions, c, d: the
// term's (high parts and area, low parts and area).  The offset is an exact
// difference of the high parts plus the low parts, |x|^2 exact squares plus
// corrections, and the softening eps, which can be larger than all of them, an exact
// sum; the residual 1 - q y^2 of the reciprocal square root and the errors of the
// products are carried to first order.
__device__ __forceinline__ float2 tile_weight(const float4 c, const float4 d, float eps, const float2 *h,
                                              const float2 *l, float2 P, const TileLaw law, float2 &wl) {
    const float2 one = dup2(1.0f);
    const float ch[3] = {c.x, c.y, c.z}, cl[3] = {d.x, d.y, d.z};
    float2 p[3], low = dup2(-3.6274936e-9f * eps);  // what FP32 leaves of 1e-15
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        // a + b = (h - ch) + (l - cl), renormalised: b is below an ulp of a
        const float2 a0 = sub2(h[k], dup2(ch[k])), bb = sub2(a0, h[k]);
        const float2 b0 = add2(sub2(sub2(h[k], sub2(a0, bb)), add2(dup2(ch[k]), bb)), sub2(l[k], dup2(cl[k])));
        const float2 a = add2(a0, b0), b = sub2(b0, sub2(a, a0));
        p[k] = mul2(a, a);
        // (a + b)^2 - a^2 = (2 a + b) b
        low = fma2(fma2(dup2(2.0f), a, b), b, add2(low, fms2(a, a, p[k])));
    }
    float2 s1, e1, s2, e2, s3, e3;
    two_sum2(p[0], p[1], s1, e1);
    two_sum2(s1, p[2], s2, e2);
    two_sum2(s2, dup2(eps), s3, e3);
    low = add2(low, add2(add2(e1, e2), e3));
    const float2 q = add2(s3, low), ql = sub2(low, sub2(q, s3));
    const float2 y = make_float2(rsqrt_normal(q.x), rsqrt_normal(q.y));
    const float2 y2 = mul2(y, y), y2l = fms2(y, y, y2);
    const float2 t0 = mul2(q, y), t0l = fms2(q, y, t0);
    // r = 1 - (q + ql) y^2
    const float2 r = fma2(neg2(ql), y2, fma2(neg2(t0l), y, fma2(neg2(t0), y, one)));
    const float2 yp = mul2(y, P);
    const float2 v = mul2(y2, yp), vl = fma2(y2l, yp, fms2(y2, yp, v));
    // u + ul = 1 + kappa y^2, whichever of the two is larger
    const float2 ky = mul2(dup2(law.kh), y2);
    float2 u, ue;
    two_sum2(ky, one, u, ue);
    const float2 ul =
        fma2(dup2(law.kl), y2, fma2(dup2(law.kh), y2l, add2(fms2(dup2(law.kh), y2, ky), ue)));
    const float2 t = mul2(v, u);
    // y (1 + r / 2) for y: v u gains v r (5 u - 2) / 2
    const float2 tl = fma2(mul2(v, fma2(dup2(2.5f), u, dup2(-1.0f))), r, fma2(vl, u, fma2(v, ul, fms2(v, u, t))));
    const float2 w0 = mul2(dup2(c.w), t);
    const float2 l0 = fma2(dup2(c.w), tl, fma2(dup2(d.w), t, fms2(dup2(c.w), t, w0)));
    // normalised: the digits take wl to be below an ulp of w (r alone is a few)
    const float2 w = add2(w0, l0);
    wl = sub2(l0, sub2(w, w0));
    return w;
}

// Keeps the weights of the nodes whose mask bits are set.  mg is the entry's
// mask shifted left by 7 - g: the bit of row g + 8 j is the sign of byte j.
__device__ __forceinline__ float2 tile_mask(float2 w, unsigned mg, int m) {
    // prmt selectors 8 + j: the sign of byte j in every byte
    unsigned a, b;
    const unsigned s = m ? mg >> 16 : mg;
    asm("prmt.b32 %0, %1, 0, 0x8888;" : "=r"(a) : "r"(s));
    asm("prmt.b32 %0, %1, 0, 0x9999;" : "=r"(b) : "r"(s));
    return make_float2(__uint_as_float(__float_as_uint(w.x) & a), __uint_as_float(__float_as_uint(w.y) & b));
}

// The four FP16 digits of the weights (w + wl) of two terms, A in the low half
// and B in the high one, at a row pair: s[.][0] row g, s[.][1] row g + 8.  A
// node's weights are scaled so that its denominator lies in [2^13, 2^14); the
// digits lie on the grids of 8, 2^-8 and 2^-19, and the last carries 2^22 times
// what is left, rounded (44 bits of the denominator in all).  FIFTH: s[0] is
// 2^22 times what those four leave (for the reverse product, where a term's own
// size counts and not the denominator's), the others are not set.
template <bool FIFTH>
__device__ __forceinline__ void tile_digits(float2 wa, float2 la, float2 wb, float2 lb, unsigned (&s)[4][2]) {
    float2 ra = dup2(0.f), rb = dup2(0.f);
    const float grid[3] = {1.5f * 67108864.0f, 1.5f * 32768.0f, 1.5f * 16.0f};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float2 M = dup2(grid[d]);
        const float2 a = sub2(add2(wa, M), M), b = sub2(add2(wb, M), M);
        if constexpr (!FIFTH) {
            s[d][0] = pack_f16(a.x, b.x);
            s[d][1] = pack_f16(a.y, b.y);
        }
        wa = sub2(wa, a);
        wb = sub2(wb, b);
        if (d == 1) {
            // the rest of w is below 2^-9 and exact; the low parts join it
            if constexpr (FIFTH) {
                two_sum2(wa, la, wa, ra);
                two_sum2(wb, lb, wb, rb);
            } else {
                wa = add2(wa, la);
                wb = add2(wb, lb);
            }
        }
    }
    const float2 S = dup2(4194304.0f);
    wa = mul2(wa, S);
    wb = mul2(wb, S);
    if constexpr (FIFTH) {
        const float2 a = make_float2(__half2float(__float2half_rn(wa.x)), __half2float(__float2half_rn(wa.y)));
        const float2 b = make_float2(__half2float(__float2half_rn(wb.x)), __half2float(__float2half_rn(wb.y)));
        wa = fma2(ra, S, sub2(wa, a));
        wb = fma2(rb, S, sub2(wb, b));
    }
    s[FIFTH ? 0 : 3][0] = pack_f16(wa.x, wb.x);
    s[FIFTH ? 0 : 3][1] = pack_f16(wa.y, wb.y);
}

// One step's weights being made, per warp.  dig: digit d of tile m as the lanes'
// fragment registers.
struct TileStage {
    int term[kTileTerms];
    unsigned mask[kTileTerms];
    uint4 dig[4][2][32];
};

__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    const unsigned d = unsigned(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16_l1(void *dst, const void *src) {
    const unsigned d = unsigned(__cvta_generic_to_shared(dst));
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Work distribution of the persistent kernels: units are taken from a global
// counter in chunks of consecutive ones, shared by the warps of a block (their
// terms overlap, so the block's L1 serves them together).  state holds the
// block's chunk as (end << 32 | next).  A warp that finds it empty takes the
// next chunk for the block; if another warp published one meanwhile, it keeps
// what was left of that to itself.  Nothing waits.
struct UnitQueue {
    unsigned long long *state;
    unsigned *counter;
    unsigned total, chunk, p, pe;
    __device__ __forceinline__ bool next(unsigned &unit) {
        unsigned u = 0xffffffffu;
        if ((threadIdx.x & 31) == 0) {
            if (p < pe) {
                u = p++;
            } else {
                const unsigned long long s = atomicAdd(state, 1ull);
                if (unsigned(s) < unsigned(s >> 32)) {
                    u = unsigned(s);
                } else {
                    const unsigned c = atomicAdd(counter, chunk);
                    if (c < total) {
                        u = c;
                        const unsigned e = min(c + chunk, total);
                        const unsigned long long o =
                            atomicExch(state, (static_cast<unsigned long long>(e) << 32) | (c + 1));
                        p = unsigned(o);
                        pe = unsigned(o >> 32);
                    }
                }
            }
        }
        unit = __shfl_sync(kFull, u, 0);
        return unit != 0xffffffffu;
    }
};

// The terms whose motion records a lane copies into a stage (one 16-byte chunk
// of each of four).
struct StageIds {
    int t[4];
};
__device__ __forceinline__ StageIds stage_ids(const int *term) {
    const int r = (threadIdx.x & 31) >> 3;
    return {{term[r], term[4 + r], term[8 + r], term[12 + r]}};
}
// Chunk g of term k lies at 8 k + (g ^ 2 (k / 4)), so that the fragment-order reads
// (lane (g, t): terms 4t .. 4t+3) meet no bank conflict.
__device__ __forceinline__ void stage_motions(uint4 *dst, const StageIds &s, const uint4 *mot) {
    const int lane = threadIdx.x & 31, g = lane & 7;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        cp_async16_l1(&dst[8 * (4 * c + (lane >> 3)) + (g ^ (2 * c))], mot + 8 * int64_t(s.t[c]) + g);
}

// The volume nodes of a lane: row pair (g + 16 m, g + 16 m + 8) of tile m.
struct TileRows {
    float2 h[3], l[3], P;
};

// The four digits of a step's weights into st.dig, or the fifth into st.dig[0],
// from its terms and masks.
template <bool FIFTH = false>
__device__ __forceinline__ void stage_weights(TileStage &st, const float4 *geo, int nPts, const TileRows *rows,
                                              const TileLaw law) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // rolled: one copy of the weight code
#pragma unroll 1
    for (int i = 0; i < 4; ++i) {
        const int p = i & 1, m = i >> 1;
        const int ta = st.term[4 * t + 2 * p], tb = st.term[4 * t + 2 * p + 1];
        const unsigned ma = st.mask[4 * t + 2 * p] << (7 - g), mb = st.mask[4 * t + 2 * p + 1] << (7 - g);
        const TileRows &R = rows[8 * m + g];
        float2 h[3], l[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            h[k] = R.h[k];
            l[k] = R.l[k];
        }
        const float2 P = R.P;
        float2 la, lb;
        float2 wa = tile_weight(ldgf4(geo + 2 * int64_t(ta)), ldgf4(geo + 2 * int64_t(ta) + 1),
                                ta < nPts ? 1e-15f : 0.f, h, l, P, law, la);
        float2 wb = tile_weight(ldgf4(geo + 2 * int64_t(tb)), ldgf4(geo + 2 * int64_t(tb) + 1),
                                tb < nPts ? 1e-15f : 0.f, h, l, P, law, lb);
        wa = tile_mask(wa, ma, m);
        la = tile_mask(la, ma, m);
        wb = tile_mask(wb, mb, m);
        lb = tile_mask(lb, mb, m);
        unsigned s[4][2];
        tile_digits<FIFTH>(wa, la, wb, lb, s);
#pragma unroll
        for (int d = 0; d < (FIFTH ? 1 : 4); ++d)
            reinterpret_cast<uint2 *>(&st.dig[d][m][lane])[p] = make_uint2(s[d][0], s[d][1]);
    }
}

// Accumulators of one unit, four digits: per 16-node tile and 8-column tile, the
// products of the first digits (exact: first digits on grids of 8, below 2^14 in
// sum), the products one digit down (a compensated pair), and the rest.
template <int ND>
struct TileAcc {
    float a0[2][2][4], a2[2][2][4];
    float2 a1[2][2][2];
};
template <int ND>
__device__ __forceinline__ void tile_zero(TileAcc<ND> &acc) {
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            acc.a1[m][n][0] = acc.a1[m][n][1] = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc.a0[m][n][j] = acc.a2[m][n][j] = 0.f;
        }
}

// The sums of a tangent: five digits of both.  A rough surface tangent has
// gradients D' far above its offsets e, which cancel near the term (D' (r - O) +
// e), and terms of large motion far from the node, so neither is good enough to
// the denominator or the largest motion only.
template <>
struct TileAcc<5> {
    float a0[2][2][4], a3[2][2][4], a4[2][2][4];  // leading products; third order and what two-sums leave; 2^22 times the rest
    float2 a1[2][2][2], a2[2][2][2];              // first and second order, by two-sums
};
template <>
__device__ __forceinline__ void tile_zero<5>(TileAcc<5> &acc) {
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            acc.a1[m][n][0] = acc.a1[m][n][1] = acc.a2[m][n][0] = acc.a2[m][n][1] = make_float2(0.f, 0.f);
#pragma unroll
            for (int j = 0; j < 4; ++j) acc.a0[m][n][j] = acc.a3[m][n][j] = acc.a4[m][n][j] = 0.f;
        }
}

// Total of column pair entry j = 2 r + k (k = 0, 1) of tiles m, n, as high and low.
template <int ND>
__device__ __forceinline__ void tile_total(const TileAcc<ND> &acc, int m, int n, int r, int k, float &s, float &low) {
    const float2 a1 = acc.a1[m][n][r];
    float e;
    two_sum(acc.a0[m][n][2 * r + k], k ? a1.y : a1.x, s, e);
    if constexpr (ND == 5) {
        const float2 a2 = acc.a2[m][n][r];
        float e2;
        two_sum(s, k ? a2.y : a2.x, s, e2);
        low = e + (e2 + fmaf(acc.a4[m][n][2 * r + k], 1.0f / 4194304.0f, acc.a3[m][n][2 * r + k]));
    } else {
        low = e + acc.a2[m][n][2 * r + k];
    }
}

// One step of the forward sums with four digits of the weights and of the motions
// (dig: digit d of 16-node tile m as the lanes' fragment registers at 64 d + 32 m;
// mot: the motion records of the step).
__device__ __forceinline__ void tile_step(const uint4 *dig, const uint4 *mot, TileAcc<4> &acc) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        // motion digits of the lane's terms: [digit][fragment register]
        unsigned C[4][2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const uint2 *q = reinterpret_cast<const uint2 *>(mot + 8 * (4 * t + 2 * p) + (g ^ (2 * t))) + n;
            const uint2 x = q[0], y = q[16];
            C[0][p] = __byte_perm(x.x, y.x, 0x5410);
            C[1][p] = __byte_perm(x.x, y.x, 0x7632);
            C[2][p] = __byte_perm(x.y, y.y, 0x5410);
            C[3][p] = __byte_perm(x.y, y.y, 0x7632);
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint4 *A = dig + 32 * m + lane;
            const uint4 A0 = A[0], A1 = A[64], A2 = A[128], A3 = A[192];
            // one digit down: exact in a step (the tensor core truncates its sums,
            // which over a list would be a bias), added by two-sums whose errors
            // join the rest; f: 2^22 times the products with a fourth digit
            float d[4], f[4];
            mma_f16_first(d, A0, C[1][0], C[1][1]);
            mma_f16_first(f, A0, C[3][0], C[3][1]);
            mma_f16(acc.a0[m][n], A0, C[0][0], C[0][1]);
            mma_f16(acc.a2[m][n], A1, C[1][0], C[1][1]);
            mma_f16(d, A1, C[0][0], C[0][1]);
            mma_f16(f, A3, C[0][0], C[0][1]);
            mma_f16(acc.a2[m][n], A0, C[2][0], C[2][1]);
            mma_f16(acc.a2[m][n], A2, C[0][0], C[0][1]);
            mma_f16(acc.a2[m][n], A1, C[2][0], C[2][1]);
            mma_f16(acc.a2[m][n], A2, C[1][0], C[1][1]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float2 s, e;
                two_sum2(acc.a1[m][n][r], make_float2(d[2 * r], d[2 * r + 1]), s, e);
                acc.a1[m][n][r] = s;
                e = fma2(make_float2(f[2 * r], f[2 * r + 1]), dup2(1.0f / 4194304.0f), e);
                acc.a2[m][n][2 * r] += e.x;
                acc.a2[m][n][2 * r + 1] += e.y;
            }
        }
    }
}

// One step of a tangent's sums.  mot5: the terms' fifth digits, chunk g of term k =
// 4 i + j in word 8 (4 i + (i + j) % 4) + g (no bank conflict for lane (g, t)).
__device__ __forceinline__ void tile_step5(const uint4 *dig, const uint4 *mot, const unsigned *mot5, TileAcc<5> &acc) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int n = 0; n < 2; ++n) {
        unsigned C[5][2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const uint2 *q = reinterpret_cast<const uint2 *>(mot + 8 * (4 * t + 2 * p) + (g ^ (2 * t))) + n;
            const uint2 x = q[0], y = q[16];
            C[0][p] = __byte_perm(x.x, y.x, 0x5410);
            C[1][p] = __byte_perm(x.x, y.x, 0x7632);
            C[2][p] = __byte_perm(x.y, y.y, 0x5410);
            C[3][p] = __byte_perm(x.y, y.y, 0x7632);
            C[4][p] = __byte_perm(mot5[8 * (4 * t + ((t + 2 * p) & 3)) + g], mot5[8 * (4 * t + ((t + 2 * p + 1) & 3)) + g],
                                  n ? 0x7632 : 0x5410);
        }
#pragma unroll
        for (int m = 0; m < 2; ++m) {
            const uint4 *A = dig + 32 * m + lane;
            const uint4 A0 = A[0], A1 = A[64], A2 = A[128], A3 = A[192], A4 = A[256];
            float d[4], f[4];
            mma_f16_first(d, A0, C[1][0], C[1][1]);
            mma_f16_first(f, A0, C[2][0], C[2][1]);
            mma_f16(acc.a3[m][n], A1, C[2][0], C[2][1]);
            mma_f16(acc.a4[m][n], A0, C[3][0], C[3][1]);
            mma_f16(d, A1, C[0][0], C[0][1]);
            mma_f16(f, A1, C[1][0], C[1][1]);
            mma_f16(acc.a3[m][n], A2, C[1][0], C[1][1]);
            mma_f16(acc.a4[m][n], A3, C[0][0], C[0][1]);
            mma_f16(acc.a0[m][n], A0, C[0][0], C[0][1]);
            mma_f16(f, A2, C[0][0], C[0][1]);
            mma_f16(acc.a4[m][n], A1, C[3][0], C[3][1]);
            mma_f16(acc.a3[m][n], A2, C[2][0], C[2][1]);
            mma_f16(acc.a4[m][n], A3, C[1][0], C[1][1]);
            mma_f16(acc.a4[m][n], A0, C[4][0], C[4][1]);
            mma_f16(acc.a4[m][n], A4, C[0][0], C[0][1]);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                // both orders are exact in a step
                float2 s, e, h;
                two_sum2(acc.a1[m][n][r], make_float2(d[2 * r], d[2 * r + 1]), s, e);
                acc.a1[m][n][r] = s;
                two_sum2(acc.a2[m][n][r], make_float2(f[2 * r], f[2 * r + 1]), s, h);
                acc.a2[m][n][r] = s;
                e = add2(e, h);
                acc.a3[m][n][2 * r] += e.x;
                acc.a3[m][n][2 * r + 1] += e.y;
            }
        }
    }
}

}  // namespace idw
