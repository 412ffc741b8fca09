// The reverse product of the tile walks (evalNode_b / evalNodeExact_b /
// evalNodeApprox_b, src/modules/kd_tree.F90:942-1031, driven as warpDeriv,
// src/warp/warpDeriv.F90:71-88): for every term the moments sum_i w_i n_i (1,
// r_i - X) over the volume nodes, with the seeds n_i = dXv_i / den_i, X the
// term's own position.
//
// The weights are the kept digits of the forward walk (idw_tile.cu) and a fifth:
// here an error counts against the term's own weights, not against the nodes'
// denominators.  Per unit (32 nodes, one mirror) the columns n (1, r - O), O the
// unit's origin, are split into five FP16 digits against each column's largest
// value; the moments of 16 terms are the product of the transposed weight tile
// (movmatrix) with them, digit products of equal order in accumulators of their
// own (the leading orders exact in FP32), summed in double-float, moved from O to
// X and landed by FP64 atomics.  The fifth digit of the columns is for that move:
// a term much nearer to a node than O is cancels against O - X.  Three of the 18
// digit products of a tile pair are left out (2^-42 of a far term's weights,
// 2^-54 of a near one's).
//
// The double-float walk that this replaces summed the 32 lanes of each term and
// seed component one after the other (idw_adjoint_precise.cu).  Against it, the
// 2M-node wing, errTol 1e-4: one seed 13.9 -> 2.9 ms, 16 seeds 105 -> 36 ms, with
// the same error (2e-14 to 2e-13 of the result for the walk alone).
// What bounds it: latency at 16 warps an SM (an instruction issues in 45% of the
// cycles, tensor pipe 28% busy, L2 atomics 5e10 sectors/s).
#include <climits>

#include "idw_tile.cuh"
#include "idwarp_gb300.h"

namespace idw {

namespace {

// Seeds taken together: two, with 16 warps an SM in the shared memory their
// columns leave, against four with 10 (the 2M-node wing, 16 seeds: 36.4 against
// 41.5 ms at one time, although the digits are read twice as often) or three with 12 (45 ms).
constexpr int kAdjSeeds = 2, kAdjWarps = 16;

// 8 x 8 FP16 tile transposed across the warp.
__device__ __forceinline__ unsigned transpose_f16(unsigned a) {
    unsigned d;
    asm("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(d) : "r"(a));
    return d;
}

// Seed columns of one unit in shared memory, S seeds: digits as the B fragments
// of column tile nt, both node tiles (x, y | z, w).  Component c (seed c / 3,
// axis c % 3) has its moments (1, x, y, z) in columns c % 2 + 0, 2, 4, 6 of tile
// c / 2, so that lane (g, t) of the product holds moment t: the four lanes of a
// term land one 32-byte sector.  off: (896 - e) << 20 for a column scaled by 2^e;
// rel: the factor from the scale of the component's moment 1 to the column's.
template <int S>
struct SeedTile {
    static constexpr int kTiles = (3 * S + 1) / 2;
    uint4 w[10][32];  // the step's weight digits, copied ahead: [2 digit + node tile][lane]
    uint4 b[5][kTiles][32];
    int off[kTiles][4][2];  // [tile][moment][component]
    float rel[kTiles][4][2];
};

// (h + l) 2^-e, |l| <= ulp(h) / 2, off = (896 - e) << 20, put together from the
// bits (an FP64 instruction holds this GPU's pipe for 16 cycles): h's, moved to
// the FP64 format, plus l in units of its last place.  Not for h = 0, nor beyond
// the range of odd_range.
__device__ __forceinline__ double join_bits(float h, float l, int off) {
    const unsigned hb = __float_as_uint(h), mag = hb & 0x7fffffffu, sgn = hb & 0x80000000u;
    const float sc = __uint_as_float((306u << 23) - (mag & 0x7f800000u));  // 2^(52 + 127 - exponent)
    int L = __float2int_rn(__uint_as_float(__float_as_uint(l) ^ sgn) * sc);
    // below a power of two the last place is half as large
    L = (mag & 0x7fffffu) == 0u && L < 0 ? 2 * L : L;
    const long long bits = ((static_cast<long long>(int(mag >> 3) + off) << 32) | (hb << 29)) + L;
    return __hiloint2double(int(bits >> 32) | int(sgn), int(bits));
}
__device__ __noinline__ double join_odd(float h, float l, int off) {
    return ldexp(double(h) + double(l), (off >> 20) - 896);
}
// Whether join_bits does not serve h (lim: 195, or 0 where the scales are extreme).
__device__ __forceinline__ bool odd_range(float h, unsigned lim) {
    return ((__float_as_uint(h) >> 23) & 0xffu) - 60u >= lim;
}

// One column (moment k of component c) scaled by 2^e0 already: the lane's value
// into its digits.  e1: the exponent of the component's moment 1.  Whether the
// scale is beyond join_bits' usual range.
template <int S>
__device__ __forceinline__ bool seed_column(SeedTile<S> &sm, int c, int k, dfl v, int e0, int &e1) {
    const int lane = threadIdx.x & 31;
    const unsigned mx = __reduce_max_sync(kFull, __float_as_uint(v.h) & 0x7fffffffu);
    // the largest value lands in [2^10, 2^11): with weights below 2^14 on a
    // grid of 8 the leading products of 32 nodes sum below 2^24 units
    const int e = mx ? max(-110, min(110, 10 - (int(mx >> 23) - 127))) : 0;
    const float sc = pow2f(e);
    float r = v.h * sc;
    const float lo = v.l * sc;
    const float M[3] = {1.5f * 67108864.0f, 1.5f * 32768.0f, 1.5f * 16.0f};
    float rest = 0.f;
    __half dg[5];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const float a = __fsub_rn(__fadd_rn(r, M[d]), M[d]);
        dg[d] = __float2half_rn(a);
        r = __fsub_rn(r, a);
        if (d == 1) two_sum(r, lo, r, rest);
    }
    r *= 4194304.0f;
    dg[3] = __float2half_rn(r);
    dg[4] = __float2half_rn(fmaf(rest, 4194304.0f, __fsub_rn(r, __half2float(dg[3]))));
    const int nt = c >> 1, col = 2 * k + (c & 1);
    const int m = lane >> 4, kk = lane & 15;
#pragma unroll
    for (int d = 0; d < 5; ++d)
        reinterpret_cast<__half *>(&sm.b[d][nt][4 * col + ((kk & 7) >> 1)])[4 * m + 2 * (kk >> 3) + (kk & 1)] = dg[d];
    if (k == 0) e1 = e;
    if (lane == 0) {
        sm.off[nt][k][c & 1] = (896 - e - e0) * (1 << 20);
        sm.rel[nt][k][c & 1] = pow2f(e - e1);
    }
    return e + e0 > 950 || e + e0 < -890;
}

// O - X on axis t - 1 of a term (high part O of the origin, both parts of X); zero
// for t = 0.
__device__ __forceinline__ dfl origin_offset(const float4 *geo, int term, int t, float O) {
    const float *p = reinterpret_cast<const float *>(geo + 2 * int64_t(term)) + (t > 0 ? t - 1 : 0);
    dfl x = {0.f, 0.f};
    if (t == 0) return x;
    two_diff(O, __ldg(p), x.h, x.l);
    return df_norm(x.h, x.l - __ldg(p + 4));
}

template <int S>
__global__ void __launch_bounds__(32 * kAdjWarps, 1)
    k_tile_adjoint(VolumeDev v, WalkRecF rec, MixedParams mp, TileDev td, TileLists lists, int nPts, unsigned nUnits,
                   unsigned chunk, const double *denInv, const double *dxv, int64_t dxvStride, double *ptAdj,
                   int64_t ptStride, double *nodeAdj, int64_t nodeStride) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ unsigned long long qstate;
    if (threadIdx.x == 0) qstate = 0ull;
    __syncthreads();
    SeedTile<S> &sm = reinterpret_cast<SeedTile<S> *>(smraw)[threadIdx.x >> 5];
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    // columns of absent components stay zero
    for (int i = lane; i < int(sizeof(sm.b) / sizeof(uint4)); i += 32) (&sm.b[0][0][0])[i] = make_uint4(0u, 0u, 0u, 0u);
    for (int i = lane; i < 8 * SeedTile<S>::kTiles; i += 32) {
        (&sm.off[0][0][0])[i] = 0;
        (&sm.rel[0][0][0])[i] = 1.0f;
    }
    __syncwarp();
    UnitQueue queue = {&qstate, td.counter, nUnits, chunk, 0u, 0u};
    unsigned unit;
    while (queue.next(unit)) {
        const int64_t group = unit / unsigned(mp.nLoop);
        const int kk = int(unit - unsigned(group) * unsigned(mp.nLoop));
        const int64_t e0 = lists.offs[unit];
        const int n = int((lists.offs[unit + 1] - e0) / kTileTerms);
        if (n <= 0) continue;
        // this lane's node: position about the unit's origin, seeds
        const int64_t slot = group * 32 + lane;
        const bool valid = slot < v.nVol;
        const int64_t at = valid ? slot : v.nVol - 1;
        const int64_t gid = td.order[at];
        const float4 hi = rec.hi[kk * v.nVol + gid], lo = rec.lo[kk * v.nVol + gid];
        const float O[3] = {__shfl_sync(kFull, hi.x, 0), __shfl_sync(kFull, hi.y, 0), __shfl_sync(kFull, hi.z, 0)};
        dfl x[3];
        two_diff(hi.x, O[0], x[0].h, x[0].l);
        two_diff(hi.y, O[1], x[1].h, x[1].l);
        two_diff(hi.z, O[2], x[2].h, x[2].l);
        x[0] = df_norm(x[0].h, x[0].l + lo.x);
        x[1] = df_norm(x[1].h, x[1].l + lo.y);
        x[2] = df_norm(x[2].h, x[2].l + lo.z);
        const int64_t vi = v.perm[gid];
        const double q = valid ? denInv[at] : 0.0;
        bool far = false;
        __syncwarp();
#pragma unroll 1
        for (int s = 0; s < S; ++s) {
            const double *dv = dxv + s * dxvStride + 3 * vi;
            double n3[3] = {dv[0] * q, dv[1] * q, dv[2] * q};
            if (!valid) n3[0] = n3[1] = n3[2] = 0.0;
            // the transpose of the numerator's reflection (getMirrorNumerator_b,
            // src/warp/initializeWarping.F90:603-635)
            for (int j = mp.nSym - 1; j >= 0; --j) {
                if ((kk >> j) & 1) {
                    const double nr[3] = {double(mp.nrm[j][0]) + double(mp.nrmLo[j][0]),
                                          double(mp.nrm[j][1]) + double(mp.nrmLo[j][1]),
                                          double(mp.nrm[j][2]) + double(mp.nrmLo[j][2])};
                    const double dp = 2.0 * (n3[0] * nr[0] + n3[1] * nr[1] + n3[2] * nr[2]);
                    n3[0] -= dp * nr[0];
                    n3[1] -= dp * nr[1];
                    n3[2] -= dp * nr[2];
                }
            }
#pragma unroll 1
            for (int a = 0; a < 3; ++a) {
                const double na = a == 0 ? n3[0] : (a == 1 ? n3[1] : n3[2]);
                // the unit's largest component to [1, 2): no range is lost in FP32
                const unsigned mx = __reduce_max_sync(kFull, unsigned(__double2hiint(na)) & 0x7fffffffu);
                const int e0 = max(-1000, min(1000, 1023 - int(mx >> 20)));
                const double ns = na * __hiloint2double((1023 + e0) << 20, 0);
                dfl w;
                w.h = float(ns);
                w.l = float(ns - double(w.h));
                int e1 = 0;
                far |= seed_column<S>(sm, 3 * s + a, 0, w, e0, e1);
#pragma unroll
                for (int k = 0; k < 3; ++k) far |= seed_column<S>(sm, 3 * s + a, k + 1, df_mul(w, x[k]), e0, e1);
            }
        }
        __syncwarp();
        const unsigned lim = far ? 0u : 195u;
        const float Ot = t == 1 ? O[0] : (t == 2 ? O[1] : O[2]);
        const uint4 *dig = lists.dig + 192 * (e0 / kTileTerms) + lane, *dig3 = lists.dig3 + 64 * (e0 / kTileTerms) + lane,
                    *dig4 = lists.dig4 + 64 * (e0 / kTileTerms) + lane;
        const int *term = lists.term + e0;
        // every lane copies what it reads itself
        auto fetch = [&](int st) {
#pragma unroll
            for (int i = 0; i < 6; ++i) cp_async16(&sm.w[i][lane], dig + 192 * int64_t(st) + 32 * i);
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                cp_async16(&sm.w[6 + m][lane], dig3 + 64 * int64_t(st) + 32 * m);
                cp_async16(&sm.w[8 + m][lane], dig4 + 64 * int64_t(st) + 32 * m);
            }
        };
        fetch(0);
        cp_async_commit();
        for (int st = 0; st < n; ++st) {
            cp_async_wait<0>();
            // terms as rows: fragment registers (nodes, terms) transposed;
            // row r is entry 4 (r / 2) + r % 2 for r < 8, two further for r >= 8
            uint4 A[5][2];
#pragma unroll
            for (int d = 0; d < 5; ++d)
#pragma unroll
                for (int m = 0; m < 2; ++m) {
                    const uint4 W = sm.w[2 * d + m][lane];
                    A[d][m] = make_uint4(transpose_f16(W.x), transpose_f16(W.z), transpose_f16(W.y), transpose_f16(W.w));
                }
            if (st + 1 < n) fetch(st + 1);
            cp_async_commit();
            // The nodes of a term, unlike the terms of a node, have no bound on their
            // weights' sum.  Up to 2^16 the products of first weight digits with second
            // column digits (below 4, on a grid of 2^-5) are exact in their accumulator.
            float rows[4];
            mma_f16_first(rows, A[0][0], 0x3c003c00u, 0x3c003c00u);
            mma_f16(rows, A[0][1], 0x3c003c00u, 0x3c003c00u);
            const bool heavy = __any_sync(kFull, fmaxf(rows[0], rows[2]) > 65536.0f);
            // the rows' terms: where they land, and O - X on the lane's axis (0 for moment 1)
            const int tA = __ldg(term + kTileTerms * st + 4 * (g >> 1) + (g & 1));
            const int tB = __ldg(term + kTileTerms * st + 4 * (g >> 1) + (g & 1) + 2);
            const dfl xA = origin_offset(td.geo, tA, t, Ot), xB = origin_offset(td.geo, tB, t, Ot);
            double *dA = (tA < nPts ? ptAdj + 12 * int64_t(tA) : nodeAdj + 12 * int64_t(tA - nPts)) + t;
            double *dB = (tB < nPts ? ptAdj + 12 * int64_t(tB) : nodeAdj + 12 * int64_t(tB - nPts)) + t;
            const int64_t sA = tA < nPts ? ptStride : nodeStride, sB = tB < nPts ? ptStride : nodeStride;
#pragma unroll 1
            for (int nt = 0; nt < SeedTile<S>::kTiles; ++nt) {
                // digit products by order; o4, o5, o6 are 2^22 times those with a
                // fourth or fifth digit.  Issued so that a sum's products are apart.
                float o0[4], o1[4], o2[4], o3[4], o4[4], o5[4], o6[4];
                {
                    uint4 B[5];
#pragma unroll
                    for (int d = 0; d < 5; ++d) B[d] = sm.b[d][nt][lane];
                    mma_f16_first(o2, A[0][0], B[2].x, B[2].y);
                    mma_f16_first(o3, A[1][0], B[2].x, B[2].y);
                    mma_f16_first(o4, A[0][0], B[3].x, B[3].y);
                    mma_f16_first(o5, A[1][0], B[3].x, B[3].y);
                    mma_f16_first(o6, A[0][0], B[4].x, B[4].y);
                    mma_f16_first(o1, A[1][0], B[0].x, B[0].y);
                    mma_f16_first(o0, A[0][0], B[0].x, B[0].y);
                    mma_f16(o2, A[1][0], B[1].x, B[1].y);
                    mma_f16(o3, A[2][0], B[1].x, B[1].y);
                    mma_f16(o4, A[3][0], B[0].x, B[0].y);
                    mma_f16(o5, A[3][0], B[1].x, B[1].y);
                    mma_f16(o2, A[2][0], B[0].x, B[0].y);
                    mma_f16(o3, A[2][0], B[2].x, B[2].y);
                    mma_f16(o4, A[4][0], B[0].x, B[0].y);
                    mma_f16(o2, A[0][1], B[2].z, B[2].w);
                    mma_f16(o3, A[1][1], B[2].z, B[2].w);
                    mma_f16(o4, A[0][1], B[3].z, B[3].w);
                    mma_f16(o5, A[1][1], B[3].z, B[3].w);
                    mma_f16(o6, A[0][1], B[4].z, B[4].w);
                    mma_f16(o1, A[1][1], B[0].z, B[0].w);
                    mma_f16(o0, A[0][1], B[0].z, B[0].w);
                    mma_f16(o2, A[1][1], B[1].z, B[1].w);
                    mma_f16(o3, A[2][1], B[1].z, B[1].w);
                    mma_f16(o4, A[3][1], B[0].z, B[0].w);
                    mma_f16(o5, A[3][1], B[1].z, B[1].w);
                    mma_f16(o2, A[2][1], B[0].z, B[0].w);
                    mma_f16(o3, A[2][1], B[2].z, B[2].w);
                    mma_f16(o4, A[4][1], B[0].z, B[0].w);
                    if (!heavy) {
                        mma_f16(o1, A[0][0], B[1].x, B[1].y);
                        mma_f16(o1, A[0][1], B[1].z, B[1].w);
                    } else {
                        // eight nodes at a time, each sum exact, added with the errors
                        // of the additions kept in the fourth order
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float part[4];
                            mma_f16_first(part, A[0][i >> 1], i & 1 ? 0u : (i & 2 ? B[1].z : B[1].x),
                                          i & 1 ? (i & 2 ? B[1].w : B[1].y) : 0u);
#pragma unroll
                            for (int j = 0; j < 4; ++j) {
                                float e;
                                two_sum(o1[j], part[j], o1[j], e);
                                o3[j] += e;
                            }
                        }
                    }
                }
                const float2 rel = *reinterpret_cast<const float2 *>(sm.rel[nt][t]);
                const int2 off = *reinterpret_cast<const int2 *>(sm.off[nt][t]);
                const int s0 = 2 * nt / 3, a0 = 2 * nt - 3 * s0, s1 = (2 * nt + 1) / 3, a1 = 2 * nt + 1 - 3 * s1;
                float2 H[2], Lo[2];
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    // o0 + o1 + o2 + o3 + 2^-22 (o4 + o5 + o6), components 2 nt and 2 nt + 1 as
                    // a pair.  o0 is a multiple of 64, o0 + o1 of 2^-5, o1 and o2 are below
                    // 2^24 of that: the three-operation sums are exact
                    const auto pair = [&](const float (&o)[4]) { return make_float2(o[2 * r], o[2 * r + 1]); };
                    float2 w = pair(o0), low = add2(pair(o4), add2(pair(o5), pair(o6)));
                    low = fma2(low, dup2(1.0f / 4194304.0f), pair(o3));
                    const auto add = [&](const float2 p) {
                        const float2 u = add2(w, p);
                        low = add2(low, sub2(p, sub2(u, w)));
                        w = u;
                    };
                    add(pair(o1));
                    add(pair(o2));
                    const float2 mh = add2(w, low), ml = sub2(low, sub2(mh, w));
                    // about the term's position: r - X = (r - O) + (O - X)
                    const dfl ox = r ? xB : xA;
                    const float2 zh = mul2(make_float2(__shfl_sync(kFull, mh.x, lane & ~3), __shfl_sync(kFull, mh.y, lane & ~3)), rel);
                    const float2 zl = mul2(make_float2(__shfl_sync(kFull, ml.x, lane & ~3), __shfl_sync(kFull, ml.y, lane & ~3)), rel);
                    const float2 p = mul2(zh, dup2(ox.h));
                    const float2 pl = fma2(zl, dup2(ox.h), fma2(zh, dup2(ox.l), fms2(zh, dup2(ox.h), p)));
                    float2 s, e;
                    two_sum2(mh, p, s, e);
                    e = add2(e, add2(ml, pl));
                    H[r] = add2(s, e);
                    Lo[r] = sub2(e, sub2(H[r], s));
                }
                double val[2][2];
                bool odd = false;
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    val[r][0] = join_bits(H[r].x, Lo[r].x, off.x);
                    val[r][1] = join_bits(H[r].y, Lo[r].y, off.y);
                    odd |= (odd_range(H[r].x, lim) && H[r].x != 0.f) || (odd_range(H[r].y, lim) && H[r].y != 0.f);
                }
                if (odd) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        val[r][0] = join_odd(H[r].x, Lo[r].x, off.x);
                        val[r][1] = join_odd(H[r].y, Lo[r].y, off.y);
                    }
                }
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    double *d = r ? dB : dA;
                    const int64_t stride = r ? sB : sA;
                    if (H[r].x != 0.f) atomicAdd(d + s0 * stride + 4 * a0, val[r][0]);
                    if ((S % 2 == 0 || 2 * nt + 1 < 3 * S) && H[r].y != 0.f) atomicAdd(d + s1 * stride + 4 * a1, val[r][1]);
                }
            }
        }
        __syncwarp();
    }
}

// Denominators from the five digits of each unit's weights, in their scaled
// units: products with ones, every order exact in its FP32 accumulator (first
// digits sum below 2^14 in eights, the others below 2^24 of their grid).
__global__ void __launch_bounds__(128) k_tile_den(int64_t nVol, int nLoop, TileLists lists, unsigned nUnits, double *part) {
    const unsigned unit = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (unit >= nUnits) return;  // whole warps only
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int64_t e0 = lists.offs[unit];
    const int n = int((lists.offs[unit + 1] - e0) / kTileTerms);
    const uint4 *dig = lists.dig + 192 * (e0 / kTileTerms) + lane, *dig3 = lists.dig3 + 64 * (e0 / kTileTerms) + lane,
                *dig4 = lists.dig4 + 64 * (e0 / kTileTerms) + lane;
    const unsigned ones = g == 0 ? 0x3c003c00u : 0u;
    float acc[5][2][4] = {};
#pragma unroll 2
    for (int st = 0; st < n; ++st)
#pragma unroll
        for (int m = 0; m < 2; ++m) {
#pragma unroll
            for (int d = 0; d < 3; ++d) mma_f16(acc[d][m], __ldcs(dig + 192 * int64_t(st) + 32 * (2 * d + m)), ones, ones);
            mma_f16(acc[3][m], __ldcs(dig3 + 64 * int64_t(st) + 32 * m), ones, ones);
            mma_f16(acc[4][m], __ldcs(dig4 + 64 * int64_t(st) + 32 * m), ones, ones);
        }
    if (t) return;
    const int64_t group = unit / unsigned(nLoop);
    const int kk = int(unit - unsigned(group) * unsigned(nLoop));
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const int64_t slot = group * 32 + 16 * m + g + 8 * r;
            if (slot < nVol)
                part[kk * nVol + slot] = (double(acc[0][m][2 * r]) + double(acc[1][m][2 * r])) +
                                         (double(acc[2][m][2 * r]) + (double(acc[3][m][2 * r]) + double(acc[4][m][2 * r])) / 4194304.0);
        }
}

__global__ void k_tile_den_inv(int64_t nVol, int nLoop, const double *part, double *denInv) {
    const int64_t slot = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (slot >= nVol) return;
    double d = 0.0;
    for (int kk = 0; kk < nLoop; ++kk) d += part[kk * nVol + slot];
    denInv[slot] = 1.0 / d;
}

template <int S>
void launch_seeds(const VolumeDev &v, const WalkRecF &rec, const MixedParams &mp, const TileDev &td,
                  const TileLists &lists, int nPts, unsigned nUnits, const double *denInv, const double *dxv,
                  int64_t dxvStride, double *ptAdj, int64_t ptStride, double *nodeAdj,
                  int64_t nodeStride, cudaStream_t st) {
    constexpr int warps = kAdjWarps;
    const int sms = tile_sms(), nb = int(min(int64_t(sms), (int64_t(nUnits) + warps - 1) / warps));
    const unsigned chunk = unsigned(max(int64_t(1), min(int64_t(32), int64_t(nUnits) / (4 * sms * warps))));
    const size_t smem = warps * sizeof(SeedTile<S>);
    cudaMemsetAsync(td.counter, 0, sizeof(unsigned), st);
    cudaFuncSetAttribute(k_tile_adjoint<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    k_tile_adjoint<S><<<nb, 32 * warps, smem, st>>>(v, rec, mp, td, lists, nPts, nUnits, chunk, denInv, dxv,
                                                    dxvStride, ptAdj, ptStride, nodeAdj, nodeStride);
}

}  // namespace

void launch_tile_den_inv(int64_t nVol, int nLoop, const TileLists &lists, double *part, double *denInv,
                         cudaStream_t st) {
    if (nVol <= 0) return;
    const int64_t units = walk_list_warps(nVol) * nLoop;
    k_tile_den<<<int((32 * units + 127) / 128), 128, 0, st>>>(nVol, nLoop, lists, unsigned(units), part);
    k_tile_den_inv<<<int((nVol + 127) / 128), 128, 0, st>>>(nVol, nLoop, part, denInv);
}

void launch_tile_adjoint(const VolumeDev &v, const WalkRecF &rec, const EvalConsts &k, const TileDev &td,
                         const TileLists &lists, int nPts, int nNodes, const double *denInv, const double *dxv,
                         int nSeeds, int64_t dxvStride, double *ptAdj, double *nodeAdj, unsigned long long *counters,
                         cudaStream_t st) {
    if (nSeeds <= 0 || v.nVol <= 0) return;
    const MixedParams mp = make_mixed_params(k);
    const unsigned nUnits = unsigned(walk_list_warps(v.nVol) * mp.nLoop);
    const int64_t ptStride = 12 * int64_t(nPts), nodeStride = 12 * int64_t(nNodes);
    // the work is counted as the other forms count it: once per group of 16, 4 or 1 seeds
    for (int i = nSeeds / 16 + (nSeeds % 16) / 4 + nSeeds % 4; i > 0; --i)
        launch_add_walk_counters(counters, lists.counters, st);
    for (int s = 0; s < nSeeds;) {
        const double *d = dxv + s * dxvStride;
        double *pa = ptAdj + s * ptStride, *na = nodeAdj + s * nodeStride;
        if (nSeeds - s >= kAdjSeeds) {
            launch_seeds<kAdjSeeds>(v, rec, mp, td, lists, nPts, nUnits, denInv, d, dxvStride, pa, ptStride, na,
                                    nodeStride, st);
            s += kAdjSeeds;
        } else {
            launch_seeds<1>(v, rec, mp, td, lists, nPts, nUnits, denInv, d, dxvStride, pa, ptStride, na, nodeStride,
                            st);
            s += 1;
        }
    }
}

}  // namespace idw
