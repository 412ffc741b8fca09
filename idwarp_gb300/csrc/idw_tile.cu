// Tile walks: the fast-mode forward sums of the default exponents (3, 5) as
// tensor-core products (evalNode, src/modules/kd_tree.F90:619-713, driven by
// warpMesh, src/warp/warpMesh.F90:46-71).
//
// Every term of a node's sums is w (D' r + e), a weight times a motion that is
// linear in the volume point, so the numerators are sum_t w_t D'_t (applied to
// r once, at the end) and sum_t w_t e_t: a product of the weights (32 nodes x
// terms) with the terms' motions (terms x 12) and a column of ones for the
// denominator.  The weights depend on set-up state and the weight law only, so
// they are formed once per mesh, in double-float, and kept as four FP16 digits in
// operand layout (8 bytes per node and term); a walk streams them and multiplies
// them with the motions' four.  The leading products sum exactly in the FP32
// accumulators and the next ones in compensated pairs, so the sums carry about 2^-44
// of the denominator and the largest motion; no term needs a second evaluation,
// however large its weight.  Three digits of both are a quarter less to stream
// (245k-node wing 235 against 258 us, 8M nodes 5.9 against 7.3 ms), but then the nodes
// beside the surface, which one term carries, and the far field are 1e-10 of the
// largest motion off where the double-float terms of the gated walk leave 1e-14.
//
// The terms are those of the reference's decisions (decide32 + resolve64, as
// k_walk_record), recorded once per den0, errTol and law.  With walkLists off a walk
// makes lists and digits for a run of groups at a time; both give the same bits.
#include <climits>
#include <type_traits>

#include <cub/cub.cuh>

#include "idw_tile.cuh"
#include "idwarp_gb300.h"

namespace idw {

namespace {

constexpr int kScaleExp = 13;   // node denominators are scaled to [2^13, 2^14)
constexpr int kMotExp = 14;     // motions are scaled to at most 2^14
inline int blocks(int64_t n, int b) { return int((n + b - 1) / b); }

// ---- set-up: node order, term geometry, scales, lists, digits ----

// Hilbert index (21 bits per axis, on a cube) of every walk slot's point: the
// groups of 32 consecutive nodes share more of their terms than on the Morton
// curve (21.4 against 20 of 32 nodes active per term on the 2M-node wing).
// The transform is J. Skilling's (AIP Conf. Proc. 707, 2004).
__global__ void k_tile_curve(VolumeDev v, double lo0, double lo1, double lo2, double scale, unsigned long long *codes,
                             int *idx) {
    const int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= v.nVol) return;
    const double *x = v.xv0 + 3 * int64_t(v.perm[i]);
    const double f[3] = {(x[0] - lo0) * scale, (x[1] - lo1) * scale, (x[2] - lo2) * scale};
    unsigned X[3];
    for (int k = 0; k < 3; ++k) X[k] = unsigned(fmin(fmax(f[k], 0.0), 2097151.0));
    for (unsigned Q = 1u << 20; Q > 1u; Q >>= 1) {
        const unsigned P = Q - 1u;
        for (int k = 0; k < 3; ++k) {
            if (X[k] & Q) {
                X[0] ^= P;
            } else {
                const unsigned t = (X[0] ^ X[k]) & P;
                X[0] ^= t;
                X[k] ^= t;
            }
        }
    }
    X[1] ^= X[0];
    X[2] ^= X[1];
    unsigned t = 0u;
    for (unsigned Q = 1u << 20; Q > 1u; Q >>= 1)
        if (X[2] & Q) t ^= Q - 1u;
    unsigned long long code = 0ull;
    for (int b = 20; b >= 0; --b)
        for (int k = 0; k < 3; ++k) code = (code << 1) | (((X[k] ^ t) >> b) & 1u);
    codes[i] = code;
    idx[i] = int(i);
}

// Geometry of every term: points, then tree nodes (their centroids); areas
// scaled by 2^areaExp (the largest is then near one).
__global__ void k_tile_geo(TreeDev t, int nPts, const dbl4 *xa, int areaExp, float4 *geo) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nPts + t.nNodes) return;
    const dbl4 p = i < nPts ? xa[i] : t.geom[i - nPts];
    const double v[4] = {p.x, p.y, p.z, ldexp(i < nPts ? p.w : t.ai[i - nPts], areaExp)};
    float h[4], l[4];
    for (int c = 0; c < 4; ++c) {
        h[c] = float(v[c]);
        l[c] = float(v[c] - double(h[c]));
    }
    geo[2 * int64_t(i)] = make_float4(h[0], h[1], h[2], h[3]);
    geo[2 * int64_t(i) + 1] = make_float4(l[0], l[1], l[2], l[3]);
}

// The traversal of one unit: emit(first, n, mask) for the n points of every leaf that
// a lane sums and (n = 1) every cluster that a lane approximates, in preorder, with
// the decisions of k_walk_record.  slot: the lane's walk slot (group 32 + lane).
template <class F>
__device__ __forceinline__ void decide_group(const TreeDev &t, const TreeDevF &tf, const VolumeDev &v,
                                             const WalkRecF &rec, const MixedParams &mp, const TileDev &td,
                                             int64_t slot, int kk, MixedCounters &cnt, unsigned long long *counters,
                                             F &&emit) {
    const bool valid = slot < v.nVol;
    const int64_t g = td.order[valid ? slot : 0];
    const float tauf = mp.errTolF * rec.hi[g].w;
    const float4 rhi = rec.hi[kk * v.nVol + g], rlo = rec.lo[kk * v.nVol + g];
    const float rh[3] = {rhi.x, rhi.y, rhi.z}, rl[3] = {rlo.x, rlo.y, rlo.z};
    int node = 0, skip = 0;
    while (node < t.nNodes) {
        const int4 inf = ldgi4(&tf.nodes[node].info);
        const bool active = valid && node >= skip;
        if (inf.w) {
            const unsigned m = __ballot_sync(kFull, active);
            if (m) emit(inf.x, inf.y - inf.x + 1, m);
            if (active) {
                cnt.leafPairs += inf.y - inf.x + 1;
                cnt.visited++;
            }
            node = inf.z;
        } else {
            int dec = 0;
            float rho0, rho1, rho2, d2, rs, wA;
            if (active) {
                cnt.visited++;
                dec = decide32(tf, node, rh, rl, tauf, rho0, rho1, rho2, d2, rs, wA);
            }
            dec = resolve64(dec, t, v, g, node, rh, rl, mp.errTol, counters);
            const unsigned m = __ballot_sync(kFull, dec == 1);
            if (m) emit(tf.nPts + node, 1, m);
            bool open = false;
            if (dec == 1) {
                skip = inf.z;
                cnt.approx++;
            } else if (active) {
                open = true;
            }
            node = __any_sync(kFull, open) ? node + 1 : inf.z;
        }
    }
}

// First guess of a node's weight scale (log2), from the estimate: den0 2^(5s) ~ 1.
__device__ __forceinline__ int first_scale(const WalkRecF &rec, int64_t gid, int lawExp) {
    return max(-110, min(110, 5 * __float_as_int(rec.lo[gid].w) + lawExp));
}

// One term's part of a node's FP32 denominator under the weight scale P.
__device__ __forceinline__ float add_den(float den, const float4 *geo, int term, int nPts, const float4 &rhi,
                                         const float4 &rlo, float P, const TileLaw &law) {
    const float4 c = ldgf4(geo + 2 * int64_t(term)), d = ldgf4(geo + 2 * int64_t(term) + 1);
    const float dx = (rhi.x - c.x) + (rlo.x - d.x), dy = (rhi.y - c.y) + (rlo.y - d.y),
                dz = (rhi.z - c.z) + (rlo.z - d.z);
    const float y = rsqrt_normal(fmaf(dx, dx, fmaf(dy, dy, fmaf(dz, dz, term < nPts ? 1e-15f : 0.f))));
    const float y2 = y * y;
    return fmaf(c.w * (y2 * (y * P)), fmaf(law.kh, y2, 1.0f), den);
}

// List lengths (whole steps) of every unit, a warp each, into counts.  DEN: also the
// unit's share of its nodes' FP32 denominators under the first guess into part
// (nLoop x nVol), as k_tile_part has it from the lists.
template <bool DEN>
__global__ void __launch_bounds__(128, 8)
    k_tile_count(TreeDev t, TreeDevF tf, VolumeDev v, WalkRecF rec, MixedParams mp, TileDev td, TileLaw law,
                 int lawExp, int64_t nGroups, int64_t *counts, float *part) {
    const int64_t unit = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t group = unit / mp.nLoop;
    if (group >= nGroups) return;  // whole warps only
    const int kk = int(unit - group * mp.nLoop), lane = threadIdx.x & 31;
    const int64_t slot = 32 * group + lane, gid = td.order[min(slot, v.nVol - 1)];
    const float P = DEN ? pow2f(first_scale(rec, gid, lawExp)) : 0.f;
    float den = 0.f;
    MixedCounters cnt;
    const float4 rhi = rec.hi[kk * v.nVol + gid], rlo = rec.lo[kk * v.nVol + gid];
    int n = 0;
    decide_group(t, tf, v, rec, mp, td, slot, kk, cnt, nullptr, [&](int first, int k, unsigned m) {
        n += k;
        if constexpr (DEN) {
            if ((m >> lane) & 1u)
                for (int i = first; i < first + k; ++i) den = add_den(den, td.geo, i, tf.nPts, rhi, rlo, P, law);
        }
    });
    if (lane == 0) counts[unit] = int64_t(n + kTileTerms - 1) / kTileTerms * kTileTerms;
    if (DEN && slot < v.nVol) part[kk * v.nVol + slot] = den;
}

// The units' shares of the FP32 denominators from the recorded lists, added in the
// order of the traversal: a new weight law needs no traversal (8M-node wing, the warp
// after a new alpha 38.5 -> 29.1 ms), and the first count does without them (2M nodes
// 3.5 -> 2.25 + 1.1 ms).
__global__ void __launch_bounds__(128)
    k_tile_part(VolumeDev v, WalkRecF rec, MixedParams mp, TileDev td, TileLists lists, TileLaw law, int lawExp,
                int nPts, int64_t nUnits, float *part) {
    const int64_t unit = (int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    if (unit >= nUnits) return;  // whole warps only
    const int64_t group = unit / mp.nLoop;
    const int kk = int(unit - group * mp.nLoop), lane = threadIdx.x & 31;
    const int64_t slot = 32 * group + lane, gid = td.order[min(slot, v.nVol - 1)];
    const float P = pow2f(first_scale(rec, gid, lawExp));
    const float4 rhi = rec.hi[kk * v.nVol + gid], rlo = rec.lo[kk * v.nVol + gid];
    float den = 0.f;
    const int64_t e1 = lists.offs[unit + 1];
    for (int64_t e = lists.offs[unit]; e < e1; e += kTileTerms) {
        const int term = lists.term[e + (lane & 15)];
        const unsigned mask = lists.mask[e + (lane & 15)];
#pragma unroll 8
        for (int k = 0; k < kTileTerms; ++k) {
            const float d = add_den(den, td.geo, __shfl_sync(kFull, term, k), nPts, rhi, rlo, P, law);
            den = (__shfl_sync(kFull, mask, k) >> lane) & 1u ? d : den;
        }
    }
    if (slot < v.nVol) part[kk * v.nVol + slot] = den;
}

// Each node's weight scale: the power of two that brings its denominator to
// [2^13, 2^14).  A node whose denominator is not a positive normal number, or
// whose scale leaves the range, raises bad (the gated walk then serves the mesh).
__global__ void k_tile_scale(VolumeDev v, WalkRecF rec, TileDev td, int nLoop, int lawExp, const float *part,
                             float *scale, int *bad) {
    const int64_t slot = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (slot >= v.nVol) return;
    float den = 0.f;
    for (int kk = 0; kk < nLoop; ++kk) den += part[kk * v.nVol + slot];
    const int ex = int((__float_as_uint(den) >> 23) & 0xffu);
    const int k = kScaleExp - (ex - 127) + first_scale(rec, td.order[slot], lawExp);
    const bool ok = den > 0.f && ex > 0 && ex < 255 && k >= -118 && k <= 118;
    if (!ok) *bad = 1;
    scale[slot] = ok ? pow2f(k) : 1.0f;
}

// The lists' entries at offs, padded with empty ones; a warp per unit.
__global__ void __launch_bounds__(128, 8)
    k_tile_record(TreeDev t, TreeDevF tf, VolumeDev v, WalkRecF rec, MixedParams mp, TileDev td, TileRange range,
                  const int64_t *offs, int *term, unsigned *mask, unsigned long long *counters) {
    const int64_t unit = range.group0 * mp.nLoop + ((int64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5);
    const int64_t group = unit / mp.nLoop;
    if (group >= range.group1) return;  // whole warps only
    const int kk = int(unit - group * mp.nLoop), lane = threadIdx.x & 31;
    MixedCounters cnt;
    int64_t pos = offs[unit] - range.entry0;
    const int64_t end = offs[unit + 1] - range.entry0;
    decide_group(t, tf, v, rec, mp, td, 32 * group + lane, kk, cnt, counters, [&](int first, int n, unsigned m) {
        for (int i = lane; i < n; i += 32) {
            term[pos + i] = first + i;
            mask[pos + i] = m;
        }
        pos += n;
    });
    if (pos + lane < end) {
        term[pos + lane] = 0;
        mask[pos + lane] = 0u;
    }
    cnt.flush(counters);
}

// The row pairs of a unit's nodes, for stage_weights; slots past the end take
// the last node (their mask bits are never set).
__device__ __forceinline__ void unit_rows(TileRows *rows, const VolumeDev &v, const WalkRecF &rec, const TileDev &td,
                                          int64_t group, int kk) {
    const int lane = threadIdx.x & 31;
    const int64_t slot = min(group * 32 + lane, v.nVol - 1);
    const int64_t gid = kk * v.nVol + td.order[slot];
    const float4 hi = rec.hi[gid], lo = rec.lo[gid];
    const float h[3] = {hi.x, hi.y, hi.z}, l[3] = {lo.x, lo.y, lo.z}, P = td.scale[slot];
    TileRows &R = rows[8 * (lane >> 4) + (lane & 7)];
    const bool up = lane & 8;
    __syncwarp();
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        (up ? R.h[c].y : R.h[c].x) = h[c];
        (up ? R.l[c].y : R.l[c].x) = l[c];
    }
    (up ? R.P.y : R.P.x) = P;
    __syncwarp();
}

// The digits of every list entry's weights: the first four, or FIFTH the fifth
// (into dig3).
template <bool FIFTH>
__global__ void __launch_bounds__(128)
    k_tile_build(VolumeDev v, WalkRecF rec, MixedParams mp, TileDev td, TileLists lists, TileLaw law, int nPts,
                 TileRange range, int64_t listEntry0, uint4 *dig, uint4 *dig3) {
    __shared__ __align__(16) TileStage stage[4];
    __shared__ TileRows rows[4][16];
    const int64_t unit = range.group0 * mp.nLoop + ((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (unit >= range.group1 * mp.nLoop) return;  // whole warps only
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    TileStage &st = stage[warp];
    unit_rows(rows[warp], v, rec, td, unit / mp.nLoop, int(unit % mp.nLoop));
    const int64_t e1 = lists.offs[unit + 1] - range.entry0;
    for (int64_t e = lists.offs[unit] - range.entry0; e < e1; e += kTileTerms) {
        if (lane < kTileTerms) {
            st.term[lane] = lists.term[listEntry0 + e + lane];
            st.mask[lane] = lists.mask[listEntry0 + e + lane];
        }
        __syncwarp();
        stage_weights<FIFTH>(st, td.geo, nPts, rows[warp], law);
        __syncwarp();
        const int64_t step = e / kTileTerms;
        const uint4 *src = &st.dig[0][0][0];
        if constexpr (!FIFTH) {
#pragma unroll
            for (int c = 0; c < 6; ++c) dig[192 * step + 32 * c + lane] = src[32 * c + lane];
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) dig3[64 * step + 32 * c + lane] = src[(FIFTH ? 0 : 192) + 32 * c + lane];
        __syncwarp();
    }
}

// ---- motions of the current surface ----

// Column pair g of a term's motion about the root centroid O: (D'_a0, D'_a2)
// for g = 2a, (D'_a1, e_a) for g = 2a + 1, with D' = M - I - Dref and
// e = D' O + b - bref (a tangent's M, ident = 0, has no I); (8, 0) for g = 6 (8 times the denominator, on the grid
// of the first digits), zero for g = 7.
__device__ __forceinline__ void motion_pair(const double *mb, const double *root, const dbl4 o, int g, int ident,
                                            double &u, double &w) {
    u = g == 6 ? 8.0 : 0.0;
    w = 0.0;
    if (g >= 6) return;
    const int a = g >> 1;
    double D[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double id = ident && a == k ? 1.0 : 0.0;
        D[k] = mb[3 * a + k] - id - (root ? root[3 * a + k] - id : 0.0);
    }
    if (!(g & 1)) {
        u = D[0];
        w = D[2];
        return;
    }
    u = D[1];
    w = D[0] * o.x + D[1] * o.y + D[2] * o.z + (mb[9 + a] - (root ? root[9 + a] : 0.0));
}

// Exponent that brings a column of largest magnitude max (float bits) to at
// most 2^14.
__device__ __forceinline__ int column_exp(unsigned maxBits) {
    if (maxBits == 0u) return 0;
    return max(-110, min(110, kMotExp - 1 - (int(maxBits >> 23) - 127)));
}

// Largest magnitude of each column over the terms (float bits; column 4a + k,
// k = 3 the offset e).  Leaves have no motion of their own: their points do.
__global__ void k_tile_max(TreeDev t, int nPts, const double *ptMB, const double *nodeMB, int ident, unsigned *colMax) {
    __shared__ unsigned sm[12];
    if (threadIdx.x < 12) sm[threadIdx.x] = 0u;
    __syncthreads();
    const int64_t tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t i = tid >> 3;
    const int g = int(tid & 7);
    if (i < nPts + t.nNodes && g < 6 && !(i >= nPts && t.info[i - nPts].w)) {
        const double *root = t.info[0].w ? nullptr : nodeMB;
        double u, w;
        motion_pair(i < nPts ? ptMB + 12 * i : nodeMB + 12 * (i - nPts), root, t.geom[0], g, ident, u, w);
        const int a = g >> 1, odd = g & 1;
        const unsigned fu = __float_as_uint(__double2float_ru(fabs(u))), fw = __float_as_uint(__double2float_ru(fabs(w)));
        if (fu > sm[4 * a + odd]) atomicMax(&sm[4 * a + odd], fu);
        if (fw > sm[4 * a + 2 + odd]) atomicMax(&sm[4 * a + 2 + odd], fw);
    }
    __syncthreads();
    if (threadIdx.x < 12 && sm[threadIdx.x]) atomicMax(colMax + threadIdx.x, sm[threadIdx.x]);
}

// The five FP16 digits of v 2^e, on the grids of the weights' digits.
__device__ __forceinline__ void motion_digits(double v, int e, unsigned (&d)[5]) {
    const double s = v * __hiloint2double((1023 + e) << 20, 0);
    const float f = float(s), lo = float(s - double(f));
    const float M[3] = {1.5f * 67108864.0f, 1.5f * 32768.0f, 1.5f * 16.0f};
    float r = f, rest = 0.f;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float g = __fsub_rn(__fadd_rn(r, M[k]), M[k]);
        d[k] = __half_as_ushort(__float2half_rn(g));
        r = __fsub_rn(r, g);
        if (k == 1) two_sum(r, lo, r, rest);
    }
    r *= 4194304.0f;
    const __half q = __float2half_rn(r);
    d[3] = __half_as_ushort(q);
    d[4] = __half_as_ushort(__float2half_rn(fmaf(rest, 4194304.0f, r - __half2float(q))));
}

// Motion records: per term 8 x 16 bytes, lane row g's digits of its two
// columns.  Thread 0 also stores the reference motion (Dref 9, bref 3; high
// parts, then low parts) that the finalisation adds back.  mot5: a tangent's
// fifth digits, 8 words a term (null: a surface).
__global__ void k_tile_mot(TreeDev t, int nPts, const double *ptMB, const double *nodeMB, const unsigned *colMax,
                           uint4 *mot, unsigned *mot5, float *refDB) {
    const int64_t tid = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t i = tid >> 3;
    const int g = int(tid & 7);
    if (i >= nPts + t.nNodes) return;
    const double *root = t.info[0].w ? nullptr : nodeMB;
    const int ident = mot5 == nullptr;
    if (tid < 12) {
        const int c = int(tid);
        const double v = root ? root[c] - (ident && c < 9 && c % 4 == 0 ? 1.0 : 0.0) : 0.0;
        refDB[c] = float(v);
        refDB[12 + c] = float(v - double(float(v)));
    }
    unsigned du[5] = {0, 0, 0, 0, 0}, dw[5] = {0, 0, 0, 0, 0};
    if (!(i >= nPts && t.info[i - nPts].w)) {
        double u, w;
        motion_pair(i < nPts ? ptMB + 12 * i : nodeMB + 12 * (i - nPts), root, t.geom[0], g, ident, u, w);
        const int a = g >> 1, odd = g & 1;
        motion_digits(u, g < 6 ? column_exp(colMax[4 * a + odd]) : 0, du);
        if (g < 6) motion_digits(w, column_exp(colMax[4 * a + 2 + odd]), dw);
    }
    mot[8 * i + g] = make_uint4(du[0] | (du[1] << 16), du[2] | (du[3] << 16), dw[0] | (dw[1] << 16), dw[2] | (dw[3] << 16));
    if (mot5) mot5[8 * i + g] = du[4] | (dw[4] << 16);
}

// ---- the walk ----

// Warps of a block (one block per SM): 16 at 128 registers, where a walk waits for
// its copies (three digits, 245k-node wing, 243 -> 236 us against 12 warps at 144
// registers); a tangent needs 166 registers.  Two surfaces sharing a step's digits,
// at 12 or 10 warps, spill beside four digits: eight surfaces on the 2M-node wing 17.0
// and 16.3 ms against 13.9 one at a time.
constexpr int tile_warps(int nd) { return nd < 5 ? 16 : 12; }
// Shared memory of a stage: nd digits and the motions (a tangent's fifth digits
// last).
constexpr size_t tile_stage_bytes(int nd) { return sizeof(uint4) * ((nd == 5 ? 10 : 8) * kTileTerms + 64 * nd); }

// The sums of one unit per warp: numerators about the reference motion and
// denominator of each node, as pairs (high, low), into out.  The weight digits
// stream from memory, the next step's copied while one is computed.  ND: 4, or 5
// for a tangent.
template <int ND>
__global__ void __launch_bounds__(32 * tile_warps(ND), 1)
    k_tile_walk(TreeDev t, TreeDevF tf, VolumeDev v, WalkRecF rec, MixedParams mp, TileDev td, TileLists lists,
                TileRange range, unsigned chunk, float4 *out) {
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ unsigned long long qstate;
    if (threadIdx.x == 0) qstate = 0ull;
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, a = lane & 3;
    constexpr size_t stageBytes = tile_stage_bytes(ND);
    unsigned char *mine = smraw + 2 * stageBytes * (threadIdx.x >> 5);
    auto motions = [&](int s) { return reinterpret_cast<uint4 *>(mine + stageBytes * (s & 1)); };
    auto digits = [&](int s) { return motions(s) + 8 * kTileTerms; };
    UnitQueue queue = {&qstate, td.counter, unsigned((range.group1 - range.group0) * mp.nLoop), chunk, 0u, 0u};
    unsigned idx;
    while (queue.next(idx)) {
        const int64_t group = range.group0 + idx / unsigned(mp.nLoop);
        const int kk = int(idx % unsigned(mp.nLoop));
        const int64_t unit = group * mp.nLoop + kk;
        TileAcc<ND> acc;
        tile_zero(acc);
        const int64_t e0 = lists.offs[unit] - range.entry0;
        const int n = int((lists.offs[unit + 1] - range.entry0 - e0) / kTileTerms);
        const int *term = lists.term + e0;
        const uint4 *dig = lists.dig + 192 * (e0 / kTileTerms), *dig3 = lists.dig3 + 64 * (e0 / kTileTerms);
        const uint4 *dig4 = ND == 5 ? lists.dig4 + 64 * (e0 / kTileTerms) : nullptr;
        StageIds ids;
        int id5 = 0;  // a tangent: the term whose fifth digits the lane copies half of
        auto issue = [&](int s) {
            uint4 *dst = digits(s);
#pragma unroll
            for (int c = 0; c < 6; ++c) cp_async16(dst + 32 * c + lane, dig + 192 * int64_t(s) + 32 * c + lane);
#pragma unroll
            for (int c = 0; c < 2; ++c) cp_async16(dst + 192 + 32 * c + lane, dig3 + 64 * int64_t(s) + 32 * c + lane);
            stage_motions(motions(s), ids, td.mot);
            if constexpr (ND == 5) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
                    cp_async16(dst + 256 + 32 * c + lane, dig4 + 64 * int64_t(s) + 32 * c + lane);
                const int k = lane >> 1;  // term 4 i + j to row 4 i + (i + j) % 4
                cp_async16_l1(dst + 320 + 2 * ((k & ~3) + ((k + (k >> 2)) & 3)) + (lane & 1),
                              reinterpret_cast<const uint4 *>(td.mot5) + 2 * int64_t(id5) + (lane & 1));
                if (s + 1 < n) id5 = term[kTileTerms * (s + 1) + (lane >> 1)];
            }
            if (s + 1 < n) ids = stage_ids(term + kTileTerms * (s + 1));
        };
        if (n > 0) {
            if constexpr (ND == 5) id5 = term[lane >> 1];
            ids = stage_ids(term);
            issue(0);
        }
        cp_async_commit();
        for (int s = 0; s < n; ++s) {
            if (s + 1 < n) issue(s + 1);
            cp_async_commit();
            cp_async_wait<1>();
            __syncwarp();
            if constexpr (ND == 5)
                tile_step5(digits(s), motions(s), reinterpret_cast<const unsigned *>(digits(s) + 320), acc);
            else
                tile_step(digits(s), motions(s), acc);
            __syncwarp();
        }
        cp_async_wait<0>();
        // component a of the numerator: D'_a . (r - O) + e_a; lane column 3: the denominator
        const float4 oh = ldgf4(td.geo + 2 * int64_t(tf.nPts)), ol = ldgf4(td.geo + 2 * int64_t(tf.nPts) + 1);
        float cs[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
            cs[k] = a < 3 ? pow2f(-column_exp(__ldg(td.colMax + 4 * a + k))) : 0.125f;
        float *o = reinterpret_cast<float *>(out);
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int64_t slot = group * 32 + g + 16 * m + 8 * r;
                if (slot >= v.nVol) continue;
                dfl M[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    // columns in the order of the motion records: D'_a0, D'_a1 | D'_a2, e_a
                    float s, low;
                    tile_total(acc, m, k >> 1, r, k & 1, s, low);
                    M[k] = df_norm(s * cs[k], low * cs[k]);
                }
                const int64_t gid = kk * v.nVol + td.order[slot];
                const float4 hi = rec.hi[gid], lo = rec.lo[gid];
                const float h[3] = {hi.x, hi.y, hi.z}, l[3] = {lo.x, lo.y, lo.z};
                const float oh3[3] = {oh.x, oh.y, oh.z}, ol3[3] = {ol.x, ol.y, ol.z};
                dfl s = M[3];
#pragma unroll
                for (int k = 0; k < 3; ++k) {
                    dfl x;
                    two_diff(h[k], oh3[k], x.h, x.l);
                    x.l += l[k] - ol3[k];
                    s = df_add(s, df_mul(M[k], df_norm(x.h, x.l)));
                }
                if (a == 3) s = M[0];
                float *p = o + 8 * (kk * v.nVol + slot);
                p[a] = s.h;
                p[4 + a] = s.l;
            }
    }
}

// The mirrors' sums of each node: reference motion added back, reflected and
// added (finish_mirror); Xv = Xv0 + num / den (a tangent: without Xv0) and the denominator in the reference's units, den L^3 / (P 2^areaExp).
__global__ void k_tile_finalize(VolumeDev v, WalkRecF rec, NodeAggF af, MixedParams mp, TileDev td, const float4 *sums,
                                double denUnit, int tangent, double *xv, double *den) {
    const int64_t slot = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (slot >= v.nVol) return;
    const int64_t gid = td.order[slot];
    float4 S = make_float4(0.f, 0.f, 0.f, 0.f), C = S;
    for (int kk = 0; kk < mp.nLoop; ++kk) {
        const float4 rhi = rec.hi[kk * v.nVol + gid], rlo = rec.lo[kk * v.nVol + gid];
        // A node on a plane is its own image there: it has one sum, so that the parts
        // along the normal cancel and the node stays on the plane to the last bit (the
        // images' steps, and with them the rounding of their sums, differ).
        int image = kk;
        for (int j = 0; j < mp.nSym; ++j) {
            if (!((image >> j) & 1)) continue;
            const int64_t other = (image ^ (1 << j)) * v.nVol + gid;
            const float4 ohi = rec.hi[other], olo = rec.lo[other];
            if (ohi.x == rhi.x && ohi.y == rhi.y && ohi.z == rhi.z && olo.x == rlo.x && olo.y == rlo.y && olo.z == rlo.z)
                image ^= 1 << j;
        }
        const int64_t at = image * v.nVol + slot;
        const float4 h = sums[2 * at], l = sums[2 * at + 1];
        const float rh[3] = {rhi.x, rhi.y, rhi.z}, rl[3] = {rlo.x, rlo.y, rlo.z};
        const float sn[3] = {h.x, h.y, h.z}, cn[3] = {l.x, l.y, l.z};
        finish_mirror(af, mp, kk, rh, rl, sn, cn, h.w, l.w, S, C);
    }
    const int vi = v.perm[gid];
    const dfl D = df_norm(S.w, C.w);
    const float oD = __frcp_rn(D.h);
    const float N[3] = {S.x, S.y, S.z}, Nl[3] = {C.x, C.y, C.z};
    if (xv) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            // quotient of two double-floats: one correction of the FP32 quotient
            const dfl n = df_norm(N[a], Nl[a]);
            const float q = n.h * oD;
            const float rem = fmaf(-q, D.l, fmaf(-q, D.h, n.h) + n.l);
            xv[3 * int64_t(vi) + a] = (tangent ? 0.0 : v.xv0[3 * int64_t(vi) + a]) + (double(q) + double(rem * oD));
        }
    }
    if (den) {
        const int k = int(__float_as_uint(td.scale[slot]) >> 23) - 127;  // P = 2^k
        den[vi] = (double(D.h) + double(D.l)) * denUnit * __hiloint2double((1023 - k) << 20, 0);
    }
}

TileLaw make_tile_law(const EvalConsts &k) {
    const double kappa = k.law.alphaToBexp * k.law.Ldef * k.law.Ldef;
    TileLaw law;
    law.kh = float(kappa);
    law.kl = float(kappa - double(law.kh));
    return law;
}

}  // namespace

int tile_sms() {
    static int cached[16] = {0};
    int dev = 0;
    cudaGetDevice(&dev);
    int &n = cached[dev & 15];
    if (n == 0 && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) n = 1;
    return n;
}

int tile_order(const VolumeDev &v, const double *lo, const double *hi, int *order, TileScratch scratch,
               cudaStream_t st) {
    if (v.nVol <= 0) return 0;
    if (v.nVol > INT_MAX) return -1;
    double ext = 0.0;
    for (int k = 0; k < 3; ++k) ext = hi[k] - lo[k] > ext ? hi[k] - lo[k] : ext;
    const size_t n = size_t(v.nVol);
    auto *codes = static_cast<unsigned long long *>(scratch.take(2 * sizeof(unsigned long long) * n));
    auto *idx = static_cast<int *>(scratch.take(sizeof(int) * n));
    if (!codes || !idx) return -2;
    k_tile_curve<<<blocks(v.nVol, 256), 256, 0, st>>>(v, lo[0], lo[1], lo[2], ext > 0.0 ? 2097151.0 / ext : 0.0, codes,
                                                      idx);
    return sort_morton(v.nVol, codes, idx, codes + v.nVol, order, st, scratch.p, scratch.left);
}

void launch_tile_geo(const TreeDev &t, int nPts, const dbl4 *xa, int areaExp, float4 *geo, cudaStream_t st) {
    k_tile_geo<<<blocks(nPts + t.nNodes, 256), 256, 0, st>>>(t, nPts, xa, areaExp, geo);
}

void launch_tile_motions(const TreeDev &t, int nPts, const double *ptMB, const double *nodeMB, unsigned *colMax,
                         uint4 *mot, unsigned *mot5, float *refDB, cudaStream_t st) {
    const int64_t n = 8 * (int64_t(nPts) + t.nNodes);
    cudaMemsetAsync(colMax, 0, 12 * sizeof(unsigned), st);
    k_tile_max<<<blocks(n, 256), 256, 0, st>>>(t, nPts, ptMB, nodeMB, mot5 == nullptr, colMax);
    k_tile_mot<<<blocks(n, 256), 256, 0, st>>>(t, nPts, ptMB, nodeMB, colMax, mot, mot5, refDB);
}

// den L^-3 2^areaExp 2^(5s) is near one
static int law_exp(const EvalConsts &k, const TileDev &td) { return 3 * ilogb(k.law.Ldef) - td.areaExp; }

int64_t count_tile_lists(const TreeDev &t, const TreeDevF &tf, const VolumeDev &v, const WalkRecF &rec,
                         const EvalConsts &k, const TileDev &td, int64_t *offs, float *part, TileScratch scratch,
                         cudaStream_t st, const std::function<void()> &meanwhile) {
    const MixedParams mp = make_mixed_params(k);
    const int64_t nGroups = walk_list_warps(v.nVol);
    const int64_t n = nGroups * mp.nLoop;
    if (n <= 0) return 0;
    if (n + 1 > int64_t(INT_MAX)) return -1;
    size_t tmpBytes = 0;
    int64_t total = 0;
    auto *counts = static_cast<int64_t *>(scratch.take(sizeof(int64_t) * size_t(n + 1)));
    if (!counts) return -2;
    bool ok = cudaMemsetAsync(counts + n, 0, sizeof(int64_t), st) == cudaSuccess;
    if (ok) {
        (part ? k_tile_count<true> : k_tile_count<false>)<<<blocks(32 * n, 128), 128, 0, st>>>(
            t, tf, v, rec, mp, td, make_tile_law(k), law_exp(k, td), nGroups, counts, part);
        ok = cudaGetLastError() == cudaSuccess;
    }
    if (ok) ok = cub::DeviceScan::ExclusiveSum(nullptr, tmpBytes, counts, offs, int(n + 1), st) == cudaSuccess;
    void *tmp = scratch.take(tmpBytes);
    if (ok && !tmp) return -2;
    if (ok) ok = cub::DeviceScan::ExclusiveSum(tmp, tmpBytes, counts, offs, int(n + 1), st) == cudaSuccess;
    meanwhile();
    if (ok) ok = cudaMemcpyAsync(&total, offs + n, sizeof(int64_t), cudaMemcpyDeviceToHost, st) == cudaSuccess;
    if (cudaStreamSynchronize(st) != cudaSuccess) ok = false;
    return ok ? total : -1;
}

void launch_tile_scales(const VolumeDev &v, const WalkRecF &rec, const EvalConsts &k, const TileDev &td,
                        const TileLists &lists, int nPts, float *part, float *scale, int *bad, cudaStream_t st) {
    if (v.nVol <= 0) return;
    const MixedParams mp = make_mixed_params(k);
    const int64_t n = walk_list_warps(v.nVol) * mp.nLoop;
    cudaMemsetAsync(bad, 0, sizeof(int), st);
    if (lists.term)
        k_tile_part<<<blocks(32 * n, 128), 128, 0, st>>>(v, rec, mp, td, lists, make_tile_law(k), law_exp(k, td), nPts, n,
                                                         part);
    k_tile_scale<<<blocks(v.nVol, 128), 128, 0, st>>>(v, rec, td, mp.nLoop, law_exp(k, td), part, scale, bad);
}

void launch_tile_record(const TreeDev &t, const TreeDevF &tf, const VolumeDev &v, const WalkRecF &rec,
                        const EvalConsts &k, const TileDev &td, const TileRange &range, const int64_t *offs, int *term,
                        unsigned *mask, unsigned long long *counters, cudaStream_t st) {
    const MixedParams mp = make_mixed_params(k);
    const int64_t units = (range.group1 - range.group0) * mp.nLoop;
    if (units > 0)
        k_tile_record<<<blocks(32 * units, 128), 128, 0, st>>>(t, tf, v, rec, mp, td, range, offs, term, mask,
                                                               counters);
}

void launch_tile_build(const VolumeDev &v, const WalkRecF &rec, const EvalConsts &k, const TileDev &td,
                       const TileLists &lists, const TileRange &range, int64_t listEntry0, int nPts, uint4 *dig,
                       uint4 *dig3, cudaStream_t st) {
    const MixedParams mp = make_mixed_params(k);
    const int64_t units = (range.group1 - range.group0) * mp.nLoop;
    if (units <= 0) return;
    (dig ? k_tile_build<false> : k_tile_build<true>)<<<blocks(32 * units, 128), 128, 0, st>>>(
        v, rec, mp, td, lists, make_tile_law(k), nPts, range, listEntry0, dig, dig3);
}

template <int ND>
static void walk_digits(const TreeDev &t, const TreeDevF &tf, const VolumeDev &v, const WalkRecF &rec,
                        const MixedParams &mp, const TileDev &td, const TileLists &lists, const TileRange &range,
                        float4 *sums, cudaStream_t st) {
    constexpr int warps = tile_warps(ND);
    const int64_t units = (range.group1 - range.group0) * mp.nLoop;
    const int sms = tile_sms(), grid = int(min(int64_t(sms), (units + warps - 1) / warps));
    const unsigned chunk = unsigned(max(int64_t(1), min(int64_t(32), units / (4 * sms * warps))));
    const size_t smem = warps * 2 * tile_stage_bytes(ND);
    cudaMemsetAsync(td.counter, 0, sizeof(unsigned), st);
    cudaFuncSetAttribute(k_tile_walk<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(smem));
    k_tile_walk<ND><<<grid, 32 * warps, smem, st>>>(t, tf, v, rec, mp, td, lists, range, chunk, sums);
}

void launch_tile_walk(const TreeDev &t, const TreeDevF &tf, const VolumeDev &v, const WalkRecF &rec,
                      const EvalConsts &k, const TileDev &td, const TileLists &lists, const TileRange &range,
                      float4 *sums, cudaStream_t st) {
    if (range.group1 <= range.group0) return;
    const MixedParams mp = make_mixed_params(k);
    if (lists.dig4) walk_digits<5>(t, tf, v, rec, mp, td, lists, range, sums, st);
    else walk_digits<4>(t, tf, v, rec, mp, td, lists, range, sums, st);
}

void launch_tile_finalize(const VolumeDev &v, const WalkRecF &rec, const EvalConsts &k, const TileDev &td,
                          const float *refDB, const float4 *sums, const WalkOut &o, cudaStream_t st) {
    if (v.nVol <= 0) return;
    const MixedParams mp = make_mixed_params(k);
    const double L = k.law.Ldef;
    NodeAggF af{};
    af.ref = refDB;
    k_tile_finalize<<<blocks(v.nVol, 128), 128, 0, st>>>(v, rec, af, mp, td, sums, ldexp(L * L * L, -td.areaExp),
                                                         o.tangent, o.xv, o.den);
}

}  // namespace idw
