// Matched forward projector: the exact transpose of the voxel-driven
// backprojector in backproject.cu (no counterpart in the reference, which has
// no forward model). The shared-memory backprojector takes the same decisions
// but for rows whose coordinate lies within one unit in the last place of an
// integer (geom.cuh), so against it the transpose holds to that rounding.
//
// The backprojector adds, for every voxel and view,
//     w * [(1-fv)((1-fu) p[v0][u0] + fu p[v0][u0+1]) + fv((1-fu) p[v0+1][u0] + fu p[v0+1][u0+1])]
// with w = U^2 * load_scale, under the cylinder, u-bounds and v-bounds masks.
// Its transpose therefore gives detector pixel (r, c) of a view the sum over
// voxels with u0 in {c-1, c} and v0 in {r-1, r} of
//     w * (u0 == c ? 1-fu : fu) * (v0 == r ? 1-fv : fv) * vol.
//
// Ray-driven gather (deterministic, no atomics), one lane per detector row. A
// warp takes kSW = 4 adjacent detector columns x 128 rows of one view, four rows
// per lane 32 apart; what depends only on (view, strip) -- which voxel columns
// can reach it -- is shared by the warp:
//  1. the warp walks the in-plane axis that is most perpendicular to the ray,
//     32 positions at a time, one position per lane; the lines u(x, y) = strip
//     edge (u is a ratio of linear functions, so they are straight) give each
//     lane a short range of candidate columns along the other axis;
//  2. step by step through those ranges, each lane evaluates one candidate
//     column with the very same FP32 expressions as the backprojector (so the
//     discrete decisions u0, v0 and the masks agree bit for bit with the
//     gather kernel's); a column that reaches the strip and the warp's rows
//     becomes a record in shared memory;
//  3. the warp takes the step's records, those with the same u0 and window
//     length together. For its row r a lane sums the column's slices z with
//     their vertical weights 1 - |vi(z) - r|, the bilinear weights 1-fv and fv
//     of rows v0 and v0+1 (exactly, the differences being exact in FP32 but for
//     vi - 1 below row 1/2, which rounds by less than 2^-24); only
//     the K = floor(2 / dv) + 1 slices from (c0 - r - 1) / dv on can have one,
//     dv the rows per slice. The sum times w (1-fu) and w fu goes to columns
//     u0 and u0+1: two registers per row within a group of records, the
//     strip's sums in shared memory between groups.
// A window that would leave the slices that count (the slab, cut to the
// reference's v run where the detector's outer rows can tell) is moved inside
// them, where its other slices weigh 0; a volume that holds an infinity or NaN (whose
// product with a zero weight must not reach rows the slice does not touch) or a value
// over 2^100 is summed slice by slice, those that do not touch a row left out.
// Elsewhere columns with fewer slices than a window take a checked sum: each slice
// weighted by its own v0 and fv (128^3 with one NaN, 120 views of 256 x 192: 1.32 ms;
// by checked sums throughout 1.64, the slice walk of the version before 1.41).
//
// What bounds it: the FP32 pipe (an FP32x2 instruction takes two of its cycles):
// per row and voxel column seven operations for each slice of the window and five
// for the row, 65 % of the issue slots used (256^3, 180 views). Integer steps that
// replace FP32 ones pay (the block of 32 by clearing bits of the magic-number
// sum: 3.50 -> 3.11 ms there, together with strips that share their edge
// column). 512^3 x 360 views of 512^2: 47 ms (1.03 TGUPS) against 97 ms for the
// version before, which walked a column's slices one per lane and added each
// to four sums in shared memory (eight shared accesses per slice, 43 % of them
// bank conflicts); 161 x 130 detector, 97 x 101 x 83 voxels of 1.6 pixels, 90
// views: 0.21 against 0.47 ms; voxels of 8 pixels (most rows see no slice)
// 0.38 against 0.41 ms. Not faster: strips of 8 (45.8 ms, but 0.26 ms on the
// small one) or 16 columns (50.8), 64 rows per warp (61 ms), 256 (51 ms),
// the strip's sums in registers (a switch per record: 75 ms), CTAs of two
// or eight warps.
//
// The volume is read in a z-fastest copy, so that a lane's slices are neighbours
// of the next lane's. Row blocks are the slowest grid dimension: the CTAs
// running at one time read the same range of slices and share it in L2.

#include <algorithm>
#include <type_traits>

#include "../ctb_internal.h"
#include "geom.cuh"

namespace ctb {

namespace {

constexpr unsigned kAll = 0xffffffffu;
// a CTA: kWarps warps of one view and one block of rows, each with a strip of kSW
// detector columns and kJ rows per lane
constexpr int kWarps = 4, kSW = 4, kJ = 4, kRows = 32 * kJ;
constexpr float kMagic = 12582912.0f;       // 1.5 * 2^23: rounds to an integer by one add
constexpr int kExtreme = 1 << 22;           // marks a window's length in an extreme volume
constexpr int kMagicBits = 0x4B400000;      // its bits: the low bits of integer + kMagic are the integer

// One voxel column that reaches a warp's strip and rows.
struct __align__(16) Hit {
    float c0, mdv;      // its row line (geom.cuh)
    float inv, za;      // 1 / dv; the window of row r starts at slice ceil(za - r inv)
    float zmin, zmax;   // first and last box slice where a window may start
    const float* line;  // box slice -kMagicBits of its line
    float wa, wb;       // weight of detector columns u0 and u0 + 1
};

// d = vi(z) - r of two rows' slices z, given as the bits of z + kMagic. vi as row_at
// forms it, fma(z mod 32, mdv, fma(z - z mod 32, mdv, c0)): the block's start is the
// integer with its low five bits cleared, z mod 32 the difference of the two floats
// (exact). The integer steps run beside the FMA pipe, which bounds this kernel.
__device__ __forceinline__ float2 row_distances(int zx, int zy, float2 nrf, float2 mdv, float2 c0) {
    const float2 zm = make_float2(__int_as_float(zx), __int_as_float(zy));
    const float2 bm = make_float2(__int_as_float(zx & ~31), __int_as_float(zy & ~31));
    const float2 zb = __fadd2_rn(bm, make_float2(-kMagic, -kMagic));
    const float2 zo = __ffma2_rn(bm, make_float2(-1.0f, -1.0f), zm);
    return __fadd2_rn(__ffma2_rn(zo, mdv, __ffma2_rn(zb, mdv, c0)), nrf);
}
// The weights 1 - |d|, 0 beyond 1.
__device__ __forceinline__ float2 weights(int zx, int zy, float2 nrf, float2 mdv, float2 c0) {
    const float2 d = row_distances(zx, zy, nrf, mdv, c0);
    return make_float2(__saturatef(1.0f - fabsf(d.x)), __saturatef(1.0f - fabsf(d.y)));
}

// The volume copy, for the bounds-checked build.
struct VolRange {
    const float* p;
    long long n;
};
__device__ __forceinline__ float fetch(const float* q, const VolRange& vol, unsigned site) {
    return CTB_FETCH_OK(q - vol.p, vol.n, site) ? __ldg(q) : 0.0f;
}

// Weighted sums over K slices for two rows whose windows start at the slices of
// bits zx, zy (lines p0, p1 start there).
template <int K>
__device__ __forceinline__ float2 window_sum(const float* __restrict__ p0, const float* __restrict__ p1, int zx,
                                             int zy, float2 nrf, float2 mdv, float2 c0, const VolRange& vol) {
    float2 v[K];
#pragma unroll
    for (int k = 0; k < K; ++k) v[k] = make_float2(fetch(p0 + k, vol, 6), fetch(p1 + k, vol, 6));
    float2 s = __fmul2_rn(weights(zx, zy, nrf, mdv, c0), v[0]);
#pragma unroll
    for (int k = 1; k < K; ++k) s = __ffma2_rn(weights(zx + k, zy + k, nrf, mdv, c0), v[k], s);
    return s;
}

// Row r's sum over the box slices za .. zb of a column among the K from z on:
// each with the weight of its own v0 and fv, as the backprojector reads it.
__device__ __forceinline__ float checked_sum(const float* __restrict__ col, float z, int K, int za, int zb, float mdv,
                                             float c0, int r, const VolRange& vol) {
    float s = 0.0f;
    const RowLine rl{mdv, c0};
    const int z0 = int(ceilf(fminf(fmaxf(z, -1.0e6f), 1.0e6f)));
    const int z1 = min(z0 + K - 1, zb);
    for (int k = max(z0, za); k <= z1; ++k) {
        const float vi = row_at(rl, k);
        const int v0 = int(vi);
        const float fv = __fsub_rn(vi, float(v0));
        const float x = fetch(col + k, vol, 7);
        if (r == v0) s = fmaf(1.0f - fv, x, s);
        if (r == v0 + 1) s = fmaf(fv, x, s);
    }
    return s;
}

// Shared memory of a warp: the records of one step, and the sums of the strip's
// columns cs0 - 1 .. cs0 + SW (the outer two belong to the neighbours' strips
// and are dropped), a column's rows contiguous.
struct WarpShared {
    Hit hits[32];
    float sum[kSW + 2][kRows];
};

// The rows of the hit columns `same` (lanes' records), all with windows of K
// slices (KC, or K at run time for KC = 0): gives their sums times w (1-fu) and
// w fu. r0: the lane's first row. EXTREME: the volume holds an infinity, a NaN or
// values near the largest float: slices that do not count or do not touch a row are
// left out (not taken times 0), and values are weighted before they are summed.
template <int JU, int KC, bool EXTREME = false>
__device__ __forceinline__ void hit_rows(const Hit* __restrict__ hits, unsigned same, int K, float r0,
                                         float2 (&ga)[kJ / 2], float2 (&gb)[kJ / 2], const VolRange& vol) {
#pragma unroll
    for (int i = 0; i < kJ / 2; ++i) ga[i] = gb[i] = make_float2(0.0f, 0.0f);
    float2 nr[JU / 2];   // the lane's rows, negated
#pragma unroll
    for (int i = 0; i < JU / 2; ++i) nr[i] = make_float2(-64.0f * i - r0, -64.0f * i - 32.0f - r0);
#pragma unroll 1
    do {
        const Hit t = hits[__ffs(same) - 1];
        same &= same - 1;
        const float2 mdv2 = make_float2(t.mdv, t.mdv), c02 = make_float2(t.c0, t.c0);
        const float za = fmaf(-r0, t.inv, t.za);
        const float2 wa2 = make_float2(t.wa, t.wa), wb2 = make_float2(t.wb, t.wb);
#pragma unroll
        for (int i = 0; i < JU / 2; ++i) {
            float2 z = make_float2(fmaf(-64.0f * i, t.inv, za), fmaf(-64.0f * i - 32.0f, t.inv, za));
            if constexpr (EXTREME) {
                // slices zmin .. zb count (the window may lie beyond them)
                const float zb = t.zmax + float(K - 1);
                z = make_float2(fminf(fmaxf(z.x, t.zmin - float(K)), zb + 1.0f),
                                fminf(fmaxf(z.y, t.zmin - float(K)), zb + 1.0f));
                const float2 zm = __fadd2_ru(z, make_float2(kMagic, kMagic));   // ceil
                const int za = kMagicBits + int(t.zmin), ze = kMagicBits + int(zb);
                const int sx = __float_as_int(zm.x), sy = __float_as_int(zm.y);
                const int k1 = min(K - 1, ze - min(sx, sy));
                for (int k = max(0, za - max(sx, sy)); k <= k1; ++k) {
                    const int zx = sx + k, zy = sy + k;
                    const float2 d = row_distances(zx, zy, nr[i], mdv2, c02);
                    // (a kept slice's row is 0 at least, as int() makes it)
                    const float dx = fmaxf(d.x, nr[i].x), dy = fmaxf(d.y, nr[i].y);
                    if (zx >= za && zx <= ze && dx >= -1.0f && dx < 1.0f) {   // r is v0 or v0 + 1
                        const float v = fetch(t.line + zx, vol, 8);
                        ga[i].x = fmaf(1.0f - fabsf(dx), t.wa * v, ga[i].x);
                        gb[i].x = fmaf(1.0f - fabsf(dx), t.wb * v, gb[i].x);
                    }
                    if (zy >= za && zy <= ze && dy >= -1.0f && dy < 1.0f) {
                        const float v = fetch(t.line + zy, vol, 8);
                        ga[i].y = fmaf(1.0f - fabsf(dy), t.wa * v, ga[i].y);
                        gb[i].y = fmaf(1.0f - fabsf(dy), t.wb * v, gb[i].y);
                    }
                }
                continue;
            }
            // a window stays inside the slices that count: one moved there has only
            // weights of 0 but for the slices it shares with the one it stands for
            z = make_float2(fminf(fmaxf(z.x, t.zmin), t.zmax), fminf(fmaxf(z.y, t.zmin), t.zmax));
            const float2 zm = __fadd2_ru(z, make_float2(kMagic, kMagic));   // ceil
            const int zx = __float_as_int(zm.x), zy = __float_as_int(zm.y);
            const float* p0 = t.line + zx;
            const float* p1 = t.line + zy;
            float2 s;
            if constexpr (KC > 0) {
                s = window_sum<KC>(p0, p1, zx, zy, nr[i], mdv2, c02, vol);
            } else {
                s = make_float2(0.0f, 0.0f);
                for (int k = 0; k < K; ++k)
                    s = __ffma2_rn(weights(zx + k, zy + k, nr[i], mdv2, c02),
                                   make_float2(fetch(p0 + k, vol, 6), fetch(p1 + k, vol, 6)), s);
            }
            ga[i] = __ffma2_rn(wa2, s, ga[i]);
            gb[i] = __ffma2_rn(wb2, s, gb[i]);
        }
    } while (same);
}

__global__ void __launch_bounds__(32 * kWarps, 7) fp_kernel(const float* __restrict__ volz,
                                                            const int* __restrict__ extreme_flag,
                                                            const float4* __restrict__ views, ProjGeom g,
                                                            float* __restrict__ proj, int accumulate) {
    constexpr int J = kJ, SW = kSW;
    static_assert(J % 2 == 0, "rows go in pairs");
    __shared__ WarpShared s_warp[kWarps];
    WarpShared& sh = s_warp[threadIdx.y];
    const int lane = threadIdx.x;
    const int R = blockIdx.z * kRows;                           // first row of the warp
    const int cs0 = (blockIdx.x * kWarps + threadIdx.y) * SW;   // first column of the strip
    // voxel columns of u0 = ulo .. cs0 + SW - 1: the share of column cs0 + SW goes to
    // the next strip through shared memory; the CTA's first strip also takes u0 =
    // cs0 - 1, whose column belongs to the CTA before (33 / 32 of the work, not 9 / 8)
    const int ulo = threadIdx.y == 0 ? cs0 - 1 : cs0;
    const int iv = blockIdx.y;
    const float4 q = __ldg(&views[iv]);
    const float sn = q.x, cs = q.y, h = q.z;
    const float D = g.D;
    const bool x_major = fabsf(cs) >= fabsf(sn);
    const int np = cs0 >= g.W ? 0 : x_major ? g.X : g.Y;   // (a strip past the detector does nothing)
    const int ns = x_major ? g.Y : g.X;
    // u = c on the line s = a(c) + b(c) p of box indices (p along the major axis, s
    // along the other): y = [T (D - x cs) + D (x sn - uOff)] / (D cs + T sn) or x =
    // [T (D - y sn) - D (y cs + uOff)] / (T cs - D sn), T = c - W/2, both linear. W < D
    // keeps the divisors at 0.35 D or more. `margin` covers the rounding of these
    // lines and of the u that decides (voxels).
    float a0, b0, a1, b1;
    {
        auto line_of = [&](double T, float* a, float* b) {
            const double d = x_major ? double(D) * cs + T * sn : T * cs - double(D) * sn;
            const double k0 = double(D) * (T - g.uOff) / d;
            const double k1 = x_major ? (double(D) * sn - T * cs) / d : -(T * sn + double(D) * cs) / d;
            const double pp = x_major ? g.xPre : g.yPre, sp = x_major ? g.yPre : g.xPre;
            *a = float(k0 / g.vs + sp - k1 * pp);
            *b = float(k1);
        };
        line_of(double(ulo) - double(g.uPre), &a0, &b0);
        line_of(double(cs0 + SW) - double(g.uPre), &a1, &b1);
    }
    const float margin = 0.05f + 1.0e-6f * (float(np + ns) + 4.0f * (float(g.W) + fabsf(g.uOff)) / g.vs);
    const int extreme = *extreme_flag != 0 ? kExtreme : 0;
    const bool edge = R <= 1 || R + kRows - 1 >= g.H - 3;   // rows the detector's bounds can cut
    const float r0 = float(R + lane);   // the lane's first row
    const VolRange vol{volz, (long long)g.X * g.Y * g.Zs};
#pragma unroll
    for (int k = 0; k < SW + 2; ++k)
#pragma unroll
        for (int j = 0; j < J; ++j) sh.sum[k][lane + 32 * j] = 0.0f;

    for (int ip0 = 0; ip0 < np; ip0 += 32) {
        // (1) candidate range of this lane's position
        const int ip = ip0 + lane;
        const float sa = fmaf(b0, float(ip), a0), sb = fmaf(b1, float(ip), a1), big = float(ns) + 2.0f;
        const int i0 = int(fmaxf(0.0f, ceilf(fminf(fmaxf(fminf(sa, sb) - margin, -2.0f), big))));
        const int i1 = int(fminf(float(ns - 1), floorf(fmaxf(fminf(fmaxf(sa, sb) + margin, big), -2.0f))));
        const int cnt = ip < np ? max(0, i1 - i0 + 1) : 0;
        const int steps = __reduce_max_sync(kAll, cnt);
        for (int st = 0; st < steps; ++st) {
            // (2) this lane's candidate column for this step; what identifies how a
            // record is taken: (u0 - c0 + 1) | checked << 7 | K << 8
            bool hit = false;
            int what = -1, ja = 0, jb = -1;   // slab slices that count
            if (st < cnt) {
                const int is = i0 + st;
                const int x = x_major ? ip : is, y = x_major ? is : ip;
                const float xw = world_coord(x, g.xPre, g.vs);
                const float yw = world_coord(y, g.yPre, g.vs);
                if (in_cylinder(xw, yw, g.r2)) {
                    float U, u;
                    column_geom(xw, yw, sn, cs, D, g.uOff, &U, &u);
                    const float ui = __fadd_rn(u, g.uPre);
                    const int u0 = int(ui);
                    if (u >= g.lbU && u <= g.ubU && u0 >= ulo && u0 <= cs0 + SW - 1) {
                        const float fu = __fsub_rn(ui, float(u0));
                        const float w = __fmul_rn(__fmul_rn(U, U), g.load_scale);
                        const RowLine rl = row_line(U, h, g.zpv, g.vs, g.vPre);
                        const float inv = 1.0f / -rl.mdv;
                        // widening of the windows (slices) for the rounding of vi (two FMAs),
                        // of the quotients and of 1/dv: each a few parts in 2^24 of the
                        // coordinates, together below 1e-6 of them
                        const float m = 1.0e-6f * (fabsf(rl.c0) + float(g.H)) * inv;
                        const float za = fmaf(rl.c0 - 1.0f, inv, -m);
                        const float span = 2.0f * inv + 2.0f * m;   // of a row's window
                        const int K = int(fminf(span, 1.0e6f)) + 1;
                        // slices of the warp's rows, R + kRows - 1 (lowest) to R (highest)
                        const float zfirst = fmaf(-float(R + kRows - 1), inv, za);
                        const float zlast = fmaf(-float(R), inv, za) + span;
                        hit = zlast >= float(g.z_begin) && zfirst <= float(g.z_begin + g.Zs - 1);
                        // the slices that count: the reference's v run where it can differ from the
                        // whole slab on the warp's rows (the detector's outer rows, slices within
                        // half a row of its bounds)
                        const float vt = row_at(rl, g.z_begin), vb = row_at(rl, g.z_begin + g.Zs - 1);
                        ja = 0;
                        jb = g.Zs - 1;
                        if (hit && edge && !(vb >= 0.5f && vt <= g.vi_hi - 0.5f))
                            v_inside_run(0, g.Zs, g.zPre, g.vs, h, U, g.lbV, g.ubV, &ja, &jb);
                        hit = hit && ja <= jb;
                        const bool check = jb - ja + 1 < K ||
                                           (edge && vb < 0.5f && row_at(rl, g.z_begin + jb) < 0.0f);
                        if (hit) {
                            what = (u0 - cs0 + 1) | int(check) << 7 | K << 8;
                            Hit& hr = sh.hits[lane];
                            hr.c0 = rl.c0;
                            hr.mdv = rl.mdv;
                            hr.inv = inv;
                            hr.za = za;
                            hr.zmin = float(g.z_begin + ja);
                            hr.zmax = float(g.z_begin + jb - K + 1);
                            hr.line = volz + (long long)(x * g.Y + y) * g.Zs - g.z_begin - kMagicBits;
                            hr.wa = w * (1.0f - fu);   // to column u0
                            hr.wb = w * fu;            // to column u0 + 1
                        }
                    }
                }
            }
            unsigned mask = __ballot_sync(kAll, hit);
            __syncwarp();
            // (3) the warp's rows of the hit columns, those taken alike together: a step's
            // columns have two or three values of u0 and one or two of K
            while (mask) {
                const int lead = __shfl_sync(kAll, what, __ffs(mask) - 1);
                const unsigned same = __ballot_sync(kAll, what == lead);
                mask &= ~same;
                const int K = lead >> 8 | extreme;
                float2 ga[J / 2], gb[J / 2];
                if ((lead & 128) && !extreme) {
#pragma unroll
                    for (int i = 0; i < J / 2; ++i) ga[i] = gb[i] = make_float2(0.0f, 0.0f);
                    for (unsigned e = same; e; e &= e - 1) {
                        const int src = __ffs(e) - 1;
                        const int a = g.z_begin + __shfl_sync(kAll, ja, src), b = g.z_begin + __shfl_sync(kAll, jb, src);
                        const Hit t = sh.hits[src];
#pragma unroll
                        for (int j = 0; j < J; ++j) {
                            const float x = checked_sum(t.line + kMagicBits, fmaf(-(r0 + 32.0f * j), t.inv, t.za), K, a,
                                                        b, t.mdv, t.c0, R + lane + 32 * j, vol);
                            float& xa = j & 1 ? ga[j / 2].y : ga[j / 2].x;
                            float& xb = j & 1 ? gb[j / 2].y : gb[j / 2].x;
                            xa = fmaf(t.wa, x, xa);
                            xb = fmaf(t.wb, x, xb);
                        }
                    }
                } else {
                    auto take = [&](auto used) {
                        constexpr int JU = decltype(used)::value;
                        switch (K) {
                            case 1: hit_rows<JU, 1>(sh.hits, same, K, r0, ga, gb, vol); break;
                            case 2: hit_rows<JU, 2>(sh.hits, same, K, r0, ga, gb, vol); break;
                            case 3: hit_rows<JU, 3>(sh.hits, same, K, r0, ga, gb, vol); break;
                            case 4: hit_rows<JU, 4>(sh.hits, same, K, r0, ga, gb, vol); break;
                            default:
                                if (K & kExtreme) hit_rows<JU, 0, true>(sh.hits, same, K & ~kExtreme, r0, ga, gb, vol);
                                else hit_rows<JU, 0>(sh.hits, same, K, r0, ga, gb, vol);
                                break;
                        }
                    };
                    // (a last row block with 64 rows or fewer skips the others)
                    if (J > 2 && R + 64 >= g.H) take(std::integral_constant<int, 2>{});
                    else take(std::integral_constant<int, J>{});
                }
                float* const sum = &sh.sum[lead & 127][lane];
#pragma unroll
                for (int i = 0; i < J / 2; ++i) {
                    sum[64 * i] += ga[i].x;
                    sum[64 * i + 32] += ga[i].y;
                    sum[64 * i + kRows] += gb[i].x;
                    sum[64 * i + 32 + kRows] += gb[i].y;
                }
            }
            __syncwarp();
        }
    }
    __syncthreads();
    // rows R .. of columns cs0 .., a warp 32 / SW rows of SW consecutive columns per step
    for (int idx = lane; idx < SW * kRows; idx += 32) {
        const int k = idx % SW, r = idx / SW;
        const int rk = R + r, ck = cs0 + k;
        if (rk >= g.H || ck >= g.W) continue;
        float* out = proj + (long long)iv * g.view_stride + (long long)rk * g.W + ck;
        float x = sh.sum[k + 1][r];
        if (k == 0 && threadIdx.y > 0) x += s_warp[threadIdx.y - 1].sum[SW + 1][r];
        *out = accumulate ? (*out + x) : x;
    }
}

// z-fastest copy of the slab, [x][y][z], through 32 x 32 shared-memory tiles;
// *extreme is set when a value is NaN or of a magnitude over 2^100: infinite, or one
// whose sums may be.
__global__ void volz_kernel(const float* __restrict__ in, int X, int Y, int Zs, float* __restrict__ out,
                            int* __restrict__ extreme) {
    __shared__ float tile[32][33];
    const int xt = blockIdx.x * 32, zt = blockIdx.z * 32, y = blockIdx.y;
    const long long plane = (long long)X * Y;
    bool bad = false;
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int z = zt + j, x = xt + threadIdx.x;
        if (z < Zs && x < X) {
            const float v = in[(long long)z * plane + (long long)y * X + x];
            bad |= !(fabsf(v) <= 1.2676506e30f);
            tile[j][threadIdx.x] = v;
        }
    }
    if (bad) *extreme = 1;
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        const int x = xt + j, z = zt + threadIdx.x;
        if (z < Zs && x < X) out[((long long)x * Y + y) * Zs + z] = tile[threadIdx.x][j];
    }
}

}  // namespace

int bounds_status_forward(unsigned* count, unsigned long long* first, int reset) {
#ifdef CTB_BOUNDS_CHECK
    CTB_CUDA_TRY(cudaMemcpyFromSymbol(count, g_bounds_count, sizeof(unsigned)));
    CTB_CUDA_TRY(cudaMemcpyFromSymbol(first, g_bounds_first, sizeof(unsigned long long)));
    if (reset) {
        const unsigned z = 0;
        const unsigned long long zz = 0;
        CTB_CUDA_TRY(cudaMemcpyToSymbol(g_bounds_count, &z, sizeof z));
        CTB_CUDA_TRY(cudaMemcpyToSymbol(g_bounds_first, &zz, sizeof zz));
    }
#else
    (void)reset;
    *count = 0;
    *first = 0;
#endif
    return CTB_OK;
}

int forward_launch(const float* vol, const float4* views, int n_views, const ProjGeom& g, float* proj,
                   int accumulate, cudaStream_t s) {
    if (n_views <= 0) return CTB_OK;
    if (n_views > 65535) {
        set_global_error("forward projector: at most 65535 views per call");
        return CTB_ERR_UNSUPPORTED;
    }
    if (g.Y > 65535) {
        set_global_error("forward projector: y too large");
        return CTB_ERR_UNSUPPORTED;
    }
    // z-fastest scratch copy of the slab, the flag before it
    const size_t n = size_t(g.X) * g.Y * g.Zs;
    char* scratch = nullptr;
    CTB_CUDA_TRY(scratch_alloc((void**)&scratch, 256 + sizeof(float) * n, s));
    int* extreme = reinterpret_cast<int*>(scratch);
    float* volz = reinterpret_cast<float*>(scratch + 256);
    int st = cuda_status(cudaMemsetAsync(extreme, 0, sizeof(int), s), "forward projector flag");
    if (st == CTB_OK) {
        volz_kernel<<<dim3((g.X + 31) / 32, g.Y, (g.Zs + 31) / 32), dim3(32, 8), 0, s>>>(vol, g.X, g.Y, g.Zs, volz,
                                                                                         extreme);
        st = cuda_status(cudaGetLastError(), "volz_kernel launch");
    }
    if (st == CTB_OK) {
        const dim3 grid((g.W + kWarps * kSW - 1) / (kWarps * kSW), n_views, (g.H + kRows - 1) / kRows);
        fp_kernel<<<grid, dim3(32, kWarps), 0, s>>>(volz, extreme, views, g, proj, accumulate);
        st = cuda_status(cudaGetLastError(), "fp_kernel launch");
    }
    cudaFreeAsync(scratch, s);
    return st;
}

namespace {
// r = a - b over n values; the sum of r^2 is added to *sumsq (double)
__global__ void residual_kernel(const float* __restrict__ a, const float* __restrict__ b, float* __restrict__ r,
                                long long n, double* __restrict__ sumsq) {
    double acc = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float d = a[i] - b[i];
        r[i] = d;
        acc += double(d) * double(d);
    }
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    __shared__ double part[8];
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < int(blockDim.x >> 5); ++w) t += part[w];
        atomicAdd(sumsq, t);
    }
}
}  // namespace

int residual_launch(const float* a, const float* b, float* r, long long n, double* sumsq, cudaStream_t s) {
    if (n <= 0) return CTB_OK;
    int dev = 0, sms = 0;
    CTB_CUDA_TRY(cudaGetDevice(&dev));
    CTB_CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    const long long blocks = std::min<long long>((n + 255) / 256, 8LL * sms);
    residual_kernel<<<int(blocks), 256, 0, s>>>(a, b, r, n, sumsq);
    return cuda_status(cudaGetLastError(), "residual_kernel launch");
}

}  // namespace ctb
