// Kernel (c): voxel-driven FDK backprojection, and the FP64 per-view geometry.
//
// Reference semantics: reconstructionCore (Ct/CtVolume.cpp:923-1046, CPU, the
// parity target) and reconstructionKernel (Ct/cuda_ct.cu:201-292, GPU):
//   x,y,z world = index - pre            (updateBoundaries :1419-1421)
//   cylinder    x^2 + y^2 < radius^2     (:980)
//   t = -x sin + y cos + uOffset, s = x cos + y sin, U = D/(D - s), u = t U
//   u in [-W/2, W-1.1-W/2]               (:998, bounds :924-925)
//   v = (z + h) U in [1.1-H/2+..., H/2]  (:1008-1011, bounds :927-928)
//   bilinear at (u + W/2, -v + H/2), weight U^2, vol += U^2 * value
//
// Design (B200): one thread owns an (x, y) column of ZC consecutive z voxels
// and keeps their sums in registers across every view of the launch, so the
// volume is written once per launch instead of read-modify-written per view
// (the reference launches once per view). u, U and U^2 depend only on
// (x, y, view) and are computed once per view for the whole column; per voxel
// only v, the row index and the bilinear sample remain. The per-view table
// {sin, cos, h} is built in FP64 on the device and staged into shared memory
// once per CTA. Warps run along x, so each z row of stores is one coalesced
// 128-byte segment of the X-fastest slab.

#include <cuda_bf16.h>
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <cuda_fp16.h>

#include "../ctb_internal.h"
#include "geom.cuh"

namespace ctb {

namespace {

__device__ __forceinline__ float4 view_record(double ang, double h) {
    // float angle_rad = (angle / 180.0) * M_PI; sine = sin(angle_rad) (:953-955)
    const float angle_rad = float((ang / 180.0) * 3.14159265358979323846);
    double s, c;
    sincos(double(angle_rad), &s, &c);
    return make_float4(float(s), float(c), float(h), 0.0f);
}

__global__ void view_table_kernel(const double* __restrict__ ang, const double* __restrict__ h, int n,
                                  float4* __restrict__ out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = view_record(ang[i], h[i]);
}

// N views' angles and heights as kernel arguments: no device copy of the host
// arrays to allocate, fill and give back (a call of the smallest scans spent more
// host time on those than on its launches).
template <int N> struct HostViews {
    double ang[N], h[N];
};
template <int N>
__global__ void view_table_args_kernel(const __grid_constant__ HostViews<N> v, int n, float4* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = view_record(v.ang[i], v.h[i]);
}

template <int N>
void view_table_args(const double* ang, const double* h, int n, float4* out, cudaStream_t s) {
    HostViews<N> v;
    std::memcpy(v.ang, ang, sizeof(double) * n);
    if (h) std::memcpy(v.h, h, sizeof(double) * n);
    else std::memset(v.h, 0, sizeof(double) * n);
    view_table_args_kernel<N><<<(n + 127) / 128, 128, 0, s>>>(v, n, out);
}

template <typename T> __device__ __forceinline__ float ld(const T* p);
template <> __device__ __forceinline__ float ld<float>(const float* p) { return __ldg(p); }
template <> __device__ __forceinline__ float ld<__half>(const __half* p) { return __half2float(__ldg(p)); }
template <> __device__ __forceinline__ float ld<__nv_bfloat16>(const __nv_bfloat16* p) {
    return __bfloat162float(__ldg(p));
}

constexpr int kBX = 32, kBY = 4;
constexpr int kViewsPerStage = 1024;   // shared-memory view table capacity (16 KB)

template <typename T, int ZC>
__global__ void __launch_bounds__(kBX * kBY) bp_kernel(const T* __restrict__ proj,
                                                       const float4* __restrict__ views, int n_views,
                                                       ProjGeom g, float* __restrict__ vol, int accumulate) {
    __shared__ float4 sviews[kViewsPerStage];
    const int x = blockIdx.x * kBX + threadIdx.x;
    const int y = blockIdx.y * kBY + threadIdx.y;
    const int z0 = blockIdx.z * ZC;
    const int tid = threadIdx.y * kBX + threadIdx.x;

    const float xw = world_coord(x, g.xPre, g.vs);
    const float yw = world_coord(y, g.yPre, g.vs);
    const bool live = x < g.X && y < g.Y && in_cylinder(xw, yw, g.r2);

    float acc[ZC];
#pragma unroll
    for (int j = 0; j < ZC; ++j) acc[j] = 0.0f;

    for (int vb = 0; vb < n_views; vb += kViewsPerStage) {
        const int nv = min(kViewsPerStage, n_views - vb);
        __syncthreads();
        for (int i = tid; i < nv; i += kBX * kBY) sviews[i] = __ldg(&views[vb + i]);
        __syncthreads();
        if (!live) continue;
        const T* pv = proj + (long long)vb * g.view_stride;
        for (int iv = 0; iv < nv; ++iv, pv += g.view_stride) {
            const float4 q = sviews[iv];  // sin, cos, h
            float U, u;
            column_geom(xw, yw, q.x, q.y, g.D, g.uOff, &U, &u);
            if (!(u >= g.lbU && u <= g.ubU)) continue;
            const float w = __fmul_rn(__fmul_rn(U, U), g.load_scale);
            const float ui = __fadd_rn(u, g.uPre);
            const int u0 = int(ui);
            const float fu = __fsub_rn(ui, float(u0));
#ifdef CTB_BOUNDS_CHECK
            const T* col = pv + (CTB_FETCH_OK(u0, g.W - 1, 6) ? u0 : 0);
#else
            const T* col = pv + u0;
#endif
            const RowLine rl = row_line(U, q.z, g.zpv, g.vs, g.vPre);
#pragma unroll
            for (int j = 0; j < ZC; ++j) {
                const float vi = row_at(rl, g.z_begin + z0 + j);
                const float zw = __fmul_rn(__fsub_rn(float(z0 + j), g.zPre), g.vs);
                if (v_inside(zw, q.z, U, g.lbV, g.ubV)) {
                    int v0 = int(vi);
                    const float fv = __fsub_rn(vi, float(v0));
#ifdef CTB_BOUNDS_CHECK
                    if (!CTB_FETCH_OK(v0, g.H - 1, 7)) v0 = 0;
#endif
                    const T* r0 = col + (long long)v0 * g.pitch;
                    const float a = (1.0f - fu) * ld(r0) + fu * ld(r0 + 1);
                    const float b = (1.0f - fu) * ld(r0 + g.pitch) + fu * ld(r0 + g.pitch + 1);
                    acc[j] += w * ((1.0f - fv) * a + fv * b);
                }
            }
        }
    }
    if (x >= g.X || y >= g.Y) return;
    const long long plane = (long long)g.X * g.Y;
    float* out = vol + (long long)z0 * plane + (long long)y * g.X + x;
#pragma unroll
    for (int j = 0; j < ZC; ++j) {
        if (z0 + j < g.Zs) {
            float* p = out + j * plane;
            *p = accumulate ? (*p + acc[j]) : acc[j];
        }
    }
}

template <typename T>
int bp_launch_typed(const T* proj, const float4* views, int n_views, const ProjGeom& g, float* vol,
                    int accumulate, cudaStream_t s) {
    constexpr int ZC = 16;
    dim3 block(kBX, kBY, 1);
    dim3 grid((g.X + kBX - 1) / kBX, (g.Y + kBY - 1) / kBY, (g.Zs + ZC - 1) / ZC);
    if (grid.x == 0 || grid.y == 0 || grid.z == 0) return CTB_OK;
    if (grid.z > 65535 || grid.y > 65535) {
        set_global_error("backproject: grid too large");
        return CTB_ERR_UNSUPPORTED;
    }
    bp_kernel<T, ZC><<<grid, block, 0, s>>>(proj, views, n_views, g, vol, accumulate);
    return cuda_status(cudaGetLastError(), "bp_kernel launch");
}

}  // namespace

int bounds_status_gather(unsigned* count, unsigned long long* first, int reset) {
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

int view_table_build(const double* angles_deg_dev, const double* heights_dev, int n, float4* out,
                     cudaStream_t s) {
    if (n <= 0) return CTB_OK;
    view_table_kernel<<<(n + 127) / 128, 128, 0, s>>>(angles_deg_dev, heights_dev, n, out);
    return cuda_status(cudaGetLastError(), "view_table_kernel launch");
}

int view_table_from_host(const double* angles_deg, const double* heights, int n, float4* out, cudaStream_t s) {
    constexpr int kMost = 1024;   // 16 KB of arguments a launch
    for (int i = 0; i < n; i += kMost) {
        const int k = std::min(kMost, n - i);
        const double* h = heights ? heights + i : nullptr;
        if (k <= 128) view_table_args<128>(angles_deg + i, h, k, out + i, s);
        else view_table_args<kMost>(angles_deg + i, h, k, out + i, s);
    }
    return cuda_status(cudaGetLastError(), "view_table_args_kernel launch");
}

static inline float __fmul_rn_host(float a, float b) { return a * b; }

ProjGeom proj_geom(const ctb_detector& det, const ctb_grid& grid, int z_begin, int z_end, float load_scale) {
    ProjGeom g;
    g.W = det.width;
    g.H = det.height;
    g.X = grid.x_to - grid.x_from;
    g.Y = grid.y_to - grid.y_from;
    g.Zs = z_end - z_begin;
    // updateBoundaries :1419-1423 (double expressions stored as float)
    g.xPre = float(float(grid.x_size) / 2.0 - float(grid.x_from));
    g.yPre = float(float(grid.y_size) / 2.0 - float(grid.y_from));
    const float zPre = float(float(grid.z_size) / 2.0 - float(grid.z_from));
    g.zPre = zPre - float(z_begin);
    g.vs = grid.voxel_pitch;
    g.D = det.fcd;
    g.uOff = det.u_offset;
    g.r2 = det.radius * det.radius;
    g.uPre = float(double(det.width) / 2.0);
    g.vPre = float(double(det.height) / 2.0);
    // reconstructionCore :924-928
    g.lbU = 0.0f - g.uPre;
    g.ubU = float(double(det.width) - 1 - 0.1) - g.uPre;
    g.lbV = (-1) * float(double(det.height) - 1 - 0.1) + g.vPre;
    g.ubV = (-1) * 0.0f + g.vPre;
    g.z_begin = z_begin;
    g.zpv = __fmul_rn_host(zPre, g.vs);
    g.vi_hi = float(double(det.height) - 1 - 0.1);
    g.load_scale = load_scale;
    g.pitch = det.width;
    g.view_stride = (long long)det.width * det.height;
    return g;
}

// z voxels per thread of the shared-memory backprojector: 32 spreads each column's
// per-view geometry over twice the voxels of 16 (8 % faster on the 128-slice slabs of
// a 1024^3 volume, with 3 instead of 4 CTAs per SM; 64 at 2 CTAs per SM was slower
// again), but a tile is summed whole, or group of eight by group of eight where it
// holds half its slices or fewer, which costs more per slice. Of 32 and 16 the
// one whose tiles take less time: 600 x 600 columns of 1.3 pixels, 60 views of 1024 x 512,
// ms a layer of tiles, FP32 / FP16: 32 whole 0.45 / 0.51, two groups 0.35 / 0.39, one 0.23 / 0.26; 16
// whole 0.26 / 0.29, one group 0.20 / 0.21. Slices 0 .. 40 0.82 in tiles of 32, 0.79 in tiles of
// 16; 16 .. 47 0.75 and 0.54; 0 .. 79 1.24 and 1.28. Up to 16 slices take 16 or 8.
int bp_pick_zc(int z_begin, int Zs) {
    if (Zs <= 16) return Zs > 8 ? 16 : 8;
    const int cost32[5] = {0, 8, 12, 16, 16}, cost16[3] = {0, 7, 9};   // by groups of eight in the slab
    auto cost = [&](int zc, const int* per_tile) {
        long long c = 0;
        for (int z = z_begin / zc * zc; z < z_begin + Zs; z += zc) {
            const int first = std::max(z, z_begin) / 8, last = (std::min(z + zc, z_begin + Zs) - 1) / 8;
            c += per_tile[last - first + 1];
        }
        return c;
    };
    return cost(16, cost16) <= cost(32, cost32) ? 16 : 32;
}

namespace {

// 16-byte pieces of the destination rows, read as aligned 32-bit words and
// shifted where the source row starts off a word (16-bit types at odd columns).
// One thread per piece, pieces of a row in adjacent threads. Bound by HBM: one
// read and one write of the rows.
template <int ES>   // element bytes: 2 or 4
__global__ void __launch_bounds__(256) repack_rows_kernel(const unsigned char* __restrict__ src, int W, int src_pitch,
                                                          long long src_stride, int row0, int rows, int pieces,
                                                          long long total, uint4* __restrict__ dst) {
    constexpr int N = 16 / ES;
    for (long long i = blockIdx.x * 256LL + threadIdx.x; i < total; i += gridDim.x * 256LL) {
        const int c = int(i % pieces) * N;
        const long long rv = i / pieces;
        const int r = int(rv % rows);
        const long long v = rv / rows;
        const unsigned char* p = src + (v * src_stride + (long long)(row0 + r) * src_pitch + c) * ES;
        uint32_t w[4];
        const bool odd = ES == 2 && (reinterpret_cast<uintptr_t>(p) & 2);
        if (c + N <= W && !odd) {
            const uint32_t* q = reinterpret_cast<const uint32_t*>(p);
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = __ldg(q + k);
        } else if (c > 0 && c + N < W) {
            // words from one element before the piece to one after it, all in the row
            const uint32_t* q = reinterpret_cast<const uint32_t*>(p - 2);
            uint32_t a[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) a[k] = __ldg(q + k);
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] = __funnelshift_r(a[k], a[k + 1], 16);
        } else {
            // a row's ends: element by element, zeros past the row
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                if constexpr (ES == 4) {
                    w[k] = c + k < W ? __ldg(reinterpret_cast<const uint32_t*>(p) + k) : 0u;
                } else {
                    const uint16_t* q = reinterpret_cast<const uint16_t*>(p);
                    const uint32_t lo = c + 2 * k < W ? __ldg(q + 2 * k) : 0u;
                    const uint32_t hi = c + 2 * k + 1 < W ? __ldg(q + 2 * k + 1) : 0u;
                    w[k] = lo | hi << 16;
                }
            }
        }
        dst[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Rows the TMA loads cannot take (a row pitch or base off 16 bytes: detector
// widths that are no multiple of 8 16-bit or 4 32-bit samples): the rows the
// slab reaches are copied, a run of views at a time, to rows of a 16-byte pitch
// and backprojected from there with the shared-memory kernel. The copy reads and
// writes each sample once; the gather kernel it replaces fetches four samples
// per voxel and view through L1. 500 views of 1021 x 777 BF16 into 333 x 301
// x 71: 3.6 ms against 15.2 ms with the gather kernel. The scratch holds 256 MB of
// views, or as many bytes as the slab if that is more: each run reads and writes the
// slab once. Returns CTB_ERR_UNSUPPORTED (nothing launched) when it has no memory.
int backproject_repacked(const void* proj, int store_type, const float4* views, int n_views, const ProjGeom& g,
                         double hmax, float* vol, int accumulate, cudaStream_t s, int zc, int nbuf) {
    const size_t es = store_bytes(store_type);
    ProjGeom b = g;
    slab_row_band(g, -hmax, hmax, &b.row0, &b.rows);
    const int n16 = int(16 / es);
    b.pitch = (g.W + n16 - 1) / n16 * n16;
    b.view_stride = (long long)b.rows * b.pitch;
    const size_t view_bytes = size_t(b.view_stride) * es;
    const size_t cap = std::max(size_t(256) << 20, sizeof(float) * size_t(g.X) * g.Y * g.Zs);
    const int run = int(std::max<size_t>(1, std::min<size_t>(size_t(n_views), cap / view_bytes)));
    void* rows = nullptr;
    if (scratch_alloc(&rows, view_bytes * run, s) != cudaSuccess) {
        cudaGetLastError();
        return CTB_ERR_UNSUPPORTED;
    }
    int st = CTB_OK;
    for (int v = 0; v < n_views && st == CTB_OK; v += run) {
        const int n = std::min(run, n_views - v);
        st = repack_rows_launch(static_cast<const char*>(proj) + size_t(v) * g.view_stride * es, store_type, g.W,
                                g.pitch, g.view_stride, b.row0, b.rows, n, rows, b.pitch, s);
        // (the kernel's base pointer is that of detector row 0)
        const char* base = static_cast<const char*>(rows) - (long long)b.row0 * b.pitch * (long long)es;
        if (st == CTB_OK)
            st = backproject_tma_launch(base, store_type, views + v, n, b, hmax, vol, v > 0 ? 1 : accumulate, s, zc,
                                        nbuf);
    }
    cudaFreeAsync(rows, s);
    return st;
}

}  // namespace

int repack_rows_launch(const void* src, int store_type, int W, int src_pitch, long long src_stride, int row0,
                       int rows, int n, void* dst, int dst_pitch, cudaStream_t s) {
    const int es = int(store_bytes(store_type));
    const int pieces = dst_pitch * es / 16;
    const long long total = (long long)n * rows * pieces;
    const int blocks = int(std::min<long long>((total + 255) / 256, 148LL * 64));
    auto kern = es == 2 ? repack_rows_kernel<2> : repack_rows_kernel<4>;
    kern<<<blocks, 256, 0, s>>>(static_cast<const unsigned char*>(src), W, src_pitch, src_stride, row0, rows, pieces,
                                total, static_cast<uint4*>(dst));
    return cuda_status(cudaGetLastError(), "repack_rows_kernel launch");
}

int backproject_launch(const void* proj, int store_type, const float4* views, int n_views,
                       const ProjGeom& g, double hmax, float* vol, int accumulate, cudaStream_t s, BpConfig cfg) {
    // shared-memory staged kernel when the footprint bound and the 16-byte TMA
    // stride rule allow it (or a copy to such rows pays); the global-gather
    // kernel otherwise.
    // CTB_BP_VARIANT=global|tma forces one of them (tma fails when ineligible).
    static const int variant = [] {
        const char* e = std::getenv("CTB_BP_VARIANT");
        if (!e) return 0;
        if (!std::strcmp(e, "global")) return 1;
        if (!std::strcmp(e, "tma")) return 2;
        return 0;
    }();
    // CTB_BP_ZC=8|16|32 fixes the z voxels per thread of the shared-memory kernel
    static const int zc_env = [] {
        const char* e = std::getenv("CTB_BP_ZC");
        const int v = e ? std::atoi(e) : 0;
        return (v == 8 || v == 16 || v == 32) ? v : 0;
    }();
    if (variant != 1) {
        const int zc = zc_env ? zc_env : cfg.zc ? cfg.zc : bp_pick_zc(g.z_begin, g.Zs);
        // tiles of 32 need two CTAs on an SM, or 16 is taken: voxels of 4 pixels FP32, whose boxes
        // leave one, 256 x 256 x 64 from 60 views of 1024 x 768 0.33 ms, tiles of 16 0.26; of 3.5 pixels (two
        // CTAs) 0.225 and 0.246
        const int ctas = zc == 32 && !zc_env && !cfg.zc ? 2 : 1;
        int st = CTB_ERR_UNSUPPORTED;
        if (backproject_tma_layout(proj, store_type, g)) {
            st = backproject_tma_launch(proj, store_type, views, n_views, g, hmax, vol, accumulate, s, zc, cfg.nbuf,
                                        ctas);
            // a taller tile's footprint may exceed the box limits where a shorter one fits
            if (st == CTB_ERR_UNSUPPORTED && !zc_env && zc > 16)
                st = backproject_tma_launch(proj, store_type, views, n_views, g, hmax, vol, accumulate, s, 16);
        } else if (variant == 0 && cfg.scratch &&
                   (store_type == CTB_FP32 || store_type == CTB_FP16 || store_type == CTB_BF16)) {
            // the copy costs about a fifth (16 bits) to two fifths (32 bits) of a gathered
            // update per sample: worth it from half an update per copied sample on (333 x 301 x
            // 71 voxels from 500 views of 1021 x 777 BF16, about 50 updates per sample: 3.6 ms
            // instead of 15.2; 32^3 voxels from 100 views of 2047 x 1500, 0.2 per sample:
            // gathered in 0.39 ms, the copy alone moves 60 MB)
            int lo = 0, rows = 0;
            slab_row_band(g, -hmax, hmax, &lo, &rows);
            const double updates = double(g.X) * g.Y * g.Zs, samples = double(g.W) * rows;
            if (2.0 * updates >= samples) {
                if (backproject_tma_fits(store_type, g, hmax, zc, cfg.nbuf, ctas))
                    st = backproject_repacked(proj, store_type, views, n_views, g, hmax, vol, accumulate, s, zc,
                                              cfg.nbuf);
                else if (!zc_env && zc > 16 && backproject_tma_fits(store_type, g, hmax, 16, 0, 1))
                    st = backproject_repacked(proj, store_type, views, n_views, g, hmax, vol, accumulate, s, 16, 0);
            }
        }
        if (st != CTB_ERR_UNSUPPORTED || variant == 2) return st;
    }
    return backproject_global_launch(proj, store_type, views, n_views, g, vol, accumulate, s);
}

int backproject_global_launch(const void* proj, int store_type, const float4* views, int n_views,
                              const ProjGeom& g, float* vol, int accumulate, cudaStream_t s) {
    switch (store_type) {
        case CTB_FP32: return bp_launch_typed((const float*)proj, views, n_views, g, vol, accumulate, s);
        case CTB_FP16: return bp_launch_typed((const __half*)proj, views, n_views, g, vol, accumulate, s);
        case CTB_BF16:
            return bp_launch_typed((const __nv_bfloat16*)proj, views, n_views, g, vol, accumulate, s);
    }
    set_global_error("backproject: unknown storage type");
    return CTB_ERR_ARG;
}

}  // namespace ctb
