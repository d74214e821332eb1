// Kernels (a)+(b): projection preprocessing fused into a shared-memory FFT ramp
// filter, plus the FP64 kernels that build the filter tables.
//
// Reference semantics (bastian-weber/Ct, CPU path, which is the parity target):
//   convertTo32bit      Ct/CtVolume.cpp:802-812  s = float(I)*alpha + beta
//   applyLogScaling     Ct/CtVolume.cpp:860-866  p = -ln(s * 1/(I0 + 1e-6*I0))
//   applyFeldkampWeight Ct/CtVolume.cpp:814-830  p *= D / sqrt(D^2 + u^2 + v^2)
//   applyFourierFilter  Ct/CtVolume.cpp:832-858  row DFT, bins 0..W/2 times
//                        window(k, W/2+1), unnormalised C2R (x W), no padding
//   windows             Ct/CtVolume.cpp:868-885
//
// Design. A row filter is a circular convolution of length W with a real, even
// kernel (the window is real and applied symmetrically by the C2R transform).
// Every case is therefore computed as
//     out = IFFT_M( FFT_M(x zero-padded to M) * K ),   K real,
// with a power-of-two M: M = W when W is a power of two (reference-exact
// circular filter), M = nextpow2(2W-1) with K = FFT of the periodically
// extended kernel otherwise (still exactly the length-W circular filter), and
// M = nextpow2(2W) with the window sampled on the padded grid for pad = 2.
// Because K is real and even, two detector rows are filtered at once as the
// real and imaginary parts of one complex signal.
//
// Lengths 256 ... 4096 run in registers (filter_rf_kernel below). Otherwise each
// group of M/8 threads owns one row pair in shared memory (M complex floats)
// and the FFT is a Stockham autosort transform with two barriers per stage. Raw
// pixels are read once, filtered values are written once: HBM traffic is the
// algorithmic minimum.

#include <type_traits>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "../ctb_internal.h"

namespace ctb {

namespace {

// ------------------------------------------------------------- FP64 tables
__global__ void twiddle_kernel(float2* tw, int M) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    double s, c;
    sincospi(-2.0 * double(k) / double(M), &s, &c);
    tw[k] = make_float2(float(c), float(s));
}

// The same factors in the order the register transforms read them (a warp's lanes
// side by side; the plain table's stride of s factors took up to 30 wavefronts a
// load): w_M^(ts) at [M + s L + t], s < 16, t < L = M / 16, and w_L^(t2 s2) at
// [2 M + s2 L2 + t2], s2 < 16, t2 < L2 = L / 16.
__global__ void twiddle_order_kernel(float2* tw, int M) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x, L = M / 16, L2 = L / 16;
    if (k < M) tw[M + k] = tw[(k / L) * (k % L)];
    else if (k < M + L) tw[M + k] = tw[16 * ((k - M) / L2) * ((k - M) % L2)];
}

// Reference window, Ct/CtVolume.cpp:868-885: rl = float(n)/float(N) in float,
// sin/cos evaluated in double on a float product, result rounded to float.
__device__ float window_ref(int filter, int k, int nyq) {
    const float rl = float(k) / float(nyq);
    if (filter == CTB_SHEPPLOGAN) {
        if (k == 0) return 0.0f;
        const double a = double(rl * 0.5f) * 3.14159265358979323846;
        return float(double(rl) * sin(a) / a);
    }
    if (filter == CTB_HANN) {
        return float(double(rl * 0.5f) * (1.0 + cos(3.14159265358979323846 * double(rl))));
    }
    return rl;
}

// Window in double on an arbitrary transform grid (padded mode).
__device__ double window_f64(int filter, int k, int nyq) {
    const double rl = double(k) / double(nyq);
    if (filter == CTB_SHEPPLOGAN) {
        if (k == 0) return 0.0;
        const double a = rl * 0.5 * 3.14159265358979323846;
        return rl * sin(a) / a;
    }
    if (filter == CTB_HANN) return rl * 0.5 * (1.0 + cos(3.14159265358979323846 * rl));
    return rl;
}

// K[k] for M == W (power of two, pad 1): the symmetric reference window.
__global__ void kernel_direct(float* K, int M, int filter) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const int kk = min(k, M - k);
    K[k] = window_ref(filter, kk, M / 2 + 1);
}

// K[k] for pad 2: (W/M) * window on the padded grid.
__global__ void kernel_padded(float* K, int M, int W, int filter) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    const int kk = min(k, M - k);
    K[k] = float(double(W) / double(M) * window_f64(filter, kk, M / 2 + 1));
}

// Spatial kernel of the length-W circular filter:
//   g[j] = sum_k Hsym[k] cos(2 pi j k / W)   (unnormalised, real, even).
__global__ void spatial_kernel(double* g, int W, int filter) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= W) return;
    const int nyq = W / 2 + 1;
    double acc = 0.0;
    for (int k = 0; k < W; ++k) {
        const int kk = min(k, W - k);
        const long long jk = (long long)j * k % W;
        acc += double(window_ref(filter, kk, nyq)) * cospi(2.0 * double(jk) / double(W));
    }
    g[j] = acc;
}

// K[k] = (1/M) sum_j G_M[j] cos(2 pi j k / M) with G_M the periodic extension
// of g placed at indices [0, W) and [M-W+1, M).
__global__ void embedded_kernel(float* K, const double* g, int W, int M) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= M) return;
    double acc = g[0];
    for (int j = 1; j < W; ++j) {
        const long long jk = (long long)j * k % M;
        acc += 2.0 * g[j] * cospi(2.0 * double(jk) / double(M));
    }
    K[k] = float(acc / double(M));
}

// ----------------------------------------------------------- storage types
template <typename T> __device__ __forceinline__ T to_store(float v);
template <> __device__ __forceinline__ float to_store<float>(float v) { return v; }
template <> __device__ __forceinline__ __half to_store<__half>(float v) { return __float2half_rn(v); }
template <> __device__ __forceinline__ __nv_bfloat16 to_store<__nv_bfloat16>(float v) {
    return __float2bfloat16_rn(v);
}

template <typename T> __device__ __forceinline__ float raw_value(const T* p, const FilterArgs& a);
template <> __device__ __forceinline__ float raw_value<uint8_t>(const uint8_t* p, const FilterArgs& a) {
    return __fadd_rn(__fmul_rn(float(*p), a.alpha), a.beta);
}
template <> __device__ __forceinline__ float raw_value<uint16_t>(const uint16_t* p, const FilterArgs& a) {
    return __fadd_rn(__fmul_rn(float(*p), a.alpha), a.beta);
}
template <> __device__ __forceinline__ float raw_value<float>(const float* p, const FilterArgs& a) {
    return *p;
}

// -ln(s * scale) * D / sqrt(D^2 + u^2 + v^2), no contraction (reference order).
__device__ __forceinline__ float log_part(float s, const FilterArgs& a) { return -logf(__fmul_rn(s, a.log_scale)); }
__device__ __forceinline__ float weight_part(int r, int c, const FilterArgs& a) {
    const float u = __fsub_rn(float(c), a.uPre);
    const float v = __fadd_rn(-float(r), a.vPre);
    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(a.D, a.D), __fmul_rn(u, u)), __fmul_rn(v, v));
    return __fdiv_rn(a.D, __fsqrt_rn(d2));
}

// TAB: the Feldkamp weight of every pixel comes from a table (exactly
// weight_part's values), loaded together with the raw samples, instead of a
// square root and a divide per pixel.

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// ------------------------------------------------------ shared-memory FFT
// Stockham autosort FFT of length M (power of two) by a group of TG = M/8
// threads: one radix-2 or radix-4 stage (when log2 M is not a multiple of 3)
// followed by radix-8 stages; every thread owns 8 elements per stage. The
// last forward stage multiplies by the kernel spectrum on its way to shared
// memory and the last inverse stage writes the filtered row pair straight to
// global memory, so each transform costs one shared-memory round trip per
// stage and no separate passes.
constexpr float kSqrtHalf = 0.70710678118654752440f;

template <bool INV>
__device__ __forceinline__ void dft2(float2* v) {
    const float2 a = v[0], b = v[1];
    v[0] = make_float2(a.x + b.x, a.y + b.y);
    v[1] = make_float2(a.x - b.x, a.y - b.y);
}

// forward: multiply by -i; inverse: by +i
template <bool INV>
__device__ __forceinline__ float2 rot90(float2 d) {
    return INV ? make_float2(-d.y, d.x) : make_float2(d.y, -d.x);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2& v0, float2& v1, float2& v2, float2& v3) {
    const float2 a0 = make_float2(v0.x + v2.x, v0.y + v2.y);
    const float2 a1 = make_float2(v0.x - v2.x, v0.y - v2.y);
    const float2 a2 = make_float2(v1.x + v3.x, v1.y + v3.y);
    const float2 a3 = rot90<INV>(make_float2(v1.x - v3.x, v1.y - v3.y));
    v0 = make_float2(a0.x + a2.x, a0.y + a2.y);
    v1 = make_float2(a1.x + a3.x, a1.y + a3.y);
    v2 = make_float2(a0.x - a2.x, a0.y - a2.y);
    v3 = make_float2(a1.x - a3.x, a1.y - a3.y);
}

// 8-point DFT in registers: two 4-point DFTs of the even and odd samples joined
// by the eighth roots of unity.
template <bool INV>
__device__ __forceinline__ void dft8(float2* v) {
    float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    float2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4<INV>(e0, e1, e2, e3);
    dft4<INV>(o0, o1, o2, o3);
    // w^1 = (1 -+ i)/sqrt2, w^2 = -+i, w^3 = (-1 -+ i)/sqrt2 (upper sign: forward)
    const float2 t1 = INV ? make_float2(kSqrtHalf * (o1.x - o1.y), kSqrtHalf * (o1.x + o1.y))
                          : make_float2(kSqrtHalf * (o1.x + o1.y), kSqrtHalf * (o1.y - o1.x));
    const float2 t2 = rot90<INV>(o2);
    const float2 t3 = INV ? make_float2(-kSqrtHalf * (o3.x + o3.y), kSqrtHalf * (o3.x - o3.y))
                          : make_float2(kSqrtHalf * (o3.y - o3.x), -kSqrtHalf * (o3.x + o3.y));
    v[0] = make_float2(e0.x + o0.x, e0.y + o0.y);
    v[4] = make_float2(e0.x - o0.x, e0.y - o0.y);
    v[1] = make_float2(e1.x + t1.x, e1.y + t1.y);
    v[5] = make_float2(e1.x - t1.x, e1.y - t1.y);
    v[2] = make_float2(e2.x + t2.x, e2.y + t2.y);
    v[6] = make_float2(e2.x - t2.x, e2.y - t2.y);
    v[3] = make_float2(e3.x + t3.x, e3.y + t3.y);
    v[7] = make_float2(e3.x - t3.x, e3.y - t3.y);
}

template <int R, bool INV>
__device__ __forceinline__ void butterfly(float2* v) {
    if (R == 2) dft2<INV>(v);
    else if (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
    else dft8<INV>(v);
}

enum { kToSmem = 0, kToSmemTimesK = 1, kToOutput = 2 };

// One radix-R stage; each of the TG threads does 8/R butterflies.
template <int R, bool INV, int DST, typename Out>
__device__ __forceinline__ void fft_stage(float2* s, int M, int Ns, const float2* __restrict__ tw,
                                          const float* __restrict__ K, int lt, int TG, const Out& out) {
    constexpr int PER = 8 / R;
    const int nb = M / R;
    const int step = M / (Ns * R);
    float2 y[PER][R];
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int b = lt + i * TG;
        const int jm = b & (Ns - 1);
#pragma unroll
        for (int r = 0; r < R; ++r) y[i][r] = s[b + r * nb];
        if (Ns > 1) {
#pragma unroll
            for (int r = 1; r < R; ++r) {
                float2 w = __ldg(&tw[(jm * r * step) & (M - 1)]);
                if (INV) w.y = -w.y;
                y[i][r] = cmul(y[i][r], w);
            }
        }
        butterfly<R, INV>(y[i]);
    }
    if (DST != kToOutput) __syncthreads();  // in place: all reads before any write
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int b = lt + i * TG;
        const int jm = b & (Ns - 1);
        const int d0 = (b - jm) * R + jm;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int idx = d0 + r * Ns;
            if (DST == kToOutput) {
                out(idx, y[i][r]);
            } else if (DST == kToSmemTimesK) {
                const float k = __ldg(&K[idx]);
                s[idx] = make_float2(y[i][r].x * k, y[i][r].y * k);
            } else {
                s[idx] = y[i][r];
            }
        }
    }
    if (DST != kToOutput) __syncthreads();
}

// Whole transform from shared memory, last stage to DSTL. All threads of the CTA must
// call it (barriers).
template <bool INV, int DSTL, typename Out>
__device__ void fft_run(float2* s, int M, int logM, const float2* __restrict__ tw, const float* __restrict__ K,
                        int lt, int TG, const Out& out) {
    const int rem = logM % 3;
    const int first = rem == 1 ? 2 : rem == 2 ? 4 : 8;
    const int nst = logM / 3 + (rem ? 1 : 0);
    int Ns = 1;
    for (int st = 0; st < nst; ++st) {
        if (st == 0) {
            if (nst == 1) fft_stage<8, INV, DSTL>(s, M, Ns, tw, K, lt, TG, out);
            else if (first == 2) fft_stage<2, INV, kToSmem>(s, M, Ns, tw, K, lt, TG, out);
            else if (first == 4) fft_stage<4, INV, kToSmem>(s, M, Ns, tw, K, lt, TG, out);
            else fft_stage<8, INV, kToSmem>(s, M, Ns, tw, K, lt, TG, out);
            Ns *= first;
        } else if (st == nst - 1) {
            fft_stage<8, INV, DSTL>(s, M, Ns, tw, K, lt, TG, out);
            Ns *= 8;
        } else {
            fft_stage<8, INV, kToSmem>(s, M, Ns, tw, K, lt, TG, out);
            Ns *= 8;
        }
    }
}

// One group of TG = M/8 threads per detector row pair; groups = blockDim/TG.
template <typename InT, typename OutT, bool TAB>
__global__ void __launch_bounds__(1024) filter_kernel(const InT* __restrict__ raw, OutT* __restrict__ out,
                                                      FilterArgs a, const float2* __restrict__ tw,
                                                      const float* __restrict__ K) {
    extern __shared__ float2 smem[];
    const int M = a.M, TG = M >> 3;
    const int g = threadIdx.x / TG, lt = threadIdx.x - g * TG;
    const int groups = blockDim.x / TG;
    float2* s = smem + (size_t)g * M;

    const int W = a.W, H = a.H;
    const int pairs = (H + 1) >> 1;
    const long long q = (long long)blockIdx.x * groups + g;
    const bool active = q < a.n_views * pairs;
    const long long view = active ? q / pairs : 0;
    const int r0 = active ? int(q - view * pairs) * 2 : 0;
    const bool has1 = r0 + 1 < H;
    const size_t base0 = (size_t)view * H * W + (size_t)r0 * W;              // raw rows (dense)
    const size_t obase = (size_t)view * H * a.out_pitch + (size_t)r0 * a.out_pitch;  // filtered rows

    auto store = [&](int c, float2 z) {
        if (active && c < W) {
            out[obase + c] = to_store<OutT>(z.x * a.store_scale);
            if (has1) out[obase + a.out_pitch + c] = to_store<OutT>(z.y * a.store_scale);
        }
    };
    // Rows r0 and r0+1 as the real and imaginary parts, zero beyond W. Preprocessing is
    // kept out of the first FFT stage (done there it raises the register footprint: it
    // involves log, sqrt and divide). All 16 raw loads of
    // a thread (8 columns x 2 rows; TG = M/8) are issued before any arithmetic,
    // so their latencies overlap instead of adding up.
    InT v0[8], v1[8];
    float w0[8], w1[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int c = lt + k * TG;
        const bool in = active && c < W;
        v0[k] = in ? raw[base0 + c] : InT(0);
        v1[k] = in && has1 ? raw[base0 + W + c] : InT(0);
        if constexpr (TAB) {
            w0[k] = in ? __ldg(&a.wt[(size_t)r0 * W + c]) : 0.0f;
            w1[k] = in && has1 ? __ldg(&a.wt[(size_t)(r0 + 1) * W + c]) : 0.0f;
        }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int c = lt + k * TG;
        float2 z = make_float2(0.f, 0.f);
        if (active && c < W) {
            const float wa = TAB ? w0[k] : weight_part(r0, c, a);
            z.x = __fmul_rn(log_part(raw_value(&v0[k], a), a), wa);
            if (has1) {
                const float wb = TAB ? w1[k] : weight_part(r0 + 1, c, a);
                z.y = __fmul_rn(log_part(raw_value(&v1[k], a), a), wb);
            }
        }
        s[c] = z;
    }
    __syncthreads();
    fft_run<false, kToSmemTimesK>(s, M, a.logM, tw, K, lt, TG, store);
    fft_run<true, kToOutput>(s, M, a.logM, tw, K, lt, TG, store);
}

// --------------------------------------- register four-step transform
// For M = 16 L with L = 16 L2 (M = 256 ... 4096) a group of L threads owns four
// detector rows: rows r0, r0+1 as the real and imaginary parts of one complex
// signal, r0+2, r0+3 of another. Every thread keeps 16 values of both, the two
// signals side by side in FP32x2 pairs (real parts in one pair, imaginary parts
// in another): every operation of the transform is one FP32x2 instruction for
// both, a multiplication by i costs nothing, and the twiddles, the kernel
// spectrum and the weights' addresses serve both. Three register passes joined
// by two shared-memory transposes:
//   1. thread t:       16-point DFT over r of x[t + L r], times w_M^(ts)
//   2. thread (s, t2): 16-point DFT over r of pass 1's values (t2 + L2 r, s),
//                      times w_L^(t2 s2)
//   3. thread (s, j):  for s2 = j + L2 q (q < 16 / L2) the L2-point DFT over t2
//                      (none for M = 256, L2 = 1),
// which leaves X[s + 16 s2 + 256 k3] in registers (k3 < L2). The kernel
// spectrum multiplies it there; the inverse runs the passes backwards with
// conjugate factors and ends with thread t holding x[t + L r] again, so raw
// rows are read and filtered rows written with the same coalesced pattern.
// The exchange between passes 2 and 3 stays inside a warp. The paddings (L2
// per 16-value row of the first transpose, 1 per s2 row and L2 per s block of
// the second) keep every shared-memory access of 16 bytes per lane at the four
// wavefronts a warp needs.
//
// HALF: W <= M / 2 (rows embedded in a longer transform): the upper eight of a
// thread's sixteen columns are zeros before and unused after the transform, so
// they are neither loaded nor computed in the outer passes.
//
// What bounds it: the FP32 pipe (an FP32x2 instruction takes two of its cycles;
// per sample of a power-of-two row about 35 operations of the transforms and 19 of
// -ln, the weight and the scales), 16 warps per SM and the L1 pipe together: 56 % of
// the issue slots, 55 % of the L1 wavefronts. 54 instructions per sample; the
// version before (one row pair per group, scalar operations, twiddles read at a
// stride) took 84. u16 to FP16, 144 views of 2048^2: 2.11 -> 1.51 ms (1.6 TB/s); 360 of
// 701 x 409 to FP32 (M = 2048): 1.21 -> 0.60; 360 of 256 x 192 to FP16: 0.104 ->
// 0.042. Not faster: one code instance for both row pairs (a loop; registers
// spill: 1.77 ms), five CTAs of 128 threads per SM (102 registers: 1.81), a
// run-time switch to logf in the whole-number instances (1.66).
template <int M> struct RF {
    static constexpr int L = M / 16, L2 = L / 16, Q = 16 / L2;
    static constexpr int SA = 16 * (L + L2);       // first transpose, float4 per group
    static constexpr int SB = 16 * (L2 + 1) + L2;  // second transpose, float4 per s block
    static constexpr int T = L > 128 ? L : 128;    // threads per CTA: small ones, whose barriers stall little
    static constexpr int G = T / L;                // groups (of four rows) per CTA
    static constexpr int SG = L2 > 1 && 16 * SB > SA ? 16 * SB : SA;   // float4 per group, both in one place
    static_assert(M >= 256 && M <= 4096 && (M & (M - 1)) == 0, "register transform lengths");
};

// two complex numbers side by side: (re of A, re of B), (im of A, im of B)
struct C2 {
    float2 x, y;
};

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 dup(float a) { return make_float2(a, a); }
__device__ __forceinline__ C2 add2(const C2& a, const C2& b) { return {add2(a.x, b.x), add2(a.y, b.y)}; }
__device__ __forceinline__ C2 sub2(const C2& a, const C2& b) { return {sub2(a.x, b.x), sub2(a.y, b.y)}; }

// a times w (CONJ: its conjugate)
template <bool CONJ>
__device__ __forceinline__ C2 mul2(const C2& a, float2 w) {
    const float2 c = dup(w.x), s = dup(w.y), n = dup(-w.y);
    return {__ffma2_rn(a.y, CONJ ? s : n, __fmul2_rn(a.x, c)), __ffma2_rn(a.x, CONJ ? n : s, __fmul2_rn(a.y, c))};
}

// 4-point DFT in place (INV: the inverse); HALF_IN: v2 and v3 are zero
template <bool INV, bool HALF_IN = false>
__device__ __forceinline__ void dft4(C2& v0, C2& v1, C2& v2, C2& v3) {
    const C2 a0 = HALF_IN ? v0 : add2(v0, v2), a1 = HALF_IN ? v0 : sub2(v0, v2);
    const C2 a2 = HALF_IN ? v1 : add2(v1, v3), d = HALF_IN ? v1 : sub2(v1, v3);
    v0 = add2(a0, a2);
    v2 = sub2(a0, a2);
    // a1 + and - (-i d forward, i d inverse)
    const C2 p = {add2(a1.x, d.y), sub2(a1.y, d.x)}, m = {sub2(a1.x, d.y), add2(a1.y, d.x)};
    v1 = INV ? m : p;
    v3 = INV ? p : m;
}

template <bool INV>
__device__ __forceinline__ void dft8(C2* v) {
    C2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6];
    C2 o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
    dft4<INV>(e0, e1, e2, e3);
    dft4<INV>(o0, o1, o2, o3);
    // w^1 = (1 -+ i)/sqrt2, w^2 = -+i, w^3 = (-1 -+ i)/sqrt2 (upper sign: forward)
    const float2 h = dup(kSqrtHalf), nh = dup(-kSqrtHalf);
    const C2 t1 = INV ? C2{__fmul2_rn(h, sub2(o1.x, o1.y)), __fmul2_rn(h, add2(o1.x, o1.y))}
                      : C2{__fmul2_rn(h, add2(o1.x, o1.y)), __fmul2_rn(h, sub2(o1.y, o1.x))};
    const C2 t3 = INV ? C2{__fmul2_rn(nh, add2(o3.x, o3.y)), __fmul2_rn(h, sub2(o3.x, o3.y))}
                      : C2{__fmul2_rn(h, sub2(o3.y, o3.x)), __fmul2_rn(nh, add2(o3.x, o3.y))};
    v[0] = add2(e0, o0);
    v[4] = sub2(e0, o0);
    v[1] = add2(e1, t1);
    v[5] = sub2(e1, t1);
    const C2 p = {add2(e2.x, o2.y), sub2(e2.y, o2.x)}, m = {sub2(e2.x, o2.y), add2(e2.y, o2.x)};
    v[2] = INV ? m : p;
    v[6] = INV ? p : m;
    v[3] = add2(e3, t3);
    v[7] = sub2(e3, t3);
}

// x times w16^m (forward: exp(-2 pi i m / 16); inverse: the conjugate)
template <bool INV, int m>
__device__ __forceinline__ C2 tw16(const C2& a) {
    constexpr float c1 = 0.92387953251128675613f, s1 = 0.38268343236508977173f;
    // cos and sin of 2 pi m / 16 for m = 0 ... 9 (m = n1 k2 <= 9)
    constexpr float cs[10] = {1.0f, c1, kSqrtHalf, s1, 0.0f, -s1, -kSqrtHalf, -c1, -1.0f, -c1};
    constexpr float sn[10] = {0.0f, s1, kSqrtHalf, c1, 1.0f, c1, kSqrtHalf, s1, 0.0f, -s1};
    static_assert(m >= 0 && m <= 9, "twiddle index");
    if constexpr (m == 0) return a;
    else if constexpr (m == 4) {
        const float2 m1 = dup(-1.0f);
        return INV ? C2{__fmul2_rn(a.y, m1), a.x} : C2{a.y, __fmul2_rn(a.x, m1)};
    } else {
        return mul2<!INV>(a, make_float2(cs[m], sn[m]));
    }
}

// 16-point DFT in registers, natural order in and out: n = n1 + 4 n2,
// k = 4 k1 + k2; 4-point DFTs over n2, twiddles w16^(n1 k2), 4-point DFTs over n1.
// HALF_IN: the inputs 8 .. 15 are zero; HALF_OUT: only the outputs 0 .. 7 are wanted.
template <bool INV, bool HALF_IN = false, bool HALF_OUT = false>
__device__ __forceinline__ void dft16(C2* v) {
    C2 a[4][4];
#pragma unroll
    for (int n1 = 0; n1 < 4; ++n1) {
        a[n1][0] = v[n1]; a[n1][1] = v[n1 + 4];
        if constexpr (!HALF_IN) {
            a[n1][2] = v[n1 + 8]; a[n1][3] = v[n1 + 12];
        }
        dft4<INV, HALF_IN>(a[n1][0], a[n1][1], a[n1][2], a[n1][3]);
    }
    a[1][1] = tw16<INV, 1>(a[1][1]); a[1][2] = tw16<INV, 2>(a[1][2]); a[1][3] = tw16<INV, 3>(a[1][3]);
    a[2][1] = tw16<INV, 2>(a[2][1]); a[2][2] = tw16<INV, 4>(a[2][2]); a[2][3] = tw16<INV, 6>(a[2][3]);
    a[3][1] = tw16<INV, 3>(a[3][1]); a[3][2] = tw16<INV, 6>(a[3][2]); a[3][3] = tw16<INV, 9>(a[3][3]);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) {
        dft4<INV>(a[0][k2], a[1][k2], a[2][k2], a[3][k2]);
#pragma unroll
        for (int k1 = 0; k1 < (HALF_OUT ? 2 : 4); ++k1) v[4 * k1 + k2] = a[k1][k2];   // (unwanted ones: dead code)
    }
}

// L2-point DFT
template <int N, bool INV>
__device__ __forceinline__ void dft_n(C2* v) {
    if constexpr (N == 2) {
        const C2 a = v[0], b = v[1];
        v[0] = add2(a, b);
        v[1] = sub2(a, b);
    } else if constexpr (N == 4) {
        dft4<INV>(v[0], v[1], v[2], v[3]);
    } else if constexpr (N == 8) {
        dft8<INV>(v);
    } else if constexpr (N == 16) {
        dft16<INV>(v);
    }
}

__device__ __forceinline__ float4 as4(const C2& a) { return make_float4(a.x.x, a.x.y, a.y.x, a.y.y); }
__device__ __forceinline__ C2 as2(const float4& a) { return {make_float2(a.x, a.y), make_float2(a.z, a.w)}; }

// -ln of two positive normal numbers. With m in [sqrt(1/2), sqrt(2)) the number's
// mantissa, e its exponent and n = 1 - m (exact): -ln m = n + n^2 Q(n), Q a degree-8
// least-maximum-error fit of the relative error over the interval (its coefficients
// rounded to floats leave 7e-9), and e ln 2 is taken off in two parts, the first
// exact for every e: Cody and Waite's reduction (Software Manual for the Elementary
// Functions, 1980) with the mantissa about 1. At most 0.9 units in the last place
// of the result, as logf; the FP32x2 form shares each step between two samples.
__device__ __forceinline__ float2 neg_ln2(float2 s) {
    const int ix = __float_as_int(s.x) - 0x3F3504F3, iy = __float_as_int(s.y) - 0x3F3504F3;   // bits of sqrt(1/2)
    const int ex = ix & 0xff800000, ey = iy & 0xff800000;                                     // e << 23
    const float2 n = sub2(dup(1.0f), make_float2(__int_as_float(__float_as_int(s.x) - ex),
                                                 __int_as_float(__float_as_int(s.y) - ey)));
    // e as a float: 1.5 * 2^23 + e less the former
    const float2 e = add2(make_float2(__int_as_float(0x4B400000 + (ix >> 23)), __int_as_float(0x4B400000 + (iy >> 23))),
                          dup(-12582912.0f));
    float2 q = dup(7.622107e-2f);
    q = __ffma2_rn(q, n, dup(1.2904692e-1f));
    q = __ffma2_rn(q, n, dup(1.3242977e-1f));
    q = __ffma2_rn(q, n, dup(1.4181779e-1f));
    q = __ffma2_rn(q, n, dup(1.6609077e-1f));
    q = __ffma2_rn(q, n, dup(2.0001977e-1f));
    q = __ffma2_rn(q, n, dup(2.5001583e-1f));
    q = __ffma2_rn(q, n, dup(3.3333326e-1f));
    q = __ffma2_rn(q, n, dup(4.9999988e-1f));
    const float2 t = __ffma2_rn(__fmul2_rn(n, n), q, __fmul2_rn(e, dup(-1.4286068e-6f)));
    return __ffma2_rn(e, dup(-0.693145752f), add2(n, t));   // 0.693145752 = 0xB1720 / 2^20
}

template <int M, bool HALF, typename InT, typename OutT>
__global__ void __launch_bounds__(RF<M>::T, 512 / RF<M>::T)
    filter_rf_kernel(const InT* __restrict__ raw, OutT* __restrict__ out, FilterArgs a, const float2* __restrict__ tw,
                     const float* __restrict__ K) {
    using C = RF<M>;
    constexpr int L = C::L, L2 = C::L2, Q = C::Q, NR = HALF ? 8 : 16;
    const float2* const tw1 = tw + M + threadIdx.x % L;              // pass 1: [s L]
    const float2* const tw2 = tw + 2 * M + threadIdx.x % L % L2;     // pass 2: [s2 L2]
    extern __shared__ float4 smem4[];
    const int g = threadIdx.x / L, lt = threadIdx.x % L;
    float4* sa = smem4 + g * C::SG;
    const int W = a.W, H = a.H;
    const int quads = (H + 3) >> 2;
    const long long q = (long long)blockIdx.x * C::G + g;
    const bool active = q < a.n_views * quads;
    const long long view = active ? q / quads : 0;
    const int r0 = active ? int(q - view * quads) * 4 : 0;
    const int rows = active ? min(4, H - r0) : 0;
    const InT* src = raw + ((size_t)view * H + r0) * W + lt;
    const float* wrow = a.wt + (size_t)r0 * W + lt;

    C2 v[16];
    // rows ra and ra + 2 at once (the same component of the two signals)
    auto load_rows = [&](auto rac, auto put) {
        constexpr int ra = decltype(rac)::value;
        InT x0[NR], x1[NR];
        float w0[NR], w1[NR];
        const bool has0 = ra < rows, has1 = ra + 2 < rows;
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const bool in = !HALF || lt + L * r < W;
            x0[r] = in && has0 ? src[ra * W + L * r] : InT(1);
            x1[r] = in && has1 ? src[(ra + 2) * W + L * r] : InT(1);
            w0[r] = in && has0 ? __ldg(wrow + ra * W + L * r) : 0.0f;
            w1[r] = in && has1 ? __ldg(wrow + (ra + 2) * W + L * r) : 0.0f;
        }
        float2 p[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r)
            p[r] = make_float2(__fmul_rn(raw_value(&x0[r], a), a.log_scale),
                               __fmul_rn(raw_value(&x1[r], a), a.log_scale));
        // whole-number samples give normal positive arguments (launch_typed); a float sample
        // may give any other (zero, negative, tiny, infinite, NaN): those go to logf
        bool odd = false;
        if constexpr (std::is_same<InT, float>::value) {
#pragma unroll
            for (int r = 0; r < NR; ++r)
                odd |= unsigned(__float_as_int(p[r].x) - 0x00800000) >= 0x7f000000u ||
                       unsigned(__float_as_int(p[r].y) - 0x00800000) >= 0x7f000000u;
        }
        if (std::is_same<InT, float>::value && odd) {
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const float2 c = p[r];
                p[r] = neg_ln2(c);
                if (unsigned(__float_as_int(c.x) - 0x00800000) >= 0x7f000000u) p[r].x = -logf(c.x);
                if (unsigned(__float_as_int(c.y) - 0x00800000) >= 0x7f000000u) p[r].y = -logf(c.y);
            }
        } else {
#pragma unroll
            for (int r = 0; r < NR; ++r) p[r] = neg_ln2(p[r]);
        }
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            p[r] = __fmul2_rn(p[r], make_float2(w0[r], w1[r]));
            if (!has0 || (HALF && lt + L * r >= W)) p[r].x = 0.0f;
            if (!has1 || (HALF && lt + L * r >= W)) p[r].y = 0.0f;
            put(r, p[r]);
        }
    };
    load_rows(std::integral_constant<int, 0>{}, [&](int r, float2 p) { v[r].x = p; });
    load_rows(std::integral_constant<int, 1>{}, [&](int r, float2 p) { v[r].y = p; });

    // pass 1
    dft16<false, HALF>(v);
#pragma unroll
    for (int s = 1; s < 16; ++s) v[s] = mul2<false>(v[s], __ldg(tw1 + s * L));
#pragma unroll
    for (int s = 0; s < 16; ++s) sa[s * (L + L2) + lt] = as4(v[s]);
    __syncthreads();
    // pass 2
    const int ps = lt / L2, t2 = lt % L2;
    float4* bs = sa + ps * C::SB;
#pragma unroll
    for (int r = 0; r < 16; ++r) v[r] = as2(sa[ps * (L + L2) + t2 + L2 * r]);
    dft16<false>(v);
    if constexpr (L2 == 1) {
        // X[s + 16 s2] is here
#pragma unroll
        for (int s2 = 0; s2 < 16; ++s2) {
            const float2 k = dup(__ldg(&K[ps + 16 * s2]));
            v[s2] = {__fmul2_rn(v[s2].x, k), __fmul2_rn(v[s2].y, k)};
        }
    } else {
#pragma unroll
        for (int s2 = 1; s2 < 16; ++s2) v[s2] = mul2<false>(v[s2], __ldg(tw2 + s2 * L2));
        __syncthreads();  // the second transpose overwrites the first
#pragma unroll
        for (int s2 = 0; s2 < 16; ++s2) bs[s2 * (L2 + 1) + t2] = as4(v[s2]);
        __syncwarp();
        // pass 3, the kernel spectrum, inverse pass 3
        {
            C2 u[Q][L2];
#pragma unroll
            for (int qq = 0; qq < Q; ++qq)
#pragma unroll
                for (int k = 0; k < L2; ++k) u[qq][k] = as2(bs[(t2 + L2 * qq) * (L2 + 1) + k]);
#pragma unroll
            for (int qq = 0; qq < Q; ++qq) {
                dft_n<L2, false>(u[qq]);
#pragma unroll
                for (int k3 = 0; k3 < L2; ++k3) {
                    const float2 kf = dup(__ldg(&K[ps + 16 * (t2 + L2 * qq) + 256 * k3]));
                    u[qq][k3] = {__fmul2_rn(u[qq][k3].x, kf), __fmul2_rn(u[qq][k3].y, kf)};
                }
                dft_n<L2, true>(u[qq]);
            }
            __syncwarp();
#pragma unroll
            for (int qq = 0; qq < Q; ++qq)
#pragma unroll
                for (int k = 0; k < L2; ++k) bs[(t2 + L2 * qq) * (L2 + 1) + k] = as4(u[qq][k]);
            __syncwarp();
        }
        // inverse pass 2
#pragma unroll
        for (int s2 = 0; s2 < 16; ++s2) v[s2] = as2(bs[s2 * (L2 + 1) + t2]);
#pragma unroll
        for (int s2 = 1; s2 < 16; ++s2) v[s2] = mul2<true>(v[s2], __ldg(tw2 + s2 * L2));
    }
    dft16<true>(v);
    __syncthreads();  // every warp has read its values of the transpose before
#pragma unroll
    for (int r = 0; r < 16; ++r) sa[ps * (L + L2) + t2 + L2 * r] = as4(v[r]);
    __syncthreads();
    // inverse pass 1 and the filtered rows
#pragma unroll
    for (int s = 0; s < 16; ++s) v[s] = as2(sa[s * (L + L2) + lt]);
#pragma unroll
    for (int s = 1; s < 16; ++s) v[s] = mul2<true>(v[s], __ldg(tw1 + s * L));
    dft16<true, false, HALF>(v);
    OutT* const dst = out + ((size_t)view * H + r0) * a.out_pitch + lt;
#pragma unroll
    for (int r = 0; r < NR; ++r) {
        if (HALF && lt + L * r >= W) continue;
        const float e[4] = {v[r].x.x, v[r].y.x, v[r].x.y, v[r].y.y};   // rows r0 .. r0 + 3
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (k < rows) dst[(size_t)k * a.out_pitch + L * r] = to_store<OutT>(e[k] * a.store_scale);
    }
}

constexpr long long kManyRows = 16384;

template <int M, bool HALF, typename InT, typename OutT>
int launch_rf(const InT* raw, OutT* out, const FilterArgs& a, const float2* tw, const float* K, cudaStream_t s) {
    using C = RF<M>;
    // Low detectors whose last group of a view would hold two rows are filtered two views
    // at a time, as views of twice the rows (the weight table repeats for them; the pairs
    // of rows that share a transform stay the same). 20000 views of 512 x 2: 98 -> 57 us, of
    // 512 x 6 195 -> 156. An odd view left over goes by a launch of its own, where that is
    // little beside the rest.
    const bool two = weight_rows(a.H) > a.H && a.n_views > 1 && (a.n_views % 2 == 0 || a.n_views * a.H > kManyRows);
    if (two && a.n_views % 2) {
        FilterArgs last = a;
        last.n_views = 1;
        const size_t rows = size_t(a.n_views - 1) * a.H;
        if (const int st = launch_rf<M, HALF>(raw + rows * a.W, out + rows * a.out_pitch, last, tw, K, s)) return st;
    }
    FilterArgs b = a;
    if (two) {
        b.H = 2 * a.H;
        b.n_views = a.n_views / 2;
    }
    const long long quads = b.n_views * ((b.H + 3) / 4);
    const long long blocks = (quads + C::G - 1) / C::G;
    if (blocks <= 0) return CTB_OK;
    if (blocks > 0x7fffffffLL) {
        set_global_error("filter: too many rows for one launch");
        return CTB_ERR_UNSUPPORTED;
    }
    const size_t smem = size_t(C::G) * C::SG * sizeof(float4);
    auto kern = filter_rf_kernel<M, HALF, InT, OutT>;
    if (const int st = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem)) return st;
    kern<<<unsigned(blocks), C::T, smem, s>>>(raw, out, b, tw, K);
    return cuda_status(cudaGetLastError(), "filter_rf_kernel launch");
}

// whole rows of a power-of-two width, or rows embedded in a transform at least twice as long
template <int M, typename InT, typename OutT>
int launch_rf_any(const InT* raw, OutT* out, const FilterArgs& a, const float2* tw, const float* K, cudaStream_t s) {
    return a.W == M ? launch_rf<M, false>(raw, out, a, tw, K, s) : launch_rf<M, true>(raw, out, a, tw, K, s);
}

template <typename InT, typename OutT>
int launch_typed(const InT* raw, OutT* out, const FilterArgs& a, const float2* tw, const float* K,
                 cudaStream_t s) {
    const int TG = a.M / 8;
    const int groups = TG >= 256 ? 1 : 256 / TG;
    const int threads = groups * TG;
    const long long pairs = a.n_views * ((a.H + 1) / 2);
    const long long blocks = (pairs + groups - 1) / groups;
    const size_t smem = (size_t)groups * a.M * sizeof(float2);
    if (blocks <= 0) return CTB_OK;
    if (blocks > 0x7fffffffLL) {
        set_global_error("filter: too many rows for one launch");
        return CTB_ERR_UNSUPPORTED;
    }
    const bool tab = a.wt != nullptr;
    // the register kernel's logarithm takes normal positive numbers: samples of 8 and 16
    // bits give arguments from beta to (1 + beta) times the scale, so any but those of a
    // negative or extreme base intensity; float samples are looked at one by one
    const bool normal = std::is_same<InT, float>::value || (a.beta > 0.0f && a.log_scale > 0.0f &&
                                                            a.beta * a.log_scale > 1e-30f && a.log_scale < 1e30f);
    if (tab && normal && (a.W == a.M || 2 * a.W <= a.M)) {
        switch (a.M) {
            case 256: return launch_rf_any<256>(raw, out, a, tw, K, s);
            case 512: return launch_rf_any<512>(raw, out, a, tw, K, s);
            case 1024: return launch_rf_any<1024>(raw, out, a, tw, K, s);
            case 2048: return launch_rf_any<2048>(raw, out, a, tw, K, s);
            case 4096: return launch_rf_any<4096>(raw, out, a, tw, K, s);
        }
    }
    auto kern = tab ? filter_kernel<InT, OutT, true> : filter_kernel<InT, OutT, false>;
    if (smem > 48 * 1024)
        if (const int st = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), smem)) return st;
    kern<<<unsigned(blocks), threads, smem, s>>>(raw, out, a, tw, K);
    return cuda_status(cudaGetLastError(), "filter_kernel launch");
}

template <typename InT>
int launch_out(const InT* raw, void* out, int store_type, const FilterArgs& a, const float2* tw,
               const float* K, cudaStream_t s) {
    switch (store_type) {
        case CTB_FP32: return launch_typed(raw, (float*)out, a, tw, K, s);
        case CTB_FP16: return launch_typed(raw, (__half*)out, a, tw, K, s);
        case CTB_BF16: return launch_typed(raw, (__nv_bfloat16*)out, a, tw, K, s);
    }
    set_global_error("filter: unknown storage type");
    return CTB_ERR_ARG;
}

}  // namespace

int filter_transform_length(int W, int pad) {
    if (W < 2) return 0;
    auto nextpow2 = [](long long n) { long long m = 1; while (m < n) m <<= 1; return m; };
    long long M;
    if (pad <= 1) M = ((W & (W - 1)) == 0) ? W : nextpow2(2LL * W - 1);
    else M = nextpow2(2LL * W);
    if (M < 8) M = 8;
    return M > kMaxFftLen ? 0 : int(M);
}

int filter_twiddle_count(int M) { return M >= 256 && M <= 4096 ? 2 * M + M / 16 : M; }

int filter_build_tables(int W, int pad, int filter, int M, float2* tw, float* K, cudaStream_t s) {
    const int T = 256;
    twiddle_kernel<<<(M + T - 1) / T, T, 0, s>>>(tw, M);
    CTB_CUDA_TRY(cudaGetLastError());
    if (filter_twiddle_count(M) > M) {
        twiddle_order_kernel<<<(M + M / 16 + T - 1) / T, T, 0, s>>>(tw, M);
        CTB_CUDA_TRY(cudaGetLastError());
    }
    if (pad >= 2) {
        kernel_padded<<<(M + T - 1) / T, T, 0, s>>>(K, M, W, filter);
    } else if (M == W) {
        kernel_direct<<<(M + T - 1) / T, T, 0, s>>>(K, M, filter);
    } else {
        double* g = nullptr;
        CTB_CUDA_TRY(cudaMallocAsync((void**)&g, sizeof(double) * W, s));
        spatial_kernel<<<(W + T - 1) / T, T, 0, s>>>(g, W, filter);
        embedded_kernel<<<(M + T - 1) / T, T, 0, s>>>(K, g, W, M);
        CTB_CUDA_TRY(cudaFreeAsync(g, s));
    }
    return cuda_status(cudaGetLastError(), "filter table kernels");
}

FilterArgs filter_args(const ctb_detector& det, int raw_type, int M, int logM, long long n_views,
                       float store_scale) {
    FilterArgs a;
    a.W = det.width;
    a.H = det.height;
    a.M = M;
    a.logM = logM;
    a.n_views = n_views;
    const double base = det.base_intensity;
    a.alpha = float(raw_type == CTB_U8 ? 1.0 / 255.0 : 1.0 / 65535.0);
    a.beta = float(0.000001 * base);
    a.log_scale = float(1.0 / (base + 0.000001 * base));
    a.D = det.fcd;
    a.uPre = float(double(det.width) / 2.0);
    a.vPre = float(double(det.height) / 2.0);
    a.store_scale = store_scale;
    a.out_pitch = det.width;
    return a;
}

namespace {
__global__ void weight_table_kernel(float* t, FilterArgs a) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const int r = blockIdx.y;
    if (c >= a.W) return;
    t[(size_t)r * a.W + c] = weight_part(r % a.H, c, a);
}
}  // namespace

int build_weight_table(const FilterArgs& a, float* t, cudaStream_t s) {
    if (a.H > 65535) return CTB_ERR_UNSUPPORTED;
    weight_table_kernel<<<dim3((a.W + 255) / 256, weight_rows(a.H)), 256, 0, s>>>(t, a);
    return cuda_status(cudaGetLastError(), "weight_table_kernel launch");
}

int filter_launch(const void* raw, int raw_type, void* out, int store_type, const FilterArgs& args,
                  const float2* tw, const float* K, cudaStream_t s) {
    FilterArgs a = args;
    std::shared_ptr<const void> pin;   // the weight table stays until the kernel is launched
    if (!a.wt) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        cudaGraph_t graph = nullptr;
        if (cudaStreamGetCaptureInfo(s, &cs, nullptr, &graph) != cudaSuccess) cudaGetLastError();
        const int st = pre_tables(&a, s, cs == cudaStreamCaptureStatusNone, &pin);
        if (st != CTB_OK) return st;
        // a graph reads the table at every launch
        if (graph && a.wt && !keep_for_graph(graph, pin)) a.wt = nullptr;
    }
    switch (raw_type) {
        case CTB_U8: return launch_out((const uint8_t*)raw, out, store_type, a, tw, K, s);
        case CTB_U16: return launch_out((const uint16_t*)raw, out, store_type, a, tw, K, s);
        case CTB_F32: return launch_out((const float*)raw, out, store_type, a, tw, K, s);
    }
    set_global_error("filter: unknown raw pixel type");
    return CTB_ERR_ARG;
}

}  // namespace ctb
