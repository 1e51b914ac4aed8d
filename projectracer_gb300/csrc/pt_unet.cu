// pt_unet.cu -- learned psi guess (no reference counterpart): the U-Net whose convolutions run on the
// tcgen05 tensor cores (pt_conv.cuh), the GEMM tile's self-check entry point, and the engine side.
#include <cuda.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "pt_internal.h"
#include "../../include/ptgpu_unet.h"
#include "pt_conv.cuh"
#include "pt_launch.cuh"
#include <cuda_bf16.h>

namespace pt {

// plain GEMM problem: C (M x N, FP32) = A (M x K) * B (N x K)^T, BF16 row-major operands
struct GemmProb {
    int M, N, K, Ntile, kc_split;
    const uint16_t* A;
    const uint16_t* B;
    float* C;
    __device__ __forceinline__ uint16_t gather_a(int r, int k) const {
        return (r < M && k < K) ? A[(size_t)r * K + k] : (uint16_t)0;
    }
    __device__ __forceinline__ uint16_t gather_b(int c, int k) const { return k < K ? B[(size_t)c * K + k] : (uint16_t)0; }
    __device__ __forceinline__ void store(int r, int c, int, float v) const { C[(size_t)r * N + c] = v; }
};


static inline unsigned nblk(size_t n, unsigned b) { return (unsigned)((n + b - 1) / b); }

// ============================================================================ U-Net kernels
using tc::PadGeo;
__device__ __forceinline__ uint16_t f2bf(float f) { return __bfloat16_as_ushort(__float2bfloat16_rn(f)); }
__device__ __forceinline__ float bf2f(uint16_t b) { return __uint_as_float((uint32_t)b << 16); }
// 8 BF16 values at a 16-byte-aligned address
__device__ __forceinline__ uint4 ld8(const uint16_t* p) { return *reinterpret_cast<const uint4*>(p); }
__device__ __forceinline__ void st8(uint16_t* p, const uint16_t (&h)[8]) {
    uint32_t w[4];
#pragma unroll
    for (int j = 0; j < 4; j++) w[j] = (uint32_t)h[2 * j] | ((uint32_t)h[2 * j + 1] << 16);
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void unpack8(const uint4& v, float (&f)[8]) {
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 8; j++) f[j] = bf2f((uint16_t)(w[j >> 1] >> (16 * (j & 1))));
}

constexpr int kImCols = 64;  // columns of the first layer's im2col rows: 36 values (tap, channel), zeros

// 32 bytes in one store: whole sectors, where 16-byte stores of a row per thread are halves of them
__device__ __forceinline__ void st32(void* p, const uint32_t (&h)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"l"(p), "r"(h[0]), "r"(h[1]), "r"(h[2]), "r"(h[3]),
                 "r"(h[4]), "r"(h[5]), "r"(h[6]), "r"(h[7])
                 : "memory");
}
// the network input, NCHW FP32, as im2col rows in BF16 at the padded positions, a pixel per thread (columns
// 40..63 stay zero from allocation).  Bound by its 128-byte rows: with a thread per 8 columns, half-sector
// stores and 64-bit divisions 77 us for 8 images of 512 x 256, now 33.
__global__ void __launch_bounds__(256) k_im2col(uint16_t* __restrict__ o, const float* __restrict__ x, PadGeo g) {
    pdl_begin();
    const unsigned q = blockIdx.x * blockDim.x + threadIdx.x;  // (positions fit in 31 bits)
    if (q >= (unsigned)g.B * g.H * g.W) return;
    const unsigned row = q / (unsigned)g.W;
    const int px = (int)(q - row * (unsigned)g.W), b = (int)(row / (unsigned)g.H), py = (int)(row - (unsigned)(b * g.H));
    const size_t plane = (size_t)g.H * g.W;
    const float* in = x + (size_t)b * 4 * plane + (size_t)py * g.W + px;
    float v[40];  // 4 tap + channel
#pragma unroll
    for (int t = 0; t < 9; t++) {
        const int y = py + t / 3 - 1, xx = px + t % 3 - 1;
        const bool in_image = y >= 0 && y < g.H && xx >= 0 && xx < g.W;
#pragma unroll
        for (int c = 0; c < 4; c++)
            v[4 * t + c] = in_image ? in[c * plane + (ptrdiff_t)(t / 3 - 1) * g.W + (t % 3 - 1)] : 0.f;
    }
#pragma unroll
    for (int c = 36; c < 40; c++) v[c] = 0.f;
    uint16_t* const out = o + g.at(b, py, px) * kImCols;
#pragma unroll
    for (int j = 0; j < 32; j += 16) {
        uint32_t h[8];
#pragma unroll
        for (int e = 0; e < 8; e++) h[e] = (uint32_t)f2bf(v[j + 2 * e]) | (uint32_t)f2bf(v[j + 2 * e + 1]) << 16;
        st32(out + j, h);
    }
    uint16_t h[8];
#pragma unroll
    for (int e = 0; e < 8; e++) h[e] = f2bf(v[32 + e]);
    st8(out + 32, h);
}

// pixel and channel octet of element q of a batch's real pixels, pixels within octets of a row adjacent; in
// 32 bits where q fits (64-bit divisions are several times as long)
template <class I>
__device__ __forceinline__ bool octet_of(I q, const PadGeo& g, int C, int& b, int& y, int& x, int& c) {
    const I noct = (I)(C >> 3), W = (I)g.W, H = (I)g.H;
    I r = q / noct;
    c = (int)(q - r * noct) * 8;
    const I row = r / W;
    x = (int)(r - row * W);
    const I im = row / H;
    y = (int)(row - im * H);
    b = (int)im;
    return im < (I)g.B;
}
__device__ __forceinline__ bool octet(size_t q, const PadGeo& g, int C, int& b, int& y, int& x, int& c) {
    return q >> 32 ? octet_of(q, g, C, b, y, x, c) : octet_of((unsigned)q, g, C, b, y, x, c);
}

// 2x2 average of a tensor at twice the resolution, ((a+b)+c)+d in FP32
__global__ void k_pool(uint16_t* __restrict__ o, const uint16_t* __restrict__ in, PadGeo g, PadGeo gf, int C) {
    pdl_begin();
    int b, y, x, c;
    if (!octet((size_t)blockIdx.x * blockDim.x + threadIdx.x, g, C, b, y, x, c)) return;
    const uint16_t* p = in + gf.at(b, 2 * y, 2 * x) * C + c;
    const size_t row = (size_t)gf.Wp() * C;
    float a[8], e[8], d[8], f[8];
    unpack8(ld8(p), a);
    unpack8(ld8(p + C), e);
    unpack8(ld8(p + row), d);
    unpack8(ld8(p + row + C), f);
    uint16_t h[8];
#pragma unroll
    for (int j = 0; j < 8; j++) h[j] = f2bf((((a[j] + e[j]) + d[j]) + f[j]) * 0.25f);
    st8(o + g.at(b, y, x) * C + c, h);
}

// epilogue of the forward GEMM: bias, ReLU, BF16; the nearest-neighbour upsampled copy beside it
// where the next layer reads that
struct FwdEpi {
    static constexpr bool kSums = false;
    static constexpr float* part = nullptr;
    uint16_t* out;
    const float* bias;
    int C;
    uint16_t* up;
    PadGeo gup;
    // the last layer: the 1x1 output convolution (linear, FP32 out), its weights and bias, [B][H][W] of g
    float* y;
    const float *ow, *ob;
    PadGeo g;
    __device__ __forceinline__ void stage(float* sb, int n, int tid) const {
        for (int c = tid; c < n; c += tc::kConvThreads) sb[c] = bias[c];
        if (y && tid <= 32) sb[32 + tid] = tid < 32 ? ow[tid] : ob[0];  // (n = 32)
    }
    __device__ __forceinline__ void operator()(int p, int b, int py, int x, int c0, const float (&v)[32],
                                               const float* sb) const {
        float s = y ? sb[64] : 0.f;
#pragma unroll
        for (int j = 0; j < 32; j += 16) {
            uint32_t h[8];
#pragma unroll
            for (int e = 0; e < 8; e++)
                h[e] = (uint32_t)f2bf(fmaxf(v[j + 2 * e] + sb[j + 2 * e], 0.f)) |
                       (uint32_t)f2bf(fmaxf(v[j + 2 * e + 1] + sb[j + 2 * e + 1], 0.f)) << 16;
            st32(out + (size_t)p * C + c0 + j, h);
            if (y)
#pragma unroll
                for (int c = 0; c < 16; c++) s += bf2f((uint16_t)(h[c >> 1] >> (16 * (c & 1)))) * sb[32 + j + c];
            if (up)
                for (int q = 0; q < 4; q++) st32(up + gup.at(b, 2 * py + (q >> 1), 2 * x + (q & 1)) * C + c0 + j, h);
        }
        if (y) y[((size_t)b * g.H + py) * g.W + x] = s;
    }
    __device__ __forceinline__ void sums(int, bool, int, const float (&)[32], float*) const {}
};
// epilogue of the backward-data GEMM: the view's gradient in FP32 at the padded positions
struct DxEpi {
    static constexpr bool kSums = false;
    static constexpr float* part = nullptr;
    float* dx;
    int N;
    __device__ __forceinline__ void stage(float*, int, int) const {}
    __device__ __forceinline__ void operator()(int p, int, int, int, int c0, const float (&v)[32], const float*) const {
        float* o = dx + (size_t)p * N + c0;
#pragma unroll
        for (int j = 0; j < 32; j += 8) {
            uint32_t h[8];
#pragma unroll
            for (int e = 0; e < 8; e++) h[e] = __float_as_uint(v[j + e]);
            st32(o + j, h);
        }
    }
    __device__ __forceinline__ void sums(int, bool, int, const float (&)[32], float*) const {}
};
// epilogue of the backward-data GEMM of a view that is a layer's output itself: that layer's dZ (the
// gradient masked by Y > 0, in BF16) and the column sums of its bias gradient, without a pass over the
// gradient in FP32
struct DzEpi {
    static constexpr bool kSums = true;
    const uint16_t* Y;
    uint16_t* dZ;
    int C;
    float* part;
    __device__ __forceinline__ void stage(float*, int, int) const {}
    __device__ __forceinline__ void operator()(int, int, int, int, int, const float (&)[32], const float*) const {}
    __device__ __forceinline__ void sums(int p, bool real, int c0, const float (&v)[32], float* sum) const {
        const size_t o = (size_t)p * C + c0;
        float g[32];
#pragma unroll
        for (int j = 0; j < 32; j += 16) {
            float y[16];
            if (real) {
                float (&y0)[8] = reinterpret_cast<float (&)[8]>(y[0]);
                float (&y1)[8] = reinterpret_cast<float (&)[8]>(y[8]);
                unpack8(ld8(Y + o + j), y0);
                unpack8(ld8(Y + o + j + 8), y1);
            }
#pragma unroll
            for (int e = 0; e < 16; e++) g[j + e] = real && y[e] > 0.f ? v[j + e] : 0.f;
            uint32_t h[8];
#pragma unroll
            for (int e = 0; e < 8; e++) h[e] = (uint32_t)f2bf(g[j + 2 * e]) | (uint32_t)f2bf(g[j + 2 * e + 1]) << 16;
            if (real) st32(dZ + o + j, h);
        }
        // lane l: the sum of column l over the warp's rows (halves exchanged, then quarters, ...)
        const int lane = threadIdx.x & 31;
#pragma unroll
        for (int w = 16; w > 0; w >>= 1) {
            const bool up = lane & w;
#pragma unroll
            for (int j = 0; j < w; j++) {
                const float other = __shfl_xor_sync(0xffffffffu, up ? g[j] : g[j + w], w);
                g[j] = (up ? g[j + w] : g[j]) + other;
            }
        }
        sum[c0 + lane] += g[0];
    }
};

// the convolutions' weights in the layouts that only the GEMMs use: wbd[ci][t][co] = w[co][8 - t][ci] (the
// K order of the backward-data GEMM), and the first layer's rows padded to the im2col width
struct PackArgs {
    int cin[14], cout[14];
    size_t woff[14];
};
__global__ void k_pack_weights(uint16_t* __restrict__ wbd, uint16_t* __restrict__ w0, const uint16_t* __restrict__ w,
                               PackArgs a) {
    const int l = blockIdx.y, cin = a.cin[l], cout = a.cout[l];
    const uint16_t* wl = w + a.woff[l];
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < cin * 9 * cout; q += gridDim.x * blockDim.x) {
        if (l == 0) {
            w0[q / 36 * kImCols + q % 36] = wl[q];
        } else {
            const int co = q % cout, t = q / cout % 9, ci = q / (9 * cout);
            wbd[a.woff[l] + q] = wl[((size_t)co * 9 + (8 - t)) * cin + ci];
        }
    }
}

// All layers' weight gradients from the splits' partial sums, dW[co][kk] = sum_z part[z][kk][co]: a warp adds
// every eighth split of 128 weights (four a lane, four loads in flight), then the eight sums are added in
// order; with two sources the rows' channels below c0 have ns0 partial sums, the others ns1.  One launch for
// the network: a launch per layer lasted longer than its reads.  8 images of 512 x 256: 114 us with one weight
// a lane, now 51.
struct ReduceArgs {
    struct Layer {
        float* dW;
        const float* part;
        int ns0, ns1, c0, cin, M, N, block0;  // block0: its first block
    } l[14];
};
constexpr int kReduce = 128;  // weights of a block (a layer's count, 9 cin cout, is a multiple)
__global__ void __launch_bounds__(256) k_wgrad_reduce(const __grid_constant__ ReduceArgs a) {
    pdl_begin();
    __shared__ float4 sh[8][32];
    int li = 13;
    while (li > 0 && (int)blockIdx.x < a.l[li].block0) li--;
    const ReduceArgs::Layer& L = a.l[li];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int q = ((int)blockIdx.x - L.block0) * kReduce + 4 * lane, kk = q / L.N, co = q - kk * L.N;  // N % 32 == 0
    const int ns = kk % L.cin < L.c0 ? L.ns0 : L.ns1;
    const size_t ld = (size_t)L.M * L.N;
    const float* part = L.part + q;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    auto add = [&](const float4& v) {
        s.x += v.x;
        s.y += v.y;
        s.z += v.z;
        s.w += v.w;
    };
    int z = warp;
    for (; z + 24 < ns; z += 32) {
        float4 v[4];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = *reinterpret_cast<const float4*>(part + (size_t)(z + 8 * j) * ld);
#pragma unroll
        for (int j = 0; j < 4; j++) add(v[j]);
    }
    for (; z < ns; z += 8) add(*reinterpret_cast<const float4*>(part + (size_t)z * ld));
    sh[warp][lane] = s;
    __syncthreads();
    if (warp) return;
#pragma unroll
    for (int j = 1; j < 8; j++) add(sh[j][lane]);
    float* const o = L.dW + (size_t)co * L.M + kk;
    o[0] = s.x;
    o[L.M] = s.y;
    o[2 * L.M] = s.z;
    o[3 * L.M] = s.w;
}

// Gradient of a layer's pre-activation as a GEMM operand, dZ = dY masked by Y > 0 in BF16, and per-block
// partial sums of its bias gradient (of the FP32 dY).  dY is where the gradient of the view that read
// the layer's output comes from:
//   pooled  the skip connection's share plus a quarter of the pooled pixel's
//   up      the sum of the four fine pixels, ((a+b)+c)+d
//   out     the output layer: dy w[c]; the partial sums of its own weights' gradients too
// One pass over the tensor, bound by its bytes (FP32 in, two BF16 tensors in and out).
enum { kDzPooled, kDzUp, kDzOut };
constexpr int kDzThreads = 256, kDzBlocks = 4 * tc::kSms;
struct DzArgs {
    PadGeo g, g2;  // of the layer, and of the other resolution (pooled: coarse, up: fine)
    int C;
    const uint16_t* Y;
    uint16_t* dZ;
    const float* dx;  // gradient of the view (out: dy)
    int ldx;          // its channels
    const float* skip;  // pooled: the skip connection's view gradient, its channels and the offset in them
    int lds, offs;
    const float* w;  // out: weights
    float* part;     // [block][C], out: [block][2 C + 1] with the weights' and the bias' sums behind
};
template <int MODE>
__global__ void __launch_bounds__(kDzThreads) k_dz(DzArgs a) {
    pdl_begin();
    constexpr int NV = MODE == kDzOut ? 2 : 1;
    __shared__ float sh[NV * 8][kDzThreads + 1];
    __shared__ float shb[kDzThreads];
    const int noct = a.C >> 3;
    const size_t total = (size_t)a.g.B * a.g.H * a.g.W * noct;
    float sum[8] = {}, wsum[8] = {}, bsum = 0.f;
    // the stride is a multiple of noct: a thread keeps its channels
    for (size_t q = (size_t)blockIdx.x * kDzThreads + threadIdx.x; q < total; q += (size_t)gridDim.x * kDzThreads) {
        int b, y, x, c;
        octet(q, a.g, a.C, b, y, x, c);
        const size_t p = a.g.at(b, y, x);
        float g[8], act[8];
        unpack8(ld8(a.Y + p * a.C + c), act);
        auto load = [&](const float* f, float (&v)[8]) {
            const float4 u = *reinterpret_cast<const float4*>(f), w = *reinterpret_cast<const float4*>(f + 4);
            v[0] = u.x; v[1] = u.y; v[2] = u.z; v[3] = u.w; v[4] = w.x; v[5] = w.y; v[6] = w.z; v[7] = w.w;
        };
        if (MODE == kDzPooled) {
            float d[8];
            load(a.skip + p * a.lds + a.offs + c, g);
            load(a.dx + a.g2.at(b, y >> 1, x >> 1) * a.ldx + c, d);
#pragma unroll
            for (int j = 0; j < 8; j++) g[j] += 0.25f * d[j];
        } else if (MODE == kDzUp) {
            const float* f = a.dx + a.g2.at(b, 2 * y, 2 * x) * a.ldx + c;
            const size_t row = (size_t)a.g2.Wp() * a.ldx;
            float d[8], e[8], h[8];
            load(f, g);
            load(f + a.ldx, d);
            load(f + row, e);
            load(f + row + a.ldx, h);
#pragma unroll
            for (int j = 0; j < 8; j++) g[j] = ((g[j] + d[j]) + e[j]) + h[j];
        } else {
            const float dy = a.dx[((size_t)b * a.g.H + y) * a.g.W + x];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                g[j] = dy * a.w[c + j];
                wsum[j] += dy * act[j];
            }
            if (c == 0) bsum += dy;
        }
        uint16_t h[8];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const bool pos = act[j] > 0.f;
            h[j] = pos ? f2bf(g[j]) : (uint16_t)0;
            if (pos) sum[j] += g[j];
        }
        st8(a.dZ + p * a.C + c, h);
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
        sh[j][threadIdx.x] = sum[j];
        if (NV == 2) sh[8 * (NV - 1) + j][threadIdx.x] = wsum[j];
    }
    shb[threadIdx.x] = bsum;
    __syncthreads();
    // threads of equal channels, in ascending order
    const int nout = NV * a.C + (MODE == kDzOut ? 1 : 0);
    for (int o = threadIdx.x; o < nout; o += kDzThreads) {
        float s = 0.f;
        if (o == NV * a.C) {
            for (int t = 0; t < kDzThreads; t++) s += shb[t];
        } else {
            const int v = o / a.C, c = o - v * a.C;
            for (int t = c >> 3; t < kDzThreads; t += noct) s += sh[8 * v + (c & 7)][t];
        }
        a.part[(size_t)blockIdx.x * nout + o] = s;
    }
}
// All layers' bias gradients (and the output layer's weights and bias) from the blocks' partial sums: a warp
// per column, lanes over blocks, then a fixed shuffle tree
struct ColsumArgs {
    struct Layer {
        float* out;
        const float* part;
        int blocks, ld, off, n, col0;  // col0: its first column among all
    } l[15];
    int total;
};
__global__ void __launch_bounds__(128) k_colsum(const __grid_constant__ ColsumArgs a) {
    pdl_begin();
    const int col = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (col >= a.total) return;
    int li = 14;
    while (li > 0 && col < a.l[li].col0) li--;
    const ColsumArgs::Layer& L = a.l[li];
    const int c = col - L.col0;
    float s = 0.f;
    for (int b = lane; b < L.blocks; b += 32) s += L.part[(size_t)b * L.ld + L.off + c];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) L.out[c] = s;
}

// loss = mean (y - t)^2; dy = 2 (y - t) / P; per-block partial sums of (y - t)^2
__global__ void k_mse(float* dy, float* lpart, const float* y, const float* t, int P) {
    pdl_begin();
    __shared__ float sh[256];
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    float e = 0.f;
    if (p < P) {
        const float d = y[p] - t[p];
        dy[p] = 2.f * d / (float)P;
        e = d * d;
    }
    sh[threadIdx.x] = e;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) lpart[blockIdx.x] = sh[0];
}

// Adam on FP32 master weights, with the BF16 copy used by the convolution GEMMs
__global__ void k_adam(float* w, float* m, float* v, uint16_t* wbf, const float* g, size_t n, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) return;
    const float gg = g[q];
    const float mm = b1 * m[q] + (1.f - b1) * gg;
    const float vv = b2 * v[q] + (1.f - b2) * gg * gg;
    m[q] = mm;
    v[q] = vv;
    const float wn = w[q] - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
    w[q] = wn;
    wbf[q] = f2bf(wn);
}
__global__ void k_to_bf16(uint16_t* o, const float* i, size_t n) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) o[q] = f2bf(i[q]);
}

// ============================================================================ U-Net host side
// 4 levels, base width 32, 3x3 convolutions with ReLU, 2x2 average pooling, nearest upsampling
// with skip concatenation, 1x1 linear output.  Activations BF16 in the padded layout of pt_conv.cuh;
// FP32 master weights with BF16 copies for the tensor-core GEMMs; FP32 gradients; Adam.
struct UConv {
    int src0, src1, mode, cin, cout, level, out;  // src -1 = network input; mode 1 pools src0, 2 upsamples
                                                  // it and appends src1
    size_t woff, boff;                            // in the flat parameter vector
};

// a layer's GEMMs for the current batch size
struct ConvPlan {
    CUtensorMap A[2], B[2];
    tc::ConvArgs a;
    dim3 grid;
};
struct LayerPlan {
    ConvPlan fwd, bwd;
    int nwg = 0, nsplit[2] = {}, c0 = 0;  // weight gradient: sources, their splits, the first one's channels
};

struct UNet {
    int H = 0, W = 0, maxB = 0;
    std::vector<UConv> L;
    int tch[14] = {}, tlev[14] = {};
    size_t nparams = 0, out_w = 0, out_b = 0;
    float *w32 = nullptr, *m = nullptr, *v = nullptr, *g = nullptr;
    uint16_t *wbf = nullptr, *wbd = nullptr, *w0 = nullptr;  // BF16 weights, k_pack_weights' layouts
    int step = 0;
    // padded tensors: im2col input, activations, their pooled and upsampled copies, masked gradients
    uint16_t *im = nullptr, *act[14] = {}, *pool[14] = {}, *up[14] = {}, *dz[14] = {};
    float *dx = nullptr, *dxcat[14] = {};  // a view's gradient; of the concatenated views, kept for the skips
    float *xin = nullptr, *y = nullptr, *dy = nullptr, *tgt = nullptr, *lpart = nullptr, *part = nullptr,
          *bpart = nullptr;
    size_t part_cap = 0, part_off[14] = {}, bpart_off[15] = {};  // of a layer's partial sums in part, in bpart
    int planB = 0;  // batch size of the plans
    LayerPlan plan[14];
    tc::WgradGroup wg;
    int* derr = nullptr;
    cudaStream_t st = nullptr;
    std::vector<void*> owned;
    PadGeo geo(int level, int B) const { return PadGeo{B, H >> level, W >> level}; }
};

static uint64_t splitmix(uint64_t& s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}
static double unit_open(uint64_t& s) { return ((double)(splitmix(s) >> 11) + 0.5) * (1.0 / 9007199254740992.0); }
static double normal01(uint64_t& s) {  // Box-Muller
    const double u1 = unit_open(s), u2 = unit_open(s);
    return std::sqrt(-2.0 * std::log(u1)) * std::cos(6.283185307179586 * u2);
}

template <class T>
static int ualloc(UNet& U, T** p, size_t n) {
    CK(cudaMalloc(p, sizeof(T) * (n ? n : 1)));
    U.owned.push_back(*p);
    CK(cudaMemsetAsync(*p, 0, sizeof(T) * (n ? n : 1), U.st));
    return 0;
}

static int pack_weights(UNet& U) {
    PackArgs a{};
    for (int l = 0; l < 14; l++) {
        a.cin[l] = U.L[l].cin;
        a.cout[l] = U.L[l].cout;
        a.woff[l] = U.L[l].woff;
    }
    k_pack_weights<<<dim3(64, 14), 256, 0, U.st>>>(U.wbd, U.w0, U.wbf, a);
    return cuda_check(cudaGetLastError(), "k_pack_weights");
}

// The shape of a source's weight gradient: columns of a tile, CTAs over blocks of channels and image rows,
// and the splits over the positions: 304 over every 128 of the layer's 9 cin rows, and at least eight chunks
// each.  (The layers share a launch, so a layer alone need not fill the chip: a third as many splits or half as
// many again change the time for 8 images of 512 x 256 by 1 %.  An accumulator's rounding error grows with its
// chain: these lengths are those of the GEMM that gathered its tiles, and the gradients of 12 batches agree
// with its own to 4e-7 to 9e-7, where other lengths leave 4e-6 to 6e-5.)
struct WgradShape {
    int ntile, units, per, ns;
};
static WgradShape wgrad_shape(int taps, int cin, int C, int cout, size_t positions) {
    WgradShape w;
    w.ntile = std::min(cout, 128);
    w.units = C / (C % 64 == 0 ? 64 : 32) * (taps == 1 ? 1 : 3);
    const int chunks = (int)((positions + tc::kWgradK - 1) / tc::kWgradK), rows = (9 * cin + 127) / 128;
    const int n0 = std::max(1, std::min((chunks + 7) / 8, 304 / rows));
    w.per = (chunks + n0 - 1) / n0;
    w.ns = (chunks + w.per - 1) / w.per;
    return w;
}

// where the layers' partial sums of a batch lie in U.part; their total
static size_t layout_partials(UNet& U, int B) {
    size_t n = 0;
    for (size_t li = 0; li < U.L.size(); li++) {
        const UConv& c = U.L[li];
        const int C0 = c.src0 < 0 ? kImCols : U.tch[c.src0], C1 = c.mode == 2 ? U.tch[c.src1] : 0;
        int ns = 0;
        for (int C : {C0, C1})
            if (C) ns = std::max(ns, wgrad_shape(c.src0 < 0 ? 1 : 9, c.cin, C, c.cout, U.geo(c.level, B).positions()).ns);
        U.part_off[li] = n;
        n += (size_t)ns * 9 * c.cin * c.cout;
    }
    return n;
}

static int unet_build(UNet& U, int H, int W, int maxB, uint64_t seed) {
    U.H = H;
    U.W = W;
    U.maxB = maxB;
    // tensor ids: 0 e1a 1 e1 2 e2a 3 e2 4 e3a 5 e3 6 b1 7 b2 8 d3a 9 d3 10 d2a 11 d2 12 d1a 13 d1
    const int spec[14][7] = {{-1, -1, 0, 4, 32, 0, 0},   {0, -1, 0, 32, 32, 0, 1},   {1, -1, 1, 32, 64, 1, 2},
                             {2, -1, 0, 64, 64, 1, 3},   {3, -1, 1, 64, 128, 2, 4},  {4, -1, 0, 128, 128, 2, 5},
                             {5, -1, 1, 128, 256, 3, 6}, {6, -1, 0, 256, 256, 3, 7}, {7, 5, 2, 384, 128, 2, 8},
                             {8, -1, 0, 128, 128, 2, 9}, {9, 3, 2, 192, 64, 1, 10},  {10, -1, 0, 64, 64, 1, 11},
                             {11, 1, 2, 96, 32, 0, 12},  {12, -1, 0, 32, 32, 0, 13}};
    size_t off = 0;
    for (auto& r : spec) {
        UConv c{r[0], r[1], r[2], r[3], r[4], r[5], r[6], 0, 0};
        c.woff = off;
        off += (size_t)c.cout * 9 * c.cin;
        c.boff = off;
        off += c.cout;
        U.L.push_back(c);
        U.tch[c.out] = c.cout;
        U.tlev[c.out] = c.level;
    }
    for (auto& c : U.L)  // the weight boxes start on 16-byte boundaries
        if (c.woff % 8) return fail(PT_ERR_CONFIG, "U-Net: weight offsets must be multiples of 8");
    U.out_w = off;
    off += 32;
    U.out_b = off;
    off += 1;
    U.nparams = off;
    if (U.geo(0, maxB).positions() > (size_t)INT32_MAX / 2) return fail(PT_ERR_ARG, "U-Net: batch of grids too large");
    int rc;
    if ((rc = ualloc(U, &U.w32, off)) || (rc = ualloc(U, &U.m, off)) || (rc = ualloc(U, &U.v, off)) ||
        (rc = ualloc(U, &U.g, off)) || (rc = ualloc(U, &U.wbf, off)) || (rc = ualloc(U, &U.wbd, off)) ||
        (rc = ualloc(U, &U.w0, 32 * kImCols)) || (rc = ualloc(U, &U.derr, 1)))
        return rc;
    // He-normal initialisation from a portable generator; biases zero
    std::vector<float> h(off, 0.f);
    uint64_t sd = seed;
    for (auto& c : U.L) {
        const double sdev = std::sqrt(2.0 / (9.0 * c.cin));
        for (size_t q = 0; q < (size_t)c.cout * 9 * c.cin; q++) h[c.woff + q] = (float)(sdev * normal01(sd));
    }
    for (int q = 0; q < 32; q++) h[U.out_w + q] = (float)(std::sqrt(1.0 / 32.0) * normal01(sd));
    CK(cudaMemcpyAsync(U.w32, h.data(), sizeof(float) * off, cudaMemcpyHostToDevice, U.st));
    k_to_bf16<<<nblk(off, 256), 256, 0, U.st>>>(U.wbf, U.w32, off);
    CK(cudaGetLastError());
    if ((rc = pack_weights(U))) return rc;
    // tensors for maxB samples; their padding stays zero from here on
    auto n = [&](int level, int ch) { return U.geo(level, maxB).positions() * (size_t)ch; };
    size_t dx = 0, part = 0, bpart = 0;
    for (auto& c : U.L) {
        if ((rc = ualloc(U, &U.act[c.out], n(c.level, c.cout))) || (rc = ualloc(U, &U.dz[c.out], n(c.level, c.cout))))
            return rc;
        if (c.mode == 1 && (rc = ualloc(U, &U.pool[c.src0], n(c.level, c.cin)))) return rc;
        if (c.mode == 2) {
            if ((rc = ualloc(U, &U.up[c.src0], n(c.level, U.tch[c.src0]))) ||
                (rc = ualloc(U, &U.dxcat[c.out], n(c.level, c.cin))))
                return rc;
        } else if (c.mode == 1) {
            dx = std::max(dx, n(c.level, c.cin));
        }
    }
    for (int B = 1; B <= maxB; B++)  // (a smaller batch may have more splits)
        part = std::max(part, layout_partials(U, B));
    for (size_t li = 0; li < U.L.size(); li++) {
        U.bpart_off[li] = bpart;
        bpart += (size_t)kDzBlocks * (li == 13 ? 2 * U.L[li].cout + 1 : U.L[li].cout);
    }
    U.part_cap = part;
    const size_t P0 = (size_t)maxB * H * W;
    if ((rc = ualloc(U, &U.im, n(0, kImCols))) || (rc = ualloc(U, &U.xin, P0 * 4)) || (rc = ualloc(U, &U.y, P0)) ||
        (rc = ualloc(U, &U.dy, P0)) || (rc = ualloc(U, &U.tgt, P0)) || (rc = ualloc(U, &U.lpart, P0 / 256 + 1)) ||
        (rc = ualloc(U, &U.dx, dx)) || (rc = ualloc(U, &U.part, part)) || (rc = ualloc(U, &U.bpart, bpart)))
        return rc;
    const int smax = 221 * 1024;  // the rings' bound and the alignment
    CK(cudaFuncSetAttribute(tc::k_conv_gemm<FwdEpi>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax));
    CK(cudaFuncSetAttribute(tc::k_conv_gemm<DxEpi>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax));
    CK(cudaFuncSetAttribute(tc::k_conv_gemm<DzEpi>, cudaFuncAttributeMaxDynamicSharedMemorySize, smax));
    CK(cudaFuncSetAttribute(tc::k_wgrad_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, smax));
    return 0;
}

// 2D tensor map of a row-major BF16 array [rows][C], boxes of boxc (64 or 32) x boxr, swizzled by the box
// row's bytes; rows outside the array read as zero
static int tensor_map(CUtensorMap* m, const uint16_t* base, size_t C, size_t rows, int boxc, int boxr) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static Encode encode = nullptr;
    if (!encode) {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        CK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q));
        if (!f) return fail(PT_ERR_CUDA, "cuTensorMapEncodeTiled is not in this driver");
        encode = reinterpret_cast<Encode>(f);
    }
    const cuuint64_t dims[2] = {C, rows}, strides[1] = {C * 2};
    const cuuint32_t box[2] = {(cuuint32_t)boxc, (cuuint32_t)boxr}, es[2] = {1, 1};
    const CUresult r = encode(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t*>(base), dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE,
                              boxc == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? 0 : fail(PT_ERR_CUDA, "U-Net: tensor map");
}

// the sources of a layer's view as padded tensors
static int view_sources(const UNet& U, const UConv& c, const uint16_t* (&t)[2], int (&C)[2]) {
    C[1] = 0;
    t[1] = nullptr;
    if (c.src0 < 0) {
        t[0] = U.im;
        C[0] = kImCols;
        return 1;
    }
    t[0] = c.mode == 1 ? U.pool[c.src0] : c.mode == 2 ? U.up[c.src0] : U.act[c.src0];
    C[0] = U.tch[c.src0];
    if (c.mode != 2) return 1;
    t[1] = U.act[c.src1];
    C[1] = U.tch[c.src1];
    return 2;
}

// one convolution GEMM: sources t (C channels each), weights w [N][Ktot], over the positions of g.  The
// column tile is the largest that still gives every SM a CTA (at least 32 columns).
static int plan_conv(ConvPlan& P, PadGeo g, int taps, int nsrc, const uint16_t* const* t, const int* C, const uint16_t* w,
                     int N, bool sums) {
    tc::ConvArgs& a = P.a;
    a.g = g;
    a.wp = PadGeo::Div(g.Wp());
    a.hp = PadGeo::Div(g.Hp());
    a.taps = taps;
    a.nsrc = nsrc;
    a.N = N;
    a.Ktot = 0;
    for (int s = 0; s < 2; s++) {
        a.C[s] = C[s];
        a.bw[s] = C[s] % 64 == 0 && C[s] > 0 ? 64 : 32;
        a.Ktot += taps * C[s];
    }
    a.first = g.Wp();
    a.last = (int)((size_t)g.B * g.Hp() * g.Wp());
    const int mt = (a.last - a.first + tc::kTileM - 1) / tc::kTileM;
    int nt = 1;
    while (N / nt > 256 || N % nt || (N / nt) % 32) nt++;
    for (int f = nt + 1; f <= N / 32 && mt * nt < 152; f++)
        if (N % f == 0 && (N / f) % 32 == 0) nt = f;
    a.Ntile = N / nt;
    a.nt = nt;
    a.tiles = mt * nt;
    tc::conv_stages(a, C[0] / a.bw[0] + (nsrc > 1 ? C[1] / a.bw[1] : 0), sums);
    P.grid = dim3(std::min(a.tiles, tc::kSms * a.ctas));
    const int brows = a.nd == 3 ? tc::kBoxRows : tc::kTileM;
    int rc;
    for (int s = 0; s < 2; s++) {
        const int q = s < nsrc ? s : 0;
        if ((rc = tensor_map(&P.A[s], t[q], C[q], g.positions(), a.bw[q], brows)) ||
            (rc = tensor_map(&P.B[s], w, a.Ktot, N, a.bw[q], a.Ntile)))
            return rc;
    }
    return 0;
}

static int plan_batch(UNet& U, int B) {
    if (U.planB == B) return 0;
    U.planB = 0;
    U.wg.n = U.wg.ctas = 0;
    U.wg.smem = 0;
    if (layout_partials(U, B) > U.part_cap) return fail(PT_ERR_STATE, "U-Net: split workspace too small");
    int rc;
    for (size_t li = 0; li < U.L.size(); li++) {
        const UConv& c = U.L[li];
        LayerPlan& P = U.plan[li];
        const PadGeo g = U.geo(c.level, B);
        const uint16_t* t[2];
        int C[2];
        const int ns = view_sources(U, c, t, C);
        const bool first = c.src0 < 0;
        if ((rc = plan_conv(P.fwd, g, first ? 1 : 9, ns, t, C, first ? U.w0 : U.wbf + c.woff, c.cout, false)))
            return rc;
        const uint16_t* z[2] = {U.dz[c.out], nullptr};
        const int Cz[2] = {c.cout, 0};
        if (!first && (rc = plan_conv(P.bwd, g, 9, 1, z, Cz, U.wbd + c.woff, c.cin, c.mode == 0))) return rc;
        P.nwg = ns;
        P.c0 = C[0];
        for (int s = 0; s < ns; s++) {
            tc::WgradGroup::Problem& w = U.wg.p[U.wg.n++];
            tc::WgradArgs& a = w.a;
            const WgradShape sh = wgrad_shape(first ? 1 : 9, c.cin, C[s], c.cout, g.positions());
            P.nsplit[s] = sh.ns;
            a.g = g;
            a.taps = first ? 1 : 9;
            a.C = C[s];
            a.bw = C[s] % 64 == 0 ? 64 : 32;
            a.c_off = s ? C[0] : 0;
            a.cin = first ? 9 * c.cin : c.cin;
            a.kk_max = 9 * c.cin;
            a.N = c.cout;
            a.Ntile = sh.ntile;
            a.bwB = c.cout % 64 == 0 ? 64 : 32;
            a.per = sh.per;
            a.chunks = (int)((g.positions() + tc::kWgradK - 1) / tc::kWgradK);
            a.ncols = (int)tc::tmem_cols((first || a.bw == 32 ? 1 : 2) * a.Ntile);
            a.abytes = tc::wgrad_box_bytes(a.bw);
            a.bbytes = a.Ntile * tc::kWgradK * 2;
            a.part = U.part + U.part_off[li];
            w.first = U.wg.ctas;
            w.gx = sh.units;
            w.gy = c.cout / a.Ntile;
            U.wg.ctas += w.gx * w.gy * sh.ns;
            a.S = std::min(std::min(110 * 1024 / (a.abytes + a.bbytes), tc::kMaxRing), sh.per);  // two CTAs on an SM
            U.wg.smem = std::max(U.wg.smem, tc::wgrad_smem(a));
            if ((rc = tensor_map(&w.A, t[s], C[s], g.positions(), a.bw, tc::kWgradBox)) ||
                (rc = tensor_map(&w.B, U.dz[c.out], c.cout, g.positions(), a.bwB, tc::kWgradK)))
                return rc;
        }
    }
    U.planB = B;
    return 0;
}

template <class E>
static int run_conv(UNet& U, const ConvPlan& P, const E& e) {
    return launch_pdl("k_conv_gemm", tc::k_conv_gemm<E>, P.grid, dim3(tc::kConvThreads), tc::conv_smem(P.a), U.st, P.A[0],
                      P.A[1], P.B[0], P.B[1], P.a, e, U.derr);
}

// network input already in U.xin (device, NCHW FP32); output in U.y ([B][H][W] FP32).
// ev (optional): 15 CUDA events recorded around the 14 convolution GEMMs
static int unet_forward(UNet& U, int B, cudaEvent_t* ev = nullptr) {
    const size_t P0 = (size_t)B * U.H * U.W;
    int rc;
    if ((rc = plan_batch(U, B))) return rc;
    if ((rc = launch_pdl("k_im2col", k_im2col, dim3(nblk(P0, 256)), dim3(256), 0, U.st, U.im, U.xin, U.geo(0, B))))
        return rc;
    int li = 0;
    if (ev) CK(cudaEventRecord(ev[0], U.st));
    for (auto& c : U.L) {
        if (c.mode == 1) {
            const PadGeo g = U.geo(c.level, B);
            const size_t n = (size_t)B * g.H * g.W * (c.cin / 8);
            if ((rc = launch_pdl("k_pool", k_pool, dim3(nblk(n, 256)), dim3(256), 0, U.st, U.pool[c.src0], U.act[c.src0], g,
                                 U.geo(c.level - 1, B), c.cin)))
                return rc;
        }
        const FwdEpi e{U.act[c.out], U.w32 + c.boff, c.cout, U.up[c.out], U.geo(c.level > 0 ? c.level - 1 : 0, B),
                       c.out == 13 ? U.y : nullptr, U.w32 + U.out_w, U.w32 + U.out_b, U.geo(0, B)};
        if ((rc = run_conv(U, U.plan[li].fwd, e))) return rc;
        li++;
        if (ev) CK(cudaEventRecord(ev[li], U.st));
    }
    return 0;
}

static int gemm_error(UNet& U) {
    int herr = 0;
    CK(cudaMemcpyAsync(&herr, U.derr, sizeof(int), cudaMemcpyDeviceToHost, U.st));
    CK(cudaStreamSynchronize(U.st));
    if (herr) return fail(PT_ERR_ITER_CAP, "U-Net tensor-core GEMM: mbarrier wait gave up");
    return 0;
}

static int dz_blocks(const UNet& U, const UConv& c, int B) {
    const size_t oct = (size_t)B * (U.H >> c.level) * (U.W >> c.level) * (c.cout / 8);
    return (int)std::min<size_t>(nblk(oct, kDzThreads), kDzBlocks);
}
// dZ of the layer that produced tensor t from where its gradient lies, and the partial sums of its bias gradient
template <int MODE>
static int run_dz(UNet& U, int t, int B, DzArgs a) {
    const UConv& c = U.L[t];  // (tensor t is layer t's output)
    a.g = U.geo(c.level, B);
    a.C = c.cout;
    a.Y = U.act[t];
    a.dZ = U.dz[t];
    a.part = U.bpart + U.bpart_off[t];
    return launch_pdl("k_dz", k_dz<MODE>, dim3(dz_blocks(U, c, B)), dim3(kDzThreads), 0, U.st, a);
}

// gradients of the MSE loss against U.tgt into U.g; loss on the host
static int unet_backward(UNet& U, int B, float* loss) {
    const int P0 = B * U.H * U.W;
    const int nb = (int)nblk(P0, 256);
    int rc;
    ReduceArgs red{};
    if ((rc = launch_pdl("k_mse", k_mse, dim3(nb), dim3(256), 0, U.st, U.dy, U.lpart, U.y, U.tgt, P0))) return rc;
    DzArgs o{};
    o.dx = U.dy;
    o.w = U.w32 + U.out_w;
    if ((rc = run_dz<kDzOut>(U, 13, B, o))) return rc;
    int bsums[14] = {};  // rows of a layer's bias partial sums
    bsums[13] = dz_blocks(U, U.L[13], B);
    for (int li = (int)U.L.size() - 1; li >= 0; li--) {
        const UConv& c = U.L[li];
        const LayerPlan& P = U.plan[li];
        // weights: split over positions; the splits are added at the end, for all layers
        const int M = 9 * c.cin;
        red.l[li] = {U.g + c.woff, U.part + U.part_off[li], P.nsplit[0], P.nsplit[1], P.nwg > 1 ? P.c0 : M,
                     P.nwg > 1 ? c.cin : M, M, c.cout, 0};
        if (c.src0 < 0) continue;  // the network input needs no gradient
        if (c.mode == 0) {
            const DzEpi e{U.act[c.src0], U.dz[c.src0], c.cin, U.bpart + U.bpart_off[c.src0]};
            if ((rc = run_conv(U, P.bwd, e))) return rc;
            bsums[c.src0] = (int)P.bwd.grid.x;
            continue;
        }
        float* dx = c.mode == 2 ? U.dxcat[c.out] : U.dx;
        if ((rc = run_conv(U, P.bwd, DxEpi{dx, c.cin}))) return rc;
        DzArgs a{};
        a.dx = dx;
        a.ldx = c.cin;
        bsums[c.src0] = dz_blocks(U, U.L[c.src0], B);
        if (c.mode == 2) {
            a.g2 = U.geo(c.level, B);
            rc = run_dz<kDzUp>(U, c.src0, B, a);
        } else {  // the skip connection's share was left by the layer that concatenates this tensor
            a.g2 = U.geo(c.level, B);
            for (auto& q : U.L)
                if (q.src1 == c.src0) {
                    a.skip = U.dxcat[q.out];
                    a.lds = q.cin;
                    a.offs = U.tch[q.src0];
                }
            rc = run_dz<kDzPooled>(U, c.src0, B, a);
        }
        if (rc) return rc;
    }
    int blocks = 0, cols = 0;
    ColsumArgs sum{};
    for (int li = 0; li < 14; li++) {
        const UConv& c = U.L[li];
        red.l[li].block0 = blocks;
        blocks += red.l[li].M * red.l[li].N / kReduce;
        sum.l[li] = {U.g + c.boff, U.bpart + U.bpart_off[li], bsums[li], li == 13 ? 2 * c.cout + 1 : c.cout, 0,
                     c.cout, cols};
        cols += c.cout;
    }
    // (the output layer's weights and bias lie next to each other)
    sum.l[14] = sum.l[13];
    sum.l[14].out = U.g + U.out_w;
    sum.l[14].off = U.L[13].cout;
    sum.l[14].n = U.L[13].cout + 1;
    sum.l[14].col0 = cols;
    sum.total = cols + sum.l[14].n;
    if ((rc = launch_pdl("k_wgrad_gemm", tc::k_wgrad_gemm, dim3(U.wg.ctas), dim3(tc::kWgradThreads), U.wg.smem, U.st, U.wg,
                         U.derr)) ||
        (rc = launch_pdl("k_wgrad_reduce", k_wgrad_reduce, dim3(blocks), dim3(256), 0, U.st, red)) ||
        (rc = launch_pdl("k_colsum", k_colsum, dim3(nblk(sum.total, 4)), dim3(128), 0, U.st, sum)))
        return rc;
    std::vector<float> lp(nb);
    CK(cudaMemcpyAsync(lp.data(), U.lpart, sizeof(float) * nb, cudaMemcpyDeviceToHost, U.st));
    if ((rc = gemm_error(U))) return rc;
    double err = 0.0;
    for (float a : lp) err += a;
    if (loss) *loss = (float)(err / P0);
    return 0;
}

static int unet_adam(UNet& U, float lr) {
    U.step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)U.step), c2 = 1.f - std::pow(b2, (float)U.step);
    k_adam<<<nblk(U.nparams, 256), 256, 0, U.st>>>(U.w32, U.m, U.v, U.wbf, U.g, U.nparams, lr, b1, b2, 1e-8f, c1, c2);
    CK(cudaGetLastError());
    return pack_weights(U);
}

// ============================================================================ engine side
// features of node (i, k), i < nx, k < nz, as the network's input planes [4][nz][nx]:
// T, C, log10(eta)/5, RHS/max|RHS| (0 on the boundary rows), and psi/max|psi| (training target)
__global__ void k_absmax_grid(const double* f, Geo g, int nx, int nz, unsigned long long* out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    double a = 0.0;
    if (i <= nx && k <= nz) a = fabs(f[g.at(i, k)]);
    for (int o = 16; o > 0; o >>= 1) a = fmax(a, __shfl_xor_sync(0xffffffffu, a, o));
    if ((threadIdx.x & 31) == 0 && a > 0.0) atomicMax(out, (unsigned long long)__double_as_longlong(a));
}
__global__ void k_features(float* x4, float* psi, const double* Tb, const double* Cb, const double* vis,
                           const double* rhs, const double* sf, Geo g, int nx, int nz, const unsigned long long* scal,
                           int comp) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (i >= nx || k >= nz) return;
    const size_t o = g.at(i, k), plane = (size_t)nx * nz, q = (size_t)k * nx + i;
    const double rmax = __longlong_as_double((long long)scal[0]), smax = __longlong_as_double((long long)scal[1]);
    x4[q] = (float)Tb[o];
    x4[plane + q] = comp ? (float)Cb[o] : 0.f;
    x4[2 * plane + q] = (float)(log10(vis[o]) * 0.2);
    x4[3 * plane + q] = (i > 0 && k > 0 && rmax > 0.0) ? (float)(rhs[o] / rmax) : 0.f;
    if (psi) psi[q] = smax > 0.0 ? (float)(sf[o] / smax) : 0.f;
}
// network output (psi shape, [nz][nx]) into the level-1 iterate: interior nodes, boundary 0
__global__ void k_guess_scatter(double* x, const float* y, Geo g, int nx, int nz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (i > nx || k > nz) return;
    x[g.at(i, k)] = (i > 0 && k > 0 && i < nx && k < nz) ? (double)y[(size_t)k * nx + i] : 0.0;
}
__global__ void k_scale_all(double* x, double a, size_t n) {
    const size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (q < n) x[q] *= a;
}

static int engine_features(Engine& E, float* x4, float* psi) {
    const Geo& g = E.g1;
    const int nx = E.cfg.nx, nz = E.cfg.nz;
    unsigned long long* scal = reinterpret_cast<unsigned long long*>(E.dscal);
    CK(cudaMemsetAsync(scal, 0, 16, E.st));
    dim3 gm(nblk(nx + 1, 128), nz + 1);
    k_absmax_grid<<<gm, 128, 0, E.st>>>(E.RHS[1], g, nx, nz, scal);
    if (psi) k_absmax_grid<<<gm, 128, 0, E.st>>>(E.SF, g, nx, nz, scal + 1);
    k_features<<<dim3(nblk(nx, 128), nz), 128, 0, E.st>>>(x4, psi, E.Tbuoy, E.Cbuoy, E.vis[1], E.RHS[1], E.SF, g, nx, nz,
                                                           scal, E.cfg.comp);
    CK(cudaGetLastError());
    return 0;
}

static int mean_resid(Engine& E, double* ratio) {
    if (int rc = residual_level1(E)) return rc;
    CK(cudaMemcpyAsync(E.hscal, E.dscal + 8, 8, cudaMemcpyDeviceToHost, E.st));
    CK(cudaStreamSynchronize(E.st));
    *ratio = E.hscal[0] / (double)(E.gl[1].nx - 2) / (double)(E.gl[1].nz - 2) / E.res_ref[1];
    return 0;
}

// Learned initial guess.  The network's psi shape g (BF16 output, grid-scale noise of order 1e-3)
// is scaled by the least-squares factor fitted on the coarsest level (coarse_scale_fit) and
// starts the solve.  The residual of the previous psi (the reference's warm start) is kept: if the
// residual after the first full cycle is not below it, the solver falls back to the previous psi
// (unet_check_fallback), so a poor guess costs one cycle.
int unet_guess(Engine& E) {
    E.unet_used = 0;
    if (!E.unet) return 0;
    UNet& U = *static_cast<UNet*>(E.unet_core);
    const Geo& g = E.g1;
    const int nx = E.cfg.nx, nz = E.cfg.nz;
    int rc;
    double r_prev = 0.0, alpha = 0.0;
    if ((rc = mean_resid(E, &r_prev))) return rc;  // err[1] holds the previous psi
    if ((rc = engine_features(E, U.xin, nullptr))) return rc;
    CK(cudaStreamSynchronize(E.st));
    if ((rc = unet_forward(U, 1)) || (rc = gemm_error(U))) return rc;
    k_guess_scatter<<<dim3(nblk(nx + 1, 128), nz + 1), 128, 0, E.st>>>(E.err[1], U.y, g, nx, nz);
    CK(cudaGetLastError());
    if ((rc = enforce_bcs_stream(E, 1, E.err[1])) || (rc = coarse_scale_fit(E, &alpha))) return rc;
    k_scale_all<<<nblk(g.elems(), 256), 256, 0, E.st>>>(E.err[1], alpha, g.elems());
    CK(cudaGetLastError());
    E.unet_r_prev = r_prev;
    E.unet_r_net = 0.0;
    E.unet_used = 1;
    return 0;
}

// Called with the residual ratio measured after the first full cycle from the network's guess:
// falls back to the previous psi when the guess did not lower the residual.  Returns 1 when the
// solve restarts from the previous psi.
int unet_check_fallback(Engine& E, double ratio) {
    if (E.unet_used != 1) return 0;
    E.unet_r_net = ratio;
    if (ratio < E.unet_r_prev) {
        E.unet_used = 2;  // kept; checked
        return 0;
    }
    E.unet_used = 0;
    if (cudaMemcpyAsync(E.err[1], E.SF, E.g1.elems() * sizeof(double), cudaMemcpyDeviceToDevice, E.st) != cudaSuccess)
        return -1;
    return 1;
}

}  // namespace pt

using namespace pt;

extern "C" {

int pt_tc_gemm_check(const uint16_t* A, const uint16_t* B, float* C, int M, int N, int K) {
    if (!A || !B || !C) return fail(PT_ERR_ARG, "null pointer");
    if (M <= 0 || K <= 0 || N < 16 || N > 256 || N % 16) return fail(PT_ERR_ARG, "pt_tc_gemm_check: N must be 16..256, a multiple of 16");
    uint16_t *dA = nullptr, *dB = nullptr;
    float* dC = nullptr;
    int* derr = nullptr;
    int rc = 0, herr = 0;
    const size_t smem = tc::smem_bytes(N);
    auto cleanup = [&]() {
        if (dA) cudaFree(dA);
        if (dB) cudaFree(dB);
        if (dC) cudaFree(dC);
        if (derr) cudaFree(derr);
    };
    if ((rc = cuda_check(cudaMalloc(&dA, sizeof(uint16_t) * (size_t)M * K), "gemm check")) ||
        (rc = cuda_check(cudaMalloc(&dB, sizeof(uint16_t) * (size_t)N * K), "gemm check")) ||
        (rc = cuda_check(cudaMalloc(&dC, sizeof(float) * (size_t)M * N), "gemm check")) ||
        (rc = cuda_check(cudaMalloc(&derr, sizeof(int)), "gemm check")) ||
        (rc = cuda_check(cudaMemcpy(dA, A, sizeof(uint16_t) * (size_t)M * K, cudaMemcpyHostToDevice), "gemm check")) ||
        (rc = cuda_check(cudaMemcpy(dB, B, sizeof(uint16_t) * (size_t)N * K, cudaMemcpyHostToDevice), "gemm check")) ||
        (rc = cuda_check(cudaMemset(derr, 0, sizeof(int)), "gemm check")) ||
        (rc = cuda_check(cudaFuncSetAttribute(tc::k_tc_gemm<GemmProb>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                         "gemm check"))) {
        cleanup();
        return rc;
    }
    GemmProb p{M, N, K, N, 0, dA, dB, dC};
    tc::k_tc_gemm<GemmProb><<<dim3((M + tc::kTileM - 1) / tc::kTileM, 1, 1), tc::kThreads, smem>>>(p, derr);
    rc = cuda_check(cudaGetLastError(), "k_tc_gemm launch");
    if (!rc) rc = cuda_check(cudaDeviceSynchronize(), "k_tc_gemm");
    if (!rc) rc = cuda_check(cudaMemcpy(&herr, derr, sizeof(int), cudaMemcpyDeviceToHost), "gemm check");
    if (!rc) rc = cuda_check(cudaMemcpy(C, dC, sizeof(float) * (size_t)M * N, cudaMemcpyDeviceToHost), "gemm check");
    cleanup();
    if (!rc && herr) rc = fail(PT_ERR_ITER_CAP, "tensor-core GEMM: mbarrier wait gave up");
    return rc;
}

struct pt_unet {
    UNet u;
};

static void unet_release(pt_unet* n) {
    for (void* p : n->u.owned) cudaFree(p);
    if (n->u.st) cudaStreamDestroy(n->u.st);
    delete n;
}

int pt_unet_create(int nz, int nx, int max_batch, uint64_t seed, pt_unet** out) {
    if (!out) return fail(PT_ERR_ARG, "null pointer");
    *out = nullptr;
    if (nz < 8 || nx < 8 || nz % 8 || nx % 8 || max_batch < 1)
        return fail(PT_ERR_ARG, "pt_unet_create: nz and nx must be positive multiples of 8, max_batch >= 1");
    pt_unet* n = new pt_unet();
    int rc = cuda_check(cudaStreamCreateWithFlags(&n->u.st, cudaStreamNonBlocking), "U-Net stream");
    if (!rc) rc = unet_build(n->u, nz, nx, max_batch, seed);
    if (!rc) rc = cuda_check(cudaStreamSynchronize(n->u.st), "U-Net init");
    if (rc) {
        std::string msg = g_err;
        unet_release(n);
        g_err = msg;
        return rc;
    }
    *out = n;
    return 0;
}

int pt_unet_destroy(pt_unet* net) {
    if (net) unet_release(net);
    return 0;
}

int pt_unet_num_params(pt_unet* net, int64_t* n) {
    if (!net || !n) return fail(PT_ERR_ARG, "null pointer");
    *n = (int64_t)net->u.nparams;
    return 0;
}

int pt_unet_get_params(pt_unet* net, float* host) {
    if (!net || !host) return fail(PT_ERR_ARG, "null pointer");
    UNet& U = net->u;
    CK(cudaMemcpyAsync(host, U.w32, sizeof(float) * U.nparams, cudaMemcpyDeviceToHost, U.st));
    CK(cudaStreamSynchronize(U.st));
    return 0;
}

int pt_unet_set_params(pt_unet* net, const float* host) {
    if (!net || !host) return fail(PT_ERR_ARG, "null pointer");
    UNet& U = net->u;
    CK(cudaMemcpyAsync(U.w32, host, sizeof(float) * U.nparams, cudaMemcpyHostToDevice, U.st));
    k_to_bf16<<<nblk(U.nparams, 256), 256, 0, U.st>>>(U.wbf, U.w32, U.nparams);
    CK(cudaGetLastError());
    if (int rc = pack_weights(U)) return rc;
    CK(cudaStreamSynchronize(U.st));
    return 0;
}

static int unet_input(UNet& U, const float* x, int batch) {
    if (batch < 1 || batch > U.maxB) return fail(PT_ERR_ARG, "U-Net: batch outside 1..max_batch");
    CK(cudaMemcpyAsync(U.xin, x, sizeof(float) * (size_t)batch * 4 * U.H * U.W, cudaMemcpyHostToDevice, U.st));
    return 0;
}

int pt_unet_forward(pt_unet* net, const float* x, int batch, float* y) {
    if (!net || !x || !y) return fail(PT_ERR_ARG, "null pointer");
    UNet& U = net->u;
    int rc;
    if ((rc = unet_input(U, x, batch)) || (rc = unet_forward(U, batch))) return rc;
    CK(cudaMemcpyAsync(y, U.y, sizeof(float) * (size_t)batch * U.H * U.W, cudaMemcpyDeviceToHost, U.st));
    return gemm_error(U);
}

int pt_unet_gradients(pt_unet* net, const float* x, const float* target, int batch, float* grads, float* loss) {
    if (!net || !x || !target || !grads) return fail(PT_ERR_ARG, "null pointer");
    UNet& U = net->u;
    int rc;
    if ((rc = unet_input(U, x, batch)) || (rc = unet_forward(U, batch))) return rc;
    CK(cudaMemcpyAsync(U.tgt, target, sizeof(float) * (size_t)batch * U.H * U.W, cudaMemcpyHostToDevice, U.st));
    if ((rc = unet_backward(U, batch, loss))) return rc;
    CK(cudaMemcpyAsync(grads, U.g, sizeof(float) * U.nparams, cudaMemcpyDeviceToHost, U.st));
    CK(cudaStreamSynchronize(U.st));
    return 0;
}

int pt_unet_train_step(pt_unet* net, const float* x, const float* target, int batch, float lr, float* loss) {
    if (!net || !x || !target) return fail(PT_ERR_ARG, "null pointer");
    UNet& U = net->u;
    int rc;
    if ((rc = unet_input(U, x, batch)) || (rc = unet_forward(U, batch))) return rc;
    CK(cudaMemcpyAsync(U.tgt, target, sizeof(float) * (size_t)batch * U.H * U.W, cudaMemcpyHostToDevice, U.st));
    if ((rc = unet_backward(U, batch, loss)) || (rc = unet_adam(U, lr))) return rc;
    CK(cudaStreamSynchronize(U.st));
    return 0;
}

int pt_unet_save(pt_unet* net, const char* path) {
    if (!net || !path) return fail(PT_ERR_ARG, "null pointer");
    UNet& U = net->u;
    std::vector<float> h(U.nparams);
    if (int rc = pt_unet_get_params(net, h.data())) return rc;
    FILE* f = std::fopen(path, "wb");
    if (!f) return fail(PT_ERR_ARG, std::string("cannot write ") + path);
    const int32_t dims[2] = {U.H, U.W};
    const int64_t n = (int64_t)U.nparams;
    bool ok = std::fwrite("PTUNET01", 1, 8, f) == 8 && std::fwrite(dims, 4, 2, f) == 2 && std::fwrite(&n, 8, 1, f) == 1 &&
              std::fwrite(h.data(), 4, h.size(), f) == h.size();
    ok = (std::fclose(f) == 0) && ok;
    return ok ? 0 : fail(PT_ERR_ARG, std::string("short write to ") + path);
}

int pt_unet_load(const char* path, int nz, int nx, int max_batch, pt_unet** out) {
    if (!path || !out) return fail(PT_ERR_ARG, "null pointer");
    *out = nullptr;
    FILE* f = std::fopen(path, "rb");
    if (!f) return fail(PT_ERR_ARG, std::string("cannot read ") + path);
    char magic[8];
    int32_t dims[2];
    int64_t n = 0;
    bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, "PTUNET01", 8) == 0 && std::fread(dims, 4, 2, f) == 2 &&
              std::fread(&n, 8, 1, f) == 1 && n > 0 && n < ((int64_t)1 << 30);
    std::vector<float> h(ok ? (size_t)n : 0);
    ok = ok && std::fread(h.data(), 4, h.size(), f) == h.size();
    std::fclose(f);
    if (!ok) return fail(PT_ERR_ARG, std::string("not a U-Net weight file: ") + path);
    int rc = pt_unet_create(nz, nx, max_batch, 0, out);
    if (rc) return rc;
    if ((int64_t)(*out)->u.nparams != n) {
        pt_unet_destroy(*out);
        *out = nullptr;
        return fail(PT_ERR_ARG, "U-Net weight file has a different parameter count");
    }
    return pt_unet_set_params(*out, h.data());
}

int pt_unet_profile_forward(pt_unet* net, const float* x, int batch, float* ms) {
    if (!net || !x || !ms) return fail(PT_ERR_ARG, "null pointer");
    UNet& U = net->u;
    if (batch < 1 || batch > U.maxB) return fail(PT_ERR_ARG, "batch out of range");
    const size_t P0 = (size_t)batch * U.H * U.W;
    CK(cudaMemcpyAsync(U.xin, x, sizeof(float) * P0 * 4, cudaMemcpyHostToDevice, U.st));
    if (int rc = unet_forward(U, batch)) return rc;  // warm-up
    cudaEvent_t ev[15];
    for (auto& e : ev) CK(cudaEventCreate(&e));
    int rc = unet_forward(U, batch, ev);
    if (!rc) rc = cuda_check(cudaStreamSynchronize(U.st), "pt_unet_profile_forward");
    for (int l = 0; l < 14 && !rc; l++) cudaEventElapsedTime(&ms[l], ev[l], ev[l + 1]);
    for (auto& e : ev) cudaEventDestroy(e);
    if (!rc) rc = gemm_error(U);
    return rc;
}

int pt_training_pair(float* x4, float* psi) {
    if (!x4 || !psi) return fail(PT_ERR_ARG, "null pointer");
    if (!g_eng) return fail(PT_ERR_STATE, "call pt_init, pt_upload_state and pt_solve_psi first");
    Engine& E = *g_eng;
    if (!E.uploaded) return fail(PT_ERR_STATE, "call pt_upload_state and pt_solve_psi first");
    const size_t plane = (size_t)E.cfg.nx * E.cfg.nz;
    if (!E.pair_buf) CK(cudaMalloc(&E.pair_buf, sizeof(float) * 5 * plane));
    if (int rc = engine_features(E, E.pair_buf, E.pair_buf + 4 * plane)) return rc;
    CK(cudaMemcpyAsync(x4, E.pair_buf, sizeof(float) * 4 * plane, cudaMemcpyDeviceToHost, E.st));
    CK(cudaMemcpyAsync(psi, E.pair_buf + 4 * plane, sizeof(float) * plane, cudaMemcpyDeviceToHost, E.st));
    CK(cudaStreamSynchronize(E.st));
    return 0;
}

int pt_pair_capture(int capacity) {
    if (!g_eng) return fail(PT_ERR_STATE, "call pt_init first");
    if (capacity < 0 || capacity > 100000) return fail(PT_ERR_ARG, "pt_pair_capture: capacity must be 0..100000");
    Engine& E = *g_eng;
    if (E.pair_ring) cudaFree(E.pair_ring);
    E.pair_ring = nullptr;
    E.pair_cap = E.pair_n = 0;
    if (capacity == 0) return 0;
    const size_t plane = (size_t)E.cfg.nx * E.cfg.nz;
    CK(cudaMalloc(&E.pair_ring, sizeof(float) * 5 * plane * (size_t)capacity));
    E.pair_cap = capacity;
    return 0;
}

int pt_pair_take(float* x4, float* psi, int max_pairs, int* taken) {
    if (!g_eng) return fail(PT_ERR_STATE, "call pt_init first");
    if ((!x4 || !psi) && max_pairs > 0) return fail(PT_ERR_ARG, "null pointer");
    Engine& E = *g_eng;
    const size_t plane = (size_t)E.cfg.nx * E.cfg.nz;
    const int n = E.pair_n < max_pairs ? E.pair_n : (max_pairs > 0 ? max_pairs : 0);
    for (int j = 0; j < n; j++) {
        const float* src = E.pair_ring + (size_t)j * 5 * plane;
        CK(cudaMemcpyAsync(x4 + (size_t)j * 4 * plane, src, sizeof(float) * 4 * plane, cudaMemcpyDeviceToHost, E.st));
        CK(cudaMemcpyAsync(psi + (size_t)j * plane, src + 4 * plane, sizeof(float) * plane, cudaMemcpyDeviceToHost,
                           E.st));
    }
    CK(cudaStreamSynchronize(E.st));
    if (taken) *taken = n;
    E.pair_n = 0;
    return 0;
}

int pt_unet_guess_info(int* used, double* resid_prev, double* resid_net) {
    if (!g_eng) return fail(PT_ERR_STATE, "call pt_init first");
    Engine& E = *g_eng;
    if (used) *used = E.unet_used;
    if (resid_prev) *resid_prev = E.unet_r_prev;
    if (resid_net) *resid_net = E.unet_r_net;
    return 0;
}

}  // extern "C"

namespace pt {
int capture_pair(Engine& E) {
    if (!E.pair_ring || E.pair_n >= E.pair_cap) return 0;
    const size_t plane = (size_t)E.cfg.nx * E.cfg.nz;
    float* slot = E.pair_ring + (size_t)E.pair_n * 5 * plane;
    if (int rc = engine_features(E, slot, slot + 4 * plane)) return rc;
    E.pair_n++;
    return 0;
}

int unet_engine_load(Engine& E, const char* path) {
    if (!path) return fail(PT_ERR_ARG, "PT_GUESS_UNET needs a weight file");
    pt_unet* net = nullptr;
    if (int rc = pt_unet_load(path, E.cfg.nz, E.cfg.nx, 1, &net)) return rc;
    unet_engine_release(E);
    E.unet = net;
    E.unet_core = &net->u;
    return 0;
}
int unet_engine_release(Engine& E) {
    if (E.unet) pt_unet_destroy(static_cast<pt_unet*>(E.unet));
    E.unet = nullptr;
    E.unet_core = nullptr;
    if (E.pair_buf) cudaFree(E.pair_buf);
    E.pair_buf = nullptr;
    if (E.pair_ring) cudaFree(E.pair_ring);
    E.pair_ring = nullptr;
    E.pair_cap = E.pair_n = 0;
    return 0;
}
}  // namespace pt
