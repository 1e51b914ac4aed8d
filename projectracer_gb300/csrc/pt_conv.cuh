// pt_conv.cuh -- the U-Net's convolutions as tcgen05 GEMMs whose operand tiles TMA loads in place.
//
// Activations are stored with their zero padding: position ((b (H+1) + y+1) (W+2) + x+1) of C BF16
// channels, so image rows are W+2 positions with a zero column on each side and every image has a zero
// row above it (the last one below too).  A 3x3 tap is then one shift of the position, the operand of
// a tap and a block of channels is a plain [128 positions x 64 channels] box of a 2D tensor, and no
// thread computes an im2col address; the padding positions cost (W+2)(H+1)/(W H) more rows, and are not
// stored.  Threads that gathered the tiles through registers kept the tensor pipe at 2.5% of its rate.
//   * k_conv_gemm (forward, backward-data): a CTA computes 128 positions x Ntile columns.  One thread
//     issues the TMA loads of a chunk (one tap, 64 or 32 channels: A box and weight box, K-major,
//     128- or 64-byte swizzle), one the MMAs (K = 16 each, taps and channels in ascending order, so an
//     output's sum does not depend on the tiling), through a ring of stages with full/empty mbarriers;
//     four warps read the accumulator from tensor memory and store.
//   * k_wgrad_gemm: M = 128 rows of (tap, input channel), N = output channels, K = positions.  Both
//     operands are the same boxes read with their channels as the leading dimension (MN-major).
// Every wait is bounded; a timeout sets an error flag and the CTA leaves after its copies have landed.
#pragma once
#include <cuda.h>

#include "pt_tc.cuh"

namespace pt {
namespace tc {

constexpr int kMaxStages = 10, kConvThreads = 192;  // warps 0-3: epilogue, 4: TMA, 5: MMA

// shared-memory descriptor with a swizzle: layout 2 = 128-byte, 4 = 64-byte; strides in bytes
__device__ __forceinline__ uint64_t smem_desc_sw(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
    return smem_desc(saddr, lbo, sbo) | ((uint64_t)layout << 61);
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
// 32 consecutive FP32 accumulator columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
        "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 32; j++) v[j] = __uint_as_float(r[j]);
}

// Padded image geometry of a batch
struct PadGeo {
    int B, H, W;
    __host__ __device__ int Wp() const { return W + 2; }
    __host__ __device__ int Hp() const { return H + 1; }
    __host__ __device__ size_t positions() const { return ((size_t)B * Hp() + 1) * Wp(); }
    __host__ __device__ size_t at(int b, int y, int x) const { return ((size_t)b * Hp() + y + 1) * Wp() + x + 1; }
    // pixel of position p; false for padding
    __device__ __forceinline__ bool pixel(int p, int& b, int& y, int& x) const {
        const int row = p / Wp();
        x = p - row * Wp() - 1;
        b = row / Hp();
        y = row - b * Hp() - 1;
        return b < B && y >= 0 && x >= 0 && x < W;
    }
};

// A convolution's operands: up to two sources (upsampled tensor, skip tensor) of C[s] channels in
// blocks of bw[s] (64 or 32); K runs over taps, then sources, then blocks, as the weights' rows do.
// taps = 9, or 1 for the first layer's im2col tensor.
struct ConvArgs {
    PadGeo g;
    int taps, nsrc, C[2], bw[2], Ktot, N, Ntile, first, last;  // positions first .. last - 1
    int stages, abytes, bbytes;                               // pipeline depth; operand bytes of a stage
};

// one role's failure ends the CTA: waits that follow return at once
__device__ __forceinline__ bool conv_wait(uint64_t* bar, uint32_t parity, volatile int* bad) {
    if (*bad) return false;
    if (mbar_wait(bar, parity)) return true;
    *bad = 1;
    return false;
}

// Pipeline depth for stages of sbytes in a grid of `ctas`: with a CTA per SM at most, as deep as the
// shared memory allows, since a chunk's load latency (1-2 us) is all there is; with more, four stages, so
// that several CTAs share an SM and one's prologue and epilogue run beside the others' loads.
static inline int conv_stages(size_t sbytes, size_t ctas, int chunks) {
    const int most = (int)((220 * 1024) / sbytes);
    int s = ctas <= 152 ? most : 4;
    s = s < most ? s : most;
    s = s < chunks ? s : chunks;
    return s < kMaxStages ? (s > 1 ? s : 1) : kMaxStages;
}

// Epilogue E: void operator()(int p, int col0, const float (&v)[32]) for columns col0 .. col0 + 31 of
// position p (called for real pixels with their coordinates)
template <class E>
__global__ void __launch_bounds__(kConvThreads) k_conv_gemm(const __grid_constant__ CUtensorMap mapA0,
                                                            const __grid_constant__ CUtensorMap mapA1,
                                                            const __grid_constant__ CUtensorMap mapB0,
                                                            const __grid_constant__ CUtensorMap mapB1, ConvArgs a, E epi,
                                                            int* err) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t full[kMaxStages], empty[kMaxStages], done;
    __shared__ uint32_t tslot;
    __shared__ int bad;
    unsigned char* const smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int p0 = a.first + blockIdx.x * kTileM, n0 = blockIdx.y * a.Ntile;
    const uint32_t ncols = tmem_cols(a.Ntile);
    const int S = a.stages;
    const size_t sbytes = (size_t)(a.abytes + a.bbytes);
    if (tid == 0) {
        bad = 0;
        for (int s = 0; s < S; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(&tslot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = tslot;
    const int nb0 = a.C[0] / a.bw[0], nb1 = a.nsrc > 1 ? a.C[1] / a.bw[1] : 0, nblk = nb0 + nb1, chunks = a.taps * nblk;
    // One thread each drives the loads and the MMAs, so a chunk's instructions are a serial chain: counters
    // instead of divisions (with them a chunk took 0.6 us).
    if (warp == 4 && lane == 0) {
        int k = 0, st = 0, dx = -1, shift = a.taps == 1 ? 0 : -a.g.Wp() - 1;
        uint32_t parity = 1;  // of the stage's previous use; the first wait for a stage passes
        bool go = true;
        for (int tap = 0; tap < a.taps && go; tap++) {
            for (int blk = 0; blk < nblk; blk++) {
                if (!conv_wait(empty + st, parity, &bad)) {
                    go = false;
                    break;
                }
                const int src = blk >= nb0, bw = a.bw[src], ch = (src ? blk - nb0 : blk) * bw;
                unsigned char* sa = smem + st * sbytes;
                mbar_expect(full + st, (uint32_t)((kTileM + a.Ntile) * bw * 2));
                tma_load_2d(sa, src ? &mapA1 : &mapA0, ch, p0 + shift, full + st);
                tma_load_2d(sa + a.abytes, bw == a.bw[0] ? &mapB0 : &mapB1, k, n0, full + st);
                k += bw;
                if (++st == S) {
                    st = 0;
                    parity ^= 1u;
                }
            }
            shift += dx < 1 ? 1 : a.g.Wp() - 2;
            dx = dx < 1 ? dx + 1 : -1;
        }
    } else if (warp == 5 && lane == 0) {
        const uint32_t idesc = idesc_bf16(a.Ntile);
        const uint64_t d64 = smem_desc_sw(0, 16, 1024, 2u), d32 = smem_desc_sw(0, 16, 512, 4u);
        int st = 0, blk = 0;
        uint32_t parity = 0, acc = 0;
        for (int c = 0; c < chunks; c++) {
            if (!conv_wait(full + st, parity, &bad)) break;
            tc_fence_after();
            const bool wide = a.bw[blk >= nb0] == 64;
            const uint32_t sa = smem_u32(smem) + (uint32_t)(st * sbytes);
            const uint64_t da = (wide ? d64 : d32) + (sa >> 4), db = da + (uint32_t)(a.abytes >> 4);
#pragma unroll
            for (int s = 0; s < 4; s++) {
                if (s >= 2 && !wide) break;
                mma_bf16(taddr, da + 2 * s, db + 2 * s, idesc, acc);  // 16 channels further: 32 bytes
                acc = 1u;
            }
            mma_commit(empty + st);
            if (++blk == nblk) blk = 0;
            if (++st == S) {
                st = 0;
                parity ^= 1u;
            }
        }
        mma_commit(&done);
    }
    __syncwarp();
    if (warp < 4) {
        const bool ok = conv_wait(&done, 0, &bad);
        tc_fence_after();
        const int p = p0 + warp * 32 + lane;
        int b = 0, y = 0, x = 0;
        const bool real = p < a.last && a.g.pixel(p, b, y, x);
        for (int c0 = 0; c0 < a.Ntile; c0 += 32) {
            float v[32];
            tmem_ld32(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
            if (ok && real) epi(p, b, y, x, n0 + c0, v);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (bad && tid == 0) {
        atomicOr(err, 1);
        for (int s = 0; s < S; s++) mbar_wait(full + s, 0);  // copies still in flight (bounded)
    }
    if (warp == 5) tmem_dealloc(taddr, ncols);
}

// Weight gradient of one source tensor: part[z][kk][co] = sum over the split's positions of
// in[p + shift(tap)][ci] dZ[p][co], kk = tap cin + c_off + ci.  A's 128 rows are `ablk` blocks of bwA
// channels (2 x 64 or 4 x 32); block q of tile t is number t ablk + q of the taps x (C / bwA) blocks.
struct WgradArgs {
    PadGeo g;
    int taps, C, bwA, c_off, cin, N, Ntile, bwB, per, chunks;  // per: chunks of 64 positions a split, of `chunks`
    int kk_max;  // rows kk >= kk_max are not stored (im2col padding)
    int stages, abytes, bbytes;
    float* part;
};
constexpr int kWgradK = 64;
// instruction descriptor with both operands MN-major
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int n) { return idesc_bf16(n) | (1u << 15) | (1u << 16); }

__global__ void __launch_bounds__(kConvThreads) k_wgrad_gemm(const __grid_constant__ CUtensorMap mapA,
                                                             const __grid_constant__ CUtensorMap mapB, WgradArgs a,
                                                             int* err) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t full[kMaxStages], empty[kMaxStages], done;
    __shared__ uint32_t tslot;
    __shared__ int bad;
    unsigned char* const smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int n0 = blockIdx.y * a.Ntile;
    const uint32_t ncols = tmem_cols(a.Ntile);
    const int S = a.stages;
    const size_t sbytes = (size_t)(a.abytes + a.bbytes);
    if (tid == 0) {
        bad = 0;
        for (int s = 0; s < S; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(&tslot, ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = tslot;
    const int cbeg = blockIdx.z * a.per, cend = min(a.chunks, cbeg + a.per), n = max(0, cend - cbeg);
    const int ablk = kTileM / a.bwA, nch = a.C / a.bwA, blocks = a.taps * nch, bblk = a.Ntile / a.bwB;
    const uint32_t abox = (uint32_t)(kWgradK * a.bwA * 2), bbox = (uint32_t)(kWgradK * a.bwB * 2);
    if (warp == 4 && lane == 0) {
        int ch[4], shift[4];  // of the A blocks; past the last one: loaded, not stored
#pragma unroll
        for (int q = 0; q < 4; q++) {
            const int blk = min((int)blockIdx.x * ablk + q, blocks - 1), tap = blk / nch;
            ch[q] = (blk - tap * nch) * a.bwA;
            shift[q] = a.taps == 1 ? 0 : (tap / 3 - 1) * a.g.Wp() + (tap % 3 - 1);
        }
        int st = 0, p = cbeg * kWgradK;
        uint32_t parity = 1;  // of the stage's previous use; the first wait for a stage passes
        for (int c = 0; c < n; c++, p += kWgradK) {
            if (!conv_wait(empty + st, parity, &bad)) break;
            unsigned char* sa = smem + st * sbytes;
            mbar_expect(full + st, (uint32_t)ablk * abox + (uint32_t)bblk * bbox);
#pragma unroll
            for (int q = 0; q < 4; q++)
                if (q < ablk) tma_load_2d(sa + q * abox, &mapA, ch[q], p + shift[q], full + st);
            for (int q = 0; q < bblk; q++) tma_load_2d(sa + a.abytes + q * bbox, &mapB, n0 + q * a.bwB, p, full + st);
            if (++st == S) {
                st = 0;
                parity ^= 1u;
            }
        }
    } else if (warp == 5 && lane == 0) {
        const uint32_t idesc = idesc_bf16_mn(a.Ntile);
        const uint32_t ra = (uint32_t)a.bwA * 2, rb = (uint32_t)a.bwB * 2;  // bytes of a position's block row
        const uint64_t da0 = smem_desc_sw(0, abox, 8 * ra, a.bwA == 64 ? 2u : 4u);
        const uint64_t db0 = smem_desc_sw(0, bbox, 8 * rb, a.bwB == 64 ? 2u : 4u);
        int st = 0;
        uint32_t parity = 0, acc = 0;
        for (int c = 0; c < n; c++) {
            if (!conv_wait(full + st, parity, &bad)) break;
            tc_fence_after();
            const uint32_t sa = smem_u32(smem) + (uint32_t)(st * sbytes);
            const uint64_t da = da0 + (sa >> 4), db = db0 + ((sa + (uint32_t)a.abytes) >> 4);
#pragma unroll
            for (int s = 0; s < kWgradK / 16; s++) {
                mma_bf16(taddr, da + s * ra, db + s * rb, idesc, acc);  // 16 positions further
                acc = 1u;
            }
            mma_commit(empty + st);
            if (++st == S) {
                st = 0;
                parity ^= 1u;
            }
        }
        mma_commit(&done);
    }
    __syncwarp();
    if (warp < 4) {
        const bool ok = conv_wait(&done, 0, &bad);
        tc_fence_after();
        const int row = warp * 32 + lane, blk = blockIdx.x * ablk + row / a.bwA, tap = blk / nch;
        const int kk = tap * a.cin + a.c_off + (blk - tap * nch) * a.bwA + row % a.bwA;
        const bool real = blk < blocks && kk < a.kk_max;
        for (int c0 = 0; c0 < a.Ntile; c0 += 32) {
            float v[32];
            tmem_ld32(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)c0, v);
            if (!ok || !real) continue;
            float* o = a.part + ((size_t)blockIdx.z * a.kk_max + kk) * a.N + n0 + c0;
#pragma unroll
            for (int j = 0; j < 32; j += 4)
                *reinterpret_cast<float4*>(o + j) = n > 0 ? make_float4(v[j], v[j + 1], v[j + 2], v[j + 3])
                                                          : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (bad && tid == 0) {
        atomicOr(err, 1);
        for (int s = 0; s < S; s++) mbar_wait(full + s, 0);  // copies still in flight (bounded)
    }
    if (warp == 5) tmem_dealloc(taddr, ncols);
}

}  // namespace tc
}  // namespace pt
