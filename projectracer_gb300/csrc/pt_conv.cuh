// pt_conv.cuh -- the U-Net's convolutions as tcgen05 GEMMs whose operand tiles TMA loads in place.
//
// Activations are stored with their zero padding: position ((b (H+1) + y+1) (W+2) + x+1) of C BF16
// channels, so image rows are W+2 positions with a zero column on each side and every image has a zero
// row above it (the last one below too).  A 3x3 tap is then one shift of the position, the operand of
// a tap and a block of channels is a plain [128 positions x 64 channels] box of a 2D tensor, and no
// thread computes an im2col address; the padding positions cost (W+2)(H+1)/(W H) more rows, and are not
// stored.  Threads that gathered the tiles through registers kept the tensor pipe at 2.5% of its rate.
//   * k_conv_gemm (forward, backward-data): tiles of 128 positions x Ntile columns.  A box of 130 positions
//     serves the three taps of a row: the swizzle goes by the shared-memory address, so an operand may
//     start at any row of a box.  Two warps issue the TMA loads (activation boxes, weight boxes; K-major,
//     128- or 64-byte swizzle), one the MMAs (K = 16 each, taps, then channels, in ascending order, so an
//     output's sum does not depend on the tiling); four read the accumulator from tensor memory and store.
//   * k_wgrad_gemm: M = (tap, input channel), N = output channels, K = positions.  The same boxes read
//     with their channels as the leading dimension (MN-major): the taps of a row are one box at row
//     offsets 0, 1 and 2, as blocks of M one position apart.
// What bounds them: on large grids the issue of one MMA per 16 channels (N = 32 takes the 64 cycles that
// reading the 128 rows takes) beside loads and stores; on small ones a chain of load latency, MMAs and
// store (set-up and weight loads run while the kernel before ends).  The forward convolutions of 8 images of 512 x 256: 1338 us with
// a CTA per tile, a box per tap and single threads issuing, now 681; backward-data 1124 and 505, weight
// gradients 1279 and 640.
// Every wait is bounded; a timeout sets an error flag and the CTA leaves after its copies have landed.
#pragma once
#include <cuda.h>

#include "pt_launch.cuh"
#include "pt_tc.cuh"

namespace pt {
namespace tc {

constexpr int kMaxRing = 12, kConvThreads = 224;  // warps 0-3: epilogue, 4 and 6: TMA, 5: MMA
constexpr int kSms = 152, kWgradThreads = 192;  // warps 0-3: epilogue, 4: TMA, 5: MMA

// shared-memory descriptor with a swizzle: layout 2 = 128-byte, 4 = 64-byte; strides in bytes
__device__ __forceinline__ uint64_t smem_desc_sw(uint32_t saddr, uint32_t lbo, uint32_t sbo, uint32_t layout) {
    return smem_desc(saddr, lbo, sbo) | ((uint64_t)layout << 61);
}
__device__ __forceinline__ void mbar_expect(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
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
    // pixel of position p; false for padding (divisions as products with the divisor's reciprocal rounded up,
    // Granlund and Montgomery, PLDI 1994: exact for p < 2^31)
    struct Div {
        int d;
        uint32_t m;
        int sh;
        explicit Div(int n) : d(n), m(0), sh(0) {
            while ((1ll << sh) < n) sh++;
            m = (uint32_t)(((1ull << (31 + sh)) + (unsigned)n - 1) / (unsigned)n);
            sh--;
        }
        Div() = default;
        __device__ __forceinline__ int operator()(int p) const { return (int)(__umulhi((uint32_t)p, m) >> sh); }
    };
    __device__ __forceinline__ bool pixel(int p, Div wp, Div hp, int& b, int& y, int& x) const {
        const int row = wp(p);
        x = p - row * wp.d - 1;
        b = hp(row);
        y = row - b * hp.d - 1;
        return b < B && y >= 0 && x >= 0 && x < W;
    }
};

// A convolution's operands: up to two sources (upsampled tensor, skip tensor) of C[s] channels in
// blocks of bw[s] (64 or 32); K runs over taps, then sources, then blocks, as the weights' rows do.
// taps = 9, or 1 for the first layer's im2col tensor.
struct ConvArgs {
    PadGeo g;
    int taps, nsrc, C[2], bw[2], Ktot, N, Ntile, first, last;  // positions first .. last - 1
    PadGeo::Div wp, hp;  // by the padded width and height
    int tiles, nt, nbuf;  // tiles, of which nt share their positions; accumulators in tensor memory
    // pipeline: S stages of G blocks and nd taps of a row (3: one box of kBoxRows positions serves them, or 1),
    // slots of abytes and bbytes; ctas: on an SM; keep: the weights stay for all tiles of a CTA
    int S, G, nd, abytes, bbytes, ctas, keep;
};
constexpr int kBoxRows = kTileM + 2;

// one role's failure ends the CTA: the others leave their waits at their next look
__device__ __forceinline__ bool conv_wait(uint64_t* bar, uint32_t parity, volatile int* bad) {
    const uint32_t a = smem_u32(bar);
    for (int it = 0; it < kWaitPolls; it++) {
        if (mbar_try(a, parity)) return true;
        if ((it & 15) == 15 && *bad) return false;
    }
    *bad = 1;
    return false;
}

// The pipeline of a convolution of nblk blocks.  A grid of more tiles than SMs runs persistent CTAs with two
// accumulators, so that one tile's stores overlap the next one's loads; as many on an SM as have three
// stages, of a whole row of taps where it fits.  There the weights stay in shared memory where they leave
// that room: all SMs reading the same 18 KB for every tile is a hot spot of L2 (32 -> 32 channels on a
// million pixels: 48 us with them kept, 74 us without; four CTAs on an SM 48 us, three 52, two 64, one 105).
// A smaller grid has an SM for each CTA, and the latency of its loads is all there is: the deepest ring.
static inline void conv_stages(ConvArgs& a, int nblk, bool sums) {
    const int bw = a.nsrc > 1 && a.bw[1] > a.bw[0] ? a.bw[1] : a.bw[0];
    const bool large = a.tiles > kSms;
    a.bbytes = a.Ntile * bw * 2;
    a.nbuf = a.Ntile <= 128 && large ? 2 : 1;
    auto stages = [&](int k, int keep) {  // of k CTAs on an SM, which has 228 KB (1 KB reserved, 2.1 KB static each, 5.1 with
        // column sums)
        const int room = (k == 1 ? 220 : 228 / k - (sums ? 8 : 4)) * 1024 - (keep ? a.taps * nblk * a.bbytes : 0);
        auto bytes = [&](int nd, int G) {
            a.nd = nd;
            a.G = G;
            a.abytes = ((nd == 3 ? kBoxRows : kTileM) * bw * 2 + 1023) / 1024 * 1024;
            return G * (a.abytes + (keep ? 0 : nd * a.bbytes));
        };
        int n;
        if (a.taps != 9 || 2 * (n = bytes(3, nblk)) > room) {
            int G = nblk;  // a divisor of nblk: three stages of it
            while (nblk % G || (3 * bytes(1, G) > room && G > 1)) G--;
            n = bytes(1, G);
        }
        a.keep = keep;
        a.ctas = k;
        a.S = room / n < kMaxRing ? room / n : kMaxRing;
        return a.S;
    };
    if (!large) {
        stages(1, 0);
        const int steps = a.taps / a.nd * (nblk / a.G);
        if (a.S > steps) a.S = steps;
        return;
    }
    const int cols = (int)tmem_cols(a.nbuf * a.Ntile);
    for (int keep = 1; keep >= 0; keep--)
        for (int k = 4; k >= 1; k--)
            if (k * cols <= 512 && (!keep || kSms * k % a.nt == 0) && stages(k, keep) >= (keep || k > 2 ? 3 : k)) return;
}
static inline size_t conv_smem(const ConvArgs& a) {
    const int nblk = a.C[0] / a.bw[0] + (a.nsrc > 1 ? a.C[1] / a.bw[1] : 0), w = a.keep ? a.taps * nblk : a.S * a.nd * a.G;
    return (size_t)a.S * a.G * a.abytes + (size_t)w * a.bbytes + 1024;
}

// barriers of a ring
struct Ring {
    uint64_t full[kMaxRing], empty[kMaxRing];
    __device__ __forceinline__ void init(int n, int fills, int frees) {
        for (int s = 0; s < n; s++) {
            mbar_init(full + s, (uint32_t)fills);
            mbar_init(empty + s, (uint32_t)frees);
        }
    }
};
// a position in a ring and the parity of its use
struct RingPos {
    int i = 0;
    uint32_t parity;
    __device__ __forceinline__ explicit RingPos(uint32_t p) : parity(p) {}
    __device__ __forceinline__ void next(int n) {
        if (++i == n) {
            i = 0;
            parity ^= 1u;
        }
    }
};

// after a failure: the loader at r waits for its copies in flight (bounded)
__device__ __forceinline__ void drain(Ring& ring, const RingPos& r, int n) {
    for (int s = 0; s < n; s++) mbar_wait(ring.full + s, s < r.i ? r.parity ^ 1u : r.parity);
}

// Epilogue E: void operator()(p, b, y, x, col0, v, bias) for columns col0 .. col0 + 31 of position p (called
// for real pixels with their coordinates); with kSums: void sums(p, real, col0, v, sum) by whole warps,
// which adds its lanes' masked values to sum[col0 ..], and part[CTA][column] for the CTA's sums
template <class E>
__global__ void __launch_bounds__(kConvThreads) k_conv_gemm(const __grid_constant__ CUtensorMap mapA0,
                                                            const __grid_constant__ CUtensorMap mapA1,
                                                            const __grid_constant__ CUtensorMap mapB0,
                                                            const __grid_constant__ CUtensorMap mapB1, ConvArgs a, E epi,
                                                            int* err) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ Ring ring, accs;  // stages; accumulators
    __shared__ uint64_t done, wfull;
    __shared__ uint32_t tslot;
    __shared__ int bad;
    __shared__ __align__(16) float sbias[256];
    __shared__ float sacc[E::kSums ? 4 * 256 : 1];  // column sums of the epilogue's warps
    unsigned char* const smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int S = a.S, G = a.G, nd = a.nd;
    const uint32_t ncols = tmem_cols(a.nbuf * a.Ntile);
    if (tid == 0) {
        bad = 0;
        ring.init(S, a.keep ? 1 : 2, 1);
        accs.init(a.nbuf, 1, 4);
        mbar_init(&done, 1);
        mbar_init(&wfull, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(&tslot, ncols);
    epi.stage(sbias, a.N, tid);
    if (E::kSums)
        for (int q = tid; q < 4 * 256; q += kConvThreads) sacc[q] = 0.f;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    // everything above, and the weights, does not depend on the kernel before this one (a parameter update
    // is at least two launches back, and a kernel lets its successor start once its predecessor has ended)
    if (warp != 6) pdl_begin();
    const uint32_t taddr = tslot;
    const int bw0 = a.bw[0], bw1 = a.bw[1], nb0 = a.C[0] / bw0, nblk = nb0 + (a.nsrc > 1 ? a.C[1] / bw1 : 0);
    const int rows = a.taps == 1 ? 1 : 3, steps = a.taps / nd, brows = nd == 3 ? kBoxRows : kTileM;
    const uint32_t boff = (uint32_t)(G * a.abytes), sbytes = boff + (uint32_t)(a.keep ? 0 : G * nd * a.bbytes);
    unsigned char* const wsm = smem + (size_t)S * sbytes;  // weights that stay
    // The loads and the MMAs are serial chains of single instructions: whole warps run the loops, so that the
    // operands stay in uniform registers, and one lane issues (by one thread alone a
    // chunk of 64 channels took 650 cycles to load and 550 to multiply, now 150 each).
    if (warp == 4) {  // activation boxes
        RingPos r(1);  // the first wait for a stage passes
        bool go = true;
        for (int tile = blockIdx.x; tile < a.tiles && go; tile += gridDim.x) {
            const int p0 = a.first + tile / a.nt * kTileM;
            int pos = a.taps == 1 ? p0 : p0 - a.g.Wp() - 1, dx = 0;
            for (int t = 0; t < steps && go; t++) {
                for (int b0 = 0; b0 < nblk; b0 += G) {
                    if (!(go = conv_wait(ring.empty + r.i, r.parity, &bad))) break;
                    if (elect_one()) {
                        unsigned char* sa = smem + r.i * sbytes;
                        uint64_t* const bar = ring.full + r.i;
                        const int k0 = min(max(nb0 - b0, 0), G);
                        mbar_expect(bar, (uint32_t)(brows * 2 * (k0 * bw0 + (G - k0) * bw1)));
                        for (int blk = b0; blk < b0 + G; blk++, sa += a.abytes)
                            if (blk < nb0)
                                tma_load_2d(sa, &mapA0, blk * bw0, pos, bar);
                            else
                                tma_load_2d(sa, &mapA1, (blk - nb0) * bw1, pos, bar);
                    }
                    __syncwarp();
                    r.next(S);
                }
                if (nd == 3 || dx == rows - 1) {
                    pos += a.g.Wp() - dx;
                    dx = 0;
                } else {
                    pos++;
                    dx++;
                }
            }
        }
        if (!go) drain(ring, r, S);
    } else if (warp == 6 && a.keep) {
        if (elect_one()) {
            unsigned char* sb = wsm;
            int x = 0;
            mbar_expect(&wfull, (uint32_t)(a.Ntile * 2 * a.Ktot));
            for (int q = 0; q < a.taps; q++)
                for (int g = 0; g < nblk; g++, sb += a.bbytes)
                    if (g < nb0 || bw1 == bw0) {
                        tma_load_2d(sb, &mapB0, x, (int)blockIdx.x % a.nt * a.Ntile, &wfull);
                        x += bw0;
                    } else {
                        tma_load_2d(sb, &mapB1, x, (int)blockIdx.x % a.nt * a.Ntile, &wfull);
                        x += bw1;
                    }
        }
        __syncwarp();
        mbar_wait(&wfull, 0);  // the CTA does not leave before its copies have landed
    } else if (warp == 6) {  // weight boxes
        RingPos r(1);
        bool go = true;
        for (int tile = blockIdx.x; tile < a.tiles && go; tile += gridDim.x) {
            const int n0 = tile % a.nt * a.Ntile;
            int k = 0;
            for (int t = 0; t < steps && go; t++)
                for (int b0 = 0; b0 < nblk; b0 += G) {
                    if (!(go = conv_wait(ring.empty + r.i, r.parity, &bad))) break;
                    const int k0 = min(max(nb0 - b0, 0), G), kw = k0 * bw0 + (G - k0) * bw1;
                    if (elect_one()) {
                        unsigned char* sb = smem + r.i * sbytes + boff;
                        uint64_t* const bar = ring.full + r.i;
                        mbar_expect(bar, (uint32_t)(nd * a.Ntile * 2 * kw));
                        int x = k;
                        for (int q = 0; q < nd; q++)
                            for (int g = 0; g < G; g++, sb += a.bbytes)
                                if (g < k0 || bw1 == bw0) {
                                    tma_load_2d(sb, &mapB0, x, n0, bar);
                                    x += bw0;
                                } else {
                                    tma_load_2d(sb, &mapB1, x, n0, bar);
                                    x += bw1;
                                }
                    }
                    __syncwarp();
                    k += nd * kw;
                    r.next(S);
                }
        }
        if (!go) drain(ring, r, S);
    } else if (warp == 5) {
        const uint32_t idesc = idesc_bf16(a.Ntile);
        const uint64_t d64 = smem_desc_sw(0, 16, 1024, 2u), d32 = smem_desc_sw(0, 16, 512, 4u);
        RingPos r(0), c(1);
        bool go = !a.keep || conv_wait(&wfull, 0, &bad);
        for (int tile = blockIdx.x; tile < a.tiles && go; tile += gridDim.x) {
            const uint32_t t0 = taddr + (uint32_t)(c.i * a.Ntile);
            uint32_t acc = 0, sw = smem_u32(wsm);
            if (!(go = conv_wait(accs.empty + c.i, c.parity, &bad))) break;
            tc_fence_after();
            for (int t = 0; t < steps && go; t++)
                for (int b0 = 0; b0 < nblk; b0 += G) {
                    if (!(go = conv_wait(ring.full + r.i, r.parity, &bad))) break;
                    tc_fence_after();
                    if (elect_one()) {
                        const uint32_t sa = smem_u32(smem) + r.i * sbytes;
                        uint32_t sb = a.keep ? sw : sa + boff;
                        for (int q = 0; q < nd; q++)
                            for (int g = 0; g < G; g++, sb += (uint32_t)a.bbytes) {
                                const bool wide = (b0 + g < nb0 ? bw0 : bw1) == 64;
                                const uint64_t d0 = wide ? d64 : d32;
                                const uint64_t da =
                                    d0 + ((sa + (uint32_t)(g * a.abytes + q * (wide ? 128 : 64))) >> 4);
                                const uint64_t db = d0 + (sb >> 4);
                                mma_bf16(t0, da, db, idesc, acc | (uint32_t)(q + g));
                                mma_bf16(t0, da + 2, db + 2, idesc, 1u);  // 16 channels further: 32 bytes
                                if (wide) {
                                    mma_bf16(t0, da + 4, db + 4, idesc, 1u);
                                    mma_bf16(t0, da + 6, db + 6, idesc, 1u);
                                }
                            }
                        mma_commit(ring.empty + r.i);
                    }
                    __syncwarp();
                    acc = 1u;
                    sw += (uint32_t)(nd * G * a.bbytes);
                    r.next(S);
                }
            if (elect_one()) mma_commit(accs.full + c.i);
            __syncwarp();
            c.next(a.nbuf);
        }
        if (!go) {  // MMAs in flight read the stages
            if (elect_one()) mma_commit(&done);
            __syncwarp();
            mbar_wait(&done, 0);
        }
    } else {
        RingPos c(0);
        for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x) {
            const int n0 = tile % a.nt * a.Ntile, p = a.first + tile / a.nt * kTileM + warp * 32 + lane;
            int b = 0, y = 0, x = 0;
            const bool real = p < a.last && a.g.pixel(p, a.wp, a.hp, b, y, x);
            int ok = 0;
            if (lane == 0) ok = conv_wait(accs.full + c.i, c.parity, &bad);  // one lane: polls take issue slots
            if (!__shfl_sync(0xffffffffu, ok, 0)) break;
            tc_fence_after();
            const uint32_t t0 = taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)(c.i * a.Ntile);
            for (int c0 = 0; c0 < a.Ntile; c0 += 32) {
                float v[32];
                __syncwarp();
                tmem_ld32(t0 + (uint32_t)c0, v);
                if (c0 + 32 == a.Ntile) {  // the accumulator is free
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(accs.empty + c.i);
                }
                if (E::kSums) epi.sums(p, real, n0 + c0, v, sacc + warp * 256);
                else if (real) epi(p, b, y, x, n0 + c0, v, sbias + n0 + c0);
            }
            c.next(a.nbuf);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (E::kSums)
        for (int c = tid; c < a.N; c += kConvThreads)
            epi.part[(size_t)blockIdx.x * a.N + c] = ((sacc[c] + sacc[256 + c]) + sacc[512 + c]) + sacc[768 + c];
    if (bad && tid == 0) atomicOr(err, 1);
    if (warp == 5) tmem_dealloc(taddr, ncols);
}

// Weight gradient of one source tensor: part[z][kk][co] = sum over the split's positions of
// in[p + shift(tap)][ci] dZ[p][co], kk = tap cin + c_off + ci.  A CTA takes a block of bw channels and the
// taps of one image row: per chunk of 128 positions a box of 132 positions, and dZ's boxes.  An accumulator
// holds 128 / bw blocks of M, one position apart: 4 x 32 (taps -1, 0, 1, and one that is not stored) or
// 2 x 64 (taps -1, 0, and in a second one tap 1).
struct WgradArgs {
    PadGeo g;
    int taps, C, bw, c_off, cin, N, Ntile, bwB, per, chunks;  // per: chunks a split, of `chunks`
    int kk_max;  // rows kk >= kk_max are not stored (im2col padding)
    int ncols;   // tensor-memory columns
    int S, abytes, bbytes;  // stages of abytes (the box of positions) and bbytes
    float* part;
};
static inline size_t wgrad_smem(const WgradArgs& a) { return (size_t)a.S * (a.abytes + a.bbytes) + 1024; }
constexpr int kWgradK = 128, kWgradBox = kWgradK + 4;
// bytes of a box of positions, to a 1024-byte boundary
__host__ __device__ constexpr int wgrad_box_bytes(int bw) { return (kWgradBox * bw * 2 + 1023) / 1024 * 1024; }
// instruction descriptor with both operands MN-major
__host__ __device__ constexpr uint32_t idesc_bf16_mn(int n) { return idesc_bf16(n) | (1u << 15) | (1u << 16); }

// The weight gradients of all layers in one launch: they depend on nothing of each other, and on a small grid
// one layer's CTAs fill part of the chip for 7 us (gradients of 3 images of 136 x 72: 500 us with a launch per
// layer and source, now 414).  first: a problem's first CTA; gx, gy: its CTAs over
// blocks of channels and rows, and over tiles of N.
constexpr int kMaxWgrads = 17;
struct WgradGroup {
    struct Problem {
        CUtensorMap A, B;
        WgradArgs a;
        int first, gx, gy;
    } p[kMaxWgrads];
    int n, ctas;
    size_t smem;
};
__global__ void __launch_bounds__(kWgradThreads) k_wgrad_gemm(const __grid_constant__ WgradGroup group, int* err) {
    int pi = group.n - 1;
    while (pi > 0 && (int)blockIdx.x < group.p[pi].first) pi--;
    const WgradGroup::Problem& P = group.p[pi];
    const WgradArgs& a = P.a;
    const int cta = (int)blockIdx.x - P.first, bz = cta / (P.gx * P.gy), bxy = cta - bz * P.gx * P.gy, by = bxy / P.gx,
              bx = bxy - by * P.gx;
    extern __shared__ unsigned char smem_raw[];
    __shared__ Ring ring;
    __shared__ uint64_t done;
    __shared__ uint32_t tslot;
    __shared__ int bad;
    unsigned char* const smem = smem_raw + ((1024 - (smem_u32(smem_raw) & 1023)) & 1023);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int n0 = by * a.Ntile, S = a.S;
    const uint32_t sbytes = (uint32_t)(a.abytes + a.bbytes);
    if (tid == 0) {
        bad = 0;
        ring.init(S, 1, 1);
        mbar_init(&done, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) tmem_alloc(&tslot, (uint32_t)a.ncols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    pdl_begin();
    const uint32_t taddr = tslot;
    const int cbeg = bz * a.per, cend = min(a.chunks, cbeg + a.per), n = max(0, cend - cbeg);
    const int nch = a.C / a.bw, unit = bx / nch, ch = (bx - unit * nch) * a.bw;
    const int bblk = a.Ntile / a.bwB, nacc = a.taps == 1 || a.bw == 32 ? 1 : 2;  // accumulators
    const int shift = a.taps == 1 ? 0 : (unit - 1) * a.g.Wp() - 1;                // of tap -1 of the row
    const uint32_t bbox = (uint32_t)(kWgradK * a.bwB * 2);
    if (warp == 4) {
        RingPos r(1);  // the first wait for a stage passes
        int p = cbeg * kWgradK;
        for (int c = 0; c < n; c++, p += kWgradK) {
            if (!conv_wait(ring.empty + r.i, r.parity, &bad)) {
                drain(ring, r, S);
                break;
            }
            unsigned char* sa = smem + r.i * sbytes;
            if (elect_one()) {
                mbar_expect(ring.full + r.i, (uint32_t)(kWgradBox * a.bw * 2) + (uint32_t)bblk * bbox);
                tma_load_2d(sa, &P.A, ch, p + shift, ring.full + r.i);
                for (int q = 0; q < bblk; q++)
                    tma_load_2d(sa + a.abytes + q * bbox, &P.B, n0 + q * a.bwB, p, ring.full + r.i);
            }
            __syncwarp();
            r.next(S);
        }
    } else if (warp == 5) {
        const uint32_t idesc = idesc_bf16_mn(a.Ntile);
        const uint32_t pa = (uint32_t)a.bw * 2, pb = (uint32_t)a.bwB * 2;  // bytes of a position
        const uint64_t da0 = smem_desc_sw(0, pa, 8 * pa, a.bw == 64 ? 2u : 4u);  // blocks of M: one position apart
        const uint64_t db0 = smem_desc_sw(0, bbox, 8 * pb, a.bwB == 64 ? 2u : 4u);
        RingPos r(0);
        uint32_t acc = 0;
        for (int c = 0; c < n; c++) {
            if (!conv_wait(ring.full + r.i, r.parity, &bad)) break;
            tc_fence_after();
            const uint32_t sa = smem_u32(smem) + r.i * sbytes;
            const uint64_t db = db0 + ((sa + (uint32_t)a.abytes) >> 4);
            if (elect_one()) {
                for (int h = 0; h < nacc; h++) {
                    const uint64_t da = da0 + ((sa + 2 * h * pa) >> 4);
#pragma unroll
                    for (int s = 0; s < kWgradK / 16; s++)  // 16 positions further
                        mma_bf16(taddr + (uint32_t)(h * a.Ntile), da + s * pa, db + s * pb, idesc, acc | (s > 0));
                }
                mma_commit(ring.empty + r.i);
            }
            __syncwarp();
            acc = 1u;
            r.next(S);
        }
        if (elect_one()) mma_commit(&done);
        __syncwarp();
        conv_wait(&done, 0, &bad);
        tc_fence_before();
    }
    __syncthreads();  // not a wait on the barrier by every thread: their polls took the driving threads' issue slots
    if (warp < 4) {
        const bool ok = !bad;
        tc_fence_after();
        const int row = warp * 32 + lane, blk = row / a.bw, ci = ch + row - blk * a.bw;
        for (int h = 0; h < nacc; h++) {
            const int dx = blk + 2 * h;  // 0, 1, 2: taps -1, 0, 1
            const int tap = a.taps == 1 ? 0 : 3 * unit + dx, kk = tap * a.cin + a.c_off + ci;
            const bool real = (a.taps == 1 ? blk == 0 : dx < 3 && (h == 0 || blk == 0)) && kk < a.kk_max;
            for (int c0 = 0; c0 < a.Ntile; c0 += 32) {
                float v[32];
                __syncwarp();
                tmem_ld32(taddr + ((uint32_t)(warp * 32) << 16) + (uint32_t)(h * a.Ntile + c0), v);
                if (!ok || !real) continue;
                float* o = a.part + ((size_t)bz * a.kk_max + kk) * a.N + n0 + c0;
#pragma unroll
                for (int j = 0; j < 32; j += 4)
                    *reinterpret_cast<float4*>(o + j) = n > 0 ? make_float4(v[j], v[j + 1], v[j + 2], v[j + 3])
                                                              : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (bad && tid == 0) atomicOr(err, 1);
    if (warp == 5) tmem_dealloc(taddr, (uint32_t)a.ncols);
}

}  // namespace tc
}  // namespace pt
