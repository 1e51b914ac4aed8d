// pt_cluster.cuh -- one multigrid level spread over one thread-block cluster, its stage values
// resident in shared memory.
//
// Below some ten thousand nodes a smoother stage is a few hundred nanoseconds of arithmetic, and a
// kernel per stage is bound by its launch and by the round trip through L2 (2.5-3.3 us a stage on
// GB300).  Here a cluster of 16 CTAs walks whole stretches of the level schedule in one launch: CTA c
// owns rows 1 + cR .. (c+1)R of the level (R = ceil((nz-1)/16)) over the full width, and holds a
// window of the stage values with the 3 rows that its stencils reach above and below.  A thread that
// has a node's new value stores it straight into the window of every CTA that reads that row
// (asynchronous stores to distributed shared memory, counted by an mbarrier of the receiver), so a
// stage waits for its neighbours' rows only and moves no global data.  Full-width strips rather than
// 2D blocks: the neighbours of a strip are known from the row alone, for strips of one row too.
// Measured per FP32 stage: 0.55-0.75 us (a cluster barrier per stage instead of the counted stores:
// 1.3 us); the part of a V-cycle below level 1, 8 stages a visit: 128x128 148 -> 77 us, 256x128
// 93 -> 62 us.  FP64 stages with exact sums: 1.5-1.7 us (4.2 with a kernel per stage).
#pragma once
#include <cstdint>

#include "pt_consts.cuh"
#include "pt_internal.h"

namespace pt {
namespace cl {

constexpr int kCtas = 16, kThreads = 512, kWarps = kThreads / 32;
constexpr size_t kMaxSmem = 227 * 1024 - 2048;  // dynamic; the static arrays take the rest
constexpr int kReach = 3;  // rows and columns that a stencil reaches

__device__ __forceinline__ uint32_t rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// all threads of all CTAs; orders shared, distributed shared and global memory in the cluster
__device__ __forceinline__ void sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t remote(uint32_t a, int cta) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(cta));
    return r;
}
// v to the shared memory of another CTA of the cluster, counted by that CTA's mbarrier
__device__ __forceinline__ void put(uint32_t a, float v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(a),
                 "r"(__float_as_uint(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void put(uint32_t a, double v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(a),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void bar_init(uint32_t bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void bar_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// 8 bytes from global to this CTA's shared memory, asynchronously; copy_wait: this thread's have arrived
__device__ __forceinline__ void copy8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(saddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }
// waits for the phase of the given parity; false once the polls run out
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < (1 << 20); it++) {
        uint32_t ok;
        asm volatile(
            "{\n .reg .pred P;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 P, [%1], %2;\n selp.u32 %0, 1, 0, P;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// A CTA's share of a level of (nx-1) x (nz-1) interior nodes.  Its window holds rows k0 - 3 ..
// k0 + R + 2 of columns -3 .. nx + 3 at a pitch that is the same for every level, so that a stencil's
// shared loads have constant offsets; cells on and outside the walls stay zero (the stencils that
// reach them are folded, see the kernels).
constexpr int kPitch = 264, kMaxRows = kWarps + 2 * kReach, kWindow = kPitch * kMaxRows;
struct Strip {
    int R, c, k0, rows, last;  // CTA c's rows k0 .. k0 + rows - 1; last: the last CTA with rows

    __host__ __device__ static int rows_per_cta(int nz) { return (nz - 1 + kCtas - 1) / kCtas; }
    __host__ __device__ static int segments(int nx) { return (nx - 1 + 31) / 32; }

    // the strip of CTA c_, or the whole level (alone)
    __device__ __forceinline__ void set(int nz, int c_, bool alone) {
        R = alone ? nz - 1 : rows_per_cta(nz);
        c = alone ? 0 : c_;
        last = alone ? 0 : (nz - 2) / R;
        k0 = 1 + c * R;
        rows = max(0, min(R, nz - k0));
    }
    // cell of node (i, k) in this CTA's window; in CTA d's it lies (c - d) R rows further
    __device__ __forceinline__ int at(int i, int k) const { return (k - k0 + kReach) * kPitch + i + kReach; }
    // how many CTAs above (below) read the strip's row r: those next to it.  (reach - 1 - r) / R + 1 and
    // (r + reach) / R, bounded by the CTAs there are
    __device__ __forceinline__ int readers_up(int r) const {
        return r >= kReach ? 0 : min(c, R >= kReach ? 1 : R == 2 ? 2 - r : 3);
    }
    __device__ __forceinline__ int readers_down(int r) const {
        return min(last - c, R >= kReach ? (r + kReach >= R ? 1 : 0) : R == 2 ? 1 + r : 3);
    }
    // rows of other CTAs in this CTA's window
    __device__ __forceinline__ int rows_received(int nz) const {
        return rows == 0 ? 0 : min(kReach, k0 - 1) + max(0, min(R + kReach, nz - k0) - rows);
    }
};

// A node's way into the windows: its cell in this CTA's first window and, counted by an mbarrier of the
// receiver, in those of the CTAs above and below that read its row.  A CTA that has received a
// stage's rows from a neighbour knows that the neighbour has finished reading the rows it gets in
// return: who reads whom is symmetric and a value is published after its stencil was read.  So two
// windows in turn need no further handshake.
template <typename T>
struct Outlet {
    uint32_t cell, bar;  // shared addresses; window q is q kWindow elements further, its mbarrier 8 q bytes
    int up, down, R, c;
    uint32_t acell[2], abar[2];  // in the next CTA above and below
    __device__ __forceinline__ void set(const Strip& s, const T* win, const uint64_t* bars, int m, int up_, int down_) {
        cell = saddr(win + m);
        bar = saddr(bars);
        up = up_;
        down = down_;
        R = s.R;
        c = s.c;
        for (int q = 0; q < 2; q++) {
            const int d = q == 0 ? 1 : -1;  // CTA c - d
            const bool any = q == 0 ? up > 0 : down > 0;
            acell[q] = any ? remote(cell + d * R * kPitch * (int)sizeof(T), c - d) : 0;
            abar[q] = any ? remote(bar, c - d) : 0;
        }
    }
    __device__ __forceinline__ void put_remote(int q, T v) const {
        const uint32_t wo = (uint32_t)(q * kWindow * (int)sizeof(T)), bo = (uint32_t)(8 * q);
        if (up) put(acell[0] + wo, v, abar[0] + bo);
        if (down) put(acell[1] + wo, v, abar[1] + bo);
        if (up > 1 || down > 1) {  // strips of one or two rows
            const int step = R * kPitch * (int)sizeof(T);
            for (int d = 2; d <= up; d++) put(remote(cell + wo + d * step, c - d), v, remote(bar + bo, c - d));
            for (int d = 2; d <= down; d++) put(remote(cell + wo - d * step, c + d), v, remote(bar + bo, c + d));
        }
    }
};

// The two windows that stages fill in turn, and the mbarriers that count the other CTAs' rows
struct Exchange {
    uint32_t bar, parity, bytes;  // parity: bit q of window q
    bool ok;                      // false once a wait has run out: later waits are skipped
    __device__ __forceinline__ void init(const uint64_t* b) {
        bar = saddr(b);
        parity = 0;
        ok = true;
        if (threadIdx.x == 0) {
            bar_init(bar);
            bar_init(bar + 8);
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
    }
    // after a stage has been published into window q: its rows from every CTA are there
    __device__ __forceinline__ void arrive(int q) {
        if (threadIdx.x == 0) bar_expect(bar + 8 * q, bytes);
        __syncthreads();
        if (ok) ok = bar_wait(bar + 8 * q, parity >> q & 1u);
        parity ^= 1u << q;
    }
};

// the stretch of a level schedule that one launch walks
struct Visit {
    signed char level;
    unsigned char flags;
};
enum { kRestrict = 1, kProlong = 2, kZero = 4, kResidual = 8, kCoarse = 16 };
constexpr int kMaxVisits = 64;  // as many as a schedule has entries: a run is never cut
static_assert(kMaxVisits >= sizeof(Engine::multi) / sizeof(int) && kMaxVisits >= sizeof(Engine::mmulti) / sizeof(int),
              "a run holds every entry of a level schedule");

// the launch of one cluster; at: one attribute
static inline void cluster_launch(cudaLaunchConfig_t& cfg, cudaLaunchAttribute* at, size_t smem, cudaStream_t st) {
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {kCtas, 1, 1};
    cfg.gridDim = dim3(kCtas);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
}

}  // namespace cl
}  // namespace pt
