// pt_bandlu.cuh -- LU of the coarse band matrix with partial pivoting (DGBTF2's operations, in panels).
//
// A panel of kPanel columns is factored by one CTA in shared memory (k_band_panel), then every column to
// its right that the panel reaches takes the panel's row interchanges, multipliers and updates in a CTA of
// its own (k_band_trail).  Every element sees the operations of the column-by-column DGBTF2 in the same
// order (interchanges permute rows, updates by ascending pivot column), so the factors are the same
// bit for bit; one CTA that updated the whole trailing block column by column was bound by its SM's FP64
// rate (two multiply-subtract pairs a cycle).  What bounds it now is the chain of a panel's columns:
// pivot search, reciprocal, scaling and the update of the next column.
// n = 2145, kl = ku = 99: 26 -> 3.2 ms; n = 561, kl = ku = 51: 2.2 -> 0.9 ms.
#pragma once
#include "pt_launch.cuh"

namespace pt {
namespace bandlu {

constexpr int kPanel = 16;

// what a panel leaves for the columns to its right: multipliers L[jj][r] in the rows' final order (r counts
// from the panel's first row), perm[r] = the row that ends at r, and the last column it reaches (1-based,
// the running maximum)
struct Work {
    double* L;
    int *perm, *ju;
};
static inline size_t work_bytes(int kl) { return sizeof(double) * kPanel * (kl + kPanel) + sizeof(int) * (kl + kPanel + 1); }
static inline Work work_of(void* base, int kl) {
    Work w;
    w.L = static_cast<double*>(base);
    w.perm = reinterpret_cast<int*>(w.L + (size_t)kPanel * (kl + kPanel));
    w.ju = w.perm + kl + kPanel;
    return w;
}
static inline int row_threads(int kl) { return (kl + kPanel + 31) / 32 * 32; }

// the band's fill-in rows
__global__ void k_band_fill(double* ab, int n, int kl, int ku, Work w) {
    const int ldab = 2 * kl + ku + 1, kv = ku + kl, j = blockIdx.x;
    if (j == 0 && threadIdx.x == 0) *w.ju = 1;
    for (int i = max(0, kv - j) + threadIdx.x; i < kl; i += blockDim.x) ab[(size_t)j * ldab + i] = 0.0;
}

// tests of FP64 values as integers: the FP64 pipe takes 64 cycles for a warp's comparison
__device__ __forceinline__ bool nonzero(double y) { return (__double_as_longlong(y) << 1) != 0; }
__device__ __forceinline__ unsigned long long magnitude_key(double x) {  // 0 for a NaN, else 1 + |x|'s bits
    const unsigned long long m = (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
    return m > 0x7ff0000000000000ull ? 0 : m + 1;
}

// Columns j0 .. j0 + kPanel - 1 (0-based).  A thread per row holds the row's kPanel entries in registers;
// rows are exchanged through shared memory.  The last warp picks the pivot among the row warps' candidates
// and takes its reciprocal, while the row warps apply the previous column's updates to the columns beyond
// the next one: FP64 instructions issue every 64 cycles, a reciprocal is a chain of them, and so is a
// column (24 us for 16 columns, kl = 99).  err: the first column without a usable pivot.
__global__ void __launch_bounds__(512) k_band_panel(double* ab, int* ipiv, int n, int kl, int ku, int j0, Work w, int* err) {
    pdl_begin();
    __shared__ double s_u[kPanel][kPanel], s_x[kPanel], s_val[16], s_rp;
    __shared__ unsigned long long s_key[16];
    __shared__ int s_row[16], s_bi, s_nz, s_id[2];
    const int ldab = 2 * kl + ku + 1, kv = ku + kl, LD = kl + kPanel, R = min(LD, n - j0), nb = min(kPanel, n - j0);
    const int r = threadIdx.x, lane = r & 31, warp = r >> 5, nw = (int)(blockDim.x >> 5) - 1;  // nw row warps
    double* const base = ab + (size_t)j0 * ldab + kv;  // row j0 + r of column j0 + c at base[r + c (ldab - 1)]
    double v[kPanel], l = 0.0;  // l: the row's multiplier of the previous column, where it has one (act)
    bool act = false;
    int id = r, ju = 1;
    unsigned usable = 0;
#pragma unroll
    for (int c = 0; c < kPanel; c++)
        v[c] = warp < nw && r < R && c < nb && r - c <= kl ? base[r + (size_t)c * (ldab - 1)] : 0.0;
#pragma unroll
    for (int jj = 0; jj < kPanel; jj++) {
        if (jj >= nb) break;
        const int km = min(kl, n - 1 - j0 - jj);
        if (warp < nw) {  // the first row of the largest |a|; a NaN never wins
            const unsigned long long key = r >= jj && r <= jj + km ? magnitude_key(v[jj]) : 0;
            const unsigned hi = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32));
            const unsigned lo = __reduce_max_sync(0xffffffffu, (unsigned)(key >> 32) == hi ? (unsigned)key : 0u);
            const unsigned long long top = ((unsigned long long)hi << 32) | lo;
            if (lane == __ffs(__ballot_sync(0xffffffffu, key == top)) - 1) {
                s_key[warp] = top;
                s_row[warp] = r;
                s_val[warp] = v[jj];
            }
        }
        __syncthreads();
        if (warp == nw) {
            if (lane == 0) {
                unsigned long long best = 0;
                int q = 0;
                for (int t = 0; t < nw; t++)
                    if (s_key[t] > best) {
                        best = s_key[t];
                        q = t;
                    }
                const int row = best ? s_row[q] : jj;  // (a column of NaNs: its first row)
                const bool nz = best > 1;              // neither NaN nor zero
                s_bi = row - jj;
                s_nz = nz;
                if (nz) {
                    s_rp = 1.0 / s_val[q];
                    ju = max(ju, min(j0 + row + 1 + ku, n));
                } else {
                    atomicCAS(err, 0, j0 + jj + 1);
                }
                ipiv[j0 + jj] = j0 + row + 1;
            }
        } else if (jj > 0) {
#pragma unroll
            for (int c = jj + 1; c < kPanel; c++) {
                const double y = s_u[jj - 1][c], t = v[c] + l * -y;
                if (act && nonzero(y)) v[c] = t;
            }
        }
        __syncthreads();
        const int bi = s_bi;
        act = false;
        if (s_nz) {
            usable |= 1u << jj;
            if (warp < nw && r == jj + bi) {
                s_id[0] = id;
#pragma unroll
                for (int c = 0; c < kPanel; c++) s_u[jj][c] = v[c];
            }
            if (bi && r == jj) {
                s_id[1] = id;
#pragma unroll
                for (int c = 0; c < kPanel; c++) s_x[c] = v[c];
            }
            __syncthreads();
            if (warp < nw) {
                if (bi && r == jj) {
                    id = s_id[0];
#pragma unroll
                    for (int c = 0; c < kPanel; c++) v[c] = s_u[jj][c];
                }
                if (bi && r == jj + bi) {
                    id = s_id[1];
#pragma unroll
                    for (int c = 0; c < kPanel; c++) v[c] = s_x[c];
                }
                act = r > jj && r <= jj + km;
                if (act) l = v[jj] = v[jj] * s_rp;
                if (jj + 1 < kPanel) {
                    const double y = s_u[jj][(jj + 1) % kPanel], t = v[(jj + 1) % kPanel] + l * -y;
                    if (act && nonzero(y)) v[(jj + 1) % kPanel] = t;
                }
            }
        }
        if (warp < nw && r <= jj + km) base[r + (size_t)jj * (ldab - 1)] = v[jj];  // final, multipliers in place
    }
    if (warp < nw) {
#pragma unroll
        for (int c = 0; c < kPanel; c++)
            if (r < R) w.L[(size_t)c * LD + r] = r > c && (usable >> c & 1u) ? v[c] : 0.0;
        if (r < R) w.perm[r] = id;
    } else if (lane == 0) {
        *w.ju = max(*w.ju, ju);
    }
}

// column j0 + kPanel + blockIdx.x: the panel's interchanges, then its updates in order; a thread per row,
// the kPanel top rows (whose values scale the updates) in the first lanes of every warp too
__global__ void __launch_bounds__(512) k_band_trail(double* ab, int n, int kl, int ku, int j0, Work w) {
    pdl_begin();
    const int ldab = 2 * kl + ku + 1, kv = ku + kl, LD = kl + kPanel, R = min(LD, n - j0);
    const int c = j0 + kPanel + blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    if (c + 1 > *w.ju) return;
    double* const col = ab + (size_t)c * ldab + kv + j0 - c;  // row j0 + r at col[r], stored from r >= r0
    const int r0 = c - kv - j0;
    auto load = [&](int r) {
        const int q = w.perm[r];
        return q >= r0 ? col[q] : 0.0;
    };
    double t = lane < kPanel ? load(lane) : 0.0, v = tid >= kPanel && tid < R ? load(tid) : 0.0;
    double lt[kPanel], lv[kPanel];
#pragma unroll
    for (int jj = 0; jj < kPanel; jj++) {
        lt[jj] = lane < kPanel ? w.L[(size_t)jj * LD + lane] : 0.0;
        lv[jj] = tid >= kPanel && tid < R ? w.L[(size_t)jj * LD + tid] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int jj = 0; jj < kPanel; jj++) {
        const double y = __shfl_sync(0xffffffffu, t, jj);
        if (nonzero(y)) {
            const double s = -y;
            if (lane > jj && lane < kPanel) t = t + lt[jj] * s;
            v = v + lv[jj] * s;
        }
    }
    if (tid < kPanel) v = t;
    if (tid < R && tid >= r0) col[tid] = v;
}

static int factor(double* ab, int* ipiv, int n, int kl, int ku, const Work& w, int* err, cudaStream_t st) {
    PT_COUNT(), k_band_fill<<<n, 128, 0, st>>>(ab, n, kl, ku, w);
    if (int rc = cuda_check(cudaGetLastError(), "k_band_fill")) return rc;
    for (int j0 = 0; j0 < n; j0 += kPanel) {
        if (int rc = launch_pdl("k_band_panel", k_band_panel, dim3(1), dim3(row_threads(kl) + 32), 0, st, ab, ipiv, n, kl, ku,
                                j0, w, err))
            return rc;
        const int nc = n - j0 - kPanel < kl + ku ? n - j0 - kPanel : kl + ku;
        if (nc <= 0) break;
        if (int rc = launch_pdl("k_band_trail", k_band_trail, dim3(nc), dim3(row_threads(kl)), 0, st, ab, n, kl,
                                ku, j0, w))
            return rc;
    }
    return 0;
}

}  // namespace bandlu
}  // namespace pt
