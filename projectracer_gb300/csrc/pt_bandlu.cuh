// pt_bandlu.cuh -- LU of the coarse band matrix with partial pivoting (DGBTF2's operations, in panels), and its
// explicit inverse.
//
// A panel of kPanel columns is factored by one CTA in shared memory (k_band_panel), then every column to
// its right that the panel reaches takes the panel's row interchanges, multipliers and updates in a CTA of
// its own (k_band_trail).  Every element sees the operations of the column-by-column DGBTF2 in the same
// order (interchanges permute rows, updates by ascending pivot column), so the factors of a finite matrix
// have the same bits; where DGBTF2 leaves an element alone, k_band_trail may add a product with a multiplier
// of zero, which turns a -0 into +0, and an infinite row spreads as NaN.  One CTA that updated the whole trailing block column by column was bound by its SM's FP64
// rate (two multiply-subtract pairs a cycle).  What bounds it now is the chain of a panel's columns:
// pivot search, reciprocal, scaling and the update of the next column.
// n = 2145, kl = ku = 99: 26 -> 3.2 ms; n = 561, kl = ku = 51: 2.2 -> 1.1 ms.
#pragma once
#include "pt_fp64.cuh"
#include "pt_launch.cuh"

namespace pt {
namespace bandlu {

constexpr int kPanel = 16;

// what panels leave for the columns to their right and for the inverse: per panel multipliers L[jj][r] in the
// rows' final order (r counts from the panel's first row), perm[r] = the row that ends at r, and top, the
// first row in which its columns of U have an entry; and the last column reached so far (1-based)
struct Work {
    double* L;
    int *perm, *top, *ju;
    int LD;  // kl + kPanel
    __host__ __device__ double* l(int panel) const { return L + (size_t)panel * kPanel * LD; }
    __host__ __device__ int* p(int panel) const { return perm + (size_t)panel * LD; }
};
static inline int panels(int n) { return (n + kPanel - 1) / kPanel; }
static inline size_t work_bytes(int n, int kl) {
    const size_t rows = (size_t)panels(n) * (kl + kPanel);
    return sizeof(double) * kPanel * rows + sizeof(int) * (rows + panels(n) + 1);
}
static inline Work work_of(void* base, int n, int kl) {
    Work w;
    w.LD = kl + kPanel;
    w.L = static_cast<double*>(base);
    w.perm = reinterpret_cast<int*>(w.L + (size_t)panels(n) * kPanel * w.LD);
    w.top = w.perm + (size_t)panels(n) * w.LD;
    w.ju = w.top + panels(n);
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
            if (r < R) w.l(j0 / kPanel)[(size_t)c * LD + r] = r > c && (usable >> c & 1u) ? v[c] : 0.0;
        if (r < R) w.p(j0 / kPanel)[r] = id;
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
        const int q = w.p(j0 / kPanel)[r];
        return q >= r0 ? col[q] : 0.0;
    };
    double t = lane < kPanel ? load(lane) : 0.0, v = tid >= kPanel && tid < R ? load(tid) : 0.0;
    double lt[kPanel], lv[kPanel];
    const double* const wl = w.l(j0 / kPanel);
#pragma unroll
    for (int jj = 0; jj < kPanel; jj++) {
        lt[jj] = lane < kPanel ? wl[(size_t)jj * LD + lane] : 0.0;
        lv[jj] = tid >= kPanel && tid < R ? wl[(size_t)jj * LD + tid] : 0.0;
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

// ---- explicit inverse G = (P L U)^{-1}, row-major, so that the coarse solve is a coalesced GEMV

// the first row in which a panel's columns of U have an entry (kv rows above the diagonal are stored, of
// which interchanges that did not happen leave the upper kl zero)
__global__ void k_band_top(const double* ab, int n, int kl, int ku, Work w) {
    const int ldab = 2 * kl + ku + 1, kv = ku + kl, j0 = blockIdx.x * kPanel;
    __shared__ int top;
    if (threadIdx.x == 0) top = j0;
    __syncthreads();
    for (int c = j0; c < min(j0 + kPanel, n); c++)
        for (int i = max(0, c - kv) + threadIdx.x; i < j0; i += blockDim.x)
            if (nonzero(ab[(size_t)c * ldab + kv + i - c])) {
                atomicMin(&top, i);
                break;  // (a thread's rows ascend)
            }
    __syncthreads();
    if (threadIdx.x == 0) w.top[blockIdx.x] = top;
}

// COLS columns of G per CTA: unit vectors through the panels' interchanges, multipliers and updates, then
// back through U, the operations of the column-by-column DGBTRS in the same order for every element.  Per
// panel the kPanel x kPanel triangle is solved with a lane per row (two columns per warp), the other rows
// with COLS / 4 threads per row, four columns each.  The window of rows that a panel reaches is in shared
// memory, twice for the forward pass, whose interchanges permute it.
// What bounds it is the FP64 rate (n^2 (kl / 2 + ku) multiply-subtract pairs): n = 2145, kl = ku = 99:
// 11.2 ms with a warp per column (a division per column and step, partly filled warps, the zeros of U
// above its entries), 6.1 now; n = 561, kl = ku = 51: 0.65 before and now.  A grid of fewer CTAs than groups
// of columns takes them in turn (see inverse).
constexpr int kInvThreads = 256, kInvCols = 4;  // columns of a thread
static inline int pow2_above(int v) {
    int w = 32;
    while (w < v) w *= 2;
    return w;
}
static inline size_t inverse_smem(int kl, int ku, int cols) {
    const int f = 2 * pow2_above(kl + 2 * kPanel), b = pow2_above(kl + ku + 2 * kPanel);
    return sizeof(double) * (size_t)(f > b ? f : b) * cols;
}
template <int COLS>
__global__ void __launch_bounds__(kInvThreads, 2) k_band_inverse(const double* __restrict__ ab, double* G, int n, int kl, int ku,
                                                            Work w, int tops, int WF, int WB, FmaForms F) {
    constexpr int H = COLS / kInvCols;  // threads per row
    extern __shared__ __align__(16) double win[];
    __shared__ __align__(16) double ys[kPanel][COLS];
    __shared__ double ut[2][kPanel][kPanel], rec[2][kPanel];  // ut[.][jj][r] = U(j0 + r, j0 + jj)
    const int ldab = 2 * kl + ku + 1, kv = ku + kl, LD = w.LD, np = (n + kPanel - 1) / kPanel;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row = lane & 15, col = 2 * warp + (lane >> 4);  // of the triangle: warps below COLS / 2
    const bool tri = warp < COLS / 2;
    const int h4 = (tid % H) * kInvCols;

    for (int c0 = blockIdx.x * COLS; c0 < n; c0 += gridDim.x * COLS) {
        const bool live = tri && c0 + col < n;

        // forward
        const int ps = max(0, (c0 - LD + kPanel) / kPanel);  // the first panel that reaches row c0
        for (int q = tid; q < min(ps * kPanel, n) * COLS; q += kInvThreads)
            if (c0 + q % COLS < n) G[(size_t)(q / COLS) * n + c0 + q % COLS] = 0.0;
        double* A = win;                      // the panel's window, row i in slot i mod WF
        double* B = win + (size_t)WF * COLS;  // the next one's
        auto enter = [&](double* W, int from, int to) {
            for (int q = from * COLS + tid; q < to * COLS; q += kInvThreads)
                W[(size_t)(q / COLS & (WF - 1)) * COLS + q % COLS] = q / COLS == c0 + q % COLS ? 1.0 : 0.0;
        };
        enter(A, ps * kPanel, min(n, ps * kPanel + LD));
        __syncthreads();
        for (int p = ps; p < np; p++) {
            const int j0 = p * kPanel, R = min(LD, n - j0), nb = min(kPanel, n - j0);
            const double* const L = w.l(p);
            const int* const perm = w.p(p);
            double l[kPanel];
            int it = tid;  // item: row kPanel + it / H, columns h4 ..
            const int items = max(0, R - kPanel) * H;
            auto load = [&](int r) {
    #pragma unroll
                for (int jj = 0; jj < kPanel; jj++) l[jj] = L[(size_t)jj * LD + r];
            };
            if (tri) {
                double t = row < nb ? A[(size_t)((j0 + perm[row]) & (WF - 1)) * COLS + col] : 0.0;
                if (row < nb) load(row);
    #pragma unroll
                for (int jj = 0; jj < kPanel; jj++) {
                    const double y = __shfl_sync(0xffffffffu, t, jj + (lane & 16));
                    const double u = F.add(t, F.mul(l[jj], -y));
                    if (row > jj && row < nb) t = u;
                }
                ys[row][col] = t;
                if (live && row < nb) G[(size_t)(j0 + row) * n + c0 + col] = t;
            }
            if (it < items) load(kPanel + it / H);
            __syncthreads();
            for (; it < items; it += kInvThreads) {
                const int r = kPanel + it / H;
                if (it != tid) load(r);
                const double* a = A + (size_t)((j0 + perm[r]) & (WF - 1)) * COLS + h4;
                double v[kInvCols];
    #pragma unroll
                for (int c = 0; c < kInvCols; c++) v[c] = a[c];
    #pragma unroll
                for (int jj = 0; jj < kPanel; jj++) {
                    const volatile double* y = &ys[jj][h4];  // (volatile: 64 values loaded ahead would fill the registers)
    #pragma unroll
                    for (int c = 0; c < kInvCols; c++) v[c] = F.add(v[c], F.mul(l[jj], -y[c]));
                }
                double* b = B + (size_t)((j0 + r) & (WF - 1)) * COLS + h4;
    #pragma unroll
                for (int c = 0; c < kInvCols; c++) b[c] = v[c];
            }
            enter(B, min(n, j0 + LD), min(n, j0 + kPanel + LD));
            __syncthreads();
            double* const x = A;
            A = B;
            B = x;
        }

        // back: row i in slot i mod WB
        auto fetch = [&](int p, int buf) {  // a panel's triangle: threads 0 .. 255, (jj, r)
            const int jj = tid / kPanel, r = tid % kPanel, j = p * kPanel + jj;
            const double u = j < n && r <= jj ? ab[(size_t)j * ldab + kv + r - jj] : 1.0;
            ut[buf][jj][r] = u;
            if (r == jj) rec[buf][jj] = 1.0 / u;
        };
        int lo = max(0, (np - 1) * kPanel - kv);  // rows lo .. are in the window
        for (int q = lo * COLS + tid; q < n * COLS; q += kInvThreads)
            win[(size_t)(q / COLS & (WB - 1)) * COLS + q % COLS] = c0 + q % COLS < n ? G[(size_t)(q / COLS) * n + c0 + q % COLS] : 0.0;
        fetch(np - 1, 0);
        __syncthreads();
        for (int p = np - 1, buf = 0; p >= 0; p--, buf ^= 1) {
            const int j0 = p * kPanel, nb = min(kPanel, n - j0), top = tops ? w.top[p] : max(0, j0 - kv);
            double u[kPanel];
            auto load = [&](int i) {
    #pragma unroll
                for (int jj = 0; jj < kPanel; jj++)
                    u[jj] = j0 + jj < n && i >= j0 + jj - kv ? ab[(size_t)(j0 + jj) * ldab + kv + i - j0 - jj] : 0.0;
            };
            // rows that enter for the next panel
            const int next = max(0, j0 - kPanel - kv), entering = (lo - next) * COLS;
            double e = 0.0;
            if (tid < entering && c0 + tid % COLS < n) e = G[(size_t)(next + tid / COLS) * n + c0 + tid % COLS];
            int it = tid;  // item: row top + it / H
            const int items = (j0 - top) * H;
            if (it < items) load(top + it / H);
            if (tri) {
                double t = row < nb ? win[(size_t)((j0 + row) & (WB - 1)) * COLS + col] : 0.0;
    #pragma unroll
                for (int jj = kPanel - 1; jj >= 0; jj--) {
                    if (jj >= nb) continue;
                    const double y = __shfl_sync(0xffffffffu, t, jj + (lane & 16)), d = ut[buf][jj][jj];
                    double x = y;
                    if (nonzero(y)) x = in_range(y, 800) && in_range(d, 100) ? quotient(y, d, rec[buf][jj]) : y / d;
                    __syncwarp();
                    const double s = F.sub(t, F.mul(x, ut[buf][jj][row]));
                    if (row < jj) t = s;
                    if (row == jj) t = x;
                }
                ys[row][col] = row < nb ? t : 0.0;
                if (live && row < nb) G[(size_t)(j0 + row) * n + c0 + col] = t;
            }
            if (p > 0) fetch(p - 1, buf ^ 1);
            __syncthreads();
            for (; it < items; it += kInvThreads) {
                const int i = top + it / H;
                if (it != tid) load(i);
                double* a = win + (size_t)(i & (WB - 1)) * COLS + h4;
                double v[kInvCols];
    #pragma unroll
                for (int c = 0; c < kInvCols; c++) v[c] = a[c];
    #pragma unroll
                for (int jj = kPanel - 1; jj >= 0; jj--) {
                    const volatile double* y = &ys[jj][h4];
    #pragma unroll
                    for (int c = 0; c < kInvCols; c++) v[c] = F.sub(v[c], F.mul(y[c], u[jj]));
                }
    #pragma unroll
                for (int c = 0; c < kInvCols; c++) a[c] = v[c];
            }
            if (tid < entering) win[(size_t)((next + tid / COLS) & (WB - 1)) * COLS + tid % COLS] = e;
            lo = next;
            __syncthreads();
        }
    }
}

// Eight columns per CTA where that leaves more than one CTA per SM, else four.
// clusters = 0: a CTA per group of columns, the whole chip.  Otherwise (beside the solves of another stream) that
// many clusters of kInvCluster CTAs, one CTA an SM: the CTAs are independent, the clusters only keep them on a
// few GPCs.  Two CTAs fill an SM's registers, and one on every SM leaves no 16 SMs of a GPC to the cycle's cluster
// kernels (pt_cluster.cuh), so a solve that met the whole-chip form waited for its end: with n = 2145 one of
// 1.6 ms took 5.0 (2048x1024), one of 0.62 took 2.95 (1024x512, five levels); beside six clusters (10.6 ms
// instead of 6.1) 2.0 and 0.72.
constexpr int kInvCluster = 16;
constexpr size_t kInvAlone = 116 * 1024;  // shared memory that a second CTA does not find on an SM
static inline size_t inverse_smem_alone(int kl, int ku, int cols) {
    const size_t b = inverse_smem(kl, ku, cols);
    return b > kInvAlone ? b : kInvAlone;
}
static inline int inverse_cols(int n) { return n > 8 * 152 ? 8 : 4; }
static int inverse(const double* ab, double* G, int n, int kl, int ku, const Work& w, cudaStream_t st, int clusters = 0) {
    const int WF = pow2_above(kl + 2 * kPanel), WB = pow2_above(kl + ku + 2 * kPanel);
    const int tops = n > 256;  // (a launch costs more than a small band's zeros)
    if (tops) PT_COUNT(), k_band_top<<<panels(n), 128, 0, st>>>(ab, n, kl, ku, w);
    const int cols = inverse_cols(n), groups = (n + cols - 1) / cols;
    const auto kernel = cols == 8 ? k_band_inverse<8> : k_band_inverse<4>;
    if (clusters == 0) {
        PT_COUNT(), kernel<<<groups, kInvThreads, inverse_smem(kl, ku, cols), st>>>(ab, G, n, kl, ku, w, tops, WF, WB,
                                                                                 FmaForms());
        return cuda_check(cudaGetLastError(), "k_band_inverse");
    }
    const int need = (groups + kInvCluster - 1) / kInvCluster;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {kInvCluster, 1, 1};
    cfg.gridDim = dim3(kInvCluster * (need < clusters ? need : clusters));
    cfg.blockDim = dim3(kInvThreads);
    cfg.dynamicSmemBytes = inverse_smem_alone(kl, ku, cols);
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    PT_COUNT();
    return cuda_check(cudaLaunchKernelEx(&cfg, kernel, ab, G, n, kl, ku, w, tops, WF, WB, FmaForms()), "k_band_inverse");
}
// *clusters: as many as can run at once, less one, so that a cycle's cluster finds its SMs; 0 where that leaves none
static int inverse_setup(int n, int kl, int ku, int* clusters) {
    const int cols = inverse_cols(n);
    const auto kernel = cols == 8 ? k_band_inverse<8> : k_band_inverse<4>;
    const size_t smem = inverse_smem_alone(kl, ku, cols);
    if (int rc = cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                            "coarse inverse"))
        return rc;
    if (int rc = cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1),
                            "coarse inverse"))
        return rc;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {kInvCluster, 1, 1};
    cfg.gridDim = dim3(kInvCluster);
    cfg.blockDim = dim3(kInvThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int fit = 0;
    if (cudaOccupancyMaxActiveClusters(&fit, kernel, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        fit = 0;
    }
    *clusters = fit > 1 ? fit - 1 : 0;
    return 0;
}

}  // namespace bandlu
}  // namespace pt
