// pt_mg.cu -- the variable-viscosity biharmonic stream-function solve (FP64): multigrid driver
// (iterative_solver.f90:124-341) with the reference's level schedule, the viscosity pipeline
// (compute_viscosity 560-634, smoother_vis smoother.f90:454-580, viscosity_gradients 472-558,
// test_eigenvalues 1147-1211), the RKC1 smoother (iterate_stream 1418-1614), residual (415-470),
// transfers (restrict 1107-1125, prolong 343-396) and the coarsest-grid banded LU
// (Compute_Matrix_coarse 1701-1844 + DGBEQU/DGBTRF/DGBTRS) -- all on the device.
//
// The RKC1 stage kernel fuses stream_derivatives + stream_space + the three-term recurrence +
// enforceBCs_stream: each thread evaluates the 10 stencil derivatives of S_{j-1} at its node
// (separable 5x5/7-point stencils), writes S_j and the antisymmetric ghost images of S_j, so one
// launch is one stage.  Error arrays keep the reference's quirk: error(:,:,2:grids) is never
// reset, so a coarse visit starts from the previous coarse correction.
#include <cmath>
#include <cstring>
#include <vector>

#include "pt_bandlu.cuh"
#include "pt_cluster.cuh"
#include "pt_consts.cuh"
#include "pt_exact.cuh"
#include "pt_launch.cuh"

namespace pt {

int upload_consts_mg(const Engine& E) { return upload_tu_consts(E); }

struct VisSet {
    double *vis, *vx, *vz, *vxx, *vzz, *vxz, *vxxpzz, *vxxmzz, *vsm, *ratio, *dtst;
};

// where a viscosity pass runs and writes: the stream, the test_eig scalars, the work arrays and
// the level arrays (the cycle's own, or the side set of the next time level)
struct VisCtx {
    cudaStream_t st;
    double *dscal, *hscal;
    double* const* visw;
    VisLevels V;
};

static VisLevels primary_levels(Engine& E) {
    VisLevels V{};
    for (int l = 0; l < PT_MAXLEV; l++) {
        V.vis[l] = E.vis[l]; V.visst[l] = E.visst[l]; V.vx[l] = E.vx[l]; V.vz[l] = E.vz[l]; V.vxx[l] = E.vxx[l];
        V.vzz[l] = E.vzz[l]; V.vxz[l] = E.vxz[l]; V.vxxpzz[l] = E.vxxpzz[l]; V.vxxmzz[l] = E.vxxmzz[l];
        V.vsm[l] = E.vsm[l]; V.ratio[l] = E.ratio[l]; V.dtst[l] = E.dtst[l];
    }
    return V;
}
static VisCtx primary_ctx(Engine& E) { return VisCtx{E.st, E.dscal, E.hscal, E.visw, primary_levels(E)}; }
static VisCtx side_ctx(Engine& E) { return VisCtx{E.st2, E.dscal2, E.hscal2, E.visw2, E.vl2}; }

static VisSet level_set(const VisLevels& V, int l) {
    return VisSet{V.vis[l], V.vx[l], V.vz[l], V.vxx[l], V.vzz[l], V.vxz[l], V.vxxpzz[l], V.vxxmzz[l],
                  V.vsm[l], V.ratio[l], V.dtst[l]};
}

// ------------------------------------------------------------------ viscosity pipeline
// visf, rheology.f90:2-23
__global__ void k_visf(double* visst, const double* Tvis, const double* Cvis, Geo g) {
    int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (i > cK.nx) return;
    double z = (double)k * cK.ds;
    if (k == 0) z = 0.0;
    if (k == cK.nz) z = 1.0;
    double v;
    if (cK.ivis == 1) v = exp(-Tvis[g.at(i, k)] * cK.lvisT + (1.0 - z) * cK.lvisP);
    else if (cK.ivis == 2 && cK.comp == 1) {
        double dot = 0.0 + Cvis[g.at(i, k)] * cK.lvisC;
        v = exp(-Tvis[g.at(i, k)] * cK.lvisT - dot + (1.0 - z) * cK.lvisP);
    } else v = 1.0;
    visst[g.at(i, k)] = v;
}

// viscosityBCs (iterative_solver.f90:666-690): phase 1 column ghosts over all rows (the row
// ghosts still hold the previous values there), phase 2 row ghosts for columns 0..nx.
__global__ void k_visbc_cols(double* v, Geo g, int nx, int nz) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 6 * (nz + 7)) return;
    int k = idx / 6 - 3, q = idx % 6;
    int j = q % 3 + 1;
    if (q < 3) v[g.at(-j, k)] = v[g.at(j, k)];
    else v[g.at(nx + j, k)] = v[g.at(nx - j, k)];
}
__global__ void k_visbc_rows(double* v, Geo g, int nx, int nz) {
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= 6 * (nx + 1)) return;
    int i = idx / 6, q = idx % 6;
    int j = q % 3 + 1;
    if (q < 3) v[g.at(i, -j)] = v[g.at(i, j)];
    else v[g.at(i, nz + j)] = v[g.at(i, nz - j)];
}
static int vis_bcs(Engine& E, double* v, int l, cudaStream_t st) {
    const Geo& g = E.gl[l];
    PT_COUNT(), k_visbc_cols<<<nblk(6 * (g.nz + 7), 128), 128, 0, st>>>(v, g, g.nx, g.nz);
    PT_COUNT(), k_visbc_rows<<<nblk(6 * (g.nx + 1), 128), 128, 0, st>>>(v, g, g.nx, g.nz);
    CKL("vis_bcs");
    return 0;
}

// c + a b: fused (fma) for the fast paths, two roundings in the reference's order for the FP64
// path with reference_rounding (this file is compiled with --fmad=false, so only fma() fuses)
template <bool FUSED>
__device__ __forceinline__ double madd(double a, double b, double c) {
    return FUSED ? fma(a, b, c) : c + a * b;
}

// viscosity_gradients, second-order stencils (uniform grid)
template <bool FUSED>
__global__ void k_vis_grad(VisSet S, Geo g, int l, int full, int ivis) {
    int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    const LevConst& L = cL[l];
    if (i > L.nx) return;
    size_t o = g.at(i, k);
    if (ivis == 0) {
        S.vx[o] = 0; S.vz[o] = 0; S.vxx[o] = 0; S.vzz[o] = 0; S.vxz[o] = 0; S.vxxpzz[o] = 0; S.vxxmzz[o] = 0;
        return;
    }
    const double* v = S.vis;
    double xx = 0.0, zz = 0.0;
    for (int j = -1; j <= 1; j++) xx = madd<FUSED>(cK.D2so[j + 1], v[g.at(i + j, k)], xx);
    xx = qdiv(xx, L.dr2, L.idr2);
    for (int j = -1; j <= 1; j++) zz = madd<FUSED>(cK.D2so[j + 1], v[g.at(i, k + j)], zz);
    zz = qdiv(zz, L.ds2, L.ids2);
    if (full) {
        double xz = 0.0, x = 0.0, z = 0.0;
        for (int k2 = -1; k2 <= 1; k2++)
            for (int i2 = -1; i2 <= 1; i2++) xz = madd<FUSED>(cK.Drsso[i2 + 1][k2 + 1], v[g.at(i + i2, k + k2)], xz);
        for (int j = -1; j <= 1; j++) x = madd<FUSED>(cK.D1so[j + 1], v[g.at(i + j, k)], x);
        for (int j = -1; j <= 1; j++) z = madd<FUSED>(cK.D1so[j + 1], v[g.at(i, k + j)], z);
        S.vxz[o] = qdiv(xz, L.drds, L.idrds);
        S.vx[o] = qdiv(x, L.dr, L.idr);
        S.vz[o] = qdiv(z, L.ds, L.ids);
        S.vxxmzz[o] = xx - zz;
    }
    S.vxx[o] = xx;
    S.vzz[o] = zz;
    S.vxxpzz[o] = xx + zz;
    S.vsm[o] = L.dt_vis * (xx + zz);
}

// test_eigenvalues (RKC1 branch): ratio, local pseudo-time step, min ratio
// FEW (mixed precision): the pseudo-time step with two divisions instead of four, by the
// reciprocals of ae and be (the step feeds an FP32 smoother there); the ratio keeps its division.
// FUSED: the sums as fused multiply-adds (not with reference_rounding).
template <bool FEW, bool FUSED>
__global__ void k_test_eig(VisSet S, Geo g, int l, double ae, double be, double ctemp, unsigned long long* rmin) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
    const LevConst& L = cL[l];
    double ratio = 1.0e100;
    if (i <= L.nx - 1) {
        size_t o = g.at(i, k);
        double vg = S.vis[o];
        double eI = madd<FUSED>(vg, L.SI2, fabs(S.vxxpzz[o] * L.SI1)) + fabs(S.vxz[o] * L.SI4) + fabs(S.vx[o] * L.SI5) +
                    fabs(S.vz[o] * L.SI6);
        double eR = madd<FUSED>(vg, L.SR2, S.vxxmzz[o] * L.SR1);
        eR = madd<FUSED>(S.vxz[o], L.SR4, eR);
        eR = madd<FUSED>(S.vx[o], L.SR5, eR);
        eR = madd<FUSED>(S.vz[o], L.SR6, eR);
        ratio = fabs(eR / eI);
        S.ratio[o] = ratio;
        const double a = FEW ? eR * ae : eR / ae, b = FEW ? eI * be : eI / be;  // FEW: ae, be are 1/ae, 1/be
        S.dtst[o] = ctemp * eR / madd<FUSED>(a, a, b * b);
    }
    double m = fmin(ratio, 1.0e100);
    for (int off = 16; off > 0; off >>= 1) m = fmin(m, __shfl_xor_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) atomicMin(rmin, (unsigned long long)__double_as_longlong(m));
}

// The smoothing update v += c vsm (smoother_vis) followed by viscosityBCs, in one pass.  Every node writes its own mirror images:
// the column and row ghosts take the updated value; a corner ghost is what viscosityBCs' column
// phase copies from the row ghost of the mirrored column, which still holds what the previous
// call wrote there: the mirrored node's value before this update.  (The first call of a smoothing
// pass is a plain vis_bcs, so that previous call always exists.)
template <bool FUSED>
__global__ void k_vis_update_bc(double* v, const double* vsm, Geo g, int nx, int nz, double c) {
    int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (i > nx) return;
    const size_t o = g.at(i, k);
    const double old = v[o];
    const double nv = madd<FUSED>(c, vsm[o], old);
    v[o] = nv;
    int xs[2], zs[2], nxm = 0, nzm = 0;
    if (i >= 1 && i <= 3) xs[nxm++] = -i;
    if (i >= nx - 3 && i <= nx - 1) xs[nxm++] = 2 * nx - i;
    if (k >= 1 && k <= 3) zs[nzm++] = -k;
    if (k >= nz - 3 && k <= nz - 1) zs[nzm++] = 2 * nz - k;
    for (int a = 0; a < nxm; a++) v[g.at(xs[a], k)] = nv;
    for (int b = 0; b < nzm; b++) v[g.at(i, zs[b])] = nv;
    for (int a = 0; a < nxm; a++)
        for (int b = 0; b < nzm; b++) v[g.at(xs[a], zs[b])] = old;
}

static const double kPi = 3.1415926535897932;

// smoother_vis (smoother.f90:454-580) on the arrays of set S at level l
static int smoother_vis(Engine& E, const VisCtx& C, int l, int interpolate, VisSet S, int record) {
    const Geo& g = E.gl[l];
    const int nx = g.nx, nz = g.nz, ivis = E.cfg.ivis;
    int rc;
    if ((rc = vis_bcs(E, S.vis, l, C.st))) return rc;
    int option, Niter;
    double lb, la;
    if (interpolate == 0) { option = 1; Niter = 3; lb = -3.0; la = -2.0; }
    else { option = 0; Niter = E.cfg.vis_iter; lb = -2.0; la = -1.0; }
    int Nvis_store = 0, nn_store = 1, n = 0, trigger = 0;
    double ratio_min = 1.0e100;
    // the pseudo-time step (test_eigenvalues) matches the smoother that will run on level l: the
    // mixed V-cycle's coarse-level smoother has its own stage count
    const bool coarse_smoother = E.cfg.precision == PT_PREC_MIXED && l >= 2;
    const double stab = coarse_smoother ? E.RKC1_stability_c : E.RKC1_stability;
    const double ae = -stab / 2.0, be = (double)(coarse_smoother ? E.nstageC : E.cfg.nstageS);
    const double ctemp = E.cfg.courant_stream * (stab / (ae * ae));
    const bool fused = !E.cfg.reference_rounding;
    dim3 gg(nblk(nx + 1, 128), nz + 1);
    for (int guard = 0; guard < 100000; guard++) {
        for (int nn = nn_store; nn <= Niter; nn++) {
            PT_COUNT(), (fused ? k_vis_grad<true> : k_vis_grad<false>)<<<gg, 128, 0, C.st>>>(S, g, l, Nvis_store != 0,
                                                                                        ivis);
            CKL("k_vis_grad");
            if (interpolate == 0 && (Nvis_store >= 1 || ivis == 0)) {
                unsigned long long* d = (unsigned long long*)C.dscal;
                unsigned long long init = (unsigned long long)__builtin_bit_cast(long long, 1.0e100);
                CK(cudaMemcpyAsync(d, &init, 8, cudaMemcpyHostToDevice, C.st));
                dim3 ge(nblk(nx - 1, 128), nz - 1);
                if (E.cfg.precision == PT_PREC_MIXED)
                    PT_COUNT(), k_test_eig<true, true><<<ge, 128, 0, C.st>>>(S, g, l, 1.0 / ae, 1.0 / be, ctemp, d);
                else if (fused)
                    PT_COUNT(), k_test_eig<false, true><<<ge, 128, 0, C.st>>>(S, g, l, ae, be, ctemp, d);
                else
                    PT_COUNT(), k_test_eig<false, false><<<ge, 128, 0, C.st>>>(S, g, l, ae, be, ctemp, d);
                CKL("k_test_eig");
                CK(cudaMemcpyAsync(C.hscal, d, 8, cudaMemcpyDeviceToHost, C.st));
                CK(cudaStreamSynchronize(C.st));
                ratio_min = C.hscal[0];
            }
            if (option == 1) {
                if ((Nvis_store >= 1 && ratio_min > E.cfg.eig_ratio_min) || ivis == 0 || n > 20) {
                    if (record) { E.eig_fine = ratio_min; E.n_eta = n; }
                    trigger = 1;
                    break;
                }
            } else if (interpolate == 0) {
                if (ratio_min > E.cfg.eig_ratio || ivis == 0) { trigger = 1; nn_store = nn; break; }
            } else if (Nvis_store >= 1 || ivis == 0) {
                trigger = 1;
                break;
            }
            int ntemp = Niter - nn + 1;
            double c = 2.0 / (-lb - la + (lb - la) * std::cos((double)(2 * ntemp - 1) * kPi / (double)(2 * Niter)));
            c = 0.99 * c;
            PT_COUNT(), (fused ? k_vis_update_bc<true> : k_vis_update_bc<false>)<<<gg, 128, 0, C.st>>>(S.vis, S.vsm, g, nx,
                                                                                                  nz, c);
            CKL("k_vis_update_bc");
        }
        if (trigger) return 0;
        Nvis_store++;
        nn_store = 1;
        if (option == 1) { Niter = 6; lb = -2.0; la = -1.0; }
        n++;
    }
    return fail(PT_ERR_ITER_CAP, "viscosity smoother exceeded its iteration cap");
}

// restrict_coefficients / restrict: full weighting onto coarse interior nodes
__device__ __forceinline__ double restrict_at(const double* in, Geo gf, int i, int k) {
    int ii = 2 * i, kk = 2 * k;
    double corners = (in[gf.at(ii - 1, kk - 1)] + in[gf.at(ii - 1, kk + 1)] + in[gf.at(ii + 1, kk + 1)] + in[gf.at(ii + 1, kk - 1)]) / 16.0;
    double sides = (in[gf.at(ii - 1, kk)] + in[gf.at(ii, kk - 1)] + in[gf.at(ii + 1, kk)] + in[gf.at(ii, kk + 1)]) / 8.0;
    double centre = in[gf.at(ii, kk)] / 4.0;
    return corners + sides + centre;
}
__global__ void k_restrict(double* out, const double* in, Geo gc, Geo gf, int nxc, int nzc) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
    if (i > nxc - 1) return;
    out[gc.at(i, k)] = restrict_at(in, gf, i, k);
}

// viscosityBCs_initialize (iterative_solver.f90:636-664)
__global__ void k_visbc_init(double* v, const double* vf, Geo g, Geo gf, int nx, int nz, int nxf, int nzf) {
    int W = nx + 7;
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= W * (nz + 7)) return;
    int i = idx % W - 3, k = idx / W - 3;
    bool xin = (i >= 0 && i <= nx), zin = (k >= 0 && k <= nz);
    if (xin && zin && i > 0 && i < nx && k > 0 && k < nz) return;  // interior: restricted values
    int mi = mirror_idx(i, nx), mk = mirror_idx(k, nz);
    // boundary value of the mirrored boundary node, taken from the finer level by injection
    double val;
    if (mk == 0) val = vf[gf.at(2 * mi, 0)];
    else if (mk == nz) val = vf[gf.at(2 * mi, nzf)];
    else if (mi == 0) val = vf[gf.at(0, 2 * mk)];
    else if (mi == nx) val = vf[gf.at(nxf, 2 * mk)];
    else val = v[g.at(mi, mk)];  // ghost of an interior node
    v[g.at(i, k)] = val;
}

static int compute_viscosity(Engine& E, const VisCtx& C, int level) {
    int rc;
    const Geo& g = E.gl[level];
    const VisLevels& V = C.V;
    if (level == 1) {
        dim3 gg(nblk(g.nx + 1, 128), g.nz + 1);
        PT_COUNT(), k_visf<<<gg, 128, 0, C.st>>>(V.visst[1], E.Tvis, E.Cvis, g);
        CKL("k_visf");
        CK(cudaMemcpyAsync(V.vis[1], V.visst[1], g.elems() * 8, cudaMemcpyDeviceToDevice, C.st));
        return smoother_vis(E, C, 1, 0, level_set(V, 1), 1);
    }
    const int lf = level - 1;
    const Geo& gf = E.gl[lf];
    // smooth a work copy of the finer static viscosity (the reference smooths in place and
    // restores the finer level's arrays afterwards)
    VisSet W{C.visw[0], C.visw[1], C.visw[2], C.visw[3], C.visw[4], C.visw[5], C.visw[6], C.visw[7],
             C.visw[8], C.visw[9], C.visw[10]};
    CK(cudaMemcpyAsync(W.vis, V.visst[lf], gf.elems() * 8, cudaMemcpyDeviceToDevice, C.st));
    if ((rc = smoother_vis(E, C, lf, 1, W, 0))) return rc;
    dim3 gr(nblk(g.nx - 1, 128), g.nz - 1);
    PT_COUNT(), k_restrict<<<gr, 128, 0, C.st>>>(V.vis[level], W.vis, g, gf, g.nx, g.nz);
    int tot = (g.nx + 7) * (g.nz + 7);
    PT_COUNT(), k_visbc_init<<<nblk(tot, 128), 128, 0, C.st>>>(V.vis[level], W.vis, g, gf, g.nx, g.nz, gf.nx, gf.nz);
    CKL("restrict_coefficients");
    CK(cudaMemcpyAsync(V.visst[level], V.vis[level], g.elems() * 8, cudaMemcpyDeviceToDevice, C.st));
    return smoother_vis(E, C, level, 0, level_set(V, level), 0);
}

// ------------------------------------------------------------------ RHS and residual norms
__global__ void k_rhs1(double* RHS, const double* Tb, const double* Cb, Geo g, int comp) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
    if (i > cK.nx - 1) return;
    double v = 0.0;
    if (cK.RaT != 0.0) {
        double tr = 0.0;
        for (int j = -2; j <= 2; j++) tr = tr + cK.D1[3 + j] * Tb[g.at(i + j, k)];
        v = cK.RaT * qdiv(tr, cK.dr, cK.inv_dr);  // (the reference's / 1.0 is exact)
    }
    if (comp) {
        double cr = 0.0;
        for (int j = -2; j <= 2; j++) cr = cr + cK.D1[3 + j] * Cb[g.at(i + j, k)];
        v = v - cK.RaC * qdiv(cr, cK.dr, cK.inv_dr);
    }
    RHS[g.at(i, k)] = v;
}

static int compute_RHS(Engine& E, int level) {
    const Geo& g = E.gl[level];
    dim3 gr(nblk(g.nx - 1, 128), g.nz - 1);
    if (level == 1) PT_COUNT(), k_rhs1<<<gr, 128, 0, E.st>>>(E.RHS[1], E.Tbuoy, E.Cbuoy, g, E.cfg.comp);
    else PT_COUNT(), k_restrict<<<gr, 128, 0, E.st>>>(E.RHS[level], E.res[level - 1], g, E.gl[level - 1], g.nx, g.nz);
    CKL("compute_RHS");
    return 0;
}

static int mean_abs(Engine& E, const double* f, int level, double* host_out) {
    const Geo& g = E.gl[level];
    int rc = reduce_sum_abs_interior(E, f, g.nx, g.nz, g.pitch, E.dscal + 8);
    if (rc) return rc;
    CK(cudaMemcpyAsync(E.hscal, E.dscal + 8, 8, cudaMemcpyDeviceToHost, E.st));
    CK(cudaStreamSynchronize(E.st));
    *host_out = E.hscal[0] / (double)(g.nx - 2) / (double)(g.nz - 2);
    return 0;
}

// ------------------------------------------------------------------ RKC1 stage kernel
struct StreamOp {
    const double *vis, *vx, *vz, *vxz, *vxxmzz, *rhs, *dtst;
};

// -(stream operator - RHS) at node (i,k) of S: stream_derivatives (iterative_solver.f90:973-1073)
// and stream_space (890-911) with the reference's operations in the reference's order -- each
// derivative a sum over its full stencil (zero weights included) divided by the spacing power,
// the cross derivatives as 25-point sums, no fused multiply-adds (this file is compiled with
// --fmad=false) -- so that the FP64 path with reference_rounding rounds like the reference.
__device__ __forceinline__ double stream_F(const double* __restrict__ S, Geo g, const LevConst& L,
                                           const StreamOp& op, int i, int k, int ivis) {
    double a = 0.0, b = 0.0, c = 0.0;
    for (int j = -2; j <= 2; j++) a += cK.D2[j + 3] * S[g.at(i + j, k)];
    for (int j = -3; j <= 3; j++) b += cK.D3[j + 3] * S[g.at(i + j, k)];
    for (int j = -3; j <= 3; j++) c += cK.D4[j + 3] * S[g.at(i + j, k)];
    const double Sxx = a / L.dr2, Sxxx = b / L.dr3, Sxxxx = c / L.dr4;
    a = 0.0; b = 0.0; c = 0.0;
    for (int j = -2; j <= 2; j++) a += cK.D2[j + 3] * S[g.at(i, k + j)];
    for (int j = -3; j <= 3; j++) b += cK.D3[j + 3] * S[g.at(i, k + j)];
    for (int j = -3; j <= 3; j++) c += cK.D4[j + 3] * S[g.at(i, k + j)];
    const double Szz = a / L.ds2, Szzz = b / L.ds3, Szzzz = c / L.ds4;
    double xz = 0.0, xxz = 0.0, xzz = 0.0, xxzz = 0.0;
    for (int k2 = -2; k2 <= 2; k2++)
        for (int i2 = -2; i2 <= 2; i2++) {
            const double v = S[g.at(i + i2, k + k2)];
            xz += cK.Drs[i2 + 2][k2 + 2] * v;
            xxz += cK.Drrs[i2 + 2][k2 + 2] * v;
            xzz += cK.Drss[i2 + 2][k2 + 2] * v;
            xxzz += cK.Drrss[i2 + 2][k2 + 2] * v;
        }
    const double Sxz = xz / L.drds, Sxxz = xxz / L.dr2ds, Sxzz = xzz / L.drds2, Sxxzz = xxzz / L.dr2ds2;
    size_t o = g.at(i, k);
    double r;
    double t2 = op.vis[o] * (Sxxxx + Szzzz + 2.0 * Sxxzz);
    if (ivis == 0) r = t2 - op.rhs[o];
    else {
        double t1 = op.vxxmzz[o] * (Sxx - Szz);
        double t4 = 4.0 * op.vxz[o] * Sxz;
        double t5 = 2.0 * op.vx[o] * (Sxxx + Sxzz);
        double t6 = 2.0 * op.vz[o] * (Szzz + Sxxz);
        r = t1 + t2 + t4 + t5 + t6 - op.rhs[o];
    }
    return -r;
}

// writes value v of interior node (i,k) of out and its free-slip ghost images: the mirror
// across a side wall flips the sign, across top/bottom it multiplies by sz (-1 free slip, +1 rigid)
__device__ __forceinline__ void store_with_ghosts(double* out, Geo g, int i, int k, int nx, int nz, double v,
                                                  double sz) {
    int xs[3], zs[3];
    double xf[3], zf[3];
    int nxp = 0, nzp = 0;
    xs[nxp] = i; xf[nxp++] = 1.0;
    if (i <= 3) { xs[nxp] = -i; xf[nxp++] = -1.0; }
    if (i >= nx - 3) { xs[nxp] = 2 * nx - i; xf[nxp++] = -1.0; }
    zs[nzp] = k; zf[nzp++] = 1.0;
    if (k <= 3) { zs[nzp] = -k; zf[nzp++] = sz; }
    if (k >= nz - 3) { zs[nzp] = 2 * nz - k; zf[nzp++] = sz; }
    for (int a = 0; a < nxp; a++)
        for (int b = 0; b < nzp; b++) out[g.at(xs[a], zs[b])] = (xf[a] * zf[b]) * v;
}

// zero the boundary lines and their ghost images (done once per buffer per pass)
__global__ void k_stream_zero_bnd(double* out, Geo g, int nx, int nz) {
    int W = nx + 7;
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= W * (nz + 7)) return;
    int i = idx % W - 3, k = idx / W - 3;
    if (i == 0 || i == nx || k == 0 || k == nz) out[g.at(i, k)] = 0.0;
    else if ((i < 0 || i > nx) && (k == 0 || k == nz)) out[g.at(i, k)] = 0.0;
}

// one RKC1 stage: out = cS0*S0 + mew*S1 + v*S2 + (mewt*c)*dt*F(S1)   (stage 1: S0 + (mewt*c)*dt*F(S0))
__global__ void __launch_bounds__(128) k_rkc_stage(double* __restrict__ out, const double* __restrict__ S1,
                                                   const double* __restrict__ S2, const double* __restrict__ S0,
                                                   StreamOp op, Geo g, int l, double cS0, double mew, double vv,
                                                   double mewtc, int first, int ivis, double sz) {
    const LevConst& L = cL[l];
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
    if (i > L.nx - 1) return;
    double F = stream_F(S1, g, L, op, i, k, ivis);
    size_t o = g.at(i, k);
    double v;
    if (first) v = S1[o] + mewtc * op.dtst[o] * F;
    else v = cS0 * S0[o] + mew * S1[o] + vv * S2[o] + mewtc * op.dtst[o] * F;
    store_with_ghosts(out, g, i, k, L.nx, L.nz, v, sz);
}

// k_rkc_stage with the stream operator's stencil sums formed exactly (pt_exact.cuh); a CTA owns a
// TG::TX x TG::TZ tile of nodes.
template <bool SQUARE, class TG>
__global__ void __launch_bounds__(TG::NT) k_rkc_stage_fx(double* __restrict__ out, const double* __restrict__ S1,
                                                         const double* __restrict__ S2, const double* __restrict__ S0,
                                                         StreamOp op, Geo g, int l, double cS0, double mew, double vv,
                                                         double mewtc, int first, int ivis, double sz, ResFxK K) {
    __shared__ int2 X[TG::HT][TG::W];
    __shared__ int emax_s;
    pdl_begin();
    const LevConst& L = cL[l];
    const int i0 = blockIdx.x * TG::TX + 1, k0 = blockIdx.y * TG::TZ + 1;
    const int emax = load_tile_fx<TG>(X, &emax_s, S1, g, i0, k0, L.nx, L.nz);
#pragma unroll 1
    for (int r = 0; r < TG::RPT; r++) {
        const int lx = threadIdx.x, lz = threadIdx.y + TG::TY * r;
        const int i = i0 + lx, k = k0 + lz;
        if (i > L.nx - 1 || k > L.nz - 1) continue;
        const size_t o = g.at(i, k);
        const double F = op.rhs[o] - tile_apply_A<SQUARE>(X, lx + TG::H, lz + TG::H, emax, op.vis, op.vx, op.vz, op.vxz,
                                                          op.vxxmzz, o, ivis, K);
        double v;
        if (first) v = S1[o] + mewtc * op.dtst[o] * F;
        else v = cS0 * S0[o] + mew * S1[o] + vv * S2[o] + mewtc * op.dtst[o] * F;
        store_with_ghosts(out, g, i, k, L.nx, L.nz, v, sz);
    }
}

// k_residual with exact stencil sums
template <bool SQUARE, class TG>
__global__ void __launch_bounds__(TG::NT) k_residual_fx64(double* __restrict__ res, const double* __restrict__ S,
                                                          StreamOp op, Geo g, int l, int ivis, ResFxK K) {
    __shared__ int2 X[TG::HT][TG::W];
    __shared__ int emax_s;
    pdl_begin();
    const LevConst& L = cL[l];
    const int i0 = blockIdx.x * TG::TX + 1, k0 = blockIdx.y * TG::TZ + 1;
    const int emax = load_tile_fx<TG>(X, &emax_s, S, g, i0, k0, L.nx, L.nz);
#pragma unroll 1
    for (int r = 0; r < TG::RPT; r++) {
        const int lx = threadIdx.x, lz = threadIdx.y + TG::TY * r;
        const int i = i0 + lx, k = k0 + lz;
        if (i > L.nx - 1 || k > L.nz - 1) continue;
        const size_t o = g.at(i, k);
        res[o] = op.rhs[o] - tile_apply_A<SQUARE>(X, lx + TG::H, lz + TG::H, emax, op.vis, op.vx, op.vz, op.vxz,
                                                  op.vxxmzz, o, ivis, K);
    }
}

// residual = -(L S - RHS) on the interior (compute_residual)
__global__ void k_residual(double* __restrict__ res, const double* __restrict__ S, StreamOp op, Geo g, int l, int ivis) {
    const LevConst& L = cL[l];
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
    if (i > L.nx - 1) return;
    res[g.at(i, k)] = stream_F(S, g, L, op, i, k, ivis);
}

// full free-slip ghost/boundary fill of a level array (enforceBCs_stream)
__global__ void k_stream_bcs(double* S, Geo g, int nx, int nz, double sz) {
    int W = nx + 7;
    int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= W * (nz + 7)) return;
    int i = idx % W - 3, k = idx / W - 3;
    bool xin = (i > 0 && i < nx), zin = (k > 0 && k < nz);
    if (xin && zin) return;
    int mi = mirror_idx(i, nx), mk = mirror_idx(k, nz);
    double v;
    if (mi == 0 || mi == nx || mk == 0 || mk == nz) v = 0.0;
    else {
        double s = 1.0;
        if (i < 0 || i > nx) s = -s;
        if (k < 0 || k > nz) s = s * sz;
        v = s * S[g.at(mi, mk)];
    }
    S[g.at(i, k)] = v;
}

int enforce_bcs_stream(Engine& E, int level, double* f) {
    const Geo& g = E.gl[level];
    int tot = (g.nx + 7) * (g.nz + 7);
    PT_COUNT(), k_stream_bcs<<<nblk(tot, 256), 256, 0, E.st>>>(f, g, g.nx, g.nz, E.cfg.Vbc == 0 ? -1.0 : 1.0);
    CKL("k_stream_bcs");
    return 0;
}

static StreamOp stream_op(Engine& E, int l) {
    return StreamOp{E.vis[l], E.vx[l], E.vz[l], E.vxz[l], E.vxxmzz[l], E.RHS[l], E.dtst[l]};
}

// one RKC1 stage / one residual on level l: the exact-sum kernels when the stencils allow them
static int launch_stage(Engine& E, int l, double* out, const double* S1, const double* S2, const double* S0,
                        const StreamOp& op, double cS0, double mew, double vv, double mewtc, int first, double sz) {
    const Geo& g = E.gl[l];
    const int ivis = E.cfg.ivis;
    if (E.res_int) {
        const bool sq = E.resfx[l].square;
        if (use_big_tiles(g.nx, g.nz)) {
            dim3 blk(TileBig::TX, TileBig::TY), grd(nblk(g.nx - 1, TileBig::TX), nblk(g.nz - 1, TileBig::TZ));
            auto kern = sq ? k_rkc_stage_fx<true, TileBig> : k_rkc_stage_fx<false, TileBig>;
            return launch_pdl("k_rkc_stage_fx", kern, grd, blk, 0, E.st, out, S1, S2, S0, op, g, l, cS0, mew, vv, mewtc,
                              first, ivis, sz, E.resfx[l]);
        }
        dim3 blk(TileSmall::TX, TileSmall::TY), grd(nblk(g.nx - 1, TileSmall::TX), nblk(g.nz - 1, TileSmall::TZ));
        auto kern = sq ? k_rkc_stage_fx<true, TileSmall> : k_rkc_stage_fx<false, TileSmall>;
        return launch_pdl("k_rkc_stage_fx", kern, grd, blk, 0, E.st, out, S1, S2, S0, op, g, l, cS0, mew, vv, mewtc, first,
                          ivis, sz, E.resfx[l]);
    }
    dim3 gs(nblk(g.nx - 1, 128), g.nz - 1);
    PT_COUNT(), k_rkc_stage<<<gs, 128, 0, E.st>>>(out, S1, S2, S0, op, g, l, cS0, mew, vv, mewtc, first, ivis, sz);
    return 0;
}
static int launch_residual(Engine& E, int l, double* res, const double* S, const StreamOp& op) {
    const Geo& g = E.gl[l];
    if (E.res_int) {
        const bool sq = E.resfx[l].square;
        if (use_big_tiles(g.nx, g.nz)) {
            dim3 blk(TileBig::TX, TileBig::TY), grd(nblk(g.nx - 1, TileBig::TX), nblk(g.nz - 1, TileBig::TZ));
            auto kern = sq ? k_residual_fx64<true, TileBig> : k_residual_fx64<false, TileBig>;
            return launch_pdl("k_residual_fx64", kern, grd, blk, 0, E.st, res, S, op, g, l, E.cfg.ivis, E.resfx[l]);
        }
        dim3 blk(TileSmall::TX, TileSmall::TY), grd(nblk(g.nx - 1, TileSmall::TX), nblk(g.nz - 1, TileSmall::TZ));
        auto kern = sq ? k_residual_fx64<true, TileSmall> : k_residual_fx64<false, TileSmall>;
        return launch_pdl("k_residual_fx64", kern, grd, blk, 0, E.st, res, S, op, g, l, E.cfg.ivis, E.resfx[l]);
    }
    PT_COUNT(), k_residual<<<dim3(nblk(g.nx - 1, 128), g.nz - 1), 128, 0, E.st>>>(res, S, op, g, l, E.cfg.ivis);
    return 0;
}

// iterate_stream (RKC1 = 1, splitting = 0) + compute_residual.  The last stage writes straight
// into error(:,:,level): a stage reads S0 only at its own node, so the update is safe in place.
// With want_sum the sum of |residual| is left in dscal[8] (no host synchronisation, so the
// sequence can be captured in a CUDA graph).  The boundary lines of the stage buffers are zero
// from allocation and are never written by the stage kernel.
static int iterate_stream(Engine& E, int l, int want_sum) {
    const Geo& g = E.gl[l];
    const int N = E.cfg.nstageS, Niter = E.cfg.Nmulti;
    const double sz = E.cfg.Vbc == 0 ? -1.0 : 1.0;
    StreamOp op = stream_op(E, l);
    double* buf[3] = {E.S0[l], E.S1[l], E.S2[l]};
    for (int n = 1; n <= Niter; n++) {
        int ntemp = Niter - n + 1;
        double temp = (E.cfg.Nmulti > 1) ? (E.cfg.c_2 - E.cfg.c_1) * (double)(ntemp - 1) / (double)(1 - Niter) : 0.0;
        double c = temp + E.cfg.c_2;
        const double* S0 = E.err[l];
        GraphTimer gt(E, 0, (l == 1 && want_sum) ? N : 0);
        int cur = 0;
        const double* none = nullptr;
        if (int rc = launch_stage(E, l, buf[cur], S0, none, none, op, 0, 0, 0, E.K.mewt[1] * c, 1, sz)) return rc;
        const double* Sm1 = buf[cur];
        const double* Sm2 = S0;
        for (int j = 2; j <= N; j++) {
            int nxt = (cur + 1) % 3;
            if (buf[nxt] == Sm2) nxt = (nxt + 1) % 3;
            double* out = (j == N) ? E.err[l] : buf[nxt];
            if (int rc = launch_stage(E, l, out, Sm1, Sm2, S0, op, E.K.cc[j], E.K.mew[j], E.K.vv[j], E.K.mewt[j] * c, 0, sz))
                return rc;
            Sm2 = Sm1;
            Sm1 = out;
            cur = nxt;
        }
        CKL("k_rkc_stage");
    }
    if (int rc = launch_residual(E, l, E.res[l], E.err[l], op)) return rc;
    CKL("k_residual");
    if (want_sum) return reduce_sum_abs_interior(E, E.res[l], g.nx, g.nz, g.pitch, E.dscal + 8);
    return 0;
}

// prolong (iterative_solver.f90:343-396): bilinear coarse correction added to the finer level
__device__ __forceinline__ double prolong_at(const double* C, Geo gc, int i, int k) {
    if (!(i & 1) && !(k & 1)) return C[gc.at(i / 2, k / 2)];
    if (!(i & 1)) return (C[gc.at(i / 2, (k - 1) / 2)] + C[gc.at(i / 2, (k + 1) / 2)]) / 2.0;
    if (!(k & 1)) return (C[gc.at((i - 1) / 2, k / 2)] + C[gc.at((i + 1) / 2, k / 2)]) / 2.0;
    return (C[gc.at((i - 1) / 2, (k - 1) / 2)] + C[gc.at((i + 1) / 2, (k - 1) / 2)] + C[gc.at((i + 1) / 2, (k + 1) / 2)] +
            C[gc.at((i - 1) / 2, (k + 1) / 2)]) / 4.0;
}
__global__ void k_prolong(double* F, const double* C, Geo gf, Geo gc, int nxf, int nzf) {
    int i = blockIdx.x * blockDim.x + threadIdx.x + 1, k = blockIdx.y + 1;
    if (i > nxf - 1) return;
    const size_t o = gf.at(i, k);
    F[o] = F[o] + prolong_at(C, gc, i, k);
}

// ------------------------------------------------------------------ levels in one cluster
// A stretch of the FP64 cycle on levels that fit one cluster (pt_cluster.cuh): the entering restriction
// or prolongation, the RKC1 stages, the residual that the next coarser level restricts; the coarsest
// level by the explicit inverse.  The stencil sums are exact, as in k_rkc_stage_fx.  A stage has three
// parts, each with the split that keeps its chain short (a few warps an SM: latency is the bound, at
// the upper end the FP64 pipe with its two lanes a clock an SM):
//   * the CTA takes the largest exponent of its window and writes the window, images included, as
//     62-bit fixed point X = Xh 2^31 + Xl (each thread keeps its few cells' places for the visit);
//   * warps form the derivative groups, five warps (or, with more tiles than that leaves warps for,
//     two) to a tile of 32 nodes: integer multiply-adds with constant weights, one rounding of the
//     78-bit sum to FP64 by integer operations, as adding its two exact halves would round it, and the
//     product with the node's coefficient; one more warp the rest of the recurrence;
//   * a thread a node adds these up and publishes the value.
// An FP64 instruction keeps a scheduler's pipe busy for some 64 cycles, so the products and the
// recurrence go to the warps that have room beside their integer work.
struct DLevel {
    Geo g;
    double *e, *rhs, *res;
    const double *vis, *vx, *vz, *vxz, *vxxmzz, *dtst;
    ResFxK K;
};
struct DRun {
    DLevel L[PT_MAXLEV];
    cl::Visit v[cl::kMaxVisits];
    int nv, N, ivis, ngc;
    double sz;
    double cc[64], mew[64], vv[64], mewtc[64];
    const double *G, *RowB;
};
constexpr int kDOwn = cl::kThreads / 2, kDGroups = 10;  // nodes of a CTA at most; derivative groups at most
constexpr int kDTiles = kDOwn / 32, kDParts = 5;         // its tiles; warps to a tile at most
constexpr int kDCells = 5;  // window cells of a thread at most: 8 rows of 263, with strips of two rows
static size_t cluster_bytes_d(int ngc) {
    return sizeof(double) * (2 * (size_t)cl::kWindow + (kDGroups + kDParts + 5) * (size_t)kDOwn + (size_t)ngc) +
           sizeof(int2) * (size_t)cl::kWindow;
}

// integer weight of the point (dx, dz) in derivative group g (tile_apply_A's sums; SQUARE: combined)
__host__ __device__ constexpr int id1(int j) { return j == -2 ? 1 : j == -1 ? -8 : j == 1 ? 8 : j == 2 ? -1 : 0; }
__host__ __device__ constexpr int id2(int j) { return j == 0 ? -30 : j == 1 || j == -1 ? 16 : j == 2 || j == -2 ? -1 : 0; }
__host__ __device__ constexpr int id3(int j) {
    return j == -3 ? 1 : j == -2 ? -8 : j == -1 ? 13 : j == 1 ? -13 : j == 2 ? 8 : j == 3 ? -1 : 0;
}
__host__ __device__ constexpr int id4(int j) {
    return j == 0 ? 56 : j == 1 || j == -1 ? -39 : j == 2 || j == -2 ? 12 : -1;
}
template <bool SQUARE>
__host__ __device__ constexpr int group_weight(int g, int dx, int dz) {
    const int x4 = dz == 0 ? id4(dx) : 0, z4 = dx == 0 ? id4(dz) : 0, x2 = dz == 0 ? id2(dx) : 0, z2 = dx == 0 ? id2(dz) : 0;
    const int x3 = dz == 0 ? id3(dx) : 0, z3 = dx == 0 ? id3(dz) : 0;
    const int i11 = id1(dx) * id1(dz), i12 = id1(dx) * id2(dz), i21 = id2(dx) * id1(dz), i22 = id2(dx) * id2(dz);
    if (SQUARE)
        return g == 0 ? 24 * (x4 + z4) + 2 * i22 : g == 1 ? x2 - z2 : g == 2 ? i11 : g == 3 ? 18 * x3 + i12 : 18 * z3 + i21;
    return g == 0 ? x4 : g == 1 ? z4 : g == 2 ? i22 : g == 3 ? x2 : g == 4 ? z2 : g == 5 ? i11 : g == 6 ? x3 : g == 7 ? i12
           : g == 8 ? z3 : i21;
}

// (h 2^31 + l) 2^-s rounded once to FP64 (|h|, |l| < 2^52, result normal or zero); s = 1084 - emax
__device__ __forceinline__ double hl_rounded(long long h, long long l, int emax) {
    long long hi = h + (l >> 31);  // hi 2^31 + lo, 0 <= lo < 2^31
    unsigned lo = (unsigned)l & 0x7FFFFFFFu;
    const bool neg = hi < 0;
    if (neg) {
        hi = lo ? ~hi : -hi;
        lo = (0x80000000u - lo) & 0x7FFFFFFFu;
    }
    if (hi == 0) {
        if (lo == 0) return 0.0;
        hi = (long long)lo;  // as hi 2^31 with the exponent 31 lower
        lo = 0;
        emax -= 31;
    }
    // the 64 leading bits of the sum, and whether any bit below them is set
    const int lz = __clzll(hi);
    unsigned long long A = (unsigned long long)hi << lz;
    bool sticky = false;
    if (lz >= 31) {
        A |= (unsigned long long)lo << (lz - 31);
    } else {
        A |= lo >> (31 - lz);
        sticky = (lo & ((1u << (31 - lz)) - 1u)) != 0;
    }
    unsigned long long q = A >> 11;
    const unsigned rem = (unsigned)A & 0x7FFu;
    if (rem > 0x400u || (rem == 0x400u && (sticky || (q & 1ull)))) q++;
    const long long ex = 1023 + 52 + 42 - lz - (1084 - emax);
    if (ex <= 0) return 0.0;  // below the normal range (S itself near underflow)
    return __longlong_as_double((long long)(((unsigned long long)neg << 63) | (((unsigned long long)(ex - 1) << 52) + q)));
}

// sum of derivative group G at cell x of the fixed-point window, rounded
template <bool SQUARE, int G>
__device__ __forceinline__ double group_sum(const int2* x, int emax) {
    long long h[2] = {0, 0}, l[2] = {0, 0};
    int n = 0;
#pragma unroll
    for (int dz = -3; dz <= 3; dz++)
#pragma unroll
        for (int dx = -3; dx <= 3; dx++) {
            const bool block = dx >= -2 && dx <= 2 && dz >= -2 && dz <= 2;
            const int w = block || dx == 0 || dz == 0 ? group_weight<SQUARE>(G, dx, dz) : 0;
            if (w == 0) continue;
            const int2 v = x[dz * cl::kPitch + dx];
            h[n & 1] += (long long)w * v.x;
            l[n & 1] += (long long)w * v.y;
            n++;
        }
    return hl_rounded(h[0] + h[1], l[0] + l[1], emax);
}
// groups G .. G + N - 1, each times its coefficient (w: kDOwn apart)
template <bool SQUARE, int G, int N>
__device__ __forceinline__ double group_part(const int2* x, int emax, const double* w) {
    double a = w[G * kDOwn] * group_sum<SQUARE, G>(x, emax);
    if constexpr (N > 1) a += group_part<SQUARE, G + 1, N - 1>(x, emax, w);
    return a;
}

template <bool SQUARE>
__global__ void __launch_bounds__(cl::kThreads, 1) k_cycle_cluster_d(const __grid_constant__ DRun P) {
    constexpr int NG = SQUARE ? 5 : 10;
    extern __shared__ __align__(16) double dm[];
    __shared__ uint64_t bars[2];
    __shared__ double cheb[64][4];
    __shared__ int emax_s[cl::kWarps];
    // of each node: the coefficients of its groups, its parts of a stage's sum, then S0, dt rhs, dt
    // and a stage's recurrence without A and its factor of A
    double *const W = dm + 2 * cl::kWindow, *const D = W + kDGroups * kDOwn, *const S0s = D + kDParts * kDOwn;
    double *const drhs = S0s + kDOwn, *const dts = drhs + kDOwn;
    double *const B = dts + kDOwn, *const M = B + kDOwn, *const cb = M + kDOwn;  // cb: the coarsest right-hand side
    int2* const X = reinterpret_cast<int2*>(cb + P.ngc);
    if (threadIdx.x < 64) {
        cheb[threadIdx.x][0] = P.cc[threadIdx.x];
        cheb[threadIdx.x][1] = P.mew[threadIdx.x];
        cheb[threadIdx.x][2] = P.vv[threadIdx.x];
        cheb[threadIdx.x][3] = P.mewtc[threadIdx.x];
    }
    const int c = (int)cl::rank(), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    cl::Exchange ex;
    ex.init(bars);
    for (int n = 0; n < P.nv; n++) {
        const int l = P.v[n].level, fl = P.v[n].flags;
        const DLevel& L = P.L[l];
        const Geo g = L.g;
        if (fl & cl::kCoarse) {  // x = G b, a warp per row over the cluster (k_coarse_apply's sums)
            const Geo gf = P.L[l - 1].g;
            const int N1 = g.nz + 1, nn = (g.nx + 1) * N1, nk = g.nz - 1, ni = (g.nx - 1) * nk;
            for (int q = threadIdx.x; q < nn; q += cl::kThreads) {
                const int ip = q / N1, kp = q - ip * N1;
                cb[q] = ip > 0 && ip < g.nx && kp > 0 && kp < g.nz ? restrict_at(P.L[l - 1].res, gf, ip, kp) * P.RowB[q] : 0.0;
            }
            __syncthreads();
            for (int r = c * cl::kWarps + warp; r < ni; r += cl::kCtas * cl::kWarps) {
                const int ip = r / nk + 1, kp = r - (ip - 1) * nk + 1;
                const double* row = P.G + (size_t)(ip * N1 + kp) * nn;
                double a = 0.0;
                for (int q = lane; q < nn; q += 32) a += row[q] * cb[q];
                for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
                if (lane == 0) L.e[g.at(ip, kp)] = a;  // (its walls stay zero, its images are not read)
            }
            cl::sync();
            continue;
        }
        cl::Strip s;
        s.set(g.nz, c, false);
        const int segs = cl::Strip::segments(g.nx), tiles = s.rows * segs, cols = g.nx + 2 * cl::kReach + 1;
        const float inv_segs = __frcp_rn((float)segs);
        // cell of lane's node in tile t (32 columns of a row); lanes past the row take its last node
        auto tile_cell = [&](int t) {
            const int r = (int)(((float)t + 0.5f) * inv_segs);
            return s.at(min((t - r * segs) * 32 + lane + 1, g.nx - 1), s.k0 + r);
        };
        // the thread's node: its coefficients, right-hand side and place
        const int r = (int)(((float)warp + 0.5f) * inv_segs), i = (warp - r * segs) * 32 + lane + 1, k = s.k0 + r;
        const bool on = warp < tiles && i <= g.nx - 1;
        const size_t o = on ? g.at(i, k) : 0;
        const int m = on ? s.at(i, k) : 0;
        double rhs = 0.0, S0 = 0.0;
        if (on) {
            double w[NG];
            const double* K = L.K.k;
            const double vis = L.vis[o];
            double c1 = 0.0, c2 = 0.0, c3 = 0.0, c4 = 0.0;
            if (P.ivis != 0) {
                c1 = L.vxxmzz[o];
                c2 = L.vxz[o];
                c3 = L.vx[o];
                c4 = L.vz[o];
            }
            const double dt = L.dtst[o];
            if (!(fl & cl::kZero)) S0 = L.e[o];
            if (fl & cl::kRestrict) {
                rhs = restrict_at(P.L[l - 1].res, P.L[l - 1].g, i, k);
                L.rhs[o] = rhs;
            } else {
                rhs = L.rhs[o];
            }
            if (fl & cl::kProlong) S0 = S0 + prolong_at(P.L[l + 1].e, P.L[l + 1].g, i, k);
            if constexpr (SQUARE) {
                w[0] = K[0] * vis; w[1] = K[1] * c1; w[2] = K[2] * c2; w[3] = K[3] * c3; w[4] = K[4] * c4;
            } else {
                w[0] = K[0] * vis; w[1] = K[1] * vis; w[2] = 2.0 * K[2] * vis; w[3] = K[3] * c1; w[4] = -K[4] * c1;
                w[5] = 4.0 * K[5] * c2; w[6] = 2.0 * K[6] * c3; w[7] = 2.0 * K[7] * c3; w[8] = 2.0 * K[8] * c4;
                w[9] = 2.0 * K[9] * c4;
            }
#pragma unroll
            for (int G = 0; G < NG; G++) W[G * kDOwn + threadIdx.x] = w[G];
            S0s[threadIdx.x] = S0;
            drhs[threadIdx.x] = dt * rhs;
            dts[threadIdx.x] = dt;
        }
        // the thread's window cells: where each goes (upper half) and where it comes from, with the sign
        // of the image; -1 where the window stays zero (walls, rows past the images)
        int place[kDCells];
        {
            const int cells = s.rows ? (s.rows + 2 * cl::kReach) * cols : 0;
            const float inv_cols = __frcp_rn((float)cols);
#pragma unroll
            for (int q = 0; q < kDCells; q++) {
                const int cell = (int)threadIdx.x + q * cl::kThreads;
                place[q] = -1;
                if (cell >= cells) continue;
                const int wr = (int)(((float)cell + 0.5f) * inv_cols), wc = cell - wr * cols;
                const int ci = wc - cl::kReach, ck = s.k0 - cl::kReach + wr;
                const int mi = mirror_idx(ci, g.nx), mk = mirror_idx(ck, g.nz);
                if (mi <= 0 || mi >= g.nx || mk <= 0 || mk >= g.nz) continue;
                const int neg = (mi != ci) != (mk != ck && P.sz < 0.0);
                place[q] = (wr * cl::kPitch + wc) << 16 | s.at(mi, mk) << 1 | neg;
            }
        }
        for (int q = threadIdx.x; q < (s.R + 2 * cl::kReach) * cl::kPitch; q += cl::kThreads) X[q] = make_int2(0, 0);
        ex.bytes = (uint32_t)(s.rows_received(g.nz) * (g.nx - 1)) * (uint32_t)sizeof(double);
        cl::Outlet<double> out;
        out.set(s, dm, bars, m, on ? s.readers_up(r) : 0, on ? s.readers_down(r) : 0);
        cl::sync();  // every CTA has left its windows of the last visit (and, the first time, its mbarriers are ready)
        auto publish = [&](int q, double v) {
            if (on) {
                dm[q * cl::kWindow + m] = v;
                if (out.up | out.down) out.put_remote(q, v);
            }
            ex.arrive(q);
        };
        // the parts of A of window q at every node of the strip, into D
        const bool fine = tiles * kDParts <= cl::kWarps;
        // the warp's part (part major: the long ones go to different schedulers), its tile's nodes
        const int part = warp < tiles ? 0 : fine ? warp / max(tiles, 1) : 1, part_tile = warp - part * tiles;
        const bool has_part = tiles > 0 && part_tile < tiles && part < (fine ? kDParts : 2);
        const int part_cell = has_part ? tile_cell(part_tile) : 0, part_node = has_part ? part_tile * 32 + lane : 0;
        const int ncell = (s.rows ? (s.rows + 2 * cl::kReach) * cols : 0) > cl::kThreads ? kDCells : 1;
        auto groups = [&](int q) {
            unsigned long long b[kDCells];
            int em = 0;
#pragma unroll
            for (int j = 0; j < kDCells; j++) {
                if (j >= ncell) break;
                b[j] = 0;
                if (place[j] >= 0)
                    b[j] = (unsigned long long)__double_as_longlong(dm[q * cl::kWindow + (place[j] >> 1 & 0x7FFF)]);
                em = max(em, (int)(b[j] >> 52) & 0x7FF);
            }
            em = __reduce_max_sync(0xffffffffu, em);
            if (lane == 0) emax_s[warp] = em;
            __syncthreads();
            const int emax = __reduce_max_sync(0xffffffffu, emax_s[lane & (cl::kWarps - 1)]);
#pragma unroll
            for (int j = 0; j < kDCells; j++) {
                if (j >= ncell) break;
                if (place[j] >= 0) {
                    const long long f = fixed_point(b[j], emax), v = place[j] & 1 ? -f : f, h = v >> 31;  // floor
                    X[place[j] >> 16] = make_int2((int)h, (int)(v - (h << 31)));
                }
            }
            __syncthreads();
            if (has_part) {
                const int2* x = X + part_cell;
                const double* w = W + part_node;
                double d;
                if (fine) {
                    switch (part) {
                        case 0: d = group_part<SQUARE, SQUARE ? 0 : 0, SQUARE ? 1 : 2>(x, emax, w); break;
                        case 1: d = group_part<SQUARE, SQUARE ? 1 : 2, SQUARE ? 1 : 2>(x, emax, w); break;
                        case 2: d = group_part<SQUARE, SQUARE ? 2 : 4, SQUARE ? 1 : 2>(x, emax, w); break;
                        case 3: d = group_part<SQUARE, SQUARE ? 3 : 6, SQUARE ? 1 : 2>(x, emax, w); break;
                        default: d = group_part<SQUARE, SQUARE ? 4 : 8, SQUARE ? 1 : 2>(x, emax, w);
                    }
                } else if (part == 0) {
                    d = group_part<SQUARE, 0, SQUARE ? 2 : 5>(x, emax, w);
                } else {
                    d = group_part<SQUARE, SQUARE ? 2 : 5, SQUARE ? 3 : 5>(x, emax, w);
                }
                D[part * kDOwn + part_node] = emax == 0x7FF ? __longlong_as_double(0x7FF8000000000000ll) : d;
            }
        };
        auto sum = [&]() {  // A at the thread's node
            const double* d = D + threadIdx.x;
            return fine ? ((d[0] + d[kDOwn]) + (d[2 * kDOwn] + d[3 * kDOwn])) + d[4 * kDOwn] : d[0] + d[kDOwn];
        };
        // what a stage adds to the sum, by the last warps, whose parts are the short ones or none
        const int spare = cl::kWarps - 1 - warp, spare_cell = spare < tiles ? tile_cell(spare) : 0;
        publish(0, S0);
        int cur = 0;
        for (int j = 1; j <= P.N; j++) {
            const bool last = j == P.N;
            groups(cur);
            if (spare < tiles) {  // cc S0 + mew S_{j-1} + vv S_{j-2} + mewt c dt rhs (stage 1: S0 + ..)
                const int q = spare * 32 + lane, cell = spare_cell;
                double base = dm[cur * cl::kWindow + cell];
                if (j > 1) base = fma(cheb[j][1], base, fma(cheb[j][2], dm[(cur ^ 1) * cl::kWindow + cell], cheb[j][0] * S0s[q]));
                B[q] = fma(cheb[j][3], drhs[q], base);
                M[q] = -cheb[j][3] * dts[q];
            }
            __syncthreads();
            double v = 0.0;
            if (on) {
                v = fma(M[threadIdx.x], sum(), B[threadIdx.x]);
                if (last) {
                    if (!ex.ok) v = __longlong_as_double(0x7FF8000000000000ll);  // a wait ran out: NaN, reported by the host
                    L.e[o] = v;
                }
            }
            if (!last || (fl & cl::kResidual)) {
                cur ^= 1;
                publish(cur, v);
            }
        }
        if (fl & cl::kResidual) {
            groups(cur);
            __syncthreads();
            if (on) L.res[o] = rhs - sum();
        }
        cl::sync();  // the correction and the residual are in global memory
    }
}

static int prolong(Engine& E, int lc) {
    const int lf = lc - 1;
    const Geo &gf = E.gl[lf], &gc = E.gl[lc];
    dim3 gp(nblk(gf.nx - 1, 128), gf.nz - 1);
    PT_COUNT(), k_prolong<<<gp, 128, 0, E.st>>>(E.err[lf], E.err[lc], gf, gc, gf.nx, gf.nz);
    CKL("k_prolong");
    return enforce_bcs_stream(E, lf, E.err[lf]);
}

// ------------------------------------------------------------------ coarsest level
// Compute_Matrix_coarse (analysis=0) rows in LAPACK band storage, one thread per row
__global__ void k_coarse_matrix(double* M, Geo g, int l, int kl, int ku, int n, double* RowB, int Vbc, int ivis,
                                const double* vis, const double* vx, const double* vz, const double* vxz,
                                const double* vxxmzz, int* err) {
    int p = blockIdx.x * blockDim.x + threadIdx.x + 1;
    if (p > n) return;
    const LevConst& L = cL[l];
    const int nxc = L.nx, nzc = L.nz, N = nzc + 1, ldab = 2 * kl + ku + 1, kk1 = kl + ku + 1;
    const int reach[7] = {0, 2, 2, 3, 2, 2, 0};
    int ip = (p - 1) / N, kp = (p - 1) % N;
#define MB(row, col) M[(size_t)((row) - 1) + (size_t)((col) - 1) * (size_t)ldab]
    for (int q = (p - kl > 1 ? p - kl : 1); q <= (p + ku < n ? p + ku : n); q++) MB(kk1 + p - q, q) = 0.0;
    if (ip > 0 && ip < nxc && kp > 0 && kp < nzc) {
        size_t o = g.at(ip, kp);
        double a1 = vxxmzz[o], a2 = vis[o], a4 = vxz[o], a5 = vx[o], a6 = vz[o];
        for (int pass = 0; pass < 2; pass++)
            for (int j = -3; j <= 3; j++) {
                int iq = j + ip;
                for (int kq = kp - reach[j + 3]; kq <= kp + reach[j + 3]; kq++) {
                    bool inside = (iq >= 0 && iq <= nxc && kq >= 0 && kq <= nzc);
                    if ((pass == 0) != inside) continue;
                    int di = iq - ip + 3, dk = kq - kp + 3;
                    double v = (ivis == 0) ? a2 * cK.SM2[di][dk]
                                           : a1 * cK.SM1[di][dk] + a2 * cK.SM2[di][dk] + a4 * cK.SM4[di][dk] +
                                                 a5 * cK.SM5[di][dk] + a6 * cK.SM6[di][dk];
                    if (pass == 0) {
                        int q = N * iq + kq + 1;
                        MB(kk1 + p - q, q) = v;
                    } else {
                        int iiq = iq, kkq = kq, sv = 1;
                        if (iq < 0) { iiq = -iq; sv = -sv; }
                        else if (iq > nxc) { iiq = 2 * nxc - iq; sv = -sv; }
                        if (kq < 0) { kkq = -kq; if (Vbc == 0) sv = -sv; }
                        else if (kq > nzc) { kkq = 2 * nzc - kq; if (Vbc == 0) sv = -sv; }
                        int q = N * iiq + kkq + 1;
                        MB(kk1 + p - q, q) = MB(kk1 + p - q, q) + (sv == -1 ? -v : v);
                    }
                }
            }
    } else {
        MB(kk1, p) = 1.0;
    }
    // row equilibration (DGBEQU row factors) and scaling
    double rmax = 0.0;
    for (int q = (p - kl > 1 ? p - kl : 1); q <= (p + ku < n ? p + ku : n); q++) rmax = fmax(rmax, fabs(MB(kk1 + p - q, q)));
    if (rmax == 0.0) { atomicOr(err, 2); rmax = 1.0; }
    const double smlnum = 2.2250738585072014e-308;
    double rf = 1.0 / fmin(fmax(rmax, smlnum), 1.0 / smlnum);
    RowB[p - 1] = rf;
    for (int q = (p - kl > 1 ? p - kl : 1); q <= (p + ku < n ? p + ku : n); q++) MB(kk1 + p - q, q) = rf * MB(kk1 + p - q, q);
#undef MB
}

// DGBTRS (forward substitution with the row interchanges and L, back substitution with U) on one
// right-hand side.  The substitutions are sequential over the n columns, so one warp carries
// them, its lanes splitting each column's band update; the band columns (and pivots) a chunk of
// steps needs are staged in shared memory by the whole CTA beforehand, so each step works from
// shared memory instead of waiting on a global load.  Same operations in the same order as the
// column-by-column DGBTRS, zero entries divided and propagated too (the optimized-BLAS behaviour
// of the shipped run, which only decides the sign of exact zeros).
constexpr int kBsChunk = 32, kBsThreads = 128;
__host__ __device__ constexpr size_t band_solve_smem(int n, int kl, int ku) {
    return sizeof(double) * ((size_t)n + (size_t)kBsChunk * (kl + ku + 1)) + sizeof(int) * kBsChunk;
}
__global__ void __launch_bounds__(kBsThreads) k_band_solve(const double* ab, const int* ipiv, double* bg, int n, int kl,
                                                         int ku) {
    extern __shared__ double b[];
    const int ldab = 2 * kl + ku + 1, kd = ku + kl + 1, kp1 = kl + ku + 1, k = kl + ku;
    double* cb = b + n;
    int* cp = reinterpret_cast<int*>(cb + (size_t)kBsChunk * kp1);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    for (int q = tid; q < n; q += kBsThreads) b[q] = bg[q];
#define AB(r, c) ab[(size_t)((r) - 1) + (size_t)((c) - 1) * (size_t)ldab]
    // forward: columns 1..n-1, rows kd+1..kd+kl of each (the multipliers of L)
    for (int c0 = 1; c0 <= n - 1; c0 += kBsChunk) {
        const int cn = min(kBsChunk, n - c0);
        __syncthreads();
        for (int q = tid; q < cn * kl; q += kBsThreads) cb[q] = AB(kd + 1 + q % kl, c0 + q / kl);
        for (int q = tid; q < cn; q += kBsThreads) cp[q] = ipiv[c0 + q - 1];
        __syncthreads();
        if (warp == 0) {
            for (int jj = 0; jj < cn; jj++) {
                const int j = c0 + jj;
                const int lm = kl < n - j ? kl : n - j;
                const int l = cp[jj];
                if (l != j && lane == 0) { double t = b[l - 1]; b[l - 1] = b[j - 1]; b[j - 1] = t; }
                __syncwarp();
                const double temp = -1.0 * b[j - 1];
                for (int i = 1 + lane; i <= lm; i += 32) b[j + i - 1] = b[j + i - 1] + cb[jj * kl + i - 1] * temp;
                __syncwarp();
            }
        }
    }
    // back substitution: columns n..1, rows 1..kp1 of each (U, diagonal in row kp1)
    for (int c1 = n; c1 >= 1; c1 -= kBsChunk) {
        const int cn = min(kBsChunk, c1);
        __syncthreads();
        for (int q = tid; q < cn * kp1; q += kBsThreads) cb[q] = AB(1 + q % kp1, c1 - q / kp1);
        __syncthreads();
        if (warp == 0) {
            for (int jj = 0; jj < cn; jj++) {
                const int j = c1 - jj;
                const double* col = cb + (size_t)jj * kp1;  // col[r - 1] = AB(r, j)
                const double x = b[j - 1] / col[kp1 - 1];
                __syncwarp();
                if (lane == 0) b[j - 1] = x;
                const int l = kp1 - j, i0 = 1 > j - k ? 1 : j - k;
                for (int i = j - 1 - lane; i >= i0; i -= 32) b[i - 1] = b[i - 1] - x * col[l + i - 1];
                __syncwarp();
            }
        }
    }
#undef AB
    __syncthreads();
    for (int q = tid; q < n; q += kBsThreads) bg[q] = b[q];
}

// coarse solve through the explicit inverse: b = RowB * RHS on interior nodes (0 on the
// boundary), x = G b (one warp per row, lanes stride the row, fixed-order shuffle reduction),
// scattered into the level array.
template <typename R>
__global__ void __launch_bounds__(256) k_coarse_apply(R* Eout, const R* RHS, const double* G, const double* RowB, Geo g,
                                                      int nxc, int nzc) {
    extern __shared__ double bsh[];
    const int N = nzc + 1, n = (nxc + 1) * N;
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
        int ip = q / N, kp = q % N;
        bsh[q] = (ip > 0 && ip < nxc && kp > 0 && kp < nzc) ? (double)RHS[g.at(ip, kp)] * RowB[q] : 0.0;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.x * (blockDim.x >> 5) + warp;
    if (p >= n) return;
    const double* row = G + (size_t)p * n;
    double a = 0.0;
    for (int q = lane; q < n; q += 32) a += row[q] * bsh[q];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) Eout[g.at(p / N, p % N)] = (R)a;
}

// The mixed-precision V-cycle's coarse solve: x = G b with the FP64 inverse and FP64 sums (the
// coarsest level stays FP64), from the FP32 restricted residual, into the FP32 correction with
// its boundary values.  A GEMV of n^2 FMAs (n = 561 at 1024x512) spread over n warps costs a few
// microseconds on the FP64 pipe.
__global__ void __launch_bounds__(256) k_coarse_apply_mixed(float* Eout, const float* RHS, const double* G,
                                                            const double* RowB, Geo g, int nxc, int nzc, float sz) {
    extern __shared__ double bsm[];
    const int N = nzc + 1, n = (nxc + 1) * N;
    for (int q = threadIdx.x; q < n; q += blockDim.x) {
        int ip = q / N, kp = q % N;
        bsm[q] = (ip > 0 && ip < nxc && kp > 0 && kp < nzc) ? (double)RHS[g.at(ip, kp)] * RowB[q] : 0.0;
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int p = blockIdx.x * (blockDim.x >> 5) + warp;
    if (p >= n) return;
    const double* row = G + (size_t)p * n;
    double a = 0.0;
    for (int q = lane; q < n; q += 32) a = fma(row[q], bsm[q], a);
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane != 0) return;
    // the correction with its boundary values: wall nodes zero, interior nodes with their free-slip
    // images (antisymmetric across the side walls, sign sz across top and bottom)
    const int ip = p / N, kp = p % N;
    if (ip == 0 || ip == nxc || kp == 0 || kp == nzc) {
        Eout[g.at(ip, kp)] = 0.0f;
        return;
    }
    const float v = (float)a;
    int xs[3], zs[3];
    float xf[3], zf[3];
    int nxp = 0, nzp = 0;
    xs[nxp] = ip; xf[nxp++] = 1.0f;
    if (ip <= 3) { xs[nxp] = -ip; xf[nxp++] = -1.0f; }
    if (ip >= nxc - 3) { xs[nxp] = 2 * nxc - ip; xf[nxp++] = -1.0f; }
    zs[nzp] = kp; zf[nzp++] = 1.0f;
    if (kp <= 3) { zs[nzp] = -kp; zf[nzp++] = sz; }
    if (kp >= nzc - 3) { zs[nzp] = 2 * nzc - kp; zf[nzp++] = sz; }
    for (int u = 0; u < nxp; u++)
        for (int w = 0; w < nzp; w++) Eout[g.at(xs[u], zs[w])] = (xf[u] * zf[w]) * v;
}

__global__ void k_coarse_rhs(double* B, const double* RHS, const double* RowB, Geo g, int nxc, int nzc) {
    int p = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int N = nzc + 1, n = (nxc + 1) * N;
    if (p > n) return;
    int ip = (p - 1) / N, kp = (p - 1) % N;
    B[p - 1] = (ip > 0 && ip < nxc && kp > 0 && kp < nzc) ? RHS[g.at(ip, kp)] * RowB[p - 1] : 0.0;
}
__global__ void k_coarse_scatter(double* E, const double* B, Geo g, int nxc, int nzc) {
    int p = blockIdx.x * blockDim.x + threadIdx.x + 1;
    int N = nzc + 1, n = (nxc + 1) * N;
    if (p > n) return;
    E[g.at((p - 1) / N, (p - 1) % N)] = B[p - 1];
}

// the panel LU for the direct solve's band (pt_direct.cu)
bool band_lu_fits(int kl) { return bandlu::row_threads(kl) + 32 <= 512; }
size_t band_lu_bytes(int n, int kl) { return bandlu::work_bytes(n, kl); }
int band_lu(double* ab, int* ipiv, int n, int kl, int ku, void* work, int* err, cudaStream_t st) {
    return bandlu::factor(ab, ipiv, n, kl, ku, bandlu::work_of(work, n, kl), err, st);
}

static int coarse_factor(Engine& E) {
    PhaseTimer tf(E, PH_FACTOR);
    const int L = E.grids, n = E.ngc;
    CK(cudaMemsetAsync(E.derr, 0, sizeof(int), E.st));
    PT_COUNT(), k_coarse_matrix<<<nblk(n, 128), 128, 0, E.st>>>(E.Mc, E.gl[L], L, E.kl, E.ku, n, E.RowB, E.cfg.Vbc,
                                                    E.cfg.ivis, E.vis[L], E.vx[L], E.vz[L], E.vxz[L], E.vxxmzz[L], E.derr);
    if (int rc = bandlu::factor(E.Mc, E.ipiv, n, E.kl, E.ku, bandlu::work_of(E.luw, n, E.kl), E.derr, E.st)) return rc;
    int h = 0;
    CK(cudaMemcpyAsync(&h, E.derr, sizeof(int), cudaMemcpyDeviceToHost, E.st));
    CK(cudaStreamSynchronize(E.st));
    if (h) return fail(PT_ERR_SINGULAR_COARSE, "coarse banded LU: zero row or pivot");
    if (E.Ginv) {
        if (int rc = bandlu::inverse(E.Mc, E.Ginv, n, E.kl, E.ku, bandlu::work_of(E.luw, n, E.kl), E.st)) return rc;
    }
    return 0;
}

// Mixed precision: build the coarse matrix, its LU and inverse for the viscosity just computed
// on st into the second buffer set on st2, overlapped with the solves that follow on st (the
// LU's panels run on one SM, the columns they reach on an SM each for a few us; the inverse on
// E.side_clusters clusters).  coarse_resolve copies the result into the live buffers.
static int coarse_factor_async(Engine& E, const VisLevels& V) {
    const int L = E.grids, n = E.ngc;
    CK(cudaMemsetAsync(E.derr2, 0, sizeof(int), E.st2));
    PT_COUNT(), k_coarse_matrix<<<nblk(n, 128), 128, 0, E.st2>>>(E.Mc2, E.gl[L], L, E.kl, E.ku, n, E.RowB2, E.cfg.Vbc,
                                                     E.cfg.ivis, V.vis[L], V.vx[L], V.vz[L], V.vxz[L], V.vxxmzz[L],
                                                     E.derr2);
    if (int rc = bandlu::factor(E.Mc2, E.ipiv2, n, E.kl, E.ku, bandlu::work_of(E.luw2, n, E.kl), E.derr2, E.st2)) return rc;
    if (int rc = bandlu::inverse(E.Mc2, E.Ginv2, n, E.kl, E.ku, bandlu::work_of(E.luw2, n, E.kl), E.st2,
                                 E.side_clusters))
        return rc;
    CK(cudaMemcpyAsync(E.hflag2, E.derr2, sizeof(int), cudaMemcpyDeviceToHost, E.st2));
    E.fact_pending = true;
    return 0;
}

// The worker thread of a new time level (mixed precision): the viscosity pipeline of levels
// 2..grids into the side set vl2 (from the snapshot of level 1's static viscosity in
// vl2.visst[1]) and the coarse factorisation from it, all on st2; ev_fact marks the end.  Reads
// only its own arrays and the engine's constant configuration; its status goes to job_rc.
static void coarse_levels_worker(Engine* Ep) {
    Engine& E = *Ep;
    int rc = 0;
    if (cudaSetDevice(E.device) != cudaSuccess || cudaStreamWaitEvent(E.st2, E.ev_in, 0) != cudaSuccess)
        rc = fail(PT_ERR_CUDA, "coarse-level worker: device or event");
    const VisCtx C = side_ctx(E);
    for (int level = 2; level <= E.grids && !rc; level++) rc = compute_viscosity(E, C, level);
    if (!rc && E.cfg.ivis > 0) rc = coarse_factor_async(E, E.vl2);
    if (!rc && cudaEventRecord(E.ev_fact, E.st2) != cudaSuccess) rc = fail(PT_ERR_CUDA, "coarse-level worker: event");
    E.job_rc = rc;
    if (rc) E.job_msg = g_err;
    E.job_done = true;
}

// Joins the worker and moves its levels into the cycle's arrays (after st2's work, in stream
// order); the factorisation follows in coarse_resolve.  Unless `wait`, only a worker whose work
// has completed on the device is joined: the solves of this time level keep the previous coarse
// levels until then (a preconditioner, O(dt) older), so a solve waits for no worker; it shares the
// SMs with the worker's kernels.
static int coarse_join(Engine& E, bool wait) {
    if (!E.job_active) return 0;
    if (!wait && !(E.job_done.load() && cudaEventQuery(E.ev_fact) == cudaSuccess)) {
        cudaGetLastError();  // a not-ready query is not an error
        return 0;
    }
    E.coarse_job.join();
    E.job_active = false;
    if (E.job_rc) return fail(E.job_rc, E.job_msg);
    CK(cudaStreamWaitEvent(E.st, E.ev_fact, 0));
    const VisLevels P = primary_levels(E);
    double* const* dst[kVisArrays] = {P.vis, P.visst, P.vx, P.vz, P.vxx, P.vzz, P.vxz, P.vxxpzz, P.vxxmzz, P.vsm, P.ratio, P.dtst};
    double* const* src[kVisArrays] = {E.vl2.vis, E.vl2.visst, E.vl2.vx, E.vl2.vz, E.vl2.vxx, E.vl2.vzz, E.vl2.vxz,
                                      E.vl2.vxxpzz, E.vl2.vxxmzz, E.vl2.vsm, E.vl2.ratio, E.vl2.dtst};
    for (int l = 2; l <= E.grids; l++)
        for (int a = 0; a < kVisArrays; a++)
            CK(cudaMemcpyAsync(dst[a][l], src[a][l], E.gl[l].elems() * 8, cudaMemcpyDeviceToDevice, E.st));
    E.coarse_fresh = true;
    return 0;
}

int coarse_resolve(Engine& E) {
    if (!E.fact_pending) return 0;
    E.fact_pending = false;
    CK(cudaEventSynchronize(E.ev_fact));
    if (*E.hflag2) return fail(PT_ERR_SINGULAR_COARSE, "coarse banded LU: zero row or pivot");
    const int n = E.ngc, ldab = 2 * E.kl + E.ku + 1;
    CK(cudaMemcpyAsync(E.Mc, E.Mc2, sizeof(double) * (size_t)ldab * n, cudaMemcpyDeviceToDevice, E.st));
    CK(cudaMemcpyAsync(E.RowB, E.RowB2, sizeof(double) * (size_t)n, cudaMemcpyDeviceToDevice, E.st));
    CK(cudaMemcpyAsync(E.ipiv, E.ipiv2, sizeof(int) * (size_t)n, cudaMemcpyDeviceToDevice, E.st));
    CK(cudaMemcpyAsync(E.Ginv, E.Ginv2, sizeof(double) * (size_t)n * n, cudaMemcpyDeviceToDevice, E.st));
    return 0;
}

// x = G b into err[L] (FP64) or ferr[L] (FP32); needs E.Ginv
int coarse_apply(Engine& E, double* out64, float* out32, const double* rhs64, const float* rhs32) {
    const int L = E.grids, n = E.ngc;
    const Geo& g = E.gl[L];
    const unsigned blocks = nblk(n, 8);
    const size_t smem = sizeof(double) * (size_t)n;
    if (out64) PT_COUNT(), k_coarse_apply<double><<<blocks, 256, smem, E.st>>>(out64, rhs64, E.Ginv, E.RowB, g, g.nx, g.nz);
    else PT_COUNT(), k_coarse_apply_mixed<<<blocks, 256, smem, E.st>>>(out32, rhs32, E.Ginv, E.RowB, g, g.nx, g.nz,
                                                                       E.cfg.Vbc == 0 ? -1.f : 1.f);
    CKL("k_coarse_apply");
    return 0;
}

static int coarse_solve(Engine& E) {
    const int L = E.grids, n = E.ngc;
    const Geo& g = E.gl[L];
    if (E.Ginv) {
        if (int rc = coarse_apply(E, E.err[L], nullptr, E.RHS[L], nullptr)) return rc;
        return enforce_bcs_stream(E, L, E.err[L]);
    }
    PT_COUNT(), k_coarse_rhs<<<nblk(n, 128), 128, 0, E.st>>>(E.Bc, E.RHS[L], E.RowB, g, g.nx, g.nz);
    PT_COUNT(), k_band_solve<<<1, kBsThreads, band_solve_smem(n, E.kl, E.ku), E.st>>>(E.Mc, E.ipiv, E.Bc, n, E.kl, E.ku);
    PT_COUNT(), k_coarse_scatter<<<nblk(n, 128), 128, 0, E.st>>>(E.err[L], E.Bc, g, g.nx, g.nz);
    CKL("coarse solve");
    return enforce_bcs_stream(E, L, E.err[L]);
}

// helpers shared with the mixed-precision solver (pt_mixed.cu)
int coarse_band_solve(Engine& E) {
    const int n = E.ngc;
    PT_COUNT(), k_band_solve<<<1, kBsThreads, band_solve_smem(n, E.kl, E.ku), E.st>>>(E.Mc, E.ipiv, E.Bc, n, E.kl, E.ku);
    CKL("k_band_solve");
    return 0;
}

int residual_level1_nosum(Engine& E) {
    if (int rc = launch_residual(E, 1, E.res[1], E.err[1], stream_op(E, 1))) return rc;
    CKL("k_residual");
    return 0;
}

int residual_level1(Engine& E) {
    const Geo& g = E.gl[1];
    if (int rc = launch_residual(E, 1, E.res[1], E.err[1], stream_op(E, 1))) return rc;
    CKL("k_residual");
    return reduce_sum_abs_interior(E, E.res[1], g.nx, g.nz, g.pitch, E.dscal + 8);
}

// ------------------------------------------------------------------ driver
int mg_setup_solve(Engine& E) {
    int rc;
    // coarse levels and factorisation built by the worker of this time level, once they are done
    // (at a new time level: always, before the next worker starts)
    const bool new_level = !(E.coarse_ready && E.coarse_time == E.time);
    if ((rc = coarse_join(E, new_level))) return rc;
    if (!E.job_active && (rc = coarse_resolve(E))) return rc;
    CK(cudaMemcpyAsync(E.err[1], E.SF, E.g1.elems() * 8, cudaMemcpyDeviceToDevice, E.st));
    if ((rc = compute_RHS(E, 1))) return rc;
    if ((rc = mean_abs(E, E.RHS[1], 1, &E.res_ref[1]))) return rc;
    // The mixed-precision cycle uses levels 2..grids only as a preconditioner inside FP64 defect
    // correction on level 1: their viscosity pipeline and the coarse factorisation are refreshed
    // once per time level (the top-of-step solve) and reused by the RK-stage solves of the step,
    // whose viscosity differs by O(dt).  Level 1, which defines the residual, is rebuilt every
    // solve.  The FP64 cycle rebuilds every level every solve, as the reference does.
    const bool mixed = E.cfg.precision == PT_PREC_MIXED;
    const bool reuse = mixed && E.coarse_ready && E.coarse_time == E.time;
    // a new time level with coarse levels in place (mixed precision): build the new ones on the
    // worker thread, off the critical path; this solve keeps the previous time level's (a
    // preconditioner, O(dt) older)
    const bool async = mixed && E.coarse_ready && !reuse && E.Ginv2 && E.vl2.vis[2];
    E.levels_reused = reuse || async;
    const VisCtx C = primary_ctx(E);
    for (int level = 1; level <= (E.levels_reused ? 1 : E.grids); level++)
        if ((rc = compute_viscosity(E, C, level))) return rc;
    if (async) {
        CK(cudaMemcpyAsync(E.vl2.visst[1], E.visst[1], E.g1.elems() * 8, cudaMemcpyDeviceToDevice, E.st));
        CK(cudaEventRecord(E.ev_in, E.st));
        E.job_rc = 0;
        E.job_done = false;
        E.coarse_job = std::thread(coarse_levels_worker, &E);
        E.job_active = true;
        E.coarse_time = E.time;
    } else if (!reuse && (E.time == 0.0 || E.cfg.ivis > 0)) {
        if ((rc = coarse_factor(E))) return rc;
        E.coarse_ready = true;
        E.coarse_time = E.time;
    }
    return 0;
}

// levels ctop.. run in one cluster, where their nodes fit its arrays and the coarsest solve is a small
// product with the explicit inverse (us a cycle in the cluster and with a kernel per stage: 256x64, n = 297 1003,
// 1893; 256x128, n = 561 1377, 1926; at n = 1089 682 and 790, which the limit of 700 leaves out)
static int cluster_setup_d(Engine& E) {
    E.ctop = E.grids + 1;
    if (E.cfg.precision != PT_PREC_FP64 || E.cfg.Nmulti != 1 || !E.res_int || !E.Ginv || E.ngc > 700) return 0;
    const size_t bytes = cluster_bytes_d(E.ngc);
    for (auto k : {k_cycle_cluster_d<true>, k_cycle_cluster_d<false>}) {
        if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) ||
            cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))
            return fail(PT_ERR_CUDA, "cluster kernel attributes");
        cudaLaunchConfig_t cfg = {};
        cudaLaunchAttribute at[1];
        cl::cluster_launch(cfg, at, bytes, E.st);
        int fit = 0;
        if (cudaOccupancyMaxActiveClusters(&fit, k, &cfg) != cudaSuccess || fit < 1) {
            (void)cudaGetLastError();  // no room for a cluster of this size: the per-stage kernels run
            return 0;
        }
    }
    auto fits = [&](int l) {
        const Geo& g = E.gl[l];
        const int R = cl::Strip::rows_per_cta(g.nz);
        const int cols = g.nx + 2 * cl::kReach + 1;
        return R * cl::Strip::segments(g.nx) <= kDTiles && cols <= cl::kPitch &&
               (R + 2 * cl::kReach) * cols <= kDCells * cl::kThreads;
    };
    E.ctop = E.grids;
    while (E.ctop > 2 && fits(E.ctop - 1)) E.ctop--;
    if (E.ctop == E.grids) E.ctop = E.grids + 1;  // nothing but the coarsest level
    return 0;
}

// the entries p.. of the schedule on levels ctop.. as one launch; *last receives the last of them
static int cluster_run_d(Engine& E, const int* multi, int nsteps, int p, int* last) {
    DRun R{};
    for (; p <= nsteps && multi[p] >= E.ctop; p++) {
        const int l = multi[p];
        cl::Visit& v = R.v[R.nv++];
        v.level = (signed char)l;
        if (l == E.grids) {
            v.flags = cl::kCoarse;
        } else {
            if (multi[p - 1] < l) {
                v.flags |= cl::kRestrict;
                if (E.cfg.mg_scheme == PT_MG_CORRECTION) v.flags |= cl::kZero;
            } else {
                v.flags |= cl::kProlong;
            }
            if (multi[p + 1] > l) v.flags |= cl::kResidual;
        }
        *last = p;
    }
    for (int l = 1; l <= E.grids; l++) {
        const StreamOp op = stream_op(E, l);
        R.L[l] = DLevel{E.gl[l], E.err[l], E.RHS[l], E.res[l], op.vis, op.vx, op.vz, op.vxz, op.vxxmzz, op.dtst, E.resfx[l]};
    }
    R.N = E.cfg.nstageS;
    R.ivis = E.cfg.ivis;
    R.ngc = E.ngc;
    R.sz = E.cfg.Vbc == 0 ? -1.0 : 1.0;
    for (int j = 1; j <= R.N; j++) {
        R.cc[j] = E.K.cc[j];
        R.mew[j] = E.K.mew[j];
        R.vv[j] = E.K.vv[j];
        R.mewtc[j] = E.K.mewt[j] * E.cfg.c_2;
    }
    R.G = E.Ginv;
    R.RowB = E.RowB;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute at[1];
    cl::cluster_launch(cfg, at, cluster_bytes_d(E.ngc), E.st);
    PT_COUNT();
    return cuda_check(cudaLaunchKernelEx(&cfg, E.resfx[1].square ? k_cycle_cluster_d<true> : k_cycle_cluster_d<false>, R),
                      "k_cycle_cluster_d");
}

// One multigrid cycle of the reference's schedule, split where the reference tests convergence
// (after the level-1 smoothing pass, iterative_solver.f90:313-315).  Part A: level-1 smoothing,
// residual and sum|r|.  Part B: the rest of the schedule (restrict, coarse visits, coarse solve,
// prolong back to level 1).  Neither part synchronises, so both are captured as CUDA graphs.
static int cycle_part(Engine& E, int part) {
    int rc;
    // the reference's schedule, or a V-cycle when asked for (mg_cycle); the parity path keeps the
    // reference's
    const bool v = E.cfg.mg_cycle == PT_CYCLE_V;
    const int grids = E.grids, nsteps = v ? E.mnsteps : E.nsteps;
    const int* multi = v ? E.mmulti : E.multi;
    if (part == 0) return iterate_stream(E, 1, 1);
    for (int p = 2; p <= nsteps; p++) {
        if (multi[p] >= E.ctop) {  // (the way out is up: the coarsest level is among them)
            if ((rc = cluster_run_d(E, multi, nsteps, p, &p)) || (rc = prolong(E, multi[p]))) return rc;
            continue;
        }
        const int level = multi[p];
        if (multi[p - 1] < multi[p]) {
            if ((rc = compute_RHS(E, level))) return rc;
            if (E.cfg.mg_scheme == PT_MG_CORRECTION && level > 1)
                CK(cudaMemsetAsync(E.err[level], 0, E.gl[level].elems() * sizeof(double), E.st));
        }
        if (level < grids) {
            if ((rc = iterate_stream(E, level, 0))) return rc;
        } else if ((rc = coarse_solve(E))) {
            return rc;
        }
        if (multi[p + 1] < multi[p] && (rc = prolong(E, level))) return rc;
    }
    return 0;
}

static int capture_part(Engine& E, int part, cudaGraphExec_t* exec, int64_t* nlaunch) {
    cudaGraph_t graph = nullptr;
    int64_t before = g_launches.load();
    CK(cudaStreamBeginCapture(E.st, cudaStreamCaptureModeThreadLocal));
    int rc = cycle_part(E, part);
    cudaError_t e = cudaStreamEndCapture(E.st, &graph);
    if (rc) {
        if (graph) cudaGraphDestroy(graph);
        return rc;
    }
    CK(e);
    CK(cudaGraphInstantiate(exec, graph, 0));
    cudaGraphDestroy(graph);
    *nlaunch = g_launches - before;
    g_launches = before;
    return 0;
}

static int run_part(Engine& E, int part) {
    cudaGraphExec_t& ex = part == 0 ? E.gA : E.gB;
    int64_t& n = part == 0 ? E.nA : E.nB;
    if (!ex) {
        int rc = capture_part(E, part, &ex, &n);
        if (rc) return rc;
    }
    CK(cudaGraphLaunch(ex, E.st));
    g_launches += n;
    return 0;
}

int multigrid(Engine& E, pt_solve_info* info) {
    int rc;
    PhaseTimer tm(E, PH_SOLVE);
    {
        PhaseTimer ts(E, PH_SETUP);
        if ((rc = mg_setup_solve(E))) return rc;
        if (E.cfg.guess_mode == PT_GUESS_UNET && (rc = unet_guess(E))) return rc;
    }
    const double norm = (double)(E.gl[1].nx - 2) * (double)(E.gl[1].nz - 2);
    int q = 1;
    double mag1 = 0.0;
    E.res_hist.clear();
    for (;;) {
        {
            PhaseTimer tp(E, PH_CYCLE_L1);
            if ((rc = run_part(E, 0))) return rc;
            CK(cudaMemcpyAsync(E.hscal, E.dscal + 8, 8, cudaMemcpyDeviceToHost, E.st));
        }
        CK(cudaStreamSynchronize(E.st));
        harvest_graph_timer(E, 0);
        mag1 = E.hscal[0] / (double)(E.gl[1].nx - 2) / (double)(E.gl[1].nz - 2);
        (void)norm;
        if (E.res_hist.size() < 100000) E.res_hist.push_back(mag1 / E.res_ref[1]);
        if (!std::isfinite(mag1)) return fail(PT_ERR_NOT_FINITE, "non-finite multigrid residual");
        if (mag1 > 1.0e10 * E.res_ref[1])
            return fail(PT_ERR_MG_DIVERGED, "Multigrid Convergence Problem: Abnormally High Residual Detected");
        if (trace_on()) fprintf(stderr, "[ptgpu] cycle %d residual ratio %.4e\n", q, mag1 / E.res_ref[1]);
        if (q == 2) {  // one full cycle from a learned guess: keep it or restart from the previous psi
            const int fb = unet_check_fallback(E, mag1 / E.res_ref[1]);
            if (fb < 0) return fail(PT_ERR_CUDA, "learned-guess fallback copy");
            if (fb) {
                q++;  // the cycle spent on the dropped guess counts
                continue;
            }
        }
        if (mag1 / E.res_ref[1] <= E.cfg.tolerance) break;
        {
            PhaseTimer tp(E, PH_CYCLE_COARSE);
            if ((rc = run_part(E, 1))) return rc;
        }
        q++;
        if (q > E.cfg.max_cycles) return fail(PT_ERR_MG_MAX_CYCLES, "Multigrid Convergence Problem: Too Many Multigrid Cycles Needed");
    }
    E.cycles = q;
    E.residual_mag1 = mag1;
    E.resid_ratio = mag1 / E.res_ref[1];
    CK(cudaMemcpyAsync(E.SF, E.err[1], E.g1.elems() * 8, cudaMemcpyDeviceToDevice, E.st));
    if (info) {
        info->cycles += q;
        info->resid_ratio = E.resid_ratio;
        info->n_eta = E.n_eta;
        info->eig_fine = E.eig_fine;
    }
    return 0;
}

int mg_alloc(Engine& E) {
    auto alloc = [&](double** p, size_t n) -> int {
        CK(cudaMalloc(p, n * sizeof(double)));
        CK(cudaMemsetAsync(*p, 0, n * sizeof(double), E.st));
        E.bytes_allocated += n * sizeof(double);
        return 0;
    };
    for (int l = 1; l <= E.grids; l++) {
        size_t n = E.gl[l].elems();
        double** arrs[] = {&E.err[l], &E.S0[l], &E.S1[l], &E.S2[l], &E.RHS[l], &E.res[l], &E.dtst[l], &E.ratio[l],
                           &E.vis[l], &E.visst[l], &E.vx[l], &E.vz[l], &E.vxx[l], &E.vzz[l], &E.vxz[l],
                           &E.vxxpzz[l], &E.vxxmzz[l], &E.vsm[l]};
        for (auto a : arrs)
            if (int rc = alloc(a, n)) return rc;
    }
    for (int q = 0; q < 11; q++)
        if (int rc = alloc(&E.visw[q], E.gl[1].elems())) return rc;
    // exact integer stencil sums unless the FP64 path is asked to round like the reference
    E.res_int = !E.cfg.reference_rounding && exact_stencils_setup(E);
    int ldab = 2 * E.kl + E.ku + 1;
    if (int rc = alloc(&E.Mc, (size_t)ldab * E.ngc)) return rc;
    if (int rc = alloc(&E.Bc, E.ngc)) return rc;
    if (int rc = alloc(&E.RowB, E.ngc)) return rc;
    CK(cudaMalloc(&E.ipiv, sizeof(int) * E.ngc));
    CK(cudaMalloc(&E.luw, bandlu::work_bytes(E.ngc, E.kl)));
    const size_t smem = sizeof(double) * (size_t)E.ngc;
    if (smem > 220 * 1024) return fail(PT_ERR_CONFIG, "coarsest grid too large for the banded solve");
    if (band_solve_smem(E.ngc, E.kl, E.ku) > 220 * 1024)
        return fail(PT_ERR_CONFIG, "coarsest grid too large for the banded solve");
    CK(cudaFuncSetAttribute(k_band_solve, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)band_solve_smem(E.ngc, E.kl, E.ku)));
    CK(cudaFuncSetAttribute(k_coarse_apply<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    CK(cudaFuncSetAttribute(k_coarse_apply_mixed, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    // explicit coarse inverse (both precisions): the coarse solve becomes a GEMV spread over the
    // SMs instead of two sequential banded substitutions on one warp of this part's narrow FP64
    // pipe; n^2 doubles, kept while it is small next to the level arrays (n <= 4096: <= 134 MB) and
    // the band is narrow next to n (the bound's second part, 16 band columns and 4 vectors in 200 KB,
    // is where the inverse has always ended)
    if (!E.cfg.reference_rounding && E.ngc <= 4096 && 16 * (E.kl + E.ku + 1) + 4 * E.ngc <= 25 * 1024) {
        CK(cudaMalloc(&E.Ginv, sizeof(double) * (size_t)E.ngc * E.ngc));
        E.bytes_allocated += sizeof(double) * (size_t)E.ngc * E.ngc;
        CK(cudaMalloc(&E.Ginv2, sizeof(double) * (size_t)E.ngc * E.ngc));
        CK(cudaMalloc(&E.Mc2, sizeof(double) * (size_t)ldab * E.ngc));
        CK(cudaMalloc(&E.RowB2, sizeof(double) * (size_t)E.ngc));
        CK(cudaMalloc(&E.ipiv2, sizeof(int) * (size_t)E.ngc));
        CK(cudaMalloc(&E.luw2, bandlu::work_bytes(E.ngc, E.kl)));
        CK(cudaMalloc(&E.derr2, sizeof(int)));
        CK(cudaMallocHost(&E.hflag2, sizeof(int)));
        *E.hflag2 = 0;
        CK(cudaStreamCreateWithFlags(&E.st2, cudaStreamNonBlocking));
        CK(cudaGetDevice(&E.device));
        // the side set of the coarse levels (and level 1's static viscosity snapshot), its work
        // arrays and scalars
        for (int l = 1; l <= E.grids; l++) {
            double** sets[kVisArrays] = {E.vl2.vis, E.vl2.visst, E.vl2.vx, E.vl2.vz, E.vl2.vxx, E.vl2.vzz, E.vl2.vxz,
                                         E.vl2.vxxpzz, E.vl2.vxxmzz, E.vl2.vsm, E.vl2.ratio, E.vl2.dtst};
            for (int a = 0; a < kVisArrays; a++) {
                if (l == 1 && a != 1) continue;  // level 1: only visst (the snapshot)
                if (int rc = alloc(&sets[a][l], E.gl[l].elems())) return rc;
            }
        }
        for (int q = 0; q < 11; q++)
            if (int rc = alloc(&E.visw2[q], E.gl[1].elems())) return rc;
        CK(cudaMalloc(&E.dscal2, 32 * sizeof(double)));
        CK(cudaMallocHost(&E.hscal2, 64 * sizeof(double)));
        CK(cudaEventCreateWithFlags(&E.ev_in, cudaEventDisableTiming));
        CK(cudaEventCreateWithFlags(&E.ev_fact, cudaEventDisableTiming));
        E.bytes_allocated += sizeof(double) * ((size_t)E.ngc * E.ngc + (size_t)ldab * E.ngc + E.ngc);
        if (int rc = bandlu::inverse_setup(E.ngc, E.kl, E.ku, &E.side_clusters)) return rc;
        // On few SMs the worker's inverse takes longer, which costs nothing while it ends within the time step (a
        // new time level waits for it).  Its work is n^2 (kl / 2 + ku) multiply-subtract pairs; a mixed step takes
        // some 5 ms and 1 ms for every 65,000 nodes.  Steps with the whole chip and with six clusters, ms:
        // 256x128 n = 561 (2.4e7) 6.0, 5.7; 384x192 n = 1225 (1.7e8) 8.7, 7.8; 1024x512 n = 2145 (6.8e8) 18.3,
        // 17.7; 2048x1024 n = 2145 36.5, 34.5; past the line 256x128 n = 2145 11.2, 14.2; 512x256 n = 2145 12.7,
        // 15.2; 1280x640 n = 3321 (2.0e9) 31.8, 40.8 (there the worker is the longer path, and a solve that
        // meets its inverse still waits)
        const double work = (double)E.ngc * E.ngc * (0.5 * E.kl + E.ku);
        if (work > 2e8 + 1e3 * (double)(E.K.nx - 1) * (double)(E.K.nz - 1)) E.side_clusters = 0;
    }
    return cluster_setup_d(E);
}

// ------------------------------------------------------------------ learned-guess support
// level-1 values at the nodes of level L (every s-th node), boundary included
__global__ void k_inject(double* c, const double* f, Geo gc, Geo gf, int nxc, int nzc, int s) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.y;
    if (i > nxc || k > nzc) return;
    c[gc.at(i, k)] = f[gf.at(i * s, k * s)];
}
// per interior row of a level: sum RHS*(RHS - r) and (RHS - r)^2  (r = RHS - A g, so RHS - r = A g)
__global__ void k_fit_rows(const double* rhs, const double* r, Geo g, int nx, double* part) {
    __shared__ double s1[128], s2[128];
    const int k = blockIdx.x + 1;
    double a = 0.0, b = 0.0;
    for (int i = 1 + threadIdx.x; i <= nx - 1; i += blockDim.x) {
        const size_t o = g.at(i, k);
        const double ag = rhs[o] - r[o];
        a += rhs[o] * ag;
        b += ag * ag;
    }
    s1[threadIdx.x] = a;
    s2[threadIdx.x] = b;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            s1[threadIdx.x] += s1[threadIdx.x + o];
            s2[threadIdx.x] += s2[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        part[2 * blockIdx.x] = s1[0];
        part[2 * blockIdx.x + 1] = s2[0];
    }
}

// Scale of a psi shape held in err[1], fitted on the coarsest level where the shape's
// grid-scale noise is averaged away: RHS restricted by full weighting (as at a descent), the shape
// injected, alpha = <RHS_L, A_L g> / <A_L g, A_L g> with the level-L operator.  Uses the level
// arrays of levels 2..L, which the cycles overwrite anyway.
int coarse_scale_fit(Engine& E, double* alpha) {
    const int L = E.grids;
    for (int l = 2; l <= L; l++) {
        const Geo& g = E.gl[l];
        PT_COUNT(), k_restrict<<<dim3(nblk(g.nx - 1, 128), g.nz - 1), 128, 0, E.st>>>(E.RHS[l], E.RHS[l - 1], g,
                                                                                       E.gl[l - 1], g.nx, g.nz);
    }
    const Geo& gc = E.gl[L];
    PT_COUNT(), k_inject<<<dim3(nblk(gc.nx + 1, 128), gc.nz + 1), 128, 0, E.st>>>(E.err[L], E.err[1], gc, E.gl[1], gc.nx,
                                                                                   gc.nz, 1 << (L - 1));
    CKL("k_inject");
    if (int rc = enforce_bcs_stream(E, L, E.err[L])) return rc;
    if (int rc = launch_residual(E, L, E.res[L], E.err[L], stream_op(E, L))) return rc;
    PT_COUNT(), k_fit_rows<<<gc.nz - 1, 128, 0, E.st>>>(E.RHS[L], E.res[L], gc, gc.nx, E.red);
    CKL("coarse_scale_fit");
    std::vector<double> part(2 * (size_t)(gc.nz - 1));
    CK(cudaMemcpyAsync(part.data(), E.red, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, E.st));
    CK(cudaStreamSynchronize(E.st));
    double a = 0.0, b = 0.0;
    for (size_t k = 0; k + 1 < part.size(); k += 2) {
        a += part[k];
        b += part[k + 1];
    }
    *alpha = b > 0.0 ? a / b : 0.0;
    return 0;
}

}  // namespace pt
