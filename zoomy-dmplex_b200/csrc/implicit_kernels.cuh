// Kernels of the fully implicit strategy (SolverStrategies.hpp:133-195): BDF
// in time, the residual F(t, X, Xdot) = Xdot - S(X) - R(X) of
// IFunctionWrapper (the transport right-hand side R comes from the ordinary
// stage kernels in MODE_RHS, the source S is the IMEX
// strategy's implicit source), and the preconditioning matrix of
// ModularSolver::FormImplicitJacobian (ModularSolver.hpp:238-371): per cell
// a I - dS/dQ (the identity times a in cells drier than 1e-4) plus the
// forward-difference Jacobians of each face's flux and fluctuations at the
// cell states, scaled by area / volume.  Matrix entries are summed in the
// reference's assembly order (all source blocks, then the faces in increasing
// original face id), so the blocks agree with the CPU restatement bit for
// bit.  The Newton-Krylov iteration around them runs on the host
// (solver.cuh); the vector kernels here serve its GMRES.
#pragma once
#include "imex_kernels.cuh"
#include "rn_div.h"

namespace zsme {

namespace implicit_fd {
constexpr double eps = 1e-7;       // ComputeFaceJacobian_FD / ComputeBoundaryJacobian_FD step
constexpr double dry_jacobian = 1e-4;
}  // namespace implicit_fd

// f = (Xdot - S(y)) - R, Xdot = xdot[id] when given, else
// (c0 y + c1 xn + c2 xnm1) / h (the BDF derivative of the step), the
// coefficients c0, c1, c2, h from device memory (coef) when given
struct BdfTerms {
    const double* xdot;
    const double* xn;
    const double* xnm1;
    double c0, c1, c2, h;
    const double* coef;
};

template <class M>
__device__ __forceinline__ void imp_residual_cell(const MeshDev& m, int c, const double* y, const double* aux,
                                                  const double* __restrict__ params, const double* R, const BdfTerms& b,
                                                  double (&f)[M::n_dof_q]) {
    constexpr int NQ = M::n_dof_q, NA = M::n_dof_qaux;
    const int C = m.C;
    const double* p = params + (size_t)cell_instance(m, c) * m.np;
    double q[NQ], a[NA], S[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) q[i] = y[(size_t)i * C + c];
#pragma unroll
    for (int i = 0; i < NA; ++i) a[i] = aux[(size_t)i * C + c];
    imex_source_cell<M>(q, a, p, S);
    const double c0 = b.coef ? b.coef[0] : b.c0, c1 = b.coef ? b.coef[1] : b.c1;
    const double c2 = b.coef ? b.coef[2] : b.c2;
    const RnDivisor by_h(b.coef ? b.coef[3] : b.h);
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
        const size_t id = (size_t)i * C + c;
        const double xd = b.xdot ? b.xdot[id] : by_h.quotient(c0 * q[i] + c1 * b.xn[id] + c2 * b.xnm1[id]);
        f[i] = (xd - S[i]) - R[id];
    }
}
template <class M>
__global__ void __launch_bounds__(128) imp_residual_kernel(MeshDev m, const double* __restrict__ y,
                                                           const double* __restrict__ aux,
                                                           const double* __restrict__ params,
                                                           const double* __restrict__ R, BdfTerms b,
                                                           double* __restrict__ f) {
    constexpr int NQ = M::n_dof_q;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= m.C) return;
    double fc[NQ];
    imp_residual_cell<M>(m, c, y, aux, params, R, b, fc);
#pragma unroll
    for (int i = 0; i < NQ; ++i) f[(size_t)i * m.C + c] = fc[i];
}

// The forward-difference blocks of a face: of an interior one
// (ComputeFaceJacobian_FD, ModularSolver.hpp:130-185) or the one block of a
// boundary face with a condition (ComputeBoundaryJacobian_FD, :187-236), each
// scaled by area / volume of its row's cell.  fj [4][NQ*NQ][F]: LL, LR, RL, RR,
// faces fastest.  Thread (f, y) perturbs columns of one state, y / kSplit = 0
// the left one (LL and RL), 1 the right one (LR and RR), y % kSplit its share of
// the columns.  A face's columns in one thread, its blocks written NQ*NQ doubles
// apart, took 215 us for 43 k level-2 faces: 24 unpipelined divisions by the step
// per column and a sector per store.
constexpr int kJacSplit = 2;
template <class M, class N>
__global__ void __launch_bounds__(128, 3) imp_face_jac_kernel(MeshDev m, const double* __restrict__ xl,
                                                           const double* __restrict__ al,
                                                           const double* __restrict__ params, double t,
                                                           double* __restrict__ fj) {
    constexpr int NQ = M::n_dof_q, NA = M::n_dof_qaux, Q2 = NQ * NQ;
    constexpr int NJ = (NQ + kJacSplit - 1) / kJacSplit;
    const int F = m.F, C = m.C;
    const int f = blockIdx.x * blockDim.x + threadIdx.x;
    if (f >= F) return;
    const int side = blockIdx.y / kJacSplit, j0 = (blockIdx.y % kJacSplit) * NJ, j1 = min(NQ, j0 + NJ);
    // entry (i, j) of the rows of L and of R
    double* const rowL = fj + (size_t)(side == 0 ? 0 : 1) * Q2 * F + f;
    double* const rowR = fj + (size_t)(side == 0 ? 2 : 3) * Q2 * F + f;
    const int L = m.face_L[f], R = m.face_R[f], bc = m.face_bc[f];
    const double area = m.farea[f];
    const bool used = area > 1e-15 && (R >= 0 || bc >= 0);
    if (!used || (R < 0 && side == 1)) {
        for (int j = j0; j < j1; ++j)
            for (int i = 0; i < NQ; ++i) rowL[(size_t)(i * NQ + j) * F] = rowR[(size_t)(i * NQ + j) * F] = 0.0;
        return;
    }
    const double* p = params + (size_t)face_instance(m, f) * m.np;
    const double X0[3] = {0.0, 0.0, 0.0};
    const double nh[3] = {m.fn[f], m.fn[F + f], 0.0};
    const double xf[3] = {m.fc[f], m.fc[F + f], 0.0};
    const double eps = implicit_fd::eps;
    const RnDivisor by_eps(eps);
    double qL[NQ], aL[NA], qR[NQ], aR[NA];
#pragma unroll
    for (int i = 0; i < NQ; ++i) qL[i] = xl[(size_t)i * C + L];
#pragma unroll
    for (int i = 0; i < NA; ++i) aL[i] = al[(size_t)i * C + L];
    const double fL = area / m.vol[L];
    double fR = 0.0;
    if (R >= 0) {
#pragma unroll
        for (int i = 0; i < NQ; ++i) qR[i] = xl[(size_t)i * C + R];
#pragma unroll
        for (int i = 0; i < NA; ++i) aR[i] = al[(size_t)i * C + R];
        fR = area / m.vol[R];
    } else {
        const auto r = M::boundary_conditions(bc, qL, aL, p, nh, xf, t, 0.0);
#pragma unroll
        for (int i = 0; i < NQ; ++i) qR[i] = r[i];
        if (NA > 0) {
            const auto ra = M::update_aux_variables(qR, aL, p, t, xf);
#pragma unroll
            for (int k = 0; k < NA; ++k) aR[k] = ra[k];
        }
    }
    const auto Fb = N::numerical_flux(qL, qR, aL, aR, p, nh);
    const auto NCb = N::numerical_fluctuations(qL, qR, aL, aR, p, nh);
#pragma unroll 1
    for (int j = j0; j < j1; ++j) {
        double pL[NQ], pR[NQ], bL[NA], bR[NA];
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
            pL[k] = side == 0 && k == j ? qL[k] + eps : qL[k];
            pR[k] = side == 1 && k == j ? qR[k] + eps : qR[k];
        }
#pragma unroll
        for (int k = 0; k < NA; ++k) { bL[k] = aL[k]; bR[k] = aR[k]; }
        if (NA > 0) {   // the perturbed state's aux
            if (side == 0) {
                const auto ra = M::update_aux_variables(pL, bL, p, R >= 0 ? 0.0 : t, R >= 0 ? X0 : xf);
#pragma unroll
                for (int k = 0; k < NA; ++k) bL[k] = ra[k];
            } else {
                const auto ra = M::update_aux_variables(pR, bR, p, 0.0, X0);
#pragma unroll
                for (int k = 0; k < NA; ++k) bR[k] = ra[k];
            }
        }
        if (R < 0) {
            const auto r = M::boundary_conditions(bc, pL, bL, p, nh, xf, t, 0.0);
#pragma unroll
            for (int k = 0; k < NQ; ++k) pR[k] = r[k];
            if (NA > 0) {
                const auto ra = M::update_aux_variables(pR, bL, p, t, xf);
#pragma unroll
                for (int k = 0; k < NA; ++k) bR[k] = ra[k];
            }
        }
        const auto Fp = N::numerical_flux(pL, pR, bL, bR, p, nh);
        const auto NCp = N::numerical_fluctuations(pL, pR, bL, bR, p, nh);
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            const double dFlux = by_eps.quotient(Fp[i] - Fb[i]);
            double eL = 0.0, eR = 0.0;
            eL += dFlux;
            eR -= dFlux;
            eL += by_eps.quotient(NCp[NQ + i] - NCb[NQ + i]);
            eR += by_eps.quotient(NCp[i] - NCb[i]);
            rowL[(size_t)(i * NQ + j) * F] = eL * fL;
            rowR[(size_t)(i * NQ + j) * F] = R >= 0 ? eR * fR : 0.0;
        }
    }
}

// The diagonal block of cell c, [NQ*NQ][C] (entry e = i NQ + j of every cell
// contiguous over the cells): the matrix starts at zero (MatZeroEntries), the
// cell's source block is added (a I - dS/dQ - dS/dAux dAux/dQ at the clamped
// state; a I in cells drier than 1e-4), then the face blocks of the cell's
// faces in increasing original face id (LL where the cell is the face's
// first cell, RR where it is the second; faces without a condition and
// degenerate faces add nothing, as in the reference's face loop).
template <class M>
__global__ void __launch_bounds__(64) imp_cell_jac_kernel(MeshDev m, const double* __restrict__ xl,
                                                          const double* __restrict__ al,
                                                          const double* __restrict__ params, double a,
                                                          const double* __restrict__ fj, double* __restrict__ pd) {
    constexpr int NQ = M::n_dof_q, NA = M::n_dof_qaux, Q2 = NQ * NQ;
    const int C = m.C, K = m.K;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const double* p = params + (size_t)cell_instance(m, c) * m.np;
    const double X0[3] = {0.0, 0.0, 0.0};
    double q[NQ], aux[NA], J[Q2];
#pragma unroll
    for (int i = 0; i < NQ; ++i) q[i] = xl[(size_t)i * C + c];
#pragma unroll
    for (int i = 0; i < NA; ++i) aux[i] = al[(size_t)i * C + c];
    if (NQ > 1 && q[1] < implicit_fd::dry_jacobian) {
#pragma unroll
        for (int e = 0; e < Q2; ++e) J[e] = 0.0;
#pragma unroll
        for (int i = 0; i < NQ; ++i) J[i * NQ + i] = a;
    } else {
        const auto dSdQ = M::source_jacobian_wrt_variables(q, aux, p);
        const auto dSdA = M::source_jacobian_wrt_aux_variables(q, aux, p);
        double dAdQ[NA * NQ + 1];
        if constexpr (HasAuxJacobian<M>::value) {
            const auto r = M::update_aux_variables_jacobian_wrt_variables(q, aux, p);
#pragma unroll
            for (int e = 0; e < NA * NQ; ++e) dAdQ[e] = r[e];
        } else {   // forward differences, SourceStep.hpp:16-53
            const auto a0 = M::update_aux_variables(q, aux, p, 0.0, X0);
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                double qp[NQ];
#pragma unroll
                for (int mm = 0; mm < NQ; ++mm) qp[mm] = q[mm];
                const double hh = 1e-7 * (fabs(q[j]) + 1e-7);
                qp[j] += hh;
                const auto a1 = M::update_aux_variables(qp, aux, p, 0.0, X0);
#pragma unroll
                for (int k = 0; k < NA; ++k) dAdQ[k * NQ + j] = (a1[k] - a0[k]) / hh;
            }
        }
#pragma unroll
        for (int i = 0; i < NQ; ++i)
#pragma unroll
            for (int j = 0; j < NQ; ++j) {
                const double val = i == j ? a : 0.0;
                double dSource = dSdQ[i * NQ + j];
#pragma unroll
                for (int k = 0; k < NA; ++k) dSource += dSdA[i * NA + k] * dAdQ[k * NQ + j];
                J[i * NQ + j] = val - dSource;
            }
    }
    // the cell's face blocks in increasing original face id
    const double* blk[4] = {nullptr, nullptr, nullptr, nullptr};
    int nblk = 0;
    const int ord = m.order[c];
    for (int jj = 0; jj < K; ++jj) {
        const int k = (ord >> (2 * jj)) & 3;
        const int f = m.slot_face[k * C + c];
        if (f < 0) continue;
        if (m.face_R[f] < 0 && m.face_bc[f] < 0) continue;
        if (!(m.farea[f] > 1e-15)) continue;
        const double* const here = fj + (size_t)(m.face_L[f] == c ? 0 : 3) * Q2 * m.F + f;
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (b == nblk) blk[b] = here;
        ++nblk;
    }
#pragma unroll
    for (int e = 0; e < Q2; ++e) {
        double acc = 0.0;
        acc += J[e];
#pragma unroll
        for (int b = 0; b < 4; ++b)
            if (b < nblk) acc += blk[b][(size_t)e * m.F];
        pd[(size_t)e * C + c] = acc;
    }
}

// LU factors of every diagonal block with partial pivoting (the block-Jacobi
// preconditioner of the Krylov solve): lu [NQ*NQ][C] with the row swaps of piv
// [NQ][C], and the reciprocals of the diagonal in rdiag [NQ][C]; a block with a
// zero or non-finite pivot is applied as the identity.  A column divides by its
// pivot's reciprocal.  The block lives in local memory (a stack frame of its
// size, 288, 512 and 1152 bytes at 6, 8 and 12 components, no spills): the row
// swaps' branches keep it out of registers, as gepp_regs.h says of blend.
template <int NQ>
__global__ void __launch_bounds__(64) imp_block_lu_kernel(int C, const double* __restrict__ pd,
                                                          double* __restrict__ lu, int* __restrict__ piv,
                                                          double* __restrict__ rdiag) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    double A[NQ][NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i)
#pragma unroll
        for (int j = 0; j < NQ; ++j) A[i][j] = pd[(size_t)(i * NQ + j) * C + c];
    int pv[NQ];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        int mr = k;
        double mv = fabs(A[k][k]);
#pragma unroll
        for (int i = k + 1; i < NQ; ++i) {
            const double v = fabs(A[i][k]);
            if (v > mv) { mv = v; mr = i; }
        }
        pv[k] = mr;
        if (mr != k) {
#pragma unroll
            for (int i = k + 1; i < NQ; ++i)
                if (mr == i) {
#pragma unroll
                    for (int j = 0; j < NQ; ++j) {
                        const double tt = A[k][j];
                        A[k][j] = A[i][j];
                        A[i][j] = tt;
                    }
                }
        }
        const double pkk = A[k][k];
        if (!(mv > 0.0) || !isfinite(pkk)) ok = false;
        const RnDivisor by_pivot(pkk);
#pragma unroll
        for (int i = k + 1; i < NQ; ++i) {
            const double l = by_pivot.quotient(A[i][k]);
            A[i][k] = l;
#pragma unroll
            for (int j = k + 1; j < NQ; ++j) A[i][j] -= l * A[k][j];
        }
    }
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
#pragma unroll
        for (int j = 0; j < NQ; ++j) lu[(size_t)(i * NQ + j) * C + c] = ok ? A[i][j] : (i == j ? 1.0 : 0.0);
        piv[(size_t)i * C + c] = ok ? pv[i] : i;
        rdiag[(size_t)i * C + c] = ok ? 1.0 / A[i][i] : 1.0;
    }
}

// b <- D^-1 b for cell c from the LU factors: each triangle is loaded before it
// is used, since the row swaps' branches would keep the loads apart, and the
// quotients are branch-free with a plain repetition behind them.
template <int NQ>
__device__ __forceinline__ void imp_block_solve(int C, int c, const double* __restrict__ lu,
                                                const int* __restrict__ piv, const double* __restrict__ rdiag,
                                                double (&b)[NQ]) {
    double T[NQ][NQ], rd[NQ], f[NQ];
    int pv[NQ];
    bool swaps = false;
#pragma unroll
    for (int k = 0; k < NQ; ++k) pv[k] = piv[(size_t)k * C + c];
#pragma unroll
    for (int i = 1; i < NQ; ++i)
#pragma unroll
        for (int j = 0; j < i; ++j) T[i][j] = lu[(size_t)(i * NQ + j) * C + c];
#pragma unroll
    for (int k = 0; k < NQ; ++k) swaps |= pv[k] != k;
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
        if (swaps) {
#pragma unroll
            for (int i = k + 1; i < NQ; ++i) {
                const double bk = b[k], bi = b[i];
                b[k] = pv[k] == i ? bi : bk;
                b[i] = pv[k] == i ? bk : bi;
            }
        }
#pragma unroll
        for (int i = k + 1; i < NQ; ++i) b[i] -= T[i][k] * b[k];
    }
#pragma unroll
    for (int i = 0; i < NQ; ++i) {
#pragma unroll
        for (int j = i; j < NQ; ++j) T[i][j] = lu[(size_t)(i * NQ + j) * C + c];
        rd[i] = rdiag[(size_t)i * C + c];
        f[i] = b[i];
    }
    auto back = [&](auto plain) {
        bool odd = false;
#pragma unroll
        for (int i = NQ - 1; i >= 0; --i) {
            double s = f[i];
#pragma unroll
            for (int j = i + 1; j < NQ; ++j) s -= T[i][j] * b[j];
            b[i] = plain ? s / T[i][i] : RnDivisor(T[i][i], rd[i]).signed_quotient_or(s, odd);
        }
        return odd;
    };
    if (back(std::false_type())) back(std::true_type());
}
// z = D^-1 r (r and z may alias)
template <int NQ>
__global__ void __launch_bounds__(128) imp_block_solve_kernel(int C, const double* __restrict__ lu,
                                                              const int* __restrict__ piv,
                                                              const double* __restrict__ rdiag, const double* r,
                                                              double* z) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    double b[NQ];
#pragma unroll
    for (int i = 0; i < NQ; ++i) b[i] = r[(size_t)i * C + c];
    imp_block_solve<NQ>(C, c, lu, piv, rdiag, b);
#pragma unroll
    for (int i = 0; i < NQ; ++i) z[(size_t)i * C + c] = b[i];
}

// UpdateState of a state: xl = the state clamped (update_variables), al = its
// aux (update_aux_variables) from the handle's aux
template <class M>
__global__ void __launch_bounds__(128) imp_update_state_kernel(MeshDev m, const double* __restrict__ y,
                                                               const double* __restrict__ aux,
                                                               const double* __restrict__ params,
                                                               double* __restrict__ xl, double* __restrict__ al) {
    constexpr int NQ = M::n_dof_q, NA = M::n_dof_qaux;
    const int C = m.C;
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= C) return;
    const double* p = params + (size_t)cell_instance(m, c) * m.np;
    double q[NQ], a[NA];
#pragma unroll
    for (int i = 0; i < NQ; ++i) q[i] = y[(size_t)i * C + c];
#pragma unroll
    for (int i = 0; i < NA; ++i) a[i] = aux[(size_t)i * C + c];
    constrain<M>(q, a, p);
#pragma unroll
    for (int i = 0; i < NQ; ++i) xl[(size_t)i * C + c] = q[i];
#pragma unroll
    for (int i = 0; i < NA; ++i) al[(size_t)i * C + c] = a[i];
}

// out = D^-1 (F(y) - F0) / hv for the perturbed state y = X + hv v whose transport
// right-hand side is R: the residual, the matrix-free Jacobian's difference
// quotient (zero when hv is zero) and the block solve of a cell in one pass
// (29 us as three kernels for 29 k level-2 cells).
template <class M>
__global__ void __launch_bounds__(128) imp_apply_kernel(MeshDev m, const double* y, const double* aux,
                                                        const double* __restrict__ params, const double* R, BdfTerms b,
                                                        const double* F0, const double* hv,
                                                        const double* __restrict__ lu, const int* __restrict__ piv,
                                                        const double* __restrict__ rdiag, double* __restrict__ out) {
    constexpr int NQ = M::n_dof_q;
    grid_release();
    grid_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x, C = m.C;
    if (c >= C) return;
    double f[NQ];
    imp_residual_cell<M>(m, c, y, aux, params, R, b, f);
    const double h = *hv;
    const RnDivisor by_h(h);
#pragma unroll
    for (int i = 0; i < NQ; ++i) f[i] = h != 0.0 ? by_h.quotient(f[i] - F0[(size_t)i * C + c]) : 0.0;
    imp_block_solve<NQ>(C, c, lu, piv, rdiag, f);
#pragma unroll
    for (int i = 0; i < NQ; ++i) out[(size_t)i * C + c] = f[i];
}

// ------------------------------------------------------------ vector kernels
static __global__ void imp_sqrt_kernel(const double* __restrict__ in, double* __restrict__ out) { *out = sqrt(*in); }
// out = 1.0 x + hv v, hv a device scalar
static __global__ void imp_perturb_kernel(long long n, const double* x, const double* v, const double* hv,
                                          double* __restrict__ out) {
    grid_release();
    grid_wait();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = 1.0 * x[i] + *hv * v[i];
}
// out = a x + b y (out may alias x or y; y may be null when b = 0)
static __global__ void imp_lincomb_kernel(long long n, double a, const double* x, double b, const double* y,
                                          double* out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    out[i] = y ? a * x[i] + b * y[i] : a * x[i];
}

// Inner products, deterministic: block b sums its chunk (a fixed stride per
// thread, a fixed tree per block) into partial[k][b], and the last block to
// arrive sums the partials the same way into out[k].  count: blocks arrived,
// zero between launches.  hv, when given: the matrix-free Jacobian's
// differencing parameter sqrt(eps) sqrt(1 + |X|) / |v| from out[0] = v.v (0 for
// a zero vector).
struct DotSink {
    double* partial;
    int* count;
    double* out;
    double* hv;
    const double* xnorm;
};
// the sum of the block's 256 values of s, in thread 0: pairs 128, 64, ... 1 apart
__device__ __forceinline__ double imp_block_sum(double s, double* sh) {
    const int t = threadIdx.x;
    sh[t] = s;
    __syncthreads();
    if (t < 128) sh[t] = s = s + sh[t + 128];
    __syncthreads();
    if (t < 64) sh[t] = s = s + sh[t + 64];
    __syncthreads();
    if (t < 32) {
        s = s + sh[t + 32];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) s = s + __shfl_down_sync(0xffffffffu, s, off);
    }
    return s;
}
// vectors k0 .. k0 + NK (below nk); group: their counter
template <int NK>
__device__ __forceinline__ void imp_finish_dots(const double (&s)[NK], int k0, int nk, int group, const DotSink& d) {
    __shared__ double sh[NK][256];
    __shared__ int arrived;
    const int nb = gridDim.x;
    double block[NK];
#pragma unroll
    for (int q = 0; q < NK; ++q) block[q] = imp_block_sum(s[q], sh[q]);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 0; q < NK; ++q)
            if (k0 + q < nk) d.partial[(size_t)(k0 + q) * nb + blockIdx.x] = block[q];
        __threadfence();
        arrived = atomicAdd(d.count + group, 1);
    }
    __syncthreads();
    if (arrived != nb - 1) return;
    __threadfence();
    double t[NK];
#pragma unroll
    for (int q = 0; q < NK; ++q) {
        t[q] = 0.0;
        if (k0 + q < nk)
            for (int b = threadIdx.x; b < nb; b += blockDim.x) t[q] += __ldcg(d.partial + (size_t)(k0 + q) * nb + b);
    }
#pragma unroll
    for (int q = 0; q < NK; ++q) {
        const double sum = imp_block_sum(t[q], sh[q]);
        if (threadIdx.x == 0 && k0 + q < nk) {
            d.out[k0 + q] = sum;
            if (d.hv && k0 + q == 0) {
                const double vn = sqrt(sum);
                *d.hv = vn > 0.0 ? 1.4901161193847656e-08 * sqrt(1.0 + *d.xnorm) / vn : 0.0;
            }
        }
    }
    if (threadIdx.x == 0) d.count[group] = 0;
}
// out[k] = V_k . w, k < nk (V_k = V + k ld): NK vectors per block row
template <int NK>
__global__ void __launch_bounds__(256) imp_multi_dot_kernel(long long n, int nk, const double* V, long long ld,
                                                            const double* w, DotSink d) {
    grid_release();
    grid_wait();
    const int k0 = blockIdx.y * NK;
    double s[NK];
    const double* v[NK];
#pragma unroll
    for (int q = 0; q < NK; ++q) {
        s[q] = 0.0;
        v[q] = V + (size_t)min(k0 + q, nk - 1) * ld;
    }
#pragma unroll 2
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double wi = w[i];
#pragma unroll
        for (int q = 0; q < NK; ++q) s[q] += v[q][i] * wi;
    }
    imp_finish_dots<NK>(s, k0, nk, blockIdx.y, d);
}
// w -= sum_k h_k V_k (classical Gram-Schmidt projection, h on the device) and
// out[0] = w.w; four elements' chains run side by side
static __global__ void __launch_bounds__(256) imp_project_kernel(long long n, int nk, const double* V, long long ld,
                                                                 const double* h, double* __restrict__ w, DotSink d) {
    grid_release();
    grid_wait();
    const long long stride = (long long)gridDim.x * blockDim.x;
    double sum[1] = {0.0};
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += 4 * stride) {
        double s[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) s[e] = i + e * stride < n ? w[i + e * stride] : 0.0;
#pragma unroll 4
        for (int k = 0; k < nk; ++k) {
            const double hk = h[k];
            const double* const v = V + (size_t)k * ld + i;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                if (i + e * stride < n) s[e] -= hk * v[e * stride];
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (i + e * stride < n) {
                w[i + e * stride] = s[e];
                sum[0] += s[e] * s[e];
            }
    }
    imp_finish_dots<1>(sum, 0, 1, 0, d);
}
// v = (1.0 / sqrt(ww)) w where ww = w.w > 0 (the next Arnoldi vector) and out[0] = v.v
static __global__ void __launch_bounds__(256) imp_normalize_kernel(long long n, const double* ww, const double* w,
                                                                   double* __restrict__ v, DotSink d) {
    grid_release();
    grid_wait();
    const double hn = sqrt(*ww), r = 1.0 / hn;
    double sum[1] = {0.0};
#pragma unroll 4
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (long long)gridDim.x * blockDim.x) {
        const double s = hn > 0.0 ? r * w[i] : v[i];
        v[i] = s;
        sum[0] += s * s;
    }
    imp_finish_dots<1>(sum, 0, 1, 0, d);
}
// x += sum_k y_k V_k (the Krylov update, y on the device)
static __global__ void imp_multi_add_kernel(long long n, int nk, const double* __restrict__ V, long long ld,
                                            const double* __restrict__ y, double* __restrict__ x) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double s = x[i];
    for (int k = 0; k < nk; ++k) s += y[k] * V[(size_t)k * ld + i];
    x[i] = s;
}

}  // namespace zsme
