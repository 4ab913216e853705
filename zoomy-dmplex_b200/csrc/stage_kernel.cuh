// One SSP stage (or one right-hand side) in one kernel: the face states of
// prep_kernel, the fluxes of face_kernel and the sums of gather_kernel over a
// tile of consecutive cells, the same operations in the same order.
//
// The separate kernels hand the stage over through HBM: 2 NQ doubles per face
// of face states and 3 NQ of contributions, written scattered (a warp's store
// touches 22 sectors of the 8 it fills) and read back.  Here a block keeps its
// tile's state with two rings of neighbours, its faces' states and their
// contributions in shared memory, so a stage reads the state and the mesh once
// and writes the next state, in one launch.  The price is repeated work on the
// tile's rim: at 256 faces a tile has about 150 cells, reconstructs 28 % more
// and evaluates 12 % more faces than it owns.
#pragma once
#include <type_traits>

#include "rn_div.h"

namespace zsme {

// One tile of the stage kernel.
struct alignas(16) StageTile {
    int c0, n, nloc, nent;      // first cell, cells, cells with both rings, cells with ring 1
    int e0, eo, f0, nown;       // first ring cell, first entry, first own face, own faces
    int in0, nf, g0, ng;        // first incoming face, faces, first ghost, ghosts
};

// Device view of the tiles (FaceTiles + StageTiles of prepared_mesh.h).
struct StageTilesDev {
    const StageTile* tile;
    const int* in_faces;
    const int* ord_lf;      // [K][C]
    const int* ext_cell;
    const int* gho_cell;
    const int* gho_face;
    const unsigned* loc;    // [K][entries]
    const double* geo;      // [2 K DIM + 2][entries]: per face the outward normal (Green-Gauss) or the
                            // weights (least squares), then face centroid - cell centroid (zero where
                            // there is no face), then the volume and its reciprocal
    int entries;
    int fst;                // row length of the face rows (> the most faces of a tile)
    int cst;                // row length of the cell rows (>= the most cells and ghosts of a tile)
};

// P threads per cell reconstruct NC components each
template <int NQ, int P>
struct StageShape {
    static constexpr int NC = (NQ + P - 1) / P;
    // row lengths are s0 modulo 16 so that the P parts of a cell (NC rows
    // apart) fall into different shared-memory banks
    static constexpr int s0() {
        for (int s = 1; s < 16; ++s)
            if ((NC * s) % 16 == 4 || (NC * s) % 16 == 12) return s;
        return 1;
    }
    static int row(int n) {
        int r = n;
        while (r % 16 != s0()) ++r;
        return r;
    }
};
// Shared memory of a block, in doubles: the raw state, the volumes and their
// reciprocals, the cells' face rows (K ints), then 3 NQ face rows whose last
// third holds the clamped state until the fluxes are formed.
template <int NQ>
inline size_t stage_smem_doubles(int fst, int cst) {
    const size_t a = (size_t)3 * NQ * fst, b = (size_t)2 * NQ * fst + (size_t)NQ * cst;
    return (size_t)(NQ + 4) * cst + (a > b ? a : b);
}
// The SSP-RK(s,2) stage combination's coefficients: the state's and the start
// state's weight in the last stage, and what the step's dt is divided by.
struct StageWeights {
    double state, start, dt_div;
};
// The positivity variants' reconstruction (prep_wb_kernel): variant and dry threshold.
struct StagePositivity {
    int variant;
    double eps;
};

// The entries' geometry, gathered once when the tiles are built, so that the
// stage kernel reads it coalesced and without waiting for indices.
static __global__ void __launch_bounds__(128) stage_entries_kernel(MeshDev m, const StageTile* __restrict__ tiles,
                                                                   const int* __restrict__ ext_cell,
                                                                   const unsigned* __restrict__ loc, int NE, int DIM,
                                                                   int least_squares, double* __restrict__ geo) {
    const StageTile t = tiles[blockIdx.x];
    const int C = m.C, K = m.K;
    for (int l = threadIdx.x; l < t.nent; l += blockDim.x) {
        const int c = l < t.n ? t.c0 + l : ext_cell[t.e0 + l - t.n];
        const size_t ent = (size_t)t.eo + l;
        for (int k = 0; k < K; ++k) {
            const unsigned e = loc[(size_t)k * NE + ent];
            const bool across = (e & 0xfffu) != kLocNone, isL = (e >> 23) & 1u, face = (e >> 26) & 1u;
            const int slot = (int)((e >> 24) & 3u), f = m.slot_face[(size_t)slot * C + c];
            for (int d = 0; d < DIM; ++d) {
                double w = 0.0;
                if (across && least_squares) w = m.slot_w[((size_t)slot * 2 + d) * C + c];
                if (across && !least_squares) w = isL ? m.fnr[(size_t)d * m.F + f] : -m.fnr[(size_t)d * m.F + f];
                geo[((size_t)k * DIM + d) * NE + ent] = w;
                geo[((size_t)(K + k) * DIM + d) * NE + ent] =
                    face ? m.slot_dx[((size_t)slot * 2 + d) * C + c] : 0.0;
            }
        }
        geo[(size_t)2 * K * DIM * NE + ent] = m.vol[c];
        geo[((size_t)2 * K * DIM + 1) * NE + ent] = 1.0 / m.vol[c];
    }
}

// WB: the face states of the positivity variants (prep_wb_kernel; order 2, P = 1).
// mode / x_in / x_out / base as gather_kernel, except that x_out never is
// x_in (another tile reads its rim there): MODE_MID and MODE_EULER write x_out.
template <class M, class N, int P, int KM, int THREADS, int MINB, bool WB = false>
__global__ void __launch_bounds__(THREADS, MINB) stage_kernel(MeshDev m, Opts o, StageTilesDev tl,
                                                              StageWeights sc, StagePositivity pos,
                                                              const double* x_in, const double* aux,
                                                              const double* __restrict__ params, double t_host,
                                                              const double* t_dev, double stage_frac,
                                                              const double* dt_step, const int* active, int mode,
                                                              double* x_out, double* base) {
    constexpr int NQ = M::n_dof_q, NA = M::n_dof_qaux, DIM = M::dimension;
    constexpr int NC = StageShape<NQ, P>::NC;
    constexpr int CH = NC <= 3 ? NC : (NC % 3 == 0 ? 3 : 2);   // components whose chains overlap
    constexpr bool KEEP = NC * KM <= 12;   // increments stay in registers, else in their face row
    extern __shared__ double smem[];
    const int C = m.C, F = m.F;
    const int K = KM == 3 ? 3 : m.K;
    const int fst = tl.fst, cst = tl.cst;
    double* const sw = smem;                           // [NQ][cst] raw stage state
    double* const sv = smem + (size_t)NQ * cst;        // [2][cst] volume, 1 / volume
    int* const srow = (int*)(sv + 2 * cst);            // [K][cst] the cells' face rows in accumulation order
    double* const rows = sv + 4 * cst;                 // [3 NQ][fst]
    double* const swl = rows + (size_t)2 * NQ * fst;   // [NQ][cst] clamped stage state
    const int tid = threadIdx.x, nt = blockDim.x;
    grid_release();
    const StageTile tile = tl.tile[blockIdx.x];
    const int n = tile.n, nloc = tile.nloc, nent = tile.nent;
    const bool second = o.order >= 2, lsq = o.gradient == 1;

    // the first task's geometry, on its way while the state is loaded
    int ent = min(tid / P, nent - 1);
    unsigned le[KM];
    double geo[KM][2 * DIM], vol, rvol;
    auto geometry = [&]() {
        const double* const g = tl.geo + tile.eo + ent;
        const size_t NE = tl.entries;
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            if (k < K) {
                le[k] = tl.loc[k * NE + tile.eo + ent];
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    geo[k][d] = g[(k * DIM + d) * NE];
                    geo[k][DIM + d] = g[((K + k) * DIM + d) * NE];
                }
            } else {
                le[k] = kLocNone | (kRowNone << 12);
#pragma unroll
                for (int d = 0; d < 2 * DIM; ++d) geo[k][d] = 0.0;
            }
        }
        vol = g[2 * K * DIM * NE];
        rvol = g[(2 * K * DIM + 1) * NE];
    };
    geometry();
    // ---- the state of the tile and its rings, raw and clamped
    for (int l = tid; l < n; l += nt)
        for (int j = 0; j < K; ++j) srow[j * cst + l] = tl.ord_lf[(size_t)j * C + tile.c0 + l];
    grid_wait();   // what follows reads the state
    bool changed = false;
    for (int l = tid; l < nloc; l += nt) {
        const int c = l < n ? tile.c0 + l : tl.ext_cell[tile.e0 + l - n];
        double q[NQ], a[NA];
        load_q<NQ>(x_in, C, c, q);
#pragma unroll
        for (int i = 0; i < NA; ++i) a[i] = aux[(size_t)i * C + c];
#pragma unroll
        for (int i = 0; i < NQ; ++i) sw[i * cst + l] = q[i];
        double ql[NQ];
#pragma unroll
        for (int i = 0; i < NQ; ++i) ql[i] = q[i];
        clamp_q<M>(ql, a, params + (size_t)cell_instance(m, c) * m.np);
#pragma unroll
        for (int i = 0; i < NQ; ++i) {
            changed |= __double_as_longlong(q[i]) != __double_as_longlong(ql[i]);
            swl[i * cst + l] = ql[i];
        }
    }
    // dt times the stage's weight; an ensemble's cells form their own instance's
    const double h0 = dt_step && !m.cell_inst ? dt_step[0] / sc.dt_div : 0.0;
    // a tile whose clamp changes nothing reads one copy
    const bool clamped = __syncthreads_or(changed);
    if (tile.ng > 0) {   // ghost values of the Green-Gauss boundary faces
        for (int g = tid; g < tile.ng; g += nt) {
            const int l = tl.gho_cell[tile.g0 + g], f = tl.gho_face[tile.g0 + g];
            double qg[NQ];
#pragma unroll
            for (int i = 0; i < NQ; ++i) qg[i] = sw[i * cst + l];
            const double nh[3] = {m.fn[f], m.fn[F + f], 0.0};
            const double xf[3] = {m.fc[f], m.fc[F + f], 0.0};
            const double* p = params + (size_t)face_instance(m, f) * m.np;
            const auto qb = M::boundary_conditions(m.face_bc[f], qg, (const double*)nullptr, p, nh, xf, 0.0, 0.0);
#pragma unroll
            for (int i = 0; i < NQ; ++i) sw[i * cst + nloc + g] = qb[i];
        }
        __syncthreads();
    }

    // ---- face states (prep_kernel), P threads per cell of the tile and ring 1.
    // The loop over the components is free of branches: the values of missing
    // faces and the plain divisions are left to the general and the odd path.
    const double* const sq = clamped ? swl : sw;
    for (int task = tid; task < ((nent * P + 31) & ~31); task += nt) {
        const int part = task % P, i0 = part * NC;
        if (task != tid) {
            ent = min(task / P, nent - 1);
            geometry();
        }
        const bool live = task < nent * P;
        int nb[KM], fso[KM];
        bool inner[KM];
        bool whole = true;   // every face has a cell behind it
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const int across = (int)(le[k] & 0xfffu), row = (int)((le[k] >> 12) & 0x7ffu);
            inner[k] = across < nloc;
            whole &= inner[k];
            nb[k] = across == (int)kLocNone ? ent : across;
            // states that no face of the tile takes go to the rows' last column
            fso[k] = (live && row != (int)kRowNone) ? ((le[k] >> 23) & 1u ? 0 : NQ * fst) + row : fst - 1;
        }
        if (!second) {
            if (live) {
#pragma unroll
                for (int ii = 0; ii < NC; ++ii) {
                    if (NC * P != NQ && i0 + ii >= NQ) break;
                    const double q = swl[(i0 + ii) * cst + ent];
#pragma unroll
                    for (int k = 0; k < KM; ++k) rows[(i0 + ii) * fst + fso[k]] = q;
                }
                if (part == 0 && ent < n) {
                    sv[ent] = vol;
                    sv[cst + ent] = rvol;
                }
            }
            continue;
        }
        const RnDivisor by_vol(vol, rvol);
        const bool divide = !lsq && vol > 1e-15;
        // a part beyond the last component repeats it: the same face states again,
        // or none where its row still holds the increment that the state is formed of
        auto component = [&](int ii) { return NC * P == NQ ? i0 + ii : min(i0 + ii, NQ - 1); };
        auto own = [&](int ii) { return KEEP || NC * P == NQ || i0 + ii < NQ; };
        auto load = [&](const double* from, int i, double& q, double (&v)[KM]) {
            q = from[i * cst + ent];
#pragma unroll
            for (int k = 0; k < KM; ++k) v[k] = from[i * cst + nb[k]];
        };
        // the bounds of a component over the cell and its neighbours
        auto bounds = [&](bool all, double q, const double (&v)[KM], double& mn, double& mx) {
            mn = mx = q;
#pragma unroll
            for (int k = 0; k < KM; ++k) {
                const double w = all || inner[k] ? v[k] : q;
                mn = w < mn ? w : mn;
                mx = w > mx ? w : mx;
            }
        };
        // the gradient of the raw state: least squares (Gradient.hpp:330-346) or
        // Green-Gauss (Gradient.hpp:91-176), before the division by the volume
        auto gradient = [&](bool least, bool all, double q, const double (&v)[KM], double (&g)[DIM]) {
#pragma unroll
            for (int d = 0; d < DIM; ++d) g[d] = 0.0;
#pragma unroll
            for (int k = 0; k < KM; ++k) {
                double fv = least ? v[k] - q : 0.5 * (q + v[k]);
                if (!all && !inner[k]) fv = v[k];   // a ghost's value; a missing face has a zero normal
#pragma unroll
                for (int d = 0; d < DIM; ++d) g[d] += geo[k][d] * fv;
            }
        };
        // the plain gradient, as prep_kernel writes it
        auto plain_gradient = [&](int i, double (&g)[DIM]) {
            double q, v[KM];
            load(sw, i, q, v);
#pragma unroll
            for (int d = 0; d < DIM; ++d) g[d] = 0.0;
#pragma unroll
            for (int k = 0; k < KM; ++k) {
                if ((le[k] & 0xfffu) == kLocNone) continue;
                const double fv = lsq ? v[k] - q : (inner[k] ? 0.5 * (q + v[k]) : v[k]);
#pragma unroll
                for (int d = 0; d < DIM; ++d) g[d] += geo[k][d] * fv;
            }
#pragma unroll
            for (int d = 0; d < DIM; ++d)
                if (divide) g[d] = g[d] / vol;
        };
        if constexpr (WB) {
            static_assert(P == 1, "one thread per cell");
            constexpr int B = 0, H = 1;
            const double eps2 = venkat_eps2<DIM>(vol);
            const double b_bar = sq[B * cst + ent], h_bar = sq[H * cst + ent];
            // the cell's face states (see prep_wb_kernel for the scheme); plain: with
            // the divisions prep_wb_kernel makes, for the cells whose branch-free
            // quotients the other form reports odd
            auto reconstruct = [&](auto plain) {
                bool odd = !lsq && !divide;
                auto gradient_of = [&](int i, double (&g)[DIM]) {
                    if (plain) {
                        plain_gradient(i, g);
                        return;
                    }
                    double q, v[KM];
                    load(sw, i, q, v);
                    gradient(lsq, whole, q, v, g);
                    odd |= !whole && exponent_word(q) >= 0x7ff00000u;
                    if (!lsq) {
#pragma unroll
                        for (int e = 0; e < DIM; ++e) g[e] = by_vol.quotient_or(g[e], odd);
                    }
                };
                // Venkatakrishnan factor: the smallest over the cell's faces
                auto factor = [&](double wc, double wmn, double wmx, const double (&g)[DIM]) {
                    double ph = 1.0;
#pragma unroll
                    for (int k = 0; k < KM; ++k) {
                        double delta = 0.0;
#pragma unroll
                        for (int e = 0; e < DIM; ++e) delta += g[e] * geo[k][DIM + e];
                        const bool skip = fabs(delta) < 1e-14 || !(le[k] >> 26 & 1u);
                        const double dm = (delta > 0) ? (wmx - wc) : (wmn - wc);
                        const double nu = dm * dm + eps2 + 2 * delta * dm;
                        const double de = dm * dm + 2 * delta * delta + delta * dm + eps2;
                        double pf;
                        if (plain) {
                            pf = (de > 1e-30) ? nu / de : 1.0;
                        } else {
                            bool far = !(de > 1e-30);
                            const RnDivisor by_de(de, rn_reciprocal(de, far));
                            pf = by_de.quotient_or(nu, far);
                            odd |= far & !skip;
                        }
                        pf = (pf < 1.0) ? pf : 1.0;   // std::min(1, pf)
                        pf = (0.0 < pf) ? pf : 0.0;   // std::max(0, pf)
                        ph = !skip && pf < ph ? pf : ph;
                    }
                    return ph;
                };
                double gb[DIM], ge[DIM], phb, phe;
                gradient_of(B, gb);
                gradient_of(H, ge);
#pragma unroll
                for (int d = 0; d < DIM; ++d) ge[d] = ge[d] + gb[d];
                {
                    double q, vb[KM], vh[KM], mn, mx;
                    load(sq, B, q, vb);
                    bounds(whole, q, vb, mn, mx);
                    phb = factor(q, mn, mx, gb);
                    load(sq, H, q, vh);
#pragma unroll
                    for (int k = 0; k < KM; ++k) vh[k] = vb[k] + vh[k];
                    bounds(whole, b_bar + h_bar, vh, mn, mx);
                    phe = factor(b_bar + h_bar, mn, mx, ge);
                }
                if (h_bar < pos.eps) phb = phe = 0.0;
                phb = (phe < phb) ? phe : phb;
                double sh[DIM];
#pragma unroll
                for (int d = 0; d < DIM; ++d) sh[d] = phe * ge[d] - phb * gb[d];
                double hmin = h_bar;
#pragma unroll
                for (int k = 0; k < KM; ++k) {
                    double hf = h_bar;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) hf += sh[d] * geo[k][DIM + d];
                    if (hf < hmin && (le[k] >> 26 & 1u)) hmin = hf;
                }
                double theta = 1.0;
                if (pos.variant != ZSME_POSITIVITY_MOOD && hmin < 0.0) {
                    const double gap = h_bar - hmin;
                    double th = h_bar / ((gap < 1e-14) ? 1e-14 : gap);
                    th = (th < 1.0) ? th : 1.0;
                    theta = (0.0 < th) ? th : 0.0;
                }
                // effective gradients: b, then eta
#pragma unroll
                for (int d = 0; d < DIM; ++d) {
                    const double gbd = gb[d];
                    gb[d] = phb * gbd;
                    ge[d] = phb * gbd + theta * sh[d];
                }
                bool dry[KM];
#pragma unroll
                for (int k = 0; k < KM; ++k) {
                    double db = 0.0, de = 0.0;
#pragma unroll
                    for (int d = 0; d < DIM; ++d) db += gb[d] * geo[k][DIM + d];
#pragma unroll
                    for (int d = 0; d < DIM; ++d) de += ge[d] * geo[k][DIM + d];
                    const double b_f = b_bar + db;
                    const double hd = (b_bar + h_bar) + de - b_f;
                    const double h_f = (hd < 0.0) ? 0.0 : hd;
                    dry[k] = h_f < pos.eps;
                    rows[B * fst + fso[k]] = b_f;
                    rows[H * fst + fso[k]] = h_f;
                }
                constexpr int CW = (NQ - 2) % 2 == 0 ? 2 : 1;
#pragma unroll 1
                for (int i = 2; i < NQ; i += CW) {
                    double out[CW][KM];
#pragma unroll
                    for (int ii = 0; ii < CW; ++ii) {
                        double g[DIM], q, v[KM], mn, mx;
                        gradient_of(i + ii, g);
                        load(sq, i + ii, q, v);
                        bounds(whole, q, v, mn, mx);
                        double ph = factor(q, mn, mx, g);
                        if (h_bar < pos.eps) ph = 0.0;
                        ph = (phe < ph) ? phe : ph;
#pragma unroll
                        for (int d = 0; d < DIM; ++d) g[d] = theta * ph * g[d];
#pragma unroll
                        for (int k = 0; k < KM; ++k) {
                            double di = 0.0;
#pragma unroll
                            for (int d = 0; d < DIM; ++d) di += g[d] * geo[k][DIM + d];
                            out[ii][k] = dry[k] ? 0.0 : (q + di);
                        }
                    }
#pragma unroll
                    for (int ii = 0; ii < CW; ++ii)
#pragma unroll
                        for (int k = 0; k < KM; ++k) rows[(i + ii) * fst + fso[k]] = out[ii][k];
                }
                return odd;
            };
            if (reconstruct(std::false_type())) reconstruct(std::true_type());
            if (live && ent < n) {
                sv[ent] = vol;
                sv[cst + ent] = rvol;
            }
            continue;
        }
        bool vac = false;
        if constexpr (NQ > 1) {   // VacuumLimiter: minimum depth over the cell and its neighbours
            double q, v[KM], mn, mx;
            load(sq, 1, q, v);
            bounds(false, q, v, mn, mx);
            vac = o.limiter && mn < 1e-2;
        }
        // alpha = min over the components of min(1, (bound - q) / dq)
        // (TVDLimiter, Reconstruction.hpp:67-78).  Rounding is monotone, so the
        // smallest rounded ratio is the smallest ratio rounded: the components
        // only compare ratios, by the sign of num |dq| - room den (p + e is
        // num |dq| exactly, s rounds room den - p: s < e and s > e decide), and
        // each face divides once.  A tie, a non-finite or a vanishing operand
        // sends the cell to the odd path, a second reconstruction: where every cell
        // ties (uniform velocity, hu = h) a step's two stages take 144 us for 99 at
        // 114 k level-2 cells, 421 for 289 at 231 k level-4 ones; the separate
        // kernels take 164 and 628 there.
        double num[KM], den[KM], al[KM], inc[KEEP ? NC : 1][KM];
        bool odd = false;
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            num[k] = vac ? 0.0 : 1.0;
            den[k] = 1.0;
        }
        // chunk after chunk in a loop: the code stays small, every warp fetches it once
        constexpr int UNROLL = KEEP ? NC : 1;
        auto pass = [&](auto least, auto all) {
#pragma unroll UNROLL
            for (int c4 = 0; c4 < NC; c4 += CH) {
                // all of a chunk's loads before its stores: the rows may overlap the state for all the compiler knows
                double q[CH], v[CH][KM], g[CH][DIM], d[CH][KM];
#pragma unroll
                for (int ii = 0; ii < CH; ++ii)
                    if (c4 + ii < NC) load(sw, component(c4 + ii), q[ii], v[ii]);
#pragma unroll
                for (int ii = 0; ii < CH; ++ii) {
                    if (c4 + ii >= NC) continue;
                    gradient(least, all, q[ii], v[ii], g[ii]);
                    if (!all) odd |= !whole && exponent_word(q[ii]) >= 0x7ff00000u;
                    if (!least) {
#pragma unroll
                        for (int e = 0; e < DIM; ++e) g[ii][e] = by_vol.quotient_or(g[ii][e], odd);
                    }
                }
                if (!all && clamped) {
#pragma unroll
                    for (int ii = 0; ii < CH; ++ii)
                        if (c4 + ii < NC) load(swl, component(c4 + ii), q[ii], v[ii]);
                }
#pragma unroll
                for (int ii = 0; ii < CH; ++ii) {
                    if (c4 + ii >= NC) continue;
                    double mn, mx;
                    bounds(all, q[ii], v[ii], mn, mx);
                    const double above = mx - q[ii], below = q[ii] - mn;
#pragma unroll
                    for (int k = 0; k < KM; ++k) {
                        double dd = 0.0;
#pragma unroll
                        for (int e = 0; e < DIM; ++e) dd += g[ii][e] * geo[k][DIM + e];
                        d[ii][k] = dd;
                        const double dq = (q[ii] + dd) - q[ii], ad = fabs(dq);
                        const double room = dq > 0 ? above : below;
                        const double p = num[k] * ad;
                        const double e = __fma_rn(num[k], ad, -p), s = __fma_rn(room, den[k], -p);
                        const bool cand = !(ad < 1e-12), less = s < e, more = s > e;
                        odd |= cand & !less & !more & (num[k] > 0.0);
                        num[k] = cand & less ? room : num[k];
                        den[k] = cand & less ? ad : den[k];
                    }
                }
#pragma unroll
                for (int ii = 0; ii < CH; ++ii) {
                    if (c4 + ii >= NC) continue;
#pragma unroll
                    for (int k = 0; k < KM; ++k) {
                        if constexpr (KEEP) inc[c4 + ii][k] = d[ii][k];
                        else if (own(c4 + ii)) rows[component(c4 + ii) * fst + fso[k]] = d[ii][k];
                    }
                }
            }
        };
        if (clamped || !__all_sync(0xffffffffu, whole)) {
            if (lsq) pass(std::true_type(), std::false_type());
            else pass(std::false_type(), std::false_type());
        } else {
            if (lsq) pass(std::true_type(), std::true_type());
            else pass(std::false_type(), std::true_type());
        }
        odd |= !lsq && !divide;
#pragma unroll
        for (int k = 0; k < KM; ++k) {
            const RnDivisor by_den(den[k], rn_reciprocal(den[k], odd));
            odd |= num[k] > 0.0 && !(num[k] >= 0x1p-800);
            al[k] = by_den.quotient_or(num[k], odd);
        }
        // an odd cell: the gradient and limiter as prep_kernel writes them
        if (odd && !vac) {
#pragma unroll
            for (int k = 0; k < KM; ++k) al[k] = 1.0;
#pragma unroll 1
            for (int ii = 0; ii < NC; ++ii) {
                double q, v[KM], g[DIM], mn, mx;
                plain_gradient(component(ii), g);
                load(sq, component(ii), q, v);
                bounds(false, q, v, mn, mx);
#pragma unroll 1
                for (int k = 0; k < KM; ++k) {
                    double d = 0.0;
#pragma unroll
                    for (int e = 0; e < DIM; ++e) {
                        double w = geo[0][DIM + e];
#pragma unroll
                        for (int kk = 1; kk < KM; ++kk) w = k == kk ? geo[kk][DIM + e] : w;
                        d += g[e] * w;
                    }
                    const double dq = (q + d) - q;
                    const bool pos = dq > 0;
                    const double rr = (pos ? mx : mn) - q;
                    const bool room = pos ? (mx > q) : (mn < q);
                    const bool lim = !(pos ? (rr >= dq) : (rr <= dq));
                    const bool small = fabs(dq) < 1e-12;
                    double a = small ? 1.0 : (room ? 1.0 : 0.0);
                    if (!small && room && lim) a = fmin(1.0, rr / dq);
#pragma unroll
                    for (int kk = 0; kk < KM; ++kk)
                        if (k == kk && a < al[kk]) al[kk] = a;
                }
            }
        }
        if (!o.limiter) {
#pragma unroll
            for (int k = 0; k < KM; ++k) al[k] = 1.0;
        }
        if constexpr (P > 1) {
#pragma unroll
            for (int k = 0; k < KM; ++k)
#pragma unroll
                for (int off = 1; off < P; off <<= 1) {
                    const double a = __shfl_xor_sync(0xffffffffu, al[k], off);
                    al[k] = a < al[k] ? a : al[k];
                }
        }
        if (part == 0 && ent < n) {
            sv[ent] = vol;
            sv[cst + ent] = rvol;
        }
        // face states q + alpha * delta
#pragma unroll UNROLL
        for (int c4 = 0; c4 < NC; c4 += CH) {
            double q[CH], d[CH][KM];
#pragma unroll
            for (int ii = 0; ii < CH; ++ii) {
                if (c4 + ii >= NC) continue;
                q[ii] = sq[component(c4 + ii) * cst + ent];
#pragma unroll
                for (int k = 0; k < KM; ++k) {
                    if constexpr (KEEP) d[ii][k] = inc[c4 + ii][k];
                    else d[ii][k] = rows[component(c4 + ii) * fst + fso[k]];
                }
            }
#pragma unroll
            for (int ii = 0; ii < CH; ++ii) {
                if (c4 + ii >= NC || !own(c4 + ii)) continue;
#pragma unroll
                for (int k = 0; k < KM; ++k) rows[component(c4 + ii) * fst + fso[k]] = q[ii] + al[k] * d[ii][k];
            }
        }
        if (odd) {
#pragma unroll 1
            for (int ii = 0; ii < NC; ++ii) {
                const int i = component(ii);
                double g[DIM];
                plain_gradient(i, g);
                const double q = sq[i * cst + ent];
#pragma unroll
                for (int k = 0; k < KM; ++k) {
                    double d = 0.0;
#pragma unroll
                    for (int e = 0; e < DIM; ++e) d += g[e] * geo[k][DIM + e];
                    rows[i * fst + fso[k]] = q + al[k] * d;
                }
            }
        }
    }
    // the first face's geometry, on its way while the block meets
    FaceGeom fg;
    if (tid < tile.nf) fg.load(m, tid < tile.nown ? tile.f0 + tid : tl.in_faces[tile.in0 + tid - tile.nown]);
    __syncthreads();

    // ---- fluxes (face_kernel): each face's states give way to its contributions
    for (int lf = tid; lf < tile.nf; lf += nt) {
        if (lf != tid) fg.load(m, lf < tile.nown ? tile.f0 + lf : tl.in_faces[tile.in0 + lf - tile.nown]);
        face_contrib<M, N>(m, fg, rows + lf, (size_t)fst, aux, params, t_host, t_dev, stage_frac, dt_step, active,
                           rows + lf, (size_t)fst);
    }
    __syncthreads();

    // ---- sums, / volume and the stage combination (gather_kernel, stage_update),
    // NCG components per thread; consecutive threads, consecutive cells
    // (the largest of 4, 3, 2, 1 that divides them: a 5-component plugin takes one each)
    constexpr int NCG = NQ % 4 == 0 ? 4 : (NQ % 3 == 0 ? 3 : (NQ % 2 == 0 ? 2 : 1)), G = NQ / NCG;
    for (int task = tid; task < n * G; task += nt) {
        const int part = task / n, l = task - part * n;
        const int i0 = part * NCG, c = tile.c0 + l;
        const int I = cell_instance(m, c);
        if (active && !active[I]) continue;
        double acc[NCG], b0[NCG];
        if (mode == MODE_FINAL) {
#pragma unroll
            for (int i = 0; i < NCG; ++i) b0[i] = base[(size_t)(i0 + i) * C + c];
        }
#pragma unroll
        for (int i = 0; i < NCG; ++i) acc[i] = 0.0;
        for (int j = 0; j < K; ++j) {
            const int e = srow[j * cst + l];
            if (e < 0) continue;
            const double* rw = rows + i0 * fst + (e >> 1);
            const bool isL = e & 1;   // the cell is the face's support[0]
#pragma unroll
            for (int i = 0; i < NCG; ++i) {
                acc[i] -= rw[(isL ? i : NQ + i) * fst];
                const double fl = rw[(2 * NQ + i) * fst];
                acc[i] += isL ? -fl : fl;
            }
        }
        const double v = sv[l];
        if (v > 1e-15) {
            const RnDivisor by_vol(v, sv[cst + l]);
            bool odd = false;
            double q[NCG];
#pragma unroll
            for (int i = 0; i < NCG; ++i) q[i] = by_vol.quotient_or(acc[i], odd);
            if (odd) {
#pragma unroll
                for (int i = 0; i < NCG; ++i) q[i] = acc[i] / v;
            }
#pragma unroll
            for (int i = 0; i < NCG; ++i) acc[i] = q[i];
        }
        const double hs = m.cell_inst && dt_step ? dt_step[I] / sc.dt_div : h0;
#pragma unroll
        for (int i = 0; i < NCG; ++i) {
            const size_t id = (size_t)(i0 + i) * C + c;
            if (mode == MODE_RHS) {
                x_out[id] = acc[i];
                continue;
            }
            const double w = sw[(i0 + i) * cst + l];
            if (mode == MODE_FINAL) base[id] = sc.state * w + hs * acc[i] + sc.start * b0[i];
            else x_out[id] = w + hs * acc[i];   // MODE_FIRST, MODE_MID, MODE_EULER
        }
    }
}

}  // namespace zsme
