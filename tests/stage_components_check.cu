// stage_kernel for component counts that no shipped plugin has: a plugin whose
// components do not act on one another beyond the limiter's minimum, and whose
// components from the fifth on repeat the third and fourth, has to give the
// four-component plugin's right-hand side for each of them, bit for bit, with 1,
// 2 and 4 threads per cell.  Argument: a mesh file (tests/test_gpu_plugin_components.py).
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "model_prelude.h"
#include "prepared_mesh.h"
#include "step_kernels.cuh"
#include "face_kernels.cuh"
#include "stage_kernel.cuh"

namespace zsme {
int set_error(int code, const std::string& msg) {
    printf("error %d: %s\n", code, msg.c_str());
    return code;
}
}  // namespace zsme
using namespace zsme;

template <int N>
struct Toy {
    static constexpr int n_dof_q = N, n_dof_qaux = 1, n_parameters = 1, dimension = 2;
    template <class... A>
    ZSME_HD static SimpleArray<double, 1> update_aux_variables(A...) { return {{0.0}}; }
    ZSME_HD static SimpleArray<double, N> boundary_conditions(int, const double* q, const double*, const double*,
                                                              const double*, const double*, double, double) {
        SimpleArray<double, N> r{};
        for (int i = 0; i < N; ++i) r[i] = 0.75 * q[i];
        return r;
    }
};
template <int N>
struct ToyNumerics {
    ZSME_HD static SimpleArray<double, N> numerical_flux(const double* l, const double* r, const double*,
                                                         const double*, const double*, const double* n) {
        const double un = n[0] + 0.5 * n[1];
        SimpleArray<double, N> f{};
        for (int i = 0; i < N; ++i) f[i] = un * (un > 0.0 ? l[i] : r[i]);
        return f;
    }
    ZSME_HD static SimpleArray<double, 2 * N> numerical_fluctuations(const double* l, const double* r, const double*,
                                                                     const double*, const double*, const double*) {
        SimpleArray<double, 2 * N> f{};
        for (int i = 0; i < N; ++i) {
            f[i] = 0.25 * (l[i] - r[i]);
            f[N + i] = 0.125 * (r[i] - l[i]);
        }
        return f;
    }
};

template <class T>
static T* upload(const std::vector<T>& v) {
    T* p = nullptr;
    cudaMalloc((void**)&p, std::max<size_t>(1, v.size()) * sizeof(T));
    cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice);
    return p;
}

struct Tables {
    MeshDev md;
    Opts opts;
    StageTilesDev tl;
    int n, max_faces, max_local;
};

static int same_as(int i) { return i < 4 ? i : 2 + i % 2; }

template <int N, int P, int KM>
static std::vector<double> rhs(Tables t, const std::vector<double>& q4) {
    const int C = t.md.C;
    std::vector<double> q((size_t)N * C), out((size_t)N * C, -1.0);
    for (int i = 0; i < N; ++i)
        memcpy(&q[(size_t)i * C], &q4[(size_t)same_as(i) * C], C * sizeof(double));
    t.tl.fst = StageShape<N, P>::row(t.max_faces + 1);
    t.tl.cst = StageShape<N, P>::row(t.max_local);
    const size_t smem = stage_smem_doubles<N>(t.tl.fst, t.tl.cst) * sizeof(double);
    double *x = upload(q), *y = upload(out), *aux = upload(std::vector<double>(C, 0.0));
    double* par = upload(std::vector<double>(1, 0.0));
    auto k = stage_kernel<Toy<N>, ToyNumerics<N>, P, KM, 256, 1>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    k<<<t.n, 256, smem>>>(t.md, t.opts, t.tl, StageWeights{0.0, 0.0, 1.0}, StagePositivity{0, 0.0}, x, aux, par, 0.0,
                          nullptr, 0.0, nullptr, nullptr, MODE_RHS, y, nullptr);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) printf("%d components: %s\n", N, cudaGetErrorString(e));
    cudaMemcpy(out.data(), y, out.size() * sizeof(double), cudaMemcpyDeviceToHost);
    for (double* p : {x, y, aux, par}) cudaFree(p);
    return out;
}

static long checks = 0, wrong = 0;

template <int N, int P, int KM>
static void compare(const Tables& t, const std::vector<double>& q4, const std::vector<double>& want) {
    const std::vector<double> got = rhs<N, P, KM>(t, q4);
    const int C = t.md.C;
    long bad = 0;
    for (int i = 0; i < N; ++i)
        bad += memcmp(&got[(size_t)i * C], &want[(size_t)same_as(i) * C], C * sizeof(double)) != 0;
    if (bad) printf("%d components, %d threads per cell, K %d: %ld rows differ\n", N, P, t.md.K, bad);
    checks += N;
    wrong += bad;
}
template <int N, int KM>
static void compare_parts(const Tables& t, const std::vector<double>& q4, const std::vector<double>& want) {
    compare<N, 1, KM>(t, q4, want);
    compare<N, 2, KM>(t, q4, want);
    compare<N, 4, KM>(t, q4, want);
}
template <int KM>
static void compare_all(const Tables& t, const std::vector<double>& q4) {
    const std::vector<double> want = rhs<4, 1, KM>(t, q4);
    compare_parts<5, KM>(t, q4, want);
    compare_parts<9, KM>(t, q4, want);
    compare_parts<13, KM>(t, q4, want);
    compare_parts<14, KM>(t, q4, want);
}

int main(int argc, char** argv) {
    FILE* f = argc > 1 ? fopen(argv[1], "rb") : nullptr;
    int h[4];
    if (!f || fread(h, sizeof(int), 4, f) != 4) return printf("no mesh file\n"), 1;
    const int C = h[1], F = h[2], K = h[3];
    std::vector<double> xc(2 * (size_t)C), vol(C), xf(2 * (size_t)F), nf(2 * (size_t)F);
    std::vector<int> cf((size_t)K * C), fcells(2 * (size_t)F), bc(F);
    auto get = [&](auto& v) { return fread(v.data(), sizeof(v[0]), v.size(), f) == v.size(); };
    if (!(get(xc) && get(vol) && get(cf) && get(fcells) && get(xf) && get(nf) && get(bc)))
        return printf("short mesh file\n"), 1;
    fclose(f);
    const zsme_mesh m{h[0], C, F, K, xc.data(), vol.data(), cf.data(), fcells.data(), xf.data(), nf.data(), bc.data(),
                      nullptr};
    std::vector<double> q4(4 * (size_t)C);
    uint64_t s = 1;
    for (size_t i = 0; i < q4.size(); ++i) {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        q4[i] = 1.0 + (double)(s >> 11) * 0x1p-54;
    }
    for (int lsq = 0; lsq < 2; ++lsq) {
        PreparedMesh p;
        if (prepare_mesh(m, p, lsq)) return 1;
        FaceTiles t;
        StageTiles st;
        if (build_tiles(p, 96, t) || build_stage_tiles(p, t, 2, !lsq, st) || !st.fits) return 1;
        std::vector<StageTile> tiles(t.n);
        for (int b = 0; b < t.n; ++b) {
            const int n = t.cell_off[b + 1] - t.cell_off[b], own = t.face_off[b + 1] - t.face_off[b];
            tiles[b] = StageTile{t.cell_off[b], n, n + st.ext_off[b + 1] - st.ext_off[b], n + st.ring1[b],
                                 st.ext_off[b], st.ent_off[b], t.face_off[b], own,
                                 t.in_off[b], own + t.in_off[b + 1] - t.in_off[b], st.gho_off[b],
                                 st.gho_off[b + 1] - st.gho_off[b]};
        }
        for (auto* v : {&st.ext_cell, &st.gho_cell, &st.gho_face})
            if (v->empty()) v->push_back(0);
        Tables d;
        d.md = MeshDev{C, K, upload(p.slot_nbr), upload(p.slot_meta), upload(p.slot_face), upload(p.slot_dx),
                       upload(p.slot_w), upload(p.vol), upload(p.rc), upload(p.order), upload(p.fn), upload(p.farea),
                       upload(p.fc), upload(p.fnr), F, upload(p.face_L), upload(p.face_R), upload(p.face_bc), nullptr,
                       nullptr, 1};
        d.opts = Opts{2, 1, lsq, 2, 0};
        const int entries = st.ent_off.back();
        double* geo = upload(std::vector<double>((size_t)(4 * K + 2) * entries));
        d.tl = StageTilesDev{upload(tiles), upload(t.in_faces), upload(t.ord_lf), upload(st.ext_cell),
                             upload(st.gho_cell), upload(st.gho_face), upload(st.loc), geo, entries, 0, 0};
        d.n = t.n;
        d.max_faces = t.max_faces;
        d.max_local = st.max_local;
        stage_entries_kernel<<<t.n, 128>>>(d.md, d.tl.tile, d.tl.ext_cell, d.tl.loc, entries, 2, lsq, geo);
        if (K == 3) compare_all<3>(d, q4);
        else compare_all<4>(d, q4);
    }
    printf("checked %ld wrong %ld\n", checks, wrong);
    return wrong != 0;
}
