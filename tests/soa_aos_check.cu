// The state store (launch_soa_to_aos) for component counts on both sides of its
// shared-memory rows, ragged cell counts and a cell range inside the arrays,
// against the plain transposition.
#include <cstdio>
#include <vector>

#include "model_prelude.h"
#include "prepared_mesh.h"
#include "step_kernels.cuh"

int main() {
    long checked = 0, wrong = 0;
    for (int nq : {1, 12, 31, 32, 33, 47, 48, 60, 100})
        for (int cn : {1, 128, 1000}) {
            const int c0 = 37, C = c0 + cn + 5;
            std::vector<double> soa((size_t)nq * C), aos((size_t)nq * cn, -1.0);
            std::vector<int> old(C, -1);
            for (size_t i = 0; i < soa.size(); ++i) soa[i] = (double)i;
            for (int r = 0; r < cn; ++r) old[c0 + r] = cn - 1 - r;   // a permutation
            double *d_soa = nullptr, *d_aos = nullptr;
            int* d_old = nullptr;
            cudaMalloc((void**)&d_soa, soa.size() * sizeof(double));
            cudaMalloc((void**)&d_aos, aos.size() * sizeof(double));
            cudaMalloc((void**)&d_old, old.size() * sizeof(int));
            cudaMemcpy(d_soa, soa.data(), soa.size() * sizeof(double), cudaMemcpyHostToDevice);
            cudaMemcpy(d_aos, aos.data(), aos.size() * sizeof(double), cudaMemcpyHostToDevice);
            cudaMemcpy(d_old, old.data(), old.size() * sizeof(int), cudaMemcpyHostToDevice);
            zsme::launch_soa_to_aos(d_soa, d_aos, d_old, c0, cn, C, nq, nullptr);
            const cudaError_t e = cudaGetLastError(), s = cudaDeviceSynchronize();
            if (e != cudaSuccess || s != cudaSuccess) printf("%d components: %s\n", nq, cudaGetErrorString(e ? e : s));
            cudaMemcpy(aos.data(), d_aos, aos.size() * sizeof(double), cudaMemcpyDeviceToHost);
            for (int r = 0; r < cn; ++r)
                for (int i = 0; i < nq; ++i)
                    wrong += aos[(size_t)(cn - 1 - r) * nq + i] != soa[(size_t)i * C + c0 + r];
            checked += (long)nq * cn;
            cudaFree(d_soa);
            cudaFree(d_aos);
            cudaFree(d_old);
        }
    printf("checked %ld wrong %ld\n", checked, wrong);
    return wrong != 0;
}
