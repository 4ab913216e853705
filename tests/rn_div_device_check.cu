// The device forms of rn_div.h (whose reciprocal starts from the hardware's
// approximation, where the host's starts from a float quotient) against the
// device's own division, bit for bit: significands of all ones, of few bits and
// random ones, over the fast exponent range, at its ends and beyond it.
#include <cstdio>

#include "rn_div.h"

using namespace zsme;

__device__ unsigned long long next(unsigned long long& s) {
    s = s * 6364136223846793005ull + 1442695040888963407ull;
    unsigned long long z = s;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}
__device__ double make(unsigned long long m, int e, unsigned long long sign) {
    return __longlong_as_double((long long)((m & ((1ull << 52) - 1)) | ((unsigned long long)(e + 1023) << 52) |
                                            (sign << 63)));
}
__device__ bool same(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}
__device__ unsigned long long significand(unsigned long long& s) {
    const unsigned long long r = next(s), kind = next(s) % 6;
    if (kind == 0) return ~0ull - (r & 63);          // all ones and its neighbours
    if (kind == 1) return r & 63;                    // one and its neighbours
    if (kind == 2) return (r | 0xffffffffull);       // a lower word of all ones
    if (kind == 3) return r << 32;                   // a lower word of zeros
    return r;
}

__global__ void check(unsigned long long seed, int per_thread, unsigned long long* wrong, unsigned long long* odds) {
    unsigned long long s = seed + (blockIdx.x * 256ull + threadIdx.x) * 0x9e3779b97f4a7c15ull, bad = 0, odd_n = 0;
    for (int i = 0; i < per_thread; ++i) {
        const int where = (int)(next(s) % 8);
        int e = (int)(next(s) % 200) - 100;                              // the fast range
        if (where == 0) e = next(s) % 2 ? -100 : 99;                     // its ends
        if (where == 1) e = (int)(next(s) % 2047) - 1023;                // any, zeros and subnormals too
        const double b = make(significand(s), e, next(s) & 1);
        int ea = (int)(next(s) % 1800) - 900;
        if (where == 2) ea = (int)(next(s) % 2048) - 1023;               // any, infinities and NaN too
        double a = make(significand(s), ea, next(s) & 1);
        if (where == 3 && next(s) % 4 == 0) a = next(s) & 1 ? -0.0 : 0.0;
        const double t = a / b;
        bool odd = false;
        const double y = rn_reciprocal(b, odd);
        odd_n += odd;
        bad += !odd && !same(y, 1.0 / b);
        const RnDivisor by(b);
        bad += !same(by.quotient(a), t);
        bool o = false;
        const double q = by.signed_quotient_or(a, o);
        bad += !o && !same(q, t);
        if (!odd) {                                                      // from the reciprocal formed here
            bool o2 = false;
            const double q2 = RnDivisor(b, y).signed_quotient_or(a, o2);
            bad += !o2 && !same(q2, t);
        }
        if (b > 0.0 && __double_as_longlong(a) != (long long)0x8000000000000000ull) {
            o = false;
            const double p = by.quotient_or(a, o);
            bad += !o && !same(p, t);
        }
    }
    if (bad) atomicAdd(wrong, bad);
    atomicAdd(odds, odd_n);
}

int main() {
    unsigned long long* n = nullptr;
    if (cudaMallocManaged(&n, 2 * sizeof *n) != cudaSuccess) return printf("no device memory\n"), 1;
    n[0] = n[1] = 0;
    const int blocks = 1024, per_thread = 256;
    check<<<blocks, 256>>>(12345, per_thread, n, n + 1);
    const cudaError_t e = cudaDeviceSynchronize();
    if (e != cudaSuccess) return printf("%s\n", cudaGetErrorString(e)), 1;
    printf("checked %lld odd %llu wrong %llu\n", (long long)blocks * 256 * per_thread, n[1], n[0]);
    return n[0] != 0;
}
