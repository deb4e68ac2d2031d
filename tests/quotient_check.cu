// Self-check of the FP64 kernels' quotient with separately tested operands
// (mquo, mout, mpos, mrcpp in multiphase-code_b200/csrc/hp_kernels.cuh)
// against the hardware IEEE division: dividends of the magnitudes given on
// the command line (2^[lo, hi), either sign, and both zeros), positive
// divisors over 2^[-100, 101), random and extreme mantissas.  Prints
// "pairs N flagged F mismatches M wrong W": M unflagged pairs whose quotient
// differs in any bit, W pairs inside the tested ranges that were flagged.
// Built and run by tests/test_quotient.py.
#include <cstdint>
#include <cstdio>
#define HP_NS v_check
#define HP_R double
#define HP_LSQ_TABLE 1
#include "../multiphase-code_b200/csrc/hp_kernels.cuh"
using namespace hp::v_check;

__device__ unsigned long long g_out[4];

__device__ double with_exponent(unsigned long long r, int e, int mode) {
    unsigned long long man = r & 0xfffffffffffffull;
    if (mode == 1) man = 0xfffffffffffffull;
    if (mode == 2) man = 0;
    if (mode == 3) man = 0xfffffffffffffull ^ (r & 0xffull);
    return __longlong_as_double((long long)(((r >> 63) << 63) | ((unsigned long long)(e + 1023) << 52) | man));
}
// test: 0 the dividend's own test (mout), 1 the test of a positive value
// (mpos), 2 none (products whose factors were tested)
__global__ void k_check(unsigned long long seed, int iters, int lo, int hi, int test) {
    unsigned long long s = seed ^ (0x9e3779b97f4a7c15ull * (blockIdx.x * blockDim.x + threadIdx.x + 1));
    unsigned long long n[4] = {0, 0, 0, 0};
    auto next = [&] { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; };
    for (int it = 0; it < iters; it++) {
        const unsigned long long r1 = next(), r2 = next() & ~(1ull << 63), r3 = next();
        const int ea = lo + (int)(r3 % (unsigned)(hi - lo)), eb = (int)((r3 >> 16) % 201) - 100;
        double a = with_exponent(r1, ea, (r3 >> 32) % 8 == 0 ? (int)((r3 >> 40) % 4) : 0);
        const double b = with_exponent(r2, eb, (r3 >> 44) % 8 == 0 ? (int)((r3 >> 50) % 4) : 0);
        if ((r3 >> 56) % 32 == 0) a = copysign(0.0, a);
        unsigned bad = 0;
        if (test == 0) mout<1>(a, bad);
        if (test == 1) mpos<1>(a, bad);
        const bool in = test == 2 || (a == 0.0 ? test == 0 : ea >= -800 && ea < 801 && (test == 0 || a > 0.0));
        const double rb = mrcpp<1>(b, bad);
        const double q = mquo<1>(a, b, rb);
        n[0]++;
        if (bad) { n[1]++; n[3] += in; continue; }
        n[2] += __double_as_longlong(q) != __double_as_longlong(a / b);
    }
    for (int k = 0; k < 4; k++) atomicAdd(&g_out[k], n[k]);
}
int main(int argc, char** argv) {
    if (argc != 4) return 2;
    k_check<<<148 * 4, 256>>>(7654321ull, 512, atoi(argv[1]), atoi(argv[2]), atoi(argv[3]));
    unsigned long long n[4];
    if (cudaDeviceSynchronize() != cudaSuccess || cudaMemcpyFromSymbol(n, g_out, sizeof n) != cudaSuccess) return 2;
    printf("pairs %llu flagged %llu mismatches %llu wrong %llu\n", n[0], n[1], n[2], n[3]);
    return 0;
}
