// Device harness of csrc/exactdiv.cuh (test only): each short quotient against the division, bit for bit.
#include <cmath>
#include <cstdint>

#include "../../pyocean_b200/csrc/exactdiv.cuh"

namespace {

__device__ bool same(double x, double y)
{
    return __double_as_longlong(x) == __double_as_longlong(y) || (x != x && y != y);
}

// wrong[0] quotient through shared_recip, [1] quot_rn from recip_newton, [2] quot_rn from 1.0 / b, [3] x / 3, [4] x / 6
__global__ void check(const double* a, const double* b, long long n, unsigned long long* wrong, double* example)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const double x = a[t], y = b[t], q = x / y;
    auto mid = [](double v, double e) { return fabs(v) >= 1.0 / e && fabs(v) <= e; };
    const bool in = y > 0.0 && mid(y, 0x1p399) && (x == 0.0 || mid(x, 0x1p499));
    bool bad[5];
    bad[0] = !same(po::quotient(x, y, po::shared_recip(y)), q);
    bad[1] = in && po::near_two_bits(y) < po::NEAR_TWO && !same(po::quot_rn(x, y, po::recip_newton(y)), q);
    bad[2] = in && !same(po::quot_rn(x, y, 1.0 / y), q);
    bad[3] = !same(po::div3_exact(x), x / 3.0);
    bad[4] = !same(po::div6_exact(x), x / 6.0);
    for (int m = 0; m < 5; ++m)
        if (bad[m]) {
            atomicAdd(wrong + m, 1ull);
            example[2 * m] = x;
            example[2 * m + 1] = y;
        }
}

}  // namespace

// a, b: n numbers on the device; wrong: 5 counters (cleared), example: 5 pairs, on the device.
extern "C" int check_quotients(const double* a, const double* b, long long n, unsigned long long* wrong, double* example)
{
    check<<<(unsigned)((n + 255) / 256), 256>>>(a, b, n, wrong, example);
    return (int)cudaDeviceSynchronize();
}
