// The FP64 arithmetic on the integer pipes (csrc/euler_device.cuh) against the
// FP64 unit, on the GPU and so with its own FP32 seeds:
//   mul_rn_alu, rcp_rn_alu, add_alu  the bits of __dmul_rn, __drcp_rn and (both
//                                    operands >= 0) __dadd_rn, NaN against NaN
//   mul_alu   as far from the exact product as __dmul_rn (its ties go away
//             from zero), the same bits outside [2^-255, 2^257)
//   rcp_alu   distance from 1/x in ulps, from the exact residual 1 - x r
//   sqrt_alu  distance from sqrt(x) in ulps, from the exact residual x - s s
// and rcp_alu, sqrt_alu outside [2^-255, 2^257) against rcp_faithful and
// sqrt_faithful.  Test harness, built and run by
// tests/test_gpu_integer_arithmetic.py; prints one JSON line of mismatch
// counts and largest distances.
#include "euler_device.cuh"

#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

namespace {

enum { kMulRn, kRcpRn, kAdd, kMul, kRcpOut, kSqrtOut, kCounts };
enum { kRcpUlps, kSqrtUlps, kMaxima };

__device__ bool same(double a, double b)
{
    return __double_as_longlong(a) == __double_as_longlong(b) || (a != a && b != b);
}

// Magnitude in [2^-255, 2^257).
__device__ bool inside(double x) { return fabs(x) >= 0x1p-255 && fabs(x) < 0x1p257; }

// Spacing of the doubles next to |x|, on the side of the exact value (rest:
// exact minus x).
__device__ double ulp(double x, double rest)
{
    long long const b = __double_as_longlong(fabs(x)) - (x < 0.0 ? rest > 0.0 : rest < 0.0);
    return __longlong_as_double(b & 0x7ff0000000000000LL) * 0x1p-52;
}

__global__ void check_kernel(const double* a, const double* b, int n, unsigned long long* bad, unsigned long long* most)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) {
        return;
    }
    double const x = a[i], y = b[i];
    double const prod = __dmul_rn(x, y);
    if (!same(eulr::mul_rn_alu(x, y), prod)) {
        atomicAdd(bad + kMulRn, 1ull);
    }
    double const m = eulr::mul_alu(x, y);
    if (!same(m, prod) && !(inside(x) && inside(y) && fabs(__fma_rn(x, y, -m)) == fabs(__fma_rn(x, y, -prod)))) {
        atomicAdd(bad + kMul, 1ull);
    }
    if (!same(eulr::add_alu(fabs(x), fabs(y)), __dadd_rn(fabs(x), fabs(y)))) {
        atomicAdd(bad + kAdd, 1ull);
    }
    if (!same(eulr::rcp_rn_alu(x), __drcp_rn(x))) {
        atomicAdd(bad + kRcpRn, 1ull);
    }
    double const r = eulr::rcp_alu(x);
    if (inside(x)) {
        double const rest = __fma_rn(-x, r, 1.0) / x;
        double const e = fabs(rest) / ulp(r, rest);
        atomicMax(most + kRcpUlps, static_cast<unsigned long long>(__double_as_longlong(e)));
    } else if (!same(r, eulr::rcp_faithful(x))) {
        atomicAdd(bad + kRcpOut, 1ull);
    }
    double const s = eulr::sqrt_alu(x);
    if (inside(x) && x > 0.0) {
        double const rest = __fma_rn(-s, s, x) / (2.0 * s);
        double const e = fabs(rest) / ulp(s, rest);
        atomicMax(most + kSqrtUlps, static_cast<unsigned long long>(__double_as_longlong(e)));
    } else if (!same(s, eulr::sqrt_faithful(x))) {
        atomicAdd(bad + kSqrtOut, 1ull);
    }
}

double from_bits(unsigned long long u)
{
    double d;
    std::memcpy(&d, &u, sizeof d);
    return d;
}

} // namespace

int main()
{
    std::vector<double> va, vb;
    unsigned long long state = 0x2545f4914f6cdd1dull;
    auto next = [&state]() {
        state ^= state << 13;
        state ^= state >> 7;
        state ^= state << 17;
        return state;
    };
    auto add = [&](double x, double y) {
        va.push_back(x);
        vb.push_back(y);
    };
    // a significand of 53 bits: any, near one, near two, of few bits
    auto significand = [&](int kind) {
        unsigned long long const u = next();
        switch (kind) {
        case 0: return 1.0 + static_cast<double>(u & 0xffull) * 0x1p-52;
        case 1: return 2.0 - static_cast<double>(1 + (u & 0xffull)) * 0x1p-52;
        case 2: return 1.0 + static_cast<double>(u >> 59) * 0x1p-5;
        default: return 1.0 + static_cast<double>(u >> 12) * 0x1p-52;
        }
    };
    for (int i = 0; i < (1 << 23); ++i) {
        unsigned long long const u = next();
        double const sx = u & 1 ? -1.0 : 1.0, sy = u & 2 ? -1.0 : 1.0;
        int const ex = static_cast<int>((u >> 8) % 540) - 270; // inside and a little outside the window
        switch (i & 7) {
        case 0: { // products on a tie: odd significands of 27 bits
            double const p = static_cast<double>((1u << 26) | ((u >> 32) & 0x3fffffeu) | 1u);
            double const q = static_cast<double>((1u << 26) | (next() & 0x3fffffeu) | 1u);
            add(sx * std::ldexp(p, ex), sy * std::ldexp(q, -ex));
            break;
        }
        case 1:
        case 2: { // sums of exponents 0 to 34 apart, every other with a tie or next to one in what is shifted out
            int const gap = static_cast<int>((u >> 20) % 35);
            unsigned long long m = (next() >> 12) | (1ull << 52);
            if (gap > 0 && (u & 4)) {
                m = (m >> gap << gap) + (1ull << (gap - 1)) + ((u >> 40) % 3) - 1;
            }
            add(sx * std::ldexp(significand(static_cast<int>((u >> 50) & 3)), ex),
                sy * std::ldexp(static_cast<double>(m), ex - gap - 52));
            break;
        }
        case 3: // any bits
            add(from_bits(next()), from_bits(next()));
            break;
        default:
            add(sx * std::ldexp(significand(static_cast<int>((u >> 50) & 3)), ex),
                sy * std::ldexp(significand(static_cast<int>((u >> 52) & 3)), static_cast<int>((u >> 20) % 540) - 270));
        }
    }
    // every binade, its edges and its middle; special values; pairwise around the window's ends
    for (int e = -1074; e <= 1023; ++e) {
        add(std::ldexp(1.0, e), std::ldexp(1.0, -e / 2));
        add(std::ldexp(std::nextafter(2.0, 1.0), e), std::ldexp(1.5, e / 3));
        add(std::ldexp(std::nextafter(1.0, 2.0), e), std::ldexp(std::nextafter(1.0, 2.0), e));
    }
    double const inf = HUGE_VAL;
    std::vector<double> special = {0.0, 1.0, 3.0, 0x1p-255, 0x1p257, std::nextafter(0x1p-255, 0.0),
                                   std::nextafter(0x1p-255, 1.0), std::nextafter(0x1p257, 0.0),
                                   std::nextafter(0x1p257, inf), 0x1p-1022, 0x1p-1074, 0x1.fffffffffffffp1023, inf,
                                   std::nan(""), 0x1.fffffffffffffp255, 0x1.0000000000001p-254, 0x1.6a09e667f3bcdp0};
    size_t const half = special.size();
    for (size_t i = 0; i < half; ++i) {
        special.push_back(-special[i]);
    }
    for (double x : special) {
        for (double y : special) {
            add(x, y);
        }
    }
    int const n = static_cast<int>(va.size());
    double *da = nullptr, *db = nullptr;
    unsigned long long* dout = nullptr;
    if (cudaMalloc(&da, sizeof(double) * n) != cudaSuccess || cudaMalloc(&db, sizeof(double) * n) != cudaSuccess ||
        cudaMalloc(&dout, sizeof(unsigned long long) * (kCounts + kMaxima)) != cudaSuccess) {
        std::printf("cudaMalloc failed\n");
        return 1;
    }
    cudaMemcpy(da, va.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemcpy(db, vb.data(), sizeof(double) * n, cudaMemcpyHostToDevice);
    cudaMemset(dout, 0, sizeof(unsigned long long) * (kCounts + kMaxima));
    check_kernel<<<(n + 255) / 256, 256>>>(da, db, n, dout, dout + kCounts);
    cudaError_t const err = cudaDeviceSynchronize();
    if (err != cudaSuccess) {
        std::printf("kernel failed: %s\n", cudaGetErrorString(err));
        return 1;
    }
    unsigned long long out[kCounts + kMaxima];
    cudaMemcpy(out, dout, sizeof out, cudaMemcpyDeviceToHost);
    cudaFree(da);
    cudaFree(db);
    cudaFree(dout);
    std::printf("{\"n\": %d, \"mul_rn\": %llu, \"rcp_rn\": %llu, \"add\": %llu, \"mul\": %llu, \"rcp_outside\": %llu, "
                "\"sqrt_outside\": %llu, \"rcp_ulps\": %.7f, \"sqrt_ulps\": %.7f}\n",
                n, out[kMulRn], out[kRcpRn], out[kAdd], out[kMul], out[kRcpOut], out[kSqrtOut],
                from_bits(out[kCounts + kRcpUlps]), from_bits(out[kCounts + kSqrtUlps]));
    return 0;
}
