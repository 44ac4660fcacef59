// div_by (device/device.cuh): largest error in ulp and largest difference from
// the division operator over random operands, for reciprocals up to 4 ulp off
// (host) and, compiled by nvcc, for the device's 1.0 / b and rsqrt(d).
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <random>
#include <vector>

#include "device.cuh"

struct Pair {
    double a, d;                              // d: the divisor, or its square
};

static Pair draw(std::mt19937_64 &rng) {
    auto value = [&](int range, bool positive) {
        const double m = 1.0 + double(rng() >> 12) * 0x1p-52;
        const int e = int(rng() % (2 * range + 1)) - range;
        return std::ldexp(!positive && (rng() & 1) ? -m : m, e);
    };
    return {value(300, false), value(200, true)};
}

struct Worst {
    double ulp = 0.0;
    long long differ = 0, apart = 0, n = 0;
    void add(double a, double b, double q) {
        const long double rest = fmal(-(long double)q, (long double)b, (long double)a);
        int e;
        std::frexp(q, &e);
        const double u = double(std::fabs(rest / b)) * std::ldexp(1.0, 53 - e);
        if (u > ulp) ulp = u;
        const double t = a / b;
        differ += q != t;
        apart += q != t && q != std::nextafter(t, INFINITY) && q != std::nextafter(t, -INFINITY);
        ++n;
    }
    void print(const char *what) const {
        std::printf("%s max_ulp_excess %.3e differ %lld apart %lld of %lld\n", what, ulp - 0.5, differ, apart, n);
    }
};

#ifdef __CUDACC__
__global__ void quotients(const Pair *p, int n, double *by_inverse, double *root, double *by_rsqrt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    by_inverse[i] = htf::div_by(p[i].a, p[i].d, 1.0 / p[i].d);
    root[i] = sqrt(p[i].d);
    by_rsqrt[i] = htf::div_by(p[i].a, root[i], rsqrt(p[i].d));
}
#endif

int main() {
    std::mt19937_64 rng(7);
    const int n = 1 << 20;
    std::vector<Pair> p(n);
    for (auto &x : p) x = draw(rng);
#ifdef __CUDACC__
    Pair *dp;
    double *dq;
    std::vector<double> q(3 * size_t(n));
    if (cudaMalloc(&dp, n * sizeof(Pair)) != cudaSuccess || cudaMalloc(&dq, q.size() * sizeof(double)) != cudaSuccess)
        return 1;
    cudaMemcpy(dp, p.data(), n * sizeof(Pair), cudaMemcpyHostToDevice);
    quotients<<<n / 256, 256>>>(dp, n, dq, dq + n, dq + 2 * size_t(n));
    if (cudaMemcpy(q.data(), dq, q.size() * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    Worst inverse, root;
    for (int i = 0; i < n; ++i) {
        inverse.add(p[i].a, p[i].d, q[i]);
        root.add(p[i].a, q[n + i], q[2 * size_t(n) + i]);
    }
    inverse.print("device 1/b");
    root.print("device rsqrt");
    cudaFree(dp);
    cudaFree(dq);
#else
    for (int off = -4; off <= 4; ++off) {
        Worst w;
        for (auto &x : p) {
            double r = 1.0 / x.d;
            for (int k = 0; k < std::abs(off); ++k) r = std::nextafter(r, off > 0 ? INFINITY : -INFINITY);
            w.add(x.a, x.d, htf::div_by(x.a, x.d, r));
        }
        char what[16];
        std::snprintf(what, sizeof what, "host %+d", off);
        w.print(what);
    }
#endif
    return 0;
}
