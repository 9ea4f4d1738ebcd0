// Accuracy of rcp_cubic and rsqrt_cubic (gkm-dns_b200/csrc/gks_device.cuh)
// against the correctly rounded reciprocal and 1/sqrt(x) in 64-bit mantissas,
// over random mantissas in every binade from 2^-1021 to 2^1021, the edges
// of the binades, and the special values.  Prints the largest errors in units
// of the last place and exits 0, or names what is out of bounds and exits 1.
#include "gks_device.cuh"

#include <cmath>
#include <cstdio>
#include <limits>
#include <random>
#include <vector>

__global__ void k_recip(const double *x, double *r, double *q, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    r[i] = gks::rcp_cubic(x[i]);
    q[i] = gks::rsqrt_cubic(x[i]);
}

static double ulps(double got, long double want)
{
    const double w = std::fabs((double)want);
    const double ulp = std::nextafter(w, std::numeric_limits<double>::infinity()) - w;
    return (double)(std::fabs((long double)got - want) / ulp);
}

int main()
{
    std::vector<double> x;
    std::mt19937_64 gen(1);
    std::uniform_real_distribution<double> mant(1.0, 2.0);
    for (int e = -1021; e <= 1020; ++e) {
        for (double m : {1.0, 1.0 + 0x1p-52, 1.0 + 0x1p-51, 1.5, 2.0 - 0x1p-51, 2.0 - 0x1p-52}) x.push_back(std::ldexp(m, e));
        for (int i = 0; i < 2000; ++i) x.push_back(std::ldexp(mant(gen), e));
    }
    const int normal = (int)x.size();
    const double inf = std::numeric_limits<double>::infinity();
    for (double s : {0.0, -0.0, inf, -inf, std::nan("")}) x.push_back(s);
    const int n = (int)x.size();
    double *dx, *dr, *dq;
    if (cudaMalloc(&dx, n * sizeof(double)) != cudaSuccess || cudaMalloc(&dr, n * sizeof(double)) != cudaSuccess ||
        cudaMalloc(&dq, n * sizeof(double)) != cudaSuccess)
        return 2;
    cudaMemcpy(dx, x.data(), n * sizeof(double), cudaMemcpyHostToDevice);
    k_recip<<<(n + 255) / 256, 256>>>(dx, dr, dq, n);
    std::vector<double> r(n), q(n);
    cudaMemcpy(r.data(), dr, n * sizeof(double), cudaMemcpyDeviceToHost);
    if (cudaMemcpy(q.data(), dq, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess) return 2;
    double er = 0.0, eq = 0.0;
    int off = 0;
    for (int i = 0; i < normal; ++i) {
        er = std::fmax(er, ulps(r[i], 1.0L / (long double)x[i]));
        eq = std::fmax(eq, ulps(q[i], 1.0L / std::sqrt((long double)x[i])));
        off += r[i] != 1.0 / x[i];
    }
    std::printf("rcp_cubic %.4f ulp (%.3f %% not correctly rounded), rsqrt_cubic %.4f ulp\n", er, 100.0 * off / normal, eq);
    int bad = !(er <= 1.0) + !(eq <= 1.0);
    for (int i = normal; i < n; ++i) // 0, inf and NaN give NaN in both
        if (!std::isnan(r[i]) || !std::isnan(q[i])) {
            std::printf("special value %g: %g %g\n", x[i], r[i], q[i]);
            ++bad;
        }
    return bad ? 1 : 0;
}
