// Host check of the kernels of the real line operators (csrc/real_line.cuh): T_s(d) of
// every line length against the plain sums over all k.  Prints the largest difference.
#include <cstdio>

#include "../../polystring_b200/csrc/real_line.cuh"

int main() {
    const long double pi = 3.141592653589793238462643383279502884L;
    long double worst = 0.0L;
    for (int N : {4, 8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 352}) {
        std::vector<double> L(N);
        for (int k = 0; k < N; k++) {
            const int r = k < N / 2 + 1 ? k : N - k;
            L[k] = exp(-0.013 * r * r);
        }
        std::vector<long double> c(N, 0.0L);
        for (int d = 0; d < N; d++) {
            for (int k = 0; k < N; k++) c[d] += (long double)L[k] * cosl(2.0L * pi * ((long)k * d % N) / N);
            c[d] /= N;
        }
        const ps::RealKernel T(N, L);
        for (int d = -N; d < 2 * N; d++)
            for (int s : {1, -1}) worst = fmaxl(worst, fabsl(T(s, d) - (c[(d + N) % N] + s * c[(d + N + N / 2) % N])));
    }
    printf("%.3Le\n", worst);
    return 0;
}
