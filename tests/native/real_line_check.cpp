// Host check of the real line operator (csrc/real_line.cuh): the warp's lane
// layout, the fold into blocks, mma.m8n8k4's index arithmetic and the block
// fragments are emulated for all 32 lanes and compared with the dense circulant
// matrix in long double.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../../polystring_b200/csrc/real_line.cuh"

using namespace ps;

template <int N>
double check() {
    using R = RealLine<N>;
    std::vector<double> L(N), kf;
    for (int k = 0; k < N; k++) {
        const int r = k < N / 2 + 1 ? k : N - k;
        L[k] = exp(-0.013 * r * r);
    }
    real_fragments(N, L, kf);
    if ((int)kf.size() != R::FRAG || R::FRAG != real_frag_doubles(N)) return 1.0;
    std::vector<double> th;
    real_parts(N, L, th);
    if ((int)th.size() != 4 * R::PARTS || (int)th.size() != real_parts_doubles(N)) return 3.0;
    double parts = 0.0;   // fragments formed from the parts, sums and differences of table entries
    for (int b = 0; b < 4; b++)
        for (int t = 0; t < R::T; t++)
            for (int s = 0; s < R::S; s++)
                for (int l = 0; l < 32; l++) {
                    const int og = real_column_orbit(l >> 2), j = l & 3, h = b >> 1;
                    if (8 * t + og >= R::O || 4 * s + j >= R::O) continue;
                    const double a = th[2 * h * R::PARTS + 4 * R::S + og - j + 8 * t - 4 * s];
                    const double c = th[(2 * h + 1) * R::PARTS + og + j + 1 + 8 * t + 4 * s];
                    parts = fmax(parts, fabs((b & 1 ? a - c : a + c) - kf[R::frag(b, t, s) + l]));
                }
    if (parts > 3e-16) return 4.0;
    std::vector<double> line(8 * N);
    srand(N);
    for (double& v : line) v = rand() / (double)RAND_MAX - 0.3;
    std::vector<std::vector<double>> x(32, std::vector<double>(R::E)), y(32, std::vector<double>(8 * R::T, 0.0));
    std::vector<int> seen(8 * N, 0);
    for (int l = 0; l < 32; l++)
        for (int s = 0; s < R::S; s++)
            for (int i = 0; i < 4; i++) {
                const int o = (l & 3) + 4 * s;
                if (o < R::O) seen[(l >> 2) * N + R::point(i, o)]++;
                x[l][4 * s + i] = o < R::O ? line[(l >> 2) * N + R::point(i, o)] : 0.0;
            }
    for (int c : seen)
        if (c != 1) return 2.0;
    for (auto& v : x) R::fold(v.data());
    for (int t = 0; t < R::T; t++)
        for (int s = 0; s < R::S; s++)
            for (int b = 0; b < 4; b++)
                for (int l = 0; l < 32; l++)   // C[g][n] += sum_k A[g][k] B[k][n]
                    for (int h = 0; h < 2; h++) {
                        const int g = l >> 2, n = 2 * (l & 3) + h;
                        for (int k = 0; k < 4; k++)
                            y[l][2 * R::T * b + 2 * t + h] += x[4 * g + k][4 * s + b] * kf[R::frag(b, t, s) + 4 * n + k];
                    }
    std::vector<double> out(8 * N, 0.0);
    for (int l = 0; l < 32; l++) {
        for (int h = 0; h < 2; h++) R::join(y[l].data() + 4 * R::T * h, h, x[l].data());
        R::unfold(x[l].data());
        for (int s = 0; s < R::S; s++)
            for (int i = 0; i < 4; i++) {
                const int o = (l & 3) + 4 * s;
                if (o < R::O) out[(l >> 2) * N + R::point(i, o)] = x[l][4 * s + i];
            }
    }
    const long double pi = 3.141592653589793238462643383279502884L;
    std::vector<long double> c(N, 0.0L);
    for (int d = 0; d < N; d++)
        for (int k = 0; k < N; k++) c[d] += L[k] * cosl(2.0L * pi * k * d / N) / N;
    double worst = 0.0;
    for (int g = 0; g < 8; g++)
        for (int n = 0; n < N; n++) {
            long double v = 0.0L;
            for (int m = 0; m < N; m++) v += c[(n - m + N) % N] * line[g * N + m];
            worst = fmax(worst, fabs((double)(v - out[g * N + n])));
        }
    return worst;
}

int main() {
    const double e[] = {check<4>(),  check<8>(),  check<12>(), check<16>(), check<24>(),
                        check<32>(), check<48>(), check<64>(), check<96>(), check<128>(), check<192>(), check<256>(), check<352>()};
    double worst = 0.0;
    for (double v : e) worst = fmax(worst, v);
    printf("%.3e\n", worst);
    return 0;
}
