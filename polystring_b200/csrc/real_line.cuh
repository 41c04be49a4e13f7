// real_line.cuh -- the diffusion step along one axis as a real matrix product
// on the FP64 tensor cores.
//
// Along one axis of N points the split step's F^-1 diag(L) F is a real
// symmetric circulant matrix C with C[n][m] = c(n - m),
//
//     c(d) = (1/N) sum_k L_k cos(2 pi k d / N),
//
// because L_k is real and even in k.  It acts on real lines: the two chains
// of a solve need no complex packing.  C commutes with the shift n -> n + N/2
// and with the reflection n -> N-1-n, which commute with each other and have
// no fixed points when 4 divides N, so the points fall into O = N/4 orbits
//
//     {o, o + N/2, N-1-o, N/2-1-o},  o = 0 .. O-1,
//
// and C splits into four O x O blocks K_rs, r, s = +-1 (the characters of the
// four-element group):
//
//     x_rs[o] = (x[o] + s x[o+N/2]) + r (x[N-1-o] + s x[N/2-1-o])
//     y_rs    = K_rs x_rs,  K_rs[o][p] = (T_s(o - p) + r T_s(o + p + 1)) / 4,
//     T_s(d)  = c(d) + s c(d + N/2)
//     y[o]    = sum_rs y_rs[o], and with the signs of the image elsewhere.
//
// A line costs N^2/4 multiply-adds and 4 N additions instead of N^2: for
// N = 64 that is 20 FP64 operations a point, as many as the two transforms of
// a fast Fourier transform take, but they run as mma.m8n8k4 instructions with no
// exchange between lanes.  Measured on a B200: 36.7 TFLOP/s of mma.m8n8k4 from
// 4 warps an SM on (one warp a scheduler, four independent accumulators; 26
// cycles of latency), against 32.5 TFLOP/s of independent FMAs from 16 warps.
//
// A warp holds 8 lines.  In mma.m8n8k4 lane 4 g + j holds A[g][j] (line g,
// contraction index j), B[j][g] and C[g][2j], C[g][2j+1].  Lane 4 g + j keeps
// the orbits j + 4 s, s < S, of line g, x[4 s + i] being image i of its orbit;
// the columns of a block's output tile are ordered so that column 2 j is
// orbit j and column 2 j + 1 orbit j + 4, hence the accumulators come out in
// the layout of the inputs and operators chain in registers.
#pragma once

#include <cmath>
#include <vector>

#include "fft_core.cuh"

namespace ps {

// the orbit of column g of an output tile
PS_HD constexpr int real_column_orbit(int g) { return (g >> 1) + 4 * (g & 1); }

// orbits of a line of N points (N a multiple of 4), orbits a lane holds, and
// output tiles of eight orbits
template <int N>
struct RealLine {
    static_assert(N % 4 == 0, "the points of a line fall into orbits of four");
    static constexpr int O = N / 4;
    static constexpr int S = (O + 3) / 4;
    static constexpr int T = (O + 7) / 8;
    static constexpr int E = 4 * S;                  // values a lane holds
    static constexpr int FRAG = 4 * T * S * 32;      // doubles of an operator's B fragments
    static constexpr int PARTS = 8 * T + 4 * S;      // entries of a part of a block (real_parts)
    static constexpr bool WHOLE = O % 4 == 0;        // every lane's orbits exist

    // image i of orbit o
    PS_HD static constexpr int point(int i, int o) {
        return i == 0 ? o : i == 1 ? o + N / 2 : i == 2 ? N - 1 - o : N / 2 - 1 - o;
    }
    // points -> block values, block b of orbit s at x[4 s + b]
    PS_HD static void fold(double* x) {
#pragma unroll
        for (int s = 0; s < S; s++) {
            const double up = x[4 * s] + x[4 * s + 1], um = x[4 * s] - x[4 * s + 1];
            const double vp = x[4 * s + 2] + x[4 * s + 3], vm = x[4 * s + 2] - x[4 * s + 3];
            x[4 * s] = up + vp;
            x[4 * s + 1] = up - vp;
            x[4 * s + 2] = um + vm;
            x[4 * s + 3] = um - vm;
        }
    }
    // results of the two blocks with s = (-1)^h (orbit s of block r at y[2 T r + s]) -> their sum and
    // difference, in the places of the blocks' values
    PS_HD static void join(const double* y, int h, double* x) {
#pragma unroll
        for (int s = 0; s < S; s++) {
            x[4 * s + 2 * h] = y[s] + y[2 * T + s];
            x[4 * s + 2 * h + 1] = y[s] - y[2 * T + s];
        }
    }
    // joined blocks -> points
    PS_HD static void unfold(double* x) {
#pragma unroll
        for (int s = 0; s < S; s++) {
            const double up = x[4 * s], vp = x[4 * s + 1], um = x[4 * s + 2], vm = x[4 * s + 3];
            x[4 * s] = up + um;
            x[4 * s + 1] = up - um;
            x[4 * s + 2] = vp + vm;
            x[4 * s + 3] = vp - vm;
        }
    }
    // the fragment of (block, output tile, orbit s)
    PS_HD static constexpr int frag(int b, int t, int s) { return ((b * T + t) * S + s) * 32; }

#ifdef __CUDACC__
    __device__ __forceinline__ static void mma(double& c0, double& c1, double a, double b) {
        asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
            : "+d"(c0), "+d"(c1)
            : "d"(a), "d"(b));
    }

    // x <- C x for the warp's eight lines; kf points at this lane's entry of
    // the operator's fragments (shared memory, consecutive lanes in consecutive
    // banks)
    __device__ __forceinline__ static void apply(double (&x)[E], const double* kf) {
        fold(x);
        // two blocks at a time: their results take the place of their inputs
#pragma unroll
        for (int h = 0; h < 2; h++) {
            double y[4 * T];
#pragma unroll
            for (int i = 0; i < 4 * T; i++) y[i] = 0.0;
#pragma unroll
            for (int s = 0; s < S; s++)
#pragma unroll
                for (int t = 0; t < T; t++)
#pragma unroll
                    for (int r = 0; r < 2; r++)
                        mma(y[2 * T * r + 2 * t], y[2 * T * r + 2 * t + 1], x[4 * s + 2 * h + r],
                            kf[frag(2 * h + r, t, s)]);
            join(y, h, x);
        }
        unfold(x);
    }
#endif
};

// blocks in the order (r, s) = (+,+), (-,+), (+,-), (-,-), as apply() uses them
constexpr int kRealBlockR[4] = {1, -1, 1, -1};
constexpr int kRealBlockS[4] = {1, 1, -1, -1};

// doubles of the B fragments of an operator on lines of N points
PS_HD constexpr int real_frag_doubles(int N) { return 4 * ((N / 4 + 7) / 8) * ((N / 4 + 3) / 4) * 32; }

// T_s(d) for s = +1, -1 and any d, in long double: half[h] of period N
struct RealKernel {
    int N;
    std::vector<long double> half[2];
    RealKernel(int n, const std::vector<double>& L) : N(n) {
        const long double pi = 3.141592653589793238462643383279502884L;
        std::vector<long double> cosn(N), c(N);
        for (int m = 0; m < N; m++) cosn[m] = cosl(2.0L * pi * m / N);
        // even in d, and its terms in k
        for (int d = 0; d <= N / 2; d++) {
            long double a = 0.0L;
            for (int k = 1, kd = d; k < N / 2; k++) {   // kd = k d mod N
                a += L[k] * cosn[kd];
                kd += d;
                if (kd >= N) kd -= N;
            }
            c[d] = c[(N - d) % N] = (2.0L * a + L[0] + (d & 1 ? -L[N / 2] : L[N / 2])) / N;
        }
        for (int h = 0; h < 2; h++)
            for (int d = 0; d < N; d++) half[h].push_back(h ? c[d] - c[(d + N / 2) % N] : c[d] + c[(d + N / 2) % N]);
    }
    long double operator()(int s, int d) const { return half[s < 0][((d % N) + N) % N]; }
};

// appends the B fragments of F^-1 diag(L) F along one axis of N points (L for
// k = 0 .. N-1, even in k), formed in long double and rounded once
inline void real_fragments(int N, const std::vector<double>& L, std::vector<double>& out) {
    const int O = N / 4, S = (O + 3) / 4, T = (O + 7) / 8;
    const RealKernel Ts(N, L);
    for (int b = 0; b < 4; b++)
        for (int t = 0; t < T; t++)
            for (int s = 0; s < S; s++)
                for (int lane = 0; lane < 32; lane++) {
                    const int o = 8 * t + real_column_orbit(lane >> 2), q = 4 * s + (lane & 3);
                    const long double k = Ts(kRealBlockS[b], o - q) + kRealBlockR[b] * Ts(kRealBlockS[b], o + q + 1);
                    out.push_back(o < O && q < O ? (double)(k / 4.0L) : 0.0);
                }
}


// doubles of the parts of an operator on lines of N points
PS_HD constexpr int real_parts_doubles(int N) { return 4 * (8 * ((N / 4 + 7) / 8) + 4 * ((N / 4 + 3) / 4)); }

// appends the parts of the same operator's blocks: for s = +1, -1 the Toeplitz
// part T_s(d) / 4 at 4 S + d, then the Hankel part T_s(d) / 4 at d.  A fragment is
// their sum (r = +1) or difference: an addition more than reading it, but 2 KB an
// operator at 128 points instead of 32 KB.
inline void real_parts(int N, const std::vector<double>& L, std::vector<double>& out) {
    const int O = N / 4, S = (O + 3) / 4, T = (O + 7) / 8, n = 8 * T + 4 * S;
    const RealKernel Ts(N, L);
    for (int s : {1, -1})
        for (int off : {4 * S, 0})
            for (int i = 0; i < n; i++) out.push_back((double)(Ts(s, i - off) / 4.0L));
}

}  // namespace ps
