// plane_sweep.cu -- RQM4 / OS2 sweeps of 1D grids, and of 2D grids of up to
// 64 x 64 points, on real line operators (real_line.cuh): one CTA runs all
// contour steps of a chain (2D) or of both chains of a solve (1D), the fields
// never leave its shared memory and registers, and only the history slices
// are written.
//
// 2D, Lx rows of Ly points in shared memory.  A tile of eight rows or of eight
// columns belongs to two warps, one for the half-step field Z and one for the
// full-step field W.  One contour step:
//
//   columns   W warps: Dx(full); Z warps: Dx(half), times e^{-w ds/2}, Dx(half)
//   rows      Z warps: Dy(half), q[t+1] = (4 e^{-w ds/4} Z - e^{-w ds/2} W) / 3
//             -> history, next e^{-w ds/4} q, Dy(half); W warps: hand their row
//             of W over, take e^{-w ds/2} q, Dy(full)
//
// OS2 has only the W warps' operators, with q = e^{-w ds/2} Dy(full) W.
// One SM's tensor cores bound a 64^2 step at 6 operators x 8 tiles x 670 cycles
// / 4 = 8000 cycles (4.2 us); it takes 9.1, 48^2 5.4, 32^2 2.3, 16^2 1.2 (a launch
// per line pass: 64^2 20).  So single solves leave it for the tiles of tile_sweep.cu
// from 32 x 64 points on, while batches and strings, whose chains fill the SMs, stay.
//
// 1D: thread (chain, orbit) keeps the orbit's four points of q and both factors
// in registers; an operator's folded values go through shared memory, its
// (block, output tile) products belong to one warp each, the two chains being
// two of the eight lines of a product.  64 points 0.82 us a step (a launch a step: 10),
// 128 1.5, 256 5.6; its chain of shared-memory trips bounds it.  (e^{-w ds/2} as the square
// of e^{-w ds/4}: 0.84, and three roundings for one.)
#include <algorithm>

#include "engine.h"
#include "ps_internal.h"
#include "fft_core.cuh"
#include "real_line.cuh"
#include "real_sweep.h"

namespace ps {

namespace {

constexpr size_t kSmemLimit = 227 * 1024 - 1024;
constexpr int kMaxLine = 64;   // longest axis of a 2D grid here

// row pitch: 4 mod 8 doubles, so that the 4 lines x 4 consecutive values of a
// half warp fall in different banks, by rows and by columns
__host__ __device__ __forceinline__ int pitch_of(int n) { return n + ((n & 7) == 4 ? 0 : 4); }
__host__ __device__ __forceinline__ constexpr int tiles_of(int n) { return (n + 7) / 8; }
__host__ __device__ __forceinline__ int values_of(int N) { return 4 * ((N / 4 + 3) / 4); }

__device__ __forceinline__ int lane_block(const RealLane& c, int t) { return t < c.sw[0] ? 0 : t < c.sw[1] ? 1 : 2; }

// barrier of a tile's two warps
__device__ __forceinline__ void pair_sync(int tile) { asm volatile("bar.sync %0, 64;" ::"r"(tile + 1) : "memory"); }

// f(value index, point) for every point that the lane holds
template <int N, class F>
__device__ __forceinline__ void each_value(int j, F f) {
    using R = RealLine<N>;
#pragma unroll
    for (int s = 0; s < R::S; s++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int o = j + 4 * s;
            if (R::WHOLE || o < R::O) f(4 * s + i, R::point(i, o));
        }
}
template <int N>
__device__ __forceinline__ void clear(double (&x)[RealLine<N>::E]) {
    if constexpr (!RealLine<N>::WHOLE) {
#pragma unroll
        for (int i = 0; i < RealLine<N>::E; i++) x[i] = 0.0;
    }
}

// What a warp knows of its chain.
struct Chain {
    const RealProblem* p;
    const RealLane* L;
    double *Z, *W;               // the fields, Lx rows of pitch pitch_of(Ly)
    const double *opx, *opy;     // fragments of the operators along x and y, full step then half step
    double *keepc, *keepr;       // this lane's kept factors of its columns and rows
    int tile, lane;
    bool zwarp;
};

// The lane's factors of its lines (point n at e[n * st]), read from memory when
// its chain has come to another block (fresh), else from where it keeps them.
template <int N>
__device__ __forceinline__ void load_factors(double (&f)[RealLine<N>::E], const double* e, int st, int j, double* keep,
                                             bool fresh) {
    clear<N>(f);
    if (fresh) {
        each_value<N>(j, [&](int i, int n) { f[i] = __ldg(e + n * st); });
#pragma unroll
        for (int i = 0; i < RealLine<N>::E; i++) keep[32 * i] = f[i];
    } else {
#pragma unroll
        for (int i = 0; i < RealLine<N>::E; i++) f[i] = keep[32 * i];
    }
}

// columns of step t (N = Lx), in place
template <int N>
__device__ __forceinline__ void columns(const Chain& c, int t) {
    using R = RealLine<N>;
    const int Ly = c.p->Ly, pitch = pitch_of(Ly), g = c.lane >> 2, j = c.lane & 3;
    if (c.tile >= tiles_of(Ly) || (c.zwarp && c.p->os2)) return;
    const bool ok = 8 * c.tile + g < Ly;
    const int y = ok ? 8 * c.tile + g : 8 * c.tile;
    double* v = (c.zwarp ? c.Z : c.W) + y;
    double x[R::E];
    clear<N>(x);
    each_value<N>(j, [&](int i, int n) { x[i] = v[n * pitch]; });
    if (c.zwarp) {
        const int b = lane_block(*c.L, t);
        double f[R::E];
        load_factors<N>(f, c.L->eF[b] + y, Ly, j, c.keepc, t == 0 || b != lane_block(*c.L, t - 1));
        R::apply(x, c.opx + R::FRAG + c.lane);
        if (c.L->keep_half && ok) {
            double* out = c.L->keep_half + (long)t * N * Ly + y;
            each_value<N>(j, [&](int i, int n) { out[n * Ly] = x[i]; });
        }
#pragma unroll
        for (int i = 0; i < R::E; i++) x[i] = __dmul_rn(x[i], f[i]);
        R::apply(x, c.opx + R::FRAG + c.lane);
    } else {
        R::apply(x, c.opx + c.lane);
    }
    __syncwarp();   // lanes past the last column read what another lane writes
    if (ok) each_value<N>(j, [&](int i, int n) { v[n * pitch] = x[i]; });
}

// rows after step t (t < 0: the head), and the next step's inputs (N = Ly)
template <int N>
__device__ __forceinline__ void rows(const Chain& c, int t) {
    using R = RealLine<N>;
    const int Lx = c.p->Lx, pitch = pitch_of(N), g = c.lane >> 2, j = c.lane & 3;
    if (c.tile >= tiles_of(Lx) || (c.zwarp && c.p->os2)) return;
    const long M = (long)Lx * N;
    const bool ok = 8 * c.tile + g < Lx, os2 = c.p->os2, next = t + 1 < c.p->Ns;
    const int r = ok ? 8 * c.tile + g : 8 * c.tile;
    double *z = c.Z + r * pitch, *w = c.W + r * pitch;
    const int now = t < 0 ? -1 : lane_block(*c.L, t), nb = lane_block(*c.L, t + 1);
    const double* const* e = os2 ? c.L->eF : c.L->eH;
    double x[R::E];
    clear<N>(x);
    if (c.zwarp || os2) {
        double f[R::E];
        if (t < 0) {
            each_value<N>(j, [&](int i, int n) { x[i] = __ldg(c.L->hist + (long)r * N + n); });
        } else {
            load_factors<N>(f, e[now] + (long)r * N, 1, j, c.keepr, false);
            each_value<N>(j, [&](int i, int n) { x[i] = (os2 ? w : z)[n]; });
            R::apply(x, c.opy + (os2 ? 0 : R::FRAG) + c.lane);
            if (os2) {
#pragma unroll
                for (int i = 0; i < R::E; i++) x[i] = __dmul_rn(x[i], f[i]);
            } else {
                each_value<N>(j, [&](int i, int n) {
                    const double h = f[i], v = __dmul_rn(x[i], h), u = __dmul_rn(w[n], __dmul_rn(h, h));
                    x[i] = div_rn(fma(4.0, v, -u), 3.0, 1.0 / 3.0);
                });
                if (c.L->keep_full && ok) {
                    double* full = c.L->keep_full + (long)t * M + (long)r * N;
                    each_value<N>(j, [&](int i, int n) { full[n] = w[n]; });
                }
                if (c.L->src_o) {
                    const double wa = c.L->src_w[0][t + 1], wb = c.L->src_w[1][t + 1];
                    const double *o = c.L->src_o + (long)(t + 1) * M + (long)r * N, *pa = c.L->src_p[0] + (long)r * N,
                                 *pb = c.L->src_p[1] + (long)r * N;
                    each_value<N>(j, [&](int i, int n) {
                        x[i] = fma(fma(wa, __ldg(pa + n), wb * __ldg(pb + n)), __ldg(o + n), x[i]);
                    });
                }
            }
            double* out = c.L->hist + (long)(t + 1) * M + (long)r * N;
            if (ok) each_value<N>(j, [&](int i, int n) { out[n] = x[i]; });
        }
        if (!next) return;
        load_factors<N>(f, e[nb] + (long)r * N, 1, j, c.keepr, nb != now);
        __syncwarp();
        if (os2) {
            if (ok) each_value<N>(j, [&](int i, int n) { w[n] = __dmul_rn(x[i], f[i]); });
            return;
        }
#pragma unroll
        for (int i = 0; i < R::E; i++) x[i] = __dmul_rn(x[i], f[i]);   // e^{-w ds/4} q
        if (ok) each_value<N>(j, [&](int i, int n) { w[n] = __dmul_rn(x[i], f[i]); });
        pair_sync(c.tile);   // e^{-w ds/2} q is there
        R::apply(x, c.opy + R::FRAG + c.lane);
        if (ok) each_value<N>(j, [&](int i, int n) { z[n] = x[i]; });
    } else if (next) {
        pair_sync(c.tile);
        each_value<N>(j, [&](int i, int n) { x[i] = w[n]; });
        R::apply(x, c.opy + c.lane);
        __syncwarp();
        if (ok) each_value<N>(j, [&](int i, int n) { w[n] = x[i]; });
    }
}

#define PL_CASES(X) X(4) X(8) X(12) X(16) X(24) X(32) X(48) X(64)

// chain k = blockIdx.x is chain k % nl of solve k / nl; many == nullptr: the solve `one`
__global__ void __launch_bounds__(512, 1) plane_sweep_kernel(const __grid_constant__ RealProblem one,
                                                             const RealProblem* __restrict__ many) {
    extern __shared__ __align__(16) double sm[];
    __shared__ RealProblem p;
    const int k = blockIdx.x;
    if (many) {
        constexpr int W = sizeof(RealProblem) / 4;
        for (int i = threadIdx.x; i < W; i += blockDim.x)
            reinterpret_cast<int*>(&p)[i] = reinterpret_cast<const int*>(many + k / one.nl)[i];
    } else if (threadIdx.x == 0) {
        p = one;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < p.nfrag; i += blockDim.x) sm[i] = p.frag[i];
    Chain c;
    c.p = &p;
    c.L = &p.lane[k % one.nl];
    c.tile = threadIdx.x >> 6;
    c.zwarp = ((threadIdx.x >> 5) & 1) == 0;
    c.lane = threadIdx.x & 31;
    c.opx = sm + p.fo[0];
    c.opy = sm + p.fo[1];
    c.Z = sm + p.nfrag;
    c.W = c.Z + p.Lx * pitch_of(p.Ly);
    const int nt = blockDim.x >> 6;
    double* keep = c.W + p.Lx * pitch_of(p.Ly);
    c.keepc = keep + c.tile * 32 * values_of(p.Lx) + c.lane;
    c.keepr = keep + nt * 32 * values_of(p.Lx) + c.tile * 32 * values_of(p.Ly) + c.lane;
    __syncthreads();
    for (int t = -1; t < p.Ns; t++) {
        if (t >= 0) {
            switch (p.Lx) {
#define X(N) case N: columns<N>(c, t); break;
                PL_CASES(X)
#undef X
            }
            __syncthreads();
        }
        switch (p.Ly) {
#define X(N) case N: rows<N>(c, t); break;
            PL_CASES(X)
#undef X
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// 1D
// ---------------------------------------------------------------------------
constexpr int k1T = 256;   // threads 0..127 the first chain's orbits, 128..255 the second's

// (block, output tile) products that a warp of eight owns, and whether their
// fragments (of both operators) stay in registers
template <int N>
struct Line1 {
    using R = RealLine<N>;
    static constexpr int U = (4 * R::T + 7) / 8;
    static constexpr bool REGS = U * R::S <= 16;
    static constexpr int OP = 4 * R::S, T8 = 8 * R::T;
};

template <int N>
__global__ void __launch_bounds__(k1T, 1) line_sweep_kernel(const __grid_constant__ RealProblem p) {
    using R = RealLine<N>;
    using Q = Line1<N>;
    constexpr int S = R::S, T = R::T, O = R::O;
    // folded values [field][block][chain][orbit], results likewise
    __shared__ double xb[2][4][2][Q::OP], yb[2][4][2][Q::T8];
    __shared__ double parts[Q::REGS ? 1 : 8 * R::PARTS];
    const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3, warp = threadIdx.x >> 5;
    const int ch = threadIdx.x >> 7, o = threadIdx.x & 127;
    const bool own = ch < p.nl && o < O, line = g < p.nl;
    const RealLane& L = p.lane[ch];
    for (int i = threadIdx.x; i < 2 * 4 * 2 * Q::OP; i += k1T) (&xb[0][0][0][0])[i] = 0.0;
    if constexpr (!Q::REGS)
        for (int i = threadIdx.x; i < 8 * R::PARTS; i += k1T) parts[i] = p.frag[i];
    // fragments of product u of operator f (0 full step, 1 half step), contraction step s
    auto fragment = [&](const double* op, int u, int s) {
        const int b = u / T, t = u - b * T, h = b >> 1, og = real_column_orbit(g);
        const double a = op[2 * h * R::PARTS + 4 * S + og - j + 8 * t - 4 * s];
        const double c = op[(2 * h + 1) * R::PARTS + og + j + 1 + 8 * t + 4 * s];
        return b & 1 ? a - c : a + c;
    };
    double kf[2][Q::REGS ? Q::U : 1][Q::REGS ? S : 1];
    if constexpr (Q::REGS) {
#pragma unroll
        for (int f = 0; f < 2; f++)
#pragma unroll
            for (int i = 0; i < Q::U; i++)
#pragma unroll
                for (int s = 0; s < S; s++)
                    kf[f][i][s] = warp + 8 * i < 4 * T ? fragment(p.frag + 4 * f * R::PARTS, warp + 8 * i, s) : 0.0;
    }
    // the warp's products of field `fld` under operator f
    auto product = [&](int fld, int f, int i) {
        const int u = warp + 8 * i;
        if (u >= 4 * T) return;
        const int b = u / T, t = u - b * T;
        const double* a = &xb[fld][b][line ? g : 0][j];
        double y0 = 0.0, y1 = 0.0;
        if constexpr (Q::REGS) {
#pragma unroll
            for (int s = 0; s < S; s++) R::mma(y0, y1, line ? a[4 * s] : 0.0, kf[f][i][s]);
        } else {
            double z0 = 0.0, z1 = 0.0;
            for (int s = 0; s + 1 < S; s += 2) {
                R::mma(y0, y1, line ? a[4 * s] : 0.0, fragment(parts + 4 * f * R::PARTS, u, s));
                R::mma(z0, z1, line ? a[4 * s + 4] : 0.0, fragment(parts + 4 * f * R::PARTS, u, s + 1));
            }
            if (S & 1) R::mma(y0, y1, line ? a[4 * (S - 1)] : 0.0, fragment(parts + 4 * f * R::PARTS, u, S - 1));
            y0 += z0;
            y1 += z1;
        }
        if (line) {
            yb[fld][b][g][8 * t + j] = y0;
            yb[fld][b][g][8 * t + 4 + j] = y1;
        }
    };
    auto put = [&](int fld, double a, double b, double c, double d) {
        const double up = a + b, um = a - b, vp = c + d, vm = c - d;
        xb[fld][0][ch][o] = up + vp;
        xb[fld][1][ch][o] = up - vp;
        xb[fld][2][ch][o] = um + vm;
        xb[fld][3][ch][o] = um - vm;
    };
    auto take = [&](int fld, double (&v)[4]) {
        const double p0 = yb[fld][0][ch][o], p1 = yb[fld][1][ch][o], p2 = yb[fld][2][ch][o], p3 = yb[fld][3][ch][o];
        const double up = p0 + p1, vp = p0 - p1, um = p2 + p3, vm = p2 - p3;
        v[0] = up + um;
        v[1] = up - um;
        v[2] = vp + vm;
        v[3] = vp - vm;
    };
    double q[4] = {0.0, 0.0, 0.0, 0.0}, e[4] = {0.0, 0.0, 0.0, 0.0}, f[4] = {0.0, 0.0, 0.0, 0.0}, w[4], z[4];
    if (own)
#pragma unroll
        for (int i = 0; i < 4; i++) q[i] = __ldg(L.hist + R::point(i, o));
    __syncthreads();
    for (int t = 0; t < p.Ns; t++) {
        if (own) {
            const int b = lane_block(L, t);
            if (t == 0 || b != lane_block(L, t - 1))
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    f[i] = __ldg(L.eF[b] + R::point(i, o));
                    e[i] = __ldg(L.eH[b] + R::point(i, o));
                }
#pragma unroll
            for (int i = 0; i < 4; i++) {
                z[i] = __dmul_rn(q[i], e[i]);
                w[i] = __dmul_rn(q[i], f[i]);
            }
            put(0, w[0], w[1], w[2], w[3]);
            if (!p.os2) put(1, z[0], z[1], z[2], z[3]);
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < Q::U; i++) {
            if (!p.os2) product(1, 1, i);
            product(0, 0, i);
        }
        __syncthreads();
        if (!p.os2) {
            if (own) {
                take(1, z);
#pragma unroll
                for (int i = 0; i < 4; i++) z[i] = __dmul_rn(z[i], f[i]);
                put(1, z[0], z[1], z[2], z[3]);
            }
            __syncthreads();
#pragma unroll
            for (int i = 0; i < Q::U; i++) product(1, 1, i);
            __syncthreads();
        }
        if (own) {
            take(0, w);
            if (!p.os2) take(1, z);
            double* out = L.hist + (long)(t + 1) * N;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                w[i] = __dmul_rn(w[i], f[i]);
                q[i] = p.os2 ? w[i] : div_rn(fma(4.0, __dmul_rn(z[i], e[i]), -w[i]), 3.0, 1.0 / 3.0);
                out[R::point(i, o)] = q[i];
            }
        }
    }
}

bool plane_line_ok(int N) {
    switch (N) {
#define X(V) case V:
        PL_CASES(X)
#undef X
        return true;
    }
    return false;
}

int pairs_of(int Lx, int Ly) { return std::max(tiles_of(Lx), tiles_of(Ly)); }

size_t plane_smem(int Lx, int Ly, int nfrag, int pairs) {
    return sizeof(double) *
           ((size_t)nfrag + 2 * (size_t)Lx * pitch_of(Ly) + (size_t)pairs * 32 * (values_of(Lx) + values_of(Ly)));
}

#define LN_CASES(X) PL_CASES(X) X(96) X(128) X(192) X(256) X(352)

}  // namespace

bool plane_sweep_supported(int Lx, int Ly) {
    return plane_line_ok(Lx) && plane_line_ok(Ly) &&
           plane_smem(Lx, Ly, 2 * (real_frag_doubles(Lx) + real_frag_doubles(Ly)), kMaxLine / 8) <= kSmemLimit;
}

void plane_sweep_prepare() {
    PS_CUDA(cudaFuncSetAttribute(plane_sweep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
}

int plane_sweep_pairs(int Lx, int Ly) { return pairs_of(Lx, Ly); }
size_t plane_sweep_smem(const RealProblem& p, int pairs) { return plane_smem(p.Lx, p.Ly, p.nfrag, pairs); }

void plane_sweep_launch(const RealProblem& p, cudaStream_t st) {
    const int pairs = pairs_of(p.Lx, p.Ly);
    plane_sweep_kernel<<<p.nl, 64 * pairs, plane_sweep_smem(p, pairs), st>>>(p, nullptr);
    PS_CUDA(cudaGetLastError());
}

void plane_sweep_launch_many(const RealProblem* d, int n, int pairs, size_t smem, cudaStream_t st) {
    RealProblem one{};
    one.nl = 2;
    plane_sweep_kernel<<<2 * n, 64 * pairs, smem, st>>>(one, d);
    PS_CUDA(cudaGetLastError());
}

bool line_sweep_supported(int Lx) {
    switch (Lx) {
#define X(V) case V:
        LN_CASES(X)
#undef X
        return true;
    }
    return false;
}

void line_sweep_launch(const RealProblem& p, cudaStream_t st) {
    for (const RealLane& L : p.lane)
        if (L.keep_half || L.keep_full || L.src_o) throw Error(-2, "the sweep of 1D grids keeps no fields and takes no source");
    switch (p.Lx) {
#define X(V) case V: line_sweep_kernel<V><<<1, k1T, 0, st>>>(p); break;
        LN_CASES(X)
#undef X
        default: throw Error(-2, "no line sweep for this grid");
    }
    PS_CUDA(cudaGetLastError());
}

}  // namespace ps
