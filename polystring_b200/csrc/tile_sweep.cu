// tile_sweep.cu -- persistent RQM4 / OS2 sweep of 2D grids on real line operators
// (real_line.cuh): those with an axis longer than 64 points, and smaller ones where many
// CTAs are faster than plane_sweep.cu's one a chain (RealSweep, BatchAB).  A CTA takes a
// tile of eight lines, whose operators' products are dealt to its eight warps.
//
// Lx rows of Ly points, fields Z (half steps) and W (full step) of every chain
// in global memory (L2).  A contour step is two phases with a barrier over the
// chain's CTAs after each:
//
//   columns   tiles of eight columns: Dx(full) W; Dx(half) Z, times e^{-w ds/2},
//             Dx(half)
//   rows      tiles of eight rows: Dy(half) Z, q[t+1] = (4 e^{-w ds/4} Z -
//             e^{-w ds/2} W) / 3 -> history, next W = Dy(full) e^{-w ds/2} q and
//             Z = Dy(half) e^{-w ds/4} q
//
// OS2 has only W.  Thread (line, orbit) holds an orbit's four points in
// registers; folded values go through shared memory to the warps, which share the
// products of (field, character s, J output tiles) so that each has one unit, and the
// results back.  So a line of 128 points takes eight warps some 300 cycles where
// one warp alone takes 2800, which is what a single solve's few lines need.
// Lines of up to 64 points read the blocks' fragments (16 KB an operator pair at
// 64), longer ones form them from the Toeplitz and Hankel parts (4 KB at 128 points
// where the fragments take 64 KB).  The arithmetic of a line does not depend on how
// tiles are spread over CTAs or threads, and is that of plane_sweep.cu.
//
// Three forms.  A chain of up to 16 tiles is a cluster with the hardware's barrier
// (us a step: 64^2 4.4, 96^2 6.4, 128^2 6.8; with the barrier in memory, 1.4 us each,
// 5.9, 7.2, 8.3; line passes 20, 21.3, 22.4; 128^2 with 8 CTAs 11.9, so it takes 16).
// Larger grids run over the whole grid with barriers in memory, rows of 256 points on
// in parts (128 x 352 13.4, whole 20.4, line passes 26.5; 256^2 18.2, 28.5).  An image
// of a string is a cluster of eight CTAs of 128 threads, three an SM, so that 40
// images are resident at once (96^2 28.9 us a step for all, line passes 48.5; 16 x 128
// 12.4 and 26).  What bounds the first two is latency: two barriers and four trips
// through L2 and shared memory a step beside 1.6 us of products (128^2); strings the
// L2, some 3 TB/s of field traffic, and the trips.
#include <algorithm>
#include <cstdio>

#include "engine.h"
#include "ps_internal.h"
#include "fft_core.cuh"
#include "real_line.cuh"
#include "real_sweep.h"
#include "sweep_barrier.cuh"

namespace ps {

namespace {

constexpr int kNT = 256;      // threads of a CTA of the grid form
constexpr int kStringNT = 128;   // and of a string's clusters: three CTAs an SM
constexpr size_t kSmemLimit = 227 * 1024 - 1024;

// barrier over the cluster's CTAs, with their writes to global memory
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ int lane_block(const RealLane& c, int t) { return t < c.sw[0] ? 0 : t < c.sw[1] ? 1 : 2; }

// threadIdx.x, read anew where a phase starts: else the index arithmetic of every
// length's phases is hoisted out of the step loop and spills (0.9 KB a thread)
__device__ __forceinline__ int thread_index() {
    int t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    return t;
}

// pitch of a line's orbits in shared memory: 4 mod 8 doubles, so that the 4 lines
// x 4 consecutive orbits of a half warp fall in different banks
__host__ __device__ constexpr int pitch_of(int n) { return (n & 7) == 4 ? n : n + 4; }

constexpr int kFragments = 64;   // longest line whose operators are held as fragments

template <int N, int NT = kNT>
struct Tile {
    using R = RealLine<N>;
    static constexpr int O = R::O, S = R::S, T = R::T;
    static constexpr int XP = pitch_of(4 * S), YP = pitch_of(8 * T);
    static constexpr int XF = 32 * XP, YF = 32 * YP;   // a field: [block][line][orbit]
    static constexpr int OP = N <= kFragments ? R::FRAG : 4 * R::PARTS;   // doubles of an operator
    static constexpr int U = (8 * O + NT - 1) / NT;  // (line, orbit) items a thread
};

// folded values of field f, results of field f
struct Shared {
    double *x, *y;
    int xf, yf;
};

template <int N>
__device__ __forceinline__ void put(double* x, int g, int o, const double (&v)[4]) {
    using Q = Tile<N>;
    const double up = v[0] + v[1], um = v[0] - v[1], vp = v[2] + v[3], vm = v[2] - v[3];
    double* p = x + g * Q::XP + o;
    p[0] = up + vp;
    p[8 * Q::XP] = up - vp;
    p[16 * Q::XP] = um + vm;
    p[24 * Q::XP] = um - vm;
}
template <int N>
__device__ __forceinline__ void take(const double* y, int g, int o, double (&v)[4]) {
    using Q = Tile<N>;
    const double* p = y + g * Q::YP + o;
    const double a = p[0], b = p[8 * Q::YP], c = p[16 * Q::YP], d = p[24 * Q::YP];
    const double up = a + b, vp = a - b, um = c + d, vm = c - d;
    v[0] = up + um;
    v[1] = up - um;
    v[2] = vp + vm;
    v[3] = vp - vm;
}

// products of NF fields, field f under the operator with parts op0 (f = 0) or
// op1.  A unit is (field, character s, J output tiles of both characters r), a
// unit a warp: the tiles share the folded values, and a tile's Toeplitz entries
// are the next tile's two steps on, its Hankel entries two steps back.
// TT output tiles from tile0 on (default: all).
template <int N, int NT, int NF, int TT = Tile<N>::T>
__device__ __forceinline__ void products(const Shared& m, const double* op0, const double* op1, int tile0 = 0) {
    using Q = Tile<N, NT>;
    constexpr int P = Q::R::PARTS, S = Q::S, T = Q::T, UF = (NT / 64) / NF;   // units a field and character
    constexpr int J = (TT + UF - 1) / UF, G = (TT + J - 1) / J;
    constexpr bool FULL = T % TT == 0 && TT % J == 0;   // no tile past the last one
    const int tid = thread_index(), warp = tid >> 5;
    if (warp >= NF * 2 * G) return;
    const int lane = tid & 31, g = lane >> 2, j = lane & 3, og = real_column_orbit(g);
    const int f = warp / (2 * G), v = warp - f * 2 * G, h = v / G, t0 = tile0 + (v - h * G) * J;
    if (t0 >= T) return;
    const double* x = m.x + f * m.xf + (16 * h + g) * Q::XP + j;
    double a[J][2], b[J][2];
#pragma unroll
    for (int i = 0; i < J; i++) a[i][0] = a[i][1] = b[i][0] = b[i][1] = 0.0;
    if constexpr (N <= kFragments) {
        const double* op = (f ? op1 : op0) + lane;
#pragma unroll
        for (int s = 0; s < S; s++)
#pragma unroll
            for (int i = 0; i < J; i++) {
                if (!FULL && t0 + i >= T) break;
                Q::R::mma(a[i][0], a[i][1], x[4 * s], op[Q::R::frag(2 * h, t0 + i, s)]);
                Q::R::mma(b[i][0], b[i][1], x[8 * Q::XP + 4 * s], op[Q::R::frag(2 * h + 1, t0 + i, s)]);
            }
    } else {
        const double* op = (f ? op1 : op0) + 2 * h * P;
        // entries that only tiles past the last one would use count as zero
        const double *tp = op + 4 * S + og - j + 8 * t0, *hp = op + P + og + j + 1 + 8 * t0;
        double k[2 * J - 1], l[2 * J - 1];   // tp[4 (i - s)], hp[4 (i + s)]
#pragma unroll
        for (int i = 0; i < 2 * J - 1; i++) {
            k[i] = t0 + (i + 1) / 2 < T ? tp[4 * i] : 0.0;
            l[i] = 8 * t0 + 4 * i + og + j + 1 < P ? hp[4 * i] : 0.0;
        }
        const int last = 2 * J - 2;
#pragma unroll
        for (int s = 0; s < S; s++) {
            const double x0 = x[4 * s], x1 = x[8 * Q::XP + 4 * s];
#pragma unroll
            for (int i = 0; i < J; i++) {
                Q::R::mma(a[i][0], a[i][1], x0, k[2 * i] + l[2 * i]);
                Q::R::mma(b[i][0], b[i][1], x1, k[2 * i] - l[2 * i]);
            }
            if (s + 1 < S) {
#pragma unroll
                for (int i = last; i > 0; i--) k[i] = k[i - 1];
                k[0] = tp[-4 * (s + 1)];
#pragma unroll
                for (int i = 0; i < last; i++) l[i] = l[i + 1];
                l[last] = FULL || 8 * t0 + 4 * (last + s + 1) + og + j + 1 < P ? hp[4 * (last + s + 1)] : 0.0;
            }
        }
    }
    double* y = m.y + f * m.yf + (16 * h + g) * Q::YP + 8 * t0 + j;
#pragma unroll
    for (int i = 0; i < J; i++) {
        if (!FULL && t0 + i >= T) break;
        y[8 * i] = a[i][0];
        y[8 * i + 4] = a[i][1];
        y[8 * Q::YP + 8 * i] = b[i][0];
        y[8 * Q::YP + 8 * i + 4] = b[i][1];
    }
}

// q[t+1] from the half steps' result, the full step's before its factor e^2, and
// e = e^{-w ds/4}
__device__ __forceinline__ double next_slice(double z, double w, double e) {
    return div_rn(fma(4.0, __dmul_rn(z, e), -__dmul_rn(w, __dmul_rn(e, e))), 3.0, 1.0 / 3.0);
}
// q plus the lane's source of slice t at point n
__device__ __forceinline__ double with_source(const RealLane& L, int t, long n, long M, double q) {
    return fma(fma(L.src_w[0][t], __ldg(L.src_p[0] + n), L.src_w[1][t] * __ldg(L.src_p[1] + n)),
               __ldg(L.src_o + (long)t * M + n), q);
}

// columns of step t (N = Lx): tile of eight columns
template <int N, int NT>
__device__ __forceinline__ void columns(const RealProblem& p, const double* op, const Shared& m, int ch, int tile, int t) {
    using Q = Tile<N, NT>;
    using R = RealLine<N>;
    constexpr int HALF = Tile<N>::OP;
    const int tid = thread_index();
    const int Ly = p.Ly;
    const long M = (long)N * Ly;
    const RealLane& L = p.lane[ch];
    const bool os2 = p.os2;
    double* const Z = p.Z + ch * M;
    double* const W = p.W + ch * M;
    const double* const e = L.eF[lane_block(L, t)];
    double f[Q::U][4];
#pragma unroll
    for (int u = 0; u < Q::U; u++) {
        const int i = tid + u * NT, g = i & 7, o = i >> 3, y = 8 * tile + g;
        if (o >= Q::O) continue;
        double z[4] = {0.0, 0.0, 0.0, 0.0}, w[4] = {0.0, 0.0, 0.0, 0.0};
        if (y < Ly) {
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int at = R::point(k, o) * Ly + y;
                if (!os2) {
                    z[k] = __ldcg(Z + at);
                    f[u][k] = __ldg(e + at);
                }
                w[k] = __ldcg(W + at);
            }
        }
        if (!os2) put<N>(m.x, g, o, z);
        put<N>(m.x + m.xf, g, o, w);
    }
    __syncthreads();
    if (os2) {
        Shared w = m;
        w.x += m.xf;
        w.y += m.yf;
        products<N, NT, 1>(w, op, op);
    } else {
        products<N, NT, 2>(m, op + HALF, op);
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < Q::U; u++) {
        const int i = tid + u * NT, g = i & 7, o = i >> 3, y = 8 * tile + g;
        if (o >= Q::O) continue;
        double v[4];
        take<N>(m.y + m.yf, g, o, v);
        if (y < Ly)
#pragma unroll
            for (int k = 0; k < 4; k++) W[R::point(k, o) * Ly + y] = v[k];
        if (os2) continue;
        take<N>(m.y, g, o, v);
        if (y < Ly) {
            if (L.keep_half) {
                double* out = L.keep_half + (long)t * M + y;
#pragma unroll
                for (int k = 0; k < 4; k++) out[R::point(k, o) * Ly] = v[k];
            }
#pragma unroll
            for (int k = 0; k < 4; k++) v[k] = __dmul_rn(v[k], f[u][k]);
        }
        put<N>(m.x, g, o, v);
    }
    if (os2) return;
    __syncthreads();
    products<N, NT, 1>(m, op + HALF, op);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < Q::U; u++) {
        const int i = tid + u * NT, g = i & 7, o = i >> 3, y = 8 * tile + g;
        if (o >= Q::O || y >= Ly) continue;
        double v[4];
        take<N>(m.y, g, o, v);
#pragma unroll
        for (int k = 0; k < 4; k++) Z[R::point(k, o) * Ly + y] = v[k];
    }
}

// rows after step t (t < 0: the head) and the next step's inputs (N = Ly): tile
// of eight rows
template <int N, int NT>
__device__ __forceinline__ void rows(const RealProblem& p, const double* op, const Shared& m, int ch, int tile, int t) {
    using Q = Tile<N, NT>;
    using R = RealLine<N>;
    constexpr int HALF = Tile<N>::OP;
    const int tid = thread_index();
    const int Lx = p.Lx;
    const long M = (long)Lx * N;
    const RealLane& L = p.lane[ch];
    const bool os2 = p.os2, next = t + 1 < p.Ns;
    constexpr bool HOLD = Q::U == 1;   // longer lines: factors and W are read after the product
    double* const Z = p.Z + ch * M;
    double* const W = p.W + ch * M;
    const double* const* eb = os2 ? L.eF : L.eH;
    const int now = t < 0 ? 0 : lane_block(L, t), nb = lane_block(L, t + 1);
    double e[Q::U][4], q[Q::U][4], w[Q::U][4];
#pragma unroll
    for (int u = 0; u < Q::U; u++) {
        const int i = tid + u * NT, g = i / Q::O, o = i - g * Q::O, r = 8 * tile + g;
        const bool on = i < 8 * Q::O && r < Lx;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            q[u][k] = w[u][k] = e[u][k] = 0.0;
            if (!on) continue;
            const long at = (long)r * N + R::point(k, o);
            if (t < 0) {
                q[u][k] = __ldg(L.hist + at);
                e[u][k] = __ldg(eb[nb] + at);
            } else {
                q[u][k] = __ldcg((os2 ? W : Z) + at);
                if (!HOLD) continue;
                if (!os2) w[u][k] = __ldcg(W + at);
                e[u][k] = __ldg(eb[now] + at);
            }
        }
        if (t >= 0 && i < 8 * Q::O) put<N>(m.x, g, o, q[u]);
    }
    if (t >= 0) {
        __syncthreads();
        products<N, NT, 1>(m, op + (os2 ? 0 : HALF), op);
        __syncthreads();
    }
#pragma unroll
    for (int u = 0; u < Q::U; u++) {
        const int i = tid + u * NT, g = i / Q::O, o = i - g * Q::O, r = 8 * tile + g;
        if (i >= 8 * Q::O) continue;
        if (t >= 0) {
            double v[4];
            take<N>(m.y, g, o, v);
            if (!HOLD && r < Lx)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const long at = (long)r * N + R::point(k, o);
                    if (!os2) w[u][k] = __ldcg(W + at);
                    e[u][k] = __ldg(eb[now] + at);
                }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (os2) q[u][k] = __dmul_rn(v[k], e[u][k]);
                else q[u][k] = next_slice(v[k], w[u][k], e[u][k]);
            }
            if (r < Lx) {
                const long row = (long)r * N;
                if (L.keep_full) {
                    double* full = L.keep_full + (long)t * M + row;
#pragma unroll
                    for (int k = 0; k < 4; k++) full[R::point(k, o)] = w[u][k];
                }
                if (L.src_o)
#pragma unroll
                    for (int k = 0; k < 4; k++) q[u][k] = with_source(L, t + 1, row + R::point(k, o), M, q[u][k]);
                double* out = L.hist + (long)(t + 1) * M + row;
#pragma unroll
                for (int k = 0; k < 4; k++) out[R::point(k, o)] = q[u][k];
            }
            if (next && nb != now && r < Lx)
#pragma unroll
                for (int k = 0; k < 4; k++) e[u][k] = __ldg(eb[nb] + (long)r * N + R::point(k, o));
        }
        if (!next) continue;
        if (os2) {
            if (r < Lx)
#pragma unroll
                for (int k = 0; k < 4; k++) W[(long)r * N + R::point(k, o)] = __dmul_rn(q[u][k], e[u][k]);
            continue;
        }
        double z[4], x[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            z[k] = __dmul_rn(q[u][k], e[u][k]);   // e^{-w ds/4} q
            x[k] = __dmul_rn(z[k], e[u][k]);      // e^{-w ds/2} q
        }
        put<N>(m.x, g, o, z);
        put<N>(m.x + m.xf, g, o, x);
    }
    if (!next || os2) return;
    __syncthreads();
    products<N, NT, 2>(m, op + HALF, op);
    __syncthreads();
#pragma unroll
    for (int u = 0; u < Q::U; u++) {
        const int i = tid + u * NT, g = i / Q::O, o = i - g * Q::O, r = 8 * tile + g;
        if (i >= 8 * Q::O || r >= Lx) continue;
        double v[4];
        take<N>(m.y, g, o, v);
#pragma unroll
        for (int k = 0; k < 4; k++) Z[(long)r * N + R::point(k, o)] = v[k];
        take<N>(m.y + m.yf, g, o, v);
#pragma unroll
        for (int k = 0; k < 4; k++) W[(long)r * N + R::point(k, o)] = v[k];
    }
}

// Rows of long lines in a launch with CTAs to spare: a task is (tile of eight
// rows, one of kParts parts of the output tiles), in two phases with a barrier
// between.  q[t+1] of the part's orbits first.
constexpr int kParts = 4;
template <int N, int NT>
__device__ __forceinline__ void rows_first(const RealProblem& p, const double* op, const Shared& m, int ch, int task, int t) {
    using Q = Tile<N, NT>;
    using R = RealLine<N>;
    constexpr int HALF = Tile<N>::OP, TT = (Q::T + kParts - 1) / kParts;
    const int tid = thread_index();
    const int Lx = p.Lx, tile = task / kParts, tile0 = (task - tile * kParts) * TT;
    const long M = (long)Lx * N;
    const RealLane& L = p.lane[ch];
    const double* const Z = p.Z + ch * M;
    const double* const W = p.W + ch * M;
    const double* const eb = L.eH[lane_block(L, t)];
#pragma unroll
    for (int u = 0; u < Q::U; u++) {
        const int i = tid + u * NT, g = i / Q::O, o = i - g * Q::O, r = 8 * tile + g;
        if (i >= 8 * Q::O) continue;
        double v[4] = {0.0, 0.0, 0.0, 0.0};
        if (r < Lx)
#pragma unroll
            for (int k = 0; k < 4; k++) v[k] = __ldcg(Z + (long)r * N + R::point(k, o));
        put<N>(m.x, g, o, v);
    }
    // the part's orbits: thread (line, orbit)
    static_assert(64 * TT <= NT, "a thread takes one orbit of a part");
    const int g = tid / (8 * TT), o = 8 * tile0 + tid - g * 8 * TT, r = 8 * tile + g;
    const bool on = g < 8 && o < Q::O && r < Lx;
    const long row = (long)r * N;
    double e[4], w[4];
    if (on)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            e[k] = __ldg(eb + row + R::point(k, o));
            w[k] = __ldcg(W + row + R::point(k, o));
        }
    __syncthreads();
    products<N, NT, 1, TT>(m, op + HALF, op, tile0);
    __syncthreads();
    if (!on) return;
    double v[4];
    take<N>(m.y, g, o, v);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const int n = R::point(k, o);
        if (L.keep_full) L.keep_full[(long)t * M + row + n] = w[k];
        double q = next_slice(v[k], w[k], e[k]);
        if (L.src_o) q = with_source(L, t + 1, row + n, M, q);
        L.hist[(long)(t + 1) * M + row + n] = q;
    }
}
// the next step's Z and W at the part's orbits
template <int N, int NT>
__device__ __forceinline__ void rows_second(const RealProblem& p, const double* op, const Shared& m, int ch, int task, int t) {
    using Q = Tile<N, NT>;
    using R = RealLine<N>;
    constexpr int HALF = Tile<N>::OP, TT = (Q::T + kParts - 1) / kParts;
    const int tid = thread_index();
    const int Lx = p.Lx, tile = task / kParts, tile0 = (task - tile * kParts) * TT;
    const long M = (long)Lx * N;
    const RealLane& L = p.lane[ch];
    const double* const q = L.hist + (long)(t + 1) * M;
    const double* const eb = L.eH[lane_block(L, t + 1)];
#pragma unroll
    for (int u = 0; u < Q::U; u++) {
        const int i = tid + u * NT, g = i / Q::O, o = i - g * Q::O, r = 8 * tile + g;
        if (i >= 8 * Q::O) continue;
        double z[4] = {0.0, 0.0, 0.0, 0.0}, x[4] = {0.0, 0.0, 0.0, 0.0};
        if (r < Lx)
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const long at = (long)r * N + R::point(k, o);
                const double e = __ldg(eb + at);
                z[k] = __dmul_rn(__ldcg(q + at), e);
                x[k] = __dmul_rn(z[k], e);
            }
        put<N>(m.x, g, o, z);
        put<N>(m.x + m.xf, g, o, x);
    }
    __syncthreads();
    products<N, NT, 2, TT>(m, op + HALF, op, tile0);
    __syncthreads();
    const int g = tid / (8 * TT), o = 8 * tile0 + tid - g * 8 * TT, r = 8 * tile + g;
    if (g >= 8 || o >= Q::O || r >= Lx) return;
    double v[4];
#pragma unroll
    for (int f = 0; f < 2; f++) {
        take<N>(m.y + f * m.yf, g, o, v);
        double* out = (f ? p.W : p.Z) + ch * M + (long)r * N;
#pragma unroll
        for (int k = 0; k < 4; k++) out[R::point(k, o)] = v[k];
    }
}

#define TS_CASES(X) X(4) X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) TS_LONG(X)
#define TS_LONG(X) X(256) X(352)
constexpr int kLong = 256;

// doubles of a field's folded values and results, for either axis
__host__ __device__ __forceinline__ int x_doubles(int N) { return 32 * pitch_of(4 * ((N / 4 + 3) / 4)); }
__host__ __device__ __forceinline__ int y_doubles(int N) { return 32 * pitch_of(8 * ((N / 4 + 7) / 8)); }
__host__ __device__ __forceinline__ int most(int a, int b) { return a > b ? a : b; }

// MAX: longest line.  CTA b works on chain b / one.ncta, solve by solve (the solves
// at `many`, or `one`).  GRID: one solve, a cooperative launch, a barrier in memory
// for each chain.  Else clusters of one or two chains' CTAs with the hardware's
// barrier, which wait for no other cluster: any number of them may queue.
template <int NT, int PER_SM, int MAX, bool GRID>
__global__ void __launch_bounds__(NT, PER_SM) tile_sweep_kernel(const __grid_constant__ RealProblem one,
                                                                const RealProblem* __restrict__ many) {
    extern __shared__ __align__(16) double sm[];
    __shared__ RealProblem p;
    const int ncta = one.ncta, chain = (int)blockIdx.x / ncta, cta = (int)blockIdx.x - chain * ncta;
    const int ch = chain % one.nl;
    if (many) {
        constexpr int W = sizeof(RealProblem) / 4;
        for (int i = threadIdx.x; i < W; i += NT)
            reinterpret_cast<int*>(&p)[i] = reinterpret_cast<const int*>(many + chain / one.nl)[i];
    } else if (threadIdx.x == 0) {
        p = one;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < p.nfrag; i += NT) sm[i] = p.frag[i];
    const double *opx = sm + p.fo[0], *opy = sm + p.fo[1];
    Shared m;
    m.xf = most(x_doubles(p.Lx), x_doubles(p.Ly));
    m.yf = most(y_doubles(p.Lx), y_doubles(p.Ly));
    m.x = sm + p.nfrag;
    m.y = m.x + 2 * m.xf;
    const int rt = (p.Lx + 7) >> 3, ct = (p.Ly + 7) >> 3;
    unsigned* bar = p.bar + 16 * ch;
    unsigned target = 0;
    auto barrier = [&]() {
        if (!GRID) {
            cluster_barrier();
            return true;
        }
        target += ncta;
        return chain_barrier(bar, p.err, &p.notice, one.hasty, target);
    };
    for (int t = -1; t < p.Ns; t++) {
        if (t >= 0) {
            // orbits past the last one count as zero (the axes' layouts differ)
            if (p.Lx & 15) {
                __syncthreads();
                for (int i = threadIdx.x; i < 2 * m.xf; i += NT) m.x[i] = 0.0;
            }
            for (int k = cta; k < ct; k += ncta) {
                __syncthreads();
                switch (p.Lx) {
#define X(N) case N: if constexpr (N <= MAX) columns<N, NT>(p, opx, m, ch, k, t); break;
                    TS_CASES(X)
#undef X
                }
            }
            if (!barrier()) return;
        }
        if (GRID && p.split) {
            if (t >= 0) {
                for (int k = cta; k < kParts * rt; k += ncta) {
                    __syncthreads();
                    switch (p.Ly) {
#define X(N) case N: if constexpr (GRID) rows_first<N, NT>(p, opy, m, ch, k, t); break;
                        TS_LONG(X)
#undef X
                    }
                }
                if (t + 1 == p.Ns) break;
                if (!barrier()) return;
            }
            for (int k = cta; k < kParts * rt; k += ncta) {
                __syncthreads();
                switch (p.Ly) {
#define X(N) case N: if constexpr (GRID) rows_second<N, NT>(p, opy, m, ch, k, t); break;
                    TS_LONG(X)
#undef X
                }
            }
        } else {
            if (p.Ly & 15) {
                __syncthreads();
                for (int i = threadIdx.x; i < 2 * m.xf; i += NT) m.x[i] = 0.0;
            }
            for (int k = cta; k < rt; k += ncta) {
                __syncthreads();
                switch (p.Ly) {
#define X(N) case N: if constexpr (N <= MAX) rows<N, NT>(p, opy, m, ch, k, t); break;
                    TS_CASES(X)
#undef X
                }
            }
        }
        if (t + 1 < p.Ns) {
            if (!barrier()) return;
        }
    }
}

bool line_ok(int N) {
    switch (N) {
#define X(V) case V:
        TS_CASES(X)
#undef X
        return true;
    }
    return false;
}

size_t tile_smem(int Lx, int Ly, int nfrag) {
    return sizeof(double) * ((size_t)nfrag + 2 * (size_t)most(x_doubles(Lx), x_doubles(Ly)) +
                             2 * (size_t)most(y_doubles(Lx), y_doubles(Ly)));
}

// the forms: one solve's chains over the grid, a cluster a chain, a cluster an image
const auto grid_kernel = tile_sweep_kernel<kNT, 1, 352, true>;
constexpr int kClusterMax = 128;                  // longest axis of the cluster forms
const auto cluster_kernel = tile_sweep_kernel<kNT, 1, kClusterMax, false>;
constexpr int kStringCtas = 4;                    // CTAs a chain, a cluster of 8 an image
const auto string_kernel = tile_sweep_kernel<kStringNT, 3, kClusterMax, false>;

cudaLaunchConfig_t cluster_config(int grid, int nt, int cluster, size_t smem, cudaStream_t st, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3((unsigned)nt, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

}  // namespace

bool tile_sweep_supported(int Lx, int Ly) {
    auto op = [](int N) { return N <= kFragments ? real_frag_doubles(N) : real_parts_doubles(N); };
    return line_ok(Lx) && line_ok(Ly) && tile_smem(Lx, Ly, 2 * (op(Lx) + op(Ly))) <= kSmemLimit;
}

int tile_sweep_fragments() { return kFragments; }

size_t tile_sweep_smem(const RealProblem& p) { return tile_smem(p.Lx, p.Ly, p.nfrag); }

int tile_sweep_tasks(int Lx, int Ly) { return std::max((Ly >= kLong ? kParts : 1) * ((Lx + 7) / 8), (Ly + 7) / 8); }

int tile_sweep_resident(size_t smem) {
    int dev = 0, sms = 0, occ = 0;
    PS_CUDA(cudaGetDevice(&dev));
    PS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PS_CUDA(cudaFuncSetAttribute(grid_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    PS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, grid_kernel, kNT, smem));
    if (occ < 1) throw Error(-2, "sweep kernel does not fit on an SM");
    return sms * occ;
}

void tile_sweep_launch(const RealProblem& p0, int ncta, cudaStream_t st) {
    RealProblem p = p0;
    p.ncta = ncta;
    // long rows in parts where that leaves no CTA two tasks: 128 x 352 13.4 us a step, whole 20.4
    p.split = p.Ly >= kLong && !p.os2 && ncta >= kParts * ((p.Lx + 7) / 8);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(ncta * p.nl), 1, 1);
    cfg.blockDim = dim3(kNT, 1, 1);
    cfg.dynamicSmemBytes = tile_sweep_smem(p);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PS_CUDA(cudaLaunchKernelEx(&cfg, grid_kernel, p, (const RealProblem*)nullptr));
}

int tile_cluster_size(int Lx, int Ly) {
    const int n = tile_sweep_tasks(Lx, Ly);
    return Lx > kClusterMax || Ly > kClusterMax || n > 16 ? 0 : n > 8 ? 16 : 8;
}

int tile_cluster_resident(int cluster, size_t smem) {
    PS_CUDA(cudaFuncSetAttribute(cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    PS_CUDA(cudaFuncSetAttribute(cluster_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cluster_config(cluster, kNT, cluster, smem, nullptr, attr);
    int n = 0;
    PS_CUDA(cudaOccupancyMaxActiveClusters(&n, cluster_kernel, &cfg));
    return n;
}

void tile_cluster_launch(const RealProblem& p, int cluster, cudaStream_t st) {
    RealProblem one = p;
    one.ncta = cluster;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cluster_config(cluster * p.nl, kNT, cluster, tile_sweep_smem(p), st, attr);
    PS_CUDA(cudaLaunchKernelEx(&cfg, cluster_kernel, one, (const RealProblem*)nullptr));
}

void tile_cluster_launch_many(const RealProblem* d, int n, int cluster, size_t smem, cudaStream_t st) {
    RealProblem one{};
    one.nl = 2;
    one.ncta = cluster;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cluster_config(n * 2 * cluster, kNT, cluster, smem, st, attr);
    PS_CUDA(cudaLaunchKernelEx(&cfg, cluster_kernel, one, d));
}

bool tile_string_supported(int Lx, int Ly) {
    return tile_sweep_supported(Lx, Ly) && Lx <= kClusterMax && Ly <= kClusterMax;
}

void tile_string_prepare(const RealProblem& p, int n) {
    const size_t smem = tile_sweep_smem(p);
    PS_CUDA(cudaFuncSetAttribute(string_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cluster_config(n * 2 * kStringCtas, kStringNT, 2 * kStringCtas, smem, nullptr, attr);
    int clusters = 0, per_sm = 0;
    PS_CUDA(cudaOccupancyMaxActiveClusters(&clusters, string_kernel, &cfg));
    PS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, string_kernel, kStringNT, smem));
    char line[200];
    std::snprintf(line, sizeof(line), "grid %dx%dx1 sweep in tiles: %d CTAs per problem, %d CTAs per SM, "
                  "%d clusters resident at once, batch %d\n", p.Lx, p.Ly, 2 * kStringCtas, per_sm, clusters, n);
    tuning_note(line);
}

void tile_string_launch(const RealProblem* d, int n, size_t smem, cudaStream_t st) {
    RealProblem one{};
    one.nl = 2;
    one.ncta = kStringCtas;
    cudaLaunchAttribute attr[1];
    const cudaLaunchConfig_t cfg = cluster_config(n * 2 * kStringCtas, kStringNT, 2 * kStringCtas, smem, st, attr);
    PS_CUDA(cudaLaunchKernelEx(&cfg, string_kernel, one, d));
}

}  // namespace ps
