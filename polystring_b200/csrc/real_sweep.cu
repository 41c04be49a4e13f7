// real_sweep.cu -- persistent RQM4 / OS2 sweep of 3D grids on real line
// operators (real_line.cuh).
//
// For an orthogonal cell the diffusion step F^-1 exp(-h k^2) F / M is the
// product Dx Dy Dz of commuting real line operators, so a chain's slices stay
// real and the two chains of a solve are independent real fields.  A contour
// step (RQM4.cc:66-92) is two grid-wide phases with a barrier after each:
//
//   x-pass   (columns (y, z), warp tasks of 8): Dx of the full step on W; Dx of
//            the first half step on Z, times e^{-w ds/2} (the two quarter-step
//            factors between the half steps), Dx of the second half step on Z
//   plane    (CTA tasks: slab x of one chain): columns: Dy of the second half
//            step on Z and Dy of the full step on W, into shared memory | rows:
//            Dz on Z, q[t+1] = (4 e^{-w ds/4} Z - e^{-w ds/2} W) / 3 -> history,
//            next inputs Dz(full) e^{-w ds/2} q -> W and Dz(half) e^{-w ds/4} q
//            | columns: Dy(half) -> Z
//
// W and Z are updated in place: an x-pass task owns its columns, a plane task
// its slab.  OS2 (PseudoSpectral.cc:248-260) has only W, with its Dz before q.  The operators carry
// the 1/M of the inverse transforms.  Every line of an operator is owned by
// one warp, whose arithmetic does not depend on how tasks are spread over warps
// and CTAs: a solve in a shared launch equals its single launch bit for bit.
//
// us a contour step, RQM4 both chains: 16^3 5.7, 32^3 7.3 (38 with packed complex
// FFTs in four phases), 48^3 12.3 (57), 64^3 17.5 (21.2 in clusters of two CTAs), 48 x
// 64 x 32 10.4 (one chain in a launch per line pass: 29).  What bounds it: small grids the two
// barriers (1.4 us and the slowest CTA each) and the phases' chains of L2 reads,
// products and writes; 64^3 the L2, which the x-pass reads and writes at 6 TB/s
// (7300 cycles of which 5300 remain without arithmetic), and the products of the
// plane, 40 % of the FP64 tensor peak while they run.  One CTA of 256 threads an SM:
// with 255 registers each the next operands are prefetched; 512 threads spill, two
// CTAs an SM gain nothing alone (19 to 20 us at 64^3), a barrier a field costs 10.2 us
// at 32^3, two columns a lane 19.1 at 64^3.  The kernel spills 2.1 KB a thread, all of it
// in the branches of 96 and 128 points; the one of shared launches, at 128 registers, 0.5 KB.
//
// Barriers (sweep_barrier.cuh) count arrivals per chain with a bounded spin; the launch
// is cooperative, so all CTAs are resident.  On a timeout the CTA raises the error
// flag, every CTA of the solve sees it and returns, and the host finds a word in its
// own memory set: RealSweep::check.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <tuple>

#include "engine.h"
#include "ps_internal.h"
#include "fft_core.cuh"
#include "real_line.cuh"
#include "real_sweep.h"
#include "sweep_barrier.cuh"

namespace ps {

namespace {

constexpr int kNT = 256;                     // threads a CTA
constexpr size_t kSmemLimit = 227 * 1024 - 1024;

// row pitch of a slab in shared memory: 4 mod 8 doubles, so that the 4 rows x 4
// consecutive values of a half warp fall in different banks, by rows and by
// columns
__host__ __device__ __forceinline__ int slab_pitch(int Lz) { return Lz + ((Lz & 7) == 4 ? 0 : 4); }

// values a lane holds of a line
__host__ __device__ __forceinline__ int line_values(int N) { return 4 * ((N / 4 + 3) / 4); }

__device__ __forceinline__ int lane_block(const RealLane& c, int t) { return t < c.sw[0] ? 0 : t < c.sw[1] ? 1 : 2; }

// A warp's eight lines: line g of the tile at element offset lo (a valid line
// also for lanes past the last one, whose results are not stored), stride st
// between the points of a line; f(offset) reads, f(offset, value) writes.
template <int N, class F>
__device__ __forceinline__ void load_lines(double (&x)[RealLine<N>::E], int j, F f) {
    using R = RealLine<N>;
#pragma unroll
    for (int s = 0; s < R::S; s++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int o = j + 4 * s;
            x[4 * s + i] = (R::WHOLE || o < R::O) ? f(R::point(i, o)) : 0.0;
        }
}
template <int N, class F>
__device__ __forceinline__ void each_point(int j, F f) {
    using R = RealLine<N>;
#pragma unroll
    for (int s = 0; s < R::S; s++)
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int o = j + 4 * s;
            if (R::WHOLE || o < R::O) f(4 * s + i, R::point(i, o));
        }
}

// x-pass of chain ch: warp w of nw takes tasks of p.xcols columns
template <int N>
__device__ __forceinline__ void x_pass(const RealProblem& p, const double* fr, double* cache, int ch, int t, int w,
                                       int nw) {
    using R = RealLine<N>;
    const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const int P = p.Ly * p.Lz;
    const long M = (long)N * P;
    const int ntile = (P + p.xcols - 1) / p.xcols;
    const int total = p.os2 ? ntile : 2 * ntile;   // Z tasks first: they are the longer ones
    const bool fresh = t == 0 || lane_block(p.lane[ch], t) != lane_block(p.lane[ch], t - 1);
    double* keep = cache + (threadIdx.x >> 5) * (R::E * 32) * p.xkeep + lane;
    for (int task = w; task < total; task += nw) {
        const bool half = !p.os2 && task < ntile;
        const int c0 = (half || p.os2 ? task : task - ntile) * p.xcols;
        for (int c8 = c0; c8 < min(c0 + p.xcols, P); c8 += 8) {
            const bool ok = c8 + g < P;
            const int c = ok ? c8 + g : c8;
            double* Z = (half ? p.Z : p.W) + ch * M + c;
            double x[R::E];
            load_lines<N>(x, j, [&](int n) { return __ldcg(Z + n * P); });
            if (half) {
                // the factors are on their way while the first operator runs
                const RealLane& L = p.lane[ch];
                const double* e = L.eF[lane_block(L, t)] + c;
                double f[R::E];
                if (p.xkeep == 0) {
                    load_lines<N>(f, j, [&](int n) { return __ldg(e + n * P); });
                } else {
                    if (fresh) {
                        load_lines<N>(f, j, [&](int n) { return __ldg(e + n * P); });
#pragma unroll
                        for (int i = 0; i < R::E; i++) keep[32 * i] = f[i];
                    } else {
#pragma unroll
                        for (int i = 0; i < R::E; i++) f[i] = keep[32 * i];
                    }
                    keep += 32 * R::E;
                }
                R::apply(x, fr + R::FRAG + lane);
                if (L.keep_half && ok) {
                    double* out = L.keep_half + (long)t * M + c;
                    each_point<N>(j, [&](int k, int n) { out[n * P] = x[k]; });
                }
#pragma unroll
                for (int i = 0; i < R::E; i++) x[i] = __dmul_rn(x[i], f[i]);
                R::apply(x, fr + R::FRAG + lane);
            } else {
                R::apply(x, fr + lane);
            }
            if (ok) each_point<N>(j, [&](int k, int n) { Z[n * P] = x[k]; });
        }
    }
}

// first stage of a plane task: Dy of Z (half step, into A) and of W (full
// step, into B)
template <int N>
__device__ __forceinline__ void plane_columns_in(const RealProblem& p, const double* fr, double* A, double* B, int slab,
                                              int ch) {
    using R = RealLine<N>;
    const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const int Lz = p.Lz, pz = slab_pitch(Lz), nt = (Lz + 7) >> 3;
    const long off = ((long)ch * p.Lx + slab) * N * Lz;
    for (int k = threadIdx.x >> 5; k < (p.os2 ? nt : 2 * nt); k += blockDim.x >> 5) {
        const bool half = !p.os2 && k < nt;
        const int z8 = (half || p.os2 ? k : k - nt) * 8;
        const bool ok = z8 + g < Lz;
        const int z = ok ? z8 + g : z8;
        const double* src = (half ? p.Z : p.W) + off + z;
        double* dst = (half ? A : B) + z;
        double x[R::E];
        load_lines<N>(x, j, [&](int n) { return __ldcg(src + n * Lz); });
        R::apply(x, fr + (half ? R::FRAG : 0) + lane);
        if (ok) each_point<N>(j, [&](int k2, int n) { dst[n * pz] = x[k2]; });
    }
}

// rows: q[t+1] from A and B (t < 0: the chain's head), the history, the next W
// and the rows of the next half-step input (into A)
template <int N>
__device__ __forceinline__ void plane_rows(const RealProblem& p, const double* fr, double* A, const double* B,
                                           double* cache, int slab, int ch, int t) {
    using R = RealLine<N>;
    const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const int Ly = p.Ly, pz = slab_pitch(N), nt = (Ly + 7) >> 3;
    const long M = (long)p.Lx * Ly * N;
    const RealLane& L = p.lane[ch];
    const bool next = t + 1 < p.Ns;
    for (int k = threadIdx.x >> 5; k < nt; k += blockDim.x >> 5) {
        const bool ok = 8 * k + g < Ly;
        const int y = ok ? 8 * k + g : 8 * k;
        const long row = ((long)slab * Ly + y) * N;
        double* a = A + y * pz;
        const double* b = B + y * pz;
        // the rows' factors, e^{-w ds/4} (OS2: e^{-w ds/2}), of a block
        double* keep = cache + k * (R::E * 32) + lane;
        auto factors = [&](double (&h)[R::E], int blk, bool kept) {
            if (p.rkeep && kept) {
#pragma unroll
                for (int i = 0; i < R::E; i++) h[i] = keep[32 * i];
                return;
            }
            const double* e = (p.os2 ? L.eF[blk] : L.eH[blk]) + row;
            load_lines<N>(h, j, [&](int n) { return __ldg(e + n); });
            if (p.rkeep) {
#pragma unroll
                for (int i = 0; i < R::E; i++) keep[32 * i] = h[i];
            }
        };
        const int now = t < 0 ? -1 : lane_block(L, t), nb = lane_block(L, t + 1);
        double q[R::E];
        if (t < 0) {
            load_lines<N>(q, j, [&](int n) { return __ldg(L.hist + row + n); });
        } else {
            double* out = L.hist + (long)(t + 1) * M + row;
            double h[R::E];   // on their way while the operator runs
            factors(h, now, true);
            if (p.os2) {
                load_lines<N>(q, j, [&](int n) { return b[n]; });
                R::apply(q, fr + lane);
#pragma unroll
                for (int i = 0; i < R::E; i++) q[i] = __dmul_rn(q[i], h[i]);
            } else {
                load_lines<N>(q, j, [&](int n) { return a[n]; });
                R::apply(q, fr + R::FRAG + lane);
                each_point<N>(j, [&](int i, int n) {
                    const double v = __dmul_rn(q[i], h[i]), u = __dmul_rn(b[n], __dmul_rn(h[i], h[i]));
                    q[i] = div_rn(fma(4.0, v, -u), 3.0, 1.0 / 3.0);
                });
                if (L.keep_full && ok) {
                    double* full = L.keep_full + (long)t * M + row;
                    each_point<N>(j, [&](int i, int n) { full[n] = b[n]; });
                }
                if (L.src_o) {
                    const double wa = L.src_w[0][t + 1], wb = L.src_w[1][t + 1];
                    const double* o = L.src_o + (long)(t + 1) * M + row;
                    each_point<N>(j, [&](int i, int n) {
                        q[i] = fma(fma(wa, __ldg(L.src_p[0] + row + n), wb * __ldg(L.src_p[1] + row + n)), __ldg(o + n), q[i]);
                    });
                }
            }
            if (ok) each_point<N>(j, [&](int i, int n) { out[n] = q[i]; });
        }
        if (next) {
            double x[R::E];
            factors(x, nb, nb == now);
            double* W = p.W + ch * M + row;
            if (p.os2) {
                if (ok) each_point<N>(j, [&](int i, int n) { W[n] = __dmul_rn(x[i], q[i]); });
                continue;
            }
#pragma unroll
            for (int i = 0; i < R::E; i++) {
                q[i] = __dmul_rn(q[i], x[i]);   // e^{-w ds/4} q, and e^{-w ds/2} q = e^{-w ds/4} (e^{-w ds/4} q)
                x[i] = __dmul_rn(x[i], q[i]);
            }
            R::apply(x, fr + lane);
            if (ok) each_point<N>(j, [&](int i, int n) { W[n] = x[i]; });
            R::apply(q, fr + R::FRAG + lane);
            if (ok) each_point<N>(j, [&](int i, int n) { a[n] = q[i]; });
        }
    }
}

// columns: Dy of the next half-step input (A) -> Z
template <int N>
__device__ __forceinline__ void plane_columns_out(const RealProblem& p, const double* fr, const double* A, int slab,
                                               int ch) {
    using R = RealLine<N>;
    const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const int Lz = p.Lz, pz = slab_pitch(Lz), nt = (Lz + 7) >> 3;
    double* dst = p.Z + ((long)ch * p.Lx + slab) * N * Lz;
    for (int k = threadIdx.x >> 5; k < nt; k += blockDim.x >> 5) {
        const bool ok = 8 * k + g < Lz;
        const int z = ok ? 8 * k + g : 8 * k;
        double x[R::E];
        load_lines<N>(x, j, [&](int n) { return A[n * pz + z]; });
        R::apply(x, fr + R::FRAG + lane);
        if (ok) each_point<N>(j, [&](int i, int n) { dst[n * Lz + z] = x[i]; });
    }
}

// line lengths of the kernel at two CTAs an SM (at most 64 points: 128
// registers a thread hold an operator's 16 inputs, 8 results of two blocks and
// 16 factors) and of the one at one CTA an SM
#define RS_CASES_64(X) X(4) X(8) X(12) X(16) X(24) X(32) X(48) X(64)
#define RS_CASES_128(X) RS_CASES_64(X) X(96) X(128)

template <bool WIDE>
__device__ __forceinline__ void run_x(const RealProblem& p, const double* fr, double* cache, int ch, int t, int w,
                                      int nw) {
    switch (p.Lx) {
#define X(N) case N: x_pass<N>(p, fr, cache, ch, t, w, nw); break;
        RS_CASES_64(X)
#undef X
        default:
            if constexpr (WIDE) {
                if (p.Lx == 96) x_pass<96>(p, fr, cache, ch, t, w, nw);
                else x_pass<128>(p, fr, cache, ch, t, w, nw);
            }
    }
}
template <bool WIDE>
__device__ __forceinline__ void run_columns_in(const RealProblem& p, const double* fr, double* A, double* B, int slab,
                                               int ch) {
    switch (p.Ly) {
#define X(N) case N: plane_columns_in<N>(p, fr, A, B, slab, ch); break;
        RS_CASES_64(X)
#undef X
        default:
            if constexpr (WIDE) {
                if (p.Ly == 96) plane_columns_in<96>(p, fr, A, B, slab, ch);
                else plane_columns_in<128>(p, fr, A, B, slab, ch);
            }
    }
}
template <bool WIDE>
__device__ __forceinline__ void run_rows(const RealProblem& p, const double* fr, double* A, const double* B,
                                         double* cache, int slab, int ch, int t) {
    switch (p.Lz) {
#define X(N) case N: plane_rows<N>(p, fr, A, B, cache, slab, ch, t); break;
        RS_CASES_64(X)
#undef X
        default:
            if constexpr (WIDE) {
                if (p.Lz == 96) plane_rows<96>(p, fr, A, B, cache, slab, ch, t);
                else plane_rows<128>(p, fr, A, B, cache, slab, ch, t);
            }
    }
}
template <bool WIDE>
__device__ __forceinline__ void run_columns_out(const RealProblem& p, const double* fr, const double* A, int slab,
                                                int ch) {
    switch (p.Ly) {
#define X(N) case N: plane_columns_out<N>(p, fr, A, slab, ch); break;
        RS_CASES_64(X)
#undef X
        default:
            if constexpr (WIDE) {
                if (p.Ly == 96) plane_columns_out<96>(p, fr, A, slab, ch);
                else plane_columns_out<128>(p, fr, A, slab, ch);
            }
    }
}

// many == nullptr: the solve `one`; else the solves many[0 .. n).  A solve's
// chains are independent: each has its own CTAs and barrier.  ONE: one CTA an
// SM, all line lengths; else two CTAs an SM and lines of at most 64 points.
template <bool ONE>
__global__ void __launch_bounds__(kNT, ONE ? 1 : 2) real_sweep_kernel(const __grid_constant__ RealProblem one,
                                                                       const RealProblem* __restrict__ many, int n) {
    extern __shared__ __align__(16) double sm[];
    __shared__ RealProblem p;
    __shared__ int which;
    if (many) {
        for (int i = threadIdx.x; i < n; i += kNT) {
            const int c = (int)blockIdx.x - many[i].cta0;
            if (c >= 0 && c < many[i].ncta * many[i].nl) which = i;
        }
        __syncthreads();
        constexpr int W = sizeof(RealProblem) / 4;
        for (int i = threadIdx.x; i < W; i += kNT)
            reinterpret_cast<int*>(&p)[i] = reinterpret_cast<const int*>(many + which)[i];
    } else if (threadIdx.x == 0) {
        p = one;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < p.nfrag; i += kNT) sm[i] = p.frag[i];
    const double *frx = sm + p.fo[0], *fry = sm + p.fo[1], *frz = sm + p.fo[2];
    double* A = sm + p.nfrag;
    double* B = A + p.Ly * slab_pitch(p.Lz);
    // factors kept by the lanes that use them: of the x-pass tasks, then of the rows
    double* xcache = B + p.Ly * slab_pitch(p.Lz);
    double* rcache = xcache + p.xkeep * (kNT / 32) * 32 * line_values(p.Lx);
    __syncthreads();

    const int ncta = p.ncta;
    const int ch = ((int)blockIdx.x - p.cta0) / ncta, cta = (int)blockIdx.x - p.cta0 - ch * ncta;
    // x-pass warp index, CTA-fastest, so that a phase's tasks spread over all SMs
    const int w = (threadIdx.x >> 5) * ncta + cta, nw = ncta * (kNT / 32);
    unsigned* bar = p.bar + 16 * ch;
    unsigned target = 0;
    for (int t = -1; t < p.Ns; t++) {
        if (t >= 0) {
            run_x<ONE>(p, frx, xcache, ch, t, w, nw);
            target += ncta;
            if (!chain_barrier(bar, p.err, &p.notice, one.hasty, target)) return;
        }
        for (int slab = cta; slab < p.Lx; slab += ncta) {
            if (t >= 0) {
                run_columns_in<ONE>(p, fry, A, B, slab, ch);
                __syncthreads();
            }
            run_rows<ONE>(p, frz, A, B, rcache, slab, ch, t);
            __syncthreads();
            if (t + 1 < p.Ns && !p.os2) {
                run_columns_out<ONE>(p, fry, A, slab, ch);
                __syncthreads();
            }
        }
        if (t + 1 < p.Ns) {
            target += ncta;
            if (!chain_barrier(bar, p.err, &p.notice, one.hasty, target)) return;
        }
    }
}

size_t smem_bytes(int Ly, int Lz, int nfrag) {
    return sizeof(double) * ((size_t)nfrag + 2 * (size_t)Ly * slab_pitch(Lz));
}

// shared memory of the kept factors
size_t xkeep_bytes(int Lx, int xkeep) { return sizeof(double) * (size_t)xkeep * kNT * line_values(Lx); }
size_t rkeep_bytes(int Ly, int Lz) { return sizeof(double) * (size_t)((Ly + 7) / 8) * 32 * line_values(Lz); }

bool line_ok(int N) {
    switch (N) {
#define X(V) case V:
        RS_CASES_128(X)
#undef X
        return true;
    }
    return false;
}

bool wide(int Lx, int Ly, int Lz) { return std::max(Lx, std::max(Ly, Lz)) > 64; }

cudaLaunchConfig_t launch_config(size_t smem, int grid, cudaStream_t st, cudaLaunchAttribute* attr) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(kNT, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cfg;
}

void launch(const RealProblem& p, const RealProblem* d, int n, size_t smem, bool one, int grid, cudaStream_t st) {
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = launch_config(smem, grid, st, attr);
    if (one) PS_CUDA(cudaLaunchKernelEx(&cfg, real_sweep_kernel<true>, p, d, n));
    else PS_CUDA(cudaLaunchKernelEx(&cfg, real_sweep_kernel<false>, p, d, n));
}

}  // namespace

std::vector<double> real_operator_tables(const int n[3], const double k[3], double ds, int fragments, int fo[3]) {
    std::vector<double> out;
    for (int a = 0; a < 3; a++) {
        fo[a] = -1;
        if (n[a] == 1) continue;
        for (int b = 0; b < a; b++)
            if (n[b] == n[a] && k[b] == k[a]) fo[a] = fo[b];
        if (fo[a] >= 0) continue;
        fo[a] = (int)out.size();
        for (double h : {ds, 0.5 * ds}) {
            std::vector<double> L(n[a]);
            for (int i = 0; i < n[a]; i++) {
                const int r = i < n[a] / 2 + 1 ? i : n[a] - i;
                L[i] = exp(h * (k[a] * r * r));
            }
            if (n[a] > fragments) real_parts(n[a], L, out);
            else real_fragments(n[a], L, out);
        }
    }
    return out;
}

bool real_sweep_supported(int Lx, int Ly, int Lz) {
    return line_ok(Lx) && line_ok(Ly) && line_ok(Lz) &&
           smem_bytes(Ly, Lz, 2 * (real_frag_doubles(Lx) + real_frag_doubles(Ly) + real_frag_doubles(Lz))) <= kSmemLimit;
}

size_t real_sweep_smem(const RealProblem& p) { return smem_bytes(p.Ly, p.Lz, p.nfrag); }
bool real_sweep_wide(const RealProblem& p) { return wide(p.Lx, p.Ly, p.Lz); }

// sets the kernels' attributes; the SMs of the device
static int prepare_kernels() {
    int dev = 0, sms = 0;
    PS_CUDA(cudaGetDevice(&dev));
    PS_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    PS_CUDA(cudaFuncSetAttribute(real_sweep_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    PS_CUDA(cudaFuncSetAttribute(real_sweep_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit));
    return sms;
}

int real_sweep_resident(size_t smem, bool one) {
    const int sms = prepare_kernels();
    int occ = 0;
    if (one) PS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, real_sweep_kernel<true>, kNT, smem));
    else PS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, real_sweep_kernel<false>, kNT, smem));
    if (occ < 1) throw Error(-2, "sweep kernel does not fit on an SM");
    return sms * occ;
}

int real_sweep_tasks(int Lx, int Ly, int Lz) {
    const int xt = 2 * ((Ly * Lz + 7) / 8);
    return std::max(Lx, (xt + kNT / 32 - 1) / (kNT / 32));
}

int real_sweep_columns(int variant) { return 8 << variant; }

void real_sweep_launch(const RealProblem& p0, int ncta, cudaStream_t st) {
    RealProblem p = p0;
    p.cta0 = 0;
    p.ncta = ncta;
    // where the shared memory allows it, factors stay there while a chain runs
    // through a block: the rows' when a CTA has one slab, the x-pass's of tasks
    // of 8 columns
    size_t smem = smem_bytes(p.Ly, p.Lz, p.nfrag);
    p.rkeep = ncta >= p.Lx && smem + rkeep_bytes(p.Ly, p.Lz) <= kSmemLimit;
    if (p.rkeep) smem += rkeep_bytes(p.Ly, p.Lz);
    const int nw = ncta * (kNT / 32), xkeep = ((p.Ly * p.Lz + 7) / 8 + nw - 1) / nw;
    p.xkeep = !p.os2 && p.xcols == 8 && smem + xkeep_bytes(p.Lx, xkeep) <= kSmemLimit ? xkeep : 0;
    smem += xkeep_bytes(p.Lx, p.xkeep);
    launch(p, nullptr, 0, smem, true, ncta * p.nl, st);
}

void real_sweep_launch_many(const RealProblem* d, int n, size_t smem, bool one, int grid, int hasty, cudaStream_t st) {
    RealProblem all{};
    all.hasty = hasty;
    launch(all, d, n, smem, one, grid, st);
}

// ---------------------------------------------------------------------------
// RealSweep
// ---------------------------------------------------------------------------
// Words of pinned host memory that kernels of every device can write, one a sweep
// alive.  A sweep returns its word for the next; a page of them (of 1024) stays for the
// process: a page each would cost every construction 2 ms.
namespace {
class Notices {
public:
    int* take() {
        std::lock_guard<std::mutex> lock(mu_);
        if (free_.empty()) {
            int* page = nullptr;
            PS_CUDA(cudaHostAlloc(&page, 1024 * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
            for (int i = 1023; i >= 0; i--) free_.push_back(page + i);
        }
        int* w = free_.back();
        free_.pop_back();
        *w = 0;
        return w;
    }
    void give(int* w) {
        std::lock_guard<std::mutex> lock(mu_);
        free_.push_back(w);
    }

private:
    std::mutex mu_;
    std::vector<int*> free_;
};
Notices& notices() {
    static Notices* n = new Notices;   // objects may be destroyed after statics are
    return *n;
}
}  // namespace

bool RealSweep::supported(int Lx, int Ly, int Lz) {
    if (Ly == 1 && Lz == 1) return line_sweep_supported(Lx);
    if (Lz == 1) return plane_sweep_supported(Lx, Ly) || tile_sweep_supported(Lx, Ly);
    return real_sweep_supported(Lx, Ly, Lz);
}

RealSweep::RealSweep(const int n[3], const double k[3], double ds, int nl, bool os2) : nl_(nl), os2_(os2) {
    try {
        init(n, k, ds, nl, os2);
    } catch (...) {
        release();
        throw;
    }
}

void RealSweep::init(const int n[3], const double k[3], double ds, int nl, bool os2) {
    std::copy(n, n + 3, n_);
    dim_ = n[2] > 1 ? 3 : n[1] > 1 ? 2 : 1;
    const size_t M = (size_t)n[0] * n[1] * n[2];
    variant_ = 0;
    ncta_ = 0;
    const bool plane = dim_ == 2 && plane_sweep_supported(n[0], n[1]);
    // a single solve's chains in tiles over many CTAs where that is faster than a CTA
    // a chain (us a step, tiles against one CTA: RQM4 64^2 4.4 / 9.1, 48^2 4.2 / 5.4,
    // 32 x 64 3.8 / 4.3, 32^2 3.5 / 2.3; OS2 64^2 3.2 / 5.1, 48^2 3.1 / 3.1, 32 x 64 3.0 / 2.5)
    tile_ = dim_ == 2 && (!plane || n[0] * n[1] >= (os2 ? 48 * 64 : 32 * 64));
    const std::vector<double> f = real_operator_tables(n, k, ds, dim_ == 1 ? 0 : dim_ == 2 ? tile_sweep_fragments() : 1 << 30, fo_);
    nfrag_ = (int)f.size();
    if (dim_ == 3) {
        ncta_ = std::max(1, std::min(prepare_kernels() / nl, real_sweep_tasks(n[0], n[1], n[2])));
        PS_CUDA(cudaMalloc(&work_, sizeof(double) * 2 * nl * M));
    }
    if (plane) plane_sweep_prepare();
    if (tile_) {
        const size_t smem = tile_sweep_smem(problem(nullptr, 0));
        cluster_ = tile_cluster_size(n[0], n[1]);
        if (cluster_ && tile_cluster_resident(cluster_, smem) < 1) cluster_ = 0;
        if (!cluster_) ncta_ = std::max(1, std::min(tile_sweep_resident(smem) / nl, tile_sweep_tasks(n[0], n[1])));
        PS_CUDA(cudaMalloc(&work_, sizeof(double) * 2 * nl * M));
    }
    PS_CUDA(cudaMalloc(&frag_, sizeof(double) * f.size()));
    upload(frag_, f.data(), sizeof(double) * f.size());
    PS_CUDA(cudaMalloc(&bar_, 33 * sizeof(unsigned)));
    const unsigned zeros[33] = {};
    upload(bar_, zeros, sizeof(zeros));
    if (dim_ == 3 || (tile_ && !cluster_)) notice_ = notices().take();
    const char* hasty = getenv("PS_B200_BARRIER_GIVE_UP");
    hasty_ = hasty && hasty[0] == '1';
}

RealSweep::~RealSweep() { release(); }

void RealSweep::release() {
    cudaFree(work_);
    cudaFree(frag_);
    cudaFree(bar_);
    if (notice_) notices().give(notice_);
}

RealProblem RealSweep::problem(const RealLane* lanes, int Ns) const {
    const size_t M = (size_t)n_[0] * n_[1] * n_[2];
    RealProblem p{};
    if (lanes) std::copy(lanes, lanes + nl_, p.lane);
    p.W = work_;
    p.Z = work_ + nl_ * M;
    p.frag = frag_;
    std::copy(fo_, fo_ + 3, p.fo);
    p.nfrag = nfrag_;
    p.bar = bar_;
    p.err = reinterpret_cast<int*>(bar_ + 32);
    p.notice = notice_;
    p.hasty = hasty_;
    p.Lx = n_[0]; p.Ly = n_[1]; p.Lz = n_[2];
    p.Ns = Ns;
    p.nl = nl_;
    p.os2 = os2_;
    p.xcols = real_sweep_columns(variant_);
    return p;
}

void RealSweep::enqueue(const RealProblem& p, cudaStream_t st) const {
    if (dim_ == 1) return line_sweep_launch(p, st);
    if (dim_ == 2 && !tile_) return plane_sweep_launch(p, st);
    if (cluster_) return tile_cluster_launch(p, cluster_, st);
    PS_CUDA(cudaMemsetAsync(bar_, 0, 32 * sizeof(unsigned), st));
    if (tile_) return tile_sweep_launch(p, ncta_, st);
    real_sweep_launch(p, ncta_, st);
}

bool RealSweep::failed() const { return notice_ && *((volatile int*)notice_); }

void RealSweep::check() const {
    if (failed()) throw Error(-3, "a propagator sweep gave up at a grid barrier (its CTAs were not all running)");
}

void RealSweep::reset() {
    if (!failed()) return;
    PS_CUDA(cudaDeviceSynchronize());   // a sweep still queued stops at the flag without a notice of its own
    const unsigned zero = 0;
    upload(bar_ + 32, &zero, sizeof(zero));
    *((volatile int*)notice_) = 0;
}

// Single Model_AB solves are tuned.  Updaters, triblocks and batch members keep 8 columns,
// the choice at most grids, rather than pay the timing at their construction.
void RealSweep::tune(const RealProblem& p0, cudaStream_t st) {
    if (dim_ < 3) return;
    const char* force = getenv("PS_B200_SWEEP_VARIANT");
    if (force && force[0] >= '0' && force[0] < '0' + kRealVariants) {
        variant_ = force[0] - '0';
        return;
    }
    const char* at = getenv("PS_B200_AUTOTUNE");
    if (at && at[0] == '0') return;
    static std::mutex mu;
    static std::map<std::tuple<int, int, int, int, int, int>, int> cache;   // (device, grid, chains, scheme) -> variant
    int dev = 0;
    PS_CUDA(cudaGetDevice(&dev));
    const auto key = std::make_tuple(dev, n_[0], n_[1], n_[2], nl_, os2_);
    std::lock_guard<std::mutex> lock(mu);
    auto it = cache.find(key);
    if (it != cache.end()) {
        variant_ = it->second;
        return;
    }
    cudaEvent_t e0, e1;
    PS_CUDA(cudaEventCreate(&e0));
    PS_CUDA(cudaEventCreate(&e1));
    RealProblem p = p0;
    p.Ns = std::min(p.Ns, 24);   // enough to tell the variants apart (64^3: 5 ms in all, 43 with 200 steps)
    double best = 1e30;
    char line[512];
    int n = std::snprintf(line, sizeof(line), "grid %dx%dx%d persistent sweep, x-tile columns (us per step):", n_[0],
                          n_[1], n_[2]);
    int pick = 0;
    for (int v = 0; v < kRealVariants; v++) {
        p.xcols = real_sweep_columns(v);
        enqueue(p, st);
        PS_CUDA(cudaEventRecord(e0, st));
        for (int r = 0; r < 3; r++) enqueue(p, st);
        PS_CUDA(cudaEventRecord(e1, st));
        PS_CUDA(cudaEventSynchronize(e1));
        float ms = 0.f;
        PS_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        const double us = 1e3 * ms / 3.0 / p.Ns;
        if (n > 0 && n < (int)sizeof(line)) n += std::snprintf(line + n, sizeof(line) - n, " %d=%.1f", p.xcols, us);
        if (us < best) {
            best = us;
            pick = v;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    check();
    variant_ = pick;
    if (n > 0 && n < (int)sizeof(line))
        std::snprintf(line + n, sizeof(line) - n, " -> %d\n", real_sweep_columns(pick));
    tuning_note(line);
    cache[key] = pick;
}

}  // namespace ps
