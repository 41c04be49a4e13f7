// etdrk4.cu -- the ETDRK4 propagator step (Etdrk4_PBC.cc:110-184) for two
// real chains packed into one complex field (lane f in the real part, lane c
// in the imaginary part).
//
// Cox-Matthews ETDRK4 with the Kassam-Trefethen coefficients: the spectrum v
// of the chain is carried from step to step, and each step is
//     Nv = F[-w q_s]
//     a  = E2 v + Q Nv              Na = F[-w Re(F^-1 a) / M]
//     b  = E2 v + Q Na              Nb = F[-w Re(F^-1 b) / M]
//     c  = E2 a + Q (2 Nb - Nv)     Nc = F[-w Re(F^-1 c) / M]
//     v  = E v + f1 Nv + 2 f2 (Na + Nb) + f3 Nc
//     q_{s+1} = Re(F^-1 v) / M
// with E = exp(ds L), E2 = exp(ds L / 2) and L = -k^2 (calc_k2_orthogonal).
// Every spectral operation multiplies by real tables that are even in k, so
// the packed field carries both lanes' spectra at once; the nonlinear term
// takes each lane's own w.  Grids of up to 1536 points of 1D and 2D run all
// steps in one CTA (etd_small_kernel); on others a stage is two (2D) or four
// (3D) passes (etd_pass_kernel).
#include "engine.h"
#include "fft_core.cuh"
#include "ps_internal.h"
#include "line_pass_body.cuh"

#include <cmath>
#include <complex>
#include <cstdlib>

namespace ps {

namespace {

constexpr int kEtdThreads = 256;

inline unsigned etd_blocks(long n) {
    long b = (n + kEtdThreads - 1) / kEtdThreads;
    return (unsigned)(b < 148 * 16 ? b : 148 * 16);
}

// T = qf + i qc (a chain's spectrum from its real slices: init) or
// T = -(wf qf) - i (wc qc) (the nonlinear term of the slices: Nv)
__global__ void etd_slices_kernel(double2* __restrict__ T, const double* __restrict__ qf,
                                  const double* __restrict__ qc, const double* __restrict__ wf,
                                  const double* __restrict__ wc, long M, int nonlin) {
    for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < M; m += (long)gridDim.x * blockDim.x) {
        const double xf = qf[m], xc = qc[m];
        T[m] = nonlin ? make_double2(-wf[m] * xf, -wc[m] * xc) : make_double2(xf, xc);
    }
}

// T = -(wf Re(T) / M) - i (wc Im(T) / M): the nonlinear term of an inverse
// transform (Etdrk4_PBC.cc, x = Re(b) / M)
__global__ void etd_nonlin_kernel(double2* __restrict__ T, const double* __restrict__ wf,
                                  const double* __restrict__ wc, long M, double rM) {
    for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < M; m += (long)gridDim.x * blockDim.x) {
        const double2 t = T[m];
        const double xf = t.x / rM, xc = t.y / rM;
        T[m] = make_double2(-wf[m] * xf, -wc[m] * xc);
    }
}

struct EtdFields {
    double2 *T, *V, *Nv, *A, *Na, *Nb;
    const double *E, *E2, *Q, *f1, *f2, *f3;
};

__device__ __forceinline__ double2 lin2(double a, double2 x, double b, double2 y) {
    return make_double2(a * x.x + b * y.x, a * x.y + b * y.y);
}

// the spectral stages of one step; T holds the forward transform of the
// stage's nonlinear term on entry and the next spectrum to invert on exit
//   0: Nv = T; a = E2 v + Q Nv; T = a
//   1: Na = T; T = E2 v + Q Na
//   2: Nb = T; T = E2 a + Q (2 Nb - Nv)
//   3: v = E v + f1 Nv + 2 f2 (Na + Nb) + f3 T; T = v
__device__ __forceinline__ double2 etd_combine(const EtdFields& f, long m, int stage, double2 t) {
    if (stage == 0) {
        f.Nv[m] = t;
        const double2 a = lin2(f.E2[m], f.V[m], f.Q[m], t);
        f.A[m] = a;
        return a;
    }
    if (stage == 1) {
        f.Na[m] = t;
        return lin2(f.E2[m], f.V[m], f.Q[m], t);
    }
    if (stage == 2) {
        f.Nb[m] = t;
        const double2 nv = f.Nv[m];
        const double2 d = make_double2(2.0 * t.x - nv.x, 2.0 * t.y - nv.y);
        return lin2(f.E2[m], f.A[m], f.Q[m], d);
    }
    const double2 v = f.V[m], nv = f.Nv[m], na = f.Na[m], nb = f.Nb[m];
    const double e = f.E[m], g1 = f.f1[m], c2 = 2.0 * f.f2[m], g3 = f.f3[m];
    const double2 r = make_double2(e * v.x + g1 * nv.x + c2 * (na.x + nb.x) + g3 * t.x,
                                   e * v.y + g1 * nv.y + c2 * (na.y + nb.y) + g3 * t.y);
    f.V[m] = r;
    return r;
}
__global__ void etd_combine_kernel(EtdFields f, long M, int stage) {
    for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < M; m += (long)gridDim.x * blockDim.x)
        f.T[m] = etd_combine(f, m, stage, f.T[m]);
}

// q_f = Re(T) / M, q_c = Im(T) / M (q_c may be null)
__global__ void etd_store_kernel(const double2* __restrict__ T, double* __restrict__ qf, double* __restrict__ qc,
                                 long M, double rM) {
    for (long m = blockIdx.x * (long)blockDim.x + threadIdx.x; m < M; m += (long)gridDim.x * blockDim.x) {
        const double2 t = T[m];
        qf[m] = t.x / rM;
        if (qc) qc[m] = t.y / rM;
    }
}

// ---------------------------------------------------------------------------
// 2D and 3D grids: a stage's two ends fused with the transforms along one axis
// ---------------------------------------------------------------------------
// The transforms' axes commute, so a stage's forward transform ends and its inverse
// one begins along the last axis, and the inverse one ends and the next stage's
// forward one begins along the first: with the spectral work between the former and
// the nonlinear term between the latter, a stage is two launches (2D) or four (3D,
// with the passes along the middle axis) where it was six or eight, and the field
// makes as many round trips through L2.  Every launch and kernel of its own, a step
// took 76 us at 128^2 (25 launches; now 31), 84 at 16^3 (33; 40), 101 at 32^3 (50),
// 184 at 48^3 (93), 130 at 64^3 (85).  What bounds a launch is its latency (2.5 us at
// 16^3, 5 at 64^3): tiles are small enough for a CTA an SM, and a launch starts before
// the one ahead has ended (128^2 35 us a step without; letting it start as early as it
// can costs 39, the waiting CTAs taking the running ones' places).
struct EtdPass {
    EtdFields f;
    int stage;
    const double *wf, *wc;   // w of the nonlinear term that follows (null: the sweep ends)
    double *qf, *qc;         // the slices after the last stage
    double M;
};

enum EtdKind {
    ETD_SPEC,   // forward, spectral stage, inverse
    ETD_REAL,   // inverse, nonlinear term (after the last stage: of the new slices), forward
    ETD_FWD, ETD_INV
};

// A launch may start while the one before it ends: it reads the twiddles, then waits
// for that launch's results.
template <int N, int KIND>
__global__ void __launch_bounds__(lp::kThreads) etd_pass_kernel(LineGeom g, EtdPass p, const double2* __restrict__ gtw) {
    constexpr bool INV = KIND == ETD_REAL || KIND == ETD_INV;   // sign of the first transform
    extern __shared__ __align__(16) double2 esm[];
    double2 *twf = esm, *twi = esm + N, *A = esm + 2 * N, *B = A + N * g.LP;
    for (int m = threadIdx.x; m < N; m += blockDim.x) {
        const double2 t = gtw[m];
        twf[m] = t;
        twi[m] = make_double2(t.x, -t.y);
    }
    const lp::TileAddr ta = lp::tile_addr(g, blockIdx.x);
    const int nel = N * g.T;
    double2* const T = p.f.T;
    using lp::kMaxEPT;
    using lp::kThreads;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    PS_ELEMS(e) {
        const lp::Elem el = lp::elem<N>(g, ta, e);
        A[el.sidx] = T[el.goff];
    }
    __syncthreads();
    double2* r = lp::tile_fft<N, INV ? +1 : -1>(A, B, g.T, g.LP, INV ? twi : twf);
    if constexpr (KIND == ETD_SPEC || KIND == ETD_REAL) {
        PS_ELEMS(e) {
            const lp::Elem el = lp::elem<N>(g, ta, e);
            if constexpr (KIND == ETD_REAL) {
                const double xf = r[el.sidx].x / p.M, xc = r[el.sidx].y / p.M;
                if (p.stage == 3) {
                    p.qf[el.goff] = xf;
                    p.qc[el.goff] = xc;
                }
                if (p.wf) r[el.sidx] = make_double2(-p.wf[el.goff] * xf, -p.wc[el.goff] * xc);
            } else {
                r[el.sidx] = etd_combine(p.f, el.goff, p.stage, r[el.sidx]);
            }
        }
        if (KIND == ETD_REAL && !p.wf) return;
        __syncthreads();
        r = lp::tile_fft<N, INV ? -1 : +1>(r, lp::other(r, A, B), g.T, g.LP, INV ? twf : twi);
    }
    asm volatile("griddepcontrol.launch_dependents;");
    PS_ELEMS(e) {
        const lp::Elem el = lp::elem<N>(g, ta, e);
        T[el.goff] = r[el.sidx];
    }
}

size_t etd_pass_smem(const LineGeom& g) { return sizeof(double2) * (2 * (size_t)g.N + 2 * (size_t)g.N * g.LP); }

template <int N, int KIND>
void etd_pass_n(const LineGeom& g, const EtdPass* p, cudaStream_t st) {
    const auto k = etd_pass_kernel<N, KIND>;
    if (!p) {
        PS_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLinePassSmemLimit));
        return;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)g.ntiles, 1, 1);
    cfg.blockDim = dim3(lp::kThreads, 1, 1);
    cfg.dynamicSmemBytes = etd_pass_smem(g);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    PS_CUDA(cudaLaunchKernelEx(&cfg, k, g, *p, twiddle_table(N)));
}

// launches the pass, or (p == nullptr) sets its kernel's attributes
template <int KIND>
void etd_pass(const LineGeom& g, const EtdPass* p, cudaStream_t st) {
    switch (g.N) {
#define X(N) case N: return etd_pass_n<N, KIND>(g, p, st);
        X(2) X(4) X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(352)
#undef X
    }
}

// ---------------------------------------------------------------------------
// small grids: all steps in one CTA
// ---------------------------------------------------------------------------
// The packed field ping-pongs between two shared-memory buffers, one Stockham
// radix pass a barrier; element (x, y) sits at x P + y with an odd pitch P, so
// that threads on consecutive lines of either axis fall in different banks.
// The spectral fields of a point stay in the registers of its thread for the whole
// solve.
// What bounds it is the chain of 8 transforms a step, each radix pass some 400
// cycles of shared-memory and FP64 latency and a barrier: 32^2 16.7 us a step,
// 1D 64 points 5.0 us (by passes 26 and 33).
constexpr long kSmallPoints = 1536;   // 32 x 48 27.0 us a step, by passes 27.9; 32 x 64 31.5 and 27.8

struct EtdSmall {
    double *hf, *hc;              // histories; hc == nullptr: lane c carries nothing
    const double *wf[2], *wc[2];  // w of each lane before and from its switch step
    int swf, swc, nsteps, Lx, Ly;
    const double *E, *E2, *Q, *f1, *f2, *f3;
    const double2 *twx, *twy;
};

extern __shared__ __align__(16) double2 esm[];

// nl lines of one axis: line l, element n at l ls + n es; magic: ceil(2^32 / nl),
// so that b / nl is the high word of b magic for b < 2^16
struct SmallAxis {
    int N, nl, ls, es, tw;
    unsigned magic;
};

// one radix pass of every line, from offset `in` of the shared memory to `out`
template <int N, int R, int NS, int SIGN, int NT>
__device__ __forceinline__ void small_pass(int in, int out, const SmallAxis& g) {
    constexpr int NB = N / R;
    for (int b = threadIdx.x; b < g.nl * NB; b += NT) {
        const int j = g.nl == 1 ? b : (int)__umulhi((unsigned)b, g.magic), l = b - j * g.nl, jm = j % NS;
        const double2* src = esm + in + l * g.ls + j * g.es;
        double2 v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = src[r * NB * g.es];
        if (NS > 1) {
#pragma unroll
            for (int r = 1; r < R; r++) {
                double2 w = esm[g.tw + (jm * r * (N / (NS * R))) % N];
                if (SIGN > 0) w.y = -w.y;
                v[r] = cmul(v[r], w);
            }
        }
        Dft<R, SIGN>::run(v);
        double2* dst = esm + out + l * g.ls + ((j / NS) * NS * R + jm) * g.es;
#pragma unroll
        for (int r = 0; r < R; r++) dst[r * NS * g.es] = v[r];
    }
    __syncthreads();
}
// transform of every line of the field at offset a (the other buffer at b);
// returns whether the field has changed places
template <int N, int SIGN, int NT>
__device__ __forceinline__ bool small_lines(int a, int b, const SmallAxis& g) {
    using P = Plan<N>;
    if constexpr (P::P >= 1) small_pass<N, P::r0, 1, SIGN, NT>(a, b, g);
    if constexpr (P::P >= 2) small_pass<N, P::r1, P::r0, SIGN, NT>(b, a, g);
    if constexpr (P::P >= 3) small_pass<N, P::r2, P::r0 * P::r1, SIGN, NT>(a, b, g);
    return P::P % 2 == 1;
}
template <int SIGN, int NT>
__device__ __forceinline__ bool small_axis(int a, int b, const SmallAxis& g) {
    switch (g.N) {
#define X(V) case V: return small_lines<V, SIGN, NT>(a, b, g);
        X(2) X(4) X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128) X(192) X(256) X(352)
#undef X
    }
    return false;
}

template <int NT, int KP>
__global__ void __launch_bounds__(NT, 1) etd_small_kernel(const __grid_constant__ EtdSmall a) {
    // the spectral fields in registers, and with the registers of up to 256
    // threads the tables and w as well (read from the L2 twice a stage otherwise)
    constexpr bool TAB = NT <= 256;
    const int M = a.Lx * a.Ly, P = a.Ly | 1, F = a.Lx * P;
    auto magic = [](int n) { return (unsigned)(((1ull << 32) + n - 1) / n); };
    const SmallAxis ax = {a.Lx, a.Ly, 1, P, 0, magic(a.Ly)}, ay = {a.Ly, a.Lx, P, 1, a.Lx, magic(a.Lx)};
    int cur = a.Lx + a.Ly, oth = cur + F;   // the field, the other buffer
    for (int i = threadIdx.x; i < a.Lx; i += NT) esm[i] = a.twx[i];
    if (a.Ly > 1)
        for (int i = threadIdx.x; i < a.Ly; i += NT) esm[a.Lx + i] = a.twy[i];
    const double Md = (double)M, rM = 1.0 / Md;
    const bool pow2 = (M & (M - 1)) == 0;
    double2 rV[KP], rN[KP], rA[KP], rS[KP];
    int place[KP];
#pragma unroll
    for (int k = 0; k < KP; k++) {
        const int m = threadIdx.x + k * NT, x = m / a.Ly;
        place[k] = x * P + (m - x * a.Ly);
    }
    auto each = [&](auto f) {   // this thread's points: (slot, point, place in the buffers)
#pragma unroll
        for (int k = 0; k < KP; k++) {
            const int m = threadIdx.x + k * NT;
            if (m < M) f(k, m, place[k]);
        }
    };
    auto flip = [&](bool moved) {
        if (moved) {
            const int c = cur;
            cur = oth;
            oth = c;
        }
    };
    auto forward = [&]() {
        __syncthreads();
        if (a.Ly > 1) flip(small_axis<-1, NT>(cur, oth, ay));
        flip(small_axis<-1, NT>(cur, oth, ax));
    };
    auto inverse = [&]() {
        __syncthreads();
        flip(small_axis<+1, NT>(cur, oth, ax));
        if (a.Ly > 1) flip(small_axis<+1, NT>(cur, oth, ay));
    };
    double2 q[KP];   // the slice
    double tab[6][TAB ? KP : 1], w[2][TAB ? KP : 1];
    const double* const tabs[6] = {a.E, a.E2, a.Q, a.f1, a.f2, a.f3};
    if constexpr (TAB)
#pragma unroll
        for (int i = 0; i < 6; i++) each([&](int k, int m, int) { tab[i][k] = __ldg(tabs[i] + m); });
    auto T = [&](int i, int k, int m) { if constexpr (TAB) return tab[i][k]; else return __ldg(tabs[i] + m); };
    for (int t = 0; t < a.nsteps; t++) {
        const double *qf = a.hf + (long)t * M, *qc = a.hc ? a.hc + (long)t * M : nullptr;
        const double *wf = a.wf[t >= a.swf], *wc = a.wc[t >= a.swc];
        if constexpr (TAB)
            if (t == 0 || t == a.swf || t == a.swc)
                each([&](int k, int m, int) {
                    w[0][k] = __ldg(wf + m);
                    w[1][k] = __ldg(wc + m);
                });
        auto W = [&](int i, int k, int m) { if constexpr (TAB) return w[i][k]; else return __ldg((i ? wc : wf) + m); };
        if (t == 0 || t == a.swf || t == a.swc) {
            each([&](int, int m, int i) { esm[cur + i] = make_double2(qf[m], qc ? qc[m] : 0.0); });
            forward();
            each([&](int k, int, int i) { rV[k] = esm[cur + i]; });
        }
        each([&](int k, int m, int i) {
            double2 x;
            if (t == 0) x = make_double2(qf[m], qc ? qc[m] : 0.0);
            else x = q[k];
            esm[cur + i] = make_double2(-W(0, k, m) * x.x, qc ? -W(1, k, m) * x.y : 0.0);
        });
#pragma unroll 1
        for (int stage = 0; stage < 4; stage++) {
            if (stage > 0)
                each([&](int k, int m, int i) {
                    const double2 z = esm[cur + i];
                    esm[cur + i] = make_double2(-W(0, k, m) * div_pow2_or_rn(z.x, Md, rM, pow2),
                                                qc ? -W(1, k, m) * div_pow2_or_rn(z.y, Md, rM, pow2) : 0.0);
                });
            forward();
            each([&](int k, int m, int i) {
                const double2 z = esm[cur + i];
                double2 r;
                if (stage == 0) {
                    rN[k] = z;
                    r = lin2(T(1, k, m), rV[k], T(2, k, m), z);
                    rA[k] = r;
                } else if (stage == 1) {
                    rS[k] = z;
                    r = lin2(T(1, k, m), rV[k], T(2, k, m), z);
                } else if (stage == 2) {
                    const double2 nv = rN[k], na = rS[k];
                    rS[k] = make_double2(na.x + z.x, na.y + z.y);
                    r = lin2(T(1, k, m), rA[k], T(2, k, m), make_double2(2.0 * z.x - nv.x, 2.0 * z.y - nv.y));
                } else {
                    const double2 v = rV[k], nv = rN[k], s = rS[k];
                    const double e = T(0, k, m), g1 = T(3, k, m), c2 = 2.0 * T(4, k, m), g3 = T(5, k, m);
                    r = make_double2(e * v.x + g1 * nv.x + c2 * s.x + g3 * z.x, e * v.y + g1 * nv.y + c2 * s.y + g3 * z.y);
                    rV[k] = r;
                }
                esm[cur + i] = r;
            });
            inverse();
        }
        double *of = a.hf + (long)(t + 1) * M, *oc = a.hc ? a.hc + (long)(t + 1) * M : nullptr;
        each([&](int k, int m, int i) {
            const double2 z = esm[cur + i];
            const double2 x = make_double2(div_pow2_or_rn(z.x, Md, rM, pow2), div_pow2_or_rn(z.y, Md, rM, pow2));
            of[m] = x.x;
            if (oc) oc[m] = x.y;
            q[k] = x;
        });
    }
}

size_t small_smem(int Lx, int Ly) { return sizeof(double2) * ((size_t)Lx + Ly + 2 * (size_t)Lx * (Ly | 1)); }

bool small_grid(int Lx, int Ly, int Lz) {
    return Lz == 1 && Lx > 1 && (long)Lx * Ly <= kSmallPoints && small_smem(Lx, Ly) <= 200 * 1024;
}

// f(kernel, threads) of the grid's kernel
template <class F>
void small_kernel(long M, F f) {
    if (M <= 128) f(etd_small_kernel<64, 2>, 64);
    else if (M <= 1024) f(etd_small_kernel<256, 4>, 256);
    else f(etd_small_kernel<512, 3>, 512);
}

}  // namespace

// Etdrk4_PBC's tables (Etdrk4_PBC.cc:14-24, :43-99): E = exp(ds L),
// E2 = exp(ds L / 2) and Q, f1, f2, f3 as ds times the mean over Mc points
// r = exp(i pi (j + 1/2) / Mc) of the upper half circle of the real parts of
//   Q  = (e^{x/2} - 1) / x,            f1 = (e^x (x^2 - 3x + 4) - x - 4) / x^3,
//   f2 = (e^x (x - 2) + x + 2) / x^3,  f3 = (e^x (4 - x) - x^2 - 3x - 4) / x^3
// at x = ds L + r (the contour integral that avoids the cancellation of the
// closed forms near L = 0).  L is the k2_orthogonal table (-|k|^2).
void PairChain::set_tables_etd(const std::vector<double>& k2, double ds, int Mc) {
    if (scheme_ != SCHEME_ETDRK4) throw Error(-2, "set_tables_etd on a chain that is not ETDRK4");
    if (Mc < 1) throw Error(-1, "ETDRK4 needs at least one contour point");
    const long M = M_;
    std::vector<double> tab(6 * (size_t)M);
    const double PI = 3.14159265358979323846;
    std::vector<std::complex<double>> r(Mc);
    for (int j = 0; j < Mc; j++) r[j] = std::exp(std::complex<double>(0.0, PI * (j + 0.5) / Mc));
    for (long m = 0; m < M; m++) {
        const double L = k2[m];
        tab[0 * M + m] = exp(ds * L);
        tab[1 * M + m] = exp(ds * L / 2.0);
        double sq = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        for (int j = 0; j < Mc; j++) {
            const std::complex<double> x = ds * L + r[j];
            const std::complex<double> ex = std::exp(x), x2 = x * x, x3 = x2 * x;
            sq += ((std::exp(x / 2.0) - 1.0) / x).real();
            s1 += ((ex * (x2 - 3.0 * x + 4.0) - x - 4.0) / x3).real();
            s2 += ((ex * (x - 2.0) + x + 2.0) / x3).real();
            s3 += ((ex * (4.0 - x) - x2 - 3.0 * x - 4.0) / x3).real();
        }
        tab[2 * M + m] = ds * (sq / Mc);
        tab[3 * M + m] = ds * (s1 / Mc);
        tab[4 * M + m] = ds * (s2 / Mc);
        tab[5 * M + m] = ds * (s3 / Mc);
    }
    // PS_B200_LINE_PASSES=1 at this point keeps the line passes
    const char* force = getenv("PS_B200_LINE_PASSES");
    small_etd_ = small_grid(Lx_, Ly_, Lz_) && !(force && force[0] == '1');
    if (small_etd_) {
        small_kernel(M_, [](auto kernel, int) {
            PS_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024));
        });
    }
    for (int a = 0; a < plan_.naxes; a++) {
        etd_pass<ETD_SPEC>(plan_.ax[a], nullptr, nullptr);
        etd_pass<ETD_REAL>(plan_.ax[a], nullptr, nullptr);
        etd_pass<ETD_FWD>(plan_.ax[a], nullptr, nullptr);
        etd_pass<ETD_INV>(plan_.ax[a], nullptr, nullptr);
    }
    etdtab_.alloc(tab.size());
    upload(etdtab_.p, tab.data(), sizeof(double) * tab.size());
}

// forward (MODE_FWD) or inverse (MODE_INV, unnormalised) transform of one
// packed field over every axis of the grid
void PairChain::transform(double2* z, int mode, cudaStream_t st) const {
    StepPtrs p{};
    p.z[0] = z;
    p.nfield = 1;
    p.M = (double)M_;
    for (int a = 0; a < plan_.naxes; a++) launch_line_pass(mode, plan_.ax[a], p, 1, st);
}

// ETDRK4 steps t = 0 .. nsteps-1 of the pair: lane f's w is lf.F(t), lane c's
// lc.F(t) (the factor slots carry the fields w themselves for this scheme).
// A lane that starts a new block at step t starts a new solve there: the
// carried spectrum is rebuilt from the real slices of both lanes at t = 0
// and at each lane's switch step (Etdrk4_PBC::solve starts from F[q_0]).
void PairChain::enqueue_etd(double* hf, double* hc, int nsteps, const LaneFactors& lf, const LaneFactors& lc,
                            cudaStream_t st, const double* c_in_fixed, double* c_out_fixed) {
    const long M = M_;
    const double rM = (double)M;
    const unsigned nb = etd_blocks(M);
    double2* T = z_[0].c();
    EtdFields f;
    f.T = T;
    f.V = etd_.c(); f.Nv = f.V + M; f.A = f.V + 2 * M; f.Na = f.V + 3 * M; f.Nb = f.V + 4 * M;
    f.E = etdtab_.p; f.E2 = f.E + M; f.Q = f.E + 2 * M; f.f1 = f.E + 3 * M; f.f2 = f.E + 4 * M; f.f3 = f.E + 5 * M;
    if (small_etd_) {
        EtdSmall a{};
        a.hf = hf;
        a.hc = c_in_fixed ? nullptr : hc;   // a fixed lane c is zero (UpdaterCtx)
        for (int i = 0; i < 2; i++) {
            a.wf[i] = lf.eF[i];
            a.wc[i] = lc.eF[i];
        }
        a.swf = lf.switch_t; a.swc = lc.switch_t;
        a.nsteps = nsteps; a.Lx = Lx_; a.Ly = Ly_;
        a.E = f.E; a.E2 = f.E2; a.Q = f.Q; a.f1 = f.f1; a.f2 = f.f2; a.f3 = f.f3;
        a.twx = twiddle_table(Lx_);
        a.twy = Ly_ > 1 ? twiddle_table(Ly_) : nullptr;
        small_kernel(M, [&](auto kernel, int threads) {
            kernel<<<1, threads, small_smem(Lx_, Ly_), st>>>(a);
        });
        PS_CUDA(cudaGetLastError());
        return;
    }
    if (plan_.naxes > 1) {
        const LineGeom &in = plan_.ax[0], &out = plan_.ax[plan_.naxes - 1];
        EtdPass p{};
        p.f = f;
        p.M = rM;
        for (int t = 0; t < nsteps; t++) {
            const double* qf = hf + (long)t * M;
            const double* qc = c_in_fixed ? c_in_fixed : hc + (long)t * M;
            if (t == 0 || t == lf.switch_t || t == lc.switch_t) {
                etd_slices_kernel<<<nb, kEtdThreads, 0, st>>>(f.V, qf, qc, nullptr, nullptr, M, 0);
                PS_CUDA(cudaGetLastError());
                transform(f.V, MODE_FWD, st);
            }
            if (t == 0) {
                etd_slices_kernel<<<nb, kEtdThreads, 0, st>>>(T, qf, qc, lf.F(0), lc.F(0), M, 1);
                PS_CUDA(cudaGetLastError());
                etd_pass<ETD_FWD>(in, &p, st);
            }
            for (int stage = 0; stage < 4; stage++) {
                const bool last = stage == 3, next = !last || t + 1 < nsteps;
                p.stage = stage;
                p.wf = next ? lf.F(last ? t + 1 : t) : nullptr;
                p.wc = next ? lc.F(last ? t + 1 : t) : nullptr;
                p.qf = hf + (long)(t + 1) * M;
                p.qc = c_in_fixed ? c_out_fixed : hc + (long)(t + 1) * M;
                if (plan_.naxes > 2) etd_pass<ETD_FWD>(plan_.ax[1], &p, st);
                etd_pass<ETD_SPEC>(out, &p, st);
                if (plan_.naxes > 2) etd_pass<ETD_INV>(plan_.ax[1], &p, st);
                etd_pass<ETD_REAL>(in, &p, st);
            }
        }
        return;
    }
    for (int t = 0; t < nsteps; t++) {
        const double* qf = hf + (long)t * M;
        const double* qc = c_in_fixed ? c_in_fixed : hc + (long)t * M;
        const double* wf = lf.F(t);
        const double* wc = lc.F(t);
        if (t == 0 || t == lf.switch_t || t == lc.switch_t) {
            etd_slices_kernel<<<nb, kEtdThreads, 0, st>>>(f.V, qf, qc, nullptr, nullptr, M, 0);
            PS_CUDA(cudaGetLastError());
            transform(f.V, MODE_FWD, st);
        }
        etd_slices_kernel<<<nb, kEtdThreads, 0, st>>>(T, qf, qc, wf, wc, M, 1);
        PS_CUDA(cudaGetLastError());
        for (int stage = 0; stage < 4; stage++) {
            if (stage > 0) {
                etd_nonlin_kernel<<<nb, kEtdThreads, 0, st>>>(T, wf, wc, M, rM);
                PS_CUDA(cudaGetLastError());
            }
            transform(T, MODE_FWD, st);
            etd_combine_kernel<<<nb, kEtdThreads, 0, st>>>(f, M, stage);
            PS_CUDA(cudaGetLastError());
            transform(T, MODE_INV, st);
        }
        double* of = hf + (long)(t + 1) * M;
        double* oc = c_in_fixed ? c_out_fixed : hc + (long)(t + 1) * M;
        etd_store_kernel<<<nb, kEtdThreads, 0, st>>>(T, of, oc, M, rM);
        PS_CUDA(cudaGetLastError());
    }
}

}  // namespace ps
