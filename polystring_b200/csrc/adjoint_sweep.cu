// adjoint_sweep.cu -- the adjoint of the RQM4 chains on grids with a persistent
// sweep (real_sweep.cu, plane_sweep.cu, tile_sweep.cu); adjoint.cu has the line-pass form.
//
// Every split step S = e (.) D e (.) is symmetric, hence so is the RQM4 step
// A = (4 S' S' - S) / 3, and lambda[t] = A lambda[t+1] + D[t] is the forward
// recursion run backwards with a source.  So the reverse sweep of both chains is
// one more launch of the forward sweep, chain f's lambda running through the
// blocks as chain c's propagator does and the other way round.  Both launches
// keep two intermediate fields of every step (the raw results
// D' e^{-w ds/4} x and D e^{-w ds/2} x), from which the w-gradient of all steps
// is one pass over the histories:
//
//   S x = e^{-w ds/2} D e^{-w ds/2} x,  S'x S'y = e^{-w ds/2} (D' e^{-w ds/4} x)(D' e^{-w ds/4} y),
//   S'S'x = (3 A x + S x) / 4
//
// The stress needs no reverse sweep: without sources lambda[t] is the
// complementary chain's slice c[Ns - t] / M, the same recursion from the same
// head.  dD/dl_i = h (8 pi^2 / l_i^3) R_i D with the line operator
// R_i = F^-1 r_i^2 F of axis i, so
//
//   lambda' (dA/dl_i) q = h 8 pi^2 / l_i^3 [ 2/3 ((D' e' lambda) . R_i (e D' e' q) + (e D' e' lambda) . R_i (D' e' q))
//                                           - 1/3 (e lambda) . R_i (D e q) ]
//
// with e = e^{-w ds/2}, e' = e^{-w ds/4}: three line operators an axis and step,
// all steps at once.  (The first term is (e' lambda) . R_i (D' e' S' q): D' is
// symmetric, commutes with R_i, and e' S' q = e D' e' q.  So only kept fields enter, and
// no quotient by e', which is zero where w is large or infinite.)
//
// 48^3, Ns 128 (B200): the reverse sweeps took about 80 us a step and chain on
// line passes (gradient 33.5 ms, stress 21.9 ms a call with the forward map); the gradient
// takes 4.5 ms now, of which the two sweeps 3.1 and the read-back of their kept fields 0.25
// at 6.4 TB/s, and 32^3's stress (11.5 ms) 1.06, of which the sweep 0.73.  What bounds the
// stress kernels is their registers, spilled from 24 points on at two CTAs an SM (56 bytes a
// thread at 32 points, 756 at 64, 3100 at 128): 105 MB an axis at 2 TB/s.
#include <algorithm>
#include <cmath>
#include <utility>
#include <vector>

#include "engine.h"
#include "field_kernels.h"
#include "real_line.cuh"

namespace ps {

namespace {

constexpr int kT = 256;
constexpr int kChunk = 16;       // steps of one block that a thread of the gradient pass sums
constexpr int kStressCtas = 592;

int grid_of(long M) { return (int)((M + kT - 1) / kT); }

// partial sums of a . b + c . d, one a block
__global__ void __launch_bounds__(kT) dot_kernel(const double* a, const double* b, const double* c, const double* d,
                                                 long M, double* partial) {
    double s = 0.0;
    for (long i = (long)blockIdx.x * kT + threadIdx.x; i < M; i += (long)gridDim.x * kT) s += a[i] * b[i] + c[i] * d[i];
    __shared__ double sh[kT / 32];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0.0;
        for (int w = 0; w < kT / 32; w++) t += sh[w];
        partial[blockIdx.x] = t;
    }
}
__global__ void dot_final_kernel(const double* partial, int n, double* out) {
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += 32) s += partial[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) *out = s;
}

// pbar = phi_bar / Q, and the heads of both adjoint chains:
// lambda_f[Ns] = (Q_bar - dot / Q) / M + (wfa pbarA + wfb pbarB) c[0], lambda_c likewise without the constant
__global__ void __launch_bounds__(kT) heads_kernel(double* pA, double* pB, const double* Q, const double* dot,
                                                   double Qbar, double wfa, double wfb, double wca, double wcb,
                                                   const double* hf0, const double* hc0, double* lf, double* lc,
                                                   long M) {
    const long i = (long)blockIdx.x * kT + threadIdx.x;
    if (i >= M) return;
    const double q = *Q, a = pA[i] / q, b = pB[i] / q;
    pA[i] = a;
    pB[i] = b;
    lf[i] = (Qbar - *dot / q) / (double)M + (wfa * a + wfb * b) * hc0[i];
    lc[i] = (wca * a + wcb * b) * hf0[i];
}

// One chain's histories: q (slice t), lambda (slice tau = Ns - t), the kept
// fields of both, and lambda's source.
struct GradChain {
    const double *q, *lam, *qhalf, *qfull, *lhalf, *lfull;
    const double *src_w[2], *src_o;
};
struct GradArgs {
    GradChain c[2];
    const double *eF[2], *pA, *pB;
    double ds[2];
    const AdjointChunk* chunk;
    double* partial;
    long M;
    int Ns;
};

// the w-gradient of chunk blockIdx.y's steps, a point a thread
__global__ void __launch_bounds__(kT) grad_kernel(const GradArgs a) {
    const long i = (long)blockIdx.x * kT + threadIdx.x;
    if (i >= a.M) return;
    const AdjointChunk k = a.chunk[blockIdx.y];
    const GradChain& c = a.c[k.chain];
    const long M = a.M;
    const double e = a.eF[k.blk][i], pA = a.pA[i], pB = a.pB[i], ds = a.ds[k.blk];
    double acc = 0.0, q0 = c.q[(long)k.t0 * M + i], l0 = c.lam[(long)(a.Ns - k.t0) * M + i];
#pragma unroll 4
    for (int t = k.t0; t < k.t1; t++) {
        const int s = a.Ns - 1 - t;   // lambda[t + 1] is slice s
        const double q1 = c.q[(long)(t + 1) * M + i], l1 = c.lam[(long)s * M + i];
        const double src = (c.src_w[0][s + 1] * pA + c.src_w[1][s + 1] * pB) * c.src_o[(long)(s + 1) * M + i];
        const double sq = e * c.qfull[(long)t * M + i], sl = e * c.lfull[(long)s * M + i];
        const double uv = e * c.qhalf[(long)t * M + i] * c.lhalf[(long)s * M + i];
        const double qt2 = 0.25 * (3.0 * q1 + sq), vv = 0.25 * (3.0 * (l0 - src) + sl);
        acc += -(ds / 3.0) * (l1 * qt2 + 2.0 * uv + q0 * vv) + (ds / 6.0) * (l1 * sq + q0 * sl);
        q0 = q1;
        l0 = l1;
    }
    a.partial[(long)blockIdx.y * M + i] = acc;
}
__global__ void __launch_bounds__(kT) grad_sum_kernel(const double* partial, const AdjointChunk* chunk, int n, long M,
                                                      double* gA, double* gB) {
    const long i = (long)blockIdx.x * kT + threadIdx.x;
    if (i >= M) return;
    double g[2] = {0.0, 0.0};
    for (int k = 0; k < n; k++) g[chunk[k].blk] += partial[(long)k * M + i];
    gA[i] = g[0];
    gB[i] = g[1];
}

// Line l of an axis with stride st between its points: offset of its first point
__device__ __forceinline__ long line_base(long l, int N, long st) { return l / st * N * st + l % st; }

struct StressArgs {
    const double *qhalf, *qfull;       // forward chain: kept fields
    const double *c, *chalf;           // complementary chain: slices, kept fields
    const double* eF[2];
    const double* frag;                // R_i
    double scale[2];                   // 8 pi^2 / l^3 times the block's ds
    double* partial;                   // [cta][3], entry `axis`
    long M, st, nlines;
    int Ns, LA, axis;
};

// sum over steps and points of one axis's terms; a unit is (step, tile of eight lines)
template <int N>
__global__ void __launch_bounds__(kT, 2) stress_axis_kernel(const StressArgs a) {
    using R = RealLine<N>;
    extern __shared__ double fr[];
    for (int i = threadIdx.x; i < R::FRAG; i += kT) fr[i] = a.frag[i];
    __syncthreads();
    const int lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const long tiles = (a.nlines + 7) / 8, units = tiles * a.Ns;
    double sum = 0.0;
    for (long u = (long)blockIdx.x * (kT / 32) + (threadIdx.x >> 5); u < units; u += (long)gridDim.x * (kT / 32)) {
        const int t = (int)(u / tiles), blk = t < a.LA ? 0 : 1;
        const long l = (u - t * tiles) * 8 + g;
        const bool ok = l < a.nlines;
        const long base = line_base(ok ? l : l - g, N, a.st), now = (long)t * a.M + base;
        const long lam = (long)(a.Ns - 1 - t) * a.M + base;   // lambda[t + 1]
        const double* eF = a.eF[blk] + base;
        double part = 0.0;
#pragma unroll 1
        for (int k = 0; k < 3; k++) {
            double x[R::E];
#pragma unroll
            for (int s = 0; s < R::S; s++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int o = j + 4 * s;
                    double v = 0.0;
                    if (R::WHOLE || o < R::O) {
                        const long n = R::point(i, o) * a.st;
                        v = k == 0 ? a.qfull[now + n] : k == 1 ? eF[n] * a.qhalf[now + n] : a.qhalf[now + n];
                    }
                    x[4 * s + i] = v;
                }
            R::apply(x, fr + lane);
            double d = 0.0;
#pragma unroll
            for (int s = 0; s < R::S; s++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int o = j + 4 * s;
                    if (R::WHOLE || o < R::O) {
                        const long n = R::point(i, o) * a.st;
                        const double y = k == 0 ? eF[n] * a.c[lam + n] : k == 1 ? a.chalf[lam + n]
                                                                                : eF[n] * a.chalf[lam + n];
                        d += x[4 * s + i] * y;
                    }
                }
            part += (k == 0 ? -1.0 / 3.0 : 2.0 / 3.0) * d;
        }
        if (ok) sum += a.scale[blk] * part;
    }
    __shared__ double sh[kT / 32];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if (lane == 0) sh[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kT / 32; w++) s += sh[w];
        a.partial[(long)blockIdx.x * 3 + a.axis] = s;
    }
}

__global__ void stress_sum_kernel(const double* partial, int n, double scale, double* out) {
    for (int i = 0; i < 3; i++) {
        double s = 0.0;
        for (int k = threadIdx.x; k < n; k += 32) s += partial[3 * k + i];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) out[i] = s * scale;
    }
}

template <int N>
void stress_launch(const StressArgs& a, cudaStream_t st) {
    const int smem = (int)(sizeof(double) * RealLine<N>::FRAG);
    PS_CUDA(cudaFuncSetAttribute(stress_axis_kernel<N>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    stress_axis_kernel<N><<<kStressCtas, kT, smem, st>>>(a);
    PS_CUDA(cudaGetLastError());
}

}  // namespace

// The chains' kept fields (and with `grad` the adjoint chains) of all steps:
// 4 (10) Ns M doubles beside the 2 (Ns + 1) M of the histories.  False where
// the grid has no sweep that keeps them (one with a single axis longer than a point,
// in a cell of any dimension, has not) or the device has no room: the line passes
// serve then, or refuse the grid.
// The buffers stay with the model.  They leave a sixteenth of the device's memory free,
// for others and for the line passes' own.
bool ModelAB::sweep_adjoint(bool grad) {
    if (!real_ || chain_->plan().naxes < 2) return false;
    // the stress keeps an axis's operator in shared memory: 32 KB at 128 points, 242 KB at 352
    if (!grad && (p_.Lx > 128 || p_.Ly > 128 || p_.Lz > 128)) return false;
    const size_t n = (size_t)Ns_ * M_;
    std::vector<std::pair<DevBuf*, size_t>> missing;
    size_t need = 0;
    auto want = [&](DevBuf& b, size_t count) {
        if (b.n > 0) return;
        missing.push_back({&b, count});
        need += sizeof(double) * count;
    };
    for (DevBuf& b : kept_) want(b, n);
    if (grad) {
        for (DevBuf& b : lkept_) want(b, n);
        for (DevBuf& b : lamh_) want(b, n + M_);
        want(gpart_, adjoint_chunks().size() * (size_t)M_);
    }
    if (missing.empty()) return true;
    size_t free = 0, total = 0;
    PS_CUDA(cudaMemGetInfo(&free, &total));
    bool room = need + total / 16 <= free;
    for (size_t i = 0; room && i < missing.size(); i++) room = missing[i].first->try_alloc(missing[i].second);
    if (!room)   // the stress's, where only the gradient's do not fit, stay
        for (auto& m : missing) m.first->release();
    return room;
}

// steps of both chains in chunks of one block each
std::vector<AdjointChunk> ModelAB::adjoint_chunks() const {
    std::vector<AdjointChunk> ch;
    auto add = [&](int chain, int blk, int t0, int t1) {
        for (int t = t0; t < t1; t += kChunk) ch.push_back({chain, blk, t, std::min(t + kChunk, t1)});
    };
    add(0, 0, 0, LA_);
    add(0, 1, LA_, Ns_);
    add(1, 1, 0, LB_);
    add(1, 0, LB_, Ns_);
    return ch;
}

// forward_only() with the kept fields
void ModelAB::forward_kept() {
    RealProblem p = sweep_descriptor();
    for (int i = 0; i < 2; i++) {
        p.lane[i].keep_half = kept_[2 * i].p;
        p.lane[i].keep_full = kept_[2 * i + 1].p;
    }
    real_->enqueue(p, st_);
    enqueue_densities(st_);
    forward_done_ = true;
}

void ModelAB::grad_w_sweep(const double* phiA_bar, const double* phiB_bar, double Q_bar, double* gA, double* gB) {
    // the steps' chunks, and the sources' weights by slice of the adjoint chains
    std::vector<double> wAf, wBf;
    adjoint_weights(wAf, wBf);
    if (adj_chunks_ == 0) {
        const std::vector<AdjointChunk> ch = adjoint_chunks();
        std::vector<double> w;
        for (int s = 0; s <= Ns_; s++) w.push_back(wAf[Ns_ - s]);
        for (int s = 0; s <= Ns_; s++) w.push_back(wBf[Ns_ - s]);
        w.insert(w.end(), wAf.begin(), wAf.end());
        w.insert(w.end(), wBf.begin(), wBf.end());
        srcw_.alloc(w.size());
        upload(srcw_.p, w.data(), sizeof(double) * w.size());
        chunks_.alloc((sizeof(AdjointChunk) * ch.size() + 7) / 8);
        upload(chunks_.p, ch.data(), sizeof(AdjointChunk) * ch.size());
        adj_chunks_ = (int)ch.size();
    }
    PS_CUDA(cudaMemcpyAsync(pbA_.p, phiA_bar, sizeof(double) * M_, cudaMemcpyHostToDevice, st_));
    PS_CUDA(cudaMemcpyAsync(pbB_.p, phiB_bar, sizeof(double) * M_, cudaMemcpyHostToDevice, st_));
    forward_kept();
    // pbar = phi_bar / Q; Qbar_total = Q_bar - (1/Q) sum(phi_bar phi)
    const int nb = std::min(grid_of(M_), (int)kRedBlocks);
    double *Q = scal_.p, *dot = scal_.p + 24;
    dot_kernel<<<nb, kT, 0, st_>>>(pbA_.p, phiA_.p, pbB_.p, phiB_.p, M_, partial_.p);
    dot_final_kernel<<<1, 32, 0, st_>>>(partial_.p, nb, dot);
    heads_kernel<<<grid_of(M_), kT, 0, st_>>>(pbA_.p, pbB_.p, Q, dot, Q_bar, wAf[Ns_], wBf[Ns_], wAf[0], wBf[0], hf_.p,
                                              hc_.p, lamh_[0].p, lamh_[1].p, M_);
    PS_CUDA(cudaGetLastError());
    // lambda of the forward chain passes block B first, as the complementary chain does
    RealProblem p = sweep_descriptor();
    std::swap(p.lane[0], p.lane[1]);
    const long W = Ns_ + 1;
    for (int i = 0; i < 2; i++) {
        RealLane& L = p.lane[i];
        L.hist = lamh_[i].p;
        L.keep_half = lkept_[2 * i].p;
        L.keep_full = lkept_[2 * i + 1].p;
        L.src_p[0] = pbA_.p;
        L.src_p[1] = pbB_.p;
        L.src_w[0] = srcw_.p + 2 * W * i;
        L.src_w[1] = srcw_.p + 2 * W * i + W;
        L.src_o = i == 0 ? hc_.p : hf_.p;
    }
    real_->enqueue(p, st_);
    GradArgs a{};
    for (int i = 0; i < 2; i++) {
        const RealLane& L = p.lane[i];
        a.c[i] = {i == 0 ? hf_.p : hc_.p, lamh_[i].p, kept_[2 * i].p, kept_[2 * i + 1].p, lkept_[2 * i].p,
                  lkept_[2 * i + 1].p, {L.src_w[0], L.src_w[1]}, L.src_o};
    }
    a.eF[0] = eFA_.p; a.eF[1] = eFB_.p;
    a.pA = pbA_.p; a.pB = pbB_.p;
    a.ds[0] = dsA_; a.ds[1] = dsB_;
    a.chunk = reinterpret_cast<const AdjointChunk*>(chunks_.p);
    a.partial = gpart_.p;
    a.M = M_;
    a.Ns = Ns_;
    grad_kernel<<<dim3(grid_of(M_), adj_chunks_), kT, 0, st_>>>(a);
    PS_CUDA(cudaGetLastError());
    grad_sum_kernel<<<grid_of(M_), kT, 0, st_>>>(gpart_.p, a.chunk, adj_chunks_, M_, gA_.p, gB_.p);
    PS_CUDA(cudaGetLastError());
    PS_CUDA(cudaMemcpyAsync(gA, gA_.p, sizeof(double) * M_, cudaMemcpyDeviceToHost, st_));
    PS_CUDA(cudaMemcpyAsync(gB, gB_.p, sizeof(double) * M_, cudaMemcpyDeviceToHost, st_));
    sync();
}

void ModelAB::stress_sweep(double* dFdl) {
    const int n[3] = {p_.Lx, p_.Ly, p_.Lz};
    const long st[3] = {(long)p_.Ly * p_.Lz, p_.Lz, 1};
    const double PI = 3.14159265358979323846;
    if (spart_.n == 0) {
        std::vector<double> f;
        for (int ax = 0; ax < 3; ax++) {
            sfo_[ax] = (int)f.size();
            if (n[ax] == 1) continue;
            std::vector<double> r2(n[ax]);
            for (int k = 0; k < n[ax]; k++) {
                const double r = k < n[ax] / 2 + 1 ? k : n[ax] - k;
                r2[k] = r * r;
            }
            real_fragments(n[ax], r2, f);
        }
        sfrag_.alloc(f.size());
        upload(sfrag_.p, f.data(), sizeof(double) * f.size());
        spart_.alloc(3 * kStressCtas);
    }
    forward_kept();
    PS_CUDA(cudaMemsetAsync(spart_.p, 0, sizeof(double) * 3 * kStressCtas, st_));
    for (int ax = 0; ax < p_.dim; ax++) {
        if (n[ax] == 1) continue;
        const double l = p_.cell.l[ax], c = l > 0 ? 8.0 * PI * PI / (l * l * l) : 0.0;
        StressArgs a{};
        a.qhalf = kept_[0].p; a.qfull = kept_[1].p;
        a.c = hc_.p; a.chalf = kept_[2].p;
        a.eF[0] = eFA_.p; a.eF[1] = eFB_.p;
        a.frag = sfrag_.p + sfo_[ax];
        a.scale[0] = c * dsA_; a.scale[1] = c * dsB_;
        a.partial = spart_.p;
        a.M = M_; a.st = st[ax]; a.nlines = M_ / n[ax];
        a.Ns = Ns_; a.LA = LA_; a.axis = ax;
        switch (n[ax]) {
#define X(N) case N: stress_launch<N>(a, st_); break;
            X(4) X(8) X(12) X(16) X(24) X(32) X(48) X(64) X(96) X(128)
#undef X
            default: throw Error(-2, "no line operator of this length");
        }
    }
    // dQ/dl = (1/M) sum over steps and points (lambda = c / M); dF/dl = -(1/Q) dQ/dl
    stress_sum_kernel<<<1, 32, 0, st_>>>(spart_.p, kStressCtas, 1.0 / (double)M_, scal_.p + 16);
    PS_CUDA(cudaGetLastError());
    double Q = 0.0, dQ[3];
    PS_CUDA(cudaMemcpyAsync(&Q, scal_.p, sizeof(double), cudaMemcpyDeviceToHost, st_));
    PS_CUDA(cudaMemcpyAsync(dQ, scal_.p + 16, sizeof(double) * 3, cudaMemcpyDeviceToHost, st_));
    sync();
    for (int i = 0; i < 3; i++) dFdl[i] = -dQ[i] / Q;
}

}  // namespace ps
