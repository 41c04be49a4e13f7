// real_sweep.h -- propagator sweeps built on real line operators
// (real_line.cuh): 3D grids in real_sweep.cu, 1D grids and 2D grids of up to
// 64 x 64 points in plane_sweep.cu, larger 2D grids in tile_sweep.cu.
#pragma once

#include <cuda_runtime.h>

#include <vector>

#include "ps_internal.h"

namespace ps {

// One chain of a solve: its history ((Ns + 1) slices, slice 0 the head) and
// the Boltzmann factors e^{-w ds/2}, e^{-w ds/4} of the blocks it runs through,
// block 0 before step sw[0], block 1 before sw[1], then block 2.
struct RealLane {
    double* hist;
    const double* eF[3];
    const double* eH[3];
    int sw[2];
    // optional, one slice a step: the first half step before its factor,
    // D' e^{-w ds/4} q, and the full step before its factor, D e^{-w ds/2} q
    double *keep_half, *keep_full;
    // optional source: slice t gets (src_w[0][t] src_p[0] + src_w[1][t] src_p[1]) src_o[t]
    const double *src_p[2], *src_w[2], *src_o;
};

// One solve of a sweep: nl chains (one or two) of Ns contour steps.
struct RealProblem {
    RealLane lane[2];
    double *W, *Z;        // work fields, nl x M each
    const double* frag;   // the axes' operators (full step, half step): B fragments, or parts (1D; 2D axes past 64)
    int fo[3], nfrag;     // where each axis's start (axes of equal length and spacing share), doubles in all
    unsigned* bar;        // barrier counters (one a chain, 16 words apart), zeroed before the launch
    int* err;             // nonzero after a barrier timeout, for the chains' CTAs
    int* notice;          // the same in host memory
    int hasty;            // barriers give up at the first poll in vain (of a launch: its `one`'s)
    int Lx, Ly, Lz, Ns, nl;
    int os2;              // second-order splitting: full steps only
    int xcols;            // columns of an x-pass task (a multiple of 8)
    int rkeep, xkeep;     // factors kept in shared memory: of the rows, of that many x-pass tasks a warp
    int split;            // long rows in parts (tile_sweep.cu)
    int cta0, ncta;       // the solve's first CTA in a shared launch, CTAs of each chain
};

// the axes' operators of an orthogonal cell, exp(h k r^2) per axis for h = ds and
// ds / 2, k = -(wave number)^2 at index 1; fo[a]: where axis a's start (axes
// of the same length and k share theirs); fragments of axes up to that many points,
// parts of longer ones
std::vector<double> real_operator_tables(const int n[3], const double k[3], double ds, int fragments, int fo[3]);

// whether a 3D grid has this sweep
bool real_sweep_supported(int Lx, int Ly, int Lz);
// CTAs one chain can keep busy
int real_sweep_tasks(int Lx, int Ly, int Lz);
// shared memory of a solve in a shared launch; whether it needs the kernel of
// one CTA an SM; CTAs resident at once in a shared launch of such solves
size_t real_sweep_smem(const RealProblem& p);
bool real_sweep_wide(const RealProblem& p);
int real_sweep_resident(size_t smem, bool wide);
// x-tile variants (columns a task; same arithmetic)
constexpr int kRealVariants = 3;
int real_sweep_columns(int variant);
// ncta CTAs a chain
void real_sweep_launch(const RealProblem& p, int ncta, cudaStream_t st);
// n solves described in device memory (shapes may differ), grid CTAs in all, the
// largest of the solves' shared memory
void real_sweep_launch_many(const RealProblem* d, int n, size_t smem, bool wide, int grid, int hasty, cudaStream_t st);

// 2D grids of up to 64 x 64 points, one CTA a chain
bool plane_sweep_supported(int Lx, int Ly);
void plane_sweep_prepare();
void plane_sweep_launch(const RealProblem& p, cudaStream_t st);
// n solves of two chains described in device memory (shapes may differ): the
// largest of their warp pairs and of their shared memory
int plane_sweep_pairs(int Lx, int Ly);
size_t plane_sweep_smem(const RealProblem& p, int pairs);
void plane_sweep_launch_many(const RealProblem* d, int n, int pairs, size_t smem, cudaStream_t st);
// 2D grids in tiles of lines; longest axis whose operators are fragments
int tile_sweep_fragments();
bool tile_sweep_supported(int Lx, int Ly);
// CTAs one chain can keep busy, shared memory of a solve
int tile_sweep_tasks(int Lx, int Ly);
size_t tile_sweep_smem(const RealProblem& p);
// over the whole grid: CTAs resident at once; ncta CTAs a chain
int tile_sweep_resident(size_t smem);
void tile_sweep_launch(const RealProblem& p, int ncta, cudaStream_t st);
// a cluster a chain: its size for a grid (0: none) and the clusters resident at
// once; a solve, or n solves of two chains described in device memory
int tile_cluster_size(int Lx, int Ly);
int tile_cluster_resident(int cluster, size_t smem);
void tile_cluster_launch(const RealProblem& p, int cluster, cudaStream_t st);
void tile_cluster_launch_many(const RealProblem* d, int n, int cluster, size_t smem, cudaStream_t st);
// n solves of two chains on one 2D grid with axes up to 128 points (the images of a
// string), a cluster each; prepare notes the clusters resident at once
bool tile_string_supported(int Lx, int Ly);
void tile_string_prepare(const RealProblem& p, int n);
void tile_string_launch(const RealProblem* d, int n, size_t smem, cudaStream_t st);
// 1D grids
bool line_sweep_supported(int Lx);
void line_sweep_launch(const RealProblem& p, cudaStream_t st);

// polls before a barrier gives up, some ten seconds (PS_B200_BARRIER_GIVE_UP=1 at the
// sweep's construction: at the first one in vain, for tests of what follows)
constexpr long long kBarrierPolls = 20000000;

// The work fields, operators and barrier words of one solve's sweep.
class RealSweep {
public:
    // k: -(wave number)^2 of index 1 along each axis; nl chains
    RealSweep(const int n[3], const double k[3], double ds, int nl, bool os2);
    ~RealSweep();
    RealSweep(const RealSweep&) = delete;
    RealSweep& operator=(const RealSweep&) = delete;
    // whether a grid has a sweep
    static bool supported(int Lx, int Ly, int Lz);
    // the solve's description: chains and number of steps
    RealProblem problem(const RealLane* lanes, int Ns) const;
    // chooses the x-tile variant by timing whole sweeps of p, once per device
    // and grid shape in a process (PS_B200_AUTOTUNE=0 keeps the default,
    // PS_B200_SWEEP_VARIANT=v forces variant v)
    void tune(const RealProblem& p, cudaStream_t st);
    void enqueue(const RealProblem& p, cudaStream_t st) const;
    bool tiled() const { return tile_; }   // 2D, the chains in tiles of lines
    int cluster() const { return cluster_; }
    // whether a sweep that has ended gave up at a barrier (the fields it wrote are not
    // the chains'), throwing if so, and a new start after that
    bool failed() const;
    void check() const;
    void reset();

private:
    void init(const int n[3], const double k[3], double ds, int nl, bool os2);
    void release();
    int n_[3], dim_, nl_, os2_, ncta_, variant_, fo_[3], nfrag_;
    bool tile_ = false;
    int cluster_ = 0;   // CTAs of a chain's cluster (0: chains over the grid)
    double *work_ = nullptr, *frag_ = nullptr;
    unsigned* bar_ = nullptr;   // 32 words, then the error flag
    int* notice_ = nullptr;     // the error flag's copy in host memory (forms with barriers in memory)
    int hasty_ = 0;
};

}  // namespace ps
