// sweep.h -- RQM4 sweeps of batches of 2D problems, one thread-block cluster
// per problem (cluster_sweep.cu).
#pragma once

#include <cuda_runtime.h>

namespace ps {

struct SweepArgs {
    double *hf, *hc;                 // histories, (Ns + 1) x M each (slice 0 = head)
    const double *eFA, *eHA, *eFB, *eHB;   // Boltzmann factors of the A and B blocks
    const double2 *twx, *twy;        // twiddles (set by the launcher)
    int LA, LB, Ns;
    long bstride_batch;              // per-problem stride of M-sized arrays
    long bstride_hist;               // per-problem stride of the histories
    const double* ktab;              // per-axis exp(h k_x^2), exp(h k_y^2), h = ds then ds/2
};

bool cluster_sweep_supported(int Lx, int Ly, int Lz);
// sets kernel attributes, builds twiddles; returns how many clusters fit at once
int cluster_sweep_prepare(int Lx, int Ly, int Lz, int nbatch);
void cluster_sweep_launch(const SweepArgs& a, int Lx, int Ly, int Lz, int nbatch, cudaStream_t st);

}  // namespace ps
