// batch_ab.h -- independent Model_AB solves of uneven grids and contour
// lengths advanced together (see batch_ab.cu).
#pragma once

#include <vector>

#include "engine.h"
#include "grouped_pass.h"

namespace ps {

class BatchAB {
public:
    // AB solves are members 0 .. ps.size() - 1, ABC triblock solves follow
    explicit BatchAB(const std::vector<ModelABParams>& ps, const std::vector<ModelABCParams>& qs = {});
    ~BatchAB();
    int size() const { return (int)(m_.size() + t_.size()); }
    int size_ab() const { return (int)m_.size(); }
    ModelAB& model(int k);
    ModelABC& model_abc(int k);   // k counts from the first ABC member (k >= size_ab())
    void set_fields(int k, const double* wA, const double* wB, bool device_ptrs);
    void set_fields_abc(int k, const double* const w[3], bool device_ptrs);
    void update(int n);
    // update() between CUDA events on the batch stream; returns the device ms
    double update_timed(int n);
    void sync();   // and the members' check()
    int launches_per_iteration() const { return launches_; }
    int launches_per_propagate() const { return launches_prop_; }
    // sum over solves of 2 Ns M: gridpoint contour steps of one iteration
    double gridpoint_steps_per_iteration() const;

private:
    struct Group {
        int naxes = 0, Ns_max = 0;
        int path[3] = {0, 0, 0};              // schedule of each axis role (in, mid, out)
        std::vector<int> members;            // solve indices, Ns descending
        std::vector<int> Ns;                  // Ns of members, same order
        GroupSolve* dev = nullptr;            // descriptors on the device
        int* prefix_dev[9] = {};              // CTA offsets per pass kind
        std::vector<int> prefix[9];
        size_t smem[9] = {};
    };
    // solves that share a sweep launch: their descriptors on the device, and
    // 32 barrier words each (3D)
    struct SweepChunk {
        int n = 0, grid = 0, pairs = 0, hasty = 0;
        int cluster = 0;
        bool plane = false, wide = false;
        size_t smem = 0;
        RealProblem* dev = nullptr;
        unsigned* bar = nullptr;
    };
    void build_group(Group& g);
    GroupSolve describe(int k) const;   // grouped-pass descriptor of member k
    PairChain* chain_of(int k) const;
    int Ns_of(int k) const;
    double points_of(int k) const;
    RealProblem sweep_descriptor(int k) const;
    const RealSweep* sweep_of(int k) const;
    void add_chunk(const std::vector<int>& ks, const std::vector<int>& per, int cluster);
    void build_sweeps(const std::vector<int>& members);
    void wait();
    void release();
    void enqueue_iteration();
    std::vector<ModelAB*> m_;
    std::vector<ModelABC*> t_;
    std::vector<Group> groups_;
    std::vector<SweepChunk> chunks_;
    std::vector<int> own_;                   // solves propagated by their own sweep launch
    cudaStream_t st_ = nullptr;
    cudaGraphExec_t graph_ = nullptr;
    int launches_ = 0, launches_prop_ = 0;
};

}  // namespace ps
