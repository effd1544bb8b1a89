// Cluster tail of the nodal V-cycle (hg_tail.cu): parameters and launchers.
#pragma once

#include "mac_internal.cuh"
#include "hg_nodal.cuh"

namespace mac {

constexpr int kHgTailLevels = 8;
constexpr int kHgTailThreads = 512;
constexpr int kHgTailSmem = 200 * 1024;
constexpr int kHgTailBottom = 640;   // unknown nodes of an exactly solved bottom at most

template <typename T>
struct HgTailParams {
    hg::Geo geo;
    int nlev;                         // levels above the bottom
    hg::LevT<T> lev[kHgTailLevels];   // of the dense 3-D hierarchy, finest first
    int iso[kHgTailLevels];           // the axis neighbours' weight is exactly 0
    const T* f0;                      // right-hand side of the first level (node array)
    T* e0;                            // its correction (unknown nodes written)
    int nu1, nu2, singular;
    // bottom: its geometry, M unknown nodes (storage indices), node -> unknown (-1: none), inverse
    hg::LevT<T> bot;
    int M;
    const int* node;
    const int* map;
    const double* binv;
    int ldb;                          // its row pitch
    // plan (hg_tail_plan)
    int spc[kHgTailLevels];           // slabs a CTA
    int off[kHgTailLevels];           // byte offset of the level's arrays
    unsigned mag[kHgTailLevels][2];   // reciprocal of a row's nodes of x parity 0 / 1
    int boff;                         // bottom: byte offset
};

// Fills the plan for a cluster of nc CTAs; the dynamic shared memory of a CTA, 0 when it does not fit.
template <typename T>
size_t hg_tail_plan(HgTailParams<T>& P, int nc);
template <typename T>
void launch_hg_tail(const HgTailParams<T>& P, size_t smem, int nc, cudaStream_t s);
int prepare_hg_tail_kernels(int* nc);

}  // namespace mac
