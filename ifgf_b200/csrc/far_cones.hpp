// Far-cone plan: the (target, far box) pairs of an operator sorted by the fine
// cone they evaluate, for the far field of the single matvec (far_cones.cuh).
#pragma once

#include <vector>

#include "devbuf.hpp"
#include "mult.hpp"

namespace ifgf
{

struct FarConePlan
{
    DevBuf<unsigned char> mem; // everything `p` points to
    FarConePtrs p;
    long long pairs = 0, places = 0;
    double ms = 0; // of the build, the kernels enqueued before it included
    bool ready = false;
    bool refused = false;  // nothing to build, or too many places
    int wait = 0;          // matvecs until another attempt, after want of memory
    bool captured = false; // a stream capture holds its addresses
    void release();
};

struct FarConeBuild
{
    const std::vector<LevelGeom>* lv;
    const LevelGeom* lv_dev;
    TreeArgs T;
    const double *tx, *ty, *tz;
    const int* fmap;
    const int* tl_first;
    const int* tl_last;
    const long long* far_off;
    // first (far box, target) pair of every target leaf, and their number
    const std::vector<long long>* leaf_off;
    const int* far_src;
    int n_tleaf;
    // fine cones of every level: box, element (device arrays)
    std::vector<const int*> cone_box, cone_el;
    unsigned long long* err;
    bool mixed = false; // lookups of the mixed pipeline
    cudaStream_t stream = nullptr; // that the build runs on
};

// A plan is one allocation.  Small ones (up to FAR_CONES_RESERVE) get it with
// the operator's other buffers at init: an allocation of 2 MB or more takes
// some 0.35 ms, as long as everything else a small plan's build does.
constexpr size_t FAR_CONES_RESERVE = size_t(64) << 20;
void reserve_far_cones(const FarConeBuild& b, FarConePlan& plan);

// Without memory a plan is tried again after this many matvecs (asking for
// the free memory takes some tens of microseconds).
constexpr int FAR_CONES_RETRY = 16;

// Fills `plan`, or leaves it empty: with `refused` set for no far pairs or 2^31
// places or more, with `wait` set where it would take more than a quarter of
// the free device memory or finds none (3.9e8 pairs take 12 ms).  Runs on the
// build's stream and waits for that one alone.
void build_far_cones(const FarConeBuild& b, FarConePlan& plan);

} // namespace ifgf
