// cfdl_amg.h -- aggregation multigrid hierarchy (host build, device view).
#pragma once
#include "cfdl_internal.h"

namespace cfdl {

constexpr int kAmgCoarsest = 64;     // dense (pseudo-)inverse at or below this many cells
constexpr int kAmgMaxLevels = 12;

// Level-0 (mesh) graph handed to the builder: ELL neighbours (-1 or >= n for
// "no interior neighbour") and the strength of each slot.
struct AmgFineView {
    int n, W;
    const int *nb;
    const double *strength;
};

// One coarse level, host side.  Slots are ELL slot indices k*n + i of the
// finer level; "fine" means the level just above.
struct AmgHostLevel {
    int n_fine = 0, n = 0, W_fine = 0, W = 0;
    FillVec<int> agg;                  // [n_fine] coarse cell of each fine cell
    FillVec<int> mem_ptr, mem;         // members of each coarse cell
    FillVec<int> nb;                   // [W][n] coarse neighbours, -1 padded
    FillVec<int> g_ptr, g_src;         // fine slots summed into coarse slot s = k*n + c
};

struct AmgHierarchy {
    std::vector<AmgHostLevel> levels;
};

int build_amg_hierarchy(const AmgFineView &fine, AmgHierarchy &H);

// One coarse level, device side (all pointers device).
struct AmgLevelDev {
    int n, W, n_fine, W_fine;
    const int *nb, *agg, *mem_ptr, *mem, *g_ptr, *g_src;
    const int *len;                           // [n] couplings of each row (its slots k < len are the valid ones)
    double *a, *dg, *rd, *r, *z, *t;          // FP64 operator and V-cycle vectors
    float *a32, *dg32, *rd32, *r32, *z32, *t32; // FP32 copies (mixed-precision form)
};

// Plan of a case's tail for one precision, built on the host when the
// hierarchy is: the levels counted from the tail level, their arrays, and the
// places (bytes from the start of the dynamic shared memory) they are staged
// at.  S slots of each row are staged: all of them unless memory runs out; the
// tail level's last slots are then read from global memory.  The rest is
// bounded: aggregation at least halves a level but for isolated cells, of
// which a usable hierarchy has at most kAmgCoarsest, so the levels hold fewer
// than 5000 rows in all and everything but the slots takes under 190 KB.
struct TailLevel {
    int n, R, S, whole;                                    // rows, rows per CTA, staged slots, done whole
    int sa, snb, srd, sdg, slen, sr;                       // the CTA's own rows
    int sz, sagg, smem_, smptr;                            // the whole level
    const void *a, *rd, *dg;
    const int *nb, *len, *agg, *mem, *mptr;
};
struct TailPlan {
    int nl, nc;                                            // smoothed levels; rows of the coarsest
    int t[2], w[2], sz, sr, sminv, total;
    const void *r, *minv;                                  // the tail level's r, the coarsest inverse
    void *z;                                               // the tail level's z
    TailLevel lv[kAmgMaxLevels];
};


}  // namespace cfdl
