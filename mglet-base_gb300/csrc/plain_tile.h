// plain_tile.h -- the plain form's single-level pressure solve on tiles.
#pragma once

#include "internal.h"
#include "sip_tile.cuh"

namespace mg {

// Arrays are [ngrid][npp], class arrays [ncls][n][npp], FP64.
struct PlainTile {
    TileDev t;
    int pair = 0;               // 1: tiles of two cells along k, 0: single cells
    int ncls = 0;
    bool unicls = false;        // every class has one value of each operator coefficient
    double* mem = nullptr;      // holds the FP64 arrays below
    int *gcls = nullptr, *fnbr = nullptr;
    double *cf = nullptr, *cb = nullptr, *lap = nullptr, *uni = nullptr;   // 4, 3, 7 arrays; [ncls][8]
    double *h = nullptr, *rhs = nullptr, *dp = nullptr, *rs[3] = {nullptr, nullptr, nullptr};
    double* gridmax = nullptr;  // [ngrid]
    double* stat = nullptr;     // device {max |rhs|, ints: converged, error, outer iterations}
    double* h_stat = nullptr;   // pinned copy
    bool lose_once = false;     // test switch: a wait of the next solve's forward sweeps runs out
};

// Set up when the context's grids take it: one level, equal dimensions, SIP in
// plane order, face neighbours on opposite faces, and the memory for it (6 FP64 arrays,
// 14 more of every class of grids with equal faces and spacing).  c->ptile stays null
// otherwise.
int plain_tile_init(Ctx* c, const mglet_grid_desc* d);
// Does the solve run on tiles?
bool plain_tile_ready(const Ctx* c);
// mglet_gpu_test_sweep_timeout
int plain_tile_test_timeout(Ctx* c);

}  // namespace mg
