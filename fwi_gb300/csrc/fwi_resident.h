// Plan of the resident kernel (fwi_resident.cu): plain structs shared by the
// host planner (fwi_resident_plan.cpp, no CUDA dependency) and the kernel.
//
// A resident launch runs the whole time loop of a few shots with their state
// (two pressure levels, CPML memory variables) in the shared memory of the
// GPU's SMs.  A shot's padded grid below the free surface -- rows
// 0..ny+dn-1, logical columns 0..nxt-1 -- is cut into a gx x gy grid of
// tiles, one thread block each; neighbouring tiles exchange the R rows and
// four columns next to their common edge every step.
#pragma once
#include <cstddef>
#include <vector>

#include "fwi_lists.h"

namespace fwi {

// Threads of one tile that do the same kind of work: a thread owns one quad
// (four columns, kinds 0 and 1) or one column (kinds 2 and 3) in `h`
// consecutive rows.  Consecutive threads take consecutive quads or columns,
// then the next band of h rows; a band takes `np` >= n threads, so that the
// quarter warps (lanes of one 128-byte shared-memory access) of a band do not
// straddle two bands.
struct ResGroup {
    int kind;        // 0 interior quads of the model rows, 1 quads of the bottom pad rows (y-CPML),
                     // 2 side-strip columns of the model rows, 3 of the bottom pad rows
    int x0, n, np;   // first logical column; number of quads / columns; threads per band
    int y0, y1;      // rows [y0, y1)
    int h;           // rows per thread
    int warp0, nwarps;
};

// A tile's step has two phases, each with groups of its own over all threads:
// the cells next to the tile's neighbours (the rows and columns they read),
// then the rest while those travel.
constexpr int RES_GROUPS = 26;
constexpr int RES_THREADS = 384;         // computing threads of a block (one block per SM) and
constexpr int RES_COMM = 128;            // threads that exchange the edges: 128 registers each (144 and 80: no faster)
constexpr int RES_BLOCK = RES_THREADS + RES_COMM;
constexpr size_t RES_STATIC_SMEM = 2048; // static shared memory of the kernel, rounded up

struct ResTile {
    int shot;                // index in the launch
    int x0, x1, y0, y1;      // logical columns [x0, x1) (x0 a multiple of 4), rows [y0, y1) below the free surface
    int nbr[4];              // tiles to the left, right, above and below in the launch (-1: none)
    int ngroups[2];          // groups of the first phase, then of the second
    ResGroup g[RES_GROUPS];
    int src0[2], src1[2];    // ResSrc ranges, forward and adjoint
    int rec0, rec1;          // ResRec range
    int lines[2];            // source lines, forward and adjoint
    int rows[2];             // first entry of the tile's row table (y1 - y0 ints), forward and adjoint
    // pairs of edge words the tile exchanges with its neighbours, the sides one after the other (each from pair0 on);
    // its outbox holds the pairs it sends, in the same order, once in the plane of the even steps and once in that of
    // the odd ones
    int npair, pair0[4];
    int out;                 // words of the outboxes before its own, of both planes
    int c2;                  // first element of the tile's c2 (rows of cp values) in global memory
    // shared memory (floats): pressure levels; x-CPML (left, right), y-CPML; c2 of the strip columns, of the bottom
    // pad rows and, where there is room, of the whole tile (o_c2; else -1); source lines, row table, factors, edge
    // pairs, receivers, sources
    int pitch, cp;           // row pitch of the pressure levels; of c2, the y-CPML arrays and the source lines
    int nl, nr;              // strip columns of the tile, left and right
    int o_p[2], o_xl, o_xr, o_y, o_cl, o_cr, o_cb, o_c2, o_line, o_row, o_fac, o_pair, o_rec, o_src;
    int floats;              // with the longer of the two source-line sets
};

struct ResSrc {
    int pos;                 // position in the tile's source lines (line * cp + column)
    int vidx;                // index into the shot's value table [vidx][nt]
};
struct ResRec {
    int off;                 // offset in a pressure level
    int ridx;                // receiver index: Rec_point(:, ridx+1)
};

// A launch: the tiles of a group of shots and their source and receiver lists.
struct ResPlan {
    bool c2_shared = false;          // c2 of the quads in shared memory
    std::vector<ResTile> tiles;      // shot after shot
    std::vector<ResSrc> src;
    std::vector<ResRec> rec;
    std::vector<int> rows;           // row tables: the row's source line, or -1
    size_t out_elems = 0;            // outbox words of all tiles
    size_t c2_elems = 0;             // c2 values of all tiles
    size_t smem = 0;                 // bytes of dynamic shared memory (the largest tile's)
};

// Device limits the planner works with.
struct ResDevice {
    int sms = 0;
    size_t smem_sm = 0;      // shared memory per SM
    size_t smem_block = 0;   // largest opt-in size per block
};

// The cut of one shot's grid: column bounds (multiples of 4, the last nxt) and
// row bounds.
struct ResCut {
    std::vector<int> xs, ys;
    double us = 0.0;          // modelled step of the slowest tile
    size_t smem = 0;          // largest tile's shared memory without sources and receivers (bytes)
};
// The cuts of the shots of a launch (they depend on the grids alone).
struct ResCuts {
    std::vector<ResCut> shots;
    bool c2_shared = false;
    double step_us = 0.0;    // modelled time of one step
};

// Cut the shots of a launch, c2 in shared memory where they fit with it (and
// c2_shared allows it); false when they do not fit the device together.
bool res_cuts(const std::vector<const Layout*>& lays, const ResDevice& dev, ResCuts& out, bool c2_shared = true);
// Plan a launch for the shots (geoms[i], lays[i]) with their cuts, or, where a
// tile's sources and receivers do not fit beside its c2, with cuts that keep
// c2 in global memory; false when they do not fit there either.
bool res_plan(const std::vector<const ShotGeom*>& geoms, const std::vector<const Layout*>& lays, const ResCuts& cuts,
              const ResDevice& dev, ResPlan& out);

// Number of shots per launch (of the shots in the given order, cut into equal
// groups of at most max_shots) with the smallest modelled time; 0 when some
// shot does not fit.  *us: that time, per step of all shots.
int res_group(const std::vector<const Layout*>& lays, const ResDevice& dev, int max_shots, double* us = nullptr);

// The launches of a survey, over its shots in the given order.
struct ResSurvey {
    int shots = 0;                  // per launch
    double us = 0.0;                // modelled time of a step of all shots
    std::vector<ResPlan> launches;
};
// The shots per launch that res_group chooses, or the next smaller choice whose
// launches hold their sources and receivers (the cuts are made for the grids
// alone); false when no choice within limit_us does.
bool res_survey(const std::vector<const ShotGeom*>& geoms, const std::vector<const Layout*>& lays, const ResDevice& dev,
                int max_shots, double limit_us, ResSurvey& out);

}  // namespace fwi
