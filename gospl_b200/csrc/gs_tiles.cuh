// Dataflow sweeps over mesh tiles (gs_tiles.cu).
#pragma once
#include <stdint.h>

struct gs_plan;

namespace gs {

// records of one graph (gs_tiles.cu): pm holds per position the predecessor
// slots and the successor flags
struct TileGraph {
    char* rec = nullptr;
    uint16_t* pm = nullptr;
};

// TG_SNAP: the snapshot flow graph (receivers of the unfilled surface), whose
// edges passed the acyclicity check; TG_CASCADE: any other donors-first graph;
// TG_UP: receivers-first graphs
enum { TG_SNAP = 0, TG_CASCADE = 1, TG_UP = 2, TG_N = 3 };
// the snapshot graph's edges with other weights, in TG_CASCADE's records
enum { TG_FLUX = TG_N };

// the plan's tiles (tl_nt = 0 when the mesh keeps the ordered sweeps; tl_cas > 0:
// but for the cascade's flow)
int tiles_setup(gs_plan* p, const int32_t* nnb, const int32_t* ngb);
void tiles_free(gs_plan* p);
// Records of graph `which` from the receiver edges rcv/rslot with a non-zero
// coefficient co ([R][n]): down = donors are solved before their receivers
// (flow), else receivers before donors (stream power); div = divide by
// 1 + sum of the vertex's co.  *bad (device) becomes 1 when an edge does not
// go down in (z, pdir, -id) (z given) or is not an edge of the donor graph
// `ref` (the pm of a graph built with down).
int tile_build(gs_plan* p, int which, bool down, bool div, const int* rcv, const double* co, const int8_t* rslot,
               const double* z, const int* pdir, const uint16_t* ref, int* bad);
// the same for the marine receivers (bit sets over the neighbour slots, one
// weight per donor) of the surface z
int tile_build_marine(gs_plan* p, int which, const unsigned short* cand, const double* w, const double* z, int* bad);
// x_v = (b_v + sum over predecessors of w x) [/ divisor] over graph `which`,
// issued on the plan's stream.  The status word is sticky: 0, GS_ETIMEOUT, or
// TILE_REJECTED when *skip (device, may be null) was set; read it with
// tile_status (synchronises) or tile_status_async and tile_status_check
int tile_solve(gs_plan* p, int which, bool div, const double* b, double* x, const int* skip);
int tile_status_async(gs_plan* p, int* host);
int tile_status_check(gs_plan* p, int st, const char* what);
int tile_status(gs_plan* p, const char* what);

constexpr unsigned TILE_REJECTED = 0x100u;   // the graph failed its check: nothing was solved

}  // namespace gs
