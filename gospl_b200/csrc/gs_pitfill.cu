// Depression filling: PITFill.fillElevation(sed=False) (pitfilling.py:849-903).
//
// Filled surface.  On one GPU the reference's three Barnes phases (per-tile
// Priority-Flood fill_tile, label-graph flood fill_edges, fill_depressions)
// reduce to the plain Priority-Flood fill: the minimax over paths to the seed
// set of the highest shifted elevation along the path.  (Each watershed label
// is created by a seed that drains to label 0, so the label-graph level of a
// watershed never exceeds the fill of its cells and fill_depressions keeps the
// flood values.)  The GPU computes that minimax without a heap:
//   1. steepest non-ascending descent (lexicographic (z, id)) links every cell
//      to a root: a seed or a local minimum (a basin);
//   2. for each pair of adjacent basins the spill height is max(z_u, z_v);
//   3. basin levels L(b) = minimax over basin-graph paths to a seed basin, by
//      contracting the graph along the components' lowest edges;
//   4. fill = max(z, L(basin)).
// Only comparisons are involved, so the result is bit-identical to the
// reference's heap-ordered flood.  Seeds and exclusions follow edge_tile
// (functions.F90:2036-2080) on z - level; cells at or below the level keep
// their elevation (fill_depressions, 2290-2329) and open-sea cells are reset
// (pitfilling.py:689-693).
//
// Pit bookkeeping follows _pitInformation (pitfilling.py:704-847):
// label_pits (equal-fill components holding a cell with no lower neighbour,
// numbered by their smallest seed id) by union-find; pits_cons renumbering;
// spill selection by smallest id; fill_dir / nghb_dir hop distances by a
// search in each depression; the (distance, id) flat receiver pick; pit volumes,
// depths and depth-volume curves (_getPitParams, getpitvol) by deterministic
// segmented reductions over pit-sorted cells.
#include <cub/cub.cuh>

#include <cfloat>
#include <climits>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>

#include "gs_plan.cuh"

namespace cg = cooperative_groups;

namespace gs {

__device__ __forceinline__ int agg_append(int* cnt) {
    cg::coalesced_group g = cg::coalesced_threads();
    int base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(cnt, (int)g.size());
    return g.shfl(base, 0) + (int)g.thread_rank();
}

// d_scalar: smallest height, fill level, level above which cells are labelled
enum { D_MINH = 0, D_LEVEL = 1, D_LABEL = 3 };
// u_scalar: min key, non-finite and block count of k_level; the fill's outcome
enum { U_LEVEL = 8, U_OUT = 12 };
// words of the outcome, as the host reads them into h_pinned + 6
enum { F_ROUNDS = 0, F_EDGES, F_PITS, F_NONFINITE, F_CELLS, F_COUNT };
enum { I_ROUNDS = 0, I_NEXT = 1, I_BASINS = 2, I_FLAGS = 5, I_NONFINITE = 13 };

// --------------------------------------------------------------------------
// reductions
// --------------------------------------------------------------------------
// Smallest height, fill level, and whether every input is finite, in one pass;
// the last block to finish (word[2] counts them, from -1) sets the scalars and
// clears the counters of the kernels that follow.  word[0] and word[1] start as
// all ones: the smallest key, and 0 once a value is not finite.
__global__ void __launch_bounds__(256) k_level(int n, const double* __restrict__ x, const double* __restrict__ b,
                                               unsigned long long* word, int sphere, double sealevel, double ofill,
                                               int sed, double* dsc, int* isc) {
    unsigned long long best = ~0ULL;
    bool bad = false;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const double v = x[i];
        const unsigned long long k = dkey(v);
        best = k < best ? k : best;
        bad |= !isfinite(v) || (b && !isfinite(b[i]));
    }
    for (int o = 16; o > 0; o >>= 1) {
        unsigned long long v = __shfl_xor_sync(0xffffffffu, best, o);
        best = v < best ? v : best;
    }
    bad = __any_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(word, best);
        if (bad) atomicExch(word + 1, 0ULL);
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x != 0 || atomicAdd(word + 2, 1ULL) + 2ULL != (unsigned long long)gridDim.x) return;
    __threadfence();
    double minh = dkey_inv(__ldcg(word));
    if (sphere) minh += 1.0e-3;
    const double base = sealevel + ofill;
    const double level = (base > minh) ? base : minh;   // Python max(minh, base)
    dsc[D_MINH] = minh;
    dsc[D_LEVEL] = level;
    dsc[D_LABEL] = sed ? level : sealevel;
    isc[I_NONFINITE] = __ldcg(word + 1) == 0ULL ? 1 : 0;
    isc[I_NEXT] = isc[I_BASINS] = 0;
    for (int k = 0; k < 3; k++) isc[I_FLAGS + k] = 0;
}

// --------------------------------------------------------------------------
// filled surface
// --------------------------------------------------------------------------
__global__ void k_classify(int n, const double* __restrict__ h, const double* __restrict__ dsc,
                           const int* __restrict__ nbr, const int8_t* __restrict__ nnb,
                           const uint8_t* __restrict__ outlet, int8_t* ledge) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    const double level = dsc[D_LEVEL];
    const double hs = h[c] - level;
    int8_t e = -1;
    if (hs < 0.0) {
        bool ge = false;
        for (int s = 0; s < nnb[c]; s++) {
            int j = nbr[(size_t)s * n + c];
            if (j >= 0 && h[j] - level >= 0.0) { ge = true; break; }
        }
        e = ge ? (outlet[c] ? 2 : 0) : -2;
    } else if (outlet[c]) {
        e = 2;
    }
    ledge[c] = e;
}

// The roots get their starting state for k_basin_levels: a seed level -inf and
// component -1, a local minimum level 0 (below every key; ~0 with `relax`), its
// own component, no outgoing edge yet (W), no claim, and a place in basin[].
// A cell at or above the level next to an excluded one would make it a seed
// when edges have both ends listed: then no neighbour needs a look at its class,
// and the cell's own class is found here (CLASS).
template <bool CLASS>
__global__ void __launch_bounds__(256) k_descend(int n, int relax, const double* __restrict__ h,
                                                 const double* __restrict__ dsc, const int* __restrict__ nbr,
                                                 const int8_t* __restrict__ nnb, const uint8_t* __restrict__ outlet,
                                                 int8_t* ledge, int* parent, unsigned long long* L,
                                                 unsigned long long* W, int* comp, int* claim, int* basin,
                                                 int* nbasin) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    bool list = false;
    if (c < n) {
        const double level = dsc[D_LEVEL];
        const double hc = h[c] - level;
        int8_t e = CLASS ? -1 : ledge[c];
        int best = c;
        if (CLASS && outlet[c]) e = 2;
        if (CLASS ? (e == -1 || hc < 0.0) : e == -1) {       // seeds and excluded cells are roots
            const int deg = nnb[c];
            double bz = hc;
            bool ge = false;
            for (int s0 = 0; s0 < deg; s0 += 6) {
                int j[6];
                double z[6];
#pragma unroll
                for (int t = 0; t < 6; t++) j[t] = s0 + t < deg ? nbr[(size_t)(s0 + t) * n + c] : -1;
#pragma unroll
                for (int t = 0; t < 6; t++) z[t] = j[t] >= 0 ? h[j[t]] - level : 0.0;
#pragma unroll
                for (int t = 0; t < 6; t++) {
                    if (j[t] < 0 || (!CLASS && ledge[j[t]] == -2)) continue;
                    ge |= z[t] >= 0.0;
                    if (z[t] < bz || (z[t] == bz && j[t] < best)) { bz = z[t]; best = j[t]; }
                }
            }
            if (CLASS && hc < 0.0) e = ge ? (outlet[c] ? 2 : 0) : -2;
            if (e != -1) best = c;
            list = e == -1 && best == c;
        }
        if (CLASS) ledge[c] = e;
        parent[c] = best;
        if (list) {
            L[c] = relax ? ~0ULL : 0ULL;
            W[c] = ~0ULL;
            comp[c] = c;
            claim[c] = 0;
        } else if (e >= 0) {
            L[c] = dkey(-INFINITY);
            comp[c] = -1;
        }
    }
    const unsigned full = 0xffffffffu, lists = __ballot_sync(full, list);
    if (!lists) return;
    const int lane = threadIdx.x & 31;
    int base = 0;
    if (lane == 0) base = atomicAdd(nbasin, __popc(lists));
    base = __shfl_sync(full, base, 0);
    if (list) basin[base + __popc(lists & ((1u << lane) - 1u))] = c;
}

// Every vertex walks to its basin's root and leaves what it has reached in its
// own parent on the way.  Other threads shorten the same chains concurrently;
// every parent value ever stored is an ancestor on the vertex's descent path,
// so reading a stale or a fresh value are both valid steps, and a path ends: it
// descends strictly (height, then id).
constexpr int JUMP_HOPS = 16;
__global__ void __launch_bounds__(256) k_jump(int n, int* parent) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    int p = parent[c], written = p;
    for (int hop = 1;; hop++) {
        const int pp = ld_relaxed_s32(parent + p);
        if (pp == p) break;
        p = pp;
        if (hop % JUMP_HOPS == 0) parent[c] = written = p;
    }
    if (p != written) parent[c] = p;
}

// Edges between basins: a cell at a basin's border emits one edge per distinct
// neighbouring basin, with the key of the smallest pass height (parallel edges
// of larger weight can never lower a level further), and lowers its basin's
// lowest outgoing edge W; a seed basin keeps level -inf, so no edge leads to it.
// Most cells lie inside: they look at their neighbours' roots, all gathers at
// once, and at no height; a warp reserves its edges at once.
__global__ void __launch_bounds__(256, 6) k_cross_edges(int n, const double* __restrict__ h,
                                                        const double* __restrict__ dsc, const int* __restrict__ nbr,
                                                        const int8_t* __restrict__ nnb,
                                                        const int8_t* __restrict__ ledge,
                                                        const int* __restrict__ root, unsigned long long* W, int* xu,
                                                        int* xv, unsigned long long* xw, int* count, int64_t cap) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int rc = -1, deg = 0;
    bool border = false;
    if (c < n && ledge[c] != -2) {
        rc = root[c];
        if (ledge[rc] < 0) {
            deg = nnb[c];
            for (int s0 = 0; s0 < deg; s0 += 6) {
                int j[6];
#pragma unroll
                for (int t = 0; t < 6; t++) j[t] = s0 + t < deg ? nbr[(size_t)(s0 + t) * n + c] : -1;
#pragma unroll
                for (int t = 0; t < 6; t++)
                    if (j[t] >= 0) border |= root[j[t]] != rc;
            }
        }
    }
    if (!__any_sync(full, border)) return;
    int rb[MAXW];
    double wb[MAXW];
    int cnt = 0;
    if (border) {
        const double level = dsc[D_LEVEL];
        const double zc = h[c] - level;
        unsigned long long low = ~0ULL;
        for (int s = 0; s < deg; s++) {
            const int j = nbr[(size_t)s * n + c];
            if (j < 0) continue;
            const int rj = root[j];
            if (rj == rc || ledge[j] == -2) continue;
            const double zj = h[j] - level;
            const double w = zc > zj ? zc : zj;
            low = min(low, dkey(w));
            int q = 0;
            while (q < cnt && rb[q] != rj) q++;
            if (q == cnt) {
                rb[cnt] = rj;
                wb[cnt] = w;
                cnt++;
            } else if (w < wb[q]) {
                wb[q] = w;
            }
        }
        if (cnt && low < __ldcg(W + rc)) atomicMin(W + rc, low);
    }
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(full, incl, o);
        if (lane >= o) incl += v;
    }
    int base = 0;
    if (lane == 31 && incl) base = atomicAdd(count, incl);
    const int64_t pos = (int64_t)__shfl_sync(full, base, 31) + incl - cnt;
    for (int q = 0; q < cnt; q++)
        if (pos + q < cap) {
            xu[pos + q] = rc;
            xv[pos + q] = rb[q];
            xw[pos + q] = dkey(wb[q]);
        }
}

// The filled surface, and the starting values of the labels and pit tables.
// An input that is not finite leaves lfill as it was.
__global__ void k_fill_final(int n, const double* __restrict__ h, const double* __restrict__ dsc,
                             double sealevel, const int8_t* __restrict__ ledge,
                             const int* __restrict__ root, const unsigned long long* __restrict__ L,
                             const int* __restrict__ isc, double* lfill, int* minseed, int* present, int* bestlid,
                             int* spill_flag, int* seg_count) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= n) return;
    minseed[c] = INT_MAX;
    present[c] = 0;
    bestlid[c] = INT_MAX;
    spill_flag[c] = 0;
    seg_count[c] = 0;
    if (c == 0) {
        present[n] = 0;
        bestlid[n] = INT_MAX;
        seg_count[n] = seg_count[n + 1] = 0;
    }
    if (isc[I_NONFINITE]) return;
    const double level = dsc[D_LEVEL];
    const double hs = h[c] - level;
    double f = hs;
    if (ledge[c] != -2) {
        unsigned long long k = L[root[c]];
        if (k != ~0ULL) {
            double lv = dkey_inv(k);
            f = lv > hs ? lv : hs;
        }
    }
    double out = (hs > 0.0) ? f : hs;          // fill_depressions: dem > lvl only
    if (out < sealevel - level) out = hs;      // open sea stays unfilled
    lfill[c] = out + level;
}

// --------------------------------------------------------------------------
// label_pits by union-find
// --------------------------------------------------------------------------
__device__ int uf_root(int* comp, int x) {
    for (int it = 0; it < 1 << 20; it++) {
        int p = ((volatile int*)comp)[x];
        if (p == x) return x;
        int gp = ((volatile int*)comp)[p];
        if (gp != p) atomicCAS(&comp[x], p, gp);
        x = p;
    }
    return x;
}

// union-find start: every cell above sea level points to its smallest-id
// equal-fill neighbour (or itself), so the linking pass starts from short
// chains instead of singletons
__global__ void k_uf_init(int n, const double* __restrict__ f, const double* __restrict__ dsc, const int* __restrict__ nbr,
                          const int8_t* __restrict__ nnb, int* comp) {
    const double sl = dsc[D_LABEL];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int best = i;
    const double fi = f[i];
    if (fi > sl) {
        for (int s = 0; s < nnb[i]; s++) {
            int j = nbr[(size_t)s * n + i];
            if (j >= 0 && j < best && f[j] == fi) best = j;
        }
    }
    comp[i] = best;
}

__global__ void k_uf_link(int n, const double* __restrict__ f, const double* __restrict__ dsc, const int* __restrict__ nbr,
                          const int8_t* __restrict__ nnb, int* comp) {
    const double sl = dsc[D_LABEL];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double fi = f[i];
    if (!(fi > sl)) return;
    for (int s = 0; s < nnb[i]; s++) {
        int j = nbr[(size_t)s * n + i];
        if (j < 0 || j > i || f[j] != fi) continue;
        for (int it = 0; it < 1 << 20; it++) {
            int a = uf_root(comp, i), b = uf_root(comp, j);
            if (a == b) break;
            if (a < b) { int t = a; a = b; b = t; }
            if (atomicCAS(&comp[a], a, b) == a) break;
        }
    }
}


__global__ void k_minseed(int n, const double* __restrict__ f, const double* __restrict__ dsc,
                          const int* __restrict__ nbr, const int8_t* __restrict__ nnb, int* comp, int* minseed) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double fi = f[i];
    if (!(fi > dsc[D_LABEL])) return;   // alone in its component
    const int r = uf_root(comp, i);
    comp[i] = r;
    for (int s = 0; s < nnb[i]; s++) {
        int j = nbr[(size_t)s * n + i];
        if (j >= 0 && fi > f[j]) return;
    }
    atomicMin(&minseed[r], i);
}

__global__ void k_seed_flag(int n, const double* __restrict__ f, const double* __restrict__ dsc, const int* __restrict__ comp,
                            const int* __restrict__ minseed, int* flag) {
    const double sl = dsc[D_LABEL];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    flag[i] = (f[i] > sl && minseed[comp[i]] == i) ? 1 : 0;
}

// label (1..P0) per cell, then outlets removed; present[label] marks survivors
__global__ void k_label(int n, const double* __restrict__ f, const double* __restrict__ dsc, const int* __restrict__ comp,
                        const int* __restrict__ minseed, const int* __restrict__ rank,
                        const uint8_t* __restrict__ outlet, int* lab, int* present) {
    const double sl = dsc[D_LABEL];
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int l = -1;
    if (f[i] > sl) {
        int ms = minseed[comp[i]];
        if (ms != INT_MAX) l = rank[ms] + 1;
    }
    if (outlet[i]) l = -1;
    lab[i] = l;
    if (l > 0) present[l] = 1;
}

// final pit ids, the sea mask when it is asked for (lFill before the flat pass
// resets open-sea cells to h: the reset keeps lFill <= sea level), the cells of
// every pit (one atomic per warp inside a pit), their flags for the compaction,
// and no flat distance.  An input that is not finite leaves pit and sea alone.
__global__ void __launch_bounds__(256) k_relabel(int n, const int* __restrict__ lab, const int* __restrict__ newid,
                                                 const int* __restrict__ isc, const double* __restrict__ f,
                                                 double sealevel, uint8_t* sea, int* pit, int* flag, int* counts,
                                                 int* pdir) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    const unsigned full = 0xffffffffu;
    const bool ok = isc[I_NONFINITE] == 0;
    int p = -1;
    if (i < n) {
        const int l = lab[i];
        p = (l > 0) ? newid[l] + 1 : -1;
        if (ok) {
            pit[i] = p;
            if (sea) sea[i] = f[i] <= sealevel ? 1 : 0;
        }
        flag[i] = p >= 0 ? 1 : 0;
        pdir[i] = -1;
    }
    const unsigned in = __ballot_sync(full, p >= 0);
    if (!in) return;
    const int first = __ffs(in) - 1, p0 = __shfl_sync(full, p, first);
    if (__all_sync(full, p < 0 || p == p0)) {
        if ((threadIdx.x & 31) == first) atomicAdd(&counts[p0], __popc(in));
    } else if (p >= 0) {
        atomicAdd(&counts[p], 1);
    }
}

// --------------------------------------------------------------------------
// spill points, flat distances, flat receivers
// --------------------------------------------------------------------------
__device__ __forceinline__ void rim_tests(int i, int n, const double* f, const int* pit,
                                          const int* nbr, const int8_t* nnb, const uint8_t* outlet,
                                          bool* lower, bool* eq) {
    bool lo = false, e = false;
    const double fi = f[i];
    for (int s = 0; s < nnb[i]; s++) {
        int j = nbr[(size_t)s * n + i];
        if (j < 0) continue;
        double fj = f[j];
        if (fj < fi) lo = true;
        else if (fj == fi && (outlet[j] || pit[j] == -1)) e = true;
    }
    *lower = lo;
    *eq = e;
}

__global__ void k_spill_qual(int n, const double* __restrict__ f, const int* __restrict__ pit,
                             const int* __restrict__ nbr, const int8_t* __restrict__ nnb,
                             const uint8_t* __restrict__ outlet, int* bestlid) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int p = pit[i];
    if (p < 0) return;
    bool lo, eq;
    rim_tests(i, n, f, pit, nbr, nnb, outlet, &lo, &eq);
    if (lo || eq) atomicMin(&bestlid[p], i);
}

__global__ void k_spill_pick(int np1, int n, const double* __restrict__ f, const int* __restrict__ pit,
                             const int* __restrict__ nbr, const int8_t* __restrict__ nnb,
                             const uint8_t* __restrict__ outlet, const int* __restrict__ bestlid,
                             int* pit_info, int* spill_flag, int* pdir) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np1) return;
    int spill = -1, rank = -1;
    int i = (p > 0) ? bestlid[p] : INT_MAX;
    if (i != INT_MAX) {
        bool lo, eq;
        rim_tests(i, n, f, pit, nbr, nnb, outlet, &lo, &eq);
        if (lo) {
            spill = i;
        } else {
            const double fi = f[i];
            int best = INT_MAX;
            for (int s = 0; s < nnb[i]; s++) {
                int j = nbr[(size_t)s * n + i];
                if (j < 0) continue;
                if (f[j] == fi && (outlet[j] || pit[j] == -1) && j < best) best = j;
            }
            spill = best;
        }
        rank = 0;
        spill_flag[spill] = 1;
        pdir[spill] = 1;
    }
    pit_info[2 * p] = spill;
    pit_info[2 * p + 1] = rank;
}

// BFS over the compacted set of reachable vertices (pit cells and spill
// nodes, local ids 0..M-1) in one block: the visited set is a shared-memory
// bitmap and the frontiers live in shared memory, so a level costs one global
// load of the adjacency rows, warp-aggregated appends and one block barrier.
__global__ void k_bfs_flag(int n, const int* __restrict__ pit, const int* __restrict__ spill_flag, int* flag) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) flag[i] = (pit[i] > -1 || spill_flag[i]) ? 1 : 0;
}

__global__ void k_bfs_local_build(int n, int S, const double* __restrict__ f, const int* __restrict__ pit,
                                  const int* __restrict__ flag, const int* __restrict__ lid,
                                  const int* __restrict__ nbr, const int8_t* __restrict__ nnb,
                                  const int* __restrict__ spill_flag, int* rows, int* l2g, int* ld,
                                  int* seeds, int* nseed) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !flag[i]) return;
    const int li = lid[i];
    l2g[li] = i;
    ld[li] = -1;
    const double fi = f[i];
    int* row = rows + (size_t)li * S;
    int k = 0;
    for (int s = 0; s < nnb[i]; s++) {
        int c = nbr[(size_t)s * n + i];
        if (c < 0 || pit[c] < 0 || !(f[c] >= fi)) continue;
        row[1 + k++] = lid[c];
    }
    row[0] = k;
    if (spill_flag[i]) seeds[agg_append(nseed)] = li;
}

__global__ void k_bfs_local_scatter(int M, const int* __restrict__ l2g, const int* __restrict__ ld, int* pdir) {
    int li = blockIdx.x * blockDim.x + threadIdx.x;
    if (li < M && ld[li] > 0) pdir[l2g[li]] = ld[li];
}

constexpr int LBFS_CAP = 6144;
constexpr int LBFS_SMEM = 200 * 1024;   // frontiers and visited set; larger sets are searched in tiles

// S4: int4 words of a packed adjacency row (S = 4 * S4 ints, row[0] the
// count).  A level's cost is the instruction chain of its busiest warp, so
// the row width is a compile-time constant and the claimed cells are
// appended by walking the set bits of the claim mask.
template <int S4>
__global__ void __launch_bounds__(1024) k_bfs_local(int M, int S, const int* __restrict__ rows,
                                                    const int* __restrict__ seeds, const int* __restrict__ nseed_p,
                                                    int* gA, int* gB, int* ld, int* levels_out) {
    extern __shared__ unsigned smem_u[];
    unsigned* vis = smem_u;                           // ceil(M/32) words
    const int nw = (M + 31) >> 5;
    int* fA = (int*)(smem_u + nw);
    int* fB = fA + LBFS_CAP;
    // three rotating frontier counters: level r reads s_cnt[r%3], appends to
    // s_cnt[(r+1)%3] and clears s_cnt[(r+2)%3], so one barrier per level
    // separates every write of a counter from its reads
    __shared__ int s_cnt[3];
    const int tid = threadIdx.x, nt = blockDim.x, lane = tid & 31;
    for (int w = tid; w < nw; w += nt) vis[w] = 0u;
    if (tid < 3) s_cnt[tid] = 0;
    __syncthreads();
    int size = *nseed_p;
    // seeds: distance 1; frontier entries beyond LBFS_CAP live in global memory
    for (int t = tid; t < size; t += nt) {
        int li = seeds[t];
        atomicOr(&vis[li >> 5], 1u << (li & 31));
        if (t < LBFS_CAP) fA[t] = li;
        else gA[t] = li;
    }
    __syncthreads();
    int* curS = fA;
    int* nxtS = fB;
    int* curG = gA;
    int* nxtG = gB;
    int d = 1, levels = 0, r = 0;
    while (size > 0 && levels <= M) {
        int* cnt = &s_cnt[(r + 1) % 3];
        if (tid == 0) s_cnt[(r + 2) % 3] = 0;
        // every warp runs the same number of batches so that ballots see all lanes
        for (int base = 0; base < size; base += nt) {
            const int t = base + tid;
            // warps past the end of the frontier go straight to the barrier
            if (!__any_sync(0xffffffffu, t < size)) break;
            constexpr int RW = 4 * S4;
            int row[RW];
            int k = 0;
            if (t < size) {
                const int li = t < LBFS_CAP ? curS[t] : curG[t];
                const int4* r4 = reinterpret_cast<const int4*>(rows + (size_t)li * S);
#pragma unroll
                for (int q = 0; q < S4; q++) {
                    int4 v = r4[q];
                    row[4 * q] = v.x; row[4 * q + 1] = v.y; row[4 * q + 2] = v.z; row[4 * q + 3] = v.w;
                }
                k = row[0];
            }
            // claim the unvisited out-neighbours: plain checks, then the
            // atomics, all independent so their latencies overlap
            unsigned cand = 0u;
#pragma unroll
            for (int q = 1; q < RW; q++)
                if (q <= k && !(vis[row[q] >> 5] & (1u << (row[q] & 31)))) cand |= 1u << q;
            unsigned olds[RW];
#pragma unroll
            for (int q = 1; q < RW; q++)
                olds[q] = (cand & (1u << q)) ? atomicOr(&vis[row[q] >> 5], 1u << (row[q] & 31)) : 0u;
#pragma unroll
            for (int q = 1; q < RW; q++)
                if (olds[q] & (1u << (row[q] & 31))) cand &= ~(1u << q);
            // warp-aggregated append of the claimed cells
            const int mine = __popc(cand);
            int incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                int v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            const int total = __shfl_sync(0xffffffffu, incl, 31);
            int pos0 = 0;
            if (lane == 31 && total > 0) pos0 = atomicAdd(cnt, total);
            pos0 = __shfl_sync(0xffffffffu, pos0, 31);
            int pos = pos0 + incl - mine;
#pragma unroll
            for (int q = 1; q < RW; q++) {
                if (cand & (1u << q)) {
                    const int c = row[q];
                    ld[c] = d + 1;
                    if (pos < LBFS_CAP) nxtS[pos] = c;
                    else nxtG[pos] = c;
                    pos++;
                }
            }
        }
        __syncthreads();
        size = *cnt;
        int* t1 = curS; curS = nxtS; nxtS = t1;
        int* t2 = curG; curG = nxtG; nxtG = t2;
        d++;
        levels++;
        r++;
    }
    if (tid == 0) *levels_out = levels;
}

// Flat distances by tiles, in one cooperative launch (delta-stepping).  The
// reachable cells are compacted in vertex order (local ids), and vertex ids
// follow a space-filling curve, so tile t = local ids [tT, tT + T) is a
// compact patch of the mesh; with no more tiles than blocks every block keeps
// its tile's adjacency rows in shared memory for the whole launch.
// Distances are settled by windows [lo, lo + window): in a round, every tile whose
// smallest pending distance falls in the window loads its distances, relaxes
// its cells of the window and then, one block barrier per wave, the cells they
// lower within the window; a cell lowered beyond the window only records the
// tile's pending minimum, and a hop out of the tile lowers the target's
// global distance (atomicMin) and the target tile's pending minimum.  Every
// pending minimum also lowers a global minimum for the round (three rotating
// slots), which all blocks read after the grid barrier: the same window again
// while it still holds pending cells, else the next window starts at the
// smallest pending distance, and no pending cell ends the launch.  Distances
// only decrease and a window is closed only when no cell of it is pending, so
// every distance is the breadth-first hop count (exact, no timed wait).
constexpr int BFT_THREADS = 512;
constexpr int BFT_SMEM = 112 * 1024;   // most of a block's shared memory

__global__ void __launch_bounds__(BFT_THREADS, 2) k_bfs_tiles(int M, int S, int T, const int* __restrict__ rows,
                                                              const int* __restrict__ seeds,
                                                              const int* __restrict__ nseed_p, int* ld, int* ctl,
                                                              int window, int* depth_out, int* rounds_out) {
    cg::grid_group grid = cg::this_grid();
    extern __shared__ int sm_bft[];
    const int INF = 0x7fffffff;
    int* rs = sm_bft;              // [T * S] adjacency rows of the tile
    int* ds = rs + T * S;          // [T] distances
    int* fl0 = ds + T;             // [T] frontier lists
    int* fl1 = fl0 + T;
    int* xc = fl1 + T;             // [T] hops out of the tile: target, distance
    int* xd = xc + T;
    __shared__ int s_cnt[3];
    __shared__ int s_over[3];
    __shared__ int s_pmin;
    __shared__ int s_nx;
    __shared__ int s_pt;
    const int ntiles = (M + T - 1) / T;
    int* gmin = ctl;               // [3] smallest pending distance after rounds r % 3
    int* pend = ctl + 3;           // [ntiles] smallest pending distance of each tile
    const int tid = threadIdx.x, nt = blockDim.x;
    const unsigned gtid = grid.thread_rank(), gsz = (unsigned)grid.size();
    for (unsigned i = gtid; i < (unsigned)M; i += gsz) ld[i] = INF;
    for (unsigned t = gtid; t < (unsigned)ntiles; t += gsz) pend[t] = INF;
    if (gtid < 3) gmin[gtid] = INF;
    grid.sync();
    const int ns = *nseed_p;
    for (unsigned q = gtid; q < (unsigned)ns; q += gsz) {
        const int li = seeds[q];
        ld[li] = 1;
        pend[li / T] = 1;
    }
    grid.sync();
    int lo = 1, hi = window;
    int cached = -1;
    int rounds = 0;
    if (ns == 0) lo = INF;
    for (int r = 0; lo != INF; r++) {
        rounds++;
        int* gnext = gmin + ((r + 1) % 3);
        if (blockIdx.x == 0 && tid == 0) gmin[(r + 2) % 3] = INF;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
            // one thread reads the tile's pending minimum for the block: other
            // blocks lower it meanwhile, and all threads must take one branch
            __syncthreads();
            if (tid == 0) s_pt = ((volatile int*)pend)[t];
            __syncthreads();
            const int pt = s_pt;
            if (pt > hi) {
                // nothing of this window here: its pending minimum stays for later
                if (tid == 0 && pt != INF) atomicMin(gnext, pt);
                continue;
            }
            const int base = t * T, len = min(T, M - base);
            if (cached != t) {
                const int4* src = reinterpret_cast<const int4*>(rows + (size_t)base * S);
                int4* dst = reinterpret_cast<int4*>(rs);
                const int nq = len * S / 4;
                for (int q = tid; q < nq; q += nt) dst[q] = src[q];
                cached = t;
            }
            if (tid == 0) {
                atomicExch(&pend[t], INF);
                __threadfence();
            }
            __syncthreads();
            for (int i = tid; i < len; i += nt) ds[i] = ((volatile int*)ld)[base + i];
            // wave 0 relaxes every cell of the tile inside the window
            if (tid < 3) {
                s_cnt[tid] = 0;
                s_over[tid] = tid == 0 ? 1 : 0;
            }
            if (tid == 0) {
                s_pmin = INF;
                s_nx = 0;
            }
            __syncthreads();
            for (int w = 0;; w++) {
                const int rd = w % 3, wr = (w + 1) % 3;
                int* lin = (w & 1) ? fl1 : fl0;
                int* lout = (w & 1) ? fl0 : fl1;
                const int full = s_over[rd];
                const int size = full ? len : s_cnt[rd];
                if (size == 0 && !full) break;
                if (tid == 0) {
                    s_cnt[(w + 2) % 3] = 0;
                    s_over[(w + 2) % 3] = 0;
                }
                for (int e = tid; e < size; e += nt) {
                    const int i = full ? e : lin[e];
                    const int d = ds[i];
                    if (d < lo || d > hi) continue;
                    const int* row = rs + i * S;
                    const int k = row[0];
                    const int nd = d + 1;
                    // lower the in-tile out-neighbours, then one append for
                    // those that dropped inside the window; hops out of the
                    // tile are buffered and applied once after the waves
                    unsigned got = 0u;
                    for (int q = 1; q <= k; q++) {
                        const int c = row[q];
                        const int lc = c - base;
                        if ((unsigned)lc < (unsigned)len) {
                            if (atomicMin(&ds[lc], nd) > nd && nd <= hi) got |= 1u << q;
                        } else {
                            const int x = atomicAdd(&s_nx, 1);
                            if (x < T) {
                                xc[x] = c;
                                xd[x] = nd;
                            } else if (atomicMin(&ld[c], nd) > nd) {
                                atomicMin(&pend[c / T], nd);
                                atomicMin(gnext, nd);
                            }
                        }
                    }
                    if (got) {
                        int pos = atomicAdd(&s_cnt[wr], __popc(got));
                        for (int q = 1; q <= k; q++) {
                            if (!(got & (1u << q))) continue;
                            if (pos < T) lout[pos] = row[q] - base;
                            else s_over[wr] = 1;
                            pos++;
                        }
                    }
                }
                __syncthreads();
            }
            // the buffered hops out of the tile, their latencies overlapped
            {
                const int nx = min(s_nx, T);
                for (int x = tid; x < nx; x += nt) {
                    const int c = xc[x], nd = xd[x];
                    if (atomicMin(&ld[c], nd) > nd) {
                        atomicMin(&pend[c / T], nd);
                        atomicMin(gnext, nd);
                    }
                }
            }
            // write back; no cell beyond the window has been relaxed yet, so
            // the smallest such distance is the tile's pending minimum
            int pmin = INF;
            for (int i = tid; i < len; i += nt) {
                const int d = ds[i];
                if (d < ((volatile int*)ld)[base + i]) atomicMin(&ld[base + i], d);
                if (d > hi && d < pmin) pmin = d;
            }
            pmin = __reduce_min_sync(0xffffffffu, pmin);
            if ((tid & 31) == 0 && pmin != INF) atomicMin(&s_pmin, pmin);
            __syncthreads();
            if (tid == 0 && s_pmin != INF) {
                atomicMin(&pend[t], s_pmin);
                atomicMin(gnext, s_pmin);
            }
        }
        grid.sync();
        // the same in every block: written before the barrier, cleared two rounds later
        const int g = ((volatile int*)gmin)[(r + 1) % 3];
        if (g == INF) break;
        if (g > hi) {
            lo = g;
            hi = g + window - 1;
        }
        if (r > 4 * M + 8) break;   // cannot happen: every round settles a pending cell or moves the window
    }
    int dmax = 0;
    for (unsigned i = gtid; i < (unsigned)M; i += gsz) {
        const int d = ld[i];
        if (d == INF) ld[i] = -1;
        else dmax = d > dmax ? d : dmax;
    }
    dmax = __reduce_max_sync(0xffffffffu, dmax);
    if ((tid & 31) == 0 && dmax > 0) atomicMax(depth_out, dmax);
    if (gtid == 0) *rounds_out = rounds;
}

// Minimax levels of the basin graph by contraction, in one cooperative launch.
// All paths of a component without a seed leave it over its lowest outgoing
// edge W or a higher one, and its members reach one another below the height
// of any edge they leave by, so every member's level is max(level, W), and the
// component joins the neighbour over one edge of height W (Boruvka's steps); a
// component that contains a seed (-1) is finished.  One edge, whichever of
// equal ones claims the component first: over two of them it could join the
// seed and a neighbour that reaches the seed only higher up.  A round at least
// halves the components, whatever the length of the chains of basins, and
// takes two grid barriers:
//   every basin notes its component, every live edge the components of its
//   ends (in place: they only coarsen) and lowers W of the first one;
//   levels are raised to W, and an edge at W joins its components.
// W is double-buffered, a component clears the other buffer's entry.  It asks
// for every edge to be listed from both its ends.  Latency bounds it: five or six rounds
// of 10 to 20 us, 87, 110 and 120 us on a plane of 20,000 and 161,000 vertices
// and a sphere of 2.6 million.  Relaxing the edges until nothing changes
// (k_relax_active, after a table of the basin pairs) took 103, 250 and 140 us.
__device__ __forceinline__ int bg_root(const int* comp, int x) {
    for (int it = 0; it < 1 << 20; it++) {
        const int p = ld_relaxed_s32(comp + x);
        if (p == x || p < 0) return p;
        x = p;
    }
    return x;
}

__global__ void __launch_bounds__(1024, 1) k_basin_levels(const int* __restrict__ m_count, int64_t cap,
                                                         const int* __restrict__ nbasin,
                                                         const int* __restrict__ basin, int* comp, int* old,
                                                         int* claim, int* xu,
                                                         int* xv, const unsigned long long* __restrict__ xw,
                                                         unsigned long long* W0, unsigned long long* W1,
                                                         unsigned long long* L, int* flags, int* rounds_out) {
    cg::grid_group grid = cg::this_grid();
    const int64_t mc = *m_count;
    const int m = (int)(mc < cap ? mc : cap), nb = *nbasin;
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gsz = gridDim.x * blockDim.x;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned long long *W = W0, *Wn = W1;
    int r = 0;
    // the first round starts with every basin its own component and W known
    for (int i = gtid; i < nb; i += gsz) {
        const int b = basin[i];
        old[b] = b;
        W1[b] = ~0ULL;
    }
    for (;; r++) {
        bool live = false;
        if (r > 0) {
            for (int i = gtid; i < nb; i += gsz) {
                const int b = basin[i];
                const int c = bg_root(comp, b);
                old[b] = c;
                if (c != b) asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(comp + b), "r"(c) : "memory");
                else Wn[b] = ~0ULL;
            }
            for (int e0 = gtid - lane; e0 < m; e0 += gsz) {
                const int e = e0 + lane;
                const int u = e < m ? xu[e] : -1;
                int cu = -1;
                unsigned long long w = ~0ULL;
                if (u >= 0) {
                    const int v = xv[e];
                    w = xw[e];
                    cu = u;
                    int cv = v;
                    for (int it = 0; it < 1 << 20; it++) {      // both ends' roots, step by step together
                        const int pu = ld_relaxed_s32(comp + cu), pv = cv < 0 ? -1 : ld_relaxed_s32(comp + cv);
                        if (pu == cu && pv == cv) break;
                        cu = pu;
                        cv = pv;
                        if (cu < 0) break;
                    }
                    if (cu == cv) cu = -1;
                    xu[e] = cu;
                    xv[e] = cv;
                }
                live |= cu >= 0;
                // late rounds have few components: one atomic per warp and component
                const unsigned same = __match_any_sync(full, cu);
                const unsigned hi = __reduce_min_sync(same, (unsigned)(w >> 32));
                const unsigned lo = __reduce_min_sync(same, (unsigned)(w >> 32) == hi ? (unsigned)w : ~0u);
                if (cu >= 0 && lane == __ffs(same) - 1) {
                    const unsigned long long low = (unsigned long long)hi << 32 | lo;
                    if (low < __ldcg(W + cu)) atomicMin(W + cu, low);
                }
            }
            if (__any_sync(0xffffffffu, live) && (threadIdx.x & 31) == 0) flags[r & 1] = 1;
            grid.sync();
            if (!*(volatile int*)&flags[r & 1]) break;
        }
        if (gtid == 0) flags[(r + 1) & 1] = 0;   // read for the last time before the last barrier but one
        for (int i = gtid; i < nb; i += gsz) {
            const int b = basin[i];
            const int c = old[b];
            if (c < 0) continue;
            const unsigned long long w = __ldcg(W + c);
            if (w != ~0ULL && w > L[b]) L[b] = w;
        }
        for (int e = gtid; e < m; e += gsz) {
            const int u = xu[e];
            if (u < 0 || xw[e] != __ldcg(W + u) || atomicMax(claim + u, r + 1) == r + 1) continue;
            const int v = xv[e];
            for (int it = 0; it < 1 << 20; it++) {
                int a = bg_root(comp, u), b = v < 0 ? -1 : bg_root(comp, v);
                if (a == b) break;
                if (a < b) { const int t = a; a = b; b = t; }
                if (atomicCAS(comp + a, a, b) == a) break;
            }
        }
        grid.sync();
        unsigned long long* t = W;
        W = Wn;
        Wn = t;
    }
    // a basin that no seed is reached from keeps no level
    for (int i = gtid; i < nb; i += gsz)
        if (old[basin[i]] >= 0) L[basin[i]] = ~0ULL;
    if (gtid == 0) *rounds_out = r;
}

// Minimax relaxation over the basin graph in one cooperative launch:
// L[u] = min(L[u], max(w, L[v])) over the edges v -> u until nothing
// changes.  A thread keeps its first RELAX_REG edges (u, v, weight and the
// level of v it last used) in registers for the whole launch, and between two
// grid barriers relaxes them RELAX_SUB times, each time only when the level
// of v changed since it last relaxed that edge: a lowered level travels along
// a chain of basins within one round instead of one basin per round.  Edges
// beyond the registers are relaxed once per round.  A round ends with a grid
// barrier and continues while any level changed in it (three rotating change
// flags: round r sets flags[r % 3], reads it after the barrier and clears
// flags[(r + 1) % 3]).  Levels only decrease and a round without any change
// used only final levels, so the result is the fixed point of the all-edges
// relaxation whatever the order of the updates.  For meshes with edges that
// only one of their ends lists.
constexpr int RELAX_REG = 2;
constexpr int RELAX_SUB = 8;

__global__ void __launch_bounds__(256) k_relax_active(const int* __restrict__ m_count, int64_t cap,
                                                      const int* __restrict__ xu, const int* __restrict__ xv,
                                                      const unsigned long long* __restrict__ xw,
                                                      unsigned long long* L, int* flags, int max_rounds,
                                                      int* rounds_out) {
    cg::grid_group grid = cg::this_grid();
    // the edge count as k_cross_edges left it (its appends stop at the capacity)
    const int64_t mc = *m_count;
    const int m = (int)(mc < cap ? mc : cap);
    const int gtid = blockIdx.x * blockDim.x + threadIdx.x, gsz = gridDim.x * blockDim.x;
    int cu[RELAX_REG], cv[RELAX_REG];
    unsigned long long cw[RELAX_REG], last[RELAX_REG];
#pragma unroll
    for (int q = 0; q < RELAX_REG; q++) {
        const int e = gtid + q * gsz;
        cv[q] = -1;
        cu[q] = 0;
        cw[q] = 0ULL;
        last[q] = ~0ULL;
        if (e < m) {
            cu[q] = xu[e];
            cv[q] = xv[e];
            cw[q] = xw[e];
        }
    }
    volatile unsigned long long* VL = L;
    int r = 1;
    for (; r <= max_rounds; r++) {
        int changed = 0;
        for (int sub = 0; sub < RELAX_SUB; sub++) {
            unsigned long long lv[RELAX_REG];
#pragma unroll
            for (int q = 0; q < RELAX_REG; q++) lv[q] = cv[q] >= 0 ? VL[cv[q]] : ~0ULL;
#pragma unroll
            for (int q = 0; q < RELAX_REG; q++) {
                if (lv[q] == ~0ULL || lv[q] == last[q]) continue;
                last[q] = lv[q];
                const unsigned long long cand = cw[q] > lv[q] ? cw[q] : lv[q];
                if (cand < atomicMin(&L[cu[q]], cand)) changed = 1;
            }
        }
        for (int e = gtid + RELAX_REG * gsz; e < m; e += gsz) {
            const unsigned long long lv = VL[xv[e]];
            if (lv == ~0ULL) continue;
            const unsigned long long w = xw[e];
            const unsigned long long cand = w > lv ? w : lv;
            const int u = xu[e];
            if (cand < VL[u] && cand < atomicMin(&L[u], cand)) changed = 1;
        }
        if (__any_sync(0xffffffffu, changed) && (threadIdx.x & 31) == 0) flags[r % 3] = 1;
        // clear the flag of the next round: its last readers (end of round
        // r - 2) have all passed the barrier of round r - 1.  The flag of
        // round r - 1 may still be unread by slow threads.
        if (gtid == 0) flags[(r + 1) % 3] = 0;
        grid.sync();
        if (!*(volatile int*)&flags[r % 3]) break;
    }
    if (gtid == 0) *rounds_out = r;
}

// ---- flat distances, one depression at a time -----------------------------
// The breadth-first search of a depression stays inside it (all its cells
// have one fill level): its sources are its own spill cells (distance 1) and
// the cells next to a spill node outside it (distance 2).  So every
// depression is searched by itself, all of them at once, and the time is that
// of the deepest lake alone: a warp for up to 32 cells, a block for more, with
// the visited set and the frontiers in shared memory and a level bound by its
// chain (adjacency row from L2, claim, append, barrier: about 0.8 us, against
// 2.5 us in one block over all depressions, whose wide early levels keep the
// block busy; a 160,000-vertex landscape with 4,411 depressions, the largest
// of 15,872 cells and 341 levels: 841 -> 275 us; a 20,000-vertex one with 99
// levels: 223 -> 77 us).
//
// A lake can also be entered from a lower lake that touches it, through a rim
// cell other than its spill cell (it takes two rim cells at exactly the same
// level).  k_flat_small and k_flat_rows list such cells, and k_flat_fix lowers
// the distances that shorten through them until none does: the fixed point of
// all edges, which is the search over all depressions.  A depression whose
// visited set does not fit shared memory (FLAT_MAX cells) makes that search run
// instead, and so does a mesh with edges that only one of their ends lists.
constexpr int FLAT_MAX = 1 << 20;   // 128 KB of visited bits
constexpr int FLAT_CAP = 4096;      // frontier entries in shared memory; the rest in global memory
enum { FL_BIG = 0, FL_MID = 1, FL_TICKET = 2, FL_RIM = 3, FL_ALL = 4, FL_DEPTH = 5, FL_NCTL = 8 };

__global__ void k_flat_inv(int m, const int* __restrict__ cells, int* inv) {
    int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q < m) inv[cells[q]] = q;
}

// sources of a cell v of depression p: its first distance (0: none), and
// whether it is a rim cell that a lower depression could enter by
__device__ __forceinline__ int flat_source(int v, int p, int n, const double* f, const int* pit, const int* nbr,
                                           const int8_t* nnb, const int* spill_flag, const int* bestlid,
                                           const int* inv, int start, int W, unsigned* adj, unsigned* row,
                                           bool* rim) {
    const double fv = f[v];
    const int deg = nnb[v];
    int d = spill_flag[v] ? 1 : 0;
    for (int s = 0; s < W; s++) {
        if (row) row[s] = ~0u;
        if (s >= deg) continue;
        const int c = nbr[(size_t)s * n + v];
        if (c < 0) continue;
        const int pc = pit[c];
        if (pc == p) {
            const int l = inv[c] - start;
            if (adj) *adj |= 1u << l;
            if (row) row[s] = (unsigned)l;
        } else {
            const double fc = f[c];
            if (spill_flag[c] && fv >= fc && d == 0) d = 2;
            if (pc >= 0 && fc < fv && v != bestlid[p]) *rim = true;
        }
    }
    return d;
}

// a warp per depression of up to 32 cells; larger ones are listed for
// k_flat_big: more than 2048 cells from the front, the others from the back
__global__ void __launch_bounds__(256) k_flat_small(int np1, int n, int W, const double* __restrict__ f,
                                                    const int* __restrict__ pit, const int* __restrict__ nbr,
                                                    const int8_t* __restrict__ nnb,
                                                    const int* __restrict__ spill_flag,
                                                    const int* __restrict__ bestlid, const int* __restrict__ start,
                                                    const int* __restrict__ counts, const int* __restrict__ cells,
                                                    const int* __restrict__ inv, int* pdir, int* list, int* rims, int* ctl) {
    const int p = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    if (p >= np1) return;
    const int cnt = counts[p], s0 = start[p];
    if (cnt == 0) return;
    if (cnt > 32) {
        if (lane == 0) {
            if (cnt > FLAT_MAX) ctl[FL_ALL] = 1;
            else if (cnt > 2048) list[atomicAdd(&ctl[FL_BIG], 1)] = p;
            else list[n - 1 - atomicAdd(&ctl[FL_MID], 1)] = p;
        }
        return;
    }
    unsigned adj = 0u;
    bool rim = false;
    int d = 0, v = -1;
    if (lane < cnt) {
        v = cells[s0 + lane];
        d = flat_source(v, p, n, f, pit, nbr, nnb, spill_flag, bestlid, inv, s0, W, &adj, nullptr, &rim);
    }
    const unsigned two = __ballot_sync(full, d == 2);
    unsigned front = __ballot_sync(full, d == 1), seen = front | two;
    for (int level = 1; front || (level == 1 && two); level++) {
        const bool now = lane < cnt && !((seen >> lane) & 1u) && (adj & front);
        if (now) d = level + 1;
        front = __ballot_sync(full, now) | (level == 1 ? two : 0u);
        seen |= front;
    }
    if (v >= 0 && d > 0) pdir[v] = d;
    if (rim) rims[atomicAdd(&ctl[FL_RIM], 1)] = v;
}

// adjacency rows (G local ids, ~0: none) and first distances of the cells of the
// larger depressions
template <int G>
__global__ void __launch_bounds__(256) k_flat_rows(int m, int n, const double* __restrict__ f,
                                                   const int* __restrict__ pit, const int* __restrict__ nbr,
                                                   const int8_t* __restrict__ nnb,
                                                   const int* __restrict__ spill_flag,
                                                   const int* __restrict__ bestlid, const int* __restrict__ start,
                                                   const int* __restrict__ counts, const int* __restrict__ keys,
                                                   const int* __restrict__ cells, const int* __restrict__ inv,
                                                   unsigned* rows, int* dist, int* rims, int* ctl) {
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= m) return;
    const int p = keys[q], cnt = counts[p];
    if (cnt <= 32 || cnt > FLAT_MAX) return;
    unsigned row[G];
    bool rim = false;
    const int v = cells[q];
    dist[q] = flat_source(v, p, n, f, pit, nbr, nnb, spill_flag, bestlid, inv, start[p], G, nullptr, row, &rim);
    uint4* out = (uint4*)(rows + (size_t)q * G);
#pragma unroll
    for (int g = 0; g < G / 4; g++)
        out[g] = make_uint4(row[4 * g], row[4 * g + 1], row[4 * g + 2], row[4 * g + 3]);
    if (rim) rims[atomicAdd(&ctl[FL_RIM], 1)] = v;
}

// a block per listed depression, the large ones first; G lanes expand one
// frontier cell, so that a claim is one shared-memory atomic per lane and the
// claimed cells are appended by one ballot
template <int G, int T>
__global__ void __launch_bounds__(T) k_flat_big(int n, const int* __restrict__ start,
                                                     const int* __restrict__ counts, const int* __restrict__ cells,
                                                     const unsigned* __restrict__ rows,
                                                     int* dist, const int* __restrict__ list, int* gA,
                                                     int* gB, int* pdir, int* ctl) {
    extern __shared__ unsigned seen[];   // a bit per cell of the largest depression
    __shared__ int fA[FLAT_CAP], fB[FLAT_CAP];
    __shared__ int s_cnt[3], s_item;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const unsigned full = 0xffffffffu;
    const int nbig = ctl[FL_BIG], nmid = ctl[FL_MID];
    for (;;) {
        if (tid == 0) s_item = atomicAdd(&ctl[FL_TICKET], 1);
        __syncthreads();
        const int item = s_item;
        if (item >= nbig + nmid) return;
        const int p = item < nbig ? list[item] : list[n - 1 - (item - nbig)];
        const int cnt = counts[p], s0 = start[p];
        for (int w = tid; w < (cnt + 31) / 32; w += T) seen[w] = 0u;
        if (tid < 3) s_cnt[tid] = 0;
        __syncthreads();
        // level 1: the cells at distance 1; those at distance 2 start the next frontier
        for (int k = tid; k < cnt; k += T) {
            const int d = dist[s0 + k];
            if (d == 0) continue;
            atomicOr(&seen[k >> 5], 1u << (k & 31));
            const int at = atomicAdd(&s_cnt[d - 1], 1);
            if (at < FLAT_CAP) (d == 1 ? fA : fB)[at] = k;
            else (d == 1 ? gA : gB)[s0 + at] = k;
        }
        __syncthreads();
        int* curS = fA;
        int* nxtS = fB;
        int* curG = gA;
        int* nxtG = gB;
        int size = s_cnt[0], r = 0, d = 1;
        for (;; r++, d++) {
            int* next = &s_cnt[(r + 1) % 3];
            if (tid == 0) s_cnt[(r + 2) % 3] = 0;   // last read before the barrier that ended the previous level
            constexpr int CW = 32 / G;               // frontier cells a warp expands at once
            for (int base = warp * CW; base < size; base += (T / 32) * CW) {
                const int t = base + lane / G;
                unsigned e = ~0u;
                if (t < size) {
                    const int k = t < FLAT_CAP ? curS[t] : curG[s0 + t];
                    e = rows[(size_t)(s0 + k) * G + lane % G];
                }
                bool got = false;
                if (e != ~0u && !((((volatile unsigned*)seen)[e >> 5] >> (e & 31u)) & 1u))
                    got = !((atomicOr(&seen[e >> 5], 1u << (e & 31u)) >> (e & 31u)) & 1u);
                const unsigned won = __ballot_sync(full, got);
                if (won) {
                    int at = 0;
                    if (lane == 0) at = atomicAdd(next, __popc(won));
                    at = __shfl_sync(full, at, 0) + __popc(won & ((1u << lane) - 1u));
                    if (got) {
                        if (at < FLAT_CAP) nxtS[at] = (int)e;
                        else nxtG[s0 + at] = (int)e;
                        dist[s0 + e] = d + 1;
                        asm volatile("prefetch.global.L1 [%0];" ::"l"(rows + (size_t)(s0 + e) * G));
                    }
                }
            }
            __syncthreads();
            size = *next;
            if (size == 0) break;
            int* ts = curS; curS = nxtS; nxtS = ts;
            int* tg = curG; curG = nxtG; nxtG = tg;
        }
        for (int k = tid; k < cnt; k += T) {
            const int v = dist[s0 + k];
            if (v > 0) pdir[cells[s0 + k]] = v;
        }
        __syncthreads();
    }
}

// Distances that shorten through the listed rim cells, lowered until none is
// left (one block: few cells, mostly none).  An unreached cell's -1 is the
// largest unsigned distance.  Sixteen lanes look at one cell's neighbours, so
// that a round is one chain of loads (cell, neighbour id, its level and
// distance, atomicMin).  A cell may be listed more than once; lists that
// outgrow their buffers hand over to the search over all depressions.
__global__ void __launch_bounds__(1024) k_flat_fix(int n, const double* __restrict__ f, const int* __restrict__ pit,
                                                   const int* __restrict__ nbr, const int8_t* __restrict__ nnb,
                                                   const int* __restrict__ rims, int* gA, int* gB, int* pdir,
                                                   int* ctl) {
    constexpr int CAP = 2048;
    __shared__ int sA[CAP], sB[CAP];
    __shared__ int s_cnt[3];
    const int tid = threadIdx.x, sub = tid & 15, nrim = ctl[FL_RIM];
    if (nrim == 0 || ctl[FL_ALL]) return;
    if (tid < 3) s_cnt[tid] = 0;
    __syncthreads();
    volatile unsigned* vd = (volatile unsigned*)pdir;
    auto lower = [&](int c, unsigned d, int* next, int* outS, int* outG) {
        if (atomicMin((unsigned*)&pdir[c], d) <= d) return;
        const int at = atomicAdd(next, 1);
        if (at < CAP) outS[at] = c;
        else if (at < n) outG[at] = c;
    };
    for (int t = tid >> 4; t < nrim; t += 64) {
        const int v = rims[t];
        const int c = sub < nnb[v] ? nbr[(size_t)sub * n + v] : -1;
        if (c < 0) continue;
        const unsigned dc = vd[c], dv = vd[v];
        if (pit[c] >= 0 && f[c] < f[v] && (int)dc > 0 && dc + 1u < dv) lower(v, dc + 1u, &s_cnt[0], sA, gA);
    }
    __syncthreads();
    int* curS = sA;
    int* nxtS = sB;
    int* curG = gA;
    int* nxtG = gB;
    for (int r = 0;; r++) {
        const int size = s_cnt[r % 3];
        if (size > n) {
            if (tid == 0) ctl[FL_ALL] = 1;
            return;
        }
        if (size == 0) return;
        int* next = &s_cnt[(r + 1) % 3];
        if (tid == 0) s_cnt[(r + 2) % 3] = 0;
        for (int t = tid >> 4; t < size; t += 64) {
            const int v = t < CAP ? curS[t] : curG[t];
            const int c = sub < nnb[v] ? nbr[(size_t)sub * n + v] : -1;
            if (c < 0) continue;
            const unsigned d = vd[v] + 1u, dc = vd[c];
            const int pc = pit[c];
            const double fv = f[v], fc = f[c];
            if (dc > d && pc >= 0 && fc >= fv) lower(c, d, next, nxtS, nxtG);
        }
        __syncthreads();
        int* t = curS; curS = nxtS; nxtS = t;
        t = curG; curG = nxtG; nxtG = t;
    }
}

__global__ void k_flat_dirs(int n, const double* __restrict__ f, const int* __restrict__ pit,
                            const int* __restrict__ pdir, const int* __restrict__ nbr,
                            const int8_t* __restrict__ nnb, const int* __restrict__ spill_flag,
                            double sl, const double* __restrict__ h, int* flat, double* lfill,
                            const int* __restrict__ skip, int* depth) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (skip && *skip) return;
    if (depth) {   // the deepest distance
        const int deep = __reduce_max_sync(0xffffffffu, i < n ? pdir[i] : -1);
        if ((threadIdx.x & 31) == 0 && deep > *(volatile int*)depth) atomicMax(depth, deep);
    }
    if (i >= n) return;
    int out = -1;
    if (pit[i] > -1) {
        const int pi = pdir[i];
        const double fi = f[i];
        int bd = INT_MAX, bj = INT_MAX;
        for (int s = 0; s < nnb[i]; s++) {
            int c = nbr[(size_t)s * n + i];
            if (c < 0) continue;
            int pc = pdir[c];
            if (pc > -1 && pc < pi && f[c] <= fi) {
                if (pc < bd || (pc == bd && c < bj)) { bd = pc; bj = c; }
            }
        }
        out = (bj != INT_MAX) ? bj : i;
    }
    if (spill_flag[i]) out = -1;
    if (f[i] <= sl) {          // open sea: unfilled, no flat routing (pitfilling.py:822-825)
        out = -1;
        lfill[i] = h[i];
    }
    flat[i] = out;
}

// --------------------------------------------------------------------------
// pit tables
// --------------------------------------------------------------------------
// pit cells in id order, and the sizes and checks that the host waits for
__global__ void k_pit_compact(int n, const int* __restrict__ flag, const int* __restrict__ pos,
                              const int* __restrict__ pit, const int* __restrict__ isc, int* keys, int* vals,
                              int* out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (i == n - 1) {
        out[F_ROUNDS] = isc[I_ROUNDS];
        out[F_EDGES] = isc[I_NEXT];
        out[F_PITS] = vals[n] + keys[n];   // labels in use: their scan and flags, not yet overwritten there
        out[F_NONFINITE] = isc[I_NONFINITE];
        out[F_CELLS] = pos[i] + flag[i];
    }
    if (!flag[i]) return;
    keys[pos[i]] = pit[i];
    vals[pos[i]] = i;
}

// Block-per-pit reductions in a fixed order (deterministic): strided partial
// sums per thread, then a fixed shared-memory tree.  A thread visits its
// cells t = lane, lane + 256, ... in order; the cells of PIT_UNROLL visits and
// their values are loaded before any is added, so that the gathers of a large
// pit overlap, and the additions keep the visiting order.
constexpr int PIT_UNROLL = 8;

template <int NV>
__device__ __forceinline__ void block_reduce(double (&v)[NV], bool is_max[NV]) {
    __shared__ double sh[NV][256];
    for (int q = 0; q < NV; q++) sh[q][threadIdx.x] = v[q];
    __syncthreads();
    for (int s = 128; s > 0; s >>= 1) {
        if (threadIdx.x < s)
            for (int q = 0; q < NV; q++)
                sh[q][threadIdx.x] = is_max[q] ? fmax(sh[q][threadIdx.x], sh[q][threadIdx.x + s])
                                               : sh[q][threadIdx.x] + sh[q][threadIdx.x + s];
        __syncthreads();
    }
    for (int q = 0; q < NV; q++) v[q] = sh[q][0];
}

// Per-pit reductions over chunks: a pit's cells (sorted by id, segments of
// seg_vals2) are cut into chunks of PIT_CHUNK = 256 * PIT_UNROLL cells, one
// block per chunk, so that a lake of tens of thousands of cells spreads over
// many blocks instead of holding one block while the others have finished.
// Within a chunk thread `lane` adds its cells lane, lane + 256, ... in order
// and the block tree combines the threads; a finishing pass adds a pit's chunk
// partials in chunk order.  A pit of one chunk therefore sums exactly as a
// block over the whole pit did.
constexpr int PIT_CHUNK = 256 * PIT_UNROLL;

__global__ void k_pit_nchunk(int np1, const int* __restrict__ counts, int* nch) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < np1) nch[p] = (counts[p] + PIT_CHUNK - 1) / PIT_CHUNK;
}

// item -> pit (items of pit p: chs[p] .. chs[p] + nch[p] - 1)
__global__ void k_pit_items(int np1, const int* __restrict__ nch, const int* __restrict__ chs, int* item_pit) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np1) return;
    const int c0 = chs[p], k = nch[p];
    for (int c = 0; c < k; c++) item_pit[c0 + c] = p;
}

// the item of this block: its pit, first cell and cell count; false past the last item
__device__ __forceinline__ bool pit_item(int np1, const int* __restrict__ nch, const int* __restrict__ chs,
                                         const int* __restrict__ item_pit, const int* __restrict__ start,
                                         const int* __restrict__ counts, int* p, int* s0, int* c) {
    const int i = blockIdx.x;
    if (i >= chs[np1 - 1] + nch[np1 - 1]) return false;
    const int q = item_pit[i];
    const int k = i - chs[q];
    *p = q;
    *s0 = start[q] + k * PIT_CHUNK;
    const int rest = counts[q] - k * PIT_CHUNK;
    *c = rest < PIT_CHUNK ? rest : PIT_CHUNK;
    return true;
}

// chunk partials of vol, max fill, max depth (cells sorted by id)
__global__ void __launch_bounds__(256) k_pit_params(int np1, const int* __restrict__ nch, const int* __restrict__ chs,
                                                    const int* __restrict__ item_pit,
                                                    const int* __restrict__ start, const int* __restrict__ counts,
                                                    const int* __restrict__ cells, const double* __restrict__ f,
                                                    const double* __restrict__ h, double sl,
                                                    const double* __restrict__ larea, double* part) {
    int p, s0, c;
    if (!pit_item(np1, nch, chs, item_pit, start, counts, &p, &s0, &c)) return;
    const int lane = threadIdx.x;
    double v[3] = {0.0, -INFINITY, -INFINITY};
    int ii[PIT_UNROLL];
    double fi[PIT_UNROLL], hi[PIT_UNROLL], ai[PIT_UNROLL];
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++) ii[u] = lane + u * 256 < c ? cells[s0 + lane + u * 256] : -1;
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++) {
        if (ii[u] < 0) continue;
        fi[u] = f[ii[u]];
        hi[u] = h[ii[u]];
        ai[u] = larea[ii[u]];
    }
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++) {
        if (ii[u] < 0) continue;
        double hc = hi[u] < sl ? sl : hi[u];
        double d = fi[u] - hc;
        v[0] += d * ai[u];
        v[1] = fmax(v[1], fi[u]);
        v[2] = fmax(v[2], d);
    }
    bool mx[3] = {false, true, true};
    block_reduce<3>(v, mx);
    if (lane == 0)
        for (int q = 0; q < 3; q++) part[3 * (size_t)blockIdx.x + q] = v[q];
}

// pit params from the chunk partials, in chunk order
__global__ void k_pit_params_fin(int np1, const int* __restrict__ nch, const int* __restrict__ chs,
                                 const double* __restrict__ part, double* params) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np1) return;
    const int k = nch[p];
    if (k == 0) {
        params[3 * p] = 0.0;
        params[3 * p + 1] = -1.0e8;   // MISSING_DATA_SENTINEL (constants.py:34)
        params[3 * p + 2] = 0.0;
        return;
    }
    const size_t i0 = chs[p];
    double vol = part[3 * i0], hmax = part[3 * i0 + 1], dmax = part[3 * i0 + 2];
    for (int j = 1; j < k; j++) {
        vol = vol + part[3 * (i0 + j)];
        hmax = fmax(hmax, part[3 * (i0 + j) + 1]);
        dmax = fmax(dmax, part[3 * (i0 + j) + 2]);
    }
    params[3 * p] = vol;
    params[3 * p + 1] = hmax;
    params[3 * p + 2] = dmax;
}

__global__ void k_filled_lvl(int np1, const double* __restrict__ params, double* lvl) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np1) return;
    double d[6] = {0, 0, 0, 0, 0, 0};
    if (params[3 * p] > 0.0) {
        d[0] = params[3 * p + 1] - params[3 * p + 2];
        double st = params[3 * p + 2] / 5.0;
        for (int k = 1; k < 6; k++) d[k] = st;
    }
    double s = d[0];
    for (int k = 1; k < 6; k++) {
        s = s + d[k];
        lvl[5 * p + k - 1] = s;
    }
}

// chunk partials of the filled volumes at the four intermediate levels
__global__ void __launch_bounds__(256) k_filled_vol(int np1, const int* __restrict__ nch, const int* __restrict__ chs,
                                                    const int* __restrict__ item_pit,
                                                    const int* __restrict__ start, const int* __restrict__ counts,
                                                    const int* __restrict__ cells, const double* __restrict__ h,
                                                    double sl, const double* __restrict__ farea,
                                                    const double* __restrict__ lvl, double* part) {
    int p, s0, c;
    if (!pit_item(np1, nch, chs, item_pit, start, counts, &p, &s0, &c)) return;
    const int lane = threadIdx.x;
    const double l0 = lvl[5 * p], l1 = lvl[5 * p + 1], l2 = lvl[5 * p + 2], l3 = lvl[5 * p + 3];
    double v[4] = {0, 0, 0, 0};
    int ii[PIT_UNROLL];
    double hi[PIT_UNROLL], ai[PIT_UNROLL];
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++) ii[u] = lane + u * 256 < c ? cells[s0 + lane + u * 256] : -1;
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++) {
        if (ii[u] < 0) continue;
        hi[u] = h[ii[u]];
        ai[u] = farea[ii[u]];
    }
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++) {
        if (ii[u] < 0) continue;
        double e = hi[u] < sl ? sl : hi[u];
        double a = ai[u];
        if (l0 > e) v[0] += (l0 - e) * a;
        if (l1 > e) v[1] += (l1 - e) * a;
        if (l2 > e) v[2] += (l2 - e) * a;
        if (l3 > e) v[3] += (l3 - e) * a;
    }
    bool mx[4] = {false, false, false, false};
    block_reduce<4>(v, mx);
    if (lane == 0)
        for (int q = 0; q < 4; q++) part[4 * (size_t)blockIdx.x + q] = v[q];
}

__global__ void k_filled_vol_fin(int np1, const int* __restrict__ nch, const int* __restrict__ chs,
                                 const double* __restrict__ part, const double* __restrict__ params, double* vol) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np1) return;
    const int k = nch[p];
    double v[4] = {0, 0, 0, 0};
    if (k > 0) {
        const size_t i0 = chs[p];
        for (int q = 0; q < 4; q++) v[q] = part[4 * i0 + q];
        for (int j = 1; j < k; j++)
            for (int q = 0; q < 4; q++) v[q] = v[q] + part[4 * (i0 + j) + q];
    }
    for (int q = 0; q < 4; q++) vol[5 * p + q] = v[q];
    vol[5 * p + 4] = params[3 * p];
}

// per-pit masked sum: chunk partials, then a pit's partials in chunk order
__global__ void __launch_bounds__(256) k_pit_masked_sum(int np1, const int* __restrict__ nch,
                                                        const int* __restrict__ chs,
                                                        const int* __restrict__ item_pit,
                                                        const int* __restrict__ start,
                                                        const int* __restrict__ counts,
                                                        const int* __restrict__ cells,
                                                        const uint8_t* __restrict__ mask,
                                                        const double* __restrict__ vals, double* part) {
    int p, s0, c;
    if (!pit_item(np1, nch, chs, item_pit, start, counts, &p, &s0, &c)) return;
    const int lane = threadIdx.x;
    double v[1] = {0.0};
    int ii[PIT_UNROLL];
    uint8_t mi[PIT_UNROLL];
    double xi[PIT_UNROLL];
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++) ii[u] = lane + u * 256 < c ? cells[s0 + lane + u * 256] : -1;
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++) {
        mi[u] = 0;
        if (ii[u] < 0) continue;
        mi[u] = mask[ii[u]];
        xi[u] = vals[ii[u]];
    }
#pragma unroll
    for (int u = 0; u < PIT_UNROLL; u++)
        if (mi[u]) v[0] += xi[u];
    bool mx[1] = {false};
    block_reduce<1>(v, mx);
    if (lane == 0) part[blockIdx.x] = v[0];
}

__global__ void k_pit_masked_fin(int np1, const int* __restrict__ nch, const int* __restrict__ chs,
                                 const double* __restrict__ part, double* out) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np1) return;
    const int k = nch[p];
    double v = 0.0;
    if (k > 0) {
        const int i0 = chs[p];
        v = part[i0];
        for (int j = 1; j < k; j++) v = v + part[i0 + j];
    }
    out[p] = v;
}

// --------------------------------------------------------------------------
// host driver
// --------------------------------------------------------------------------
static int launch_coop(gs_plan* p, const void* fn, int blocks, int threads, void** args) {
    cudaEvent_t stop = nullptr;
    if (p->profiling) prof_begin(p, fn, &stop);
    GS_CUDA(cudaLaunchCooperativeKernel(fn, blocks, threads, args, 0, p->stream));
    if (stop) cudaEventRecord(stop, p->stream);
    p->launches++;
    return GS_OK;
}

// Tiled flat-distance BFS (k_bfs_tiles) over the M compacted cells whose
// rows, seeds (front0, count in i_scalar[6]) and local ids k_bfs_local_build
// wrote; distances into ld (-1 unreached), depth into i_scalar[4].  Tiles of
// T cells with T * (S + 5) ints of shared memory (<= 112 KB), as many blocks
// as stay co-resident.
static int bfs_tiles(gs_plan* p, int M, int S, const int* rows, int* ld) {
    int T = 4096;
    while (T > 256 && (size_t)T * (S + 5) * sizeof(int) > BFT_SMEM) T >>= 1;
    const size_t smem = (size_t)T * (S + 5) * sizeof(int);
    int occ = 0;
    GS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_bfs_tiles, BFT_THREADS, smem));
    if (occ < 1) {
        set_error(GS_ECUDA, "flat BFS: tile kernel cannot be resident");
        return GS_ECUDA;
    }
    const int ntiles = (M + T - 1) / T;
    const int grid = std::max(1, std::min(ntiles, p->sm_count * occ));
    if (3 + ntiles > (int)p->n + 1) {
        set_error(GS_EINVAL, "flat BFS: tile marks exceed their buffer");
        return GS_EINVAL;
    }
    GS_CUDA(cudaMemsetAsync(p->i_scalar + 4, 0, sizeof(int), p->stream));
    int m = M, s = S, t = T;
    const int* seeds = p->front0;
    const int* nseed = p->i_scalar + 6;
    int* ctl = p->front1;
    int* depth = p->i_scalar + 4;
    int* rounds = p->i_scalar + 15;
    // the search over all depressions also comes here with the knob at 0, when
    // the visited set is too large for one block
    int window = p->bfs_window > 0 ? p->bfs_window : 64;
    void* args[] = {(void*)&m, (void*)&s, (void*)&t, (void*)&rows, (void*)&seeds, (void*)&nseed, (void*)&ld,
                    (void*)&ctl, (void*)&window, (void*)&depth, (void*)&rounds};
    cudaEvent_t stop = nullptr;
    if (p->profiling) prof_begin(p, (const void*)k_bfs_tiles, &stop);
    GS_CUDA(cudaLaunchCooperativeKernel((const void*)k_bfs_tiles, grid, BFT_THREADS, args, smem, p->stream));
    if (stop) cudaEventRecord(stop, p->stream);
    p->launches++;
    GS_LAUNCH();
    return GS_OK;
}

static int exclusive_scan(gs_plan* p, const int* in, int* out, int count) {
    size_t bytes = p->cub_bytes;
    GS_CUDA(cub::DeviceScan::ExclusiveSum(p->cub_tmp, bytes, in, out, count, p->stream));
    p->launches++;
    return GS_OK;
}

// chunk items of the pit segments (after seg_count and seg_start): at most
// np1 + ncell / PIT_CHUNK of them, the grid of the chunk kernels
static int pit_chunks(gs_plan* p, int np1, int ncell) {
    const int B = 256;
    const int64_t imax = (int64_t)np1 + ncell / PIT_CHUNK + 1;
    if (imax > INT_MAX) {
        set_error(GS_ENOMEM, "pit tables: too many chunk items");
        return GS_ENOMEM;
    }
    if (!p->pit_nch) {
        GS_CUDA(cudaMalloc((void**)&p->pit_nch, sizeof(int) * ((size_t)p->n + 2)));
        GS_CUDA(cudaMalloc((void**)&p->pit_chs, sizeof(int) * ((size_t)p->n + 2)));
    }
    if (imax > p->pit_item_cap) {
        const int64_t cap = std::max<int64_t>(imax, 2 * p->pit_item_cap);
        if (p->pit_item) cudaFree(p->pit_item);
        if (p->pit_part) cudaFree(p->pit_part);
        p->pit_item = nullptr;
        p->pit_part = nullptr;
        p->pit_item_cap = 0;
        GS_CUDA(cudaMalloc((void**)&p->pit_item, sizeof(int) * (size_t)cap));
        GS_CUDA(cudaMalloc((void**)&p->pit_part, sizeof(double) * 4 * (size_t)cap));
        p->pit_item_cap = cap;
    }
    launch(p, k_pit_nchunk, grid_for(np1, B), B, np1, (const int*)p->seg_count, p->pit_nch);
    GS_LAUNCH();
    GS_TRY(exclusive_scan(p, p->pit_nch, p->pit_chs, np1));
    launch(p, k_pit_items, grid_for(np1, B), B, np1, (const int*)p->pit_nch, (const int*)p->pit_chs, p->pit_item);
    GS_LAUNCH();
    p->pit_items_max = (int)imax;
    return GS_OK;
}

int group_sum_by_pit(gs_plan* p, const int* /*pit_ids*/, const uint8_t* mask, const double* vals,
                     double* out, int npits) {
    const int np1 = npits + 1;
    launch(p, k_pit_masked_sum, p->pit_items_max, 256, np1, (const int*)p->pit_nch, (const int*)p->pit_chs,
           (const int*)p->pit_item, (const int*)p->seg_start, (const int*)p->seg_count, (const int*)p->seg_vals2,
           mask, vals, p->pit_part);
    launch(p, k_pit_masked_fin, grid_for(np1, 256), 256, np1, (const int*)p->pit_nch, (const int*)p->pit_chs,
           (const double*)p->pit_part, out);
    GS_LAUNCH();
    return GS_OK;
}

// The flat-distance search over all depressions at once: rows of the
// compacted reachable cells, one block (or tiles when the visited set does not
// fit, or by GS_TUNE_FLAT_BFS), distances into pdir, depth into i_scalar[4].
// M: number of compacted cells (flags and local ids in flagbuf / scanbuf).
static int flat_search_all(gs_plan* p, int M, const double* lfill, const int* pit_ids) {
    const int n = (int)p->n;
    const int B = 256, G = grid_for(n, B);
    // packed adjacency rows: [count, ids...], stride S ints (16-byte multiple)
    const int S = ((p->W + 1 + 3) / 4) * 4;
    int* rows = p->bfs_rows;
    int* ldv = p->lab;
    GS_CUDA(cudaMemsetAsync(p->i_scalar + 6, 0, sizeof(int), p->stream));
    launch(p, k_bfs_local_build, G, B, n, S, lfill, pit_ids, (const int*)p->flagbuf, (const int*)p->scanbuf,
           (const int*)p->nbr, (const int8_t*)p->nnb, (const int*)p->spill_flag, rows, p->comp, ldv, p->front0,
           p->i_scalar + 6);
    GS_LAUNCH();
    const size_t smem1 = sizeof(unsigned) * (size_t)((M + 31) / 32) + sizeof(int) * 2 * LBFS_CAP;
    if (p->bfs_window > 0 || smem1 > LBFS_SMEM) {
        GS_TRY(bfs_tiles(p, M, S, rows, ldv));
    } else {
        // one block: visited bitmap and frontiers in shared memory
        auto run = [&](auto kern) -> int {
            cudaEvent_t stop = nullptr;
            if (p->profiling) prof_begin(p, (const void*)kern, &stop);
            kern<<<1, 1024, smem1, p->stream>>>(M, S, (const int*)rows, (const int*)p->front0, p->i_scalar + 6,
                                                p->front1, p->minseed, ldv, p->i_scalar + 4);
            if (stop) cudaEventRecord(stop, p->stream);
            return GS_OK;
        };
        const int S4 = S / 4;
        if (S4 <= 1) GS_TRY(run(k_bfs_local<1>));
        else if (S4 == 2) GS_TRY(run(k_bfs_local<2>));
        else if (S4 == 3) GS_TRY(run(k_bfs_local<3>));
        else GS_TRY(run(k_bfs_local<4>));
        p->launches++;
        GS_LAUNCH();
    }
    launch(p, k_bfs_local_scatter, grid_for(M, B), B, M, (const int*)p->comp, (const int*)ldv, p->pdir);
    GS_LAUNCH();
    return GS_OK;
}

// flags of the cells the search can reach (pit cells, spill nodes) and their
// local ids
static int flat_compact(gs_plan* p, const int* pit_ids) {
    const int n = (int)p->n;
    launch(p, k_bfs_flag, grid_for(n, 256), 256, n, pit_ids, (const int*)p->spill_flag, p->flagbuf);
    GS_LAUNCH();
    return exclusive_scan(p, p->flagbuf, p->scanbuf, n);
}

static int flat_dirs_launch(gs_plan* p, const FlatArgs& a, const int* skip, int* depth) {
    const int n = (int)p->n;
    launch(p, k_flat_dirs, grid_for(n, 256), 256, n, (const double*)a.lfill, a.pit_ids, (const int*)p->pdir,
           (const int*)p->nbr, (const int8_t*)p->nnb, (const int*)p->spill_flag, a.sealevel, a.h, a.flat_dirs,
           a.lfill, skip, depth);
    GS_LAUNCH();
    return GS_OK;
}

// The flat pass by depressions (k_flat_*), on the current stream: m pit cells
// sorted by (pit, id) in seg_keys2 / seg_vals2 with seg_start / seg_count.
static int flat_search_pits(gs_plan* p, int m, const FlatArgs& a) {
    const int n = (int)p->n, np1 = p->npits + 1;
    const int B = 256;
    int* ctl = p->front1;
    int* inv = p->comp;
    unsigned* rows = (unsigned*)p->bfs_rows;   // at least G ids a vertex (plan creation)
    int* dist = p->lab;
    int* rims = p->scanbuf;
    GS_CUDA(cudaMemsetAsync(ctl, 0, sizeof(int) * FL_NCTL, p->stream));
    launch(p, k_flat_inv, grid_for(m, B), B, m, (const int*)p->seg_vals2, inv);
    launch(p, k_flat_small, grid_for((int64_t)np1 * 32, B), B, np1, n, p->W, (const double*)a.lfill, a.pit_ids,
           (const int*)p->nbr, (const int8_t*)p->nnb, (const int*)p->spill_flag, (const int*)p->bestlid,
           (const int*)p->seg_start, (const int*)p->seg_count, (const int*)p->seg_vals2, (const int*)inv, p->pdir,
           p->front0, rims, ctl);
    auto larger = [&](auto g) -> int {
        constexpr int G = decltype(g)::value;
        launch(p, k_flat_rows<G>, grid_for(m, B), B, m, n, (const double*)a.lfill, a.pit_ids, (const int*)p->nbr,
               (const int8_t*)p->nnb, (const int*)p->spill_flag, (const int*)p->bestlid, (const int*)p->seg_start,
               (const int*)p->seg_count, (const int*)p->seg_keys2, (const int*)p->seg_vals2, (const int*)inv, rows,
               dist, rims, ctl);
        // 1024 threads where a lake may be large: the widest levels of a
        // 15,872-cell lake gain (314 -> 275 us), small ones lose the barrier's
        // cost (77 -> 83 us at 9,186 pit cells)
        const bool wide = m > 32768;
        const int T = wide ? 1024 : 512, smem = (std::min(m, FLAT_MAX) + 31) / 32 * 4;
        auto kern = wide ? k_flat_big<G, 1024> : k_flat_big<G, 512>;
        cudaEvent_t stop = nullptr;
        if (p->profiling) prof_begin(p, (const void*)kern, &stop);
        kern<<<std::min(p->sm_count * 2, np1), T, smem, p->stream>>>(
            n, (const int*)p->seg_start, (const int*)p->seg_count, (const int*)p->seg_vals2, (const unsigned*)rows,
            dist, (const int*)p->front0, p->minseed, p->flagbuf, p->pdir, ctl);
        if (stop) cudaEventRecord(stop, p->stream);
        p->launches++;
        return GS_OK;
    };
    if (p->W <= 8) GS_TRY(larger(std::integral_constant<int, 8>{}));
    else GS_TRY(larger(std::integral_constant<int, 16>{}));
    launch(p, k_flat_fix, 1, 1024, n, (const double*)a.lfill, a.pit_ids, (const int*)p->nbr, (const int8_t*)p->nnb,
           (const int*)rims, p->minseed, p->flagbuf, p->pdir, ctl);
    GS_LAUNCH();
    GS_TRY(flat_dirs_launch(p, a, ctl + FL_ALL, ctl + FL_DEPTH));
    GS_CUDA(cudaMemcpyAsync(p->h_pinned + 2, ctl + FL_DEPTH, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
    GS_CUDA(cudaMemcpyAsync(p->h_pinned + 3, ctl + FL_ALL, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
    return GS_OK;
}

// The shared memory that the flat searches of a mesh of W slots may ask for.  The
// limit belongs to the kernel and the device, not to the plan, and plans of other
// threads launch meanwhile: it is set once per plan, always to the same value,
// and never lowered to what one launch needs.
int flat_limits(int W) {
    const auto limit = [](auto kern, int bytes) {
        return cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    };
    const int S4 = (W + 1 + 3) / 4, seen = FLAT_MAX / 8;
    GS_CUDA(limit(k_bfs_tiles, BFT_SMEM));
    if (S4 <= 1) GS_CUDA(limit(k_bfs_local<1>, LBFS_SMEM));
    else if (S4 == 2) GS_CUDA(limit(k_bfs_local<2>, LBFS_SMEM));
    else if (S4 == 3) GS_CUDA(limit(k_bfs_local<3>, LBFS_SMEM));
    else GS_CUDA(limit(k_bfs_local<4>, LBFS_SMEM));
    if (W <= 8) {
        GS_CUDA(limit(k_flat_big<8, 512>, seen));
        GS_CUDA(limit(k_flat_big<8, 1024>, seen));
    } else {
        GS_CUDA(limit(k_flat_big<16, 512>, seen));
        GS_CUDA(limit(k_flat_big<16, 1024>, seen));
    }
    return GS_OK;
}

__global__ void k_pdir_init(int n, const int* __restrict__ spill_flag, int* pdir) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) pdir[i] = spill_flag[i] ? 1 : -1;
}

int fill_join(gs_plan* p, gs_stats* st) {
    if (!p->bfs_pending) return GS_OK;
    const int by_pits = p->bfs_pending == 2;
    p->bfs_pending = 0;
    GS_CUDA(cudaStreamWaitEvent(p->stream, p->ev_b, 0));
    GS_CUDA(cudaEventSynchronize(p->ev_b));
    if (by_pits && p->h_pinned[3]) {
        // a depression with too many cells (or a k_flat_fix that outgrew its
        // lists): search over all of them, then the flat directions
        const FlatArgs a = p->flat_args;
        const int n = (int)p->n;
        launch(p, k_pdir_init, grid_for(n, 256), 256, n, (const int*)p->spill_flag, p->pdir);
        GS_LAUNCH();
        GS_TRY(flat_compact(p, a.pit_ids));
        int last[2];
        GS_CUDA(cudaMemcpyAsync(&last[0], p->scanbuf + n - 1, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
        GS_CUDA(cudaMemcpyAsync(&last[1], p->flagbuf + n - 1, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
        GS_CUDA(cudaStreamSynchronize(p->stream));
        GS_TRY(flat_search_all(p, last[0] + last[1], a.lfill, a.pit_ids));
        GS_TRY(flat_dirs_launch(p, a, nullptr, nullptr));
        GS_CUDA(cudaMemcpyAsync(p->h_pinned + 2, p->i_scalar + 4, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
        GS_CUDA(cudaStreamSynchronize(p->stream));
    }
    if (st) st->flat_rounds = p->h_pinned[2];
    p->pdir_bound = p->h_pinned[2] + 2;   // the deepest distance is the BFS depth
    return GS_OK;
}


int fill_elevation(gs_plan* p, const double* h, double sealevel, double ofill, double* lfill,
                   int* pit_ids, int* flat_dirs, gs_stats* st, bool defer_flats, uint8_t* sea_out, bool sed,
                   const double* check_b) {
    const int n = (int)p->n;
    if (p->bfs_pending) {   // left by a call that stopped on an error: only wait for it
        p->bfs_pending = 0;
        GS_CUDA(cudaStreamWaitEvent(p->stream, p->ev_b, 0));
    }
    if (n == 0) { p->npits = 0; return GS_OK; }
    const int B = 256, G = grid_for(n, B);
    // smallest height, level, and whether the inputs are finite: the host reads
    // that with the sizes, the kernels until then leave the outputs alone if not
    // (launches and host waits bound a fill of a small mesh: with a wait for the
    // check and the roots, one for the pits and one for their cells, and a kernel
    // or memset per array, a flow accumulation of 20,000 vertices took 790 us, now
    // 680)
    unsigned long long* word = p->u_scalar + U_LEVEL;
    int* out = (int*)(p->u_scalar + U_OUT);
    GS_CUDA(cudaMemsetAsync(word, 0xff, 3 * sizeof(unsigned long long), p->stream));
    launch(p, k_level, std::min(p->sm_count * 4, G), 256, n, h, check_b, word, p->flat ? 0 : 1, sealevel, ofill,
           sed ? 1 : 0, p->d_scalar, p->i_scalar);
    // Filling with sediment (pitfilling.py:557-702, 704-847 with sed=True):
    // open-sea depressions are filled too, pits are labelled above the fill
    // level instead of sea level, and pit volumes use the unclipped surface.
    const double clip_sl = sed ? -INFINITY : sealevel, marine_sl = sed ? -INFINITY : sealevel;
    const double* dsc = p->d_scalar;

    // seeds, descent links, roots; W lies in the diffusion's vectors, which no
    // fill runs beside
    unsigned long long *w0 = (unsigned long long*)p->cg_p, *w1 = (unsigned long long*)p->cg_ap;
    if (!p->mutual)
        launch(p, k_classify, G, B, n, h, dsc, (const int*)p->nbr, (const int8_t*)p->nnb, (const uint8_t*)p->outlet,
               p->ledge);
    launch(p, p->mutual ? k_descend<true> : k_descend<false>, G, B, n, p->mutual ? 0 : 1, h, dsc, (const int*)p->nbr,
           (const int8_t*)p->nnb, (const uint8_t*)p->outlet, p->ledge, p->parent, p->basinL, w0, p->comp, p->flagbuf,
           p->lab, p->i_scalar + I_BASINS);
    launch(p, k_jump, G, B, n, p->parent);
    // basin graph and minimax levels
    {
        // the counts stay on the device: the contraction reads them, and the
        // host checks the edges against the capacity with the sizes
        const int* mc = p->i_scalar + I_NEXT;
        const int* nbs = p->i_scalar + I_BASINS;
        int* flags = p->i_scalar + I_FLAGS;
        int* rout = p->i_scalar + I_ROUNDS;
        int64_t cap = std::min<int64_t>(p->xe_cap, INT_MAX);
        launch(p, k_cross_edges, G, B, n, h, (const double*)p->d_scalar, (const int*)p->nbr, (const int8_t*)p->nnb,
               (const int8_t*)p->ledge, (const int*)p->parent, w0, p->xe_u, p->xe_v, p->xe_w, p->i_scalar + I_NEXT,
               cap);
        GS_LAUNCH();
        if (p->mutual) {
            void* args[] = {(void*)&mc,      (void*)&cap,     (void*)&nbs, (void*)&p->lab, (void*)&p->comp,
                            (void*)&p->minseed, (void*)&p->flagbuf, (void*)&p->xe_u, (void*)&p->xe_v, (void*)&p->xe_w, (void*)&w0,
                            (void*)&w1,      (void*)&p->basinL, (void*)&flags, (void*)&rout};
            GS_TRY(launch_coop(p, (const void*)k_basin_levels, std::min(p->sm_count, grid_for(n, 1024)), 1024, args));
        } else {
            int maxr = 1000000;
            void* args[] = {(void*)&mc,      (void*)&cap,     (void*)&p->xe_u, (void*)&p->xe_v, (void*)&p->xe_w,
                            (void*)&p->basinL, (void*)&flags, (void*)&maxr,    (void*)&rout};
            GS_TRY(launch_coop(p, (const void*)k_relax_active, p->coop_blocks, 256, args));
        }
    }
    launch(p, k_fill_final, G, B, n, h, dsc, marine_sl, (const int8_t*)p->ledge, (const int*)p->parent,
           (const unsigned long long*)p->basinL, (const int*)p->i_scalar, lfill, p->minseed, p->seg_keys, p->bestlid,
           p->spill_flag, p->seg_count);
    GS_LAUNCH();

    // label_pits: equal-fill components of cells above the label level
    launch(p, k_uf_init, G, B, n, (const double*)lfill, dsc, (const int*)p->nbr, (const int8_t*)p->nnb, p->comp);
    launch(p, k_uf_link, G, B, n, (const double*)lfill, dsc, (const int*)p->nbr, (const int8_t*)p->nnb, p->comp);
    launch(p, k_minseed, G, B, n, (const double*)lfill, dsc, (const int*)p->nbr, (const int8_t*)p->nnb, p->comp,
           p->minseed);
    launch(p, k_seed_flag, G, B, n, (const double*)lfill, dsc, (const int*)p->comp, (const int*)p->minseed,
           p->flagbuf);
    GS_LAUNCH();
    GS_TRY(exclusive_scan(p, p->flagbuf, p->scanbuf, n));
    launch(p, k_label, G, B, n, (const double*)lfill, dsc, (const int*)p->comp, (const int*)p->minseed,
           (const int*)p->scanbuf, (const uint8_t*)p->outlet, p->lab, p->seg_keys);
    GS_LAUNCH();
    // consecutive ids over surviving labels (pits_cons); pit cells, compacted in
    // id order for the flat pass and the per-pit reductions
    GS_TRY(exclusive_scan(p, p->seg_keys, p->seg_vals, n + 1));
    launch(p, k_relabel, G, B, n, (const int*)p->lab, (const int*)p->seg_vals, (const int*)p->i_scalar,
           (const double*)lfill, sealevel, sea_out, pit_ids, p->pflag, p->seg_count, p->pdir);
    GS_LAUNCH();
    GS_TRY(exclusive_scan(p, p->pflag, p->pscan, n));
    launch(p, k_pit_compact, G, B, n, (const int*)p->pflag, (const int*)p->pscan, (const int*)pit_ids,
           (const int*)p->i_scalar, p->seg_keys, p->seg_vals, out);
    GS_LAUNCH();
    GS_CUDA(cudaMemcpyAsync(p->h_pinned + 6, out, sizeof(int) * F_COUNT, cudaMemcpyDeviceToHost, p->stream));
    GS_CUDA(cudaStreamSynchronize(p->stream));
    const int* res = p->h_pinned + 6;
    if (res[F_NONFINITE]) {
        set_error(GS_ENONFINITE, check_b ? "non-finite elevation or rain volume (NaN or Inf)"
                                         : "non-finite elevation (NaN or Inf)");
        return GS_ENONFINITE;
    }
    p->npits = res[F_PITS];
    const int ncell = res[F_CELLS];
    if ((int64_t)res[F_EDGES] > p->xe_cap) {
        set_error(GS_ENOMEM, "pit fill: cross-edge capacity exceeded");
        return GS_ENOMEM;
    }
    if (st) st->fill_rounds = res[F_ROUNDS];
    const int P = p->npits, np1 = P + 1;
    if (st) st->npits = P;

    // spill points
    launch(p, k_spill_qual, G, B, n, (const double*)lfill, (const int*)pit_ids, (const int*)p->nbr,
           (const int8_t*)p->nnb, (const uint8_t*)p->outlet, p->bestlid);
    launch(p, k_spill_pick, grid_for(np1, B), B, np1, n, (const double*)lfill, (const int*)pit_ids,
           (const int*)p->nbr, (const int8_t*)p->nnb, (const uint8_t*)p->outlet,
           (const int*)p->bestlid, p->pit_info, p->spill_flag, p->pdir);
    GS_LAUNCH();

    // flat distances (fill_dir + nghb_dir fixed point = BFS hop distance).
    // The search and the flat directions run on side_b, beside the pit tables
    // on the main stream: they share only read-only inputs, and the sea reset
    // of lFill in k_flat_dirs touches open-sea cells, which hold no pit.
    p->pdir_bound = 0;
    // GS_TUNE_FLAT_BFS > 0 asks for the search over all depressions in tiles.
    // An edge that only one of its ends lists is walked from that end alone: the
    // search over all depressions follows the list of the cell it has reached,
    // the one by depression looks into the lists of the cells it has not.
    const bool all_at_once = p->bfs_window > 0 || !p->mutual;
    int last[2] = {0, 0};
    if (all_at_once) {
        GS_TRY(flat_compact(p, pit_ids));
        GS_CUDA(cudaMemcpyAsync(&last[0], p->scanbuf + n - 1, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
        GS_CUDA(cudaMemcpyAsync(&last[1], p->flagbuf + n - 1, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
        GS_CUDA(cudaStreamSynchronize(p->stream));
    }
    // pit cells sorted by (pit, id): segments for the flat pass and the per-pit
    // reductions.  The ordered compaction keeps id order; the stable radix sort
    // by pit then lists every pit's cells in increasing id.
    if (ncell > 0) {
        int bits = 1;
        while ((1 << bits) <= P && bits < 31) bits++;
        size_t bytes = p->cub_bytes;
        GS_CUDA(cub::DeviceRadixSort::SortPairs(p->cub_tmp, bytes, p->seg_keys, p->seg_keys2, p->seg_vals,
                                                p->seg_vals2, ncell, 0, bits, p->stream));
        p->launches++;
    }
    GS_TRY(exclusive_scan(p, p->seg_count, p->seg_start, np1));
    auto pit_tables = [&]() -> int {
        GS_TRY(pit_chunks(p, np1, ncell));
        const int NI = p->pit_items_max;
        const int* nch = p->pit_nch;
        const int* chs = p->pit_chs;
        const int* itp = p->pit_item;
        launch(p, k_pit_params, NI, 256, np1, nch, chs, itp, (const int*)p->seg_start, (const int*)p->seg_count,
               (const int*)p->seg_vals2, (const double*)lfill, h, clip_sl, (const double*)p->larea, p->pit_part);
        launch(p, k_pit_params_fin, grid_for(np1, B), B, np1, nch, chs, (const double*)p->pit_part,
               p->pit_params);
        launch(p, k_filled_lvl, grid_for(np1, B), B, np1, (const double*)p->pit_params, p->filled_lvl);
        launch(p, k_filled_vol, NI, 256, np1, nch, chs, itp, (const int*)p->seg_start, (const int*)p->seg_count,
               (const int*)p->seg_vals2, h, clip_sl, (const double*)p->farea, (const double*)p->filled_lvl,
               p->pit_part);
        launch(p, k_filled_vol_fin, grid_for(np1, B), B, np1, nch, chs, (const double*)p->pit_part,
               (const double*)p->pit_params, p->filled_vol);
        GS_LAUNCH();
        return GS_OK;
    };
    // Without sediment the pit cells are above sea level and the flat pass
    // rewrites lFill only at open-sea cells, so that it and the pit tables read
    // and write disjoint data.  The flat pass is queued first: a deep lake makes
    // it the longer of the two.
    p->flat_args = FlatArgs{lfill, pit_ids, flat_dirs, h, sealevel};
    if (ncell > 0) {
        GS_CUDA(cudaEventRecord(p->ev_fork_b, p->stream));
        GS_CUDA(cudaStreamWaitEvent(p->side_b, p->ev_fork_b, 0));
        {
            StreamSwap sw(p, p->side_b, nullptr);
            if (all_at_once) {
                GS_TRY(flat_search_all(p, last[0] + last[1], lfill, pit_ids));
                GS_TRY(flat_dirs_launch(p, p->flat_args, nullptr, nullptr));
                GS_CUDA(cudaMemcpyAsync(p->h_pinned + 2, p->i_scalar + 4, sizeof(int), cudaMemcpyDeviceToHost,
                                        p->stream));
            } else {
                GS_TRY(flat_search_pits(p, ncell, p->flat_args));
            }
        }
        GS_CUDA(cudaEventRecord(p->ev_b, p->side_b));
        p->bfs_pending = all_at_once ? 1 : 2;
    } else {
        if (st) st->flat_rounds = 0;
        p->pdir_bound = 2;
        GS_TRY(flat_dirs_launch(p, p->flat_args, nullptr, nullptr));
    }
    if (!sed) GS_TRY(pit_tables());

    // With sediment the open-sea reset of lFill in k_flat_dirs touches pit
    // cells (marine depressions are labelled), and the pit tables read the
    // reset lFill (pitfilling.py:820-846): join the BFS first.
    if (sed) {
        GS_TRY(fill_join(p, st));
        GS_TRY(pit_tables());
    }
    if (!defer_flats) GS_TRY(fill_join(p, st));
    return GS_OK;
}


// smallest per-SM residency of the cooperative kernels at 256 threads
int coop_occupancy(int* per_sm) {
    int a = 0, b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, k_relax_active, 256, 0) != cudaSuccess) return 1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_cg_coop, 256, 0) != cudaSuccess) return 1;
    int c = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&c, k_cg_coop32, 256, 0) != cudaSuccess) return 1;
    *per_sm = std::min(std::min(a, b), c);
    return 0;
}

}  // namespace gs
