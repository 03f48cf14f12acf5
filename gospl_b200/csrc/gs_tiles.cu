// Exact solves of the triangular systems over the receiver graph by dataflow
// over mesh tiles.
//
// The mesh is cut into compact tiles of at most T vertices, one resident
// block per tile (one per SM).  A block keeps the values of its vertices, the
// count of their unsolved predecessors and a ready queue in shared memory; a
// vertex whose last predecessor is solved is taken up at once by the thread
// that solved it (or put in the queue), so a dependency hop inside a tile
// costs shared-memory operations and one read of the vertex's record instead
// of a store to L2 seen by a polling loop.  Only hops between tiles go through
// global memory: a vertex with a successor in another tile publishes its
// value there, and a few warps of each block poll the values its cut edges
// still wait for.
//
// What bounds it: the longest dependency chain (24 hops in the snapshot graph
// and 633 in the lake cascade's on a 160,000-vertex planar landscape, whose
// lakes are long single-receiver chains), at about 0.33 us a hop in shared
// memory (some 80 dependent instructions), plus two to three microseconds for
// each hop that leaves a tile; the tiles are compact patches so that few do
// (22 on that chain).  Measured against the ordered sweeps, B200, per sweep:
// cascade graph 390 -> 235 us at 160,000 vertices and 139 -> 90 us at 20,000; no
// order of the vertices has to be sorted or merged for it, which saves the
// cascade pass of those meshes another 300 us of launches and host round trips.
//
// No order of the vertices is needed: predecessors are summed in a fixed order
// (donors ascending by id, receivers in slot order), so results do not depend
// on scheduling.  The graph must be acyclic, which the build pass checks edge by
// edge against (surface, flat distance, id), a total order.  Every wait is
// bounded by the plan's sweep budget (GS_ETIMEOUT).
#include <algorithm>
#include <cmath>
#include <vector>

#include "gs_plan.cuh"
#include "gs_tiles.cuh"

namespace gs {

namespace {

// one 512-thread block per tile; its last POLL_WARPS warps poll the cut edges
// first and join the others when none is left
constexpr int TS_THREADS = 512;
constexpr int POLL_WARPS = 4;
constexpr int POLL_LANES = POLL_WARPS * 32;
constexpr int POLL_EDGES = 8;                // cut edges a polling lane holds at a time
constexpr unsigned short Q_EMPTY = 0xffff;   // queue slot not filled yet
constexpr int TILE_MAX = 0xf000;             // local ids and cut edges share 16 bits
constexpr int TILE_MIN = 512;
constexpr int SM_SPARE = 4;                  // SMs left to the flat-distance BFS beside the sweep
constexpr int CHAIN = 8;                      // hops a lane follows before it looks at the queue again
constexpr uint16_t PM_IN = 1 << 12;          // flags above the predecessor slots
constexpr uint16_t PM_OUT = 1 << 13;
constexpr uint16_t PM_PRED = 0x0fff;

constexpr unsigned long long XSENT = 0x7ff4dead0badf00dULL;   // a value not published yet

__device__ __forceinline__ double ld_pub(const double* p) {
    unsigned long long v;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return __longlong_as_double((long long)v);
}
__device__ __forceinline__ void st_pub(double* p, double v) {
    asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"((unsigned long long)__double_as_longlong(v)) : "memory");
}
__device__ __forceinline__ bool pending_val(double v) {
    return (unsigned long long)__double_as_longlong(v) == XSENT;
}

// shared-memory accesses by 32-bit address (the hop's critical path)
__device__ __forceinline__ unsigned sm_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ double lds_f64(unsigned a) {
    double v;
    asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void sts_f64(unsigned a, double v) {
    asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ uint4 lds_u128(unsigned a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ double2 lds_2f64(unsigned a) {
    double2 v;
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ unsigned lds_u16(unsigned a) {
    unsigned short v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ unsigned atoms_add(unsigned a, unsigned v) {
    unsigned o;
    asm volatile("atom.shared.add.u32 %0, [%1], %2;" : "=r"(o) : "r"(a), "r"(v) : "memory");
    return o;
}
__device__ __forceinline__ void fence_cta() { asm volatile("fence.acq_rel.cta;" ::: "memory"); }

// Record of a vertex with room for NP predecessors and successors (NP = 6, 8 or
// 12 by the mesh's largest degree).  Predecessors are 16-bit indices into the
// block's values: a local vertex, or T + k for the value that arrived over cut
// edge k.  The first 48 bytes hold all that a vertex of up to four
// predecessors and three successors in its tile needs (most of them):
//   0  successors 0..2, then the counts (RI_*); predecessors 0..3 (16 bits each)
//  16  weights 0..3, in summation order
// and the rest follows: weights 4.., predecessors 4.., successors 3..,
// the divisor.
constexpr unsigned RI_ND = 0xf, RI_NS_SHIFT = 4, RI_OUT = 0x100;
template <int NP>
struct Rec {
    static constexpr int OFF_W = 16;
    static constexpr int OFF_P4 = OFF_W + 8 * NP;
    static constexpr int OFF_S3 = OFF_P4 + 2 * (NP - 4);
    static constexpr int OFF_DIV = (OFF_S3 + 2 * (NP - 3) + 7) / 8 * 8;
    static constexpr int BYTES = (OFF_DIV + 8 + 31) / 32 * 32;
};

struct SweepArgs {
    int n, T;
    const int* perm;          // tile-major position -> vertex (null: identity)
    const char* rec;
    const uint16_t* pm;
    const double* b;          // right-hand side, by vertex
    double* x;                // solution, by vertex
    double* xb;               // published values of this solve, by position
    double* xb_next;          // those of the next solve, reset here
    const int* cut0;          // [nt + 1] first cut edge of each tile
    const unsigned* cut_q;    // position of the neighbour across the edge
    const unsigned* cut_l;    // local vertex | slot << 16
    int cut_cap;
    unsigned* status;
    const int* skip;          // non-zero: the graph failed its check, nothing is solved (null: not checked)
    unsigned long long budget_ns;
};

// shared memory of a tile: values (vertices, then cut edges), records (whole, or
// the hot part and the divisors), counts and a spare word per lane, queue, list
// of the cut edges in use
constexpr int HOT = 48;
__host__ __device__ inline size_t tile_values(int T, int cut_cap) {
    return (((size_t)T + cut_cap) * 8 + 15) / 16 * 16;
}
// words of the counts: one each, or one for four vertices when no record is kept
__host__ __device__ inline int tile_count_words(int T, bool bytes) {
    return bytes ? (T + 7) / 8 * 2 : (T + 1) / 2 * 2;
}
__host__ __device__ inline size_t tile_smem(int T, int cut_cap, int rec_bytes) {
    const size_t t2 = (size_t)(T + 1) / 2 * 2;
    return tile_values(T, cut_cap) + (size_t)T * rec_bytes + (size_t)tile_count_words(T, rec_bytes == 0) * 4 + 128 +
           t2 * 2 + (size_t)cut_cap * 2;
}

// KEEP 2: the tile's whole records are copied to shared memory first; 1: only
// their first HOT bytes and the divisors, and a vertex with more than four
// predecessors or three successors reads the rest from L2; 0: none, every record
// is read from L2 and a count takes a byte.
template <int NP, bool DIV, int KEEP>
__global__ void __launch_bounds__(TS_THREADS, 1) k_tile_sweep(SweepArgs a) {
    extern __shared__ double sm_tile[];
    __shared__ unsigned s_head, s_tail, s_ncut;
    __shared__ int s_left, s_stop;
    using R = Rec<NP>;
    const int T = a.T, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NW = TS_THREADS / 32, NWORK = NW - POLL_WARPS;   // warps that start with work
    const unsigned full = 0xffffffffu;
    constexpr bool FULL = KEEP == 2, HOTS = KEEP == 1;
    constexpr int RB = FULL ? R::BYTES : HOTS ? HOT : 0;
    double* sx = sm_tile;
    char* srec = (char*)sm_tile + tile_values(T, a.cut_cap);
    double* sdiv = (double*)(srec + (size_t)T * RB);   // with the hot parts
    unsigned* cntw = (unsigned*)(sdiv + (HOTS ? T : 0));   // unsolved predecessors of l
    const int nw = tile_count_words(T, KEEP == 0);
    unsigned* spare = cntw + nw;
    unsigned short* queue = (unsigned short*)(spare + 32);
    unsigned short* act_cut = queue + (T + 1) / 2 * 2;
    volatile unsigned short* vq = queue;
    const int p0 = blockIdx.x * T;
    const int m = min(T, a.n - p0);
    const int c0 = a.cut0[blockIdx.x], nc = a.cut0[blockIdx.x + 1] - c0;
    const char* grec = a.rec + (size_t)p0 * R::BYTES;
    const unsigned long long t0 = globaltimer_ns();
    if (tid == 0) {
        s_head = NWORK * 32;   // the first tickets are handed out below
        s_tail = 0u;
        s_ncut = 0u;
        s_left = 0;
        s_stop = ld_relaxed_u32(a.status) != 0u;
        if (!s_stop && a.skip && *a.skip) {
            atomicCAS(a.status, 0u, TILE_REJECTED);
            s_stop = 1;
        }
    }
    __syncthreads();
    if (s_stop) return;
    // the values start as the right-hand side; a vertex without predecessors
    // and successors is done unless it is divided
    int work = 0;
    for (int l = tid; l < m; l += TS_THREADS) {
        const int p = p0 + l;
        const unsigned f = a.pm[p];
        const unsigned nd = __popc(f & PM_PRED);
        sx[l] = a.b[a.perm ? a.perm[p] : p];
        if (KEEP == 0) ((uint8_t*)cntw)[l] = (uint8_t)nd;
        else cntw[l] = nd;
        queue[l] = Q_EMPTY;
        if (DIV || nd || (f & (PM_IN | PM_OUT))) {
            work++;
            if (HOTS && DIV) sdiv[l] = __ldg((const double*)(grec + (size_t)l * R::BYTES + R::OFF_DIV));
        }
    }
    for (int e = tid; e < nc; e += TS_THREADS) sx[T + e] = __longlong_as_double((long long)XSENT);
    if constexpr (KEEP != 0)
        for (int q = tid; q < m * (RB / 16); q += TS_THREADS) {
            const int l = FULL ? 0 : q / (RB / 16), o = FULL ? q : q - l * (RB / 16);
            ((uint4*)srec)[q] = __ldg((const uint4*)(grec + (size_t)l * R::BYTES) + o);
        }
    if (tid < 32) spare[tid] = 0x40000000u;
    work = __reduce_add_sync(full, work);
    if (lane == 0 && work) atomicAdd(&s_left, work);
    for (int e = tid; e < nc; e += TS_THREADS) {
        const unsigned ls = a.cut_l[c0 + e], l = ls & 0xffffu;
        a.xb_next[p0 + l] = __longlong_as_double((long long)XSENT);
        if ((a.pm[p0 + l] >> (ls >> 16)) & 1u) act_cut[atomicAdd(&s_ncut, 1u)] = (unsigned short)e;
    }
    if (tid == 0 && globaltimer_ns() - t0 > a.budget_ns) {
        atomicCAS(a.status, 0u, (unsigned)GS_ETIMEOUT);
        s_stop = 1;
    }
    __syncthreads();
    if (s_stop) return;

    // one predecessor of l solved: its count before
    const unsigned cnt_a = sm_addr(cntw), x_a = sm_addr(sx), rec_a = sm_addr(srec), div_a = sm_addr(sdiv);
    auto arrive = [&](unsigned l) -> unsigned {
        if (KEEP != 0) return atoms_add(cnt_a + 4u * l, ~0u);
        const unsigned sh = 8u * (l & 3u);   // a count never goes below zero: no borrow
        return (atoms_add(cnt_a + (l & ~3u), 0u - (1u << sh)) >> sh) & 0xffu;
    };
    // absent successors count down a word of their lane that nothing reads
    const unsigned none = (unsigned)(nw + lane) * (KEEP == 0 ? 4u : 1u);
    // The values that l's other predecessors released with their counts reach the
    // taker through this thread, which saw the last count: a fence between that
    // count and the queue entry (the taker's own stands behind its read of the entry)
    auto push = [&](unsigned l) {
        fence_cta();
        const unsigned pos = atomicAdd(&s_tail, 1u);   // a vertex is pushed at most once: pos < T
        vq[pos] = (unsigned short)l;
    };
    // lane 0 watches the budget and other blocks' status; the whole warp leaves together
    auto stopped = [&](bool look) -> bool {
        int st = 0;
        if (lane == 0) {
            st = *(volatile int*)&s_stop;
            if (!st && look) {
                if (ld_relaxed_u32(a.status) != 0u) st = 1;
                else if (globaltimer_ns() - t0 > a.budget_ns) {
                    atomicCAS(a.status, 0u, (unsigned)GS_ETIMEOUT);
                    st = 1;
                }
                if (st) *(volatile int*)&s_stop = 1;
            }
        }
        return __shfl_sync(full, st, 0) != 0;
    };

    bool leave = false;
    if (warp >= NWORK) {
        // poll the cut edges in use: the pollers own edges e, e + POLL_LANES, ...,
        // PE of them at a time with their addresses in registers, so that a pass
        // is one round trip to L2
        constexpr int PE = POLL_EDGES;
        const int ncut = (int)s_ncut, first = tid - (TS_THREADS - POLL_LANES);
        const int groups = (ncut + POLL_LANES * PE - 1) / (POLL_LANES * PE);
        unsigned long long left_g = 0ull;   // groups of this lane with edges still waited for (at most 64)
        unsigned rounds = 0;
        unsigned todo0 = 0u, el0[PE];
        const double* ad0[PE];
        auto load_group = [&](int g, unsigned& todo, unsigned (&el)[PE], const double* (&ad)[PE]) {
            todo = 0u;
#pragma unroll
            for (int u = 0; u < PE; u++) {
                const int k = (g * PE + u) * POLL_LANES + first;
                ad[u] = a.xb;
                el[u] = 0u;
                if (k < ncut) {
                    const unsigned e = act_cut[k];
                    if (pending_val(((volatile double*)sx)[T + e])) {
                        ad[u] = a.xb + __ldg(a.cut_q + c0 + e);
                        el[u] = e | ((__ldg(a.cut_l + c0 + e) & 0xffffu) << 16);
                        todo |= 1u << u;
                    }
                }
            }
        };
        for (int g = 0; g < groups; g++) left_g |= 1ull << g;
        int g = 0;
        if (groups > 0) load_group(0, todo0, el0, ad0);
        while (!leave && __any_sync(full, left_g != 0ull)) {
            double v[PE];
#pragma unroll
            for (int u = 0; u < PE; u++)
                if ((todo0 >> u) & 1u) v[u] = ld_pub(ad0[u]);
            bool got = false;
#pragma unroll
            for (int u = 0; u < PE; u++) {
                if (!((todo0 >> u) & 1u) || pending_val(v[u])) continue;
                todo0 &= ~(1u << u);
                got = true;
                sts_f64(x_a + 8u * (T + (el0[u] & 0xffffu)), v[u]);
                fence_cta();
                if (arrive(el0[u] >> 16) == 1u) push(el0[u] >> 16);
            }
            if (todo0 == 0u) left_g &= ~(1ull << g);
            if (!__any_sync(full, got) && (++rounds & 31u) == 0u) leave = stopped(true);
            if (groups > 1) {   // more edges than registers: the next group that still waits
                do g = g + 1 < groups ? g + 1 : 0;
                while (__any_sync(full, left_g != 0ull) && !__any_sync(full, (left_g >> g) & 1ull));
                load_group(g, todo0, el0, ad0);
            }
        }
    }

    // the sources of this thread first, then the queue; consecutive tickets go
    // to different warps, so that vertices that become ready one after the
    // other do not share (and wait for) one warp's loads
    int src = warp < NWORK ? tid : m;   // (the polling warps take no sources: nobody would wait for them)
    unsigned slot = (unsigned)(lane * NWORK + warp);
    bool ticket = warp < NWORK;
    int cur = -1;
    unsigned rounds = 0;
    while (!leave) {
        // a ticket for each lane without work that has none
        const unsigned need = __ballot_sync(full, cur < 0 && !ticket);
        if (need) {
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(&s_head, (unsigned)__popc(need));
            base = __shfl_sync(full, base, 0);
            if (cur < 0 && !ticket) {
                slot = base + __popc(need & ((1u << lane) - 1u));
                ticket = true;
            }
        }
        if (cur < 0) {
            while (src < m) {
                const int l = src;
                src += NWORK * 32;
                const unsigned f = a.pm[p0 + l];
                if (!(f & PM_PRED) && (DIV || (f & (PM_IN | PM_OUT)))) { cur = l; break; }
            }
            if (cur < 0 && slot < (unsigned)m) {   // at most m vertices are ever pushed
                const unsigned short v = vq[slot];
                if (v != Q_EMPTY) {
                    cur = v;
                    ticket = false;
                }
            }
        }
        if (!__any_sync(full, cur >= 0)) {
            int left = 0;
            if (lane == 0) left = *(volatile int*)&s_left;
            if (__shfl_sync(full, left, 0) <= 0) break;
            if ((++rounds & 63u) == 0u) leave = stopped(true);
            else __nanosleep(20);
            continue;
        }
        int done = 0;
        for (int hop = 0; hop < CHAIN && cur >= 0; hop++) {
            const unsigned l = (unsigned)cur;
            const unsigned rs = rec_a + l * RB;
            const char* rg = grec + (size_t)l * R::BYTES;
            const uint4 hd = KEEP != 0 ? lds_u128(rs) : __ldg((const uint4*)rg);
            const double2 w01 = KEEP != 0 ? lds_2f64(rs + R::OFF_W) : __ldg((const double2*)(rg + R::OFF_W)),
                          w23 = KEEP != 0 ? lds_2f64(rs + R::OFF_W + 16) : __ldg((const double2*)(rg + R::OFF_W + 16));
            const double dv = !DIV ? 1.0 : FULL ? lds_f64(rs + R::OFF_DIV) : lds_f64(div_a + 8u * l);
            const unsigned info = hd.y >> 16;
            const int nd = (int)(info & RI_ND), ns = (int)((info >> RI_NS_SHIFT) & 0xfu);
            fence_cta();   // the predecessors' values, after their counts
            double acc = lds_f64(x_a + 8u * l);
            if (nd > 0) {
                // an absent predecessor's index is a valid one and its product is dropped
                const double v0 = lds_f64(x_a + 8u * (hd.z & 0xffffu)), v1 = lds_f64(x_a + 8u * (hd.z >> 16));
                acc = acc + w01.x * v0;
                const double s1 = acc + w01.y * v1;
                acc = nd > 1 ? s1 : acc;
                if (nd > 2) {
                    const double v2 = lds_f64(x_a + 8u * (hd.w & 0xffffu)), v3 = lds_f64(x_a + 8u * (hd.w >> 16));
                    acc = acc + w23.x * v2;
                    const double s3 = acc + w23.y * v3;
                    acc = nd > 3 ? s3 : acc;
                    for (int q = 4; q < nd; q++) {
                        const unsigned pi = FULL ? lds_u16(rs + R::OFF_P4 + 2 * (q - 4))
                                                 : __ldg((const unsigned short*)(rg + R::OFF_P4) + (q - 4));
                        const double wq = FULL ? lds_f64(rs + R::OFF_W + 8 * q)
                                               : __ldg((const double*)(rg + R::OFF_W) + q);
                        acc = acc + wq * lds_f64(x_a + 8u * pi);
                    }
                }
            }
            if (DIV) acc = acc / dv;
            sts_f64(x_a + 8u * l, acc);
            fence_cta();
            // the counts of the first three successors, all in flight together,
            // then what became ready: this lane goes on with one of them
            const unsigned s0 = hd.x & 0xffffu, s1 = hd.x >> 16, s2 = hd.y & 0xffffu;
            const unsigned o0 = arrive(ns > 0 ? s0 : none), o1 = arrive(ns > 1 ? s1 : none),
                           o2 = arrive(ns > 2 ? s2 : none);
            const bool r0 = o0 == 1u && ns > 0, r1 = o1 == 1u && ns > 1, r2 = o2 == 1u && ns > 2;
            int next = r0 ? (int)s0 : r1 ? (int)s1 : r2 ? (int)s2 : -1;
            if ((r0 && r1) || (r2 && (r0 || r1)) || ns > 3) {
                if (r0 && r1) push(s1);
                if (r2 && (r0 || r1)) push(s2);
                for (int q = 3; q < ns; q++) {
                    const unsigned sq = FULL ? lds_u16(rs + R::OFF_S3 + 2 * (q - 3))
                                             : __ldg((const unsigned short*)(rg + R::OFF_S3) + (q - 3));
                    if (arrive(sq) != 1u) continue;
                    if (next < 0) next = (int)sq;
                    else push(sq);
                }
            }
            if (info & RI_OUT) st_pub(&a.xb[p0 + l], acc);
            cur = next;
            done++;
        }
        done = __reduce_add_sync(full, done);
        if (lane == 0) atomicSub(&s_left, done);
    }
    __syncthreads();
    if (s_stop) return;
    for (int l = tid; l < m; l += TS_THREADS) a.x[a.perm ? a.perm[p0 + l] : p0 + l] = sx[l];
}

__global__ void k_fill_pending(int n, double* a, double* b) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    a[i] = b[i] = __longlong_as_double((long long)XSENT);
}

// ---------------------------------------------------------------------------
// Build passes: one thread per tile-major position writes the vertex's record
// and its predecessor slots.
struct BuildArgs {
    int n, T, R;
    const int* perm;
    const int* loc;           // vertex -> position (null: identity)
    const int* nbr;
    const int8_t* nnb;
    const int8_t* rev;
    const unsigned long long* sorder;
    const int* rcv;           // [R][n]
    const int8_t* rslot;
    const double* co;         // [R][n] weight or coefficient of each receiver edge, 0: no edge
    const double* z;          // order check: surface, flat distance (null: none)
    const int* pdir;
    const uint16_t* ref;      // edges must be among those of this donor graph (null: not checked)
    int div;
    const uint16_t* cut_idx;  // [W][n] by position: cut edge of each slot within its tile
    char* rec;
    uint16_t* pm;
    int* bad;
};

// a record while it is put together; slots are filled by compile-time index
template <int NP>
struct RecOut {
    double w[NP];
    unsigned short suc[NP];
    unsigned short pr[NP];
    double dv = 1.0;
    int nd = 0, ns = 0;
    bool out = false;
    unsigned mask = 0u;
    __device__ __forceinline__ void pred(double wq, unsigned short idx, int slot) {
#pragma unroll
        for (int c = 0; c < NP; c++)
            if (c == nd) {
                w[c] = wq;
                pr[c] = idx;
            }
        nd++;
        mask |= 1u << slot;
    }
    __device__ __forceinline__ void succ(unsigned short idx) {
#pragma unroll
        for (int c = 0; c < NP; c++)
            if (c == ns) suc[c] = idx;
        ns++;
    }
};

// writes the parts of a record that its readers touch
template <int NP>
__device__ __forceinline__ void rec_store(const BuildArgs& a, int p, RecOut<NP>& o) {
    using R = Rec<NP>;
    a.pm[p] = (uint16_t)(o.mask | (o.ns ? PM_IN : 0) | (o.out ? PM_OUT : 0));
    if (!o.nd && !o.ns && !o.out && !a.div) return;
    char* r = a.rec + (size_t)p * R::BYTES;
    const unsigned info = (unsigned)o.nd | ((unsigned)o.ns << RI_NS_SHIFT) | (o.out ? RI_OUT : 0u);
    auto two = [](unsigned short x, unsigned short y) { return (unsigned)x | ((unsigned)y << 16); };
    uint4 hd;
    hd.x = two(o.ns > 0 ? o.suc[0] : 0, o.ns > 1 ? o.suc[1] : 0);
    hd.y = two(o.ns > 2 ? o.suc[2] : 0, (unsigned short)info);
    hd.z = two(o.nd > 0 ? o.pr[0] : 0, o.nd > 1 ? o.pr[1] : 0);
    hd.w = two(o.nd > 2 ? o.pr[2] : 0, o.nd > 3 ? o.pr[3] : 0);
    *(uint4*)r = hd;
    if (o.nd > 0) *(double2*)(r + R::OFF_W) = make_double2(o.w[0], o.nd > 1 ? o.w[1] : 0.0);
    if (o.nd > 2) *((double2*)(r + R::OFF_W) + 1) = make_double2(o.w[2], o.nd > 3 ? o.w[3] : 0.0);
#pragma unroll
    for (int q = 4; q < NP; q++)
        if (q < o.nd) {
            ((double*)(r + R::OFF_W))[q] = o.w[q];
            ((unsigned short*)(r + R::OFF_P4))[q - 4] = o.pr[q];
        }
#pragma unroll
    for (int q = 3; q < NP; q++)
        if (q < o.ns) ((unsigned short*)(r + R::OFF_S3))[q - 3] = o.suc[q];
    if (a.div) *(double*)(r + R::OFF_DIV) = o.dv;
}

// index of the value of the neighbour at position pj over slot t of position p
__device__ __forceinline__ unsigned short pred_index(const BuildArgs& a, int p, int tile, int t, int pj) {
    const int l = pj - tile * a.T;
    if (l >= 0 && l < a.T) return (unsigned short)l;
    return (unsigned short)(a.T + a.cut_idx[(size_t)t * a.n + p]);
}

// Donors as predecessors, receivers as successors (flow accumulation; with
// div the transposed stream-power system).  The receiver edge of a donor is
// found through its receiver slots; donors are taken in ascending id.  The
// loads of all slots go out together, level by level (ids, receiver slots,
// coefficients), since each level's addresses come from the one before.
template <int NP>
__global__ void __launch_bounds__(128) k_build_down(BuildArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const int n = a.n, i = a.perm ? a.perm[p] : p, tile = p / a.T;
    RecOut<NP> o;
    const int deg = a.nnb[i];
    const double zi = a.z ? a.z[i] : 0.0;
    const int di = a.pdir ? a.pdir[i] : 0;
    int bad = 0;
    int j[NP], rt[NP];
    double w[NP];
#pragma unroll
    for (int t = 0; t < NP; t++) {
        j[t] = t < deg ? a.nbr[(size_t)t * n + i] : -1;
        rt[t] = t < deg ? (int)a.rev[(size_t)t * n + i] : -1;
        w[t] = 0.0;
    }
    unsigned hit = 0u;
    unsigned kk[NP];
    for (int k = 0; k < a.R; k++)
#pragma unroll
        for (int t = 0; t < NP; t++)
            if (rt[t] >= 0 && j[t] >= 0 && a.rslot[(size_t)k * n + j[t]] == rt[t] && !((hit >> t) & 1u)) {
                kk[t] = k;
                hit |= 1u << t;
            }
#pragma unroll
    for (int t = 0; t < NP; t++)
        if ((hit >> t) & 1u) w[t] = a.co[(size_t)kk[t] * n + j[t]];
#pragma unroll
    for (int t = 0; t < NP; t++) {
        if (!((hit >> t) & 1u)) continue;
        if (!(w[t] != 0.0)) {
            hit &= ~(1u << t);
            continue;
        }
        if (a.z) {
            const double zj = a.z[j[t]];
            if (!(zj > zi)) {
                const int dj = a.pdir ? a.pdir[j[t]] : 0;
                if (!(zj == zi && (dj > di || (dj == di && j[t] < i)))) bad = 1;
            }
        }
    }
    if (a.ref && (hit & ~(unsigned)a.ref[p])) bad = 1;
    unsigned long long ord = a.sorder[i];
    for (unsigned left = hit; left;) {
        const int t = (int)(ord & 15ULL);
        ord >>= 4;
        if (!((left >> t) & 1u)) continue;
        left &= ~(1u << t);
        double wt = 0.0;
        int jt = 0;
#pragma unroll
        for (int c = 0; c < NP; c++)
            if (c == t) {
                wt = w[c];
                jt = j[c];
            }
        o.pred(wt, pred_index(a, p, tile, t, a.loc ? a.loc[jt] : jt), t);
    }
    double den = 1.0;
    for (int k = 0; k < a.R; k++) {
        const int s = a.rslot[(size_t)k * n + i];
        const double c = a.co[(size_t)k * n + i];
        den = den + c;
        if (s < 0 || !(c != 0.0)) continue;
        int r = -1, back = -1;
#pragma unroll
        for (int t = 0; t < NP; t++)
            if (t == s) {
                r = j[t];
                back = rt[t];
            }
        if (back < 0) continue;
        if (a.rcv[(size_t)k * n + i] != r || ((hit >> s) & 1u)) bad = 1;
        const int pr = a.loc ? a.loc[r] : r;
        if (pr / a.T == tile) o.succ((unsigned short)(pr - tile * a.T));
        else o.out = true;
    }
    o.dv = den;
    if (bad) *a.bad = 1;
    rec_store<NP>(a, p, o);
}

// Receivers as predecessors (in receiver order), donors as successors
// (stream power, div; without div the transposed flow system).  Latency bounds it
// (a wave of blocks takes as long as its chain of loads): 23 and 35 us on lattices
// of 160,000 and 300,000 vertices, 31 and 44 when the coefficient of a slot was
// loaded behind the test of its receiver slots, one slot after the other.
template <int NP>
__global__ void __launch_bounds__(128) k_build_up(BuildArgs a) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const int n = a.n, i = a.perm ? a.perm[p] : p, tile = p / a.T;
    RecOut<NP> o;
    const int deg = a.nnb[i];
    int bad = 0;
    // only a donor of the reference graph can be a successor: any other edge is
    // found by the vertex it leaves, and the graph is rejected
    const unsigned may = a.ref ? a.ref[p] & PM_PRED : PM_PRED;
    int j[NP], rt[NP];
#pragma unroll
    for (int t = 0; t < NP; t++) {
        j[t] = t < deg ? a.nbr[(size_t)t * n + i] : -1;
        rt[t] = t < deg ? (int)a.rev[(size_t)t * n + i] : -1;
    }
    // (the loads of all slots together, as in k_build_down)
    unsigned hit = 0u;
    unsigned kk[NP];
    for (int k = 0; k < a.R; k++)
#pragma unroll
        for (int t = 0; t < NP; t++)
            if (((may >> t) & 1u) && rt[t] >= 0 && j[t] >= 0 && a.rslot[(size_t)k * n + j[t]] == rt[t]) {
                kk[t] = k;
                hit |= 1u << t;
            }
    double w[NP];
#pragma unroll
    for (int t = 0; t < NP; t++) w[t] = (hit >> t) & 1u ? a.co[(size_t)kk[t] * n + j[t]] : 0.0;
#pragma unroll
    for (int t = 0; t < NP; t++)
        if (!(w[t] != 0.0)) hit &= ~(1u << t);
    double den = 1.0;
    for (int k = 0; k < a.R; k++) {
        const double c = a.co[(size_t)k * n + i];
        den = den + c;
        const int r = a.rcv[(size_t)k * n + i];
        if (r == i || !(c != 0.0)) continue;
        const int s = a.rslot[(size_t)k * n + i];
        int rs = -1, back = -1;
#pragma unroll
        for (int t = 0; t < NP; t++)
            if (t == s) {
                rs = j[t];
                back = rt[t];
            }
        if (back < 0 || rs != r || ((o.mask >> s) & 1u) || ((hit >> s) & 1u)) {
            bad = 1;
            continue;
        }
        const int pr = a.loc ? a.loc[r] : r;
        if (a.ref && !((a.ref[pr] >> back) & 1)) bad = 1;
        o.pred(c, pred_index(a, p, tile, s, pr), s);
    }
#pragma unroll
    for (int t = 0; t < NP; t++) {
        if (!((hit >> t) & 1u)) continue;
        const int pj = a.loc ? a.loc[j[t]] : j[t];
        if (pj / a.T == tile) o.succ((unsigned short)(pj - tile * a.T));
        else o.out = true;
    }
    o.dv = den;
    if (bad) *a.bad = 1;
    rec_store<NP>(a, p, o);
}

// Marine flow (the coupled marine system): donors as predecessors, a donor
// being a neighbour whose receiver bit set (over its neighbour slots) holds the
// slot of this vertex; the weight is the donor's own.
template <int NP>
__global__ void __launch_bounds__(128) k_build_marine(BuildArgs a, const unsigned short* __restrict__ cand) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.n) return;
    const int n = a.n, i = a.perm ? a.perm[p] : p, tile = p / a.T;
    RecOut<NP> o;
    unsigned long long ord = a.sorder[i];
    const int deg = a.nnb[i];
    const double zi = a.z[i];
    const unsigned mine = cand[i];
    int bad = 0;
    for (int q = 0; q < deg; q++) {
        const int t = (int)(ord & 15ULL);
        ord >>= 4;
        if (t >= deg) break;   // slots without a neighbour end the list
        const int j = a.nbr[(size_t)t * n + i];
        const int rt = a.rev[(size_t)t * n + i];
        if (rt < 0) continue;
        const int pj = a.loc ? a.loc[j] : j;
        const bool don = (cand[j] >> rt) & 1u, rcv = (mine >> t) & 1u;
        if (don && rcv) bad = 1;
        if (don) {
            const double zj = a.z[j];
            if (!(zj > zi || (zj == zi && j < i))) bad = 1;
            o.pred(a.co[j], pred_index(a, p, tile, t, pj), t);
        }
        if (rcv) {
            if (pj / a.T == tile) o.succ((unsigned short)(pj - tile * a.T));
            else o.out = true;
        }
    }
    if (bad) *a.bad = 1;
    rec_store<NP>(a, p, o);
}

template <class F>
int by_width(const gs_plan* p, F f) {
    if (p->tl_np == 6) return f(std::integral_constant<int, 6>{});
    if (p->tl_np == 8) return f(std::integral_constant<int, 8>{});
    return f(std::integral_constant<int, 12>{});
}

template <int NP>
const void* sweep_kernel(bool div, int keep) {
    if (keep == 2) return div ? (const void*)k_tile_sweep<NP, true, 2> : (const void*)k_tile_sweep<NP, false, 2>;
    if (keep == 1) return div ? (const void*)k_tile_sweep<NP, true, 1> : (const void*)k_tile_sweep<NP, false, 1>;
    return div ? nullptr : (const void*)k_tile_sweep<NP, false, 0>;
}

}  // namespace

// Cut edges of a tile (one block): their number, or with FILL their tables from
// c0[tile] on, by position and slot.  On the device, which has the neighbour rows
// already: two passes on the host and the upload of the tables took 12 ms of a
// plan's creation at 160,000 vertices and 30 at 655,000.
constexpr int CUT_THREADS = 256;
template <bool FILL>
__global__ void __launch_bounds__(CUT_THREADS) k_cuts(int n, int T, const int* __restrict__ perm,
                                                      const int* __restrict__ loc, const int* __restrict__ nbr,
                                                      const int8_t* __restrict__ nnb, int* count,
                                                      const int* __restrict__ c0, unsigned* cut_q, unsigned* cut_l,
                                                      uint16_t* cut_idx) {
    constexpr int NW = CUT_THREADS / 32;
    __shared__ int s_warp[NW];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tile = blockIdx.x;
    const int p0 = tile * T, m = min(T, n - p0);
    int run = 0;
    for (int base = 0; base < m; base += CUT_THREADS) {
        const int p = p0 + base + tid;
        int cnt = 0, i = 0;
        unsigned cut = 0u;
        if (base + tid < m) {
            i = perm ? perm[p] : p;
            const int deg = nnb[i];
            for (int s = 0; s < deg; s++) {
                const int j = nbr[(size_t)s * n + i];
                if (j >= 0 && j < n && (loc ? loc[j] : j) / T != tile) cut |= 1u << s;
            }
            cnt = __popc(cut);
        }
        int incl = cnt;
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += v;
        }
        __syncthreads();   // the sums of the batch before are read
        if (lane == 31) s_warp[warp] = incl;
        __syncthreads();
        int before = 0, all = 0;
        for (int w = 0; w < NW; w++) {
            if (w < warp) before += s_warp[w];
            all += s_warp[w];
        }
        if (FILL) {
            int at = run + before + incl - cnt;
            for (; cut; cut &= cut - 1u, at++) {
                const int s = __ffs(cut) - 1, j = nbr[(size_t)s * n + i];
                cut_idx[(size_t)s * n + p] = (uint16_t)at;
                cut_q[c0[tile] + at] = (unsigned)(loc ? loc[j] : j);
                cut_l[c0[tile] + at] = (unsigned)(p - p0) | ((unsigned)s << 16);
            }
        }
        run += all;
    }
    if (!FILL && tid == 0) count[tile] = run;
}

__global__ void k_loc(int n, const int* __restrict__ perm, int* loc) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < n) loc[perm[p]] = p;
}

// cut edges of each tile for the positions loc (null: identity); scratch: scanbuf
static int count_cuts(gs_plan* p, int T, int nt, const int* perm, const int* loc, std::vector<int>& cuts) {
    cuts.resize(nt);
    k_cuts<false><<<nt, CUT_THREADS>>>((int)p->n, T, perm, loc, p->nbr, p->nnb, p->scanbuf, nullptr, nullptr, nullptr,
                                       nullptr);
    GS_LAUNCH();
    GS_CUDA(cudaMemcpy(cuts.data(), p->scanbuf, sizeof(int) * nt, cudaMemcpyDeviceToHost));
    return GS_OK;
}

// Tile-major order of the vertices by growing one tile after the other
// breadth-first from an unassigned vertex next to the tiles already grown; by
// id within a tile, so that neighbours in memory stay together.
static void grow_tiles(int n, const int32_t* nnb, const int32_t* ngb, int T, int nt, std::vector<int>& perm) {
    std::vector<int> tile_of(n, -1), mark(n, -1), front, rest;
    size_t rh = 0;
    int scan = 0, done = 0;
    for (int tile = 0; done < n; tile++) {
        front.clear();
        size_t h = 0;
        for (int cnt = 0; cnt < T && done < n;) {
            if (h == front.size()) {
                int seed = -1;
                while (rh < rest.size() && seed < 0) {
                    const int c = rest[rh++];
                    if (tile_of[c] < 0) seed = c;
                }
                if (seed < 0) {
                    while (tile_of[scan] >= 0) scan++;
                    seed = scan;
                }
                mark[seed] = tile;
                front.push_back(seed);
            }
            const int v = front[h++];
            if (tile_of[v] >= 0) continue;
            tile_of[v] = tile;
            done++;
            cnt++;
            for (int s = 0; s < nnb[v]; s++) {
                const int j = ngb[(size_t)v * 12 + s];
                if (j < 0 || j >= n || tile_of[j] >= 0 || mark[j] == tile) continue;
                mark[j] = tile;
                front.push_back(j);
            }
        }
        for (; h < front.size(); h++)
            if (tile_of[front[h]] < 0) rest.push_back(front[h]);
    }
    std::vector<int> at(nt);
    for (int t = 0; t < nt; t++) at[t] = t * T;   // every tile but the last is full
    perm.resize(n);
    for (int v = 0; v < n; v++) perm[at[tile_of[v]]++] = v;
}

// The plan's tiles: one per SM but SM_SPARE (a cooperative launch waits for
// every SM it needs, and the one-block BFS of the fill runs beside the first
// sweep), at least TILE_MIN vertices each (512 and 1024 measured alike at 20,000
// and 160,000 vertices).  Consecutive ids are kept as they are when their tiles
// cut at most twice the edges of grown ones (meshes numbered along a
// space-filling curve: values then stay in vertex order); other numberings
// (rows of a lattice, mesh generators) get grown tiles (3 ms on the host at
// 160,000 vertices).
// A tile must fit its block's shared memory with the hot part of its records
// (about 3,200 vertices a tile, 460,000 in all).  Larger meshes keep the
// ordered sweeps (tl_nt = 0) but for the cascade's flow (tl_cas), which would
// have to merge an order first: with records left in L2 a tile solves about 100
// vertices/us and a hop takes 0.65 us, and the two flow sweeps of a step took
// 260 + 350 us at 655,362 vertices and 740 + 1,060 us at 2,621,442, against 380 +
// 820 us in the ordered form there (flow_needs_order).  Loading the first
// successor's record ahead made it 10 % slower: the fences wait for it.  Values, a byte of count
// and a queue slot per vertex fit for 2.7 million vertices.
// Not called for a mesh with an edge that only one of its ends lists (a vertex
// of more than twelve neighbours, of which the reference keeps the first
// twelve), nor where a vertex lists a neighbour twice: solved vertices are
// announced through the neighbour lists, once per edge.
int tiles_setup(gs_plan* p, const int32_t* nnb, const int32_t* ngb) {
    const int n = (int)p->n;
    p->tl_nt = 0;
    if (n == 0) return GS_OK;
    int dev = 0, smem_max = 0;
    GS_CUDA(cudaGetDevice(&dev));
    GS_CUDA(cudaDeviceGetAttribute(&smem_max, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    const size_t room = (size_t)std::max(smem_max - 1024, 0);   // beside the static shared memory
    const int blocks = std::max(p->sm_count - SM_SPARE, 1);
    const int64_t per = ((int64_t)n + blocks - 1) / blocks;
    const int64_t T64 = std::max<int64_t>(TILE_MIN, (per + 31) / 32 * 32);
    if (T64 > TILE_MAX || tile_smem((int)T64, 0, 0) > room) return GS_OK;
    const int T = (int)T64;
    const bool cas = tile_smem(T, 0, HOT + 8) > room;   // the cascade's flow alone
    const int nt = (n + T - 1) / T;
    std::vector<int> cuts, gcuts;
    const int* d_perm = nullptr;   // tile-major order, in scratch until the pool is there
    const int* d_loc = nullptr;
    GS_TRY(count_cuts(p, T, nt, nullptr, nullptr, cuts));
    int64_t total = 0;
    for (int c : cuts) total += c;
    const double side = sqrt((double)T) * nt;
    if (cas) {
        // consecutive ids as they are, or not at all: growing tiles of so many
        // vertices costs the host more than many steps save.  A compact patch cuts
        // about 8 sqrt(T) edges, one along a space-filling curve up to twice that,
        // the strips of a lattice's rows some 60 sqrt(T).
        if ((double)total > 24.0 * side) return GS_OK;
    } else if (nt > 1 && !(T > TILE_MIN && (double)total <= 16.0 * side)) {
        // (a curve's tiles are kept without growing others where that costs
        // milliseconds, 6 at 164,000 vertices; grown ones cut 8.0 to 8.4 sqrt(T))
        std::vector<int> perm;
        grow_tiles(n, nnb, ngb, T, nt, perm);
        GS_CUDA(cudaMemcpy(p->comp, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice));
        k_loc<<<grid_for(n, 256), 256>>>(n, p->comp, p->lab);
        GS_LAUNCH();
        GS_TRY(count_cuts(p, T, nt, p->comp, p->lab, gcuts));
        int64_t grown = 0;
        for (int c : gcuts) grown += c;
        if (total > 2 * grown) {
            cuts.swap(gcuts);
            d_perm = p->comp;
            d_loc = p->lab;
        }
    }
    const int cap = std::max(1, *std::max_element(cuts.begin(), cuts.end()));
    // (64 groups of the pollers' cut edges, 16-bit value indices)
    if (cap > 64 * POLL_LANES * POLL_EDGES || T + cap > 0xffff) return GS_OK;
    std::vector<int> c0(nt + 1, 0);
    for (int t = 0; t < nt; t++) c0[t + 1] = c0[t] + cuts[t];
    p->tl_T = T;
    p->tl_cap = cap;
    p->tl_np = p->W <= 6 ? 6 : p->W <= 8 ? 8 : 12;
    // the sweep kernels must be resident, one block per SM
    int ok = 1;
    by_width(p, [&](auto w) -> int {
        constexpr int NP = decltype(w)::value;
        p->tl_keep = cas ? 0 : tile_smem(T, cap, Rec<NP>::BYTES) <= room ? 2 : 1;
        p->tl_smem = tile_smem(T, cap, p->tl_keep == 2 ? Rec<NP>::BYTES : p->tl_keep == 1 ? HOT + 8 : 0);
        if (p->tl_smem > room) ok = 0;
        for (int div = 0; div < (cas ? 1 : 2) && ok; div++) {
            const void* k = sweep_kernel<NP>(div != 0, p->tl_keep);
            int o = 0;
            // (the limit is the kernel's, not the plan's: the device's own for every
            // plan, so that no thread lowers it under another's launch)
            if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)room) != cudaSuccess ||
                cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k, TS_THREADS, p->tl_smem) != cudaSuccess || o < 1)
                ok = 0;
        }
        return GS_OK;
    });
    cudaGetLastError();
    if (!ok) return GS_OK;
    // one allocation: the tile tables, the published values, the status word and
    // the records of the three graphs
    const size_t N = (size_t)n, ncut = (size_t)std::max(c0[nt], 1);
    size_t rec_bytes = 0;
    by_width(p, [&](auto w) -> int {
        rec_bytes = N * Rec<decltype(w)::value>::BYTES;
        return GS_OK;
    });
    size_t pool = 0;
    auto take = [&](size_t bytes) {
        const size_t at = pool;
        pool += (bytes + 31) / 32 * 32;
        return at;
    };
    const size_t ids = d_perm ? sizeof(int) * N : 0;
    const size_t o_status = take(sizeof(unsigned)), o_c0 = take(sizeof(int) * c0.size()),
                 o_cq = take(sizeof(unsigned) * ncut), o_cl = take(sizeof(unsigned) * ncut),
                 o_ci = take(sizeof(uint16_t) * p->W * N), o_pm = take(ids), o_lc = take(ids),
                 o_xb = take(2 * N * sizeof(double)), o_g = pool;
    const size_t g_bytes = rec_bytes + (N * sizeof(uint16_t) + 31) / 32 * 32;
    if (cudaMalloc((void**)&p->tl_pool, o_g + (cas ? 1 : TG_N) * g_bytes) != cudaSuccess) {
        p->tl_pool = nullptr;
        cudaGetLastError();
        return GS_OK;   // no room for the records: the ordered sweeps need none
    }
    p->tl_status = (unsigned*)(p->tl_pool + o_status);
    p->tl_cut0 = (int*)(p->tl_pool + o_c0);
    p->tl_cut_q = (unsigned*)(p->tl_pool + o_cq);
    p->tl_cut_l = (unsigned*)(p->tl_pool + o_cl);
    p->tl_cut_idx = (uint16_t*)(p->tl_pool + o_ci);
    p->tl_perm = d_perm ? (int*)(p->tl_pool + o_pm) : nullptr;
    p->tl_loc = d_perm ? (int*)(p->tl_pool + o_lc) : nullptr;
    p->tl_xb = (double*)(p->tl_pool + o_xb);
    GS_CUDA(cudaMemset(p->tl_status, 0, sizeof(unsigned)));
    GS_CUDA(cudaMemcpy(p->tl_cut0, c0.data(), sizeof(int) * c0.size(), cudaMemcpyHostToDevice));
    if (d_perm) {
        GS_CUDA(cudaMemcpy(p->tl_perm, d_perm, ids, cudaMemcpyDeviceToDevice));
        GS_CUDA(cudaMemcpy(p->tl_loc, d_loc, ids, cudaMemcpyDeviceToDevice));
    }
    k_cuts<true><<<nt, CUT_THREADS>>>(n, T, p->tl_perm, p->tl_loc, p->nbr, p->nnb, nullptr, p->tl_cut0, p->tl_cut_q,
                                      p->tl_cut_l, p->tl_cut_idx);
    GS_LAUNCH();
    GS_CUDA(cudaDeviceSynchronize());
    for (int g = 0; g < TG_N; g++) {
        if (cas && g != TG_CASCADE) continue;
        p->tl_graph[g].rec = p->tl_pool + o_g + (cas ? 0 : g) * g_bytes;
        p->tl_graph[g].pm = (uint16_t*)(p->tl_graph[g].rec + rec_bytes);
    }
    p->tl_dirty = 1;
    p->tl_nt = cas ? 0 : nt;
    p->tl_cas = cas ? nt : 0;
    return GS_OK;
}

void tiles_free(gs_plan* p) {
    if (p->tl_pool) cudaFree(p->tl_pool);
    p->tl_pool = nullptr;
    p->tl_nt = p->tl_cas = 0;
}

static BuildArgs build_args(gs_plan* p, const TileGraph& g) {
    // solves that a call queued and did not see the end of (it stopped on an
    // error, or its stream was capturing and nothing ran) left the halves of
    // tl_xb in a state that is not known
    if (p->tl_open) p->tl_dirty = 1;
    p->tl_open = 0;
    BuildArgs a = {};
    a.n = (int)p->n;
    a.T = p->tl_T;
    a.R = p->R;
    a.perm = p->tl_perm;
    a.loc = p->tl_loc;
    a.nbr = p->nbr;
    a.nnb = p->nnb;
    a.rev = p->rev;
    a.sorder = p->sorder;
    a.cut_idx = p->tl_cut_idx;
    a.rec = g.rec;
    a.pm = g.pm;
    return a;
}

int tile_build(gs_plan* p, int which, bool down, bool div, const int* rcv, const double* co, const int8_t* rslot,
               const double* z, const int* pdir, const uint16_t* ref, int* bad) {
    const TileGraph& g = p->tl_graph[which];
    BuildArgs a = build_args(p, g);
    a.rcv = rcv;
    a.rslot = rslot;
    a.co = co;
    a.z = z;
    a.pdir = pdir;
    a.ref = ref;
    a.div = div ? 1 : 0;
    a.bad = bad;
    by_width(p, [&](auto w) -> int {
        constexpr int NP = decltype(w)::value;
        if (down) launch(p, k_build_down<NP>, grid_for(a.n, 128), 128, a);
        else launch(p, k_build_up<NP>, grid_for(a.n, 128), 128, a);
        return GS_OK;
    });
    GS_LAUNCH();
    return GS_OK;
}

int tile_build_marine(gs_plan* p, int which, const unsigned short* cand, const double* w, const double* z, int* bad) {
    const TileGraph& g = p->tl_graph[which];
    BuildArgs a = build_args(p, g);
    a.co = w;
    a.z = z;
    a.bad = bad;
    by_width(p, [&](auto np) -> int {
        launch(p, k_build_marine<decltype(np)::value>, grid_for(a.n, 128), 128, a, cand);
        return GS_OK;
    });
    GS_LAUNCH();
    return GS_OK;
}

int tile_solve(gs_plan* p, int which, bool div, const double* b, double* x, const int* skip) {
    const int n = (int)p->n;
    if (p->tl_dirty) {
        // first solve of the plan, or the one after a solve that stopped early
        launch(p, k_fill_pending, grid_for(n, 256), 256, n, p->tl_xb, p->tl_xb + n);
        GS_CUDA(cudaMemsetAsync(p->tl_status, 0, sizeof(unsigned), p->stream));
        GS_LAUNCH();
        p->tl_dirty = 0;
    }
    const TileGraph& g = p->tl_graph[which];
    SweepArgs a;
    a.n = n;
    a.T = p->tl_T;
    a.perm = p->tl_perm;
    a.rec = g.rec;
    a.pm = g.pm;
    a.b = b;
    a.x = x;
    a.xb = p->tl_xb + (size_t)p->tl_par * n;
    a.xb_next = p->tl_xb + (size_t)(1 - p->tl_par) * n;
    a.cut0 = p->tl_cut0;
    a.cut_q = p->tl_cut_q;
    a.cut_l = p->tl_cut_l;
    a.cut_cap = p->tl_cap;
    a.status = p->tl_status;
    a.skip = skip;
    a.budget_ns = p->sweep_budget_ns;
    p->tl_par = 1 - p->tl_par;
    p->tl_open = 1;
    return by_width(p, [&](auto w) -> int {
        constexpr int NP = decltype(w)::value;
        const void* fn = sweep_kernel<NP>(div, p->tl_keep);
        void* args[] = {(void*)&a};
        cudaEvent_t stop = nullptr;
        if (p->profiling) prof_begin(p, fn, &stop);
        // the blocks wait on one another: a cooperative launch keeps them all resident
        GS_CUDA(cudaLaunchCooperativeKernel(fn, std::max(p->tl_nt, p->tl_cas), TS_THREADS, args, p->tl_smem, p->stream));
        if (stop) cudaEventRecord(stop, p->stream);
        p->launches++;
        return GS_OK;
    });
}

int tile_status_async(gs_plan* p, int* host) {
    GS_CUDA(cudaMemcpyAsync(host, p->tl_status, sizeof(int), cudaMemcpyDeviceToHost, p->stream));
    return GS_OK;
}

int tile_status_check(gs_plan* p, int st, const char* what) {
    p->tl_open = 0;
    if (st == 0) return GS_OK;
    p->tl_dirty = 1;   // values of the stopped solve are published: reset before the next
    if ((unsigned)st != TILE_REJECTED) set_error(st, what);
    return st;
}

int tile_status(gs_plan* p, const char* what) {
    int st = 0;
    GS_TRY(tile_status_async(p, &st));
    GS_CUDA(cudaStreamSynchronize(p->stream));
    return tile_status_check(p, st, what);
}

}  // namespace gs
