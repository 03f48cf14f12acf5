// Multiple-flow-direction receivers and the flow-direction post-processing.
//
// k_mfd_receivers restates fortran/functions.F90:1544-1671 (mfdreceivers):
// one thread per vertex over the slot-major neighbour arrays, adaptive
// exponent, gid-keyed 1e-15 tie perturbation, top-R selection.  The top-R
// order for distinct slopes is the descending order the reference's quicksort
// produces; when two candidate slopes are exactly equal the reference
// quicksort/split pair (functions.F90:683-762) is replayed literally so tie
// order matches.  As in the reference, the distance of output receiver o is
// the edge length of candidate kk-1-o in candidate order (the sort permutes
// slopes and ids but not distances).
//
// k_flow_direction_post restates flowplex.py:480-540: flat routing on filled
// pits when down=True, self-sink outlets on flat models, the lsink mask.
#include <type_traits>

#include "gs_plan.cuh"

namespace gs {

// --- literal replay of the reference quicksort on <=12 candidates ----------
__device__ void dev_split(double* a, int low, int high, int* mid, int* ix) {
    int left = low, right = high;
    double pivot = a[low - 1];
    int ipivot = ix[low - 1];
    for (;;) {
        if (left >= right) break;
        for (;;) {
            if (left >= right || a[right - 1] < pivot) break;
            right = right - 1;
        }
        for (;;) {
            if (left > 12) break;
            if (a[left - 1] > pivot) break;
            left = left + 1;
        }
        if (left < right) {
            double sw = a[left - 1]; a[left - 1] = a[right - 1]; a[right - 1] = sw;
            int is = ix[left - 1]; ix[left - 1] = ix[right - 1]; ix[right - 1] = is;
        }
    }
    a[low - 1] = a[right - 1];
    a[right - 1] = pivot;
    *mid = right;
    ix[low - 1] = ix[right - 1];
    ix[right - 1] = ipivot;
}

__device__ void dev_quicksort(double* a, int first, int last, int* ix) {
    // explicit stack replaying the recursion order (left part first)
    int stf[32], stl[32];
    int sp = 0;
    stf[sp] = first; stl[sp] = last; sp++;
    while (sp > 0) {
        sp--;
        int f = stf[sp], l = stl[sp];
        if (f < l) {
            int mid;
            dev_split(a, f, l, &mid, ix);
            // recursion: quicksort(first, mid-1) then quicksort(mid+1, last)
            stf[sp] = mid + 1; stl[sp] = l; sp++;
            stf[sp] = f; stl[sp] = mid - 1; sp++;
        }
    }
}

// One vertex of mfdreceivers with its candidates in arrays: any R, and the
// literal quicksort replay when candidate slopes tie exactly.  Not inlined:
// it is the only code here that needs a stack frame, and the register form
// below calls it for tied vertices only.
__device__ __noinline__ void mfd_vertex_general(int k, int n, int R, double expo, const double* __restrict__ elev,
                                                double sl, const int* __restrict__ gid, const int* __restrict__ nbr,
                                                const double* __restrict__ elen, const int8_t* __restrict__ nnb,
                                                int* __restrict__ rcv, double* __restrict__ dist,
                                                double* __restrict__ wgt, int8_t* __restrict__ rslot) {
    const double hk = elev[k];
    for (int o = 0; o < R; o++) {
        rcv[(size_t)o * n + k] = k;
        dist[(size_t)o * n + k] = 0.0;
        wgt[(size_t)o * n + k] = 0.0;
        if (rslot) rslot[(size_t)o * n + k] = -1;
    }
    if (hk <= sl) return;
    const int deg = nnb[k];
    double e = 0.0;
    for (int s = 0; s < deg; s++) {
        int nb = nbr[(size_t)s * n + k];
        double L = elen[(size_t)s * n + k];
        if (nb >= 0 && L > 0.0) {
            double val = (hk - elev[nb]) / L;
            e = (val > e) ? val : e;
        }
    }
    double fexp;
    if (e > 0) {
        double me = (e < 1.0) ? e : 1.0;
        fexp = 5.0 * me + expo;
    } else {
        fexp = 1.0;
    }
    const bool fexp_int = (fexp == floor(fexp));
    double slp[12], dst[12];
    int cid[12], cs[12];
    int kk = 0;
    for (int s = 0; s < deg; s++) {
        int nb = nbr[(size_t)s * n + k];
        double L = elen[(size_t)s * n + k];
        if (nb >= 0 && L > 0.0) {
            double d = hk - elev[nb];
            double val;
            if (d > 0.0) val = pow(d, fexp) / L;
            else if (d == 0.0) val = 0.0;
            else val = fexp_int ? pow(d, fexp) / L : -1.0;   // non-integer power of a
                                                             // negative base is NaN: no receiver
            if (val > 0.0) {
                slp[kk] = val * (1.0 - 1.0e-15 * (double)(gid ? gid[nb] : nb));
                cid[kk] = nb;
                cs[kk] = s;
                dst[kk] = L;
                kk++;
            }
        }
    }
    if (kk == 0) return;
    if (kk <= R) {
        double val = 0.0;
        for (int p = 0; p < kk; p++) {
            rcv[(size_t)p * n + k] = cid[p];
            dist[(size_t)p * n + k] = dst[p];
            if (rslot) rslot[(size_t)p * n + k] = (int8_t)cs[p];
            val = val + slp[p];
        }
        for (int p = 0; p < kk; p++) wgt[(size_t)p * n + k] = slp[p] / val;
        return;
    }
    // kk > R: top-R in descending slope order
    int top[12];
    bool tie = false;
    for (int a = 0; a < kk && !tie; a++)
        for (int b = a + 1; b < kk; b++)
            if (slp[a] == slp[b]) { tie = true; break; }
    if (!tie) {
        unsigned used = 0;
        for (int o = 0; o < R; o++) {
            int best = -1;
            for (int a = 0; a < kk; a++) {
                if (used & (1u << a)) continue;
                if (best < 0 || slp[a] > slp[best]) best = a;
            }
            used |= 1u << best;
            top[o] = best;
        }
    } else {
        double sa[12];
        int ix[12];
        for (int a = 0; a < 12; a++) { sa[a] = (a < kk) ? slp[a] : 0.0; ix[a] = a; }
        dev_quicksort(sa, 1, kk, ix);
        for (int o = 0; o < R; o++) top[o] = ix[kk - 1 - o];
    }
    double val = 0.0;
    double slope[12];
    for (int o = 0; o < R; o++) {
        int a = top[o];
        slope[o] = slp[a];
        rcv[(size_t)o * n + k] = cid[a];
        dist[(size_t)o * n + k] = dst[kk - 1 - o];
        if (rslot) rslot[(size_t)o * n + k] = (int8_t)cs[a];
        val = val + slp[a];
    }
    for (int o = 0; o < R; o++) wgt[(size_t)o * n + k] = slope[o] / val;
}

__global__ void k_mfd_receivers(int n, int W, int R, double expo, const double* __restrict__ elev,
                                double sl, const int* __restrict__ gid, const int* __restrict__ nbr,
                                const double* __restrict__ elen, const int8_t* __restrict__ nnb,
                                int* __restrict__ rcv, double* __restrict__ dist,
                                double* __restrict__ wgt, int8_t* __restrict__ rslot) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k < n) mfd_vertex_general(k, n, R, expo, elev, sl, gid, nbr, elen, nnb, rcv, dist, wgt, rslot);
}

// What k_flow_direction_post does to the receivers of the unfilled surface, in
// the kernel that finds them: outlets of flat models drain to themselves (flat),
// and the masks when they are asked for (lsink).
struct DirPost {
    const uint8_t* flat = nullptr;      // outlet flags, null: none drain to themselves
    const uint8_t* outlet = nullptr;
    const double* lfill = nullptr;
    uint8_t* lsink = nullptr;
    uint8_t* sea = nullptr;
};
__device__ __forceinline__ void dir_masks(const DirPost& post, int k, double sl, bool none) {
    if (!post.lsink) return;
    const bool is_sea = post.lfill[k] <= sl;
    post.lsink[k] = (none && !post.outlet[k] && !is_sea) ? 1 : 0;
    post.sea[k] = is_sea ? 1 : 0;
}

// neighbours c (-1: none), edge lengths l and drops d of a vertex, all gathers
// in flight together, and the exponent from its steepest gradient
template <int NP>
__device__ __forceinline__ void mfd_gather(int k, int n, double hk, const double* __restrict__ elev,
                                           const int* __restrict__ nbr, const double* __restrict__ elen,
                                           const int8_t* __restrict__ nnb, double expo, int (&c)[NP], double (&l)[NP],
                                           double (&d)[NP], double& fexp) {
    const int deg = nnb[k];
#pragma unroll
    for (int s = 0; s < NP; s++) {
        c[s] = s < deg ? nbr[(size_t)s * n + k] : -1;
        l[s] = s < deg ? elen[(size_t)s * n + k] : 0.0;
    }
#pragma unroll
    for (int s = 0; s < NP; s++) d[s] = c[s] >= 0 ? hk - elev[c[s]] : 0.0;
    double e = 0.0;
#pragma unroll
    for (int s = 0; s < NP; s++) {
        if (!(l[s] > 0.0)) c[s] = -1;
        if (c[s] < 0) continue;
        const double g = d[s] / l[s];
        e = (g > e) ? g : e;
    }
    fexp = e > 0 ? 5.0 * ((e < 1.0) ? e : 1.0) + expo : 1.0;
}

__device__ __forceinline__ double mfd_slope(double d, double l, double fexp, bool fexp_int) {
    if (d > 0.0) return pow(d, fexp) / l;
    if (d == 0.0) return 0.0;
    return fexp_int ? pow(d, fexp) / l : -1.0;   // non-integer power of a negative base is NaN
}

// R >= the mesh's neighbour slots: every candidate is a receiver, in slot order,
// and nothing has to be ranked.  The powers of the land vertices bound it, then
// the stores: eight directions of 655,362 vertices and their masks take 56 us,
// where the general form (arrays in local memory) and a pass for the masks took
// 73.  Six slots: 64 registers for eight blocks an SM, 4 % faster than 78.  MINB,
// the blocks an SM that the registers have to allow: see two_waves.
template <int NP, int MINB>
__global__ void __launch_bounds__(128, MINB) k_mfd_all(int n, int R, double expo, const double* __restrict__ elev,
                                                  double sl, const int* __restrict__ gid, const int* __restrict__ nbr,
                                                  const double* __restrict__ elen, const int8_t* __restrict__ nnb,
                                                  int* __restrict__ rcv, double* __restrict__ dist,
                                                  double* __restrict__ wgt, int8_t* __restrict__ rslot,
                                                  const DirPost post) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double hk = elev[k];
    int c[NP], kk = 0;
    double l[NP], x[NP], tot = 0.0;
    unsigned mask = 0u;
    if (!(hk <= sl) && !(post.flat && post.flat[k])) {
        double d[NP], fexp;
        mfd_gather<NP>(k, n, hk, elev, nbr, elen, nnb, expo, c, l, d, fexp);
        const bool fexp_int = (fexp == floor(fexp));
#pragma unroll
        for (int s = 0; s < NP; s++) {
            x[s] = 0.0;
            if (c[s] < 0) continue;
            const double val = mfd_slope(d[s], l[s], fexp, fexp_int);
            if (!(val > 0.0)) continue;
            x[s] = val * (1.0 - 1.0e-15 * (double)(gid ? gid[c[s]] : c[s]));
            tot = tot + x[s];
            mask |= 1u << s;
            kk++;
        }
    }
    double sw = 0.0;
    for (int o = 0; o < R; o++) {
        int r = k, slot = -1;
        double dd = 0.0, w = 0.0;
        if (o < kk) {
            slot = __ffs(mask) - 1;
            mask &= mask - 1u;
#pragma unroll
            for (int s = 0; s < NP; s++)
                if (s == slot) {
                    r = c[s];
                    dd = l[s];
                    w = x[s] / tot;
                }
        }
        rcv[(size_t)o * n + k] = r;
        dist[(size_t)o * n + k] = dd;
        wgt[(size_t)o * n + k] = w;
        sw = sw + w;
        if (rslot) rslot[(size_t)o * n + k] = (int8_t)slot;
    }
    dir_masks(post, k, sl, sw == 0.0);
}

// Register form for R = RM < the neighbour slots NP: every candidate slope is
// formed and summed in slot order, and the RM + 1 steepest are kept by
// insertion.  Without exact ties among the kept candidates the descending order
// is the one the reference quicksort leaves, so the result is bit-identical to
// the general form; a vertex whose new candidate equals a kept one goes to
// mfd_vertex_general (literal replay).  gid == nullptr means the identity
// numbering (one partition).  The gathers of a vertex are in flight together: in
// a loop over its slots, and once more in the second pass over them, three
// directions took 22 us on 20,000 vertices and 125 on 2.6 million, now 18 and 112.
// NP = 0 is that loop: 64 registers whatever the slots, for the meshes that
// two_waves sends here.
template <int RM, int NP>
__global__ void __launch_bounds__(128, NP == 6 || NP == 0 ? 8 : 1) k_mfd_receivers_r(int n, double expo, const double* __restrict__ elev,
                                                          double sl, const int* __restrict__ gid,
                                                          const int* __restrict__ nbr, const double* __restrict__ elen,
                                                          const int8_t* __restrict__ nnb, int* __restrict__ rcv,
                                                          double* __restrict__ dist, double* __restrict__ wgt,
                                                          int8_t* __restrict__ rslot, const DirPost post) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const double hk = elev[k];
    if (!(hk > sl) || (post.flat && post.flat[k])) {
#pragma unroll
        for (int o = 0; o < RM; o++) {
            rcv[(size_t)o * n + k] = k;
            dist[(size_t)o * n + k] = 0.0;
            wgt[(size_t)o * n + k] = 0.0;
            if (rslot) rslot[(size_t)o * n + k] = -1;
        }
        dir_masks(post, k, sl, true);
        return;
    }
    const int deg = nnb[k];
    constexpr int NG = NP ? NP : 1;
    int c[NG];
    double l[NG], d[NG], fexp;
    if constexpr (NP != 0) mfd_gather<NP>(k, n, hk, elev, nbr, elen, nnb, expo, c, l, d, fexp);
    else {
        double e = 0.0;
        for (int s = 0; s < deg; s++) {
            const int j = nbr[(size_t)s * n + k];
            const double ls = elen[(size_t)s * n + k];
            if (j < 0 || !(ls > 0.0)) continue;
            const double g = (hk - elev[j]) / ls;
            e = (g > e) ? g : e;
        }
        fexp = e > 0 ? 5.0 * ((e < 1.0) ? e : 1.0) + expo : 1.0;
    }
    const bool fexp_int = (fexp == floor(fexp));
    // candidates: slope (scaled by the global-id tie-break), kept descending;
    // strict > keeps the earlier slot ahead of an equal value
    double tv[RM + 1];
    int ts[RM + 1], tid[RM + 1];
#pragma unroll
    for (int j = 0; j <= RM; j++) {
        tv[j] = -1.0;
        ts[j] = -1;
        tid[j] = -1;
    }
    unsigned mask = 0u;
    int kk = 0;
    double tot_all = 0.0;
    bool tie = false;
    auto take = [&](int s, int j, double ls, double ds) {
        const double val = mfd_slope(ds, ls, fexp, fexp_int);
        if (!(val > 0.0)) return;
        double x = val * (1.0 - 1.0e-15 * (double)(gid ? gid[j] : j));
        mask |= 1u << s;
        kk++;
        tot_all = tot_all + x;
        int xs = s, xi = j;
#pragma unroll
        for (int q = 0; q <= RM; q++) tie |= (x == tv[q]);
#pragma unroll
        for (int q = 0; q <= RM; q++) {
            if (x > tv[q]) {
                const double t = tv[q];
                const int a = ts[q], b = tid[q];
                tv[q] = x;
                ts[q] = xs;
                tid[q] = xi;
                x = t;
                xs = a;
                xi = b;
            }
        }
    };
    if constexpr (NP != 0) {
#pragma unroll
        for (int s = 0; s < NP; s++)
            if (c[s] >= 0) take(s, c[s], l[s], d[s]);
    } else {
        for (int s = 0; s < deg; s++) {
            const int j = nbr[(size_t)s * n + k];
            const double ls = elen[(size_t)s * n + k];
            if (j >= 0 && ls > 0.0) take(s, j, ls, hk - elev[j]);
        }
    }
    double sw = 0.0;
    if (kk <= RM) {
        // every candidate is kept: receivers in slot order, weights over the
        // sum of all candidates taken in slot order
#pragma unroll
        for (int j = 0; j < RM; j++) {
            if (j < kk) {
                int o = 0;
#pragma unroll
                for (int i = 0; i < RM; i++) o += (i < kk && ts[i] < ts[j]) ? 1 : 0;
                rcv[(size_t)o * n + k] = tid[j];
                dist[(size_t)o * n + k] = elen[(size_t)ts[j] * n + k];
                const double w = tv[j] / tot_all;
                sw = sw + w;
                wgt[(size_t)o * n + k] = w;
                if (rslot) rslot[(size_t)o * n + k] = (int8_t)ts[j];
            } else {
                rcv[(size_t)j * n + k] = k;
                dist[(size_t)j * n + k] = 0.0;
                wgt[(size_t)j * n + k] = 0.0;
                if (rslot) rslot[(size_t)j * n + k] = -1;
            }
        }
        dir_masks(post, k, sl, sw == 0.0);
        return;
    }
    if (tie) {
        mfd_vertex_general(k, n, RM, expo, elev, sl, gid, nbr, elen, nnb, rcv, dist, wgt, rslot);
        if (post.lsink)
            for (int o = 0; o < RM; o++) sw = sw + wgt[(size_t)o * n + k];
        dir_masks(post, k, sl, sw == 0.0);
        return;
    }
    // reference quirk: receiver o takes the edge length of candidate kk-1-o
    // in slot order (the sort permutes slopes and ids, not distances), i.e.
    // of the (o+1)-th highest candidate slot
    double tot = 0.0;
#pragma unroll
    for (int o = 0; o < RM; o++) tot = tot + tv[o];
    unsigned m = mask;
#pragma unroll
    for (int o = 0; o < RM; o++) {
        const int hs = 31 - __clz(m);
        m &= ~(1u << hs);
        rcv[(size_t)o * n + k] = tid[o];
        dist[(size_t)o * n + k] = elen[(size_t)hs * n + k];
        const double w = tv[o] / tot;
        sw = sw + w;
        wgt[(size_t)o * n + k] = w;
        if (rslot) rslot[(size_t)o * n + k] = (int8_t)ts[o];
    }
    dir_masks(post, k, sl, sw == 0.0);
}

__global__ void k_flow_direction_post(int n, int W, int R, int flat, const double* __restrict__ h,
                                      int down, const double* __restrict__ lfill,
                                      const int* __restrict__ pit, const int* __restrict__ fdir,
                                      double sl, const uint8_t* __restrict__ outlet,
                                      const int* __restrict__ nbr, int* rcv, double* dist,
                                      double* wgt, int8_t* rslot, uint8_t* lsink, uint8_t* sea) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (down) {
        double sw = 0.0;
        for (int k = 0; k < R; k++) sw = sw + wgt[(size_t)k * n + i];
        if (h[i] == lfill[i] && pit[i] > -1 && fdir[i] > -1 && sw == 0.0) {
            int f = fdir[i];
            int slot = -1;
            if (f != i)
                for (int s = 0; s < W; s++)
                    if (nbr[(size_t)s * n + i] == f) { slot = s; break; }
            for (int k = 0; k < R; k++) {
                rcv[(size_t)k * n + i] = (k == 0) ? f : i;
                wgt[(size_t)k * n + i] = (k == 0) ? 1.0 : 0.0;
                rslot[(size_t)k * n + i] = (k == 0) ? (int8_t)slot : (int8_t)-1;
            }
        }
    }
    if (flat && outlet[i]) {
        for (int k = 0; k < R; k++) {
            rcv[(size_t)k * n + i] = i;
            dist[(size_t)k * n + i] = 0.0;
            wgt[(size_t)k * n + i] = 0.0;
            rslot[(size_t)k * n + i] = -1;
        }
    }
    if (!lsink) return;  // graph only: the masks are set by k_sink_mask once lFill exists
    const bool is_sea = lfill[i] <= sl;
    double sw = 0.0;
    for (int k = 0; k < R; k++) sw = sw + wgt[(size_t)k * n + i];
    lsink[i] = (sw == 0.0 && !outlet[i] && !is_sea) ? 1 : 0;
    sea[i] = is_sea ? 1 : 0;
}

// seaID (lFill <= sea level, flowplex.py:493) as a mask
__global__ void k_sea_mask(int n, const double* __restrict__ lfill, double sl, uint8_t* sea) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) sea[i] = lfill[i] <= sl ? 1 : 0;
}

// lsink (flowplex.py:531-540) from the weights and a precomputed sea mask
__global__ void k_sink_mask(int n, int R, const double* __restrict__ wgt, const uint8_t* __restrict__ outlet,
                            const uint8_t* __restrict__ sea, uint8_t* lsink) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double sw = 0.0;
    for (int k = 0; k < R; k++) sw = sw + wgt[(size_t)k * n + i];
    lsink[i] = (sw == 0.0 && !outlet[i] && !sea[i]) ? 1 : 0;
}

int sea_mask(gs_plan* p, const double* lfill, double sl, uint8_t* sea) {
    if (p->n == 0) return GS_OK;
    launch(p, k_sea_mask, grid_for(p->n, 256), 256, (int)p->n, lfill, sl, sea);
    GS_LAUNCH();
    return GS_OK;
}

int sink_mask(gs_plan* p, const double* wgt, const uint8_t* sea, uint8_t* lsink) {
    if (p->n == 0) return GS_OK;
    launch(p, k_sink_mask, grid_for(p->n, 256), 256, (int)p->n, p->R, wgt, (const uint8_t*)p->outlet, sea,
           lsink);
    GS_LAUNCH();
    return GS_OK;
}

// More vertices than two waves of a form with `blocks` blocks of 128 an SM.  With
// up to two, the unrolled forms gain from their gathers in flight; with more, the
// blocks of 94 to 118 registers for 8 or 12 slots (and the spills of four
// directions at 6) cost more than that gives, and 64 registers are faster.  B200,
// us for the receivers and masks, lattices of 8 slots, unrolled and 64 registers:
// three directions 14 and 18 at 20,000 vertices, 33.0 and 34.3 at 160,000, 73 and 65
// at 400,000, 170 and 140 at 900,000; four 14 and 18, 41 and 37, 84 and 70, 209 and
// 151; eight (all kept) 15.4 and 16.5, 43 and 37, 96 and 80, 194 and 163.  Spheres,
// four directions: 30.5 and 30.2 at 163,842, 77 and 70 at 655,362.
static bool two_waves(const gs_plan* p, int blocks) { return p->n > (int64_t)2 * p->sm_count * blocks * 128; }

// `post` runs in the receivers' kernel where *fused comes back true
static int receivers_post(gs_plan* p, int nrcv, double exp, const double* elev, double sl, const int* gid, int* rcv,
                          double* dist, double* wgt, int8_t* rslot, const DirPost& post, bool* fused) {
    if (nrcv < 1 || nrcv > 12) {
        set_error(GS_EINVAL, "mfdreceivers: nrcv must be in 1..12");
        return GS_EINVAL;
    }
    *fused = nrcv >= p->W || nrcv <= 4;
    if (p->n == 0) return GS_OK;
    const int* g = gid == p->gid ? nullptr : gid;   // the plan's own numbering is the identity
    const int G = grid_for(p->n, 128), n = (int)p->n;
    // slots of the unrolled forms (6: spheres, 8: jittered lattices, 12)
    auto width = [&](auto f) {
        if (p->W <= 6) f(std::integral_constant<int, 6>{});
        else if (p->W <= 8) f(std::integral_constant<int, 8>{});
        else f(std::integral_constant<int, 12>{});
    };
    auto ranked = [&](auto w) {
        constexpr int NP = decltype(w)::value;
        launch(p, nrcv == 1 ? k_mfd_receivers_r<1, NP> : nrcv == 2 ? k_mfd_receivers_r<2, NP>
                  : nrcv == 3 ? k_mfd_receivers_r<3, NP> : k_mfd_receivers_r<4, NP>,
               G, 128, n, exp, elev, sl, g, p->nbr, p->elen, p->nnb, rcv, dist, wgt, rslot, post);
    };
    if (nrcv >= p->W)
        width([&](auto w) {
            constexpr int NP = decltype(w)::value;
            constexpr int FEW = NP == 6 ? 8 : 1, MANY = NP == 12 ? 6 : 8;
            launch(p, two_waves(p, 4) ? k_mfd_all<NP, MANY> : k_mfd_all<NP, FEW>, G, 128, n, nrcv, exp, elev, sl, g,
                   p->nbr, p->elen, p->nnb, rcv, dist, wgt, rslot, post);
        });
    else if (nrcv <= 4) {
        const bool loop = p->W <= 6 ? nrcv == 4 && two_waves(p, 8) : two_waves(p, p->W <= 8 && nrcv <= 3 ? 5 : 4);
        if (loop) ranked(std::integral_constant<int, 0>{});
        else width(ranked);
    } else
        launch(p, k_mfd_receivers, G, 128, n, p->W, nrcv, exp, elev, sl, g, p->nbr, p->elen, p->nnb, rcv, dist, wgt,
               rslot);
    GS_LAUNCH();
    return GS_OK;
}

int receivers(gs_plan* p, int nrcv, double exp, const double* elev, double sl, const int* gid,
              int* rcv, double* dist, double* wgt, int8_t* rslot) {
    bool fused;
    return receivers_post(p, nrcv, exp, elev, sl, gid, rcv, dist, wgt, rslot, DirPost{}, &fused);
}

int flow_direction(gs_plan* p, const double* h, bool down, const double* lfill, const int* pit_ids,
                   const int* flat_dirs, double sealevel, int* rcv, double* dist, double* wgt,
                   int8_t* rslot, uint8_t* lsink, uint8_t* sea) {
    DirPost post;
    if (!down) post = DirPost{p->flat ? p->outlet : nullptr, p->outlet, lfill, lsink, sea};
    bool fused = false;
    GS_TRY(receivers_post(p, p->R, 1.1, h, sealevel, p->gid, rcv, dist, wgt, rslot, post, &fused));
    if (fused && !down) return GS_OK;
    return flow_direction_post(p, h, down, lfill, pit_ids, flat_dirs, sealevel, rcv, dist, wgt, rslot, lsink, sea);
}

int flow_direction_post(gs_plan* p, const double* h, bool down, const double* lfill, const int* pit_ids,
                        const int* flat_dirs, double sealevel, int* rcv, double* dist, double* wgt,
                        int8_t* rslot, uint8_t* lsink, uint8_t* sea) {
    if (p->n == 0) return GS_OK;
    launch(p, k_flow_direction_post, grid_for(p->n, 256), 256, (int)p->n, p->W, p->R, p->flat, h,
           down ? 1 : 0, lfill, pit_ids, flat_dirs, sealevel, p->outlet, p->nbr, rcv, dist, wgt,
           rslot, lsink, sea);
    GS_LAUNCH();
    return GS_OK;
}

}  // namespace gs

namespace gs {

// Reverse of the slope-weight computation of k_mfd_receivers with the
// receiver choice held fixed (the slots in rslot): given gw[o][k] = dJ/dw_ok,
// writes dJ/dz_k to gself[k] and dJ/dz of the neighbour in slot s to
// gnb[s][k].  The weights are w_o = slp_o / sum(slp), slp_o = (z_k - z_o)^f /
// L_o (1 - 1e-15 gid_o), and the adaptive exponent f = 5 min(e, 1) + expo
// with e the steepest descent (z_k - z_a) / L_a.  Cells without MFD receivers
// (sea, outlets, flat-routed cells) carry no derivative.
__global__ void k_mfd_weights_adj(int n, int W, int R, double expo, const double* __restrict__ z, double sl,
                                  const int* __restrict__ gid, const int* __restrict__ nbr,
                                  const double* __restrict__ elen, const int8_t* __restrict__ nnb,
                                  const int8_t* __restrict__ rslot, const double* __restrict__ gw,
                                  double* gself, double* gnb) {
    int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    for (int s = 0; s < W; s++) gnb[(size_t)s * n + k] = 0.0;
    gself[k] = 0.0;
    const double hk = z[k];
    if (hk <= sl) return;
    int so[MAXR];
    int nsel = 0;
    for (int o = 0; o < R; o++) {
        int s = rslot[(size_t)o * n + k];
        so[o] = s;
        if (s >= 0) nsel++;
    }
    if (nsel == 0) return;
    const int deg = nnb[k];
    double e = 0.0;
    int a = -1;
    for (int s = 0; s < deg; s++) {
        int nb = nbr[(size_t)s * n + k];
        double L = elen[(size_t)s * n + k];
        if (nb >= 0 && L > 0.0) {
            double val = (hk - z[nb]) / L;
            if (val > e) { e = val; a = s; }
        }
    }
    double fexp, dfe = 0.0;
    if (e > 0) {
        double me = (e < 1.0) ? e : 1.0;
        fexp = 5.0 * me + expo;
        if (e < 1.0) dfe = 5.0;
    } else {
        fexp = 1.0;
    }
    double slp[MAXR], dval[MAXR], fval[MAXR], gfac[MAXR];
    double V = 0.0;
    for (int o = 0; o < R; o++) {
        slp[o] = 0.0;
        int s = so[o];
        if (s < 0) continue;
        int nb = nbr[(size_t)s * n + k];
        double L = elen[(size_t)s * n + k];
        double d = hk - z[nb];
        if (!(d > 0.0) || !(L > 0.0)) return;   // not an MFD receiver (flat routing): no derivative
        double val = pow(d, fexp) / L;
        gfac[o] = 1.0 - 1.0e-15 * (double)gid[nb];
        slp[o] = val * gfac[o];
        dval[o] = fexp * pow(d, fexp - 1.0) / L;
        fval[o] = val * log(d);
        V = V + slp[o];
    }
    if (!(V > 0.0)) return;
    double sw = 0.0;
    for (int o = 0; o < R; o++)
        if (so[o] >= 0) sw += gw[(size_t)o * n + k] * (slp[o] / V);
    double gs_ = 0.0, gf = 0.0;
    for (int o = 0; o < R; o++) {
        int s = so[o];
        if (s < 0) continue;
        double gslp = (gw[(size_t)o * n + k] - sw) / V;
        double gval = gslp * gfac[o];
        double gd = gval * dval[o];
        gf += gval * fval[o];
        gs_ += gd;
        gnb[(size_t)s * n + k] -= gd;
    }
    if (dfe != 0.0 && a >= 0) {
        double La = elen[(size_t)a * n + k];
        double ge = gf * dfe / La;
        gs_ += ge;
        gnb[(size_t)a * n + k] -= ge;
    }
    gself[k] = gs_;
}

// gz[v] += gself[v] + sum over the cells k that have v as neighbour of gnb[slot of v at k][k]
__global__ void k_nb_gather(int n, const int* __restrict__ nbr, const int8_t* __restrict__ nnb,
                            const int8_t* __restrict__ rev, const double* __restrict__ gself,
                            const double* __restrict__ gnb, double* gz) {
    int v = blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= n) return;
    double acc = gself[v];
    for (int t = 0; t < nnb[v]; t++) {
        int k = nbr[(size_t)t * n + v];
        if (k < 0) continue;
        int s = rev[(size_t)t * n + v];
        if (s >= 0) acc += gnb[(size_t)s * n + k];
    }
    gz[v] += acc;
}

// dJ/dz of the surface the receivers were built on, accumulated into gz,
// from dJ/dw (gw, receiver-major [R][n]); gself/gnb are [n] / [W][n] scratch.
int receivers_adjoint(gs_plan* p, const double* z, double sl, const int8_t* rslot, const double* gw, double* gself,
                      double* gnb, double* gz) {
    const int n = (int)p->n;
    if (n == 0) return GS_OK;
    launch(p, k_mfd_weights_adj, grid_for(n, 128), 128, n, p->W, p->R, 1.1, z, sl, (const int*)p->gid,
           (const int*)p->nbr, (const double*)p->elen, (const int8_t*)p->nnb, rslot, gw, gself, gnb);
    launch(p, k_nb_gather, grid_for(n, 256), 256, n, (const int*)p->nbr, (const int8_t*)p->nnb,
           (const int8_t*)p->rev, (const double*)gself, (const double*)gnb, gz);
    GS_LAUNCH();
    return GS_OK;
}

}  // namespace gs
