// The contact query by one warp.
//
// A query is a chain of short dependent operations (cell ranges, list heads,
// list entries, the swept tests of a few neighbours), so a block answers it
// hardly faster than a warp: its barriers, and the uniform FP64 work on every
// warp, cost what its threads gain. One warp takes the neighbours through a
// queue in shared memory, 32 list entries a round of loads, and three lanes
// per swept test, one axis each. Queries beyond the scratch (long neighbour
// lists, many sphere pairs) are left to block_query; both give the same bits.
#pragma once
#include <type_traits>

#include "box.cuh"

namespace mcacg {

constexpr int kWarpCells = 128;  // cells a query visits (four per lane)
constexpr int kWarpEarly = 8;    // spheres of an aggregate whose pairs are counted before the filter too
constexpr int kWarpCands = 32;   // neighbours past the FP32 screen; sphere pairs to refine

// The cells that a query read, an axis each: x the first (periodic), y how many
// of them, plus kFineLists when they are fine cells, not Verlet cells. (One
// store for three lanes: what a round notes costs every query of it.)
constexpr int kFineLists = 1 << 16;
struct QueryLists {
    int2 axis[3];
};
struct NoQueryLists {};

// Scratch of a one-warp query: up to Queue aggregates listed and Pairs sphere
// pairs screened. 'Lists' (QueryLists): the query notes the lists it read.
template <int Queue, int Pairs, class Lists = NoQueryLists>
struct WarpQueryScratch {
    static constexpr int kQueue = Queue;
    static constexpr int kPairs = Pairs;
    static constexpr bool kNotesLists = !std::is_same<Lists, NoQueryLists>::value;
    Lists lists;
    int queue[Queue];
    // neighbours past the FP32 screen, with their scan keys
    int scr_slot[kWarpCands];
    long long scr_key[kWarpCands];
    // candidates as found, and in filter order (distances as ordered keys)
    unsigned long long c_db[kWarpCands];
    long long c_key[kWarpCands];
    int c_slot[kWarpCands];
    unsigned long long s_db[kWarpCands];
    int s_slot[kWarpCands], s_off[kWarpCands], s_pre[kWarpCands];
    // sphere pairs to refine
    unsigned long long p_key[kWarpCands], p_ij[kWarpCands];
    int p_r[kWarpCands], p_si[kWarpCands], p_sj[kWarpCands];
};

__device__ __forceinline__ double shfl_d(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ int shfl_i(int v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ float shfl_f(float v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ __forceinline__ unsigned clock_lo() { return static_cast<unsigned>(clock()); }
__device__ __forceinline__ unsigned lanes_below(int lane) { return (1u << lane) - 1u; }

// x + y + z in that order, from the three lanes of a group whose first lane is g
__device__ __forceinline__ double sum3(double v, int g) {
    const double x = shfl_d(v, g), y = shfl_d(v, g + 1), z = shfl_d(v, g + 2);
    return (x + y) + z;
}

// sweep_contact_fast by three lanes, one axis each: lane g + ax of a group
// holds the two positions' coordinate ax (pa, pb); the direction's are on
// lanes 0-2 (u). The result is valid on every lane of the group. All lanes
// of the warp call it.
__device__ __forceinline__ double warp_sweep(int g, int ax, double pa, double pb, double r1, double r2, double u,
                                             double dist, double L) {
    const double dc = r1 + r2;
    const double dc2 = dc * dc;
    const double ua = shfl_d(u, ax), u1 = shfl_d(u, ax == 2 ? 0 : ax + 1), u2 = shfl_d(u, ax == 0 ? 2 : ax - 1);
    const double d0 = wrap_distance(pa - pb, L);
    const bool touch = nonneg_le(sum3(d0 * d0, g), dc2);
    const double td = ua * dist;
    const double moved = pa + td;
    const bool back = dbits(td) < 0;
    const double base = (back ? moved : pa) - dc;
    const double end = (back ? pa : moved) + dc;
    const double zone = end - base;
    bool usual = abs_lt(zone, L);
    double w = pb - base;
    if (!abs_lt(w, L)) {
        // fmod(w, L) for L <= |w| < 2 L: one exact subtraction
        usual = usual && (dbits(w) & 0x7fffffffffffffffLL) < dbits(L) + (1LL << 52);
        w = dbits(w) < 0 ? w + L : w - L;
    }
    if (neg(w)) w += L;
    const double q = w + base;
    const double d = q - pa;
    const bool outside = (dbits(d) & 0x7fffffffffffffffLL) > dbits(zone);
    const double e = moved - q;
    const double proj = sum3(d * ua, g);
    const double e2 = sum3(e * e, g);
    const double d1 = shfl_d(d, ax == 2 ? g : g + ax + 1), d2 = shfl_d(d, ax == 0 ? g + 2 : g + ax - 1);
    const double c = d1 * u2 - d2 * u1;
    const double axis = sum3(c * c, g);
    const unsigned unusual3 = (__ballot_sync(0xffffffffu, !usual) >> g) & 7u;
    const unsigned outside3 = (__ballot_sync(0xffffffffu, outside) >> g) & 7u;
    double res = CUDART_INF;
    if (unusual3 == 0u && outside3 == 0u && !neg(proj) && nonneg_le(axis, dc2) &&
        (nonneg_le(e2, dc2) || !(dkey(dist) < dkey(proj))))
        res = proj - fp64_sqrt(dc2 - axis);
    const unsigned any = __ballot_sync(0xffffffffu, unusual3 != 0u);
    if (any != 0u) {  // several periodic images can matter: the general routine
        const Vec3 p1{shfl_d(pa, g), shfl_d(pa, g + 1), shfl_d(pa, g + 2)};
        const Vec3 p2{shfl_d(pb, g), shfl_d(pb, g + 1), shfl_d(pb, g + 2)};
        const Vec3 dir{shfl_d(u, 0), shfl_d(u, 1), shfl_d(u, 2)};
        if (unusual3 != 0u) res = sweep_contact_general(p1, r1, p2, r2, dir, dist, L);
    }
    return touch ? 0.0 : res;
}

// The picked slot's record, spread over the warp: lane f holds field f of
// the FP64 table (f < 21), and lane k entry k of RecInt. Each lane keeps its
// own row's address (rec_ptr), so that a record is one load instruction
// per table: chosen among the tables by lane at each use, the loads went out
// one after another (4400 cycles a record instead of about 600).
enum RecInt : int { REC_N, REC_OFF, REC_CELL, REC_POS, REC_FINE, REC_PREV, REC_NEXT, REC_F4, REC_INTS = REC_F4 + 4 };
struct WarpRec {
    double f;
    int i;
};
struct RecRows {
    const double *f;
    const int *i;
    int shift;  // entry stride of the integer row, as a shift
};
__device__ __forceinline__ RecRows record_rows(const DevBox &b, const int *const *rec_ptr, int lane) {
    return RecRows{b.agg + size_t(lane < AGG_NFIELDS ? lane : 0) * size_t(b.nslots),
                   lane < REC_INTS ? rec_ptr[lane] : nullptr, lane >= REC_F4 ? 2 : 0};
}
__device__ __forceinline__ WarpRec load_record(const RecRows &rows, int slot) {
    WarpRec r;
    r.f = rows.f[slot];
    r.i = rows.i != nullptr ? rows.i[size_t(slot) << rows.shift] : -1;
    return r;
}
// The rows' addresses (one thread, once a launch; null: no such table).
__device__ inline void record_rows_init(const DevBox &b, const int **rec_ptr) {
    const bool fine = b.fine_div > 0;
    rec_ptr[REC_N] = b.agg_n;
    rec_ptr[REC_OFF] = b.agg_off;
    rec_ptr[REC_CELL] = b.agg_cell;
    rec_ptr[REC_POS] = b.cell_pos;
    rec_ptr[REC_FINE] = fine ? b.fine_cell : nullptr;
    rec_ptr[REC_PREV] = fine ? b.fine_prev : nullptr;
    rec_ptr[REC_NEXT] = fine ? b.fine_next : nullptr;
    for (int k = 0; k < 4; ++k) rec_ptr[REC_F4 + k] = reinterpret_cast<const int *>(b.agg_f4) + k;
}

// The contact query of slot 'src' by one warp: the same neighbours, filter,
// pairs and walk as block_query. 'dl' is the direction's component on lanes
// 0-2; 'live' lists the live slots (n_live of them) or is null. Returns false when the block has to run it (long
// lists or many pairs); then nothing was changed. Otherwise the answer and
// the work counts are in 'o'.
struct WarpAnswer {
    double distance;
    int ms, os, oslot, status;
    int scanned, cells, cands, cand_spheres, refined;
    unsigned t_scan;  // clock after the neighbourhood and the filter
};
template <class WS>
__device__ __forceinline__ bool warp_query(const DevBox &b, const DevScalars *sc, WS &W, const int *live, int n_live,
                                           int src, const WarpRec &rec, double dl, double full, WarpAnswer &o) {
    const int lane = threadIdx.x & 31;
    const unsigned all = 0xffffffffu;
    // the comparisons with the length below order its bits
    if (!is_finite(full)) return false;
    // FP32 forms of the direction (lanes 0-2), the length and the largest
    // r_max: one conversion for all of them
    const float cf = float(lane == 3 ? full : (lane == 4 ? sc->maxradius : dl));
    Sweep32 w;
    w.px = __int_as_float(shfl_i(rec.i, REC_F4));
    w.py = __int_as_float(shfl_i(rec.i, REC_F4 + 1));
    w.pz = __int_as_float(shfl_i(rec.i, REC_F4 + 2));
    const float rmax_f = __int_as_float(shfl_i(rec.i, REC_F4 + 3));
    w.ux = shfl_f(cf, 0);
    w.uy = shfl_f(cf, 1);
    w.uz = shfl_f(cf, 2);
    w.dist = shfl_f(cf, 3);
    w.cx = 0.5f * w.dist * w.ux;
    w.cy = 0.5f * w.dist * w.uy;
    w.cz = 0.5f * w.dist * w.uz;
    w.L = b.Lf;
    w.invL = b.inv_Lf;
    const float margin = b.margin_f + 1e-6f * w.dist;
    w.zmax = fmaxf(fabsf(w.dist * w.ux), fmaxf(fabsf(w.dist * w.uy), fabsf(w.dist * w.uz)));
    w.margin = margin;
    const float reach_f = rmax_f + shfl_f(cf, 4);
    // the Verlet and fine cell ranges, one axis on each of lanes 0-2
    int lo = 0, n_c = 0, flo = 0, fn = 0;
    const double x_ax = shfl_d(rec.f, AGG_X + (lane < 3 ? lane : 0));
    const double rmax = shfl_d(rec.f, AGG_RMAX);
    if (lane < 3) {
        const float pf = lane == 0 ? w.px : (lane == 1 ? w.py : w.pz);
        const float vf = w.dist * cf;
        int hi = 0;
        if (!neighborhood_axis_f32(pf, vf, reach_f, b.n_div, b.step_f, &lo, &hi))
            neighborhood_axis_call(x_ax, full * dl, rmax + sc->maxradius, b.n_div, b.L, b.inv_L, &lo, &hi);
        n_c = hi - lo + 1;
        lo = near_cell(lo, b.n_div);
        if (b.fine_div > 0) {  // widened as in block_query
            const float flof = floorf((pf - reach_f + fminf(vf, 0.f)) * b.fine_step_f - 2e-3f);
            const float fhif = floorf((pf + reach_f + fmaxf(vf, 0.f)) * b.fine_step_f + 2e-3f);
            const bool part = (fhif - flof + 1.f < float(b.fine_div)) && flof > -1e6f && fhif < 1e6f;
            flo = part ? near_cell(int(flof), b.fine_div) : 0;
            fn = part ? int(fhif - flof + 1.f) : b.fine_div;
        }
    }
    const int nd = b.n_div;
    const int rlo0 = shfl_i(lo, 0), rlo1 = shfl_i(lo, 1), rlo2 = shfl_i(lo, 2);
    const int nx = shfl_i(n_c, 0), ny = shfl_i(n_c, 1), nz = shfl_i(n_c, 2);
    bool fine = false;
    int n_scan = nx * ny * nz;
    int total = 0;  // entries in the list
    const int *list = W.queue;
    if (live != nullptr) {
        list = live;
        total = n_live;
        o.cells = 0;
    } else {
        int fn0 = 0, fn1 = 0, fn2 = 0, n_fine = 0;
        if (b.fine_div > 0) {
            fn0 = shfl_i(fn, 0);
            fn1 = shfl_i(fn, 1);
            fn2 = shfl_i(fn, 2);
            n_fine = fn0 * fn1 * fn2;
            const float alive = float(sc->n_alive);
            const float cost_fine = float(n_fine) * (1.f + alive * b.inv_fine_cells);
            const float cost_coarse = float(n_scan) * (1.f + alive * b.inv_cells);
            fine = n_fine <= kFineMaxCells && cost_fine < cost_coarse;
        }
        const int n_cells = fine ? n_fine : n_scan;
        if (n_cells > kWarpCells) return false;
        if constexpr (WS::kNotesLists) {
            if (lane < 3) W.lists.axis[lane] = fine ? make_int2(flo, fn | kFineLists) : make_int2(lo, n_c);
        }
        o.cells = n_cells;
        const int dy = fine ? fn1 : ny, dz = fine ? fn2 : nz, nf = fine ? b.fine_div : nd;
        const int l0 = fine ? shfl_i(flo, 0) : rlo0, l1 = fine ? shfl_i(flo, 1) : rlo1, l2 = fine ? shfl_i(flo, 2) : rlo2;
        // g -> (a, bb, c) by FP32 reciprocals, exact for these sizes
        const int dyz = dy * dz;
        const float inv_yz = 1.f / float(dyz), inv_z = 1.f / float(dz);
        const int *heads = fine ? b.fine_head : b.cell_n;
        int lin[kWarpCells / 32], h[kWarpCells / 32];
#pragma unroll
        for (int u = 0; u < kWarpCells / 32; ++u) {
            const int g = u * 32 + lane;
            h[u] = fine ? -1 : 0;
            lin[u] = 0;
            if (g < n_cells) {
                const int a = int((float(g) + 0.5f) * inv_yz), r = g - a * dyz;
                const int bb = int((float(r) + 0.5f) * inv_z), c = r - bb * dz;
                lin[u] = (wrap_cell(l0 + a, nf) * nf + wrap_cell(l1 + bb, nf)) * nf + wrap_cell(l2 + c, nf);
                h[u] = heads[lin[u]];
            }
        }
        if (fine) {
#pragma unroll
            for (int u = 0; u < kWarpCells / 32; ++u) {
                const unsigned m = __ballot_sync(all, h[u] >= 0);
                if (h[u] >= 0) W.queue[total + __popc(m & lanes_below(lane))] = h[u];
                total += __popc(m);
            }
        } else {
            int cnt = 0;
#pragma unroll
            for (int u = 0; u < kWarpCells / 32; ++u) cnt += h[u];
            int incl = cnt;
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const int y = __shfl_up_sync(all, incl, s);
                if (lane >= s) incl += y;
            }
            total = shfl_i(incl, 31);
            if (total > WS::kQueue) return false;
            int at = incl - cnt;
#pragma unroll
            for (int u = 0; u < kWarpCells / 32; ++u) {
                const int *items = b.cell_items + size_t(lin[u]) * b.cell_cap;
#pragma unroll 1
                for (int k = 0; k < h[u]; ++k) W.queue[at + k] = items[k];
                at += h[u];
            }
        }
        __syncwarp();
    }
    // the listed aggregates: those in the reference's neighbourhood that pass
    // the FP32 screen wait for the FP64 filter, with their scan keys
    bool found = false, sure = false;
    int n_screen = 0;
    // the shortened sweep of 'sure': both its reach and its length less by a
    // margin than the exact ones
    Sweep32 ws = w;
    ws.dist = w.dist - margin;
    for (int k0 = 0, cnt = 0; k0 < total; k0 += cnt) {
        cnt = min(32, total - k0);
        const int slot = lane < cnt ? list[k0 + lane] : -1;
        int nxt = -1, key = 0;
        float4 of = make_float4(0.f, 0.f, 0.f, 0.f);
        if (slot >= 0) {
            if (fine) nxt = b.fine_next[slot];
            key = b.agg_cell[slot];
            of = b.agg_f4[slot];
        }
        const int oa = wrap_cell((key & 1023) - rlo0, nd);
        const int ob = wrap_cell(((key >> 10) & 1023) - rlo1, nd);
        const int oc = wrap_cell((key >> 20) - rlo2, nd);
        const bool in = slot >= 0 && oa < nx && ob < ny && oc < nz;
        // the fine walk and the cells always hold the source; the live list
        // counts it when its cell is in the neighbourhood
        found = found || (slot == src && (live == nullptr || in));
        const bool pass = in && slot != src && capsule_hit(w, of.x, of.y, of.z, rmax_f + of.w + margin);
        const unsigned m = __ballot_sync(all, pass);
        if (n_screen + __popc(m) > kWarpCands) return false;
        if (m != 0u) {
            const float inner = rmax_f + of.w - 2.f * margin;
            sure = __any_sync(all, pass && ws.dist > 0.f && inner > 0.f &&
                                       w.zmax + 2.f * (rmax_f + of.w + margin) + 8.f * margin < w.L &&
                                       capsule_hit(ws, of.x, of.y, of.z, inner));
        }
        if (pass) {
            const int at = n_screen + __popc(m & lanes_below(lane));
            W.scr_slot[at] = slot;
            W.scr_key[at] = (long long)((oa * ny + ob) * nz + oc) * b.nslots + slot;
        }
        n_screen += __popc(m);
        if (fine) {
            const unsigned mn = __ballot_sync(all, nxt >= 0);
            if (total + __popc(mn) > WS::kQueue) return false;
            if (nxt >= 0) W.queue[total + __popc(mn & lanes_below(lane))] = nxt;
            total += __popc(mn);
        }
        __syncwarp();
    }
    // The screen's spheres bound the filter's: more pairs than a warp takes are
    // the block's, before the FP64 work on them.
    if (n_screen > 0) {
        const int n_src = shfl_i(rec.i, REC_N);
        if (n_src >= kWarpEarly) {
            const int near = __reduce_add_sync(all, lane < n_screen ? b.agg_n[W.scr_slot[lane]] : 0);
            if (float(n_src) * float(near) > float(WS::kPairs)) return false;
        }
    }
    o.scanned = total;
    o.status = ST_OK;
    o.distance = CUDART_INF;
    o.ms = o.os = o.oslot = -1;
    o.cands = o.cand_spheres = o.refined = 0;
    if (!__any_sync(all, found)) {
        o.status = ST_VERLET;  // "Aggregate not on the verlet list"
        o.t_scan = clock_lo();
        return true;
    }
    // the exact bounding-sphere filter, ten neighbours at a time
    const int gi = lane / 3, ax = lane - 3 * gi, g = 3 * gi;
    const double x_g = shfl_d(rec.f, AGG_X + ax);
    int nc = 0;
    if (n_screen == 1 && sure) {
        // one neighbour, within reach before the sweep's end by more than the
        // screen's margins: a candidate without the FP64 sweep, whose value
        // would only order it among others
        nc = 1;
        if (lane == 0) {
            W.c_db[0] = 0ULL;
            W.c_key[0] = W.scr_key[0];
            W.c_slot[0] = W.scr_slot[0];
        }
    }
    for (int k0 = nc > 0 ? n_screen : 0; k0 < n_screen; k0 += 10) {
        const bool act = lane < 30 && k0 + gi < n_screen;
        const int slot = act ? W.scr_slot[k0 + gi] : src;
        const double pb = A(b, AGG_X + ax, slot), r2 = A(b, AGG_RMAX, slot);
        const double db = warp_sweep(g, ax, x_g, pb, rmax, r2, dl, full, b.L);
        const bool pass = act && ax == 0 && dkey(db) < dkey(full);
        const unsigned m = __ballot_sync(all, pass);
        if (pass) {
            const int at = nc + __popc(m & lanes_below(lane));
            W.c_db[at] = dkey(db);
            W.c_key[at] = W.scr_key[k0 + gi];
            W.c_slot[at] = slot;
        }
        nc += __popc(m);
    }
    const bool filtered = !(n_screen == 1 && sure);  // the candidates' d_b are known
    __syncwarp();
    o.cands = nc;
    o.t_scan = clock_lo();
    if (nc == 0) return true;
    // candidates in the order (d_b, scan key), with their spheres' prefix
    const unsigned long long my_db = lane < nc ? W.c_db[lane] : ~0ULL;
    const long long my_key = lane < nc ? W.c_key[lane] : 0;
    const int my_slot = lane < nc ? W.c_slot[lane] : src;
    const int my_n = b.agg_n[my_slot], my_off = b.agg_off[my_slot];
    int rank = lane;
    if (nc > 1) {
        rank = 0;
        for (int m = 0; m < nc; ++m) {
            const unsigned long long dm = W.c_db[m];
            rank += dm < my_db || (dm == my_db && W.c_key[m] < my_key);
        }
    }
    __syncwarp();
    if (lane < nc) {
        W.s_db[rank] = my_db;
        W.s_slot[rank] = my_slot;
        W.s_off[rank] = my_off;
        W.s_pre[rank] = my_n;
    }
    __syncwarp();
    int n_other = 0;
    {
        const int cnt = lane < nc ? W.s_pre[lane] : 0;
        int incl = cnt;
        if (nc > 1) {
#pragma unroll
            for (int s = 1; s < 32; s <<= 1) {
                const int y = __shfl_up_sync(all, incl, s);
                if (lane >= s) incl += y;
            }
        }
        n_other = shfl_i(incl, nc - 1);
        __syncwarp();
        if (lane < nc) W.s_pre[lane] = incl - cnt;
    }
    __syncwarp();
    const int n_mov = shfl_i(rec.i, REC_N), off_m = shfl_i(rec.i, REC_OFF);
    // pairs for the block: its screens and tiles pay off for more
    if (n_mov > WS::kPairs || n_other > WS::kPairs || n_mov * n_other > WS::kPairs) return false;
    o.cand_spheres = n_other;
    const int *pool_id = sc->pool_sel ? b.pool_id[1] : b.pool_id[0];
    const float4 *pool_pos = sc->pool_sel ? b.pool_pos[1] : b.pool_pos[0];
    const int n_pairs = n_mov * n_other;
    const float inv_mov = 1.f / float(n_mov);
    int n_hit = 0;
    for (int p0 = 0; p0 < n_pairs; p0 += 32) {
        const int p = p0 + lane;
        bool hit = false;
        int r = 0, i = 0, jl = 0, pj = 0;
        if (p < n_pairs) {
            const int f = int((float(p) + 0.5f) * inv_mov);
            i = p - f * n_mov;
            while (r + 1 < nc && W.s_pre[r + 1] <= f) ++r;
            jl = f - W.s_pre[r];
            pj = W.s_off[r] + jl;
            const float4 q = pool_pos[pj], pm = pool_pos[off_m + i];
            Sweep32 wi = w;
            wi.px = pm.x;
            wi.py = pm.y;
            wi.pz = pm.z;
            hit = capsule_hit(wi, q.x, q.y, q.z, pm.w + q.w + margin);
        }
        const unsigned m = __ballot_sync(all, hit);
        if (n_hit + __popc(m) > kWarpCands) return false;
        if (hit) {
            const int at = n_hit + __popc(m & lanes_below(lane));
            W.p_r[at] = r;
            W.p_ij[at] = (static_cast<unsigned long long>(i) << 32) | static_cast<unsigned>(jl);
            W.p_si[at] = pool_id[off_m + i];
            W.p_sj[at] = pool_id[pj];
        }
        n_hit += __popc(m);
    }
    __syncwarp();
    o.refined = n_hit;
    if (n_hit == 0) return true;
    for (int k0 = 0; k0 < n_hit; k0 += 10) {
        const bool act = lane < 30 && k0 + gi < n_hit;
        const int k = act ? k0 + gi : 0;
        const int si = W.p_si[k], sj = W.p_sj[k];
        const double xi = S(b, SPH_X + ax, si), xj = S(b, SPH_X + ax, sj), ri = S(b, SPH_R, si), rj = S(b, SPH_R, sj);
        // two single spheres at their aggregates' centres: the filter's sweep
        // was this one
        const int oslot = W.s_slot[W.p_r[k]];
        const bool same = filtered && ((dbits(xi) ^ dbits(x_g)) | (dbits(ri) ^ dbits(rmax)) |
                                       (dbits(xj) ^ dbits(A(b, AGG_X + ax, oslot))) |
                                       (dbits(rj) ^ dbits(A(b, AGG_RMAX, oslot)))) == 0;
        double res;
        if (__all_sync(all, same || !act))
            res = dkey_inv(W.s_db[W.p_r[k]]);
        else
            res = warp_sweep(g, ax, xi, xj, ri, rj, dl, full, b.L);
        if (act && ax == 0) W.p_key[k] = res < CUDART_INF ? dkey(res) : ~0ULL;
    }
    __syncwarp();
    // the reference's ordered walk with early exits
    const unsigned long long my_res = lane < n_hit ? W.p_key[lane] : ~0ULL;
    const int my_r = lane < n_hit ? W.p_r[lane] : -1;
    unsigned long long best = dkey(CUDART_INF);
    int best_r = -1;
    for (int r = 0; r < nc; ++r) {
        if (best_r >= 0 && (best <= dkey(0.0) || best < W.s_db[r])) break;
        unsigned long long v = my_r == r ? my_res : ~0ULL;
        const unsigned m = __ballot_sync(all, v != ~0ULL);
        if (m == 0u) continue;  // no finite pair: +inf never wins
        if ((m & (m - 1u)) == 0u) {
            v = __shfl_sync(all, v, __ffs(m) - 1);
        } else {
#pragma unroll
            for (int s = 16; s > 0; s >>= 1) {
                const unsigned long long y = __shfl_xor_sync(all, v, s);
                v = y < v ? y : v;
            }
        }
        if (v < best) {
            best = v;
            best_r = r;
        }
    }
    if (best_r < 0) return true;
    // among the candidate's equal minima the first (moving, other) pair
    unsigned long long ij = my_r == best_r && my_res == best ? W.p_ij[lane] : ~0ULL;
    unsigned m = __ballot_sync(all, ij != ~0ULL);
    if ((m & (m - 1u)) != 0u) {
        unsigned long long v = ij;
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) {
            const unsigned long long y = __shfl_xor_sync(all, v, s);
            v = y < v ? y : v;
        }
        m = __ballot_sync(all, ij == v);
    }
    const int win = __ffs(m) - 1;
    o.distance = dkey_inv(best);
    o.ms = W.p_si[win];
    o.os = W.p_sj[win];
    o.oslot = W.s_slot[best_r];
    return true;
}

}  // namespace mcacg
