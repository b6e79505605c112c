// MC steps of the device loop by one warp.
//
// Most steps of a run are small: an aggregate of a few spheres moves, a
// handful of neighbours lie in its reach, and usually none is hit. Such a
// step is a chain of short dependent operations -- loads that wait for one
// another, FP64 instructions at 64 cycles each, barriers -- so it takes the
// same time on 512 threads as on 32, and the barriers and the other warps'
// copies of the uniform FP64 work come on top. Here warp 0 runs the whole
// step alone, without a block barrier:
//
//   pick    the tree descent; the direction's FP64 work fills the wait for
//           the tree's leaves;
//   record  every field of the picked slot in one round of loads (lane f
//           reads field f of the FP64 table and of the integer tables), and
//           the members' relative positions behind it, used after the query;
//   query   the same neighbours, filter, pairs and walk as block_query: the
//           neighbours come through a queue in shared memory, so that a
//           round of loads serves 32 list entries; a swept test takes three
//           lanes, one axis each (warp_sweep, ~40 FP64 instructions for up
//           to ten tests at once);
//   move    member positions, three lanes a sphere;
//   merge   up to 32 spheres, one per lane (warp_merge).
//
// Whatever is larger (long neighbour lists, many sphere pairs, aggregates of
// many spheres, surface reactions, tree rebuilds) goes to the
// block's routines: warp_steps returns the operation, all threads run it
// (block_op), and warp 0 goes on from there. Both ways give the same bits.
//
// What bounds it: about 2000 warp instructions a step in one dependent
// chain (9.5 cycles each on a box alone: 2.7 fixed latency, 3.0 waiting for
// L2, 1.7 for FP64 and shared memory). Measured against the block's loop:
// one box of 4096 monomers 15.4 -> 8.6 us a step; 2000 boxes of 1000
// monomers, a warp each, 35.6 -> 17.5 us; the 512-box ensemble's 4000 early
// steps 158 -> 97 ms; 48 served runs 559 -> 390 ms. The limits (kWarp*, in
// warp_query.cuh and run.cuh) lie where a warp's rounds over the work cost about what the
// block's barriers and set-up do: four rounds of cells, two of members,
// thirty-two of pair screens at two instructions a cycle.
#pragma once
#include "run.cuh"

namespace mcacg {

// What warp_steps asks the block to do.
enum StepOp : int { STEP_EXIT, STEP_QUERY, STEP_MOVE, STEP_REACT, STEP_MERGE, STEP_TREE, STEP_LIVE, STEP_UPDATE,
                     STEP_NEXT };
// Where warp 0 goes on.
enum StepPhase : int { PH_START, PH_QUERIED, PH_MOVED, PH_REACTED, PH_MERGED, PH_END };

// A slot's place after a move: the new centre (lanes 0-2 an axis each) and
// its cells.
struct WarpPlace {
    double x;
    float xf;
    int key, fcell;
};
__device__ __forceinline__ WarpPlace warp_place(const DevBox &b, double x0, double dl, double move) {
    const int lane = threadIdx.x & 31;
    WarpPlace p;
    int vc = 0, fc = 0;
    p.x = 0.0;
    p.xf = 0.f;
    if (lane < 3) {
        p.x = wrap_position(x0 + dl * move, b.L);
        p.xf = float(p.x);
        vc = verlet_coord_dev(b, p.x, p.xf);
        if (b.fine_div > 0) fc = fine_index_near(p.xf, b.fine_step_f, b.fine_div);
    }
    p.key = cell_key(shfl_i(vc, 0), shfl_i(vc, 1), shfl_i(vc, 2));
    const int nf = b.fine_div;
    p.fcell = nf > 0 ? (shfl_i(fc, 0) * nf + shfl_i(fc, 1)) * nf + shfl_i(fc, 2) : -1;
    return p;
}

// Aggregate::translate (aggregat.cpp:148-161) of the picked slot's fields and
// members by warp 0 (as block_translate), without the grids. The members'
// first ten (sid, rel: member lane / 3, axis lane % 3) are already loaded.
__device__ __forceinline__ void warp_translate(const DevBox &b, int pool_sel, int slot, const WarpRec &rec,
                                               const WarpPlace &to, int sid, double rel) {
    const int lane = threadIdx.x & 31;
    const int gi = lane / 3, ax = lane - 3 * gi;
    const int n = shfl_i(rec.i, REC_N), off = shfl_i(rec.i, REC_OFF);
    const double r0 = shfl_d(rec.f, AGG_RX + (lane < 3 ? lane : 0));
    if (lane < 3) {
        A(b, AGG_X + lane, slot) = to.x;
        reinterpret_cast<float *>(b.agg_f4 + slot)[lane] = to.xf;
    }
    const double ref_ax = shfl_d(to.x - r0, ax);
    const int *pool_id = pool_sel ? b.pool_id[1] : b.pool_id[0];
    float *pf = reinterpret_cast<float *>((pool_sel ? b.pool_pos[1] : b.pool_pos[0]) + off);
    if (sid >= 0) {
        const double v = ref_ax + rel;
        S(b, SPH_X + ax, sid) = v;
        pf[4 * gi + ax] = float(v);  // the entry's radius stays as it is
    }
#pragma unroll 1
    for (int k0 = 10; k0 < n; k0 += 40) {
        int s[4];
        double rl[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const int k = k0 + 10 * u + gi;
            s[u] = lane < 30 && k < n ? pool_id[off + k] : -1;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) rl[u] = s[u] >= 0 ? S(b, SPH_RX + ax, s[u]) : 0.0;
#pragma unroll
        for (int u = 0; u < 4; ++u)
            if (s[u] >= 0) {
                const double v = ref_ax + rl[u];
                S(b, SPH_X + ax, s[u]) = v;
                pf[4 * (k0 + 10 * u + gi) + ax] = float(v);
            }
    }
}

// What regrid_to reads to move the slot to 'to', loaded ahead: in 'a' lane 0
// has the length of the new Verlet cell's list, lane 1 that of the old one's,
// lane 2 the head of the new fine cell's (a second round of loads then
// depends on it: warp_regrid_items).
struct WarpGrid {
    int a, b;
};
__device__ __forceinline__ int warp_regrid_heads(const DevBox &b, const WarpRec &rec, const WarpPlace &to) {
    const int lane = threadIdx.x & 31;
    const int old_key = shfl_i(rec.i, REC_CELL);
    if (lane == 2 && b.fine_div > 0) return b.fine_head[to.fcell];
    return lane < 2 ? b.cell_n[cell_index(b, lane == 0 ? to.key : old_key)] : -1;
}
// Lane 0: the old cell's last item, lane 1: its item at the slot's place.
__device__ __forceinline__ int warp_regrid_items(const DevBox &b, const WarpRec &rec, int heads) {
    const int lane = threadIdx.x & 31;
    const int n_old = shfl_i(heads, 1), pos = shfl_i(rec.i, REC_POS), old_key = shfl_i(rec.i, REC_CELL);
    const int k = lane == 0 ? n_old - 1 : pos;
    return lane < 2 && k >= 0 && k < n_old ? b.cell_items[size_t(cell_index(b, old_key)) * b.cell_cap + k] : -1;
}
// regrid_to from those loads (lane 0 stores).
__device__ __forceinline__ void warp_regrid(const DevBox &b, int slot, const WarpRec &rec, const WarpPlace &to,
                                            const WarpGrid &g) {
    const int lane = threadIdx.x & 31;
    const int old_key = shfl_i(rec.i, REC_CELL), pos = shfl_i(rec.i, REC_POS);
    const int fold = shfl_i(rec.i, REC_FINE), fprev = shfl_i(rec.i, REC_PREV), fnext = shfl_i(rec.i, REC_NEXT);
    const int n_new = shfl_i(g.a, 0), n_old = shfl_i(g.a, 1), fhead = shfl_i(g.a, 2);
    const int last = shfl_i(g.b, 0), item = shfl_i(g.b, 1);
    if (to.key != old_key && (item != slot || n_new >= b.cell_cap)) {
        // not where recorded, or a full cell: the general form
        if (lane == 0) regrid_to(b, slot, to.key, to.fcell);
        return;
    }
    if (lane == 0) {
        if (to.key != old_key) {
            const int c = cell_index(b, to.key), old = cell_index(b, old_key);
            b.cell_items[size_t(old) * b.cell_cap + pos] = last;
            b.cell_pos[last] = pos;
            b.cell_n[old] = n_old - 1;
            b.cell_items[size_t(c) * b.cell_cap + n_new] = slot;
            b.cell_pos[slot] = n_new;
            b.cell_n[c] = n_new + 1;
            b.agg_cell[slot] = to.key;
        }
        if (to.fcell != fold) {
            if (fold >= 0) {
                if (fprev >= 0) b.fine_next[fprev] = fnext; else b.fine_head[fold] = fnext;
                if (fnext >= 0) b.fine_prev[fnext] = fprev;
            }
            b.fine_next[slot] = fhead;
            b.fine_prev[slot] = -1;
            if (fhead >= 0) b.fine_prev[fhead] = slot;
            b.fine_head[to.fcell] = slot;
            b.fine_cell[slot] = to.fcell;
        }
    }
}

// The merge of the step's contact by warp 0: block_merge (with no volume and
// surface correction), the physics and the pick tree of commit_merge, one
// sphere of the merged aggregate per lane. The FP64 chains are cut by doing
// what is independent on different lanes of one instruction: the seven
// ordered sums and the overlap's, the five quotients at the end, the two
// reciprocals after the physics; a tree update adds differences to the
// ancestors (the weights are integers, so the sums are the same) instead of
// reading 32 children a level. Returns WM_BLOCK when the block has to do it
// (more than 32 spheres, or the member pool is full; nothing was changed).
enum WarpMergeResult : int { WM_BLOCK, WM_DONE, WM_TREE, WM_LIVE };
template <class LS>
__device__ __noinline__ int warp_merge() {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LS &sm = *reinterpret_cast<LS *>(smem_raw);
    const BoxRun &R = sm.R;
    const DevBox &b = R.box;
    DevScalars *sc = &sm.sc;
    RunState &st = sm.st;
    auto &M = sm.u.wm;
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, a3 = lane < 3 ? lane : 0;
    const int ms = sm.ms, os = sm.os, mslot = sm.mslot, cslot = sm.cslot;
    const int keep = min(mslot, cslot), removed = max(mslot, cslot);
    const int my = mslot == keep ? ms : os, oth = mslot == keep ? os : ms;
    // round 1: both records, the two spheres, the leaves
    const RecRows rows = record_rows(sm.R.box, sm.rec_ptr, lane);
    const WarpRec rk = load_record(rows, keep), rr = load_record(rows, removed);
    const double pm = S(b, SPH_X + a3, ms), po = S(b, SPH_X + a3, os);
    const double rms = S(b, SPH_R, ms), ros = S(b, SPH_R, os);
    const double rel_my = S(b, SPH_RX + a3, my), rel_oth = S(b, SPH_RX + a3, oth);
    const unsigned long long w_keep = R.tree[R.tree_off[0] + keep], w_removed = R.tree[R.tree_off[0] + removed];
    const int nk = shfl_i(rk.i, REC_N), nr = shfl_i(rr.i, REC_N), n = nk + nr;
    const int off_keep = shfl_i(rk.i, REC_OFF), off_rem = shfl_i(rr.i, REC_OFF);
    const int new_off = sc->pool_top;
    if (n > 32 || keep == removed || new_off + n > b.pool_cap) return WM_BLOCK;
    {
        const double d = wrap_distance(pm - po, b.L);
        const double d2 = sum3(d * d, 0);
        const double s = rms + ros;
        const double gap = d2 - s * s;
        if (!(dkey(gap) <= dkey(kContactEpsilon)) || is_nan(gap)) return WM_DONE;  // the spheres no longer touch
    }
    const double diff = (rel_my + wrap_distance(my == ms ? po - pm : pm - po, b.L)) - rel_oth;
    // round 2: the members, and the removed slot's cell
    int *pool_id = sc->pool_sel ? b.pool_id[1] : b.pool_id[0];
    float4 *pool_pos = sc->pool_sel ? b.pool_pos[1] : b.pool_pos[0];
    const bool act = lane < n, gone = act && lane >= nk;
    const int at = lane < nk ? off_keep + lane : off_rem + (lane - nk);
    const int sid = act ? pool_id[at] : 0;
    float4 pp = make_float4(0.f, 0.f, 0.f, 0.f);
    if (act) pp = pool_pos[at];
    const int cell_r = cell_index(b, shfl_i(rr.i, REC_CELL)), pos_r = shfl_i(rr.i, REC_POS);
    const int n_cell_r = b.cell_n[cell_r];
    // round 3: the spheres
    double r = 0.0, vol = 0.0, surf = 0.0, rx = 0.0, ry = 0.0, rz = 0.0;
    if (act) {
        r = S(b, SPH_R, sid);
        vol = S(b, SPH_VOLUME, sid);
        surf = S(b, SPH_SURFACE, sid);
        rx = S(b, SPH_RX, sid);
        ry = S(b, SPH_RY, sid);
        rz = S(b, SPH_RZ, sid);
    }
    const double ref = S(b, SPH_X + a3, shfl_i(sid, 0));
    int *items = b.cell_items + size_t(cell_r) * b.cell_cap;
    const bool listed = pos_r >= 0 && pos_r < n_cell_r;
    const int at_pos = listed ? items[pos_r] : -1, last = listed ? items[n_cell_r - 1] : -1;
    {
        const double dx = shfl_d(diff, 0), dy = shfl_d(diff, 1), dz = shfl_d(diff, 2);
        const double fx = shfl_d(ref, 0), fy = shfl_d(ref, 1), fz = shfl_d(ref, 2);
        if (gone) {  // relabel and shift the removed aggregate's spheres
            rx = rx + dx;
            ry = ry + dy;
            rz = rz + dz;
            const double x = rx + fx, y = ry + fy, z = rz + fz;
            b.sph_slot[sid] = keep;
            S(b, SPH_RX, sid) = rx;
            S(b, SPH_RY, sid) = ry;
            S(b, SPH_RZ, sid) = rz;
            S(b, SPH_X, sid) = x;
            S(b, SPH_Y, sid) = y;
            S(b, SPH_Z, sid) = z;
            pp.x = float(x);
            pp.y = float(y);
            pp.z = float(z);
        }
    }
    if (act) {
        pool_id[new_off + lane] = sid;
        pool_pos[new_off + lane] = pp;
        b.sph_volw[sid] = vol;
        M.rel[0][lane] = rx;
        M.rel[1][lane] = ry;
        M.rel[2][lane] = rz;
        M.term[0][lane] = vol;
        M.term[1][lane] = surf;
        M.term[2][lane] = rx * vol;
        M.term[3][lane] = ry * vol;
        M.term[4][lane] = rz * vol;
        M.term[5][lane] = vol * (r * r);
        M.term[6][lane] = r;
    }
    if (lane == 0) {
        b.agg_off[keep] = new_off;
        b.agg_n[keep] = n;
        b.agg_n[removed] = 0;
        sc->pool_top = new_off + n;
        sc->n_alive -= 1;
    }
    // the removed slot leaves the grids
    const int prev_r = shfl_i(rr.i, REC_PREV), next_r = shfl_i(rr.i, REC_NEXT), fine_r = shfl_i(rr.i, REC_FINE);
    if (lane == 0) {
        if (at_pos == removed) {
            items[pos_r] = last;
            b.cell_pos[last] = pos_r;
            b.cell_pos[removed] = -1;
            b.cell_n[cell_r] = n_cell_r - 1;
        } else {
            cell_remove(b, cell_r, removed);
        }
        if (fine_r >= 0) {
            if (prev_r >= 0) b.fine_next[prev_r] = next_r; else b.fine_head[fine_r] = next_r;
            if (next_r >= 0) b.fine_prev[next_r] = prev_r;
            b.fine_cell[removed] = -1;
        }
    }
    __syncwarp();
    // contact pairs i < j in (i, j) order: an FP32 screen with the margins of
    // block_pair_scan, then the exact test
    int P = 1;
    if (n == 2) {
        if (lane == 0) M.pair[0] = 1;  // i = 0, j = 1
    } else {
        const float fx = float(rx), fy = float(ry), fz = float(rz), fr = pp.w;
        const float ext = act ? fabsf(fx) + fabsf(fy) + fabsf(fz) + fr : 0.f;
        const float margin = 1.0e-5f * __int_as_float(__reduce_max_sync(all, __float_as_int(ext)));
        P = 0;
        for (int i = 0; i + 1 < n; ++i) {
            const float dx = shfl_f(fx, i) - fx, dy = shfl_f(fy, i) - fy, dz = shfl_f(fz, i) - fz;
            const float reach = (shfl_f(fr, i) + fr) * 1.0001f + margin;
            const bool hit = act && lane > i && __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, dz * dz)) <= reach * reach;
            const unsigned m = __ballot_sync(all, hit);
            if (hit) M.pair[P + __popc(m & lanes_below(lane))] = static_cast<unsigned short>((i << 8) | lane);
            P += __popc(m);
        }
    }
    __syncwarp();
    int Pc = 0;
    for (int p0 = 0; p0 < P; p0 += 32) {
        const bool has = p0 + lane < P;
        const int ij = has ? M.pair[p0 + lane] : 1;
        const int i = ij >> 8, j = ij & 255;
        const double ex = M.rel[0][i] - M.rel[0][j], ey = M.rel[1][i] - M.rel[1][j], ez = M.rel[2][i] - M.rel[2][j];
        const double dist = fp64_sqrt(ex * ex + ey * ey + ez * ez);
        const double rsum = M.term[6][i] + M.term[6][j];
        const bool pass = has && nonneg_le(dist, (1. + kCoordinationEpsilon) * rsum);
        const double term = 2.0 * fp64_div(rsum - dist, rsum);
        const unsigned m = __ballot_sync(all, pass);
        if (pass) M.ov[Pc + __popc(m & lanes_below(lane))] = term;
        Pc += __popc(m);
    }
    __syncwarp();
    // the ordered sums: the seven series on lanes 0-6, the overlap's on lane 7
    double acc = 0.0;
    {
        const double *v = lane < 7 ? M.term[lane] : M.ov;
        const int lim = lane < 7 ? n : (lane == 7 ? Pc : 0), most = max(n, Pc);
#pragma unroll 4
        for (int k = 0; k < most; ++k) acc = acc + (k < lim ? v[k] : 0.0);
    }
    const double V = shfl_d(acc, 0), Sf = shfl_d(acc, 1);
    if (not_positive(V) || not_positive(Sf)) {
        if (lane == 0) {
            sc->status = ST_VOL_SURF;
            st.status = ST_VOL_SURF;
            sm.stop = 1;
        }
        __syncwarp();
        return WM_DONE;
    }
    const double cm = fp64_div(acc, V);  // lanes 2-4: the centre of mass
    const double cx = shfl_d(cm, 2), cy = shfl_d(cm, 3), cz = shfl_d(cm, 4);
    const double dx = rx - cx, dy = ry - cy, dz = rz - cz;
    const double dcen = fp64_sqrt(dx * dx + dy * dy + dz * dz);
    long long rmax_bits = act ? nonneg_max_bits(0, dbits(r + dcen)) : 0;  // non-negative: integer order
    M.term[7][lane] = vol * (dcen * dcen);
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        const long long y = __shfl_xor_sync(all, rmax_bits, s);
        rmax_bits = y > rmax_bits ? y : rmax_bits;
    }
    const double rmax = __longlong_as_double(rmax_bits);
    __syncwarp();
    double arg = 0.0;
#pragma unroll 4
    for (int k = 0; k < n; ++k) arg = arg + M.term[7][k];
    // the quotients of the fields, one per lane: Rg's, the mean diameter, the
    // mean sphere volume, overlap and coordination
    const double nd = double(n), pd = double(2 * Pc);
    const double brg = shfl_d(acc, 5), sum_r = shfl_d(acc, 6), sum_ov = shfl_d(acc, 7);
    const double prod = (lane == 0 ? 3. / 5. : 2.0) * (lane == 0 ? brg : sum_r);
    const double num = lane == 0 ? arg + prod : (lane == 1 ? prod : (lane == 2 ? V : (lane == 3 ? sum_ov : pd)));
    const double den = lane == 0 ? V : (lane == 3 ? pd : nd);
    const double quo = fp64_div(num, den);
    const double rg = fp64_sqrt(fabs(shfl_d(quo, 0)));
    const double dp = shfl_d(quo, 1), vol_pp = shfl_d(quo, 2);
    const double overlapping = Pc > 0 ? shfl_d(quo, 3) : 0.0, coordination = Pc > 0 ? shfl_d(quo, 4) : 0.0;
    const double x = wrap_position(ref + shfl_d(cm, 2 + a3), b.L);  // lanes 0-2
    const float cf = float(lane < 3 ? x : (lane == 3 ? rmax : (lane == 4 ? V : (lane == 5 ? vol_pp : half_any(dp)))));
    const float4 ph = physics_f32(R.phys, shfl_f(cf, 6), shfl_f(cf, 4), shfl_f(cf, 5));
    const double phd = double(lane == 0 ? ph.x : (lane == 1 ? ph.y : (lane == 2 ? ph.z : ph.w)));
    // lane 0: Rg / (dp / 2), lane 2: 1 / time step
    const double rec = fp64_div(lane == 0 ? rg : 1.0, lane == 0 ? half_any(dp) : phd);
    unsigned long long wk = __double2ull_rn(fmin(rec * st.tree_scale, double(kTreeHeadroom)));
    wk = __shfl_sync(all, wk > 0ULL ? wk : 1ULL, 2);
    const double time = (shfl_d(rk.f, AGG_TIME) + shfl_d(rr.f, AGG_TIME)) - st.time;
    if (lane < 3) {
        A(b, AGG_X + lane, keep) = x;
        reinterpret_cast<float *>(b.agg_f4 + keep)[lane] = cf;
    }
    if (lane >= 2 && lane < 5) A(b, AGG_RX + lane - 2, keep) = cm;
    if (lane < 4) A(b, lane == 0 ? AGG_F_AGG : (lane == 1 ? AGG_D_M : (lane == 2 ? AGG_TIME_STEP : AGG_LPM)), keep) = phd;
    if (lane == 3) reinterpret_cast<float *>(b.agg_f4 + keep)[3] = cf;
    int vc = 0, fc = 0;
    if (lane < 3) {
        vc = verlet_coord_dev(b, x, cf);
        if (b.fine_div > 0) fc = fine_index(cf, b.fine_step_f, b.fine_div);
    }
    const int nf = b.fine_div;
    const int key = cell_key(shfl_i(vc, 0), shfl_i(vc, 1), shfl_i(vc, 2));
    const int fcell = nf > 0 ? (shfl_i(fc, 0) * nf + shfl_i(fc, 1)) * nf + shfl_i(fc, 2) : -1;
    const int cell_k = shfl_i(rk.i, REC_CELL), fine_k = shfl_i(rk.i, REC_FINE);
    const unsigned long long total = st.tree_total - w_keep - w_removed + wk;
    if (lane == 0) {
        A(b, AGG_RG, keep) = rg;
        A(b, AGG_RMAX, keep) = rmax;
        A(b, AGG_VOLUME, keep) = V;
        A(b, AGG_SURFACE, keep) = Sf;
        A(b, AGG_DP, keep) = dp;
        A(b, AGG_OVERLAPPING, keep) = overlapping;
        A(b, AGG_COORDINATION_NUMBER, keep) = coordination;
        A(b, AGG_DG_OVER_DP, keep) = rec;
        A(b, AGG_TIME, keep) = time;
        if (key != cell_k || fcell != fine_k) regrid_to(b, keep, key, fcell);
        if (dkey(rmax) > dkey(sc->maxradius) && !is_nan(sc->maxradius)) sc->maxradius = rmax;
        sm.merged = 1;
        st.c_merged_spheres += n;
        st.c_merge_pairs += Pc;
    }
    tree_merge(R, sm.tree, 0ULL, keep, removed, w_keep, w_removed, wk);
    const bool rescale = total > kTreeHeadroom;  // a new scale keeps the total clear of 2^64
    if (lane == 0) tree_total_to_state(st, total);
    if (sm.live.on) warp_live_merge(sm.live, keep, removed, wk);
    __syncwarp();
    if (rescale) return WM_TREE;
    return !sm.live.on && sm.live.allow && sc->n_alive <= sm.live.max ? WM_LIVE : WM_DONE;
}

// A step's pick and direction by one warp, from the step's three rand() values
// on lanes 0-2: the slot (-1: the tree has lost a live slot), its record and
// the direction's components on lanes 0-2.
struct WarpPicked {
    WarpRec rec;
    double dl;
    int slot;
};
template <class LS>
__device__ __forceinline__ WarpPicked warp_pick(LS &sm, int rnd) {
    const int lane = threadIdx.x & 31;
    const BoxRun &R = sm.R;
    WarpPicked p;
    const unsigned long long r0 = static_cast<unsigned long long>(shfl_i(rnd, 0)), total = sm.st.tree_total;
    unsigned long long t = (__umul64hi(r0, total) << 33) | ((r0 * total) >> 31);
    // the leaves' load is under way while the direction (direction_from, an
    // axis on each of lanes 0-2) is formed
    const bool live = sm.live.on != 0;
    int base = 0;
    unsigned long long leaf = 0ULL;
    if (!live) {
        int node = 0;
#pragma unroll 1
        for (int lev = R.tree_levels - 1; lev > 0; --lev)
            node = node * kTreeFan + tree_pick_child(tree_children(R, sm.tree, lev, node * kTreeFan), t);
        base = node * kTreeFan;
        leaf = tree_children(R, sm.tree, 0, base);
    }
    {
        const float u1 = float(shfl_i(rnd, 1)) * (1.0f / 2147483647.0f);
        const float u2 = float(shfl_i(rnd, 2)) * (1.0f / 2147483647.0f);
        const float cpf = 1.f - 2.f * u2;
        const float spf = 2.f * sqrtf(u2 * (1.f - u2));
        float sth, cth;
        sincospif(2.f * u1, &sth, &cth);
        const double d = double(lane == 0 ? spf * cth : (lane == 1 ? spf * sth : cpf));
        const double k = 1.5 - 0.5 * sum3(d * d, 0);
        p.dl = d * k;
    }
    const int slot = live ? live_sample(sm.live, t) : base + tree_pick_child(leaf, t);
    const bool ok = slot >= 0 && slot < R.box.nslots;
    p.rec = load_record(record_rows(R.box, sm.rec_ptr, lane), ok ? slot : 0);
    p.slot = ok && shfl_i(p.rec.i, REC_N) != 0 ? slot : -1;
    return p;
}

// warp_query on the scratch of the round's step k. Where the last kMissRun
// queries of larger aggregates were the block's (dense boxes of few aggregates),
// the next ones go there without a try, all but every eighth. (64 boxes of 200
// spheres in 8 aggregates at 8000 ppm, 600 steps on 128 threads: 12.9 -> 12.3
// ms; after a run of 4, boxes of 100 aggregates of a few spheres lost 4%.)
template <class LS>
__device__ __forceinline__ bool loop_query(LS &sm, int k, int src, const WarpRec &rec, double dl, double full,
                                           WarpAnswer &o) {
    const int *live = sm.live.on ? sm.live.slot : nullptr;
    const bool large = shfl_i(rec.i, REC_N) >= kWarpEarly;
    // (warp 0 alone reads and writes its count while a round is under way)
    const int missed = k == 0 ? sm.misses : sm.round_misses;
    bool ok = false;
    if (!large || missed < kMissRun || (missed & 7) == 0) {
        if constexpr (LS::kRounds > 1)
            ok = warp_query(sm.R.box, &sm.sc, sm.u.r[k], live, sm.live.n, src, rec, dl, full, o);
        else
            ok = warp_query(sm.R.box, &sm.sc, sm.u.w, live, sm.live.n, src, rec, dl, full, o);
    }
    if (large && k == 0 && (!ok || missed != 0)) {
        __syncwarp();
        if ((threadIdx.x & 31) == 0) sm.misses = ok ? 0 : missed + 1;
        __syncwarp();
    }
    return ok;
}

// A picked slot's move, prepared: its place, the members' first ten and what
// its change of cells reads, all loaded together; and carried out.
struct WarpMove {
    WarpPlace to;
    WarpGrid grid;
    int sid;
    double rel;
};
template <class LS>
__device__ __forceinline__ WarpMove loop_prepare(LS &sm, const WarpRec &rec, double dl, double move) {
    const DevBox &b = sm.R.box;
    const int lane = threadIdx.x & 31, gi = lane / 3, ax = lane - 3 * gi;
    const int n = shfl_i(rec.i, REC_N), off = shfl_i(rec.i, REC_OFF);
    WarpMove m;
    m.sid = lane < 30 && gi < n ? (sm.sc.pool_sel ? b.pool_id[1] : b.pool_id[0])[off + gi] : -1;
    m.to = warp_place(b, shfl_d(rec.f, AGG_X + (lane < 3 ? lane : 0)), dl, move);
    const bool cell = m.to.key != shfl_i(rec.i, REC_CELL);
    m.grid = WarpGrid{-1, -1};
    if (cell || m.to.fcell != shfl_i(rec.i, REC_FINE)) m.grid.a = warp_regrid_heads(b, rec, m.to);
    m.rel = m.sid >= 0 ? S(b, SPH_RX + ax, m.sid) : 0.0;
    if (cell) m.grid.b = warp_regrid_items(b, rec, m.grid.a);
    return m;
}
// 'grids': the cells are changed here (else by the caller).
template <class LS>
__device__ __forceinline__ void loop_move(LS &sm, int slot, const WarpRec &rec, const WarpMove &m, bool grids) {
    const DevBox &b = sm.R.box;
    const bool moves = m.to.key != shfl_i(rec.i, REC_CELL) || m.to.fcell != shfl_i(rec.i, REC_FINE);
    if (moves && grids) warp_regrid(b, slot, rec, m.to, m.grid);
    warp_translate(b, sm.sc.pool_sel, slot, rec, m.to, m.sid, m.rel);
}
template <class LS>
__device__ __noinline__ void loop_move_call(int slot, WarpRec rec, WarpMove m, bool grids) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    loop_move(*reinterpret_cast<LS *>(smem_raw), slot, rec, m, grids);
}

// Warp 0: MC steps until the block is needed or the run ends (sm.left counts
// the steps still allowed; t_phase is the clock at the start of the phase).
// Returns the operation (StepOp). The counters are summed in registers and
// added to the loop state every so often.
// In a loop of rounds (block_rounds) it only carries a step on from its query,
// and returns STEP_NEXT at its end.
template <class LS>
__device__ __forceinline__ int warp_steps(LS &sm, int phase, unsigned &t_phase) {
    const int lane = threadIdx.x & 31;
    const BoxRun &R = sm.R;
    const DevBox &b = R.box;
    RunState &st = sm.st;
    const RecRows rows = record_rows(sm.R.box, sm.rec_ptr, lane);
    const int a3 = lane < 3 ? lane : 0;
    const bool growth = R.phys.growth != 0;
    // members translated here; more are the block's (one warp does them all)
    const int move_max = blockDim.x > 32 ? kWarpMove : INT_MAX;
    bool finished = st.finished || st.status != ST_OK || sm.stop;
    // steps until the counters are added to the loop state
    int quota = 0, n_done = 0;
    unsigned n_mov = 0, n_scanned = 0, n_cells = 0, cyc_pick = 0, cyc_query = 0, cyc_scan = 0, cyc_move = 0, cyc_end = 0;
    int n_query = 0;
    // the step under way
    int slot = sm.slot, contact = sm.contact, status = ST_OK;
    double full = sm.full, move = sm.move, dl = lane < 3 ? sm.dir[lane] : 0.0;
    WarpRec rec{0.0, -1};
    bool have = false;  // the record is loaded
    auto flush = [&]() {
        if (lane == 0) {
            sm.left -= n_done;
            st.n_iter_without_event += n_done;
            st.steps += n_done;
            st.c_queries += n_query;
            st.c_mov += n_mov;
            st.c_scanned += n_scanned;
            st.c_cells += n_cells;
            st.cyc_pick += cyc_pick;
            st.cyc_query += cyc_query;
            st.cyc_qscan += cyc_scan;
            if (n_query > 0) st.cyc_qpairs += (long long)cyc_query - (long long)cyc_scan;
            st.cyc_move += cyc_move;
            st.cyc_merge += cyc_end;
        }
        __syncwarp();
        n_done = n_query = 0;
        n_mov = n_scanned = n_cells = cyc_pick = cyc_query = cyc_scan = cyc_move = cyc_end = 0;
    };
    int op = STEP_EXIT;
    for (;;) {
        if (phase == PH_START) {
            op = LS::kRounds > 1 ? STEP_NEXT : STEP_EXIT;
            if (LS::kRounds > 1) break;
            if (n_done >= quota) {
                flush();
                quota = int(min(sm.left, 256LL));
            }
            if (quota <= 0 || finished) break;
            if (sm.deadline != 0ULL) {
                // a time-capped launch: checked before every step, so that a
                // box of expensive steps does not hold the launch past the cap
                const int over = lane == 0 && global_ns() >= sm.deadline;
                if (shfl_i(over, 0)) break;
            }
            t_phase = clock_lo();
            // the step's three rand() values, one on each of lanes 0-2 (each
            // needs values at least three places back)
            int rnd = 0;
            {
                const int pos = st.rng.pos;
                int k = pos + a3;
                k -= k >= 34 ? 34 : 0;
                const uint32_t v = st.rng.r[k >= 3 ? k - 3 : k + 31] + st.rng.r[k >= 31 ? k - 31 : k + 3];
                __syncwarp();
                if (lane < 3) st.rng.r[k] = v;
                if (lane == 0) st.rng.pos = pos >= 31 ? pos - 31 : pos + 3;
                rnd = int(v >> 1);
                __syncwarp();
            }
            const WarpPicked p = warp_pick(sm, rnd);
            rec = p.rec;
            dl = p.dl;
            if (p.slot < 0) {
                status = ST_UNKNOWN;  // the tree lost a live slot: stop this box
                break;
            }
            slot = p.slot;
            const int n = shfl_i(rec.i, REC_N);
            have = true;
            contact = 0;
            full = shfl_d(rec.f, AGG_LPM);
            move = full;
            const unsigned now = clock_lo();
            cyc_pick += now - t_phase;
            t_phase = now;
            if (R.lim.with_collisions) {
                WarpAnswer o;
                if (!loop_query(sm, 0, slot, rec, dl, full, o)) {
                    op = STEP_QUERY;
                    break;
                }
                n_query += 1;
                n_mov += n;
                n_scanned += o.scanned;
                n_cells += o.cells;
                if (o.cands > 0 && lane == 0) {
                    st.c_candidates += o.cands;
                    st.c_cand_spheres += o.cand_spheres;
                    st.c_refined += o.refined;
                }
                if (o.status != ST_OK) {
                    status = o.status;
                    break;
                }
                if (o.oslot >= 0 && dkey(o.distance) <= dkey(full)) {
                    contact = 1;
                    move = o.distance;
                    if (lane == 0) {
                        sm.ms = o.ms;
                        sm.os = o.os;
                        sm.oslot = o.oslot;
                    }
                }
                const unsigned done = clock_lo();
                cyc_scan += o.t_scan - t_phase;
                cyc_query += done - t_phase;
                t_phase = done;
            }
            phase = PH_QUERIED;
        }
        if (phase == PH_QUERIED) {
            if (!have) {  // back from the block's query
                if (finished) break;
                rec = load_record(rows, slot);
                have = true;
                const unsigned now = clock_lo();
                if (lane == 0) st.cyc_query += now - t_phase;
                t_phase = now;
            }
            if (shfl_i(rec.i, REC_N) > move_max) {
                op = STEP_MOVE;
                break;
            }
            loop_move(sm, slot, rec, loop_prepare(sm, rec, dl, move), true);
            phase = PH_MOVED;
        }
        if (phase == PH_MOVED) {
            // without contact the move is the full lpm and the ratio is 1; the
            // aggregate's proper time and the box's advance together
            if (!have && lane == AGG_TIME) rec.f = A(b, AGG_TIME, slot);
            const double ratio = contact ? fp64_div(move, full) + 0.0 : 1.0;
            const double dt = contact ? st.inv_weight * ratio : st.inv_weight;
            const double then = (lane == AGG_TIME ? rec.f : st.time) + dt;
            if (lane == AGG_TIME) A(b, AGG_TIME, slot) = then;
            __syncwarp();
            if (lane == 0) st.time = then;
            const unsigned now = clock_lo();
            cyc_move += now - t_phase;
            t_phase = now;
            if (contact || growth) {
                const double own = have ? shfl_d(rec.f, AGG_TIME_STEP) : sm.dt_indiv;
                if (lane == 0) {
                    sm.slot = slot;
                    sm.mslot = slot;
                    sm.cslot = sm.oslot;
                    sm.merged = 0;
                    sm.try_merge = contact;
                    sm.step_dt = dt;
                    sm.step_dt_indiv = contact ? own * ratio : own;
                }
                __syncwarp();
                if (growth) {
                    op = STEP_REACT;
                    break;
                }
                phase = PH_REACTED;
            }
        }
        if (phase == PH_REACTED) {
            op = STEP_EXIT;
            if (finished) break;
            if (sm.try_merge) {
                op = STEP_MERGE;
                const int did = !growth && b.volsurf == VS_NONE ? warp_merge<LS>() : WM_BLOCK;
                if (did == WM_BLOCK) break;
                op = did == WM_TREE ? STEP_TREE : STEP_LIVE;
                if (did != WM_DONE) break;
            }
            phase = PH_MERGED;
        }
        if (phase == PH_MERGED) {
            op = STEP_EXIT;
            if (finished || sm.stop) break;
            if (growth) {
                op = STEP_UPDATE;
                break;
            }
            phase = PH_END;
        }
        // the end of the step
        __syncwarp();
        if (phase == PH_END) {  // after a contact or surface reactions
            flush();
            if (lane == 0) {
                sm.left -= 1;
                step_end(R, sm);
            }
            __syncwarp();
            quota = 0;
            finished = st.finished != 0;
        } else {
            n_done += 1;
            const long long iter_limit = R.lim.n_iter_without_event_limit;
            const double time_limit = R.lim.physical_time_limit;
            finished = (iter_limit > 0 && st.n_iter_without_event + n_done >= iter_limit) ||
                       (dbits(time_limit) > 0 && nonneg_le(time_limit, st.time));
            if (finished && lane == 0) st.finished = 1;
        }
        const unsigned now = clock_lo();
        cyc_end += now - t_phase;
        t_phase = now;
        have = false;
        phase = PH_START;
    }
    // what the block's operation and the next entry need
    flush();
    if (lane < 3) sm.dir[lane] = dl;
    if (have && lane == AGG_TIME_STEP) sm.dt_indiv = rec.f;
    if (lane == 0) {
        if (status != ST_OK) st.status = status;
        sm.slot = slot;
        sm.full = full;
        sm.dt = st.inv_weight;
        sm.contact = contact;
        sm.move = move;
    }
    __syncwarp();
    return op;
}

// What warp 0 asked for, by the whole block; returns where warp 0 goes on.
// Out of line (and on the shared memory itself, so that its accesses are
// known to be shared): the steps' own registers and code stay small.
template <class LS>
__device__ __noinline__ int block_op(int op) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    LS &sm = *reinterpret_cast<LS *>(smem_raw);
    const BoxRun &R = sm.R;
    typename LS::Base &rs = sm;
    const int tid = threadIdx.x;
    if (op == STEP_QUERY) {
        const unsigned t0 = clock_lo();
        block_query(R.box, sm.slot, Vec3{sm.dir[0], sm.dir[1], sm.dir[2]}, sm.full, sm.u.q, &sm.live);
        if (tid == 0) {
            apply_query(sm.st, rs, sm.u.q.out);
            sm.far = sm.st.status == ST_OK && blockDim.x > 32 && R.box.agg_n[sm.slot] > kWarpMove;
        }
        __syncthreads();
        if (!sm.far) return PH_QUERIED;
        // a move for the block too: carried out without going back first
        if (tid == 0) {
            const unsigned cyc = clock_lo() - t0;
            sm.st.cyc_query += cyc;
            sm.st.cyc_move -= (long long)cyc;  // (the caller counts both as the move's)
        }
        op = STEP_MOVE;
    }
    if (op == STEP_MOVE) {
        block_translate(R.box, sm.slot, tid < 3 ? sm.dir[tid] * sm.move : 0.0, sm.refpos);
        return PH_MOVED;
    }
    if (op == STEP_REACT) {
        commit_reactions(R, rs);
        return PH_REACTED;
    }
    if (op == STEP_MERGE) {
        commit_merge(R, rs);
        return PH_MERGED;
    }
    if (op == STEP_TREE || op == STEP_LIVE) {
        if (op == STEP_TREE) {
            block_tree_build(R);
            tree_cache_load(R, sm.tree);
        }
        live_load(R, sm.live, sm.u.q.warp_tmp);
        return PH_MERGED;
    }
    commit_update(R, rs);
    return PH_END;
}

// One step of a round (block_rounds), as its warp prepared it.
struct RoundJob {
    int slot;    // -1: no live slot picked
    int status, heavy;  // heavy: the block's query or translation
    int n, contact, ms, os, oslot;
    int scanned, cells, cands, cand_spheres, refined;
    int old_key, key, old_fine, fine;
    uint32_t rnd[3];
    float centre[4];  // and r_max, as the record has them
    float ux, uy, uz, full_f, move_f;
    double dir[3], full, move, dt_indiv;
};

// The shared memory of the loop: the block routines' plan, and the box's
// record, loop state and scalars, kept on chip for the launch.
template <class RS, int Rounds>
struct LoopSmemT : RS {
    using Base = RS;
    static constexpr int kRounds = Rounds;  // steps of a round (block_rounds); 1: one after another
    RoundJob job[Rounds];
    int seq;                       // steps to run one after another before the next round
    int round_n, round_sum;        // rounds since the last look, and the steps they took
    int alone_n, looks, back;      // steps one after another of this stretch; looks won; length of the next stretch
    unsigned round_cyc, alone_cyc;  // cycles of those rounds and steps
    float alone_pace;               // cycles a step one after another
    int n_jobs, n_commit, serial;  // steps drawn, steps committed, those whose cell changes wait for others'
    double commit_dt;              // time increment of the round's last step
    BoxRun R;
    RunState st;
    DevScalars sc;
    long long left;  // steps still allowed in this launch
    int misses;      // queries of larger aggregates in a row that were the block's (loop_query),
    int round_misses;  // and as they were at the round's start
    int far;         // block_op: the query's aggregate is the block's to move
    const int *rec_ptr[REC_INTS];  // the integer tables of a slot's record
};

// ------------------------------------------------------------------ rounds
// With more than one warp a box's next steps are taken in rounds: between two
// events the pick tree does not change, so the picks and directions of the
// next steps depend on the box's rand() stream alone. Warp k draws, picks and
// queries the round's step k on the state at the round's start and prepares
// its move; then the steps are committed in order, up to the first one that
// an earlier step of the round could have changed, the first with a contact
// (it is committed, its merge ends the round), or the first that the block
// has to run. What is not committed is drawn again from the same place of
// the stream, so the runs are the sequential loop's, bit for bit: a query's
// answer depends on the aggregates whose bounding spheres its swept bounding
// sphere can meet, and an aggregate whose whole move stays clear of that
// sweep is none of them before or after its move.
//
// What bounds it: a step is one warp's chain of dependent operations, so a
// box that has the SM (or half of it) to itself leaves it idle; a round takes
// about 1.5 steps' time and commits up to kRoundMax of them. Seven: the
// stream's 31-value recurrence gives 21 values ahead, and the pairs of seven
// fit a warp. Measured, kernel time: one box of 4096 monomers, 2000 steps,
// 18.2 -> 7.1 ms; 48 served runs 390 -> 250 ms in all. The steps of 152 boxes
// late in their run (few aggregates, whose sweeps meet) stay one after
// another, 13.25 against 13.2 ms, and so do most of the first 4000 steps of
// 152 or 304 dense boxes (69.9 against 71.5 ms and 88.5 against 88.0).
//
// Could the sweep of step a (its move) come within reach of the sweep of step
// b (its whole length)? Conservative, in FP32: the distance of the two
// segments against the sum of the radii with four screening margins (one is
// more than ten times the FP32 error, see DevBox::margin); true also when the
// two are long enough for a second periodic image to matter.
__device__ inline bool rounds_conflict(const DevBox &b, const RoundJob &a, const RoundJob &c) {
    if (a.slot == c.slot) return true;
    const float reach = a.centre[3] + c.centre[3] + 4.f * b.margin_f;
    if (!(a.move_f + c.full_f + reach < 0.45f * b.Lf)) return true;
    float wx = c.centre[0] - a.centre[0], wy = c.centre[1] - a.centre[1], wz = c.centre[2] - a.centre[2];
    wx -= b.Lf * rintf(wx * b.inv_Lf);
    wy -= b.Lf * rintf(wy * b.inv_Lf);
    wz -= b.Lf * rintf(wz * b.inv_Lf);
    // closest points of w + s u (s in [0, lc]) and t v (t in [0, la]); u and v
    // are unit vectors: minimise by clamping, from the unclamped optimum
    const float la = a.move_f, lc = c.full_f;
    const float uv = c.ux * a.ux + c.uy * a.uy + c.uz * a.uz;
    const float uw = c.ux * wx + c.uy * wy + c.uz * wz, vw = a.ux * wx + a.uy * wy + a.uz * wz;
    const float den = 1.f - uv * uv;
    float s = den > 1e-6f ? (uv * vw - uw) / den : 0.f;
    s = fminf(fmaxf(s, 0.f), lc);
    float t = fminf(fmaxf(vw + s * uv, 0.f), la);
    s = fminf(fmaxf(t * uv - uw, 0.f), lc);
    t = fminf(fmaxf(vw + s * uv, 0.f), la);
    const float dx = wx + s * c.ux - t * a.ux, dy = wy + s * c.uy - t * a.uy, dz = wz + s * c.uz - t * a.uz;
    // The closest points up to the rounding of s, some 3e-7 L / den, which
    // lengthens the distance by at most den times its square over twice the
    // distance: 5e-7 L for den > 1e-3, far below the margins.
    if (dx * dx + dy * dy + dz * dz <= reach * reach) return true;
    if (den > 1e-3f) return false;
    // nearly parallel: a lower bound from the segments' middles
    const float mx = wx + 0.5f * (lc * c.ux - la * a.ux), my = wy + 0.5f * (lc * c.uy - la * a.uy),
                mz = wz + 0.5f * (lc * c.uz - la * a.uz);
    return sqrtf(mx * mx + my * my + mz * mz) <= reach + 0.5f * (la + lc);
}

// Warp 0, after the round's warps: how many steps are committed (in order),
// with their counters, the stream's advance and the box's time. Sets
// n_commit, serial, and op where the block has to go on (the round's first
// step, which was left whole).
template <class LS>
__device__ inline void rounds_decide(LS &sm, unsigned t_start) {
    const unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, K = sm.n_jobs;
    const BoxRun &R = sm.R;
    const DevBox &b = R.box;
    RunState &st = sm.st;
    const RoundJob &mine = sm.job[lane < K ? lane : 0];
    const bool sound = mine.slot >= 0 && mine.status == ST_OK;
    const bool light = sound && !mine.heavy;
    const unsigned ok = __ballot_sync(all, lane < K && light);
    const unsigned hit = __ballot_sync(all, lane < K && light && mine.contact);
    // pairs (i, j), i < j, at bit j (j - 1) / 2 + i
    int pj = 1;
    while (lane >= (pj * (pj + 1)) / 2) ++pj;
    const int pi_ = lane - (pj * (pj - 1)) / 2;
    const bool pair = pj < K && ((ok >> pj) & 1u) && ((ok >> pi_) & 1u);
    const unsigned clash = __ballot_sync(all, pair && rounds_conflict(b, sm.job[pi_], sm.job[pj]));
    int c = 0;
    while (c < K && ((ok >> c) & 1u) && ((clash >> ((c * (c - 1)) / 2)) & ((1u << c) - 1u)) == 0u) {
        ++c;
        if ((hit >> (c - 1)) & 1u) break;  // its merge ends the round
    }
    // the stop criteria that a step without event can meet
    const long long iter_limit = R.lim.n_iter_without_event_limit;
    if (iter_limit > 0) c = int(min((long long)c, max(1LL, iter_limit - st.n_iter_without_event)));
    const bool contact = c > 0 && ((hit >> (c - 1)) & 1u);
    double time = st.time, last_dt = st.inv_weight;
    if (contact) last_dt = st.inv_weight * (fp64_div(sm.job[c - 1].move, sm.job[c - 1].full) + 0.0);
    bool ended = false;
    for (int k = 0; k < c; ++k) {
        time = time + (k == c - 1 ? last_dt : st.inv_weight);
        if (dbits(R.lim.physical_time_limit) > 0 && nonneg_le(R.lim.physical_time_limit, time) &&
            !(contact && k == c - 1)) {
            c = k + 1;
            ended = true;
        }
    }
    if (ended) last_dt = st.inv_weight;
    const bool with_hit = contact && !ended;
    const int plain = c - (with_hit ? 1 : 0);  // committed steps without contact
    if (c > 0 && iter_limit > 0 && st.n_iter_without_event + plain >= iter_limit && !with_hit) ended = true;
    // cell changes: two steps that touch a common list go one after the other
    auto fine_moves = [&](const RoundJob &x) { return x.fine != x.old_fine; };
    auto cell_moves = [&](const RoundJob &x) { return x.key != x.old_key; };
    bool common = false;
    if (pair && pj < c) {
        const RoundJob &x = sm.job[pi_], &y = sm.job[pj];
        if (fine_moves(x) && fine_moves(y))
            common = x.old_fine == y.old_fine || x.old_fine == y.fine || x.fine == y.old_fine || x.fine == y.fine;
        if (cell_moves(x) && cell_moves(y))
            common = common || x.old_key == y.old_key || x.old_key == y.key || x.key == y.old_key || x.key == y.key;
    }
    const unsigned shared = __ballot_sync(all, common);
    unsigned serial = 0u;
    for (int j = 1; j < c; ++j)
        if (((shared >> ((j * (j - 1)) / 2)) & ((1u << j) - 1u)) != 0u) serial |= 1u << j;
    const bool done = lane < c;
    const int n_mov = __reduce_add_sync(all, done ? mine.n : 0), n_sc = __reduce_add_sync(all, done ? mine.scanned : 0);
    const int n_ce = __reduce_add_sync(all, done ? mine.cells : 0), n_ca = __reduce_add_sync(all, done ? mine.cands : 0);
    const int n_cs = __reduce_add_sync(all, done ? mine.cand_spheres : 0);
    const int n_re = __reduce_add_sync(all, done ? mine.refined : 0);
    // the stream: three values a step (a step that is left to the block has
    // drawn them too)
    const bool first = c == 0;  // the round's first step goes on by itself, or stops the box
    const int draws = 3 * (first ? 1 : c);
    {
        const int pos = st.rng.pos;
        if (lane < draws) {
            int k = pos + lane;
            k -= k >= 34 ? 34 : 0;
            st.rng.r[k] = sm.job[lane / 3].rnd[lane % 3];
        }
        __syncwarp();
        if (lane == 0) st.rng.pos = pos + draws >= 34 ? pos + draws - 34 : pos + draws;
    }
    if (lane == 0) {
        sm.n_commit = c;
        sm.round_n += 1;
        st.c_rounds += 1;
        st.c_round_steps += c;
        sm.round_sum += first ? 1 : c;
        sm.serial = int(serial);
        sm.commit_dt = last_dt;
        sm.op = STEP_NEXT;
        const unsigned now = clock_lo();
        st.cyc_query += now - t_start;
        if (first) {
            if (mine.slot < 0) {
                st.status = ST_UNKNOWN;  // the tree lost a live slot: stop this box
                sm.op = STEP_EXIT;
            } else if (mine.status != ST_OK) {
                st.status = mine.status;
                sm.op = STEP_EXIT;
            }
        } else {
            st.time = time;
            st.steps += plain;
            st.n_iter_without_event += plain;
            sm.left -= plain;
            if (ended) st.finished = 1;
        }
        // the step that goes on by itself: the block's, or the last committed
        // one with its contact
        const RoundJob &on = sm.job[first ? 0 : c - 1];
        sm.contact = first ? on.contact : with_hit;
        sm.slot = on.slot;
        for (int l = 0; l < 3; ++l) sm.dir[l] = on.dir[l];
        sm.full = on.full;
        sm.move = on.move;
        sm.dt = st.inv_weight;
        sm.dt_indiv = on.dt_indiv;
        sm.ms = on.ms;
        sm.os = on.os;
        sm.oslot = on.oslot;
        if (with_hit) {
            sm.mslot = on.slot;
            sm.cslot = on.oslot;
            sm.merged = 0;
            sm.try_merge = 1;
        }
        if (R.lim.with_collisions && !(first && (!sound || (mine.heavy & 1)))) {
            st.c_queries += first ? 1 : c;
            st.c_mov += first ? mine.n : n_mov;
            st.c_scanned += first ? mine.scanned : n_sc;
            st.c_cells += first ? mine.cells : n_ce;
            st.c_candidates += first ? mine.cands : n_ca;
            st.c_cand_spheres += first ? mine.cand_spheres : n_cs;
            st.c_refined += first ? mine.refined : n_re;
        }
    }
    __syncwarp();
}

// A warp without a step, while the others carry out theirs: a query read its
// lists as they were at the round's start, so what the earlier steps of the
// round moved into or out of them is added to the count of scanned aggregates,
// which is then that of the steps one after another.
template <class LS>
__device__ inline void rounds_count(LS &sm) {
    const int lane = threadIdx.x & 31, c = sm.n_commit;
    if (c < 2) return;
    const DevBox &b = sm.R.box;
    int pj = 1;  // pairs as in rounds_decide
    while (lane >= (pj * (pj + 1)) / 2) ++pj;
    int listed = 0;
    if (pj < c && !sm.live.on) {
        const RoundJob &x = sm.job[lane - (pj * (pj - 1)) / 2];
        const QueryLists &y = sm.u.r[pj].lists;
        auto in = [&](int i, int j, int k, int n) {
            return int(wrap_cell(i - y.axis[0].x, n) < (y.axis[0].y & (kFineLists - 1)) &&
                       wrap_cell(j - y.axis[1].x, n) < (y.axis[1].y & (kFineLists - 1)) &&
                       wrap_cell(k - y.axis[2].x, n) < (y.axis[2].y & (kFineLists - 1)));
        };
        auto verlet = [&](int key) { return in(key & 1023, (key >> 10) & 1023, key >> 20, b.n_div); };
        auto fine = [&](int cell) {
            // quotients by an FP32 reciprocal: exact below 2^21 cells
            const int n = b.fine_div;
            const float inv = 1.f / float(n);
            const int row = int((float(cell) + 0.5f) * inv), i = int((float(row) + 0.5f) * inv);
            return in(i, row - i * n, cell - row * n, n);
        };
        if (y.axis[0].y & kFineLists) {
            if (x.fine != x.old_fine) listed = fine(x.fine) - fine(x.old_fine);
        } else if (x.key != x.old_key) {
            listed = verlet(x.key) - verlet(x.old_key);
        }
    }
    if (!__any_sync(0xffffffffu, listed != 0)) return;
    listed = __reduce_add_sync(0xffffffffu, listed);
    if (lane == 0 && sm.R.lim.with_collisions) sm.st.c_scanned += listed;
}

template <class LS>
__device__ __noinline__ int warp_steps_call(int phase, unsigned t_phase) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    return warp_steps(*reinterpret_cast<LS *>(smem_raw), phase, t_phase);
}

// MC steps of one box in rounds, by the whole block: at most max_steps, until
// a stop criterion, an error or the deadline (checked before every round).
template <class LS>
__device__ inline void block_rounds(LS &sm, long long max_steps) {
    constexpr int kMax = LS::kRounds;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, a3 = lane < 3 ? lane : 0;
    const BoxRun &R = sm.R;
    const DevBox &b = R.box;
    RunState &st = sm.st;
    unsigned t_phase = 0;
    if (threadIdx.x == 0) {
        record_rows_init(b, sm.rec_ptr);
        sm.stop = 0;
        sm.misses = 0;
        sm.left = max_steps;
        // the criteria may have changed since the last launch; afterwards
        // they are checked at the end of every step
        if (!st.finished && st.status == ST_OK && run_finished(R, st, sm.sc.n_alive)) st.finished = 1;
        sm.merged = 0;
        sm.op = STEP_NEXT;
        // (surface reactions change every radius in every step)
        sm.seq = R.phys.growth ? INT_MAX : kRoundAlone;
        sm.back = kRoundBack;
        sm.round_n = sm.round_sum = sm.alone_n = sm.looks = 0;
        sm.round_cyc = sm.alone_cyc = 0u;
    }
    int phase = PH_START;  // the same in all threads
    __syncthreads();
    for (;;) {
        int jobs = 0;  // warps with a step to take
        bool alone = true;
        if (phase == PH_START) {
            // A round costs more than a step (its slowest query, the others on
            // the same FP64 pipes and three barriers), how much more and how
            // many steps it commits depends on the box: both forms are timed
            // as they run, in cycles a step without events' and the block's
            // work, and the slower one is only tried again now and then. The
            // results do not depend on the form.
            if (threadIdx.x == 0) {
                int k = sm.left < kMax ? int(sm.left) : kMax;
                if (sm.seq <= 0) {
                    if (sm.alone_n > 0) {
                        sm.alone_pace = float(sm.alone_cyc) / float(sm.alone_n);
                        sm.alone_n = 0;
                        sm.alone_cyc = sm.round_cyc = 0u;
                        sm.round_n = sm.round_sum = 0;
                    } else if (sm.round_n >= kRoundLook) {
                        if (float(sm.round_cyc) > sm.alone_pace * float(sm.round_sum)) {
                            sm.seq = sm.back;
                            sm.back = sm.back * 2 < kRoundBackMax ? sm.back * 2 : kRoundBackMax;
                        } else {
                            sm.back = kRoundBack;
                            if (++sm.looks % kRoundAgain == 0) sm.seq = kRoundAlone;
                        }
                        sm.round_cyc = 0u;
                        sm.round_n = sm.round_sum = 0;
                    }
                }
                if (st.finished || st.status != ST_OK || sm.stop) k = 0;
                if (k > 0 && sm.deadline != 0ULL && global_ns() >= sm.deadline) k = 0;
                sm.round_misses = sm.misses;
                sm.n_jobs = k > 0 && sm.seq > 0 ? -1 : k;  // -1: warp 0 alone
            }
            __syncthreads();
            jobs = sm.n_jobs;
            if (jobs == 0) return;  // block-uniform
            alone = jobs < 0;
            if (alone) jobs = 1;
        } else if (wid == 0) {  // a step goes on after the block's operation, and the next may follow
            const int op = warp_steps_call<LS>(phase, t_phase);
            jobs = op == STEP_NEXT && sm.seq > 0 && sm.left > 0 && !st.finished && st.status == ST_OK && !sm.stop &&
                   sm.deadline == 0ULL;
            if (lane == 0) sm.op = op;
        }
        if (wid < jobs || !alone) {
            unsigned t_start = clock_lo();
            WarpRec rec{0.0, -1};
            WarpMove mv{WarpPlace{0.0, 0.f, 0, -1}, WarpGrid{-1, -1}, -1, 0.0};
            int slot = -1;
            // counters of steps taken alone, added to the loop state at the end
            int n_done = 0, n_query = 0, quota = int(min(sm.left, 256LL)), seq = sm.seq;
            unsigned n_mov = 0, n_scanned = 0, n_cells = 0, cyc_pick = 0, cyc_scan = 0, cyc_pairs = 0, cyc_move = 0;
            // a warp's job: step wid of the round, or (warp 0 alone) one step
            // after another until the block is needed
            while (wid < jobs) {
                // rand() values 3 wid .. 3 wid + 2 from here: each lane follows
                // its own residue of three
                const int pos = st.rng.pos;
                int k = pos + a3;
                uint32_t v = st.rng.r[k >= 3 ? (k >= 37 ? k - 37 : k - 3) : k + 31];
                for (int g = 0; g <= (alone ? 0 : wid); ++g, k += 3) v += st.rng.r[k + 3 >= 34 ? k - 31 : k + 3];
                const WarpPicked p = warp_pick(sm, int(v >> 1));
                const double dl = p.dl;
                rec = p.rec;
                slot = p.slot;
                const unsigned t_pick = clock_lo();
                WarpAnswer o;
                o.distance = CUDART_INF;
                o.status = ST_OK;
                o.ms = o.os = o.oslot = -1;
                o.scanned = o.cells = o.cands = o.cand_spheres = o.refined = 0;
                o.t_scan = t_pick;
                const int n = shfl_i(rec.i, REC_N);
                const double full = shfl_d(rec.f, AGG_LPM);
                int heavy = 0;  // 1: the block's query; 2: its translation, or surface reactions
                if (slot >= 0) {
                    if (R.lim.with_collisions && !loop_query(sm, wid, slot, rec, dl, full, o)) heavy = 1;
                    if (R.phys.growth || n > kWarpMove) heavy |= 2;
                }
                const int contact = o.oslot >= 0 && dkey(o.distance) <= dkey(full);
                const double move = contact ? o.distance : full;
                const bool sound = slot >= 0 && o.status == ST_OK;
                if (sound && heavy == 0) mv = loop_prepare(sm, rec, dl, move);
                if (!alone) {
                    RoundJob &J = sm.job[wid];
                    if (lane < 3) {
                        J.rnd[lane] = v;
                        J.dir[lane] = dl;
                    }
                    const float df = float(lane == 3 ? full : (lane == 4 ? move : dl));
                    const float ux = shfl_f(df, 0), uy = shfl_f(df, 1), uz = shfl_f(df, 2);
                    const float full_f = shfl_f(df, 3), move_f = shfl_f(df, 4);
                    const double dt_indiv = shfl_d(rec.f, AGG_TIME_STEP);
                    if (lane == REC_CELL) J.old_key = rec.i;
                    if (lane == REC_FINE) J.old_fine = rec.i;
                    if (lane >= REC_F4 && lane < REC_F4 + 4) J.centre[lane - REC_F4] = __int_as_float(rec.i);
                    if (lane == 0) {
                        J.slot = slot;
                        J.status = o.status;
                        J.heavy = heavy;
                        J.n = n;
                        J.contact = contact;
                        J.ms = o.ms;
                        J.os = o.os;
                        J.oslot = o.oslot;
                        J.scanned = o.scanned;
                        J.cells = o.cells;
                        J.cands = o.cands;
                        J.cand_spheres = o.cand_spheres;
                        J.refined = o.refined;
                        J.key = mv.to.key;
                        J.fine = mv.to.fcell;
                        J.ux = ux;
                        J.uy = uy;
                        J.uz = uz;
                        J.full_f = full_f;
                        J.move_f = move_f;
                        J.full = full;
                        J.move = move;
                        J.dt_indiv = dt_indiv;
                        if (wid == 0) {
                            st.cyc_pick += t_pick - t_start;
                            st.cyc_qscan += o.t_scan - t_pick;
                            st.cyc_qpairs += clock_lo() - o.t_scan;
                            t_phase = t_pick;
                        }
                    }
                    break;
                }
                // alone: the step is committed at once
                if (lane < 3) st.rng.r[pos + lane >= 34 ? pos + lane - 34 : pos + lane] = v;
                if (lane == 0) st.rng.pos = pos >= 31 ? pos - 31 : pos + 3;
                cyc_pick += t_pick - t_start;
                if (slot >= 0 && !(heavy & 1)) {
                    n_query += 1;
                    n_mov += n;
                    n_scanned += o.scanned;
                    n_cells += o.cells;
                    if (o.cands > 0 && lane == 0) {
                        st.c_candidates += o.cands;
                        st.c_cand_spheres += o.cand_spheres;
                        st.c_refined += o.refined;
                    }
                    cyc_scan += o.t_scan - t_pick;
                    cyc_pairs += clock_lo() - o.t_scan;
                }
                t_phase = heavy & 1 ? t_pick : clock_lo();
                int go = STEP_NEXT, on = PH_START;  // where the step goes on, if not here
                if (!sound) {
                    if (lane == 0) st.status = slot < 0 ? ST_UNKNOWN : o.status;  // (the tree lost a live slot)
                    go = STEP_EXIT;
                } else if (heavy) {
                    go = heavy & 1 ? STEP_QUERY : STEP_MOVE;
                    on = PH_QUERIED;
                } else {
                    loop_move_call<LS>(slot, rec, mv, true);
                    double dt = st.inv_weight;
                    if (contact) dt = dt * (fp64_div(move, full) + 0.0);
                    const double then = (lane == AGG_TIME ? rec.f : st.time) + dt;
                    if (lane == AGG_TIME) A(b, AGG_TIME, slot) = then;
                    __syncwarp();
                    if (lane == 0) st.time = then;
                    if (contact) {
                        go = STEP_MERGE;
                        on = PH_REACTED;
                    }
                    const unsigned now = clock_lo();
                    cyc_move += now - t_phase;
                    t_phase = now;
                }
                if (go != STEP_NEXT && go != STEP_EXIT) {
                    if (lane < 3) sm.dir[lane] = dl;
                    if (lane == AGG_TIME_STEP) sm.dt_indiv = rec.f;
                    if (lane == 0) {
                        sm.slot = slot;
                        sm.full = full;
                        sm.move = move;
                        sm.contact = contact;
                        sm.dt = st.inv_weight;
                        sm.ms = o.ms;
                        sm.os = o.os;
                        sm.oslot = o.oslot;
                        sm.mslot = slot;
                        sm.cslot = o.oslot;
                        sm.merged = 0;
                        sm.try_merge = contact;
                    }
                }
                bool finished = false;
                if (go == STEP_NEXT) {
                    n_done += 1;
                    const long long iter_limit = R.lim.n_iter_without_event_limit;
                    const double time_limit = R.lim.physical_time_limit;
                    __syncwarp();
                    finished = (iter_limit > 0 && st.n_iter_without_event + n_done >= iter_limit) ||
                               (dbits(time_limit) > 0 && nonneg_le(time_limit, st.time));
                    if (finished && lane == 0) st.finished = 1;
                }
                seq -= 1;
                const bool over = go != STEP_NEXT || finished || seq <= 0 || n_done >= quota ||
                                  (sm.deadline != 0ULL && __shfl_sync(0xffffffffu, int(global_ns() >= sm.deadline), 0));
                if (over) {
                    __syncwarp();
                    if (lane == 0) {
                        sm.left -= n_done;
                        sm.seq = R.phys.growth ? INT_MAX : seq;
                        sm.alone_n += n_done + (on != PH_START ? 1 : 0);
                        sm.alone_cyc += cyc_pick + cyc_scan + cyc_pairs + cyc_move;
                        st.n_iter_without_event += n_done;
                        st.steps += n_done;
                        if (R.lim.with_collisions) {
                            st.c_queries += n_query;
                            st.c_mov += n_mov;
                            st.c_scanned += n_scanned;
                            st.c_cells += n_cells;
                        }
                        st.cyc_pick += cyc_pick;
                        st.cyc_query += cyc_scan + cyc_pairs;
                        st.cyc_qscan += cyc_scan;
                        st.cyc_qpairs += cyc_pairs;
                        st.cyc_move += cyc_move;
                    }
                    n_done = n_query = 0;
                    n_mov = n_scanned = n_cells = cyc_pick = cyc_scan = cyc_pairs = cyc_move = 0;
                    __syncwarp();
                    if (on != PH_START && go != STEP_QUERY) go = warp_steps_call<LS>(on, t_phase);
                    __syncwarp();
                    // a merge that needed no block: on to the next step
                    const bool more = go == STEP_NEXT && on != PH_START && seq > 0 && sm.left > 0 && !st.finished &&
                                      st.status == ST_OK && sm.deadline == 0ULL;
                    if (!more) {
                        if (lane == 0) sm.op = go;
                        break;
                    }
                    quota = int(min(sm.left, 256LL));
                }
                t_start = clock_lo();
            }
            if (!alone) {
                __syncthreads();
                if (wid == 0) rounds_decide(sm, __shfl_sync(0xffffffffu, t_phase, 0));
                t_phase = clock_lo();
                __syncthreads();
                const int c = sm.n_commit;
                if (wid == kMax) rounds_count(sm);  // (256 threads and more: a warp beyond the round's)
                if (wid < c) {
                    loop_move_call<LS>(slot, rec, mv, !((sm.serial >> wid) & 1));
                    const double dt = wid == c - 1 ? sm.commit_dt : st.inv_weight;
                    if (lane == AGG_TIME) A(b, AGG_TIME, slot) = rec.f + dt;
                }
                __syncthreads();
                if (wid == 0) {
                    if (sm.serial != 0 && lane == 0)
                        for (int j = 1; j < c; ++j)
                            if ((sm.serial >> j) & 1) regrid_to(b, sm.job[j].slot, sm.job[j].key, sm.job[j].fine);
                    __syncwarp();
                    const unsigned now = clock_lo();
                    if (lane == 0 && c > 0) st.cyc_move += now - t_phase;
                    if (lane == 0) sm.round_cyc += now - t_start;
                    t_phase = now;
                    int op = sm.op;
                    if (op == STEP_NEXT && c == 0)
                        op = (sm.job[0].heavy & 1) ? int(STEP_QUERY) : warp_steps_call<LS>(PH_QUERIED, t_phase);
                    else if (op == STEP_NEXT && sm.contact)
                        op = warp_steps_call<LS>(PH_REACTED, t_phase);
                    __syncwarp();
                    if (lane == 0) sm.op = op;
                }
            }
        }
        __syncthreads();
        const int op = sm.op;
        if (op == STEP_EXIT) return;  // block-uniform
        phase = op == STEP_NEXT ? int(PH_START) : block_op<LS>(op);
        __syncthreads();
    }
}

// MC steps of one box, one after another (kRounds 1): at most max_steps,
// until a stop criterion, an error or the deadline.
template <class LS>
__device__ inline void block_steps(LS &sm, long long max_steps) {
    unsigned t_phase = 0;
    int phase = PH_START;  // the same in all threads
    if (threadIdx.x == 0) {
        record_rows_init(sm.R.box, sm.rec_ptr);
        sm.stop = 0;
        sm.misses = 0;
        sm.left = max_steps;
        // the criteria may have changed since the last launch; afterwards
        // they are checked at the end of every step
        RunState &st = sm.st;
        if (!st.finished && st.status == ST_OK && run_finished(sm.R, st, sm.sc.n_alive)) st.finished = 1;
    }
    __syncthreads();
    for (;;) {
        if (threadIdx.x < 32) {
            const int op = warp_steps(sm, phase, t_phase);
            if (threadIdx.x == 0) sm.op = op;
        }
        __syncthreads();
        const int op = sm.op;
        if (op == STEP_EXIT) break;  // block-uniform
        phase = block_op<LS>(op);
        __syncthreads();
    }
}

}  // namespace mcacg
