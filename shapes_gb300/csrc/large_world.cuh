/*
 * Solver paths for one very large world (hundreds of thousands of bodies),
 * where a warp per world cannot expose the parallelism.
 *
 * Ordered (exact): the reference's sequence of updates — warm-start pass over
 * the cache hits, then `iterations` sweeps, each in contact order
 * (Solvers/Contact.hs:74-157) — is executed as a dataflow.  Update u touching
 * body a must run after every earlier update on a.  If r_a(u) is the number of
 * earlier updates on a, u may run exactly when a's completion counter equals
 * r_a(u).  The ranks come from each body's contacts sorted by contact order:
 * for a contact k at position r_a(k) in a's list, with h_a of a's contacts
 * being cache hits (hr_a(k) of them before k) and n_a contacts in all,
 *   warm-start pass:  r = hr_a(k)
 *   sweep p (1-based): r = h_a + (p - 1) n_a + r_a(k).
 * Contacts are in descending (i, j) order with i > j the first body, so a
 * pass is a sequence of rows, one per first body i; within a pass no update
 * after i's row touches i.  A row is one unit of work ("ticket"): eight lanes
 * wait for i's earlier updates, keep i's velocity in registers through the
 * row and wait per contact only for the second body's.  Tickets are handed out
 * in the order p S + r (pass p, row r, S the pass skew: row r of pass p + 1
 * waits on nothing of pass p at a row >= r + S), which puts every wait on an
 * earlier ticket and lets the tickets in flight cover several passes'
 * wavefronts; the earliest unfinished ticket can always run.  Lanes never
 * block: a warp polls each row's next dependency once and the rows whose
 * dependency is met run their updates together (split_update, eight lanes
 * each).
 * A velocity component travels with its body's completion count in one 16-byte
 * word, a Lagrangian with its pass, so that one load at L2 both finds whether
 * the update may run and brings its operand: no fences, no separate counters.
 * Waits are bounded: past the limit the kernel raises an error flag
 * (SHAPES_E_TIMEOUT) that stays set for the rest of the run, and stops.
 * Static bodies take no part in the ordering (they are never written).
 * Results are bit-identical to the sequential sweep.
 *
 * Coloured (not the reference's order): contacts are coloured so that no two
 * contacts of a colour share a dynamic body (Jones-Plassmann: a contact takes
 * the smallest colour free among its neighbours once its hash priority beats
 * all uncoloured neighbours), then each pass updates one colour at a time,
 * every contact of a colour in parallel.  Judged against the ordered path by
 * residual and penetration.
 */
#pragma once
#include "frontier.cuh"
#include "lw_order.cuh"

namespace shapes {

/* Per large world scratch (device). */
struct LW {
  int wld;                  /* the world */
  int b0, nb;               /* bodies [b0, b0 + nb) */
  int c0, nc;               /* contacts [c0, c0 + nc): set on the device by k_lw_setup */
  int32_t* bcnt;            /* [nb + 1] refs per body, then scanned starts, then ends */
  int32_t* bstart;          /* [nb + 1] */
  int32_t* refs;            /* [2 nc] (local contact << 1 | side), grouped by body */
  int32_t* rank;            /* [2 nc] r_s(k) */
  int32_t* hrank;           /* [2 nc] hr_s(k) */
  int32_t* bh;              /* [nb] hits per body */
  int32_t* bn;              /* [nb] contacts per body */
  ulonglong2* vel;          /* [3 nb] ordered path: {velocity component, updates of the body completed} */
  ulonglong2* lag;          /* [2 nc] ordered path: {Lagrangian, pass that wrote it} */
  int32_t* hitflag;         /* [nc] */
  int32_t* hitoff;          /* [nc + 1] scanned */
  int32_t* color;           /* [nc] */
  int32_t* color_cnt;       /* [kMaxColors + 1] then scanned */
  int32_t* color_list;      /* [nc] contacts grouped by colour */
  int32_t* seqflag;         /* [nc] 1 = left over by the colouring */
  int32_t* seqoff;          /* [nc + 1] scanned seqflag */
  int32_t* seq_list;        /* [nc] left-over contacts in contact order */
  unsigned long long* ctl;  /* [8] ticket, timeout flag, round counter, colours used (coloured) or pass skew
                               (ordered by rows), nc, c0, round counters */
  int32_t* rowflag;         /* [nc] 1 where a contact starts a row (a run of contacts with one first body) */
  int32_t* rowoff;          /* [nc + 1] scanned rowflag: rowoff[nc] rows */
  int32_t* row_start;       /* [rows] first local contact of each row */
  int4* side;               /* [2 nc] per contact side: see k_lw_side */
};

/* 16-byte words read and written whole, at L2 (other SMs write them). */
__device__ __forceinline__ ulonglong2 ld_word(const ulonglong2* p) {
  ulonglong2 v;
  asm volatile("{\n\t.reg .b128 q;\n\tld.relaxed.gpu.global.b128 q, [%2];\n\tmov.b128 {%0, %1}, q;\n\t}"
               : "=l"(v.x), "=l"(v.y)
               : "l"(p)
               : "memory");
  return v;
}

__device__ __forceinline__ void st_word(ulonglong2* p, double x, uint64_t tag) {
  asm volatile("{\n\t.reg .b128 q;\n\tmov.b128 q, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], q;\n\t}" ::"l"(p),
               "l"(__double_as_longlong(x)), "l"(tag)
               : "memory");
}

constexpr int kMaxColors = 64;
constexpr int kSeqColor = kMaxColors - 1; /* contacts left over by the colouring: updated one by one */

/* Reads the world's contact range from the device (kernels read w.c0 / w.nc
 * through lw_range) and resets the per-step state.  A timeout (ctl[1]) stays
 * raised for the rest of the run: later steps' ordered solves return at once
 * and the host reports the error. */
__global__ void k_lw_setup(Dev d, LW w) {
  const int c0 = d.world_contact_off[w.wld], c1 = d.world_contact_off[w.wld + 1];
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b <= w.nb; b += gridDim.x * blockDim.x) w.bcnt[b] = 0;
  if (blockIdx.x == 0 && threadIdx.x < 8 && threadIdx.x != 1) { /* ctl[1], the timeout flag, is cleared per run */
    const int t = threadIdx.x;
    w.ctl[t] = t == 4 ? (unsigned long long)(c1 - c0) : (t == 5 ? (unsigned long long)c0 : 0ull);
  }
  if (blockIdx.x == 0) {
    for (int t = threadIdx.x; t <= kMaxColors; t += blockDim.x) w.color_cnt[t] = 0;
  }
}

__device__ __forceinline__ void lw_range(LW& w) {
  w.nc = (int)w.ctl[4];
  w.c0 = (int)w.ctl[5];
}

/* Body of a contact side, or -1 for a static body (no ordering). */
__device__ __forceinline__ int lw_body(const Dev& d, const LW& w, int k, int side) {
  const int c = w.c0 + k;
  const uint8_t info = d.c_hit[c];
  if (side == 0) return (info & kInfoDynA) ? d.c_ga[c] - w.b0 : -1;
  return (info & kInfoDynB) ? d.c_gb[c] - w.b0 : -1;
}

__global__ void k_lw_count(Dev d, LW w) {
  lw_range(w);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x) {
    const int c = w.c0 + k;
    w.hitflag[k] = (d.c_hit[c] & kInfoHit) ? 1 : 0;
    for (int s = 0; s < 2; ++s) {
      const int b = lw_body(d, w, k, s);
      if (b >= 0) atomicAdd(&w.bcnt[b], 1);
    }
  }
}

/* bstart holds exclusive starts; the atomics turn them into ends. */
__global__ void k_lw_scatter(Dev d, LW w) {
  lw_range(w);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x) {
    for (int s = 0; s < 2; ++s) {
      const int b = lw_body(d, w, k, s);
      if (b >= 0) w.refs[atomicAdd(&w.bstart[b], 1)] = (k << 1) | s;
    }
  }
}

/* One thread per body: sort its refs by contact order, then ranks. */
__global__ void k_lw_rank(Dev d, LW w) {
  lw_range(w);
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < w.nb; b += gridDim.x * blockDim.x) {
    const int r0 = b > 0 ? w.bstart[b - 1] : 0, r1 = w.bstart[b];
    for (int x = r0 + 1; x < r1; ++x) {
      const int v = w.refs[x];
      int y = x - 1;
      while (y >= r0 && w.refs[y] > v) {
        w.refs[y + 1] = w.refs[y];
        --y;
      }
      w.refs[y + 1] = v;
    }
    int hits = 0;
    for (int x = r0; x < r1; ++x) {
      const int ref = w.refs[x];
      w.rank[ref] = x - r0;
      w.hrank[ref] = hits;
      hits += w.hitflag[ref >> 1];
    }
    w.bh[b] = hits;
    w.bn[b] = r1 - r0;
  }
}

/* The step's statistics: cache hits and updates (hits + iterations x contacts). */
__global__ void k_lw_item_counts(LW w, unsigned long long* hits, unsigned long long* items, int iterations) {
  lw_range(w);
  atomicAdd(hits, (unsigned long long)w.hitoff[w.nc]);
  atomicAdd(items, (unsigned long long)w.hitoff[w.nc] + (unsigned long long)iterations * (unsigned long long)w.nc);
}

__global__ void k_lw_gravity(Dev d, LW w, double ax, double ay, double dt) {
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < w.nb; b += gridDim.x * blockDim.x) {
    const int g = w.b0 + b;
    if (!(0.0 == d.iml[g]) && !(d.flags[g] & kFlagInactive)) {
      d.vx[g] = d.vx[g] + ax * dt;
      d.vy[g] = d.vy[g] + ay * dt;
    }
  }
}

/* One update of a contact from its record, the velocities v of its two bodies
 * (updated in place) and its accumulated Lagrangians lam2
 * (Solvers/Contact.hs:74-157; warm = the warm-start pass's application of the
 * cached impulses). */
__device__ __forceinline__ void lw_contact_math(const Con* con, double v[6], double2* lam2, bool warm) {
  const double2* cp = reinterpret_cast<const double2*>(con);
  const double2 n0 = cp[0], n1 = cp[1], f0 = cp[2], f1 = cp[3], ma = cp[7], mb = cp[8];
  const double rn[4] = {n0.x, n0.y, n1.x, n1.y}, rf[4] = {f0.x, f0.y, f1.x, f1.y}, im[4] = {ma.x, ma.y, mb.x, mb.y};
  const double2 cached = __ldcg(lam2);
  double ln = cached.x, lf = cached.y;
  if (!warm) {
    double2 now;
    contact_impulses(con, rn, rf, v, cached, &ln, &lf, &now);
    __stcg(lam2, now);
  }
  row_apply(rn, ln, v, im);
  row_apply(rf, lf, v, im);
}

/* The update of contact c (global index), with the generic velocity store. */
template <typename Store>
__device__ __forceinline__ void lw_solve_item(const Dev& d, uint32_t item, const Store& vs) {
  const int c = (int)(item & ~kWarmBit);
  const int ga = d.c_ga[c], gb = d.c_gb[c];
  double v[6];
  vs.load(ga, 0, v[0], v[1], v[2]);
  vs.load(gb, 0, v[3], v[4], v[5]);
  lw_contact_math(d.con + c, v, reinterpret_cast<double2*>(d.lam) + c, (item & kWarmBit) != 0);
  const uint8_t info = d.c_hit[c];
  if (info & kInfoDynA) vs.store(ga, 0, v[0], v[1], v[2]);
  if (info & kInfoDynB) vs.store(gb, 0, v[3], v[4], v[5]);
}

/* Rows: contacts are in the reference's order, descending (i, j) with i the
 * first body, so the contacts of one first body form a contiguous run. */
__global__ void k_lw_rowflag(Dev d, LW w) {
  lw_range(w);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x)
    w.rowflag[k] = (k == 0 || d.c_ga[w.c0 + k] != d.c_ga[w.c0 + k - 1]) ? 1 : 0;
}

__global__ void k_lw_row_list(LW w) {
  lw_range(w);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x)
    if (w.rowflag[k]) w.row_start[w.rowoff[k]] = k;
}

__device__ __forceinline__ int lw_row_of(const LW& w, int k) { return w.rowoff[k] + w.rowflag[k] - 1; }

/* Pass skew S = 1 + the largest (last row of the pass touching body b) - (row
 * of a contact on b), over the contacts' dynamic bodies (ctl[3]).  A body's
 * contacts are refs[bstart[b - 1] .. bstart[b]) in contact order, so its last
 * row is the row of its last ref.  Row r of pass p + 1 then waits on nothing
 * of pass p at a row >= r + S. */
__global__ void k_lw_skew(Dev d, LW w) {
  lw_range(w);
  int best = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x) {
    const int r = lw_row_of(w, k);
    for (int s = 0; s < 2; ++s) {
      const int b = lw_body(d, w, k, s);
      if (b >= 0) best = max(best, lw_row_of(w, w.refs[w.bstart[b] - 1] >> 1) - r + 1);
    }
  }
  for (int o = 16; o; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(&w.ctl[3], (unsigned long long)best);
}

/* Per contact side (ref = k << 1 | side): {global body, hr_b(k) or -1 for a
 * static body, h_b - n_b + r_b(k), n_b}, so that the body's completed count
 * wanted before the update of pass p is lw_want(e, p) with one load. */
__global__ void k_lw_side(Dev d, LW w) {
  lw_range(w);
  for (int ref = blockIdx.x * blockDim.x + threadIdx.x; ref < 2 * w.nc; ref += gridDim.x * blockDim.x) {
    const int k = ref >> 1, s = ref & 1;
    const int c = w.c0 + k;
    const int g = s ? d.c_gb[c] : d.c_ga[c];
    const int b = lw_body(d, w, k, s);
    w.side[ref] = b >= 0 ? make_int4(g, w.hrank[ref], w.bh[b] - w.bn[b] + w.rank[ref], w.bn[b])
                         : make_int4(g, -1, 0, 0);
  }
}

__device__ __forceinline__ int lw_want(int4 e, int pass) { return pass == 0 ? e.y : e.z + pass * e.w; }

/* The ordered path's words: velocities after gravity with no update completed,
 * Lagrangians of pass 0. */
__global__ void k_lw_begin(Dev d, LW w, int external, double ax, double ay, double dt) {
  lw_range(w);
  const int stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (int b = t0; b < w.nb; b += stride) {
    const int g = w.b0 + b;
    double vx = d.vx[g], vy = d.vy[g];
    if (external && !(0.0 == d.iml[g]) && !(d.flags[g] & kFlagInactive)) {
      vx = vx + ax * dt;
      vy = vy + ay * dt;
    }
    w.vel[3 * (size_t)b] = make_ulonglong2((uint64_t)__double_as_longlong(vx), 0);
    w.vel[3 * (size_t)b + 1] = make_ulonglong2((uint64_t)__double_as_longlong(vy), 0);
    w.vel[3 * (size_t)b + 2] = make_ulonglong2((uint64_t)__double_as_longlong(d.w[g]), 0);
  }
  for (int q = t0; q < 2 * w.nc; q += stride)
    w.lag[q] = make_ulonglong2((uint64_t)__double_as_longlong(d.lam[2 * (size_t)w.c0 + q]), 0);
}

__global__ void k_lw_end(Dev d, LW w) {
  if (d.counters[kCntOverflow]) return;
  lw_range(w);
  const int stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  for (int b = t0; b < w.nb; b += stride) {
    const int g = w.b0 + b;
    d.vx[g] = __longlong_as_double((long long)w.vel[3 * (size_t)b].x);
    d.vy[g] = __longlong_as_double((long long)w.vel[3 * (size_t)b + 1].x);
    d.w[g] = __longlong_as_double((long long)w.vel[3 * (size_t)b + 2].x);
  }
  for (int q = t0; q < 2 * w.nc; q += stride)
    d.lam[2 * (size_t)w.c0 + q] = __longlong_as_double((long long)w.lag[q].x);
}

/* The ordered solve of one large world.  Rows are tickets in the skewed order
 * (lw_ticket); eight lanes hold one row: lanes 0-2 wait for the row's first
 * body i and keep its velocity, lanes 3-5 wait for each contact's second body
 * and hand its velocity on after the update, lanes 0 and 1 do so with the
 * contact's Lagrangians; at the end of the row lanes 0-2 hand i on, its count
 * raised by the row's updates.  No lane blocks: each pass of a warp's loop
 * polls what every row still waits for once, then the rows that have all of it
 * run their update together.  A row that is finished takes the next ticket on
 * the following pass (one atomic per warp).  The earliest unfinished ticket
 * finds its dependencies met on its warp's next poll, so the solve always
 * progresses; a row that polls one dependency poll_limit times (default
 * kPollLimit, shapes_batch_set_wait_limit) raises the timeout flag and every
 * warp returns.
 * What bounds it: the chain of dependent updates, each a hand-over through L2
 * and 20 FP64 instructions of 64 cycles, and how far the rows in flight reach
 * along the ticket order.  A settled pile of 32,771 bodies (1518 levels, 562 k
 * updates a step): 7.13 ms with a row on one lane, counters beside the
 * velocities and fences between them; 3.07 ms so.  Rows in flight (rows an SM:
 * time): 4: 8.1 ms, 16: 3.83, 32: 3.32, 64: 3.07, 64 in one block: 3.29. */
constexpr int kOrderedThreads = 256;
constexpr long long kPollLimit = 1ll << 22; /* polls of one dependency before giving up */
constexpr int kOrderedBlocksPerSM = 2;

__global__ void __launch_bounds__(kOrderedThreads) k_lw_ordered(Dev d, LW w, int iterations, int warm_start,
                                                                  long long poll_limit) {
  if (d.counters[kCntOverflow]) return;
  lw_range(w);
  const unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned row_mask = 0xffu << (lane & 24), leaders_below = 0x01010101u & ((1u << (lane & 24)) - 1u);
  const SplitLane t;
  const int n_rows = w.rowoff[w.nc];
  const int passes = warm_start ? iterations + 1 : iterations;
  const long long total = (long long)passes * n_rows;
  const int skew = max(1, min((int)w.ctl[3], n_rows));
  /* the same in the eight lanes of a row */
  bool has = false, exhausted = total == 0;
  int pass = 0, k = 0, k1 = 0;
  long long polls = 0;
  /* this lane's */
  int m = 0;              /* updates of the row (lanes of i) */
  int4 side = make_int4(0, -1, 0, 0);
  bool have_v = false, have_l = false;
  double v = 0.0, cached = 0.0;
  LaneConstants x;
  const Con* con = d.con;
  int empty = 0;
  auto take_contact = [&]() { /* contact k of the row becomes current: what this lane waits for, and its constants */
    if (t.side) {
      side = w.side[(k << 1) | 1];
      have_v = false;
    }
    have_l = false;
    con = d.con + w.c0 + k;
    load_split(con, x);
  };
  for (;;) {
    if (!exhausted) { /* rows that are free take the next tickets, in order */
      const unsigned need = __ballot_sync(kAll, !has) & 0x01010101u;
      if (need) {
        unsigned long long base = 0;
        if (lane == 0) base = atomicAdd(&w.ctl[0], (unsigned long long)__popc(need));
        base = __shfl_sync(kAll, base, 0);
        const long long ticket = (long long)base + __popc(need & leaders_below);
        if (!has && ticket < total) {
          int pi, r;
          lw_ticket(ticket, passes, skew, n_rows, pi, r);
          pass = pi + (warm_start ? 0 : 1);
          k = w.row_start[r];
          k1 = r + 1 < n_rows ? w.row_start[r + 1] : w.nc;
          m = k1 - k;
          if (pass == 0) { /* the warm-start pass updates the cache hits only */
            while (k < k1 && !w.hitflag[k]) ++k;
            m = 0;
            for (int q = k; q < k1; ++q) m += w.hitflag[q];
          }
          if (m > 0) {
            has = true;
            polls = 0;
            have_v = false;
            if (!t.side) side = w.side[k << 1];
            take_contact();
          }
        }
        if ((long long)base + __popc(need) >= total) exhausted = true;
      }
    }
    if (exhausted && !__any_sync(kAll, has)) break;
    /* poll what this lane still waits for, once */
    if (has && !have_v) {
      const ulonglong2 q = ld_word(w.vel + 3 * (size_t)(side.x - w.b0) + t.k);
      have_v = side.y < 0 || q.y == (uint64_t)lw_want(side, pass);
      if (have_v) v = __longlong_as_double((long long)q.x);
    }
    if (has && !have_l) {
      const ulonglong2 q = ld_word(w.lag + 2 * (size_t)k + t.fric);
      have_l = q.y == (uint64_t)(pass > 0 ? pass - 1 : 0);
      if (have_l) cached = __longlong_as_double((long long)q.x);
    }
    const unsigned have = __ballot_sync(kAll, has & have_v & have_l);
    const bool ready = (have & row_mask) == row_mask;
    if (__any_sync(kAll, ready)) {
      double now;
      const double v1 = split_update(con, x, pass == 0, ready ? v : 0.0, ready ? cached : 0.0, &now);
      if (ready) {
        const bool dynamic = side.y >= 0;
        if (dynamic) v = v1;
        if (t.j < 2 && pass > 0) st_word(w.lag + 2 * (size_t)k + t.fric, now, (uint64_t)pass);
        if (t.side && t.j < 6 && dynamic)
          st_word(w.vel + 3 * (size_t)(side.x - w.b0) + t.k, v, (uint64_t)lw_want(side, pass) + 1);
        ++k;
        if (pass == 0)
          while (k < k1 && !w.hitflag[k]) ++k;
        polls = 0;
        if (k < k1) {
          take_contact();
        } else {
          if (!t.side && dynamic)
            st_word(w.vel + 3 * (size_t)(side.x - w.b0) + t.k, v, (uint64_t)lw_want(side, pass) + (uint64_t)m);
          has = false;
        }
      }
      empty = 0;
    } else {
      if ((++empty & 15) == 0) {
        const unsigned long long flag = *reinterpret_cast<volatile unsigned long long*>(&w.ctl[1]);
        if (__shfl_sync(kAll, flag, 0)) break; /* an update timed out */
      }
      if (empty > 64) __nanosleep(64);
    }
    if (has && !ready && ++polls > poll_limit) atomicExch(&w.ctl[1], 1ull);
  }
}

/* Jones-Plassmann colouring round over the contact graph. */
__device__ __forceinline__ uint32_t lw_prio(int k) {
  uint32_t x = (uint32_t)k * 0x9e3779b1u;
  x ^= x >> 15;
  x *= 0x85ebca6bu;
  x ^= x >> 13;
  return x;
}

/* Round r of the colouring counts the contacts it leaves uncoloured in
 * ctl[slot(r)], slots rotating over ctl[2], ctl[6], ctl[7]: round r reads
 * slot(r - 1) (a round after one that left none returns at once, so the host
 * can launch a generous number of rounds), counts into slot(r), and clears
 * slot(r + 1), which no block of round r reads. */
__device__ __forceinline__ unsigned long long* lw_round_slot(const LW& w, int round) {
  const int m = round % 3;
  return w.ctl + (m == 0 ? 2 : (m == 1 ? 6 : 7));
}

__global__ void k_lw_color_round(Dev d, LW w, int round) {
  lw_range(w);
  if (round > 0 && *lw_round_slot(w, round - 1) == 0) return;
  if (blockIdx.x == 0 && threadIdx.x == 0) *lw_round_slot(w, round + 1) = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x) {
    if (w.color[k] >= 0) continue;
    const uint64_t mine = ((uint64_t)lw_prio(k) << 32) | (uint32_t)k;
    bool top = true;
    uint64_t used = 0;
    for (int s = 0; s < 2 && top; ++s) {
      const int b = lw_body(d, w, k, s);
      if (b < 0) continue;
      const int r0 = b > 0 ? w.bstart[b - 1] : 0, r1 = w.bstart[b];
      for (int x = r0; x < r1; ++x) {
        const int k2 = w.refs[x] >> 1;
        if (k2 == k) continue;
        const int col = w.color[k2];
        if (col < 0) {
          const uint64_t other = ((uint64_t)lw_prio(k2) << 32) | (uint32_t)k2;
          if (other > mine) {
            top = false;
            break;
          }
        } else if (col < kSeqColor) {
          used |= 1ull << col;
        }
      }
    }
    if (!top) {
      atomicAdd(lw_round_slot(w, round), 1ull);
      continue;
    }
    int col = __ffsll((long long)~used) - 1;
    if (col < 0 || col >= kSeqColor) col = kSeqColor;
    w.color[k] = col;
    atomicMax(&w.ctl[3], (unsigned long long)(col + 1));
  }
}

/* After the rounds, contacts still uncoloured go to the sequential colour. */
__global__ void k_lw_color_count(LW w) {
  lw_range(w);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x) {
    if (w.color[k] < 0) w.color[k] = kSeqColor;
    atomicAdd(&w.color_cnt[w.color[k]], 1);
    w.seqflag[k] = w.color[k] == kSeqColor ? 1 : 0;
  }
}

__global__ void k_lw_color_init(LW w) {
  lw_range(w);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x) w.color[k] = -1;
}

__global__ void k_lw_color_scatter(LW w) {
  lw_range(w);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x)
    w.color_list[atomicAdd(&w.color_cnt[w.color[k]], 1)] = k;
}

/* Global velocities with plain loads/stores (one colour per launch: no other
 * update of the launch touches the same body). */
struct GlobalVel {
  const Dev* d;
  __device__ __forceinline__ void load(int g, int, double& x, double& y, double& w) const {
    x = d->vx[g];
    y = d->vy[g];
    w = d->w[g];
  }
  __device__ __forceinline__ void store(int g, int, double x, double y, double w) const {
    d->vx[g] = x;
    d->vy[g] = y;
    d->w[g] = w;
  }
};

/* The left-over contacts, in contact order (ordered compaction of seqflag). */
__global__ void k_lw_seq_list(LW w) {
  lw_range(w);
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x)
    if (w.seqflag[k]) w.seq_list[w.seqoff[k]] = k;
}

/* One colour of one pass: contacts [lo, hi) of the colour list.  The
 * left-over contacts run on one thread in contact order. */
__global__ void k_lw_color_seq(Dev d, LW w, int warm) {
  if (d.counters[kCntOverflow]) return;
  lw_range(w);
  if (blockIdx.x != 0 || threadIdx.x != 0) return;
  const int n = w.seqoff[w.nc];
  for (int t = 0; t < n; ++t) {
    const int k = w.seq_list[t];
    const int c = w.c0 + k;
    if (warm && !(d.c_hit[c] & kInfoHit)) continue;
    lw_solve_item(d, (uint32_t)c | (warm ? kWarmBit : 0u), GlobalVel{&d});
  }
}

__global__ void k_lw_color_pass(Dev d, LW w, int lo_color, int warm) {
  if (d.counters[kCntOverflow]) return;
  lw_range(w);
  const int lo = lo_color > 0 ? w.color_cnt[lo_color - 1] : 0, hi = w.color_cnt[lo_color];
  for (int t = lo + blockIdx.x * blockDim.x + threadIdx.x; t < hi; t += gridDim.x * blockDim.x) {
    const int k = w.color_list[t];
    const int c = w.c0 + k;
    if (warm && !(d.c_hit[c] & kInfoHit)) continue;
    lw_solve_item(d, (uint32_t)c | (warm ? kWarmBit : 0u), GlobalVel{&d});
  }
}

}  // namespace shapes
