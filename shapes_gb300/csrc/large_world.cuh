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
 * every contact of a colour in parallel, all in one cooperative launch.  Judged against the ordered path by
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
  int32_t* color;           /* [nc] colour | depth << 8, see ColourSearch */
  int32_t* color_cnt;       /* [kMaxColors + 1] */
  unsigned long long* ctl;  /* [8] ticket, timeout flag, round counter, colours used (coloured) or pass skew
                               (ordered by rows), nc, c0, round counters */
  int32_t* rowflag;         /* [nc] 1 where a contact starts a row (a run of contacts with one first body) */
  int32_t* rowoff;          /* [nc + 1] scanned rowflag: rowoff[nc] rows */
  int32_t* row_start;       /* [rows] first local contact of each row */
  int4* side;               /* [2 nc] ordered: per contact side, see k_lw_rows; coloured: the updates by colour */
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

/* Per contact: its bodies' counts, whether it was a cache hit, whether it
 * starts a row (contacts are in the reference's order, descending (i, j) with i
 * the first body, so the contacts of one first body form a contiguous run); and
 * the step's statistics: cache hits and updates (hits + iterations x contacts). */
__global__ void k_lw_count(Dev d, LW w, int iterations) {
  lw_range(w);
  int hits = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x) {
    const int c = w.c0 + k;
    const int hit = (d.c_hit[c] & kInfoHit) ? 1 : 0;
    hits += hit;
    w.hitflag[k] = hit;
    w.rowflag[k] = (k == 0 || d.c_ga[c] != d.c_ga[c - 1]) ? 1 : 0;
    for (int s = 0; s < 2; ++s) {
      const int b = lw_body(d, w, k, s);
      if (b >= 0) atomicAdd(&w.bcnt[b], 1);
    }
  }
  hits = __reduce_add_sync(0xffffffffu, hits);
  if ((threadIdx.x & 31) == 0 && hits) {
    atomicAdd(&d.counters[kCntHits], (unsigned long long)hits);
    atomicAdd(&d.counters[kCntItems], (unsigned long long)hits);
  }
  if (blockIdx.x == 0 && threadIdx.x == 0)
    atomicAdd(&d.counters[kCntItems], (unsigned long long)iterations * (unsigned long long)w.nc);
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

__device__ __forceinline__ int lw_row_of(const LW& w, int k) { return w.rowoff[k] + w.rowflag[k] - 1; }

/* What the ordered path reads per row, contact and side:
 * - the first contact of each row;
 * - the pass skew S = 1 + the largest (last row of the pass touching body b) -
 *   (row of a contact on b), over the contacts' dynamic bodies (ctl[3]).  A
 *   body's contacts are refs[bstart[b - 1] .. bstart[b]) in contact order, so
 *   its last row is the row of its last ref.  Row r of pass p + 1 then waits on
 *   nothing of pass p at a row >= r + S;
 * - per contact side (k << 1 | side): {global body, hr_b(k) or -1 for a static
 *   body, h_b - n_b + r_b(k), n_b}, so that the body's completed count wanted
 *   before the update of pass p is lw_want(e, p) with one load. */
__global__ void k_lw_rows(Dev d, LW w) {
  lw_range(w);
  int best = 0;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < w.nc; k += gridDim.x * blockDim.x) {
    const int r = lw_row_of(w, k), c = w.c0 + k;
    if (w.rowflag[k]) w.row_start[w.rowoff[k]] = k;
    for (int s = 0; s < 2; ++s) {
      const int ref = k << 1 | s, g = s ? d.c_gb[c] : d.c_ga[c];
      const int b = lw_body(d, w, k, s);
      if (b >= 0) best = max(best, lw_row_of(w, w.refs[w.bstart[b] - 1] >> 1) - r + 1);
      w.side[ref] = b >= 0 ? make_int4(g, w.hrank[ref], w.bh[b] - w.bn[b] + w.rank[ref], w.bn[b])
                           : make_int4(g, -1, 0, 0);
    }
  }
  for (int o = 16; o; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0 && best > 0) atomicMax(&w.ctl[3], (unsigned long long)best);
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
constexpr long long kPollLimit = 1ll << 22; /* polls of one dependency, or at one barrier, before giving up */
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

/* A barrier over all blocks of a cooperative launch, counting up on *arrived.
 * False when it gave up (with the default limit it never does while every block runs). */
__device__ __forceinline__ bool grid_barrier(unsigned long long* arrived, unsigned long long& target,
                                             int poll_limit) {
  __syncthreads();
  target += gridDim.x;
  bool ok = true;
  if (threadIdx.x == 0) {
    __threadfence();
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(arrived) : "memory");
    for (int n = 0;;) {
      unsigned long long now;
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(now) : "l"(arrived) : "memory");
      if (now >= target) break;
      if (++n > poll_limit) {
        ok = false;
        break;
      }
    }
  }
  return __syncthreads_and(ok);
}

/* The colouring of one contact: it takes the smallest colour its neighbours of
 * higher priority leave free, once all of those have theirs (the lower ones
 * cannot have theirs before).  Words hold colour | depth << 8, depth 1 + the
 * deepest of those neighbours: the round in which Jones and Plassmann's rounds
 * would colour it; past kColourRounds, or without a colour left, it goes to the
 * sequential colour.  The search through the neighbours stops at one still
 * missing and goes on from there the next time. */
constexpr int kColourRounds = 128;
struct ColourSearch {
  int x, end, x2, end2; /* references left on the first body, and those of the second */
  int depth;
  uint64_t used;
  __device__ __forceinline__ void begin(const Dev& d, const LW& w, int k) {
    const int a = lw_body(d, w, k, 0), b = lw_body(d, w, k, 1);
    x = a > 0 ? w.bstart[a - 1] : 0;
    end = a >= 0 ? w.bstart[a] : x;
    x2 = b > 0 ? w.bstart[b - 1] : 0;
    end2 = b >= 0 ? w.bstart[b] : x2;
    depth = 0;
    used = 0;
  }
  /* true when contact k can be coloured now, with its word */
  __device__ __forceinline__ bool go_on(const LW& w, int k, int32_t* word) {
    const uint64_t mine = ((uint64_t)lw_prio(k) << 32) | (uint32_t)k;
    for (;;) {
      if (x == end) {
        if (x2 == end2) break;
        x = x2;
        end = end2;
        x2 = end2;
      }
      const int k2 = w.refs[x] >> 1;
      if ((((uint64_t)lw_prio(k2) << 32) | (uint32_t)k2) > mine) {
        const int32_t c2 = __ldcg(w.color + k2);
        if (c2 < 0) return false;
        depth = max(depth, c2 >> 8);
        if ((c2 & 0xff) < kSeqColor) used |= 1ull << (c2 & 0xff);
      }
      ++x;
    }
    const int deep = min(depth + 1, kColourRounds + 1), col = __ffsll((long long)~used) - 1;
    *word = (deep > kColourRounds || col < 0 || col >= kSeqColor ? kSeqColor : col) | deep << 8;
    return true;
  }
};

/* Velocities and Lagrangians at L2: in one launch other SMs write them. */
struct L2Store {
  const Dev* d;
  __device__ __forceinline__ void load(int g, double& x, double& y, double& w) const {
    x = __ldcg(d->vx + g);
    y = __ldcg(d->vy + g);
    w = __ldcg(d->w + g);
  }
  __device__ __forceinline__ void store(int g, double x, double y, double w) const {
    __stcg(d->vx + g, x);
    __stcg(d->vy + g, y);
    __stcg(d->w + g, w);
  }
  __device__ __forceinline__ double* at(const int4 u, int fric) const {
    return d->lam + 2 * (size_t)((uint32_t)u.x & ~kWarmBit) + fric;
  }
  __device__ __forceinline__ double lagrangian(const int4 u, int fric) const { return __ldcg(at(u, fric)); }
  __device__ __forceinline__ void set_lagrangian(const int4 u, int fric, double x) const { __stcg(at(u, fric), x); }
};

/* The coloured solve of one large world, one cooperative launch:
 * - gravity;
 * - colouring (ColourSearch): every thread keeps trying its contacts, polling
 *   for each the neighbour it last found missing; a contact of the highest
 *   priority among its uncoloured neighbours can always be coloured, so the
 *   colouring ends without barriers between rounds;
 * - the contacts grouped by colour, the sequential ones in contact order;
 * - the warm-start pass and the sweeps, colour after colour, two lanes to an
 *   update; the sequential colour one update after another on one warp.
 * A colour's work is a few microseconds: what bounds the sweeps is the barrier
 * between colours and the latency of one round of updates, of which the
 * constants are loaded before the barrier.  A container of 65,539 bodies (165 k
 * contacts, 15 colours, 5 passes): 0.69 ms a step, 2.55 ms as a launch per
 * round and colour (459 launches). */
constexpr int kColourThreads = 512;
constexpr int kColourBlocksPerSM = 1;

__global__ void __launch_bounds__(kColourThreads, kColourBlocksPerSM)
    k_lw_coloured(Dev d, LW w, int iterations, int warm_start, int external, double ax, double ay, double dt,
                  int poll_limit) {
  if (d.counters[kCntOverflow]) return;
  lw_range(w);
  const int stride = gridDim.x * blockDim.x, t0 = blockIdx.x * blockDim.x + threadIdx.x;
  unsigned long long target = 0;
  auto barrier = [&]() {
    const bool ok = grid_barrier(&w.ctl[0], target, poll_limit);
    if (!ok && threadIdx.x == 0) atomicExch(&w.ctl[1], 1ull);
    return ok;
  };
  if (external)
    for (int b = t0; b < w.nb; b += stride) {
      const int g = w.b0 + b;
      if (!(0.0 == d.iml[g]) && !(d.flags[g] & kFlagInactive)) {
        d.vx[g] = d.vx[g] + ax * dt;
        d.vy[g] = d.vy[g] + ay * dt;
      }
    }
  for (int k = t0; k < w.nc; k += stride) __stcg(w.color + k, -1);
  if (!barrier()) return;
  {
    constexpr int kOwn = 3; /* contacts of a thread whose search is kept between its turns */
    ColourSearch search[kOwn];
    bool coloured[kOwn];
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
      const int k = t0 + i * stride;
      coloured[i] = k >= w.nc;
      if (!coloured[i]) search[i].begin(d, w, k);
    }
    int idle = 0;
    for (bool left = true; left;) {
      left = false;
      bool any = false;
      int32_t word;
#pragma unroll
      for (int i = 0; i < kOwn; ++i) {
        const int k = t0 + i * stride;
        if (!coloured[i] && search[i].go_on(w, k, &word)) {
          __stcg(w.color + k, word);
          coloured[i] = any = true;
        }
        left |= !coloured[i];
      }
      for (long long k = t0 + (long long)kOwn * stride; k < w.nc; k += stride) {
        if (__ldcg(w.color + k) >= 0) continue;
        ColourSearch fresh;
        fresh.begin(d, w, (int)k);
        if (fresh.go_on(w, (int)k, &word)) {
          __stcg(w.color + k, word);
          any = true;
        } else {
          left = true;
        }
      }
      idle = any ? 0 : idle + 1;
      if (idle > poll_limit) {
        atomicExch(&w.ctl[1], 1ull);
        break;
      }
    }
  }
  if (!barrier()) return;
  if (__syncthreads_or(__ldcg(&w.ctl[1]) != 0)) return; /* a wait gave up, here or in an earlier step */
  for (int k = t0; k < w.nc; k += stride) {
    const int col = __ldcg(w.color + k) & 0xff;
    const unsigned same = __match_any_sync(__activemask(), col);
    if ((threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&w.color_cnt[col], __popc(same));
  }
  if (!barrier()) return;
  __shared__ int32_t start[kMaxColors + 1]; /* every block its own copy */
  if (threadIdx.x == 0) {
    int run = 0;
    for (int col = 0; col < kMaxColors; ++col) {
      start[col] = run;
      run += __ldcg(w.color_cnt + col);
    }
    start[kMaxColors] = run;
  }
  if (!barrier()) return;
  /* a colour's contacts in any order: they share no dynamic body */
  auto place = [&](int at, int k) {
    const int c = w.c0 + k;
    __stcg(w.side + at, make_int4(c, d.c_ga[c], d.c_gb[c], d.c_hit[c]));
  };
  for (int k0 = t0 - (int)(threadIdx.x & 31); k0 < w.nc; k0 += stride) {
    const int lane = threadIdx.x & 31, k = k0 + lane;
    const int col = k < w.nc ? __ldcg(w.color + k) & 0xff : kSeqColor;
    const unsigned same = __match_any_sync(0xffffffffu, col);
    const int leader = __ffs(same) - 1;
    int base = 0;
    if (lane == leader && col != kSeqColor) base = atomicSub(&w.color_cnt[col], __popc(same)) - __popc(same);
    base = __shfl_sync(0xffffffffu, base, leader);
    if (col != kSeqColor) place(start[col] + base + __popc(same & ((1u << lane) - 1u)), k);
  }
  const int n_seq = start[kMaxColors] - start[kSeqColor];
  if (n_seq > 0 && blockIdx.x == 0 && threadIdx.x < 32) { /* the left-over contacts in contact order */
    int at = start[kSeqColor];
    for (int base = 0; base < w.nc; base += 32) {
      const int k = base + (int)threadIdx.x;
      const bool mine = k < w.nc && (__ldcg(w.color + k) & 0xff) == kSeqColor;
      const unsigned m = __ballot_sync(0xffffffffu, mine);
      if (mine) place(at + __popc(m & ((1u << threadIdx.x) - 1u)), k);
      at += __popc(m);
    }
  }
  if (!barrier()) return;
  const L2Store store{&d};
  /* chunks of a colour are dealt to the blocks first, then to a block's warps */
  const int warp = (int)(threadIdx.x >> 5) * gridDim.x + blockIdx.x, warps = stride >> 5, lane = threadIdx.x & 31;
  int4 u = make_int4(0, 0, 0, 0);
  LaneConstants x;
  auto fetch = [&](int at) { /* the update at place `at` of the list and its constants */
    u = __ldcg(w.side + at);
    load_pair(d, u, x);
  };
  auto update = [&](bool live, bool warm) {
    int4 v = u;
    if (warm) v.x = (int)((uint32_t)v.x | kWarmBit);
    solve_pair(d, v, x, live && !(warm && !(v.w & kInfoHit)), store);
  };
  auto first_of = [&](int col) { return start[col] + 16 * warp; };
  auto next_colour = [&](int col) { /* the next colour with contacts, around to the next pass's first */
    do {
      col = col + 1 < kSeqColor ? col + 1 : 0;
    } while (start[col] == start[col + 1]);
    return col;
  };
  const bool any_colour = start[kSeqColor] > 0;
  int col = any_colour ? next_colour(kSeqColor - 1) : 0;
  if (any_colour && first_of(col) < start[col + 1]) fetch(min(first_of(col) + (lane >> 1), start[col + 1] - 1));
  for (int pass = warm_start ? 0 : 1; pass <= iterations; ++pass) {
    for (bool more = any_colour; more;) {
      const int hi = start[col + 1];
      for (int base = first_of(col); base < hi; base += 16 * warps) {
        const int at = base + (lane >> 1);
        if (base != first_of(col)) fetch(min(at, hi - 1));
        update(at < hi, pass == 0);
      }
      const int next = next_colour(col);
      more = next > col; /* else the pass is over */
      col = next;
      if (first_of(col) < start[col + 1]) fetch(min(first_of(col) + (lane >> 1), start[col + 1] - 1));
      if (!barrier()) return;
    }
    if (n_seq > 0) {
      if (warp == 0) {
        const int4 keep_u = u;
        const LaneConstants keep_x = x;
        for (int at = start[kSeqColor]; at < start[kMaxColors]; ++at) {
          fetch(at);
          update(lane < 2, pass == 0);
          __syncwarp();
        }
        u = keep_u;
        x = keep_x;
      }
      if (!barrier()) return;
    }
  }
}

}  // namespace shapes
