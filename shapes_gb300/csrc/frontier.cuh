/*
 * The ordered solve of small worlds: dependency frontiers found while the
 * updates run.
 *
 * The reference applies warm starts, then `iterations` sweeps, strictly in
 * contact order (Solvers/Contact.hs:74-157).  Each update reads and writes only
 * its two bodies' velocities and its own Lagrangians, so running update u after
 * every earlier update that shares a non-static body with it reproduces the
 * sequential result bit for bit; static bodies are never written in the step.
 * With level(u) = 1 + max(level of the previous update on each of its dynamic
 * bodies), the updates of one level touch disjoint bodies and run together.
 * The levels pipeline the sweeps: sweep s + 1 starts on a body as soon as
 * sweep s is done with it.
 *
 * A CTA owns one solver group (whole worlds packed by the host): one warp
 * schedules, the other P warps solve, level by level.
 *
 * Scheduling.  A body's updates are the same list of contacts in every pass:
 * first the contacts it is the second body of, then the row of contacts it is
 * the first body of (contacts come in descending (i, j) order, i > j, so the
 * rows of larger first bodies come earlier).  Each body has a cursor (pass,
 * position) into that list.  A contact whose two cursors both stand on it has
 * no predecessor left: the frontier of level L + 1 is found by advancing the
 * cursors of level L's bodies, one arrival bit per contact telling the second
 * arrival from the first.  This costs work per update, not per world, needs
 * no levels stored, no sort, and no pass over the contacts beforehand but the
 * building of the lists; and because it looks at no velocity it runs ahead of
 * the solver warps.  It replaces a walk over every update in contact order
 * (or chunks of them raised to a fixed point) and a counting sort by level,
 * which together took 27-30 % of the solve (901-body stack: 1.9 of 6.6
 * million cycles; 1024 x 256 bodies: 0.63 of 2.3 million).
 *
 * Solving.  The FP64 pipe takes one warp instruction per 64 cycles and SM
 * sub-partition (76 with all four busy), whatever lanes are active, and a
 * dependent instruction can follow at once: the cost of a level is the number
 * of FP64 warp instructions its slowest warp issues.  On one lane an update is
 * 65 of them for 32 updates; on two lanes (solve_pair) 34 for sixteen, about the
 * same pipe time at half the latency; on four (solve_quad) 24 for eight; on eight
 * (solve_split) 20 for four.
 */
#pragma once
#include "step_kernels.cuh"

namespace shapes {

constexpr int kMaxGroupWorlds = 32;
constexpr int kEndRing = 64;              /* published level ends in flight */
constexpr uint32_t kSlotBits = 14;        /* shared-memory groups hold fewer than 2^14 bodies */
constexpr uint32_t kSlotMask = (1u << kSlotBits) - 1u;
constexpr int kMoves = 2;                 /* cursors a lane of the scheduling warp moves together */
constexpr int kFrontierPollLimit = 1 << 24; /* polls of a wait between a group's warps before giving up */

/* Entries of the ring that hands frontiers to the solver: a power of two, at
 * least two levels (a level has at most one update per body). */
__host__ __device__ __forceinline__ int frontier_ring(long long bodies) {
  int n = 64;
  while (n < 2 * bodies) n <<= 1;
  return n;
}

/* Bytes of shared memory a group of `bodies` bodies and `contacts` contacts
 * keeps: velocities, the per-body lists and cursor, the ring, the contacts'
 * bodies and flags, list entry and arrival bit, and with `lam` their
 * accumulated Lagrangians. */
__host__ __device__ __forceinline__ size_t frontier_bytes(long long bodies, long long contacts, bool lam) {
  return (size_t)(bodies * (24 + 4 + 8) + 2 * frontier_ring(bodies) + contacts * (8 + 2) + ((contacts + 31) >> 5) * 4 +
                  (lam ? 16 * contacts : 0) + 32);
}

/* Where a group's lists live.  In shared memory the slots and contacts are
 * numbered within the group; in global memory (a group too large for the
 * launch's shared memory) by their index in the batch.  An update is described
 * by {contact and warm bit, slot a, slot b, flags | its number in the group << 4}. */
struct SmemLists {
  uint2* info;    /* [contacts] {contact, slot a | slot b << 14 | flags << 28} */
  uint32_t* cur;  /* [bodies] pass << 16 | position; counts while the lists are built */
  uint32_t* bits; /* [contacts / 32] arrival bits */
  uint16_t* list; /* [contacts] second-body lists */
  uint16_t* unsorted;
  uint16_t* ring; /* [ring_mask + 1] contact | warm << 15 */
  uint16_t* b0;   /* [bodies] start and length of the second-body list, and of the first-body row */
  uint16_t* bn;
  uint16_t* r0;
  uint16_t* r1;
  int ring_mask;
  __device__ __forceinline__ void set_info(int q, int c, int sa, int sb, uint32_t fl) {
    info[q] = make_uint2((uint32_t)c, (uint32_t)sa | (uint32_t)sb << kSlotBits | fl << (2 * kSlotBits));
  }
  __device__ __forceinline__ uint32_t flags(int q) const { return info[q].y >> (2 * kSlotBits); }
  __device__ __forceinline__ int second(int q) const { return (int)(info[q].y >> kSlotBits & kSlotMask); }
  __device__ __forceinline__ bool arrive(int q) { /* true for the second arrival */
    const uint32_t b = 1u << (q & 31);
    return (atomicXor(&bits[q >> 5], b) & b) != 0;
  }
  __device__ __forceinline__ void set_row(int s, int first, int last, int q) {
    if (first) r0[s] = (uint16_t)q;
    if (last) r1[s] = (uint16_t)(q + 1);
  }
  __device__ __forceinline__ int pass_of(uint32_t u) const { return (int)(u >> 16); }
  __device__ __forceinline__ int pos_of(uint32_t u) const { return (int)(u & 0xffffu); }
  __device__ __forceinline__ uint32_t pack(int pass, int pos) const { return (uint32_t)pass << 16 | (uint32_t)pos; }
  __device__ __forceinline__ void put(int at, int q, bool warm) {
    ring[at & ring_mask] = (uint16_t)(q | (warm ? 0x8000 : 0));
  }
  __device__ __forceinline__ int4 get(int at) const {
    const uint32_t r = ring[at & ring_mask];
    const int q = (int)(r & 0x7fffu);
    const uint2 u = info[q];
    return make_int4((int)(u.x | ((r & 0x8000u) ? kWarmBit : 0u)), (int)(u.y & kSlotMask),
                     (int)(u.y >> kSlotBits & kSlotMask),
                     (int)(u.y >> (2 * kSlotBits) | (uint32_t)q << 4));
  }
  __device__ __forceinline__ int space(int pos, int solved) const { return ring_mask + 1 - (pos - solved); }
};

struct GlobalLists {
  int4* info;
  int4* run;     /* the group's updates, level by level */
  uint32_t* cur; /* [N] pass << 24 | position (a body has fewer than 2^24 contacts) */
  int32_t* arr;  /* [contact_cap] arrival flags */
  int32_t* list;
  int32_t* unsorted;
  int32_t* b0;
  int32_t* bn;
  int32_t* r0;
  int32_t* r1;
  __device__ __forceinline__ void set_info(int q, int c, int sa, int sb, uint32_t fl) {
    info[q] = make_int4(c, sa, sb, (int)fl);
  }
  __device__ __forceinline__ uint32_t flags(int q) const { return (uint32_t)info[q].w; }
  __device__ __forceinline__ int second(int q) const { return info[q].z; }
  __device__ __forceinline__ bool arrive(int q) { return (atomicXor(&arr[q], 1) & 1) != 0; }
  __device__ __forceinline__ void set_row(int s, int first, int last, int q) {
    if (first) r0[s] = q;
    if (last) r1[s] = q + 1;
  }
  __device__ __forceinline__ int pass_of(uint32_t u) const { return (int)(u >> 24); }
  __device__ __forceinline__ int pos_of(uint32_t u) const { return (int)(u & 0xffffffu); }
  __device__ __forceinline__ uint32_t pack(int pass, int pos) const { return (uint32_t)pass << 24 | (uint32_t)pos; }
  __device__ __forceinline__ void put(int at, int q, bool warm) {
    int4 e = info[q];
    if (warm) e.x = (int)((uint32_t)e.x | kWarmBit);
    run[at] = e;
  }
  __device__ __forceinline__ int4 get(int at) const { return run[at]; }
  __device__ __forceinline__ int space(int, int) const { return 0x7fffffff; }
};

/* Control block shared by a group's warps. */
struct FrontierCtl {
  int32_t delta[kMaxGroupWorlds];    /* slot = body + delta of its world */
  int32_t c0[kMaxGroupWorlds];       /* first contact of each world */
  int32_t coff[kMaxGroupWorlds + 1]; /* prefix of the worlds' contact counts */
  int32_t boff[kMaxGroupWorlds + 1]; /* prefix of the worlds' body counts */
  int32_t ends[kEndRing];            /* end of each published level in the group's run of gdesc */
  int32_t bump, n0, hits;
  volatile int32_t published; /* levels published */
  volatile int32_t total;     /* levels in all once known, else -1 */
  volatile int32_t done;      /* levels solved */
  volatile int32_t solved;    /* updates of those levels */
  volatile int32_t err;       /* a wait between the warps gave up */
  volatile int32_t stop;      /* the level at which the solver warps stop for it */
  unsigned long long base;
};

__device__ __forceinline__ int32_t ld_acquire_cta(const volatile int32_t* shared) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(const_cast<const int32_t*>(shared));
  int32_t v;
  asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(at) : "memory");
  return v;
}

__device__ __forceinline__ void st_release_cta(volatile int32_t* shared, int32_t v) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(const_cast<int32_t*>(shared));
  asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(at), "r"(v) : "memory");
}

__device__ __forceinline__ void solver_barrier(int threads) {
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}

/* A body's cursor on the move from (pass, pos) on to its next update, skipping
 * contacts without a cache entry in the warm-start pass.  In steps, so that a lane
 * can move several cursors with their loads in flight together. */
template <class Lists>
struct Advance {
  int s, p, pos, n, nb, r0, b0, q;
  uint32_t fl;
  bool on; /* a cursor to move, until it runs past the last pass */
  __device__ __forceinline__ void load(const Lists& ls) {
    nb = ls.bn[s];
    r0 = ls.r0[s];
    n = nb + (int)ls.r1[s] - r0;
    b0 = ls.b0[s];
  }
  __device__ __forceinline__ void next() { /* a position past the list is the first of the next pass */
    if (pos >= n) {
      pos = 0;
      ++p;
    }
  }
  __device__ __forceinline__ void contact(const Lists& ls) {
    q = pos < nb ? (int)ls.list[b0 + pos] : r0 + pos - nb;
  }
  __device__ __forceinline__ void skip(const Lists& ls, int iterations) { /* warm-start pass only */
    while (p == 0 && !(fl & kInfoHit)) {
      ++pos;
      next();
      if (p > iterations) {
        on = false;
        return;
      }
      contact(ls);
      fl = ls.flags(q);
    }
  }
  /* That update's contact when its other body already waits there (or is
   * static) so that it joins the frontier, else -1. */
  __device__ __forceinline__ int arrive(Lists& ls) {
    ls.cur[s] = ls.pack(p, pos);
    const bool both = (fl & kInfoDynA) && (fl & kInfoDynB);
    return both && !ls.arrive(q) ? -1 : q;
  }
};

/* Builds the group's lists and the first frontier (all the CTA's threads).
 * SM: slots and contacts numbered within the group. */
template <bool SM, class Lists>
__device__ __forceinline__ void frontier_build(const Dev& d, Lists& ls, FrontierCtl& ctl, const int32_t* worlds, int nw,
                                               int iterations, int p0) {
  const int NC = ctl.coff[nw], NB = ctl.boff[nw], nt = blockDim.x;
  int k = 0;
  auto slot = [&](int t) { /* t-th body of the group (t ascending per thread) */
    while (k + 1 < nw && ctl.boff[k + 1] <= t) ++k;
    return SM ? t : d.world_body_off[worlds[k]] + (t - ctl.boff[k]);
  };
  for (int t = threadIdx.x; t < NB; t += nt) {
    const int s = slot(t);
    ls.cur[s] = 0;
    ls.r0[s] = 0;
    ls.r1[s] = 0;
  }
  if constexpr (SM)
    for (int t = threadIdx.x; t < ((NC + 31) >> 5); t += nt) ls.bits[t] = 0;
  __syncthreads();
  int hits = 0;
  k = 0;
  for (int t = threadIdx.x; t < NC; t += nt) {
    while (k + 1 < nw && ctl.coff[k + 1] <= t) ++k;
    const int c = ctl.c0[k] + (t - ctl.coff[k]);
    const int q = SM ? t : c;
    const int ga = d.c_ga[c], gb = d.c_gb[c];
    const uint32_t fl = d.c_hit[c];
    const int sa = SM ? ga + ctl.delta[k] : ga, sb = SM ? gb + ctl.delta[k] : gb;
    hits += (fl & kInfoHit) ? 1 : 0;
    ls.set_info(q, c, sa, sb, fl);
    if constexpr (!SM) ls.arr[q] = 0;
    if (fl & kInfoDynB) atomicAdd(&ls.cur[sb], 1u);
    if (fl & kInfoDynA)
      ls.set_row(sa, t == ctl.coff[k] || d.c_ga[c - 1] != ga, t + 1 == ctl.coff[k + 1] || d.c_ga[c + 1] != ga, q);
  }
  hits = __reduce_add_sync(0xffffffffu, hits);
  if ((threadIdx.x & 31) == 0 && hits) atomicAdd(&ctl.hits, hits);
  __syncthreads();
  k = 0;
  for (int t = threadIdx.x; t < NB; t += nt) { /* where each list lies does not matter: any free run will do */
    const int s = slot(t);
    const uint32_t n = ls.cur[s];
    ls.bn[s] = n;
    ls.b0[s] = n ? atomicAdd(&ctl.bump, (int)n) : 0;
    ls.cur[s] = 0;
  }
  __syncthreads();
  k = 0;
  for (int t = threadIdx.x; t < NC; t += nt) {
    while (k + 1 < nw && ctl.coff[k + 1] <= t) ++k;
    const int q = SM ? t : ctl.c0[k] + (t - ctl.coff[k]);
    if (ls.flags(q) & kInfoDynB) {
      const int s = ls.second(q);
      ls.unsorted[(int)ls.b0[s] + (int)atomicAdd(&ls.cur[s], 1u)] = q;
    }
  }
  __syncthreads();
  k = 0;
  for (int t = threadIdx.x; t < NC; t += nt) { /* contact order within each list: rank by counting */
    while (k + 1 < nw && ctl.coff[k + 1] <= t) ++k;
    const int q = SM ? t : ctl.c0[k] + (t - ctl.coff[k]);
    if (!(ls.flags(q) & kInfoDynB)) continue;
    const int s = ls.second(q), b0 = ls.b0[s], n = ls.bn[s];
    int r = 0;
    for (int j = 0; j < n; ++j) r += (int)ls.unsorted[b0 + j] < q;
    ls.list[b0 + r] = q;
  }
  __syncthreads();
  k = 0;
  for (int t = threadIdx.x; t < NB; t += nt) {
    const int s = slot(t);
    Advance<Lists> a;
    a.s = s;
    a.p = p0;
    a.pos = 0;
    a.load(ls);
    if (a.n == 0 || p0 > iterations) continue;
    a.on = true;
    a.contact(ls);
    a.fl = ls.flags(a.q);
    a.skip(ls, iterations);
    if (!a.on) continue;
    const int q = a.arrive(ls);
    if (q >= 0) ls.put(atomicAdd(&ctl.n0, 1), q, a.p == 0);
  }
}

/* Waits until `ready` (a volatile read of the control block) holds; false when
 * the group gave up, after poll_limit polls here or elsewhere. */
template <class F>
__device__ __forceinline__ bool frontier_wait(FrontierCtl& ctl, int poll_limit, F&& ready) {
  for (int n = 0; n < poll_limit; ++n) {
    if (ready()) return true;
    if (ctl.err) return false;
    if (n > 64) __nanosleep(40);
  }
  ctl.err = 1;
  return false;
}

/* The scheduling warp: level after level, the frontier that the previous
 * one's updates open.  Lanes take (update, side) pairs, two each: a cursor's move
 * is a chain of six shared-memory accesses, and a level of 17 to 32 updates took
 * two of them in turn.  It waits when the ring of level ends or of updates is
 * full. */
template <class Lists>
__device__ __forceinline__ void frontier_schedule(const Dev& d, Lists& ls, FrontierCtl& ctl, int bodies,
                                                  int iterations, int poll_limit) {
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int begin = 0, end = ctl.n0, level = 0;
  while (end > begin) {
    __syncwarp();
    if (lane == 0) {
      ctl.ends[level % kEndRing] = end;
      st_release_cta(&ctl.published, level + 1);
    }
    const int need = level + 3 - kEndRing; /* levels solved before the next level's end may overwrite a slot */
    const bool room = ctl.done >= need && ls.space(end, ctl.solved) >= bodies;
    if (!__all_sync(0xffffffffu, room)) {
      const bool ok =
          frontier_wait(ctl, poll_limit, [&]() { return ctl.done >= need && ls.space(end, ctl.solved) >= bodies; });
      if (!__all_sync(0xffffffffu, ok)) break;
    }
    int pos = end;
    for (int base = begin; base < end; base += 16 * kMoves) {
      Advance<Lists> a[kMoves];
      int4 u[kMoves];
#pragma unroll
      for (int k = 0; k < kMoves; ++k) {
        const int i = base + 16 * k + (lane >> 1);
        u[k] = ls.get(min(i, end - 1));
        a[k].s = (lane & 1) ? u[k].z : u[k].y;
        a[k].on = i < end && (u[k].w & ((lane & 1) ? kInfoDynB : kInfoDynA));
      }
#pragma unroll
      for (int k = 0; k < kMoves; ++k) {
        const uint32_t cu = ls.cur[a[k].s];
        a[k].load(ls);
        a[k].p = ls.pass_of(cu);
        a[k].pos = ls.pos_of(cu) + 1;
        a[k].next();
      }
      bool last[kMoves];
#pragma unroll
      for (int k = 0; k < kMoves; ++k) {
        last[k] = a[k].on && a[k].p > iterations;
        a[k].on = a[k].on && a[k].p <= iterations;
        a[k].q = 0;
        if (a[k].on) a[k].contact(ls);
      }
#pragma unroll
      for (int k = 0; k < kMoves; ++k) a[k].fl = ls.flags(a[k].q);
#pragma unroll
      for (int k = 0; k < kMoves; ++k) {
        if (a[k].on && a[k].p == 0) {
          a[k].skip(ls, iterations);
          last[k] = !a[k].on;
        }
        int q = -1;
        if (a[k].on) q = a[k].arrive(ls);
        if (last[k]) { /* the body's last update: its world has at least this many levels */
          const int c = (int)((uint32_t)u[k].x & ~kWarmBit);
          atomicMax(&d.world_levels[d.body_world[d.c_ga[c]]], level + 1);
        }
        const unsigned m = __ballot_sync(0xffffffffu, q >= 0);
        if (q >= 0) ls.put(pos + __popc(m & below), q, a[k].p == 0);
        pos += __popc(m);
      }
    }
    begin = end;
    end = pos;
    ++level;
  }
  if (lane == 0) {
    atomicAdd(&d.counters[kCntLevels], (unsigned long long)level);
    __threadfence_block();
    ctl.total = level;
  }
}

/* Where the solver keeps a group's velocities: shared memory by slot, else
 * the batch's arrays by body; and the Lagrangians: shared memory by the
 * contact's number in the group, else the batch's array. */
template <bool SM>
struct BodyStore {
  const Dev* d;
  double* vel; /* [3 * bodies] */
  double* lam;
  bool lam_local;
  __device__ __forceinline__ double* lagrangians(const int4 u) const {
    return lam + 2 * (size_t)(SM && lam_local ? (uint32_t)u.w >> 4 : (uint32_t)u.x & ~kWarmBit);
  }
  __device__ __forceinline__ void load(int s, double& x, double& y, double& w) const {
    if (SM) {
      x = vel[3 * s]; y = vel[3 * s + 1]; w = vel[3 * s + 2];
    } else {
      x = d->vx[s]; y = d->vy[s]; w = d->w[s];
    }
  }
  __device__ __forceinline__ void store(int s, double x, double y, double w) const {
    if (SM) {
      vel[3 * s] = x; vel[3 * s + 1] = y; vel[3 * s + 2] = w;
    } else {
      d->vx[s] = x; d->vy[s] = y; d->w[s] = w;
    }
  }
  __device__ __forceinline__ double lagrangian(const int4 u, int fric) const { return lagrangians(u)[fric]; }
  __device__ __forceinline__ void set_lagrangian(const int4 u, int fric, double x) const { lagrangians(u)[fric] = x; }
  __device__ __forceinline__ double component(int s, int k) const {
    if (SM) return vel[3 * s + k];
    return k == 0 ? d->vx[s] : (k == 1 ? d->vy[s] : d->w[s]);
  }
  __device__ __forceinline__ void set_component(int s, int k, double x) const {
    if (SM) vel[3 * s + k] = x;
    else if (k == 0) d->vx[s] = x;
    else if (k == 1) d->vy[s] = x;
    else d->w[s] = x;
  }
};

__device__ __forceinline__ void prefetch_l1(const char* p) { asm volatile("prefetch.global.L1 [%0];" ::"l"(p)); }

/* An update is spread over two, four or eight lanes.  Of the lanes' rows, the even
 * lanes carry the normal row and the odd lanes the friction row: its fold, its
 * quotient and its accumulated Lagrangian `cached`.  Warm: applySln of the
 * cached Lagrangians (Solvers/Contact.hs:105-113).  Otherwise improveContactSln
 * (Solvers/Contact.hs:124-143), see contact_impulses; adding +0.0 to the
 * friction fold is the reference's `+ 0`.  update_impulse finishes an update
 * from the row's fold: the impulses (non-penetration, friction) to apply, and
 * the row's new accumulated Lagrangian. */
__device__ __forceinline__ double2 update_impulse(bool warm, double dot, double bias, double mc, double rc, double mu,
                                                  double cached, double* now) {
  const unsigned kAll = 0xffffffffu;
  const bool fric = threadIdx.x & 1;
  const double fresh = div_rn(flip_sign(dot + bias), mc, rc);
  const double neg = flip_sign(cached);
  /* even lanes: the normal impulse, clamped so that the total stays non-negative */
  const double amount = !fric & f_le(fresh, neg) ? neg : fresh;
  const double total = cached + amount;
  const double thr = __shfl_sync(kAll, total * mu, threadIdx.x & 30);
  const double held = clamp_abs(total, thr); /* odd lanes: the friction total */
  const double slide = held - cached;
  *now = fric ? held : total;
  const double mine = warm ? cached : (fric ? slide : amount);
  const double other = __shfl_xor_sync(kAll, mine, 1);
  return fric ? make_double2(other, mine) : make_double2(mine, other);
}

/* The constants of one lane's part of an update, as loaded: nothing is computed
 * from them before the update runs, so that they can be on their way while
 * another level runs. */
struct LaneConstants {
  double mc, rc, mu, bn0;
  double c[7]; /* pair: own row, the other row's arm on this lane's body, inverse masses; quad: own row on this lane's body,
                * inverse masses; split: both rows' entry, mass */
  int32_t no_bounce;
};

__device__ __forceinline__ void load_common(const Con* con, int fric, LaneConstants& x) {
  x.mc = con->mc[fric];
  x.rc = con->rc[fric];
  x.mu = con->mu;
  x.bn0 = con->bn0;
  x.no_bounce = con->no_bounce;
}

__device__ __forceinline__ const Con* con_of(const Dev& d, const int4 u) {
  return d.con + (int)((uint32_t)u.x & ~kWarmBit);
}

__device__ __forceinline__ void load_pair(const Dev& d, const int4 u, LaneConstants& x) {
  const int fric = threadIdx.x & 1;
  const Con* con = con_of(d, u);
  const double2* own = reinterpret_cast<const double2*>(con->row[fric]);
  const double2 r0 = own[0], r1 = own[1];
  const double2 im = reinterpret_cast<const double2*>(con->im)[fric];
  x.c[0] = r0.x;
  x.c[1] = r0.y;
  x.c[2] = r1.x;
  x.c[3] = r1.y;
  x.c[4] = con->row[1 - fric][2 + fric];
  x.c[5] = im.x;
  x.c[6] = im.y;
  load_common(con, fric, x);
}

/* Two lanes to an update, sixteen updates a warp: each lane folds its row from
 * all six velocity components, then moves one body (the even lane a, the odd
 * lane b).  A row's linear products are the same for both bodies but for their
 * sign: its own lane forms them and the two trade.  34 FP64 instructions for
 * sixteen updates; one lane to an update took 65 for 32, the same pipe time for
 * twice the latency. */
template <class Store>
__device__ __forceinline__ void solve_pair(const Dev& d, const int4 u, const LaneConstants& k, bool live,
                                           const Store& bs) {
  const int fric = threadIdx.x & 1;
  double v[6];
  bs.load(u.y, v[0], v[1], v[2]);
  bs.load(u.z, v[3], v[4], v[5]);
  const double cached = bs.lagrangian(u, fric);
  const double dot = row_dot(k.c, v);
  const bool bounce = !((k.no_bounce != 0) & small_velocities(v));
  double bias = fric ? 0.0 : k.bn0;
  if (__any_sync(0xffffffffu, bounce)) { /* some update of the warp has a restitution term */
    if (bounce && !fric) bias = con_of(d, u)->bn + bounce_term(con_of(d, u), v);
  }
  const bool warm = ((uint32_t)u.x & kWarmBit) != 0;
  double now;
  const double2 l = update_impulse(warm, dot, bias, k.mc, k.rc, k.mu, cached, &now);
  if (live & !warm) bs.set_lagrangian(u, fric, now);
  const double mine = fric ? l.y : l.x;
  const double px = k.c[0] * mine, py = k.c[1] * mine; /* on b; the negative on a */
  const double qx = __shfl_xor_sync(0xffffffffu, px, 1), qy = __shfl_xor_sync(0xffffffffu, py, 1);
  const double nx = fric ? qx : flip_sign(px), ny = fric ? qy : flip_sign(py), na = fric ? k.c[4] : k.c[2];
  const double fx = fric ? px : flip_sign(qx), fy = fric ? py : flip_sign(qy), fa = fric ? k.c[3] : k.c[4];
  double x = fric ? v[3] : v[0], y = fric ? v[4] : v[1], w = fric ? v[5] : v[2];
  x = x + nx * k.c[5];
  y = y + ny * k.c[5];
  w = w + (na * l.x) * k.c[6];
  x = x + fx * k.c[5];
  y = y + fy * k.c[5];
  w = w + (fa * l.y) * k.c[6];
  if (live && (u.w & (fric ? kInfoDynB : kInfoDynA))) bs.store(fric ? u.z : u.y, x, y, w);
}

/* Lane j of eight: velocity component, and side and component of the body it
 * belongs to.  Lanes 6 and 7 repeat 4 and 5 and store nothing. */
struct SplitLane {
  int j, side, k, fric;
  __device__ __forceinline__ SplitLane() {
    j = threadIdx.x & 7;
    const int comp = j < 6 ? j : j - 2;
    side = comp >= 3;
    k = comp - 3 * side;
    fric = j & 1;
  }
};

__device__ __forceinline__ void load_split(const Con* con, LaneConstants& x) {
  const SplitLane t;
  const int at = t.k < 2 ? t.k : 2 + t.side;
  x.c[0] = con->row[0][at];
  x.c[1] = con->row[1][at];
  x.c[2] = con->im[2 * t.side + (t.k == 2)];
  load_common(con, t.fric, x);
}

/* Eight lanes to an update, four updates a warp (all 32 lanes call it, live or
 * not): from this lane's velocity component v0 and its row's Lagrangian, the
 * new component and Lagrangian.  The lanes' products change places so that
 * every even lane has the normal row's six and every odd lane the friction
 * row's.  20 FP64 instructions. */
__device__ __forceinline__ double split_update(const Con* con, const LaneConstants& x, bool warm, double v0,
                                               double cached, double* now) {
  const unsigned kAll = 0xffffffffu;
  const SplitLane t;
  const bool flip = t.side == 0 && t.k < 2;
  const double jn = flip ? flip_sign(x.c[0]) : x.c[0], jf = flip ? flip_sign(x.c[1]) : x.c[1], m = x.c[2];
  const double pn = jn * v0, pf = jf * v0;
  /* pairs of lanes trade: an even lane 2 i ends with the normal row's products 2 i and 2 i + 1, its neighbour with the
   * friction row's */
  const double got = __shfl_xor_sync(kAll, t.fric ? pn : pf, 1);
  const double lo = t.fric ? got : pn, hi = t.fric ? pf : got;
  double dot = __shfl_sync(kAll, lo, t.fric, 8);
  dot = dot + __shfl_sync(kAll, hi, t.fric, 8);
  dot = dot + __shfl_sync(kAll, lo, 2 + t.fric, 8);
  dot = dot + __shfl_sync(kAll, hi, 2 + t.fric, 8);
  dot = dot + __shfl_sync(kAll, lo, 4 + t.fric, 8);
  dot = dot + __shfl_sync(kAll, hi, 4 + t.fric, 8);
  const unsigned slow = __ballot_sync(kAll, !((x.no_bounce != 0) & small_mag(v0)));
  double bias = t.fric ? 0.0 : x.bn0;
  if (slow) { /* some update of the warp has a restitution term */
    double v[6];
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] = __shfl_sync(kAll, v0, q, 8);
    if (!t.fric && ((slow >> (threadIdx.x & 24)) & 0xffu)) bias = con->bn + bounce_term(con, v);
  }
  const double2 l = update_impulse(warm, dot, bias, x.mc, x.rc, x.mu, cached, now);
  const double v1 = v0 + (jn * l.x) * m;
  return v1 + (jf * l.y) * m;
}

template <bool SM>
__device__ __forceinline__ void solve_split(const Dev& d, const int4 u, const LaneConstants& x, bool live,
                                            const BodyStore<SM>& bs) {
  const SplitLane t;
  const int s = t.side ? u.z : u.y;
  const bool warm = ((uint32_t)u.x & kWarmBit) != 0;
  double now;
  const double v1 = split_update(con_of(d, u), x, warm, bs.component(s, t.k), bs.lagrangian(u, t.fric), &now);
  if (live & !warm & (t.j < 2)) bs.set_lagrangian(u, t.fric, now);
  if (live && t.j < 6 && (u.w & (t.side ? kInfoDynB : kInfoDynA))) bs.set_component(s, t.k, v1);
}

/* Four lanes to an update, eight updates a warp (all 32 lanes call it, live or
 * not): lane 2 * side + fric has its row's three entries on its side's body.  The
 * second side continues the first one's fold; a lane forms the three changes that
 * its row makes to its side's body, and the two lanes of a side trade: the normal
 * one moves x and y, the friction one w.  24 FP64 instructions: for levels of
 * 17 to 32 updates that is one chunk per sub-partition, where two lanes to an
 * update keep half of them idle for 34 (a step of 901 stacked bodies, 27 updates
 * a level: 715 -> 671 us), and a remainder of five to eight costs 24 instead of
 * 34 (4096 worlds of columns 715 -> 672 us).  In all three forms the fold comes
 * before the test for a restitution term: a branch ahead of it would keep the
 * other instructions out of the FP64 ones' shadow. */
__device__ __forceinline__ void load_quad(const Con* con, LaneConstants& x) {
  const int fric = threadIdx.x & 1, side = (threadIdx.x >> 1) & 1;
  const double2 lin = *reinterpret_cast<const double2*>(con->row[fric]);
  const double2 im = reinterpret_cast<const double2*>(con->im)[side];
  x.c[0] = lin.x;
  x.c[1] = lin.y;
  x.c[2] = con->row[fric][2 + side];
  x.c[3] = im.x;
  x.c[4] = im.y;
  load_common(con, fric, x);
}

template <bool SM>
__device__ __forceinline__ void solve_quad(const Dev& d, const int4 u, const LaneConstants& k, bool live,
                                           const BodyStore<SM>& bs) {
  const unsigned kAll = 0xffffffffu;
  const int fric = threadIdx.x & 1, side = (threadIdx.x >> 1) & 1;
  const int s = side ? u.z : u.y;
  const bool warm = ((uint32_t)u.x & kWarmBit) != 0;
  double x, y, w;
  bs.load(s, x, y, w);
  const double cached = bs.lagrangian(u, fric);
  const double jx = side ? k.c[0] : flip_sign(k.c[0]), jy = side ? k.c[1] : flip_sign(k.c[1]), ja = k.c[2];
  const double px = jx * x, py = jy * y, pw = ja * w;
  const double first = (px + py) + pw; /* of the first side */
  double dot = ((__shfl_sync(kAll, first, fric, 4) + px) + py) + pw; /* of the second */
  dot = __shfl_sync(kAll, dot, 2 + fric, 4);
  const unsigned slow = __ballot_sync(kAll, !((k.no_bounce != 0) & small_mag(x) & small_mag(y) & small_mag(w)));
  double bias = fric ? 0.0 : k.bn0;
  if (slow) { /* some update of the warp has a restitution term */
    double v[6];
#pragma unroll
    for (int q = 0; q < 2; ++q) {
      v[3 * q] = __shfl_sync(kAll, x, 2 * q, 4);
      v[3 * q + 1] = __shfl_sync(kAll, y, 2 * q, 4);
      v[3 * q + 2] = __shfl_sync(kAll, w, 2 * q, 4);
    }
    const Con* con = con_of(d, u);
    if (!fric && ((slow >> (threadIdx.x & 28)) & 0xfu)) bias = con->bn + bounce_term(con, v);
  }
  double now;
  const double2 l = update_impulse(warm, dot, bias, k.mc, k.rc, k.mu, cached, &now);
  if (live & !warm & (side == 0)) bs.set_lagrangian(u, fric, now);
  const double mine = fric ? l.y : l.x;
  /* the row's linear products, the same for both sides but for their sign: x by the second side, y by the first */
  const double half = (side ? k.c[0] : k.c[1]) * mine, traded = __shfl_xor_sync(kAll, half, 2);
  const double dx = (side ? half : flip_sign(traded)) * k.c[3], dy = (side ? traded : flip_sign(half)) * k.c[3];
  const double dw = (ja * mine) * k.c[4];
  const double got = __shfl_xor_sync(kAll, fric ? dx : dw, 1), got_y = __shfl_xor_sync(kAll, dy, 1);
  double a = fric ? w : x;
  a = a + (fric ? got : dx);
  a = a + (fric ? dw : got);
  y = y + dy;
  y = y + got_y;
  if (live && (u.w & (side ? kInfoDynB : kInfoDynA))) {
    bs.set_component(s, fric ? 2 : 0, a);
    if (!fric) bs.set_component(s, 1, y);
  }
}

/* How a level of `count` updates is dealt: first `pairs` chunks of sixteen
 * updates with two lanes each, then `quads` of eight with four, then the rest
 * four to a warp with eight (34, 24 and 20 FP64 instructions a chunk). */
struct Deal {
  int pairs, quads, units;
  __device__ __forceinline__ Deal(int count, int split_limit) {
    int split = 0;
    pairs = quads = 0;
    if (count <= split_limit) {
      split = count;
    } else if (count <= 2 * split_limit) { /* as many chunks as the line above has */
      quads = (count + 7) >> 3;
    } else {
      const int rest = count & 15;
      if (rest <= 4) split = rest;
      else if (rest <= 8) quads = 1;
      pairs = (count - split - (quads ? rest : 0) + 15) >> 4;
    }
    units = pairs + quads + ((split + 3) >> 2);
  }
  /* unit t's update of this lane, counted from the level's begin */
  __device__ __forceinline__ int at(int t, int lane) const {
    if (t < pairs) return 16 * t + (lane >> 1);
    if (t < pairs + quads) return 16 * pairs + 8 * (t - pairs) + (lane >> 2);
    return 16 * pairs + 8 * quads + 4 * (t - pairs - quads) + (lane >> 3);
  }
};

/* The solver warps: every published level (see split_limit).  A level is dealt
 * to the warps starting half of them further each level: a partly filled chunk
 * does not always fall to the same sub-partition, and where a level keeps at
 * most half of the warps busy the others prepare the next one.  Preparing, if
 * that level is published, is reading which updates the warp's first unit has
 * and sending for their constants: into registers (kStage: a group with an SM
 * to itself, where nothing else hides that latency and registers are plenty),
 * else to L1. */
template <int P, bool SM, class Lists>
__device__ __forceinline__ void frontier_solve(const Dev& d, FrontierCtl& ctl, const Lists& ls,
                                               const BodyStore<SM>& bs, int split_limit, int poll_limit) {
  constexpr bool kStage = P == 8;
  constexpr int kTurn = P > 1 ? P / 2 : 1;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  /* this lane's update of unit t of the level [begin, end) */
  auto update_of = [&](const Deal& deal, int t, int begin, int end, bool* live) {
    const int i = begin + deal.at(t, lane);
    *live = i < end;
    return ls.get(min(i, end - 1));
  };
  auto load = [&](const Deal& deal, int t, const int4 u, LaneConstants& k) {
    if (t < deal.pairs) load_pair(d, u, k);
    else if (t < deal.pairs + deal.quads) load_quad(con_of(d, u), k);
    else load_split(con_of(d, u), k);
  };
  int begin = 0;
  bool ahead = false, live = false;
  int4 u = make_int4(0, 0, 0, 0);
  LaneConstants k;
  int known = 0; /* levels that this warp has seen published */
  for (int level = 0;; ++level) {
    if (wib == 0 && known <= level) {
      const bool ok = frontier_wait(
          ctl, poll_limit, [&]() { return ld_acquire_cta(&ctl.published) > level || ld_acquire_cta(&ctl.total) >= 0; });
      if (!__all_sync(0xffffffffu, ok) && lane == 0) ctl.stop = level; /* every warp stops at the same level */
    }
    solver_barrier(32 * P); /* the level before is solved, this one is published */
    const int published = ld_acquire_cta(&ctl.published);
    if (ctl.stop <= level || published <= level) break; /* published holds all levels once total is known */
    if (threadIdx.x == 0) {
      ctl.solved = begin;
      ctl.done = level;
    }
    const int end = ctl.ends[level % kEndRing];
    const Deal deal(end - begin, split_limit);
    const int first = (wib + kTurn * level) % P;
    if (first < deal.units) {
      if (!ahead) u = update_of(deal, first, begin, end, &live);
      if (!(kStage && ahead)) load(deal, first, u, k);
    }
    for (int t = first; t < deal.units; t += P) {
      if (t != first) {
        u = update_of(deal, t, begin, end, &live);
        load(deal, t, u, k);
      }
      if (t < deal.pairs) solve_pair(d, u, k, live, bs);
      else if (t < deal.pairs + deal.quads) solve_quad(d, u, k, live, bs);
      else solve_split(d, u, k, live, bs);
    }
    known = published;
    ahead = known > level + 1;
    if (ahead) {
      const int end2 = ctl.ends[(level + 1) % kEndRing];
      const Deal deal2(end2 - end, split_limit);
      const int t = (wib + kTurn * (level + 1)) % P;
      if (t < deal2.units) {
        u = update_of(deal2, t, end, end2, &live);
        if constexpr (kStage) load(deal2, t, u, k);
        else prefetch_l1(reinterpret_cast<const char*>(con_of(d, u)) + ((lane & 1) ? kConHot - 8 : 0));
      }
    }
    begin = end;
  }
}

/* Step 1 is applyExternal (World.hs:156-158, constantAccel External.hs:23-28)
 * on the group's bodies.  Groups come sorted heaviest first; with heavy_first
 * = h > 0 the first h CTAs (one wave over the SMs) take the h heaviest groups
 * and the rest take the others lightest first, so that a heavy group starts
 * beside light ones instead of beside the next heaviest.
 *
 * split_limit: levels of at most this many updates run eight lanes to an
 * update, of at most twice as many four: sixteen for a group alone on its SM (so
 * that a level is one chunk on each of the four sub-partitions), four where
 * several groups share the SM and the pipe's total work counts. */
template <int P>
__global__ void __launch_bounds__(32 * (P + 1), P == 8 ? 1 : (P == 4 ? 4 : 6))
    k_frontier(Dev d, int iterations, int warm_start, int external, double ax, double ay, double dt, int n_groups,
               int smem_bytes, int heavy_first, int split_limit, int poll_limit) {
  chained_wait(); /* the next kernel's blocks would hold places through the whole solve, that other streams can use */
  extern __shared__ __align__(16) unsigned char s_dyn[];
  __shared__ FrontierCtl ctl;
  if (d.counters[kCntOverflow]) return; /* buffers incomplete: the host retries */
  const int tid = threadIdx.x, nt = blockDim.x;
  const int hf = min(heavy_first, n_groups);
  const int grp = (int)blockIdx.x < hf ? (int)blockIdx.x : n_groups - 1 - ((int)blockIdx.x - hf);
  if (grp >= n_groups) return;
  const int o0 = d.group_world_off[grp], nw = d.group_world_off[grp + 1] - o0;
  const int32_t* worlds = d.group_worlds + o0;
  const int p0 = warm_start ? 0 : 1;
  if (d.phase_clock && tid == 0) d.phase_clock[8 * grp + 0] = clock64();
  if (tid == 0) {
    int nb = 0, nc = 0;
    for (int k = 0; k < nw; ++k) {
      const int w = worlds[k], b0 = d.world_body_off[w], c0 = d.world_contact_off[w];
      ctl.delta[k] = nb - b0;
      ctl.c0[k] = c0;
      ctl.boff[k] = nb;
      ctl.coff[k] = nc;
      nb += d.world_body_off[w + 1] - b0;
      nc += d.world_contact_off[w + 1] - c0;
    }
    ctl.boff[nw] = nb;
    ctl.coff[nw] = nc;
    ctl.bump = ctl.n0 = ctl.hits = 0;
    ctl.published = ctl.done = ctl.solved = ctl.err = 0;
    ctl.total = -1;
    ctl.stop = 0x7fffffff;
    ctl.base = atomicAdd(&d.counters[kCntGroupAlloc], (unsigned long long)(iterations + 1) * nc + 1);
  }
  if (tid < nw) d.world_levels[worlds[tid]] = 0;
  __syncthreads();
  const int NB = ctl.boff[nw], NC = ctl.coff[nw];
  const bool fits = NB <= (int)kSlotMask && NC < 32768 && NC <= 12 * NB &&
                    frontier_bytes(NB, NC, false) <= (size_t)smem_bytes;
  const bool lam_local = fits && frontier_bytes(NB, NC, true) <= (size_t)smem_bytes;
  unsigned char* p = s_dyn;
  double* vel = reinterpret_cast<double*>(p);
  p += (size_t)((NB + 1) & ~1) * 24;
  double* lam = d.lam;
  SmemLists ls;
  GlobalLists lg;
  if (fits) {
    if (lam_local) {
      lam = reinterpret_cast<double*>(p);
      p += (size_t)NC * 16;
    }
    ls.info = reinterpret_cast<uint2*>(p);
    p += (size_t)NC * 8;
    ls.cur = reinterpret_cast<uint32_t*>(p);
    p += (size_t)NB * 4;
    ls.bits = reinterpret_cast<uint32_t*>(p);
    p += (size_t)((NC + 31) >> 5) * 4;
    ls.ring_mask = frontier_ring(NB) - 1;
    ls.ring = reinterpret_cast<uint16_t*>(p);
    ls.list = ls.ring + ls.ring_mask + 1;
    ls.b0 = ls.list + NC;
    ls.bn = ls.b0 + NB;
    ls.r0 = ls.bn + NB;
    ls.r1 = ls.r0 + NB;
    ls.unsorted = reinterpret_cast<uint16_t*>(vel); /* before the velocities move in */
    frontier_build<true>(d, ls, ctl, worlds, nw, iterations, p0);
  } else {
    lg.info = d.sched_info;
    lg.run = d.gdesc + ctl.base;
    lg.cur = d.sched_cur;
    lg.arr = d.sched_arr;
    if (tid == 0) ctl.bump = (int)atomicAdd(&d.counters[kCntListAlloc], (unsigned long long)NC);
    lg.list = d.sched_list;
    lg.unsorted = d.sched_list + d.contact_cap;
    lg.b0 = d.sched_body;
    lg.bn = d.sched_body + (size_t)d.n_bodies;
    lg.r0 = d.sched_body + 2 * (size_t)d.n_bodies;
    lg.r1 = d.sched_body + 3 * (size_t)d.n_bodies;
    __syncthreads();
    frontier_build<false>(d, lg, ctl, worlds, nw, iterations, p0);
  }
  {
    int k = 0;
    for (int t = tid; t < NB; t += nt) {
      while (k + 1 < nw && ctl.boff[k + 1] <= t) ++k;
      const int g = d.world_body_off[worlds[k]] + (t - ctl.boff[k]);
      double vx = d.vx[g], vy = d.vy[g];
      const double im = d.iml[g];
      if (external && !(0.0 == im) && !(d.flags[g] & kFlagInactive)) {
        vx = vx + ax * dt;
        vy = vy + ay * dt;
        if (!fits) {
          d.vx[g] = vx;
          d.vy[g] = vy;
        }
      }
      if (fits) {
        vel[3 * t] = vx;
        vel[3 * t + 1] = vy;
        vel[3 * t + 2] = d.w[g];
      }
    }
    k = 0;
    if (lam_local)
      for (int t = tid; t < NC; t += nt) {
        while (k + 1 < nw && ctl.coff[k + 1] <= t) ++k;
        reinterpret_cast<double2*>(lam)[t] = reinterpret_cast<const double2*>(d.lam)[ctl.c0[k] + (t - ctl.coff[k])];
      }
  }
  __syncthreads();
  if (d.phase_clock && tid == 0) d.phase_clock[8 * grp + 1] = clock64();
  if (tid >= 32 * P) { /* the scheduling warp */
    if (tid == 32 * P) {
      const unsigned long long h = warm_start ? (unsigned long long)ctl.hits : 0ull;
      atomicAdd(&d.counters[kCntHits], h);
      atomicAdd(&d.counters[kCntItems], h + (unsigned long long)iterations * NC);
    }
    if (fits) frontier_schedule(d, ls, ctl, NB, iterations, poll_limit);
    else frontier_schedule(d, lg, ctl, NB, iterations, poll_limit);
    if (d.phase_clock && tid == 32 * P) d.phase_clock[8 * grp + 2] = clock64();
    return;
  }
  if (fits) frontier_solve<P>(d, ctl, ls, BodyStore<true>{&d, vel, lam, lam_local}, split_limit, poll_limit);
  else frontier_solve<P>(d, ctl, lg, BodyStore<false>{&d, nullptr, lam, false}, split_limit, poll_limit);
  if (ctl.err && tid == 0) atomicOr(&d.counters[kCntSolveErr], 1ull);
  {
    int k = 0;
    if (fits)
      for (int t = tid; t < NB; t += 32 * P) {
        while (k + 1 < nw && ctl.boff[k + 1] <= t) ++k;
        const int g = d.world_body_off[worlds[k]] + (t - ctl.boff[k]);
        d.vx[g] = vel[3 * t];
        d.vy[g] = vel[3 * t + 1];
        d.w[g] = vel[3 * t + 2];
      }
    k = 0;
    if (lam_local)
      for (int t = tid; t < NC; t += 32 * P) {
        while (k + 1 < nw && ctl.coff[k + 1] <= t) ++k;
        reinterpret_cast<double2*>(d.lam)[ctl.c0[k] + (t - ctl.coff[k])] = reinterpret_cast<const double2*>(lam)[t];
      }
  }
  if (d.phase_clock && tid == 0) {
    d.phase_clock[8 * grp + 3] = clock64();
    d.phase_clock[8 * grp + 4] = ctl.total;
    d.phase_clock[8 * grp + 5] = (warm_start ? ctl.hits : 0) + iterations * NC;
    d.phase_clock[8 * grp + 6] = NB;
    d.phase_clock[8 * grp + 7] = nw;
  }
}

}  // namespace shapes
