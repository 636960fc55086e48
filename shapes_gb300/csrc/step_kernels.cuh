/*
 * Device kernels of the GB300 world step.
 *
 * Arithmetic contract (shared with the CPU oracle): IEEE binary64, every sum a
 * left fold in the reference's source order, no contraction (-fmad=false), the
 * reference's comparison spellings.  Floating-point comparisons whose only job
 * is ordering (AABB overlap) are done on order-preserving 64-bit integer keys,
 * which give the same answers as the IEEE comparisons for every non-NaN value;
 * NaN operands take the IEEE path.  On GB300 the FP64 pipe retires about 0.05
 * warp-instructions per clock per SM and charges masked-off lanes in full, so
 * every kernel here keeps warps full across its FP64 work and moves what it
 * can to the integer pipes.
 */
#pragma once
#include <cstdint>

#include "fp64_ops.cuh"
#include "scan.cuh"
#include "shapes_sincos.h"

namespace shapes {

constexpr int kMaxVerts = 64;
constexpr uint32_t kWarmBit = 0x80000000u;
constexpr uint8_t kFlagStatic = 1;
constexpr uint8_t kFlagBoxNaN = 2;
constexpr uint8_t kFlagInactive = 4; /* empty slot (World.delete): no pairs, no motion */
constexpr uint8_t kFlagCircle = 8;
/* per-contact info byte */
constexpr uint8_t kInfoHit = 1;
constexpr uint8_t kInfoDynA = 2;
constexpr uint8_t kInfoDynB = 4;

/* Per-contact constraint data, built once per step (constraintGen,
 * Constraints/Contact.hs:60-72) plus the step-invariant factors of the solver:
 * effective-mass denominators (effMassM2, Constraint.hs:173-179), pairMu
 * (Friction.hs:46-48) and min bounciness (Restitution.hs:51). */
struct __align__(16) Con {
  /* normal and friction row, {x, y, angular of a, angular of b}: the Jacobian
   * row is (-x, -y, angular of a, x, y, angular of b), because the normal and the
   * tangent enter the two bodies with opposite signs and a Flip only swaps the
   * halves */
  double row[2][4];
  double mc[2];       /* effective-mass denominators */
  double rc[2];       /* RN(1 / mc) for div_rn, or 0 when out of its range */
  double mu, bn0;     /* bn0 = bn + 0.0 */
  double im[4];       /* inverse masses: linear and rotational of a, then of b */
  int32_t no_bounce;  /* 1 when e is a zero, both radii are below 2^500 and the normal below 2: the bounce term is +0
                         for velocities below 2^500 */
  int32_t pad;
  double bn;          /* baumgarte term */
  /* a solver needs the 160 bytes above, two 128-byte lines wherever the record starts */
  double e;
  double ra[4];       /* contact point from a's and from b's position */
  double rn[2];
};
static_assert(sizeof(Con) == 224, "records start on 32-byte sectors");
constexpr int kConHot = 160;

/* Device view of a batch; passed by value to every kernel. */
struct Dev {
  int32_t n_worlds, n_bodies, n_verts;
  int32_t pair_cap, contact_cap, item_cap;
  const int32_t* world_body_off; /* [W+1] */
  const int32_t* body_world;     /* [N] */
  const int32_t* vert_off;       /* [N+1] */
  const double* lx;
  const double* ly;
  int32_t* emin;
  int32_t* emax;
  double* vx;
  double* vy;
  double* w;
  double* px;
  double* py;
  double* th;
  const double* iml;
  const double* imr;
  const double* mu;
  const double* bounce;
  double* wx;
  double* wy;
  double* nx;
  double* ny;
  float4* vf;       /* [V] posed vertex and its edge's normal in binary32 (the narrowphase's filter) */
  float2* ef;       /* [V] per edge: least and largest projection of its hull on its normal in binary32 */
  double* box;      /* [4N] x0 x1 y0 y1 */
  uint64_t* boxk;   /* [4N] ordered keys of box */
  uint8_t* flags;   /* [N] */
  /* grid broadphase (worlds with grid_T[w] > 0) */
  const int32_t* grid_T;    /* [W] bucket table size (power of two), 0 = brute force */
  const int32_t* grid_base; /* [W] first bucket of the world */
  double* grid_inv_s;       /* [W] 1 / cell size, 0 = no usable grid this step */
  double* grid_lim;         /* [W] (1 - 2^-20) * cell size: bodies below it in x and y use the grid */
  int32_t* bucket_cnt;      /* [n_buckets + 1] counts, then scanned offsets */
  int32_t* bucket_off;      /* [n_buckets + 1] */
  int4* grid_ent;           /* [N] {body, cell x, cell y, flags} sorted by bucket: all that a searching row needs of
                             * a candidate in another cell, in one access where id, cells and flags were four */
  int2* cell;               /* [N] */
  uint8_t* row_mode;        /* [N] 1 = row found through the grid */
  int32_t* large_cnt;       /* [W] bodies of the world off the grid */
  int32_t* large_ids;       /* [N] per-world region at world_body_off[w] */
  int32_t n_buckets;
  /* incremental grid pairs (fat boxes); null when off */
  uint64_t* fatk;        /* [4N] ordered keys of each grid body's fat box */
  int32_t* nbr;          /* [N * nbr_cap] bodies whose fat boxes overlap (either index); -1 = removed */
  int32_t* nbr_cnt;      /* [N] entries used in nbr */
  uint8_t* moved;        /* [N] kMoved* bits of this frame */
  int32_t* inc_state;    /* [W] 0 = rebuild the adjacency next frame, 1 = valid */
  int32_t* inc_rebuild;  /* [W] this frame rebuilds the world's adjacency */
  int32_t* inc_moved;    /* [W] bodies re-inserted this frame */
  int32_t* inc_frames;   /* [W] consecutive quiet frames of a FULL world */
  double* inc_margin;    /* [W] fat-box margin */
  int32_t nbr_cap;
  int32_t* row_cnt; /* [N] mirrored per-row pair counts */
  int32_t* row_hits; /* [kRowHits * N] the pairs of rows with few, descending j */
  int32_t* row_off; /* [N+1] scanned */
  int32_t* pair_a;  /* [pair_cap] global body index, the larger */
  int32_t* pair_b;  /* [pair_cap] */
  int32_t* slot_cnt;   /* [pair_cap] contacts per pair (0..2) */
  int32_t* slot_off;   /* [pair_cap+1] scanned */
  int32_t* slot_feat;  /* [2*pair_cap] fa | fb<<12 | flip<<24 */
  int32_t* np_perm;    /* [pair_cap] pairs in processing order, grouped by vertex-count class */
  const int32_t* ext_chunk;     /* [2 * n_ext_chunks] body range [b0, b1) of each extent-reduction chunk */
  const int32_t* ext_chunk_off; /* [n_worlds + 1] each world's chunks */
  double* ext_part_sum;         /* [n_ext_chunks] chunk sums of box extents */
  int32_t* ext_part_cnt;        /* [n_ext_chunks] chunk counts */
  int32_t* ext_done;            /* [W] chunks of the world summed so far this step */
  int32_t n_ext_chunks;
  const uint8_t* world_sap; /* [n_worlds] 1: the world's small bodies pair by sweep and prune (null: none) */
  const int32_t* sap_base;  /* [n_worlds] first of the world's kSapBuckets buckets */
  int32_t* sap_cnt;         /* [n_sap_buckets + 1] bucket counts */
  int32_t* sap_off;         /* [n_sap_buckets + 1] their exclusive scan: bucket starts, then ends */
  int32_t n_sap_buckets;
  int32_t* sap_ids;         /* [n_bodies] small bodies of sweep worlds, in bucket order */
  int32_t* sap_qs;          /* [n_bodies] their buckets, in the same order */
  int32_t* sap_cursor;      /* [n_bodies] per row (mirrored index): the next free slot of the row */
  uint64_t* sap_range;      /* [2 * n_worlds] min and max order key of the small bodies' lower x */
  int32_t* sap_end;         /* [n_worlds] end of the world's run in sap_ids */
  int32_t* np_cls;     /* [2 * kNpClasses + 1] class counts, then offsets and cursors */
  double* slot_val;    /* [2*pair_cap*5] nx ny px py depth */
  uint64_t* c_key;     /* [contact_cap] packed world-local key */
  int32_t* c_ga;       /* [contact_cap] */
  int32_t* c_slot;     /* [contact_cap] each contact's slot t = 2 pair + s (k_contact_slots), or null */
  int32_t* c_gb;       /* [contact_cap] */
  uint8_t* c_flip;     /* [contact_cap] */
  uint8_t* c_hit;      /* [contact_cap] kInfo* bits */
  double* c_val;       /* [contact_cap*5] */
  Con* con;            /* [contact_cap] */
  double* lam;         /* [2*contact_cap] this step's cache Lagrangians */
  const uint64_t* old_key; /* previous cache keys */
  const double* old_lam;   /* previous cache Lagrangians */
  const int32_t* old_cwo;  /* [W+1] previous cache world offsets */
  int32_t* world_pair_off;    /* [W+1] */
  int32_t* world_contact_off; /* [W+1] */
  int4* sched_info;           /* [contact_cap] lists of groups too large for shared memory (frontier.cuh) */
  int32_t* sched_list;        /* [2 * contact_cap] */
  int32_t* sched_arr;         /* [contact_cap] */
  int32_t* sched_body;        /* [4 * N] */
  uint32_t* sched_cur;        /* [N] */
  int4* gdesc;                /* [item_cap + W + 1] per-group updates, level by level: {contact and warm bit, slots, flags} */
  long long* phase_clock;     /* [G * 8] per-group phase clocks when profiling, else null */
  int32_t* world_levels;      /* [W] dependency levels of each small world's last solve */
  const int32_t* group_world_off; /* [G+1] offsets into group_worlds */
  const int32_t* group_worlds;    /* [W] world ids, grouped */
  unsigned long long* counters;   /* [kCntSlots] see kCnt* */
  double* world_residual;         /* [W] */
  double* world_depth;            /* [W] */
  /* learned warm start (null / zero when off) */
  uint8_t* learned_mask;       /* [W] 1 = contacts without a cache entry start from the network */
  int32_t* miss_flag;          /* [contact_cap] 1 = contact gets a feature row */
  int32_t* miss_off;           /* [contact_cap + 1] scanned miss_flag */
  int32_t* miss_ids;           /* [contact_cap] contact of each row */
  int32_t* miss_n;             /* [1] rows this step */
  float* mfeat;                /* [contact_cap x 16] raw features */
  int32_t collect_all;         /* 1 = rows for every world's misses (sample collection) */
  const double* judge_res;     /* [W] residual limit of the judge */
  const double* judge_depth;   /* [W] depth limit of the judge */
  const uint8_t* active;       /* [N] 0 = empty slot (World.delete); null when every slot is filled */
  const double* radius;        /* [N] > 0: a circle (one local point, the centre); 0: a hull */
};

enum {
  /* set anew every step (the first two by the scans, the others by k_contact_slots), the others every call */
  kCntPairs = 0,
  kCntContacts = 1,
  kCntGroupAlloc = 2, /* bump allocator of the groups' runs of updates kept in global memory */
  kCntListAlloc = 3,  /* bump allocator of the lists kept in global memory */
  kCntHits = 4,
  kCntItems = 5,
  kCntLevels = 6,
  kCntOverflow = 7,
  kCntBadInput = 8,
  kCntPredicted = 9, /* contacts started from the network (summed over the call) */
  kCntReverted = 10, /* worlds the judge switched back to the plain start */
  kCntMlpErr = 11,   /* set when a tensor-core wait of the network gave up */
  kCntSolveErr = 12, /* set when a wait between a solver group's warps or a scan's blocks gave up */
  kCntSlots = 16,
};

/* Narrowphase work classes: (min(nv_a, 9) - 3) * 7 + (min(nv_b, 9) - 3). */
constexpr int kNpHullClasses = 49;            /* hull pairs by vertex counts 3..9+ each */
constexpr int kNpClasses = kNpHullClasses + 15; /* then circle-circle, circle-hull, hull-circle */

/* Flags any non-finite value among n bodies' ten state arrays. */
__global__ void k_check_finite(const double* a0, const double* a1, const double* a2, const double* a3,
                               const double* a4, const double* a5, const double* a6, const double* a7,
                               const double* a8, const double* a9, int n, unsigned long long* flag) {
  const double* arr[10] = {a0, a1, a2, a3, a4, a5, a6, a7, a8, a9};
  bool bad = false;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < 10LL * n;
       t += (long long)gridDim.x * blockDim.x) {
    const double v = arr[t / n][t % n];
    bad |= !isfinite(v);
  }
  if (__any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(flag, 1ull);
}

/* Ten arrays of n doubles copied in one launch (blockIdx.y = array), with an
 * optional finiteness check of what passes through.  Either side may be
 * pinned host memory mapped into the device address space: on a Grace host
 * the loads and stores then cross NVLink-C2C from every SM at once instead of
 * through the copy engines. */
struct Ptr10 {
  const double* src[10];
  double* dst[10];
};

/* Ten arrays of n doubles, array blockIdx.y; non-finite values set *bad_flag.
 * When both ends are 16-byte aligned each thread keeps four 16-byte loads in
 * flight, so a copy over the host link needs few blocks (copy10_grid sizes
 * the grid for kCopy10PerThread doubles a thread) and leaves the SMs to the
 * steps of other handles. */
constexpr int kCopy10PerThread = 8;

__global__ void k_copy10(Ptr10 p, int n, unsigned long long* bad_flag) {
  const double* __restrict__ src = p.src[blockIdx.y];
  double* __restrict__ dst = p.dst[blockIdx.y];
  bool bad = false;
  const int stride = gridDim.x * blockDim.x;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15u) == 0) {
    const double2* __restrict__ s2 = reinterpret_cast<const double2*>(src);
    double2* __restrict__ d2 = reinterpret_cast<double2*>(dst);
    const int n2 = n >> 1;
    for (; i + 3 * stride < n2; i += 4 * stride) {
      double2 v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = s2[i + u * stride];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        bad |= !isfinite(v[u].x) || !isfinite(v[u].y);
        d2[i + u * stride] = v[u];
      }
    }
    for (; i < n2; i += stride) {
      const double2 v = s2[i];
      bad |= !isfinite(v.x) || !isfinite(v.y);
      d2[i] = v;
    }
    if ((n & 1) && blockIdx.x == 0 && threadIdx.x == 0) {
      const double v = src[n - 1];
      bad |= !isfinite(v);
      dst[n - 1] = v;
    }
  } else {
    for (; i < n; i += stride) {
      const double v = src[i];
      bad |= !isfinite(v);
      dst[i] = v;
    }
  }
  if (bad_flag && __any_sync(0xffffffffu, bad) && (threadIdx.x & 31) == 0) atomicOr(bad_flag, 1ull);
}

/* Up to kMaxSegments device-to-device copies in one launch (the retry
 * snapshot of a step and its restore): blockIdx.y picks the segment; every
 * segment starts on an allocation base (8-byte aligned), so whole 8-byte
 * words are copied and the last bytes singly. */
constexpr int kMaxSegments = 12;
struct Segments {
  const void* src[kMaxSegments];
  void* dst[kMaxSegments];
  unsigned long long bytes[kMaxSegments];
};

__global__ void k_copy_segments(Segments s) {
  const int k = blockIdx.y;
  const unsigned long long nb = s.bytes[k], nw = nb >> 3;
  const uint64_t* __restrict__ sw = static_cast<const uint64_t*>(s.src[k]);
  uint64_t* __restrict__ dw = static_cast<uint64_t*>(s.dst[k]);
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  const unsigned long long t = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
  for (unsigned long long i = t; i < nw; i += stride) dw[i] = sw[i];
  if (t < (nb & 7ull)) {
    const unsigned long long b = (nw << 3) + t;
    static_cast<uint8_t*>(s.dst[k])[b] = static_cast<const uint8_t*>(s.src[k])[b];
  }
}

/* Contacts in the caller's layout (keys i, j, fa, fb, flip and values nx, ny,
 * px, py, depth, five each), written to device memory or to mapped pinned
 * host memory.  The key fields follow pack_key. */
__global__ void k_export_contacts(const uint64_t* key, const uint8_t* flip, const double* val, int n,
                                  int32_t* keys5, double* vals5) {
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
    const uint64_t k = key[c];
    int32_t* ko = keys5 + 5 * (size_t)c;
    ko[0] = (int32_t)(k >> 44);
    ko[1] = (int32_t)((k >> 24) & 0xfffff);
    ko[2] = (int32_t)((k >> 12) & 0xfff);
    ko[3] = (int32_t)(k & 0xfff);
    ko[4] = flip[c];
    const double* vi = val + 5 * (size_t)c;
    double* vo = vals5 + 5 * (size_t)c;
#pragma unroll
    for (int q = 0; q < 5; ++q) vo[q] = vi[q];
  }
}

/* Staged body state -> live arrays, one thread per body; changed[g] = 1 when
 * a field the pose depends on (position, rotation, inverse masses, which set
 * the static flag) differs bit for bit from the live value. */
__global__ void k_commit_bodies(Ptr10 p, int n, uint8_t* changed, const unsigned long long* bad = nullptr) {
  const bool skip = bad && *bad != 0; /* refused input: the live state stays */
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < n; g += gridDim.x * blockDim.x) {
    if (skip) {
      changed[g] = 0;
      continue;
    }
    bool c = false;
#pragma unroll
    for (int k = 0; k < 10; ++k) {
      const double v = p.src[k][g];
      if (k >= 3 && k <= 7) c |= __double_as_longlong(v) != __double_as_longlong(p.dst[k][g]);
      p.dst[k][g] = v;
    }
    changed[g] = c ? 1 : 0;
  }
}

/* ------------------------------------------------------------------------ */
/* helpers                                                                    */
/* ------------------------------------------------------------------------ */

__device__ __forceinline__ bool is_nan(double d) { return d != d; }



__device__ __forceinline__ uint64_t pack_key(int i, int j, int fa, int fb) {
  return ((uint64_t)i << 44) | ((uint64_t)j << 24) | ((uint64_t)fa << 12) | (uint64_t)fb;
}

/* ------------------------------------------------------------------------ */
/* A2 pose + A11 integrate                                                    */
/* ------------------------------------------------------------------------ */

/* listToHull extents (ConvexHull.hs:151-167): for each local edge, the first
 * strict min / max vertex along its local unit normal (extentAlong',
 * ConvexHull.hs:81-92).  One thread per edge. */
__global__ void k_init_extents(Dev d) {
  chained_entry();
  for (int v = blockIdx.x * blockDim.x + threadIdx.x; v < d.n_verts; v += gridDim.x * blockDim.x) {
    /* find the owning body by binary search over vert_off */
    int lo = 0, hi = d.n_bodies - 1;
    while (lo < hi) {
      int mid = (lo + hi + 1) >> 1;
      if (d.vert_off[mid] <= v) lo = mid; else hi = mid - 1;
    }
    const int b0 = d.vert_off[lo], nv = d.vert_off[lo + 1] - b0, e = v - b0;
    if (nv < 3) { /* a circle: no edges */
      d.emin[v] = 0;
      d.emax[v] = 0;
      continue;
    }
    const int n1 = e < nv - 1 ? e + 1 : 0;
    const double ddx = d.lx[b0 + n1] - d.lx[b0 + e], ddy = d.ly[b0 + n1] - d.ly[b0 + e];
    const double ex = ddy, ey = -ddx;
    const double len = sqrt(ex * ex + ey * ey);
    const double nx = ex / len, ny = ey / len;
    double lo_d = d.lx[b0] * nx + d.ly[b0] * ny, hi_d = lo_d;
    int imin = 0, imax = 0;
    for (int k = 1; k < nv; ++k) {
      const double t = d.lx[b0 + k] * nx + d.ly[b0 + k] * ny;
      if (t < lo_d) { lo_d = t; imin = k; }
      if (t > hi_d) { hi_d = t; imax = k; }
    }
    d.emin[v] = imin;
    d.emax[v] = imax;
  }
}

/* A body's box, its ordered keys and its flags. */
__device__ __forceinline__ void write_box(const Dev& d, int g, double x0, double x1, double y0, double y1, uint8_t f) {
  d.box[4 * g + 0] = x0;
  d.box[4 * g + 1] = x1;
  d.box[4 * g + 2] = y0;
  d.box[4 * g + 3] = y1;
  d.boxk[4 * g + 0] = okey(x0);
  d.boxk[4 * g + 1] = okey(x1);
  d.boxk[4 * g + 2] = okey(y0);
  d.boxk[4 * g + 3] = okey(y1);
  if (is_zero(d.iml[g]) && is_zero(d.imr[g])) f |= kFlagStatic;
  if (nan_bits(x0) || nan_bits(x1) || nan_bits(y0) || nan_bits(y1)) f |= kFlagBoxNaN;
  d.flags[g] = f;
}

/* advanceObj (Constraint.hs:225-229) when `advance`, then moveShape
 * (World.hs:132-133): rotation matrix from shapes_sincos, the 3x3 product of
 * toTransform (Transform.hs:34-38, 73-77; MatrixTemplate.hs:47-67), afmul
 * (Linear.hs:217-220) per vertex, unitEdgeNormal (ConvexHull.hs:218-226) per
 * edge, then hullToAabb (Aabb.hs:81-84, 106-110) and its ordered keys.
 * A block takes per_block bodies (a warp's worth in small batches, so that
 * their vertices are one round of its threads) in turns: a thread per body for the angle
 * and the matrix, a thread per vertex for the points, a thread per edge for the
 * normals (a square root and two divisions, two thirds of a hull's FP64 work),
 * a thread per body for the box.  The FP64 pipe charges a warp instruction in
 * full whatever its active lanes, and here every warp but a block's last is
 * full however many vertices the hulls have; with a thread per body the vertex
 * loop was also one long chain.  1024 x 256 mixed worlds: 0.181 ms a step as a
 * thread per body (bodies ordered by vertex count). */
constexpr int kPoseThreads = 128;
__global__ void __launch_bounds__(kPoseThreads) k_integrate_pose(Dev d, double dt, int advance, int per_block,
                                                                 const uint8_t* only = nullptr) {
  chained_entry();
  __shared__ double mat[6][kPoseThreads];   /* the matrix's two rows */
  __shared__ int32_t vstart[kPoseThreads + 1];
  __shared__ uint8_t kind[kPoseThreads];    /* a hull to pose: 1, with a NaN translation: 2; else 0 */
  const int tid = threadIdx.x;
  for (int base = blockIdx.x * per_block; base < d.n_bodies; base += gridDim.x * per_block) {
    const int nb = min(per_block, d.n_bodies - base), g = base + tid;
    if (tid < nb) {
      vstart[tid] = d.vert_off[g];
      if (tid == nb - 1) vstart[nb] = d.vert_off[g + 1];
      kind[tid] = 0;
      if (only && !only[g]) { /* re-pose: this body's pose inputs did not change */
      } else if (d.active && !d.active[g]) { /* empty slot: left as it was, out of the broadphase */
        d.flags[g] = kFlagInactive;
      } else {
        double px = d.px[g], py = d.py[g], th = d.th[g];
        if (advance) {
          const double vx = d.vx[g], vy = d.vy[g], w = d.w[g];
          px = (vx * dt) + px;
          py = (vy * dt) + py;
          th = (dt * w) + th;
          d.px[g] = px;
          d.py[g] = py;
          d.th[g] = th;
        }
        double s, c;
        shapes_sincos(th, &s, &c);
        const double ms = flip_sign(s);
        /* rows of translate(px,py) times columns of rotate(c,s), summed in the
         * reference's order (joinTransforms, Transform.hs:73-77) */
        double m00, m01, m02, m10, m11, m12;
        if (finite_bits(c) && finite_bits(s) && finite_bits(px) && finite_bits(py)) {
          /* every product by 1.0 or 0.0 is exact, so the sums reduce to
           * signed-zero rules on the integer pipe */
          const double zc = signed_zero(c), zs = signed_zero(s), zms = signed_zero(ms);
          const double zpx = signed_zero(px), zpy = signed_zero(py);
          m00 = add_zero(add_zero(c, zs), zpx);
          m01 = add_zero(add_zero(ms, zc), zpx);
          m02 = plus_zero(px);
          m10 = add_zero(add_zero(s, zc), zpy);
          m11 = add_zero(add_zero(c, zms), zpy);
          m12 = plus_zero(py);
        } else {
          m00 = (1.0 * c + 0.0 * s) + px * 0.0;
          m01 = (1.0 * ms + 0.0 * c) + px * 0.0;
          m02 = (1.0 * 0.0 + 0.0 * 0.0) + px * 1.0;
          m10 = (0.0 * c + 1.0 * s) + py * 0.0;
          m11 = (0.0 * ms + 1.0 * c) + py * 0.0;
          m12 = (0.0 * 0.0 + 1.0 * 0.0) + py * 1.0;
        }
        /* m02 * 1.0 == m02 and m12 * 1.0 == m12 unless NaN (then both are NaN) */
        const bool t_nan = nan_bits(m02) || nan_bits(m12);
        const double rad = d.radius ? d.radius[g] : 0.0;
        if (rad > 0.0) {
          /* setCircleTransform (Circle.hs:60-64): the transformed local origin;
           * circleToAabb (Aabb.hs:86-89): centre -+ radius */
          const int b0 = vstart[tid];
          const double lx = d.lx[b0], ly = d.ly[b0];
          const double x = t_nan ? (m00 * lx + m01 * ly) + m02 * 1.0 : (mul_rn_int(m00, lx) + m01 * ly) + m02;
          const double y = t_nan ? (m10 * lx + m11 * ly) + m12 * 1.0 : (mul_rn_int(m10, lx) + m11 * ly) + m12;
          d.wx[b0] = x;
          d.wy[b0] = y;
          d.nx[b0] = 0.0;
          d.ny[b0] = 0.0;
          write_box(d, g, x - rad, x + rad, y - rad, y + rad, kFlagCircle);
        } else {
          kind[tid] = t_nan ? 2 : 1;
          mat[0][tid] = m00;
          mat[1][tid] = m01;
          mat[2][tid] = m02;
          mat[3][tid] = m10;
          mat[4][tid] = m11;
          mat[5][tid] = m12;
        }
      }
    }
    __syncthreads();
    const int v0 = vstart[0], v1 = vstart[nb];
    auto owner = [&](int v) { /* the body of vertex v */
      int lo = 0, hi = nb;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (vstart[mid] <= v) lo = mid;
        else hi = mid;
      }
      return lo;
    };
    for (int v = v0 + tid; v < v1; v += kPoseThreads) {
      const int k = owner(v);
      if (!kind[k]) continue;
      const double lx = d.lx[v], ly = d.ly[v], m02 = mat[2][k], m12 = mat[5][k];
      const bool t_nan = kind[k] == 2;
      /* one product per coordinate on the integer pipe (exact), as in SAT */
      const double m00 = mat[0][k], m01 = mat[1][k], m10 = mat[3][k], m11 = mat[4][k];
      d.wx[v] = t_nan ? (m00 * lx + m01 * ly) + m02 * 1.0 : (mul_rn_int(m00, lx) + m01 * ly) + m02;
      d.wy[v] = t_nan ? (m10 * lx + m11 * ly) + m12 * 1.0 : (mul_rn_int(m10, lx) + m11 * ly) + m12;
    }
    __syncthreads();
    for (int v = v0 + tid; v < v1; v += kPoseThreads) {
      const int k = owner(v);
      if (!kind[k]) continue;
      const int n1 = v + 1 < vstart[k + 1] ? v + 1 : vstart[k];
      const double x = d.wx[v], y = d.wy[v];
      const double ddx = d.wx[n1] - x, ex = d.wy[n1] - y, ey = flip_sign(ddx);
      const double len = sqrt(ex * ex + ey * ey);
      const double nx = ex / len, ny = ey / len;
      d.nx[v] = nx;
      d.ny[v] = ny;
      d.vf[v] = make_float4(to_float(x), to_float(y), to_float(nx), to_float(ny));
    }
    __syncthreads();
    for (int v = v0 + tid; v < v1; v += kPoseThreads) { /* extentAlongSelf (ConvexHull.hs:107-118) */
      const int k = owner(v);
      if (!kind[k]) continue;
      const float4 n = d.vf[v], lo = d.vf[vstart[k] + d.emin[v]], hi = d.vf[vstart[k] + d.emax[v]];
      d.ef[v] = make_float2(__fmaf_rn(lo.x, n.z, lo.y * n.w), __fmaf_rn(hi.x, n.z, hi.y * n.w));
    }
    if (tid < nb && kind[tid]) {
      const int b0 = vstart[tid], b1 = vstart[tid + 1];
      double bx0 = d.wx[b0], bx1 = bx0, by0 = d.wy[b0], by1 = by0;
      for (int v = b0 + 1; v < b1; ++v) {
        const double x = d.wx[v], y = d.wy[v];
        bx0 = f_lt(bx0, x) ? bx0 : x;
        bx1 = f_lt(x, bx1) ? bx1 : x;
        by0 = f_lt(by0, y) ? by0 : y;
        by1 = f_lt(y, by1) ? by1 : y;
      }
      write_box(d, g, bx0, bx1, by0, by1, 0);
    }
    __syncthreads();
  }
}

/* ------------------------------------------------------------------------ */
/* A3 broadphase                                                              */
/* ------------------------------------------------------------------------ */

/* culledKeys (Aabb.hs:168-183): not both static, and boundsOverlap
 * (Aabb.hs:69-72) on x and y, i.e. not (c > b || d < a) with (a,b) = box i,
 * (c,d) = box j.  The flags and the box of j are loaded together by the
 * callers: one trip to L2 instead of two. */
__device__ __forceinline__ bool keys_overlap(const Dev& d, int gi, int gj, uint8_t fi, uint8_t fj,
                                             const uint64_t ki[4], ulonglong2 kj01, ulonglong2 kj23) {
  if ((fi | fj) & kFlagInactive) return false;
  if ((fi & fj & kFlagStatic)) return false;
  if ((fi | fj) & kFlagBoxNaN) {
    const double* a = d.box + 4 * gi;
    const double* b = d.box + 4 * gj;
    return !(b[0] > a[1] || b[1] < a[0]) && !(b[2] > a[3] || b[3] < a[2]);
  }
  return !(kj01.x > ki[1] || kj01.y < ki[0]) && !(kj23.x > ki[3] || kj23.y < ki[2]);
}

__device__ __forceinline__ bool box_overlaps(const Dev& d, int gi, int gj, uint8_t fi, uint8_t fj,
                                             const uint64_t ki[4]) {
  const ulonglong2 kj01 = *reinterpret_cast<const ulonglong2*>(d.boxk + 4 * gj);
  const ulonglong2 kj23 = *reinterpret_cast<const ulonglong2*>(d.boxk + 4 * gj + 2);
  return keys_overlap(d, gi, gj, fi, fj, ki, kj01, kj23);
}

__device__ __forceinline__ bool pair_overlaps(const Dev& d, int gi, int gj, uint8_t fi,
                                              const uint64_t ki[4]) {
  return box_overlaps(d, gi, gj, fi, d.flags[gj], ki);
}

constexpr int kRowHits = 8;        /* pairs of a row that the counting pass keeps */
constexpr int kRowSorted = 256;    /* pairs of a row that a warp sorts in shared memory */
constexpr int kRowThreads = 256;

/* Lanes per grid row.  While all of the batch's rows run at once with eight
 * lanes each (2048 threads an SM), the chain of loads of one lane is what takes
 * the time, and eight are the fastest; above that two are, because each lane of a
 * row repeats the row's own loads.  The incremental broadphase with 8, 4, 2 and 1
 * lanes, us: 9,075 bodies 64, 70, 82, 104; 32,771: 65, 63, 74, 97; 65,539: 89,
 * 83, 88, 118; 262,144: 198, 178, 171, 196; 505,800: 279, 245, 203, 196. */
constexpr int kRowTeam = 8, kRowPair = 2;
inline bool row_teams(long long n) { return n * kRowTeam <= 152 * 2048; }

/* Row i (the larger index of a pair, body g) by brute force, a warp together:
 * lanes test j = i-1, i-2, ... 64 at a time (two loads in flight per lane),
 * so ballot order is the reference's descending j order.  COUNT: writes the
 * row's pair count at its mirrored position q = off + (n_w - 1 - i), so that an
 * exclusive scan over q lays rows out in descending i within each world, and
 * keeps the first kRowHits pairs.  !COUNT: writes the pairs at row_off[q]. */
template <bool COUNT>
__device__ __forceinline__ void brute_row(const Dev& d, int g) {
  constexpr int kU = 2;
  const int lane = threadIdx.x & 31;
  const int wld = d.body_world[g];
  const int off = d.world_body_off[wld];
  const int n = d.world_body_off[wld + 1] - off;
  const int i = g - off;
  const int q = off + (n - 1 - i);
  const uint8_t fi = d.flags[g];
  uint64_t ki[4];
  ki[0] = d.boxk[4 * g + 0];
  ki[1] = d.boxk[4 * g + 1];
  ki[2] = d.boxk[4 * g + 2];
  ki[3] = d.boxk[4 * g + 3];
  int count = 0;
  const int base_out = COUNT ? 0 : d.row_off[q];
  for (int base = 0; base < i; base += 32 * kU) {
    uint8_t fj[kU];
    ulonglong2 k01[kU], k23[kU];
    const int j0 = i - 1 - base - lane;
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      if (j0 - 32 * u < 0) continue;
      const int gj = off + j0 - 32 * u;
      fj[u] = d.flags[gj];
      k01[u] = *reinterpret_cast<const ulonglong2*>(d.boxk + 4 * gj);
      k23[u] = *reinterpret_cast<const ulonglong2*>(d.boxk + 4 * gj + 2);
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const int jl = j0 - 32 * u;
      bool hit = false;
      if (jl >= 0) hit = keys_overlap(d, g, off + jl, fi, fj[u], ki, k01[u], k23[u]);
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (hit) {
        const int at = count + __popc(m & ((1u << lane) - 1u));
        if (COUNT) {
          if (at < kRowHits) d.row_hits[kRowHits * (size_t)g + at] = off + jl;
        } else if (base_out + at < d.pair_cap) {
          d.pair_a[base_out + at] = g;
          d.pair_b[base_out + at] = off + jl;
        }
      }
      count += __popc(m);
    }
  }
  if (COUNT && lane == 0) d.row_cnt[q] = count;
}

/* Counts the rows of a batch without a grid world: a warp per row. */
__global__ void k_count_brute(Dev d) {
  chained_entry();
  const int wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nw_total = (gridDim.x * blockDim.x) >> 5;
  for (int g = wid; g < d.n_bodies; g += nw_total) brute_row<true>(d, g);
}

/* Grid broadphase for larger worlds.  It finds exactly the pairs the
 * brute-force rows find, faster: the cell size s is twice the mean AABB extent
 * of the world; a body is "small" when its width and height are below
 * s (1 - 2^-20), its box is finite and its cell index fits 30 bits.  A small
 * body is binned by the cell of its box's min corner, floor(x0 / s) and
 * floor(y0 / s) (computed as x0 * (1/s): monotone in x0).  Two small bodies
 * whose closed boxes overlap have |x0_i - x0_j| < s (1 - 2^-20) and likewise in
 * y, so their cells differ by at most one in each axis: every such pair is
 * found by scanning the 3x3 cells around a body.  Cells are hashed into a
 * table of 2^k >= 2n buckets by their Morton code; a bucket may hold other
 * cells, so candidates are kept only when their exact cell matches.  Bodies
 * that are not small are listed per world and checked against everything:
 * their own rows take the brute-force path, and every grid row also checks
 * them.  Grid rows are written unordered and then sorted (descending j), so
 * the final list is the reference's descending (i, j) order. */

__device__ __forceinline__ uint32_t spread16(uint32_t x) {
  x &= 0xffffu;
  x = (x | (x << 8)) & 0x00ff00ffu;
  x = (x | (x << 4)) & 0x0f0f0f0fu;
  x = (x | (x << 2)) & 0x33333333u;
  x = (x | (x << 1)) & 0x55555555u;
  return x;
}

__device__ __forceinline__ uint32_t cell_bucket(int cx, int cy, int T) {
  return (spread16((uint32_t)cx) | (spread16((uint32_t)cy) << 1)) & (uint32_t)(T - 1);
}

/* Twice the mean extent over a world's chunks, added in chunk order. */
__device__ __forceinline__ double world_cell_size(const Dev& d, int wld) {
  double t = 0.0;
  int c = 0;
  for (int k = d.ext_chunk_off[wld]; k < d.ext_chunk_off[wld + 1]; ++k) {
    t += __ldcg(d.ext_part_sum + k);
    c += __ldcg(d.ext_part_cnt + k);
  }
  return c > 0 ? 2.0 * t / c : 0.0;
}

/* Mean box extent of each grid world, which sets its cell size (2x the mean),
 * its reciprocal, the size limit of a grid body and the fat-box margin.  The
 * cell size only decides how fast the grid finds the pairs, never which pairs
 * it finds (any positive size gives the pairs of culledKeys), so the sum may be
 * split: one block per chunk of at most 4096 bodies of one world, and the last
 * block of a world to finish adds its chunks in order (deterministic; a world
 * of one chunk sums exactly as one block would).  A single large world thus
 * spreads over the GPU instead of one SM.  With incremental pairs only a world
 * that rebuilds needs a cell size.  Every world's large list and moved count
 * start empty here. */
__global__ void k_grid_stats(Dev d, int inc) {
  chained_entry();
  __shared__ double s_sum[32];
  __shared__ int s_cnt[32];
  const int k = blockIdx.x;
  if (k >= d.n_ext_chunks) return;
  const int b0 = d.ext_chunk[2 * k], b1 = d.ext_chunk[2 * k + 1];
  const int wld = d.body_world[b0];
  if (d.grid_T[wld] == 0) return;
  if (threadIdx.x == 0 && k == d.ext_chunk_off[wld]) {
    d.large_cnt[wld] = 0;
    if (inc) d.inc_moved[wld] = 0;
    if (d.world_sap && d.world_sap[wld]) { /* the small bodies' range of lower x, gathered by k_grid_bin */
      d.sap_range[2 * wld] = ~0ull;
      d.sap_range[2 * wld + 1] = 0ull;
    }
  }
  if (inc && d.inc_state[wld] != 0) return;
  double sum = 0.0;
  int cnt = 0;
  for (int g = b0 + threadIdx.x; g < b1; g += blockDim.x) {
    const double w = d.box[4 * g + 1] - d.box[4 * g + 0];
    const double h = d.box[4 * g + 3] - d.box[4 * g + 2];
    const double e = w > h ? w : h;
    if (small_mag(e)) {
      sum += e;
      ++cnt;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  if ((threadIdx.x & 31) == 0) {
    s_sum[threadIdx.x >> 5] = sum;
    s_cnt[threadIdx.x >> 5] = cnt;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  double t = 0.0;
  int c = 0;
  for (int q = 0; q < (int)(blockDim.x >> 5); ++q) {
    t += s_sum[q];
    c += s_cnt[q];
  }
  __stcg(d.ext_part_sum + k, t);
  __stcg(d.ext_part_cnt + k, c);
  __threadfence();
  const int chunks = d.ext_chunk_off[wld + 1] - d.ext_chunk_off[wld];
  if (atomicAdd(d.ext_done + wld, 1) + 1 < chunks) return;
  d.ext_done[wld] = 0; /* for the next step */
  __threadfence();
  const double sz = world_cell_size(d, wld);
  const double inv = (sz > 0.0 && small_mag(sz) && small_mag(1.0 / sz)) ? 1.0 / sz : 0.0;
  d.grid_inv_s[wld] = inv;
  d.grid_lim[wld] = inv > 0.0 ? (1.0 - 0x1p-20) / inv : 0.0;
  if (inc) d.inc_margin[wld] = inv > 0.0 ? 0.03125 / inv : 0.0;
}

/* One thread per body: grid bodies get a cell and a bucket count, the rest go
 * on their world's list of large bodies. */
__global__ void k_grid_bin(Dev d) {
  chained_entry();
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < d.n_bodies; g += gridDim.x * blockDim.x) {
    const int wld = d.body_world[g];
    const int T = d.grid_T[wld];
    uint8_t mode = 0;
    if (T > 0) {
      const double inv_s = d.grid_inv_s[wld];
      bool small = false;
      int cx = 0, cy = 0;
      if (inv_s > 0.0 && !(d.flags[g] & kFlagBoxNaN)) {
        const double x0 = d.box[4 * g + 0], x1 = d.box[4 * g + 1];
        const double y0 = d.box[4 * g + 2], y1 = d.box[4 * g + 3];
        const double lim = d.grid_lim[wld];
        const double qx = x0 * inv_s, qy = y0 * inv_s;
        if (small_mag(x0) && small_mag(x1) && small_mag(y0) && small_mag(y1) && (x1 - x0) < lim &&
            (y1 - y0) < lim && fabs(qx) < 0x1p30 && fabs(qy) < 0x1p30) {
          small = true;
          cx = (int)floor(qx);
          cy = (int)floor(qy);
        }
      }
      if (small) {
        mode = 1;
        d.cell[g] = make_int2(cx, cy);
        if (d.world_sap && d.world_sap[wld]) {
          const uint64_t k = okey(d.box[4 * g + 0]);
          atomicMin(reinterpret_cast<unsigned long long*>(&d.sap_range[2 * wld]), (unsigned long long)k);
          atomicMax(reinterpret_cast<unsigned long long*>(&d.sap_range[2 * wld + 1]), (unsigned long long)k);
        } else {
          atomicAdd(&d.bucket_cnt[d.grid_base[wld] + cell_bucket(cx, cy, T)], 1);
        }
      } else {
        const int k = atomicAdd(&d.large_cnt[wld], 1);
        d.large_ids[d.world_body_off[wld] + k] = g;
      }
    }
    d.row_mode[g] = mode;
  }
}

/* Places grid bodies into their buckets (bucket_off turns from starts into ends). */
__global__ void k_grid_scatter(Dev d) {
  chained_entry();
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < d.n_bodies; g += gridDim.x * blockDim.x) {
    if (!d.row_mode[g]) continue;
    const int wld = d.body_world[g];
    if (d.world_sap && d.world_sap[wld]) continue; /* swept, not binned */
    const int2 c = d.cell[g];
    const int pos = atomicAdd(&d.bucket_off[d.grid_base[wld] + cell_bucket(c.x, c.y, d.grid_T[wld])], 1);
    d.grid_ent[pos] = make_int4(g, c.x, c.y, d.flags[g]);
  }
}

/* ---- sweep and prune ------------------------------------------------------
 * For large single worlds, the small bodies (the grid's classification: box
 * below the cell limit) can be paired by sweep and prune along x instead of
 * the 3x3 cell search.  The bodies are sorted by their box's lower x
 * quantised to kSapBuckets buckets over the world's range, q(x) =
 * floor((x - xmin) * (kSapBuckets - 1) / (xmax - xmin)) clamped to the last
 * bucket; q is non-decreasing in x (each operation is a monotone rounding),
 * so two small bodies whose closed boxes overlap, x0_j <= x1_i, have
 * q(x0_j) <= q(x1_i).  A counting sort (one 16-bit radix digit) orders them;
 * from each body the sweep walks forward while q(x0) <= q(x1) of the body
 * and tests every candidate with the exact test every path uses
 * (pair_overlaps).  Each overlapping pair is met once, from the body earlier
 * in the order (within a bucket the order is arbitrary: the walk from the
 * earlier one still reaches the later one).  It is added to the row of its
 * larger index with an atomic slot after that row's large-body pairs, and the
 * rows are then sorted descending like the grid's, so the pairs and their
 * order are exactly those of culledKeys. */
constexpr int kSapBuckets = 65536;

__device__ __forceinline__ double from_okey(uint64_t k) {
  const uint64_t u = (k >> 63) ? (k & 0x7fffffffffffffffull) : ~k;
  return __longlong_as_double((long long)u);
}

__device__ __forceinline__ int sap_bucket(const Dev& d, int wld, double x) {
  const double lo = from_okey(d.sap_range[2 * wld]), hi = from_okey(d.sap_range[2 * wld + 1]);
  const double span = hi - lo;
  const double scale = span > 0.0 && small_mag(span) ? (double)(kSapBuckets - 1) / span : 0.0;
  const double t = (x - lo) * scale;
  if (!(t > 0.0)) return 0;
  return t >= (double)(kSapBuckets - 1) ? kSapBuckets - 1 : (int)t;
}

__global__ void k_sap_count(Dev d) {
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < d.n_bodies; g += gridDim.x * blockDim.x) {
    if (!d.row_mode[g]) continue;
    const int wld = d.body_world[g];
    if (!d.world_sap[wld]) continue;
    atomicAdd(&d.sap_cnt[d.sap_base[wld] + sap_bucket(d, wld, d.box[4 * g + 0])], 1);
  }
}

/* Places the swept bodies by bucket (sap_cnt turns from starts into ends);
 * records the end of each world's run. */
__global__ void k_sap_scatter(Dev d) {
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < d.n_bodies; g += gridDim.x * blockDim.x) {
    if (!d.row_mode[g]) continue;
    const int wld = d.body_world[g];
    if (!d.world_sap[wld]) continue;
    const int q = sap_bucket(d, wld, d.box[4 * g + 0]);
    const int pos = atomicAdd(&d.sap_off[d.sap_base[wld] + q], 1);
    d.sap_ids[pos] = g;
    d.sap_qs[pos] = q;
  }
}

__global__ void k_sap_ends(Dev d) {
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < d.n_worlds; w += gridDim.x * blockDim.x)
    if (d.world_sap[w]) d.sap_end[w] = d.sap_off[d.sap_base[w] + kSapBuckets - 1];
}

/* One thread per position of the sorted run: the forward sweep.  COUNT adds
 * to the rows' counts; otherwise writes the pairs at atomic slots. */
template <bool COUNT>
__global__ void k_sap_rows(Dev d) {
  const int n_swept = d.sap_off[d.n_sap_buckets - 1]; /* end of the last bucket */
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n_swept; p += gridDim.x * blockDim.x) {
    const int g = d.sap_ids[p];
    const int wld = d.body_world[g];
    const int off = d.world_body_off[wld];
    const int n = d.world_body_off[wld + 1] - off;
    const int end = d.sap_end[wld];
    const int q1 = sap_bucket(d, wld, d.box[4 * g + 1]);
    const uint8_t fi = d.flags[g];
    uint64_t ki[4];
    ki[0] = d.boxk[4 * g + 0];
    ki[1] = d.boxk[4 * g + 1];
    ki[2] = d.boxk[4 * g + 2];
    ki[3] = d.boxk[4 * g + 3];
    for (int t = p + 1; t < end && d.sap_qs[t] <= q1; ++t) {
      const int j = d.sap_ids[t];
      if (!pair_overlaps(d, g, j, fi, ki)) continue;
      const int hi = g > j ? g : j, lo = g > j ? j : g;
      const int q = off + (n - 1 - (hi - off));
      if (COUNT) {
        atomicAdd(&d.row_cnt[q], 1);
      } else {
        const int pos = d.row_off[q] + atomicAdd(&d.sap_cursor[q], 1);
        if (pos < d.pair_cap) {
          d.pair_a[pos] = hi;
          d.pair_b[pos] = lo;
        }
      }
    }
  }
}

/* Sorts each grid row's j descending once the sweep has added its pairs (a
 * handful per row). */
__global__ void k_sap_sort_rows(Dev d) {
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < d.n_bodies; g += gridDim.x * blockDim.x) {
    if (!d.row_mode[g]) continue;
    const int wld = d.body_world[g];
    if (!d.world_sap[wld]) continue;
    const int off = d.world_body_off[wld];
    const int n = d.world_body_off[wld + 1] - off;
    const int q = off + (n - 1 - (g - off));
    const int r0 = d.row_off[q], r1 = min(d.row_off[q + 1], d.pair_cap);
    for (int a = r0 + 1; a < r1; ++a) {
      const int v = d.pair_b[a];
      int b = a - 1;
      while (b >= r0 && d.pair_b[b] < v) {
        d.pair_b[b + 1] = d.pair_b[b];
        --b;
      }
      d.pair_b[b + 1] = v;
    }
  }
}

/* ---- incremental grid pairs ------------------------------------------------
 * The grid rows above search the 3x3 cells of every body every frame.  Most
 * bodies move far less than a cell per frame, so the incremental variant keeps
 * for each grid body a fat box (its box grown by a margin of s/32, s the
 * world's cell size) and the list of bodies whose fat boxes overlap it (an
 * adjacency, symmetric: each overlap is listed at both bodies).  While a
 * body's box stays inside its fat box nothing about it is searched again:
 * boxes inside overlapping-or-not fat boxes overlap only if the fat boxes do,
 * so the exact pairs of a row are its adjacency entries j < i whose current
 * boxes overlap (pair_overlaps, the same test as every other path).  A body
 * whose box left its fat box (or that changed between grid and large) is
 * "moved": it is removed from its old neighbours' lists, gets a new fat box,
 * searches the 3x3 cells of the fat-box grid (binned only in worlds with
 * moved bodies) and is appended to each unmoved neighbour's list.
 * Each world picks one of three modes per frame: LIST (the above), BUILD
 * (every grid body searches and the lists are written afresh: a new world,
 * every world after a retry, and a world coming back from FULL) and FULL
 * (more than a quarter of the world moved: no lists; the rows search the
 * 3x3 cells of the fat-box grid directly, like the plain grid rows).  A FULL
 * world keeps counting the bodies that leave their fat boxes and returns
 * through BUILD once that share stays below an eighth for four frames.  Large bodies (fat box not small, or a non-finite
 * box) stay on the per-world large list as before.
 * Rows come out unordered and are sorted like grid rows, so the pair list is
 * exactly the brute-force rows' list.  A list that would exceed nbr_cap sets
 * overflow bit 4 and the host retries with a larger capacity. */

constexpr int kIncList = 0, kIncBuild = 1, kIncFull = 2; /* per-world mode of a frame */
constexpr int kIncStateNew = 0, kIncStateList = 1, kIncStateFull = 2;
constexpr uint8_t kMovedBit = 1;     /* re-inserted this frame */
constexpr uint8_t kMovedWasGrid = 2; /* was in the adjacency before this frame */
constexpr uint8_t kMovedNowGrid = 4; /* is in the adjacency after this frame */

/* Fat box of a body's current box, its cell, and whether it is small enough
 * for the grid (the same finiteness and size rules as k_grid_bin, on the fat
 * box). */
__device__ __forceinline__ bool fat_box(const Dev& d, int g, int wld, double fb[4], int* cx, int* cy) {
  const double inv_s = d.grid_inv_s[wld];
  if (!(inv_s > 0.0) || (d.flags[g] & kFlagBoxNaN)) return false;
  const double m = d.inc_margin[wld];
  fb[0] = d.box[4 * g + 0] - m;
  fb[1] = d.box[4 * g + 1] + m;
  fb[2] = d.box[4 * g + 2] - m;
  fb[3] = d.box[4 * g + 3] + m;
  const double lim = d.grid_lim[wld];
  const double qx = fb[0] * inv_s, qy = fb[2] * inv_s;
  if (!(small_mag(fb[0]) && small_mag(fb[1]) && small_mag(fb[2]) && small_mag(fb[3]) && (fb[1] - fb[0]) < lim &&
        (fb[3] - fb[2]) < lim && fabs(qx) < 0x1p30 && fabs(qy) < 0x1p30))
    return false;
  *cx = (int)floor(qx);
  *cy = (int)floor(qy);
  return true;
}

/* One thread per body of a grid world: moved or not, and the large list. */
__global__ void k_inc_mark(Dev d) {
  chained_entry();
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < d.n_bodies; g += gridDim.x * blockDim.x) {
    const int wld = d.body_world[g];
    if (d.grid_T[wld] == 0) continue;
    const bool rebuild = d.inc_state[wld] == 0;
    const bool was = !rebuild && d.row_mode[g];
    bool inside = false;
    if (was) {
      const uint64_t* f = d.fatk + 4 * g;
      const ulonglong2 b01 = *reinterpret_cast<const ulonglong2*>(d.boxk + 4 * g);
      const ulonglong2 b23 = *reinterpret_cast<const ulonglong2*>(d.boxk + 4 * g + 2);
      inside = !(d.flags[g] & kFlagBoxNaN) && f[0] <= b01.x && b01.y <= f[1] && f[2] <= b23.x && b23.y <= f[3];
    }
    bool fits = false;
    if (!inside) { /* only a body that is not staying needs the fat-box verdict */
      double fb[4];
      int cx = 0, cy = 0;
      fits = fat_box(d, g, wld, fb, &cx, &cy);
      if (fits) { /* its new fat box (read by nothing before k_inc_scatter) */
        for (int k = 0; k < 4; ++k) d.fatk[4 * g + k] = okey(fb[k]);
        d.cell[g] = make_int2(cx, cy);
      }
    }
    const bool moved = rebuild || (!inside && (was || fits));
    const bool now = inside || fits;
    d.moved[g] = (moved ? kMovedBit : 0) | (was ? kMovedWasGrid : 0) | (now ? kMovedNowGrid : 0);
    if (moved && !rebuild) { /* one atomic for the warp's bodies of a world: its counter is one address */
      const unsigned peers = __match_any_sync(__activemask(), wld);
      if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&d.inc_moved[wld], __popc(peers));
    }
    if (!now) {
      const int k = atomicAdd(&d.large_cnt[wld], 1);
      d.large_ids[d.world_body_off[wld] + k] = g;
    }
  }
}

/* A world's mode this frame, from what its state was before the frame and how
 * many of its bodies moved (k_inc_mark): read by k_inc_update, which writes it
 * to inc_rebuild; the state follows in k_inc_scatter. */
__device__ __forceinline__ int inc_mode(const Dev& d, int w) {
  const int n = d.world_body_off[w + 1] - d.world_body_off[w];
  const int st = d.inc_state[w], moved = d.inc_moved[w];
  if (st == kIncStateNew) return kIncBuild;
  if (st == kIncStateList) return 4 * moved > n ? kIncFull : kIncList;
  /* FULL: back through BUILD after 4 quiet-enough frames */
  return 8 * moved < n && d.inc_frames[w] + 1 >= 4 ? kIncBuild : kIncFull;
}

/* One thread per body.  A moved body that was in the adjacency of a LIST world:
 * its entry in each unmoved neighbour's list becomes -1 (every entry is removed
 * by the thread of the body it names, so the stores never collide).  Then a
 * moved body's grid membership (its fat box and cell were written by k_inc_mark;
 * a staying body keeps the ones it has, which still contain its box), and the
 * grid bodies of worlds that search this frame are counted into the buckets. */
__global__ void k_inc_update(Dev d) {
  chained_entry();
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < d.n_bodies; g += gridDim.x * blockDim.x) {
    const int wld = d.body_world[g];
    if (d.grid_T[wld] == 0) continue;
    const int mode = inc_mode(d, wld);
    if (g == d.world_body_off[wld]) d.inc_rebuild[wld] = mode;
    const uint8_t mg = d.moved[g];
    if (mode == kIncList && (mg & kMovedBit) && (mg & kMovedWasGrid)) {
      const int32_t* lst = d.nbr + (size_t)g * d.nbr_cap;
      const int n = min(d.nbr_cnt[g], d.nbr_cap);
      for (int k = 0; k < n; ++k) {
        const int j = lst[k];
        if (j < 0 || (d.moved[j] & kMovedBit)) continue;
        int32_t* lj = d.nbr + (size_t)j * d.nbr_cap;
        const int nj = min(d.nbr_cnt[j], d.nbr_cap);
        for (int t = 0; t < nj; ++t)
          if (lj[t] == g) {
            lj[t] = -1;
            break;
          }
      }
    }
    const bool now = (mg & kMovedNowGrid) != 0;
    if (mg & kMovedBit) d.row_mode[g] = now ? 1 : 0;
    if (mode == kIncBuild) d.nbr_cnt[g] = 0;
    if (now && (mode != kIncList || d.inc_moved[wld] > 0)) {
      const int2 c = d.cell[g];
      atomicAdd(&d.bucket_cnt[d.grid_base[wld] + cell_bucket(c.x, c.y, d.grid_T[wld])], 1);
    }
  }
}

/* Places the grid bodies of worlds that search; and each world's state for the
 * next frame. */
__global__ void k_inc_scatter(Dev d) {
  chained_entry();
  for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < d.n_bodies; g += gridDim.x * blockDim.x) {
    const int wld = d.body_world[g];
    if (d.grid_T[wld] == 0) continue;
    const int mode = d.inc_rebuild[wld];
    if (g == d.world_body_off[wld]) {
      const int n = d.world_body_off[wld + 1] - g;
      if (d.inc_state[wld] == kIncStateFull)
        d.inc_frames[wld] = 8 * d.inc_moved[wld] < n ? d.inc_frames[wld] + 1 : 0;
      else if (mode == kIncFull)
        d.inc_frames[wld] = 0;
      d.inc_state[wld] = mode == kIncFull ? kIncStateFull : kIncStateList;
    }
    if (!d.row_mode[g] || !(mode != kIncList || d.inc_moved[wld] > 0)) continue;
    const int2 c = d.cell[g];
    const int pos = atomicAdd(&d.bucket_off[d.grid_base[wld] + cell_bucket(c.x, c.y, d.grid_T[wld])], 1);
    d.grid_ent[pos] = make_int4(g, c.x, c.y, d.flags[g]);
  }
}

__device__ __forceinline__ bool fat_overlap(const uint64_t* a, const uint64_t* b) {
  return !(b[0] > a[1] || b[1] < a[0]) && !(b[2] > a[3] || b[3] < a[2]);
}

/* The lanes of this thread's team of TEAM neighbours in a warp. */
template <int TEAM>
__device__ __forceinline__ unsigned team_mask() {
  return TEAM == 32 ? 0xffffffffu : ((1u << (TEAM & 31)) - 1u) << (threadIdx.x & 31 & ~(TEAM - 1));
}

/* TEAM lanes per re-inserted grid body: its new list from the 3x3 cells of
 * the fat-box grid, a cell per lane; in an incremental frame it is also appended
 * to each unmoved neighbour's list.  (The order within a list is arbitrary: the
 * rows are sorted.)  A thread walking all nine cells took 40 us on 75 worlds of
 * 121 bodies; the chain of its loads, not their number, is what takes the time. */
template <int TEAM>
__global__ void __launch_bounds__(kRowThreads) k_inc_query(Dev d) {
  chained_entry();
  __shared__ int s_cnt[kRowThreads / TEAM];
  const int lane = threadIdx.x % TEAM, team = threadIdx.x / TEAM;
  const unsigned mates = team_mask<TEAM>();
  for (int g = blockIdx.x * (kRowThreads / TEAM) + team; g < d.n_bodies;
       g += gridDim.x * (kRowThreads / TEAM)) {
    const int wld = d.body_world[g];
    if (d.grid_T[wld] == 0 || !d.row_mode[g]) continue;
    const int mode = d.inc_rebuild[wld];
    const bool rebuild = mode == kIncBuild;
    if (mode == kIncFull || (!rebuild && !(d.moved[g] & kMovedBit))) continue;
    const int T = d.grid_T[wld], base = d.grid_base[wld];
    const int2 cell = d.cell[g];
    uint64_t fg[4];
    for (int k = 0; k < 4; ++k) fg[k] = d.fatk[4 * g + k];
    int32_t* lst = d.nbr + (size_t)g * d.nbr_cap;
    if (lane == 0) s_cnt[team] = 0;
    __syncwarp(mates);
    bool over = false;
    for (int c = lane; c < 9; c += TEAM) {
      const int ncx = cell.x + c % 3 - 1, ncy = cell.y + c / 3 - 1;
      const int b = base + cell_bucket(ncx, ncy, T);
      const int k0 = b > 0 ? d.bucket_off[b - 1] : 0, k1 = d.bucket_off[b];
      for (int k = k0; k < k1; ++k) {
        const int4 e = d.grid_ent[k];
        const int j = e.x;
        if (j == g || e.y != ncx || e.z != ncy) continue;
        if (!fat_overlap(fg, d.fatk + 4 * j)) continue;
        const int cnt = atomicAdd(&s_cnt[team], 1);
        if (cnt < d.nbr_cap) lst[cnt] = j; else over = true;
        if (!rebuild && !(d.moved[j] & kMovedBit)) {
          const int pos = atomicAdd(&d.nbr_cnt[j], 1);
          if (pos < d.nbr_cap) d.nbr[(size_t)j * d.nbr_cap + pos] = g; else over = true;
        }
      }
    }
    __syncwarp(mates);
    if (lane == 0) d.nbr_cnt[g] = s_cnt[team];
    if (over) atomicOr(&d.counters[kCntOverflow], 4ull);
  }
}

/* Calls hit(j) for the partners j < g of grid row g, its candidates dealt over
 * LANES lanes: with adjacency lists the entries of its list (COMPACT: removed
 * entries are dropped from it on the way), else the bodies of the 3x3 cells
 * around it; then the world's large bodies.  A world that is swept finds the
 * partners among its small bodies elsewhere. */
template <int LANES, bool INC, bool COMPACT, class Hit>
__device__ __forceinline__ void grid_partners(const Dev& d, int g, Hit&& hit) {
  const int lane = threadIdx.x % LANES;
  const unsigned mates = team_mask<LANES>();
  const int wld = d.body_world[g];
  const uint8_t fi = d.flags[g];
  uint64_t ki[4];
  ki[0] = d.boxk[4 * g + 0];
  ki[1] = d.boxk[4 * g + 1];
  ki[2] = d.boxk[4 * g + 2];
  ki[3] = d.boxk[4 * g + 3];
  if (INC && d.inc_rebuild[wld] != kIncFull) {
    int32_t* lst = d.nbr + (size_t)g * d.nbr_cap;
    const int listed = d.nbr_cnt[g], nl = min(listed, d.nbr_cap);
    int kept = 0;
    for (int k0 = 0; k0 < nl; k0 += LANES) {
      const int j = k0 + lane < nl ? lst[k0 + lane] : -1;
      if (COMPACT) {
        const unsigned m = LANES == 1 ? (j >= 0 ? mates : 0u) : __ballot_sync(mates, j >= 0);
        const int at = kept + __popc(m & ((1u << (threadIdx.x & 31)) - 1u));
        if (j >= 0 && at != k0 + lane) lst[at] = j;
        kept += __popc(m);
      }
      if (j >= 0 && j < g && pair_overlaps(d, g, j, fi, ki)) hit(j);
    }
    if (COMPACT && lane == 0 && listed <= d.nbr_cap) d.nbr_cnt[g] = kept;
  } else if (INC || !(d.world_sap && d.world_sap[wld])) {
    const int T = d.grid_T[wld], base = d.grid_base[wld];
    const int2 cell = d.cell[g];
    for (int c = lane; c < 9; c += LANES) {
      const int ncx = cell.x + c % 3 - 1, ncy = cell.y + c / 3 - 1;
      const int b = base + cell_bucket(ncx, ncy, T);
      const int k0 = b > 0 ? d.bucket_off[b - 1] : 0, k1 = d.bucket_off[b];
      for (int k = k0; k < k1; ++k) {
        const int4 e = d.grid_ent[k];
        if (e.x >= g || e.y != ncx || e.z != ncy) continue;
        if (box_overlaps(d, g, e.x, fi, (uint8_t)e.w, ki)) hit(e.x);
      }
    }
  }
  const int nlarge = d.large_cnt[wld];
  const int32_t* large = d.large_ids + d.world_body_off[wld];
  for (int k = lane; k < nlarge; k += LANES) {
    const int j = large[k];
    if (j < g && pair_overlaps(d, g, j, fi, ki)) hit(j);
  }
}

/* Counts the rows of a batch with grid worlds and keeps each row's pairs, in
 * descending j, where it has at most kRowHits: TEAM lanes per grid row; the
 * rows of bodies outside the grid (large ones, small worlds) a warp each, dealt
 * over the block.  A row is a chain of dependent loads, so the latency of one
 * lane's share counts.  A thread per row, which tested everything once to count
 * and once more to write, took 53 us for one world of 401 bodies and 135 us for
 * 4096 worlds of 505,800; counting and writing now take 13 and 100. */
template <bool INC, int TEAM>
__global__ void __launch_bounds__(kRowThreads, 5) k_count_rows(Dev d) {
  chained_entry();
  constexpr int kTeams = kRowThreads / TEAM;
  __shared__ int s_cnt[kTeams], s_hits[kTeams][kRowHits + 1], s_brute[kTeams], s_nbrute;
  const int lane = threadIdx.x % TEAM, team = threadIdx.x / TEAM;
  const unsigned mates = team_mask<TEAM>();
  for (int base = blockIdx.x * kTeams; base < d.n_bodies; base += gridDim.x * kTeams) {
    if (threadIdx.x == 0) s_nbrute = 0;
    if (lane == 0) s_cnt[team] = 0;
    __syncthreads();
    const int g = base + team;
    if (g < d.n_bodies) {
      if (d.row_mode[g]) {
        grid_partners<TEAM, INC, true>(d, g, [&](int j) {
          const int k = atomicAdd(&s_cnt[team], 1);
          if (k < kRowHits) s_hits[team][k] = j;
        });
        __syncwarp(mates);
        const int count = s_cnt[team];
        for (int e = lane; e < count && count <= kRowHits; e += TEAM) {
          const int j = s_hits[team][e];
          int rank = 0;
          for (int k = 0; k < count; ++k) rank += s_hits[team][k] > j;
          d.row_hits[kRowHits * (size_t)g + rank] = j;
        }
        if (lane == 0) {
          const int wld = d.body_world[g];
          const int off = d.world_body_off[wld];
          const int q = off + (d.world_body_off[wld + 1] - 1 - g);
          d.row_cnt[q] = count;
          if (!INC && d.world_sap && d.world_sap[wld]) d.sap_cursor[q] = count; /* the sweep's pairs follow */
        }
      } else if (lane == 0) {
        s_brute[atomicAdd(&s_nbrute, 1)] = g;
      }
    }
    __syncthreads();
    for (int k = threadIdx.x >> 5; k < s_nbrute; k += kRowThreads / 32) brute_row<true>(d, s_brute[k]);
    __syncthreads();
  }
}

/* Writes the pairs: a thread per row that kept its pairs; the others a warp
 * each, tested again (in a grid row sorted in shared memory, or by brute force,
 * which finds them in order, where there are more than that holds).  In a swept
 * world a thread writes its row's pairs with large bodies. */
template <bool GRID, bool INC>
__global__ void __launch_bounds__(kRowThreads) k_write_rows(Dev d) {
  chained_entry();
  constexpr int kWarps = kRowThreads / 32;
  __shared__ int s_heavy[kRowThreads], s_nheavy, s_cnt[kWarps], s_hits[GRID ? kWarps : 1][kRowSorted];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int base = blockIdx.x * kRowThreads; base < d.n_bodies; base += gridDim.x * kRowThreads) {
    if (threadIdx.x == 0) s_nheavy = 0;
    __syncthreads();
    const int g = base + threadIdx.x;
    if (g < d.n_bodies) {
      const int wld = d.body_world[g];
      const int off = d.world_body_off[wld];
      const int q = off + (d.world_body_off[wld + 1] - 1 - g);
      const int out = d.row_off[q], count = d.row_off[q + 1] - out;
      auto put = [&](int k, int j) {
        if (out + k < d.pair_cap) {
          d.pair_a[out + k] = g;
          d.pair_b[out + k] = j;
        }
      };
      if (GRID && !INC && d.world_sap && d.world_sap[wld] && d.row_mode[g]) {
        int k = 0;
        grid_partners<1, false, false>(d, g, [&](int j) { put(k++, j); });
      } else if (count <= kRowHits) {
        const int32_t* hits = d.row_hits + kRowHits * (size_t)g;
        for (int k = 0; k < count; ++k) put(k, hits[k]);
      } else {
        s_heavy[atomicAdd(&s_nheavy, 1)] = g;
      }
    }
    __syncthreads();
    for (int h = warp; h < s_nheavy; h += kWarps) {
      const int gh = s_heavy[h];
      const int wld = d.body_world[gh];
      const int off = d.world_body_off[wld];
      const int q = off + (d.world_body_off[wld + 1] - 1 - gh);
      const int out = d.row_off[q], count = d.row_off[q + 1] - out;
      if (!GRID || !d.row_mode[gh] || count > kRowSorted) {
        brute_row<false>(d, gh);
        continue;
      }
      if (lane == 0) s_cnt[warp] = 0;
      __syncwarp();
      grid_partners<32, INC, false>(d, gh, [&](int j) {
        const int k = atomicAdd(&s_cnt[warp], 1);
        if (k < kRowSorted) s_hits[GRID ? warp : 0][k] = j;
      });
      __syncwarp();
      const int found = min(s_cnt[warp], kRowSorted);
      for (int e = lane; e < found; e += 32) {
        const int j = s_hits[GRID ? warp : 0][e];
        int rank = 0;
        for (int k = 0; k < found; ++k) rank += s_hits[GRID ? warp : 0][k] > j;
        if (out + rank < d.pair_cap) {
          d.pair_a[out + rank] = gh;
          d.pair_b[out + rank] = j;
        }
      }
      __syncwarp();
    }
    __syncthreads();
  }
}

/* ------------------------------------------------------------------------ */
/* A5-A7 narrowphase                                                          */
/* ------------------------------------------------------------------------ */

struct HullView {
  const double* wx;
  const double* wy;
  const double* nx;
  const double* ny;
  const int32_t* emin;
  const int32_t* emax;
  const float4* vf;
  const float2* ef;
  int nv;
};

__device__ __forceinline__ HullView hull_view(const Dev& d, int g) {
  const int b0 = d.vert_off[g];
  HullView h;
  h.wx = d.wx + b0;
  h.wy = d.wy + b0;
  h.nx = d.nx + b0;
  h.ny = d.ny + b0;
  h.emin = d.emin + b0;
  h.emax = d.emax + b0;
  h.vf = d.vf + b0;
  h.ef = d.ef + b0;
  h.nv = d.vert_off[g + 1] - b0;
  return h;
}

/* overlap (SAT.hs:103-118): extentAlongSelf with the precomputed extent
 * indices (ConvexHull.hs:111-118), extentAlong over the penetrator
 * (ConvexHull.hs:81-100), overlapTest/overlapAmount (SAT.hs:74-95). */
/* The comparisons run on the integer pipe through order-preserving keys; a
 * NaN projection compares false exactly as in IEEE arithmetic (a NaN first
 * projection pins lo and hi, later NaNs never replace them). */
__device__ __forceinline__ bool sat_axis(const HullView& se, int e, const HullView& sp,
                                         double* depth, int* pen) {
  const double dx = se.nx[e], dy = se.ny[e];
  const int mi = se.emin[e], ma = se.emax[e];
  const double sa = se.wx[mi] * dx + se.wy[mi] * dy;
  const double sb = se.wx[ma] * dx + se.wy[ma] * dy;
  /* one product of each projection on the integer pipe (mul_rn_int, exact),
   * the other on the FP64 pipe: the kernel is bound by FP64 throughput at
   * high occupancy, so the two pipes share the work */
  const double t0 = mul_rn_int(sp.wx[0], dx) + sp.wy[0] * dy;
  double lo = t0, hi = t0;
  uint64_t klo = okey(t0), khi = klo;
  const bool pinned = nan_bits(t0);
  int pmin = 0;
  for (int k = 1; k < sp.nv; ++k) {
    const double t = mul_rn_int(sp.wx[k], dx) + sp.wy[k] * dy;
    if (pinned || nan_bits(t)) continue;
    const uint64_t kt = okey(t);
    if (kt < klo) { lo = t; klo = kt; pmin = k; }
    if (kt > khi) { hi = t; khi = kt; }
  }
  *pen = pmin;
  if (f_lt(sb, lo) || f_lt(hi, sa)) return false; /* Separated */
  *depth = sb - lo;
  return true;
}

/* minOverlap (SAT.hs:121-138): first Separated axis, else first strict
 * minimum depth.  Returns false when separated. */
__device__ __forceinline__ bool min_overlap(const HullView& se, const HullView& sp, int* edge,
                                            double* depth, int* pen) {
  double best = 0.0;
  int be = 0, bp = 0;
  for (int e = 0; e < se.nv; ++e) {
    double dep;
    int p;
    if (!sat_axis(se, e, sp, &dep, &p)) return false;
    if (e == 0 || f_lt(dep, best)) { best = dep; be = e; bp = p; }
  }
  *edge = be;
  *depth = best;
  *pen = bp;
  return true;
}

enum { kClipNone = 0, kClipLeft = 1, kClipRight = 2, kClipBoth = 3 };

/* The binary32 filter.  Every coordinate in vf is within 2^-23 of its double,
 * so a projection computed from them is within 3 * 2^-23 M of the double one,
 * M bounding |x| + |y| of both hulls (normals are unit vectors), and an overlap
 * of two such within kFilter M = 2^-20 M.  Decisions that hold by more than
 * that are the doubles' decisions; the others are made in binary64.  On a
 * reference normal of length L the bound for a difference of two points is
 * kFilterEdge M L, with room to spare. */
constexpr float kFilter = 0x1p-20f, kFilterEdge = 0x1p-18f, kFilterMax = 1e15f;

/* contact_ (SAT.hs:261-267): penetratingEdge (SAT.hs:152-166), clipEdge
 * (SAT.hs:190-218, clipSegment, Linear.hs:327-343) and flattenContactPoints
 * (SAT.hs:181-187).  Writes up to two (index, x, y) points, descending index.
 * m bounds |x| + |y| of both hulls for the filter, an infinity leaves it out.
 * The incident edge is clipped at three lines: the sides of the reference edge
 * and the edge itself.  An end is cut off when it lies below the crossing of
 * incident edge and line along the line's normal.  The crossing lies on the line
 * up to rounding, so comparing with the crossing is comparing with the line
 * wherever the two are far from parallel: ends clear of the line by the
 * filter's bound then need neither the comparison nor, unless an end is
 * replaced, the crossing.  The lanes of a warp go on to the next line that
 * needs a crossing before they compute one together. */
__device__ __forceinline__ int manifold(const HullView& se, int e, const HullView& sp, int pen, float m,
                                        int idx[2], double xs[2], double ys[2]) {
  const int ne = e < se.nv - 1 ? e + 1 : 0;
  const double ax = se.wx[e], ay = se.wy[e], bx = se.wx[ne], by = se.wy[ne];
  const double nx = se.nx[e], ny = se.ny[e];
  const int vb = pen, vc = pen < sp.nv - 1 ? pen + 1 : 0, va = pen > 0 ? pen - 1 : sp.nv - 1;
  bool second;
  {
    const float4 n = se.vf[e], fa = sp.vf[va], fb = sp.vf[vb], fc = sp.vf[vc];
    const float ab = fabsf((fb.x - fa.x) * n.z + (fb.y - fa.y) * n.w);
    const float bc = fabsf((fc.x - fb.x) * n.z + (fc.y - fb.y) * n.w);
    second = bc < ab;
    if (!(fabsf(bc - ab) > kFilterEdge * m)) {
      const double abn = (sp.wx[vb] - sp.wx[va]) * nx + (sp.wy[vb] - sp.wy[va]) * ny;
      const double bcn = (sp.wx[vc] - sp.wx[vb]) * nx + (sp.wy[vc] - sp.wy[vb]) * ny;
      second = no_nan(abn, bcn) & (mag_bits(bcn) < mag_bits(abn));
    }
  }
  int ci, di;
  if (second) { ci = vb; di = vc; } else { ci = va; di = vb; }
  double cx = sp.wx[ci], cy = sp.wy[ci], dx = sp.wx[di], dy = sp.wy[di];
  const double ipx = cx, ipy = cy, inx = dy - cy, iny = flip_sign(dx - cx);
  const double ex = bx - ax, ey = by - ay;
  const float lx = to_float(inx), ly = to_float(iny), ilen = fabsf(lx) + fabsf(ly);
  int line = 0, kind = kClipNone;
#pragma unroll 1
  for (int round = 0; round < 3; ++round) {
    double px = 0.0, py = 0.0, wx = 0.0, wy = 0.0; /* a point of the line and its normal */
    bool known = false;
    for (; line < 3; ++line) {
      px = line == 1 ? bx : ax;
      py = line == 1 ? by : ay;
      wx = line == 0 ? ex : flip_sign(line == 1 ? ex : nx);
      wy = line == 0 ? ey : flip_sign(line == 1 ? ey : ny);
      const float fx = to_float(wx), fy = to_float(wy), qx = to_float(px), qy = to_float(py);
      const float fcx = to_float(cx), fcy = to_float(cy), fdx = to_float(dx), fdy = to_float(dy);
      const float dc = (fcx - qx) * fx + (fcy - qy) * fy, dd = (fdx - qx) * fx + (fdy - qy) * fy;
      const float len = fabsf(fx) + fabsf(fy);
      /* an end may be a crossing far away */
      const float clear = kFilterEdge * len * fmaxf(m, fmaxf(fabsf(fcx) + fabsf(fcy), fabsf(fdx) + fabsf(fdy)));
      known = (fabsf(fx * ly - fy * lx) > 0.0625f * len * ilen) & (fabsf(dc) > clear) & (fabsf(dd) > clear);
      kind = dc < 0.0f ? (dd < 0.0f ? kClipBoth : kClipLeft) : (dd < 0.0f ? kClipRight : kClipNone);
      if (!known) break;
      if (kind == kClipBoth) return 0;
      if (line < 2 && kind != kClipNone) break; /* an end is replaced */
    }
    if (line == 3) break;
    /* intersect2 (Linear.hs:244-251), invM2x2 (Linear.hs:194-199) */
    const double b0 = px * wx + py * wy;
    const double b1 = ipx * inx + ipy * iny;
    const double det = wx * iny - wy * inx;
    const double inv = 1.0 / det;
    const double m00 = iny * inv, m01 = (-wy) * inv, m10 = (-inx) * inv, m11 = wx * inv;
    const double qx = m00 * b0 + m01 * b1, qy = m10 * b0 + m11 * b1;
    if (!known) {
      const double c_ = cx * wx + cy * wy, d_ = dx * wx + dy * wy, q_ = qx * wx + qy * wy;
      const bool below_c = f_lt(c_, q_), below_d = f_lt(d_, q_);
      kind = below_c ? (below_d ? kClipBoth : kClipLeft) : (below_d ? kClipRight : kClipNone);
      if (kind == kClipBoth) return 0;
    }
    if (line < 2) {
      if (kind == kClipLeft) { cx = qx; cy = qy; }
      if (kind == kClipRight) { dx = qx; dy = qy; }
    }
    ++line;
  }
  /* kind is the last line's */
  if (kind == kClipLeft) { idx[0] = di; xs[0] = dx; ys[0] = dy; return 1; }
  if (kind == kClipRight) { idx[0] = ci; xs[0] = cx; ys[0] = cy; return 1; }
  const bool c_first = ci > di;
  idx[0] = c_first ? ci : di;
  xs[0] = c_first ? cx : dx;
  ys[0] = c_first ? cy : dy;
  idx[1] = c_first ? di : ci;
  xs[1] = c_first ? dx : cx;
  ys[1] = c_first ? dy : cy;
  return 2;
}

/* The contacts of one pair of hulls once both directions' least overlaps are
 * known (SAT.contact, SAT.hs:238-258): into slots 2 p and 2 p + 1. */
__device__ __forceinline__ int write_contacts(const Dev& d, int p, const HullView& a, const HullView& b, int e_ab,
                                              double dep_ab, int pen_ab, int e_ba, double dep_ba, int pen_ba, float m) {
  const bool flip = !f_lt(dep_ab, dep_ba);
  const HullView& se = flip ? b : a;
  const HullView& sp = flip ? a : b;
  const int e = flip ? e_ba : e_ab;
  int idx[2];
  double xs[2], ys[2];
  const int cnt = manifold(se, e, sp, flip ? pen_ba : pen_ab, m, idx, xs, ys);
  if (cnt == 0) return 0;
  const double nx = se.nx[e], ny = se.ny[e];
  const double vdot = se.wx[e] * nx + se.wy[e] * ny;
  for (int q = 0; q < cnt; ++q) {
    const int fa = flip ? idx[q] : e;
    const int fb = flip ? e : idx[q];
    d.slot_feat[2 * p + q] = fa | (fb << 12) | ((flip ? 1 : 0) << 24);
    double* v = d.slot_val + 5 * (2 * (size_t)p + q);
    v[0] = nx;
    v[1] = ny;
    v[2] = xs[q];
    v[3] = ys[q];
    v[4] = vdot - (xs[q] * nx + ys[q] * ny);
  }
  return cnt;
}

/* ---- circles (Contact.hs:22-40, Contact/Circle.hs, CircleVsHull.hs, GJK.hs) */

__device__ __forceinline__ double dot2(double ax, double ay, double bx, double by) { return ax * bx + ay * by; }

/* crossV2V2 (Linear.hs:135-139): (a x b) x c. */
__device__ __forceinline__ void cross3(double ax, double ay, double bx, double by, double cx, double cy,
                                       double* x, double* y) {
  const double abz = ax * by - ay * bx;
  *x = -(abz * cy);
  *y = abz * cx;
}

/* sameDirection (GJK.hs:137-138): a . b > 0, compared on the integer pipe. */
__device__ __forceinline__ bool same_dir(double ax, double ay, double bx, double by) {
  return f_lt(0.0, dot2(ax, ay, bx, by));
}

/* support (ConvexHull.hs:124-128): the first vertex of largest projection. */
__device__ __forceinline__ int gjk_support(const HullView& h, double dx, double dy) {
  int best = 0;
  double bd = dot2(h.wx[0], h.wy[0], dx, dy);
  for (int k = 1; k < h.nv; ++k) {
    const double t = dot2(h.wx[k], h.wy[k], dx, dy);
    if (f_lt(bd, t)) { bd = t; best = k; }
  }
  return best;
}

/* GJK.closestSimplex (GJK.hs:52-135) from vertex 0 toward (ox, oy): returns
 * the simplex size (3 = encloses the point), s[0] the vertex added last.  The
 * reference loop is unbounded; this one gives up after 4 nv + 8 extensions
 * (a failed search), a bound an ordinary convex hull never reaches. */
__device__ int gjk_closest(const HullView& h, double ox, double oy, int s[3]) {
  int n = 1;
  s[0] = 0;
  double dx = ox - h.wx[0], dy = oy - h.wy[0];
  for (int it = 0; it < 4 * h.nv + 8; ++it) {
    const int a = gjk_support(h, dx, dy);
    if (n == 1) {
      if (a == s[0]) return 1;
      s[1] = s[0];
      s[0] = a;
      n = 2;
      const double abx = h.wx[s[1]] - h.wx[a], aby = h.wy[s[1]] - h.wy[a];
      const double aox = ox - h.wx[a], aoy = oy - h.wy[a];
      if (same_dir(abx, aby, aox, aoy)) {
        cross3(abx, aby, aox, aoy, abx, aby, &dx, &dy);
      } else {
        n = 1;
        dx = aox;
        dy = aoy;
      }
      continue;
    }
    if (a == s[0] || a == s[1]) return 2;
    const int b = s[0], c = s[1];
    const double ax = h.wx[a], ay = h.wy[a];
    const double abx = h.wx[b] - ax, aby = h.wy[b] - ay;
    const double acx = h.wx[c] - ax, acy = h.wy[c] - ay;
    const double aox = ox - ax, aoy = oy - ay;
    const double abc = abx * acy - aby * acx;
    const double abcacx = -(abc * acy), abcacy = abc * acx;
    const double ababcx = aby * abc, ababcy = -(abx * abc);
    int mode; /* 0 star, 1 (a, c), 2 enclosed */
    if (same_dir(abcacx, abcacy, aox, aoy)) mode = same_dir(acx, acy, aox, aoy) ? 1 : 0;
    else mode = same_dir(ababcx, ababcy, aox, aoy) ? 0 : 2;
    if (mode == 2) {
      s[0] = a; s[1] = b; s[2] = c;
      return 3;
    }
    if (mode == 1) {
      s[0] = a; s[1] = c; n = 2;
      cross3(acx, acy, aox, aoy, acx, acy, &dx, &dy);
    } else if (same_dir(abx, aby, aox, aoy)) {
      s[0] = a; s[1] = b; n = 2;
      cross3(abx, aby, aox, aoy, abx, aby, &dx, &dy);
    } else {
      s[0] = a; n = 1;
      dx = aox; dy = aoy;
    }
  }
  return n;
}

/* Circle.contact (Contact/Circle.hs:27-56): a is penetrated, b penetrates. */
__device__ bool circle_circle(double ax, double ay, double ra, double bx, double by, double rb, double* v) {
  const double abx = bx - ax, aby = by - ay;
  const double rab = ra + rb;
  const double ab_sq = abx * abx + aby * aby;
  if (!f_le(ab_sq, rab * rab)) return false;
  const double len = sqrt(ab_sq);
  const double ux = abx / len, uy = aby / len;
  const double a1x = ux * ra + ax, a1y = uy * ra + ay;
  const double b1x = ux * (-rb) + bx, b1y = uy * (-rb) + by;
  v[0] = ux;
  v[1] = uy;
  v[2] = (a1x + b1x) / 2.0;
  v[3] = (a1y + b1y) / 2.0;
  v[4] = ra + rb - len;
  return true;
}

/* CircleVsHull.generateContacts (CircleVsHull.hs:18-69): the circle
 * penetrates; one contact at the closest hull point, keyed by the vertex the
 * simplex ended on; none for a 3-point simplex. */
__device__ bool circle_hull(double ox, double oy, double r, const HullView& hull, int* feature, double* v) {
  int s[3];
  const int n = gjk_closest(hull, ox, oy, s);
  if (n == 3) return false;
  double qx, qy;
  if (n == 1) {
    qx = hull.wx[s[0]];
    qy = hull.wy[s[0]];
  } else { /* closestAlong (CircleVsHull.hs:61-69) */
    const double ax = hull.wx[s[0]], ay = hull.wy[s[0]];
    const double aox = ox - ax, aoy = oy - ay;
    const double abx = hull.wx[s[1]] - ax, aby = hull.wy[s[1]] - ay;
    const double l = sqrt(abx * abx + aby * aby);
    const double ux = abx / l, uy = aby / l;
    const double t = dot2(aox, aoy, ux, uy);
    qx = ux * t + ax;
    qy = uy * t + ay;
  }
  const double bx = ox - qx, by = oy - qy;
  const double ab_sq = bx * bx + by * by;
  if (f_lt(r * r, ab_sq)) return false; /* processSimplex_ (CircleVsHull.hs:44-59) */
  const double len = sqrt(ab_sq);
  *feature = s[0];
  v[0] = -(bx / len);
  v[1] = -(by / len);
  v[2] = qx;
  v[3] = qy;
  v[4] = r - len;
  return true;
}

/* With several lanes per pair, pairs are processed grouped by the vertex counts of their two hulls, so
 * that the lanes of a warp run SAT loops of the same trip counts (one thread
 * per pair, the warp pays for its longest loop), and pairs with a circle
 * (circle-circle, or GJK against a hull of a given vertex count) apart from
 * them, so that no warp runs both the SAT and the circle code.  The grouping
 * is a permutation of the processing order only: every pair still writes its
 * own slots, so the results do not depend on it. */
__device__ __forceinline__ int np_class(const Dev& d, int p) {
  const int ga = d.pair_a[p], gb = d.pair_b[p];
  const int na = max(3, min(d.vert_off[ga + 1] - d.vert_off[ga], 9));
  const int nb = max(3, min(d.vert_off[gb + 1] - d.vert_off[gb], 9));
  const bool ca = d.radius && d.radius[ga] > 0.0, cb = d.radius && d.radius[gb] > 0.0;
  if (ca && cb) return kNpHullClasses;
  if (ca) return kNpHullClasses + 1 + (nb - 3);
  if (cb) return kNpHullClasses + 8 + (na - 3);
  return (na - 3) * 7 + (nb - 3);
}

__global__ void k_np_count(Dev d) {
  __shared__ int32_t h[kNpClasses];
  for (int k = threadIdx.x; k < kNpClasses; k += blockDim.x) h[k] = 0;
  __syncthreads();
  const int P = min((int)d.counters[kCntPairs], d.pair_cap);
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < P; p += gridDim.x * blockDim.x)
    atomicAdd(&h[np_class(d, p)], 1);
  __syncthreads();
  for (int k = threadIdx.x; k < kNpClasses; k += blockDim.x)
    if (h[k]) atomicAdd(&d.np_cls[k], h[k]);
}

/* counts -> offsets (np_cls[kNpClasses + k]) and cursors (np_cls[k]). */
__global__ void k_np_offsets(Dev d) {
  if (threadIdx.x == 0) {
    int run = 0;
    for (int k = 0; k < kNpClasses; ++k) {
      const int c = d.np_cls[k];
      d.np_cls[kNpClasses + k] = run;
      d.np_cls[k] = run;
      run += c;
    }
    d.np_cls[2 * kNpClasses] = run;
  }
}

__global__ void k_np_scatter(Dev d) {
  __shared__ int32_t h[kNpClasses];
  __shared__ int32_t base[kNpClasses];
  const int P = min((int)d.counters[kCntPairs], d.pair_cap);
  const int stride = gridDim.x * blockDim.x;
  for (int p0 = blockIdx.x * blockDim.x; p0 < P; p0 += stride) {
    for (int k = threadIdx.x; k < kNpClasses; k += blockDim.x) h[k] = 0;
    __syncthreads();
    const int p = p0 + threadIdx.x;
    int cls = -1, rank = 0;
    if (p < P) {
      cls = np_class(d, p);
      rank = atomicAdd(&h[cls], 1);
    }
    __syncthreads();
    for (int k = threadIdx.x; k < kNpClasses; k += blockDim.x)
      base[k] = h[k] ? atomicAdd(&d.np_cls[k], h[k]) : 0;
    __syncthreads();
    if (cls >= 0) d.np_perm[base[cls] + rank] = p;
    __syncthreads();
  }
}

/* One pair with a circle (Contact.generateContacts, Contact.hs:22-40). */
__device__ __forceinline__ int circle_pair(const Dev& d, int p, int ga, int gb) {
  const HullView a = hull_view(d, ga), b = hull_view(d, gb);
  const double ra = d.radius[ga], rb = d.radius[gb];
  double v[5];
  int f = 0, fa = 0, fb = 0, flip = 0;
  bool hit;
  if (ra > 0.0 && rb > 0.0) {
    hit = circle_circle(a.wx[0], a.wy[0], ra, b.wx[0], b.wy[0], rb, v);
  } else if (ra > 0.0) {
    hit = circle_hull(a.wx[0], a.wy[0], ra, b, &f, v);
    fb = f;
  } else {
    hit = circle_hull(b.wx[0], b.wy[0], rb, a, &f, v);
    fa = f;
    flip = 1;
  }
  if (!hit) return 0;
  d.slot_feat[2 * p] = fa | (fb << 12) | (flip << 24);
  double* o = d.slot_val + 5 * (2 * (size_t)p);
  for (int k = 0; k < 5; ++k) o[k] = v[k];
  return 1;
}

/* What the filter leaves of one direction's axes: those that may have the
 * least overlap, and those that may separate. */
struct AxisSets {
  uint64_t least, doubtful;
};

/* Eight vertices from number k0 of a hull on, its last one repeated past its
 * end (repeats change no minimum or maximum), so that the loops over them have
 * one length and no branches. */
struct Eight {
  float x[8], y[8];
  __device__ __forceinline__ Eight(const HullView& h, int k0) {
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float4 v = h.vf[min(k0 + q, h.nv - 1)];
      x[q] = v.x;
      y[q] = v.y;
    }
  }
  __device__ __forceinline__ float bound(float m) const { /* |x| + |y|; a NaN stays one */
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const float t = fabsf(x[q]) + fabsf(y[q]);
      m = (m == m) & !(t <= m) ? t : m;
    }
    return m;
  }
  __device__ __forceinline__ void project(float nx, float ny, float t[8]) const {
#pragma unroll
    for (int q = 0; q < 8; ++q) t[q] = __fmaf_rn(x[q], nx, y[q] * ny);
  }
};

/* One direction in binary32: false when an axis separates for certain.  first:
 * sp's first eight vertices.  bad is set when a normal is not an ordinary
 * vector (the vertices are, see bound). */
__device__ __forceinline__ bool filter_axes(const HullView& se, const HullView& sp, const Eight& first, float bound,
                                            AxisSets& sets, bool* bad) {
  float best = 0.0f, normals = 0.0f;
  bool touch = true;
  sets.least = sets.doubtful = 0;
  for (int e = 0; e < se.nv && touch; ++e) {
    const float4 n = se.vf[e];
    const float2 self = se.ef[e];
    normals += fabsf(n.z) + fabsf(n.w);
    float t[8];
    first.project(n.z, n.w, t);
    float lo = fminf(fminf(fminf(t[0], t[1]), fminf(t[2], t[3])), fminf(fminf(t[4], t[5]), fminf(t[6], t[7])));
    float hi = fmaxf(fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3])), fmaxf(fmaxf(t[4], t[5]), fmaxf(t[6], t[7])));
    for (int k = 8; k < sp.nv; ++k) {
      const float4 v = sp.vf[k];
      const float u = __fmaf_rn(v.x, n.z, v.y * n.w);
      lo = fminf(lo, u);
      hi = fmaxf(hi, u);
    }
    const float depth = self.y - lo, back = hi - self.x;
    touch = !((depth < -bound) | (back < -bound));
    if ((depth <= bound) | (back <= bound)) sets.doubtful |= 1ull << e;
    if (e == 0 || depth < best - 2.0f * bound) sets.least = 1ull << e;
    else if (depth <= best + 2.0f * bound) sets.least |= 1ull << e;
    best = e ? fminf(best, depth) : depth;
  }
  *bad |= !(normals < 1e3f);
  return touch;
}

/* minOverlap (SAT.hs:121-138) over the axes the filter left, in order: on a
 * doubtful axis as sat_axis does, else the largest self projection and the
 * first vertex of least projection among those the filter cannot tell apart. */
__device__ __forceinline__ bool least_overlap(const HullView& se, const HullView& sp, const AxisSets& sets,
                                              float bound, int* edge, double* depth, int* pen) {
  bool first = true;
  for (uint64_t left = sets.least | sets.doubtful; left; left &= left - 1) {
    const int e = __ffsll((long long)left) - 1;
    double dep;
    int p = 0;
    if (sets.doubtful >> e & 1) {
      if (!sat_axis(se, e, sp, &dep, &p)) return false;
    } else {
      const float4 n = se.vf[e];
      uint64_t near = 0;
      {
        float t[8], least;
        const Eight eight(sp, 0);
        eight.project(n.z, n.w, t);
        least = fminf(fminf(fminf(t[0], t[1]), fminf(t[2], t[3])), fminf(fminf(t[4], t[5]), fminf(t[6], t[7])));
        for (int k = 8; k < sp.nv; ++k) {
          const float4 v = sp.vf[k];
          least = fminf(least, __fmaf_rn(v.x, n.z, v.y * n.w));
        }
        const float limit = least + 2.0f * bound;
#pragma unroll
        for (int q = 0; q < 8; ++q) near |= (uint64_t)(t[q] <= limit && q < sp.nv) << q;
        for (int k = 8; k < sp.nv; ++k) {
          const float4 v = sp.vf[k];
          near |= (uint64_t)(__fmaf_rn(v.x, n.z, v.y * n.w) <= limit) << k;
        }
      }
      const double dx = se.nx[e], dy = se.ny[e];
      const int ma = se.emax[e];
      double lo = 0.0;
      for (bool any = false; near; near &= near - 1, any = true) {
        const int k = __ffsll((long long)near) - 1;
        const double t = sp.wx[k] * dx + sp.wy[k] * dy;
        if (!any || f_lt(t, lo)) {
          lo = t;
          p = k;
        }
      }
      dep = (se.wx[ma] * dx + se.wy[ma] * dy) - lo;
    }
    if (first || f_lt(dep, *depth)) {
      *depth = dep;
      *edge = e;
      *pen = p;
    }
    first = false;
  }
  return true;
}

/* HullVsHull.generateContacts (HullVsHull.hs:54-90) over SAT.contact
 * (SAT.hs:238-258) for every broadphase pair; results go to two fixed slots
 * per pair and are compacted after a scan.
 * The FP64 pipe is what bounds this (about 64 cycles an instruction and
 * sub-partition), so binary32 decides all it can (filter_axes): about half the
 * pairs of a settled pile separate by more than its error, and of the others
 * it leaves one axis a direction and a vertex or two on it, where the full
 * search computes every vertex on every axis.  The block's remaining pairs are
 * then taken close-packed, so that whole warps work on them, hull pairs and
 * pairs with a circle apart.  Values that are not ordinary numbers (or beyond
 * kFilterMax) take the full binary64 search.
 * 1024 x 256 mixed worlds, 530 k pairs: 0.178 ms a step; 0.331 ms with every
 * projection in binary64 and the pairs sorted by vertex counts beforehand
 * (three launches).  65,536-polygon field, 50 k pairs: 0.035 ms, 0.096 before. */
constexpr int kNpThreads = 128;
constexpr int kNpRounds = 4; /* pairs a thread filters before the block goes on, at most */

__global__ void __launch_bounds__(kNpThreads) k_narrowphase(Dev d) {
  chained_entry();
  struct Entry {
    AxisSets ab, ba;
    int p;
    float m; /* |x| + |y| bound; infinite: no filter */
  };
  __shared__ Entry queue[kNpThreads * kNpRounds];
  __shared__ int32_t circles[kNpThreads * kNpRounds];
  __shared__ int32_t n_hulls, n_circles;
  const int P = min((int)d.counters[kCntPairs], d.pair_cap);
  const int rounds = max(1, min(kNpRounds, P / (kNpThreads * (int)gridDim.x / 2 + 1)));
  const int chunk = rounds * kNpThreads, tid = threadIdx.x;
  for (int base = blockIdx.x * chunk; base < P; base += gridDim.x * chunk) {
    if (tid == 0) n_hulls = n_circles = 0;
    __syncthreads();
    for (int r = 0; r < rounds; ++r) {
      const int p = base + r * kNpThreads + tid;
      if (p >= P) continue;
      const int ga = d.pair_a[p], gb = d.pair_b[p];
      if (d.radius && (d.radius[ga] > 0.0 || d.radius[gb] > 0.0)) {
        circles[atomicAdd(&n_circles, 1)] = p;
        continue;
      }
      const HullView a = hull_view(d, ga), b = hull_view(d, gb);
      Entry q;
      q.p = p;
      const Eight va(a, 0), vb(b, 0);
      q.m = vb.bound(va.bound(0.0f));
      for (int k = 8; k < a.nv; k += 8) q.m = Eight(a, k).bound(q.m);
      for (int k = 8; k < b.nv; k += 8) q.m = Eight(b, k).bound(q.m);
      bool bad = !(q.m < kFilterMax), apart = false;
      const float bound = kFilter * q.m + 1e-30f;
      if (!bad)
        apart = !filter_axes(a, b, vb, bound, q.ab, &bad) || !filter_axes(b, a, va, bound, q.ba, &bad);
      if (apart && !bad) {
        d.slot_cnt[p] = 0;
        continue;
      }
      if (bad) q.m = __int_as_float(0x7f800000);
      queue[atomicAdd(&n_hulls, 1)] = q;
    }
    __syncthreads();
    /* the first warps get the last, partly filled round; which those are turns
     * with the block, as a block's warps sit on fixed sub-partitions */
    const int at = (tid + 32 * (int)blockIdx.x) & (kNpThreads - 1);
    for (int t = at; t < n_hulls; t += kNpThreads) {
      const Entry q = queue[t];
      const HullView a = hull_view(d, d.pair_a[q.p]), b = hull_view(d, d.pair_b[q.p]);
      int e_ab = 0, pen_ab = 0, e_ba = 0, pen_ba = 0, cnt = 0;
      double dep_ab = 0.0, dep_ba = 0.0;
      const float bound = kFilter * q.m + 1e-30f;
      const bool touch =
          q.m < kFilterMax
              ? least_overlap(a, b, q.ab, bound, &e_ab, &dep_ab, &pen_ab) &&
                    least_overlap(b, a, q.ba, bound, &e_ba, &dep_ba, &pen_ba)
              : min_overlap(a, b, &e_ab, &dep_ab, &pen_ab) && min_overlap(b, a, &e_ba, &dep_ba, &pen_ba);
      if (touch) cnt = write_contacts(d, q.p, a, b, e_ab, dep_ab, pen_ab, e_ba, dep_ba, pen_ba, q.m);
      d.slot_cnt[q.p] = cnt;
    }
    for (int t = at; t < n_circles; t += kNpThreads) {
      const int p = circles[t];
      d.slot_cnt[p] = circle_pair(d, p, d.pair_a[p], d.pair_b[p]);
    }
    __syncthreads();
  }
}

/* ---- L lanes per pair: the axis search spread over lanes, shuffle-reduced ----
 * The same contacts as k_narrowphase, with each pair's separating-axis search
 * split over L lanes of a warp (L = 32: one warp per pair; 32 / L pairs per
 * warp).  Lane e of a pair's lanes tests axes e, e + L, ... of both hulls
 * (sat_axis, unchanged); the lanes then agree, by shuffles, on whether any
 * axis separates and on each direction's minimum, taken exactly as
 * min_overlap's fold takes it: the first axis of the least depth, except that
 * a NaN depth on axis 0 keeps axis 0 and a NaN on any other axis is never
 * chosen.  The manifold, circles and the writes run on the pair's first
 * lane.  Selected by shapes_batch_set_narrowphase_lanes. */
struct AxisBest {
  uint64_t key; /* okey of the depth; ~0 when the lane holds no eligible axis */
  int e;        /* axis (kNoAxis when none) */
  int pen;
  double dep;
};
constexpr int kNoAxis = 0x7fffffff;

__device__ __forceinline__ void axis_take(AxisBest& b, int e, double dep, int pen) {
  if (nan_bits(dep)) return; /* never the fold's choice except on axis 0 (handled apart) */
  const uint64_t k = okey(dep);
  if (k < b.key || (k == b.key && e < b.e)) {
    b.key = k;
    b.e = e;
    b.pen = pen;
    b.dep = dep;
  }
}

template <int L>
__device__ __forceinline__ void axis_reduce(AxisBest& b) {
#pragma unroll
  for (int o = L / 2; o; o >>= 1) {
    const uint64_t k = __shfl_xor_sync(0xffffffffu, b.key, o, L);
    const int e = __shfl_xor_sync(0xffffffffu, b.e, o, L);
    const int pen = __shfl_xor_sync(0xffffffffu, b.pen, o, L);
    const double dep = __shfl_xor_sync(0xffffffffu, b.dep, o, L);
    if (k < b.key || (k == b.key && e < b.e)) {
      b.key = k;
      b.e = e;
      b.pen = pen;
      b.dep = dep;
    }
  }
}

/* One direction of minOverlap over this lane's axes: sep is set when one of
 * them separates; axis 0's depth and penetrator (on lane 0 of the pair) are
 * kept in d0 and p0. */
template <int L>
__device__ __forceinline__ void axes_lane(const HullView& se, const HullView& sp, int sub, AxisBest& best, bool* sep,
                                          double* d0, int* p0) {
  for (int e = sub; e < se.nv; e += L) {
    double dep;
    int pen;
    if (!sat_axis(se, e, sp, &dep, &pen)) {
      *sep = true;
      continue;
    }
    if (e == 0) {
      *d0 = dep;
      *p0 = pen;
    }
    axis_take(best, e, dep, pen);
  }
}

template <int L>
__global__ void k_narrowphase_lanes(Dev d) {
  const int P = min((int)d.counters[kCntPairs], d.pair_cap);
  constexpr int G = 32 / L; /* pairs per warp */
  const int lane = threadIdx.x & 31, sub = lane & (L - 1);
  const long long warp = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long n_warps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long base = warp * G; base < P; base += n_warps * G) { /* warp-uniform */
    const int i = (int)base + lane / L;
    const bool live = i < P;
    const int p = live ? (d.np_perm ? d.np_perm[i] : i) : 0;
    const int ga = live ? d.pair_a[p] : 0, gb = live ? d.pair_b[p] : 0;
    HullView a{}, b{};
    double ra = 0.0, rb = 0.0;
    if (live) {
      a = hull_view(d, ga);
      b = hull_view(d, gb);
      ra = d.radius ? d.radius[ga] : 0.0;
      rb = d.radius ? d.radius[gb] : 0.0;
    }
    const bool circ = ra > 0.0 || rb > 0.0;
    AxisBest ab{~0ull, kNoAxis, 0, 0.0}, ba{~0ull, kNoAxis, 0, 0.0};
    bool sep = false;
    double d0_ab = 0.0, d0_ba = 0.0;
    int p0_ab = 0, p0_ba = 0;
    if (live && !circ) {
      axes_lane<L>(a, b, sub, ab, &sep, &d0_ab, &p0_ab);
      axes_lane<L>(b, a, sub, ba, &sep, &d0_ba, &p0_ba);
    }
    axis_reduce<L>(ab);
    axis_reduce<L>(ba);
    const unsigned group_mask = (L == 32 ? 0xffffffffu : ((1u << L) - 1u)) << (lane & ~(L - 1));
    sep = (__ballot_sync(0xffffffffu, sep) & group_mask) != 0;
    if (!live || sub != 0) continue;
    if (circ) {
      d.slot_cnt[p] = circle_pair(d, p, ga, gb);
      continue;
    }
    int cnt = 0;
    if (!sep) {
      /* axis 0 with a NaN depth stays the fold's choice */
      const int e_ab = nan_bits(d0_ab) ? 0 : ab.e, pen_ab = nan_bits(d0_ab) ? p0_ab : ab.pen;
      const double dep_ab = nan_bits(d0_ab) ? d0_ab : ab.dep;
      const int e_ba = nan_bits(d0_ba) ? 0 : ba.e, pen_ba = nan_bits(d0_ba) ? p0_ba : ba.pen;
      const double dep_ba = nan_bits(d0_ba) ? d0_ba : ba.dep;
      cnt = write_contacts(d, p, a, b, e_ab, dep_ab, pen_ab, e_ba, dep_ba, pen_ba, __int_as_float(0x7f800000));
    }
    d.slot_cnt[p] = cnt;
  }
}

/* ------------------------------------------------------------------------ */
/* A8-A9 constraint build + warm-start lookup                                 */
/* ------------------------------------------------------------------------ */

constexpr int kBuildThreads = 128;

/* Whether k_build stages its constants in shared memory: a warp's constants lie one
 * after another, and staged they leave 512 bytes to a store instruction, where a
 * thread storing its own 224 touches a line for each (521 thousand contacts: 76 us
 * in place of 110, 165 thousand: 39 in place of 51).  Few contacts gain nothing, and
 * the group solver's block, which may need all of an SM's shared memory, then cannot
 * take its place before k_build is done (401 boxes: 12 us a step lost); nor can
 * those of other handles in flight (eight handles of 30 thousand contacts: 1.3 %).
 * The line is drawn in the contacts that the buffers hold, because a captured step
 * is launched before its contacts are counted: a new handle has room for 16 a body,
 * so it lies at 4,096 bodies.  Whole steps of one handle, us, plain and staged, by
 * the contacts they had: 2 to 50 thousand (17 handles of 2,048 to 34,018 bodies)
 * within 1.1 % of each other either way; 35 thousand in 512 ragged columns 469 and
 * 404, 76 thousand 566 and 474, 100 thousand 589 and 503, 200 thousand 685 and 677;
 * 62 thousand in 512 worlds of 64 bodies, two sweeps, 209 and 219. */
inline bool build_staged(long long contact_cap) { return contact_cap >= 65536; }

/* The slot of every contact, so that k_build's threads take contacts rather
 * than slots: about half the slots of a settled pile are empty (separated
 * pairs, pairs with one contact), and an idle lane still costs its warp's FP64
 * instructions; and the worlds' first pairs (row_off at their first row in
 * mirrored order) and first contacts; and the group solver's allocators. */
__global__ void k_contact_slots(Dev d) {
  chained_entry();
  const int P = min((int)d.counters[kCntPairs], d.pair_cap);
  const int C = (int)d.counters[kCntContacts];
  if (blockIdx.x == 0 && threadIdx.x == 0) d.counters[kCntGroupAlloc] = d.counters[kCntListAlloc] = 0;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w <= d.n_worlds; w += gridDim.x * blockDim.x) {
    const int p = d.row_off[d.world_body_off[w]];
    d.world_pair_off[w] = p;
    d.world_contact_off[w] = d.slot_off[min(p, d.pair_cap)];
  }
  if (C > d.contact_cap) return;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < 2 * P; t += gridDim.x * blockDim.x) {
    const int p = t >> 1, s = t & 1;
    if (s < d.slot_cnt[p]) d.c_slot[d.slot_off[p] + s] = t;
  }
}

/* One thread per contact (or contact slot, where k_contact_slots did not run).  Compacts the contact, builds its
 * ContactConstraint (NonPenetration.hs:16-56, Friction.hs:18-44,
 * Restitution.hs:21-31, flip handling Utils.hs:175-215 / Constraint.hs:96-98),
 * the step-invariant solver factors, and looks the key up in the previous
 * cache: descZipVector (Utils/Descending.hs:47-71) over two strictly
 * descending key lists pairs each new key with an equal old key exactly when
 * one exists, which a search over the world's old entries finds.
 * `build_solver` = 0 compacts contacts only (collide). */
__global__ void __launch_bounds__(kBuildThreads) k_build(Dev d, double beta_dt, double slop, int warm_start,
                                                         int build_solver, int staged) {
  extern __shared__ __align__(16) unsigned char s_build[];
  Con* s_con = reinterpret_cast<Con*>(s_build); /* [kBuildThreads] if staged */
  chained_entry();
  const int lane = threadIdx.x & 31;
  const int P = min((int)d.counters[kCntPairs], d.pair_cap);
  const int C = (int)d.counters[kCntContacts];
  if (C > d.contact_cap) return;
  const int n = d.c_slot ? C : 2 * P; /* contacts (k_contact_slots ran), else slots */
  auto one = [&](int i) {
    int t = i, c = i;
    if (d.c_slot) {
      t = d.c_slot[i];
    } else {
      if ((t & 1) >= d.slot_cnt[t >> 1]) return;
      c = d.slot_off[t >> 1] + (t & 1);
    }
    const int p = t >> 1;
    const int ga = d.pair_a[p], gb = d.pair_b[p];
    const int wld = d.body_world[ga];
    const int off = d.world_body_off[wld];
    const int feat = d.slot_feat[t];
    const int fa = feat & 0xfff, fb = (feat >> 12) & 0xfff, flip = (feat >> 24) & 1;
    const double* v = d.slot_val + 5 * (size_t)t;
    const double nx = v[0], ny = v[1], px = v[2], py = v[3], depth = v[4];
    const uint64_t key = pack_key(ga - off, gb - off, fa, fb);
    d.c_key[c] = key;
    d.c_ga[c] = ga;
    d.c_gb[c] = gb;
    d.c_flip[c] = (uint8_t)flip;
    double* cv = d.c_val + 5 * (size_t)c;
    cv[0] = nx;
    cv[1] = ny;
    cv[2] = px;
    cv[3] = py;
    cv[4] = depth;
    if (!build_solver) return;
    /* constraintGen: positions of (a, b) = (i, j); a Flip contact is built
     * with the bodies swapped, then its Jacobian halves are swapped back.  The
     * differences and products that the two rows, the restitution radii and the
     * effective masses share up to sign are computed once: (-p) * q is -(p * q)
     * and p - q is -(q - p) exactly, and the rows' linear parts are each other's
     * swapped, so (x m) x and (y m) y serve both folds. */
    Con cc;
    cc.ra[0] = px - d.px[ga];
    cc.ra[1] = py - d.py[ga];
    cc.ra[2] = px - d.px[gb];
    cc.ra[3] = py - d.py[gb];
    const double dxa = flip ? cc.ra[2] : cc.ra[0], dya = flip ? cc.ra[3] : cc.ra[1];
    const double dxb = flip ? cc.ra[0] : cc.ra[2], dyb = flip ? cc.ra[1] : cc.ra[3];
    const double na = dya * nx - dxa * ny, nb = dxb * ny - dyb * nx;       /* cross2 of the arms and the normal */
    const double fa_ = dxa * nx + dya * ny, fb_ = -(dxb * nx) - dyb * ny; /* and the tangent (ny, -nx) */
    cc.row[0][0] = flip ? flip_sign(nx) : nx;
    cc.row[0][1] = flip ? flip_sign(ny) : ny;
    cc.row[0][2] = flip ? nb : na;
    cc.row[0][3] = flip ? na : nb;
    cc.row[1][0] = cc.row[0][1];
    cc.row[1][1] = flip_sign(cc.row[0][0]);
    cc.row[1][2] = flip ? fb_ : fa_;
    cc.row[1][3] = flip ? fa_ : fb_;
    cc.bn = f_lt(slop, depth) ? beta_dt * (slop - depth) : 0.0;
    cc.bn0 = plus_zero(cc.bn);
    cc.rn[0] = flip ? flip_sign(nx) : nx;
    cc.rn[1] = flip ? flip_sign(ny) : ny;
    const double ima = d.iml[ga], ira = d.imr[ga], imb = d.iml[gb], irb = d.imr[gb];
    const double xa2 = (nx * ima) * nx, ya2 = (ny * ima) * ny, xb2 = (nx * imb) * nx, yb2 = (ny * imb) * ny;
    const double lin_a = xa2 + ya2;
    cc.mc[0] = ((lin_a + (cc.row[0][2] * ira) * cc.row[0][2]) + xb2) + yb2;
    cc.mc[0] = cc.mc[0] + (cc.row[0][3] * irb) * cc.row[0][3];
    cc.mc[1] = ((lin_a + (cc.row[1][2] * ira) * cc.row[1][2]) + yb2) + xb2;
    cc.mc[1] = cc.mc[1] + (cc.row[1][3] * irb) * cc.row[1][3];
    for (int k = 0; k < 2; ++k) cc.rc[k] = recip_ok(cc.mc[k]) ? 1.0 / cc.mc[k] : 0.0;
    cc.im[0] = ima;
    cc.im[1] = ira;
    cc.im[2] = imb;
    cc.im[3] = irb;
    cc.mu = (d.mu[ga] + d.mu[gb]) / 2.0;
    const double ea = d.bounce[ga], eb = d.bounce[gb];
    cc.e = f_le(ea, eb) ? ea : eb;
    cc.no_bounce = (small_mag(cc.ra[0]) & small_mag(cc.ra[1]) & small_mag(cc.ra[2]) & small_mag(cc.ra[3]) &
                    below_two(nx) & below_two(ny) & (mag_bits(cc.e) == 0)) ? 1 : 0;
    cc.pad = 0;
    if (staged) s_con[threadIdx.x] = cc;
    else d.con[c] = cc;
    /* warm-start lookup */
    double l0 = 0.0, l1 = 0.0;
    uint8_t hit = 0;
    if (warm_start) {
      /* keys strictly descending.  From one step to the next a world's contacts hardly change: the search starts at the
       * contact's place of now and widens from there (a settled world: one access, its neighbours' the same line, in
       * place of one per bit of the world's contact count, each waiting for the last) */
      const int first = d.old_cwo[wld], end = d.old_cwo[wld + 1];
      int lo = first, hi = end - 1, at = min(first + (c - d.world_contact_off[wld]), hi), step = 1;
      bool below = false, above = false; /* bounded by a key that was read */
      while (lo <= hi) {
        const uint64_t k = d.old_key[at];
        if (k == key) {
          hit = 1;
          l0 = d.old_lam[2 * at];
          l1 = d.old_lam[2 * at + 1];
          break;
        }
        if (k > key) {
          lo = at + 1;
          below = true;
        } else {
          hi = at - 1;
          above = true;
        }
        if (below && above) {
          at = (lo + hi) >> 1;
        } else {
          at = below ? min(lo + step - 1, hi) : max(hi - step + 1, lo);
          step <<= 1;
        }
      }
    }
    if (d.miss_flag)
      d.miss_flag[c] = (warm_start && !hit && (d.collect_all || d.learned_mask[wld])) ? 1 : 0;
    uint8_t info = hit ? kInfoHit : 0;
    if (!(d.flags[ga] & kFlagStatic)) info |= kInfoDynA;
    if (!(d.flags[gb] & kFlagStatic)) info |= kInfoDynB;
    d.c_hit[c] = info;
    d.lam[2 * c] = l0;
    d.lam[2 * c + 1] = l1;
  };
  for (int base = blockIdx.x * blockDim.x + (threadIdx.x & ~31); base < n; base += gridDim.x * blockDim.x) {
    if (base + lane < n) one(base + lane);
    if (!build_solver || !staged) continue;
    __syncwarp();
    const int4* src = reinterpret_cast<const int4*>(s_con + (threadIdx.x & ~31));
    int4* dst = reinterpret_cast<int4*>(d.con + base);
    const int words = min(32, n - base) * (int)(sizeof(Con) / 16);
    for (int k = lane; k < words; k += 32) dst[k] = src[k];
    __syncwarp();
  }
}

/* ------------------------------------------------------------------------ */
/* A9-A10 one update                                                          */
/* ------------------------------------------------------------------------ */

/* J . v as a left fold (Shapes/Linear/Template.hs:108-110) of a stored row. */
__device__ __forceinline__ double row_dot(const double r[4], const double v[6]) {
  double s = (-r[0]) * v[0];
  s = s + (-r[1]) * v[1];
  s = s + r[2] * v[2];
  s = s + r[0] * v[3];
  s = s + r[1] * v[4];
  return s + r[3] * v[5];
}

/* The restitution term (bounceB, Restitution.hs:34-51): min 0 (e * (closing
 * velocity . n)), closing velocity ((-va + (-wa) z x ra) + vb) + wb z x rb. */
__device__ __forceinline__ double bounce_term(const Con* con, const double v[6]) {
  const double nwa = -v[2];
  const double cvx = ((-v[0] + (-(nwa * con->ra[1]))) + v[3]) + (-(v[5] * con->ra[3]));
  const double cvy = ((-v[1] + nwa * con->ra[0]) + v[4]) + v[5] * con->ra[2];
  const double tb = con->e * (cvx * con->rn[0] + cvy * con->rn[1]);
  return f_le(0.0, tb) ? 0.0 : tb;
}

/* Every velocity component below 2^500 in magnitude. */
__device__ __forceinline__ bool small_velocities(const double v[6]) {
  return small_mag(v[0]) & small_mag(v[1]) & small_mag(v[2]) & small_mag(v[3]) & small_mag(v[4]) & small_mag(v[5]);
}

/* improveContactSln (Solvers/Contact.hs:124-143) up to the clamps, on one
 * lane: the impulses to apply and the new accumulated Lagrangians.  Both new
 * Lagrangians come from the same velocities (contactLagrangian,
 * Constraints/Contact.hs:86-95; lagrangian2, Constraint.hs:164-169), then
 * positive / clampAbs (SolutionProcessors.hs:33-53).  Where no_bounce holds and
 * the velocities are below 2^500 the bounce product is a signed zero and its
 * minimum with 0 is +0, so b + bounceB is the stored b + 0.0 bit for bit. */
__device__ __forceinline__ void contact_impulses(const Con* con, const double rn[4], const double rf[4],
                                                 const double v[6], double2 cached, double* ln, double* lf,
                                                 double2* now) {
  double bias = con->bn0;
  if (!(con->no_bounce && small_velocities(v))) bias = con->bn + bounce_term(con, v);
  const double ln_new = div_rn(flip_sign(row_dot(rn, v) + bias), con->mc[0], con->rc[0]);
  const double lf_new = div_rn(flip_sign(plus_zero(row_dot(rf, v))), con->mc[1], con->rc[1]);
  const double neg_cn = flip_sign(cached.x);
  *ln = f_le(ln_new, neg_cn) ? neg_cn : ln_new;
  now->x = cached.x + *ln;
  now->y = clamp_abs(cached.y + lf_new, now->x * con->mu);
  *lf = now->y - cached.y;
}

/* Per-world solver residual after the last sweep: one more improveContactSln
 * pass over the world's contacts that applies nothing (every contact sees the
 * final velocities), reporting sqrt(mean over contacts of the normal and
 * friction amounts it would apply, squared).  The squared amounts of one
 * contact: */
__device__ __forceinline__ double residual_term(const Dev& d, int c) {
  const int ga = d.c_ga[c], gb = d.c_gb[c];
  const Con* con = d.con + c;
  const double v[6] = {d.vx[ga], d.vy[ga], d.w[ga], d.vx[gb], d.vy[gb], d.w[gb]};
  double ln, lf;
  double2 now;
  contact_impulses(con, con->row[0], con->row[1], v, reinterpret_cast<const double2*>(d.lam)[c], &ln, &lf, &now);
  return ln * ln + lf * lf;
}

/* One warp per world (fixed summation order); worlds of `split_from` bodies
 * or more are left to k_residual_part / k_metric_final. */
__global__ void k_residual(Dev d, int split_from) {
  const int lane = threadIdx.x & 31;
  const int wld = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (wld >= d.n_worlds) return;
  if (d.world_body_off[wld + 1] - d.world_body_off[wld] >= split_from) return;
  const int c0 = d.world_contact_off[wld], c1 = d.world_contact_off[wld + 1];
  double sum = 0.0;
  for (int c = c0 + lane; c < c1; c += 32) sum += residual_term(d, c);
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if (lane == 0) d.world_residual[wld] = c1 > c0 ? sqrt(sum / (2.0 * (c1 - c0))) : 0.0;
}

/* Per-world maximum penetration depth over the contacts of the last collide.
 * One warp per world; worlds of `split_from` bodies or more are left to
 * k_depth_part / k_metric_final. */
__global__ void k_world_depth(Dev d, int split_from) {
  const int lane = threadIdx.x & 31;
  const int wld = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (wld >= d.n_worlds) return;
  if (d.world_body_off[wld + 1] - d.world_body_off[wld] >= split_from) return;
  const int c0 = d.world_contact_off[wld], c1 = d.world_contact_off[wld + 1];
  double m = 0.0;
  for (int c = c0 + lane; c < c1; c += 32) m = fmax(m, d.c_val[5 * (size_t)c + 4]);
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) d.world_depth[wld] = m;
}

/* The same metrics for one large world over kMetricParts warps: warp k takes
 * the k-th contiguous chunk of the world's contacts, and k_metric_final
 * combines the parts in order (a fixed summation order for the residual). */
constexpr int kMetricParts = 256;

template <bool RESIDUAL>
__global__ void k_metric_part(Dev d, int wld, double* part) {
  const int lane = threadIdx.x & 31;
  const int k = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (k >= kMetricParts) return;
  const int c0 = d.world_contact_off[wld], c1 = d.world_contact_off[wld + 1];
  const int chunk = (c1 - c0 + kMetricParts - 1) / kMetricParts;
  const int a = c0 + k * chunk, b = min(c1, a + chunk);
  double acc = 0.0;
  for (int c = a + lane; c < b; c += 32) acc = RESIDUAL ? acc + residual_term(d, c) : fmax(acc, d.c_val[5 * (size_t)c + 4]);
  for (int o = 16; o > 0; o >>= 1) {
    const double t = __shfl_xor_sync(0xffffffffu, acc, o);
    acc = RESIDUAL ? acc + t : fmax(acc, t);
  }
  if (lane == 0) part[k] = acc;
}

template <bool RESIDUAL>
__global__ void k_metric_final(Dev d, int wld, const double* part) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  double acc = 0.0;
  for (int k = 0; k < kMetricParts; ++k) acc = RESIDUAL ? acc + part[k] : fmax(acc, part[k]);
  const int n = d.world_contact_off[wld + 1] - d.world_contact_off[wld];
  if (RESIDUAL)
    d.world_residual[wld] = n > 0 ? sqrt(acc / (2.0 * n)) : 0.0;
  else
    d.world_depth[wld] = acc;
}

}  // namespace shapes
