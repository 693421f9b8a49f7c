// tree.cu -- octree construction in HBM (replaces src/tree.jl:3-122).
//
// The reference builds its octree top-down, sorting each splitting branch's
// bodies into octants with a stable counting sort, where the octant of a body
// is decided by strict `>` comparisons against the branch's FP64 centre, and
// child centres are parent_centre +- parent_box/2 (src/tree.jl:433-592).
// Here every body computes its whole octant path at once: the centre
// recursion is replayed per body with the same FP64 operations (this file is
// compiled with -fmad=false, so every product and sum is rounded exactly as
// in the reference), giving a 63-bit key (21 levels x 3 bits).  One radix sort
// of the keys then yields the branch structure level by level: a branch
// splits iff exceeds(n_bodies) (src/tree.jl:492-569), its children are the
// runs of the next key digit, emitted in octant order, so branches come out in
// the reference's breadth-first order with identical body ranges.  Finally the
// bodies inside each leaf are put back in input order (the reference's
// per-level sorts are stable and leaves are never sorted), by one kernel that also
// moves the bodies, shrinks the leaves and, from the last child of every parent to
// finish, the branches above them.
//
// The levels are built without the host: one cluster of CTAs takes level after level
// while a level is small (all of a small tree), and larger levels take two launches each
// whose bounds are read from device memory.  The host waits once for a small tree and once
// per kLevelBatch large levels.  (Before: six launches and a host round trip per level, a second
// radix sort for the order inside the leaves, a launch per level to shrink the branches.  Tree and
// lists of 1,000 bodies 0.43 -> 0.20 ms, of 10,000 0.68 -> 0.31 ms, of 1e6 2.36 -> 1.80 ms; bound by
// the latency of dependent small launches and of the radix passes.)
#include <cooperative_groups.h>

#include <climits>
#include <utility>

#include <cub/cub.cuh>

#include "context.cuh"

namespace cg = cooperative_groups;

namespace fmmb {

namespace {

constexpr int kThreads = 256;
constexpr int kRankMax = 1024;  // largest leaf ordered by comparisons (n^2 / 32 of them per warp)

inline int blocks_for(int64_t n, int t = kThreads) {
  int64_t b = (n + t - 1) / t;
  if (b < 1) b = 1;
  if (b > 148 * 64) b = 148 * 64;
  return (int)b;
}

struct RootGeom {
  double c[3];
  double bmax;
  double radius;
};

__global__ void k_unpack(const double* __restrict__ buf, int64_t n, int64_t stride, int ns, int has_r,
                         double4* __restrict__ pos, double4* __restrict__ str) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* b = buf + i * stride;
    pos[i] = make_double4(b[0], b[1], b[2], has_r ? b[3] : 0.0);
    double4 s = make_double4(0, 0, 0, 0);
    if (ns >= 1) s.x = b[4];
    if (ns >= 3) {
      s.y = b[5];
      s.z = b[6];
    }
    str[i] = s;
  }
}

// Progress of a build, in device memory.
enum : int { kIdle = 0, kRunning, kDone, kNoRoom, kFullSort, kTooDeep };
struct TreeState {
  int status;                // how the build ended (kIdle: not yet)
  int ticket;                // blocks of k_bbox that have finished
  int n_levels;              // levels that exist; the last one is still to split when kIdle
  int max_leaf;              // bodies of the largest leaf
  int lev[kMaxDepth + 3];    // first branch of every level
  int leaf0[kMaxDepth + 3];  // leaves before every level
  int run[kMaxDepth + 3];    // kRunning: the level is to be split
  int stop[kMaxDepth + 3];   // why a level cannot be split
};

// extents of the bodies, then (the last block to finish) center_box / get_center_box
// (src/tree.jl:894-924) and the cubic root cell (src/tree.jl:20-26); min / max are exact in any order
__global__ void k_bbox(const double4* __restrict__ pos, int64_t n, double* __restrict__ part, TreeState* st,
                       RootGeom* root) {
  double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double4 p = pos[i];
    mn[0] = fmin(mn[0], p.x); mx[0] = fmax(mx[0], p.x);
    mn[1] = fmin(mn[1], p.y); mx[1] = fmax(mx[1], p.y);
    mn[2] = fmin(mn[2], p.z); mx[2] = fmax(mx[2], p.z);
  }
  __shared__ double s[6][kThreads / 32];
  __shared__ bool last;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  auto reduce = [&](int nw) {  // the block's (nw warps') extents into s[..][0]
    for (int k = 0; k < 3; ++k)
      for (int o = 16; o > 0; o >>= 1) {
        mn[k] = fmin(mn[k], __shfl_xor_sync(0xffffffffu, mn[k], o));
        mx[k] = fmax(mx[k], __shfl_xor_sync(0xffffffffu, mx[k], o));
      }
    if (lane == 0)
      for (int k = 0; k < 3; ++k) s[k][w] = mn[k], s[3 + k][w] = mx[k];
    __syncthreads();
    if (threadIdx.x == 0)
      for (int q = 1; q < nw; ++q)
        for (int k = 0; k < 3; ++k) s[k][0] = fmin(s[k][0], s[k][q]), s[3 + k][0] = fmax(s[3 + k][0], s[3 + k][q]);
  };
  reduce(kThreads / 32);
  if (threadIdx.x == 0) {
    for (int k = 0; k < 6; ++k) part[6 * blockIdx.x + k] = s[k][0];
    __threadfence();
    last = atomicAdd(&st->ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  for (int k = 0; k < 3; ++k) mn[k] = INFINITY, mx[k] = -INFINITY;
  for (int b = threadIdx.x; b < (int)gridDim.x; b += kThreads)
    for (int k = 0; k < 3; ++k) {
      mn[k] = fmin(mn[k], __ldcg(part + 6 * b + k));
      mx[k] = fmax(mx[k], __ldcg(part + 6 * b + 3 + k));
    }
  reduce(kThreads / 32);
  if (threadIdx.x != 0) return;
  double box[3];
  for (int k = 0; k < 3; ++k) {
    root->c[k] = (s[3 + k][0] + s[k][0]) * 0.5;
    box[k] = s[3 + k][0] - root->c[k];
  }
  double bmax = fmax(fmax(box[0], box[1]), box[2]);
  root->bmax = bmax;
  root->radius = sqrt(bmax * bmax * 3.0);
}

// octant path of every body: get_octant (src/tree.jl:474-480) applied level by
// level with the child-centre recursion of get_child_center (src/tree.jl:581-592)
__global__ void k_keys(const double4* __restrict__ pos, int64_t n, const RootGeom* __restrict__ root,
                       unsigned long long* __restrict__ keys, int* __restrict__ vals) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double4 p = pos[i];
    double cx = root->c[0], cy = root->c[1], cz = root->c[2];
    double box = root->bmax;
    unsigned long long key = 0;
    for (int d = 0; d < kMaxDepth; ++d) {
      int o = (p.x > cx ? 1 : 0) | (p.y > cy ? 2 : 0) | (p.z > cz ? 4 : 0);
      key = (key << 3) | (unsigned long long)o;
      double delta = box * 0.5;
      cx = cx + ((o & 1) ? delta : -delta);
      cy = cy + ((o & 2) ? delta : -delta);
      cz = cz + ((o & 4) ? delta : -delta);
      box = box * 0.5;
    }
    keys[i] = key;
    vals[i] = (int)i;
  }
}

__device__ __forceinline__ int key_digit(unsigned long long k, int l) {
  return (int)((k >> (3 * (kMaxDepth - 1 - l))) & 7ull);
}

// first position in [lo, hi) whose level-l digit is >= o (three probes a round: the rounds' loads,
// not the comparisons, take the time)
__device__ int lower_bound_digit(const unsigned long long* keys, int lo, int hi, int l, int o) {
  while (hi - lo > 3) {
    const int q = (hi - lo) >> 2, a = lo + q, b = a + q, c = b + q;
    const bool pa = key_digit(keys[a], l) < o, pb = key_digit(keys[b], l) < o, pc = key_digit(keys[c], l) < o;
    if (pb) {
      lo = (pc ? c : b) + 1;
      if (!pc) hi = c;
    } else {
      hi = pa ? b : a;
      if (pa) lo = a + 1;
    }
  }
  while (lo < hi && key_digit(keys[lo], l) < o) ++lo;
  return lo;
}

// exceeds(..., method), src/tree.jl:492-569 (same FP operations)
__device__ __forceinline__ bool exceeds(int n, int64_t ls, int method) {
  if (method == FMM_LIST_BARBA) return n > ls;
  double fraction = 0.0;
  fraction = fraction + (double)n / (double)(ls * ls);
  fraction = fraction * (double)ls;
  if (method == FMM_LIST_SELF_TUNING) return fraction > 0.5 && n > 1;
  return fraction > 2.8284271247461903 && n > 1;
}

// The children of a splitting level-l branch are the runs of key digit l among its
// bodies.  Eight lanes per branch: lane o finds where octant o starts (a binary search
// over the branch's keys, in parallel instead of seven chained searches), lane o + 1
// where it ends.
constexpr unsigned kFullMask = 0xffffffffu;
struct Branches {
  int *body_start, *body_count, *child_start, *n_children, *parent, *level, *i_leaf, *leaf_index, *done;
  double *gcenter, *gbox, *gradius;
  int cap;
};
struct Rules {
  const unsigned long long* keys;
  int64_t leaf_size;
  int method;
  int depth;  // levels that the keys are sorted for
};
struct Octants {
  int o;       // this lane's octant
  bool in;     // the lane's group holds a branch
  bool leaf;   // which does not split
  int b, e;    // bodies of octant o: [b, e)
  int cnt;     // bodies of the branch
  unsigned nonempty;  // bit q: octant q holds bodies (all lanes of the group)
};
// stop: kTooDeep / kFullSort when the branch would split below the keys' depth (all lanes), else 0
__device__ __forceinline__ Octants octants_of(const Rules& R, const Branches& B, int k, bool in, int level, int& stop) {
  Octants r;
  r.o = threadIdx.x & 7;
  r.in = in;
  r.cnt = in ? B.body_count[k] : 0;
  bool split = in && exceeds(r.cnt, R.leaf_size, R.method);
  if (split && level >= R.depth) {
    stop = level >= kMaxDepth ? kTooDeep : kFullSort;
    split = false;
  }
  r.leaf = in && !split;
  const int lo = split ? B.body_start[k] : 0, hi = lo + (split ? r.cnt : 0);
  r.b = r.o == 0 ? lo : lower_bound_digit(R.keys, lo, hi, level, r.o);
  const int nb = __shfl_down_sync(kFullMask, r.b, 1, 8);
  r.e = r.o == 7 ? hi : nb;
  const unsigned ball = __ballot_sync(kFullMask, split && r.e > r.b);
  r.nonempty = (ball >> ((threadIdx.x & 31) & ~7)) & 0xffu;
  return r;
}

// (children, leaves) of the groups before this one in the block, one warp-wide value per group;
// total: of the block.  sh: two ints per warp.  Every thread of the block calls it.
__device__ __forceinline__ int2 scan_groups(int children, int leaf, int2* sh, int2& total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
  int c = (lane & 7) == 0 ? children : 0, f = (lane & 7) == 0 ? leaf : 0;
  const int c0 = c, f0 = f;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int x = __shfl_up_sync(kFullMask, c, o), y = __shfl_up_sync(kFullMask, f, o);
    if (lane >= o) c += x, f += y;
  }
  if (lane == 31) sh[w] = make_int2(c, f);
  __syncthreads();
  int2 ex = make_int2(c - c0, f - f0);
  ex.x = __shfl_sync(kFullMask, ex.x, lane & ~7);
  ex.y = __shfl_sync(kFullMask, ex.y, lane & ~7);
  total = make_int2(0, 0);
  for (int q = 0; q < nw; ++q) {
    if (q < w) ex.x += sh[q].x, ex.y += sh[q].y;
    total.x += sh[q].x;
    total.y += sh[q].y;
  }
  __syncthreads();
  return ex;
}

// branch k of one level: its children at base .. (breadth-first order), or its leaf ordinal
__device__ __forceinline__ void emit(const Branches& B, const Octants& r, int k, int level, int base, int leaf) {
  if (!r.in) return;
  const int o = r.o;
  if (o == 0) {
    B.child_start[k] = base;
    B.n_children[k] = __popc(r.nonempty);
    B.i_leaf[k] = r.leaf ? leaf : -1;
    B.done[k] = 0;
    if (r.leaf) B.leaf_index[leaf] = k;
  }
  if (!((r.nonempty >> o) & 1u)) return;
  const int c = base + __popc(r.nonempty & ((1u << o) - 1u));
  const double pbox = B.gbox[k], prad = B.gradius[k];
  B.body_start[c] = r.b;
  B.body_count[c] = r.e - r.b;
  B.parent[c] = k;
  B.level[c] = level + 1;
  const double delta = pbox * 0.5;  // get_child_center: parent box is a cube of half width pbox
  B.gcenter[3 * c] = B.gcenter[3 * k] + ((o & 1) ? delta : -delta);
  B.gcenter[3 * c + 1] = B.gcenter[3 * k + 1] + ((o & 2) ? delta : -delta);
  B.gcenter[3 * c + 2] = B.gcenter[3 * k + 2] + ((o & 4) ? delta : -delta);
  B.gbox[c] = pbox * 0.5;
  B.gradius[c] = prad * 0.5;
}

// The root and the levels of up to kCluMaxLevel branches: one cluster, 512 branches at a time,
// each CTA's share counted, the shares' sums exchanged through distributed shared memory.
constexpr int kClu = 8, kCluThreads = 512, kCluGroups = kCluThreads / 8;
constexpr int kCluMaxLevel = 4096;
__global__ void __cluster_dims__(kClu, 1, 1) __launch_bounds__(kCluThreads)
    k_levels_cluster(Rules R, Branches B, int n, const RootGeom* __restrict__ root, TreeState* st) {
  cg::cluster_group clu = cg::this_cluster();
  __shared__ int2 sh[kCluThreads / 32];
  __shared__ int2 mine[2];  // this CTA's (children, leaves), double-buffered over the exchanges
  __shared__ int stopped[2];
  const int rank = (int)clu.block_rank();
  if (rank == 0 && threadIdx.x == 0) {
    B.body_start[0] = 0;
    B.body_count[0] = n;
    B.parent[0] = -1;
    B.level[0] = 0;
    for (int k = 0; k < 3; ++k) B.gcenter[k] = root->c[k];
    B.gbox[0] = root->bmax;
    B.gradius[0] = root->radius;
    st->lev[0] = 0;
    st->lev[1] = 1;
    st->leaf0[0] = 0;
  }
  clu.sync();
  int ls = 0, le = 1, level = 0, leaves = 0, status = kIdle, buf = 0, max_leaf = 0;
  for (;;) {
    int made = 0;
    for (int g0 = 0; g0 < le - ls; g0 += kClu * kCluGroups) {
      const int k = ls + g0 + rank * kCluGroups + (threadIdx.x >> 3);
      int stop = 0;
      const Octants r = octants_of(R, B, k, k < le, level, stop);
      if (threadIdx.x == 0) stopped[buf] = 0;
      int2 total;
      const int2 ex = scan_groups(__popc(r.nonempty), r.leaf ? 1 : 0, sh, total);
      if (stop) stopped[buf] = stop;
      if (threadIdx.x == 0) mine[buf] = total;
      clu.sync();
      int2 before = make_int2(0, 0), all = make_int2(0, 0);
      int stop_all = 0;
      for (int q = 0; q < kClu; ++q) {
        const int2 v = *clu.map_shared_rank(&mine[buf], q);
        stop_all = max(stop_all, *clu.map_shared_rank(&stopped[buf], q));
        if (q < rank) before.x += v.x, before.y += v.y;
        all.x += v.x;
        all.y += v.y;
      }
      buf ^= 1;
      if (stop_all) status = stop_all;
      if (le + made + all.x > B.cap) status = status ? status : (int)kNoRoom;
      if (status) break;
      emit(B, r, k, level, le + made + before.x + ex.x, leaves + before.y + ex.y);
      if (r.leaf) max_leaf = max(max_leaf, r.cnt);
      made += all.x;
      leaves += all.y;
    }
    if (status) break;
    if (rank == 0 && threadIdx.x == 0) {
      st->lev[level + 2] = le + made;
      st->leaf0[level + 1] = leaves;
    }
    if (made == 0) {
      status = kDone;
      break;
    }
    ls = le;
    le += made;
    ++level;
    clu.sync();  // the children are read by every CTA
    if (le - ls > kCluMaxLevel) break;
  }
  for (int o = 16; o > 0; o >>= 1) max_leaf = max(max_leaf, __shfl_xor_sync(kFullMask, max_leaf, o));
  if ((threadIdx.x & 31) == 0 && max_leaf) atomicMax(&st->max_leaf, max_leaf);
  if (rank == 0 && threadIdx.x == 0) {
    st->status = status;
    st->n_levels = level + 1;
    st->run[level] = status == kIdle ? kRunning : kIdle;
  }
  clu.sync();  // no CTA leaves while its shared memory may be read
}

// A larger level: every block counts a contiguous share of its branches (children, leaves), then
// adds up the shares before its own and emits.  Bounds come from the state, so that levels are
// launched without the host knowing them; a level past the last does nothing.
constexpr int kLvlThreads = 128, kLvlGroups = kLvlThreads / 8, kLvlBlocks = 148 * 8, kLevelBatch = 4;
__device__ __forceinline__ bool level_share(const TreeState* st, int level, int& ls, int& le, int& b, int& e) {
  if (st->run[level] != kRunning) return false;
  ls = st->lev[level];
  le = st->lev[level + 1];
  const int per = ((le - ls + (int)gridDim.x * kLvlGroups - 1) / ((int)gridDim.x * kLvlGroups)) * kLvlGroups;
  b = min(ls + (int)blockIdx.x * per, le);
  e = min(b + per, le);
  return true;
}
__global__ void __launch_bounds__(kLvlThreads) k_level_count(Rules R, Branches B, int level, TreeState* st,
                                                             int2* __restrict__ share) {
  __shared__ int2 sh[kLvlThreads / 32];
  int ls, le, b, e;
  if (!level_share(st, level, ls, le, b, e)) return;
  int2 sum = make_int2(0, 0);
  for (int k0 = b; k0 < e; k0 += kLvlGroups) {
    const int k = k0 + (threadIdx.x >> 3);
    int stop = 0;
    const Octants r = octants_of(R, B, k, k < e, level, stop);
    int2 total;
    scan_groups(__popc(r.nonempty), r.leaf ? 1 : 0, sh, total);
    sum.x += total.x;
    sum.y += total.y;
    if (stop) atomicMax(&st->stop[level], stop);
  }
  if (threadIdx.x == 0) share[blockIdx.x] = sum;
}
__global__ void __launch_bounds__(kLvlThreads) k_level_emit(Rules R, Branches B, int level, TreeState* st,
                                                            const int2* __restrict__ share) {
  __shared__ int2 sh[kLvlThreads / 32];
  __shared__ int2 acc[2];
  int ls, le, b, e;
  if (!level_share(st, level, ls, le, b, e)) return;
  // shares before this block's, and all of them
  int2 before = make_int2(0, 0), all = make_int2(0, 0);
  for (int q = threadIdx.x; q < (int)gridDim.x; q += kLvlThreads) {
    const int2 v = share[q];
    if (q < (int)blockIdx.x) before.x += v.x, before.y += v.y;
    all.x += v.x;
    all.y += v.y;
  }
  if (threadIdx.x < 2) acc[threadIdx.x] = make_int2(0, 0);
  __syncthreads();
  atomicAdd(&acc[0].x, before.x);
  atomicAdd(&acc[0].y, before.y);
  atomicAdd(&acc[1].x, all.x);
  atomicAdd(&acc[1].y, all.y);
  __syncthreads();
  before = acc[0];
  all = acc[1];
  const int stop = st->stop[level];
  const int end = stop ? stop : le + all.x > B.cap ? (int)kNoRoom : all.x == 0 ? (int)kDone : (int)kIdle;
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->lev[level + 2] = le + all.x;
    st->leaf0[level + 1] = st->leaf0[level] + all.y;
    st->n_levels = level + 1 + (all.x > 0);
    st->status = end;
    if (end == kIdle) st->run[level + 1] = kRunning;
  }
  if (end == kNoRoom || stop) return;
  const int leaf0 = st->leaf0[level];
  int max_leaf = 0;
  for (int k0 = b; k0 < e; k0 += kLvlGroups) {
    const int k = k0 + (threadIdx.x >> 3);
    int s_ = 0;
    const Octants r = octants_of(R, B, k, k < e, level, s_);
    int2 total;
    const int2 ex = scan_groups(__popc(r.nonempty), r.leaf ? 1 : 0, sh, total);
    emit(B, r, k, level, le + before.x + ex.x, leaf0 + before.y + ex.y);
    if (r.leaf) max_leaf = max(max_leaf, r.cnt);
    before.x += total.x;
    before.y += total.y;
  }
  for (int o = 16; o > 0; o >>= 1) max_leaf = max(max_leaf, __shfl_xor_sync(kFullMask, max_leaf, o));
  if ((threadIdx.x & 31) == 0 && max_leaf) atomicMax(&st->max_leaf, max_leaf);
}

// key of the final order: the body_start of the leaf holding sorted position i,
// scattered to the body's input index
__global__ void k_leaf_keys(const int* __restrict__ leaf_index, int n_leaves, const int* __restrict__ body_start,
                            const int* __restrict__ body_count, const int* __restrict__ perm,
                            unsigned int* __restrict__ key_by_input) {
  int lane = threadIdx.x & 31;
  int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= n_leaves) return;
  int b = leaf_index[w];
  int s = body_start[b], c = body_count[b];
  for (int i = lane; i < c; i += 32) key_by_input[perm[s + i]] = (unsigned int)s;
}

__global__ void k_iota(int* v, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    v[i] = (int)i;
}

__global__ void k_permute(const double4* __restrict__ in_pos, const double4* __restrict__ in_str,
                          const int* __restrict__ sort_index, int64_t n, double4* __restrict__ pos,
                          double4* __restrict__ str) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int j = sort_index[i];
    pos[i] = in_pos[j];
    str[i] = in_str[j];
  }
}

// geometric cells without shrinking
__global__ void k_copy_geometry(int nb, const double* gcenter, const double* gbox, const double* gradius,
                                double* tc, double* sc, double* tr, double* sr, double* tb, double* sb) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= nb) return;
  for (int d = 0; d < 3; ++d) {
    tc[3 * k + d] = sc[3 * k + d] = gcenter[3 * k + d];
    tb[3 * k + d] = sb[3 * k + d] = gbox[k];
  }
  tr[k] = sr[k] = gradius[k];
}

// min / max over an aligned group of G lanes (exact, so the grouping does not matter)
template <int G = 32>
__device__ __forceinline__ double wmin(double v) {
  for (int o = G / 2; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
template <int G = 32>
__device__ __forceinline__ double wmax(double v) {
  for (int o = G / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// branch geometry of one tree (k_leaf_bodies)
struct Geometry {
  double *tc, *sc, *tr, *sr, *tb, *sb;
};

// min / max over the first eight lanes of a group, by that group's lanes alone (mask)
__device__ __forceinline__ double min8(unsigned mask, double v) {
  for (int o = 4; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(mask, v, o));
  return v;
}
__device__ __forceinline__ double max8(unsigned mask, double v) {
  for (int o = 4; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(mask, v, o));
  return v;
}

// shrink_branch! (src/tree.jl:1163-1174), one lane per child (eight lanes; those past the children
// repeat the first); the children were written by other SMs
__device__ __forceinline__ void shrink_branch(const Geometry& G, unsigned mask, int lane, int k, int c0, int nc) {
  const int c = c0 + (lane < nc ? lane : 0);
  double tc[3], sc[3], tcen[3], scen[3], tb[3], sb[3];
  for (int d = 0; d < 3; ++d) {
    tc[d] = __ldcg(G.tc + 3 * c + d);
    sc[d] = __ldcg(G.sc + 3 * c + d);
    tb[d] = __ldcg(G.tb + 3 * c + d);
    sb[d] = __ldcg(G.sb + 3 * c + d);
  }
  const double tr = __ldcg(G.tr + c), sr = __ldcg(G.sr + c);
  for (int d = 0; d < 3; ++d) {
    // the first child's centre takes part too, as in the reference
    const double tmn = min8(mask, fmin(tc[d], tc[d] - tb[d])), tmx = max8(mask, fmax(tc[d], tc[d] + tb[d]));
    const double smn = min8(mask, fmin(sc[d], sc[d] - sb[d])), smx = max8(mask, fmax(sc[d], sc[d] + sb[d]));
    tcen[d] = (tmn + tmx) * 0.5;
    scen[d] = (smn + smx) * 0.5;
    tb[d] = tmx - tcen[d];
    sb[d] = smx - scen[d];
  }
  double dx = tc[0] - tcen[0], dy = tc[1] - tcen[1], dz = tc[2] - tcen[2];
  const double trad = max8(mask, fmax(0.0, sqrt(dx * dx + dy * dy + dz * dz) + tr));
  dx = sc[0] - scen[0];
  dy = sc[1] - scen[1];
  dz = sc[2] - scen[2];
  const double srad = max8(mask, fmax(0.0, sqrt(dx * dx + dy * dy + dz * dz) + sr));
  if (lane != 0) return;
  for (int d = 0; d < 3; ++d) {
    G.tc[3 * k + d] = tcen[d];
    G.sc[3 * k + d] = scen[d];
    G.tb[3 * k + d] = tb[d];
    G.sb[3 * k + d] = sb[d];
  }
  G.tr[k] = trad;
  G.sr[k] = srad;
}

// One leaf per group of G lanes (32, or 8 when the leaves hold a few bodies).
// MOVE: puts the leaf's bodies back in input order (the rank of a body is the number of the leaf's
// bodies with a smaller input index) and moves them to their sorted places; perm holds the input
// index of every position of the key order.  Otherwise the bodies are in place.
// shrink: shrink_leaf! (src/tree.jl:1141-1161), then shrink_branch! of every ancestor whose last
// child this is (done counts the finished children).
template <int G, bool MOVE>
__global__ void k_leaf_bodies(Branches B, int n_leaves, const int* __restrict__ perm,
                              const double4* __restrict__ in_pos, const double4* __restrict__ in_str,
                              int* __restrict__ sort_index, double4* __restrict__ pos, double4* __restrict__ str,
                              int shrink, Geometry geo) {
  const int lane = threadIdx.x & (G - 1);
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) / G;
  const bool valid = w < n_leaves;
  const int b = B.leaf_index[valid ? w : n_leaves - 1];
  const int s = B.body_start[b], c = valid ? B.body_count[b] : 0;
  if (MOVE) {
    int top = c;
    for (int o = 16; o >= G; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
    for (int i0 = 0; i0 < top; i0 += G) {
      const int i = i0 + lane;
      const int v = i < c ? perm[s + i] : INT_MAX;
      int rank = 0;
      for (int j0 = 0; j0 < top; j0 += G) {
        const int u = j0 + lane < c ? perm[s + j0 + lane] : INT_MAX;
#pragma unroll
        for (int q = 0; q < G; ++q) rank += __shfl_sync(0xffffffffu, u, q, G) < v;
      }
      if (i < c) {
        sort_index[s + rank] = v;
        pos[s + rank] = in_pos[v];
        str[s + rank] = in_str[v];
      }
    }
  }
  if (!shrink) return;
  auto body = [&](int i) { return MOVE ? in_pos[perm[s + i]] : pos[s + i]; };
  const double4 p0 = body(0);
  double tmn[3] = {p0.x, p0.y, p0.z}, tmx[3] = {p0.x, p0.y, p0.z};
  double smn[3] = {p0.x, p0.y, p0.z}, smx[3] = {p0.x, p0.y, p0.z};
  for (int i = lane; i < c; i += G) {
    double4 p = body(i);
    double x[3] = {p.x, p.y, p.z};
    for (int d = 0; d < 3; ++d) {
      tmn[d] = fmin(tmn[d], x[d]);
      tmx[d] = fmax(tmx[d], x[d]);
      smn[d] = fmin(smn[d], x[d] - p.w);
      smx[d] = fmax(smx[d], x[d] + p.w);
    }
  }
  double tcen[3], scen[3];
  for (int d = 0; d < 3; ++d) {
    tmn[d] = wmin<G>(tmn[d]);
    tmx[d] = wmax<G>(tmx[d]);
    smn[d] = wmin<G>(smn[d]);
    smx[d] = wmax<G>(smx[d]);
    tcen[d] = (tmx[d] + tmn[d]) * 0.5;
    scen[d] = (smx[d] + smn[d]) * 0.5;
  }
  double trad = 0.0, srad = 0.0;
  for (int i = lane; i < c; i += G) {
    double4 p = body(i);
    double dx = p.x - tcen[0], dy = p.y - tcen[1], dz = p.z - tcen[2];
    trad = fmax(trad, sqrt(dx * dx + dy * dy + dz * dz));
    dx = p.x - scen[0];
    dy = p.y - scen[1];
    dz = p.z - scen[2];
    srad = fmax(srad, sqrt(dx * dx + dy * dy + dz * dz) + p.w);
  }
  trad = wmax<G>(trad);
  srad = wmax<G>(srad);
  if (!valid || lane >= 8) return;
  if (lane == 0) {
    for (int d = 0; d < 3; ++d) {
      geo.tc[3 * b + d] = tcen[d];
      geo.sc[3 * b + d] = scen[d];
      geo.tb[3 * b + d] = tmx[d] - tcen[d];
      geo.sb[3 * b + d] = smx[d] - scen[d];
    }
    geo.tr[b] = trad;
    geo.sr[b] = srad;
  }
  const unsigned mask = 0xffu << (threadIdx.x & 31 & ~7);  // the group's first eight lanes
  for (int k = B.parent[b]; k >= 0; k = B.parent[k]) {
    const int nc = B.n_children[k];
    int last = 0;
    if (lane == 0) {
      __threadfence();
      last = atomicAdd(B.done + k, 1) == nc - 1;
      __threadfence();
    }
    if (!__shfl_sync(mask, last, 0, 8)) break;
    __syncwarp(mask);  // the other lanes' loads of the children after lane 0's fence (a shuffle orders no memory)
    shrink_branch(geo, mask, lane, k, B.child_start[k], nc);
    __syncwarp(mask);
  }
}

// estimate_influence! tail (src/fmm.jl:1236-1262): max |grad| over each branch's bodies
// of a leaf's bodies, then into every ancestor (non-negative doubles order as their bits do); a
// walk ends where an equal or larger value has already passed
__global__ void k_leaf_maxinf(const int* __restrict__ leaf_index, int n_leaves, const int* __restrict__ body_start,
                              const int* __restrict__ body_count, const int* __restrict__ parent,
                              const int* __restrict__ sort_index, const double* __restrict__ gnorm, double* mi) {
  int lane = threadIdx.x & 31;
  int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (w >= n_leaves) return;
  int b = leaf_index[w];
  int s = body_start[b], c = body_count[b];
  double m = 0.0;
  for (int i = lane; i < c; i += 32) {
    m = fmax(m, gnorm[sort_index[s + i]]);
  }
  m = wmax(m);
  if (lane != 0 || !(m > 0.0)) return;
  const unsigned long long v = (unsigned long long)__double_as_longlong(m);
  for (int k = b; k >= 0; k = parent[k])
    if (atomicMax(reinterpret_cast<unsigned long long*>(mi) + k, v) >= v) break;
}

}  // namespace

void unpack_bodies(DevTree& t, const double* dev_buf, int64_t n, int64_t stride, int n_strength, bool has_radius,
                   cudaStream_t st) {
  t.n_bodies = n;
  t.pos.grow(n);
  t.str.grow(n);
  if (n == 0) return;
  note_launch();
  k_unpack<<<blocks_for(n), kThreads, 0, st>>>(dev_buf, n, stride, n_strength, has_radius ? 1 : 0, t.pos.ptr,
                                               t.str.ptr);
  FMM_CUDA_TRY(cudaGetLastError());
}

void build_tree(DevTree& t, Scratch& sc, cudaStream_t st, int64_t leaf_size, int method, bool shrink) {
  const int64_t n = t.n_bodies;
  FMM_CHECK(n > 0, FMM_ERR_ARGUMENT, "build_tree: empty system");
  FMM_CHECK(n < (1ll << 31) - 64, FMM_ERR_ARGUMENT, "build_tree: more than 2^31 bodies");
  FMM_CHECK(leaf_size >= 1, FMM_ERR_ARGUMENT, "leaf_size must be >= 1");

  const size_t st_ints = (sizeof(TreeState) + 3) / 4;
  int nb_part = (int)std::min<int64_t>(blocks_for(n), 148 * 4);
  sc.tmp_d.grow(6 * (size_t)nb_part + 8);
  double* part = sc.tmp_d.ptr;
  RootGeom* root = reinterpret_cast<RootGeom*>(part + 6 * nb_part);
  sc.counts.grow(st_ints + 2 * kLvlBlocks + 2);
  TreeState* state = reinterpret_cast<TreeState*>(sc.counts.ptr);
  int2* share = reinterpret_cast<int2*>(sc.counts.ptr + ((st_ints + 1) & ~(size_t)1));
  FMM_CUDA_TRY(cudaMemsetAsync(state, 0, sizeof(TreeState), st));
  // root cell
  note_launch();
  k_bbox<<<nb_part, kThreads, 0, st>>>(t.pos.ptr, n, part, state, root);

  // octant-path keys, sorted (stable) with the body index
  sc.keys_a.grow(n);
  sc.keys_b.grow(n);
  sc.vals_a.grow(n);
  sc.vals_b.grow(n);
  note_launch();
  k_keys<<<blocks_for(n), kThreads, 0, st>>>(t.pos.ptr, n, root, sc.keys_a.ptr, sc.vals_a.ptr);
  FMM_CUDA_TRY(cudaGetLastError());
  // the digits of as many levels first as a density 8^6 times the mean would split to (four or five
  // radix passes instead of eight); all of them when a branch below still has to split
  auto sort_keys = [&](int depth) {
    const int lo = 3 * (kMaxDepth - depth);
    size_t tmp_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, sc.keys_a.ptr, sc.keys_b.ptr, sc.vals_a.ptr, sc.vals_b.ptr,
                                    (int)n, lo, 3 * kMaxDepth, st);
    sc.cub.grow(tmp_bytes);
    FMM_CUDA_TRY(cub::DeviceRadixSort::SortPairs(sc.cub.ptr, tmp_bytes, sc.keys_a.ptr, sc.keys_b.ptr, sc.vals_a.ptr,
                                                 sc.vals_b.ptr, (int)n, lo, 3 * kMaxDepth, st));
  };
  int depth = 6;
  for (int64_t m = n; m > leaf_size && depth < kMaxDepth; m >>= 3) ++depth;
  depth = std::min(kMaxDepth, (3 * depth + 7) / 8 * 8 / 3);  // to the end of a radix pass
  sort_keys(depth);
  const int* perm = sc.vals_b.ptr;

  // branches
  size_t cap = (size_t)(2 * n / std::max<int64_t>(leaf_size, 1) + 1024);
  TreeState h;
  for (;;) {
    for (DevBuf<int>* q : {&t.body_start, &t.body_count, &t.child_start, &t.n_children, &t.parent, &t.level, &t.i_leaf,
                           &t.leaf_index, &sc.tmp_k})
      q->grow(cap);
    t.gcenter.grow(3 * cap);
    t.gbox.grow(cap);
    t.gradius.grow(cap);
    const Rules R{sc.keys_b.ptr, leaf_size, method, depth};
    size_t room = std::min(t.gcenter.cap / 3, std::min(t.gbox.cap, t.gradius.cap));
    for (DevBuf<int>* q : {&t.body_start, &t.body_count, &t.child_start, &t.n_children, &t.parent, &t.level, &t.i_leaf,
                           &t.leaf_index, &sc.tmp_k})
      room = std::min(room, q->cap);
    const Branches B{t.body_start.ptr, t.body_count.ptr, t.child_start.ptr, t.n_children.ptr, t.parent.ptr,
                     t.level.ptr,      t.i_leaf.ptr,     t.leaf_index.ptr,  sc.tmp_k.ptr,     t.gcenter.ptr,
                     t.gbox.ptr,       t.gradius.ptr,    (int)std::min<size_t>(room, INT_MAX)};
    note_launch();
    k_levels_cluster<<<kClu, kCluThreads, 0, st>>>(R, B, (int)n, root, state);
    FMM_CUDA_TRY(cudaGetLastError());
    for (;;) {
      FMM_CUDA_TRY(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
      FMM_CUDA_TRY(cudaStreamSynchronize(st));
      if (h.status != kIdle) break;
      for (int l = h.n_levels - 1; l < std::min(h.n_levels - 1 + kLevelBatch, kMaxDepth + 1); ++l) {
        note_launch();
        k_level_count<<<kLvlBlocks, kLvlThreads, 0, st>>>(R, B, l, state, share);
        note_launch();
        k_level_emit<<<kLvlBlocks, kLvlThreads, 0, st>>>(R, B, l, state, share);
      }
      FMM_CUDA_TRY(cudaGetLastError());
    }
    if (h.status == kDone) break;
    FMM_CHECK(h.status != kTooDeep, FMM_ERR_TREE_DEPTH,
              "octree deeper than 21 levels: bodies are (nearly) coincident; spread them or raise leaf_size");
    if (h.status == kFullSort) {
      depth = kMaxDepth;
      sort_keys(depth);
    } else {
      cap = 4 * std::max(cap, room);
    }
    FMM_CUDA_TRY(cudaMemsetAsync(state, 0, sizeof(TreeState), st));
  }
  t.n_levels = h.n_levels;
  t.levels_start.assign(h.lev, h.lev + h.n_levels);
  t.levels_end.assign(h.lev + 1, h.lev + h.n_levels + 1);
  const int nb = h.lev[h.n_levels], nleaves = h.leaf0[h.n_levels];
  t.n_branches = nb;
  t.n_leaves = nleaves;

  // bodies into leaf order (input order inside a leaf), branch geometry: shrink_recenter!
  // (src/tree.jl:1176-1188) or the geometric cells
  t.sort_index.grow(n);
  t.tcenter.grow(3 * nb);
  t.scenter.grow(3 * nb);
  t.tradius.grow(nb);
  t.sradius.grow(nb);
  t.tbox.grow(3 * nb);
  t.sbox.grow(3 * nb);
  t.max_influence.grow(nb);
  FMM_CUDA_TRY(cudaMemsetAsync(t.max_influence.ptr, 0, nb * sizeof(double), st));
  if (!shrink) {
    note_launch();
    k_copy_geometry<<<(nb + 255) / 256, 256, 0, st>>>(nb, t.gcenter.ptr, t.gbox.ptr, t.gradius.ptr, t.tcenter.ptr,
                                                      t.scenter.ptr, t.tradius.ptr, t.sradius.ptr, t.tbox.ptr,
                                                      t.sbox.ptr);
  }
  // the unpacked bodies (input order) change places with the scratch, and back in leaf order
  sc.alt_pos.grow(n);
  sc.alt_str.grow(n);
  std::swap(t.pos, sc.alt_pos);
  std::swap(t.str, sc.alt_str);
  const Branches B{t.body_start.ptr, t.body_count.ptr, t.child_start.ptr, t.n_children.ptr, t.parent.ptr,
                   t.level.ptr,      t.i_leaf.ptr,     t.leaf_index.ptr,  sc.tmp_k.ptr,     t.gcenter.ptr,
                   t.gbox.ptr,       t.gradius.ptr,    nb};
  const Geometry geo{t.tcenter.ptr, t.scenter.ptr, t.tradius.ptr, t.sradius.ptr, t.tbox.ptr, t.sbox.ptr};
  const bool small = n <= 8 * (int64_t)nleaves;
  const int grid = (int)((nleaves * (small ? 8ll : 32ll) + 127) / 128);
  if (h.max_leaf <= kRankMax) {
    note_launch();
    if (small)
      k_leaf_bodies<8, true><<<grid, 128, 0, st>>>(B, nleaves, perm, sc.alt_pos.ptr, sc.alt_str.ptr, t.sort_index.ptr,
                                                   t.pos.ptr, t.str.ptr, shrink ? 1 : 0, geo);
    else
      k_leaf_bodies<32, true><<<grid, 128, 0, st>>>(B, nleaves, perm, sc.alt_pos.ptr, sc.alt_str.ptr,
                                                    t.sort_index.ptr, t.pos.ptr, t.str.ptr, shrink ? 1 : 0, geo);
  } else {
    // leaves too large for ranks by comparison: one radix sort by leaf of the input indices
    unsigned int* key_in = reinterpret_cast<unsigned int*>(sc.keys_a.ptr);
    unsigned int* key_out = key_in + n;
    note_launch();
    k_leaf_keys<<<(int)((nleaves * 32ll + 255) / 256), 256, 0, st>>>(t.leaf_index.ptr, nleaves, t.body_start.ptr,
                                                                      t.body_count.ptr, perm, key_in);
    note_launch();
    k_iota<<<blocks_for(n), kThreads, 0, st>>>(sc.vals_a.ptr, n);
    int bits = 1;
    while ((1ll << bits) <= n) ++bits;
    size_t tmp_bytes = 0;
    cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, key_in, key_out, sc.vals_a.ptr, t.sort_index.ptr, (int)n, 0,
                                    bits, st);
    sc.cub.grow(tmp_bytes);
    FMM_CUDA_TRY(cub::DeviceRadixSort::SortPairs(sc.cub.ptr, tmp_bytes, key_in, key_out, sc.vals_a.ptr,
                                                 t.sort_index.ptr, (int)n, 0, bits, st));
    note_launch();
    k_permute<<<blocks_for(n), kThreads, 0, st>>>(sc.alt_pos.ptr, sc.alt_str.ptr, t.sort_index.ptr, n, t.pos.ptr,
                                                  t.str.ptr);
    if (shrink) {
      note_launch();
      k_leaf_bodies<32, false><<<(int)((nleaves * 32ll + 127) / 128), 128, 0, st>>>(
          B, nleaves, perm, nullptr, nullptr, t.sort_index.ptr, t.pos.ptr, t.str.ptr, 1, geo);
    }
  }
  FMM_CUDA_TRY(cudaGetLastError());
}

void branch_max_influence(DevTree& t, const double* gnorm_orig, cudaStream_t st) {
  int nl = (int)t.n_leaves;
  note_launch();
  k_leaf_maxinf<<<(int)((nl * 32ll + 255) / 256), 256, 0, st>>>(t.leaf_index.ptr, nl, t.body_start.ptr,
                                                                t.body_count.ptr, t.parent.ptr, t.sort_index.ptr,
                                                                gnorm_orig, t.max_influence.ptr);
  FMM_CUDA_TRY(cudaGetLastError());
}

}  // namespace fmmb
