// lists.cu -- dual-tree traversal in HBM (replaces src/interaction_list.jl:3-213).
//
// The reference recurses from (root, root) and, per (target, source) branch
// pair, either records a P2P pair, records an M2L pair (multipole acceptance
// criterion d^2 * mac^2 > (r_s + r_t)^2) or descends into the children of one
// side, with three rule sets (Barba, SelfTuning, SelfTuningTreeStop).  Here the
// same per-pair decision runs on a breadth-first frontier of pairs, one kernel
// per step with no host round trip in between: a pair at step k has depth(t) +
// depth(s) = k, so (levels of the target tree + levels of the source tree - 1)
// steps exhaust the recursion.  Outputs and the next frontier take their slots
// with warp-aggregated atomics, and the pairs of every target are counted.  The
// decisions are the reference's, with the same FP64 operations (-fmad=false), so
// the pair sets are identical.  A scan of the per-target counts, a scatter into
// the target rows and a segmented sort of every row give the target-sorted lists
// of sort_by_target (src/interaction_list.jl:183-213) with a canonical order inside
// each target (the reference's is depth-first): by source index, or, for the M2L
// rows of an error-controlled solve, by decreasing (r_s + r_t) / separation and then
// source index, so that the pairs of one lane-per-pair pass stop at similar orders.
// The result does not depend on the order in which the atomics were served.
// Both lists go through each stage in one launch, and the host synchronises once per build:
// after the row compaction (totals, capacity check, row counts).
#include <climits>
#include <cstring>

#include <cub/cub.cuh>
#include <cub/block/block_merge_sort.cuh>
#include <cub/warp/warp_merge_sort.cuh>

#include "context.cuh"

namespace fmmb {

namespace {

enum : int { A_NONE = 0, A_DIRECT = 1, A_M2L = 2, A_SPLIT_T = 3, A_SPLIT_S = 4 };

// per branch of one tree in its role: centre and radius (target ones for the target
// tree, source ones for the source tree), and (n_children, child_start, body_count)
struct TreeRef {
  const double4* geo;
  const int4* info;
};

struct Rule {
  double mac;
  int64_t ls;  // source leaf size (SelfTuning)
  int method;
  bool ff, nf, si;
};

__device__ __forceinline__ bool mac_accept(const double4& tg, const double4& sg, double mac) {
  double dx = tg.x - sg.x;
  double dy = tg.y - sg.y;
  double dz = tg.z - sg.z;
  double sep2 = dx * dx + dy * dy + dz * dz;
  double summed = sg.w + tg.w;
  return sep2 * mac * mac > summed * summed;
}

// one step of build_interaction_lists! for the three rule sets
// (src/interaction_list.jl:23-64, 66-120, 122-166); for a split, n_next children
// starting at child0 (of the target for A_SPLIT_T, of the source for A_SPLIT_S); pairs: the body pairs
__device__ int decide(const TreeRef& T, int t, const TreeRef& S, int s, const Rule& R, int& n_next, int& child0,
                      unsigned long long& pairs) {
  n_next = 0;
  child0 = 0;
  const int4 ti = T.info[t], si = S.info[s];
  const int nct = ti.x, ncs = si.x;
  const int bt = ti.z, bs = si.z;
  pairs = (unsigned long long)bt * (unsigned)bs;
  bool both_leaves = (nct == 0) && (ncs == 0);
  bool dir_ok = (R.nf || (t == s && R.si)) && (t != s || R.si);
  if (R.method == FMM_LIST_BARBA) {
    const double4 tg = T.geo[t], sg = S.geo[s];
    if (mac_accept(tg, sg, R.mac)) return R.ff ? A_M2L : A_NONE;
    if (both_leaves) return dir_ok ? A_DIRECT : A_NONE;
    // target radius decides the side (src/interaction_list.jl:48)
    if (ncs == 0 || (tg.w >= sg.w && nct != 0)) {
      n_next = nct;
      child0 = ti.y;
      return A_SPLIT_T;
    }
    n_next = ncs;
    child0 = si.y;
    return A_SPLIT_S;
  }
  if (R.method == FMM_LIST_SELF_TUNING) {
    double fraction = 0.0;
    fraction = fraction + (double)bs / (double)(R.ls * R.ls);
    fraction = fraction * (double)bt;
    if (fraction < 1.0 || both_leaves) return (R.nf && (t != s || R.si)) ? A_DIRECT : A_NONE;
    if (mac_accept(T.geo[t], S.geo[s], R.mac)) return R.ff ? A_M2L : A_NONE;
  } else {  // SelfTuningTreeStop
    if (both_leaves) return dir_ok ? A_DIRECT : A_NONE;
    if (mac_accept(T.geo[t], S.geo[s], R.mac)) return R.ff ? A_M2L : A_NONE;
  }
  if (ncs == 0 || (bt >= bs && nct != 0)) {
    n_next = nct;
    child0 = ti.y;
    return A_SPLIT_T;
  }
  n_next = ncs;
  child0 = si.y;
  return A_SPLIT_S;
}

// branch records of one tree in one role, and (front given) the root pair of a traversal
struct NodeIn {
  int n;
  const double *center, *radius;
  const int *n_children, *child_start, *body_count;
  double4* geo;
  int4* info;
};
__global__ void k_pack_nodes(NodeIn T, NodeIn S, int2* front, int* ctr) {
  const NodeIn& a = blockIdx.y ? S : T;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n; i += gridDim.x * blockDim.x) {
    a.geo[i] = make_double4(a.center[3 * i], a.center[3 * i + 1], a.center[3 * i + 2], a.radius[i]);
    a.info[i] = make_int4(a.n_children[i], a.child_start[i], a.body_count[i], 0);
  }
  if (front && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) {
    front[0] = make_int2(0, 0);
    ctr[0] = 1;
  }
}

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxSteps = 64;  // frontier counters; a traversal takes levels_t + levels_s - 1 steps
enum : int {
  C_DIR = kMaxSteps,
  C_M2L,
  C_FLAG,
  C_ROWS_DIR,
  C_ROWS_M2L = C_ROWS_DIR + 8,
  C_PAIRS = C_ROWS_M2L + 9,
  C_N = 128
};
static_assert(C_PAIRS % 2 == 0, "the body pairs of the direct list are a 64-bit counter");
constexpr int kStepThreads = 128;
constexpr int kStepMinBlocks = 9;  // per SM, 56 registers (62 left alone: 150,001 bodies 459 -> 442 us)
constexpr int kStepMaxBlocks = 148 * 16;

// Add one to cnt[t] for the lanes that pass, one atomic per distinct target of the warp.
__device__ __forceinline__ void count_targets(bool on, int t, int lane, int* __restrict__ cnt) {
  const unsigned grp = __match_any_sync(kFull, on ? t : -1 - lane);
  if (on && lane == __ffs(grp) - 1) atomicAdd(cnt + t, __popc(grp));
}

constexpr int kStepItems = 4;                              // pairs per thread and chunk (most)
constexpr int kStepChunk = kStepThreads * kStepItems;      // pairs per block and chunk (most)

// Step k of the traversal: every pair of the frontier (ctr[k] pairs) is decided;
// direct and M2L pairs go to the raw lists and count for their target, split
// pairs put their children into the next frontier (ctr[k + 1] pairs).  A block
// takes the slots of a whole chunk with one atomic per counter.  Slots past a
// capacity are not written and raise the flag, which stops the later steps (the
// host grows the buffers and repeats).
__global__ void __launch_bounds__(kStepThreads, kStepMinBlocks)
    k_step(const int2* __restrict__ fin, int2* __restrict__ fout, int k, TreeRef T, TreeRef S, Rule R,
           int2* __restrict__ rdir, int2* __restrict__ rm2l, int* __restrict__ cdir, int* __restrict__ cm2l,
           int* __restrict__ ctr, int cap_f, int cap_d, int cap_m) {
  constexpr int NW = kStepThreads / 32;
  __shared__ int wsum[3][NW];
  __shared__ int bbase[3];
  __shared__ int stop;
  __shared__ unsigned long long bpairs;
  // after an overflow the frontier holds unwritten slots: the steps that follow do
  // nothing, and the host grows the buffers and repeats the traversal.  Another block
  // of this step may raise the flag meanwhile, so one thread reads it for the block:
  // the block leaves or stays as a whole (its barriers and block sums need every warp)
  if (threadIdx.x == 0) stop = *reinterpret_cast<volatile int*>(ctr + C_FLAG), bpairs = 0;
  __syncthreads();
  if (stop) return;
  const int n = min(ctr[k], cap_f);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  bool bad = false;
  // a frontier that the launch's threads cover takes one pair per thread
  const int items = n > (int)gridDim.x * kStepThreads ? kStepItems : 1, chunk = items * kStepThreads;
  for (int c0 = blockIdx.x * chunk; c0 < n; c0 += gridDim.x * chunk) {
    int2 p[kStepItems];
    int a[kStepItems], nn[kStepItems], ch[kStepItems];
    int cd = 0, cm = 0, cf = 0;
    unsigned long long pairs = 0;  // body pairs of this thread's direct pairs
#pragma unroll
    for (int r = 0; r < kStepItems; ++r) {
      const int i = c0 + r * kStepThreads + threadIdx.x;
      p[r] = make_int2(0, 0);
      a[r] = A_NONE;
      nn[r] = 0;
      ch[r] = 0;
      if (r < items && i < n) {
        p[r] = fin[i];
        unsigned long long v;
        a[r] = decide(T, p[r].x, S, p[r].y, R, nn[r], ch[r], v);
        if (a[r] == A_DIRECT) pairs += v;
      }
      if (a[r] != A_SPLIT_T && a[r] != A_SPLIT_S) nn[r] = 0;
      cd += a[r] == A_DIRECT;
      cm += a[r] == A_M2L;
      cf += nn[r];
    }
    // block exclusive scan of (cd, cm, cf)
    int id = cd, im = cm, jf = cf;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(kFull, id, o), y = __shfl_up_sync(kFull, im, o), z = __shfl_up_sync(kFull, jf, o);
      if (lane >= o) id += x, im += y, jf += z;
    }
    if (lane == 31) wsum[0][w] = id, wsum[1][w] = im, wsum[2][w] = jf;
    __syncthreads();
    if (threadIdx.x < 3) {
      int tot = 0;
      for (int q = 0; q < NW; ++q) tot += wsum[threadIdx.x][q];
      const int slot = threadIdx.x == 0 ? C_DIR : threadIdx.x == 1 ? C_M2L : k + 1;
      bbase[threadIdx.x] = tot ? atomicAdd(ctr + slot, tot) : 0;
    }
    __syncthreads();
    int od = bbase[0] + id - cd, om = bbase[1] + im - cm, of = bbase[2] + jf - cf;
    for (int q = 0; q < w; ++q) od += wsum[0][q], om += wsum[1][q], of += wsum[2][q];
#pragma unroll
    for (int r = 0; r < kStepItems; ++r) {
      if (a[r] == A_DIRECT) {
        if (od < cap_d)
          rdir[od] = p[r];
        else
          bad = true;
        ++od;
      } else if (a[r] == A_M2L) {
        if (om < cap_m)
          rm2l[om] = p[r];
        else
          bad = true;
        ++om;
      } else if (nn[r]) {
        if (of + nn[r] > cap_f) {
          bad = true;
        } else if (a[r] == A_SPLIT_T) {
          for (int c = 0; c < nn[r]; ++c) fout[of + c] = make_int2(ch[r] + c, p[r].y);
        } else {
          for (int c = 0; c < nn[r]; ++c) fout[of + c] = make_int2(p[r].x, ch[r] + c);
        }
        of += nn[r];
      }
      if (r < items) {
        count_targets(a[r] == A_DIRECT, p[r].x, lane, cdir);
        count_targets(a[r] == A_M2L, p[r].x, lane, cm2l);
      }
    }
    if (__any_sync(kFull, cd > 0)) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) pairs += __shfl_xor_sync(kFull, pairs, o);
      if (lane == 0) atomicAdd(&bpairs, pairs);
    }
    __syncthreads();  // wsum / bbase are rewritten by the next chunk, bpairs is complete
  }
  if (bad) atomicOr(ctr + C_FLAG, 1);
  // one addition per block to the launch's counter
  if (threadIdx.x == 0 && bpairs) atomicAdd(reinterpret_cast<unsigned long long*>(ctr + C_PAIRS), bpairs);
}

// per target: (count << 32) | (count > 0), so that one exclusive scan gives both the
// row offset (high word) and the row ordinal among the non-empty targets (low word); the
// direct and the M2L counts one after the other, n + 1 entries each (the last one 0)
__global__ void k_pack_counts(const int* __restrict__ cnt, int n, unsigned long long* __restrict__ pk) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int c = cnt[t];
    pk[t] = ((unsigned long long)(unsigned)c << 32) | (c > 0 ? 1ull : 0ull);
  }
}

constexpr int kSmallRow = 256;  // rows up to this length: one warp each (merge sort in registers)
constexpr int kMidRow = 4096;   // up to this length: one block each; longer: segmented radix sort
constexpr int kMidClasses = 4;  // block sorts of 512, 1024, 2048 and 4096 keys
constexpr int kLongestSlot = 2 + kMidClasses;
static_assert(C_ROWS_DIR + kLongestSlot < C_ROWS_M2L, "counters of a list");

__host__ __device__ constexpr int mid_class(int c) { return c <= 512 ? 0 : c <= 1024 ? 1 : c <= 2048 ? 2 : 3; }

// one list (direct or M2L) on its way into target rows
struct Rows {
  const int* cnt;        // pairs per target
  const int2* raw;       // pairs in arrival order
  int n;                 // pairs
  int *off, *tgt, *roff; // offsets of all targets, the CSR of the non-empty ones
  int* ctr;              // rows, rows per block class, big rows, longest row
  int *mid, *big_b, *big_e, *big_r;  // rows per block class (n_targets + 1 each), longer rows
  int *cursor, *tmp;     // slots taken per target, rows before their sort
  int *out_t, *out_s;
  const double4 *tgeo, *sgeo;  // non-null: rows up to kMidRow ordered by separation (RowKey)
};
struct RowsPair {
  Rows l[2];
};

// offsets of all targets (off, n + 1), the CSR of the non-empty ones (tgt, roff),
// and the rows too long for a warp sort: row ordinals per block class (mid, n + 1
// per class) and the bounds of the longer rows (big).  blockIdx.y: the list.
__global__ void k_rows(RowsPair P, const unsigned long long* __restrict__ scan, int n) {
  const Rows& L = P.l[blockIdx.y];
  const unsigned long long* ex = scan + (size_t)blockIdx.y * (n + 1);
  const unsigned long long base = ex[0];
  int longest = 0;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t <= n; t += gridDim.x * blockDim.x) {
    const unsigned long long e = ex[t] - base;
    const int o = (int)(e >> 32), r = (int)(e & 0xffffffffu);
    L.off[t] = o;
    if (t < n) {
      L.cursor[t] = 0;
      const int c = L.cnt[t];
      longest = max(longest, c);
      if (c > 0) {
        L.tgt[r] = t;
        L.roff[r] = o;
      }
      if (c > kMidRow) {
        const int q = atomicAdd(L.ctr + 1 + kMidClasses, 1);
        L.big_b[q] = o;
        L.big_e[q] = o + c;
        L.big_r[q] = r;
      } else if (c > kSmallRow) {
        const int k = mid_class(c);
        L.mid[(size_t)k * (n + 1) + atomicAdd(L.ctr + 1 + k, 1)] = r;
      }
    } else {
      L.roff[r] = o;
      L.ctr[0] = r;
    }
  }
  longest = __reduce_max_sync(kFull, longest);
  if ((threadIdx.x & 31) == 0 && longest > 0) atomicMax(L.ctr + kLongestSlot, longest);
}

// raw pairs into their target's row, sources only (order inside a row fixed by the
// sort that follows); one cursor atomic per distinct target of a warp
__global__ void k_scatter(RowsPair P) {
  const Rows& L = P.l[blockIdx.y];
  const int lane = threadIdx.x & 31;
  for (int w0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); w0 < L.n; w0 += gridDim.x * blockDim.x) {
    const int i = w0 + lane;
    const bool on = i < L.n;
    const int2 p = on ? L.raw[i] : make_int2(-1 - lane, 0);
    const unsigned grp = __match_any_sync(kFull, p.x);
    const int leader = __ffs(grp) - 1;
    int b = 0;
    if (on && lane == leader) b = atomicAdd(L.cursor + p.x, __popc(grp));
    b = __shfl_sync(kFull, b, leader);
    if (on) L.tmp[L.off[p.x] + b + __popc(grp & ((1u << lane) - 1u))] = p.y;
  }
}

struct KeyLess {
  __device__ __forceinline__ bool operator()(unsigned a, unsigned b) const { return a < b; }
};

// Sort key of a row entry: its source index, or, for M2L rows ordered by separation,
// (4095 - q) << 20 | source with q = floor(4095 (r_s + r_t) / |c_t - c_s|) clamped to
// [0, 4095]: the pairs of one target that need high expansion orders come first and
// neighbouring pairs need similar orders (source indices < 2^20 on that path).
constexpr int kSepShift = 20;
struct RowKey {
  const double4* sgeo;  // null: source order
  double4 tg;
  __device__ __forceinline__ unsigned enc(int s) const {
    if (!sgeo) return (unsigned)s;
    const double4 sg = sgeo[s];
    const double dx = tg.x - sg.x, dy = tg.y - sg.y, dz = tg.z - sg.z;
    const double rho = (sg.w + tg.w) / sqrt(dx * dx + dy * dy + dz * dz);
    const int q = (int)fmin(4095.0, fmax(0.0, rho * 4095.0));
    return ((unsigned)(4095 - q) << kSepShift) | (unsigned)s;
  }
  __device__ __forceinline__ int dec(unsigned k) const {
    return sgeo ? (int)(k & ((1u << kSepShift) - 1u)) : (int)k;
  }
};
__device__ __forceinline__ RowKey row_key(const double4* tgeo, const double4* sgeo, int t) {
  RowKey k;
  k.sgeo = sgeo;
  k.tg = sgeo ? tgeo[t] : make_double4(0, 0, 0, 0);
  return k;
}

constexpr int kSortWarps = 8;

// one row of up to 32 ITEMS entries, sorted by a warp
template <int ITEMS, class Temp>
__device__ __forceinline__ void sort_row_warp(Temp& tmp, const Rows& L, int b, int len, int t, int lane) {
  using WMS = cub::WarpMergeSort<unsigned, ITEMS, 32>;
  WMS ws(reinterpret_cast<typename WMS::TempStorage&>(tmp));
  const RowKey rk = row_key(L.tgeo, L.sgeo, t);
  unsigned keys[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = lane * ITEMS + j;
    keys[j] = i < len ? rk.enc(L.tmp[b + i]) : UINT_MAX;
  }
  ws.Sort(keys, KeyLess(), len, UINT_MAX);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = lane * ITEMS + j;
    if (i < len) L.out_t[b + i] = t, L.out_s[b + i] = rk.dec(keys[j]);
  }
  __syncwarp();
}

// rows of up to kSmallRow entries: one warp each.  blockIdx.y: the list
__global__ void __launch_bounds__(kSortWarps * 32) k_sort_warp(RowsPair P) {
  using Temp = typename cub::WarpMergeSort<unsigned, 8, 32>::TempStorage;
  __shared__ Temp tmp[kSortWarps];
  const Rows& L = P.l[blockIdx.y];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n_rows = L.ctr[0];
  for (int r = blockIdx.x * kSortWarps + w; r < n_rows; r += gridDim.x * kSortWarps) {
    const int b = L.roff[r], len = L.roff[r + 1] - b;
    if (len > kSmallRow) continue;
    const int t = L.tgt[r];
    if (len == 1) {
      if (lane == 0) L.out_t[b] = t, L.out_s[b] = L.tmp[b];
    } else if (len <= 32) {
      sort_row_warp<1>(tmp[w], L, b, len, t, lane);
    } else if (len <= 64) {
      sort_row_warp<2>(tmp[w], L, b, len, t, lane);
    } else if (len <= 128) {
      sort_row_warp<4>(tmp[w], L, b, len, t, lane);
    } else {
      sort_row_warp<8>(tmp[w], L, b, len, t, lane);
    }
  }
}

// rows of one block class: one block of THREADS x ITEMS keys per row (n0 rows of the first
// list, the others of the second)
template <int THREADS, int ITEMS>
__global__ void __launch_bounds__(THREADS) k_sort_block(RowsPair P, size_t mid0, int n0) {
  using BMS = cub::BlockMergeSort<unsigned, THREADS, ITEMS>;
  __shared__ typename BMS::TempStorage tmp;
  const int q = (int)blockIdx.x < n0 ? 0 : 1;
  const Rows& L = P.l[q];
  const int r = L.mid[mid0 + blockIdx.x - (q ? n0 : 0)];
  const int b = L.roff[r], len = L.roff[r + 1] - b, t = L.tgt[r];
  const RowKey rk = row_key(L.tgeo, L.sgeo, t);
  unsigned keys[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = threadIdx.x * ITEMS + j;
    keys[j] = i < len ? rk.enc(L.tmp[b + i]) : UINT_MAX;
  }
  BMS(tmp).Sort(keys, KeyLess(), len, UINT_MAX);
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = threadIdx.x * ITEMS + j;
    if (i < len) L.out_t[b + i] = t, L.out_s[b + i] = rk.dec(keys[j]);
  }
}

// target column of the rows sorted by the segmented radix sort
__global__ void k_fill_rows(const int* __restrict__ big_r, const int* __restrict__ tgt, const int* __restrict__ roff,
                            int* __restrict__ out_t) {
  const int r = big_r[blockIdx.x];
  const int b = roff[r], e = roff[r + 1], t = tgt[r];
  for (int i = b + threadIdx.x; i < e; i += blockDim.x) out_t[i] = t;
}

int blocks_for(int64_t n, int threads) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, kStepMaxBlocks));
}

// rows sorted, both lists in one launch per kind of row (h0, h1: the lists' counters)
template <int THREADS, int ITEMS>
void sort_block_class(const RowsPair& P, int k, size_t stride, const int* h0, const int* h1, cudaStream_t st) {
  const int n0 = h0[1 + k], n1 = h1[1 + k];
  if (n0 + n1 == 0) return;
  note_launch();
  k_sort_block<THREADS, ITEMS><<<n0 + n1, THREADS, 0, st>>>(P, (size_t)k * stride, n0);
  FMM_CUDA_TRY(cudaGetLastError());
}

void sort_rows(const RowsPair& P, int nt, const int* h0, const int* h1, int nbits, Scratch& sc, cudaStream_t st) {
  const int n = std::max(P.l[0].n, P.l[1].n), rows = std::max(h0[0], h1[0]);
  if (n == 0) return;
  note_launch();
  k_scatter<<<dim3(blocks_for(n, 256), 2), 256, 0, st>>>(P);
  note_launch();
  k_sort_warp<<<dim3(blocks_for((int64_t)rows * 32, kSortWarps * 32), 2), kSortWarps * 32, 0, st>>>(P);
  FMM_CUDA_TRY(cudaGetLastError());
  const size_t stride = (size_t)nt + 1;
  sort_block_class<128, 4>(P, 0, stride, h0, h1, st);
  sort_block_class<256, 4>(P, 1, stride, h0, h1, st);
  sort_block_class<256, 8>(P, 2, stride, h0, h1, st);
  sort_block_class<256, 16>(P, 3, stride, h0, h1, st);
  for (int q = 0; q < 2; ++q) {
    const Rows& L = P.l[q];
    const int n_big = (q ? h1 : h0)[1 + kMidClasses];
    if (n_big == 0) continue;
    size_t tb = 0;
    cub::DeviceSegmentedRadixSort::SortKeys(nullptr, tb, L.tmp, L.out_s, L.n, n_big, L.big_b, L.big_e, 0, nbits, st);
    sc.cub.grow(tb);
    FMM_CUDA_TRY(cub::DeviceSegmentedRadixSort::SortKeys(sc.cub.ptr, tb, L.tmp, L.out_s, L.n, n_big, L.big_b, L.big_e,
                                                         0, nbits, st));
    note_launch();
    k_fill_rows<<<n_big, 256, 0, st>>>(L.big_r, L.tgt, L.roff, L.out_t);
    FMM_CUDA_TRY(cudaGetLastError());
  }
}

NodeIn target_nodes(const DevTree& t, Scratch& sc) {
  return NodeIn{(int)t.n_branches,  t.tcenter.ptr,    t.tradius.ptr,     t.n_children.ptr,
                t.child_start.ptr, t.body_count.ptr, sc.node_geo_t.ptr, sc.node_info_t.ptr};
}
NodeIn source_nodes(const DevTree& t, Scratch& sc) {
  return NodeIn{(int)t.n_branches,  t.scenter.ptr,    t.sradius.ptr,     t.n_children.ptr,
                t.child_start.ptr, t.body_count.ptr, sc.node_geo_s.ptr, sc.node_info_s.ptr};
}

}  // namespace

void build_lists(DevLists& L, const DevTree& tt, const DevTree& stt, Scratch& sc, cudaStream_t st,
                 int64_t leaf_size_source, double mac, bool ff, bool nf, bool si, int method,
                 bool m2l_by_separation) {
  const int nt = (int)tt.n_branches, ns = (int)stt.n_branches;
  sc.node_geo_t.grow((size_t)nt);
  sc.node_info_t.grow((size_t)nt);
  sc.node_geo_s.grow((size_t)ns);
  sc.node_info_s.grow((size_t)ns);
  TreeRef T{sc.node_geo_t.ptr, sc.node_info_t.ptr};
  TreeRef S{sc.node_geo_s.ptr, sc.node_info_s.ptr};
  Rule R{mac, leaf_size_source, method, ff, nf, si};
  const int n_steps = tt.n_levels + stt.n_levels - 1;
  FMM_CHECK(n_steps + 1 < kMaxSteps, FMM_ERR_TREE_DEPTH, "interaction-list traversal deeper than supported");
  // counters, then the pairs per target of the two lists (nt + 1 each): one buffer, cleared at once
  const size_t n1 = (size_t)nt + 1;
  sc.cnt_a.grow(C_N + 2 * n1);
  int* ctr = sc.cnt_a.ptr;
  int *cnt_d = ctr + C_N, *cnt_m = cnt_d + n1;
  sc.row_mid.grow(2 * (size_t)kMidClasses * n1);
  sc.row_big_b.grow(2 * n1);
  sc.row_big_e.grow(2 * n1);
  sc.row_big_r.grow(2 * n1);
  sc.row_cur.grow(2 * n1);
  sc.row_off_a.grow(n1);
  sc.row_off_b.grow(n1);
  L.dir_tgt.grow(n1);
  L.dir_off.grow(n1 + 1);
  L.m2l_tgt.grow(n1);
  L.m2l_off.grow(n1 + 1);
  sc.keys_a.grow(2 * n1);
  sc.keys_b.grow(2 * n1);
  // capacities: kept from earlier builds, grown when a traversal reports more
  size_t cap_f = std::max<size_t>(4096, (size_t)nt * 32), cap_d = std::max<size_t>(4096, (size_t)tt.n_leaves * 64);
  size_t cap_m = std::max<size_t>(4096, (size_t)nt * 96);
  std::vector<int> h(C_N, 0);
  RowsPair P;
  for (int attempt = 0;; ++attempt) {
    FMM_CHECK(attempt < 8, FMM_ERR_MEMORY, "interaction-list capacities did not converge");
    sc.front_a.grow(cap_f);
    sc.front_b.grow(cap_f);
    sc.dir_raw.grow(cap_d);
    sc.m2l_raw.grow(cap_m);
    const int cf = (int)std::min<size_t>(sc.front_a.cap, sc.front_b.cap);
    const int cd = (int)sc.dir_raw.cap, cm = (int)sc.m2l_raw.cap;
    FMM_CUDA_TRY(cudaMemsetAsync(ctr, 0, (C_N + 2 * n1) * sizeof(int), st));
    note_launch();
    k_pack_nodes<<<dim3(blocks_for(std::max(nt, ns), 256), 2), 256, 0, st>>>(target_nodes(tt, sc),
                                                                              source_nodes(stt, sc),
                                                                              sc.front_a.ptr, ctr);
    FMM_CUDA_TRY(cudaGetLastError());
    for (int k = 0; k < n_steps; ++k) {
      const int2* fin = (k & 1) ? sc.front_b.ptr : sc.front_a.ptr;
      int2* fout = (k & 1) ? sc.front_a.ptr : sc.front_b.ptr;
      // grid from this scratch's previous build (the kernel strides over any frontier)
      const int64_t hint = k < (int)sc.step_hint.size() ? sc.step_hint[k] : (int64_t)kStepChunk * kStepMaxBlocks;
      note_launch();
      k_step<<<blocks_for(hint + hint / 4 + 32, kStepThreads), kStepThreads, 0, st>>>(
          fin, fout, k, T, S, R, sc.dir_raw.ptr, sc.m2l_raw.ptr, cnt_d, cnt_m, ctr, cf, cd, cm);
      FMM_CUDA_TRY(cudaGetLastError());
    }
    // row offsets of both lists (of partial counts after an overflow, which are then not used)
    note_launch();
    k_pack_counts<<<blocks_for(2 * (int64_t)n1, 256), 256, 0, st>>>(cnt_d, (int)(2 * n1), sc.keys_a.ptr);
    size_t tb = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tb, sc.keys_a.ptr, sc.keys_b.ptr, (int)(2 * n1), st);
    sc.cub.grow(tb);
    FMM_CUDA_TRY(cub::DeviceScan::ExclusiveSum(sc.cub.ptr, tb, sc.keys_a.ptr, sc.keys_b.ptr, (int)(2 * n1), st));
    auto rows = [&](int q, int* cnt, const int2* raw, int* off, int* tgt, int* roff, int slot) {
      Rows& r = P.l[q];
      r.cnt = cnt;
      r.raw = raw;
      r.n = 0;
      r.off = off;
      r.tgt = tgt;
      r.roff = roff;
      r.ctr = ctr + slot;
      r.mid = sc.row_mid.ptr + q * kMidClasses * n1;
      r.big_b = sc.row_big_b.ptr + q * n1;
      r.big_e = sc.row_big_e.ptr + q * n1;
      r.big_r = sc.row_big_r.ptr + q * n1;
      r.cursor = sc.row_cur.ptr + q * n1;
      r.tmp = r.out_t = r.out_s = nullptr;
      r.tgeo = r.sgeo = nullptr;
    };
    rows(0, cnt_d, sc.dir_raw.ptr, sc.row_off_a.ptr, L.dir_tgt.ptr, L.dir_off.ptr, C_ROWS_DIR);
    rows(1, cnt_m, sc.m2l_raw.ptr, sc.row_off_b.ptr, L.m2l_tgt.ptr, L.m2l_off.ptr, C_ROWS_M2L);
    note_launch();
    k_rows<<<dim3(blocks_for((int64_t)n1, 256), 2), 256, 0, st>>>(P, sc.keys_b.ptr, nt);
    FMM_CUDA_TRY(cudaGetLastError());
    FMM_CUDA_TRY(cudaMemcpyAsync(h.data(), ctr, C_N * sizeof(int), cudaMemcpyDeviceToHost, st));
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
    size_t max_f = 0;
    for (int k = 0; k <= n_steps; ++k) max_f = std::max(max_f, (size_t)(unsigned)h[k]);
    const size_t nd = (size_t)(unsigned)h[C_DIR], nm = (size_t)(unsigned)h[C_M2L];
    if (h[C_FLAG] || max_f > (size_t)cf || nd > (size_t)cd || nm > (size_t)cm) {
      // the counts after an overflow are partial: grow past them and at least double
      cap_f = std::max(2 * (size_t)cf, max_f + max_f / 4 + 64);
      cap_d = std::max(nd > (size_t)cd ? 2 * (size_t)cd : (size_t)cd, nd + nd / 4 + 64);
      cap_m = std::max(nm > (size_t)cm ? 2 * (size_t)cm : (size_t)cm, nm + nm / 4 + 64);
      continue;
    }
    FMM_CHECK(h[n_steps] == 0, FMM_ERR_TREE_DEPTH, "interaction-list traversal did not terminate");
    sc.step_hint.assign(h.begin(), h.begin() + n_steps);
    break;
  }
  const int n_dir = h[C_DIR], n_m2l = h[C_M2L];
  int nbits = 1;
  while ((1ll << nbits) <= stt.n_branches) ++nbits;
  L.dir_t.grow((size_t)n_dir + 1);
  L.dir_s.grow((size_t)n_dir + 1);
  L.m2l_t.grow((size_t)n_m2l + 1);
  L.m2l_s.grow((size_t)n_m2l + 1);
  sc.row_tmp_a.grow((size_t)n_dir + 1);
  sc.row_tmp_b.grow((size_t)n_m2l + 1);
  P.l[0].n = n_dir;
  P.l[0].tmp = sc.row_tmp_a.ptr;
  P.l[0].out_t = L.dir_t.ptr;
  P.l[0].out_s = L.dir_s.ptr;
  P.l[1].n = n_m2l;
  P.l[1].tmp = sc.row_tmp_b.ptr;
  P.l[1].out_t = L.m2l_t.ptr;
  P.l[1].out_s = L.m2l_s.ptr;
  if (m2l_by_separation && ns < (1 << kSepShift)) {
    P.l[1].tgeo = sc.node_geo_t.ptr;
    P.l[1].sgeo = sc.node_geo_s.ptr;
  }
  const int *h_d = h.data() + C_ROWS_DIR, *h_m = h.data() + C_ROWS_M2L;
  sort_rows(P, nt, h_d, h_m, nbits, sc, st);
  const int rows[2] = {h_d[0], h_m[0]};
  L.n_direct = n_dir;
  L.n_m2l = n_m2l;
  std::memcpy(&L.n_pairs, h.data() + C_PAIRS, sizeof(L.n_pairs));
  L.n_source_bodies = stt.n_bodies;
  L.n_dir_targets = rows[0];
  L.n_m2l_targets = rows[1];
  L.m2l_longest = h_m[kLongestSlot];
  L.rule_method = method;
}

namespace {

// The reference's recursion reaches the pairs of one target in the depth-first order of their
// sources: the paths of (t, s1) and (t, s2) from (root, root) are the same, split by split, up to
// the pair that splits the lowest common ancestor of s1 and s2 on the source side, where the
// children are taken in order.  The sources of a row are disjoint, so that order is the order of
// their first bodies: rows are sorted by (first body, source).
struct ExportRows {
  const int *tgt, *off, *src, *first_body;
  int2* out;
};
using ExportKey = unsigned long long;
__device__ __forceinline__ ExportKey export_key(const ExportRows& E, int i) {
  const int s = E.src[i];
  return ((ExportKey)(unsigned)E.first_body[s] << 32) | (unsigned)s;
}
struct ExportLess {
  __device__ __forceinline__ bool operator()(ExportKey a, ExportKey b) const { return a < b; }
};
constexpr int kExportRow = 4096;  // longest row of the block sort

// rows of up to 128 entries: a warp each
__global__ void __launch_bounds__(kSortWarps * 32) k_export_warp(ExportRows E, int rows) {
  using WMS = cub::WarpMergeSort<ExportKey, 4, 32>;
  __shared__ typename WMS::TempStorage tmp[kSortWarps];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int r = blockIdx.x * kSortWarps + w; r < rows; r += gridDim.x * kSortWarps) {
    const int b = E.off[r], len = E.off[r + 1] - b, t = E.tgt[r];
    if (len > 128) continue;
    ExportKey k[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) k[j] = lane * 4 + j < len ? export_key(E, b + lane * 4 + j) : ~0ull;
    WMS(tmp[w]).Sort(k, ExportLess(), len, ~0ull);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (lane * 4 + j < len) E.out[b + lane * 4 + j] = make_int2(t, (int)(unsigned)k[j]);
    __syncwarp();
  }
}
// rows of more than LO and up to THREADS x ITEMS entries: a block each
template <int THREADS, int ITEMS, int LO>
__global__ void __launch_bounds__(THREADS) k_export_block(ExportRows E, int rows) {
  using BMS = cub::BlockMergeSort<ExportKey, THREADS, ITEMS>;
  __shared__ typename BMS::TempStorage tmp;
  for (int r = blockIdx.x; r < rows; r += gridDim.x) {
    const int b = E.off[r], len = E.off[r + 1] - b, t = E.tgt[r];
    if (len <= LO || len > THREADS * ITEMS) continue;
    ExportKey k[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int i = threadIdx.x * ITEMS + j;
      k[j] = i < len ? export_key(E, b + i) : ~0ull;
    }
    BMS(tmp).Sort(k, ExportLess(), len, ~0ull);
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int i = threadIdx.x * ITEMS + j;
      if (i < len) E.out[b + i] = make_int2(t, (int)(unsigned)k[j]);
    }
    __syncthreads();
  }
}
// longer rows: keys for a segmented sort, and its result as pairs (rows of up to kExportRow are done)
__global__ void k_export_keys(ExportRows E, int n, ExportKey* __restrict__ keys) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) keys[i] = export_key(E, i);
}
__global__ void k_export_long(ExportRows E, const ExportKey* __restrict__ keys) {
  const int r = blockIdx.x, b = E.off[r], e = E.off[r + 1], t = E.tgt[r];
  if (e - b <= kExportRow) return;
  for (int i = b + threadIdx.x; i < e; i += blockDim.x) E.out[i] = make_int2(t, (int)(unsigned)keys[i]);
}
// the longest row
__global__ void k_longest_row(const int* __restrict__ off, int rows, int* __restrict__ longest) {
  int m = 0;
  for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < rows; r += gridDim.x * blockDim.x)
    m = max(m, off[r + 1] - off[r]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(kFull, m, o));
  if ((threadIdx.x & 31) == 0) atomicMax(longest, m);
}

}  // namespace

void export_lists_reference_order(const DevLists& L, const DevTree& stt, Scratch& sc, cudaStream_t st, int32_t* m2l,
                                  int32_t* direct) {
  struct One {
    const DevBuf<int>*tgt, *s, *off;
    int64_t n, rows;
    int32_t* dst;
  } lists[2] = {{&L.m2l_tgt, &L.m2l_s, &L.m2l_off, L.n_m2l, L.n_m2l_targets, m2l},
                {&L.dir_tgt, &L.dir_s, &L.dir_off, L.n_direct, L.n_dir_targets, direct}};
  sc.flag.grow(2);
  FMM_CUDA_TRY(cudaMemsetAsync(sc.flag.ptr, 0, 2 * sizeof(int), st));
  for (int q = 0; q < 2; ++q) {
    if (!lists[q].dst || lists[q].n == 0) continue;
    note_launch();
    k_longest_row<<<blocks_for(lists[q].rows, 256), 256, 0, st>>>(lists[q].off->ptr, (int)lists[q].rows,
                                                                  sc.flag.ptr + q);
  }
  int longest[2] = {0, 0};
  FMM_CUDA_TRY(cudaMemcpyAsync(longest, sc.flag.ptr, sizeof(longest), cudaMemcpyDeviceToHost, st));
  FMM_CUDA_TRY(cudaStreamSynchronize(st));
  for (int k = 0; k < 2; ++k) {
    const One& q = lists[k];
    if (!q.dst || q.n == 0) continue;
    const int n = (int)q.n, rows = (int)q.rows;
    sc.front_a.grow((size_t)n);
    const ExportRows E{q.tgt->ptr, q.off->ptr, q.s->ptr, stt.body_start.ptr, sc.front_a.ptr};
    note_launch();
    k_export_warp<<<blocks_for((int64_t)rows * 32, kSortWarps * 32), kSortWarps * 32, 0, st>>>(E, rows);
    if (longest[k] > 128) {
      note_launch();
      k_export_block<128, 4, 128><<<std::min(rows, kStepMaxBlocks), 128, 0, st>>>(E, rows);
    }
    if (longest[k] > 512) {
      note_launch();
      k_export_block<256, 16, 512><<<std::min(rows, kStepMaxBlocks), 256, 0, st>>>(E, rows);
    }
    FMM_CUDA_TRY(cudaGetLastError());
    if (longest[k] > kExportRow) {
      sc.keys_a.grow((size_t)n);
      sc.keys_b.grow((size_t)n);
      note_launch();
      k_export_keys<<<blocks_for(n, 256), 256, 0, st>>>(E, n, sc.keys_a.ptr);
      size_t tb = 0;
      FMM_CUDA_TRY(cub::DeviceSegmentedSort::SortKeys(nullptr, tb, sc.keys_a.ptr, sc.keys_b.ptr, n, rows, E.off,
                                                      E.off + 1, st));
      sc.cub.grow(tb);
      FMM_CUDA_TRY(cub::DeviceSegmentedSort::SortKeys(sc.cub.ptr, tb, sc.keys_a.ptr, sc.keys_b.ptr, n, rows, E.off,
                                                      E.off + 1, st));
      note_launch();
      k_export_long<<<rows, 256, 0, st>>>(E, sc.keys_b.ptr);
      FMM_CUDA_TRY(cudaGetLastError());
    }
    FMM_CUDA_TRY(cudaMemcpyAsync(q.dst, sc.front_a.ptr, (size_t)n * sizeof(int2), cudaMemcpyDeviceToHost, st));
    FMM_CUDA_TRY(cudaStreamSynchronize(st));
  }
}

}  // namespace fmmb
