// vecchia_grid.cu -- exact Vecchia ordering and neighbour sets on uniform grids, O(n log n) work instead of O(n^2).
//
// Definition (Kriging::make_vecchia_sets, src/lib/Kriging.cpp:736-804): the order starts at the point closest to the
// centroid and then repeatedly takes the point whose smallest squared distance to the points already ordered is
// largest (argmax ties to the lowest index); the neighbours of the point at position t are its min(m, t) nearest
// points among positions 0 .. t - 1, by (squared distance, index).  Squared distances are sums of (a_k - b_k)^2
// rounded term by term, as the reference's loop computes them (no fused multiply-add).
//
// Maxmin order.  The points are counting-sorted into the cells of a uniform grid.  When point p is taken with
// running distance r2 = mind2[p] (the current maximum), only points q with d2(q, p) < mind2[q] <= r2 change, so only
// the cells that intersect the cube of half-width sqrt(r2) around p are visited: a few cells per step once the
// ordering has covered the domain.  The argmax runs on a two-level 64-ary tournament tree in shared memory (level 1
// holds one (max, index) per 64 grid slots, level 2 one per 64 level-1 nodes) that is updated only where distances
// changed.  One CTA runs the steps; a launch runs a bounded number of them and rebuilds the tree from the distances it
// left behind.
//
// Steps are taken in rounds.  All points whose distance reaches a threshold tau (the current maximum times a ratio, so
// that there are at most 512 of them) are the round's candidates.  As long as the largest distance among them reaches
// tau, it is the global maximum, because no other point does and distances only fall: the candidates alone decide the
// next steps.  They are sorted by (distance, index), and all pairs are compared in FP32 with error bounds: taking one
// leaves another one alone, or brings it below tau (out of the round), or neither is sure.  One warp then takes the steps
// 32 candidates at a time from these bits; pairs that are not sure, or that come down to a distance that still reaches
// tau, go step by step with FP64 distances (146 of 32768 steps).  The other warps meanwhile update the neighbourhoods of
// the points taken, with atomic minima, and the tree follows.  A step alone costs 5.3 us, a chain of dependent loads and
// FP64 operations.  More candidates than 512 make the pairs dearer than the rounds they save (an argmax over up to 1024
// candidates and their distances to the point taken, step after step, cost 0.65 us a step).  An infinite
// maximum, and ties in more than 2048 nodes of the tree, fall back to a step alone.  Measured, n = 32768, d = 3: 172.6 ms by single steps,
// 29.5 ms with an argmax per step, 11.1 ms with the pairs: neighbourhoods 6 ms, then finding the candidates, sorting
// them, the pairs and the tree about 1 ms each.  Where more than 512 points share the maximum (lattices), a round takes
// those of the lowest indices: lattices of 32768 points 179 ms by single steps, 20 ms.
// The cell range of a query is computed
// with the same monotone floating-point map as the cells of the points, with a 1e-12 relative margin on the radius,
// so every point that can change lies in a visited cell.
//
// Neighbour sets.  For the points at positions t in (2^(j-1), 2^j] a grid over the first 2^j ordered points (about
// two per cell) holds at least half earlier points, so a ring-by-ring search around the query's cell finds the m
// nearest earlier points after O(m) visited points; it stops once the m-th best squared distance is below the
// squared distance to the next ring of cells (minus a margin for the cell rounding).  Positions t <= 2048 scan the
// earlier points directly.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdint>
#include <vector>

#include "common.cuh"
#include "stats.hpp"
#include "vecchia.hpp"

namespace lkg {

namespace {

constexpr unsigned FULL = 0xffffffffu;
constexpr int MAXD = 8;
constexpr int G1 = 64;                 // grid slots per level-1 node
constexpr int NG1_MAX = 8192;          // level-1 nodes in shared memory (n <= 2^19 at G1 = 64; larger n widens G1)
constexpr int NG2_MAX = 128;           // level-2 nodes (64 level-1 nodes each)
constexpr int LIST_MAX = 2048;         // dirty level-1 nodes tracked per step; more -> every node is rebuilt
constexpr int MM_THREADS = 1024;
constexpr int CAND_MAX = 512;          // candidates of a round
constexpr int CWORDS = CAND_MAX / 32;
constexpr int ROUND_FROM = 1;           // steps taken one by one before the first round
constexpr int QUEUE = 64;              // a warp's queue of distances to take in FP64
constexpr int KNN_BRUTE = 2048;        // positions up to this scan the earlier points directly
constexpr double RADIUS_MARGIN = 1e-12;

struct GridDesc {
  int d;
  int G[MAXD];          // cells per dimension
  long long stride[MAXD];
  double lo[MAXD], inv_h[MAXD];
  double h_min;         // smallest cell width
  double slack;         // absolute margin for the rounding of the cell map
};

__device__ __forceinline__ int cell_coord(const GridDesc& g, int k, double x) {
  const double f = (x - g.lo[k]) * g.inv_h[k];  // monotone in x: the same map for points and query bounds
  int c = (f >= 0.0) ? (int)fmin(f, 2.0e9) : 0;
  return c < 0 ? 0 : (c >= g.G[k] ? g.G[k] - 1 : c);
}

__device__ __forceinline__ double sqdist(const double* a, const double* b, int d) {
  double s = 0.0;
  for (int k = 0; k < d; ++k) {
    const double dk = __dsub_rn(a[k], b[k]);
    s = __dadd_rn(s, __dmul_rn(dk, dk));
  }
  return s;
}

// (value, index) pairs: larger value wins, ties to the lower index.  Values are running squared distances (>= 0,
// +inf before the first step, -inf once ordered); for these, the IEEE bit patterns read as signed 64-bit integers
// order exactly like the doubles, so the tree compares integers (FP64 throughput is scarce on this part).
__device__ __forceinline__ long long key_of(double v) { return __double_as_longlong(v); }
__device__ __forceinline__ bool beats(long long v, int i, long long bv, int bi) { return v > bv || (v == bv && i < bi); }

__device__ __forceinline__ void warp_argmax(long long& v, int& i) {
  for (int o = 16; o > 0; o >>= 1) {
    const long long ov = __shfl_xor_sync(FULL, v, o);
    const int oi = __shfl_xor_sync(FULL, i, o);
    if (beats(ov, oi, v, i)) {
      v = ov;
      i = oi;
    }
  }
}

// ------------------------------------------------------------------------------------------------ grid building
__global__ void k_grid_cells(int n, const double* __restrict__ P, int pstride_pts, GridDesc g, int* __restrict__ cell,
                             int* __restrict__ count) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  long long c = 0;
  for (int k = 0; k < g.d; ++k) c += (long long)cell_coord(g, k, P[(int64_t)i * pstride_pts + k]) * g.stride[k];
  cell[i] = (int)c;
  atomicAdd(&count[c], 1);
}

// exclusive scan of a[0 .. len) in place, one block, 1024 threads, len any size (sequential chunks)
__global__ void __launch_bounds__(1024) k_scan_exclusive(int len, int* __restrict__ a, int* __restrict__ total) {
  __shared__ int warp_sums[32];
  __shared__ int carry_s;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int base = 0; base < len; base += 1024) {
    const int i = base + threadIdx.x;
    const int v = i < len ? a[i] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(FULL, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[w] = x;
    __syncthreads();
    if (w == 0) {
      int s = warp_sums[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(FULL, s, o);
        if (lane >= o) s += y;
      }
      warp_sums[lane] = s;
    }
    __syncthreads();
    const int carry = carry_s;
    const int incl = x + (w > 0 ? warp_sums[w - 1] : 0) + carry;
    if (i < len) a[i] = incl - v;
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = incl;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry_s;
}

// slot of every point: cursor starts as a copy of cell_start
__global__ void k_grid_scatter(int n, const int* __restrict__ cell, int* __restrict__ cursor, int* __restrict__ perm) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  perm[atomicAdd(&cursor[cell[i]], 1)] = i;
}

// slot arrays of the maxmin grid: coordinates, original index, slot of every point, running distance = +inf
// (Xf: FP32 differences from the grid's lower corner)
__global__ void k_grid_slots(int n, int d, const double* __restrict__ Xp, const int* __restrict__ perm, GridDesc g,
                             double* __restrict__ Xs, float* __restrict__ Xf, int* __restrict__ orig,
                             int* __restrict__ slot_of, double* __restrict__ dist) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n) return;
  const int i = perm[s];
  for (int k = 0; k < d; ++k) {
    const double x = Xp[(int64_t)i * d + k];
    Xs[(int64_t)s * d + k] = x;
    Xf[(int64_t)s * d + k] = (float)(x - g.lo[k]);
  }
  orig[s] = i;
  slot_of[i] = s;
  dist[s] = INFINITY;
}

// ------------------------------------------------------------------------------------------------ maxmin steps
struct MaxminArgs {
  int n, d, t0, t1, first, g1;  // steps [t0, t1); t0 == 0 takes `first` with an infinite radius
  int singles;                  // steps below this position are taken one by one
  int ng1, ng2;
  GridDesc g;
  const int* cell_start;
  const double* Xs;
  const float* Xf;
  const int* orig;
  const int* slot_of;
  double* dist;  // read past L1 (rounds update it with atomics)
  int* order;
  int* err;                    // set when a wait gave up; the launches after it do nothing
  unsigned long long wait_ns;  // limit of a wait for a round's next step
  float eps_length;  // no less than the length of eps, from FP64: in FP32 its squares are zero for sides below 1e-16
  float eps[MAXD];  // bound on the error of a difference of two Xf in dimension k
};

// a float above the non-negative double with these bits (its 24 leading bits, plus one unit), by integer operations
__device__ __forceinline__ float f32_above(long long bits) {
  const int hi = (int)(bits >> 32), e = (hi >> 20) & 0x7FF;
  if (e <= 896) return 1.2e-38f;
  if (e >= 1150) return NAN;  // beyond FP32: no bound (every comparison with it fails)
  return __int_as_float((((e - 896) << 23) | ((hi & 0xFFFFF) << 3) | (int)((unsigned)bits >> 29)) + 1);
}

// the largest (key, lowest index) of a warp and the lane that holds it; -1 keys mean none (index INT_MAX)
__device__ __forceinline__ void redux_argmax(long long key, int idx, long long& mkey, int& midx, int& mlane) {
  const int hi = (int)(key >> 32), mh = __reduce_max_sync(FULL, hi);
  const unsigned lo = hi == mh ? (unsigned)key : 0u, ml = __reduce_max_sync(FULL, lo);
  const bool top = hi == mh && (unsigned)key == ml;
  midx = __reduce_min_sync(FULL, top ? idx : INT_MAX);
  mlane = __ffs(__ballot_sync(FULL, top && idx == midx)) - 1;
  mkey = ((long long)mh << 32) | ml;
}

// coordinates a candidate takes in shared memory: FP32, and FP64 up to d = 4 (for more there is no room)
__host__ __device__ constexpr int cand_stride(int d) { return d <= 4 ? 4 : 8; }
__host__ __device__ constexpr int cand_stride64(int d) { return d <= 4 ? 4 : 0; }

size_t maxmin_smem(int ng1, int d) {
  return sizeof(long long) * ng1 + sizeof(int) * ((ng1 + 1) & ~1) + (sizeof(long long) + sizeof(int)) * NG2_MAX +
         sizeof(unsigned) * (NG1_MAX / 32) + sizeof(int) * LIST_MAX + sizeof(int2) * QUEUE * (MM_THREADS / 32) +
         CAND_MAX * (sizeof(uint2) * CWORDS + sizeof(long long) + sizeof(double) * cand_stride64(d) + 3 * sizeof(int) +
                     (cand_stride(d) + 1) * sizeof(float));
}

template <int DM>  // d <= DM
__global__ void __launch_bounds__(MM_THREADS, 1) k_maxmin_grid(MaxminArgs a) {
  constexpr int DP = cand_stride(DM);
  extern __shared__ long long mm_smem[];
  long long* l1v = mm_smem;                                  // ng1 keys
  int* l1i = reinterpret_cast<int*>(l1v + a.ng1);            // ng1
  long long* l2v = reinterpret_cast<long long*>(l1i + ((a.ng1 + 1) & ~1));
  int* l2i = reinterpret_cast<int*>(l2v + NG2_MAX);          // 256
  unsigned* dirty1 = reinterpret_cast<unsigned*>(l2i + NG2_MAX);  // ng1 bits
  int* list1 = reinterpret_cast<int*>(dirty1 + NG1_MAX / 32);     // LIST_MAX
  int2* queue = reinterpret_cast<int2*>(list1 + LIST_MAX);  // QUEUE per warp: (slot, candidate taken)
  // a round's candidates (CAND_MAX each) by descending distance: FP64 key and coordinates, FP32 coordinates, conflicts
  // with the others (.x: a point that may fall when this one is taken, .y: that surely falls below the threshold)
  long long* skey = reinterpret_cast<long long*>(queue + QUEUE * (MM_THREADS / 32));
  double* cxd = reinterpret_cast<double*>(skey + CAND_MAX);
  float* cx = reinterpret_cast<float*>(cxd + cand_stride64(DM) * CAND_MAX);
  uint2* pairs = reinterpret_cast<uint2*>(cx + DP * CAND_MAX);
  float* cthr = reinterpret_cast<float*>(pairs + CWORDS * CAND_MAX);
  int* cslot = reinterpret_cast<int*>(cthr + CAND_MAX);
  int* cidx = cslot + CAND_MAX;
  int* taken = cidx + CAND_MAX;  // the candidates taken, in order
  // as they were found: where the conflicts go once they are sorted
  long long* ukey = reinterpret_cast<long long*>(pairs);
  int* uslot = reinterpret_cast<int*>(ukey + CAND_MAX);
  int* uidx = uslot + CAND_MAX;
  int* rank = uidx + CAND_MAX;
  __shared__ unsigned dirty2[NG2_MAX / 32];
  __shared__ int nlist1, overflow;
  // the step's scalars, computed by warp 0 and read by every warp: the point taken, its slot and coordinates, and
  // the range of cells that can hold a changing point
  __shared__ int st_snext, st_clo[MAXD], st_chi[MAXD], st_rows;
  __shared__ double st_xn[MAXD];
  // a round's: threshold, radius, sizes; number of steps (-1 while they are being taken)
  __shared__ long long rd_max, rd_tau;
  __shared__ float rd_radius;
  __shared__ int rd_nodes, rd_cands, rd_count[32];
  __shared__ volatile int rd_taken;
  __shared__ int rd_expired;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = MM_THREADS / 32;
  const int d = a.d, n = a.n, gs = a.g1, per = gs / 32;

  auto mark_dirty = [&](int gidx) {
    const unsigned bit = 1u << (gidx & 31);
    if (!(atomicOr(&dirty1[gidx >> 5], bit) & bit)) {
      const int pos = atomicAdd(&nlist1, 1);
      if (pos < LIST_MAX)
        list1[pos] = gidx;
      else
        overflow = 1;
    }
  };
  // level-1 nodes: argmax of dist over the slots [g gs, (g + 1) gs), ties to the lowest original index.  A warp takes
  // four nodes at a time (-1: none), so that their loads are in flight together.
  auto reduce_l1 = [&](const int (&gi)[4]) {
    long long bv[4];
    int bi[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      bv[u] = LLONG_MIN;
      bi[u] = INT_MAX;
    }
    for (int q = 0; q < per; ++q) {
      long long v[4];
      int i[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int s = gi[u] * gs + q * 32 + lane;
        const bool in = gi[u] >= 0 && s < n;
        v[u] = in ? key_of(__ldcg(a.dist + s)) : LLONG_MIN;
        i[u] = in ? a.orig[s] : INT_MAX;
      }
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (beats(v[u], i[u], bv[u], bi[u])) {
          bv[u] = v[u];
          bi[u] = i[u];
        }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      long long mv;
      int mi, ml;
      redux_argmax(bv[u], bi[u], mv, mi, ml);
      if (lane == 0 && gi[u] >= 0) {
        l1v[gi[u]] = mv;
        l1i[gi[u]] = mi;
      }
    }
  };
  auto reduce_l2 = [&](int gidx) {
    long long bv = LLONG_MIN;
    int bi = INT_MAX;
    for (int q = 0; q < 2; ++q) {
      const int c = gidx * 64 + q * 32 + lane;
      if (c < a.ng1 && beats(l1v[c], l1i[c], bv, bi)) {
        bv = l1v[c];
        bi = l1i[c];
      }
    }
    int ml;
    redux_argmax(bv, bi, bv, bi, ml);
    if (lane == 0) {
      l2v[gidx] = bv;
      l2i[gidx] = bi;
    }
  };

  if (*a.err != 0) return;  // uniform: written only by an earlier launch's kernel here

  // rebuild the tree from the distances of the previous launch
  for (int g0 = w; g0 < a.ng1; g0 += 4 * nw) {
    int gi[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) gi[u] = g0 + u * nw < a.ng1 ? g0 + u * nw : -1;
    reduce_l1(gi);
  }
  for (int q = tid; q < NG1_MAX / 32; q += MM_THREADS) dirty1[q] = 0u;
  if (tid < NG2_MAX / 32) dirty2[tid] = 0u;
  if (tid == 0) {
    nlist1 = 0;
    overflow = 0;
    rd_expired = 0;
  }
  __syncthreads();
  for (int gidx = w; gidx < a.ng2; gidx += nw) reduce_l2(gidx);
  __syncthreads();

  // (c), (d): the tree where distances changed (every node after an overflowing list), then the marks are cleared
  auto refresh_tree = [&]() {
    const bool full = overflow != 0;
    const int cnt = full ? a.ng1 : nlist1;
    for (int q0 = w; q0 < cnt; q0 += 4 * nw) {
      int gi[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int q = q0 + u * nw;
        gi[u] = q < cnt ? (full ? q : list1[q]) : -1;
        if (lane == 0 && q < cnt) atomicOr(&dirty2[(gi[u] >> 6) >> 5], 1u << ((gi[u] >> 6) & 31));
      }
      reduce_l1(gi);
    }
    __syncthreads();
    for (int c = w; c < a.ng2; c += nw)
      if (dirty2[c >> 5] & (1u << (c & 31))) reduce_l2(c);
    if (full) {
      for (int q = tid; q < NG1_MAX / 32; q += MM_THREADS) dirty1[q] = 0u;
    } else {
      for (int q = tid; q < cnt; q += MM_THREADS) {
        const int gidx = list1[q];
        atomicAnd(&dirty1[gidx >> 5], ~(1u << (gidx & 31)));
      }
    }
    __syncthreads();
    if (tid < NG2_MAX / 32) dirty2[tid] = 0u;
    if (tid == 0) {
      nlist1 = 0;
      overflow = 0;
    }
    __syncthreads();
  };

  double ratio = 0.9;         // uniform over the block, like the next two
  int singles = a.singles;    // position up to which steps are taken alone
  int wait = 512;             // steps alone after ties that no round can list, doubled each time they come again
  bool ties = false;          // more than CAND_MAX points share the maximum: the round takes those of them below index cut
  int cut = n;
  int t = a.t0;
  while (t < a.t1) {
    bool single = t < singles;
    double now = ratio;
    int lo = 0, hi = n + 1;
    while (!single) {  // the round's candidates; a smaller range of distances when there are too many
      if (w == 0) {
        long long bv = LLONG_MIN;
        for (int c = lane; c < a.ng2; c += 32) bv = l2v[c] > bv ? l2v[c] : bv;
        for (int o = 16; o > 0; o >>= 1) {
          const long long ov = __shfl_xor_sync(FULL, bv, o);
          bv = ov > bv ? ov : bv;
        }
        if (lane == 0) {
          const double mx = __longlong_as_double(bv);
          rd_max = bv;
          rd_tau = ties ? bv : key_of(mx * now);
          rd_radius = __double2float_ru(sqrt(mx) * (1.0 + 1e-6));
          rd_nodes = 0;
          rd_cands = 0;
          rd_taken = -1;
        }
      }
      __syncthreads();
      if (rd_max >= key_of(INFINITY)) {
        single = true;
        break;
      }
      if (rd_max == 0) {  // every point left coincides with one already taken: they follow by ascending index
        for (int i0 = 0; i0 < n && t < a.t1; i0 += MM_THREADS) {
          const int i = i0 + tid, s = i < n ? a.slot_of[i] : 0;
          const bool left = i < n && key_of(__ldcg(a.dist + s)) >= 0;
          const unsigned mask = __ballot_sync(FULL, left);
          if (lane == 0) rd_count[w] = __popc(mask);
          __syncthreads();
          int before = __popc(mask & ((1u << lane) - 1u)), total = 0;
          for (int q = 0; q < nw; ++q) {
            before += q < w ? rd_count[q] : 0;
            total += rd_count[q];
          }
          if (left && t + before < a.t1) {
            a.order[t + before] = i;
            __stcg(a.dist + s, -INFINITY);
          }
          t = min(t + total, a.t1);
          __syncthreads();
        }
        return;  // the last step of this launch; the next one rebuilds the tree
      }
      const long long tau = rd_tau;
      for (int g = tid; g < a.ng1; g += MM_THREADS)
        if (l1v[g] >= tau) {
          const int pos = atomicAdd(&rd_nodes, 1);
          if (pos < LIST_MAX) list1[pos] = g;
        }
      __syncthreads();
      const int nodes = rd_nodes;
      if (nodes <= LIST_MAX)
        for (int q0 = w; q0 < nodes; q0 += 4 * nw)
          for (int h = 0; h < per; ++h) {
            int s[4];
            long long v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) {  // four nodes' loads in flight
              const int q = q0 + u * nw;
              s[u] = q < nodes ? list1[q] * gs + h * 32 + lane : n;
              v[u] = s[u] < n ? key_of(__ldcg(a.dist + s[u])) : -1;
              if (ties && v[u] >= tau && a.orig[s[u]] >= cut) v[u] = -1;
            }
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              const unsigned mask = __ballot_sync(FULL, v[u] >= tau);
              int base = 0;
              if (lane == 0 && mask) base = atomicAdd(&rd_cands, __popc(mask));
              base = __shfl_sync(FULL, base, 0);
              const int pos = base + __popc(mask & ((1u << lane) - 1u));
              if (v[u] >= tau && pos < CAND_MAX) {
                uslot[pos] = s[u];
                ukey[pos] = v[u];
              }
            }
          }
      __syncthreads();
      const int nc = nodes <= LIST_MAX ? rd_cands : CAND_MAX + 1;
      __syncthreads();
      if (ties && nodes <= LIST_MAX) {
        // equal distances go by index, so the lowest of them are the next steps
        // (none below lo, too many below hi)
        if (nc > CAND_MAX) {
          hi = cut;
          cut = lo + max(CAND_MAX, (int)((hi - lo) * (0.75 * CAND_MAX / nc)));
          continue;
        }
        if (nc == 0) {
          lo = cut;
          cut = hi <= n ? lo + max(CAND_MAX, (hi - lo) / 2) : lo > n / 4 ? n : 4 * lo;
          continue;
        }
        if (cut == n) ties = false;
        if (nc < CAND_MAX / 4) cut = cut > n / 2 ? n : 2 * cut;
        break;
      }
      if (nc <= CAND_MAX) {
        // the next round's range of distances: about 3/4 of the candidates there is room for
        ratio = fmax(0.5, 1.0 - (1.0 - now) * fmin(1.5, 0.75 * CAND_MAX / nc));
        break;
      }
      now = 1.0 - (nc < 4 * CAND_MAX ? 0.5 : 0.125) * (1.0 - now);
      if (now > 1.0 - 1e-9) {  // more than CAND_MAX points share the maximum, or nearly: that may last for a while
        ties = nodes <= LIST_MAX;
        if (ties) {
          cut = max(CAND_MAX, (int)(n * (0.75 * CAND_MAX / nc)));
          now = ratio;  // for when the ties are through
        } else {
          singles = t + wait;
          wait *= 2;
          single = true;
        }
      }
    }
    if (!single) {
      const int nc = rd_cands;
      const long long tau = rd_tau;
      // by descending distance, ties by ascending index: a candidate's rank is the number of those that beat it
      if (tid < nc) {
        uidx[tid] = a.orig[uslot[tid]];
        rank[tid] = 0;
        taken[tid] = -1;
      }
      __syncthreads();
      {
        constexpr int PARTS = MM_THREADS / CAND_MAX;
        const int i = tid % CAND_MAX;
        if (i < nc) {
          const long long key = ukey[i];
          const int idx = uidx[i];
          int r = 0;
          for (int j = tid / CAND_MAX; j < nc; j += PARTS) r += beats(ukey[j], uidx[j], key, idx);
          atomicAdd(&rank[i], r);
        }
      }
      __syncthreads();
      // FP32 bounds: with E the length of the error bounds of the differences and d2 the FP32 squared distance, the true one
      // is at least (sqrt(d2) - E)^2 and at most (sqrt(d2) + E)^2, up to 2^-19 for the rounding of at most 8 terms and of the
      // square roots
      const float E = a.eps_length;
      if (tid < nc) {
        const int r = rank[tid], s = uslot[tid];
        skey[r] = ukey[tid];
        cslot[r] = s;
        cidx[r] = uidx[tid];
#pragma unroll
        for (int k = 0; k < DM; ++k) {
          cx[r * DP + k] = k < d ? a.Xf[(int64_t)s * d + k] : 0.0f;
          if (DM <= 4 && k < d) cxd[r * 4 + k] = a.Xs[(int64_t)s * d + k];
        }
        const float v = sqrtf(f32_above(ukey[tid])) + E;
        cthr[r] = v * v * (1.0f + 0x1p-17f);  // d2 at least this: it keeps its distance
      }
      __syncthreads();
      // (a) every pair: lane j of a warp against all rows
      {
        const float tauf = __double2float_rd(__longlong_as_double(tau)), vd = fmaxf(sqrtf(tauf) - E, 0.0f);
        const float thr_gone = tauf > 1e-30f ? vd * vd * (1.0f - 0x1p-17f) : 0.0f;  // d2 below this: it falls below tau
        const int word = w % CWORDS, j = word * 32 + lane;
        if (word * 32 < nc) {
          float xj[DM];
#pragma unroll
          for (int k = 0; k < DM; ++k) xj[k] = cx[j * DP + k];
          const float thr = cthr[j];
#pragma unroll 4
          for (int i = w / CWORDS; i < nc; i += nw / CWORDS) {
            float d2 = 0.0f;
#pragma unroll
            for (int k = 0; k < DM; ++k) {
              const float dx = xj[k] - cx[i * DP + k];
              d2 = fmaf(dx, dx, d2);
            }
            const unsigned may = __ballot_sync(FULL, !(d2 >= thr)), gone = __ballot_sync(FULL, d2 < thr_gone);
            if (lane == 0) pairs[i * CWORDS + word] = make_uint2(may, gone);
          }
        }
      }
      __syncthreads();
      if (w == 0) {
        // (b) the steps.  Lane l holds the candidates 32 l .. 32 l + 31: those still in place (alive), and those that came
        // down but not below tau (late).
        unsigned alive = lane < CWORDS ? (nc >= lane * 32 + 32 ? FULL : nc > lane * 32 ? (1u << (nc - lane * 32)) - 1u : 0u) : 0u;
        unsigned late = 0u;
        long long lkey = -1;
        int lidx = INT_MAX, lcand = -1, s = 0, hold = 0;
        for (;;) {
          const unsigned m = __ballot_sync(FULL, alive != 0u);
          // 32 candidates at once, as long as every conflict of theirs puts a point out of the round (most do): a
          // candidate is taken when no earlier one that it conflicts with is
          if (m && lkey < 0 && --hold < 0) {
            const int l0 = __ffs(m) - 1;
            const unsigned A = __shfl_sync(FULL, alive, l0);
            unsigned may = 0u, gone = 0u;  // bit j: candidate j of the 32 takes this lane's away (surely)
#pragma unroll 8
            for (int j = 0; j < 32; ++j) {
              const uint2 pr = pairs[(l0 * 32 + j) * CWORDS + l0];
              may |= ((pr.x >> lane) & 1u) << j;
              gone |= ((pr.y >> lane) & 1u) << j;
            }
            const bool in = (A >> lane) & 1u;
            may &= in ? A & ((1u << lane) - 1u) : 0u;
            if (!__any_sync(FULL, (may & ~gone) != 0u)) {
              unsigned T = 0u;
              for (unsigned U = A; U;) {  // the first of U is decided every time
                const bool open = (U >> lane) & 1u, out = open && (may & T);
                const unsigned tk = __ballot_sync(FULL, open && !out && !(may & U));
                U &= ~(tk | __ballot_sync(FULL, out));
                T |= tk;
              }
              unsigned go = 0u, stay = 0u;  // what they do to the other candidates
#pragma unroll 8
              for (int j = 0; j < 32; ++j)
                if (((T >> j) & 1u) && lane < CWORDS) {
                  const uint2 pr = pairs[(l0 * 32 + j) * CWORDS + lane];
                  go |= pr.y;
                  stay |= pr.x & ~pr.y;
                }
              const unsigned others = lane == l0 ? 0u : alive;
              if (!__any_sync(FULL, (stay & others) != 0u)) {
                alive = others & ~go;
                const int pos = s + __popc(T & ((1u << lane) - 1u));
                if (((T >> lane) & 1u) && t + pos < a.t1) *(volatile int*)(taken + pos) = l0 * 32 + lane;
                s += __popc(T);
                if (t + s >= a.t1) {
                  s = a.t1 - t;
                  break;
                }
                continue;
              }
            }
            hold = 8;
          }
          // one step: the first candidate in place or the best of the late ones
          int c = lcand;
          if (m) {
            const int l0 = __ffs(m) - 1;
            const int h = l0 * 32 + __ffs(__shfl_sync(FULL, alive, l0)) - 1;
            if (lkey < 0 || beats(skey[h], cidx[h], lkey, lidx)) c = h;
          } else if (lkey < 0) {
            break;  // no candidate reaches the threshold any more
          }
          if (lane == 0) *(volatile int*)(taken + s) = c;
          ++s;
          if (t + s == a.t1) break;
          const uint2 pr = lane < CWORDS ? pairs[c * CWORDS + lane] : make_uint2(0u, 0u);
          const unsigned self = lane == (c >> 5) ? 1u << (c & 31) : 0u;
          const unsigned hit = pr.x & (alive | late) & ~self, gone = hit & pr.y;
          unsigned open = hit & ~gone;
          const bool look = open != 0u || (late & (gone | self)) != 0u;
          alive &= ~(gone | self);
          late &= ~(gone | self);
          if (__any_sync(FULL, look)) {
            for (; open; open &= open - 1u) {
              const unsigned bit = open & (0u - open);
              const int j = lane * 32 + __ffs(open) - 1;
              const long long dk = key_of(DM <= 4 ? sqdist(cxd + j * 4, cxd + c * 4, d)
                                                  : sqdist(a.Xs + (int64_t)cslot[j] * d, a.Xs + (int64_t)cslot[c] * d, d));
              if (dk < skey[j]) {
                alive &= ~bit;
                late &= ~bit;
                if (dk >= tau) {
                  late |= bit;
                  skey[j] = dk;
                }
              }
            }
            long long bk = -1;
            int bi = INT_MAX, bc = -1, ml;
            for (unsigned u = late; u; u &= u - 1u) {
              const int j = lane * 32 + __ffs(u) - 1;
              if (beats(skey[j], cidx[j], bk, bi)) {
                bk = skey[j];
                bi = cidx[j];
                bc = j;
              }
            }
            redux_argmax(bk, bi, lkey, lidx, ml);
            lcand = __shfl_sync(FULL, bc, ml);
            __syncwarp();
          }
        }
        // the lanes' entries of taken[] before their number: __syncwarp orders them before lane 0's fence
        __syncwarp();
        if (lane == 0) {
          __threadfence_block();
          rd_taken = s;
        }
      } else {
        // (c) meanwhile the other warps: the neighbourhoods of the points taken, one warp per point, its cells' slots
        // spread over the lanes; the FP32 bound clears most of them, the others wait in the warp's queue for 32 FP64
        // distances at a time
        int2* qu = queue + w * QUEUE;
        int qn = 0;
        auto drain = [&](int cnt) {
          __syncwarp();
          if (lane < cnt) {
            const int2 e = qu[lane];
            const long long dk = key_of(sqdist(a.Xs + (int64_t)e.x * d, a.Xs + (int64_t)cslot[e.y] * d, d));
            if (atomicMin(reinterpret_cast<long long*>(a.dist + e.x), dk) > dk) mark_dirty(e.x / gs);
          }
          __syncwarp();
        };
        const float rf = rd_radius;
        // with few candidates several warps share a point's rows of cells
        const int share = min(32, max(1, 512 / nc));
        for (int unit = w - 1; unit < nc * share; unit += nw - 1) {
          const int q = unit / share, part = unit % share;
          int c = -1;
          unsigned long long since = 0;
          for (;;) {  // until step q is there, or the number of steps says that it will not come
            if (lane == 0) {
              const int steps = rd_taken;
              __threadfence_block();
              c = steps >= 0 && q >= steps ? -2 : *(volatile int*)(taken + q);
              if (c == -1) {
                const unsigned long long now = global_ns();
                if (since == 0) since = now;
                if (now - since >= a.wait_ns) {
                  rd_expired = 1;
                  c = -3;
                }
              }
            }
            c = __shfl_sync(FULL, c, 0);
            if (c != -1) break;
            __nanosleep(100);
          }
          if (c < 0) break;
          if (lane == 0 && part == 0) {
            a.order[t + q] = cidx[c];
            __stcg(a.dist + cslot[c], -INFINITY);
            mark_dirty(cslot[c] / gs);
          }
          // cells within the radius, in FP32 with a margin for its rounding
          int clo = 0, chi = 0;
          if (lane < d) {
            const float x = cx[c * DP + lane], ih = (float)a.g.inv_h[lane];
            const float marg = 1e-3f + (float)a.g.G[lane] * 0x1p-19f;
            clo = (int)fminf(fmaxf((x - rf) * ih - marg, 0.0f), (float)(a.g.G[lane] - 1));
            chi = (int)fminf(fmaxf((x + rf) * ih + marg, 0.0f), (float)(a.g.G[lane] - 1));
          }
          int rows = 1;
          for (int k = 1; k < d; ++k)
            rows *= __shfl_sync(FULL, chi, k) - __shfl_sync(FULL, clo, k) + 1;
          const int c0 = __shfl_sync(FULL, clo, 0), c1 = __shfl_sync(FULL, chi, 0);
          for (int r0 = part * 32; r0 < rows; r0 += 32 * share) {
            int rem = r0 + lane;
            long long cb = c0;
            for (int k = 1; k < d; ++k) {
              const int lo = __shfl_sync(FULL, clo, k), span = __shfl_sync(FULL, chi, k) - lo + 1;
              cb += (long long)(lo + rem % span) * a.g.stride[k];
              rem /= span;
            }
            int s0 = 0, len = 0;
            if (r0 + lane < rows) {
              s0 = a.cell_start[cb];
              len = a.cell_start[cb + (c1 - c0) + 1] - s0;
            }
            int inc = len;  // slots of this row and the rows before it
            for (int o = 1; o < 32; o <<= 1) {
              const int y = __shfl_up_sync(FULL, inc, o);
              if (lane >= o) inc += y;
            }
            const int total = __shfl_sync(FULL, inc, 31);
            for (int e0 = 0; e0 < total; e0 += 32) {
              const int e = e0 + lane;
              int row = 0;  // the row that holds entry e: rows whose running count is at most e lie before it
              for (int o = 16; o > 0; o >>= 1)
                if (__shfl_sync(FULL, inc, row + o - 1) <= e) row += o;
              row = min(row, 31);
              const int s = __shfl_sync(FULL, s0, row) + e - (__shfl_sync(FULL, inc, row) - __shfl_sync(FULL, len, row));
              bool hit = false;
              if (e < total) {
                const long long dv = key_of(__ldcg(a.dist + s));
                if (dv >= 0) {
                  float lb = 0.0f;
#pragma unroll
                  for (int k = 0; k < DM; ++k)
                    if (k < d) {
                      const float dl = fmaxf(fabsf(a.Xf[(int64_t)s * d + k] - cx[c * DP + k]) - a.eps[k], 0.0f);
                      lb = fmaf(dl, dl, lb);
                    }
                  hit = !(lb * (1.0f - 0x1p-18f) >= f32_above(dv));
                }
              }
              const unsigned mask = __ballot_sync(FULL, hit);
              if (hit) qu[qn + __popc(mask & ((1u << lane) - 1u))] = make_int2(s, c);
              qn += __popc(mask);
              if (qn >= 32) {
                drain(32);
                int2 keep = make_int2(0, 0);
                if (lane < qn - 32) keep = qu[32 + lane];
                __syncwarp();
                if (lane < qn - 32) qu[lane] = keep;
                qn -= 32;
                __syncwarp();
              }
            }
          }
        }
        drain(qn);
      }
      __syncthreads();
      if (rd_expired) {
        if (tid == 0) *a.err = 1;
        return;
      }
      t += rd_taken;
      refresh_tree();
      continue;
    }
    // ---- one step alone ----
    // (a) warp 0: the next point (the root of the tree) and the cells that can hold a changing point
    if (w == 0) {
      int next;
      double r2;
      if (t == 0) {
        next = a.first;
        r2 = INFINITY;
      } else {
        long long bv = LLONG_MIN;
        int bi = 0x7fffffff;
        for (int c = lane; c < a.ng2; c += 32)
          if (beats(l2v[c], l2i[c], bv, bi)) {
            bv = l2v[c];
            bi = l2i[c];
          }
        warp_argmax(bv, bi);
        next = bi;
        r2 = __longlong_as_double(bv);
      }
      const int snext = a.slot_of[next];
      const bool all = !(r2 < INFINITY);
      double r = 0.0;
      if (lane == 0 && !all) r = sqrt(r2) * (1.0 + RADIUS_MARGIN);
      r = __shfl_sync(FULL, r, 0);
      if (lane < d) {
        const double x = a.Xs[(int64_t)snext * d + lane];
        st_xn[lane] = x;
        st_clo[lane] = all ? 0 : cell_coord(a.g, lane, x - r);
        st_chi[lane] = all ? a.g.G[lane] - 1 : cell_coord(a.g, lane, x + r);
      }
      __syncwarp();
      if (lane == 0) {
        int rows = 1;
        for (int k = 1; k < d; ++k) rows *= (st_chi[k] - st_clo[k] + 1);
        st_rows = rows;
        st_snext = snext;
        a.order[t] = next;
        a.dist[snext] = -INFINITY;
        mark_dirty(snext / gs);
      }
    }
    __syncthreads();
    // (b) distance updates, one warp per row of cells along dimension 0 (contiguous slots)
    {
      const int snext = st_snext, rows = st_rows;
      double xn[MAXD];
      for (int k = 0; k < d; ++k) xn[k] = st_xn[k];
      for (int rho = w; rho < rows; rho += nw) {
        int rem = rho;
        long long cbase = st_clo[0];
        for (int k = 1; k < d; ++k) {
          const int span = st_chi[k] - st_clo[k] + 1;
          cbase += (long long)(st_clo[k] + rem % span) * a.g.stride[k];
          rem /= span;
        }
        const int s0 = a.cell_start[cbase], s1 = a.cell_start[cbase + (st_chi[0] - st_clo[0]) + 1];
        for (int s = s0 + lane; s < s1; s += 32) {
          if (s == snext) continue;
          const long long dv = key_of(__ldcg(a.dist + s));
          if (dv < 0) continue;  // already ordered (-inf)
          const double d2 = sqdist(a.Xs + (int64_t)s * d, xn, d);
          if (key_of(d2) < dv) {
            a.dist[s] = d2;
            mark_dirty(s / gs);
          }
        }
      }
    }
    __syncthreads();
    refresh_tree();
    ++t;
  }
}

// sorted per-warp list of the best k (squared distance, index) keys: insert the qualifying lanes' candidates
__device__ __forceinline__ void knn_offer(double dj, int ij, bool valid, int k, int lane, double* kd, int* ki,
                                          int& cnt, double& thr, int& thri) {
  const bool qual = valid && (cnt < k || dj < thr || (dj == thr && ij < thri));
  unsigned mask = __ballot_sync(FULL, qual);
  while (mask) {
    const int src = __ffs(mask) - 1;
    mask &= mask - 1;
    const double cd = __shfl_sync(FULL, dj, src);
    const int ci = __shfl_sync(FULL, ij, src);
    if (lane == 0) {
      const bool fullq = cnt >= k;
      if (!fullq || cd < kd[k - 1] || (cd == kd[k - 1] && ci < ki[k - 1])) {
        int pos = fullq ? k - 1 : cnt;
        while (pos > 0 && (kd[pos - 1] > cd || (kd[pos - 1] == cd && ki[pos - 1] > ci))) {
          kd[pos] = kd[pos - 1];
          ki[pos] = ki[pos - 1];
          --pos;
        }
        kd[pos] = cd;
        ki[pos] = ci;
      }
    }
    cnt = cnt < k ? cnt + 1 : k;
    __syncwarp();
  }
  __syncwarp();
  if (cnt >= k && k > 0) {
    thr = kd[k - 1];
    thri = ki[k - 1];
  }
}

// positions t in [t0, t1) with t <= KNN_BRUTE: scan positions 0 .. t - 1
__global__ void __launch_bounds__(256) k_knn_brute(int t0, int t1, int d, int m, const double* __restrict__ Xo,
                                                   const int32_t* __restrict__ order, int32_t* __restrict__ nbr) {
  __shared__ double kd[8][VECCHIA_MAX_M];
  __shared__ int ki[8][VECCHIA_MAX_M];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = t0 + blockIdx.x * 8 + w;
  if (t >= t1) return;
  const int k = t < m ? t : m;
  double xt[MAXD];
  for (int q = 0; q < d; ++q) xt[q] = Xo[(int64_t)t * d + q];
  int cnt = 0;
  double thr = INFINITY;
  int thri = 0x7fffffff;
  for (int j0 = 0; j0 < t; j0 += 32) {
    const int j = j0 + lane;
    double dj = INFINITY;
    int ij = 0x7fffffff;
    if (j < t) {
      dj = sqdist(xt, Xo + (int64_t)j * d, d);
      ij = order[j];
    }
    knn_offer(dj, ij, j < t, k, lane, kd[w], ki[w], cnt, thr, thri);
  }
  for (int q = lane; q < m; q += 32) nbr[(int64_t)t * m + q] = (q < k) ? ki[w][q] : -1;
}

// positions t in [t0, t1) on the grid over positions 0 .. np - 1 (slots hold positions; a slot qualifies when its
// position is below t): rings of cells around the query's cell, stopping once no unvisited cell can hold a better key
__global__ void __launch_bounds__(256) k_knn_grid(int t0, int t1, int m, GridDesc g, const int* __restrict__ cell_start,
                                                  const int* __restrict__ spos, const double* __restrict__ Xo,
                                                  const int32_t* __restrict__ order, int32_t* __restrict__ nbr) {
  __shared__ double kd[8][VECCHIA_MAX_M];
  __shared__ int ki[8][VECCHIA_MAX_M];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = t0 + blockIdx.x * 8 + w;
  if (t >= t1) return;
  const int d = g.d, k = t < m ? t : m;
  double xt[MAXD];
  int cq[MAXD];
  int rmax = 0;
  for (int q = 0; q < d; ++q) {
    xt[q] = Xo[(int64_t)t * d + q];
    cq[q] = cell_coord(g, q, xt[q]);
    rmax = max(rmax, max(cq[q], g.G[q] - 1 - cq[q]));
  }
  int cnt = 0;
  double thr = INFINITY;
  int thri = 0x7fffffff;
  for (int R = 0; R <= rmax; ++R) {
    // cells of the cube [cq - R, cq + R] (clamped) on its surface: max_k |c_k - cq_k| == R
    long long cube = 1;
    int lo[MAXD], span[MAXD];
    for (int q = 0; q < d; ++q) {
      lo[q] = max(0, cq[q] - R);
      span[q] = min(g.G[q] - 1, cq[q] + R) - lo[q] + 1;
      cube *= span[q];
    }
    for (long long c0 = 0; c0 < cube; c0 += 32) {
      const long long c = c0 + lane;
      int s0 = 0, s1 = 0;
      if (c < cube) {
        long long rem = c, cid = 0;
        int cheb = 0;
        for (int q = 0; q < d; ++q) {
          const int cc = lo[q] + (int)(rem % span[q]);
          rem /= span[q];
          cheb = max(cheb, abs(cc - cq[q]));
          cid += (long long)cc * g.stride[q];
        }
        if (cheb == R) {
          s0 = cell_start[cid];
          s1 = cell_start[cid + 1];
        }
      }
      // the lanes' cells one slot at a time; lanes with fewer slots offer nothing
      int more = __any_sync(FULL, s0 < s1);
      while (more) {
        double dj = INFINITY;
        int ij = 0x7fffffff;
        bool valid = false;
        if (s0 < s1) {
          const int pos = spos[s0];
          if (pos < t) {
            dj = sqdist(xt, Xo + (int64_t)pos * d, d);
            ij = order[pos];
            valid = true;
          }
          ++s0;
        }
        knn_offer(dj, ij, valid, k, lane, kd[w], ki[w], cnt, thr, thri);
        more = __any_sync(FULL, s0 < s1);
      }
    }
    // every unvisited point is at least R cell widths away in some dimension (less the rounding of the cell map)
    if (cnt >= k) {
      const double gap = (double)R * g.h_min - g.slack;
      if (gap > 0.0 && thr < gap * gap * (1.0 - 1e-12)) break;
    }
  }
  for (int q = lane; q < m; q += 32) nbr[(int64_t)t * m + q] = (q < k) ? ki[w][q] : -1;
}

__global__ void k_points_major(int n, int d, const double* __restrict__ X, const int32_t* __restrict__ order,
                               double* __restrict__ Xp, double* __restrict__ Xo) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int q = 0; q < d; ++q) {
    if (Xp) Xp[i * d + q] = X[i + (int64_t)q * n];
    if (Xo) Xo[i * d + q] = X[order[i] + (int64_t)q * n];
  }
}

template <class P>
struct DevBuf {
  P* p = nullptr;
  explicit DevBuf(size_t count) { LKG_CUDA(cudaMalloc(&p, sizeof(P) * std::max<size_t>(count, 1))); }
  ~DevBuf() { cudaFree(p); }
  DevBuf(const DevBuf&) = delete;
  DevBuf& operator=(const DevBuf&) = delete;
};

// a grid over np points (point-major P with stride d) with about `per_cell` points per cell
GridDesc make_grid(int np, int d, const double* lo, const double* hi, double per_cell) {
  GridDesc g{};
  g.d = d;
  const double cells = std::max(1.0, np / per_cell);
  const int per_dim = std::max(1, (int)std::floor(std::pow(cells, 1.0 / d)));
  long long stride = 1;
  g.h_min = INFINITY;
  double ext_max = 0.0;
  for (int k = 0; k < d; ++k) {
    const double ext = hi[k] - lo[k];
    g.G[k] = ext > 0.0 ? per_dim : 1;
    g.lo[k] = lo[k];
    g.inv_h[k] = ext > 0.0 ? g.G[k] / ext : 0.0;
    g.stride[k] = stride;
    stride *= g.G[k];
    if (ext > 0.0) g.h_min = std::min(g.h_min, ext / g.G[k]);
    ext_max = std::max(ext_max, std::max(std::fabs(lo[k]), std::fabs(hi[k])));
  }
  if (!(g.h_min < INFINITY)) g.h_min = 0.0;  // all points coincide: every query scans every cell
  g.slack = 1e-9 * std::max(ext_max, 1e-300);
  return g;
}

long long grid_cells(const GridDesc& g) {
  long long c = 1;
  for (int k = 0; k < g.d; ++k) c *= g.G[k];
  return c;
}

// counting sort of np points into the cells of g: cell_start (cells + 1) and perm (slot -> point)
void grid_sort(int np, const double* P, const GridDesc& g, int* cell, int* cell_start, int* cursor, int* perm,
               cudaStream_t st) {
  const long long nc = grid_cells(g);
  LKG_CUDA(cudaMemsetAsync(cell_start, 0, sizeof(int) * (nc + 1), st));
  k_grid_cells<<<ceil_div(np, 256), 256, 0, st>>>(np, P, g.d, g, cell, cell_start);
  LKG_LAUNCH("k_grid_cells");
  k_scan_exclusive<<<1, 1024, 0, st>>>((int)nc + 1, cell_start, nullptr);
  LKG_LAUNCH("k_scan_exclusive");
  LKG_CUDA(cudaMemcpyAsync(cursor, cell_start, sizeof(int) * nc, cudaMemcpyDeviceToDevice, st));
  k_grid_scatter<<<ceil_div(np, 256), 256, 0, st>>>(np, cell, cursor, perm);
  LKG_LAUNCH("k_grid_scatter");
}

}  // namespace

void vecchia_sets_grid(int n, int d, const double* hX, const double* dX, int first, int m, int32_t* dorder,
                       int32_t* dnbr, cudaStream_t st, unsigned long long wait_ns) {
  if (d < 1 || d > MAXD) throw std::invalid_argument("Vecchia sets on the GPU support 1 <= d <= 8");
  if (m > VECCHIA_MAX_M) throw std::invalid_argument("Vecchia sets on the GPU support m <= 32");
  // bounding box of the points (the grids' extent)
  std::vector<double> lo(d, INFINITY), hi(d, -INFINITY);
  for (int k = 0; k < d; ++k)
    for (int i = 0; i < n; ++i) {
      lo[k] = std::min(lo[k], hX[i + (size_t)k * n]);
      hi[k] = std::max(hi[k], hX[i + (size_t)k * n]);
    }
  DevBuf<double> Xp((size_t)n * d), Xs((size_t)n * d), dist(n);
  DevBuf<float> Xf((size_t)n * d);
  DevBuf<int> cell(n), perm(n), orig(n), slot_of((size_t)n + 1);
  int* const err = slot_of.p + n;  // the error word of the order's kernel
  LKG_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
  k_points_major<<<ceil_div(n, 256), 256, 0, st>>>(n, d, dX, nullptr, Xp.p, nullptr);
  LKG_LAUNCH("k_points_major");

  // ---- maxmin order on a grid of about 2 points per cell
  {
    const GridDesc g = make_grid(n, d, lo.data(), hi.data(), 2.0);
    const long long nc = grid_cells(g);
    DevBuf<int> cstart(nc + 1), cursor(nc);
    grid_sort(n, Xp.p, g, cell.p, cstart.p, cursor.p, perm.p, st);
    k_grid_slots<<<ceil_div(n, 256), 256, 0, st>>>(n, d, Xp.p, perm.p, g, Xs.p, Xf.p, orig.p, slot_of.p, dist.p);
    LKG_LAUNCH("k_grid_slots");
    int gs = G1;
    while (ceil_div(n, gs) > NG1_MAX) gs *= 2;
    MaxminArgs a{};
    a.n = n;
    a.d = d;
    a.first = first;
    a.g1 = gs;
    a.ng1 = ceil_div(n, gs);
    a.ng2 = ceil_div(a.ng1, 64);
    a.g = g;
    a.cell_start = cstart.p;
    a.Xs = Xs.p;
    a.Xf = Xf.p;
    // |x - lo| <= ext: two roundings to FP32 and the subtraction's own
    double length2 = 0.0;
    for (int k = 0; k < d; ++k) {
      a.eps[k] = std::nextafter((float)((hi[k] - lo[k]) * 0x1p-22), INFINITY);
      length2 += (double)a.eps[k] * a.eps[k];
    }
    a.eps_length = (float)(std::sqrt(length2) * (1.0 + 0x1p-20));
    a.orig = orig.p;
    a.slot_of = slot_of.p;
    a.dist = dist.p;
    a.order = dorder;
    a.err = err;
    a.wait_ns = wait_ns;
    // FP32 squares of differences between 1e-18 and 1e18 stay in range; other boxes take every step alone
    a.singles = ROUND_FROM;
    for (int k = 0; k < d; ++k)
      if (hi[k] > lo[k] && !(hi[k] - lo[k] > 1e-18 && hi[k] - lo[k] < 1e18)) a.singles = n;
    const auto kernel = d <= 2 ? k_maxmin_grid<2> : d == 3 ? k_maxmin_grid<3> : d == 4 ? k_maxmin_grid<4> : k_maxmin_grid<8>;
    const size_t smem = maxmin_smem(a.ng1, d);
    LKG_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int chunk = 65536;  // steps per launch: each launch stays well under a second
    for (int t0 = 0; t0 < n; t0 += chunk) {
      a.t0 = t0;
      a.t1 = std::min(n, t0 + chunk);
      LaunchTimer lt("k_maxmin_grid", st, 0.0, 8.0 * (a.t1 - t0) * 64.0);
      kernel<<<1, MM_THREADS, smem, st>>>(a);
      LKG_LAUNCH("k_maxmin_grid");
    }
    int expired = 0;
    LKG_CUDA(cudaMemcpyAsync(&expired, err, sizeof(int), cudaMemcpyDeviceToHost, st));
    LKG_CUDA(cudaStreamSynchronize(st));  // cstart / cursor are freed at scope exit
    // the order is incomplete then, and nothing may read it
    if (expired) throw std::runtime_error("Vecchia sets: a round of the maxmin order did not complete (timed out)");
  }
  if (m <= 0 || n < 2) return;
  // ---- neighbour sets (rows of m = min(m, n - 1) entries): ordered coordinates, then one grid per prefix of
  // 2^j positions serving the positions in (2^(j-1), 2^j]
  const int mm = std::min(m, n - 1);
  DevBuf<double> Xo((size_t)n * d);
  k_points_major<<<ceil_div(n, 256), 256, 0, st>>>(n, d, dX, dorder, nullptr, Xo.p);
  LKG_LAUNCH("k_points_major");
  const int tb = std::min(n, KNN_BRUTE + 1);
  {
    LaunchTimer lt("k_knn_brute", st, 0.0, 8.0 * d * (double)tb * tb / 2.0);
    k_knn_brute<<<ceil_div(tb, 8), 256, 0, st>>>(0, tb, d, mm, Xo.p, dorder, dnbr);
    LKG_LAUNCH("k_knn_brute");
  }
  DevBuf<int> pos_cell(n), spos(n);
  for (long long np = 2LL * KNN_BRUTE; np / 2 + 1 < n; np *= 2) {
    const int t0 = (int)(np / 2 + 1), t1 = (int)std::min<long long>(n, np + 1);
    const GridDesc g = make_grid(t1, d, lo.data(), hi.data(), 2.0);  // positions 0 .. t1 - 1
    const long long nc = grid_cells(g);
    DevBuf<int> cstart(nc + 1), cursor(nc);
    grid_sort(t1, Xo.p, g, pos_cell.p, cstart.p, cursor.p, spos.p, st);
    LaunchTimer lt("k_knn_grid", st, 0.0, 8.0 * (d + 1) * (double)(t1 - t0) * 8.0 * mm);
    k_knn_grid<<<ceil_div(t1 - t0, 8), 256, 0, st>>>(t0, t1, mm, g, cstart.p, spos.p, Xo.p, dorder, dnbr);
    LKG_LAUNCH("k_knn_grid");
  }
  // the grids' buffers are freed at scope exit: make sure their last users have run
  LKG_CUDA(cudaStreamSynchronize(st));
}

}  // namespace lkg
