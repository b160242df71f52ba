// fmm.cu — fast many-body: the 2-D FMM of fmm.zig on the device, bit-identical
// to its serial recursion (fmm.zig:247-354).
//
// The reference computes, per target, sums whose order is fixed by a serial
// dual-tree recursion from (root, root). Every accumulation here runs in that
// order, so the device result equals the reference's bit for bit:
//
//  keys     square extent, 16-bit quantised Morton keys, stable 4-pass sort
//           (tree.zig:287-309, 346-364).
//  cells    level-order cells over the sorted keys, leaf at <= 32 points or
//           depth 16, children contiguous (fmm.zig:685-717); all levels at
//           once from each point's shared digits (four launches, no level
//           barriers).
//  upward   from the leaves: bounding box, centre and radius (fmm.zig:721-754),
//           P2M at leaves and M2M from the children (fmm.zig:757-806), then
//           M_k /= k! (fmm.zig:629-642).
//  lists    the recursion's calls, each cell's after its parent's. A call (A, B)
//           either ends (M2L of B into A, P2P of B into A's points, or nothing
//           past distanceMax), or splits B (the calls (A, B_j) follow at once,
//           in order), or splits A (the call goes to every child of A). So
//           every child of A receives the same ordered list of B's — the
//           "forward" list of A — and each cell's M2L and P2P lists come out
//           in the order the serial recursion meets them.
//  m2l      per cell, its M2L sources in list order: a lane per (source, three
//           l) computes the two-lane correlation of fmm.zig:561-610, then a
//           lane per coefficient adds the sources in order; L_l is unscaled by
//           (-1)^l / l! (fmm.zig:645-657).
//  p2p      per leaf, one to four lanes per target point run fmm.zig:477-553
//           against each source leaf of its list in order.
//  downward per cell with leaf children: L2L along its path from the root and
//           into the children (fmm.zig:823-849), L2P there (fmm.zig:853-886).
#include <cstdlib>

#include "fast.cuh"
#include "scan_sort.cuh"

namespace d3 {

constexpr uint32_t FMM_MAX_ORDER = 24;
constexpr uint32_t FMM_DEFAULT_ORDER = 8;
constexpr double FMM_DEFAULT_OPENING = 1.4;
constexpr uint32_t FMM_LEAF = 32;
constexpr uint32_t FMM_LEVELS = 16;
constexpr double FMM_MIN_SEP2 = 1e-28;
constexpr uint32_t FMM_TAB = 2 * FMM_MAX_ORDER + 2;  // rows of the binomial table
constexpr unsigned LISTS_THREADS = 128;
constexpr unsigned UP_THREADS = 64, M2L_THREADS = 32, P2P_THREADS = 32, DOWN_THREADS = 64;
// A P2P list of more than LONG_LIST source leaves (a leaf beside a far denser
// region) goes by segments of 32; the terms of a segment and 16 targets take a
// unit of 32 KB, LONG_UNITS_MAX of them at most (256 MB, held once a run wanted
// some; lists past that or past what the device has left, and leaves of more
// than LONG_POINTS points, go by k_fmm_p2p). LONG_LIST 32 / 64 / 128: a tick of
// 80,000 clustered nodes 494 / 503 / 579 us, 80,000 in tighter clusters 945 /
// 945 / 1,014.
constexpr uint32_t LONG_LIST = 64, LONG_POINTS = 64, LONG_UNITS_MAX = 8192;
constexpr uint32_t LONG_UNIT = 32 * 4 * 16;  // terms: source leaf, three pairs and a sum, target

// The two launches and their chains take 45 to 60 us, which only a list that
// is long against k_fmm_p2p's own chain gives back: they are taken when the
// longest list of the last run passed LONG_WORTH, or LONG_WORTH_FEW where the
// cells are few and k_fmm_p2p has four lanes a target. A tick with / without
// them, by the longest list. Few cells: 77 leaves 366 / 305 us, 96 408 / 360,
// 120 424 / 402, 160 404 / 410, 230 421 / 482, 340 450 / 608. More cells: 80
// 441 / 386, 137 497 / 517, 245 459 / 523, 677 947 / 1,522.
constexpr uint32_t LONG_WORTH_FEW = 192, LONG_WORTH = 96;

constexpr uint32_t P2P_FEW_CELLS = 4096;  // some 30,000 nodes; measured at k_fmm_p2p
constexpr uint32_t FMM_STACK = 64;


struct FmmTables {
  double fact[FMM_TAB];
  double ifact[FMM_TAB];            // 1 / fact
  double binom[FMM_TAB * FMM_TAB];  // binom[n * FMM_TAB + k]
};

// info words (device, mirrored to the host after the cell build)
enum : uint32_t { FI_CELLS = 0, FI_OVERFLOW, FI_LEVELS, FI_POOL_M2L, FI_POOL_P2P, FI_POOL_FWD,
                  FI_LIST_OVERFLOW,              // 1: a pool, 2: a call stack, 4: a wait ran out
                  FI_TICKET,                     // k_fmm_lists' blocks so far
                  FI_LVL = 8,  // FI_LVL + d: first cell of level d
                  FI_LONG_UNITS = 36, FI_LONGS,  // long P2P lists: units of terms, leaves,
                  FI_LONG_MAX,                   // the longest list's source leaves
                  FI_DONE,                       // counts on while k_fmm_lists makes progress
                  FI_M = 40,                     // points to act on (0 when the extent is bad)
                  FI_BAD = 41 };                 // 1: the extent is not finite and positive

struct FmmDev {
  uint32_t pcap = 0, ccap = 0;
  size_t coef_cap = 0, cap_m2l = 0, cap_p2p = 0, cap_fwd = 0;
  double *px = nullptr, *py = nullptr, *ps = nullptr, *ux = nullptr, *uy = nullptr;
  FCell *cells = nullptr;
  double *bx0 = nullptr, *by0 = nullptr, *bx1 = nullptr, *by1 = nullptr;
  uint32_t *m2l_off = nullptr, *m2l_cnt = nullptr, *p2p_off = nullptr, *p2p_cnt = nullptr;
  uint32_t *fwd_off = nullptr, *fwd_cnt = nullptr;
  uint32_t *m2l = nullptr, *p2p = nullptr, *fwd = nullptr;
  double *mco = nullptr, *lco = nullptr;
  FmmTables *tab = nullptr;
  uint32_t tab_p = 0;
  uint32_t *info = nullptr, *arrive = nullptr;
  uint2 *long_items = nullptr;
  uint32_t *long_at = nullptr, *longs = nullptr, *long_flags = nullptr;
  double2 *long_terms = nullptr;
  SpareRoom long_room{0, 0, LONG_UNITS_MAX};  // units
  uint32_t long_max = 0, longs_last = 0;      // the last run's longest P2P list, its leaves in segments
  cudaEvent_t lists_read = nullptr;  // the lists' words are in h_info
  double *square = nullptr;      // box x0, y0, side
  uint32_t *h_info = nullptr;    // pinned mirror of info
  double *h_geom = nullptr;      // pinned: the geometry read back (w, 1 / w, ox, oy)
  double *geom = nullptr;        // device: w, 1 / w, ox, oy (k_fmm_geom)
  size_t last_m2l = 0, last_p2p = 0, last_fwd = 0;  // list sizes of the previous run
  // the cell build: per-block counts per level, each cell's start and level
  uint32_t *cb_count = nullptr, *start_of = nullptr;
  uint16_t *pt_levels = nullptr;  // per point: the levels it starts cells at, d0 << 8 | d1
  uint8_t *level_of = nullptr;
  size_t cb_count_cap = 0, start_cap = 0, level_cap = 0;
};

struct FmmArgs {
  const uint64_t *keys;
  const uint32_t *perm;
  const double *px, *py, *ps, *ux, *uy;
  FCell *cells;
  double *bx0, *by0, *bx1, *by1;
  double *mco, *lco;
  const FmmTables *tab;
  double *vx, *vy;
  uint32_t *m2l, *p2p, *fwd;
  uint32_t *m2l_off, *m2l_cnt, *p2p_off, *p2p_cnt, *fwd_off, *fwd_cnt;
  uint32_t *info, *arrive;
  uint2 *long_items;  // per unit: the leaf and its item (NONE: not an item's first unit)
  uint32_t *long_at, *longs, *long_flags;  // per cell: first unit or NONE; the leaves; see there
  double2 *long_terms;
  uint32_t long_cap;
  uint32_t by_level;               // k_fmm_lists: a launch a level, nothing to wait for
  unsigned long long wait_ns;      // k_fmm_lists: a wait's limit
  size_t cap_m2l, cap_p2p, cap_fwd;
  uint32_t ncells, p;
  double mac_far, dmax_scaled, dmin_scaled, dmin2, dmax2, inv_w;
  int ring, has_dmax;
  const double *seed;
};

__device__ inline double ldg_cg(const double *p) { return __ldcg(p); }
__device__ inline uint32_t ldg_cg(const uint32_t *p) { return __ldcg(p); }

// zig @min / @max on finite operands
__device__ inline double zmin(double a, double b) { return b < a ? b : a; }
__device__ inline double zmax(double a, double b) { return b > a ? b : a; }

// ---- keys and gather --------------------------------------------------------

// tree.zig:346-364, 688-695
__device__ inline uint64_t spread16(uint32_t v) {
  uint64_t x = v & 0xFFFF;
  x = (x | (x << 8)) & 0x00FF00FF;
  x = (x | (x << 4)) & 0x0F0F0F0F;
  x = (x | (x << 2)) & 0x33333333;
  x = (x | (x << 1)) & 0x55555555;
  return x;
}

// Sort value: the node, with bit 31 for a NaN coordinate (partitioned last).
__global__ void k_fmm_keys(const double *xs, const double *ys, uint32_t n, const double *square,
                           uint64_t *keys, uint32_t *sv) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double x = xs[i], y = ys[i];
  if (x != x || y != y) {
    keys[i] = 0;
    sv[i] = i | 0x80000000u;
    return;
  }
  const double b0 = square[0], b1 = square[1], scale = 65536.0 / square[2];
  const double fx = floor((x - b0) * scale), fy = floor((y - b1) * scale);
  const uint32_t qx = (uint32_t)(fx < 65535 ? fx : 65535);
  const uint32_t qy = (uint32_t)(fy < 65535 ? fy : 65535);
  keys[i] = spread16(qx) | (spread16(qy) << 1);
  sv[i] = i;
}

// fmm.zig:668-682
// The run's geometry from the square's extent (tree.zig:287-309): geom =
// {w, 1 / w, ox, oy}; FI_M = the finite points, or 0 with FI_BAD = 1 when
// there are some but the extent is not finite and positive (the exact kernel
// runs instead). The
// same IEEE f64 operations the host would do, so the values are the same.
__global__ void k_fmm_geom(const double *extent, const uint32_t *tinfo, double *geom,
                           uint32_t *info) {
  const double e0 = extent[0], e1 = extent[1], e2 = extent[2], e3 = extent[3];
  const double w = e2 - e0;
  const bool ok = w > 0 && w < INFINITY;
  geom[0] = w;
  geom[1] = 1 / w;
  geom[2] = (e0 + e2) / 2;
  geom[3] = (e1 + e3) / 2;
  const uint32_t m = tinfo[0];
  info[FI_M] = ok ? m : 0;
  info[FI_BAD] = m > 0 && !ok ? 1 : 0;
}

__global__ void k_fmm_gather(const uint32_t *perm, const double *xs, const double *ys,
                             const double *strength, const uint32_t *info, double alpha,
                             const double *geom, double *px, double *py, double *ps, double *ux,
                             double *uy) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= info[FI_M]) return;
  const double inv_w = geom[1], ox = geom[2], oy = geom[3];
  const uint32_t i = perm[j];
  const double x = xs[i], y = ys[i];
  px[j] = x;
  py[j] = y;
  const double st = strength[i] * alpha;
  ps[j] = st != st ? 0 : st;
  ux[j] = (x - ox) * inv_w;
  uy[j] = (y - oy) * inv_w;
}

// ---- cells (fmm.zig:685-717) ---------------------------------------------------

// The child ranges of a cell at depth d: bnd[q] .. bnd[q + 1] holds digit q.
// Returns the number of non-empty children (0 for a leaf).
__device__ uint32_t child_ranges(const uint64_t *keys, uint32_t first, uint32_t count, uint32_t d,
                                 uint32_t *bnd) {
  if (count <= FMM_LEAF || d >= FMM_LEVELS) return 0;
  const unsigned shift = 2 * (FMM_LEVELS - 1 - d);
  const uint32_t end = first + count;
  bnd[0] = first;
  bnd[4] = end;
  for (uint32_t q = 1; q < 4; ++q) {
    uint32_t lo = bnd[q - 1], hi = end;
    while (lo < hi) {
      const uint32_t mid = lo + (hi - lo) / 2;
      if (((keys[mid] >> shift) & 3) < q) lo = mid + 1;
      else hi = mid;
    }
    bnd[q] = lo;
  }
  uint32_t nc = 0;
  for (uint32_t q = 0; q < 4; ++q) nc += bnd[q + 1] > bnd[q];
  return nc;
}

// ---- cells, all levels at once -------------------------------------------------------
//
// The same cells as fmm.zig:685-717 (level order, each level in key order,
// children contiguous in digit order), built without a pass per level. A
// level-d cell is a maximal run of sorted keys sharing d digits whose
// enclosing level-(d-1) run holds more than FMM_LEAF points (d <= 16). So a
// point k starts cells at the levels d in (lcp(k), top(k)], where lcp(k) is
// the digits it shares with point k - 1, provided the level-lcp(k) run around
// it holds more than FMM_LEAF points, and top(k) = min(16, max(lcp + 1,
// A(k) + 1)) with A(k) the digits keys k and k + FMM_LEAF share (a run that
// starts at k holds more than FMM_LEAF points exactly at the levels <= A(k)).
// Passes: per point the flags and per-block counts per level; a scan of the
// counts; per point the cells' places (level start + block offset + rank in
// the block); per cell its range, children and parent by binary searches.

constexpr uint32_t CB_THREADS = 256;
constexpr uint32_t CB_LEVELS = FMM_LEVELS + 1;  // levels 0 .. 16

__device__ inline int shared_digits(uint32_t a, uint32_t b) {
  return a == b ? 16 : __clz(a ^ b) >> 1;
}

// First index in [lo, hi) whose key >= t (keys sorted; low 32 bits).
__device__ inline uint32_t key_lower(const uint64_t *keys, uint32_t lo, uint32_t hi, uint64_t t) {
  while (lo < hi) {
    const uint32_t mid = lo + (hi - lo) / 2;
    if ((uint64_t)(uint32_t)keys[mid] < t) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// The same first index for a run known to hold k - 1 (keys[k - 1] >= t):
// galloping back from k - 1, then a binary search of the last stride, so a
// short run costs a few loads.
__device__ inline uint32_t key_lower_back(const uint64_t *keys, uint32_t k, uint64_t t) {
  uint32_t hi = k - 1;  // keys[hi] >= t
  uint32_t lo = 0;
  for (uint32_t step = 1; step <= hi; step <<= 1) {
    const uint32_t probe = hi - step;
    if ((uint64_t)(uint32_t)keys[probe] < t) {
      lo = probe + 1;
      break;
    }
    hi = probe;
  }
  return key_lower(keys, lo, hi, t);
}

// First index in [k, m) whose key >= t, for keys[k] < t: galloping forward
// from k, then a binary search of the last stride (a short run costs a few
// loads).
__device__ inline uint32_t key_lower_fwd(const uint64_t *keys, uint32_t k, uint32_t m, uint64_t t) {
  uint32_t lo = k + 1, hi = m;  // the answer is in [lo, hi]
  for (uint32_t step = 1; lo < m; step <<= 1) {
    const uint32_t probe = step < m - lo ? lo + step - 1 : m - 1;
    if ((uint64_t)(uint32_t)keys[probe] >= t) {
      hi = probe;
      break;
    }
    lo = probe + 1;
  }
  return key_lower(keys, lo, hi, t);
}

// The levels at which point k starts cells: [d0, d1] (empty when d1 < d0).
__device__ void cell_levels(const uint64_t *keys, uint32_t m, uint32_t k, int &d0, int &d1) {
  const uint32_t key = (uint32_t)keys[k];
  const int lcp = k == 0 ? -1 : shared_digits((uint32_t)keys[k - 1], key);
  d0 = lcp + 1;
  d1 = -1;
  if (lcp >= (int)FMM_LEVELS) return;
  if (k > 0) {
    // the level-lcp run around k must hold more than FMM_LEAF points
    const uint64_t t = lcp ? (uint64_t)(key >> (32 - 2 * lcp)) << (32 - 2 * lcp) : 0;
    const uint32_t s0 = key_lower_back(keys, k, t);
    if (s0 + FMM_LEAF >= m) return;
    if (shared_digits((uint32_t)keys[s0], (uint32_t)keys[s0 + FMM_LEAF]) < lcp) return;
  }
  const int A = k + FMM_LEAF < m ? shared_digits(key, (uint32_t)keys[k + FMM_LEAF]) : -1;
  int top = A + 1 > d0 ? A + 1 : d0;
  d1 = top < (int)FMM_LEVELS ? top : (int)FMM_LEVELS;
}

__global__ void __launch_bounds__(CB_THREADS) k_cells_count(const uint64_t *keys,
                                                            const uint32_t *info, uint32_t *bcount,
                                                            uint16_t *levels) {
  const uint32_t m = info[FI_M];
  __shared__ uint32_t wc[CB_LEVELS][CB_THREADS / 32];
  const uint32_t k = blockIdx.x * CB_THREADS + threadIdx.x;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int d0 = 0, d1 = -1;
  if (k < m) {
    cell_levels(keys, m, k, d0, d1);
    levels[k] = (uint16_t)(((uint32_t)d0 << 8) | ((uint32_t)d1 & 0xFFu));  // for k_cells_place
  }
  for (int d = 0; d < (int)CB_LEVELS; ++d) {
    const unsigned b = __ballot_sync(0xffffffffu, d >= d0 && d <= d1);
    if (lane == 0) wc[d][warp] = __popc(b);
  }
  __syncthreads();
  if (threadIdx.x < CB_LEVELS) {
    uint32_t t = 0;
    for (uint32_t w = 0; w < CB_THREADS / 32; ++w) t += wc[threadIdx.x][w];
    bcount[(size_t)threadIdx.x * gridDim.x + blockIdx.x] = t;
  }
}

// One block per level: the exclusive scan of that level's block counts; the
// level's cell count goes to info FI_LVL + d (k_cells_starts turns the counts
// into starts).
__global__ void __launch_bounds__(1024) k_cells_scan(uint32_t *bcount, uint32_t nb,
                                                     uint32_t *info) {
  __shared__ uint32_t sw[32];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint32_t d = blockIdx.x;
  uint32_t *v = bcount + (size_t)d * nb;
  uint32_t run = 0;
  for (uint32_t base = 0; base < nb; base += blockDim.x) {
    const uint32_t i = base + threadIdx.x;
    const uint32_t x = i < nb ? v[i] : 0;
    uint32_t incl = x;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (unsigned)o) incl += y;
    }
    if (lane == 31) sw[warp] = incl;
    __syncthreads();
    uint32_t wpre = 0, tile = 0;
    for (unsigned w = 0; w < nw; ++w) {
      if (w < warp) wpre += sw[w];
      tile += sw[w];
    }
    if (i < nb) v[i] = run + wpre + incl - x;
    run += tile;
    __syncthreads();
  }
  if (threadIdx.x == 0) info[FI_LVL + d] = run;
}

// One warp: the level starts (info FI_LVL + d) from the per-level counts, the
// cell total, the level count, and the overflow word when the cells do not
// fit `ccap`.
__global__ void __launch_bounds__(32) k_cells_starts(uint32_t ccap, uint32_t *info) {
  static_assert(CB_LEVELS <= 32, "one lane per level");
  const unsigned lane = threadIdx.x;
  const uint32_t x = lane < CB_LEVELS ? info[FI_LVL + lane] : 0;
  uint32_t incl = x;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (unsigned)o) incl += y;
  }
  const uint32_t at = __shfl_sync(0xffffffffu, incl, 31);
  const unsigned used = __ballot_sync(0xffffffffu, x != 0);
  if (lane < CB_LEVELS) info[FI_LVL + lane] = incl - x;
  if (lane == 0) {
    info[FI_LONG_UNITS] = info[FI_LONGS] = info[FI_LONG_MAX] = 0;
    info[FI_LVL + CB_LEVELS] = at;
    info[FI_CELLS] = at;
    info[FI_LEVELS] = used ? 32 - __clz(used) : 0;
    info[FI_OVERFLOW] = at > ccap ? at : 0;
  }
}

// start_of[cell] = the point that starts it; level_of[cell] = its level.
// (the point's levels as k_cells_count found them)
__global__ void __launch_bounds__(CB_THREADS) k_cells_place(const uint16_t *levels,
                                                            const uint32_t *bcount,
                                                            const uint32_t *info,
                                                            uint32_t *start_of,
                                                            uint8_t *level_of) {
  __shared__ uint32_t wc[CB_LEVELS][CB_THREADS / 32];
  if (__ldcg(&info[FI_OVERFLOW])) return;
  const uint32_t m = info[FI_M];
  const uint32_t k = blockIdx.x * CB_THREADS + threadIdx.x;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int d0 = 0, d1 = -1;
  if (k < m) {
    const uint32_t v = levels[k];
    d0 = (int)(v >> 8);
    d1 = (int)(int8_t)(v & 0xFFu);
  }
  uint32_t rank[CB_LEVELS];
  for (int d = 0; d < (int)CB_LEVELS; ++d) {
    const unsigned b = __ballot_sync(0xffffffffu, d >= d0 && d <= d1);
    rank[d] = __popc(b & ((1u << lane) - 1));
    if (lane == 0) wc[d][warp] = __popc(b);
  }
  __syncthreads();
  if (k >= m) return;
  for (int d = d0; d <= d1; ++d) {
    uint32_t pre = 0;
    for (uint32_t w = 0; w < warp; ++w) pre += wc[d][w];
    const uint32_t c = __ldcg(&info[FI_LVL + d]) + bcount[(size_t)d * gridDim.x + blockIdx.x] +
                       pre + rank[d];
    start_of[c] = k;
    level_of[c] = (uint8_t)d;
  }
}

__global__ void __launch_bounds__(CB_THREADS) k_cells_fill(const uint64_t *keys,
                                                           const uint32_t *start_of,
                                                           const uint8_t *level_of,
                                                           const uint32_t *info, FCell *cells,
                                                           uint32_t *arrive, uint32_t *fwd_cnt) {
  const uint32_t m = info[FI_M];
  const uint32_t total = __ldcg(&info[FI_CELLS]);
  if (__ldcg(&info[FI_OVERFLOW])) return;
  const uint32_t c = blockIdx.x * CB_THREADS + threadIdx.x;
  if (c >= total) return;
  const uint32_t k = start_of[c];
  const int d = level_of[c];
  const uint32_t key = (uint32_t)keys[k];
  // the run: the points sharing d digits with k
  uint32_t end = m;
  if (d > 0) {
    const uint64_t pre = key >> (32 - 2 * d);
    end = key_lower_fwd(keys, k, m, (pre + 1) << (32 - 2 * d));
  }
  FCell f;
  f.cx = f.cy = f.r = 0;
  f.first = k;
  f.count = end - k;
  f.depth = (uint32_t)d;
  f.child0 = 0;
  f.nchild = 0;
  if (f.count > FMM_LEAF && d < (int)FMM_LEVELS) {
    uint32_t bnd[5];
    f.nchild = child_ranges(keys, k, f.count, (uint32_t)d, bnd);
    // the first child starts at k: its place among level d + 1's starts
    const uint32_t lo = __ldcg(&info[FI_LVL + d + 1]), hi = __ldcg(&info[FI_LVL + d + 2]);
    uint32_t a = lo, b = hi;
    while (a < b) {
      const uint32_t mid = a + (b - a) / 2;
      if (start_of[mid] < k) a = mid + 1;
      else b = mid;
    }
    f.child0 = a;
  }
  f.parent = NONE;
  if (d > 0) {
    // the level d - 1 cell holding k: the last start <= k among that level's
    const uint32_t lo = __ldcg(&info[FI_LVL + d - 1]), hi = __ldcg(&info[FI_LVL + d]);
    uint32_t a = lo, b = hi;
    while (a < b) {
      const uint32_t mid = a + (b - a) / 2;
      if (start_of[mid] <= k) a = mid + 1;
      else b = mid;
    }
    f.parent = a - 1;
  }
  cells[c] = f;
  arrive[c] = 0;       // children k_fmm_upward has finished
  fwd_cnt[c] = NONE;   // k_fmm_lists' forward list is not there yet
}

// ---- upward: geometry, P2M, M2M, scale ------------------------------------------

// fmm.zig:614-623: powers of d = (dre, dim) into pw[0..p] (re) and pw[q..] (im).
__device__ inline void shift_powers(double dre, double dim, uint32_t p, double *pw) {
  const uint32_t q = p + 1;
  double re = 1, im = 0;
  pw[0] = 1;
  pw[q] = 0;
  for (uint32_t k = 1; k <= p; ++k) {
    const double nre = re * dre - im * dim;
    const double nim = re * dim + im * dre;
    re = nre;
    im = nim;
    pw[k] = re;
    pw[q + k] = im;
  }
}

// Minimum / maximum as the serial scan's strict comparisons: the first
// occurrence in point order wins a tie.
__device__ inline void minmax_merge(double &mn, uint32_t &imn, double &mx, uint32_t &imx,
                                    double omn, uint32_t oimn, double omx, uint32_t oimx) {
  if (omn < mn || (omn == mn && oimn < imn)) { mn = omn; imn = oimn; }
  if (omx > mx || (omx == mx && oimx < imx)) { mx = omx; imx = oimx; }
}

__device__ inline void write_box(const FmmArgs &a, uint32_t c, double x0, double y0, double x1,
                                 double y1, double cx, double cy) {
  a.bx0[c] = x0; a.by0[c] = y0; a.bx1[c] = x1; a.by1[c] = y1;
  const double dx = x1 - x0, dy = y1 - y0;
  a.cells[c].cx = cx;
  a.cells[c].cy = cy;
  a.cells[c].r = 0.5 * sqrt(dx * dx + dy * dy);
}

// Real r of cell c's multipole; the root's, which no parent reads, scaled.
__device__ inline void store_sums(const FmmArgs &a, uint32_t c, uint32_t q, uint32_t r, double v) {
  if (r >= 2 * q) return;
  const uint32_t o = r % q;
  a.mco[(size_t)c * 2 * q + r] = c == 0 && o >= 2 ? v * a.tab->ifact[o] : v;
}

// Shared doubles a warp of k_fmm_upward needs: 32 rows of a point's terms (odd
// rows: no bank conflicts), more than four children's coefficients, powers and
// sums take.
__host__ __device__ constexpr uint32_t up_row(uint32_t stride) { return stride | 1; }

// A warp per leaf: box, centre and P2M. The warp that finishes a cell's last
// child (`arrive` counts them) goes on with the cell: box from the children's,
// M2M with a lane per (child, coefficient), up to the root. A plain launch, and
// a chain of one or two microseconds a level: with a grid barrier a level, the
// children one after another and the coefficients read from L2 inside the sums
// it was a chain of 16 us a level (6,000 nodes: 98 -> 31 us; 1 M: 358 ->
// 193 us). A parent is the last reader of its children's sums, so it also
// scales them (fmm.zig:629-642: M_k /= k!); no pass of its own. P fixes the
// order at compile time (0: the order of the arguments) so that the sums unroll.
template <uint32_t P>
__global__ void __launch_bounds__(UP_THREADS) k_fmm_upward(FmmArgs a) {
  extern __shared__ double fmm_smem[];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t p = P ? P : a.p, q = p + 1, stride = 2 * q, row = up_row(stride);
  double *ws = fmm_smem + warp * 32 * row;
  uint32_t c = blockIdx.x * (UP_THREADS / 32) + warp;
  if (c >= a.ncells || a.cells[c].nchild) return;
  {
    const uint32_t first = a.cells[c].first, count = a.cells[c].count;
    double mnx = INFINITY, mxx = -INFINITY, mny = INFINITY, mxy = -INFINITY;
    uint32_t imnx = NONE, imxx = NONE, imny = NONE, imxy = NONE;
    for (uint32_t k = first + lane; k < first + count; k += 32) {
      const double x = a.ux[k], y = a.uy[k];
      if (x < mnx) { mnx = x; imnx = k; }
      if (x > mxx) { mxx = x; imxx = k; }
      if (y < mny) { mny = y; imny = k; }
      if (y > mxy) { mxy = y; imxy = k; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const double a0 = __shfl_xor_sync(0xffffffffu, mnx, o), a1 = __shfl_xor_sync(0xffffffffu, mxx, o);
      const uint32_t i0 = __shfl_xor_sync(0xffffffffu, imnx, o), i1 = __shfl_xor_sync(0xffffffffu, imxx, o);
      const double b0 = __shfl_xor_sync(0xffffffffu, mny, o), b1 = __shfl_xor_sync(0xffffffffu, mxy, o);
      const uint32_t j0 = __shfl_xor_sync(0xffffffffu, imny, o), j1 = __shfl_xor_sync(0xffffffffu, imxy, o);
      minmax_merge(mnx, imnx, mxx, imxx, a0, i0, a1, i1);
      minmax_merge(mny, imny, mxy, imxy, b0, j0, b1, j1);
    }
    const double cx = (mnx + mxx) / 2, cy = (mny + mxy) / 2;
    if (lane == 0) write_box(a, c, mnx, mny, mxx, mxy, cx, cy);
    // P2M (fmm.zig:757-780): lane t holds point t's terms; then lane r adds
    // real r (re 0..q-1, im q..2q-1) over the points in order.
    double acc0 = 0, acc1 = 0;
    const uint32_t r0 = lane, r1 = lane + 32;
    for (uint32_t base = first; base < first + count; base += 32) {
      const uint32_t k = base + lane;
      const uint32_t np = min(32u, first + count - base);
      double *rt = ws + lane * row;
      if (k < first + count) {
        const double sv = a.ps[k];
        if (sv != sv) {
          rt[0] = NAN;  // skipped point
        } else {
          const double zre = a.ux[k] - cx, zim = a.uy[k] - cy;
          double pre = 1, pim = 0;
          rt[0] = sv;
          rt[q] = 0;
#pragma unroll 8
          for (uint32_t o = 1; o < q; ++o) {
            const double nre = pre * zre - pim * zim;
            const double nim = pre * zim + pim * zre;
            pre = nre;
            pim = nim;
            rt[o] = sv * pre;
            rt[q + o] = sv * pim;
          }
        }
      }
      __syncwarp();
#pragma unroll 4
      for (uint32_t t = 0; t < np; ++t) {
        const double *ot = ws + t * row;
        const double sv = ot[0];
        if (sv != sv) continue;
        if (r0 < stride && r0 != q) acc0 += ot[r0];
        if (r1 < stride && r1 != q) acc1 += ot[r1];
      }
      __syncwarp();
    }
    store_sums(a, c, q, r0, acc0);
    store_sums(a, c, q, r1, acc1);
  }
  const uint32_t S = 32 / q, nn = lane % q;
  double bn[P + 1];  // the lane's row of the binomials, on its way during the first wait
  if (P) {
#pragma unroll
    for (uint32_t k = 0; k <= P; ++k) bn[k] = a.tab->binom[nn * FMM_TAB + k];
  }
  while (c != 0) {
    const uint32_t parent = a.cells[c].parent;
    const uint32_t nchild = a.cells[parent].nchild, child0 = a.cells[parent].child0;
    __threadfence();
    __syncwarp();
    uint32_t before = 0;
    if (lane == 0) before = atomicAdd(&a.arrive[parent], 1u);
    if (__shfl_sync(0xffffffffu, before, 0) + 1 != nchild) return;
    __threadfence();
    c = parent;
    // the box: lane j holds child j's
    double b0 = 0, b1 = 0, b2 = 0, b3 = 0, ccx = 0, ccy = 0;
    if (lane < nchild) {
      const uint32_t ch = child0 + lane;
      b0 = ldg_cg(&a.bx0[ch]); b1 = ldg_cg(&a.by0[ch]);
      b2 = ldg_cg(&a.bx1[ch]); b3 = ldg_cg(&a.by1[ch]);
      ccx = ldg_cg(&a.cells[ch].cx); ccy = ldg_cg(&a.cells[ch].cy);
    }
    double *Ms = ws, *pw = ws + 4 * stride, *Cs = ws + 8 * stride;
    for (uint32_t idx = lane; idx < nchild * stride; idx += 32) {
      double *m = a.mco + (size_t)child0 * stride + idx;
      const uint32_t o = idx % q;  // stride is 2 q
      const double v = ldg_cg(m);
      Ms[idx] = v;
      if (o >= 2) *m = v * a.tab->ifact[o];
    }
    double x0 = INFINITY, y0 = INFINITY, x1 = -INFINITY, y1 = -INFINITY;
    for (uint32_t j = 0; j < nchild; ++j) {
      x0 = zmin(x0, __shfl_sync(0xffffffffu, b0, j));
      y0 = zmin(y0, __shfl_sync(0xffffffffu, b1, j));
      x1 = zmax(x1, __shfl_sync(0xffffffffu, b2, j));
      y1 = zmax(y1, __shfl_sync(0xffffffffu, b3, j));
    }
    const double cx = (x0 + x1) / 2, cy = (y0 + y1) / 2;
    if (lane == 0) write_box(a, c, x0, y0, x1, y1, cx, cy);
    if (lane < nchild) shift_powers(ccx - cx, ccy - cy, p, pw + lane * stride);
    __syncwarp();
    // M2M (fmm.zig:782-806): lane (child, nn) its sum over k, then lane r the
    // children in order
    for (uint32_t j = lane / q; j < nchild && lane < S * q; j += S) {
      const double *cre = Ms + j * stride, *cim = cre + q, *w = pw + j * stride;
      double sre = 0, sim = 0;
#pragma unroll
      for (uint32_t k = 0; k < (P ? P + 1 : nn + 1); ++k) {
        if (k > nn) continue;
        const double b = P ? bn[P ? k : 0] : a.tab->binom[nn * FMM_TAB + k];
        const double xre = cre[k] * b, xim = cim[k] * b;
        sre += xre * w[nn - k] - xim * w[q + nn - k];
        sim += xre * w[q + nn - k] + xim * w[nn - k];
      }
      Cs[j * stride + nn] = sre;
      Cs[j * stride + q + nn] = sim;
    }
    __syncwarp();
    for (uint32_t r = lane; r < stride; r += 32) {
      double acc = 0;
      for (uint32_t j = 0; j < nchild; ++j) acc += Cs[j * stride + r];
      store_sums(a, c, q, r, acc);
    }
    __syncwarp();
  }
}

// ---- interaction lists (fmm.zig:400-453) -------------------------------------------

// Expands one call (A, b) of cell c = A with the recursion's order: splits of
// B are followed at once, depth first. WRITE false: counts only (nm, np, nf
// are added to); WRITE true: the events are written from om / op / of on.
// Returns false if the local stack overflowed.
template <bool WRITE>
__device__ bool expand_call(const FmmArgs &a, uint32_t c, const FCell &A, uint32_t b, uint32_t &nm,
                            uint32_t &np, uint32_t &nf, uint32_t om, uint32_t op, uint32_t of) {
  uint32_t stack[FMM_STACK];
  const bool la = A.nchild == 0;
  uint32_t sp = 0;
  stack[sp++] = b;
  while (sp) {
    const uint32_t B = stack[--sp];
    if (B == c) {
      if (la) {
        if (WRITE) a.p2p[op + np] = c;
        ++np;
      } else {
        for (uint32_t j = 0; j < A.nchild; ++j) {
          if (WRITE) a.fwd[of + nf] = A.child0 + j;
          ++nf;
        }
      }
      continue;
    }
    const FCell Bc = a.cells[B];
    const double ra = A.r, rb = Bc.r;
    const double dx = A.cx - Bc.cx, dy = A.cy - Bc.cy;
    const double d2 = dx * dx + dy * dy;
    const double rmax = zmax(ra, rb), rmin = zmin(ra, rb);
    const double thr = a.mac_far * rmax + rmin;
    if (d2 > FMM_MIN_SEP2 && d2 >= thr * thr) {
      bool separated = true;
      if (a.ring) {
        const double gap = sqrt(d2) - ra - rb;
        if (gap >= a.dmax_scaled) continue;
        if (gap + 2 * (ra + rb) > a.dmax_scaled || gap < a.dmin_scaled) separated = false;
      }
      if (separated) {
        if (WRITE) a.m2l[om + nm] = B;
        ++nm;
        continue;
      }
    }
    const bool lb = Bc.nchild == 0;
    if (la && lb) {
      if (WRITE) a.p2p[op + np] = B;
      ++np;
    } else if (la || (!lb && rb > ra)) {
      if (sp + Bc.nchild > FMM_STACK) return false;
      for (uint32_t j = Bc.nchild; j-- > 0;) stack[sp++] = Bc.child0 + j;
    } else {
      if (WRITE) a.fwd[of + nf] = B;
      ++nf;
    }
  }
  return true;
}

__device__ inline unsigned long long fmm_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ inline uint32_t ld_acquire(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ inline void st_release(uint32_t *p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ inline uint32_t warp_excl(uint32_t v, uint32_t &total) {
  const unsigned lane = threadIdx.x & 31;
  uint32_t incl = v;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (unsigned)o) incl += y;
  }
  total = __shfl_sync(0xffffffffu, incl, 31);
  return incl - v;
}

// A cell in three 16-byte loads.
__device__ inline FCell load_cell(const FCell *p) {
  union {
    uint4 w[3];
    FCell c;
  } u;
#pragma unroll
  for (int i = 0; i < 3; ++i) u.w[i] = reinterpret_cast<const uint4 *>(p)[i];
  return u.c;
}

// What cell c's call with B comes to: an event, B's children in its place
// (n of them from v), or nothing. The decision of expand_call above.
constexpr uint32_t EV_CALL = 0, EV_M2L = 1u << 30, EV_P2P = 2u << 30, EV_FWD = 3u << 30;
constexpr uint32_t EV_CELL = EV_M2L - 1;

__device__ inline uint32_t decide_call(const FmmArgs &a, uint32_t c, const FCell &A, uint32_t B,
                                       uint32_t &v) {
  const bool la = A.nchild == 0;
  if (B == c) {
    v = la ? c | EV_P2P : A.child0 | EV_FWD;
    return la ? 1 : A.nchild;
  }
  const FCell Bc = load_cell(a.cells + B);
  const double ra = A.r, rb = Bc.r;
  const double dx = A.cx - Bc.cx, dy = A.cy - Bc.cy;
  const double d2 = dx * dx + dy * dy;
  const double rmax = zmax(ra, rb), rmin = zmin(ra, rb);
  const double thr = a.mac_far * rmax + rmin;
  if (d2 > FMM_MIN_SEP2 && d2 >= thr * thr) {
    bool separated = true;
    if (a.ring) {
      const double gap = sqrt(d2) - ra - rb;
      if (gap >= a.dmax_scaled) return 0;
      if (gap + 2 * (ra + rb) > a.dmax_scaled || gap < a.dmin_scaled) separated = false;
    }
    if (separated) {
      v = B | EV_M2L;
      return 1;
    }
  }
  const bool lb = Bc.nchild == 0;
  if (la && lb) {
    v = B | EV_P2P;
    return 1;
  }
  if (la || (!lb && rb > ra)) {
    v = Bc.child0;
    return Bc.nchild;
  }
  v = B | EV_FWD;
  return 1;
}

// Reserves cell c's places in the pools; false if they do not fit.
__device__ bool reserve_lists(const FmmArgs &a, uint32_t c, uint32_t tm, uint32_t tp, uint32_t tf,
                              uint32_t &om, uint32_t &op, uint32_t &of) {
  const unsigned lane = threadIdx.x & 31;
  uint32_t at = 0;
  if (lane < 3) {
    const uint32_t t = lane == 0 ? tm : lane == 1 ? tp : tf;
    if (t) at = atomicAdd(&a.info[FI_POOL_M2L + lane], t);
    (lane == 0 ? a.m2l_off : lane == 1 ? a.p2p_off : a.fwd_off)[c] = at;
    if (lane < 2) (lane == 0 ? a.m2l_cnt : a.p2p_cnt)[c] = t;
  }
  om = __shfl_sync(0xffffffffu, at, 0);
  op = __shfl_sync(0xffffffffu, at, 1);
  of = __shfl_sync(0xffffffffu, at, 2);
  if ((size_t)om + tm > a.cap_m2l || (size_t)op + tp > a.cap_p2p || (size_t)of + tf > a.cap_fwd) {
    if (lane == 0) atomicOr(&a.info[FI_LIST_OVERFLOW], 1u);
    return false;
  }
  return true;
}

// The calls of cell c (`in`, in order; null: (root, root)) by one warp, where
// their expansion passes the shared lists: lane k expands calls k, k + 32, ...
// depth first; each call's events are placed after those of the calls before
// it (a warp scan of the counts). Counts, then a reservation in the pools, then
// counts again and the writes. Returns the forward list's length; tp the P2P
// list's.
__device__ uint32_t expand_long(const FmmArgs &a, uint32_t c, const FCell &A, const uint32_t *in,
                                uint32_t nin, uint32_t &tp) {
  const unsigned lane = threadIdx.x & 31;
  uint32_t tm = 0, tf = 0;
  tp = 0;
  bool ok = true;
  for (uint32_t u0 = 0; u0 < nin; u0 += 32) {
    const uint32_t u = u0 + lane;
    uint32_t nm = 0, np = 0, nf = 0;
    if (u < nin && !expand_call<false>(a, c, A, in ? ldg_cg(&in[u]) : 0, nm, np, nf, 0, 0, 0)) ok = false;
    uint32_t t;
    warp_excl(nm, t); tm += t;
    warp_excl(np, t); tp += t;
    warp_excl(nf, t); tf += t;
  }
  ok = __all_sync(0xffffffffu, ok);
  if (!ok) {
    tm = tp = tf = 0;
    if (lane == 0) atomicOr(&a.info[FI_LIST_OVERFLOW], 2u);
  }
  uint32_t om, op, of;
  if (!reserve_lists(a, c, tm, tp, tf, om, op, of) || !ok) return 0;
  for (uint32_t u0 = 0; u0 < nin; u0 += 32) {
    const uint32_t u = u0 + lane;
    const uint32_t b = u < nin && in ? ldg_cg(&in[u]) : 0;
    uint32_t nm = 0, np = 0, nf = 0;
    if (u < nin) expand_call<false>(a, c, A, b, nm, np, nf, 0, 0, 0);
    uint32_t t0, t1, t2;
    const uint32_t xm = warp_excl(nm, t0), xp = warp_excl(np, t1), xf = warp_excl(nf, t2);
    if (u < nin) {
      uint32_t wm = 0, wp = 0, wf = 0;
      expand_call<true>(a, c, A, b, wm, wp, wf, om + xm, op + xp, of + xf);
    }
    om += t0;
    op += t1;
    of += t2;
  }
  return tf;
}

// The same in shared memory: the calls as one ordered list, and in each round
// every call in it (a lane each) is replaced by what it comes to, until only
// events are left. Each cell is read once, by as many lanes as there are calls;
// the depth-first form reads it three times, in one lane's chain of dependent
// loads a call. `buf` holds two lists of LIST_CAP words; a longer list (a leaf
// beside a far denser region) takes the depth-first form. LIST_CAP 256 / 512 /
// 1,024: a tick of 200,003 clustered nodes 985 / 992 / 737 us, of 80,000 in
// tighter clusters 944 / 946 / 637 (their lists pass 512); 6,000 to 80,000
// clustered or even nodes the same.
constexpr uint32_t LIST_CAP = 512;
__device__ uint32_t expand_cell(const FmmArgs &a, uint32_t c, const FCell &A, const uint32_t *in,
                                uint32_t nin, uint32_t *buf, uint32_t &tp) {
  const unsigned lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1;
  if (nin > LIST_CAP) return expand_long(a, c, A, in, nin, tp);
  for (uint32_t u = lane; u < nin; u += 32) buf[u] = in ? ldg_cg(&in[u]) : 0;
  __syncwarp();
  uint32_t cnt = nin, tm = 0;
  uint32_t *src = buf, *dst = buf + LIST_CAP;
  for (bool more = true; more;) {
    more = false;
    tm = tp = 0;
    uint32_t out = 0;
    for (uint32_t w0 = 0; w0 < cnt; w0 += 32) {
      uint32_t k = 0, v = 0;
      if (w0 + lane < cnt) {
        v = src[w0 + lane];
        k = 1;
        if (v < EV_M2L) k = decide_call(a, c, A, v, v);
      }
      const unsigned b0 = __ballot_sync(0xffffffffu, k & 1), b1 = __ballot_sync(0xffffffffu, k & 2),
                     b2 = __ballot_sync(0xffffffffu, k & 4);
      const uint32_t at = out + __popc(b0 & lt) + 2 * __popc(b1 & lt) + 4 * __popc(b2 & lt);
      out += __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
      if (out > LIST_CAP) return expand_long(a, c, A, in, nin, tp);
      for (uint32_t j = 0; j < k; ++j) dst[at + j] = v + j;
      const uint32_t type = v & ~EV_CELL;
      tm += __popc(__ballot_sync(0xffffffffu, k && type == EV_M2L));
      tp += __popc(__ballot_sync(0xffffffffu, k && type == EV_P2P));
      if (__any_sync(0xffffffffu, k && type == EV_CALL)) more = true;
    }
    __syncwarp();
    cnt = out;
    uint32_t *t = src; src = dst; dst = t;
  }
  const uint32_t tf = cnt - tm - tp;
  uint32_t om, op, of;
  if (!reserve_lists(a, c, tm, tp, tf, om, op, of)) return 0;
  for (uint32_t w0 = 0; w0 < cnt; w0 += 32) {
    const uint32_t v = w0 + lane < cnt ? src[w0 + lane] : 0;
    const uint32_t type = v & ~EV_CELL;
    const unsigned bm = __ballot_sync(0xffffffffu, type == EV_M2L),
                   bp = __ballot_sync(0xffffffffu, type == EV_P2P),
                   bf = __ballot_sync(0xffffffffu, type == EV_FWD);
    if (type == EV_M2L) a.m2l[om + __popc(bm & lt)] = v & EV_CELL;
    if (type == EV_P2P) a.p2p[op + __popc(bp & lt)] = v & EV_CELL;
    if (type == EV_FWD) a.fwd[of + __popc(bf & lt)] = v & EV_CELL;
    om += __popc(bm);
    op += __popc(bp);
    of += __popc(bf);
  }
  return tf;
}

// A leaf with a long P2P list (tp > LONG_LIST): its units, if they fit;
// long_at[c] = the first.
__device__ void plan_long(const FmmArgs &a, uint32_t c, uint32_t count, uint32_t tp) {
  const unsigned lane = threadIdx.x & 31;
  uint32_t at = NONE;
  if (count <= LONG_POINTS) {
    const uint32_t per = count <= 16 ? 1 : 2;  // units an item: targets in lanes / 16
    const uint32_t items = (tp + 31) / 32 * ((count + 31) / 32), units = items * per;
    if (lane == 0) at = atomicAdd(&a.info[FI_LONG_UNITS], units);
    at = __shfl_sync(0xffffffffu, at, 0);
    const bool fits = (size_t)at + units <= a.long_cap;
    for (uint32_t j = lane; j < units; j += 32)
      if ((size_t)at + j < a.long_cap)
        a.long_items[at + j] = make_uint2(fits && j % per == 0 ? c : NONE, j / per);
    if (!fits) at = NONE;
    else if (lane == 0) a.longs[atomicAdd(&a.info[FI_LONGS], 1u)] = c;
  }
  if (lane == 0) a.long_at[c] = at;
}

// A warp per cell, in level order (blocks numbered as they start, so a block's
// cells wait only for cells of running blocks): a cell waits for its parent's
// forward list (`fwd_cnt`, NONE until the list is there) and no level waits as
// a whole. With a grid barrier a level and the depth-first form 6,000 nodes
// took 174 us (now 37), 1 M 584 us (now 151). A wait ends after 20 ms in which
// no counted cell was finished (the first 1,024 and every 64th: a count of all
// would be a chain of atomics on one word); the lists are then built again with
// a launch a level (by_level), whose cells find their parents' lists there.
__global__ void __launch_bounds__(LISTS_THREADS) k_fmm_lists(FmmArgs a, uint32_t c0, uint32_t c1) {
  __shared__ uint32_t buf[LISTS_THREADS / 32][2 * LIST_CAP];
  __shared__ uint32_t ticket;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) ticket = a.by_level ? blockIdx.x : atomicAdd(&a.info[FI_TICKET], 1u);
  __syncthreads();
  const uint32_t c = c0 + ticket * (LISTS_THREADS / 32) + warp;
  if (c >= c1) return;
  const FCell A = load_cell(a.cells + c);
  const uint32_t *in = nullptr;
  uint32_t nin = 1;
  if (c != 0) {
    if (lane == 0) {
      nin = ld_acquire(&a.fwd_cnt[A.parent]);
      if (nin == NONE) {
        unsigned long long t0 = fmm_timer_ns();
        uint32_t seen = ld_acquire(&a.info[FI_DONE]);
        while ((nin = ld_acquire(&a.fwd_cnt[A.parent])) == NONE) {
          if (fmm_timer_ns() - t0 > a.wait_ns) {
            const uint32_t done = ld_acquire(&a.info[FI_DONE]);
            if (done == seen) {
              atomicOr(&a.info[FI_LIST_OVERFLOW], 4u);
              nin = 0;
              break;
            }
            seen = done;
            t0 = fmm_timer_ns();
          }
          __nanosleep(64);
        }
      }
    }
    nin = __shfl_sync(0xffffffffu, nin, 0);
    in = a.fwd + (nin ? ldg_cg(&a.fwd_off[A.parent]) : 0);
  }
  uint32_t tp = 0;
  const uint32_t tf = expand_cell(a, c, A, in, nin, buf[warp], tp);
  if (A.nchild) {
    __threadfence();
    __syncwarp();
    if (lane == 0) st_release(&a.fwd_cnt[c], tf);
  } else if (tp > LONG_LIST) {
    plan_long(a, c, A.count, tp);
    if (lane == 0) atomicMax(&a.info[FI_LONG_MAX], tp);
  }
  if (lane == 0 && (c < 1024 || (c & 63) == 0)) atomicAdd(&a.info[FI_DONE], 1u);
}

// ---- M2L (fmm.zig:561-610) and the unscale of L (fmm.zig:645-657) --------------------

// A warp per cell. The powers T of 32 sources' offsets at a time, a lane per
// source; then per source M2L_R of the q outputs a lane, so that a T and an M
// read from shared memory (both as (re, im) pairs) feed M2L_R multiplications
// and S = 32 / ceil(q / M2L_R) sources run side by side; then a lane per real
// adds the sources in order. One output a lane and three sources at a time,
// three lanes busy in the powers, were bound by shared-memory reads and by those
// idle lanes: 1 M nodes 731 -> 256 us, 6,000 36 -> 10 us.
constexpr uint32_t M2L_R = 3;
__host__ __device__ constexpr uint32_t m2l_lanes(uint32_t q) { return (q + M2L_R - 1) / M2L_R; }
__host__ __device__ constexpr uint32_t m2l_side(uint32_t q) { return 32 / m2l_lanes(q); }
__host__ __device__ constexpr uint32_t m2l_chunk(uint32_t q) { return 32 / m2l_side(q) * m2l_side(q); }
// doubles a warp: T (and a lane's reads past the last row), M, C
__host__ __device__ constexpr uint32_t m2l_words(uint32_t q) {
  return 2 * (m2l_chunk(q) * (2 * q - 1) + 2 * M2L_R) + 4 * m2l_side(q) * q;
}

template <uint32_t P>
__global__ void __launch_bounds__(M2L_THREADS, 18) k_fmm_m2l(FmmArgs a) {
  extern __shared__ __align__(16) double fmm_smem[];
  if (a.info[FI_LIST_OVERFLOW]) return;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t p = P ? P : a.p, q = p + 1, stride = 2 * q, nt = 2 * p + 1;
  const uint32_t G = m2l_lanes(q), S = m2l_side(q), CH = m2l_chunk(q);
  double2 *T = reinterpret_cast<double2 *>(fmm_smem + (size_t)warp * m2l_words(q));
  double2 *M = T + CH * nt + 2 * M2L_R;
  double *C = reinterpret_cast<double *>(M + S * q);
  const uint32_t s = lane / G, l0 = lane % G * M2L_R;
  const uint32_t c = blockIdx.x * (M2L_THREADS / 32) + warp;
  if (c >= a.ncells) return;
  const double acx = a.cells[c].cx, acy = a.cells[c].cy;
  const uint32_t cnt = a.m2l_cnt[c], off = a.m2l_off[c];
  double acc0 = 0, acc1 = 0;
  for (uint32_t base = 0; base < cnt; base += CH) {
    const uint32_t nc = min(CH, cnt - base);
    uint32_t B = 0;
    if (lane < nc) {
      B = a.m2l[off + base + lane];
      const double dx = acx - a.cells[B].cx, dy = acy - a.cells[B].cy;
      const double d2 = dx * dx + dy * dy;
      const double ire = dx / d2, iim = -dy / d2;
      double are = ire, aim = iim;
      double2 *t = T + lane * nt;
      t[0] = make_double2(are, aim);
#pragma unroll
      for (uint32_t mm = 1; mm < (P ? 2 * P + 1 : nt); ++mm) {
        const double nre = are * ire - aim * iim;
        const double nim = are * iim + aim * ire;
        are = nre;
        aim = nim;
        const double f = a.tab->fact[mm];
        t[mm] = make_double2(are * f, aim * f);
      }
    }
    // a round's multipoles: real idx of S x stride a lane, the next round's
    // (default order) loaded while this one's are multiplied
    constexpr uint32_t LOADS = P ? (m2l_side(P + 1) * 2 * (P + 1) + 31) / 32 : 1;
    double next[LOADS];
    auto load = [&](uint32_t r0, uint32_t i) {
      const uint32_t ss = (i * 32 + lane) / stride, r = (i * 32 + lane) % stride;
      const uint32_t Bs = __shfl_sync(0xffffffffu, B, (r0 + ss) & 31);
      return ss < S && r0 + ss < nc ? a.mco[(size_t)Bs * stride + r] : 0.0;
    };
    auto put = [&](uint32_t i, double v) {
      const uint32_t ss = (i * 32 + lane) / stride, r = (i * 32 + lane) % stride;
      if (ss < S) reinterpret_cast<double *>(M + ss * q + r % q)[r / q] = v;
    };
    if (P) {
#pragma unroll
      for (uint32_t i = 0; i < LOADS; ++i) next[i] = load(0, i);
    }
    for (uint32_t r0 = 0; r0 < nc; r0 += S) {
      const uint32_t ns = min(S, nc - r0);
      if (P) {
#pragma unroll
        for (uint32_t i = 0; i < LOADS; ++i) {
          put(i, next[i]);
          next[i] = load(r0 + S, i);
        }
      } else {
        for (uint32_t i = 0; i * 32 < ns * stride; ++i) put(i, load(r0, i));
      }
      __syncwarp();
      if (s < ns) {
        const double2 *t = T + (r0 + s) * nt + l0, *m = M + s * q;
        double vre[2][M2L_R], vim[2][M2L_R];
        double2 w[M2L_R];
#pragma unroll
        for (uint32_t j = 0; j < M2L_R; ++j) {
          vre[0][j] = vre[1][j] = vim[0][j] = vim[1][j] = 0;
          w[j] = t[j];
        }
        uint32_t k = 0;
#pragma unroll
        for (; k + 2 <= (P ? P + 1 : q); k += 2) {
#pragma unroll
          for (uint32_t h = 0; h < 2; ++h) {
            const double2 mk = m[k + h];
#pragma unroll
            for (uint32_t j = 0; j < M2L_R; ++j) {
              vre[h][j] += mk.x * w[j].x - mk.y * w[j].y;
              vim[h][j] += mk.x * w[j].y + mk.y * w[j].x;
            }
#pragma unroll
            for (uint32_t j = 0; j + 1 < M2L_R; ++j) w[j] = w[j + 1];
            w[M2L_R - 1] = t[k + h + M2L_R];
          }
        }
#pragma unroll
        for (uint32_t j = 0; j < M2L_R; ++j) {
          double sre = vre[0][j] + vre[1][j], sim = vim[0][j] + vim[1][j];
          if (k < q) {
            const double2 mk = m[k];
            sre += mk.x * w[j].x - mk.y * w[j].y;
            sim += mk.x * w[j].y + mk.y * w[j].x;
          }
          if (l0 + j < q) {
            C[s * stride + l0 + j] = sre;
            C[s * stride + q + l0 + j] = sim;
          }
        }
      }
      __syncwarp();
#pragma unroll 4
      for (uint32_t t = 0; t < ns; ++t) {
        if (lane < stride) acc0 += C[t * stride + lane];
        if (lane + 32 < stride) acc1 += C[t * stride + lane + 32];
      }
      __syncwarp();
    }
  }
  double *L = a.lco + (size_t)c * stride;
  for (uint32_t r = lane; r < stride; r += 32) {
    const uint32_t l = r % q;
    const double inv = ((l & 1) ? -1.0 : 1.0) / a.tab->fact[l];
    L[r] = (r < 32 ? acc0 : acc1) * inv;
  }
}

// ---- P2P (fmm.zig:477-553) ------------------------------------------------------------

// One pair's term, or false where it has none.
__device__ inline bool pair_term(const FmmArgs &a, uint64_t seed, uint32_t ti, uint32_t tj, double sj,
                                 double xj, double yj, double xi, double yi, double &tx, double &ty) {
  if (tj == ti) return false;
  double x = xj - xi, y = yj - yi;
  double l = x * x + y * y;
  if (l >= a.dmax2) return false;
  if (x == 0 || y == 0) {
    const uint32_t i = a.perm[ti], j = a.perm[tj];
    if (x == 0) { x = hash_jiggle(seed, i, j, 0); l += x * x; }
    if (y == 0) { y = hash_jiggle(seed, i, j, 1); l += y * y; }
  }
  if (l < a.dmin2) l = sqrt(a.dmin2 * l);
  const double wj = sj / l;
  tx = x * wj;
  ty = y * wj;
  return true;
}

// The points of a source leaf, up to 32 at a time, in a warp's shared memory.
struct Sources {
  double x[32], y[32], s[32];
};

// Four pairs of a target by one division, on two lanes (sum 0: k, k + 2; sum 1:
// k + 1, k + 3); false, with nothing added, if they have to go one by one.
__device__ inline bool group_four(const FmmArgs &a, uint32_t ti, uint32_t b0, uint32_t k,
                                  const Sources &src, double xi, double yi, double &ax0, double &ay0,
                                  double &ax1, double &ay1) {
  const double xa0 = src.x[k] - xi, xa1 = src.x[k + 1] - xi;
  const double ya0 = src.y[k] - yi, ya1 = src.y[k + 1] - yi;
  const double xb0 = src.x[k + 2] - xi, xb1 = src.x[k + 3] - xi;
  const double yb0 = src.y[k + 2] - yi, yb1 = src.y[k + 3] - yi;
  const double la0 = xa0 * xa0 + ya0 * ya0, la1 = xa1 * xa1 + ya1 * ya1;
  const double lb0 = xb0 * xb0 + yb0 * yb0, lb1 = xb1 * xb1 + yb1 * yb1;
  const double z0 = xa0 * ya0 * xb0 * yb0, z1 = xa1 * ya1 * xb1 * yb1;
  const double mn = zmin(zmin(la0, lb0), zmin(la1, lb1));
  if (z0 == 0 || z1 == 0 || !(mn >= a.dmin2) || ti - (b0 + k) < 4) return false;
  const double pa = la0 * la1, pb = lb0 * lb1;
  const double inv = 1 / (pa * pb);
  double wa0 = src.s[k] * la1 * pb * inv, wa1 = src.s[k + 1] * la0 * pb * inv;
  double wb0 = src.s[k + 2] * lb1 * pa * inv, wb1 = src.s[k + 3] * lb0 * pa * inv;
  if (a.has_dmax) {
    if (!(la0 < a.dmax2)) wa0 = 0;
    if (!(la1 < a.dmax2)) wa1 = 0;
    if (!(lb0 < a.dmax2)) wb0 = 0;
    if (!(lb1 < a.dmax2)) wb1 = 0;
  }
  ax0 += xa0 * wa0 + xb0 * wb0;
  ax1 += xa1 * wa1 + xb1 * wb1;
  ay0 += ya0 * wa0 + yb0 * wb0;
  ay1 += ya1 * wa1 + yb1 * wb1;
  return true;
}

// A target's sums within one source leaf: its groups of four, pairs that cannot
// go that way added to the velocity one by one. One thread has both sums; `b0`
// is the chunk's first point.
__device__ inline void leaf_one(const FmmArgs &a, uint64_t seed, uint32_t ti, uint32_t b0, uint32_t cn,
                                const Sources &src, double xi, double yi, double &vx, double &vy,
                                double &ax0, double &ay0, double &ax1, double &ay1) {
  uint32_t k = 0;
  for (; k + 4 <= cn; k += 4) {
    if (group_four(a, ti, b0, k, src, xi, yi, ax0, ay0, ax1, ay1)) continue;
#pragma unroll 1
    for (uint32_t u = 0; u < 4; ++u) {
      double tx, ty;
      if (pair_term(a, seed, ti, b0 + k + u, src.s[k + u], src.x[k + u], src.y[k + u], xi, yi, tx, ty)) {
        vx += tx;
        vy += ty;
      }
    }
  }
#pragma unroll 1
  for (; k < cn; ++k) {
    double tx, ty;
    if (pair_term(a, seed, ti, b0 + k, src.s[k], src.x[k], src.y[k], xi, yi, tx, ty)) {
      vx += tx;
      vy += ty;
    }
  }
}

// Pairs [k, k + np), np <= 4, of a target that LANES neighbouring lanes hold
// (all keep the whole velocity): each takes every LANES-th pair, the terms are
// added in order. Every lane of the warp calls it; `mine` says whose terms count.
template <uint32_t LANES>
__device__ inline void pairs_many(const FmmArgs &a, uint64_t seed, uint32_t ti, uint32_t b0, uint32_t k,
                                  uint32_t np, const Sources &src, double xi, double yi, bool mine,
                                  double &vx, double &vy) {
  constexpr uint32_t PER = 4 / LANES;
  const uint32_t lane = threadIdx.x & 31, r = lane % LANES, l0 = lane - r;
  double tx[PER], ty[PER];
  uint32_t has = 0;
#pragma unroll
  for (uint32_t i = 0; i < PER; ++i) {
    const uint32_t u = i * LANES + r, j = (k + u) & 31;
    tx[i] = ty[i] = 0;
    if (mine && u < np &&
        pair_term(a, seed, ti, b0 + j, src.s[j], src.x[j], src.y[j], xi, yi, tx[i], ty[i]))
      has |= 1u << u;
  }
#pragma unroll
  for (uint32_t o = 1; o < LANES; o <<= 1) has |= __shfl_xor_sync(0xffffffffu, has, o);
#pragma unroll
  for (uint32_t u = 0; u < 4; ++u) {
    const double x = __shfl_sync(0xffffffffu, tx[u / LANES], l0 + u % LANES),
                 y = __shfl_sync(0xffffffffu, ty[u / LANES], l0 + u % LANES);
    if (has >> u & 1u) {
      vx += x;
      vy += y;
    }
  }
}

// leaf_one for a target that LANES neighbouring lanes hold: LANES / 2 groups of
// four pairs at a time, a lane per group and sum; both sums are kept by every
// second lane, the groups' terms added in order. (The pairs that go to the
// velocity one by one do not meet the sums before the leaf ends.)
template <uint32_t LANES>
__device__ inline void leaf_many(const FmmArgs &a, uint64_t seed, uint32_t ti, uint32_t b0, uint32_t cn,
                                 const Sources &src, double xi, double yi, double &vx, double &vy,
                                 double &ax, double &ay) {
  constexpr uint32_t G = LANES / 2;
  const uint32_t lane = threadIdx.x & 31, h = lane & 1, g = lane % LANES / 2, l0 = lane - lane % LANES;
  for (uint32_t k = 0; k + 4 <= cn; k += 4 * G) {
    const bool in = G == 1 || k + 4 * g + 4 <= cn;
    const uint32_t ja = in ? k + 4 * g + h : h, jb = ja + 2;
    const double xa = src.x[ja] - xi, ya = src.y[ja] - yi;
    const double xb = src.x[jb] - xi, yb = src.y[jb] - yi;
    const double la = xa * xa + ya * ya, lb = xb * xb + yb * yb;
    const double oa = __shfl_xor_sync(0xffffffffu, la, 1), ob = __shfl_xor_sync(0xffffffffu, lb, 1);
    const double z = xa * ya * xb * yb;
    const double mn = zmin(zmin(la, lb), zmin(oa, ob));
    int bad = z == 0 || !(mn >= a.dmin2) || ti - (b0 + k + 4 * g) < 4;
    bad |= __shfl_xor_sync(0xffffffffu, bad, 1);
    const double pa = la * oa, pb = lb * ob;
    const double inv = 1 / (pa * pb);
    double wa = src.s[ja] * oa * pb * inv, wb = src.s[jb] * ob * pa * inv;
    if (a.has_dmax) {
      if (!(la < a.dmax2)) wa = 0;
      if (!(lb < a.dmax2)) wb = 0;
    }
    const double tx = xa * wa + xb * wb, ty = ya * wa + yb * wb;
    if (G == 1) {
      if (!bad) {
        ax += tx;
        ay += ty;
      }
      if (__any_sync(0xffffffffu, bad))
        pairs_many<LANES>(a, seed, ti, b0, k, 4, src, xi, yi, bad, vx, vy);
    } else {
      const int state = in ? 1 + bad : 0;
#pragma unroll
      for (uint32_t gg = 0; gg < G; ++gg) {
        const uint32_t from = l0 + 2 * gg + h;
        const double x = __shfl_sync(0xffffffffu, tx, from), y = __shfl_sync(0xffffffffu, ty, from);
        const int st = __shfl_sync(0xffffffffu, state, from);
        if (st == 1) {
          ax += x;
          ay += y;
        }
        if (__any_sync(0xffffffffu, st == 2))
          pairs_many<LANES>(a, seed, ti, b0, k + 4 * gg, 4, src, xi, yi, st == 2, vx, vy);
      }
    }
  }
  if (cn & 3) pairs_many<LANES>(a, seed, ti, b0, cn & ~3u, cn & 3, src, xi, yi, true, vx, vy);
}

// A warp per leaf: the source leaves of its list one after another, the next
// one's points on their way into registers while this one's, in shared memory,
// are summed. A lane holds a target, or two lanes where the leaf has at most 16
// (six in ten leaves of evenly spread nodes: half the lanes were idle). Sources
// read from L2 as the sums went, a chain of three loads a source leaf, took 104
// us at 6,000 nodes (now 52) and 759 us at 1 M (now 620). FEW: four warps
// a leaf, eight targets each and four lanes a target, where the leaves do not
// fill the chip: shorter chains for a sixth more work. Against a lane or two a
// target, evenly spread / clustered (long lists included): 6,000 nodes 25 / 64
// us for 37 / 84; 20,000 39 / 150 for 35 / 200; 80,000 104 / 360 for 68 / 478.
template <bool FEW>
__global__ void __launch_bounds__(P2P_THREADS) k_fmm_p2p(FmmArgs a) {
  __shared__ Sources sources[P2P_THREADS / 32];
  if (a.info[FI_LIST_OVERFLOW]) return;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Sources &src = sources[warp];
  const uint64_t seed = (uint64_t)__double_as_longlong(*a.seed);
  const uint32_t gw = blockIdx.x * (P2P_THREADS / 32) + warp;
  const uint32_t c = FEW ? gw >> 2 : gw, skip = FEW ? (gw & 3) * 8 : 0;
  if (c >= a.ncells) return;
  const uint32_t cnt = a.p2p_cnt[c];
  if (!cnt || (cnt > LONG_LIST && a.long_at[c] != NONE)) return;
  const uint32_t off = a.p2p_off[c], first = a.cells[c].first, count = a.cells[c].count;
  const bool two = count <= 16;
  for (uint32_t base = first + skip; base < first + count; base += 32) {
    const uint32_t at = base + (FEW ? lane >> 2 : two ? lane >> 1 : lane);
    const bool live = at < first + count;
    const uint32_t ti = live ? at : first;
    const uint32_t i = a.perm[ti];
    const double xi = a.px[ti], yi = a.py[ti];
    double vx = a.vx[i], vy = a.vy[i];
    for (uint32_t e0 = 0; e0 < cnt; e0 += 32) {
      const uint32_t ne = min(32u, cnt - e0);
      uint32_t lb = 0, ln = 0;
      if (lane < ne) {
        const uint32_t B = a.p2p[off + e0 + lane];
        lb = a.cells[B].first;
        ln = a.cells[B].count;
      }
      uint32_t b0 = __shfl_sync(0xffffffffu, lb, 0), bn = __shfl_sync(0xffffffffu, ln, 0);
      double rx = 0, ry = 0, rs = 0;
      if (lane < bn) { rx = a.px[b0 + lane]; ry = a.py[b0 + lane]; rs = a.ps[b0 + lane]; }
      double ax0 = 0, ax1 = 0, ay0 = 0, ay1 = 0;
      for (uint32_t e = 0; e < ne;) {
        const uint32_t cb = b0, cn = min(32u, bn);
        __syncwarp();
        src.x[lane] = rx;
        src.y[lane] = ry;
        src.s[lane] = rs;
        __syncwarp();
        const bool ends = bn <= 32;  // this source leaf ends with this chunk
        if (ends) {
          ++e;
          b0 = __shfl_sync(0xffffffffu, lb, e & 31);
          bn = __shfl_sync(0xffffffffu, ln, e & 31);
        } else {
          b0 += 32;
          bn -= 32;
        }
        if (e < ne && lane < bn) { rx = a.px[b0 + lane]; ry = a.py[b0 + lane]; rs = a.ps[b0 + lane]; }
        if (FEW) leaf_many<4>(a, seed, ti, cb, cn, src, xi, yi, vx, vy, ax0, ay0);
        else if (two) leaf_many<2>(a, seed, ti, cb, cn, src, xi, yi, vx, vy, ax0, ay0);
        else leaf_one(a, seed, ti, cb, cn, src, xi, yi, vx, vy, ax0, ay0, ax1, ay1);
        if (ends) {
          if (FEW || two) {
            ax1 = __shfl_xor_sync(0xffffffffu, ax0, 1);
            ay1 = __shfl_xor_sync(0xffffffffu, ay0, 1);
          }
          vx += ax0 + ax1;
          vy += ay0 + ay1;
          ax0 = ax1 = ay0 = ay1 = 0;
        }
      }
    }
    if (live && (FEW ? lane % 4 == 0 : !two || lane % 2 == 0)) {
      a.vx[i] = vx;
      a.vy[i] = vy;
    }
  }
}

// Long lists. A target's velocity is a chain over all pairs of its list, but
// within a source leaf the chain's terms do not depend on the velocity: the sums
// of the groups of four, after up to three pairs of their own. So a warp per
// segment of 32 source leaves writes every leaf's terms (a pair without a term
// writes -0, which changes nothing), and a warp per leaf then adds them in
// order; a source leaf with groups that go pair by pair (`long_flags`, a bit a
// leaf of the segment) is summed there as before. Where this pays, and what it
// measured: at LONG_WORTH.
constexpr unsigned LONG_THREADS = 64, LONG_BLOCKS = 2368;

__global__ void __launch_bounds__(LONG_THREADS) k_fmm_p2p_terms(FmmArgs a) {
  __shared__ Sources sources[LONG_THREADS / 32];
  if (a.info[FI_LIST_OVERFLOW]) return;
  const unsigned lane = threadIdx.x & 31;
  Sources &src = sources[threadIdx.x >> 5];
  const uint64_t seed = (uint64_t)__double_as_longlong(*a.seed);
  const uint32_t units = min(a.info[FI_LONG_UNITS], a.long_cap);
  for (uint32_t u = (blockIdx.x * LONG_THREADS + threadIdx.x) >> 5; u < units;
       u += gridDim.x * LONG_THREADS >> 5) {
    const uint2 item = a.long_items[u];
    const uint32_t c = item.x;
    if (c == NONE) continue;
    const uint32_t cnt = a.p2p_cnt[c], off = a.p2p_off[c];
    const uint32_t first = a.cells[c].first, count = a.cells[c].count;
    const uint32_t nseg = (cnt + 31) / 32, chunk = item.y / nseg, e0 = item.y % nseg * 32;
    const uint32_t wide = count <= 16 ? 16 : 32;
    const uint32_t at = first + chunk * 32 + lane;
    const bool live = at < first + count;  // (lanes past `wide` are not)
    const uint32_t ti = live ? at : first;
    const double xi = a.px[ti], yi = a.py[ti];
    double2 *terms = a.long_terms + (size_t)u * LONG_UNIT;
    const uint32_t ne = min(32u, cnt - e0);
    uint32_t lb = 0, ln = 0;
    if (lane < ne) {
      const uint32_t B = a.p2p[off + e0 + lane];
      lb = a.cells[B].first;
      ln = a.cells[B].count;
    }
    uint32_t flags = 0;
    uint32_t b0 = __shfl_sync(0xffffffffu, lb, 0), bn = __shfl_sync(0xffffffffu, ln, 0);
    double rx = 0, ry = 0, rs = 0;
    if (lane < bn) { rx = a.px[b0 + lane]; ry = a.py[b0 + lane]; rs = a.ps[b0 + lane]; }
    for (uint32_t e = 0; e < ne; ++e) {
      const uint32_t cb = b0, cn = bn;
      __syncwarp();
      src.x[lane] = rx;
      src.y[lane] = ry;
      src.s[lane] = rs;
      __syncwarp();
      b0 = __shfl_sync(0xffffffffu, lb, (e + 1) & 31);
      bn = __shfl_sync(0xffffffffu, ln, (e + 1) & 31);
      if (e + 1 < ne && lane < bn) { rx = a.px[b0 + lane]; ry = a.py[b0 + lane]; rs = a.ps[b0 + lane]; }
      if (cn > 32) {
        flags |= 1u << e;
        continue;
      }
      double ax0 = 0, ax1 = 0, ay0 = 0, ay1 = 0;
      bool bad = false;
      uint32_t k = 0;
      for (; k + 4 <= cn; k += 4)
        bad |= !group_four(a, ti, cb, k, src, xi, yi, ax0, ay0, ax1, ay1);
      if (bad) flags |= 1u << e;
      for (uint32_t t = 0; k < cn; ++k, ++t) {
        double tx, ty;
        if (!pair_term(a, seed, ti, cb + k, src.s[k], src.x[k], src.y[k], xi, yi, tx, ty)) tx = ty = -0.0;
        if (live) terms[(e * 4 + t) * wide + lane] = make_double2(tx, ty);
      }
      if (live) terms[(e * 4 + 3) * wide + lane] = make_double2(ax0 + ax1, ay0 + ay1);
    }
    if (live) a.long_flags[(size_t)u * 16 + lane] = flags;
  }
}

__global__ void __launch_bounds__(LONG_THREADS) k_fmm_p2p_add(FmmArgs a) {
  __shared__ Sources sources[LONG_THREADS / 32];
  if (a.info[FI_LIST_OVERFLOW]) return;
  const unsigned lane = threadIdx.x & 31;
  Sources &src = sources[threadIdx.x >> 5];
  const uint64_t seed = (uint64_t)__double_as_longlong(*a.seed);
  const uint32_t longs = 2 * a.info[FI_LONGS];  // two chunks of targets a leaf
  for (uint32_t w = (blockIdx.x * LONG_THREADS + threadIdx.x) >> 5; w < longs;
       w += gridDim.x * LONG_THREADS >> 5) {
    const uint32_t c = a.longs[w >> 1], chunk = w & 1;
    const uint32_t cnt = a.p2p_cnt[c], off = a.p2p_off[c];
    const uint32_t first = a.cells[c].first, count = a.cells[c].count;
    if (chunk * 32 >= count) continue;
    const uint32_t nseg = (cnt + 31) / 32, per = count <= 16 ? 1 : 2, wide = 16 * per;
    const uint32_t at = first + chunk * 32 + lane;
    const bool live = at < first + count;
    const uint32_t ti = live ? at : first;
    const uint32_t i = a.perm[ti], row = live ? lane : 0;
    const double xi = a.px[ti], yi = a.py[ti];
    double vx = a.vx[i], vy = a.vy[i];
    for (uint32_t sg = 0; sg < nseg; ++sg) {
      const uint32_t u = a.long_at[c] + (chunk * nseg + sg) * per;
      const double2 *terms = a.long_terms + (size_t)u * LONG_UNIT + row;
      const uint32_t flags = live ? a.long_flags[(size_t)u * 16 + lane] : 0;
      const uint32_t e0 = sg * 32, ne = min(32u, cnt - e0);
      uint32_t lb = 0, ln = 0;
      if (lane < ne) {
        const uint32_t B = a.p2p[off + e0 + lane];
        lb = a.cells[B].first;
        ln = a.cells[B].count;
      }
      // four source leaves' terms at a time on their way
      constexpr uint32_t AHEAD = 4;
      double2 buf[AHEAD][4];
#pragma unroll
      for (uint32_t q = 0; q < AHEAD; ++q)
#pragma unroll
        for (uint32_t t = 0; t < 4; ++t) buf[q][t] = terms[(q * 4 + t) * wide];
      for (uint32_t eb = 0; eb < ne; eb += AHEAD) {
#pragma unroll
        for (uint32_t q = 0; q < AHEAD; ++q) {
          const uint32_t e = eb + q;
          if (e >= ne) break;
          const uint32_t b0 = __shfl_sync(0xffffffffu, lb, e), bn = __shfl_sync(0xffffffffu, ln, e);
          const bool by_pairs = flags >> e & 1u;
          if (!by_pairs) {
#pragma unroll
            for (uint32_t t = 0; t < 3; ++t)
              if (t < (bn & 3)) {
                vx += buf[q][t].x;
                vy += buf[q][t].y;
              }
            vx += buf[q][3].x;
            vy += buf[q][3].y;
          }
          if (e + AHEAD < 32)
#pragma unroll
            for (uint32_t t = 0; t < 4; ++t) buf[q][t] = terms[((e + AHEAD) * 4 + t) * wide];
          if (__any_sync(0xffffffffu, by_pairs)) {
            double ax0 = 0, ax1 = 0, ay0 = 0, ay1 = 0;
            for (uint32_t o = 0; o < bn; o += 32) {
              const uint32_t cn = min(32u, bn - o);
              __syncwarp();
              if (lane < cn) {
                src.x[lane] = a.px[b0 + o + lane];
                src.y[lane] = a.py[b0 + o + lane];
                src.s[lane] = a.ps[b0 + o + lane];
              }
              __syncwarp();
              if (by_pairs) leaf_one(a, seed, ti, b0 + o, cn, src, xi, yi, vx, vy, ax0, ay0, ax1, ay1);
            }
            if (by_pairs) {
              vx += ax0 + ax1;
              vy += ay0 + ay1;
            }
          }
        }
      }
    }
    if (live) {
      a.vx[i] = vx;
      a.vy[i] = vy;
    }
  }
}

// ---- downward: L2L (fmm.zig:823-849), L2P (fmm.zig:853-886) ---------------------------

// L2L's sum for one coefficient: local `L` (re 0..q-1, im q..) shifted by the
// powers `pw`.
template <uint32_t P>
__device__ inline void l2l_sum(const FmmArgs &a, const double *L, const double *pw, uint32_t mm,
                               uint32_t q, double &sre, double &sim) {
  sre = sim = 0;
#pragma unroll
  for (uint32_t u = 0; u < (P ? P + 1 : q - mm); ++u) {
    const uint32_t l = mm + u;
    if (l >= q) continue;
    const double b = a.tab->binom[l * FMM_TAB + mm];
    const double xre = L[l] * b, xim = L[q + l] * b;
    sre += xre * pw[u] - xim * pw[q + u];
    sim += xre * pw[q + u] + xim * pw[u];
  }
}

// Rows of a warp's shared memory: a local and the powers of the step to it for
// each cell of the path from the root and for four children.
constexpr uint32_t DOWN_ROWS = FMM_LEVELS + 1 + 4;

// A warp per cell with leaf children: it takes the locals down the path from
// the root itself, in shared memory, then to its children, and on to their
// points. The path's upper cells are recomputed by every warp below them (the
// same operations on the same values): eight short sums a warp at 1 M nodes,
// where a grid barrier a level and a cell's children one after another made a
// chain of 19 us a level (6,000 nodes: 116 -> 15 us; 1 M: 415 -> 106 us).
template <uint32_t P>
__global__ void __launch_bounds__(DOWN_THREADS) k_fmm_down(FmmArgs a) {
  extern __shared__ double fmm_smem[];
  if (a.info[FI_LIST_OVERFLOW]) return;
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t p = P ? P : a.p, q = p + 1, stride = 2 * q, row = up_row(stride);
  double *Ls = fmm_smem + (size_t)warp * 2 * DOWN_ROWS * row, *pw = Ls + DOWN_ROWS * row;
  const uint32_t c = blockIdx.x * (DOWN_THREADS / 32) + warp;
  if (c >= a.ncells) return;
  const FCell A = load_cell(a.cells + c);
  if (A.nchild == 0 && c != 0) return;
  const uint32_t d = A.depth;  // path rows 0 .. d, children's rows d + 1 ..
  // lane k: the path's cell at depth k, then the children
  uint32_t id = c, at = c;
  for (uint32_t k = d; k-- > 0;) {
    at = a.cells[at].parent;
    if (k == lane) id = at;
  }
  if (lane > d && lane <= d + A.nchild) id = A.child0 + lane - d - 1;
  const uint32_t rows = d + 1 + A.nchild;
  FCell mine = {};
  if (lane < rows) mine = load_cell(a.cells + id);
  const unsigned leaves = __ballot_sync(0xffffffffu, lane < rows && mine.nchild == 0);
  if (!leaves) return;
  for (uint32_t i0 = 0; i0 < rows * stride; i0 += 32) {
    const uint32_t k = (i0 + lane) / stride, r = (i0 + lane) % stride;
    const uint32_t from = __shfl_sync(0xffffffffu, id, k & 31);
    if (k < rows) Ls[k * row + r] = a.lco[(size_t)from * stride + r];
  }
  {
    // the step to row k: from the row before, or from c to a child
    const uint32_t before = lane > d ? d : lane ? lane - 1 : 0;
    const double bx = __shfl_sync(0xffffffffu, mine.cx, before),
                 by = __shfl_sync(0xffffffffu, mine.cy, before);
    if (lane > 0 && lane < rows) shift_powers(mine.cx - bx, mine.cy - by, p, pw + lane * row);
  }
  __syncwarp();
  for (uint32_t k = 1; k <= d; ++k) {
    if (lane < q) {
      double sre, sim;
      l2l_sum<P>(a, Ls + (k - 1) * row, pw + k * row, lane, q, sre, sim);
      double *L = Ls + k * row;
      L[lane] = L[lane] + sre;
      L[q + lane] = L[q + lane] + sim;
    }
    __syncwarp();
  }
  const uint32_t S = 32 / q;
  for (uint32_t j = lane / q; j < A.nchild && lane < S * q; j += S) {
    const uint32_t k = d + 1 + j, mm = lane % q;
    double sre, sim;
    l2l_sum<P>(a, Ls + d * row, pw + k * row, mm, q, sre, sim);
    double *L = Ls + k * row;
    L[mm] = L[mm] + sre;
    L[q + mm] = L[q + mm] + sim;
  }
  __syncwarp();
  // the leaves' points, one leaf after another over the lanes
  const uint32_t held = leaves >> lane & 1u ? mine.count : 0;
  for (uint32_t k0 = 0;; k0 += 32) {
    uint32_t rk = 0, k = NONE, before = 0;
    for (uint32_t j = d; j < rows; ++j) {
      const uint32_t n = __shfl_sync(0xffffffffu, held, j), f = __shfl_sync(0xffffffffu, mine.first, j);
      if (k0 + lane - before < n) { rk = j; k = f + k0 + lane - before; }
      before += n;
    }
    if (k0 >= before) break;
    const double cx = __shfl_sync(0xffffffffu, mine.cx, rk), cy = __shfl_sync(0xffffffffu, mine.cy, rk);
    if (k == NONE) continue;
    const double *L = Ls + rk * row;
    const uint32_t j = a.perm[k];
    const double wre = a.ux[k] - cx, wim = a.uy[k] - cy;
    double are = L[p], aim = L[q + p];
#pragma unroll 8
    for (uint32_t l = p; l > 0;) {
      --l;
      const double nre = are * wre - aim * wim + L[l];
      const double nim = are * wim + aim * wre + L[q + l];
      are = nre;
      aim = nim;
    }
    a.vx[j] = a.vx[j] - are * a.inv_w;
    a.vy[j] = a.vy[j] + aim * a.inv_w;
  }
}

// ---- host ------------------------------------------------------------------------------

// Makes p hold at least `need` elements, with headroom so a slowly growing
// need does not reallocate every run.
template <typename T>
int grow(T *&p, size_t &cap, size_t need) {
  if (need <= cap && p) return 0;
  cudaFree(p);
  p = nullptr;
  cap = need + need / 2;
  D3_CUDA_OK(cudaMalloc(&p, cap * sizeof(T)));
  return 0;
}

int fmm_reserve_points(FmmDev &f, uint32_t n) {
  if (n <= f.pcap && f.pcap) return 0;
  uint32_t cap = n < 1024 ? 1024 : n;
  f.pcap = 0;
  device_give(f.px, f.py, f.ps, f.ux, f.uy, f.pt_levels);
  if (!device_take({{(void **)&f.px, cap * 8ull},
                    {(void **)&f.py, cap * 8ull},
                    {(void **)&f.ps, cap * 8ull},
                    {(void **)&f.ux, cap * 8ull},
                    {(void **)&f.uy, cap * 8ull},
                    {(void **)&f.pt_levels, cap * 2ull}}))
    return -1;
  f.pcap = cap;
  return 0;
}

int fmm_reserve_cells(FmmDev &f, uint32_t ccap) {
  if (ccap <= f.ccap && f.ccap) return 0;
  f.ccap = 0;
  device_give(f.cells, f.bx0, f.by0, f.bx1, f.by1, f.m2l_off, f.m2l_cnt, f.p2p_off, f.p2p_cnt, f.fwd_off,
              f.fwd_cnt, f.arrive, f.long_at);
  if (!device_take({{(void **)&f.cells, ccap * sizeof(FCell)},
                    {(void **)&f.bx0, ccap * 8ull},
                    {(void **)&f.by0, ccap * 8ull},
                    {(void **)&f.bx1, ccap * 8ull},
                    {(void **)&f.by1, ccap * 8ull},
                    {(void **)&f.m2l_off, ccap * 4ull},
                    {(void **)&f.m2l_cnt, ccap * 4ull},
                    {(void **)&f.p2p_off, ccap * 4ull},
                    {(void **)&f.p2p_cnt, ccap * 4ull},
                    {(void **)&f.fwd_off, ccap * 4ull},
                    {(void **)&f.fwd_cnt, ccap * 4ull},
                    {(void **)&f.arrive, ccap * 4ull},
                    {(void **)&f.long_at, ccap * 4ull}}))
    return -1;
  f.ccap = ccap;
  return 0;
}

void fmm_free(FastScratch &s) {
  FmmDev *f = static_cast<FmmDev *>(s.fmm);
  if (!f) return;
  cudaFree(f->px); cudaFree(f->py); cudaFree(f->ps); cudaFree(f->ux); cudaFree(f->uy);
  cudaFree(f->pt_levels);
  cudaFree(f->cells); cudaFree(f->bx0); cudaFree(f->by0); cudaFree(f->bx1); cudaFree(f->by1);
  cudaFree(f->m2l_off); cudaFree(f->m2l_cnt); cudaFree(f->p2p_off);
  cudaFree(f->p2p_cnt); cudaFree(f->fwd_off); cudaFree(f->fwd_cnt); cudaFree(f->m2l);
  cudaFree(f->p2p); cudaFree(f->fwd); cudaFree(f->mco); cudaFree(f->lco); cudaFree(f->tab);
  cudaFree(f->info); cudaFree(f->arrive); cudaFree(f->long_at); cudaFree(f->longs);
  cudaFree(f->long_items); cudaFree(f->long_flags); cudaFree(f->long_terms); cudaFree(f->square); cudaFree(f->geom);
  cudaFree(f->cb_count); cudaFree(f->start_of); cudaFree(f->level_of);
  cudaFreeHost(f->h_info); cudaFreeHost(f->h_geom);
  if (f->lists_read) cudaEventDestroy(f->lists_read);
  delete f;
  s.fmm = nullptr;
}

// The limit of a wait in k_fmm_lists: 20 ms, or D3_LISTS_WAIT_NS (0: every wait
// runs out at once, a test of what follows).
static unsigned long long lists_wait_ns() {
  static const unsigned long long v = [] {
    const char *e = getenv("D3_LISTS_WAIT_NS");
    return e ? strtoull(e, nullptr, 10) : 20000000ull;
  }();
  return v;
}

// Dynamic shared memory of a block, at q coefficients.
static int up_smem(uint32_t q) { return (int)(UP_THREADS / 32 * 32 * up_row(2 * q) * 8); }
static int m2l_smem(uint32_t q) { return (int)(M2L_THREADS / 32 * m2l_words(q) * 8); }
static int down_smem(uint32_t q) { return (int)(DOWN_THREADS / 32 * 2 * DOWN_ROWS * up_row(2 * q) * 8); }

uint32_t fmm_longs(const FastScratch &s) {
  const FmmDev *f = static_cast<const FmmDev *>(s.fmm);
  return f ? f->longs_last : 0;
}

static int sync_read(FmmDev &f, cudaStream_t st) {
  if (cudaMemcpyAsync(f.h_info, f.info, 64 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st) !=
          cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return -1;
  return 0;
}

int fmm_prepare(FastScratch &s, TreeDev &t, const NodeArrays &a, const double *strengths,
                double alpha, FmmPrep &out, cudaStream_t st) {
  const uint32_t n = a.n;
  if (!s.fmm) {
    FmmDev *f = new FmmDev();
    s.fmm = f;
    D3_CUDA_OK(cudaMalloc(&f->info, 64 * sizeof(uint32_t)));
    D3_CUDA_OK(cudaMemsetAsync(f->info, 0, 64 * sizeof(uint32_t), st));
    D3_CUDA_OK(cudaMalloc(&f->square, 4 * sizeof(double)));
    D3_CUDA_OK(cudaMalloc(&f->tab, sizeof(FmmTables)));
    D3_CUDA_OK(cudaMalloc(&f->geom, 4 * sizeof(double)));
    D3_CUDA_OK(cudaHostAlloc(&f->h_info, 64 * sizeof(uint32_t), cudaHostAllocDefault));
    D3_CUDA_OK(cudaHostAlloc(&f->h_geom, 8 * sizeof(double), cudaHostAllocDefault));
    D3_CUDA_OK(cudaEventCreateWithFlags(&f->lists_read, cudaEventDisableTiming));
    // shared memory past the default 48 KB (up to order 24)
    int up = 0, m2l = 0, down = 0;
    for (uint32_t q = 2; q <= FMM_MAX_ORDER + 1; ++q) {
      if (up_smem(q) > up) up = up_smem(q);
      if (m2l_smem(q) > m2l) m2l = m2l_smem(q);
      if (down_smem(q) > down) down = down_smem(q);
    }
    cudaFuncSetAttribute(k_fmm_upward<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, up);
    cudaFuncSetAttribute(k_fmm_m2l<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, m2l);
    cudaFuncSetAttribute(k_fmm_down<0>, cudaFuncAttributeMaxDynamicSharedMemorySize, down);
  }
  FmmDev &f = *static_cast<FmmDev *>(s.fmm);
  if (fmm_reserve_points(f, n)) return -1;
  // keys: square extent, quantised Morton keys, stable sort (NaN nodes last)
  fast_box(t, a.x, a.y, n, f.square, st);
  D3_LAUNCH(k_fmm_keys, blocks_for(n, 256), 256, 0, st)(a.x, a.y, n, f.square, t.keys, t.sv);
  SortScratch ss{t.keys_tmp, t.sv_tmp, t.hist};
  radix_sort_u64(t.keys, t.sv, n, 0, 4, true, ss, st);
  // the geometry, the point count and the gather stay on the device: the
  // host reads them with the cell counts, in one synchronisation
  D3_LAUNCH(k_fmm_geom, 1, 1, 0, st)(t.extent, t.info, f.geom, f.info);
  D3_LAUNCH(k_fmm_gather, blocks_for(n, 256), 256, 0, st)(t.sv, a.x, a.y, strengths, f.info, alpha,
                                                          f.geom, f.px, f.py, f.ps, f.ux, f.uy);
  // cells (level order); grow and rebuild if they do not fit
  uint32_t want = 2 * (n / FMM_LEAF + 1) + 64;
  for (int attempt = 0;; ++attempt) {
    if (fmm_reserve_cells(f, want > f.ccap ? want : f.ccap)) return -1;
    {
      const uint32_t nb = (n + CB_THREADS - 1) / CB_THREADS;
      if (grow(f.cb_count, f.cb_count_cap, (size_t)nb * CB_LEVELS) ||
          grow(f.start_of, f.start_cap, (size_t)f.ccap) || grow(f.level_of, f.level_cap, (size_t)f.ccap))
        return -1;
      D3_LAUNCH(k_cells_count, nb, CB_THREADS, 0, st)(t.keys, f.info, f.cb_count, f.pt_levels);
      D3_LAUNCH(k_cells_scan, CB_LEVELS, 1024, 0, st)(f.cb_count, nb, f.info);
      D3_LAUNCH(k_cells_starts, 1, 32, 0, st)(f.ccap, f.info);
      D3_LAUNCH(k_cells_place, nb, CB_THREADS, 0, st)(f.pt_levels, f.cb_count, f.info, f.start_of,
                                                    f.level_of);
      D3_LAUNCH(k_cells_fill, blocks_for(f.ccap, CB_THREADS), CB_THREADS, 0, st)(
          t.keys, f.start_of, f.level_of, f.info, f.cells, f.arrive, f.fwd_cnt);
    }
    if (cudaMemcpyAsync(f.h_geom, f.geom, 4 * sizeof(double), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        sync_read(f, st))
      return -1;
    if (f.h_info[FI_BAD]) return 0;  // the exact kernel runs instead
    if (!f.h_info[FI_M]) return 2;   // nothing to do (tree.zig:287-309 with an empty box)
    if (!f.h_info[FI_OVERFLOW]) break;
    if (attempt > 8) return -1;
    want = 2 * f.h_info[FI_OVERFLOW] + 64;
  }
  const uint32_t m = f.h_info[FI_M];
  const double w = f.h_geom[0], inv_w = f.h_geom[1], ox = f.h_geom[2], oy = f.h_geom[3];
  out.m = m;
  out.ncells = f.h_info[FI_CELLS];
  out.nlev = f.h_info[FI_LEVELS];
  for (uint32_t d = 0; d <= out.nlev && d < FMM_LEVELS + 2; ++d) out.lvl[d] = f.h_info[FI_LVL + d];
  out.w = w;
  out.inv_w = inv_w;
  out.ox = ox;
  out.oy = oy;
  out.keys = t.keys;
  out.perm = t.sv;
  out.px = f.px; out.py = f.py; out.ps = f.ps; out.ux = f.ux; out.uy = f.uy;
  out.cells = f.cells;
  out.info = f.info;
  return 1;
}

int fmm_run(FastScratch &s, TreeDev &t, const NodeArrays &a, const double *strengths,
            const FmmParams &prm, const double *seed, uint32_t *status, cudaStream_t st) {
  (void)status;
  FmmPrep pr;
  const int pre = fmm_prepare(s, t, a, strengths, prm.alpha, pr, st);
  if (pre == 2) return 1;
  if (pre <= 0) return pre;
  FmmDev &f = *static_cast<FmmDev *>(s.fmm);
  const double w = pr.w;
  uint32_t p = FMM_DEFAULT_ORDER;
  if (prm.order >= 1 && prm.order <= (double)FMM_MAX_ORDER) p = (uint32_t)prm.order;
  double kappa = prm.opening;
  if (!(kappa > 1)) kappa = FMM_DEFAULT_OPENING;
  if (f.tab_p != p) {
    // fmm.zig:223-238
    FmmTables h;
    memset(&h, 0, sizeof h);
    const size_t nmax = 2 * p + 2;
    for (size_t nn = 0; nn < nmax; ++nn) {
      h.binom[nn * FMM_TAB] = 1;
      for (size_t k = 1; k <= nn; ++k)
        h.binom[nn * FMM_TAB + k] =
            h.binom[(nn - 1) * FMM_TAB + k - 1] + (k < nn ? h.binom[(nn - 1) * FMM_TAB + k] : 0);
    }
    h.fact[0] = 1;
    for (size_t k = 1; k < nmax; ++k) h.fact[k] = h.fact[k - 1] * (double)k;
    for (size_t k = 0; k < nmax; ++k) h.ifact[k] = 1 / h.fact[k];
    if (cudaMemcpyAsync(f.tab, &h, sizeof h, cudaMemcpyHostToDevice, st) != cudaSuccess ||
        cudaStreamSynchronize(st) != cudaSuccess)
      return -1;
    f.tab_p = p;
  }
  const uint32_t q = p + 1, stride = 2 * q;
  FmmArgs args;
  memset(&args, 0, sizeof args);
  args.keys = t.keys;
  args.perm = t.sv;
  args.px = f.px; args.py = f.py; args.ps = f.ps; args.ux = f.ux; args.uy = f.uy;
  args.tab = f.tab;
  args.vx = a.vx; args.vy = a.vy;
  args.info = f.info;
  args.p = p;
  args.inv_w = pr.inv_w;
  args.mac_far = 2 * kappa - 1;
  double dmax_scaled = INFINITY;
  if (prm.dmax2 < INFINITY) dmax_scaled = sqrt(prm.dmax2) / w;
  const double dmin_scaled = prm.dmin2 > 0 ? sqrt(prm.dmin2) / w : 0;
  args.dmax_scaled = dmax_scaled;
  args.dmin_scaled = dmin_scaled;
  args.ring = dmin_scaled > 0 || dmax_scaled < INFINITY;
  args.has_dmax = dmax_scaled < INFINITY;
  args.dmin2 = prm.dmin2;
  args.dmax2 = prm.dmax2;
  args.seed = seed;
  const uint32_t ncells = pr.ncells;
  args.cells = f.cells;
  args.bx0 = f.bx0; args.by0 = f.by0; args.bx1 = f.bx1; args.by1 = f.by1;
  args.ncells = ncells;
  if ((size_t)ncells * stride > f.coef_cap || !f.mco) {
    f.coef_cap = 0;
    device_give(f.mco, f.lco);
    const size_t cap = (size_t)ncells * stride + (size_t)ncells * stride / 4;
    if (!device_take({{(void **)&f.mco, cap * 8}, {(void **)&f.lco, cap * 8}})) return -1;
    f.coef_cap = cap;
  }
  args.mco = f.mco;
  args.lco = f.lco;
  args.arrive = f.arrive;
  const bool few = ncells <= P2P_FEW_CELLS, longs = f.long_max > (few ? LONG_WORTH_FEW : LONG_WORTH);
  if (longs) f.long_room.grow([&](size_t cap) {
    device_give(f.longs, f.long_items, f.long_flags, f.long_terms);
    return device_take({{(void **)&f.longs, cap * 4},
                        {(void **)&f.long_items, cap * sizeof(uint2)},
                        {(void **)&f.long_flags, cap * 16 * 4},
                        {(void **)&f.long_terms, cap * LONG_UNIT * sizeof(double2)}});
  });
  args.long_items = f.long_items;
  args.long_at = f.long_at;
  args.longs = f.longs;
  args.long_flags = f.long_flags;
  args.long_terms = f.long_terms;
  args.long_cap = longs ? f.long_room.cap : 0;
  args.m2l_off = f.m2l_off; args.m2l_cnt = f.m2l_cnt;
  args.p2p_off = f.p2p_off; args.p2p_cnt = f.p2p_cnt;
  args.fwd_off = f.fwd_off; args.fwd_cnt = f.fwd_cnt;
  const bool dflt = p == FMM_DEFAULT_ORDER;  // its own kernels: the sums unroll
  const unsigned ub = blocks_for(ncells, UP_THREADS / 32), mb = blocks_for(ncells, M2L_THREADS / 32),
                 pb = blocks_for(ncells, P2P_THREADS / 32), db = blocks_for(ncells, DOWN_THREADS / 32);
  if (dflt) D3_LAUNCH(k_fmm_upward<FMM_DEFAULT_ORDER>, ub, UP_THREADS, up_smem(q), st)(args);
  else D3_LAUNCH(k_fmm_upward<0>, ub, UP_THREADS, up_smem(q), st)(args);
  // interaction lists; grow the pools and redo on overflow
  // first guesses from the cell count, then what the previous run needed
  size_t need_m2l = (size_t)ncells * 48 + 1024, need_p2p = (size_t)ncells * 16 + 1024,
         need_fwd = (size_t)ncells * 16 + 1024;
  if (f.last_m2l) {
    need_m2l = f.last_m2l + f.last_m2l / 4 + 1024;
    need_p2p = f.last_p2p + f.last_p2p / 4 + 1024;
    need_fwd = f.last_fwd + f.last_fwd / 4 + 1024;
  }
  args.by_level = 0;
  args.wait_ns = lists_wait_ns();
  for (int attempt = 0;; ++attempt) {
    if (grow(f.m2l, f.cap_m2l, need_m2l) || grow(f.p2p, f.cap_p2p, need_p2p) ||
        grow(f.fwd, f.cap_fwd, need_fwd))
      return -1;
    args.m2l = f.m2l; args.p2p = f.p2p; args.fwd = f.fwd;
    args.cap_m2l = f.cap_m2l; args.cap_p2p = f.cap_p2p; args.cap_fwd = f.cap_fwd;
    if (cudaMemsetAsync(f.info + FI_POOL_M2L, 0, 5 * sizeof(uint32_t), st) != cudaSuccess) return -1;
    if (attempt && (cudaMemsetAsync(f.fwd_cnt, 0xFF, (size_t)ncells * 4, st) != cudaSuccess ||
                    cudaMemsetAsync(f.info + FI_LONG_UNITS, 0, 12, st) != cudaSuccess))
      return -1;
    const uint32_t launches = args.by_level ? pr.nlev : 1;
    for (uint32_t lev = 0; lev < launches; ++lev) {
      const uint32_t c0 = args.by_level ? pr.lvl[lev] : 0, c1 = args.by_level ? pr.lvl[lev + 1] : ncells;
      if (c1 > c0)
        D3_LAUNCH(k_fmm_lists, blocks_for(c1 - c0, LISTS_THREADS / 32), LISTS_THREADS, 0, st)(args, c0, c1);
    }
    // the rest follows at once (it does nothing where a list overflowed), and
    // the host reads the lists' words while it runs
    if (cudaMemcpyAsync(f.h_info, f.info, 64 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st) !=
            cudaSuccess ||
        cudaEventRecord(f.lists_read, st) != cudaSuccess)
      return -1;
    if (dflt) D3_LAUNCH(k_fmm_m2l<FMM_DEFAULT_ORDER>, mb, M2L_THREADS, m2l_smem(q), st)(args);
    else D3_LAUNCH(k_fmm_m2l<0>, mb, M2L_THREADS, m2l_smem(q), st)(args);
    if (few)
      D3_LAUNCH(k_fmm_p2p<true>, blocks_for(4 * ncells, P2P_THREADS / 32), P2P_THREADS, 0, st)(args);
    else D3_LAUNCH(k_fmm_p2p<false>, pb, P2P_THREADS, 0, st)(args);
    if (args.long_cap) {
      D3_LAUNCH(k_fmm_p2p_terms, LONG_BLOCKS, LONG_THREADS, 0, st)(args);
      D3_LAUNCH(k_fmm_p2p_add, LONG_BLOCKS / 8, LONG_THREADS, 0, st)(args);
    }
    if (dflt) D3_LAUNCH(k_fmm_down<FMM_DEFAULT_ORDER>, db, DOWN_THREADS, down_smem(q), st)(args);
    else D3_LAUNCH(k_fmm_down<0>, db, DOWN_THREADS, down_smem(q), st)(args);
    if (cudaEventSynchronize(f.lists_read) != cudaSuccess) return -1;
    const uint32_t ovf = f.h_info[FI_LIST_OVERFLOW];
    if (!ovf) {
      f.last_m2l = f.h_info[FI_POOL_M2L];
      f.last_p2p = f.h_info[FI_POOL_P2P];
      f.last_fwd = f.h_info[FI_POOL_FWD];
      f.long_room.want = f.h_info[FI_LONG_UNITS];
      f.long_max = f.h_info[FI_LONG_MAX];
      f.longs_last = args.long_cap ? f.h_info[FI_LONGS] : 0;
      break;
    }
    if ((ovf & 2) || attempt > 8) return -1;  // a call stack overflowed
    if (ovf & 4) {  // a wait ran out (what it left out also says too little of the pools)
      args.by_level = 1;
      s.lists_by_level += 1;
    }
    if (!(ovf & 1)) continue;
    need_m2l = 2 * (size_t)(f.h_info[FI_POOL_M2L] > need_m2l ? f.h_info[FI_POOL_M2L] : need_m2l);
    need_p2p = 2 * (size_t)(f.h_info[FI_POOL_P2P] > need_p2p ? f.h_info[FI_POOL_P2P] : need_p2p);
    need_fwd = 2 * (size_t)(f.h_info[FI_POOL_FWD] > need_fwd ? f.h_info[FI_POOL_FWD] : need_fwd);
  }
  return cudaGetLastError() == cudaSuccess ? 1 : -1;
}

}  // namespace d3
