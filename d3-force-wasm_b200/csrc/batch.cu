// batch.cu — batched fast mode (no reference counterpart): thousands of
// independent graphs of uneven sizes tick in ONE persistent launch per tick,
// a run of ticks is captured in one CUDA graph, and the launch shape is
// picked by an autotuner.
//
// Each graph is a d3 simulation of its own with forceManyBody (FMM order 8,
// opening 1.5, distanceMin 1, strength -30), forceLink (distance 30, d3's
// default strength 1 / min(degree) and bias, one iteration) and forceCollide
// (radius 3, strength 1, one iteration), in FP32, with d3's alpha schedule
// and velocity decay 0.4. The fast forms follow the reference's fast mode:
// the link and the collide are Jacobi passes over a snapshot x + vx
// (link_fast.zig, grid.zig: each node adds only its own side), the
// many-body force an FMM (fmm.zig's expansions) — here on a complete
// quadtree over the graph's square box, with the level-free lattice
// operators of fmm_tc.cu (geometric centres, expansions normalised by the
// cell side), so every cell's interaction list is a fixed set of offsets.
//
// 2,048 graphs (6.0 M nodes, log-uniform 64 .. 16,384): ticks 2 and 12 from
// the phyllotaxis start take 3.8 and 5.1 ms (8.2 and 11 ms with bitonic sorts,
// Morton cells and the expansions in global memory); 40 graphs of at most
// 2,048 nodes 0.19 ms (0.9 ms). One 1024-thread CTA on each SM issues on 58 %
// of its cycles with 148 graphs of 16,000 nodes.
//
// Persistent kernel, one launch per tick: the CTAs take graphs from the
// tick's queue counter, largest first, and run the graph's whole tick in the
// CTA (shared memory and a per-CTA scratch region in global memory):
//   FMM   box; leaf of each node at level L (chosen per graph from the
//         autotuned leaf size); a counting sort by (leaf, node) (the order -
//         and every sum - is the same in any run and on any schedule); P2M;
//         M2M by level; M2L (39 offsets per quadrant) of all levels at once;
//         L2L by level; L2P; P2P over the 13 near leaves; v += kick.
//   link  snapshot x + vx; each node sums its links' own sides.
//   collide snapshot sorted by grid cell; each node scans the 3 x 3 cells
//         around it; then v *= 0.6, x += v.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

#include "common.cuh"
#include "pages.cuh"

namespace d3 {
namespace {

constexpr int BQ = 9;           // order 8: q = p + 1
constexpr int BQS = 10;         // a row of 9 coefficients and a pad (16-byte rows)
constexpr int BSLOT = 39;       // M2L offsets per quadrant at opening 1.5
constexpr int BCLASS_MAX = 60;  // distinct M2L offsets
constexpr uint32_t BMAX_N = 16384;
constexpr int BMAX_L = 6;
constexpr uint32_t BCELLS = (((1u << (2 * (BMAX_L + 1))) - 1) / 3);  // levels 0..6
constexpr float BDMIN2 = 1.f, BSTRENGTH = -30.f, BDIST = 30.f, BRADIUS = 3.f;

struct BTables {
  float2 k[BCLASS_MAX][BQ][BQS];  // M2L [class][l][k]
  float2 m2m[4][BQ][BQ];          // [b][n][k]
  float2 l2l[4][BQ][BQ];          // [b][m][l]
  int8_t slot_dx[4][BSLOT + 1], slot_dy[4][BSLOT + 1];
  uint8_t slot_class[4][BSLOT + 1];
};

static_assert(sizeof(BTables) % 16 == 0, "the tables are copied to shared memory in 16-byte units");

// One adjacency entry in one 16-byte load: the other node (local index),
// strength, this side's share, and +1 at the source / -1 at the target.
struct alignas(16) BLink {
  uint32_t j;
  float strength, share, sign;
};

struct BArgs {
  const BTables *tab;
  uint32_t graphs;
  const uint32_t *order;     // graphs, largest first
  const uint32_t *node_off;  // [graphs + 1]
  const uint8_t *level;      // FMM leaf level per graph
  const uint32_t *adj_off;   // [N + 1] per node (global index)
  const BLink *adj;
  float *x, *y, *vx, *vy;
  unsigned char *scratch;    // per CTA: what does not fit its shared memory
  size_t scratch_stride;     // bytes per CTA
  uint32_t smem;             // dynamic shared memory of the launch
  uint32_t *queue;           // this tick's counter
  float alpha;
  uint32_t tick;
  float2 *kick_out;          // non-null: many-body kick only (per global node), no other force
};

__host__ __device__ __forceinline__ uint32_t cells_before(int level) {  // cells at levels < level
  return ((1u << (2 * level)) - 1) / 3;
}
__host__ __device__ __forceinline__ size_t up16(size_t v) { return (v + 15) / 16 * 16; }
// Bytes of the 16-bit starts of `cells` cells (one more entry, whole words).
__host__ __device__ __forceinline__ size_t start_bytes(uint32_t cells) {
  return up16((cells + 2) / 2 * 4ull);
}
// Collide cells of a graph of n nodes (grid.zig: at most 4 n + 16).
__host__ __device__ __forceinline__ uint32_t grid_cap(uint32_t n) { return 4 * n + 16; }

// Shared memory that would hold every working array of a graph.
__host__ __forceinline__ size_t work_bytes(uint32_t n, int L) {
  const size_t nodes = up16(n * 8ull) + 2 * up16(n * 2ull);
  const size_t fmm = sizeof(BTables) + start_bytes(1u << (2 * L)) + nodes +
                     2 * (size_t)cells_before(L + 1) * BQS * 8;
  const size_t collide = start_bytes(grid_cap(n)) + nodes;
  return fmm > collide ? fmm : collide;
}

__host__ __device__ constexpr size_t scratch_bytes() {
  return (4 * BMAX_N + 16 + 32) * 2ull + BMAX_N * 12ull + 2ull * BCELLS * BQS * 8 + 256;
}

// The working arrays of a phase, taken in order: from shared memory while
// they fit, else from the CTA's scratch (L2).
struct Carve {
  unsigned char *sh, *gl;
  size_t left;
  template <typename T>
  __device__ __forceinline__ T *take(size_t bytes) {
    unsigned char *p;
    if (bytes <= left) {
      p = sh;
      sh += bytes;
      left -= bytes;
    } else {
      p = gl;
      gl += bytes;
    }
    return reinterpret_cast<T *>(p);
  }
};

// Sorting a graph's nodes by cell: the cells' counts, then starts (16 bits:
// at most 16,384 nodes), and per node its slot, then its place.
struct BSort {
  uint32_t *cnt;  // two 16-bit entries a word
  float2 *pos;    // sorted positions
  uint16_t *a;    // arrival slots by node, then sorted node indices
  uint16_t *b;    // nodes by cell, unordered
  __device__ __forceinline__ uint32_t start(uint32_t c) const {
    return reinterpret_cast<const uint16_t *>(cnt)[c];
  }
  // counts a node into cell c; returns its arrival slot
  __device__ __forceinline__ uint32_t arrive(uint32_t c) const {
    const uint32_t sh = 16 * (c & 1);
    return (atomicAdd(&cnt[c >> 1], 1u << sh) >> sh) & 0xFFFFu;
  }
};

// Complex product and product plus term, with the roundings spelled out: the
// layouts are chaotic within a few ticks (one unit in a velocity's last place
// moves close pairs visibly), so a compiler's choice of contraction should
// not change them.
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)),
                     __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float2 cmul_add(float2 a, float2 b, float2 c) {
  const float2 p = cmul(a, b);
  return make_float2(__fadd_rn(p.x, c.x), __fadd_rn(p.y, c.y));
}
__device__ __forceinline__ float norm2(float x, float y) {
  return __fmaf_rn(x, x, __fmul_rn(y, y));
}

// The block's bounding box {min x, min y, max x, max y} (every thread gets it).
__device__ float4 block_box(float4 v, float4 *sh) {
  auto merge = [](float4 p, float4 q) {
    return make_float4(fminf(p.x, q.x), fminf(p.y, q.y), fmaxf(p.z, q.z), fmaxf(p.w, q.w));
  };
  auto warp_box = [&](float4 p) {
    for (int o = 16; o > 0; o >>= 1)
      p = merge(p, make_float4(__shfl_xor_sync(0xffffffffu, p.x, o),
                               __shfl_xor_sync(0xffffffffu, p.y, o),
                               __shfl_xor_sync(0xffffffffu, p.z, o),
                               __shfl_xor_sync(0xffffffffu, p.w, o)));
    return p;
  };
  const uint32_t lane = threadIdx.x & 31, nw = blockDim.x / 32;
  v = warp_box(v);
  __syncthreads();
  if (lane == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  return warp_box(lane < nw ? sh[lane] : make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY));
}

// A level's cells quadrant by quadrant (of their parents), each quadrant row
// by row: the sources that neighbouring lanes of M2L read for one slot are
// then neighbours, whose 80-byte rows fall in distinct banks.
__device__ __forceinline__ uint32_t cell_at(int level, uint32_t ix, uint32_t iy) {
  return cells_before(level) + (((iy & 1) << 1 | (ix & 1)) << (2 * level - 2)) +
         ((iy >> 1) << (level - 1)) + (ix >> 1);
}

// Clears the counts of n cells (and the entry after them).
__device__ void clear_counts(uint32_t *cnt, uint32_t n) {
  for (uint32_t k = threadIdx.x; k < (n + 2) / 2; k += blockDim.x) cnt[k] = 0;
}

// Counts of n cells to exclusive prefix sums, entry n their total: a run of
// words per thread; barriers before and after.
__device__ void block_starts(uint32_t *cnt, uint32_t n, uint32_t *sh) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x / 32;
  const uint32_t words = (n + 2) / 2, per = (words + blockDim.x - 1) / blockDim.x;
  const uint32_t k0 = min(words, threadIdx.x * per), k1 = min(words, k0 + per);
  __syncthreads();
  uint32_t sum = 0;
  for (uint32_t k = k0; k < k1; ++k) sum += (cnt[k] & 0xFFFFu) + (cnt[k] >> 16);
  uint32_t incl = sum;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= (uint32_t)o) incl += y;
  }
  if (lane == 31) sh[warp] = incl;
  __syncthreads();
  uint32_t wi = lane < nw ? sh[lane] : 0;
  const uint32_t w = wi;
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, wi, o);
    if (lane >= (uint32_t)o) wi += y;
  }
  uint32_t run = __shfl_sync(0xffffffffu, wi - w, warp) + incl - sum;
  for (uint32_t k = k0; k < k1; ++k) {
    const uint32_t lo = cnt[k] & 0xFFFFu, hi = cnt[k] >> 16;
    cnt[k] = run | (run + lo) << 16;
    run += lo + hi;
  }
  __syncthreads();
}

// The counting sort's second half: with S.a[i] node i's arrival slot and
// S.cnt the starts, S.pos and S.a become the positions and nodes in (cell,
// node) order. The slots come in the order of the counting atomics, so a
// node's place in its cell is its rank among the cell's nodes: the same on
// every launch shape. node(i): the node's position; cell(p): its cell;
// keep(p): what S.pos holds.
template <typename Node, typename Cell, typename Keep>
__device__ void sort_by_cell(uint32_t n, const BSort &S, Node node, Cell cell, Keep keep) {
  const uint32_t t = threadIdx.x, nt = blockDim.x;
  for (uint32_t i = t; i < n; i += nt) S.b[S.start(cell(node(i))) + S.a[i]] = (uint16_t)i;
  __syncthreads();
  for (uint32_t p = t; p < n; p += nt) {
    const uint32_t i = S.b[p];
    const float2 q = node(i);
    const uint32_t c = cell(q), s0 = S.start(c), s1 = S.start(c + 1);
    uint32_t rank = 0;
    for (uint32_t k = s0; k < s1; ++k) rank += S.b[k] < i;
    S.a[s0 + rank] = (uint16_t)i;
    S.pos[s0 + rank] = keep(q);
  }
  __syncthreads();
}

// One pair of the near field: d3's formula with distanceMin 1, the hashed
// jiggle per zero component. (dx, dy) in, the force's factor out.
__device__ __forceinline__ float pair_factor(float &dx, float &dy, float strength, uint32_t i,
                                             uint32_t j, uint64_t seed) {
  float l = norm2(dx, dy);
  if (dx == 0.f || dy == 0.f) {
    if (dx == 0.f) {
      dx = (float)hash_jiggle(seed, i, j, 0);
      l += dx * dx;
    }
    if (dy == 0.f) {
      dy = (float)hash_jiggle(seed, i, j, 1);
      l += dy * dy;
    }
  }
  if (l < BDMIN2) l = sqrtf(BDMIN2 * l);
  return strength / l;
}

// The many-body force of one graph, into the velocities (or kick_out).
//
// Bound by issue in the near field (150 pairs a node on an even layout, up to
// 1,000 after a few ticks have drawn it together; about half of a tick) and
// M2L (39 slots a cell; a quarter), by latency and barriers elsewhere. Leaves
// are sorted row by row, so the 13 near leaves of a target are five contiguous runs
// of the sorted positions (same order as leaf by leaf); a target's sums stay
// in one thread and in that order, a pair's two components in packed FP32
// (FADD2, FMUL2, FFMA2), and four pairs share the test for zero deltas and
// distances inside distanceMin. M2L: a thread takes three coefficients of
// a cell, so a slot's multipole is read three times and not nine, the lanes
// of a warp take cells of one quadrant, whose operator reads are broadcasts,
// and all levels run in one pass.
__device__ void graph_many_body(const BArgs &a, unsigned char *smem, uint32_t g, uint32_t n0,
                                uint32_t n, float4 *red) {
  const uint32_t t = threadIdx.x, nt = blockDim.x;
  const int L = a.level[g];
  const uint32_t side = 1u << L, nleaf = side * side;
  const float *X = a.x + n0, *Y = a.y + n0;
  Carve cv{smem, a.scratch + (size_t)blockIdx.x * a.scratch_stride, a.smem};
  BSort S;
  S.cnt = cv.take<uint32_t>(start_bytes(nleaf));
  S.a = cv.take<uint16_t>(up16(n * 2ull));
  unsigned char *const low = cv.sh;  // from here on: free again by the near field
  const size_t low_bytes = cv.left;
  BTables &T = *cv.take<BTables>(sizeof(BTables));
  const size_t coef = (size_t)cells_before(L + 1) * BQS * 8, pos_bytes = up16(n * 8ull);
  float2 *const SM = cv.take<float2>(coef);
  S.b = cv.take<uint16_t>(up16(n * 2ull));
  // positions that do not fit beside the multipoles move in when those are
  // done with (the local expansions then stay out of their way)
  const bool late = pos_bytes > cv.left;
  if (late) cv.left = 0;
  S.pos = cv.take<float2>(pos_bytes);
  float2 *const SL = cv.take<float2>(coef);
  // the tables (the last graph's collide used their place)
  {
    const uint4 *src = reinterpret_cast<const uint4 *>(a.tab);
    uint4 *dst = reinterpret_cast<uint4 *>(&T);
    for (uint32_t k = t; k < sizeof(BTables) / 16; k += nt) dst[k] = src[k];
  }
  float4 box = make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
  for (uint32_t i = t; i < n; i += nt) {
    const float x = X[i], y = Y[i];
    box = make_float4(fminf(box.x, x), fminf(box.y, y), fmaxf(box.z, x), fmaxf(box.w, y));
  }
  clear_counts(S.cnt, nleaf);
  box = block_box(box, red);
  float w = fmaxf(box.z - box.x, box.w - box.y);
  if (!(w > 0)) w = 1;
  w *= 1.0001f;  // the largest coordinate stays inside the last cell
  const float inv_w = 1.f / w;
  auto node = [&](uint32_t i) { return make_float2(X[i], Y[i]); };
  // scaled coordinates: [0, 1) x [0, 1)
  auto scaled = [&](float2 p) {
    return make_float2((p.x - box.x) * inv_w, (p.y - box.y) * inv_w);
  };
  auto place = [&](float u) { return min(side - 1, (uint32_t)(u * side)); };
  auto leaf = [&](float2 p) {
    const float2 u = scaled(p);
    return place(u.y) * side + place(u.x);
  };
  for (uint32_t i = t; i < n; i += nt) S.a[i] = (uint16_t)S.arrive(leaf(node(i)));
  block_starts(S.cnt, nleaf, reinterpret_cast<uint32_t *>(red));
  sort_by_cell(n, S, node, leaf, scaled);
  // P2M: M'_k = sum s ((u - c) / s_L)^k, the points in order
  const float sL = 1.f / side, strength = BSTRENGTH * a.alpha;
  for (uint32_t c = t; c < nleaf; c += nt) {
    const uint32_t ix = c & (side - 1), iy = c >> L;
    const float cx = (ix + 0.5f) * sL, cy = (iy + 0.5f) * sL;
    float2 m[BQ];
#pragma unroll
    for (int k = 0; k < BQ; ++k) m[k] = make_float2(0, 0);
    const uint32_t k1 = S.start(c + 1);
    for (uint32_t k = S.start(c); k < k1; ++k) {
      const float2 u = S.pos[k];
      const float2 z = make_float2((u.x - cx) * side, (u.y - cy) * side);
      float2 p = make_float2(strength, 0);
#pragma unroll
      for (int o = 0; o < BQ; ++o) {
        m[o].x += p.x;
        m[o].y += p.y;
        p = cmul(p, z);
      }
    }
#pragma unroll
    for (int k = 0; k < BQ; ++k) SM[(size_t)cell_at(L, ix, iy) * BQS + k] = m[k];
  }
  __syncthreads();
  // M2M up to level 2
  for (int l = L - 1; l >= 2; --l) {
    const uint32_t nc = 1u << (2 * l);
    for (uint32_t e = t; e < nc * BQ; e += nt) {
      const uint32_t c = e / BQ, nn = e % BQ, ix = c & ((1u << l) - 1), iy = c >> l;
      float2 acc = make_float2(0, 0);
      for (uint32_t b = 0; b < 4; ++b) {
        const float2 *cm = SM + (size_t)cell_at(l + 1, 2 * ix + (b & 1), 2 * iy + (b >> 1)) * BQS;
        for (uint32_t k = 0; k <= nn; ++k) acc = cmul_add(cm[k], T.m2m[b][nn][k], acc);
      }
      SM[(size_t)cell_at(l, ix, iy) * BQS + nn] = acc;
    }
    __syncthreads();
  }
  // M2L of every level >= 2 (the lattice offsets of the cell's quadrant)
  const uint32_t first = cells_before(2), cells = cells_before(L + 1) - first;
  for (uint32_t e = t; e < 3 * cells; e += nt) {
    const uint32_t part = e / cells;
    uint32_t c = e - part * cells;
    int l = 2;
    while (c >= (1u << (2 * l))) {
      c -= 1u << (2 * l);
      ++l;
    }
    const uint32_t base = cells_before(l), l0 = 3 * part, row = base + c;
    const uint32_t qd = c >> (2 * l - 2), cq = c & ((1u << (2 * l - 2)) - 1);
    const int sl = 1 << l;
    const int ix = (int)((cq & ((1u << (l - 1)) - 1)) * 2 + (qd & 1));
    const int iy = (int)((cq >> (l - 1)) * 2 + (qd >> 1));
    float2 acc[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) acc[r] = make_float2(0, 0);
    for (int j = 0; j < BSLOT; ++j) {
      const int bx = ix + T.slot_dx[qd][j], by = iy + T.slot_dy[qd][j];
      if (bx < 0 || by < 0 || bx >= sl || by >= sl) continue;
      const float4 *mb = reinterpret_cast<const float4 *>(SM + (size_t)cell_at(l, bx, by) * BQS);
      const float4 *kk = reinterpret_cast<const float4 *>(&T.k[T.slot_class[qd][j]][l0][0]);
      float4 m[BQS / 2];
#pragma unroll
      for (int h = 0; h < BQS / 2; ++h) m[h] = mb[h];
#pragma unroll
      for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int h = 0; h < BQS / 2; ++h) {
          const float4 k = kk[r * (BQS / 2) + h];
          acc[r] = cmul_add(make_float2(m[h].x, m[h].y), make_float2(k.x, k.y), acc[r]);
          if (2 * h + 1 < BQ)
            acc[r] = cmul_add(make_float2(m[h].z, m[h].w), make_float2(k.z, k.w), acc[r]);
        }
    }
    float2 *lo = SL + (size_t)row * BQS + l0;
#pragma unroll
    for (int r = 0; r < 3; ++r) lo[r] = acc[r];
  }
  __syncthreads();
  // L2L down
  for (int l = 2; l < L; ++l) {
    const uint32_t nc = 1u << (2 * (l + 1));
    for (uint32_t e = t; e < nc * BQ; e += nt) {
      const uint32_t c = e / BQ, mm = e % BQ;
      const uint32_t ix = c & ((2u << l) - 1), iy = c >> (l + 1);
      const uint32_t b = (ix & 1) | ((iy & 1) << 1);
      const float2 *pl = SL + (size_t)cell_at(l, ix >> 1, iy >> 1) * BQS;
      float2 *const row = SL + (size_t)cell_at(l + 1, ix, iy) * BQS;
      float2 acc = row[mm];
      for (uint32_t l2 = mm; l2 < BQ; ++l2) acc = cmul_add(pl[l2], T.l2l[b][mm][l2], acc);
      row[mm] = acc;
    }
    __syncthreads();
  }
  // L2P and P2P, a thread per sorted point
  if (late && pos_bytes <= low_bytes) {
    const float4 *from = reinterpret_cast<const float4 *>(S.pos);
    float4 *to = reinterpret_cast<float4 *>(low);
    for (uint32_t k = t; k < pos_bytes / 16; k += nt) to[k] = from[k];
    S.pos = reinterpret_cast<float2 *>(low);
    __syncthreads();
  }
  const uint64_t seed = 0x5DEECE66Dull * (a.tick + 1);
  for (uint32_t k = t; k < n; k += nt) {
    const float2 p = S.pos[k];
    const uint32_t qx = place(p.x), qy = place(p.y), i = S.a[k];
    const float cx = (qx + 0.5f) * sL, cy = (qy + 0.5f) * sL;
    const float2 z = make_float2((p.x - cx) * side, (p.y - cy) * side);
    const float2 *Lc = SL + (size_t)cell_at(L, qx, qy) * BQS;
    float2 phi = Lc[BQ - 1];
#pragma unroll
    for (int l = BQ - 2; l >= 0; --l) phi = cmul_add(phi, z, Lc[l]);
    // phi / s_L in scaled units; the world kick divides by w
    float2 kick = make_float2(-phi.x * side * inv_w, phi.y * side * inv_w);
    const float2 np = make_float2(-p.x, -p.y), w2 = make_float2(w, w);
    // four sources from j on; the ones past j1 add nothing
    auto four = [&](uint32_t j, uint32_t j1, bool tail) {
      float2 d[4];
      float f[4], zero = 1.f, close = BDMIN2;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        d[u] = __fmul2_rn(__fadd2_rn(S.pos[tail ? min(j + u, j1 - 1) : j + u], np), w2);
        const float l = norm2(d[u].x, d[u].y);
        zero = fminf(zero, fminf(fabsf(d[u].x), fabsf(d[u].y)));
        close = fminf(close, l);
        f[u] = __fdividef(strength, l);
        if (tail && j + u >= j1) f[u] = 0.f;
      }
      if (zero != 0.f && !(close < BDMIN2)) {
#pragma unroll
        for (int u = 0; u < 4; ++u) kick = __ffma2_rn(d[u], make_float2(f[u], f[u]), kick);
      } else {
        // a zero delta or a pair inside distanceMin among them
#pragma unroll 1
        for (uint32_t u = j; u < min(j + 4, j1); ++u) {
          const float2 q = S.pos[u];
          float dx = (q.x - p.x) * w, dy = (q.y - p.y) * w;
          const float s = pair_factor(dx, dy, strength, i, S.a[u], seed);
          kick.x += dx * s;
          kick.y += dy * s;
        }
      }
    };
    // the five rows of near leaves, the target's own row as the runs before
    // and after it
#pragma unroll 1
    for (int r = 0; r < 6; ++r) {
      const int dy = r < 3 ? r - 2 : r - 3, by = (int)qy + dy, hw = 2 - abs(dy);
      if (by < 0 || by >= (int)side) continue;
      const int x0 = max((int)qx - hw, 0), x1 = min((int)qx + hw, (int)side - 1);
      uint32_t j = r == 3 ? k + 1 : S.start(by * side + x0);
      const uint32_t j1 = r == 2 ? k : S.start(by * side + x1 + 1);
      for (; j + 4 <= j1; j += 4) four(j, j1, false);
      if (j < j1) four(j, j1, true);
    }
    const float kx = kick.x, ky = kick.y;
    if (a.kick_out) {
      a.kick_out[n0 + i] = make_float2(kx, ky);
    } else {
      a.vx[n0 + i] += kx;
      a.vy[n0 + i] += ky;
    }
  }
  __syncthreads();
}

// link_fast.zig: each node adds its own side of each of its links, from the
// snapshot x + vx (in shared memory, up to the largest graph). Returns the
// box of x + vx after it (per thread).
__device__ float4 graph_link(const BArgs &a, unsigned char *smem, uint32_t n0, uint32_t n) {
  const uint32_t t = threadIdx.x, nt = blockDim.x;
  Carve cv{smem, a.scratch + (size_t)blockIdx.x * a.scratch_stride, a.smem};
  float2 *const P = cv.take<float2>(up16(n * 8ull));
  for (uint32_t i = t; i < n; i += nt)
    P[i] = make_float2(a.x[n0 + i] + a.vx[n0 + i], a.y[n0 + i] + a.vy[n0 + i]);
  __syncthreads();
  float4 box = make_float4(INFINITY, INFINITY, -INFINITY, -INFINITY);
  for (uint32_t i = t; i < n; i += nt) {
    const float2 p = P[i];
    float dvx = 0, dvy = 0;
    const uint32_t e1 = a.adj_off[n0 + i + 1];
    for (uint32_t e = a.adj_off[n0 + i]; e < e1; ++e) {
      const BLink k = a.adj[e];
      const float2 q = P[k.j];
      // the link's vector target - source
      float dx = (q.x - p.x) * k.sign, dy = (q.y - p.y) * k.sign;
      if (dx == 0.f) dx = (float)hash_jiggle(0x9E37ull * (a.tick + 1), min(i, k.j), max(i, k.j), 2);
      if (dy == 0.f) dy = (float)hash_jiggle(0x9E37ull * (a.tick + 1), min(i, k.j), max(i, k.j), 3);
      const float l = sqrtf(norm2(dx, dy));
      const float f = (l - BDIST) / l * a.alpha * k.strength;
      // target: v -= d f b; source: v += d f (1 - b)  (the sign picks the side)
      dvx += k.sign * dx * f * k.share;
      dvy += k.sign * dy * f * k.share;
    }
    const float vx = a.vx[n0 + i] + dvx, vy = a.vy[n0 + i] + dvy;
    a.vx[n0 + i] = vx;
    a.vy[n0 + i] = vy;
    const float x = a.x[n0 + i] + vx, y = a.y[n0 + i] + vy;
    box = make_float4(fminf(box.x, x), fminf(box.y, y), fmaxf(box.z, x), fmaxf(box.w, y));
  }
  return box;
}

// grid.zig: radius 3 for every node, strength 1; Jacobi from the snapshot
// x + vx (whose box is `box`, per thread); then v *= 0.6, x += v. The cells
// lie row by row, so a node's 3 x 3 cells are three runs of the sorted
// snapshot.
__device__ void graph_collide(const BArgs &a, unsigned char *smem, uint32_t n0, uint32_t n,
                              float4 box, float4 *red) {
  const uint32_t t = threadIdx.x, nt = blockDim.x;
  box = block_box(box, red);
  const float r2 = 2 * BRADIUS;
  // cell side 2r, coarsened until the grid has at most 4n + 16 cells
  float h = r2;
  uint32_t gx = 1, gy = 1;
  bool fits = false;
  for (int it = 0; it < 64 && !fits; ++it) {
    if (it) h *= 2;
    gx = (uint32_t)fminf((box.z - box.x) / h, 1e6f) + 1;
    gy = (uint32_t)fminf((box.w - box.y) / h, 1e6f) + 1;
    fits = (uint64_t)gx * gy <= grid_cap(n);
  }
  if (!fits) gx = gy = 1;  // a box that is not finite
  const float inv_h = 1.f / h;
  Carve cv{smem, a.scratch + (size_t)blockIdx.x * a.scratch_stride, a.smem};
  BSort S;
  S.cnt = cv.take<uint32_t>(start_bytes(gx * gy));
  S.pos = cv.take<float2>(up16(n * 8ull));
  S.a = cv.take<uint16_t>(up16(n * 2ull));
  S.b = cv.take<uint16_t>(up16(n * 2ull));
  clear_counts(S.cnt, gx * gy);
  __syncthreads();
  auto node = [&](uint32_t i) {
    return make_float2(a.x[n0 + i] + a.vx[n0 + i], a.y[n0 + i] + a.vy[n0 + i]);
  };
  auto col = [&](float x) { return min(gx - 1, (uint32_t)((x - box.x) * inv_h)); };
  auto row = [&](float y) { return min(gy - 1, (uint32_t)((y - box.y) * inv_h)); };
  auto cell = [&](float2 p) { return row(p.y) * gx + col(p.x); };
  for (uint32_t i = t; i < n; i += nt) S.a[i] = (uint16_t)S.arrive(cell(node(i)));
  block_starts(S.cnt, gx * gy, reinterpret_cast<uint32_t *>(red));
  sort_by_cell(n, S, node, cell, [](float2 p) { return p; });
  const float rr = r2 * r2;
  for (uint32_t k = t; k < n; k += nt) {
    const float2 p = S.pos[k];
    const int cx = (int)col(p.x), cy = (int)row(p.y);
    const uint32_t i = S.a[k];
    const int x0 = max(cx - 1, 0), x1 = min(cx + 1, (int)gx - 1);
    const int y1 = min(cy + 1, (int)gy - 1);
    float dvx = 0, dvy = 0;
    for (int by = max(cy - 1, 0); by <= y1; ++by) {
      const uint32_t m1 = S.start(by * gx + x1 + 1);
      for (uint32_t m = S.start(by * gx + x0); m < m1; ++m) {
        const float2 q = S.pos[m];
        float dx = p.x - q.x, dy = p.y - q.y;
        float l = norm2(dx, dy);
        if (!(l < rr) || m == k) continue;
        if (dx == 0.f || dy == 0.f) {
          const uint32_t j = S.a[m];
          const uint64_t seed = 0xC2B2AE35ull * (a.tick + 1);
          const float sg = i < j ? 1.f : -1.f;  // the pair's two sides push apart
          if (dx == 0.f) {
            dx = sg * (float)hash_jiggle(seed, min(i, j), max(i, j), 4);
            l += dx * dx;
          }
          if (dy == 0.f) {
            dy = sg * (float)hash_jiggle(seed, min(i, j), max(i, j), 5);
            l += dy * dy;
          }
        }
        l = sqrtf(l);
        const float push = (r2 - l) / l * 0.5f;  // equal radii: an even share
        dvx += dx * push;
        dvy += dy * push;
      }
    }
    const float vx = (a.vx[n0 + i] + dvx) * 0.6f, vy = (a.vy[n0 + i] + dvy) * 0.6f;
    a.vx[n0 + i] = vx;
    a.vy[n0 + i] = vy;
    a.x[n0 + i] += vx;
    a.y[n0 + i] += vy;
  }
  __syncthreads();
}

__global__ void __launch_bounds__(1024) k_batch_tick(BArgs a) {
  extern __shared__ __align__(16) unsigned char b_smem[];
  __shared__ float4 red[32];
  __shared__ uint32_t next;
  for (;;) {
    if (threadIdx.x == 0) next = atomicAdd(a.queue, 1u);
    __syncthreads();
    const uint32_t pos = next;
    __syncthreads();
    if (pos >= a.graphs) break;
    const uint32_t g = a.order[pos];
    const uint32_t n0 = a.node_off[g], n = a.node_off[g + 1] - n0;
    if (n == 0) continue;
    graph_many_body(a, b_smem, g, n0, n, red);
    if (a.kick_out) continue;
    const float4 box = graph_link(a, b_smem, n0, n);
    graph_collide(a, b_smem, n0, n, box, red);
  }
}

// ---- host ------------------------------------------------------------------------------------

double binom_h(int n, int k) {
  double r = 1;
  for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
  return r;
}

struct Cx {
  double re, im;
};
Cx cx_mul(Cx a, Cx b) { return {a.re * b.re - a.im * b.im, a.re * b.im + a.im * b.re}; }

void build_btables(BTables &T) {
  memset(&T, 0, sizeof T);
  const double k2 = 2 * 1.5 * 1.5;
  auto sep = [&](int x, int y) { return (double)(x * x + y * y) >= k2; };
  // the 13 near offsets: |dx| <= 2 - |dy|, as the near-field rows take them
  std::vector<std::pair<int, int>> near;
  for (int y = -2; y <= 2; ++y)
    for (int x = -2; x <= 2; ++x)
      if (!sep(x, y)) near.push_back({x, y});
  std::vector<std::pair<int, int>> classes;
  for (int aq = 0; aq < 4; ++aq) {
    const int ax = aq & 1, ay = aq >> 1;
    int ns = 0;
    for (const auto &o : near)
      for (int b = 0; b < 4; ++b) {
        const int vx = 2 * o.first + (b & 1) - ax, vy = 2 * o.second + (b >> 1) - ay;
        if (!sep(vx, vy)) continue;
        size_t c = 0;
        while (c < classes.size() && !(classes[c].first == vx && classes[c].second == vy)) ++c;
        if (c == classes.size()) classes.push_back({vx, vy});
        T.slot_dx[aq][ns] = (int8_t)vx;
        T.slot_dy[aq][ns] = (int8_t)vy;
        T.slot_class[aq][ns] = (uint8_t)c;
        ++ns;
      }
  }
  for (size_t c = 0; c < classes.size(); ++c) {
    // z0 = c_A - c_B = -(B - A)
    const Cx v{-(double)classes[c].first, -(double)classes[c].second};
    const double d2 = v.re * v.re + v.im * v.im;
    const Cx inv{v.re / d2, -v.im / d2};
    Cx pw[2 * BQ + 2];
    pw[0] = {1, 0};
    for (int e = 1; e < 2 * BQ + 2; ++e) pw[e] = cx_mul(pw[e - 1], inv);
    for (int l = 0; l < BQ; ++l)
      for (int k = 0; k < BQ; ++k) {
        const double f = ((l & 1) ? -1.0 : 1.0) * binom_h(k + l, l);
        T.k[c][l][k] = make_float2((float)(f * pw[k + l + 1].re), (float)(f * pw[k + l + 1].im));
      }
  }
  for (int b = 0; b < 4; ++b) {
    const Cx delta{(double)(2 * (b & 1) - 1), (double)(2 * (b >> 1) - 1)};
    for (int nn2 = 0; nn2 < BQ; ++nn2)
      for (int k = 0; k <= nn2; ++k) {
        Cx p{1, 0};
        for (int e = 0; e < nn2 - k; ++e) p = cx_mul(p, delta);
        const double f = binom_h(nn2, k) * std::ldexp(1.0, -k) * std::ldexp(1.0, -2 * (nn2 - k));
        T.m2m[b][nn2][k] = make_float2((float)(f * p.re), (float)(f * p.im));
      }
    for (int mm = 0; mm < BQ; ++mm)
      for (int l = mm; l < BQ; ++l) {
        Cx p{1, 0};
        for (int e = 0; e < l - mm; ++e) p = cx_mul(p, delta);
        const double f = binom_h(l, mm) * std::ldexp(1.0, -2 * (l - mm)) * std::ldexp(1.0, -(mm + 1));
        T.l2l[b][mm][l] = make_float2((float)(f * p.re), (float)(f * p.im));
      }
  }
}

// Reads of device arrays into the caller's pageable memory. One cudaMemcpy
// stages through one thread, which also takes every page fault of memory that
// was never touched. Here up to READ_WORKERS threads take pieces of READ_PIECE
// bytes in turn, each with two pinned slots (one being filled by the copy
// engine while the other is copied out). 96 MB, cudaMemcpy / threads: untouched
// 49 / 14 ms, touched 4.9 / 4.4 ms. The slots, 8 MB at most, stay with the batch
// and go with it; pinning them takes the first such read 8 to 18 ms more, so it
// needs READ_MIN bytes of untouched memory (48 MB: 25 ms by cudaMemcpy, 14 ms
// with the pinning, 7 ms without); other reads take cudaMemcpy until there are
// slots.
constexpr unsigned READ_WORKERS = 8, READ_SLOTS = 2;
constexpr size_t READ_PIECE = 1u << 19, READ_MIN = 48u << 20;

struct ReadSpan {
  void *dst;
  const void *src;
  size_t bytes;
};

class Reader {
 public:
  // Copies the spans; false on a CUDA error. One call at a time (a second
  // thread waits).
  bool read(const ReadSpan *spans, unsigned count) {
    size_t total = 0, untouched = 0;
    for (unsigned i = 0; i < count; ++i) total += spans[i].bytes;
    std::lock_guard<std::mutex> hold(lock_);
    if (total >= READ_MIN && !workers_)
      for (unsigned i = 0; i < count; ++i) untouched += untouched_bytes(spans[i].dst, spans[i].bytes);
    if (total < READ_MIN || (!workers_ && (untouched < READ_MIN || !reserve()))) {
      for (unsigned i = 0; i < count; ++i)
        if (cudaMemcpy(spans[i].dst, spans[i].src, spans[i].bytes, cudaMemcpyDeviceToHost) !=
            cudaSuccess)
          return false;
      return true;
    }
    int dev = 0;
    cudaGetDevice(&dev);
    spans_ = spans;
    count_ = count;
    next_ = 0;
    failed_ = false;
    std::thread threads[READ_WORKERS - 1];
    unsigned started = 0;
    try {
      for (; started + 1 < workers_; ++started)
        threads[started] = std::thread([this, dev, started] {
          if (cudaSetDevice(dev) == cudaSuccess) work(started + 1);
          else failed_ = true;
        });
    } catch (...) {  // no more threads: those that run take the pieces
    }
    work(0);
    for (unsigned t = 0; t < started; ++t) threads[t].join();
    return !failed_;
  }

  ~Reader() {
    if (stream_) cudaStreamDestroy(stream_);
    for (unsigned w = 0; w < READ_WORKERS; ++w)
      for (unsigned q = 0; q < READ_SLOTS; ++q)
        if (filled_[w][q]) cudaEventDestroy(filled_[w][q]);
    if (slots_) cudaFreeHost(slots_);
  }

 private:
  // The pinned slots, once. (A blocking stream: it waits for work on the
  // default stream, as cudaMemcpy does.)
  bool reserve() {
    if (workers_) return true;
    const unsigned cores = std::thread::hardware_concurrency();
    const unsigned n = cores && cores < READ_WORKERS ? cores : READ_WORKERS;
    bool ok = slots_ || cudaHostAlloc(reinterpret_cast<void **>(&slots_), n * READ_SLOTS * READ_PIECE,
                                      cudaHostAllocDefault) == cudaSuccess;
    ok = ok && (stream_ || cudaStreamCreate(&stream_) == cudaSuccess);
    for (unsigned w = 0; ok && w < n; ++w)
      for (unsigned q = 0; ok && q < READ_SLOTS; ++q)
        ok = filled_[w][q] ||
             cudaEventCreateWithFlags(&filled_[w][q], cudaEventDisableTiming) == cudaSuccess;
    if (ok) workers_ = n;
    else cudaGetLastError();
    return ok;
  }

  // Piece `i` of the spans in order; false past the last.
  bool piece(size_t i, ReadSpan &out) const {
    for (unsigned k = 0; k < count_; ++k) {
      const size_t pieces = (spans_[k].bytes + READ_PIECE - 1) / READ_PIECE;
      if (i < pieces) {
        const size_t at = i * READ_PIECE;
        out = {static_cast<char *>(spans_[k].dst) + at, static_cast<const char *>(spans_[k].src) + at,
               std::min(READ_PIECE, spans_[k].bytes - at)};
        return true;
      }
      i -= pieces;
    }
    return false;
  }

  void work(unsigned w) {
    ReadSpan held[READ_SLOTS];
    bool full[READ_SLOTS] = {};
    auto fill = [&](unsigned q) {
      full[q] = !failed_ && piece(next_++, held[q]);
      if (full[q] && (cudaMemcpyAsync(slot(w, q), held[q].src, held[q].bytes, cudaMemcpyDeviceToHost,
                                      stream_) != cudaSuccess ||
                      cudaEventRecord(filled_[w][q], stream_) != cudaSuccess)) {
        failed_ = true;
        full[q] = false;
      }
    };
    for (unsigned q = 0; q < READ_SLOTS; ++q) fill(q);
    for (unsigned q = 0; full[q]; q = (q + 1) % READ_SLOTS) {
      if (cudaEventSynchronize(filled_[w][q]) != cudaSuccess) {
        failed_ = true;
        break;
      }
      std::memcpy(held[q].dst, slot(w, q), held[q].bytes);
      fill(q);
    }
    if (failed_) cudaStreamSynchronize(stream_);  // no copy into a slot is left behind
  }

  char *slot(unsigned w, unsigned q) const { return slots_ + (w * READ_SLOTS + q) * READ_PIECE; }

  std::mutex lock_;
  unsigned workers_ = 0;
  char *slots_ = nullptr;
  cudaStream_t stream_ = nullptr;
  cudaEvent_t filled_[READ_WORKERS][READ_SLOTS] = {};
  const ReadSpan *spans_ = nullptr;
  unsigned count_ = 0;
  std::atomic<size_t> next_{0};
  std::atomic<bool> failed_{false};
};

struct Batch {
  uint32_t graphs = 0, nodes = 0;
  std::vector<uint32_t> h_off, h_order;
  std::vector<uint8_t> h_level;
  std::vector<uint32_t> h_counts;
  BTables *tab = nullptr;
  uint32_t *order = nullptr, *node_off = nullptr, *adj_off = nullptr;
  uint8_t *level = nullptr;
  BLink *adj = nullptr;
  float *x = nullptr, *y = nullptr, *vx = nullptr, *vy = nullptr;
  unsigned char *scratch = nullptr;
  uint32_t *queues = nullptr;
  uint32_t queue_cap = 0;
  float2 *kick = nullptr;
  double alpha = 1, alpha_decay = 0;
  uint32_t tick = 0;
  int threads = 512, per_sm = 1, sms = 148;
  uint32_t leaf_size = 16;
  size_t scratch_ctas = 0, smem = 0;
  cudaStream_t st = nullptr;
  cudaGraphExec_t graph = nullptr;
  uint32_t graph_ticks = 0;
  Reader reader;
};

std::vector<Batch *> g_batches;

Batch *get_batch(uint32_t h) {
  return h >= 1 && h <= g_batches.size() ? g_batches[h - 1] : nullptr;
}

// Dynamic shared memory a launch may take with `per_sm` CTAs on an SM: 227 KB
// less the kernel's static part for one, half of the SM's 228 KB less the
// 1 KB reserved per CTA and the static part for two.
size_t smem_cap(int per_sm) { return per_sm == 1 ? 226 * 1024 : 112 * 1024; }

void set_levels(Batch &b) {
  b.h_level.resize(b.graphs);
  for (uint32_t g = 0; g < b.graphs; ++g) {
    int L = 2;
    while (L < BMAX_L && (double)b.h_counts[g] / (double)(1u << (2 * L)) > b.leaf_size) ++L;
    b.h_level[g] = (uint8_t)L;
  }
  cudaMemcpyAsync(b.level, b.h_level.data(), b.graphs, cudaMemcpyHostToDevice, b.st);
  // what the largest working set takes, up to the cap: more of the SM's
  // memory stays L1 for the loads through the node and link arrays
  b.smem = 0;
  for (uint32_t g = 0; g < b.graphs; ++g) {
    const size_t sum = work_bytes(b.h_counts[g], b.h_level[g]);
    b.smem = sum > b.smem ? sum : b.smem;
  }
  b.smem = b.smem < smem_cap(b.per_sm) ? b.smem : smem_cap(b.per_sm);
}

int ensure_scratch(Batch &b) {
  const size_t ctas = (size_t)b.sms * b.per_sm;
  if (ctas <= b.scratch_ctas) return 0;
  cudaFree(b.scratch);
  b.scratch = nullptr;
  if (cudaMalloc(&b.scratch, ctas * scratch_bytes()) != cudaSuccess) return -1;
  b.scratch_ctas = ctas;
  return 0;
}

BArgs args_of(Batch &b, float alpha, uint32_t tick, uint32_t *queue, float2 *kick) {
  BArgs a;
  a.tab = b.tab;
  a.graphs = b.graphs;
  a.order = b.order;
  a.node_off = b.node_off;
  a.level = b.level;
  a.adj_off = b.adj_off;
  a.adj = b.adj;
  a.x = b.x; a.y = b.y; a.vx = b.vx; a.vy = b.vy;
  a.scratch = b.scratch;
  a.scratch_stride = scratch_bytes();
  a.smem = (uint32_t)b.smem;
  a.queue = queue;
  a.alpha = alpha;
  a.tick = tick;
  a.kick_out = kick;
  return a;
}

int launch_tick(Batch &b, float alpha, uint32_t tick, uint32_t *queue, float2 *kick) {
  BArgs a = args_of(b, alpha, tick, queue, kick);
  D3_LAUNCH(k_batch_tick, b.sms * b.per_sm, b.threads, b.smem, b.st)(a);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}

int ensure_queues(Batch &b, uint32_t n) {
  if (n <= b.queue_cap) return 0;
  cudaFree(b.queues);
  b.queues = nullptr;
  if (cudaMalloc(&b.queues, (size_t)n * 4) != cudaSuccess) return -1;
  b.queue_cap = n;
  return 0;
}

}  // namespace
}  // namespace d3

using namespace d3;

extern "C" {

uint32_t batch_create(uint32_t graphs, const uint32_t *node_counts, const uint32_t *link_counts,
                      const uint32_t *src, const uint32_t *tgt, const float *x, const float *y) {
  if (graphs == 0 || !node_counts || !link_counts || !x || !y) return 0;
  Batch *b = new Batch();
  b->graphs = graphs;
  b->h_counts.assign(node_counts, node_counts + graphs);
  b->h_off.resize(graphs + 1, 0);
  size_t links = 0;
  for (uint32_t g = 0; g < graphs; ++g) {
    if (node_counts[g] > BMAX_N) {
      delete b;
      return 0;
    }
    b->h_off[g + 1] = b->h_off[g] + node_counts[g];
    links += link_counts[g];
  }
  const uint32_t N = b->h_off[graphs];
  b->nodes = N;
  // per-node adjacency: d3's default link strength 1 / min(degree) and bias
  // degree(source) / (degree(source) + degree(target)) (link.js:30-67)
  std::vector<uint32_t> deg(N, 0), adj_off(N + 1, 0);
  std::vector<BLink> adj(2 * links);
  size_t e0 = 0;
  for (uint32_t g = 0; g < graphs; ++g) {
    for (uint32_t e = 0; e < link_counts[g]; ++e) {
      const uint32_t s = src[e0 + e], t = tgt[e0 + e];
      if (s >= node_counts[g] || t >= node_counts[g]) {
        delete b;
        return 0;
      }
      ++deg[b->h_off[g] + s];
      ++deg[b->h_off[g] + t];
    }
    e0 += link_counts[g];
  }
  for (uint32_t i = 0; i < N; ++i) adj_off[i + 1] = adj_off[i] + deg[i];
  std::vector<uint32_t> fill(adj_off.begin(), adj_off.end() - 1);
  e0 = 0;
  for (uint32_t g = 0; g < graphs; ++g) {
    const uint32_t o = b->h_off[g];
    for (uint32_t e = 0; e < link_counts[g]; ++e) {
      const uint32_t s = src[e0 + e], t = tgt[e0 + e];
      const float ds = (float)deg[o + s], dt = (float)deg[o + t];
      const float k = 1.f / fminf(ds, dt), bias = ds / (ds + dt);
      // an entry's sign turns (other - self) into d = target - source and
      // gives its side's direction: the target gets -d f bias, the source
      // +d f (1 - bias)
      adj[fill[o + t]++] = BLink{s, k, bias, -1.f};
      adj[fill[o + s]++] = BLink{t, k, 1.f - bias, 1.f};
    }
    e0 += link_counts[g];
  }
  // largest graphs first
  b->h_order.resize(graphs);
  for (uint32_t g = 0; g < graphs; ++g) b->h_order[g] = g;
  std::stable_sort(b->h_order.begin(), b->h_order.end(),
                   [&](uint32_t p, uint32_t q) { return node_counts[p] > node_counts[q]; });
  BTables T;
  build_btables(T);
  int dev = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, dev);
  bool ok = cudaStreamCreateWithFlags(&b->st, cudaStreamNonBlocking) == cudaSuccess &&
            cudaMalloc(&b->tab, sizeof(BTables)) == cudaSuccess &&
            cudaMalloc(&b->order, graphs * 4) == cudaSuccess &&
            cudaMalloc(&b->node_off, (graphs + 1) * 4) == cudaSuccess &&
            cudaMalloc(&b->level, graphs) == cudaSuccess &&
            cudaMalloc(&b->adj_off, (N + 1) * 4ull) == cudaSuccess &&
            cudaMalloc(&b->adj, (2 * links + 1) * sizeof(BLink)) == cudaSuccess &&
            cudaMalloc(&b->x, N * 4ull) == cudaSuccess && cudaMalloc(&b->y, N * 4ull) == cudaSuccess &&
            cudaMalloc(&b->vx, N * 4ull) == cudaSuccess && cudaMalloc(&b->vy, N * 4ull) == cudaSuccess &&
            cudaMalloc(&b->kick, N * sizeof(float2)) == cudaSuccess;
  // on the batch's stream, which does not wait for the default one
  auto put = [&](void *to, const void *from, size_t bytes) {
    return cudaMemcpyAsync(to, from, bytes, cudaMemcpyHostToDevice, b->st) == cudaSuccess;
  };
  ok = ok && put(b->tab, &T, sizeof T) && put(b->order, b->h_order.data(), graphs * 4) &&
       put(b->node_off, b->h_off.data(), (graphs + 1) * 4) &&
       put(b->adj_off, adj_off.data(), (N + 1) * 4ull) &&
       (links == 0 || put(b->adj, adj.data(), 2 * links * sizeof(BLink))) &&
       put(b->x, x, N * 4ull) && put(b->y, y, N * 4ull) &&
       cudaMemsetAsync(b->vx, 0, N * 4ull, b->st) == cudaSuccess &&
       cudaMemsetAsync(b->vy, 0, N * 4ull, b->st) == cudaSuccess;
  cudaFuncSetAttribute(k_batch_tick, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)smem_cap(1));
  b->alpha_decay = 1 - std::pow(0.001, 1.0 / 300);
  if (ok) {
    set_levels(*b);
    ok = ensure_scratch(*b) == 0 && cudaStreamSynchronize(b->st) == cudaSuccess;
  }
  if (!ok) {
    delete b;
    return 0;
  }
  g_batches.push_back(b);
  return (uint32_t)g_batches.size();
}

int32_t batch_destroy(uint32_t h) {
  Batch *b = get_batch(h);
  if (!b) return D3_BAD_HANDLE;
  if (b->graph) cudaGraphExecDestroy(b->graph);
  cudaFree(b->tab); cudaFree(b->order); cudaFree(b->node_off); cudaFree(b->level);
  cudaFree(b->adj_off); cudaFree(b->adj); cudaFree(b->x); cudaFree(b->y);
  cudaFree(b->vx); cudaFree(b->vy); cudaFree(b->scratch); cudaFree(b->queues); cudaFree(b->kick);
  cudaStreamDestroy(b->st);
  delete b;
  g_batches[h - 1] = nullptr;
  return D3_OK;
}

// Launch shape: threads per CTA, CTAs per SM, target points per FMM leaf.
int32_t batch_set_shape(uint32_t h, uint32_t threads, uint32_t per_sm, uint32_t leaf_size) {
  Batch *b = get_batch(h);
  if (!b) return D3_BAD_HANDLE;
  if ((threads != 256 && threads != 512 && threads != 1024) || per_sm < 1 || per_sm > 2 ||
      leaf_size < 2 || leaf_size > 256)
    return D3_BAD_ARGUMENT;
  int per = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_batch_tick, (int)threads,
                                                smem_cap((int)per_sm));
  if ((int)per_sm > per) return D3_BAD_ARGUMENT;
  b->threads = (int)threads;
  b->per_sm = (int)per_sm;
  b->leaf_size = leaf_size;
  set_levels(*b);
  if (ensure_scratch(*b)) return D3_OUT_OF_MEMORY;
  if (b->graph) {
    cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
    b->graph_ticks = 0;
  }
  return D3_OK;
}

// Capturing and instantiating a graph costs 0.13 - 0.18 ms whatever its length
// (1 to 128 ticks of 40 graphs of up to 2,048 nodes, 0.35 ms a tick), which a
// run of a few ticks does not get back: those are launched one by one (one
// tick 0.50 -> 0.37 ms, 8 ticks 2.97 -> 2.81 ms, 64 ticks 22.5 -> 22.3 ms).
constexpr uint32_t GRAPH_TICKS = 16;

// Runs `ticks` ticks (d3's alpha schedule continues from the batch's
// state). graph != 0: GRAPH_TICKS ticks or more are captured once into a CUDA
// graph (one kernel node per tick) and replayed. *ms: device time (CUDA events).
int32_t batch_run(uint32_t h, uint32_t ticks, uint32_t graph, double *ms) {
  Batch *b = get_batch(h);
  if (!b) return D3_BAD_HANDLE;
  if (ticks == 0) return D3_OK;
  if (ensure_queues(*b, ticks)) return D3_OUT_OF_MEMORY;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  int32_t rc = D3_OK;
  // alphas of these ticks (simulation.js:64 per tick)
  std::vector<float> alphas(ticks);
  double al = b->alpha;
  for (uint32_t k = 0; k < ticks; ++k) {
    al += (0 - al) * b->alpha_decay;
    alphas[k] = (float)al;
  }
  if (cudaMemsetAsync(b->queues, 0, (size_t)ticks * 4, b->st) != cudaSuccess) rc = D3_WORKER_FAILED;
  if (graph && ticks >= GRAPH_TICKS && rc == D3_OK) {
    // a captured run is tied to its alphas and tick numbers: capture anew
    if (b->graph) {
      cudaGraphExecDestroy(b->graph);
      b->graph = nullptr;
    }
    cudaGraph_t gr = nullptr;
    if (cudaStreamBeginCapture(b->st, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      rc = D3_WORKER_FAILED;
    } else {
      for (uint32_t k = 0; k < ticks; ++k)
        if (launch_tick(*b, alphas[k], b->tick + k, b->queues + k, nullptr)) rc = D3_WORKER_FAILED;
      if (cudaStreamEndCapture(b->st, &gr) != cudaSuccess) rc = D3_WORKER_FAILED;
    }
    if (rc == D3_OK && cudaGraphInstantiate(&b->graph, gr, 0) != cudaSuccess) rc = D3_WORKER_FAILED;
    if (gr) cudaGraphDestroy(gr);
    if (rc == D3_OK) {
      cudaEventRecord(e0, b->st);
      if (cudaGraphLaunch(b->graph, b->st) != cudaSuccess) rc = D3_WORKER_FAILED;
      cudaEventRecord(e1, b->st);
    }
  } else if (rc == D3_OK) {
    cudaEventRecord(e0, b->st);
    for (uint32_t k = 0; k < ticks; ++k)
      if (launch_tick(*b, alphas[k], b->tick + k, b->queues + k, nullptr)) rc = D3_WORKER_FAILED;
    cudaEventRecord(e1, b->st);
  }
  if (cudaStreamSynchronize(b->st) != cudaSuccess) rc = D3_WORKER_FAILED;
  float f = 0;
  cudaEventElapsedTime(&f, e0, e1);
  if (ms) *ms = f;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (rc == D3_OK) {
    b->alpha = al;
    b->tick += ticks;
  }
  return rc;
}

// The many-body kick alone (FMM, the batch's next alpha) at the current
// positions, per node (x, y pairs), into host `out` (2 x nodes floats).
int32_t batch_kick(uint32_t h, float *out, double *alpha_used) {
  Batch *b = get_batch(h);
  if (!b || !out) return b ? D3_BAD_ARGUMENT : D3_BAD_HANDLE;
  if (ensure_queues(*b, 1)) return D3_OUT_OF_MEMORY;
  const double al = b->alpha + (0 - b->alpha) * b->alpha_decay;
  if (alpha_used) *alpha_used = (float)al;
  if (cudaMemsetAsync(b->queues, 0, 4, b->st) != cudaSuccess ||
      launch_tick(*b, (float)al, b->tick, b->queues, b->kick) ||
      cudaStreamSynchronize(b->st) != cudaSuccess)
    return D3_WORKER_FAILED;
  const ReadSpan span{out, b->kick, b->nodes * sizeof(float2)};
  return b->reader.read(&span, 1) ? D3_OK : D3_WORKER_FAILED;
}

int32_t batch_read(uint32_t h, float *x, float *y, float *vx, float *vy) {
  Batch *b = get_batch(h);
  if (!b) return D3_BAD_HANDLE;
  const size_t bytes = b->nodes * 4ull;
  const ReadSpan all[4] = {{x, b->x, bytes}, {y, b->y, bytes}, {vx, b->vx, bytes}, {vy, b->vy, bytes}};
  ReadSpan spans[4];
  unsigned count = 0;
  for (const ReadSpan &sp : all)
    if (sp.dst) spans[count++] = sp;
  return b->reader.read(spans, count) ? D3_OK : D3_WORKER_FAILED;
}

// Autotuner: times `ticks` ticks (from a copy of the current state, which is
// restored) for every launch shape - threads 256 / 512 / 1024, 1 or 2 CTAs
// per SM where they fit, leaf sizes 8 / 16 / 32 - and keeps the fastest.
// out[0..3]: threads, CTAs per SM, leaf size, ms per tick of the choice.
int32_t batch_autotune(uint32_t h, uint32_t ticks, double *out) {
  Batch *b = get_batch(h);
  if (!b) return D3_BAD_HANDLE;
  const size_t bytes = b->nodes * 4ull;
  float *save = nullptr;
  if (cudaMalloc(&save, 4 * bytes) != cudaSuccess) return D3_OUT_OF_MEMORY;
  float *arr[4] = {b->x, b->y, b->vx, b->vy};
  for (int k = 0; k < 4; ++k)
    cudaMemcpyAsync(save + k * b->nodes, arr[k], bytes, cudaMemcpyDeviceToDevice, b->st);
  const double alpha0 = b->alpha;
  const uint32_t tick0 = b->tick;
  double best = 1e30;
  uint32_t bt = 512, bp = 1, bl = 16;
  int32_t rc = D3_OK;
  for (uint32_t th : {256u, 512u, 1024u})
    for (uint32_t ps : {1u, 2u})
      for (uint32_t ls : {8u, 16u, 32u}) {
        if (batch_set_shape(h, th, ps, ls) != D3_OK) continue;
        double ms = 0;
        if (batch_run(h, 1, 0, &ms) != D3_OK || batch_run(h, ticks, 0, &ms) != D3_OK) {
          rc = D3_WORKER_FAILED;
          break;
        }
        ms /= ticks;
        if (ms < best) {
          best = ms;
          bt = th;
          bp = ps;
          bl = ls;
        }
        for (int k = 0; k < 4; ++k)
          cudaMemcpyAsync(arr[k], save + k * b->nodes, bytes, cudaMemcpyDeviceToDevice, b->st);
        b->alpha = alpha0;
        b->tick = tick0;
      }
  if (cudaStreamSynchronize(b->st) != cudaSuccess) rc = D3_WORKER_FAILED;  // the state is back
  cudaFree(save);
  if (rc != D3_OK) return rc;
  batch_set_shape(h, bt, bp, bl);
  if (out) {
    out[0] = bt;
    out[1] = bp;
    out[2] = bl;
    out[3] = best;
  }
  return D3_OK;
}

}  // extern "C"
