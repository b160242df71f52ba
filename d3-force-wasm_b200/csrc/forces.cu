// forces.cu — exact-mode forces on the device, bit-exact with d3-force.
//
// All arithmetic keeps d3's statement order (no FMA contraction: the file is
// built with -fmad=false). Traversals are stackless: cells are in d3's visit
// preorder, so "descend" is c + 1 and "do not descend" is skip[c].
#include <climits>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>

#include "forces.cuh"
#include "scan_sort.cuh"

namespace cg = cooperative_groups;

namespace d3 {

size_t csum_rec_bytes(uint32_t n);
size_t csum_count_words(uint32_t n);
size_t csum_part_words(uint32_t n);

int scratch_reserve(ForceScratch &s, uint32_t n, cudaStream_t st) {
  if (!s.counters) {
    D3_CUDA_OK(cudaMalloc(&s.counters, 16 * sizeof(uint32_t)));
    D3_CUDA_OK(cudaMemsetAsync(s.counters, 0, 16 * sizeof(uint32_t), st));
    D3_CUDA_OK(cudaMalloc(&s.center, 2 * sizeof(double)));
    D3_CUDA_OK(cudaMalloc(&s.csum_stamps, 8 * sizeof(unsigned long long)));
    D3_CUDA_OK(cudaMemsetAsync(s.csum_stamps, 0, 8 * sizeof(unsigned long long), st));
  }
  if (n <= s.cap && s.cap) return 0;
  uint32_t cap = n < 1024 ? 1024 : n;
  cudaFree(s.draws); cudaFree(s.offsets); cudaFree(s.scan_part);
  cudaFree(s.csum_recs); cudaFree(s.csum_counts); cudaFree(s.csum_part); cudaFree(s.csum_scan_part);
  D3_CUDA_OK(cudaMalloc(&s.csum_recs, csum_rec_bytes(cap)));
  D3_CUDA_OK(cudaMalloc(&s.csum_counts, 2 * csum_count_words(cap) * 4));  // counts, offsets
  D3_CUDA_OK(cudaMalloc(&s.csum_part, csum_part_words(cap) * 8));
  D3_CUDA_OK(cudaMalloc(&s.csum_scan_part, scan_partial_words(csum_count_words(cap)) * 4));
  D3_CUDA_OK(cudaMalloc(&s.draws, (cap + 1) * 4ull));
  D3_CUDA_OK(cudaMalloc(&s.offsets, (cap + 1) * 4ull));
  // also the grid partials of k_mb_draws (one word per block)
  const size_t sp = scan_partial_words(cap + 1);
  D3_CUDA_OK(cudaMalloc(&s.scan_part, (sp > 1024 ? sp : 1024) * 4));
  s.cap = cap;
  return 0;
}

void scratch_free(ForceScratch &s) {
  cudaFree(s.draws); cudaFree(s.offsets); cudaFree(s.scan_part); cudaFree(s.counters);
  cudaFree(s.center); cudaFree(s.csum_recs); cudaFree(s.csum_counts); cudaFree(s.csum_part);
  cudaFree(s.csum_scan_part); cudaFree(s.csum_stamps);
  s = ForceScratch();
}

// ---------------------------------------------------------------------------
// Bottom-up passes (visitAfter). The many-body accumulation: the last child to
// finish computes its parent. The collide radii: a maximum, so each leaf
// raises its ancestors directly.
// ---------------------------------------------------------------------------

__device__ inline double ld_cg(const double *p) { return __ldcg(p); }

// A cell as the exact many-body traversal reads it, in one 64-byte load.
struct alignas(64) MRec {
  double x, y, value;
  double wt;              // (x1 - x0)^2 / theta2, as the opening test forms it
  uint32_t skip, head;    // head: the leaf's head node; NONE for an internal cell
  uint32_t first, count;  // the leaf's points in perm
};
static_assert(sizeof(MRec) == 64, "record layout");

// A parent's step of the accumulation: its children are the ones listed
// in its cell (several), or only the child just finished (one: no counter,
// and the child's values are still in registers).
struct Climb {
  uint32_t p;      // the parent (NONE at the root)
  uint32_t nch;    // its child count
};

__device__ inline Climb climb_up(const uint32_t *parent, const uint8_t *pnch, uint32_t cur) {
  Climb c;
  c.p = parent[cur];
  c.nch = pnch[cur];
  return c;
}

// A child's arrival at its parent: release orders the child's values before
// the count, acquire makes the earlier children's values visible to the last
// one (the counts on one parent form a release sequence).
__device__ inline uint32_t arrive_acq_rel(uint32_t *p) {
  uint32_t old;
  asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
  return old;
}

// many_body.zig:101-135 (accumulate). Leaf: head position, strength summed
// over the chain from perm[first + count - 1] down. Internal: children 0..3
// with a truthy |value|. Every cell's traversal record: the thread visiting
// an internal cell writes its fixed part (width test, skip link); the climb
// writes its centroid and charge.
// BLOCK: all by one block, `counter` in its shared memory.
template <bool BLOCK>
__device__ __forceinline__ void accumulate(Cell *cells, const uint32_t *parent, const uint8_t *pnch,
                                           uint32_t *counter, const uint32_t *perm,
                                           const uint32_t *skip, const double *xs, const double *ys,
                                           const double *strengths, double theta2, MRec *rec,
                                           uint32_t len) {
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < len; c += gridDim.x * blockDim.x) {
    Cell *q = &cells[c];
    if (!is_leaf(*q)) {
      const double w = q->x1 - q->x0;
      rec[c].wt = w * w / theta2;
      rec[c].skip = skip[c];
      rec[c].head = NONE;
      rec[c].first = 0;
      rec[c].count = 0;
      continue;
    }
    const uint32_t first = q->first, count = q->count;
    uint32_t head = perm[first + count - 1];
    double strength = 0;
    for (uint32_t k = first + count; k > first;) {
      --k;
      strength += strengths[perm[k]];
    }
    double cx = xs[head], cy = ys[head], cv = strength;
    q->x = cx;
    q->y = cy;
    q->value = cv;
    {
      const double w = q->x1 - q->x0;
      MRec r;
      r.x = cx; r.y = cy; r.value = cv; r.wt = w * w / theta2;
      r.skip = skip[c]; r.head = head; r.first = first; r.count = count;
      rec[c] = r;
    }
    auto finish = [&](uint32_t x) {
      cells[x].x = cx;
      cells[x].y = cy;
      cells[x].value = cv;
      rec[x].x = cx;
      rec[x].y = cy;
      rec[x].value = cv;
    };
    Climb up = climb_up(parent, pnch, c);
    for (;;) {
      const uint32_t p = up.p;
      if (p == NONE) break;
      if (up.nch == 1) {
        // A run of only children: p's only child is done, so p, p - 1, ...
        // (in preorder an only child follows its parent) while each is an
        // only child itself; their child counts read 8 at a time.
        uint8_t pk[8];
#pragma unroll
        for (int t = 0; t < 8; ++t) pk[t] = (uint32_t)t <= p ? pnch[p - t] : 0;
        bool out = false;
#pragma unroll
        for (int t = 0; t < 8; ++t) {
          const uint32_t x = p - t;
          double st = 0, weight = 0, sx = 0, sy = 0;
          const double w = fabs(cv);
          if (w > 0) {
            st += cv;
            weight += w;
            sx += w * cx;
            sy += w * cy;
          }
          cx = sx / weight;
          cy = sy / weight;
          cv = st;
          finish(x);
          if (pk[t] != 1) {
            up = climb_up(parent, pnch, x);
            out = true;
            break;
          }
        }
        if (!out) {
          up.p = p - 8;  // the eighth cell was an only child too
          up.nch = 1;
        }
        continue;
      }
      // The parent's links and child list were written by the tree build:
      // loaded before the arrival, so only the children's values wait on it.
      const Climb next = climb_up(parent, pnch, p);
      uint32_t ch[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) ch[k] = cells[p].child[k];
      if (BLOCK) {
        __threadfence_block();
        const uint32_t old = atomicAdd(&counter[p], 1u);
        __threadfence_block();
        if (old != up.nch - 1) break;
      } else if (arrive_acq_rel(&counter[p]) != up.nch - 1) {
        break;
      }
      double2 cxy[4], cvw[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (ch[k] == NONE) continue;
        const double2 *q0 = (const double2 *)&rec[ch[k]].x, *q1 = (const double2 *)&rec[ch[k]].value;
        cxy[k] = BLOCK ? *q0 : __ldcg(q0);
        cvw[k] = BLOCK ? *q1 : __ldcg(q1);
      }
      double st = 0, weight = 0, x = 0, y = 0;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (ch[k] == NONE) continue;
        double v = cvw[k].x;
        double w = fabs(v);
        if (w > 0) {
          st += v;
          weight += w;
          x += w * cxy[k].x;
          y += w * cxy[k].y;
        }
      }
      cx = x / weight;
      cy = y / weight;
      cv = st;
      finish(p);
      up = next;
    }
  }
}

__global__ void k_mb_accumulate(Cell *cells, const uint32_t *parent, const uint8_t *pnch,
                                uint32_t *counter, const uint32_t *perm, const uint32_t *skip,
                                const double *xs, const double *ys, const double *strengths,
                                double theta2, MRec *rec, const uint32_t *info) {
  accumulate<false>(cells, parent, pnch, counter, perm, skip, xs, ys, strengths, theta2, rec, info[1]);
}

// Small trees by one block: an arrival is a shared-memory atomic and the
// children's values come from this SM's L1, where the grid's arrivals go
// through L2 (1 us a level): 77 nodes 17 -> 12 us (event time). At 1,000
// nodes the one SM is busy longer than the grid's chain takes (27 / 22 us).
constexpr uint32_t ACC_BLOCK_NODES = 384, ACC_BLOCK_CELLS = 5120;  // (buffers of up to 1,024 nodes)

__global__ void __launch_bounds__(512) k_mb_accumulate_block(
    Cell *cells, const uint32_t *parent, const uint8_t *pnch, uint32_t *counter, const uint32_t *perm,
    const uint32_t *skip, const double *xs, const double *ys, const double *strengths, double theta2,
    MRec *rec, const uint32_t *info) {
  __shared__ uint32_t count[ACC_BLOCK_CELLS];
  const uint32_t len = info[1];
  if (len > ACC_BLOCK_CELLS) {  // (cell buffers of a simulation that was larger before)
    accumulate<false>(cells, parent, pnch, counter, perm, skip, xs, ys, strengths, theta2, rec, len);
    return;
  }
  for (uint32_t c = threadIdx.x; c < len; c += blockDim.x) count[c] = 0;
  __syncthreads();
  accumulate<true>(cells, parent, pnch, count, perm, skip, xs, ys, strengths, theta2, rec, len);
}

// collide.zig:117-129 (prepare): leaf radius of its head, internal the largest
// child radius (strict >, from 0). The internal rule makes a cell's radius
// max(+0, the positive radii of the leaf heads below it): a maximum, exact in
// any order. So no cell waits for its children: the tree build leaves every
// radius +0, each leaf with a positive radius raises its ancestors by 64-bit
// atomic maxima on the radius bits (the bit order of positive doubles is their
// numeric order), and stops at the first ancestor that already holds at least
// as much (whoever raised that one goes on from there). NaN, negative and zero
// leaf radii raise nothing, as in the strict comparison from 0.
__global__ void k_collide_prep(Cell *cells, const uint32_t *parent, const uint32_t *perm,
                               const double *radii, const uint32_t *info) {
  const uint32_t len = info[1];
  for (uint32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < len; c += gridDim.x * blockDim.x) {
    Cell *q = &cells[c];
    if (!is_leaf(*q)) continue;
    const double cr = radii[perm[q->first + q->count - 1]];
    q->r = cr;
    if (!(cr > 0)) continue;
    const unsigned long long bits = (unsigned long long)__double_as_longlong(cr);
    uint32_t p = parent[c];
    while (p != NONE) {
      // the next link is static: loaded alongside the maximum
      const uint32_t pp = parent[p];
      const unsigned long long old =
          atomicMax(reinterpret_cast<unsigned long long *>(&cells[p].r), bits);
      if (old >= bits) break;
      p = pp;
    }
  }
}

// ---------------------------------------------------------------------------
// Exact many-body traversal (many_body.zig:176-263)
// ---------------------------------------------------------------------------

// One target. RECORD: stop accumulating at the first zero delta d3 would
// jiggle, count the draws it would make, and do not write. Otherwise draws
// come from the stream at `draw0`.
template <bool RECORD>
__device__ __forceinline__ uint32_t mb_node(const MRec *rec, const uint32_t *perm,
                                   uint32_t len, const double *xs, const double *ys,
                                   double *vxs, double *vys, const double *strengths,
                                   const ManyBodyParams p, uint32_t i, const Rng *rng,
                                   uint64_t draw0) {
  const double nx = xs[i], ny = ys[i];
  double vx = vxs[i], vy = vys[i];
  uint32_t draws = 0;
  bool flagged = false;
  // The next cell follows from the current record alone (its skip link when
  // the cell is empty or far enough, else c + 1), so its load is issued
  // before this cell's arithmetic.
  uint32_t c = 0;
  MRec q;
  if (len) q = rec[0];
  while (c < len) {
    const MRec cq = q;
    const double value = cq.value;
    const bool live = value != 0 && value == value;
    double x = cq.x - nx, y = cq.y - ny;
    double l = x * x + y * y;
    const bool far = live && cq.wt < l;
    const uint32_t next = !live || far ? cq.skip : c + 1;
    if (next < len) q = rec[next];
    c = next;
    if (!live) continue;
    if (far) {
      if (l < p.dmax2) {
        if (RECORD && (x == 0 || y == 0)) {
          flagged = true;
          draws += (x == 0) + (y == 0);
        } else if (!flagged) {
          if (!RECORD) {
            if (x == 0) { x = (rng_draw_at(*rng, draw0 + draws++) - 0.5) * 1e-6; l += x * x; }
            if (y == 0) { y = (rng_draw_at(*rng, draw0 + draws++) - 0.5) * 1e-6; l += y * y; }
          }
          if (l < p.dmin2) l = sqrt(p.dmin2 * l);
          vx += x * value * p.alpha / l;
          vy += y * value * p.alpha / l;
        }
      }
      continue;
    }
    if (cq.head == NONE) continue;
    if (l >= p.dmax2) continue;
    const uint32_t first = cq.first, count = cq.count;
    const uint32_t head = cq.head;
    if (head != i || count > 1) {
      if (RECORD && (x == 0 || y == 0)) {
        flagged = true;
        draws += (x == 0) + (y == 0);
      } else if (!flagged) {
        if (!RECORD) {
          if (x == 0) { x = (rng_draw_at(*rng, draw0 + draws++) - 0.5) * 1e-6; l += x * x; }
          if (y == 0) { y = (rng_draw_at(*rng, draw0 + draws++) - 0.5) * 1e-6; l += y * y; }
        }
        if (l < p.dmin2) l = sqrt(p.dmin2 * l);
      }
    }
    if (!flagged) {
      for (uint32_t k = first + count; k > first;) {
        --k;
        const uint32_t j = perm[k];
        if (j != i) {
          const double wj = strengths[j] * p.alpha / l;
          vx += x * wj;
          vy += y * wj;
        }
      }
    }
  }
  if (!flagged) {
    vxs[i] = vx;
    vys[i] = vy;
  }
  return flagged ? draws : 0;
}

template <bool RECORD>
__device__ __noinline__ uint32_t mb_node_call(const MRec *rec, const uint32_t *perm, uint32_t len,
                                              const double *xs, const double *ys, double *vxs,
                                              double *vys, const double *strengths,
                                              const ManyBodyParams &p, uint32_t i, const Rng *rng,
                                              uint64_t draw0) {
  return mb_node<RECORD>(rec, perm, len, xs, ys, vxs, vys, strengths, p, i, rng, draw0);
}

// A warp's shared memory for one target (mb_warp): a bit per record, a stack
// of cells to visit (later the accepted records in order), a window's terms.
constexpr uint32_t MB_STACK = 1024;
__host__ __device__ inline uint32_t mb_warp_words(uint32_t records) {
  return MB_STACK + (records + 127) / 128 * 4;  // whole 16-byte units
}

// One target by a warp (all lanes with the same arguments). A thread per
// target is a chain of dependent steps, one per visited record (500 cycles
// each), and a small graph has no other targets to hide it; here the visit is
// spread over the lanes and only the sum is a chain. The visit itself needs no
// order: cells are popped 32 at a time from a stack, tested, and opened ones
// push their children; a record that adds a term sets its bit. Records are in
// preorder, so the set bits from the lowest up are the terms in visit order:
// they are formed 32 at a time and added one after the other, which gives
// mb_node's sums. (A stack that would overflow, at opening angles far below
// d3's, leaves the target to mb_node on one lane.) Returns as mb_node does.
template <bool RECORD>
__device__ uint32_t mb_warp(const MRec *rec, const Cell *cells, const uint32_t *perm, uint32_t len,
                            const double *xs, const double *ys, double *vxs, double *vys,
                            const double *strengths, const ManyBodyParams &p, uint32_t i,
                            const Rng *rng, uint64_t draw0, uint32_t *work, double2 *terms) {
  const unsigned lane = threadIdx.x & 31, full = 0xffffffffu, before = (1u << lane) - 1u;
  uint32_t *const stack = work, *const bits = work + MB_STACK;
  const uint32_t words = (len + 31) / 32;
  const double nx = xs[i], ny = ys[i];
  for (uint32_t w = lane; w < words; w += 32) bits[w] = 0;
  if (lane == 0) stack[0] = 0;
  __syncwarp();
  for (uint32_t sp = 1; sp;) {
    const uint32_t take = sp < 32 ? sp : 32;
    sp -= take;
    const bool in = lane < take;
    const uint32_t c = in ? stack[sp + lane] : 0;
    __syncwarp();
    uint2 ch[2] = {{NONE, NONE}, {NONE, NONE}};
    if (in) {
      const double x = rec[c].x - nx, y = rec[c].y - ny, value = rec[c].value, wt = rec[c].wt;
      const uint32_t head = rec[c].head;
      const double l = x * x + y * y;
      if (value != 0 && value == value) {
        if (wt < l) {
          if (l < p.dmax2) atomicOr(&bits[c >> 5], 1u << (c & 31));
        } else if (head != NONE) {
          if (!(l >= p.dmax2) && (head != i || rec[c].count > 1)) atomicOr(&bits[c >> 5], 1u << (c & 31));
        } else {
          const uint2 *child = reinterpret_cast<const uint2 *>(cells[c].child);
          ch[0] = child[0];
          ch[1] = child[1];
        }
      }
    }
    const uint32_t nch = (ch[0].x != NONE) + (ch[0].y != NONE) + (ch[1].x != NONE) + (ch[1].y != NONE);
    const unsigned b0 = __ballot_sync(full, nch & 1), b1 = __ballot_sync(full, nch & 2),
                   b2 = __ballot_sync(full, nch & 4);
    const uint32_t total = __popc(b0) + 2 * __popc(b1) + 4 * __popc(b2);
    if (sp + total > MB_STACK) {
      uint32_t d = 0;
      if (lane == 0)
        d = mb_node_call<RECORD>(rec, perm, len, xs, ys, vxs, vys, strengths, p, i, rng, draw0);
      return __shfl_sync(full, d, 0);
    }
    uint32_t at = sp + __popc(b0 & before) + 2 * __popc(b1 & before) + 4 * __popc(b2 & before);
    if (ch[0].x != NONE) stack[at++] = ch[0].x;
    if (ch[0].y != NONE) stack[at++] = ch[0].y;
    if (ch[1].x != NONE) stack[at++] = ch[1].x;
    if (ch[1].y != NONE) stack[at++] = ch[1].y;
    sp += total;
    __syncwarp();
  }
  double vx = vxs[i], vy = vys[i];
  uint32_t draws = 0;
  for (uint32_t w0 = 0; w0 < words; w0 += 32) {
    // the accepted records of 32 words, in order, into the stack's place
    unsigned set = w0 + lane < words ? bits[w0 + lane] : 0;
    if (!__any_sync(full, set)) continue;
    uint32_t incl = __popc(set);
    const uint32_t own = incl;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(full, incl, o);
      if (lane >= (unsigned)o) incl += v;
    }
    const uint32_t count = __shfl_sync(full, incl, 31);
    for (uint32_t at = incl - own; set; set &= set - 1) stack[at++] = (w0 + lane) * 32 + __ffs(set) - 1;
    __syncwarp();
    for (uint32_t k0 = 0; k0 < count; k0 += 32) {
      const uint32_t nt = count - k0 < 32 ? count - k0 : 32;
      const bool in = lane < nt;
      double x = 0, y = 0, l = 1;
      MRec q;
      q.head = q.first = 0;
      q.count = 1;
      if (in) {
        q = rec[stack[k0 + lane]];
        x = q.x - nx;
        y = q.y - ny;
        l = x * x + y * y;
      }
      const bool far = in && q.wt < l, zx = in && x == 0, zy = in && y == 0;
      if (__any_sync(full, zx || zy)) {
        const unsigned bx = __ballot_sync(full, zx), by = __ballot_sync(full, zy);
        if (!RECORD) {
          uint64_t d = draw0 + draws + __popc(bx & before) + __popc(by & before);
          if (zx) { x = (rng_draw_at(*rng, d++) - 0.5) * 1e-6; l += x * x; }
          if (zy) { y = (rng_draw_at(*rng, d) - 0.5) * 1e-6; l += y * y; }
        }
        draws += __popc(bx) + __popc(by);
      }
      if (RECORD && draws) continue;  // flagged: only the draws still count
      if (in && l < p.dmin2) l = sqrt(p.dmin2 * l);
      if (in) {
        // far: x value alpha / l, y value alpha / l; a leaf's point: x and y
        // times strength alpha / l (the same two divisions for both kinds)
        const double sv = far ? q.value : strengths[q.head];
        const double a = far ? x * sv * p.alpha : sv * p.alpha, b = far ? y * sv * p.alpha : a;
        const double qa = a / l, qb = b / l;
        terms[lane] = make_double2(far ? qa : x * qa, far ? qb : y * qa);
      }
      const unsigned many = __ballot_sync(full, in && !far && q.count > 1);
      __syncwarp();
      if (!many && nt == 32) {
#pragma unroll 8
        for (uint32_t k = 0; k < 32; ++k) {
          const double2 t = terms[k];
          vx += t.x;
          vy += t.y;
        }
      } else {
        for (uint32_t k = 0; k < nt; ++k) {
          if (!((many >> k) & 1u)) {
            vx += terms[k].x;
            vy += terms[k].y;
            continue;
          }
          // a leaf of coincident points: its points one by one
          const uint32_t first = __shfl_sync(full, q.first, k), points = __shfl_sync(full, q.count, k);
          const double lx = __shfl_sync(full, x, k), ly = __shfl_sync(full, y, k);
          const double ll = __shfl_sync(full, l, k);
          for (uint32_t k2 = first + points; k2 > first;) {
            --k2;
            const uint32_t j = perm[k2];
            if (j != i) {
              const double wj = strengths[j] * p.alpha / ll;
              vx += lx * wj;
              vy += ly * wj;
            }
          }
        }
      }
      __syncwarp();
    }
  }
  if (RECORD && draws) return draws;  // flagged: nothing written
  if (lane == 0) {
    vxs[i] = vx;
    vys[i] = vy;
  }
  return draws;
}

// Record pass over all nodes in Morton order (perm, then the NaN nodes).
__global__ void __launch_bounds__(128) k_mb_traverse(const MRec *rec,
                                                     const uint32_t *perm, const uint32_t *info,
                                                     const double *xs, const double *ys, double *vxs,
                                                     double *vys, const double *strengths,
                                                     ManyBodyParams p, uint32_t n, uint32_t *draws,
                                                     uint32_t *counters) {
  const uint32_t pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= n) return;
  // no tree this call (cell buffer overflow or a failed build launch): perm
  // may be stale, the velocities stay as they are
  if (info[5]) return;
  const uint32_t len = info[1];
  const uint32_t i = perm[pos];
  uint32_t d = len ? mb_node<true>(rec, perm, len, xs, ys, vxs, vys, strengths, p, i,
                                   nullptr, 0)
                   : 0;
  draws[i] = d;
  if (d) atomicAdd(&counters[1], 1u);
}

// The same by a warp a target (mb_warp); `words` of shared memory a warp.
__global__ void __launch_bounds__(128) k_mb_traverse_warp(
    const MRec *rec, const Cell *cells, const uint32_t *perm, const uint32_t *info, const double *xs,
    const double *ys, double *vxs, double *vys, const double *strengths, ManyBodyParams p, uint32_t n,
    uint32_t *draws, uint32_t *counters, uint32_t words) {
  extern __shared__ uint4 mb_smem[];
  __shared__ double2 terms[4][32];
  const uint32_t pos = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, warp = threadIdx.x >> 5;
  if (pos >= n || info[5]) return;
  const uint32_t len = info[1];
  const uint32_t i = perm[pos];
  uint32_t *work = reinterpret_cast<uint32_t *>(mb_smem) + (size_t)warp * words;
  const uint32_t d = len ? mb_warp<true>(rec, cells, perm, len, xs, ys, vxs, vys, strengths, p, i,
                                         nullptr, 0, work, terms[warp])
                         : 0;
  if ((threadIdx.x & 31) != 0) return;
  draws[i] = d;
  if (d) atomicAdd(&counters[1], 1u);
}

// The flagged ones of nodes i0 .. i0 + 31: one after the other by the whole
// warp when a bit per record fits its `words` of shared memory (a flagged
// node, 4 % of them where coincident ones are in play, is a chain that takes
// one thread as long as the whole record pass), else a lane each.
__device__ void mb_rerun_warp(const MRec *rec, const Cell *cells, const uint32_t *perm, uint32_t len,
                              const double *xs, const double *ys, double *vxs, double *vys,
                              const double *strengths, const ManyBodyParams &p, uint32_t n,
                              uint32_t i0, const uint32_t *draws, const uint32_t *offsets,
                              const Rng *rng, uint32_t *work, uint32_t words, double2 *terms) {
  const uint32_t i = i0 + (threadIdx.x & 31);
  const bool mine = i < n && __ldcg(&draws[i]) != 0;
  const uint32_t off = mine ? __ldcg(&offsets[i]) : 0;
  if (mb_warp_words(len) > words) {
    if (mine) mb_node_call<false>(rec, perm, len, xs, ys, vxs, vys, strengths, p, i, rng, off);
    return;
  }
  unsigned flagged = __ballot_sync(0xffffffffu, mine);
  while (flagged) {
    const unsigned b = __ffs(flagged) - 1;
    flagged &= flagged - 1;
    mb_warp<false>(rec, cells, perm, len, xs, ys, vxs, vys, strengths, p, i0 + b, rng,
                   __shfl_sync(0xffffffffu, off, b), work, terms);
    __syncwarp();
  }
}

// Flagged nodes again, each from its own offset in the draw stream (the
// exclusive scan of draws over node index = d3's draw order).
__global__ void __launch_bounds__(128) k_mb_rerun(const MRec *rec, const Cell *cells,
                                                  const uint32_t *perm, const uint32_t *info,
                                                  const double *xs, const double *ys, double *vxs,
                                                  double *vys, const double *strengths,
                                                  ManyBodyParams p, uint32_t n,
                                                  const uint32_t *draws, const uint32_t *offsets,
                                                  const uint32_t *counters, const Rng *rng,
                                                  uint32_t words) {
  extern __shared__ uint4 mb_smem[];
  if (counters[1] == 0 || info[5]) return;
  __shared__ double2 terms[4][32];
  const uint32_t i0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u;
  mb_rerun_warp(rec, cells, perm, info[1], xs, ys, vxs, vys, strengths, p, n, i0, draws, offsets, rng,
                reinterpret_cast<uint32_t *>(mb_smem) + (size_t)(threadIdx.x >> 5) * words, words,
                terms[threadIdx.x >> 5]);
}

// The jiggle draws of the flagged targets, after the record pass, in one
// cooperative launch (device LCG): the exclusive scan of the draw counts over
// node index (d3's draw order), the flagged targets again from their stream
// positions, then the LCG advanced past all the draws. Nothing to do (the
// usual case) is decided by every block alike from the flagged count.
__global__ void __launch_bounds__(256) k_mb_draws(const MRec *rec, const Cell *cells, const uint32_t *perm,
                                                  const uint32_t *info, const double *xs,
                                                  const double *ys, double *vxs, double *vys,
                                                  const double *strengths, ManyBodyParams p,
                                                  uint32_t n, const uint32_t *draws,
                                                  uint32_t *offsets, uint32_t *counters,
                                                  uint32_t *bsum, Rng *rng, uint32_t words) {
  extern __shared__ uint4 mb_smem[];
  __shared__ double2 terms[8][32];
  if (__ldcg(&counters[1]) == 0 || __ldcg(&info[5])) return;
  cg::grid_group g = cg::this_grid();
  const uint32_t total = grid_excl_scan(g, draws, offsets, n, bsum);
  g.sync();
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  const uint32_t len = info[1];
  for (uint32_t i0 = tid & ~31u; i0 < n; i0 += nth)
    mb_rerun_warp(rec, cells, perm, len, xs, ys, vxs, vys, strengths, p, n, i0, draws, offsets, rng,
                  reinterpret_cast<uint32_t *>(mb_smem) + (size_t)(threadIdx.x >> 5) * words, words,
                  terms[threadIdx.x >> 5]);
  g.sync();
  if (tid == 0) {
    counters[0] = total;
    if (rng->mode == 0) rng->lcg = lcg_skip(rng->lcg, total);
    else rng->pos += total;
  }
}

__global__ void k_rng_advance(Rng *rng, const uint32_t *total) {
  uint32_t t = *total;
  if (t == 0) return;
  if (rng->mode == 0) rng->lcg = lcg_skip(rng->lcg, t);
  else rng->pos += t;
}

static void climb_grid(unsigned &blocks, unsigned &threads, uint32_t cap) {
  threads = 256;
  blocks = blocks_for(cap, threads);
  if (blocks > 148 * 16) blocks = 148 * 16;
}

// Shared memory of k_mb_draws, two blocks of 8 warps an SM: a bit per record
// up to 32,000 records (the trees of about 19,000 nodes). No more: the center
// sum on the side stream holds 64 KB of one SM, and a cooperative launch waits
// until all its blocks have room.
constexpr size_t MB_DRAWS_SMEM = 64 * 1024;

// The record pass: a warp per target up to MB_WARP_NODES nodes, a thread per
// target above (event time, warp / thread: 77 nodes 22 / 41 us, 1,000 27 / 62,
// 3,000 35 / 70, 5,003 56 / 72, 7,000 67 / 75, 10,000 113 / 80: a target takes
// about 3,300 warp instructions, which 148 SMs issue in the time of the
// longest serial visit at 8,000 targets).
constexpr uint32_t MB_WARP_NODES = 7000;

static bool launch_traverse(TreeDev &t, const NodeArrays &a, const double *strengths,
                            const ManyBodyParams &p, ForceScratch &s, cudaStream_t st) {
  const uint32_t n = a.n;
  const MRec *rec = (const MRec *)t.rec;
  // four warps a block: at most 42 KB (the cell buffers may be larger than n asks for)
  const uint32_t words = mb_warp_words(t.cells_cap);
  if (n <= MB_WARP_NODES && 16 * words <= 42 * 1024 &&
      launch(k_mb_traverse_warp, blocks_for(n * 32ull, 128), 128, 16 * words, st, rec, t.cells, t.perm,
             t.info, a.x, a.y, a.vx, a.vy, strengths, p, n, s.draws, s.counters, words))
    return true;
  return launch(k_mb_traverse, blocks_for(n, 128), 128, 0, st, rec, t.perm, t.info, a.x, a.y, a.vx,
                a.vy, strengths, p, n, s.draws, s.counters);
}

void many_body_exact(TreeDev &t, const NodeArrays &a, const double *strengths,
                     const ManyBodyParams &p, Rng *rng, ForceScratch &s, uint32_t *status,
                     bool host_draws, cudaStream_t st, const std::function<void(int)> &mark) {
  const uint32_t n = a.n;
  tree_build(t, a.x, a.y, n, status, st);
  if (mark) mark(0);
  if (n == 0) return;
  unsigned cb, ct;
  climb_grid(cb, ct, t.cells_cap);
  bool ran = n <= ACC_BLOCK_NODES &&
             launch(k_mb_accumulate_block, 1, 512, 0, st, t.cells, t.parent, t.pnch, t.counter, t.perm,
                    t.skip, a.x, a.y, strengths, p.theta2, (MRec *)t.rec, t.info);
  ran = ran || launch(k_mb_accumulate, cb, ct, 0, st, t.cells, t.parent, t.pnch, t.counter, t.perm,
                      t.skip, a.x, a.y, strengths, p.theta2, (MRec *)t.rec, t.info);
  if (mark) mark(1);
  cudaMemsetAsync(s.counters, 0, 2 * sizeof(uint32_t), st);
  if (!ran || !launch_traverse(t, a, strengths, p, s, st)) tree_failed(t, status, st);
  if (host_draws) {
    scan_u32(s.draws, s.offsets, n, s.scan_part, s.counters, st);
    return;
  }
  static int blocks = 0;
  if (!blocks) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    open_shared<k_mb_draws>(MB_DRAWS_SMEM);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_mb_draws, 256, MB_DRAWS_SMEM);
    blocks = sms * (per >= 2 ? 2 : (per > 0 ? per : 1));
  }
  const MRec *rec = (const MRec *)t.rec;
  const Cell *cells = t.cells;
  const uint32_t *perm = t.perm, *info = t.info;
  const double *x = a.x, *y = a.y;
  double *vx = a.vx, *vy = a.vy;
  ManyBodyParams pp = p;
  uint32_t nn = n, words = (uint32_t)(MB_DRAWS_SMEM / 32);  // of 8 warps
  const uint32_t *draws = s.draws;
  uint32_t *offsets = s.offsets, *counters = s.counters, *bsum = s.scan_part;
  void *params[] = {&rec, &cells, &perm, &info, &x, &y, &vx, &vy, &strengths, &pp, &nn, &draws,
                    &offsets, &counters, &bsum, &rng, &words};
  ++g_launches;
  if (!open_shared<k_mb_draws>(MB_DRAWS_SMEM) ||
      cudaLaunchCooperativeKernel((const void *)k_mb_draws, blocks, 256, params, MB_DRAWS_SMEM, st) !=
          cudaSuccess) {
    cudaGetLastError();
    scan_u32(s.draws, s.offsets, n, s.scan_part, s.counters, st);
    many_body_rerun(t, a, strengths, p, rng, s, st);
  }
}

void many_body_rerun(TreeDev &t, const NodeArrays &a, const double *strengths,
                     const ManyBodyParams &p, Rng *rng, ForceScratch &s, cudaStream_t st) {
  const uint32_t n = a.n;
  constexpr uint32_t words = 48 * 1024 / 16;  // of 4 warps, 47 KB in all
  D3_LAUNCH(k_mb_rerun, blocks_for(n, 128), 128, (words - 256) * 16, st)(
      (const MRec *)t.rec, t.cells, t.perm, t.info, a.x, a.y, a.vx, a.vy, strengths, p, n, s.draws,
      s.offsets, s.counters, rng, words - 256);
  D3_LAUNCH(k_rng_advance, 1, 1, 0, st)(rng, s.counters);
}

// ---------------------------------------------------------------------------
// Exact link (link.zig:8-40)
// ---------------------------------------------------------------------------

static bool link_in_block(uint32_t nodes);

int link_plan_build(LinkPlan &plan, const uint32_t *src, const uint32_t *tgt, uint32_t m,
                    cudaStream_t st) {
  // level(e) = 1 + the largest level of an earlier link sharing a node, so
  // every link sees exactly the velocities its predecessors wrote.
  uint32_t nmax = 0;
  bool self = false;
  for (uint32_t e = 0; e < m; ++e) {
    if (src[e] + 1 > nmax) nmax = src[e] + 1;
    if (tgt[e] + 1 > nmax) nmax = tgt[e] + 1;
    self = self || src[e] == tgt[e];
  }
  std::vector<uint32_t> node_level(nmax, 0), level(m);
  uint32_t levels = 0;
  for (uint32_t e = 0; e < m; ++e) {
    uint32_t l = (node_level[src[e]] > node_level[tgt[e]] ? node_level[src[e]] : node_level[tgt[e]]) + 1;
    level[e] = l;
    node_level[src[e]] = l;
    node_level[tgt[e]] = l;
    if (l > levels) levels = l;
  }
  std::vector<uint32_t> start(levels + 2, 0), order(m > 0 ? m : 1), place(m > 0 ? m : 1);
  for (uint32_t e = 0; e < m; ++e) start[level[e]]++;
  uint32_t run = 0, width = 0;
  for (uint32_t l = 0; l <= levels + 1; ++l) {
    uint32_t c = start[l];
    start[l] = run;
    run += c;
    width = c > width ? c : width;
  }
  std::vector<uint32_t> fill(start.begin(), start.end());
  for (uint32_t e = 0; e < m; ++e) {
    place[e] = fill[level[e]]++;
    order[place[e]] = e;
  }
  // per link in level order: its ends, each marked if no earlier link touches
  // it, and where each end's velocity goes on to: the next link's input
  // (2 x its place, + 1 for its target side) or nowhere (NONE: the last one)
  std::vector<LinkEnds> ends(m > 0 ? m : 1);
  std::vector<uint32_t> later(nmax, NONE);
  for (uint32_t e = m; e-- > 0;) {
    LinkEnds &r = ends[place[e]];
    r.next_src = later[src[e]];
    r.next_tgt = later[tgt[e]];
    r.src = src[e];
    r.tgt = tgt[e];
    later[src[e]] = 2 * place[e];
    later[tgt[e]] = 2 * place[e] + 1;
  }
  for (uint32_t i = 0; i < nmax; ++i)
    if (later[i] != NONE) {
      LinkEnds &r = ends[later[i] >> 1];
      if (later[i] & 1) r.tgt |= LINK_FIRST;
      else r.src |= LINK_FIRST;
    }
  link_plan_free(plan);
  const bool in_block = link_in_block(nmax);
  // one allocation and one copy: the plan's tables and the zeroed tally, then
  // the constants and (for k_link_flow) the messages. Copy and fill go on the
  // stream of the launches that read them: it does not wait for the default
  // stream, where either may still be under way when the call returns, and a
  // link would take what the memory held before for its velocity.
  const auto room = [](size_t bytes) { return (bytes + 255) / 256 * 256; };
  const size_t at_order = room(ends.size() * sizeof(LinkEnds)),
               at_start = at_order + room(order.size() * 4), at_tally = at_start + room(start.size() * 4),
               at_par = at_tally + room(3 * sizeof(uint32_t)),
               at_msg = at_par + room(ends.size() * 3 * sizeof(double)),
               msg_bytes = in_block ? 0 : ends.size() * 2 * sizeof(double2);
  std::vector<unsigned char> image(at_par, 0);
  memcpy(image.data(), ends.data(), ends.size() * sizeof(LinkEnds));
  memcpy(image.data() + at_order, order.data(), order.size() * 4);
  memcpy(image.data() + at_start, start.data(), start.size() * 4);
  unsigned char *block = nullptr;
  D3_CUDA_OK(cudaMalloc(&block, at_msg + msg_bytes));
  plan.ends = reinterpret_cast<LinkEnds *>(block);
  plan.order = reinterpret_cast<uint32_t *>(block + at_order);
  plan.level_start = reinterpret_cast<uint32_t *>(block + at_start);
  plan.tally = reinterpret_cast<uint32_t *>(block + at_tally);
  plan.par = reinterpret_cast<double *>(block + at_par);
  plan.msg = reinterpret_cast<double2 *>(block + at_msg);
  D3_CUDA_OK(cudaMemcpyAsync(block, image.data(), at_par, cudaMemcpyHostToDevice, st));
  if (msg_bytes) D3_CUDA_OK(cudaMemsetAsync(plan.msg, 0xff, msg_bytes, st));  // no message yet
  plan.h_level_start = new uint32_t[start.size()];
  for (size_t k = 0; k < start.size(); ++k) plan.h_level_start[k] = start[k];
  plan.m = m;
  plan.levels = levels;
  plan.nodes = nmax;
  plan.width = width;
  plan.self = self;
  plan.in_block = in_block;
  plan.gathered = false;
  return 0;
}

void link_plan_free(LinkPlan &plan) {
  cudaFree(plan.ends);  // the block of all device arrays
  delete[] plan.h_level_start;
  plan = LinkPlan();
}

// The links' distance, strength and bias in plan order (three planes), once
// per plan (an upload of the link force makes a new plan).
__global__ void k_link_params(LinkArrays l, const uint32_t *order, double *par) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= l.m) return;
  const uint32_t e = order[p];
  par[p] = l.distance[e];
  par[(size_t)l.m + p] = l.strength[e];
  par[2 * (size_t)l.m + p] = l.bias[e];
}

// One link, d3's statement order. Returns false (writing nothing) where d3
// would draw from `random`.
__device__ inline bool link_one(double *xs, double *ys, double *vxs, double *vys, const LinkArrays l,
                                uint32_t e, double alpha) {
  const uint32_t src = l.source[e], tgt = l.target[e];
  double x = xs[tgt] + vxs[tgt] - xs[src] - vxs[src];
  double y = ys[tgt] + vys[tgt] - ys[src] - vys[src];
  if (x == 0 || x != x || y == 0 || y != y) return false;
  double len = sqrt(x * x + y * y);
  len = (len - l.distance[e]) / len * alpha * l.strength[e];
  x *= len;
  y *= len;
  double b = l.bias[e];
  vxs[tgt] -= x * b;
  vys[tgt] -= y * b;
  b = 1 - b;
  vxs[src] += x * b;
  vys[src] += y * b;
  return true;
}

__global__ void k_link_level(double *xs, double *ys, double *vxs, double *vys, LinkArrays l,
                             const uint32_t *order, uint32_t lo, uint32_t hi, double alpha,
                             uint32_t *flag) {
  uint32_t k = lo + blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= hi) return;
  if (!link_one(xs, ys, vxs, vys, l, order[k], alpha)) atomicOr(flag, 1u);
}

__global__ void k_restore_v(double *vx, double *vy, const double *svx, const double *svy, uint32_t n,
                            const uint32_t *flag) {
  if (*flag == 0) return;
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  vx[i] = svx[i];
  vy[i] = svy[i];
}

__global__ void k_save_v(double *svx, double *svy, const double *vx, const double *vy, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  svx[i] = vx[i];
  svy[i] = vy[i];
}

// link.zig:8-40 on one thread, drawing from the device LCG.
__device__ void link_serial_lcg(const double *xs, const double *ys, double *vxs, double *vys,
                                const LinkArrays &l, double alpha, double iterations, Rng *rng,
                                uint32_t *status, uint32_t why = ST_LINK_JIGGLE) {
  atomicOr(status, why);
  uint32_t s = rng->lcg;
  for (double k = 0; k < iterations; k += 1) {
    for (uint32_t i = 0; i < l.m; ++i) {
      const uint32_t src = l.source[i], tgt = l.target[i];
      double x = xs[tgt] + vxs[tgt] - xs[src] - vxs[src];
      if (x == 0 || x != x) { s = lcg_step(s); x = (lcg_value(s) - 0.5) * 1e-6; }
      double y = ys[tgt] + vys[tgt] - ys[src] - vys[src];
      if (y == 0 || y != y) { s = lcg_step(s); y = (lcg_value(s) - 0.5) * 1e-6; }
      double len = sqrt(x * x + y * y);
      len = (len - l.distance[i]) / len * alpha * l.strength[i];
      x *= len;
      y *= len;
      double b = l.bias[i];
      vxs[tgt] -= x * b;
      vys[tgt] -= y * b;
      b = 1 - b;
      vxs[src] += x * b;
      vys[src] += y * b;
    }
  }
  rng->lcg = s;
}

__global__ void k_link_serial(double *xs, double *ys, double *vxs, double *vys, LinkArrays l,
                              double alpha, double iterations, Rng *rng, const uint32_t *flag,
                              uint32_t *status) {
  if (*flag == 0) return;
  link_serial_lcg(xs, ys, vxs, vys, l, alpha, iterations, rng, status);
}

// The same with draws pulled by the host: resumes at (resume[0], resume[1]),
// stops before a link whose draws are not in the buffer yet.
__global__ void k_link_serial_host(double *xs, double *ys, double *vxs, double *vys, LinkArrays l,
                                   double alpha, double iterations, Rng *rng, uint32_t *resume) {
  uint64_t used = 0, avail = rng->avail - rng->pos;
  const double *buf = rng->buf + rng->pos;
  uint32_t it = resume[0], i0 = resume[1];
  for (double k = (double)it; k < iterations; k += 1, ++it, i0 = 0) {
    for (uint32_t i = i0; i < l.m; ++i) {
      const uint32_t src = l.source[i], tgt = l.target[i];
      double x = xs[tgt] + vxs[tgt] - xs[src] - vxs[src];
      double y = ys[tgt] + vys[tgt] - ys[src] - vys[src];
      uint32_t need = (x == 0 || x != x) + (y == 0 || y != y);
      if (used + need > avail) {
        resume[0] = it;
        resume[1] = i;
        resume[2] = (uint32_t)(used + need - avail);
        rng->pos += used;
        return;
      }
      if (x == 0 || x != x) x = (buf[used++] - 0.5) * 1e-6;
      if (y == 0 || y != y) y = (buf[used++] - 0.5) * 1e-6;
      double len = sqrt(x * x + y * y);
      len = (len - l.distance[i]) / len * alpha * l.strength[i];
      x *= len;
      y *= len;
      double b = l.bias[i];
      vxs[tgt] -= x * b;
      vys[tgt] -= y * b;
      b = 1 - b;
      vxs[src] += x * b;
      vys[src] += y * b;
    }
  }
  resume[2] = 0;
  rng->pos += used;
}

__device__ inline unsigned long long globaltimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

struct LinkFlowArgs {
  const double *xs, *ys;
  double *vxs, *vys, *svx, *svy;
  LinkArrays l;
  const LinkEnds *ends;
  const double *par;           // distance, strength, bias planes
  const uint32_t *level_start; // k_link_block
  ulonglong2 *msg;             // k_link_flow: two inputs per link, all ones = nothing yet
  uint32_t *tally;             // k_link_flow: blocks done, failure bits, progress
  uint32_t levels, nodes;
  double alpha, iterations;
  uint32_t *flag;
  Rng *rng;           // with serial_lcg: the serial pass's draws
  uint32_t *status;
  int serial_lcg;     // a met jiggle is resolved in the launch (device LCG)
  unsigned sleep_ns;  // pause between polls of a wait (after the first eight)
};

struct LinkPar {
  double dist, str, bias;
};

// One link on the velocities of its ends, d3's statement order. False
// (nothing changed) where d3 would draw from `random`.
__device__ __forceinline__ bool link_apply(const LinkPar &c, double xt, double yt, double xs,
                                           double ys, double alpha, double2 &vt, double2 &vs) {
  double x = xt + vt.x - xs - vs.x;
  double y = yt + vt.y - ys - vs.y;
  if (x == 0 || x != x || y == 0 || y != y) return false;
  double len = sqrt(x * x + y * y);
  len = (len - c.dist) / len * alpha * c.str;
  x *= len;
  y *= len;
  double b = c.bias;
  vt.x -= x * b;
  vt.y -= y * b;
  b = 1 - b;
  vs.x += x * b;
  vs.y += y * b;
  return true;
}

__device__ __forceinline__ LinkPar link_par(const LinkFlowArgs &a, uint32_t p) {
  return {a.par[p], a.par[(size_t)a.l.m + p], a.par[2 * (size_t)a.l.m + p]};
}

// The pass of a graph whose nodes fit one SM: a block keeps every node's
// velocity and position in shared memory and takes the links level by level,
// a barrier between levels. A level costs the chain of one link (shared
// loads, sqrt, division) and the barrier, about 1 us; its links' constants are
// loaded during the level before. The node arrays are written only if no link
// met a jiggle; if one did, they are still the pass's start for the serial
// pass. A level's links share no node: at most half the nodes, so the block is
// as wide as the widest level.
constexpr uint32_t LINK_BLOCK_NODES = 7000;  // 32 bytes each in 227 KB

__global__ void __launch_bounds__(1024) k_link_block(LinkFlowArgs a) {
  extern __shared__ double2 link_smem[];
  double2 *const V = link_smem, *const P = link_smem + a.nodes;
  const uint32_t t = threadIdx.x, nt = blockDim.x, m = a.l.m;
  for (uint32_t i = t; i < a.nodes; i += nt) {
    V[i] = make_double2(a.vxs[i], a.vys[i]);
    P[i] = make_double2(a.xs[i], a.ys[i]);
  }
  bool bad = false;
  auto run = [&](const LinkEnds &r, const LinkPar &c) {
    const uint32_t s = r.src & ~LINK_FIRST, d = r.tgt & ~LINK_FIRST;
    const double2 pt = P[d], ps = P[s];
    double2 vt = V[d], vs = V[s];
    if (!link_apply(c, pt.x, pt.y, ps.x, ps.y, a.alpha, vt, vs)) {
      bad = true;
      return;
    }
    V[d] = vt;
    V[s] = vs;
  };
  for (double k = 0; k < a.iterations; k += 1) {
    uint32_t lo = 0, hi = a.level_start[2];  // level 1 starts at place 0
    LinkEnds r;
    LinkPar c;
    if (t < hi) {
      r = a.ends[t];
      c = link_par(a, t);
    }
    __syncthreads();
    for (uint32_t lv = 1; lv <= a.levels; ++lv) {
      const uint32_t nhi = lv < a.levels ? a.level_start[lv + 2] : m;
      LinkEnds rn;
      LinkPar cn;
      if (lv < a.levels && hi + t < nhi) {
        rn = a.ends[hi + t];
        cn = link_par(a, hi + t);
      }
      if (lo + t < hi) run(r, c);
      for (uint32_t p = lo + nt + t; p < hi; p += nt) run(a.ends[p], link_par(a, p));
      __syncthreads();
      r = rn;
      c = cn;
      lo = hi;
      hi = nhi;
    }
  }
  bad = __syncthreads_or(bad);
  if (t == 0) *a.flag = bad;
  if (bad) {
    if (a.serial_lcg && t == 0)
      link_serial_lcg(a.xs, a.ys, a.vxs, a.vys, a.l, a.alpha, a.iterations, a.rng, a.status);
    return;
  }
  for (uint32_t i = t; i < a.nodes; i += nt) {
    a.vxs[i] = V[i].x;
    a.vys[i] = V[i].y;
  }
}

// Whether a plan over `nodes` nodes runs in one block.
static bool link_in_block(uint32_t nodes) {
  return nodes <= LINK_BLOCK_NODES && open_shared<k_link_block>(LINK_BLOCK_NODES * 2 * sizeof(double2));
}

// A link's input from the link before it on one of its nodes, or all ones in
// either half while that has not come. Each half is a 64-bit access and is
// looked at by itself, so the halves need not arrive together; the value is
// the message, so nothing else is ordered by it. (A velocity whose bits are
// all ones, a NaN no arithmetic gives, runs the wait out: the serial pass.)
__device__ __forceinline__ ulonglong2 msg_read(const ulonglong2 *p) {
  ulonglong2 v;
  asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(v.x), "=l"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void msg_write(ulonglong2 *p, unsigned long long x, unsigned long long y) {
  asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(x), "l"(y) : "memory");
}

constexpr uint32_t LINK_MET_JIGGLE = 1, LINK_GAVE_UP = 2;

// The pass as messages, in one cooperative launch: threads take the links in
// level order; a link waits (until no 64th link was done for 20 ms: a chain of
// any length goes on) for the velocities of its two nodes from the links before it there, each a 16-byte message in a place
// of its own, and hands them on to the links after it. A level costs one
// message through L2 and one link's arithmetic (1.6 us; 5 us with finished
// counts and the velocities read after an acquire). The first link on a node
// reads its velocity and saves it, the last one writes it. A read message is
// cleared for the next pass. If a link met a zero or NaN delta or gave up, the
// last block puts the saved velocities back and runs the serial pass.
// The work of a ready link is inside the polling loop: a lane never waits at
// a convergence point for a lane that waits for its message.
__global__ void __launch_bounds__(256) k_link_flow(LinkFlowArgs a) {
  const uint32_t tid = blockIdx.x * blockDim.x + threadIdx.x, nth = gridDim.x * blockDim.x;
  const uint32_t m = a.l.m;
  const unsigned long long none = ~0ull;
  uint32_t bad = 0;
  for (double k = 0; k < a.iterations; k += 1) {
    if (k > 0) cg::this_grid().sync();  // the last iteration's velocities and cleared messages
    uint32_t p = tid;
    LinkEnds r;
    LinkPar c;
    double2 pt, ps;
    ulonglong2 in_s, in_t;
    bool fresh = true;
    unsigned long long t0 = 0;
    uint32_t polls = 0, seen = 0;
    while (p < m) {
      if (fresh) {
        fresh = false;
        polls = 0;
        r = a.ends[p];
        c = link_par(a, p);
        const uint32_t s = r.src & ~LINK_FIRST, d = r.tgt & ~LINK_FIRST;
        pt = make_double2(a.xs[d], a.ys[d]);
        ps = make_double2(a.xs[s], a.ys[s]);
        in_s = in_t = make_ulonglong2(none, none);
        if (r.src & LINK_FIRST) {
          const double x = __ldcg(&a.vxs[s]), y = __ldcg(&a.vys[s]);
          if (k == 0) {
            a.svx[s] = x;
            a.svy[s] = y;
          }
          in_s = make_ulonglong2(__double_as_longlong(x), __double_as_longlong(y));
        }
        if (r.tgt & LINK_FIRST) {
          const double x = __ldcg(&a.vxs[d]), y = __ldcg(&a.vys[d]);
          if (k == 0) {
            a.svx[d] = x;
            a.svy[d] = y;
          }
          in_t = make_ulonglong2(__double_as_longlong(x), __double_as_longlong(y));
        }
      }
      bool gave_up = false;
      if (!(r.src & LINK_FIRST) && (in_s.x == none || in_s.y == none)) in_s = msg_read(&a.msg[2 * (size_t)p]);
      if (!(r.tgt & LINK_FIRST) && (in_t.x == none || in_t.y == none)) in_t = msg_read(&a.msg[2 * (size_t)p + 1]);
      const bool have_s = (r.src & LINK_FIRST) || (in_s.x != none && in_s.y != none);
      const bool have_t = (r.tgt & LINK_FIRST) || (in_t.x != none && in_t.y != none);
      if (!(have_s && have_t)) {
        if (polls == 0) t0 = globaltimer_ns();
        ++polls;
        if (polls > 8 && a.sleep_ns) __nanosleep(a.sleep_ns);
        if ((polls & 15) == 0 && globaltimer_ns() - t0 > 20000000ull) {
          const uint32_t done = *(volatile const uint32_t *)&a.tally[2];
          gave_up = done == seen;  // (counted on from 0: a first look sees any progress)
          seen = done;
          t0 = globaltimer_ns();
        }
      }
      if ((have_s && have_t) || gave_up) {
        const uint32_t s = r.src & ~LINK_FIRST, d = r.tgt & ~LINK_FIRST;
        if (gave_up) bad |= LINK_GAVE_UP;
        double2 vs = make_double2(__longlong_as_double(in_s.x), __longlong_as_double(in_s.y));
        double2 vt = make_double2(__longlong_as_double(in_t.x), __longlong_as_double(in_t.y));
        if (gave_up) vs = vt = make_double2(0, 0);  // the pass is put back: only keep the others going
        else if (!link_apply(c, pt.x, pt.y, ps.x, ps.y, a.alpha, vt, vs)) bad |= LINK_MET_JIGGLE;
        if (r.next_src != NONE) {
          msg_write(&a.msg[r.next_src], __double_as_longlong(vs.x), __double_as_longlong(vs.y));
        } else {
          a.vxs[s] = vs.x;
          a.vys[s] = vs.y;
        }
        if (r.next_tgt != NONE) {
          msg_write(&a.msg[r.next_tgt], __double_as_longlong(vt.x), __double_as_longlong(vt.y));
        } else {
          a.vxs[d] = vt.x;
          a.vys[d] = vt.y;
        }
        if (!(r.src & LINK_FIRST)) msg_write(&a.msg[2 * (size_t)p], none, none);
        if (!(r.tgt & LINK_FIRST)) msg_write(&a.msg[2 * (size_t)p + 1], none, none);
        if ((p & 63) == 0) atomicAdd(&a.tally[2], 1u);
        p += nth;
        fresh = true;
      }
    }
  }
  // the block that ends last sees every block's writes
  __shared__ uint32_t bits;
  const bool any_jiggle = __syncthreads_or(bad & LINK_MET_JIGGLE);
  const bool any_gave_up = __syncthreads_or(bad & LINK_GAVE_UP);
  if (threadIdx.x == 0) {
    if (any_jiggle || any_gave_up)
      atomicOr(&a.tally[1], (any_jiggle ? LINK_MET_JIGGLE : 0u) | (any_gave_up ? LINK_GAVE_UP : 0u));
    __threadfence();
    bits = NONE;
    if (atomicAdd(&a.tally[0], 1u) == gridDim.x - 1) {
      __threadfence();
      bits = atomicExch(&a.tally[1], 0u);
      a.tally[0] = a.tally[2] = 0;
      *a.flag = bits != 0;
    }
  }
  __syncthreads();
  if (bits == NONE || bits == 0) return;
  for (uint32_t p = threadIdx.x; p < m; p += blockDim.x) {
    const LinkEnds r = a.ends[p];
    const uint32_t s = r.src & ~LINK_FIRST, d = r.tgt & ~LINK_FIRST;
    if (r.src & LINK_FIRST) {
      a.vxs[s] = __ldcg(&a.svx[s]);
      a.vys[s] = __ldcg(&a.svy[s]);
    }
    if (r.tgt & LINK_FIRST) {
      a.vxs[d] = __ldcg(&a.svx[d]);
      a.vys[d] = __ldcg(&a.svy[d]);
    }
    if (bits & LINK_GAVE_UP) {  // messages nobody took
      msg_write(&a.msg[2 * (size_t)p], none, none);
      msg_write(&a.msg[2 * (size_t)p + 1], none, none);
    }
  }
  __syncthreads();
  if (a.serial_lcg && threadIdx.x == 0)
    link_serial_lcg(a.xs, a.ys, a.vxs, a.vys, a.l, a.alpha, a.iterations, a.rng, a.status,
                    (bits & LINK_MET_JIGGLE ? ST_LINK_JIGGLE : 0) | (bits & LINK_GAVE_UP ? ST_LINK_GAVE_UP : 0));
}

__global__ void k_link_flag(uint32_t *flag) { *flag = 1; }

void link_exact(const NodeArrays &a, const LinkArrays &l, LinkPlan &plan, double alpha,
                double iterations, Rng *rng, uint32_t *flag, uint32_t *status, bool serial_lcg,
                cudaStream_t st) {
  if (l.m == 0) return;
  const uint32_t n = a.n;
  if (plan.self) {
    // a link from a node to itself always draws: the pass is serial
    D3_LAUNCH(k_link_flag, 1, 1, 0, st)(flag);
    if (serial_lcg) link_fallback_lcg(a, l, alpha, iterations, rng, flag, status, st);
    return;
  }
  if (!plan.gathered) {
    D3_LAUNCH(k_link_params, blocks_for(l.m, 256), 256, 0, st)(l, plan.order, plan.par);
    plan.gathered = true;
  }
  LinkFlowArgs c;
  c.xs = a.x; c.ys = a.y; c.vxs = a.vx; c.vys = a.vy; c.svx = a.snap_vx; c.svy = a.snap_vy;
  c.l = l; c.ends = plan.ends; c.par = plan.par; c.level_start = plan.level_start;
  c.msg = reinterpret_cast<ulonglong2 *>(plan.msg); c.tally = plan.tally;
  c.levels = plan.levels; c.nodes = plan.nodes; c.alpha = alpha; c.iterations = iterations;
  c.flag = flag; c.rng = rng; c.status = status; c.serial_lcg = serial_lcg;
  c.sleep_ns = wait_sleep_ns();
  // One SM when its shared memory holds the nodes: no messages, and the gain
  // ends about there (block / messages: 77 nodes 13 / 21 us; 1,000 nodes, 2,000
  // links 16 / 27; 5,003 nodes, two iterations 52 / 56).
  if (plan.in_block) {
    const uint32_t w = plan.width > 1024 ? 1024 : (plan.width + 31) / 32 * 32;
    if (launch(k_link_block, 1, w, plan.nodes * 2 * sizeof(double2), st, c)) return;
  }
  static int sms = 0, per_sm = 0;
  if (!per_sm) {
    int dev = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_link_flow, 256, 0);
    // blocks per SM: at most 2, or D3_LINK_BLOCKS_PER_SM (1 .. occupancy)
    int want = per >= 2 ? 2 : 1;
    if (const char *e = getenv("D3_LINK_BLOCKS_PER_SM")) {
      const int v = atoi(e);
      if (v >= 1 && v <= per) want = v;
    }
    per_sm = want;
  }
  if (!plan.in_block) {
    void *params[] = {&c};
    const unsigned most = (unsigned)(sms * per_sm), blocks = blocks_for(l.m, 256);
    ++g_launches;
    if (cudaLaunchCooperativeKernel((const void *)k_link_flow, blocks < most ? blocks : most, 256,
                                    params, 0, st) == cudaSuccess)
      return;
    cudaGetLastError();
  }
  // (without either launch: one per level)
  cudaMemsetAsync(flag, 0, sizeof(uint32_t), st);
  D3_LAUNCH(k_save_v, blocks_for(n, 256), 256, 0, st)(a.snap_vx, a.snap_vy, a.vx, a.vy, n);
  for (double k = 0; k < iterations; k += 1) {
    for (uint32_t lv = 1; lv <= plan.levels; ++lv) {
      uint32_t lo = plan.h_level_start[lv], hi = plan.h_level_start[lv + 1];
      if (hi > lo)
        D3_LAUNCH(k_link_level, blocks_for(hi - lo, 128), 128, 0, st)(a.x, a.y, a.vx, a.vy, l, plan.order,
                                                                lo, hi, alpha, flag);
    }
  }
  D3_LAUNCH(k_restore_v, blocks_for(n, 256), 256, 0, st)(a.vx, a.vy, a.snap_vx, a.snap_vy, n, flag);
  if (serial_lcg) link_fallback_lcg(a, l, alpha, iterations, rng, flag, status, st);
}

void link_serial_host(const NodeArrays &a, const LinkArrays &l, double alpha, double iterations,
                      Rng *rng, uint32_t *resume, cudaStream_t st) {
  D3_LAUNCH(k_link_serial_host, 1, 1, 0, st)(a.x, a.y, a.vx, a.vy, l, alpha, iterations, rng, resume);
}

// Serial link on the device LCG, after a DAG pass that met a jiggle.
void link_fallback_lcg(const NodeArrays &a, const LinkArrays &l, double alpha, double iterations,
                       Rng *rng, const uint32_t *flag, uint32_t *status, cudaStream_t st) {
  D3_LAUNCH(k_link_serial, 1, 1, 0, st)(a.x, a.y, a.vx, a.vy, l, alpha, iterations, rng, flag, status);
}

// ---------------------------------------------------------------------------
// Exact collide (collide.zig:17-102), serial node order
// ---------------------------------------------------------------------------

__global__ void k_shift(const double *x, const double *y, const double *vx, const double *vy,
                        double *px, double *py, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  px[i] = x[i] + vx[i];
  py[i] = y[i] + vy[i];
}

// The node loop of collide.zig:47-100 from node i0. In host-draw mode a turn
// first counts its draws (decided by the state at the turn's start) and stops
// before the turn when the buffer is short.
__global__ void k_collide_serial(const Cell *cells, const uint32_t *skip, const uint32_t *perm,
                                 const uint32_t *info, const double *xs, const double *ys, double *vxs,
                                 double *vys, const double *radii, double strength, uint32_t n,
                                 Rng *rng, bool host_draws, uint32_t *resume) {
  const uint32_t len = info[1];
  if (len == 0) {
    if (resume) resume[2] = 0;
    return;
  }
  uint32_t s = rng->lcg;
  uint64_t used = 0, avail = host_draws ? rng->avail - rng->pos : 0;
  const double *buf = host_draws ? rng->buf + rng->pos : nullptr;
  uint32_t i0 = resume ? resume[0] : 0;
  for (uint32_t i = i0; i < n; ++i) {
    const double ri = radii[i], ri2 = ri * ri;
    const double xi = xs[i] + vxs[i], yi = ys[i] + vys[i];
    if (host_draws) {
      uint32_t need = 0;
      for (uint32_t c = 0; c < len;) {
        const Cell &q = cells[c];
        double r = ri + q.r;
        if (is_leaf(q)) {
          uint32_t j = perm[q.first + q.count - 1];
          if (j > i) {
            double x = xi - xs[j] - vxs[j], y = yi - ys[j] - vys[j];
            if (x * x + y * y < r * r) need += (x == 0) + (y == 0);
          }
          c = c + 1;
          continue;
        }
        if (q.x0 > xi + r || q.x1 < xi - r || q.y0 > yi + r || q.y1 < yi - r) c = skip[c];
        else c = c + 1;
      }
      if (used + need > avail) {
        resume[0] = i;
        resume[2] = (uint32_t)(used + need - avail);
        rng->pos += used;
        return;
      }
    }
    for (uint32_t c = 0; c < len;) {
      const Cell &q = cells[c];
      double rj = q.r;
      double r = ri + rj;
      if (is_leaf(q)) {
        const uint32_t j = perm[q.first + q.count - 1];
        if (j > i) {
          double x = xi - xs[j] - vxs[j];
          double y = yi - ys[j] - vys[j];
          double l = x * x + y * y;
          if (l < r * r) {
            if (x == 0) {
              double u;
              if (host_draws) u = buf[used++]; else { s = lcg_step(s); u = lcg_value(s); }
              x = (u - 0.5) * 1e-6;
              l += x * x;
            }
            if (y == 0) {
              double u;
              if (host_draws) u = buf[used++]; else { s = lcg_step(s); u = lcg_value(s); }
              y = (u - 0.5) * 1e-6;
              l += y * y;
            }
            l = sqrt(l);
            l = (r - l) / l * strength;
            x *= l;
            y *= l;
            rj *= rj;
            r = rj / (ri2 + rj);
            vxs[i] += x * r;
            vys[i] += y * r;
            r = 1 - r;
            vxs[j] -= x * r;
            vys[j] -= y * r;
          }
        }
        c = c + 1;
        continue;
      }
      if (q.x0 > xi + r || q.x1 < xi - r || q.y0 > yi + r || q.y1 < yi - r) c = skip[c];
      else c = c + 1;
    }
  }
  if (host_draws) rng->pos += used;
  else rng->lcg = s;
  if (resume) resume[2] = 0;
}

void shift_positions(const NodeArrays &a, cudaStream_t st) {
  if (a.n == 0) return;
  D3_LAUNCH(k_shift, blocks_for(a.n, 256), 256, 0, st)(a.x, a.y, a.vx, a.vy, a.px, a.py, a.n);
}

void collide_setup(TreeDev &t, const NodeArrays &a, const double *radii, uint32_t *status,
                   cudaStream_t st) {
  const uint32_t n = a.n;
  tree_build_shifted(t, a.x, a.y, a.vx, a.vy, a.px, a.py, n, status, st);
  if (n == 0) return;
  unsigned cb, ct;
  climb_grid(cb, ct, t.cells_cap);
  D3_LAUNCH(k_collide_prep, cb, ct, 0, st)(t.cells, t.parent, t.perm, radii, t.info);
}

void collide_serial(TreeDev &t, const NodeArrays &a, const double *radii, double strength, Rng *rng,
                    bool host_draws, uint32_t *resume, cudaStream_t st) {
  if (a.n == 0) return;
  D3_LAUNCH(k_collide_serial, 1, 1, 0, st)(t.cells, t.skip, t.perm, t.info, a.x, a.y, a.vx, a.vy, radii,
                                    strength, a.n, rng, host_draws, resume);
}

// ---------------------------------------------------------------------------
// center, x, y, radial, integrate (simple.zig)
// ---------------------------------------------------------------------------

// simple.zig:14-31: sx += x[i] for i = 0..n-1 (and sy), reproduced exactly
// in parallel. While the running sum s stays inside one binade [2^e, 2^e+1)
// (or its negative) and never meets a rounding tie, fl(s + v) = s + R(v) u
// with u = 2^(e-52) the ulp there and R(v) = v / u rounded to the nearest
// integer: the chain is an integer prefix sum. The launches:
//  part     approximate sums of chunks of values (a warp per chunk);
//  records  per chunk (a thread each), from the approximate prefix, the chunk
//           as records {lo, hi, a}, each applied as "s must lie in [lo, hi];
//           s += a" — run twice, to count and then to write at the scanned
//           offsets. A stretch record covers a run where the approximate sum
//           stays in one binade: [lo, hi] holds the exact entry sums for which
//           every partial sum provably stays there, and a = T, the run's exact
//           total (s + T is itself exact: both are multiples of u and the
//           result lies in the binade). A value record adds one value (binade
//           crossings, ties, short runs) and always applies.
//  walk     one thread per axis applies the records in order with the exact s,
//           streaming them into shared memory by bulk async copies
//           (cp.async.bulk, completion on an mbarrier). A batch runs first
//           with the entry tests off the dependent chain (one add per record);
//           if any test failed, the batch reruns from its entry sum, adding a
//           failed stretch's values one by one from global memory.
constexpr unsigned CSUM_CHUNK_MIN = 128;   // values per chunk (at least)
constexpr unsigned CSUM_MAX_CHUNKS = 8192; // chunks per axis (at most)
constexpr unsigned CSUM_BUFS = 4;          // record copies in flight per axis
constexpr unsigned CSUM_BATCH = 256;       // records per copy
constexpr unsigned CSUM_MIN_RUN = 2;       // shorter runs go into value records
constexpr unsigned long long CSUM_WAIT_NS = 20000000ull;  // 20 ms per copy, far above need

__device__ inline uint32_t smem_addr(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ inline unsigned long long gtimer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A record; meta = (start << 16) | len for a stretch, 0 for a value.
struct CsumRec {
  double lo, hi, a;
  unsigned long long meta;
};

struct CsumGeom {
  uint32_t L, nc;  // values per chunk, chunks
};

__host__ __device__ inline CsumGeom csum_geom(uint32_t n) {
  CsumGeom g;
  uint32_t L = CSUM_CHUNK_MIN;
  if ((n + L - 1) / L > CSUM_MAX_CHUNKS) L = ((n + CSUM_MAX_CHUNKS - 1) / CSUM_MAX_CHUNKS + 31) / 32 * 32;
  g.L = L;
  g.nc = (n + L - 1) / L;
  return g;
}

// Every record covers at least one value: at most n records per axis.
size_t csum_rec_bytes(uint32_t n) { return 2ull * ((size_t)n + 1) * sizeof(CsumRec); }
size_t csum_count_words(uint32_t n) { return 2ull * csum_geom(n).nc + 1; }
size_t csum_part_words(uint32_t n) { return 2ull * csum_geom(n).nc; }

__device__ inline int binade_of(double s) {
  int e;
  frexp(s, &e);  // s = f 2^e, f in [0.5, 1): binade [2^(e-1), 2^e)
  return e - 1;
}

// part[ax * nc + c]: the sum of chunk c, in any order.
__global__ void k_csum_part(const double *x, const double *y, uint32_t n, CsumGeom g, double *part) {
  const uint32_t c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const unsigned lane = threadIdx.x & 31;
  if (c >= g.nc) return;
  const uint32_t k0 = c * g.L, k1 = min(n, k0 + g.L);
  double ax = 0, ay = 0;
  for (uint32_t k = k0 + lane; k < k1; k += 32) {
    ax += x[k];
    ay += y[k];
  }
  for (int o = 16; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ay += __shfl_xor_sync(0xffffffffu, ay, o);
  }
  if (lane == 0) {
    part[c] = ax;
    part[g.nc + c] = ay;
  }
}

// One thread per chunk, both axes. WRITE false: counts[ax nc + c] = the
// chunk's records; WRITE true: the records at out + offsets[ax nc + c].
template <bool WRITE>
__global__ void __launch_bounds__(256) k_csum_records(const double *x, const double *y, uint32_t n,
                                                      CsumGeom g, const double *part,
                                                      uint32_t *counts, const uint32_t *offsets,
                                                      CsumRec *out, uint32_t *status) {
  __shared__ double sred[2][8];
  __shared__ double swarp[2][8];
  const uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const uint32_t c0 = blockIdx.x * blockDim.x;
  // approximate prefix: the chunks before this block, then a block scan
  double before[2] = {0, 0};
  for (int ax = 0; ax < 2; ++ax) {
    double a = 0;
    for (uint32_t k = t; k < c0; k += blockDim.x) a += part[ax * g.nc + k];
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) sred[ax][warp] = a;
  }
  __syncthreads();
  for (int ax = 0; ax < 2; ++ax) {
    double b = 0;
    for (unsigned w = 0; w < blockDim.x / 32; ++w) b += sred[ax][w];
    before[ax] = b;
  }
  double start[2];
  for (int ax = 0; ax < 2; ++ax) {
    const double mine = c < g.nc ? part[ax * g.nc + c] : 0;
    double incl = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const double yv = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= (unsigned)o) incl += yv;
    }
    if (lane == 31) swarp[ax][warp] = incl;
    __syncthreads();
    double wpre = 0;
    for (unsigned w = 0; w < warp; ++w) wpre += swarp[ax][w];
    start[ax] = before[ax] + wpre + incl - mine;
    __syncthreads();
  }
  if (c >= g.nc) return;
  const long long LO = (1ll << 52) + 1, HI = (1ll << 53) - 1;
  const uint32_t k0 = c * g.L, k1 = min(n, k0 + g.L);
  for (int ax = 0; ax < 2; ++ax) {
    const double *v = ax ? y : x;
    CsumRec *o = nullptr;
    uint32_t limit = 0;
    if (WRITE) {
      o = out + offsets[ax * g.nc + c];
      limit = counts[ax * g.nc + c];
    }
    uint32_t count = 0;
    auto put = [&](const CsumRec &r) {
      if (WRITE) {
        if (count < limit) o[count] = r;
        else atomicOr(status, ST_CENTER_RECORDS);  // cannot happen: both passes agree
      }
      ++count;
    };
    double run = start[ax];
    bool open = false, neg = false;
    double scale = 0, u = 0, blo = 0, bhi = 0;  // 1 / u, u, binade [blo, bhi)
    long long tot = 0, pmin = 0, pmax = 0;
    uint32_t st0 = 0;
    auto start_at = [&](uint32_t k) {
      open = false;
      if (!(run != 0) || !isfinite(run)) return;
      const int e = binade_of(run);
      if (!(e > -1000 && e < 1000)) return;
      neg = run < 0;
      st0 = k;
      tot = pmin = pmax = 0;
      scale = ldexp(1.0, 52 - e);
      u = ldexp(1.0, e - 52);
      blo = ldexp(1.0, e);
      bhi = ldexp(1.0, e + 1);
      open = true;
    };
    // closes the open run [st0, end): a stretch record, or its values
    auto close = [&](uint32_t end) {
      if (!open) return;
      open = false;
      if (end - st0 >= CSUM_MIN_RUN) {
        // entry S (|s| = S u) keeps every partial S +- P in [LO, HI]
        long long a, b;
        if (!neg) { a = LO - pmin; b = HI - pmax; }
        else { a = LO + pmax; b = HI + pmin; }
        if (a <= b && a >= LO && b <= HI) {
          CsumRec r;
          if (!neg) { r.lo = (double)a * u; r.hi = (double)b * u; }
          else { r.lo = -(double)b * u; r.hi = -(double)a * u; }
          r.a = (double)tot * u;
          r.meta = ((unsigned long long)st0 << 16) | (unsigned long long)(end - st0);
          put(r);
          return;
        }
      }
      for (uint32_t k = st0; k < end; ++k) put(CsumRec{-INFINITY, INFINITY, v[k], 0ull});
    };
    start_at(k0);
    for (uint32_t k = k0; k < k1; ++k) {
      const double vv = v[k];
      run += vv;
      if (open) {
        const double q = vv * scale;  // exact: a power-of-two scaling in range
        const double ar = fabs(run);
        if (fabs(q) < 4.0e15 && fabs(q - trunc(q)) != 0.5 && ar >= blo && ar < bhi &&
            (run < 0) == neg) {
          tot += (long long)rint(q);
          pmin = tot < pmin ? tot : pmin;
          pmax = tot > pmax ? tot : pmax;
          continue;
        }
      }
      close(k);
      put(CsumRec{-INFINITY, INFINITY, vv, 0ull});  // element k is added on its own
      start_at(k + 1);
    }
    close(k1);
    if (!WRITE) counts[ax * g.nc + c] = count;
  }
}

__device__ inline bool mbar_test(uint32_t a, uint32_t parity) {
  uint32_t done;
  asm volatile(
      "{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; "
      "selp.u32 %0, 1, 0, p; }"
      : "=r"(done)
      : "r"(a), "r"(parity)
      : "memory");
  return done != 0;
}

// Waits on an mbarrier phase with a time budget; false if it ran out. It
// spins on the test first, then polls against the timer.
__device__ bool mbar_wait_for(uint64_t *bar, uint32_t parity, unsigned long long budget_ns) {
  const uint32_t a = smem_addr(bar);
  for (int k = 0; k < 4096; ++k)
    if (mbar_test(a, parity)) return true;
  const unsigned long long t0 = gtimer_ns();
  for (;;) {
    if (mbar_test(a, parity)) return true;
    if (gtimer_ns() - t0 > budget_ns) return false;
    __nanosleep(32);
  }
}

__device__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
  return mbar_wait_for(bar, parity, CSUM_WAIT_NS);
}

// The bounded wait's failure path, on purpose: a wait on an mbarrier that
// nothing arrives at (no copy is issued), with a short budget. The wait gives
// up, the status word records it, and the kernel returns.
__global__ void k_wait_selftest(uint32_t *status, unsigned long long budget_ns) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x != 0) return;
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  if (!mbar_wait_for(&bar, 0, budget_ns)) atomicOr(status, ST_WAIT_TIMEOUT);
}

void wait_selftest(uint32_t *status, uint32_t budget_us, cudaStream_t st) {
  D3_LAUNCH(k_wait_selftest, 1, 32, 0, st)(status, (unsigned long long)budget_us * 1000ull);
}

// A buffer is refilled only after this thread has used the values it read
// from it, so the copy needs no proxy fence before it.
__device__ void bulk_copy(void *dst, const void *src, uint32_t bytes, uint64_t *bar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)),
               "r"(bytes)
               : "memory");
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_addr(dst)),
      "l"(src), "r"(bytes), "r"(smem_addr(bar))
      : "memory");
}

constexpr size_t CSUM_WALK_SMEM = 2ull * CSUM_BUFS * CSUM_BATCH * sizeof(CsumRec);

// One block: thread 0 walks x and thread 32 walks y, over the records
// [offsets[ax nc], offsets[(ax + 1) nc]).
// stamps (globaltimer ns): 0-2 walk start, 3 / 4 end of the x / y walk;
// 5 / 6 / 7 the x walk's batches rerun / stretches added one by one /
// records in all.
__global__ void k_csum_walk(const double *x, const double *y, CsumGeom g, const CsumRec *recs,
                            const uint32_t *offsets, double *out, uint32_t *status,
                            unsigned long long *stamps) {
  extern __shared__ __align__(128) unsigned char csum_smem[];
  __shared__ __align__(8) uint64_t bars[2][CSUM_BUFS];
  const unsigned t = threadIdx.x;
  if ((t & 31) != 0) return;
  const int ax = t >> 5;
  if (ax > 1) return;
  if (ax == 0) stamps[0] = stamps[1] = stamps[2] = gtimer_ns();
  CsumRec *bufs = reinterpret_cast<CsumRec *>(csum_smem) + (size_t)ax * CSUM_BUFS * CSUM_BATCH;
  uint64_t *bar = bars[ax];
  for (uint32_t q = 0; q < CSUM_BUFS; ++q)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar[q])) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  const double *v = ax ? y : x;
  const uint32_t r0 = offsets[ax * g.nc], r1 = offsets[(ax + 1) * g.nc];
  const uint32_t nrec = r1 - r0, nb = (nrec + CSUM_BATCH - 1) / CSUM_BATCH;
  const CsumRec *rec = recs + r0;
  auto issue = [&](uint32_t b) {
    const uint32_t m = min(CSUM_BATCH, nrec - b * CSUM_BATCH);
    bulk_copy(bufs + (size_t)(b % CSUM_BUFS) * CSUM_BATCH, rec + (size_t)b * CSUM_BATCH,
              m * (uint32_t)sizeof(CsumRec), &bar[b % CSUM_BUFS]);
  };
  for (uint32_t b = 0; b < CSUM_BUFS && b < nb; ++b) issue(b);
  bool ok = true;
  double s = 0;
  uint32_t reruns = 0, failed = 0;
  uint32_t b = 0;
  for (; b < nb; ++b) {
    if (!mbar_wait(&bar[b % CSUM_BUFS], (b / CSUM_BUFS) & 1u)) {
      ok = false;
      break;
    }
    const CsumRec *r = bufs + (size_t)(b % CSUM_BUFS) * CSUM_BATCH;
    const uint32_t m = min(CSUM_BATCH, nrec - b * CSUM_BATCH);
    // the tests do not feed the chain: one dependent add per record
    const double s_in = s;
    bool bad = false;
#pragma unroll 4
    for (uint32_t k = 0; k < m; ++k) {
      const double lo = r[k].lo, hi = r[k].hi, a = r[k].a;
      bad |= !(s >= lo && s <= hi);
      s += a;
    }
    if (bad) {
      // some entry test failed (or s is not finite): rerun with the tests
      ++reruns;
      s = s_in;
      for (uint32_t k = 0; k < m; ++k) {
        const CsumRec d = r[k];
        if (d.meta == 0 || (s >= d.lo && s <= d.hi)) {
          s += d.a;
        } else {
          const uint32_t i0 = (uint32_t)(d.meta >> 16), len = (uint32_t)(d.meta & 0xffffu);
          for (uint32_t i = i0; i < i0 + len; ++i) s += v[i];
          ++failed;
        }
      }
    }
    if (b + CSUM_BUFS < nb) issue(b + CSUM_BUFS);
  }
  // every copy in flight lands before the block exits
  for (uint32_t q = b; q < nb && q < b + CSUM_BUFS; ++q)
    mbar_wait(&bar[q % CSUM_BUFS], (q / CSUM_BUFS) & 1u);
  if (!ok) atomicOr(status, ST_WAIT_TIMEOUT);
  out[ax] = s;
  stamps[3 + ax] = gtimer_ns();
  if (ax == 0) {
    stamps[5] = reruns;
    stamps[6] = failed;
    stamps[7] = nrec;
  }
}

// Small node counts: the two serial sums themselves, one warp on one SM
// (lane 0 x, lane 1 y, in lockstep: one dependent add per value), the values
// staged into shared memory by bulk copies. At 50k values this is ~0.27 ms
// and overlaps the forces entirely, where the record pipeline above spreads
// over many SMs and launches and, on a running sum that keeps crossing zero
// (short stretches), walks nearly as many records as values.
constexpr uint32_t CSUM_SERIAL_MAX = 1u << 16;
constexpr unsigned CSUM_TILE = 1024;  // values per copy and axis (8 KB)
constexpr unsigned CSUM_STAGES = 4;
constexpr size_t CSUM_SERIAL_SMEM = 2ull * CSUM_STAGES * CSUM_TILE * sizeof(double);

// stamps as k_csum_walk's (5-7 zero: no records).
__global__ void __launch_bounds__(32) k_csum_serial(const double *x, const double *y, uint32_t n,
                                                    double *out, uint32_t *status,
                                                    unsigned long long *stamps) {
  extern __shared__ __align__(128) unsigned char csum_smem[];
  __shared__ __align__(8) uint64_t bar[CSUM_STAGES];
  double *buf = reinterpret_cast<double *>(csum_smem);  // [stage][axis][CSUM_TILE]
  const unsigned lane = threadIdx.x;
  if (lane == 0) {
    stamps[0] = stamps[1] = stamps[2] = gtimer_ns();
    for (unsigned q = 0; q < CSUM_STAGES; ++q)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar[q])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncwarp();
  const uint32_t nt = (n + CSUM_TILE - 1) / CSUM_TILE;
  // tile t: its even-length head by two bulk copies (sizes in 16-byte
  // units), an odd last value by a plain load
  auto issue = [&](uint32_t t) {
    const uint32_t k0 = t * CSUM_TILE, m = min(CSUM_TILE, n - k0), mb = m & ~1u;
    uint64_t *b = &bar[t % CSUM_STAGES];
    double *d = buf + (size_t)(t % CSUM_STAGES) * 2 * CSUM_TILE;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)),
                 "r"(mb * 16u)
                 : "memory");
    if (mb) {
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_addr(d)),
          "l"(x + k0), "r"(mb * 8u), "r"(smem_addr(b))
          : "memory");
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_addr(d + CSUM_TILE)),
          "l"(y + k0), "r"(mb * 8u), "r"(smem_addr(b))
          : "memory");
    }
  };
  if (lane == 0)
    for (uint32_t t = 0; t < CSUM_STAGES && t < nt; ++t) issue(t);
  __syncwarp();
  const double *v = lane == 1 ? y : x;
  double s = 0;
  bool ok = true;
  uint32_t t = 0;
  for (; t < nt; ++t) {
    bool w = true;
    if (lane < 2) w = mbar_wait(&bar[t % CSUM_STAGES], (t / CSUM_STAGES) & 1u);
    if (!__all_sync(0xffffffffu, w)) {
      ok = false;
      break;
    }
    const uint32_t k0 = t * CSUM_TILE, m = min(CSUM_TILE, n - k0), mb = m & ~1u;
    if (lane < 2) {
      const double *d = buf + ((size_t)(t % CSUM_STAGES) * 2 + lane) * CSUM_TILE;
      if (mb == CSUM_TILE) {
#pragma unroll 16
        for (uint32_t k = 0; k < CSUM_TILE; ++k) s += d[k];
      } else {
        for (uint32_t k = 0; k < mb; ++k) s += d[k];
      }
      if (mb < m) s += v[k0 + mb];
    }
    // the stage is refilled after both lanes have added its values
    __syncwarp();
    if (lane == 0 && t + CSUM_STAGES < nt) issue(t + CSUM_STAGES);
  }
  // every copy in flight lands before the block exits
  if (lane == 0)
    for (uint32_t q = t; q < nt && q < t + CSUM_STAGES; ++q)
      mbar_wait(&bar[q % CSUM_STAGES], (q / CSUM_STAGES) & 1u);
  if (lane < 2) {
    out[lane] = s;
    stamps[3 + lane] = gtimer_ns();
  }
  if (lane == 0) {
    stamps[5] = stamps[6] = stamps[7] = 0;
    if (!ok) atomicOr(status, ST_WAIT_TIMEOUT);
  }
}

__global__ void k_center_apply(double *x, double *y, uint32_t n, const double *sums, double cx,
                               double cy, double strength) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double nf = (double)n;
  const double sx = (sums[0] / nf - cx) * strength;
  const double sy = (sums[1] / nf - cy) * strength;
  x[i] -= sx;
  y[i] -= sy;
}

__global__ void k_set_status(uint32_t *status, uint32_t bits) { atomicOr(status, bits); }

void set_status(uint32_t *status, uint32_t bits, cudaStream_t st) {
  D3_LAUNCH(k_set_status, 1, 1, 0, st)(status, bits);
}

void center_sum(const NodeArrays &a, ForceScratch &s, uint32_t *status, cudaStream_t st) {
  if (a.n == 0) return;
  if (a.n <= CSUM_SERIAL_MAX && ((uintptr_t)a.x & 15) == 0 && ((uintptr_t)a.y & 15) == 0) {
    const bool sattr = open_shared<k_csum_serial>(CSUM_SERIAL_SMEM);
    D3_LAUNCH(k_csum_serial, 1, 32, CSUM_SERIAL_SMEM, st)(a.x, a.y, a.n, s.center, status,
                                                          s.csum_stamps);
    if (!sattr || cudaGetLastError() != cudaSuccess) set_status(status, ST_CENTER_RECORDS, st);
    return;
  }
  const bool attr = open_shared<k_csum_walk>(CSUM_WALK_SMEM);
  const CsumGeom g = csum_geom(a.n);
  CsumRec *recs = static_cast<CsumRec *>(s.csum_recs);
  uint32_t *counts = s.csum_counts, *offsets = s.csum_counts + 2 * g.nc + 1;
  const unsigned cb = blocks_for(g.nc, 256);
  D3_LAUNCH(k_csum_part, blocks_for((size_t)g.nc * 32, 256), 256, 0, st)(a.x, a.y, a.n, g, s.csum_part);
  D3_LAUNCH(k_csum_records<false>, cb, 256, 0, st)(a.x, a.y, a.n, g, s.csum_part, counts, nullptr,
                                                   nullptr, status);
  // offsets of both axes' records; offsets[2 nc] = the total
  scan_u32(counts, offsets, 2 * g.nc, s.csum_scan_part, offsets + 2 * g.nc, st);
  D3_LAUNCH(k_csum_records<true>, cb, 256, 0, st)(a.x, a.y, a.n, g, s.csum_part, counts, offsets,
                                                  recs, status);
  D3_LAUNCH(k_csum_walk, 1, 64, CSUM_WALK_SMEM, st)(a.x, a.y, g, recs, offsets, s.center, status,
                                                    s.csum_stamps);
  // a launch that did not happen leaves stale sums: report it as a failure
  if (!attr || cudaGetLastError() != cudaSuccess) set_status(status, ST_CENTER_RECORDS, st);
}

// One block: s.center = the sums of the chunk sums in chunk order (a fixed
// tree: lane-strided partials, then a shuffle tree).
__global__ void __launch_bounds__(1024) k_csum_tree(const double *part, uint32_t nc, double *out) {
  __shared__ double wx[32], wy[32];
  double ax = 0, ay = 0;
  for (uint32_t c = threadIdx.x; c < nc; c += blockDim.x) {
    ax += part[c];
    ay += part[nc + c];
  }
  for (int o = 16; o > 0; o >>= 1) {
    ax += __shfl_xor_sync(0xffffffffu, ax, o);
    ay += __shfl_xor_sync(0xffffffffu, ay, o);
  }
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    wx[warp] = ax;
    wy[warp] = ay;
  }
  __syncthreads();
  if (warp == 0) {
    const unsigned nw = blockDim.x >> 5;
    ax = lane < nw ? wx[lane] : 0.0;
    ay = lane < nw ? wy[lane] : 0.0;
    for (int o = 16; o > 0; o >>= 1) {
      ax += __shfl_xor_sync(0xffffffffu, ax, o);
      ay += __shfl_xor_sync(0xffffffffu, ay, o);
    }
    if (lane == 0) {
      out[0] = ax;
      out[1] = ay;
    }
  }
}

void center_sum_tree(const NodeArrays &a, ForceScratch &s, cudaStream_t st) {
  if (a.n == 0) return;
  const CsumGeom g = csum_geom(a.n);
  D3_LAUNCH(k_csum_part, blocks_for((size_t)g.nc * 32, 256), 256, 0, st)(a.x, a.y, a.n, g, s.csum_part);
  D3_LAUNCH(k_csum_tree, 1, 1024, 0, st)(s.csum_part, g.nc, s.center);
}

void center_apply(const NodeArrays &a, double cx, double cy, double strength, ForceScratch &s,
                  cudaStream_t st) {
  if (a.n == 0) return;
  D3_LAUNCH(k_center_apply, blocks_for(a.n, 256), 256, 0, st)(a.x, a.y, a.n, s.center, cx, cy, strength);
}

// src/core.js:130 on the device: fixed = (fx set) | (fy set) << 1, a missing
// value being NaN.
__global__ void k_fixed_from_f(const double *fx, const double *fy, uint8_t *fixed, uint32_t n) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double a = fx[i], b = fy[i];
  fixed[i] = (uint8_t)((a == a ? 1u : 0u) | (b == b ? 2u : 0u));
}

void fixed_from_f(const double *fx, const double *fy, uint8_t *fixed, uint32_t n, cudaStream_t st) {
  if (n == 0) return;
  D3_LAUNCH(k_fixed_from_f, blocks_for(n, 256), 256, 0, st)(fx, fy, fixed, n);
}

// simulation.js:157-178 (find). The serial scan keeps the first node whose d2
// is strictly below its best so far (starting at radius^2): the lowest index
// of the least d2 below radius^2. One block: each thread runs that scan over
// its own nodes (ascending indices), then the block keeps the least (d2,
// index) pair. A NaN d2 never passes the strict test.
constexpr unsigned FIND_THREADS = 1024;

__device__ inline void find_merge(double &d, uint32_t &i, double d2, uint32_t i2) {
  if (i2 != NONE && (i == NONE || d2 < d || (d2 == d && i2 < i))) {
    d = d2;
    i = i2;
  }
}

__global__ void __launch_bounds__(FIND_THREADS) k_find(const double *xs, const double *ys, uint32_t n,
                                                       double x, double y, double r2,
                                                       uint32_t *out) {
  __shared__ double sd[FIND_THREADS / 32];
  __shared__ uint32_t si[FIND_THREADS / 32];
  double best = r2;
  uint32_t bi = NONE;
  for (uint32_t k = threadIdx.x; k < n; k += blockDim.x) {
    const double dx = x - xs[k], dy = y - ys[k];
    const double d2 = dx * dx + dy * dy;
    if (d2 < best) {
      best = d2;
      bi = k;
    }
  }
  for (int o = 16; o > 0; o >>= 1)
    find_merge(best, bi, __shfl_xor_sync(0xffffffffu, best, o), __shfl_xor_sync(0xffffffffu, bi, o));
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    sd[warp] = best;
    si[warp] = bi;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (unsigned w = 1; w < blockDim.x / 32; ++w) find_merge(best, bi, sd[w], si[w]);
    *out = bi;
  }
}

void find_closest(const NodeArrays &a, double x, double y, double r2, uint32_t *out,
                  cudaStream_t st) {
  D3_LAUNCH(k_find, 1, FIND_THREADS, 0, st)(a.x, a.y, a.n, x, y, r2, out);
}

// simple.zig:51-62
__global__ void k_axis(double *pos, double *v, const double *strength, const double *target,
                       double alpha, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  v[i] += (target[i] - pos[i]) * strength[i] * alpha;
}

void axis_force(const NodeArrays &a, const double *strength, const double *target, double alpha,
                int dim, cudaStream_t st) {
  if (a.n == 0) return;
  D3_LAUNCH(k_axis, blocks_for(a.n, 256), 256, 0, st)(dim ? a.y : a.x, dim ? a.vy : a.vx, strength, target,
                                               alpha, a.n);
}

// simple.zig:64-86
__global__ void k_radial(const double *x, const double *y, double *vx, double *vy,
                         const double *strength, const double *radius, double cx, double cy,
                         double alpha, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double dx = x[i] - cx;
  if (dx == 0 || dx != dx) dx = 1e-6;
  double dy = y[i] - cy;
  if (dy == 0 || dy != dy) dy = 1e-6;
  double l = sqrt(dx * dx + dy * dy);
  double k = (radius[i] - l) * strength[i] * alpha / l;
  vx[i] += dx * k;
  vy[i] += dy * k;
}

void radial_force(const NodeArrays &a, const double *strength, const double *radius, double cx,
                  double cy, double alpha, cudaStream_t st) {
  if (a.n == 0) return;
  D3_LAUNCH(k_radial, blocks_for(a.n, 256), 256, 0, st)(a.x, a.y, a.vx, a.vy, strength, radius, cx, cy,
                                                 alpha, a.n);
}

// simple.zig:90-123
__global__ void k_integrate(double *x, double *y, double *vx, double *vy, const double *fx,
                            const double *fy, const uint8_t *fixed, double decay, uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint8_t f = fixed[i];
  if ((f & 1) == 0) {
    double v = vx[i] * decay;
    vx[i] = v;
    x[i] += v;
  } else {
    x[i] = fx[i];
    vx[i] = 0;
  }
  if ((f & 2) == 0) {
    double v = vy[i] * decay;
    vy[i] = v;
    y[i] += v;
  } else {
    y[i] = fy[i];
    vy[i] = 0;
  }
}

// k_center_apply then k_integrate, per node in one pass (both are per node).
__global__ void k_center_integrate(double *x, double *y, double *vx, double *vy, const double *fx,
                                   const double *fy, const uint8_t *fixed, const double *sums,
                                   double cx, double cy, double strength, double decay,
                                   uint32_t n) {
  uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double nf = (double)n;
  const double sx = (sums[0] / nf - cx) * strength;
  const double sy = (sums[1] / nf - cy) * strength;
  const double x0 = x[i] - sx, y0 = y[i] - sy;
  const uint8_t f = fixed[i];
  if ((f & 1) == 0) {
    double v = vx[i] * decay;
    vx[i] = v;
    x[i] = x0 + v;
  } else {
    x[i] = fx[i];
    vx[i] = 0;
  }
  if ((f & 2) == 0) {
    double v = vy[i] * decay;
    vy[i] = v;
    y[i] = y0 + v;
  } else {
    y[i] = fy[i];
    vy[i] = 0;
  }
}

void center_apply_integrate(const NodeArrays &a, double cx, double cy, double strength,
                            ForceScratch &s, double decay, cudaStream_t st) {
  if (a.n == 0) return;
  D3_LAUNCH(k_center_integrate, blocks_for(a.n, 256), 256, 0, st)(a.x, a.y, a.vx, a.vy, a.fx, a.fy,
                                                           a.fixed, s.center, cx, cy, strength,
                                                           decay, a.n);
}

void integrate(const NodeArrays &a, double decay, cudaStream_t st) {
  if (a.n == 0) return;
  D3_LAUNCH(k_integrate, blocks_for(a.n, 256), 256, 0, st)(a.x, a.y, a.vx, a.vy, a.fx, a.fy, a.fixed, decay,
                                                    a.n);
}

}  // namespace d3
