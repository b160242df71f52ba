// scan_sort.cu — device-wide exclusive scan and stable LSD radix sort.
#include "scan_sort.cuh"

namespace d3 {

// ---- exclusive scan --------------------------------------------------------

// Block-wide exclusive scan of one value per thread (blockDim a multiple of
// 32, at most 1024); the block total goes to *total.
__device__ inline uint32_t block_exclusive_scan(uint32_t v, uint32_t *sw, uint32_t *total) {
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= (unsigned)o) x += y;
  }
  if (lane == 31) sw[warp] = x;
  __syncthreads();
  const unsigned nw = blockDim.x >> 5;
  if (warp == 0) {
    uint32_t w = lane < nw ? sw[lane] : 0;
    uint32_t t = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= (unsigned)o) t += y;
    }
    if (lane < nw) sw[lane] = t - w;
    if (lane == nw - 1) sw[32] = t;
  }
  __syncthreads();
  uint32_t r = sw[warp] + x - v;
  *total = sw[32];
  __syncthreads();
  return r;
}

// Each block scans 4 * blockDim values (4 consecutive per thread).
__global__ void k_scan_local(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *partials) {
  __shared__ uint32_t sw[33];
  const size_t base = (size_t)blockIdx.x * blockDim.x * 4 + threadIdx.x * 4;
  uint32_t v[4];
  uint32_t s = 0;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[k] = base + k < n ? in[base + k] : 0;
    s += v[k];
  }
  uint32_t tot;
  uint32_t ex = block_exclusive_scan(s, sw, &tot);
  uint32_t run = ex;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    if (base + k < n) out[base + k] = run;
    run += v[k];
  }
  if (threadIdx.x == 0) partials[blockIdx.x] = tot;
}

// Scans the block partials in place (one block; loops if many).
__global__ void k_scan_partials(uint32_t *partials, uint32_t nb, uint32_t *total) {
  __shared__ uint32_t sw[33];
  __shared__ uint32_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (uint32_t off = 0; off < nb; off += blockDim.x) {
    uint32_t i = off + threadIdx.x;
    uint32_t v = i < nb ? partials[i] : 0;
    uint32_t tot;
    uint32_t ex = block_exclusive_scan(v, sw, &tot);
    if (i < nb) partials[i] = carry + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry;
}

__global__ void k_scan_add(uint32_t *out, uint32_t n, const uint32_t *partials) {
  const size_t base = (size_t)blockIdx.x * blockDim.x * 4 + threadIdx.x * 4;
  uint32_t p = partials[blockIdx.x];
  if (p == 0) return;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (base + k < n) out[base + k] += p;
}

void scan_u32(const uint32_t *in, uint32_t *out, uint32_t n, uint32_t *partials, uint32_t *total,
              cudaStream_t st) {
  unsigned nb = blocks_for(n, SCAN_BLOCK * 4);
  D3_LAUNCH(k_scan_local, nb, SCAN_BLOCK, 0, st)(in, out, n, partials);
  D3_LAUNCH(k_scan_partials, 1, SCAN_BLOCK, 0, st)(partials, nb, total);
  if (nb > 1) D3_LAUNCH(k_scan_add, nb, SCAN_BLOCK, 0, st)(out, n, partials);
}

// ---- radix sort -------------------------------------------------------------

// Digit modes: BYTE, the key's byte at `shift` (256 buckets); PART_BYTE, the
// value's bit 31 above the key's byte at `shift` (512 buckets: the partition
// on bit 31 folded into the last byte pass, the same stable order as a byte
// pass followed by a partition pass).
enum : int { BYTE = 0, PART_BYTE = 1 };

template <int MODE>
__host__ __device__ constexpr unsigned buckets() {
  return MODE == PART_BYTE ? 512u : 256u;
}

template <int MODE>
__device__ inline uint32_t digit_of(uint64_t k, uint32_t v, int shift) {
  const uint32_t b = (uint32_t)(k >> shift) & 255u;
  return MODE == PART_BYTE ? ((v >> 31) << 8) | b : b;
}

// The lanes whose digit of `bits` bits is this lane's, among the valid ones: a
// ballot a bit (a warp match takes a turn per distinct digit, up to 32).
__device__ inline unsigned same_digit(uint32_t d, bool valid, int bits) {
  unsigned peers = __ballot_sync(0xffffffffu, valid);
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    if (b >= bits) break;
    const unsigned on = __ballot_sync(0xffffffffu, d >> b & 1u);
    peers &= d >> b & 1u ? on : ~on;
  }
  return peers;
}

// The whole array's digit counts of every pass (they do not depend on the
// order), so that a pass is one launch: tot[pass * 512 + digit].
__global__ void __launch_bounds__(SORT_THREADS) k_sort_totals(const uint64_t *keys, const uint32_t *vals,
                                                              uint32_t n, int byte_lo, int passes,
                                                              int part, uint32_t *tot) {
  __shared__ uint32_t h[SORT_PASSES * 512];
  for (unsigned d = threadIdx.x; d < SORT_PASSES * 512; d += blockDim.x) h[d] = 0;
  __syncthreads();
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const uint64_t k = keys[i] >> (8 * byte_lo);
    for (int p = 0; p < passes; ++p) {
      uint32_t d = (uint32_t)(k >> (8 * p)) & 255u;
      if (part && p + 1 == passes) d |= (vals[i] >> 31) << 8;
      atomicAdd(&h[p * 512 + d], 1u);
    }
  }
  __syncthreads();
  for (unsigned d = threadIdx.x; d < passes * 512u; d += blockDim.x)
    if (h[d]) atomicAdd(&tot[d], h[d]);
}

// A tile's counts as its successors read them, one word per digit: nothing
// yet, the tile's own count, or the count of it and every tile before it.
constexpr uint32_t TILE_OWN = 1u << 30, TILE_ALL = 2u << 30, TILE_COUNT = TILE_OWN - 1;
constexpr unsigned LOOK_BACK = 8;                       // words read at a time
constexpr unsigned long long SORT_WAIT_NS = 2000000ull;   // 2 ms, far above need

__device__ inline unsigned long long sort_timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ inline uint32_t tile_read(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ inline void tile_write(uint32_t *p, uint32_t v) {
  asm volatile("st.relaxed.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The count of one digit in the tiles before `tile`: words read backwards
// until one that holds all before it. False if a word did not come in time.
template <unsigned NB>
__device__ bool look_back(const uint32_t *words, uint32_t tile, uint32_t d, uint32_t &before) {
  before = 0;
  unsigned long long t0 = 0;
  int64_t at = (int64_t)tile - 1;
  while (at >= 0) {
    uint32_t w[LOOK_BACK];
#pragma unroll
    for (unsigned q = 0; q < LOOK_BACK; ++q)
      w[q] = at - (int64_t)q >= 0 ? tile_read(&words[(size_t)(at - q) * NB + d]) : TILE_ALL;
    bool waiting = false;
#pragma unroll
    for (unsigned q = 0; q < LOOK_BACK; ++q) {
      if (waiting) continue;
      if (w[q] < TILE_OWN) {
        waiting = true;
        continue;
      }
      before += w[q] & TILE_COUNT;
      --at;
      if (w[q] & TILE_ALL) return true;
    }
    if (waiting) {
      if (!t0) t0 = sort_timer_ns();
      else if (sort_timer_ns() - t0 > SORT_WAIT_NS) return false;
      __nanosleep(20);
    } else {
      t0 = 0;
    }
  }
  return true;
}

// Stable scatter of one tile of SORT_TILE keys, a launch a pass (the published
// single-pass prefix with decoupled look-back of Merrill and Garland 2016, and
// its use in a radix sort, Adinets and Merrill 2022): warp w takes the tile's
// w-th run of 32 x PER keys, in PER rounds of 32. In a round a key's rank
// among equal digits is the warp's count of that digit so far plus the lanes
// below it with the same digit (same_digit). The warps' counts then give
// each key its place in the tile sorted by digit (stable); the tile is
// reordered in shared memory and written in that order, so consecutive
// threads write consecutive places of one digit's run. Where the tile's run of
// a digit starts follows from the whole array's counts (`all`) and the counts
// of the tiles before it, which every tile publishes as soon as it has its
// own (`words`): one launch and one read of the keys a pass, where a counting
// pass and three scan launches came first. Tiles are numbered in the order
// their blocks start (`ticket`), so a tile only waits for running blocks; where
// a wait runs out all the same, the tile counts the keys before it itself. A pass over
// 1 M keys 37 -> 27 us, over 41,000 24 -> 11 us, its share of k_sort_totals
// in it.
template <int MODE>
__global__ void __launch_bounds__(SORT_THREADS) k_sort_scatter(const uint64_t *keys, const uint32_t *vals,
                                                               uint64_t *okeys, uint32_t *ovals,
                                                               uint32_t n, int shift,
                                                               const uint32_t *all, uint32_t *words,
                                                               uint32_t *ticket) {
  constexpr unsigned NB = buckets<MODE>();
  __shared__ uint32_t tile_id;
  constexpr unsigned WARPS = SORT_THREADS / 32, PER = SORT_TILE / SORT_THREADS;
  __shared__ uint32_t wh[WARPS][NB];
  __shared__ uint32_t lstart[NB], gbase[NB];
  __shared__ uint64_t skey[SORT_TILE];
  __shared__ uint32_t sval[SORT_TILE];
  __shared__ uint32_t wsum[WARPS], wall[WARPS];
  const unsigned lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const unsigned lt = (1u << lane) - 1;
  // every key has the same digit (cell numbers' high bytes): the order stands
  if (all[digit_of<MODE>(keys[0], vals[0], shift)] == n) {
    const size_t base = (size_t)blockIdx.x * SORT_TILE;
    for (unsigned r = threadIdx.x; r < SORT_TILE; r += SORT_THREADS)
      if (base + r < n) {
        okeys[base + r] = keys[base + r];
        ovals[base + r] = vals[base + r];
      }
    return;
  }
  if (threadIdx.x == 0) tile_id = atomicAdd(ticket, 1u);
  for (unsigned d = threadIdx.x; d < WARPS * NB; d += blockDim.x) (&wh[0][0])[d] = 0;
  __syncthreads();
  const uint32_t tile = tile_id;
  const size_t tbase = (size_t)tile * SORT_TILE;
  const size_t wbase = tbase + (size_t)warp * 32 * PER;
  const uint32_t tn = n - tbase < SORT_TILE ? (uint32_t)(n - tbase) : SORT_TILE;
  uint64_t k[PER];
  uint32_t v[PER], dg[PER], rk[PER];
#pragma unroll
  for (unsigned r = 0; r < PER; ++r) {
    const size_t i = wbase + r * 32 + lane;
    k[r] = i < n ? keys[i] : 0;
    v[r] = i < n ? vals[i] : 0;
  }
  __syncthreads();
#pragma unroll
  for (unsigned r = 0; r < PER; ++r) {
    const bool valid = wbase + r * 32 + lane < n;
    const uint32_t d = valid ? digit_of<MODE>(k[r], v[r], shift) : NB + lane;  // never matches
    const unsigned peers = same_digit(d, valid, MODE == PART_BYTE ? 9 : 8);
    const unsigned below = __popc(peers & lt);
    const uint32_t cnt = valid ? wh[warp][d] : 0;
    __syncwarp();
    if (valid && below == 0) wh[warp][d] = cnt + __popc(peers);
    __syncwarp();
    dg[r] = d;
    rk[r] = cnt + below;
  }
  __syncthreads();
  // per digit: the earlier warps' counts (in place) and the tile's count;
  // the tile's digit starts by a block scan of the counts
  uint32_t tot[NB / SORT_THREADS];
#pragma unroll
  for (unsigned j = 0; j < NB / SORT_THREADS; ++j) {
    const unsigned d = j * SORT_THREADS + threadIdx.x;
    uint32_t run = 0;
#pragma unroll
    for (unsigned w = 0; w < WARPS; ++w) {
      const uint32_t t = wh[w][d];
      wh[w][d] = run;
      run += t;
    }
    tot[j] = run;
    tile_write(&words[(size_t)tile * NB + d], run | (tile ? TILE_OWN : TILE_ALL));
  }
  // exclusive scans of the NB tile counts and of the whole array's, a chunk
  // of SORT_THREADS digits at a time (thread t holds digit j * SORT_THREADS + t
  // of chunk j)
  uint32_t gstart[NB / SORT_THREADS];
  {
    uint32_t chunk_base = 0, chunk_all = 0;
#pragma unroll
    for (unsigned j = 0; j < NB / SORT_THREADS; ++j) {
      const uint32_t x = tot[j], g = all[j * SORT_THREADS + threadIdx.x];
      uint32_t in = x, gin = g;
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, in, o), z = __shfl_up_sync(0xffffffffu, gin, o);
        if (lane >= (unsigned)o) {
          in += y;
          gin += z;
        }
      }
      __syncthreads();
      if (lane == 31) {
        wsum[warp] = in;
        wall[warp] = gin;
      }
      __syncthreads();
      uint32_t pre = 0, sum = 0, gpre = 0, gsum = 0;
      for (unsigned w = 0; w < WARPS; ++w) {
        if (w < warp) {
          pre += wsum[w];
          gpre += wall[w];
        }
        sum += wsum[w];
        gsum += wall[w];
      }
      lstart[j * SORT_THREADS + threadIdx.x] = chunk_base + pre + in - x;
      gstart[j] = chunk_all + gpre + gin - g;
      chunk_base += sum;
      chunk_all += gsum;
    }
  }
  bool ok = true;
#pragma unroll
  for (unsigned j = 0; j < NB / SORT_THREADS; ++j) {
    const unsigned d = j * SORT_THREADS + threadIdx.x;
    uint32_t before;
    if (look_back<NB>(words, tile, d, before)) {
      if (tile) tile_write(&words[(size_t)tile * NB + d], (before + tot[j]) | TILE_ALL);
      gbase[d] = gstart[j] + before;
    } else {
      ok = false;
    }
  }
  if (__syncthreads_or(!ok)) {
    uint32_t *h = reinterpret_cast<uint32_t *>(skey);
    for (unsigned d = threadIdx.x; d < NB; d += SORT_THREADS) h[d] = 0;
    __syncthreads();
    for (size_t i = threadIdx.x; i < tbase; i += SORT_THREADS)
      atomicAdd(&h[digit_of<MODE>(keys[i], vals[i], shift)], 1u);
    __syncthreads();
#pragma unroll
    for (unsigned j = 0; j < NB / SORT_THREADS; ++j) {
      const unsigned d = j * SORT_THREADS + threadIdx.x;
      tile_write(&words[(size_t)tile * NB + d], (h[d] + tot[j]) | TILE_ALL);
      gbase[d] = gstart[j] + h[d];
    }
    __syncthreads();
  }
  // each key into its place in the tile's digit order
#pragma unroll
  for (unsigned r = 0; r < PER; ++r)
    if (wbase + r * 32 + lane < n) {
      const uint32_t at = lstart[dg[r]] + wh[warp][dg[r]] + rk[r];
      skey[at] = k[r];
      sval[at] = v[r];
    }
  __syncthreads();
  // write in tile order: place i of digit d goes to gbase[d] + i - lstart[d]
  for (uint32_t i = threadIdx.x; i < tn; i += blockDim.x) {
    const uint64_t kk = skey[i];
    const uint32_t vv = sval[i];
    const uint32_t d = digit_of<MODE>(kk, vv, shift);
    const uint32_t pos = gbase[d] + (i - lstart[d]);
    okeys[pos] = kk;
    ovals[pos] = vv;
  }
}

// Up to SORT_BLOCK_MAX keys: all passes in one block, keys (the sorted bytes,
// at most 32 bits) and values in registers and shared memory. A pass is the
// ranking above without the other tiles: no launch, no wait. Four passes: 3,000
// keys 35 us, 8,192 41 us, for 39 us and the gaps of six launches; the one SM's
// ranking rounds grow with the keys, the tiles' time does not, so the line is
// what registers and shared memory hold.
constexpr uint32_t SORT_BLOCK_MAX = 8192;
constexpr unsigned SB_THREADS = 1024, SB_WARPS = SB_THREADS / 32,
                   SB_PER = SORT_BLOCK_MAX / SB_THREADS;
constexpr size_t SB_SMEM = SORT_BLOCK_MAX * 8 + SB_WARPS * 512 * 2;

__global__ void __launch_bounds__(SB_THREADS) k_sort_block(uint64_t *keys, uint32_t *vals, uint32_t n,
                                                           int byte_lo, int passes, int part) {
  extern __shared__ uint32_t sb_smem[];
  uint32_t *skey = sb_smem, *sval = skey + SORT_BLOCK_MAX;
  uint16_t *wh = reinterpret_cast<uint16_t *>(sval + SORT_BLOCK_MAX);  // [warp][digit]
  __shared__ uint32_t seg[SB_THREADS], lstart[512], wsum[16];
  const unsigned tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1;
  const uint32_t base = warp * 32 * SB_PER + lane;
  uint32_t k[SB_PER], v[SB_PER];
  uint16_t rk[SB_PER];
#pragma unroll
  for (unsigned r = 0; r < SB_PER; ++r) {
    const uint32_t i = base + r * 32;
    k[r] = i < n ? (uint32_t)(keys[i] >> (8 * byte_lo)) : 0;
    v[r] = i < n ? vals[i] : 0;
  }
  for (int p = 0; p < passes; ++p) {
    const bool wide = part && p + 1 == passes;  // the partition's bit on top of the byte
    const unsigned nb = wide ? 512 : 256;
    uint16_t *mine = wh + warp * nb;
    for (unsigned d = lane; d < nb; d += 32) mine[d] = 0;
    __syncwarp();
#pragma unroll
    for (unsigned r = 0; r < SB_PER; ++r) {
      const bool valid = base + r * 32 < n;
      const uint32_t b = (k[r] >> (8 * p)) & 255u;
      const uint32_t d = !valid ? nb + lane : wide ? (v[r] >> 31) << 8 | b : b;
      const unsigned peers = same_digit(d, valid, wide ? 9 : 8);
      const unsigned below = __popc(peers & lt);
      const uint32_t cnt = valid ? mine[d] : 0;
      __syncwarp();
      if (valid && below == 0) mine[d] = (uint16_t)(cnt + __popc(peers));
      __syncwarp();
      rk[r] = (uint16_t)(cnt + below);
    }
    __syncthreads();
    // per digit: the earlier warps' counts (in place) and the count of all,
    // the warps in SB_THREADS / nb stretches
    const unsigned d = tid & (nb - 1), part_of = tid / nb, stretch = SB_WARPS * nb / SB_THREADS;
    uint32_t run = 0;
#pragma unroll 4
    for (unsigned w = part_of * stretch; w < (part_of + 1) * stretch; ++w) {
      const uint32_t t = wh[w * nb + d];
      wh[w * nb + d] = (uint16_t)run;
      run += t;
    }
    seg[tid] = run;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (unsigned q = 0; q < SB_THREADS / nb; ++q) {
      if (q < part_of) before += seg[q * nb + d];
      total += seg[q * nb + d];
    }
    // every key has the same digit: the order stands
    if (__syncthreads_or(total == n)) continue;
    uint32_t in = total;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t y = __shfl_up_sync(0xffffffffu, in, o);
      if (lane >= (unsigned)o) in += y;
    }
    if (tid < nb && lane == 31) wsum[warp] = in;
    seg[tid] = before;
    __syncthreads();
    if (tid < nb) {
      uint32_t pre = 0;
      for (unsigned w = 0; w < warp; ++w) pre += wsum[w];
      lstart[tid] = pre + in - total;
    }
    __syncthreads();
#pragma unroll
    for (unsigned r = 0; r < SB_PER; ++r) {
      if (base + r * 32 < n) {
        const uint32_t b = (k[r] >> (8 * p)) & 255u;
        const uint32_t dd = wide ? (v[r] >> 31) << 8 | b : b;
        const uint32_t to = lstart[dd] + seg[warp / stretch * nb + dd] + mine[dd] + rk[r];
        skey[to] = k[r];
        sval[to] = v[r];
      }
    }
    __syncthreads();
#pragma unroll
    for (unsigned r = 0; r < SB_PER; ++r) {
      const uint32_t i = base + r * 32;
      if (i < n) {
        k[r] = skey[i];
        v[r] = sval[i];
      }
    }
    // (the next pass writes skey only after its own barriers)
  }
#pragma unroll
  for (unsigned r = 0; r < SB_PER; ++r) {
    const uint32_t i = base + r * 32;
    if (i < n) {
      keys[i] = (uint64_t)k[r] << (8 * byte_lo);
      vals[i] = v[r];
    }
  }
}

void radix_sort_u64(uint64_t *keys, uint32_t *vals, uint32_t n, int byte_lo, int byte_hi,
                    bool partition_hi_bit, const SortScratch &s, cudaStream_t st) {
  if (n == 0) return;
  if (n <= SORT_BLOCK_MAX && open_shared<k_sort_block>(SB_SMEM) &&
      launch(k_sort_block, 1, SB_THREADS, SB_SMEM, st, keys, vals, n, byte_lo, byte_hi - byte_lo,
             partition_hi_bit))
    return;
  uint64_t *ak = keys, *bk = s.keys_tmp;
  uint32_t *av = vals, *bv = s.vals_tmp;
  const uint32_t tiles = (n + SORT_TILE - 1) / SORT_TILE;
  const int passes = byte_hi - byte_lo;
  // hist: the passes' totals, tickets, then a word per tile, digit and pass
  uint32_t *tot = s.hist, *ticket = tot + SORT_PASSES * 512, *words = ticket + SORT_PASSES;
  cudaMemsetAsync(s.hist, 0, (SORT_PASSES * 513 + (size_t)tiles * 256 * (passes + partition_hi_bit)) * 4, st);
  const unsigned hb = blocks_for(n, SORT_THREADS * 2);
  D3_LAUNCH(k_sort_totals, hb < 592 ? hb : 592, SORT_THREADS, 0, st)(keys, vals, n, byte_lo, passes,
                                                                  partition_hi_bit, tot);
  for (int p = 0; p < passes; ++p) {
    const int shift = 8 * (byte_lo + p);
    // the partition on bit 31 rides on the last byte pass
    if (partition_hi_bit && p + 1 == passes)
      D3_LAUNCH(k_sort_scatter<PART_BYTE>, tiles, SORT_THREADS, 0, st)(ak, av, bk, bv, n, shift,
                                                                      tot + p * 512, words, ticket + p);
    else
      D3_LAUNCH(k_sort_scatter<BYTE>, tiles, SORT_THREADS, 0, st)(ak, av, bk, bv, n, shift,
                                                                 tot + p * 512, words, ticket + p);
    words += (size_t)tiles * 256;  // (the 9-bit digit comes last)
    uint64_t *tk = ak; ak = bk; bk = tk;
    uint32_t *tv = av; av = bv; bv = tv;
  }
  if (ak != keys) {
    cudaMemcpyAsync(keys, ak, (size_t)n * 8, cudaMemcpyDeviceToDevice, st);
    cudaMemcpyAsync(vals, av, (size_t)n * 4, cudaMemcpyDeviceToDevice, st);
  }
}

}  // namespace d3
