// K2: leaf binning and the cell lists behind the influence tree, the splat and
// PSE neighbour lists.
//
// Replaces Particles::PartitionParticles (Particles/particle.cpp:398-437),
// which appends each vorton index to the list of the cell
// UniformGridGeometry::OffsetOfPosition names (uniformGrid.h:536-574,
// 645-651), in vorton-index order.  Here a counting sort by cell:
//   1. k_bin: one thread per vorton computes the leaf offset with the
//      reference's FP32 binning (bit-exact) and takes a place among the cell's
//      vortons from the cell's counter (places in no particular order);
//   2. an exclusive scan of the counts gives each cell's first slot;
//   3. k_place puts each vorton's index into its cell's slots;
//   4. k_order, one thread per slot, puts the cell's indices into ascending
//      order -- the order in which the reference accumulates them -- by
//      counting the smaller ones; cells of more than kCountMax vortons are left
//      to k_order_large, which sorts up to kSortMax indices in shared memory and
//      marks the indices of larger cells in a bitmap.
// The result does not depend on thread timing.
//
// Bound by launches and the latency of dependent accesses: seven small kernels,
// 262,144 vortons on a 129^3 grid in 26 us.  (A stable radix sort by cell in two
// passes of 11 bits, fifteen kernels, took 69 us; its scatter, three barriers to
// every 256 keys of a tile, 13 us a pass.)
#include "vg_internal.cuh"

namespace vg {

namespace {

__global__ void k_bin(Geom g, const float4* __restrict__ pos, int n, unsigned* __restrict__ key,
                      unsigned* __restrict__ place, unsigned* __restrict__ count, unsigned ncells) {
  pdl_entry();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;  // n may be within a block of 2^31
  const bool valid = i < (unsigned)n;
  unsigned off = 0xffffffffu;
  if (valid) {
    const float4 p = pos[i];
    const unsigned ix = bin_axis(p.x, g.mn[0], g.cpe[0]);
    const unsigned iy = bin_axis(p.y, g.mn[1], g.cpe[1]);
    const unsigned iz = bin_axis(p.z, g.mn[2], g.cpe[2]);
    off = ix + g.np[0] * (iy + g.np[1] * iz);
    // Vortons outside the grid's points (undefined behaviour in the reference;
    // negative cells wrap to large values), and non-finite ones, go to an extra
    // slot, ncells, that no consumer of the lists reads: they drop out of the
    // splat, the tree and PSE.
    if (ix >= g.np[0] || iy >= g.np[1] || iz >= g.np[2] || off >= ncells || !(p.x == p.x && p.y == p.y && p.z == p.z))
      off = ncells;
  }
  // one addition for the vortons of a warp in the same cell: a counter that all share would take them one by one
  const unsigned peers = __match_any_sync(0xffffffffu, off);
  const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
  unsigned base = 0;
  if (valid && lane == leader) base = atomicAdd(&count[off], (unsigned)__popc(peers));
  base = __shfl_sync(0xffffffffu, base, leader);
  if (!valid) return;
  key[i] = off;
  place[i] = base + __popc(peers & ((1u << lane) - 1u));
}

// ---- exclusive scan ----------------------------------------------------------
// Two kernels over at most kScanCtas chunks of whole tiles: the chunks' sums, then
// every chunk's scan from the sum of the chunks before it.  No kernel waits for
// another block; up to one tile takes the second kernel alone.
constexpr int kScanThreads = 512, kScanItems = 8, kScanTile = kScanThreads * kScanItems;
constexpr int kScanCtas = 1024;

__device__ __forceinline__ unsigned warp_inclusive(unsigned x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Sum over the block's threads of v, for all of them (kThreads up to 1024).
template <int kThreads>
__device__ __forceinline__ unsigned block_sum(unsigned v, unsigned* sh) {
  v = __reduce_add_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x / 32] = v;
  __syncthreads();
  unsigned t = (threadIdx.x & 31) < kThreads / 32 ? sh[threadIdx.x & 31] : 0;
  t = __reduce_add_sync(0xffffffffu, t);
  __syncthreads();
  return t;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_sums(const unsigned* __restrict__ in, size_t n, size_t chunk,
                                                            unsigned* __restrict__ sums) {
  pdl_entry();
  __shared__ unsigned sh[32];
  const size_t begin = blockIdx.x * chunk, end = begin + chunk < n ? begin + chunk : n;
  unsigned v = 0;
  for (size_t base = begin; base < end; base += kScanTile)
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      const size_t i = base + k * kScanThreads + threadIdx.x;
      if (i < end) v += in[i];
    }
  v = block_sum<kScanThreads>(v, sh);
  if (threadIdx.x == 0) sums[blockIdx.x] = v;
}

__global__ void __launch_bounds__(kScanThreads) k_scan_chunks(const unsigned* __restrict__ in, size_t n, size_t chunk,
                                                              const unsigned* __restrict__ sums,
                                                              unsigned* __restrict__ out, int write_total) {
  pdl_entry();
  __shared__ unsigned sh[32], warp_sum[kScanThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  const size_t begin = blockIdx.x * chunk, end = begin + chunk < n ? begin + chunk : n;
  unsigned before = 0;
  for (unsigned b = threadIdx.x; b < blockIdx.x; b += kScanThreads) before += sums[b];
  before = block_sum<kScanThreads>(before, sh);
  for (size_t base = begin; base < end; base += kScanTile) {
    // a warp scans 256 consecutive values, 32 at a time
    const size_t w0 = base + (size_t)wid * 32 * kScanItems + lane;
    unsigned v[kScanItems], run = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) v[k] = w0 + 32 * k < end ? in[w0 + 32 * k] : 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      const unsigned inc = warp_inclusive(v[k]);
      const unsigned total = __shfl_sync(0xffffffffu, inc, 31);
      v[k] = run + inc - v[k];
      run += total;
    }
    if (lane == 0) warp_sum[wid] = run;
    __syncthreads();
    const unsigned ws_ = lane < kScanThreads / 32 ? warp_sum[lane] : 0;
    const unsigned inc = warp_inclusive(ws_);
    const unsigned mine = __shfl_sync(0xffffffffu, inc - ws_, wid);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k)
      if (w0 + 32 * k < end) out[w0 + 32 * k] = before + mine + v[k];
    before += __shfl_sync(0xffffffffu, inc, 31);
    __syncthreads();
  }
  if (write_total && blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = before;
}

// ---- a cell's indices in ascending order -------------------------------------
// kCountMax: a thread's count costs as many loads as its cell has vortons, from
// the first-level cache mostly; 512 of them take about 1 us.  kSortMax: 32 KB.
constexpr unsigned kCountMax = 512, kSortMax = 8192;
constexpr int kOrderThreads = 1024;
constexpr unsigned kWindow = kSortMax * 32;  // indices of one bitmap
constexpr unsigned kMidCtas = 304, kBigCtas = 152;

__global__ void k_place(int n, const unsigned* __restrict__ key, const unsigned* __restrict__ place,
                        const unsigned* __restrict__ start, uint2* __restrict__ slot) {
  pdl_entry();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (unsigned)n) return;
  const unsigned k = key[i];
  slot[start[k] + place[i]] = make_uint2(k, i);
}

// big[0], big[1]: the numbers of mid and big cells; their offsets follow, mid ones from mid_list, big ones from big_list.
__global__ void k_order(int n, const uint2* __restrict__ slot, const unsigned* __restrict__ start,
                        unsigned* __restrict__ items, unsigned* __restrict__ big, unsigned* __restrict__ mid_list,
                        unsigned* __restrict__ big_list) {
  pdl_entry();
  const unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (unsigned)n) return;
  const uint2 me = slot[p];
  const unsigned s = start[me.x], e = start[me.x + 1], m = e - s;
  if (m <= kCountMax) {
    unsigned rank = 0;
    if (m > 1)
#pragma unroll 4
      for (unsigned q = s; q < e; ++q) rank += slot[q].y < me.y;
    items[s + rank] = me.y;
  } else if (p == s) {
    if (m <= kSortMax)
      mid_list[atomicAdd(&big[0], 1u)] = me.x;
    else
      big_list[atomicAdd(&big[1], 1u)] = me.x;
  }
}

// Bitonic sort of one cell's indices at a time (v: kSortMax values in shared memory).
__device__ __forceinline__ void order_mid(unsigned cta, unsigned ctas, const uint2* __restrict__ slot,
                                          const unsigned* __restrict__ start, const unsigned* __restrict__ big,
                                          const unsigned* __restrict__ mid_list, unsigned* __restrict__ items,
                                          unsigned* v) {
  for (unsigned b = cta; b < big[0]; b += ctas) {
    const unsigned cell = mid_list[b], s = start[cell], m = start[cell + 1] - s;
    unsigned pow2 = 2;
    while (pow2 < m) pow2 *= 2;
    for (unsigned i = threadIdx.x; i < pow2; i += kOrderThreads) v[i] = i < m ? slot[s + i].y : 0xffffffffu;
    __syncthreads();
    for (unsigned k = 2; k <= pow2; k *= 2)
      for (unsigned j = k / 2; j > 0; j /= 2) {
        for (unsigned t = threadIdx.x; t < pow2 / 2; t += kOrderThreads) {
          const unsigned lo = 2 * t - (t & (j - 1)), hi = lo + j;
          const unsigned a = v[lo], c = v[hi];
          if ((a > c) == ((lo & k) == 0)) v[lo] = c, v[hi] = a;
        }
        __syncthreads();
      }
    for (unsigned i = threadIdx.x; i < m; i += kOrderThreads) items[s + i] = v[i];
    __syncthreads();
  }
}

// One cell and one window of kWindow indices at a time: the cell's indices in
// the window are marked in a bitmap (kSortMax words) and read off it, after those
// before the window.
__device__ __forceinline__ void order_big(unsigned cta, unsigned ctas, int n, const uint2* __restrict__ slot,
                                          const unsigned* __restrict__ start, const unsigned* __restrict__ big,
                                          const unsigned* __restrict__ big_list, unsigned* __restrict__ items,
                                          unsigned* bits) {
  constexpr unsigned kWords = kSortMax, kPer = kWords / kOrderThreads;
  __shared__ unsigned sh[32], warp_sum[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  const unsigned windows = ((unsigned)n + kWindow - 1) / kWindow;
  const unsigned long long units = (unsigned long long)big[1] * windows;
  for (unsigned long long u = cta; u < units; u += ctas) {
    const unsigned cell = big_list[u / windows], first = (unsigned)(u % windows) * kWindow;
    const unsigned s = start[cell], e = start[cell + 1];
    for (unsigned w = threadIdx.x; w < kWords; w += kOrderThreads) bits[w] = 0;
    __syncthreads();
    unsigned before = 0;
#pragma unroll 4
    for (unsigned q = s + threadIdx.x; q < e; q += kOrderThreads) {
      const unsigned i = slot[q].y;
      before += i < first;
      if (i >= first && i - first < kWindow) atomicOr(&bits[(i - first) / 32], 1u << (i & 31));
    }
    before = block_sum<kOrderThreads>(before, sh);  // its barriers also end the marking
    unsigned cnt = 0;
#pragma unroll
    for (unsigned w = 0; w < kPer; ++w) cnt += __popc(bits[threadIdx.x * kPer + w]);
    const unsigned inc = warp_inclusive(cnt);
    if (lane == 31) warp_sum[wid] = inc;
    __syncthreads();
    const unsigned ws_ = warp_sum[lane], winc = warp_inclusive(ws_);
    unsigned at = s + before + __shfl_sync(0xffffffffu, winc - ws_, wid) + inc - cnt;
    for (unsigned w = 0; w < kPer; ++w)
      for (unsigned x = bits[threadIdx.x * kPer + w]; x; x &= x - 1)
        items[at++] = first + (threadIdx.x * kPer + w) * 32 + __ffs(x) - 1;
    __syncthreads();
  }
}

// The cells that k_order left: the first mid_ctas CTAs take the mid ones, the others the big ones.
__global__ void __launch_bounds__(kOrderThreads) k_order_large(int n, unsigned mid_ctas, const uint2* __restrict__ slot,
                                                               const unsigned* __restrict__ start,
                                                               const unsigned* __restrict__ big,
                                                               const unsigned* __restrict__ mid_list,
                                                               const unsigned* __restrict__ big_list,
                                                               unsigned* __restrict__ items) {
  pdl_entry();
  __shared__ unsigned v[kSortMax];
  if (blockIdx.x < mid_ctas)
    order_mid(blockIdx.x, mid_ctas, slot, start, big, mid_list, items, v);
  else
    order_big(blockIdx.x - mid_ctas, gridDim.x - mid_ctas, n, slot, start, big, big_list, items, v);
}

}  // namespace

// Exclusive scan of n values; out[n] receives the total when out has n+1 slots.
vg_status exclusive_scan(Ctx* c, const unsigned* in, size_t n, unsigned* out, bool write_total) {
  const size_t tiles = (n + kScanTile - 1) / kScanTile;
  const size_t chunk = ((tiles + kScanCtas - 1) / kScanCtas) * kScanTile;
  const unsigned ctas = n ? (unsigned)((n + chunk - 1) / chunk) : 1;
  vg_status st = VG_OK;
  unsigned* sums = (unsigned*)ws(c, S_SCAN, kScanCtas * sizeof(unsigned), &st);
  if (st != VG_OK) return st;
  if (ctas > 1) {
    pdl_launch(c->stream, ctas, kScanThreads, 0, k_scan_sums, in, n, chunk, sums);
    VG_LAUNCHED(c);
  }
  pdl_launch(c->stream, ctas, kScanThreads, 0, k_scan_chunks, in, n, chunk, (const unsigned*)sums, out,
             write_total ? 1 : 0);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status build_cell_lists(Ctx* c, const Geom& g, const float4* ps, size_t n, CellLists* out) {
  const size_t ncells = g.points();
  if (n > 0x7fffffff || ncells >= 0xffffffffu) return fail(c, VG_TOO_LARGE, "cell lists: too many vortons or cells");
  vg_status st = VG_OK;
  // one slot per grid point and one for vortons outside the grid
  const size_t slots = ncells + 1;
  // S_CELL: slot (2 n), key and later items, place (n each), lists of the mid and the big cells
  const size_t mids = n / (kCountMax + 1) + 1, bigs = n / (kSortMax + 1) + 1;
  uint2* slot = (uint2*)ws(c, S_CELL, (4 * n + mids + bigs) * sizeof(unsigned), &st);
  if (st != VG_OK) return st;
  // S_COUNT: count (slots), numbers of mid and big cells
  unsigned* count = (unsigned*)ws(c, S_COUNT, (slots + 2) * sizeof(unsigned), &st);
  if (st != VG_OK) return st;
  unsigned* start = (unsigned*)ws(c, S_START, (slots + 1) * sizeof(unsigned), &st);
  if (st != VG_OK) return st;
  unsigned* key = (unsigned*)(slot + n);
  unsigned *place = key + n, *items = key, *mid_list = place + n, *big_list = mid_list + mids;
  unsigned* big = count + slots;
  VG_CUDA(c, cudaMemsetAsync(count, 0, (slots + 2) * sizeof(unsigned), c->stream));
  if (n > 0) {
    pdl_launch(c->stream, blocks_for(n, 256), 256, 0, k_bin, g, ps, (int)n, key, place, count, (unsigned)ncells);
    VG_LAUNCHED(c);
  }
  st = exclusive_scan(c, count, slots, start, true);
  if (st != VG_OK) return st;
  if (n > 0) {
    pdl_launch(c->stream, blocks_for(n, 256), 256, 0, k_place, (int)n, (const unsigned*)key, (const unsigned*)place,
               (const unsigned*)start, slot);
    VG_LAUNCHED(c);
    pdl_launch(c->stream, blocks_for(n, 256), 256, 0, k_order, (int)n, (const uint2*)slot, (const unsigned*)start, items,
               big, mid_list, big_list);
    VG_LAUNCHED(c);
  }
  if (n > kCountMax) {
    const unsigned mid_ctas = (unsigned)(mids - 1 < kMidCtas ? mids - 1 : kMidCtas), big_ctas = n > kSortMax ? kBigCtas : 0;
    pdl_launch(c->stream, mid_ctas + big_ctas, kOrderThreads, 0, k_order_large, (int)n, mid_ctas, (const uint2*)slot,
               (const unsigned*)start, (const unsigned*)big, (const unsigned*)mid_list, (const unsigned*)big_list, items);
    VG_LAUNCHED(c);
  }
  VG_CUDA(c, cudaGetLastError());
  out->start = start;
  out->items = items;
  return VG_OK;
}

}  // namespace vg
