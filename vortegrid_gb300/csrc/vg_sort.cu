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
//      to k_order_large, where a warp, a group of warps or a CTA sorts their
//      indices in registers or marks them in bitmaps, a window of indices at a time.
// The result does not depend on thread timing.
//
// Bound by launches and the latency of dependent accesses: seven small kernels,
// 262,144 vortons on a 129^3 grid in 26 us.  (A stable radix sort by cell in two
// passes of 11 bits, fifteen kernels, took 69 us; its scatter, three barriers to
// every 256 keys of a tile, 13 us a pass.)
#include <algorithm>

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
// Up to kCountMax vortons each counts the smaller indices of its cell, as many
// loads as the cell has vortons; up to kWarpMax a warp sorts them, up to kGroupMax
// eight warps, up to sort_max a CTA; bitmaps order larger cells.  Whole builds of
// 10^6 vortons, us, by a radix sort / counts up to 512 and sorts in shared memory /
// this: 82 a cell 114 / 79 / 80, 125 a cell 114 / 87 / 80, 455 a cell 116 / 156 / 77,
// 578 a cell 117 / 152 / 89, 1,371 a cell 121 / 129 / 94, 2,915 a cell 132 / 135 / 107.
// With kCountMax 192, 125 a cell take 88; with 48, four million at 41 a cell take 172,
// not 166.  CTAs of 512 threads: of 1,024 with as many registers each, one fills an
// SM and waits for it to drain (32 steps at once on streams 0.9 % longer).
constexpr unsigned kCountMax = 96, kWarpMax = 512, kGroupMax = 2048, kSortMax = 8192;
constexpr int kOrderThreads = 512, kOrderWarps = kOrderThreads / 32, kGroup = 256;
constexpr unsigned kMaxWindowBits = 18, kMinWindowBits = 12;  // log2 of a bitmap's indices: 32 KB and 512 B
constexpr unsigned kOrderCtas = 304, kWindows = 152;
constexpr unsigned kChunk = 32;  // slots whose extreme indices k_order writes down: a warp's

__global__ void k_place(int n, const unsigned* __restrict__ key, const unsigned* __restrict__ place,
                        const unsigned* __restrict__ start, uint2* __restrict__ slot) {
  pdl_entry();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (unsigned)n) return;
  const unsigned k = key[i];
  slot[start[k] + place[i]] = make_uint2(k, i);
}

// Lists of the cells that k_order leaves, and their lengths.
struct LargeCells {
  unsigned* count;    // of each list
  unsigned* cell[4];  // for a warp, for a group, for a CTA, for bitmaps
};

// range: of a warp's slots in cells for bitmaps, the least and the greatest index.
__global__ void k_order(int n, unsigned sort_max, const uint2* __restrict__ slot, const unsigned* __restrict__ start,
                        unsigned* __restrict__ items, LargeCells large, uint2* __restrict__ range) {
  pdl_entry();
  const unsigned p = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = p < (unsigned)n;
  uint2 me = make_uint2(0, 0);
  unsigned s = 0, e = 0;
  if (valid) {
    me = slot[p];
    s = start[me.x];
    e = start[me.x + 1];
  }
  const unsigned m = e - s;
  const bool big = m > sort_max;
  if (__any_sync(0xffffffffu, big)) {
    const unsigned lo = __reduce_min_sync(0xffffffffu, big ? me.y : 0xffffffffu);
    const unsigned hi = __reduce_max_sync(0xffffffffu, big ? me.y : 0u);
    if ((threadIdx.x & 31) == 0) range[p / kChunk] = make_uint2(lo, hi);
  }
  if (m > kCountMax) {
    if (p == s) {
      const int k = (m > kWarpMax) + (m > kGroupMax) + big;
      (k < 2 ? k == 0 ? large.cell[0] : large.cell[1]
             : k == 2 ? large.cell[2] : large.cell[3])[atomicAdd(&large.count[k], 1u)] = me.x;
    }
  } else if (valid) {
    unsigned rank = 0;
    if (m > 1)
#pragma unroll 4
      for (unsigned q = s; q < e; ++q) rank += slot[q].y < me.y;
    items[s + rank] = me.y;
  }
}

// Barrier of the kThreads threads that sort a cell.
template <int kThreads>
__device__ __forceinline__ void sort_sync() {
  if constexpr (kThreads == kOrderThreads)
    __syncthreads();
  else
    asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / kThreads), "n"(kThreads) : "memory");
}

// Bound by the latency of a cell's chain (list, start, slots, then the exchanges),
// hence few barriers: only pairs in different warps meet in shared memory.
// Bitonic sort of m indices (up to kThreads R) from slot to items, R of them in a
// thread's registers: thread t ends with those of ranks t R to t R + R - 1.  Pairs
// R or more apart are exchanged between the lanes of a warp, those 32 R or more
// apart by v (kThreads R values; unused for a warp).
template <int kThreads, int R>
__device__ __forceinline__ void sort_cell(int t, unsigned m, const uint2* __restrict__ slot,
                                          unsigned* __restrict__ items, unsigned* v) {
  unsigned x[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const unsigned i = r * kThreads + t;
    x[r] = i < m ? slot[i].y : 0xffffffffu;  // no index: those of vortons are below 2^31
  }
  auto pass = [&](int a, int b, bool up) {
    const unsigned lo = min(x[a], x[b]), hi = max(x[a], x[b]);
    x[a] = up ? lo : hi;
    x[b] = up ? hi : lo;
  };
#pragma unroll
  for (int k = 2; k < R; k *= 2)
#pragma unroll
    for (int j = k / 2; j > 0; j /= 2)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (!(r & j)) pass(r, r + j, !(r & k));
  // k, j: in threads from here on, runs of k sorted; the last run is all
#pragma unroll 1
  for (int k = 1; k <= kThreads; k *= 2) {
    const bool up = !(t & k);
#pragma unroll 1
    for (int j = k / 2; j > 0; j /= 2) {
      const bool low = up == !(t & j);
      if (kThreads == 32 || j < 32) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const unsigned y = __shfl_xor_sync(0xffffffffu, x[r], j);
          x[r] = low ? min(x[r], y) : max(x[r], y);
        }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) v[r * kThreads + t] = x[r];
        sort_sync<kThreads>();
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const unsigned y = v[r * kThreads + (t ^ j)];
          x[r] = low ? min(x[r], y) : max(x[r], y);
        }
        sort_sync<kThreads>();
      }
    }
#pragma unroll
    for (int j = R / 2; j > 0; j /= 2)
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (!(r & j)) pass(r, r + j, up);
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    if ((unsigned)(t * R + r) < m) items[t * R + r] = x[r];
}

// One cell and one window of indices at a time: the cell's indices in the window
// are marked in a bitmap and read off it, after those before the window.  The
// windows are as wide as leaves every SM one (304 of them instead of 152: 16 million
// vortons in one cell 2,173 us, not 1,499: every window reads all ranges).  Vortons get their places as
// k_bin's blocks run, so that the indices of a chunk of slots lie close together:
// by their range most chunks are before the window or behind it as a whole.
// Whole builds, us, by a radix sort / windows of 2^18 that read all slots of their
// cell, and a sort of every cell up to 8,192 / this: 10,000 vortons, half of them
// outside 74 / 78 / 47; 100,000 in one cell 135 / 144 / 53; 16 million in 64 cells
// 1,733 / 2,026 / 1,280, in one cell 11,277 / 3,132 / 1,499, scattered 1,018 / 623 / 628.
__device__ __forceinline__ void order_big(unsigned cta, unsigned ctas, int n, const uint2* __restrict__ slot,
                                          const uint2* __restrict__ range, const unsigned* __restrict__ start,
                                          unsigned cells, const unsigned* big_list, unsigned* __restrict__ items,
                                          unsigned* bits) {
  __shared__ unsigned sh[32], warp_sum[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
  unsigned log = kMaxWindowBits;
  auto windows_of = [&](unsigned b) { return ((unsigned)n + (1u << b) - 1) >> b; };
  while (log > kMinWindowBits && (unsigned long long)cells * windows_of(log) < min(ctas, kWindows)) --log;
  const unsigned window = 1u << log, words = window / 32, per = words > kOrderThreads ? words / kOrderThreads : 1;
  const unsigned windows = windows_of(log);
  const unsigned long long units = (unsigned long long)cells * windows;
  for (unsigned long long u = cta; u < units; u += ctas) {
    const unsigned cell = big_list[u / windows], first = (unsigned)(u % windows) << log;
    const unsigned s = start[cell], e = start[cell + 1], c1 = (e - 1) / kChunk;
    for (unsigned w = threadIdx.x; w < words; w += kOrderThreads) bits[w] = 0;
    __syncthreads();
    unsigned before = 0;
    // a warp looks at every kOrderWarps-th chunk, 32 of them at a time, then at the slots of those that it has to,
    // 8 at a time
    for (unsigned c0 = s / kChunk + wid; c0 <= c1; c0 += kOrderThreads) {
      const unsigned c = c0 + kOrderWarps * lane;
      bool in = false;
      if (c <= c1) {
        const uint2 r = range[c];
        if (r.y < first)
          before += min(c * kChunk + kChunk, e) - max(c * kChunk, s);
        else
          in = r.x < first + window;
      }
      unsigned todo = __ballot_sync(0xffffffffu, in);
      while (todo) {
        constexpr int kAt = 8;
        unsigned i[kAt];
#pragma unroll
        for (int k = 0; k < kAt; ++k, todo &= todo - 1) {
          const unsigned q = (c0 + kOrderWarps * (__ffs(todo) - 1)) * kChunk + lane;
          i[k] = todo && q >= s && q < e ? slot[q].y : 0xffffffffu;
        }
#pragma unroll
        for (int k = 0; k < kAt; ++k) {
          before += i[k] < first;
          if (i[k] >= first && i[k] - first < window) atomicOr(&bits[(i[k] - first) / 32], 1u << (i[k] & 31));
        }
      }
    }
    before = block_sum<kOrderThreads>(before, sh);  // its barriers also end the marking
    const unsigned w0 = threadIdx.x * per;  // this thread's words; none past the bitmap
    unsigned cnt = 0;
    if (w0 < words)
      for (unsigned w = 0; w < per; ++w) cnt += __popc(bits[w0 + w]);
    const unsigned inc = warp_inclusive(cnt);
    if (lane == 31) warp_sum[wid] = inc;
    __syncthreads();
    const unsigned ws_ = lane < kOrderWarps ? warp_sum[lane] : 0, winc = warp_inclusive(ws_);
    unsigned at = s + before + __shfl_sync(0xffffffffu, winc - ws_, wid) + inc - cnt;
    if (__shfl_sync(0xffffffffu, winc, 31) > 4 * words) {  // a word a warp, its indices side by side
      for (unsigned l = 0; l < 32; ++l) {
        unsigned to = __shfl_sync(0xffffffffu, at, l);
        const unsigned wl = (wid * 32 + l) * per;
        if (wl >= words) break;
        for (unsigned w = wl; w < wl + per; ++w) {
          const unsigned x = bits[w];
          if ((x >> lane) & 1u) items[to + __popc(x & ((1u << lane) - 1u))] = first + w * 32 + lane;
          to += __popc(x);
        }
      }
    } else if (w0 < words) {
      for (unsigned w = w0; w < w0 + per; ++w)
        for (unsigned x = bits[w]; x; x &= x - 1) items[at++] = first + w * 32 + __ffs(x) - 1;
    }
    __syncthreads();
  }
}

// The cells that k_order left.  Every thread works by the same counts, those
// that its block read: they decide who meets at the barriers.
__global__ void __launch_bounds__(kOrderThreads) k_order_large(int n, const uint2* __restrict__ slot,
                                                               const uint2* __restrict__ range,
                                                               const unsigned* __restrict__ start,
                                                               const LargeCells large, unsigned* __restrict__ items) {
  pdl_entry();
  __shared__ unsigned v[kSortMax], count[4];
  unsigned any = 0;
  if (threadIdx.x < 4) count[threadIdx.x] = any = large.count[threadIdx.x];
  if (!__syncthreads_or(any)) return;
  const int t = threadIdx.x, lane = t & 31;
  for (unsigned b = blockIdx.x + gridDim.x * (t / 32); b < count[0]; b += gridDim.x * kOrderWarps) {
    const unsigned cell = large.cell[0][b], s = start[cell], m = start[cell + 1] - s;
    if (m <= 128)
      sort_cell<32, 4>(lane, m, slot + s, items + s, nullptr);
    else if (m <= 256)
      sort_cell<32, 8>(lane, m, slot + s, items + s, nullptr);
    else
      sort_cell<32, 16>(lane, m, slot + s, items + s, nullptr);
  }
  static_assert(kGroupMax == 8 * kGroup && kSortMax == 16 * kOrderThreads, "what a thread holds");
  const int group = t / kGroup;
  for (unsigned b = blockIdx.x + gridDim.x * group; b < count[1]; b += gridDim.x * (kOrderThreads / kGroup)) {
    const unsigned cell = large.cell[1][b], s = start[cell], m = start[cell + 1] - s;
    if (m <= 4 * kGroup)
      sort_cell<kGroup, 4>(t % kGroup, m, slot + s, items + s, v + kGroupMax * group);
    else
      sort_cell<kGroup, 8>(t % kGroup, m, slot + s, items + s, v + kGroupMax * group);
  }
  __syncthreads();  // v is one from here on
  for (unsigned b = blockIdx.x; b < count[2]; b += gridDim.x) {
    const unsigned cell = large.cell[2][b], s = start[cell], m = start[cell + 1] - s;
    if (m <= 8 * kOrderThreads)
      sort_cell<kOrderThreads, 8>(t, m, slot + s, items + s, v);
    else
      sort_cell<kOrderThreads, 16>(t, m, slot + s, items + s, v);
  }
  order_big(blockIdx.x, gridDim.x, n, slot, range, start, count[3], large.cell[3], items, v);
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
  // A cell's bitmaps cost by the windows that all n indices fill, its sort by its
  // own vortons.  Whole builds, us, all sorted / all by bitmaps: 262,144 vortons, 4,096
  // a cell 66 / 54; 600,000, 2,777 a cell 85 / 98, 4,800 a cell 107 / 94; 10^6, 2,915 a cell
  // 106 / 134, 8,000 a cell 136 / 121; two million, 5,830 a cell 174 / 223.
  const unsigned sort_max = (unsigned)std::clamp<size_t>(((n >> kMaxWindowBits) + 1) * 1024, kGroupMax, kSortMax);
  // S_CELL: slot (2 n), ranges (2 chunks), key and later items, place (n each), the lists of large cells
  const size_t chunks = (n + kChunk - 1) / kChunk;
  const size_t of_warps = n / (kCountMax + 1), of_groups = n / (kWarpMax + 1), of_ctas = n / (kGroupMax + 1),
               of_bitmaps = n / (sort_max + 1);
  uint2* slot = (uint2*)ws(
      c, S_CELL, (4 * n + 2 * chunks + of_warps + of_groups + of_ctas + of_bitmaps + 2) * sizeof(unsigned), &st);
  if (st != VG_OK) return st;
  // S_COUNT: count (slots), the lists' lengths
  unsigned* count = (unsigned*)ws(c, S_COUNT, (slots + 4) * sizeof(unsigned), &st);
  if (st != VG_OK) return st;
  unsigned* start = (unsigned*)ws(c, S_START, (slots + 1) * sizeof(unsigned), &st);
  if (st != VG_OK) return st;
  uint2* range = slot + n;
  unsigned* key = (unsigned*)(range + chunks);
  unsigned *place = key + n, *items = key;
  LargeCells large = {count + slots, {place + n}};
  large.cell[1] = large.cell[0] + of_warps;
  large.cell[2] = large.cell[1] + of_groups;
  large.cell[3] = large.cell[2] + of_ctas;
  VG_CUDA(c, cudaMemsetAsync(count, 0, (slots + 4) * sizeof(unsigned), c->stream));
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
    pdl_launch(c->stream, blocks_for(n, 256), 256, 0, k_order, (int)n, sort_max, (const uint2*)slot,
               (const unsigned*)start, items, large, range);
    VG_LAUNCHED(c);
  }
  if (n > kCountMax) {
    // as many as there can be cells, or windows of those for bitmaps
    const unsigned ctas =
        (unsigned)std::min<size_t>(std::max(of_warps, of_bitmaps * ((n >> kMinWindowBits) + 1)), kOrderCtas);
    pdl_launch(c->stream, ctas, kOrderThreads, 0, k_order_large, (int)n, (const uint2*)slot, (const uint2*)range,
               (const unsigned*)start, large, items);
    VG_LAUNCHED(c);
  }
  VG_CUDA(c, cudaGetLastError());
  out->start = start;
  out->items = items;
  return VG_OK;
}

}  // namespace vg
