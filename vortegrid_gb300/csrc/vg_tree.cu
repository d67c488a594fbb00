// K3/K4/K5: NestedGrid influence tree, treecode evaluation, boundary vector
// potential and the vorticity splat.
//
//  * k_leaf      -- MakeBaseVortonGrid (VortonFluid/vortonSim.cpp:1192-1321):
//                   one thread per leaf point sums its cell's vortons in index
//                   order (|w|-weighted centroid with the FLT_MIN-seeded weight
//                   of vortonClusterAux.h:71, vorticity sum, last size);
//  * k_aggregate -- AggregateClusters (vortonSim.cpp:1337-1569), one launch
//                   per parent layer, children in the reference's z,y,x order;
//  * k_tree_eval -- ComputeVelocity_Tree / ComputeVectorPotential_Tree
//                   (vortonSim.cpp:1650-1905) as an explicit-stack walk that
//                   keeps one partial sum per open layer and adds it to its
//                   parent exactly where the recursion returns, so REFERENCE
//                   numerics reproduce the recursive sum bit for bit;
//  * boundary    -- ComputeVectorPotentialAtGridpoints_Slice with
//                   boundariesOnly (vortonSim.cpp:2055-2138): one thread per
//                   face point;
//  * k_splat     -- PopulateVorticityGridFromVortons + UniformGrid::Accumulate
//                   (vortonSim.cpp:2372-2436, uniformGrid.h:1278-1342) as a
//                   gather: each grid point merges the index-sorted lists of
//                   its 8 adjacent cells and adds their trilinear shares in
//                   vorton-index order -- the reference's summation order --
//                   with no atomics.
// The tree build and the splat always use the reference's operation order
// (they are a small share of the step); FAST numerics change only the
// per-pair law inside the tree walk.
#include <float.h>

#include "vg_internal.cuh"

namespace vg {

namespace {

struct TreeParams {
  int depth;
  Geom layer[kMaxLayers];
  unsigned decim[kMaxLayers][3];
  unsigned long long base[kMaxLayers];
};

__device__ __forceinline__ float ref_vort_mag(float4 w) {
  const float a = __fmul_rn(w.x, 2.0f), b = __fmul_rn(w.y, 2.0f), c = __fmul_rn(w.z, 2.0f);
  return __fsqrt_rn(ref_dot_self(a, b, c));
}

// Two vortons at a time: a leaf's vortons cost two dependent memory latencies each
// otherwise (14 us for the eight rings, now 8 us); four take registers that the
// many empty leaves of a large grid pay for (75 us for 7 million, two 63 us).
constexpr unsigned kLeafBatch = 2;
__global__ void k_leaf(Geom g, const float4* __restrict__ ps, const float4* __restrict__ w,
                       const unsigned* __restrict__ start, const unsigned* __restrict__ items,
                       float4* __restrict__ out_pos, float4* __restrict__ out_w) {
  pdl_entry();
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.points()) return;
  float px = 0.f, py = 0.f, pz = 0.f, wx = 0.f, wy = 0.f, wz = 0.f, size = 0.f, aux = FLT_MIN;
  const unsigned b = start[c], e = start[c + 1];
  for (unsigned k = b; k < e; k += kLeafBatch) {  // a batch's loads at a time: two latencies for all of them
    unsigned i[kLeafBatch];
    float4 p[kLeafBatch], a[kLeafBatch];
#pragma unroll
    for (unsigned u = 0; u < kLeafBatch; ++u) i[u] = items[k + u < e ? k + u : k];
#pragma unroll
    for (unsigned u = 0; u < kLeafBatch; ++u)
      if (k + u < e) {
        p[u] = ps[i[u]];
        a[u] = w[i[u]];
      }
#pragma unroll
    for (unsigned u = 0; u < kLeafBatch; ++u) {
      if (k + u >= e) break;
      const float mag = ref_vort_mag(a[u]);
      px = __fadd_rn(px, __fmul_rn(p[u].x, mag));
      py = __fadd_rn(py, __fmul_rn(p[u].y, mag));
      pz = __fadd_rn(pz, __fmul_rn(p[u].z, mag));
      wx = __fadd_rn(wx, a[u].x);
      wy = __fadd_rn(wy, a[u].y);
      wz = __fadd_rn(wz, a[u].z);
      size = p[u].w;
      aux = __fadd_rn(aux, mag);
    }
  }
  if (aux != FLT_MIN) {
    const float r = __fdiv_rn(1.0f, aux);
    px = __fmul_rn(px, r);
    py = __fmul_rn(py, r);
    pz = __fmul_rn(pz, r);
  }
  out_pos[c] = make_float4(px, py, pz, size);
  out_w[c] = make_float4(wx, wy, wz, 0.f);
}

// AggregateClusters for parent point k of layer P from its children in C
// (decimation d): vorticity-weighted centroid, summed angular velocity, the
// last child's nonzero size.
constexpr unsigned kBatch = 4;
__device__ __forceinline__ void aggregate_point(const Geom& P, const Geom& C, uint3 d, const float4* __restrict__ cpos,
                                                const float4* __restrict__ cw, float4* __restrict__ ppos,
                                                float4* __restrict__ pw, size_t k) {
  const unsigned k32 = (unsigned)k;  // a tree's layers have fewer than 2^32 points
  const unsigned px = k32 % P.np[0], py = k32 / P.np[0] % P.np[1], pz = k32 / P.np[0] / P.np[1];
  float x = 0.f, y = 0.f, z = 0.f, wx = 0.f, wy = 0.f, wz = 0.f, size = 0.f;
  if (px < P.np[0] - 1 && py < P.np[1] - 1 && pz < P.np[2] - 1) {
    float aux = FLT_MIN;
    // the children in z, y, x order, kBatch of them loaded at a time: one memory latency for the batch
    const size_t o0 = px * d.x + (size_t)C.np[0] * (py * d.y + (size_t)C.np[1] * (pz * d.z));
    const unsigned total = d.x * d.y * d.z;
    unsigned ix = 0, iy = 0, iz = 0;
    for (unsigned k0 = 0; k0 < total; k0 += kBatch) {
      float4 p[kBatch], a[kBatch];
#pragma unroll
      for (unsigned u = 0; u < kBatch; ++u)
        if (k0 + u < total) {
          const size_t o = o0 + ix + (size_t)C.np[0] * (iy + (size_t)C.np[1] * iz);
          p[u] = cpos[o];
          a[u] = cw[o];
          if (++ix == d.x) {
            ix = 0;
            if (++iy == d.y) {
              iy = 0;
              ++iz;
            }
          }
        }
#pragma unroll
      for (unsigned u = 0; u < kBatch; ++u) {
        if (k0 + u >= total) break;
        const float mag = ref_vort_mag(a[u]);
        x = __fadd_rn(x, __fmul_rn(p[u].x, mag));
        y = __fadd_rn(y, __fmul_rn(p[u].y, mag));
        z = __fadd_rn(z, __fmul_rn(p[u].z, mag));
        wx = __fadd_rn(wx, a[u].x);
        wy = __fadd_rn(wy, a[u].y);
        wz = __fadd_rn(wz, a[u].z);
        aux = __fadd_rn(aux, mag);
        if (p[u].w != 0.0f) size = p[u].w;
      }
    }
    const float r = __fdiv_rn(1.0f, aux);
    x = __fmul_rn(x, r);
    y = __fmul_rn(y, r);
    z = __fmul_rn(z, r);
  }
  ppos[k] = make_float4(x, y, z, size);
  pw[k] = make_float4(wx, wy, wz, 0.f);
}

__global__ void k_aggregate(Geom P, Geom C, uint3 d, const float4* __restrict__ cpos, const float4* __restrict__ cw,
                            float4* __restrict__ ppos, float4* __restrict__ pw) {
  pdl_entry();
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= P.points()) return;
  aggregate_point(P, C, d, cpos, cw, ppos, pw, k);
}

// The small top layers l0 .. depth-1 in one CTA, layer after layer (a barrier
// between them makes each layer's writes visible to the next): the same cells
// as one k_aggregate launch per layer, without a launch per few hundred points.
// Layers of up to 512 points, one to a thread: all layers up to 4,096 points took
// 12 to 18 us, now 8 us and a launch of 4.7 us where there is one between.
constexpr size_t kTopLayerPoints = 512;  // layers of at most this many points go to k_aggregate_top
constexpr int kTopThreads = 512;
__global__ void __launch_bounds__(kTopThreads) k_aggregate_top(const __grid_constant__ TreeParams T, int l0,
                                                               float4* __restrict__ sv_pos, float4* __restrict__ sv_w) {
  pdl_entry();
  for (int l = l0; l < T.depth; ++l) {
    const Geom& P = T.layer[l];
    const Geom& C = T.layer[l - 1];
    const uint3 d = make_uint3(T.decim[l][0], T.decim[l][1], T.decim[l][2]);
    for (size_t k = threadIdx.x; k < P.points(); k += blockDim.x)
      aggregate_point(P, C, d, sv_pos + T.base[l - 1], sv_w + T.base[l - 1], sv_pos + T.base[l], sv_w + T.base[l], k);
    __syncthreads();
  }
}

template <int KIND, bool REF>
__device__ __forceinline__ void add_pair(float3& acc, float qx, float qy, float qz, float4 p, float4 a, float sr,
                                         float sc) {
  if (REF)
    ref_accum<KIND>(acc, qx, qy, qz, p, a, sr, sc);
  else
    fast_accum<KIND>(acc, qx, qy, qz, p, a, sr, sc);
}

struct Frame {
  unsigned ix, iy, iz;
  int layer;
  unsigned counter;
  float ax, ay, az;
};

// Walk the tree from the root for query q (vortonSim.cpp:1650-1905).
template <int KIND, bool REF>
__device__ float3 tree_walk(const TreeParams& T, const float4* __restrict__ sp, const float4* __restrict__ sw,
                            const float4* __restrict__ ps, const float4* __restrict__ w, int n, float qx, float qy,
                            float qz, float sr, float sc) {
  float3 res = make_float3(0.f, 0.f, 0.f);
  if (T.depth <= 1) {  // no tree: direct sum (vortonSim.cpp:2125-2128)
    for (int i = 0; i < n; ++i) add_pair<KIND, REF>(res, qx, qy, qz, ps[i], w[i], sr, sc);
    return res;
  }
  Frame st[kMaxLayers];
  int top = 0;
  st[0] = Frame{0u, 0u, 0u, T.depth - 1, 0u, 0.f, 0.f, 0.f};
  const float mfac = 0.0001f;
  for (;;) {
    Frame& F = st[top];
    const int L = F.layer;
    const unsigned d0 = T.decim[L][0], d1 = T.decim[L][1], d2 = T.decim[L][2];
    if (F.counter == d0 * d1 * d2) {
      if (top == 0) {
        res = make_float3(F.ax, F.ay, F.az);
        break;
      }
      const float cx = F.ax, cy = F.ay, cz = F.az;
      --top;
      Frame& Pf = st[top];
      if (REF) {
        Pf.ax = __fadd_rn(Pf.ax, cx);
        Pf.ay = __fadd_rn(Pf.ay, cy);
        Pf.az = __fadd_rn(Pf.az, cz);
      } else {
        Pf.ax += cx;
        Pf.ay += cy;
        Pf.az += cz;
      }
      Pf.counter++;
      continue;
    }
    const Geom& C = T.layer[L - 1];
    const unsigned c = F.counter;
    const unsigned ix = c % d0, iy = (c / d0) % d1, iz = c / (d0 * d1);
    const unsigned chx = F.ix * d0 + ix, chy = F.iy * d1 + iy, chz = F.iz * d2 + iz;
    bool open = false;
    if (L > 1) {
      const float mx = __fmul_rn(mfac, C.cell[0]);
      const float my = __fmul_rn(mfac, C.cell[1]);
      const float mz = __fadd_rn(__fmul_rn(mfac, C.cell[2]), (0.0f == C.cell[2]) ? FLT_MIN : 0.0f);
      const float lox = __fadd_rn(C.mn[0], __fmul_rn((float)chx, C.cell[0]));
      const float hix = __fadd_rn(C.mn[0], __fmul_rn((float)(chx + 1), C.cell[0]));
      const float loy = __fadd_rn(C.mn[1], __fmul_rn((float)chy, C.cell[1]));
      const float hiy = __fadd_rn(C.mn[1], __fmul_rn((float)(chy + 1), C.cell[1]));
      const float loz = __fadd_rn(C.mn[2], __fmul_rn((float)chz, C.cell[2]));
      const float hiz = __fadd_rn(C.mn[2], __fmul_rn((float)(chz + 1), C.cell[2]));
      open = (qx >= __fsub_rn(lox, mx)) && (qy >= __fsub_rn(loy, my)) && (qz >= __fsub_rn(loz, mz)) &&
             (qx < __fadd_rn(hix, mx)) && (qy < __fadd_rn(hiy, my)) && (qz < __fadd_rn(hiz, mz));
    }
    if (open) {
      ++top;
      st[top] = Frame{chx, chy, chz, L - 1, 0u, 0.f, 0.f, 0.f};
      continue;
    }
    const size_t o = T.base[L - 1] + chx + (size_t)C.np[0] * (chy + (size_t)C.np[1] * chz);
    float3 acc = make_float3(F.ax, F.ay, F.az);
    add_pair<KIND, REF>(acc, qx, qy, qz, sp[o], sw[o], sr, sc);
    F.ax = acc.x;
    F.ay = acc.y;
    F.az = acc.z;
    F.counter++;
  }
  return res;
}

// FAST walk's per-cell constants for one call's spread factors sr, sc:
// tp = (centroid, 1 / R), tw = (angular velocity x 2/3 R^3 sc, R^2), R =
// size / 2 x sr -- what fast_accum derives from (sp, sw) at every pair.
__device__ __forceinline__ void prepare_cell(float4& p, float4& a, float sr, float sc) {
  const float radius = p.w * 0.5f * sr;
  const float s = VG_TWO_THIRDS * radius * radius * radius * sc;
  p.w = 1.0f / radius;
  a = make_float4(a.x * s, a.y * s, a.z * s, radius * radius);
}

__global__ void k_tree_prep(const float4* __restrict__ sp, const float4* __restrict__ sw, size_t total, float sr,
                            float sc, float4* __restrict__ tp, float4* __restrict__ tw) {
  pdl_entry();
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= total) return;
  float4 p = sp[k], a = sw[k];
  prepare_cell(p, a, sr, sc);
  tp[k] = p;
  tw[k] = a;
}

// fast_accum's law from prepared constants (the same mathematics, the scale
// folded into the angular velocity).
template <int KIND>
__device__ __forceinline__ void prep_accum(float3& acc, float qx, float qy, float qz, float4 tp, float4 tw) {
  const float d0 = qx - tp.x, d1 = qy - tp.y, d2 = qz - tp.z;
  const float dist2 = fmaf(d0, d0, fmaf(d1, d1, d2 * d2));
  if (KIND == 0) {
    const float inv = fminf(rsqrtf(dist2), tp.w);
    const float law = inv * inv * inv;
    const float b0 = d0 * law, b1 = d1 * law, b2 = d2 * law;
    acc.x = fmaf(tw.y, b2, fmaf(-tw.z, b1, acc.x));
    acc.y = fmaf(tw.z, b0, fmaf(-tw.x, b2, acc.y));
    acc.z = fmaf(tw.x, b1, fmaf(-tw.y, b0, acc.z));
  } else {
    const float law = (dist2 < tw.w) ? dist2 * tp.w * tp.w * tp.w : rsqrtf(dist2);
    acc.x = fmaf(tw.x, law, acc.x);
    acc.y = fmaf(tw.y, law, acc.y);
    acc.z = fmaf(tw.z, law, acc.z);
  }
}

// FAST form of the same walk.  The opening test is geometric and separable
// per axis (the query lies in the child's box widened by 1e-4 cells along x,
// y and z), so the cells opened at a layer always form a box of 1 or 2 cells
// per axis (2 where the query is within the margin of a face -- every grid
// point is).  Walk the layers with that box in registers: the children of the
// open cells that are not themselves opened add their monopoles, the opened
// ones form the next layer's box.  Same cells as tree_walk, summed layer by
// layer instead of depth first (FAST numerics sum in any order).
//
// kRawLeaf: the leaf layer's cells are prepared where they are read.  kLanes
// neighbouring lanes walk for one query, each taking every kLanes-th row of a
// layer's cells; all of them return the sum.
template <int KIND, bool kRawLeaf, int kLanes>
__device__ float3 tree_walk_fast(const TreeParams& T, const float4* __restrict__ sp, const float4* __restrict__ sw,
                                 const float4* __restrict__ tp, const float4* __restrict__ tw,
                                 const float4* __restrict__ ps, const float4* __restrict__ w, int n, float qx,
                                 float qy, float qz, float sr, float sc) {
  float3 acc = make_float3(0.f, 0.f, 0.f);
  const unsigned sub = threadIdx.x % kLanes;
  if (T.depth <= 1)  // no tree: direct sum (vortonSim.cpp:2125-2128)
    for (int i = (int)sub; i < n; i += kLanes) fast_accum<KIND>(acc, qx, qy, qz, ps[i], w[i], sr, sc);
  const float mfac = 0.0001f;
  const float q[3] = {qx, qy, qz};
  unsigned f0[3] = {0u, 0u, 0u}, fn[3] = {1u, 1u, 1u};  // open box of layer L: [f0, f0 + fn) per axis
  for (int L = T.depth - 1; L >= 1; --L) {
    const Geom& C = T.layer[L - 1];
    unsigned c0[3], cn[3], o0[3], on[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const unsigned d = T.decim[L][a];
      c0[a] = f0[a] * d;
      cn[a] = fn[a] * d;
      on[a] = 0;
      o0[a] = 0;
      if (L > 1) {  // children open along this axis: a contiguous run of 1 or 2
        const float m = (a == 2) ? __fadd_rn(__fmul_rn(mfac, C.cell[2]), (0.0f == C.cell[2]) ? FLT_MIN : 0.0f)
                                 : __fmul_rn(mfac, C.cell[a]);
        for (unsigned i = 0; i < cn[a]; ++i) {
          const unsigned ch = c0[a] + i;
          const float lo = __fadd_rn(C.mn[a], __fmul_rn((float)ch, C.cell[a]));
          const float hi = __fadd_rn(C.mn[a], __fmul_rn((float)(ch + 1), C.cell[a]));
          if (q[a] >= __fsub_rn(lo, m) && q[a] < __fadd_rn(hi, m)) {
            if (on[a] == 0) o0[a] = ch;
            ++on[a];
          }
        }
      }
    }
    const bool any = on[0] && on[1] && on[2];
    // the layer's cells (fewer than 2^32 in a layer); a row's cells are
    // consecutive, visited up to 4 at a time with their loads issued
    // together; an opened cell's term is computed and dropped (acc kept)
    const bool raw = kRawLeaf && L == 1;
    const float4* __restrict__ lp = (raw ? sp : tp) + T.base[L - 1];
    const float4* __restrict__ lw = (raw ? sw : tw) + T.base[L - 1];
    const unsigned sy = C.np[0], sz = C.np[0] * C.np[1];
    auto add_row = [&](unsigned iy, unsigned iz) {
      const unsigned chy = c0[1] + iy, chz = c0[2] + iz;
      const bool oyz = any && chz - o0[2] < on[2] && chy - o0[1] < on[1];
      const unsigned row = c0[0] + sy * chy + sz * chz;
      for (unsigned ix0 = 0; ix0 < cn[0]; ix0 += 4) {
        float4 cp[4], cw[4];
#pragma unroll
        for (unsigned u = 0; u < 4; ++u)
          if (ix0 + u < cn[0]) {
            cp[u] = lp[row + ix0 + u];
            cw[u] = lw[row + ix0 + u];
          }
#pragma unroll
        for (unsigned u = 0; u < 4; ++u) {
          const unsigned ix = ix0 + u;
          if (ix >= cn[0]) break;
          float3 next = acc;
          if (raw) prepare_cell(cp[u], cw[u], sr, sc);
          prep_accum<KIND>(next, qx, qy, qz, cp[u], cw[u]);
          if (!(oyz && c0[0] + ix - o0[0] < on[0])) acc = next;
        }
      }
    };
    if (kLanes == 1) {
      for (unsigned iz = 0; iz < cn[2]; ++iz)
        for (unsigned iy = 0; iy < cn[1]; ++iy) add_row(iy, iz);
    } else {
      for (unsigned iy = sub, iz = 0;; iy += kLanes) {
        while (iy >= cn[1] && iz < cn[2]) {
          iy -= cn[1];
          ++iz;
        }
        if (iz >= cn[2]) break;
        add_row(iy, iz);
      }
    }
    if (!any) break;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      f0[a] = o0[a];
      fn[a] = on[a];
    }
  }
  // the query's lanes only: others may be at another query, or have none
  const unsigned lanes = ((1u << kLanes) - 1u) << (threadIdx.x % 32 / kLanes * kLanes);
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) {
    acc.x += __shfl_xor_sync(lanes, acc.x, o);
    acc.y += __shfl_xor_sync(lanes, acc.y, o);
    acc.z += __shfl_xor_sync(lanes, acc.z, o);
  }
  return acc;
}

// REFERENCE numerics walk the raw cells (sp, sw); FAST the prepared ones (tp, tw),
// but with kRawLeaf the raw leaf cells.
template <int KIND, bool REF, bool kRawLeaf, int kLanes>
__device__ __forceinline__ float3 walk(const TreeParams& T, const float4* __restrict__ sp,
                                       const float4* __restrict__ sw, const float4* __restrict__ tp,
                                       const float4* __restrict__ tw, const float4* __restrict__ ps,
                                       const float4* __restrict__ w, int n, float qx, float qy, float qz, float sr,
                                       float sc) {
  if (REF) return tree_walk<KIND, true>(T, sp, sw, ps, w, n, qx, qy, qz, sr, sc);
  return tree_walk_fast<KIND, kRawLeaf, kLanes>(T, sp, sw, tp, tw, ps, w, n, qx, qy, qz, sr, sc);
}

template <int KIND, bool REF, bool kRawLeaf, int kLanes>
__global__ void __launch_bounds__(128) k_tree_eval(const __grid_constant__ TreeParams T, const float4* __restrict__ sp,
                                                    const float4* __restrict__ sw, const float4* __restrict__ tp,
                                                    const float4* __restrict__ tw, const float4* __restrict__ ps,
                                                    const float4* __restrict__ w, int n, const float4* __restrict__ q,
                                                    int m, float sr, float sc, float4* __restrict__ out) {
  pdl_entry();
  const int j = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  if (j >= m) return;
  const float4 v = q[j];
  const float3 r = walk<KIND, REF, kRawLeaf, kLanes>(T, sp, sw, tp, tw, ps, w, n, v.x, v.y, v.z, sr, sc);
  if (threadIdx.x % kLanes == 0) out[j] = make_float4(r.x, r.y, r.z, 0.f);
}

// Boundary queries, row by row of nq: z faces (nq * ny each), y faces (nq * (nz - 2)),
// then the points of the x faces ((ny - 2) * (nz - 2)).  step: points along x to a query of a row.
struct BoundaryQueries {
  size_t fz, fy, fx;  // queries of one face
  unsigned nq, step;
};

BoundaryQueries boundary_queries(const Geom& g, bool copy_odd_x) {
  BoundaryQueries b;
  b.step = copy_odd_x ? 2 : 1;
  b.nq = (g.np[0] + b.step - 1) / b.step;
  const size_t iy = g.np[1] > 2 ? g.np[1] - 2 : 0, iz = g.np[2] > 2 ? g.np[2] - 2 : 0;
  b.fz = (size_t)b.nq * g.np[1];
  b.fy = b.nq * iz;
  b.fx = iy * iz;
  return b;
}

__device__ __forceinline__ bool face_point(const Geom& g, const BoundaryQueries& b, size_t t, unsigned& x, unsigned& y,
                                           unsigned& z, bool& row) {
  const size_t nx = g.np[0], ny = g.np[1], nz = g.np[2];
  row = true;
  if (t < 2 * b.fz) {
    z = (t < b.fz) ? 0 : (unsigned)(nz - 1);
    const size_t r = t % b.fz;
    x = (unsigned)(r % b.nq) * b.step;
    y = (unsigned)(r / b.nq);
    return nz > 1 || t < b.fz;
  }
  t -= 2 * b.fz;
  if (t < 2 * b.fy) {
    y = (t < b.fy) ? 0 : (unsigned)(ny - 1);
    const size_t r = t % b.fy;
    x = (unsigned)(r % b.nq) * b.step;
    z = (unsigned)(r / b.nq) + 1;
    return ny > 1 || t < b.fy;
  }
  t -= 2 * b.fy;
  row = false;
  if (t < 2 * b.fx) {
    x = (t < b.fx) ? 0 : (unsigned)(nx - 1);
    const size_t r = t % b.fx, iy = ny - 2;
    y = (unsigned)(r % iy) + 1;
    z = (unsigned)(r / iy) + 1;
    return nx > 1 || t < b.fx;
  }
  return false;
}

// Vector potential of the tree at the grid's boundary points.  With copy_odd_x
// (step 2) an odd x has the value of the point before it, which is walked for
// once and written twice; on rows that only have their two x faces' points
// the point before the last was not computed and still holds zero.
template <bool REF, bool kRawLeaf, int kLanes>
__global__ void __launch_bounds__(128) k_boundary_vecpot(const __grid_constant__ TreeParams T, Geom g,
                                                          const float4* __restrict__ sp, const float4* __restrict__ sw,
                                                          const float4* __restrict__ tp, const float4* __restrict__ tw,
                                                          const float4* __restrict__ ps, const float4* __restrict__ w,
                                                          int n, BoundaryQueries b, float* __restrict__ grid3) {
  pdl_entry();
  const size_t t = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes;
  unsigned x, y, z;
  bool row;
  if (!face_point(g, b, t, x, y, z, row)) return;
  unsigned xq = x;
  bool zero = false;
  if (!row && b.step == 2 && (x & 1u)) {
    if (x == 1)
      xq = 0;
    else
      zero = true;
  }
  const float nudge = 1.0f - 2.0f * FLT_EPSILON;  // vortonSim.cpp:2063-2064
  float3 r = make_float3(0.f, 0.f, 0.f);
  if (!zero) {
    const float qx = __fadd_rn(g.mn[0], __fmul_rn((float)xq, __fmul_rn(g.cell[0], nudge)));
    const float qy = __fadd_rn(g.mn[1], __fmul_rn((float)y, __fmul_rn(g.cell[1], nudge)));
    const float qz = __fadd_rn(g.mn[2], __fmul_rn((float)z, __fmul_rn(g.cell[2], nudge)));
    r = walk<1, REF, kRawLeaf, kLanes>(T, sp, sw, tp, tw, ps, w, n, qx, qy, qz, 1.0f, 1.0f);
  }
  const unsigned sub = threadIdx.x % kLanes;
  if (sub) return;
  const size_t o = x + (size_t)g.np[0] * (y + (size_t)g.np[1] * z);
  grid3[3 * o] = r.x;
  grid3[3 * o + 1] = r.y;
  grid3[3 * o + 2] = r.z;
  if (row && b.step == 2 && x + 1 < g.np[0]) {
    grid3[3 * o + 3] = r.x;
    grid3[3 * o + 4] = r.y;
    grid3[3 * o + 5] = r.z;
  }
}

// Gather-form splat: point P accumulates from the 8 cells P - {0,1}^3 in
// ascending vorton index (k-way merge of the cells' sorted lists).
__global__ void __launch_bounds__(128) k_splat(Geom g, const float4* __restrict__ ps, const float4* __restrict__ w,
                                               const unsigned* __restrict__ start, const unsigned* __restrict__ items,
                                               float scale, float four_pi_over3, float cell_volume,
                                               float* __restrict__ grid3) {
  pdl_entry();
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= g.points()) return;
  // volumeCorrection = scale * (4 pi / 3 * r^3) / cellVolume, r = first vorton's radius
  const float radius = __fmul_rn(ps[0].w, 0.5f);
  const float vorton_volume = __fmul_rn(four_pi_over3, __fmul_rn(__fmul_rn(radius, radius), radius));
  const float corr = __fdiv_rn(__fmul_rn(scale, vorton_volume), cell_volume);
  const unsigned nx = g.np[0], ny = g.np[1];
  unsigned X, Y, Z;
  grid_index(k, nx, ny, X, Y, Z);
  CellMerge merge(start, items, nx, ny, X, Y, Z);
  float ax = 0.f, ay = 0.f, az = 0.f;
  for (;;) {
    unsigned best;
    const int bo = merge.next(items, best);
    if (bo < 0) break;
    const float4 p = ps[best];
    const float4 a = w[best];
    // Accumulate (uniformGrid.h:1278-1342): this point is corner `bo` of the vorton's cell.
    const float pp[3] = {p.x, p.y, p.z};
    float tw[3], om[3];
#pragma unroll
    for (int ax3 = 0; ax3 < 3; ++ax3) {
      const unsigned idx = bin_axis(pp[ax3], g.mn[ax3], g.cpe[ax3]);
      const float cmin = __fadd_rn(g.mn[ax3], __fmul_rn((float)idx, g.cell[ax3]));
      const float t = __fmul_rn(__fsub_rn(pp[ax3], cmin), g.cpe[ax3]);
      const float lo = t > 0.0f ? t : 0.0f;  // Clamp0to1 = Min2(Max2(x, 0), 1) (vec3.h:565-571)
      tw[ax3] = lo < 1.0f ? lo : 1.0f;
      om[ax3] = __fsub_rn(1.0f, tw[ax3]);
    }
    const float fx = (bo & 1) ? tw[0] : om[0];
    const float fy = (bo & 2) ? tw[1] : om[1];
    const float fz = (bo & 4) ? tw[2] : om[2];
    const float wt = __fmul_rn(__fmul_rn(fx, fy), fz);
    const float ix = __fmul_rn(__fmul_rn(a.x, 2.0f), corr);
    const float iy = __fmul_rn(__fmul_rn(a.y, 2.0f), corr);
    const float iz = __fmul_rn(__fmul_rn(a.z, 2.0f), corr);
    ax = __fadd_rn(ax, __fmul_rn(wt, ix));
    ay = __fadd_rn(ay, __fmul_rn(wt, iy));
    az = __fadd_rn(az, __fmul_rn(wt, iz));
  }
  grid3[3 * k] = ax;
  grid3[3 * k + 1] = ay;
  grid3[3 * k + 2] = az;
}

TreeParams make_params(const Tree& t) {
  TreeParams T;
  T.depth = t.depth;
  for (int l = 0; l < t.depth; ++l) {
    T.layer[l] = t.layer[l];
    for (int a = 0; a < 3; ++a) T.decim[l][a] = t.decim[l][a];
    T.base[l] = t.base[l];
  }
  return T;
}

}  // namespace

vg_status build_tree(Ctx* c, const Geom& g, const float4* ps, const float4* w, size_t n, const CellLists& cl,
                     Tree* t) {
  t->depth = nested_shape(g, t->layer, t->decim);
  if (t->depth <= 0 || t->depth > kMaxLayers) return fail(c, VG_TOO_LARGE, "influence tree: too many layers");
  size_t total = 0;
  for (int l = 0; l < t->depth; ++l) {
    t->base[l] = total;
    total += t->layer[l].points();
  }
  t->total = total;
  vg_status st = VG_OK;
  float4* mem = (float4*)ws(c, S_TREE, 2 * total * sizeof(float4), &st);
  if (st != VG_OK) return st;
  t->sv_pos = mem;
  t->sv_w = mem + total;
  const Geom& leaf = t->layer[0];
  pdl_launch(c->stream, blocks_for(leaf.points(), 256), 256, 0, k_leaf, leaf, ps, w, cl.start, cl.items, t->sv_pos,
                                                                  t->sv_w);
  VG_LAUNCHED(c);
  // the first layer from which every layer is small: those run in one CTA
  int l0 = t->depth;
  while (l0 > 1 && t->layer[l0 - 1].points() <= kTopLayerPoints) --l0;
  for (int l = 1; l < l0; ++l) {
    const Geom& P = t->layer[l];
    const uint3 d = make_uint3(t->decim[l][0], t->decim[l][1], t->decim[l][2]);
    pdl_launch(c->stream, blocks_for(P.points(), 128), 128, 0, k_aggregate, P, t->layer[l - 1], d, t->sv_pos + t->base[l - 1],
                                                                     t->sv_w + t->base[l - 1], t->sv_pos + t->base[l],
                                                                     t->sv_w + t->base[l]);
    VG_LAUNCHED(c);
  }
  if (l0 < t->depth) {
    pdl_launch(c->stream, 1, kTopThreads, 0, k_aggregate_top, make_params(*t), l0, t->sv_pos, t->sv_w);
    VG_LAUNCHED(c);
  }
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

// Whether m queries read the leaf layer's cells as they are and prepare them
// themselves: the leaf layer has seven eighths of a tree's cells, few of which lie
// next to a boundary point.  1.0 million vortons on 225 x 161 x 193 points (192,000
// queries): 75 us of preparation and 67 us of walks, now 13 and 75 us; 129^3
// (98,000): 26 and 47 us, now 4 and 57 us.  A query in every cell pays for the
// preparation (65,536 vortons' velocity grid: 3 and 86 us, else 2 and 108 us).
static bool raw_leaf(const Tree& t, size_t m) { return m < t.layer[0].points() / 8; }

// The FAST walk's prepared cells (workspace slot S_TREEPREP) for spread
// factors sr, sc: tp, tw are indexed as sv_pos, sv_w, the leaf layer left out when
// raw; nothing when the tree has no layers (the walk then sums the vortons
// directly).
static vg_status tree_prep(Ctx* c, const Tree& t, bool raw, float sr, float sc, float4** tp, float4** tw) {
  if (t.depth <= 1 || t.total == 0) return VG_OK;
  const size_t first = raw ? t.base[1] : 0, count = t.total - first;
  vg_status st = VG_OK;
  float4* buf = (float4*)ws(c, S_TREEPREP, 2 * count * sizeof(float4), &st);
  if (st != VG_OK) return st;
  *tp = buf - first;
  *tw = buf + count - first;
  pdl_launch(c->stream, blocks_for(count, 256), 256, 0, k_tree_prep, t.sv_pos + first, t.sv_w + first, count, sr, sc,
             buf, buf + count);
  VG_LAUNCHED(c);
  return VG_OK;
}

// Lanes to a query: four where the queries alone leave most of the chip idle.
// 6,146 boundary points: 22.8 us with one lane, 9.8 us with four; 25,000 points
// of a 65^3 grid: 56 and 33 us by themselves, but 32 such solves at a time 2.5 %
// slower, so the line is below; 98,000: 60 and 58 us; 192,000: 78 and 83 us.
static int walk_lanes(size_t m) { return m < 16384 ? 4 : 1; }

vg_status launch_tree_eval(Ctx* c, int kind, bool ref, const Tree& t, const float4* ps, const float4* w, size_t n,
                           const float4* q, size_t m, float sr, float sc, float4* out) {
  if (m == 0) return VG_OK;
  const TreeParams T = make_params(t);
  float4 *tp = nullptr, *tw = nullptr;
  const bool raw = !ref && raw_leaf(t, m);
  const int lanes = ref ? 1 : walk_lanes(m);
  const unsigned blocks = blocks_for(lanes * m, 128);
  if (!ref) {
    vg_status st = tree_prep(c, t, raw, sr, sc, &tp, &tw);
    if (st != VG_OK) return st;
  }
  auto launch = [&](auto kernel) {
    pdl_launch(c->stream, blocks, 128, 0, kernel, T, t.sv_pos, t.sv_w, tp, tw, ps, w, (int)n, q, (int)m, sr, sc, out);
  };
  if (kind == 0) {
    if (ref) launch(k_tree_eval<0, true, false, 1>);
    else if (lanes == 4) launch(raw ? k_tree_eval<0, false, true, 4> : k_tree_eval<0, false, false, 4>);
    else launch(raw ? k_tree_eval<0, false, true, 1> : k_tree_eval<0, false, false, 1>);
  } else {
    if (ref) launch(k_tree_eval<1, true, false, 1>);
    else if (lanes == 4) launch(raw ? k_tree_eval<1, false, true, 4> : k_tree_eval<1, false, false, 4>);
    else launch(raw ? k_tree_eval<1, false, true, 1> : k_tree_eval<1, false, false, 1>);
  }
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_boundary_vecpot(Ctx* c, const Tree& t, const Geom& g, const float4* ps, const float4* w, size_t n,
                                 bool copy_odd_x, bool ref, float* grid3) {
  const TreeParams T = make_params(t);
  const BoundaryQueries b = boundary_queries(g, copy_odd_x);
  const size_t m = 2 * (b.fz + b.fy + b.fx);
  if (m == 0) return VG_OK;
  float4 *tp = nullptr, *tw = nullptr;
  const bool raw = !ref && raw_leaf(t, m);
  const int lanes = ref ? 1 : walk_lanes(m);
  if (!ref) {
    vg_status st = tree_prep(c, t, raw, 1.0f, 1.0f, &tp, &tw);
    if (st != VG_OK) return st;
  }
  auto launch = [&](auto kernel) {
    pdl_launch(c->stream, blocks_for(lanes * m, 128), 128, 0, kernel, T, g, t.sv_pos, t.sv_w, tp, tw, ps, w, (int)n, b,
               grid3);
  };
  if (ref) launch(k_boundary_vecpot<true, false, 1>);
  else if (lanes == 4) launch(raw ? k_boundary_vecpot<false, true, 4> : k_boundary_vecpot<false, false, 4>);
  else launch(raw ? k_boundary_vecpot<false, true, 1> : k_boundary_vecpot<false, false, 1>);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_splat(Ctx* c, const Geom& g, const float4* ps, const float4* w, size_t n, const CellLists& cl,
                       float scale, float radius, float* grid3) {
  const size_t pts = g.points();
  if (n == 0) {
    VG_CUDA(c, cudaMemsetAsync(grid3, 0, pts * 3 * sizeof(float), c->stream));
    return VG_OK;
  }
  // volume correction (vortonSim.cpp:2398-2402) from the first vorton's radius,
  // evaluated in the kernel from ps[0].w so no host round trip is needed
  volatile float cell_volume = g.cell[0] * g.cell[1];
  cell_volume = cell_volume * g.cell[2];
  const float four_pi = 4.0f * 3.1415926535897932384626433832795f;
  const float four_pi_over3 = four_pi / 3.0f;
  (void)radius;
  pdl_launch(c->stream, blocks_for(pts, 128), 128, 0, k_splat, g, ps, w, cl.start, cl.items, scale, four_pi_over3,
                                                        cell_volume, grid3);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

}  // namespace vg
