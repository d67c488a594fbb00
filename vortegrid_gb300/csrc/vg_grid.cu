// Grid and particle stages of the VortonSim step (HBM / L2 bound):
//  * k_sor_rows      -- StepTowardVectorPoissonSolution, red then black,
//                       Dirichlet (Core/SpatialPartition/uniformGridMath.cpp:
//                       1116-1339): the reference colours whole x-rows by
//                       (y + z) parity and sweeps each row in +x, so one thread
//                       owns one row and walks it in order (bit-exact);
//  * k_downsample    -- UniformGrid::DownSampleSlice (uniformGrid.h:1453-1585);
//  * k_upsample      -- UniformGrid::UpSampleSlice (uniformGrid.h:1637-1700);
//  * k_jacobian      -- ComputeJacobian (uniformGridMath.cpp:304-451);
//  * k_curl          -- ComputeJacobian + ComputeCurlFromJacobian fused: only
//                       the six off-diagonal derivatives the curl needs;
//  * k_stretch       -- StretchAndTiltVortons (VortonFluid/vortonSim.cpp:
//                       2748-2820);
//  * k_pse           -- DiffuseAndDissipateVorticityPSE (vortonSim.cpp:
//                       3616-3879), order-independent form;
//  * k_gather_advect -- AssignParticleVelocityFromField (gain 1) +
//                       EvolveParticlesSlice (Particles/Operation/
//                       pclOpAdvect.cpp:42-81, pclOpEvolve.cpp:36-58);
//  * k_bbox          -- FindBoundingBox (pclOpFindBoundingBox.cpp:102-140).
// All arithmetic that the reference performs in FP32 is written with
// round-to-nearest intrinsics in the reference's order.
#include <float.h>

#include "vg_internal.cuh"

namespace vg {

namespace {

__global__ void k_sor_rows(Geom g, float* __restrict__ s, const float* __restrict__ lap, unsigned color, float r2x,
                           float r2y, float r2z, float H) {
  pdl_entry();
  // rows (y, z) interior with (z % 2 == color) ? y odd-shifted : ...
  const unsigned ny = g.np[1], nz = g.np[2], nx = g.np[0];
  const unsigned rows_per_z = (ny - 2 + 1) / 2 + 1;
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t zi = t / rows_per_z;
  const unsigned z = (unsigned)zi + 1;
  if (z + 1 > nz - 1 + 0 || z >= nz - 1) return;
  const unsigned yshift = (z % 2 == color) ? 1u : 0u;
  const unsigned y = 1 + yshift + 2 * (unsigned)(t % rows_per_z);
  if (y >= ny - 1) return;
  const size_t nxy = (size_t)nx * ny;
  const float relax = 1.72f;
  const float omr = __fsub_rn(1.0f, relax);
  size_t c = 1 + (size_t)nx * y + nxy * z;
  for (unsigned x = 1; x + 1 < nx; ++x, ++c) {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float t1 = __fmul_rn(__fadd_rn(s[3 * (c + 1) + a], s[3 * (c - 1) + a]), r2x);
      const float t2 = __fmul_rn(__fadd_rn(s[3 * (c + nx) + a], s[3 * (c - nx) + a]), r2y);
      const float t3 = __fmul_rn(__fadd_rn(s[3 * (c + nxy) + a], s[3 * (c - nxy) + a]), r2z);
      const float v = __fmul_rn(__fsub_rn(__fadd_rn(__fadd_rn(t1, t2), t3), lap[3 * c + a]), H);
      s[3 * c + a] = __fadd_rn(__fmul_rn(omr, s[3 * c + a]), __fmul_rn(relax, v));
    }
  }
}

__global__ void k_downsample(Geom F, const float* __restrict__ f, Geom C, uint3 cd, int inject,
                             float* __restrict__ out) {
  pdl_entry();
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= C.points()) return;
  const unsigned x = (unsigned)(k % C.np[0]), y = (unsigned)((k / C.np[0]) % C.np[1]),
                 z = (unsigned)(k / ((size_t)C.np[0] * C.np[1]));
  const unsigned mx = x * cd.x, my = y * cd.y, mz = z * cd.z;
  const size_t fnx = F.np[0], fnxy = (size_t)F.np[0] * F.np[1];
  if (inject) {
    const size_t o = mx + my * fnx + mz * fnxy;
    out[3 * k] = f[3 * o];
    out[3 * k + 1] = f[3 * o + 1];
    out[3 * k + 2] = f[3 * o + 2];
    return;
  }
  const float table[4] = {8.0f, 4.0f, 2.0f, 1.0f};
  const unsigned sh[3] = {cd.x / 2, cd.y / 2, cd.z / 2};
  float ax = 0.f, ay = 0.f, az = 0.f;
  for (unsigned iz = 0; iz < cd.z + sh[2]; ++iz) {
    const int s2 = (int)iz - (int)sh[2];
    const unsigned hz = mz + (unsigned)s2;
    if (hz >= F.np[2]) continue;
    for (unsigned iy = 0; iy < cd.y + sh[1]; ++iy) {
      const int s1 = (int)iy - (int)sh[1];
      const unsigned hy = my + (unsigned)s1;
      if (hy >= F.np[1]) continue;
      for (unsigned ix = 0; ix < cd.x + sh[0]; ++ix) {
        const int s0 = (int)ix - (int)sh[0];
        const unsigned hx = mx + (unsigned)s0;
        if (hx >= F.np[0]) continue;
        const float wt = table[abs(s0) + abs(s1) + abs(s2)];
        const size_t o = hx + hy * fnx + hz * fnxy;
        ax = __fadd_rn(ax, __fmul_rn(wt, f[3 * o]));
        ay = __fadd_rn(ay, __fmul_rn(wt, f[3 * o + 1]));
        az = __fadd_rn(az, __fmul_rn(wt, f[3 * o + 2]));
      }
    }
  }
  const float r = 1.0f / 64.0f;
  out[3 * k] = __fmul_rn(ax, r);
  out[3 * k + 1] = __fmul_rn(ay, r);
  out[3 * k + 2] = __fmul_rn(az, r);
}

__global__ void k_upsample(Geom C, const float* __restrict__ cv, Geom F, int interior, float* __restrict__ fv) {
  pdl_entry();
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= F.points()) return;
  const unsigned x = (unsigned)(k % F.np[0]), y = (unsigned)((k / F.np[0]) % F.np[1]),
                 z = (unsigned)(k / ((size_t)F.np[0] * F.np[1]));
  if (interior && (x == 0 || y == 0 || z == 0 || x + 1 >= F.np[0] || y + 1 >= F.np[1] || z + 1 >= F.np[2])) return;
  const float two_eps = 2.0f * FLT_EPSILON;
  const float shrink = 1.0f - 4.0f * FLT_EPSILON;
  float p[3];
  const unsigned id[3] = {x, y, z};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const float pmin = __fadd_rn(F.mn[a], __fmul_rn(__fmul_rn(fabsf(F.mn[a]), 2.0f), FLT_EPSILON));
    const float sp = __fmul_rn(F.cell[a], shrink);
    p[a] = __fadd_rn(pmin, __fmul_rn((float)id[a], sp));
  }
  (void)two_eps;
  if (!inside_cells(C, p[0], p[1], p[2])) return;
  interp<3>(C, cv, p[0], p[1], p[2], fv + 3 * k);
}

// Per-axis derivative factor and neighbours (uniformGridMath.cpp:326-344, 348-356).
__device__ __forceinline__ void diff_axis(size_t c, unsigned i, unsigned n, size_t stride, float rs, float hrs,
                                          size_t& hi, size_t& lo, float& f) {
  if (i == 0) {
    hi = c + stride; lo = c; f = rs;
  } else if (i == n - 1) {
    hi = c; lo = c - stride; f = rs;
  } else {
    hi = c + stride; lo = c - stride; f = hrs;
  }
}

__global__ void k_jacobian(Geom g, float rsx, float rsy, float rsz, const float* __restrict__ v,
                           float* __restrict__ jac) {
  pdl_entry();
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.points()) return;
  const unsigned nx = g.np[0], ny = g.np[1];
  unsigned id[3];
  grid_index(c, nx, ny, id[0], id[1], id[2]);
  const size_t stride[3] = {1, nx, (size_t)nx * ny};
  const float rs[3] = {rsx, rsy, rsz};
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    size_t hi, lo;
    float f;
    diff_axis(c, id[a], g.np[a], stride[a], rs[a], __fmul_rn(0.5f, rs[a]), hi, lo, f);
#pragma unroll
    for (int b = 0; b < 3; ++b) jac[9 * c + 3 * a + b] = __fmul_rn(__fsub_rn(v[3 * hi + b], v[3 * lo + b]), f);
  }
}

__global__ void k_curl(Geom g, float rsx, float rsy, float rsz, const float* __restrict__ v,
                       float* __restrict__ curl) {
  pdl_entry();
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= g.points()) return;
  const unsigned nx = g.np[0], ny = g.np[1];
  unsigned id[3];
  grid_index(c, nx, ny, id[0], id[1], id[2]);
  const size_t stride[3] = {1, nx, (size_t)nx * ny};
  const float rs[3] = {rsx, rsy, rsz};
  float J[3][3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    size_t hi, lo;
    float f;
    diff_axis(c, id[a], g.np[a], stride[a], rs[a], __fmul_rn(0.5f, rs[a]), hi, lo, f);
#pragma unroll
    for (int b = 0; b < 3; ++b) J[a][b] = (a == b) ? 0.f : __fmul_rn(__fsub_rn(v[3 * hi + b], v[3 * lo + b]), f);
  }
  curl[3 * c] = __fsub_rn(J[1][2], J[2][1]);
  curl[3 * c + 1] = __fsub_rn(J[2][0], J[0][2]);
  curl[3 * c + 2] = __fsub_rn(J[0][1], J[1][0]);
}

// order (optional): the vortons grouped by cell, so that a warp's vortons
// interpolate from the same few cells' corners (each vorton's update is the
// same whichever thread runs it).
__global__ void k_stretch(Geom g, const float* __restrict__ jac, const float4* __restrict__ ps,
                          float4* __restrict__ w, int n, float dt, const unsigned* __restrict__ order,
                          int* __restrict__ flag) {
  pdl_entry();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int i = order ? (int)order[t] : t;
  const float4 p = ps[i];
  if (!inside_cells(g, p.x, p.y, p.z)) {
    atomicOr(flag, (int)DF_OUT_OF_GRID);
    return;
  }
  float J[9];
  interp<9>(g, jac, p.x, p.y, p.z, J);
  float4 a = w[i];
  const float s0 = __fadd_rn(__fadd_rn(__fmul_rn(J[0], a.x), __fmul_rn(J[1], a.y)), __fmul_rn(J[2], a.z));
  const float s1 = __fadd_rn(__fadd_rn(__fmul_rn(J[3], a.x), __fmul_rn(J[4], a.y)), __fmul_rn(J[5], a.z));
  const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(J[6], a.x), __fmul_rn(J[7], a.y)), __fmul_rn(J[8], a.z));
  a.x = __fadd_rn(a.x, __fmul_rn(__fmul_rn(0.5f, s0), dt));
  a.y = __fadd_rn(a.y, __fmul_rn(__fmul_rn(0.5f, s1), dt));
  a.z = __fadd_rn(a.z, __fmul_rn(__fmul_rn(0.5f, s2), dt));
  w[i] = a;
}

// k_jacobian and k_stretch fused: the velocity Jacobian is formed at the 8
// corners of each vorton's cell from the velocity grid (the differences of
// k_jacobian at those grid points) and interpolated as interp<9> would from
// the Jacobian grid, so the 9-float-per-point grid is never written.  Same
// float operations on the same values as the two kernels; order as k_stretch.
__global__ void k_stretch_vel(Geom g, float rsx, float rsy, float rsz, const float* __restrict__ v,
                              const float4* __restrict__ ps, float4* __restrict__ w, int n, float dt,
                              const unsigned* __restrict__ order, int* __restrict__ flag) {
  pdl_entry();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int i = order ? (int)order[t] : t;
  const float4 p = ps[i];
  if (!inside_cells(g, p.x, p.y, p.z)) {
    atomicOr(flag, (int)DF_OUT_OF_GRID);
    return;
  }
  const float pp[3] = {p.x, p.y, p.z};
  unsigned idx[3];
  float tw[3], om[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    idx[a] = bin_axis(pp[a], g.mn[a], g.cpe[a]);
    const float cmin = __fadd_rn(g.mn[a], __fmul_rn((float)idx[a], g.cell[a]));
    tw[a] = __fmul_rn(__fsub_rn(pp[a], cmin), g.cpe[a]);
    om[a] = __fsub_rn(1.0f, tw[a]);
  }
  const unsigned nx = g.np[0], ny = g.np[1];
  const size_t stride[3] = {1, nx, (size_t)nx * ny};
  const float rs[3] = {rsx, rsy, rsz};
  float J[9];
  auto interpolate = [&](const float (&cv)[8]) {  // corners (dx, dy, dz), x fastest: v000, v100, v010, v110, v001, ...
    const float y0 = __fadd_rn(__fmul_rn(__fadd_rn(__fmul_rn(om[0], cv[0]), __fmul_rn(tw[0], cv[1])), om[1]),
                               __fmul_rn(__fadd_rn(__fmul_rn(om[0], cv[2]), __fmul_rn(tw[0], cv[3])), tw[1]));
    const float y1 = __fadd_rn(__fmul_rn(__fadd_rn(__fmul_rn(om[0], cv[4]), __fmul_rn(tw[0], cv[5])), om[1]),
                               __fmul_rn(__fadd_rn(__fmul_rn(om[0], cv[6]), __fmul_rn(tw[0], cv[7])), tw[1]));
    return __fadd_rn(__fmul_rn(y0, om[2]), __fmul_rn(y1, tw[2]));
  };
  // A cell whose corners all lie inside the grid differences every one of them
  // centrally, from fixed offsets; selecting each corner's neighbours took three
  // quarters of the instructions (2^18 vortons at 129^3: 42 us, now 19; 10^6 at
  // 225 x 161 x 193: 118 us, now 50).
  if (idx[0] - 1 < nx - 3 && idx[1] - 1 < ny - 3 && idx[2] - 1 < g.np[2] - 3 && nx > 3 && ny > 3 && g.np[2] > 3) {
    const float* base = v + 3 * (idx[0] + (size_t)nx * (idx[1] + (size_t)ny * idx[2]));
    const ptrdiff_t step[3] = {3, 3 * (ptrdiff_t)nx, 3 * (ptrdiff_t)nx * ny};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float hrs = __fmul_rn(0.5f, rs[a]);
      float cv[3][8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float* c = base + ((q & 1) ? step[0] : 0) + ((q & 2) ? step[1] : 0) + ((q & 4) ? step[2] : 0);
#pragma unroll
        for (int b = 0; b < 3; ++b) cv[b][q] = __fmul_rn(__fsub_rn(c[step[a] + b], c[b - step[a]]), hrs);
      }
#pragma unroll
      for (int b = 0; b < 3; ++b) J[3 * a + b] = interpolate(cv[b]);
    }
  } else {
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      const float hrs = __fmul_rn(0.5f, rs[a]);
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        float cv[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const unsigned ci[3] = {idx[0] + (q & 1), idx[1] + ((q >> 1) & 1), idx[2] + (q >> 2)};
          const size_t c = ci[0] + (size_t)nx * (ci[1] + (size_t)ny * ci[2]);
          size_t hi, lo;
          float f;
          diff_axis(c, ci[a], g.np[a], stride[a], rs[a], hrs, hi, lo, f);
          cv[q] = __fmul_rn(__fsub_rn(v[3 * hi + b], v[3 * lo + b]), f);
        }
        J[3 * a + b] = interpolate(cv);
      }
    }
  }
  float4 wa = w[i];
  const float s0 = __fadd_rn(__fadd_rn(__fmul_rn(J[0], wa.x), __fmul_rn(J[1], wa.y)), __fmul_rn(J[2], wa.z));
  const float s1 = __fadd_rn(__fadd_rn(__fmul_rn(J[3], wa.x), __fmul_rn(J[4], wa.y)), __fmul_rn(J[5], wa.z));
  const float s2 = __fadd_rn(__fadd_rn(__fmul_rn(J[6], wa.x), __fmul_rn(J[7], wa.y)), __fmul_rn(J[8], wa.z));
  wa.x = __fadd_rn(wa.x, __fmul_rn(__fmul_rn(0.5f, s0), dt));
  wa.y = __fadd_rn(wa.y, __fmul_rn(__fmul_rn(0.5f, s1), dt));
  wa.z = __fadd_rn(wa.z, __fmul_rn(__fmul_rn(0.5f, s2), dt));
  w[i] = wa;
}

// Order-independent PSE: vorton i exchanges with every vorton of the pair set
// the reference visits (same cell, or cells offset by {0,1}^3 either way with
// the lower cell strictly inside the point range), using pre-step values.
// Pre-step positions and angular velocities in cell order (pss[t], w0s[t] of
// vorton items[t]), so that each cell's vortons are contiguous for k_pse.
__global__ void k_pse_gather(const float4* __restrict__ ps, const float4* __restrict__ w, int n,
                             const unsigned* __restrict__ items, float4* __restrict__ pss, float4* __restrict__ w0s) {
  pdl_entry();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const unsigned j = items[t];
  pss[t] = ps[j];
  w0s[t] = w[j];
}

// The neighbour cells of a particle at slot t of the cell lists: its own cell
// and, on the side s = -1 and then +1 of it, those at offset s along each of
// the axes in k's bits (kAll: k = 1 .. 7) or along axis k - 1 (k = 1 .. 3).
// body(slot, here): every other particle of them in that order; here tells
// whether the pair is evaluated in this particle's cell (or, within the cell,
// at this particle, the earlier one) rather than the other's.
//
// Bound by latency: a particle's neighbours are few, and in up to 15 lists.  All
// list bounds are loaded at once, the lists that are not empty put down in
// shared memory, and their particles visited in one loop -- a warp runs as long
// as its longest particle, not the sum of its longest lists -- that loads the
// next one's values before it uses this one's.  Slots ascend with the particles'
// indices within a cell, so the order of two particles of a cell is that of
// their slots.  kLanes neighbouring lanes take a particle's lists in turn; the
// caller adds their sums (sum_lanes).  k_pse, 10^6 vortons at 225 x 161 x 193: 177 -> 118 us, 262,144 at
// 129^3: 57 -> 36 us, 32 sets of 32,768: 65 -> 26 us each.
//
// In dense cells a warp's particles have the same lists, and finding the next one's place costs more than the longest
// list does.  Warps with kDense particles a list or more on average (one lane to a particle) go list by list, the own
// cell's apart because the particle itself is in it, four particles' loads at a time.  Whole calls, us, a loop to every
// list as before / one loop / this: 600,000 vortons on 33^3 points (17 a cell) 444 / 493 / 362, 400,000 on 49 x 33 x 41
// (6) 214 / 185 / 162, 1.5 million on 17^3 (305) 12,022 / 16,956 / 10,066; below kDense the same as one loop.  By a line
// of their own, without the warp, particles near it took both loops: up to 30 % more.
constexpr int kPseThreads = 128;
constexpr unsigned kDense = 5;
template <bool kAll, int kLanes, typename Load, typename Body>
__device__ __forceinline__ void for_neighbours(int nx, int ny, int nz, int cx, int cy, int cz, unsigned t,
                                               const unsigned* __restrict__ start, const Load& load,
                                               const Body& body) {
  constexpr int kSide = kAll ? 8 : 4, kLists = 2 * kSide - 1, kMine = (kLists + kLanes - 1) / kLanes;
  __shared__ uint2 lists[kMine][kPseThreads];
  uint2 range[kMine];
#pragma unroll
  for (int q = 0; q < kMine; ++q) {
    const int r = q * kLanes + (int)(threadIdx.x % kLanes);
    const int s = r < kSide ? -1 : 1, k = r < kSide ? r : r - kSide + 1;
    const int ox = s * (kAll ? (k & 1) : (k == 1)), oy = s * (kAll ? ((k >> 1) & 1) : (k == 2));
    const int oz = s * (kAll ? ((k >> 2) & 1) : (k == 3));
    const int ncx = cx + ox, ncy = cy + oy, ncz = cz + oz;
    // the lower of the two cells has to be one that the reference's loop visits
    const int lx = s == 1 ? cx : ncx, ly = s == 1 ? cy : ncy, lz = s == 1 ? cz : ncz;
    range[q] = make_uint2(0, 0);
    if (r < kLists && ncx >= 0 && ncy >= 0 && ncz >= 0 && ncx < nx && ncy < ny && ncz < nz && lx < nx - 1 &&
        ly < ny - 1 && lz < nz - 1) {
      const size_t cell = (size_t)ncx + (size_t)nx * ((size_t)ncy + (size_t)ny * ncz);
      range[q] = make_uint2(start[cell], start[cell + 1]);
    }
  }
  int cnt = 0, own = 0, lower = 0;  // lists kept, and of them the own cell's, and those up to the lower side's
  unsigned total = 0;               // particles in them
#pragma unroll
  for (int q = 0; q < kMine; ++q) {
    const int r = q * kLanes + (int)(threadIdx.x % kLanes);
    if (range[q].x < range[q].y) lists[cnt++][threadIdx.x] = range[q];
    total += range[q].y - range[q].x;
    if (r == 0) own = cnt;
    if (r < kSide) lower = cnt;
  }
  // the warp's lanes that are here: one loop for all of them
  const unsigned active = __activemask();
  const bool dense = kLanes == 1 && __reduce_add_sync(active, min(total, 1u << 20)) >= kDense * kLists * __popc(active);
  if (cnt == 0) return;
  if (dense) {
    for (int r = 0; r < cnt; ++r) {
      const uint2 list = lists[r][threadIdx.x];
      if (r < own) {
        for (unsigned slot = list.x; slot < list.y; ++slot)
          if (slot != t) body(load(slot), t < slot);
      } else {
        const bool here = r >= lower;
#pragma unroll 4
        for (unsigned slot = list.x; slot < list.y; ++slot) body(load(slot), here);
      }
    }
    return;
  }
  int r = 0;
  uint2 at = lists[0][threadIdx.x];
  auto value = load(at.x);
  for (;;) {
    const unsigned slot = at.x;
    const bool here = r < own ? t < slot : r >= lower;
    const auto cur = value;
    bool more = true;
    if (++at.x == at.y) {
      more = ++r < cnt;
      if (more) at = lists[r][threadIdx.x];
    }
    if (more) value = load(at.x);
    if (slot != t) body(cur, here);
    if (!more) break;
  }
}

// A particle's sum over its lanes, for all of them.
template <int kLanes>
__device__ __forceinline__ float sum_lanes(float v) {
  const unsigned mask = ((1u << kLanes) - 1u) << (threadIdx.x % 32 / kLanes * kLanes);
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) v += __shfl_xor_sync(mask, v, o);
  return v;
}

// Four lanes to a particle where the particles alone do not fill the chip: 3,001
// vortons 18.2 us with one lane, 7.6 with four; 32,000 in a puff 114 and 48; 32
// sets of 1,000 to 65,536 at a time 25 and 12 each; but 262,144 36.2 and 38.5 (heat
// 19.0 and 22.9).
int pse_lanes(size_t n) { return n < 131072 ? 4 : 1; }

template <int kLanes>
__global__ void __launch_bounds__(kPseThreads) k_pse(Geom g, const float4* __restrict__ pss, const float4* __restrict__ w0s,
                                             float4* __restrict__ w, int n, const unsigned* __restrict__ start,
                                             const unsigned* __restrict__ items, float nu, float dt) {
  pdl_entry();
  // threads take the vortons in cell order, so a warp's vortons share their
  // neighbour cells and read them contiguously (each vorton's sums are the
  // same whichever thread runs them)
  const int t = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  if (t >= n) return;
  const int i = (int)items[t];
  const float4 p = pss[t];
  const float4 wi = w0s[t];
  const int nx = (int)g.np[0], ny = (int)g.np[1], nz = (int)g.np[2];
  // cell coordinates clamped to [-2, n + 1]: beyond that every neighbour test
  // below fails the same way, and ncx = cx + ox cannot overflow
  const int cx = min(max(__float2int_rz(__fmul_rn(__fsub_rn(p.x, g.mn[0]), g.cpe[0])), -2), nx + 1);
  const int cy = min(max(__float2int_rz(__fmul_rn(__fsub_rn(p.y, g.mn[1]), g.cpe[1])), -2), ny + 1);
  const int cz = min(max(__float2int_rz(__fmul_rn(__fsub_rn(p.z, g.mn[2]), g.cpe[2])), -2), nz + 1);
  if (cx < 0 || cy < 0 || cz < 0 || cx >= nx || cy >= ny || cz >= nz) {
    w[i] = wi;  // outside the grid's points: in no cell list, so no exchange
    return;
  }
  const bool here_ok = cx >= 0 && cy >= 0 && cz >= 0 && cx < nx - 1 && cy < ny - 1 && cz < nz - 1;
  const float twonudt = 2.0f * nu * dt;
  float ax = 0.f, ay = 0.f, az = 0.f;
  struct Neighbour {
    float4 p, w;
  };
  for_neighbours<true, kLanes>(
      nx, ny, nz, cx, cy, cz, (unsigned)t, start, [&](unsigned slot) { return Neighbour{pss[slot], w0s[slot]}; },
      [&](const Neighbour& v, bool here) {
        const float range = 4.0f * (here ? p.w : v.p.w);
        const float dx = p.x - v.p.x, dy = p.y - v.p.y, dz = p.z - v.p.z;
        const float dist2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const float law = __expf(-dist2 / (range * range));
        const float frac = fminf(fmaxf(twonudt * law, -0.5f), 0.5f);
        ax = fmaf(frac, v.w.x - wi.x, ax);
        ay = fmaf(frac, v.w.y - wi.y, ay);
        az = fmaf(frac, v.w.z - wi.z, az);
      });
  ax = sum_lanes<kLanes>(ax);
  ay = sum_lanes<kLanes>(ay);
  az = sum_lanes<kLanes>(az);
  if (threadIdx.x % kLanes) return;
  float vx = wi.x + ax, vy = wi.y + ay, vz = wi.z + az;
  if (here_ok) {
    const float f = nu * dt;
    vx -= f * vx;
    vy -= f * vy;
    vz -= f * vz;
  }
  w[i] = make_float4(vx, vy, vz, wi.w);
}

// DiffuseAndDissipateHeatPSE (vortonSim.cpp:3880-4093) in the order-independent
// form of k_pse: vorton i (threads in cell order, reading cell-sorted copies)
// exchanges density with every vorton of its own cell and of the face
// neighbours along +-x, +-y, +-z that the reference pairs it with (the pair's
// "here" cell strictly inside the point range; the range 4 x the "here"
// vorton's size), using the densities from before the step, then relaxes
// toward the ambient density when its own cell is a "here" cell.
__global__ void k_heat_gather(const float4* __restrict__ ps, const float* __restrict__ d, int n,
                              const unsigned* __restrict__ items, float4* __restrict__ pss, float* __restrict__ d0s) {
  pdl_entry();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const unsigned j = items[t];
  pss[t] = ps[j];
  d0s[t] = d[j];
}

template <int kLanes>
__global__ void __launch_bounds__(kPseThreads) k_heat_pse(Geom g, const float4* __restrict__ pss, const float* __restrict__ d0s,
                                                  float* __restrict__ d, int n, const unsigned* __restrict__ start,
                                                  const unsigned* __restrict__ items, float kappa, float ambient,
                                                  float dt) {
  pdl_entry();
  const int t = (int)(((size_t)blockIdx.x * blockDim.x + threadIdx.x) / kLanes);
  if (t >= n) return;
  const int i = (int)items[t];
  const float4 p = pss[t];
  const float di = d0s[t];
  const int nx = (int)g.np[0], ny = (int)g.np[1], nz = (int)g.np[2];
  const int cx = min(max(__float2int_rz(__fmul_rn(__fsub_rn(p.x, g.mn[0]), g.cpe[0])), -2), nx + 1);
  const int cy = min(max(__float2int_rz(__fmul_rn(__fsub_rn(p.y, g.mn[1]), g.cpe[1])), -2), ny + 1);
  const int cz = min(max(__float2int_rz(__fmul_rn(__fsub_rn(p.z, g.mn[2]), g.cpe[2])), -2), nz + 1);
  if (cx < 0 || cy < 0 || cz < 0 || cx >= nx || cy >= ny || cz >= nz) {
    d[i] = di;  // in no cell list: no exchange
    return;
  }
  const bool here_ok = cx < nx - 1 && cy < ny - 1 && cz < nz - 1;
  const float twokdt = 2.0f * kappa * dt;
  float acc = 0.f;
  struct Neighbour {
    float4 p;
    float d;
  };
  for_neighbours<false, kLanes>(
      nx, ny, nz, cx, cy, cz, (unsigned)t, start, [&](unsigned slot) { return Neighbour{pss[slot], d0s[slot]}; },
      [&](const Neighbour& v, bool here) {
        const float range = 4.0f * (here ? p.w : v.p.w);
        const float dx = p.x - v.p.x, dy = p.y - v.p.y, dz = p.z - v.p.z;
        const float dist2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        const float law = __expf(-dist2 / (range * range));
        const float ratio = fminf(fmaxf(twokdt * law, -0.5f), 0.5f);
        acc = fmaf(ratio, v.d - di, acc);
      });
  acc = sum_lanes<kLanes>(acc);
  if (threadIdx.x % kLanes) return;
  float v = di + acc;
  if (here_ok) v += fminf(fmaxf(kappa * dt, -0.5f), 0.5f) * (ambient - v);
  d[i] = v;
}

// order (optional): the particles grouped by cell, as in k_stretch.
__global__ void k_gather_advect(Geom g, const float* __restrict__ vel3, float4* __restrict__ pos,
                                float4* __restrict__ vel, int m, float dt, int evolve,
                                const unsigned* __restrict__ order, int* __restrict__ flag) {
  pdl_entry();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= m) return;
  const int i = order ? (int)order[t] : t;
  float4 p = pos[i];
  if (!inside_cells(g, p.x, p.y, p.z)) {
    atomicOr(flag, (int)DF_OUT_OF_GRID);
    if (vel) vel[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  float u[3];
  interp<3>(g, vel3, p.x, p.y, p.z, u);
  if (vel) vel[i] = make_float4(u[0], u[1], u[2], 0.f);
  if (evolve) {
    p.x = __fadd_rn(p.x, __fmul_rn(u[0], dt));
    p.y = __fadd_rn(p.y, __fmul_rn(u[1], dt));
    p.z = __fadd_rn(p.z, __fmul_rn(u[2], dt));
    pos[i] = p;
  }
}

// AssignParticleVelocityFromField (gain 1) + EvolveParticlesSlice on staged
// particle records (position at bytes 0-11, velocity at 12-23, pitch bytes
// apart), in place: k_gather_advect without copying positions and velocities
// out of and back into the records.  A record outside the grid's cells keeps
// its position and gets zero velocity, as on the copy path.
__global__ void k_gather_advect_records(Geom g, const float* __restrict__ vel3, unsigned char* __restrict__ rec,
                                        size_t pitch, int m, float dt, int* __restrict__ flag) {
  pdl_entry();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= m) return;
  float* r = (float*)(rec + (size_t)i * pitch);
  const float px = r[0], py = r[1], pz = r[2];
  if (!inside_cells(g, px, py, pz)) {
    atomicOr(flag, (int)DF_OUT_OF_GRID);
    r[3] = 0.f;
    r[4] = 0.f;
    r[5] = 0.f;
    return;
  }
  float u[3];
  interp<3>(g, vel3, px, py, pz, u);
  r[0] = __fadd_rn(px, __fmul_rn(u[0], dt));
  r[1] = __fadd_rn(py, __fmul_rn(u[1], dt));
  r[2] = __fadd_rn(pz, __fmul_rn(u[2], dt));
  r[3] = u[0];
  r[4] = u[1];
  r[5] = u[2];
}

// The velocity grid as float4 points, for k_gather_advect_points.
__global__ void k_vel_points(size_t pts, const float* __restrict__ v3, float4* __restrict__ vp) {
  pdl_entry();
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k < pts) vp[k] = make_float4(v3[3 * k], v3[3 * k + 1], v3[3 * k + 2], 0.f);
}

// k_gather_advect reading the float4 points: the same cell, weights and sums bit
// for bit.  Eight lanes take the corners of a tracer, lane q corner q (x in bit
// 0, y in bit 1, z in bit 2), for the eight tracers of those lanes in turn; the
// sums along x, y and z are then exchanges between lanes 1, 2 and 4 apart, each
// of which halves the number of tracers a lane holds, so that lane q ends with
// its own tracer's.
//
// Bound by the first-level cache's lines a cycle: a tracer's corners lie in
// four rows, and one load of eight lanes takes each row's line once, where a
// thread that loads its tracer's corners itself takes one for every corner.
// 2^22 tracers on 129^3 points: 99 us, and 7 us for the float4 points, against
// 228 us from the three-float grid (a thread to a tracer, 24 loads) and 136 us + 84 us
// from a copy of the grid with each cell's corners in a line of their own.
//
// Neighbouring tracers in one line's cells need none of that: a warp in which fewer
// than kFewLines lanes change the line loads by thread (tracers in the order of
// their cells 63 us, all eight lanes 107; in one cell 49 and 90, from the
// three-float grid 46).  Six blocks an SM: 40 registers, 48 else (69 and 56 us).
constexpr int kFewLines = 16;
__global__ void __launch_bounds__(256, 6) k_gather_advect_points(Geom g, const float4* __restrict__ vp,
                                                                 float4* __restrict__ pos, float4* __restrict__ vel,
                                                                 int m, float dt, int evolve, int* __restrict__ flag) {
  pdl_entry();
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool valid = i < (unsigned)m;  // all lanes take part in the exchanges
  float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
  if (valid) p = pos[i];
  const bool inside = valid && inside_cells(g, p.x, p.y, p.z);
  const float pp[3] = {p.x, p.y, p.z};
  unsigned idx[3] = {0, 0, 0};  // a lane without a tracer in the grid reads the first cell
  float tw[3] = {0.f, 0.f, 0.f};
  if (inside)
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      idx[a] = bin_axis(pp[a], g.mn[a], g.cpe[a]);
      const float cmin = __fadd_rn(g.mn[a], __fmul_rn((float)idx[a], g.cell[a]));
      tw[a] = __fmul_rn(__fsub_rn(pp[a], cmin), g.cpe[a]);
    }
  const unsigned nx = g.np[0], nxy = g.np[0] * g.np[1];
  const unsigned base = idx[0] + nx * idx[1] + nxy * idx[2];
  const int lane = threadIdx.x & 31, q = lane & 7, group = lane & 24;
  const unsigned bx = q & 1, by = (q >> 1) & 1, bz = q >> 2;
  const unsigned corner = bx + nx * by + nxy * bz;
  float4 c[8], u;
  // lanes whose tracer's cell lies in another line than the lane's before it; 8 points of a row to a line
  const unsigned before = __shfl_up_sync(0xffffffffu, base, 1);
  if (__popc(__ballot_sync(0xffffffffu, base >> 3 != before >> 3)) < kFewLines) {
    if (!valid) return;
#pragma unroll
    for (unsigned k = 0; k < 8; ++k) c[k] = vp[base + (k & 1) + nx * ((k >> 1) & 1) + nxy * (k >> 2)];
    auto mix = [](float4 a, float4 b, float t) {  // (1 - t) a + t b
      const float s = __fsub_rn(1.0f, t);
      return make_float4(__fadd_rn(__fmul_rn(s, a.x), __fmul_rn(t, b.x)), __fadd_rn(__fmul_rn(s, a.y), __fmul_rn(t, b.y)),
                         __fadd_rn(__fmul_rn(s, a.z), __fmul_rn(t, b.z)), 0.f);
    };
    u = mix(mix(mix(c[0], c[1], tw[0]), mix(c[2], c[3], tw[0]), tw[1]),
            mix(mix(c[4], c[5], tw[0]), mix(c[6], c[7], tw[0]), tw[1]), tw[2]);
  } else {
#pragma unroll
    for (int r = 0; r < 8; ++r) c[r] = vp[__shfl_sync(0xffffffffu, base, group + r) + corner];
    auto weight = [&](float t, unsigned bit, int from) {  // 1 - t or t of the tracer of lane `from`
      const float w = __shfl_sync(0xffffffffu, t, from);
      return bit ? w : __fsub_rn(1.0f, w);
    };
    auto times = [](float4 v, float w) {
      return make_float4(__fmul_rn(v.x, w), __fmul_rn(v.y, w), __fmul_rn(v.z, w), 0.f);
    };
    // keeps one of two tracers' terms, by the lane's bit, and adds the partner's term of the same tracer
    auto exchange = [](float4 t0, float4 t1, unsigned bit, int apart) {
      const float4 keep = bit ? t1 : t0, give = bit ? t0 : t1;
      return make_float4(__fadd_rn(keep.x, __shfl_xor_sync(0xffffffffu, give.x, apart)),
                         __fadd_rn(keep.y, __shfl_xor_sync(0xffffffffu, give.y, apart)),
                         __fadd_rn(keep.z, __shfl_xor_sync(0xffffffffu, give.z, apart)), 0.f);
    };
    float4 sx[4], sy[2];
#pragma unroll
    for (int r = 0; r < 4; ++r)
      sx[r] = exchange(times(c[2 * r], weight(tw[0], bx, group + 2 * r)),
                       times(c[2 * r + 1], weight(tw[0], bx, group + 2 * r + 1)), bx, 1);
#pragma unroll
    for (int r = 0; r < 2; ++r)
      sy[r] = exchange(times(sx[2 * r], weight(tw[1], by, group + 4 * r + bx)),
                       times(sx[2 * r + 1], weight(tw[1], by, group + 4 * r + 2 + bx)), by, 2);
    u = exchange(times(sy[0], weight(tw[2], bz, group + 2 * by + bx)),
                 times(sy[1], weight(tw[2], bz, group + 4 + 2 * by + bx)), bz, 4);
    if (!valid) return;
  }
  if (!inside) {
    atomicOr(flag, (int)DF_OUT_OF_GRID);
    if (vel) vel[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    return;
  }
  if (vel) vel[i] = make_float4(u.x, u.y, u.z, 0.f);
  if (evolve) {
    p.x = __fadd_rn(p.x, __fmul_rn(u.x, dt));
    p.y = __fadd_rn(p.y, __fmul_rn(u.y, dt));
    p.z = __fadd_rn(p.z, __fmul_rn(u.z, dt));
    pos[i] = p;
  }
}

// Order-preserving float <-> uint map, for the warp's integer reductions.
__device__ __forceinline__ unsigned f2key(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// Each block's extremes to part[6 block]; k_bbox_finish takes them together.
// (Atomics by every warp to the same six words, with a kernel to set them first,
// took 19 us for 65,536 particles; these two kernels take 3.9.)
constexpr int kBoxThreads = 256;
__global__ void __launch_bounds__(kBoxThreads) k_bbox(const float4* __restrict__ pos, int n,
                                                      unsigned* __restrict__ part, int* __restrict__ flag) {
  pdl_entry();
  __shared__ unsigned sh[kBoxThreads / 32][6];
  float mn[3] = {FLT_MAX, FLT_MAX, FLT_MAX}, mx[3] = {-FLT_MAX, -FLT_MAX, -FLT_MAX};
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < (unsigned)n; i += gridDim.x * blockDim.x) {
    const float4 p = pos[i];
    if (!(isfinite(p.x) && isfinite(p.y) && isfinite(p.z))) atomicOr(flag, (int)DF_NONFINITE);
    mn[0] = fminf(mn[0], p.x); mn[1] = fminf(mn[1], p.y); mn[2] = fminf(mn[2], p.z);
    mx[0] = fmaxf(mx[0], p.x); mx[1] = fmaxf(mx[1], p.y); mx[2] = fmaxf(mx[2], p.z);
  }
  const int lane = threadIdx.x & 31, wid = threadIdx.x / 32;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
    const unsigned lo = __reduce_min_sync(0xffffffffu, f2key(mn[a])), hi = __reduce_max_sync(0xffffffffu, f2key(mx[a]));
    if (lane == 0) sh[wid][a] = lo, sh[wid][3 + a] = hi;
  }
  __syncthreads();
  if (threadIdx.x < 6) {
    unsigned k = sh[0][threadIdx.x];
    for (int w = 1; w < kBoxThreads / 32; ++w)
      k = threadIdx.x < 3 ? min(k, sh[w][threadIdx.x]) : max(k, sh[w][threadIdx.x]);
    part[6 * blockIdx.x + threadIdx.x] = k;
  }
}

// One warp for each of the six extremes.
__global__ void __launch_bounds__(192) k_bbox_finish(const unsigned* __restrict__ part, int nb, float* __restrict__ out6) {
  pdl_entry();
  const int a = threadIdx.x / 32, lane = threadIdx.x & 31;
  unsigned k = a < 3 ? 0xffffffffu : 0u;
  for (int b = lane; b < nb; b += 32) k = a < 3 ? min(k, part[6 * b + a]) : max(k, part[6 * b + a]);
  k = a < 3 ? __reduce_min_sync(0xffffffffu, k) : __reduce_max_sync(0xffffffffu, k);
  if (lane == 0) out6[a] = __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

}  // namespace

static void recip_spacing(const Geom& g, float rs[3]) {
  // reciprocalSpacing (uniformGridMath.cpp:1124, 317)
  rs[0] = 1.0f / g.cell[0];
  rs[1] = 1.0f / g.cell[1];
  rs[2] = g.cell[2] > FLT_EPSILON ? 1.0f / g.cell[2] : 0.0f;
}

vg_status launch_sor(Ctx* c, const Geom& g, float* s, const float* lap, int steps) {
  if (g.np[0] < 3 || g.np[1] < 3 || g.np[2] < 3 || steps <= 0) return VG_OK;
  float rs[3];
  recip_spacing(g, rs);
  volatile float r2x = rs[0] * rs[0], r2y = rs[1] * rs[1], r2z = rs[2] * rs[2];
  volatile float sum = r2x + r2y;
  sum = sum + r2z;
  const float H = 0.5f / sum;
  const unsigned rows_per_z = (g.np[1] - 2 + 1) / 2 + 1;
  const size_t threads = (size_t)rows_per_z * (g.np[2] - 2);
  for (int it = 0; it < steps; ++it)
    for (unsigned color = 0; color < 2; ++color) {
      pdl_launch(c->stream, blocks_for(threads, 64), 64, 0, k_sor_rows, g, s, lap, color, r2x, r2y, r2z, H);
      VG_LAUNCHED(c);
    }
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_downsample(Ctx* c, const Geom& F, const float* f3, const Geom& C, bool inject, float* c3) {
  const uint3 cd = make_uint3((F.np[0] - 1) / (C.np[0] - 1), (F.np[1] - 1) / (C.np[1] - 1), (F.np[2] - 1) / (C.np[2] - 1));
  pdl_launch(c->stream, blocks_for(C.points(), 128), 128, 0, k_downsample, F, f3, C, cd, inject ? 1 : 0, c3);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_upsample(Ctx* c, const Geom& C, const float* c3, const Geom& F, bool interior, float* f3) {
  pdl_launch(c->stream, blocks_for(F.points(), 128), 128, 0, k_upsample, C, c3, F, interior ? 1 : 0, f3);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status run_cascade(Ctx* c, const Geom& g, float* soln3, const float* rhs3, int steps) {
  Geom L[kMaxLayers];
  unsigned dec[kMaxLayers][3];
  const int depth = nested_shape(g, L, dec);
  size_t total = 0, base[kMaxLayers];
  for (int l = 0; l < depth; ++l) {
    base[l] = total;
    total += L[l].points();
  }
  vg_status st = VG_OK;
  float* mem = (float*)ws(c, S_MG, 2 * total * 3 * sizeof(float), &st);
  if (st != VG_OK) return st;
  float* a[kMaxLayers];
  float* b[kMaxLayers];
  for (int l = 0; l < depth; ++l) {
    a[l] = mem + 3 * base[l];
    b[l] = mem + 3 * (total + base[l]);
  }
  a[0] = soln3;
  b[0] = const_cast<float*>(rhs3);
  if ((st = launch_sor(c, L[0], a[0], b[0], steps)) != VG_OK) return st;
  int max_valid = 0;
  for (int l = 1; l < depth; ++l) {
    unsigned mind = L[l].np[0] < L[l].np[1] ? L[l].np[0] : L[l].np[1];
    if (L[l].np[2] < mind) mind = L[l].np[2];
    if (mind > 2) {
      if ((st = launch_downsample(c, L[l - 1], b[l - 1], L[l], true, b[l])) != VG_OK) return st;
      if ((st = launch_downsample(c, L[l - 1], a[l - 1], L[l], true, a[l])) != VG_OK) return st;
      if ((st = launch_sor(c, L[l], a[l], b[l], steps)) != VG_OK) return st;
    } else {
      max_valid = l - 1;
      break;
    }
  }
  for (int l = max_valid; l >= 1; --l) {
    if ((st = launch_upsample(c, L[l], a[l], L[l - 1], true, a[l - 1])) != VG_OK) return st;
    if ((st = launch_sor(c, L[l - 1], a[l - 1], b[l - 1], steps)) != VG_OK) return st;
  }
  return VG_OK;
}

vg_status launch_jacobian(Ctx* c, const Geom& g, const float* v3, float* jac9) {
  float rs[3];
  recip_spacing(g, rs);
  pdl_launch(c->stream, blocks_for(g.points(), 128), 128, 0, k_jacobian, g, rs[0], rs[1], rs[2], v3, jac9);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_curl(Ctx* c, const Geom& g, const float* v3, float* curl3) {
  float rs[3];
  recip_spacing(g, rs);
  pdl_launch(c->stream, blocks_for(g.points(), 128), 128, 0, k_curl, g, rs[0], rs[1], rs[2], v3, curl3);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_stretch_vel(Ctx* c, const Geom& g, const float* v3, const float4* ps, float4* w, size_t n, float dt,
                             const unsigned* order) {
  if (0.0f == g.ext[0] || 0.0f == g.ext[1] || 0.0f == g.ext[2]) return VG_OK;  // 2D: no stretching
  if (n == 0) return VG_OK;
  float rs[3];
  recip_spacing(g, rs);
  pdl_launch(c->stream, blocks_for(n, 128), 128, 0, k_stretch_vel, g, rs[0], rs[1], rs[2], v3, ps, w, (int)n, dt, order,
             outside_flag(c));
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_stretch(Ctx* c, const Geom& g, const float* jac9, const float4* ps, float4* w, size_t n, float dt,
                         const unsigned* order) {
  if (0.0f == g.ext[0] || 0.0f == g.ext[1] || 0.0f == g.ext[2]) return VG_OK;  // 2D: no stretching
  if (n == 0) return VG_OK;
  pdl_launch(c->stream, blocks_for(n, 128), 128, 0, k_stretch, g, jac9, ps, w, (int)n, dt, order, outside_flag(c));
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_heat_pse(Ctx* c, const Geom& g, const CellLists& cl, const float4* ps, float* density, size_t n,
                          float kappa, float ambient, float dt) {
  vg_status st = VG_OK;
  char* tmp = (char*)ws(c, S_WOLD, n * (sizeof(float4) + sizeof(float)), &st);
  if (st != VG_OK) return st;
  float4* pss = (float4*)tmp;
  float* d0s = (float*)(pss + n);
  pdl_launch(c->stream, blocks_for(n, 256), 256, 0, k_heat_gather, ps, density, (int)n, cl.items, pss, d0s);
  const int lanes = pse_lanes(n);
  pdl_launch(c->stream, blocks_for(lanes * n, kPseThreads), kPseThreads, 0, lanes == 4 ? k_heat_pse<4> : k_heat_pse<1>,
             g, pss, d0s, density, (int)n, cl.start, cl.items, kappa, ambient, dt);
  c->launches += 2;
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_pse(Ctx* c, const Geom& g, const CellLists& cl, const float4* ps, float4* w, size_t n, float nu,
                     float dt) {
  if (n == 0) return VG_OK;
  vg_status st = VG_OK;
  float4* pss = (float4*)ws(c, S_WOLD, 2 * n * sizeof(float4), &st);
  if (st != VG_OK) return st;
  float4* w0s = pss + n;
  pdl_launch(c->stream, blocks_for(n, 256), 256, 0, k_pse_gather, ps, w, (int)n, cl.items, pss, w0s);
  const int lanes = pse_lanes(n);
  pdl_launch(c->stream, blocks_for(lanes * n, kPseThreads), kPseThreads, 0, lanes == 4 ? k_pse<4> : k_pse<1>, g, pss, w0s,
             w, (int)n, cl.start, cl.items, nu, dt);
  c->launches += 2;
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

// Staged records are taken apart into float4 positions and velocities, and put
// together again, for two tracers or more per cell of a grid of 2^17 cells.
bool unpack_records(const Geom& g, size_t m) {
  if (g.np[0] < 2 || g.np[1] < 2 || g.np[2] < 2) return false;
  const size_t cells = (size_t)(g.np[0] - 1) * (g.np[1] - 1) * (size_t)(g.np[2] - 1);
  return cells >= ((size_t)1 << 17) && m >= 2 * cells;
}

// Tracers of the step's own grid gather from its float4 points where the copy
// (made once per step) pays: it costs 4 ns per 1000 points, and saves 25 to
// 35 ns per 1000 tracers in no order.  2^18 tracers, copy included, against the three-float
// grid: 9.3 against 10.7 us on 33^3 points, 10.2 against 15.6 on 65^3, 16.2
// against 16.8 on 129^3 (eight points to a tracer); 2^20 tracers on 193^3
// points (seven to a tracer) 62.5 against 64.1.  Tracers in the order of their
// cells gain nothing from it and pay the copy (10^6 on 129^3 24 us and 7).
static bool gather_points(const Geom& g, size_t m) {
  const size_t pts = g.points();
  return g.np[0] >= 2 && g.np[1] >= 2 && g.np[2] >= 2 && pts < ((size_t)1 << 31) && m >= ((size_t)1 << 18) &&
         6 * m >= pts;
}

vg_status launch_gather_advect_records(Ctx* c, const Geom& g, const float* vel3, unsigned char* rec, size_t pitch,
                                       size_t m, float dt) {
  if (m == 0) return VG_OK;
  if (m > 0x7fffffff) return fail(c, VG_TOO_LARGE, "advect: more than 2^31 particles");
  pdl_launch(c->stream, blocks_for(m, 256), 256, 0, k_gather_advect_records, g, vel3, rec, pitch, (int)m, dt,
             outside_flag(c));
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_gather_advect(Ctx* c, const Geom& g, const float* vel3, float4* pos, float4* vel, size_t m, float dt,
                               bool evolve, const unsigned* order, bool step_grid) {
  if (m == 0) return VG_OK;
  if (m > 0x7fffffff) return fail(c, VG_TOO_LARGE, "advect: more than 2^31 particles");
  // (inside a graph capture the copy is always made, so that every replay
  // remakes it from that replay's grid)
  if (step_grid && !order && gather_points(g, m)) {
    vg_status st = VG_OK;
    float4* vp = (float4*)ws(c, S_VELPOINTS, g.points() * sizeof(float4), &st);
    if (st != VG_OK) return st;
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    VG_CUDA(c, cudaStreamIsCapturing(c->stream, &cap));
    if (cap != cudaStreamCaptureStatusNone || c->vel_uncounted || c->velpoints_gen != c->vel_gen) {
      pdl_launch(c->stream, blocks_for(g.points(), 256), 256, 0, k_vel_points, g.points(), vel3, vp);
      VG_LAUNCHED(c);
      c->velpoints_gen = cap != cudaStreamCaptureStatusNone ? ~0ull : c->vel_gen;
    }
    pdl_launch(c->stream, blocks_for(m, 256), 256, 0, k_gather_advect_points, g, (const float4*)vp, pos, vel, (int)m,
               dt, evolve ? 1 : 0, outside_flag(c));
    VG_LAUNCHED(c);
    VG_CUDA(c, cudaGetLastError());
    return VG_OK;
  }
  pdl_launch(c->stream, blocks_for(m, 256), 256, 0, k_gather_advect, g, vel3, pos, vel, (int)m, dt, evolve ? 1 : 0, order,
                                                              outside_flag(c));
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

vg_status launch_bbox(Ctx* c, const float4* pos, size_t n, float* out6) {
  vg_status st = VG_OK;
  const unsigned most = 2u * (unsigned)sm_count();
  unsigned blocks = n > 0 ? blocks_for(n, kBoxThreads) : 0;
  if (blocks > most) blocks = most;
  unsigned* part = (unsigned*)ws(c, S_BBOX, 6 * most * sizeof(unsigned), &st);
  if (st != VG_OK) return st;
  if (blocks) {
    pdl_launch(c->stream, blocks, kBoxThreads, 0, k_bbox, pos, (int)n, part, c->dflag);
    VG_LAUNCHED(c);
  }
  pdl_launch(c->stream, 1, 192, 0, k_bbox_finish, (const unsigned*)part, (int)blocks, out6);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

}  // namespace vg
