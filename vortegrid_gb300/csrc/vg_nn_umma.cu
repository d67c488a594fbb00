// 3x3x3 convolution on the 5th-generation tensor cores (tcgen05, sm_103a).
//
// Implicit GEMM: M = 128 output voxels (a tile of 8 x 16 voxels in x, y at one z), K = 27 taps x 16-channel slices.  A slab
// (one z plane of the tile's zero-padded halo, 10 x 18 voxels, 16 channels) is stored "chunk-planar": channels 0..7 of
// every voxel, 16 bytes each, then channels 8..15.  In that layout the A operand of any tap is a K-major, no-swizzle
// shared-memory matrix: 8 consecutive voxels of one x row form a core matrix (8 rows x 16 bytes, contiguous), successive y
// rows are 10 voxels (160 bytes) apart (the stride between 8-row groups) and the second 8 channels are one plane further
// (the stride between K-adjacent core matrices), so each tap reads the halo in place.
//
// The three z taps share one MMA: a slab at z feeds the output planes z - 1, z and z + 1, whose accumulators are
// neighbouring columns of tensor memory, so for every (dy, dx) one tcgen05.mma of N = 3 CO_T takes the slab's 4 KB window
// for all three.  What bounds these layers is that window's way through shared memory, about 60 cycles an MMA however small
// N is: 9 MMAs a slab and tile instead of 27, and every slab is copied once instead of three times.
//
// A CTA marches an item (a tile x up to 256 / CO_T planes, all accumulators in 256 columns) slice by slice, plane by plane,
// so that the products of an output are added in the order slice, z tap, y tap, x tap.  Its output planes are drained while
// the next ones are summed; two CTAs share an SM and hide each other's waits.  The weights of the CTA's output-channel
// group stay in shared memory.
//
// Measured on GB300, us a launch, against one MMA of N = CO_T per tap with three halo planes copied for every output plane
// (and mma.sync for 128 and more input channels); the results are the same bit for bit:
//   16 -> 16 on 128^3   141 -> 55..72     48 -> 16 on 128^3   430 -> 107     16 -> 48 on 128^3   190 -> 102
//   32 -> 32 on  64^3    51 -> 26         96 -> 32 on  64^3   339 -> 63
//   64 -> 64 on  32^3    44 -> 20        192 -> 64 on  32^3   147 -> 49     128 -> 128 on 16^3   65 -> 17
//
// Warps: 0..3 epilogue, 4..7 copy the slabs (cp.async into a ring; the first input may be read through a nearest 2x
// upsampling, so that neither the upsampled nor the concatenated tensor exists in memory), 8 issues the MMAs.  Every wait
// is bounded: one that runs out (2 s) sets an abort word that ends all later waits at once; the roles then run through
// their work without waiting (every access stays in its buffers), the kernel raises DF_TIMEOUT and frees its tensor memory.
#include <algorithm>

#include "vg_nn.cuh"

namespace vg {
namespace nn {

namespace {

constexpr int kTX = 8, kTY = 16;                 // tile: 8 x 16 voxels = M 128
constexpr int kHX = kTX + 2, kHY = kTY + 2;       // halo 10 x 18
constexpr int kChunks = kHX * kHY * 2;            // 16-byte chunks of a slab
constexpr unsigned kXPlane = kHX * kHY * 16;      // bytes of 8 channels of a slab
constexpr unsigned kSlab = 2 * kXPlane;
constexpr int kEpiWarps = 4, kCopyWarps = 4, kCopyThreads = kCopyWarps * 32;
constexpr int kMmaWarp = kEpiWarps + kCopyWarps, kThreads = (kMmaWarp + 1) * 32;
constexpr int kMaxSlabs = 8, kMinSlabs = 4;       // slabs in the ring
constexpr int kCols = 256;                        // tensor-memory columns of a CTA
constexpr int kMaxPlanes = 16;
constexpr size_t kSmemTwo = 113 * 1024, kSmemOne = 226 * 1024;  // shared memory of a CTA at two and at one per SM
constexpr size_t kTail = (2 * kMaxSlabs + 2 * kMaxPlanes) * 8 + 64;

// No-swizzle K-major descriptors: the low word holds the address and the distance of the second 8 channels, the high word
// the distance of 8-row groups (and the descriptor version).
__device__ __forceinline__ unsigned desc_lo(unsigned addr, unsigned plane) {
  return ((addr >> 4) & 0x3fff) | ((plane >> 4) << 16);
}
constexpr unsigned kDescHiA = ((kHX * 16u) >> 4) | (1u << 14), kDescHiB = (128u >> 4) | (1u << 14);

// kind::f16 instruction descriptor: FP32 accumulate, BF16 A and B, both K-major, M = 128.
__host__ __device__ constexpr unsigned idesc_bf16(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void mma(unsigned d, unsigned a_lo, unsigned b_lo, unsigned idesc, unsigned acc) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 da, db;\nsetp.ne.b32 p, %6, 0;\nmov.b64 da, {%1, %4};\nmov.b64 db, {%2, %5};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}" ::"r"(d),
      "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(kDescHiA), "r"(kDescHiB), "r"(acc)
      : "memory");
}

struct UmmaPlan {
  int nxt, nyt;  // tiles along x and y
  int zr, nz;    // planes per item, items along z
  int ncog;      // output-channel groups
  int slabs;     // slabs in the ring
};

template <int CO_T>
__global__ void __launch_bounds__(kThreads, 2) k_conv3_umma(const ConvIn in, const __nv_bfloat16* __restrict__ wt,
                                                            const ConvOut out, const UmmaPlan P, int* __restrict__ err) {
  pdl_entry();
  extern __shared__ __align__(1024) unsigned char smem[];
  constexpr int N = 3 * CO_T;
  constexpr unsigned kWPlane = 9u * N * 16u;  // 8 channels of a slice's weights
  const int Ci = in.C1 + in.C2, nsl = Ci / 16, Co = out.Co, H = in.H, W = in.W, D = in.D;
  const unsigned wbytes = (unsigned)nsl * 2u * kWPlane;
  const unsigned s_w = su32(smem), s_x = s_w + wbytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + wbytes + (size_t)P.slabs * kSlab);
  const unsigned b_full = su32(bars), b_empty = b_full + 8 * kMaxSlabs, b_accf = b_empty + 8 * kMaxSlabs,
                 b_acce = b_accf + 8 * kMaxPlanes;
  unsigned* tslot = reinterpret_cast<unsigned*>(bars + 2 * kMaxSlabs + 2 * kMaxPlanes);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tslot + 1);
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int co0 = (blockIdx.x % P.ncog) * CO_T;
  const int item0 = blockIdx.x / P.ncog, item_step = gridDim.x / P.ncog, items = P.nxt * P.nyt * P.nz;

  // weights of this channel group: slice, 8-channel chunk, (dy, dx), row j CO_T + co for dz = 1 - j
  for (int i = tid; i < nsl * 9 * N * 2; i += kThreads) {
    const int c = i & 1, r = i >> 1, n = r % N, q = r / N, yx = q % 9, sl = q / 9, j = n / CO_T, co = n % CO_T;
    const __nv_bfloat16* src = wt + ((size_t)((2 - j) * 9 + yx) * Co + co0 + co) * Ci + sl * 16 + c * 8;
    cp_async16(s_w + (unsigned)(sl * 2 + c) * kWPlane + (unsigned)(yx * N + n) * 16u, src, 16);
  }
  asm volatile("cp.async.commit_group;\n" ::);
  if (tid == 0) {
    for (int b = 0; b < P.slabs; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b_full + 8 * b), "r"(kCopyWarps));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_empty + 8 * b));
    }
    for (int p = 0; p < kMaxPlanes; ++p) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_accf + 8 * p));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b_acce + 8 * p), "r"(kEpiWarps));
    }
    *abort_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::);
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(tslot)), "n"(kCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("cp.async.wait_all;\n" ::: "memory");
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::);
  const unsigned tmem = *tslot;
  auto item_of = [&](int it, int& x0, int& y0, int& z0, int& z1) {
    x0 = (it % P.nxt) * kTX;
    it /= P.nxt;
    y0 = (it % P.nyt) * kTY;
    z0 = (it / P.nyt) * P.zr;
    z1 = min(z0 + P.zr, D);
  };

  if (warp >= kEpiWarps && warp < kMmaWarp) {
    // ---- slab copies
    constexpr int kPer = (kChunks + kCopyThreads - 1) / kCopyThreads;
    const int t = tid - kEpiWarps * 32;
    unsigned b = 0, phase = 1, pend = 0, pb = 0;  // ring position; slabs in flight and the oldest one's position
    for (int it = item0; it < items; it += item_step) {
      int x0, y0, z0, z1;
      item_of(it, x0, y0, z0, z1);
      for (int sl = 0; sl < nsl; ++sl) {
        const int ci = sl * 16;
        const bool one = ci < in.C1;
        const int C = one ? in.C1 : in.C2, sh = one && in.up1 ? 1 : 0;
        const __nv_bfloat16* base = one ? in.x1 + ci : in.x2 + (ci - in.C1);
        // this thread's chunks: place in the plane (or outside the volume) and in the slab
        int src[kPer];
        unsigned dst[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
          const int i = t + k * kCopyThreads, c = i & 1, v = i >> 1, y = y0 + v / kHX - 1, x = x0 + v % kHX - 1;
          const bool inside = (unsigned)y < (unsigned)H && (unsigned)x < (unsigned)W;
          src[k] = inside ? ((y >> sh) * (W >> sh) + (x >> sh)) * C + c * 8 : -1;
          dst[k] = (unsigned)c * kXPlane + (unsigned)v * 16u;
        }
        const size_t plane = (size_t)(H >> sh) * (W >> sh) * C;
        for (int zi = max(z0 - 1, 0); zi <= min(z1, D - 1); ++zi) {
          wait_phase(b_empty + 8 * b, phase, abort_word);
          const __nv_bfloat16* p = base + (size_t)(zi >> sh) * plane;
          const unsigned to = s_x + b * kSlab;
#pragma unroll
          for (int k = 0; k < kPer; ++k)
            if ((k + 1) * kCopyThreads <= kChunks || t + k * kCopyThreads < kChunks)
              cp_async16(to + dst[k], p + max(src[k], 0), src[k] >= 0 ? 16 : 0);
          asm volatile("cp.async.commit_group;\n" ::);
          if (++b == (unsigned)P.slabs) {
            b = 0;
            phase ^= 1;
          }
          // the slab two copies back is complete: hand it to the tensor cores
          if (++pend > 2) {
            asm volatile("cp.async.wait_group 2;\n" ::: "memory");
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            arrive(b_full + 8 * pb);
            pb = pb + 1 == (unsigned)P.slabs ? 0 : pb + 1;
            --pend;
          }
        }
      }
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (; pend; --pend) {
      arrive(b_full + 8 * pb);
      pb = pb + 1 == (unsigned)P.slabs ? 0 : pb + 1;
    }
  } else if (warp == kMmaWarp) {
    // ---- MMAs: a slab at zi into the output planes zi - 1 + j, j = 0, 1, 2 (dz = 1 - j), those of the item
    unsigned b = 0, phase = 0;
    unsigned pe = 0xffffffffu;  // parity to wait for before a plane is summed anew, by plane
    for (int it = item0; it < items; it += item_step) {
      int x0, y0, z0, z1;
      item_of(it, x0, y0, z0, z1);
      const int zf = max(z0 - 1, 0), zl = min(z1, D - 1);
      for (int sl = 0; sl < nsl; ++sl) {
        const unsigned w0 = desc_lo(s_w + (unsigned)sl * 2u * kWPlane, kWPlane);
        for (int zi = zf; zi <= zl; ++zi) {
          const int jlo = max(0, z0 - zi + 1), jhi = min(2, z1 - zi);
          const int jnew = min(max(sl ? 3 : (zi == 0 ? 1 : 2), jlo), jhi + 1);  // planes from here on start with this slab
          wait_phase(b_full + 8 * b, phase, abort_word);
          for (int j = jnew; j <= jhi; ++j) {
            const int k = zi - 1 + j - z0;
            wait_phase(b_acce + 8 * k, (pe >> k) & 1, abort_word);
            pe ^= 1u << k;
          }
          asm volatile("tcgen05.fence::after_thread_sync;" ::);
          const unsigned a0 = desc_lo(s_x + b * kSlab, kXPlane);
          const unsigned d = tmem + (unsigned)((zi - 1 - z0 + jlo) * CO_T), wj = w0 + (unsigned)(jlo * CO_T);
          const unsigned idesc = idesc_bf16(0) + ((unsigned)((jhi - jlo + 1) * CO_T / 8) << 17);
          if (elect_one()) {
            if (jnew > jhi) {
              mma(d, a0, wj, idesc, 1u);
            } else {  // the first tap pair overwrites in the planes that start here
              if (jnew > jlo) mma(d, a0, wj, idesc_bf16(0) + ((unsigned)((jnew - jlo) * CO_T / 8) << 17), 1u);
              mma(d + (unsigned)((jnew - jlo) * CO_T), a0, w0 + (unsigned)(jnew * CO_T),
                  idesc_bf16(0) + ((unsigned)((jhi - jnew + 1) * CO_T / 8) << 17), 0u);
            }
#pragma unroll
            for (int q = 1; q < 9; ++q) mma(d, a0 + (unsigned)((q / 3) * kHX + q % 3), wj + (unsigned)(q * N), idesc, 1u);
            commit_to(b_empty + 8 * b);
            if (sl == nsl - 1) {  // output planes whose last slab this was
              if (zi - 1 >= z0) commit_to(b_accf + 8 * (zi - 1 - z0));
              if (zi == D - 1 && zi < z1) commit_to(b_accf + 8 * (zi - z0));
            }
          }
          __syncwarp();
          if (++b == (unsigned)P.slabs) {
            b = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else {
    // ---- epilogue: thread (warp w, lane l) owns accumulator row 32 w + l, voxel (x0 + row % 8, y0 + row / 8)
    const int m = warp * 32 + lane;
    const float slope = out.relu ? out.slope : 1.f;  // v > 0 ? v : slope v = max(v, slope v) for slopes up to 1
    unsigned pf = 0;
    for (int it = item0; it < items; it += item_step) {
      int x0, y0, z0, z1;
      item_of(it, x0, y0, z0, z1);
      size_t at0 = (((size_t)z0 * H + (y0 + (m >> 3))) * W + (x0 + (m & 7))) * Co + co0;
      for (int zo = z0; zo < z1; ++zo, at0 += (size_t)H * W * Co) {
        const int k = zo - z0;
        wait_phase(b_accf + 8 * k, (pf >> k) & 1, abort_word);
        pf ^= 1u << k;
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::);
        unsigned r[CO_T];
#pragma unroll
        for (int j = 0; j < CO_T / 16; ++j)
          tmem_ld16(tmem + ((unsigned)(warp * 32) << 16) + (unsigned)(k * CO_T + 16 * j), r + 16 * j);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < CO_T; ++q) asm volatile("" : "+r"(r[q]));  // uses stay after the wait
        asm volatile("tcgen05.fence::before_thread_sync;" ::);
        arrive(b_acce + 8 * k);
#pragma unroll
        for (int c8 = 0; c8 < CO_T / 8; ++c8) {
          float v[8];
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            float t = __uint_as_float(r[c8 * 8 + q]);
            if (out.bias) t += __ldg(out.bias + co0 + c8 * 8 + q);
            v[q] = fmaxf(t, slope * t);
          }
          const size_t at = at0 + c8 * 8;
          if (out.mask) {
            const uint4 mk = *reinterpret_cast<const uint4*>(out.mask + at);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&mk);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (!(__low2float(h[q]) > 0.f)) v[2 * q] *= out.mask_slope;
              if (!(__high2float(h[q]) > 0.f)) v[2 * q + 1] *= out.mask_slope;
            }
          }
          if (out.yf) {
            float4* d = reinterpret_cast<float4*>(out.yf + at);
            d[0] = make_float4(v[0], v[1], v[2], v[3]);
            d[1] = make_float4(v[4], v[5], v[6], v[7]);
          } else {
            __align__(16) __nv_bfloat162 h[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) h[q] = __floats2bfloat162_rn(v[2 * q], v[2 * q + 1]);
            *reinterpret_cast<uint4*>(out.y + at) = *reinterpret_cast<const uint4*>(h);
          }
        }
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::);
  __syncthreads();
  if (tid == 0 && *abort_word) atomicOr(err, DF_TIMEOUT);
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::);
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kCols));
  }
}

constexpr size_t weight_bytes(int Ci, int co_t) { return (size_t)27 * Ci * co_t * 2; }

template <int CO_T>
vg_status launch_umma(Ctx* c, const ConvIn& in, const __nv_bfloat16* wt, const ConvOut& out) {
  const size_t wbytes = weight_bytes(in.C1 + in.C2, CO_T);
  const bool two = wbytes + kMinSlabs * kSlab + kTail <= kSmemTwo;
  UmmaPlan P;
  P.nxt = in.W / kTX;
  P.nyt = in.H / kTY;
  P.ncog = out.Co / CO_T;
  P.slabs = (int)std::min<size_t>(kMaxSlabs, ((two ? kSmemTwo : kSmemOne) - wbytes - kTail) / kSlab);
  // planes per item: the fewest rounds of items over the CTAs, counting the two extra input planes of an item
  const int ctas = std::max(1, (two ? 2 : 1) * sm_count() / P.ncog), zmax = std::min(in.D, kCols / CO_T);
  double best = 1e30;
  P.zr = 1;
  for (int zr = 1; zr <= zmax; ++zr) {
    const int nz = (in.D + zr - 1) / zr;
    const double cost = (double)((P.nxt * P.nyt * nz + ctas - 1) / ctas) * (zr + 2);
    if (cost < best - 1e-9) {
      best = cost;
      P.zr = zr;
    }
  }
  P.nz = (in.D + P.zr - 1) / P.zr;
  const size_t smem = wbytes + P.slabs * (size_t)kSlab + kTail;
  VG_CUDA(c, cudaFuncSetAttribute(k_conv3_umma<CO_T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  VG_CUDA(c, cudaFuncSetAttribute(k_conv3_umma<CO_T>, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
  const int grid = P.ncog * std::min(ctas, P.nxt * P.nyt * P.nz);
  pdl_launch(c->stream, (unsigned)grid, kThreads, smem, k_conv3_umma<CO_T>, in, wt, out, P, c->dflag);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

}  // namespace

bool conv3_umma_fits(const ConvIn& in, int Co) {
  return in.W % kTX == 0 && in.H % kTY == 0 && Co % 16 == 0 && (in.C1 + in.C2) % 16 == 0;
}

vg_status conv3_fwd_umma(Ctx* c, const ConvIn& in, const __nv_bfloat16* wt, const ConvOut& out, bool* handled) {
  *handled = false;
  if (!conv3_umma_fits(in, out.Co) || !c->dflag) return VG_OK;
  const int Ci = in.C1 + in.C2;
  auto fits = [&](int co_t, size_t smem) {
    return out.Co % co_t == 0 && weight_bytes(Ci, co_t) + kMinSlabs * kSlab + kTail <= smem;
  };
  *handled = true;
  // the widest group at two CTAs per SM, else at one
  for (const size_t smem : {kSmemTwo, kSmemOne}) {
    if (fits(48, smem) && out.Co % 32) return launch_umma<48>(c, in, wt, out);
    if (fits(32, smem)) return launch_umma<32>(c, in, wt, out);
    if (fits(16, smem)) return launch_umma<16>(c, in, wt, out);
  }
  *handled = false;
  return VG_OK;
}

}  // namespace nn
}  // namespace vg
