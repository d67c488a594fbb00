// Weight and bias gradients of the 3x3x3 convolutions on the 5th-generation tensor cores (tcgen05, sm_103a).
//
//   dW[dz][dy][dx][co][ci] = sum over voxels v of dY[v][co] X[v + (dx, dy, dz)][ci],  db[co] = sum of dY[v][co]
//
// A GEMM whose contraction runs over the voxels.  Channels-last rows of 16 channels are MN-major operands as they lie in
// memory: K = 16 voxels along x, 16 channels a group.  The taps are groups at constant strides:
//   A (M = 64)  four x rows y - 1 .. y + 2 of one plane of X, 16 input channels each;
//   B (N = 96)  the two rows y, y + 1 of dY, each in three copies shifted by dx = -1, 0, 1, 16 output channels each;
// so that D[(row, ci)][(row, dx, co)] holds the three dy taps of either dY row (three of its four row pairs) at once, and
// three accumulators (dz = -1, 0, 1; 288 columns of tensor memory) hold all 27 taps of a 16 x 16 block of channels.  They
// stay in tensor memory over a third of the CTA's share of the volume, and then are added to dW atomically: the tensor cores
// round their running sums toward zero, and with one drain for the whole share the error against 64 bits was twice that of
// the mma.sync kernel that this one replaces (with three it is smaller).
//
// A CTA owns one block of channels and a run of steps; a step is one plane z of a block of 256 / W rows (256 voxels): the
// X slab of plane z + 1 (the planes z - 1 and z are still in the ring) and the dY slab of plane z, then 24 MMAs.
// Warps 0..7 copy (X by cp.async; dY through registers, stored three times, and summed for db by the CTAs of the first
// input block), warps 8..11 drain the accumulators, warp 12 issues the MMAs.  Every wait is bounded, as in the
// forward kernel.
//
// Measured on GB300, db included, us a launch, against the mma.sync kernel and a separate column sum: 16 -> 16 on 128^3
// 248 + 85 -> 64, 48 -> 16 on 128^3 1213 + 89 -> 163, 96 -> 32 on 64^3 558 + 14 -> 91, 192 -> 64 on 32^3 280 + 5 -> 51; the
// network's 15 layers at edge 128 3590 + 517 -> 763.  What is left is a step's chain of waits (half of a step without its
// MMAs) and MMAs of 64 x 96 x 16 one after another.  Error against 64 bits at edge 128, root mean square over seeds, layer
// by layer: 0.6 to 0.9 of the mma.sync kernel's, at the 16-wide levels of small networks up to 1.09 of it (1.4e-7, FP32's
// own rounding); db about half of the column sum's.
#include <algorithm>

#include "vg_nn.cuh"

namespace vg {
namespace nn {

namespace {

constexpr int kCopyThreads = 256, kMmaWarp = kCopyThreads / 32 + 4, kThreads = kCopyThreads + 128 + 32;
constexpr int kDrains = 3;
constexpr int kXSlabs = 6, kYSlabs = 5;
constexpr unsigned kYSlab = 256 * 3 * 32;  // bytes of a dY slab: 256 voxels, three copies

// MN-major operands of 16-channel groups (32-byte rows, 32-byte swizzle): 8-voxel groups 256 bytes apart, channel groups
// one x row (W x 32 bytes) apart.
constexpr unsigned kDescHi = (256u >> 4) | (1u << 14) | (6u << 29);
// kind::f16: FP32 accumulators, BF16, both operands MN-major, N = 96, M = 64
constexpr unsigned kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((96u >> 3) << 17) | ((64u >> 4) << 24);

__device__ __forceinline__ void mma_wgrad(unsigned d, unsigned a_lo, unsigned b_lo) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 da, db;\nsetp.ne.b32 p, 1, 0;\nmov.b64 da, {%1, %4};\nmov.b64 db, {%2, %4};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n}" ::"r"(d),
      "r"(a_lo), "r"(b_lo), "r"(kIdesc), "r"(kDescHi)
      : "memory");
}

__device__ __forceinline__ void st16_zero(unsigned taddr) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};" ::"r"(taddr),
               "r"(0)
               : "memory");
}

template <int LW>
struct Shape {
  static constexpr int W = 1 << LW, P = 128 / W, XR = 2 * P + 2;  // row pairs a step, X rows of a slab
  static constexpr unsigned kXSlab = (unsigned)XR * W * 32u;
  static constexpr size_t smem = (size_t)kXSlabs * kXSlab + (size_t)kYSlabs * kYSlab + 256;
};

template <int LW>
__global__ void __launch_bounds__(kThreads, 1) k_conv3_wgrad_rows(const ConvIn in, const __nv_bfloat16* __restrict__ dy,
                                                                  int Co, float* __restrict__ dw, float* __restrict__ db,
                                                                  int* __restrict__ err) {
  pdl_entry();
  using S = Shape<LW>;
  constexpr int W = S::W, P = S::P, XR = S::XR;
  constexpr unsigned kXSlab = S::kXSlab;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
  const int H = in.H, D = in.D, Ci = in.C1 + in.C2, nci = Ci / 16;
  const int co0 = (blockIdx.x / nci) * 16, ci0 = (blockIdx.x % nci) * 16;
  const int steps = (H / (2 * P)) * D;
  const int s0 = (int)((long long)steps * blockIdx.y / gridDim.y), s1 = (int)((long long)steps * (blockIdx.y + 1) / gridDim.y);
  if (s0 >= s1) return;  // the whole CTA
  const int drains = min(kDrains, s1 - s0);  // drain k (from 0) comes after the first (k + 1) / drains of the steps
  const unsigned s_x = su32(smem), s_y = s_x + kXSlabs * kXSlab;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kXSlabs * kXSlab + kYSlabs * kYSlab);
  const unsigned b_xf = su32(bars), b_xe = b_xf + 8 * kXSlabs, b_yf = b_xe + 8 * kXSlabs, b_ye = b_yf + 8 * kYSlabs,
                 b_done = b_ye + 8 * kYSlabs, b_free = b_done + 8;
  unsigned* tslot = reinterpret_cast<unsigned*>(bars + 2 * kXSlabs + 2 * kYSlabs + 2);
  volatile int* abort_word = reinterpret_cast<volatile int*>(tslot + 1);
  if (tid == 0) {
    for (int b = 0; b < kXSlabs; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b_xf + 8 * b), "r"(kCopyThreads / 32));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_xe + 8 * b));
    }
    for (int b = 0; b < kYSlabs; ++b) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(b_yf + 8 * b), "r"(kCopyThreads / 32));
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_ye + 8 * b));
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_done));
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(b_free));
    *abort_word = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::);
  }
  // the shifted copies' ends (dY past a row's end) are never written: zero
  for (unsigned i = tid; i < kYSlabs * kYSlab / 16; i += kThreads)
    reinterpret_cast<uint4*>(smem + kXSlabs * kXSlab)[i] = make_uint4(0, 0, 0, 0);
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(su32(tslot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  asm volatile("tcgen05.fence::before_thread_sync;" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::);
  const unsigned tmem = *tslot;
  if (warp < 4) {  // the accumulators start from zero
    for (int j = 0; j < 18; ++j) st16_zero(tmem + ((unsigned)(warp * 32) << 16) + 16 * j);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::);
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::);

  if (warp < kCopyThreads / 32) {
    // ---- copies
    const int c = tid & 1, v0 = tid >> 1;  // 16-byte half of a voxel's 16 channels; first voxel
    const bool one = ci0 < in.C1;
    const int C = one ? in.C1 : in.C2, sh = one && in.up1 ? 1 : 0;
    const __nv_bfloat16* xbase = (one ? in.x1 + ci0 : in.x2 + (ci0 - in.C1)) + c * 8;
    const int xrow_c = (W >> sh) * C;
    const __nv_bfloat16* ybase = dy + co0 + c * 8;
    float sum[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) sum[j] = 0.f;
    const bool want_db = db && ci0 == 0;
    uint4 next[2];
    int z = s0 % D, yb = s0 / D;
    auto load_y = [&]() {  // this thread's two pieces of the step (yb, z)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int v = v0 + i * 128, row = v >> LW, x = v & (W - 1);
        next[i] = __ldg(reinterpret_cast<const uint4*>(ybase + (((size_t)z * H + yb * (2 * P) + row) * W + x) * Co));
      }
    };
    load_y();
    unsigned xb = 0, xphase = 1, yb_ = 0, yphase = 1, pend = 0, pb = 0;  // ring positions; X slabs in flight
   
    for (int s = s0; s < s1; ++s) {
      const int y0 = yb * (2 * P) - 1;
      // X planes this step is the first to need
      for (int zi = (s == s0 || z == 0) ? max(z - 1, 0) : z + 1; zi <= min(z + 1, D - 1); ++zi) {
        wait_phase(b_xe + 8 * xb, xphase, abort_word);
        const __nv_bfloat16* plane = xbase + (size_t)(zi >> sh) * (H >> sh) * xrow_c;
        const unsigned dst = s_x + xb * kXSlab + (unsigned)v0 * 32u + (unsigned)((c ^ ((v0 >> 2) & 1)) * 16);
#pragma unroll
        for (int i = 0; i < (XR * W + 127) / 128; ++i) {
          const int v = v0 + i * 128, row = v >> LW, x = v & (W - 1), y = y0 + row;
          if (XR * W % 128 == 0 || v < XR * W) {
            const bool in_y = (unsigned)y < (unsigned)H;
            const __nv_bfloat16* p = plane + (in_y ? (y >> sh) * xrow_c + (x >> sh) * C : 0);
            cp_async16(dst + i * 4096u, p, in_y ? 16 : 0);
          }
        }
        asm volatile("cp.async.commit_group;\n" ::);
        if (++xb == kXSlabs) {
          xb = 0;
          xphase ^= 1;
        }
        ++pend;
      }
      // dY: three copies, x shifted by dx
      wait_phase(b_ye + 8 * yb_, yphase, abort_word);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int v = v0 + i * 128, row = v >> LW, x = v & (W - 1);
        const uint4 q = next[i];
        unsigned char* rowp = smem + kXSlabs * kXSlab + yb_ * kYSlab + (unsigned)(row * 3) * W * 32u;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const int xs = x + d - 1;
          if ((unsigned)xs < (unsigned)W)
            *reinterpret_cast<uint4*>(rowp + d * W * 32 + xs * 32 + ((c ^ ((xs >> 2) & 1)) * 16)) = q;
        }
        if (want_db) {
          const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            sum[2 * j] += __low2float(h[j]);
            sum[2 * j + 1] += __high2float(h[j]);
          }
        }
      }
      // the X slabs but the newest two are complete; one fence for them and for dY
      asm volatile("cp.async.wait_group 2;\n" ::: "memory");
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      for (; pend > 2; --pend) {
        arrive(b_xf + 8 * pb);
        pb = pb + 1 == kXSlabs ? 0 : pb + 1;
      }
      arrive(b_yf + 8 * yb_);
      if (++yb_ == kYSlabs) {
        yb_ = 0;
        yphase ^= 1;
      }
      if (++z == D) {
        z = 0;
        ++yb;
      }
      if (s + 1 < s1) load_y();
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    for (; pend; --pend) {
      arrive(b_xf + 8 * pb);
      pb = pb + 1 == kXSlabs ? 0 : pb + 1;
    }
    if (want_db) {  // lanes of equal parity hold the same 8 channels
      __shared__ float sh_db[kCopyThreads / 32][16];
#pragma unroll
      for (int j = 0; j < 8; ++j)
        for (int o = 16; o > 1; o >>= 1) sum[j] += __shfl_xor_sync(0xffffffffu, sum[j], o);
      if (lane < 2)
#pragma unroll
        for (int j = 0; j < 8; ++j) sh_db[warp][c * 8 + j] = sum[j];
      // one addition to db a CTA: its rounding is of the whole sum, so that one a warp made the error 1.4 times the column
      // sum kernel's
      asm volatile("bar.sync 1, %0;" ::"n"(kCopyThreads) : "memory");
      if (tid < 16) {
        float t = 0.f;
        for (int w = 0; w < kCopyThreads / 32; ++w) t += sh_db[w][tid];
        atomicAdd(db + co0 + tid, t);
      }
    }
  } else if (warp == kMmaWarp) {
    // ---- MMAs.  Ring positions of X: xl the newest slab received (plane zt), xo the oldest not given back.
    int end = s0 + (s1 - s0) / drains, drained = 0;  // the drain after the steps before `end`; drains asked for
    bool fresh = false;                              // the step before asked for a drain
    unsigned xl = kXSlabs - 1, xphase = 0, xo = 0, held = 0, yb_ = 0, yphase = 0;
    int z = s0 % D;
    bool start = true;  // a new run of planes
    for (int s = s0; s < s1; ++s) {
      const int zt = min(z + 1, D - 1);
      for (int zi = start ? max(z - 1, 0) : z + 1; zi <= zt; ++zi, ++held) {
        if (++xl == kXSlabs) xl = 0;
        wait_phase(b_xf + 8 * xl, xphase, abort_word);
        if (xl == kXSlabs - 1) xphase ^= 1;
      }
      wait_phase(b_yf + 8 * yb_, yphase, abort_word);
      if (fresh) wait_phase(b_free, (drained - 1) & 1, abort_word);
      fresh = s + 1 == end;
      asm volatile("tcgen05.fence::after_thread_sync;" ::);
      const unsigned blo = ((s_y + yb_ * kYSlab) >> 4) | ((unsigned)(W * 32 / 16) << 16);
      start = s + 1 == s1 || z == D - 1;  // the end of a run: every slab held goes back, else those before plane z
      const unsigned keep = start ? 0 : 1 + (unsigned)(zt - z);
      if (elect_one()) {
#pragma unroll
        for (int dz = -1; dz <= 1; ++dz) {
          const int zi = z + dz;
          if (zi < 0 || zi >= D) continue;
          const unsigned back = (unsigned)(zt - zi), at = xl >= back ? xl - back : xl + kXSlabs - back;
          const unsigned alo = ((s_x + at * kXSlab) >> 4) | ((unsigned)(W * 32 / 16) << 16);
#pragma unroll
          for (int p = 0; p < P; ++p)
#pragma unroll
            for (int k = 0; k < W / 16; ++k)
              mma_wgrad(tmem + (unsigned)(dz + 1) * 96u, alo + (unsigned)(2 * p * W * 2 + k * 32),
                        blo + (unsigned)(p * 6 * W * 2 + k * 32));
        }
        commit_to(b_ye + 8 * yb_);
        for (unsigned x = xo, h = held; h > keep; --h) {
          commit_to(b_xe + 8 * x);
          if (++x == kXSlabs) x = 0;
        }
        if (fresh) commit_to(b_done);
      }
      __syncwarp();
      for (; held > keep; --held)
        if (++xo == kXSlabs) xo = 0;
      if (fresh) {
        ++drained;
        end = s0 + (int)((long long)(s1 - s0) * (drained + 1) / drains);
      }
      if (++z == D) z = 0;
      if (++yb_ == kYSlabs) {
        yb_ = 0;
        yphase ^= 1;
      }
    }
  } else {
    // ---- drains: warp r (of four) holds X row r, lanes 0..15 the input channels; columns (dz, dY row, dx, co)
    const int w4 = warp & 3;
    for (int round = 0; round < drains; ++round) {
      wait_phase(b_done, round & 1, abort_word);
      __syncwarp();
      asm volatile("tcgen05.fence::after_thread_sync;" ::);
      for (int j = 0; j < 18; ++j) {
        const int dz = j / 6, row = (j / 3) % 2, dx = j % 3, dyt = w4 - row;  // tap dy + 1 of this X row and dY row
        const unsigned at = tmem + ((unsigned)(w4 * 32) << 16) + 16 * j;
        unsigned r[16];
        tmem_ld16(at, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int q = 0; q < 16; ++q) asm volatile("" : "+r"(r[q]));
        st16_zero(at);
        if (dyt >= 0 && dyt < 3 && lane < 16) {
          float* p = dw + ((size_t)((dz * 3 + dyt) * 3 + dx) * Co + co0) * Ci + ci0 + lane;
#pragma unroll
          for (int q = 0; q < 16; ++q) atomicAdd(p + (size_t)q * Ci, __uint_as_float(r[q]));
        }
      }
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      asm volatile("tcgen05.fence::before_thread_sync;" ::);
      arrive(b_free);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::);
  __syncthreads();
  if (tid == 0 && *abort_word) atomicOr(err, DF_TIMEOUT);
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::);
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

template <int LW>
vg_status launch_wgrad(Ctx* c, const ConvIn& in, const __nv_bfloat16* dy, int Co, float* dw, float* db) {
  using S = Shape<LW>;
  VG_CUDA(c, cudaFuncSetAttribute(k_conv3_wgrad_rows<LW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::smem));
  const int blocks = (Co / 16) * ((in.C1 + in.C2) / 16), steps = (in.H / (2 * S::P)) * in.D;
  const int splits = std::max(1, std::min(steps, sm_count() / blocks));
  pdl_launch(c->stream, dim3((unsigned)blocks, (unsigned)splits), kThreads, S::smem, k_conv3_wgrad_rows<LW>, in, dy, Co, dw, db,
                                                                                                    c->dflag);
  VG_LAUNCHED(c);
  VG_CUDA(c, cudaGetLastError());
  return VG_OK;
}

}  // namespace

vg_status conv3_wgrad_rows(Ctx* c, const ConvIn& in, const __nv_bfloat16* dy, int Co, float* dw, float* db, bool* handled) {
  *handled = false;
  int lw = 4;
  while (lw < 7 && (1 << lw) != in.W) ++lw;
  if (!c->dflag || (1 << lw) != in.W || in.H % (256 / in.W) || in.C1 % 16 || in.C2 % 16 || Co % 16) return VG_OK;
  if (((uintptr_t)in.x1 | (uintptr_t)in.x2 | (uintptr_t)dy) & 15) return VG_OK;
  *handled = true;
  switch (lw) {
    case 4: return launch_wgrad<4>(c, in, dy, Co, dw, db);
    case 5: return launch_wgrad<5>(c, in, dy, Co, dw, db);
    case 6: return launch_wgrad<6>(c, in, dy, Co, dw, db);
    default: return launch_wgrad<7>(c, in, dy, Co, dw, db);
  }
}

}  // namespace nn
}  // namespace vg
