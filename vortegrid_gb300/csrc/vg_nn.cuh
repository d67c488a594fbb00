// Declarations shared by the learned warm-start kernels (vg_nn_conv.cu, vg_nn.cu).
//
// Tensors are channels-last BF16 ([D][H][W][C], C a multiple of 16); weights
// of a 3x3x3 convolution are [27][Co][Ci] BF16 with tap = (dz+1)*9 + (dy+1)*3 + (dx+1).
#pragma once

#include <cuda_bf16.h>

#include "vg_internal.cuh"

namespace vg {
namespace nn {

// Input of a convolution: x1 (C1 channels), optionally read through a
// nearest-neighbour 2x upsampling (x1 then has dims D/2, H/2, W/2), followed
// by x2 (C2 channels, may be 0) at the output resolution D x H x W.
struct ConvIn {
  const __nv_bfloat16* x1;
  const __nv_bfloat16* x2;
  int C1, C2;
  int up1;
  int D, H, W;
};

// Output: y (BF16) or yf (FP32), Co channels; + bias, then the leaky ReLU
// (v > 0 ? v : slope v) when relu != 0, then, with a mask tensor (same layout
// as the output), a factor mask_slope wherever the mask entry is <= 0 (the
// derivative of that activation, for input gradients).
struct ConvOut {
  __nv_bfloat16* y;
  float* yf;
  const float* bias;
  const __nv_bfloat16* mask;
  int Co;
  int relu;
  float slope;
  float mask_slope;
};

bool conv_shape_ok(int D, int H, int W, int C1, int C2, int Co);
size_t conv3_fwd_smem(int D, int H, int W, int co_t);
vg_status conv3_fwd(Ctx* c, const ConvIn& in, const __nv_bfloat16* wt, const ConvOut& out);
// The tcgen05 form (tiles of 8 x 16 voxels; needs W % 8 == 0, H % 16 == 0, the
// weights of one output-channel group within shared memory, and c->dflag for
// its timeout bit); *handled says whether it ran.
vg_status conv3_fwd_umma(Ctx* c, const ConvIn& in, const __nv_bfloat16* wt, const ConvOut& out, bool* handled);
// dW[27][Co][Ci] += sum over voxels of dY (x) X_tap  (FP32, accumulated atomically)
vg_status conv3_wgrad(Ctx* c, const ConvIn& in, const __nv_bfloat16* dy, int Co, float* dw);
// The same, and db[Co] += sum over voxels of dY, over whole x rows (W = 16, 32, 64 or 128; vg_nn_wgrad.cu).
vg_status conv3_wgrad_rows(Ctx* c, const ConvIn& in, const __nv_bfloat16* dy, int Co, float* dw, float* db, bool* handled);

// ---- mbarriers, asynchronous copies and tensor memory, as the tcgen05 kernels use them

__device__ __forceinline__ unsigned su32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ bool try_wait(unsigned mbar, unsigned parity) {
  unsigned done;
  asm volatile(
      "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}"
      : "=r"(done)
      : "r"(mbar), "r"(parity)
      : "memory");
  return done != 0;
}

// Waits for a phase, 2 s at most; a wait that runs out sets the abort word, which ends every later wait at once.
constexpr unsigned long long kWaitNs = 2000000000ull;
__device__ __forceinline__ void wait_phase(unsigned mbar, unsigned parity, volatile int* abort_word) {
  for (int k = 0; k < 512; ++k)
    if (try_wait(mbar, parity)) return;
  unsigned long long t0, t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t0));
  while (!*abort_word) {
    for (int k = 0; k < 16; ++k)
      if (try_wait(mbar, parity)) return;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    if (t - t0 > kWaitNs) *abort_word = 1;
  }
}

// One arrival for the warp, after all of its lanes.
__device__ __forceinline__ void arrive(unsigned mbar) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ void commit_to(unsigned mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
}

__device__ __forceinline__ bool elect_one() {
  unsigned r;
  asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}" : "=r"(r));
  return r != 0;
}

__device__ __forceinline__ void cp_async16(unsigned dst, const void* src, int src_bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// 16 consecutive FP32 accumulator columns of this thread's TMEM lane.
__device__ __forceinline__ void tmem_ld16(unsigned taddr, unsigned* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}

}  // namespace nn
}  // namespace vg
