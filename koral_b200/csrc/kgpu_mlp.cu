// The warm-start network: a 16 -> 128 -> 128 -> 7 multilayer perceptron with
// SiLU activations, BF16 weights and activations and FP32 accumulation on
// the tensor cores (mma.sync m16n8k16), trained on the device by the
// kernels below (forward, backward, Adam) and evaluated on the device to
// give every cell of a batched implicit solve its initial iterate.
//
// Tile of work: in inference a warp carries 16 samples (the M dimension of
// one mma) through all layers in registers, sixteen warps a block; a training
// block has sixteen warps on 64 samples, each 16 samples by 32 columns.
// Weights sit in shared memory as BF16, laid out [output][input], and reach
// the tensor cores by ldmatrix.  FP32 master weights, their gradients and
// Adam moments stay in global memory.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <vector>

#include "../../include/koral_b200.h"
#include "kgpu_mlp.cuh"

using namespace kgpu;

int kgpu_report_cuda(const char *what, cudaError_t e);

namespace {

#define MCK(call)                                              \
  do {                                                         \
    cudaError_t e_ = (call);                                   \
    if (e_ != cudaSuccess) return kgpu_report_cuda(#call, e_); \
  } while (0)

typedef __nv_bfloat16 bf16;

// FP32 parameter blob: W1[16][128], b1[128], W2[128][128], b2[128],
// W3[128][8] (output 7 unused, kept zero), b3[8]; then the output
// standardisation mean[8], scale[8].
constexpr int OW1 = 0;
constexpr int OB1 = OW1 + MLP_IN * MLP_H;
constexpr int OW2 = OB1 + MLP_H;
constexpr int OB2 = OW2 + MLP_H * MLP_H;
constexpr int OW3 = OB2 + MLP_H;
constexpr int OB3 = OW3 + MLP_H * MLP_OUTP;
constexpr int NPARAM = OB3 + MLP_OUTP;
constexpr int OMEAN = NPARAM, OSCALE = NPARAM + MLP_OUTP;
constexpr int NBLOB = NPARAM + 2 * MLP_OUTP;

// padded leading dimensions of the shared-memory tiles (bf16 elements)
constexpr int LDX = MLP_IN + 8;    // 24
constexpr int LDH = MLP_H + 8;     // 136

// BF16 weights in the [output][input] layout the fragments want
struct Bf16Weights {
  bf16 *w1t;   // [128][16]
  bf16 *w2t;   // [128][128]
  bf16 *w3t;   // [8][128]
};

__device__ inline int lane_id() { return threadIdx.x & 31; }

__device__ inline void mma16816(float c[4], const uint32_t a[4], const uint32_t b[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

__device__ inline uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// four 8x8 tiles of 16-bit elements, lane l giving the address of row l % 8
// of tile l / 8; with trans, each tile transposed
__device__ inline void ldsm4(uint32_t r[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ inline void ldsm4t(uint32_t r[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// Fragments by ldmatrix.  A (m16 x k16 at m0, k0) of a matrix stored [m][ld]
// or [k][ld]; two B fragments (k16 x n8 at n0 and n0 + 8, in b[0..1] and
// b[2..3]) of a matrix stored [n][ld] or [k][ld].
__device__ inline void frag_a_mk(uint32_t a[4], const bf16 *A, int ld, int m0, int k0) {
  const int l = lane_id();
  ldsm4(a, smem_addr(A + (m0 + (l & 15)) * ld + k0 + (l >> 4) * 8));
}
__device__ inline void frag_a_km(uint32_t a[4], const bf16 *A, int ld, int m0, int k0) {
  const int l = lane_id();
  ldsm4t(a, smem_addr(A + (k0 + (l & 7) + ((l >> 4) & 1) * 8) * ld + m0 + ((l >> 3) & 1) * 8));
}
__device__ inline void frag_b2_nk(uint32_t b[4], const bf16 *B, int ld, int n0, int k0) {
  const int l = lane_id();
  ldsm4(b, smem_addr(B + (n0 + (l & 7) + ((l >> 4) & 1) * 8) * ld + k0 + ((l >> 3) & 1) * 8));
}
__device__ inline void frag_b2_kn(uint32_t b[4], const bf16 *B, int ld, int n0, int k0) {
  const int l = lane_id();
  ldsm4t(b, smem_addr(B + (k0 + (l & 7) + ((l >> 3) & 1) * 8) * ld + n0 + ((l >> 4) & 1) * 8));
}
__device__ inline uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t *>(&v);
}

__device__ inline float silu(float z) { return z / (1.f + __expf(-z)); }
__device__ inline float dsilu(float z) {
  const float s = 1.f / (1.f + __expf(-z));
  return s * (1.f + z * (1.f - s));
}

// shared-memory image of the weights of one block
struct alignas(16) SmemW {
  bf16 w1t[MLP_H * LDX];
  bf16 w2t[MLP_H * LDH];
  bf16 w3t[MLP_OUTP * LDH];
  float b1[MLP_H], b2[MLP_H], b3[MLP_OUTP];
};
// 16 bytes (8 elements of a row) at a time
__device__ void load_weights(SmemW &w, const Bf16Weights W, const float *blob) {
  for (int i = threadIdx.x; i < MLP_H * MLP_IN / 8; i += blockDim.x) {
    const int n = i / (MLP_IN / 8), k = i % (MLP_IN / 8) * 8;
    *(uint4 *)(w.w1t + n * LDX + k) = ((const uint4 *)W.w1t)[i];
  }
  for (int i = threadIdx.x; i < MLP_H * MLP_H / 8; i += blockDim.x) {
    const int n = i / (MLP_H / 8), k = i % (MLP_H / 8) * 8;
    *(uint4 *)(w.w2t + n * LDH + k) = ((const uint4 *)W.w2t)[i];
  }
  for (int i = threadIdx.x; i < MLP_OUTP * MLP_H / 8; i += blockDim.x) {
    const int n = i / (MLP_H / 8), k = i % (MLP_H / 8) * 8;
    *(uint4 *)(w.w3t + n * LDH + k) = ((const uint4 *)W.w3t)[i];
  }
  for (int i = threadIdx.x; i < MLP_H; i += blockDim.x) {
    w.b1[i] = blob[OB1 + i];
    w.b2[i] = blob[OB2 + i];
  }
  for (int i = threadIdx.x; i < MLP_OUTP; i += blockDim.x) w.b3[i] = blob[OB3 + i];
}

// two 8-column accumulator tiles (columns 16 ks .. 16 ks + 15 of a layer's
// pre-activations) as the A fragment of k-step ks of the next layer: the
// layouts agree, so activations never leave the registers
__device__ inline void activate(uint32_t a[4], const float c0[4], const float c1[4]) {
  a[0] = pack2(silu(c0[0]), silu(c0[1]));
  a[1] = pack2(silu(c0[2]), silu(c0[3]));
  a[2] = pack2(silu(c1[0]), silu(c1[1]));
  a[3] = pack2(silu(c1[2]), silu(c1[3]));
}

// neighbouring floats of the caller's arrays: one access where they are
// aligned for it (WIDE: X to 16 bytes and Y to 8), else one by one
template <bool WIDE>
__device__ inline float2 load2(const float *p) {
  return WIDE ? *(const float2 *)p : make_float2(p[0], p[1]);
}
template <bool WIDE>
__device__ inline float4 load4(const float *p) {
  return WIDE ? *(const float4 *)p : make_float4(p[0], p[1], p[2], p[3]);
}
template <bool WIDE>
__device__ inline void store2(float *p, float a, float b) {
  if (WIDE) {
    *(float2 *)p = make_float2(a, b);
  } else {
    p[0] = a;
    p[1] = b;
  }
}

// 16 warps of 124 registers fill the register file of an SM
constexpr int kInferWarps = 16;

// Inference: Y[n][8] = unstandardised outputs; the block's warps share the
// weights.  A warp takes 16 samples at a time through the three layers in
// registers; all 16 output tiles of the second layer are in flight, so the
// tensor-core latency of one chain is hidden by the others.  What bounds it is
// the issue of the activations (128 exponentials and divisions a lane and
// tile).  With the activations passed through shared memory and fragments
// from 32-bit loads 2^20 samples took 394 us, now 337.
template <bool WIDE>
__global__ void __launch_bounds__(32 * kInferWarps) k_mlp_forward(const float *blob, Bf16Weights W, const float *X,
                                                                  int n, float *Y) {
  extern __shared__ __align__(16) unsigned char smem[];
  SmemW &w = *reinterpret_cast<SmemW *>(smem);
  load_weights(w, W, blob);
  __syncthreads();
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int g = lane_id() >> 2, t = lane_id() & 3;
  const float sc0 = blob[OSCALE + 2 * t], sc1 = blob[OSCALE + 2 * t + 1];
  const float mn0 = blob[OMEAN + 2 * t], mn1 = blob[OMEAN + 2 * t + 1];
  // the third layer's weights stay in registers
  uint32_t w3[MLP_H / 16][2];
#pragma unroll
  for (int ks = 0; ks < MLP_H / 16; ks++) {
    w3[ks][0] = *(const uint32_t *)(w.w3t + g * LDH + ks * 16 + 2 * t);
    w3[ks][1] = *(const uint32_t *)(w.w3t + g * LDH + ks * 16 + 2 * t + 8);
  }
  for (int s0 = warp * 16; s0 < n; s0 += nwarps * 16) {
    const int r0 = s0 + g, r1 = s0 + g + 8;
    const float2 zero = make_float2(0.f, 0.f);
    const float2 x0 = r0 < n ? load2<WIDE>(X + (long)r0 * MLP_IN + 2 * t) : zero;
    const float2 x1 = r1 < n ? load2<WIDE>(X + (long)r1 * MLP_IN + 2 * t) : zero;
    const float2 x2 = r0 < n ? load2<WIDE>(X + (long)r0 * MLP_IN + 2 * t + 8) : zero;
    const float2 x3 = r1 < n ? load2<WIDE>(X + (long)r1 * MLP_IN + 2 * t + 8) : zero;
    const uint32_t ax[4] = {pack2(x0.x, x0.y), pack2(x1.x, x1.y), pack2(x2.x, x2.y), pack2(x3.x, x3.y)};
    float c[MLP_H / 8][4];
#pragma unroll
    for (int nt = 0; nt < MLP_H / 8; nt++) {
      const float2 b = *(const float2 *)(w.b2 + nt * 8 + 2 * t);
      c[nt][0] = c[nt][2] = b.x;
      c[nt][1] = c[nt][3] = b.y;
    }
    // layer 1 (16 x 16 . 16 x 128) 16 columns at a time, each the k-step of
    // layer 2 (16 x 128 . 128 x 128)
#pragma unroll
    for (int ks = 0; ks < MLP_H / 16; ks++) {
      float h[2][4];
      uint32_t b[4], a[4];
      frag_b2_nk(b, w.w1t, LDX, ks * 16, 0);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const float2 bb = *(const float2 *)(w.b1 + ks * 16 + j * 8 + 2 * t);
        h[j][0] = h[j][2] = bb.x;
        h[j][1] = h[j][3] = bb.y;
        mma16816(h[j], ax, b + 2 * j);
      }
      activate(a, h[0], h[1]);
#pragma unroll
      for (int nt = 0; nt < MLP_H / 8; nt += 2) {
        frag_b2_nk(b, w.w2t, LDH, nt * 8, ks * 16);
        mma16816(c[nt], a, b);
        mma16816(c[nt + 1], a, b + 2);
      }
    }
    // layer 3: 16 x 128 . 128 x 8
    float y[4] = {w.b3[2 * t], w.b3[2 * t + 1], w.b3[2 * t], w.b3[2 * t + 1]};
#pragma unroll
    for (int ks = 0; ks < MLP_H / 16; ks++) {
      uint32_t a[4];
      activate(a, c[2 * ks], c[2 * ks + 1]);
      mma16816(y, a, w3[ks]);
    }
    if (r0 < n) store2<WIDE>(Y + (long)r0 * MLP_OUTP + 2 * t, y[0] * sc0 + mn0, y[1] * sc1 + mn1);
    if (r1 < n) store2<WIDE>(Y + (long)r1 * MLP_OUTP + 2 * t, y[2] * sc0 + mn0, y[3] * sc1 + mn1);
  }
}

// the samples and activations of a training block
constexpr int kTrainWarps = 16, kTile = 64;
constexpr int LDZ = MLP_H + 4;   // FP32 rows
struct alignas(16) SmemTrain {
  bf16 x[kTile * LDX];
  bf16 a1[kTile * LDH], a2[kTile * LDH], dz2[kTile * LDH];
  float dz1[kTile * LDZ];
  float y[kTile * MLP_OUTP];   // outputs, then dL/dy
};
__device__ inline void red2(float *p, float a, float b) {   // two neighbours, 8-byte aligned
  asm volatile("red.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(p), "f"(a), "f"(b) : "memory");
}

// One training batch: forward and backward of 64 samples per block; the
// loss is the mean over the batch of the squared error of the standardised
// outputs; gradients are added to grad (FP32, zeroed by the caller).
// A batch of 8192 is 128 blocks, one wave of one block an SM: its time is the
// chain of one tile.  So sixteen warps share a tile, each 16 samples (mt) by 32
// columns (cg): the pre-activations of its part stay in its registers until
// the backward pass wants them, and the weight gradients read the activations
// transposed (ldmatrix.trans) instead of copies.  With four warps of 16
// samples each an epoch of 2^18 samples took 4.17 ms, now 1.58 (a launch 104 us
// under the profiler before).
template <bool WIDE>
__global__ void __launch_bounds__(32 * kTrainWarps) k_mlp_train(const float *blob, Bf16Weights W, const float *X,
                                                                const float *T, const int *order, int n, int nbatch,
                                                                float *grad, double *loss) {
  extern __shared__ __align__(16) unsigned char smem[];
  SmemW &w = *reinterpret_cast<SmemW *>(smem);
  SmemTrain &sb = *reinterpret_cast<SmemTrain *>(smem + sizeof(SmemW));
  const int tid = threadIdx.x, wi = tid >> 5, mt = wi >> 2, cg = wi & 3;
  const int g = lane_id() >> 2, t = lane_id() & 3;
  load_weights(w, W, blob);
  const float inv = 1.f / (float)nbatch;
  (void)n;
  for (int b0 = blockIdx.x * kTile; b0 < nbatch; b0 += gridDim.x * kTile) {
    __syncthreads();   // the weights are there; the tile before is done with
    // gather the samples of this tile
    for (int i = tid; i < kTile * MLP_IN / 4; i += blockDim.x) {
      const int r = i / (MLP_IN / 4), f = i % (MLP_IN / 4) * 4;
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      if (b0 + r < nbatch) v = load4<WIDE>(X + (long)order[b0 + r] * MLP_IN + f);
      *(uint2 *)(sb.x + r * LDX + f) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
    }
    __syncthreads();
    // layers 1 and 2: this warp's 16 x 32 part of the pre-activations
    float z1[4][4], z2[4][4];
    uint32_t a[4], b[4];
    frag_a_mk(a, sb.x, LDX, mt * 16, 0);
#pragma unroll
    for (int j = 0; j < 4; j += 2) {
      frag_b2_nk(b, w.w1t, LDX, cg * 32 + j * 8, 0);
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int c0 = cg * 32 + (j + q) * 8 + 2 * t;
        float *z = z1[j + q];
        z[0] = z[2] = w.b1[c0];
        z[1] = z[3] = w.b1[c0 + 1];
        mma16816(z, a, b + 2 * q);
        *(uint32_t *)(sb.a1 + (mt * 16 + g) * LDH + c0) = pack2(silu(z[0]), silu(z[1]));
        *(uint32_t *)(sb.a1 + (mt * 16 + g + 8) * LDH + c0) = pack2(silu(z[2]), silu(z[3]));
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int c0 = cg * 32 + j * 8 + 2 * t;
      z2[j][0] = z2[j][2] = w.b2[c0];
      z2[j][1] = z2[j][3] = w.b2[c0 + 1];
    }
#pragma unroll
    for (int ks = 0; ks < MLP_H / 16; ks++) {
      frag_a_mk(a, sb.a1, LDH, mt * 16, ks * 16);
#pragma unroll
      for (int j = 0; j < 4; j += 2) {
        frag_b2_nk(b, w.w2t, LDH, cg * 32 + j * 8, ks * 16);
        mma16816(z2[j], a, b);
        mma16816(z2[j + 1], a, b + 2);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
      const int c0 = cg * 32 + j * 8 + 2 * t;
      *(uint32_t *)(sb.a2 + (mt * 16 + g) * LDH + c0) = pack2(silu(z2[j][0]), silu(z2[j][1]));
      *(uint32_t *)(sb.a2 + (mt * 16 + g + 8) * LDH + c0) = pack2(silu(z2[j][2]), silu(z2[j][3]));
    }
    __syncthreads();
    // layer 3 and the output error (standardised targets): one warp per 16
    // samples
    if (cg == 0) {
      const int c0 = 2 * t;
      float y[4] = {w.b3[c0], w.b3[c0 + 1], w.b3[c0], w.b3[c0 + 1]};
#pragma unroll
      for (int ks = 0; ks < MLP_H / 16; ks++) {
        frag_a_mk(a, sb.a2, LDH, mt * 16, ks * 16);
        b[0] = *(const uint32_t *)(w.w3t + g * LDH + ks * 16 + 2 * t);
        b[1] = *(const uint32_t *)(w.w3t + g * LDH + ks * 16 + 2 * t + 8);
        mma16816(y, a, b);
      }
      float lsum = 0.f;
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = mt * 16 + g + (q >> 1) * 8, o = c0 + (q & 1);
        float d = 0.f;
        if (b0 + r < nbatch && o < MLP_OUT) {
          const float tt = (T[(long)order[b0 + r] * MLP_OUT + o] - blob[OMEAN + o]) / blob[OSCALE + o];
          const float e = y[q] - tt;
          lsum += e * e;
          d = 2.f * e * inv;
        }
        sb.y[r * MLP_OUTP + o] = d;
      }
      for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
      if (lane_id() == 0 && lsum != 0.f) atomicAdd(loss, (double)(lsum * inv));
    }
    __syncthreads();
    // dL/da2 = dy . W3^T (K = 8: in FP32), dz2 = da2 silu'(z2)
    {
      float dy[2][MLP_OUTP];
#pragma unroll
      for (int h = 0; h < 2; h++)
#pragma unroll
        for (int o = 0; o < MLP_OUTP; o++) dy[h][o] = sb.y[(mt * 16 + g + 8 * h) * MLP_OUTP + o];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int c0 = cg * 32 + j * 8 + 2 * t;
        float da[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int o = 0; o < MLP_OUTP; o++) {
          const float2 w3 = __bfloat1622float2(*(const __nv_bfloat162 *)(w.w3t + o * LDH + c0));
          da[0] += dy[0][o] * w3.x;
          da[1] += dy[0][o] * w3.y;
          da[2] += dy[1][o] * w3.x;
          da[3] += dy[1][o] * w3.y;
        }
        *(uint32_t *)(sb.dz2 + (mt * 16 + g) * LDH + c0) = pack2(da[0] * dsilu(z2[j][0]), da[1] * dsilu(z2[j][1]));
        *(uint32_t *)(sb.dz2 + (mt * 16 + g + 8) * LDH + c0) = pack2(da[2] * dsilu(z2[j][2]), da[3] * dsilu(z2[j][3]));
      }
    }
    __syncthreads();
    // dL/da1 = dz2 . W2 (tensor cores: K = outputs of layer 2), dz1 = da1 silu'(z1)
    {
      float da[4][4];
#pragma unroll
      for (int j = 0; j < 4; j++) da[j][0] = da[j][1] = da[j][2] = da[j][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < MLP_H / 16; ks++) {
        frag_a_mk(a, sb.dz2, LDH, mt * 16, ks * 16);
#pragma unroll
        for (int j = 0; j < 4; j += 2) {
          frag_b2_kn(b, w.w2t, LDH, cg * 32 + j * 8, ks * 16);
          mma16816(da[j], a, b);
          mma16816(da[j + 1], a, b + 2);
        }
      }
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int c0 = cg * 32 + j * 8 + 2 * t;
        *(float2 *)(sb.dz1 + (mt * 16 + g) * LDZ + c0) = make_float2(da[j][0] * dsilu(z1[j][0]), da[j][1] * dsilu(z1[j][1]));
        *(float2 *)(sb.dz1 + (mt * 16 + g + 8) * LDZ + c0) =
            make_float2(da[j][2] * dsilu(z1[j][2]), da[j][3] * dsilu(z1[j][3]));
      }
    }
    // W2 gradient = a1^T . dz2 over the tile's samples (tensor cores: M = in
    // i, N = out j, K = samples); a warp takes 16 inputs by 64 outputs
    {
      const int m0 = (wi >> 1) * 16, n0 = (wi & 1) * 64;
      float c[8][4];
#pragma unroll
      for (int j = 0; j < 8; j++) c[j][0] = c[j][1] = c[j][2] = c[j][3] = 0.f;
#pragma unroll
      for (int ks = 0; ks < kTile / 16; ks++) {
        frag_a_km(a, sb.a1, LDH, m0, ks * 16);
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
          frag_b2_kn(b, sb.dz2, LDH, n0 + j * 8, ks * 16);
          mma16816(c[j], a, b);
          mma16816(c[j + 1], a, b + 2);
        }
      }
#pragma unroll
      for (int j = 0; j < 8; j++) {
        float *p = grad + OW2 + (m0 + g) * MLP_H + n0 + j * 8 + 2 * t;
        red2(p, c[j][0], c[j][1]);
        red2(p + 8 * MLP_H, c[j][2], c[j][3]);
      }
    }
    __syncthreads();   // dz1
    // the other gradients in FP32: a thread takes column i and a quarter of
    // the inputs (W1) and of the outputs (W3)
    {
      const int i = tid & (MLP_H - 1), q = tid >> 7;
      float gw1[4] = {0.f, 0.f, 0.f, 0.f}, gw3[2] = {0.f, 0.f}, s = 0.f;
#pragma unroll 8
      for (int r = 0; r < kTile; r++) {
        const float dz = sb.dz1[r * LDZ + i];
        const float2 xa = __bfloat1622float2(*(const __nv_bfloat162 *)(sb.x + r * LDX + 4 * q));
        const float2 xb = __bfloat1622float2(*(const __nv_bfloat162 *)(sb.x + r * LDX + 4 * q + 2));
        gw1[0] += xa.x * dz;
        gw1[1] += xa.y * dz;
        gw1[2] += xb.x * dz;
        gw1[3] += xb.y * dz;
        const float a2 = __bfloat162float(sb.a2[r * LDH + i]);
        const float2 dy = *(const float2 *)(sb.y + r * MLP_OUTP + 2 * q);
        gw3[0] += a2 * dy.x;
        gw3[1] += a2 * dy.y;
        if (q == 0) s += dz;
        else if (q == 1) s += __bfloat162float(sb.dz2[r * LDH + i]);
      }
#pragma unroll
      for (int f = 0; f < 4; f++) atomicAdd(&grad[OW1 + (4 * q + f) * MLP_H + i], gw1[f]);
      red2(grad + OW3 + i * MLP_OUTP + 2 * q, gw3[0], 2 * q + 1 < MLP_OUT ? gw3[1] : 0.f);
      if (q == 0) atomicAdd(&grad[OB1 + i], s);
      else if (q == 1) atomicAdd(&grad[OB2 + i], s);
      if (q == 2 && i < MLP_OUTP) {
        float sy = 0.f;
        for (int r = 0; r < kTile; r++) sy += sb.y[r * MLP_OUTP + i];
        atomicAdd(&grad[OB3 + i], sy);
      }
    }
  }
}

// the BF16 copy of parameter i, [output][input]
__device__ inline void store_bf16(const Bf16Weights &W, int i, float v) {
  if (i < OB1) {
    const int k = (i - OW1) / MLP_H, c = (i - OW1) % MLP_H;
    W.w1t[c * MLP_IN + k] = __float2bfloat16(v);
  } else if (i >= OW2 && i < OB2) {
    const int k = (i - OW2) / MLP_H, c = (i - OW2) % MLP_H;
    W.w2t[c * MLP_H + k] = __float2bfloat16(v);
  } else if (i >= OW3 && i < OB3) {
    const int k = (i - OW3) / MLP_OUTP, c = (i - OW3) % MLP_OUTP;
    W.w3t[c * MLP_H + k] = __float2bfloat16(v);
  }
}

// Adam on the FP32 master weights, and their BF16 copies
__global__ void k_mlp_adam(float *blob, float *grad, float *m, float *v, Bf16Weights W, float lr, float b1, float b2,
                           float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NPARAM) return;
  const bool pad = (i >= OW3 && i < OB3 && (i - OW3) % MLP_OUTP >= MLP_OUT) || (i >= OB3 && i - OB3 >= MLP_OUT);
  const float gr = pad ? 0.f : grad[i];
  m[i] = b1 * m[i] + (1.f - b1) * gr;
  v[i] = b2 * v[i] + (1.f - b2) * gr * gr;
  if (!pad) {
    blob[i] -= lr * (m[i] / c1) / (sqrtf(v[i] / c2) + eps);
    store_bf16(W, i, blob[i]);
  }
  grad[i] = 0.f;
}

__global__ void k_mlp_to_bf16(const float *blob, Bf16Weights W) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < MLP_IN * MLP_H) {   // w1t[n][k] = W1[k][n]
    const int n = i / MLP_IN, k = i % MLP_IN;
    W.w1t[i] = __float2bfloat16(blob[OW1 + k * MLP_H + n]);
  }
  if (i < MLP_H * MLP_H) {
    const int n = i / MLP_H, k = i % MLP_H;
    W.w2t[i] = __float2bfloat16(blob[OW2 + k * MLP_H + n]);
  }
  if (i < MLP_OUTP * MLP_H) {
    const int n = i / MLP_H, k = i % MLP_H;
    W.w3t[i] = __float2bfloat16(blob[OW3 + k * MLP_OUTP + n]);
  }
}

size_t smem_forward() { return sizeof(SmemW); }
size_t smem_train() { return sizeof(SmemW) + sizeof(SmemTrain); }

int sm_count_mlp() {
  int dev = 0, n = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

}  // namespace

struct kgpu_mlp {
  float *blob = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
  Bf16Weights W{};
  double *dloss = nullptr;
  int *order = nullptr;
  int order_n = 0;
  long long step = 0;
};

static void launch_train(const kgpu_mlp &M, const float *X, const float *T, const int *order, int n, int batch) {
  const int blocks = (batch + kTile - 1) / kTile;
  if ((uintptr_t)X & 15)
    k_mlp_train<false><<<blocks, 32 * kTrainWarps, smem_train()>>>(M.blob, M.W, X, T, order, n, batch, M.grad, M.dloss);
  else
    k_mlp_train<true><<<blocks, 32 * kTrainWarps, smem_train()>>>(M.blob, M.W, X, T, order, n, batch, M.grad, M.dloss);
}

extern "C" int kgpu_mlp_blob_size(void) { return NBLOB; }

extern "C" int kgpu_mlp_create(kgpu_mlp **out, unsigned long long seed) {
  if (!out) return KGPU_EINVAL;
  kgpu_mlp *M = new kgpu_mlp();
  std::vector<float> h(NBLOB, 0.f);
  // He-style initialisation from a 64-bit linear congruential stream
  unsigned long long s = seed * 6364136223846793005ULL + 1442695040888963407ULL;
  auto unif = [&]() {
    s = s * 6364136223846793005ULL + 1442695040888963407ULL;
    return (double)(s >> 11) / 9007199254740992.0;
  };
  auto fill = [&](int off, int fan_in, int rows, int cols, int used_cols) {
    const double a = sqrt(6.0 / fan_in);
    for (int r = 0; r < rows; r++)
      for (int c = 0; c < cols; c++) h[off + r * cols + c] = c < used_cols ? (float)((2. * unif() - 1.) * a) : 0.f;
  };
  fill(OW1, MLP_IN, MLP_IN, MLP_H, MLP_H);
  fill(OW2, MLP_H, MLP_H, MLP_H, MLP_H);
  fill(OW3, MLP_H, MLP_H, MLP_OUTP, MLP_OUT);
  for (int o = 0; o < MLP_OUTP; o++) h[OSCALE + o] = 1.f;
  cudaError_t e = cudaSuccess;
  auto al = [&](void **p, size_t b) {
    if (e == cudaSuccess) e = cudaMalloc(p, b);
  };
  al((void **)&M->blob, NBLOB * 4);
  al((void **)&M->grad, NPARAM * 4);
  al((void **)&M->m, NPARAM * 4);
  al((void **)&M->v, NPARAM * 4);
  al((void **)&M->W.w1t, MLP_IN * MLP_H * 2);
  al((void **)&M->W.w2t, MLP_H * MLP_H * 2);
  al((void **)&M->W.w3t, MLP_OUTP * MLP_H * 2);
  al((void **)&M->dloss, sizeof(double));
  if (e == cudaSuccess) e = cudaMemcpy(M->blob, h.data(), NBLOB * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(M->grad, 0, NPARAM * 4);
  if (e == cudaSuccess) e = cudaMemset(M->m, 0, NPARAM * 4);
  if (e == cudaSuccess) e = cudaMemset(M->v, 0, NPARAM * 4);
  if (e == cudaSuccess) {
    k_mlp_to_bf16<<<(MLP_H * MLP_H + 255) / 256, 256>>>(M->blob, M->W);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_mlp_train<true>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem_train());
  if (e == cudaSuccess) e = cudaFuncSetAttribute(k_mlp_train<false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem_train());
  if (e != cudaSuccess) {
    kgpu_report_cuda("kgpu_mlp_create", e);
    delete M;
    return KGPU_ECUDA;
  }
  *out = M;
  return 0;
}

extern "C" int kgpu_mlp_destroy(kgpu_mlp *M) {
  if (!M) return KGPU_EINVAL;
  cudaFree(M->blob);
  cudaFree(M->grad);
  cudaFree(M->m);
  cudaFree(M->v);
  cudaFree(M->W.w1t);
  cudaFree(M->W.w2t);
  cudaFree(M->W.w3t);
  cudaFree(M->dloss);
  cudaFree(M->order);
  delete M;
  return 0;
}

extern "C" int kgpu_mlp_get(kgpu_mlp *M, float *blob) {
  if (!M || !blob) return KGPU_EINVAL;
  MCK(cudaMemcpy(blob, M->blob, NBLOB * 4, cudaMemcpyDeviceToHost));
  return 0;
}

extern "C" int kgpu_mlp_set(kgpu_mlp *M, const float *blob) {
  if (!M || !blob) return KGPU_EINVAL;
  MCK(cudaMemcpy(M->blob, blob, NBLOB * 4, cudaMemcpyHostToDevice));
  k_mlp_to_bf16<<<(MLP_H * MLP_H + 255) / 256, 256>>>(M->blob, M->W);
  MCK(cudaGetLastError());
  MCK(cudaDeviceSynchronize());
  return 0;
}

extern "C" int kgpu_mlp_forward(kgpu_mlp *M, const float *X, int n, float *Y, void *stream) {
  if (!M || n < 0 || (n > 0 && (!X || !Y))) return KGPU_EINVAL;
  if (n == 0) return 0;
  const int tiles = (n + 15) / 16;
  int blocks = (tiles + kInferWarps - 1) / kInferWarps;
  const int cap = sm_count_mlp();
  if (blocks > cap) blocks = cap;
  cudaStream_t st = (cudaStream_t)stream;
  if (((uintptr_t)X | ((uintptr_t)Y << 1)) & 15)
    k_mlp_forward<false><<<blocks, 32 * kInferWarps, smem_forward(), st>>>(M->blob, M->W, X, n, Y);
  else
    k_mlp_forward<true><<<blocks, 32 * kInferWarps, smem_forward(), st>>>(M->blob, M->W, X, n, Y);
  MCK(cudaGetLastError());
  return 0;
}

// Gradient of the batch loss (mean over the n samples, targets
// standardised with the blob's mean and scale) at the current weights,
// without an update: for checking the backward pass.
extern "C" int kgpu_mlp_gradient(kgpu_mlp *M, const float *X, const float *T, int n, float *grad_host,
                                 double *loss) {
  if (!M || n <= 0 || !X || !T || !grad_host || !loss) return KGPU_EINVAL;
  int *order = nullptr;
  MCK(cudaMalloc(&order, (size_t)n * 4));
  std::vector<int> h(n);
  for (int i = 0; i < n; i++) h[i] = i;
  cudaError_t e = cudaMemcpy(order, h.data(), (size_t)n * 4, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(M->grad, 0, NPARAM * 4);
  if (e == cudaSuccess) e = cudaMemset(M->dloss, 0, sizeof(double));
  if (e == cudaSuccess) {
    launch_train(*M, X, T, order, n, n);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaMemcpy(grad_host, M->grad, NPARAM * 4, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(loss, M->dloss, sizeof(double), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemset(M->grad, 0, NPARAM * 4);
  cudaFree(order);
  if (e != cudaSuccess) return kgpu_report_cuda("kgpu_mlp_gradient", e);
  return 0;
}

// One epoch of Adam over n samples (X [n][16], raw targets T [n][5], both
// device pointers), shuffled with `seed`, in batches of `batch`.  The mean
// batch loss goes to *mean_loss.
extern "C" int kgpu_mlp_train_epoch(kgpu_mlp *M, const float *X, const float *T, int n, int batch, float lr,
                                    unsigned long long seed, double *mean_loss) {
  if (!M || n <= 0 || batch <= 0 || !X || !T) return KGPU_EINVAL;
  if (M->order_n < n) {
    cudaFree(M->order);
    M->order = nullptr;
    MCK(cudaMalloc(&M->order, (size_t)n * 4));
    M->order_n = n;
  }
  std::vector<int> h(n);
  for (int i = 0; i < n; i++) h[i] = i;
  unsigned long long s = seed ^ 0x9e3779b97f4a7c15ULL;
  for (int i = n - 1; i > 0; i--) {
    s = s * 6364136223846793005ULL + 1442695040888963407ULL;
    const int j = (int)((unsigned)(s >> 33) % (unsigned)(i + 1));   // both below 2^31
    const int tmp = h[i];
    h[i] = h[j];
    h[j] = tmp;
  }
  MCK(cudaMemcpy(M->order, h.data(), (size_t)n * 4, cudaMemcpyHostToDevice));
  MCK(cudaMemset(M->dloss, 0, sizeof(double)));
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  int nb = 0;
  for (int b0 = 0; b0 + batch <= n; b0 += batch, nb++) {
    launch_train(*M, X, T, M->order + b0, n, batch);
    MCK(cudaGetLastError());
    M->step++;
    const float c1 = 1.f - powf(b1, (float)M->step), c2 = 1.f - powf(b2, (float)M->step);
    k_mlp_adam<<<(NPARAM + 127) / 128, 128>>>(M->blob, M->grad, M->m, M->v, M->W, lr, b1, b2, eps, c1, c2);
    MCK(cudaGetLastError());
  }
  double l = 0.;
  MCK(cudaMemcpy(&l, M->dloss, sizeof(double), cudaMemcpyDeviceToHost));
  if (mean_loss) *mean_loss = nb ? l / nb : 0.;
  return 0;
}
