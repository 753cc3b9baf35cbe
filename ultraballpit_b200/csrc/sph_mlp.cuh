// sph_mlp.cuh - device pieces of the closure network (16 -> 64 -> 64 -> 4,
// SiLU): BF16 tensor-core tiles (mma.sync.m16n8k16, FP32 accumulation) over
// 16 samples per warp, operands staged in shared memory.
#pragma once
#include <cstdint>

#include <cuda_bf16.h>

namespace sphmlp {

constexpr int kIn = 16, kHid = 64, kOut = 4;
constexpr int kOffW1 = 0, kOffB1 = 1024, kOffW2 = 1088, kOffB2 = 5184, kOffW3 = 5248, kOffB3 = 5504;
constexpr int kParams = 5508;
constexpr int kParamBias = 132;   // b1 | b2 | b3 in shared memory
constexpr int kBf16Count = 5376;  // W1 | W2 | W3 in BF16

// Index of master parameter i in the BF16 weight array, -1 for biases.
__host__ __device__ inline int bf16_index(int i) {
  if (i < kOffB1) return i;
  if (i >= kOffW2 && i < kOffB2) return 1024 + (i - kOffW2);
  if (i >= kOffW3 && i < kOffB3) return 5120 + (i - kOffW3);
  return -1;
}

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
  float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

// C(16x8) += A(16x16) B(16x8) on the tensor cores, A(m,k) = A[m*sam + k*sak],
// B(k,n) = B[k*sbk + n*sbn] (BF16 in shared memory). Fragment layout of the
// PTX ISA for mma.m16n8k16: g = lane/4, t = lane%4; A rows g and g+8, columns
// 2t, 2t+1 (+8); B rows 2t, 2t+1 (+8), column g; C rows g, g+8, columns 2t, 2t+1.
__device__ __forceinline__ void mma_tile(const __nv_bfloat16* A, int sam, int sak, const __nv_bfloat16* B,
                                         int sbk, int sbn, float c[4], int lane) {
  int g = lane >> 2, t = lane & 3;
  int k0 = 2 * t;
  uint32_t a0 = pack2(A[g * sam + k0 * sak], A[g * sam + (k0 + 1) * sak]);
  uint32_t a1 = pack2(A[(g + 8) * sam + k0 * sak], A[(g + 8) * sam + (k0 + 1) * sak]);
  uint32_t a2 = pack2(A[g * sam + (k0 + 8) * sak], A[g * sam + (k0 + 9) * sak]);
  uint32_t a3 = pack2(A[(g + 8) * sam + (k0 + 8) * sak], A[(g + 8) * sam + (k0 + 9) * sak]);
  uint32_t b0 = pack2(B[k0 * sbk + g * sbn], B[(k0 + 1) * sbk + g * sbn]);
  uint32_t b1 = pack2(B[(k0 + 8) * sbk + g * sbn], B[(k0 + 9) * sbk + g * sbn]);
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Block-wide copy of the BF16 weights (W3 padded with zero rows to 16) and
// FP32 biases into shared memory.
__device__ __forceinline__ void load_weights_smem(const __nv_bfloat16* __restrict__ wb, const float* __restrict__ w,
                                                  __nv_bfloat16* w1, __nv_bfloat16* w2, __nv_bfloat16* w3,
                                                  float* b) {
  for (int i = threadIdx.x; i < 1024; i += blockDim.x) w1[i] = wb[i];
  for (int i = threadIdx.x; i < 4096; i += blockDim.x) w2[i] = wb[1024 + i];
  for (int i = threadIdx.x; i < 1024; i += blockDim.x) w3[i] = i < 256 ? wb[5120 + i] : __float2bfloat16_rn(0.0f);
  for (int i = threadIdx.x; i < kParamBias; i += blockDim.x)
    b[i] = i < 64 ? w[kOffB1 + i] : (i < 128 ? w[kOffB2 + i - 64] : w[kOffB3 + i - 128]);
}

// Forward pass of one 16-sample tile: x[16][16] (BF16) -> z1/h1, z2/h2
// ([16][64], FP32 pre-activations and BF16 activations) -> y[16][4] (FP32).
__device__ __forceinline__ void forward_tile(const __nv_bfloat16* x, const __nv_bfloat16* w1,
                                             const __nv_bfloat16* w2, const __nv_bfloat16* w3, const float* b,
                                             float* z1, __nv_bfloat16* h1, float* z2, __nv_bfloat16* h2,
                                             float* y, int lane) {
  int g = lane >> 2, t = lane & 3;
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    mma_tile(x, 16, 1, w1 + nt * 8 * 16, 1, 16, c, lane);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      int r = g + (e >> 1) * 8, col = nt * 8 + 2 * t + (e & 1);
      float z = c[e] + b[col];
      z1[r * 64 + col] = z;
      h1[r * 64 + col] = __float2bfloat16_rn(silu(z));
    }
  }
  __syncwarp();
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) mma_tile(h1 + kt * 16, 64, 1, w2 + nt * 8 * 64 + kt * 16, 1, 64, c, lane);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      int r = g + (e >> 1) * 8, col = nt * 8 + 2 * t + (e & 1);
      float z = c[e] + b[64 + col];
      z2[r * 64 + col] = z;
      h2[r * 64 + col] = __float2bfloat16_rn(silu(z));
    }
  }
  __syncwarp();
  {
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) mma_tile(h2 + kt * 16, 64, 1, w3 + kt * 16, 1, 64, c, lane);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      int r = g + (e >> 1) * 8, col = 2 * t + (e & 1);
      if (col < 4) y[r * 4 + col] = c[e] + b[128 + col];
    }
  }
  __syncwarp();
}

// One m16n8k16 step with the operands already in registers.
__device__ __forceinline__ void mma_regs(float c[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                         uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// The weights in the order the forward pass's lanes take them: per lane 22
// quads of words, 4 of W1 (two n-tiles' B fragments each), 16 of W2 (two
// k-tiles' each) and 2 of W3 (two k-tiles' each; its columns 4..7 are zero
// rows), quad q of lane l at word (q * 32 + l) * 4. A quad is one coalesced
// load; a word at a time from the row-major matrices is 72 loads of eight
// lines each (density pass of a 42k-particle tank, two lanes a particle: 127
// -> 123 us; 88 -> 86 at 24k).
constexpr int kFragQuads = 22, kFragWords = kFragQuads * 32 * 4;

// Word `at` of that array as the index of its lower BF16 in W1 | W2 | W3
// (the upper one follows it), -1 for a zero.
__host__ __device__ inline int frag_index(int at) {
  const int e = at & 3, lane = (at >> 2) & 31, q = at >> 7;
  const int g = lane >> 2, k0 = 2 * (lane & 3) + (e & 1) * 8, odd = e >> 1;
  if (q < 4) return ((2 * q + odd) * 8 + g) * 16 + k0;
  if (q < 20) return 1024 + (((q - 4) >> 1) * 8 + g) * 64 + (((q - 4) & 1) * 2 + odd) * 16 + k0;
  return g < 4 ? 5120 + g * 64 + ((q - 20) * 2 + odd) * 16 + k0 : -1;
}

// The forward pass of forward_tile with the activations kept in registers:
// the C fragment of two adjacent n-tiles of one layer is the A fragment of
// one k-tile of the next (rows g, g+8; columns 2t, 2t+1 and 2t+8, 2t+9), so
// only the input tile x[16][16] (BF16, shared) and the output y[16][4]
// (FP32, shared) leave the registers. The weights come from global memory in
// the lanes' order (wq, frag_index; the master FP32 parameters wf for the
// biases) and stay in L1. Same instructions, operands and rounding points as
// forward_tile, so the outputs are identical.
__device__ __forceinline__ void forward_tile_regs(const __nv_bfloat16* x, const uint4* __restrict__ wq,
                                                  const float* __restrict__ wf, float* y, int lane) {
  int g = lane >> 2, t = lane & 3;
  int k0 = 2 * t;
  uint32_t xa0 = pack2(x[g * 16 + k0], x[g * 16 + k0 + 1]);
  uint32_t xa1 = pack2(x[(g + 8) * 16 + k0], x[(g + 8) * 16 + k0 + 1]);
  uint32_t xa2 = pack2(x[g * 16 + k0 + 8], x[g * 16 + k0 + 9]);
  uint32_t xa3 = pack2(x[(g + 8) * 16 + k0 + 8], x[(g + 8) * 16 + k0 + 9]);
  wq += lane;
  uint32_t h1[16], h2[16];
  // an n-tile's sums with their biases through the SiLU, as half an A fragment
  auto activate = [&](const float c[4], int off, int nt, uint32_t* h) {
    const float2 b = __ldg(reinterpret_cast<const float2*>(wf + off + nt * 8 + k0));
    h[(nt >> 1) * 4 + (nt & 1) * 2] = pack2(__float2bfloat16_rn(silu(c[0] + b.x)), __float2bfloat16_rn(silu(c[1] + b.y)));
    h[(nt >> 1) * 4 + (nt & 1) * 2 + 1] =
        pack2(__float2bfloat16_rn(silu(c[2] + b.x)), __float2bfloat16_rn(silu(c[3] + b.y)));
  };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint4 w = __ldg(wq + q * 32);
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f}, d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    mma_regs(c, xa0, xa1, xa2, xa3, w.x, w.y);
    mma_regs(d, xa0, xa1, xa2, xa3, w.z, w.w);
    activate(c, kOffB1, 2 * q, h1);
    activate(d, kOffB1, 2 * q + 1, h1);
  }
#pragma unroll
  for (int nt = 0; nt < 8; ++nt) {
    const uint4 u = __ldg(wq + (4 + 2 * nt) * 32), v = __ldg(wq + (5 + 2 * nt) * 32);
    float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    mma_regs(c, h1[0], h1[1], h1[2], h1[3], u.x, u.y);
    mma_regs(c, h1[4], h1[5], h1[6], h1[7], u.z, u.w);
    mma_regs(c, h1[8], h1[9], h1[10], h1[11], v.x, v.y);
    mma_regs(c, h1[12], h1[13], h1[14], h1[15], v.z, v.w);
    activate(c, kOffB2, nt, h2);
  }
  const uint4 u = __ldg(wq + 20 * 32), v = __ldg(wq + 21 * 32);
  float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
  mma_regs(c, h2[0], h2[1], h2[2], h2[3], u.x, u.y);
  mma_regs(c, h2[4], h2[5], h2[6], h2[7], u.z, u.w);
  mma_regs(c, h2[8], h2[9], h2[10], h2[11], v.x, v.y);
  mma_regs(c, h2[12], h2[13], h2[14], h2[15], v.z, v.w);
  if (t < 2) {
    float bl = __ldg(&wf[kOffB3 + k0]), bh = __ldg(&wf[kOffB3 + k0 + 1]);
    y[g * 4 + k0] = c[0] + bl;
    y[g * 4 + k0 + 1] = c[1] + bh;
    y[(g + 8) * 4 + k0] = c[2] + bl;
    y[(g + 8) * 4 + k0 + 1] = c[3] + bh;
  }
}

// Sum of a C-fragment column over the 16 rows (lanes with equal t), in lanes
// 0..3 (columns 2t, 2t+1).
__device__ __forceinline__ void colsum(float c[4], float& s0, float& s1) {
  s0 = c[0] + c[2];
  s1 = c[1] + c[3];
#pragma unroll
  for (int o = 4; o < 32; o <<= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
  }
}

// Fragments by ldmatrix: four (two) 8x8 BF16 matrices of a row-major array
// in shared memory, each lane naming the 16-byte row it provides. Rows are
// padded so that eight of them fall into distinct banks.
constexpr int kPad16 = 24, kPad64 = 72;  // row strides of 16- and 64-wide arrays
__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldm4(uint32_t r[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldm4t(uint32_t r[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldm2(uint32_t r[2], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"(smem_addr(p)));
}
__device__ __forceinline__ void ldm2t(uint32_t r[2], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1]) : "r"(smem_addr(p)));
}
// A(16x16) of M[row][col] at (0, col): rows the samples
__device__ __forceinline__ void frag_a(uint32_t a[4], const __nv_bfloat16* M, int ld, int col, int lane) {
  ldm4(a, M + (lane & 15) * ld + col + (lane >> 4) * 8);
}
// A = M^T for M[k][m] at column m (k the 16 samples)
__device__ __forceinline__ void frag_at(uint32_t a[4], const __nv_bfloat16* M, int ld, int m, int lane) {
  ldm4t(a, M + ((lane & 7) + ((lane >> 4) & 1) * 8) * ld + m + ((lane >> 3) & 1) * 8);
}
// B(16x8) of W[n][k] at (n, k): the layer's weights
__device__ __forceinline__ void frag_b(uint32_t b[2], const __nv_bfloat16* W, int ld, int n, int k, int lane) {
  ldm2(b, W + (n + (lane & 7)) * ld + k + ((lane >> 3) & 1) * 8);
}
// B of M[k][n] at (k, n)
__device__ __forceinline__ void frag_bt(uint32_t b[2], const __nv_bfloat16* M, int ld, int k, int n, int lane) {
  ldm2t(b, M + (k + (lane & 15)) * ld + n);
}
__device__ __forceinline__ void mma_frag(float c[4], const uint32_t a[4], const uint32_t b[2]) {
  mma_regs(c, a[0], a[1], a[2], a[3], b[0], b[1]);
}

}  // namespace sphmlp
