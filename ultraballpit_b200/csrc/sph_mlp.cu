// sph_mlp.cu - the learned near-wall closure network: 16 -> 64 -> 64 -> 4,
// SiLU, trained and evaluated with BF16 operands on the tensor cores
// (mma.sync m16n8k16, FP32 accumulation). FP32 master weights and Adam state;
// BF16 copies feed the matrix products. No reference counterpart.
//
// Parameter layout (5,508 floats): W1[64][16], b1[64], W2[64][64], b2[64],
// W3[4][64], b3[4]; W[out][in], so y = W x + b.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "sph_cuda.h"
#include "sph_mlp.cuh"

using namespace sphmlp;

namespace sph {
__attribute__((visibility("hidden"))) cudaMemPool_t device_pool(int dev);  // sph_api.cu: null if there is none
}

struct SphMlp {
  int dev = 0;
  cudaStream_t st = nullptr;
  float* w = nullptr;        // FP32 master parameters
  float* m = nullptr;        // Adam first moment
  float* v = nullptr;        // Adam second moment
  __nv_bfloat16* wb = nullptr;  // BF16 copies of W1, W2, W3 (biases stay FP32)
  float* grad = nullptr;     // summed gradient of a mini-batch
  float* part = nullptr;     // gradient partials, a row per CTA
  int part_rows = 0;
  float* loss = nullptr;     // loss per tile of an epoch
  size_t loss_tiles = 0;
  // samples, targets (or outputs) and permutation on the device; these, the
  // partials and the losses are pieces of `work`, kept from call to call up to
  // kKeep bytes. `mu` is held by the call that uses them.
  std::mutex mu;
  unsigned char* work = nullptr;
  size_t work_bytes = 0;
  bool work_pooled = false;  // from device_pool
  float *dx = nullptr, *dt = nullptr;
  uint32_t* dp = nullptr;
  size_t cap = 0;  // samples they hold
  int64_t step = 0;
  int sms = 148;             // SMs of the device (queried at creation)
  std::vector<void*> allocs;
};

namespace {

template <class T>
cudaError_t mal(SphMlp* h, T** p, size_t n) {
  cudaError_t e = cudaMalloc((void**)p, std::max<size_t>(n, 1) * sizeof(T));
  if (e == cudaSuccess) h->allocs.push_back(*p);
  return e;
}

int status(cudaError_t e) {
  if (e == cudaSuccess) return SPH_OK;
  return e == cudaErrorMemoryAllocation ? SPH_ERR_OOM : SPH_ERR_CUDA;
}

uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

double uniform01(uint64_t& s) { return (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0); }

constexpr int kWarps = 4;
constexpr int kCtaSamples = kWarps * 16;  // samples whose gradients are added first (a group of four tiles)

// Shared memory of the forward kernel: weights, and a tile per warp.
struct WarpSmem {
  __nv_bfloat16 x[16 * 16];
  float z1[16 * 64];
  __nv_bfloat16 h1[16 * 64];
  float z2[16 * 64];
  __nv_bfloat16 h2[16 * 64];
  float y[16 * 4];
};
struct CtaSmem {
  __nv_bfloat16 w1[64 * 16];
  __nv_bfloat16 w2[64 * 64];
  __nv_bfloat16 w3[16 * 64];   // W3 padded to 16 output rows
  float b[kParamBias];          // b1, b2, b3
  WarpSmem wp[kWarps];
};

// Shared memory of the training kernel: weights and one tile of 16 samples.
struct __align__(16) TrainSmem {
  __nv_bfloat16 w1[64 * kPad16], w2[64 * kPad64], w3[16 * kPad64];
  __nv_bfloat16 x[16 * kPad16], dy[16 * kPad16];
  __nv_bfloat16 h1[16 * kPad64], h2[16 * kPad64], dz2[16 * kPad64], dz1[16 * kPad64];
  float b[kParamBias];
  float y[16 * 4];
};

// Forward and backward of the closure network on BF16 tensor-core tiles of 16
// samples. A CTA's four warps share a tile, two 8-column blocks of each layer
// each, with fragments by ldmatrix; the pre-activations and the gradients stay
// in the registers of the warp that made them. `tiles` tiles per CTA, their
// gradients added in order and written to the CTA's row of `part` (no
// atomics): four for a large batch, one where four would leave most SMs
// without a CTA (k_adam then adds the rows in the same groups of four). A
// mini-batch of 1024 is bound by the chain of one tile and by the two launches:
// an epoch of 49 took 3890 us with a warp per tile, fragments gathered 2 bytes
// at a time, gradients in shared memory and a read of the loss after every
// mini-batch, and takes 1160 us here (16.5 us a mini-batch).
__global__ void __launch_bounds__(kWarps * 32)
k_mlp_train(const __nv_bfloat16* __restrict__ wb, const float* __restrict__ w, const float* __restrict__ x,
            const float* __restrict__ t, const uint32_t* __restrict__ perm, int batch_lo, int batch_n, int tiles,
            float* __restrict__ part, float* __restrict__ loss_part) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrainSmem& S = *reinterpret_cast<TrainSmem*>(smem_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, q = lane & 3;
  {
    const uint4* src = reinterpret_cast<const uint4*>(wb);  // eight weights each
    for (int i = tid; i < 128; i += kWarps * 32)
      *reinterpret_cast<uint4*>(&S.w1[(i >> 1) * kPad16 + (i & 1) * 8]) = src[i];
    for (int i = tid; i < 512; i += kWarps * 32)
      *reinterpret_cast<uint4*>(&S.w2[(i >> 3) * kPad64 + (i & 7) * 8]) = src[128 + i];
    for (int i = tid; i < 128; i += kWarps * 32)  // rows 4..15 are padding
      *reinterpret_cast<uint4*>(&S.w3[(i >> 3) * kPad64 + (i & 7) * 8]) = i < 32 ? src[640 + i] : make_uint4(0u, 0u, 0u, 0u);
    for (int i = tid; i < kParamBias; i += kWarps * 32)
      S.b[i] = i < 64 ? w[kOffB1 + i] : (i < 128 ? w[kOffB2 + i - 64] : w[kOffB3 + i - 128]);
  }
  // the sums over the CTA's tiles, in fragment layout (bias sums in lanes 0..3)
  float gw1[2][4] = {}, gw2[8][4] = {}, gw3[2][4] = {}, gb1[2][2] = {}, gb2[2][2] = {}, gb3 = 0.0f;
  const float scale = 2.0f / (float)(batch_n * kOut);
  for (int tile = 0; tile < tiles; ++tile) {
    const int base = (blockIdx.x * tiles + tile) * 16;  // within the mini-batch
    if (base >= batch_n) break;
    __syncthreads();  // the last tile's reads are done, the weights are in
    for (int i = tid; i < 256; i += kWarps * 32) {  // rows past the batch are zero with zero target weight
      const int r = i >> 4, c = i & 15, j = base + r;
      S.x[r * kPad16 + c] = __float2bfloat16_rn(j < batch_n ? x[(size_t)perm[batch_lo + j] * kIn + c] : 0.0f);
    }
    __syncthreads();
    float z1[2][4], z2[2][4];
    uint32_t a[4], b[2];
    frag_a(a, S.x, kPad16, 0, lane);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int nt = warp * 2 + u;
      float c[4] = {};
      frag_b(b, S.w1, kPad16, nt * 8, 0, lane);
      mma_frag(c, a, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = g + (e >> 1) * 8, col = nt * 8 + 2 * q + (e & 1);
        z1[u][e] = c[e] + S.b[col];
        S.h1[r * kPad64 + col] = __float2bfloat16_rn(silu(z1[u][e]));
      }
    }
    __syncthreads();
    {
      float c[2][4] = {};
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        frag_a(a, S.h1, kPad64, kt * 16, lane);
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          frag_b(b, S.w2, kPad64, (warp * 2 + u) * 8, kt * 16, lane);
          mma_frag(c[u], a, b);
        }
      }
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int r = g + (e >> 1) * 8, col = (warp * 2 + u) * 8 + 2 * q + (e & 1);
          z2[u][e] = c[u][e] + S.b[64 + col];
          S.h2[r * kPad64 + col] = __float2bfloat16_rn(silu(z2[u][e]));
        }
    }
    __syncthreads();
    if (warp == 0) {  // the output, the loss and dL/dy
      float c[4] = {};
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        frag_a(a, S.h2, kPad64, kt * 16, lane);
        frag_b(b, S.w3, kPad64, 0, kt * 16, lane);
        mma_frag(c, a, b);
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = g + (e >> 1) * 8, col = 2 * q + (e & 1);
        if (col < 4) S.y[r * 4 + col] = c[e] + S.b[128 + col];
      }
      __syncwarp();
      // mean squared error over batch_n x 4 outputs
      float lsum = 0.0f;
      for (int i = lane; i < 256; i += 32) {
        const int r = i >> 4, c4 = i & 15, j = base + r;
        float d = 0.0f;
        if (j < batch_n && c4 < kOut) {
          const float err = S.y[r * 4 + c4] - t[(size_t)perm[batch_lo + j] * kOut + c4];
          lsum += err * err;
          d = scale * err;
        }
        S.dy[r * kPad16 + c4] = __float2bfloat16_rn(d);
      }
      for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
      if (lane == 0) loss_part[base >> 4] = lsum;
    }
    __syncthreads();
    // dW3[o][k] = sum_m dy[m][o] h2[m][k] (rows o >= 4 are padding); dz2 = (dy W3) silu'(z2)
    uint32_t at[4];
    frag_at(at, S.dy, kPad16, 0, lane);
    frag_a(a, S.dy, kPad16, 0, lane);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int nt = warp * 2 + u;
      float c[4] = {};
      frag_bt(b, S.h2, kPad64, 0, nt * 8, lane);
      mma_frag(c, at, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) gw3[u][e] += c[e];
      float d[4] = {};
      frag_bt(b, S.w3, kPad64, 0, nt * 8, lane);
      mma_frag(d, a, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = g + (e >> 1) * 8, col = nt * 8 + 2 * q + (e & 1);
        d[e] *= silu_grad(z2[u][e]);
        S.dz2[r * kPad64 + col] = __float2bfloat16_rn(d[e]);
      }
      float s0, s1;
      colsum(d, s0, s1);
      gb2[u][0] += s0;
      gb2[u][1] += s1;
    }
    if (warp == 0 && lane < 4) {
      float s = 0.0f;
      for (int m = 0; m < 16; ++m) s += __bfloat162float(S.dy[m * kPad16 + lane]);
      gb3 += s;
    }
    __syncthreads();
    // dW2[o][k] = sum_m dz2[m][o] h1[m][k]: warp w has the columns k of its two blocks
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) {
      frag_at(at, S.dz2, kPad64, mt * 16, lane);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float c[4] = {};
        frag_bt(b, S.h1, kPad64, 0, (warp * 2 + u) * 8, lane);
        mma_frag(c, at, b);
#pragma unroll
        for (int e = 0; e < 4; ++e) gw2[mt * 2 + u][e] += c[e];
      }
    }
    // dz1 = (dz2 W2) silu'(z1)
    float d1[2][4] = {};
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) {
      frag_a(a, S.dz2, kPad64, kt * 16, lane);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        frag_bt(b, S.w2, kPad64, kt * 16, (warp * 2 + u) * 8, lane);
        mma_frag(d1[u], a, b);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int r = g + (e >> 1) * 8, col = (warp * 2 + u) * 8 + 2 * q + (e & 1);
        d1[u][e] *= silu_grad(z1[u][e]);
        S.dz1[r * kPad64 + col] = __float2bfloat16_rn(d1[u][e]);
      }
      float s0, s1;
      colsum(d1[u], s0, s1);
      gb1[u][0] += s0;
      gb1[u][1] += s1;
    }
    __syncthreads();
    // dW1[o][k] = sum_m dz1[m][o] x[m][k]: warp w has the rows o of its 16
    frag_at(at, S.dz1, kPad64, warp * 16, lane);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      float c[4] = {};
      frag_bt(b, S.x, kPad16, 0, u * 8, lane);
      mma_frag(c, at, b);
#pragma unroll
      for (int e = 0; e < 4; ++e) gw1[u][e] += c[e];
    }
  }
  float* out = part + (size_t)blockIdx.x * kParams;
  auto put = [&](int off, int row, int ld, int col, const float c[4]) {  // rows row, row + 8; columns col, col + 1
    *reinterpret_cast<float2*>(out + off + row * ld + col) = make_float2(c[0], c[1]);
    *reinterpret_cast<float2*>(out + off + (row + 8) * ld + col) = make_float2(c[2], c[3]);
  };
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int col = (warp * 2 + u) * 8 + 2 * q;
    put(kOffW1, warp * 16 + g, 16, u * 8 + 2 * q, gw1[u]);
#pragma unroll
    for (int mt = 0; mt < 4; ++mt) put(kOffW2, mt * 16 + g, 64, col, gw2[mt * 2 + u]);
    if (g < 4) *reinterpret_cast<float2*>(out + kOffW3 + g * 64 + col) = make_float2(gw3[u][0], gw3[u][1]);
    if (lane < 4) {
      out[kOffB1 + col] = gb1[u][0];
      out[kOffB1 + col + 1] = gb1[u][1];
      out[kOffB2 + col] = gb2[u][0];
      out[kOffB2 + col + 1] = gb2[u][1];
    }
  }
  if (warp == 0 && lane < 4) out[kOffB3 + lane] = gb3;
}

// Sum the rows of partials in order, `group` of them first (the groups of four
// tiles that a CTA adds when it has four), then one Adam step (bias-corrected)
// on the FP32 masters and refresh of the BF16 copies. Bound by the latency of
// the rows' loads, sixteen of which are in flight. ONE: group is 1, for the
// many rows of a large batch (50,000 samples in batches of 20,000: 493 us an
// epoch with a load at a time, 236 so).
template <bool ONE>
__global__ void k_adam(int rows, int group, const float* __restrict__ part, float* __restrict__ grad,
                       float* __restrict__ w, float* __restrict__ m, float* __restrict__ v,
                       __nv_bfloat16* __restrict__ wb, float lr, float b1, float b2, float eps, float c1, float c2,
                       int apply) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  float g = 0.0f;
  int c = 0;
  if (!ONE && group == 4) {
    const float* p = part + i;
    for (; c + 15 < rows; c += 16, p += 16 * (size_t)kParams) {  // sixteen rows' loads in flight
      float r[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) r[u] = p[u * (size_t)kParams];
#pragma unroll
      for (int u = 0; u < 16; u += 4) g += ((r[u] + r[u + 1]) + r[u + 2]) + r[u + 3];
    }
  }
  if (ONE) {
    const float* p = part + i;
    for (; c + 15 < rows; c += 16, p += 16 * (size_t)kParams) {
      float r[16];
#pragma unroll
      for (int u = 0; u < 16; ++u) r[u] = p[u * (size_t)kParams];
#pragma unroll
      for (int u = 0; u < 16; ++u) g += r[u];
    }
  }
  for (; c < rows; c += group) {
    float a = 0.0f;
    for (int u = c; u < min(c + group, rows); ++u) a += part[(size_t)u * kParams + i];
    g += a;
  }
  grad[i] = g;
  if (!apply) return;
  float mi = b1 * m[i] + (1.0f - b1) * g;
  float vi = b2 * v[i] + (1.0f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  float mh = mi / c1, vh = vi / c2;
  float wi = w[i] - lr * mh / (sqrtf(vh) + eps);
  w[i] = wi;
  int bi = bf16_index(i);
  if (bi >= 0) wb[bi] = __float2bfloat16_rn(wi);
}

__global__ void k_refresh_bf16(const float* __restrict__ w, __nv_bfloat16* __restrict__ wb) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  int bi = bf16_index(i);
  if (bi >= 0) wb[bi] = __float2bfloat16_rn(w[i]);
}

__global__ void __launch_bounds__(kWarps * 32)
k_mlp_forward(const __nv_bfloat16* __restrict__ wb, const float* __restrict__ w, const float* __restrict__ x,
              int n, float* __restrict__ y) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CtaSmem& S = *reinterpret_cast<CtaSmem*>(smem_raw);
  int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  load_weights_smem(wb, w, S.w1, S.w2, S.w3, S.b);
  __syncthreads();
  WarpSmem& W = S.wp[warp];
  for (int base = (blockIdx.x * kWarps + warp) * 16; base < n; base += gridDim.x * kWarps * 16) {
    for (int q = lane; q < 16 * 16; q += 32) {
      int r = q >> 4, c = q & 15;
      W.x[q] = __float2bfloat16_rn(base + r < n ? x[(size_t)(base + r) * kIn + c] : 0.0f);
    }
    __syncwarp();
    forward_tile(W.x, S.w1, S.w2, S.w3, S.b, W.z1, W.h1, W.z2, W.h2, W.y, lane);
    for (int q = lane; q < 16 * 4; q += 32) {
      int r = q >> 2;
      if (base + r < n) y[(size_t)(base + r) * kOut + (q & 3)] = W.y[q];
    }
    __syncwarp();
  }
}

constexpr size_t kKeep = (size_t)64 << 20;

void free_work(SphMlp* h) {
  if (h->work) {
    if (h->work_pooled) cudaFreeAsync(h->work, h->st);
    else cudaFree(h->work);
  }
  h->work = nullptr;
  h->dx = h->dt = h->part = h->loss = nullptr;
  h->dp = nullptr;
  h->work_bytes = h->cap = h->loss_tiles = 0;
  h->part_rows = 0;
}

// Room for n samples, `rows` of partials and the losses of `tiles` tiles, in one
// allocation: allocations and frees wait for the device, and three a call
// were a third of a short training run (a net's first epoch of 50,000 samples:
// 2.5 to 7.8 ms with five that it kept, 1.7 with this one; later ones 1.2).
cudaError_t ensure_work(SphMlp* h, size_t n, int rows, size_t tiles) {
  if (n <= h->cap && rows <= h->part_rows && tiles <= h->loss_tiles) return cudaSuccess;
  n = std::max(n, h->cap);
  rows = std::max(rows, h->part_rows);
  tiles = std::max(tiles, h->loss_tiles);
  free_work(h);
  size_t bytes = 0;
  auto piece = [&](size_t words) {
    const size_t at = bytes;
    bytes += (words * 4 + 255) / 256 * 256;
    return at;
  };
  const size_t x = piece(n * kIn), t = piece(n * kOut), p = piece(n), part = piece((size_t)rows * kParams),
               loss = piece(tiles);
  // What a net keeps comes from the library's pool: mapping 2 MB and more anew
  // takes 0.5 ms (a net created for one gradient of 2,400 samples: 1.30 ms, 0.81
  // from the pool); less than that has room in what the process has mapped.
  const cudaMemPool_t pool = bytes > (1u << 20) && bytes <= kKeep ? sph::device_pool(h->dev) : nullptr;
  h->work_pooled = pool != nullptr;
  const cudaError_t e = pool ? cudaMallocFromPoolAsync((void**)&h->work, bytes, pool, h->st)
                             : cudaMalloc((void**)&h->work, bytes);
  if (e != cudaSuccess) {
    h->work = nullptr;
    return e;
  }
  h->dx = reinterpret_cast<float*>(h->work + x);
  h->dt = reinterpret_cast<float*>(h->work + t);
  h->dp = reinterpret_cast<uint32_t*>(h->work + p);
  h->part = reinterpret_cast<float*>(h->work + part);
  h->loss = reinterpret_cast<float*>(h->work + loss);
  h->work_bytes = bytes;
  h->cap = n;
  h->part_rows = rows;
  h->loss_tiles = tiles;
  return cudaSuccess;
}
struct KeepSmall {  // gives large buffers back at the end of a call
  SphMlp* h;
  ~KeepSmall() {
    if (h->work_bytes > kKeep) free_work(h);
  }
};

// Rows of partials, tiles per CTA and rows per group of a mini-batch: four
// tiles a CTA once those CTAs cover the SMs.
struct Split {
  int rows, tiles, group;
  Split(const SphMlp* h, size_t n) {
    const size_t ctas = (n + kCtaSamples - 1) / kCtaSamples;
    tiles = ctas >= (size_t)h->sms ? 4 : 1;
    rows = (int)(tiles == 4 ? ctas : (n + 15) / 16);
    group = tiles == 4 ? 1 : 4;
  }
};

// The gradient of samples [lo, lo + bn) of the permutation, then the sum over
// its rows (and the update where `apply`)
void enqueue_batch(SphMlp* h, size_t lo, int bn, float* loss, float lr, float c1, float c2, int apply) {
  const Split sp(h, (size_t)bn);
  k_mlp_train<<<sp.rows, kWarps * 32, sizeof(TrainSmem), h->st>>>(h->wb, h->w, h->dx, h->dt, h->dp, (int)lo, bn,
                                                                  sp.tiles, h->part, loss);
  auto* adam = sp.group == 1 ? k_adam<true> : k_adam<false>;
  adam<<<(kParams + 63) / 64, 64, 0, h->st>>>(sp.rows, sp.group, h->part, h->grad, h->w, h->m, h->v, h->wb, lr, 0.9f,
                                              0.999f, 1e-8f, c1, c2, apply);
}

// Adds a mini-batch's loss from its tiles': groups of four in FP32 first
void add_loss(const float* lp, size_t tiles, double& L) {
  for (size_t a = 0; a < tiles; a += 4) {
    float s = 0.0f;
    for (size_t q = a; q < std::min(a + 4, tiles); ++q) s += lp[q];
    L += s;
  }
}

}  // namespace

extern "C" {

int sph_mlp_create(int device, uint64_t seed, SphMlp** out) {
  if (!out) return SPH_ERR_INVALID_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
    cudaGetLastError();
    return SPH_ERR_NO_DEVICE;
  }
  SphMlp* h = new SphMlp();
  h->dev = device;
  cudaSetDevice(device);
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) == cudaSuccess && sms > 0) h->sms = sms;
  cudaError_t e = cudaStreamCreateWithFlags(&h->st, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = mal(h, &h->w, kParams);
  if (e == cudaSuccess) e = mal(h, &h->m, kParams);
  if (e == cudaSuccess) e = mal(h, &h->v, kParams);
  if (e == cudaSuccess) e = mal(h, &h->wb, kBf16Count);
  if (e == cudaSuccess) e = mal(h, &h->grad, kParams);
  if (e == cudaSuccess && cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               (int)sizeof(CtaSmem)) != cudaSuccess)
    e = cudaErrorInvalidValue;
  if (e != cudaSuccess) {
    sph_mlp_destroy(h);
    return status(e);
  }
  // uniform(-1/sqrt(fan_in), 1/sqrt(fan_in)) weights and biases
  std::vector<float> w(kParams);
  uint64_t s = seed;
  const int fan[3] = {kIn, kHid, kHid};
  const int off_w[3] = {kOffW1, kOffW2, kOffW3}, nw[3] = {kHid * kIn, kHid * kHid, kOut * kHid};
  const int off_b[3] = {kOffB1, kOffB2, kOffB3}, nb[3] = {kHid, kHid, kOut};
  for (int l = 0; l < 3; ++l) {
    double a = 1.0 / std::sqrt((double)fan[l]);
    for (int i = 0; i < nw[l]; ++i) w[off_w[l] + i] = (float)((2.0 * uniform01(s) - 1.0) * a);
    for (int i = 0; i < nb[l]; ++i) w[off_b[l] + i] = (float)((2.0 * uniform01(s) - 1.0) * a);
  }
  int st = sph_mlp_set_params(h, w.data());
  if (st != SPH_OK) {
    sph_mlp_destroy(h);
    return st;
  }
  *out = h;
  return SPH_OK;
}

void sph_mlp_destroy(SphMlp* h) {
  if (!h) return;
  cudaSetDevice(h->dev);
  if (h->st) cudaStreamSynchronize(h->st);
  for (void* p : h->allocs) cudaFree(p);
  free_work(h);
  if (h->st) cudaStreamDestroy(h->st);
  delete h;
}

int sph_mlp_set_params(SphMlp* h, const float* params) {
  if (!h || !params) return SPH_ERR_INVALID_ARG;
  cudaSetDevice(h->dev);
  cudaError_t e = cudaMemcpyAsync(h->w, params, kParams * sizeof(float), cudaMemcpyHostToDevice, h->st);
  if (e == cudaSuccess) e = cudaMemsetAsync(h->m, 0, kParams * sizeof(float), h->st);
  if (e == cudaSuccess) e = cudaMemsetAsync(h->v, 0, kParams * sizeof(float), h->st);
  if (e == cudaSuccess) {
    k_refresh_bf16<<<(kParams + 255) / 256, 256, 0, h->st>>>(h->w, h->wb);
    e = cudaStreamSynchronize(h->st);
  }
  h->step = 0;
  return status(e);
}

int sph_mlp_get_params(SphMlp* h, float* params) {
  if (!h || !params) return SPH_ERR_INVALID_ARG;
  cudaSetDevice(h->dev);
  cudaError_t e = cudaMemcpyAsync(params, h->w, kParams * sizeof(float), cudaMemcpyDeviceToHost, h->st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(h->st);
  return status(e);
}

int sph_mlp_forward(SphMlp* h, const float* x, size_t n, float* y) {
  if (!h || (n && (!x || !y)) || n > 0x7fffffffull) return SPH_ERR_INVALID_ARG;
  if (n == 0) return SPH_OK;
  cudaSetDevice(h->dev);
  auto run = [&](float* dx, float* dy) {
    cudaError_t e = cudaMemcpyAsync(dx, x, n * kIn * sizeof(float), cudaMemcpyHostToDevice, h->st);
    if (e == cudaSuccess) {
      int blocks = (int)std::min<size_t>((n + kCtaSamples - 1) / kCtaSamples, (size_t)h->sms * 4);
      k_mlp_forward<<<blocks, kWarps * 32, sizeof(CtaSmem), h->st>>>(h->wb, h->w, dx, (int)n, dy);
      e = cudaMemcpyAsync(y, dy, n * kOut * sizeof(float), cudaMemcpyDeviceToHost, h->st);
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->st);
    return e;
  };
  std::unique_lock<std::mutex> lock(h->mu, std::try_to_lock);
  if (!lock.owns_lock()) {  // another thread's call has the kept buffers, perhaps for a whole training
    float* own = nullptr;
    cudaError_t e = cudaMalloc((void**)&own, n * (kIn + kOut) * sizeof(float));
    if (e == cudaSuccess) e = run(own, own + n * kIn);
    if (own) cudaFree(own);
    return status(e);
  }
  KeepSmall keep{h};
  cudaError_t e = ensure_work(h, n, 0, 0);
  if (e == cudaSuccess) e = run(h->dx, h->dt);
  return status(e);
}

int sph_mlp_loss_grad(SphMlp* h, const float* x, const float* t, size_t n, float* loss, float* grad) {
  if (!h || !x || !t || n == 0 || n > (1u << 24)) return SPH_ERR_INVALID_ARG;
  cudaSetDevice(h->dev);
  std::lock_guard<std::mutex> lock(h->mu);
  KeepSmall keep{h};
  const size_t tiles = (n + 15) / 16;
  cudaError_t e = ensure_work(h, n, Split(h, n).rows, tiles);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h->dx, x, n * kIn * sizeof(float), cudaMemcpyHostToDevice, h->st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h->dt, t, n * kOut * sizeof(float), cudaMemcpyHostToDevice, h->st);
  std::vector<uint32_t> perm(n);
  for (size_t i = 0; i < n; ++i) perm[i] = (uint32_t)i;
  if (e == cudaSuccess) e = cudaMemcpyAsync(h->dp, perm.data(), n * 4, cudaMemcpyHostToDevice, h->st);
  if (e == cudaSuccess) {
    enqueue_batch(h, 0, (int)n, h->loss, 0.0f, 1.0f, 1.0f, 0);
    std::vector<float> lp(tiles);
    e = cudaMemcpyAsync(lp.data(), h->loss, tiles * sizeof(float), cudaMemcpyDeviceToHost, h->st);
    if (e == cudaSuccess && grad) e = cudaMemcpyAsync(grad, h->grad, kParams * 4, cudaMemcpyDeviceToHost, h->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->st);
    double L = 0.0;
    add_loss(lp.data(), tiles, L);
    if (loss) *loss = (float)(L / (double)(n * kOut));
  }
  return status(e);
}

int sph_mlp_train(SphMlp* h, const float* x, const float* t, size_t n, int batch, int epochs, float lr,
                  uint64_t shuffle_seed, float* epoch_loss) {
  if (!h || !x || !t || n == 0 || n > 0x7fffffffull || batch < 16 || epochs < 1 || !(lr > 0.0f))
    return SPH_ERR_INVALID_ARG;
  cudaSetDevice(h->dev);
  std::lock_guard<std::mutex> lock(h->mu);
  KeepSmall keep{h};
  // tiles of an epoch, mini-batch by mini-batch
  const size_t full = n / (size_t)batch, per = ((size_t)batch + 15) / 16, rest = n % (size_t)batch;
  const size_t tiles = full * per + (rest + 15) / 16;
  cudaError_t e =
      ensure_work(h, n, std::max(Split(h, std::min(n, (size_t)batch)).rows, Split(h, rest).rows), tiles);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h->dx, x, n * kIn * sizeof(float), cudaMemcpyHostToDevice, h->st);
  if (e == cudaSuccess) e = cudaMemcpyAsync(h->dt, t, n * kOut * sizeof(float), cudaMemcpyHostToDevice, h->st);
  std::vector<uint32_t> perm(n);
  std::vector<float> lp(tiles);
  uint64_t rs = shuffle_seed;
  const float b1 = 0.9f, b2 = 0.999f;
  auto shuffle = [&] {
    for (size_t i = 0; i < n; ++i) perm[i] = (uint32_t)i;
    for (size_t i = n - 1; i > 0; --i) std::swap(perm[i], perm[splitmix(rs) % (i + 1)]);
  };
  shuffle();
  for (int ep = 0; ep < epochs && e == cudaSuccess; ++ep) {
    // an epoch's mini-batches follow one another on the stream; the losses come
    // back once, after the host has shuffled the next epoch
    e = cudaMemcpyAsync(h->dp, perm.data(), n * 4, cudaMemcpyHostToDevice, h->st);
    float* loss = h->loss;
    for (size_t lo = 0; lo < n && e == cudaSuccess; lo += (size_t)batch) {
      const int bn = (int)std::min<size_t>((size_t)batch, n - lo);
      h->step += 1;
      float c1 = 1.0f - powf(b1, (float)h->step), c2 = 1.0f - powf(b2, (float)h->step);
      enqueue_batch(h, lo, bn, loss, lr, c1, c2, 1);
      e = cudaGetLastError();
      loss += ((size_t)bn + 15) / 16;
    }
    if (ep + 1 < epochs) shuffle();
    if (e == cudaSuccess) e = cudaMemcpyAsync(lp.data(), h->loss, tiles * sizeof(float), cudaMemcpyDeviceToHost, h->st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(h->st);
    double L = 0.0;
    for (size_t k = 0; k < full; ++k) add_loss(lp.data() + k * per, per, L);
    if (rest) add_loss(lp.data() + full * per, tiles - full * per, L);
    if (epoch_loss) epoch_loss[ep] = (float)(L / (double)(n * kOut));
  }
  return status(e);
}

}  // extern "C"
