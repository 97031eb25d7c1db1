// Fused softmax cross-entropy over bf16 logits: the per-row loss and, where a gradient is wanted, the logits' gradient
// (softmax - onehot) * scale in the same kernel, so no fp32 [T, V] tensor exists.  The mean's 1 / (number of valid
// targets) is known before the rows run and is part of that scale; a loss gradient of 1 then leaves nothing to do
// in the backward pass.  One CTA per row.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "dbgcheck.cuh"
#include "launch.cuh"

extern "C" void pb_count_launch(int n);

namespace pbx {

constexpr int THREADS = 512;
constexpr int ROW_NARROW = 4096;  // classes up to which 128 threads per row are enough (32 columns each)
constexpr int ROW_WIDE = 56000;   // classes of a row that fits shared memory twice per SM (2 x 112 KB of 227)

__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const __nv_bfloat162* b = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float2 t = __bfloat1622float2(b[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 u;
  __nv_bfloat162* b = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) b[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// Rows that fit shared memory twice per SM (V <= ROW_WIDE).  What bounds it: bytes in flight, then the two exponentials
// per element on the special-function unit (2 V / 16 cycles per row and SM).  The whole row is requested at once with
// asynchronous 16-byte copies, every thread reads back only what it copied itself, and three short passes run over
// shared memory: maximum, sum, gradient.  The two-pass kernel below keeps one 16-byte load per thread in flight, rescales its sum at
// each vector and compares every column with the target.
// On a B200, loss and gradient: 8192 x 32000 276 -> 246 us, 2048 x 50257 123 -> 117 us, 512 x 1024 17.5 -> 7.7 us; loss
// alone: 8192 x 32000 279 -> 132 us.  (1 024 threads per row: 342, 137 us.)
__device__ __forceinline__ float block_max(float v, float* red, int nwarps) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int i = 1; i < nwarps; ++i) v = fmaxf(v, red[i]);
  return v;
}
__device__ __forceinline__ float block_add(float v, float* red, int nwarps) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  v = red[0];
  for (int i = 1; i < nwarps; ++i) v += red[i];
  return v;
}

template <int kThreads>
__global__ void __launch_bounds__(kThreads) xent_row_kernel(const __nv_bfloat16* logits, __nv_bfloat16* dlogits,
                                                            const long long* __restrict__ targets,
                                                            float* __restrict__ loss_rows,
                                                            const float* __restrict__ n_valid, int V, long long ld,
                                                            long long ignore_index PB_DBG_PARAMS) {
  extern __shared__ uint4 buf[];  // the row's ceil(V / 8) vectors
  __shared__ float red_m[kThreads / 32], red_s[kThreads / 32];
  const long long row = blockIdx.x;
  const uint4* lr = reinterpret_cast<const uint4*>(logits + row * ld);
  const int nvec = (V + 7) / 8, ldvec = (int)(ld / 8);
  const uint32_t sbase = (uint32_t)__cvta_generic_to_shared(buf);
  for (int c = threadIdx.x; c < nvec; c += kThreads)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sbase + c * 16), "l"(lr + c) : "memory");
  long long tgt = targets[row];
  if (tgt != ignore_index && !PB_DBG_IN_RANGE(tgt)) tgt = ignore_index;  // debug build: reported, row skipped
  const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= V;
  asm volatile("cp.async.wait_all;" ::: "memory");
  if ((V & 7) && threadIdx.x == (nvec - 1) % kThreads) {  // padding columns of the last vector count as -inf
    __nv_bfloat16* tail = reinterpret_cast<__nv_bfloat16*>(buf) + (nvec - 1) * 8;
    for (int j = V & 7; j < 8; ++j) tail[j] = __float2bfloat16(-CUDART_INF_F);
  }
  float m = -CUDART_INF_F;
  for (int c = threadIdx.x; c < nvec; c += kThreads) {
    float v[8];
    unpack8(buf[c], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) m = fmaxf(m, v[j]);
  }
  m = block_max(m, red_m, kThreads / 32);  // its barrier also publishes the row to every thread
  float s = 0.f;
  for (int c = threadIdx.x; c < nvec; c += kThreads) {
    float v[8];
    unpack8(buf[c], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) s += __expf(v[j] - m);
  }
  s = block_add(s, red_s, kThreads / 32);
  const float x_t = ignored ? 0.f : __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(buf)[tgt]);
  if (threadIdx.x == 0) loss_rows[row] = ignored ? 0.f : (m + __logf(s) - x_t);
  if (dlogits == nullptr) return;
  const float gs = ignored ? 0.f : (n_valid ? 1.f / *n_valid : 1.f);
  const float scale = gs / s;
  uint4* dr = reinterpret_cast<uint4*>(dlogits + row * ld);
  const int tvec = ignored ? -1 : (int)(tgt / 8);
  for (int c = threadIdx.x; c < nvec; c += kThreads) {
    float v[8];
    unpack8(buf[c], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) v[j] = __expf(v[j] - m) * scale;
    if (c == tvec) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j == (int)(tgt & 7)) v[j] = (__expf(x_t - m) / s - 1.f) * gs;
    }
    dr[c] = pack8(v);
  }
  for (int c = nvec + threadIdx.x; c < ldvec; c += kThreads) dr[c] = make_uint4(0u, 0u, 0u, 0u);
}

// *n_valid = max(1, number of targets that are not ignored); one CTA.
__global__ void __launch_bounds__(1024) xent_count_kernel(const long long* __restrict__ targets, long long T,
                                                          long long ignore_index, float* __restrict__ n_valid) {
  __shared__ int total;
  if (threadIdx.x == 0) total = 0;
  __syncthreads();
  int n = 0;
#pragma unroll 4
  for (long long i = threadIdx.x; i < T; i += 1024) n += targets[i] != ignore_index;
  n = __reduce_add_sync(0xffffffffu, n);
  if ((threadIdx.x & 31) == 0) atomicAdd(&total, n);
  __syncthreads();
  if (threadIdx.x == 0) *n_valid = (float)(total > 1 ? total : 1);
}

// *loss = sum of the rows' losses (over n_valid), in a fixed order; one CTA.
__global__ void __launch_bounds__(1024) xent_loss_kernel(const float* __restrict__ loss_rows, long long T,
                                                         const float* __restrict__ n_valid, float* __restrict__ loss) {
  __shared__ float red[32];
  float s = 0.f;
#pragma unroll 4
  for (long long i = threadIdx.x; i < T; i += 1024) s += loss_rows[i];
  s = block_add(s, red, 32);
  if (threadIdx.x == 0) *loss = n_valid ? s / *n_valid : s;
}

// Any V: the row is read twice, the second time from L2.
// logits: [T, ld] bf16, first V columns are classes (ld >= V, ld % 8 == 0; columns >= V are padding and get
// zero gradient).  targets: int64 [T], ignore_index rows contribute nothing.  loss_rows: fp32 [T].
// On exit dlogits (null = not wanted; it may alias logits) holds (softmax - onehot) / n_valid (null = not divided).
__global__ void __launch_bounds__(THREADS) xent_fwd_bwd_kernel(const __nv_bfloat16* logits, __nv_bfloat16* dlogits,
                                                               const long long* __restrict__ targets,
                                                               float* __restrict__ loss_rows, int V, long long ld,
                                                               const float* __restrict__ n_valid,
                                                               long long ignore_index
                                                               PB_DBG_PARAMS) {
  __shared__ float red_m[THREADS / 32];
  __shared__ float red_s[THREADS / 32];
  __shared__ float bc[2];
  const long long row = blockIdx.x;
  const __nv_bfloat16* lr = logits + row * ld;
  __nv_bfloat16* dr = dlogits + row * ld;
  long long tgt = targets[row];
  if (tgt != ignore_index && !PB_DBG_IN_RANGE(tgt)) tgt = ignore_index;  // debug build: reported, row skipped
  const int nvec = V / 8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  float m = -CUDART_INF_F, s = 0.f;
  for (int c = threadIdx.x; c < nvec; c += THREADS) {
    float v[8];
    unpack8(reinterpret_cast<const uint4*>(lr)[c], v);
    float cm = v[0];
#pragma unroll
    for (int j = 1; j < 8; ++j) cm = fmaxf(cm, v[j]);
    const float nm = fmaxf(m, cm);
    const float base = nm == -CUDART_INF_F ? 0.f : nm;  // nothing but masked columns so far: they add 0, not NaN
    float add = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) add += __expf(v[j] - base);
    s = s * __expf(m - base) + add;
    m = nm;
  }
  for (int c = nvec * 8 + threadIdx.x; c < V; c += THREADS) {  // ragged tail
    const float v = __bfloat162float(lr[c]);
    const float nm = fmaxf(m, v);
    const float base = nm == -CUDART_INF_F ? 0.f : nm;
    s = s * __expf(m - base) + __expf(v - base);
    m = nm;
  }
  // block combine of (m, s)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float om = __shfl_xor_sync(0xffffffffu, m, o);
    const float os = __shfl_xor_sync(0xffffffffu, s, o);
    const float nm = fmaxf(m, om);
    s = (nm == -CUDART_INF_F) ? 0.f : s * __expf(m - nm) + os * __expf(om - nm);
    m = nm;
  }
  if (lane == 0) {
    red_m[warp] = m;
    red_s[warp] = s;
  }
  __syncthreads();
  if (warp == 0) {
    m = lane < THREADS / 32 ? red_m[lane] : -CUDART_INF_F;
    s = lane < THREADS / 32 ? red_s[lane] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float om = __shfl_xor_sync(0xffffffffu, m, o);
      const float os = __shfl_xor_sync(0xffffffffu, s, o);
      const float nm = fmaxf(m, om);
      s = (nm == -CUDART_INF_F) ? 0.f : s * __expf(m - nm) + os * __expf(om - nm);
      m = nm;
    }
    if (lane == 0) {
      bc[0] = m;
      bc[1] = s;
    }
  }
  __syncthreads();
  m = bc[0];
  s = bc[1];
  const float lse = m + __logf(s);
  const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= V;
  if (threadIdx.x == 0) loss_rows[row] = ignored ? 0.f : (lse - __bfloat162float(lr[tgt]));
  if (dlogits == nullptr) return;
  __syncthreads();  // the target logit was read before anything is overwritten
  const float gs = ignored ? 0.f : (n_valid ? 1.f / *n_valid : 1.f);
  const float inv = 1.f / s;
  for (int c = threadIdx.x; c < nvec; c += THREADS) {
    float v[8];
    unpack8(reinterpret_cast<const uint4*>(lr)[c], v);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float p = __expf(v[j] - m) * inv;
      if ((long long)c * 8 + j == tgt) p -= 1.f;
      v[j] = p * gs;
    }
    reinterpret_cast<uint4*>(dr)[c] = pack8(v);
  }
  for (int c = nvec * 8 + threadIdx.x; c < ld; c += THREADS) {
    float p = 0.f;
    if (c < V) {
      p = __expf(__bfloat162float(lr[c]) - m) * inv;
      if (c == tgt) p -= 1.f;
    }
    dr[c] = __float2bfloat16(p * gs);
  }
}

}  // namespace pbx

extern "C" {

// loss (fp32 scalar) = sum over the rows of lse - logit[target], over the number of valid targets when `n_valid`
// (fp32 scratch scalar) is given.  dlogits: null, or [T, ld] bf16 (may alias logits): the gradient of that loss.
// loss_rows: fp32 [T] scratch.
int pb_xent(const void* logits, void* dlogits, const long long* targets, float* loss_rows, float* n_valid, float* loss,
            long long T, int V, long long ld, long long ignore_index, void* stream_) {
  using namespace pbx;
  if (ld % 8 != 0 || ld < V) return -1;
  cudaStream_t stream = reinterpret_cast<cudaStream_t>(stream_);
  auto L = reinterpret_cast<const __nv_bfloat16*>(logits);
  auto D = reinterpret_cast<__nv_bfloat16*>(dlogits);
  if (n_valid) {
    xent_count_kernel<<<1, 1024, 0, stream>>>(targets, T, ignore_index, n_valid);
    pb_count_launch(1);
  }
  const int smem = (V + 7) / 8 * 16;
  if (V <= ROW_NARROW) {
    xent_row_kernel<128><<<(unsigned)T, 128, smem, stream>>>(L, D, targets, loss_rows, n_valid, V, ld,
                                                             ignore_index PB_DBG_ARGS(V));
  } else if (V <= ROW_WIDE) {
    if (cudaError_t e = pb::allow_smem<xent_row_kernel<THREADS>, ROW_WIDE * 2>(); e != cudaSuccess) return (int)e;
    xent_row_kernel<THREADS><<<(unsigned)T, THREADS, smem, stream>>>(L, D, targets, loss_rows, n_valid, V, ld,
                                                                     ignore_index PB_DBG_ARGS(V));
  } else {
    xent_fwd_bwd_kernel<<<(unsigned)T, THREADS, 0, stream>>>(L, D, targets, loss_rows, V, ld, n_valid,
                                                             ignore_index PB_DBG_ARGS(V));
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return (int)e;
  xent_loss_kernel<<<1, 1024, 0, stream>>>(loss_rows, T, n_valid, loss);
  pb_count_launch(2);
  return (int)cudaGetLastError();
}

}  // extern "C"
