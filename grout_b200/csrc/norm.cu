// RMSNorm with the residual sum folded in.
//
//   v   = res_in[s, :] + delta[s, :]        (either may be absent; 32-bit sum)
//   res_out[r, :] = v                       (32-bit residual stream, optional)
//   y[r, :] = v / sqrt(mean(v^2) + eps) * w
//
// s = rows[r] when a row list is given (gather before the final norm), else r.
// The reference's rms_norm_f16 (src/kernels.rs:304-343) and add_rms_norm_f16
// (src/kernels.rs:3013-3074) keep the sum in f32 only inside the kernel and
// store a 16-bit residual; here the residual stream itself stays 32-bit.
// In 32-bit the kernel, and with it the reduction tree, is chosen by N only, so
// a row's result does not depend on the batch it is in; in bfloat16 few rows of a
// wide model take a cluster of blocks per row (another order of sums, which
// bfloat16's rounding of y hides).
#include <cooperative_groups.h>

#include <type_traits>

#include "common.cuh"

namespace cg = cooperative_groups;

// `parts`: instead of (or beside) delta, n_parts 32-bit partial sums [n_parts]
// [rows_total, N], part_stride floats apart, added in order: the split-K product
// of the projection before this norm leaves its reduction to this kernel.
template <typename T, typename WT>
__global__ void add_rmsnorm_kernel(const float* res_in, const T* delta, const float* parts,
                                   int n_parts, long long part_stride,
                                   const int* __restrict__ rows, const WT* __restrict__ w,
                                   float eps, float* res_out, T* __restrict__ y, int N) {
  __shared__ float scratch[32];
  pdl_launch_dependents_if_small();
  pdl_wait();
  const int r = blockIdx.x;
  const size_t s = rows ? (size_t)rows[r] : (size_t)r;
  const float* rin = res_in ? res_in + s * N : nullptr;
  const T* din = delta ? delta + s * N : nullptr;
  float* rout = res_out ? res_out + (size_t)r * N : nullptr;
  const float* pin = parts ? parts + s * N : nullptr;
  auto value = [&](int i) {
    float d = din ? to_f32<T>(din[i]) : 0.f;
    for (int k = 0; k < n_parts; ++k) d += pin[(size_t)k * part_stride + i];
    return (rin ? rin[i] : 0.f) + d;
  };
  float ss = 0.f;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    float v = value(i);
    if (rout) rout[i] = v;
    ss += v * v;
  }
  ss = block_sum(ss, scratch);
  pdl_launch_dependents_if_large();
  const float inv = 1.0f / sqrtf(ss / (float)N + eps);
  T* yo = y + (size_t)r * N;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    // the same thread wrote rout[i] above, so it reads its own store here
    float v = rout ? rout[i] : value(i);
    yo[i] = from_f32<T>(v * inv * to_f32<WT>(w[i]));
  }
}

// The same operation for widths that are a multiple of 4 and at most 16384:
// every thread keeps its (up to 16) values in registers between the sum of
// squares and the scaling, and all traffic is in 8- or 16-byte pieces.
#define NV_MAX 4
template <typename T> struct Vec4;
template <> struct Vec4<float> {
  static __device__ __forceinline__ void load(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
  }
  static __device__ __forceinline__ void store(float* p, const float (&v)[4]) {
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  }
};
template <> struct Vec4<bf16> {
  static __device__ __forceinline__ void load(const bf16* p, float (&v)[4]) {
    const uint2 x = *reinterpret_cast<const uint2*>(p);
    const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&x.x);
    const __nv_bfloat162 b = *reinterpret_cast<const __nv_bfloat162*>(&x.y);
    v[0] = __low2float(a); v[1] = __high2float(a); v[2] = __low2float(b); v[3] = __high2float(b);
  }
  static __device__ __forceinline__ void store(bf16* p, const float (&v)[4]) {
    __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    uint2 x;
    x.x = *reinterpret_cast<uint32_t*>(&a);
    x.y = *reinterpret_cast<uint32_t*>(&b);
    *reinterpret_cast<uint2*>(p) = x;
  }
};

template <typename T, typename WT>
__global__ void add_rmsnorm_vec_kernel(const float* res_in, const T* delta, const float* parts,
                                       int n_parts, long long part_stride,
                                       const int* __restrict__ rows, const WT* __restrict__ w,
                                       float eps, float* res_out, T* __restrict__ y, int N) {
  __shared__ float scratch[32];
  pdl_launch_dependents_if_small();
  // the weight vector is no kernel's output: fetch it while the producer drains
  float wv[NV_MAX][4];
#pragma unroll
  for (int j = 0; j < NV_MAX; ++j) {
    const int i = (threadIdx.x + j * blockDim.x) * 4;
    if (i < N) Vec4<WT>::load(w + i, wv[j]);
  }
  pdl_wait();
  const int r = blockIdx.x;
  const size_t s = rows ? (size_t)rows[r] : (size_t)r;
  const float* rin = res_in ? res_in + s * N : nullptr;
  const T* din = delta ? delta + s * N : nullptr;
  float* rout = res_out ? res_out + (size_t)r * N : nullptr;
  const float* pin = parts ? parts + s * N : nullptr;
  float v[NV_MAX][4];
  float ss = 0.f;
  // all of a thread's loads first, then the sums: the memory system sees every
  // request of the row at once
  float av[NV_MAX][4], dv[NV_MAX][4];
#pragma unroll
  for (int j = 0; j < NV_MAX; ++j) {
    const int i = (threadIdx.x + j * blockDim.x) * 4;
#pragma unroll
    for (int e = 0; e < 4; ++e) av[j][e] = dv[j][e] = 0.f;
    if (i < N) {
      if (rin) Vec4<float>::load(rin + i, av[j]);
      if (din) Vec4<T>::load(din + i, dv[j]);
    }
  }
#pragma unroll
  for (int j = 0; j < NV_MAX; ++j) {
    const int i = (threadIdx.x + j * blockDim.x) * 4;
    if (i < N) {
      for (int k0 = 0; k0 < n_parts; k0 += 4) {   // four at once, added in order
        float pk[4][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int k = k0 + u < n_parts ? k0 + u : n_parts - 1;
          Vec4<float>::load(pin + (size_t)k * part_stride + i, pk[u]);
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (k0 + u < n_parts) {
#pragma unroll
            for (int e = 0; e < 4; ++e) dv[j][e] += pk[u][e];
          }
      }
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        v[j][e] = av[j][e] + dv[j][e];
        ss += v[j][e] * v[j][e];
      }
      if (rout) Vec4<float>::store(rout + i, v[j]);
    }
  }
  ss = block_sum(ss, scratch);
  pdl_launch_dependents_if_large();
  const float inv = 1.0f / sqrtf(ss / (float)N + eps);
  T* yo = y + (size_t)r * N;
#pragma unroll
  for (int j = 0; j < NV_MAX; ++j) {
    const int i = (threadIdx.x + j * blockDim.x) * 4;
    if (i < N) {
      float o[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) o[e] = v[j][e] * inv * wv[j][e];
      Vec4<T>::store(yo + i, o);
    }
  }
}

// A handful of rows (a decode step) would keep a handful of SMs busy.  Here a
// cluster of NC_CLUSTER blocks shares a row: each block owns a quarter of the
// columns, the sums of squares meet through distributed shared memory (added in
// rank order, so the result is a fixed sum), and every block scales its columns.
// The cluster barrier is the hardware's; no block spins on memory.
#ifndef NC_CLUSTER
#define NC_CLUSTER 4
#endif
template <typename T, typename WT>
__global__ void add_rmsnorm_cluster_kernel(const float* res_in, const T* delta, const float* parts, int n_parts,
                           long long part_stride, const int* __restrict__ rows,
                           const WT* __restrict__ w, float eps, float* res_out,
                           T* __restrict__ y, int N) {
  __shared__ float scratch[32];
  __shared__ float ss_all[NC_CLUSTER];
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = (int)cluster.block_rank();
  pdl_launch_dependents_if_small();
  const int cols = N / NC_CLUSTER;              // a multiple of 4
  const int c0 = rank * cols;
  const int i = c0 + threadIdx.x * 4;           // this thread's four columns
  const bool active = threadIdx.x * 4 < cols;
  float wv[4] = {0.f, 0.f, 0.f, 0.f};
  if (active) Vec4<WT>::load(w + i, wv);        // no kernel's output: before the wait
  pdl_wait();
  const int r = blockIdx.x / NC_CLUSTER;
  const size_t s = rows ? (size_t)rows[r] : (size_t)r;
  float v[4] = {0.f, 0.f, 0.f, 0.f};
  float ss = 0.f;
  if (active) {
    float a[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
    if (res_in) Vec4<float>::load(res_in + s * N + i, a);
    if (delta) Vec4<T>::load(delta + s * N + i, d);
    // eight partials are requested at once and then added in order: one at a time, each
    // load would wait for the one before it to have been added (a round trip to L2 each;
    // a product is split at most eight ways, so this is one trip)
    for (int k0 = 0; k0 < n_parts; k0 += 8) {
      float pk[8][4];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int k = k0 + u < n_parts ? k0 + u : n_parts - 1;
        Vec4<float>::load(parts + (size_t)k * part_stride + s * N + i, pk[u]);
      }
#pragma unroll
      for (int u = 0; u < 8; ++u)
        if (k0 + u < n_parts) {
#pragma unroll
          for (int e = 0; e < 4; ++e) d[e] += pk[u][e];
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      v[e] = a[e] + d[e];
      ss += v[e] * v[e];
    }
    if (res_out) Vec4<float>::store(res_out + (size_t)r * N + i, v);
  }
  ss = block_sum(ss, scratch);
  // every block puts its sum into every block's table (thread k writes to block k), so
  // that one cluster barrier is enough: after it each block reads its own shared memory
  // only, and nobody is read from after it has left
  if (threadIdx.x < NC_CLUSTER) cluster.map_shared_rank(ss_all, threadIdx.x)[rank] = ss;
  cluster.sync();
  float total = 0.f;
#pragma unroll
  for (int k = 0; k < NC_CLUSTER; ++k) total += ss_all[k];
  const float inv = 1.0f / sqrtf(total / (float)N + eps);
  if (active) {
    float o[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) o[e] = v[e] * inv * wv[e];
    Vec4<T>::store(y + (size_t)r * N + i, o);
  }
}

static int norm_threads(int N) {
  int t = (N + 3) / 4;
  t = ((t + 31) / 32) * 32;
  if (t < 32) t = 32;
  if (t > 1024) t = 1024;
  return t;
}

template <typename T, typename WT>
static int launch(const float* res_in, const void* delta, const float* parts, int n_parts,
                  long long part_stride, const int* rows, const void* w, float eps,
                  float* res_out, void* y, int n_rows, int N, cudaStream_t stream) {
  if (n_rows < 0 || N <= 0 || !w || !y || (!res_in && !delta && !parts)) return GB_ERR_BAD_ARG;
  if ((parts != nullptr) != (n_parts > 0) || n_parts < 0) return GB_ERR_BAD_ARG;
  // in place is allowed only without a row list (each block then owns its row)
  if (rows && res_out && res_out == res_in) return GB_ERR_BAD_ARG;
  if (n_rows == 0) return 0;
  const bool aligned = ((((uintptr_t)res_in) | ((uintptr_t)delta) | ((uintptr_t)w) |
                         ((uintptr_t)res_out) | ((uintptr_t)y) | ((uintptr_t)parts) |
                         ((uintptr_t)(part_stride * 4))) & 15) == 0;
  // The cluster kernel is chosen by the number of rows and sums in another order
  // than the kernels below.  The 32-bit path never takes it: there the order of
  // a row's sums may depend on the width alone, so that a token's result is the
  // same in a step of one row and in a step of thousands.
  constexpr bool by_rows_too = !std::is_same<T, float>::value;
#ifndef NC_MAX_ROWS
#define NC_MAX_ROWS 64
#endif
  if (by_rows_too && aligned && n_rows <= NC_MAX_ROWS && N >= 1024 && N % (4 * NC_CLUSTER) == 0 &&
      N / NC_CLUSTER <= 4096) {
    int threads = ((N / NC_CLUSTER / 4 + 31) / 32) * 32;
    return gb_launch_cluster(add_rmsnorm_cluster_kernel<T, WT>, dim3(n_rows * NC_CLUSTER),
                             dim3(threads), 0, stream, NC_CLUSTER, res_in, (const T*)delta, parts,
                             n_parts, part_stride, rows, (const WT*)w, eps, res_out, (T*)y, N);
  }
  if (N % 4 == 0 && N <= 4 * 1024 * NV_MAX && aligned) {
    int threads = (N / 4 + NV_MAX - 1) / NV_MAX;      // vectors per thread <= NV_MAX
    threads = ((threads + 31) / 32) * 32;
    if (threads < 64) threads = 64;
    if (threads > 1024) threads = 1024;
    return gb_launch(add_rmsnorm_vec_kernel<T, WT>, dim3(n_rows), dim3(threads), 0, stream, res_in,
                     (const T*)delta, parts, n_parts, part_stride, rows, (const WT*)w, eps, res_out,
                     (T*)y, N);
  }
  return gb_launch(add_rmsnorm_kernel<T, WT>, dim3(n_rows), dim3(norm_threads(N)), 0, stream, res_in,
                   (const T*)delta, parts, n_parts, part_stride, rows, (const WT*)w, eps, res_out,
                   (T*)y, N);
}

// w_is_f32: the weight vector is stored in 32-bit although the activations are bf16.
GB_EXPORT int gb_add_rmsnorm_f32(const float* res_in, const void* delta, const float* parts,
                                 int n_parts, long long part_stride, const int* rows,
                                 const void* w, int w_is_f32, float eps, float* res_out, void* y,
                                 int n_rows, int N, cudaStream_t s) {
  if (!w_is_f32) return GB_ERR_UNSUPPORTED;
  return launch<float, float>(res_in, delta, parts, n_parts, part_stride, rows, w, eps, res_out, y,
                              n_rows, N, s);
}
GB_EXPORT int gb_add_rmsnorm_bf16(const float* res_in, const void* delta, const float* parts,
                                  int n_parts, long long part_stride, const int* rows,
                                  const void* w, int w_is_f32, float eps, float* res_out, void* y,
                                  int n_rows, int N, cudaStream_t s) {
  if (w_is_f32)
    return launch<bf16, float>(res_in, delta, parts, n_parts, part_stride, rows, w, eps, res_out, y,
                               n_rows, N, s);
  return launch<bf16, bf16>(res_in, delta, parts, n_parts, part_stride, rows, w, eps, res_out, y,
                            n_rows, N, s);
}

// ---- a contribution that passes through an RMS norm of its own ------------------
//
//   d   = delta[s, :]  (or the sum of n_parts 32-bit partial sums of it)
//   c   = post_w ? d / sqrt(mean(d^2) + post_eps) * post_w : d
//   c   = scale ? c * scale : c                      (a learned factor per channel)
//   v   = res_in[s, :] + c                           (either may be absent; 32-bit)
//   res_out[r, :] = v                                (optional)
//   y[r, :] = w ? v / sqrt(mean(v^2) + eps) * w : v  (rounded to the activation type)
//
// for layers that normalise a sublayer's output instead of its input: the
// sublayer that follows reads y = the stream itself.  All vectors are 32-bit.
// One block per row keeps the row in shared memory between its passes; the
// block's size, and with it the tree of its sums, depends on N only.
struct PostNormArgs {
  const float* res_in;
  const void* delta;
  const float* parts;
  int n_parts;
  long long part_stride;
  const int* rows;
  const float* post_w;
  float post_eps;
  const float* scale;
  const float* w;
  float eps;
  float* res_out;
  void* y;
  int n_rows, N;
};

template <typename T>
__global__ void add_postnorm_kernel(const PostNormArgs a) {
  extern __shared__ float row[];   // [N]
  __shared__ float scratch[32];
  pdl_launch_dependents_if_small();
  pdl_wait();
  const int N = a.N, r = blockIdx.x;
  const size_t s = a.rows ? (size_t)a.rows[r] : (size_t)r;
  const T* din = a.delta ? (const T*)a.delta + s * N : nullptr;
  const float* pin = a.parts ? a.parts + s * N : nullptr;
  const float* rin = a.res_in ? a.res_in + s * N : nullptr;
  const bool has_d = din || pin;
  float ss = 0.f;
  if (has_d) {
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
      float d = din ? to_f32<T>(din[i]) : 0.f;
      // partial sums are asked for eight (or four) at a time and added in their order: one
      // trip to memory for the lot instead of one each
      int k = 0;
      for (; k + 8 <= a.n_parts; k += 8) {
        float p[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) p[u] = pin[(size_t)(k + u) * a.part_stride + i];
#pragma unroll
        for (int u = 0; u < 8; ++u) d += p[u];
      }
      if (k + 4 <= a.n_parts) {
        float p[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) p[u] = pin[(size_t)(k + u) * a.part_stride + i];
#pragma unroll
        for (int u = 0; u < 4; ++u) d += p[u];
        k += 4;
      }
      for (; k < a.n_parts; ++k) d += pin[(size_t)k * a.part_stride + i];
      row[i] = d;
      ss += d * d;
    }
  }
  float inv_d = 1.f;
  if (has_d && a.post_w) inv_d = 1.0f / sqrtf(block_sum(ss, scratch) / (float)N + a.post_eps);
  float* rout = a.res_out ? a.res_out + (size_t)r * N : nullptr;
  ss = 0.f;
  for (int i = threadIdx.x; i < N; i += blockDim.x) {
    float v = rin ? rin[i] : 0.f;
    if (has_d) {
      float c = row[i];
      if (a.post_w) c = c * inv_d * a.post_w[i];
      if (a.scale) c *= a.scale[i];
      v += c;
    }
    if (rout) rout[i] = v;
    row[i] = v;
    ss += v * v;
  }
  pdl_launch_dependents_if_large();
  T* yo = (T*)a.y + (size_t)r * N;
  if (a.w) {
    const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)N + a.eps);
    for (int i = threadIdx.x; i < N; i += blockDim.x) yo[i] = from_f32<T>(row[i] * inv * a.w[i]);
  } else {
    for (int i = threadIdx.x; i < N; i += blockDim.x) yo[i] = from_f32<T>(row[i]);
  }
}

// The same with the row in registers, V pieces of four values a thread: for widths that are multiples of four up to
// 16,384 on 16-byte boundaries.  A decode step's row is a chain of latencies (the partial sums, two block-wide sums), so
// the weights are on their way to L2 before the wait (a kernel in front may have made them, so they are read behind it),
// and all of the row is asked for at once behind it; a prompt's rows are bound by memory, and small blocks keep many of
// them in flight.  Rows of 2,048, inside a step of one row: 4.3 us exposed (7.9 with the row in shared memory, a value at a time).  One row of eight partial
// sums and 1,024 rows of one, back to back, us, with the row in shared memory behind the stroke: 2,048 wide 2.7, 7.9 / 5.3,
// 13.8; 8,192 4.6, 23 / 14.9, 46; 8,196 6.9, 35 / 15.3, 45; 10,240 7.2, 44 / 17.9, 66; 16,384 9.0, 64 / 27, 144.
template <typename T> __device__ __forceinline__ float4 pn_load4(const T* p);
template <> __device__ __forceinline__ float4 pn_load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <> __device__ __forceinline__ float4 pn_load4<bf16>(const bf16* p) {
  const uint2 v = *reinterpret_cast<const uint2*>(p);
  const __nv_bfloat162 a = *reinterpret_cast<const __nv_bfloat162*>(&v.x), b = *reinterpret_cast<const __nv_bfloat162*>(&v.y);
  return make_float4(__low2float(a), __high2float(a), __low2float(b), __high2float(b));
}
__device__ __forceinline__ void pn_store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void pn_store4(bf16* p, float4 v) {
  __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
  uint2 u;
  u.x = *reinterpret_cast<uint32_t*>(&a), u.y = *reinterpret_cast<uint32_t*>(&b);
  *reinterpret_cast<uint2*>(p) = u;
}

// EARLY: the weights are asked for with the row; the threads of wide rows, of which there are up to 1,024, have no
// registers to hold them (64, and 64 bytes of spills in bfloat16), and read them where they are used.
template <typename T, int V, int THREADS, bool EARLY>
__global__ void __launch_bounds__(THREADS) add_postnorm_vec_kernel(const PostNormArgs a) {
  __shared__ float scratch[32];
  pdl_launch_dependents_if_small();
  const int N = a.N, r = blockIdx.x, tid = threadIdx.x, step = blockDim.x;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f), one = make_float4(1.f, 1.f, 1.f, 1.f);
  float4 wp[V], ws[V], wy[V];      // what multiplies the delta, the same again, and the row
  const auto weight = [&](const float* w, int at) { return at < N && w ? *reinterpret_cast<const float4*>(w + at) : one; };
  if constexpr (EARLY) {
    const auto fetch = [&](const float* w, int at) { if (at < N && w) prefetch_l2(w + at); };
    if (tid % 8 == 0)              // (eight threads' pieces are a line)
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int at = (tid + i * step) * 4;
        fetch(a.post_w, at), fetch(a.scale, at), fetch(a.w, at);
      }
  }
  pdl_wait();
  if constexpr (EARLY) {
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int at = (tid + i * step) * 4;
      wp[i] = weight(a.post_w, at);
      ws[i] = weight(a.scale, at);
      wy[i] = weight(a.w, at);
    }
  }
  const size_t s = a.rows ? (size_t)a.rows[r] : (size_t)r;
  float4 v[V], d[V];
  float ss = 0.f;
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int at = (tid + i * step) * 4;
    const bool in = at < N;
    v[i] = in && a.res_in ? *reinterpret_cast<const float4*>(a.res_in + s * N + at) : zero;
    d[i] = in && a.delta ? pn_load4<T>((const T*)a.delta + s * N + at) : zero;
  }
  if (a.parts) {
    const float* pin = a.parts + s * N;
    constexpr int U = V <= 2 ? 4 : EARLY ? 2 : 1;
    int k = 0;
    for (; k + U <= a.n_parts; k += U) {       // asked for U at a time, added in their order
      float4 p[U][V];
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < V; ++i) {
          const int at = (tid + i * step) * 4;
          p[u][i] = at < N ? *reinterpret_cast<const float4*>(pin + (size_t)(k + u) * a.part_stride + at) : zero;
        }
#pragma unroll
      for (int u = 0; u < U; ++u)
#pragma unroll
        for (int i = 0; i < V; ++i) d[i].x += p[u][i].x, d[i].y += p[u][i].y, d[i].z += p[u][i].z, d[i].w += p[u][i].w;
    }
    for (; k < a.n_parts; ++k)
#pragma unroll
      for (int i = 0; i < V; ++i) {
        const int at = (tid + i * step) * 4;
        if (at >= N) continue;
        const float4 p = *reinterpret_cast<const float4*>(pin + (size_t)k * a.part_stride + at);
        d[i].x += p.x, d[i].y += p.y, d[i].z += p.z, d[i].w += p.w;
      }
  }
  if (a.delta || a.parts) {
    float inv_d = 1.f;
    if (a.post_w) {
#pragma unroll
      for (int i = 0; i < V; ++i) ss += d[i].x * d[i].x + d[i].y * d[i].y + (d[i].z * d[i].z + d[i].w * d[i].w);
      inv_d = 1.0f / sqrtf(block_sum(ss, scratch) / (float)N + a.post_eps);
    }
#pragma unroll
    for (int i = 0; i < V; ++i) {
      if constexpr (!EARLY) wp[i] = weight(a.post_w, (tid + i * step) * 4), ws[i] = weight(a.scale, (tid + i * step) * 4);
      v[i].x += d[i].x * inv_d * wp[i].x * ws[i].x, v[i].y += d[i].y * inv_d * wp[i].y * ws[i].y;
      v[i].z += d[i].z * inv_d * wp[i].z * ws[i].z, v[i].w += d[i].w * inv_d * wp[i].w * ws[i].w;
    }
  }
  if (a.res_out)
#pragma unroll
    for (int i = 0; i < V; ++i) {
      const int at = (tid + i * step) * 4;
      if (at < N) pn_store4(a.res_out + (size_t)r * N + at, v[i]);
    }
  float inv = 1.f;
  if (a.w) {
    ss = 0.f;
#pragma unroll
    for (int i = 0; i < V; ++i) ss += v[i].x * v[i].x + v[i].y * v[i].y + (v[i].z * v[i].z + v[i].w * v[i].w);
    inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)N + a.eps);
  }
#pragma unroll
  for (int i = 0; i < V; ++i) {
    const int at = (tid + i * step) * 4;
    if constexpr (!EARLY) wy[i] = weight(a.w, at);
    if (at < N)
      pn_store4((T*)a.y + (size_t)r * N + at, make_float4(v[i].x * inv * wy[i].x, v[i].y * inv * wy[i].y,
                                                          v[i].z * inv * wy[i].z, v[i].w * inv * wy[i].w));
  }
  pdl_launch_dependents_if_large();
}

template <typename T, int V, int THREADS, bool EARLY>
static int add_postnorm_vec_launch(const PostNormArgs& a, cudaStream_t stream) {
  const int threads = ((a.N / 4 + V - 1) / V + 31) / 32 * 32;    // by N only
  return gb_launch(add_postnorm_vec_kernel<T, V, THREADS, EARLY>, dim3(a.n_rows), dim3(threads), 0, stream, a);
}

template <typename T>
static int add_postnorm_launch(const PostNormArgs& a, cudaStream_t stream) {
  if (a.n_rows < 0 || a.N <= 0 || !a.y || (!a.res_in && !a.delta && !a.parts)) return GB_ERR_BAD_ARG;
  if (a.parts && a.n_parts <= 0) return GB_ERR_BAD_ARG;
  if (a.n_rows == 0) return 0;
  const uintptr_t vectors = (uintptr_t)a.res_in | (uintptr_t)a.parts | (uintptr_t)a.post_w | (uintptr_t)a.scale |
                            (uintptr_t)a.w | (uintptr_t)a.res_out;
  if (a.N % 4 == 0 && a.N <= 16384 && !(vectors & 15) && !(((uintptr_t)a.delta | (uintptr_t)a.y) & (4 * sizeof(T) - 1)) &&
      !(a.parts && a.part_stride % 4)) {
    // (by N only, so that a row's sums do not depend on the step; the alignment is the same for every step's buffers)
    if (a.N <= 4096) return add_postnorm_vec_launch<T, 2, 512, true>(a, stream);
    if (a.N <= 8192) return add_postnorm_vec_launch<T, 4, 512, true>(a, stream);
    return add_postnorm_vec_launch<T, 4, 1024, false>(a, stream);
  }
  const size_t smem = (size_t)a.N * sizeof(float);
  if (smem > 200 * 1024) return GB_ERR_UNSUPPORTED;
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(add_postnorm_kernel<T>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
  }
  int threads = ((a.N + 3) / 4 + 31) / 32 * 32;   // by N only
  threads = threads < 64 ? 64 : (threads > 512 ? 512 : threads);
  return gb_launch(add_postnorm_kernel<T>, dim3(a.n_rows), dim3(threads), smem, stream, a);
}

GB_EXPORT int gb_add_postnorm_f32(const PostNormArgs* a, cudaStream_t s) {
  return add_postnorm_launch<float>(*a, s);
}
GB_EXPORT int gb_add_postnorm_bf16(const PostNormArgs* a, cudaStream_t s) {
  return add_postnorm_launch<bf16>(*a, s);
}
