// True 32-bit matrix product C[M, N] = A[M, K] . W[N, K]^T on the CUDA cores
// (FFMA only: no tensor cores, no TF32), the linear layer of the 32-bit path.
// Weights are row-major [out, in] and activations [tokens, in], as in the
// reference (src/cublas.rs:287-307 does the same product through cuBLAS).
//
// Every output element is summed over k = 0..K-1 in one fixed order, whatever M
// and N are and whichever kernel below runs, so a row's result does not depend on
// how many other rows the step holds.  The order is a sum of sums: fused
// multiply-adds over 32 consecutive k (a chain), 32 chains added in turn (a chunk
// of 1,024 k), and the chunks added in turn.  One chain over all of K would let the
// rounding error grow with sqrt(K): at K = 25,600 (the down projection of the widest
// model) that showed as 5e-5 on logits of order one, beyond the bar the 32-bit path
// is held to; in three levels the longest chain has 32 links.
//
// Two kernels share that order.
#include "common.cuh"

#include <cooperative_groups.h>
namespace cg = cooperative_groups;

#define CHAIN 32      // terms of one fused-multiply-add chain
#define CHUNK 1024    // terms of 32 chains, whose sums are added in turn

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 (or 4) bytes to shared memory; zeros when !in
__device__ __forceinline__ void copy16(void* dst, const float* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(in ? 16 : 0));
}
__device__ __forceinline__ void copy4(void* dst, const float* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(in ? 4 : 0));
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

// ---- few rows: the weights as one stream ------------------------------------
// Bound by reading W once.  A block of 16 ROWS_N threads takes ROWS_N weight rows and MT <= 8
// activation rows, a chunk of 1,024 k at a time, through a ring of cp.async stages (32 KB of
// weights each for eight rows; two blocks an SM keep up to 200 KB in flight).  The chains of a chunk are
// independent, so eight lanes of a warp hold eight chains and the other bits of the lane choose
// among the weight rows: warp w has chains 8 (w % 4) .. + 7 of rows 2g, 2g + 1, g = 4 (w / 4) + lane / 8.
// The chains' sums meet in shared memory, where one thread per output adds them in turn.  16-byte pieces
// are stored at piece ^ (chain % 8), so that eight lanes that read the same piece of eight chains touch
// all banks once.  Blocks are persistent over a whole number of tiles each.
// One row: 65,536 x 2,048 in 83 us (6.4 TB/s), 12,288 x 2,048 in 20, 2,048 x 2,048 in 5.4 (the tiles of the kernel
// before: 328 us on average over such a step's products); four rows 104, 26 and 6.7 us.
__device__ __forceinline__ int swizzled(int k) {   // float index of k in a chunk's row
  const int chain = k >> 5, piece = (k >> 2) & 7;
  return (chain << 5) | ((piece ^ (chain & 7)) << 2) | (k & 3);
}

// R rows of a [rows, ld] matrix into dst[R][CHUNK], columns k0 .. k0 + CHUNK; zeros outside
template <int R, int THREADS, bool VEC>
__device__ __forceinline__ void stage_rows(float* dst, const float* src, int row0, int rows, int k0, int K, int ld,
                                           int tid) {
  constexpr int PER = VEC ? 4 : 1;                    // floats a copy
  constexpr int STEPS = CHUNK / PER / THREADS;        // copies of a thread in one row
#pragma unroll
  for (int h = 0; h < STEPS; ++h) {
    const int k = (h * THREADS + tid) * PER;
    const float* p = src + (size_t)row0 * ld + k0 + k;
    float* d = dst + swizzled(k);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const bool in = row0 + r < rows && k0 + k < K;
      if (VEC) copy16(d + r * CHUNK, in ? p + (size_t)r * ld : src, in);
      else copy4(d + r * CHUNK, in ? p + (size_t)r * ld : src, in);
    }
  }
}

template <int MT, int ROWS_N, int ROWS_STAGES, bool VEC>
__global__ void __launch_bounds__(ROWS_N * 16)
f32_rows_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ C, int M, int N,
                int K, int lda, int ldw, int ldc, int tiles, int m_tiles, int settled) {
  constexpr int ROWS_THREADS = ROWS_N * 16;
  extern __shared__ float4 sm4[];
  float* sm = (float*)sm4;
  constexpr int STAGE = (ROWS_N + MT) * CHUNK;            // weights, then activations
  constexpr int OUTS = ROWS_N * MT;
  float* red = sm + ROWS_STAGES * STAGE;                  // [32 chains][OUTS + 1]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int chain = (warp & 3) * 8 + (lane & 7), g = (warp >> 2) * 4 + (lane >> 3);
  const int chunks = (K + CHUNK - 1) / CHUNK;
  const int mine = (tiles - (int)blockIdx.x + (int)gridDim.x - 1) / (int)gridDim.x;
  const int total_units = mine * chunks;                  // (tile, chunk) pairs, chunk fastest

  auto place = [&](int u, int& n0, int& m0, int& k0) {
    const int tile = blockIdx.x + (u / chunks) * gridDim.x;
    n0 = tile / m_tiles * ROWS_N, m0 = tile % m_tiles * MT, k0 = u % chunks * CHUNK;
  };
  // the first weights are asked for before the wait where no kernel still writes them
  if (!settled) pdl_wait();
#pragma unroll
  for (int s = 0; s < ROWS_STAGES; ++s) {
    if (s < total_units) {
      int n0, m0, k0;
      place(s, n0, m0, k0);
      stage_rows<ROWS_N, ROWS_THREADS, VEC>(sm + s * STAGE, W, n0, N, k0, K, ldw, tid);
    }
    copies_commit();
  }
  pdl_wait();
  // and their activations by plain loads, so that they do not queue behind all of those copies
#pragma unroll
  for (int s = 0; s < ROWS_STAGES; ++s) {
    if (s < total_units) {
      int n0, m0, k0;
      place(s, n0, m0, k0);
      float* x = sm + s * STAGE + ROWS_N * CHUNK;
      if (VEC) {
#pragma unroll
        for (int at = tid; at < MT * (CHUNK / 4); at += ROWS_THREADS) {
          const int r = at / (CHUNK / 4), k = (at % (CHUNK / 4)) * 4;
          float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
          if (m0 + r < M && k0 + k < K) v = *(const float4*)(A + (size_t)(m0 + r) * lda + k0 + k);
          *(float4*)(x + r * CHUNK + swizzled(k)) = v;
        }
      } else {
        for (int at = tid; at < MT * CHUNK; at += ROWS_THREADS) {
          const int r = at / CHUNK, k = at % CHUNK;
          x[r * CHUNK + swizzled(k)] = (m0 + r < M && k0 + k < K) ? A[(size_t)(m0 + r) * lda + k0 + k] : 0.f;
        }
      }
    }
  }

  float total = 0.f;
  int slot = 0;
  for (int u = 0; u < total_units; ++u) {
    copies_wait<ROWS_STAGES - 1>();
    __syncthreads();
    float* w_s = sm + slot * STAGE;
    const float* x_s = w_s + ROWS_N * CHUNK;
    float acc[2][MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[0][i] = acc[1][i] = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int at = (chain << 5) | ((j ^ (chain & 7)) << 2);
      const float4 w0 = *(const float4*)(w_s + (2 * g) * CHUNK + at);
      const float4 w1 = *(const float4*)(w_s + (2 * g + 1) * CHUNK + at);
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        const float4 x = *(const float4*)(x_s + i * CHUNK + at);
        acc[0][i] = fmaf(x.x, w0.x, acc[0][i]);
        acc[1][i] = fmaf(x.x, w1.x, acc[1][i]);
        acc[0][i] = fmaf(x.y, w0.y, acc[0][i]);
        acc[1][i] = fmaf(x.y, w1.y, acc[1][i]);
        acc[0][i] = fmaf(x.z, w0.z, acc[0][i]);
        acc[1][i] = fmaf(x.z, w1.z, acc[1][i]);
        acc[0][i] = fmaf(x.w, w0.w, acc[0][i]);
        acc[1][i] = fmaf(x.w, w1.w, acc[1][i]);
      }
    }
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      red[chain * (OUTS + 1) + i * ROWS_N + 2 * g] = acc[0][i];
      red[chain * (OUTS + 1) + i * ROWS_N + 2 * g + 1] = acc[1][i];
    }
    __syncthreads();   // everyone is done with the stage, and the chains' sums are there
    int n0, m0, k0;
    if (u + ROWS_STAGES < total_units) {
      place(u + ROWS_STAGES, n0, m0, k0);
      stage_rows<ROWS_N, ROWS_THREADS, VEC>(w_s, W, n0, N, k0, K, ldw, tid);
      stage_rows<MT, ROWS_THREADS, VEC>(w_s + ROWS_N * CHUNK, A, m0, M, k0, K, lda, tid);
    }
    copies_commit();
    if (tid < OUTS) {
      float mid = 0.f;
#pragma unroll
      for (int c = 0; c < 32; ++c) mid += red[c * (OUTS + 1) + tid];
      total += mid;
      if (u % chunks == chunks - 1) {
        place(u, n0, m0, k0);
        const int m = m0 + tid / ROWS_N, n = n0 + tid % ROWS_N;
        if (m < M && n < N) C[(size_t)m * ldc + n] = total;
        total = 0.f;
      }
    }
    slot = slot + 1 == ROWS_STAGES ? 0 : slot + 1;
  }
  pdl_launch_dependents();
}

// ---- more rows: register tiles ----------------------------------------------
// Bound by the FFMA rate (packed: one-by-one multiply-adds issue at half the rate here), of which it reaches 57 %
// (1,200 x 12,288 x 2,048 in 1.39 ms, 43 TFLOP/s; one-by-one 1.72).  Copies through a ring of cp.async stages that
// each thread reads back itself; a block of 128 threads makes a BM x BN tile, TM x TN outputs a thread, from k-major
// tiles of 16 k in shared memory (two buffers; the next tile waits in registers).  Two neighbouring columns are one
// packed multiply-add (fma.rn.f32x2: two independent roundings).  A chain's and a chunk's sums are in registers, the
// chunks' in C.  The k-major rows are stored at column ^ (8 (k / 4)), so that the
// transposing stores touch all banks once.  A cluster of blocks shares a tile, each
// with its own chunks, and adds them in turn through distributed shared memory, wherever K has more than one chunk and
// their sums leave room for a second block on the SM: by K alone, not by how many tiles there are.  With the kernel that the
// rule takes, shared / whole tiles, us: 128 rows x 2,048 of 2,048 55 / 94, 600 rows 168 / 197, 1,200 rows 285 / 313 (of
// 6,144 782 / 920), x 12,288 1,401 / 1,407; only 2,048 rows x 12,288 would gain (2,338 / 2,258).  (Activations stored
// twice, so that no register pair has to be made, were slower: 1.60 ms, shared memory then being the bound.)
#define TILE_K 16
#define TILE_THREADS 128
#define TILE_STAGES 3

typedef unsigned long long pair_t;   // two 32-bit floats
__device__ __forceinline__ pair_t both(float a) {
  pair_t r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ void fma2(pair_t& d, pair_t a, pair_t b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void add2(pair_t& d, pair_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }

template <int BM, int BN>
constexpr size_t tile_smem(int slots) {     // tiles, ring, and the chunks' sums where they do not fit in these
  return (size_t)((2 + TILE_STAGES) * TILE_K * (BM + BN) + (slots > 1 ? slots : 0) * BM * BN) * sizeof(float);
}

template <int BM, int BN, int TM, int TN, bool VEC>
__global__ void __launch_bounds__(TILE_THREADS)
f32_tile_kernel(const float* __restrict__ A, const float* __restrict__ W, float* C, int M, int N, int K, int lda,
                int ldw, int ldc, int split, int per_rank, int settled) {
  static_assert((BM / TM) * (BN / TN) == TILE_THREADS, "threads");
  static_assert((TM == 4 || TM == 8) && (TN == 4 || TN == 8), "outputs of a thread");
  static_assert(tile_smem<BM, BN>(1) >= BM * BN * sizeof(float), "one slot of sums fits where the tiles were");
  constexpr int LA = BM * TILE_K / 4 / TILE_THREADS, LW = BN * TILE_K / 4 / TILE_THREADS;
  constexpr int TXW = BN / TN >= 8 ? 8 : BN / TN;          // a warp's threads along the columns
  constexpr int TX = BN / TN;
  constexpr int PAIRS = TM * TN / 2;
  extern __shared__ float4 sm4[];
  float4* ring = sm4;                                      // [TILE_STAGES][LA + LW][TILE_THREADS]
  float* As = (float*)(ring + TILE_STAGES * (LA + LW) * TILE_THREADS);   // [2][TILE_K][BM]
  float* Ws = As + 2 * TILE_K * BM;                        // [2][TILE_K][BN]
  pair_t* sums = (pair_t*)(per_rank > 1 ? Ws + 2 * TILE_K * BN : (float*)sm4);   // [slots][PAIRS][TILE_THREADS]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tx = (warp % (TX / TXW)) * TXW + lane % TXW;
  const int ty = (warp / (TX / TXW)) * (32 / TXW) + lane / TXW;
  const int rank = blockIdx.x % split, m0 = blockIdx.x / split * BM, n0 = blockIdx.y * BN;
  const int lr = tid >> 2, lk = (tid & 3) * 4;             // this thread's row (+32 i) and k of a tile's copies

  const int chunks = (K + CHUNK - 1) / CHUNK;
  const int c_lo = rank * per_rank, c_hi = min(chunks, c_lo + per_rank);
  const int k_lo = c_lo * CHUNK, k_hi = min(K, c_hi * CHUNK);
  const int steps = (k_hi - k_lo + TILE_K - 1) / TILE_K;

  // A thread copies and reads back its own places of the ring, so only its own copies have to have landed.
  auto copy = [&](int s, int i, const float* src, int row, int rows, int ld) {
    float4* dst = ring + ((s % TILE_STAGES) * (LA + LW) + i) * TILE_THREADS + tid;
    const int k = k_lo + s * TILE_K + lk;
    const float* p = src + (size_t)row * ld + k;
    if (VEC) copy16(dst, row < rows && k < K ? p : src, row < rows && k < K);
    else
      for (int u = 0; u < 4; ++u)
        copy4((float*)dst + u, row < rows && k + u < K ? p + u : src, row < rows && k + u < K);
  };
  auto copy_w = [&](int s) {
#pragma unroll
    for (int i = 0; i < LW; ++i) copy(s, LA + i, W, n0 + lr + 32 * i, N, ldw);
  };
  auto copy_a = [&](int s) {
#pragma unroll
    for (int i = 0; i < LA; ++i) copy(s, i, A, m0 + lr + 32 * i, M, lda);
  };
  auto put = [&](int s) {      // tile s from the ring to its k-major buffer
    const float4* from = ring + (s % TILE_STAGES) * (LA + LW) * TILE_THREADS + tid;
    float* a = As + (s & 1) * TILE_K * BM;
    float* w = Ws + (s & 1) * TILE_K * BN;
#pragma unroll
    for (int i = 0; i < LA; ++i) {
      const int col = (lr + 32 * i) ^ (lk << 1);
      const float4 v = from[i * TILE_THREADS];
      a[(lk + 0) * BM + col] = v.x, a[(lk + 1) * BM + col] = v.y;
      a[(lk + 2) * BM + col] = v.z, a[(lk + 3) * BM + col] = v.w;
    }
#pragma unroll
    for (int i = 0; i < LW; ++i) {
      const int col = (lr + 32 * i) ^ (lk << 1);
      const float4 v = from[(LA + i) * TILE_THREADS];
      w[(lk + 0) * BN + col] = v.x, w[(lk + 1) * BN + col] = v.y;
      w[(lk + 2) * BN + col] = v.z, w[(lk + 3) * BN + col] = v.w;
    }
  };
  // output pair e of this thread: v, or v added to what is there
  auto store = [&](int e, pair_t v, bool add) {
    const int i = e / (TN / 2), j = e % (TN / 2);
    const int m = m0 + (i / 4) * (BM / 2) + ty * 4 + i % 4;
    const int n = n0 + (j / 2) * (BN / 2) + tx * 4 + (j % 2) * 2;
    if (m >= M) return;
    float* c = C + (size_t)m * ldc + n;
    float lo = __uint_as_float((uint32_t)v), hi = __uint_as_float((uint32_t)(v >> 32));
    if (n + 1 < N && !(((size_t)c) & 7)) {
      if (add) {
        const float2 was = *(float2*)c;
        lo = was.x + lo, hi = was.y + hi;
      }
      *(float2*)c = make_float2(lo, hi);
    } else {
      if (n < N) c[0] = add ? c[0] + lo : lo;
      if (n + 1 < N) c[1] = add ? c[1] + hi : hi;
    }
  };

  pair_t acc[TM][TN / 2], mid[TM][TN / 2];
#pragma unroll
  for (int i = 0; i < TM; ++i)
#pragma unroll
    for (int j = 0; j < TN / 2; ++j) acc[i][j] = mid[i][j] = 0ull;

  if (!settled) pdl_wait();
  for (int s = 0; s < TILE_STAGES; ++s)
    if (s < steps) copy_w(s);
  pdl_wait();
  for (int s = 0; s < TILE_STAGES; ++s) {
    if (s < steps) copy_a(s);
    copies_commit();
  }
  copies_wait<TILE_STAGES - 1>();
  put(0);
  if (TILE_STAGES < steps) copy_w(TILE_STAGES), copy_a(TILE_STAGES);
  copies_commit();
  __syncthreads();
  for (int s = 0; s < steps; ++s) {
    const float* a_s = As + (s & 1) * TILE_K * BM;
    const float* w_s = Ws + (s & 1) * TILE_K * BN;
#pragma unroll
    for (int k = 0; k < TILE_K; ++k) {
      const int x = (k >> 2) << 3;
      float a[TM];
      pair_t w[TN / 2];
#pragma unroll
      for (int h = 0; h < TM / 4; ++h)
        *(float4*)(a + 4 * h) = *(const float4*)(a_s + k * BM + ((h * (BM / 2) + ty * 4) ^ x));
#pragma unroll
      for (int h = 0; h < TN / 4; ++h)
        *(ulonglong2*)(w + 2 * h) = *(const ulonglong2*)(w_s + k * BN + ((h * (BN / 2) + tx * 4) ^ x));
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const pair_t aa = both(a[i]);
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], aa, w[j]);
      }
    }
    if ((s + 1) % (CHAIN / TILE_K) == 0 || s + 1 == steps) {        // the chains end here
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) add2(mid[i][j], acc[i][j]), acc[i][j] = 0ull;
    }
    if (s + 1 < steps) {
      if ((s + 1) % (CHUNK / TILE_K) == 0) {                        // and the chunk, with more to come
        const int c = s / (CHUNK / TILE_K);
#pragma unroll
        for (int e = 0; e < PAIRS; ++e) {
          pair_t& v = mid[e / (TN / 2)][e % (TN / 2)];
          if (split > 1) sums[((size_t)c * PAIRS + e) * TILE_THREADS + tid] = v;
          else store(e, v, c > 0);
          v = 0ull;
        }
      }
      copies_wait<TILE_STAGES - 1>();
      put(s + 1);
      if (s + 1 + TILE_STAGES < steps) copy_w(s + 1 + TILE_STAGES), copy_a(s + 1 + TILE_STAGES);
      copies_commit();
    }
    __syncthreads();
  }
  pdl_launch_dependents();

  const int last = (steps - 1) / (CHUNK / TILE_K);
  if (split == 1) {
#pragma unroll
    for (int e = 0; e < PAIRS; ++e) store(e, mid[e / (TN / 2)][e % (TN / 2)], last > 0);
    return;
  }
#pragma unroll
  for (int e = 0; e < PAIRS; ++e) sums[((size_t)last * PAIRS + e) * TILE_THREADS + tid] = mid[e / (TN / 2)][e % (TN / 2)];
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int e = rank; e < PAIRS; e += split) {
    pair_t v = 0ull;
    for (int c = 0; c < chunks; ++c) {
      const pair_t* from = cluster.map_shared_rank(sums, c / per_rank);
      add2(v, from[((size_t)(c % per_rank) * PAIRS + e) * TILE_THREADS + tid]);
    }
    store(e, v, false);
  }
  cluster.sync();     // the sums stay until every block of the cluster has read them
}

static int sm_count() {
  int dev = 0, n = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n;
}

template <int MT, int ROWS_N, int ROWS_STAGES, bool VEC>
static int launch_rows(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                       int sms, int settled, cudaStream_t stream) {
  constexpr size_t smem = (ROWS_STAGES * (ROWS_N + MT) * CHUNK + 32 * (ROWS_N * MT + 1)) * sizeof(float);
  auto* kernel = f32_rows_kernel<MT, ROWS_N, ROWS_STAGES, VEC>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return (int)e;
  const int m_tiles = (M + MT - 1) / MT;
  const long long tiles = (long long)((N + ROWS_N - 1) / ROWS_N) * m_tiles;
  if (tiles > (1 << 30)) return GB_ERR_UNSUPPORTED;
  const int fit = sms * (int)((227 * 1024) / (smem + 1024));
  const int each = (int)((tiles + fit - 1) / fit);           // whole tiles a block, as even as they come
  const int blocks = (int)((tiles + each - 1) / each);
  return gb_launch(kernel, dim3(blocks), dim3(ROWS_N * 16), smem, stream, A, W, C, M, N, K, lda, ldw, ldc,
                   (int)tiles, m_tiles, settled);
}

template <int BM, int BN, int TM, int TN, bool VEC>
static int launch_tile(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                       int settled, cudaStream_t stream) {
  const int chunks = (K + CHUNK - 1) / CHUNK;
  // one block for each chunk of a tile, or for a few where the cluster of eight would not do; sums of several chunks
  // take shared memory that two blocks of the large tile would not have
  int per_rank = (chunks + 7) / 8;
  int split = (chunks + per_rank - 1) / per_rank;
  if (split == 1 || (per_rank > 1 && tile_smem<BM, BN>(per_rank) > 113 * 1024)) split = 1, per_rank = chunks;
  const size_t smem = tile_smem<BM, BN>(split > 1 ? per_rank : 1);
  auto* kernel = f32_tile_kernel<BM, BN, TM, TN, VEC>;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  if (e != cudaSuccess) return (int)e;
  dim3 grid((M + BM - 1) / BM * split, (N + BN - 1) / BN);
  if (grid.y > 65535) return GB_ERR_UNSUPPORTED;
  return gb_launch_cluster(kernel, grid, dim3(TILE_THREADS), smem, stream, split, A, W, C, M, N, K, lda, ldw, ldc,
                           split, per_rank, settled);
}

template <bool VEC>
static int launch(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int kind,
                  int settled, cudaStream_t stream) {
  const int sms = sm_count();
  if (kind == 0) {
    // Measured on 2,048-wide layers (us; rows / small / medium / large): 16 rows x 12,288 62 / 70 / 98 / 121; 24 rows
    // x 2,048 19 / 39 / 47 / 75, x 12,288 90 / 70 / 98 / 121; 45 rows x 2,048 37 / 39 / 48 / 76, x 12,288 - / 115 /
    // 99 / 122; 600 rows x 2,048 - / 169 / 158 / 182, x 12,288 - / 904 / 775 / 734.  The stream of weights costs by
    // M / 8 passes over W, a tile by its 64 (32) rows whether they are there or not.
    // The stream takes any number of weight rows, the tiles as many as a grid has blocks.
    const double passes = (double)((M + 7) / 8) * N * K;
    if (M <= 16 || (M <= 48 && passes <= 4e7) || N > 65535 * 64) kind = 1;
    else if (M <= 32) kind = 2;
    else kind = (long long)((M + 63) / 64) * ((N + 127) / 128) >= 4 * sms ? 4 : 3;
  }
  switch (kind) {
    case 1:
      // two blocks an SM up to four rows (three stages for one), a larger block from there
      if (M <= 1) return launch_rows<1, 8, 3, VEC>(A, W, C, M, N, K, lda, ldw, ldc, sms, settled, stream);
      if (M <= 2) return launch_rows<2, 8, 2, VEC>(A, W, C, M, N, K, lda, ldw, ldc, sms, settled, stream);
      if (M <= 4) return launch_rows<4, 8, 2, VEC>(A, W, C, M, N, K, lda, ldw, ldc, sms, settled, stream);
      return launch_rows<8, 16, 2, VEC>(A, W, C, M, N, K, lda, ldw, ldc, sms, settled, stream);
    case 2: return launch_tile<32, 64, 4, 4, VEC>(A, W, C, M, N, K, lda, ldw, ldc, settled, stream);
    case 3: return launch_tile<64, 64, 8, 4, VEC>(A, W, C, M, N, K, lda, ldw, ldc, settled, stream);
    case 4: return launch_tile<64, 128, 8, 8, VEC>(A, W, C, M, N, K, lda, ldw, ldc, settled, stream);
  }
  return GB_ERR_BAD_ARG;
}

// kind: 0 chooses; 1 the stream of weights, 2, 3 and 4 the small, the medium and the large tile.  All give the same
// bits.  settled: no kernel that may still run writes W (a model's weights), so that its first tiles may be read before
// the kernel in front has finished.
GB_EXPORT int gb_gemm_nt_f32(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                             int kind, int settled, cudaStream_t stream) {
  if (M < 0 || N <= 0 || K <= 0 || lda < K || ldw < K || ldc < N) return GB_ERR_BAD_ARG;
  if (M == 0) return 0;
  // 16-byte loads want every row to start on 16 bytes and to end on a whole piece
  const bool vec = !(K % 4 || lda % 4 || ldw % 4 || ((size_t)A & 15) || ((size_t)W & 15));
  return vec ? launch<true>(A, W, C, M, N, K, lda, ldw, ldc, kind, settled, stream)
             : launch<false>(A, W, C, M, N, K, lda, ldw, ldc, kind, settled, stream);
}
