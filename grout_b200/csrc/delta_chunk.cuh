// The delta rule chunk by chunk: what the chunked forms of delta.cu (one decay per head) and channel_delta.cu (one per
// channel) share.  Both write the same record for every chunk of every head; with S_0 the state in front of a chunk,
//
//   U = U0 - W S_0;   S_n = diag(gC) S_0 + Kd^T U;   O = [e^L q | B] [S_0 ; U]
//
//   chain   walks a sequence's chunks in order, a block per head and COLS columns of S with the state in shared
//           memory: U and the next state, tiled 32-bit products; it leaves U and the state in front of every chunk
//           in the record
//   out     takes every chunk of every head at the same time: the read-outs, and their norm and gate
//
// The including file's arguments have cu_q, slots, state, state_stride, taps, H, dk, dv, n_seqs, norm_eps, norm_w, y and
// chunks, and for them cc_channels(a) (the convolved channels), cc_gate(a, t, h) (the gate's logits of a row and head),
// cc_gate_of(a, x), cc_out_done(a, seq, h) (called by a sequence's first block of every head), and, where a launch takes a
// part of the chunks only, the first of them cc_from(a), the end of them cc_to(a, chunks) and the place of a record
// cc_place(a, first, z, seq) (else 0, chunks and cc_entry).
#pragma once

#define CC_ROWS 32       // rows of a chunk
#define CC_MAX_DK 128
#define CC_MAX_DV 1024

// A chunk's record for one head: W [dk][32] (per channel the 32 rows) | Kd [32][dk] (e^{L_n - L} k) |
// gC [dk] (e^{L_n}) | QB [dk + 32][32] (per channel the rows of e^L q, then per row i the column of
// B) | SU [dk + 32][dv] (S_0, then U0, which becomes U)
__host__ __device__ __forceinline__ size_t cc_record(int dk, int dv) {
  return (size_t)2 * dk * CC_ROWS + dk + (size_t)(dk + CC_ROWS) * (CC_ROWS + dv);
}
__host__ __device__ __forceinline__ int cc_at_qb(int dk) { return 2 * dk * CC_ROWS + dk; }
__host__ __device__ __forceinline__ int cc_at_su(int dk) { return cc_at_qb(dk) + (dk + CC_ROWS) * CC_ROWS; }
// Chunk z of a sequence whose rows start at `first` has an entry that no other chunk has.
__host__ __device__ __forceinline__ size_t cc_entry(int first, int z, int seq) {
  return (size_t)(first / CC_ROWS + z + seq);
}

__device__ __forceinline__ void cc_copy16(float* smem, const float* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem));
}

// floats of a chain block's stage: W | Kd | gC | U0's columns
__host__ __device__ __forceinline__ int cc_stage(int dk, int cols) { return 2 * dk * CC_ROWS + dk + CC_ROWS * cols; }
__host__ __device__ __forceinline__ size_t cc_chain_smem(int dk, int cols) {   // two stages, S, partial sums, U
  return (size_t)(2 * cc_stage(dk, cols) + dk * cols + (128 / cols + 1) * CC_ROWS * cols) * sizeof(float);
}

// Bound by a chunk's chain of three steps with a barrier behind each and, in a block of 32 columns, by their
// multiply-adds; so where a step has few sequences and heads a block has 16 columns: 64 chunks of one sequence and 16
// heads of 128 in 149 us, 2.3 a chunk.  (Multiply-adds packed two by two were no faster, 140 us where one by one took 135:
// every pair of equal factors has to be made first.)
// The sums are taken so that no error grows beyond the row-by-row form's: W S in parts that are added up before they are
// subtracted, a chunk's share of the state before the state is added to it, the read-outs by 32 terms (135 us and 64
// for the read-outs otherwise, and with the products of the preparation in one chain the read-outs of 2,048 rows are
// 1.4e-7 off where row by row they are 1.04e-7, with slow decays 2.5e-7 where they are 1.55e-7; so 1.05e-7 and 1.53e-7).
template <typename Args, int COLS>
__global__ void __launch_bounds__(256) delta_chain_kernel(const Args a) {
  static_assert(COLS == 16 || COLS == 32, "columns of a block");
  extern __shared__ __align__(16) float sm[];
  constexpr int CT = COLS / 4;                   // threads along the columns of W S, four columns each
  constexpr int SPLITS = 256 / (8 * CT);         // parts of the channels' sum: 4 or 8
  constexpr int SC = COLS / 8;                   // columns of the state a thread updates
  pdl_launch_dependents_if_small();
  const int tid = threadIdx.x;
  const int h = blockIdx.y, seq = blockIdx.z, col0 = blockIdx.x * COLS;
  const int H = a.H, dk = a.dk, dv = a.dv, Cc = cc_channels(a);
  const int stage = cc_stage(dk, COLS);
  float* S = sm + 2 * stage;                     // [dk][COLS]
  float* P = S + dk * COLS;                      // [SPLITS][CC_ROWS][COLS]: a part of the channels' share of W S each
  float* U = P + SPLITS * CC_ROWS * COLS;        // [CC_ROWS][COLS]
  pdl_wait();
  const int first = a.cu_q[seq], n_seq = a.cu_q[seq + 1] - first;
  if (n_seq <= 0) return;
  const int slot = a.slots[seq];
  float* sp = slot >= 0 ? a.state + (size_t)slot * a.state_stride + (size_t)(a.taps - 1) * Cc + (size_t)h * dv * dk
                        : nullptr;
  const int z_lo = cc_from(a), z_hi = cc_to(a, (n_seq + CC_ROWS - 1) / CC_ROWS);
  if (z_lo >= z_hi) return;
  auto record = [&](int z) { return a.chunks + (cc_place(a, first, z, seq) * H + h) * cc_record(dk, dv); };
  const int whole = 2 * dk * CC_ROWS + dk;                 // (dk is a multiple of four)
  auto stage_in = [&](int z) {
    float* dst = sm + (z & 1) * stage;
    const float* src = record(z);
    for (int i = tid * 4; i < whole; i += 1024) cc_copy16(dst + i, src + i);
    const int t = tid / CT, c = (tid % CT) * 4;
    if (t < CC_ROWS && col0 + c < dv)
      cc_copy16(dst + whole + t * COLS + c, src + cc_at_su(dk) + (size_t)(dk + t) * dv + col0 + c);
    cp_async_commit();
  };
  for (int s = 0; s < 2 && col0 + COLS > dv; ++s)          // columns no copy brings
    for (int i = tid; i < CC_ROWS * COLS; i += 256)
      if (col0 + i % COLS >= dv) sm[s * stage + whole + i] = 0.f;
  stage_in(z_lo);
  // the state: element (k, c) of the head's matrix lies at c dk + k
  for (int i = tid; i < dk * COLS; i += 256) {
    const int c = i / dk, k = i % dk;
    S[k * COLS + c] = sp && col0 + c < dv ? sp[(size_t)(col0 + c) * dk + k] : 0.f;
  }
  // tiles: 4 rows by 4 columns of W S a thread, a part of the channels each; 4 rows by SC columns of the state
  const int part = tid / (8 * CT), tr = tid % (8 * CT) / CT * 4, tc = tid % CT * 4;
  const int per = (dk + SPLITS - 1) / SPLITS, k_lo = part * per, k_hi = min(dk, k_lo + per);
  const int sk = tid / 8 * 4, sc = tid % 8 * SC;
  const bool col_in = col0 + sc < dv;                      // (dv is a multiple of four)
  for (int z = z_lo; z < z_hi; ++z) {
    if (z + 1 < z_hi) { stage_in(z + 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
    __syncthreads();
    const float* w = sm + (z & 1) * stage;
    const float* kd = w + dk * CC_ROWS;
    const float* gc = kd + CC_ROWS * dk;
    const float* u0 = gc + dk;
    float* su = record(z) + cc_at_su(dk) + col0;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
#pragma unroll 8
    for (int k = k_lo; k < k_hi; ++k) {
      const float4 x = *reinterpret_cast<const float4*>(w + k * CC_ROWS + tr);
      const float xv[4] = {x.x, x.y, x.z, x.w};
      const float4 y = *reinterpret_cast<const float4*>(S + k * COLS + tc);
      const float yv[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(xv[i], yv[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *reinterpret_cast<float4*>(P + (part * CC_ROWS + tr + i) * COLS + tc) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    __syncthreads();
    for (int i = tid * 4; i < CC_ROWS * COLS; i += 1024) {  // U = U0 - W S, four columns of a row a thread
      float4 u = *reinterpret_cast<const float4*>(u0 + i);
      float4 x[SPLITS];
#pragma unroll
      for (int q = 0; q < SPLITS; ++q) x[q] = *reinterpret_cast<const float4*>(P + q * CC_ROWS * COLS + i);
#pragma unroll
      for (int n = SPLITS / 2; n > 0; n /= 2)
#pragma unroll
        for (int q = 0; q < n; ++q) x[q].x += x[q + n].x, x[q].y += x[q + n].y, x[q].z += x[q + n].z, x[q].w += x[q + n].w;
      u.x -= x[0].x, u.y -= x[0].y, u.z -= x[0].z, u.w -= x[0].w;
      *reinterpret_cast<float4*>(U + i) = u;
      if (col0 + i % COLS < dv) *reinterpret_cast<float4*>(su + (size_t)(dk + i / COLS) * dv + i % COLS) = u;
    }
    __syncthreads();
    if (sk < dk) {                               // S <- diag(gC) S + Kd^T U
      float s[4][SC], was[4][SC];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float* x = was[i];
        if constexpr (SC == 4) *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(S + (sk + i) * COLS + sc);
        else *reinterpret_cast<float2*>(x) = *reinterpret_cast<const float2*>(S + (sk + i) * COLS + sc);
        if (col_in) {
          float* to = su + (size_t)(sk + i) * dv + sc;
          if constexpr (SC == 4) *reinterpret_cast<float4*>(to) = *reinterpret_cast<const float4*>(x);
          else *reinterpret_cast<float2*>(to) = *reinterpret_cast<const float2*>(x);
        }
#pragma unroll
        for (int j = 0; j < SC; ++j) s[i][j] = 0.f;
      }
#pragma unroll 8
      for (int t = 0; t < CC_ROWS; ++t) {
        const float4 x = *reinterpret_cast<const float4*>(kd + t * dk + sk);
        const float xv[4] = {x.x, x.y, x.z, x.w};
        float y[SC];
        if constexpr (SC == 4) *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(U + t * COLS + sc);
        else *reinterpret_cast<float2*>(y) = *reinterpret_cast<const float2*>(U + t * COLS + sc);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < SC; ++j) s[i][j] = fmaf(xv[i], y[j], s[i][j]);
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float* to = S + (sk + i) * COLS + sc;
        const float g = gc[sk + i];
#pragma unroll
        for (int j = 0; j < SC; ++j) s[i][j] = fmaf(g, was[i][j], s[i][j]);
        if constexpr (SC == 4) *reinterpret_cast<float4*>(to) = make_float4(s[i][0], s[i][1], s[i][2], s[i][3]);
        else *reinterpret_cast<float2*>(to) = make_float2(s[i][0], s[i][1]);
      }
    }
    __syncthreads();                             // S is whole, the stage and P may be overwritten
  }
  pdl_launch_dependents_if_large();
  if (sp)
    for (int i = tid; i < dk * COLS; i += 256) {
      const int c = i / dk, k = i % dk;
      if (col0 + c < dv) sp[(size_t)(col0 + c) * dk + k] = S[k * COLS + c];
    }
}

// The read-outs of a chunk: [32 x (dk + 32)] times [(dk + 32) x dv], 128 columns at a time, a thread 4 rows
// (its warp's) by 4 columns, 32 elements of the sum staged together (two stages); then the norm
// over a row's dv numbers, the weight and the gate.
#define CO_COLS 128
#define CO_STAGE (CC_ROWS * (CC_ROWS + CO_COLS))
template <typename T, typename Args>
__global__ void __launch_bounds__(256, 4) delta_out_kernel(const Args a) {
  extern __shared__ __align__(16) float sm[];    // two stages [A: 32 x 32 | B: 32 x CO_COLS] | the read-outs [32][dv]
  pdl_launch_dependents_if_small();
  const int tid = threadIdx.x, lane = tid & 31, row = tid / 32 * 4;
  const int h = blockIdx.y, seq = blockIdx.z, z = cc_from(a) + blockIdx.x;
  const int H = a.H, dk = a.dk, dv = a.dv, K = dk + CC_ROWS;
  float* os = sm + 2 * CO_STAGE;
  pdl_wait();
  const int first = a.cu_q[seq], n = min(CC_ROWS, a.cu_q[seq + 1] - first - z * CC_ROWS);
  if (n <= 0) return;
  if (z == 0) cc_out_done(a, seq, h);
  const float* rec = a.chunks + (cc_place(a, first, z, seq) * H + h) * cc_record(dk, dv);
  const float* qb = rec + cc_at_qb(dk);
  const float* su = rec + cc_at_su(dk);
  const int tiles = (K + CC_ROWS - 1) / CC_ROWS, col_tiles = (dv + CO_COLS - 1) / CO_COLS;
  auto stage_in = [&](int s) {                   // stage s: column tile s / tiles, rows (s % tiles) 32 ..
    float* as = sm + (s & 1) * CO_STAGE;
    float* bs = as + CC_ROWS * CC_ROWS;
    const int k0 = s % tiles * CC_ROWS, c0 = s / tiles * CO_COLS;
    {
      const int k = tid / 8, r = (tid % 8) * 4;
      if (k0 + k < K) cc_copy16(as + k * CC_ROWS + r, qb + (size_t)(k0 + k) * CC_ROWS + r);
    }
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int k = tid / 32 + 8 * it, c = lane * 4;
      if (k0 + k < K && c0 + c < dv) cc_copy16(bs + k * CO_COLS + c, su + (size_t)(k0 + k) * dv + c0 + c);
    }
    cp_async_commit();
  };
  float acc[4][4];                               // the sum over the stages' sums
  stage_in(0);
  const int stages = tiles * col_tiles;
  for (int s = 0; s < stages; ++s) {
    if (s + 1 < stages) { stage_in(s + 1); cp_async_wait<1>(); } else { cp_async_wait<0>(); }
    __syncthreads();
    const float* as = sm + (s & 1) * CO_STAGE;
    const float* bs = as + CC_ROWS * CC_ROWS;
    if (s % tiles == 0) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
    }
    // The terms of U go up to a row's own: those of later rows, whose factors are zero, may not be finite.  (All bounds
    // are multiples of four: `below` terms are all four rows', the next four one row's less each.)
    const int k0 = s % tiles * CC_ROWS, nk = min(CC_ROWS, K - k0), own = dk + row - k0, below = max(0, min(nk, own));
    float part[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) part[i][j] = 0.f;
    const auto term = [&](int k, int from) {     // (columns beyond dv hold what no one reads)
      const float4 x = *reinterpret_cast<const float4*>(as + k * CC_ROWS + row);
      const float4 y = *reinterpret_cast<const float4*>(bs + k * CO_COLS + lane * 4);
      const float xv[4] = {x.x, x.y, x.z, x.w}, yv[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (i >= from) part[i][j] = fmaf(xv[i], yv[j], part[i][j]);
    };
    if (below == nk) {
#pragma unroll 8
      for (int k = 0; k < nk; ++k) term(k, 0);
    } else {
#pragma unroll 1
      for (int k = 0; k < below; k += 4)
#pragma unroll
        for (int u = 0; u < 4; ++u) term(k + u, 0);
      if (own >= 0)
#pragma unroll
        for (int u = 0; u < 4; ++u) term(own + u, u);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j];
    const int c = s / tiles * CO_COLS + lane * 4;
    if (s % tiles == tiles - 1 && c < dv) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(os + (row + i) * dv + c) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
    }
    __syncthreads();
  }
  pdl_launch_dependents_if_large();
#pragma unroll
  for (int i = 0; i < 4; ++i) {                  // (a warp finishes the rows it has made)
    const int r = row + i;
    if (r >= n) break;
    const size_t t = (size_t)first + z * CC_ROWS + r;
    float ss = 0.f;
    for (int j = lane; j < dv; j += 32) ss = fmaf(os[r * dv + j], os[r * dv + j], ss);
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)dv + a.norm_eps);
    const float* gate = cc_gate(a, t, h);
    T* y = (T*)a.y + (t * H + h) * dv;
    for (int j = lane; j < dv; j += 32) y[j] = from_f32<T>(os[r * dv + j] * inv * a.norm_w[j] * cc_gate_of(a, gate[j]));
  }
}

template <typename Args, int COLS>
static int delta_chain(const Args& a, cudaStream_t s) {
  size_t smem = cc_chain_smem(a.dk, COLS);
  const dim3 grid((a.dv + COLS - 1) / COLS, a.H, a.n_seqs);
  // a grid that has an SM for every block: one block an SM, wherever it finds room first (two would
  // halve each other's pace while other SMs stand idle)
  if ((long long)grid.x * grid.y * grid.z <= 148 && smem < 120 * 1024) smem = 120 * 1024;
  const cudaError_t e = cudaFuncSetAttribute(delta_chain_kernel<Args, COLS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)smem);
  if (e != cudaSuccess) return (int)e;
  return gb_launch(delta_chain_kernel<Args, COLS>, grid, dim3(256), smem, s, a);
}

// The two kernels behind the records of a launch that takes at most `chunks` chunks of every sequence.
template <typename T, typename Args>
static int delta_chain_and_out(const Args& a, int chunks, cudaStream_t s) {
  // 16 columns a block while that gives an SM at most one block
  const long long narrow = (long long)((a.dv + 15) / 16) * a.H * a.n_seqs;
  int e = narrow <= 148 ? delta_chain<Args, 16>(a, s) : delta_chain<Args, 32>(a, s);
  if (e) return e;
  const size_t smem = (2 * CO_STAGE + CC_ROWS * a.dv) * sizeof(float);
  const cudaError_t ce = cudaFuncSetAttribute(delta_out_kernel<T, Args>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                              (int)smem);
  if (ce != cudaSuccess) return (int)ce;
  return gb_launch(delta_out_kernel<T, Args>, dim3(chunks, a.H, a.n_seqs), dim3(256), smem, s, a);
}
