// The gated delta rule: a mixer whose memory is one matrix S [dk, dv] per head and
// sequence, updated token by token,
//
//   S <- g S;   u = beta (v - S^T k);   S <- S + k u^T;   o = S^T q
//
// with g in (0, 1) a decay per head and token, beta in (0, 1) a step size, k a
// unit vector and q a unit vector times dk^(-1/2).  q, k and v come out of short
// causal convolutions over time (one filter per channel, no bias, zeros before
// the sequence's start) followed by silu; the read-out o is RMS-normalised over
// dv, multiplied by a weight shared by the heads and by silu of a gate.
//
// Everything here is 32-bit whatever the activation type: the one projection
// that feeds it arrives as 32-bit sums, and only y, the o projection's input, is
// rounded.  Four kernels (and, further down, the forms of a decode step and of long prompts):
//
//   prepare  one block per token and kv head (its q and k) or run of value
//            channels: convolution (from the rows of this step and, for the first
//            tokens of a continued sequence, from the kept tail), silu, unit
//            vectors, beta, decay
//   gram     one block per group of 4 consecutive rows of a sequence and head: the
//            products k_i . k_j (i < j) and k_i . q_j (i <= j) inside the group, and
//            with them and the group's g and beta every scalar of the group that
//            does not depend on the column
//   scan     the recurrence.  The columns of S are independent recurrences, so a
//            column is held in the registers of 8 lanes (dk / 8 elements each),
//            16 columns a block, and a sequence's rows are walked in order, four
//            at a time: with c_j = g_1 .. g_j and s_0 the column before the group,
//              s_{j-1} . k_j = c_{j-1} (s_0 . k_j) + sum_{i<j} (c_{j-1} / c_i) (k_i . k_j) u_i
//              o_j = c_j (s_0 . q_j) + sum_{i<=j} (c_j / c_i) (k_i . q_j) u_i
//              s_4 = c_4 s_0 + sum_i (c_4 / c_i) k_i u_i
//            so the eight sums over dk that a group needs are taken from the column
//            as it stands, in one pass of shuffles, and what is sequential is a few
//            operations on scalars (the quotients are products of the g between, never
//            divisions).  The operands of 16 tokens at a time (their head's k and q,
//            the block's 16 values, beta, g, the group's products) reach shared memory
//            by asynchronous copies, two chunks in flight.  Groups are counted from the
//            first row a step brings, so a sequence cut elsewhere gives the same
//            result up to rounding, not bit for bit.
//   finish   one warp per (token, head): norm over dv, weight, gate; the block of a
//            sequence's first row then keeps the new tail of taps - 1 inputs
//
// Columns of the projection: q [G dk] | k [G dk] | v [H dv] | gate [H dv] | b [H] | a [H].
// A sequence's state is one row of floats: the tail [taps - 1, Cc] (Cc = the
// convolved channels q | k | v), then S as [H, dv, dk], a column's dk elements
// side by side.  Rows of slot < 0 (padding) read zeros and store nothing.
#include "attn_mma.cuh"   // the asynchronous-copy helpers
#include "short_conv.cuh"

struct DeltaArgs {
  const float* proj;       // [n_tokens, C_all]
  const float* conv_w;     // [Cc, taps], the last column is the current token's
  const float* a_log;      // [H]
  const float* dt_bias;    // [H]
  const float* norm_w;     // [dv]
  const int* token_seq;    // [n_tokens]
  const int* cu_q;         // [n_seqs + 1]
  const int* slots;        // [n_seqs]
  float* state;            // [slots, state_stride]
  long long state_stride;
  float* prep;             // [n_tokens, prep_stride]: unit q | unit k | v | beta | decay | (pad to 4) |
                           //   on a group's first row: its scalars [H, 48]
  float* o;                // [n_tokens, H, dv]
  void* y;                 // [n_tokens, H dv] in the activation type
  int n_tokens, n_seqs, H, G, dk, dv, taps;
  float unit_eps, norm_eps;
  int prep_stride;         // floats between rows of prep: round4(Cc + 2 H) + 48 H
  int few_rows;            // 1: no sequence brings more than DELTA_B rows, 2: none more than one (a decode
                           //   step): the scan works out its one group's scalars itself, `gram` is not launched
  int max_rows;            // the most rows any sequence brings (0: unknown)
  float* chunks;           // scratch of a step that goes chunk by chunk, or null: [n_tokens / 32 + n_seqs, H, record], or
                           //   with `window` [group, window, H, record]
  int group, window;       // window > 0: the step goes by `group` sequences and `window` of their chunks at a time
  int z0;                  // the first chunk of the launch's window
};

__device__ __forceinline__ void delta_keep_tail(const DeltaArgs& a, int seq, int first, int step);
__device__ __forceinline__ int cc_channels(const DeltaArgs& a) { return 2 * a.G * a.dk + a.H * a.dv; }
__device__ __forceinline__ const float* cc_gate(const DeltaArgs& a, size_t t, int h) {
  const int Cc = cc_channels(a);
  return a.proj + t * (Cc + a.H * a.dv + 2 * a.H) + Cc + (size_t)h * a.dv;
}
__device__ __forceinline__ float cc_gate_of(const DeltaArgs&, float x) { return silu_f(x); }
// (every reader of the old tail, the prepare kernel, has finished)
__device__ __forceinline__ void cc_out_done(const DeltaArgs& a, int seq, int h) {
  delta_keep_tail(a, seq, h * blockDim.x + threadIdx.x, a.H * blockDim.x);
}
#include "delta_chunk.cuh"
__device__ __forceinline__ int cc_from(const DeltaArgs& a) { return a.z0; }
__device__ __forceinline__ int cc_to(const DeltaArgs& a, int chunks) {
  return a.window ? min(chunks, a.z0 + a.window) : chunks;
}
__device__ __forceinline__ size_t cc_place(const DeltaArgs& a, int first, int z, int seq) {
  return a.window ? (size_t)seq * a.window + (z - a.z0) : cc_entry(first, z, seq);
}

// One block per (token, unit): unit g < G is kv head g's q and k together, the units after that are runs of
// DELTA_PREP_V value channels; the block of unit 0 also takes beta and the decay.
#define DELTA_PREP_V 256

__device__ __forceinline__ float delta_conv(const DeltaArgs& a, const float* tail, int t, int r,
                                            int c, int Cc, int C_all) {
  return short_conv_silu(a.proj, C_all, a.conv_w, a.taps, tail, Cc, t, r, c);
}

__global__ void __launch_bounds__(256) delta_prepare_kernel(const DeltaArgs a) {
  extern __shared__ float row[];   // [2 dk]: a kv head's q and k after the convolution
  __shared__ float scratch[32];
  pdl_launch_dependents_if_small();
  const int t = blockIdx.x, unit = blockIdx.y, tid = threadIdx.x;
  const int H = a.H, G = a.G, dk = a.dk, dv = a.dv;
  const int Cc = 2 * G * dk + H * dv, C_all = Cc + H * dv + 2 * H, P = a.prep_stride;
  const int seq = a.token_seq[t];
  const int slot = a.slots[seq];
  const int r = t - a.cu_q[seq];                 // the token's place among its sequence's rows
  const float* tail = slot >= 0 ? a.state + (size_t)slot * a.state_stride : nullptr;
  float* out = a.prep + (size_t)t * P;
  pdl_wait();
  if (unit >= G) {                               // value channels: convolution and silu
    const int c = 2 * G * dk + (unit - G) * DELTA_PREP_V + tid;
    if (tid < DELTA_PREP_V && c < Cc) out[c] = delta_conv(a, tail, t, r, c, Cc, C_all);
    return;
  }
  float sq = 0.f, sk = 0.f;
  for (int i = tid; i < 2 * dk; i += blockDim.x) {
    const int c = i < dk ? unit * dk + i : (G + unit) * dk + (i - dk);
    const float v = delta_conv(a, tail, t, r, c, Cc, C_all);
    row[i] = v;
    if (i < dk) sq += v * v; else sk += v * v;
  }
  sq = block_sum(sq, scratch);
  sk = block_sum(sk, scratch);
  const float iq = 1.0f / sqrtf(sq + a.unit_eps) * (1.0f / sqrtf((float)dk));
  const float ik = 1.0f / sqrtf(sk + a.unit_eps);
  for (int d = tid; d < dk; d += blockDim.x) {
    out[unit * dk + d] = row[d] * iq;
    out[(G + unit) * dk + d] = row[dk + d] * ik;
  }
  if (unit == 0) {
    for (int h = tid; h < H; h += blockDim.x) {
      const float b = a.proj[(size_t)t * C_all + Cc + H * dv + h];
      const float al = a.proj[(size_t)t * C_all + Cc + H * dv + H + h];
      out[Cc + h] = 1.0f / (1.0f + expf(-b));
      out[Cc + H + h] = expf(-expf(a.a_log[h]) * softplus_f(al + a.dt_bias[h]));
    }
  }
  pdl_launch_dependents_if_large();
}

// The same for steps of many rows: a block takes a run of DP_RUN rows, a thread a channel of them (q and k of one kv
// head, or 256 value channels), so an input is read once instead of once for each tap, all of a run's are on
// their way together, and the sums of squares of all rows meet behind one barrier.  Bound by memory; 2,048 rows of 4,096
// channels 32 us (80 with a block a row).  From 256 rows on, eight a sequence: a whole rule of 100 rows takes 47 us with
// runs and 43 without (16 heads of 128), 64 sequences of one and two rows 106 and 92, 316 rows in 61 sequences 200 and
// 190, 256 rows 86 and 88, 63 sequences of 16 rows 203 and 220.
#define DP_RUN 16
#define DP_TAPS 8
__global__ void __launch_bounds__(256) delta_prepare_rows_kernel(const DeltaArgs a) {
  __shared__ float sums[DP_RUN][8];
  pdl_launch_dependents_if_small();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, unit = blockIdx.y;
  const int H = a.H, G = a.G, dk = a.dk, dv = a.dv, taps = a.taps;
  const int Cc = 2 * G * dk + H * dv, C_all = Cc + H * dv + 2 * H, P = a.prep_stride;
  const bool qk = unit < G, is_q = tid < dk;
  const int c = !qk ? 2 * G * dk + (unit - G) * 256 + tid : is_q ? unit * dk + tid : (G + unit) * dk + (tid - dk);
  const bool mine = qk ? tid < 2 * dk : c < Cc;
  if (mine) prefetch_l2(a.conv_w + (size_t)c * taps);
  int seq, run;
  run_of_block(a.cu_q, a.n_seqs, DP_RUN, false, blockIdx.x, seq, run);
  const int first = a.cu_q[seq], n = min(DP_RUN, a.cu_q[seq + 1] - first - run * DP_RUN), row0 = first + run * DP_RUN;
  if (n <= 0) return;
  const int slot = a.slots[seq];
  pdl_wait();
  float w[DP_TAPS];                    // [j] meets the input j rows back
#pragma unroll
  for (int j = 0; j < DP_TAPS; ++j) w[j] = mine && j < taps ? a.conv_w[(size_t)c * taps + taps - 1 - j] : 0.f;
  float x[DP_RUN + DP_TAPS - 1];       // the DP_TAPS - 1 inputs in front of the run, then the run's
#pragma unroll
  for (int i = 0; i < DP_TAPS - 1; ++i) {
    const int back = DP_TAPS - 1 - i;  // so many rows in front of the run's first
    x[i] = 0.f;
    if (!mine || back >= taps) continue;
    if (run > 0) x[i] = a.proj[(size_t)(row0 - back) * C_all + c];
    else if (slot >= 0) x[i] = a.state[(size_t)slot * a.state_stride + (size_t)(taps - 1 - back) * Cc + c];
  }
#pragma unroll
  for (int i = 0; i < DP_RUN; ++i) x[DP_TAPS - 1 + i] = mine && i < n ? a.proj[(size_t)(row0 + i) * C_all + c] : 0.f;
  float y[DP_RUN];
#pragma unroll
  for (int i = 0; i < DP_RUN; ++i) {
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < DP_TAPS; ++j) acc = fmaf(w[j], x[DP_TAPS - 1 + i - j], acc);
    y[i] = silu_f(acc);
  }
  float* out = a.prep + (size_t)row0 * P + c;
  if (!qk) {
#pragma unroll
    for (int i = 0; i < DP_RUN; ++i)
      if (mine && i < n) out[(size_t)i * P] = y[i];
    return;
  }
#pragma unroll
  for (int i = 0; i < DP_RUN; ++i) {   // (a warp is all q, all k or idle)
    const float ss = warp_sum(mine ? y[i] * y[i] : 0.f);
    if (lane == 0) sums[i][warp] = ss;
  }
  __syncthreads();
  const int w0 = is_q ? 0 : dk / 32;
  const float scale = is_q ? 1.0f / sqrtf((float)dk) : 1.0f;
#pragma unroll
  for (int i = 0; i < DP_RUN; ++i) {
    float ss = 0.f;
    for (int u = 0; u < dk / 32; ++u) ss += sums[i][min(7, w0 + u)];
    if (mine && i < n) out[(size_t)i * P] = y[i] * (1.0f / sqrtf(ss + a.unit_eps) * scale);
  }
  if (unit == 0)
    for (int i = tid; i < n * H; i += 256) {
      const int t = row0 + i / H, h = i % H;
      const float* row = a.proj + (size_t)t * C_all + Cc + H * dv;
      a.prep[(size_t)t * P + Cc + h] = 1.0f / (1.0f + expf(-row[h]));
      a.prep[(size_t)t * P + Cc + H + h] = expf(-expf(a.a_log[h]) * softplus_f(row[H + h] + a.dt_bias[h]));
    }
  pdl_launch_dependents_if_large();
}

// The new tail of a sequence; the caller's threads share the channels: first, first + step, ...
__device__ __forceinline__ void delta_keep_tail(const DeltaArgs& a, int seq, int first, int step) {
  const int slot = a.slots[seq];
  const int row0 = a.cu_q[seq], n = a.cu_q[seq + 1] - row0;
  if (slot < 0 || n <= 0) return;
  const int Cc = 2 * a.G * a.dk + a.H * a.dv, C_all = Cc + a.H * a.dv + 2 * a.H;
  short_conv_keep_tail(a.proj, C_all, a.taps, a.state + (size_t)slot * a.state_stride, Cc, row0, n, first, step);
}

#define DELTA_LANES 8       // lanes that share a column of S
#define DELTA_COLS 16       // columns of S per block
#define DELTA_TT 16         // tokens whose operands are staged together
#define DELTA_B 4           // rows of a group

__host__ __device__ __forceinline__ int delta_gram_offset(int Cc, int H) { return (Cc + 2 * H + 3) / 4 * 4; }

// The scalars of a group of DELTA_B rows and one head that do not depend on the column
// (c_j = g_1 .. g_j, c_0 = 1; quotients c_j / c_i are products of the g between):
//   [0, 4)   A_j  = beta_j g_j c_{j-1}                       u_j = beta_j v_j - A_j (s_0 . k_j)
//   [4, 20)  C_ij = beta_j g_j (c_{j-1} / c_i) (k_i . k_j)          - sum_{i<j} C_ij u_i
//   [20, 24) c_j                                              o_j = c_j (s_0 . q_j)
//   [24, 40) D_ij = (c_j / c_i) (k_i . q_j)                         + sum_{i<=j} D_ij u_i
//   [40, 44) E_i  = c_4 / c_i                                 s_4 = c_4 s_0 + sum_i E_i u_i k_i
//   [44, 48) beta_j
// Rows beyond the sequence's end are neutral (beta 0, g 1, products 0).
#define DELTA_COEF 48
// Where the pieces lie for groups of B rows (B = 4: the table above); the whole is filled up
// to a multiple of four floats.
template <int B> struct DeltaCoef {
  static constexpr int A = 0, C = B, CUM = B + B * B, D = 2 * B + B * B, E = 2 * B + 2 * B * B,
                       BETA = 3 * B + 2 * B * B, SIZE = (4 * B + 2 * B * B + 3) / 4 * 4;
};
static_assert(DeltaCoef<DELTA_B>::SIZE == DELTA_COEF, "the scalars of a group of four rows are 48 floats");

template <int B>
__device__ __forceinline__ void delta_group_scalars(float* out, const float* dots,
                                                    const float (&beta)[B], const float (&g)[B]) {
  using L = DeltaCoef<B>;
  float quot[B][B], cum[B + 1];
  cum[0] = 1.f;
  for (int j = 0; j < B; ++j) {
    cum[j + 1] = cum[j] * g[j];
    quot[j][j] = 1.f;
    for (int i = 0; i < j; ++i) quot[i][j] = quot[i][j - 1] * g[j];
  }
  for (int j = 0; j < B; ++j) {
    out[L::A + j] = beta[j] * g[j] * cum[j];
    out[L::CUM + j] = cum[j + 1];
    out[L::E + j] = quot[j][B - 1];
    out[L::BETA + j] = beta[j];
    for (int i = 0; i < B; ++i) {
      out[L::C + i * B + j] = i < j ? beta[j] * g[j] * quot[i][j - 1] * dots[i * B + j] : 0.f;
      out[L::D + i * B + j] = i <= j ? quot[i][j] * dots[B * B + i * B + j] : 0.f;
    }
  }
}

__global__ void __launch_bounds__(128) delta_gram_kernel(const DeltaArgs a) {
  __shared__ float dots[2 * DELTA_B * DELTA_B];
  pdl_launch_dependents_if_small();
  constexpr int B = DELTA_B;
  const int t = blockIdx.x, h = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int G = a.G, H = a.H, dk = a.dk, P = a.prep_stride;
  const int Cc = 2 * G * dk + H * a.dv, kvh = h / (H / G);
  const int seq = a.token_seq[t];
  const int row0 = a.cu_q[seq], r = t - row0;
  if (r % B) return;
  const int nb = min(B, a.cu_q[seq + 1] - t);
  pdl_wait();
  for (int e = warp; e < 2 * B * B; e += 4) {       // e < 16: k_i . k_j, else k_i . q_j
    const int with_q = e / (B * B), i = (e % (B * B)) / B, j = e % B;
    float acc = 0.f;
    if (i < nb && j < nb && (with_q ? i <= j : i < j)) {
      const float* ki = a.prep + (size_t)(t + i) * P + (G + kvh) * dk;
      const float* xj = a.prep + (size_t)(t + j) * P + (with_q ? kvh : G + kvh) * dk;
      for (int d = lane; d < dk; d += 32) acc = fmaf(ki[d], xj[d], acc);
      acc = warp_sum(acc);
    }
    if (lane == 0) dots[e] = acc;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    float beta[B], g[B];
    for (int j = 0; j < B; ++j) {
      beta[j] = j < nb ? a.prep[(size_t)(t + j) * P + Cc + h] : 0.f;
      g[j] = j < nb ? a.prep[(size_t)(t + j) * P + Cc + H + h] : 1.f;
    }
    delta_group_scalars<DELTA_B>(a.prep + (size_t)t * P + delta_gram_offset(Cc, H) + h * DELTA_COEF, dots, beta, g);
  }
  pdl_launch_dependents_if_large();
}

__device__ __forceinline__ void cp_async4(void* smem, const void* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(s), "l"(gmem));
}

// R floats of a column per lane, in pieces of four: piece i of lane l holds the
// elements (i * 8 + l) * 4 .. + 3, so that the lanes of a column read contiguous
// bytes of shared memory, and of the state, at a time.
// B = 4 rows a turn; B = 1 for a step in which every sequence brings one row (a decode step):
// one staged row, one group, far fewer registers, so that more of its many short blocks fit an SM.
template <int R, int B>
__global__ void __launch_bounds__(DELTA_LANES * DELTA_COLS) delta_scan_kernel(const DeltaArgs a) {
  extern __shared__ __align__(16) float sm[];
  using L = DeltaCoef<B>;
  constexpr int TT = B == 1 ? 1 : DELTA_TT;            // rows of a stage
  constexpr int DKP = DELTA_LANES * R;                       // dk filled up with zeros
  constexpr int GRAM = L::SIZE;
  // q | k | v | the groups' scalars
  constexpr int STAGE = TT * (2 * DKP + DELTA_COLS) + (TT / B) * GRAM;
  pdl_launch_dependents_if_small();
  const int seq = blockIdx.z, h = blockIdx.y, tid = threadIdx.x;
  const int col0 = blockIdx.x * DELTA_COLS;
  const int col = col0 + tid / DELTA_LANES, l = tid % DELTA_LANES;
  const int H = a.H, G = a.G, dk = a.dk, dv = a.dv;
  const int Cc = 2 * G * dk + H * dv, P = a.prep_stride;
  const int gram_off = delta_gram_offset(Cc, H);
  const int kvh = h / (H / G);
  const bool active = col < dv;
  if (dk < DKP)   // what no copy writes stays zero (a step of few rows has one stage only)
    for (int i = tid; i < (a.few_rows ? 1 : 2) * STAGE; i += blockDim.x) sm[i] = 0.f;
  pdl_wait();
  const int row0 = a.cu_q[seq], n = a.cu_q[seq + 1] - row0;
  if (n <= 0) return;
  __syncthreads();
  const int slot = a.slots[seq];
  float* sp = slot >= 0 && active
                  ? a.state + (size_t)slot * a.state_stride + (size_t)(a.taps - 1) * Cc +
                        ((size_t)h * dv + col) * dk
                  : nullptr;
  const bool wide = (dk & 3) == 0;     // 16-byte copies; prep rows are 16-byte aligned
  const bool wide_state = wide && sp && (((uintptr_t)sp) & 15) == 0;
  float S[R];
#pragma unroll
  for (int i = 0; i < R / 4; ++i) {
    const int e = (i * DELTA_LANES + l) * 4;
    if (wide_state) {
      const float4 x = e < dk ? *reinterpret_cast<const float4*>(sp + e) : make_float4(0.f, 0.f, 0.f, 0.f);
      S[4 * i] = x.x, S[4 * i + 1] = x.y, S[4 * i + 2] = x.z, S[4 * i + 3] = x.w;
    } else {
#pragma unroll
      for (int x = 0; x < 4; ++x) S[4 * i + x] = sp && e + x < dk ? sp[e + x] : 0.f;
    }
  }
  const int warp = tid >> 5, lane = tid & 31, nwarps = blockDim.x >> 5;
  auto stage_in = [&](int chunk, int st) {
    float* base = sm + st * STAGE;
    float* vs = base + 2 * TT * DKP;
    float* gr = vs + TT * DELTA_COLS;
    const int t0 = row0 + chunk * TT;
    const int nt = min(TT, row0 + n - t0);
    for (int tt = warp; tt < nt; tt += nwarps) {          // a warp per token: its q, its k, its values
      const float* src = a.prep + (size_t)(t0 + tt) * P;
      if (wide) {
        for (int pc = lane; pc < dk / 4; pc += 32) {
          cp_async16(base + tt * DKP + pc * 4, src + kvh * dk + pc * 4, true);
          cp_async16(base + (TT + tt) * DKP + pc * 4, src + (G + kvh) * dk + pc * 4, true);
        }
      } else {
        for (int d = lane; d < dk; d += 32) {
          cp_async4(base + tt * DKP + d, src + kvh * dk + d);
          cp_async4(base + (TT + tt) * DKP + d, src + (G + kvh) * dk + d);
        }
      }
      if (lane < DELTA_COLS && col0 + lane < dv)
        cp_async4(vs + tt * DELTA_COLS + lane, src + 2 * G * dk + h * dv + col0 + lane);
    }
    if (!a.few_rows)
      for (int gi = warp; gi * B < nt; gi += nwarps)      // a warp per group: its scalars
        for (int e = lane; e < GRAM / 4; e += 32)
          cp_async16(gr + gi * GRAM + e * 4, a.prep + (size_t)(t0 + gi * B) * P + gram_off + h * GRAM + e * 4, true);
    cp_async_commit();
    const int fill = ((nt + B - 1) / B) * B - nt;   // the sequence ends inside a group: its other rows are zeros
    if (fill > 0) {
      for (int i = tid; i < fill * DKP; i += blockDim.x) {
        base[nt * DKP + i] = 0.f;
        base[(TT + nt) * DKP + i] = 0.f;
      }
      for (int i = tid; i < fill * DELTA_COLS; i += blockDim.x) vs[nt * DELTA_COLS + i] = 0.f;
    }
  };
  const int n_chunks = (n + TT - 1) / TT;
  float beta_f[B], g_f[B];      // a step of few rows: the one group's beta and g, asked for early
#pragma unroll
  for (int j = 0; j < B; ++j) {
    beta_f[j] = 0.f, g_f[j] = 1.f;
    if (a.few_rows && tid == 0 && j < n) {
      beta_f[j] = a.prep[(size_t)(row0 + j) * P + Cc + h];
      g_f[j] = a.prep[(size_t)(row0 + j) * P + Cc + H + h];
    }
  }
  stage_in(0, 0);
  for (int c = 0; c < n_chunks; ++c) {
    const int st = c & 1;
    if (c + 1 < n_chunks) {
      stage_in(c + 1, st ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float* base = sm + st * STAGE;
    const float* vs = base + 2 * TT * DKP;
    const float* gr = vs + TT * DELTA_COLS;
    const int t0 = row0 + c * TT;
    const int nt = min(TT, row0 + n - t0);
    if (a.few_rows) {       // the one group's products from the staged rows, then its scalars
      __shared__ float dots[2 * B * B];
      for (int e = warp; e < 2 * B * B; e += nwarps) {
        const int with_q = e / (B * B), i = (e % (B * B)) / B, j = e % B;
        float acc = 0.f;
        if (i < nt && j < nt && (with_q ? i <= j : i < j)) {
          const float* ki = base + (TT + i) * DKP;
          const float* xj = base + (with_q ? j : TT + j) * DKP;
          for (int d = lane; d < dk; d += 32) acc = fmaf(ki[d], xj[d], acc);
          acc = warp_sum(acc);
        }
        if (lane == 0) dots[e] = acc;
      }
      __syncthreads();
      if (tid == 0)
        delta_group_scalars<B>(sm + st * STAGE + 2 * TT * DKP + TT * DELTA_COLS, dots, beta_f, g_f);
      __syncthreads();
    }
    for (int g0 = 0; g0 < nt; g0 += B) {
      float k[B][R], sk[B], sq[B];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        const float4* qp = reinterpret_cast<const float4*>(base + (g0 + j) * DKP) + l;
        const float4* kp = reinterpret_cast<const float4*>(base + (TT + g0 + j) * DKP) + l;
        float d1 = 0.f, d2 = 0.f;
#pragma unroll
        for (int i = 0; i < R / 4; ++i) {
          const float4 kk = kp[i * DELTA_LANES], qq = qp[i * DELTA_LANES];
          k[j][4 * i] = kk.x, k[j][4 * i + 1] = kk.y, k[j][4 * i + 2] = kk.z, k[j][4 * i + 3] = kk.w;
          d1 = fmaf(S[4 * i], kk.x, d1), d1 = fmaf(S[4 * i + 1], kk.y, d1);
          d1 = fmaf(S[4 * i + 2], kk.z, d1), d1 = fmaf(S[4 * i + 3], kk.w, d1);
          d2 = fmaf(S[4 * i], qq.x, d2), d2 = fmaf(S[4 * i + 1], qq.y, d2);
          d2 = fmaf(S[4 * i + 2], qq.z, d2), d2 = fmaf(S[4 * i + 3], qq.w, d2);
        }
        sk[j] = d1, sq[j] = d2;
      }
#pragma unroll
      for (int m = 1; m < DELTA_LANES; m <<= 1)
#pragma unroll
        for (int j = 0; j < B; ++j) {
          sk[j] += __shfl_xor_sync(0xffffffffu, sk[j], m);
          sq[j] += __shfl_xor_sync(0xffffffffu, sq[j], m);
        }
      // what is left of the group's scalars depends on the column: every lane computes the same
      const float4* cf = reinterpret_cast<const float4*>(gr + (g0 / B) * GRAM);
      float co[GRAM];
#pragma unroll
      for (int i = 0; i < GRAM / 4; ++i) {
        const float4 x = cf[i];
        co[4 * i] = x.x, co[4 * i + 1] = x.y, co[4 * i + 2] = x.z, co[4 * i + 3] = x.w;
      }
      float u[B], w[B];
#pragma unroll
      for (int j = 0; j < B; ++j) {
        const float v = vs[(g0 + j) * DELTA_COLS + (tid / DELTA_LANES)];
        float uj = fmaf(co[L::BETA + j], v, -co[L::A + j] * sk[j]);
#pragma unroll
        for (int i = 0; i < j; ++i) uj = fmaf(-co[L::C + i * B + j], u[i], uj);
        u[j] = uj;
        float o = co[L::CUM + j] * sq[j];
#pragma unroll
        for (int i = 0; i <= j; ++i) o = fmaf(co[L::D + i * B + j], u[i], o);
        if (l == 0 && active && g0 + j < nt) a.o[((size_t)(t0 + g0 + j) * H + h) * dv + col] = o;
      }
#pragma unroll
      for (int i = 0; i < B; ++i) w[i] = co[L::E + i] * u[i];
      const float cum = co[L::CUM + B - 1];
#pragma unroll
      for (int x = 0; x < R; ++x) {
        float sx = cum * S[x];
#pragma unroll
        for (int i = 0; i < B; ++i) sx = fmaf(k[i][x], w[i], sx);
        S[x] = sx;
      }
    }
    __syncthreads();   // the stage is refilled by the next turn's copies
  }
  pdl_launch_dependents_if_large();
  if (sp) {
#pragma unroll
    for (int i = 0; i < R / 4; ++i) {
      const int e = (i * DELTA_LANES + l) * 4;
      if (wide_state) {
        if (e < dk) *reinterpret_cast<float4*>(sp + e) = make_float4(S[4 * i], S[4 * i + 1], S[4 * i + 2], S[4 * i + 3]);
      } else {
#pragma unroll
        for (int x = 0; x < 4; ++x)
          if (e + x < dk) sp[e + x] = S[4 * i + x];
      }
    }
  }
}

template <typename T>
__global__ void delta_finish_kernel(const DeltaArgs a) {
  pdl_launch_dependents_if_small();
  pdl_wait();
  const int t = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nwarps = blockDim.x >> 5;
  const int H = a.H, dv = a.dv;
  const int Cc = 2 * a.G * a.dk + H * dv, C_all = Cc + H * dv + 2 * H;
  for (int h = blockIdx.y * nwarps + warp; h < H; h += gridDim.y * nwarps) {
    const float* o = a.o + ((size_t)t * H + h) * dv;
    const float* gate = a.proj + (size_t)t * C_all + Cc + h * dv;
    float ss = 0.f;
    for (int j = lane; j < dv; j += 32) ss += o[j] * o[j];
    ss = warp_sum(ss);
    const float inv = 1.0f / sqrtf(ss / (float)dv + a.norm_eps);
    T* y = (T*)a.y + ((size_t)t * H + h) * dv;
    for (int j = lane; j < dv; j += 32) y[j] = from_f32<T>(o[j] * inv * a.norm_w[j] * silu_f(gate[j]));
  }
  // the block of a sequence's first row also keeps the convolutions' tail (every reader
  // of the old one, the prepare kernel, has finished)
  if (a.taps > 1) {
    const int seq = a.token_seq[t];
    if (t == a.cu_q[seq]) delta_keep_tail(a, seq, blockIdx.y * blockDim.x + threadIdx.x, gridDim.y * blockDim.x);
  }
  pdl_launch_dependents_if_large();
}

// ---- a decode step in one kernel ---------------------------------------------
// Every sequence brings one row: a block per head and sequence does all of the mixer for it.  Bound by latency (a
// head's state is 64 KB; three kernels of few blocks were 20 us of a step of one sequence and 16 heads of 128, each its
// own hand-over; this is 4.7), so the weights, which no kernel writes, are requested before the wait, and the state and
// the kept inputs are on their way to L2 by then.  They are read behind it: the kernel in front may be another step of
// the same sequences, which writes both at its end.  A column of the state is in eight lanes' registers, four columns a
// thread.  The heads that share q and k are a cluster: all of them read the kept inputs of q and k, and the first
// replaces them when all have.
// From some ten sequences on it is bound by the states' way through memory, and two blocks an SM (128 registers a thread)
// keep it busy while one of them waits.  Projection, rule and output product of a layer of 16 heads on 8 at 1, 4, 8, 16,
// 32 and 64 sequences, us: 20.7, 23.2, 23.2, 25.3, 39.5 and 67.4; with one block an SM 21.1, 22.9, 23.0, 29.8, 47.0 and
// 80.5; prepare, scan and finish 28.6, 31.0, 30.8, 35.3, 48.5 and 74.9.
#define DS_COLS 128       // columns of a head: 4 passes of 32
#define DS_TAPS 8
template <typename T>
__global__ void __launch_bounds__(256, 2) delta_step_kernel(const DeltaArgs a) {
  __shared__ float q_s[128], k_s[128], v_s[DS_COLS], o_s[DS_COLS], sums[2][8];
  pdl_launch_dependents_if_small();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.x, seq = blockIdx.y, H = a.H, G = a.G, dk = a.dk, dv = a.dv, taps = a.taps;
  const int kvh = h / (H / G), Cc = 2 * G * dk + H * dv, C_all = Cc + H * dv + 2 * H;
  const int slot = a.slots[seq], t = a.cu_q[seq];
  if (a.cu_q[seq + 1] <= t) return;              // (the same for the whole cluster)
  float* st = slot >= 0 ? a.state + (size_t)slot * a.state_stride : nullptr;
  float* sp = st ? st + (size_t)(taps - 1) * Cc + (size_t)h * dv * dk : nullptr;
  const int l = tid & 7, c0 = tid >> 3;
  // this thread's channel of q or k, and of v
  const bool is_q = tid < dk, is_qk = tid < 2 * dk, is_v = tid < dv;
  const int cq = is_q ? kvh * dk + tid : (G + kvh) * dk + (tid - dk), cv = 2 * G * dk + h * dv + tid;
  if (st) {                                      // (32 bytes a request of the kept inputs, whose rows start anywhere)
    for (int i = tid * 32; i < dk * dv; i += 256 * 32) prefetch_l2(sp + i);
    if (lane % 8 == 0)
      for (int j = 1; j < taps; ++j) {
        if (is_qk) prefetch_l2(st + (size_t)(taps - 1 - j) * Cc + cq);
        if (is_v) prefetch_l2(st + (size_t)(taps - 1 - j) * Cc + cv);
      }
  }
  // (the weights as well: a kernel in front may have made them)
  if (is_qk) prefetch_l2(a.conv_w + (size_t)cq * taps);
  if (is_v) prefetch_l2(a.conv_w + (size_t)cv * taps);
  if (is_v && lane == 0) prefetch_l2(a.norm_w + tid);
  if (tid == 0) prefetch_l2(a.a_log + h), prefetch_l2(a.dt_bias + h);
  pdl_wait();
  float w_q[DS_TAPS], w_v[DS_TAPS];              // [j]: of the input j rows back
#pragma unroll
  for (int j = 0; j < DS_TAPS; ++j) {
    w_q[j] = j < taps && is_qk ? a.conv_w[(size_t)cq * taps + taps - 1 - j] : 0.f;
    w_v[j] = j < taps && is_v ? a.conv_w[(size_t)cv * taps + taps - 1 - j] : 0.f;
  }
  const float rate = expf(a.a_log[h]), dt = a.dt_bias[h], nw = is_v ? a.norm_w[tid] : 0.f;
  float kept_q[DS_TAPS], kept_v[DS_TAPS];
#pragma unroll
  for (int j = 1; j < DS_TAPS; ++j) {
    kept_q[j] = st && j < taps && is_qk ? st[(size_t)(taps - 1 - j) * Cc + cq] : 0.f;
    kept_v[j] = st && j < taps && is_v ? st[(size_t)(taps - 1 - j) * Cc + cv] : 0.f;
  }
  kept_q[0] = kept_v[0] = 0.f;
  float4 S[4][4];
#pragma unroll
  for (int p = 0; p < 4; ++p)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int c = p * 32 + c0, e = (i * 8 + l) * 4;
      S[p][i] = sp && c < dv && e < dk ? *reinterpret_cast<const float4*>(sp + (size_t)c * dk + e)
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  const float* row = a.proj + (size_t)t * C_all;
  if (is_qk) kept_q[0] = row[cq];
  float gate = 0.f;
  if (is_v) kept_v[0] = row[cv], gate = row[Cc + h * dv + tid];
  const float b = row[Cc + H * dv + h], al = row[Cc + H * dv + H + h];
  float x = 0.f, v = 0.f;
#pragma unroll
  for (int j = 0; j < DS_TAPS; ++j) x = fmaf(w_q[j], kept_q[j], x), v = fmaf(w_v[j], kept_v[j], v);
  // (the kept inputs have been used, so they have been read)
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  x = silu_f(x);
  if (is_v) v_s[tid] = silu_f(v);
  const float sq = warp_sum(is_q ? x * x : 0.f), sk = warp_sum(is_qk && !is_q ? x * x : 0.f);
  if (lane == 0) sums[0][warp] = sq, sums[1][warp] = sk;
  __syncthreads();
  if (is_qk) {
    float ss = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) ss += sums[is_q ? 0 : 1][i];
    const float inv = 1.0f / sqrtf(ss + a.unit_eps);
    if (is_q) q_s[tid] = x * inv * (1.0f / sqrtf((float)dk));
    else k_s[tid - dk] = x * inv;
  }
  __syncthreads();
  const float beta = 1.0f / (1.0f + expf(-b)), g = expf(-rate * softplus_f(al + dt));
  float4 q[4], k[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = (i * 8 + l) * 4;
    q[i] = e < dk ? *reinterpret_cast<const float4*>(q_s + e) : make_float4(0.f, 0.f, 0.f, 0.f);
    k[i] = e < dk ? *reinterpret_cast<const float4*>(k_s + e) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  float kq = 0.f, dq[4], dks[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    kq = fmaf(k[i].x, q[i].x, kq), kq = fmaf(k[i].y, q[i].y, kq);
    kq = fmaf(k[i].z, q[i].z, kq), kq = fmaf(k[i].w, q[i].w, kq);
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float d1 = 0.f, d2 = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 s = S[p][i];
      d1 = fmaf(s.x, k[i].x, d1), d1 = fmaf(s.y, k[i].y, d1), d1 = fmaf(s.z, k[i].z, d1), d1 = fmaf(s.w, k[i].w, d1);
      d2 = fmaf(s.x, q[i].x, d2), d2 = fmaf(s.y, q[i].y, d2), d2 = fmaf(s.z, q[i].z, d2), d2 = fmaf(s.w, q[i].w, d2);
    }
    dks[p] = d1, dq[p] = d2;
  }
#pragma unroll
  for (int m = 1; m < 8; m <<= 1) {
    kq += __shfl_xor_sync(0xffffffffu, kq, m);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      dks[p] += __shfl_xor_sync(0xffffffffu, dks[p], m);
      dq[p] += __shfl_xor_sync(0xffffffffu, dq[p], m);
    }
  }
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    const int c = p * 32 + c0;
    const float u = c < dv ? beta * (v_s[c] - g * dks[p]) : 0.f;
    if (l == 0 && c < dv) o_s[c] = fmaf(u, kq, g * dq[p]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float4 s = S[p][i];
      s.x = fmaf(k[i].x, u, g * s.x), s.y = fmaf(k[i].y, u, g * s.y);
      s.z = fmaf(k[i].z, u, g * s.z), s.w = fmaf(k[i].w, u, g * s.w);
      const int e = (i * 8 + l) * 4;
      if (sp && c < dv && e < dk) *reinterpret_cast<float4*>(sp + (size_t)c * dk + e) = s;
    }
  }
  __syncthreads();
  float ss = 0.f;
  for (int j = lane; j < dv; j += 32) ss += o_s[j] * o_s[j];
  const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)dv + a.norm_eps);
  if (is_v) ((T*)a.y)[((size_t)t * H + h) * dv + tid] = from_f32<T>(o_s[tid] * inv * nw * silu_f(gate));
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (st) {
#pragma unroll
    for (int j = 0; j < DS_TAPS; ++j)
      if (j < taps - 1) {
        if (is_v) st[(size_t)(taps - 2 - j) * Cc + cv] = kept_v[j];
        if (is_qk && h % (H / G) == 0) st[(size_t)(taps - 2 - j) * Cc + cq] = kept_q[j];
      }
  }
  pdl_launch_dependents_if_large();
}

// Heads of up to 128 by 128 in whole pieces of four on 16-byte boundaries, up to eight taps and clusters of eight.
static bool delta_step_takes(const DeltaArgs& a) {
  const int Cc = 2 * a.G * a.dk + a.H * a.dv;
  return a.few_rows == 2 && a.dk <= 128 && a.dk % 4 == 0 && a.dv <= DS_COLS && a.taps <= DS_TAPS && a.H / a.G <= 8 &&
         a.n_seqs <= 65535 && a.state_stride % 4 == 0 && ((long long)(a.taps - 1) * Cc) % 4 == 0 &&
         (((uintptr_t)a.state) & 15) == 0;
}

// ---- many rows: chunk by chunk (delta_chunk.cuh) -------------------------------
// With c_t = g_1 .. g_t inside a chunk, what that file calls e^L is one number a row:
//   A_ti = (c_t / c_i) (k_t . k_i),  B_ti = (c_t / c_i) (q_t . k_i),  u_t = beta_t (v_t - S_0^T c_t k_t - sum_{i<t} A_ti u_i)
// (quotients are products of the g between).  This kernel takes every chunk of every head at the same time, solves
// the triangular system for the right-hand sides beta v and beta c k, and leaves the record.  The scan below
// walks 2,048 rows (16 heads of 128) in 512 turns of a microsecond, 502 us and 36 for their products; this kernel takes
// 58 us, the two behind it 149 and 67 (with the norm and the gate, which took 40 more behind the scan).  Decays are
// multiplied up with the rounding of each product carried along, and the products of two rows are sums of chains of eight.
__global__ void __launch_bounds__(256, 2) delta_local_kernel(const DeltaArgs a) {
  constexpr int LD = CC_MAX_DK + 4;
  extern __shared__ __align__(16) float sm[];
  float *Ks = sm, *Qs = Ks + CC_ROWS * LD, *As = Qs + CC_ROWS * LD, *Bs = As + CC_ROWS * CC_ROWS;
  float *quot = Bs + CC_ROWS * CC_ROWS, *beta = quot + CC_ROWS * (CC_ROWS + 1), *cum = beta + CC_ROWS;
  pdl_launch_dependents_if_small();
  const int tid = threadIdx.x, lane = tid & 31;
  const int h = blockIdx.y, seq = blockIdx.z, z = cc_from(a) + blockIdx.x;
  const int H = a.H, G = a.G, dk = a.dk, dv = a.dv, kvh = h / (H / G), Cc = cc_channels(a), P = a.prep_stride;
  pdl_wait();
  const int first = a.cu_q[seq], n_seq = a.cu_q[seq + 1] - first;
  const int n = min(CC_ROWS, n_seq - z * CC_ROWS), row0 = first + z * CC_ROWS;
  if (n <= 0) return;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
  for (int i = 0; i < CC_ROWS * (CC_MAX_DK / 4) / 256; ++i) {
    const int at = i * 256 + tid, t = at / (CC_MAX_DK / 4), d = at % (CC_MAX_DK / 4) * 4;
    const float* p = a.prep + (size_t)(row0 + t) * P;
    const bool in = t < n && d < dk;
    *reinterpret_cast<float4*>(Qs + t * LD + d) = in ? *reinterpret_cast<const float4*>(p + kvh * dk + d) : zero;
    *reinterpret_cast<float4*>(Ks + t * LD + d) = in ? *reinterpret_cast<const float4*>(p + (G + kvh) * dk + d) : zero;
  }
  if (tid < 32) {          // a warp: lane i has the quotients c_t / c_i of row i, and c_t in front of all of them
    const float* p = a.prep + (size_t)(row0 + lane) * P + Cc + h;
    beta[lane] = lane < n ? p[0] : 0.f;
    const float g = lane < n ? p[H] : 1.f;
    float run = 0.f, run_lost = 0.f, all = 1.f, all_lost = 0.f;      // (lost: what the products' roundings left out)
#pragma unroll
    for (int t = 0; t < CC_ROWS; ++t) {
      const float gt = __shfl_sync(0xffffffffu, g, t);
      const float r = __fmul_rn(run, gt), p = __fmul_rn(all, gt);
      run_lost = t == lane ? 0.f : fmaf(run_lost, gt, fmaf(run, gt, -r));
      run = t == lane ? 1.f : r;
      all_lost = fmaf(all_lost, gt, fmaf(all, gt, -p));
      all = p;
      quot[t * (CC_ROWS + 1) + lane] = run + run_lost;               // (zero for t < i)
      if (lane == 0) cum[t] = all + all_lost;
    }
  }
  __syncthreads();
  const size_t entry = (cc_place(a, first, z, seq) * H + h) * cc_record(dk, dv);
  float* wq = a.chunks + entry;
  float* kd = wq + (size_t)dk * CC_ROWS;
  float* gc = kd + (size_t)CC_ROWS * dk;
  float* qb = wq + cc_at_qb(dk);
  float* u0 = wq + cc_at_su(dk) + (size_t)dk * dv;
  {                        // two rows by two of both products a thread
    const int t0 = tid / 16, i0 = tid % 16;
    float kk[2][2][4], qk[2][2][4];              // a sum for every fourth channel, of chains of eight
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y)
#pragma unroll
        for (int j = 0; j < 4; ++j) kk[x][y][j] = qk[x][y][j] = 0.f;
#pragma unroll 1
    for (int d0 = 0; d0 < dk; d0 += 32) {        // (channels beyond dk are zero)
      float ck[2][2][4], cq[2][2][4];
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
          for (int j = 0; j < 4; ++j) ck[x][y][j] = cq[x][y][j] = 0.f;
#pragma unroll 2
      for (int d = d0; d < d0 + 32; d += 4) {
        float4 ki[2], kt[2], qt[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          ki[x] = *reinterpret_cast<const float4*>(Ks + (i0 + 16 * x) * LD + d);
          kt[x] = *reinterpret_cast<const float4*>(Ks + (t0 + 16 * x) * LD + d);
          qt[x] = *reinterpret_cast<const float4*>(Qs + (t0 + 16 * x) * LD + d);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            ck[x][y][0] = fmaf(kt[x].x, ki[y].x, ck[x][y][0]), cq[x][y][0] = fmaf(qt[x].x, ki[y].x, cq[x][y][0]);
            ck[x][y][1] = fmaf(kt[x].y, ki[y].y, ck[x][y][1]), cq[x][y][1] = fmaf(qt[x].y, ki[y].y, cq[x][y][1]);
            ck[x][y][2] = fmaf(kt[x].z, ki[y].z, ck[x][y][2]), cq[x][y][2] = fmaf(qt[x].z, ki[y].z, cq[x][y][2]);
            ck[x][y][3] = fmaf(kt[x].w, ki[y].w, ck[x][y][3]), cq[x][y][3] = fmaf(qt[x].w, ki[y].w, cq[x][y][3]);
          }
      }
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y)
#pragma unroll
          for (int j = 0; j < 4; ++j) kk[x][y][j] += ck[x][y][j], qk[x][y][j] += cq[x][y][j];
    }
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 2; ++y) {
        const int t = t0 + 16 * x, i = i0 + 16 * y;
        const float w = quot[t * (CC_ROWS + 1) + i];
        const float *u = kk[x][y], *v = qk[x][y];
        As[t * CC_ROWS + i] = i < t ? w * ((u[0] + u[1]) + (u[2] + u[3])) : 0.f;
        Bs[t * CC_ROWS + i] = i <= t ? w * ((v[0] + v[1]) + (v[2] + v[3])) : 0.f;
      }
  }
  __syncthreads();
  // the substitution: a thread takes one right-hand side (dv of values, then dk of c k)
  for (int c = tid; c < dv + dk; c += 256) {
    float x[CC_ROWS];
    const int d = c - dv;
#pragma unroll
    for (int t = 0; t < CC_ROWS; ++t) {
      if (d < 0) x[t] = t < n ? a.prep[(size_t)(row0 + t) * P + 2 * G * dk + h * dv + c] : 0.f;
      else x[t] = Ks[t * LD + d] * cum[t];
    }
#pragma unroll
    for (int t = 0; t < CC_ROWS; ++t) {
      float s = 0.f;
#pragma unroll
      for (int i0 = 0; i0 < t; i0 += 4) {        // (entries of A from the diagonal on are zero, x there still finite)
        const float4 w = *reinterpret_cast<const float4*>(As + t * CC_ROWS + i0);
        s = fmaf(w.x, x[i0], s);
        if (i0 + 1 < t) s = fmaf(w.y, x[i0 + 1], s);
        if (i0 + 2 < t) s = fmaf(w.z, x[i0 + 2], s);
        if (i0 + 3 < t) s = fmaf(w.w, x[i0 + 3], s);
      }
      x[t] = beta[t] * (x[t] - s);
    }
    if (d < 0) {
#pragma unroll
      for (int t = 0; t < CC_ROWS; ++t) u0[(size_t)t * dv + c] = x[t];
    } else {
      float4* out = reinterpret_cast<float4*>(wq + (size_t)d * CC_ROWS);
#pragma unroll
      for (int t = 0; t < CC_ROWS; t += 4) out[t / 4] = make_float4(x[t], x[t + 1], x[t + 2], x[t + 3]);
    }
  }
  pdl_launch_dependents_if_large();
  for (int i = tid; i < 8 * dk; i += 256) {      // c q, four rows of a channel a thread
    const int d = i / 8, t = (i % 8) * 4;
    *reinterpret_cast<float4*>(qb + (size_t)d * CC_ROWS + t) =
        make_float4(Qs[t * LD + d] * cum[t], Qs[(t + 1) * LD + d] * cum[t + 1], Qs[(t + 2) * LD + d] * cum[t + 2],
                    Qs[(t + 3) * LD + d] * cum[t + 3]);
  }
  for (int i = tid; i < CC_ROWS * CC_ROWS; i += 256)     // B by columns
    qb[(size_t)dk * CC_ROWS + i] = Bs[(i % CC_ROWS) * CC_ROWS + i / CC_ROWS];
  for (int i = tid; i < CC_ROWS * dk; i += 256) {        // what is left of a row's key at the chunk's end
    const int t = i / dk, d = i % dk;
    kd[i] = Ks[t * LD + d] * quot[(CC_ROWS - 1) * (CC_ROWS + 1) + t];
  }
  for (int d = tid; d < dk; d += 256) gc[d] = cum[CC_ROWS - 1];
}

static bool delta_chunks_take(const DeltaArgs& a) {
  return a.chunks && !a.few_rows && a.max_rows > 0 && a.dk <= CC_MAX_DK && a.dk % 4 == 0 && a.dv % 4 == 0 &&
         a.dv <= CC_MAX_DV && a.H <= 65535 && (a.window ? a.group : a.n_seqs) <= 65535 &&
         (((uintptr_t)a.chunks) & 15) == 0;
}

// All at once, or, where the scratch would be too large, by groups of sequences and windows of their chunks: the state
// goes from one window to the next through its place in the cache, in the same 32 bits.  (A padding sequence has no
// place: its read-outs, which nobody reads, start anew with every window.)
template <typename T>
static int delta_by_chunks(DeltaArgs a, cudaStream_t s) {
  const size_t smem = (2 * CC_ROWS * (CC_MAX_DK + 4) + 2 * CC_ROWS * CC_ROWS + CC_ROWS * (CC_ROWS + 1) + 2 * CC_ROWS) *
                      sizeof(float);
  cudaError_t ce = cudaFuncSetAttribute(delta_local_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (ce != cudaSuccess) return (int)ce;
  const int all = (a.max_rows + CC_ROWS - 1) / CC_ROWS, n_seqs = a.n_seqs, *cu_q = a.cu_q, *slots = a.slots;
  const int window = a.window ? a.window : all, group = a.window ? a.group : n_seqs;
  for (int q = 0; q < n_seqs; q += group) {
    a.cu_q = cu_q + q, a.slots = slots + q, a.n_seqs = n_seqs - q < group ? n_seqs - q : group;
    for (a.z0 = 0; a.z0 < all; a.z0 += window) {
      const int chunks = all - a.z0 < window ? all - a.z0 : window;
      int e = gb_launch(delta_local_kernel, dim3(chunks, a.H, a.n_seqs), dim3(256), smem, s, a);
      if (!e) e = delta_chain_and_out<T>(a, chunks, s);
      if (e) return e;
    }
  }
  return 0;
}

template <int R, int B>
static int scan_launch_b(const DeltaArgs& a, cudaStream_t s) {
  const dim3 grid((a.dv + DELTA_COLS - 1) / DELTA_COLS, a.H, a.n_seqs), block(DELTA_LANES * DELTA_COLS);
  constexpr int TT = B == 1 ? 1 : DELTA_TT;
  const size_t smem = (size_t)(a.few_rows ? 1 : 2) * (TT * (2 * DELTA_LANES * R + DELTA_COLS) +
                                                      (TT / B) * DeltaCoef<B>::SIZE) * sizeof(float);
  if (smem > 48 * 1024) {
    cudaError_t ce = cudaFuncSetAttribute(delta_scan_kernel<R, B>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (ce != cudaSuccess) return (int)ce;
  }
  return gb_launch(delta_scan_kernel<R, B>, grid, block, smem, s, a);
}

template <int R>
static int scan_launch(const DeltaArgs& a, cudaStream_t s) {
  return a.few_rows == 2 ? scan_launch_b<R, 1>(a, s) : scan_launch_b<R, DELTA_B>(a, s);
}

static int delta_check(const DeltaArgs& a) {
  if (a.n_tokens < 0 || a.n_seqs <= 0 || a.H <= 0 || a.G <= 0 || a.H % a.G || a.dk <= 0 ||
      a.dv <= 0 || a.taps <= 0 || !a.proj || !a.state || !a.prep || (!a.o && !a.chunks) || !a.y)
    return GB_ERR_BAD_ARG;
  if (a.dk > 32 * DELTA_LANES) return GB_ERR_UNSUPPORTED;
  const int Cc = 2 * a.G * a.dk + a.H * a.dv;
  if (a.prep_stride != delta_gram_offset(Cc, a.H) + DELTA_COEF * a.H ||
      (((uintptr_t)a.prep) & 15))
    return GB_ERR_BAD_ARG;
  return 0;
}

template <typename T>
static int delta_forward(const DeltaArgs& a, cudaStream_t s) {
  int e = delta_check(a);
  if (e) return e;
  if (a.n_tokens == 0) return 0;
  if (delta_step_takes(a))
    return gb_launch_cluster(delta_step_kernel<T>, dim3(a.H, a.n_seqs), dim3(256), 0, s, a.H / a.G, a);
  const int units = a.G + (a.H * a.dv + DELTA_PREP_V - 1) / DELTA_PREP_V;
  if (!a.few_rows && a.n_tokens >= 256 && a.n_tokens / 8 >= a.n_seqs && a.dk % 32 == 0 && a.dk <= 128 && a.taps <= DP_TAPS) {
    const int runs = a.n_tokens / DP_RUN + a.n_seqs;         // (run_of_block)
    e = gb_launch(delta_prepare_rows_kernel, dim3(runs, a.G + (a.H * a.dv + 255) / 256), dim3(256), 0, s, a);
  } else {
    e = gb_launch(delta_prepare_kernel, dim3(a.n_tokens, units), dim3(256), (size_t)2 * a.dk * sizeof(float), s, a);
  }
  if (e) return e;
  if (a.window && (a.window < 0 || a.group < 1)) return GB_ERR_BAD_ARG;
  if (delta_chunks_take(a)) return delta_by_chunks<T>(a, s);
  if (!a.o) return GB_ERR_BAD_ARG;
  if (!a.few_rows) {
    e = gb_launch(delta_gram_kernel, dim3(a.n_tokens, a.H), dim3(128), 0, s, a);
    if (e) return e;
  }
  const int per_lane = (a.dk + DELTA_LANES - 1) / DELTA_LANES;
  if (per_lane <= 4) e = scan_launch<4>(a, s);
  else if (per_lane <= 8) e = scan_launch<8>(a, s);
  else if (per_lane <= 12) e = scan_launch<12>(a, s);
  else if (per_lane <= 16) e = scan_launch<16>(a, s);
  else if (per_lane <= 24) e = scan_launch<24>(a, s);
  else e = scan_launch<32>(a, s);
  if (e) return e;
  const int warps = a.H < 8 ? a.H : 8;
  int rows_y = (a.H + warps - 1) / warps;            // blocks of a row: enough for its heads, and
  const int Cc = 2 * a.G * a.dk + a.H * a.dv;        //   for the tail's channels four to a thread
  const int for_tail = a.taps > 1 ? (Cc + warps * 32 * 4 - 1) / (warps * 32 * 4) : 1;
  if (for_tail > rows_y) rows_y = for_tail < 64 ? for_tail : 64;
  return gb_launch(delta_finish_kernel<T>, dim3(a.n_tokens, rows_y), dim3(warps * 32), 0, s, a);
}

// One launch for a decode step; prepare, local, chain and out by chunks; else prepare, gram (not for a step of few rows a
// sequence), scan and finish.
GB_EXPORT int gb_delta_forward_f32(const DeltaArgs* a, cudaStream_t s) { return delta_forward<float>(*a, s); }
GB_EXPORT int gb_delta_forward_bf16(const DeltaArgs* a, cudaStream_t s) { return delta_forward<bf16>(*a, s); }
