// The delta rule with a decay per channel, chunk by chunk (included by channel_delta.cu; the
// notation is that file's).  With L_t the sums of log g from a chunk's first row to row t
// (per channel) and S_0 the state in front of the chunk, the rows of a chunk obey
//
//   u_t = beta_t (v_t - S_0^T (e^{L_t} k_t) - sum_{i<t} A_ti u_i),   A_ti = sum_d k_td k_id e^{L_td - L_id}
//   o_t = S_0^T (e^{L_t} q_t) + sum_{i<=t} B_ti u_i,                 B_ti = sum_d q_td k_id e^{L_td - L_id}
//   S_n = diag(e^{L_n}) S_0 + sum_i (e^{L_n - L_i} k_i) u_i^T
//
// The first line is a triangular system: u = X v - (W) S_0 with both X v and W from one forward
// substitution that knows nothing of S_0.  So
//
//   local   takes every chunk of every head at the same time: A, B, the substitution for the dv + dk
//           right-hand sides beta v and beta e^{L} k, and leaves the chunk's record
//   chain, out   (delta_chunk.cuh) walk a sequence's chunks in order, and take every chunk again
//
// Every exponent that is taken is not positive and is summed up from logarithms of one sign, never a
// difference of two running sums (rows of the same half chunk directly, others by way of the end of
// the first half): no quotient of decays overflows, and none loses its digits behind a strong one.
#pragma once

__device__ __forceinline__ int cc_channels(const ChannelDeltaArgs& a) { return cd_channels(a); }
__device__ __forceinline__ const float* cc_gate(const ChannelDeltaArgs& a, size_t t, int h) {
  return a.wide + t * a.H * (a.dk + a.dv) + (size_t)a.H * a.dk + (size_t)h * a.dv;
}
__device__ __forceinline__ float cc_gate_of(const ChannelDeltaArgs&, float x) { return cd_sigmoid(x); }
__device__ __forceinline__ void cc_out_done(const ChannelDeltaArgs&, int, int) {}
#include "delta_chunk.cuh"
__device__ __forceinline__ int cc_from(const ChannelDeltaArgs&) { return 0; }
__device__ __forceinline__ int cc_to(const ChannelDeltaArgs&, int chunks) { return chunks; }
__device__ __forceinline__ size_t cc_place(const ChannelDeltaArgs&, int first, int z, int seq) { return cc_entry(first, z, seq); }

#define CC_HALF 16
#define CC_MIN 64        // a step goes chunk by chunk when a sequence brings this many rows
#define CC_LOG2E 1.4426950408889634f   // the kernels keep logarithms to base 2: one operation less per power

// Sums over the warp's lanes of 32 values a lane holds: lane i gets the sum of value i.
__device__ __forceinline__ float cc_transpose_sum(float (&v)[32], int lane) {
#pragma unroll
  for (int m = 16; m > 0; m >>= 1) {
    const bool up = lane & m;
#pragma unroll
    for (int i = 0; i < m; ++i) {
      const float give = up ? v[i] : v[i + m], keep = up ? v[i + m] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, m);
    }
  }
  return v[0];
}

template <int E>
__device__ __forceinline__ void cc_read(const float* p, float (&o)[E]) {
  if constexpr (E == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    o[0] = x.x, o[1] = x.y, o[2] = x.z, o[3] = x.w;
  } else if constexpr (E == 2) {
    const float2 x = *reinterpret_cast<const float2*>(p);
    o[0] = x.x, o[1] = x.y;
  } else {
    o[0] = p[0];
  }
}

// E channels a lane: heads of up to 32 E.  The block's rows, zero beyond dk and beyond the chunk's end.
template <int E>
__global__ void __launch_bounds__(256, 2) channel_delta_local_kernel(const ChannelDeltaArgs a) {
  constexpr int DKP = 32 * E, LD = DKP + 4;      // (16-byte rows; a column's rows on different banks)
  extern __shared__ __align__(16) float sm[];
  float *Ks = sm, *Qs = Ks + CC_ROWS * LD, *Ls = Qs + CC_ROWS * LD, *Fs = Ls + CC_ROWS * LD;
  float *Kr = Fs + CC_ROWS * LD;                 // [16][LD]: the first half's keys, faded to its end
  float *As = Kr + CC_HALF * LD, *Bs = As + CC_ROWS * CC_ROWS, *beta = Bs + CC_ROWS * CC_ROWS;
  pdl_launch_dependents_if_small();
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int h = blockIdx.y, seq = blockIdx.z, z = blockIdx.x;
  const int H = a.H, G = a.G, dk = a.dk, dv = a.dv, kvh = h / (H / G), Cc = cd_channels(a);
  const float rate = expf(a.a_log[h]);
  pdl_wait();
  const int first = a.cu_q[seq], n_seq = a.cu_q[seq + 1] - first;
  const int n = min(CC_ROWS, n_seq - z * CC_ROWS), row0 = first + z * CC_ROWS;
  if (n <= 0) return;
#pragma unroll 4
  for (int i = tid; i < CC_ROWS * DKP; i += 256) {
    const int t = i / DKP, d = i % DKP;
    float q = 0.f, k = 0.f, lg = 0.f;
    if (t < n && d < dk) {
      const float* p = a.prep + (size_t)(row0 + t) * a.prep_stride;
      q = p[kvh * dk + d], k = p[(G + kvh) * dk + d];
      lg = CC_LOG2E * cd_log_decay(a.wide[(size_t)(row0 + t) * H * (dk + dv) + h * dk + d], a.dt_bias[h * dk + d], rate);
    }
    Qs[t * LD + d] = q, Ks[t * LD + d] = k, Ls[t * LD + d] = lg;
  }
  if (tid < CC_ROWS) beta[tid] = tid < n ? a.prep[(size_t)(row0 + tid) * a.prep_stride + Cc + h] : 0.f;
  __syncthreads();
  const size_t entry = (cc_entry(first, z, seq) * H + h) * cc_record(dk, dv);
  float* wq = a.chunks + entry;
  float* kd = wq + (size_t)dk * CC_ROWS;
  float* gc = kd + (size_t)CC_ROWS * dk;
  float* qb = wq + cc_at_qb(dk);
  float* u0 = wq + cc_at_su(dk) + (size_t)dk * dv;
  // per channel: Fs, the logarithms summed up from the start of a row's half chunk on; and, from the
  // chunk's end back, what is left of a row's key at the end of its half and of the chunk (rows
  // beyond the chunk's end have no decay)
  if (tid < DKP) {
    float s = 0.f;
#pragma unroll 8
    for (int t = 0; t < CC_ROWS; ++t) {
      if (t == CC_HALF) s = 0.f;
      s += Ls[t * LD + tid];
      Fs[t * LD + tid] = s;
    }
  } else if (tid >= 128 && tid - 128 < DKP) {
    const int d = tid - 128;
    float s = 0.f, in_half = 0.f;
#pragma unroll 4
    for (int t = CC_ROWS - 1; t >= 0; --t) {
      const float k = Ks[t * LD + d], lg = Ls[t * LD + d];
      if (d < dk) kd[t * dk + d] = k * exp2f(s);
      if (t < CC_HALF) {
        Kr[t * LD + d] = k * exp2f(in_half);
        in_half += lg;
      }
      s += lg;
    }
    if (d < dk) gc[d] = exp2f(s);
  }
  __syncthreads();
  // A and B: a warp takes rows warp, warp + 8, ...; its lanes share the channels
  for (int t = warp; t < CC_ROWS; t += 8) {
    float kt[E], qt[E], ki[E], li[E], since[E], part[32];
    cc_read<E>(Ks + t * LD + lane * E, kt);
    cc_read<E>(Qs + t * LD + lane * E, qt);
    const int base = t & CC_HALF;                // the first row of t's half chunk
#pragma unroll
    for (int x = 0; x < E; ++x) since[x] = 0.f;  // the logarithms behind row base + j, up to t's
#pragma unroll
    for (int j = CC_HALF - 1; j >= 0; --j) {
      part[j] = part[CC_HALF + j] = 0.f;
      if (base + j <= t) {
        cc_read<E>(Ks + (base + j) * LD + lane * E, ki);
        cc_read<E>(Ls + (base + j) * LD + lane * E, li);
#pragma unroll
        for (int x = 0; x < E; ++x) {
          const float w = ki[x] * exp2f(since[x]);
          since[x] += li[x];
          part[j] = fmaf(kt[x], w, part[j]);
          part[CC_HALF + j] = fmaf(qt[x], w, part[CC_HALF + j]);
        }
      }
    }
    float sum = cc_transpose_sum(part, lane);    // lanes 0 .. 15: A, 16 .. 31: B
    const int j = lane & (CC_HALF - 1);
    if (lane < CC_HALF) As[t * CC_ROWS + base + j] = base + j < t ? sum : 0.f;
    else Bs[t * CC_ROWS + base + j] = base + j <= t ? sum : 0.f;
    if (base) {                                  // the other half, by way of its last row
      cc_read<E>(Fs + t * LD + lane * E, li);
#pragma unroll
      for (int x = 0; x < E; ++x) {
        const float w = exp2f(li[x]);
        kt[x] *= w, qt[x] *= w;
      }
#pragma unroll
      for (int i = 0; i < CC_HALF; ++i) {
        part[i] = part[CC_HALF + i] = 0.f;
        cc_read<E>(Kr + i * LD + lane * E, ki);
#pragma unroll
        for (int x = 0; x < E; ++x) {
          part[i] = fmaf(kt[x], ki[x], part[i]);
          part[CC_HALF + i] = fmaf(qt[x], ki[x], part[CC_HALF + i]);
        }
      }
      sum = cc_transpose_sum(part, lane);
      (lane < CC_HALF ? As : Bs)[t * CC_ROWS + j] = sum;
    } else {
      (lane < CC_HALF ? As : Bs)[t * CC_ROWS + CC_HALF + j] = 0.f;
    }
  }
  __syncthreads();
  // the substitution: a thread takes one right-hand side (dv of values, then dk of e^{L} k)
  for (int c = tid; c < dv + dk; c += 256) {
    float x[CC_ROWS];
    const int d = c - dv;
#pragma unroll
    for (int t = 0; t < CC_ROWS; ++t) {
      if (d < 0) x[t] = t < n ? a.prep[(size_t)(row0 + t) * a.prep_stride + 2 * G * dk + h * dv + c] : 0.f;
      else x[t] = Ks[t * LD + d] * exp2f(Fs[t * LD + d] + (t < CC_HALF ? 0.f : Fs[(CC_HALF - 1) * LD + d]));
    }
#pragma unroll
    for (int t = 0; t < CC_ROWS; ++t) {
      float s = x[t];
#pragma unroll
      for (int i0 = 0; i0 < t; i0 += 4) {        // (entries of A from the diagonal on are zero, x there still finite)
        const float4 w = *reinterpret_cast<const float4*>(As + t * CC_ROWS + i0);
        s = fmaf(-w.x, x[i0], s);
        if (i0 + 1 < t) s = fmaf(-w.y, x[i0 + 1], s);
        if (i0 + 2 < t) s = fmaf(-w.z, x[i0 + 2], s);
        if (i0 + 3 < t) s = fmaf(-w.w, x[i0 + 3], s);
      }
      x[t] = beta[t] * s;
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
  for (int i = tid; i < 8 * dk; i += 256) {      // e^{L} q, four rows of a channel a thread
    const int d = i / 8, t = (i % 8) * 4;
    const float before = t < CC_HALF ? 0.f : Fs[(CC_HALF - 1) * LD + d];
    float v[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) v[x] = Qs[(t + x) * LD + d] * exp2f(Fs[(t + x) * LD + d] + before);
    *reinterpret_cast<float4*>(qb + (size_t)d * CC_ROWS + t) = make_float4(v[0], v[1], v[2], v[3]);
  }
  for (int i = tid; i < CC_ROWS * CC_ROWS; i += 256)     // B by columns
    qb[(size_t)dk * CC_ROWS + i] = Bs[(i % CC_ROWS) * CC_ROWS + i / CC_ROWS];
}

static bool cc_takes(const ChannelDeltaArgs& a) {
  return a.chunks && a.max_rows >= CC_MIN && a.dk <= CC_MAX_DK && a.dk % 4 == 0 && a.dv % 4 == 0 &&
         a.dv <= CC_MAX_DV && (((uintptr_t)a.chunks) & 15) == 0;
}

template <int E>
static int cc_local(const ChannelDeltaArgs& a, int chunks, cudaStream_t s) {
  constexpr int LD = 32 * E + 4;
  const size_t smem = ((4 * CC_ROWS + CC_HALF) * LD + 2 * CC_ROWS * CC_ROWS + CC_ROWS) * sizeof(float);
  static bool configured = false;
  if (smem > 48 * 1024 && !configured) {
    cudaError_t e = cudaFuncSetAttribute(channel_delta_local_kernel<E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)smem);
    if (e != cudaSuccess) return (int)e;
    configured = true;
  }
  return gb_launch(channel_delta_local_kernel<E>, dim3(chunks, a.H, a.n_seqs), dim3(256), smem, s, a);
}

template <typename T>
static int cc_run(const ChannelDeltaArgs& a, cudaStream_t s) {
  const int chunks = (a.max_rows + CC_ROWS - 1) / CC_ROWS;
  int e = a.dk <= 32 ? cc_local<1>(a, chunks, s) : a.dk <= 64 ? cc_local<2>(a, chunks, s) : cc_local<4>(a, chunks, s);
  if (e) return e;
  return delta_chain_and_out<T>(a, chunks, s);
}
