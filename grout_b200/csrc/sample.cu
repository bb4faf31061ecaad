// Next-token choice on the device from rows of 32-bit logits.
//
// gb_argmax_f32: first maximum (ties go to the lowest index, as the reference's
// argmax kernels do, src/kernels.rs:379-385, 502-508).
//
// gb_sample_f32: the reference's sample_next (src/model.rs:2212-2270) without a
// sort of the vocabulary.  s_i = logit_i / temperature; the top_k largest are
// kept (0 < top_k < V; equal scores keep index order); p_i = exp(s_i - max);
// with top_p < 1 the shortest prefix, in descending order, whose normalised
// mass reaches top_p is kept; then u * sum(p) is walked over the kept set.
// "The k-th largest" and "the prefix that reaches top_p" are both thresholds on
// the score (by counts for top_k, by probability mass for top_p), with ties at the
// threshold resolved by index.  The walk is in index order (the reference walks in
// descending order of probability; the distribution is the same).
// Two kernels: a cluster of blocks that holds a row's scores in shared memory, and
// one block per row that reads them again in every pass, for rows too long for that.
// temperature <= 1e-5 falls back to argmax (src/model.rs:2216-2218).
#include "common.cuh"
#include <cooperative_groups.h>
#include <limits.h>

namespace cg = cooperative_groups;

#define ST 1024

__device__ __forceinline__ uint32_t okey(float s) {
  if (s != s) return 0u;  // NaN sorts below everything
  const uint32_t b = __float_as_uint(s);
  return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_to_float(uint32_t k) {
  const uint32_t b = (k & 0x80000000u) ? (k & 0x7fffffffu) : ~k;
  return __uint_as_float(b);
}

struct ArgBest {
  float v;
  int i;
};
__device__ __forceinline__ ArgBest better(ArgBest a, ArgBest b) {
  if (b.v > a.v || (b.v == a.v && b.i < a.i)) return b;
  return a;
}

// every thread returns the block's first maximum
__device__ ArgBest block_argmax(const float* row, int V, float mul, ArgBest* sh) {
  ArgBest best{-INFINITY, INT_MAX};
  for (int i = threadIdx.x; i < V; i += ST) {
    float v = row[i] * mul;
    if (v != v) v = -INFINITY;
    if (v > best.v || (v == best.v && i < best.i)) best = ArgBest{v, i};
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgBest other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = best;
  __syncthreads();
  ArgBest r = sh[0];
  for (int w = 1; w < ST / 32; ++w) r = better(r, sh[w]);
  if (r.i == INT_MAX) r.i = 0;  // a row of NaN or -inf
  return r;
}

// Stage 1: block (chunk, row) finds the first maximum of its slice of the row.
// Stage 2: one warp per row picks the first maximum among the chunks.  Two short
// launches instead of one block per row, which left most of the GPU idle.
#define ARGMAX_CHUNKS 32

__global__ void __launch_bounds__(256) argmax_partial_kernel(const float* logits, int V,
                                                             float* part_v, int* part_i) {
  __shared__ ArgBest sh[8];
  pdl_launch_dependents_if_small();
  pdl_wait();
  const int row = blockIdx.y, chunk = blockIdx.x;
  const int per = (V + ARGMAX_CHUNKS - 1) / ARGMAX_CHUNKS;
  const int lo = chunk * per, hi = min(V, lo + per);
  const float* r = logits + (size_t)row * V;
  ArgBest best{-INFINITY, INT_MAX};
  for (int i = lo + threadIdx.x; i < hi; i += 256) {
    float v = r[i];
    if (v != v) v = -INFINITY;
    if (v > best.v || (v == best.v && i < best.i)) best = ArgBest{v, i};
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgBest other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = best;
  __syncthreads();
  if (threadIdx.x == 0) {
    ArgBest b = sh[0];
    for (int w = 1; w < 8; ++w) b = better(b, sh[w]);
    part_v[row * ARGMAX_CHUNKS + chunk] = b.v;
    part_i[row * ARGMAX_CHUNKS + chunk] = b.i;
  }
}

__global__ void __launch_bounds__(32) argmax_final_kernel(const float* part_v, const int* part_i,
                                                          int* out) {
  pdl_launch_dependents_if_small();
  pdl_wait();
  const int row = blockIdx.x;
  ArgBest best{part_v[row * ARGMAX_CHUNKS + threadIdx.x], part_i[row * ARGMAX_CHUNKS + threadIdx.x]};
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ArgBest other{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)};
    best = better(best, other);
  }
  if (threadIdx.x == 0) out[row] = best.i == INT_MAX ? 0 : best.i;
}

// scratch: n_rows * 32 floats followed by n_rows * 32 ints (the caller's).
GB_EXPORT int gb_argmax_f32(const float* logits, int n_rows, int V, int* out, void* scratch,
                            cudaStream_t s) {
  if (n_rows < 0 || V <= 0 || !scratch) return GB_ERR_BAD_ARG;
  if (n_rows == 0) return 0;
  if (n_rows > 65535) return GB_ERR_UNSUPPORTED;
  float* pv = (float*)scratch;
  int* pi = (int*)(pv + (size_t)n_rows * ARGMAX_CHUNKS);
  int e = gb_launch(argmax_partial_kernel, dim3(ARGMAX_CHUNKS, n_rows), dim3(256), 0, s, logits, V,
                    pv, pi);
  if (e) return e;
  return gb_launch(argmax_final_kernel, dim3(n_rows), dim3(32), 0, s, (const float*)pv,
                   (const int*)pi, out);
}

// ---------------------------------------------------------------------------
struct Members {       // i is kept when key > thr, or key == thr and i <= cut
  uint32_t thr;
  int cut;
};
__device__ __forceinline__ bool member(const Members& m, uint32_t key, int i) {
  return key > m.thr || (key == m.thr && i <= m.cut);
}

__device__ double block_sum_f64(double v, double* sh) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0.0;
  for (int w = 0; w < ST / 32; ++w) r += sh[w];
  return r;
}

// Inclusive scan of one value per thread over the block; returns the thread's
// inclusive prefix and the block total.
template <typename T>
__device__ T block_scan(T v, T* sh, T* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T n = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += n;
  }
  __syncthreads();
  if (lane == 31) sh[warp] = v;
  __syncthreads();
  T before = 0, all = 0;
  for (int w = 0; w < ST / 32; ++w) {
    if (w < warp) before += sh[w];
    all += sh[w];
  }
  *total = all;
  return v + before;
}

struct Shared {
  unsigned int cnt[256];
  double mass[256];
  ArgBest best[ST / 32];
  double red[ST / 32];
  int ired[ST / 32];
  uint32_t sel_prefix;
  unsigned int sel_count;   // elements in the chosen bin
  double rest_mass;         // mass still wanted inside the chosen bin
  unsigned int rest_count;  // rank still wanted inside the chosen bin
  int found;
};

// The index of the r-th element (1-based, index order) whose key equals `key`
// among the members of `base`.
__device__ int find_tie_cut(const float* row, int V, float inv_t, const Members& base, uint32_t key,
                            unsigned int r, Shared& sh) {
  unsigned int seen = 0;
  if (threadIdx.x == 0) sh.found = INT_MAX;
  __syncthreads();
  for (int c = 0; c < V; c += ST) {
    const int i = c + threadIdx.x;
    int flag = 0;
    if (i < V) {
      const uint32_t k = okey(row[i] * inv_t);
      flag = (k == key && member(base, k, i)) ? 1 : 0;
    }
    int total;
    const int incl = block_scan<int>(flag, sh.ired, &total);
    if (flag && seen + incl == r) sh.found = i;
    seen += total;
    __syncthreads();
    if (seen >= r) break;
  }
  __syncthreads();
  return sh.found;
}

// What the rows of a launch ask for: arrays on the device, or, without them, the
// values themselves, which then travel with the launch and need no copy.
#define SAMPLE_ROWS 64
struct SampleAsk {
  const float* temperature_dev;
  const int* top_k_dev;
  const float* top_p_dev;
  const float* u_dev;
  float temperature[SAMPLE_ROWS];
  int top_k[SAMPLE_ROWS];
  float top_p[SAMPLE_ROWS];
  float u[SAMPLE_ROWS];
};
__device__ __forceinline__ void asked_of(const SampleAsk& a, int b, float& temp, int& K, float& P, float& u) {
  temp = a.temperature_dev ? a.temperature_dev[b] : a.temperature[b];
  K = a.top_k_dev ? a.top_k_dev[b] : a.top_k[b];
  P = a.top_p_dev ? a.top_p_dev[b] : a.top_p[b];
  u = a.u_dev ? a.u_dev[b] : a.u[b];
}

// One block per row, every pass over the row from memory (L2): 2,537 us for 64 rows of
// 151,936, so it is kept for rows that the cluster kernel's shared memory cannot hold.
__global__ void __launch_bounds__(ST)
sample_kernel(const float* __restrict__ logits, int V, const __grid_constant__ SampleAsk asked,
              int* __restrict__ out) {
  __shared__ Shared sh;
  const int b = blockIdx.x, tid = threadIdx.x;
  const float* row = logits + (size_t)b * V;
  float temp, P, u;
  int K;
  asked_of(asked, b, temp, K, P, u);
  if (!(temp > 1.0e-5f)) {
    const ArgBest r = block_argmax(row, V, 1.0f, sh.best);
    if (tid == 0) out[b] = r.i;
    return;
  }
  const float inv_t = 1.0f / temp;
  const ArgBest top = block_argmax(row, V, inv_t, sh.best);
  const float smax = top.v;
  P = fminf(fmaxf(P, 0.f), 1.f);

  Members mem{0u, INT_MAX};

  // ---- top-k: the k-th largest key, by counts --------------------------------
  if (K > 0 && K < V) {
    uint32_t prefix = 0;
    unsigned int want = (unsigned int)K;
    unsigned int eq = 0;
    for (int d = 3; d >= 0; --d) {
      for (int j = tid; j < 256; j += ST) sh.cnt[j] = 0;
      __syncthreads();
      const int shift = 8 * d;
      for (int i = tid; i < V; i += ST) {
        const uint32_t k = okey(row[i] * inv_t);
        if (d == 3 || (k >> (shift + 8)) == (prefix >> (shift + 8)))
          atomicAdd(&sh.cnt[(k >> shift) & 255u], 1u);
      }
      __syncthreads();
      if (tid == 0) {
        unsigned int w = want;
        int bin = 0;
        for (int j = 255; j >= 0; --j) {
          if (w <= sh.cnt[j]) { bin = j; break; }
          w -= sh.cnt[j];
        }
        sh.sel_prefix = prefix | ((uint32_t)bin << shift);
        sh.rest_count = w;
        sh.sel_count = sh.cnt[bin];
      }
      __syncthreads();
      prefix = sh.sel_prefix;
      want = sh.rest_count;
      eq = sh.sel_count;
      __syncthreads();
    }
    mem.thr = prefix;
    if (want < eq) mem.cut = find_tie_cut(row, V, inv_t, Members{0u, INT_MAX}, prefix, want, sh);
  }

  // ---- mass of the kept set ---------------------------------------------------
  double local = 0.0;
  for (int i = tid; i < V; i += ST) {
    const float s = row[i] * inv_t;
    const uint32_t k = okey(s);
    if (member(mem, k, i)) local += (double)expf(s - smax);
  }
  double total = block_sum_f64(local, sh.red);

  // ---- top-p: the key at which the descending cumulative mass reaches P * total
  if (P < 1.0f) {
    uint32_t prefix = 0;
    double want = (double)P * total;
    unsigned int eq = 0;
    for (int d = 3; d >= 0; --d) {
      for (int j = tid; j < 256; j += ST) { sh.cnt[j] = 0; sh.mass[j] = 0.0; }
      __syncthreads();
      const int shift = 8 * d;
      for (int i = tid; i < V; i += ST) {
        const float s = row[i] * inv_t;
        const uint32_t k = okey(s);
        if (member(mem, k, i) && (d == 3 || (k >> (shift + 8)) == (prefix >> (shift + 8)))) {
          atomicAdd(&sh.cnt[(k >> shift) & 255u], 1u);
          atomicAdd(&sh.mass[(k >> shift) & 255u], (double)expf(s - smax));
        }
      }
      __syncthreads();
      if (tid == 0) {
        double w = want;
        int bin = -1, lowest = 0;
        for (int j = 255; j >= 0; --j) {
          if (!sh.cnt[j]) continue;
          lowest = j;
          if (sh.mass[j] >= w) { bin = j; break; }
          w -= sh.mass[j];
        }
        if (bin < 0) { bin = lowest; w = sh.mass[lowest]; }  // rounding left a crumb: keep all
        sh.sel_prefix = prefix | ((uint32_t)bin << shift);
        sh.rest_mass = w;
        sh.sel_count = sh.cnt[bin];
      }
      __syncthreads();
      prefix = sh.sel_prefix;
      want = sh.rest_mass;
      eq = sh.sel_count;
      __syncthreads();
    }
    // `want` is the mass still needed from the eq elements equal to the threshold
    const double pv = (double)expf(key_to_float(prefix) - smax);
    unsigned int r = eq;
    if (pv > 0.0) {
      const double need = ceil(want / pv);
      r = need < 1.0 ? 1u : (need > (double)eq ? eq : (unsigned int)need);
    }
    Members narrowed{prefix, INT_MAX};
    // ties at a shared threshold obey the tighter of the two limits
    if (prefix == mem.thr && mem.cut != INT_MAX) {
      narrowed.cut = mem.cut;
      // r counts members only; find_tie_cut below counts members of `mem` too
    }
    if (r < eq) {
      const int cut = find_tie_cut(row, V, inv_t, mem, prefix, r, sh);
      narrowed.cut = cut < narrowed.cut ? cut : narrowed.cut;
    }
    mem = narrowed;
    local = 0.0;
    for (int i = tid; i < V; i += ST) {
      const float s = row[i] * inv_t;
      const uint32_t k = okey(s);
      if (member(mem, k, i)) local += (double)expf(s - smax);
    }
    total = block_sum_f64(local, sh.red);
  }

  if (!(total > 0.0) || total != total || isinf(total)) {  // src/model.rs:2260-2263
    if (tid == 0) out[b] = top.i;
    return;
  }

  // ---- the draw: first index whose running mass reaches u * total --------------
  const double threshold = (double)u * total;
  double seen = 0.0;
  if (tid == 0) sh.found = INT_MAX;
  __syncthreads();
  int last_member = -1;
  for (int c = 0; c < V; c += ST) {
    const int i = c + tid;
    double p = 0.0;
    bool in = false;
    if (i < V) {
      const float s = row[i] * inv_t;
      const uint32_t k = okey(s);
      in = member(mem, k, i);
      if (in) p = (double)expf(s - smax);
    }
    if (in) last_member = i;
    double ctotal;
    const double incl = block_scan<double>(p, sh.red, &ctotal);
    if (in && seen + incl >= threshold) atomicMin(&sh.found, i);
    seen += ctotal;
    __syncthreads();
    if (sh.found != INT_MAX) break;
  }
  __syncthreads();
  int token = sh.found;
  if (token == INT_MAX) {  // rounding left the threshold above the last sum
    int lm = last_member;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) lm = max(lm, __shfl_xor_sync(0xffffffffu, lm, o));
    __syncthreads();
    if ((tid & 31) == 0) sh.ired[tid >> 5] = lm;
    __syncthreads();
    if (tid == 0) {
      int best = -1;
      for (int w = 0; w < ST / 32; ++w) best = max(best, sh.ired[w]);
      sh.found = best < 0 ? top.i : best;
    }
    __syncthreads();
    token = sh.found;
  }
  if (tid == 0) out[b] = token;
}

// ---------------------------------------------------------------------------
// A row per cluster of eight blocks.  What bounds it: the passes over a row are short
// (152,000 scores are 19,000 a block) and depend on one another, so the time of a single
// row is the number of dependent steps; of a full batch, the instructions of the passes.
// The scores are read from memory once and kept in shared memory; a threshold costs one
// histogram pass over 2,048 bins that divide the row's own range of scores evenly (the
// bits of the float key put most of a row into a dozen bins, whose atomics then queue),
// combined over the blocks through distributed shared memory, and one pass that gathers
// the few scores of the bin on which the threshold falls, which are ranked directly.
// A bin with more than SC_GATHER of them (equal scores, far outliers that stretch the
// range) is divided again by the key's bits, 11 at a time.
// Measured at 151,936 scores against the one-block kernel above, us: one row with
// temperature, top-k and top-p 415 -> 31, 64 rows of four kinds of limits 2,537 -> 90
// (temperature alone 43, with top-k 63, with top-k and top-p 80, with top-p alone 116: the
// 64-bit masses of a whole row's histogram are what that costs).
#define SC_BLOCKS 8
#define SC_THREADS 512
#define SC_WARPS (SC_THREADS / 32)
#define SC_BINS 2048
#define SC_SLICE (SC_BINS / SC_BLOCKS)   // bins that a block adds up for its cluster
#define SC_GATHER 1024                   // scores that are ranked directly
#define SC_STRIDE 8                      // groups of 32 scores that the draw passes at once
#define SC_SCORES 50000                  // scores a block's shared memory holds

struct __align__(16) ClusterShared {
  unsigned int cnt[SC_BINS];       // later: all the gathered elements, 64 bits each
  double mass[SC_BINS];            // later: this block's gathered elements, then their masses
  unsigned int slice_cnt[SC_SLICE];
  double slice_mass[SC_SLICE];
  double slice_mass_sum;
  unsigned int slice_cnt_sum;
  unsigned int n_mine;
  ArgBest best;
  float lowest;
  ArgBest warp_best[SC_WARPS];
  float warp_low[SC_WARPS];
  double warp_mass[SC_WARPS];      // mass and number of the members in every warp's run of scores
  unsigned int warp_cnt[SC_WARPS];
  double block_mass;
  unsigned int block_cnt;
  int pick_bin;                    // what a histogram pass found
  unsigned int pick_n, pick_rest;
  double pick_mass_rest;
  uint32_t thr;                    // what a ranking found
  int cut, rank;
};
static_assert(SC_GATHER * 8 <= SC_BINS * 4 && 2 * SC_GATHER * 8 <= SC_BINS * 8, "gathered elements fit the bins");

// A block's share of the row and where it lies in it.
struct RowPart {
  const float* s;      // scores, in shared memory
  int first, n;        // s[0] is the row's element `first`
  int lo, hi;          // this warp's run of them, in index order over the warps
};

// The bin, in descending order of the scores, on which a threshold falls: the `want`-th
// element (by counts) or the element at which the mass reaches `frac` of the whole (first
// pass) or `want_mass` (a pass inside a bin).  bin_of(i, score) is the element's bin or -1;
// it must not grow with the score.  All blocks of the cluster return the same.
struct Pick {
  int bin;
  unsigned int n, rest;    // elements in the bin; rank still wanted inside it
  double rest_mass;        // mass still wanted inside it
  double total;            // mass of all elements (by mass only)
};
template <bool MASS, typename BinOf>
__device__ Pick pick_bin(cg::cluster_group& cl, ClusterShared& sh, const RowPart& part, float smax, BinOf bin_of,
                         unsigned int want, double want_mass, double frac) {
  const int tid = threadIdx.x, lane = tid & 31, rank = (int)cl.block_rank();
  cl.sync();               // the others are done with what the last pass left here
  for (int j = tid; j < SC_BINS; j += SC_THREADS) {
    sh.cnt[j] = 0;
    if (MASS) sh.mass[j] = 0.0;
  }
  __syncthreads();
  for (int i = tid; i < part.n; i += SC_THREADS) {
    const float s = part.s[i];
    const int b = bin_of(i, s);
    if (b >= 0) {
      atomicAdd(&sh.cnt[b], 1u);
      if (MASS) {
        // adding nothing changes nothing, and far below the maximum there is little else
        const double p = (double)expf(s - smax);
        if (p != 0.0) atomicAdd(&sh.mass[b], p);
      }
    }
  }
  cl.sync();
  if (tid < SC_SLICE) {
    unsigned int c = 0;
    double m = 0.0;
#pragma unroll
    for (int r = 0; r < SC_BLOCKS; ++r) {
      const ClusterShared* peer = cl.map_shared_rank(&sh, r);
      c += peer->cnt[rank * SC_SLICE + tid];
      if (MASS) m += peer->mass[rank * SC_SLICE + tid];
    }
    sh.slice_cnt[tid] = c;
    if (MASS) sh.slice_mass[tid] = m;
  }
  __syncthreads();
  if (tid < 32) {
    unsigned int c = 0;
    double m = 0.0;
    for (int j = lane; j < SC_SLICE; j += 32) {
      c += sh.slice_cnt[j];
      if (MASS) m += sh.slice_mass[j];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      c += __shfl_xor_sync(0xffffffffu, c, o);
      if (MASS) m += __shfl_xor_sync(0xffffffffu, m, o);
    }
    if (lane == 0) {
      sh.slice_cnt_sum = c;
      sh.slice_mass_sum = m;
    }
  }
  cl.sync();
  Pick got{-1, 0u, 0u, 0.0, 0.0};
  unsigned int slice_n[SC_BLOCKS];
  double slice_m[SC_BLOCKS];
#pragma unroll
  for (int r = 0; r < SC_BLOCKS; ++r) {
    const ClusterShared* peer = cl.map_shared_rank(&sh, r);
    slice_n[r] = peer->slice_cnt_sum;
    slice_m[r] = MASS ? peer->slice_mass_sum : 0.0;
    got.total += slice_m[r];
  }
  if (MASS && frac >= 0.0) want_mass = frac * got.total;
  // the slice, then the bin in it; where rounding leaves the wanted mass a crumb above all
  // that there is, the lowest element that there is
  int slice = -1, last = 0;
  unsigned int n_before = 0, n_last = 0;
  double m_before = 0.0, m_last = 0.0;
  {
    unsigned int n = 0;
    double m = 0.0;
#pragma unroll
    for (int r = 0; r < SC_BLOCKS; ++r) {
      if (slice < 0 && slice_n[r]) {
        if (MASS ? m + slice_m[r] >= want_mass : n + slice_n[r] >= want) {
          slice = r, n_before = n, m_before = m;
        }
        last = r, n_last = n, m_last = m;
      }
      n += slice_n[r];
      m += slice_m[r];
    }
    if (slice < 0) slice = last, n_before = n_last, m_before = m_last;
  }
  if (tid < 32) {
    const ClusterShared* peer = cl.map_shared_rank(&sh, slice);
    constexpr int PER = SC_SLICE / 32;
    unsigned int c[PER], c_all = 0;
    double m[PER], m_all = 0.0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      c[j] = peer->slice_cnt[lane * PER + j];
      m[j] = MASS ? peer->slice_mass[lane * PER + j] : 0.0;
      c_all += c[j];
      m_all += m[j];
    }
    unsigned int c_in = c_all;
    double m_in = m_all;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned int cn = __shfl_up_sync(0xffffffffu, c_in, o);
      const double mn = __shfl_up_sync(0xffffffffu, m_in, o);
      if (lane >= o) c_in += cn, m_in += mn;
    }
    unsigned int n = n_before + c_in - c_all;
    double mm = __shfl_up_sync(0xffffffffu, m_in, 1);
    mm = m_before + (lane ? mm : 0.0);
    int hit = -1, low = -1;
    unsigned int n_hit = 0, n_low = 0, rest_hit = 0, rest_low = 0;
    double mass_hit = 0.0, mass_low = 0.0;
#pragma unroll
    for (int j = 0; j < PER; ++j) {
      if (hit < 0 && c[j]) {
        if (MASS ? mm + m[j] >= want_mass : n + c[j] >= want) {
          hit = lane * PER + j, n_hit = c[j], rest_hit = want - n, mass_hit = want_mass - mm;
        }
        low = lane * PER + j, n_low = c[j], rest_low = c[j], mass_low = m[j];
      }
      n += c[j];
      mm += m[j];
    }
    const unsigned int hits = __ballot_sync(0xffffffffu, hit >= 0), lows = __ballot_sync(0xffffffffu, low >= 0);
    const int from = hits ? __ffs(hits) - 1 : 31 - __clz(lows | 1u);
    if (lane == from) {
      sh.pick_bin = slice * SC_SLICE + (hits ? hit : low);
      sh.pick_n = hits ? n_hit : n_low;
      sh.pick_rest = hits ? rest_hit : rest_low;
      sh.pick_mass_rest = hits ? mass_hit : mass_low;
    }
  }
  __syncthreads();
  got.bin = sh.pick_bin;
  got.n = sh.pick_n;
  got.rest = sh.pick_rest;
  got.rest_mass = sh.pick_mass_rest;
  return got;
}

// The threshold among at most SC_GATHER elements in_bin(i, score): the `rest`-th in
// descending order (equal scores in index order), or the one at which their mass in that
// order reaches `rest_mass`, or, with frac >= 0, frac * (the mass of all of them), which is
// then left in *total.  Every block gathers all of them and finds the same.
template <bool MASS, typename InBin>
__device__ Members rank_gathered(cg::cluster_group& cl, ClusterShared& sh, const RowPart& part, float smax, InBin in_bin,
                                 unsigned int rest, double rest_mass, double frac = -1.0, double* total = nullptr) {
  const int tid = threadIdx.x;
  unsigned long long* mine = (unsigned long long*)sh.mass;
  unsigned long long* all = (unsigned long long*)sh.cnt;
  double* p = sh.mass + SC_GATHER;
  // (the others read this block's bins for the last time before pick_bin's last cl.sync)
  if (tid == 0) sh.n_mine = 0;
  __syncthreads();
  for (int i = tid; i < part.n; i += SC_THREADS) {
    const float s = part.s[i];
    if (in_bin(i, s)) {
      const unsigned int at = atomicAdd(&sh.n_mine, 1u);
      if (at < SC_GATHER) mine[at] = ((unsigned long long)okey(s) << 32) | (0xffffffffu - (uint32_t)(part.first + i));
    }
  }
  cl.sync();
  unsigned int n = 0;
  for (int r = 0; r < SC_BLOCKS; ++r) {
    const ClusterShared* peer = cl.map_shared_rank(&sh, r);
    const unsigned int n_r = min(peer->n_mine, (unsigned int)SC_GATHER - n);
    const unsigned long long* theirs = (const unsigned long long*)peer->mass;
    for (unsigned int t = tid; t < n_r; t += SC_THREADS) {
      const unsigned long long e = theirs[t];
      all[n + t] = e;
      if (MASS) p[n + t] = (double)expf(key_to_float((uint32_t)(e >> 32)) - smax);
    }
    n += n_r;
  }
  if (tid == 0) sh.rank = (int)n - 1;          // by mass: the lowest, unless one above it reaches
  __syncthreads();
  if (MASS && frac >= 0.0) {
    double all_mass = 0.0;
    for (unsigned int j = 0; j < n; ++j) all_mass += p[j];
    *total = all_mass;
    rest_mass = frac * all_mass;
  }
  int rank[SC_GATHER / SC_THREADS];
#pragma unroll
  for (int k = 0; k < SC_GATHER / SC_THREADS; ++k) {
    const unsigned int t = tid + k * SC_THREADS;
    rank[k] = -1;
    if (t < n) {
      const unsigned long long e = all[t];
      int above = 0;
      double m = MASS ? p[t] : 0.0;
      for (unsigned int j = 0; j < n; ++j) {
        const bool up = all[j] > e;
        above += up;
        if (MASS && up) m += p[j];
      }
      rank[k] = above;
      if (MASS && m >= rest_mass) atomicMin(&sh.rank, above);
    }
  }
  __syncthreads();
  const int pick = MASS ? sh.rank : (int)rest - 1;
#pragma unroll
  for (int k = 0; k < SC_GATHER / SC_THREADS; ++k)
    if (rank[k] == pick && rank[k] >= 0) {
      const unsigned long long e = all[tid + k * SC_THREADS];
      sh.thr = (uint32_t)(e >> 32);
      sh.cut = (int)(0xffffffffu - (uint32_t)e);
    }
  __syncthreads();
  return Members{sh.thr, sh.cut};
}

// The index of the r-th element (1-based, index order) for which is_tie(i, score) holds.
template <typename IsTie>
__device__ int cluster_tie_cut(cg::cluster_group& cl, ClusterShared& sh, const RowPart& part, IsTie is_tie,
                               unsigned int r) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, rank = (int)cl.block_rank();
  cl.sync();
  unsigned int n = 0;
  for (int c = part.lo; c < part.hi; c += 32) {
    const int i = c + lane;
    n += __popc(__ballot_sync(0xffffffffu, i < part.hi && is_tie(i, part.s[min(i, part.hi - 1)])));
  }
  if (lane == 0) sh.warp_cnt[warp] = n;
  if (threadIdx.x == 0) sh.cut = INT_MAX;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned int all = 0;
    for (int w = 0; w < SC_WARPS; ++w) all += sh.warp_cnt[w];
    sh.block_cnt = all;
  }
  cl.sync();
  unsigned int before = 0;
  for (int q = 0; q < rank; ++q) before += cl.map_shared_rank(&sh, q)->block_cnt;
  for (int w = 0; w < warp; ++w) before += sh.warp_cnt[w];
  if (before < r && before + n >= r) {          // the element is in this warp's run
    for (int c = part.lo; c < part.hi; c += 32) {
      const int i = c + lane;
      const unsigned int hits = __ballot_sync(0xffffffffu, i < part.hi && is_tie(i, part.s[min(i, part.hi - 1)]));
      if (before + __popc(hits) >= r) {
        const int skip = (int)(r - before) - 1;   // the hit with `skip` hits below it
        if ((hits >> lane) & 1u && __popc(hits & ((1u << lane) - 1u)) == skip)
          for (int q = 0; q < SC_BLOCKS; ++q) cl.map_shared_rank(&sh, q)->cut = part.first + i;
        break;
      }
      before += __popc(hits);
    }
  }
  cl.sync();
  return sh.cut;
}

// The members of `base` above a threshold: rank `want` by counts, or the mass frac * (their
// whole mass).  *total is that mass (by mass only).
template <bool MASS>
__device__ Members narrow(cg::cluster_group& cl, ClusterShared& sh, const RowPart& part, float smax, float scale,
                          const Members base, unsigned int want, double frac, double* total) {
  const auto linear = [=](float s) { return (int)fminf((smax - s) * scale, (float)(SC_BINS - 1)); };   // NaN: the last
  const auto inside = [=](int i, float s) { return member(base, okey(s), part.first + i); };
  Pick got = pick_bin<MASS>(cl, sh, part, smax, [=](int i, float s) { return inside(i, s) ? linear(s) : -1; }, want,
                            0.0, frac);
  if (MASS) {
    *total = got.total;
    if (!(got.total > 0.0) || isinf(got.total)) return base;   // the caller falls back to the maximum
  }
  const int bin = got.bin;
  if (got.n <= SC_GATHER)
    return rank_gathered<MASS>(cl, sh, part, smax, [=](int i, float s) { return inside(i, s) && linear(s) == bin; },
                               got.rest, got.rest_mass);
  // divide the bin by the key's bits
  uint32_t prefix = 0, known = 0;
  const int shifts[3] = {21, 10, 0}, widths[3] = {11, 11, 10};
#pragma unroll 1
  for (int d = 0; d < 3; ++d) {
    const int shift = shifts[d], top = (1 << widths[d]) - 1;
    got = pick_bin<MASS>(cl, sh, part, smax, [=](int i, float s) {
      const uint32_t k = okey(s);
      return inside(i, s) && linear(s) == bin && (k & known) == prefix ? top - (int)((k >> shift) & top) : -1;
    }, got.rest, got.rest_mass, -1.0);
    prefix |= (uint32_t)(top - got.bin) << shift;
    known |= (uint32_t)top << shift;
    const uint32_t pre = prefix, kn = known;
    if (got.n <= SC_GATHER)
      return rank_gathered<MASS>(cl, sh, part, smax,
                                 [=](int i, float s) { return inside(i, s) && (okey(s) & kn) == pre && linear(s) == bin; },
                                 got.rest, got.rest_mass);
  }
  unsigned int r = got.rest;                    // only equal scores are left
  if (MASS) {
    const double pv = (double)expf(key_to_float(prefix) - smax);
    r = got.n;
    if (pv > 0.0) {
      const double need = ceil(got.rest_mass / pv);
      r = need < 1.0 ? 1u : (need > (double)got.n ? got.n : (unsigned int)need);
    }
  }
  const uint32_t key = prefix;
  return Members{key, cluster_tie_cut(cl, sh, part, [=](int i, float s) { return inside(i, s) && okey(s) == key; }, r)};
}

__global__ void __launch_bounds__(SC_THREADS, 2)
sample_cluster_kernel(const float* __restrict__ logits, int V, int per_block, const __grid_constant__ SampleAsk asked,
                      int* __restrict__ out) {
  extern __shared__ __align__(16) float scores[];
  __shared__ ClusterShared sh;
  cg::cluster_group cl = cg::this_cluster();
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, rank = (int)cl.block_rank(), row_no = blockIdx.y;
  pdl_launch_dependents_if_small();
  pdl_wait();
  float temp, P, u;
  int K;
  asked_of(asked, row_no, temp, K, P, u);
  const bool greedy = !(temp > 1.0e-5f);
  const float inv_t = greedy ? 1.0f : 1.0f / temp;
  P = fminf(fmaxf(P, 0.f), 1.f);
  RowPart part;
  part.s = scores;
  part.first = min(rank * per_block, V);
  part.n = min(per_block, V - part.first);
  const int run = (per_block + SC_WARPS - 1) / SC_WARPS;
  part.lo = min(warp * run, part.n);
  part.hi = min(part.lo + run, part.n);

  // ---- the scores, their first maximum and their lowest finite value -------------
  const float* row = logits + (size_t)row_no * V + part.first;
  ArgBest best{-INFINITY, INT_MAX};
  float low = INFINITY;
  const auto take = [&](int i, float v) {
    const float s = v * inv_t, w = s != s ? -INFINITY : s;
    if (isfinite(s)) low = fminf(low, s);
    if (w > best.v || (w == best.v && part.first + i < best.i)) best = ArgBest{w, part.first + i};
    return s;
  };
  constexpr int U = 5;                          // 16-byte loads in flight a thread
  const int n4 = ((uintptr_t)row & 15) == 0 ? part.n & ~3 : 0;   // 16 bytes at a time where the row starts on them
  for (int c = 0; c < n4; c += 4 * U * SC_THREADS) {
    float4 v[U];
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int i = c + 4 * (k * SC_THREADS + tid);
      if (i < n4) v[k] = *(const float4*)(row + i);
    }
#pragma unroll
    for (int k = 0; k < U; ++k) {
      const int i = c + 4 * (k * SC_THREADS + tid);
      if (i < n4)
        *(float4*)(scores + i) = make_float4(take(i, v[k].x), take(i + 1, v[k].y), take(i + 2, v[k].z), take(i + 3, v[k].w));
    }
  }
  constexpr int U1 = 16;
  for (int c = n4; c < part.n; c += U1 * SC_THREADS) {
    float v[U1];
#pragma unroll
    for (int k = 0; k < U1; ++k) {
      const int i = c + k * SC_THREADS + tid;
      v[k] = i < part.n ? row[i] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < U1; ++k) {
      const int i = c + k * SC_THREADS + tid;
      if (i < part.n) scores[i] = take(i, v[k]);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    best = better(best, ArgBest{__shfl_xor_sync(0xffffffffu, best.v, o), __shfl_xor_sync(0xffffffffu, best.i, o)});
    low = fminf(low, __shfl_xor_sync(0xffffffffu, low, o));
  }
  if (lane == 0) sh.warp_best[warp] = best, sh.warp_low[warp] = low;
  __syncthreads();
  if (tid == 0) {
    for (int w = 1; w < SC_WARPS; ++w) {
      best = better(best, sh.warp_best[w]);
      low = fminf(low, sh.warp_low[w]);
    }
    sh.best = best;
    sh.lowest = low;
  }
  cl.sync();
  ArgBest top{-INFINITY, INT_MAX};
  low = INFINITY;
#pragma unroll
  for (int r = 0; r < SC_BLOCKS; ++r) {
    const ClusterShared* peer = cl.map_shared_rank(&sh, r);
    top = better(top, peer->best);
    low = fminf(low, peer->lowest);
  }
  if (top.i == INT_MAX) top.i = 0;
  const float smax = top.v;
  // No finite maximum: every mass would be NaN, and the choice falls to the maximum.
  if (greedy || !isfinite(smax)) {
    if (rank == 0 && tid == 0) out[row_no] = top.i;
    cl.sync();                                  // the others may still read this block's maximum
    return;
  }
  const float range = fminf(smax - low, 128.f);          // exp(-128) is nothing beside 1 in 32 bits
  const float scale = range > 0.f ? (float)(SC_BINS - 1) / range : 0.f;

  Members mem{0u, INT_MAX};
  double total = 1.0;
  if (K > 0 && K < V) mem = narrow<false>(cl, sh, part, smax, scale, mem, (unsigned int)K, -1.0, &total);
  if (P < 1.0f) {
    if (K > 0 && K < V && K <= SC_GATHER) {     // what top-k left is ranked as it is
      const Members base = mem;
      cl.sync();                                // the others are done with what top-k gathered
      mem = rank_gathered<true>(cl, sh, part, smax, [=](int i, float s) { return member(base, okey(s), part.first + i); },
                                0u, 0.0, (double)P, &total);
    } else {
      mem = narrow<true>(cl, sh, part, smax, scale, mem, 0u, (double)P, &total);
    }
  }

  // ---- mass of the kept set, by runs of scores in index order ---------------------
  double m = 0.0;
  unsigned int n = 0;
  for (int i = part.lo + lane; i < part.hi; i += 32) {
    const float s = scores[i];
    if (member(mem, okey(s), part.first + i)) {
      m += (double)expf(s - smax);
      ++n;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    m += __shfl_xor_sync(0xffffffffu, m, o);
    n += __shfl_xor_sync(0xffffffffu, n, o);
  }
  __syncthreads();
  if (lane == 0) sh.warp_mass[warp] = m, sh.warp_cnt[warp] = n;
  __syncthreads();
  if (tid == 0) {
    double bm = 0.0;
    unsigned int bn = 0;
    for (int w = 0; w < SC_WARPS; ++w) bm += sh.warp_mass[w], bn += sh.warp_cnt[w];
    sh.block_mass = bm;
    sh.block_cnt = bn;
  }
  cl.sync();
  double bm[SC_BLOCKS];
  unsigned int bn[SC_BLOCKS];
  double sum = 0.0;
#pragma unroll
  for (int r = 0; r < SC_BLOCKS; ++r) {
    const ClusterShared* peer = cl.map_shared_rank(&sh, r);
    bm[r] = peer->block_mass;
    bn[r] = peer->block_cnt;
    sum += bm[r];
  }
  cl.sync();                                    // nothing of another block is read below
  if (!(total > 0.0) || isinf(total) || !(sum > 0.0) || isinf(sum)) {  // src/model.rs:2260-2263
    if (rank == 0 && tid == 0) out[row_no] = top.i;
    return;
  }

  // ---- the draw: first member whose running mass reaches u * sum -------------------
  // block, warp and element in turn; where rounding leaves the threshold above a part's
  // own last sum, its last member
  const double threshold = (double)u * sum;
  int owner = -1, last = -1;
  double before = 0.0, owner_before = 0.0, last_before = 0.0;
#pragma unroll
  for (int r = 0; r < SC_BLOCKS; ++r) {
    if (bn[r]) {
      if (owner < 0 && before + bm[r] >= threshold) owner = r, owner_before = before;
      last = r, last_before = before;
    }
    before += bm[r];
  }
  if (owner < 0) owner = last, owner_before = last_before;
  if (rank != owner) return;
  before = owner_before;
  owner = last = -1;
  for (int w = 0; w < SC_WARPS; ++w) {
    if (sh.warp_cnt[w]) {
      if (owner < 0 && before + sh.warp_mass[w] >= threshold) owner = w, owner_before = before;
      last = w, last_before = before;
    }
    before += sh.warp_mass[w];
  }
  if (owner < 0) owner = last, owner_before = last_before;
  if (warp != owner) return;
  double seen = owner_before;
  int token = -1;
  const auto mass_at = [&](int i, bool& in) {
    const float s = i < part.hi ? scores[i] : 0.f;
    in = i < part.hi && member(mem, okey(s), part.first + i);
    return in ? (double)expf(s - smax) : 0.0;
  };
  // the stride of groups first (a scan of 32 masses is a long chain), then the group in it
  int at = part.lo;                             // the last stride with members so far
  bool reached = false;
  for (int c = part.lo; c < part.hi && !reached; c += 32 * SC_STRIDE) {
    double p = 0.0;
    bool any = false, in;
#pragma unroll
    for (int k = 0; k < SC_STRIDE; ++k) {
      p += mass_at(c + k * 32 + lane, in);
      any |= in;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) p += __shfl_xor_sync(0xffffffffu, p, o);
    any = __any_sync(0xffffffffu, any);
    if (any) at = c;
    reached = any && seen + p >= threshold;     // (a draw of zero is reached by the first member, not in front of it)
    if (!reached) seen += p;
  }
  for (int k = 0; k < SC_STRIDE; ++k) {
    const int c = at + k * 32;
    bool in;
    double p = mass_at(c + lane, in);
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double other = __shfl_up_sync(0xffffffffu, p, o);
      if (lane >= o) p += other;
    }
    const unsigned int ins = __ballot_sync(0xffffffffu, in);
    const unsigned int hits = __ballot_sync(0xffffffffu, in && reached && seen + p >= threshold);
    if (hits) {
      token = part.first + c + __ffs(hits) - 1;
      break;
    }
    if (ins) token = part.first + c + 31 - __clz(ins);
    seen += __shfl_sync(0xffffffffu, p, 31);
  }
  if (lane == 0) out[row_no] = token;
}

static int sample_launch(const float* logits, int n_rows, int V, const SampleAsk& asked, int* out, cudaStream_t s) {
  // whole groups of four, so that every block's share starts on 16 bytes when the row does
  const int per_block = ((V + SC_BLOCKS - 1) / SC_BLOCKS + 3) / 4 * 4;
  if (per_block > SC_SCORES) {
    sample_kernel<<<n_rows, ST, 0, s>>>(logits, V, asked, out);
    return gb_status();
  }
  static bool set[64] = {};                      // per device
  int dev = 0;
  cudaError_t ce = cudaGetDevice(&dev);
  if (ce == cudaSuccess && (dev >= 64 || !set[dev])) {
    ce = cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              SC_SCORES * (int)sizeof(float));
    if (ce == cudaSuccess && dev < 64) set[dev] = true;
  }
  if (ce != cudaSuccess) return (int)ce;
  for (int r = 0; r < n_rows; r += 65535) {      // rows are the grid's y
    SampleAsk a = asked;
    if (a.temperature_dev) a.temperature_dev += r, a.top_k_dev += r, a.top_p_dev += r, a.u_dev += r;
    const int n = n_rows - r < 65535 ? n_rows - r : 65535;
    const int e = gb_launch_cluster(sample_cluster_kernel, dim3(SC_BLOCKS, n), dim3(SC_THREADS),
                                    (size_t)per_block * sizeof(float), s, SC_BLOCKS, logits + (size_t)r * V, V,
                                    per_block, a, out + r);
    if (e) return e;
  }
  return 0;
}

// What the rows ask for lies on the device.
GB_EXPORT int gb_sample_f32(const float* logits, int n_rows, int V, const float* temperature,
                            const int* top_k, const float* top_p, const float* u, int* out,
                            cudaStream_t s) {
  if (n_rows < 0 || V <= 0 || !temperature || !top_k || !top_p || !u) return GB_ERR_BAD_ARG;
  if (n_rows == 0) return 0;
  SampleAsk a = {};
  a.temperature_dev = temperature, a.top_k_dev = top_k, a.top_p_dev = top_p, a.u_dev = u;
  return sample_launch(logits, n_rows, V, a, out, s);
}

// What the rows ask for lies on the host: it is read before this returns and travels with
// the launches (64 rows each), so that nothing is copied and nothing waits.
GB_EXPORT int gb_sample_host_f32(const float* logits, int n_rows, int V, const float* temperature,
                                 const int* top_k, const float* top_p, const float* u, int* out,
                                 cudaStream_t s) {
  if (n_rows < 0 || V <= 0 || !temperature || !top_k || !top_p || !u) return GB_ERR_BAD_ARG;
  for (int r = 0; r < n_rows; r += SAMPLE_ROWS) {
    SampleAsk a = {};
    const int n = n_rows - r < SAMPLE_ROWS ? n_rows - r : SAMPLE_ROWS;
    for (int k = 0; k < n; ++k) {
      a.temperature[k] = temperature[r + k];
      a.top_k[k] = top_k[r + k];
      a.top_p[k] = top_p[r + k];
      a.u[k] = u[r + k];
    }
    const int e = sample_launch(logits + (size_t)r * V, n, V, a, out + r, s);
    if (e) return e;
  }
  return 0;
}
