// Attention over the paged cache with all arithmetic in 32-bit on the CUDA cores, for prompts and for decode steps: the
// attention of the 32-bit path where the head size is a multiple of 4 up to 128 and no first keys are kept (the plain
// kernel, attn_generic.cu, has the rest; the masks, the cap and the sinks mean what they mean there).
//
// Keys go in tiles of 64 at fixed places.  A tile gives each row a maximum, a sum of exponentials and a sum of values by
// itself, and the tiles of a row are merged in turn.  A prompt's block (the rows of a few tokens and of query heads that
// share a kv head; sixteen neighbouring threads a row) walks its tiles and merges as it goes, keys and values by
// cp.async, the keys of the next tile while the values of this one are worked on and the other way round.  A decode step
// has a block for each tile, a thread for each score and then for each column, and merges in a second kernel.  Every sum
// has the same order in both, so a row's result is the same bits whichever way its tokens were cut into steps, and
// depends on its own keys only.
//
// Bound by the multiply-adds of its two products for prompts and by latency for decode steps.  Measured with 16 heads of
// 128 on 8 kv heads, us (the plain kernel, one block a token and query head, a thread a key): a decode step of 57 keys
// 7.2 (17.1), 500 keys 8.0 (117), eight sequences of 3,000 keys 63 (1,184); prompts of 45 tokens 15 (25), 100 + 180 + 330
// + 600 tokens 142 (2,485), 2,048 tokens 885 (19,570).
#include "common.cuh"

#define AF_BN 64
#define AF_LANES 16          // threads of a row

struct AttnF32Args {
  const float* q;            // [n_tokens, nq, D]
  const float* k_pages;      // [n_pages, nkv, page, D]
  const float* v_pages;
  const int* block_table;    // [slots, max_pages]
  const int* cu_q;           // [n_seqs + 1]
  const int* slots;          // [n_seqs]
  const int* kv_len;         // [n_seqs]
  float* out;                // [n_tokens, nq, D]
  float* parts;              // [n_seqs of a launch, nq, n_parts, D + 2], decode steps
  const float* sinks;        // [nq] or null
  int n_seqs, nq, nkv, D, page, max_pages, window, chunk, heads, n_qblocks, n_parts, page_shift;   // page_shift: log2(page), or -1
  float scale, softcap;
};

__device__ __forceinline__ void af_copy16(void* dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
               "r"(in ? 16 : 0));
}
__device__ __forceinline__ void af_commit() { asm volatile("cp.async.commit_group;"); }
template <int N> __device__ __forceinline__ void af_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N)); }

// exp of a maximum (or score) against a maximum that is not below it; nothing seen: 0
__device__ __forceinline__ float af_scale(float m, float m_new) { return m == -INFINITY ? 0.f : expf(m - m_new); }

// o += p v over a tile's keys in turn
template <int RT, int TY, bool SOME>
__device__ __forceinline__ void add_values(float (&o)[RT][8], const float* p_s, const float* v_s, int D, int tx, int ty) {
  const int D4 = D / 4;
#pragma unroll 2
  for (int j = 0; j < AF_BN; j += 4) {
    float4 p[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) p[r] = *(const float4*)(p_s + (ty + TY * r) * (AF_BN + 4) + j);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int c = tx + 16 * h;
        if (c >= D4) continue;
        const float4 v = *(const float4*)(v_s + (j + u) * D + c * 4);
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          const float x = u == 0 ? p[r].x : u == 1 ? p[r].y : u == 2 ? p[r].z : p[r].w;
          float* to = o[r] + 4 * h;
          if (!SOME || x != 0.f) {
            to[0] = fmaf(x, v.x, to[0]);
            to[1] = fmaf(x, v.y, to[1]);
            to[2] = fmaf(x, v.z, to[2]);
            to[3] = fmaf(x, v.w, to[3]);
          }
        }
      }
  }
}

// RT rows a thread, TY groups of sixteen threads
template <int RT, int TY>
__global__ void __launch_bounds__(TY * AF_LANES)
attn_f32_prompt_kernel(AttnF32Args a) {
  constexpr int ROWS = RT * TY, THREADS = TY * AF_LANES;
  extern __shared__ float4 af_sm[];
  const int D = a.D, LD = D + 4, D4 = D / 4;
  float* q_s = (float*)af_sm;                    // [ROWS][LD]
  float* k_s = q_s + ROWS * LD;                  // [64][LD]
  float* v_s = k_s + AF_BN * LD;                 // [64][D]
  float* p_s = v_s + AF_BN * D;                  // [ROWS][68]
  constexpr int LP = AF_BN + 4;
  const int tid = threadIdx.x, tx = tid % AF_LANES, ty = tid / AF_LANES;
  const int group = a.nq / a.nkv, subs = group / a.heads;
  const int hx = blockIdx.x % (a.nkv * subs), kvh = hx / subs, head0 = kvh * group + hx % subs * a.heads;
  pdl_wait();

  // the block's sequence and its tokens
  const int per = ROWS / a.heads, b = a.n_qblocks - 1 - (int)(blockIdx.x / (a.nkv * subs));    // heavy blocks first
  int first_block;
  const int seq = find_query_block(a.cu_q, a.n_seqs, per, b, first_block);
  if (seq >= a.n_seqs) return;
  const int q0 = (b - first_block) * per;
  const int tok0 = a.cu_q[seq] + q0, q_len = a.cu_q[seq + 1] - a.cu_q[seq];
  const int tokens = min(per, q_len - q0), rows = tokens * a.heads;
  const int slot = a.slots[seq];
  auto row_at = [&](int row) { return ((size_t)(tok0 + row / a.heads) * a.nq + head0 + row % a.heads) * D; };
  if (slot < 0) {
    for (int i = tid; i < rows * D; i += THREADS) a.out[row_at(i / D) + i % D] = 0.f;
    return;
  }
  const int pos0 = a.kv_len[seq] - q_len + q0, key_hi = pos0 + tokens - 1;
  const int key_lo = first_key(pos0, a.window, a.chunk);
  int tile = key_lo / AF_BN;
  const int tile_end = key_hi / AF_BN + 1;
  const int* table = a.block_table + (size_t)slot * a.max_pages;
  auto load = [&](float* dst, const float* pages, int t, int ld) {
#pragma unroll 4
    for (int r = ty; r < AF_BN; r += TY) {
      const int key = t * AF_BN + r;
      const bool in = key >= key_lo && key <= key_hi;   // others may have no page
      const float* src = pages;
      if (in) {
        // (a division a row would be most of a tile's instructions)
        const int at = a.page_shift >= 0 ? key >> a.page_shift : key / a.page;
        src += (((size_t)table[at] * a.nkv + kvh) * a.page + (key - at * a.page)) * D;
      }
      if (tx < D4) af_copy16(dst + r * ld + tx * 4, in ? src + tx * 4 : src, in);
      if (tx + 16 < D4) af_copy16(dst + r * ld + (tx + 16) * 4, in ? src + (tx + 16) * 4 : src, in);
    }
  };
#pragma unroll
  for (int k = 0; k < RT; ++k) {
    const int r = ty + TY * k;
    const float* src = r < rows ? a.q + row_at(r) : a.q;
    if (tx < D4) af_copy16(q_s + r * LD + tx * 4, r < rows ? src + tx * 4 : src, r < rows);
    if (tx + 16 < D4) af_copy16(q_s + r * LD + (tx + 16) * 4, r < rows ? src + (tx + 16) * 4 : src, r < rows);
  }
  load(k_s, a.k_pages, tile, LD);
  af_commit();
  load(v_s, a.v_pages, tile, D);
  af_commit();

  float m[RT], l[RT], o[RT][8], was[RT], now[RT];
  int lo[RT], hi[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    m[r] = -INFINITY, l[r] = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) o[r][c] = 0.f;
    const int row = ty + TY * r, pos = pos0 + row / a.heads;
    hi[r] = row < rows ? pos : -1;              // rows beyond the block see nothing
    lo[r] = first_key(pos, a.window, a.chunk);
  }
  for (; tile < tile_end; ++tile) {
    af_wait<1>();
    __syncthreads();                            // the keys are there
    float s[RT][4];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int i = 0; i < 4; ++i) s[r][i] = 0.f;
#pragma unroll 4
    for (int d = 0; d < D; d += 4) {
      float4 k[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) k[i] = *(const float4*)(k_s + (tx + 16 * i) * LD + d);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const float4 x = *(const float4*)(q_s + (ty + TY * r) * LD + d);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          s[r][i] = fmaf(x.x, k[i].x, s[r][i]);
          s[r][i] = fmaf(x.y, k[i].y, s[r][i]);
          s[r][i] = fmaf(x.z, k[i].z, s[r][i]);
          s[r][i] = fmaf(x.w, k[i].w, s[r][i]);
        }
      }
    }
    const int key0 = tile * AF_BN;
#pragma unroll
    for (int r = 0; r < RT; ++r) {
      float top = -INFINITY;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int key = key0 + tx + 16 * i;
        float v = s[r][i] * a.scale;
        if (a.softcap > 0.f) v = a.softcap * tanhf(v / a.softcap);
        s[r][i] = key <= hi[r] && key >= lo[r] ? v : -INFINITY;
        top = fmaxf(top, s[r][i]);
      }
#pragma unroll
      for (int x = 1; x < AF_LANES; x *= 2) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float p = af_scale(s[r][i], top);
        p_s[(ty + TY * r) * LP + tx + 16 * i] = p;
        sum += p;
      }
#pragma unroll
      for (int x = 1; x < AF_LANES; x *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, x);
      const float m_new = fmaxf(m[r], top);
      was[r] = af_scale(m[r], m_new), now[r] = af_scale(top, m_new);
      l[r] = fmaf(l[r], was[r], sum * now[r]);
      m[r] = m_new;
    }
    __syncthreads();                            // the keys are read; the probabilities are there
    if (tile + 1 < tile_end) load(k_s, a.k_pages, tile + 1, LD);
    af_commit();
    af_wait<1>();
    __syncthreads();                            // the values are there
    float t[RT][8];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int c = 0; c < 8; ++c) t[r][c] = 0.f;
    // Where a row does not see all of the tile's keys, their values are not multiplied: they may be infinite.
    if (key0 + AF_BN - 1 > pos0 || key0 < first_key(key_hi, a.window, a.chunk)) add_values<RT, TY, true>(t, p_s, v_s, D, tx, ty);
    else add_values<RT, TY, false>(t, p_s, v_s, D, tx, ty);
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
      for (int c = 0; c < 8; ++c) o[r][c] = fmaf(o[r][c], was[r], t[r][c] * now[r]);
    __syncthreads();                            // the values and probabilities are read
    if (tile + 1 < tile_end) load(v_s, a.v_pages, tile + 1, D);
    af_commit();
  }
  pdl_launch_dependents();
  af_wait<0>();
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    const int row = ty + TY * r;
    if (row >= rows) continue;
    const int h = head0 + row % a.heads;
    float mm = m[r], ll = l[r], f = 1.f;
    if (a.sinks) {
      const float m_new = fmaxf(mm, a.sinks[h]);
      f = expf(mm - m_new);
      ll = fmaf(ll, f, expf(a.sinks[h] - m_new));
    }
    f = f * (1.0f / ll);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const int at = (tx + 16 * c) * 4;
      if (at >= D) continue;
      const float* x = o[r] + 4 * c;
      *(float4*)(a.out + row_at(row) + at) = make_float4(x[0] * f, x[1] * f, x[2] * f, x[3] * f);
    }
  }
}

// One tile of keys of a decode step's sequence for `heads` query heads; the tiles of a sequence count from the one that
// holds its first visible key.  A score is one thread's, a column's sum over the keys is one thread's; the sums of
// exponentials are added by sixteen threads a row as in the kernel above.
#define AD_THREADS 256
__global__ void __launch_bounds__(AD_THREADS)
attn_f32_decode_kernel(AttnF32Args a) {
  extern __shared__ float4 af_sm[];
  const int D = a.D, LD = D + 4, D4 = D / 4;
  float* k_s = (float*)af_sm;                    // [64][LD]
  float* v_s = k_s + AF_BN * LD;                 // [64][D]
  float* q_s = v_s + AF_BN * D;                  // [heads][D]
  float* p_s = q_s + a.heads * D;                // [heads][64]
  const int tid = threadIdx.x;
  const int group = a.nq / a.nkv, subs = group / a.heads;
  const int hx = blockIdx.x % (a.nkv * subs), kvh = hx / subs, head0 = kvh * group + hx % subs * a.heads;
  pdl_wait();
  const int at = blockIdx.x / (a.nkv * subs), seq = at / a.n_parts, part = at % a.n_parts;
  const int slot = a.slots[seq];
  const size_t row0 = (size_t)a.cu_q[seq] * a.nq + head0;
  if (slot < 0) {
    if (part == 0)
      for (int i = tid; i < a.heads * D; i += AD_THREADS) a.out[row0 * D + i] = 0.f;
    return;
  }
  const int pos = a.kv_len[seq] - 1, lo = first_key(pos, a.window, a.chunk), key0 = (lo / AF_BN + part) * AF_BN;
  if (key0 > pos) return;                        // (the merge does not look at this part either)
  const int* table = a.block_table + (size_t)slot * a.max_pages;
  auto load = [&](float* dst, const float* pages, int ld) {
#pragma unroll 4
    for (int i = tid; i < AF_BN * 32; i += AD_THREADS) {   // a warp a row, so that the row's page is found once
      const int r = i / 32, c = i % 32, key = key0 + r;
      const bool in = key >= lo && key <= pos;
      const float* src = pages;
      if (in) {
        const int at = a.page_shift >= 0 ? key >> a.page_shift : key / a.page;
        src += (((size_t)table[at] * a.nkv + kvh) * a.page + (key - at * a.page)) * D;
      }
      if (c < D4) af_copy16(dst + r * ld + c * 4, in ? src + c * 4 : src, in);
    }
  };
  load(k_s, a.k_pages, LD);
  for (int i = tid; i < a.heads * D4; i += AD_THREADS) af_copy16(q_s + i * 4, a.q + row0 * D + i * 4, true);
  af_commit();
  load(v_s, a.v_pages, D);
  af_commit();
  af_wait<1>();
  __syncthreads();
  for (int i = tid; i < a.heads * AF_BN; i += AD_THREADS) {
    const float *q = q_s + i / AF_BN * D, *k = k_s + i % AF_BN * LD;
    float s = 0.f;
#pragma unroll 8
    for (int d = 0; d < D; d += 4) {
      const float4 x = *(const float4*)(q + d), y = *(const float4*)(k + d);
      s = fmaf(x.x, y.x, s);
      s = fmaf(x.y, y.y, s);
      s = fmaf(x.z, y.z, s);
      s = fmaf(x.w, y.w, s);
    }
    float v = s * a.scale;
    if (a.softcap > 0.f) v = a.softcap * tanhf(v / a.softcap);
    const int key = key0 + i % AF_BN;
    p_s[i] = key <= pos && key >= lo ? v : -INFINITY;
  }
  __syncthreads();
  float* parts = a.parts + (((size_t)seq * a.nq + head0) * a.n_parts + part) * (D + 2);
  const size_t part_ld = (size_t)a.n_parts * (D + 2);
  if (tid < 8 * AF_LANES) {                      // whole warps, whatever the number of heads
    const int r = tid / AF_LANES, tx = tid % AF_LANES;
    float s[4], top = -INFINITY, sum = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = r < a.heads ? p_s[r * AF_BN + tx + 16 * i] : -INFINITY, top = fmaxf(top, s[i]);
#pragma unroll
    for (int x = 1; x < AF_LANES; x *= 2) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      s[i] = af_scale(s[i], top);
      if (r < a.heads) p_s[r * AF_BN + tx + 16 * i] = s[i];
      sum += s[i];
    }
#pragma unroll
    for (int x = 1; x < AF_LANES; x *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, x);
    if (tx == 0 && r < a.heads) parts[r * part_ld + D] = top, parts[r * part_ld + D + 1] = sum;
  }
  af_wait<0>();
  __syncthreads();
  pdl_launch_dependents();
  const bool some = key0 + AF_BN - 1 > pos || key0 < lo;   // (unseen keys' values may be infinite)
  for (int i = tid; i < a.heads * D; i += AD_THREADS) {
    const int r = i / D, d = i % D;
    const float *p = p_s + r * AF_BN, *v = v_s + d;
    float o = 0.f;
    if (some) {
      for (int j = 0; j < AF_BN; ++j)
        if (p[j] != 0.f) o = fmaf(p[j], v[j * D], o);
    } else {
#pragma unroll 16
      for (int j = 0; j < AF_BN; ++j) o = fmaf(p[j], v[j * D], o);
    }
    parts[r * part_ld + d] = o;
  }
}

// The tiles of a decode step's rows in turn: one block a sequence and query head, a thread a column.
__global__ void attn_f32_merge_kernel(AttnF32Args a) {
  pdl_wait();
  pdl_launch_dependents_if_small();
  const int seq = blockIdx.x, h = blockIdx.y, D = a.D;
  if (a.slots[seq] < 0) return;
  const int pos = a.kv_len[seq] - 1;
  const int parts = pos / AF_BN - first_key(pos, a.window, a.chunk) / AF_BN + 1;
  const float* p = a.parts + ((size_t)seq * a.nq + h) * a.n_parts * (D + 2);
  const int d = threadIdx.x;
  float m = -INFINITY, l = 0.f, o = 0.f;
#pragma unroll 8
  for (int i = 0; i < parts; ++i) {
    const float pm = p[(size_t)i * (D + 2) + D], pl = p[(size_t)i * (D + 2) + D + 1], po = p[(size_t)i * (D + 2) + d];
    const float m_new = fmaxf(m, pm), was = af_scale(m, m_new), now = af_scale(pm, m_new);
    l = fmaf(l, was, pl * now);
    o = fmaf(o, was, po * now);
    m = m_new;
  }
  float f = 1.f;
  if (a.sinks) {
    const float m_new = fmaxf(m, a.sinks[h]);
    f = expf(m - m_new);
    l = fmaf(l, f, expf(a.sinks[h] - m_new));
  }
  f = f * (1.0f / l);
  a.out[((size_t)a.cu_q[seq] * a.nq + h) * D + d] = o * f;
}

// heads: query heads of a block's rows, a divisor of those that share a kv head, at most 8.  decode: every sequence
// brings one token; n_parts: the most tiles that a sequence's visible keys lie in; `group` sequences go at a time, whose
// parts the scratch holds.  Blocks are numbered along one axis, heads first, so that no number of sequences, tiles or
// tokens that a step can have is beyond a grid.
GB_EXPORT int gb_attn_f32(const AttnF32Args* args, int decode, int group, cudaStream_t stream) {
  AttnF32Args a = *args;
  if (a.n_seqs <= 0 || a.nq <= 0 || a.nkv <= 0 || a.nq % a.nkv || a.max_pages <= 0 || a.page <= 0 || a.n_qblocks < 0 ||
      a.chunk < 0 || a.n_parts < 1 || a.heads < 1 || a.heads > 8 || (a.nq / a.nkv) % a.heads)
    return GB_ERR_BAD_ARG;
  if (a.D % 4 || a.D < 4 || a.D > 128 || a.nq > 65535 || ((size_t)a.q & 15) || ((size_t)a.out & 15) ||
      ((size_t)a.k_pages & 15) || ((size_t)a.v_pages & 15))
    return GB_ERR_UNSUPPORTED;
  const long long heads = a.nq / a.heads;
  if (!decode) {
    constexpr int RT = 4, TY = 8;
    if (heads * a.n_qblocks > 0x7fffffffll) return GB_ERR_UNSUPPORTED;
    if (!a.n_qblocks) return 0;
    const size_t smem = ((size_t)(RT * TY + AF_BN) * (a.D + 4) + AF_BN * a.D + RT * TY * (AF_BN + 4)) * sizeof(float);
    auto* kernel = attn_f32_prompt_kernel<RT, TY>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return (int)e;
    return gb_launch(kernel, dim3((unsigned)(heads * a.n_qblocks)), dim3(TY * AF_LANES), smem, stream, a);
  }
  if (!a.parts || group < 1) return GB_ERR_BAD_ARG;
  if (heads * a.n_parts * (group < a.n_seqs ? group : a.n_seqs) > 0x7fffffffll) return GB_ERR_UNSUPPORTED;
  const size_t smem = ((size_t)AF_BN * (a.D + 4) + AF_BN * a.D + a.heads * (a.D + AF_BN)) * sizeof(float);
  cudaError_t e = cudaFuncSetAttribute(attn_f32_decode_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 80 * 1024);
  if (e != cudaSuccess) return (int)e;
  for (int s = 0; s < args->n_seqs; s += group) {
    a.cu_q = args->cu_q + s, a.slots = args->slots + s, a.kv_len = args->kv_len + s;
    a.n_seqs = args->n_seqs - s < group ? args->n_seqs - s : group;
    int rc = gb_launch(attn_f32_decode_kernel, dim3((unsigned)(heads * a.n_seqs * a.n_parts)), dim3(AD_THREADS), smem, stream,
                       a);
    if (!rc) rc = gb_launch(attn_f32_merge_kernel, dim3(a.n_seqs, a.nq), dim3(a.D), 0, stream, a);
    if (rc) return rc;
  }
  return 0;
}
