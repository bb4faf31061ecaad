// All layers of a decode step of few rows as one persistent kernel.
//
// A decode step of few sequences reads every weight once and does next to nothing with it, so it
// is bound by HBM; launched kernel by kernel it is bound by the hand-overs instead (eight or nine
// dependent kernels a layer, some 3 to 4 us each, while nothing streams).  Here one block per SM
// runs the whole stack: one lane streams everything this block will read in the step, weights and
// cached keys and values of every layer in order, through a ring of shared memory, and never
// waits for a result: none of that data is written in this step.  The other warps compute from
// the ring and meet the other blocks at a grid-wide barrier after each product; while they do,
// the ring (some 200 KB a block, 4.5 us of the GPU's copy rate) fills with the next product's
// weights.
//
// A layer is five phases, each ended by a barrier:
//   qkv        the block's share of the rows of the fused q|k|v weight;
//   attention  the block's share of the (sequence, kv head) pairs or of their key tiles: per-head
//              norm and rotation of q and the new key, the new key and value into the pages, the
//              tiles, the splits' partial results (when no pair is split, the finished output);
//   merge      (only when a pair is split) the splits of the block's (sequence, head) rows;
//   o          the block's columns of the residual stream, x += W_o a, which stay in its
//              registers for the whole step;
//   gate|up    silu(gate) * up of the block's features;
//   down       x += W_d h.
// A norm is no phase: whoever owns a column of x publishes bf16(x * w) (w: the weight of the
// norm in front of the next product) and its share of the sum of squares; 1 / rms is a factor of
// the next product's finished sums.  (The rounding is that of the normalised value: scaling by a
// common factor changes no relative error.)
//
// Products: mma.sync m16n8k16 with 16 weight rows as A (ldmatrix from the ring's 128-byte
// swizzled tiles) and up to eight activation rows as B.  tcgen05 has no tile this narrow in use:
// an SM gets 23 bytes of weights a clock, one such instruction every 22 clocks.  The activations
// lie in global memory in the order of B's fragments (stack_fragment); a lane of its own has
// them copied into the ring's slots beside the weights as soon as the barrier in front of them is passed.
// The warps divide a stage's columns or rows, and their sums meet in shared memory in a fixed
// order.  Sums are 32-bit throughout.
//
// Every wait (a stage of the ring, the grid barrier) is bounded by wall-clock time; a block that
// gives up records a code and says so to the others, and each block lets its copies in flight land
// and leaves.  The launch is cooperative: all blocks are resident or none.
#include <stddef.h>

#include "tc_common.cuh"

#include "attn_mma.cuh"

#define DS_FOURS 3                          // fours of consumer warps, which take turns at the ring's stages
#define DS_WARPS (4 * DS_FOURS)             // consumer warps; warp DS_WARPS feeds the ring (128 registers a thread)
#define DS_CONSUMERS (DS_WARPS * 32)
#define DS_THREADS (DS_CONSUMERS + 64)      // warp DS_WARPS + 1 brings the activations
#define DS_BLOCKS_MOST 160
#define DS_ROWS 8                           // most activation rows
#define DS_FEW 4                            // up to so many, o and down have longer stages
#define DS_TILES 3                          // most 16-row tiles a warp holds sums of
#define DS_SLOTS_MOST 12
#define DS_SPLITS_MOST 32
#define DS_UNITS_MOST 2                     // attention units of a block
#define DS_RED_BYTES 17408                  // where the warps' sums meet
#define DS_OWN_MOST 32                      // most columns of the stream a block owns
#define DS_TILE_BYTES (64 * 128)            // 64 keys x 64 elements
#define DS_SMEM_MOST 232448
#define DS_PAGES 128
#define DS_QLD 136                          // row pitch of the queries in shared memory

#define GB_ERR_STACK_STAGE 151     // a stage of the ring never arrived
#define GB_ERR_STACK_RING 152      // a stage of the ring was never released
#define GB_ERR_STACK_BARRIER 153   // the grid's barrier was never complete

struct StackLayer {
  // [0]: boxes of the smaller, [1]: of the larger number of rows a block has
  CUtensorMap qkv[2], o[2][2], gate_up[2], down[2][2];     // (o, down: [few, more rows of activations][..])
  CUtensorMap half;                // half a group of eight gates and their ups: 4 + 4 rows
  CUtensorMap k, v;
};
// What else a layer has: its pages and the weights of its norms (in front of qkv and of gate|up, of q and of k) where
// they lie, and whether these are bfloat16 or 32-bit.  Both are read from there by every launch.
struct StackRow {
  bf16* pages[2];
  const void* norm[4];
  int narrow[4];
};
static_assert(sizeof(StackRow) == 64, "copied in four pieces");
static_assert(sizeof(StackLayer) % 64 == 0, "tensor maps are 64-byte aligned");

struct StackArgs {
  const StackLayer* layers;
  const StackRow* rows;                      // [n_layers]
  int n_layers, T, hidden, ff, nq, nkv;      // T: activation rows = sequences, head size 128
  int slot_bytes, n_slots, act_at;           // the ring, where a slot's activations begin
  int kb_qkv, kb_o, kb_down;                 // 64-column blocks of a stage
  int qk_norm;                               // whether the heads of q and k have norms
  float eps, qk_eps, scale_log2;
  const bf16* x_in;                          // [T, hidden]: the stream in front of the first layer
  const float* res_in;                       // or the same in 32-bit
  float* x_out;                              // [T, hidden]: the stream behind the last layer
  const float* inv_freq;                     // [64] or null
  const int *slots, *kv_len;                 // [T]
  const int* block_table;
  int max_pages;
  bf16 *xb, *ab, *hb;                        // activations in fragment order
  float* ss;                                 // [T, P] sums of squares
  float* qkv;                                // [T, (nq + 2 nkv) * 128]
  float *part_o, *part_ml;                   // [T, nq, DS_SPLITS_MOST, 128 | 2]
  unsigned* sync;                            // [3]: arrivals, blocks that are done, whether one gave up; zero between launches
  int* error;
  unsigned long long wait_ns;                // the bound of a wait
  unsigned long long* stamps;                // optional [blocks][16] %globaltimer stamps of a layer's phases, or null
};

// Where element k of row t of T rows lies: 32 columns of a row are one 64-byte piece in which
// the lane c = 0..3 of a fragment finds its eight values (k % 8 / 2 == c) side by side.
__host__ __device__ __forceinline__ int stack_fragment(int k, int t, int T) {
  return ((k >> 5) * T + t) * 32 + ((k & 7) >> 1) * 8 + ((k >> 3) & 3) * 2 + (k & 1);
}

// The rows of a product of N rows fall to the P blocks in order, N / P or one more to a block.
__host__ __device__ __forceinline__ int stack_first_row(int N, int p, int P) { return (int)((unsigned)N * p / P); }

// Gates and ups lie in groups of eight gate rows and their eight up rows; a block's share counts
// half groups (four gates, four ups).  Blocks with an odd number of halves come first, two of
// them to an odd number of whole groups, so a share is whole groups and at most one half, behind
// them (even block) or in front (odd block).
struct StackShare {
  int first, whole, half;      // first whole group, whole groups, the half group's number in halves or -1
};
__host__ __device__ __forceinline__ StackShare stack_share(int groups, int p, int P) {
  const int H = 2 * groups, base = H / P, rem = H - base * P;
  const int odd = (base & 1) ? base : base + 1, even = (base & 1) ? base + 1 : base;
  const int n_odd = (base & 1) ? P - rem : rem;
  StackShare s;
  if (p < n_odd) {
    const int start = (p >> 1) * 2 * odd + (p & 1) * odd;
    s.whole = odd >> 1;
    s.first = (start + (p & 1)) >> 1;
    s.half = (p & 1) ? start : start + odd - 1;
  } else {
    s.first = (n_odd * odd + (p - n_odd) * even) >> 1;
    s.whole = even >> 1;
    s.half = -1;
  }
  return s;
}

__device__ __forceinline__ void ds_sync() { asm volatile("bar.sync 1, %0;" ::"n"(DS_CONSUMERS) : "memory"); }
// The same, and whether any of the threads says so.
__device__ __forceinline__ bool ds_sync_or(bool mine) {
  uint32_t any;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.u32 p, %1, 0;\n\t"
      "barrier.cta.red.or.pred q, 1, %2, p;\n\t"
      "selp.b32 %0, 1, 0, q;\n\t}"
      : "=r"(any)
      : "r"((uint32_t)mine), "n"(DS_CONSUMERS)
      : "memory");
  return any != 0;
}
__device__ __forceinline__ uint32_t ds_load_acquire(const unsigned* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void ds_add_release(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z, void* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tma_load_4d(void* dst, const CUtensorMap* map, int x, int y, int z, int w, void* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5, %6}], [%2];" ::"r"(smem_u32(dst)),
      "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y), "r"(z), "r"(w)
      : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void lds4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
// Writes to global memory that other blocks' bulk copies will read.
__device__ __forceinline__ void ds_fence_async() { asm volatile("fence.proxy.async.global;" ::: "memory"); }
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, int bytes, void* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst), "l"(src),
      "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ uint32_t transposed8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}

// The attention's work: a unit is one split of one (sequence, kv head) pair.
struct StackUnit {
  int seq, kvh, tile0, tiles, split, splits, slot, len, page;      // page: of the new key
};

// Tiles a unit takes: the fewest, DS_FOURS or more (as many tiles are taken at once), that make no
// more units than there are blocks.  A pair of so few tiles is one unit.
__device__ __forceinline__ int stack_unit_tiles(const int* tiles, int T, int nkv, int P) {
  int longest = 1, sum = 0;
#pragma unroll 1
  for (int t = 0; t < T; ++t) longest = max(longest, tiles[t]), sum += tiles[t];
#pragma unroll 1
  for (int u = max(DS_FOURS, sum * nkv / P); u < longest; ++u) {
    int total = 0, most = 0;
#pragma unroll 1
    for (int t = 0; t < T; ++t) {
      const int s = (tiles[t] + u - 1) / u;
      total += s * nkv;
      most = max(most, s);
    }
    if (total <= P && most <= DS_SPLITS_MOST) return u;
  }
  return max(longest, DS_FOURS);
}

struct StackShared {
  uint64_t full[DS_SLOTS_MOST], empty[DS_SLOTS_MOST];
  float2 turn[DS_UNITS_MOST][64];        // cosine and sine of a unit's new position
  float rstd[DS_ROWS];
  float ss[DS_ROWS * DS_BLOCKS_MOST];    // the blocks' sums of squares, on their way while a product runs
  uint32_t norm[DS_ROWS * 32];           // the weights of the norm behind o or down as they lie in memory, a copy a row
  uint32_t qk_w[256];                    // those of the layer's norms of q and k, 128 words each
  StackRow rows[2];                      // of the layers with even and odd numbers
  float red_m[DS_WARPS * 8], red_l[DS_WARPS * 8];
  StackUnit units[DS_UNITS_MOST];
  int n_units, split_any;
  int tiles[DS_ROWS];
  int pages[DS_PAGES];                   // of the block's tiles, as far as there is room
  int abort, issued, go;                 // issued: stages asked for; go: phases whose activations are there
};

static_assert(offsetof(StackShared, turn) % 16 == 0 && offsetof(StackShared, qk_w) % 16 == 0 &&
                  offsetof(StackShared, rows) % 16 == 0,
              "copied or read by 16 bytes");

// A place in the order of stages, which is the same for the warps that fill the ring and for
// those that empty it: every phase's loop counts stages from the same numbers.
struct StackRing {
  int slot;
  uint32_t round;
  __device__ __forceinline__ void skip(int k, int n) {        // k <= n
    slot += k;
    if (slot >= n) {
      slot -= n;
      ++round;
    }
  }
};

// Waits, as a whole warp, until a counter of the block is beyond a value; false when a wait has given up.
__device__ __forceinline__ bool stack_until(volatile int* count, int more_than, volatile int* abort_flag,
                                            unsigned long long wait_ns) {
  if (__all_sync(0xffffffffu, *count > more_than)) return true;
  const unsigned long long t0 = now_ns();
#pragma unroll 1
  for (int i = 1;; ++i) {
    if (__all_sync(0xffffffffu, *count > more_than)) return true;
    if ((i & 63) == 0 && __any_sync(0xffffffffu, *abort_flag || now_ns() - t0 > wait_ns)) return false;
  }
}

// A wait of this block has given up: the launch's results are void, and the block and the others leave.  (The error flag
// is the host's; another kernel's error, which it may hold from before, is no reason to leave.)
__device__ __forceinline__ void stack_give_up(const StackArgs& a, StackShared& sh, int code) {
  if (!*(volatile int*)&sh.abort) atomicCAS(a.error, 0, code);
  *(volatile int*)&sh.abort = 1;
  *(volatile unsigned*)(a.sync + 2) = 1;
}

struct StackConsumer {
  const StackArgs& a;
  StackShared& sh;
  uint8_t* ring;
  float* red;
  StackRing at;                // the first stage of the phase
  int tid, warp, lane, p, P, c0, c_rows;
  bool bad;
  int gone;
  unsigned arrived;            // arrivals the grid barrier has had when all have come

  __device__ __forceinline__ void give_up(int code) {
    if (lane == 0) stack_give_up(a, sh, code);
    bad = true;
  }
  // (A slot's stage may be another four's than the one before it, which may not have landed yet: before a barrier is
  // asked about a stage, the stage has to be on its way, or the answer may be about the stage before the last.)
  __device__ __forceinline__ void wait_full(const StackRing& r) {
    if (bad) return;
    if (!stack_until(&sh.issued, (int)r.round * a.n_slots + r.slot, &sh.abort, a.wait_ns) ||
        !mbar_wait_warp(&sh.full[r.slot], r.round & 1, &sh.abort, a.wait_ns))
      give_up(GB_ERR_STACK_STAGE);
  }
  // (Not behind a wait that has given up: the stage may be on its way, and another must not be copied over it.)
  __device__ __forceinline__ void release(const StackRing& r) {
    __syncwarp();
    if (lane == 0 && !bad) mbar_arrive(&sh.empty[r.slot]);
  }
  __device__ __forceinline__ void pass(int stages) {
    const int to = at.slot + stages, rounds = to / a.n_slots;
    at.round += rounds;
    at.slot = to - rounds * a.n_slots;
  }

  // All blocks have come this far, and what they have written can be read.  False: some wait gave up.
  __device__ __forceinline__ bool grid_sync() {
    if (ds_sync_or(bad)) {
      bad = true;
      return false;
    }
    arrived += P;
    if (tid == 0) {
      ds_add_release(a.sync, 1);
      const unsigned long long t0 = now_ns();
#pragma unroll 1
      for (int i = 1; ds_load_acquire(a.sync) < arrived; ++i) {
        if ((i & 255) == 0 && (now_ns() - t0 > a.wait_ns || *(volatile unsigned*)(a.sync + 2))) {
          stack_give_up(a, sh, GB_ERR_STACK_BARRIER);
          bad = true;
          break;
        }
      }
    }
    if (ds_sync_or(bad)) {
      bad = true;
      return false;
    }
    return true;
  }
  // The activations of the phase that begins can be brought in.
  __device__ __forceinline__ void go() {
    if (tid == 0) {
      __threadfence_block();
      *(volatile int*)&sh.go = ++gone;
    }
  }

  // What the phase needs behind its product, asked for in front of it: read where it is used, each cost a trip to
  // L2 or, the weights between one step and the next having been through it, to memory.
  // In front of a product of normalised rows the blocks' sums of squares (a warp a row), of qkv the attention's vectors
  // and where the next layer's lie too; else the weights of the next norm, `which` of `row`.
  __device__ __forceinline__ void ask(int layer, const StackRow& row, int which, bool normed, bool qkv) {
    if (warp < a.T) {
      if (normed) {
        for (int i = lane; i < P; i += 32)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(sh.ss + warp * DS_BLOCKS_MOST + i)),
                       "l"(a.ss + warp * P + i)
                       : "memory");
      } else {
        // (the words in which the block's columns lie, two columns a word where they are bfloat16)
        const int narrow = row.narrow[which], word0 = c0 >> narrow, words = ((c0 + c_rows - 1) >> narrow) - word0 + 1;
        if (lane < words)
          asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(sh.norm + warp * 32 + lane)),
                       "l"(static_cast<const uint32_t*>(row.norm[which]) + word0 + lane)
                       : "memory");
      }
    } else if (qkv && warp >= DS_ROWS) {
      const int j = warp - DS_ROWS;                // q's, k's, the next layer's
      if (j < 2) {
        if (a.qk_norm && lane < (row.narrow[2 + j] ? 16 : 32))
          cp_async16(sh.qk_w + j * 128 + lane * 4, static_cast<const uint32_t*>(row.norm[2 + j]) + lane * 4, true);
      } else if (j == 2 && lane < 4 && layer + 1 < a.n_layers) {
        cp_async16(reinterpret_cast<uint4*>(&sh.rows[(layer + 1) & 1]) + lane,
                   reinterpret_cast<const uint4*>(a.rows + layer + 1) + lane, true);
      }
    }
    cp_async_commit();
  }
  // Element i of weights that begin with the word at `w`.
  __device__ __forceinline__ static float widened(const uint32_t* w, int i, int narrow) {
    if (!narrow) return __uint_as_float(w[i]);
    return __uint_as_float((i & 1) ? w[i >> 1] & 0xffff0000u : w[i >> 1] << 16);
  }
  // Elements 2 i and 2 i + 1.
  __device__ __forceinline__ static float2 widened2(const uint32_t* w, int i, int narrow) {
    if (!narrow) return reinterpret_cast<const float2*>(w)[i];
    return make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
  }
  // 1 / rms of the rows
  __device__ __forceinline__ void row_factors() {
    if (warp < a.T) {
      float s = 0.f;
      for (int i = lane; i < P; i += 32) s += sh.ss[warp * DS_BLOCKS_MOST + i];      // (what this lane asked for)
      s = warp_sum(s);
      if (lane == 0) sh.rstd[warp] = rsqrtf(s / (float)a.hidden + a.eps);
    }
  }

  // The product of `rows` weight rows with the T activation rows, K columns, kb blocks of 64 a stage: the warps' sums
  // in `red` as [part][activation row][pitch], summed up by whoever reads them over the `parts` it returns.
  //
  // Four warps take a stage, the fours taking turns, so that a four has the time of several stages for its waits and
  // instructions; among them they divide the stage's steps of 32 columns, or its 16-row tiles where there are more than
  // three, or both two by two where twelve partial sums of three tiles have no room.  A warp asks for the operands of
  // two steps before it multiplies: one step after the other a stage of six steps took it 0.85 us.
  __device__ __forceinline__ int product(int K, int rows, int kb, int& pitch) {
    const int steps = 2 * kb, K32 = K >> 5, tiles = (rows + 15) >> 4;
    const int stages = (K / 64 + kb - 1) / kb;
    pitch = ((rows + 11) & ~15) + 4;
    const int j = warp & 3, quad = warp >> 2;
    // log2 of the ways in which the tiles are divided; the steps are divided in 4 >> ways
    const int ways = tiles > 3 ? 2 : (DS_WARPS * a.T * pitch * 4 > DS_RED_BYTES ? 1 : 0);
    const int t_off = j & ((1 << ways) - 1), s_off = j >> ways, s_inc = 4 >> ways;
    const int part = quad * s_inc + s_off, parts = DS_FOURS * s_inc;
    const int n_tiles = (tiles - t_off + (1 << ways) - 1) >> ways;
    const int g = lane >> 2, c = lane & 3;
    // Two sums a tile, so that no product waits for the one before it: a warp issues in order, and one chain of eight
    // took a four 0.97 us a stage.  The odd tile's are the last ones.
    float acc[DS_TILES][2][4];
#pragma unroll
    for (int i = 0; i < DS_TILES; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][0][e] = acc[i][1][e] = 0.f;
    // (columns beyond the rows get some other row's values: nobody reads what becomes of them)
    const uint32_t act = a.act_at + min(g, a.T - 1) * 64 + c * 16, act_pitch = a.T * 64;
    const uint32_t ring32 = smem_u32(ring), tile_pitch = 2048u << ways;
    const uint32_t half = lane >> 4, lane_row = (lane & 15) + t_off * 16;
    int s = quad;
    StackRing r = at;
    r.skip(s, a.n_slots);
#pragma unroll 1
    for (; s < stages; s += DS_FOURS) {
      wait_full(r);
      const uint32_t base = ring32 + (uint32_t)r.slot * a.slot_bytes;
      const int end = min(steps, K32 - s * steps);
#pragma unroll
      for (int i = 0; i < 4; i += 2) {
        const int step0 = s_off + i * s_inc;
        if (step0 < end) {
          const bool two = step0 + s_inc < end;
          const int step1 = two ? step0 + s_inc : step0;
          const uint32_t row0 = (step0 >> 1) * rows + lane_row, row1 = (step1 >> 1) * rows + lane_row;
          // (a step is four 16-byte chunks of a 64-column block; the second pair of them is two chunks on)
          const uint32_t w0 = base + row0 * 128 + ((((step0 & 1) * 4 + half) ^ (row0 & 7)) << 4);
          const uint32_t w1 = base + row1 * 128 + ((((step1 & 1) * 4 + half) ^ (row1 & 7)) << 4);
          uint32_t f0[4], f1[4], w[2][4][4];
          lds4(f0, base + act + step0 * act_pitch);
          lds4(f1, base + act + step1 * act_pitch);
          auto load = [&](int t, uint32_t (&v)[4][4]) {
            ldsm4(v[0], w0 + t * tile_pitch);
            ldsm4(v[1], (w0 ^ 32u) + t * tile_pitch);
            ldsm4(v[2], w1 + t * tile_pitch);
            ldsm4(v[3], (w1 ^ 32u) + t * tile_pitch);
          };
          if (n_tiles > 1) {
            load(0, w[0]);
            load(1, w[1]);
            mma_16816(acc[0][0], w[0][0], f0[0], f0[1]);
            mma_16816(acc[1][0], w[1][0], f0[0], f0[1]);
            mma_16816(acc[0][1], w[0][1], f0[2], f0[3]);
            mma_16816(acc[1][1], w[1][1], f0[2], f0[3]);
            if (two) {
              mma_16816(acc[0][0], w[0][2], f1[0], f1[1]);
              mma_16816(acc[1][0], w[1][2], f1[0], f1[1]);
              mma_16816(acc[0][1], w[0][3], f1[2], f1[3]);
              mma_16816(acc[1][1], w[1][3], f1[2], f1[3]);
            }
          }
          if (n_tiles & 1) {                     // (the third, or the only one)
            float(&last)[2][4] = acc[2];
            load(n_tiles - 1, w[0]);
            mma_16816(last[0], w[0][0], f0[0], f0[1]);
            mma_16816(last[1], w[0][1], f0[2], f0[3]);
            if (two) {
              mma_16816(last[0], w[0][2], f1[0], f1[1]);
              mma_16816(last[1], w[0][3], f1[2], f1[3]);
            }
          }
        }
      }
      release(r);
      r.skip(DS_FOURS, a.n_slots);
    }
    pass(stages);
    float* out = red + part * a.T * pitch;
#pragma unroll
    for (int i = 0; i < DS_TILES; ++i) {
      const int t = i == 2 ? n_tiles - 1 : i;
      if (i == 2 ? (n_tiles & 1) : n_tiles > 1) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int rr = (t_off + (t << ways)) * 16 + g + (e >> 1) * 8, col = 2 * c + (e & 1);
          if (rr < rows && col < a.T) out[col * pitch + rr] = acc[i][0][e] + acc[i][1][e];
        }
      }
    }
    return parts;
  }

  // A sum over the parts, in their order, from loads that do not wait for one another.
  __device__ __forceinline__ float summed(const float* at0, int parts, int stride) {
    float v[DS_WARPS], s = 0.f;
#pragma unroll
    for (int i = 0; i < DS_WARPS; ++i) v[i] = i < parts ? at0[i * stride] : 0.f;
#pragma unroll
    for (int i = 0; i < DS_WARPS; ++i) s += v[i];
    return s;
  }

  // The block's share of a row's sum of squares.
  __device__ __forceinline__ void publish(int row, float sq) {
    sq = warp_sum(sq);
    if (lane == 0) a.ss[row * P + p] = sq;
  }

  // ---- attention -----------------------------------------------------------------------------
  __device__ __forceinline__ void attention(const StackRow& row) {
    const int G = a.nq / a.nkv, N = (a.nq + 2 * a.nkv) * 128;
    const int g = lane >> 2, c = lane & 3;
    bf16* q_s = reinterpret_cast<bf16*>(red);              // [8][DS_QLD]
    bf16* k_new = q_s + 8 * DS_QLD;                        // [128] each
    bf16* v_new = k_new + 128;
    const uint32_t ring32 = smem_u32(ring);
#pragma unroll 1
    for (int ui = 0; ui < sh.n_units; ++ui) {
      const StackUnit u = sh.units[ui];
      const int pos = u.len - 1;
      const bool fresh = u.tiles > 0 && u.tile0 + u.tiles == (u.len + 63) / 64;      // the unit with the new key
      // queries and the new key: a warp a head (four values a lane: j, j + 1 and their partners
      // 64 further on); the new value
      if (warp < G || (warp <= G + 1 && fresh)) {
        const int head = warp < G ? u.kvh * G + warp : (warp == G ? a.nq + u.kvh : a.nq + a.nkv + u.kvh);
        const bool is_v = warp == G + 1;
        const float* src = a.qkv + (size_t)u.seq * N + head * 128;
        const float2 lo = __ldcg(reinterpret_cast<const float2*>(src) + lane);
        const float2 hi = __ldcg(reinterpret_cast<const float2*>(src + 64) + lane);
        float x0 = lo.x, x1 = lo.y, y0 = hi.x, y1 = hi.y;
        if (a.qk_norm && !is_v) {
          const uint32_t* w = sh.qk_w + (warp < G ? 0 : 128);
          const int narrow = row.narrow[warp < G ? 2 : 3];
          const float ssq = warp_sum(x0 * x0 + x1 * x1 + y0 * y0 + y1 * y1);
          const float f = rsqrtf(ssq / 128.f + a.qk_eps);
          const float2 wl = widened2(w, lane, narrow), wh = widened2(w, 32 + lane, narrow);
          x0 = x0 * f * wl.x, x1 = x1 * f * wl.y, y0 = y0 * f * wh.x, y1 = y1 * f * wh.y;
        }
        if (a.inv_freq && !is_v) {
          const float4 cs = reinterpret_cast<const float4*>(sh.turn[ui])[lane];
          const float r0 = x0 * cs.x - y0 * cs.y, r1 = x1 * cs.z - y1 * cs.w;
          y0 = y0 * cs.x + x0 * cs.y, y1 = y1 * cs.z + x1 * cs.w;
          x0 = r0, x1 = r1;
        }
        bf16* dst = warp < G ? q_s + warp * DS_QLD : (is_v ? v_new : k_new);
        const uint32_t p0 = pack2(x0, x1), p1 = pack2(y0, y1);
        reinterpret_cast<uint32_t*>(dst)[lane] = p0;
        reinterpret_cast<uint32_t*>(dst + 64)[lane] = p1;
        if (warp >= G) {
          bf16* page = row.pages[is_v] + (((size_t)u.page * a.nkv + u.kvh) * 64 + (pos & 63)) * 128;
          reinterpret_cast<uint32_t*>(page)[lane] = p0;
          reinterpret_cast<uint32_t*>(page + 64)[lane] = p1;
        }
      } else if (warp >= G + 2 && warp < 10) {       // the rows without a head are zero
        uint32_t* row = reinterpret_cast<uint32_t*>(q_s + (warp - 2) * DS_QLD);
        row[lane] = 0u, row[lane + 32] = 0u;
      }
      ds_sync();
      uint32_t q[8][2];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        q[k][0] = *reinterpret_cast<const uint32_t*>(q_s + g * DS_QLD + k * 16 + 2 * c);
        q[k][1] = *reinterpret_cast<const uint32_t*>(q_s + g * DS_QLD + k * 16 + 8 + 2 * c);
      }
      float o[8][4];
#pragma unroll
      for (int i = 0; i < 8; ++i) o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f;
      float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
      // four warps a tile, 16 keys each
      const int key_w = (warp & 3) * 16;
      StackRing r = at;
      r.skip(2 * (warp >> 2), a.n_slots);
#pragma unroll 1
      for (int i = warp >> 2; i < u.tiles; i += DS_FOURS) {
        wait_full(r);
        const int tile = u.tile0 + i;
        const bool last = tile * 64 + 63 >= pos;           // holds the new key, and rows beyond it
        const int row_new = pos - tile * 64;               // (of the tile)
        uint8_t* tile_p = ring + (size_t)r.slot * a.slot_bytes;
        bool wrote = false;
        if (last && row_new >= key_w && row_new < key_w + 16) {
          if (lane < 16)
            *reinterpret_cast<uint4*>(tile_p + (lane >> 3) * DS_TILE_BYTES + row_new * 128 +
                                      (((lane & 7) ^ (row_new & 7)) << 4)) = *reinterpret_cast<const uint4*>(k_new + lane * 8);
          wrote = true;
          __syncwarp();
        }
        float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
        {
          const int kr = key_w + (lane & 15);
          const uint32_t rb = ring32 + (uint32_t)r.slot * a.slot_bytes + kr * 128;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            uint32_t w[4];
            const int ch = (k & 3) * 2 + (lane >> 4);
            ldsm4(w, rb + (k >> 2) * DS_TILE_BYTES + ((ch ^ (kr & 7)) << 4));
            mma_16816((k & 1) ? s1 : s0, w, q[k][0], q[k][1]);
          }
        }
        if (wrote) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        release(r);
        r.skip(1, a.n_slots);
        // rows: keys g and g + 8; columns: heads 2c and 2c + 1
        float s[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[e] = (s0[e] + s1[e]) * a.scale_log2;
          if (last && tile * 64 + key_w + g + (e >> 1) * 8 > pos) s[e] = -INFINITY;
        }
        float corr[2], pr[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          float mx = fmaxf(s[h], s[h + 2]);
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
          const float mn = fmaxf(m[h], mx);
          const float from = mn == -INFINITY ? 0.f : mn;
          corr[h] = m[h] == -INFINITY ? 0.f : exp2f(m[h] - from);
          m[h] = mn;
          pr[h] = exp2f(s[h] - from);
          pr[h + 2] = exp2f(s[h + 2] - from);
          l[h] = l[h] * corr[h] + pr[h] + pr[h + 2];
        }
        const uint32_t b0 = transposed8x8(pack2(pr[0], pr[1])), b1 = transposed8x8(pack2(pr[2], pr[3]));
#pragma unroll
        for (int d = 0; d < 8; ++d) o[d][0] *= corr[0], o[d][1] *= corr[1], o[d][2] *= corr[0], o[d][3] *= corr[1];
        wait_full(r);
        tile_p = ring + (size_t)r.slot * a.slot_bytes;
        wrote = false;
        if (last && row_new < key_w + 16) {                // the new value; zeros where there is no key yet
#pragma unroll 1
          for (int j = lane; j < 256; j += 32) {
            const int vr = key_w + (j >> 4), ch = j & 15;
            if (vr >= row_new) {
              uint4 v = make_uint4(0, 0, 0, 0);
              if (vr == row_new) v = *reinterpret_cast<const uint4*>(v_new + ch * 8);
              *reinterpret_cast<uint4*>(tile_p + (ch >> 3) * DS_TILE_BYTES + vr * 128 + (((ch & 7) ^ (vr & 7)) << 4)) = v;
            }
          }
          wrote = true;
          __syncwarp();
        }
        {
          const int vr = key_w + (lane & 7) + ((lane >> 4) & 1) * 8;
          const uint32_t rb = ring32 + (uint32_t)r.slot * a.slot_bytes + vr * 128;
#pragma unroll
          for (int d = 0; d < 8; ++d) {
            uint32_t w[4];
            const int ch = (d & 3) * 2 + ((lane >> 3) & 1);
            ldsm4_t(w, rb + (d >> 2) * DS_TILE_BYTES + ((ch ^ (vr & 7)) << 4));
            mma_16816(o[d], w, b0, b1);
          }
        }
        if (wrote) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        release(r);
        r.skip(2 * DS_FOURS - 1, a.n_slots);
      }
      pass(2 * u.tiles);
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 4);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 8);
        l[h] += __shfl_xor_sync(0xffffffffu, l[h], 16);
        if (g == 0) {
          sh.red_m[warp * 8 + 2 * c + h] = m[h];
          sh.red_l[warp * 8 + 2 * c + h] = l[h];
        }
      }
      ds_sync();                                           // (everyone is done with q_s, k_new, v_new)
      const int nw = 4 * min(DS_FOURS, u.tiles);           // warps that took a tile
      float f[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        float M = -INFINITY;
#pragma unroll 1
        for (int w = 0; w < nw; w += 4) {
          const float* x = sh.red_m + w * 8 + 2 * c + h;
          M = fmaxf(fmaxf(fmaxf(M, x[0]), fmaxf(x[8], x[16])), x[24]);
        }
        f[h] = m[h] == -INFINITY ? 0.f : exp2f(m[h] - M);
      }
      // as many of the 128 columns at once as there is room for
      const int sh_cols = nw * G <= 32 ? 7 : (nw * G <= 48 ? 6 : 5), cols = 1 << sh_cols;
      const int pitch = cols + 8;
#pragma unroll 1
      for (int d0 = 0; d0 < 128; d0 += cols) {
        if (d0) ds_sync();
        if (warp < nw) {
#pragma unroll
          for (int d = 0; d < 8; ++d) {
            const int col = d * 16 - d0;
            if (col >= 0 && col < cols) {
              float* x = red + (warp * G + 2 * c) * pitch + col + g;
              if (2 * c < G) x[0] = o[d][0] * f[0], x[8] = o[d][2] * f[0];
              if (2 * c + 1 < G) x[pitch] = o[d][1] * f[1], x[pitch + 8] = o[d][3] * f[1];
            }
          }
        }
        ds_sync();
#pragma unroll 1
        for (int i = tid; i < (G << sh_cols); i += DS_CONSUMERS) {
          const int h = i >> sh_cols, col = i & (cols - 1);
          float O = 0.f;
          const float* x = red + h * pitch + col;
#pragma unroll 1
          for (int w = 0; w < nw; w += 4) {
            const float v0 = x[0], v1 = x[G * pitch], v2 = x[2 * G * pitch], v3 = x[3 * G * pitch];
            O += v0, O += v1, O += v2, O += v3;
            x += 4 * G * pitch;
          }
          const int head = u.kvh * G + h;
          if (u.splits == 1 || col + d0 == 0) {
            float M = -INFINITY, Ls = 0.f;
#pragma unroll 1
            for (int w = 0; w < nw; w += 4) {
              const float* y = sh.red_m + w * 8 + h;
              M = fmaxf(fmaxf(fmaxf(M, y[0]), fmaxf(y[8], y[16])), y[24]);
            }
#pragma unroll 4
            for (int w = 0; w < nw; ++w) Ls += sh.red_l[w * 8 + h] * exp2f(sh.red_m[w * 8 + h] - M);   // (0 of a -inf)
            if (u.splits == 1) {
              a.ab[stack_fragment(head * 128 + d0 + col, u.seq, a.T)] = __float2bfloat16(O / Ls);
              continue;
            }
            float* ml = a.part_ml + (((size_t)u.seq * a.nq + head) * DS_SPLITS_MOST + u.split) * 2;
            ml[0] = M, ml[1] = Ls;
          }
          a.part_o[(((size_t)u.seq * a.nq + head) * DS_SPLITS_MOST + u.split) * 128 + d0 + col] = O;
        }
      }
      if (ui + 1 < sh.n_units) ds_sync();                  // red is the next unit's queries
    }
    ds_fence_async();
  }

  // The splits of the block's (sequence, head) rows, a warp a row.
  __device__ __forceinline__ void merge(int unit_tiles) {
#pragma unroll 1
    for (int item = p + P * warp; item < a.T * a.nq; item += P * DS_WARPS) {
      const int seq = item / a.nq, head = item - seq * a.nq;
      const int S = (sh.tiles[seq] + unit_tiles - 1) / unit_tiles;
      if (S <= 1) continue;              // finished already (or no sequence)
      const size_t at0 = (size_t)item * DS_SPLITS_MOST;
      float ms = -INFINITY, ls = 0.f;
      if (lane < S) {
        const float2 v = __ldcg(reinterpret_cast<const float2*>(a.part_ml) + at0 + lane);
        ms = v.x, ls = v.y;
      }
      const float4* part = reinterpret_cast<const float4*>(a.part_o + at0 * 128) + lane;
      float4 O = make_float4(0.f, 0.f, 0.f, 0.f);
      float fl = 0.f, total = 0.f;
#pragma unroll 1
      for (int s0 = 0; s0 < S; s0 += 8) {
        float4 v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = __ldcg(part + min(s0 + i, S - 1) * 32);
        if (s0 == 0) {
          const float M = warp_max(ms);
          fl = ms == -INFINITY ? 0.f : exp2f(ms - M);      // (and where there is no split: 0)
          total = warp_sum(ls * fl);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float f = s0 + i < S ? __shfl_sync(0xffffffffu, fl, (s0 + i) & 31) : 0.f;
          O.x += v[i].x * f, O.y += v[i].y * f, O.z += v[i].z * f, O.w += v[i].w * f;
        }
      }
      const float inv = 1.f / total;
      const int k = head * 128 + lane * 4;
      *reinterpret_cast<uint32_t*>(a.ab + stack_fragment(k, seq, a.T)) = pack2(O.x * inv, O.y * inv);
      *reinterpret_cast<uint32_t*>(a.ab + stack_fragment(k + 2, seq, a.T)) = pack2(O.z * inv, O.w * inv);
    }
    ds_fence_async();
  }
};

#define DS_STAMP(i)                                                                                         \
  do {                                                                                                      \
    if (a.stamps && tid == 0 && layer == a.n_layers - 2) a.stamps[(size_t)blockIdx.x * 16 + (i)] = now_ns(); \
  } while (0)

__global__ void __launch_bounds__(DS_THREADS, 1) decode_stack_kernel(const __grid_constant__ StackArgs a) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* ring = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  float* red = reinterpret_cast<float*>(ring + (size_t)a.n_slots * a.slot_bytes);
  StackShared& sh = *reinterpret_cast<StackShared*>((uint8_t*)red + DS_RED_BYTES);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int p = blockIdx.x, P = gridDim.x;
  const int N = (a.nq + 2 * a.nkv) * 128;

  if (tid == 0) {
    for (int i = 0; i < a.n_slots; ++i) {
      mbar_init(&sh.full[i], 1);
      mbar_init(&sh.empty[i], 4);
    }
    sh.abort = 0;
    sh.issued = sh.go = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1 && lane < 4) reinterpret_cast<uint4*>(&sh.rows[0])[lane] = reinterpret_cast<const uint4*>(a.rows)[lane];
  if (tid < a.T) sh.tiles[tid] = a.slots[tid] < 0 ? 0 : (a.kv_len[tid] + 63) / 64;
  __syncthreads();
  // rows of the products that are this block's
  const int q0 = stack_first_row(N, p, P), q_rows = stack_first_row(N, p + 1, P) - q0;
  const int c0 = stack_first_row(a.hidden, p, P), c_rows = stack_first_row(a.hidden, p + 1, P) - c0;
  const StackShare share = stack_share(a.ff / 8, p, P);
  const int gu_rows = share.whole * 16 + (share.half >= 0 ? 8 : 0);
  const int unit_tiles = stack_unit_tiles(sh.tiles, a.T, a.nkv, P);
  if (tid == 0) {
    int n = 0, first = 0, any = 0;
    for (int t = 0; t < a.T; ++t) {
      const int S = (sh.tiles[t] + unit_tiles - 1) / unit_tiles;
      any |= S > 1;
      const int here = S * a.nkv;
      // units p, p + P, ... of the line; unit = (sequence, kv head, split)
      for (int u = p + (first > p ? (first - p + P - 1) / P * P : 0); u < first + here; u += P) {
        if (n == DS_UNITS_MOST) break;
        StackUnit& w = sh.units[n++];
        const int r = u - first;
        w.seq = t, w.kvh = r / S, w.split = r - w.kvh * S, w.splits = S;
        const int per = (sh.tiles[t] + S - 1) / S;       // even shares of the tiles
        w.tile0 = min(sh.tiles[t], w.split * per);
        w.tiles = min(sh.tiles[t], w.tile0 + per) - w.tile0;
        w.slot = a.slots[t], w.len = a.kv_len[t];
        w.page = a.block_table[(size_t)w.slot * a.max_pages + (w.len - 1) / 64];
      }
      first += here;
    }
    sh.n_units = n;
    sh.split_any = any;
  }
  __syncthreads();
  for (int ui = 0, first = 0; ui < sh.n_units; first += sh.units[ui++].tiles)
    for (int i = tid; i < sh.units[ui].tiles && first + i < DS_PAGES; i += DS_THREADS)
      sh.pages[first + i] = a.block_table[(size_t)sh.units[ui].slot * a.max_pages + sh.units[ui].tile0 + i];
  if (a.inv_freq) {
#pragma unroll 1
    for (int i = tid; i < sh.n_units * 64; i += DS_THREADS) {
      float sn, cs;
      sincosf((float)(sh.units[i >> 6].len - 1) * a.inv_freq[i & 63], &sn, &cs);
      sh.turn[i >> 6][i & 63] = make_float2(cs, sn);
    }
  }
  __syncthreads();

  // The phases in turn, one copy of the code of each: what all warps run through again and again must stay in the
  // instruction caches (as 300 KB, with products, barriers and polls written out, fetching it took most of the time:
  // 3,240 us a step of one row at the 4B sizes).
  enum { QKV, ATTENTION, MERGE, O, GATE_UP, DOWN };

  if (warp == DS_WARPS) {
    // ------------------------------------------------------------------ the stream
    // One lane, and few instructions a stage: with a page broadcast, a vote and divisions in the loop a stage took
    // 0.45 us to ask for, whatever its size.  A stage's barrier expects its activations too, which come later.
    if (elect_one()) {
      StackRing at = {0, 0};
      bool ok = true;
      // the next stage's place, once it is free; its barrier expects `bytes`
      auto next_stage = [&](uint32_t bytes) -> uint8_t* {
        if (at.round > 0 && !mbar_wait(&sh.empty[at.slot], (at.round & 1) ^ 1, &sh.abort, a.wait_ns)) {
          stack_give_up(a, sh, GB_ERR_STACK_RING);
          ok = false;
          return nullptr;
        }
        mbar_expect_tx(&sh.full[at.slot], bytes);
        return ring + at.slot * a.slot_bytes;
      };
      auto sent = [&] {
        at.skip(1, a.n_slots);
        *(volatile int*)&sh.issued = (int)at.round * a.n_slots + at.slot;
      };
      const int more = a.T > DS_FEW, big_q = q_rows > N / P, big_c = c_rows > a.hidden / P;
      const int big_g = share.whole > 2 * (a.ff / 8) / P / 2;
#pragma unroll 1
      for (int layer = 0; layer < a.n_layers && ok; ++layer) {
        const StackLayer* L = a.layers + layer;
        if (layer + 1 < a.n_layers) {
          const StackLayer* next = L + 1;
          tma_prefetch_map(&next->qkv[big_q]);
          tma_prefetch_map(&next->o[more][big_c]);
          tma_prefetch_map(&next->gate_up[big_g]);
          tma_prefetch_map(&next->half);
          tma_prefetch_map(&next->down[more][big_c]);
          tma_prefetch_map(&next->k);
          tma_prefetch_map(&next->v);
        }
#pragma unroll 1
        for (int phase = QKV; phase <= DOWN && ok; ++phase) {
          if (phase == MERGE) continue;
          if (phase == ATTENTION) {
            int at_page = 0;
#pragma unroll 1
            for (int ui = 0; ui < sh.n_units && ok; ++ui) {
              const StackUnit& u = sh.units[ui];
              const int tiles = u.tiles, kvh = u.kvh;
              const int* table = a.block_table + (size_t)u.slot * a.max_pages + u.tile0;
#pragma unroll 1
              for (int i = 0; i < 2 * tiles && ok; ++i) {
                const int page = at_page < DS_PAGES ? sh.pages[at_page] : table[i >> 1];
                at_page += i & 1;
                const CUtensorMap* map = (i & 1) ? &L->v : &L->k;
                const int row = (page * a.nkv + kvh) * 64;
                uint8_t* dst = next_stage(2 * DS_TILE_BYTES);
                if (!ok) break;
                tma_load_2d(dst, map, 0, row, &sh.full[at.slot]);
                tma_load_2d(dst + DS_TILE_BYTES, map, 64, row, &sh.full[at.slot]);
                sent();
              }
            }
          } else if (phase == GATE_UP) {
            const int k_end = a.hidden, row0 = share.first * 16;
            const bool half = share.half >= 0;
            const int act = 128 * a.T;
            const int half_row = (share.half & 1) * 4, half_group = share.half >> 1, whole_bytes = share.whole * 2048;
#pragma unroll 1
            for (int k = 0; k < k_end; k += 64) {
              uint8_t* dst = next_stage(gu_rows * 128 + act);
              if (!ok) break;
              tma_load_2d(dst, &L->gate_up[big_g], k, row0, &sh.full[at.slot]);
              if (half) tma_load_4d(dst + whole_bytes, &L->half, k, half_row, 0, half_group, &sh.full[at.slot]);
              sent();
            }
          } else {
            const CUtensorMap* map = phase == QKV ? &L->qkv[big_q] : (phase == O ? &L->o[more][big_c] : &L->down[more][big_c]);
            const int blocks = (phase == QKV ? a.hidden : (phase == O ? a.nq * 128 : a.ff)) / 64;
            const int kb = phase == QKV ? a.kb_qkv : (phase == O ? a.kb_o : a.kb_down);
            const int row0 = phase == QKV ? q0 : c0, bytes = (phase == QKV ? q_rows : c_rows) * 128 * kb, act = 128 * a.T;
#pragma unroll 1
            for (int k = 0; k < blocks; k += kb) {
              uint8_t* dst = next_stage(bytes + act * min(kb, blocks - k));
              if (!ok) break;
              tma_load_3d(dst, map, 0, row0, k, &sh.full[at.slot]);
              sent();
            }
          }
        }
      }
    }
    __syncwarp();
  } else if (warp == DS_WARPS + 1) {
    // ------------------------------------------------------------------ the activations
    // They go where the consumers find them beside the weights, in the same order and under the same barrier, a bulk
    // copy a stage: loaded by the consumers themselves, into registers and a few stages ahead, each stage cost them a
    // trip to L2 (0.48 us), and 16-byte copies whose 32 lanes each arrive at the barrier took a warp 0.45 us a stage.
    if (elect_one()) {
      StackRing at = {0, 0};
      int gone = 0, stage = 0, issued = 0;       // issued: as last looked at
      bool ok = true;
      const uint32_t ring32 = smem_u32(ring);
      auto until = [&](volatile int* count, int more_than) -> int {
        int n = *count;
        if (n > more_than) return n;
        const unsigned long long t0 = now_ns();
#pragma unroll 1
        for (int i = 1; (n = *count) <= more_than; ++i)
          if ((i & 63) == 0 && (*(volatile int*)&sh.abort || now_ns() - t0 > a.wait_ns)) {
            ok = false;
            break;
          }
        return n;
      };
#pragma unroll 1
      for (int layer = 0; layer < a.n_layers && ok; ++layer) {
#pragma unroll 1
        for (int phase = QKV; phase <= DOWN && ok; ++phase) {
          if (phase == MERGE) continue;
          if (phase == ATTENTION) {
            int stages = 0;
            for (int ui = 0; ui < sh.n_units; ++ui) stages += 2 * sh.units[ui].tiles;
            stage += stages;
            const int to = at.slot + stages, rounds = to / a.n_slots;
            at.round += rounds;
            at.slot = to - rounds * a.n_slots;
            continue;
          }
          const int K = phase == O ? a.nq * 128 : (phase == DOWN ? a.ff : a.hidden);
          const int kb = phase == QKV ? a.kb_qkv : (phase == O ? a.kb_o : (phase == DOWN ? a.kb_down : 1));
          const int bytes = kb * 128 * a.T;
          int left = K * 2 * a.T;
          const uint8_t* src = reinterpret_cast<const uint8_t*>(phase == O ? a.ab : (phase == DOWN ? a.hb : a.xb));
          until(&sh.go, gone++);
          __threadfence_block();
          ds_fence_async();
#pragma unroll 1
          for (; left > 0 && ok; left -= bytes) {
            if (issued <= stage) issued = until(&sh.issued, stage);
            if (!ok) break;
            bulk_load(ring32 + at.slot * a.slot_bytes + a.act_at, src, min(bytes, left), &sh.full[at.slot]);
            src += bytes;
            ++stage;
            at.skip(1, a.n_slots);
          }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ the work
    StackConsumer w = {a, sh, ring, red, {0, 0}, tid, warp, lane, p, P, c0, c_rows, false, 0, 0u};
    // the block's columns of the stream: a warp a row of the batch, a lane a column
    float x = 0.f;
    if (warp < a.T) {
      if (lane < c_rows) {
        const size_t i = (size_t)warp * a.hidden + c0 + lane;
        x = a.res_in ? a.res_in[i] : __bfloat162float(a.x_in[i]);
        const StackRow& row = sh.rows[0];
        const float weight = row.narrow[0] ? __bfloat162float(static_cast<const bf16*>(row.norm[0])[c0 + lane])
                                           : static_cast<const float*>(row.norm[0])[c0 + lane];
        a.xb[stack_fragment(c0 + lane, warp, a.T)] = __float2bfloat16(x * weight);
      }
      w.publish(warp, x * x);
      ds_fence_async();
    }
    int phase = -1, layer = 0;
    bool ok = true;
#pragma unroll 1
    for (;;) {
      if (!(ok = w.grid_sync())) break;
      if (phase == DOWN) ++layer;
      phase = phase == DOWN ? QKV : phase + 1;
      if (phase == MERGE && !sh.split_any) ++phase;
      DS_STAMP(phase * 2);
      if (phase == ATTENTION) {
        w.attention(sh.rows[layer & 1]);
        DS_STAMP(phase * 2 + 1);
      } else if (phase == MERGE) {
        w.merge(unit_tiles);
        DS_STAMP(phase * 2 + 1);
      } else {
        const bool normed = phase == QKV || phase == GATE_UP;
        const int rows = phase == QKV ? q_rows : (phase == GATE_UP ? gu_rows : c_rows);
        const bool last = phase == DOWN && layer + 1 == a.n_layers;
        // whose norm comes behind the product (behind the last layer none of the stack's: its weights are read and not used)
        const int which = phase == O ? 1 : 0;
        const StackRow& row = sh.rows[(phase == DOWN && !last ? layer + 1 : layer) & 1];
        w.go();
        w.ask(layer, row, which, normed, phase == QKV);
        int pitch;
        const int parts = w.product(normed ? a.hidden : (phase == O ? a.nq * 128 : a.ff), rows,
                                    phase == QKV ? a.kb_qkv : (phase == O ? a.kb_o : (phase == DOWN ? a.kb_down : 1)), pitch);
        DS_STAMP(phase * 2 + 1);
        cp_async_wait<0>();
        if (normed) w.row_factors();
        ds_sync();
        const int stride = a.T * pitch;
        if (!normed) {
          if (warp < a.T) {
            if (lane < c_rows) {
              const int narrow = row.narrow[which];
              const float weight = w.widened(sh.norm + warp * 32, narrow ? lane + (c0 & 1) : lane, narrow);
              x += w.summed(red + warp * pitch + lane, parts, stride);
              a.xb[stack_fragment(c0 + lane, warp, a.T)] = __float2bfloat16(x * weight);
              if (last) a.x_out[(size_t)warp * a.hidden + c0 + lane] = x;
            }
            w.publish(warp, x * x);
            ds_fence_async();
          }
          if (last) break;
        } else if (phase == QKV) {
#pragma unroll 1
          for (int t = warp; t < a.T; t += DS_WARPS)
#pragma unroll 1
            for (int r = lane; r < q_rows; r += 32)
              a.qkv[(size_t)t * N + q0 + r] = w.summed(red + t * pitch + r, parts, stride) * sh.rstd[t];
        } else {
          const int whole = share.whole * 8, n = whole + (share.half >= 0 ? 4 : 0);
          const int chunks = (n + 31) >> 5;
#pragma unroll 1
          for (int i = warp; i < chunks * a.T; i += DS_WARPS) {
            const int t = i / chunks, f = (i - t * chunks) * 32 + lane;
            if (f >= n) continue;
            const bool in_whole = f < whole;
            const int rg = in_whole ? (f >> 3) * 16 + (f & 7) : share.whole * 16 + f - whole;
            const int ru = in_whole ? rg + 8 : rg + 4;
            const int feature = in_whole ? share.first * 8 + f : share.half * 4 + f - whole;
            const float* s = red + t * pitch;
            const float gate = w.summed(s + rg, parts, stride) * sh.rstd[t];
            const float up = w.summed(s + ru, parts, stride) * sh.rstd[t];
            a.hb[stack_fragment(feature, t, a.T)] = __float2bfloat16(__fdividef(gate, 1.0f + __expf(-gate)) * up);
          }
          ds_fence_async();
        }
      }
    }
    if (!ok) *(volatile int*)&sh.abort = 1;
  }
  __syncthreads();
  if (tid == 0) {
    if (sh.abort) {
      // No warp asks for copies any more: let those that were asked for land before the block leaves, each slot's last
      // stage (10 ms: where its activations were never asked for, its barrier does not complete).
      const int rounds = sh.issued / a.n_slots, more = sh.issued - rounds * a.n_slots;
#pragma unroll 1
      for (int i = 0; i < a.n_slots; ++i) {
        const int n = rounds + (i < more);
        if (n > 0) mbar_wait(&sh.full[i], (n - 1) & 1, nullptr, 10000000ull);
      }
    }
    // the last block to leave sets the counters back: nobody polls them any more
    __threadfence();
    if (atomicAdd(a.sync + 1, 1u) == (unsigned)P - 1) {
      a.sync[0] = a.sync[1] = a.sync[2] = 0;
      __threadfence();
    }
  }
}

// ---- host ----------------------------------------------------------------------------------------
static int stack_map(CUtensorMap* map, const void* base, int dims, const cuuint64_t* size, const cuuint64_t* pitch,
                     const cuuint32_t* box) {
  EncodeTiledFn fn = tc_encode_fn();
  if (!fn) return GB_ERR_UNSUPPORTED;
  const cuuint32_t one[5] = {1, 1, 1, 1, 1};
  if (((uintptr_t)base) & 15) return GB_ERR_BAD_ARG;
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, dims, const_cast<void*>(base), size, pitch, box, one,
                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                        CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : GB_ERR_BAD_ARG;
}
// [rows, K] in boxes of `box_rows` rows x kb blocks of 64 columns
static int stack_map_wide(CUtensorMap* map, const void* base, int rows, int K, int box_rows, int kb) {
  const cuuint64_t size[3] = {64, (cuuint64_t)rows, (cuuint64_t)K / 64};
  const cuuint64_t pitch[2] = {(cuuint64_t)K * 2, 128};
  const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, (cuuint32_t)kb};
  return stack_map(map, base, 3, size, pitch, box);
}

struct StackPlan {
  int slot_bytes, n_slots, act_at, kb_qkv, kb_o[2];    // kb_o: of o and down with up to DS_FEW rows, with more
};
// The ring's shape for a model on P blocks and T rows, or why there is none.
static int stack_plan(int hidden, int ff, int nq, int nkv, int P, int T, StackPlan* plan) {
  const int N = (nq + 2 * nkv) * 128, groups = ff / 8;
  if (hidden <= 0 || ff <= 0 || nq <= 0 || nkv <= 0 || P <= 0) return GB_ERR_BAD_ARG;
  if (hidden % 64 || ff % 64 || nq % nkv || nq / nkv > 8 || N > (1 << 20) || ff > (1 << 20))
    return GB_ERR_UNSUPPORTED;
  const int c_most = (hidden + P - 1) / P, q_most = (N + P - 1) / P, h_most = (2 * groups + P - 1) / P;
  const int h_least = 2 * groups / P;
  // every block has a share of everything, and it fits where it is kept
  if (hidden < P || N < P || h_least < 2 || c_most > DS_OWN_MOST || q_most > 256 || P > DS_BLOCKS_MOST) return GB_ERR_UNSUPPORTED;
  if (DS_ROWS * nkv > DS_UNITS_MOST * P) return GB_ERR_UNSUPPORTED;
  const int gu_rows = h_most * 8;
  int at = gu_rows * 128;
  at = (at < 2 * DS_TILE_BYTES ? 2 * DS_TILE_BYTES : at + 1023) / 1024 * 1024;
  // 64-column blocks a stage: as the slot holds, at most `most`, and none where the warps' sums do not fit
  auto blocks = [&](int rows, int most) {
    const int tiles = (rows + 15) / 16, parts = DS_FOURS * (tiles > 3 ? 1 : 2), pitch = (rows + 11) / 16 * 16 + 4;
    if (tiles > 4 * DS_TILES || parts * DS_ROWS * pitch * 4 > DS_RED_BYTES) return 0;
    const int fits = at / (rows * 128);
    if (tiles > 3 && most > 2) most = 2;       // (a warp takes up to four steps of a stage)
    return fits < most ? fits : most;
  };
  plan->act_at = at;
  plan->kb_qkv = blocks(q_most, 4), plan->kb_o[0] = blocks(c_most, 8), plan->kb_o[1] = blocks(c_most, 4);
  // (o and down: two tiles at most, whose twelve partial sums always fit, so eight blocks are four steps a warp)
  static_assert(DS_WARPS * DS_ROWS * 36 * 4 <= DS_RED_BYTES, "");
  if (plan->kb_qkv < 1 || plan->kb_o[1] < 1 || blocks(gu_rows, 1) < 1 || h_most / 2 * 16 > 256) return GB_ERR_UNSUPPORTED;
  const int kb_o = plan->kb_o[T > DS_FEW], kb = kb_o > plan->kb_qkv ? kb_o : plan->kb_qkv;
  plan->slot_bytes = (at + kb * 128 * T + 1023) / 1024 * 1024;
  const int n = (DS_SMEM_MOST - 1024 - DS_RED_BYTES - (int)sizeof(StackShared)) / plan->slot_bytes;
  plan->n_slots = n > DS_SLOTS_MOST ? DS_SLOTS_MOST : n;
  return plan->n_slots < 2 * DS_FOURS ? GB_ERR_UNSUPPORTED : 0;
}

// Bytes of a layer's entry, or 0 when the sizes have no plan.
GB_EXPORT int gb_decode_stack_layer_bytes(int hidden, int ff, int nq, int nkv, int P) {
  StackPlan plan;
  return stack_plan(hidden, ff, nq, nkv, P, DS_ROWS, &plan) ? 0 : (int)sizeof(StackLayer);
}

// Block p's share of the work, for tests on the host: out[0..3] first row and rows of qkv, of o and down; out[4..6] first
// whole group, whole groups and half group of gate|up; out[7..] the plan for T rows: bytes of a slot, slots, where a
// slot's activations begin, 64-column blocks a stage of qkv and of o and down.
GB_EXPORT int gb_decode_stack_share(int hidden, int ff, int nq, int nkv, int P, int T, int p, int* out) {
  StackPlan plan;
  const int e = stack_plan(hidden, ff, nq, nkv, P, T, &plan);
  if (e) return e;
  const int N = (nq + 2 * nkv) * 128;
  const StackShare g = stack_share(ff / 8, p, P);
  out[0] = stack_first_row(N, p, P), out[1] = stack_first_row(N, p + 1, P) - out[0];
  out[2] = stack_first_row(hidden, p, P), out[3] = stack_first_row(hidden, p + 1, P) - out[2];
  out[4] = g.first, out[5] = g.whole, out[6] = g.half;
  out[7] = plan.slot_bytes, out[8] = plan.n_slots, out[9] = plan.act_at;
  out[10] = plan.kb_qkv, out[11] = plan.kb_o[T > DS_FEW];
  return 0;
}
GB_EXPORT int gb_decode_stack_fragment(int k, int t, int T) { return stack_fragment(k, t, T); }

// Writes a layer's entry (its tensor maps) to host memory.
GB_EXPORT int gb_decode_stack_encode(void* entry, int hidden, int ff, int nq, int nkv, int P, const void* w_qkv,
                                     const void* w_o, const void* w_gate_up, const void* w_down, void* k_pages,
                                     void* v_pages, long long n_pages) {
  StackPlan plan;
  int e = stack_plan(hidden, ff, nq, nkv, P, DS_ROWS, &plan);
  if (e) return e;
  if (!entry || ((uintptr_t)entry & 63) || !w_qkv || !w_o || !w_gate_up || !w_down || !k_pages || !v_pages || n_pages <= 0)
    return GB_ERR_BAD_ARG;
  if ((unsigned long long)n_pages * nkv * 64 > 0x7fffffffull) return GB_ERR_UNSUPPORTED;
  StackLayer* L = (StackLayer*)entry;
  const int N = (nq + 2 * nkv) * 128, base = 2 * (ff / 8) / P;
  for (int i = 0; i < 2; ++i) {
    if ((e = stack_map_wide(&L->qkv[i], w_qkv, N, hidden, N / P + i, plan.kb_qkv))) return e;
    for (int j = 0; j < 2; ++j) {
      if ((e = stack_map_wide(&L->o[j][i], w_o, hidden, nq * 128, hidden / P + i, plan.kb_o[j]))) return e;
      if ((e = stack_map_wide(&L->down[j][i], w_down, hidden, ff, hidden / P + i, plan.kb_o[j]))) return e;
    }
    // (whole groups of a share: base / 2, or one more)
    const int whole = base / 2 + i;
    if ((e = tc_make_map_2d(&L->gate_up[i], w_gate_up, 2 * (uint64_t)ff, hidden, (uint64_t)hidden * 2,
                            whole * 16 > 256 ? 256 : whole * 16, 64)))
      return e;
  }
  const cuuint64_t size[4] = {(cuuint64_t)hidden, 8, 2, (cuuint64_t)ff / 8};
  const cuuint64_t pitch[3] = {(cuuint64_t)hidden * 2, (cuuint64_t)hidden * 16, (cuuint64_t)hidden * 32};
  const cuuint32_t box[4] = {64, 4, 2, 1};
  if ((e = stack_map(&L->half, w_gate_up, 4, size, pitch, box))) return e;
  const uint64_t rows = (uint64_t)n_pages * nkv * 64;
  if ((e = tc_make_map_2d(&L->k, k_pages, rows, 128, 256, 64, 64))) return e;
  if ((e = tc_make_map_2d(&L->v, v_pages, rows, 128, 256, 64, 64))) return e;
  return 0;
}

// One launch: args' plan fields are filled in here.
GB_EXPORT int gb_decode_stack(StackArgs* a, int P, cudaStream_t s) {
  StackPlan plan;
  if (a->T < 1 || a->T > DS_ROWS) return GB_ERR_BAD_ARG;
  int e = stack_plan(a->hidden, a->ff, a->nq, a->nkv, P, a->T, &plan);
  if (e) return e;
  if (a->n_layers < 1 || a->max_pages <= 0 || !a->layers || !a->rows || ((uintptr_t)a->rows & 15) || !a->x_out || (!a->x_in && !a->res_in) || !a->slots ||
      !a->kv_len || !a->block_table || !a->xb || !a->ab || !a->hb || !a->ss || !a->qkv || !a->part_o || !a->part_ml ||
      !a->sync || !a->error)
    return GB_ERR_BAD_ARG;
  if (!a->wait_ns) a->wait_ns = TC_WAIT_LIMIT_NS;
  a->slot_bytes = plan.slot_bytes, a->n_slots = plan.n_slots;
  a->act_at = plan.act_at, a->kb_qkv = plan.kb_qkv, a->kb_o = a->kb_down = plan.kb_o[a->T > DS_FEW];
  const size_t smem = 1024 + (size_t)plan.n_slots * plan.slot_bytes + DS_RED_BYTES + sizeof(StackShared);
  // (each launch, which is once a capture: the attribute is a device's)
  const cudaError_t set = cudaFuncSetAttribute(decode_stack_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, DS_SMEM_MOST);
  if (set != cudaSuccess) return (int)set;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(P);
  cfg.blockDim = dim3(DS_THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t r = cudaLaunchKernelEx(&cfg, decode_stack_kernel, *a);
  if (r != cudaSuccess) return (int)r;
  return (int)cudaGetLastError();
}
