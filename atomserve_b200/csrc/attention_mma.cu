// Paged grouped-query attention for bfloat16 on the tensor cores (mma.sync m16n8k16, float32
// accumulation), head sizes 64 and 128. Two kernels share one tile machinery:
//
//   decode   the token's G query heads are the rows of a 16-row tile, so keys and values are read
//            once for all of them. The block's four warps take the keys of each 64-key tile sixteen
//            apiece, keep their own running softmax, and merge at the end. The tiles of all rows are
//            one sequence, cut into equal ranges, a block per range and kv head; what a range cuts is
//            written as (max, sum, accumulator) and merged by a second kernel.
//            Serves every request that brings at most kShortRows tokens in the step; each of
//            those tokens is its own row with its own context length.
//   prefill  one block per (request, tile of query tokens, kv head): 128 rows = (token, head)
//            pairs, sixteen per warp, all key tiles up to the tile's last position, causal and
//            window masks from absolute positions. Serves the longer portions.
//
// Keys and values come straight from the cache pages through the block table with 16-byte
// cp.async copies into shared memory (two stages), swizzled so that ldmatrix reads are free of
// bank conflicts. Scores, maxima, sums and the output accumulator are float32; probabilities are
// rounded to bfloat16 only as the tensor-core operand of the second product, the output once
// (atomserve/kernels.py:147-334 is the reference's scalar decode kernel; its prefill is a
// library call, atomserve/model.py:225-231).
//
// Key tiles start at absolute multiples of 64; how a row's tiles are grouped into sums may depend on
// the rest of the batch (the decode kernel's ranges), which keys it sees does not.
#include "attention_mma.cuh"
#include "gemm_partials.cuh"

namespace {

using namespace asb::mma;

constexpr int kThreads = 128;
constexpr int kKeyTile = 64;
constexpr int kShortRows = 8;  // requests with at most this many new tokens go row by row

struct MmaParams {
  const __nv_bfloat16* q;    // [T, H, HD]
  __nv_bfloat16* out;        // [T, H, HD]
  const __nv_bfloat16* k_cache;  // [num_blocks, KV, bs, HD]
  const __nv_bfloat16* v_cache;
  const int* block_tables;   // [R, table_width]
  const int* req_q_start;    // [R + 1]
  const int* req_pos_start;  // [R]
  const float* sink;         // [H] or null: a logit per head that joins the softmax's denominator once
  int T, R, H, KV, bs, table_width;
  int G, GC, HC;             // heads per kv head, heads per block (<= 16), chunks per kv head
  int QT;                    // tokens per 128-row tile
  int window;
  int chunk;                 // 0: none; else a query sees only the keys of its own run of `chunk` positions
  float softcap;             // 0: none; else score <- softcap tanh(score / softcap)
  float scale;
};

// cap * tanh(x / cap) through one exponential: tanh(y) = 1 - 2 / (exp(2y) + 1); exact limits at both ends
__device__ __forceinline__ float capped(float x, float cap) {
  return cap * (1.f - __fdividef(2.f, __expf(2.f * x / cap) + 1.f));
}

// Copy keys [kt0, kt0 + 64) of one kv head into a tile; rows outside [key_lo, key_hi) are zero.
// A thread copies one 16-byte chunk column of a run of consecutive keys, so that when a run lies
// inside one page (pages of at least that many tokens, a power of two) it looks the page up once.
template <int HD, int NT>
__device__ __forceinline__ void load_kv_tile(uint32_t k_tile, uint32_t v_tile, const MmaParams& p,
                                             const int* table, int kvh, int kt0, int key_lo, int key_hi) {
  constexpr int kChunks = HD / 8;                        // 16-byte chunks per row
  constexpr int kRun = kKeyTile / (NT / kChunks);        // consecutive keys per thread
  const int chunk = threadIdx.x % kChunks;
  const int run0 = (threadIdx.x / kChunks) * kRun;
  const int j0 = kt0 + run0;
  const bool one_page = p.bs >= kRun && (p.bs & (p.bs - 1)) == 0;
  size_t page_at = 0;
  if (one_page && j0 < key_hi && j0 + kRun > key_lo) {
    const int blk = table[j0 / p.bs];
    page_at = (((size_t)blk * p.KV + kvh) * p.bs + (j0 & (p.bs - 1))) * HD + chunk * 8;
  }
#pragma unroll
  for (int i = 0; i < kRun; ++i) {
    const int j = j0 + i;
    const bool valid = j >= key_lo && j < key_hi;
    size_t at = 0;
    if (valid) {
      if (one_page) {
        at = page_at + (size_t)i * HD;
      } else {
        const int blk = table[j / p.bs];
        at = (((size_t)blk * p.KV + kvh) * p.bs + (j % p.bs)) * HD + chunk * 8;
      }
    }
    const uint32_t off = tile_offset<HD>(run0 + i, chunk);
    cp_async16(k_tile + off, p.k_cache + at, valid);
    cp_async16(v_tile + off, p.v_cache + at, valid);
  }
}

// One warp: scores of its 16 rows against all 64 keys of a tile. The eight accumulators advance together along the head
// dimension, so eight independent MMA chains are in flight. Q fragments are read from shared memory as they are needed, which frees the
// HD/4 registers that holding them costs (the prefill kernel runs two blocks per SM that way).
template <int HD>
__device__ __forceinline__ void qk_64keys_smem_q(float (&s)[kKeyTile / 8][4], uint32_t q_tile, int q_row0,
                                                 uint32_t k_tile, int lane, float scale) {
#pragma unroll
  for (int j = 0; j < kKeyTile / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
  const int krow = (lane & 7) + ((lane >> 4) << 3);
  const int kchunk = (lane >> 3) & 1;
  const int qrow = q_row0 + (lane & 7) + (((lane >> 3) & 1) << 3);
  const int qchunk = lane >> 4;
#pragma unroll
  for (int kc = 0; kc < HD / 16; ++kc) {
    uint32_t a[4];
    ldmatrix_x4(a, q_tile + tile_offset<HD>(qrow, kc * 2 + qchunk));
#pragma unroll
    for (int sub = 0; sub < kKeyTile / 16; ++sub) {
      uint32_t b[4];
      ldmatrix_x4(b, k_tile + tile_offset<HD>(sub * 16 + krow, kc * 2 + kchunk));
      mma_bf16(s[sub * 2], a, b[0], b[1]);
      mma_bf16(s[sub * 2 + 1], a, b[2], b[3]);
    }
  }
#pragma unroll
  for (int j = 0; j < kKeyTile / 8; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[j][e] *= scale;
}

template <int HD>
__device__ __forceinline__ void qk_16keys_smem_q(float (&s)[2][4], uint32_t q_tile, int q_row0, uint32_t k_tile,
                                                 int key0, int lane, float scale) {
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[j][e] = 0.f;
  const int krow = key0 + (lane & 7) + ((lane >> 4) << 3);
  const int kchunk = (lane >> 3) & 1;
  const int qrow = q_row0 + (lane & 7) + (((lane >> 3) & 1) << 3);
  const int qchunk = lane >> 4;
#pragma unroll
  for (int kc = 0; kc < HD / 16; ++kc) {
    uint32_t a[4], b[4];
    ldmatrix_x4(a, q_tile + tile_offset<HD>(qrow, kc * 2 + qchunk));
    ldmatrix_x4(b, k_tile + tile_offset<HD>(krow, kc * 2 + kchunk));
    mma_bf16(s[0], a, b[0], b[1]);
    mma_bf16(s[1], a, b[2], b[3]);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) s[j][e] *= scale;
}

// ---- decode ------------------------------------------------------------------------------------

constexpr int kDecodeStages = 2;
constexpr float kLog2e = 1.4426950408889634f;

// What the decode kernel and its merge share: the shape, the per-step index arrays, and how the keys are dealt out.
// The rows' 64-key tiles make one sequence, cut into `ranges` equal ranges; a block has one range and one lane, a kv
// head (or 16 of its heads). Blocks of the same range and different lanes are neighbours: they read the same pages at
// about the same time, and a page's kv heads lie side by side in memory.
struct DecodeParams {
  const __nv_bfloat16* q;    // [T, H, HD]
  __nv_bfloat16* out;        // [T, H, HD]
  const __nv_bfloat16* k_cache;  // [num_blocks, KV, bs, HD]
  const __nv_bfloat16* v_cache;
  const int* block_tables;   // [R, table_width]
  const int* req_q_start;    // [R + 1]
  const int* req_pos_start;  // [R]
  int4* cuts;                // [rows]: the first and the last range that hold a share of the row, and its flat row
  float* part_acc;           // [2 * ranges * lanes, GC, HD]: a block's first row, if it began in another range, and its
  float* part_ml;            // [2 * ranges * lanes, GC, 2]   last, if it ends in another one; (max, sum)
  const float* sink;         // [H] or null: a logit per head that joins the softmax's denominator once
  int rows, R, H, KV, bs, table_width;
  int G, GC, HC;             // heads per kv head, heads per block (<= 16), chunks per kv head
  int lanes;                 // KV * HC
  int window;
  int chunk;                 // 0: none; else a query sees only the keys of its own run of `chunk` positions
  float softcap;             // 0: none; else score <- softcap tanh(score / softcap)
  int all_single;            // every request brings exactly one token: request = row
  int short_rows;            // > 0: rows count only those of requests with at most kShortRows tokens
  int early;                 // 1: the index arrays, and the keys below a request's first new position, were written before the
                             // stream's previous kernel was launched; else nothing is read before the wait for it
  int ranges;                // 0: a range is a row, whatever its length
  float scale;
};

// One row of the launch. The index arrays may be read before the wait for the previous kernel (`early`), and so from
// L2: an SM's L1 could still hold their lines from an earlier step.
struct DecodeRow {
  int row, r, pos, fresh;    // flat row, request, position, first position that this step writes
  int lo, tile0, tiles;      // first visible key, its tile, tiles to walk (0: not a row of this kernel)
};

// Flat row `row`, of request r whose rows begin at q_start.
__device__ __forceinline__ DecodeRow make_row(const DecodeParams& p, int row, int r, int q_start) {
  DecodeRow d;
  d.row = row;
  d.r = r;
  d.fresh = __ldcg(p.req_pos_start + r);
  d.pos = d.fresh + (row - q_start);
  d.lo = p.window > 0 ? max(0, d.pos - p.window + 1) : 0;
  if (p.chunk > 0) d.lo = max(d.lo, d.pos - d.pos % p.chunk);
  d.tile0 = d.lo / kKeyTile;
  d.tiles = d.pos / kKeyTile - d.tile0 + 1;
  return d;
}

__device__ __forceinline__ DecodeRow no_row() {
  DecodeRow d;
  d.row = -1;
  d.r = d.pos = d.fresh = d.lo = d.tile0 = d.tiles = 0;
  return d;
}

// req_q_start as the searches below read it: a copy in shared memory where it fits (they read many entries, one after
// the other), and never through an SM's L1. Not needed where every request brings one token.
constexpr int kStarts = 512;
typedef const volatile int* Starts;
__device__ __forceinline__ Starts copy_starts(const DecodeParams& p, int* to) {
  if (p.all_single || p.R >= kStarts) return p.req_q_start;
  for (int r = threadIdx.x; r <= p.R; r += kThreads) to[r] = __ldcg(p.req_q_start + r);
  __syncthreads();
  return to;
}

__device__ __noinline__ DecodeRow decode_row(const DecodeParams& p, Starts starts, int i) {
  if (p.all_single) return make_row(p, i, i, i);
  if (p.short_rows > 0) {  // row number i among the short requests' rows (the lanes of a warp leave the walk together)
    int begin = starts[0], left = i, row = -1, r_of = 0, begin_of = 0;
#pragma unroll 4
    for (int r = 0; r < p.R; ++r) {
      const int end = starts[r + 1], n = end - begin;
      if (n <= kShortRows) {
        if (left >= 0 && left < n) { row = begin + left; r_of = r; begin_of = begin; }
        left -= n;
      }
      begin = end;
    }
    return row >= 0 ? make_row(p, row, r_of, begin_of) : no_row();
  }
  int lo = 0, hi = p.R - 1;  // flat row i, of the last request that begins at or before it
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (starts[mid] <= i) lo = mid; else hi = mid - 1;
  }
  const int begin = starts[lo], end = starts[lo + 1];
  return i < end && end - begin <= kShortRows ? make_row(p, i, lo, begin) : no_row();  // (longer ones: the prefill kernel's)
}

// Row i, the one after `d`: what decode_row gives, without its walk over the requests.
__device__ __forceinline__ DecodeRow row_after(const DecodeParams& p, Starts starts, const DecodeRow& d, int i) {
  if (p.short_rows == 0 || d.row < 0) return decode_row(p, starts, i);
  int r = d.r, begin = starts[r], end = starts[r + 1];
  if (d.row + 1 < end) return make_row(p, d.row + 1, r, begin);
  while (++r < p.R) {
    begin = end;
    end = starts[r + 1];
    if (end > begin && end - begin <= kShortRows) return make_row(p, begin, r, begin);
  }
  return no_row();
}

// Sum over the block (every thread gets it; `scratch`: one word per warp).
__device__ __forceinline__ int block_total(int v, int* scratch) {
  v = __reduce_add_sync(0xffffffffu, v);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = v;
  __syncthreads();
  int s = 0;
#pragma unroll
  for (int w = 0; w < kThreads / 32; ++w) s += scratch[w];
  return s;
}

// Sum of the tiles of the rows below `upto`.
__device__ __forceinline__ int tiles_below(const DecodeParams& p, Starts starts, int upto, int* scratch) {
  int s = 0;
  for (int i = threadIdx.x; i < upto; i += kThreads) s += decode_row(p, starts, i).tiles;
  return block_total(s, scratch);
}

// Ranges that end with their rows: the fewest tiles a range such that every row cut into equal ranges of at most that many
// leaves no more than p.ranges of them, if that is within what the equal ranges of the whole sequence have and kCrossing more;
// else 0 (also with more rows than threads; `mine`: the tiles of row threadIdx.x). A block that walks from one row into
// the next pays for a second merge and a second start, about three tiles' time: three requests of 500 to 1,500 keys, 32 heads
// over 8, 12.5 -> 9.3 us.
constexpr int kCrossing = 3;
__device__ __forceinline__ int tiles_a_range(const DecodeParams& p, int mine, int total, int* scratch) {
  if (p.rows > kThreads) return 0;
  const int least = (total + p.ranges - 1) / p.ranges;
  for (int c = least; c < least + kCrossing; ++c)
    if (c > 0 && block_total((mine + c - 1) / c, scratch) <= p.ranges) return c;
  return 0;
}

// A place in the sequence of tiles.
struct DecodeCursor {
  int i, t;                  // row of the launch, tile of the row
  DecodeRow d;
  __device__ __forceinline__ void next(const DecodeParams& p, Starts starts) {
    if (++t < d.tiles) return;
    t = 0;
    do { ++i; d = row_after(p, starts, d, i); } while (d.tiles == 0 && i + 1 < p.rows);
  }
};

// What bounds it: the keys' and values' bytes with many or long rows, the chain of one warp's instructions per tile
// with few (about 0.95 us a tile, from 1.4: whole tiles copied and scored without masks, and with up to 8 heads a kv head
// the heads as the 8 columns of the products instead of half of 16 rows). Three blocks share an SM, two stages of
// 64 keys each, which run on across rows. Each warp copies the keys that it reads, so the block meets only at a row's
// end. The sequence of tiles is cut into equal ranges because rows of one step have contexts of all lengths: with a grid of
// (row, kv head, partition of the longest context) a block had up to twice the mean of work and many had none. A
// first tile of keys that earlier steps wrote is asked for before the wait. Measured with the merge, before and after: 64
// requests of 300 to 3,000 keys, 32 heads over 8: 87.5 -> 78.2 us (5.5 TB/s); 13 of 6,000 to 12,000, 64 over 8: 114.8 ->
// 89.1 us; 8 of 2,048: 19.2 -> 17.9; one of 2,048: 12.3 -> 8.5 us. (Three stages and two blocks an SM: 88.7, 96.8,
// 21.9, 9.4 on an earlier form; neighbouring blocks on neighbouring ranges of one kv head instead: 144 us for the second.)
template <int HD, bool Half>
__global__ void __launch_bounds__(kThreads, 3)
decode_attention_kernel(const __grid_constant__ DecodeParams p) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr int kTileBytes = kKeyTile * HD * 2;
  constexpr int kChunks = HD / 8;
  __shared__ int scan[kThreads / 32], found[3], starts_at[kStarts];
  __shared__ float mm[4 * 16], ml[4 * 16];
  // [K stage 0][V stage 0][K stage 1][V stage 1][Q of two rows, 8 or 16 heads]; a merge uses the K and V of a tile
  // that has been read
  const uint32_t smem = (smem_u32(smem_raw) + 255u) & ~255u;  // rows of the tiles begin where the swizzle's bits are zero
  unsigned char* const smem_at = smem_raw + (smem - smem_u32(smem_raw));
  auto k_stage = [&](int stage) { return smem + (uint32_t)(2 * stage) * kTileBytes; };
  auto v_stage = [&](int stage) { return smem + (uint32_t)(2 * stage + 1) * kTileBytes; };
  constexpr int q_rows = Half ? 8 : 16;
  auto q_tile = [&](int i) { return smem + 2 * kDecodeStages * kTileBytes + (uint32_t)(i % kDecodeStages) * q_rows * HD * 2; };

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int range = blockIdx.x / p.lanes, head_lane = blockIdx.x - range * p.lanes;
  const int kvh = head_lane / p.HC, head0 = kvh * p.G + (head_lane - kvh * p.HC) * p.GC;
  const int gc = min(p.GC, kvh * p.G + p.G - head0);
  if (!p.early) asb::pdl_wait();
  const Starts starts = copy_starts(p, starts_at);
  DecodeCursor at;           // the tile being computed
  int n;                     // tiles of this block
  // A block without work waits for the previous kernel before it leaves: a launch whose blocks all left without
  // waiting would be over before that kernel, and whatever waits for this launch would not have waited for that one.
  if (p.ranges > 0) {
    // A scan over a value per row, as many rows at a time as there are threads: this thread's row holds [from, to).
    int from, to, above = 0;
    auto scan_rows = [&](int mine) {
      int upto = mine;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, upto, o);
        if (lane >= o) upto += u;
      }
      __syncthreads();
      if (lane == 31) scan[warp] = upto;
      if (threadIdx.x == 0) found[0] = -1;
      __syncthreads();
      int round = 0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) {
        if (w < warp) upto += scan[w];
        round += scan[w];
      }
      to = above + upto;
      from = to - mine;
      above += round;
    };
    int mine = (int)threadIdx.x < p.rows ? decode_row(p, starts, threadIdx.x).tiles : 0;
    const int total = p.rows <= kThreads ? block_total(mine, scan) : tiles_below(p, starts, p.rows, scan);
    const int per = tiles_a_range(p, mine, total, scan);
    if (per > 0) {           // ranges that end with their rows
      const int cuts = (mine + per - 1) / per;
      scan_rows(cuts);
      if (range >= above) {    // (uniform; with no rows of this kernel's in the step, every block comes here)
        asb::pdl_wait();
        return;
      }
      if (range >= from && range < to) {
        const int k = range - from;
        found[0] = threadIdx.x;
        found[1] = mine * k / cuts;
        found[2] = mine * (k + 1) / cuts - found[1];
      }
      __syncthreads();
      n = found[2];
    } else {
      const int ranges = min(p.ranges, total);
      if (range >= ranges) {
        asb::pdl_wait();
        return;
      }
      const int begin = (int)asb::range_begin(total, ranges, range);
      n = (int)asb::range_begin(total, ranges, range + 1) - begin;
      for (int i0 = 0;;) {   // the row that tile `begin` belongs to
        scan_rows(mine);
        if (begin >= from && begin < to) { found[0] = i0 + threadIdx.x; found[1] = begin - from; }
        __syncthreads();
        if (found[0] >= 0) break;
        i0 += kThreads;
        mine = i0 + (int)threadIdx.x < p.rows ? decode_row(p, starts, i0 + threadIdx.x).tiles : 0;
      }
    }
    at.i = found[0];
    at.t = found[1];
    at.d = decode_row(p, starts, at.i);
  } else {
    at.i = range;
    at.t = 0;
    at.d = decode_row(p, starts, at.i);
    n = at.d.tiles;
    if (n == 0) {
      asb::pdl_wait();
      return;
    }
  }

  // A thread copies one 16-byte column of kRun consecutive keys. Where these lie in one page (pages of at least that
  // many tokens, a power of two), its number is looked up a tile before the copies need it.
  constexpr int kRun = kKeyTile / (kThreads / kChunks);
  const int column = threadIdx.x % kChunks, run0 = (threadIdx.x / kChunks) * kRun;
  const bool one_page = p.bs >= kRun && (p.bs & (p.bs - 1)) == 0;
  const int page_shift = 31 - __clz(p.bs);
  auto look_up = [&](const DecodeCursor& u) {
    const int j = (u.d.tile0 + u.t) * kKeyTile + run0;
    return one_page && j <= u.d.pos && j + kRun > u.d.lo ? __ldcg(p.block_tables + (size_t)u.d.r * p.table_width + (j >> page_shift)) : 0;
  };
  uint32_t put[kRun];        // where the run's 16-byte columns go in a tile
#pragma unroll
  for (int i = 0; i < kRun; ++i) put[i] = tile_offset<HD>(run0 + i, column);
  auto load_tile = [&](const DecodeCursor& u, int page, int stage) {
    const int kt0 = (u.d.tile0 + u.t) * kKeyTile, j0 = kt0 + run0;
    const size_t page_at = (((size_t)page * p.KV + kvh) * p.bs + (j0 & (p.bs - 1))) * HD + column * 8;
    if (one_page && kt0 >= u.d.lo && kt0 + kKeyTile <= u.d.pos + 1) {  // a whole tile
      const __nv_bfloat16 *k_from = p.k_cache + page_at, *v_from = p.v_cache + page_at;
#pragma unroll
      for (int i = 0; i < kRun; ++i) {
        cp_async16(k_stage(stage) + put[i], k_from + i * HD);
        cp_async16(v_stage(stage) + put[i], v_from + i * HD);
      }
      return;
    }
#pragma unroll 1
    for (int i = 0; i < kRun; ++i) {
      const int j = j0 + i;
      const bool valid = j >= u.d.lo && j <= u.d.pos;
      size_t from = 0;
      if (valid) {
        if (one_page) from = page_at + (size_t)i * HD;
        else from = (((size_t)__ldcg(p.block_tables + (size_t)u.d.r * p.table_width + j / p.bs) * p.KV + kvh) * p.bs + j % p.bs) * HD + column * 8;
      }
      const uint32_t to = tile_offset<HD>(run0 + i, column);
      cp_async16(k_stage(stage) + to, p.k_cache + from, valid);
      cp_async16(v_stage(stage) + to, p.v_cache + from, valid);
    }
  };
  // Every warp brings all of the queries (the same bytes to the same place), so that it waits for its own copies only.
  // Rows beyond the chunk's heads are zero.
  auto load_q = [&](const DecodeCursor& u, int index) {
    const __nv_bfloat16* src = p.q + ((size_t)u.d.row * p.H + head0) * HD;
    for (int i = lane; i < q_rows * kChunks; i += 32) {
      const bool valid = i < gc * kChunks;
      cp_async16(q_tile(index) + tile_offset<HD>(i / kChunks, i % kChunks), src + (valid ? (size_t)i * 8 : 0), valid);
    }
  };

  DecodeCursor next = at;    // the loads run kDecodeStages - 1 tiles ahead
  const bool early = p.early && (at.d.tile0 + at.t + 1) * kKeyTile <= at.d.fresh;
  int page = look_up(next);
  if (early) load_tile(next, page, 0);
  asb::pdl_wait();  // the stream's previous kernel has completed (programmatic dependent launch)
  asb::pdl_launch_dependents();
  if (!early) load_tile(next, page, 0);
  int next_row = 0, row = 0;  // rows met so far by the loads, by the arithmetic
  load_q(next, next_row);
  cp_async_commit();
  int loaded = 1;            // tiles whose copies have been issued
  auto look_ahead = [&]() {
    if (loaded < n) {
      next.next(p, starts);
      page = look_up(next);
    }
  };
  auto load_next = [&](int stage) {
    if (loaded < n) {
      load_tile(next, page, stage);
      if (next.t == 0) load_q(next, ++next_row);
      ++loaded;
      look_ahead();
    }
    cp_async_commit();
  };
  look_ahead();
#pragma unroll
  for (int i = 1; i < kDecodeStages - 1; ++i) load_next(i);
  int stage = 0;

  // With up to 8 heads (Half) the keys are the 16 rows of the products and the heads their 8 columns: scores^T = K . Q^T,
  // out^T = V^T . P^T; a thread then has heads 2 (lane % 4) and one more in both. With more, the heads are the rows:
  // a thread has heads lane / 4 and 8 more. m (in units of log2(e)) and l (this thread's share of the sum) are theirs.
  constexpr int kOut = Half ? HD / 16 : HD / 8;
  uint32_t qf[HD / 16][Half ? 2 : 4];
  float m[2], l[2], acc[kOut][4];
  bool fresh_row = true;
  int first_t = at.t;        // the row's tile that this block began with
  const float scale = p.scale * kLog2e, cap = p.softcap * kLog2e;
  const int key0 = warp * 16;  // this warp's keys inside a tile
  // where this lane's ldmatrix rows begin in a tile; 16 columns further is an exclusive or (tile_offset's swizzle)
  const uint32_t rows_first = tile_offset<HD>(key0 + (lane & 15), lane >> 4);
  const uint32_t columns_first = tile_offset<HD>(key0 + (lane & 7) + ((lane >> 4) << 3), (lane >> 3) & 1);
  const uint32_t k_off = Half ? rows_first : columns_first, v_off = Half ? columns_first : rows_first;

  for (int it = 0; it < n; ++it) {
    load_next(stage == 0 ? kDecodeStages - 1 : stage - 1);
    cp_async_wait<kDecodeStages - 1>();
    __syncwarp();  // a warp reads the keys that it copied: there is no barrier of the block but at a row's end

    if (fresh_row) {
#pragma unroll
      for (int kc = 0; kc < HD / 16; kc += Half ? 2 : 1) {
        uint32_t f[4];
        if constexpr (Half) {
          ldmatrix_x4(f, q_tile(row) + tile_offset<HD>(lane & 7, kc * 2 + (lane >> 3)));
          qf[kc][0] = f[0]; qf[kc][1] = f[1];
          qf[kc + 1][0] = f[2]; qf[kc + 1][1] = f[3];
        } else {
          ldmatrix_x4(f, q_tile(row) + tile_offset<HD>(lane & 15, kc * 2 + (lane >> 4)));
#pragma unroll
          for (int k = 0; k < 4; ++k) qf[kc][k] = f[k];
        }
      }
#pragma unroll
      for (int i = 0; i < kOut; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
      m[0] = m[1] = -INFINITY;
      l[0] = l[1] = 0.f;
      first_t = at.t;
      fresh_row = false;
    }
    const int kt0 = (at.d.tile0 + at.t) * kKeyTile;
    if (kt0 + key0 <= at.d.pos && kt0 + key0 + 16 > at.d.lo) {
      // Scores in fragments of 4: element e of fragment j is head e % 2 (Half) or e / 2 of the thread, and key
      // `key_of(j, e)` of the warp's 16. Two chains of products a fragment.
      constexpr int kFrags = Half ? 1 : 2;
      auto key_of = [&](int j, int e) { return Half ? (lane >> 2) + (e >> 1) * 8 : j * 8 + (lane & 3) * 2 + (e & 1); };
      auto head_of = [](int e) { return Half ? e & 1 : e >> 1; };
      float s[kFrags][4], s_odd[kFrags][4];
#pragma unroll
      for (int j = 0; j < kFrags; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[j][e] = s_odd[j][e] = 0.f;
      const uint32_t k_at = k_stage(stage) + k_off;
#pragma unroll
      for (int kc = 0; kc < HD / 16; ++kc) {
        uint32_t b[4];
        ldmatrix_x4(b, k_at ^ (uint32_t)(kc << 5));
        if constexpr (Half) {
          mma_bf16(kc & 1 ? s_odd[0] : s[0], b, qf[kc][0], qf[kc][1]);
        } else {
          mma_bf16(kc & 1 ? s_odd[0] : s[0], qf[kc], b[0], b[1]);
          mma_bf16(kc & 1 ? s_odd[1] : s[1], qf[kc], b[2], b[3]);
        }
      }
#pragma unroll
      for (int j = 0; j < kFrags; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) s[j][e] = (s[j][e] + s_odd[j][e]) * scale;
      if (cap > 0.f) {
#pragma unroll
        for (int j = 0; j < kFrags; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[j][e] = capped(s[j][e], cap);
      }
      if (kt0 + key0 < at.d.lo || kt0 + key0 + 15 > at.d.pos) {
        // mask by absolute key position; all heads share the token, hence the mask
#pragma unroll
        for (int j = 0; j < kFrags; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int key = kt0 + key0 + key_of(j, e);
            if (key < at.d.lo || key > at.d.pos) s[j][e] = -INFINITY;
          }
      }
      float top[2] = {-INFINITY, -INFINITY}, corr[2];
#pragma unroll
      for (int j = 0; j < kFrags; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) top[head_of(e)] = fmaxf(top[head_of(e)], s[j][e]);
#pragma unroll
      for (int o = Half ? 4 : 1; o <= (Half ? 16 : 2); o <<= 1) {
        top[0] = fmaxf(top[0], __shfl_xor_sync(0xffffffffu, top[0], o));
        top[1] = fmaxf(top[1], __shfl_xor_sync(0xffffffffu, top[1], o));
      }
      bool grown = false;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const float m_new = fmaxf(m[h], top[h]);  // finite: at least one key of the 16 is visible
        corr[h] = fast_exp2(m[h] - m_new);
        grown |= m_new != m[h];
        m[h] = m_new;
      }
      if (__any_sync(0xffffffffu, grown)) {
        l[0] *= corr[0];
        l[1] *= corr[1];
#pragma unroll
        for (int i = 0; i < kOut; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][e] *= corr[head_of(e)];
      }
#pragma unroll
      for (int j = 0; j < kFrags; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          s[j][e] = fast_exp2(s[j][e] - m[head_of(e)]);
          l[head_of(e)] += s[j][e];
        }
      const uint32_t v_at = v_stage(stage) + v_off;
      if constexpr (Half) {
        // (key, two heads) a thread -> (head, two keys): the column operand of the second product
        const uint32_t p0 = transposed(pack_bf16(s[0][0], s[0][1])), p1 = transposed(pack_bf16(s[0][2], s[0][3]));
#pragma unroll
        for (int nc = 0; nc < HD / 16; ++nc) {
          uint32_t b[4];
          ldmatrix_x4_trans(b, v_at ^ (uint32_t)(nc << 5));
          mma_bf16(acc[nc], b, p0, p1);
        }
      } else {
        const uint32_t pf[4] = {pack_bf16(s[0][0], s[0][1]), pack_bf16(s[0][2], s[0][3]),
                                pack_bf16(s[kFrags - 1][0], s[kFrags - 1][1]), pack_bf16(s[kFrags - 1][2], s[kFrags - 1][3])};
#pragma unroll
        for (int nc = 0; nc < HD / 16; ++nc) {
          uint32_t b[4];
          ldmatrix_x4_trans(b, v_at ^ (uint32_t)(nc << 5));
          mma_bf16(acc[(nc * 2) % kOut], pf, b[0], b[1]);
          mma_bf16(acc[(nc * 2 + 1) % kOut], pf, b[2], b[3]);
        }
      }
    }
    __syncwarp();  // the warp's keys of the stage have been read
    if (at.t + 1 == at.d.tiles || it + 1 == n) {
      __syncthreads();
      // The row, or this block's share of it, is complete: merge the four warps through the stage just read.
      float* ma = reinterpret_cast<float*>(smem_at + (k_stage(stage) - smem));  // [4][gc][HD], at most a K and a V tile
      {
        const int g = lane >> 2, t = lane & 3;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
#pragma unroll
          for (int o = Half ? 4 : 1; o <= (Half ? 16 : 2); o <<= 1) l[h] += __shfl_xor_sync(0xffffffffu, l[h], o);
          const int head = Half ? 2 * t + h : g + 8 * h;
          if (Half ? g == 0 : t == 0) {
            mm[warp * 16 + head] = m[h];
            ml[warp * 16 + head] = l[h];
          }
          if (head >= gc) continue;
          float* to = ma + (size_t)(warp * gc + head) * HD;
#pragma unroll
          for (int i = 0; i < kOut; ++i) {
            if constexpr (Half) {
              to[i * 16 + g] = acc[i][h];
              to[i * 16 + g + 8] = acc[i][2 + h];
            } else {
              *reinterpret_cast<float2*>(to + i * 8 + t * 2) = make_float2(acc[i][2 * h], acc[i][2 * h + 1]);
            }
          }
        }
      }
      __syncthreads();
      const bool whole = first_t == 0 && at.t + 1 == at.d.tiles;
      const size_t slot = 2 * (size_t)blockIdx.x + (first_t == 0 ? 1 : 0);
      if (p.ranges > 0 && !p.all_single && head_lane == 0 && threadIdx.x == 0) {
        if (first_t == 0) { p.cuts[at.i].x = range; p.cuts[at.i].z = at.d.row; }
        if (at.t + 1 == at.d.tiles) p.cuts[at.i].y = range;
      }
      for (int i = threadIdx.x; i < gc * HD; i += kThreads) {
        const int qr = i / HD, col = i - qr * HD;
        float mx = -INFINITY;
#pragma unroll
        for (int w = 0; w < 4; ++w)
          if (ml[w * 16 + qr] != 0.f) mx = fmaxf(mx, mm[w * 16 + qr]);  // (zero: the warp saw no key; a sum that is NaN counts)
        float a = 0.f, den = 0.f;
#pragma unroll
        for (int w = 0; w < 4; ++w)
          if (ml[w * 16 + qr] != 0.f) {
            const float f = fast_exp2(mm[w * 16 + qr] - mx);
            den += ml[w * 16 + qr] * f;
            a += ma[(size_t)(w * gc + qr) * HD + col] * f;
          }
        if (p.sink && first_t == 0) {  // the sink counts once per row: with its first tile
          const float sk = p.sink[head0 + qr] * kLog2e;
          if (den != 0.f) {
            den += exp2f(sk - mx);  // (the sums stay relative to mx: nothing is rescaled)
          } else {
            mx = sk;
            den = 1.f;
            a = 0.f;
          }
        }
        if (whole) {
          p.out[((size_t)at.d.row * p.H + head0 + qr) * HD + col] = __float2bfloat16_rn(a / den);
        } else {
          p.part_acc[(slot * p.GC + qr) * HD + col] = a;
          if (col == 0) *reinterpret_cast<float2*>(p.part_ml + (slot * p.GC + qr) * 2) = make_float2(mx, den);
        }
      }
      __syncthreads();  // the next loads may fill the stage
      ++row;
      fresh_row = true;
    }
    if (it + 1 < n) at.next(p, starts);
    if (++stage == kDecodeStages) stage = 0;
  }
  cp_async_wait<0>();
}

// Merges the rows that the ranges of the decode kernel cut: a block per (row, head). Which ranges hold a share of a row
// follows from the rows' tiles: where a row's tiles are at hand (every request brings one token) that is worked out before
// the wait, from index arrays that are there: the decode kernel lets this one start after its own wait (or `early` says so) (one request of 12,000 keys: 19.5 -> 17.5 us with the decode kernel), elsewhere the decode kernel says it.
template <int HD>
__global__ void __launch_bounds__(kThreads)
decode_merge_kernel(const __grid_constant__ DecodeParams p) {
  constexpr int kWarps = kThreads / 32, V = HD / 32;  // columns per lane
  __shared__ int scan[kWarps];
  __shared__ float2 warp_ml[kWarps];
  __shared__ float warp_acc[kWarps][HD];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x / p.H, head = blockIdx.x - i * p.H;
  const int kvh = head / p.G, in_group = head - kvh * p.G, head_lane = kvh * p.HC + in_group / p.GC, qr = in_group % p.GC;
  int first = 0, last = 0, row = i;
  bool served = true;
  if (p.all_single) {
    const int mine = (int)threadIdx.x < p.rows ? decode_row(p, nullptr, threadIdx.x).tiles : 0;
    const int total = p.rows <= kThreads ? block_total(mine, scan) : tiles_below(p, nullptr, p.rows, scan);
    const int per = tiles_a_range(p, mine, total, scan), tiles = decode_row(p, nullptr, i).tiles;
    if (per > 0) {
      first = block_total((int)threadIdx.x < i ? (mine + per - 1) / per : 0, scan);
      last = first + (tiles + per - 1) / per - 1;
    } else {
      const int ranges = min(p.ranges, total), begin = tiles_below(p, nullptr, i, scan);
      first = asb::block_of(total, ranges, begin);
      last = asb::block_of(total, ranges, begin + tiles - 1);
    }
  } else if (p.short_rows == 0) {  // a launch over all rows of a step meets longer requests', which the decode kernel left alone
    served = decode_row(p, p.req_q_start, i).tiles > 0;
  }
  asb::pdl_wait();  // the stream's previous kernel has completed (programmatic dependent launch)
  asb::pdl_launch_dependents();
  if (!served) return;
  if (!p.all_single) {
    const int4 cut = p.cuts[i];
    first = cut.x;
    last = cut.y;
    row = cut.z;
  }
  if (first == last) return;  // one block had it all and stored it
  // a warp takes every fourth block of the row, four of them at a time
  float mx = -INFINITY, den = 0.f, a[V];
#pragma unroll
  for (int k = 0; k < V; ++k) a[k] = 0.f;
  struct alignas(4 * V) Vec { float v[V]; };
  for (int j0 = first + warp; j0 <= last; j0 += 4 * kWarps) {
    float2 s[4];
    Vec v[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = j0 + u * kWarps;
      s[u] = make_float2(-INFINITY, 0.f);
      if (j > last) continue;
      const size_t at = (2 * ((size_t)j * p.lanes + head_lane) + (j == first ? 1 : 0)) * p.GC + qr;
      s[u] = *reinterpret_cast<const float2*>(p.part_ml + at * 2);
      v[u] = *reinterpret_cast<const Vec*>(p.part_acc + at * HD + lane * V);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (s[u].y == 0.f) continue;
      const float m_new = fmaxf(mx, s[u].x), f_old = exp2f(mx - m_new), f = exp2f(s[u].x - m_new);
      den = den * f_old + s[u].y * f;
#pragma unroll
      for (int k = 0; k < V; ++k) a[k] = a[k] * f_old + v[u].v[k] * f;
      mx = m_new;
    }
  }
  if (lane == 0) warp_ml[warp] = make_float2(mx, den);
#pragma unroll
  for (int k = 0; k < V; ++k) warp_acc[warp][lane * V + k] = a[k];
  __syncthreads();
  const int col = threadIdx.x;
  if (col >= HD) return;
  float m_all = -INFINITY;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) m_all = fmaxf(m_all, warp_ml[w].x);  // (the row's first block has a finite one)
  float sum = 0.f, value = 0.f;
#pragma unroll
  for (int w = 0; w < kWarps; ++w) {
    const float f = exp2f(warp_ml[w].x - m_all);
    sum += warp_ml[w].y * f;
    value += warp_acc[w][col] * f;
  }
  p.out[((size_t)row * p.H + head) * HD + col] = __float2bfloat16_rn(value / sum);
}

// ---- prefill -----------------------------------------------------------------------------------

constexpr int kPrefillThreads = 256;  // eight warps of sixteen rows
constexpr int kPrefillRows = 128;

template <int HD>
__device__ __forceinline__ void prefill_rows(const MmaParams& p) {
  asb::pdl_wait();  // the stream's previous kernel has completed (programmatic dependent launch)
  asb::pdl_launch_dependents();
  extern __shared__ __align__(128) unsigned char smem_raw[];
  constexpr int kTileBytes = kKeyTile * HD * 2;
  const uint32_t smem = smem_u32(smem_raw);
  auto k_stage = [&](int i) { return smem + (uint32_t)(i & 1) * kTileBytes; };
  auto v_stage = [&](int i) { return smem + (uint32_t)(2 + (i & 1)) * kTileBytes; };
  const uint32_t q_tile = smem + 4 * kTileBytes;  // 128 rows

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // Which request and tile of its tokens? Only requests with more than kShortRows tokens count.
  // (blocks are numbered head chunk fastest, so that every kv head's longest block starts first)
  const int chunks = p.KV * p.HC;
  const int chunk = blockIdx.x % chunks;
  int tile = blockIdx.x / chunks, r = 0, q_len = 0;
  for (; r < p.R; ++r) {
    q_len = p.req_q_start[r + 1] - p.req_q_start[r];
    if (q_len <= kShortRows) continue;
    const int tiles = (q_len + p.QT - 1) / p.QT;
    if (tile < tiles) {
      tile = tiles - 1 - tile;  // late tiles see the most keys: start them first
      break;
    }
    tile -= tiles;
  }
  if (r >= p.R) return;
  const int q0 = tile * p.QT;
  const int nq = min(p.QT, q_len - q0);
  const int row0 = p.req_q_start[r] + q0;
  const int pos0 = p.req_pos_start[r] + q0;
  const int kvh = chunk / p.HC;
  const int head0 = kvh * p.G + (chunk % p.HC) * p.GC;
  const int gc = min(p.GC, kvh * p.G + p.G - head0);
  const int num_rows = nq * gc;  // tile row rr = qi * gc + g
  const int* table = p.block_tables + (size_t)r * p.table_width;

  int key_lo = p.window > 0 ? max(0, pos0 - p.window + 1) : 0;
  if (p.chunk > 0) key_lo = max(key_lo, pos0 - pos0 % p.chunk);
  const int key_hi = pos0 + nq;

  {
    constexpr int kChunks = HD / 8;
    for (int i = threadIdx.x; i < kPrefillRows * kChunks; i += kPrefillThreads) {
      const int rr = i / kChunks, c = i % kChunks;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (rr < num_rows) {
        const int qi = rr / gc, g = rr - qi * gc;
        const __nv_bfloat162* src = reinterpret_cast<const __nv_bfloat162*>(
            p.q + ((size_t)(row0 + qi) * p.H + head0 + g) * HD + c * 8);
        v = *reinterpret_cast<const uint4*>(src);
      }
      *reinterpret_cast<uint4*>(smem_raw + (q_tile - smem) + tile_offset<HD>(rr, c)) = v;
    }
  }

  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  float acc[HD / 8][4];
#pragma unroll
  for (int i = 0; i < HD / 8; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;

  // positions of this thread's two rows (rows warp*16 + g and + 8)
  const int g4 = lane >> 2;
  int qpos[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int rr = warp * 16 + g4 + h * 8;
    qpos[h] = rr < num_rows ? pos0 + rr / gc : -1;  // -1: a padding row, sees nothing
  }
  // keys this warp's rows can see at all
  const int warp_first = warp * 16, warp_last = min(warp * 16 + 15, num_rows - 1);
  const int warp_hi = warp_first < num_rows ? pos0 + warp_last / gc + 1 : 0;
  const int warp_min_pos = pos0 + warp_first / gc;            // position of the warp's first row
  const int warp_max_pos = warp_hi - 1;                       // and of its last real row
  int warp_lo = p.window > 0 ? max(0, warp_min_pos - p.window + 1) : 0;
  if (p.chunk > 0) warp_lo = max(warp_lo, warp_min_pos - warp_min_pos % p.chunk);
  // where the last row's run of positions begins: tiles from there on lie in every row's run
  const int warp_chunk_lo = p.chunk > 0 && warp_max_pos >= 0 ? warp_max_pos - warp_max_pos % p.chunk : 0;
  const float cap2 = p.softcap * 1.4426950408889634f;         // the cap in the scores' log2 units
  const bool warp_full = warp_first + 15 < num_rows;          // no padding rows in this warp

  const int kt_begin = (key_lo / kKeyTile) * kKeyTile;
  const int num_tiles = (key_hi - kt_begin + kKeyTile - 1) / kKeyTile;
  load_kv_tile<HD, kPrefillThreads>(k_stage(0), v_stage(0), p, table, kvh, kt_begin, key_lo, key_hi);
  cp_async_commit();
  __syncthreads();  // the Q tile is in shared memory; fragments are read from it as needed

  for (int it = 0; it < num_tiles; ++it) {
    const int kt0 = kt_begin + it * kKeyTile;
    if (it + 1 < num_tiles)
      load_kv_tile<HD, kPrefillThreads>(k_stage(it + 1), v_stage(it + 1), p, table, kvh, kt0 + kKeyTile, key_lo, key_hi);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();

    if (kt0 < warp_hi && kt0 + kKeyTile > warp_lo) {
      // Scores of this warp's 16 rows against all 64 keys of the tile, in units of log2(e) so that
      // the exponentials are bare ex2 instructions; 16-key groups no row can see are skipped.
      float s[kKeyTile / 8][4];
      bool live[kKeyTile / 16];
      const bool all_live = kt0 + kKeyTile <= warp_hi && kt0 >= warp_lo;  // uniform in the warp
      if (all_live) {
#pragma unroll
        for (int sub = 0; sub < kKeyTile / 16; ++sub) live[sub] = true;
        qk_64keys_smem_q<HD>(s, q_tile, warp * 16, k_stage(it), lane, p.scale * 1.4426950408889634f);
      } else
#pragma unroll
      for (int sub = 0; sub < kKeyTile / 16; ++sub) {
        live[sub] = kt0 + sub * 16 < warp_hi && kt0 + sub * 16 + 16 > warp_lo;  // uniform in the warp
        if (live[sub]) {
          float part[2][4];
          qk_16keys_smem_q<HD>(part, q_tile, warp * 16, k_stage(it), sub * 16, lane, p.scale * 1.4426950408889634f);
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            s[sub * 2][e] = part[0][e];
            s[sub * 2 + 1][e] = part[1][e];
          }
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) s[sub * 2][e] = s[sub * 2 + 1][e] = -INFINITY;
        }
      }
      // Masks are needed only where the tile touches a row's own position, the window's edge or
      // the ends of the key range; tiles strictly inside every row's view skip them.
      const bool inside = warp_full && kt0 + kKeyTile <= warp_min_pos + 1 && kt0 >= key_lo && kt0 + kKeyTile <= key_hi &&
                          (p.window <= 0 || kt0 > warp_max_pos - p.window) && kt0 >= warp_chunk_lo;
      float rmax[2] = {-INFINITY, -INFINITY};
      if (cap2 > 0.f) {
        // (a group no row sees holds -inf, which the cap turns into -cap: such tiles are never `inside`)
#pragma unroll
        for (int j = 0; j < kKeyTile / 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) s[j][e] = capped(s[j][e], cap2);
      }
#pragma unroll
      for (int j = 0; j < kKeyTile / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          if (!inside) {
            const int key = kt0 + j * 8 + (lane & 3) * 2 + (e & 1);
            const int qp = qpos[e >> 1];
            const bool visible = key <= qp && key >= key_lo && (p.window <= 0 || key > qp - p.window) &&
                                 (p.chunk <= 0 || key >= qp - qp % p.chunk);
            if (!visible) s[j][e] = -INFINITY;
          }
          rmax[e >> 1] = fmaxf(rmax[e >> 1], s[j][e]);
        }
      float corr[2], rsum[2] = {0.f, 0.f}, m_use[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        rmax[h] = fmaxf(rmax[h], __shfl_xor_sync(0xffffffffu, rmax[h], 1));
        rmax[h] = fmaxf(rmax[h], __shfl_xor_sync(0xffffffffu, rmax[h], 2));
        const float m_new = fmaxf(m[h], rmax[h]);
        // a row that has seen nothing yet keeps max -inf: use 0 in the exponent to avoid inf - inf
        m_use[h] = m_new == -INFINITY ? 0.f : m_new;
        corr[h] = fast_exp2(m[h] - m_use[h]);
        m[h] = m_new;
      }
#pragma unroll
      for (int j = 0; j < kKeyTile / 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float pe = fast_exp2(s[j][e] - m_use[e >> 1]);
          s[j][e] = pe;
          rsum[e >> 1] += pe;
        }
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        rsum[h] += __shfl_xor_sync(0xffffffffu, rsum[h], 1);
        rsum[h] += __shfl_xor_sync(0xffffffffu, rsum[h], 2);
        l[h] = l[h] * corr[h] + rsum[h];
      }
#pragma unroll
      for (int i = 0; i < HD / 8; ++i) {
        acc[i][0] *= corr[0]; acc[i][1] *= corr[0];
        acc[i][2] *= corr[1]; acc[i][3] *= corr[1];
      }
#pragma unroll
      for (int sub = 0; sub < kKeyTile / 16; ++sub) {
        if (!live[sub]) continue;
        const uint32_t pf[4] = {pack_bf16(s[sub * 2][0], s[sub * 2][1]), pack_bf16(s[sub * 2][2], s[sub * 2][3]),
                                pack_bf16(s[sub * 2 + 1][0], s[sub * 2 + 1][1]), pack_bf16(s[sub * 2 + 1][2], s[sub * 2 + 1][3])};
        pv_16keys<HD>(acc, pf, v_stage(it), sub * 16, lane);
      }
    }
    __syncthreads();
  }
  cp_async_wait<0>();

  const int t = lane & 3;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int rr = warp * 16 + g4 + h * 8;
    if (rr >= num_rows) continue;
    const int qi = rr / gc, g = rr - qi * gc;
    __nv_bfloat16* o = p.out + ((size_t)(row0 + qi) * p.H + head0 + g) * HD;
    if (p.sink) l[h] += exp2f(p.sink[head0 + g] * 1.4426950408889634f - m[h]);  // scores and maxima are in log2 units here
    const float inv = 1.f / l[h];
#pragma unroll
    for (int i = 0; i < HD / 8; ++i)
      *reinterpret_cast<__nv_bfloat162*>(o + i * 8 + t * 2) =
          __floats2bfloat162_rn(acc[i][h * 2] * inv, acc[i][h * 2 + 1] * inv);
  }
}

// At the 128 registers that two blocks an SM leave, how the compiler reaches the parameters decides what it spills: from the
// constant bank 20 / 44 bytes with head size 64 (64 / 112 with 128), copied 24 / 72 (8 / 4). 512 tokens at position 7,000, 32 heads
// over 8: head size 64 309 us against 333, head size 128 577 against 547.
template <int HD>
__global__ void __launch_bounds__(kPrefillThreads, 2) prefill_attention_kernel(const __grid_constant__ MmaParams p) { prefill_rows<HD>(p); }
template <int HD>
__global__ void __launch_bounds__(kPrefillThreads, 2) prefill_attention_copied_kernel(const MmaParams p) { prefill_rows<HD>(p); }

template <int HD>
int launch_prefill(const MmaParams& p, cudaStream_t stream) {
  const int smem = 4 * kKeyTile * HD * 2 + kPrefillRows * HD * 2;
  auto kern = HD == 64 ? prefill_attention_kernel<64> : prefill_attention_copied_kernel<128>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return asb::fail("prefill_attention: %s", cudaGetErrorString(e));
  const long long blocks = (long long)((p.T + p.QT - 1) / p.QT + p.R) * p.KV * p.HC;
  if (blocks > 0x7fffffffLL) return asb::fail("prefill_attention: %lld blocks exceed the grid", blocks);
  asb::launch(kern, dim3((unsigned)blocks), kPrefillThreads, smem, stream, p);
  return asb::check_launch("prefill_attention");
}

int decode_smem(int hd, int gc) { return kDecodeStages * (2 * kKeyTile + (gc <= 8 ? 8 : 16)) * hd * 2 + 128; }  // (a base of 128 bytes to one of 256)

template <int HD>
int launch_decode(const DecodeParams& p, cudaStream_t stream) {
  const int smem = decode_smem(HD, p.GC);
  auto kern = p.GC <= 8 ? decode_attention_kernel<HD, true> : decode_attention_kernel<HD, false>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return asb::fail("decode_attention: %s", cudaGetErrorString(e));
  asb::launch(kern, dim3((p.ranges > 0 ? p.ranges : p.rows) * p.lanes), kThreads, smem, stream, p);
  if (int rc = asb::check_launch("decode_attention")) return rc;
  if (p.ranges == 0) return 0;
  asb::launch(decode_merge_kernel<HD>, dim3(p.rows * p.H), kThreads, 0, stream, p);
  return asb::check_launch("decode_merge");
}

template <int HD, bool Half>
int resident_blocks(int sms) {
  int per_sm = 0;
  auto kern = decode_attention_kernel<HD, Half>;
  const int smem = decode_smem(HD, Half ? 8 : 16);
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  asb::prefer_shared_carveout((const void*)kern);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem) != cudaSuccess) return 0;
  return per_sm * sms;
}

}  // namespace

// How many blocks of the decode kernel for `group` heads a kv head the device holds at once (blocks per SM x SMs), which
// is what the caller's choice of ranges aims to fill; 0 for a head size not served. (Head size 64 with up to 8 heads: four
// an SM; with three counted, 128 rows of 2,048 keys, 32 heads over 8, took 100 us instead of 97.)
extern "C" int asb_decode_attention_resident(int hd, int group) {
  if (hd != 64 && hd != 128) return 0;
  static int cached[4] = {0, 0, 0, 0};
  int& slot = cached[2 * (hd == 128) + (group <= 8)];
  if (slot) return slot;
  int device = 0, sms = 0;
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess)
    return 0;
  if (group <= 8) return slot = hd == 64 ? resident_blocks<64, true>(sms) : resident_blocks<128, true>(sms);
  return slot = hd == 64 ? resident_blocks<64, false>(sms) : resident_blocks<128, false>(sms);
}

// The same for more than 8 heads a kv head, the least of them.
extern "C" int asb_decode_attention_resident_blocks(int hd) { return asb_decode_attention_resident(hd, 16); }

// 1 if this (head size, group) is served by the tensor-core kernels.
extern "C" int asb_attention_mma_supported(int hd, int group) {
  return (hd == 64 || hd == 128) && group >= 1 ? 1 : 0;
}

// The rows of requests that bring at most 8 new tokens each (all_single: every request brings one). short_rows > 0: the
// number of such rows in a step that also holds longer portions, whose rows are left alone; 0: T rows, those of
// longer requests left alone.
// ranges: the keys of all rows are cut into as many equal ranges, each for KV * ceil(H / KV / 16) thread blocks; 0: each
// row is a range. scratch: float32, 16-byte aligned, 4 * rows + 2 * ranges * KV * ceil(H / KV / 16) * min(H / KV, 16) *
// (hd + 2) elements (null with 0 ranges).
// chunk, softcap (0: none), early: see DecodeParams. (Letting the last block to arrive merge the shares inside the
// kernel was measured and was slower than the second launch.)
extern "C" int asb_decode_attention(void* out, const void* q, const void* k_cache, const void* v_cache,
                                    const int* block_tables, const int* req_q_start, const int* req_pos_start,
                                    float* scratch, const float* sink, int T, int R, int H, int KV, int hd, int bs,
                                    int table_width, int window, int chunk, int ranges, float scale, float softcap,
                                    int all_single, int short_rows, int early, cudaStream_t stream) {
  if (chunk < 0 || softcap < 0.f) return asb::fail("decode_attention: chunk %d and softcap %f must not be negative", chunk, (double)softcap);
  if (T == 0 || R == 0) return 0;
  if (short_rows < 0 || short_rows > T || (short_rows > 0 && all_single) || (all_single && R != T))
    return asb::fail("decode_attention: %d short rows of %d tokens", short_rows, T);
  if (KV < 1 || H % KV) return asb::fail("decode_attention: %d heads over %d kv heads", H, KV);
  if (!asb_attention_mma_supported(hd, H / KV)) return asb::fail("decode_attention: head_dim %d is not 64 or 128", hd);
  if (ranges < 0 || (ranges > 0 && (!scratch || ((uintptr_t)scratch & 15)))) return asb::fail("decode_attention: %d ranges need scratch", ranges);
  DecodeParams p;
  p.q = (const __nv_bfloat16*)q; p.out = (__nv_bfloat16*)out;
  p.k_cache = (const __nv_bfloat16*)k_cache; p.v_cache = (const __nv_bfloat16*)v_cache;
  p.block_tables = block_tables; p.req_q_start = req_q_start; p.req_pos_start = req_pos_start;
  p.sink = sink;
  p.rows = short_rows > 0 ? short_rows : T;
  p.R = R; p.H = H; p.KV = KV; p.bs = bs; p.table_width = table_width;
  p.G = H / KV;
  p.GC = p.G < 16 ? p.G : 16;
  p.HC = (p.G + p.GC - 1) / p.GC;
  p.lanes = KV * p.HC;
  if ((long long)p.rows * H > 0x7fffffffLL || (long long)ranges * p.lanes > 0x7fffffffLL)
    return asb::fail("decode_attention: %d rows of %d heads, %d ranges exceed the grid", p.rows, H, ranges);
  p.window = window; p.chunk = chunk; p.softcap = softcap; p.scale = scale;
  p.all_single = all_single; p.short_rows = short_rows;
  p.early = early;
  p.ranges = ranges;
  p.cuts = (int4*)scratch;
  p.part_acc = scratch ? scratch + 4 * (size_t)p.rows : nullptr;
  p.part_ml = scratch ? p.part_acc + 2 * (size_t)ranges * p.lanes * p.GC * hd : nullptr;
  return hd == 64 ? launch_decode<64>(p, stream) : launch_decode<128>(p, stream);
}

// The longer portions (requests that bring more than 8 new tokens; the others' rows are left alone).
// chunk, softcap (0: none): see MmaParams.
extern "C" int asb_prefill_attention_mma(void* out, const void* q, const void* k_cache, const void* v_cache,
                                         const int* block_tables, const int* req_q_start, const int* req_pos_start,
                                         const float* sink, int num_tokens, int R, int H, int KV, int hd, int bs,
                                         int table_width, int window, int chunk, float scale, float softcap,
                                         cudaStream_t stream) {
  if (chunk < 0 || softcap < 0.f) return asb::fail("prefill_attention: chunk %d and softcap %f must not be negative", chunk, (double)softcap);
  if (num_tokens == 0 || R == 0) return 0;
  if (KV < 1 || H % KV) return asb::fail("prefill_attention: %d heads over %d kv heads", H, KV);
  if (!asb_attention_mma_supported(hd, H / KV)) return asb::fail("prefill_attention: head_dim %d is not 64 or 128", hd);
  MmaParams p;
  p.q = (const __nv_bfloat16*)q; p.out = (__nv_bfloat16*)out;
  p.k_cache = (const __nv_bfloat16*)k_cache; p.v_cache = (const __nv_bfloat16*)v_cache;
  p.block_tables = block_tables; p.req_q_start = req_q_start; p.req_pos_start = req_pos_start;
  p.sink = sink;
  p.T = num_tokens; p.R = R; p.H = H; p.KV = KV; p.bs = bs; p.table_width = table_width;
  p.G = H / KV;
  p.GC = p.G < 16 ? p.G : 16;
  p.HC = (p.G + p.GC - 1) / p.GC;
  p.QT = kPrefillRows / p.GC;
  p.window = window; p.scale = scale; p.chunk = chunk; p.softcap = softcap;
  return hd == 64 ? launch_prefill<64>(p, stream) : launch_prefill<128>(p, stream);
}
