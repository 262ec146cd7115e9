// The projections between one layer's attention and the next one's, for few tokens, as one persistent kernel:
//
//   x1 = attn . Wo^T + x;  h = SiLU(N(x1) . Wg^T) * (N(x1) . Wu^T);  x2 = h . Wd^T + x1;  p = N'(x2) . Wqkv^T
//
// (atomserve/model.py:336, 354-360, 378-382 and the next layer's :326-329), N the RMS norms. With up to 8 tokens, one column
// of tiles, each product is a read of its matrix, and as separate kernels a layer's four products left memory idle for 2 to 3
// us at each of nine kernel boundaries. Here the matrices are one stream: every block owns 1 / gridDim of each matrix's
// rows, and its loader warps walk the block's rows of all four matrices in order through one ring of stages, stopping
// for nothing but a full ring. Where a product needs what all blocks made of the one before (a grid barrier, about 3 us
// until the first multiply-add that follows), the loaders have the next matrix's first 180 KB under way or landed, which
// at the device's memory rate is 4 us' worth: memory does not see the barriers.
//
// A stage holds 14 weight rows x 512 elements of K, copied row by row (`cp.async.bulk`, 1 KB each, any number of rows;
// rows 1088 bytes apart, so that the fragment reads below meet no bank conflict; a loader issues such a copy every 37 ns,
// so that four of them stay ahead of memory). The eight multiplying warps share a stage along K, 64 elements each, with
// the weights as the rows of mma.sync's m16n8k16 and the tokens as its columns: per 14 KB of weights and SM, which memory
// delivers in some 600 cycles, a warp issues 4 shared loads and 4 mma. (tcgen05's tiles have 64 or 128 rows:
// they would have to be cut along K to give every SM its share of 4096 rows, and the cut sums met again behind one
// barrier more.) K runs outside, the block's row tiles inside: a token's elements are read once per K step from L2 into
// registers, a step ahead, multiplied there by the norm's gains where the product's input is a norm's output, and serve
// all row tiles. The warps' sums meet in shared memory at the end of a product, in a fixed order, where the epilogue
// multiplies by the norm's factor of the token, rounds and stores them.
//
// The norms' sums of squares: every block leaves its rows' share per token, and all blocks add up the shares of all
// blocks in one order, so that each token's factor is the same everywhere, and the same for any number of tokens.
//
// Measured in a CUDA graph of such layers, 1 and 8 tokens, in us, as separate kernels and as one, beside the matrices' time
// at 6,549 GB/s: Qwen3-8B's sizes 78.3, 80.8 -> 70.0, 73.0 (58.9); 14B's 118.7, 121.7 -> 106.8, 110.3 (100.9); 32B's 163.6,
// 167.0 -> 152.6, 156.8 (148.9); a hidden size of 512 (1.0) 19.2, 19.5 -> 13.5, 14.2: no size in between was slower, so
// the sizes do not decide. What is left: the first product's start, and about 1.5 us at each barrier. Loads held to 84 KB
// in flight an SM (so that the SMs stay level) were slower, 72 -> 73 us; without the gains' early loads, the factor's sums
// beside the first K step and the early residual it took 74.
//
// Waits are bounded; one that runs out reports through the status word and the block goes on to its end without waiting.
#include "tcgen05.cuh"

#include "glu.cuh"

namespace {

using asb::t5::mbar_arrive;
using asb::t5::mbar_expect_tx;
using asb::t5::mbar_init;
using asb::t5::smem_u32;

constexpr int kWarps = 8;            // multiplying warps
constexpr int kLoaders = 4;          // loader warps, which take the stages in turn (a warpgroup: they give registers to the others)
constexpr int kThreads = (kWarps + kLoaders) * 32;
constexpr int kTileRows = 14;        // of the 16 of a fragment: 28 and 42 rows a block, as the served sizes have, fill their stages
constexpr int kStepK = 512;          // elements of K per stage, 64 per warp
constexpr int kPitch = kStepK * 2 + 64;
constexpr int kStageBytes = kTileRows * kPitch;
constexpr int kStages = 13;
constexpr int kMaxTiles = 12;        // row tiles that a warp holds sums of at once (48 registers)
constexpr int kSumFloats = 5376;     // shared memory in which the warps' sums meet (it follows the ring: a fragment's rows
                                     // past the last stage's lie in it, and belong to no result)
constexpr uint32_t kBarrierPolls = 1u << 22;
constexpr int kMaxPhases = 4;
constexpr int kMaxTokens = 8;        // the columns of a fragment, and one token a warp where the norm's factors are worked out
constexpr int kMaxBlocks = 160;      // a multiple of 32
constexpr int kGroup = kSumFloats / (kWarps * kTileRows * kMaxTokens);  // row tiles whose sums meet at once

enum Epilogue : int { kResidual = 0, kSwiglu = 1, kPlain = 2 };

struct Phase {
  const __nv_bfloat16* w;         // [rows, k]
  const __nv_bfloat16* x;         // [tokens, k]
  const float* gain;              // not null: x is normed on the way in, with the sums of squares `squares_in`
  const float* squares_in;        // [tokens, gridDim]
  const __nv_bfloat16* residual;  // [tokens, rows] (kResidual)
  __nv_bfloat16* out;             // [tokens, rows], or [tokens, rows / 2] (kSwiglu)
  float* squares_out;             // [tokens, gridDim] (kResidual)
  float eps;
  int rows, k, epilogue;
};

struct Chain {
  Phase phase[kMaxPhases];
  int phases, tokens;
  unsigned* arrived;  // [kMaxPhases] zeroed
  int* status;
};

struct Shared {
  unsigned long long full[kStages], empty[kStages];
  float rstd[kMaxTokens];
  float part[kWarps][kMaxTokens];
  int dead;
};

constexpr int kSharedBytes = kStages * kStageBytes + kSumFloats * 4 + (int)sizeof(Shared);

__device__ __forceinline__ bool given_up(const Shared& s) { return *(const volatile int*)&s.dead; }

// A bounded wait that ends at once where another one of the block has run out.
__device__ __forceinline__ void wait_or_give_up(Shared& s, uint32_t bar, uint32_t parity, int* status, int code) {
  for (uint32_t i = 0; i < asb::t5::kMaxPolls; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done || given_up(s)) return;
  }
  atomicExch(status, code);
  *(volatile int*)&s.dead = 1;
}

__device__ __forceinline__ void sync_multipliers() { asm volatile("bar.sync 1, %0;" ::"n"(kWarps * 32) : "memory"); }

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar, uint64_t policy) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
      "l"(src), "r"(bytes), "r"(bar), "l"(policy)
      : "memory");
}

__device__ __forceinline__ void lds128(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ld.shared.v4.b32 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

__device__ __forceinline__ void mma16816(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// This block's rows of a matrix of `rows` (even) rows: whole pairs, as the gated rows are.
__device__ __forceinline__ int first_row(int rows, int block, int blocks) { return 2 * (int)((long long)(rows / 2) * block / blocks); }
// How they are walked: in equal passes of at most kMaxTiles tiles.
__device__ __forceinline__ int pass_rows(int own) {
  const int passes = (own + kMaxTiles * kTileRows - 1) / (kMaxTiles * kTileRows);
  return passes ? ((own / 2 + passes - 1) / passes) * 2 : 2;
}

__device__ void load_matrices(const Chain& c, Shared& s, uint32_t ring, int loader, int lane) {
  uint64_t policy;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(policy));
  int stage = 0, round = 0, turn = 0;
  for (int p = 0; p < c.phases; ++p) {
    const Phase& ph = c.phase[p];
    const int begin = first_row(ph.rows, blockIdx.x, gridDim.x), end = first_row(ph.rows, blockIdx.x + 1, gridDim.x);
    const int step = pass_rows(end - begin);
    for (int r0 = begin; r0 < end; r0 += step) {
      const int r1 = min(end, r0 + step);
      for (int k0 = 0; k0 < ph.k; k0 += kStepK) {
        for (int r = r0; r < r1; r += kTileRows) {
          if (turn == loader) {
            const uint32_t full = smem_u32(&s.full[stage]);
            wait_or_give_up(s, smem_u32(&s.empty[stage]), (round & 1) ^ 1, c.status, 41);
            if (__any_sync(0xffffffffu, given_up(s))) return;
            const int n = min(kTileRows, r1 - r);
            if (lane == 0) mbar_expect_tx(full, (uint32_t)n * kStepK * 2);
            __syncwarp();
            if (lane < n)
              bulk_load(ring + stage * kStageBytes + lane * kPitch, ph.w + (size_t)(r + lane) * ph.k + k0, kStepK * 2, full, policy);
            __syncwarp();
          }
          turn = turn + 1 == kLoaders ? 0 : turn + 1;
          if (++stage == kStages) stage = 0, ++round;
        }
      }
    }
  }
}

// 64 elements of K (this warp's share of a step) of the lane's token: element group lane % 4 of each half.
__device__ __forceinline__ void load_tokens(uint4 (&x)[2], const Phase& ph, int tokens, int k, int lane) {
  const int t = lane >> 2;
  const __nv_bfloat16* at = ph.x + (size_t)t * ph.k + k + (lane & 3) * 8;
  x[0] = x[1] = make_uint4(0, 0, 0, 0);
  if (t < tokens) {
    x[0] = __ldcg(reinterpret_cast<const uint4*>(at));
    x[1] = __ldcg(reinterpret_cast<const uint4*>(at + 32));
  }
}

// The gains of the same elements.
__device__ __forceinline__ void load_gains(float4 (&g)[2][2], const Phase& ph, int k, int lane) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float4* at = reinterpret_cast<const float4*>(ph.gain + k + h * 32 + (lane & 3) * 8);
    g[h][0] = __ldg(at);
    g[h][1] = __ldg(at + 1);
  }
}

__device__ __forceinline__ void scale_tokens(uint4 (&x)[2], const float4 (&gains)[2][2]) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const float* g = reinterpret_cast<const float*>(&gains[h]);
    __nv_bfloat162* v = reinterpret_cast<__nv_bfloat162*>(&x[h]);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float2 f = __bfloat1622float2(v[i]);
      v[i] = __floats2bfloat162_rn(f.x * g[2 * i], f.y * g[2 * i + 1]);
    }
  }
}

struct Walk {
  int stage, parity;
};

__device__ void multiply_phase(const Chain& c, const Phase& ph, Shared& s, uint32_t ring, float* sums, Walk& walk, float4 (&gains)[2][2],
                               int warp, int lane) {
  const int T = c.tokens, tid = warp * 32 + lane;
  // Tokens to a power of two: how the epilogue's threads divide. Where they add up squares, always the most tokens there are:
  // the order of a token's sum is then the same whatever else is in the step (and a block has few rows there: 14 to 18 pairs).
  int columns = ph.epilogue == kResidual ? kMaxTokens : 1;
  while (columns < T) columns *= 2;
  constexpr int TP = kMaxTokens;  // token columns
  static_assert(kMaxTokens <= kWarps, "a warp works out one token's factor");
  uint4 next[2];
  load_tokens(next, ph, T, warp * 64, lane);
  // The norm's factor of a token multiplies its sums: it is worked out beside the first K step. (This warp's token.)
  float shares[kMaxBlocks / 32];
  if (ph.gain) {
#pragma unroll
    for (int i = 0; i < kMaxBlocks / 32; ++i)
      shares[i] = warp < T && i * 32 + lane < gridDim.x ? __ldcg(ph.squares_in + (size_t)warp * gridDim.x + i * 32 + lane) : 0.f;
  }
  const int begin = first_row(ph.rows, blockIdx.x, gridDim.x), end = first_row(ph.rows, blockIdx.x + 1, gridDim.x);
  const int step = pass_rows(end - begin);
  const uint32_t lane_at = (uint32_t)((lane >> 2) * kPitch + warp * 128 + (lane & 3) * 16);
  uint32_t residual = 0;  // of the first pair of rows that the thread stores
  if (ph.epilogue == kResidual && (tid & (columns - 1)) < T && tid / columns * 2 < min(end - begin, kGroup * kTileRows))
    residual = __ldcg(reinterpret_cast<const unsigned*>(ph.residual + (size_t)(tid & (columns - 1)) * ph.rows + begin + tid / columns * 2));
  float squares = 0.f;  // of this thread's token, tid % columns
  for (int r0 = begin; r0 < end; r0 += step) {
    const int own = min(end, r0 + step) - r0, tiles = (own + kTileRows - 1) / kTileRows;
    float acc[kMaxTiles][4];
#pragma unroll
    for (int m = 0; m < kMaxTiles; ++m) acc[m][0] = acc[m][1] = acc[m][2] = acc[m][3] = 0.f;
    if (r0 != begin) {
      load_tokens(next, ph, T, warp * 64, lane);
      if (ph.gain) load_gains(gains, ph, warp * 64, lane);
    }
    for (int k0 = 0; k0 < ph.k; k0 += kStepK) {
      uint4 x[2] = {next[0], next[1]};
      if (k0 + kStepK < ph.k) load_tokens(next, ph, T, k0 + kStepK + warp * 64, lane);
      if (ph.gain) {
        scale_tokens(x, gains);
        if (k0 + kStepK < ph.k) load_gains(gains, ph, k0 + kStepK + warp * 64, lane);
      }
#pragma unroll
      for (int m = 0; m < kMaxTiles; ++m) {
        if (m >= tiles) break;
        wait_or_give_up(s, smem_u32(&s.full[walk.stage]), walk.parity, c.status, 42);
        const uint32_t at = ring + walk.stage * kStageBytes + lane_at;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          uint32_t a[4], b[4];  // rows lane / 4 and 8 further on, eight elements of K each: two K steps of the mma
          lds128(a, at + h * 64);
          lds128(b, at + h * 64 + 8 * kPitch);
          mma16816(acc[m], a[0], b[0], a[1], b[1], x[h].x, x[h].y);
          mma16816(acc[m], a[2], b[2], a[3], b[3], x[h].z, x[h].w);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&s.empty[walk.stage]));
        if (++walk.stage == kStages) walk.stage = 0, walk.parity ^= 1;
      }
      if (k0 == 0 && r0 == begin && ph.gain) {
        float v = 0.f;
#pragma unroll
        for (int i = 0; i < kMaxBlocks / 32; ++i) v += shares[i];
        v = asb::warp_sum(v);
        if (lane == 0 && warp < T) s.rstd[warp] = rsqrtf(v / (float)ph.k + ph.eps);
      }
    }
    // the warps' sums, kGroup row tiles at a time: [warp][row][token]
#pragma unroll
    for (int m0 = 0; m0 < kMaxTiles; m0 += kGroup) {
      if (m0 >= tiles) break;
      if (m0) sync_multipliers();  // (the group before has been read)
      float* mine = sums + warp * (kGroup * kTileRows * TP);
#pragma unroll
      for (int g = 0; g < kGroup; ++g) {
        if (m0 + g < kMaxTiles) {
          float* at = mine + (g * kTileRows + (lane >> 2)) * TP + (lane & 3) * 2;
          *reinterpret_cast<float2*>(at) = make_float2(acc[m0 + g][0], acc[m0 + g][1]);
          if ((lane >> 2) + 8 < kTileRows) *reinterpret_cast<float2*>(at + 8 * TP) = make_float2(acc[m0 + g][2], acc[m0 + g][3]);
        }
      }
      sync_multipliers();
      const int rows_here = min(own - m0 * kTileRows, kGroup * kTileRows), t = tid & (columns - 1);
      if (t < T) {
        for (int pair = tid / columns; pair < rows_here / 2; pair += kWarps * 32 / columns) {
          float v0 = 0.f, v1 = 0.f;
#pragma unroll
          for (int w = 0; w < kWarps; ++w) {
            const float* at = sums + (w * kGroup * kTileRows + pair * 2) * TP + t;
            v0 += at[0];
            v1 += at[TP];
          }
          const int row = r0 + m0 * kTileRows + pair * 2;
          if (ph.gain) v0 *= s.rstd[t], v1 *= s.rstd[t];
          if (ph.epilogue == kSwiglu) {
            ph.out[(size_t)t * (ph.rows / 2) + row / 2] = __float2bfloat16_rn(asb::glu_value<asb::kGluSilu>(v0, v1));
          } else {
            const size_t to = (size_t)t * ph.rows + row;
            if (ph.epilogue == kResidual) {
              const uint32_t raw = row == begin + tid / columns * 2 ? residual : __ldcg(reinterpret_cast<const unsigned*>(ph.residual + to));
              const float2 r = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw));
              v0 += r.x;
              v1 += r.y;
            }
            const __nv_bfloat162 o = __floats2bfloat162_rn(v0, v1);
            *reinterpret_cast<__nv_bfloat162*>(ph.out + to) = o;
            const float2 f = __bfloat1622float2(o);
            squares = fmaf(f.x, f.x, fmaf(f.y, f.y, squares));
          }
        }
      }
    }
    sync_multipliers();  // (the next pass or phase writes the sums again)
  }
  if (ph.epilogue == kResidual) {
    for (int o = columns; o < 32; o <<= 1) squares += __shfl_xor_sync(0xffffffffu, squares, o);
    if (lane < columns) s.part[warp][lane] = squares;
    sync_multipliers();
    if (tid < T) {
      float v = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) v += s.part[w][tid];
      ph.squares_out[(size_t)tid * gridDim.x + blockIdx.x] = v;
    }
  }
}

// All blocks' multiplying warps: everything stored before is visible to all after.
__device__ void grid_barrier(const Chain& c, Shared& s, int index, int tid) {
  sync_multipliers();
  if (tid == 0) {
    unsigned* at = c.arrived + index;
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(at) : "memory");
    bool done = false;
    for (uint32_t i = 0; i < kBarrierPolls && !done && !given_up(s); ++i) {
      unsigned seen;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(at) : "memory");
      done = seen >= gridDim.x;
    }
    if (!done && !given_up(s)) {
      atomicExch(c.status, 43);
      *(volatile int*)&s.dead = 1;
    }
  }
  sync_multipliers();
}

__global__ void __launch_bounds__(kThreads, 1) decode_chain_kernel(const __grid_constant__ Chain c) {
  extern __shared__ __align__(128) unsigned char memory[];
  float* sums = reinterpret_cast<float*>(memory + kStages * kStageBytes);
  Shared& s = *reinterpret_cast<Shared*>(memory + kStages * kStageBytes + kSumFloats * 4);
  const uint32_t ring = smem_u32(memory);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < kStages; ++i) {
      mbar_init(smem_u32(&s.full[i]), 1);
      mbar_init(smem_u32(&s.empty[i]), kWarps);
    }
    s.dead = 0;
    asb::t5::mbar_init_fence();
  }
  __syncthreads();
  if (warp >= kWarps) {
    // (128 x 40 + 256 x 224 = 62,464 registers, of the 384 x 168 = 64,512 that the block is launched with)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    load_matrices(c, s, ring, warp - kWarps, lane);  // weights: no kernel writes them, so nothing is waited for
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    // A load from every line of the gains, for nothing but to have them in L2 before their first product reads them. (With
    // prefetches in their place 70.6 us at Qwen3-8B's sizes instead of 70.0.)
    for (int p = 0; p < c.phases; ++p)
      if (c.phase[p].gain)
        for (int i = threadIdx.x * 32; i < c.phase[p].k; i += kWarps * 32 * 32) {
          float unused;
          asm volatile("ld.global.nc.L1::no_allocate.f32 %0, [%1];" : "=f"(unused) : "l"(c.phase[p].gain + i));
          (void)unused;
        }
    asb::pdl_wait();
    asb::pdl_launch_dependents();
    Walk walk = {0, 0};
    for (int p = 0; p < c.phases; ++p) {
      float4 gains[2][2];  // of the first K step: they wait for no other block
      if (c.phase[p].gain) load_gains(gains, c.phase[p], warp * 64, lane);
      if (p) grid_barrier(c, s, p - 1, threadIdx.x);
      multiply_phase(c, c.phase[p], s, ring, sums, walk, gains, warp, lane);
    }
  }
  __syncthreads();
  if (s.dead) {
    // copies may still be under way into this block's memory: give them the time that any copy takes
    for (int i = 0; i < 1 << 14; ++i) __nanosleep(1000);
  }
}

}  // namespace

// Tokens that the kernel takes, and the multiple that every product's K has to be.
extern "C" int asb_decode_chain_limits(int* tokens, int* k_multiple) {
  *tokens = kMaxTokens;
  *k_multiple = kStepK;
  return 0;
}

// Blocks that run at once on the current device (one an SM): the squares' scratch is [2, tokens, blocks] floats.
extern "C" int asb_decode_chain_blocks() {
  static int blocks[64] = {};
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= 64) return 0;
  if (!blocks[device]) {
    int n = 0;
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return 0;
    blocks[device] = n < kMaxBlocks ? n : kMaxBlocks;
  }
  return blocks[device];
}

// x1 = attn . wo^T + x; act = SiLU and product of N(x1) . wgu^T (rows of wgu alternate gate, up); x2 = act . wd^T + x1; and
// where wn is given, out = N'(x2) . wn^T. All bfloat16 but the gains; attn [tokens, attn_k], x, x1, x2 [tokens, hidden],
// act [tokens, ff], out [tokens, next_rows]; squares: 2 * tokens * blocks floats; arrived: four zeroed words.
extern "C" int asb_decode_chain(const void* attn, const void* wo, const void* x, void* x1, const float* gain, float eps, const void* wgu,
                                void* act, const void* wd, void* x2, const float* next_gain, float next_eps, const void* wn, void* out,
                                float* squares, unsigned* arrived, int tokens, int hidden, int attn_k, int ff, int next_rows, int* status,
                                cudaStream_t stream) {
  if (tokens < 1 || tokens > kMaxTokens) return asb::fail("decode_chain: %d tokens, it takes 1 to %d", tokens, kMaxTokens);
  if (hidden % kStepK || attn_k % kStepK || ff % kStepK || hidden < 1 || attn_k < 1 || ff < 1 || next_rows < 0 || next_rows % 2)
    return asb::fail("decode_chain: sizes %d, %d, %d must be multiples of %d, and %d rows even", hidden, attn_k, ff, kStepK, next_rows);
  if (((uintptr_t)attn | (uintptr_t)wo | (uintptr_t)x | (uintptr_t)x1 | (uintptr_t)gain | (uintptr_t)wgu | (uintptr_t)act | (uintptr_t)wd |
       (uintptr_t)x2 | (uintptr_t)next_gain | (uintptr_t)wn | (uintptr_t)out) & 15)
    return asb::fail("decode_chain: pointers must be 16-byte aligned");
  const int blocks = asb_decode_chain_blocks();
  if (!blocks) return asb::fail("decode_chain: the device does not say how many SMs it has");
  using B = __nv_bfloat16;
  float* squares2 = squares + (size_t)tokens * blocks;
  Chain c = {};
  c.phase[0] = {(const B*)wo, (const B*)attn, nullptr, nullptr, (const B*)x, (B*)x1, squares, 0.f, hidden, attn_k, kResidual};
  c.phase[1] = {(const B*)wgu, (const B*)x1, gain, squares, nullptr, (B*)act, nullptr, eps, 2 * ff, hidden, kSwiglu};
  c.phase[2] = {(const B*)wd, (const B*)act, nullptr, nullptr, (const B*)x1, (B*)x2, squares2, 0.f, hidden, ff, kResidual};
  c.phase[3] = {(const B*)wn, (const B*)x2, next_gain, squares2, nullptr, (B*)out, nullptr, next_eps, next_rows, hidden, kPlain};
  c.phases = wn ? 4 : 3;
  c.tokens = tokens;
  c.arrived = arrived;
  c.status = status;
  const cudaError_t set = cudaFuncSetAttribute((const void*)decode_chain_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSharedBytes);
  if (set != cudaSuccess) return asb::fail("decode_chain: %s", cudaGetErrorString(set));
  if (const int refused = asb::launch_cooperative(decode_chain_kernel, blocks, kThreads, kSharedBytes, stream, c)) return refused;
  return asb::check_launch("decode_chain");
}
