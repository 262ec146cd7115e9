// out[M, N] = x[M, K] . w[N, K]^T (+ residual[M, N]) on CUDA cores with float32 multiply-adds:
// the matrix product of the true 32-bit path (no tensor-core mode of reduced precision is
// involved), also instantiated for bfloat16 inputs as the fallback and the checker of the
// tensor-core kernels. Weights keep the checkpoint layout [out_features, in_features], so
// both operands are contiguous along K (atomserve/model.py:15-16; the residual form is the
// reference's addmm, atomserve/quant.py:89-91).
//
// Each output element is summed in a fixed order that depends on k and K alone: a chain of fused
// multiply-adds over each run of kRun consecutive k, the runs' sums added up in ascending order
// within each quarter of the runs, the quarters' sums in ascending order, whatever M and N are,
// wherever the element lies in its tile and whichever kernel computes it. A row's result
// therefore does not depend on which other rows share the batch. The levels keep the
// rounding error of a long sum (K = 12,288 in the served models) near that of a sum of
// sqrt(K) terms: one chain over all of K drifted 2.5e-5 of the largest logit from a float64
// oracle through two full-width layers, the blocked sum a fifth of that.
//
// Two kernels. Up to 16 rows the weights' bytes are the bound (rows_kernel); beyond, the multiply-adds (tile_kernel).
// The quarters are there so that both can share one output's K among the blocks of a cluster: a matrix of few
// rows (4,096) has too few tiles for the device otherwise.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kRun = 256;   // k per chain
constexpr int kQuarters = 4;
constexpr int BK = 16;      // k per stage; kRun is a multiple
constexpr int kSMs = 148;

// Two multiply-adds in one instruction, each rounded as fmaf rounds: d = a * b + d on both halves.
__device__ __forceinline__ void fma2(unsigned long long& d, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ unsigned long long both(float a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ float2 halves(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

// Four consecutive k of one row; what lies outside the matrix is zero. VEC: K a multiple of 4 and the rows aligned
// for one load.
template <typename T, bool VEC>
__device__ __forceinline__ float4 load4(const T* base, int row, int rows, int k, int K) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (row >= rows) return v;
  const T* at = base + (size_t)row * K + k;
  if (VEC) {
    if (k < K) {
      if constexpr (sizeof(T) == 4) {
        v = *reinterpret_cast<const float4*>(at);
      } else {
        const uint2 raw = *reinterpret_cast<const uint2*>(at);
        const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&raw.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&raw.y);
        v = make_float4(__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi));
      }
    }
  } else {
    if (k < K) v.x = asb::to_float(at[0]);
    if (k + 1 < K) v.y = asb::to_float(at[1]);
    if (k + 2 < K) v.z = asb::to_float(at[2]);
    if (k + 3 < K) v.w = asb::to_float(at[3]);
  }
  return v;
}

// ---- many rows: tiles of BM x 128, a quarter of K per block of a cluster ------------------------------------------

constexpr int BN = 128;

template <int BM>
struct Tile {
  static constexpr int LDX = BM + 4, LDW = BN + 4;  // 4 more: the transposing stores of one instruction hit 32 banks
  static constexpr int kStage = BK * (LDX + LDW);   // floats
  static constexpr size_t kSmem = sizeof(float) * (2 * kStage + BM * BN);
};

// What bounds it: the multiply-adds. A thread holds TM x 8 sums as pairs along n, so that per k it reads TM + 8 floats
// from shared memory for TM x 8 multiply-adds in half as many instructions; both operands lie k-major there, put
// so by the stores (the loads run along k), two stages, the next one's loads under way during the arithmetic. The
// runs' sums are banked in shared memory, which keeps a thread within 168 registers (124 with 32 rows) and three blocks on an SM.
template <typename TIn, typename TOut, int BM, int CLUSTER, bool VEC>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(kThreads, 3)
tile_kernel(TOut* __restrict__ out, const TIn* __restrict__ x, const TIn* __restrict__ w,
            const TOut* __restrict__ residual, int M, int N, int K) {
  using L = Tile<BM>;
  constexpr int TM = BM / 8;
  constexpr int XL = BM / 32, WL = BN / 32;  // loads of four k per thread and stage
  asb::pdl_wait();  // the stream's previous kernel has completed (programmatic dependent launch)
  asb::pdl_launch_dependents();
  extern __shared__ __align__(16) float smem[];
  float* total = smem + 2 * L::kStage;  // [BM][BN]: the sums of the runs so far
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tx = tid & 15, ty = tid >> 4;  // rows ty * TM .., columns tx * 4 .. and 64 + tx * 4 ..
  const int tile = (int)(blockIdx.x / CLUSTER), tiles_m = (M + BM - 1) / BM;  // tiles of the same weights side by side
  const int m0 = tile % tiles_m * BM, n0 = tile / tiles_m * BN;
  const int runs = (K + kRun - 1) / kRun;
  const int quarter = (int)(blockIdx.x % CLUSTER);
  const int k_begin = (int)((long long)quarter * runs / CLUSTER) * kRun;
  const int k_end = min(K, (int)((long long)(quarter + 1) * runs / CLUSTER) * kRun);

  // A warp's load covers 16 rows of 8 consecutive k (32 bytes of float32).
  float4 xr[XL], wr[WL];
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < XL; ++u) {
      const int task = u * kWarps + warp;
      xr[u] = load4<TIn, VEC>(x, m0 + (task >> 1) * 16 + (lane >> 1), M, k0 + ((task & 1) * 2 + (lane & 1)) * 4, K);
    }
#pragma unroll
    for (int u = 0; u < WL; ++u) {
      const int task = u * kWarps + warp;
      wr[u] = load4<TIn, VEC>(w, n0 + (task >> 1) * 16 + (lane >> 1), N, k0 + ((task & 1) * 2 + (lane & 1)) * 4, K);
    }
  };
  auto put = [&](int stage) {
    float* xs = smem + stage * L::kStage;
    float* ws = xs + BK * L::LDX;
#pragma unroll
    for (int u = 0; u < XL; ++u) {
      const int task = u * kWarps + warp, row = (task >> 1) * 16 + (lane >> 1), kq = ((task & 1) * 2 + (lane & 1)) * 4;
      xs[kq * L::LDX + row] = xr[u].x;
      xs[(kq + 1) * L::LDX + row] = xr[u].y;
      xs[(kq + 2) * L::LDX + row] = xr[u].z;
      xs[(kq + 3) * L::LDX + row] = xr[u].w;
    }
#pragma unroll
    for (int u = 0; u < WL; ++u) {
      const int task = u * kWarps + warp, row = (task >> 1) * 16 + (lane >> 1), kq = ((task & 1) * 2 + (lane & 1)) * 4;
      ws[kq * L::LDW + row] = wr[u].x;
      ws[(kq + 1) * L::LDW + row] = wr[u].y;
      ws[(kq + 2) * L::LDW + row] = wr[u].z;
      ws[(kq + 3) * L::LDW + row] = wr[u].w;
    }
  };

  unsigned long long acc[TM][4];  // [row][pair of columns]
#pragma unroll
  for (int i = 0; i < TM; ++i) {
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    float4* t = reinterpret_cast<float4*>(total + (ty * TM + i) * BN);  // (each thread banks where it alone reads)
    t[tx] = t[16 + tx] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  if (k_begin < k_end) {
    load(k_begin);
    put(0);
  }
  __syncthreads();
  int stage = 0;
  for (int k0 = k_begin; k0 < k_end; k0 += BK) {
    const bool more = k0 + BK < k_end;
    if (more) load(k0 + BK);
    const float* xs = smem + stage * L::kStage;
    const float* ws = xs + BK * L::LDX;
#pragma unroll
    for (int kk = 0; kk < BK; ++kk) {
      float a[TM];
#pragma unroll
      for (int i = 0; i < TM; i += 4) {
        const float4 v = *reinterpret_cast<const float4*>(xs + kk * L::LDX + ty * TM + i);
        a[i] = v.x; a[i + 1] = v.y; a[i + 2] = v.z; a[i + 3] = v.w;
      }
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(ws + kk * L::LDW + tx * 4);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(ws + kk * L::LDW + 64 + tx * 4);
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        const unsigned long long aa = both(a[i]);
        fma2(acc[i][0], aa, b0.x);
        fma2(acc[i][1], aa, b0.y);
        fma2(acc[i][2], aa, b1.x);
        fma2(acc[i][3], aa, b1.y);
      }
    }
    if ((k0 + BK) % kRun == 0 || !more) {  // the run is complete: bank its sum
#pragma unroll
      for (int i = 0; i < TM; ++i) {
        float4* t = reinterpret_cast<float4*>(total + (ty * TM + i) * BN);
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const float2 lo = halves(acc[i][2 * j]), hi = halves(acc[i][2 * j + 1]);
          float4 v = t[16 * j + tx];
          v.x += lo.x; v.y += lo.y; v.z += hi.x; v.w += hi.y;
          t[16 * j + tx] = v;
          acc[i][2 * j] = acc[i][2 * j + 1] = 0ull;
        }
      }
    }
    if (more) put(stage ^ 1);
    __syncthreads();
    stage ^= 1;
  }

  // Each block of the cluster adds up its share of the tile's rows over the quarters.
  const cg::cluster_group cluster = cg::this_cluster();
  if (CLUSTER > 1) cluster.sync();
  constexpr int kRows = BM / CLUSTER;
  for (int r = warp; r < kRows; r += kWarps) {
    const int row = quarter * kRows + r, m = m0 + row;
    if (m >= M) break;
#pragma unroll
    for (int c = 0; c < BN; c += 32) {
      const int n = n0 + c + lane;
      if (n >= N) break;
      float v = 0.f;
#pragma unroll
      for (int q = 0; q < CLUSTER; ++q) {
        const float* t = CLUSTER > 1 ? cluster.map_shared_rank(total, q) : total;
        v += t[row * BN + c + lane];
      }
      if (residual) v += asb::to_float(residual[(size_t)m * N + n]);
      out[(size_t)m * N + n] = asb::from_float<TOut>(v);
    }
  }
  if (CLUSTER > 1) cluster.sync();  // no block leaves while another reads its sums
}

// ---- up to 16 rows of float32: a warp walks whole runs of 64 weight rows -------------------------------------------

constexpr int kRowsN = 64;      // weight rows per block
constexpr int kLd = BK + 4;     // floats per row of a stage: eight lanes' 16-byte reads hit 32 banks
constexpr int kRowStages = 3;

template <int MR>
constexpr int row_stage() { return (kRowsN + MR) * kLd; }  // floats

__device__ __forceinline__ void copy16(float* to, const float* from, bool valid) {
  const uint32_t at = (uint32_t)__cvta_generic_to_shared(to);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at), "l"(from), "r"(valid ? 16 : 0) : "memory");
}

// What bounds it: the weights' bytes (with 16 rows, 16 multiply-adds a weight come close to the bound too). The runs of
// K are dealt out to the blocks of a cluster and to their warps; each warp brings its own weights through three
// stages of 64 rows x 16 k with cp.async and needs no barrier but its own, so eight warps keep 64 KB under way on an
// SM. A lane owns two weight rows (16-byte reads along k free of bank conflicts) and reads the rows of x as
// broadcasts. A run's sums go to shared memory, and once all runs are there the blocks of the cluster add them up.
template <int MR, int CLUSTER>
__global__ void __cluster_dims__(CLUSTER, 1, 1) __launch_bounds__(kThreads)
rows_kernel(float* __restrict__ out, const float* __restrict__ x, const float* __restrict__ w,
            const float* __restrict__ residual, int M, int N, int K, int w_stored) {
  extern __shared__ __align__(16) float smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)(blockIdx.x % CLUSTER);
  const int n0 = (int)(blockIdx.x / CLUSTER) * kRowsN;
  const int runs = (K + kRun - 1) / kRun;
  const int run_begin = (int)((long long)rank * runs / CLUSTER), run_end = (int)((long long)(rank + 1) * runs / CLUSTER);
  float* stages = smem + warp * kRowStages * row_stage<MR>();
  float* sums = smem + kWarps * kRowStages * row_stage<MR>();  // [run of this block][MR][kRowsN]

  // this warp's runs: run_begin + warp, + kWarps, ..; its stages in one sequence
  const int mine = run_end - run_begin > warp ? (run_end - run_begin - warp + kWarps - 1) / kWarps : 0;
  constexpr int kPerRun = kRun / BK;
  int steps = mine * kPerRun;
  if (mine > 0 && run_begin + warp + (mine - 1) * kWarps == runs - 1) steps -= kPerRun - ((K - (runs - 1) * kRun) + BK - 1) / BK;
  auto fetch_rows = [&](int step, int first, int last, const float* base, int base_row, int rows) {
    const int k0 = (run_begin + warp + (step / kPerRun) * kWarps) * kRun + (step % kPerRun) * BK;
    float* to = stages + (step % kRowStages) * row_stage<MR>();
#pragma unroll
    for (int i = first * 4 + lane; i < last * 4; i += 32) {
      const int r = i >> 2, k = k0 + (i & 3) * 4, row = base_row + r - first;
      const bool valid = row < rows && k < K;
      copy16(to + r * kLd + (i & 3) * 4, base + (valid ? (size_t)row * K + k : 0), valid);
    }
  };
  auto fetch_w = [&](int step) { if (step < steps) fetch_rows(step, 0, kRowsN, w, n0, N); };
  auto fetch_x = [&](int step) { if (step < steps) fetch_rows(step, kRowsN, kRowsN + MR, x, 0, M); };
  // a model's weights, which no kernel of a step writes, come before the wait for the stream's previous kernel
  if (!w_stored) asb::pdl_wait();
#pragma unroll
  for (int s = 0; s < kRowStages - 1; ++s) fetch_w(s);
  asb::pdl_wait();
  asb::pdl_launch_dependents();
#pragma unroll
  for (int s = 0; s < kRowStages - 1; ++s) {
    fetch_x(s);
    asm volatile("cp.async.commit_group;" ::: "memory");  // (the first group holds all weights asked for so far)
  }

  float acc[2][MR];
#pragma unroll
  for (int i = 0; i < MR; ++i) acc[0][i] = acc[1][i] = 0.f;
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;" ::"n"(kRowStages - 2) : "memory");
    __syncwarp();  // every lane's copies of this stage have landed, and every lane has read the stage before
    fetch_w(step + kRowStages - 1);
    fetch_x(step + kRowStages - 1);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const float* ws = stages + (step % kRowStages) * row_stage<MR>();
    const float* xs = ws + kRowsN * kLd;
#pragma unroll
    for (int kq = 0; kq < BK; kq += 4) {
      const float4 w0 = *reinterpret_cast<const float4*>(ws + lane * kLd + kq);
      const float4 w1 = *reinterpret_cast<const float4*>(ws + (32 + lane) * kLd + kq);
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        const float4 v = *reinterpret_cast<const float4*>(xs + m * kLd + kq);
        acc[0][m] = fmaf(v.w, w0.w, fmaf(v.z, w0.z, fmaf(v.y, w0.y, fmaf(v.x, w0.x, acc[0][m]))));
        acc[1][m] = fmaf(v.w, w1.w, fmaf(v.z, w1.z, fmaf(v.y, w1.y, fmaf(v.x, w1.x, acc[1][m]))));
      }
    }
    if ((step + 1) % kPerRun == 0 || step + 1 == steps) {
      float* to = sums + (size_t)(warp + (step / kPerRun) * kWarps) * MR * kRowsN;
#pragma unroll
      for (int m = 0; m < MR; ++m) {
        to[m * kRowsN + lane] = acc[0][m];
        to[m * kRowsN + 32 + lane] = acc[1][m];
        acc[0][m] = acc[1][m] = 0.f;
      }
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");

  const cg::cluster_group cluster = cg::this_cluster();
  if (CLUSTER > 1) cluster.sync();
  else __syncthreads();
  for (int i = rank * kThreads + tid; i < M * kRowsN; i += CLUSTER * kThreads) {
    const int m = i / kRowsN, col = i % kRowsN, n = n0 + col;
    if (n >= N) continue;
    float v = 0.f;
    if (CLUSTER == 1) {  // fewer runs than quarters: each is a quarter's
      for (int r = 0; r < runs; ++r) v += sums[((size_t)r * MR + m) * kRowsN + col];
    } else {
      constexpr int kEach = CLUSTER >= kQuarters ? CLUSTER / kQuarters : 1;  // blocks per quarter
      for (int q = 0; q < kQuarters; ++q) {
        float t = 0.f;
#pragma unroll
        for (int b = 0; b < kEach; ++b) {
          const int c = q * kEach + b;
          const float* from = cluster.map_shared_rank(sums, c) + m * kRowsN + col;
          const int count = (int)((long long)(c + 1) * runs / CLUSTER) - (int)((long long)c * runs / CLUSTER);
#pragma unroll 4
          for (int r = 0; r < count; ++r) t += from[(size_t)r * MR * kRowsN];
        }
        v += t;
      }
    }
    if (residual) v += residual[(size_t)m * N + n];
    out[(size_t)m * N + n] = v;
  }
  if (CLUSTER > 1) cluster.sync();  // no block leaves while another reads its sums
}

template <typename K>
int allow_smem(K kernel, size_t bytes) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  return e == cudaSuccess ? 0 : asb::fail("gemm_simt: shared memory %lld: %s", (long long)bytes, cudaGetErrorString(e));
}

template <typename TIn, typename TOut, int BM, int CLUSTER, bool VEC>
int launch_tile(void* out, const void* x, const void* w, const void* residual, int M, int N, int K, cudaStream_t stream) {
  const long long blocks = (long long)CLUSTER * ((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  if (blocks > 0x7fffffffLL) return asb::fail("gemm_simt: [%d, %d] exceeds the grid", M, N);
  auto kernel = tile_kernel<TIn, TOut, BM, CLUSTER, VEC>;
  if (int rc = allow_smem(kernel, Tile<BM>::kSmem)) return rc;
  asb::launch(kernel, dim3((unsigned)blocks), kThreads, Tile<BM>::kSmem, stream, (TOut*)out, (const TIn*)x, (const TIn*)w, (const TOut*)residual, M, N, K);
  return 0;
}

template <typename TIn, typename TOut>
int tiles(void* out, const void* x, const void* w, const void* residual, int M, int N, int K, cudaStream_t stream) {
  const bool vec = K % 4 == 0 && ((((uintptr_t)x) | ((uintptr_t)w)) & (4 * sizeof(TIn) - 1)) == 0;
  const bool cut = K > (kQuarters - 1) * kRun;  // a run for every block of a cluster
  // Tiles of 32 rows for up to 32 (half the multiply-adds would be padding in the other), and where they come to one block
  // an SM: a block's chain of stages is then what counts, and half as long (300 rows of 96 over 512: 9.8 us with 64 rows a
  // tile, 7.3 with 32; of 2,048 over 2,048, 64 rows: 36.3 and 34.9; just beyond one block an SM, 1,000 rows of 256 over
  // 640: 19.6 and 22.8).
  const long long blocks = (long long)(cut ? kQuarters : 1) * ((M + 31) / 32) * ((N + BN - 1) / BN);
#define ASB_TILE(BM_, C_, V_) return launch_tile<TIn, TOut, BM_, C_, V_>(out, x, w, residual, M, N, K, stream)
  if (M <= 32 || blocks <= kSMs) {
    if (cut) { if (vec) ASB_TILE(32, kQuarters, true); ASB_TILE(32, kQuarters, false); }
    if (vec) ASB_TILE(32, 1, true);
    ASB_TILE(32, 1, false);
  }
  if (cut) { if (vec) ASB_TILE(64, kQuarters, true); ASB_TILE(64, kQuarters, false); }
  if (vec) ASB_TILE(64, 1, true);
  ASB_TILE(64, 1, false);
#undef ASB_TILE
}

constexpr size_t kMostSmem = 227 * 1024;

// The rows kernel's shared memory for MR rows and a cluster of `blocks`.
size_t rows_smem(int mr, int blocks, int runs) {
  return sizeof(float) * ((size_t)kWarps * kRowStages * (kRowsN + mr) * kLd + (size_t)((runs + blocks - 1) / blocks) * mr * kRowsN);
}

template <int MR, int CLUSTER>
int launch_rows(float* out, const float* x, const float* w, const float* residual, int M, int N, int K, int w_stored, cudaStream_t stream) {
  const size_t smem = rows_smem(MR, CLUSTER, (K + kRun - 1) / kRun);
  auto kernel = rows_kernel<MR, CLUSTER>;
  if (int rc = allow_smem(kernel, smem)) return rc;
  asb::launch(kernel, dim3(CLUSTER * (unsigned)((N + kRowsN - 1) / kRowsN)), kThreads, smem, stream, out, x, w, residual, M, N, K, w_stored);
  return 0;
}

template <int MR>
int rows(float* out, const float* x, const float* w, const float* residual, int M, int N, int K, int w_stored, cudaStream_t stream) {
  // eight blocks a cluster where four would have more than eight runs each to keep the sums of
  if (K > 32 * kRun) return launch_rows<MR, 8>(out, x, w, residual, M, N, K, w_stored, stream);
  if (K > (kQuarters - 1) * kRun) return launch_rows<MR, kQuarters>(out, x, w, residual, M, N, K, w_stored, stream);
  return launch_rows<MR, 1>(out, x, w, residual, M, N, K, w_stored, stream);
}

}  // namespace

// in_dtype: element type of x and w. out_dtype: element type of out and residual (float32 out
// from bfloat16 inputs gives logits straight from the accumulator). w_stored: w was written before the stream's
// previous kernel was launched, and may be read while that kernel runs.
extern "C" int asb_gemm_simt(void* out, const void* x, const void* w, const void* residual,
                             int M, int N, int K, int in_dtype, int out_dtype, int w_stored,
                             cudaStream_t stream) {
  if (M == 0 || N == 0) return 0;
  if (K < 1) return asb::fail("gemm_simt: K = %d", K);
  if (M > 65535 * 64) return asb::fail("gemm_simt: M = %d exceeds the grid", M);
  int rc = 0;
  if (in_dtype == asb::kFloat32 && out_dtype == asb::kFloat32) {
    const bool aligned = K % 4 == 0 && ((((uintptr_t)x) | ((uintptr_t)w)) & 15) == 0;
    const int mr = M <= 4 ? 4 : (M <= 8 ? 8 : 16);
    const float* xf = (const float*)x;
    const float* wf = (const float*)w;
    const float* rf = (const float*)residual;
    if (M > 16 || !aligned || rows_smem(mr, 8, (K + kRun - 1) / kRun) > kMostSmem)
      rc = tiles<float, float>(out, x, w, residual, M, N, K, stream);
    else if (mr == 4) rc = rows<4>((float*)out, xf, wf, rf, M, N, K, w_stored, stream);
    else if (mr == 8) rc = rows<8>((float*)out, xf, wf, rf, M, N, K, w_stored, stream);
    else rc = rows<16>((float*)out, xf, wf, rf, M, N, K, w_stored, stream);
  } else if (in_dtype == asb::kBFloat16 && out_dtype == asb::kBFloat16) {
    rc = tiles<__nv_bfloat16, __nv_bfloat16>(out, x, w, residual, M, N, K, stream);
  } else if (in_dtype == asb::kBFloat16 && out_dtype == asb::kFloat32) {
    rc = tiles<__nv_bfloat16, float>(out, x, w, residual, M, N, K, stream);
  } else {
    return asb::fail("gemm_simt: unsupported dtypes in=%d out=%d", in_dtype, out_dtype);
  }
  if (rc) return rc;
  return asb::check_launch("gemm_simt");
}
