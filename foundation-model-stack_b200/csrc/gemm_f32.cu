// y[M, N] = x[M, K] . w[N, K]^T (+ bias[N]) in true float32: FFMA on the CUDA cores, no tensor-core mode,
// no reduced-precision product.  K is cut into up to RUNS runs whose length depends on K alone; an element is the sum,
// in the runs' order, of one sequential fmaf chain a run, whichever kernel makes it and whatever M is, so a row's result
// does not depend on what else is in the batch.  The runs of a tile belong to the blocks of one thread-block cluster,
// which add their sums through distributed shared memory: that many more and smaller blocks fill 148 multiprocessors
// evenly, and the shorter chains round less than one chain over all of K.
#include "common.cuh"

#include <cooperative_groups.h>

namespace {
namespace cg = cooperative_groups;
constexpr int RUNS = 8, BK = 16;

// length of a run: a multiple of 32, at least 128 (shorter ones are not worth a sum of their own)
int run_length(int K) {
  const int even = ((K + RUNS - 1) / RUNS + 31) / 32 * 32;
  return even < 128 ? 128 : even;
}
// blocks of a cluster: a power of two that covers the runs
int ranks_for(int K) {
  const int runs = (K + run_length(K) - 1) / run_length(K);
  return runs <= 1 ? 1 : runs <= 2 ? 2 : runs <= 4 ? 4 : 8;
}

template <typename... KArgs, typename... Args>
int launch_clusters(void (*kernel)(KArgs...), long long tiles, int ranks, int threads, size_t smem, cudaStream_t stream, Args... args) {
  if (tiles * ranks > 0x7fffffffLL) return fms_fail("gemm_f32: %lld tiles are more than one launch takes", tiles);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(tiles * ranks));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = ranks;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = fms_pdl_enabled() ? 2 : 1;
  cudaLaunchKernelEx(&cfg, kernel, KArgs(args)...);
  return fms_launch_status("gemm_f32");
}

typedef unsigned long long f32x2;  // two floats side by side in registers
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 swapped(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(b), "f"(a));
  return r;
}

// ---- many rows: tiles of 64 x 128, 8 x 8 elements a thread, a block a run ---------------------------------------------
// Bound by what shared memory returns to registers (128 bytes a cycle, whoever reads what: 16 words a thread and k for 64
// multiply-adds take it as long as the FMA pipe) and by issue slots, which fma.rn.f32x2 halves: two elements an
// instruction, the same roundings.  A warp's elements are four by eight lanes of two runs of four rows and of four
// columns, so that its reads of a k are 64 and 128 contiguous bytes.  The next 16 k are on their way from global memory
// (in registers) while these are multiplied.  Measured (1,100 x 6,144 x 4,096; 72 TFLOP/s is what the FMA pipe gives): 45
// TFLOP/s; one element an instruction 38; 16 x 8 elements a thread 46 (and 20% less at 40 rows); tiles of 128 x 128 43;
// the tiles of 64 x 64 with 4 x 4 elements and one chain over K that were here before 26.
constexpr int BM = 64, BN = 128, TM = 8, TILE_THREADS = BM * BN / (TM * 8);
constexpr size_t TILE_SMEM = sizeof(float) * BM * BN;  // the block's sums; before, the operands of two steps
static_assert(2 * BK * (BM + 4 + BN + 4) <= BM * BN, "operands");

__global__ void __launch_bounds__(TILE_THREADS, 4)
    gemm_f32_tile_kernel(const float* __restrict__ x, const float* __restrict__ w, const float* __restrict__ bias,
                         float* __restrict__ y, int M, int N, int K, int run_len, int ranks, int vec) {
  constexpr int THREADS = TILE_THREADS, LDX = BM + 4, LDW = BN + 4, NX = BM * 4 / THREADS, NW = BN * 4 / THREADS;
  extern __shared__ __align__(16) float sm[];
  float* xs = sm;                 // [2][BK][LDX]
  float* ws = xs + 2 * BK * LDX;  // [2][BK][LDW]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int tile = blockIdx.x / ranks, rank = blockIdx.x - tile * ranks;
  // rows vary fastest over the tiles: clusters side by side read the same rows of w
  const int tiles_m = (M + BM - 1) / BM;
  const int m0 = (tile % tiles_m) * BM, n0 = (tile / tiles_m) * BN;
  const int tm = (warp / (BN / 64)) * (4 * TM) + (lane >> 3) * 4, tn = (warp % (BN / 64)) * 64 + (lane & 7) * 4;
  const int k_begin = min(rank * run_len, K), k_end = min(k_begin + run_len, K);

  float4 px[NX], pw[NW];
  auto four = [&](const float* base, int row, int rows, int k) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (row < rows) {
      const float* p = base + (size_t)row * K + k;
      if (vec) {
        if (k < k_end) v = *reinterpret_cast<const float4*>(p);
      } else {
        if (k < k_end) v.x = p[0];
        if (k + 1 < k_end) v.y = p[1];
        if (k + 2 < k_end) v.z = p[2];
        if (k + 3 < k_end) v.w = p[3];
      }
    }
    return v;
  };
  auto fetch = [&](int k0) {
#pragma unroll
    for (int i = 0; i < NX; ++i) px[i] = four(x, m0 + (tid + i * THREADS) / 4, M, k0 + (tid & 3) * 4);
#pragma unroll
    for (int i = 0; i < NW; ++i) pw[i] = four(w, n0 + (tid + i * THREADS) / 4, N, k0 + (tid & 3) * 4);
  };
  auto put = [&](int buf) {
    float* xb = xs + buf * BK * LDX + (tid & 3) * 4 * LDX;
    float* wb = ws + buf * BK * LDW + (tid & 3) * 4 * LDW;
#pragma unroll
    for (int i = 0; i < NX; ++i) {
      const int r = (tid + i * THREADS) / 4;
      xb[r] = px[i].x;
      xb[LDX + r] = px[i].y;
      xb[2 * LDX + r] = px[i].z;
      xb[3 * LDX + r] = px[i].w;
    }
#pragma unroll
    for (int i = 0; i < NW; ++i) {
      const int r = (tid + i * THREADS) / 4;
      wb[r] = pw[i].x;
      wb[LDW + r] = pw[i].y;
      wb[2 * LDW + r] = pw[i].z;
      wb[3 * LDW + r] = pw[i].w;
    }
  };

  f32x2 acc2[TM / 2][8];  // of rows 2 i and 2 i + 1: columns j and j ^ 1
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc2[i][j] = 0;

  pdl_launch_dependents();
  pdl_wait();
  const int steps = (k_end - k_begin + BK - 1) / BK;
  if (steps > 0) {
    fetch(k_begin);
    put(0);
  }
  __syncthreads();
  for (int step = 0; step < steps; ++step) {
    const int buf = step & 1;
    if (step + 1 < steps) fetch(k_begin + (step + 1) * BK);
    const float* xb = xs + buf * BK * LDX;
    const float* wb = ws + buf * BK * LDW;
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      f32x2 a[TM / 2], b[4], c[4];
#pragma unroll
      for (int i = 0; i < TM / 4; ++i) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(xb + k * LDX + tm + 16 * i);
        a[2 * i] = v.x;
        a[2 * i + 1] = v.y;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(wb + k * LDW + tn + 32 * j);
        b[2 * j] = v.x;
        b[2 * j + 1] = v.y;
        c[2 * j] = swapped(v.x);
        c[2 * j + 1] = swapped(v.y);
      }
#pragma unroll
      for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc2[i][2 * j] = fma2(a[i], b[j], acc2[i][2 * j]);
          acc2[i][2 * j + 1] = fma2(a[i], c[j], acc2[i][2 * j + 1]);
        }
    }
    if (step + 1 < steps) put(buf ^ 1);
    __syncthreads();
  }

  float acc[TM][8];
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      unpack2(acc2[i][2 * j], acc[2 * i][2 * j], acc[2 * i + 1][2 * j + 1]);
      unpack2(acc2[i][2 * j + 1], acc[2 * i][2 * j + 1], acc[2 * i + 1][2 * j]);
    }
  const bool vec_y = (N % 4) == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
  // four number i of this thread: row i / 2, columns of its run i % 2
  auto store4 = [&](int i, float4 v) {
    const int row = i >> 1, gm = m0 + tm + (row & 3) + (row >> 2) * 16, gn = n0 + tn + (i & 1) * 32;
    if (gm >= M || gn >= N) return;
    float* p = y + (size_t)gm * N + gn;
    if (gn + 3 < N && vec_y) {
      if (!FMS_IN((size_t)gm * N + gn + 3, (size_t)M * N)) return;
      if (bias) v = make_float4(v.x + bias[gn], v.y + bias[gn + 1], v.z + bias[gn + 2], v.w + bias[gn + 3]);
      *reinterpret_cast<float4*>(p) = v;
      return;
    }
    const float e[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (gn + j < N && FMS_IN((size_t)gm * N + gn + j, (size_t)M * N)) p[j] = bias ? e[j] + bias[gn + j] : e[j];
  };
  if (ranks == 1) {
#pragma unroll
    for (int i = 0; i < 2 * TM; ++i)
      store4(i, make_float4(acc[i >> 1][(i & 1) * 4], acc[i >> 1][(i & 1) * 4 + 1], acc[i >> 1][(i & 1) * 4 + 2], acc[i >> 1][(i & 1) * 4 + 3]));
    return;
  }
  // the block's sums lie where its operands were, thread by thread
#pragma unroll
  for (int i = 0; i < 2 * TM; ++i)
    *reinterpret_cast<float4*>(sm + ((size_t)i * THREADS + tid) * 4) =
        make_float4(acc[i >> 1][(i & 1) * 4], acc[i >> 1][(i & 1) * 4 + 1], acc[i >> 1][(i & 1) * 4 + 2], acc[i >> 1][(i & 1) * 4 + 3]);
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int runs = (K + run_len - 1) / run_len, share = 2 * TM / ranks;
  for (int h = 0; h < share; ++h) {
    const int i = rank * share + h;
    float4 p[RUNS];
#pragma unroll
    for (int s = 0; s < RUNS; ++s)
      if (s < runs) p[s] = *reinterpret_cast<const float4*>(cluster.map_shared_rank(sm, s) + ((size_t)i * THREADS + tid) * 4);
    float4 v = p[0];
#pragma unroll
    for (int s = 1; s < RUNS; ++s)
      if (s < runs) v = make_float4(v.x + p[s].x, v.y + p[s].y, v.z + p[s].z, v.w + p[s].w);
    store4(i, v);
  }
  cluster.sync();  // nobody leaves while its sums are still read
}

int launch_tiles(const float* x, const float* w, const float* bias, float* y, int M, int N, int K, int vec, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_SMEM);
    if (e != cudaSuccess) return fms_fail("gemm_f32: %zu bytes of shared memory refused: %s", TILE_SMEM, cudaGetErrorString(e));
    configured = true;
  }
  const long long tiles = (long long)((M + BM - 1) / BM) * ((N + BN - 1) / BN);
  return launch_clusters(gemm_f32_tile_kernel, tiles, ranks_for(K), TILE_THREADS, TILE_SMEM, stream, x, w, bias, y, M, N, K,
                         run_length(K), ranks_for(K), vec);
}

// ---- few rows (a decode step): a warp a run ---------------------------------------------------------------------------
// Bound by the bytes of w, and next to them by what shared memory returns to registers.  A cluster owns 32 rows of w (32
// columns of y), each of its blocks is one warp with one run and a ring of its own: FEW_KT k of the 32 rows and of the
// rows of x at a time by 16-byte asynchronous copies, no barrier but the cluster's at the end.  The lanes are G by XG: a
// lane holds 32 / G rows of w and ROWS / XG rows of x, which share each other's reads (a row of w and eight of x a lane
// read 36 words for 32 multiply-adds, two and four 24).  Rows are padded to 36 floats: no bank conflicts.  Measured (8 rows, w of 28,672 x 4,096 / 4,096 x
// 14,336, L2 flushed): 114 / 71 us (4.1 / 3.3 TB/s); all runs in one block of eight warps 131 / 72; one chain over K, where a
// thread walks a row of w for two or four rows of x, as here before, 138 / 138.
constexpr int FEW_MAX_ROWS = 32, FEW_WROWS = 32, FEW_KT = 32, FEW_STRIDE = FEW_KT + 4;
template <int ROWS> constexpr int FEW_STAGES = ROWS <= 16 ? 4 : 3;
template <int ROWS> constexpr int FEW_STAGE_FLOATS = (FEW_WROWS + ROWS) * FEW_STRIDE;
template <int ROWS> constexpr size_t FEW_SMEM = (size_t)FEW_STAGES<ROWS> * FEW_STAGE_FLOATS<ROWS> * sizeof(float);

__device__ __forceinline__ void few_copy16(void* smem, const void* gmem, bool valid) {
  const int bytes = valid ? 16 : 0;  // 0: the destination is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(smem)), "l"(gmem), "r"(bytes) : "memory");
}

template <int ROWS, int G>
__global__ void __launch_bounds__(32) gemm_f32_few_rows_kernel(const float* __restrict__ x, const float* __restrict__ w,
                                                               const float* __restrict__ bias, float* __restrict__ y, int M, int N,
                                                               int K, int run_len, int ranks) {
  extern __shared__ __align__(16) float sm[];
  constexpr int STAGES = FEW_STAGES<ROWS>, STAGE = FEW_STAGE_FLOATS<ROWS>, PIECES = FEW_KT / 4;
  constexpr int R = FEW_WROWS / G, XG = 32 / G, XR = ROWS / XG;
  static_assert(R * G == FEW_WROWS && XR * XG == ROWS, "lanes");
  const int lane = threadIdx.x, group = blockIdx.x / ranks, rank = blockIdx.x - group * ranks;
  const int n0 = group * FEW_WROWS, wl = lane % G, xl = lane / G;
  const int k_begin = min(rank * run_len, K), k_end = min(k_begin + run_len, K);  // K is a multiple of 4 here
  const int steps = (k_end - k_begin + FEW_KT - 1) / FEW_KT;
  const int piece = lane % PIECES, sub = lane / PIECES;

  auto issue_w = [&](int step) {
    float* ws = sm + (step % STAGES) * STAGE;
    const int k = k_begin + step * FEW_KT + 4 * piece;
#pragma unroll
    for (int r = 0; r < FEW_WROWS; r += 32 / PIECES) {
      const int n = min(n0 + r + sub, N - 1);  // rows beyond N repeat the last one; their results are not stored
      few_copy16(ws + (r + sub) * FEW_STRIDE + 4 * piece, w + (size_t)n * K + min(k, K - 4), k < k_end);
    }
  };
  auto issue_x = [&](int step) {
    float* xs = sm + (step % STAGES) * STAGE + FEW_WROWS * FEW_STRIDE;
    const int k = k_begin + step * FEW_KT + 4 * piece;
#pragma unroll
    for (int r = 0; r < ROWS; r += 32 / PIECES) {
      const int m = r + sub;
      if (m < ROWS) few_copy16(xs + m * FEW_STRIDE + 4 * piece, x + (size_t)min(m, M - 1) * K + min(k, K - 4), m < M && k < k_end);
    }
  };

  float acc[XR][R];
#pragma unroll
  for (int i = 0; i < XR; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) acc[i][j] = 0.f;
  // w may be what the kernel in front makes: before the wait it is only asked into the second-level cache
  for (int s = 0; s < STAGES - 1; ++s)
    if (s < steps) prefetch_l2(w + (size_t)min(n0 + lane, N - 1) * K + k_begin + s * FEW_KT);
  pdl_launch_dependents();
  pdl_wait();
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < steps) {
      issue_w(s);
      issue_x(s);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  }
  for (int step = 0; step < steps; ++step) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncwarp();  // every lane's copies of this stage are there, and all are done with the one that is filled next
    if (step + STAGES - 1 < steps) {
      issue_w(step + STAGES - 1);
      issue_x(step + STAGES - 1);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");  // an empty group keeps the count of groups in step
    const float* ws = sm + (step % STAGES) * STAGE + wl * FEW_STRIDE;
    const float* xs = sm + (step % STAGES) * STAGE + (FEW_WROWS + xl) * FEW_STRIDE;
#pragma unroll(ROWS <= 8 ? PIECES : 2)
    for (int u = 0; u < PIECES; ++u) {  // beyond the run the stage holds zeros: a chain sees terms of 0 x 0
      float4 wv[R];
#pragma unroll
      for (int j = 0; j < R; ++j) wv[j] = *reinterpret_cast<const float4*>(ws + j * G * FEW_STRIDE + 4 * u);
#pragma unroll
      for (int i = 0; i < XR; ++i) {
        const float4 xv = *reinterpret_cast<const float4*>(xs + i * XG * FEW_STRIDE + 4 * u);
#pragma unroll
        for (int j = 0; j < R; ++j) {
          acc[i][j] = fmaf(xv.x, wv[j].x, acc[i][j]);
          acc[i][j] = fmaf(xv.y, wv[j].y, acc[i][j]);
          acc[i][j] = fmaf(xv.z, wv[j].z, acc[i][j]);
          acc[i][j] = fmaf(xv.w, wv[j].w, acc[i][j]);
        }
      }
    }
  }
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncwarp();  // the ring is free: the run's sums go where it was, [ROWS][32]
#pragma unroll
  for (int i = 0; i < XR; ++i)
#pragma unroll
    for (int j = 0; j < R; ++j) sm[(i * XG + xl) * FEW_WROWS + j * G + wl] = acc[i][j];
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  const int runs = (K + run_len - 1) / run_len, n = n0 + lane;
  const float b = bias && n < N ? bias[n] : 0.f;
  for (int m = rank; m < min(M, ROWS); m += ranks) {
    float p[RUNS];
#pragma unroll
    for (int s = 0; s < RUNS; ++s)
      if (s < runs) p[s] = cluster.map_shared_rank(sm, s)[m * FEW_WROWS + lane];
    float v = p[0];
#pragma unroll
    for (int s = 1; s < RUNS; ++s)
      if (s < runs) v += p[s];
    if (n < N && FMS_IN((size_t)m * N + n, (size_t)M * N)) y[(size_t)m * N + n] = bias ? v + b : v;
  }
  cluster.sync();  // nobody leaves while its sums are still read
}

template <int ROWS, int G>
int launch_few_rows(const float* x, const float* w, const float* bias, float* y, int M, int N, int K, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_rows_kernel<ROWS, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FEW_SMEM<ROWS>);
    if (e != cudaSuccess) return fms_fail("gemm_f32: %zu bytes of shared memory refused: %s", FEW_SMEM<ROWS>, cudaGetErrorString(e));
    configured = true;
  }
  return launch_clusters(gemm_f32_few_rows_kernel<ROWS, G>, (N + FEW_WROWS - 1) / FEW_WROWS, ranks_for(K), 32, FEW_SMEM<ROWS>, stream, x, w,
                         bias, y, M, N, K, run_length(K), ranks_for(K));
}
}  // namespace

FMS_API int fms_gemm_f32(const float* x, const float* w, const float* bias, float* y, int M, int N, int K,
                         cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) return fms_fail("gemm_f32: K %d", K);
  // 16-byte loads only where every row starts on 16 bytes; else the tiles take one value at a time, in the same order
  const bool vec = K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15) == 0;
  // from 33 rows on the tiles of 64 rows are the faster ones (32 rows of 28,672 x 4,096: 251 against 330 us)
  if (M <= FEW_MAX_ROWS && vec) {
    if (M <= 1) return launch_few_rows<1, 32>(x, w, bias, y, M, N, K, stream);
    if (M <= 2) return launch_few_rows<2, 16>(x, w, bias, y, M, N, K, stream);
    if (M <= 4) return launch_few_rows<4, 16>(x, w, bias, y, M, N, K, stream);
    if (M <= 8) return launch_few_rows<8, 16>(x, w, bias, y, M, N, K, stream);
    if (M <= 16) return launch_few_rows<16, 8>(x, w, bias, y, M, N, K, stream);
    return launch_few_rows<32, 8>(x, w, bias, y, M, N, K, stream);
  }
  return launch_tiles(x, w, bias, y, M, N, K, vec, stream);
}
