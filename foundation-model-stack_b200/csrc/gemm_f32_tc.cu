// y[M, N] = x[M, K] . w[N, K]^T (+ bias[N]) in float32 for large matrices, on the tensor cores without losing a bit of the
// operands: a float32 value is the sum of three bfloat16 values (8 + 8 + 8 bits of mantissa: nearest, nearest of the rest, the
// rest), and six of the nine products of parts hold everything above 2^-26 of a product.  tcgen05.mma adds them in tensor memory.
//
// Its sums there are cut off, not rounded: 8.5e-9 of an element for every 16 k that go into one accumulator, always towards
// zero (measured: 6.4e-8 after 64 k, 4.7e-7 after 512).  So an accumulator takes 32 k only, the five small products first (they
// are 2^-8 of the sum, so is what they lose), then the large one; what it holds goes through registers into the run's sum, rounded
// to nearest.  Runs of K (run_length, a function of K alone) are added in their order at the end.  An element is thus one fixed
// sequence of operations whatever M is and wherever its row lies: a row's result does not depend on the rows beside it.  Error
// against 64 bits for normal values, K = 1,024 / 4,096 / 14,336: 5.6e-8 / 1.0e-7 / 1.9e-7 (multiply-adds of gemm_f32.cu 2.1e-7 /
// 4.1e-7 / 7.6e-7).
//
// x and w are split times 2^SPLIT_SCALE, and sums are scaled back when they are complete: parts of the smallest float32 values are
// normal bfloat16 values then, and sums of products down to 2^-174 normal float32 ones (additions in memory flush what is smaller, the
// others do so too).  Values that are not finite or beyond 2^30 do not split (products of parts of both signs could overflow where the
// sum does not): a row of x or of w with such values is noted while it is split, and its elements are made by multiply-adds instead, by
// persistent blocks once all their tiles are done (the other warps' waits are bounded, and many such rows take long).
//
// x is split by a kernel of its own (it is read by every tile of w's rows; 27 MB written for 1,100 rows of 4,096).  w is split on
// its way, since writing it split would take longer than the product reads it.  A block owns 128 rows of w (the instruction's
// rows) and nt rows of x (its columns):
//   epilogue    eight warps.  Each owns 32 lanes of tensor memory and half of the columns and keeps the run's sums in registers
//   mma, TMA    a warp each: one lane issues the products of a step, one brings the parts of x
//   splitting   4 or 16 warps.  Read the next rows of w into registers while they split these, and store the parts into a ring of
//               stages (rows of 64 bytes, 64-byte swizzle).  Plain loads: they go through registers anyway
// A step fills two accumulators (nt 256: one, for there is no more tensor memory), while the epilogue drains those of the step
// before: handing over costs 600 cycles, whatever a step holds (w of 4,096 x 14,336 and 64 rows: 124 us by single accumulators, 91 so).
// Few tiles: the blocks of a cluster take a run each and add their sums through distributed shared memory.  Many: persistent
// blocks take all runs of a tile and add a run's sums to y where it lies, which nobody waits for; the last run's meet them in registers.
// Measured (us, CUDA cores / here; six products of bfloat16 at the tensor cores' rate would be 279 TFLOP/s): 1,100 rows of 6,144 x 4,096
// 1,217 / 304 (182 TFLOP/s), 4,096 x 4,096 824 / 241; 2,048 of 4,096 x 14,336 4,870 / 1,183 (203); 64 of 28,672 x 4,096 645 / 200.  The scale
// costs 1% of that, the last run's way through registers 1 to 3%.
// What is left: tiles of 128 x 256 read 96 bytes of shared memory a cycle for the products and 48 for what is brought in, of 128;
// the last round of tiles; adding a run to y stalls the products by a tenth.
#include <cooperative_groups.h>
#include <cuda.h>

#include <type_traits>

#include "common.cuh"

namespace {
namespace cg = cooperative_groups;
#include "tcgen05.cuh"
#include "split_f32.cuh"

constexpr int RUNS = 4, BK = 32, WROWS = 128;
constexpr int SPLIT_UP_TO = 30 + SPLIT_SCALE, MOST_K = 1 << 18;  // 2^18 products of two operands of 2^54 are below 2^127
constexpr float UNSCALE = power_of_two(-2 * SPLIT_SCALE);
constexpr int OTHER_REGS = 48;  // registers of the threads that neither split nor drain, where the kinds differ
constexpr int W_PART = WROWS * BK * 2;  // bytes of one part of a stage's rows of w

int run_length(int K) {
  const int even = ((K + RUNS - 1) / RUNS + 63) / 64 * 64;
  return even < 128 ? 128 : even;
}
int ranks_for(int K) {
  const int runs = (K + run_length(K) - 1) / run_length(K);
  return runs <= 1 ? 1 : runs <= 2 ? 2 : 4;
}

// NT: most rows of x a block takes.  SUB: accumulators (32 k each) that a step fills.  CONV, EPI: warps that split and that drain.
// DEPTH: steps of w that a splitting warp has on their way, AHEAD: steps before those for which w is asked into the second-level cache.
// CONV_REGS, EPI_REGS: registers of a thread of either kind, 0: as launched
template <int NT_, int SUB_, int CONV_, int EPI_, int STAGES_, int DEPTH_, int AHEAD_, int CONV_REGS_, int EPI_REGS_>
struct Shape {
  static constexpr int NT = NT_, SUB = SUB_, CONV = CONV_, EPI = EPI_, STAGES = STAGES_, DEPTH = DEPTH_, AHEAD = AHEAD_;
  static constexpr int CONV_REGS = CONV_REGS_, EPI_REGS = EPI_REGS_;
  static constexpr int PIECE = NT > 128 ? 32 : 16;           // columns that a warp reads at a time
  static constexpr int LAST = NT > 64 ? 16 : 8;              // sums of earlier runs that a thread reads at a time with the last
  static constexpr int SPAN = CONV * 8, UNITS = WROWS / SPAN;  // rows of w that the splitting warps take at a time, and how often
  static constexpr int MMA = EPI, TMA = EPI + 1, CONV_AT = EPI + 4;  // warps: first those that drain
  static constexpr int THREADS = 32 * (CONV_AT + CONV), COLS = NT / (EPI / 4);
  static constexpr int STEP = SUB * BK, STAGE = 3 * (WROWS + NT) * STEP * 2, TMEM = 2 * SUB * NT;
  static constexpr size_t SMEM = (size_t)STAGES * STAGE + 1024;
  static_assert((size_t)NT * WROWS * 4 <= (size_t)STAGES * STAGE, "the run's sums lie where the stages were");
  static_assert(EPI_REGS == 0 || (CONV % 4 == 0 && EPI % 4 == 0 && 32 * (CONV_REGS * CONV + OTHER_REGS * 4 + EPI_REGS * EPI) <= 65536), "registers");
};

struct Product {
  const float *x, *w, *bias;
  float* y;
  const unsigned char* x_kinds;  // of every row of x (row_kind)
  unsigned char* w_kinds;        // of every row of w, for a block's own use
  int M, N, K, run_len, ranks, nt, tiles_x, tiles, vec;
  int* error_flag;
};

// One 128 x nt x 16 product.  Operands by the low words of their shared-memory descriptors: K-major rows of 64 bytes with the 64-byte
// swizzle, groups of 8 rows 512 bytes apart (the high word, made here so that no pair of registers is kept for each of them)
__device__ __forceinline__ uint32_t operand(uint32_t smem_addr) { return ((smem_addr >> 4) & 0x3FFF) | (1u << 16); }
template <bool ACCUMULATE>
__device__ __forceinline__ void umma_64(uint32_t tmem_d, uint32_t a, uint32_t b, uint32_t idesc) {
  asm volatile(
      "{\n.reg .pred p;\n.reg .b64 da, db;\nsetp.ne.b32 p, %4, 0;\nmov.b64 da, {%1, %5};\nmov.b64 db, {%2, %5};\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, {%6, %6, %6, %6}, p;\n}\n" ::"r"(tmem_d),
      "r"(a), "r"(b), "r"(idesc), "n"(ACCUMULATE ? 1 : 0), "r"((512u >> 4) | (1u << 14) | (4u << 29)), "r"(0u)
      : "memory");
}
// If wanted, *at = v, or *at += v where it lies, rounded to nearest, subnormal values as zeros; only this thread writes there, so its
// additions happen in their order.  Under a predicate: a branch a column would cost more than the store
template <bool ADD>
__device__ __forceinline__ void put_to(float* at, float v, bool wanted) {
  if constexpr (ADD)
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %2, 0;\n@p red.relaxed.gpu.global.add.f32 [%0], %1;\n}\n" ::"l"(at), "f"(v), "r"((int)wanted) : "memory");
  else
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %2, 0;\n@p st.global.f32 [%0], %1;\n}\n" ::"l"(at), "f"(v), "r"((int)wanted) : "memory");
}

// what additions in memory have made of *at, if wanted, else 0
__device__ __forceinline__ float sum_at(const float* at, bool wanted) {
  float v = 0.f;
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %2, 0;\n@p ld.relaxed.gpu.global.f32 %0, [%1];\n}\n" : "+f"(v) : "l"(at), "r"((int)wanted) : "memory");
  return v;
}
// a + b as additions in memory make it
__device__ __forceinline__ float add_runs(float a, float b) {
  float r;
  asm("add.rn.ftz.f32 %0, %1, %2;\n" : "=f"(r) : "f"(a), "f"(b));
  return r;
}

// Eight values from `at` on, if they are wanted; `left`: so many of them exist, the others are zeros.  vec: 2 rows of 32 bytes alignment, 1 of
// 16, 0 of 4.  FAST: vec 2 and nothing missing; one instruction under a predicate, so that its registers stay where they are
template <bool FAST>
__device__ __forceinline__ void load8(float* v, const float* at, int vec, int left, bool wanted) {
  if constexpr (FAST) {
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %9, 0;\n@p ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n}\n"
                 : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7])
                 : "l"(at), "r"((int)wanted));
  } else if (wanted) {
    if (vec && left >= 8) {
      const float4 a = *reinterpret_cast<const float4*>(at), b = *reinterpret_cast<const float4*>(at + 4);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
      v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = j < left ? at[j] : 0.f;
    }
  }
}

// A wait of a whole warp: its lanes look for themselves, so one can see the phase complete when another sees that a role gave up, and
// what follows takes all of them
__device__ __forceinline__ bool warp_waits(void* bar, uint32_t parity, volatile int* failed) {
  return __all_sync(0xffffffffu, wait_or_abort(bar, parity, failed));
}

// asks for a run of bytes (16-byte aligned, a multiple of 16) to be brought into the second-level cache
__device__ __forceinline__ void prefetch_l2_run(const void* p, unsigned bytes) {
  asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;\n" ::"l"(p), "r"(bytes) : "memory");
}

// an element one of whose rows does not split, by a warp: every lane its share of k, the lanes' sums in a fixed order
__device__ __forceinline__ float whole_element(const float* __restrict__ x, const float* __restrict__ w, int K, int lane) {
  float v = 0.f;
#pragma unroll 4
  for (int k = lane; k < K; k += 32) v = fmaf(x[k], w[k], v);
  return warp_sum(v);
}

// x as three matrices of bfloat16 parts [3][M][pitch], zeros behind K, and its rows' kinds: a block a row
__global__ void __launch_bounds__(256) split_rows_kernel(const float* __restrict__ x, uint4* __restrict__ parts, unsigned char* __restrict__ kinds,
                                                         int M, int K, int pitch, int vec) {
  pdl_launch_dependents();
  pdl_wait();
  const int m = blockIdx.x;
  uint32_t most = 0;
  for (int k = threadIdx.x * 8; k < pitch; k += blockDim.x * 8) {
    const float* at = x + (size_t)m * K + k;
    float v[8];
    if (vec && k + 8 <= K) {
      const float4 a = *reinterpret_cast<const float4*>(at), b = *reinterpret_cast<const float4*>(at + 4);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = k + j < K ? at[j] : 0.f;
    }
    uint4 hi, mid, lo;
    split8<SPLIT_SCALE>(v, &hi, &mid, &lo, most);
    const size_t part = (size_t)M * (pitch / 8), to = (size_t)m * (pitch / 8) + k / 8;
    if (!FMS_IN(to, part)) continue;
    parts[to] = hi;
    parts[part + to] = mid;
    parts[2 * part + to] = lo;
  }
  const unsigned char kind = row_kind<SPLIT_UP_TO>(most);
  const int any = __syncthreads_or(kind != 0), none = __syncthreads_or(kind == 2);
  if (threadIdx.x == 0) kinds[m] = none ? 2 : any ? 1 : 0;
}

template <typename S>
__global__ void __launch_bounds__(S::THREADS, 1) gemm_f32_split_kernel(const Product p, const __grid_constant__ CUtensorMap map_x) {
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)smem_unaligned + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full[S::STAGES], empty[S::STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int failed_flag, whole_any;  // whole_any: some row of this block's run may have to stay whole
  __shared__ unsigned char w_kinds[2][WROWS];  // by the parity of the block's tile
  volatile int* failed = &failed_flag;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int x_part = p.nt * BK * 2, sub_bytes = 3 * (W_PART + x_part), stage_bytes = S::SUB * sub_bytes;
  const bool alone = p.ranks == 1;
  const int rank = alone ? 0 : (int)(blockIdx.x % p.ranks);
  const int first_tile = alone ? (int)blockIdx.x : (int)(blockIdx.x / p.ranks), tile_step = alone ? (int)gridDim.x : p.tiles;
  const int k_begin = alone ? 0 : min(rank * p.run_len, p.K), k_end = alone ? p.K : min(k_begin + p.run_len, p.K);
  const int steps = (k_end - k_begin + S::STEP - 1) / S::STEP;

  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    failed_flag = 0;
    whole_any = 0;
    for (int s = 0; s < S::STAGES; ++s) {
      mbar_init(&full[s], S::CONV + 1);
      mbar_init(&empty[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&acc_full[a], 1);
      mbar_init(&acc_empty[a], S::EPI);
    }
    mbar_fence_init();
  }
  if (warp == S::MMA) tmem_alloc(&tmem_slot, S::TMEM);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;

  if (warp >= S::CONV_AT) {
    if constexpr (S::CONV_REGS > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(S::CONV_REGS > 0 ? S::CONV_REGS : 24));
    const int member = warp - S::CONV_AT;
    const int row = member * 8 + (lane >> 2), kk = (lane & 3) * 8;  // of every SPAN rows
    // bits 4 and 5 of a place within the part are crossed with bits 7 and 8
    unsigned char* const to = ring + row * 64 + (((lane & 3) ^ ((row >> 1) & 3)) << 4);
    float v[S::DEPTH][S::UNITS][S::SUB][8] = {};
    uint32_t most[S::UNITS];
    const float* at[S::UNITS];
    int load_tile = first_tile, load_step = 0;  // the step that is asked for next
    auto aim = [&]() {  // rows behind the last repeat it; what they give is not stored
#pragma unroll
      for (int u = 0; u < S::UNITS; ++u)
        at[u] = p.w + (size_t)min(load_tile / p.tiles_x * WROWS + u * S::SPAN + row, p.N - 1) * p.K + k_begin + kk;
    };
    auto loaded = [&]() {  // on to the next step
      if (++load_step < steps) {
#pragma unroll
        for (int u = 0; u < S::UNITS; ++u) at[u] += S::STEP;
      } else {
        load_step = 0;
        load_tile += tile_step;
        if (load_tile < p.tiles) aim();
      }
    };
    // for the bounds-checked build: what is read of a row of w lies in the matrix
    auto inside = [&](const float* from, int left) { return left <= 0 || FMS_IN(from - p.w + min(left, 8) - 1, (size_t)p.N * p.K); };
    if (first_tile < p.tiles) {  // w may be what the kernel in front makes: only asked for
      const int n = first_tile / p.tiles_x * WROWS + member * 32 + lane;
      for (int s = 0; s < S::DEPTH; ++s)
        for (int k = k_begin + s * S::STEP; k < min(k_begin + (s + 1) * S::STEP, k_end); k += BK)
          if (member < WROWS / 32 && n < p.N) prefetch_l2(p.w + (size_t)n * p.K + k);
    }
    pdl_wait();
    const bool active = first_tile < p.tiles && steps > 0;
    const int n_tiles = first_tile < p.tiles ? (p.tiles - first_tile + tile_step - 1) / tile_step : 0, total = n_tiles * steps;
    // The whole loop for either kind of load: where one follows the other in it, what is loaded is moved, and so waited for, at once
    auto work = [&](auto kind) {
      constexpr bool fast = decltype(kind)::value;
      if (active) {
        aim();
#pragma unroll
        for (int d = 0; d < S::DEPTH; ++d)
          if (load_tile < p.tiles) {
#pragma unroll
            for (int u = 0; u < S::UNITS; ++u)
#pragma unroll
              for (int h = 0; h < S::SUB; ++h) {
                const int left = k_end - (k_begin + load_step * S::STEP + h * BK + kk);
                load8<fast>(v[d][u][h], at[u] + h * BK, p.vec, left, inside(at[u] + h * BK, left));
              }
            loaded();
          }
      }
#pragma unroll
      for (int u = 0; u < S::UNITS; ++u) most[u] = 0;
      int i = 0, turn = 0, s = 0, round = 1;  // round: parity of the stage's phase
      bool go = true;
      for (int it0 = 0; it0 < total && go; it0 += S::DEPTH) {
#pragma unroll
        for (int d = 0; d < S::DEPTH; ++d) {
          if (it0 + d >= total) break;
          go = warp_waits(&empty[s], round, failed);
          if (!go) break;
          if (active) {
            unsigned char* const stage = to + s * stage_bytes;
            const int left = k_end - (k_begin + load_step * S::STEP + kk);
            const bool more = load_tile < p.tiles;
#pragma unroll
            for (int u = 0; u < S::UNITS; ++u) {
#pragma unroll
              for (int h = 0; h < S::SUB; ++h) {
                uint4 hi, mid, lo;
                split8<SPLIT_SCALE>(v[d][u][h], &hi, &mid, &lo, most[u]);
                unsigned char* const place = stage + h * sub_bytes + u * S::SPAN * 64;
                *reinterpret_cast<uint4*>(place) = hi;
                *reinterpret_cast<uint4*>(place + W_PART) = mid;
                *reinterpret_cast<uint4*>(place + 2 * W_PART) = lo;
                load8<fast>(v[d][u][h], at[u] + h * BK, p.vec, left - h * BK, more && inside(at[u] + h * BK, left - h * BK));
              }
            }
            if (more) {
              // a row's values of a step are one run of bytes
              if (S::AHEAD > 0 && fast && (lane & 3) == 0 && load_step + S::AHEAD < steps) {
#pragma unroll
                for (int u = 0; u < S::UNITS; ++u) prefetch_l2_run(at[u] + S::AHEAD * S::STEP, S::STEP * 4);
              }
              loaded();
            }
            if (i + 1 == steps) {
#pragma unroll
              for (int u = 0; u < S::UNITS; ++u) {
                uint32_t m = most2(most[u], __shfl_xor_sync(0xffffffffu, most[u], 1));
                m = most2(m, __shfl_xor_sync(0xffffffffu, m, 2));
                if ((lane & 3) == 0) w_kinds[turn][u * S::SPAN + row] = row_kind<SPLIT_UP_TO>(m);
                most[u] = 0;
              }
            }
            fence_proxy_async();
            __syncwarp();
          }
          if (lane == 0) mbar_arrive(&full[s]);
          if (++i == steps) {
            i = 0;
            turn ^= 1;
          }
          if (++s == S::STAGES) {
            s = 0;
            round ^= 1;
          }
        }
      }
    };
    if (p.vec == 2 && (k_end - k_begin) % S::STEP == 0) work(std::true_type());
    else work(std::false_type());
  } else if (warp > S::MMA) {
    if constexpr (S::EPI_REGS > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(OTHER_REGS));
    if (warp == S::TMA && elect_one()) {
      pdl_wait();
      int it = 0;
      for (int tile = first_tile; tile < p.tiles && !*failed; tile += tile_step) {
        const int x0 = tile % p.tiles_x * p.nt;
        for (int i = 0; i < steps; ++i, ++it) {
          const int s = it % S::STAGES;
          if (!wait_or_abort(&empty[s], ((it / S::STAGES) & 1) ^ 1, failed)) break;
          mbar_arrive_expect_tx(&full[s], S::SUB * 3 * x_part);
          for (int h = 0; h < S::SUB; ++h)
            for (int q = 0; q < 3; ++q)  // rows behind x's last are the next part's: columns that nobody stores
              tma_load_2d(ring + (size_t)s * stage_bytes + h * sub_bytes + 3 * W_PART + q * x_part, &map_x, k_begin + i * S::STEP + h * BK, q * p.M + x0, &full[s]);
        }
      }
    }
  } else if (warp == S::MMA) {
    if constexpr (S::EPI_REGS > 0) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;\n" ::"n"(OTHER_REGS));
    if (elect_one()) {
      const int n_tiles = first_tile < p.tiles ? (p.tiles - first_tile + tile_step - 1) / tile_step : 0, total = n_tiles * steps;
      const uint32_t idesc = umma_idesc(WROWS, p.nt);
      auto ready = [&](int it) {  // the accumulators are drained and the stage is filled
        return wait_or_abort(&acc_empty[it & 1], ((it >> 1) & 1) ^ 1, failed) && wait_or_abort(&full[it % S::STAGES], (it / S::STAGES) & 1, failed);
      };
      bool go = total > 0 && ready(0);
      for (int it = 0; go; ++it) {
        bool next = false;
        const int s = it % S::STAGES;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < S::SUB; ++h) {
          // parts (of w, of x): the small products of both 16 k, then the large ones.  32 bytes of a row are two units of a descriptor
          const uint32_t at = smem_u32(ring + (size_t)s * stage_bytes + h * sub_bytes), d = tmem + ((it & 1) * S::SUB + h) * S::NT, xq = x_part >> 4;
          const uint32_t w = operand(at), x = operand(at + 3 * W_PART);
          constexpr uint32_t WQ = W_PART >> 4;
          umma_64<false>(d, w + 2 * WQ, x, idesc);
          umma_64<true>(d, w, x + 2 * xq, idesc);
          umma_64<true>(d, w + WQ, x + xq, idesc);
          umma_64<true>(d, w + WQ, x, idesc);
          umma_64<true>(d, w, x + xq, idesc);
          umma_64<true>(d, w + 2 * WQ + 2, x + 2, idesc);
          umma_64<true>(d, w + 2, x + 2 * xq + 2, idesc);
          umma_64<true>(d, w + WQ + 2, x + xq + 2, idesc);
          umma_64<true>(d, w + WQ + 2, x + 2, idesc);
          umma_64<true>(d, w + 2, x + xq + 2, idesc);
          // the wait for the next step while these products are still on their way
          if (h == S::SUB - 1) next = it + 1 < total && ready(it + 1);
          umma_64<true>(d, w, x, idesc);
          umma_64<true>(d, w + 2, x + 2, idesc);
        }
        tc_commit(&empty[s]);
        tc_commit(&acc_full[it & 1]);
        go = next;
      }
    }
  } else {
    if constexpr (S::EPI_REGS > 0) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;\n" ::"n"(S::EPI_REGS > 0 ? S::EPI_REGS : 24));
    const int e = warp, quarter = warp & 3, cols = p.nt / (S::EPI / 4), col0 = (e >> 2) * cols;
    const int my_row = quarter * 32 + lane;
    pdl_wait();
    float acc[S::COLS];
    int it = 0, turn = 0;
    bool some_whole = false, go = true;
    for (int tile = first_tile; tile < p.tiles && go; tile += tile_step, turn ^= 1) {
      const int w0 = tile / p.tiles_x * WROWS, x0 = tile % p.tiles_x * p.nt, n = w0 + my_row;
#pragma unroll
      for (int c = 0; c < S::COLS; ++c) acc[c] = 0.f;
      int run_end = alone ? p.run_len / S::STEP : steps;
      bool first_run = true;
      for (int i = 0; i < steps; ++i, ++it) {
        go = warp_waits(&acc_full[it & 1], (it >> 1) & 1, failed);
        if (!go) break;
        tc_fence_after();
#pragma unroll
        for (int h = 0; h < S::SUB; ++h) {
          const uint32_t from = tmem + ((it & 1) * S::SUB + h) * S::NT + col0 + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
          for (int c = 0; c < S::COLS; c += S::PIECE)
            if (c < cols) {
              float t[S::PIECE];
              if constexpr (S::PIECE == 32) tmem_load_32(from + c, t);
              else tmem_load_16(from + c, t);
#pragma unroll
              for (int j = 0; j < S::PIECE; ++j) acc[c + j] += t[j];
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&acc_empty[it & 1]);
        if (alone && (i + 1 == run_end || i + 1 == steps)) {  // the run is complete: to those before it
          const bool end = i + 1 == steps;
          const float b = end && p.bias && n < p.N ? p.bias[n] : 0.f;
          float* at = p.y + (size_t)(x0 + col0) * p.N + n;
          const int left = n < p.N ? min(cols, p.M - (x0 + col0)) : 0;
          if (end) {
#pragma unroll
            for (int c0 = 0; c0 < S::COLS; c0 += S::LAST) {
              float before[S::LAST];
              float* from = at;
#pragma unroll
              for (int j = 0; j < S::LAST; ++j) {
                before[j] = sum_at(from, !first_run && c0 + j < left && FMS_IN(from - p.y, (size_t)p.M * p.N));
                from += p.N;
                asm volatile("" : "+l"(from));  // one column after the other: no addresses kept for all of them
              }
#pragma unroll
              for (int j = 0; j < S::LAST; ++j) {
                put_to<false>(at, __fadd_rn(__fmul_rn(add_runs(before[j], acc[c0 + j]), UNSCALE), b), c0 + j < left && FMS_IN(at - p.y, (size_t)p.M * p.N));
                at += p.N;
                asm volatile("" : "+l"(at));
              }
            }
          } else if (first_run) {
#pragma unroll
            for (int c = 0; c < S::COLS; ++c) {
              put_to<false>(at, acc[c], c < left && FMS_IN(at - p.y, (size_t)p.M * p.N));
              at += p.N;
              asm volatile("" : "+l"(at));
            }
          } else {
#pragma unroll
            for (int c = 0; c < S::COLS; ++c) {
              put_to<true>(at, acc[c], c < left && FMS_IN(at - p.y, (size_t)p.M * p.N));
              at += p.N;
              asm volatile("" : "+l"(at));
            }
          }
#pragma unroll
          for (int c = 0; c < S::COLS; ++c) acc[c] = 0.f;
          first_run = false;
          run_end += p.run_len / S::STEP;
          if (end) {
            bool any = false;
            for (int j = lane; j < WROWS; j += 32) any |= w_kinds[turn][j] != 0;
            for (int j = lane; j < min(p.nt, p.M - x0); j += 32) any |= p.x_kinds[x0 + j] != 0;
            some_whole |= __any_sync(0xffffffffu, any) != 0;
            if (n < p.N && FMS_IN(n, p.N)) p.w_kinds[n] = w_kinds[turn][my_row];  // the same from every block that has the row
          }
        }
      }
    }
    // the rows that do not split, when no warp waits for this one any more
    for (int tile = some_whole && go ? first_tile : p.tiles; tile < p.tiles; tile += tile_step) {
      const int w0 = tile / p.tiles_x * WROWS, x0 = tile % p.tiles_x * p.nt, n = w0 + my_row;
      const unsigned kind_w = n < p.N ? p.w_kinds[n] : 0;
      const float b = p.bias && n < p.N ? p.bias[n] : 0.f;
      for (int c = 0; c < cols && x0 + col0 + c < p.M; ++c) {
        const int m = x0 + col0 + c;
        const unsigned kind = max(kind_w, (unsigned)p.x_kinds[m]);
        if (n < p.N && kind == 2) p.y[(size_t)m * p.N + n] = NAN;
        for (unsigned rows = __ballot_sync(0xffffffffu, n < p.N && kind == 1); rows; rows &= rows - 1) {
          const int r = __ffs(rows) - 1;
          const float v = whole_element(p.x + (size_t)m * p.K, p.w + (size_t)(w0 + quarter * 32 + r) * p.K, p.K, lane);
          if (lane == r) p.y[(size_t)m * p.N + n] = v + b;
        }
      }
    }
    if (!alone) {  // every step's mma are done: the run's sums lie where the stages were, [nt][128]
      float* own = reinterpret_cast<float*>(ring);
      if (steps > 0) {
#pragma unroll
        for (int c = 0; c < S::COLS; ++c)
          if (c < cols) own[(col0 + c) * WROWS + my_row] = acc[c];
        const int x0 = first_tile % p.tiles_x * p.nt;
        bool any = false;
        for (int j = lane; j < WROWS; j += 32) any |= w_kinds[0][j] != 0;
        for (int j = lane; j < min(p.nt, p.M - x0); j += 32) any |= p.x_kinds[x0 + j] != 0;
        if (__any_sync(0xffffffffu, any) && lane == 0) whole_any = 1;
      }
      __syncwarp();
      cluster_sync_all();
      cg::cluster_group cluster = cg::this_cluster();
      const int runs = (p.K + p.run_len - 1) / p.run_len, row = lane * 4, n = first_tile / p.tiles_x * WROWS + row;
      const int x0 = first_tile % p.tiles_x * p.nt;
      uint32_t sums[RUNS];
      bool any = false;
#pragma unroll
      for (int s = 0; s < RUNS; ++s)
        if (s < runs) {
          asm("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(sums[s]) : "r"(smem_u32(ring) + row * 4), "r"(s));
          any |= *cluster.map_shared_rank(&whole_any, s) != 0;
        }
      const bool four = p.N % 4 == 0 && ((uintptr_t)p.y & 15) == 0;
      // a warp a column, four rows of w a lane
      for (int c = warp * p.ranks + rank; c < p.nt && x0 + c < p.M; c += S::EPI * p.ranks) {
        float4 t[RUNS];
#pragma unroll
        for (int s = 0; s < RUNS; ++s)
          if (s < runs)
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(t[s].x), "=f"(t[s].y), "=f"(t[s].z), "=f"(t[s].w) : "r"(sums[s] + c * WROWS * 4));
        float4 q = t[0];
#pragma unroll
        for (int s = 1; s < RUNS; ++s)
          if (s < runs) q = make_float4(add_runs(q.x, t[s].x), add_runs(q.y, t[s].y), add_runs(q.z, t[s].z), add_runs(q.w, t[s].w));
        float v[4] = {__fmul_rn(q.x, UNSCALE), __fmul_rn(q.y, UNSCALE), __fmul_rn(q.z, UNSCALE), __fmul_rn(q.w, UNSCALE)};
        float* const at = p.y + (size_t)(x0 + c) * p.N + n;
        if (any) {
          const unsigned kind_x = p.x_kinds[x0 + c];
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            unsigned kind = kind_x;
            for (int s = 0; s < runs; ++s) kind = max(kind, (unsigned)cluster.map_shared_rank(w_kinds[0], s)[row + j]);
            if (kind == 2) v[j] = NAN;
            unsigned rows = __ballot_sync(0xffffffffu, n + j < p.N && kind == 1);
            for (; rows; rows &= rows - 1) {
              const int r = __ffs(rows) - 1;
              const float t = whole_element(p.x + (size_t)(x0 + c) * p.K, p.w + (size_t)(n + j + (r - lane) * 4) * p.K, p.K, lane);
              if (lane == r) v[j] = t;
            }
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (n + j < p.N) v[j] = __fadd_rn(v[j], p.bias ? p.bias[n + j] : 0.f);
        if (four && n + 3 < p.N) {
          if (FMS_IN(at + 3 - p.y, (size_t)p.M * p.N)) *reinterpret_cast<float4*>(at) = make_float4(v[0], v[1], v[2], v[3]);
        } else {
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (n + j < p.N && FMS_IN(at + j - p.y, (size_t)p.M * p.N)) at[j] = v[j];
        }
      }
    }
    tc_fence_before();
  }
  if (warp >= S::EPI) {
    __syncwarp();
    if (!alone) cluster_sync_all();
  }
  __syncthreads();
  if (warp == S::MMA) {
    tc_fence_after();
    tmem_dealloc(tmem, S::TMEM);
  }
  if (!alone) cluster_sync_all();  // nobody leaves while its sums are still read
  if (threadIdx.x == 0 && *failed && p.error_flag) atomicExch(p.error_flag, 4);
}

// Rows of float32 out of or into places of a matrix of `extent` rows: a block a row, bound by what it copies
template <bool INTO>
__global__ void __launch_bounds__(256) copy_rows_kernel(const float* __restrict__ from, float* __restrict__ to, const int* __restrict__ places,
                                                        int width, int extent, int vec) {
  pdl_launch_dependents();
  pdl_wait();
  const int place = places[blockIdx.x];
  if (!FMS_IN(place, extent)) return;
  const float* a = from + (size_t)(INTO ? (int)blockIdx.x : place) * width;
  float* b = to + (size_t)(INTO ? place : (int)blockIdx.x) * width;
  if (vec)
    for (int i = threadIdx.x; i < width / 4; i += blockDim.x) reinterpret_cast<float4*>(b)[i] = reinterpret_cast<const float4*>(a)[i];
  else
    for (int i = threadIdx.x; i < width; i += blockDim.x) b[i] = a[i];
}

int multiprocessors() {
  static int sms = 0;
  if (sms == 0) {
    int device = 0;
    cudaGetDevice(&device);
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0) sms = 148;
  }
  return sms;
}

int make_parts_map(CUtensorMap* map, const void* base, long rows, int pitch, int box_rows) {
  EncodeTiled enc = encode_tiled();
  if (enc == nullptr) return fms_fail("gemm_f32_tc: the driver does not export cuTensorMapEncodeTiled");
  const cuuint64_t dims[2] = {(cuuint64_t)pitch, (cuuint64_t)rows}, strides[1] = {(cuuint64_t)pitch * 2};
  const cuuint32_t box[2] = {BK, (cuuint32_t)box_rows}, elem[2] = {1, 1};
  CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fms_fail("gemm_f32_tc: cuTensorMapEncodeTiled failed with %d (rows %ld, pitch %d)", (int)r, rows, pitch);
  return 0;
}

template <typename S>
int launch_shape(const Product& p, const CUtensorMap& map_x, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_split_kernel<S>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
    cudaFuncAttributes made;
    if (e == cudaSuccess) e = cudaFuncGetAttributes(&made, gemm_f32_split_kernel<S>);
    if (e != cudaSuccess) return fms_fail("gemm_f32_tc: %zu bytes of shared memory refused: %s", S::SMEM, cudaGetErrorString(e));
    // the shares that the warps take come out of what the block is launched with
    if (S::EPI_REGS > 0 && 32 * (S::CONV * S::CONV_REGS + 4 * OTHER_REGS + S::EPI * S::EPI_REGS) > made.numRegs * S::THREADS)
      return fms_fail("gemm_f32_tc: built with %d registers a thread", made.numRegs);
    configured = true;
  }
  cudaLaunchConfig_t cfg = {};
  const int sms = multiprocessors();
  cfg.gridDim = dim3((unsigned)(p.ranks > 1 ? p.tiles * p.ranks : p.tiles < sms ? p.tiles : sms));
  cfg.blockDim = dim3(S::THREADS);
  cfg.dynamicSmemBytes = S::SMEM;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = fms_pdl_enabled() ? 1 : 0;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = p.ranks;
  attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  cudaLaunchKernelEx(&cfg, gemm_f32_split_kernel<S>, p, map_x);
  return fms_launch_status("gemm_f32_tc");
}

int pitch_of(int K) { return (K + 63) / 64 * 64; }

// How a product of M rows is cut: rows of x a block and whether a cluster shares a tile's runs
void plan(int M, int N, int K, Product& p) {
  const long long tiles_w = (N + WROWS - 1) / WROWS;
  const int sms = multiprocessors(), all_ranks = ranks_for(K);
  long long best = -1;
  auto consider = [&](int nt) {
    const long long tiles_x = (M + nt - 1) / nt, tiles = tiles_w * tiles_x;
    const long long mma = 12 * (nt < 64 ? 32 : nt / 2), shared = (12 * (4096 + nt * 32) + (WROWS + nt) * 192) / 128;
    const long long step = (mma > shared ? mma : shared > 800 ? shared : 800) + 100;
    for (int ranks = 1; ranks <= all_ranks; ranks += all_ranks > 1 ? all_ranks - 1 : 1) {
      const int runs = (K + p.run_len - 1) / p.run_len;
      const long long each = (ranks > 1 ? (p.run_len + BK - 1) / BK * step + 45 * nt : (K + BK - 1) / BK * step + 45LL * nt * runs) + (ranks > 1 ? 15000 : 5000);
      const long long cost = (tiles * ranks + sms - 1) / sms * each;
      if (best < 0 || cost < best) {
        best = cost;
        p.nt = nt;
        p.ranks = ranks;
        p.tiles_x = (int)tiles_x;
        p.tiles = (int)(tiles < 0x7fffffffLL ? tiles : 0x7fffffffLL);
      }
      if (all_ranks == 1) break;
    }
  };
  for (int t = (M + 255) / 256; t <= (M + 255) / 256 + 4; ++t) consider(((M + t - 1) / t + 31) / 32 * 32);
}
}  // namespace

// scratch: 128-byte aligned, 6 bytes for every row of x and k (K rounded up to a multiple of 64) and one for every row of x and of w
FMS_API int fms_gemm_f32_tc(const float* x, const float* w, const float* bias, float* y, void* scratch, long long scratch_bytes, int M, int N,
                            int K, int* error_flag, cudaStream_t stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0 || K > MOST_K) return fms_fail("gemm_f32_tc: K %d, at most %d", K, MOST_K);
  Product p = {};
  p.x = x; p.w = w; p.bias = bias; p.y = y;
  p.M = M; p.N = N; p.K = K;
  p.error_flag = error_flag;
  p.run_len = run_length(K);
  const uintptr_t at = (uintptr_t)x | (uintptr_t)w;
  p.vec = K % 8 == 0 && (at & 31) == 0 ? 2 : K % 4 == 0 && (at & 15) == 0 ? 1 : 0;
  plan(M, N, K, p);
  if ((long long)p.tiles * p.ranks > 0x7fffffffLL) return fms_fail("gemm_f32_tc: %d x %d are more tiles than one launch takes", M, N);
  CUtensorMap map_x = {};
  const int pitch = pitch_of(K);
  if (3LL * M > 0x7fffffffLL) return fms_fail("gemm_f32_tc: %d rows", M);
  if (scratch == nullptr || ((uintptr_t)scratch & 127) || scratch_bytes < (long long)M * pitch_of(K) * 6 + M + N)
    return fms_fail("gemm_f32_tc: %lld bytes of scratch at %p", scratch_bytes, scratch);
  unsigned char* kinds = (unsigned char*)scratch + (size_t)M * pitch * 6;
  fms_launch(split_rows_kernel, dim3(M), dim3(256), 0, stream, x, (uint4*)scratch, kinds, M, K, pitch, p.vec);
  if (fms_launch_status("gemm_f32_tc")) return 1;
  p.x_kinds = kinds;
  p.w_kinds = kinds + M;
  if (make_parts_map(&map_x, scratch, 3L * M, pitch, p.nt)) return 1;
  if (p.nt <= 64) return launch_shape<Shape<64, 2, 16, 8, 3, 2, 4, 0, 0>>(p, map_x, stream);
  if (p.nt <= 128) return launch_shape<Shape<128, 2, 16, 8, 2, 1, 0, 56, 112>>(p, map_x, stream);
  return launch_shape<Shape<256, 1, 4, 8, 3, 1, 0, 88, 184>>(p, map_x, stream);
}

// to[r] = from[places[r]], or with `into` to[places[r]] = from[r], for r < rows; places lie within `extent` rows
FMS_API int fms_copy_rows_f32(const float* from, float* to, const int* places, int rows, int width, int extent, int into, cudaStream_t stream) {
  if (rows <= 0 || width <= 0) return 0;
  const int vec = width % 4 == 0 && (((uintptr_t)from | (uintptr_t)to) & 15) == 0;
  if (into) fms_launch(copy_rows_kernel<true>, dim3(rows), dim3(256), 0, stream, from, to, places, width, extent, vec);
  else fms_launch(copy_rows_kernel<false>, dim3(rows), dim3(256), 0, stream, from, to, places, width, extent, vec);
  return fms_launch_status("copy_rows_f32");
}
