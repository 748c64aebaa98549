// State matrices under one decay a head, over many tokens at once.  Per head, with a and b one number a token each,
//
//   S_t = a_t S_(t-1) + b_t k_t v_t^T        o_t = S_t^T q_t            S [dim, vdim], float32 throughout
//
// is, for a run of C = 64 tokens behind the state S (D(t, s) = b_s a_(s+1) .. a_t, G_t = a_1 .. a_t),
//
//   o_t = G_t S^T q_t + sum_(s <= t) D(t, s) (q_t . k_s) v_s        S' = G_C S + sum_s D(C, s) k_s v_s^T
//
// four products a run instead of a walk over its tokens, whose every step was a chain of shared-memory loads, few
// multiply-adds and shuffles (csrc/state_scan.cu, which short prompts and decode steps keep).  Four kernels:
//
//   chunk_scores   q_t . k_s of every run and key head
//   chunk_states   sum_s D(C, s) k_s v_s^T of every run and head, and G_C
//   chunk_carry    the states before every run: elementwise, in the order of the runs, over what chunk_states left
//   chunk_outputs  o of every run and head
//
// All but the third take every run at once.  The states of the runs of one pass lie in at most `runs` runs' worth of scratch;
// longer steps take several passes, between which the one sequence that a boundary cuts has its state in `carry`.  Products of decays
// are taken as products in the order of the tokens (no logarithms: a decay of zero and a run of tiny ones need no case), and a
// token's results never touch later tokens' rows, not even times zero.
//
// KIND 0: a = decay[head], b = 1.  KIND 1: (a, b, e) = gates[token, head]; a normalizer n_t = a n + b k beside S, and o is divided
// by max(|n . q|, e) + 1e-6.  KIND 2: a = exp(-exp(a_log) dt), b = dt = softplus(raw + bias), and o += d_skip v; key heads
// are shared by groups of heads.
#include "common.cuh"

namespace {
constexpr int C = 64;        // tokens of a run
constexpr int COLS = 128;    // value columns of a block: one head of 128 values, two of 64, four of 32
constexpr int SLICE = 32;    // state rows (key channels) brought into shared memory at a time
constexpr int SROW = SLICE + 4;  // 16-byte reads of neighbouring rows meet different banks
constexpr int PROW = C + 4;

struct ChunkArgs {
  const float* q;  // token t, key head g: q + t * row + g * dim; k alike; v: v + t * row + head * vdim
  const float* k;
  const float* v;
  long row;
  const int* runs;       // [runs, 2]: first row and end of every run
  const int* first_run;  // [n_seqs + 1]
  const int* slots;
  const float* decay;    // KIND 0
  const float* gates;    // KIND 1
  float* norm_in;        // KIND 1: [n_seqs, heads, dim], n before the step; carries n from pass to pass
  float* norm_state;     // KIND 1: [slots, heads, dim + 1]
  const void* dt_raw;    // KIND 2: column `head` of rows of dt_stride values
  const float* dt_bias;
  const float* a_log;
  const float* d_skip;
  long dt_stride;
  int dt_is_bf16;
  float* state;   // [slots, heads, vdim, dim]
  float* carry;   // [2, heads, vdim, dim], written by every other pass, or null (one pass)
  float* scores;  // scratch: [runs of a pass, key heads, C, C], row t
  float* states;  // scratch: [runs of a pass, heads, vdim, dim]
  float* norms;   // scratch, KIND 1: [runs of a pass, heads, dim]
  float* totals;  // scratch: [runs of a pass, heads]
  float* o;       // [tokens, heads * vdim]
  int heads, key_heads, n_seqs, n_slots, write_state;
  int run_lo, run_hi, pass;  // this pass
};

__device__ __forceinline__ void copy16(float* smem, const float* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(smem)), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// (a, b) of a token and head; beyond the run's end (1, 0), which changes nothing
template <int KIND>
__device__ __forceinline__ float2 token_gates(const ChunkArgs& g, int t, int end, int head) {
  if (t >= end) return make_float2(1.f, 0.f);
  if (KIND == 0) return make_float2(g.decay[head], 1.f);
  if (KIND == 1) {
    const float* p = g.gates + ((size_t)t * g.heads + head) * 3;
    return make_float2(p[0], p[1]);
  }
  // in double, rounded once: a decay's error compounds over a sequence
  const size_t at = (size_t)t * g.dt_stride + head;
  const double x = (g.dt_is_bf16 ? (double)__bfloat162float(((const __nv_bfloat16*)g.dt_raw)[at]) : (double)((const float*)g.dt_raw)[at]) +
                   (double)g.dt_bias[head];
  const double dt = x > 40.0 ? x : log1p(exp(x));
  return make_float2((float)exp(-exp((double)g.a_log[head]) * dt), (float)dt);
}

// ---- scores: 64 x 64 a block, 8 x 4 a thread ---------------------------------------------------------------------------
template <int DIM>
__global__ void __launch_bounds__(128) chunk_scores_kernel(ChunkArgs g) {
  __shared__ __align__(16) float sm[2][2][C][SROW];
  pdl_launch_dependents();
  pdl_wait();
  const int run = g.run_lo + blockIdx.x, kh = blockIdx.y, tid = threadIdx.x;
  const int row0 = g.runs[2 * run], rows = g.runs[2 * run + 1] - row0;
  const float* q = g.q + (size_t)row0 * g.row + (size_t)kh * DIM;
  const float* k = g.k + (size_t)row0 * g.row + (size_t)kh * DIM;
  auto issue = [&](int d0, int buf) {
    for (int i = tid; i < C * (SLICE / 4); i += 128) {
      const int t = i / (SLICE / 4), d = (i % (SLICE / 4)) * 4;
      const size_t at = (size_t)min(t, rows - 1) * g.row + d0 + d;
      copy16(&sm[buf][0][t][d], q + at, t < rows);
      copy16(&sm[buf][1][t][d], k + at, t < rows);
    }
    copies_commit();
  };
  const int ty = tid >> 4, tx = tid & 15;  // rows ty * 8 + i, columns tx + 16 j
  float acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  issue(0, 0);
#pragma unroll 1
  for (int d0 = 0; d0 < DIM; d0 += SLICE) {
    const int buf = (d0 / SLICE) & 1;
    if (d0 + SLICE < DIM) {
      issue(d0 + SLICE, buf ^ 1);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncthreads();
#pragma unroll
    for (int d = 0; d < SLICE; d += 4) {
      float4 kx[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) kx[j] = *reinterpret_cast<const float4*>(&sm[buf][1][tx + 16 * j][d]);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 qx = *reinterpret_cast<const float4*>(&sm[buf][0][ty * 8 + i][d]);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          acc[i][j] = fmaf(qx.x, kx[j].x, acc[i][j]);
          acc[i][j] = fmaf(qx.y, kx[j].y, acc[i][j]);
          acc[i][j] = fmaf(qx.z, kx[j].z, acc[i][j]);
          acc[i][j] = fmaf(qx.w, kx[j].w, acc[i][j]);
        }
      }
    }
    __syncthreads();
  }
  float* out = g.scores + ((size_t)blockIdx.x * g.key_heads + kh) * C * C;
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) out[(ty * 8 + i) * C + tx + 16 * j] = acc[i][j];
}

// ---- a run's own state: 128 value columns x DIM a block, 8 x DIM / 16 a thread ----------------------------------------
template <int DIM, int VDIM, int KIND>
__global__ void __launch_bounds__(256) chunk_states_kernel(ChunkArgs g) {
  constexpr int HB = COLS / VDIM, N = DIM / 16;
  extern __shared__ __align__(16) float sm[];
  float* vs = sm;                    // [C][COLS], times D(C, s)
  float* ks = vs + C * COLS;         // [C][DIM]
  __shared__ float ab[HB][2][C], weight[HB][C];
  pdl_launch_dependents();
  pdl_wait();
  const int run = g.run_lo + blockIdx.x, head0 = blockIdx.y * HB, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = g.runs[2 * run], end = g.runs[2 * run + 1], rows = end - row0;
  const int kh = head0 / (g.heads / g.key_heads);
  for (int i = tid; i < C * (DIM / 4); i += 256) {
    const int t = i / (DIM / 4), d = (i % (DIM / 4)) * 4;
    copy16(ks + t * DIM + d, g.k + (size_t)(row0 + min(t, rows - 1)) * g.row + (size_t)kh * DIM + d, t < rows);
  }
  for (int i = tid; i < C * (COLS / 4); i += 256) {
    const int t = i / (COLS / 4), c = (i % (COLS / 4)) * 4;
    copy16(vs + t * COLS + c, g.v + (size_t)(row0 + min(t, rows - 1)) * g.row + (size_t)head0 * VDIM + c, t < rows);
  }
  copies_commit();
  if (tid < HB * C) {
    const float2 w = token_gates<KIND>(g, row0 + tid % C, end, head0 + tid / C);
    ab[tid / C][0][tid % C] = w.x;
    ab[tid / C][1][tid % C] = w.y;
  }
  __syncthreads();
  if (warp < HB) {  // weight[s] = b_s a_(s+1) .. a_(C-1): a lane two neighbouring tokens, the products behind it by shuffles
    const float a0 = ab[warp][0][2 * lane], a1 = ab[warp][0][2 * lane + 1];
    float behind = a0 * a1;  // inclusive product over this lane's tokens and all later ones
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float other = __shfl_down_sync(0xffffffffu, behind, o);
      if (lane + o < 32) behind *= other;
    }
    if (lane == 0) g.totals[(size_t)blockIdx.x * g.heads + head0 + warp] = behind;
    float after = __shfl_down_sync(0xffffffffu, behind, 1);
    if (lane == 31) after = 1.f;
    weight[warp][2 * lane + 1] = ab[warp][1][2 * lane + 1] * after;
    weight[warp][2 * lane] = ab[warp][1][2 * lane] * (a1 * after);
  }
  copies_wait<0>();
  __syncthreads();
  for (int i = tid; i < C * (COLS / 4); i += 256) {
    const int t = i / (COLS / 4), c = (i % (COLS / 4)) * 4;
    const float w = weight[c / VDIM][t];
    float4* p = reinterpret_cast<float4*>(vs + t * COLS + c);
    const float4 x = *p;
    *p = t < rows ? make_float4(x.x * w, x.y * w, x.z * w, x.w * w) : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  const int ty = tid >> 4, tx = tid & 15;  // value columns ty * 4 + i (+ 64), key channels tx * 4 + j (+ 64)
  float acc[8][N];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) acc[i][j] = 0.f;
#pragma unroll 8
  for (int s = 0; s < C; ++s) {
    float a[8], b[N];
    *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(vs + s * COLS + ty * 4);
    *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(vs + s * COLS + 64 + ty * 4);
#pragma unroll
    for (int j = 0; j < N; j += 4) *reinterpret_cast<float4*>(b + j) = *reinterpret_cast<const float4*>(ks + s * DIM + j * 16 + tx * 4);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < N; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
  }
  float* out = g.states + ((size_t)blockIdx.x * g.heads + head0) * VDIM * DIM;  // the block's heads lie side by side
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < N; j += 4)
      *reinterpret_cast<float4*>(out + (size_t)((i >> 2) * 64 + ty * 4 + (i & 3)) * DIM + j * 16 + tx * 4) =
          make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
  if (KIND == 1 && tid < DIM) {
    float n = 0.f;
#pragma unroll 8
    for (int s = 0; s < C; ++s)
      if (s < rows) n = fmaf(weight[0][s], ks[s * DIM + tid], n);
    g.norms[((size_t)blockIdx.x * g.heads + head0) * DIM + tid] = n;
  }
}

// ---- the states before every run, in place of the runs' own -----------------------------------------------------------
// A thread four neighbouring state values (blockIdx.z 0) or, KIND 1, one of the normalizer's (blockIdx.z 1) of one sequence.
template <int DIM, int VDIM, int KIND>
__global__ void __launch_bounds__(256) chunk_carry_kernel(ChunkArgs g) {
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.y;
  const int lo = max(g.first_run[seq], g.run_lo), hi = min(g.first_run[seq + 1], g.run_hi);
  if (lo >= hi) return;
  const int slot = __ldcg(g.slots + seq);
  if (!FMS_IN(slot, g.n_slots)) return;
  const bool begins = lo == g.first_run[seq], ends = hi == g.first_run[seq + 1];
  const size_t e = (size_t)blockIdx.x * 256 + threadIdx.x;
  if (KIND == 1 && blockIdx.z == 1) {
    if (e >= (size_t)g.heads * DIM) return;
    const int head = (int)(e / DIM);
    float* in = g.norm_in + (size_t)seq * g.heads * DIM + e;
    float n = *in;
    for (int r = lo - g.run_lo; r < hi - g.run_lo; ++r) {
      float* p = g.norms + (size_t)r * g.heads * DIM + e;
      const float own = *p;
      *p = n;
      n = fmaf(g.totals[(size_t)r * g.heads + head], n, own);
    }
    *in = n;
    if (ends && g.write_state) g.norm_state[((size_t)slot * g.heads + head) * (DIM + 1) + e % DIM] = n;
    return;
  }
  const size_t per_seq = (size_t)g.heads * VDIM * DIM / 4;
  if (e >= per_seq) return;
  const int head = (int)(e * 4 / (VDIM * DIM));
  float4* held = reinterpret_cast<float4*>(g.state + (size_t)slot * per_seq * 4) + e;
  float4* between = reinterpret_cast<float4*>(g.carry) + e;
  float4 s = begins ? *held : between[(g.pass & 1) * per_seq];
  float4* p = reinterpret_cast<float4*>(g.states) + (size_t)(lo - g.run_lo) * per_seq + e;
  const float* total = g.totals + (size_t)(lo - g.run_lo) * g.heads + head;
  constexpr int AHEAD = 4;  // runs whose own states are on their way
  float4 own[AHEAD];
  float a[AHEAD];
  const int n = hi - lo;
#pragma unroll
  for (int i = 0; i < AHEAD; ++i)
    if (i < n) {
      own[i] = p[i * per_seq];
      a[i] = total[(size_t)i * g.heads];
    }
  for (int r0 = 0; r0 < n; r0 += AHEAD) {
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int r = r0 + i;
      if (r >= n) break;
      const float4 x = own[i];
      const float w = a[i];
      if (r + AHEAD < n) {
        own[i] = p[(size_t)(r + AHEAD) * per_seq];
        a[i] = total[(size_t)(r + AHEAD) * g.heads];
      }
      p[(size_t)r * per_seq] = s;
      s = make_float4(fmaf(w, s.x, x.x), fmaf(w, s.y, x.y), fmaf(w, s.z, x.z), fmaf(w, s.w, x.w));
    }
  }
  if (!ends) between[((g.pass + 1) & 1) * per_seq] = s;
  else if (g.write_state) *held = s;
}

// ---- outputs: 64 tokens x 128 value columns a block, 8 x 8 a thread ---------------------------------------------------
// Threads (ty, tx): tokens ty * 8 + i, columns tx + 16 j.  First q against the state before the run (32 state rows at a
// time, two buffers), then the run's own tokens, each thread only as far as its own rows reach.  The heavier rows go to
// another scheduler in every block.
template <int VDIM>
constexpr size_t OUT_SMEM = (size_t)(2 * (C + COLS) * SROW + COLS / VDIM * C * PROW) * sizeof(float);

template <int DIM, int VDIM, int KIND>
__global__ void __launch_bounds__(128, VDIM == 128 ? 3 : 2) chunk_outputs_kernel(ChunkArgs g) {
  constexpr int HB = COLS / VDIM;
  extern __shared__ __align__(16) float sm[];
  float* buffers = sm;                       // [2]: q [C][SROW], state [COLS][SROW]; afterwards v [C][COLS]
  float* P = sm + 2 * (C + COLS) * SROW;     // [HB][C][PROW], row t
  static_assert(C * COLS <= 2 * (C + COLS) * SROW, "v fits where the slices were");
  __shared__ float as[HB][C], bs[HB][C], G[HB][C], nq[C];
  pdl_launch_dependents();
  pdl_wait();
  const int local = blockIdx.x, run = g.run_lo + local, head0 = blockIdx.y * HB, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = g.runs[2 * run], end = g.runs[2 * run + 1], rows = end - row0;
  const int kh = head0 / (g.heads / g.key_heads);
  const float* q = g.q + (size_t)row0 * g.row + (size_t)kh * DIM;
  const float* S = g.states + ((size_t)local * g.heads + head0) * VDIM * DIM;
  auto issue = [&](int d0, int buf) {
    float* qd = buffers + buf * (C + COLS) * SROW;
    float* sd = qd + C * SROW;
    for (int i = tid; i < C * (SLICE / 4); i += 128) {
      const int t = i / (SLICE / 4), d = (i % (SLICE / 4)) * 4;
      copy16(qd + t * SROW + d, q + (size_t)min(t, rows - 1) * g.row + d0 + d, t < rows);
    }
    for (int i = tid; i < COLS * (SLICE / 4); i += 128) {
      const int c = i / (SLICE / 4), d = (i % (SLICE / 4)) * 4;
      copy16(sd + c * SROW + d, S + (size_t)c * DIM + d0 + d, true);
    }
    copies_commit();
  };
  issue(0, 0);
  for (int i = tid; i < HB * C; i += 128) {
    const float2 w = token_gates<KIND>(g, row0 + i % C, end, head0 + i / C);
    as[i / C][i % C] = w.x;
    bs[i / C][i % C] = w.y;
  }
  __syncthreads();
  // P[t][s] = D(t, s) (q_t . k_s), a thread a column s: the products run down the tokens
  for (int i = tid; i < HB * C; i += 128) {
    const int h = i / C, s = i % C;
    const float* raw = g.scores + ((size_t)local * g.key_heads + kh) * C * C + s;
    float* p = P + h * C * PROW + s;
    float d = bs[h][s];
#pragma unroll 8
    for (int t = 0; t < C; ++t) {
      const float x = raw[t * C];
      if (t > s) d *= as[h][t];
      p[t * PROW] = t >= s ? x * d : 0.f;
    }
  }
  if (warp < HB) {  // G[t] = a_0 .. a_t
    const float a0 = as[warp][2 * lane], a1 = as[warp][2 * lane + 1];
    float upto = a0 * a1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float other = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto *= other;
    }
    float before = __shfl_up_sync(0xffffffffu, upto, 1);
    if (lane == 0) before = 1.f;
    G[warp][2 * lane] = before * a0;
    G[warp][2 * lane + 1] = upto;
  }
  const int turned = (warp + local + blockIdx.y) & 3;
  const int ty = turned * 2 + (lane >> 4), tx = lane & 15;
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
  float own_nq = 0.f;  // KIND 1, threads 0..63: q_t . n
  const float* n_before = KIND == 1 ? g.norms + ((size_t)local * g.heads + head0) * DIM : nullptr;
#pragma unroll 1
  for (int d0 = 0; d0 < DIM; d0 += SLICE) {
    const int buf = (d0 / SLICE) & 1;
    if (d0 + SLICE < DIM) {
      issue(d0 + SLICE, buf ^ 1);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    __syncthreads();
    const float* qd = buffers + buf * (C + COLS) * SROW;
    const float* sd = qd + C * SROW;
#pragma unroll 2
    for (int d = 0; d < SLICE; d += 4) {
      float4 x[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) x[j] = *reinterpret_cast<const float4*>(sd + (tx + 16 * j) * SROW + d);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float4 y = *reinterpret_cast<const float4*>(qd + (ty * 8 + i) * SROW + d);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          acc[i][j] = fmaf(y.x, x[j].x, acc[i][j]);
          acc[i][j] = fmaf(y.y, x[j].y, acc[i][j]);
          acc[i][j] = fmaf(y.z, x[j].z, acc[i][j]);
          acc[i][j] = fmaf(y.w, x[j].w, acc[i][j]);
        }
      }
    }
    if (KIND == 1 && tid < C) {
#pragma unroll
      for (int d = 0; d < SLICE; d += 4) {
        const float4 y = *reinterpret_cast<const float4*>(qd + tid * SROW + d);
        const float4 n = *reinterpret_cast<const float4*>(n_before + d0 + d);
        own_nq = fmaf(y.x, n.x, fmaf(y.y, n.y, fmaf(y.z, n.z, fmaf(y.w, n.w, own_nq))));
      }
    }
    __syncthreads();  // the buffer is free (and P and G are complete)
  }
  for (int i = tid; i < C * (COLS / 4); i += 128) {
    const int t = i / (COLS / 4), c = (i % (COLS / 4)) * 4;
    copy16(buffers + t * COLS + c, g.v + (size_t)(row0 + min(t, rows - 1)) * g.row + (size_t)head0 * VDIM + c, t < rows);
  }
  copies_commit();
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] *= G[16 * j / VDIM][ty * 8 + i];
  if (KIND == 1 && tid < C) {  // n_t . q_t = G_t (n . q_t) + the sum of the row of P
    float sum = G[0][tid] * own_nq;
    for (int s = 0; s <= tid; ++s) sum += P[tid * PROW + s];
    nq[tid] = sum;
  }
  copies_wait<0>();
  __syncthreads();
  // tokens before this thread's rows: four at a time for all its rows
#pragma unroll 1
  for (int s = 0; s < ty * 8; s += 4) {
#pragma unroll
    for (int h = 0; h < HB; ++h) {
      float4 p[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) p[i] = *reinterpret_cast<const float4*>(P + (h * C + ty * 8 + i) * PROW + s);
#pragma unroll
      for (int j = h * 8 / HB; j < (h + 1) * 8 / HB; ++j) {
        const float* v = buffers + s * COLS + tx + 16 * j;
        const float v0 = v[0], v1 = v[COLS], v2 = v[2 * COLS], v3 = v[3 * COLS];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          acc[i][j] = fmaf(p[i].x, v0, acc[i][j]);
          acc[i][j] = fmaf(p[i].y, v1, acc[i][j]);
          acc[i][j] = fmaf(p[i].z, v2, acc[i][j]);
          acc[i][j] = fmaf(p[i].w, v3, acc[i][j]);
        }
      }
    }
  }
  // its own rows: token ty * 8 + s reaches the rows from itself on
#pragma unroll
  for (int h = 0; h < HB; ++h)
#pragma unroll
    for (int s = 0; s < 8; ++s) {
      float p[8];
#pragma unroll
      for (int i = s; i < 8; ++i) p[i] = P[(h * C + ty * 8 + i) * PROW + ty * 8 + s];
#pragma unroll
      for (int j = h * 8 / HB; j < (h + 1) * 8 / HB; ++j) {
        const float v = buffers[(ty * 8 + s) * COLS + tx + 16 * j];
#pragma unroll
        for (int i = s; i < 8; ++i) acc[i][j] = fmaf(p[i], v, acc[i][j]);
      }
    }
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int t = ty * 8 + i;
    if (t >= rows) continue;
    float scale = 1.f;
    if (KIND == 1) scale = 1.f / (fmaxf(fabsf(nq[t]), g.gates[((size_t)(row0 + t) * g.heads + head0) * 3 + 2]) + 1e-6f);
    float* out = g.o + (size_t)(row0 + t) * g.heads * VDIM + (size_t)head0 * VDIM + tx;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float x = acc[i][j];
      if (KIND == 1) x *= scale;
      if (KIND == 2) x = fmaf(g.d_skip[head0 + 16 * j / VDIM], buffers[t * COLS + tx + 16 * j], x);
      out[16 * j] = x;
    }
  }
}

template <int DIM, int VDIM, int KIND>
int launch_passes(ChunkArgs g, int n_runs, int pass_runs, cudaStream_t stream) {
  constexpr int HB = COLS / VDIM;
  constexpr size_t state_smem = (size_t)C * (COLS + DIM) * sizeof(float);
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(chunk_states_kernel<DIM, VDIM, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)state_smem);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(chunk_outputs_kernel<DIM, VDIM, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OUT_SMEM<VDIM>);
    if (e != cudaSuccess) return fms_fail("chunk_scan: shared memory refused: %s", cudaGetErrorString(e));
    configured = true;
  }
  for (int lo = 0; lo < n_runs; lo += pass_runs) {
    g.pass = lo / pass_runs;
    g.run_lo = lo;
    g.run_hi = lo + pass_runs < n_runs ? lo + pass_runs : n_runs;
    const int n = g.run_hi - lo;
    const size_t quads = (size_t)g.heads * VDIM * DIM / 4;
    fms_launch(chunk_scores_kernel<DIM>, dim3(n, g.key_heads), dim3(128), 0, stream, g);
    fms_launch(chunk_states_kernel<DIM, VDIM, KIND>, dim3(n, g.heads / HB), dim3(256), state_smem, stream, g);
    fms_launch(chunk_carry_kernel<DIM, VDIM, KIND>, dim3((unsigned)((quads + 255) / 256), g.n_seqs, KIND == 1 ? 2 : 1), dim3(256), 0, stream, g);
    fms_launch(chunk_outputs_kernel<DIM, VDIM, KIND>, dim3(n, g.heads / HB), dim3(128), OUT_SMEM<VDIM>, stream, g);
    if (fms_launch_status("chunk_scan")) return 1;
  }
  return 0;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
}  // namespace

FMS_API int fms_chunk_scan_tokens() { return C; }
// Whether heads of these sizes, `shared` of them to a key head, go through the kernels above.
FMS_API int fms_chunk_scan_takes(int dim, int vdim, int shared) {
  return dim == 128 && (vdim == 128 || (vdim == 64 && shared % 2 == 0)) ? 1 : 0;
}

// kind, q, k, v, row, gates and the rest: see ChunkArgs and the head of this file.  runs, first_run: the step's rows cut into runs
// of fms_chunk_scan_tokens() rows of one sequence.  pass_runs: how many runs' states the scratch holds; with fewer than n_runs,
// `carry` is needed.  For kind 1 norm_in holds n before the step and is written.
FMS_API int fms_chunk_scan(int kind, const float* q, const float* k, const float* v, long row, const int* runs, const int* first_run,
                           int n_runs, int pass_runs, const int* slots, int n_seqs, const float* decay, const float* gates,
                           float* norm_in, float* norm_state, const void* dt_raw, int dt_dtype, long dt_stride, const float* dt_bias,
                           const float* a_log, const float* d_skip, float* state, float* carry, float* scores, float* states,
                           float* norms, float* totals, float* o, int heads, int key_heads, int dim, int vdim, int write_state,
                           int n_slots, cudaStream_t stream) {
  if (n_runs <= 0 || n_seqs <= 0) return 0;
  if (heads <= 0 || key_heads <= 0 || heads % key_heads || !fms_chunk_scan_takes(dim, vdim, heads / key_heads) || (kind == 1 && vdim != 128))
    return fms_fail("chunk_scan: %d heads over %d, dim %d, vdim %d", heads, key_heads, dim, vdim);
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || row % 4 || !aligned16(state) || !aligned16(states) || (carry && !aligned16(carry)))
    return fms_fail("chunk_scan: rows of %ld values, or a pointer, not on 16 bytes", row);
  if (pass_runs <= 0 || (pass_runs < n_runs && carry == nullptr)) return fms_fail("chunk_scan: %d runs of %d a pass without a carry", pass_runs, n_runs);
  if (n_seqs > 65535 || heads > 65535) return fms_fail("chunk_scan: %d sequences, %d heads", n_seqs, heads);
  if (!scores || !states || !totals || (kind == 0 && !decay) || (kind == 1 && (!gates || !norm_in || !norm_state || !norms)) ||
      (kind == 2 && (!dt_raw || !dt_bias || !a_log || !d_skip)))
    return fms_fail("chunk_scan: kind %d without what it reads", kind);
  if (kind == 2 && dt_dtype != FMS_F32 && dt_dtype != FMS_BF16) return fms_fail("chunk_scan: dtype code %d", dt_dtype);
  ChunkArgs g = {};
  g.q = q; g.k = k; g.v = v; g.row = row; g.runs = runs; g.first_run = first_run; g.slots = slots; g.decay = decay; g.gates = gates;
  g.norm_in = norm_in; g.norm_state = norm_state; g.dt_raw = dt_raw; g.dt_bias = dt_bias; g.a_log = a_log; g.d_skip = d_skip;
  g.dt_stride = dt_stride; g.dt_is_bf16 = dt_dtype == FMS_BF16; g.state = state; g.carry = carry; g.scores = scores; g.states = states;
  g.norms = norms; g.totals = totals; g.o = o; g.heads = heads; g.key_heads = key_heads; g.n_seqs = n_seqs; g.n_slots = n_slots;
  g.write_state = write_state;
  if (kind == 0) return vdim == 128 ? launch_passes<128, 128, 0>(g, n_runs, pass_runs, stream) : launch_passes<128, 64, 0>(g, n_runs, pass_runs, stream);
  if (kind == 1) return launch_passes<128, 128, 1>(g, n_runs, pass_runs, stream);
  if (kind == 2) return vdim == 128 ? launch_passes<128, 128, 2>(g, n_runs, pass_runs, stream) : launch_passes<128, 64, 2>(g, n_runs, pass_runs, stream);
  return fms_fail("chunk_scan: kind %d", kind);
}
