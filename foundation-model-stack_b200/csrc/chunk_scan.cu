// State matrices under one decay a head, over many tokens at once.  Per head, with a and b one number a token each,
//
//   S_t = a_t S_(t-1) + b_t k_t v_t^T        o_t = S_t^T q_t            S [dim, vdim], float32 throughout
//
// is, for a run of C = 64 tokens behind the state S (D(t, s) = b_s a_(s+1) .. a_t, G_t = a_1 .. a_t),
//
//   o_t = G_t S^T q_t + sum_(s <= t) D(t, s) (q_t . k_s) v_s        S' = G_C S + sum_s D(C, s) k_s v_s^T
//
// four products a run instead of a walk over its tokens, whose every step was a chain of shared-memory loads, few
// multiply-adds and shuffles (csrc/state_scan.cu, which short prompts and decode steps keep).  Three kernels:
//
//   chunk_scores   q_t . k_s of every run and key head; a, b, G and D(C, .) of every run and head
//   chunk_states   a block a head's (or half or quarter head's) columns of one sequence, run after run with the state in
//                  registers: leaves the state before every run
//   chunk_outputs  o of every run and head, all runs at once
//
// Bound by the FMA pipe and by what shared memory returns to registers: 8 x 8 elements a thread, two elements a multiply-add
// instruction (fma.rn.f32x2, the same roundings).  (On the tensor cores, with three bfloat16 parts a value and six products of
// parts, the results were ten times further from 64 bits, 9e-7 instead of 8e-8 of a row, and no sooner there.)
// Products of decays are taken as products (no logarithms: a decay of zero and a run of tiny ones need no case), and a token's
// values never touch earlier tokens' rows, not even times zero.  The states of the runs of one pass lie in at most pass_runs runs'
// worth of scratch; longer steps take several passes, between which the one sequence that a boundary cuts has its state in
// `carry`.
//
// KIND 0: a = decay[head], b = 1.  KIND 1: (a, b, e) = gates[token, head]; a normalizer n_t = a n + b k beside S, and o is divided
// by max(|n . q|, e) + 1e-6.  KIND 2: a = exp(-exp(a_log) dt), b = dt = softplus(raw + bias), and o += d_skip v; key heads
// are shared by groups of heads.
//
// KIND 3, the delta rule: S_t = a_t S_(t-1) + k_t u_t^T with u_t = beta_t (v_t - a_t S_(t-1)^T k_t).  Within a run the u hang
// together by a lower triangle, (I + A) U = diag(beta) (V - diag(G) K S), A[t][s] = beta_t a_(s+1) .. a_t (k_t . k_s) for s < t:
//
//   chunk_solve    T' = (I + A)^-1 diag(beta) of every run and head, all at once
//   delta_states   as chunk_states, with Y = V - diag(G) K S and U = T' Y first; U goes where o will be
//
// and chunk_outputs takes U for the values (b = 1).
//
// So that neither an output nor a state is further from 64 bits than the walk's: scores (and k . k) are summed in 64 bits and
// rounded once, as products of decays are; the other sums of an output and of a u are made of float32 runs of 16 terms, which
// under fixed decays 64 bits add up.  A run's part of the state and of the normalizer is one float32 chain of its 64 tokens.
// Errors of outputs and of states as parts of the walk's (400 and 2,048 tokens): fixed decays 0.77 and 0.94, 0.46 and 0.41; under a
// normalizer 0.88 and 0.83, 0.96 and 0.98; state space 0.98 and 0.99, 0.85 and 0.80; delta rule 0.99 and 0.90, 0.87 and 0.77.  (With
// float32 sums throughout outputs were at 1.05 to 1.15 of it, and a layer of 2,048 tokens under fixed decays took 531 us instead of
// 590, prompts of 1,062 and 638 tokens with a normalizer 503 instead of 516.)
#include "common.cuh"

namespace {
constexpr int C = 64;        // tokens of a run
constexpr int COLS = 128;    // value columns of a block of outputs: one head of 128 values or two of 64
constexpr int DIM = 128;     // key channels
constexpr int PART = 16;     // terms that a sum takes together before they are added to the rest: a single chain loses more
constexpr int SLICE = 16, SROW = SLICE + 2;  // of the scores: channels brought into shared memory at a time, rows padded by two
constexpr int TROW = C + 4, CROW = COLS + 4; // rows of 64 tokens, of 128 columns, padded by four floats

struct ChunkArgs {
  const float* q;  // token t, key head g: q + t * row + g * dim; k alike; v: v + t * row + head * vdim
  const float* k;
  const float* v;
  long row;
  const int* runs;       // [runs, 2]: first row and end of every run
  const int* first_run;  // [n_seqs + 1]
  const int* slots;
  long v_row;            // of v: row, or the stride of o where chunk_outputs reads U there
  const float* decay;    // KIND 0: [heads]; KIND 3: [tokens, heads]
  const float* gates;    // KIND 1; KIND 3: beta [tokens, heads]
  float* solve;          // scratch, KIND 3: [runs of a pass, heads, C, C]: T', element [s][t]
  float* norm_in;        // KIND 1: [n_seqs, heads, dim], n before the step; carries n from pass to pass
  float* norm_state;     // KIND 1: [slots, heads, dim + 1]
  const void* dt_raw;    // KIND 2: column `head` of rows of dt_stride values
  const float* dt_bias;
  const float* a_log;
  const float* d_skip;
  long dt_stride;
  int dt_is_bf16;
  float* state;    // [slots, heads, vdim, dim]
  float* carry;    // [2, heads, vdim, dim], written by every other pass, or null (one pass)
  float* scores;   // scratch: [runs of a pass, key heads, C, C], element [s][t]
  float* factors;  // scratch: [runs of a pass, heads, 4, C]: a, b, G, D(C, .)
  float* totals;   // scratch: [runs of a pass, heads]: G_C
  float* states;   // scratch: [runs of a pass, heads * vdim / COLS, dim, COLS]
  float* norms;    // scratch, KIND 1: [runs of a pass, heads, dim]
  int* flags;      // scratch: [runs of a pass, heads]: a value of the run's is not finite
  float* o;        // [tokens, heads * vdim]
  int heads, key_heads, n_seqs, n_slots, write_state;
  int run_lo, run_hi, pass;  // this pass
};

__device__ __forceinline__ void copy16(float* smem, const float* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(smem)), "l"(gmem), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

typedef unsigned long long f32x2;  // two floats side by side in registers
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;\n" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 d;
  asm("add.rn.f32x2 %0, %1, %2;\n" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;\n" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 pack2(float a, float b) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};\n" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ f32x2 swapped(f32x2 v) {
  float a, b;
  unpack2(v, a, b);
  return pack2(b, a);
}
// acc [rows 2 i, 2 i + 1][columns j, j ^ 1] += a [rows] x b [columns]: one step of an outer product of 8 rows (two runs of
// four, RS apart) by 2 P columns (runs of four, CS apart)
template <int P, int RS, int CS>
__device__ __forceinline__ void outer_step(const float* a, const float* b, f32x2 (&acc)[4][2 * P]) {
  f32x2 x[4], y[P], z[P];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(a + RS * i);
    x[2 * i] = v.x;
    x[2 * i + 1] = v.y;
  }
#pragma unroll
  for (int j = 0; j < P / 2; ++j) {
    const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(b + CS * j);
    y[2 * j] = v.x;
    y[2 * j + 1] = v.y;
    z[2 * j] = swapped(v.x);
    z[2 * j + 1] = swapped(v.y);
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < P; ++j) {
      acc[i][2 * j] = fma2(x[i], y[j], acc[i][2 * j]);
      acc[i][2 * j + 1] = fma2(x[i], z[j], acc[i][2 * j + 1]);
    }
}
template <int P>
__device__ __forceinline__ void outer_unpack(const f32x2 (&acc)[4][2 * P], float (&out)[8][2 * P]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < P; ++j) {
      unpack2(acc[i][2 * j], out[2 * i][2 * j], out[2 * i + 1][2 * j + 1]);
      unpack2(acc[i][2 * j + 1], out[2 * i][2 * j + 1], out[2 * i + 1][2 * j]);
    }
}

// (a, b) of a token and head; beyond the run's end (1, 0), which changes nothing
template <int KIND>
__device__ __forceinline__ float2 token_gates(const ChunkArgs& g, int t, int end, int head) {
  if (t >= end) return make_float2(1.f, 0.f);
  if (KIND == 0) return make_float2(g.decay[head], 1.f);
  if (KIND == 1) {
    const float* p = g.gates + ((size_t)t * g.heads + head) * 3;
    return make_float2(p[0], p[1]);
  }
  if (KIND == 3) return make_float2(g.decay[(size_t)t * g.heads + head], 1.f);
  // in double, rounded once: a decay's error compounds over a sequence
  const size_t at = (size_t)t * g.dt_stride + head;
  const double x = (g.dt_is_bf16 ? (double)__bfloat162float(((const __nv_bfloat16*)g.dt_raw)[at]) : (double)((const float*)g.dt_raw)[at]) +
                   (double)g.dt_bias[head];
  const double dt = x > 40.0 ? x : log1p(exp(x));
  return make_float2((float)exp(-exp((double)g.a_log[head]) * dt), (float)dt);
}

// ---- products of 64 x 64 tokens of a run: sum[i][j] = x_t . y_s over all channels, t = product_row(i), s = tid % 16 + 16 j ------
// Only blocks of 16 x 16 that hold an s <= t are made (20 of every thread's 32 products), the others are left at zero.
// In 64 bits, rounded once: an output is a sum of few of them where decays are short, and with float32 sums of 16 terms (7e-8 of
// a score's size, once rounded 2.5e-8) it was up to 20% further from 64 bits than the walk's.  Half the FMA pipe's rate, but a
// twentieth of the scan's products.  A slice's values are widened on their way from registers to shared memory, the next slice's
// loads are on their way meanwhile.  SAME: y is x.  sm: [2][SAME ? 1 : 2][C][SROW].
__device__ __forceinline__ int product_row(int i) { return 2 * (threadIdx.x >> 4) + (i & 1) + 16 * (i >> 1); }

template <bool SAME>
__device__ __forceinline__ void run_products(const float* x, const float* y, long row, int rows, double* sm, double (&sum)[8][4]) {
  constexpr int OPERANDS = SAME ? 1 : 2;
  const int tid = threadIdx.x, t0 = tid >> 2, d0 = (tid & 3) * 4;  // of a slice: rows t0 and t0 + 32, channels d0 .. + 3
  float4 next[OPERANDS][2];
  auto fetch = [&](int d) {
#pragma unroll
    for (int o = 0; o < OPERANDS; ++o)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int t = t0 + 32 * h;
        next[o][h] = t < rows ? *reinterpret_cast<const float4*>((o ? y : x) + (size_t)t * row + d + d0) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
  };
  auto put = [&](int buf) {
#pragma unroll
    for (int o = 0; o < OPERANDS; ++o)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        double2* p = reinterpret_cast<double2*>(sm + ((buf * OPERANDS + o) * C + t0 + 32 * h) * SROW + d0);
        p[0] = make_double2(next[o][h].x, next[o][h].y);
        p[1] = make_double2(next[o][h].z, next[o][h].w);
      }
  };
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) sum[i][j] = 0.0;
  const int ty = tid >> 4, tx = tid & 15;
  fetch(0);
  put(0);
  __syncthreads();
#pragma unroll 1
  for (int d = 0; d < DIM; d += SLICE) {
    const int buf = (d / SLICE) & 1;
    if (d + SLICE < DIM) fetch(d + SLICE);
    const double* xs = sm + (buf * OPERANDS * C + 2 * ty) * SROW;
    const double* ys = sm + ((buf * OPERANDS + OPERANDS - 1) * C + tx) * SROW;
#pragma unroll
    for (int e = 0; e < SLICE; e += 2) {
      double2 b[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const double2*>(ys + 16 * j * SROW + e);
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const double2 a = *reinterpret_cast<const double2*>(xs + ((i & 1) + 16 * (i >> 1)) * SROW + e);
#pragma unroll
        for (int j = 0; j <= (i >> 1); ++j) sum[i][j] = fma(a.y, b[j].y, fma(a.x, b[j].x, sum[i][j]));
      }
    }
    if (d + SLICE < DIM) put(buf ^ 1);
    __syncthreads();
  }
}

// ---- scores: a block a run and key head; the factors of the key head's heads, a warp a head ----------------------------
template <int KIND>
__global__ void __launch_bounds__(128) chunk_scores_kernel(ChunkArgs g) {
  __shared__ __align__(16) double sm[2 * 2 * C * SROW];
  pdl_wait();
  const int run = g.run_lo + blockIdx.x, kh = blockIdx.y, tid = threadIdx.x, lane = tid & 31;
  const int row0 = g.runs[2 * run], end = g.runs[2 * run + 1], rows = end - row0;
  const int shared = g.heads / g.key_heads;
  for (int head = kh * shared + (tid >> 5); head < (kh + 1) * shared; head += 4) {  // a lane two neighbouring tokens
    const float2 w0 = token_gates<KIND>(g, row0 + 2 * lane, end, head), w1 = token_gates<KIND>(g, row0 + 2 * lane + 1, end, head);
    // inclusive products over this lane's tokens and all earlier, all later ones, in 64 bits: a constant decay's roundings
    // would add up alike from run to run
    double upto = (double)w0.x * w1.x, behind = upto;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double x = __shfl_up_sync(0xffffffffu, upto, o), y = __shfl_down_sync(0xffffffffu, behind, o);
      if (lane >= o) upto *= x;
      if (lane + o < 32) behind *= y;
    }
    double before = __shfl_up_sync(0xffffffffu, upto, 1), after = __shfl_down_sync(0xffffffffu, behind, 1);
    if (lane == 0) before = 1.0;
    if (lane == 31) after = 1.0;
    float2* f = reinterpret_cast<float2*>(g.factors + ((size_t)blockIdx.x * g.heads + head) * 4 * C) + lane;
    f[0] = make_float2(w0.x, w1.x);
    f[C / 2] = make_float2(w0.y, w1.y);
    f[2 * C / 2] = make_float2((float)(before * w0.x), (float)upto);
    f[3 * C / 2] = make_float2((float)(w0.y * (w1.x * after)), (float)(w1.y * after));
    if (lane == 0) {
      g.totals[(size_t)blockIdx.x * g.heads + head] = (float)behind;
      g.flags[(size_t)blockIdx.x * g.heads + head] = 0;
    }
  }
  const int tx = tid & 15;  // tokens t = product_row(i), s = tx + 16 j
  double sum[8][4];
  run_products<false>(g.q + (size_t)row0 * g.row + (size_t)kh * DIM, g.k + (size_t)row0 * g.row + (size_t)kh * DIM, g.row, rows, sm, sum);
  // only now: blocks of the states' kernel that come earlier gather on the multiprocessors that are free first, two together
  // where every one could have its own (a layer of two prompts, 1,062 and 638 tokens: 498 instead of 552 us)
  pdl_launch_dependents();
  float* out = g.scores + ((size_t)blockIdx.x * g.key_heads + kh) * C * C;
#pragma unroll
  for (int i = 0; i < 8; i += 2)
#pragma unroll
    for (int j = 0; j <= (i >> 1); ++j)  // what lies above is not read
      *reinterpret_cast<float2*>(out + (tx + 16 * j) * C + product_row(i)) = make_float2((float)sum[i][j], (float)sum[i + 1][j]);
}

// ---- the states before every run: 128 key channels x VT value columns a block, 8 x VT / 8 a thread ------------------------
// A sequence's runs in order, the state and a run's own part of it in registers; the next run's keys and values are on their
// way meanwhile.  VT = 64, or 32 where that gives a single prompt's blocks to more multiprocessors.
template <int VT> constexpr size_t STATES_SMEM = (size_t)2 * C * (DIM + VT) * sizeof(float);

template <int VDIM, int KIND, int VT>
__global__ void __launch_bounds__(128, 2) chunk_states_kernel(ChunkArgs g) {
  constexpr int P = VT / 16;  // pairs of columns a thread
  extern __shared__ __align__(16) float sm[];
  __shared__ float weight[C];
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.y, tid = threadIdx.x;
  const int lo = max(g.first_run[seq], g.run_lo), hi = min(g.first_run[seq + 1], g.run_hi);
  if (lo >= hi) return;
  const int slot = __ldcg(g.slots + seq);
  if (!FMS_IN(slot, g.n_slots)) return;
  const bool begins = lo == g.first_run[seq], ends = hi == g.first_run[seq + 1];
  const int col0 = blockIdx.x * VT, head = col0 / VDIM, kh = head / (g.heads / g.key_heads);  // columns over all heads
  auto issue = [&](int run, int buf) {
    float* ks = sm + buf * C * (DIM + VT);
    float* vs = ks + C * DIM;
    const int row0 = g.runs[2 * run], rows = g.runs[2 * run + 1] - row0;
    const float* k = g.k + (size_t)row0 * g.row + (size_t)kh * DIM;
    const float* v = g.v + (size_t)row0 * g.row + col0;
    for (int i = tid; i < C * (DIM / 4); i += 128) {
      const int t = i / (DIM / 4), d = (i % (DIM / 4)) * 4;
      copy16(ks + t * DIM + d, k + (size_t)min(t, rows - 1) * g.row + d, t < rows);
    }
    for (int i = tid; i < C * (VT / 4); i += 128) {
      const int t = i / (VT / 4), c = (i % (VT / 4)) * 4;
      copy16(vs + t * VT + c, v + (size_t)min(t, rows - 1) * g.row + c, t < rows);
    }
    copies_commit();
  };
  issue(lo, 0);
  const int td = (tid >> 3) * 4, tv = (tid & 7) * 4;  // channels td .. + 3 and td + 64 .., columns tv .. + 3 and tv + 32 ..
  const size_t per_seq = (size_t)g.heads * VDIM * DIM;
  const float* from = (begins ? g.state + (size_t)slot * per_seq : g.carry + (g.pass & 1) * per_seq) + (size_t)col0 * DIM;
  float S[8][2 * P];
#pragma unroll
  for (int j = 0; j < 2 * P; ++j)
#pragma unroll
    for (int i = 0; i < 8; i += 4) {
      const float4 x = *reinterpret_cast<const float4*>(from + (size_t)(tv + (j & 3) + (j >> 2) * 32) * DIM + td + (i >> 2) * 64);
      S[i][j] = x.x;
      S[i + 1][j] = x.y;
      S[i + 2][j] = x.z;
      S[i + 3][j] = x.w;
    }
  const bool norms = KIND == 1 && col0 % VDIM == 0;  // this block walks the head's normalizer: thread d its channel d
  float n = 0.f;
  float* n_at = KIND == 1 ? g.norm_in + ((size_t)seq * g.heads + head) * DIM + tid : nullptr;
  if (norms) n = *n_at;
#pragma unroll 1
  for (int run = lo; run < hi; ++run) {
    const int local = run - g.run_lo, buf = (run - lo) & 1;
    if (run + 1 < hi) {
      issue(run + 1, buf ^ 1);
      copies_wait<1>();
    } else {
      copies_wait<0>();
    }
    const float total = g.totals[(size_t)local * g.heads + head];
    if (tid < C) weight[tid] = g.factors[(((size_t)local * g.heads + head) * 4 + 3) * C + tid];
    __syncthreads();
    const float* ks = sm + buf * C * (DIM + VT);
    float* vs = sm + buf * C * (DIM + VT) + C * DIM;
    int bad = 0;
    for (int i = tid; i < C * (VT / 4); i += 128) {
      const float w = weight[i / (VT / 4)];
      float4* p = reinterpret_cast<float4*>(vs) + i;
      const float4 x = *p;
      bad |= !(fabsf(x.x) <= 3.4028235e38f && fabsf(x.y) <= 3.4028235e38f && fabsf(x.z) <= 3.4028235e38f && fabsf(x.w) <= 3.4028235e38f);
      *p = make_float4(x.x * w, x.y * w, x.z * w, x.w * w);
    }
    if (__syncthreads_or(bad) && tid == 0) g.flags[(size_t)local * g.heads + head] = 1;
    // what is before the run goes out, [dim][COLS] of the block of heads that outputs takes together
    float* out = g.states + ((size_t)local * (g.heads * VDIM / COLS) + col0 / COLS) * DIM * COLS + col0 % COLS + tv;
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 2 * P; j += 4)
        *reinterpret_cast<float4*>(out + (size_t)(td + (i & 3) + (i >> 2) * 64) * COLS + (j >> 2) * 32) =
            make_float4(S[i][j], S[i][j + 1], S[i][j + 2], S[i][j + 3]);
    f32x2 acc[4][2 * P];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2 * P; ++j) acc[i][j] = 0;
#pragma unroll 8
    for (int s = 0; s < C; ++s) outer_step<P, 64, 32>(ks + s * DIM + td, vs + s * VT + tv, acc);
    float T[8][2 * P];
    outer_unpack<P>(acc, T);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 2 * P; ++j) S[i][j] = fmaf(total, S[i][j], T[i][j]);
    if (norms) {
      g.norms[((size_t)local * g.heads + head) * DIM + tid] = n;
      float own = 0.f;
#pragma unroll 8
      for (int s = 0; s < C; ++s) own = fmaf(weight[s], ks[s * DIM + tid], own);  // rows beyond the run's end are zeros
      n = fmaf(total, n, own);
    }
    __syncthreads();  // the stage and the weights are free
  }
  if (!ends || g.write_state) {
    float* to = (ends ? g.state + (size_t)slot * per_seq : g.carry + ((g.pass + 1) & 1) * per_seq) + (size_t)col0 * DIM;
#pragma unroll
    for (int j = 0; j < 2 * P; ++j)
#pragma unroll
      for (int i = 0; i < 8; i += 4)
        *reinterpret_cast<float4*>(to + (size_t)(tv + (j & 3) + (j >> 2) * 32) * DIM + td + (i >> 2) * 64) =
            make_float4(S[i][j], S[i + 1][j], S[i + 2][j], S[i + 3][j]);
  }
  if (norms) {
    *n_at = n;
    if (ends && g.write_state) g.norm_state[((size_t)slot * g.heads + head) * (DIM + 1) + tid] = n;
  }
}

// ---- outputs: 64 tokens x 128 value columns a block, 8 x 8 a thread ---------------------------------------------------
// Bound by the FMA pipe and by registers: 64 sums in 64 bits beside 64 of a run of terms leave two blocks a multiprocessor.
// First q against the state before the run, 16 channels at a time (q transposed on its way through registers, the state by
// asynchronous copies), then the run's own tokens: P^T, a thread a token t walking s downwards.  A warp's 64 columns belong to one
// head; it takes the tokens up to its last row, earlier rows with zeros of P (or, where a value is not finite, by selection).
constexpr int OSLICE = 16;  // channels brought into shared memory at a time
// whether 64 bits add up the float32 runs of terms: where float32 would leave outputs further from 64 bits than the walk's
template <int KIND> constexpr bool WIDE = KIND == 0;
template <int VDIM>
constexpr size_t OUT_SMEM = (size_t)(C * CROW + COLS / VDIM * C * TROW) * sizeof(float);
static_assert(OSLICE == PART);
static_assert(2 * OSLICE * (TROW + CROW) <= C * CROW, "the slices lie where the values go afterwards");

// A thread's 8 x 8 sums of runs of terms, in float32 pairs as outer_step leaves them, or in 64 bits
template <bool IN_64_BITS> struct RunSums {
  f32x2 sum[4][8];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[i][j] = 0;
  }
  __device__ __forceinline__ void add(f32x2 (&part)[4][8]) {  // and part is cleared
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        sum[i][j] = add2(sum[i][j], part[i][j]);
        part[i][j] = 0;
      }
  }
  __device__ __forceinline__ void scale(const float* of_row) {  // row i's factor at (i & 3) + (i >> 2) * 16
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float* f = of_row + (i >> 1) * 16 + (i & 1) * 2;
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[i][j] = fma2(sum[i][j], pack2(f[0], f[1]), 0ull);
    }
  }
  __device__ __forceinline__ void get(float (&out)[8][8]) const { outer_unpack<4>(sum, out); }
};
template <> struct RunSums<true> {
  double sum[8][8];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[i][j] = 0.0;
  }
  __device__ __forceinline__ void add(f32x2 (&part)[4][8]) {
    float own[8][8];
    outer_unpack<4>(part, own);
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[i][j] += (double)own[i][j];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) part[i][j] = 0;
  }
  __device__ __forceinline__ void scale(const float* of_row) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) sum[i][j] *= (double)of_row[(i & 3) + (i >> 2) * 16];
  }
  __device__ __forceinline__ void get(float (&out)[8][8]) const {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) out[i][j] = (float)sum[i][j];
  }
};

template <int VDIM, int KIND>
__global__ void __launch_bounds__(128, WIDE<KIND> ? 2 : 3) chunk_outputs_kernel(ChunkArgs g) {
  constexpr int HB = COLS / VDIM;
  extern __shared__ __align__(16) float sm[];
  float* qs = sm;                                 // [2][OSLICE][TROW], then the values [C][CROW] over both
  float* ss = sm + 2 * OSLICE * TROW;             // [2][OSLICE][CROW]
  float* Pt = sm + C * CROW;                      // [HB][C][TROW]: row s, column t
  __shared__ float as[HB][C], bs[HB][C], G[HB][C], nq[KIND == 1 ? C : 1];
  pdl_launch_dependents();
  pdl_wait();
  const int local = blockIdx.x, run = g.run_lo + local, head0 = blockIdx.y * HB, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = g.runs[2 * run], rows = g.runs[2 * run + 1] - row0;
  const int kh = head0 / (g.heads / g.key_heads);
  const float* q = g.q + (size_t)row0 * g.row + (size_t)kh * DIM;
  const float* S = g.states + ((size_t)local * gridDim.y + blockIdx.y) * DIM * COLS;
  float4 pq[2];
  auto fetch_q = [&](int d0) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int t = (tid >> 2) + 32 * i;
      pq[i] = t < rows ? *reinterpret_cast<const float4*>(q + (size_t)t * g.row + d0 + (tid & 3) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
  };
  auto put_q = [&](int buf) {
    float* p = qs + buf * OSLICE * TROW + (tid & 3) * 4 * TROW + (tid >> 2);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      p[32 * i] = pq[i].x;
      p[32 * i + TROW] = pq[i].y;
      p[32 * i + 2 * TROW] = pq[i].z;
      p[32 * i + 3 * TROW] = pq[i].w;
    }
  };
  auto issue_s = [&](int d0, int buf) {
    float* p = ss + buf * OSLICE * CROW;
    for (int i = tid; i < OSLICE * (COLS / 4); i += 128) {
      const int d = i / (COLS / 4), c = (i % (COLS / 4)) * 4;
      copy16(p + d * CROW + c, S + (size_t)(d0 + d) * COLS + c, true);
    }
    copies_commit();
  };
  issue_s(0, 0);
  fetch_q(0);
  for (int i = tid; i < HB * C; i += 128) {
    const float* f = g.factors + ((size_t)local * g.heads + head0 + i / C) * 4 * C + i % C;
    as[i / C][i % C] = f[0];
    bs[i / C][i % C] = f[C];
    G[i / C][i % C] = f[2 * C];
  }
  put_q(0);
  __syncthreads();
  double p_sum = 0.0;
  if (tid < HB * C) {  // P^T[s][t] = b_s a_(s+1) .. a_t (q_t . k_s)
    const int h = tid / C, t = tid % C;
    const float* raw = g.scores + ((size_t)local * g.key_heads + kh) * C * C + t;
    float* p = Pt + h * C * TROW + t;
    double e = 1.0;
#pragma unroll 8
    for (int s = C - 1; s >= 0; --s) {
      const float x = raw[s * C];
      const float w = s <= t ? (float)(x * (e * bs[h][s])) : 0.f;
      if (s <= t) e *= as[h][s];
      p[s * TROW] = w;
      p_sum += w;
    }
  }
  const int tm = (warp >> 1) * 32 + (lane >> 3) * 4, tn = (warp & 1) * 64 + (lane & 7) * 4;
  const int my_head = (warp & 1) * 64 / VDIM;  // of the block's
  f32x2 part[4][8];
  RunSums<WIDE<KIND>> sums;
  sums.clear();
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) part[i][j] = 0;
  double own_nq = 0.0;  // KIND 1, threads 0..63: q_t . n
  const float* n_before = KIND == 1 ? g.norms + ((size_t)local * g.heads + head0) * DIM : nullptr;
#pragma unroll 1
  for (int d0 = 0; d0 < DIM; d0 += OSLICE) {
    const int buf = (d0 / OSLICE) & 1;
    const bool more = d0 + OSLICE < DIM;
    copies_wait<0>();
    __syncthreads();  // this slice is there, and everyone is done with the one before it
    if (more) {
      issue_s(d0 + OSLICE, buf ^ 1);
      fetch_q(d0 + OSLICE);
    }
    const float* x = qs + buf * OSLICE * TROW;
    const float* y = ss + buf * OSLICE * CROW;
#pragma unroll
    for (int d = 0; d < OSLICE; ++d) outer_step<4, 16, 32>(x + d * TROW + tm, y + d * CROW + tn, part);
    sums.add(part);
    if (KIND == 1 && tid < C) {
#pragma unroll
      for (int d = 0; d < OSLICE; ++d) own_nq = fma((double)x[d * TROW + tid], (double)n_before[d0 + d], own_nq);
    }
    if (more) put_q(buf ^ 1);
  }
  __syncthreads();  // the slices are free: the values go there
  for (int i = tid; i < C * (COLS / 4); i += 128) {
    const int t = i / (COLS / 4), c = (i % (COLS / 4)) * 4;
    copy16(sm + t * CROW + c, g.v + (size_t)(row0 + min(t, rows - 1)) * g.v_row + (size_t)head0 * VDIM + c, t < rows);
  }
  copies_commit();
  sums.scale(G[my_head] + tm);  // G_t times what the state gives
  if (KIND == 1 && tid < C) {  // of n_t . q_t, what divides the row; here, since a load between the row's stores would wait for each
    const float least = tid < rows ? g.gates[((size_t)(row0 + tid) * g.heads + head0) * 3 + 2] : 1.f;
    nq[tid] = 1.f / (fmaxf(fabsf((float)fma((double)G[0][tid], own_nq, p_sum)), least) + 1e-6f);
  }
  const bool bad = g.flags[(size_t)local * g.heads + head0 + my_head] != 0;
  copies_wait<0>();
  __syncthreads();
  const float* p = Pt + my_head * C * TROW + tm;
  const int reach = (warp >> 1) * 32 + 32;
  float acc[8][8];
  if (!bad) {
#pragma unroll 1
    for (int s0 = 0; s0 < reach; s0 += PART) {
#pragma unroll 8
      for (int s = s0; s < s0 + PART; ++s) outer_step<4, 16, 32>(p + s * TROW, sm + s * CROW + tn, part);
      sums.add(part);
    }
    sums.get(acc);
  } else {
    sums.get(acc);
    for (int s = 0; s < reach; ++s)
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (s <= tm + (i & 3) + (i >> 2) * 16) {
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(p[s * TROW + (i & 3) + (i >> 2) * 16], sm[s * CROW + tn + (j & 3) + (j >> 2) * 32], acc[i][j]);
        }
  }
  const float skip = KIND == 2 ? g.d_skip[head0 + my_head] : 0.f;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int t = tm + (i & 3) + (i >> 2) * 16;
    if (t >= rows) continue;
    float scale = 1.f;
    if (KIND == 1) scale = nq[t];
    float* out = g.o + (size_t)(row0 + t) * g.heads * VDIM + (size_t)head0 * VDIM + tn;
#pragma unroll
    for (int j = 0; j < 8; j += 4) {
      float4 x = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
      if (KIND == 1) x = make_float4(x.x * scale, x.y * scale, x.z * scale, x.w * scale);
      if (KIND == 2) {
        const float4 v = *reinterpret_cast<const float4*>(sm + t * CROW + tn + (j >> 2) * 32);
        x = make_float4(fmaf(skip, v.x, x.x), fmaf(skip, v.y, x.y), fmaf(skip, v.z, x.z), fmaf(skip, v.w, x.w));
      }
      *reinterpret_cast<float4*>(out + (j >> 2) * 32) = x;
    }
  }
}

// ---- the delta rule's triangles: a block a run and head -----------------------------------------------------------------
// k . k^T as the scores, then the inverse of the 64 x 64 triangle by blocks of 16: the diagonal ones by substitution,
// a thread a column; those below, diagonal by diagonal, T_ij = -T_ii sum_(j <= m < i) A_im T_mj.  A row takes no term of a later one.
__global__ void __launch_bounds__(128) chunk_solve_kernel(ChunkArgs g) {
  __shared__ __align__(16) double sm[2 * C * SROW];  // slices of k, then T over them
  __shared__ float A[C][C + 1], W[3][16][16], as[C], bt[C];
  constexpr int TP = C + 1;
  static_assert(C * TP <= 2 * 2 * C * SROW, "T lies where the slices were");
  float* T = reinterpret_cast<float*>(sm);
  pdl_wait();
  const int local = blockIdx.x, run = g.run_lo + local, head = blockIdx.y, kh = head / (g.heads / g.key_heads), tid = threadIdx.x;
  const int row0 = g.runs[2 * run], end = g.runs[2 * run + 1], rows = end - row0;
  if (tid < C) {
    const size_t at = (size_t)(row0 + tid) * g.heads + head;
    as[tid] = tid < rows ? g.decay[at] : 1.f;
    bt[tid] = tid < rows ? g.gates[at] : 0.f;
  }
  const int tx = tid & 15;  // rows t = product_row(i), columns s = tx + 16 j
  double sum[8][4];
  const float* k = g.k + (size_t)row0 * g.row + (size_t)kh * DIM;
  run_products<true>(k, k, g.row, rows, sm, sum);
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) A[product_row(i)][tx + 16 * j] = (float)sum[i][j];
  for (int i = tid; i < C * TP; i += 128) T[i] = 0.f;
  __syncthreads();
  if (tid < C) {  // a row a thread, s downwards
    double e = bt[tid];
    for (int s = tid - 1; s >= 0; --s) {
      e *= as[s + 1];
      A[tid][s] = (float)(A[tid][s] * e);
    }
  }
  __syncthreads();
  if (tid < C) {  // the diagonal blocks
    const int base = tid & ~15, c = tid & 15;
    float x[16];
#pragma unroll
    for (int t = 0; t < 16; ++t) {
      float y = t == c ? 1.f : 0.f;
#pragma unroll
      for (int s = 0; s < t; ++s)
        if (s >= c) y = fmaf(-A[base + t][base + s], x[s], y);
      x[t] = y;
      T[(base + t) * TP + tid] = y;
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int far = 1; far < 4; ++far) {
    const int items = (4 - far) * 256;
    for (int e = tid; e < items; e += 128) {  // W_b = sum_m A_im T_mj for j = b, i = b + far
      const int b = e >> 8, r = (e >> 4) & 15, c = e & 15, i0 = (b + far) * 16 + r, j0 = b * 16;
      float y = 0.f;
#pragma unroll 16
      for (int m = 0; m < far * 16; ++m) y = fmaf(A[i0][j0 + m], T[(j0 + m) * TP + j0 + c], y);
      W[b][r][c] = y;
    }
    __syncthreads();
    for (int e = tid; e < items; e += 128) {
      const int b = e >> 8, r = (e >> 4) & 15, c = e & 15, i0 = (b + far) * 16;
      float y = 0.f;
#pragma unroll
      for (int m = 0; m < 16; ++m)
        if (m <= r) y = fmaf(-T[(i0 + r) * TP + i0 + m], W[b][m][c], y);
      T[(i0 + r) * TP + b * 16 + c] = y;
    }
    __syncthreads();
  }
  pdl_launch_dependents();
  float* out = g.solve + ((size_t)local * g.heads + head) * C * C;
  for (int i = tid; i < C * C; i += 128) {
    const int s = i / C, t = i % C;
    out[i] = s <= t ? T[t * TP + s] * bt[s] : 0.f;
  }
}

// ---- the delta rule's states: 128 key channels x 16 value columns a block, 4 x 4 a thread ---------------------------------
// As chunk_states, a sequence's runs in order, with U in front of every run's part of the state; three products in a row that wait
// for one another, so narrow columns and more blocks.  Bound by what shared memory returns (half a word a multiply-add) and by the
// three products' order: 4.6 us a run of 64 tokens, which the walk takes 28 us for (one sequence, 16 heads of 128: 149 us of
// 2,048 tokens; the walk 912).
constexpr int DVT = 16, KROW = DIM + 4;
constexpr size_t DELTA_SMEM = (size_t)(2 * C * KROW + 2 * C * DVT + C * TROW + DVT * KROW + C * DVT) * sizeof(float);

__global__ void __launch_bounds__(128, 2) delta_states_kernel(ChunkArgs g) {
  constexpr int VDIM = 128;
  extern __shared__ __align__(16) float sm[];
  float* kbuf = sm;                      // [2][C][KROW]
  float* vbuf = kbuf + 2 * C * KROW;     // [2][C][DVT]: v, then Y in place
  float* ts = vbuf + 2 * C * DVT;        // [C][TROW]: T', row s
  float* st = ts + C * TROW;             // [DVT][KROW]: the state, a row a column
  float* uw = st + DVT * KROW;           // [C][DVT]: U times the decays behind it
  __shared__ float weight[C], upto[C];
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.y, tid = threadIdx.x;
  const int lo = max(g.first_run[seq], g.run_lo), hi = min(g.first_run[seq + 1], g.run_hi);
  if (lo >= hi) return;
  const int slot = __ldcg(g.slots + seq);
  if (!FMS_IN(slot, g.n_slots)) return;
  const bool begins = lo == g.first_run[seq], ends = hi == g.first_run[seq + 1];
  const int col0 = blockIdx.x * DVT, head = col0 / VDIM, kh = head / (g.heads / g.key_heads);
  auto issue = [&](int run, int buf) {
    const int row0 = g.runs[2 * run], rows = g.runs[2 * run + 1] - row0;
    const float* k = g.k + (size_t)row0 * g.row + (size_t)kh * DIM;
    const float* v = g.v + (size_t)row0 * g.row + col0;
    for (int i = tid; i < C * (DIM / 4); i += 128) {
      const int t = i / (DIM / 4), d = (i % (DIM / 4)) * 4;
      copy16(kbuf + (buf * C + t) * KROW + d, k + (size_t)min(t, rows - 1) * g.row + d, t < rows);
    }
    for (int i = tid; i < C * (DVT / 4); i += 128) {
      const int t = i / (DVT / 4), c = (i % (DVT / 4)) * 4;
      copy16(vbuf + (buf * C + t) * DVT + c, v + (size_t)min(t, rows - 1) * g.row + c, t < rows);
    }
  };
  auto issue_solve = [&](int run) {
    const float* from = g.solve + ((size_t)(run - g.run_lo) * g.heads + head) * C * C;
    for (int i = tid; i < C * (C / 4); i += 128) copy16(ts + i / (C / 4) * TROW + i % (C / 4) * 4, from + i * 4, true);
  };
  issue(lo, 0);
  issue_solve(lo);
  copies_commit();
  const int td = (tid >> 2) * 4, tv = (tid & 3) * 4;   // of the state: channels td .. + 3, columns tv .. + 3
  const int ky = tid >> 3, kx = tid & 7;               // of Y: tokens ky + 16 i, columns kx + 8 j
  const int ut = (tid >> 3) * 4, uc = (tid & 7) * 2;   // of U: tokens ut .. + 3, columns uc, uc + 1
  const size_t per_seq = (size_t)g.heads * VDIM * DIM;
  const float* from = (begins ? g.state + (size_t)slot * per_seq : g.carry + (g.pass & 1) * per_seq) + (size_t)col0 * DIM;
  float S[4][4];  // [channel][column]
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const float4 x = *reinterpret_cast<const float4*>(from + (size_t)(tv + j) * DIM + td);
    S[0][j] = x.x;
    S[1][j] = x.y;
    S[2][j] = x.z;
    S[3][j] = x.w;
  }
#pragma unroll 1
  for (int run = lo; run < hi; ++run) {
    const int local = run - g.run_lo, buf = (run - lo) & 1;
    const int row0 = g.runs[2 * run], rows = g.runs[2 * run + 1] - row0;
    const float* ks = kbuf + buf * C * KROW;
    float* vs = vbuf + buf * C * DVT;
    const float total = g.totals[(size_t)local * g.heads + head];
    if (tid < C) {
      const float* f = g.factors + ((size_t)local * g.heads + head) * 4 * C + tid;
      upto[tid] = f[2 * C];
      weight[tid] = f[3 * C];
    }
    float* out = g.states + ((size_t)local * (g.heads * VDIM / COLS) + col0 / COLS) * DIM * COLS + col0 % COLS + tv;
#pragma unroll
    for (int i = 0; i < 4; ++i)  // what is before the run goes out, and to where this block's threads read it
      *reinterpret_cast<float4*>(out + (size_t)(td + i) * COLS) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(st + (tv + j) * KROW + td) = make_float4(S[0][j], S[1][j], S[2][j], S[3][j]);
    copies_wait<0>();
    __syncthreads();
    if (run + 1 < hi) {
      issue(run + 1, buf ^ 1);
      copies_commit();
    }
    // Y = V - G (K S)
    f32x2 even[4][2], odd[4][2];  // channels 0, 1 and 2, 3 of every four
#pragma unroll
    for (int i = 0; i < 4; ++i) even[i][0] = even[i][1] = odd[i][0] = odd[i][1] = 0;
#pragma unroll 8
    for (int d = 0; d < DIM; d += 4) {
      ulonglong2 x[4], y[2];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const ulonglong2*>(ks + (ky + 16 * i) * KROW + d);
#pragma unroll
      for (int j = 0; j < 2; ++j) y[j] = *reinterpret_cast<const ulonglong2*>(st + (kx + 8 * j) * KROW + d);
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          even[i][j] = fma2(x[i].x, y[j].x, even[i][j]);
          odd[i][j] = fma2(x[i].y, y[j].y, odd[i][j]);
        }
    }
    int bad = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        float a, b;
        unpack2(add2(even[i][j], odd[i][j]), a, b);
        float* y = vs + (ky + 16 * i) * DVT + kx + 8 * j;
        const float x = fmaf(-upto[ky + 16 * i], a + b, *y);
        *y = x;
        bad |= !(fabsf(x) <= 3.4028235e38f);
      }
    bad = __syncthreads_or(bad);
    // U = T' Y: rows up to the warp's last, later ones with zeros of T' (or, where a value is not finite, by selection)
    float U[4][2], part[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) U[i][0] = U[i][1] = part[i][0] = part[i][1] = 0.f;
    const int reach = (tid >> 5) * 16 + 16;
#pragma unroll 1
    for (int s0 = 0; s0 < reach; s0 += PART) {
#pragma unroll
      for (int s = s0; s < s0 + PART; ++s) {
        const float4 x = *reinterpret_cast<const float4*>(ts + s * TROW + ut);
        const float2 y = *reinterpret_cast<const float2*>(vs + s * DVT + uc);
        const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (!bad || s <= ut + i) {
            part[i][0] = fmaf(xs[i], y.x, part[i][0]);
            part[i][1] = fmaf(xs[i], y.y, part[i][1]);
          }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        U[i][0] += part[i][0];
        U[i][1] += part[i][1];
        part[i][0] = part[i][1] = 0.f;
      }
    }
    bad = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int t = ut + i;
      const float w = weight[t];
      *reinterpret_cast<float2*>(uw + t * DVT + uc) = make_float2(U[i][0] * w, U[i][1] * w);
      if (t < rows) *reinterpret_cast<float2*>(g.o + (size_t)(row0 + t) * g.heads * VDIM + col0 + uc) = make_float2(U[i][0], U[i][1]);
      bad |= !(fabsf(U[i][0]) <= 3.4028235e38f && fabsf(U[i][1]) <= 3.4028235e38f);
    }
    if (__syncthreads_or(bad) && tid == 0) g.flags[(size_t)local * g.heads + head] = 1;
    if (run + 1 < hi) {
      issue_solve(run + 1);
      copies_commit();
    }
    // S = total S + K^T (U times the decays behind it)
    f32x2 acc[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0;
#pragma unroll 8
    for (int s = 0; s < C; ++s) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(ks + s * KROW + td);
      const ulonglong2 y = *reinterpret_cast<const ulonglong2*>(uw + s * DVT + tv);
      const f32x2 z0 = swapped(y.x), z1 = swapped(y.y);
      acc[0][0] = fma2(x.x, y.x, acc[0][0]);
      acc[0][1] = fma2(x.x, z0, acc[0][1]);
      acc[0][2] = fma2(x.x, y.y, acc[0][2]);
      acc[0][3] = fma2(x.x, z1, acc[0][3]);
      acc[1][0] = fma2(x.y, y.x, acc[1][0]);
      acc[1][1] = fma2(x.y, z0, acc[1][1]);
      acc[1][2] = fma2(x.y, y.y, acc[1][2]);
      acc[1][3] = fma2(x.y, z1, acc[1][3]);
    }
    float own[4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        unpack2(acc[i][2 * j], own[2 * i][2 * j], own[2 * i + 1][2 * j + 1]);
        unpack2(acc[i][2 * j + 1], own[2 * i][2 * j + 1], own[2 * i + 1][2 * j]);
      }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) S[i][j] = fmaf(total, S[i][j], own[i][j]);
    __syncthreads();  // the stage, the state's copy, U and the factors are free
  }
  if (!ends || g.write_state) {
    float* to = (ends ? g.state + (size_t)slot * per_seq : g.carry + ((g.pass + 1) & 1) * per_seq) + (size_t)col0 * DIM;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      *reinterpret_cast<float4*>(to + (size_t)(tv + j) * DIM + td) = make_float4(S[0][j], S[1][j], S[2][j], S[3][j]);
  }
}

template <int VDIM, int KIND, int VT>
int launch_states(const ChunkArgs& g, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(chunk_states_kernel<VDIM, KIND, VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STATES_SMEM<VT>);
    if (e != cudaSuccess) return fms_fail("chunk_scan: shared memory refused: %s", cudaGetErrorString(e));
    configured = true;
  }
  fms_launch(chunk_states_kernel<VDIM, KIND, VT>, dim3(g.heads * VDIM / VT, g.n_seqs), dim3(128), STATES_SMEM<VT>, stream, g);
  return 0;
}

// A block walks a sequence's runs one by one: 32 columns a block instead of 64 give twice the blocks, whose instructions fill the gaps
// of one another (two prompts of 32 heads, 128 blocks of 64 or 256 of 32: 94 -> 78 us of 1,700 tokens; one of 128 heads of 64 values:
// 167 -> 161 of 2,048).  Whole layers, 16 blocks of 64 a sequence, 32 columns' time over that of 64, in the three kinds alike: 64 blocks
// 0.86-0.99 (2,048 and 640 tokens), 128 0.92-1.00, 144 0.86-0.98, 160 0.94-0.98, 224 0.94-0.96, 384 0.89-0.98, 448 0.87-1.03 (1,100 and 520
// tokens), 1,024 0.85-1.00, 1,536 0.84-1.02.  So the line has nothing slower on its side; beyond it 32 would mostly win as well.
bool columns_32(const ChunkArgs& g, int vdim) { return (long)g.n_seqs * g.heads * vdim / 64 <= 148; }

template <int VDIM, int KIND>
int launch_passes(ChunkArgs g, int n_runs, int pass_runs, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(chunk_outputs_kernel<VDIM, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OUT_SMEM<VDIM>);
    if (KIND == 3 && e == cudaSuccess) e = cudaFuncSetAttribute(delta_states_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DELTA_SMEM);
    if (e != cudaSuccess) return fms_fail("chunk_scan: shared memory refused: %s", cudaGetErrorString(e));
    configured = true;
  }
  for (int lo = 0; lo < n_runs; lo += pass_runs) {
    g.pass = lo / pass_runs;
    g.run_lo = lo;
    g.run_hi = lo + pass_runs < n_runs ? lo + pass_runs : n_runs;
    const int n = g.run_hi - lo;
    fms_launch(chunk_scores_kernel<KIND>, dim3(n, g.key_heads), dim3(128), 0, stream, g);
    if constexpr (KIND == 3) {
      fms_launch(chunk_solve_kernel, dim3(n, g.heads), dim3(128), 0, stream, g);
      fms_launch(delta_states_kernel, dim3(g.heads * VDIM / DVT, g.n_seqs), dim3(128), DELTA_SMEM, stream, g);
      ChunkArgs u = g;
      u.v = g.o;
      u.v_row = (long)g.heads * VDIM;
      fms_launch(chunk_outputs_kernel<VDIM, KIND>, dim3(n, g.heads * VDIM / COLS), dim3(128), OUT_SMEM<VDIM>, stream, u);
    } else {
      if (columns_32(g, VDIM) ? launch_states<VDIM, KIND, 32>(g, stream) : launch_states<VDIM, KIND, 64>(g, stream)) return 1;
      fms_launch(chunk_outputs_kernel<VDIM, KIND>, dim3(n, g.heads * VDIM / COLS), dim3(128), OUT_SMEM<VDIM>, stream, g);
    }
    if (fms_launch_status("chunk_scan")) return 1;
  }
  return 0;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }
}  // namespace

FMS_API int fms_chunk_scan_tokens() { return C; }
// Whether heads of these sizes, `shared` of them to a key head, go through the kernels above.
FMS_API int fms_chunk_scan_takes(int dim, int vdim, int shared) {
  return dim == DIM && (vdim == 128 || (vdim == 64 && shared % 2 == 0)) ? 1 : 0;
}

// kind, q, k, v, row, gates and the rest: see ChunkArgs and the head of this file.  runs, first_run: the step's rows cut into runs
// of fms_chunk_scan_tokens() rows of one sequence.  pass_runs: how many runs' states the scratch holds; with fewer than n_runs,
// `carry` is needed.  For kind 1 norm_in holds n before the step and is written.
FMS_API int fms_chunk_scan(int kind, const float* q, const float* k, const float* v, long row, const int* runs, const int* first_run,
                           int n_runs, int pass_runs, const int* slots, int n_seqs, const float* decay, const float* gates,
                           float* norm_in, float* norm_state, const void* dt_raw, int dt_dtype, long dt_stride, const float* dt_bias,
                           const float* a_log, const float* d_skip, float* state, float* carry, float* scores, float* factors,
                           float* totals, float* states, float* norms, float* solve, int* flags, float* o, int heads, int key_heads, int dim, int vdim,
                           int write_state, int n_slots, cudaStream_t stream) {
  if (n_runs <= 0 || n_seqs <= 0) return 0;
  if (heads <= 0 || key_heads <= 0 || heads % key_heads || !fms_chunk_scan_takes(dim, vdim, heads / key_heads) || (kind != 2 && vdim != 128))
    return fms_fail("chunk_scan: %d heads over %d, dim %d, vdim %d", heads, key_heads, dim, vdim);
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || row % 4 || !aligned16(state) || !aligned16(states) || (carry && !aligned16(carry)))
    return fms_fail("chunk_scan: rows of %ld values, or a pointer, not on 16 bytes", row);
  if (pass_runs <= 0 || (pass_runs < n_runs && carry == nullptr)) return fms_fail("chunk_scan: %d runs of %d a pass without a carry", pass_runs, n_runs);
  if (n_seqs > 65535 || heads > 65535) return fms_fail("chunk_scan: %d sequences, %d heads", n_seqs, heads);
  if (!scores || !factors || !states || !totals || !flags || (kind == 0 && !decay) || (kind == 1 && (!gates || !norm_in || !norm_state || !norms)) ||
      (kind == 3 && (!decay || !gates || !solve)) || (kind == 2 && (!dt_raw || !dt_bias || !a_log || !d_skip)))
    return fms_fail("chunk_scan: kind %d without what it reads", kind);
  if (kind == 2 && dt_dtype != FMS_F32 && dt_dtype != FMS_BF16) return fms_fail("chunk_scan: dtype code %d", dt_dtype);
  ChunkArgs g = {};
  g.q = q; g.k = k; g.v = v; g.row = g.v_row = row; g.solve = solve; g.runs = runs; g.first_run = first_run; g.slots = slots; g.decay = decay; g.gates = gates;
  g.norm_in = norm_in; g.norm_state = norm_state; g.dt_raw = dt_raw; g.dt_bias = dt_bias; g.a_log = a_log; g.d_skip = d_skip;
  g.dt_stride = dt_stride; g.dt_is_bf16 = dt_dtype == FMS_BF16; g.state = state; g.carry = carry; g.scores = scores; g.factors = factors;
  g.states = states; g.norms = norms; g.totals = totals; g.flags = flags; g.o = o; g.heads = heads; g.key_heads = key_heads;
  g.n_seqs = n_seqs; g.n_slots = n_slots; g.write_state = write_state;
  if (kind == 0) return launch_passes<128, 0>(g, n_runs, pass_runs, stream);
  if (kind == 1) return launch_passes<128, 1>(g, n_runs, pass_runs, stream);
  if (kind == 2) return vdim == 128 ? launch_passes<128, 2>(g, n_runs, pass_runs, stream) : launch_passes<64, 2>(g, n_runs, pass_runs, stream);
  if (kind == 3) return launch_passes<128, 3>(g, n_runs, pass_runs, stream);
  return fms_fail("chunk_scan: kind %d", kind);
}
