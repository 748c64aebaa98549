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
// The products are float32 products on the tensor cores: every operand is the sum of three bfloat16 (8 bits of it each, 24 in
// all), and the six products of parts that matter are added in float32 (what is left out is 2^-24 of a product and less, as much as
// float32 rounds).  On the FMA pipe shared memory returns its 128 bytes a cycle as slowly as the pipe multiplies (8 x 8 elements a
// thread), and a single prompt's states are few warps' work.  Products of decays are taken as products (no logarithms: a decay of
// zero and a run of tiny ones need no case), and a token's values never touch earlier tokens' rows, not even times zero.  The
// states of the runs of one pass lie in at most pass_runs runs' worth of scratch; longer steps take several passes, between which the
// one sequence that a boundary cuts has its state in `carry`.
//
// KIND 0: a = decay[head], b = 1.  KIND 1: (a, b, e) = gates[token, head]; a normalizer n_t = a n + b k beside S, and o is divided
// by max(|n . q|, e) + 1e-6.  KIND 2: a = exp(-exp(a_log) dt), b = dt = softplus(raw + bias), and o += d_skip v; key heads
// are shared by groups of heads.
#include "common.cuh"

namespace {
constexpr int C = 64;        // tokens of a run
constexpr int COLS = 128;    // value columns of a block of outputs: one head of 128 values or two of 64
constexpr int DIM = 128;     // key channels
constexpr int ROW128 = 128 + 8, ROW64 = 64 + 8;  // strides of tiles of 128 and of 64 values a row

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
  float* state;    // [slots, heads, vdim, dim]
  float* carry;    // [2, heads, vdim, dim], written by every other pass, or null (one pass)
  float* scores;   // scratch: [runs of a pass, key heads, C, C], element [s][t], quarters with s > t left out
  float* factors;  // scratch: [runs of a pass, heads, 4, C]: a, b, G, D(C, .)
  float* totals;   // scratch: [runs of a pass, heads]: G_C
  float* states;   // scratch: [runs of a pass, heads, vdim, dim]
  float* norms;    // scratch, KIND 1: [runs of a pass, heads, dim]
  int* flags;      // scratch: [runs of a pass, heads]: a value of the run's is not finite
  float* o;        // [tokens, heads * vdim]
  int heads, key_heads, n_seqs, n_slots, write_state;
  int run_lo, run_hi, pass;  // this pass
};

// ---- float32 operands in three bfloat16 parts, tiles in shared memory [part][row][stride] ------------------------------
typedef __nv_bfloat16 bf16;
constexpr int PARTS = 3;

__device__ __forceinline__ uint32_t pack(float x, float y) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t*>(&v);
}
// two neighbouring values into the parts' words
__device__ __forceinline__ void split2(float x, float y, uint32_t (&w)[PARTS]) {
#pragma unroll
  for (int p = 0; p < PARTS; ++p) {
    w[p] = pack(x, y);
    x -= __uint_as_float(w[p] << 16);  // exact: the remainder has fewer bits than the value
    y -= __uint_as_float(w[p] & 0xffff0000u);
  }
}
// four neighbouring values at `at` of a tile whose parts lie `part` elements apart
__device__ __forceinline__ void put4(bf16* at, int part, float4 v) {
  uint32_t a[PARTS], b[PARTS];
  split2(v.x, v.y, a);
  split2(v.z, v.w, b);
#pragma unroll
  for (int p = 0; p < PARTS; ++p) *reinterpret_cast<uint2*>(at + p * part) = make_uint2(a[p], b[p]);
}
template <bool TRANS>
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], const bf16* p) {
  if (TRANS)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(smem_u32(p)));
}
// The 16 x 16 operand A at (m, k): stored [m][k], or [k][m] (ACROSS).  Rows of every tile are 16 bytes longer than a multiple of 64 of
// them: the eight rows of a matrix meet different banks.
template <bool ACROSS>
__device__ __forceinline__ void load_a(uint32_t (&r)[4], const bf16* tile, int stride, int m, int k, int lane) {
  if (ACROSS) ldmatrix4<true>(r, tile + (k + (lane & 7) + ((lane >> 4) << 3)) * stride + m + ((lane >> 3) & 1) * 8);
  else ldmatrix4<false>(r, tile + (m + (lane & 15)) * stride + k + (lane >> 4) * 8);
}
// The operands B of two neighbouring 8 columns at (n, k): stored [n][k], or [k][n] (ACROSS)
template <bool ACROSS>
__device__ __forceinline__ void load_b(uint32_t (&r)[4], const bf16* tile, int stride, int n, int k, int lane) {
  if (ACROSS) ldmatrix4<true>(r, tile + (k + (lane & 7) + ((lane >> 3) & 1) * 8) * stride + n + (lane >> 4) * 8);
  else ldmatrix4<false>(r, tile + (n + (lane & 7) + ((lane >> 4) << 3)) * stride + k + ((lane >> 3) & 1) * 8);
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// acc [MT x 16 rows][NT x 8 columns] += A[m0 .., ka ..] B[kb .., n0 ..] for 16 k: six products of parts, the smallest first.
// Element e of a lane: row lane / 4 + 8 (e / 2), column 2 (lane % 4) + e % 2 of its 16 x 8.
template <int MT, int NT, bool A_ACROSS, bool B_ACROSS>
__device__ __forceinline__ void step16(float (&acc)[MT][NT][4], const bf16* a, int a_part, int a_stride, int m0, int ka, const bf16* b,
                                       int b_part, int b_stride, int n0, int kb, int lane) {
  uint32_t x[PARTS][MT][4];
#pragma unroll
  for (int p = 0; p < PARTS; ++p)
#pragma unroll
    for (int i = 0; i < MT; ++i) load_a<A_ACROSS>(x[p][i], a + p * a_part, a_stride, m0 + 16 * i, ka, lane);
#pragma unroll
  for (int j = 0; j < NT; j += 2) {
    uint32_t y[PARTS][4];
#pragma unroll
    for (int p = 0; p < PARTS; ++p) load_b<B_ACROSS>(y[p], b + p * b_part, b_stride, n0 + 8 * j, kb, lane);
    constexpr int PA[6] = {0, 2, 1, 0, 1, 0}, PB[6] = {2, 0, 1, 1, 0, 0};
#pragma unroll
    for (int t = 0; t < 6; ++t)
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h) mma(acc[i][j + h], x[PA[t]][i], y[PB[t]][2 * h], y[PB[t]][2 * h + 1]);
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
  // in double, rounded once: a decay's error compounds over a sequence
  const size_t at = (size_t)t * g.dt_stride + head;
  const double x = (g.dt_is_bf16 ? (double)__bfloat162float(((const __nv_bfloat16*)g.dt_raw)[at]) : (double)((const float*)g.dt_raw)[at]) +
                   (double)g.dt_bias[head];
  const double dt = x > 40.0 ? x : log1p(exp(x));
  return make_float2((float)exp(-exp((double)g.a_log[head]) * dt), (float)dt);
}

// ---- scores: [s][t] of 64 x 64 a block, a warp 32 x 32; the factors of the key head's heads, a warp a head ------------------
constexpr size_t SCORES_SMEM = (size_t)2 * PARTS * C * ROW128 * sizeof(bf16);

template <int KIND>
__global__ void __launch_bounds__(128) chunk_scores_kernel(ChunkArgs g) {
  extern __shared__ __align__(16) bf16 tiles[];
  bf16* ks = tiles;                        // [PARTS][C][ROW128]
  bf16* qs = tiles + PARTS * C * ROW128;
  pdl_launch_dependents();
  pdl_wait();
  const int run = g.run_lo + blockIdx.x, kh = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = g.runs[2 * run], end = g.runs[2 * run + 1], rows = end - row0;
  const float* q = g.q + (size_t)row0 * g.row + (size_t)kh * DIM;
  const float* k = g.k + (size_t)row0 * g.row + (size_t)kh * DIM;
#pragma unroll 4
  for (int i = tid; i < C * (DIM / 4); i += 128) {
    const int t = i / (DIM / 4), d = (i % (DIM / 4)) * 4;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    put4(ks + t * ROW128 + d, C * ROW128, t < rows ? *reinterpret_cast<const float4*>(k + (size_t)t * g.row + d) : zero);
    put4(qs + t * ROW128 + d, C * ROW128, t < rows ? *reinterpret_cast<const float4*>(q + (size_t)t * g.row + d) : zero);
  }
  const int shared = g.heads / g.key_heads;
  for (int head = kh * shared + warp; head < (kh + 1) * shared; head += 4) {  // a lane two neighbouring tokens
    const float2 w0 = token_gates<KIND>(g, row0 + 2 * lane, end, head), w1 = token_gates<KIND>(g, row0 + 2 * lane + 1, end, head);
    float upto = w0.x * w1.x, behind = upto;  // inclusive products over this lane's tokens and all earlier, all later ones
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float x = __shfl_up_sync(0xffffffffu, upto, o), y = __shfl_down_sync(0xffffffffu, behind, o);
      if (lane >= o) upto *= x;
      if (lane + o < 32) behind *= y;
    }
    float before = __shfl_up_sync(0xffffffffu, upto, 1), after = __shfl_down_sync(0xffffffffu, behind, 1);
    if (lane == 0) before = 1.f;
    if (lane == 31) after = 1.f;
    float2* f = reinterpret_cast<float2*>(g.factors + ((size_t)blockIdx.x * g.heads + head) * 4 * C) + lane;
    f[0] = make_float2(w0.x, w1.x);
    f[C / 2] = make_float2(w0.y, w1.y);
    f[2 * C / 2] = make_float2(before * w0.x, upto);
    f[3 * C / 2] = make_float2(w0.y * (w1.x * after), w1.y * after);
    if (lane == 0) {
      g.totals[(size_t)blockIdx.x * g.heads + head] = behind;
      g.flags[(size_t)blockIdx.x * g.heads + head] = 0;
    }
  }
  __syncthreads();
  const int s0 = (warp >> 1) * 32, t0 = (warp & 1) * 32;
  if (s0 > t0) return;  // tokens behind every query of this quarter: never read
  float acc[2][4][4] = {};
#pragma unroll 1
  for (int d = 0; d < DIM; d += 16)
    step16<2, 4, false, false>(acc, ks, C * ROW128, ROW128, s0, d, qs, C * ROW128, ROW128, t0, d, lane);
  float* out = g.scores + ((size_t)blockIdx.x * g.key_heads + kh) * C * C;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        *reinterpret_cast<float2*>(out + (s0 + 16 * i + (lane >> 2) + 4 * e) * C + t0 + 8 * j + 2 * (lane & 3)) = make_float2(acc[i][j][e], acc[i][j][e + 1]);
}

// ---- the states before every run: VT value columns x 128 key channels a block, a warp 32 x 32 (VT = 32: 32 x 16) -----------------
// A sequence's runs in order, the state in registers as the tensor cores leave it; the next run's keys and values are on their
// way from global memory (in registers) meanwhile.  VT = 32 where 64 would leave multiprocessors without a block.
template <int VT> constexpr size_t STATES_SMEM = (size_t)PARTS * C * (ROW128 + VT + 8) * sizeof(bf16);

template <int VDIM, int KIND, int VT>
__global__ void __launch_bounds__(256) chunk_states_kernel(ChunkArgs g) {
  constexpr int WARPS_D = 8 / (VT / 32), NT = DIM / WARPS_D / 8, VROW = VT + 8, NK = C * DIM / 4 / 256, NV = C * VT / 4 / 256;
  extern __shared__ __align__(16) bf16 tiles[];
  bf16* ks = tiles;                        // [PARTS][C][ROW128]
  bf16* vs = tiles + PARTS * C * ROW128;   // [PARTS][C][VROW], times D(C, s)
  pdl_launch_dependents();
  pdl_wait();
  const int seq = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int lo = max(g.first_run[seq], g.run_lo), hi = min(g.first_run[seq + 1], g.run_hi);
  if (lo >= hi) return;
  const int slot = __ldcg(g.slots + seq);
  if (!FMS_IN(slot, g.n_slots)) return;
  const bool begins = lo == g.first_run[seq], ends = hi == g.first_run[seq + 1];
  const int col0 = blockIdx.x * VT, head = col0 / VDIM, kh = head / (g.heads / g.key_heads);  // columns over all heads
  float4 pk[NK], pv[NV];
  float pw[NV], total_next = 0.f;
  auto fetch = [&](int run) {
    const int row0 = g.runs[2 * run], rows = g.runs[2 * run + 1] - row0;
    const float* k = g.k + (size_t)row0 * g.row + (size_t)kh * DIM;
    const float* v = g.v + (size_t)row0 * g.row + col0;
    const float* w = g.factors + (((size_t)(run - g.run_lo) * g.heads + head) * 4 + 3) * C;
#pragma unroll
    for (int n = 0; n < NK; ++n) {
      const int i = tid + 256 * n, t = i / (DIM / 4), d = (i % (DIM / 4)) * 4;
      pk[n] = t < rows ? *reinterpret_cast<const float4*>(k + (size_t)t * g.row + d) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int n = 0; n < NV; ++n) {
      const int i = tid + 256 * n, t = i / (VT / 4), c = (i % (VT / 4)) * 4;
      pv[n] = t < rows ? *reinterpret_cast<const float4*>(v + (size_t)t * g.row + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      pw[n] = w[t];
    }
    total_next = g.totals[(size_t)(run - g.run_lo) * g.heads + head];
  };
  fetch(lo);
  const int c0 = (warp / WARPS_D) * 32, d0 = (warp % WARPS_D) * (NT * 8);
  const size_t per_seq = (size_t)g.heads * VDIM * DIM;
  // element e of tile (i, j): column c0 + 16 i + lane / 4 + 8 (e / 2), channel d0 + 8 j + 2 (lane % 4) + e % 2
  const size_t mine = (size_t)(col0 + c0 + (lane >> 2)) * DIM + d0 + 2 * (lane & 3);
  const float* from = (begins ? g.state + (size_t)slot * per_seq : g.carry + (g.pass & 1) * per_seq) + mine;
  float S[2][NT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const float2 x = *reinterpret_cast<const float2*>(from + (size_t)(16 * i + 4 * e) * DIM + 8 * j);
        S[i][j][e] = x.x;
        S[i][j][e + 1] = x.y;
      }
  const bool norms = KIND == 1 && col0 % VDIM == 0 && tid < DIM;  // this thread walks the normalizer's channel tid
  float n = 0.f;
  float* n_at = KIND == 1 ? g.norm_in + ((size_t)seq * g.heads + head) * DIM + (tid % DIM) : nullptr;
  if (norms) n = *n_at;
#pragma unroll 1
  for (int run = lo; run < hi; ++run) {
    const int local = run - g.run_lo;
    const float total = total_next;
    int bad = 0;
#pragma unroll
    for (int m = 0; m < NK; ++m) {
      const int i = tid + 256 * m;
      put4(ks + (i / (DIM / 4)) * ROW128 + (i % (DIM / 4)) * 4, C * ROW128, pk[m]);
    }
#pragma unroll
    for (int m = 0; m < NV; ++m) {
      const int i = tid + 256 * m;
      const float4 x = pv[m];
      const float w = pw[m];
      bad |= !(fabsf(x.x) <= 3.3e38f && fabsf(x.y) <= 3.3e38f && fabsf(x.z) <= 3.3e38f && fabsf(x.w) <= 3.3e38f);
      put4(vs + (i / (VT / 4)) * VROW + (i % (VT / 4)) * 4, C * VROW, make_float4(x.x * w, x.y * w, x.z * w, x.w * w));
    }
    if (__syncthreads_or(bad) && tid == 0) g.flags[(size_t)local * g.heads + head] = 1;
    if (run + 1 < hi) fetch(run + 1);
    // what is before the run goes out
    float* out = g.states + (size_t)local * per_seq + mine;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; e += 2) *reinterpret_cast<float2*>(out + (size_t)(16 * i + 4 * e) * DIM + 8 * j) = make_float2(S[i][j][e], S[i][j][e + 1]);
    float T[2][NT][4] = {};
#pragma unroll 1
    for (int s = 0; s < C; s += 16)
      step16<2, NT, true, true>(T, vs, C * VROW, VROW, c0, s, ks, C * ROW128, ROW128, d0, s, lane);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) S[i][j][e] = fmaf(total, S[i][j][e], T[i][j][e]);
    if (norms) {
      g.norms[((size_t)local * g.heads + head) * DIM + tid] = n;
      const float* w = g.factors + (((size_t)local * g.heads + head) * 4 + 3) * C;
      float own = 0.f;
#pragma unroll 8
      for (int s = 0; s < C; ++s) {  // rows beyond the run's end are zeros; the three parts add up to the value
        const bf16* at = ks + s * ROW128 + tid;
        own = fmaf(w[s], __bfloat162float(at[0]) + (__bfloat162float(at[C * ROW128]) + __bfloat162float(at[2 * C * ROW128])), own);
      }
      n = fmaf(total, n, own);
    }
    __syncthreads();  // the tiles are free
  }
  if (!ends || g.write_state) {
    float* to = (ends ? g.state + (size_t)slot * per_seq : g.carry + ((g.pass + 1) & 1) * per_seq) + mine;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; e += 2) *reinterpret_cast<float2*>(to + (size_t)(16 * i + 4 * e) * DIM + 8 * j) = make_float2(S[i][j][e], S[i][j][e + 1]);
  }
  if (norms) {
    *n_at = n;
    if (ends && g.write_state) g.norm_state[((size_t)slot * g.heads + head) * (DIM + 1) + tid] = n;
  }
}

// ---- outputs: 64 tokens x 128 value columns a block, a warp 32 x 32 -----------------------------------------------------
// First q against the state before the run, 64 channels at a time, then the run's own tokens: P as [s][t], a thread a token t
// walking s downwards.  A warp's 32 columns belong to one head; it takes the tokens up to its last row, earlier rows with zeros
// of P (or, where a value is not finite, by selection).
constexpr int Q_TILE = PARTS * C * ROW64, S_TILE = PARTS * COLS * ROW64, P_TILE = PARTS * C * ROW64, V_TILE = PARTS * C * ROW128;
template <int VDIM>
constexpr size_t OUT_SMEM = sizeof(bf16) * (size_t)(Q_TILE + S_TILE > COLS / VDIM * P_TILE + V_TILE ? Q_TILE + S_TILE : COLS / VDIM * P_TILE + V_TILE);

template <int VDIM, int KIND>
__global__ void __launch_bounds__(256, 2) chunk_outputs_kernel(ChunkArgs g) {
  constexpr int HB = COLS / VDIM;
  extern __shared__ __align__(16) bf16 tiles[];
  bf16* qs = tiles;                // [PARTS][C][ROW64], then P: [HB][PARTS][C][ROW64], row s, column t
  bf16* ss = tiles + Q_TILE;       // [PARTS][COLS][ROW64]
  bf16* vs = tiles + HB * P_TILE;  // [PARTS][C][ROW128], afterwards
  __shared__ float as[HB][C], bs[HB][C], G[HB][C], nq[KIND == 1 ? C : 1];
  pdl_launch_dependents();
  pdl_wait();
  const int local = blockIdx.x, run = g.run_lo + local, head0 = blockIdx.y * HB, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int row0 = g.runs[2 * run], rows = g.runs[2 * run + 1] - row0;
  const int kh = head0 / (g.heads / g.key_heads);
  const float* q = g.q + (size_t)row0 * g.row + (size_t)kh * DIM;
  const float* S = g.states + ((size_t)local * g.heads + head0) * VDIM * DIM;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  if (tid < HB * C) {
    const float* f = g.factors + ((size_t)local * g.heads + head0 + tid / C) * 4 * C + tid % C;
    as[tid / C][tid % C] = f[0];
    bs[tid / C][tid % C] = f[C];
    G[tid / C][tid % C] = f[2 * C];
  }
  const int t0 = (warp >> 2) * 32, c0 = (warp & 3) * 32, my_head = c0 / VDIM;
  float acc[2][4][4] = {};
#pragma unroll 1
  for (int d0 = 0; d0 < DIM; d0 += 64) {
    if (d0) __syncthreads();
#pragma unroll
    for (int n = 0; n < 4; ++n) {
      const int i = tid + 256 * n, t = i / 16, d = (i % 16) * 4;
      put4(qs + t * ROW64 + d, C * ROW64, t < rows ? *reinterpret_cast<const float4*>(q + (size_t)t * g.row + d0 + d) : zero);
    }
#pragma unroll
    for (int n = 0; n < 8; ++n) {
      const int i = tid + 256 * n, c = i / 16, d = (i % 16) * 4;
      put4(ss + c * ROW64 + d, COLS * ROW64, *reinterpret_cast<const float4*>(S + (size_t)c * DIM + d0 + d));
    }
    __syncthreads();
#pragma unroll 1
    for (int d = 0; d < 64; d += 16)
      step16<2, 4, false, false>(acc, qs, C * ROW64, ROW64, t0, d, ss, COLS * ROW64, ROW64, c0, d, lane);
  }
  __syncthreads();  // q and the state have been read; P and the values go where they were
  float p_sum = 0.f;
  if (tid < HB * C) {  // P[s][t] = b_s a_(s+1) .. a_t (q_t . k_s)
    const int h = tid / C, t = tid % C;
    const float* raw = g.scores + ((size_t)local * g.key_heads + kh) * C * C + t;
    bf16* p = qs + h * P_TILE + t;
    float e = 1.f;
#pragma unroll 8
    for (int s = C - 1; s >= 0; --s) {
      float w = 0.f;
      if (s <= t) {
        w = raw[s * C] * (e * bs[h][s]);
        e *= as[h][s];
      }
      p_sum += w;
      uint32_t parts[PARTS];
      split2(w, 0.f, parts);
#pragma unroll
      for (int k = 0; k < PARTS; ++k) reinterpret_cast<uint16_t*>(p + k * C * ROW64)[s * ROW64] = (uint16_t)parts[k];
    }
  }
#pragma unroll
  for (int n = 0; n < 8; ++n) {
    const int i = tid + 256 * n, t = i / 32, c = (i % 32) * 4;
    put4(vs + t * ROW128 + c, C * ROW128, t < rows ? *reinterpret_cast<const float4*>(g.v + (size_t)(row0 + t) * g.row + (size_t)head0 * VDIM + c) : zero);
  }
  // G_t times what the state gives
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      const float x = G[my_head][t0 + 16 * i + (lane >> 2) + 4 * e];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j][e] *= x;
        acc[i][j][e + 1] *= x;
      }
    }
  if (KIND == 1) {  // n_t . q_t = G_t (n . q_t) + the sum of the row of P: a warp eight tokens
    const float4 x = reinterpret_cast<const float4*>(g.norms + ((size_t)local * g.heads + head0) * DIM)[lane];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int t = warp * 8 + i;
      const float4 y = t < rows ? reinterpret_cast<const float4*>(q + (size_t)t * g.row)[lane] : zero;
      const float sum = warp_sum(fmaf(x.x, y.x, fmaf(x.y, y.y, fmaf(x.z, y.z, x.w * y.w))));
      if (lane == 0) nq[t] = G[0][t] * sum;
    }
  }
  const bool bad = g.flags[(size_t)local * g.heads + head0 + my_head] != 0;
  __syncthreads();
  if (KIND == 1 && tid < C) nq[tid] += p_sum;
  if (!bad) {
#pragma unroll 1
    for (int s = 0; s < t0 + 32; s += 16)
      step16<2, 4, true, true>(acc, qs + my_head * P_TILE, C * ROW64, ROW64, t0, s, vs, C * ROW128, ROW128, c0, s, lane);
  } else {  // rarely: value by value, earlier rows left out
    const bf16* P = qs + my_head * P_TILE;
    const float* v = g.v + (size_t)row0 * g.row + (size_t)head0 * VDIM + c0;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = t0 + 16 * i + (lane >> 2) + 8 * (e >> 1);
        for (int s = 0; s <= min(t, rows - 1); ++s) {
          const bf16* at = P + s * ROW64 + t;
          const float p = __bfloat162float(at[0]) + (__bfloat162float(at[C * ROW64]) + __bfloat162float(at[2 * C * ROW64]));
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j][e] = fmaf(p, v[(size_t)s * g.row + 8 * j + 2 * (lane & 3) + (e & 1)], acc[i][j][e]);
        }
      }
  }
  if (KIND == 1) __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
      const int t = t0 + 16 * i + (lane >> 2) + 4 * e;
      if (t >= rows) continue;
      float scale = 1.f, skip = 0.f;
      if (KIND == 1) scale = 1.f / (fmaxf(fabsf(nq[t]), g.gates[((size_t)(row0 + t) * g.heads + head0) * 3 + 2]) + 1e-6f);
      if (KIND == 2) skip = g.d_skip[head0 + my_head];
      const size_t at = (size_t)head0 * VDIM + c0 + 2 * (lane & 3);
      float* out = g.o + (size_t)(row0 + t) * g.heads * VDIM + at;
      const float* v = g.v + (size_t)(row0 + t) * g.row + at;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float2 x = make_float2(acc[i][j][e], acc[i][j][e + 1]);
        if (KIND == 1) x = make_float2(x.x * scale, x.y * scale);
        if (KIND == 2) {
          const float2 y = *reinterpret_cast<const float2*>(v + 8 * j);
          x = make_float2(fmaf(skip, y.x, x.x), fmaf(skip, y.y, x.y));
        }
        *reinterpret_cast<float2*>(out + 8 * j) = x;
      }
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
  fms_launch(chunk_states_kernel<VDIM, KIND, VT>, dim3(g.heads * VDIM / VT, g.n_seqs), dim3(256), STATES_SMEM<VT>, stream, g);
  return 0;
}

// a block walks a sequence's runs one by one: 32 columns a block where 64 would leave multiprocessors without one
bool columns_32(const ChunkArgs& g, int vdim) { return (long)g.n_seqs * g.heads * vdim / 64 < 128; }

template <int VDIM, int KIND>
int launch_passes(ChunkArgs g, int n_runs, int pass_runs, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(chunk_outputs_kernel<VDIM, KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)OUT_SMEM<VDIM>);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(chunk_scores_kernel<KIND>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SCORES_SMEM);
    if (e != cudaSuccess) return fms_fail("chunk_scan: shared memory refused: %s", cudaGetErrorString(e));
    configured = true;
  }
  for (int lo = 0; lo < n_runs; lo += pass_runs) {
    g.pass = lo / pass_runs;
    g.run_lo = lo;
    g.run_hi = lo + pass_runs < n_runs ? lo + pass_runs : n_runs;
    const int n = g.run_hi - lo;
    fms_launch(chunk_scores_kernel<KIND>, dim3(n, g.key_heads), dim3(128), SCORES_SMEM, stream, g);
    if (columns_32(g, VDIM) ? launch_states<VDIM, KIND, 32>(g, stream) : launch_states<VDIM, KIND, 64>(g, stream)) return 1;
    fms_launch(chunk_outputs_kernel<VDIM, KIND>, dim3(n, g.heads * VDIM / COLS), dim3(256), OUT_SMEM<VDIM>, stream, g);
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
                           float* totals, float* states, float* norms, int* flags, float* o, int heads, int key_heads, int dim, int vdim,
                           int write_state, int n_slots, cudaStream_t stream) {
  if (n_runs <= 0 || n_seqs <= 0) return 0;
  if (heads <= 0 || key_heads <= 0 || heads % key_heads || !fms_chunk_scan_takes(dim, vdim, heads / key_heads) || (kind == 1 && vdim != 128))
    return fms_fail("chunk_scan: %d heads over %d, dim %d, vdim %d", heads, key_heads, dim, vdim);
  if (!aligned16(q) || !aligned16(k) || !aligned16(v) || row % 4 || !aligned16(state) || !aligned16(states) || (carry && !aligned16(carry)))
    return fms_fail("chunk_scan: rows of %ld values, or a pointer, not on 16 bytes", row);
  if (pass_runs <= 0 || (pass_runs < n_runs && carry == nullptr)) return fms_fail("chunk_scan: %d runs of %d a pass without a carry", pass_runs, n_runs);
  if (n_seqs > 65535 || heads > 65535) return fms_fail("chunk_scan: %d sequences, %d heads", n_seqs, heads);
  if (!scores || !factors || !states || !totals || !flags || (kind == 0 && !decay) || (kind == 1 && (!gates || !norm_in || !norm_state || !norms)) ||
      (kind == 2 && (!dt_raw || !dt_bias || !a_log || !d_skip)))
    return fms_fail("chunk_scan: kind %d without what it reads", kind);
  if (kind == 2 && dt_dtype != FMS_F32 && dt_dtype != FMS_BF16) return fms_fail("chunk_scan: dtype code %d", dt_dtype);
  ChunkArgs g = {};
  g.q = q; g.k = k; g.v = v; g.row = row; g.runs = runs; g.first_run = first_run; g.slots = slots; g.decay = decay; g.gates = gates;
  g.norm_in = norm_in; g.norm_state = norm_state; g.dt_raw = dt_raw; g.dt_bias = dt_bias; g.a_log = a_log; g.d_skip = d_skip;
  g.dt_stride = dt_stride; g.dt_is_bf16 = dt_dtype == FMS_BF16; g.state = state; g.carry = carry; g.scores = scores; g.factors = factors;
  g.states = states; g.norms = norms; g.totals = totals; g.flags = flags; g.o = o; g.heads = heads; g.key_heads = key_heads;
  g.n_seqs = n_seqs; g.n_slots = n_slots; g.write_state = write_state;
  if (kind == 0) return vdim == 128 ? launch_passes<128, 0>(g, n_runs, pass_runs, stream) : launch_passes<64, 0>(g, n_runs, pass_runs, stream);
  if (kind == 1) return launch_passes<128, 1>(g, n_runs, pass_runs, stream);
  if (kind == 2) return vdim == 128 ? launch_passes<128, 2>(g, n_runs, pass_runs, stream) : launch_passes<64, 2>(g, n_runs, pass_runs, stream);
  return fms_fail("chunk_scan: kind %d", kind);
}
