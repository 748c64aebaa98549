// float32 prefill attention on the tensor cores, for head sizes of 64 and 128 and an even number of query heads a key head: both
// products over operands in three bfloat16 parts (split_f32.cuh), six products of parts in accumulators of 32 terms (they cut
// their sums off), which registers add up rounded to nearest; softmax, probabilities and sums in float32 as in the kernel on the
// CUDA cores.  A block takes 64 positions by two heads (the instruction's 128 rows) and walks its keys 64 at a time:
//
//   the keys' parts -> S = Q K^T, while the values are split -> softmax -> the probabilities' parts where the keys were -> O' = P V,
//   while the next keys are on their way -> O = alpha O + O'
//
// A thread has a row and half of its scores and of its results.  One block a multiprocessor: the parts of 128 queries, 64 keys and 64
// values are 192 KB.  Bound by the steps' order, some 12,000 cycles a block of keys, of which 3,800 are products.  Measured (three
// prompts of 1,100 tokens together, 32 heads of 128 over 8): 95 us, the kernel on the CUDA cores 207; 64 tokens onto 1,000 cached ones
// 125 and 271; 17 alone 27 and 29.
// Operands that are not finite or beyond 2^30 do not split: zeros stand for them, and the rows that see them (or that they belong to)
// go on the CUDA cores instead, as do rows whose sum of probabilities is no number (a scale beyond 2^60 can make scores infinite):
// a warp a row, a lane a key, every score by the multiply-adds of the kernel there in their order.  All operands
// are split times 2^SPLIT_SCALE, so that small ones lose nothing.  A row's result depends on its own keys only, block by block of
// the cache, whatever tile it lies in.
#pragma once

constexpr int FT_THREADS = 256, FT_ATOMS = HD / 64;
constexpr int FT_QPART = FT_ATOMS * 128 * 128, FT_KPART = FT_ATOMS * BLK * 128, FT_PPART = 128 * 128;
constexpr int FT_KREGION = 3 * (FT_KPART > FT_PPART ? FT_KPART : FT_PPART);
constexpr size_t FT_SMEM = 3 * FT_QPART + FT_KREGION + 3 * FT_KPART + 1024;
constexpr int FT_O = 256;             // tensor memory: scores from column 0, results from here
constexpr int FT_PER_ROW = HD / 8;    // threads a row of keys or values, eight values each
constexpr int FT_UNITS = BLK * FT_PER_ROW / FT_THREADS;

constexpr float FT_UNSCALE = power_of_two(-2 * SPLIT_SCALE);  // of a product of two operands

// eight values to 16 bytes of each of three parts; whether they split (else zeros)
__device__ __forceinline__ bool ft_put(unsigned char* p, int part, const float* v) {
  uint4 hi, mid, lo;
  uint32_t most = 0;
  split8<SPLIT_SCALE>(v, &hi, &mid, &lo, most);
  const bool fine = !beyond<30 + SPLIT_SCALE>(most);
  if (!fine) hi = mid = lo = make_uint4(0, 0, 0, 0);
  *reinterpret_cast<uint4*>(p) = hi;
  *reinterpret_cast<uint4*>(p + part) = mid;
  *reinterpret_cast<uint4*>(p + 2 * part) = lo;
  return fine;
}
__device__ __forceinline__ void ft_read(float* v, const float* at, bool there) {
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const float4 a = there ? *reinterpret_cast<const float4*>(at) : zero, b = there ? *reinterpret_cast<const float4*>(at + 4) : zero;
  v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
  v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
}
// an accumulator of 32 terms, two steps of 16: a, b the descriptors of the first parts' first 16 terms, the others `ap`, `bp` behind it
// (in descriptors' units of 16 bytes), the second step `as`, `bs`
__device__ __forceinline__ void ft_accumulate(uint32_t d, uint64_t a, uint64_t b, uint32_t ap, uint32_t bp, uint32_t as, uint32_t bs, uint32_t idesc) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const uint64_t x = a + h * as, y = b + h * bs;
    umma(d, x + 2 * ap, y, idesc, h > 0);
    umma(d, x, y + 2 * bp, idesc, true);
    umma(d, x + ap, y + bp, idesc, true);
    umma(d, x + ap, y, idesc, true);
    umma(d, x, y + bp, idesc, true);
  }
  umma(d, a, b, idesc, true);
  umma(d, a + as, b + bs, idesc, true);
}

__global__ void __launch_bounds__(FT_THREADS, 1) attn_prefill_f32_tc_kernel(AttnArgs a, const int* __restrict__ tiles, int n_tiles,
                                                                             int n_seqs, int n_rows, int* __restrict__ error_flag) {
  extern __shared__ unsigned char smem_unaligned[];
  unsigned char* qs = reinterpret_cast<unsigned char*>(((uintptr_t)smem_unaligned + 1023) & ~(uintptr_t)1023);
  unsigned char *ks = qs + 3 * FT_QPART, *vs = ks + FT_KREGION;
  __shared__ uint64_t done_s, done_o;
  __shared__ uint32_t tmem_slot;
  __shared__ int failed_flag;
  __shared__ unsigned odd_keys[2][2];  // by the parity of the step and by halves: the block's positions whose key or value does not split
  __shared__ unsigned char odd[128];   // rows that go on the CUDA cores
  __shared__ float top[2][128], sums[2][128];
  volatile int* failed = &failed_flag;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, half = warp >> 2, row = (warp & 3) * 32 + lane;
  pdl_launch_dependents();
  if (tid == 0) {
    failed_flag = 0;
    mbar_init(&done_s, 1);
    mbar_init(&done_o, 1);
    mbar_fence_init();
  }
  if (tid < 128) odd[tid] = 0;
  if (tid < 4) odd_keys[tid >> 1][tid & 1] = 0;
  if (warp == 0) tmem_alloc(&tmem_slot, 512);
  __syncthreads();
  pdl_wait();
  const int pairs = a.nheads / 2, pair = blockIdx.x % pairs, tile = n_tiles - 1 - blockIdx.x / pairs;  // the longest tiles first
  const int seq = FMS_IN(tiles[2 * tile], n_seqs) ? tiles[2 * tile] : 0, r0 = tiles[2 * tile + 1];
  const int row_begin = a.first_row[seq], n_new = a.first_row[seq + 1] - row_begin, len = a.len_after[seq];
  const int rows_here = min(TQ, n_new - r0), slot = a.slots[seq], p_first = len - n_new + r0, p_last = p_first + rows_here - 1;
  const int head0 = 2 * pair, kvh = head0 / (a.nheads / a.kvheads), head = head0 + (row >> 6), pos = row & 63, my_pos = p_first + pos;
  const int my_first = first_visible(a, my_pos), kb_hi = p_last / BLK;
  const bool mine = pos < rows_here;
  const float* q = (const float*)a.q + (size_t)(row_begin + r0) * a.q_stride + (size_t)head0 * HD;
  const int k_row = tid / FT_PER_ROW, piece = tid % FT_PER_ROW;  // of keys and values: rows k_row, + 256 / FT_PER_ROW, ...
  constexpr int K_STEP = FT_THREADS / FT_PER_ROW;
  for (int i = tid; i < 128 * FT_PER_ROW; i += FT_THREADS) {
    const int r = i / FT_PER_ROW, c = i % FT_PER_ROW;
    float v[8];
    ft_read(v, q + (size_t)(r & 63) * a.q_stride + (r >> 6) * HD + 8 * c, (r & 63) < rows_here && FMS_IN(row_begin + r0 + (r & 63), n_rows));
    if (!ft_put(qs + (c >> 3) * (128 * 128) + r * 128 + (((c & 7) ^ (r & 7)) << 4), FT_QPART, v)) odd[r] = 1;
  }
  float x[FT_UNITS][8];
  auto read_block = [&](const void* cache, int kb, int blk) {
    const float* base = (const float*)cache + ((size_t)blk * a.kvheads + kvh) * BLK * HD;
#pragma unroll
    for (int u = 0; u < FT_UNITS; ++u) ft_read(x[u], base + (size_t)(k_row + u * K_STEP) * HD + 8 * piece, kb * BLK + k_row + u * K_STEP < len);
  };
  auto put_block = [&](unsigned char* to, int parity) {
#pragma unroll
    for (int u = 0; u < FT_UNITS; ++u) {
      const int r = k_row + u * K_STEP;
      if (!ft_put(to + (piece >> 3) * (BLK * 128) + r * 128 + (((piece & 7) ^ (r & 7)) << 4), FT_KPART, x[u]))
        atomicOr(&odd_keys[parity][r >> 5], 1u << (r & 31));
    }
  };
  // the next block of keys from kb on, or one behind the last (a block that left the window has no place in the cache)
  auto next_block = [&](int kb, int& blk) {
    for (blk = -1; kb <= kb_hi; ++kb)
      if ((blk = block_of(a, slot, kb)) >= 0) break;
    return kb;
  };
  int blk = -1, kb = next_block(first_visible(a, p_first) / BLK, blk);
  if (kb <= kb_hi) read_block(a.keys, kb, blk);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot, lane_base = (uint32_t)((warp & 3) * 32) << 16;
  float m = -INFINITY, l = 0.f, acc[HD / 2];  // l: of this thread's half of the keys
#pragma unroll
  for (int c = 0; c < HD / 2; ++c) acc[c] = 0.f;
  bool ok = true, sees_odd = false;
  for (int it = 0; kb <= kb_hi; ++it) {
    put_block(ks, it & 1);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();  // the keys' parts are there, and every row is done with the block before
    tc_fence_after();
    if (warp == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc(128, BLK);
#pragma unroll
      for (int i = 0; i < HD / 32; ++i) {  // 32 of the head's values: half of an atom's 64
        const uint32_t aq = smem_u32(qs) + (i >> 1) * (128 * 128) + (i & 1) * 64, bk = smem_u32(ks) + (i >> 1) * (BLK * 128) + (i & 1) * 64;
        ft_accumulate(tmem + i * BLK, umma_desc(aq), umma_desc(bk), FT_QPART >> 4, FT_KPART >> 4, 2, 2, idesc);
      }
      tc_commit(&done_s);
    }
    __syncwarp();
    read_block(a.values, kb, blk);
    put_block(vs, it & 1);
    const int this_kb = kb;
    kb = next_block(kb + 1, blk);
    if (kb <= kb_hi) read_block(a.keys, kb, blk);
    ok = __all_sync(0xffffffffu, ok && wait_or_abort(&done_s, it & 1, failed));
    float s[32];
#pragma unroll
    for (int j = 0; j < 32; ++j) s[j] = 0.f;
    if (ok) {
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < HD / 32; ++i) {
        float t[32];
        tmem_load_32(tmem + lane_base + i * BLK + half * 32, t);
#pragma unroll
        for (int j = 0; j < 32; ++j) s[j] += t[j];
      }
    }
    float most_here = -INFINITY;
    const int from = my_first - (this_kb * BLK + half * 32), upto = mine ? my_pos - (this_kb * BLK + half * 32) : -1;  // visible: from .. upto
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      s[j] = j >= from && j <= upto ? s[j] * FT_UNSCALE * a.scale : -INFINITY;
      most_here = fmaxf(most_here, s[j]);
    }
    top[half][row] = most_here;
    if (tid < 2) odd_keys[(it + 1) & 1][tid] = 0;  // every row has read what the step before found
    __syncthreads();
    // of this block's positions the row's own visible ones, so that nothing depends on the tile's other rows
    const unsigned own = from < 32 && upto >= 0 ? (0xffffffffu << max(from, 0)) & (0xffffffffu >> (31 - min(upto, 31))) : 0u;
    sees_odd |= (odd_keys[it & 1][half] & own) != 0;
    const float m_new = fmaxf(m, fmaxf(top[0][row], top[1][row])), m_use = m_new == -INFINITY ? 0.f : m_new;
    const float alpha = m == -INFINITY ? 0.f : expf(m - m_use);
    float psum = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      s[j] = s[j] == -INFINITY ? 0.f : expf(s[j] - m_use);
      psum += s[j];
    }
    l = l * alpha + psum;
    m = m_new;
#pragma unroll
    for (int j = 0; j < 4; ++j) ft_put(ks + row * 128 + (((half * 4 + j) ^ (row & 7)) << 4), FT_PPART, s + 8 * j);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();  // the probabilities' and the values' parts are there
    tc_fence_after();
    if (warp == 0 && elect_one()) {
      constexpr uint32_t idesc = umma_idesc(128, HD, true);
#pragma unroll
      for (int i = 0; i < 2; ++i)  // 32 keys
        ft_accumulate(tmem + FT_O + i * HD, umma_desc(smem_u32(ks) + i * 64), umma_desc_offsets(smem_u32(vs) + i * 32 * 128, BLK * 128, 1024),
                      FT_PPART >> 4, FT_KPART >> 4, 2, 16 * 128 >> 4, idesc);
      tc_commit(&done_o);
    }
    __syncwarp();
#pragma unroll
    for (int c = 0; c < HD / 2; ++c) acc[c] *= alpha;
    ok = __all_sync(0xffffffffu, ok && wait_or_abort(&done_o, it & 1, failed));
    if (ok) {
      tc_fence_after();
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int c = 0; c < HD / 2; c += 32) {
          float t[32];
          tmem_load_32(tmem + lane_base + FT_O + i * HD + half * (HD / 2) + c, t);
#pragma unroll
          for (int j = 0; j < 32; ++j) acc[c + j] += t[j];
        }
    }
  }
  sums[half][row] = l;
  if (sees_odd || !(l == l)) odd[row] = 1;
  __syncthreads();
  if (mine && !odd[row] && FMS_IN(row_begin + r0 + pos, n_rows)) {
    float sum = sums[0][row] + sums[1][row];
    if (a.sink != nullptr) sum += expf(a.sink[head] - (m == -INFINITY ? 0.f : m));
    const float inv = sum > 0.f ? 1.f / sum : 0.f;
    float4* o = reinterpret_cast<float4*>((float*)a.out + (size_t)(row_begin + r0 + pos) * a.nheads * HD + (size_t)head * HD + half * (HD / 2));
#pragma unroll
    for (int c = 0; c < HD / 2; c += 4)
      o[c / 4] = make_float4(acc[c] * inv * FT_UNSCALE, acc[c + 1] * inv * FT_UNSCALE, acc[c + 2] * inv * FT_UNSCALE, acc[c + 3] * inv * FT_UNSCALE);
  }
  {  // the other rows: a warp a row, a lane a key and HD / 32 of the results
    constexpr int PER = HD / 32;
    for (int r = warp; r < 128; r += FT_THREADS / 32) {
      if ((r & 63) >= rows_here || !odd[r] || !FMS_IN(row_begin + r0 + (r & 63), n_rows)) continue;
      const int at = p_first + (r & 63), h = head0 + (r >> 6);
      const float* qr = q + (size_t)(r & 63) * a.q_stride + (r >> 6) * HD;
      const int first = first_visible(a, at);
      float o[PER] = {}, mr = -INFINITY, lr = 0.f;
      for (int base = first / 32 * 32; base <= at; base += 32) {
        const int b = block_of(a, slot, base / BLK);
        if (b < 0) continue;
        const size_t place = (((size_t)b * a.kvheads + kvh) * BLK + base % BLK) * HD;
        const bool visible = base + lane >= first && base + lane <= at;
        float score = -INFINITY;
        if (visible) {
          const float* key = (const float*)a.keys + place + (size_t)lane * HD;
          float dot = 0.f;
#pragma unroll 4
          for (int d = 0; d < HD; d += 4) {
            const float4 x = *reinterpret_cast<const float4*>(qr + d), y = *reinterpret_cast<const float4*>(key + d);
            dot = fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, fmaf(x.x, y.x, dot))));
          }
          score = dot * a.scale;
        }
        const float m_new = fmaxf(mr, warp_max(score)), m_use = m_new == -INFINITY ? 0.f : m_new;
        const float before = mr == -INFINITY ? 0.f : expf(mr - m_use), p = score == -INFINITY ? 0.f : expf(score - m_use);
        lr = lr * before + warp_sum(p);
        mr = m_new;
#pragma unroll
        for (int d = 0; d < PER; ++d) o[d] *= before;
        const float* values = (const float*)a.values + place + lane * PER;
        for (int j = max(first - base, 0); j <= min(at - base, 31); ++j) {
          const float pj = __shfl_sync(0xffffffffu, p, j);
#pragma unroll
          for (int d = 0; d < PER; ++d) o[d] = fmaf(pj, values[j * HD + d], o[d]);
        }
      }
      if (a.sink != nullptr) lr += expf(a.sink[h] - (mr == -INFINITY ? 0.f : mr));
      const float inv = lr > 0.f ? 1.f / lr : 0.f;  // where lr is no number, o is none
#pragma unroll
      for (int d = 0; d < PER; ++d) ((float*)a.out)[(size_t)(row_begin + r0 + (r & 63)) * a.nheads * HD + (size_t)h * HD + lane * PER + d] = o[d] * inv;
    }
  }
  tc_fence_before();
  __syncthreads();
  if (tid == 0 && *failed && error_flag) atomicExch(error_flag, 4);
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
}
