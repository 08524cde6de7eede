// Softmax attention of prompt rows over the paged cache with shaped scores (`attention_scored.cu` says what a score can be
// given), on the tensor cores: bfloat16 queries, keys and values, 32-bit scores, softmax weights and sums.
//
//   s = q . k        mma.sync m16n8k16, 32-bit accumulation (products of bfloat16 numbers are exact)
//   p = exp(s - m)   32-bit, in the accumulators' own registers
//   o += p v         p is cut into three bfloat16 pieces, p = h + m + l exactly: a weight keeps its 24 bits, the pieces are
//                    multiplied one after another.  The tensor core's truncating accumulation is kept to 64 keys, whose sum
//                    then joins the 32-bit running sum by a rounded addition: over all pages it left the sums of 8 k even weights
//                    8e-5 short.
//
// A block works 64 (token, head) pairs that share a key head - 64 / hp consecutive tokens of one sequence times hp heads of the
// group, a warp 16 of them - against the cache's pages of 64 keys, by two halves of four warps that take the pages the block sees in
// turn and put their sums together at the end (`layout_of`: or by one half alone).  What bounds it is the chain through one
// warp, more than 1000 instructions and 5000 cycles a page with the products' latency; more warps at once and half as many pages a warp is what helps, and
// four warps a barrier, so that halves and blocks are out of step and one's softmax runs under another's products.  A page comes into
// shared memory by cp.async while the one before is worked on (values that are the keys' first entries come once).  Queries stay in shared
// memory, all of the running output in registers.  Rows are padded to an odd number of 16-byte pieces, so ldmatrix meets no bank twice.
// Pages that no pair of the block sees are skipped.  Tiles are launched longest first.
//
// Why: on the CUDA cores (`attention_scored.cu`) 2 x 1024 rows of 16 heads over a latent of 256 took 1102 us (15.6 TFLOP/s) and take 127 here,
// 16 heads of 64 on 4 key heads with capped scores, gates and a window of 512 took 358 us and take 64.
#include <algorithm>

#include "common.cuh"

using namespace kvad;

namespace {

constexpr int PAGE = 64, WARPS = 4, HALF = 32 * WARPS, THREADS = 2 * HALF, ROWS = 16 * WARPS;
constexpr size_t SMEM_MOST = 220 * 1024, SMEM_HALF = 112 * 1024;      // (a block's; so that two fit an SM)
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;

struct PromptArgs {
  const __nv_bfloat16* q; int64_t ld_q;
  void* out; int64_t ld_out;
  const __nv_bfloat16* gate; int64_t ld_gate; int gate_heads;    // gate_heads: one number per row and head
  const float* sinks;
  const int* seq_starts; const int* kv_lens; const int* page_table; int table_width;
  const __nv_bfloat16* k_pages; const __nv_bfloat16* v_pages;
  int64_t k_page_stride, v_page_stride;                           // in entries; a head's page is PAGE x dk (PAGE x dv)
  int n_heads, n_kv_heads, dk, dv, hp, alias, key_maps, halves;
  int columns;                                                    // tiles of one place in their sequence: sequences x heads / hp (the grid is these, the last place first)
  float scale, softcap, slope_span;
  float cap_in, cap_out;                                          // a capped score: cap_out * tanh(cap_in * (q . k)), in units of log2
  int window, keep_first, chunk;
  int k_steps, k_stride, v_stride;                                // 16-entry steps of a key; row strides in shared memory, in entries
};

__device__ __forceinline__ uint32_t smem_at(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm4(uint32_t at, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t at, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// 16 bytes to shared memory, zeros where `live` is false (places of the cache that no row sees yet may hold anything)
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool live) {
  const int bytes = live ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
// 2^x by the special-function unit (2 units in the last place; a weight below 2^-126 of its row's largest is zero).  With it a 32-bit output is off
// by 1.4e-7 (16 heads of 64) to 1.8e-7 (a latent of 128) over 1024 rows, the CUDA-core kernel's by 2.6e-7 to 3.2e-7.
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// The upper halves of two floats as a pair of bfloat16 (truncated), and what is left of each.
__device__ __forceinline__ uint32_t cut(float& a, float& b) {
  const uint32_t x = __float_as_uint(a), y = __float_as_uint(b);
  a -= __uint_as_float(x & 0xffff0000u);
  b -= __uint_as_float(y & 0xffff0000u);
  return __byte_perm(x, y, 0x7632);
}
__device__ __forceinline__ uint32_t pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// NV: 16-entry groups of a value.
template <int NV, bool F32OUT>
__global__ void __launch_bounds__(NV <= 4 ? THREADS : HALF, 2) scored_prompt_kernel(const PromptArgs a) {
  extern __shared__ uint8_t smem_raw[];
  __nv_bfloat16* smem = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  const int hp = a.hp, tok = ROWS / hp, group = a.n_heads / a.n_kv_heads, chunks = group / hp;
  const int per_seq = a.n_kv_heads * chunks, from_end = blockIdx.x / a.columns, column = blockIdx.x - from_end * a.columns;
  const int s = column / per_seq, part = column - s * per_seq, kvh = part / chunks, h0 = kvh * group + (part - kvh * chunks) * hp;
  const int half = threadIdx.x / HALF, tid = threadIdx.x - half * HALF, lane = tid & 31, warp = tid >> 5;      // (tid, warp: within the half)
  const int kst = a.k_stride, vst = a.v_stride;
  __nv_bfloat16* Qs = smem;                                     // [ROWS][kst]
  const int stage_size = PAGE * kst + (a.alias ? 0 : PAGE * vst);
  __nv_bfloat16* stages = Qs + ROWS * kst + half * 2 * stage_size;      // each half: two of: keys [PAGE][kst], values [PAGE][vst] (or none: the keys)
  pdl_launch_dependents();
  // The last step's entries past the key that no copy writes must not be NaN: zeros.  (Values past the last reach only outputs that are not written.)
  if (a.dk % 16 != 0) {
    for (int i = tid; i < ROWS + 2 * PAGE; i += HALF) {
      __nv_bfloat16* at = i < ROWS ? Qs + i * kst : stages + ((i - ROWS) / PAGE) * stage_size + ((i - ROWS) % PAGE) * kst;
      *reinterpret_cast<uint4*>(at + a.dk) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  pdl_wait();
  const int start = a.seq_starts[s], n_new = a.seq_starts[s + 1] - start, tok0 = ((int)gridDim.x / a.columns - 1 - from_end) * tok;
  if (tok0 >= n_new) return;
  const int n_tok = min(tok, n_new - tok0), pos0 = a.kv_lens[s] - n_new + tok0, last_pos = pos0 + n_tok - 1;
  const int* pages = a.page_table + (int64_t)s * a.table_width;
  const int q_pieces = a.dk / 8, v_pieces = a.dv / 8;
  for (int i = threadIdx.x; i < ROWS * q_pieces; i += blockDim.x) {
    const int r = i / q_pieces, c = i - r * q_pieces, ti = r / hp, hi = r - ti * hp;
    const bool live = ti < n_tok;
    copy16(smem_at(Qs + r * kst + c * 8), a.q + (int64_t)(start + tok0 + (live ? ti : 0)) * a.ld_q + (int64_t)(h0 + hi) * a.dk + c * 8, live);
  }
  const int first_key = a.chunk > 0 ? pos0 - pos0 % a.chunk : ((a.window > 0 && pos0 - a.window + 1 > 0) ? pos0 - a.window + 1 : 0);   // of the block's first token
  auto next_page = [&](int t) {                                 // the next page that a pair of the block sees (the same for every thread)
    while (t * PAGE <= last_pos && t * PAGE + PAGE <= first_key && t * PAGE >= a.keep_first) ++t;
    return t;
  };
  // A thread steps from one of its pieces to the next by additions (a division a piece cost as much as the scores); where registers are to spare the
  // first step is worked out once, not once a page.
  struct Steps { int r, c, rows, rest; };
  auto steps_of = [&](int pieces) {
    const int rows = HALF / pieces, r = tid / pieces;
    return Steps{r, tid - r * pieces, rows, HALF - rows * pieces};
  };
  constexpr bool ONCE = NV == 8;
  const Steps k_once = ONCE ? steps_of(q_pieces) : Steps{}, v_once = ONCE ? steps_of(v_pieces) : Steps{};
  auto bring_rows = [&](__nv_bfloat16* dst, int stride, const __nv_bfloat16* src, int pieces, const Steps& z, int n_live) {
    int r = z.r, c = z.c;
#pragma unroll 4
    for (int i = tid; i < PAGE * pieces; i += HALF) {
      copy16(smem_at(dst + r * stride + c * 8), src + (int64_t)i * 8, r < n_live);
      r += z.rows;
      c += z.rest;
      if (c >= pieces) { c -= pieces; ++r; }
    }
  };
  auto bring = [&](int t, int stage) {
    const int page = pages[t], n_live = last_pos - t * PAGE + 1;
    __nv_bfloat16* ks = stages + stage * stage_size;
    const __nv_bfloat16* src = a.k_pages + (int64_t)page * a.k_page_stride + (int64_t)kvh * PAGE * a.dk;
    bring_rows(ks, kst, src, q_pieces, ONCE ? k_once : steps_of(q_pieces), n_live);
    if (!a.alias) {
      __nv_bfloat16* vs = ks + PAGE * kst;
      const __nv_bfloat16* vsrc = a.v_pages + (int64_t)page * a.v_page_stride + (int64_t)(kvh / a.key_maps) * PAGE * a.dv;
      bring_rows(vs, vst, vsrc, v_pieces, ONCE ? v_once : steps_of(v_pieces), n_live);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // this thread's two rows of the warp's 16: lane / 4 and that plus 8
  int pos[2], first[2], head[2];
  bool live[2];
  float slope[2], run_max[2] = {-INFINITY, -INFINITY}, run_sum[2] = {0.f, 0.f};      // (maxima in units of log2)
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    const int row = warp * 16 + (lane >> 2) + u * 8, ti = row / hp;
    head[u] = h0 + row - ti * hp;
    live[u] = ti < n_tok;
    pos[u] = pos0 + ti;
    first[u] = a.window > 0 ? pos[u] - a.window + 1 : (a.chunk > 0 ? pos[u] - pos[u] % a.chunk : 0);
    slope[u] = a.slope_span > 0.f ? exp2f(-a.slope_span * (float)(head[u] + 1) / (float)a.n_heads) * LOG2E : 0.f;
  }
  // keys from `clear_from` up to `clear_to` (and the kept first ones) are seen by every live row of the warp
  const int warp_ti0 = warp * 16 / hp, warp_ti1 = min((warp * 16 + 15) / hp, n_tok - 1);
  const bool warp_live = warp_ti0 < n_tok;
  const int clear_to = pos0 + warp_ti0;
  const int far = pos0 + warp_ti1;
  const int clear_from = a.window > 0 ? far - a.window + 1 : (a.chunk > 0 ? far - far % a.chunk : 0);
  float o[2 * NV][4];
#pragma unroll
  for (int j = 0; j < 2 * NV; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[j][e] = 0.f;
  const float scale2 = a.scale * LOG2E;
  const bool plain = !(a.softcap > 0.f) && !(a.slope_span > 0.f) && a.scale > 0.f;
  const float unit = plain ? scale2 : 1.f;
  const uint32_t q_at = smem_at(Qs + (warp * 16 + (lane & 15)) * kst + (lane >> 4) * 8);

  // the pages that the block sees, dealt out to the halves in turn
  int t = next_page(0), stage = 0;
  if (half == 1) t = next_page(t + 1);
  if (t * PAGE <= last_pos) bring(t, 0);
  asm volatile("cp.async.wait_all;" ::: "memory");              // (a half without pages has queries on their way)
  __syncthreads();                                              // the queries, brought by both halves, and each half's first page
  bool first_page = true;
  while (t * PAGE <= last_pos) {
    if (!first_page) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (half == 0) asm volatile("bar.sync 1, %0;" ::"n"(HALF) : "memory");      // this page is there, and the one before has been used up
      else asm volatile("bar.sync 2, %0;" ::"n"(HALF) : "memory");
    }
    first_page = false;
    int t_next = next_page(t + 1);
    if (a.halves == 2) t_next = next_page(t_next + 1);
    if (t_next * PAGE <= last_pos) bring(t_next, stage ^ 1);
    const int key0 = t * PAGE;
    const __nv_bfloat16* ks = stages + stage * stage_size;
    const __nv_bfloat16* vs = a.alias ? ks : ks + PAGE * kst;
    t = t_next;
    stage ^= 1;
    if (!warp_live) continue;
    float sc[8][4];
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) sc[j][e] = 0.f;
    const uint32_t k_at = smem_at(ks + ((lane & 7) + (lane >> 4) * 8) * kst + ((lane >> 3) & 1) * 8);
#pragma unroll 2
    for (int kk = 0; kk < a.k_steps; ++kk) {
      uint32_t qa[4];
      ldsm4(q_at + kk * 32, qa);
#pragma unroll
      for (int ng = 0; ng < 4; ++ng) {
        uint32_t kb[4];
        ldsm4(k_at + kk * 32 + ng * 16 * kst * 2, kb);
        mma(sc[2 * ng], qa, kb[0], kb[1]);
        mma(sc[2 * ng + 1], qa, kb[2], kb[3]);
      }
    }
    // Scores in units of log2, or, where nothing but a positive factor is on them, as they are with the factor `unit` still owed.
    // (Whole passes over the 32 scores under tests that are the same for every thread: this part is bound by instructions.)
    if (!plain) {
      if (a.softcap > 0.f) {                                    // cap tanh(s / cap): by `tanhf`, whose error follows its result (1 - 2 / (exp(2 y) + 1): off by 2^-22 of the CAP)
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            sc[j][e] = a.cap_out * tanhf(sc[j][e] * a.cap_in);
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) sc[j][e] *= scale2;
      }
      if (a.slope_span > 0.f) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) sc[j][e] -= slope[e >> 1] * (float)(pos[e >> 1] - (key0 + j * 8 + (lane & 3) * 2 + (e & 1)));
      }
    }
    if (!(key0 + PAGE - 1 <= clear_to && (key0 >= clear_from || key0 + PAGE <= a.keep_first))) {      // some pair does not see all of the page
#pragma unroll
      for (int j = 0; j < 8; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int u = e >> 1, key = key0 + j * 8 + (lane & 3) * 2 + (e & 1);
          if (!(key <= pos[u] && (key >= first[u] || key < a.keep_first))) sc[j][e] = -INFINITY;
        }
    }
    float top[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) top[e >> 1] = fmaxf(top[e >> 1], sc[j][e]);
    float base[2], keep[2], sum[2] = {0.f, 0.f};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      top[u] = fmaxf(top[u], __shfl_xor_sync(0xffffffffu, top[u], 1));
      top[u] = fmaxf(top[u], __shfl_xor_sync(0xffffffffu, top[u], 2));
      const float new_max = fmaxf(run_max[u], top[u] * unit);
      base[u] = new_max == -INFINITY ? 0.f : new_max;
      keep[u] = run_max[u] == -INFINITY ? 0.f : exp2_fast(run_max[u] - base[u]);
      run_max[u] = new_max;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int u = e >> 1;
        sc[j][e] = exp2_fast(fmaf(sc[j][e], unit, -base[u]));
        sum[u] += sc[j][e];
      }
#pragma unroll
    for (int u = 0; u < 2; ++u) run_sum[u] = run_sum[u] * keep[u] + sum[u];      // (of this thread's keys; the row's four threads meet at the end)
    const uint32_t v_at = smem_at(vs + ((lane & 7) + ((lane >> 3) & 1) * 8) * vst + (lane >> 4) * 8);
    uint32_t ph[4][4], pm[4][4], pl[4][4];
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        float x = sc[2 * kk + (f >> 1)][(f & 1) * 2], y = sc[2 * kk + (f >> 1)][(f & 1) * 2 + 1];
        ph[kk][f] = cut(x, y);
        pm[kk][f] = cut(x, y);
        pl[kk][f] = pack(x, y);
      }
#pragma unroll
    for (int ng = 0; ng < NV; ++ng) {
      float low[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, page[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        uint32_t vb[4];
        ldsm4_t(v_at + kk * 16 * vst * 2 + ng * 32, vb);
#pragma unroll
        for (int w = 0; w < 2; ++w) mma(low[w], pl[kk], vb[2 * w], vb[2 * w + 1]);
#pragma unroll
        for (int w = 0; w < 2; ++w) mma(page[w], ph[kk], vb[2 * w], vb[2 * w + 1]);
#pragma unroll
        for (int w = 0; w < 2; ++w) mma(low[w], pm[kk], vb[2 * w], vb[2 * w + 1]);
      }
#pragma unroll
      for (int w = 0; w < 2; ++w)
#pragma unroll
        for (int e = 0; e < 4; ++e) o[2 * ng + w][e] = fmaf(o[2 * ng + w][e], keep[e >> 1], page[w][e] + low[w][e]);
    }
  }

  // The second half's sums join the first's: its threads hold the same rows and entries.
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    run_sum[u] += __shfl_xor_sync(0xffffffffu, run_sum[u], 1);
    run_sum[u] += __shfl_xor_sync(0xffffffffu, run_sum[u], 2);
  }
  if (a.halves == 2) {
    float* meet = reinterpret_cast<float*>(smem_raw) + tid;
    __syncthreads();                                              // nobody reads queries or pages any more
    if (half == 1) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        meet[u * HALF] = run_max[u];
        meet[(2 + u) * HALF] = run_sum[u];
      }
#pragma unroll
      for (int j = 0; j < 2 * NV; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) meet[(4 + j * 4 + e) * HALF] = o[j][e];
    }
    __syncthreads();
    if (half == 1) return;
    float mine[2], theirs[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float their_max = meet[u * HALF], m = fmaxf(run_max[u], their_max), base = m == -INFINITY ? 0.f : m;
      mine[u] = exp2_fast(run_max[u] - base);
      theirs[u] = exp2_fast(their_max - base);
      run_sum[u] = run_sum[u] * mine[u] + meet[(2 + u) * HALF] * theirs[u];
      run_max[u] = m;
    }
#pragma unroll
    for (int j = 0; j < 2 * NV; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[j][e] = o[j][e] * mine[e >> 1] + meet[(4 + j * 4 + e) * HALF] * theirs[e >> 1];
  }

#pragma unroll
  for (int u = 0; u < 2; ++u) {
    if (!live[u]) continue;
    const int row = warp * 16 + (lane >> 2) + u * 8, h = head[u];
    const int64_t grow = start + tok0 + row / hp;
    float inv;
    if (a.sinks == nullptr) {
      inv = 1.0f / run_sum[u];
    } else {                                                    // a sink is one more term of the denominator
      const float mine = run_max[u] * LN2, sink = a.sinks[h], m = fmaxf(mine, sink), f = expf(mine - m);
      inv = f / fmaf(run_sum[u], f, expf(sink - m));
    }
    float head_factor = 1.f;
    if (a.gate != nullptr && a.gate_heads) head_factor = 1.0f / (1.0f + expf(-__bfloat162float(a.gate[grow * a.ld_gate + h])));
#pragma unroll
    for (int j = 0; j < 2 * NV; ++j) {
      const int d = j * 8 + (lane & 3) * 2;                     // (dv is a multiple of 8)
      if (d >= a.dv) continue;
      float x = o[j][2 * u] * inv, y = o[j][2 * u + 1] * inv;
      if (F32OUT) {
        *reinterpret_cast<float2*>(reinterpret_cast<float*>(a.out) + grow * a.ld_out + (int64_t)h * a.dv + d) = make_float2(x, y);
      } else {
        if (a.gate != nullptr && !a.gate_heads) {
          const __nv_bfloat162 z = *reinterpret_cast<const __nv_bfloat162*>(a.gate + grow * a.ld_gate + (int64_t)h * a.dv + d);
          x *= 1.0f / (1.0f + expf(-__bfloat162float(z.x)));
          y *= 1.0f / (1.0f + expf(-__bfloat162float(z.y)));
        } else {
          x *= head_factor;
          y *= head_factor;
        }
        *reinterpret_cast<uint32_t*>(reinterpret_cast<__nv_bfloat16*>(a.out) + grow * a.ld_out + (int64_t)h * a.dv + d) = pack(x, y);
      }
    }
  }
}

template <int NV, bool F32OUT>
int launch(const PromptArgs& a, int max_new, size_t smem, cudaStream_t stream) {
  static size_t configured = 0;
  if (smem > configured) {
    cudaError_t e = cudaFuncSetAttribute(scored_prompt_kernel<NV, F32OUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "attention (scored, prompts): cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    configured = smem;
  }
  const int tok = ROWS / a.hp;
  const int64_t tiles = (int64_t)a.columns * ((max_new + tok - 1) / tok);
  KVAD_REQUIRE(tiles < (1ll << 31), "attention (scored, prompts): %lld tiles are more than one launch takes", (long long)tiles);
  kvad_launch(scored_prompt_kernel<NV, F32OUT>, dim3((unsigned)tiles), dim3(a.halves * HALF), smem, stream, a);
  KVAD_CHECK_LAUNCH("attention_scored_prompt");
  return KVAD_OK;
}

// 16-entry groups of a value that the kernel is built for.
int groups_of(int dv) { return dv <= 32 ? 2 : (dv <= 64 ? 4 : (dv <= 128 ? 8 : (dv <= 192 ? 12 : 16))); }

struct Layout { int k_stride, v_stride, halves; size_t smem; };
// Row strides of an odd number of 16-byte pieces over whole 16-entry steps; all of shared memory with the slack that the last row's unused
// value columns may read (values are read in the kernel's groups of 16 entries), and room for the second half's sums at the end.
Layout layout_of(int dk, int dv, bool alias) {
  Layout z;
  z.k_stride = (dk + 15) / 16 * 16 + 8;
  z.v_stride = alias ? z.k_stride : (dv + 15) / 16 * 16 + 8;
  // Two halves where two such blocks fit an SM (values of up to 64 entries: 128 registers a thread), else one: two halves that are the SM's
  // only block leave it idle where they begin and end.  (Measured when weights went through in two pieces, 2 x 1024 rows, two halves against one: 12 heads of 64: 36 us and 50; 32 heads of
  // 128 on 8: 148 and 112; 16 heads over a latent of 256: 152 and 108.)
  auto need = [&](int halves) {
    return ((size_t)ROWS * z.k_stride + 2 * halves * ((size_t)PAGE * z.k_stride + (alias ? 0 : (size_t)PAGE * z.v_stride)) + 256 + 16) * 2;
  };
  z.halves = groups_of(dv) <= 4 && need(2) <= SMEM_HALF ? 2 : 1;
  z.smem = need(z.halves);
  if (z.halves == 2) z.smem = std::max(z.smem, (size_t)(8 * groups_of(dv) + 4) * HALF * sizeof(float));
  return z;
}

}  // namespace

// 1 if prompts of these sizes run here: whole 16-byte pieces, values up to 256 entries (128 where the output is 32-bit), everything in shared memory.
KVAD_EXPORT int kvad_attention_scored_prompt_takes(int dk, int dv, int alias, int out_f32) {
  return dk > 0 && dv > 0 && dk % 8 == 0 && dv % 8 == 0 && dv <= (out_f32 ? 128 : 256) && layout_of(dk, dv, alias != 0).smem <= SMEM_MOST ? 1 : 0;
}

KVAD_EXPORT int kvad_attention_scored_prompt(const void* q, int64_t ld_q, void* out, int64_t ld_out, const void* gate, int64_t ld_gate, int gate_heads,
                                             const float* sinks, const int* seq_starts, const int* kv_lens, const int* page_table, int table_width,
                                             const void* k_pages, const void* v_pages, int n_seqs, int n_heads, int n_kv_heads, int dk, int dv,
                                             int page_size, int max_new, float scale, float softcap, float slope_span, int window, int keep_first,
                                             int chunk, int key_maps, int out_f32, cudaStream_t stream) {
  KVAD_REQUIRE(n_seqs >= 0 && n_heads > 0 && n_kv_heads > 0 && dk > 0 && dv > 0 && table_width > 0 && max_new >= 0 && keep_first >= 0,
               "attention (scored, prompts): bad sizes seqs=%d heads=%d kv_heads=%d dk=%d dv=%d", n_seqs, n_heads, n_kv_heads, dk, dv);
  KVAD_REQUIRE(n_heads % n_kv_heads == 0, "attention (scored, prompts): %d heads do not divide into %d key/value heads", n_heads, n_kv_heads);
  KVAD_REQUIRE(chunk <= 0 || window <= 0, "attention (scored, prompts): a chunk goes without a window");
  const bool alias = v_pages == k_pages;
  KVAD_REQUIRE(key_maps >= 1 && n_kv_heads % key_maps == 0 && (key_maps == 1 || !alias), "attention (scored, prompts): %d key heads do not share values %d by %d", n_kv_heads, key_maps, key_maps);
  KVAD_REQUIRE(!out_f32 || gate == nullptr, "attention (scored, prompts): a 32-bit output takes no gate");
  KVAD_REQUIRE(!alias || dv <= dk, "attention (scored, prompts): values read from the keys cannot be longer than a key");
  if (page_size != PAGE || !kvad_attention_scored_prompt_takes(dk, dv, alias, out_f32))
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "attention (scored, prompts): pages of %d, keys of %d, values of %d are not taken", page_size, dk, dv);
  const uintptr_t all = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages);
  if ((all & 15) || ld_q % 8 != 0 || (reinterpret_cast<uintptr_t>(out) & 7) || ld_out % 2 != 0 ||
      (gate != nullptr && ((reinterpret_cast<uintptr_t>(gate) & 3) || ld_gate % 2 != 0)))
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "attention (scored, prompts): rows must lie on 16-byte boundaries");
  if (n_seqs == 0 || max_new == 0) return KVAD_OK;
  PromptArgs a;
  a.q = (const __nv_bfloat16*)q; a.ld_q = ld_q; a.out = out; a.ld_out = ld_out; a.gate = (const __nv_bfloat16*)gate; a.ld_gate = ld_gate;
  a.gate_heads = gate_heads; a.sinks = sinks; a.seq_starts = seq_starts; a.kv_lens = kv_lens; a.page_table = page_table; a.table_width = table_width;
  a.k_pages = (const __nv_bfloat16*)k_pages; a.v_pages = (const __nv_bfloat16*)v_pages;
  a.k_page_stride = (int64_t)n_kv_heads * PAGE * dk; a.v_page_stride = (int64_t)(n_kv_heads / key_maps) * PAGE * dv;
  a.n_heads = n_heads; a.n_kv_heads = n_kv_heads; a.dk = dk; a.dv = dv; a.alias = alias ? 1 : 0; a.key_maps = key_maps;
  a.scale = scale; a.softcap = softcap; a.slope_span = slope_span; a.window = window > 0 ? window : 0; a.keep_first = window > 0 ? keep_first : 0;
  a.chunk = chunk > 0 ? chunk : 0;
  // (scale / cap stays an ordinary number: a cap above 2^100 moves no score below 2^87, one of nothing makes every score but 0 the cap)
  const float cap = std::min(softcap, 1.2676506e30f), ratio = scale / cap;
  a.cap_in = softcap > 0.f ? std::max(-3.402823466e38f, std::min(3.402823466e38f, ratio)) : 0.f; a.cap_out = cap * LOG2E;
  // heads a tile: as many of the group as divide it, up to a warp's 16 rows (a tile then spans few tokens: little of its last page is masked)
  a.hp = 1;
  while (a.hp < 16 && (n_heads / n_kv_heads) % (a.hp * 2) == 0) a.hp *= 2;
  KVAD_REQUIRE((int64_t)n_seqs * (n_heads / a.hp) < (1ll << 31), "attention (scored, prompts): %d sequences x %d heads are more than one launch takes", n_seqs, n_heads);
  a.columns = n_seqs * (n_heads / a.hp);
  const Layout z = layout_of(dk, dv, alias);
  a.halves = z.halves; a.k_steps = (dk + 15) / 16; a.k_stride = z.k_stride; a.v_stride = z.v_stride;
#define KVAD_SP(N)                                                                          \
  do {                                                                                      \
    if (out_f32) return launch<(N > 8 ? 8 : N), true>(a, max_new, z.smem, stream);  \
    return launch<N, false>(a, max_new, z.smem, stream);                            \
  } while (0)
  switch (groups_of(dv)) {
    case 2: KVAD_SP(2);
    case 4: KVAD_SP(4);
    case 8: KVAD_SP(8);
    case 12: KVAD_SP(12);
    default: KVAD_SP(16);
  }
#undef KVAD_SP
}

KVAD_DEFINE_LAST_ERROR()
