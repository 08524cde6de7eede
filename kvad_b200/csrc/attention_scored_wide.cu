// Softmax attention of prompt rows over the paged cache with shaped scores (`attention_scored.cu` says what a score can be given), 32-bit queries, keys
// and values on the 5th-generation tensor cores: the float32 engine's prompts.
//
// As `attention_scored_prompt.cu` (128 (token, head) pairs a block, pages of 64 keys, a page's weights against its own maximum, sums of one page in the
// tensor core, 32-bit registers beyond), with every operand cut into bfloat16 pieces x = h + m + l (exact above about 2^-110) and the six products of
// pieces that reach 2^-24 (h h, h m, m h, h l, m m, l h, the smallest first): S takes 24 products of 128 x 64 x 16 for keys of 64, P V as many.
// The tensor core truncates where it accumulates, so S leaves it after 64 entries of a key, P V after 64 keys with its h h in an accumulator of their own; all
// joins are rounded.  Queries are cut once; a page's keys and values are cut by four warps (of eight that take pages in turn) into the ring that the tensor core reads.
//
// What bounds it: cutting a page (1000 instructions a thread of four warps) about as much as its 48 products (1150 + 770 cycles for 64 + 64 entries); one page at a time
// where keys and values are above 64 entries.  us against the CUDA cores: 2 x 1024 rows of 16 heads of 64 on 4 key heads: 56 against 381; capped, window 512: 63 against 313
// (scores beyond 0.45 caps among them: 87); heads of 128: 132 against 472; a latent of 96 with 32 more key entries: 78 against 640; two new rows of four sequences behind 300
// positions: 17 against 54; one prompt of 17: 9.6 against 15.6.  (With one group of warps cutting a batch ahead by way of registers: 90 where it was 54.  One accumulator for all
// of S and one for all of P V: 53, 64, 130, 71.)
// Relative error against 64 bits, here and there (heads of 64; of 128): 2 x 1024 rows 2.2e-7, 3.3e-7; 2.0e-7, 3.9e-7; operands of one sign 1.3e-7, 3.4e-7 in both; 2000 cached positions
// 3.1e-7, 8.5e-7; one prompt of 17 1.2e-7, 1.2e-7; 1.3e-7, 1.8e-7.  It is larger only where the weights of few keys are nearly even (17 rows, scores below 0.1: 8.8e-8 for 6.0e-8).
//
// A number that is not finite has no pieces: rows whose outputs it reaches are worked out again by fmaf (`row_again`).  Every wait is bounded.
#include <algorithm>
#include <type_traits>

#include "scored_tiles.cuh"

using namespace kvad;

namespace {

constexpr int THREADS = 640, MAX_STAGES = 3, CW = 64, SLOTS = 3;
constexpr int STATS = 8;             // pages whose statistics are kept: weights run up to two pages ahead of P V, P V up to three of the output
// tensor-memory columns: the places of P V, S of two pages, the weights' pieces of two pages (32 columns each: two bfloat16 a column)
constexpr uint32_t TM_T = 0, TM_S = SLOTS * CW, TM_P = TM_S + 128, P_STEP = 96, TM_COLS = 512;
constexpr size_t SMEM_MOST = 226 * 1024, SMEM_REST = STATS * ROWS * 8 + 320 + 1024;      // (statistics, barriers, alignment)

struct WideArgs {
  const float* q; int64_t ld_q;
  float* out; int64_t ld_out;
  const float* gate; int64_t ld_gate; int gate_heads;            // gate_heads: one number per row and head
  const float* sinks;
  const int* seq_starts; const int* kv_lens; const int* page_table; int table_width;
  const float* k_pages; const float* v_pages;
  int n_heads, n_kv_heads, dk, dv, hp, alias, key_maps, stages;
  int columns;                                                    // tiles of one place in their sequence: sequences x heads / hp (the grid is these, the last place first)
  float scale, softcap, slope_span;
  float cap_in, cap_out;                                          // a capped score: cap_out * tanh(cap_in * (q . k)), in units of log2
  int window, keep_first, chunk;
  int shorter;                                                    // sequences of up to so many positions are left alone (attention_simt.cu takes them)
  int skip_copy;                                                  // (tests: a block's first page is not said to be there, so that the wait for it runs out)
};

int g_skip_copy = 0;

// Eight neighbours into three pieces of 16 bytes, `step` bytes apart.  (Of a number that is not finite the last pieces are no number.)
__device__ __forceinline__ void put8(uint8_t* dst, uint32_t step, const float4& a, const float4& b) {
  float x[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
  for (int piece = 0; piece < 2; ++piece) {
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = cut(x[2 * i], x[2 * i + 1]);
    *reinterpret_cast<uint4*>(dst + piece * step) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  uint32_t w[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) w[i] = __byte_perm(__float_as_uint(x[2 * i]), __float_as_uint(x[2 * i + 1]), 0x7632);
  *reinterpret_cast<uint4*>(dst + 2 * step) = make_uint4(w[0], w[1], w[2], w[3]);
}

// CPW: 64-column pieces of the output.
template <int CPW>
__global__ void __launch_bounds__(THREADS, 1) scored_wide_kernel(const __grid_constant__ WideArgs a) {
  constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};      // which pieces meet, the smallest products first
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int k_blocks = (a.dk + 63) / 64, v_blocks = (a.dv + 63) / 64, stages = a.stages;
  const uint32_t q_piece = k_blocks * Q_BLOCK, k_piece = k_blocks * PAGE_BLOCK, v_piece = a.alias ? k_piece : v_blocks * PAGE_BLOCK;
  const uint32_t v_off = a.alias ? 0u : 3 * k_piece, stage_bytes = 3 * k_piece + (a.alias ? 0u : 3 * v_piece);
  uint8_t* q_tile = smem;                                         // [piece][block of 64 entries][row]
  uint8_t* ring = smem + 3 * q_piece;                             // stage: keys [piece][block][key], then values (or none: the keys)
  float2* stats = reinterpret_cast<float2*>(ring + stages * stage_bytes);      // [STATS][ROWS] a page's largest score and sum of weights, per row
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(stats + STATS * ROWS);       // [stages] a page's pieces are there
  uint64_t* kv_empty = kv_full + MAX_STAGES;                      // [stages] it has been used up
  uint64_t* s_full = kv_empty + MAX_STAGES;                       // [2] S is in tensor memory
  uint64_t* s_empty = s_full + 2;                                 // [2] S has been read
  uint64_t* p_full = s_empty + 2;                                 // [2] the weights' pieces are in tensor memory
  uint64_t* p_empty = p_full + 2;                                 // [2] P V has read them
  uint64_t* st_full = p_empty + 2;                                // [STATS] a page's statistics are there
  uint64_t* t_full = st_full + STATS;                             // [3] a piece of P V is in tensor memory
  uint64_t* t_empty = t_full + 3;                                 // [3] it has been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(t_empty + 3);
  uint32_t* again = tmem_slot + 1;                                // [4] rows with an entry that is not finite, a bit a row
  volatile uint32_t* failed = again + 4;                          // a wait of the block has run out
  const int hp = a.hp, tok = ROWS / hp, group = a.n_heads / a.n_kv_heads, chunks = group / hp;
  const int per_seq = a.n_kv_heads * chunks, from_end = blockIdx.x / a.columns, column = blockIdx.x - from_end * a.columns;
  const int s = column / per_seq, part = column - s * per_seq, kvh = part / chunks, h0 = kvh * group + (part - kvh * chunks) * hp;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    for (int i = 0; i < MAX_STAGES; ++i) { mbar_init(&kv_full[i], 4); mbar_init(&kv_empty[i], 1); }
    for (int i = 0; i < 2; ++i) { mbar_init(&s_full[i], 1); mbar_init(&s_empty[i], 128); mbar_init(&p_full[i], 128); mbar_init(&p_empty[i], 1); }
    for (int i = 0; i < STATS; ++i) mbar_init(&st_full[i], 128);
    for (int i = 0; i < 3; ++i) { mbar_init(&t_full[i], 1); mbar_init(&t_empty[i], 128); }
    for (int i = 0; i < 4; ++i) again[i] = 0;
    *failed = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    fence_async_shared();
  }
  pdl_wait();
  const int start = a.seq_starts[s], n_new = a.seq_starts[s + 1] - start, tok0 = ((int)gridDim.x / a.columns - 1 - from_end) * tok;
  const int kv_len = a.kv_lens[s];
  if (tok0 >= n_new || kv_len <= a.shorter) return;
  if (warp == 1) tmem_alloc(tmem_slot, TM_COLS);
  const int n_tok = min(tok, n_new - tok0), pos0 = kv_len - n_new + tok0, last_pos = pos0 + n_tok - 1;
  const int first_key = a.chunk > 0 ? pos0 - pos0 % a.chunk : ((a.window > 0 && pos0 - a.window + 1 > 0) ? pos0 - a.window + 1 : 0);   // of the block's first token
  const int keep_first = a.keep_first;                            // (arguments that a loop over pages wants are read before it: every wait in it would have them read again)
  auto next_page = [&](int t) {                                   // the next page that a pair of the block sees (the same for every thread)
    while (t * PAGE <= last_pos && t * PAGE + PAGE <= first_key && t * PAGE >= keep_first) ++t;
    return t;
  };
  const int* pages = a.page_table + (int64_t)s * a.table_width;
  const int k_eights = (a.dk + 15) / 16 * 2, v_eights = a.alias ? 0 : (a.dv + 15) / 16 * 2;      // pieces of eight entries of a row, up to whole sixteens (zeros)
  {                                                               // the queries, by all
#pragma unroll 2
    for (int i = threadIdx.x; i < ROWS * k_eights; i += THREADS) {
      const int r = i / k_eights, c = i - r * k_eights, ti = r / hp;
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
      if (ti < n_tok && c * 8 < a.dk) {
        const float4* src = reinterpret_cast<const float4*>(a.q + (int64_t)(start + tok0 + ti) * a.ld_q + (int64_t)(h0 + r - ti * hp) * a.dk + c * 8);
        x = src[0];
        y = src[1];
      }
      put8(q_tile + (c >> 3) * Q_BLOCK + r * 128 + (((c & 7) ^ (r & 7)) << 4), q_piece, x, y);
    }
    fence_async_shared();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (mbar_wait(bar, parity)) return true;
    *failed = 1;
    return false;
  };
  // after a role's last page: the rows that have to be worked out again, by all warps that have the registers
  auto finish = [&]() {
    asm volatile("bar.sync 1, 256;" ::: "memory");
    if ((again[0] | again[1] | again[2] | again[3]) != 0) rows_again<2 * CPW, float, float>(a, again, 12, 8);
  };

  if (warp < 4) {
    regs_fewer<32>();
    if (warp == 1) {                                              // S = Q K^T (the whole warp, its elected lane issues: see elect_one)
      const int k_steps = (a.dk + 15) / 16;
      const uint32_t idesc = umma_instr_desc(ROWS, PAGE);
      const uint64_t q_desc = sw128_desc(smem_u32(q_tile)), k_desc = sw128_desc(smem_u32(ring));
      const bool one = elect_one();
      bool ok = true;
      int u = 0, st = 0;                                          // u: blocks of 64 entries so far, each an accumulator of its own (the tensor core truncates where it accumulates)
      uint32_t turn = 0;
      for (int t = next_page(0); t * PAGE <= last_pos && ok; t = next_page(t + 1)) {
        if (!wait(&kv_full[st], turn)) { ok = false; break; }
        const uint64_t k_at = k_desc + st * (stage_bytes >> 4);
        int left = k_steps;
        for (int kb = 0; kb < k_blocks; ++kb, ++u, left -= 4) {
          const int b = u & 1;
          if (u >= 2 && !wait(&s_empty[b], ((u >> 1) & 1) ^ 1)) { ok = false; break; }
          tc_fence_after();
          const uint32_t d = tmem_base + TM_S + b * 64;
          if (one) {
#pragma unroll
            for (int x = 0; x < 6; ++x) {
              const uint64_t qd = q_desc + PA[x] * (q_piece >> 4) + kb * (Q_BLOCK >> 4), kd = k_at + PB[x] * (k_piece >> 4) + kb * (PAGE_BLOCK >> 4);
              if (left >= 4) {
#pragma unroll
                for (int k = 0; k < 4; ++k) umma(d, qd + k * 2, kd + k * 2, idesc, (x > 0 || k > 0) ? 1u : 0u);
              } else {
                for (int k = 0; k < left; ++k) umma(d, qd + k * 2, kd + k * 2, idesc, (x > 0 || k > 0) ? 1u : 0u);
              }
            }
            umma_commit(&s_full[b]);
          }
        }
        if (++st == stages) { st = 0; turn ^= 1; }
      }
    } else if (warp == 2) {                                       // T = P V, by another warp
      const uint64_t v_desc = sw128_mn_desc(smem_u32(ring) + v_off);
      const bool one = elect_one();
      const int dv = a.dv;
      bool ok = true;
      int i = 0, st = 0, slot = 0, g = 0;
      uint32_t slot_turn = 0;
      for (int t = next_page(0); t * PAGE <= last_pos && ok; t = next_page(t + 1), ++i) {
        const int b = i & 1;
        if (!wait(&p_full[b], (i >> 1) & 1)) { ok = false; break; }
        const uint32_t p_at = tmem_base + TM_P + b * P_STEP;
        const uint64_t v_at = v_desc + st * (stage_bytes >> 4);
        for (int c = 0; c < 2 * v_blocks; ++c, ++g) {             // 64 columns' small products, then their h h: apart, so that nothing truncates what is small once it is large
          if (g >= SLOTS && !wait(&t_empty[slot], slot_turn ^ 1)) { ok = false; break; }
          tc_fence_after();
          const uint32_t idesc = umma_instr_desc(ROWS, min(CW, (dv - (c >> 1) * CW + 15) & ~15), false, true), d = tmem_base + TM_T + slot * CW;
          const uint64_t vd = v_at + (c >> 1) * (PAGE_BLOCK >> 4);
          if (one) {
            if ((c & 1) == 0) {
#pragma unroll
              for (int x = 0; x < 5; ++x)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) umma_ta(d, p_at + PA[x] * 32 + kk * 8, vd + PB[x] * (v_piece >> 4) + kk * (2048 >> 4), idesc, (x > 0 || kk > 0) ? 1u : 0u);
            } else {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_ta(d, p_at + kk * 8, vd + kk * (2048 >> 4), idesc, kk > 0 ? 1u : 0u);
            }
            umma_commit(&t_full[slot]);
          }
          if (++slot == SLOTS) { slot = 0; slot_turn ^= 1; }
        }
        if (!ok) break;
        if (one) {
          umma_commit(&p_empty[b]);
          umma_commit(&kv_empty[st]);
        }
        if (++st == stages) st = 0;
      }
    }
  } else if (warp < 12) {
    // ---- keys and values into pieces, by two groups of four warps that take pages in turn; four eights of a row a thread at a time
    regs_fewer<80>();
    const int tid = threadIdx.x & 127, mine = (warp >> 2) - 1;
    const int64_t k_step = (int64_t)a.n_kv_heads * PAGE * a.dk, v_step = (int64_t)(a.n_kv_heads / a.key_maps) * PAGE * a.dv;
    bool ok = true;
    auto bring = [&](uint8_t* dst, uint32_t step, const float* src, int width, int eights, int n_live) {
      const int rows = 128 / eights, rest = 128 - rows * eights;  // (from one of a thread's places to the next)
      int r = tid / eights, c = tid - r * eights;
      for (int i = tid; i < PAGE * eights; i += 512) {
        float4 x[4], y[4];
        int at[4];
#pragma unroll
        for (int f = 0; f < 4; ++f) {
          x[f] = y[f] = make_float4(0.f, 0.f, 0.f, 0.f);
          at[f] = r < PAGE ? (c >> 3) * (int)PAGE_BLOCK + r * 128 + (((c & 7) ^ (r & 7)) << 4) : -1;
          if (r < n_live && c * 8 < width) {                      // (places past the block's last position may hold anything)
            const float4* from = reinterpret_cast<const float4*>(src + r * width + c * 8);
            x[f] = from[0];
            y[f] = from[1];
          }
          r += rows;
          c += rest;
          if (c >= eights) { c -= eights; ++r; }
        }
#pragma unroll
        for (int f = 0; f < 4; ++f)
          if (at[f] >= 0) put8(dst + at[f], step, x[f], y[f]);
      }
    };
    // (with room for one page only the first group works: a group that waits for a place to be given back must not be two givings behind)
    const int takers = stages > 1 ? 2 : 1;
    int j = mine, t = next_page(0);
    if (mine == 1) t = next_page(t + 1);
    for (; mine < takers && t * PAGE <= last_pos && ok; j += takers) {
      const int page = pages[t], st = j % stages, n_live = min(PAGE, last_pos + 1 - t * PAGE);
      if (j >= stages && !wait(&kv_empty[st], ((j / stages) & 1) ^ 1)) { ok = false; break; }
      uint8_t* at = ring + st * stage_bytes;
      bring(at, k_piece, a.k_pages + (int64_t)page * k_step + (int64_t)kvh * PAGE * a.dk, a.dk, k_eights, n_live);
      if (v_eights > 0) bring(at + v_off, v_piece, a.v_pages + (int64_t)page * v_step + (int64_t)(kvh / a.key_maps) * PAGE * a.dv, a.dv, v_eights, n_live);
      fence_async_shared();
      __syncwarp();
      if (lane == 0 && !(a.skip_copy && j == 0)) mbar_arrive_one(&kv_full[st]);
      t = next_page(t + 1);
      if (takers == 2) t = next_page(t + 1);
    }
  } else if (warp < 16) {
    // ---- scores into weights: a thread a row
    if (CPW == 1) regs_more<152>(); else regs_more<112>();
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int ti = row / hp, pos = pos0 + ti;
    const int first = a.window > 0 ? pos - a.window + 1 : (a.chunk > 0 ? pos - pos % a.chunk : 0);
    const float slope = a.slope_span > 0.f ? exp2f(-a.slope_span * (float)(h0 + row - ti * hp + 1) / (float)a.n_heads) * LOG2E : 0.f;
    // keys from `clear_from` up to `clear_to` (and the kept first ones) are seen by every live row of the warp
    const int clear_to = pos0 + quarter * 32 / hp, far = pos0 + min((quarter * 32 + 31) / hp, n_tok - 1);
    const int clear_from = a.window > 0 ? far - a.window + 1 : (a.chunk > 0 ? far - far % a.chunk : 0);
    const float scale2 = a.scale * LOG2E;
    const bool capped = a.softcap > 0.f, sloped = a.slope_span > 0.f, plain = !capped && !sloped && a.scale > 0.f;
    const float cap_in = a.cap_in, cap_out = a.cap_out;
    const float unit = plain ? scale2 : 1.f;
    const uint64_t unit2 = pair(unit, unit);
    int j = 0, u = 0;
    for (int t = next_page(0); t * PAGE <= last_pos; t = next_page(t + 1), ++j) {
      const int b = j & 1, key0 = t * PAGE;
      const uint32_t turn = (j >> 1) & 1;
      float sc[64];
      bool come = true;
      for (int kb = 0; kb < k_blocks; ++kb, ++u) {
        if (!wait(&s_full[u & 1], (u >> 1) & 1)) { come = false; break; }
        tc_fence_after();
        if (kb == 0) {
          uint32_t* raw = reinterpret_cast<uint32_t*>(sc);
          tmem_ld32(lanes + TM_S + (u & 1) * 64, raw);
          tmem_ld32(lanes + TM_S + (u & 1) * 64 + 32, raw + 32);
          tmem_ld_wait();
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float more[16];
            tmem_ld16(lanes + TM_S + (u & 1) * 64 + q * 16, more);
#pragma unroll
            for (int e = 0; e < 16; ++e) sc[q * 16 + e] += more[e];
          }
        }
        tc_fence_before();
        mbar_arrive_one(&s_empty[u & 1]);
      }
      if (!come) break;
      // Scores in units of log2, or, where nothing but a positive factor is on them, as they are with the factor `unit` still owed.
      if (!plain) shape_scores(sc, capped, cap_in, cap_out, scale2, sloped, slope, pos - key0);
      if (!(key0 + PAGE - 1 <= clear_to && (key0 >= clear_from || key0 + PAGE <= keep_first)))      // some pair does not see all of the page
        hide_scores(sc, pos - key0, first - key0, keep_first - key0);
      float top[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int c = 0; c < 64; ++c) top[c & 3] = fmaxf(top[c & 3], sc[c]);
      const float most = ceilf(fmaxf(fmaxf(top[0], top[1]), fmaxf(top[2], top[3])) * unit), base = most == -INFINITY ? 0.f : most;
      if (j >= 2 && !wait(&p_empty[b], turn ^ 1)) break;
      tc_fence_after();
      const uint64_t less = pair(-base, -base);
      uint64_t sum2[2] = {0ull, 0ull};
      const uint32_t p_at = lanes + TM_P + b * P_STEP, low_at = p_at + 64;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t ph[8], pm[8], pl[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          float x, y;
          unpair(fma2(pair(sc[q * 16 + 2 * e], sc[q * 16 + 2 * e + 1]), unit2, less), x, y);
          x = exp2_fast(x);
          y = exp2_fast(y);
          sum2[e & 1] = add2(sum2[e & 1], pair(x, y));
          ph[e] = cut(x, y);
          pm[e] = cut(x, y);
          pl[e] = pack(x, y);
        }
        tmem_st8(p_at + q * 8, ph);
        tmem_st8(p_at + 32 + q * 8, pm);
        tmem_st8(low_at + q * 8, pl);
      }
      float s0, s1;
      unpair(add2(sum2[0], sum2[1]), s0, s1);
      stats[(j % STATS) * ROWS + row] = make_float2(most, s0 + s1);
      mbar_arrive_one(&st_full[j % STATS]);
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive_one(&p_full[b]);
    }
    finish();
  } else {
    // ---- the running output: a thread a row and CPW x 64 of its columns
    if (CPW == 1) regs_more<120>(); else regs_more<176>();
    const int quarter = warp & 3, row = quarter * 32 + lane;
    const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16) + TM_T;
    const int ti = row / hp, h = h0 + row - ti * hp;
    const int64_t grow = start + tok0 + ti;
    const float* gate = a.gate == nullptr ? nullptr : (a.gate_heads ? a.gate + grow * a.ld_gate + h : a.gate + grow * a.ld_gate + (int64_t)h * a.dv);
    if (gate != nullptr && ti < n_tok) {                          // (the gate is asked for now: it is wanted after the last page)
      const int bytes = a.gate_heads ? 4 : 4 * a.dv;
      for (int at = 0; at < bytes; at += 128) asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const char*>(gate) + at));
    }
    float run_max = -INFINITY, run_sum = 0.f;
    uint64_t o[CPW * 32];
#pragma unroll
    for (int c = 0; c < CPW * 32; ++c) o[c] = 0ull;
    bool ok = true;
    int j = 0;
    for (int t = next_page(0); t * PAGE <= last_pos && ok; t = next_page(t + 1), ++j) {
      if (!wait(&st_full[j % STATS], (j / STATS) & 1)) { ok = false; break; }
      const float2 st = stats[(j % STATS) * ROWS + row];
      const float new_max = fmaxf(run_max, st.x);
      const float keep = run_max == -INFINITY ? 0.f : exp2_whole(run_max - new_max), take = st.x == -INFINITY ? 0.f : exp2_whole(st.x - new_max);
      // (a page that the row sees nothing of has weights of zero and a sum of zero, or NaN, which stays)
      run_sum = fmaf(run_sum, keep, st.y * (st.x == -INFINITY ? 1.f : take));
      run_max = new_max;
      const uint64_t keep2 = pair(keep, keep), take2 = pair(take, take);
#pragma unroll
      for (int c = 0; c < CPW; ++c) {
        if (c >= v_blocks) continue;
        const int g = (j * v_blocks + c) * 2, turns = g / SLOTS, slot = g - turns * SLOTS, slot2 = slot + 1 == SLOTS ? 0 : slot + 1;
        if (!wait(&t_full[slot], turns & 1) || !wait(&t_full[slot2], (slot2 == 0 ? turns + 1 : turns) & 1)) { ok = false; break; }
        tc_fence_after();
        constexpr int Q = CPW == 1 ? 16 : 8;                      // columns at a time, as registers allow
#pragma unroll
        for (int q = 0; q < CW / Q; ++q) {
          uint64_t v[Q / 2];
          tmem_ld_sum<Q>(lanes + slot * CW + q * Q, lanes + slot2 * CW + q * Q, v);
#pragma unroll
          for (int e = 0; e < Q / 2; ++e) {
            uint64_t& x = o[c * (CW / 2) + q * (Q / 2) + e];
            x = fma2(x, keep2, mul2(v[e], take2));
          }
        }
        tc_fence_before();
        mbar_arrive_one(&t_empty[slot]);
        mbar_arrive_one(&t_empty[slot2]);
      }
    }
    bool bad = false;                                             // some entry is not finite (0 times it is none)
    if (ok && ti < n_tok) {
      uint64_t odd = 0ull;
      float inv;
      if (a.sinks == nullptr) {
        inv = 1.0f / run_sum;
      } else {                                                    // a sink is one more term of the denominator
        const float most = run_max * LN2, sink = a.sinks[h], m = fmaxf(most, sink), f = expf(most - m);
        inv = f / fmaf(run_sum, f, expf(sink - m));
      }
      if (gate != nullptr && a.gate_heads) inv *= sigmoid(*gate);
      float* dst = a.out + grow * a.ld_out + (int64_t)h * a.dv;
      auto leave = [&](auto gated) {                              // (apart: what gates take makes the way of those without any longer by fetching it)
#pragma unroll
        for (int d = 0; d < CPW * 64; d += 4) {                   // (dv is a multiple of 8)
          if (d >= a.dv) continue;
          float x[4];
          unpair(o[d / 2], x[0], x[1]);
          unpair(o[d / 2 + 1], x[2], x[3]);
          odd = fma2(o[d / 2 + 1], 0ull, fma2(o[d / 2], 0ull, odd));
#pragma unroll
          for (int e = 0; e < 4; ++e) x[e] *= inv;
          if (gated.value) {
            const float4 z = *reinterpret_cast<const float4*>(gate + d);
            x[0] *= sigmoid(z.x); x[1] *= sigmoid(z.y); x[2] *= sigmoid(z.z); x[3] *= sigmoid(z.w);
          }
          *reinterpret_cast<float4*>(dst + d) = make_float4(x[0], x[1], x[2], x[3]);
        }
      };
      if (gate != nullptr && !a.gate_heads) leave(std::true_type());
      else leave(std::false_type());
      float odd0, odd1;
      unpair(odd, odd0, odd1);
      bad = !(odd0 + odd1 == 0.f) || not_finite(inv);
    }
    note_again(again, quarter, bad);
    finish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*failed != 0) outlast_what_is_in_flight();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, TM_COLS);
  }
}

struct Layout { int stages; size_t smem; };
Layout layout_of(int dk, int dv, bool alias) {
  const size_t kb = (dk + 63) / 64, vb = alias ? 0 : (dv + 63) / 64, fixed = 3 * kb * Q_BLOCK + SMEM_REST, stage = 3 * (kb + vb) * PAGE_BLOCK;
  Layout z;
  z.stages = fixed >= SMEM_MOST ? 0 : (int)std::min<size_t>(MAX_STAGES, (SMEM_MOST - fixed) / stage);
  z.smem = fixed + z.stages * stage;
  return z;
}

template <int CPW>
int launch(const WideArgs& a, int max_new, size_t smem, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(scored_wide_kernel<CPW>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MOST);
    if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "attention (scored, 32-bit prompts): cannot reserve %zu bytes of shared memory: %s", SMEM_MOST, cudaGetErrorString(e));
    configured = true;
  }
  const int tok = ROWS / a.hp;
  const int64_t tiles = (int64_t)a.columns * ((max_new + tok - 1) / tok);
  KVAD_REQUIRE(tiles < (1ll << 31), "attention (scored, 32-bit prompts): %lld tiles are more than one launch takes", (long long)tiles);
  kvad_launch(scored_wide_kernel<CPW>, dim3((unsigned)tiles), dim3(THREADS), smem, stream, a);
  KVAD_CHECK_LAUNCH("attention_scored_wide");
  return KVAD_OK;
}

}  // namespace

// 1 if prompts of these sizes run here: rows in eights of entries, values up to 128 entries, the queries' pieces and a page's in shared memory.
KVAD_EXPORT int kvad_attention_scored_wide_takes(int dk, int dv, int alias) {
  return dk > 0 && dv > 0 && dk % 8 == 0 && dv % 8 == 0 && dv <= 128 && layout_of(dk, dv, alias != 0).stages >= 1 ? 1 : 0;
}

// `shorter`: sequences of up to so many positions are left alone.
KVAD_EXPORT int kvad_attention_scored_wide(const float* q, int64_t ld_q, float* out, int64_t ld_out, const float* gate, int64_t ld_gate, int gate_heads,
                                           const float* sinks, const int* seq_starts, const int* kv_lens, const int* page_table, int table_width,
                                           const float* k_pages, const float* v_pages, int n_seqs, int n_heads, int n_kv_heads, int dk, int dv,
                                           int page_size, int max_new, float scale, float softcap, float slope_span, int window, int keep_first,
                                           int chunk, int key_maps, int shorter, cudaStream_t stream) {
  KVAD_REQUIRE(n_seqs >= 0 && n_heads > 0 && n_kv_heads > 0 && dk > 0 && dv > 0 && table_width > 0 && max_new >= 0 && keep_first >= 0,
               "attention (scored, 32-bit prompts): bad sizes seqs=%d heads=%d kv_heads=%d dk=%d dv=%d", n_seqs, n_heads, n_kv_heads, dk, dv);
  KVAD_REQUIRE(n_heads % n_kv_heads == 0, "attention (scored, 32-bit prompts): %d heads do not divide into %d key/value heads", n_heads, n_kv_heads);
  KVAD_REQUIRE(chunk <= 0 || window <= 0, "attention (scored, 32-bit prompts): a chunk goes without a window");
  const bool alias = v_pages == k_pages;
  KVAD_REQUIRE(key_maps >= 1 && n_kv_heads % key_maps == 0 && (key_maps == 1 || !alias), "attention (scored, 32-bit prompts): %d key heads do not share values %d by %d", n_kv_heads, key_maps, key_maps);
  KVAD_REQUIRE(!alias || dv <= dk, "attention (scored, 32-bit prompts): values read from the keys cannot be longer than a key");
  if (page_size != PAGE || !kvad_attention_scored_wide_takes(dk, dv, alias))
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "attention (scored, 32-bit prompts): pages of %d, keys of %d, values of %d are not taken", page_size, dk, dv);
  const uintptr_t all = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_pages) | reinterpret_cast<uintptr_t>(v_pages) | reinterpret_cast<uintptr_t>(out);
  if ((all & 15) || ld_q % 4 != 0 || ld_out % 4 != 0 || (gate != nullptr && !gate_heads && ((reinterpret_cast<uintptr_t>(gate) & 15) || ld_gate % 4 != 0)))
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "attention (scored, 32-bit prompts): rows must lie on 16-byte boundaries");
  if (n_seqs == 0 || max_new == 0) return KVAD_OK;
  WideArgs a;
  a.q = q; a.ld_q = ld_q; a.out = out; a.ld_out = ld_out; a.gate = gate; a.ld_gate = ld_gate; a.gate_heads = gate_heads; a.sinks = sinks;
  a.seq_starts = seq_starts; a.kv_lens = kv_lens; a.page_table = page_table; a.table_width = table_width; a.k_pages = k_pages; a.v_pages = v_pages;
  a.n_heads = n_heads; a.n_kv_heads = n_kv_heads; a.dk = dk; a.dv = dv; a.alias = alias ? 1 : 0; a.key_maps = key_maps;
  a.scale = scale; a.softcap = softcap; a.slope_span = slope_span; a.window = window > 0 ? window : 0; a.keep_first = window > 0 ? keep_first : 0;
  a.chunk = chunk > 0 ? chunk : 0;
  const float cap = std::min(softcap, 1.2676506e30f), ratio = scale / cap;      // (see attention_scored_prompt.cu)
  a.cap_in = softcap > 0.f ? std::max(-3.402823466e38f, std::min(3.402823466e38f, ratio)) : 0.f; a.cap_out = cap * LOG2E;
  a.hp = 1;
  while (a.hp < 16 && (n_heads / n_kv_heads) % (a.hp * 2) == 0) a.hp *= 2;
  KVAD_REQUIRE((int64_t)n_seqs * (n_heads / a.hp) < (1ll << 31), "attention (scored, 32-bit prompts): %d sequences x %d heads are more than one launch takes", n_seqs, n_heads);
  a.columns = n_seqs * (n_heads / a.hp);
  a.shorter = shorter;
  a.skip_copy = g_skip_copy;
  g_skip_copy = 0;
  const Layout z = layout_of(dk, dv, alias);
  a.stages = z.stages;
  return dv <= 64 ? launch<1>(a, max_new, z.smem, stream) : launch<2>(a, max_new, z.smem, stream);
}

// How many bounded waits have run out since the library was loaded (0 in a healthy run).  Synchronises the device.
KVAD_EXPORT int kvad_attention_scored_wide_status() {
  int n = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&n, g_wait_timeouts, sizeof(int));
  if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "attention_scored_wide_status: %s", cudaGetErrorString(e));
  return n;
}

// Tests of the bounded waits: `wait_limit` > 0 sets how many polls a wait makes before it gives up (0: the library's own limit); `skip_copy` leaves the first page out of
// the NEXT launch's blocks, so that the wait for it runs out.  Synchronises the device.
KVAD_EXPORT int kvad_attention_scored_wide_test_hooks(unsigned wait_limit, int skip_copy) {
  g_skip_copy = skip_copy;
  return set_wait_limit(wait_limit);
}

KVAD_DEFINE_LAST_ERROR()
