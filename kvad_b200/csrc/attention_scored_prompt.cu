// Softmax attention of prompt rows over the paged cache with shaped scores (`attention_scored.cu` says what a score can be
// given), on the 5th-generation tensor cores: bfloat16 queries, keys and values, 32-bit scores, softmax weights and sums.
//
//   S = Q K^T        tcgen05.mma, 128 (token, head) pairs x 64 keys of a page, in tensor memory
//   p = exp(s - m)   32-bit, m the page's own largest score of the row (a whole power of two): a page's weights wait for no other page
//   T = P V          p is cut into three bfloat16 pieces, p = h + m + l exactly (a weight keeps its 24 bits), which lie in tensor memory as the
//                    product's first operand, the smallest first.  The tensor core's truncating accumulation is kept to one page,
//   O = a O + b T    whose sum joins the 32-bit running sum in registers by rounded operations (a, b: 2^(old maximum - new), 2^(m - new), both exact)
//
// A block works 128 (token, head) pairs that share a key head: 128 / hp consecutive tokens of one sequence times hp heads of the group.
// Roles, so that the tensor core's queue never waits for one thread's chain: one warp brings the queries once and the pages' keys and
// values by TMA into a ring; one warp issues S = Q K^T, up to two pages ahead of P V, which another issues; NS groups of four warps turn the pages' scores
// into weights (a thread a row, pages in turn); NA groups of four warps keep the running output (a thread a row and up to 128 of its
// columns).  NS = 2, NA = 1 for values of up to 128 entries, where softmax takes the time; NS = 1, NA = 2 above, where the products do.
// P V goes in pieces of columns through two or three places of tensor memory, so that one can be read while the next is worked out.
// Pages that no pair of the block sees are skipped; tiles are launched longest first.  Every wait is bounded (`kvad_attention_scored_prompt_status`).
//
// What bounds it.  Keys and values of 256: a page takes 16 products of 128 x 64 x 16 (48 cycles each: both operands in shared memory) and 24 of
// 128 x 128 x 16 (64), 2300 cycles, and runs in 2850.  Values of up to 64: the weights, ~1000 instructions a row and page, 1400 cycles a page; then the
// start of a block (~5 us with the first page's chain), of which two go one after another where there are more than 148 tiles.
// Graph-replayed launches, us: 2 x 1024 rows of 16 heads over a latent of 256: 1100 on the CUDA cores, 127 by mma.sync, 40 here; 16 heads of 64 on 4 key heads, capped,
// window 512: 358, 55, 28 (42 where scores lie beyond 0.45 caps); without cap and window 46, 23.  64 new rows of 4 sequences with 300 cached positions: latent 47.6, 17.7; 16 heads of 64: 15.4, 10.4;
// 2 new rows: 38.4, 14.0; 12.3, 9.1.  With a head a group many short sequences were faster by mma.sync, two blocks an SM: 32 of 2 rows 14, 26; of 32 rows 17, 26.  (On the way: products issued by a
// branch of one lane 64, by the whole warp 50, S and P V by warps of their own with wide P V 40.)
#include <algorithm>
#include <type_traits>

#include "scored_tiles.cuh"

using namespace kvad;

namespace {

constexpr int THREADS = 512, MAX_STAGES = 4;
constexpr int STATS = 8;             // pages whose statistics are kept: weights run up to two pages ahead of P V, P V up to three of the output
constexpr uint32_t TM_COLS = 512;
constexpr size_t SMEM_MOST = 226 * 1024, SMEM_REST = STATS * ROWS * 8 + 320 + 1024;      // (statistics, barriers, alignment)

struct PromptArgs {
  const __nv_bfloat16* q; int64_t ld_q; const __nv_bfloat16* k_pages; const __nv_bfloat16* v_pages;      // (read by `row_again` alone: the products' operands come by TMA)
  void* out; int64_t ld_out;
  const __nv_bfloat16* gate; int64_t ld_gate; int gate_heads;    // gate_heads: one number per row and head
  const float* sinks;
  const int* seq_starts; const int* kv_lens; const int* page_table; int table_width;
  int n_heads, n_kv_heads, dk, dv, hp, alias, key_maps, stages, vec;
  int columns;                                                    // tiles of one place in their sequence: sequences x heads / hp (the grid is these, the last place first)
  float scale, softcap, slope_span;
  float cap_in, cap_out;                                          // a capped score: cap_out * tanh(cap_in * (q . k)), in units of log2
  int window, keep_first, chunk;
  int skip_copy;                                                  // (tests: a block's first page is left out, so that the wait for it runs out)
};

int g_skip_copy = 0;

// NS: groups of four warps that turn scores into weights; CPW: 64-column pieces of the output that a group of four warps keeps.  IN_TURN: there is room for a page's keys or
// its values only, which come into the same place one after the other.
template <int NS, int CPW, bool F32OUT, bool IN_TURN>
__global__ void __launch_bounds__(THREADS, 1)
scored_prompt_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v, const __grid_constant__ PromptArgs a) {
  // Tensor-memory columns: the places of P V, S of two pages (64 each), the weights' pieces of two pages (32 columns each: two bfloat16 a column).  With values
  // above 128 entries P V takes two places of 128 (products 128 wide leave the issuing warp time for its waits), and the third piece takes its page's S' place.
  constexpr bool S_IS_P = NS == 1;
  constexpr int NI = NS == 1 ? 8 : 2 * CPW, FINISHERS = THREADS / 32 - 4;      // 32s of a value's entries; warps that finish a block together
  constexpr int CW = NS == 1 ? 128 : 64, SLOTS = NS == 1 ? 2 : 3;
  // With a 32-bit output the small pieces' products have an accumulator of their own, so that nothing truncates what is small once it is large; a rounding to bfloat16 hides it.
  constexpr int PARTS = F32OUT ? 2 : 1;
  constexpr bool TOGETHER = PARTS == 2 && NS == 2;      // the two meet before they join the running output (where two groups of warps share the places, a group has one of its own)
  constexpr uint32_t TM_T = 0, TM_S = SLOTS * CW, TM_P = TM_S + 128, P_STEP = S_IS_P ? 64 : 96;
  static_assert(TM_P + 2 * P_STEP <= TM_COLS, "tensor memory");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  const int k_blocks = (a.dk + 63) / 64, v_blocks = (a.dv + 63) / 64, n_chunks = (a.dv + CW - 1) / CW, stages = a.stages;
  const uint32_t k_bytes = k_blocks * PAGE_BLOCK, v_bytes = a.alias ? 0 : v_blocks * PAGE_BLOCK, v_off = a.alias || IN_TURN ? 0 : k_bytes;
  const uint32_t stage_bytes = IN_TURN ? max(k_bytes, v_bytes) : k_bytes + v_bytes;
  uint8_t* q_tile = smem;
  uint8_t* ring = smem + k_blocks * Q_BLOCK;                      // stage: keys, then values (or none: the keys)
  float2* stats = reinterpret_cast<float2*>(ring + stages * stage_bytes);      // [STATS][ROWS] a page's largest score and sum of weights, per row
  uint64_t* q_full = reinterpret_cast<uint64_t*>(stats + STATS * ROWS);
  uint64_t* kv_full = q_full + 1;                                 // [stages] a page has come (in turn: its keys, and [1] its values)
  uint64_t* kv_empty = kv_full + MAX_STAGES;                      // [stages] it has been used up
  uint64_t* s_full = kv_empty + MAX_STAGES;                       // [2] S is in tensor memory
  uint64_t* s_empty = s_full + 2;                                 // [2] S has been read
  uint64_t* p_full = s_empty + 2;                                 // [2] the weights' pieces are in tensor memory
  uint64_t* p_empty = p_full + 2;                                 // [2] P V has read them
  uint64_t* st_full = p_empty + 2;                                // [STATS] a page's statistics are there
  uint64_t* t_full = st_full + STATS;                                 // [3] a piece of P V is in tensor memory
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
    prefetch_tensormap(&map_q);
    prefetch_tensormap(&map_k);
    prefetch_tensormap(&map_v);
    mbar_init(q_full, 1);
    for (int i = 0; i < MAX_STAGES; ++i) { mbar_init(&kv_full[i], 1); mbar_init(&kv_empty[i], 1); }
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
  if (tok0 >= n_new) return;
  const int kv_len = a.kv_lens[s];
  if (warp == 1) tmem_alloc(tmem_slot, TM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const int n_tok = min(tok, n_new - tok0), pos0 = kv_len - n_new + tok0, last_pos = pos0 + n_tok - 1;
  const int first_key = a.chunk > 0 ? pos0 - pos0 % a.chunk : ((a.window > 0 && pos0 - a.window + 1 > 0) ? pos0 - a.window + 1 : 0);   // of the block's first token
  const int keep_first = a.keep_first;                            // (arguments that a loop over pages wants are read before it: every wait in it would have them read again)
  auto next_page = [&](int t) {                                   // the next page that a pair of the block sees (the same for every thread)
    while (t * PAGE <= last_pos && t * PAGE + PAGE <= first_key && t * PAGE >= keep_first) ++t;
    return t;
  };
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (mbar_wait(bar, parity)) return true;
    *failed = 1;
    return false;
  };
  // after a role's last page: the rows that have to be worked out again, by all warps that have the registers
  auto finish = [&]() {
    asm volatile("bar.sync 1, %0;" ::"n"(FINISHERS * 32) : "memory");
    if ((again[0] | again[1] | again[2] | again[3]) != 0) rows_again<NI, __nv_bfloat16, typename std::conditional<F32OUT, float, __nv_bfloat16>::type>(a, again, 4, FINISHERS);
  };

  if (warp < 4) {
    regs_fewer<40>();
    if (warp == 0 && lane == 0) {
      const int* pages = a.page_table + (int64_t)s * a.table_width;
      const int n_kv = a.n_kv_heads, n_v = n_kv / a.key_maps, v_head = kvh / a.key_maps;
      const bool alias = a.alias;
      int t = next_page(0), page_next = pages[t];
      mbar_expect_tx(q_full, k_blocks * Q_BLOCK);
      for (int b = 0; b < k_blocks; ++b) tma_load_3d(q_tile + b * Q_BLOCK, &map_q, q_full, b * 64, h0, start + tok0);
      int j = 0, st = 0;
      uint32_t turn = 0;
      for (int t_next; t * PAGE <= last_pos; t = t_next, ++j) {
        const int page = page_next;                               // (a page's place is looked up one page ahead)
        t_next = next_page(t + 1);
        if (t_next * PAGE <= last_pos) page_next = pages[t_next];
        if (j >= stages && !wait(&kv_empty[st], turn ^ 1)) break;
        uint8_t* at = ring + st * stage_bytes;
        if (!(a.skip_copy && j == 0)) {
          mbar_expect_tx(&kv_full[st], IN_TURN ? k_bytes : stage_bytes);
          const int y = (page * n_kv + kvh) * PAGE;
          for (int b = 0; b < k_blocks; ++b) tma_load_2d(at + b * PAGE_BLOCK, &map_k, &kv_full[st], b * 64, y);
          if (!alias) {
            uint64_t* come = IN_TURN ? &kv_full[1] : &kv_full[st];
            if (IN_TURN) {
              if (!wait(&s_full[j & 1], (j >> 1) & 1)) break;     // (the keys have been read)
              mbar_expect_tx(come, v_bytes);
            }
            const int yv = (page * n_v + v_head) * PAGE;
            for (int b = 0; b < v_blocks; ++b) tma_load_2d(at + v_off + b * PAGE_BLOCK, &map_v, come, b * 64, yv);
          }
        }
        if (++st == stages) { st = 0; turn ^= 1; }
      }
    } else if (warp == 1) {                                       // S = Q K^T (the whole warp, its elected lane issues: see elect_one)
      const int k_steps = (a.dk + 15) / 16;
      const uint32_t idesc = umma_instr_desc(ROWS, PAGE);
      const uint64_t q_desc = sw128_desc(smem_u32(q_tile)), k_desc = sw128_desc(smem_u32(ring));
      const uint32_t stage_step = stage_bytes >> 4;               // (descriptors count sixteens of bytes)
      const bool one = elect_one();
      bool ok = wait(q_full, 0);
      int j = 0, st = 0;
      uint32_t turn = 0;
      for (int t = next_page(0); t * PAGE <= last_pos && ok; t = next_page(t + 1), ++j) {
        const int b = j & 1;
        if (!wait(&kv_full[st], turn) || (j >= 2 && !wait(S_IS_P ? &p_empty[b] : &s_empty[b], ((j >> 1) & 1) ^ 1))) { ok = false; break; }
        tc_fence_after();
        const uint64_t k_at = k_desc + st * stage_step;
        const uint32_t d = tmem_base + TM_S + b * 64;
        if (one) {
          int left = k_steps;
          for (int kb = 0; kb < k_blocks; ++kb, left -= 4) {
            const uint64_t qd = q_desc + kb * (Q_BLOCK >> 4), kd = k_at + kb * (PAGE_BLOCK >> 4);
            if (left >= 4) {
#pragma unroll
              for (int k = 0; k < 4; ++k) umma(d, qd + k * 2, kd + k * 2, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            } else {
              for (int k = 0; k < left; ++k) umma(d, qd + k * 2, kd + k * 2, idesc, (kb > 0 || k > 0) ? 1u : 0u);
            }
          }
          umma_commit(&s_full[b]);
        }
        if (++st == stages) { st = 0; turn ^= 1; }
      }
    } else if (warp == 2) {                                       // T = P V, by another warp: a wait takes a hundred cycles even when it is over
      const uint64_t v_desc = sw128_mn_desc(smem_u32(ring) + v_off);
      const uint32_t stage_step = stage_bytes >> 4;
      const bool one = elect_one();
      const int dv = a.dv;
      bool ok = true;
      int i = 0, st = 0, slot = 0, g = 0;
      uint32_t slot_turn = 0;
      for (int t = next_page(0); t * PAGE <= last_pos && ok; t = next_page(t + 1), ++i) {
        const int b = i & 1;
        if (!wait(&p_full[b], (i >> 1) & 1) || (IN_TURN && !wait(&kv_full[1], i & 1))) { ok = false; break; }
        const uint32_t p_at = tmem_base + TM_P + b * P_STEP, low_at = tmem_base + (S_IS_P ? TM_S + b * 64 : TM_P + b * P_STEP + 64);
        const uint64_t v_at = v_desc + st * stage_step;
        for (int c = 0; c < n_chunks * PARTS; ++c, ++g) {
          if (g >= SLOTS && !wait(&t_empty[slot], slot_turn ^ 1)) { ok = false; break; }
          tc_fence_after();
          // (where two groups of warps share the places: all chunks' small products, then all their h h, so that each meets every turn of its own place)
          const int part = TOGETHER ? c & 1 : (c >= n_chunks ? 1 : 0), chunk = TOGETHER ? c >> 1 : c - part * n_chunks;
          const uint32_t idesc = umma_instr_desc(ROWS, min(CW, (dv - chunk * CW + 15) & ~15), false, true), d = tmem_base + TM_T + slot * CW;
          const uint64_t vd = v_at + chunk * (CW / 64) * (PAGE_BLOCK >> 4);
          if (one) {
            if (part == 0) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_ta(d, low_at + kk * 8, vd + kk * (2048 >> 4), idesc, kk > 0 ? 1u : 0u);
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_ta(d, p_at + 32 + kk * 8, vd + kk * (2048 >> 4), idesc, 1u);
            }
            if (part == PARTS - 1) {
#pragma unroll
              for (int kk = 0; kk < 4; ++kk) umma_ta(d, p_at + kk * 8, vd + kk * (2048 >> 4), idesc, (PARTS == 1 || kk > 0) ? 1u : 0u);
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
  } else if (warp < 4 + 4 * NS) {
    // ---- scores into weights: a thread a row
    if (NS == 2) { if (CPW == 1) regs_more<176>(); else regs_more<152>(); } else regs_more<136>();
    const int mine = (warp >> 2) - 1, quarter = warp & 3, row = quarter * 32 + lane;
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
    int t = next_page(0), j = mine;
    if (mine == 1) t = next_page(t + 1);
    for (; t * PAGE <= last_pos; j += NS) {
      const int b = j & 1, key0 = t * PAGE;
      const uint32_t turn = (j >> 1) & 1;
      if (!wait(&s_full[b], turn)) break;
      tc_fence_after();
      float sc[64];
      {
        uint32_t* raw = reinterpret_cast<uint32_t*>(sc);
        tmem_ld32(lanes + TM_S + b * 64, raw);
        tmem_ld32(lanes + TM_S + b * 64 + 32, raw + 32);
        tmem_ld_wait();
      }
      tc_fence_before();
      if (!S_IS_P) mbar_arrive_one(&s_empty[b]);
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
      const uint32_t p_at = lanes + TM_P + b * P_STEP, low_at = S_IS_P ? lanes + TM_S + b * 64 : p_at + 64;
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
      // Places past the sequence's end may hold anything: no weight is on them, but their values must not be NaN.  (Hidden places before the end hold numbers in earnest;
      // where one is not finite, `rows_again` sees to it.  Clearing those too took 2 x 1024 rows of 16 heads of 64 from 23.6 to 24.6 us, a latent of 256 from 40.1 to 42.0.)
      const int valid = kv_len - key0;
      if (valid < PAGE) {
        const int st = j % stages;
        if (IN_TURN ? !wait(&kv_full[1], j & 1) : !wait(&kv_full[st], (j / stages) & 1)) break;
        uint8_t* v_tile = ring + st * stage_bytes + v_off;
        for (int vb = 0; vb < v_blocks; ++vb)
          for (int x = row; x < (PAGE - valid) * 8; x += 128) *reinterpret_cast<uint4*>(v_tile + vb * PAGE_BLOCK + valid * 128 + x * 16) = make_uint4(0u, 0u, 0u, 0u);
        fence_async_shared();
      }
      tmem_st_wait();
      tc_fence_before();
      mbar_arrive_one(&p_full[b]);
      t = next_page(t + 1);
      if (NS == 2) t = next_page(t + 1);
    }
    finish();
  } else {
    // ---- the running output: a thread a row and CPW x 64 of its columns
    if (CPW == 1) regs_fewer<104>(); else regs_more<168>();
    const int quarter = warp & 3, row = quarter * 32 + lane, c0 = ((warp >> 2) - 1 - NS) * CPW;
    const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16) + TM_T;
    const int ti = row / hp, h = h0 + row - ti * hp;
    const int64_t grow = start + tok0 + ti;
    const __nv_bfloat16* gate = a.gate == nullptr ? nullptr : (a.gate_heads ? a.gate + grow * a.ld_gate + h : a.gate + grow * a.ld_gate + (int64_t)h * a.dv + c0 * 64);
    if (gate != nullptr && ti < n_tok) {                          // (the gate is asked for now: it is wanted after the last page)
      const int bytes = a.gate_heads ? 2 : 2 * min(CPW * 64, a.dv - c0 * 64);
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
      auto take_page = [&](int part, uint64_t stay) {             // this group's chunks of P V, one part of them
#pragma unroll
        for (int c = 0; c < CPW * 64 / CW; ++c) {
          if (c0 * 64 / CW + c >= n_chunks) continue;
          const int g = TOGETHER ? (j * n_chunks + c) * 2 : (j * PARTS + part) * n_chunks + c0 * 64 / CW + c, turns = g / SLOTS, slot = g - turns * SLOTS;
          const int slot2 = slot + 1 == SLOTS ? 0 : slot + 1;
          if (!wait(&t_full[slot], turns & 1) || (TOGETHER && !wait(&t_full[slot2], (slot2 == 0 ? turns + 1 : turns) & 1))) { ok = false; break; }
          tc_fence_after();
#pragma unroll
          for (int q = 0; q < CW / 16; ++q) {
            uint64_t v[8];
            if (TOGETHER) {
              tmem_ld_sum<16>(lanes + slot * CW + q * 16, lanes + slot2 * CW + q * 16, v);
            } else {
              float one[16];
              tmem_ld16(lanes + slot * CW + q * 16, one);
#pragma unroll
              for (int e = 0; e < 8; ++e) v[e] = pair(one[2 * e], one[2 * e + 1]);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              uint64_t& x = o[c * (CW / 2) + q * 8 + e];
              x = fma2(x, stay, mul2(v[e], take2));
            }
          }
          tc_fence_before();
          mbar_arrive_one(&t_empty[slot]);
          if (TOGETHER) mbar_arrive_one(&t_empty[slot2]);
        }
      };
      if (PARTS == 1 || TOGETHER) {
        take_page(0, keep2);
      } else {
#pragma unroll 1
        for (int part = 0; part < 2 && ok; ++part) take_page(part, part == 0 ? keep2 : pair(1.f, 1.f));
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
      if (gate != nullptr && a.gate_heads) inv *= sigmoid(__bfloat162float(*gate));
      auto leave = [&](auto gated) {                              // (apart: what gates take makes the way of those without any longer by fetching it: 8 us for 9.8, 17 rows of 8 heads of 128)
#pragma unroll
        for (int c = 0; c < CPW * 8; ++c) {
          const int d = c0 * 64 + c * 8;                            // (dv is a multiple of 8)
          if (d >= a.dv) continue;
          float x[8];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            unpair(o[c * 4 + e], x[2 * e], x[2 * e + 1]);
            odd = fma2(o[c * 4 + e], 0ull, odd);
          }
#pragma unroll
          for (int e = 0; e < 8; ++e) x[e] *= inv;
          if (F32OUT) {
            float* dst = reinterpret_cast<float*>(a.out) + grow * a.ld_out + (int64_t)h * a.dv + d;
            if (a.vec) {
              reinterpret_cast<float4*>(dst)[0] = make_float4(x[0], x[1], x[2], x[3]);
              reinterpret_cast<float4*>(dst)[1] = make_float4(x[4], x[5], x[6], x[7]);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) reinterpret_cast<float2*>(dst)[e] = make_float2(x[2 * e], x[2 * e + 1]);
            }
          } else {
            __nv_bfloat16* dst = reinterpret_cast<__nv_bfloat16*>(a.out) + grow * a.ld_out + (int64_t)h * a.dv + d;
            if (gated.value) {
              uint32_t z[4];
              if (a.vec) {
                const uint4 w = *reinterpret_cast<const uint4*>(gate + c * 8);
                z[0] = w.x; z[1] = w.y; z[2] = w.z; z[3] = w.w;
              } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) z[e] = *reinterpret_cast<const uint32_t*>(gate + c * 8 + 2 * e);
              }
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                x[2 * e] *= sigmoid(__uint_as_float(z[e] << 16));
                x[2 * e + 1] *= sigmoid(__uint_as_float(z[e] & 0xffff0000u));
              }
            }
            uint32_t w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = pack(x[2 * e], x[2 * e + 1]);
            if (a.vec) {
              *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
            } else {
#pragma unroll
              for (int e = 0; e < 4; ++e) *reinterpret_cast<uint32_t*>(dst + 2 * e) = w[e];
            }
          }
        }
      };
      if (!F32OUT && gate != nullptr && !a.gate_heads) leave(std::true_type());
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

int make_map(CUtensorMap* map, const void* at, int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
  EncodeTiledFn fn = encode_fn();
  if (fn == nullptr) KVAD_FAIL(KVAD_ERR_CUDA, "attention (scored, prompts): the driver has no cuTensorMapEncodeTiled");
  const cuuint32_t ones[3] = {1, 1, 1};
  const CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, const_cast<void*>(at), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) KVAD_FAIL(KVAD_ERR_CUDA, "attention (scored, prompts): cuTensorMapEncodeTiled failed (%d)", (int)r);
  return KVAD_OK;
}

template <int NS, int CPW, bool F32OUT, bool IN_TURN>
int launch(const CUtensorMap& q, const CUtensorMap& k, const CUtensorMap& v, const PromptArgs& a, int max_new, size_t smem, cudaStream_t stream) {
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(scored_prompt_kernel<NS, CPW, F32OUT, IN_TURN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MOST);
    if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "attention (scored, prompts): cannot reserve %zu bytes of shared memory: %s", SMEM_MOST, cudaGetErrorString(e));
    configured = true;
  }
  const int tok = ROWS / a.hp;
  const int64_t tiles = (int64_t)a.columns * ((max_new + tok - 1) / tok);
  KVAD_REQUIRE(tiles < (1ll << 31), "attention (scored, prompts): %lld tiles are more than one launch takes", (long long)tiles);
  kvad_launch(scored_prompt_kernel<NS, CPW, F32OUT, IN_TURN>, dim3((unsigned)tiles), dim3(THREADS), smem, stream, q, k, v, a);
  KVAD_CHECK_LAUNCH("attention_scored_prompt");
  return KVAD_OK;
}

struct Layout { int stages, in_turn; size_t smem; };
// As many pages on their way as fit (three keep all roles busy; one, for the longest keys, gives the same sums page by page; of keys above 512 entries, and above 448 with
// values above 192, a page's keys and values come in turn).
Layout layout_of(int dk, int dv, bool alias) {
  const size_t kb = (dk + 63) / 64, vb = alias ? 0 : (dv + 63) / 64, fixed = kb * Q_BLOCK + SMEM_REST, stage = (kb + vb) * PAGE_BLOCK;
  Layout z;
  z.stages = fixed >= SMEM_MOST ? 0 : (int)std::min<size_t>(MAX_STAGES, (SMEM_MOST - fixed) / stage);
  z.in_turn = 0;
  z.smem = fixed + z.stages * stage;
  if (z.stages == 0 && !alias && fixed + std::max(kb, vb) * PAGE_BLOCK <= SMEM_MOST) {
    z.stages = z.in_turn = 1;
    z.smem = fixed + std::max(kb, vb) * PAGE_BLOCK;
  }
  return z;
}

}  // namespace

// 1 if prompts of these sizes run here: whole 16-byte pieces, values up to 256 entries, the queries and a page in shared memory (whatever the output's type).
KVAD_EXPORT int kvad_attention_scored_prompt_takes(int dk, int dv, int alias, int) {
  return dk > 0 && dv > 0 && dk % 8 == 0 && dv % 8 == 0 && dv <= 256 && layout_of(dk, dv, alias != 0).stages >= 1 ? 1 : 0;
}

// `n_rows`, `n_pages`: how many rows q has and how many pages the cache.
KVAD_EXPORT int kvad_attention_scored_prompt(const void* q, int64_t ld_q, int n_rows, void* out, int64_t ld_out, const void* gate, int64_t ld_gate, int gate_heads,
                                         const float* sinks, const int* seq_starts, const int* kv_lens, const int* page_table, int table_width,
                                         const void* k_pages, const void* v_pages, int n_pages, int n_seqs, int n_heads, int n_kv_heads, int dk, int dv,
                                         int page_size, int max_new, float scale, float softcap, float slope_span, int window, int keep_first,
                                         int chunk, int key_maps, int out_f32, cudaStream_t stream) {
  KVAD_REQUIRE(n_seqs >= 0 && n_heads > 0 && n_kv_heads > 0 && dk > 0 && dv > 0 && table_width > 0 && max_new >= 0 && keep_first >= 0 && n_rows >= 0 && n_pages > 0,
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
  KVAD_REQUIRE((int64_t)n_pages * n_kv_heads * PAGE < (1ll << 31), "attention (scored, prompts): %d pages of %d heads are more than a coordinate counts", n_pages, n_kv_heads);
  if (n_seqs == 0 || max_new == 0 || n_rows == 0) return KVAD_OK;
  PromptArgs a;
  a.q = (const __nv_bfloat16*)q; a.ld_q = ld_q; a.k_pages = (const __nv_bfloat16*)k_pages; a.v_pages = (const __nv_bfloat16*)v_pages;
  a.out = out; a.ld_out = ld_out; a.gate = (const __nv_bfloat16*)gate; a.ld_gate = ld_gate;
  a.gate_heads = gate_heads; a.sinks = sinks; a.seq_starts = seq_starts; a.kv_lens = kv_lens; a.page_table = page_table; a.table_width = table_width;
  a.n_heads = n_heads; a.n_kv_heads = n_kv_heads; a.dk = dk; a.dv = dv; a.alias = alias ? 1 : 0; a.key_maps = key_maps;
  a.scale = scale; a.softcap = softcap; a.slope_span = slope_span; a.window = window > 0 ? window : 0; a.keep_first = window > 0 ? keep_first : 0;
  a.chunk = chunk > 0 ? chunk : 0;
  // (scale / cap stays an ordinary number: a cap above 2^100 moves no score below 2^87, one of nothing makes every score but 0 the cap)
  const float cap = std::min(softcap, 1.2676506e30f), ratio = scale / cap;
  a.cap_in = softcap > 0.f ? std::max(-3.402823466e38f, std::min(3.402823466e38f, ratio)) : 0.f; a.cap_out = cap * LOG2E;
  // heads a tile: as many of the group as divide it, up to 16 (a tile then spans few tokens: little of its last page is masked)
  a.hp = 1;
  while (a.hp < 16 && (n_heads / n_kv_heads) % (a.hp * 2) == 0) a.hp *= 2;
  KVAD_REQUIRE((int64_t)n_seqs * (n_heads / a.hp) < (1ll << 31), "attention (scored, prompts): %d sequences x %d heads are more than one launch takes", n_seqs, n_heads);
  a.columns = n_seqs * (n_heads / a.hp);
  a.skip_copy = g_skip_copy;
  g_skip_copy = 0;
  const int item = out_f32 ? 4 : 2;
  a.vec = (reinterpret_cast<uintptr_t>(out) & 15) == 0 && ld_out * item % 16 == 0 &&
          (gate == nullptr || gate_heads || ((reinterpret_cast<uintptr_t>(gate) & 15) == 0 && ld_gate % 8 == 0)) ? 1 : 0;
  const Layout z = layout_of(dk, dv, alias);
  a.stages = z.stages;
  CUtensorMap mq, mk, mv;
  const cuuint64_t q_dims[3] = {(cuuint64_t)dk, (cuuint64_t)n_heads, (cuuint64_t)n_rows}, q_strides[2] = {(cuuint64_t)dk * 2, (cuuint64_t)ld_q * 2};
  const cuuint32_t q_box[3] = {64, (cuuint32_t)a.hp, (cuuint32_t)(ROWS / a.hp)}, page_box[2] = {64, PAGE};
  const cuuint64_t k_dims[2] = {(cuuint64_t)dk, (cuuint64_t)n_pages * n_kv_heads * PAGE}, k_strides[1] = {(cuuint64_t)dk * 2};
  const cuuint64_t v_dims[2] = {(cuuint64_t)dv, (cuuint64_t)n_pages * (n_kv_heads / key_maps) * PAGE}, v_strides[1] = {(cuuint64_t)dv * 2};
  int rc = make_map(&mq, q, 3, q_dims, q_strides, q_box);
  if (rc == KVAD_OK) rc = make_map(&mk, k_pages, 2, k_dims, k_strides, page_box);
  if (rc != KVAD_OK) return rc;
  mv = mk;
  if (!alias && (rc = make_map(&mv, v_pages, 2, v_dims, v_strides, page_box)) != KVAD_OK) return rc;
#define KVAD_TC(NS, CPW)                                                                                                      \
  do {                                                                                                                        \
    if (z.in_turn && out_f32) return launch<NS, CPW, true, true>(mq, mk, mv, a, max_new, z.smem, stream);                     \
    if (z.in_turn) return launch<NS, CPW, false, true>(mq, mk, mv, a, max_new, z.smem, stream);                               \
    if (out_f32) return launch<NS, CPW, true, false>(mq, mk, mv, a, max_new, z.smem, stream);                                 \
    return launch<NS, CPW, false, false>(mq, mk, mv, a, max_new, z.smem, stream);                                             \
  } while (0)
  if (dv <= 64) KVAD_TC(2, 1);
  if (dv <= 128) KVAD_TC(2, 2);
  KVAD_TC(1, 2);
#undef KVAD_TC
}

// How many bounded waits have run out since the library was loaded (0 in a healthy run).  Synchronises the device.
KVAD_EXPORT int kvad_attention_scored_prompt_status() {
  int n = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&n, g_wait_timeouts, sizeof(int));
  if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "attention_scored_prompt_status: %s", cudaGetErrorString(e));
  return n;
}

// Tests of the bounded waits: `wait_limit` > 0 sets how many polls a wait makes before it gives up (0: the library's own limit); `skip_copy` leaves the first page out of
// the NEXT launch's blocks, so that the wait for it runs out.  Synchronises the device.
KVAD_EXPORT int kvad_attention_scored_prompt_test_hooks(unsigned wait_limit, int skip_copy) {
  g_skip_copy = skip_copy;
  return set_wait_limit(wait_limit);
}

KVAD_DEFINE_LAST_ERROR()
