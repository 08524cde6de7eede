// What the prompt attention kernels with shaped scores share (`attention_scored_prompt.cu`: bfloat16, `attention_scored_wide.cu`: 32-bit): 128 rows against
// pages of 64 keys on tcgen05, a thread a row where scores become weights.
#pragma once
#include "tcgen05.cuh"

namespace kvad {

constexpr int PAGE = 64, ROWS = 128;
constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
constexpr uint32_t Q_BLOCK = ROWS * 128, PAGE_BLOCK = PAGE * 128;      // 64 entries (128 bytes of bfloat16, swizzled) of the queries, of a page

__device__ __forceinline__ void fence_async_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
template <int N> __device__ __forceinline__ void regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_fewer() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }

__device__ __forceinline__ void tmem_ld32(uint32_t addr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tmem_st8(uint32_t addr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// D += A B with A in tensor memory (a lane a row, two neighbours along K a column)
__device__ __forceinline__ void umma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
// Values as the second operand of P V: rows are keys (the product's K), 128 contiguous bytes are 64 of its columns.
__device__ __forceinline__ uint64_t sw128_mn_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)((PAGE_BLOCK >> 4) & 0x3FFFu) << 16;        // leading byte offset: between blocks of 64 columns (products of 128 step over two)
  d |= (uint64_t)(1024 >> 4) << 32;                          // stride byte offset: between groups of 8 keys
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;                                    // SWIZZLE_128B
  return d;
}

__device__ __forceinline__ void tmem_ld_issue(uint32_t addr, uint32_t (&r)[16]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                 "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(addr) : "memory");
}
__device__ __forceinline__ void tmem_ld_issue(uint32_t addr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(addr) : "memory");
}

// Two 32-bit numbers at once (an instruction for both).
__device__ __forceinline__ uint64_t pair(float a, float b) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpair(uint64_t r, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(r)); }
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
// What two places of N (8 or 16) columns hold, added up, two columns a number.
template <int N>
__device__ __forceinline__ void tmem_ld_sum(uint32_t at, uint32_t and_at, uint64_t (&v)[N / 2]) {
  uint32_t x[N], y[N];
  tmem_ld_issue(at, x);
  tmem_ld_issue(and_at, y);
  tmem_ld_wait();
#pragma unroll
  for (int i = 0; i < N / 2; ++i)
    v[i] = add2(pair(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1])), pair(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1])));
}
// 2^x by the special-function unit (2 units in the last place; a weight below 2^-126 of its row's largest is zero).
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 2^x of a whole number x <= 0 (exactly; 0 below -126).  Pages are brought to whole powers of two of one another, so that joining them rounds nothing but the sums: with each
// page's own largest score as its unit, factors of exp2_fast's errors went into every page's share (2000 keys, values of one sign: 1.4e-7 off, so 1.0e-7).
__device__ __forceinline__ float exp2_whole(float x) { return __int_as_float((int)(fmaxf(x, -127.f) + 127.f) << 23); }
// 1 / (1 + e^(-z)) from e = e^(-|z|), so that the denominator lies in (1, 2]: its reciprocal by the special-function unit and one step of Newton's method, without a branch.  (A fast
// division of 1 + e^(-z) gives 0 for gates below -87.3; a full one has a way for every number, which took 31 us to 39: 2 x 1024 rows of 16 gated heads of 64.)
__device__ __forceinline__ float sigmoid(float z) {
  const float e = expf(-fabsf(z)), d = 1.0f + e;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
  r = fmaf(r, fmaf(-d, r, 1.0f), r);
  return z >= 0.f ? r : e * r;
}
// The upper halves of two floats as a pair of bfloat16 (truncated), and what is left of each.
__device__ __forceinline__ uint32_t cut(float& a, float& b) {
  const uint32_t x = __float_as_uint(a), y = __float_as_uint(b);
  unpair(add2(pair(a, b), pair(-__uint_as_float(x & 0xffff0000u), -__uint_as_float(y & 0xffff0000u))), a, b);
  return __byte_perm(x, y, 0x7632);
}
__device__ __forceinline__ uint32_t pack(float a, float b) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&v);
}

// tanh(y) = y + y^3 P(y^2) up to |y| = 0.45 (P fitted to (tanh(y) / y - 1) / y^2 by reweighted least squares: off by 7.8e-9 of tanh with these coefficients).
constexpr float TANH_NEAR = 0.45f, TANH0 = -0.3333325f, TANH1 = 0.13329249f, TANH2 = -0.05334366f, TANH3 = 0.01802476f;

// A row's 64 scores of a page, in units of log2: capped or scaled, less the slope times the distance (`ahead`: the row's position less the page's first).
// (Whole passes under tests that are the same for every thread: this part is bound by instructions.)
__device__ __forceinline__ void shape_scores(float (&sc)[64], bool capped, float cap_in, float cap_out, float scale2, bool sloped, float slope, int ahead) {
  if (capped) {                             // cap tanh(s / cap): which formula a score takes is its own affair (by `tanhf`, whose error follows its result too, far out)
    const uint64_t in2 = pair(cap_in, cap_in), out2 = pair(cap_out, cap_out);
    auto near2 = [&](int c) {
      const uint64_t y = mul2(pair(sc[c], sc[c + 1]), in2), z = mul2(y, y);
      uint64_t p = fma2(z, pair(TANH3, TANH3), pair(TANH2, TANH2));
      p = fma2(z, p, pair(TANH1, TANH1));
      p = fma2(z, p, pair(TANH0, TANH0));
      return mul2(out2, fma2(mul2(y, z), p, y));
    };
    float most = 0.f;
#pragma unroll
    for (int c = 0; c < 64; ++c) most = fmaxf(most, fabsf(sc[c]));
    if (__any_sync(0xffffffffu, most * fabsf(cap_in) > TANH_NEAR)) {      // (the vote only saves work: whoever is not far out has the polynomial's result either way)
#pragma unroll
      for (int c = 0; c < 64; c += 2) {
        float n0, n1;
        unpair(near2(c), n0, n1);
        const float y0 = sc[c] * cap_in, y1 = sc[c + 1] * cap_in, f0 = cap_out * tanhf(y0), f1 = cap_out * tanhf(y1);
        asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %1, %2;\n\tselp.f32 %0, %3, %4, p;\n\t}" : "=f"(sc[c]) : "f"(fabsf(y0)), "f"(TANH_NEAR), "f"(f0), "f"(n0));      // (no branch an entry)
        asm("{\n\t.reg .pred p;\n\tsetp.gt.f32 p, %1, %2;\n\tselp.f32 %0, %3, %4, p;\n\t}" : "=f"(sc[c + 1]) : "f"(fabsf(y1)), "f"(TANH_NEAR), "f"(f1), "f"(n1));
      }
    } else {
#pragma unroll
      for (int c = 0; c < 64; c += 2) unpair(near2(c), sc[c], sc[c + 1]);
    }
  } else {
#pragma unroll
    for (int c = 0; c < 64; ++c) sc[c] *= scale2;
  }
  if (sloped) {
#pragma unroll
    for (int c = 0; c < 64; ++c) sc[c] -= slope * (float)(ahead - c);
  }
}
// Scores of keys the row does not see: it sees those up to `hi` and from `lo` on, and the first `kept` (all counted from the page's first key).
__device__ __forceinline__ void hide_scores(float (&sc)[64], int hi, int lo, int kept) {
  uint64_t see = hi < 0 ? 0ull : (hi >= 63 ? ~0ull : (2ull << hi) - 1ull);
  const uint64_t below = lo <= 0 ? 0ull : (lo >= 64 ? ~0ull : (1ull << lo) - 1ull);
  const uint64_t held = kept <= 0 ? 0ull : (kept >= 64 ? ~0ull : (1ull << kept) - 1ull);
  see &= ~below | held;
  const uint32_t see0 = (uint32_t)see, see1 = (uint32_t)(see >> 32);
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    if (!(see0 >> c & 1)) sc[c] = -INFINITY;
    if (!(see1 >> c & 1)) sc[32 + c] = -INFINITY;
  }
}

// A row worked out once more by a whole warp, key by key, from what it sees alone.  In the products a key that a row does not see has weight 0, and 0 times a
// value that is not a finite number is none: where such a number is in a tile's pages, rows that do not see it lose the entries it meets.  So every entry that came
// out as no finite number is worked out here again (a lane a key for the scores, a lane a column for the output), and is one only if the row sees the cause.
// A block's rows are noted (`note_again`) and shared out over its warps at its end.  Nothing of it runs otherwise.  (2 x 1024 rows of 16 heads of 64 on 4 key heads, ms:
// all keys NaN, 0.25 where finite ones take 0.024 in bfloat16, 0.60 for 0.048 in 32 bits; one NaN value 0.12 and 3.2; a thread a row, all rows of a tile: 24 in 32 bits.)
template <typename T> struct RowAgain {
  const T* q;                                     // the row's query
  const T* k; const T* v;                         // the head's keys and values in page 0
  const int* pages;
  int64_t k_step, v_step;                         // from page to page
  int dk, dv, ld_v, pos, first, kept;
  float scale2, cap_in, cap_out, slope;
  int capped;
  const float* sink;                              // or null
  const T* gate; int gate_step;                   // or null; gate_step 0: one number for all entries
};
__device__ __forceinline__ void load8(const float* p, float (&x)[8]) {
  const float4 a = reinterpret_cast<const float4*>(p)[0], b = reinterpret_cast<const float4*>(p)[1];
  x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w; x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
}
__device__ __forceinline__ void load8(const __nv_bfloat16* p, float (&x)[8]) {
  const uint4 raw = *reinterpret_cast<const uint4*>(p);
  const uint32_t w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    x[2 * i] = __uint_as_float(w[i] << 16);
    x[2 * i + 1] = __uint_as_float(w[i] & 0xffff0000u);
  }
}
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }
// `out`: the row's entries of this head, of which those that are not finite are written again.
// NI: 32s of entries.  An entry that has become NaN stays so: the row is left as it is as soon as all that are worked out again have.
template <int NI, typename T, typename TO>
__device__ __forceinline__ void row_again(const RowAgain<T>& z, TO* out) {
  const int lane = threadIdx.x & 31;
  float o[NI], most = -INFINITY, sum = 0.f;
  uint32_t need = 0;
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    o[i] = 0.f;
    if (lane + 32 * i < z.dv && not_finite(to_f32(out[lane + 32 * i]))) need |= 1u << i;
  }
  for (int j0 = 0; j0 <= z.pos; j0 += 32) {       // (half a page)
    if (j0 + 32 <= z.first && j0 >= z.kept) continue;
    const int64_t page = z.pages[j0 / PAGE];
    const int j = j0 + lane, place = j % PAGE;
    const bool seen = j <= z.pos && (j >= z.first || j < z.kept);
    float s = 0.f;
    if (seen) {
      const T* k = z.k + page * z.k_step + (int64_t)place * z.dk;
#pragma unroll 2
      for (int d = 0; d < z.dk; d += 8) {
        float a[8], b[8];
        load8(z.q + d, a);
        load8(k + d, b);
#pragma unroll
        for (int e = 0; e < 8; ++e) s = fmaf(a[e], b[e], s);
      }
      s = z.capped ? z.cap_out * tanhf(s * z.cap_in) : s * z.scale2;
      s -= z.slope * (float)(z.pos - j);
    }
    const float top = fmaxf(most, warp_max(seen ? s : -INFINITY)), base = top == -INFINITY ? 0.f : top, keep = most == -INFINITY ? 0.f : exp2f(most - base);
    const float p = seen ? exp2f(s - base) : 0.f;
    most = top;
    sum = fmaf(sum, keep, warp_sum(p));
#pragma unroll
    for (int i = 0; i < NI; ++i) o[i] *= keep;
    const uint32_t live = __ballot_sync(0xffffffffu, seen);
    const T* v = z.v + page * z.v_step + (int64_t)(j0 % PAGE) * z.ld_v + lane;
#pragma unroll 4
    for (int at = 0; at < 32; ++at, v += z.ld_v) {
      const float w = __shfl_sync(0xffffffffu, p, at);
      if (!(live >> at & 1)) continue;
#pragma unroll
      for (int i = 0; i < NI; ++i)
        if (need >> i & 1) o[i] = fmaf(w, to_f32(v[32 * i]), o[i]);
    }
    bool settled = true;
#pragma unroll
    for (int i = 0; i < NI; ++i) settled = settled && (!(need >> i & 1) || o[i] != o[i]);
    if (__all_sync(0xffffffffu, settled)) return;
  }
  float inv = 1.f / sum;
  if (z.sink != nullptr) {
    const float sink = *z.sink * LOG2E, m = fmaxf(most, sink), f = exp2f(most - m);
    inv = f / fmaf(sum, f, exp2f(sink - m));
  }
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    const int d = lane + 32 * i;
    if (!(need >> i & 1)) continue;
    float y = o[i] * inv;
    if (z.gate != nullptr) y *= 1.f / (1.f + expf(-to_f32(z.gate[(int64_t)d * z.gate_step])));
    out[d] = from_f32<TO>(y);
  }
}

// The 32 rows of a warp: which have an entry that is not finite.  `again`: a bit a row.
__device__ __forceinline__ void note_again(uint32_t* again, int quarter, bool bad) {
  const uint32_t rows = __ballot_sync(0xffffffffu, bad);
  if (rows != 0 && (threadIdx.x & 31) == 0) atomicOr(again + quarter, rows);
}
// The noted rows of a block, by `warps` of its warps from `first` on, which all call it at the end of their roles (where they still have the registers that they took).
// Args: the kernels' arguments (in constant memory).  It finds the block's place again: nothing of it is kept in the kernels' registers.
template <int NI, typename T, typename TO, typename Args>
__device__ __noinline__ void rows_again(const Args& a, const uint32_t* again, int first, int warps) {
  const int hp = a.hp, tok = ROWS / hp, group = a.n_heads / a.n_kv_heads, chunks = group / hp, per_seq = a.n_kv_heads * chunks;
  const int from_end = blockIdx.x / a.columns, column = blockIdx.x - from_end * a.columns, s = column / per_seq, part = column - s * per_seq, kvh = part / chunks;
  const int h0 = kvh * group + (part - kvh * chunks) * hp, start = a.seq_starts[s], n_new = a.seq_starts[s + 1] - start;
  const int tok0 = ((int)gridDim.x / a.columns - 1 - from_end) * tok, pos0 = a.kv_lens[s] - n_new + tok0, n_tok = min(tok, n_new - tok0);
  for (int r = (threadIdx.x >> 5) - first; r < ROWS; r += warps) {
    const int ti = r / hp, h = h0 + r - ti * hp;
    if (!(again[r >> 5] >> (r & 31) & 1) || ti >= n_tok) continue;
    const int64_t at = start + tok0 + ti;
    RowAgain<T> z;
    z.q = a.q + at * a.ld_q + (int64_t)h * a.dk;
    z.k = a.k_pages + (int64_t)kvh * PAGE * a.dk;
    z.v = a.alias ? z.k : a.v_pages + (int64_t)(kvh / a.key_maps) * PAGE * a.dv;
    z.pages = a.page_table + (int64_t)s * a.table_width;
    z.k_step = (int64_t)a.n_kv_heads * PAGE * a.dk;
    z.v_step = a.alias ? z.k_step : (int64_t)(a.n_kv_heads / a.key_maps) * PAGE * a.dv;
    z.dk = a.dk; z.dv = a.dv; z.ld_v = a.alias ? a.dk : a.dv;
    z.pos = pos0 + ti;
    z.first = a.window > 0 ? z.pos - a.window + 1 : (a.chunk > 0 ? z.pos - z.pos % a.chunk : 0);
    z.kept = a.keep_first;
    z.scale2 = a.scale * LOG2E; z.cap_in = a.cap_in; z.cap_out = a.cap_out; z.capped = a.softcap > 0.f;
    z.slope = a.slope_span > 0.f ? exp2f(-a.slope_span * (float)(h + 1) / (float)a.n_heads) * LOG2E : 0.f;
    z.sink = a.sinks == nullptr ? nullptr : a.sinks + h;
    z.gate = a.gate == nullptr ? nullptr : (a.gate_heads ? a.gate + at * a.ld_gate + h : a.gate + at * a.ld_gate + (int64_t)h * a.dv);
    z.gate_step = a.gate_heads ? 0 : 1;
    row_again<NI>(z, reinterpret_cast<TO*>(a.out) + at * a.ld_out + (int64_t)h * a.dv);
  }
}

}  // namespace kvad
