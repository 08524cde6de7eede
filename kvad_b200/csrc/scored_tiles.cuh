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
  d |= (uint64_t)((PAGE_BLOCK >> 4) & 0x3FFFu) << 16;        // leading byte offset: between blocks of 64 columns (one at a time is used)
  d |= (uint64_t)(1024 >> 4) << 32;                          // stride byte offset: between groups of 8 keys
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;                                    // SWIZZLE_128B
  return d;
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
// 2^x by the special-function unit (2 units in the last place; a weight below 2^-126 of its row's largest is zero).
__device__ __forceinline__ float exp2_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / (1 + 2^(-z log2 e)) by the special-function unit (3 units in the last place, before a rounding to bfloat16).
__device__ __forceinline__ float sigmoid_fast(float z) { return __fdividef(1.0f, 1.0f + exp2_fast(-z * LOG2E)); }
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

// tanh(y) = y + y^3 P(y^2) up to |y| = 0.45 (P fitted to (tanh(y) / y - 1) / y^2 by reweighted least squares: off by 5e-9 of tanh).
constexpr float TANH_NEAR = 0.45f, TANH0 = -0.3333325f, TANH1 = 0.13329249f, TANH2 = -0.05334366f, TANH3 = 0.01802476f;

// A row's 64 scores of a page, in units of log2: capped or scaled, less the slope times the distance (`ahead`: the row's position less the page's first).
// (Whole passes under tests that are the same for every thread: this part is bound by instructions.)
__device__ __forceinline__ void shape_scores(float (&sc)[64], bool capped, float cap_in, float cap_out, float scale2, bool sloped, float slope, int ahead) {
  if (capped) {                             // cap tanh(s / cap): by `tanhf` where some score is far out, whose error follows its result too
    float most = 0.f;
#pragma unroll
    for (int c = 0; c < 64; ++c) most = fmaxf(most, fabsf(sc[c]));
    if (__any_sync(0xffffffffu, most * fabsf(cap_in) > TANH_NEAR)) {
#pragma unroll
      for (int c = 0; c < 64; ++c) sc[c] = cap_out * tanhf(sc[c] * cap_in);
    } else {
      const uint64_t in2 = pair(cap_in, cap_in), out2 = pair(cap_out, cap_out);
#pragma unroll
      for (int c = 0; c < 64; c += 2) {
        const uint64_t y = mul2(pair(sc[c], sc[c + 1]), in2), z = mul2(y, y);
        uint64_t p = fma2(z, pair(TANH3, TANH3), pair(TANH2, TANH2));
        p = fma2(z, p, pair(TANH1, TANH1));
        p = fma2(z, p, pair(TANH0, TANH0));
        unpair(mul2(out2, fma2(mul2(y, z), p, y)), sc[c], sc[c + 1]);
      }
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

}  // namespace kvad
