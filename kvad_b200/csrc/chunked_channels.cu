// Recurrences of prompts whose state decays by one number per KEY CHANNEL and row, 64 rows at a time: the gated delta rule and the gated
// linear kind of `gated_recurrence.cu`,
//
//   S_t = diag(g_t) S_(t-1) + k_t u_t^T,   o_t = S_t^T q_t,   u_t = v_t   or   u_t = beta_t (v_t - (diag(g_t) S_(t-1))^T k_t)  (delta rule).
//
// Walking the rows is a chain of ~0.4 us a row.  Within a chunk of 64 rows, with P(j -> i) the channels' decay from row j to row i and
// B_i the one from the chunk's start:
//
//   o_i = sum_(j <= i) A_ij u_j + (q_i B_i)^T S,          A_ij = sum_d q_i k_j P(j -> i)
//   delta rule: u_i + beta_i sum_(j < i) M_ij u_j = beta_i v_i - beta_i (k_i B_i)^T S,   M_ij = sum_d k_i k_j P(j -> i),
//   so u = X - W S with (I + beta M) [X | W] = beta [v | k B]
//   S' = diag(B_63) S + sum_j (k_j P(j -> 63)) u_j^T
//
// Decays appear only as PRODUCTS of the g's over the rows between, never as quotients of two products, so a channel that forgets at
// once (g = 0) or never (g = 1) is nothing special: 16 rows form a block; pairs of rows of different blocks take the decay up to the later
// block's first row from the earlier row (a product over the rest of its block, times whole blocks between) and from there on from the
// later row; pairs within a block take the product row by row.
//
// Two kernels.  `prepare`, a block per (chunk, head): A, the decayed keys and queries, and for the delta rule X and W by forward
// substitution, a column a thread, all of it in registers.  `walk`, a block per (sequence, head, 16 value columns): from chunk to chunk,
// four products a chunk.  All 32-bit on the CUDA cores; sums of 16 terms added up and decays whose products carry what they lose keep the
// error beside the walk's: over 1024 rows of 128 x 128 the delta rule's outputs are off by 1.21e-7 (row by row 1.17e-7, with longer chains and
// plain products 1.43e-7) and its states by 8.9e-8 (8.9e-8, 9.9e-8), the gated linear kind's by 1.30e-7 (1.27e-7, 1.71e-7) and 9.0e-8 (1.00e-7, 1.26e-7).
//
// Measured, delta rule, 2 x 1024 rows of 8 heads of 128 x 128: 434 -> 155 us (the walk 92 of them: 16 chunks one after another).
#include "common.cuh"

using namespace kvad;

namespace {

constexpr int C = 64, B = 16, THREADS = 256, LDT = C + 4, COLS = 16, LDC = COLS + 4;

struct ChannelArgs {
  const void* q; const void* k; const void* v;
  int64_t ld_q, ld_k, ld_v;
  const float* gates; int64_t ld_gates;        // [rows, heads * dk]: the decays
  const float* beta; int64_t ld_beta;          // [rows, heads], or null: the gated linear kind
  const int* seq_starts; const int* seq_slots;
  int n_seqs, heads, group, dk, dv;
  int from;                 // only sequences of so many new rows or more (the others: gated_recurrence.cu)
  int place0, places;       // the span of the list of chunks that the scratch holds: its first place, how many (see chunked_recurrence.cu)
  float q_scale;
  float* wq;          // [places, heads, DK, 128]: columns 0..63 W (delta rule), 64..127 q B, transposed
  float* kt;          // [places, heads, 64, DK]: keys decayed to the chunk's end
  float* x;           // [places, heads, 64, dv]: X (the delta rule), or unused
  float* at;          // [places, heads, 64, 64]: A transposed
  float* whole;       // [places, heads, DK]: decay over the chunk
  float* out; int64_t ld_out;
  float* state; int64_t state_stride;          // [slots][heads][dv][dk]
};

struct Place { int s, row0, n; };
__device__ __forceinline__ Place find(const ChannelArgs& a, int place) {
  int lo = 0, hi = a.n_seqs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) / 2;
    if (a.seq_starts[mid] / C + mid <= place) lo = mid;
    else hi = mid - 1;
  }
  Place p;
  const int start = a.seq_starts[lo], n_new = a.seq_starts[lo + 1] - start, first = (place - (start / C + lo)) * C;
  p.s = lo;
  p.row0 = start + first;
  p.n = n_new < a.from ? 0 : max(0, min(C, n_new - first));
  return p;
}

__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
// A chunk's rows of one head, transposed [entry][row]; what does not exist is `fill`.  `width_to` is a multiple of 16: a warp takes 8 rows by 4
// neighbouring quads, whole sectors of memory, and its stores meet a bank twice.
template <typename TI>
__device__ __forceinline__ void bring(float* dst, const TI* src, int64_t ld, const Place& p, int width, int width_to, float scale, float fill) {
#pragma unroll 4
  for (int i = threadIdx.x; i < C * width_to / 4; i += THREADS) {
    const int r = (i & 7) + (i >> 5) % (C / 8) * 8, d = (((i >> 3) & 3) + (i >> 5) / (C / 8) * 4) * 4;
    float4 x = make_float4(fill, fill, fill, fill);
    if (r < p.n && d < width) {
      x = load4(src + (int64_t)(p.row0 + r) * ld + d);
      x.x *= scale; x.y *= scale; x.z *= scale; x.w *= scale;
    }
    dst[d * LDT + r] = x.x;
    dst[(d + 1) * LDT + r] = x.y;
    dst[(d + 2) * LDT + r] = x.z;
    dst[(d + 3) * LDT + r] = x.w;
  }
}
// 16 rows of one channel, in quads.
__device__ __forceinline__ void get16(float (&v)[B], const float* src) {
#pragma unroll
  for (int i = 0; i < B; i += 4) *reinterpret_cast<float4*>(v + i) = *reinterpret_cast<const float4*>(src + i);
}
__device__ __forceinline__ void put16(float* dst, const float (&v)[B]) {
#pragma unroll
  for (int i = 0; i < B; i += 4) *reinterpret_cast<float4*>(dst + i) = *reinterpret_cast<const float4*>(v + i);
}

// ---- prepare -----------------------------------------------------------------------------------------------------------------
// The channels come 64 at a time, so that two blocks fit an SM.
constexpr int HD = 64;

// A product of decays that carries what its roundings lose (up to 64 of them in a row otherwise, which every state and output would inherit).
struct Decay {
  float w = 1.f, lost = 0.f;
  __device__ __forceinline__ void by(float g) {
    const float p = w * g;
    lost = fmaf(lost, g, fmaf(w, g, -p));
    w = p;
  }
  __device__ __forceinline__ float value() const { return w + lost; }
};

template <typename TI, int DK, bool DELTA>
__global__ void __launch_bounds__(THREADS, 2) channel_prepare_kernel(const ChannelArgs a) {
  extern __shared__ float smem[];
  float* qt = smem;                    // [HD][LDT] q, then q times the decay from its block's first row on
  float* kt = qt + HD * LDT;           // k likewise
  float* gt = kt + HD * LDT;           // decays
  float* kh = gt + HD * LDT;           // keys times the decay over the rest of their block
  float* As = kh + HD * LDT;           // [64 (j)][LDT (i)]
  float* Ms = As + C * LDT;            // [64 (i)][LDT (j)] (delta rule)
  float* block_g = Ms + C * LDT;       // [4][HD]: decay over a block
  __shared__ float sbeta[C];
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.y, qh = h / a.group, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const Place p = find(a, a.place0 + blockIdx.x);
  if (p.n == 0) return;
  const int64_t at = (int64_t)blockIdx.x * a.heads + h;
  for (int i = tid; i < 2 * C * LDT; i += THREADS) As[i] = 0.f;
  if (tid < C) sbeta[tid] = DELTA && tid < p.n ? a.beta[(int64_t)(p.row0 + tid) * a.ld_beta + h] : 0.f;

#pragma unroll 1
  for (int h0 = 0; h0 < DK; h0 += HD) {
    __syncthreads();                   // the half before has been used up
    bring<TI>(qt, (const TI*)a.q + qh * a.dk + h0, a.ld_q, p, a.dk - h0, HD, a.q_scale, 0.f);
    bring<TI>(kt, (const TI*)a.k + qh * a.dk + h0, a.ld_k, p, a.dk - h0, HD, 1.f, 0.f);
    bring<float>(gt, a.gates + h * a.dk + h0, a.ld_gates, p, a.dk - h0, HD, 1.f, 1.f);
    __syncthreads();
    // pairs of rows within a block: a lane owns row j and a quarter of the channels (two warps a block), its key decaying as i goes on
    {
      const int blk = warp >> 1, j = lane & 15, quarter = (warp & 1) * 2 + (lane >> 4), d0 = quarter * (HD / 4), i0 = blk * B;
      float sq[B], sk[B];
#pragma unroll
      for (int i = 0; i < B; ++i) sq[i] = sk[i] = 0.f;
#pragma unroll 1
      for (int d = d0; d < d0 + HD / 4; ++d) {
        float qv[B], kv[B], gv[B];
        get16(qv, qt + d * LDT + i0);
        get16(gv, gt + d * LDT + i0);
        if (DELTA) get16(kv, kt + d * LDT + i0);
        const float own = kt[d * LDT + i0 + j];
        float w = 0.f, lost = 0.f;                 // (the key's entry as it decays, and what the roundings of that lose)
#pragma unroll
        for (int i = 0; i < B; ++i) {
          const float next = w * gv[i];
          lost = i == j ? 0.f : fmaf(lost, gv[i], fmaf(w, gv[i], -next));
          w = i == j ? own : next;                 // (before row j: zero)
          const float key = w + lost;
          sq[i] = fmaf(qv[i], key, sq[i]);
          if (DELTA) sk[i] = fmaf(kv[i], key, sk[i]);
        }
      }
      // the quarters meet: neighbouring half-warps by shuffles, the two warps in shared memory
#pragma unroll
      for (int i = 0; i < B; ++i) {
        sq[i] += __shfl_xor_sync(0xffffffffu, sq[i], 16);
        if (DELTA) sk[i] += __shfl_xor_sync(0xffffffffu, sk[i], 16);
      }
#pragma unroll
      for (int turn = 0; turn < 2; ++turn) {
        if ((warp & 1) == turn && lane < 16) {
#pragma unroll
          for (int i = 0; i < B; ++i)
            if (i >= j) {
              As[(i0 + j) * LDT + i0 + i] += sq[i];
              if (DELTA && i > j) Ms[(i0 + i) * LDT + i0 + j] += sk[i];
            }
        }
        __syncthreads();
      }
    }
    // decays along a block, a (channel, block) a thread
    {
      const int d = tid % HD, blk = tid / HD, at_d = d * LDT + blk * B;
      float g[B], k[B], x[B];
      Decay after, before;
      get16(g, gt + at_d);
      get16(k, kt + at_d);
#pragma unroll
      for (int r = B - 1; r >= 0; --r) {
        x[r] = k[r] * after.value();
        after.by(g[r]);
      }
      put16(kh + at_d, x);
      block_g[blk * HD + d] = after.value();
      get16(x, qt + at_d);
#pragma unroll
      for (int r = 0; r < B; ++r) {
        before.by(g[r]);
        x[r] *= before.value();
        k[r] *= before.value();
      }
      put16(qt + at_d, x);
      if (DELTA) put16(kt + at_d, k);
    }
    __syncthreads();
    // pairs of rows of different blocks: a warp a pair of blocks, its half-warps for q and k, 4 x 4 a lane
    if (warp < 6) {
      const int late = warp == 0 ? 1 : (warp <= 2 ? 2 : 3), early = warp == 0 ? 0 : (warp <= 2 ? warp - 1 : warp - 3);
      const float* rows = lane < 16 ? qt : kt;
      const int i0 = late * B + (lane & 3) * 4, j0 = early * B + ((lane >> 2) & 3) * 4;
      if (DELTA || lane < 16) {
        float s[4][4] = {};
#pragma unroll 1
        for (int d0 = 0; d0 < HD; d0 += 16) {      // (sums of 16 terms, added up)
          float part[4][4] = {};
#pragma unroll 4
          for (int d = d0; d < d0 + 16; ++d) {
            float x[4], y[4], w = 1.f;
            *reinterpret_cast<float4*>(x) = *reinterpret_cast<const float4*>(rows + d * LDT + i0);
            *reinterpret_cast<float4*>(y) = *reinterpret_cast<const float4*>(kh + d * LDT + j0);
            if (late - early > 1) w = block_g[(early + 1) * HD + d];
            if (late - early > 2) w *= block_g[(early + 2) * HD + d];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const float xi = x[i] * w;
#pragma unroll
              for (int j = 0; j < 4; ++j) part[i][j] = fmaf(xi, y[j], part[i][j]);
            }
          }
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] += part[i][j];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (lane < 16) As[(j0 + j) * LDT + i0 + i] += s[i][j];
            else Ms[(i0 + i) * LDT + j0 + j] += s[i][j];
          }
      }
    }
    // the keys decayed to the chunk's end, the queries decayed from its start, the decay over the chunk
    {
      const int d = tid % HD, blk = tid / HD;
      float after = 1.f, x[B];
      for (int m = blk + 1; m < 4; ++m) after *= block_g[m * HD + d];
      get16(x, kh + d * LDT + blk * B);
#pragma unroll
      for (int r = 0; r < B; ++r) a.kt[(at * C + blk * B + r) * DK + h0 + d] = x[r] * after;
      if (blk == 0) a.whole[at * DK + h0 + d] = block_g[d] * after;
    }
    for (int i = tid; i < HD * C / 4; i += THREADS) {
      const int d = i / (C / 4), c = i % (C / 4) * 4;
      float before = 1.f;
      for (int m = 0; m < c / B; ++m) before *= block_g[m * HD + d];
      float4 x = *reinterpret_cast<const float4*>(qt + d * LDT + c);
      x.x *= before; x.y *= before; x.z *= before; x.w *= before;
      *reinterpret_cast<float4*>(a.wq + (at * DK + h0 + d) * 128 + 64 + c) = x;
    }
  }
  __syncthreads();
  for (int i = tid; i < C * C / 4; i += THREADS) {
    const int j = i / (C / 4), c = i % (C / 4) * 4;
    *reinterpret_cast<float4*>(a.at + at * C * C + j * C + c) = *reinterpret_cast<const float4*>(As + j * LDT + c);
  }
  if (DELTA) {
    // (I + beta M) [X | W] = beta [v | k B]: a column a thread
    const TI* v = (const TI*)a.v + h * a.dv;
    const TI* k = (const TI*)a.k + qh * a.dk;
    const float* g = a.gates + h * a.dk;
#pragma unroll 1
    for (int col = tid; col < DK + a.dv; col += THREADS) {
      const bool is_w = col < DK;
      float x[C];
      // (every load is of a row and a column that exist, so that none waits for a test)
      const bool there = !is_w || col < a.dk;
      const int own = there ? col : 0;
      const TI* src = is_w ? k + (int64_t)p.row0 * a.ld_k + own : v + (int64_t)p.row0 * a.ld_v + col - DK;
      const int64_t step = is_w ? a.ld_k : a.ld_v;
#pragma unroll
      for (int i = 0; i < C; ++i) {
        const float y = to_f32(*src);
        x[i] = there && i < p.n ? y : 0.f;
        src += i + 1 < p.n ? step : 0;
      }
      if (is_w) {
        const float* decay = g + (int64_t)p.row0 * a.ld_gates + own;
        Decay before;
#pragma unroll
        for (int i0 = 0; i0 < C; i0 += B) {
          float y[B];
#pragma unroll
          for (int i = 0; i < B; ++i) {
            y[i] = *decay;
            decay += i0 + i + 1 < p.n ? a.ld_gates : 0;
          }
#pragma unroll
          for (int i = 0; i < B; ++i) {
            before.by(y[i]);
            x[i0 + i] *= before.value();
          }
        }
      }
#pragma unroll
      for (int i = 0; i < C; ++i) {
        asm volatile("" ::: "memory");                          // (a row of M at a time: the registers are full of the column)
        float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
#pragma unroll
        for (int j = 0; j < (i + 3) / 4 * 4; j += 4) {          // (entries of M from the diagonal on are zeros)
          const float4 m = *reinterpret_cast<const float4*>(Ms + i * LDT + j);
          s0 = fmaf(m.x, x[j], s0);
          if (j + 1 < i) s1 = fmaf(m.y, x[j + 1], s1);
          if (j + 2 < i) s2 = fmaf(m.z, x[j + 2], s2);
          if (j + 3 < i) s3 = fmaf(m.w, x[j + 3], s3);
        }
        x[i] = sbeta[i] * (x[i] - ((s0 + s1) + (s2 + s3)));
      }
      if (is_w) {
#pragma unroll
        for (int i = 0; i < C; i += 4) *reinterpret_cast<float4*>(a.wq + (at * DK + col) * 128 + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
      } else {
        float* dst = a.x + at * C * a.dv + col - DK;
#pragma unroll
        for (int i = 0; i < C; ++i) {
          *dst = x[i];
          dst += a.dv;
        }
      }
    }
  }
}

// ---- walk --------------------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void copy16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// The walk's tiles of 16 columns ([rows][COLS]) keep row r at place (r % 4) * (rows / 4) + r / 4, places LDC apart: 4 x 4 tiles of eight
// neighbouring lanes then go to and come from different banks (with the rows in order they all meet in the same four).
template <int ROWS>
__device__ __forceinline__ int place_of(int r) { return ((r & 3) * (ROWS / 4) + (r >> 2)) * LDC; }
// acc[4][4] += sum over n of X[n][0 .. 3] Y[row n][0 .. 3]; Y points at the place of a row that is a multiple of 4, n is a multiple of 16.
// Sums of 16 terms, added up: less rounding than one chain (of 8: less again by 2 %, for 6 us of 148).
template <int ROWS>
__device__ __forceinline__ void product(float (&acc)[4][4], const float* X, int ldx, const float* Y, int n) {
#pragma unroll 1
  for (int t0 = 0; t0 < n / 4; t0 += 4) {
    float part[4][4] = {};
#pragma unroll
    for (int t4 = t0; t4 < t0 + 4; ++t4) {
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float4 x = *reinterpret_cast<const float4*>(X + (t4 * 4 + e) * ldx), y = *reinterpret_cast<const float4*>(Y + (e * (ROWS / 4) + t4) * LDC);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) part[i][j] = fmaf(xs[i], ys[j], part[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j];
  }
}
// Rows 4 q .. + 3 of a tile.
template <int ROWS>
__device__ __forceinline__ void put_tile(float* dst, int q, const float (&v)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) *reinterpret_cast<float4*>(dst + (i * (ROWS / 4) + q) * LDC) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
}
template <int ROWS>
__device__ __forceinline__ void add_tile(const float* src, int q, float (&v)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float4 o = *reinterpret_cast<const float4*>(src + (i * (ROWS / 4) + q) * LDC);
    v[i][0] += o.x; v[i][1] += o.y; v[i][2] += o.z; v[i][3] += o.w;
  }
}

template <typename TI, int DK, bool DELTA>
__global__ void __launch_bounds__(THREADS, 1) channel_walk_kernel(const ChannelArgs a) {
  constexpr int WROWS = DELTA ? 128 : 64;             // W and q B, or q B alone
  extern __shared__ float smem[];
  float* wq = smem;                                   // [DK][WROWS]
  float* kt = wq + DK * WROWS;                        // [64][DK]
  float* at = kt + C * DK;                            // [64][64]
  float* S = at + C * C;                              // [DK][COLS]
  float* D = S + DK * LDC;                            // [64][COLS]: u
  float* part = D + C * LDC;                          // partial sums: 3 x [64][COLS], or [128][COLS]
  float* part2 = part + 3 * C * LDC;                  // [DK][COLS]
  pdl_launch_dependents();
  pdl_wait();
  const int s = blockIdx.x / a.heads, h = blockIdx.x - s * a.heads, c0 = blockIdx.y * COLS, tid = threadIdx.x;
  const int start = a.seq_starts[s], n_new = a.seq_starts[s + 1] - start;
  if (n_new <= 0 || n_new < a.from) return;
  // the chunks that lie in the span, and where chunk 0 would lie in its scratch
  const int n_chunks = (n_new + C - 1) / C, first = start / C + s - a.place0, c_begin = max(0, -first), c_end = min(n_chunks, a.places - first);
  if (c_begin >= c_end) return;
  float* st = a.state + (int64_t)a.seq_slots[s] * a.state_stride + (int64_t)h * a.dv * a.dk;
  for (int i = tid; i < DK * COLS; i += THREADS) {
    const int c = i / DK, d = i - c * DK;
    S[place_of<DK>(d) + c] = d < a.dk && c0 + c < a.dv ? st[(int64_t)(c0 + c) * a.dk + d] : 0.f;
  }
  auto bring_wq = [&](int c) {
    const float* src = a.wq + ((int64_t)(first + c) * a.heads + h) * DK * 128 + (128 - WROWS);
    for (int i = tid; i < DK * WROWS / 4; i += THREADS) {
      const int d = i / (WROWS / 4), r = i % (WROWS / 4) * 4;
      copy16(wq + d * WROWS + r, src + (int64_t)d * 128 + r);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto bring_rest = [&](int c) {
    const int64_t place = (int64_t)(first + c) * a.heads + h;
    for (int i = tid; i < C * DK / 4; i += THREADS) copy16(kt + i * 4, a.kt + place * C * DK + i * 4);
    for (int i = tid; i < C * C / 4; i += THREADS) copy16(at + i * 4, a.at + place * C * C + i * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  // A thread has 4 rows x 4 columns of a product and a share of its sum.  A warp's lanes are 32 quads of rows against ONE quad of columns, so that
  // its second operand is a broadcast.
  const int group = tid >> 7;                         // halves of a sum
  const int r4 = tid & 31, c4 = ((tid >> 5) & 3) * 4;
  const int q4 = tid & 15, quarter = (tid >> 4 & 1) + 2 * group;      // 64 rows: quarters of a sum
  bring_wq(c_begin);
  for (int c = c_begin; c < c_end; ++c) {
    const int64_t place = (int64_t)(first + c) * a.heads + h;
    const int n = min(C, n_new - c * C), row0 = start + c * C;
    bring_rest(c);                                    // on its way under the first product
    // what the first product is taken from, and the decay, into registers meanwhile
    const int ur = tid >> 2, uc = (tid & 3) * 4;      // row, four columns
    float given[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      given[e] = 0.f;
      if (ur < n && c0 + uc + e < a.dv)
        given[e] = DELTA ? a.x[(place * C + ur) * a.dv + c0 + uc + e] : to_f32(((const TI*)a.v)[(int64_t)(row0 + ur) * a.ld_v + h * a.dv + c0 + uc + e]);
    }
    float keep[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) keep[i] = r4 * 4 + i < DK ? a.whole[place * DK + r4 * 4 + i] : 0.f;
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    // [W | q B]^T S: rows r4 of both, a half of the channels a group (without W: 64 rows, a quarter of the channels)
    float acc[4][4] = {};
    if (DELTA) {
      product<DK>(acc, wq + group * (DK / 2) * WROWS + r4 * 4, WROWS, S + place_of<DK>(group * (DK / 2)) + c4, DK / 2);
      if (group == 1) put_tile<128>(part + c4, r4, acc);
      __syncthreads();
      if (group == 0) {
        add_tile<128>(part + c4, r4, acc);
        if (r4 < 16) put_tile<C>(D + c4, r4, acc);
      }
      __syncthreads();
      const float4 w = *reinterpret_cast<const float4*>(D + place_of<C>(ur) + uc);      // u = X - W S
      given[0] -= w.x; given[1] -= w.y; given[2] -= w.z; given[3] -= w.w;
      *reinterpret_cast<float4*>(D + place_of<C>(ur) + uc) = make_float4(given[0], given[1], given[2], given[3]);
    } else {
      *reinterpret_cast<float4*>(D + place_of<C>(ur) + uc) = make_float4(given[0], given[1], given[2], given[3]);
      product<DK>(acc, wq + quarter * (DK / 4) * WROWS + q4 * 4, WROWS, S + place_of<DK>(quarter * (DK / 4)) + c4, DK / 4);
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // u lies, keys and A are there, W and q B have been used up
    const bool odd = __syncthreads_or(given[0] * 0.f + given[1] * 0.f + given[2] * 0.f + given[3] * 0.f != 0.f);
    if (c + 1 < c_end) bring_wq(c + 1);
    // the state: S' = B S + K^T u, a half of the rows a group
    float add[4][4] = {};
    if (r4 * 4 < DK) product<C>(add, kt + group * 32 * DK + r4 * 4, DK, D + place_of<C>(group * 32) + c4, 32);
    if (group == 1 && r4 * 4 < DK) put_tile<DK>(part2 + c4, r4, add);
    // the read-outs: A u, a quarter of the rows j a thread, plus (q B)^T S
    float read[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) read[i][j] = DELTA ? 0.f : acc[i][j];
    if (!odd) {
      product<C>(read, at + quarter * B * C + q4 * 4, C, D + place_of<C>(quarter * B) + c4, B);
    } else {                                          // a row u is not finite: A's zeros would make NaN of it, so only the rows that a row sees
      float sum[4][4] = {};                           // (in the same order, for the same bits)
#pragma unroll 1
      for (int j = quarter * B; j < min(quarter * B + B, q4 * 4 + 4); ++j) {
        const float4 x = *reinterpret_cast<const float4*>(at + j * C + q4 * 4), y = *reinterpret_cast<const float4*>(D + place_of<C>(j) + c4);
        const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (j <= q4 * 4 + i) {
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[i][e] = fmaf(xs[i], ys[e], sum[i][e]);
          }
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) read[i][e] += sum[i][e];
    }
    // (delta rule: the threads of group 0 with rows from 64 on hold (q B)^T S: they are the second quarter, for the same rows and columns)
    if (DELTA && quarter == 1) {
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) read[i][j] += acc[i][j];
    }
    if (quarter > 0) put_tile<C>(part + (quarter - 1) * C * LDC + c4, q4, read);
    __syncthreads();
    if (quarter == 0) {
#pragma unroll
      for (int m = 0; m < 3; ++m) add_tile<C>(part + m * C * LDC + c4, q4, read);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int r = q4 * 4 + i;
        if (r < n) {
          float* o = a.out + (int64_t)(row0 + r) * a.ld_out + h * a.dv + c0 + c4;
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (c0 + c4 + e < a.dv) o[e] = read[i][e];
        }
      }
    }
    if (group == 0 && r4 * 4 < DK) {
      add_tile<DK>(part2 + c4, r4, add);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float4* at_s = reinterpret_cast<float4*>(S + (i * (DK / 4) + r4) * LDC + c4);
        const float4 was = *at_s;
        *at_s = make_float4(fmaf(keep[i], was.x, add[i][0]), fmaf(keep[i], was.y, add[i][1]), fmaf(keep[i], was.z, add[i][2]), fmaf(keep[i], was.w, add[i][3]));
      }
    }
    __syncthreads();                                  // the new state lies; keys, A and the partial sums have been used up
  }
  for (int i = tid; i < DK * COLS; i += THREADS) {
    const int c = i / DK, d = i - c * DK;
    if (d < a.dk && c0 + c < a.dv) st[(int64_t)(c0 + c) * a.dk + d] = S[place_of<DK>(d) + c];
  }
}

template <typename TI, int DK, bool DELTA>
int launch(ChannelArgs a, int span, cudaStream_t stream) {
  constexpr size_t prepare_smem = ((size_t)4 * HD * LDT + 2 * C * LDT + 4 * HD) * 4;
  constexpr size_t walk_smem = ((size_t)DK * (DELTA ? 128 : 64) + C * DK + C * C + 2 * DK * LDC + 4 * C * LDC) * 4;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(channel_prepare_kernel<TI, DK, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)prepare_smem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(channel_walk_kernel<TI, DK, DELTA>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_smem);
    if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "chunked channels: cannot reserve shared memory: %s", cudaGetErrorString(e));
    configured = true;
  }
  const int total = a.places;
  for (a.place0 = 0; a.place0 < total; a.place0 += span) {
    a.places = total - a.place0 < span ? total - a.place0 : span;
    kvad_launch(channel_prepare_kernel<TI, DK, DELTA>, dim3(a.places, a.heads), dim3(THREADS), prepare_smem, stream, a);
    kvad_launch(channel_walk_kernel<TI, DK, DELTA>, dim3(a.n_seqs * a.heads, (a.dv + COLS - 1) / COLS), dim3(THREADS), walk_smem, stream, a);
  }
  KVAD_CHECK_LAUNCH("chunked channels");
  return KVAD_OK;
}

template <typename TI>
int dispatch(const ChannelArgs& a, bool delta, int span, cudaStream_t stream) {
  if (a.dk <= 64) return delta ? launch<TI, 64, true>(a, span, stream) : launch<TI, 64, false>(a, span, stream);
  return delta ? launch<TI, 128, true>(a, span, stream) : launch<TI, 128, false>(a, span, stream);
}

inline int64_t work_per(int dk, int dv) {
  const int64_t DK = dk <= 64 ? 64 : 128;
  return DK * 128 + C * DK + (int64_t)C * ((dv + 3) / 4 * 4) + C * C + DK;
}

}  // namespace

// Scratch in floats for one chunk of one head; `n` rows of `s` sequences are n / 64 + s places of chunks, and `work` holds `span` of them at a time.
KVAD_EXPORT int kvad_channels_work(int dk, int dv) { return (int)work_per(dk, dv); }

// The gated delta rule (`beta` given) or the gated linear kind over prompt rows; `gates` are the decays themselves (see kvad_gated_recurrence).
KVAD_EXPORT int kvad_channels_chunked(int dtype, const void* q, int64_t ld_q, const void* k, int64_t ld_k, const void* v, int64_t ld_v, const float* gates,
                                      int64_t ld_gates, const float* beta, int64_t ld_beta, float* out, int64_t ld_out, int n_rows, float* state,
                                      int64_t state_stride, const int* seq_starts, const int* seq_slots, int n_seqs, int heads, int kv_heads, int dk, int dv,
                                      float q_scale, float* work, int span, int from, cudaStream_t stream) {
  KVAD_REQUIRE(n_rows >= 0 && n_seqs > 0 && heads > 0 && kv_heads > 0 && heads % kv_heads == 0 && dk > 0 && dv > 0, "chunked channels: bad sizes seqs=%d heads=%d dk=%d dv=%d",
               n_seqs, heads, dk, dv);
  KVAD_REQUIRE(q && k && v && gates && out && state && seq_starts && seq_slots && work && span > 0, "chunked channels: bad arguments");
  KVAD_REQUIRE(heads <= 65535 && (int64_t)n_seqs * heads < (1ll << 31) && (dv + COLS - 1) / COLS <= 65535, "chunked channels: more than one launch takes");
  const uintptr_t unit = dtype == KVAD_DTYPE_F32 ? 15 : 7;
  if (dk > 128 || dk % 4 || ld_q % 4 || ld_k % 4 || ld_gates % 4 || ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k)) & unit) ||
      ((reinterpret_cast<uintptr_t>(work) | reinterpret_cast<uintptr_t>(gates)) & 15))
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "chunked channels: keys of %d entries a head; up to 128, all in whole quads, are taken", dk);
  ChannelArgs a = {};
  a.q = q; a.k = k; a.v = v; a.ld_q = ld_q; a.ld_k = ld_k; a.ld_v = ld_v; a.gates = gates; a.ld_gates = ld_gates; a.beta = beta; a.ld_beta = ld_beta;
  a.seq_starts = seq_starts; a.seq_slots = seq_slots; a.n_seqs = n_seqs; a.heads = heads; a.group = heads / kv_heads; a.dk = dk; a.dv = dv;
  a.from = from; a.places = n_rows / C + n_seqs; a.q_scale = q_scale; a.out = out; a.ld_out = ld_out; a.state = state; a.state_stride = state_stride;
  const int64_t DK = dk <= 64 ? 64 : 128, places = (int64_t)span * heads;
  a.wq = work;
  a.kt = a.wq + places * DK * 128;
  a.at = a.kt + places * C * DK;
  a.whole = a.at + places * C * C;
  a.x = a.whole + places * DK;
  if (dtype == KVAD_DTYPE_F32) return dispatch<float>(a, beta != nullptr, span, stream);
  if (dtype == KVAD_DTYPE_BF16) return dispatch<__nv_bfloat16>(a, beta != nullptr, span, stream);
  KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "chunked channels: unknown dtype %d", dtype);
}

KVAD_DEFINE_LAST_ERROR()
