// Linear recurrences of prompts, 64 rows at a time: retention (`retention.cu`) and the matrix memory (`gated_recurrence.cu`),
// whose state decays by one number per head and row,
//
//   S_t = f_t S_(t-1) + w_t k_t v_t^T,   o_t = S_t^T q_t.
//
// Walking the rows one after another (what those kernels do, and still do for few rows) is a chain of ~0.35 us a row whatever the
// arithmetic.  Here a sequence's rows are cut into chunks of 64 and the same sums are taken in another order, as products:
//
//   1  U_c = sum_j (decay from row j to the chunk's end) w_j k_j v_j^T          every chunk and head by itself
//   2  S_(c+1) = (decay over chunk c) S_c + U_c                                 from chunk to chunk, entry by entry
//   3  o_i = sum_(j <= i) (decay from j to i) w_j (q_i . k_j) v_j + (decay to i) S_c^T q_i      every chunk and head by itself
//
// The products run on mma.sync with 32-bit operands cut into bfloat16 pieces x = h + m + l (exact above about 2^-110; an operand that is bfloat16 as it
// comes is one piece): the six products that reach 2^-24, or three, or one.  The tensor core truncates where it accumulates, so h h joins the 32-bit sums by
// rounded additions after every 16 terms; the others, 2^-8 of it, have an accumulator of their own.  A thread cuts its fragments itself
// from 32-bit rows in shared memory.  Numbers that are not finite have no pieces: a block that meets one leaves them out of the products and adds their terms by fmaf.  Decays are powers of the head's constant (retention), or exponentials of
// differences of logarithms that are summed up in 64 bits within the chunk (matrix memory), so that a difference of two large sums
// keeps its last places.  The matrix memory's running maximum goes along: a chunk's own maximum at its end, the maximum carried over
// the chunks in step 2, and per row m_i = F_i + max(m_c, max_(j <= i) (i_j - F_j)); every weight is at most 1.
//
// Measured: 2 x 1024 rows of 8 heads of 128 x 128 (rotated, normed, gated, bfloat16) 387 us walked, 84 with fmaf chains, 68 so; the matrix memory over
// 1000 + 517 + 37 rows of 8 heads of 64 x 128 334, 48 and 39.  Of the 68: kernel 1 15 (rows 4, turning and weights 4, product 6), kernel 2 6, kernel 3 42 (rows 5,
// turning 4, scores 7, state 17, values 1, norm, gate and rows out 6), the rest between them.  At six products mma.sync is no faster than the CUDA cores' peak; what it
// saves is the shared-memory traffic that kept them at a fifth of it.
//
// Chunks of all sequences lie in one list: chunk c of sequence s is place seq_starts[s] / 64 + s + c, which never collides.  The list is taken in
// spans of as many places as the scratch holds, one after another: the sequences' own states carry over from one to the next.
#include "common.cuh"

using namespace kvad;

namespace {

constexpr int C = 64, THREADS = 256, LDT = C + 4;      // rows a chunk; row stride of transposed tiles
constexpr int RETENTION = 0, MEMORY = 1;

__device__ __forceinline__ float silu_f(float z) { return z / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_f(float z) { return fmaxf(z, 0.f) + log1pf(expf(-fabsf(z))); }

struct ChunkArgs {
  const void* q; const void* k; const void* v;
  int64_t ld_q, ld_k, ld_v;
  const int* seq_starts; const int* kv_lens; const int* seq_slots;
  int n_seqs, heads, group, dk, dv;
  int from;                 // only sequences of so many new rows or more (the others: retention.cu, gated_recurrence.cu)
  int place0, places;       // the span: its first place, how many
  float* work;              // [places, heads, dk * dv]: U of a chunk, then the state before it (in the state's own order of entries)
  float* state; int64_t state_stride;
  // retention
  const float* decay; const float* inv_freq; int rot_dims, interleaved, act;
  float k_scale, q_scale;
  // matrix memory
  const float* gates; int64_t ld_gates; float cap;
  float* work_n;            // [places, heads, dk + 2]: the normaliser like U (after step 2: before the chunk), then the chunk's decay and maximum (logarithms)
  float* work_m;            // [places, heads]: the running maximum before the chunk
  int tiles;
  // out: 32-bit read-outs, or finished rows
  float* raw; int64_t ld_raw;
  void* out; int64_t ld_out; const void* gate; int64_t ld_gate; int unit_norm, finish, vec_out;      // vec_out: rows of `out` begin on whole quads
  float eps;
};

// The upper halves of two floats as a pair of bfloat16 (truncated), and what is left of each.
__device__ __forceinline__ uint32_t cut(float& a, float& b) {
  const uint32_t x = __float_as_uint(a), y = __float_as_uint(b);
  a -= __uint_as_float(x & 0xffff0000u);
  b -= __uint_as_float(y & 0xffff0000u);
  return __byte_perm(x, y, 0x7632);
}
__device__ __forceinline__ uint32_t upper(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }
__device__ __forceinline__ void mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// the same into zeros
__device__ __forceinline__ void mma_first(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}
__device__ __forceinline__ bool not_finite(float x) { return (__float_as_uint(x) & 0x7f800000u) == 0x7f800000u; }

// acc[i][j] += sum over k in [0, n) of A[k][row0 + 16 i ..] B[k][col0 + 8 j ..] by a warp, in mma.sync's layout: entry e of a tile is row lane / 4 + 8 (e / 2),
// column 2 (lane % 4) + e % 2.  PA, PB: pieces of the operands.  n in whole sixteens; row strides of 4 more than a multiple of 32 meet no bank twice.
// CLEAN: entries that are not finite count as zeros (`leftover` adds what they give).
template <int MT, int NT, int PA, int PB, bool CLEAN = false>
__device__ __forceinline__ void product(float (&acc)[MT][NT][4], const float* A, int lda, const float* B, int ldb, int n) {
  const int g = (threadIdx.x & 31) >> 2, t2 = (threadIdx.x & 3) * 2;
  float low[MT][NT][4] = {};
  A += t2 * lda + g;
  B += t2 * ldb + g;
#pragma unroll 1
  for (int k = 0; k < n; k += 16, A += 16 * lda, B += 16 * ldb) {
    uint32_t ap[PA][MT][4];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const float* at = A + (f >> 1) * 8 * lda + i * 16 + (f & 1) * 8;
        float x = at[0], y = at[lda];
        if (CLEAN) x = not_finite(x) ? 0.f : x, y = not_finite(y) ? 0.f : y;
        if (PA == 1) {
          ap[0][i][f] = upper(x, y);
        } else {
          ap[0][i][f] = cut(x, y);
          ap[PA > 1 ? 1 : 0][i][f] = cut(x, y);
          ap[PA > 2 ? 2 : 0][i][f] = upper(x, y);
        }
      }
    // (two columns of tiles at a time: a product follows three others before it meets its own accumulator again)
    constexpr int W = NT < 2 ? NT : 2;
#pragma unroll
    for (int j0 = 0; j0 < NT; j0 += W) {
      uint32_t bp[PB][W][2];
#pragma unroll
      for (int j = 0; j < W; ++j)
#pragma unroll
        for (int f = 0; f < 2; ++f) {
          const float* at = B + f * 8 * ldb + (j0 + j) * 8;
          float x = at[0], y = at[ldb];
          if (CLEAN) x = not_finite(x) ? 0.f : x, y = not_finite(y) ? 0.f : y;
          if (PB == 1) {
            bp[0][j][f] = upper(x, y);
          } else {
            bp[0][j][f] = cut(x, y);
            bp[PB > 1 ? 1 : 0][j][f] = cut(x, y);
            bp[PB > 2 ? 2 : 0][j][f] = upper(x, y);
          }
        }
      float high[MT][W][4];
      constexpr int PRODUCTS = PA == 3 && PB == 3 ? 6 : (PA == 3 || PB == 3 ? 3 : 1);
      // which pieces meet: h h, then the small ones from the smallest on
      constexpr int XA[6] = {0, PA == 3 ? 2 : 0, PA == 3 && PB == 3 ? 0 : (PA == 3 ? 1 : 0), 1, 1, 0}, XB[6] = {0, PA == 3 ? 0 : 2, PA == 3 && PB == 3 ? 2 : (PA == 3 ? 0 : 1), 1, 0, 1};
#pragma unroll
      for (int t = 0; t < PRODUCTS; ++t)
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
          for (int i = 0; i < MT; ++i) {
            if (t == 0) mma_first(high[i][j], ap[0][i], bp[0][j]);
            else mma(low[i][j0 + j], ap[XA[t] % PA][i], bp[XB[t] % PB][j]);
          }
#pragma unroll
      for (int j = 0; j < W; ++j)
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][j0 + j][e] += high[i][j][e];
    }
  }
  if (PA == 3 || PB == 3) {
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] += low[i][j][e];
  }
}
// The terms of which an operand is not finite, by fmaf: what they give is what 32-bit arithmetic gives, the other terms' sums keep their bits.  TRIANGLE: a row takes
// the terms k <= row only (row0: its first row's number).
template <int MT, int NT, bool TRIANGLE>
__device__ __noinline__ void leftover_terms(float* acc, const float* A, int lda, const float* B, int ldb, int n, int row0) {
  const int g = (threadIdx.x & 31) >> 2, t2 = (threadIdx.x & 3) * 2;
  for (int at = 0; at < MT * NT * 4; ++at) {
    const int e = at & 3, j = (at >> 2) % NT, i = (at >> 2) / NT;
    const int r = i * 16 + g + (e >> 1) * 8, c = j * 8 + t2 + (e & 1), m = TRIANGLE ? min(n, row0 + r + 1) : n;
    float sum = acc[at];
    for (int k = 0; k < m; ++k) {
      const float x = A[k * lda + r], y = B[k * ldb + c];
      if (not_finite(x) || not_finite(y)) sum = fmaf(x, y, sum);
    }
    acc[at] = sum;
  }
}
template <int MT, int NT, bool TRIANGLE>
__device__ __forceinline__ void leftover(float (&acc)[MT][NT][4], const float* A, int lda, const float* B, int ldb, int n, int row0) {
  float copy[MT * NT * 4];                  // (the accumulators themselves stay in registers)
#pragma unroll
  for (int at = 0; at < MT * NT * 4; ++at) copy[at] = acc[(at >> 2) / NT][(at >> 2) % NT][at & 3];
  leftover_terms<MT, NT, TRIANGLE>(copy, A, lda, B, ldb, n, row0);
#pragma unroll
  for (int at = 0; at < MT * NT * 4; ++at) acc[(at >> 2) / NT][(at >> 2) % NT][at & 3] = copy[at];
}
// As many pieces as the operands need: PA, PB where rows are bfloat16 as they come (`as_is`), three and three elsewhere; `bad`: some operand is not finite.
template <int MT, int NT, int PA, int PB, bool TRIANGLE, typename TI>
__device__ __forceinline__ void product_of(float (&acc)[MT][NT][4], const float* A, int lda, const float* B, int ldb, int n, bool as_is, bool bad, int n_bad, int row0) {
  if (!bad) {
    if (sizeof(TI) == 2 && as_is) product<MT, NT, PA, PB>(acc, A, lda, B, ldb, n);
    else product<MT, NT, 3, 3>(acc, A, lda, B, ldb, n);
  } else {
    if (sizeof(TI) == 2 && as_is) product<MT, NT, PA, PB, true>(acc, A, lda, B, ldb, n);
    else product<MT, NT, 3, 3, true>(acc, A, lda, B, ldb, n);
    leftover<MT, NT, TRIANGLE>(acc, A, lda, B, ldb, n_bad, row0);
  }
}

struct Place { int s, row0, n, pos0; };      // sequence, first row, rows (0: no such chunk), position of the first row
__device__ __forceinline__ Place find(const ChunkArgs& a, int place) {
  int lo = 0, hi = a.n_seqs - 1;
  while (lo < hi) {                            // the last sequence whose first place is not behind this one
    const int mid = (lo + hi + 1) / 2;
    if (a.seq_starts[mid] / C + mid <= place) lo = mid;
    else hi = mid - 1;
  }
  Place p;
  const int start = a.seq_starts[lo], n_new = a.seq_starts[lo + 1] - start, first = (place - (start / C + lo)) * C;
  p.s = lo;
  p.row0 = start + first;
  p.n = n_new < a.from ? 0 : max(0, min(C, n_new - first));
  p.pos0 = a.kv_lens != nullptr ? a.kv_lens[lo] - n_new + first : 0;
  return p;
}
// The chunks of sequence `s` that lie in the span: from `begin` up to `end`, and where chunk 0 would lie in the span's scratch.
struct Run { int begin, end, n_new, n_chunks, base; };
__device__ __forceinline__ Run run_of(const ChunkArgs& a, int s) {
  Run r;
  const int start = a.seq_starts[s];
  r.n_new = a.seq_starts[s + 1] - start;
  r.n_chunks = r.n_new >= a.from ? (r.n_new + C - 1) / C : 0;
  r.base = start / C + s - a.place0;
  r.begin = max(0, -r.base);
  r.end = min(r.n_chunks, a.places - r.base);
  return r;
}

// The matrix memory's gates of a chunk's rows, by the block's first 64 threads: F (the forget gates' logarithms summed up from the chunk's
// first row on), the input gate, and the running maximum of (input - F).
__device__ __forceinline__ void chunk_gates(const ChunkArgs& a, const Place& p, int h, double* F, float* in, float* best, float* scratch) {
  const int t = threadIdx.x;
  if (t < C) {
    double f = 0.0;
    float i = -INFINITY;
    if (t < p.n) {
      const float* g = a.gates + (int64_t)(p.row0 + t) * a.ld_gates;
      i = a.cap * tanhf(g[h] / a.cap);
      f = (double)-softplus_f(-a.cap * tanhf(g[a.heads + h] / a.cap));
    }
    const int lane = t & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const double up = __shfl_up_sync(0xffffffffu, f, o);
      if (lane >= o) f += up;
    }
    F[t] = f;
    in[t] = i;
  }
  __syncthreads();
  if (t < C) {
    const double f = F[t] + (t >= 32 ? F[31] : 0.0);
    float m = in[t] == -INFINITY ? -INFINITY : (float)((double)in[t] - f);
    const int lane = t & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float up = __shfl_up_sync(0xffffffffu, m, o);
      if (lane >= o) m = fmaxf(m, up);
    }
    best[t] = m;
    if (t == 31) *scratch = m;
    __syncwarp();
  }
  __syncthreads();
  double whole = 0.0;
  if (t < C) whole = F[t] + (t >= 32 ? F[31] : 0.0);
  __syncthreads();
  if (t < C) {
    F[t] = whole;
    if (t >= 32) best[t] = fmaxf(best[t], *scratch);
  }
  __syncthreads();
}

// A chunk's rows of one head on their way into shared memory, W entries wide: transposed [entry][row] or plain [row][entry]; entries and rows that
// do not exist are zeros.  `ask` starts the loads (of several operands, before the first `put`), `put` says whether any of the thread's entries is not finite.
__device__ __forceinline__ float4 widen(const float4& x) { return x; }
__device__ __forceinline__ float4 widen(const uint2& raw) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
template <typename TI> struct Quad { using type = float4; };
template <> struct Quad<__nv_bfloat16> { using type = uint2; };
template <typename TI, int W, bool TRANSPOSED>
struct Rows {
  using Raw = typename Quad<TI>::type;
  static constexpr int N = C * (W / 4) / THREADS;
  Raw raw[N];
  static __device__ __forceinline__ void place(int f, int& r, int& c) {
    const int i = threadIdx.x + f * THREADS;
    // transposed: a warp takes 8 rows by 4 neighbouring quads (whole 32-byte sectors of bfloat16, and stores that meet a bank twice)
    r = TRANSPOSED ? (i & 7) + (i >> 5) % (C / 8) * 8 : i / (W / 4);
    c = (TRANSPOSED ? ((i >> 3) & 3) + (i >> 5) / (C / 8) * 4 : i % (W / 4)) * 4;
  }
  __device__ __forceinline__ void ask(const TI* src, int64_t ld_src, const Place& p, int width) {
#pragma unroll
    for (int f = 0; f < N; ++f) {
      int r, c;
      place(f, r, c);
      raw[f] = Raw{};
      if (r < p.n && c < width) raw[f] = *reinterpret_cast<const Raw*>(src + (int64_t)(p.row0 + r) * ld_src + c);
    }
  }
  __device__ __forceinline__ bool put(float* dst, int ld, bool act, float scale_from, int scaled_from) const {
    bool bad = false;
#pragma unroll
    for (int f = 0; f < N; ++f) {
      int r, c;
      place(f, r, c);
      const float4 x = widen(raw[f]);
      float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        if (act) v[e] = silu_f(v[e]);
        if (c + e >= scaled_from) v[e] *= scale_from;
        bad |= not_finite(v[e]);
        if (TRANSPOSED) dst[(c + e) * ld + r] = v[e];
      }
      if (!TRANSPOSED) *reinterpret_cast<float4*>(dst + r * ld + c) = make_float4(v[0], v[1], v[2], v[3]);
    }
    return bad;
  }
};

// Pairs of q (or null) and k turned by the rows' positions where they lie, k scaled after turning.
template <bool TRANSPOSED>
__device__ __forceinline__ void turn(const ChunkArgs& a, const Place& p, float* q, float* k, int ld) {
  const int half = a.rot_dims / 2;
#pragma unroll 4
  for (int i = threadIdx.x; i < C * half; i += THREADS) {
    const int r = TRANSPOSED ? i % C : i / half, pr = TRANSPOSED ? i / C : i % half;
    const int ea = a.interleaved ? 2 * pr : pr, eb = a.interleaved ? 2 * pr + 1 : pr + half;
    const int ia = TRANSPOSED ? ea * ld + r : r * ld + ea, ib = TRANSPOSED ? eb * ld + r : r * ld + eb;
    float sn, cs;
    sincosf((float)(p.pos0 + r) * a.inv_freq[pr], &sn, &cs);
    if (q != nullptr) {
      const float x = q[ia], y = q[ib];
      q[ia] = x * cs - y * sn;
      q[ib] = y * cs + x * sn;
    }
    const float x = k[ia], y = k[ib];
    k[ia] = (x * cs - y * sn) * a.k_scale;
    k[ib] = (y * cs + x * sn) * a.k_scale;
  }
}

// ---- 1: what a chunk leaves in the state ---------------------------------------------------------------------------------
template <int KIND, typename TI, int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2) chunk_sum_kernel(const ChunkArgs a) {
  constexpr int LDK = DK + 4, LDV = DV + 4;
  extern __shared__ float smem[];
  float* ks = smem;                         // [C][LDK]
  float* vs = ks + C * LDK;                 // [C][LDV]
  __shared__ double F[KIND == MEMORY ? C : 1];
  __shared__ float in[C], best[C], weight[C], scratch;
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.y, qh = h / a.group;
  const Place p = find(a, a.place0 + blockIdx.x);
  if (p.n == 0) return;
  const bool half = KIND == RETENTION && a.rot_dims > 0;
  bool bad;
  {
    Rows<TI, DK, false> k;
    Rows<TI, DV, false> v;
    k.ask((const TI*)a.k + qh * a.dk, a.ld_k, p, a.dk);
    v.ask((const TI*)a.v + h * a.dv, a.ld_v, p, a.dv);
    k.put(ks, LDK, KIND == RETENTION && a.act, a.k_scale, a.rot_dims);
    bad = v.put(vs, LDV, KIND == RETENTION && a.act, 1.f, DV);
  }
  if (KIND == MEMORY) {
    chunk_gates(a, p, h, F, in, best, &scratch);
    if (threadIdx.x < C) {                  // weights at the chunk's end, against its own maximum there
      const int t = threadIdx.x;
      weight[t] = t < p.n ? expf((float)((double)in[t] - F[t] - (double)best[p.n - 1])) : 0.f;
    }
  } else {
    if (half) {
      __syncthreads();
      turn<false>(a, p, nullptr, ks, LDK);
    }
    if (threadIdx.x < C) weight[threadIdx.x] = powf(a.decay[h], (float)max(0, p.n - 1 - (int)threadIdx.x));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C * (DK / 4); i += THREADS) {
    float4* at = reinterpret_cast<float4*>(ks + i / (DK / 4) * LDK + i % (DK / 4) * 4);
    const float w = weight[i / (DK / 4)];
    float4 x = *at;
    x.x *= w; x.y *= w; x.z *= w; x.w *= w;
    bad |= not_finite(x.x) || not_finite(x.y) || not_finite(x.z) || not_finite(x.w);
    *at = x;
  }
  bad = __syncthreads_or(bad);
  // (entries in the state's own order: retention [dk][dv], the matrix memory [dv][dk]; a warp has half of the rows, 32 at a time, and a quarter of the columns)
  constexpr int NR = KIND == MEMORY ? DV : DK, NC = KIND == MEMORY ? DK : DV, NT = NC / 32;
  const int warp = threadIdx.x >> 5, col0 = (warp >> 1) * (NC / 4), n16 = (p.n + 15) & ~15;
  const float* A = KIND == MEMORY ? vs : ks;
  const float* B = (KIND == MEMORY ? ks : vs) + col0;
  constexpr int LDA = KIND == MEMORY ? LDV : LDK, LDB = KIND == MEMORY ? LDK : LDV, EA = KIND == MEMORY ? 1 : 3, EB = KIND == MEMORY ? 3 : 1;
  const int rows = KIND == MEMORY ? a.dv : a.dk, cols = KIND == MEMORY ? a.dk : a.dv;
  float* u = a.work + ((int64_t)blockIdx.x * a.heads + h) * a.dk * a.dv;
  const int g = (threadIdx.x & 31) >> 2, t2 = (threadIdx.x & 3) * 2;
#pragma unroll 1
  for (int row0 = (warp & 1) * 32; row0 < NR; row0 += 64) {
    float acc[2][NT][4] = {};
    product_of<2, NT, EA, EB, false, TI>(acc, A + row0, LDA, B, LDB, n16, !(KIND == RETENTION && a.act), bad, p.n, 0);
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e = 0; e < 4; e += 2) {
        const int r = row0 + i * 16 + g + e * 4;
        if (r >= rows) continue;
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const int c = col0 + j * 8 + t2;
          if (c < cols) *reinterpret_cast<float2*>(u + r * cols + c) = make_float2(acc[i][j][e], acc[i][j][e + 1]);
        }
      }
  }
  if (KIND == MEMORY) {
    float* un = a.work_n + ((int64_t)blockIdx.x * a.heads + h) * (a.dk + 2);
    for (int d = threadIdx.x; d < a.dk; d += THREADS) {
      float sum = 0.f;
      for (int t = 0; t < p.n; ++t) sum += ks[t * LDK + d];
      un[d] = sum;
    }
    if (threadIdx.x == 0) {
      un[a.dk] = (float)F[p.n - 1];
      un[a.dk + 1] = (float)(F[p.n - 1] + (double)best[p.n - 1]);
    }
  }
}

// ---- 2: the state from chunk to chunk --------------------------------------------------------------------------------------
// A thread carries four entries; its loads of several chunks are on their way at once.  `work` holds the state before each chunk afterwards.
template <int KIND>
__global__ void __launch_bounds__(THREADS) chunk_scan_kernel(const ChunkArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int s = blockIdx.x / a.heads, h = blockIdx.x - s * a.heads;
  const Run run = run_of(a, s);
  if (run.begin >= run.end) return;
  const int entries = a.dk * a.dv;
  const int at = (blockIdx.y * THREADS + threadIdx.x) * 4;
  float* slot = a.state + (int64_t)a.seq_slots[s] * a.state_stride;
  float* st = slot + (int64_t)h * entries;
  float m = KIND == MEMORY ? slot[(int64_t)a.heads * entries + (int64_t)a.heads * a.tiles * a.dk + (int64_t)h * a.tiles] : 0.f;
  const bool mine = at < entries;
  // the normaliser (one copy of it is carried; the state keeps one a tile) by the first block's first threads
  const bool norm = KIND == MEMORY && blockIdx.y == 0 && (int)threadIdx.x < a.dk;
  float4 S = mine ? *reinterpret_cast<float4*>(st + at) : make_float4(0.f, 0.f, 0.f, 0.f);
  float* n_st = slot + (int64_t)a.heads * entries + (int64_t)h * a.tiles * a.dk;
  float N = norm ? n_st[threadIdx.x] : 0.f;
  const float lambda = KIND == RETENTION ? a.decay[h] : 0.f;
  const float whole = KIND == RETENTION ? powf(lambda, (float)C) : 0.f;
  const int64_t step = (int64_t)a.heads * entries, n_step = (int64_t)a.heads * (a.dk + 2);
  float* w = a.work + (int64_t)run.base * step + (int64_t)h * entries + at;
  float* wn = KIND == MEMORY ? a.work_n + (int64_t)run.base * n_step + (int64_t)h * (a.dk + 2) : nullptr;
  constexpr int AHEAD = 8;
  for (int c0 = run.begin; c0 < run.end; c0 += AHEAD) {
    float4 u[AHEAD];
    float f[AHEAD], top[AHEAD], un[AHEAD];
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const bool in = c0 + i < run.end;
      u[i] = in && mine ? *reinterpret_cast<const float4*>(w + (c0 + i) * step) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (KIND == MEMORY) {
        f[i] = in ? wn[(c0 + i) * n_step + a.dk] : 0.f;
        top[i] = in ? wn[(c0 + i) * n_step + a.dk + 1] : 0.f;
        un[i] = in && norm ? wn[(c0 + i) * n_step + threadIdx.x] : 0.f;
      }
    }
#pragma unroll
    for (int i = 0; i < AHEAD; ++i) {
      const int c = c0 + i;
      if (c >= run.end) break;
      float keep = whole, take = 1.f;
      if (mine) *reinterpret_cast<float4*>(w + c * step) = S;
      if (KIND == MEMORY) {
        const float next = fmaxf(f[i] + m, top[i]);
        keep = expf(f[i] + m - next);
        take = expf(top[i] - next);
        if (norm) wn[c * n_step + threadIdx.x] = N;
        if (blockIdx.y == 0 && threadIdx.x == 0) a.work_m[(int64_t)(run.base + c) * a.heads + h] = m;
        m = next;
        N = fmaf(keep, N, take * un[i]);
      } else if (c == run.n_chunks - 1) {
        keep = powf(lambda, (float)(run.n_new - c * C));
      }
      S.x = fmaf(keep, S.x, take * u[i].x);
      S.y = fmaf(keep, S.y, take * u[i].y);
      S.z = fmaf(keep, S.z, take * u[i].z);
      S.w = fmaf(keep, S.w, take * u[i].w);
    }
  }
  if (mine) *reinterpret_cast<float4*>(st + at) = S;
  if (KIND == MEMORY) {
    if (norm)
      for (int i = 0; i < a.tiles; ++i) n_st[(int64_t)i * a.dk + threadIdx.x] = N;
  }
}
// The running maxima at their new place in the state: a launch of its own, because every block of the scan starts from the old one.
__global__ void chunk_max_kernel(const ChunkArgs a) {
  pdl_launch_dependents();
  pdl_wait();
  const int s = blockIdx.x;
  const Run run = run_of(a, s);
  if (run.begin >= run.end) return;
  const int last = run.base + run.end - 1;
  float* slot = a.state + (int64_t)a.seq_slots[s] * a.state_stride + (int64_t)a.heads * a.dk * a.dv + (int64_t)a.heads * a.tiles * a.dk;
  for (int h = threadIdx.x; h < a.heads; h += blockDim.x) {
    const float* end = a.work_n + ((int64_t)last * a.heads + h) * (a.dk + 2) + a.dk;
    const float m = fmaxf(end[0] + a.work_m[(int64_t)last * a.heads + h], end[1]);
    for (int i = 0; i < a.tiles; ++i) slot[(int64_t)h * a.tiles + i] = m;
  }
}

// ---- 3: the read-outs ------------------------------------------------------------------------------------------------------
// A warp has 32 of the chunk's rows and a quarter of the columns.
template <int KIND, typename TI, int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2) chunk_read_kernel(const ChunkArgs a) {
  constexpr int PIECE = 32, LDS = DV + 4;                               // rows of the state that come at a time
  constexpr int REGION = DK * LDT > C * LDT + PIECE * LDS ? DK * LDT : C * LDT + PIECE * LDS;
  extern __shared__ float smem[];
  float* qt = smem;                         // [DK][LDT]
  float* kt = qt + DK * LDT;                // [DK][LDT], later the weighted scores [j][i] and a piece of the state
  float* vs = kt + REGION;                  // [C][LDS]
  float* pt = kt;
  float* ss = kt + C * LDT;
  __shared__ double F[KIND == MEMORY ? C : 1];
  __shared__ float in[C], best[C], power[C + 1], carried[C], den[5][C], sq_sum[4][C], scratch, mx[C];
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.y, qh = h / a.group;
  const Place p = find(a, a.place0 + blockIdx.x);
  if (p.n == 0) return;
  const bool act = KIND == RETENTION && a.act;
  // Rows that are bfloat16 as they come stay so (one piece); their factors go to the scores and to what the state gives.
  const bool as_is = sizeof(TI) == 2 && !act && (KIND == MEMORY || a.rot_dims == 0);
  bool bad;
  {
    Rows<TI, DK, true> q, k;
    Rows<TI, DV, false> v;
    q.ask((const TI*)a.q + qh * a.dk, a.ld_q, p, a.dk);
    k.ask((const TI*)a.k + qh * a.dk, a.ld_k, p, a.dk);
    v.ask((const TI*)a.v + h * a.dv, a.ld_v, p, a.dv);
    bad = q.put(qt, LDT, act, a.q_scale, as_is ? DK : 0);
    bad |= k.put(kt, LDT, act, a.k_scale, as_is ? DK : a.rot_dims);
    bad |= v.put(vs, LDS, act, 1.f, DV);
  }
  const float owed_q = as_is ? a.q_scale : 1.f, owed_k = as_is ? a.k_scale : 1.f;
  const int warp = threadIdx.x >> 5, wr = (warp & 1) * 32, wc = warp >> 1, g = (threadIdx.x & 31) >> 2, t2 = (threadIdx.x & 3) * 2;
  if (KIND == MEMORY) {
    const float m_c = a.work_m[(int64_t)blockIdx.x * a.heads + h];
    chunk_gates(a, p, h, F, in, best, &scratch);
    if (threadIdx.x < C) {
      const int t = threadIdx.x;
      const float top = fmaxf(m_c, best[t]);               // m_i = F_i + this
      mx[t] = top;
      carried[t] = expf(m_c - top);
    }
  } else {
    if (a.rot_dims > 0) {
      __syncthreads();
      turn<true>(a, p, qt, kt, LDT);
    }
    if (threadIdx.x <= C) power[threadIdx.x] = powf(a.decay[h], (float)threadIdx.x);
  }
  bad = __syncthreads_or(bad);

  // The state before the chunk comes a piece at a time by way of registers, each piece asked for before the arithmetic that runs ahead of it.
  // (The matrix memory's is [dv][dk]: a thread takes four neighbours along dk of one column.)
  constexpr int FETCH = DV / 32;
  const float* S = a.work + ((int64_t)blockIdx.x * a.heads + h) * a.dk * a.dv;
  float4 piece[FETCH];
  auto fetch = [&](int d0) {
    const int nd = min(PIECE, a.dk - d0);
#pragma unroll
    for (int f = 0; f < FETCH; ++f) {
      const int i = threadIdx.x + f * THREADS;
      const int c = KIND == MEMORY ? i % DV : i % (DV / 4) * 4, d = KIND == MEMORY ? i / DV * 4 : i / (DV / 4);
      piece[f] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < a.dv && d < nd) piece[f] = *reinterpret_cast<const float4*>(KIND == MEMORY ? S + (int64_t)c * a.dk + d0 + d : S + (int64_t)(d0 + d) * a.dv + c);
    }
  };
  fetch(0);

  float sc[2][2][4] = {};
  if (wr + 31 >= wc * 16)                   // (tiles above the diagonal are not seen)
    product_of<2, 2, 1, 1, false, TI>(sc, qt + wr, LDT, kt + wc * 16, LDT, DK, as_is, bad, a.dk, 0);
  // weights; the matrix memory's sums of a row's weighted scores meet over its four threads and the four warps of its columns
  bool wild = false;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2) {
      const int r = wr + i * 16 + g + e2 * 8;
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e1 = 0; e1 < 2; ++e1) {
          const int c = wc * 16 + j * 8 + t2 + e1;
          float& x = sc[i][j][e2 * 2 + e1];
          // (a row that is not seen counts for nothing, also where its score is no number)
          if (c <= r && r < p.n) x *= owed_q * owed_k * (KIND == MEMORY ? expf((float)((double)in[c] - F[c] - (double)mx[r])) : power[r - c]);
          else x = 0.f;
          wild |= not_finite(x);
          sum += x;
        }
      if (KIND == MEMORY) {
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        if (t2 == 0) den[wc][r] = sum;
      }
    }
  wild = __syncthreads_or(wild) || bad;     // (the keys have been used up)
  if (KIND == MEMORY) {                     // ... and the normaliser before the chunk along the row's query
    const float* n_c = a.work_n + ((int64_t)blockIdx.x * a.heads + h) * (a.dk + 2);
    const int r = threadIdx.x >> 2, part = threadIdx.x & 3;
    float sum = 0.f;
    for (int d = part; d < a.dk; d += 4) sum = fmaf(qt[d * LDT + r], n_c[d], sum);
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    if (part == 0) den[4][r] = fmaf(carried[r], sum * owed_q, (den[0][r] + den[1][r]) + (den[2][r] + den[3][r]));
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) pt[(wc * 16 + j * 8 + t2 + (e & 1)) * LDT + wr + i * 16 + g + (e >> 1) * 8] = sc[i][j][e];

  constexpr int NT = DV / 32;
  const int col0 = wc * (DV / 4);
  float acc[2][NT][4] = {};
  for (int d0 = 0; d0 < a.dk; d0 += PIECE) {
    if (d0 > 0) __syncthreads();
    bool odd = false;
#pragma unroll
    for (int f = 0; f < FETCH; ++f) {
      const int i = threadIdx.x + f * THREADS;
      odd |= not_finite(piece[f].x) || not_finite(piece[f].y) || not_finite(piece[f].z) || not_finite(piece[f].w);
      if (KIND == MEMORY) {
        const int c = i % DV, d = i / DV * 4;
        ss[d * LDS + c] = piece[f].x;
        ss[(d + 1) * LDS + c] = piece[f].y;
        ss[(d + 2) * LDS + c] = piece[f].z;
        ss[(d + 3) * LDS + c] = piece[f].w;
      } else {
        *reinterpret_cast<float4*>(ss + i / (DV / 4) * LDS + i % (DV / 4) * 4) = piece[f];
      }
    }
    if (d0 + PIECE < a.dk) fetch(d0 + PIECE);
    odd = __syncthreads_or(odd) || bad;
    product_of<2, NT, 1, 3, false, TI>(acc, qt + d0 * LDT + wr, LDT, ss + col0, LDS, PIECE, as_is, odd, min(PIECE, a.dk - d0), 0);
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int r = wr + i * 16 + g + (e >> 1) * 8;
      const float w = (KIND == MEMORY ? carried[r] : power[r + 1]) * owed_q;
#pragma unroll
      for (int j = 0; j < NT; ++j) acc[i][j][e] *= w;
    }
  // values of the rows that a row sees (the others' weights are zeros)
  product_of<2, NT, 3, 1, true, TI>(acc, pt + wr, LDT, vs + col0, LDS, wr + 32, !act, wild, p.n, wr);

  Rows<TI, DV, false> gate;                 // (asked for now, wanted with the rows)
  if (KIND == RETENTION && a.finish && a.gate != nullptr) gate.ask((const TI*)a.gate + h * a.dv, a.ld_gate, p, a.dv);
  float factor[2][2];
  if (KIND == RETENTION && a.finish && a.unit_norm) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int e2 = 0; e2 < 2; ++e2) {
        float sq = 0.f;
#pragma unroll
        for (int j = 0; j < NT; ++j)        // (columns beyond dv are zeros)
          sq = fmaf(acc[i][j][e2 * 2], acc[i][j][e2 * 2], fmaf(acc[i][j][e2 * 2 + 1], acc[i][j][e2 * 2 + 1], sq));
        sq += __shfl_xor_sync(0xffffffffu, sq, 1);
        sq += __shfl_xor_sync(0xffffffffu, sq, 2);
        if (t2 == 0) sq_sum[wc][wr + i * 16 + g + e2 * 8] = sq;
      }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2) {
      const int r = wr + i * 16 + g + e2 * 8;
      factor[i][e2] = 1.f;
      if (KIND == MEMORY) factor[i][e2] = 1.f / (fmaxf(fabsf(den[4][r]), r < p.n ? expf(-(float)(F[r] + (double)mx[r])) : 1.f) + 1e-6f);
      if (KIND == RETENTION && a.finish && a.unit_norm)
        factor[i][e2] = 1.0f / sqrtf(((sq_sum[0][r] + sq_sum[1][r]) + (sq_sum[2][r] + sq_sum[3][r])) / (float)a.dv + a.eps);
    }
  // rows leave by way of shared memory, whole quads side by side (a thread's own entries are pairs)
  __syncthreads();                          // nobody reads queries, scores or pieces any more
  float* os = smem;                         // [C][LDS]
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int e2 = 0; e2 < 2; ++e2)
#pragma unroll
      for (int j = 0; j < NT; ++j)
        *reinterpret_cast<float2*>(os + (wr + i * 16 + g + e2 * 8) * LDS + col0 + j * 8 + t2) =
            make_float2(acc[i][j][e2 * 2] * factor[i][e2], acc[i][j][e2 * 2 + 1] * factor[i][e2]);
  __syncthreads();
#pragma unroll
  for (int f = 0; f < gate.N; ++f) {
    int r, c;
    gate.place(f, r, c);
    if (r >= p.n || c >= a.dv) continue;
    const int64_t row = p.row0 + r;
    const float4 x = *reinterpret_cast<const float4*>(os + r * LDS + c);
    if (KIND == RETENTION && a.finish) {
      float y[4] = {x.x, x.y, x.z, x.w};
      if (a.gate != nullptr) {
        const float4 g4 = widen(gate.raw[f]);
        const float gt[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) y[e] *= silu_f(gt[e]);
      }
      TI* o = (TI*)a.out + row * a.ld_out + h * a.dv + c;
      if (a.vec_out) {
        typename Quad<TI>::type w;
        TI* parts = reinterpret_cast<TI*>(&w);
#pragma unroll
        for (int e = 0; e < 4; ++e) parts[e] = from_f32<TI>(y[e]);
        *reinterpret_cast<typename Quad<TI>::type*>(o) = w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = from_f32<TI>(y[e]);
      }
    } else {
      *reinterpret_cast<float4*>(a.raw + row * a.ld_raw + h * a.dv + c) = x;
    }
  }
}

template <typename K>
int room(K kernel, size_t smem) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "chunked recurrence: cannot reserve %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
  return KVAD_OK;
}

template <int KIND, typename TI, int DK, int DV>
int launch(ChunkArgs a, int span, cudaStream_t stream) {
  constexpr size_t sum_smem = (size_t)C * (DK + DV + 8) * 4;
  constexpr int LDS = DV + 4, region = DK * LDT > C * LDT + 32 * LDS ? DK * LDT : C * LDT + 32 * LDS;
  constexpr size_t read_smem = ((size_t)DK * LDT + region + C * LDS) * 4;
  static_assert((size_t)C * LDS * 4 <= read_smem, "the rows leave through shared memory");
  static bool configured = false;
  if (!configured) {
    int rc = room(chunk_sum_kernel<KIND, TI, DK, DV>, sum_smem);
    if (rc == KVAD_OK) rc = room(chunk_read_kernel<KIND, TI, DK, DV>, read_smem);
    if (rc != KVAD_OK) return rc;
    configured = true;
  }
  const int entries = a.dk * a.dv;
  const int total = a.places;
  for (a.place0 = 0; a.place0 < total; a.place0 += span) {
    a.places = total - a.place0 < span ? total - a.place0 : span;
    kvad_launch(chunk_sum_kernel<KIND, TI, DK, DV>, dim3(a.places, a.heads), dim3(THREADS), sum_smem, stream, a);
    kvad_launch(chunk_scan_kernel<KIND>, dim3(a.n_seqs * a.heads, (entries / 4 + THREADS - 1) / THREADS), dim3(THREADS), 0, stream, a);
    if (KIND == MEMORY) kvad_launch(chunk_max_kernel, dim3(a.n_seqs), dim3(64), 0, stream, a);
    kvad_launch(chunk_read_kernel<KIND, TI, DK, DV>, dim3(a.places, a.heads), dim3(THREADS), read_smem, stream, a);
  }
  KVAD_CHECK_LAUNCH("chunked recurrence");
  return KVAD_OK;
}

template <int KIND, typename TI>
int dispatch(const ChunkArgs& a, int span, cudaStream_t stream) {
  if (a.dk <= 64) return a.dv <= 64 ? launch<KIND, TI, 64, 64>(a, span, stream) : launch<KIND, TI, 64, 128>(a, span, stream);
  return a.dv <= 64 ? launch<KIND, TI, 128, 64>(a, span, stream) : launch<KIND, TI, 128, 128>(a, span, stream);
}

int check(const ChunkArgs& a, int dtype, int n_rows, int span) {
  const uintptr_t unit = dtype == KVAD_DTYPE_F32 ? 15 : 7;
  KVAD_REQUIRE(a.n_seqs > 0 && a.heads > 0 && a.dk > 0 && a.dv > 0 && n_rows >= 0, "chunked recurrence: bad sizes seqs=%d heads=%d dk=%d dv=%d", a.n_seqs, a.heads, a.dk, a.dv);
  KVAD_REQUIRE(span > 0, "chunked recurrence: scratch for no chunk at all");
  KVAD_REQUIRE(a.state && a.seq_starts && a.seq_slots && a.work, "chunked recurrence: needs state, sequences and scratch");
  KVAD_REQUIRE(a.heads <= 65535 && (int64_t)a.n_seqs * a.heads < (1ll << 31), "chunked recurrence: %d sequences x %d heads are more than one launch takes", a.n_seqs, a.heads);
  if (a.dk > 128 || a.dv > 128 || a.dk % 4 || a.dv % 4 || a.ld_q % 4 || a.ld_k % 4 || a.ld_v % 4 ||
      ((reinterpret_cast<uintptr_t>(a.q) | reinterpret_cast<uintptr_t>(a.k) | reinterpret_cast<uintptr_t>(a.v)) & unit) ||
      ((reinterpret_cast<uintptr_t>(a.state) | reinterpret_cast<uintptr_t>(a.work) | reinterpret_cast<uintptr_t>(a.raw)) & 15) || a.state_stride % 4 || a.ld_raw % 4)
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "chunked recurrence: sizes of up to 128 entries a head, all in whole quads");
  return KVAD_OK;
}

}  // namespace

// Places of chunks that `n_rows` rows of `n_seqs` sequences may take.
KVAD_EXPORT int kvad_chunk_places(int n_rows, int n_seqs) { return n_rows / C + n_seqs; }

// Retention of prompt rows (see kvad_retention for the arguments).  `work`: float32 [span, heads, dk, dv] for `span` places at a time.  With `finish` the rows of `out` are
// written, else the 32-bit read-outs [rows, heads * dv] to `raw`.
KVAD_EXPORT int kvad_retention_chunked(int dtype, const void* q, int64_t ld_q, const void* k, int64_t ld_k, const void* v, int64_t ld_v, const void* gate,
                                       int64_t ld_gate, void* out, int64_t ld_out, float* raw, int n_rows, float* state, const int* seq_starts,
                                       const int* kv_lens, const int* seq_slots, const float* decay, const float* inv_freq, int rot_dims,
                                       int interleaved, int n_seqs, int heads, int dk, int dv, float k_scale, float eps, int unit_norm, int act,
                                       int finish, float* work, int span, int from, cudaStream_t stream) {
  ChunkArgs a = {};
  a.q = q; a.k = k; a.v = v; a.ld_q = ld_q; a.ld_k = ld_k; a.ld_v = ld_v; a.seq_starts = seq_starts; a.kv_lens = kv_lens; a.seq_slots = seq_slots;
  a.n_seqs = n_seqs; a.heads = heads; a.group = 1; a.dk = dk; a.dv = dv; a.places = kvad_chunk_places(n_rows, n_seqs); a.work = work;
  a.state = state; a.state_stride = (int64_t)heads * dk * dv; a.decay = decay; a.inv_freq = inv_freq; a.rot_dims = inv_freq != nullptr ? rot_dims : 0;
  a.interleaved = interleaved; a.act = act; a.k_scale = k_scale; a.q_scale = 1.f; a.raw = finish ? nullptr : raw; a.ld_raw = (int64_t)heads * dv;
  a.out = out; a.ld_out = ld_out; a.gate = gate; a.ld_gate = ld_gate; a.unit_norm = unit_norm; a.finish = finish; a.eps = eps;
  a.from = from;
  int rc = check(a, dtype, n_rows, span);
  if (rc != KVAD_OK) return rc;
  KVAD_REQUIRE(kv_lens && decay && (finish ? out != nullptr : raw != nullptr), "retention (chunked): bad arguments");
  KVAD_REQUIRE(rot_dims >= 0 && rot_dims % 2 == 0 && rot_dims <= dk, "retention (chunked): %d rotated entries of %d", rot_dims, dk);
  const uintptr_t unit = dtype == KVAD_DTYPE_F32 ? 15 : 7;
  if (gate != nullptr && (ld_gate % 4 || (reinterpret_cast<uintptr_t>(gate) & unit)))
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "retention (chunked): the gate comes in whole quads");
  a.vec_out = ld_out % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & unit) == 0 ? 1 : 0;
  if (dtype == KVAD_DTYPE_F32) return dispatch<RETENTION, float>(a, span, stream);
  if (dtype == KVAD_DTYPE_BF16) return dispatch<RETENTION, __nv_bfloat16>(a, span, stream);
  KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "retention (chunked): unknown dtype %d", dtype);
}

// The matrix memory over prompt rows (see kvad_gated_recurrence).  `work`: float32 [span, heads, dk * dv]; `work_n`: float32 span x heads x (dk + 3).
KVAD_EXPORT int kvad_matrix_memory_chunked(int dtype, const void* q, int64_t ld_q, const void* k, int64_t ld_k, const void* v, int64_t ld_v, const float* gates,
                                           int64_t ld_gates, float* out, int64_t ld_out, int n_rows, float* state, int64_t state_stride, const int* seq_starts,
                                           const int* seq_slots, int n_seqs, int heads, int kv_heads, int dk, int dv, float q_scale, float cap, float* work,
                                           float* work_n, int span, int from, cudaStream_t stream) {
  KVAD_REQUIRE(kv_heads > 0 && heads % kv_heads == 0 && gates && work_n && out, "matrix memory (chunked): bad arguments");
  ChunkArgs a = {};
  a.q = q; a.k = k; a.v = v; a.ld_q = ld_q; a.ld_k = ld_k; a.ld_v = ld_v; a.seq_starts = seq_starts; a.seq_slots = seq_slots;
  a.n_seqs = n_seqs; a.heads = heads; a.group = heads / kv_heads; a.dk = dk; a.dv = dv; a.places = kvad_chunk_places(n_rows, n_seqs); a.work = work;
  a.state = state; a.state_stride = state_stride; a.k_scale = 1.f; a.q_scale = q_scale; a.gates = gates; a.ld_gates = ld_gates; a.cap = cap;
  a.work_n = work_n; a.work_m = work_n + (int64_t)span * heads * (dk + 2); a.tiles = (dv + 15) / 16; a.raw = out; a.ld_raw = ld_out;
  a.from = from;
  int rc = check(a, dtype, n_rows, span);
  if (rc != KVAD_OK) return rc;
  if (dtype == KVAD_DTYPE_F32) return dispatch<MEMORY, float>(a, span, stream);
  if (dtype == KVAD_DTYPE_BF16) return dispatch<MEMORY, __nv_bfloat16>(a, span, stream);
  KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "matrix memory (chunked): unknown dtype %d", dtype);
}

KVAD_DEFINE_LAST_ERROR()
