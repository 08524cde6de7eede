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
// All of it is 32-bit arithmetic on the CUDA cores (fmaf chains of 32 to 64 terms; 0.8 G multiply-adds for 2 x 1024 rows of 8
// heads of 128 x 128, 22 us at their peak).  Decays are powers of the head's constant (retention), or exponentials of
// differences of logarithms that are summed up in 64 bits within the chunk (matrix memory), so that a difference of two large sums
// keeps its last places.  The matrix memory's running maximum goes along: a chunk's own maximum at its end, the maximum carried over
// the chunks in step 2, and per row m_i = F_i + max(m_c, max_(j <= i) (i_j - F_j)); every weight is at most 1.
//
// Measured: 2 x 1024 rows of 8 heads of 128 x 128 (rotated, normed, gated, bfloat16) 387 -> 85 us; the matrix memory over 1000 + 517 + 37 rows of 8
// heads of 64 x 128 334 -> 50 us.  (92 and 53 before the state came a piece ahead by way of registers and rows by whole sectors.)
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
  void* out; int64_t ld_out; const void* gate; int64_t ld_gate; int unit_norm, finish;
  float eps;
};

// Four neighbouring entries of a row as floats.
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
  const uint2 raw = *reinterpret_cast<const uint2*>(p);
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x)), b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
  return make_float4(a.x, a.y, b.x, b.y);
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

// A chunk's rows of one head into shared memory, `width_to` entries wide: transposed [entry][row] or plain [row][entry]; entries and rows that
// do not exist are zeros.
template <typename TI, bool TRANSPOSED>
__device__ __forceinline__ void bring(float* dst, int ld, const TI* src, int64_t ld_src, const Place& p, int width, int width_to, bool act, float scale_from, int scaled_from) {
  const int quads = width_to / 4;
#pragma unroll 4
  for (int i = threadIdx.x; i < C * quads; i += THREADS) {
    // transposed: a warp takes 8 rows by 4 neighbouring quads (whole 32-byte sectors of bfloat16, and stores that meet a bank twice)
    const int r = TRANSPOSED ? (i & 7) + (i >> 5) % (C / 8) * 8 : i / quads, c = (TRANSPOSED ? ((i >> 3) & 3) + (i >> 5) / (C / 8) * 4 : i % quads) * 4;
    float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
    if (r < p.n && c < width) x = load4(src + (int64_t)(p.row0 + r) * ld_src + c);
    float v[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (act) v[e] = silu_f(v[e]);
      if (c + e >= scaled_from) v[e] *= scale_from;
      if (TRANSPOSED) dst[(c + e) * ld + r] = v[e];
    }
    if (!TRANSPOSED) *reinterpret_cast<float4*>(dst + r * ld + c) = make_float4(v[0], v[1], v[2], v[3]);
  }
}

// Pairs of q (or null) and k turned by the rows' positions where they lie, k scaled after turning.
template <bool TRANSPOSED>
__device__ __forceinline__ void turn(const ChunkArgs& a, const Place& p, float* q, float* k, int ld) {
  const int half = a.rot_dims / 2;
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

// acc[i][j] += sum over n of A[n][rows] B[n][cols], both read in quads; a thread's rows are ty * 4 .. + 3 (and the same 64 further), its columns likewise.
template <int TR, int TC>
__device__ __forceinline__ void outer(float (&acc)[TR][TC], const float* A, int lda, const float* B, int ldb, int n, int ty, int tx) {
#pragma unroll 4
  for (int t = 0; t < n; ++t) {
    float x[TR], y[TC];
#pragma unroll
    for (int g = 0; g < TR; g += 4) *reinterpret_cast<float4*>(x + g) = *reinterpret_cast<const float4*>(A + t * lda + ty * 4 + g * 16);
#pragma unroll
    for (int g = 0; g < TC; g += 4) *reinterpret_cast<float4*>(y + g) = *reinterpret_cast<const float4*>(B + t * ldb + tx * 4 + g * 16);
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j) acc[i][j] = fmaf(x[i], y[j], acc[i][j]);
  }
}

// ---- 1: what a chunk leaves in the state ---------------------------------------------------------------------------------
template <int KIND, typename TI, int DK, int DV>
__global__ void __launch_bounds__(THREADS) chunk_sum_kernel(const ChunkArgs a) {
  extern __shared__ float smem[];
  float* ks = smem;                         // [C][DK]
  float* vs = ks + C * DK;                  // [C][DV]
  __shared__ double F[KIND == MEMORY ? C : 1];
  __shared__ float in[C], best[C], weight[C], scratch;
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.y, qh = h / a.group;
  const Place p = find(a, a.place0 + blockIdx.x);
  if (p.n == 0) return;
  const bool half = KIND == RETENTION && a.rot_dims > 0;
  bring<TI, false>(ks, DK, (const TI*)a.k + qh * a.dk, a.ld_k, p, a.dk, DK, KIND == RETENTION && a.act, a.k_scale, a.rot_dims);
  bring<TI, false>(vs, DV, (const TI*)a.v + h * a.dv, a.ld_v, p, a.dv, DV, KIND == RETENTION && a.act, 1.f, DV);
  if (KIND == MEMORY) {
    chunk_gates(a, p, h, F, in, best, &scratch);
    if (threadIdx.x < C) {                  // weights at the chunk's end, against its own maximum there
      const int t = threadIdx.x;
      weight[t] = t < p.n ? expf((float)((double)in[t] - F[t] - (double)best[p.n - 1])) : 0.f;
    }
  } else {
    if (half) {
      __syncthreads();
      turn<false>(a, p, nullptr, ks, DK);
    }
    if (threadIdx.x < C) weight[threadIdx.x] = powf(a.decay[h], (float)max(0, p.n - 1 - (int)threadIdx.x));
  }
  __syncthreads();
  for (int i = threadIdx.x; i < C * DK; i += THREADS) ks[i] *= weight[i / DK];
  __syncthreads();
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  // (entries in the state's own order: retention [dk][dv], the matrix memory [dv][dk])
  constexpr int TR = (KIND == MEMORY ? DV : DK) / 16, TC = (KIND == MEMORY ? DK : DV) / 16;
  float acc[TR][TC];
#pragma unroll
  for (int i = 0; i < TR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j) acc[i][j] = 0.f;
  if (KIND == MEMORY) outer<TR, TC>(acc, vs, DV, ks, DK, p.n, ty, tx);
  else outer<TR, TC>(acc, ks, DK, vs, DV, p.n, ty, tx);
  const int rows = KIND == MEMORY ? a.dv : a.dk, cols = KIND == MEMORY ? a.dk : a.dv;
  float* u = a.work + ((int64_t)blockIdx.x * a.heads + h) * a.dk * a.dv;
#pragma unroll
  for (int i = 0; i < TR; ++i) {
    const int r = ty * 4 + (i & 3) + (i >> 2) * 64;
    if (r >= rows) continue;
#pragma unroll
    for (int j = 0; j < TC; j += 4) {
      const int c = tx * 4 + (j >> 2) * 64;
      if (c < cols) *reinterpret_cast<float4*>(u + r * cols + c) = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
    }
  }
  if (KIND == MEMORY) {
    float* un = a.work_n + ((int64_t)blockIdx.x * a.heads + h) * (a.dk + 2);
    for (int d = threadIdx.x; d < a.dk; d += THREADS) {
      float sum = 0.f;
      for (int t = 0; t < p.n; ++t) sum += ks[t * DK + d];
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
template <int KIND, typename TI, int DK, int DV>
__global__ void __launch_bounds__(THREADS, 2) chunk_read_kernel(const ChunkArgs a) {
  constexpr int PIECE = 32, LDS = DV + 4;                               // rows of the state that come at a time
  constexpr int REGION = DK * LDT > C * LDT + PIECE * LDS ? DK * LDT : C * LDT + PIECE * LDS;
  extern __shared__ float smem[];
  float* qt = smem;                         // [DK][LDT]
  float* kt = qt + DK * LDT;                // [DK][LDT], later the weighted scores [j][i] and a piece of the state
  float* vs = kt + REGION;                  // [C][DV]
  float* pt = kt;
  float* ss = kt + C * LDT;
  __shared__ double F[KIND == MEMORY ? C : 1];
  __shared__ float in[C], best[C], power[C + 1], carried[C], den[4][C], scratch, mx[C];
  pdl_launch_dependents();
  pdl_wait();
  const int h = blockIdx.y, qh = h / a.group;
  const Place p = find(a, a.place0 + blockIdx.x);
  if (p.n == 0) return;
  const bool act = KIND == RETENTION && a.act;
  bring<TI, true>(qt, LDT, (const TI*)a.q + qh * a.dk, a.ld_q, p, a.dk, DK, act, a.q_scale, 0);
  bring<TI, true>(kt, LDT, (const TI*)a.k + qh * a.dk, a.ld_k, p, a.dk, DK, act, a.k_scale, a.rot_dims);
  bring<TI, false>(vs, DV, (const TI*)a.v + h * a.dv, a.ld_v, p, a.dv, DV, act, 1.f, DV);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
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
  __syncthreads();

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

  float sc[4][4] = {};
#pragma unroll 1
  for (int d0 = 0; d0 < DK; d0 += PIECE) {              // (sums of 32 terms, added up: less rounding than one chain of 128)
    float part[4][4] = {};
    outer<4, 4>(part, qt + d0 * LDT, LDT, kt + d0 * LDT, LDT, PIECE, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) sc[i][j] += part[i][j];
  }
  // weights; the matrix memory's sums of a row's weighted scores meet over its 16 threads
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    float sum = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int c = tx * 4 + j;
      // (a row that is not seen counts for nothing, also where its score is no number)
      if (c <= r && r < p.n) sc[i][j] *= KIND == MEMORY ? expf((float)((double)in[c] - F[c] - (double)mx[r])) : power[r - c];
      else sc[i][j] = 0.f;
      sum += sc[i][j];
    }
    if (KIND == MEMORY) {
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (tx == 0) den[0][r] = sum;
    }
  }
  if (KIND == MEMORY) {                     // ... and the normaliser before the chunk along the row's query
    const float* n_c = a.work_n + ((int64_t)blockIdx.x * a.heads + h) * (a.dk + 2);
    const int r = threadIdx.x & (C - 1), part = threadIdx.x / C;
    float sum = 0.f;
    for (int d = part; d < a.dk; d += 4) sum = fmaf(qt[d * LDT + r], n_c[d], sum);
    __syncthreads();
    if (part > 0) den[part][r] = sum;
    __syncthreads();
    if (part == 0) den[0][r] = fmaf(carried[r], (sum + den[1][r]) + (den[2][r] + den[3][r]), den[0][r]);
  }
  __syncthreads();                          // the keys have been used up
#pragma unroll
  for (int j = 0; j < 4; ++j) *reinterpret_cast<float4*>(pt + (tx * 4 + j) * LDT + ty * 4) = make_float4(sc[0][j], sc[1][j], sc[2][j], sc[3][j]);

  constexpr int TC = DV / 16;
  float acc[4][TC] = {};
  for (int d0 = 0; d0 < a.dk; d0 += PIECE) {
    const int nd = min(PIECE, a.dk - d0);
    if (d0 > 0) __syncthreads();
#pragma unroll
    for (int f = 0; f < FETCH; ++f) {
      const int i = threadIdx.x + f * THREADS;
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
    __syncthreads();
    float part[4][TC] = {};
    outer<4, TC>(part, qt + d0 * LDT, LDT, ss, LDS, nd, ty, tx);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j) acc[i][j] += part[i][j];
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float w = KIND == MEMORY ? carried[ty * 4 + i] : power[ty * 4 + i + 1];
#pragma unroll
    for (int j = 0; j < TC; ++j) acc[i][j] *= w;
  }
  // values of the rows that a row sees, and no others: a zero weight would make NaN of a value that is not finite
  outer<4, TC>(acc, pt, LDT, vs, DV, min(p.n, ty * 4), ty, tx);
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const int t = ty * 4 + e;
    if (t >= p.n) break;
    float y[TC];
#pragma unroll
    for (int g = 0; g < TC; g += 4) *reinterpret_cast<float4*>(y + g) = *reinterpret_cast<const float4*>(vs + t * DV + tx * 4 + g * 16);
#pragma unroll
    for (int i = e; i < 4; ++i) {
      const float x = pt[t * LDT + ty * 4 + i];
#pragma unroll
      for (int j = 0; j < TC; ++j) acc[i][j] = fmaf(x, y[j], acc[i][j]);
    }
  }

#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = ty * 4 + i;
    float factor = 1.f;
    if (KIND == MEMORY) factor = 1.f / (fmaxf(fabsf(den[0][r]), r < p.n ? expf(-(float)(F[r] + (double)mx[r])) : 1.f) + 1e-6f);
    if (KIND == RETENTION && a.finish && a.unit_norm) {
      float sq = 0.f;
#pragma unroll
      for (int j = 0; j < TC; ++j) sq = fmaf(acc[i][j], acc[i][j], sq);      // (columns beyond dv are zeros)
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
      factor = 1.0f / sqrtf(sq / (float)a.dv + a.eps);
    }
    if (r >= p.n) continue;
    const int64_t row = p.row0 + r;
#pragma unroll
    for (int j = 0; j < TC; j += 4) {
      const int c = tx * 4 + (j >> 2) * 64;
      if (c >= a.dv) continue;
      float y[4];
#pragma unroll
      for (int e = 0; e < 4; ++e) y[e] = acc[i][j + e] * factor;
      if (KIND == RETENTION && a.finish) {
        if (a.gate != nullptr) {
          const float4 g4 = load4((const TI*)a.gate + row * a.ld_gate + h * a.dv + c);
          const float g[4] = {g4.x, g4.y, g4.z, g4.w};
#pragma unroll
          for (int e = 0; e < 4; ++e) y[e] *= g[e] / (1.0f + expf(-g[e]));
        }
        TI* o = (TI*)a.out + row * a.ld_out + h * a.dv + c;
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] = from_f32<TI>(y[e]);
      } else {
        *reinterpret_cast<float4*>(a.raw + row * a.ld_raw + h * a.dv + c) = make_float4(y[0], y[1], y[2], y[3]);
      }
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
  constexpr size_t sum_smem = (size_t)C * (DK + DV) * 4;
  constexpr int LDS = DV + 4, region = DK * LDT > C * LDT + 32 * LDS ? DK * LDT : C * LDT + 32 * LDS;
  constexpr size_t read_smem = ((size_t)DK * LDT + region + C * DV) * 4;
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
