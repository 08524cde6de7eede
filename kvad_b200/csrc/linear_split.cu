// out[M,N] = epilogue(A[M,K] . W[N,K]^T + bias) of 32-bit operands on the 5th-generation tensor cores, without giving up
// 32-bit accuracy: the float32 engine's products of many rows and short K, and its head-wise maps (longer K: linear_pieces.cu, which cuts the weights once a product).
//
// Every operand x is cut into three bfloat16 pieces by truncation, x = h + m + l exactly (24 bits of significand = 3 x 8), and
//   a.w = h_a h_w + (h_a m_w + m_a h_w) + (h_a l_w + m_a m_w + l_a h_w)       (what is left out is below 2^-24 of |a||w|)
// are six bfloat16 products with 32-bit accumulation.  (Exactly while x is above about 2^-110: below, the last places of l fall under bfloat16's smallest number,
// 2^-133, and are left out.)  The tensor core accumulates by TRUNCATING (measured: a product of
// K = 768 is off by 7e-7 of its norm when summed in one accumulator, the CUDA cores' fmaf chain by 2.1e-7), so a sum stays in
// tensor memory for 32 of K only - small products first, so that only the two steps of h_a h_w meet the full magnitude - and
// then goes into 32-bit registers by ordinary rounded additions: off by 1.4e-7 at K = 768, less than the fmaf chain.
//
// A CTA walks tiles of 128 rows x BN outputs, 32 of K at a time.  Sixteen worker warps bring the block of A and W into
// registers (the next two blocks' loads are in flight while this one is worked), cut it up and write the pieces into shared
// memory in the layout the tensor core reads (K-major, 128-byte swizzle; a block is half of such a row); one thread issues the 12
// MMAs of the block.  Four slots of shared memory, each with an accumulator of its own, go round: the MMAs run up to three blocks
// behind the cutting, and the workers collect an accumulator right before they reuse its slot.  An output's sum depends on K
// only: the same bits whatever its company and its tile.
//
// An operand that is not finite makes the pieces' differences NaN; an output that comes out NaN is summed again with
// fmaf from the operands themselves (k = 0..K-1), so infinities and NaN give what 32-bit arithmetic gives.
#include "common.cuh"
#include "tcgen05.cuh"

using namespace kvad;

namespace {

constexpr int BM = 128, BK = 32, SLOTS = 4, WORKERS = 512, THREADS = WORKERS + 32;

// A piece of two neighbouring slots is one tile of 128-byte rows: slot 2i has the first 64 bytes of each, slot 2i + 1 the others.
template <int BN> struct SplitTile {
  static constexpr uint32_t A_PIECE = BM * 128, W_PIECE = BN * 128;
  static constexpr uint32_t PAIR = 3 * (A_PIECE + W_PIECE);
  static constexpr uint32_t TMEM_COLS = SLOTS * BN;
  static constexpr size_t SMEM = (SLOTS / 2) * (size_t)PAIR + 2 * SLOTS * 8 + 16 + 1024;
};

// Four neighbours along K as three rows of four bfloat16 pieces each (x = h + m + l exactly, by truncation).
__device__ __forceinline__ void cut4(const float4& x, uint2& h, uint2& m, uint2& l) {
  const float v[4] = {x.x, x.y, x.z, x.w};
  uint32_t hb[4], mb[4], lb[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    hb[i] = __float_as_uint(v[i]);
    const float r1 = v[i] - __uint_as_float(hb[i] & 0xffff0000u);
    mb[i] = __float_as_uint(r1);
    lb[i] = __float_as_uint(r1 - __uint_as_float(mb[i] & 0xffff0000u));
  }
  h = make_uint2(__byte_perm(hb[0], hb[1], 0x7632), __byte_perm(hb[2], hb[3], 0x7632));
  m = make_uint2(__byte_perm(mb[0], mb[1], 0x7632), __byte_perm(mb[2], mb[3], 0x7632));
  l = make_uint2(__byte_perm(lb[0], lb[1], 0x7632), __byte_perm(lb[2], lb[3], 0x7632));
}

struct SplitArgs {
  const float* A; int64_t lda;
  const float* W;
  const void* bias; int bias_f32;
  float* out; int64_t ldo;
  int M, N, K, vec_out;
  int heads; int64_t a_head, out_head;      // `heads` products side by side: head z reads A from column z * a_head, its own [N, K] of W, and writes from column z * out_head
};

__device__ __noinline__ float plain_dot(const float* a, const float* w, int K) {
  float s = 0.f;
  for (int k = 0; k < K; ++k) s = fmaf(a[k], w[k], s);
  return s;
}

template <int BN, int EPI>
__global__ void __launch_bounds__(THREADS, 1) linear_split_kernel(const SplitArgs p) {
  using T = SplitTile<BN>;
  constexpr int QR = BK / 4, RQ = WORKERS / QR;                      // lanes that share a row's block, rows that the workers take at a time
  constexpr int AQ = BM / RQ, WQ = BN / RQ;      // quads of 4 along K that a worker brings of a block
  constexpr int SHARE = BN / (WORKERS / 128);                        // the warps that share a quarter of the accumulator's lanes take a share of its columns each
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + SLOTS / 2 * T::PAIR);   // [SLOTS] the workers have written a slot and emptied its accumulator
  uint64_t* done_bar = full_bar + SLOTS;                                      // [SLOTS] the block's MMAs have run
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + SLOTS);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  pdl_launch_dependents();
  if (tid == 0) {
    for (int s = 0; s < SLOTS; ++s) {
      mbar_init(&full_bar[s], WORKERS / 32);
      mbar_init(&done_bar[s], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == WORKERS / 32) tmem_alloc(tmem_slot, T::TMEM_COLS);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  const int tiles_n = (p.N + BN - 1) / BN, tiles_mn = tiles_n * ((p.M + BM - 1) / BM), tiles = tiles_mn * p.heads, num_kb = (p.K + BK - 1) / BK;
  const int mine = (int)blockIdx.x < tiles ? (tiles - (int)blockIdx.x - 1) / (int)gridDim.x + 1 : 0;   // tiles of this CTA
  const int blocks = mine * num_kb;

  if (warp == WORKERS / 32) {
    if (lane == 0) {
      constexpr uint32_t idesc = umma_instr_desc(BM, BN);
      for (int j = 0; j < blocks; ++j) {
        const int s = j % SLOTS;
        if (!mbar_wait(&full_bar[s], (j / SLOTS) & 1)) break;
        tc_fence_after();
        const uint32_t base = smem_u32(smem + (s >> 1) * T::PAIR), acc = tmem_base + (uint32_t)(s * BN);
        uint64_t a[3], w[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          a[i] = sw128_desc(base + i * T::A_PIECE) + (uint64_t)((s & 1) * 4);      // (32 entries: 64 bytes further along the rows)
          w[i] = sw128_desc(base + 3 * T::A_PIECE + i * T::W_PIECE) + (uint64_t)((s & 1) * 4);
        }
        constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PW[6] = {0, 2, 1, 0, 1, 0};      // the smallest products first
#pragma unroll
        for (int t = 0; t < 6; ++t)
#pragma unroll
          for (int k = 0; k < BK / 16; ++k)
            umma(acc, a[PA[t]] + (uint64_t)(k * 2), w[PW[t]] + (uint64_t)(k * 2), idesc, (t > 0 || k > 0) ? 1u : 0u);
        umma_commit(&done_bar[s]);
      }
    }
  } else {
    const int quarter = warp & 3, share = warp >> 2;
    float4 ra[2][AQ], rw[2][WQ];                                     // the next two blocks
    float acc[SHARE];
#pragma unroll
    for (int i = 0; i < SHARE; ++i) acc[i] = 0.f;
    auto corner = [&](int t, int* m0, int* n0, int* z) {
      const int g = (int)blockIdx.x + t * (int)gridDim.x;
      *z = g / tiles_mn;
      const int in_head = g - *z * tiles_mn;
      *n0 = (in_head % tiles_n) * BN;
      *m0 = (in_head / tiles_n) * BM;
    };
    // where this worker's quads of a block come from: 8 lanes take a row's 32 of K, 128 bytes side by side.  The block is kept
    // by counting (divisions cost as much as the cutting); rows and K that do not exist are zeros.
    const int row_of = tid / QR, quad_of = tid % QR;
    const float *a_at = nullptr, *w_at = nullptr;
    const int64_t a_step = (int64_t)RQ * p.lda, w_step = (int64_t)RQ * p.K;
    int a_left = 0, w_left = 0, load_t = 0, load_kb = 0, whole = 0;
    auto fetch = [&](float4* fa, float4* fw) {
      if (load_t >= mine) return;
      if (load_kb == 0) {
        int m0, n0, z;
        corner(load_t, &m0, &n0, &z);
        a_at = p.A + (int64_t)(m0 + row_of) * p.lda + z * p.a_head + quad_of * 4;
        w_at = p.W + ((int64_t)z * p.N + n0 + row_of) * p.K + quad_of * 4;
        a_left = p.M - m0 - row_of;
        w_left = p.N - n0 - row_of;
        whole = m0 + BM <= p.M && n0 + BN <= p.N;
      }
      if (whole && (load_kb + 1) * BK <= p.K) {                      // (the same for all workers)
#pragma unroll
        for (int i = 0; i < AQ; ++i) fa[i] = *reinterpret_cast<const float4*>(a_at + i * a_step);
#pragma unroll
        for (int i = 0; i < WQ; ++i) fw[i] = *reinterpret_cast<const float4*>(w_at + i * w_step);
      } else {
        const bool in_k = load_kb * BK + quad_of * 4 < p.K;          // (K is a multiple of 4)
#pragma unroll
        for (int i = 0; i < AQ; ++i)
          fa[i] = in_k && i * RQ < a_left ? *reinterpret_cast<const float4*>(a_at + i * a_step) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < WQ; ++i)
          fw[i] = in_k && i * RQ < w_left ? *reinterpret_cast<const float4*>(w_at + i * w_step) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
      a_at += BK;
      w_at += BK;
      if (++load_kb == num_kb) {
        load_kb = 0;
        ++load_t;
      }
    };
    // (rows RQ = 64 apart have the same place in the swizzle)
    const uint32_t put_row = row_of * 128, put_x = row_of & 7;
    auto put = [&](uint8_t* piece0, uint32_t piece_bytes, int r, uint32_t half, const float4& x) {
      uint2 h, m, l;
      cut4(x, h, m, l);
      uint8_t* at = piece0 + put_row + r * 128 + (((half * 4 + (quad_of >> 1)) ^ put_x) << 4) + ((quad_of & 1) << 3);
      *reinterpret_cast<uint2*>(at) = h;
      *reinterpret_cast<uint2*>(at + piece_bytes) = m;
      *reinterpret_cast<uint2*>(at + 2 * piece_bytes) = l;
    };
    auto outcome = [&](float x, int col) {
      if (p.bias != nullptr) x += load_param(p.bias, col, p.bias_f32);
      if (EPI == EPI_GELU_TANH) x = gelu_tanh(x);
      if (EPI == EPI_GELU_ERF) x = gelu_erf(x);
      return x;
    };
    auto finish = [&](int t) {                                       // the tile's sums leave the registers
      int m0, n0, z;
      corner(t, &m0, &n0, &z);
      const int row = m0 + quarter * 32 + lane, col0 = n0 + share * SHARE;
      uint32_t again = 0;                                            // columns whose sum came out NaN
      if (row < p.M) {
        float* o = p.out + (int64_t)row * p.ldo + z * p.out_head + col0;
#pragma unroll
        for (int c = 0; c < SHARE; c += 4) {
          float x[4];
          uint32_t bad = 0;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            x[e] = acc[c + e];
            if (x[e] != x[e]) bad |= 1u << e;
            if (col0 + c + e < p.N) x[e] = outcome(x[e], col0 + c + e);
            else bad |= 1u << e;
          }
          if (p.vec_out && bad == 0) {
            float4 y = make_float4(x[0], x[1], x[2], x[3]);
            if (EPI == EPI_RESIDUAL) {
              const float4 old = *reinterpret_cast<const float4*>(o + c);
              y.x += old.x; y.y += old.y; y.z += old.z; y.w += old.w;
            }
            *reinterpret_cast<float4*>(o + c) = y;
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (!(bad >> e & 1)) o[c + e] = EPI == EPI_RESIDUAL ? o[c + e] + x[e] : x[e];
            again |= bad << c;
          }
        }
      }
#pragma unroll
      for (int i = 0; i < SHARE; ++i) acc[i] = 0.f;
      while (again) {
        const int c = __ffs((int)again) - 1, col = col0 + c;
        again &= again - 1;
        if (col >= p.N) break;
        const float x = outcome(plain_dot(p.A + (int64_t)row * p.lda + z * p.a_head, p.W + ((int64_t)z * p.N + col) * p.K, p.K), col);
        float* o = p.out + (int64_t)row * p.ldo + z * p.out_head + col;
        *o = EPI == EPI_RESIDUAL ? *o + x : x;
      }
    };
    int got_t = 0, got_kb = 0;                                       // the block that is collected next
    auto collect = [&](int j) -> bool {                              // block j's sums join the registers, rounded
      const int s = j % SLOTS;
      if (!mbar_wait(&done_bar[s], (j / SLOTS) & 1)) return false;
      tc_fence_after();
      const uint32_t at = tmem_base + (uint32_t)(s * BN + share * SHARE) + ((uint32_t)(quarter * 32) << 16);
#pragma unroll
      for (int c = 0; c < SHARE; c += 16) {
        float v[16];
        tmem_ld16(at + (uint32_t)c, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[c + i] += v[i];
      }
      tc_fence_before();
      if (++got_kb == num_kb) {
        got_kb = 0;
        finish(got_t++);
      }
      return true;
    };
    pdl_wait();
    bool ok = true;
    fetch(ra[0], rw[0]);
    fetch(ra[1], rw[1]);
    for (int j0 = 0; j0 < blocks && ok; j0 += 2) {
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int j = j0 + u;
        if (j >= blocks || !ok) break;
        if (j >= SLOTS && !(ok = collect(j - SLOTS))) break;
        uint8_t* pair = smem + (j % SLOTS / 2) * T::PAIR;
#pragma unroll
        for (int i = 0; i < AQ; ++i) put(pair, T::A_PIECE, i * RQ, u, ra[u][i]);
#pragma unroll
        for (int i = 0; i < WQ; ++i) put(pair + 3 * T::A_PIECE, T::W_PIECE, i * RQ, u, rw[u][i]);
        fetch(ra[u], rw[u]);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0) mbar_arrive_one(&full_bar[j % SLOTS]);       // (one arrival a warp)
      }
    }
    for (int j = blocks > SLOTS ? blocks - SLOTS : 0; j < blocks && ok; ++j) ok = collect(j);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == WORKERS / 32) {
    __syncwarp();
    tmem_dealloc(tmem_base, T::TMEM_COLS);
  }
}

int sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
  }
  return n;
}

template <int BN, int EPI>
int launch_split(const SplitArgs& a, cudaStream_t stream) {
  using T = SplitTile<BN>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(linear_split_kernel<BN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM);
    if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "linear_split: cannot reserve %zu bytes of shared memory: %s", T::SMEM, cudaGetErrorString(e));
    configured = true;
  }
  const int64_t tiles = (int64_t)((a.N + BN - 1) / BN) * ((a.M + BM - 1) / BM) * a.heads;
  KVAD_REQUIRE(tiles * ((a.K + BK - 1) / BK) < (1ll << 30), "linear_split: %lld tiles are more than one launch takes", (long long)tiles);
  const int ctas = tiles < sm_count() ? (int)tiles : sm_count();
  kvad_launch(linear_split_kernel<BN, EPI>, dim3(ctas), dim3(THREADS), T::SMEM, stream, a);
  KVAD_CHECK_LAUNCH("linear_split");
  return KVAD_OK;
}

template <int BN>
int launch_epi(int epilogue, const SplitArgs& a, cudaStream_t stream) {
  switch (epilogue) {
    case EPI_STORE:
    case EPI_STORE_F32: return launch_split<BN, EPI_STORE>(a, stream);
    case EPI_GELU_TANH: return launch_split<BN, EPI_GELU_TANH>(a, stream);
    case EPI_GELU_ERF: return launch_split<BN, EPI_GELU_ERF>(a, stream);
    case EPI_RESIDUAL: return launch_split<BN, EPI_RESIDUAL>(a, stream);
  }
  KVAD_FAIL(KVAD_ERR_ARGUMENT, "linear_split: unknown epilogue %d", epilogue);
}

int split(const float* A, int64_t lda, const float* W, const void* bias, int bias_f32, float* out, int64_t ldo, int M, int N, int K, int epilogue,
          int force_bn, int heads, int64_t a_head, int64_t out_head, cudaStream_t stream) {
  KVAD_REQUIRE(M >= 0 && N > 0 && K > 0, "linear_split: bad sizes M=%d N=%d K=%d", M, N, K);
  if (K % 4 != 0 || lda % 4 != 0 || a_head % 4 != 0 || (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(W) & 15))
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "linear_split: K and the strides must be multiples of 4, the operands on 16-byte boundaries");
  KVAD_REQUIRE(force_bn == 0 || force_bn == 64 || force_bn == 128, "linear_split: tile width %d is not 64 or 128", force_bn);
  if (M == 0) return KVAD_OK;
  SplitArgs a;
  a.A = A; a.lda = lda; a.W = W; a.bias = bias; a.bias_f32 = bias_f32; a.out = out; a.ldo = ldo; a.M = M; a.N = N; a.K = K;
  a.heads = heads; a.a_head = a_head; a.out_head = out_head;
  a.vec_out = (ldo % 4 == 0 && out_head % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) ? 1 : 0;
  int bn = force_bn;
  if (bn == 0) {
    const int64_t rows = (int64_t)((M + BM - 1) / BM) * heads, sms = sm_count();
    const int64_t w128 = (rows * ((N + 127) / 128) + sms - 1) / sms, w64 = (rows * ((N + 63) / 64) + sms - 1) / sms;
    bn = (float)w64 * 0.62f < (float)w128 ? 64 : 128;
  }
  return bn == 64 ? launch_epi<64>(epilogue, a, stream) : launch_epi<128>(epilogue, a, stream);
}

}  // namespace

// `force_bn`: 0, or the tile width (64 or 128).
KVAD_EXPORT int kvad_linear_split(const float* A, int64_t lda, const float* W, const void* bias, int bias_f32, float* out, int64_t ldo,
                                  int M, int N, int K, int epilogue, int force_bn, cudaStream_t stream) {
  KVAD_REQUIRE(lda >= K && ldo >= N, "linear_split: leading dimensions lda=%lld ldo=%lld too small", (long long)lda, (long long)ldo);
  return split(A, lda, W, bias, bias_f32, out, ldo, M, N, K, epilogue, force_bn, 1, 0, 0, stream);
}

// out[r, z * out_head + j] = W[z, j, :] . A[r, z * a_head : + K] for every head z, in one launch.
KVAD_EXPORT int kvad_linear_split_heads(const float* A, int64_t lda, int64_t a_head, const float* W, float* out, int64_t ldo, int64_t out_head,
                                        int M, int heads, int N, int K, cudaStream_t stream) {
  KVAD_REQUIRE(heads > 0 && lda >= (heads - 1) * a_head + K && ldo >= (heads - 1) * out_head + N, "linear_split_heads: the heads do not fit the rows");
  return split(A, lda, W, nullptr, 0, out, ldo, M, N, K, EPI_STORE, 0, heads, a_head, out_head, stream);
}

// How many bounded waits have run out since the library was loaded (0 in a healthy run).  Synchronises the device.
KVAD_EXPORT int kvad_linear_split_status() {
  int n = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&n, g_wait_timeouts, sizeof(int));
  if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "linear_split_status: %s", cudaGetErrorString(e));
  return n;
}

KVAD_DEFINE_LAST_ERROR()
