// out[M,N] = epilogue(A[M,K] . W[N,K]^T + bias) of 32-bit operands on the 5th-generation tensor cores, for many rows: the same six products of bfloat16
// pieces as `linear_split.cu` (x = h + m + l exactly; a.w = hh + hm + mh + hl + mm + lh), in the same order, 32 of K at a time, so the same bits.
//
// There every tile cuts both operands, and the sixteen warps that cut (3400 cycles per 64 of K) are slower than the products (1536 at 128 outputs).
// What bounds the products themselves is shared memory: six products read a piece of A and one of W each, 128 bytes a cycle.  Here
//   - one pass writes the pieces of W to scratch in the very order that the tensor core reads: [tile of outputs][32 of K][piece][output], 64-byte
//     swizzle, zeros where they end; a block comes by one bulk copy;
//   - eight warps bring A's rows from global memory into registers, cut them and put them into TENSOR memory, the products' first operand, so that of shared
//     memory only W's side is left (576 cycles of 768 at 128 outputs);
//   - a converged warp issues the twelve products of a block into one of ACC accumulators, eight warps add each accumulator to their 32-bit registers by
//     rounded additions (the tensor core truncates where it accumulates).
// Tiles are 128 rows by 64, 128 or 192 outputs, whichever gives the fewest cycles in waves of one tile an SM.
//
// Outputs that are no number (an infinity has no pieces) are summed again with fmaf from the operands themselves.  Every wait is bounded.
#include "common.cuh"
#include "tcgen05.cuh"

using namespace kvad;

namespace {

constexpr int BM = 128, BK = 32, THREADS = 640, A_COLS = 48;      // A_COLS: tensor-memory columns of a block's pieces of A (two bfloat16 each)

template <int BN> struct PieceTile {
  static constexpr uint32_t W_PIECE = BN * 64, STAGE = 3 * W_PIECE;
  static constexpr int RING = BN == 64 ? 5 : (BN == 128 ? 4 : 2), ACC = BN == 64 ? 3 : 2;      // blocks of W and A on their way; accumulators
  static constexpr size_t SMEM = (size_t)RING * STAGE + 2 * RING * 8 + 16 + 1024;
  static_assert(ACC * BN + RING * A_COLS <= 512 && SMEM <= 227 * 1024, "an SM's memory");
};

struct PieceArgs {
  const float* A; int64_t lda;
  const float* W;
  const void* bias; int bias_f32;
  float* out; int64_t ldo;
  int M, N, K, vec_out;
  int skip_copy;                                // (tests: the first copy is left out, so that the wait for it runs out)
};

int g_skip_copy = 0;

// The upper halves of two floats as a pair of bfloat16 (truncated), and what is left of each.
__device__ __forceinline__ uint32_t cut(float& a, float& b) {
  const uint32_t x = __float_as_uint(a), y = __float_as_uint(b);
  a -= __uint_as_float(x & 0xffff0000u);
  b -= __uint_as_float(y & 0xffff0000u);
  return __byte_perm(x, y, 0x7632);
}

// W into scratch, eight neighbours along K a thread: 32 bytes in, 16 out for every piece.  Bound by memory: 10 bytes an entry.
__global__ void __launch_bounds__(256) pieces_kernel(const PieceArgs p, uint8_t* w_pieces, int bn) {
  pdl_launch_dependents();
  pdl_wait();                                   // (the scratch may still be read by the product before)
  const int num_kb = (p.K + BK - 1) / BK;
  const int64_t units = (int64_t)((p.N + bn - 1) / bn) * num_kb * bn * 4;
  for (int64_t u = (int64_t)blockIdx.x * 256 + threadIdx.x; u < units; u += (int64_t)gridDim.x * 256) {
    const int c = (int)(u & 3);
    const int64_t block = (u >> 2) / bn, tile = block / num_kb;
    const int r = (int)((u >> 2) - block * bn), k = (int)(block - tile * num_kb) * BK + c * 8;
    const int64_t row = tile * bn + r;
    float4 x0 = make_float4(0.f, 0.f, 0.f, 0.f), x1 = x0;
    if (row < p.N) {
      const float* src = p.W + row * p.K + k;
      if (k < p.K) x0 = *reinterpret_cast<const float4*>(src);
      if (k + 4 < p.K) x1 = *reinterpret_cast<const float4*>(src + 4);
    }
    float x[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
    uint8_t* dst = w_pieces + block * 3 * bn * 64 + r * 64 + ((c ^ ((r >> 1) & 3)) << 4);
#pragma unroll
    for (int piece = 0; piece < 3; ++piece) {
      uint32_t w[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) w[i] = cut(x[2 * i], x[2 * i + 1]);
      *reinterpret_cast<uint4*>(dst + piece * bn * 64) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
}

template <int N> __device__ __forceinline__ void regs_more() { asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N)); }
template <int N> __device__ __forceinline__ void regs_fewer() { asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N)); }
// D += A B with A in tensor memory (a lane a row, two neighbours along K a column)
__device__ __forceinline__ void umma_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
      ::"r"(tmem_d), "r"(tmem_a), "l"(b_desc), "r"(idesc), "r"(accumulate) : "memory");
}
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
// 16 lanes x 16 columns: r[0], r[1]: lane (thread / 4), columns 2 (thread % 4) and + 1; r[2], r[3]: eight lanes further; r[4 ..]: eight columns further.
__device__ __forceinline__ void tmem_st_16x16(uint32_t addr, const uint32_t (&r)[8]) {
  asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};"
               ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]) : "memory");
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
               ::"r"(smem_u32(dst)), "l"(src), "r"(bytes), "r"(smem_u32(bar)) : "memory");
}

__device__ __noinline__ float plain_dot(const float* a, const float* w, int K) {
  float s = 0.f;
  for (int k = 0; k < K; ++k) s = fmaf(a[k], w[k], s);
  return s;
}

// K-major tile whose rows are 64 bytes, 64-byte swizzle: groups of 8 rows are 512 bytes apart.
__device__ __forceinline__ uint64_t sw64_desc(uint32_t smem_addr) {
  uint64_t d = 0;
  d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;
  d |= (uint64_t)(512 >> 4) << 32;
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)4 << 61;                       // SWIZZLE_64B
  return d;
}

template <int BN, int EPI>
__global__ void __launch_bounds__(THREADS, 1) linear_pieces_kernel(const uint8_t* __restrict__ w_pieces, const PieceArgs p) {
  using T = PieceTile<BN>;
  constexpr int ACC = T::ACC, RING = T::RING, SHARE = BN / 2;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  // One barrier says that a block can be worked out: its W has come (a copy's bytes), its A lies in tensor memory (four warps) and its accumulator is free (eight
  // warps); one that its products have run.  (To the issuing warp a wait is 90 cycles and a commit 120: with a barrier for each of these things a block took it 1060.)
  uint64_t* ready = reinterpret_cast<uint64_t*>(smem + RING * T::STAGE);           // [RING]
  uint64_t* done = ready + RING;                                                    // [RING]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + RING);
  volatile uint32_t* failed = tmem_slot + 1;                                        // a wait of the block has run out
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_launch_dependents();
  if (threadIdx.x == 0) {
    *failed = 0;
    for (int s = 0; s < RING; ++s) { mbar_init(&ready[s], 1 + 4 + 8); mbar_init(&done[s], 1); }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 1) tmem_alloc(tmem_slot, 512);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot, tmem_a = tmem_base + ACC * BN;
  const int tiles_n = (p.N + BN - 1) / BN, tiles = tiles_n * ((p.M + BM - 1) / BM), num_kb = (p.K + BK - 1) / BK;
  const int mine = (int)blockIdx.x < tiles ? (tiles - (int)blockIdx.x - 1) / (int)gridDim.x + 1 : 0, blocks = mine * num_kb;      // of this CTA
  pdl_wait();

  if (warp < 4) {
    regs_fewer<32>();
    if (warp == 0 && lane == 0) {
      const int from = p.skip_copy ? 1 : 0;
      int s = 0, j = 0;
      uint32_t turn = 0;
      bool ok = true;
      for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        const uint8_t* w_at = w_pieces + (int64_t)(t % tiles_n) * num_kb * T::STAGE;
        for (int kb = 0; kb < num_kb; ++kb, ++j, w_at += T::STAGE) {
          if (j >= RING && !mbar_wait(&done[s], turn ^ 1)) { ok = false; break; }
          if (j >= from) {
            mbar_expect_tx(&ready[s], T::STAGE);
            bulk_load(smem + s * T::STAGE, w_at, T::STAGE, &ready[s]);
          }
          if (++s == RING) { s = 0; turn ^= 1; }
        }
      }
    } else if (warp == 1) {
      constexpr uint32_t idesc = umma_instr_desc(BM, BN);
      const uint64_t w0 = sw64_desc(smem_u32(smem));
      const bool one = elect_one();
      int s = 0, acc = 0;
      uint32_t turn = 0;
      for (int j = 0; j < blocks; ++j) {
        if (!mbar_wait(&ready[s], turn)) break;
        tc_fence_after();
        const uint64_t w = w0 + (uint32_t)s * (T::STAGE >> 4);
        const uint32_t d = tmem_base + (uint32_t)(acc * BN), a = tmem_a + (uint32_t)(s * A_COLS);
        if (one) {
          constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PW[6] = {0, 2, 1, 0, 1, 0};      // the smallest products first
#pragma unroll
          for (int x = 0; x < 6; ++x)
#pragma unroll
            for (int k = 0; k < BK / 16; ++k) umma_ta(d, a + PA[x] * 16 + k * 8, w + (uint64_t)(PW[x] * (T::W_PIECE >> 4) + k * 2), idesc, (x > 0 || k > 0) ? 1u : 0u);
          umma_commit(&done[s]);
        }
        if (++s == RING) { s = 0; turn ^= 1; }
        if (++acc == ACC) acc = 0;
      }
    }
  } else if (warp < 12) {
    // ---- A into tensor memory, by two groups of four warps in turn (a block takes one 1000 cycles): a warp has 32 rows; of each 16, a thread has two rows'
    // four neighbours along K, so that 4 threads read 64 bytes of a row
    regs_fewer<80>();
    const int group = (warp >> 2) - 1, quarter = warp & 3, r0 = quarter * 32 + (lane >> 2), k0 = (lane & 3) * 4;
    const uint32_t at = tmem_a + ((uint32_t)(quarter * 32) << 16);
    float4 f[8];                                // the group's next block: [row of four][half of the block]
    int load_t = 0, load_kb = group;
    auto fetch = [&]() {
      while (load_kb >= num_kb) {
        load_kb -= num_kb;
        ++load_t;
      }
      if (load_t >= mine) return;
      const int m0 = ((int)blockIdx.x + load_t * (int)gridDim.x) / tiles_n * BM, left = p.M - m0 - r0, k = load_kb * BK + k0;
      const float* row_at = p.A + (int64_t)(m0 + r0) * p.lda + k;
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int h = 0; h < 2; ++h)
          f[i * 2 + h] = i * 8 < left && h * 16 + k < p.K ? *reinterpret_cast<const float4*>(row_at + (int64_t)i * 8 * p.lda + h * 16) : make_float4(0.f, 0.f, 0.f, 0.f);
      load_kb += 2;
    };
    fetch();
    for (int j = group; j < blocks; j += 2) {
      const int ring = j % RING;
      if (j >= RING && !mbar_wait(&done[ring], ((j / RING) & 1) ^ 1)) break;
      tc_fence_after();
#pragma unroll
      for (int pair = 0; pair < 2; ++pair) {    // 16 rows: i = 2 pair and 2 pair + 1
        float4 x[4] = {f[pair * 4], f[pair * 4 + 2], f[pair * 4 + 1], f[pair * 4 + 3]};      // [half of the block][rows, eight further]
#pragma unroll
        for (int piece = 0; piece < 3; ++piece) {
          uint32_t w[8];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            w[2 * q] = cut(x[q].x, x[q].y);
            w[2 * q + 1] = cut(x[q].z, x[q].w);
          }
          tmem_st_16x16(at + ((uint32_t)(pair * 16) << 16) + (uint32_t)(ring * A_COLS + piece * 16), w);
        }
      }
      fetch();
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive_one(&ready[ring]);
    }
  } else {
    // ---- sums and what leaves: a thread a row and half of the tile's columns
    regs_more<144>();
    const int quarter = warp & 3, share = warp >= 16 ? 1 : 0;
    const uint32_t lanes = tmem_base + ((uint32_t)(quarter * 32) << 16) + share * SHARE;
    int acc = 0, j = 0;
    bool ok = true;
    if (lane == 0)
      for (int b = 0; b < min(ACC, blocks); ++b) mbar_arrive_one(&ready[b]);      // (every accumulator is free)
    auto outcome = [&](float x, int col) {
      if (p.bias != nullptr) x += load_param(p.bias, col, p.bias_f32);
      if (EPI == EPI_GELU_TANH) x = gelu_tanh(x);
      if (EPI == EPI_GELU_ERF) x = gelu_erf(x);
      return x;
    };
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
      float sum[SHARE];
#pragma unroll
      for (int i = 0; i < SHARE; ++i) sum[i] = 0.f;
      for (int kb = 0; kb < num_kb; ++kb, ++j) {
        if (!mbar_wait(&done[j % RING], (j / RING) & 1)) { ok = false; break; }
        tc_fence_after();
        {
          uint32_t v[32];
#pragma unroll
          for (int c = 0; c < SHARE; c += 32) {
            tmem_ld32(lanes + (uint32_t)(acc * BN + c), v);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 32; ++i) sum[c + i] += __uint_as_float(v[i]);
          }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0 && j + ACC < blocks) mbar_arrive_one(&ready[(j + ACC) % RING]);
        if (++acc == ACC) acc = 0;
      }
      if (!ok) break;
      const int row = t / tiles_n * BM + quarter * 32 + lane, col0 = t % tiles_n * BN + share * SHARE;
      if (row >= p.M) continue;
      float* o = p.out + (int64_t)row * p.ldo + col0;
#pragma unroll
      for (int c = 0; c < SHARE; c += 4) {
        float x[4];
        bool whole = p.vec_out != 0, wrong = false;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          x[e] = sum[c + e];
          wrong |= x[e] != x[e];
          if (col0 + c + e < p.N) x[e] = outcome(x[e], col0 + c + e);
          else whole = false;
        }
        if (whole && !wrong) {
          float4 y = make_float4(x[0], x[1], x[2], x[3]);
          if (EPI == EPI_RESIDUAL) {
            const float4 old = *reinterpret_cast<const float4*>(o + c);
            y.x += old.x; y.y += old.y; y.z += old.z; y.w += old.w;
          }
          *reinterpret_cast<float4*>(o + c) = y;
        } else {
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int col = col0 + c + e;
            if (col >= p.N) continue;
            const float y = sum[c + e] == sum[c + e] ? x[e] : outcome(plain_dot(p.A + (int64_t)row * p.lda, p.W + (int64_t)col * p.K, p.K), col);
            o[c + e] = EPI == EPI_RESIDUAL ? o[c + e] + y : y;
          }
        }
      }
    }
    if (!ok) *failed = 1;                       // (whichever role gave up: then there are products that this one has waited for in vain)
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (*failed != 0) outlast_what_is_in_flight();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tmem_base, 512);
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
int launch(const uint8_t* wp, const PieceArgs& a, cudaStream_t stream) {
  using T = PieceTile<BN>;
  static bool configured = false;
  if (!configured) {
    cudaError_t e = cudaFuncSetAttribute(linear_pieces_kernel<BN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::SMEM);
    if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "linear_pieces: cannot reserve %zu bytes of shared memory: %s", T::SMEM, cudaGetErrorString(e));
    configured = true;
  }
  const int64_t tiles = (int64_t)((a.N + BN - 1) / BN) * ((a.M + BM - 1) / BM);
  KVAD_REQUIRE(tiles < (1ll << 30), "linear_pieces: %lld tiles are more than one launch takes", (long long)tiles);
  kvad_launch(linear_pieces_kernel<BN, EPI>, dim3((unsigned)(tiles < sm_count() ? tiles : sm_count())), dim3(THREADS), T::SMEM, stream, wp, a);
  KVAD_CHECK_LAUNCH("linear_pieces");
  return KVAD_OK;
}

template <int BN>
int launch_epi(int epilogue, const uint8_t* wp, const PieceArgs& a, cudaStream_t stream) {
  switch (epilogue) {
    case EPI_STORE:
    case EPI_STORE_F32: return launch<BN, EPI_STORE>(wp, a, stream);
    case EPI_GELU_TANH: return launch<BN, EPI_GELU_TANH>(wp, a, stream);
    case EPI_GELU_ERF: return launch<BN, EPI_GELU_ERF>(wp, a, stream);
    case EPI_RESIDUAL: return launch<BN, EPI_RESIDUAL>(wp, a, stream);
  }
  KVAD_FAIL(KVAD_ERR_ARGUMENT, "linear_pieces: unknown epilogue %d", epilogue);
}

}  // namespace

// `work`: scratch, 192 bytes for each row of W (rounded up to whole tiles) and 32 of K.  `force_bn`: 0, or the tile width (64, 128 or 192).
KVAD_EXPORT int kvad_linear_pieces(const float* A, int64_t lda, const float* W, const void* bias, int bias_f32, float* out, int64_t ldo, int M, int N, int K,
                                   int epilogue, int force_bn, void* work, int64_t work_bytes, cudaStream_t stream) {
  KVAD_REQUIRE(M >= 0 && N > 0 && K > 0 && lda >= K && ldo >= N, "linear_pieces: bad sizes M=%d N=%d K=%d lda=%lld ldo=%lld", M, N, K, (long long)lda, (long long)ldo);
  KVAD_REQUIRE(force_bn == 0 || force_bn == 64 || force_bn == 128 || force_bn == 192, "linear_pieces: tile width %d is not 64, 128 or 192", force_bn);
  if (K % 4 != 0 || lda % 4 != 0 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(work)) & 15))
    KVAD_FAIL(KVAD_ERR_UNSUPPORTED, "linear_pieces: K and strides in quads, rows on 16-byte boundaries");
  if (M == 0) return KVAD_OK;
  KVAD_REQUIRE(work != nullptr, "linear_pieces: needs scratch");
  PieceArgs a;
  a.A = A; a.lda = lda; a.W = W; a.bias = bias; a.bias_f32 = bias_f32; a.out = out; a.ldo = ldo; a.M = M; a.N = N; a.K = K;
  a.skip_copy = g_skip_copy;
  g_skip_copy = 0;
  a.vec_out = (ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0) ? 1 : 0;
  int bn = force_bn;
  if (bn == 0) {        // waves of one tile an SM times a block's products (half a cycle a column each; a narrow tile's cutting takes longer than its products)
    const int64_t rows = (M + BM - 1) / BM, sms = sm_count();
    int64_t best = 0;
    for (int w = 64; w <= 192; w += 64) {
      const int64_t cost = (rows * ((N + w - 1) / w) + sms - 1) / sms * (w == 64 ? 44 : w / 2);
      if (bn == 0 || cost < best) { bn = w; best = cost; }
    }
  }
  const int64_t n_rows = (int64_t)(N + bn - 1) / bn * bn, num_kb = (K + BK - 1) / BK;
  KVAD_REQUIRE(n_rows * num_kb * 192 <= work_bytes, "linear_pieces: %lld bytes of scratch are too few", (long long)work_bytes);
  KVAD_REQUIRE((int64_t)((M + BM - 1) / BM) * n_rows / bn * num_kb < (1ll << 30), "linear_pieces: more blocks than one launch counts");
  uint8_t* wp = (uint8_t*)work;
  const int64_t blocks = (n_rows * num_kb * 4 + 255) / 256;
  kvad_launch(pieces_kernel, dim3((unsigned)(blocks < 8 * sm_count() ? blocks : 8 * sm_count())), dim3(256), 0, stream, a, wp, bn);
  KVAD_CHECK_LAUNCH("linear_pieces (cut)");
  if (bn == 64) return launch_epi<64>(epilogue, wp, a, stream);
  if (bn == 128) return launch_epi<128>(epilogue, wp, a, stream);
  return launch_epi<192>(epilogue, wp, a, stream);
}

// How many bounded waits have run out since the library was loaded (0 in a healthy run).  Synchronises the device.
KVAD_EXPORT int kvad_linear_pieces_status() {
  int n = 0;
  cudaError_t e = cudaMemcpyFromSymbol(&n, g_wait_timeouts, sizeof(int));
  if (e != cudaSuccess) KVAD_FAIL(KVAD_ERR_CUDA, "linear_pieces_status: %s", cudaGetErrorString(e));
  return n;
}

// Tests of the bounded waits: `wait_limit` > 0 sets how many polls a wait makes before it gives up (0: the library's own limit); `skip_copy` leaves the first copy out of
// the NEXT launch's blocks, so that the wait for it runs out.  Synchronises the device.
KVAD_EXPORT int kvad_linear_pieces_test_hooks(unsigned wait_limit, int skip_copy) {
  g_skip_copy = skip_copy;
  return set_wait_limit(wait_limit);
}

KVAD_DEFINE_LAST_ERROR()
