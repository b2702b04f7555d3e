// y = x · Wᵀ for a weight [N, K] and any M, N, K and any mix of float32 / bfloat16 operands,
// with float32 multiply-adds on the CUDA cores (no tensor-core or reduced-precision mode):
// the matrix product of the true 32-bit path for few rows, and the fallback for sizes that the
// tensor-core kernels refuse (gemm_split.cu has the 32-bit path's products of many rows). The role of the reference's `gemm8` and `linear8`
// (tools/cuda/linear.cu:418-463, :517-606 of the reference project), without its
// quantized formats.
//
// Epilogues: store; add into a float32 residual; SwiGLU over a weight [2N, K] (out =
// silu(gate) * up) whose rows are either [0, N) gate and [N, 2N) up, or alternate gate, up,
// gate, up ... (the layout that the tensor-core kernel's fused epilogue uses).
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

MB_DEFINE_LAST_ERROR

enum { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU = 2, EPI_SWIGLU_PAIRS = 3 };

#define BM 64
#define BN 64
#define BK 16

// The output's type is looked at when a result is stored, not compiled in: eight variants of
// every kernel less to build.
__device__ __forceinline__ void put_out(void* C, int c_bf16, size_t at, float v, bool add) {
  if (c_bf16) {
    ((__nv_bfloat16*)C)[at] = __float2bfloat16_rn(v);  // a residual add is float32 only
  } else {
    float* out = (float*)C + at;
    *out = add ? *out + v : v;
  }
}

// SwiGLU over a weight whose gate rows come first and whose up rows follow, for more rows of A than
// gemm_few_rows_kernel takes: 64 x 64 outputs a block, two sums each.
template <typename TA, typename TW>
__global__ void __launch_bounds__(256)
gemm_swiglu_halves_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W,
                          void* __restrict__ C, int c_bf16, int ldc, int M, int N, int K) {
  __shared__ float As[BK][BM + 4];
  __shared__ float Ws[2][BK][BN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  const int tr = (tid / 16) * 4, tc = (tid % 16) * 4;
  float acc[2][4][4];
#pragma unroll
  for (int w = 0; w < 2; ++w)
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[w][i][j] = 0.f;

  for (int k0 = 0; k0 < K; k0 += BK) {
    // 64 x 16 elements per tile, 256 threads: 4 each
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + i * 256;
      const int r = e / BK, c = e % BK;
      const int gm = m0 + r, gk = k0 + c;
      As[c][r] = (gm < M && gk < K) ? to_f32<TA>(A[(size_t)gm * lda + gk]) : 0.f;
      const int gn = n0 + r;
#pragma unroll
      for (int w = 0; w < 2; ++w)
        Ws[w][c][r] = (gn < N && gk < K) ? to_f32<TW>(W[((size_t)w * N + gn) * K + gk]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < BK; ++k) {
      float a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) a[i] = As[k][tr + i];
#pragma unroll
      for (int w = 0; w < 2; ++w) {
        float b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Ws[w][k][tc + j];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[w][i][j] = fmaf(a[i], b[j], acc[w][i][j]);
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int gm = m0 + tr + i;
    if (gm >= M) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int gn = n0 + tc + j;
      if (gn >= N) continue;
      const float g = acc[0][i][j];
      put_out(C, c_bf16, (size_t)gm * ldc + gn, g / (1.0f + expf(-g)) * acc[1][i][j], false);
    }
  }
}

// ---------------------------------------------------------------------------- few rows
// The same product for at most 16 rows of A (a decode step): the weight streams through once, and
// its bytes are what bounds it. A warp owns four weight rows at a time (four output features, or two
// with their gate and up rows) and walks K in chunks of 128 (every lane 4 consecutive values of each
// of its rows, 16 bytes of float32), against up to eight rows of A. Three chunks are under way or at
// work at a time, over the border from one group of rows to the next, and the blocks stay for the
// whole weight, so that enough bytes are asked for at every moment; the rows of A lie in shared
// memory where they fit (FEW_STAGED: two blocks a multiprocessor) and a warp has work enough, and come
// four reads at a time elsewhere, with two chunks under way. One or two rows' values are asked for with
// the weight's (four reads of which three are the same row's took a quarter longer). More than eight
// rows take two passes, group by group where all rows lie in shared memory, else over the whole weight.
// The 32 sums are reduced by halves, a value a lane at the end. A weight with few rows has KW warps of a
// block share each four rows along K. Eight rows, float32, from memory, one chunk ahead and a block for
// every eight groups -> this form: 151,936 x 1,024 163 -> 119 us (5.2 TB/s), 2 x 12,288 x 4,096 182 ->
// 123, 4,096 x 12,288 147 -> 84, 2 x 3,072 x 1,024 27 -> 18.5, 1,024 x 3,072 18.5 -> 13.3. One row, in a
// graph: 151,936 x 1,024 117 -> 89, 1,024 x 3,072 4.3 -> 3.5, 1,024 x 1,024 2.5 -> 2.4; nine rows,
// 151,936 x 1,024 190 -> 154 (a walk through the weight for each pass: 190).
// A weight row's values are used once: they pass by the L1 cache. Predicated, zeros where not `ok`: a
// load behind a branch would be waited for where the branch ends.
template <typename T> __device__ __forceinline__ float4 load4_once(const T* p, bool ok);
template <> __device__ __forceinline__ float4 load4_once<float>(const float* p, bool ok) {
  float4 v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
      "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
      "@p ld.global.nc.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}\n"
      : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w)
      : "l"(p), "r"((int)ok));
  return v;
}
template <> __device__ __forceinline__ float4 load4_once<__nv_bfloat16>(const __nv_bfloat16* p, bool ok) {
  uint2 raw;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t"
      "@p ld.global.nc.L1::no_allocate.v2.u32 {%0, %1}, [%2];\n\t}\n"
      : "=&r"(raw.x), "=&r"(raw.y)
      : "l"(p), "r"((int)ok));
  const float2 lo = __bfloat1622float2(*(const __nv_bfloat162*)&raw.x);
  const float2 hi = __bfloat1622float2(*(const __nv_bfloat162*)&raw.y);
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

// The same of a value that is used again
template <typename T> __device__ __forceinline__ float4 load4_ok(const T* p, bool ok);
template <> __device__ __forceinline__ float4 load4_ok<float>(const float* p, bool ok) {
  float4 v;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
      "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
      "@p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}\n"
      : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w)
      : "l"(p), "r"((int)ok)
      : "memory");
  return v;
}
template <> __device__ __forceinline__ float4 load4_ok<__nv_bfloat16>(const __nv_bfloat16* p, bool ok) {
  uint2 raw;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %3, 0;\n\t"
      "mov.b32 %0, 0;\n\tmov.b32 %1, 0;\n\t"
      "@p ld.global.v2.u32 {%0, %1}, [%2];\n\t}\n"
      : "=&r"(raw.x), "=&r"(raw.y)
      : "l"(p), "r"((int)ok)
      : "memory");
  const float2 lo = __bfloat1622float2(*(const __nv_bfloat162*)&raw.x);
  const float2 hi = __bfloat1622float2(*(const __nv_bfloat162*)&raw.y);
  return make_float4(lo.x, lo.y, hi.x, hi.y);
}

#define FEW_ROWS 8   // rows of A in one pass
#define FEW_MAX 16   // the most rows that take this kernel

#define FEW_STAGED (96 * 1024)   // bytes of A's rows that still go into shared memory

// ROWS: rows of A in one pass. TWO_PASSES (STAGED only): more than ROWS of them lie in shared memory, and
// a group's weights are read for all passes before the next group's, the second time from L2.
template <typename TA, typename TW, int EPI, int ROWS, bool STAGED, bool TWO_PASSES>
__global__ void __launch_bounds__(256, 2)
gemm_few_rows_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W,
                     void* __restrict__ C, int c_bf16, int ldc, int M, int N, int K, int KW,
                     int groups, int settled) {
  constexpr bool GLU = EPI == EPI_SWIGLU || EPI == EPI_SWIGLU_PAIRS;
  constexpr int FEATS = GLU ? 2 : 4;  // output features of a warp
  constexpr bool AHEAD = ROWS <= 2;   // A's values are asked for with the weights'
  constexpr int DEPTH = STAGED || AHEAD ? 3 : 2;      // chunks under way or at work
  extern __shared__ __align__(16) float As[];      // STAGED: [rows of a walk through the weight][K]
  __shared__ float part[8][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per_block = 8 / KW, kw = warp % KW, step = gridDim.x * per_block;
  const int k_first = kw * 128 + lane * 4, k_step = KW * 128;
  const int chunks = (K + k_step - 1) / k_step;
  const int g_block = blockIdx.x * per_block, g0 = g_block + warp / KW;
  // the chunk that is asked for next: its group and pass (rows of A), place and the group's four weight
  // rows; a row beyond the weight is read as its last and not stored
  int ask_g, ask_m, ask_k;
  const TW* wr[4];
  auto enter = [&](int g) {
    ask_g = g;
    ask_m = 0;
    ask_k = k_first;
    const int n0 = g * FEATS;
    if (g < groups) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        int row;
        if (EPI == EPI_SWIGLU) row = (j >> 1) * N + min(n0 + (j & 1), N - 1);     // g0 g1 u0 u1
        else if (EPI == EPI_SWIGLU_PAIRS) row = 2 * min(n0 + (j >> 1), N - 1) + (j & 1);  // g0 u0 g1 u1
        else row = min(n0 + j, N - 1);
        wr[j] = W + (size_t)row * K;
      }
    }
  };
  struct Chunk { float4 w[4], a[AHEAD ? ROWS : 1]; };
  auto ask_a = [&](Chunk& c, int k, bool ok) {
#pragma unroll
    for (int i = 0; i < ROWS; ++i) c.a[i] = load4_ok<TA>(A + (size_t)i * lda + k, ok && i < M);
  };
  auto ask = [&](Chunk& c, bool rows) {
    const bool ok = ask_k < K && ask_g < groups;
#pragma unroll
    for (int j = 0; j < 4; ++j) c.w[j] = load4_once<TW>(wr[j] + ask_k, ok);
    if (AHEAD && rows) ask_a(c, ask_k, ok);
    ask_k += k_step;
    if (ask_k - k_first >= chunks * k_step) {
      ask_k = k_first;
      if (!TWO_PASSES || (ask_m += ROWS) >= M) enter(ask_g + step);
    }
  };
  Chunk c0, c1, c2;
  auto begin = [&]() {
#pragma unroll
    for (int j = 0; j < 4; ++j) wr[j] = W;
    enter(g0);
    ask(c0, false);
    ask(c1, false);
    if (DEPTH > 2) ask(c2, false);
  };
  // the first chunks ahead of the wait, where the kernel before does not write the weight
  if (settled) begin();
  mb_grid_wait();
  mb_grid_launch_next();
  if (!settled) begin();
  if (AHEAD) {
    int k = k_first, left = chunks;
    auto next = [&](Chunk& c) {
      ask_a(c, k, k < K);
      k += k_step;
      if (--left == 0) { left = chunks; k = k_first; }
    };
    next(c0);
    next(c1);
    next(c2);
  }
  // walks through the weight, one for all rows (TWO_PASSES) or one for every ROWS of them
  const int per_walk = TWO_PASSES ? M : ROWS;
  for (int m_walk = 0; m_walk < M; m_walk += per_walk) {
    const int walk_rows = min(M - m_walk, per_walk);
    if (m_walk) begin();
    if (STAGED) {
      if (m_walk) __syncthreads();
      const int per_row = K >> 2;
      for (int m = 0; m < walk_rows; ++m)
        for (int i = threadIdx.x; i < per_row; i += 256)
          *(float4*)(As + m * K + 4 * i) = load4<TA>(A + (size_t)(m_walk + m) * lda + 4 * i);
      __syncthreads();
    }
    float acc[4 * ROWS];
    int g = g0, m0 = 0, k = k_first, chunk = 0;
    bool more = g_block < groups;      // the same for the whole block
    auto row_of = [&](const Chunk& c, float4 a, int m) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float& s = acc[j * ROWS + m];
        s = fmaf(a.x, c.w[j].x, fmaf(a.y, c.w[j].y, fmaf(a.z, c.w[j].z, fmaf(a.w, c.w[j].w, s))));
      }
    };
    auto work = [&](Chunk& c) {
      if (chunk == 0) {
#pragma unroll
        for (int j = 0; j < 4 * ROWS; ++j) acc[j] = 0.f;
      }
      const int rows = walk_rows - m0;      // ROWS of them, or what is left: the same for the block
      if (AHEAD) {
#pragma unroll
        for (int m = 0; m < ROWS; ++m)
          if (m < rows) row_of(c, c.a[m], m);
      } else if (k < K) {
        constexpr int BATCH = STAGED ? 1 : 4;      // reads of A under way together
#pragma unroll
        for (int mb = 0; mb < ROWS; mb += BATCH) {
          if (mb >= rows) break;
          float4 a[BATCH];
#pragma unroll
          for (int i = 0; i < BATCH; ++i)
            a[i] = STAGED ? *(const float4*)(As + (m0 + mb) * K + k)
                          : load4<TA>(A + (size_t)(m_walk + min(mb + i, rows - 1)) * lda + k);
#pragma unroll
          for (int i = 0; i < BATCH; ++i) row_of(c, a[i], mb + i);
        }
      }
      ask(c, true);
      k += k_step;
      if (++chunk < chunks) return;
      // the group's end
      float v = sums_by_lane<4 * ROWS>(acc, lane);
      if (KW > 1) {
        __syncthreads();      // the sums of the group before have been read
        part[warp][lane] = v;
        __syncthreads();
        if (kw == 0)
          for (int i = 1; i < KW; ++i) v += part[warp + i][lane];
      }
      constexpr int EACH = 8 / ROWS;      // lanes that have the sum of weight row j and row m of A
      const int j = lane >> 3, m = m_walk + m0 + (lane & 7) / EACH;
      const float up = GLU ? __shfl_sync(0xffffffffu, v, (lane + (EPI == EPI_SWIGLU ? 16 : 8)) & 31) : 0.f;
      const int f = EPI == EPI_SWIGLU_PAIRS ? j >> 1 : j, n0 = g * FEATS;
      const bool has = (EPI == EPI_SWIGLU_PAIRS ? !(j & 1) : (EPI != EPI_SWIGLU || j < 2)) && lane % EACH == 0;
      if (kw == 0 && m < M && has && n0 + f < N)
        put_out(C, c_bf16, (size_t)m * ldc + n0 + f, GLU ? v / (1.0f + expf(-v)) * up : v, EPI == EPI_ADD);
      chunk = 0;
      k = k_first;
      if (TWO_PASSES && (m0 += ROWS) < walk_rows) return;
      m0 = 0;
      g += step;
      more = g - warp / KW < groups;
    };
    while (more) {
      work(c0);
      if (more) work(c1);
      if (DEPTH > 2 && more) work(c2);
    }
  }
}

// ---------------------------------------------------------------------------- many rows
// The same product for many rows where an operand is bfloat16 or K is short (float32 operands
// otherwise go through gemm_split.cu), bound by the latencies of multiply-adds and of shared memory
// with the 7.6 warps a multiprocessor that the registers leave (the multiply-adds' pipe is 0.57
// busy). Reads of shared memory come close behind: a 16-byte read of a warp takes four cycles
// whatever its lanes share, so a thread has 16 x 8 results (six reads per 128 multiply-adds; 8 x 8
// would need as many cycles for the one as for the other). Multiply-adds go two rows an
// instruction (`fma.rn.f32x2`, each half rounded like a single one), which leaves issue slots for
// the reads. Blocks are small (64 threads, 64 x 128 results, four to a multiprocessor), K goes in
// steps of 8 through two buffers with the next step's global loads under way; where tiles are few
// or would leave a last round half empty, K is dealt out over a cluster whose CTAs add their sums
// up through shared memory, in K's order. Epilogues: store, residual add, and SwiGLU over weight
// rows that alternate gate and up (NW = 2 N weight rows, neighbouring columns pair up). 1,728
// rows, 6,144 x 1,024 (SwiGLU): 639 us with 128 x 128 tiles, 8 x 8 results a thread -> 519 (42
// TFLOP/s); 1,024 x 2,048: 247 -> 216, with 400 rows 246 -> 68. Lanes of a row-wise load that
// stand in 32 rows cost a tenth of it: a row's LK values lie with neighbouring lanes.
#define LM 64
#define LN 128
#define LK 8
#define LMP (LM + 4)
#define LNP (LN + 4)

// four values k .. k + 3 of a row as float32, zeros beyond K or for a row that does not exist
template <typename T>
__device__ __forceinline__ float4 row_piece(const T* __restrict__ base, bool row_ok, int k, int K,
                                            bool vec) {
  if (!row_ok || k >= K) return make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec) return load4<T>(base + k);
  float4 v;
  v.x = to_f32<T>(base[k]);
  v.y = k + 1 < K ? to_f32<T>(base[k + 1]) : 0.f;
  v.z = k + 2 < K ? to_f32<T>(base[k + 2]) : 0.f;
  v.w = k + 3 < K ? to_f32<T>(base[k + 3]) : 0.f;
  return v;
}

template <typename TA, typename TW, int EPI>
__global__ void __launch_bounds__(64, 4)
gemm_many_rows_kernel(const TA* __restrict__ A, int lda, const TW* __restrict__ W,
                      void* __restrict__ C, int c_bf16, int ldc, int M, int NW, int K, int vec_a,
                      int vec_w, int splits, int k_split) {
  // [buffer][K step][rows of A | rows of W]; a split's sums [LM][LN] reuse it
  extern __shared__ __align__(16) float sm[];
  constexpr int BUF = LK * (LMP + LNP);
  const int tid = threadIdx.x;
  const int split = blockIdx.x % splits;
  const int m0 = blockIdx.y * LM, n0 = (blockIdx.x / splits) * LN;
  const int k_lo = split * k_split, k_hi = min(K, k_lo + k_split);
  // loads: a row's LK values lie with LK / 4 neighbouring lanes; a pass brings RP rows
  constexpr int PER = LK / 4, RP = 64 / PER, PA = LM / RP, PW = LN / RP;
  const int lr = tid / PER, lk = 4 * (tid % PER);
  const int ty = tid >> 4, tx = tid & 15;
  // rows 16 g + 4 ty + (0 .. 3), two a pair; columns 64 h + 4 tx + (0 .. 3)
  f32_pair acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0ull;
  mb_grid_wait();
  mb_grid_launch_next();

  float4 r[PA + PW];
  auto fetch = [&](int k) {
#pragma unroll
    for (int i = 0; i < PA; ++i) {
      const int m = m0 + lr + RP * i;
      r[i] = row_piece<TA>(A + (size_t)m * lda, m < M, k + lk, k_hi, vec_a);
    }
#pragma unroll
    for (int i = 0; i < PW; ++i) {
      const int n = n0 + lr + RP * i;
      r[PA + i] = row_piece<TW>(W + (size_t)n * K, n < NW, k + lk, k_hi, vec_w);
    }
  };
  auto put = [&](float* buf) {
#pragma unroll
    for (int i = 0; i < PA + PW; ++i) {
      const int pitch = i < PA ? LMP : LNP;
      float* d = buf + (i < PA ? RP * i : LK * LMP + RP * (i - PA)) + lr + lk * pitch;
      d[0] = r[i].x;
      d[pitch] = r[i].y;
      d[2 * pitch] = r[i].z;
      d[3 * pitch] = r[i].w;
    }
  };
  int cur = 0;
  fetch(k_lo);
  put(sm);
  __syncthreads();
  for (int k0 = k_lo; k0 < k_hi; k0 += LK) {
    const bool more = k0 + LK < k_hi;
    if (more) fetch(k0 + LK);
    const float* as = sm + cur * BUF + 4 * ty;
    const float* ws = sm + cur * BUF + LK * LMP + 4 * tx;
#pragma unroll
    for (int k = 0; k < LK; ++k) {
      ulonglong2 a[4];
      float4 b[2];
#pragma unroll
      for (int g = 0; g < 4; ++g) a[g] = *(const ulonglong2*)(as + k * LMP + 16 * g);
#pragma unroll
      for (int h = 0; h < 2; ++h) b[h] = *(const float4*)(ws + k * LNP + 64 * h);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 bq = b[j >> 2];
        const float bj = (j & 3) == 0 ? bq.x : ((j & 3) == 1 ? bq.y : ((j & 3) == 2 ? bq.z : bq.w));
        const f32_pair bb = pair_of(bj, bj);
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          pair_fma(acc[2 * g][j], a[g].x, bb);
          pair_fma(acc[2 * g + 1][j], a[g].y, bb);
        }
      }
    }
    if (more) {
      put(sm + (cur ^ 1) * BUF);
      __syncthreads();
      cur ^= 1;
    }
  }
  // four neighbouring columns of a row
  auto finish = [&](int gm, int gn, float4 v) {
    if (gm >= M) return;
    const float c[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (gn + j >= NW) return;
      if (EPI == EPI_SWIGLU_PAIRS) {
        // gate at the even weight row, up at the odd one after it
        if (!(j & 1))
          put_out(C, c_bf16, (size_t)gm * ldc + ((gn + j) >> 1), c[j] / (1.0f + expf(-c[j])) * c[j + 1], false);
      } else {
        put_out(C, c_bf16, (size_t)gm * ldc + gn + j, c[j], EPI == EPI_ADD);
      }
    }
  };
  if (splits > 1) __syncthreads();      // the last step's reads are done
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int row = 16 * (i >> 2) + 4 * ty + (i & 3);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const f32_pair* p = acc[i >> 1] + 4 * h;
      const float4 v = make_float4(pair_half(p[0], i & 1), pair_half(p[1], i & 1),
                                   pair_half(p[2], i & 1), pair_half(p[3], i & 1));
      if (splits == 1) finish(m0 + row, n0 + 64 * h + 4 * tx, v);
      else *(float4*)(sm + row * LN + 64 * h + 4 * tx) = v;
    }
  }
  if (splits == 1) return;
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  for (int e = 4 * (split * 64 + tid); e < LM * LN; e += 4 * 64 * splits) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < splits; ++k) {
      const float4 o = *(const float4*)(cluster.map_shared_rank(sm, k) + e);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    finish(m0 + e / LN, n0 + e % LN, v);
  }
  cluster.sync();      // nobody leaves while its sums are still read
}

template <typename TA, typename TW>
static int launch(const void* A, int lda, const void* W, void* C, int c_bf16, int ldc, int M, int N,
                  int K, int epi, int settled, int sms, cudaStream_t s) {
  // few rows, and every row piece of 4 values a whole aligned load
  const int a_align = sizeof(TA) == 4 ? 15 : 7, w_align = sizeof(TW) == 4 ? 15 : 7;
  if (M <= FEW_MAX && K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A & a_align) == 0 &&
      ((uintptr_t)W & w_align) == 0) {
    const int feats = (epi == EPI_SWIGLU || epi == EPI_SWIGLU_PAIRS) ? 2 : 4;
    const int groups = (N + feats - 1) / feats;
    // Warps that share a group's K: as many as leave the least to do for the busiest warp, in chunks of
    // 128 with one more for what a group's end takes, when two blocks of eight warps a multiprocessor
    // are all that run
    const int room = 2 * sms;
    int kw = 1;
    long long least = 1ll << 60;
    for (int n = 1; n <= 8 && (n == 1 || n / 2 * 128 < K); n *= 2) {
      const long long work = (long long)((groups + (8 / n) * room - 1) / ((8 / n) * room)) *
                             ((K + 128 * n - 1) / (128 * n) + 1);
      if (work < least) { least = work; kw = n; }
    }
    const int all = (groups + 8 / kw - 1) / (8 / kw), blocks = all < room ? all : room;
    // the rows of A that a walk through the weight has in shared memory: all of them where they fit
    const int walk_rows = M <= FEW_ROWS || (size_t)M * K * sizeof(float) <= FEW_STAGED ? M : FEW_ROWS;
    const size_t bytes = (size_t)walk_rows * K * sizeof(float);
    // The rows of A into shared memory where a warp has at least eight chunks: the copy costs a wait
    // of its own. Eight rows, us with | without: 151,936 x 1,024 119 | 134 and 2 x 3,072 x 1,024 (8
    // chunks a warp) 18.5 | 20.5, but 4,096 x 1,024 (4) 16.4 | 14.5 and 1,024 x 3,072 (3) 16.4 | 13.3.
    const long long rounds = (groups + (8 / kw) * (long long)blocks - 1) / ((8 / kw) * (long long)blocks);
    const bool staged = bytes <= FEW_STAGED && rounds * ((K + 128 * kw - 1) / (128 * kw)) >= 8;
#define FEW2(E, R_, S_, T_)                                                                   \
  {                                                                                           \
    static unsigned long long allowed = 0;                                                    \
    const auto kernel = gemm_few_rows_kernel<TA, TW, E, R_, S_, T_>;                          \
    const cudaError_t e =                                                                     \
        S_ ? mb_allow_smem((const void*)kernel, FEW_STAGED, &allowed) : cudaSuccess;          \
    if (e != cudaSuccess) MB_FAIL("mb_gemm_simt: %s", cudaGetErrorString(e));                 \
    mb_launch(kernel, dim3(blocks), dim3(256), S_ ? bytes : 0, s, (const TA*)A, lda,          \
              (const TW*)W, C, c_bf16, ldc, M, N, K, kw, groups, settled);                    \
  }
#define FEW(E)                                                                                \
  if (M <= 2) FEW2(E, 2, false, false)                                                        \
  else if (!staged) FEW2(E, FEW_ROWS, false, false)                                           \
  else if (walk_rows > FEW_ROWS) FEW2(E, FEW_ROWS, true, true)                                \
  else FEW2(E, FEW_ROWS, true, false)
    switch (epi) {
      case EPI_STORE: FEW(EPI_STORE) break;
      case EPI_ADD: FEW(EPI_ADD) break;
      case EPI_SWIGLU: FEW(EPI_SWIGLU) break;
      default: FEW(EPI_SWIGLU_PAIRS)
    }
#undef FEW
#undef FEW2
    MB_CHECK_LAUNCH("mb_gemm_simt");
  }
  if (epi != EPI_SWIGLU) {
    const int NW = epi == EPI_SWIGLU_PAIRS ? 2 * N : N;
    const int tiles_n = (NW + LN - 1) / LN, tiles_m = (M + LM - 1) / LM;
    if (tiles_m > 65535) MB_FAIL("mb_gemm_simt: %d rows are too many for one launch", M);
    const int vec_a = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A & a_align) == 0;
    const int vec_w = K % 4 == 0 && ((uintptr_t)W & w_align) == 0;
    // splits of K, at least 128 values each: what a multiprocessor has to do in units of one whole
    // tile, where fewer than three CTAs take as long as three
    const int tiles = tiles_n * tiles_m;
    int splits = 1;
    double best = 1e30;
    for (int n = 1; n <= 8 && (n == 1 || K >= 128 * n); ++n) {
      const int each = (int)(((long long)tiles * n + sms - 1) / sms);
      const double cost = (double)(each < 3 ? 3 : each) / n + 0.02 * n;
      if (cost < best) { best = cost; splits = n; }
    }
    const int k_split = ((K + splits - 1) / splits + LK - 1) / LK * LK;
    splits = (K + k_split - 1) / k_split;
    const size_t buffers = 2 * LK * (LMP + LNP) * sizeof(float), sums = LM * LN * sizeof(float);
    const size_t smem = splits > 1 && sums > buffers ? sums : buffers;
#define MANY(E)                                                                               \
  mb_launch_clusters(gemm_many_rows_kernel<TA, TW, E>, dim3(tiles_n * splits, tiles_m), dim3(64), smem, s, \
                     splits, (const TA*)A, lda, (const TW*)W, C, c_bf16, ldc, M, NW, K, vec_a, \
                     vec_w, splits, k_split)
    if (epi == EPI_STORE) MANY(EPI_STORE);
    else if (epi == EPI_ADD) MANY(EPI_ADD);
    else MANY(EPI_SWIGLU_PAIRS);
#undef MANY
    MB_CHECK_LAUNCH("mb_gemm_simt");
  }
  dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
  if (grid.y > 65535) MB_FAIL("mb_gemm_simt: %d rows are too many for one launch", M);
  gemm_swiglu_halves_kernel<TA, TW><<<grid, 256, 0, s>>>((const TA*)A, lda, (const TW*)W, C, c_bf16,
                                                         ldc, M, N, K);
  MB_CHECK_LAUNCH("mb_gemm_simt");
}

// C[M, N] (row stride ldc) = A[M, K] (row stride lda) · W[N, K]ᵀ. For EPI_ADD, C must be
// float32. For the SwiGLU epilogues, W is [2N, K]. `settled`: W was not written by the kernel just
// before in the stream, so that reading it need not wait for that kernel. `sms`: the number of SMs
// of the device.
MB_EXPORT int mb_gemm_simt(const void* A, int a_dtype, int lda, const void* W, int w_dtype,
                           void* C, int c_dtype, int ldc, int M, int N, int K, int epilogue,
                           int settled, int sms, void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) MB_FAIL("mb_gemm_simt: K = %d", K);
  if (epilogue < 0 || epilogue > 3) MB_FAIL("mb_gemm_simt: epilogue %d", epilogue);
  if (epilogue == EPI_ADD && c_dtype != MB_F32) MB_FAIL("mb_gemm_simt: the residual is float32");
  cudaStream_t s = (cudaStream_t)stream;
  typedef __nv_bfloat16 bf;
  const int c_bf16 = c_dtype == MB_BF16;
  if (a_dtype == MB_F32 && w_dtype == MB_F32)
    return launch<float, float>(A, lda, W, C, c_bf16, ldc, M, N, K, epilogue, settled, sms, s);
  if (a_dtype == MB_F32) return launch<float, bf>(A, lda, W, C, c_bf16, ldc, M, N, K, epilogue, settled, sms, s);
  if (w_dtype == MB_F32) return launch<bf, float>(A, lda, W, C, c_bf16, ldc, M, N, K, epilogue, settled, sms, s);
  return launch<bf, bf>(A, lda, W, C, c_bf16, ldc, M, N, K, epilogue, settled, sms, s);
}
