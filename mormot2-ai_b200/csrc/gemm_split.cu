// y = x · Wᵀ of float32 operands on the tensor cores, for more rows than gemm_simt.cu's kernel of
// few rows takes. Every float32 value from 2^-110 up is the exact sum of three bfloat16 parts of 8
// significant bits each (hi + mid + lo: its 24 bits cut in three), so a product of two values is a sum of nine
// products of parts; six of them are computed, the other three lie 2^-24 and less below the whole.
// (The method: G. Henry, P. Tang, A. Heinecke, Leveraging the bfloat16 artificial intelligence datatype
// for higher-precision computations, 2019.)
// tcgen05 multiplies exactly and adds in float32, but cuts off what falls behind the accumulator's
// last place instead of rounding. So no long sum is left to it: hi·hi is drained from tensor memory
// every 64 values of K and added up in registers, rounded to nearest; only the five products that
// stand 2^-8 and more below gather there over all of K. Error against float64, normal values, as a
// share of the result's norm, a chain of fma beside it: K of 128 1.2e-7 (2.0e-7), 1,024 1.3e-7
// (2.1e-7), 3,072 1.4e-7 (3.6e-7), 12,288 1.9e-7 (7.0e-7).
//
// Layout: 128 weight rows are the MMA's lanes, up to 128 rows of x its columns. x is cut once, by a
// kernel of its own, into three bfloat16 planes that TMA brings in (cut by every CTA that needs it,
// it took the cutting warps as long as the weight). The weight is cut on its way: per 32 values of K
// four warps load it straight from memory and store its parts in tensor memory (tcgen05.st 16x256b:
// four lanes hold 16 neighbouring values of a row, so the loads are whole sectors), where they are
// the MMA's first operand: read from shared memory, the twelve MMAs of a stage would ask for more
// than its 128 bytes a cycle. Two groups of four warps take the stages in turn, two warps issue, eight
// drain. What bounds it: the way of a stage round from the cutting warps to the MMAs and back (900 to
// 1,150 cycles; the MMAs themselves take 576 with 96 columns, 768 with 128), with two to four stages
// in tensor memory. Measured with inputs from memory, beside gemm_many_rows_kernel of gemm_simt.cu:
// 1,728 rows, 4,096 x 1,024 376 -> 93 us (156 TFLOP/s of float32 products), 1,024 x 3,072 316 -> 87,
// 6,144 x 1,024 with SwiGLU 525 -> 142; 24 rows, 1,024 x 2,048 41 -> 19; 400 rows 72 -> 28.
//
// Values that the parts do not sum up to (below 2^-110, where bits fall behind bfloat16's last place;
// infinities and NaNs) get a NaN for their lo, so that what they take part in comes out as a NaN of the
// smaller products' accumulator. Results that are no numbers, those and overflows, are made again by
// multiply-adds in the drain (`again`): a value's loss, and what it costs, stays with the rows that have
// it. The look at what a cut loses takes 1 to 2 in a hundred.
#include <cooperative_groups.h>

#include "attention_tc.cuh"

namespace cg = cooperative_groups;

MB_DEFINE_LAST_ERROR

enum { EPI_STORE = 0, EPI_ADD = 1, EPI_SWIGLU_PAIRS = 3 };

constexpr int GS_ROWS = 128;      // weight rows of a tile: the MMA's lanes
constexpr int GS_COLS = 128;      // rows of x of a tile, at most: the MMA's columns
constexpr int GS_K = 32;          // values of K of a stage of the weight
constexpr int GS_BK = 64;         // values of K of a stage of x
constexpr int GS_GROUP = 2;       // stages of the weight between two drains of hi·hi
constexpr int GS_A_MAX = 4, GS_B_MAX = 6;    // stages, at most
constexpr int GS_A_COLS = 3 * GS_K / 2;      // tensor memory of a stage: hi, mid, lo
constexpr int GS_THREADS = 32 * 20;  // 8 warps cut the weight, 8 drain, 1 loads, 2 issue, 1 has no part
constexpr int GS_SMEM = 200 * 1024;  // of the stages of x
constexpr uint32_t GS_NAN2 = 0x7fff7fffu;    // two bfloat16 NaNs

// 16 lanes x 16 columns of tensor memory: registers 4 j .. 4 j + 3 hold columns 8 j + 2 (lane % 4)
// and the next of row lane / 4, then of row lane / 4 + 8
__device__ __forceinline__ void tmem_st_rows16(uint32_t taddr, const uint32_t* w) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
      ::"r"(taddr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]),
        "r"(w[7])
      : "memory");
}

// Four values of a row from `at` on, of which the first `have` exist (all of them or none where VEC;
// the others read as zeros): predicated loads, since one behind a branch would be waited for where
// the branch ends.
template <bool VEC>
__device__ __forceinline__ float4 piece4(const float* at, int have) {
  float4 v;
  if (VEC) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %5, 0;\n\t"
        "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
        "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
        "@p ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}\n"
        : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w)
        : "l"(at), "r"(have));
  } else {
    float x[4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
      asm volatile(
          "{\n\t.reg .pred p;\n\tsetp.gt.s32 p, %2, 0;\n\t"
          "mov.f32 %0, 0f00000000;\n\t@p ld.global.nc.f32 %0, [%1];\n\t}\n"
          : "=&f"(x[i])
          : "l"(at + i), "r"(have - i));
    v = make_float4(x[0], x[1], x[2], x[3]);
  }
  return v;
}

// ---------------------------------------------------------------------------- x in parts
// planes [3][M][Kp] bfloat16 (hi, mid, lo; zeros from K to Kp) of A [M, K] with rows lda apart:
// eight values a thread, bound by its 10 bytes a value
template <bool VEC>
__global__ void __launch_bounds__(256)
cut_rows_kernel(const float* __restrict__ A, int lda, int M, int K, int Kp,
                __nv_bfloat16* __restrict__ planes) {
  mb_grid_wait();
  mb_grid_launch_next();
  const int per_row = Kp / 8;
  const long long total = (long long)M * per_row;
  for (long long i = blockIdx.x * 256ll + threadIdx.x; i < total; i += gridDim.x * 256ll) {
    const int m = (int)(i / per_row), k = 8 * (int)(i - (long long)m * per_row);
    const float* at = A + (size_t)m * lda + k;
    const float4 u = piece4<VEC>(at, K - k), v = piece4<VEC>(at + 4, K - k - 4);
    Cut2 c[4] = {cut(u.x, u.y), cut(u.z, u.w), cut(v.x, v.y), cut(v.z, v.w)};
    if (cut_is_inexact(c[0].rest | c[1].rest | c[2].rest | c[3].rest))
      c[0].lo = c[1].lo = c[2].lo = c[3].lo = GS_NAN2;
    uint4* out = (uint4*)(planes + (size_t)m * Kp + k);
    const size_t plane = (size_t)M * Kp / 8;
    out[0] = make_uint4(c[0].hi, c[1].hi, c[2].hi, c[3].hi);
    out[plane] = make_uint4(c[0].mid, c[1].mid, c[2].mid, c[3].mid);
    out[2 * plane] = make_uint4(c[0].lo, c[1].lo, c[2].lo, c[3].lo);
  }
}

// ---------------------------------------------------------------------------- the product
struct SplitArgs {
  const float *A, *W;
  void* C;
  int lda, ldc, c_bf16, M, NW, K, epi;
  int cols, a_stages, b_stages, splits, k_split, tiles_m, num_tiles, vec_a;
  int* error;
};

__device__ __forceinline__ void put_out(const SplitArgs& p, size_t at, float v) {
  if (p.c_bf16) ((__nv_bfloat16*)p.C)[at] = __float2bfloat16_rn(v);
  else ((float*)p.C)[at] = v;
}

// Whether a phase is over, without waiting for it
__device__ __forceinline__ bool mbar_test(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.b32 %0, 1, 0, p;\n\t}\n"
      : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
  return ok != 0;
}

// v[j] += the products of row `w` of the weight and row m + j of x over k_lo .. k_hi, by multiply-adds: 64
// values of K to a chain (one over all of K would round more often). All lanes of a warp, which share m.
template <bool VEC>
__device__ __forceinline__ void columns_again(const SplitArgs& p, const float* w, int m, int k_lo, int k_hi, float (&v)[8]) {
#pragma unroll 1
  for (int k = k_lo; k < k_hi; k += 64) {
    float u[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) u[j] = 0.f;
#pragma unroll 1
    for (int i = k; i < min(k + 64, k_hi); i += 4) {
      const float4 a = piece4<VEC>(w + i, k_hi - i);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float4 x = piece4<VEC>(p.A + (size_t)min(m + j, p.M - 1) * p.lda + i, k_hi - i);
        u[j] = fmaf(x.x, a.x, fmaf(x.y, a.y, fmaf(x.z, a.z, fmaf(x.w, a.w, u[j]))));
      }
    }
    bool number = false;      // a NaN stays one
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      v[j] += u[j];
      number |= v[j] == v[j];
    }
    if (!__any_sync(0xffffffffu, number)) return;
  }
}

template <bool VEC>
__global__ void __launch_bounds__(GS_THREADS, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap tm_x, const SplitArgs p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  const uint32_t tile_bytes = p.cols * 128, b_stage = 3 * tile_bytes;      // hi, mid, lo
  const uint32_t bars = base + max(p.b_stages * b_stage, p.splits > 1 ? p.cols * GS_ROWS * 4u : 0u);
  const uint32_t a_full0 = bars, a_empty0 = a_full0 + 8 * GS_A_MAX;
  const uint32_t b_full0 = a_empty0 + 8 * GS_A_MAX, b_empty0 = b_full0 + 8 * GS_B_MAX;
  const uint32_t main_full0 = b_empty0 + 8 * GS_B_MAX, main_empty0 = main_full0 + 16;
  const uint32_t low_full = main_empty0 + 16, low_empty = low_full + 8, slot = low_empty + 8;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < p.a_stages; ++s) {
      mbar_init(a_full0 + 8 * s, 4);
      mbar_init(a_empty0 + 8 * s, 2);
    }
    for (int s = 0; s < p.b_stages; ++s) {
      mbar_init(b_full0 + 8 * s, 1);
      mbar_init(b_empty0 + 8 * s, 2);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(main_full0 + 8 * b, 1);
      mbar_init(main_empty0 + 8 * b, 8);
    }
    mbar_init(low_full, 1);
    mbar_init(low_empty, 8);
    mbar_fence_init();
    tma_prefetch_desc(&tm_x);
  }
  if (warp == 17) tmem_alloc(slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *(volatile uint32_t*)(smem_raw + (slot - raw));
  // hi·hi of two groups in turn, the other products, the weight's parts of every stage
  const uint32_t t_main = tmem, t_low = tmem + 2 * p.cols, t_a = tmem + 3 * p.cols;

  // a CTA's work: whole tiles in turn, or one tile's share of K (a cluster shares a tile)
  const int split = blockIdx.x % p.splits;
  const int tile0 = blockIdx.x / p.splits, tile_step = gridDim.x / p.splits;
  const int k_lo = split * p.k_split, k_hi = min(p.K, k_lo + p.k_split);
  const int nkb = (k_hi - k_lo + GS_K - 1) / GS_K;
  const int groups = (nkb + GS_GROUP - 1) / GS_GROUP;
  // x comes from the kernel before (cut_rows_kernel), which began after the one before it had ended:
  // the weight, which cut_rows_kernel does not write, need not wait
  if (warp >= 8 && warp != 16) mb_grid_wait();
  mb_grid_launch_next();

  // Registers: 96 a thread at the start (61,440 in all). The four warps that load and issue give
  // theirs to the eight that cut: 256 x 120 + 256 x 96 + 128 x 40 = 60,416.
  if (warp < 8) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 120;");
    // Two groups of four warps take the stages in turn. Piece 4 h + 2 j + i of a thread is row
    // 32 w + 16 h + lane / 4 + 8 i, k 16 j + 4 (lane % 4).
    const int w = warp & 3, turn = warp >> 2;
    const size_t step8 = (size_t)8 * p.K;
    int tile = tile0, kb = turn;      // the stage that this group fetches next
    const float* row0 = nullptr;
    int rows = 0;      // weight rows from this thread's first on
    auto enter = [&]() {
      while (kb >= nkb && tile < p.num_tiles) { kb -= nkb; tile += tile_step; }
      if (tile < p.num_tiles) {
        const int n = (tile / p.tiles_m) * GS_ROWS + 32 * w + (lane >> 2);
        rows = p.NW - n;
        row0 = p.W + (size_t)n * p.K + k_lo + 4 * (lane & 3);
      }
    };
    float4 r[8];
    auto fetch = [&](int h) {
      const int left = k_hi - k_lo - kb * GS_K - 4 * (lane & 3);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const int dr = 2 * h + (i & 1), dk = 16 * (i >> 1);
        r[4 * h + i] = piece4<VEC>(row0 + dr * step8 + kb * GS_K + dk, 8 * dr < rows ? left - dk : 0);
      }
    };
    enter();
    bool more = tile < p.num_tiles;
    if (more) {
      fetch(0);
      fetch(1);
    }
    int st = turn % p.a_stages, it = turn;
    while (more) {
      kb += 2;
      if (kb >= nkb) enter();
      more = tile < p.num_tiles;
      const uint32_t ph = ((it / p.a_stages) & 1) ^ 1;
      uint32_t hi[16], mid[16], lo[16], rest = 0;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 4 * h; i < 4 * h + 4; ++i) {
          const Cut2 a = cut(r[i].x, r[i].y), b = cut(r[i].z, r[i].w);
          hi[2 * i] = a.hi; mid[2 * i] = a.mid; lo[2 * i] = a.lo;
          hi[2 * i + 1] = b.hi; mid[2 * i + 1] = b.mid; lo[2 * i + 1] = b.lo;
          rest |= a.rest | b.rest;
        }
        if (more) fetch(h);
      }
      if (cut_is_inexact(rest)) {      // somewhere in this thread's four rows
#pragma unroll
        for (int i = 0; i < 16; ++i) lo[i] = GS_NAN2;
      }
      __syncwarp();
      mbar_wait(a_empty0 + 8 * st, ph, p.error, 41);
      tc_fence_after_sync();
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const uint32_t ta = t_a + st * GS_A_COLS + ((uint32_t)(32 * w + 16 * h) << 16);
        tmem_st_rows16(ta, hi + 8 * h);
        tmem_st_rows16(ta + GS_K / 2, mid + 8 * h);
        tmem_st_rows16(ta + GS_K, lo + 8 * h);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(a_full0 + 8 * st);
      it += 2;
      st += 2;
      while (st >= p.a_stages) st -= p.a_stages;
    }
  } else if (warp >= 16) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 40;");
    if (warp == 16) {
    if (elect_one()) {
      // A tile's weight rows into L2 ahead of their use: the CTAs that work on the same rows ask for
      // them at the same time, which leaves few bytes of memory's under way (1,728 rows, 1,024 x 2,048
      // from memory: 65 us without). They share the rows out among them.
      auto ahead = [&](int tile) {
        if (!VEC || tile >= p.num_tiles) return;
        const int n = min(8, p.tiles_m), n0 = (tile / p.tiles_m) * GS_ROWS;
        const int end = min(p.NW, n0 + GS_ROWS);
        for (int row = n0 + tile % p.tiles_m % n; row < end; row += n)
          asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;"
                       ::"l"(p.W + (size_t)row * p.K + k_lo), "r"((k_hi - k_lo) * 4) : "memory");
      };
      ahead(tile0);
      mb_grid_wait();
      int st = 0;
      uint32_t ph = 1;
      for (int tile = tile0; tile < p.num_tiles; tile += tile_step) {
        ahead(tile + tile_step);
        const int m0 = (tile % p.tiles_m) * p.cols;
        for (int k = k_lo; k < k_hi; k += GS_BK) {
          mbar_wait(b_empty0 + 8 * st, ph, p.error, 47);
          mbar_expect_tx(b_full0 + 8 * st, b_stage);
#pragma unroll
          for (int part = 0; part < 3; ++part)      // rows beyond M are another part's: never stored
            tma_load_2d(base + st * b_stage + part * tile_bytes, &tm_x, k, part * p.M + m0,
                        b_full0 + 8 * st);
          if (++st == p.b_stages) { st = 0; ph ^= 1; }
        }
      }
    }
    __syncwarp();
    } else if (warp < 19) {
    // Two warps issue, each in its own accumulators: warp 17 hi·hi, warp 18 the other products. What a
    // stage costs an issuing thread (its waits, its commits, a dozen instructions an MMA) is about
    // what the MMAs themselves take; one warp for all of them: 1,690 cycles a stage.
    const bool is_main = warp == 17, one = elect_one();
    const uint32_t idesc = umma_idesc_bf16(GS_ROWS, p.cols);
    constexpr uint32_t MID = GS_K / 2, LO = GS_K;
    int sa = 0, sb = 0, g = 0;
    uint32_t pa = 0, pb = 0, low_ph = 1;
    bool a_here = false, b_here = false;      // the next stage has been seen full already
    for (int tile = tile0; tile < p.num_tiles; tile += tile_step) {
      if (!is_main) {
        mbar_wait(low_empty, low_ph, p.error, 44);
        low_ph ^= 1;
      }
#pragma unroll 1
      for (int kb = 0; kb < nkb; ++kb) {
        const bool first = kb % GS_GROUP == 0, last = kb == nkb - 1, b_done = (kb & 1) || last;
        if (!(kb & 1) && !b_here) mbar_wait(b_full0 + 8 * sb, pb, p.error, 48);
        if (is_main && first) mbar_wait(main_empty0 + 8 * (g & 1), ((g >> 1) & 1) ^ 1, p.error, 43);
        if (!a_here) mbar_wait(a_full0 + 8 * sa, pa, p.error, 42);
        tc_fence_after_sync();
        const uint32_t ta = t_a + sa * GS_A_COLS;
        const uint32_t a_bar = a_empty0 + 8 * sa, b_bar = b_empty0 + 8 * sb;
        const uint64_t b_hi = umma_desc_k128(base + sb * b_stage + (kb & 1) * 64);
        // a look at the next stage, whose answer comes while this stage's products are issued
        if (++sa == p.a_stages) { sa = 0; pa ^= 1; }
        if (b_done && ++sb == p.b_stages) { sb = 0; pb ^= 1; }
        a_here = mbar_test(a_full0 + 8 * sa, pa);
        b_here = b_done && mbar_test(b_full0 + 8 * sb, pb);
        if (is_main) {
          const uint32_t tm = t_main + (g & 1) * p.cols;
          const bool group_done = kb % GS_GROUP == GS_GROUP - 1 || last;
          if (one) {
#pragma unroll
            for (int k = 0; k < GS_K / 16; ++k)
              umma_bf16_ts(tm, ta + 8 * k, b_hi + 2 * k, idesc, !first || k > 0);
            if (group_done) umma_commit(main_full0 + 8 * (g & 1));
            umma_commit(a_bar);
            if (b_done) umma_commit(b_bar);
          }
          if (group_done) ++g;
        } else if (one) {
          const uint64_t b_mid = b_hi + (tile_bytes >> 4), b_lo = b_mid + (tile_bytes >> 4);
#pragma unroll
          for (int k = 0; k < GS_K / 16; ++k) {
            umma_bf16_ts(t_low, ta + LO + 8 * k, b_hi + 2 * k, idesc, kb > 0 || k > 0);
            umma_bf16_ts(t_low, ta + 8 * k, b_lo + 2 * k, idesc, 1);
            umma_bf16_ts(t_low, ta + MID + 8 * k, b_mid + 2 * k, idesc, 1);
            umma_bf16_ts(t_low, ta + MID + 8 * k, b_hi + 2 * k, idesc, 1);
            umma_bf16_ts(t_low, ta + 8 * k, b_mid + 2 * k, idesc, 1);
          }
          umma_commit(a_bar);
          if (b_done) umma_commit(b_bar);
          if (last) umma_commit(low_full);
        }
      }
    }
    __syncwarp();
    }
  } else {
    // lanes 32 (warp % 4) .. + 31, columns of one half: 16 i of them where i < parts
    const int q = warp & 3, half = (warp - 8) >> 2;
    const int c0 = half ? (p.cols / 16 + 1) / 2 * 16 : 0;
    const int parts = half ? p.cols / 32 : (p.cols / 16 + 1) / 2;
    const uint32_t lanes = ((uint32_t)(32 * q) << 16) + c0;
    const int row = 32 * q + lane;
    int g = 0;
    uint32_t low_ph = 0;
    // Results that are no numbers, by multiply-adds over this CTA's share of K, eight columns at a time, so
    // that a weight's values serve them all. 1,728 rows, 4,096 x 1,024: 0.1 ms without, 2.1 where every
    // row has such a value (a lane a result at a time: 27, and other warps' waits are limited).
    auto again = [&](float (&s)[4][16], int tile) {
      float t[64];
#pragma unroll
      for (int i = 0; i < 64; ++i) t[i] = s[i / 16][i % 16];
      const int n = (tile / p.tiles_m) * GS_ROWS + row, m0 = (tile % p.tiles_m) * p.cols + c0;
      const int valid = n < p.NW ? min(16 * parts, p.M - m0) : 0;      // this lane's results that are stored
      const float* w = p.W + (size_t)min(n, p.NW - 1) * p.K;
#pragma unroll 1
      for (int g = 0; g < 2 * parts; ++g) {
        bool bad = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) bad |= 8 * g + j < valid && !(fabsf(t[8 * g + j]) <= 3.402823466e38f);
        if (!__any_sync(0xffffffffu, bad)) continue;
        float v[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) v[j] = 0.f;
        if (VEC && p.vec_a) columns_again<true>(p, w, m0 + 8 * g, k_lo, k_hi, v);
        else columns_again<false>(p, w, m0 + 8 * g, k_lo, k_hi, v);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (!(fabsf(t[8 * g + j]) <= 3.402823466e38f)) t[8 * g + j] = v[j];
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 64; ++i) s[i / 16][i % 16] = t[i];
    };
    for (int tile = tile0; tile < p.num_tiles; tile += tile_step) {
      float s[4][16];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 16; ++j) s[i][j] = 0.f;
      for (int n = 0; n < groups; ++n, ++g) {
        mbar_wait(main_full0 + 8 * (g & 1), (g >> 1) & 1, p.error, 45);
        tc_fence_after_sync();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if (i < parts) {
            float v[16];
            tmem_ld16(t_main + (g & 1) * p.cols + lanes + 16 * i, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) s[i][j] += v[j];
          }
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(main_empty0 + 8 * (g & 1));
      }
      mbar_wait(low_full, low_ph, p.error, 46);
      low_ph ^= 1;
      tc_fence_after_sync();
      float no_number = 0.f;      // turns NaN
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        if (i < parts) {
          float v[16];
          tmem_ld16(t_low + lanes + 16 * i, v);
#pragma unroll
          for (int j = 0; j < 16; ++j) {
            s[i][j] += v[j];
            no_number = fmaf(s[i][j], 0.f, no_number);
          }
        }
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(low_empty);
      if (__any_sync(0xffffffffu, no_number != 0.f)) again(s, tile);
      if (p.splits > 1) {      // [rows of x][weight rows], over the stages that nobody reads any more
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (i < parts)
              *(float*)(smem_raw + (base - raw) + ((c0 + 16 * i + j) * GS_ROWS + row) * 4) = s[i][j];
        continue;
      }
      // A loop per form, each with little code: 64 results a thread, unrolled, with the choice of the
      // form inside took 15,000 cycles, most of them for instructions that no cache held.
      const int n = (tile / p.tiles_m) * GS_ROWS + row, m0 = (tile % p.tiles_m) * p.cols + c0;
      const bool pairs = p.epi == EPI_SWIGLU_PAIRS;
      const int left = n < p.NW ? min(16 * parts, p.M - m0) : 0;
      const size_t at = (size_t)m0 * p.ldc + (pairs ? n >> 1 : n);
      if (pairs) {
        // gate in the even lane, up in the odd one: of two rows of x each takes the one, so that
        // both have a result to finish
        const bool odd = lane & 1;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 16; j += 2) {
            const float got = __shfl_xor_sync(0xffffffffu, odd ? s[i][j] : s[i][j + 1], 1);
            const float g = odd ? got : s[i][j], up = odd ? s[i][j + 1] : got;
            if (16 * i + j + odd < left)
              put_out(p, at + (size_t)(16 * i + j + odd) * p.ldc, g / (1.0f + expf(-g)) * up);
          }
      } else if (p.c_bf16) {
        __nv_bfloat16* out = (__nv_bfloat16*)p.C + at;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 16; ++j)
            if (16 * i + j < left) out[(size_t)(16 * i + j) * p.ldc] = __float2bfloat16_rn(s[i][j]);
      } else {
        float* out = (float*)p.C + at;
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 16; j += 8) {
            if (p.epi == EPI_ADD) {
              float old[8];
#pragma unroll
              for (int u = 0; u < 8; ++u) old[u] = 16 * i + j + u < left ? out[(size_t)u * p.ldc] : 0.f;
#pragma unroll
              for (int u = 0; u < 8; ++u) s[i][j + u] = old[u] + s[i][j + u];
            }
#pragma unroll
            for (int u = 0; u < 8; ++u)
              if (16 * i + j + u < left) out[(size_t)u * p.ldc] = s[i][j + u];
            out += 8 * (size_t)p.ldc;
          }
      }
    }
  }
  __syncthreads();
  if (warp == 17) tmem_dealloc(tmem, 512);
  if (p.splits == 1) return;
  // a tile's sums over the cluster's shares of K, in K's order
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  float* sums = (float*)(smem_raw + (base - raw));
  const int n0 = (tile0 / p.tiles_m) * GS_ROWS, m0 = (tile0 % p.tiles_m) * p.cols;
  constexpr int step = 4 * 512;      // by the warps that have their registers still
  for (int e = 4 * threadIdx.x + split * step; warp < 16 && e < p.cols * GS_ROWS; e += step * p.splits) {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < p.splits; ++k) {
      const float4 o = *(const float4*)(cluster.map_shared_rank(sums, k) + e);
      v.x += o.x; v.y += o.y; v.z += o.z; v.w += o.w;
    }
    const int m = m0 + e / GS_ROWS, n = n0 + e % GS_ROWS;
    if (m >= p.M) continue;
    const float c[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (n + j >= p.NW) break;
      if (p.epi == EPI_SWIGLU_PAIRS) {
        if (!(j & 1))
          put_out(p, (size_t)m * p.ldc + ((n + j) >> 1), c[j] / (1.0f + expf(-c[j])) * c[(j + 1) & 3]);
      } else {
        const size_t at = (size_t)m * p.ldc + n + j;
        put_out(p, at, p.epi == EPI_ADD ? ((const float*)p.C)[at] + c[j] : c[j]);
      }
    }
  }
  cluster.sync();      // nobody leaves while its sums are still read
}

typedef void (*SplitKernel)(CUtensorMap, SplitArgs);

// How many clusters of `n` CTAs run at once on the current device: 148 SMs hold 45 of 3, 33 of 4, 15
// of 7 or 8, since a cluster stays within a group of SMs. Asked for once a device and size.
static int clusters_at_once(SplitKernel kernel, int n, int smem) {
  static int known[64][9];
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return 0;
  const bool keep = device >= 0 && device < 64;
  if (keep) {
    const int v = __atomic_load_n(&known[device][n], __ATOMIC_RELAXED);
    if (v) return v - 1;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(n);
  cfg.blockDim = dim3(GS_THREADS);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = n;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int v = 0;
  if (cudaOccupancyMaxActiveClusters(&v, kernel, &cfg) != cudaSuccess) return 0;
  if (keep) __atomic_store_n(&known[device][n], v + 1, __ATOMIC_RELAXED);
  return v;
}

// The values of a row of the planes: K up to whole 16 bytes.
static long long padded_k(int K) { return (K + 7ll) / 8 * 8; }

// Bytes of scratch of a product of M rows, with no more than `most` (but one row's).
MB_EXPORT long long mb_gemm_split_scratch(int M, int K, long long most) {
  const long long row = 6 * padded_k(K), fit = most / row;
  return row * (M <= fit ? M : fit >= GS_COLS ? fit / GS_COLS * GS_COLS : fit > 0 ? fit : 1);
}

// M rows whose parts fit into the scratch: the two kernels
static int split_rows(const void* A, int lda, const void* W, void* C, int c_dtype, int ldc, int M, int N,
                      int K, int epilogue, int sms, int force_cols, int force_splits, void* scratch,
                      void* error, cudaStream_t s) {
  const int Kp = (int)padded_k(K);
  SplitArgs p;
  p.A = (const float*)A; p.W = (const float*)W; p.C = C;
  p.lda = lda; p.ldc = ldc; p.c_bf16 = c_dtype == MB_BF16; p.M = M; p.K = K; p.epi = epilogue;
  p.NW = epilogue == EPI_SWIGLU_PAIRS ? 2 * N : N;
  p.error = (int*)error;
  const int tiles_n = (p.NW + GS_ROWS - 1) / GS_ROWS;
  const bool vec_w = K % 4 == 0 && ((uintptr_t)W & 15) == 0;
  const bool vec_a = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A & 15) == 0;
  p.vec_a = vec_a;
  const SplitKernel kernel = vec_w ? gemm_split_kernel<true> : gemm_split_kernel<false>;
  static unsigned long long allowed[2] = {0, 0};
  cudaError_t e = mb_allow_smem((const void*)kernel, GS_SMEM + 2048, &allowed[vec_w]);
  if (e != cudaSuccess) MB_FAIL("mb_gemm_split: %s", cudaGetErrorString(e));
  double best = 1e30;
  p.cols = p.splits = 0;
  for (int cols = 16; cols <= GS_COLS; cols += 16) {
    if (force_cols && cols != force_cols) continue;
    const long long tiles = (long long)tiles_n * ((M + cols - 1) / cols);
    for (int splits = 1; splits <= 8 && (splits == 1 || K >= 128 * splits); ++splits) {
      if (force_splits && splits != force_splits) continue;
      // a cluster a tile, all of them at once
      if (!force_splits && splits > 1 && tiles > clusters_at_once(kernel, splits, GS_SMEM + 2048)) continue;
      const long long rounds = splits > 1 ? 1 : (tiles + sms - 1) / sms;
      // cycles: what a stage takes the warps that cut and issue, or its products; a tile's beginning
      // and end; the sums' way through the cluster (fitted to 17 to 3,000 rows of the sizes above)
      const double stage = cols <= 96 ? 900.0 : 190.0 + 7.4 * cols;
      const double cost = rounds * (((K + splits - 1) / splits + GS_K - 1) / GS_K * stage + 2000.0) +
                          (splits > 1 ? 2000.0 : 0.0) + 0.5 * tiles * splits;
      if (cost < best) { best = cost; p.cols = cols; p.splits = splits; }
    }
  }
  if (!p.cols) MB_FAIL("mb_gemm_split: no plan with %d columns and %d splits", force_cols, force_splits);
  p.k_split = ((K + p.splits - 1) / p.splits + GS_BK - 1) / GS_BK * GS_BK;
  p.splits = (K + p.k_split - 1) / p.k_split;
  p.tiles_m = (M + p.cols - 1) / p.cols;
  const long long tiles = (long long)tiles_n * p.tiles_m;
  if (tiles * p.splits > 0x7fffffff) MB_FAIL("mb_gemm_split: %d rows are too many for one launch", M);
  p.num_tiles = (int)tiles;
  p.a_stages = (512 - 3 * p.cols) / GS_A_COLS;
  if (p.a_stages > GS_A_MAX) p.a_stages = GS_A_MAX;
  p.b_stages = GS_SMEM / (3 * 128 * p.cols);
  if (p.b_stages > GS_B_MAX) p.b_stages = GS_B_MAX;
  const int stages = p.b_stages * 3 * 128 * p.cols, sums = p.splits > 1 ? p.cols * GS_ROWS * 4 : 0;
  const int smem = 1024 + (stages > sums ? stages : sums) + 512;
  CUtensorMap map;
  if (!mb_make_map_bf16(&map, scratch, 3ll * M, Kp, Kp, p.cols, "mb_gemm_split")) return -1;
  const long long pieces = (long long)M * (Kp / 8), blocks = (pieces + 255) / 256;
  e = mb_launch(vec_a ? cut_rows_kernel<true> : cut_rows_kernel<false>,
                dim3((unsigned)(blocks < 16 * sms ? blocks : 16 * sms)), dim3(256), 0, s, (const float*)A,
                lda, M, K, Kp, (__nv_bfloat16*)scratch);
  if (e != cudaSuccess) MB_FAIL("mb_gemm_split: %s", cudaGetErrorString(e));
  const int grid = p.splits > 1 ? p.num_tiles * p.splits : (p.num_tiles < sms ? p.num_tiles : sms);
  if (p.splits > 1)
    mb_launch_clusters(kernel, dim3(grid), dim3(GS_THREADS), smem, s, p.splits, map, p);
  else
    mb_launch(kernel, dim3(grid), dim3(GS_THREADS), smem, s, map, p);
  MB_CHECK_LAUNCH("mb_gemm_split");
}

// C[M, N] (row stride ldc) = A[M, K] (row stride lda) · W[N, K]ᵀ, all float32 (C may be bfloat16,
// except for EPI_ADD). For EPI_SWIGLU_PAIRS, W is [2N, K] and its rows alternate gate and up.
// `scratch`: on a 16-byte boundary, mb_gemm_split_scratch bytes; with less than all rows' room the rows
// go in bands, one after the other through the same scratch (a band's cut waits for the product
// before it). `force_cols`, `force_splits`: 0 for the rule's choice.
MB_EXPORT int mb_gemm_split(const void* A, int lda, const void* W, void* C, int c_dtype, int ldc,
                            int M, int N, int K, int epilogue, int sms, int force_cols,
                            int force_splits, void* scratch, long long scratch_bytes, void* error,
                            void* stream) {
  if (M <= 0 || N <= 0) return 0;
  if (K <= 0) MB_FAIL("mb_gemm_split: K = %d", K);
  if (epilogue != EPI_STORE && epilogue != EPI_ADD && epilogue != EPI_SWIGLU_PAIRS)
    MB_FAIL("mb_gemm_split: epilogue %d", epilogue);
  if (epilogue == EPI_ADD && c_dtype != MB_F32) MB_FAIL("mb_gemm_split: the residual is float32");
  const long long fit = scratch_bytes / (6 * padded_k(K));
  if (fit < 1) MB_FAIL("mb_gemm_split: %lld bytes of scratch, a row needs %lld", scratch_bytes, 6 * padded_k(K));
  if ((fit < M ? fit : M) > 0x7fffffff / 3) MB_FAIL("mb_gemm_split: %d rows are too many for one launch", M);
  for (long long m = 0; m < M; m += fit) {
    const int rows = (int)(M - m < fit ? M - m : fit);
    const int rc = split_rows((const float*)A + m * lda, lda, W,
                              (char*)C + m * ldc * (c_dtype == MB_BF16 ? 2 : 4), c_dtype, ldc, rows, N, K,
                              epilogue, sms, force_cols, force_splits, scratch, error, (cudaStream_t)stream);
    if (rc) return rc;
  }
  return 0;
}
