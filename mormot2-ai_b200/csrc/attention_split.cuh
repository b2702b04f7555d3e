// Causal attention of many new tokens in float32 on the tensor cores, for heads of 128 values: every
// float32 value is cut into three bfloat16 parts that sum up to it (common.cuh), and both products are sums of six
// products of parts, as in gemm_split.cu. 128 new tokens of one sequence and one head per CTA, a
// page of 64 keys at a time.
//
// q's parts lie in tensor memory (192 columns) and are the scores' first operand for all pages. Eight
// warps cut a page's keys and values into shared memory; one thread issues; four warps, a row a
// thread, turn scores into probabilities, cut them and put them in tensor memory over the scores they
// came from; the eight warps add the page's part of the output to what they hold in registers, 64
// values of a row a thread. tcgen05 cuts off what falls behind an accumulator's last place instead
// of rounding, so no long sum is left to it: the scores' leading products go 64 values of the head to
// an accumulator (two, and one for all the rest), the output's a page; sums over those are float32
// additions. The softmax is the float32 kernel's, with all its options.
//
// A CTA whose inputs may be no exact sums of three parts (values below 2^-110, infinities, NaNs) or whose
// results are no numbers somewhere (an overflow, a row that sees no key) says so in `redo`, and
// attention_many_kernel, launched behind, does that tile again. A probability below 2^-110 may lose up
// to 2^-133, beside a sum of at least one.
//
// What bounds it: a page's chain, products of scores, softmax (64 exponentials and cuts a thread), products
// of values, one after the other, since tensor memory has no room for a second tile. 1,728 tokens of
// three prompts, 16 heads on 8: 321 us with multiply-adds, 105 here; 2,048 of one 693 -> 174.
#pragma once
#include "attention_simt.cuh"
#include "attention_tc.cuh"

constexpr int AS_ROWS = 128;
constexpr int AS_THREADS = 32 * 13;                 // 8 warps cut and hold the output, 4 softmax, 1 issues
constexpr int AS_HALF = MB_PAGE * 128;              // 64 keys x 64 values of a part
constexpr int AS_PART = 2 * AS_HALF;
constexpr int AS_TILE = 3 * AS_PART;                // a page's keys (or values): hi, mid, lo
constexpr int AS_SMEM = 1024 + 3 * AS_TILE + 2 * AS_ROWS * 4 + AS_ROWS * 4 + 256;
constexpr uint32_t AS_TQ = 0, AS_TS = 192, AS_TO = 384;      // tensor memory: q, scores (and p), output

__device__ __forceinline__ void as_st_rows16(uint32_t taddr, const uint32_t* w) {
  asm volatile(
      "tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};\n"
      ::"r"(taddr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]),
        "r"(w[7])
      : "memory");
}
__device__ __forceinline__ void as_st_v2(uint32_t addr, uint32_t a, uint32_t b) {
  asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ float4 as_load4(const float* at, bool ok) {
  float4 v;      // predicated: a load behind a branch would be waited for where the branch ends
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %5, 0;\n\t"
      "mov.f32 %0, 0f00000000;\n\tmov.f32 %1, 0f00000000;\n\t"
      "mov.f32 %2, 0f00000000;\n\tmov.f32 %3, 0f00000000;\n\t"
      "@p ld.global.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}\n"
      : "=&f"(v.x), "=&f"(v.y), "=&f"(v.z), "=&f"(v.w)
      : "l"(at), "r"((int)ok)
      : "memory");
  return v;
}
__device__ __forceinline__ bool as_no_number(float4 v) {
  return !(0.f * v.x + 0.f * v.y + 0.f * v.z + 0.f * v.w == 0.f);
}

__global__ void __launch_bounds__(AS_THREADS, 1)
attention_split_kernel(const AttArgs<float> a, int fewest, int* __restrict__ redo, int* __restrict__ error) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
  const uint32_t sK = base, sV = base + 2 * AS_TILE;      // two pages of keys, one of values
  float* corr = (float*)(smem_raw + (base - raw) + 3 * AS_TILE);      // [2][128] of a page's turn
  float* sums = corr + 2 * AS_ROWS;                                    // [128] the rows' sums at the end
  const uint32_t bars = base + 3 * AS_TILE + 3 * AS_ROWS * 4;
  const uint32_t q_full = bars, k_full0 = bars + 8, v_full = bars + 24, s_done = bars + 32, o_done = bars + 40,
                 o_read = bars + 48, p_full0 = bars + 56, slot = bars + 72;
  volatile uint32_t* slot_ptr = (volatile uint32_t*)(smem_raw + (slot - raw));
  int* bad = (int*)(smem_raw + (slot - raw) + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    mbar_init(q_full, 8);
    mbar_init(k_full0, 8);
    mbar_init(k_full0 + 8, 8);
    mbar_init(v_full, 8);
    mbar_init(s_done, 1);
    mbar_init(p_full0, 4);
    mbar_init(p_full0 + 8, 4);
    mbar_init(o_done, 1);
    mbar_init(o_read, 8);
    mbar_fence_init();
    *bad = 0;
  }
  mb_grid_wait();
  mb_grid_launch_next();
  const int h = blockIdx.x, g = h / (a.nh / a.nkv), b = blockIdx.z;
  const int t0 = a.seq_start[b], n_new = a.seq_start[b + 1] - t0;
  const int tiles = (n_new + AS_ROWS - 1) / AS_ROWS;
  if ((int)blockIdx.y >= tiles || n_new < fewest) return;
  const int tile = tiles - 1 - blockIdx.y, r0 = tile * AS_ROWS;      // the tiles that see the most keys first
  const int cnt = min(AS_ROWS, n_new - r0);
  const int seq_slot = a.seq_slot[b], p0 = a.tok_pos[t0 + r0], last = p0 + cnt - 1;
  if (warp == 12) tmem_alloc(slot, 512);
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *slot_ptr;
  // pages that some row sees: those of the kept first positions, then from the first row's window
  const int lo0 = a.window > 0 ? max(0, p0 + 1 - a.window) : 0;
  const int first_page = lo0 / MB_PAGE, kept_pages = min((a.keep_first + MB_PAGE - 1) / MB_PAGE, first_page);
  const int pages = kept_pages + last / MB_PAGE - first_page + 1;
  auto page_of = [&](int j) { return j < kept_pages ? j : first_page + j - kept_pages; };

  if (warp < 8) {
    const int w = warp & 3, half = warp >> 2;
    bool odd = false;
    {
      // q: rows 32 w + 16 half + lane / 4 (+ 8), 16 values to four lanes
      const int row = 32 * w + 16 * half + (lane >> 2);
      const float* at = a.q + (size_t)(t0 + r0 + row) * a.q_stride + (size_t)h * 128 + 4 * (lane & 3);
#pragma unroll
      for (int kb = 0; kb < 4; ++kb) {
        uint32_t hi[8], mid[8], lo[8];
        float4 v[4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
          v[i] = as_load4(at + (size_t)(8 * (i & 1)) * a.q_stride + 32 * kb + 16 * (i >> 1), row + 8 * (i & 1) < cnt);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          odd |= as_no_number(v[i]) | too_small_to_cut(v[i]);
          const Cut2 x = cut(v[i].x, v[i].y), y = cut(v[i].z, v[i].w);
          hi[2 * i] = x.hi; mid[2 * i] = x.mid; lo[2 * i] = x.lo;
          hi[2 * i + 1] = y.hi; mid[2 * i + 1] = y.mid; lo[2 * i + 1] = y.lo;
        }
        const uint32_t ta = tmem + AS_TQ + 16 * kb + ((uint32_t)(32 * w + 16 * half) << 16);
        as_st_rows16(ta, hi);
        as_st_rows16(ta + 64, mid);
        as_st_rows16(ta + 128, lo);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(q_full);
    }
    // a page's rows of `pool`, eight pieces of four values a thread: a row a warp at a time
    float4 r[8];
    auto fetch = [&](const float* pool, int j) {
      const int k0 = page_of(j) * MB_PAGE, keys = min(MB_PAGE, last + 1 - k0);
      const size_t row = kv_row(a.page_table, a.max_pages, a.ring_pages, seq_slot, k0, a.nkv, g);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        r[i] = as_load4(pool + (row + warp + 8 * i) * 128 + 4 * lane, warp + 8 * i < keys);
    };
    auto put = [&](uint32_t to) {
      const uint32_t at = to + (lane >> 4) * AS_HALF + (lane & 1) * 8, ch = (lane & 15) >> 1;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int row = warp + 8 * i;
        odd |= as_no_number(r[i]) | too_small_to_cut(r[i]);
        const Cut2 x = cut(r[i].x, r[i].y), y = cut(r[i].z, r[i].w);
        const uint32_t p = at + row * 128 + ((ch ^ (row & 7)) << 4);
        as_st_v2(p, x.hi, y.hi);
        as_st_v2(p + AS_PART, x.mid, y.mid);
        as_st_v2(p + 2 * AS_PART, x.lo, y.lo);
      }
      fence_async_smem();
      __syncwarp();
    };
    fetch(a.kpool, 0);
    put(sK);
    if (lane == 0) mbar_arrive(k_full0);
    float o[64];
#pragma unroll
    for (int i = 0; i < 64; ++i) o[i] = 0.f;
    const uint32_t tO = tmem + AS_TO + 64 * half + ((uint32_t)(32 * w) << 16);
    fetch(a.vpool, 0);
    for (int j = 0; j < pages; ++j) {
      put(sV);      // the page before has been multiplied: its output has been read
      if (lane == 0) mbar_arrive(v_full);
      if (j + 1 < pages) {
        fetch(a.kpool, j + 1);
        put(sK + ((j + 1) & 1) * AS_TILE);      // the keys of page j - 1: multiplied before page j - 1's values
        if (lane == 0) mbar_arrive(k_full0 + 8 * ((j + 1) & 1));
        fetch(a.vpool, j + 1);
      }
      mbar_wait(p_full0 + 8 * (j & 1), (j >> 1) & 1, error, 51);      // the page's corrections are there
      const float c = corr[(j & 1) * AS_ROWS + 32 * w + lane];
      mbar_wait(o_done, j & 1, error, 52);
      tc_fence_after_sync();
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float v[16];
        tmem_ld16(tO + 16 * i, v);
#pragma unroll
        for (int e = 0; e < 16; ++e) o[16 * i + e] = fmaf(o[16 * i + e], c, v[e]);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(o_read);
    }
    asm volatile("bar.sync 1, 384;" ::: "memory");      // the rows' sums are there
    const int row = 32 * w + lane, t = t0 + r0 + row;
    if (row < cnt) {
      const float inv = 1.f / sums[row];
      float* out = a.out + (size_t)t * a.out_stride + (size_t)h * 128 + 64 * half;
      if (a.gate) {
#pragma unroll
        for (int i = 0; i < 64; ++i) o[i] *= att_gate(a, t, h, 64 * half + i);
      }
#pragma unroll
      for (int i = 0; i < 64; i += 4) {
        const float4 v = make_float4(o[i] * inv, o[i + 1] * inv, o[i + 2] * inv, o[i + 3] * inv);
        odd |= as_no_number(v);
        *(float4*)(out + i) = v;
      }
    }
    if (__any_sync(0xffffffffu, odd) && lane == 0) atomicOr(bad, 1);
  } else if (warp < 12) {
    const int w = warp & 3, row = 32 * w + lane, pos = p0 + row;
    const uint32_t lanes = (uint32_t)(32 * w) << 16;
    const uint32_t tS = tmem + AS_TS + lanes;
    const float slope = a.slopes ? a.slopes[h] : 0.f;
    float m = a.sink ? a.sink[h] : -INFINITY, l = a.sink ? 1.f : 0.f;
    for (int j = 0; j < pages; ++j) {
      const int k0 = page_of(j) * MB_PAGE;
      mbar_wait(s_done, j & 1, error, 53);
      tc_fence_after_sync();
      float s[64];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        float x[16];
        tmem_ld16(tS + 16 * i, s + 16 * i);
        tmem_ld16(tS + 64 + 16 * i, x);
#pragma unroll
        for (int e = 0; e < 16; ++e) s[16 * i + e] += x[e];
        tmem_ld16(tS + 128 + 16 * i, x);
#pragma unroll
        for (int e = 0; e < 16; ++e) s[16 * i + e] += x[e];
      }
      // Each option in a loop of its own, so that the common way through is short: all in one loop, the
      // unrolled code was more than the instruction caches hold and a page took three times as long.
#pragma unroll
      for (int e = 0; e < 64; ++e) s[e] *= a.scale;
      if (a.softcap > 0.f) {
#pragma unroll
        for (int e = 0; e < 64; ++e) s[e] = a.softcap * tanhf(s[e] / a.softcap);
      }
      if (a.slopes) {
#pragma unroll
        for (int e = 0; e < 64; ++e) s[e] -= slope * (float)(pos - k0 - e);
      }
      // a page that every row of the warp sees whole needs no mask
      if (k0 + 63 > pos - lane || (a.window > 0 && k0 <= pos - lane + 31 - a.window)) {
#pragma unroll
        for (int e = 0; e < 64; ++e) {
          const int key = k0 + e;
          if (!(key <= pos && (a.window <= 0 || key > pos - a.window || key < a.keep_first))) s[e] = -INFINITY;
        }
      }
      float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
      for (int e = 0; e < 64; ++e) mx4[e & 3] = fmaxf(mx4[e & 3], s[e]);
      const float m_new = fmaxf(m, fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])));
      // a row that has seen no key yet keeps its zeros
      const float c = m_new == -INFINITY ? 1.f : expf(m - m_new), ref = m_new == -INFINITY ? 0.f : m_new;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int e = 0; e < 64; ++e) {
        s[e] = expf(s[e] - ref);
        sum[e & 3] += s[e];
      }
      l = l * c + ((sum[0] + sum[1]) + (sum[2] + sum[3]));
      m = m_new;
      corr[(j & 1) * AS_ROWS + row] = c;
#pragma unroll
      for (int i = 0; i < 2; ++i) {      // 32 keys' parts: 16 columns each
        uint32_t hi[16], mid[16], lo[16];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          const Cut2 x = cut(s[32 * i + 2 * e], s[32 * i + 2 * e + 1]);
          hi[e] = x.hi; mid[e] = x.mid; lo[e] = x.lo;
        }
        tmem_st16_u32(tS + 16 * i, hi);
        tmem_st16_u32(tS + 32 + 16 * i, mid);
        tmem_st16_u32(tS + 64 + 16 * i, lo);
      }
      tmem_wait_st();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full0 + 8 * (j & 1));
    }
    sums[row] = l;
    asm volatile("bar.sync 1, 384;" ::: "memory");
  } else if (elect_one()) {
    constexpr uint32_t idesc_s = umma_idesc_bf16(AS_ROWS, MB_PAGE);              // K-major both
    constexpr uint32_t idesc_o = umma_idesc_bf16(AS_ROWS, 64) | (1u << 16);      // B MN-major
    const uint32_t tQ = tmem + AS_TQ, tS = tmem + AS_TS, tO = tmem + AS_TO;
    // the six products of parts, the smallest first: part of the first operand, of the second
    constexpr uint32_t PA = 0x001102, PB = 0x010120;      // a hexadecimal digit each, the first lowest
    mbar_wait(q_full, 0, error, 54);
    for (int j = 0; j < pages; ++j) {
      mbar_wait(k_full0 + 8 * (j & 1), (j >> 1) & 1, error, 55);
      if (j > 0) mbar_wait(o_done, (j - 1) & 1, error, 56);      // the probabilities there have been read
      tc_fence_after_sync();
      const uint64_t dk = umma_desc_k128(sK + (j & 1) * AS_TILE);
      // the leading products go to two accumulators of four steps, the others to one
#pragma unroll
      for (int k = 0; k < 8; ++k)
        umma_bf16_ts(tS + 64 * (k / 4), tQ + 8 * k, dk + (k / 4) * (AS_HALF >> 4) + (k % 4) * 2, idesc_s, k % 4 > 0);
#pragma unroll 1
      for (int x = 0; x < 5; ++x) {
        const uint32_t tA = tQ + 64 * ((PA >> (4 * x)) & 3);
        const uint64_t db = dk + ((PB >> (4 * x)) & 3) * (AS_PART >> 4);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          umma_bf16_ts(tS + 128, tA + 8 * k, db + (k / 4) * (AS_HALF >> 4) + (k % 4) * 2, idesc_s, x > 0 || k > 0);
      }
      umma_commit(s_done);
      mbar_wait(v_full, j & 1, error, 57);
      mbar_wait(p_full0 + 8 * (j & 1), (j >> 1) & 1, error, 58);
      if (j > 0) mbar_wait(o_read, (j - 1) & 1, error, 59);
      tc_fence_after_sync();
      const uint64_t dv = umma_desc_mn128(sV, AS_HALF);
#pragma unroll 1
      for (int x = 0; x < 6; ++x) {
        const uint32_t tA = tS + 32 * ((PA >> (4 * x)) & 3);
        const uint64_t db = dv + ((PB >> (4 * x)) & 3) * (AS_PART >> 4);
#pragma unroll
        for (int half = 0; half < 2; ++half)
#pragma unroll
          for (int k = 0; k < 4; ++k)
            umma_bf16_ts(tO + 64 * half, tA + 8 * k, db + half * (AS_HALF >> 4) + k * (2048 >> 4), idesc_o, x > 0 || k > 0);
      }
      umma_commit(o_done);
    }
  }
  __syncthreads();
  if (warp == 12) tmem_dealloc(tmem, 512);
  if (threadIdx.x == 0) redo[((size_t)b * gridDim.y + tile) * a.nh + h] = *bad;
}

// (the dispatch is compiled for both types)
static int launch_split(const AttArgs<__nv_bfloat16>&, int, int, int, int*, int*, cudaStream_t) { return 0; }
static int launch_split(const AttArgs<float>& a, int B, int max_new, int fewest, int* redo, int* error,
                        cudaStream_t s) {
  static unsigned long long allowed = 0;
  const cudaError_t e = mb_allow_smem((const void*)attention_split_kernel, AS_SMEM, &allowed);
  if (e != cudaSuccess) MB_FAIL("mb_attention_simt: %s", cudaGetErrorString(e));
  mb_launch(attention_split_kernel, dim3(a.nh, (max_new + AS_ROWS - 1) / AS_ROWS, B), dim3(AS_THREADS), AS_SMEM, s,
            a, fewest, redo, error);
  return 0;
}
