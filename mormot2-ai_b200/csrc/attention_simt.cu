// Causal grouped-query attention over the paged cache for any head size up to 1024 (value rows up
// to 256) and any number of heads and groups, in float32 arithmetic on the CUDA cores, for float32
// or bfloat16 storage. It serves prefill and decode of the true 32-bit path and is the fallback
// of the bfloat16 path. Sizes that are multiples of four (heads of up to 256) with rows on the
// boundaries of four values go through two kernels: `attention_few_kernel` for a step that brings
// few tokens a sequence and `attention_many_kernel` for tiles of 64 new tokens (float32 heads of 128
// values that see many keys: attention_split.cuh, on the tensor cores). For all else one
// warp per (token, query head) walks the keys of the token's own sequence in tiles of 32 with an
// online softmax (a lane has one key of the tile for q·k and four neighbouring values of every
// key's row for p·v).
//
// The formula is the reference's (paths within the reference project):
// src/infer/mormot.ai.infer.backend.cpu.pas:1296-1353 — head h reads KV head
// h div (heads div kv_heads); keys max(0, pos+1-window)..pos; s = q·k·scale; p = exp(s - max);
// y = (sum p v) / (sum p) — and the tiled form of tools/cuda/ops.cu:352-540.
#include <cooperative_groups.h>

#include "attention_split.cuh"

namespace cg = cooperative_groups;

MB_DEFINE_LAST_ERROR

#define ATT_WARPS 4
#define ATT_MAX_D 8  // head sizes up to 32 * 8

template <typename T, bool VEC>
__global__ void __launch_bounds__(ATT_WARPS * 32)
attention_simt_kernel(const T* __restrict__ q, int q_stride, T* __restrict__ out, int out_stride,
                      const T* __restrict__ kpool, const T* __restrict__ vpool,
                      const int* __restrict__ page_table, int max_pages, int ring_pages,
                      const int* __restrict__ tok_seq, const int* __restrict__ tok_pos,
                      const int* __restrict__ seq_slot, int nh, int nkv, int hd, int window,
                      float scale, int vd, const float* __restrict__ sink, float softcap,
                      const T* __restrict__ gate, int gate_stride, int gate_dim,
                      const float* __restrict__ slopes, int keep_first) {
  extern __shared__ __align__(16) float qs[];  // ATT_WARPS x hd
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int t = blockIdx.x;
  const int h = blockIdx.y * ATT_WARPS + warp;
  if (h >= nh) return;
  const int g = h / (nh / nkv);
  const int pos = tok_pos[t];
  const int slot = seq_slot[tok_seq[t]];
  float* qv = qs + warp * hd;
  const T* qp = q + (size_t)t * q_stride + (size_t)h * hd;
  for (int i = lane; i < hd; i += 32) qv[i] = to_f32<T>(qp[i]);
  __syncwarp();

  int lo = 0;
  if (window > 0 && pos + 1 > window) lo = pos + 1 - window;
  // the first keep_first positions stay visible when the window has moved past them: the
  // keys are walked in two runs, [0, kept) and [lo, pos]
  const int kept = min(keep_first, lo);
  const float slope = slopes ? slopes[h] : 0.f;
  // a sink: one more term exp(sink[h]) in the denominator, as a key of that score (not
  // scaled) whose value is zero
  float m = sink ? sink[h] : -INFINITY, l = sink ? 1.f : 0.f;
  // VEC: values 4 * lane .. + 3 of every 128; else values lane, lane + 32, ...
  float acc[ATT_MAX_D];
#pragma unroll
  for (int d = 0; d < ATT_MAX_D; ++d) acc[d] = 0.f;

  for (int run = 0; run < 2; ++run) {
  const int first = run ? lo : 0, last = run ? pos : kept - 1;
  for (int k0 = first; k0 <= last; k0 += 32) {
    const int kp = k0 + lane;
    const bool valid = kp <= last;
    size_t row = 0;
    float s = -INFINITY;
    if (valid) {
      row = kv_row(page_table, max_pages, ring_pages, slot, kp, nkv, g);
      const T* kr = kpool + row * hd;
      float dot = 0.f;
      if (VEC) {
        for (int i = 0; i < hd; i += 4) {
          const float4 kk = load4<T>(kr + i), qq = *(const float4*)(qv + i);
          dot = fmaf(qq.x, kk.x, fmaf(qq.y, kk.y, fmaf(qq.z, kk.z, fmaf(qq.w, kk.w, dot))));
        }
      } else {
        for (int i = 0; i < hd; ++i) dot = fmaf(qv[i], to_f32<T>(kr[i]), dot);
      }
      s = dot * scale;
      if (softcap > 0.f) s = softcap * tanhf(s / softcap);
      s -= slope * (float)(pos - kp);      // a bias that grows with the distance
    }
    const float m_new = fmaxf(m, warp_max(s));
    const float corr = expf(m - m_new);  // 0 on the first tile (m = -inf)
    const float p = valid ? expf(s - m_new) : 0.f;
    l = l * corr + warp_sum(p);
#pragma unroll
    for (int d = 0; d < ATT_MAX_D; ++d) acc[d] *= corr;
    m = m_new;
    const int n = min(32, last - k0 + 1);
    for (int j = 0; j < n; ++j) {
      const float pj = __shfl_sync(0xffffffffu, p, j);
      const unsigned lo32 = __shfl_sync(0xffffffffu, (unsigned)(row & 0xffffffffu), j);
      const unsigned hi32 = __shfl_sync(0xffffffffu, (unsigned)(row >> 32), j);
      const T* vr = vpool + (((size_t)hi32 << 32) | lo32) * vd;
      if (VEC) {
#pragma unroll
        for (int d = 0; d < ATT_MAX_D / 4; ++d) {
          const int i = 4 * lane + 128 * d;
          if (i < vd) {
            const float4 vv = load4<T>(vr + i);
            acc[4 * d] = fmaf(pj, vv.x, acc[4 * d]);
            acc[4 * d + 1] = fmaf(pj, vv.y, acc[4 * d + 1]);
            acc[4 * d + 2] = fmaf(pj, vv.z, acc[4 * d + 2]);
            acc[4 * d + 3] = fmaf(pj, vv.w, acc[4 * d + 3]);
          }
        }
      } else {
#pragma unroll
        for (int d = 0; d < ATT_MAX_D; ++d) {
          const int i = lane + 32 * d;
          if (i < vd) acc[d] = fmaf(pj, to_f32<T>(vr[i]), acc[d]);
        }
      }
    }
  }
  }
  // a gate per head: the head's output times the sigmoid of the token's logit for this head;
  // or one per value
  const float inv = (gate && gate_dim == 0
                         ? sigmoid_f32(to_f32<T>(gate[(size_t)t * gate_stride + h])) : 1.0f) / l;
  if (gate && gate_dim > 0) {
    const T* gp = gate + (size_t)t * gate_stride + (size_t)h * gate_dim;
#pragma unroll
    for (int d = 0; d < ATT_MAX_D; ++d) {
      const int i = VEC ? 4 * lane + 128 * (d / 4) + d % 4 : lane + 32 * d;
      if (i < vd) acc[d] *= sigmoid_f32(to_f32<T>(gp[i]));
    }
  }
  T* op = out + (size_t)t * out_stride + (size_t)h * vd;
  if (VEC) {
#pragma unroll
    for (int d = 0; d < ATT_MAX_D / 4; ++d) {
      const int i = 4 * lane + 128 * d;
      if (i < vd)
        store4<T>(op + i, make_float4(acc[4 * d] * inv, acc[4 * d + 1] * inv, acc[4 * d + 2] * inv,
                                      acc[4 * d + 3] * inv));
    }
  } else {
#pragma unroll
    for (int d = 0; d < ATT_MAX_D; ++d) {
      const int i = lane + 32 * d;
      if (i < vd) op[i] = from_f32<T>(acc[d] * inv);
    }
  }
}

// ---------------------------------------------------------------------------- few new tokens
// One token and up to RT query heads of one KV head per cluster of S CTAs; the tiles of 16 visible
// keys are dealt out over the cluster's 4 S warps in turn, each with a softmax of its own, and the
// partial results meet in shared memory, the CTAs' through the cluster's. It is the reading of the
// cache that bounds it, so every warp asks for whole rows with 16-byte loads, 16 keys at a time:
// eight lanes share a key for q.k (three shuffles a score), a lane has four values of a row for
// p.v, and a key's row serves all heads of its group. Before, a warp walked a (token, head) alone,
// with 32 lanes in 32 different rows: a decode step of 8 sequences of 200 to 1,500 positions (16
// heads on 8 of 128 values, float32, 55 MB) took 744 us; now 25 (2.2 TB/s).
// `per_seq` > 0: a step in which other sequences bring many tokens (for the kernel below); the
// clusters then stand for the first per_seq tokens of every sequence and leave those alone.
#define ATF_WARPS 4
#define ATF_KEYS 16

template <typename T, int RT, bool WHOLE>   // WHOLE: hd = vd = 128
__global__ void __launch_bounds__(ATF_WARPS * 32)
attention_few_kernel(const AttArgs<T> a, int splits, int chunks, int per_seq) {
  mb_grid_wait();
  mb_grid_launch_next();
  int t = blockIdx.x / splits;
  const int split = blockIdx.x - t * splits;
  if (per_seq > 0) {
    const int b = t / per_seq, n_new = a.seq_start[b + 1] - a.seq_start[b];
    if (n_new >= ATT_MANY || t - b * per_seq >= n_new) return;      // the whole cluster
    t = a.seq_start[b] + t - b * per_seq;
  }
  extern __shared__ __align__(16) float sm[];
  const int hd = WHOLE ? 128 : a.hd, vd = WHOLE ? 128 : a.vd;
  constexpr int ND = WHOLE ? 1 : 2;
  float* qs = sm;                                    // [RT][hd]
  float* ps = qs + RT * hd;                          // [warps][RT][16] scores, then probabilities
  float* po = ps + ATF_WARPS * RT * ATF_KEYS;        // [warps][RT][vd] partial sums of values
  float* pml = po + ATF_WARPS * RT * vd;             // [warps][RT][2] maximum and sum
  float* bo = pml + ATF_WARPS * RT * 2;              // [RT][vd] the block's, and [RT][2]
  float* bml = bo + RT * vd;
  size_t* rows = (size_t*)(bml + RT * 2);            // [warps][16]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = blockIdx.y / chunks, R = a.nh / a.nkv;
  const int h0 = g * R + (blockIdx.y - g * chunks) * RT, heads = min(RT, (g + 1) * R - h0);
  const int pos = a.tok_pos[t], slot = a.seq_slot[a.tok_seq[t]];
  for (int e = threadIdx.x; e < RT * hd; e += ATF_WARPS * 32) {
    const int r = e / hd;
    qs[e] = r < heads ? to_f32<T>(a.q[(size_t)t * a.q_stride + (size_t)(h0 + r) * hd + e - r * hd]) : 0.f;
  }
  __syncthreads();
  int lo = 0;
  if (a.window > 0 && pos + 1 > a.window) lo = pos + 1 - a.window;
  // visible keys 0 .. n - 1: first the positions that the window never loses, then lo .. pos
  const int kept = min(a.keep_first, lo), n = kept + pos + 1 - lo;
  float slope[RT], m[RT], l[RT], acc[RT][4 * ND];
#pragma unroll
  for (int r = 0; r < RT; ++r) {
    slope[r] = a.slopes && r < heads ? a.slopes[h0 + r] : 0.f;
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int d = 0; d < 4 * ND; ++d) acc[r][d] = 0.f;
  }
  float* pw = ps + warp * RT * ATF_KEYS;
  size_t* rw = rows + warp * ATF_KEYS;
  const int sub = lane >> 3, l8 = lane & 7;
  for (int k0 = (split * ATF_WARPS + warp) * ATF_KEYS; k0 < n; k0 += splits * ATF_WARPS * ATF_KEYS) {
    const int cnt = min(ATF_KEYS, n - k0);
    __syncwarp();
    if (lane < ATF_KEYS) {      // places behind the last key repeat it: its row exists
      const int kk = k0 + min(lane, cnt - 1);
      rw[lane] = kv_row(a.page_table, a.max_pages, a.ring_pages, slot,
                        kk < kept ? kk : lo + kk - kept, a.nkv, g);
    }
    __syncwarp();
    float dot[4][RT];
    const T* kr[4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      kr[p] = a.kpool + rw[4 * p + sub] * hd;
#pragma unroll
      for (int r = 0; r < RT; ++r) dot[p][r] = 0.f;
    }
#pragma unroll 4
    for (int i = 4 * l8; i < hd; i += 32) {
      float4 kk[4];
#pragma unroll
      for (int p = 0; p < 4; ++p) kk[p] = load4<T>(kr[p] + i);
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        const float4 qq = *(const float4*)(qs + r * hd + i);
#pragma unroll
        for (int p = 0; p < 4; ++p)
          dot[p][r] = fmaf(qq.x, kk[p].x, fmaf(qq.y, kk[p].y, fmaf(qq.z, kk[p].z,
                                                                  fmaf(qq.w, kk[p].w, dot[p][r]))));
      }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int r = 0; r < RT; ++r) {
        float d = dot[p][r];
        d += __shfl_xor_sync(0xffffffffu, d, 1);
        d += __shfl_xor_sync(0xffffffffu, d, 2);
        d += __shfl_xor_sync(0xffffffffu, d, 4);
        if (l8 == r) pw[r * ATF_KEYS + 4 * p + sub] = d;
      }
    __syncwarp();
    const int key = lane & 15, kk = k0 + key;
    const int dist = pos - (kk < kept ? kk : lo + kk - kept);
#pragma unroll
    for (int r0 = 0; r0 < RT; r0 += 2) {      // two heads at a time, a half warp each
      const int r = r0 + (RT > 1 ? lane >> 4 : 0);
      const float sl = RT > 1 && lane >= 16 ? slope[r0 + (RT > 1 ? 1 : 0)] : slope[r0];
      float mine = RT > 1 && lane >= 16 ? m[r0 + (RT > 1 ? 1 : 0)] : m[r0];
      const float s = key < cnt ? att_score(a, pw[r * ATF_KEYS + key], sl, dist) : -INFINITY;
      float mx = s;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
      // a warp's keys so far may all have the score -infinity: they weigh nothing (not 0 / 0)
      const float m_new = fmaxf(mine, mx), corr = m_new == -INFINITY ? 1.f : expf(mine - m_new);
      const float p = s == -INFINITY ? 0.f : expf(s - m_new);
      float sum = p;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (RT > 1 || lane < 16) pw[r * ATF_KEYS + key] = p;
#pragma unroll
      for (int q = 0; q < (RT > 1 ? 2 : 1); ++q) {
        const float c = __shfl_sync(0xffffffffu, corr, 16 * q);
        m[r0 + q] = __shfl_sync(0xffffffffu, m_new, 16 * q);
        l[r0 + q] = l[r0 + q] * c + __shfl_sync(0xffffffffu, sum, 16 * q);
#pragma unroll
        for (int d = 0; d < 4 * ND; ++d) acc[r0 + q][d] *= c;
      }
    }
    __syncwarp();
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      const int i = 4 * lane + 128 * d;
      if (i >= vd) break;
      auto add = [&](int j, float4 vv) {
#pragma unroll
        for (int r = 0; r < RT; ++r) {
          const float p = pw[r * ATF_KEYS + j];
          acc[r][4 * d] = fmaf(p, vv.x, acc[r][4 * d]);
          acc[r][4 * d + 1] = fmaf(p, vv.y, acc[r][4 * d + 1]);
          acc[r][4 * d + 2] = fmaf(p, vv.z, acc[r][4 * d + 2]);
          acc[r][4 * d + 3] = fmaf(p, vv.w, acc[r][4 * d + 3]);
        }
      };
      if (cnt == ATF_KEYS) {
#pragma unroll
        for (int j = 0; j < ATF_KEYS; j += 8) {
          float4 vv[8];
#pragma unroll
          for (int u = 0; u < 8; ++u) vv[u] = load4<T>(a.vpool + rw[j + u] * vd + i);
#pragma unroll
          for (int u = 0; u < 8; ++u) add(j + u, vv[u]);
        }
      } else {
        for (int j = 0; j < cnt; ++j) add(j, load4<T>(a.vpool + rw[j] * vd + i));
      }
    }
  }
#pragma unroll
  for (int r = 0; r < RT; ++r) {
#pragma unroll
    for (int d = 0; d < ND; ++d) {
      const int i = 4 * lane + 128 * d;
      if (i < vd)
        *(float4*)(po + (warp * RT + r) * vd + i) =
            make_float4(acc[r][4 * d], acc[r][4 * d + 1], acc[r][4 * d + 2], acc[r][4 * d + 3]);
    }
    if (lane == 0) {
      pml[(warp * RT + r) * 2] = m[r];
      pml[(warp * RT + r) * 2 + 1] = l[r];
    }
  }
  __syncthreads();
  // the four warps' results, in their order; a part without keys has the maximum -inf
  for (int e = threadIdx.x; e < RT * vd; e += ATF_WARPS * 32) {
    const int r = e / vd;
    float M = -INFINITY, L = 0.f, o = 0.f;
#pragma unroll
    for (int w = 0; w < ATF_WARPS; ++w) M = fmaxf(M, pml[(w * RT + r) * 2]);
#pragma unroll
    for (int w = 0; w < ATF_WARPS; ++w) {
      const float mw = pml[(w * RT + r) * 2], f = mw == -INFINITY ? 0.f : expf(mw - M);
      L = fmaf(f, pml[(w * RT + r) * 2 + 1], L);
      if (f != 0.f) o = fmaf(f, po[(w * RT + r) * vd + e - r * vd], o);
    }
    bo[e] = o;
    if (e == r * vd) {
      bml[2 * r] = M;
      bml[2 * r + 1] = L;
    }
  }
  cg::cluster_group cluster = cg::this_cluster();
  if (splits > 1) cluster.sync();
  else __syncthreads();
  // the cluster's CTAs each finish a share of the outputs, the splits in their order
  for (int e = split * ATF_WARPS * 32 + threadIdx.x; e < heads * vd; e += splits * ATF_WARPS * 32) {
    const int r = e / vd, i = e - r * vd, h = h0 + r;
    float M = a.sink ? a.sink[h] : -INFINITY, L = 0.f, o = 0.f;
    for (int k = 0; k < splits; ++k)
      M = fmaxf(M, splits > 1 ? cluster.map_shared_rank(bml, k)[2 * r] : bml[2 * r]);
    if (a.sink) L = expf(a.sink[h] - M);
    for (int k = 0; k < splits; ++k) {
      const float* kml = splits > 1 ? cluster.map_shared_rank(bml, k) : bml;
      const float* ko = splits > 1 ? cluster.map_shared_rank(bo, k) : bo;
      const float mk = kml[2 * r], f = mk == -INFINITY ? 0.f : expf(mk - M);
      L = fmaf(f, kml[2 * r + 1], L);
      if (f != 0.f) o = fmaf(f, ko[e], o);
    }
    a.out[(size_t)t * a.out_stride + (size_t)h * vd + i] = from_f32<T>(o * att_gate(a, t, h, i) / L);
  }
  if (splits > 1) cluster.sync();      // nobody leaves while its results are still read
}

template <typename T>
static int launch_few(const AttArgs<T>& a, int tokens, int per_seq, int sms, cudaStream_t s) {
  const int R = a.nh / a.nkv, RT = R > 4 ? 8 : (R > 2 ? 4 : R), chunks = (R + RT - 1) / RT;
  const bool whole = a.hd == 128 && a.vd == 128;
  // about four CTAs an SM, at most the eight of a portable cluster; it depends on nothing that
  // changes between the steps that a captured launch is replayed for
  int splits = 4 * sms / (tokens * a.nkv * chunks);
  splits = splits > 8 ? 8 : (splits < 1 ? 1 : splits);
  if (splits > a.max_pages) splits = a.max_pages;
  const size_t smem = (size_t)(RT * a.hd + ATF_WARPS * RT * (ATF_KEYS + a.vd + 2) + RT * (a.vd + 2)) *
                          sizeof(float) + ATF_WARPS * ATF_KEYS * sizeof(size_t);
  const dim3 grid(tokens * splits, a.nkv * chunks);
#define GO(R_, W_)                                                                             \
  {                                                                                            \
    if (smem > 48 * 1024) { /* heads of 256 and eight to a KV head: 53 KB */                   \
      static unsigned long long allowed = 0;                                                   \
      const cudaError_t e =                                                                    \
          mb_allow_smem((const void*)attention_few_kernel<T, R_, W_>, 56 * 1024, &allowed);    \
      if (e != cudaSuccess) MB_FAIL("mb_attention_simt: %s", cudaGetErrorString(e));           \
    }                                                                                          \
    mb_launch_clusters(attention_few_kernel<T, R_, W_>, grid, dim3(ATF_WARPS * 32), smem, s,   \
                       splits, a, splits, chunks, per_seq);                                             \
  }
#define GOW(R_) if (whole) GO(R_, true) else GO(R_, false)
  if (RT == 1) GOW(1) else if (RT == 2) GOW(2) else if (RT == 4) GOW(4) else GOW(8)
#undef GOW
#undef GO
  MB_CHECK_LAUNCH("mb_attention_simt");
}

// ---------------------------------------------------------------------------- many new tokens
// 64 new tokens of one sequence and one head per CTA, a page of 64 keys at a time through shared
// memory: a tile of 64 x 64 scores gives each of 256 threads 4 x 4 of them (every value read from
// shared memory serves four multiply-adds) and 4 x 8 values of the output (128 threads with twice
// the rows take 385 us where these take 335: too few warps). Rows of q and k keep their order in
// shared memory (pitch hd + 4: a warp's 16 keys lie on different banks) and are read four values
// along the head at a time. K and V take turns in one tile, so that two CTAs fit an SM and one
// computes while the other loads. The reads of shared memory bound it (issue slots 0.51 busy, the
// pipe of the multiply-adds 0.24; warps wait for operands first of all).
// Before, a warp walked a (token, head) alone: 1,728 tokens of three prompts (16 heads on 8 of
// 128 values, float32) took 1,907 us; now 335 (17 TFLOP/s).
#define ATM_ROWS 64
#define ATM_THREADS 256
#define ATM_R 4           // rows of a thread
#define ATM_PITCH 68      // of a row of probabilities

template <typename T>
__global__ void __launch_bounds__(ATM_THREADS, 2)
attention_many_kernel(const AttArgs<T> a, int fewest, const int* __restrict__ redo) {
  // fewest: new tokens of a sequence; redo: [B][tiles of 128][heads], the tiles to do (null: all)
  mb_grid_wait();
  mb_grid_launch_next();
  extern __shared__ __align__(16) float sm[];
  const int hd = a.hd, vd = a.vd, pitch = hd + 4, kv_pitch = max(pitch, vd);
  float* qs = sm;                             // [64][pitch]
  float* kv = qs + ATM_ROWS * pitch;          // [64][pitch] keys, then [64][vd] values
  float* ps = kv + ATM_ROWS * kv_pitch;       // [64][ATM_PITCH]
  const int h = blockIdx.x, g = h / (a.nh / a.nkv), b = blockIdx.z;
  const int t0 = a.seq_start[b], n_new = a.seq_start[b + 1] - t0;
  const int tiles = (n_new + ATM_ROWS - 1) / ATM_ROWS;
  if ((int)blockIdx.y >= tiles || n_new < fewest) return;
  const int r0 = (tiles - 1 - blockIdx.y) * ATM_ROWS;   // the tiles that see the most keys first
  if (redo && !redo[((size_t)b * ((gridDim.y * ATM_ROWS + 127) / 128) + r0 / 128) * a.nh + h]) return;
  const int cnt = min(ATM_ROWS, n_new - r0);
  const int slot = a.seq_slot[b], p0 = a.tok_pos[t0 + r0];   // row r stands at position p0 + r
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int hp = hd >> 2, vp = vd >> 2;
  for (int e = threadIdx.x; e < ATM_ROWS * hp; e += ATM_THREADS) {
    const int r = e / hp, c = 4 * (e - r * hp);
    *(float4*)(qs + r * pitch + c) =
        r < cnt ? load4<T>(a.q + (size_t)(t0 + r0 + r) * a.q_stride + (size_t)h * hd + c)
                : make_float4(0.f, 0.f, 0.f, 0.f);
  }
  const float slope = a.slopes ? a.slopes[h] : 0.f;
  const float sink = a.sink ? a.sink[h] : -INFINITY;
  float m[ATM_R], l[ATM_R], o[ATM_R][8];
#pragma unroll
  for (int i = 0; i < ATM_R; ++i) {
    m[i] = sink;
    l[i] = a.sink ? 1.f : 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) o[i][j] = 0.f;
  }
  auto sees = [&](int pos, int key) {
    return key <= pos && (a.window <= 0 || key > pos - a.window || key < a.keep_first);
  };
  const int last = p0 + cnt - 1;
  // pages that some row sees: those of the kept first positions, then from the first row's window
  const int lo0 = a.window > 0 ? max(0, p0 + 1 - a.window) : 0;
  const int first_page = lo0 / MB_PAGE, kept_pages = min((a.keep_first + MB_PAGE - 1) / MB_PAGE, first_page);
  for (int it = 0; it < kept_pages + last / MB_PAGE - first_page + 1; ++it) {
    const int page = it < kept_pages ? it : first_page + it - kept_pages, k0 = page * MB_PAGE;
    const int keys = min(MB_PAGE, last + 1 - k0);
    const size_t row = kv_row(a.page_table, a.max_pages, a.ring_pages, slot, k0, a.nkv, g);
    __syncthreads();      // the values (and probabilities) of the page before have been read
    for (int e = threadIdx.x; e < MB_PAGE * hp; e += ATM_THREADS) {
      const int r = e / hp, c = 4 * (e - r * hp);
      *(float4*)(kv + r * pitch + c) = r < keys ? load4<T>(a.kpool + (row + r) * hd + c)
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    __syncthreads();
    float s[ATM_R][4];
#pragma unroll
    for (int i = 0; i < ATM_R; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) s[i][j] = 0.f;
#pragma unroll 2
    for (int c = 0; c < hd; c += 4) {
      float4 kk[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) kk[j] = *(const float4*)(kv + (tx + 16 * j) * pitch + c);
#pragma unroll
      for (int i = 0; i < ATM_R; ++i) {
        const float4 qq = *(const float4*)(qs + (ATM_R * ty + i) * pitch + c);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          s[i][j] = fmaf(qq.x, kk[j].x, fmaf(qq.y, kk[j].y, fmaf(qq.z, kk[j].z,
                                                                fmaf(qq.w, kk[j].w, s[i][j]))));
      }
    }
    __syncthreads();      // the keys have been read: the values may come
    bool odd = false;     // an infinity or NaN among the values
    for (int e = threadIdx.x; e < MB_PAGE * vp; e += ATM_THREADS) {
      const int r = e / vp, c = 4 * (e - r * vp);
      const float4 v = r < keys ? load4<T>(a.vpool + (row + r) * vd + c)
                                : make_float4(0.f, 0.f, 0.f, 0.f);
      odd |= !(0.f * v.x + 0.f * v.y + 0.f * v.z + 0.f * v.w == 0.f);
      *(float4*)(kv + r * vd + c) = v;
    }
#pragma unroll
    for (int i = 0; i < ATM_R; ++i) {
      const int pos = p0 + ATM_R * ty + i;
      float mx = -INFINITY;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kp = k0 + tx + 16 * j;
        s[i][j] = sees(pos, kp) ? att_score(a, s[i][j], slope, pos - kp) : -INFINITY;
        mx = fmaxf(mx, s[i][j]);
      }
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
      const float m_new = fmaxf(m[i], mx);
      // a row that has seen no key yet keeps its zeros
      const float corr = m_new == -INFINITY ? 1.f : expf(m[i] - m_new);
      float sum = 0.f;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float p = s[i][j] == -INFINITY ? 0.f : expf(s[i][j] - m_new);
        ps[(ATM_R * ty + i) * ATM_PITCH + tx + 16 * j] = p;
        sum += p;
      }
#pragma unroll
      for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
      m[i] = m_new;
      l[i] = l[i] * corr + sum;
#pragma unroll
      for (int j = 0; j < 8; ++j) o[i][j] *= corr;
    }
    if (__syncthreads_or(odd)) {
      // a value that no number is reaches only the rows that see its key: 0 times it is NaN
      for (int k = 0; k < keys; ++k)
#pragma unroll
        for (int i = 0; i < ATM_R; ++i) {
          if (!sees(p0 + ATM_R * ty + i, k0 + k)) continue;
          const float p = ps[(ATM_R * ty + i) * ATM_PITCH + k];
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const int c = 4 * tx + 64 * (j >> 2) + (j & 3);
            if (c < vd) o[i][j] = fmaf(p, kv[k * vd + c], o[i][j]);
          }
        }
      continue;
    }
    for (int k = 0; k < keys; k += 4) {
      float4 pp[ATM_R];
#pragma unroll
      for (int i = 0; i < ATM_R; ++i) pp[i] = *(const float4*)(ps + (ATM_R * ty + i) * ATM_PITCH + k);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const int c = 4 * tx + 64 * half;
          if (c >= vd) continue;
          const float4 vv = *(const float4*)(kv + (k + u) * vd + c);
#pragma unroll
          for (int i = 0; i < ATM_R; ++i) {
            const float p = u == 0 ? pp[i].x : (u == 1 ? pp[i].y : (u == 2 ? pp[i].z : pp[i].w));
            o[i][4 * half] = fmaf(p, vv.x, o[i][4 * half]);
            o[i][4 * half + 1] = fmaf(p, vv.y, o[i][4 * half + 1]);
            o[i][4 * half + 2] = fmaf(p, vv.z, o[i][4 * half + 2]);
            o[i][4 * half + 3] = fmaf(p, vv.w, o[i][4 * half + 3]);
          }
        }
    }
  }
#pragma unroll
  for (int i = 0; i < ATM_R; ++i) {
    const int r = ATM_R * ty + i;
    if (r >= cnt) continue;
    const int t = t0 + r0 + r;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      const int c = 4 * tx + 64 * half;
      if (c >= vd) continue;
      const float inv = 1.f / l[i];
      store4<T>(a.out + (size_t)t * a.out_stride + (size_t)h * vd + c,
                make_float4(o[i][4 * half] * inv * att_gate(a, t, h, c),
                            o[i][4 * half + 1] * inv * att_gate(a, t, h, c + 1),
                            o[i][4 * half + 2] * inv * att_gate(a, t, h, c + 2),
                            o[i][4 * half + 3] * inv * att_gate(a, t, h, c + 3)));
    }
  }
}

template <typename T>
static int launch_many(const AttArgs<T>& a, int B, int max_new, int fewest, const int* redo, cudaStream_t s) {
  const int pitch = a.hd + 4, kv_pitch = pitch > a.vd ? pitch : a.vd;
  const size_t smem = (size_t)ATM_ROWS * (pitch + kv_pitch + ATM_PITCH) * sizeof(float);
  static unsigned long long allowed = 0;      // heads of 128: 85 KB
  const cudaError_t e = mb_allow_smem((const void*)attention_many_kernel<T>, 88 * 1024, &allowed);
  if (e != cudaSuccess) MB_FAIL("mb_attention_simt: %s", cudaGetErrorString(e));
  mb_launch(attention_many_kernel<T>, dim3(a.nh, (max_new + ATM_ROWS - 1) / ATM_ROWS, B),
            dim3(ATM_THREADS), smem, s, a, fewest, redo);
  MB_CHECK_LAUNCH("mb_attention_simt");
}

// out[t, h, :] for every token t of the step and head h. q: head h of token t at
// q + t * q_stride + h * hd (the q part of the fused qkv rows); out: head h at
// out + t * out_stride + h * vd. `vd`: the size of a value row (0: hd). `sink`: float32 [nh]
// or null, one more term exp(sink[h]) in every softmax denominator of head h. `softcap` > 0:
// every score s (after the scale) becomes softcap * tanh(s / softcap). `gate` (may be null):
// head h's output of token t is multiplied by sigmoid(gate[t * gate_stride + h]), or, with
// `gate_dim` > 0, its value d by sigmoid(gate[t * gate_stride + h * gate_dim + d]). `slopes`:
// float32 [nh] or null: slopes[h] * (query's position - key's position) is taken off every
// score of head h after the cap. `keep_first` > 0: with a window, the first keep_first
// positions of a sequence stay visible to every later one. `few_new`: the most new tokens of a
// sequence that brings fewer than ATT_MANY of them (0: there is none). `redo`: null, or room for an
// int per sequence, 128 of max_new tokens (rounded up) and head: many new tokens of float32 heads of
// 128 values then go through the tensor cores (attention_split.cuh). `error`: its waits' error word.
MB_EXPORT int mb_attention_simt(const void* q, int q_stride, void* out, int out_stride,
                                const void* kpool, const void* vpool, int dtype,
                                const int* page_table, int max_pages, int ring_pages,
                                const int* tok_seq, const int* tok_pos, const int* seq_slot,
                                const int* seq_start, int B, int max_new, int few_new,
                                int T, int nh, int nkv, int hd, int window, float scale,
                                int vd, const float* sink, float softcap, const void* gate,
                                int gate_stride, int gate_dim, const float* slopes, int keep_first,
                                int sms, int* redo, int* error, void* stream) {
  if (T <= 0) return 0;
  if (vd <= 0) vd = hd;
  if (hd <= 0 || hd > 1024 || vd > 32 * ATT_MAX_D)
    MB_FAIL("mb_attention_simt: heads of %d and %d values are not supported (at most 1024 "
            "and %d)", hd, vd, 32 * ATT_MAX_D);
  if (nkv <= 0 || nh % nkv) MB_FAIL("mb_attention_simt: %d heads on %d KV heads", nh, nkv);
  cudaStream_t s = (cudaStream_t)stream;
  dim3 grid(T, (nh + ATT_WARPS - 1) / ATT_WARPS);
  const size_t smem = (size_t)ATT_WARPS * hd * sizeof(float);
  // four values with one load: the size of four values divides every row's address
  const int four = dtype == MB_F32 ? 15 : 7;
  const bool vec = hd % 4 == 0 && vd % 4 == 0 && q_stride % 4 == 0 && out_stride % 4 == 0 &&
                   (((uintptr_t)q | (uintptr_t)out | (uintptr_t)kpool | (uintptr_t)vpool) & four) == 0;
  if (vec && hd <= 256) {
    const bool many = max_new >= ATT_MANY && hd <= 128 && vd <= 128 && B <= 65535;
    const bool mixed = many && few_new > 0;
    if (mixed && few_new >= ATT_MANY) MB_FAIL("mb_attention_simt: %d are not few new tokens", few_new);
#define GOA(T_)                                                                               \
  {                                                                                           \
    const AttArgs<T_> a = {(const T_*)q, (T_*)out, (const T_*)kpool, (const T_*)vpool,        \
                           page_table, tok_seq, tok_pos, seq_slot, seq_start, sink, slopes,   \
                           (const T_*)gate, q_stride, out_stride, max_pages, ring_pages, nh,  \
                           nkv, hd, vd, window, gate_stride, gate_dim, keep_first, scale,     \
                           softcap};                                                          \
    if (mixed && launch_few<T_>(a, B * few_new, few_new, sms, s)) return -1;                  \
    const int fewest = mixed ? ATT_MANY : 0;                                                  \
    if (!many || hd != 128 || vd != 128 || sizeof(T_) != 4) redo = nullptr;                   \
    if (redo && launch_split(a, B, max_new, fewest, redo, error, s)) return -1;               \
    return many ? launch_many<T_>(a, B, max_new, fewest, redo, s)                             \
                : launch_few<T_>(a, T, 0, sms, s);                                            \
  }
    if (dtype == MB_F32) GOA(float) else GOA(__nv_bfloat16)
#undef GOA
  }
#define GO(T_, V_)                                                                            \
  attention_simt_kernel<T_, V_><<<grid, ATT_WARPS * 32, smem, s>>>(                           \
      (const T_*)q, q_stride, (T_*)out, out_stride, (const T_*)kpool, (const T_*)vpool,       \
      page_table, max_pages, ring_pages, tok_seq, tok_pos, seq_slot, nh, nkv, hd, window, scale, \
      vd, sink, softcap, (const T_*)gate, gate_stride, gate_dim, slopes, keep_first)
  if (dtype == MB_F32) {
    if (vec) GO(float, true); else GO(float, false);
  } else {
    if (vec) GO(__nv_bfloat16, true); else GO(__nv_bfloat16, false);
  }
#undef GO
  MB_CHECK_LAUNCH("mb_attention_simt");
}
