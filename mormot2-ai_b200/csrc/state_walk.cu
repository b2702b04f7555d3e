// The matrix-state recurrences of linear_state.cu and recurrent.cu, four tokens at a time, for
// steps that bring many tokens of a sequence. With S0 the state (D x DV per head) before a group of
// four tokens, every recurrence here is
//
//   r_t = S0^T q'_t                                        (S0's part of the output)
//   o_t = og_t r_t + sum_{s <= t} N_ts x_s                 (the group's own tokens)
//   S   = A S0 + sum_s k'_s (h_s x_s)^T
//
//   delta    x_t = c_t v_t - e_t (S0^T k_t) - sum_{s < t} M_ts x_s, A a scalar
//   mlstm    x = v, A a scalar; the normalizer n is one more column whose values are one
//   gla, wkv x = v, A per key channel; q' and k' carry the decays of the group's tokens
//
// Long sequences of the first two go in chunks of 32 tokens instead (state_chunks.cuh).
//
// (definitions of the mixers in linear_state.cu and recurrent.cu; products of decays are formed as
// products, never as quotients). Walked token by token a state element costs four instructions a
// token and every token ends in a chain of shuffles that the next one waits for; by fours it is
// two and a quarter to three, and one chain for four tokens. N, M and the factors are small
// products of keys and queries alone: CT / 4 warps of the block (a group each) prepare the next
// chunk of CT tokens (32, or 16 where shared memory does not allow it) and copy in the chunk after
// it while the others walk this one. A walking thread has 8 or 16 rows of two neighbouring columns
// of the state in registers, P lanes share a pair of columns. What bounds it: the chain of a group
// in the walking warps, of which a scheduler has one (of its three warps; issue slots 0.44 busy,
// the preparing warps wait at the chunk's barrier, the walking ones for fixed latencies and shared
// memory); a block takes as few columns as leave it one walking warp a scheduler while the step
// has few (sequence, head) pairs, so that one prompt spreads over the device. All of it float32.
// One prompt of 2,048 tokens, 16 heads of 128 x 128: delta 936 -> 366 us, gated linear attention
// 960 -> 365; 8 heads of 128 x 128, mlstm: 1,660 -> 298; 32 heads of 64 x 64, wkv: 870 -> 258.
// Tried on the way: one column a thread (delta 424: reads of shared memory, 512 bytes each
// whatever lanes share, bound it).
#include "common.cuh"

MB_DEFINE_LAST_ERROR

enum { WALK_GLA = 0, WALK_DELTA = 1, WALK_MLSTM = 2, WALK_WKV = 3 };

#define SW_MOST_CT 32   // most tokens of a chunk
#define SW_COEF 56      // numbers of a group
// places of a group's numbers
#define SW_N 0          // [t][s]
#define SW_M 16         // [t][s]
#define SW_C 32
#define SW_E 36
#define SW_OG 40
#define SW_H 44
#define SW_A 48
#define SW_EM 52        // mlstm: e^-m of the four tokens

// As kernels.py lays it out: pointers to column 0 of head 0, row strides in floats.
struct WalkArgs {
  const float* q;
  const float* k;
  const float* v;
  const float* a;         // gla, wkv: the decays' logits
  const float* s0;        // delta: beta's and the decay's logits; mlstm: the gates' logits
  const float* s1;
  const float* gate;
  const float* abias;     // gla: bias [H D]; wkv: w0 [H D]
  const float* u;         // wkv: [H D]
  const float* p0;        // per head: delta a_log, mlstm the input gate's bias
  const float* p1;        // ... dt_bias, the forget gate's bias
  const float* normw;
  float* state;
  const int* seq_start;
  const int* seq_slot;
  const void* h;          // wkv: the mixer's input rows, whose last goes before the states
  void* out;              // [T, H DV] of the activation type
  float* raw;             // scratch: [T, H DV], [T, H] (mlstm), [B, H] (mlstm)
  long long state_stride, state_off, head_stride;   // of a slot, of a head's state in it
  int ldq, ldk, ldv, lda, lds, ldg, group, mode, gate_kind, norm_stride, T, B, H, D, DV, W,
      out_bf16, h_bf16, vec;
  float q_scale, inv_tau, unit_eps, cap, eps;
};

static_assert(sizeof(WalkArgs) == 264, "as kernels.py packs it");

__device__ __forceinline__ float sw_log_sigmoid(float x) {
  return fminf(x, 0.f) - log1pf(expf(-fabsf(x)));
}
__device__ __forceinline__ float sw_softplus(float x) {
  return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x)));
}
#include "state_chunks.cuh"

template <int BYTES> __device__ __forceinline__ void sw_copy(float* dst, const float* src) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (BYTES == 16)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void sw_prep_sync(int threads) {
  asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
}
__device__ __forceinline__ float sw_added(f32_pair v) { return pair_half(v, 0) + pair_half(v, 1); }

// Shared memory: three buffers [q | k | decays (gla, wkv)] of CT x DP + CT x CW of v + CT x 2
// logits; two of coefficients; two of CT x CW outputs. mlstm: the block behind the slices of the
// columns has the one column of the normalizer.
template <int MODE, int R>   // R: rows of a walking thread
__global__ void __launch_bounds__(128 + SW_MOST_CT * 8, 1)
state_walk_kernel(const WalkArgs g, int P, int CW, int CT) {
  mb_grid_wait();
  mb_grid_launch_next();
  extern __shared__ __align__(16) float sw_smem[];
  constexpr bool CHANNEL = MODE == WALK_GLA || MODE == WALK_WKV;
  constexpr int NV = CHANNEL ? 3 : 2;
  constexpr int RP = R + 4;      // pitch of R rows in shared memory: a column's lanes on different banks
  const int D = g.D, DV = g.DV, DP = P * RP;
  const int BUF = NV * CT * DP + CT * CW + CT * 2;
  const int b = blockIdx.x, hd = blockIdx.y;
  const int t0 = g.seq_start[b], n = g.seq_start[b + 1] - t0;
  if (n <= 0) return;
  const int slices = (DV + CW - 1) / CW;
  const bool norm_col = MODE == WALK_MLSTM && (int)blockIdx.z == slices;
  const int c0 = norm_col ? 0 : blockIdx.z * CW, cw = norm_col ? 1 : min(CW, DV - c0);
  float* slot = g.state + (size_t)g.seq_slot[b] * g.state_stride + g.state_off;
  float* Sg = slot + (size_t)hd * g.head_stride + (norm_col ? (size_t)D * DV : (size_t)c0);
  const int s_row = norm_col ? 1 : DV;                    // from one row of the state to the next
  const int chunks = (n + CT - 1) / CT;
  const int walkers = CW / 2 * P, PREP = 8 * CT, warps = CT / 4;
  const int lane = threadIdx.x & 31;
  // places that no copy writes stay zero
  float* coefs = sw_smem + 3 * BUF;                       // [2][CT / 4][SW_COEF]
  float* so = coefs + 2 * warps * SW_COEF;                // [2][CT][CW]
  for (int e = threadIdx.x; e < 3 * BUF; e += blockDim.x) sw_smem[e] = 0.f;
  __syncthreads();

  if ((int)threadIdx.x >= walkers) {
    // ------------------------------------------------------------------ preparing warps
    const int tid = threadIdx.x - walkers, w = tid >> 5;
    const float* qh = g.q + (size_t)(hd / g.group) * D;
    const float* kh = g.k + (size_t)(hd / g.group) * D;
    const float* vh = g.v + (size_t)hd * DV + c0;
    const float* ah = CHANNEL ? g.a + (size_t)hd * D : nullptr;
    auto issue = [&](int ci) {
      if (ci < chunks) {
        float* qb = sw_smem + (ci % 3) * BUF;
        const int cn = min(CT, n - ci * CT);
        const size_t row0 = (size_t)t0 + ci * CT;
        float* vb = qb + NV * CT * DP;
        for (int tt = w; tt < cn; tt += warps) {      // a warp a token
          const float* qr = qh + (row0 + tt) * g.ldq;
          const float* kr = kh + (row0 + tt) * g.ldk;
          const float* ar = CHANNEL ? ah + (row0 + tt) * g.lda : nullptr;
          const float* vr = vh + (row0 + tt) * g.ldv;
          float* row = qb + tt * DP;
          if (g.vec) {
            for (int i = lane; i < D >> 2; i += 32) {
              float* d = row + (4 * i / R) * RP + (4 * i) % R;
              sw_copy<16>(d, qr + 4 * i);
              sw_copy<16>(d + CT * DP, kr + 4 * i);
              if (CHANNEL) sw_copy<16>(d + 2 * CT * DP, ar + 4 * i);
            }
            if (!norm_col && lane < cw >> 2) sw_copy<16>(vb + tt * CW + 4 * lane, vr + 4 * lane);
          } else {
            for (int i = lane; i < D; i += 32) {
              float* d = row + (i / R) * RP + (i % R);
              sw_copy<4>(d, qr + i);
              sw_copy<4>(d + CT * DP, kr + i);
              if (CHANNEL) sw_copy<4>(d + 2 * CT * DP, ar + i);
            }
            if (!norm_col)
              for (int i = lane; i < cw; i += 32) sw_copy<4>(vb + tt * CW + i, vr + i);
          }
        }
        if (!CHANNEL && tid < 2 * cn) {
          const int tt = tid >> 1;
          sw_copy<4>(vb + CT * CW + tid, ((tid & 1) ? g.s1 : g.s0) + (row0 + tt) * g.lds + hd);
        }
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float m = MODE == WALK_MLSTM ? slot[(size_t)hd * g.head_stride + (size_t)D * DV + D] : 0.f;
    const float par0 = !CHANNEL ? g.p0[hd] : 0.f, par1 = !CHANNEL ? g.p1[hd] : 0.f;

    auto prepare = [&](int ci) {
      float* qb = sw_smem + (ci % 3) * BUF + 4 * w * DP;      // this warp's group
      float* kb = qb + CT * DP;
      float* vb = sw_smem + (ci % 3) * BUF + NV * CT * DP;
      const float* sc = vb + CT * CW;                      // [CT][2]
      float* co = coefs + ((ci & 1) * warps + w) * SW_COEF;
      const int cn = min(CT, n - ci * CT), have = min(4, cn - 4 * w);
      // tokens behind the sequence's last: zeros, so that what an older chunk left has no part
      for (int tt = max(have, 0); tt < 4; ++tt) {
        for (int e = lane; e < DP; e += 32) qb[tt * DP + e] = kb[tt * DP + e] = 0.f;
        for (int e = lane; e < CW; e += 32) vb[(4 * w + tt) * CW + e] = 0.f;
      }
      if (norm_col && lane < 4) vb[(4 * w + lane) * CW] = lane < have ? 1.f : 0.f;
      __syncwarp();
      float a_tok = 1.f, b_tok = 0.f, em_tok = 0.f;           // mlstm, of token `lane`
      if (MODE == WALK_MLSTM) {
        float gi = -INFINITY, gf = 0.f, mo = 0.f, mn = 0.f;
        if (lane < cn) {
          gi = g.cap * tanhf((sc[2 * lane] + par0) / g.cap);
          gf = sw_log_sigmoid(g.cap * tanhf((sc[2 * lane + 1] + par1) / g.cap));
        }
        for (int tt = 0; tt < cn; ++tt) {                     // the running maximum, by all warps
          const float f = __shfl_sync(0xffffffffu, gf, tt), i = __shfl_sync(0xffffffffu, gi, tt);
          const float m_new = fmaxf(f + m, i);
          if (lane == tt) { mo = m; mn = m_new; }
          m = m_new;
        }
        if (lane < cn) {
          a_tok = expf(gf + mo - mn);
          b_tok = expf(gi - mn);
          em_tok = expf(-mn);
        }
      }
      if (have <= 0) return;
      float sums[32];
#pragma unroll
      for (int i = 0; i < 32; ++i) sums[i] = 0.f;
      for (int i = lane; i < D; i += 32) {
        const int at = (i / R) * RP + (i % R);
        float q[4], k[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          q[t] = qb[t * DP + at];
          k[t] = kb[t * DP + at];
        }
        if (CHANNEL) {
          float* ab = kb + CT * DP;
          float a[4];
          const float bias = g.abias[hd * D + i];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            const float z = ab[t * DP + at] + bias;
            a[t] = MODE == WALK_GLA ? expf(sw_log_sigmoid(z) * g.inv_tau) : expf(-expf(z));
            if (t >= have) a[t] = 1.f;
            if (MODE == WALK_GLA) q[t] *= g.q_scale;
          }
          // N_ts: gla counts the decays of s + 1 .. t, wkv of s + 1 .. t - 1 and u at t = s
          const float uk = MODE == WALK_WKV ? g.u[hd * D + i] : 1.f;
          int at_pair = 0;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            float left[4];
            left[t] = uk;
            if (t > 0) left[t - 1] = MODE == WALK_GLA ? a[t] : 1.f;
#pragma unroll
            for (int s = t - 2; s >= 0; --s) left[s] = left[s + 1] * a[s + 1];
#pragma unroll
            for (int s = 0; s <= t; ++s) sums[at_pair + s] = fmaf(q[t] * k[s], left[s], sums[at_pair + s]);
            at_pair += t + 1;
          }
          float pre = 1.f;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            if (MODE == WALK_GLA) pre *= a[t];
            qb[t * DP + at] = q[t] * pre;
            if (MODE == WALK_WKV) pre *= a[t];
          }
          float suf = 1.f;
#pragma unroll
          for (int t = 3; t >= 0; --t) {
            kb[t * DP + at] = k[t] * suf;
            suf *= a[t];
          }
          ab[at] = suf;                                       // the group's whole decay
        } else {
          int at_pair = 0;
#pragma unroll
          for (int t = 0; t < 4; ++t) {
#pragma unroll
            for (int s = 0; s <= t; ++s) sums[at_pair + s] = fmaf(q[t], k[s], sums[at_pair + s]);
            at_pair += t + 1;
          }
          if (MODE == WALK_DELTA) {
            at_pair = 10;
#pragma unroll
            for (int t = 1; t < 4; ++t) {
#pragma unroll
              for (int s = 0; s < t; ++s) sums[at_pair + s] = fmaf(k[t], k[s], sums[at_pair + s]);
              at_pair += t;
            }
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              sums[16 + t] = fmaf(q[t], q[t], sums[16 + t]);
              sums[20 + t] = fmaf(k[t], k[t], sums[20 + t]);
            }
          }
        }
      }
      const float sum = sums_by_lane<32>(sums, lane);
      const int t = (lane >> 2) & 3, s = lane & 3;
      const float qk = __shfl_sync(0xffffffffu, sum, t * (t + 1) / 2 + min(s, t));
      if (CHANNEL) {
        if (lane < 16) co[SW_N + lane] = s <= t ? qk : 0.f;
        return;
      }
      float dec, beta = 0.f, fq = g.q_scale, fk = 1.f;        // of token s = lane & 3
      if (MODE == WALK_DELTA) {
        const float ssq = __shfl_sync(0xffffffffu, sum, 16 + s), ssk = __shfl_sync(0xffffffffu, sum, 20 + s);
        const float zb = sc[2 * (4 * w + s)], zd = sc[2 * (4 * w + s) + 1];
        dec = s < have ? expf(-expf(par0) * sw_softplus(zd + par1)) : 1.f;
        beta = s < have ? 1.0f / (1.0f + expf(-zb)) : 0.f;
        // by choice: the zeros in a missing token's place have no unit length where unit_eps is 0
        fq = s < have ? g.q_scale / sqrtf(ssq + g.unit_eps) : 0.f;
        fk = s < have ? 1.0f / sqrtf(ssk + g.unit_eps) : 0.f;
      } else {
        dec = __shfl_sync(0xffffffffu, a_tok, 4 * w + s);
        beta = __shfl_sync(0xffffffffu, b_tok, 4 * w + s);
      }
      const float em = __shfl_sync(0xffffffffu, em_tok, 4 * w + s);
      float d[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) d[r] = __shfl_sync(0xffffffffu, dec, r);
      float between = 1.f, upto = 1.f, after = 1.f;           // s + 1 .. t; .. s; s + 1 ..
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        if (r > s && r <= t) between *= d[r];
        if (r <= s) upto *= d[r];
        if (r > s) after *= d[r];
      }
      const float fq_t = __shfl_sync(0xffffffffu, fq, t);
      if (MODE == WALK_DELTA) {
        const float c_t = __shfl_sync(0xffffffffu, beta * fk, t), fk_t = __shfl_sync(0xffffffffu, fk, t);
        const float kk = __shfl_sync(0xffffffffu, sum, 10 + (s < t ? t * (t - 1) / 2 + s : 0));
        if (lane < 16) {
          co[SW_N + lane] = s <= t ? fq_t * between * qk : 0.f;
          co[SW_M + lane] = s < t ? c_t * fk_t * between * kk : 0.f;
        }
        if (lane < 4) {
          co[SW_C + lane] = beta * fk;
          co[SW_E + lane] = beta * fk * fk * upto;
          co[SW_OG + lane] = fq * upto;
          co[SW_H + lane] = after;
        }
      } else {
        if (lane < 16) co[SW_N + lane] = s <= t ? fq_t * between * beta * qk : 0.f;
        if (lane < 4) {
          co[SW_OG + lane] = fq * upto;
          co[SW_H + lane] = beta * after;
          co[SW_EM + lane] = em;
        }
      }
      if (lane == 3) co[SW_A] = upto;
    };
    float* den = g.raw + (size_t)g.T * g.H * DV;              // mlstm: [T][H], then [B][H]
    auto store = [&](int ci) {
      const int cn = min(CT, n - ci * CT);
      const float* o = so + (ci & 1) * CT * CW;
      for (int tt = w; tt < cn; tt += warps) {
        const size_t row = (size_t)t0 + ci * CT + tt;
        if (norm_col) {
          if (lane == 0) den[row * g.H + hd] = o[tt * CW];
          continue;
        }
        float* r = g.raw + row * g.H * DV + (size_t)hd * DV + c0;
        for (int i = lane; i < cw; i += 32) r[i] = o[tt * CW + i];
      }
    };
    issue(0);
    issue(1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    sw_prep_sync(PREP);
    prepare(0);
    __syncthreads();
    for (int ci = 0; ci < chunks; ++ci) {
      if (ci + 1 < chunks) {
        issue(ci + 2);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        sw_prep_sync(PREP);
        prepare(ci + 1);
      }
      if (ci > 0) store(ci - 1);
      __syncthreads();
    }
    store(chunks - 1);
    if (norm_col && tid == 0) den[(size_t)g.T * g.H + (size_t)b * g.H + hd] = m;
    if (MODE == WALK_WKV && hd == 0 && blockIdx.z == 0) {
      const size_t row = ((size_t)t0 + n - 1) * g.W;
      for (int c = tid; c < g.W; c += PREP)
        (slot - g.W)[c] = g.h_bf16 ? __bfloat162float(((const __nv_bfloat16*)g.h)[row + c])
                           : ((const float*)g.h)[row + c];
    }
    return;
  }

  // -------------------------------------------------------------------- walking warps
  // a thread has R rows of two neighbouring columns; half of a pair of columns' lanes finish the
  // sums of the one, half those of the other
  const int j = 2 * (threadIdx.x / P), p = threadIdx.x % P, hc = P >> 1;
  const bool second = p & hc;
  const int mine = j + (second ? 1 : 0), pl = p & (hc - 1), my_t = pl & 3;
  f32_pair S[2][R / 2];
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < R / 2; ++r) {
      const int i = p * R + 2 * r;
      const bool own = j + c < cw;
      S[c][r] = pair_of(own && i < D ? Sg[(size_t)i * s_row + j + c] : 0.f,
                        own && i + 1 < D ? Sg[(size_t)(i + 1) * s_row + j + c] : 0.f);
    }
  __syncthreads();
  for (int ci = 0; ci < chunks; ++ci) {
    const float* buf = sw_smem + (ci % 3) * BUF;
    const int cn = min(CT, n - ci * CT), groups = (cn + 3) >> 2;
    for (int gr = 0; gr < groups; ++gr) {
      const float* qb = buf + 4 * gr * DP + p * RP;
      const float* kb = qb + CT * DP;
      const float* vb = buf + NV * CT * DP + 4 * gr * CW;
      const float* co = coefs + ((ci & 1) * warps + gr) * SW_COEF;
      // x of this lane's own column, of its neighbour's, and the group's numbers
      float x[4], other[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        x[t] = vb[t * CW + mine];
        if (MODE != WALK_DELTA) other[t] = vb[t * CW + (mine ^ 1)];
      }
      float4 c4, e4, m1, m2, m3, h4;
      float A1 = 1.f, og = 1.f, em = 0.f;
      if (MODE == WALK_DELTA) {
        c4 = *(const float4*)(co + SW_C);
        e4 = *(const float4*)(co + SW_E);
        m1 = *(const float4*)(co + SW_M + 4);
        m2 = *(const float4*)(co + SW_M + 8);
        m3 = *(const float4*)(co + SW_M + 12);
      }
      if (!CHANNEL) {
        h4 = *(const float4*)(co + SW_H);
        A1 = co[SW_A];
        og = co[SW_OG + my_t];
        if (MODE == WALK_MLSTM) em = co[SW_EM + my_t];
      }
      const float4 nn = *(const float4*)(co + SW_N + 4 * my_t);
      f32_pair rd[4][2], pd[4][2];
#pragma unroll
      for (int t = 0; t < 4; ++t) rd[t][0] = rd[t][1] = pd[t][0] = pd[t][1] = 0ull;
#pragma unroll
      for (int r = 0; r < R / 2; r += 2) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const ulonglong2 q = *(const ulonglong2*)(qb + t * DP + 2 * r);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            pair_fma(rd[t][c], S[c][r], q.x);
            pair_fma(rd[t][c], S[c][r + 1], q.y);
          }
          if (MODE == WALK_DELTA) {
            const ulonglong2 k = *(const ulonglong2*)(kb + t * DP + 2 * r);
#pragma unroll
            for (int c = 0; c < 2; ++c) {
              pair_fma(pd[t][c], S[c][r], k.x);
              pair_fma(pd[t][c], S[c][r + 1], k.y);
            }
          }
        }
      }
      // the four tokens' sums over the P lanes, the lane's own column's; both kinds side by side
      float q[4], rs[4];
#pragma unroll
      for (int t = 0; t < 4; ++t) {
        if (MODE == WALK_DELTA) {
          const float a = sw_added(pd[t][0]), b = sw_added(pd[t][1]);
          q[t] = (second ? b : a) + __shfl_xor_sync(0xffffffffu, second ? a : b, hc);
        }
        const float a = sw_added(rd[t][0]), b = sw_added(rd[t][1]);
        rs[t] = (second ? b : a) + __shfl_xor_sync(0xffffffffu, second ? a : b, hc);
      }
      for (int o = hc >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (MODE == WALK_DELTA) q[t] += __shfl_xor_sync(0xffffffffu, q[t], o);
          rs[t] += __shfl_xor_sync(0xffffffffu, rs[t], o);
        }
      if (MODE == WALK_DELTA) {
        x[0] = c4.x * x[0] - e4.x * q[0];
        x[1] = (c4.y * x[1] - e4.y * q[1]) - m1.x * x[0];
        x[2] = (c4.z * x[2] - e4.z * q[2] - m2.x * x[0]) - m2.y * x[1];
        x[3] = (c4.w * x[3] - e4.w * q[3] - m3.x * x[0] - m3.y * x[1]) - m3.z * x[2];
#pragma unroll
        for (int t = 0; t < 4; ++t) other[t] = __shfl_xor_sync(0xffffffffu, x[t], hc);
      }
      f32_pair xp[4][2];
      {
        const float h[4] = {CHANNEL ? 1.f : h4.x, CHANNEL ? 1.f : h4.y, CHANNEL ? 1.f : h4.z,
                            CHANNEL ? 1.f : h4.w};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float a = h[t] * (second ? other[t] : x[t]), b = h[t] * (second ? x[t] : other[t]);
          xp[t][0] = pair_of(a, a);
          xp[t][1] = pair_of(b, b);
        }
      }
      if (!CHANNEL) {
        const f32_pair A = pair_of(A1, A1);
#pragma unroll
        for (int r = 0; r < R / 2; ++r) {
          pair_mul(S[0][r], A);
          pair_mul(S[1][r], A);
        }
      } else {
        const float* ab = kb + CT * DP;
#pragma unroll
        for (int r = 0; r < R / 2; r += 2) {
          const ulonglong2 a = *(const ulonglong2*)(ab + 2 * r);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            pair_mul(S[c][r], a.x);
            pair_mul(S[c][r + 1], a.y);
          }
        }
      }
#pragma unroll
      for (int r = 0; r < R / 2; r += 2)
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const ulonglong2 k = *(const ulonglong2*)(kb + t * DP + 2 * r);
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            pair_fma(S[c][r], k.x, xp[t][c]);
            pair_fma(S[c][r + 1], k.y, xp[t][c]);
          }
        }
      // the outputs, a token a lane (a column's two lanes, P = 4, have two each)
      auto output = [&](int t, float r, float4 n4, float factor, float floor_) {
        float o = CHANNEL ? r : r * factor;
        // not by zeros for the later ones: an infinity of theirs must not reach this token
        o = fmaf(n4.x, x[0], o);
        if (t >= 1) o = fmaf(n4.y, x[1], o);
        if (t >= 2) o = fmaf(n4.z, x[2], o);
        if (t >= 3) o = fmaf(n4.w, x[3], o);
        // the normalizer's column leaves the denominator
        if (MODE == WALK_MLSTM && norm_col) o = fmaxf(fabsf(o), floor_) + 1e-6f;
        so[((ci & 1) * CT + 4 * gr + t) * CW + mine] = o;
      };
      if (pl < 4) output(my_t, my_t == 0 ? rs[0] : my_t == 1 ? rs[1] : my_t == 2 ? rs[2] : rs[3], nn, og, em);
      if (hc == 2)
        output(my_t + 2, my_t == 0 ? rs[2] : rs[3], *(const float4*)(co + SW_N + 4 * my_t + 8),
               CHANNEL ? 1.f : co[SW_OG + my_t + 2], MODE == WALK_MLSTM ? co[SW_EM + my_t + 2] : 0.f);
    }
    __syncthreads();
  }
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = p * R + r;
      if (j + c < cw && i < D) Sg[(size_t)i * s_row + j + c] = pair_half(S[c][r >> 1], r & 1);
    }
}

// out[t, hd, :] = o / rms(o) * normw * gate for every (token, head), a warp each; mlstm: o is first
// divided by its denominator, and the running maxima go into the state (here, since every block of
// the walk reads them when it begins).
template <typename T, bool VEC>
__global__ void state_walk_norm_kernel(const WalkArgs g) {
  mb_grid_wait();
  mb_grid_launch_next();
  const int idx = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int H = g.H, DV = g.DV;
  const float* den = g.raw + (size_t)g.T * H * DV;
  if (g.mode == WALK_MLSTM) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < g.B * H && g.seq_start[e / H + 1] > g.seq_start[e / H])
      g.state[(size_t)g.seq_slot[e / H] * g.state_stride + g.state_off +
              (size_t)(e % H) * g.head_stride + (size_t)g.D * DV + g.D] = den[(size_t)g.T * H + e];
  }
  if (idx >= g.T * H) return;
  const int t = idx / H, hd = idx - t * H;
  const float* o = g.raw + (size_t)idx * DV;
  const float* gr = g.gate + (size_t)t * g.ldg + (size_t)hd * DV;
  const float* nw = g.normw + (size_t)hd * g.norm_stride;
  T* out = (T*)g.out + (size_t)idx * DV;
  const float d = g.mode == WALK_MLSTM ? 1.0f / den[idx] : 1.0f;
  auto gated = [&](float ov, float gi, float w, float inv) {
    const float sig = 1.0f / (1.0f + expf(-gi));
    return ov * inv * w * (g.gate_kind ? sig : gi * sig);
  };
  float ss = 0.f;
  if (VEC) {
    for (int i = 4 * lane; i < DV; i += 128) {
      const float4 v = *(const float4*)(o + i);
      const float x = v.x * d, y = v.y * d, z = v.z * d, u = v.w * d;
      ss = fmaf(x, x, fmaf(y, y, fmaf(z, z, fmaf(u, u, ss))));
    }
    const float inv = d / sqrtf(warp_sum(ss) / (float)DV + g.eps);
    for (int i = 4 * lane; i < DV; i += 128) {
      const float4 v = *(const float4*)(o + i), gi = *(const float4*)(gr + i), w = *(const float4*)(nw + i);
      store4<T>(out + i, make_float4(gated(v.x, gi.x, w.x, inv), gated(v.y, gi.y, w.y, inv),
                                     gated(v.z, gi.z, w.z, inv), gated(v.w, gi.w, w.w, inv)));
    }
  } else {
    for (int i = lane; i < DV; i += 32) ss = fmaf(o[i] * d, o[i] * d, ss);
    const float inv = d / sqrtf(warp_sum(ss) / (float)DV + g.eps);
    for (int i = lane; i < DV; i += 32) out[i] = from_f32<T>(gated(o[i], gr[i], nw[i], inv));
  }
}

static int launch_norm(const WalkArgs& g, cudaStream_t s) {
  const bool vec = g.DV % 4 == 0 && g.ldg % 4 == 0 && g.norm_stride % 4 == 0 &&
                   (((uintptr_t)g.raw | (uintptr_t)g.gate | (uintptr_t)g.normw) & 15) == 0 &&
                   ((uintptr_t)g.out & (g.out_bf16 ? 7 : 15)) == 0;
  const dim3 grid((g.T * g.H + 7) / 8);
#define NORM(T_)                                                                   \
  if (vec) mb_launch(state_walk_norm_kernel<T_, true>, grid, dim3(256), 0, s, g);  \
  else mb_launch(state_walk_norm_kernel<T_, false>, grid, dim3(256), 0, s, g)
  if (g.out_bf16) { NORM(__nv_bfloat16); } else { NORM(float); }
#undef NORM
  MB_CHECK_LAUNCH("mb_state_walk");
}

static int walk_lanes(int D, int R) {
  int p = 4;
  while (p * R < D) p *= 2;
  return p;
}

static size_t walk_smem(int mode, int P, int R, int CW, int CT) {
  const int nv = mode == WALK_GLA || mode == WALK_WKV ? 3 : 2;
  return (3 * ((size_t)nv * CT * P * (R + 4) + CT * CW + CT * 2) + 2 * (CT / 4) * SW_COEF +
          2 * CT * CW) * sizeof(float);
}

// Heads of up to 256 x 1024 values. `raw` needs T H DV floats, for mlstm T H + B H more.
MB_EXPORT int mb_state_walk(const WalkArgs* args, int sms, void* stream) {
  WalkArgs g = *args;
  if (g.T <= 0 || g.B <= 0) return 0;
  if (g.D <= 0 || g.D > 256 || g.DV <= 0 || g.DV > (g.mode == WALK_MLSTM ? 512 : 1024))
    MB_FAIL("mb_state_walk: heads of %d x %d values (at most 256 x 1024, mlstm 256 x 512)", g.D, g.DV);
  if (g.group <= 0 || g.H % g.group) MB_FAIL("mb_state_walk: %d heads in groups of %d", g.H, g.group);
  if (g.mode < 0 || g.mode > 3) MB_FAIL("mb_state_walk: mode %d", g.mode);
  // blocks of a step with R rows a walking thread and so many walking threads a block
  const auto blocks = [&](int R, int threads) {
    const int cw = 2 * threads / walk_lanes(g.D, R);
    return (long long)g.B * g.H * ((g.DV + cw - 1) / cw + (g.mode == WALK_MLSTM ? 1 : 0));
  };
  // Rows of a walking thread: 8 (twice the lanes a column) shorten a group's chain and serve a step
  // whose blocks all run at once (one fits a multiprocessor), as long as chunks of 32 tokens fit; 16
  // read least from shared memory and have half the blocks. 500 tokens a prompt, us with 8 | 16:
  // delta, 16 heads of 128 x 128, one prompt 101 | 133, two 198 | 142, four 394 | 281; mlstm, 8 heads
  // of 128 x 128, two 89 | 94, three 172 | 101, four 174 | 191 (of 111 to 900 tokens 240 | 170); wkv,
  // 32 heads of 64 x 64, two 85 | 93, three 162 | 107.
  const int P8 = walk_lanes(g.D, 8);
  const int R = blocks(8, 128) <= sms && walk_smem(g.mode, P8, 8, 2 * 128 / P8, 32) <= 200 * 1024 ? 8 : 16;
  const int P = walk_lanes(g.D, R);
  // walking threads of a block: 128, or 64 where even twice as many blocks all run at once
  const int threads = blocks(R, 64) <= sms ? 64 : 128;
  const int CW = 2 * threads / P, slices = (g.DV + CW - 1) / CW;
  const int CT = walk_smem(g.mode, P, R, CW, 32) <= 200 * 1024 ? 32 : 16;
  g.vec = g.D % 4 == 0 && g.DV % 4 == 0 && CW % 4 == 0 && g.ldq % 4 == 0 && g.ldk % 4 == 0 &&
          g.ldv % 4 == 0 && g.lda % 4 == 0 &&
          (((uintptr_t)g.q | (uintptr_t)g.k | (uintptr_t)g.v | (uintptr_t)g.a) & 15) == 0;
  const size_t smem = walk_smem(g.mode, P, R, CW, CT);
  const dim3 grid(g.B, g.H, slices + (g.mode == WALK_MLSTM ? 1 : 0));
  cudaStream_t s = (cudaStream_t)stream;
#define GO(M_, R_)                                                                             \
  {                                                                                            \
    static unsigned long long allowed = 0;                                                     \
    const cudaError_t e =                                                                      \
        mb_allow_smem((const void*)state_walk_kernel<M_, R_>, 224 * 1024, &allowed);           \
    if (e != cudaSuccess) MB_FAIL("mb_state_walk: %s", cudaGetErrorString(e));                 \
    mb_launch(state_walk_kernel<M_, R_>, grid, dim3(threads + 8 * CT), smem, s, g, P, CW, CT); \
  }
#define GOR(M_) if (R == 8) GO(M_, 8) else GO(M_, 16)
  switch (g.mode) {
    case WALK_GLA: GOR(WALK_GLA) break;
    case WALK_DELTA: GOR(WALK_DELTA) break;
    case WALK_MLSTM: GOR(WALK_MLSTM) break;
    default: GOR(WALK_WKV)
  }
#undef GOR
#undef GO
  return launch_norm(g, s);
}

// The delta rule and the matrix memory in chunks of 32 tokens (state_chunks.cuh): heads of up to 128 x
// 1024 (mlstm 128 x 512) values, multiples of 16 both, rows on 16-byte boundaries. `scratch`:
// `scratch_floats` floats, at least mb_state_chunks_scratch of one chunk a sequence; with less than all
// chunks' room the chunks go in several passes. `longest`: the most new tokens of a sequence.
MB_EXPORT long long mb_state_chunks_scratch(int mode, int B, int H, int D, int DV, int chunks) {
  return (long long)B * H * ((long long)sc_chunk_floats(mode == WALK_DELTA, D, DV) * chunks + 2);
}

MB_EXPORT int mb_state_chunks(const WalkArgs* args, float* scratch, long long scratch_floats, int longest,
                              int sms, void* stream) {
  const WalkArgs g = *args;
  if (g.T <= 0 || g.B <= 0) return 0;
  const bool delta = g.mode == WALK_DELTA;
  if (!delta && g.mode != WALK_MLSTM) MB_FAIL("mb_state_chunks: mode %d", g.mode);
  if (g.D <= 0 || g.D > 128 || g.D % 16 || g.DV <= 0 || g.DV % 16 || g.DV > (delta ? 1024 : 512))
    MB_FAIL("mb_state_chunks: heads of %d x %d values", g.D, g.DV);
  if (g.group <= 0 || g.H % g.group) MB_FAIL("mb_state_chunks: %d heads in groups of %d", g.H, g.group);
  if (g.ldq % 4 || g.ldk % 4 || g.ldv % 4 ||
      (((uintptr_t)g.q | (uintptr_t)g.k | (uintptr_t)g.v | (uintptr_t)scratch) & 15))
    MB_FAIL("mb_state_chunks: rows off the 16-byte boundaries");
  const int all = (longest + SC_C - 1) / SC_C;
  const long long each = (long long)g.B * g.H * sc_chunk_floats(delta, g.D, g.DV), maxima = 2ll * g.B * g.H;
  const long long fit = (scratch_floats - maxima) / each;
  const int per_seq = fit < all ? (int)fit : all;
  if (all < 1 || per_seq < 1) MB_FAIL("mb_state_chunks: %lld floats of scratch are too few", scratch_floats);
  cudaStream_t s = (cudaStream_t)stream;
  const size_t prep_smem = (2 * SC_C * (g.D + 8) + SC_C * 33 + 2 * SC_C * 36 + 16 * 17 + 3 * SC_C +
                            (delta ? (g.DV <= SC_V_HERE ? SC_C * (size_t)(g.DV + 8) : 0) : 2 * (size_t)per_seq)) * 4;
  const int warps = g.D / 16, rows = delta ? 2 * SC_C : SC_C, threads = 32 * (warps < 4 ? 4 : warps);
  const dim3 walk(g.B, g.H, g.DV / SC_COLS + (delta ? 0 : 1));
  size_t walk_smem = ((size_t)warps * rows * SC_PART + SC_C * SC_PART + 3 * SC_COLS * 20) * 4;
  // Where every walking CTA can have a multiprocessor for itself it asks for more than half of the shared
  // memory: the CTAs come while preparing blocks still run, and two of them on one multiprocessor made
  // the walk a fifth longer (mlstm, 1,000 tokens, us of the whole call without | with: 8 heads of 128 x
  // 128 124 | 104, 16 of 64 x 128 120 | 105; delta, 8 heads of 64 x 128 98 | 89).
  if ((long long)walk.x * walk.y * walk.z <= sms && walk_smem < 116 * 1024) walk_smem = 116 * 1024;
  if (prep_smem > 200 * 1024) MB_FAIL("mb_state_chunks: %d chunks in one pass", per_seq);
  static unsigned long long allowed[4] = {0, 0, 0, 0};
  const void* kernels[4] = {(const void*)state_chunk_prep_kernel<false>, (const void*)state_chunk_prep_kernel<true>,
                            (const void*)state_chunk_walk_kernel<false>, (const void*)state_chunk_walk_kernel<true>};
  for (int i = 0; i < 4; ++i) {
    const cudaError_t e = mb_allow_smem(kernels[i], 200 * 1024, &allowed[i]);
    if (e != cudaSuccess) MB_FAIL("mb_state_chunks: %s", cudaGetErrorString(e));
  }
  float* m[2] = {scratch + scratch_floats - maxima, scratch + scratch_floats - maxima / 2};
  int pass = 0;
  for (int c = 0; c < all; c += per_seq, ++pass) {
    const int now = all - c < per_seq ? all - c : per_seq;
    const dim3 grid((unsigned)(g.B * now), g.H);
    if (delta) {
      mb_launch(state_chunk_prep_kernel<true>, grid, dim3(256), prep_smem, s, g, scratch, c, now,
                (const float*)m[pass & 1], m[1 - (pass & 1)]);
      mb_launch(state_chunk_walk_kernel<true>, walk, dim3(threads), walk_smem, s, g, (const float*)scratch, c, now);
    } else {
      mb_launch(state_chunk_prep_kernel<false>, grid, dim3(256), prep_smem, s, g, scratch, c, now,
                (const float*)m[pass & 1], m[1 - (pass & 1)]);
      mb_launch(state_chunk_walk_kernel<false>, walk, dim3(threads), walk_smem, s, g, (const float*)scratch, c, now);
    }
  }
  return launch_norm(g, s);
}
