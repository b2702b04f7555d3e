// The delta rule and the matrix memory in chunks of 32 tokens, for steps whose sequences are long
// (state_walk.cu holds the recurrences, their other forms and the entry points). With S0 the state
// before a chunk, dec_t the decays, D_ts the product of those of s + 1 .. t, G_t that of all up to t:
//
//   delta    (I + M) U = beta V - diag(beta G) K S0,  M_ts = beta_t D_ts (k_t . k_s), s < t
//            U = U1 - W S0 with T = (I + M)^-1, U1 = T beta V, W = T diag(beta G) K
//   mlstm    U = V
//   both     o_t = G_t q_t . S0 + sum_{s <= t} N_ts u_s,  N_ts = D_ts (q_t . k_s) (mlstm: times b_s)
//            S = G_31 S0 + sum_s D_31,s k_s u_s^T (mlstm: times b_s)
//
// (The delta rule in chunks: S. Yang et al., Parallelizing linear transformers with the delta rule over
// sequence length, 2024.)
//
// All that does not need S0 is made by a block per chunk and head (state_chunk_prep_kernel), all chunks
// at once, and left in scratch as the operands that the walk's lanes will hold. The walk
// (state_chunk_walk_kernel) is then three small products a chunk with two barriers between them, a CTA
// per head and 16 columns of the state; its operands come straight from L2 into registers, a chunk
// ahead.
//
// Products go through mma.sync (m16n8k16) with every float32 value cut into three bfloat16 parts that
// sum up to it (common.cuh), six products of parts, the smallest first: an accumulator cuts off what falls
// behind its last place, so the leading products come last and few to an accumulator, and sums over
// warps and chunks are made with float32 additions. What goes into the state chunk after chunk leans to
// neither side: the first operand's leading part is the nearest one, and what an accumulator cut off its
// leading products is made once more and added (2,000 tokens, 128 x 128, delta, the mean over three
// inputs of the state's relative error against float64: by fours 1.16e-7, this 1.08e-7; on the first of
// them 0.94e-7 and 1.20e-7, without either 1.67e-7). Decays are products, never quotients. The state
// stands as fragments in registers, transposed, so that a chunk's result is the next one's operand.
// What bounds the walk: a chunk's chain of two rounds of MMAs, two barriers and a sum over the warps
// (some 4,000 cycles, of which the tensor pipe works 1,500); the preparing blocks: instructions (issue
// slots half busy, most of them cut values). One prompt of 2,048 tokens, 16 heads of 128 x 128, delta:
// by fours 366 us -> 56 + 150; four prompts of 111 to 900, 8 heads, mlstm: 185 -> 23 + 86 (before what
// keeps the sums from leaning was added: 9 and 7 us more; the whole mixers 491 -> 323, 261 -> 180). With the
// operands in shared memory and cut there a chunk took twice the instructions (97 + 234 us).
// Keys, queries, a state or an update that may be no exact sums of three parts (an infinity, a NaN, a value
// below 2^-110) and products of keys and queries that overflow take the chunk through a form that goes
// token by token, so that they reach no earlier token and keep their 24 bits. A state or an output that
// overflows at the end of a chunk is an infinity there. Factors with decays in them may lose up to 2^-133,
// bfloat16's last place, beside the token's own, which is not decayed.
#pragma once
#include "mma_common.cuh"

constexpr int SC_C = 32;          // tokens of a chunk
constexpr int SC_COLS = 16;       // columns of the state of a walking CTA
constexpr int SC_V_HERE = 256;   // values of a row that the preparing block brings into shared memory
constexpr int SC_META = 192;      // G_31, whether something is no number; of each token: see below
constexpr int SC_FQ = 32, SC_FK = 64, SC_DEC = 96, SC_BETA = 128, SC_EM = 160;

// A fragment of the second operand (16 x 8), cut: 32 lanes' hi and mid (16 bytes each), then lo (8)
constexpr int SC_FRAG = 192;

// A chunk's place in scratch: meta; N, fragment (8 tokens t, 16 tokens s) at 2 nt + kt; of each 16 rows
// of the state q times G (4 fragments of 8 tokens), k times D_31,s (fragment (8 rows, 16 tokens) at
// 2 j + kt); delta: W like q, then U1 [32][DV]
__host__ __device__ inline size_t sc_chunk_floats(bool delta, int D, int DV) {
  return SC_META + 8 * SC_FRAG + (size_t)(delta ? 12 : 8) * SC_FRAG * (D / 16) + (delta ? SC_C * (size_t)DV : 0);
}

struct FragA { uint32_t hi[4], mid[4], lo[4]; };
struct FragB { uint32_t hi[2], mid[2], lo[2]; };
// The first operand's cut: the first part is the nearest, so that what the six products leave out (its
// rest times the second operand's) has either sign
__device__ __forceinline__ Cut2 cut_near(float a, float b) {
  Cut2 c;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(c.hi) : "f"(b), "f"(a));
  const f32_pair v = pair_of(a - __uint_as_float(c.hi << 16), b - __uint_as_float(c.hi & 0xffff0000u));
  c.mid = upper_halves(v);
  const f32_pair q = pair_sub_upper(v);
  c.lo = upper_halves(q);
  c.rest = (uint32_t)q | (uint32_t)(q >> 32);
  return c;
}
__device__ __forceinline__ uint32_t put_a(FragA& f, int i, float a, float b) {      // gives the cut's rest
  const Cut2 c = cut_near(a, b);
  f.hi[i] = c.hi; f.mid[i] = c.mid; f.lo[i] = c.lo;
  return c.rest;
}
__device__ __forceinline__ void put_b(FragB& f, int i, float a, float b) {
  const Cut2 c = cut(a, b);
  f.hi[i] = c.hi; f.mid[i] = c.mid; f.lo[i] = c.lo;
}
__device__ __forceinline__ void mma_parts(float* d, const uint32_t* a, const uint32_t* b) {
  mma_bf16(d, a[0], a[1], a[2], a[3], b[0], b[1]);
}
// The six products for N accumulators, one kind for all of them after the other: no product waits for
// the one before it
template <int N> __device__ __forceinline__ void mma_low(float (*d)[4], const FragA& a, const FragB* b) {
#pragma unroll
  for (int i = 0; i < N; ++i) mma_parts(d[i], a.lo, b[i].hi);
#pragma unroll
  for (int i = 0; i < N; ++i) mma_parts(d[i], a.hi, b[i].lo);
#pragma unroll
  for (int i = 0; i < N; ++i) mma_parts(d[i], a.mid, b[i].mid);
#pragma unroll
  for (int i = 0; i < N; ++i) mma_parts(d[i], a.mid, b[i].hi);
#pragma unroll
  for (int i = 0; i < N; ++i) mma_parts(d[i], a.hi, b[i].mid);
}
template <int N> __device__ __forceinline__ void mma_high(float (*d)[4], const FragA& a, const FragB* b) {
#pragma unroll
  for (int i = 0; i < N; ++i) mma_parts(d[i], a.hi, b[i].hi);
}
// The leading products, to which an accumulator that starts at zero leaves what it cuts off: the same
// products again less their sum
template <int N> __device__ __forceinline__ void mma_rest(float (*low)[4], const float (*high)[4], const FragA& a, const FragB* b) {
  float d[N][4];
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) d[i][e] = -high[i][e];
  mma_high<N>(d, a, b);
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int e = 0; e < 4; ++e) low[i][e] += d[i][e];
}
__device__ __forceinline__ void store_frag(float* at, int lane, const FragB& f) {
  ((uint4*)at)[lane] = make_uint4(f.hi[0], f.hi[1], f.mid[0], f.mid[1]);
  ((uint2*)(at + 128))[lane] = make_uint2(f.lo[0], f.lo[1]);
}
// (volatile: a load stays behind the products that use what stood in its registers before; moved ahead
// of them it would need registers of its own and a copy that waits for it)
__device__ __forceinline__ void load_frag(FragB& f, const float* at, int lane) {
  asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(f.hi[0]), "=r"(f.hi[1]), "=r"(f.mid[0]), "=r"(f.mid[1])
               : "l"((const uint4*)at + lane));
  asm volatile("ld.global.nc.v2.u32 {%0, %1}, [%2];"
               : "=r"(f.lo[0]), "=r"(f.lo[1]) : "l"((const uint2*)(at + 128) + lane));
}
__device__ __forceinline__ float4 load_once4(const float* p) {
  float4 v;
  asm volatile("ld.global.nc.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ bool no_number(float4 v) {
  return !(0.f * v.x + 0.f * v.y + 0.f * v.z + 0.f * v.w == 0.f);
}
__device__ __forceinline__ void sc_copy16(float* dst, const float* src, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;"
               ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(valid ? 16 : 0) : "memory");
}

// ---------------------------------------------------------------------------- a chunk's factors
// Block (sequence and chunk of this pass, head). `chunk0`: the pass's first chunk of every sequence,
// `per_seq` chunks of each; `m_in`, `m_out`: mlstm's running maxima at the pass's ends, [B][H] each.
template <bool DELTA>
__global__ void __launch_bounds__(256, DELTA ? 2 : 3)
state_chunk_prep_kernel(const WalkArgs g, float* __restrict__ scratch, int chunk0, int per_seq,
                        const float* __restrict__ m_in, float* __restrict__ m_out) {
  mb_grid_wait();
  mb_grid_launch_next();
  const int b = blockIdx.x / per_seq, ci = blockIdx.x - b * per_seq, chunk = chunk0 + ci;
  const int hd = blockIdx.y, D = g.D, DV = g.DV, DP = D + 8;
  const int t0 = g.seq_start[b], n = g.seq_start[b + 1] - t0, cn = min(SC_C, n - chunk * SC_C);
  if (cn <= 0) return;
  const size_t row0 = (size_t)t0 + chunk * SC_C;
  extern __shared__ __align__(16) float sm[];
  const int VP = DV + 8;
  const bool v_here = DELTA && DV <= SC_V_HERE;
  float* ks = sm;                        // [32][DP] keys, of unit length for delta
  float* qs = ks + SC_C * DP;            // [32][DP]
  float* Dm = qs + SC_C * DP;            // [32][33] D_ts (mlstm: b_s D_ts), zero for s > t
  float* Mx = Dm + SC_C * 33;            // [32][36]
  float* Tx = Mx + SC_C * 36;            // [32][36]
  float* Px = Tx + SC_C * 36;            // [16][17]
  float* G = Px + 16 * 17;               // of each token: [32] each
  float* last = G + SC_C;                // D_31,s (mlstm: times b_s)
  float* beta = last + SC_C;
  float* vs = beta + SC_C;               // delta: [32][VP] values, where they fit
  float* tf = vs;                        // mlstm: [per_seq][2] of the chunks so far
  float* out = scratch + ((size_t)blockIdx.x * g.H + hd) * sc_chunk_floats(DELTA, D, DV);
  float* oN = out + SC_META;
  float* oQ = oN + 8 * SC_FRAG;
  float* oK = oQ + 4 * SC_FRAG * (D / 16);
  float* oW = oK + 4 * SC_FRAG * (D / 16);
  float* oU = oW + 4 * SC_FRAG * (D / 16);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  bool odd = false;

  const float* vb = g.v + row0 * g.ldv + (size_t)hd * DV;
  if (v_here) {
    for (int t = warp; t < SC_C; t += 8)
      for (int i = 4 * lane; i < DV; i += 128) sc_copy16(vs + t * VP + i, vb + (t < cn ? (size_t)t * g.ldv + i : 0), t < cn);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  {
    float4 q[4], k[4];
    const int i = 4 * lane;
    const size_t at = (size_t)(hd / g.group) * D + i;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = warp + 8 * r;
      const bool ok = t < cn && i < D;
      q[r] = ok ? *(const float4*)(g.q + (row0 + t) * g.ldq + at) : make_float4(0.f, 0.f, 0.f, 0.f);
      k[r] = ok ? *(const float4*)(g.k + (row0 + t) * g.ldk + at) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int t = warp + 8 * r;
      odd |= no_number(q[r]) || no_number(k[r]);
      float fq = g.q_scale, fk = 1.f;
      if (DELTA) {
        const float sq = warp_sum(q[r].x * q[r].x + q[r].y * q[r].y + q[r].z * q[r].z + q[r].w * q[r].w);
        const float sk = warp_sum(k[r].x * k[r].x + k[r].y * k[r].y + k[r].z * k[r].z + k[r].w * k[r].w);
        fq = t < cn ? g.q_scale / sqrtf(sq + g.unit_eps) : 0.f;
        fk = t < cn ? 1.0f / sqrtf(sk + g.unit_eps) : 0.f;
        odd |= !(0.f * fq + 0.f * fk == 0.f);
      }
      if (i < D) {
        const float4 x = make_float4(q[r].x * fq, q[r].y * fq, q[r].z * fq, q[r].w * fq);
        const float4 y = make_float4(k[r].x * fk, k[r].y * fk, k[r].z * fk, k[r].w * fk);
        odd |= too_small_to_cut(x) | too_small_to_cut(y);
        *(float4*)(qs + t * DP + i) = x;
        *(float4*)(ks + t * DP + i) = y;
      }
      if (lane == 0) {
        out[SC_FQ + t] = fq;
        out[SC_FK + t] = fk;
      }
    }
  }
  // mlstm: what a chunk's gates do to the running maximum, m -> max(F + m, M), of token `lane` from the
  // chunk's first on
  const float p0 = g.p0[hd], p1 = g.p1[hd];
  auto gates_of = [&](int c, float& gi, float& gf, float& F, float& M) {
    const int t = c * SC_C + lane;
    gi = -INFINITY;
    gf = 0.f;
    if (t < n) {
      const size_t at = ((size_t)t0 + t) * g.lds + hd;
      gi = g.cap * tanhf((g.s0[at] + p0) / g.cap);
      gf = sw_log_sigmoid(g.cap * tanhf((g.s1[at] + p1) / g.cap));
    }
    F = gf;
    M = gi;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float Fb = __shfl_up_sync(0xffffffffu, F, o), Mb = __shfl_up_sync(0xffffffffu, M, o);
      if (lane >= o) {
        M = fmaxf(Mb + F, M);
        F += Fb;
      }
    }
  };
  if (!DELTA)
    for (int c = warp; c < ci; c += 8) {
      float gi, gf, F, M;
      gates_of(chunk0 + c, gi, gf, F, M);
      if (lane == 31) {
        tf[2 * c] = F;
        tf[2 * c + 1] = M;
      }
    }
  __syncthreads();
  if (warp == 0) {
    float dec = 1.f, be = 0.f, em = 0.f;
    if (DELTA) {
      if (lane < cn) {
        const float* s = g.s0 + (row0 + lane) * g.lds + hd;
        be = 1.0f / (1.0f + expf(-*s));
        dec = expf(-expf(p0) * sw_softplus(g.s1[(row0 + lane) * g.lds + hd] + p1));
      }
    } else {
      float gi, gf, F, M;
      gates_of(chunk, gi, gf, F, M);
      float m = chunk0 ? m_in[(size_t)b * g.H + hd]
                       : (g.state + (size_t)g.seq_slot[b] * g.state_stride + g.state_off)
                             [(size_t)hd * g.head_stride + (size_t)D * DV + D];
      for (int c = 0; c < ci; ++c) m = fmaxf(tf[2 * c] + m, tf[2 * c + 1]);
      const float mt = fmaxf(F + m, M), up = __shfl_up_sync(0xffffffffu, mt, 1), before = lane ? up : m;
      dec = expf(gf + before - mt);
      be = expf(gi - mt);
      em = expf(-mt);
      if (lane == 31) {
        if (ci == per_seq - 1) m_out[(size_t)b * g.H + hd] = mt;
        if (chunk * SC_C + cn == n)
          g.raw[(size_t)g.T * g.H * DV + (size_t)g.T * g.H + (size_t)b * g.H + hd] = mt;
      }
    }
    odd |= !(0.f * dec + 0.f * be == 0.f);
    float pre = dec, suf = dec;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float a = __shfl_up_sync(0xffffffffu, pre, o), z = __shfl_down_sync(0xffffffffu, suf, o);
      if (lane >= o) pre *= a;
      if (lane + o < 32) suf *= z;
    }
    const float next = __shfl_down_sync(0xffffffffu, suf, 1), after = lane < 31 ? next : 1.f;
    G[lane] = pre;
    beta[lane] = be;
    last[lane] = DELTA ? after : after * be;
    out[SC_DEC + lane] = dec;
    out[SC_BETA + lane] = be;
    out[SC_EM + lane] = em;
    if (lane == 31) out[0] = pre;
    float p = DELTA ? 1.f : be;
#pragma unroll
    for (int t = 0; t < 32; ++t) {
      const float d = __shfl_sync(0xffffffffu, dec, t);
      if (t > lane) p *= d;
      Dm[t * 33 + lane] = t >= lane ? p : 0.f;
    }
  }
  __syncthreads();

  // q . k and k . k: warps of (which, 16 rows t, 16 columns s)
  const int gr = lane >> 2, tq = lane & 3;
  {
    const bool kk = warp >= 4;
    const int mt = (warp >> 1) & 1, nh = warp & 1;
    if (DELTA || !kk) {
      const float* a0 = (kk ? ks : qs) + (16 * mt + gr) * DP + 2 * tq;
      float sum[2][4] = {}, low[2][4] = {};
      if (mt >= nh)
        for (int k = 0; k < D; k += 16) {
          FragA a;
          FragB f[2];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float2 x = *(const float2*)(a0 + (e & 1) * 8 * DP + k + 8 * (e >> 1));
            put_a(a, e, x.x, x.y);
          }
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float2 y = *(const float2*)(ks + (16 * nh + 8 * j + gr) * DP + 2 * tq + k + 8 * e);
              put_b(f[j], e, y.x, y.y);
            }
          mma_low<2>(low, a, f);
          float high[2][4] = {};
          mma_high<2>(high, a, f);
#pragma unroll
          for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[j][e] += high[j][e];
        }
      FragB f[2];      // of N: tokens t of row r's eight, s of the 16 nh on
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int t = 16 * mt + gr + 8 * r, s = 16 * nh + 8 * j + 2 * tq;
          float v[2];
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float x = sum[j][2 * r + e] + low[j][2 * r + e];
            odd |= !(fabsf(x) <= 3.402823466e38f);      // an overflow
            if (!kk) v[e] = s + e <= t ? x * Dm[t * 33 + s + e] : 0.f;
            else v[e] = s + e < t ? beta[t] * Dm[t * 33 + s + e] * x : 0.f;
          }
          if (kk) *(float2*)(Mx + t * 36 + s) = make_float2(v[0], v[1]);
          else put_b(f[r], j, v[0], v[1]);
        }
      if (!kk) {
        store_frag(oN + (4 * mt + nh) * SC_FRAG, lane, f[0]);
        store_frag(oN + (4 * mt + 2 + nh) * SC_FRAG, lane, f[1]);
      }
    }
  }
  const int any_odd = __syncthreads_or(odd);
  if (threadIdx.x == 0) out[1] = any_odd ? 1.f : 0.f;
  if (DELTA) {
    // T = (I + M)^-1: its two blocks of 16 on the diagonal by forward substitution, a column a lane,
    // then the one below them
    if (warp == 0) {
      const int h = 16 * (lane >> 4), c = lane & 15;
      float x[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) {
        float s[4] = {i == c ? 1.f : 0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int r = 0; r < i; r += 4) {
          const float4 m = *(const float4*)(Mx + (h + i) * 36 + h + r);
          s[0] = fmaf(-m.x, x[r], s[0]);
          if (r + 1 < i) s[1] = fmaf(-m.y, x[r + 1], s[1]);
          if (r + 2 < i) s[2] = fmaf(-m.z, x[r + 2], s[2]);
          if (r + 3 < i) s[3] = fmaf(-m.w, x[r + 3], s[3]);
        }
        x[i] = (s[0] + s[1]) + (s[2] + s[3]);
        Tx[(h + i) * 36 + h + c] = x[i];
        if (h == 0) Tx[i * 36 + 16 + c] = 0.f;
      }
    }
  }
  // q times G and k times D_31,s as the walk's fragments
  const int frags = D / 16 * 4, first = DELTA ? warp - 1 : warp, others = DELTA ? 7 : 8;
  if (first >= 0)
    for (int e = first; e < 2 * frags; e += others) {
      FragB f;
      if (e < frags) {
        const int t = 8 * (e & 3) + gr;
        const float* q = qs + t * DP + 16 * (e >> 2) + 2 * tq;
        const float2 x = *(const float2*)q, y = *(const float2*)(q + 8);
        put_b(f, 0, x.x * G[t], x.y * G[t]);
        put_b(f, 1, y.x * G[t], y.y * G[t]);
        store_frag(oQ + e * SC_FRAG, lane, f);
      } else {
        const int r = e - frags, t = 16 * (r & 1) + 2 * tq;
        const float* k = ks + t * DP + 8 * (r >> 1) + gr;
        put_b(f, 0, k[0] * last[t], k[DP] * last[t + 1]);
        put_b(f, 1, k[8 * DP] * last[t + 8], k[9 * DP] * last[t + 9]);
        store_frag(oK + r * SC_FRAG, lane, f);
      }
    }
  if (!DELTA) return;
  __syncthreads();
  {
    const int i = threadIdx.x >> 4, c = threadIdx.x & 15;      // M21 T11, then T21 = -T22 (M21 T11)
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < 16; ++r) s = fmaf(Mx[(16 + i) * 36 + r], Tx[r * 36 + c], s);
    Px[i * 17 + c] = s;
    __syncthreads();
    s = 0.f;
#pragma unroll
    for (int r = 0; r < 16; ++r) s = fmaf(Tx[(16 + i) * 36 + 16 + r], Px[r * 17 + c], s);
    Tx[(16 + i) * 36 + c] = -s;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
  // W = T diag(beta G) K by warps 0 to 3, U1 = T diag(beta) V by warps 4 to 7: 16 columns at a time
  const bool is_u = warp >= 4;
  FragA a[2][2];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int kt = 0; kt < 2; ++kt)
#pragma unroll
      for (int e = 0; e < 4; ++e) {      // rows gr, gr + 8; columns 2 tq, 2 tq + 8 on
        const int t = 16 * mt + gr + 8 * (e & 1), s = 16 * kt + 2 * tq + 8 * (e >> 1);
        const float2 x = *(const float2*)(Tx + t * 36 + s);
        put_a(a[mt][kt], e, x.x * beta[s] * (is_u ? 1.f : G[s]), x.y * beta[s + 1] * (is_u ? 1.f : G[s + 1]));
      }
  for (int ct = warp & 3; ct < (is_u ? DV : D) / 16; ct += 4) {
    FragB f[2][2];      // [16 tokens][8 columns]
#pragma unroll
    for (int kt = 0; kt < 2; ++kt)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int s = 16 * kt + 8 * e + 2 * tq, col = 16 * ct + 8 * j + gr;
          float x, y;
          if (is_u && !v_here) {
            x = s < cn ? vb[(size_t)s * g.ldv + col] : 0.f;
            y = s + 1 < cn ? vb[(size_t)(s + 1) * g.ldv + col] : 0.f;
          } else {
            const float* p = is_u ? vs + s * VP + col : ks + s * DP + col;
            x = p[0];
            y = p[is_u ? VP : DP];
          }
          put_b(f[kt][j], e, x, y);
        }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) {
      float acc[2][4] = {}, h0[2][4] = {}, h1[2][4] = {};
      mma_low<2>(acc, a[mt][0], f[0]);
      if (mt) mma_low<2>(acc, a[mt][1], f[1]);      // T is zero above its diagonal
      mma_high<2>(h0, a[mt][0], f[0]);
      if (mt) mma_high<2>(h1, a[mt][1], f[1]);
      mma_rest<2>(acc, h0, a[mt][0], f[0]);
      if (mt) mma_rest<2>(acc, h1, a[mt][1], f[1]);
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[j][e] = h0[j][e] + (h1[j][e] + acc[j][e]);
      if (is_u) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          float* at = oU + (16 * mt + gr) * DV + 16 * ct + 8 * j + 2 * tq;
          *(float2*)at = make_float2(acc[j][0], acc[j][1]);
          *(float2*)(at + 8 * DV) = make_float2(acc[j][2], acc[j][3]);
        }
      } else {
        // a result's neighbours in a row are neighbours in the walk's operand
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          FragB w;
          put_b(w, 0, acc[0][2 * r], acc[0][2 * r + 1]);
          put_b(w, 1, acc[1][2 * r], acc[1][2 * r + 1]);
          store_frag(oW + (4 * ct + 2 * mt + r) * SC_FRAG, lane, w);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------- the walk
constexpr int SC_PART = 20;       // pitch of a token's 16 columns in shared memory

// CTA (sequence, head, 16 columns; mlstm: one more for the normalizer's column), a warp for every 16
// rows of the state (and at least four). The state is held transposed in the accumulators' layout:
// columns gr and gr + 8, rows 16 warp + 8 j + 2 tq + (0, 1).
template <bool DELTA>
__global__ void __launch_bounds__(256, DELTA ? 1 : 2)
state_chunk_walk_kernel(const WalkArgs g, const float* __restrict__ scratch, int chunk0, int per_seq) {
  mb_grid_wait();
  mb_grid_launch_next();
  extern __shared__ __align__(16) float sm[];
  const int D = g.D, DV = g.DV, H = g.H, warps = D / 16;
  const int b = blockIdx.x, hd = blockIdx.y;
  const bool norm_col = !DELTA && (int)blockIdx.z == DV / SC_COLS;
  const int c0 = norm_col ? 0 : blockIdx.z * SC_COLS;
  const int t0 = g.seq_start[b], n = g.seq_start[b + 1] - t0;
  const int chunks = min(per_seq, (n + SC_C - 1) / SC_C - chunk0);
  if (chunks <= 0) return;
  constexpr int ROWS = DELTA ? 2 * SC_C : SC_C;      // rows that meet S0: W's, then q's
  constexpr int NT = ROWS / 8;
  float* part = sm;                                  // [warps][ROWS][SC_PART]
  float* so = part + warps * ROWS * SC_PART;         // [32][SC_PART] q's part of the outputs
  uint32_t* up = (uint32_t*)(so + SC_C * SC_PART);   // U cut: [3][16 columns][20 words of 2 tokens]
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gr = lane >> 2, tq = lane & 3;
  const bool own = warp < warps;                     // has rows of the state
  const size_t per = sc_chunk_floats(DELTA, D, DV), step = (size_t)H * per;
  const float* base = scratch + ((size_t)b * per_seq * H + hd) * per;
  float* slot = g.state + (size_t)g.seq_slot[b] * g.state_stride + g.state_off;
  float* Sg = slot + (size_t)hd * g.head_stride + (norm_col ? (size_t)D * DV : (size_t)c0);
  const int s_row = norm_col ? 1 : DV;
  float* den = g.raw + (size_t)g.T * H * DV;

  // this lane's operands of the chunk that comes next
  FragB fr[NT], fk[4], fn[2];
  float4 u1;
  float2 head;
  const int my_row = threadIdx.x >> 2, my_col = 4 * (threadIdx.x & 3);      // a thread's place in a sum
  // (without conditions, warps that have no part read another's: a load behind a branch would be waited
  // for where the branch ends)
  const int rows_of = min(warp, warps - 1), u_row = my_row & (SC_C - 1);
  auto load_rows = [&](int ci) {
    const float* q = base + (size_t)ci * step + SC_META + 8 * SC_FRAG + 4 * SC_FRAG * rows_of;
#pragma unroll
    for (int i = 0; i < NT; ++i)
      load_frag(fr[i], DELTA && i < 4 ? q + (size_t)8 * SC_FRAG * warps + i * SC_FRAG : q + (i % 4) * SC_FRAG, lane);
  };
  auto load_u = [&](int ci) {
    const float* at = base + (size_t)ci * step;
    asm volatile("ld.global.nc.v2.f32 {%0, %1}, [%2];" : "=f"(head.x), "=f"(head.y) : "l"(at));
    const int t = min((chunk0 + ci) * SC_C + u_row, n - 1);
    u1 = load_once4(DELTA ? at + SC_META + 8 * SC_FRAG + (size_t)12 * SC_FRAG * warps + u_row * DV + c0 + my_col
                          : g.v + ((size_t)t0 + t) * g.ldv + (size_t)hd * DV + c0 + my_col);
  };
  auto load_keys = [&](int ci) {
    const float* at = base + (size_t)ci * step + SC_META;
#pragma unroll
    for (int i = 0; i < 4; ++i)
      load_frag(fk[i], at + 8 * SC_FRAG + (size_t)4 * SC_FRAG * (warps + rows_of) + i * SC_FRAG, lane);
#pragma unroll
    for (int i = 0; i < 2; ++i) load_frag(fn[i], at + (2 * (warp & 3) + i) * SC_FRAG, lane);
  };
  load_rows(0);
  load_u(0);
  load_keys(0);
  float S[2][4];      // [j][column gr or gr + 8][row, the next]
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int col = gr + 8 * (e >> 1), i = 16 * warp + 8 * j + 2 * tq + (e & 1);
      S[j][e] = !own || (norm_col && col) ? 0.f : Sg[(size_t)i * s_row + col];
    }
  for (int ci = 0; ci < chunks; ++ci) {
    const int next = min(ci + 1, chunks - 1);
    const int first = (chunk0 + ci) * SC_C, cn = min(SC_C, n - first);
    const float decay = head.x;
    bool odd = head.y != 0.f;
    if (own) {
      // S0^T [16 x 16 of this warp's rows] times the rows of W and q
      FragA a;
      odd |= cut_is_inexact(put_a(a, 0, S[0][0], S[0][1]) | put_a(a, 1, S[0][2], S[0][3]) |
                            put_a(a, 2, S[1][0], S[1][1]) | put_a(a, 3, S[1][2], S[1][3]));
      float acc[NT][4] = {};
      mma_low<NT>(acc, a, fr);
      mma_high<NT>(acc, a, fr);
      float* p = part + warp * ROWS * SC_PART + 2 * tq * SC_PART + gr;
#pragma unroll
      for (int i = 0; i < NT; ++i) {
        float* o = p + 8 * i * SC_PART;
        o[0] = acc[i][0];
        o[SC_PART] = acc[i][1];
        o[8] = acc[i][2];
        o[SC_PART + 8] = acc[i][3];
      }
    }
    load_rows(next);
    __syncthreads();
    // four columns of a row a thread: the warps' sums in their order
    for (int r = my_row; r < ROWS; r += blockDim.x >> 2) {
      float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
      for (int k = 0; k < warps; ++k) {
        const float4 x = *(const float4*)(part + (k * ROWS + r) * SC_PART + my_col);
        v.x += x.x; v.y += x.y; v.z += x.z; v.w += x.w;
      }
      const int t = r & (SC_C - 1);
      if (!DELTA || r >= SC_C) {
        *(float4*)(so + t * SC_PART + my_col) = v;
        odd |= no_number(v);
      }
      if (!DELTA || r < SC_C) {
        float4 u = u1;
        if (!DELTA && (norm_col || t >= cn)) u = make_float4(my_col == 0 && t < cn ? 1.f : 0.f, 0.f, 0.f, 0.f);
        if (DELTA) u = make_float4(u.x - v.x, u.y - v.y, u.z - v.z, u.w - v.w);
        const Cut2 a = cut_near(u.x, u.y), z = cut_near(u.z, u.w);
        odd |= cut_is_inexact(a.rest | z.rest);
        unsigned short* h = (unsigned short*)up + my_col * 40 + t;
        const uint32_t words[6] = {a.hi, z.hi, a.mid, z.mid, a.lo, z.lo};
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          unsigned short* at = h + (q >> 1) * 16 * 40 + (q & 1) * 80;
          at[0] = (unsigned short)words[q];
          at[40] = (unsigned short)(words[q] >> 16);
        }
      }
    }
    load_u(next);
    if (__syncthreads_or(odd)) {
      // token by token, from what the tokens themselves are
      const float* meta = base + (size_t)ci * step;
      for (int t = 0; t < cn; ++t) {
        const size_t row = (size_t)t0 + first + t;
        const float dec = meta[SC_DEC + t], be = meta[SC_BETA + t], qf = meta[SC_FQ + t], kf = meta[SC_FK + t];
        float k[2][2], q[2][2], sums[5] = {0.f, 0.f, 0.f, 0.f, 0.f};      // S.k and S.q of two columns, q.k
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const int i = 16 * warp + 8 * j + 2 * tq + e;
            k[j][e] = own ? g.k[row * g.ldk + (size_t)(hd / g.group) * D + i] * kf : 0.f;
            q[j][e] = own ? g.q[row * g.ldq + (size_t)(hd / g.group) * D + i] * qf : 0.f;
            sums[4] = fmaf(q[j][e], k[j][e], sums[4]);
          }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            S[j][e] *= dec;
            if (DELTA) sums[e >> 1] = fmaf(S[j][e], k[j][e & 1], sums[e >> 1]);
            sums[2 + (e >> 1)] = fmaf(S[j][e], q[j][e & 1], sums[2 + (e >> 1)]);
          }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 5; ++c) {
          sums[c] += __shfl_xor_sync(0xffffffffu, sums[c], 1);
          sums[c] += __shfl_xor_sync(0xffffffffu, sums[c], 2);
          if (own && tq == 0) part[(warp * 8 + gr) * 5 + c] = sums[c];
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < 5; ++c) {
          sums[c] = 0.f;
          for (int r = 0; r < warps; ++r) sums[c] += part[(r * 8 + gr) * 5 + c];
        }
        float x[2], o[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int col = gr + 8 * c;
          const float v = norm_col ? (col == 0 ? 1.f : 0.f) : g.v[row * g.ldv + (size_t)hd * DV + c0 + col];
          x[c] = DELTA ? be * (v - sums[c]) : be * v;
          o[c] = fmaf(sums[4], x[c], sums[2 + c]);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) S[j][e] = fmaf(k[j][e & 1], x[e >> 1], S[j][e]);
        if (warp == 0 && tq == 0) {
          if (norm_col) {
            if (gr == 0) den[row * H + hd] = fmaxf(fabsf(o[0]), meta[SC_EM + t]) + 1e-6f;
          } else {
            float* r = g.raw + row * H * DV + (size_t)hd * DV + c0 + gr;
            r[0] = o[0];
            r[8] = o[1];
          }
        }
      }
      load_keys(next);
      __syncthreads();
      continue;
    }
    FragA ua[2];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const uint32_t* at = up + (gr + 8 * (e & 1)) * 20 + 8 * k + tq + 4 * (e >> 1);
        ua[k].hi[e] = at[0];
        ua[k].mid[e] = at[16 * 20];
        ua[k].lo[e] = at[2 * 16 * 20];
      }
    // U^T times k of this warp's rows, and times N of eight tokens: three accumulators
    float acc[3][4] = {}, h0[3][4] = {}, h1[3][4] = {};
    {
      const FragB f0[3] = {fk[0], fk[2], fn[0]}, f1[3] = {fk[1], fk[3], fn[1]};
      mma_low<3>(acc, ua[0], f0);
      mma_low<3>(acc, ua[1], f1);
      mma_high<3>(h0, ua[0], f0);
      mma_high<3>(h1, ua[1], f1);
      mma_rest<3>(acc, h0, ua[0], f0);
      mma_rest<3>(acc, h1, ua[1], f1);
#pragma unroll
      for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          // an overflow of the leading products stands for itself: what they cut off is no number then
          const float sum = h0[i][e] + (h1[i][e] + acc[i][e]);
          acc[i][e] = sum == sum ? sum : h0[i][e] + h1[i][e];
        }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) S[j][e] = fmaf(decay, S[j][e], acc[j][e]);
    if (warp < SC_C / 8) {
      float* raw = g.raw + ((size_t)t0 + first) * H * DV + (size_t)hd * DV + c0;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int t = 8 * warp + 2 * tq + (e & 1), col = gr + 8 * (e >> 1);
        const float o = so[t * SC_PART + col] + acc[2][e];
        if (t >= cn) continue;
        if (!norm_col) raw[(size_t)t * H * DV + col] = o;
        else if (col == 0)
          den[((size_t)t0 + first + t) * H + hd] = fmaxf(fabsf(o), base[(size_t)ci * step + SC_EM + t]) + 1e-6f;
      }
    }
    load_keys(next);
  }
#pragma unroll
  for (int j = 0; j < 2; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int col = gr + 8 * (e >> 1), i = 16 * warp + 8 * j + 2 * tq + (e & 1);
      if (own && (!norm_col || col == 0)) Sg[(size_t)i * s_row + col] = S[j][e];
    }
}
