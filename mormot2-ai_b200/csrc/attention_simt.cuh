// What the general attention's kernels share: their arguments, a score's way from the dot product to
// the softmax, an output's factor.
#pragma once
#include "common.cuh"

// From so many new tokens on a sequence goes in tiles: 16 fill a quarter of a tile of 64; with fewer
// the tile costs more than reading the keys once per token. Each sequence by itself: a tile with
// one token in it walks the token's keys in a row on one CTA a head (63 sequences of 2,000
// positions beside a prompt of 16: 2,700 us with tiles for all, 225 with both kernels).
#define ATT_MANY 16

// A score s (after the scale) goes through softcap and slopes as in attention_simt_kernel;
// `max_pages`, `ring_pages`, `keep_first`, `gate` likewise.
template <typename T> struct AttArgs {
  const T* q;
  T* out;
  const T* kpool;
  const T* vpool;
  const int* page_table;
  const int* tok_seq;
  const int* tok_pos;
  const int* seq_slot;
  const int* seq_start;
  const float* sink;
  const float* slopes;
  const T* gate;
  int q_stride, out_stride, max_pages, ring_pages, nh, nkv, hd, vd, window, gate_stride, gate_dim,
      keep_first;
  float scale, softcap;
};

template <typename T>
__device__ __forceinline__ float att_score(const AttArgs<T>& a, float dot, float slope, int dist) {
  float s = dot * a.scale;
  if (a.softcap > 0.f) s = a.softcap * tanhf(s / a.softcap);
  return s - slope * (float)dist;
}

// The factor of value i of head h in token t's output: a gate per head or per value, or none.
template <typename T>
__device__ __forceinline__ float att_gate(const AttArgs<T>& a, int t, int h, int i) {
  if (!a.gate) return 1.f;
  const size_t at = (size_t)t * a.gate_stride + (a.gate_dim > 0 ? (size_t)h * a.gate_dim + i : h);
  return sigmoid_f32(to_f32<T>(a.gate[at]));
}
