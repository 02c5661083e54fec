// Bit-sliced helpers of the word kernels (words.cu, observables.cu): 32 replicas per int32 word, one replica per
// bit position. Counts of several words are formed for all 32 replicas at once in carry-save adders.
#pragma once

#include "spec_site.cuh"

namespace sck {

constexpr int bit_length(int v) { return v <= 0 ? 0 : 1 + bit_length(v >> 1); }

// planes[p] bit j = bit p of the number of in[i] that have bit j set, i < N. Full adders take the inputs of one
// weight two at a time with the running sum and pass their carries to the next weight: 2 logic operations per
// input and weight step (8 for 6 inputs, against 15 for a ripple adder fed one input at a time).
template <int N>
__device__ __forceinline__ void bit_counts(const uint32_t (&in)[N], uint32_t* planes) {
  if constexpr (N == 1) {
    planes[0] = in[0];
  } else {
    uint32_t carry[N / 2];
    uint32_t s = in[0];
#pragma unroll
    for (int i = 0; i < (N - 1) / 2; ++i) {
      const uint32_t a = in[1 + 2 * i], b = in[2 + 2 * i];
      carry[i] = (s & a) | (s & b) | (a & b);
      s = s ^ a ^ b;
    }
    if constexpr (N % 2 == 0) {
      carry[N / 2 - 1] = s & in[N - 1];
      s = s ^ in[N - 1];
    }
    planes[0] = s;
    bit_counts<N / 2>(carry, planes + 1);
  }
}

// Counts of the in[i] that differ from s: the first adders take the raw words three at a time, since the sum and
// the carry of three complemented words are the complements of theirs (two operations per three words saved).
template <int N>
__device__ __forceinline__ void differ_counts(uint32_t s, const uint32_t (&in)[N], uint32_t* planes) {
  constexpr int T = N / 3, R = N % 3;
  uint32_t sum[T + R], carry[T + (T + R) / 2];
#pragma unroll
  for (int i = 0; i < T; ++i) {
    const uint32_t a = in[3 * i], b = in[3 * i + 1], c = in[3 * i + 2];
    sum[i] = s ^ (a ^ b ^ c);
    carry[i] = s ^ ((a & b) | (a & c) | (b & c));
  }
#pragma unroll
  for (int i = 0; i < R; ++i) sum[T + i] = s ^ in[3 * T + i];
  // the sums add up to plane 0; their carries join the first ones one weight up
  uint32_t v = sum[0];
  constexpr int S = T + R;
#pragma unroll
  for (int i = 0; i < (S - 1) / 2; ++i) {
    const uint32_t a = sum[1 + 2 * i], b = sum[2 + 2 * i];
    carry[T + i] = (v & a) | (v & b) | (a & b);
    v = v ^ a ^ b;
  }
  if constexpr (S % 2 == 0) {
    carry[T + S / 2 - 1] = v & sum[S - 1];
    v = v ^ sum[S - 1];
  }
  planes[0] = v;
  bit_counts<T + S / 2>(carry, planes + 1);
}

// The lanes' entry m[count], count given by its bit planes: a tree of bit selects, one logic operation each.
// Entries past M (counts that cannot occur) are never selected.
template <int M>
__device__ __forceinline__ uint32_t bit_select(const uint32_t (&m)[M], const uint32_t* planes) {
  if constexpr (M == 1) {
    return m[0];
  } else {
    uint32_t t[(M + 1) / 2];
#pragma unroll
    for (int i = 0; i < M / 2; ++i) t[i] = (planes[0] & m[2 * i + 1]) | (~planes[0] & m[2 * i]);
    if constexpr (M % 2 == 1) t[M / 2] = m[M - 1];
    return bit_select<(M + 1) / 2>(t, planes + 1);
  }
}

// 4-byte word offsets, within one word plane, of the neighbours of site (x, y, z) of sublattice A (periodic box).
template <class Lat, int A>
__device__ __forceinline__ void word_neighbours(const Geometry& g, int x, int y, int z,
                                                uint32_t (&off)[Lat::max_bonds]) {
  const Around<Lat::reach, true> nb(g, x, y, z);
  static_for<0, Lat::n_bonds(A)>([&](auto ic) {
    constexpr int i = decltype(ic)::value;
    constexpr BondC bd = Lat::bond(A, i);
    off[i] = (uint32_t)nb.index(g, bd);
  });
}

// Number of threads of the warp whose mask has bit `lane` set, for every lane at once: the warp's 32 masks as a
// 32 x 32 bit matrix (row = thread, column = bit) transposed by exchanging off-diagonal blocks of 16, 8, 4, 2 and
// 1 across lane ^ s, then the popcount of the lane's column.
__device__ __forceinline__ unsigned warp_lane_counts(uint32_t x, int lane) {
  const uint32_t lo[5] = {0x0000FFFFu, 0x00FF00FFu, 0x0F0F0F0Fu, 0x33333333u, 0x55555555u};
#pragma unroll
  for (int i = 0, sh = 16; i < 5; ++i, sh >>= 1) {
    const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x, sh);
    x = (lane & sh) ? ((x & ~lo[i]) | ((y & ~lo[i]) >> sh)) : ((x & lo[i]) | ((y & lo[i]) << sh));
  }
  return (unsigned)__popc(x);
}

// Philox4x32-10 of counter (c0, 0, 0, 0) with the ten round keys spelled out, for kernels whose threads draw many
// times under one key. A call for one output is 18 wide multiplies and 18 logic operations; the multiplies set its
// pace (a warp's takes four cycles of its scheduler's multiply pipe: 70 cycles a call measured alone, hence at most
// about 510 draws a nanosecond on 148 SMs at 1.9 GHz).
struct RoundKeys {
  uint32_t a[10], b[10];
};

// The same through shared memory, formed once per block: threads 0 .. 9 write round i's pair to k[2 i], k[2 i + 1].
__device__ __forceinline__ void write_keys(uint4* keys, int32_t key, int i) {
  uint32_t* k = reinterpret_cast<uint32_t*>(keys) + 2 * i;
  k[0] = key_lo(key) + (uint32_t)i * 0x9E3779B9u;
  k[1] = key_hi(key) + (uint32_t)i * 0xBB67AE85u;
}

__device__ __forceinline__ RoundKeys shared_keys(const uint4* k) {
  RoundKeys r;
#pragma unroll
  for (int i = 0; i < 5; ++i) {
    const uint4 v = k[i];
    r.a[2 * i] = v.x;
    r.b[2 * i] = v.y;
    r.a[2 * i + 1] = v.z;
    r.b[2 * i + 1] = v.w;
  }
  return r;
}

__device__ __forceinline__ Philox4 philox_keys(uint32_t c0, const RoundKeys& k) {
  uint32_t c1 = 0u, c2 = 0u, c3 = 0u;
#pragma unroll
  for (int i = 0; i < 10; ++i) {
    const unsigned long long pa = (unsigned long long)0xD2511F53u * c0;
    const unsigned long long pb = (unsigned long long)0xCD9E8D57u * c2;
    c0 = (uint32_t)(pb >> 32) ^ c1 ^ k.a[i];
    c2 = (uint32_t)(pa >> 32) ^ c3 ^ k.b[i];
    c1 = (uint32_t)pb;
    c3 = (uint32_t)pa;
  }
  return Philox4{c0, c1, c2, c3};
}

// All ones where u < t, for u finite and t a number (or NaN: zero): the sign of the rounded difference, which the
// FMA pipe forms (a compare and a select are two operations of the busier logic pipe).
__device__ __forceinline__ uint32_t below_mask(float u, float t) {
  return (uint32_t)(__float_as_int(__fsub_rn(u, t)) >> 31);
}

}  // namespace sck
