// Class kernels of 32-replica words on periodic boxes with a compile-time bond table (lattices.h), no mask: the
// packed chain and the two bitwise chains of bitwise.cu / sweep.cu, which keep every other system. Same draws,
// same tables, same decisions.
//
// The kernels are bound by instruction issue, not by memory (a word and site is 4 bytes for 32 attempts), so every
// step that the 32 replicas can share is taken once per word:
//   - neighbour offsets once per site, for all words of the thread;
//   - the neighbour counts of 32 replicas in a carry-save adder (words.cuh);
//   - bitwise: one flip mask per possible count, chosen for all lanes by a tree of bit selects on the count planes
//     (bitwise.cu forms every count's lane set and ORs it in);
//   - the sweep's Philox round keys once per block, acceptance entries of the block's words in shared memory.
//
// Measured on a B200 against the kernels of bitwise.cu and sweep.cu, one class launch:
//   bitwise shared, simple cubic 128^3, 512 replicas   240 -> 82 us (DRAM 214 MB, 2.6 TB/s; logic pipe the limit)
//   bitwise independent, triangular 510^2, 200 replicas, field, Barker   53 -> 28 us
//   packed, simple cubic 64^3, 128 replicas   418 -> 50 us; its 16.8 M Philox calls alone are 33 us
#include "words.cuh"

namespace sck {

struct WordParams {
  Common c;
  int colour, alpha;
  int u0, per_block;     // first unit (bitwise shared: group of four words; packed: part of a word) and units per block
};

constexpr int kWordUnits = 8;   // units a block handles at most (their acceptance entries fit 8 KB)

// Offsets of own site and neighbours of class site t, false when the thread owns none.
template <class Lat>
__device__ __forceinline__ bool word_site(const WordParams& p, uint32_t t, uint32_t& own,
                                          uint32_t (&off)[Lat::max_bonds]) {
  const Common& c = p.c;
  const uint32_t per = (uint32_t)c.rows * (uint32_t)c.bx;
  int x, y, z;
  if (t >= per || !class_site(c, p.colour, p.alpha, t, x, y, z)) return false;
  own = (uint32_t)(p.alpha * c.g.plane + (z * c.g.L2 + y) * c.g.L1 + x);
  static_for<0, Lat::b>([&](auto ac) {
    constexpr int a = decltype(ac)::value;
    if (a == p.alpha) word_neighbours<Lat, a>(c.g, x, y, z, off);
  });
  return true;
}

// Lanes whose count (at most Z) is H or more.
template <int Z, int H>
__device__ __forceinline__ uint32_t lanes_from(const uint32_t* cp) {
  uint32_t m[Z + 1];
#pragma unroll
  for (int k = 0; k <= Z; ++k) m[k] = k >= H ? 0xFFFFFFFFu : 0u;
  return bit_select<Z + 1>(m, cp);
}

// ----------------------------------------------------------------------------------- bitwise, shared draws
// Grid (class sites / 256, group rows). Output q of one Philox call serves word 4 grp + q.
template <class Lat, bool FIELD>
__global__ void __launch_bounds__(256, 5) bitwise_shared_lattice_kernel(const __grid_constant__ WordParams p) {
  constexpr int Z = Lat::max_bonds, NP = bit_length(Z), ROW = (Z + 4) / 4 * 4, F = FIELD ? 2 : 1;
  constexpr int H = Z / 2;
  __shared__ float4 thr4[4 * kWordUnits][F][ROW / 4];
  __shared__ uint4 keys[5];
  __shared__ unsigned upper;     // bit w: word 4 u0 + w accepts every count from H on (energy not raised)
  const Common& c = p.c;
  const int units = (c.W + 3) / 4;
  const int u0 = p.u0 + (int)blockIdx.y * p.per_block;
  const int u1 = u0 + p.per_block < units ? u0 + p.per_block : units;
  float* thr = reinterpret_cast<float*>(thr4);
  follow_previous();
  if (threadIdx.x < 10) write_keys(keys, sweep_key_at(c.state, c.sweep_offset), threadIdx.x);
  if (threadIdx.x == 32) upper = FIELD ? 0u : 0xFFFFFFFFu;
  __syncthreads();
  for (int i = threadIdx.x; i < 4 * p.per_block * F * (Z + 1); i += blockDim.x) {
    const int k = i % (Z + 1), ws = i / (Z + 1), s = ws % F, w = ws / F;
    if (4 * u0 + w < c.W) {
      const float t = ((const float*)c.table)[(size_t)(4 * u0 + w) * c.NT + (s * c.Z1 + Z) * c.Z1 + k];
      thr[ws * ROW + k] = t;
      if (k >= H && !(t >= 1.0f)) atomicAnd(&upper, ~(1u << w));
    }
  }
  __syncthreads();
  uint32_t own, off[Z];
  if (!word_site<Lat>(p, blockIdx.x * blockDim.x + threadIdx.x, own, off)) return;
  const RoundKeys rk = shared_keys(keys);
  const uint32_t nsite = (uint32_t)c.g.nsite;
  const unsigned up = upper;
  for (int u = u0; u < u1; ++u) {
    const Philox4 r = philox_keys((uint32_t)u * nsite + own, rk);
    const uint32_t rx[4] = {r.x0, r.x1, r.x2, r.x3};
    uint32_t* plane = (uint32_t*)c.dst + (size_t)(4 * u) * nsite;
    const int left = c.W - 4 * u;
    auto word = [&](int q, uint32_t s0, const uint32_t (&x)[Z]) {
      uint32_t cp[NP], m[Z + 1];
      differ_counts<Z>(s0, x, cp);
      const float uq = to_uniform(rx[q]);
      const float* tb = thr + (4 * (u - u0) + q) * F * ROW;
      uint32_t acc;
      if (!FIELD && ((up >> (4 * (u - u0) + q)) & 1u)) {
        // u < 1 <= every entry from H on: only the counts below H compare
        uint32_t mh[H + 1];
#pragma unroll
        for (int k = 0; k < H; ++k) mh[k] = below_mask(uq, tb[k]);
        mh[H] = 0xFFFFFFFFu;
        acc = bit_select<H + 1>(mh, cp) | lanes_from<Z, H>(cp);
      } else {
#pragma unroll
        for (int k = 0; k <= Z; ++k) m[k] = below_mask(uq, tb[k]);
        acc = bit_select<Z + 1>(m, cp);
      }
      if constexpr (FIELD) {
#pragma unroll
        for (int k = 0; k <= Z; ++k) m[k] = below_mask(uq, tb[ROW + k]);
        acc = (s0 & bit_select<Z + 1>(m, cp)) | (~s0 & acc);
      }
      plane[(size_t)q * nsite + own] = s0 ^ acc;
    };
    // the words' loads first, two or four words at a time: their latency, not their number, is what they cost
    constexpr int BATCH = 2;
    if (left >= 4) {
#pragma unroll
      for (int q0 = 0; q0 < 4; q0 += BATCH) {
        uint32_t s0[BATCH], x[BATCH][Z];
#pragma unroll
        for (int q = 0; q < BATCH; ++q) {
          const uint32_t* pw = plane + (size_t)(q0 + q) * nsite;
          s0[q] = pw[own];
#pragma unroll
          for (int i = 0; i < Z; ++i) x[q][i] = pw[off[i]];
        }
#pragma unroll
        for (int q = 0; q < BATCH; ++q) word(q0 + q, s0[q], x[q]);
      }
    } else {
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (q < left) {
          const uint32_t* pw = plane + (size_t)q * nsite;
          uint32_t x[Z];
#pragma unroll
          for (int i = 0; i < Z; ++i) x[i] = pw[off[i]];
          word(q, pw[own], x);
        }
    }
  }
}

// ------------------------------------------------------------------------------ bitwise, independent draws
// Lane j accepts when its 32-bit integer U is below P[s, count]: compared from the most significant bit, four bits
// per Philox call (bitwise.cu). The bit planes of P over the counts are masks in shared memory, one row per
// (word, s, bit); a tree of selects turns a row into every lane's bit of its own P.
template <class Lat, bool FIELD>
__global__ void __launch_bounds__(256, 4) bitwise_independent_lattice_kernel(const __grid_constant__ WordParams p) {
  constexpr int Z = Lat::max_bonds, NP = bit_length(Z), ROW = (Z + 4) / 4 * 4, F = FIELD ? 2 : 1;
  constexpr int BITS = 34;        // rows 0..31: bit 31 - row of P; 32: P = 2^32 (accepts); 33: 0 < P < 2^32
  __shared__ uint4 mask4[F][BITS][ROW / 4];
  __shared__ uint4 keys[8][5];   // round keys of the eight bit groups
  const Common& c = p.c;
  uint32_t* mask = reinterpret_cast<uint32_t*>(mask4);
  follow_previous();
  if (threadIdx.x < 80) {
    const int grp = threadIdx.x / 10;
    const long long kg = (long long)sweep_key_at(c.state, c.sweep_offset) + (long long)(grp + 1) * 104729LL;
    write_keys(keys[grp], (int32_t)(kg % 2147483629LL), threadIdx.x % 10);
  }
  uint32_t own = 0, off[Z];
  const bool live = word_site<Lat>(p, blockIdx.x * blockDim.x + threadIdx.x, own, off);
  const uint32_t nsite = (uint32_t)c.g.nsite;
  const int w0 = p.u0 + (int)blockIdx.y * p.per_block;
  const int w1 = w0 + p.per_block < c.W ? w0 + p.per_block : c.W;
  for (int w = w0; w < w1; ++w) {
    __syncthreads();
    for (int i = threadIdx.x; i < F * BITS * (Z + 1); i += blockDim.x) {
      const int k = i % (Z + 1), sb = i / (Z + 1), b = sb % BITS, s = sb / BITS;
      const long long P = ((const long long*)c.table)[(size_t)w * c.NT + (s * c.Z1 + Z) * c.Z1 + k];
      const bool all = P >= (1LL << 32);
      const bool set = b < 32 ? (((unsigned long long)P >> (31 - b)) & 1ull) != 0 : (b == 32 ? all : (P > 0 && !all));
      mask[sb * ROW + k] = set ? 0xFFFFFFFFu : 0u;
    }
    __syncthreads();
    if (!live) continue;
    uint32_t* plane = (uint32_t*)c.dst + (size_t)w * nsite;
    const uint32_t s0 = plane[own];
    uint32_t x[Z], cp[NP];
#pragma unroll
    for (int i = 0; i < Z; ++i) x[i] = plane[off[i]];
    differ_counts<Z>(s0, x, cp);
    auto lanes = [&](int b) {
      uint32_t m[Z + 1];
#pragma unroll
      for (int k = 0; k <= Z; ++k) m[k] = mask[b * ROW + k];
      uint32_t v = bit_select<Z + 1>(m, cp);
      if constexpr (FIELD) {
#pragma unroll
        for (int k = 0; k <= Z; ++k) m[k] = mask[(BITS + b) * ROW + k];
        v = (s0 & bit_select<Z + 1>(m, cp)) | (~s0 & v);
      }
      return v;
    };
    uint32_t acc = lanes(32), und = lanes(33);
    const uint32_t ctr = (uint32_t)w * nsite + own;
#pragma unroll 1
    for (int grp = 0; grp < 8; ++grp) {
      if (und == 0u) break;
      const Philox4 r = philox_keys(ctr, shared_keys(keys[grp]));
      const uint32_t rw4[4] = {r.x0, r.x1, r.x2, r.x3};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const uint32_t pb = lanes(4 * grp + q), rw = rw4[q];
        acc |= und & ~rw & pb;
        und &= ~(rw ^ pb);
      }
    }
    plane[own] = s0 ^ acc;
  }
}

// ---------------------------------------------------------------------------------------------- packed
// One thread per (class site, part of a word): the neighbour counts of the word's 32 replicas in bit planes, then
// one Philox draw and one table entry per replica of its part. Each replica's entries of the sublattice, indexed by
// own spin and number of up neighbours, sit in shared memory (bank = entry: lanes of one warp read one row). Grid
// (class sites / 256, word parts); a part is a word, a half or a quarter (LANES = 32, 16, 8), stored as its own
// 4, 2 or 1 bytes.
template <class Lat, int LANES, bool BARKER>
__global__ void __launch_bounds__(256, 4) packed_lattice_kernel(const __grid_constant__ WordParams p) {
  constexpr int Z = Lat::max_bonds, NP = bit_length(Z), ROW = 2 << NP, PARTS = 32 / LANES;
  static_assert(NP == 3 || NP == 4, "the count planes pack into nibbles");
  __shared__ float tab[LANES * ROW];
  const Common& c = p.c;
  const int unit = p.u0 + (int)blockIdx.y, w = unit / PARTS, part = unit % PARTS;
  __shared__ uint4 keys[5];
  follow_previous();
  if (threadIdx.x < 10) write_keys(keys, sweep_key_at(c.state, c.sweep_offset), threadIdx.x);
  for (int i = threadIdx.x; i < LANES * 2 * (Z + 1); i += blockDim.x) {
    const int up = i % (Z + 1), s = i / (Z + 1) % 2, j = i / (2 * (Z + 1));
    const float e =
        ((const float*)c.table)[(size_t)(LANES * unit + j) * c.lut_rep_stride + p.alpha * c.keys + s + 4 * up];
    tab[j * ROW + (s << NP) + up] = BARKER ? __fadd_rn(1.0f, e) : e;
  }
  __syncthreads();
  uint32_t own, off[Z];
  if (!word_site<Lat>(p, blockIdx.x * blockDim.x + threadIdx.x, own, off)) return;
  const RoundKeys rk = shared_keys(keys);
  const uint32_t nsite = (uint32_t)c.g.nsite;
  uint32_t* plane = (uint32_t*)c.dst + (size_t)w * nsite;
  uint32_t sown;                 // own spins of the part, alone: other blocks write the word's other parts
  if constexpr (LANES == 32) sown = plane[own];
  else if constexpr (LANES == 16) sown = reinterpret_cast<const uint16_t*>(plane + own)[part];
  else sown = reinterpret_cast<const uint8_t*>(plane + own)[part];
  uint32_t x[Z], cp[4];
#pragma unroll
  for (int i = 0; i < Z; ++i) x[i] = plane[off[i]];
  bit_counts<Z>(x, cp);
  if constexpr (NP == 3) cp[3] = sown << (LANES * part);
  // nibble m of nib[q] = planes 0..3 of lane 4 m + q
  uint32_t nib[4];
  {
    const uint32_t m1 = 0x55555555u, m2 = 0x33333333u;
    const uint32_t a0 = (cp[0] & m1) | ((cp[1] << 1) & ~m1), a1 = ((cp[0] >> 1) & m1) | (cp[1] & ~m1);
    const uint32_t b0 = (cp[2] & m1) | ((cp[3] << 1) & ~m1), b1 = ((cp[2] >> 1) & m1) | (cp[3] & ~m1);
    nib[0] = (a0 & m2) | ((b0 << 2) & ~m2);
    nib[2] = ((a0 >> 2) & m2) | (b0 & ~m2);
    nib[1] = (a1 & m2) | ((b1 << 2) & ~m2);
    nib[3] = ((a1 >> 2) & m2) | (b1 & ~m2);
  }
  if constexpr (PARTS > 1) {
#pragma unroll
    for (int q = 0; q < 4; ++q) nib[q] >>= LANES * part;
  }
  uint32_t flip = 0u;            // the decisions, latest in the lowest bit
  uint32_t ctr = (uint32_t)(LANES * unit) * nsite + own;
  const float* row = tab;
#pragma unroll 1
  for (int m = 0; m < LANES / 4; ++m) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t idx = nib[q] & 15u;
      nib[q] >>= 4;
      if constexpr (NP == 4) idx |= ((sown >> (4 * m + q)) & 1u) << NP;
      const float e = row[q * ROW + idx];
      const float u = to_uniform(philox_keys(ctr, rk).x0);
      ctr += nsite;
      // accept: u < e, or u (1 + e) < 1 (below_mask's sign, shifted in)
      const float d = BARKER ? __fsub_rn(__fmul_rn(u, e), 1.0f) : __fsub_rn(u, e);
      flip = __funnelshift_l(__float_as_uint(d), flip, 1);
    }
    row += 4 * ROW;
  }
  const uint32_t out = sown ^ (__brev(flip) >> (32 - LANES));
  if constexpr (LANES == 32) plane[own] = out;
  else if constexpr (LANES == 16) reinterpret_cast<uint16_t*>(plane + own)[part] = (uint16_t)out;
  else reinterpret_cast<uint8_t*>(plane + own)[part] = (uint8_t)out;
}

// The compile-time table these kernels serve for a plan of word storage, or 0: one coupling group, every axis
// periodic, no mask.
int find_word_spec(const sck_plan* plan) {
  if (plan->mode != SCK_MODE_PACKED && plan->mode != SCK_MODE_BITWISE && plan->mode != SCK_MODE_BITWISE_INDEP) return 0;
  if (plan->geom.has_mask) return 0;
  const int id = match_lattice(plan);
  if (id == 0 || id == Lat_bcc_1_2::id || !lattice_periodic_box(plan, id)) return 0;
  return id;
}

// ------------------------------------------------------------------------------------ FP64 observables
// Per replica of a word: A = anti-aligned pairs, each bond visited once from its forward end, and U_a = up spins of
// sublattice a, in integers; then E = -J (P - 2 A) - h (2 U - S) and M_a = 2 U_a - S_a with P pairs and S sites.
// A thread walks a column of the box (along z, in two dimensions along y): the words s ^ s_j of a few sites go
// through the carry-save adder and into per-thread counters kept as bit planes, so that the 32 replicas cost
// about two operations per pair. Only at the end of a column does the warp transpose the planes into one integer
// per replica (warp_lane_counts), where the kernel for other systems (observables.cu) transposes every word of
// every bond. Grid (blocks per word, words); a block takes the word's (column block, chunk) items in turn.
// Bound by the logic pipe: 1083 -> 90 us for 128^3 x 512 replicas (1.5 TB/s of words), 40 -> 11 us for 64^3 x 128.
constexpr int kPairPlanes = 11, kUpPlanes = 8;     // per-thread counters: chunks of at most 128 sites, 12 pairs each

template <int N, int M>
__device__ __forceinline__ void planes_add(uint32_t (&cnt)[M], const uint32_t* v) {
  uint32_t carry = 0u;
#pragma unroll
  for (int i = 0; i < M; ++i) {
    const uint32_t a = cnt[i], b = i < N ? v[i] : 0u;
    cnt[i] = a ^ b ^ carry;
    carry = (a & b) | (carry & (a | b));
  }
}

template <class Lat, int A>
__host__ __device__ constexpr int forward_bonds() {
  int n = 0;
  for (int i = 0; i < Lat::n_bonds(A); ++i) n += forward_bond<Lat, A>(i) ? 1 : 0;
  return n;
}

// A bond to the next site of the same column.
template <class Lat, int A>
__host__ __device__ constexpr bool ahead_bond(int i) {
  const BondC b = Lat::bond(A, i);
  return b.a2 == A && b.dx == 0 && (Lat::dim == 3 ? (b.dy == 0 && b.dz == 1) : b.dy == 1);
}
template <class Lat, int A>
__host__ __device__ constexpr bool has_ahead() {
  for (int i = 0; i < Lat::n_bonds(A); ++i)
    if (ahead_bond<Lat, A>(i)) return true;
  return false;
}

template <class Lat>
__global__ void __launch_bounds__(256) observables_columns_kernel(const __grid_constant__ ObsParams p, int chunk) {
  constexpr int B = Lat::b;
  const Geometry& g = p.g;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t* words = (const uint32_t*)p.spins + (size_t)blockIdx.y * g.nsite;
  const int ncol = Lat::dim == 3 ? g.L1 * g.L2 : g.L1;       // columns, sites of a column, words between them
  const int len = Lat::dim == 3 ? g.L3 : g.L2;
  const int step = Lat::dim == 3 ? ncol : g.L1;
  const int colblocks = (ncol + 255) / 256, items = colblocks * ((len + chunk - 1) / chunk);
  unsigned pairs = 0u, up[B];                                // of replica `lane`
#pragma unroll
  for (int a = 0; a < B; ++a) up[a] = 0u;
  unsigned long long sites = 0;                              // sites of one sublattice this block visited
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    const int cb = it % colblocks, z0 = it / colblocks * chunk, z1 = min(len, z0 + chunk);
    const int col = cb * 256 + (int)threadIdx.x;
    const bool live = col < ncol;
    sites += (unsigned long long)min(256, ncol - cb * 256) * (unsigned)(z1 - z0);
    const int y = Lat::dim == 3 && live ? (int)fdiv((uint32_t)col, p.fd_L1) : 0;
    const int x = live ? col - y * g.L1 : 0;
    const Around<1, true> nb(g, x, y, 0);
    static_for<0, B>([&](auto ac) {
      constexpr int a = decltype(ac)::value;
      constexpr int F = forward_bonds<Lat, a>(), U = F <= 3 ? 8 : (F <= 8 ? 4 : 2);
      uint32_t cp[kPairPlanes], cu[kUpPlanes];
#pragma unroll
      for (int i = 0; i < kPairPlanes; ++i) cp[i] = 0u;
#pragma unroll
      for (int i = 0; i < kUpPlanes; ++i) cu[i] = 0u;
      // sites z .. z + N - 1 of the column; the own word of the next site serves as the forward neighbour along it
      const uint32_t* base = words + (Lat::dim == 3 ? 0 : nb.xo[1]);
      auto take = [&](int z, auto nc) {
        constexpr int N = decltype(nc)::value;
        uint32_t in[N * F > 0 ? N * F : 1], s[N + 1];
        const int xy = Lat::dim == 3 ? nb.yo[1] + nb.xo[1] : 0;
#pragma unroll
        for (int u = 0; u < N; ++u) s[u] = __ldg(base + a * g.plane + (z + u) * step + xy);
        const int zn = z + N < len ? z + N : 0;
        if constexpr (has_ahead<Lat, a>()) s[N] = __ldg(base + a * g.plane + zn * step + xy);
#pragma unroll
        for (int u = 0; u < N; ++u) {
          const int zz = z + u;
          const int zo[3] = {(zz > 0 ? zz - 1 : len - 1) * step, zz * step, (u + 1 < N ? zz + 1 : zn) * step};
          int f = 0;
          static_for<0, Lat::n_bonds(a)>([&](auto ic) {
            constexpr int i = decltype(ic)::value;
            if constexpr (forward_bond<Lat, a>(i)) {
              constexpr BondC bd = Lat::bond(a, i);
              uint32_t t;
              if constexpr (ahead_bond<Lat, a>(i)) {
                t = s[u + 1];
              } else {
                const int q = bd.a2 * g.plane + (Lat::dim == 3 ? zo[bd.dz + 1] + nb.yo[bd.dy + 1] + nb.xo[bd.dx + 1]
                                                               : zo[bd.dy + 1] + nb.xo[bd.dx + 1]);
                t = __ldg(words + q);
              }
              in[u * F + f] = s[u] ^ t;
              ++f;
            }
          });
        }
        uint32_t sv[N];
#pragma unroll
        for (int u = 0; u < N; ++u) sv[u] = s[u];
        uint32_t v[bit_length(N * F) + 1], vs[bit_length(N)];
        if constexpr (F > 0) {
          bit_counts<N * F>(in, v);
          planes_add<bit_length(N * F)>(cp, v);
        }
        bit_counts<N>(sv, vs);
        planes_add<bit_length(N)>(cu, vs);
      };
      if (live) {
        int z = z0;
        for (; z + U <= z1; z += U) take(z, std::integral_constant<int, U>{});
        for (; z < z1; ++z) take(z, std::integral_constant<int, 1>{});
      }
      if constexpr (F > 0) {
#pragma unroll
        for (int i = 0; i < kPairPlanes; ++i) pairs += warp_lane_counts(cp[i], lane) << i;
      }
#pragma unroll
      for (int i = 0; i < kUpPlanes; ++i) up[a] += warp_lane_counts(cu[i], lane) << i;
    });
  }
  __shared__ unsigned red[8][1 + B][32];
  red[warp][0][lane] = pairs;
#pragma unroll
  for (int a = 0; a < B; ++a) red[warp][1 + a][lane] = up[a];
  __syncthreads();
  if (threadIdx.x < 32) {
    unsigned long long n[1 + B];
#pragma unroll
    for (int i = 0; i <= B; ++i) {
      n[i] = 0;
      for (int wi = 0; wi < 8; ++wi) n[i] += red[wi][i][lane];
    }
    int zsum = 0;                                            // forward bonds of a cell
    static_for<0, B>([&](auto ac) { zsum += forward_bonds<Lat, decltype(ac)::value>(); });
    const int rep = 32 * (int)blockIdx.y + lane;
    if (rep < p.B) {
      double* out = p.partial + ((size_t)rep * p.blocks_per_rep + blockIdx.x) * OBS_VALUES;
      double m = 0.0;
#pragma unroll
      for (int a = 0; a < B; ++a) {
        const double ma = 2.0 * (double)n[1 + a] - (double)sites;
        out[1 + a] = ma;
        m += ma;
      }
      out[0] = -p.obs[0].J[0] * ((double)(zsum * sites) - 2.0 * (double)n[0]) - p.h64[0] * m;
    }
  }
}

// A word observables call takes the column kernel: the systems of find_word_spec with one coupling on every bond.
bool word_columns_ok(const sck_plan* plan) {
  if (find_word_spec(plan) == 0) return false;
  for (int a = 0; a < plan->geom.b; ++a)
    for (int i = 0; i < plan->obs[a].n_bonds; ++i)
      if (plan->obs[a].J[i] != plan->obs[0].J[0]) return false;
  return true;
}

// Sites of a column one item takes: whole columns when these give the GPU eight blocks per SM, shorter chunks (at
// least 8, so that the transposes stay a small part) when the box has few columns or words.
static int word_column_chunk(const sck_plan* plan, int batch) {
  const Geometry& g = plan->geom;
  const int ncol = g.dim == 3 ? g.L1 * g.L2 : g.L1, len = g.dim == 3 ? g.L3 : g.L2;
  const long long blocks = (long long)((ncol + 255) / 256) * ((batch + 31) / 32);
  const long long split = (148 * 8 + blocks - 1) / blocks;
  long long chunk = (len + split - 1) / split;
  chunk = chunk < 8 ? 8 : (chunk > 128 ? 128 : chunk);
  return (int)chunk;
}

int word_column_blocks(const sck_plan* plan, int batch) {
  const Geometry& g = plan->geom;
  const int ncol = g.dim == 3 ? g.L1 * g.L2 : g.L1, len = g.dim == 3 ? g.L3 : g.L2;
  const int chunk = word_column_chunk(plan, batch);
  const long long items = (long long)((ncol + 255) / 256) * ((len + chunk - 1) / chunk);
  const int words = (batch + 31) / 32;
  const long long want = (148 * 16 + words - 1) / words;     // more items than that share blocks
  return (int)(items < want ? items : want);
}

int launch_word_columns(const sck_plan* plan, const ObsParams& p, cudaStream_t s) {
  const dim3 grid((unsigned)p.blocks_per_rep, (unsigned)((p.B + 31) / 32));
  const int chunk = word_column_chunk(plan, p.B);
  switch (find_word_spec(plan)) {
    case Lat_square_1::id: observables_columns_kernel<Lat_square_1><<<grid, 256, 0, s>>>(p, chunk); break;
    case Lat_triangular_1::id: observables_columns_kernel<Lat_triangular_1><<<grid, 256, 0, s>>>(p, chunk); break;
    case Lat_sc_1::id: observables_columns_kernel<Lat_sc_1><<<grid, 256, 0, s>>>(p, chunk); break;
    case Lat_bcc_1::id: observables_columns_kernel<Lat_bcc_1><<<grid, 256, 0, s>>>(p, chunk); break;
    default: observables_columns_kernel<Lat_fcc_1><<<grid, 256, 0, s>>>(p, chunk); break;
  }
  return cuda_status(cudaGetLastError(), "word observables");
}

// --------------------------------------------------------------------------------------------- host side
// Word launches overlap the class before them at every size. What they save, about a microsecond, is a fifth of a short
// launch (packed fcc 18^3 x 37, 184 blocks: 4.9 us a class, 6.2 plain); where a grid crowds the SMs left over (one block
// per SM in one launch of 75 to 148 blocks, two in the next) they lose more than that (packed fcc 10^3 x 256, 128
// blocks: 6.0 us, 4.0 plain).
template <class Lat, bool BARKER>
static void launch_packed(const WordParams& p, int parts, dim3 grid, cudaStream_t s) {
  if (parts == 1) launch_dependent(packed_lattice_kernel<Lat, 32, BARKER>, grid, 256, s, p);
  else if (parts == 2) launch_dependent(packed_lattice_kernel<Lat, 16, BARKER>, grid, 256, s, p);
  else launch_dependent(packed_lattice_kernel<Lat, 8, BARKER>, grid, 256, s, p);
}

template <class Lat>
static void launch_word_t(const sck_plan* plan, const WordParams& p, int parts, dim3 grid, cudaStream_t s) {
  if (plan->mode == SCK_MODE_PACKED) {
    if (plan->geom.acceptance == SCK_BARKER) launch_packed<Lat, true>(p, parts, grid, s);
    else launch_packed<Lat, false>(p, parts, grid, s);
  } else if (plan->mode == SCK_MODE_BITWISE) {
    if (p.c.field) launch_dependent(bitwise_shared_lattice_kernel<Lat, true>, grid, 256, s, p);
    else launch_dependent(bitwise_shared_lattice_kernel<Lat, false>, grid, 256, s, p);
  } else {
    if (p.c.field) launch_dependent(bitwise_independent_lattice_kernel<Lat, true>, grid, 256, s, p);
    else launch_dependent(bitwise_independent_lattice_kernel<Lat, false>, grid, 256, s, p);
  }
}

// One class of every word, in place. A block of the bitwise kernels handles several units (groups of four words, or
// words) when the class sites alone fill the GPU (eight blocks per SM): its threads then form offsets and its round
// keys once. A block of the packed kernel takes one word, or a half or a quarter of one where whole words would
// leave SMs idle (fewer than four blocks per SM); halves cost more work per attempt (59 against 50 us a class at
// 64^3, 128 replicas).
int launch_word_class(const sck_plan* plan, const Common& c, int colour, int alpha, cudaStream_t s) {
  WordParams p;
  p.c = c;
  p.colour = colour;
  p.alpha = alpha;
  const uint32_t per = (uint32_t)c.rows * (uint32_t)c.bx;
  const int bx = (int)((per + 255) / 256);
  int units = plan->mode == SCK_MODE_BITWISE ? (c.W + 3) / 4 : c.W;
  p.per_block = 1;
  int parts = 1;
  if (plan->mode == SCK_MODE_PACKED) {
    while (parts < 4 && (long long)bx * units * parts < 148 * 4) parts *= 2;
    units *= parts;
  } else {
    const int rows = (148 * 8 + bx - 1) / bx;                // grid rows that fill the GPU
    p.per_block = rows > units ? 1 : (units + rows - 1) / rows;
    if (p.per_block > kWordUnits) p.per_block = kWordUnits;
  }
  const int most = 65535;
  for (p.u0 = 0; p.u0 < units; p.u0 += most * p.per_block) {
    const int left = (units - p.u0 + p.per_block - 1) / p.per_block;
    const dim3 grid((unsigned)bx, (unsigned)(left < most ? left : most));
    switch (plan->word_spec) {
      case Lat_square_1::id: launch_word_t<Lat_square_1>(plan, p, parts, grid, s); break;
      case Lat_triangular_1::id: launch_word_t<Lat_triangular_1>(plan, p, parts, grid, s); break;
      case Lat_sc_1::id: launch_word_t<Lat_sc_1>(plan, p, parts, grid, s); break;
      case Lat_bcc_1::id: launch_word_t<Lat_bcc_1>(plan, p, parts, grid, s); break;
      default: launch_word_t<Lat_fcc_1>(plan, p, parts, grid, s); break;
    }
    const int rc = cuda_status(cudaGetLastError(), "word class launch");
    if (rc != SCK_OK) return rc;
  }
  return SCK_OK;
}

}  // namespace sck
