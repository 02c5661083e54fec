// Whole sweeps of small replicas on systems with a compile-time bond table (lattices.h): one block per replica keeps
// its spins in shared memory for all sweeps of a call, as the generic kernel of sweep.cu does, with constant
// neighbour offsets. Vector models may carry extra matrices (DMI) on their bonds, masks and open axes. Arithmetic,
// its order and the math functions are the generic kernel's (site.cuh), so the chain is the same bit for bit.
//
// One block per replica leaves a class step to one SM, so what counts is a step's instructions and the chain of
// dependent ones between two barriers. The generic kernel walks the bond list at run time, forms every neighbour's
// index with its axis checks and keeps extra neighbours in local memory; here offsets are constants, neighbours stay
// in registers, the sweeps' keys are formed 32 at a time and the Ising table row sits beside the spins.
#include <cooperative_groups.h>

#include <algorithm>

#include "site.cuh"
#include "words.cuh"

namespace sck {

struct LatticeResidentParams {
  Common c;
  float J[SCK_MAX_BASIS][SCK_MAX_GROUPS];
  int8_t extra[SCK_MAX_BASIS][16];        // extra-matrix slot of each bond, -1 none
  float E[SCK_MAX_BASIS][SCK_MAX_EXTRA][9];
  int Enz[SCK_MAX_BASIS][SCK_MAX_EXTRA];
  int has_extra;
  int single;                             // no row of an extra matrix has two non-zero entries: the next three hold
  uint8_t live[SCK_MAX_BASIS][16];        //   bit k: bond's row k has an entry
  int at[SCK_MAX_BASIS][16][3];           //   its column's offset among the listed spins (component x slots)
  float Erow[SCK_MAX_BASIS][16][3];       //   its value
  int n_classes;
  int classes[128][2];
  int n_sweeps;
  int table_floats;                       // Ising: entries of a replica's table row kept in shared memory, 0 none
  int spin_bytes;                         // bytes of the replica in shared memory (multiple of 16)
};

constexpr int kResidentKeys = 32;

// v += E t of every bond with an extra matrix, in bond order; only the matrix's non-zero entries enter, as in vec_site
// (-0 + a is a and a + -0 is a, so -0 stands for an empty sum).
template <int Z, int N>
__device__ __forceinline__ void add_extras(const LatticeResidentParams& p, int A, const float (&t)[Z][N],
                                           float (&v)[N]) {
#pragma unroll
  for (int i = 0; i < Z; ++i) {
    const int e = p.extra[A][i];
    if (e < 0) continue;
    const int nz = p.Enz[A][e];
#pragma unroll
    for (int k = 0; k < N; ++k) {
      float tot = -0.0f;
#pragma unroll
      for (int l = 0; l < N; ++l)
        if ((nz >> (3 * k + l)) & 1) tot = __fadd_rn(tot, __fmul_rn(p.E[A][e][3 * k + l], t[i][l]));
      v[k] = __fadd_rn(v[k], tot);
    }
  }
}

template <class Lat, int A, int N, bool PER>
__device__ __forceinline__ void resident_vec(const LatticeResidentParams& p, int rep, int x, int y, int z, int32_t key,
                                             float* S) {
  const Common& c = p.c;
  const Geometry& g = c.g;
  const int own = A * g.plane + (z * g.L2 + y) * g.L1 + x;
  if (g.has_mask && c.mask[own] == 0) return;
  const Around<Lat::reach, PER> nb(g, x, y, z);
  constexpr int Z = Lat::n_bonds(A);
  const int NS = g.nsite;
  float s[N], v[N], t[Z][N];
#pragma unroll
  for (int k = 0; k < N; ++k) {
    s[k] = S[k * NS + own];
    v[k] = 0.0f;
  }
  static_for<0, Lat::groups>([&](auto gc) {
    constexpr int gi = decltype(gc)::value;
    using R = GroupRange<Lat, A, gi>;
    float gs[N];
#pragma unroll
    for (int k = 0; k < N; ++k) gs[k] = 0.0f;
    static_for<R::begin, R::end>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      constexpr BondC bd = Lat::bond(A, i);
      const int q = nb.index(g, bd);
      const bool ok = nb.valid(bd);
#pragma unroll
      for (int k = 0; k < N; ++k) {
        t[i][k] = ok ? S[k * NS + q] : 0.0f;
        gs[k] = __fadd_rn(gs[k], t[i][k]);
      }
    });
#pragma unroll
    for (int k = 0; k < N; ++k) v[k] = __fadd_rn(v[k], __fmul_rn(p.J[A][gi], gs[k]));
  });
  if (p.has_extra) add_extras<Z, N>(p, A, t, v);
  vec_finish<N>(c, own, rep, key, s, v, S, S);
}

template <class Lat, int A, typename ST, bool PER>
__device__ __forceinline__ void resident_ising(const LatticeResidentParams& p, int rep, int x, int y, int z,
                                               int32_t key, const float* tab, ST* S) {
  const Common& c = p.c;
  const Geometry& g = c.g;
  const int own = A * g.plane + (z * g.L2 + y) * g.L1 + x;
  if (g.has_mask && c.mask[own] == 0) return;
  const Around<Lat::reach, PER> nb(g, x, y, z);
  const int s = sgn(S[own]);
  int k = s > 0 ? 1 : 0, stride = 2;
  static_for<0, Lat::groups>([&](auto gc) {
    using R = GroupRange<Lat, A, decltype(gc)::value>;
    int G = 0;
    static_for<R::begin, R::end>([&](auto ic) {
      constexpr BondC bd = Lat::bond(A, decltype(ic)::value);
      G += nb.valid(bd) ? sgn(S[nb.index(g, bd)]) : 0;
    });
    k += (G + (R::end - R::begin)) * stride;
    stride *= 2 * (R::end - R::begin) + 1;
  });
  const float e = tab[A * c.keys + k];
  const Philox4 r = philox4x32_10(counter32(rep, g.nsite, own), 0u, key_lo(key), key_hi(key));
  const float u = to_uniform(r.x0);
  const bool acc = g.acceptance == SCK_BARKER ? __fmul_rn(u, __fadd_rn(1.0f, e)) < 1.0f : u < e;
  if (acc) S[own] = (ST)(-s);
}

template <class Lat, int N, typename ST, bool PER>
__global__ void __launch_bounds__(1024) lattice_resident_kernel(const __grid_constant__ LatticeResidentParams p) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int32_t keys[kResidentKeys];
  const Common& c = p.c;
  ST* S = reinterpret_cast<ST*>(smem_raw);
  float* row = reinterpret_cast<float*>(smem_raw + p.spin_bytes);
  const int rep = blockIdx.x;
  const int n = N * c.g.nsite;
  ST* home = (ST*)c.dst + (size_t)rep * n;
  const float* tab = N == 1 ? (const float*)c.table + (size_t)rep * c.lut_rep_stride : nullptr;
  for (int i = threadIdx.x; i < n; i += blockDim.x) S[i] = home[i];
  if (N == 1 && p.table_floats) {
    for (int i = threadIdx.x; i < p.table_floats; i += blockDim.x) row[i] = tab[i];
    tab = row;
  }
  const uint32_t per = (uint32_t)c.rows * (uint32_t)c.bx;
  for (int sw = 0; sw < p.n_sweeps; ++sw) {
    if (sw % kResidentKeys == 0) {
      __syncthreads();                       // the sweep before has read its key
      if (threadIdx.x < kResidentKeys && sw + (int)threadIdx.x < p.n_sweeps)
        keys[threadIdx.x] = sweep_key_at(c.state, sw + (int)threadIdx.x);
      __syncthreads();
    }
    const int32_t key = keys[sw % kResidentKeys];
    for (int ci = 0; ci < p.n_classes; ++ci) {
      const int colour = p.classes[ci][0], alpha = p.classes[ci][1];
      for (uint32_t t = threadIdx.x; t < per; t += blockDim.x) {
        int x, y, z;
        if (!class_site(c, colour, alpha, t, x, y, z)) continue;
        static_for<0, Lat::b>([&](auto ac) {
          constexpr int A = decltype(ac)::value;
          if (A != alpha) return;
          if constexpr (N == 1) resident_ising<Lat, A, ST, PER>(p, rep, x, y, z, key, tab, S);
          else resident_vec<Lat, A, N, PER>(p, rep, x, y, z, key, S);
        });
      }
      __syncthreads();
    }
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) home[i] = S[i];
}

// ------------------------------------------------------------------------------------------ listed sweeps
// Calls of several sweeps first write, beside the spins, every site's neighbours as shared-memory slots, and then
// update from the list alone: no coordinates, no axis checks, no inactive sites. Slots follow the sweep (class by
// class, inactive sites last), so that a warp's own spins are consecutive and its neighbours nearly so (sites of one
// class are two apart in the box: every access a two-way bank conflict). A neighbour outside an open box is the
// slot after the last, which holds zeros.
//
// A cluster of CL blocks shares a replica when replicas are too few for the SMs and classes large: every block
// holds all spins and lists, takes every CL-th run of a class's slots and stores accepted spins in every block's
// copy; classes are separated by cluster barriers. Slots are assigned by ordered block scans, the same in every block.
template <class Lat>
constexpr int list_words() { return Lat::max_bonds + 1 <= 8 ? 1 : 2; }   // uint4 per site: own index, neighbour slots

__device__ __forceinline__ int list_entry(const uint32_t* w, int i) { return (int)((w[i >> 1] >> (16 * (i & 1))) & 0xFFFFu); }

// Rank of this thread's flag among the block's set flags, in thread order; total in `sum`. Every thread calls it.
__device__ __forceinline__ int block_rank(bool flag, int* warp_sums, int& sum) {
  const unsigned m = __ballot_sync(0xFFFFFFFFu, flag);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) warp_sums[warp] = __popc(m);
  __syncthreads();
  // every warp scans the block's sums for itself, one per lane
  const int own = lane < (int)(blockDim.x >> 5) ? warp_sums[lane] : 0;
  int incl = own;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int up = __shfl_up_sync(0xFFFFFFFFu, incl, o);
    if (lane >= o) incl += up;
  }
  const int before = __shfl_sync(0xFFFFFFFFu, incl - own, warp);
  sum = __shfl_sync(0xFFFFFFFFu, incl, 31);
  __syncthreads();
  return before + __popc(m & ((1u << lane) - 1u));
}

template <class Lat, int N, typename ST, bool PER, int CL>
__global__ void __launch_bounds__(1024) list_resident_kernel(const __grid_constant__ LatticeResidentParams p) {
  namespace cg = cooperative_groups;
  constexpr int Z = Lat::max_bonds, W = list_words<Lat>();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ int32_t keys[kResidentKeys];
  __shared__ int first[129], warp_sums[32];
  const Common& c = p.c;
  const Geometry& g = c.g;
  const int n = g.nsite, NS = n + 1;
  ST* S = reinterpret_cast<ST*>(smem_raw);                              // [N][NS], slot order
  uint16_t* slot_of = reinterpret_cast<uint16_t*>(smem_raw);            // set-up only, before the spins arrive
  uint32_t* list = reinterpret_cast<uint32_t*>(smem_raw + p.spin_bytes);
  float* row = reinterpret_cast<float*>(smem_raw + p.spin_bytes + (size_t)16 * W * n);
  const int rank = CL > 1 ? (int)cg::this_cluster().block_rank() : 0;
  const int rep = (int)blockIdx.x / CL;
  ST* home = (ST*)c.dst + (size_t)rep * N * n;
  const float* tab = N == 1 ? (const float*)c.table + (size_t)rep * c.lut_rep_stride : nullptr;
  if (N == 1 && p.table_floats) {
    for (int i = threadIdx.x; i < p.table_floats; i += blockDim.x) row[i] = tab[i];
    tab = row;
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) slot_of[i] = 0xFFFFu;
  __syncthreads();
  const uint32_t per = (uint32_t)c.rows * (uint32_t)c.bx;
  int base = 0;
  for (int ci = 0; ci < p.n_classes; ++ci) {
    if (threadIdx.x == 0) first[ci] = base;
    for (uint32_t t0 = 0; t0 < per; t0 += blockDim.x) {
      const uint32_t t = t0 + threadIdx.x;
      int x, y, z, own = 0, sum;
      bool on = t < per && class_site(c, p.classes[ci][0], p.classes[ci][1], t, x, y, z);
      if (on) {
        own = p.classes[ci][1] * g.plane + (z * g.L2 + y) * g.L1 + x;
        on = !g.has_mask || c.mask[own] != 0;
      }
      const int r = block_rank(on, warp_sums, sum);
      if (on) {
        slot_of[own] = (uint16_t)(base + r);
        list[(base + r) * 4 * W] = (uint32_t)own;
      }
      base += sum;
    }
  }
  if (threadIdx.x == 0) first[p.n_classes] = base;
  for (int i0 = 0; base < n && i0 < n; i0 += blockDim.x) {   // inactive sites
    __syncthreads();
    const int i = i0 + (int)threadIdx.x;
    int sum;
    const bool on = i < n && slot_of[i] == 0xFFFFu;
    const int r = block_rank(on, warp_sums, sum);
    if (on) {
      slot_of[i] = (uint16_t)(base + r);
      list[(base + r) * 4 * W] = (uint32_t)i;
    }
    base += sum;
  }
  __syncthreads();
  const int active = first[p.n_classes];
  for (int sl = threadIdx.x; sl < active; sl += blockDim.x) {
    const int own = (int)list[sl * 4 * W];
    int a = 0, in = own;
    while (in >= g.plane) {
      in -= g.plane;
      ++a;
    }
    const int rw = (int)fdiv((uint32_t)in, c.fd_L1), x = in - rw * g.L1;
    const int z = (int)fdiv((uint32_t)rw, c.fd_L2), y = rw - z * g.L2;
    const Around<Lat::reach, PER> nb(g, x, y, z);
    uint32_t w[4 * W];
#pragma unroll
    for (int i = 0; i < 4 * W; ++i) w[i] = 0u;
    w[0] = (uint32_t)own;
    static_for<0, Lat::b>([&](auto ac) {
      constexpr int A = decltype(ac)::value;
      if (A != a) return;
      static_for<0, Z>([&](auto ic) {
        constexpr int i = decltype(ic)::value;
        constexpr BondC bd = Lat::bond(A, i);
        const uint32_t q = nb.valid(bd) ? slot_of[nb.index(g, bd)] : (uint32_t)n;
        w[(i + 1) >> 1] |= q << (16 * ((i + 1) & 1));
      });
    });
#pragma unroll
    for (int i = 0; i < W; ++i)
      reinterpret_cast<uint4*>(list)[sl * W + i] = make_uint4(w[4 * i], w[4 * i + 1], w[4 * i + 2], w[4 * i + 3]);
  }
  __syncthreads();                                     // slot_of is done: the spins take its place
  for (int sl = threadIdx.x; sl < n; sl += blockDim.x) {
    const int own = list_entry(list + sl * 4 * W, 0);
#pragma unroll
    for (int k = 0; k < N; ++k) S[k * NS + sl] = home[k * n + own];
  }
  if (threadIdx.x < N) S[threadIdx.x * NS + n] = (ST)0;
  if constexpr (CL > 1) cg::this_cluster().sync();
  const uint4* list4 = reinterpret_cast<const uint4*>(list);
  for (int sw = 0; sw < p.n_sweeps; ++sw) {
    if (sw % kResidentKeys == 0) {
      __syncthreads();
      if (threadIdx.x < kResidentKeys && sw + (int)threadIdx.x < p.n_sweeps)
        keys[threadIdx.x] = sweep_key_at(c.state, sw + (int)threadIdx.x);
      __syncthreads();
    }
    const int32_t key = keys[sw % kResidentKeys];
    for (int ci = 0; ci < p.n_classes; ++ci) {
      const int alpha = p.classes[ci][1], end = first[ci + 1];
      // the sublattice as a constant: its couplings are then constant-bank operands (indexed, every one is a load
      // through the address unit; 57 of them an update held the nanodisk step at 155 us)
      static_for<0, Lat::b>([&](auto ac) {
      constexpr int A = decltype(ac)::value;
      if (A != alpha) return;
      for (int sl = first[ci] + rank * (int)blockDim.x + (int)threadIdx.x; sl < end; sl += CL * (int)blockDim.x) {
        uint32_t w[4 * W];
#pragma unroll
        for (int i = 0; i < W; ++i) {
          const uint4 v4 = list4[sl * W + i];
          w[4 * i] = v4.x;
          w[4 * i + 1] = v4.y;
          w[4 * i + 2] = v4.z;
          w[4 * i + 3] = v4.w;
        }
        const int own = list_entry(w, 0);
        if constexpr (N == 1) {
          const int s = sgn(S[sl]);
          int k = s > 0 ? 1 : 0, stride = 2;
          static_for<0, Lat::groups>([&](auto gc) {
            using R = GroupRange<Lat, A, decltype(gc)::value>;
            int G = 0;
#pragma unroll
            for (int i = R::begin; i < R::end; ++i) G += sgn(S[list_entry(w, i + 1)]);
            k += (G + (R::end - R::begin)) * stride;
            stride *= 2 * (R::end - R::begin) + 1;
          });
          const float e = tab[A * c.keys + k];
          const Philox4 r = philox4x32_10(counter32(rep, n, own), 0u, key_lo(key), key_hi(key));
          const float u = to_uniform(r.x0);
          const bool acc = g.acceptance == SCK_BARKER ? __fmul_rn(u, __fadd_rn(1.0f, e)) < 1.0f : u < e;
          if (acc) {
            S[sl] = (ST)(-s);
            if constexpr (CL > 1)
              for (int o = 1; o < CL; ++o) *cg::this_cluster().map_shared_rank(S + sl, (rank + o) % CL) = (ST)(-s);
          }
        } else {
          float s[N], v[N], t[Z][N], x[N];
#pragma unroll
          for (int k = 0; k < N; ++k) {
            s[k] = S[k * NS + sl];
            v[k] = 0.0f;
          }
          static_for<0, Lat::groups>([&](auto gc) {
            constexpr int gi = decltype(gc)::value;
            using R = GroupRange<Lat, A, gi>;
            float gs[N];
#pragma unroll
            for (int k = 0; k < N; ++k) gs[k] = 0.0f;
#pragma unroll
            for (int i = R::begin; i < R::end; ++i) {
              const ST* q = S + list_entry(w, i + 1);
#pragma unroll
              for (int k = 0; k < N; ++k) {
                t[i][k] = q[k * NS];
                gs[k] = __fadd_rn(gs[k], t[i][k]);
              }
            }
#pragma unroll
            for (int k = 0; k < N; ++k) v[k] = __fadd_rn(v[k], __fmul_rn(p.J[A][gi], gs[k]));
          });
          if (p.single) {
            // DMI and the like: one product a row, its neighbour component read again at a uniform offset (testing
            // all nine entries of every bond's matrix cost as much as half the update: 53 of 155 us a ladder step)
#pragma unroll
            for (int i = 0; i < Z; ++i) {
              if (!p.live[A][i]) continue;
              const ST* q = S + list_entry(w, i + 1);
#pragma unroll
              for (int k = 0; k < N; ++k)
                if ((p.live[A][i] >> k) & 1) v[k] = __fadd_rn(v[k], __fmul_rn(p.Erow[A][i][k], q[p.at[A][i][k]]));
            }
          } else if (p.has_extra) {
            add_extras<Z, N>(p, A, t, v);
          }
          if (vec_decide<N>(c, own, rep, key, s, v, x)) {
#pragma unroll
            for (int k = 0; k < N; ++k) {
              S[k * NS + sl] = x[k];
              if constexpr (CL > 1)
                for (int o = 1; o < CL; ++o) *cg::this_cluster().map_shared_rank(S + k * NS + sl, (rank + o) % CL) = x[k];
            }
          }
        }
      }
      });
      if constexpr (CL > 1) cg::this_cluster().sync();
      else __syncthreads();
    }
  }
  for (int sl = rank * (int)blockDim.x + (int)threadIdx.x; sl < active; sl += CL * (int)blockDim.x) {
    const int own = list_entry(list + sl * 4 * W, 0);
#pragma unroll
    for (int k = 0; k < N; ++k) home[k * n + own] = S[k * NS + sl];
  }
}

// --------------------------------------------------------------------------------------------- host side
// The compile-time table a resident sweep of this plan runs on, or 0: the table's bonds and coupling groups, extra
// matrices (vector models) one per bond in bond order, as the field adds them.
int find_resident_spec(const sck_plan* plan) {
  if (plan->mode != SCK_MODE_INT8 && plan->mode != SCK_MODE_F32) return 0;
  const sck_system_desc& d = plan->desc;
  for (int a = 0; a < d.b; ++a) {
    const sck_sublattice& s = d.sub[a];
    if (s.n_extra > 0 && d.n == 1) return 0;
    int next = 0;
    for (int i = 0; i < s.n_bonds; ++i)
      if (s.bonds[i].extra >= 0 && s.bonds[i].extra != next++) return 0;
    if (next != s.n_extra) return 0;
  }
  return match_lattice(plan, true);
}

// Sweeps of a call from which the lists pay for their set-up (about a sweep's time), and their size in shared memory.
// us constant offsets / lists: int8 square 64^2 x 148, 1 sweep 10.5 / 14.1, 2: 17.0 / 17.6, 3: 23.5 / 21.1, 4: 30.0 / 24.6,
// 8: 55.8 / 38.7; Heisenberg bcc 8^3 x 148, 3: 12.3 / 13.2, 4: 15.1 / 15.6, 5: 17.7 / 17.8, 8: 25.9 / 24.8; nanodisk
// 39 x 39 x 5 x 148, 1: 40.4 / 38.5, 4: 125 / 76. Lists take 16 or 32 bytes a site, which leaves fewer blocks to an
// SM; in large batches they pay all the same from three or four sweeps on: int8 square 110^2 x 1,024 (one block
// to an SM with lists), 3 sweeps 373 / 346, 4: 491 / 412; 64^2 x 1,024, 3: 135 / 119; Heisenberg fcc 8^3 x 1,024, 3: 126 / 131,
// 4: 164 / 160.
constexpr int kListSweeps = 4;
constexpr size_t kResidentSmem = 222 << 10;

// Entries of a replica's Ising table row kept in shared memory beside the spins, 0 none.
static int table_floats(const sck_plan* plan) {
  if (plan->geom.n != 1) return 0;
  const size_t spins = (resident_bytes(plan) + 15) / 16 * 16;
  const int floats = plan->geom.b * plan->keys;
  return floats <= 2048 && spins + 4 * (size_t)floats <= (220 << 10) ? floats : 0;
}

// Spins in slot order with the slot of missing neighbours; the same bytes hold two per site during set-up.
static size_t list_spin_bytes(const sck_plan* plan) {
  const int nsite = plan->geom.nsite;
  const size_t spins = (size_t)plan->geom.n * (nsite + 1) * (plan->mode == SCK_MODE_INT8 ? 1 : 4);
  return (std::max(spins, (size_t)2 * nsite) + 15) / 16 * 16;
}

static size_t list_bytes(const sck_plan* plan) {
  const int words = plan->resident_spec == Lat_square_1::id       ? list_words<Lat_square_1>()
                    : plan->resident_spec == Lat_triangular_1::id ? list_words<Lat_triangular_1>()
                    : plan->resident_spec == Lat_sc_1::id         ? list_words<Lat_sc_1>()
                    : plan->resident_spec == Lat_bcc_1::id        ? list_words<Lat_bcc_1>()
                    : plan->resident_spec == Lat_bcc_1_2::id      ? list_words<Lat_bcc_1_2>()
                                                                  : list_words<Lat_fcc_1>();
  return list_spin_bytes(plan) + (size_t)16 * words * plan->geom.nsite + sizeof(float) * table_floats(plan);
}

// Calls of kListSweeps sweeps and more run from neighbour lists: 16-bit slots, everything in shared memory, and no
// class named twice. Every entry of the class list takes slots of its own, so a sweep order that repeats a class
// (the C ABI accepts it) would need more slots than sites; it stays on lattice_resident_kernel, which walks the list.
bool resident_lists_ok(const sck_plan* plan) {
  if (plan->resident_spec == 0 || plan->geom.nsite >= 65535 || list_bytes(plan) > kResidentSmem) return false;
  const sck_system_desc& d = plan->desc;
  for (int i = 0; i < d.n_classes; ++i)
    for (int j = 0; j < i; ++j)
      if (d.classes[i][0] == d.classes[j][0] && d.classes[i][1] == d.classes[j][1]) return false;
  return true;
}

template <class K>
static int launch_resident_kernel(K kernel, const LatticeResidentParams& p, int cluster, int threads, size_t smem,
                                  cudaStream_t s) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_status(e, "resident kernel shared memory");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(p.c.B * cluster));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at;
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)cluster;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = cluster > 1 ? 1 : 0;
  return cuda_status(cudaLaunchKernelEx(&cfg, kernel, p), "resident launch");
}

static int block_threads(int sites) {
  const int rounds = (sites + 1023) / 1024;
  const int threads = ((sites + rounds - 1) / rounds + 31) / 32 * 32;
  return threads < 128 ? 128 : threads;
}

template <class Lat, int N, typename ST, bool PER>
static int launch_lattice_resident_t(const sck_plan* plan, LatticeResidentParams& p, cudaStream_t s) {
  const int per = p.c.rows * p.c.bx, B = p.c.B;
  if (p.n_sweeps >= kListSweeps && plan->resident_lists) {
    LatticeResidentParams q = p;
    q.spin_bytes = (int)list_spin_bytes(plan);
    const size_t smem = list_bytes(plan);
    // two blocks a replica when that still leaves a block to an SM and a class gives each block a round of threads. Ten
    // sweeps in us, one block / two: nanodisk 39 x 39 x 5 (3,808 sites a class) x 74 151 / 123, x 75 151 / 239; XY square 90^2
    // x 74 97 / 73, 64^2 (2,048) 54 / 46, 56^2 (1,568) 46 / 42, 40^2 (800) 29 / 35
    if (N > 1 && 2 * B <= 148 && per >= 2048)
      return launch_resident_kernel(list_resident_kernel<Lat, N, ST, PER, (N > 1 ? 2 : 1)>, q, 2,
                                    block_threads((per + 1) / 2), smem, s);
    return launch_resident_kernel(list_resident_kernel<Lat, N, ST, PER, 1>, q, 1, block_threads(per), smem, s);
  }
  return launch_resident_kernel(lattice_resident_kernel<Lat, N, ST, PER>, p, 1, block_threads(per),
                                (size_t)p.spin_bytes + sizeof(float) * p.table_floats, s);
}

template <class Lat, bool PER>
static int launch_lattice_resident_n(const sck_plan* plan, LatticeResidentParams& p, cudaStream_t s) {
  if (plan->mode == SCK_MODE_INT8) return launch_lattice_resident_t<Lat, 1, int8_t, PER>(plan, p, s);
  switch (plan->geom.n) {
    case 1: return launch_lattice_resident_t<Lat, 1, float, PER>(plan, p, s);
    case 2: return launch_lattice_resident_t<Lat, 2, float, PER>(plan, p, s);
    default: return launch_lattice_resident_t<Lat, 3, float, PER>(plan, p, s);
  }
}

template <class Lat>
static int launch_lattice_resident_per(const sck_plan* plan, LatticeResidentParams& p, cudaStream_t s) {
  return lattice_periodic_box(plan, Lat::id) ? launch_lattice_resident_n<Lat, true>(plan, p, s)
                                             : launch_lattice_resident_n<Lat, false>(plan, p, s);
}

int launch_lattice_resident(const sck_plan* plan, const Common& c, int n_sweeps, cudaStream_t s) {
  LatticeResidentParams p;
  memset(&p, 0, sizeof(p));
  p.c = c;
  for (int a = 0; a < plan->geom.b; ++a) {
    const SubDev& sub = plan->sub[a];
    for (int gi = 0; gi < SCK_MAX_GROUPS; ++gi) p.J[a][gi] = sub.J[gi];
    for (int i = 0; i < 16; ++i) p.extra[a][i] = i < sub.n_bonds ? sub.bonds[i].extra : (int8_t)-1;
    for (int e = 0; e < sub.n_extra; ++e) {
      for (int k = 0; k < 9; ++k) p.E[a][e][k] = sub.E[e][k];
      p.Enz[a][e] = sub.Enz[e];
    }
    if (sub.n_extra > 0) p.has_extra = 1;
  }
  p.single = p.has_extra;
  for (int a = 0; a < plan->geom.b; ++a)
    for (int i = 0; i < 16; ++i) {
      if (p.extra[a][i] < 0) continue;
      const int e = p.extra[a][i], nz = p.Enz[a][e];
      for (int k = 0; k < 3; ++k) {
        const int row = (nz >> (3 * k)) & 7;
        if (row == 0) continue;
        if (row != 1 && row != 2 && row != 4) p.single = 0;
        const int l = row == 1 ? 0 : (row == 2 ? 1 : 2);
        p.live[a][i] |= (uint8_t)(1 << k);
        p.at[a][i][k] = l * (plan->geom.nsite + 1);
        p.Erow[a][i][k] = p.E[a][e][3 * k + l];
      }
    }
  p.n_classes = plan->desc.n_classes;
  for (int i = 0; i < p.n_classes; ++i) {
    p.classes[i][0] = plan->desc.classes[i][0];
    p.classes[i][1] = plan->desc.classes[i][1];
  }
  p.n_sweeps = n_sweeps;
  p.spin_bytes = (int)((resident_bytes(plan) + 15) / 16 * 16);
  p.table_floats = table_floats(plan);
  switch (plan->resident_spec) {
    case Lat_square_1::id: return launch_lattice_resident_per<Lat_square_1>(plan, p, s);
    case Lat_triangular_1::id: return launch_lattice_resident_per<Lat_triangular_1>(plan, p, s);
    case Lat_sc_1::id: return launch_lattice_resident_per<Lat_sc_1>(plan, p, s);
    case Lat_bcc_1::id: return launch_lattice_resident_per<Lat_bcc_1>(plan, p, s);
    case Lat_bcc_1_2::id: return launch_lattice_resident_per<Lat_bcc_1_2>(plan, p, s);
    default: return launch_lattice_resident_per<Lat_fcc_1>(plan, p, s);
  }
}

}  // namespace sck
