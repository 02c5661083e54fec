// Whole sweeps of small replicas on systems with a compile-time bond table (lattices.h): one block per replica keeps
// its spins in shared memory for all sweeps of a call, as the generic kernel of sweep.cu does, with constant
// neighbour offsets. Vector models may carry extra matrices (DMI) on their bonds, masks and open axes. Arithmetic,
// its order and the math functions are the generic kernel's (site.cuh), so the chain is the same bit for bit.
//
// One block per replica leaves a class step to one SM, so what counts is a step's instructions and the chain of
// dependent ones between two barriers. The generic kernel walks the bond list at run time, forms every neighbour's
// index with its axis checks and keeps extra neighbours in local memory; here offsets are constants, neighbours stay
// in registers, the sweeps' keys are formed 32 at a time and the Ising table row sits beside the spins.
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
  int n_classes;
  int classes[128][2];
  int n_sweeps;
  int table_floats;                       // Ising: entries of a replica's table row kept in shared memory, 0 none
  int spin_bytes;                         // bytes of the replica in shared memory (multiple of 16)
};

constexpr int kResidentKeys = 32;

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
  if (p.has_extra) {
    static_for<0, Z>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      const int e = p.extra[A][i];
      if (e < 0) return;
#pragma unroll
      for (int k = 0; k < N; ++k) {
        float tot = 0.0f;
        bool any = false;
#pragma unroll
        for (int l = 0; l < N; ++l) {
          if ((p.Enz[A][e] >> (3 * k + l)) & 1) {
            const float term = __fmul_rn(p.E[A][e][3 * k + l], t[i][l]);
            tot = any ? __fadd_rn(tot, term) : term;
            any = true;
          }
        }
        if (any) v[k] = __fadd_rn(v[k], tot);
      }
    });
  }
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

template <class Lat, int N, typename ST, bool PER>
static int launch_lattice_resident_t(const sck_plan* plan, LatticeResidentParams& p, int threads, cudaStream_t s) {
  size_t smem = (size_t)p.spin_bytes + sizeof(float) * p.table_floats;
  const cudaError_t e = cudaFuncSetAttribute(lattice_resident_kernel<Lat, N, ST, PER>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return cuda_status(e, "resident kernel shared memory");
  lattice_resident_kernel<Lat, N, ST, PER><<<p.c.B, threads, smem, s>>>(p);
  return cuda_status(cudaGetLastError(), "resident launch");
}

template <class Lat, bool PER>
static int launch_lattice_resident_n(const sck_plan* plan, LatticeResidentParams& p, int threads, cudaStream_t s) {
  if (plan->mode == SCK_MODE_INT8) return launch_lattice_resident_t<Lat, 1, int8_t, PER>(plan, p, threads, s);
  switch (plan->geom.n) {
    case 1: return launch_lattice_resident_t<Lat, 1, float, PER>(plan, p, threads, s);
    case 2: return launch_lattice_resident_t<Lat, 2, float, PER>(plan, p, threads, s);
    default: return launch_lattice_resident_t<Lat, 3, float, PER>(plan, p, threads, s);
  }
}

template <class Lat>
static int launch_lattice_resident_per(const sck_plan* plan, LatticeResidentParams& p, int threads, cudaStream_t s) {
  return lattice_periodic_box(plan, Lat::id) ? launch_lattice_resident_n<Lat, true>(plan, p, threads, s)
                                             : launch_lattice_resident_n<Lat, false>(plan, p, threads, s);
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
  p.n_classes = plan->desc.n_classes;
  for (int i = 0; i < p.n_classes; ++i) {
    p.classes[i][0] = plan->desc.classes[i][0];
    p.classes[i][1] = plan->desc.classes[i][1];
  }
  p.n_sweeps = n_sweeps;
  p.spin_bytes = (int)((resident_bytes(plan) + 15) / 16 * 16);
  if (plan->geom.n == 1) {
    const int floats = plan->geom.b * plan->keys;
    if (floats <= 2048 && p.spin_bytes + 4 * floats <= (220 << 10)) p.table_floats = floats;
  }
  const uint32_t per = (uint32_t)c.rows * (uint32_t)c.bx;
  int threads = (int)((per + 31) / 32 * 32);
  threads = threads < 128 ? 128 : (threads > 1024 ? 1024 : threads);
  switch (plan->resident_spec) {
    case Lat_square_1::id: return launch_lattice_resident_per<Lat_square_1>(plan, p, threads, s);
    case Lat_triangular_1::id: return launch_lattice_resident_per<Lat_triangular_1>(plan, p, threads, s);
    case Lat_sc_1::id: return launch_lattice_resident_per<Lat_sc_1>(plan, p, threads, s);
    case Lat_bcc_1::id: return launch_lattice_resident_per<Lat_bcc_1>(plan, p, threads, s);
    case Lat_bcc_1_2::id: return launch_lattice_resident_per<Lat_bcc_1_2>(plan, p, threads, s);
    default: return launch_lattice_resident_per<Lat_fcc_1>(plan, p, threads, s);
  }
}

}  // namespace sck
