// Specialised class kernels for the common crystals and the L2-resident group pipeline.
//
// Specialisation. When a system's bond lists equal one of the compile-time tables of lattices.h (one coupling
// group per shell, no extra matrices), its class launches run kernels in which every neighbour offset is a
// constant: the wrapped coordinates of a site are formed once for offsets -R..R per axis and every bond costs
// one add and one load per component. Ising keeps the integer key and the host table (bit-exact); vector models
// run two replicas per thread in packed float32x2 arithmetic (add.rn.f32x2 / mul.rn.f32x2, round-to-nearest
// per lane, same operation order as the generic kernel), with proposal trigonometry and exp on the SFU
// (__sinf / __cosf on [-pi, pi], __expf): per-spin differences from the reference stay ~1e-6. Vector models on
// lattices whose classes alternate along x run the segment kernels of segment.cu instead when the tuning level
// asks for them and their box allows it.
//
// Group pipeline. A sweep visits its C classes in order, and each class launch reads the whole state. When the
// state is larger than L2, the replicas are cut into groups whose C-group working set fits in L2, and launch k
// runs class c on group k - c for every c at once (a diagonal over (group, class)): the C launches that touch a
// group run back to back, so after its first read from HBM a group stays in L2 until its sweep is done. Each
// replica's chain is unchanged: its classes still run in order, one launch after another.
#include "words.cuh"

namespace sck {

// ------------------------------------------------------------------------------------------------- kernels
// Grid (ceil(rows * bx / 256), n_tasks * units_per_task). Block y-slot -> (task, `pairs` replica pairs): a thread forms
// its class site, its neighbours' offsets and the sweep's key once for all of them. Bound by instruction issue (304
// instructions per attempt with one pair a thread, 75 % of the issue slots, on Heisenberg bcc 32^3 x 2). Five blocks
// per SM: attempts/ns without a bound / at four / five / six, Heisenberg bcc J1-J2 64^3 x 2 x 64: 60 / 67 / 69 / 60;
// XY square 512^2 x 33: 157 / 157 / 162 / 160; the quick-start case 511 / 474 / 482 / 475 us.
template <class Lat, int N, bool PER, int NSL>
__global__ void __launch_bounds__(256, 5) spec_task_kernel(const __grid_constant__ SpecParams p) {
  follow_previous();
  const uint32_t per = (uint32_t)p.c.rows * (uint32_t)p.c.bx;
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= per) return;
  const int ti = blockIdx.y / p.units_per_task;
  const int unit = blockIdx.y - ti * p.units_per_task;
  const Task task = p.tasks[ti];
  const int rep0 = task.rep_begin + unit * 2 * p.pairs;
  const int rep1 = rep0 + 2 * p.pairs < task.rep_end ? rep0 + 2 * p.pairs : task.rep_end;
  if (rep0 >= rep1) return;
  int x, y, z;
  if (!class_site(p.c, task.colour, task.alpha, t, x, y, z)) return;
  const int32_t key = sweep_key_at(p.c.state, task.sweep_offset);
  static_for<0, Lat::b>([&](auto ac) {
    constexpr int a = decltype(ac)::value;
    if (a != task.alpha) return;
#pragma unroll 1
    for (int rep = rep0; rep < rep1; rep += 2)
      vec_spec_pair<Lat, a, N, PER, NSL>(p.c, p.J[a], rep, rep + 1 < rep1, x, y, z, key);
  });
}

// One class of int8 or float32 Ising replicas. A thread keeps its class site for several replicas: site, neighbour
// offsets and, per block, the sweep's round keys are formed once, and two replicas' loads are in flight together.
// Bound by instruction issue; the Philox call alone (36 instructions, 70 cycles of a scheduler's multiply pipe) is
// 131 us a sweep of 64^3 x 256 sites. Grid (class sites / 256, replica rows of p.per).
struct IsingClassParams {
  Common c;
  int colour, alpha, per;
};

template <class Lat, typename ST, bool PER>
__global__ void __launch_bounds__(256, 4) ising_class_kernel(const __grid_constant__ IsingClassParams p) {
  __shared__ uint4 keys[5];
  const Common& c = p.c;
  const Geometry& g = c.g;
  follow_previous();
  if (threadIdx.x < 10) write_keys(keys, sweep_key_at(c.state, c.sweep_offset), threadIdx.x);
  __syncthreads();
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  int x, y, z;
  if (t >= (uint32_t)c.rows * (uint32_t)c.bx || !class_site(c, p.colour, p.alpha, t, x, y, z)) return;
  const uint32_t own = (uint32_t)(p.alpha * g.plane + (z * g.L2 + y) * g.L1 + x);
  if (g.has_mask && c.mask[own] == 0) return;
  const RoundKeys rk = shared_keys(keys);
  const bool barker = g.acceptance == SCK_BARKER;
  const Around<Lat::reach, PER> nb(g, x, y, z);
  static_for<0, Lat::b>([&](auto ac) {
    constexpr int A = decltype(ac)::value;
    if (A != p.alpha) return;
    constexpr int Z = Lat::n_bonds(A);
    uint32_t off[Z];
    bool ok[Z];
    static_for<0, Z>([&](auto ic) {
      constexpr int i = decltype(ic)::value;
      constexpr BondC bd = Lat::bond(A, i);
      off[i] = (uint32_t)nb.index(g, bd);
      ok[i] = nb.valid(bd);
    });
    const int r0 = (int)blockIdx.y * p.per, r1 = r0 + p.per < c.B ? r0 + p.per : c.B;
    const uint32_t nsite = (uint32_t)g.nsite;
    const ST* src = (const ST*)c.src + (size_t)r0 * nsite;
    ST* dst = (ST*)c.dst + (size_t)r0 * nsite;
    const float* tab = (const float*)c.table + (size_t)r0 * c.lut_rep_stride + A * c.keys;
    uint32_t ctr = counter_of(r0, g.nsite, (int)own);
    auto replicas = [&](auto nc) {
      constexpr int N = decltype(nc)::value;
      int s[N], v[N][Z];
#pragma unroll
      for (int r = 0; r < N; ++r) {
        const ST* sr = src + (size_t)r * nsite;
        s[r] = sgn(sr[own]);
#pragma unroll
        for (int i = 0; i < Z; ++i) v[r][i] = ok[i] ? sgn(__ldg(sr + off[i])) : 0;
      }
      float e[N];
#pragma unroll
      for (int r = 0; r < N; ++r) {
        int k = s[r] > 0 ? 1 : 0, stride = 2;
        static_for<0, Lat::groups>([&](auto gc) {
          using R = GroupRange<Lat, A, decltype(gc)::value>;
          int G = 0;
#pragma unroll
          for (int i = R::begin; i < R::end; ++i) G += v[r][i];
          k += (G + (R::end - R::begin)) * stride;
          stride *= 2 * (R::end - R::begin) + 1;
        });
        e[r] = tab[(size_t)r * c.lut_rep_stride + k];
      }
#pragma unroll
      for (int r = 0; r < N; ++r) {
        const float u = to_uniform(philox_keys(ctr + (uint32_t)r * nsite, rk).x0);
        const bool acc = barker ? __fmul_rn(u, __fadd_rn(1.0f, e[r])) < 1.0f : u < e[r];
        if (acc) dst[(size_t)r * nsite + own] = (ST)(-s[r]);
      }
      src += (size_t)N * nsite;
      dst += (size_t)N * nsite;
      tab += (size_t)N * c.lut_rep_stride;
      ctr += (uint32_t)N * nsite;
    };
    int r = r0;
    for (; r + 2 <= r1; r += 2) replicas(std::integral_constant<int, 2>{});
    if (r < r1) replicas(std::integral_constant<int, 1>{});
  });
}

// The same for int8 spins on the square and simple cubic lattices, two colours, periodic, rows of whole 4-byte words:
// a thread takes one word of a row (two class sites) and walks along the last axis. Spins become codes 1 + sign, four
// at a time, and the codes of the neighbours add up byte by byte; a word's codes serve its own step and its
// neighbours' along the walk, so a step converts three words and loads three words and a byte for two attempts (the
// kernel above loads and converts seven bytes for each). What is left is mostly the Philox call. Grid (words of a
// plane or row / 256, chunks of the walk, replicas).
struct IsingMarchParams {
  Common c;
  int colour, chunk, r0;
};

// 1 + sign of four int8 spins.
__device__ __forceinline__ uint32_t spin_codes(uint32_t v) {
  const uint32_t nonneg = ~v & 0x80808080u;
  const uint32_t pos = nonneg & ((v & 0x7F7F7F7Fu) + 0x7F7F7F7Fu);
  return (nonneg >> 7) + (pos >> 7);
}

template <bool CUBIC, bool BARKER>
__global__ void __launch_bounds__(256, 4) ising_march_kernel(const __grid_constant__ IsingMarchParams p) {
  constexpr int Z = CUBIC ? 6 : 4;
  __shared__ uint4 keys[5];
  __shared__ float tab[2 * (2 * Z + 1)];
  const Common& c = p.c;
  const Geometry& g = c.g;
  follow_previous();
  const int rep = p.r0 + (int)blockIdx.z;
  if (threadIdx.x < 10) write_keys(keys, sweep_key_at(c.state, c.sweep_offset), threadIdx.x);
  for (int i = threadIdx.x; i < 2 * (2 * Z + 1); i += blockDim.x) {
    const float e = ((const float*)c.table)[(size_t)rep * c.lut_rep_stride + i];
    tab[i] = BARKER ? __fadd_rn(1.0f, e) : e;
  }
  __syncthreads();
  const int words = g.L1 >> 2;                       // of a row
  const int col = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (col >= words * (CUBIC ? g.L2 : 1)) return;
  const int y = CUBIC ? col / words : 0, xw = col - y * words;
  const int step = CUBIC ? g.L1 * g.L2 : g.L1, len = CUBIC ? g.L3 : g.L2;
  const int z0 = (int)blockIdx.y * p.chunk, z1 = min(len, z0 + p.chunk);
  const RoundKeys rk = shared_keys(keys);
  const int8_t* src = (const int8_t*)c.src + (size_t)rep * g.nsite;
  int8_t* dst = (int8_t*)c.dst + (size_t)rep * g.nsite;
  const int row = y * g.L1 + 4 * xw;                 // this word, and those beside it, within a plane
  const int ym = (y > 0 ? y - 1 : g.L2 - 1) * g.L1 + 4 * xw, yp = (y + 1 < g.L2 ? y + 1 : 0) * g.L1 + 4 * xw;
  const int left = y * g.L1 + (xw > 0 ? 4 * xw : g.L1) - 1, right = y * g.L1 + (xw + 1 < words ? 4 * xw + 4 : 0);
  // plain loads: a word holds bytes of the class that this launch writes, its own threads' and its neighbours', so the
  // read-only path, which needs memory that stays as it is for the whole kernel, is not for them
  auto word = [&](int at) { return *reinterpret_cast<const uint32_t*>(src + at); };
  // parity of the class in this row: it alternates along the walk
  int ph = CUBIC ? first_class_x(c, p.colour, 0, y, z0) : first_class_x(c, p.colour, 0, z0, 0);
  uint32_t below = spin_codes(word((z0 > 0 ? z0 - 1 : len - 1) * step + row)), here = spin_codes(word(z0 * step + row));
  const uint32_t ctr0 = counter_of(rep, g.nsite, row);
  // the next step's words are loaded ahead of this step's stores, past which the compiler may not move them
  uint32_t w_above, w_ym = 0u, w_yp = 0u;
  int8_t w_edge;
  auto load = [&](int z, int p1) {
    w_above = word((z + 1 < len ? z + 1 : 0) * step + row);
    if constexpr (CUBIC) {
      w_ym = word(z * step + ym);
      w_yp = word(z * step + yp);
    }
    w_edge = src[z * step + (p1 ? right : left)];
  };
  load(z0, ph);
#pragma unroll 2
  for (int z = z0; z < z1; ++z) {
    const int at = z * step;
    const uint32_t above = spin_codes(w_above);
    uint32_t sum = below + above;
    if constexpr (CUBIC) sum += spin_codes(w_ym) + spin_codes(w_yp);
    const uint32_t edge = (uint32_t)(1 + sgn(w_edge));
    load(min(z + 1, z1 - 1), ph ^ 1);
    const uint32_t even = here & 0x00FF00FFu, odd = (here >> 8) & 0x00FF00FFu;
    const uint32_t own = ph ? odd : even, other = ph ? even : odd;
    // neighbours along the row: the other residue's two, and one of them or the edge on the far side
    const uint32_t side = other + (ph ? (even >> 16) | (edge << 16) : (odd << 16) | edge);
    const uint32_t key2 = 2u * (((sum >> (8 * ph)) & 0x00FF00FFu) + side) + ((own >> 1) & 0x00010001u);
    const uint32_t ctr = ctr0 + (uint32_t)(at + ph);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float e = tab[j ? key2 >> 16 : key2 & 0xFFFFu];
      const float u = to_uniform(philox_keys(ctr + 2u * j, rk).x0);
      const bool acc = BARKER ? __fmul_rn(u, e) < 1.0f : u < e;
      if (acc) dst[at + row + ph + 2 * j] = (int8_t)(1 - (int)((own >> (16 * j)) & 0xFFu));
    }
    below = here;
    here = above;
    ph ^= 1;
  }
}

// ----------------------------------------------------------------------------------- the streamed pipeline
// One launch runs the group pipeline of several sweeps. Tickets, taken from a counter in the order blocks start,
// enumerate stages k = 0, 1, ...; stage k holds class ci of unit k - ci (unit = sweep-major group) for every ci,
// each class task split into T tickets (slot of the group x chunk of site blocks). Before touching spins a
// block waits until every ticket of the task it follows has finished: class ci - 1 of its unit, or, for class
// 0, class C - 1 of the same group's previous sweep. That task holds smaller tickets, so its blocks started
// before this one and are running or done: the wait ends. Tasks of one group are therefore serialised exactly
// as class launches are, tasks of different groups overlap freely, and a group's state is read from HBM once
// per sweep while its C classes pass over it from L2.
constexpr int kStreamSiteBlocks = 1;                 // site blocks of 256 threads per ticket
static __device__ unsigned long long g_stream_wait_timeouts;

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* a) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(a) : "memory");
  return v;
}

struct StreamTask {
  int go;            // 0: no task (pipeline fill / drain) or a wait that gave up
  int rep, rep_end;  // first replica of this block's slot, end of its group
  int colour, alpha, sweep;
  int done;          // index of this task's completion counter
  uint32_t t0;       // first class-site thread of this block
};

template <class Lat, int N, typename ST, bool PER, int NSL>
__global__ void __launch_bounds__(256, 5) stream_kernel(const __grid_constant__ StreamParams p) {
  __shared__ StreamTask s;
  if (threadIdx.x == 0) {
    const unsigned tk = atomicAdd(p.ticket, 1u);
    const unsigned stage = (unsigned)p.C * (unsigned)p.T;
    const unsigned k = tk / stage;
    const unsigned r = tk - k * stage;
    const int ci = (int)(r / (unsigned)p.T), j = (int)(r - (unsigned)ci * (unsigned)p.T);
    const int u = (int)k - ci;
    s.go = 0;
    s.done = -1;
    if (u >= 0 && u < p.units) {
      const int sw = u / p.ngroups, g = u - sw * p.ngroups;
      const int q = j / p.chunks, chunk = j - q * p.chunks;
      constexpr int per_slot = N == 1 ? 1 : 2;
      s.rep = g * p.group + q * per_slot;
      s.rep_end = min(p.c.B, (g + 1) * p.group);
      s.colour = p.cls[ci][0];
      s.alpha = p.cls[ci][1];
      s.sweep = p.sweep_base + sw;
      s.done = g * p.C + ci;
      s.t0 = (uint32_t)chunk * (kStreamSiteBlocks * 256u);
      const unsigned* dep = nullptr;
      unsigned need = 0;
      if (ci > 0) {
        dep = p.done + s.done - 1;
        need = (unsigned)(sw + 1) * (unsigned)p.T;
      } else if (sw > 0) {
        dep = p.done + g * p.C + p.C - 1;
        need = (unsigned)sw * (unsigned)p.T;
      }
      int go = 1;
      if (dep != nullptr) {
        unsigned polls = 0;
        while (ld_acquire_u32(dep) < need) {
          if (++polls > p.c.wait_limit) {
            go = 0;
            atomicAdd(&g_stream_wait_timeouts, 1ull);
            if (p.c.giveup != nullptr) atomicExch_system(p.c.giveup, 1);
            break;
          }
          __nanosleep(100);
        }
      }
      s.go = go && s.rep < s.rep_end;
    }
  }
  __syncthreads();
  if (s.done < 0) return;                              // the pipeline's fill and drain: no task
  if (s.go) {
    const int rep = s.rep, rep_end = s.rep_end, alpha = s.alpha;
    const int32_t key = sweep_key_at(p.c.state, s.sweep);
    const uint32_t per = (uint32_t)p.c.rows * (uint32_t)p.c.bx;
#pragma unroll 1
    for (int sb = 0; sb < kStreamSiteBlocks; ++sb) {
      const uint32_t t = s.t0 + sb * 256u + threadIdx.x;
      int x, y, z;
      if (t < per && class_site(p.c, s.colour, alpha, t, x, y, z)) {
        static_for<0, Lat::b>([&](auto ac) {
          constexpr int a = decltype(ac)::value;
          if (a != alpha) return;
          if constexpr (N == 1) {
            ising_spec_site<Lat, a, ST, PER>(p.c, rep, x, y, z, key);
          } else {
            vec_spec_pair<Lat, a, N, PER, NSL>(p.c, p.J[a], rep, rep + 1 < rep_end, x, y, z, key);
          }
        });
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    atomicAdd(p.done + s.done, 1u);   // finished (or given up): later tasks of this group may start
  }
}

int stream_wait_timeouts(unsigned long long* count) {
  return cuda_status(cudaMemcpyFromSymbol(count, g_stream_wait_timeouts, sizeof(*count)), "stream wait timeouts");
}

// ------------------------------------------------------------------------------------------ host: matching
template <class Lat>
static bool matches(const sck_plan* p, bool extras) {
  const sck_system_desc& d = p->desc;
  if (d.b != Lat::b || d.dim != Lat::dim) return false;
  for (int a = 0; a < d.b; ++a) {
    const sck_sublattice& s = d.sub[a];
    if (s.n_groups != Lat::groups || s.n_bonds != Lat::n_bonds(a) || (s.n_extra != 0 && !extras))
      return false;
    for (int gi = 0; gi < s.n_groups; ++gi)
      if (!s.group_apply[gi] || s.group_end[gi] != Lat::group_end(a, gi)) return false;
    for (int i = 0; i < s.n_bonds; ++i) {
      const BondC b = Lat::bond(a, i);
      const sck_bond& e = s.bonds[i];
      if (e.alpha2 != b.a2 || e.d[0] != b.dx || e.d[1] != b.dy || e.d[2] != b.dz || (e.extra != -1 && !extras))
        return false;
    }
  }
  return true;
}

// Id of the compile-time table that equals the plan's bond lists, or 0; with `extras`, extra matrices on its bonds are left
// aside.
int match_lattice(const sck_plan* p, bool extras) {
  if (matches<Lat_square_1>(p, extras)) return Lat_square_1::id;
  if (matches<Lat_triangular_1>(p, extras)) return Lat_triangular_1::id;
  if (matches<Lat_sc_1>(p, extras)) return Lat_sc_1::id;
  if (matches<Lat_bcc_1>(p, extras)) return Lat_bcc_1::id;
  if (matches<Lat_bcc_1_2>(p, extras)) return Lat_bcc_1_2::id;
  if (matches<Lat_fcc_1>(p, extras)) return Lat_fcc_1::id;
  return 0;
}

int find_spec(const sck_plan* p) {
  if (p->mode != SCK_MODE_INT8 && p->mode != SCK_MODE_F32 && p->mode != SCK_MODE_QUAD) return 0;
  return match_lattice(p);
}

// ------------------------------------------------------------------------------------------- host: launches
// Grids of the vector class kernel that overlap the class before them: those of at most half a block per SM, of two to
// two and a half blocks per SM, and of four fifths of the GPU's 740 places and more. Between these, the blocks that come early
// share the SMs that the previous launch leaves room on, several to one while others stay empty, and the launch takes longer
// than one that spreads over all SMs. Time of plain over overlapping launches, mean and range of 262 sweeps:
//   blocks   up to 74    75-148     149-222    223-296    297-370    371-444    445-591    592-1,183  more
//   mean     1.06        0.85       0.77       0.78       1.01       0.80       0.95       1.08       1.01-1.05
//   range    0.96-1.18   0.68-1.02  0.65-0.92  0.67-1.04  0.94-1.10  0.76-0.88  0.90-1.03  1.04-1.12
static bool overlap_pays(dim3 grid) {
  constexpr long long kSms = 148, kPlaces = 5 * kSms;
  const long long blocks = (long long)grid.x * grid.y;
  return 2 * blocks <= kSms || (blocks > 2 * kSms && 2 * blocks <= 5 * kSms) || 5 * blocks >= 4 * kPlaces;
}

template <class Lat, int N, typename ST, bool PER, int NSL, class P>
static void launch_one(const P& p, dim3 grid, cudaStream_t s) {
  if constexpr (std::is_same_v<P, SpecParams>)
    launch_dependent(spec_task_kernel<Lat, N, PER, NSL>, grid, 256, s, p, overlap_pays(grid));
  else
    stream_kernel<Lat, N, ST, PER, NSL><<<grid, 256, 0, s>>>(p);
}

template <class Lat, int N, bool PER, class P>
static void launch_vec(const sck_plan* plan, const P& p, dim3 grid, cudaStream_t s) {
  // replicas of 2^16 .. 2^19 sites on periodic boxes: component strides up to 2 MiB fit a load's immediate offset
  if constexpr (PER) {
    const int64_t ns = plan->geom.nsite;
    if (ns == (1 << 16)) return launch_one<Lat, N, float, PER, 16>(p, grid, s);
    if (ns == (1 << 17)) return launch_one<Lat, N, float, PER, 17>(p, grid, s);
    if (ns == (1 << 18)) return launch_one<Lat, N, float, PER, 18>(p, grid, s);
    if (ns == (1 << 19)) return launch_one<Lat, N, float, PER, 19>(p, grid, s);
  }
  launch_one<Lat, N, float, PER, 0>(p, grid, s);
}

template <class Lat, bool PER, class P>
static void launch_lat_per(const sck_plan* plan, const P& p, dim3 grid, cudaStream_t s) {
  if (plan->geom.n == 1) {
    if constexpr (!std::is_same_v<P, SpecParams>) {      // launch_tasks refuses Ising plans
      if (plan->mode == SCK_MODE_INT8)
        launch_one<Lat, 1, int8_t, PER, 0>(p, grid, s);
      else
        launch_one<Lat, 1, float, PER, 0>(p, grid, s);
    }
  } else if (plan->geom.n == 2) {
    launch_vec<Lat, 2, PER>(plan, p, grid, s);
  } else {
    launch_vec<Lat, 3, PER>(plan, p, grid, s);
  }
}

// All axes periodic (2D: x and y) with every extent >= the bond reach: the branch-free wrap applies.
template <class Lat>
static bool periodic_box(const sck_plan* plan) {
  const Geometry& g = plan->geom;
  if (!g.per[0] || !g.per[1] || g.L1 < Lat::reach || g.L2 < Lat::reach) return false;
  return g.dim == 2 || (g.per[2] && g.L3 >= Lat::reach);
}

int lattice_periodic_box(const sck_plan* plan, int id) {
  switch (id) {
    case Lat_square_1::id: return periodic_box<Lat_square_1>(plan) ? 1 : 0;
    case Lat_triangular_1::id: return periodic_box<Lat_triangular_1>(plan) ? 1 : 0;
    case Lat_sc_1::id: return periodic_box<Lat_sc_1>(plan) ? 1 : 0;
    case Lat_bcc_1::id: return periodic_box<Lat_bcc_1>(plan) ? 1 : 0;
    case Lat_bcc_1_2::id: return periodic_box<Lat_bcc_1_2>(plan) ? 1 : 0;
    case Lat_fcc_1::id: return periodic_box<Lat_fcc_1>(plan) ? 1 : 0;
    default: return 0;
  }
}

int spec_periodic_box(const sck_plan* plan) { return lattice_periodic_box(plan, plan->spec); }

template <class Lat, class P>
static void launch_lat(const sck_plan* plan, const P& p, dim3 grid, cudaStream_t s) {
  if (periodic_box<Lat>(plan))
    launch_lat_per<Lat, true>(plan, p, grid, s);
  else
    launch_lat_per<Lat, false>(plan, p, grid, s);
}

// replicas per grid y-slot: vector models pair two replicas per thread in the lattice kernels
template <class P>
static void launch_spec_grid(const sck_plan* plan, const P& p, dim3 grid, cudaStream_t s) {
  switch (plan->spec) {
    case Lat_square_1::id: launch_lat<Lat_square_1>(plan, p, grid, s); break;
    case Lat_triangular_1::id: launch_lat<Lat_triangular_1>(plan, p, grid, s); break;
    case Lat_sc_1::id: launch_lat<Lat_sc_1>(plan, p, grid, s); break;
    case Lat_bcc_1::id: launch_lat<Lat_bcc_1>(plan, p, grid, s); break;
    case Lat_bcc_1_2::id: launch_lat<Lat_bcc_1_2>(plan, p, grid, s); break;
    default: launch_lat<Lat_fcc_1>(plan, p, grid, s); break;
  }
}

static int slot_replicas(const sck_plan* plan) { return seg_kernel_ok(plan) ? 1 : 2; }

// Class tasks of vector models. Ising classes have kernels of their own (launch_ising_class, launch_ising_march).
static int launch_tasks(const sck_plan* plan, SpecParams& p, cudaStream_t s) {
  if (plan->geom.n == 1) return cuda_status(cudaErrorInvalidValue, "task launch of an Ising plan");
  int per_unit = slot_replicas(plan);
  int most = 1;
  for (int i = 0; i < p.n_tasks; ++i) {
    const int n = p.tasks[i].rep_end - p.tasks[i].rep_begin;
    if (n > most) most = n;
  }
  const uint32_t per = (uint32_t)p.c.rows * (uint32_t)p.c.bx;
  p.pairs = 1;
  // up to four pairs a thread while eight blocks per SM are left: attempts/ns at one / two / four pairs, XY square 512^2
  // x 33: 116 / 142 / 166; Heisenberg sc 40^3 x 100: 82 / 89 / 92; bcc 32^3 x 64: 86 / 96 / 96; bcc J1-J2 64^3 x 2 x 64,
  // whose 42 neighbour loads outweigh what pairs share: 64 / 63 / 62
  if (per_unit == 2)
    while (p.pairs < 4 && (long long)((per + 255) / 256) * p.n_tasks * ((most + 4 * p.pairs - 1) / (4 * p.pairs)) >= 148 * 8)
      p.pairs *= 2;
  per_unit *= p.pairs;
  p.units_per_task = (most + per_unit - 1) / per_unit;
  const long long ys = (long long)p.units_per_task * p.n_tasks;
  if (ys > 65535) return cuda_status(cudaErrorInvalidConfiguration, "task launch: too many replicas per launch");
  if (seg_kernel_ok(plan)) return launch_seg_tasks(plan, p, (int)ys, s);
  launch_spec_grid(plan, p, dim3((per + 255) / 256, (unsigned)ys), s);
  return cuda_status(cudaGetLastError(), "specialised class launch");
}

static SpecParams spec_params(const sck_plan* plan, const Common& c) {
  SpecParams p;
  memset(&p, 0, sizeof(p));
  p.c = c;
  for (int a = 0; a < SCK_MAX_BASIS; ++a)
    for (int gi = 0; gi < SCK_MAX_GROUPS; ++gi) p.J[a][gi] = plan->sub[a].J[gi];
  return p;
}

template <class Lat>
static void launch_ising_t(const sck_plan* plan, const IsingClassParams& p, dim3 grid, cudaStream_t s) {
  const bool per = periodic_box<Lat>(plan);
  if (plan->mode == SCK_MODE_INT8) {
    if (per) ising_class_kernel<Lat, int8_t, true><<<grid, 256, 0, s>>>(p);
    else ising_class_kernel<Lat, int8_t, false><<<grid, 256, 0, s>>>(p);
  } else {
    if (per) ising_class_kernel<Lat, float, true><<<grid, 256, 0, s>>>(p);
    else ising_class_kernel<Lat, float, false><<<grid, 256, 0, s>>>(p);
  }
}

// The marching kernel's systems: the walk and both row directions alternate between the two colours, the words of a
// plane or row fill at least 7/16 of its blocks' threads, and there are enough walks of eight sites to occupy the GPU.
// Everything else takes ising_class_kernel. Class kernel against marching, us a sweep:
//   filled:  square 4 x 60,000 x 100 (1 word of 256) 129 / 4,425; 256 x 1,024 x 33 (64) 50.2 / 57.8;
//            500^2 x 33 (125) 48.6 / 45.4; 1,024 x 256 x 33 (256) 50.2 / 44.6
//   walks:   sc 64^3 x 1 (8,192) 7.6 / 14.0, x 3 (24,576) 14.7 / 15.1, x 4 (32,768) 18.1 / 15.2; sc 96^3 x 1 (27,648)
//            15.8 / 14.4; square 512^2 x 2 (16,384) 10.6 / 10.9, x 3 (24,576) 13.4 / 11.7
constexpr long long kMarchWalks = 26000, kMarchWalks2 = 20000;   // three dimensions, two

bool ising_march_plan(const sck_plan* plan) {
  const Geometry& g = plan->geom;
  if (plan->mode != SCK_MODE_INT8 || g.has_mask || g.L1 % 4 != 0 || !spec_periodic_box(plan)) return false;
  if (plan->spec != Lat_square_1::id && plan->spec != Lat_sc_1::id) return false;
  const Colouring& col = plan->col;
  if (col.r != 1 || col.m[0] != 2) return false;
  for (int k = 0; k < g.dim; ++k)
    if (col.K[0][k] != 1) return false;
  const int cols = g.L1 / 4 * (g.dim == 3 ? g.L2 : 1), len = g.dim == 3 ? g.L3 : g.L2;
  if (16 * (long long)cols < 7 * 256 * (long long)((cols + 255) / 256)) return false;
  return (long long)cols * ((len + 7) / 8) * plan->Bp >= (g.dim == 3 ? kMarchWalks : kMarchWalks2);
}

// Its 4-byte loads need spins that start on 4 bytes.
static bool ising_march_ok(const sck_plan* plan, const void* spins, int colour) {
  return colour <= 1 && ((uintptr_t)spins & 3u) == 0 && ising_march_plan(plan);
}

// Chunks of the walk: long ones convert fewer words twice, short ones keep 16 blocks per SM; at least 8 sites.
static int launch_ising_march(const sck_plan* plan, const Common& c, int colour, cudaStream_t s) {
  const Geometry& g = plan->geom;
  const bool cubic = g.dim == 3, barker = g.acceptance == SCK_BARKER;
  IsingMarchParams p;
  p.c = c;
  p.colour = colour;
  const int cols = g.L1 / 4 * (cubic ? g.L2 : 1), len = cubic ? g.L3 : g.L2;
  const long long blocks = (long long)((cols + 255) / 256) * c.B;
  const long long split = (148 * 16 + blocks - 1) / blocks;
  p.chunk = (int)((len + split - 1) / split);
  if (p.chunk < 8) p.chunk = 8;
  for (p.r0 = 0; p.r0 < c.B; p.r0 += 65535) {
    const int n = c.B - p.r0 < 65535 ? c.B - p.r0 : 65535;
    const dim3 grid((unsigned)((cols + 255) / 256), (unsigned)((len + p.chunk - 1) / p.chunk), (unsigned)n);
    if (cubic) {
      if (barker) ising_march_kernel<true, true><<<grid, 256, 0, s>>>(p);
      else ising_march_kernel<true, false><<<grid, 256, 0, s>>>(p);
    } else {
      if (barker) ising_march_kernel<false, true><<<grid, 256, 0, s>>>(p);
      else ising_march_kernel<false, false><<<grid, 256, 0, s>>>(p);
    }
    const int rc = cuda_status(cudaGetLastError(), "Ising class launch");
    if (rc != SCK_OK) return rc;
  }
  return SCK_OK;
}

// Replicas per thread: up to eight, as long as the launch keeps sixteen blocks per SM (four rounds of its four).
static int launch_ising_class(const sck_plan* plan, const Common& c, int colour, int alpha, cudaStream_t s) {
  IsingClassParams p;
  p.c = c;
  p.colour = colour;
  p.alpha = alpha;
  const uint32_t per = (uint32_t)c.rows * (uint32_t)c.bx;
  const unsigned bx = (per + 255) / 256;
  p.per = 1;
  while (p.per < 8 && (long long)bx * ((c.B + 2 * p.per - 1) / (2 * p.per)) >= 148 * 16) p.per *= 2;
  if ((c.B + p.per - 1) / p.per > 65535) p.per = (c.B + 65534) / 65535;
  const dim3 grid(bx, (unsigned)((c.B + p.per - 1) / p.per));
  switch (plan->spec) {
    case Lat_square_1::id: launch_ising_t<Lat_square_1>(plan, p, grid, s); break;
    case Lat_triangular_1::id: launch_ising_t<Lat_triangular_1>(plan, p, grid, s); break;
    case Lat_sc_1::id: launch_ising_t<Lat_sc_1>(plan, p, grid, s); break;
    case Lat_bcc_1::id: launch_ising_t<Lat_bcc_1>(plan, p, grid, s); break;
    case Lat_bcc_1_2::id: launch_ising_t<Lat_bcc_1_2>(plan, p, grid, s); break;
    default: launch_ising_t<Lat_fcc_1>(plan, p, grid, s); break;
  }
  return cuda_status(cudaGetLastError(), "Ising class launch");
}

// One class over all replicas, in chunks of at most 65535 grid rows.
int launch_spec_class(const sck_plan* plan, const Common& c, int colour, int alpha, cudaStream_t s) {
  if (plan->geom.n == 1)
    return ising_march_ok(plan, c.src, colour) ? launch_ising_march(plan, c, colour, s) : launch_ising_class(plan, c, colour, alpha, s);
  if (tile_kernel_ok(plan)) return launch_tile_class(plan, c, colour, alpha, s);
  SpecParams p = spec_params(plan, c);
  const int chunk = 65535 * slot_replicas(plan);
  for (int r0 = 0; r0 < c.B; r0 += chunk) {
    p.n_tasks = 1;
    p.tasks[0] = Task{colour, alpha, r0, r0 + chunk < c.B ? r0 + chunk : c.B, c.sweep_offset};
    const int rc = launch_tasks(plan, p, s);
    if (rc != SCK_OK) return rc;
  }
  return SCK_OK;
}

size_t stream_counter_bytes(const sck_plan* plan, int group) {
  const int ngroups = (plan->Bp + group - 1) / group;
  return (size_t)(1 + ngroups * plan->desc.n_classes) * sizeof(unsigned);
}

// n sweeps of the group pipeline (streamed kernel, one launch per chunk of sweeps); state[1] is advanced by
// the caller. `counters` holds stream_counter_bytes(plan, group) bytes of device memory, zeroed here before
// every launch.
int launch_spec_pipeline(const sck_plan* plan, const Common& c, int n_sweeps, int group, void* counters,
                         cudaStream_t s) {
  if (counters == nullptr) {
    set_error("the group pipeline has no completion counters (set an L2 budget with sck_plan_tune)");
    return SCK_ERR_INVALID;
  }
  const int C = plan->desc.n_classes;
  StreamParams p;
  memset(&p, 0, sizeof(p));
  p.c = c;
  for (int a = 0; a < SCK_MAX_BASIS; ++a)
    for (int gi = 0; gi < SCK_MAX_GROUPS; ++gi) p.J[a][gi] = plan->sub[a].J[gi];
  p.C = C;
  for (int ci = 0; ci < C; ++ci) {
    p.cls[ci][0] = plan->desc.classes[ci][0];
    p.cls[ci][1] = plan->desc.classes[ci][1];
  }
  p.group = group;
  p.ngroups = (c.B + group - 1) / group;
  const int per_slot = plan->geom.n == 1 ? 1 : 2;
  const long long site_blocks = ((long long)c.rows * c.bx + 255) / 256;
  p.chunks = (int)((site_blocks + kStreamSiteBlocks - 1) / kStreamSiteBlocks);
  p.T = ((group + per_slot - 1) / per_slot) * p.chunks;
  p.ticket = (unsigned*)counters;
  p.done = p.ticket + 1;
  // tickets of a launch, (units + C - 1) x C x T, stay below 2^30
  const long long stage = (long long)C * p.T;
  const long long most_units = (1ll << 30) / stage - (C - 1);
  const long long sweeps_per_launch = most_units / p.ngroups;
  if (sweeps_per_launch < 1) return cuda_status(cudaErrorInvalidConfiguration, "group pipeline: too many tickets");
  const size_t bytes = stream_counter_bytes(plan, group);
  for (int sw0 = 0; sw0 < n_sweeps; sw0 += (int)sweeps_per_launch) {
    const int n = (int)((long long)(n_sweeps - sw0) < sweeps_per_launch ? n_sweeps - sw0 : sweeps_per_launch);
    p.units = n * p.ngroups;
    p.sweep_base = sw0;
    int rc = cuda_status(cudaMemsetAsync(counters, 0, bytes, s), "group pipeline counters");
    if (rc != SCK_OK) return rc;
    launch_spec_grid(plan, p, dim3((unsigned)((p.units + C - 1) * stage)), s);
    rc = cuda_status(cudaGetLastError(), "group pipeline launch");
    if (rc != SCK_OK) return rc;
  }
  return SCK_OK;
}

}  // namespace sck
