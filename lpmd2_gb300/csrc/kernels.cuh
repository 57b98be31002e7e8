// kernels.cuh -- the sm_103a kernels of the MD timestep.
//
//   k_rebuild_list the systems of a batch that rebuild, for the kernels of the chain
//   k_decide       per system: does this force evaluation need a cell/list rebuild?
//                  (LinkedCell rebuilds at every UpdateCell, plugins/linkedcell.cc:112-267;
//                   the Verlet list on displacement > skin/2 and/or every `each` UpdateCell
//                   calls, plugins/verletlist.cc:124-131)
//   k_bin          FP64 cell index of every atom (plugins/linkedcell.cc:249-253) + histogram
//   k_scan         per-system exclusive scan of the cell histogram
//   k_scatter      counting-sort scatter into cells
//   k_cellsort     orders each cell by original atom index (the reference's linked-list order)
//   k_permute      gathers every per-atom field into the new cell-sorted order (scratch)
//   k_copyback     writes the sorted fields back, refreshes gather copies and home cells
//   k_sort_cluster the same sort in one launch, for small systems
//   k_buildlist_block, k_buildlist_warp
//                  Verlet list from the 27/125-cell stencil with per-pair cell-shift codes, a block or
//                  a warp for each home cell
//   k_scale_*      velocity rescaling between steps
//   k_drift        VelocityVerlet::AdvancePosition (plugins/velocityverlet.cc:60-68) + wrap,
//                  gather copies, displacement tracking (stand-alone; a step's drift is part of the
//                  force pass before it)
// The force, density and thermo kernels are in forces.cuh (mixed precision) and force64.cuh (FP64).
#pragma once

#include <type_traits>

#include "device.cuh"
#include "potentials.cuh"

namespace gbmd {

enum EpiMode { EPI_FORCES = 0, EPI_KICK = 1, EPI_KICK_DRIFT = 2 };

struct StepParams {
  double dt;
  double half_dt;       // 0.5 * dt, as AdvanceVelocity computes it
  double half_dt2;      // 0.5 * dt * dt (mixed drift)
  int epi;              // EpiMode of the final force pass
  int first;            // first potential pass of this evaluation (overwrite partials)
  int last;             // last potential pass (write accelerations)
  int count_step;       // k_thermo advances the step counter
  int kinetic;          // compute kinetic sums in the epilogue
  int raw_acc;          // keep fixedvel atoms' accelerations (a bare UpdateForces, no integrator)
};

// ---------------------------------------------------------------------------------------------
// Rebuild decision
// ---------------------------------------------------------------------------------------------

// ucall_inc: how many emulated UpdateCell calls this evaluation stands for (verletlist "each").
// Rebuild decision of one system for the next force evaluation (one warp): clears the system's
// fixed-point accumulators and returns whether its cells/list are rebuilt.
__device__ __forceinline__ int decide_system(const Dev& D, int s, int ucall_inc, int force_all) {
  const SysDev& S = D.sysd[s];
  SysState& st = D.sst[s];
  const int lane = threadIdx.x & 31;
  if (!S.active) {
    if (lane == 0) st.need_rebuild = 0;
    return 0;
  }
  if (lane < SA_LEN) D.sys_acc[(long long)s * SA_LEN + lane] = 0ull;
  int need = 0;
  if (lane == 0) {
    need = force_all | st.force_rebuild;
    const long long ucalls = st.ucalls;
    if (S.mode == NB_CELLS) need = 1;
    if (S.mode == NB_LIST) {
      float md2 = __int_as_float((int)__ldcg(&st.maxdisp2));  // atomics of the previous launch
      if ((S.rebuild_policy == REBUILD_SKIN || S.rebuild_policy == REBUILD_BOTH) && (double)md2 > S.thresh2)
        need = 1;
      if (S.rebuild_policy == REBUILD_EACH || S.rebuild_policy == REBUILD_BOTH) {
        for (int k = 0; k < ucall_inc; ++k)
          if (((ucalls + k) % S.each) == 0) need = 1;
      }
    }
    st.ucalls = ucalls + ucall_inc;
    if (S.mode == NB_ALLPAIRS) need = 0;
    st.need_rebuild = need;
    st.force_rebuild = 0;
    if (need) {
      D.outside[s] = 0;
      st.maxdisp2 = 0u;
      st.rebuilds += (S.mode == NB_LIST) ? 1 : 0;
    }
  }
  return __shfl_sync(0xffffffffu, need, 0);
}

// One warp per system.  Inside a graph the conditional of the step starts at 0 at every graph
// launch (cudaGraphCondAssignDefault): a warp raises it when its system rebuilds.
constexpr int SYS_WARPS = 4;  // systems per block of the per-system kernels
__global__ void __launch_bounds__(32 * SYS_WARPS) k_decide(Dev D, int nsys, int ucall_inc, int force_all,
                                                           unsigned long long cond_handle, int use_cond) {
  const int s = blockIdx.x * SYS_WARPS + (threadIdx.x >> 5);
  if (s >= nsys) return;
  const int need = decide_system(D, s, ucall_inc, force_all);
  if (need && use_cond && (threadIdx.x & 31) == 0)
    cudaGraphSetConditional((cudaGraphConditionalHandle)cond_handle, 1u);
}

// ---------------------------------------------------------------------------------------------
// Binning and counting sort
// ---------------------------------------------------------------------------------------------

// Work of the rebuild chain.  A batch rebuilds a few of its systems at a time (each by its own
// displacements), so the chain's kernels do not run over every atom and cell of the batch: their
// units (chunks of REBUILD_CHUNK atoms, or cells) are numbered over the rebuilding systems alone,
// listed by k_rebuild_list.  A single system needs no list.
constexpr int REBUILD_CHUNK = 256;

constexpr int RLIST_THREADS = 1024;
__global__ void __launch_bounds__(RLIST_THREADS) k_rebuild_list(Dev D) {
  __shared__ int part[RLIST_THREADS / 32][3];
  __shared__ int carry[3];
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < 3) carry[threadIdx.x] = 0;
  __syncthreads();
  for (int base = 0; base < D.nsys; base += RLIST_THREADS) {
    const int s = base + (int)threadIdx.x;
    const bool need = s < D.nsys && D.sst[s].need_rebuild;
    int v[3] = {need ? 1 : 0, need ? (D.sysd[s].natoms + REBUILD_CHUNK - 1) / REBUILD_CHUNK : 0,
                need ? D.sysd[s].ncells : 0};
    int x[3];
    for (int k = 0; k < 3; ++k) {
      x[k] = v[k];
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(all, x[k], o);
        if (lane >= o) x[k] += y;
      }
      if (lane == 31) part[w][k] = x[k];
    }
    __syncthreads();
    if (w < 3) {
      int t = part[lane][w];
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(all, t, o);
        if (lane >= o) t += y;
      }
      part[lane][w] = t;
    }
    __syncthreads();
    for (int k = 0; k < 3; ++k) x[k] += carry[k] + (w > 0 ? part[w - 1][k] : 0);
    if (need) {
      const int r = x[0] - 1;
      D.rb_sys[r] = s;
      D.rb_chunk0[r] = x[1] - v[1];
      D.rb_cell0[r] = x[2] - v[2];
    }
    __syncthreads();
    if (threadIdx.x == RLIST_THREADS - 1)
      for (int k = 0; k < 3; ++k) carry[k] = x[k];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *D.rb_n = carry[0];
    D.rb_chunk0[carry[0]] = carry[1];
    D.rb_cell0[carry[0]] = carry[2];
  }
}

// System and chunk (CELLS: cell) of unit u, false past the last one.
template <bool CELLS>
__device__ __forceinline__ bool rebuild_unit(const Dev& D, int u, int& s, int& v) {
  if (D.nsys == 1) {
    s = 0;
    v = u;
    if (!D.sst[0].need_rebuild) return false;
    return u < (CELLS ? D.sysd[0].ncells : (D.sysd[0].natoms + REBUILD_CHUNK - 1) / REBUILD_CHUNK);
  }
  const int* pre = CELLS ? D.rb_cell0 : D.rb_chunk0;
  int lo = 0, hi = *D.rb_n;
  if (u >= pre[hi]) return false;
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (pre[mid] <= u)
      lo = mid;
    else
      hi = mid;
  }
  s = D.rb_sys[lo];
  v = u - pre[lo];
  return true;
}

// Calls body(system, atom) for this thread's atoms of the rebuilding systems.
template <class F>
__device__ __forceinline__ void for_rebuild_atoms(const Dev& D, F&& body) {
  int s, v;
  for (int u = blockIdx.x; rebuild_unit<false>(D, u, s, v); u += gridDim.x) {
    const int k = v * REBUILD_CHUNK + (int)threadIdx.x;
    if (k < D.sysd[s].natoms) body(s, D.sysd[s].atom_base + k);
  }
}

__device__ __forceinline__ void bin_atom(const Dev& D, int s, long long i) {
  const SysDev& S = D.sysd[s];
  bool ok = true;
  int cx, cy, cz;
  if (S.mode == NB_LIST) {
    // Verlet-list grid: cells are wider than the list radius by a margin, so the binning may
    // round differently from LinkedCell's; one multiply instead of a division per axis
    cx = list_cell_coord(D.x[i] * S.ninv[0], S.n[0], ok);
    cy = list_cell_coord(D.y[i] * S.ninv[1], S.n[1], ok);
    cz = list_cell_coord(D.z[i] * S.ninv[2], S.n[2], ok);
  } else {
    cx = ref_cell_coord(D.x[i], S.L[0], S.n[0], ok);
    cy = ref_cell_coord(D.y[i], S.L[1], S.n[1], ok);
    cz = ref_cell_coord(D.z[i], S.L[2], S.n[2], ok);
    // a coordinate n is the first cell of the next row or plane, as in the reference (linkedcell.cc:253);
    // past the last plane, where the reference keeps the atom in no cell, it is cell 0
    if ((cz * S.n[1] + cy) * S.n[0] + cx >= S.ncells) {
      if (cx == S.n[0]) cx = 0;
      if (cy == S.n[1]) cy = 0;
      if (cz == S.n[2]) cz = 0;
    }
  }
  if (!ok) {
    atomicOr(&D.sst[s].error, ERR_OUTSIDE);
    cx = cy = cz = 0;
  }
  const int c = S.cell_base + (cz * S.n[1] + cy) * S.n[0] + cx;
  D.acell[i] = c;
  // consecutive atoms mostly share a cell (the arrays are in the previous cell order): one
  // atomic per cell and warp
  const unsigned peers = __match_any_sync(__activemask(), c);
  if ((threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(&D.ccount[c], __popc(peers));
}

__global__ void __launch_bounds__(REBUILD_CHUNK) k_bin(Dev D) {
  for_rebuild_atoms(D, [&](int s, long long i) { bin_atom(D, s, i); });
}

// One block per system: exclusive scan of the cell counts; resets counts and cursors.  A thread takes
// 16 consecutive cells as four 16-byte words (from the aligned word that holds the system's first
// cell on), so that a pass of the block covers 16,384 cells: the block's chain of load, scan and
// barriers, not bandwidth, is the time (4 cells a thread: 123 us for the 110,592 cells of a 2 M atom
// liquid, 63 so; 16 -> 9 us for 13,824).
constexpr int SCAN_CELLS = 16;
__device__ __forceinline__ void scan_cells(const Dev& D, int s) {
  const SysDev& S = D.sysd[s];
  const int cb = S.cell_base, ce = cb + S.ncells, a0 = cb & ~3;
  __shared__ int warp_tot[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int carry = (int)S.atom_base;  // global slots
  for (int base = a0; base < ce; base += 1024 * SCAN_CELLS) {
    const int c0 = base + threadIdx.x * SCAN_CELLS;
    int v[SCAN_CELLS];
    int sum = 0;
#pragma unroll
    for (int k = 0; k < SCAN_CELLS; k += 4) {
      const bool whole = c0 + k >= cb && c0 + k + 4 <= ce;
      int4 x = make_int4(0, 0, 0, 0);
      if (whole) {
        x = *reinterpret_cast<const int4*>(D.ccount + c0 + k);
      } else {
        if (c0 + k >= cb && c0 + k < ce) x.x = D.ccount[c0 + k];
        if (c0 + k + 1 >= cb && c0 + k + 1 < ce) x.y = D.ccount[c0 + k + 1];
        if (c0 + k + 2 >= cb && c0 + k + 2 < ce) x.z = D.ccount[c0 + k + 2];
        if (c0 + k + 3 >= cb && c0 + k + 3 < ce) x.w = D.ccount[c0 + k + 3];
      }
      v[k] = x.x;
      v[k + 1] = x.y;
      v[k + 2] = x.z;
      v[k + 3] = x.w;
      sum += (x.x + x.y) + (x.z + x.w);
    }
    int x = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[w] = x;
    __syncthreads();
    int t = warp_tot[lane];  // every warp scans the 32 totals for itself
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, t, o);
      if (lane >= o) t += y;
    }
    const int before = __shfl_sync(0xffffffffu, t, w > 0 ? w - 1 : 0);
    int excl = x - sum + (w > 0 ? before : 0) + carry;
    carry += __shfl_sync(0xffffffffu, t, 31);
#pragma unroll
    for (int k = 0; k < SCAN_CELLS; k += 4) {
      const int4 st = make_int4(excl, excl + v[k], excl + v[k] + v[k + 1], excl + v[k] + v[k + 1] + v[k + 2]);
      if (c0 + k >= cb && c0 + k + 4 <= ce) {
        *reinterpret_cast<int4*>(D.cstart + c0 + k) = st;
        *reinterpret_cast<int4*>(D.ccnt + c0 + k) = make_int4(v[k], v[k + 1], v[k + 2], v[k + 3]);
        *reinterpret_cast<int4*>(D.ccount + c0 + k) = make_int4(0, 0, 0, 0);
        *reinterpret_cast<int4*>(D.ccursor + c0 + k) = make_int4(0, 0, 0, 0);
      } else {
        const int start[4] = {st.x, st.y, st.z, st.w};
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c0 + k + q >= cb && c0 + k + q < ce) {
            D.cstart[c0 + k + q] = start[q];
            D.ccnt[c0 + k + q] = v[k + q];
            D.ccount[c0 + k + q] = 0;
            D.ccursor[c0 + k + q] = 0;
          }
      }
      excl += v[k] + v[k + 1] + v[k + 2] + v[k + 3];
    }
    __syncthreads();  // warp_tot is written again
  }
}
__global__ void __launch_bounds__(1024) k_scan(Dev D) {
  if (D.sst[blockIdx.x].need_rebuild) scan_cells(D, blockIdx.x);
}

// LCBinary::UpdateCell keeps at most one atom per sub-cell (plugins/lcbinary.cc:162-193): flags
// the systems whose re-sort put two atoms into one cell (their grid then grows by 2 per axis).
__global__ void k_binary_collide(Dev D) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= D.total_cells) return;
  const int s = D.cell_sys[g];
  if (!D.sysd[s].active || !D.sst[s].need_rebuild) return;
  if (D.ccnt[g] > 1) atomicOr(&D.sst[s].collide, 1);
}

__global__ void k_binary_clear(Dev D) {
  for (int s = threadIdx.x; s < D.nsys; s += blockDim.x) D.sst[s].collide = 0;
}

__device__ __forceinline__ void scatter_atom(const Dev& D, long long i) {
  const int c = D.acell[i];
  // the warp's atoms of one cell take consecutive slots from one atomic (their order inside
  // the cell is set by k_cellsort either way)
  const unsigned peers = __match_any_sync(__activemask(), c);
  const int lane = threadIdx.x & 31, lead = __ffs(peers) - 1;
  int first = 0;
  if (lane == lead) first = atomicAdd(&D.ccursor[c], __popc(peers));
  first = __shfl_sync(peers, first, lead);
  D.perm[D.cstart[c] + first + __popc(peers & ((1u << lane) - 1u))] = (int)i;
}

__global__ void __launch_bounds__(REBUILD_CHUNK) k_scatter(Dev D) {
  for_rebuild_atoms(D, [&](int, long long i) { scatter_atom(D, i); });
}

// One warp per cell of the rebuilding systems: orders the cell's slots by original index, the order in which LinkedCell's head/next lists
// visit them.  Each atom's rank is the number of smaller tags in its cell: up to 32 atoms the
// lanes compare through shuffles, up to SORT_STAGE atoms (dense cells of a liquid, coarse
// LinkedCell grids) through a copy of the cell's tags in shared memory, and beyond that through
// global scratch (n^2/32 compares per lane).
constexpr int SORT_WARPS = 4;    // cells per block
constexpr int SORT_STAGE = 256;  // atoms per cell ranked in shared memory
__device__ __forceinline__ void sort_cell(const Dev& D, int g, int* tg, int* ix) {
  const int lane = threadIdx.x & 31;
  const int b = D.cstart[g], n = D.ccnt[g];
  if (n <= 32) {
    int v = lane < n ? D.perm[b + lane] : 0;
    int tv = lane < n ? D.tag[v] : 0x7fffffff;
    int rank = 0;
    for (int k = 0; k < n; ++k) {
      int tk = __shfl_sync(0xffffffffu, tv, k);
      rank += (tk < tv) ? 1 : 0;
    }
    __syncwarp();
    if (lane < n) D.perm[b + rank] = v;
    return;
  }
  if (n <= SORT_STAGE) {
    for (int k = lane; k < n; k += 32) {
      const int v = D.perm[b + k];
      ix[k] = v;
      tg[k] = D.tag[v];
    }
    __syncwarp();  // every slot is read before any is rewritten
    for (int k = lane; k < n; k += 32) {
      const int t = tg[k];
      int rank = 0;
      for (int m = 0; m < n; ++m) rank += (tg[m] < t) ? 1 : 0;
      D.perm[b + rank] = ix[k];
    }
    return;
  }
  // larger cells: the same ranks through global scratch, the cell's own slots [b, b + n) of the
  // permutation staging (free until k_permute fills it)
  int* const tags = D.sint;
  int* const sorted = D.sint + D.N;
  for (int k = lane; k < n; k += 32) tags[b + k] = D.tag[D.perm[b + k]];
  __syncwarp();
  for (int k = lane; k < n; k += 32) {
    const int t = tags[b + k];
    int rank = 0;
    for (int m = 0; m < n; ++m) rank += (tags[b + m] < t) ? 1 : 0;
    sorted[b + rank] = D.perm[b + k];
  }
  __syncwarp();
  for (int k = lane; k < n; k += 32) D.perm[b + k] = sorted[b + k];
}
__global__ void __launch_bounds__(32 * SORT_WARPS) k_cellsort(Dev D) {
  __shared__ int s_tag[SORT_WARPS][SORT_STAGE];
  __shared__ int s_idx[SORT_WARPS][SORT_STAGE];
  const int w = threadIdx.x >> 5;
  int s, v;
  for (int u = blockIdx.x * SORT_WARPS + w; rebuild_unit<true>(D, u, s, v); u += gridDim.x * SORT_WARPS) {
    sort_cell(D, D.sysd[s].cell_base + v, s_tag[w], s_idx[w]);
    __syncwarp();
  }
}

__device__ __forceinline__ void permute_atom(const Dev& D, long long p) {
  const long long N = D.N;
  const int o = D.perm[p];
  double* sd = D.sdbl;
  sd[0 * N + p] = D.x[o];
  sd[1 * N + p] = D.y[o];
  sd[2 * N + p] = D.z[o];
  sd[3 * N + p] = D.vx[o];
  sd[4 * N + p] = D.vy[o];
  sd[5 * N + p] = D.vz[o];
  sd[6 * N + p] = D.ax[o];
  sd[7 * N + p] = D.ay[o];
  sd[8 * N + p] = D.az[o];
  sd[9 * N + p] = D.mass[o];
  sd[10 * N + p] = D.fm[o];
  int* si = D.sint;
  si[0 * N + p] = D.type[o];
  si[1 * N + p] = D.tag[o];
  si[2 * N + p] = D.acell[o];
  if (D.has_flags) D.sflags[p] = D.flags[o];
  if (D.ist)
    for (int k = 0; k < IST_K; ++k) D.ist_alt[k * N + p] = D.ist[k * N + o];
}

__global__ void __launch_bounds__(REBUILD_CHUNK) k_permute(Dev D) {
  for_rebuild_atoms(D, [&](int, long long i) { permute_atom(D, i); });
}

// Offset of x from the centre xc of its home cell, wrapped into [-L/2, L/2).  Two FP64-pipe
// operations on the common path (the FP64 unit is GB300's scarcest); the wrap is only taken
// for atoms far from their home cell (outside the box in the input).
__device__ __forceinline__ float home_offset(double x, double xc, double L, double Lh) {
  double o = x - xc;
  float of = (float)o;
  if (fabsf(of) >= 0.999f * (float)Lh) {
    if (o >= Lh) o = dsub(o, L);
    if (o < -Lh) o = dadd(o, L);
    of = (float)o;
  }
  return of;
}

// Gather copies of atom p at position (xx, yy, zz): the FP64 double4 (not by the mixed path's
// fused drift, WRITE64 = 0: no mixed kernel reads it, and a change of precision re-sorts, which
// rewrites it) and, for Verlet lists, the FP32 offset from the home-cell centre (returned, for
// displacement tracking).
template <int WRITE64 = 1>
__device__ __forceinline__ float4 write_gather(const Dev& D, const SysDev& S, long long p, double xx, double yy,
                                               double zz, int t, double4_32a* g64, float4* g32) {
  if (WRITE64) g64[p] = make_double4_32a(xx, yy, zz, (double)t);
  float4 g = make_float4(0.f, 0.f, 0.f, __int_as_float(t));
  if (S.mode == NB_LIST) {
    const double* c = D.ccentre + 3 * (long long)D.home[p];
    g = make_float4(home_offset(xx, c[0], S.L[0], S.Lh[0]), home_offset(yy, c[1], S.L[1], S.Lh[1]),
                    home_offset(zz, c[2], S.L[2], S.Lh[2]), __int_as_float(t));
    g32[p] = g;
  }
  return g;
}

__device__ __forceinline__ void refresh_gather(const Dev& D, const SysDev& S, long long p, bool set_ref) {
  float4 g = write_gather(D, S, p, D.x[p], D.y[p], D.z[p], D.type[p], D.g64, D.g32);
  if (set_ref && S.mode == NB_LIST) D.ref[p] = g;
}

// Squared displacement since the last list build (FP32 offsets, home cell unchanged).
__device__ __forceinline__ float displacement2(const Dev& D, long long p, float4 g) {
  float4 r = D.ref[p];
  float dx = g.x - r.x, dy = g.y - r.y, dz = g.z - r.z;
  return dx * dx + dy * dy + dz * dz;
}

// Largest displacement^2 of a warp whose lanes all belong to system s (whole tiles/blocks).
__device__ __forceinline__ void track_displacement_warp(const Dev& D, int s, float d2) {
  unsigned m = __reduce_max_sync(0xffffffffu, (unsigned)__float_as_int(d2));
  if ((threadIdx.x & 31) == 0 && m) atomicMax(&D.sst[s].maxdisp2, m);
}

__device__ __forceinline__ void copyback_atom(const Dev& D, int s, long long p) {
  const long long N = D.N;
  const double* sd = D.sdbl;
  D.x[p] = sd[0 * N + p];
  D.y[p] = sd[1 * N + p];
  D.z[p] = sd[2 * N + p];
  D.vx[p] = sd[3 * N + p];
  D.vy[p] = sd[4 * N + p];
  D.vz[p] = sd[5 * N + p];
  D.ax[p] = sd[6 * N + p];
  D.ay[p] = sd[7 * N + p];
  D.az[p] = sd[8 * N + p];
  D.mass[p] = sd[9 * N + p];
  D.fm[p] = sd[10 * N + p];
  const int* si = D.sint;
  D.type[p] = si[0 * N + p];
  D.tag[p] = si[1 * N + p];
  D.home[p] = si[2 * N + p];
  if (D.has_flags) D.flags[p] = D.sflags[p];
  if (D.ist)
    for (int k = 0; k < IST_K; ++k) D.ist[k * N + p] = D.ist_alt[k * N + p];
  const SysDev& S = D.sysd[s];
  // atoms that move are folded into the box before the next re-sort, those with a fixed position stay
  if (S.mode == NB_LIST && (outside_bits(D.x[p], S.L[0]) || outside_bits(D.y[p], S.L[1]) || outside_bits(D.z[p], S.L[2])))
    D.outside[s] = 1;
  refresh_gather(D, S, p, true);
}

__global__ void __launch_bounds__(REBUILD_CHUNK) k_copyback(Dev D) {
  for_rebuild_atoms(D, [&](int s, long long i) { copyback_atom(D, s, i); });
}

// ---------------------------------------------------------------------------------------------
// The same sort in one launch: a cluster of blocks per system goes through the phases above with
// the hardware's cluster barrier between them (release / acquire, so that each phase sees the others'
// writes to global memory).  Bound by latency: six phases on at most 8 SMs.  It replaces six launches
// when the system rebuilds, and when it does not it costs one empty launch, with which a graph step
// does without its conditional node.  Measured against the chain of kernels (conditional node
// included), us a step: single LJ liquids of 500 / 4,000 / 8,788 / 16,384 / 32,000 atoms 21.2 / 24.8 /
// 25.8 / 30.0 / 38.5 against 27.8 / 28.0 / 29.9 / 32.9 / 37.3; batches of 512 x 256 atoms 101 against
// 110, of 33 systems up to 4,000 87 against 77.  Cells cost as well: gases of 500 atoms on 8,000 cells
// 20.8 against 26.3, 2,000 on 32,768 32.9 / 32.3, 8,000 on 2,197 / 15,625 cells 31.0 / 34.2 against
// 31.0 / 32.8, 20,000 on 2,197 / 39,304 36.9 / 54.0 against 35.2 / 46.8 (with one cell a
// warp at a time and no line by cells 37.0, 115, 42.0 and 66.2, and 3,820 for 1,000 on 1.2 M: 240 so).
// ---------------------------------------------------------------------------------------------
constexpr int CLUSTER_ATOMS = 24000;       // a single system
constexpr int CLUSTER_ATOMS_BATCH = 2048;  // the largest system of a batch
constexpr int CLUSTER_CELLS = 4096;        // of a system on several blocks
constexpr int CLUSTER_CELLS_ONE = 32768;   // of a system on one
constexpr int CLUSTER_THREADS = 1024;
constexpr int CLUSTER_SORT_BYTES = CLUSTER_THREADS / 32 * 2 * SORT_STAGE * (int)sizeof(int);

// Blocks of a system's cluster (at most 8, the portable size): two or more atoms a thread.
inline int cluster_blocks(long long natoms) {
  int b = 1;
  while (b < 8 && (long long)b * 2 * CLUSTER_THREADS < natoms) b *= 2;
  return b;
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__global__ void __launch_bounds__(CLUSTER_THREADS, 1) k_sort_cluster(Dev D, int blocks) {
  extern __shared__ int stage[];  // SORT_STAGE tags and indices per warp
  const int s = blockIdx.x / blocks, rank = blockIdx.x % blocks;
  if (!D.sst[s].need_rebuild) return;  // the whole cluster
  const SysDev& S = D.sysd[s];
  const int n = S.natoms, t0 = rank * CLUSTER_THREADS + (int)threadIdx.x, step = blocks * CLUSTER_THREADS;
  for (int k = t0; k < n; k += step) bin_atom(D, s, S.atom_base + k);
  cluster_barrier();
  if (rank == 0) scan_cells(D, s);
  cluster_barrier();
  for (int k = t0; k < n; k += step) scatter_atom(D, S.atom_base + k);
  cluster_barrier();
  const int w = threadIdx.x >> 5;
  int* const mine = stage + w * 2 * SORT_STAGE;
  if (S.ncells <= step) {
    for (int c = rank * (CLUSTER_THREADS / 32) + w; c < S.ncells; c += blocks * (CLUSTER_THREADS / 32)) {
      sort_cell(D, S.cell_base + c, mine, mine + SORT_STAGE);
      __syncwarp();
    }
  } else {  // 32 cells at a time, of which most have one atom or none
    const int lane = threadIdx.x & 31;
    for (int c0 = (w * blocks + rank) * 32; c0 < S.ncells; c0 += step) {
      const int c = c0 + lane;
      for (unsigned todo = __ballot_sync(0xffffffffu, c < S.ncells && D.ccnt[S.cell_base + c] > 1); todo; todo &= todo - 1) {
        sort_cell(D, S.cell_base + c0 + __ffs(todo) - 1, mine, mine + SORT_STAGE);
        __syncwarp();
      }
    }
  }
  cluster_barrier();
  for (int k = t0; k < n; k += step) permute_atom(D, S.atom_base + k);
  cluster_barrier();
  for (int k = t0; k < n; k += step) copyback_atom(D, s, S.atom_base + k);
}

// ---------------------------------------------------------------------------------------------
// Verlet list with cell-shift codes
// ---------------------------------------------------------------------------------------------

__device__ __forceinline__ int shift_code(int kx, int ky, int kz) { return (kx + 2) + 5 * ((ky + 2) + 5 * (kz + 2)); }

// The Verlet list is built by one of two kernels, by the size of the system's grid: up to
// LIST_BLOCK_CELLS cells a block works on a home cell, above that a warp.  Both make the same list.
// A warp per cell needs fewer instructions an atom, but is a serial chain 27 cells long, which is
// all there is where the grid does not fill the GPU several times over, or where a few systems of a
// batch rebuild in a step; the block's chain is a quarter of that.  Measured (block / warp per cell):
// 729 cells (16,000 LJ atoms) 24 / 29 us, 1,728 (32,000) 31 / 30, 3,375 (54,000 of copper) 109 / 114,
// an ensemble of 128 systems 95 / 125 us a step; but 5,832 (32,000 of iron) 46 / 33, 13,824
// (495,000 of copper) 590 / 578, 97,336 (2 M LJ atoms) 1396 / 1092.
constexpr int LIST_BLOCK_CELLS = 4096;
constexpr int LIST_WARPS = 8;
constexpr int LIST_STAGE = 1024;
constexpr int LIST_STENCIL = 125;       // cells of the widest stencil (radius 2)
constexpr int LIST_ROWS_BYTES = 28672;  // shared memory of the rows (the rest is 20 KB)

// Home atoms whose rows fit in shared memory (0: none, entries then go straight to the list).
inline int list_batch(int maxnb) {
  const int n = LIST_ROWS_BYTES / ((maxnb + 4) * 4);
  return n > 32 ? 32 : n;
}

// The list's test of entry e of an atom at offset gi, in k_buildlist_warp's operation order.
__device__ __noinline__ bool list_pair(const SysDev& S, const float4& gi, const float4* g32, unsigned e) {
  const int code = (int)(e >> CODE_SHIFT);
  const float4 g = g32[e & LOCAL_MASK];
  const float ox = (float)(code % 5 - 2) * S.df[0] - gi.x, oy = (float)(code / 5 % 5 - 2) * S.df[1] - gi.y,
              oz = (float)(code / 25 - 2) * S.df[2] - gi.z;
  const float rx = ox + g.x, ry = oy + g.y, rz = oz + g.z;
  return fmaf(rx, rx, fmaf(ry, ry, rz * rz)) < S.rlist2f;
}

// One block per home cell.  The atoms of the stencil's cells are staged in shared memory as one
// run, LIST_STAGE at a time, each shifted by its cell's offset from the home cell and with its list
// entry beside it; each warp takes home atoms in turn and tests 64 candidates at a time (two a
// lane, in packed FP32 pairs), the hits' places in the atom's row by ballot.  The rows of `batch`
// home atoms are put together in shared memory and leave as whole 16-byte groups of neighbouring
// atoms (written straight to the list, the half-filled sectors cost more than the tests).
// (A pair so close to the list radius that the staged sums' rounding could decide it, by at most
// 4e-6 rl^2, sends its atom through the same loop once more with k_buildlist_warp's operation order,
// one atom in a few hundred: so the lists are the same.)
// ROWS: `batch` rows are put together in shared memory; else the entries go straight to the list.
template <bool ROWS>
__global__ void __launch_bounds__(32 * LIST_WARPS, 4) k_buildlist_block(Dev D, int batch) {
  extern __shared__ __align__(16) unsigned rows[];  // batch rows of maxnb + 4 words
  __shared__ __align__(16) float cx[LIST_STAGE], cy[LIST_STAGE], cz[LIST_STAGE];
  __shared__ __align__(16) unsigned ce[LIST_STAGE];
  __shared__ float4 c_shift[LIST_STENCIL];  // offset of the stencil cell, and its entries' code bits
  __shared__ int c_first[LIST_STENCIL];     // its first atom (index within the system)
  __shared__ int c_off[LIST_STENCIL + 4];   // running total of the atoms of the cells before it
  __shared__ int count[32];                 // entries of the batch's atoms
  const unsigned all = 0xffffffffu;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  const int maxnb = D.maxnb, rs = maxnb + 4, nbatch = ROWS ? batch : 32;
  int s, c;
  for (int u = blockIdx.x; rebuild_unit<true>(D, u, s, c); u += gridDim.x) {
    const SysDev& S = D.sysd[s];
    const int cell_base = S.cell_base;
    const int n0 = D.ccnt[cell_base + c];
    if (S.mode != NB_LIST || S.ncells > LIST_BLOCK_CELLS || n0 == 0) continue;
    const long long atom_base = S.atom_base;
    const int b0 = (int)(D.cstart[cell_base + c] - atom_base);
    const int R = S.stencil_r, W = 2 * R + 1, nst = W * W * W;
    const int nx = S.n[0], ny = S.n[1], nz = S.n[2];
    for (int t = threadIdx.x; t < nst; t += blockDim.x) {
      const int dx = t % W - R, dy = (t / W) % W - R, dz = t / (W * W) - R;
      const int xc = wrap_around(c % nx + dx, nx), yc = wrap_around((c / nx) % ny + dy, ny),
                zc = wrap_around(c / (nx * ny) + dz, nz);
      const int g = cell_base + (zc * ny + yc) * nx + xc;
      c_first[t] = (int)(D.cstart[g] - atom_base);
      c_off[t + 1] = D.ccnt[g];
      c_shift[t] = make_float4((float)dx * S.df[0], (float)dy * S.df[1], (float)dz * S.df[2],
                               __uint_as_float((unsigned)shift_code(dx, dy, dz) << CODE_SHIFT));
    }
    __syncthreads();
    if (w == 0) {  // exclusive running totals, four cells a lane
      int v[4], sum = 0;
      for (int k = 0; k < 4; ++k) {
        v[k] = 4 * lane + k < nst ? c_off[4 * lane + k + 1] : 0;
        sum += v[k];
      }
      int x = sum;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(all, x, o);
        if (lane >= o) x += y;
      }
      x -= sum;
      __syncwarp();
      for (int k = 0; k < 4; ++k) {
        if (4 * lane + k <= nst) c_off[4 * lane + k] = x;
        x += v[k];
      }
    }
    __syncthreads();
    const int total = c_off[nst];
    const float4* __restrict__ g32 = D.g32 + atom_base;
    unsigned* const nl = D.nl + S.nl_base;
    const long long na = S.natoms;
    const float rl2 = S.rlist2f;
    const float tol = 1e-5f * rl2;
    int most = 0, staged = -1;
    for (int a0 = 0; a0 < n0; a0 += nbatch) {
      const int nb = min(nbatch, n0 - a0);
      if ((int)threadIdx.x < nb) count[threadIdx.x] = 0;
      for (int w0 = 0; w0 < total; w0 += LIST_STAGE) {
        const int m = min(LIST_STAGE, total - w0), mp = (m + 63) & ~63;
        if (staged != w0) {
          for (int t = w; t < nst; t += LIST_WARPS) {
            const int n = c_off[t + 1] - c_off[t], p0 = c_off[t] - w0, first = c_first[t];
            const float4 sh = c_shift[t];
            for (int k = lane; k < n; k += 32)
              if (p0 + k >= 0 && p0 + k < LIST_STAGE) {
                const float4 g = g32[first + k];
                cx[p0 + k] = g.x + sh.x;
                cy[p0 + k] = g.y + sh.y;
                cz[p0 + k] = g.z + sh.z;
                ce[p0 + k] = __float_as_uint(sh.w) | (unsigned)(first + k);
              }
          }
          // far-away sentinels fill the last 64 (r^2 ~ 1e36 never hits)
          for (int k = m + (int)threadIdx.x; k < mp; k += blockDim.x) {
            cx[k] = 1e18f;
            cy[k] = cz[k] = 0.0f;
            ce[k] = 0u;
          }
          staged = w0;
        }
        __syncthreads();
        for (int a = w; a < nb; a += LIST_WARPS) {
          const int li = b0 + a0 + a;
          const float4 gi = g32[li];
          const f32x2 gx = f2_pack(gi.x, gi.x), gy = f2_pack(gi.y, gi.y), gz = f2_pack(gi.z, gi.z),
                      out2 = f2_pack(-rl2, -rl2);
          const unsigned self = ((unsigned)shift_code(0, 0, 0) << CODE_SHIFT) | (unsigned)li;
          unsigned* const row = rows + a * rs;
          const int cnt0 = count[a];
          int cnt = 0;
          bool near = false;
          auto scan = [&](auto exact) {
            cnt = cnt0;
            int k = 2 * lane;
            unsigned h0, h1;
            bool in0, in1;
            uint2 e;
            auto test = [&]() {
              e = *reinterpret_cast<const uint2*>(ce + k);
              if (decltype(exact)::value) {
                in0 = k < m && list_pair(S, gi, g32, e.x);
                in1 = k + 1 < m && list_pair(S, gi, g32, e.y);
              } else {
                const float2 X = *reinterpret_cast<const float2*>(cx + k), Y = *reinterpret_cast<const float2*>(cy + k),
                             Z = *reinterpret_cast<const float2*>(cz + k);
                const f32x2 rx = f2_sub(f2_pack(X.x, X.y), gx), ry = f2_sub(f2_pack(Y.x, Y.y), gy),
                            rz = f2_sub(f2_pack(Z.x, Z.y), gz);
                float d0, d1;  // r^2 - rl^2
                f2_unpack(f2_fma(rx, rx, f2_fma(ry, ry, f2_fma(rz, rz, out2))), d0, d1);
                in0 = d0 < 0.0f;
                in1 = d1 < 0.0f;
                near = near || fminf(fabsf(d0), fabsf(d1)) < tol;
              }
              in0 = in0 && e.x != self;
              in1 = in1 && e.y != self;
              h0 = __ballot_sync(all, in0);
              h1 = __ballot_sync(all, in1);
            };
            if (ROWS) {
              // while 64 more entries surely fit
              const int room = maxnb - 64;
              for (; k < mp && cnt <= room; k += 64) {
                test();
                unsigned* at = row + (cnt + __popc(h0 & below) + __popc(h1 & below));
                if (in0) *at++ = e.x;
                if (in1) *at = e.y;
                cnt += __popc(h0) + __popc(h1);
              }
            }
            for (; k < mp; k += 64) {
              test();
              int p = cnt + __popc(h0 & below) + __popc(h1 & below);
              auto put = [&](unsigned v) {
                if (p < maxnb) {
                  if (ROWS)
                    row[p] = v;
                  else
                    nl[((long long)(p >> 2) * na + li) * 4 + (p & 3)] = v;
                }
                ++p;
              };
              if (in0) put(e.x);
              if (in1) put(e.y);
              cnt += __popc(h0) + __popc(h1);
            }
          };
          scan(std::false_type());
          if (__any_sync(all, near)) scan(std::true_type());
          __syncwarp();  // every lane has read the atom's count
          if (lane == 0) count[a] = cnt;
        }
        __syncthreads();
      }
      // lane = atom of the batch, warps over the groups of four; words past the end are written as
      // entry 0, which the force passes may load but do not count
      const int cnt = lane < nb ? count[lane] : 0;
      const int kept = min(cnt, maxnb);
      most = max(most, cnt);
      if (ROWS) {
        const int ng = (int)__reduce_max_sync(all, (unsigned)(kept + 3) >> 2);
        for (int q = w; q < ng; q += LIST_WARPS)
          if (4 * q < kept) {
            uint4 v = *reinterpret_cast<const uint4*>(rows + lane * rs + 4 * q);
            const int left = kept - 4 * q;
            if (left < 2) v.y = 0u;
            if (left < 3) v.z = 0u;
            if (left < 4) v.w = 0u;
            reinterpret_cast<uint4*>(nl)[q * na + b0 + a0 + lane] = v;
          }
      }
      if (w == 0 && lane < nb) D.ncount[atom_base + b0 + a0 + lane] = kept;
      __syncthreads();
    }
    if (w == 0) {
      most = (int)__reduce_max_sync(all, (unsigned)most);
      if (lane == 0) {
        if (most > *(volatile int*)&D.sst[s].max_count) atomicMax(&D.sst[s].max_count, most);
        if (most > maxnb) atomicOr(&D.sst[s].error, ERR_LIST);
      }
    }
  }
}

// The atoms of home cell c of system S, up to 32 at a time a lane each: the atoms of each stencil
// cell are staged through shared memory 32 at a time; every lane then tests the staged candidates
// against its own atom (broadcast reads, no divergence between lanes, since all atoms of a cell share
// the stencil and its cell-shift codes; the sign of r^2 - rl^2 shifts into a mask), and appends its
// hits in candidate order.  Bound by instruction issue (64 %, the integer unit 60 %), half of it
// tests and half the appending, with latency behind.  The lanes look the stencil's cells up together,
// and the next candidates are loaded while the last are tested; with 72 registers seven blocks fit
// an SM.  Measured, a cell looked up at a time with its own load / this at 4 / 7 / 8 blocks an SM:
// 2,048,000 LJ atoms 1167 / 1173 / 1092 / 1130 us, 107,963 75 / 72 / 69 / 74, 32,000 of iron
// 40 / 34 / 33 / 37, 495,000 of copper 578 / 574 / 578 / 605.  (A group of four entries gathered
// in registers and written as 16 bytes instead of an entry at a time: 1272 us for 2,048,000.)
constexpr int LIST_CELLS = 4;  // home cells (warps) of a block
// A warp's shared memory: the staged candidates' coordinates as three arrays, so that one 16-byte
// load gives the x (y, z) of four consecutive candidates (two packed pairs), and up to 32 cells of
// the stencil: first atom (index within the system) and atoms, offset from the home cell and code bits.
struct ListStage {
  float x[32], y[32], z[32];
  float4 shift[32];
  int2 run[32];
};
__device__ __forceinline__ void list_cell(const Dev& D, const SysDev& S, int s, int c, ListStage& st) {
  const int lane = threadIdx.x & 31;
  // the system's grid in registers: the list stores below may alias any global memory, so
  // fields read through the SysDev reference would be re-read after every store
  const int nx = S.n[0], ny = S.n[1], nz = S.n[2];
  const float dfx = S.df[0], dfy = S.df[1], dfz = S.df[2];
  const int cell_base = S.cell_base;
  const long long atom_base = S.atom_base;
  const float rlist2 = S.rlist2f;
  const int R = S.stencil_r;
  const int na = S.natoms;
  unsigned* const nl = D.nl + S.nl_base;
  const int* __restrict__ cstart = D.cstart;
  const int* __restrict__ ccnt = D.ccnt;
  const float4* __restrict__ g32 = D.g32 + atom_base;
  const int maxnb = D.maxnb;
  const int W = 2 * R + 1, nst = W * W * W;
  const int b0 = cstart[cell_base + c], n0 = ccnt[cell_base + c];
  const int cx = c % nx, cy = (c / nx) % ny, cz = c / (nx * ny);
  int most = 0;
  for (int base = 0; base < n0; base += 32) {
    const bool has = base + lane < n0;
    const long long i = (long long)b0 + base + lane;
    const int li = (int)(i - atom_base);
    const float4 gi = has ? g32[li] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float out = has ? -rlist2 : 1.0f;  // lanes without an atom never match
    const f32x2 out2 = f2_pack(out, out);
    const long long gstride = (long long)na * 4;  // words between consecutive groups of four
    int cnt = 0;
    unsigned* wp = nl + (long long)li * 4;
    for (int t0 = 0; t0 < nst; t0 += 32) {
      __syncwarp();
      if (t0 + lane < nst) {
        const int t = t0 + lane, dx = t % W - R, dy = (t / W) % W - R, dz = t / (W * W) - R;
        const int xc = wrap_around(cx + dx, nx), yc = wrap_around(cy + dy, ny), zc = wrap_around(cz + dz, nz);
        const int g = cell_base + (zc * ny + yc) * nx + xc;
        st.run[lane] = make_int2((int)(cstart[g] - atom_base), ccnt[g]);
        st.shift[lane] = make_float4((float)dx * dfx, (float)dy * dfy, (float)dz * dfz,
                                     __uint_as_float((unsigned)shift_code(dx, dy, dz) << CODE_SHIFT));
      }
      __syncwarp();
      const int cells = min(32, nst - t0);
      // the next 32 candidates (of one cell) on their way while the last are tested
      int t = -1, from = 0, left = 0;
      float4 gj;
      auto fetch = [&]() -> bool {
        while (left <= 0) {
          if (++t >= cells) return false;
          const int2 run = st.run[t];
          from = run.x;
          left = run.y;
        }
        gj = lane < left ? g32[from + lane] : make_float4(1e18f, 1e18f, 1e18f, 0.f);
        return true;
      };
      for (bool more = fetch(); more;) {
        __syncwarp();
        st.x[lane] = gj.x;
        st.y[lane] = gj.y;
        st.z[lane] = gj.z;
        __syncwarp();
        const int m = min(32, left), jl0 = from;
        const float4 sh = st.shift[t];
        const unsigned code = __float_as_uint(sh.w);
        from += 32;
        left -= 32;
        more = fetch();
        const float ox = sh.x - gi.x, oy = sh.y - gi.y, oz = sh.z - gi.z;
        const f32x2 ox2 = f2_pack(ox, ox), oy2 = f2_pack(oy, oy), oz2 = f2_pack(oz, oz);
        // pass 1: a bit per staged candidate inside the list radius (branch-free), candidate k
        // in bit 31 - k
        unsigned hits = 0u;
        for (int k = 0; k < m; k += 4) {
          // candidates k..k+3 as two packed pairs
          const float4 X = *reinterpret_cast<const float4*>(st.x + k);
          const float4 Y = *reinterpret_cast<const float4*>(st.y + k);
          const float4 Z = *reinterpret_cast<const float4*>(st.z + k);
          const f32x2 rx01 = f2_add(ox2, f2_pack(X.x, X.y)), rx23 = f2_add(ox2, f2_pack(X.z, X.w));
          const f32x2 ry01 = f2_add(oy2, f2_pack(Y.x, Y.y)), ry23 = f2_add(oy2, f2_pack(Y.z, Y.w));
          const f32x2 rz01 = f2_add(oz2, f2_pack(Z.x, Z.y)), rz23 = f2_add(oz2, f2_pack(Z.z, Z.w));
          const f32x2 q01 = f2_fma(rx01, rx01, f2_fma(ry01, ry01, f2_mul(rz01, rz01)));
          const f32x2 q23 = f2_fma(rx23, rx23, f2_fma(ry23, ry23, f2_mul(rz23, rz23)));
          float d0, d1, d2, d3;  // r^2 - rl^2, whose sign no rounding changes
          f2_unpack(f2_add(q01, out2), d0, d1);
          f2_unpack(f2_add(q23, out2), d2, d3);
          hits = __funnelshift_l(__float_as_uint(d0), hits, 1);
          hits = __funnelshift_l(__float_as_uint(d1), hits, 1);
          hits = __funnelshift_l(__float_as_uint(d2), hits, 1);
          hits = __funnelshift_l(__float_as_uint(d3), hits, 1);
        }
        hits <<= 32 - ((m + 3) & ~3);
        const int self = li - jl0;  // drop the atom itself
        if (self >= 0 && self < 32) hits &= ~(0x80000000u >> self);
        // pass 2: append the hits in candidate order
        while (hits) {
          const int k = __clz(hits);
          hits ^= 0x80000000u >> k;
          // running write position: entry cnt of the atom lives at group cnt/4, slot cnt%4
          if (cnt < maxnb) *wp = code | (unsigned)(jl0 + k);
          wp += (cnt & 3) == 3 ? gstride - 3 : 1;
          ++cnt;
        }
      }
    }
    if (has) {
      D.ncount[i] = cnt < maxnb ? cnt : maxnb;
      most = max(most, cnt);
    }
  }
  most = (int)__reduce_max_sync(0xffffffffu, (unsigned)most);
  if (lane == 0) {
    if (most > *(volatile int*)&D.sst[s].max_count) atomicMax(&D.sst[s].max_count, most);
    if (most > maxnb) atomicOr(&D.sst[s].error, ERR_LIST);
  }
}

__global__ void __launch_bounds__(32 * LIST_CELLS, 7) k_buildlist_warp(Dev D) {
  __shared__ __align__(16) ListStage stage[LIST_CELLS];
  const int w = threadIdx.x >> 5;
  int s, c;
  for (int u = blockIdx.x * LIST_CELLS + w; rebuild_unit<true>(D, u, s, c); u += gridDim.x * LIST_CELLS)
    if (D.sysd[s].mode == NB_LIST && D.sysd[s].ncells > LIST_BLOCK_CELLS)
      list_cell(D, D.sysd[s], s, c, stage[w]);
}

// ---------------------------------------------------------------------------------------------
// Integration: drift half of velocity Verlet
// ---------------------------------------------------------------------------------------------

// Velocity rescaling between steps.  The temperature is measured afresh, as the modifiers do:
// k_kinetic_clear + k_scale_kinetic sum the kinetic energy of the current velocities into the
// system's int64 kinetic slot (2^-44 units; each warp's FP64 sum rounded once, so the total is
// order-independent), then k_scale_velocities scales.
//   mode 0, SimulationBuilder::SetTemperature (liblpmd/simulation/simulationbuilder.cc:53-72,
//     called by plugins/tempscaling.cc:66-71 and plugins/temperature.cc:58-62 with tag = "any
//     atom has fixedvel/fixedpos"): T over the untagged atoms, tagged atoms keep their velocity,
//     v *= sqrt(target / T);
//   mode 1, BerendsenModifier::Apply (plugins/berendsen.cc:72-99): T over all atoms
//     (lpmd::Temperature with tag false, liblpmd/lpmd/properties.h:40-53), every atom scaled by
//     sqrt(1 + dt/tau * (target / T - 1)).
// The kinetic slot is free between steps: the next force evaluation's decision clears it.
// A system at T = 0 is left as it is (the reference would divide by zero).
__global__ void k_kinetic_clear(Dev D) {
  for (int s = threadIdx.x; s < D.nsys; s += blockDim.x) D.sys_acc[(long long)s * SA_LEN + SA_KE] = 0ull;
}

__global__ void __launch_bounds__(TILE) k_scale_kinetic(Dev D, int sys, int mode) {
  const int tile = blockIdx.x;
  const int s = D.tile_sys[tile];
  if ((sys >= 0 && s != sys) || !D.sysd[s].active) return;  // whole block: one tile, one system
  const long long i = D.tile_first[tile] + threadIdx.x;
  double ke = 0.0;
  if ((int)threadIdx.x < D.tile_count[tile] &&
      !(mode == 0 && D.has_flags && (D.flags[i] & (FLAG_FIXEDVEL | FLAG_FIXEDPOS)))) {
    const double vx = D.vx[i], vy = D.vy[i], vz = D.vz[i];
    ke = dmul(dmul(0.5, D.mass[i]), ref_sq(vx, vy, vz));
  }
  const double kw = warp_sum(ke);
  __shared__ long long part[TILE / 32];
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = __double2ll_rn(kw * FIX_KE);
  __syncthreads();
  if (threadIdx.x == 0) {
    long long t = 0;
    for (int w = 0; w < TILE / 32; ++w) t += part[w];
    atomicAdd(D.sys_acc + (long long)s * SA_LEN + SA_KE, (unsigned long long)t);
  }
}

__global__ void k_scale_velocities(Dev D, int sys, int mode, double target, double dt_over_tau) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= D.N) return;
  const int s = D.sysid[i];
  const SysDev& S = D.sysd[s];
  if ((sys >= 0 && s != sys) || !S.active) return;
  const double KIN2EV = 103.64269, KBOLTZMANN = 8.6173422E-05;  // liblpmd/lpmd/properties.h:10-11
  const double ke = (double)(long long)__ldcg(D.sys_acc + (long long)s * SA_LEN + SA_KE) * (1.0 / FIX_KE);
  const double kbn = mode == 0 ? S.kbn : dmul(KBOLTZMANN, (double)S.natoms);
  const double T = ddiv(dmul(2.0 / 3.0, dmul(ke, KIN2EV)), kbn);
  if (!(T > 0.0)) return;
  if (mode == 0 && D.has_flags && (D.flags[i] & (FLAG_FIXEDVEL | FLAG_FIXEDPOS))) return;
  const double f = mode == 0 ? sqrt(ddiv(target, T)) : sqrt(dadd(1.0, dmul(dt_over_tau, dsub(ddiv(target, T), 1.0))));
  D.vx[i] = dmul(D.vx[i], f);
  D.vy[i] = dmul(D.vy[i], f);
  D.vz[i] = dmul(D.vz[i], f);
}

// Centre of every Verlet-list cell: ((c + 1/2) * d) per axis, FP64.
__global__ void k_cell_centres(Dev D) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= D.total_cells) return;
  const SysDev& S = D.sysd[D.cell_sys[g]];
  const int c = g - S.cell_base;
  const int cx = c % S.n[0], cy = (c / S.n[0]) % S.n[1], cz = c / (S.n[0] * S.n[1]);
  D.ccentre[3 * (long long)g] = fma((double)cx, S.d[0], 0.5 * S.d[0]);
  D.ccentre[3 * (long long)g + 1] = fma((double)cy, S.d[1], 0.5 * S.d[1]);
  D.ccentre[3 * (long long)g + 2] = fma((double)cz, S.d[2], 0.5 * S.d[2]);
}

// VelocityVerlet::AdvancePosition of atom i from the evaluation buffer into the output buffer:
// newpos = x + v*dt + 0.5*a*dt*dt, then FittedInside.  The FP64 path rounds every product and
// sum separately as the reference does; the mixed path uses two FP64 fused multiply-adds per
// coordinate.  Returns the squared displacement since the last list build.
template <int MIXED>
__device__ __forceinline__ float drift_atom(const Dev& D, const SysDev& S, long long i, double dt, double h2,
                                            double vx, double vy, double vz, double ax, double ay, double az) {
  double nx = D.x[i], ny = D.y[i], nz = D.z[i];
  if (!(D.has_flags && (D.flags[i] & FLAG_FIXEDPOS))) {
    if (MIXED) {  // h2 = 0.5 * dt * dt
      nx = fma(h2, ax, fma(dt, vx, nx));
      ny = fma(h2, ay, fma(dt, vy, ny));
      nz = fma(h2, az, fma(dt, vz, nz));
    } else {
      nx = dadd(dadd(nx, dmul(vx, dt)), dmul(dmul(dmul(0.5, ax), dt), dt));
      ny = dadd(dadd(ny, dmul(vy, dt)), dmul(dmul(dmul(0.5, ay), dt), dt));
      nz = dadd(dadd(nz, dmul(vz, dt)), dmul(dmul(dmul(0.5, az), dt), dt));
    }
    nx = ref_fitted(nx, S.L[0]);
    ny = ref_fitted(ny, S.L[1]);
    nz = ref_fitted(nz, S.L[2]);
  }
  D.xo[i] = nx;
  D.yo[i] = ny;
  D.zo[i] = nz;
  float4 g = write_gather<!MIXED>(D, S, i, nx, ny, nz, D.type[i], D.g64o, D.g32o);
  return S.mode == NB_LIST ? displacement2(D, i, g) : 0.0f;
}

// Keeps an inactive system's committed positions in place across a launch that writes the
// other position buffer.  A fused force+drift launch reads the pending buffer (x) and writes
// the committed one (xo), after which the buffers swap roles: copy xo -> x (to_read = true).
// A stand-alone drift reads the committed buffer (x) and writes the pending one (xo): copy
// x -> xo (to_read = false).
__device__ __forceinline__ void hold_range(const Dev& D, const SysDev& S, int first, int count, bool to_read) {
  if ((int)threadIdx.x >= count) return;
  const long long i = first + threadIdx.x;
  if (to_read) {
    D.x[i] = D.xo[i];
    D.y[i] = D.yo[i];
    D.z[i] = D.zo[i];
    D.g64[i] = D.g64o[i];
    if (S.mode == NB_LIST) D.g32[i] = D.g32o[i];
  } else {
    D.xo[i] = D.x[i];
    D.yo[i] = D.y[i];
    D.zo[i] = D.z[i];
    D.g64o[i] = D.g64[i];
    if (S.mode == NB_LIST) D.g32o[i] = D.g32[i];
  }
}
__device__ __forceinline__ void hold_tile(const Dev& D, const SysDev& S, int tile, bool to_read) {
  hold_range(D, S, D.tile_first[tile], D.tile_count[tile], to_read);
}

// Stand-alone drift (the first step of a run, before any fused force/drift launch).
template <int MIXED>
__global__ void __launch_bounds__(TILE) k_drift(Dev D, double dt, double h2) {
  const int tile = blockIdx.x;
  const int s = D.tile_sys[tile];
  const SysDev& S = D.sysd[s];
  if (!S.active) {
    hold_tile(D, S, tile, false);
    return;
  }
  const long long i = D.tile_first[tile] + threadIdx.x;
  float d2 = 0.0f;
  if ((int)threadIdx.x < D.tile_count[tile])
    d2 = drift_atom<MIXED>(D, S, i, dt, h2, D.vx[i], D.vy[i], D.vz[i], D.ax[i], D.ay[i], D.az[i]);
  track_displacement_warp(D, s, d2);
}

}  // namespace gbmd
