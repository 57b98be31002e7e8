// forces.cuh -- mixed-precision force and density kernels, and the thermo kernels of both precisions.
// A block works on atoms of one system, an atom has one lane or several; every atom gathers over its
// full neighbour list, so forces need no atomics.  Sums over a system are int64 fixed point (mixed) or
// have a fixed order (FP64).
//
//   k_eam_density32  MetalPotential rho pass + embedding (liblpmd/simulation/metalpotential.cc:118-132,168)
//   k_force32        PairPotential::UpdateForces (liblpmd/simulation/pairpotential.cc:35-84) or
//                    MetalPotential's force pass (liblpmd/simulation/metalpotential.cc:137-169), with
//                    VelocityVerlet::AdvanceVelocity (plugins/velocityverlet.cc:70-75), the next step's
//                    drift and the thermo sums
//   ..._lanes        the same with several lanes an atom
//   k_tail, k_thermo thermo record (SetSimulationTags, liblpmd/simulation/simulationbuilder.cc:84-124) and
//                    the next step's rebuild decision
#pragma once

#include "kernels.cuh"

namespace gbmd {

enum PotClass { PC_PAIR = 0, PC_EAM = 1 };


// Visits the candidate neighbours j of atom i under neighbour mode NB (compile-time).
template <int NB, class F>
__device__ __forceinline__ void for_each_candidate(const Dev& D, const SysDev& S, long long i, F&& f) {
  if (NB == NB_LIST) {
    const int na = S.natoms;
    const uint4* L = list_group(D, S, (int)(i - S.atom_base), 0);
    const int cnt = D.ncount[i];
    for (int k = 0; k < cnt; k += 4) {
      const uint4 e4 = __ldg(L);
      L += na;
      const unsigned e[4] = {e4.x, e4.y, e4.z, e4.w};
      for (int u = 0; u < 4 && k + u < cnt; ++u) f(S.atom_base + (long long)(e[u] & LOCAL_MASK), e[u] >> CODE_SHIFT);
    }
  } else if (NB == NB_CELLS) {
    // The reference stencil of LinkedCell (plugins/linkedcell.cc:221-240), duplicates included.
    const int h = D.home[i] - S.cell_base;
    const int cx = h % S.n[0], cy = (h / S.n[0]) % S.n[1], cz = h / (S.n[0] * S.n[1]);
    const int sd = S.lc_side;
    for (int dz = -sd; dz <= sd; ++dz) {
      int zc = wrap_around(cz + dz, S.n[2]);
      for (int dy = -sd; dy <= sd; ++dy) {
        int yc = wrap_around(cy + dy, S.n[1]);
        for (int dx = -sd; dx <= sd; ++dx) {
          int xc = wrap_around(cx + dx, S.n[0]);
          int g = S.cell_base + (zc * S.n[1] + yc) * S.n[0] + xc;
          int b = D.cstart[g], e = b + D.ccnt[g];
          for (int j = b; j < e; ++j)
            if (j != i) f((long long)j, 0u);
        }
      }
    }
  } else {
    for (long long j = S.atom_base; j < S.atom_base + S.natoms; ++j)
      if (j != i) f(j, 0u);
  }
}

// Exact FP64 reference cutoff test of pair (i, j) from the master positions.
__device__ __forceinline__ bool exact_inside(const Dev& D, const SysDev& S, long long i, long long j, double rc2) {
  double dx = ref_wrap(dsub(D.x[j], D.x[i]), S.L[0], S.Lh[0]);
  double dy = ref_wrap(dsub(D.y[j], D.y[i]), S.L[1], S.Lh[1]);
  double dz = ref_wrap(dsub(D.z[j], D.z[i]), S.L[2], S.Lh[2]);
  return ref_sq(dx, dy, dz) < rc2;
}

// Out-of-line copy for the hot loops: the guard-band recheck is rare (a few pairs per thousand
// atoms), and keeping its FP64 code out of the loop body keeps the body small.
__device__ __noinline__ bool exact_inside_cold(const Dev* D, const SysDev* S, long long i, long long j, double rc2) {
  return exact_inside(*D, *S, i, j, rc2);
}

// The cell-shift table (k * cell edge, k in -2..2 per axis) of a block in shared memory, an array
// per axis: a 4-byte word a lane takes one pass of the shared-memory port for most code patterns
// (a code's bank is code mod 32), the 16 bytes of a float4 a lane at least four, and that port,
// which the neighbour gathers use too, is what the mixed passes wait for most (80 % busy at
// 2,048,000 atoms).  Measured, float4 / float2 + float / three floats: LJ forces of 2,048,000
// atoms 526 / 520 / 511 us, of 128 systems of 6,400 atoms 226 / 222 / 218; 495,000 copper atoms'
// forces 254 / 248 / 246 us, densities 159 / 152 / 147.
template <int N = 125>
struct ShiftTable {
  float x[N], y[N], z[N];
  __device__ __forceinline__ float4 operator[](unsigned code) const {
    return make_float4(x[code], y[code], z[code], 0.f);
  }
};

// Fills the table for system S (whole block).
__device__ __forceinline__ void load_shifts(const SysDev& S, ShiftTable<>& sh) {
  for (int c = threadIdx.x; c < 125; c += blockDim.x) {
    int kx = c % 5 - 2, ky = (c / 5) % 5 - 2, kz = c / 25 - 2;
    sh.x[c] = (float)kx * S.df[0];
    sh.y[c] = (float)ky * S.df[1];
    sh.z[c] = (float)kz * S.df[2];
  }
  __syncthreads();
}

// Epilogue shared by the force kernels: turns the total force on atom i into its acceleration
// (a = F * forcefactor/m, liblpmd/simulation/pairpotential.cc:62), applies fixedvel, and unless
// EPI_FORCES advances the velocity: v = v + (0.5*dt) * (a_old + a) (plugins/velocityverlet.cc:73-74).
// EPI_KICK_DRIFT then also advances the position for the next step (AdvancePosition) into the
// output position buffer.  Returns the kinetic terms of the updated velocity and the squared
// displacement since the last list build.
template <int MIXED>
__device__ __forceinline__ float finish_atom(const Dev& D, const SysDev& S, long long i, double Fx, double Fy,
                                             double Fz, const StepParams& sp, double& ke, double& px, double& py,
                                             double& pz) {
  // mixed: F arrives in 2^-32 eV/A units; scaling fm by the power of two is exact and gives
  // the same products as scaling F
  const double fm = MIXED ? D.fm[i] * (1.0 / FIX_F) : D.fm[i];
  double ax = dmul(Fx, fm), ay = dmul(Fy, fm), az = dmul(Fz, fm);
  unsigned char fl = D.has_flags ? D.flags[i] : 0;
  if ((fl & FLAG_FIXEDVEL) && !sp.raw_acc) ax = ay = az = 0.0;
  double vx = D.vx[i], vy = D.vy[i], vz = D.vz[i];
  if (sp.epi != EPI_FORCES && !(fl & FLAG_FIXEDPOS)) {
    if (MIXED) {
      vx = fma(sp.half_dt, D.ax[i] + ax, vx);
      vy = fma(sp.half_dt, D.ay[i] + ay, vy);
      vz = fma(sp.half_dt, D.az[i] + az, vz);
    } else {
      vx = dadd(vx, dmul(sp.half_dt, dadd(D.ax[i], ax)));
      vy = dadd(vy, dmul(sp.half_dt, dadd(D.ay[i], ay)));
      vz = dadd(vz, dmul(sp.half_dt, dadd(D.az[i], az)));
    }
    D.vx[i] = vx;
    D.vy[i] = vy;
    D.vz[i] = vz;
  }
  D.ax[i] = ax;
  D.ay[i] = ay;
  D.az[i] = az;
  ke = 0.0;
  px = py = pz = 0.0;
  // KineticEnergy/Momentum skip tagged atoms (liblpmd/lpmd/properties.h:22-37,64-81)
  if (sp.kinetic && !(fl & (FLAG_FIXEDVEL | FLAG_FIXEDPOS))) {
    const double m = D.mass[i];
    ke = MIXED ? (0.5 * m) * fma(vx, vx, fma(vy, vy, vz * vz)) : dmul(dmul(0.5, m), ref_sq(vx, vy, vz));
    px = dmul(vx, m);
    py = dmul(vy, m);
    pz = dmul(vz, m);
  }
  if (sp.epi == EPI_KICK_DRIFT) return drift_atom<MIXED>(D, S, i, sp.dt, sp.half_dt2, vx, vy, vz, ax, ay, az);
  return 0.0f;
}

// Kinetic energy and momentum of the calling warp's atoms as int64 fixed point (2^-44 units):
// FP64 warp sums in a fixed shuffle order, rounded once; lane l returns value l / 8 of the four.  A warp
// never spans two systems (tiles start at a system's first atom), so the sums are the same in a
// batch and alone.
__device__ __forceinline__ long long warp_kinetic_fix(double ke, double px, double py, double pz) {
  double v[4] = {ke, px, py, pz};
  return __double2ll_rn(warp_sums(v) * FIX_KE);
}

// The eight sums of a mixed pass -- energy, virial, and the stress's xx, xy, xz, yy, yz, zz -- as
// the system's eleven accumulator slots hold them: the sum that goes to slot k.
__device__ __forceinline__ int sum_of_slot(int k) {
  const int from[11] = {0, 1, 2, 3, 4, 3, 5, 6, 4, 6, 7};
  int f = 0;
#pragma unroll
  for (int q = 0; q < 11; ++q)
    if (k == q) f = from[q];
  return f;
}

// ------------------------------------------------------------------------------------------
// Mixed force pass: FP32 pair maths, int64 fixed-point force sums, FP64 cutoff test inside a
// guard band around rc^2 so the set of interacting pairs is the FP64 reference's.
// ------------------------------------------------------------------------------------------

// Thermo record of system s (one warp, a lane per sum and per field): SetSimulationTags' quantities
// from the FP64 sums `sums` (PD_* order; FP64 path) or, with sums == nullptr, from the system's int64
// accumulators.
__device__ __forceinline__ void thermo_record(const Dev& D, int s, const double* sums, int count_step) {
  const unsigned all = 0xffffffffu;
  const SysDev& S = D.sysd[s];
  SysState& st = D.sst[s];
  const int lane = threadIdx.x & 31;
  const long long step = st.step + (count_step ? 1 : 0);
  double x = 0.0;
  if (lane < PART_D) {
    if (sums) {
      x = sums[lane];
    } else {
      // the accumulators hold the same slots with the embedding energy last
      const int slot = lane == PD_EEMBED ? (int)SA_EEMBED : lane == PD_EPAIR ? (int)SA_EPAIR : lane - 1;
      x = (double)(long long)__ldcg(D.sys_acc + (long long)s * SA_LEN + slot) *
          (lane >= PD_KE ? 1.0 / FIX_KE : 1.0 / FIX_E);
    }
  }
  const double epot = __shfl_sync(all, x, PD_EPAIR) + __shfl_sync(all, x, PD_EEMBED);
  const double vir = __shfl_sync(all, x, PD_VIR);
  const double KIN2EV = 103.64269;  // liblpmd/lpmd/properties.h:10
  const double kin = dmul(__shfl_sync(all, x, PD_KE), KIN2EV);
  const double sum = __shfl_sync(all, x, lane >= 13 ? lane - 13 + PD_STRESS : PD_PX + ((lane - 6) & 3));
  const double vol = S.vol, pv = S.pv;  // volume and pressfactor/volume, computed on the host
  double r = sum;                       // momentum (6..8) and stress (13..21)
  if (lane == 0) r = (double)step;
  if (lane == 1) r = epot;
  if (lane == 2) r = kin;
  if (lane == 3) r = epot + kin;
  if (lane == 4) r = (S.natoms == 0) ? 0.0 : ddiv(dmul(2.0 / 3.0, kin), S.kbn);
  if (lane == 5) r = vir;
  if (lane == 9) r = vol;
  if (lane == 10) r = dmul(dmul(pv, 1.0 / 3.0), vir);
  if (lane == 11) r = dmul(dmul(pv, 2.0 / 3.0), kin);
  if (lane == 12) r = dmul(pv, dadd(dmul(2.0 / 3.0, kin), dmul(1.0 / 3.0, vir)));
  if (lane < THERMO_LEN) {
    D.thermo_last[(long long)s * THERMO_LEN + lane] = r;
    if (count_step) D.thermo_log[((long long)s * D.log_cap + (step % D.log_cap)) * THERMO_LEN + lane] = r;
  }
  __syncwarp();
  if (lane == 0 && count_step) st.step = step;
}

// Tail of a mixed force evaluation, one warp per system: the thermo records from the int64
// accumulators and, inside a step sequence, the next step's rebuild decision and graph
// conditional -- one launch instead of a k_thermo and a k_decide.  The conditional starts every
// graph launch at 0 (cudaGraphCondAssignDefault), so a warp raises it only when its system
// rebuilds and none ever lowers it.  (One thread per system wrote the 44 doubles of a record one
// after the other: 4.6 us for one system, 12 us for 128; a warp 3.7 and 4.7 us.)
__global__ void __launch_bounds__(32 * SYS_WARPS) k_tail(Dev D, int count_step, int decide_next,
                                                         unsigned long long cond_next) {
  const int s = blockIdx.x * SYS_WARPS + (threadIdx.x >> 5);
  if (s >= D.nsys) return;
  if (D.sysd[s].active) thermo_record(D, s, nullptr, count_step);
  if (decide_next && decide_system(D, s, 2, 0) && cond_next && (threadIdx.x & 31) == 0)
    cudaGraphSetConditional((cudaGraphConditionalHandle)cond_next, 1u);
}

// Resident blocks per SM the register allocation of the mixed force kernel is sized for.
#ifndef GBMD_FORCE_MIN_BLOCKS
#define GBMD_FORCE_MIN_BLOCKS 8
#endif
// Packed displacement arithmetic in the EAM force pass as well (the pair force pass always
// uses it when GBMD_F32X2 is on).
#ifndef GBMD_F32X2_EAM_FORCE
#define GBMD_F32X2_EAM_FORCE 1
#endif
// Pair functions of two list entries at a time in packed pairs (LJ; folded Sutton-Chen).
#ifndef GBMD_F32X2_PAIRMATH_LJ
#define GBMD_F32X2_PAIRMATH_LJ 1
#endif
#ifndef GBMD_F32X2_PAIRMATH_EAM
#define GBMD_F32X2_PAIRMATH_EAM 1
#endif

// The same for the mixed EAM density pass (0: no minimum, the compiler's own choice).
#ifndef GBMD_DENSITY_MIN_BLOCKS
#define GBMD_DENSITY_MIN_BLOCKS 0
#endif
#if GBMD_DENSITY_MIN_BLOCKS > 0
#define GBMD_DENSITY_BOUNDS __launch_bounds__(TILE, GBMD_DENSITY_MIN_BLOCKS)
#else
#define GBMD_DENSITY_BOUNDS __launch_bounds__(TILE)
#endif

// List groups per ring iteration of the pair and the EAM force passes (1 or 2).
#ifndef GBMD_EAM_RING_GROUPS
#define GBMD_EAM_RING_GROUPS 2
#endif
#ifndef GBMD_PAIR_RING_GROUPS
#define GBMD_PAIR_RING_GROUPS 2
#endif

// After a bounded wait gave up at group q no further copies are issued; lane 0 then waits (again
// bounded) for the copies already in flight -- groups q .. q+RING-1 below ngw, one per stage --
// so the warp never leaves while the copy engine still writes into its stages.
__device__ __forceinline__ void ring_drain(unsigned long long* bar, int q, int ngw) {
  if ((threadIdx.x & 31) == 0)
    for (int g = q; g < q + RING && g < ngw; ++g) mbar_wait_bounded(&bar[g & (RING - 1)], (unsigned)((g / RING) & 1));
  __syncwarp();
}

// Streams the list groups of the calling warp's 32 atoms (32 x 16 bytes, contiguous for a
// fixed group index) through the warp's RING-stage shared-memory ring with bulk asynchronous
// copies, calling body(group q, this lane's uint4 of that group) for q < ngw, the warp's
// largest group count.  Lane 0 issues the copies; every wait is bounded.  Returns false if a
// wait gave up: the warp then stops (uniformly), drains its copies in flight and skips the
// remaining groups.
template <class F>
__device__ __forceinline__ bool warp_list_ring(const Dev& D, const SysDev& S, int wfirst, int wcount, int ngw,
                                               uint4 (*ring)[32], unsigned long long* bar, F&& body) {
  const int lane = threadIdx.x & 31;
  const uint4* src0 = list_group(D, S, wfirst, 0);
  const unsigned bytes = (unsigned)wcount * 16u;
  const int na = S.natoms;
  if (lane == 0 && ngw > 0) {
    for (int r = 0; r < RING; ++r) mbar_init(&bar[r], 1);
    mbar_init_fence();
    for (int r = 0; r < RING && r < ngw; ++r) {
      mbar_expect_tx(&bar[r], bytes);
      bulk_g2s(ring[r], src0 + (long long)r * na, bytes, &bar[r]);
    }
  }
  __syncwarp();
  for (int q = 0; q < ngw; ++q) {
    const int r = q & (RING - 1);
    if (!__all_sync(0xffffffffu, mbar_wait_bounded(&bar[r], (unsigned)((q / RING) & 1)))) {
      ring_drain(bar, q, ngw);
      return false;
    }
    const uint4 cur = ring[r][lane];
    __syncwarp();  // every lane has its entry: the stage can be refilled
    if (lane == 0 && q + RING < ngw) {
      fence_proxy_async_shared();
      mbar_expect_tx(&bar[r], bytes);
      bulk_g2s(ring[r], src0 + (long long)(q + RING) * na, bytes, &bar[r]);
    }
    body(q, cur);
  }
  return true;
}

// As warp_list_ring, two groups per iteration: both stages are read before either body runs,
// so the two groups' neighbour gathers can be in flight together (for latency-bound bodies).
template <class F>
__device__ __forceinline__ bool warp_list_ring2(const Dev& D, const SysDev& S, int wfirst, int wcount, int ngw,
                                                uint4 (*ring)[32], unsigned long long* bar, F&& body) {
  const int lane = threadIdx.x & 31;
  const uint4* src0 = list_group(D, S, wfirst, 0);
  const unsigned bytes = (unsigned)wcount * 16u;
  const int na = S.natoms;
  if (lane == 0 && ngw > 0) {
    for (int r = 0; r < RING; ++r) mbar_init(&bar[r], 1);
    mbar_init_fence();
    for (int r = 0; r < RING && r < ngw; ++r) {
      mbar_expect_tx(&bar[r], bytes);
      bulk_g2s(ring[r], src0 + (long long)r * na, bytes, &bar[r]);
    }
  }
  __syncwarp();
  for (int q = 0; q < ngw; q += 2) {
    const bool two = q + 1 < ngw;
    const int r0 = q & (RING - 1), r1 = (q + 1) & (RING - 1);
    bool ok = mbar_wait_bounded(&bar[r0], (unsigned)((q / RING) & 1));
    if (two && ok) ok = mbar_wait_bounded(&bar[r1], (unsigned)(((q + 1) / RING) & 1));
    if (!__all_sync(0xffffffffu, ok)) {
      ring_drain(bar, q, ngw);
      return false;
    }
    const uint4 c0 = ring[r0][lane];
    const uint4 c1 = two ? ring[r1][lane] : make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();  // every lane has its entries: the stages can be refilled
    if (lane == 0) {
      fence_proxy_async_shared();
      if (q + RING < ngw) {
        mbar_expect_tx(&bar[r0], bytes);
        bulk_g2s(ring[r0], src0 + (long long)(q + RING) * na, bytes, &bar[r0]);
      }
      if (two && q + 1 + RING < ngw) {
        mbar_expect_tx(&bar[r1], bytes);
        bulk_g2s(ring[r1], src0 + (long long)(q + 1 + RING) * na, bytes, &bar[r1]);
      }
    }
    body(q, c0);
    if (two) body(q + 1, c1);
  }
  return true;
}

// Streaming 16-byte load that does not allocate in L1 (the list is read once per launch; L1 is
// left to the neighbour gathers).
__device__ __forceinline__ uint4 ld_stream(const uint4* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// As warp_list_ring2 with the list rows in registers instead of shared memory: each lane loads
// its own 16-byte entry of rows q + 2 and q + 3 while rows q and q + 1 are evaluated.  Lanes
// without an atom (has = false) load nothing; rows up to the warp's largest group count lie
// inside every atom's list capacity.
template <class F>
__device__ __forceinline__ void warp_list_prefetch2(const Dev& D, const SysDev& S, int li, bool has, int ngw, F&& body) {
  const uint4* src = list_group(D, S, li, 0);
  const long long row = S.natoms;
  const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
  uint4 n0 = (has && ngw > 0) ? ld_stream(src) : zero;
  uint4 n1 = (has && ngw > 1) ? ld_stream(src + row) : zero;
  for (int q = 0; q < ngw; q += 2) {
    const uint4 c0 = n0, c1 = n1;
    if (has && q + 2 < ngw) n0 = ld_stream(src + (long long)(q + 2) * row);
    if (has && q + 3 < ngw) n1 = ld_stream(src + (long long)(q + 3) * row);
    body(q, c0);
    if (q + 1 < ngw) body(q + 1, c1);
  }
}

// How the mixed force and density passes read their list rows (template parameter FEED, chosen
// per launch): FEED_REGS, each lane loads its own entries into registers with L1-bypassing loads;
// FEED_RING, bulk asynchronous copies into a per-warp shared-memory ring.  Results are bitwise
// the same.  The ring hides the list's latency best; registers leave the L1 that serves the
// neighbour gathers 32 KB larger per SM, which the density pass (a gather and little else) uses
// better.  The figures stand at the choice between them (launch_force_passes).
constexpr int FEED_REGS = 0, FEED_RING = 1;

template <int PC, int SPECIES, int SCN, int SCM, int FEED>
__device__ __forceinline__ void force32_tile(const Dev& D, const PotParams& P, const StepParams& sp, const Blk32 B) {
  const int s = B.sys;
  const SysDev& S = D.sysd[s];
  if (!S.active) {  // whole block: its atoms belong to one system
    if (sp.epi == EPI_KICK_DRIFT && sp.last) hold_range(D, S, B.first, B.count, true);
    return;
  }
  __shared__ ShiftTable<> shifts;
  load_shifts(S, shifts);
  const ShiftCorr corr = shift_corr(S);
  const int li = B.first - (int)S.atom_base + (int)threadIdx.x;  // index within the system
  const long long i = S.atom_base + li;
  const bool active = (int)threadIdx.x < B.count;
  const float4* __restrict__ g32 = D.g32 + S.atom_base;
  // EAM without a species filter gathers the density pass's copy, whose w holds the
  // neighbour's embedding factor (one 16-byte gather per pair instead of 16 + 4 bytes)
  constexpr bool PHI_IN_W = PC == PC_EAM && !SPECIES;
  const float4* __restrict__ gsrc = PHI_IN_W ? D.g32e + S.atom_base : g32;
  // force, energy and virial: each group of four list entries is summed in FP32 and the group
  // sum rounded into int64 fixed point (forces 2^-32 eV/A; energy and virial 2^-26 eV, scaled
  // to the system accumulators' 2^-32 by an exact integer shift); stress components are summed
  // in FP32 per atom (sab = sum of f_a * r_b with f = g * r; stress_ab = -sab/2), rounded once
  Fix fqx, fqy, fqz, fqe, fqv;
  float sxx = 0.f, sxy = 0.f, sxz = 0.f, syy = 0.f, syz = 0.f, szz = 0.f;
  const float rc2_lo = P.f[12], rc2_hi = P.f[13];
  unsigned rechecks = 0;
  bool bad = false;
  // Each warp streams its 32 atoms' list groups (32 x 16 bytes, contiguous for a fixed group
  // index), with FEED_RING through its own ring of shared-memory stages filled by bulk
  // asynchronous copies (TMA engine) that run RING groups ahead of the force evaluation, with
  // FEED_REGS through registers loaded two groups ahead.  Warps never wait on each other
  // inside the loop.
  __shared__ __align__(16) uint4 ring[TILE / 32][RING][32];
  __shared__ __align__(8) unsigned long long bar[TILE / 32][RING];
  {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float4 gi = active ? g32[li] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int ti = __float_as_int(gi.w);
    // the embedding factor as the loop uses it: the density pass's copy (f[14] x 1/sqrt(rho),
    // f[14] = the Sutton-Chen many-body prefactor in the folded form, else 1) where gathered
    const float phi_i = (PC == PC_EAM && active) ? (PHI_IN_W ? gsrc[li].w : D.phif[i]) : 0.f;
    constexpr bool FOLDED = PHI_IN_W && SCN > 0;
    constexpr bool PACKED_R2 = GBMD_F32X2 && (PC == PC_PAIR || GBMD_F32X2_EAM_FORCE);
    const int na = S.natoms;
    const int cnt = active ? D.ncount[i] : 0;
    const int ng = (cnt + 3) >> 2;
    // Guard-band entries (a few per thousand atoms) are only noted in the loop and decided in
    // FP64 afterwards; their forces then go straight into the fixed-point sums.
    constexpr unsigned NO_BAND = 0xffffffffu;
    unsigned band_e = NO_BAND;
    bool band_more = false;
    float ge = 0.f, gv = 0.f;  // the current group's energy and sum of g r^2
    // Branch-free body: every candidate is evaluated and out-of-range pairs are masked to
    // zero, so lanes never diverge on the cutoff test (70% of Verlet-list entries are inside).
    // Returns g with f = g * d; the caller sums a group's four forces in FP32 and adds the
    // group sum to the int64 fixed-point accumulators.
    auto pair = [&](unsigned e, bool valid, float& dx, float& dy, float& dz) -> float {
      const int j = (int)(e & LOCAL_MASK);
      const float4 gj = gsrc[j];
      const float r2 = entry_r2<PACKED_R2>(gi, gj, shifts[e >> CODE_SHIFT], corr, dx, dy, dz);
      bool in = valid && r2 < rc2_lo;
      if (valid && r2 >= rc2_lo && r2 < rc2_hi) {  // guard band: decided in FP64 after the loop
        if (band_e == NO_BAND)
          band_e = e;
        else
          band_more = true;
      }
      if (SPECIES) in = in && applies_to(P.spc_sum, ti, __float_as_int(gj.w));
      float g, en;
      if (PC == PC_PAIR) {
        lj_pair32(P, rcp_approx(r2), g, en);
      } else if constexpr (FOLDED) {
        eam_sc_pair32_q<SCN, SCM>(P, r2, phi_i, gj.w, g, en);
      } else {
        eam_pair32_t<SCN, SCM>(P, r2, phi_i, PHI_IN_W ? gj.w : D.phif[S.atom_base + j], g, en);
      }
      g = in ? g : 0.0f;
      ge += in ? en : 0.0f;
      gv = fmaf(g, r2, gv);
      const float fx = g * dx, fy = g * dy, fz = g * dz;
      sxx = fmaf(fx, dx, sxx);
      sxy = fmaf(fx, dy, sxy);
      sxz = fmaf(fx, dz, sxz);
      syy = fmaf(fy, dy, syy);
      syz = fmaf(fy, dz, syz);
      szz = fmaf(fz, dz, szz);
      return g;
    };
    // The same two entries at a time, with the pair functions' products of variables as packed
    // FP32 pairs (LJ and folded Sutton-Chen; bitwise the values of `pair`).
    auto geom = [&](unsigned e, bool valid, float& dx, float& dy, float& dz, bool& in, float& qj) -> float {
      const int j = (int)(e & LOCAL_MASK);
      const float4 gj = gsrc[j];
      const float r2 = entry_r2<PACKED_R2>(gi, gj, shifts[e >> CODE_SHIFT], corr, dx, dy, dz);
      in = valid && r2 < rc2_lo;
      if (valid && r2 >= rc2_lo && r2 < rc2_hi) {
        if (band_e == NO_BAND)
          band_e = e;
        else
          band_more = true;
      }
      if (SPECIES) in = in && applies_to(P.spc_sum, ti, __float_as_int(gj.w));
      qj = gj.w;
      return r2;
    };
    auto accum = [&](float g, float en, bool in, float r2, float dx, float dy, float dz) -> float {
      g = in ? g : 0.0f;
      ge += in ? en : 0.0f;
      gv = fmaf(g, r2, gv);
      const float fx = g * dx, fy = g * dy, fz = g * dz;
      sxx = fmaf(fx, dx, sxx);
      sxy = fmaf(fx, dy, sxy);
      sxz = fmaf(fx, dz, sxz);
      syy = fmaf(fy, dy, syy);
      syz = fmaf(fy, dz, syz);
      szz = fmaf(fz, dz, szz);
      return g;
    };
    auto two = [&](unsigned ea, unsigned eb, bool va, bool vb, float& ax, float& ay, float& az, float& bx,
                   float& by, float& bz, float& ga, float& gb) {
      bool ina, inb;
      float qa, qb;
      const float r2a = geom(ea, va, ax, ay, az, ina, qa);
      const float r2b = geom(eb, vb, bx, by, bz, inb, qb);
      float sa, sb, ena, enb;
      if constexpr (PC == PC_PAIR) {
        lj_pair32_x2(P, rcp_approx(r2a), rcp_approx(r2b), sa, sb, ena, enb);
      } else if constexpr (FOLDED) {
        eam_sc_pair32_q_x2<SCN, SCM>(P, r2a, r2b, phi_i, qa, qb, sa, sb, ena, enb);
      } else {
        sa = sb = ena = enb = 0.0f;  // not reached: `two` serves the LJ and folded forms only
      }
      ga = accum(sa, ena, ina, r2a, ax, ay, az);
      gb = accum(sb, enb, inb, r2b, bx, by, bz);
    };
    constexpr bool PAIRED =
        GBMD_F32X2 && ((PC == PC_PAIR && GBMD_F32X2_PAIRMATH_LJ) || (FOLDED && GBMD_F32X2_PAIRMATH_EAM));
    // One group of four entries (rem = entries left in the atom's list from this group on).
    auto group = [&](const uint4& cur, int rem) {
      ge = 0.f;
      gv = 0.f;
      float ax, ay, az, bx, by, bz;
      float g0, g1;
      if constexpr (PAIRED) {
        two(cur.x, cur.y, true, rem > 1, ax, ay, az, bx, by, bz, g0, g1);
      } else {
        g0 = pair(cur.x, true, ax, ay, az);
        g1 = pair(cur.y, rem > 1, bx, by, bz);
      }
      float gx = fmaf(g1, bx, g0 * ax), gy = fmaf(g1, by, g0 * ay), gz = fmaf(g1, bz, g0 * az);
      if constexpr (PAIRED) {
        two(cur.z, cur.w, rem > 2, rem > 3, ax, ay, az, bx, by, bz, g0, g1);
      } else {
        g0 = pair(cur.z, rem > 2, ax, ay, az);
        g1 = pair(cur.w, rem > 3, bx, by, bz);
      }
      gx = fmaf(g1, bx, fmaf(g0, ax, gx));
      gy = fmaf(g1, by, fmaf(g0, ay, gy));
      gz = fmaf(g1, bz, fmaf(g0, az, gz));
      fqx.add_scaled32(gx);
      fqy.add_scaled32(gy);
      fqz.add_scaled32(gz);
      // halved: the full list counts each pair twice; virial = -sum g r^2 / 2
      fqe.add_scaled26(0.5f * ge);
      fqv.add_scaled26(-0.5f * gv);
      // |group force| < 4096 eV/A keeps the force split exact
      bad |= fmaxf(fabsf(gx), fmaxf(fabsf(gy), fabsf(gz))) > 4000.0f;
    };
    const int ngw = __reduce_max_sync(0xffffffffu, (unsigned)ng);
    const int wfirst = B.first - (int)S.atom_base + 32 * w;
    const int wcount = min(32, max(0, B.count - 32 * w));
    bool waited = true;
    if constexpr (FEED == FEED_REGS &&
                  ((PC == PC_PAIR && GBMD_PAIR_RING_GROUPS == 2) || (PC == PC_EAM && GBMD_EAM_RING_GROUPS == 2))) {
      warp_list_prefetch2(D, S, li, lane < wcount, ngw, [&](int q, const uint4& cur) {
        if (q < ng) group(cur, cnt - 4 * q);
      });
    } else if constexpr ((PC == PC_PAIR && GBMD_PAIR_RING_GROUPS == 2) || (PC == PC_EAM && GBMD_EAM_RING_GROUPS == 2)) {
      // two list groups per iteration: eight neighbour gathers in flight per lane
      waited = warp_list_ring2(D, S, wfirst, wcount, ngw, ring[w], bar[w], [&](int q, const uint4& cur) {
        if (q < ng) group(cur, cnt - 4 * q);
      });
    } else {
      // one group per iteration, written out here: through the helper the EAM body spills more
      const uint4* src0 = list_group(D, S, wfirst, 0);
      const unsigned bytes = (unsigned)wcount * 16u;
      unsigned long long* wbar = bar[w];
      if (lane == 0 && ngw > 0) {
        for (int r = 0; r < RING; ++r) mbar_init(&wbar[r], 1);
        mbar_init_fence();
        for (int r = 0; r < RING && r < ngw; ++r) {
          mbar_expect_tx(&wbar[r], bytes);
          bulk_g2s(ring[w][r], src0 + (long long)r * na, bytes, &wbar[r]);
        }
      }
      __syncwarp();
      for (int q = 0; q < ngw; ++q) {
        const int r = q & (RING - 1);
        if (!__all_sync(0xffffffffu, mbar_wait_bounded(&wbar[r], (unsigned)((q / RING) & 1)))) {
          ring_drain(wbar, q, ngw);  // stop issuing, wait for the copies in flight, skip the rest
          waited = false;
          break;
        }
        const uint4 cur = ring[w][r][lane];
        __syncwarp();  // every lane has its entry: the stage can be refilled
        if (lane == 0 && q + RING < ngw) {
          fence_proxy_async_shared();
          mbar_expect_tx(&wbar[r], bytes);
          bulk_g2s(ring[w][r], src0 + (long long)(q + RING) * na, bytes, &wbar[r]);
        }
        if (q < ng) group(cur, cnt - 4 * q);
      }
    }
    if (!waited) atomicOr(&D.sst[s].error, ERR_WAIT);
    if (band_e != NO_BAND) {
      // exact FP64 cutoff decision (the reference's Displacement and r^2) for the guard-band
      // entries; one noted entry per atom, else a rescan of the atom's list
      auto settle = [&](unsigned e) {
        const int j = (int)(e & LOCAL_MASK);
        const float4 gj = g32[j];
        float dx, dy, dz;
        const float r2 = entry_r2(gi, gj, shifts[e >> CODE_SHIFT], corr, dx, dy, dz);
        if (!(r2 >= rc2_lo && r2 < rc2_hi)) return;
        ++rechecks;
        if (!exact_inside_cold(&D, &S, i, S.atom_base + j, P.rc2)) return;
        if (SPECIES && !applies_to(P.spc_sum, ti, __float_as_int(gj.w))) return;
        float g, en;
        if (PC == PC_PAIR) {
          lj_pair32(P, rcp_approx(r2), g, en);
        } else {
          // the unscaled embedding factors of both atoms (rare path)
          eam_pair32_t<SCN, SCM>(P, r2, D.phif[i], D.phif[S.atom_base + j], g, en);
        }
        const float fx = g * dx, fy = g * dy, fz = g * dz;
        fqx.add_scaled32(fx);
        fqy.add_scaled32(fy);
        fqz.add_scaled32(fz);
        fqe.add_scaled26(0.5f * en);
        fqv.add_scaled26(-0.5f * (g * r2));
        bad |= fmaxf(fabsf(fx), fmaxf(fabsf(fy), fabsf(fz))) > 4000.0f;
        sxx = fmaf(fx, dx, sxx);
        sxy = fmaf(fx, dy, sxy);
        sxz = fmaf(fx, dz, sxz);
        syy = fmaf(fy, dy, syy);
        syz = fmaf(fy, dz, syz);
        szz = fmaf(fz, dz, szz);
      };
      if (!band_more) {
        settle(band_e);
      } else {
        const uint4* L = list_group(D, S, li, 0);
        for (int q = 0; q < ng; ++q) {
          const uint4 e4 = __ldg(L + (long long)q * na);
          const int rem = cnt - 4 * q;
          settle(e4.x);
          if (rem > 1) settle(e4.y);
          if (rem > 2) settle(e4.z);
          if (rem > 3) settle(e4.w);
        }
      }
    }
  }
  double ke = 0.0, px = 0.0, py = 0.0, pz = 0.0;
  float d2 = 0.0f;
  if (active) {
    const long long N = D.N;
    long long qx = fqx.value(), qy = fqy.value(), qz = fqz.value();
    if (!sp.first) {
      qx += D.facc[i];
      qy += D.facc[N + i];
      qz += D.facc[2 * N + i];
    }
    if (sp.last) {
      d2 = finish_atom<1>(D, S, i, (double)qx, (double)qy, (double)qz, sp, ke, px, py, pz);
    } else {
      D.facc[i] = qx;
      D.facc[N + i] = qy;
      D.facc[2 * N + i] = qz;
    }
    if (rechecks) atomicAdd(&D.sst[s].rechecks, (unsigned long long)rechecks);
    if (bad) atomicOr(&D.sst[s].error, ERR_FIXED);
  }
  track_displacement_warp(D, s, d2);
  // energy and virial already in fixed point; per-atom stress (halved: full list) rounded to
  // int64 once, kinetic energy and momentum as FP64 warp sums in a fixed order rounded once per warp;
  // exact int64 sums from there on, one integer atomic per quantity into the system's slots.  The warp
  // sums halve the values a lane carries with each exchange: 9 additions a lane instead of 55 for the
  // eight integers, 6 on the FP64 unit instead of 20 for the four kinetic ones (a third of the
  // epilogue's FP64 instructions with their roundings): 2,048,000 LJ atoms 511 -> 473 us, 495,000 of
  // copper 241 -> 233, 128 systems 218 -> 200.
  __shared__ long long esum[TILE / 32][8], ksum[TILE / 32][4];
  {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float ms = (float)(-0.5 * FIX_E);
    long long v[8] = {fqe.value() * 64, fqv.value() * 64, fix64(sxx * ms), fix64(sxy * ms), fix64(sxz * ms),
                      fix64(syy * ms),  fix64(syz * ms),  fix64(szz * ms)};
    const long long t = warp_sums(v);
    if ((lane & 3) == 0) esum[w][lane >> 2] = t;
    if (sp.last) {
      const long long k = warp_kinetic_fix(ke, px, py, pz);
      if ((lane & 7) == 0) ksum[w][lane >> 3] = k;
    }
  }
  __syncthreads();
  const int slot = threadIdx.x;
  if (slot < (sp.last ? 15 : 11)) {
    const long long* from = slot < 11 ? &esum[0][sum_of_slot(slot)] : &ksum[0][slot - 11];
    const int stride = slot < 11 ? 8 : 4;
    long long t = 0;
    for (int w = 0; w < TILE / 32; ++w) t += from[w * stride];
    static_assert(SA_STRESS == 2 && SA_KE == 11 && SA_P == 12, "slots in the order of the sums");
    atomicAdd(D.sys_acc + (long long)s * SA_LEN + slot, (unsigned long long)t);
  }
}


template <int PC, int SPECIES, int SCN = 0, int SCM = 0, int FEED = FEED_REGS>
__global__ void __launch_bounds__(TILE, GBMD_FORCE_MIN_BLOCKS) k_force32(Dev D, PotParams P, StepParams sp, const Blk32* blk) {
  force32_tile<PC, SPECIES, SCN, SCM, FEED>(D, P, sp, blk[blockIdx.x]);
}

// ------------------------------------------------------------------------------------------
// Mixed force pass with LANES lanes per atom (TILE / LANES atoms a block), for systems too small to
// fill the GPU one lane per atom: there a warp's time is its own chain of some ten iterations of
// gathers and arithmetic (26 us with the tail for 4,000 and for 16,384 atoms of LJ liquid alike, 15 and 18 here),
// which LANES lanes cut to two or three.  The atom's list groups go round-robin to its lanes (plain
// cached loads); each group is evaluated and summed exactly as in k_force32, and the lanes'
// fixed-point partials are combined with integer shuffles.  Stress, an FP32 sum over the whole list in
// k_force32, is handed from lane to lane: after each round of groups every lane in turn adds its four
// entries and all go on from its sums (0.9 us of the pass at 16,384 LJ atoms, 1.3 at 32,000 of iron; through
// shared memory 5 and 3).  So every result is bitwise that of k_force32, and what a
// system gets does not depend on the lanes, which go by what else is in the batch.  The per-atom
// epilogue -- FP64 instructions, as long for one atom as for 32 -- runs one thread per atom in as few
// warps as hold the block's atoms (in every warp, with a few lanes at work, it took longer than the
// pairs: 15.1 us at 4 lanes and 16,384 atoms, 14.3 so; 20 and 15.3 at 8).  A block has whole groups of
// 32 atoms of its system, whose kinetic terms are summed in FP64 as a warp of k_force32 sums them.
// ------------------------------------------------------------------------------------------

// g and pair energy of one entry; qi, qj: the embedding factors (metals), folded: times the prefactor.
template <int PC, bool FOLDED, int SCN, int SCM>
__device__ __forceinline__ void pair32(const PotParams& P, float r2, float qi, float qj, float& g, float& en) {
  if constexpr (PC == PC_PAIR)
    lj_pair32(P, rcp_approx(r2), g, en);
  else if constexpr (FOLDED)
    eam_sc_pair32_q<SCN, SCM>(P, r2, qi, qj, g, en);
  else
    eam_pair32_t<SCN, SCM>(P, r2, qi, qj, g, en);
}

// Sum of an atom's fixed-point partials over its LANES adjacent lanes.
template <int LANES>
__device__ __forceinline__ void lanes_sum(Fix& f) {
#pragma unroll
  for (int m = 1; m < LANES; m <<= 1) {
    f.hi += __shfl_xor_sync(0xffffffffu, f.hi, m);
    f.lo += __shfl_xor_sync(0xffffffffu, f.lo, m);
  }
}

// Atoms and threads of a block with `lanes` lanes an atom.
constexpr int lanes_atoms(int lanes) { return lanes <= TILE / 32 ? TILE / lanes : 32; }
constexpr int lanes_threads(int lanes) { return lanes * lanes_atoms(lanes); }

template <int PC, int SPECIES, int SCN, int SCM, int LANES>
__global__ void __launch_bounds__(lanes_threads(LANES), 8 * TILE / lanes_threads(LANES))
    k_force32_lanes(Dev D, PotParams P, StepParams sp, const Blk32* blk) {
  constexpr int APB = lanes_atoms(LANES), WARPS = lanes_threads(LANES) / 32;
  __shared__ ShiftTable<> shifts;
  __shared__ long long fsum[3][APB];
  __shared__ long long esum[WARPS][8];
  const Blk32 B = blk[blockIdx.x];
  const int s = B.sys;
  const SysDev& S = D.sysd[s];
  if (!S.active) {  // whole block: its atoms belong to one system
    if (sp.epi == EPI_KICK_DRIFT && sp.last) hold_range(D, S, B.first, B.count, true);
    return;
  }
  load_shifts(S, shifts);
  const ShiftCorr corr = shift_corr(S);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sub = threadIdx.x % LANES, slot = (int)threadIdx.x / LANES;
  const float4* __restrict__ g32 = D.g32 + S.atom_base;
  // as in k_force32: metals without a species filter gather the embedding factor with the position
  constexpr bool PHI_IN_W = PC == PC_EAM && !SPECIES;
  constexpr bool FOLDED = PHI_IN_W && SCN > 0;
  const float4* __restrict__ gsrc = PHI_IN_W ? D.g32e + S.atom_base : g32;
  const float rc2_lo = P.f[12], rc2_hi = P.f[13];
  unsigned rechecks = 0;
  bool bad = false;
  Fix fqe, fqv;
  const bool active = slot < B.count;
  const int li = B.first - (int)S.atom_base + (active ? slot : 0);
  const long long i = S.atom_base + li;
  Fix fqx, fqy, fqz;
  float stress[6] = {};  // xx, xy, xz, yy, yz, zz of the atom, in each of its lanes
  const float4 gi = active ? g32[li] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int ti = __float_as_int(gi.w);
  const float phi_i = (PC == PC_EAM && active) ? (PHI_IN_W ? gsrc[li].w : D.phif[i]) : 0.f;
  const int na = S.natoms;
  const int cnt = active ? D.ncount[i] : 0;
  const int ng = (cnt + 3) >> 2;
  constexpr unsigned NO_BAND = 0xffffffffu;
  unsigned band_e = NO_BAND;
  bool band_more = false;
  const uint4* L = active ? list_group(D, S, li, 0) : nullptr;
  const int ngw = (int)__reduce_max_sync(0xffffffffu, (unsigned)ng);
  for (int q0 = 0; q0 < ngw; q0 += LANES) {
    const int q = q0 + sub;
    float f[3][4] = {}, d[3][4] = {};
    if (q < ng) {
      const uint4 cur = __ldg(L + (long long)q * na);
      const unsigned e[4] = {cur.x, cur.y, cur.z, cur.w};
      const int rem = cnt - 4 * q;
      float4 gj[4];
      float pj[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        gj[u] = gsrc[e[u] & LOCAL_MASK];
        pj[u] = (PC == PC_EAM && !PHI_IN_W) ? D.phif[S.atom_base + (e[u] & LOCAL_MASK)] : gj[u].w;
      }
      float ge = 0.f, gv = 0.f, gx = 0.f, gy = 0.f, gz = 0.f;
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool valid = u == 0 || rem > u;
        float dx, dy, dz;
        const float r2 = entry_r2(gi, gj[u], shifts[e[u] >> CODE_SHIFT], corr, dx, dy, dz);
        bool in = valid && r2 < rc2_lo;
        if (valid && r2 >= rc2_lo && r2 < rc2_hi) {  // guard band: decided in FP64 after the loop
          if (band_e == NO_BAND)
            band_e = e[u];
          else
            band_more = true;
        }
        if (SPECIES) in = in && applies_to(P.spc_sum, ti, __float_as_int(gj[u].w));
        float g, en;
        pair32<PC, FOLDED, SCN, SCM>(P, r2, phi_i, pj[u], g, en);
        g = in ? g : 0.0f;
        ge += in ? en : 0.0f;
        gv = fmaf(g, r2, gv);
        d[0][u] = dx;
        d[1][u] = dy;
        d[2][u] = dz;
        f[0][u] = g * dx;
        f[1][u] = g * dy;
        f[2][u] = g * dz;
        // the group's force in k_force32's order: ((g0 d0 + g1 d1) + g2 d2) + g3 d3, fused
        gx = u == 0 ? g * dx : fmaf(g, dx, gx);
        gy = u == 0 ? g * dy : fmaf(g, dy, gy);
        gz = u == 0 ? g * dz : fmaf(g, dz, gz);
      }
      fqx.add_scaled32(gx);
      fqy.add_scaled32(gy);
      fqz.add_scaled32(gz);
      fqe.add_scaled26(0.5f * ge);
      fqv.add_scaled26(-0.5f * gv);
      bad |= fmaxf(fabsf(gx), fmaxf(fabsf(gy), fabsf(gz))) > 4000.0f;
    }
    // the round's groups in list order: each lane in turn adds its own, and all go on from its sums (a
    // lane without a group adds zeros, which change none)
#pragma unroll
    for (int l = 0; l < LANES; ++l) {
#pragma unroll
      for (int k = 0; k < 6; ++k) {
        const int a = k < 3 ? 0 : k < 5 ? 1 : 2, b = k < 3 ? k : k < 5 ? k - 2 : 2;
        float t = stress[k];
#pragma unroll
        for (int u = 0; u < 4; ++u) t = fmaf(f[a][u], d[b][u], t);
        stress[k] = __shfl_sync(0xffffffffu, t, l, LANES);
      }
    }
  }
  // guard-band entries, as in k_force32 in list order: all lanes of the atom settle each of them, and
  // the first one adds it to the fixed-point sums
  const unsigned mine = (LANES == 32 ? 0xffffffffu : (1u << (LANES & 31)) - 1u) << (lane - sub);
  const unsigned noted = __ballot_sync(0xffffffffu, band_e != NO_BAND) & mine;
  const unsigned more = __ballot_sync(0xffffffffu, band_more) & mine;
  if (noted) {
    auto settle = [&](unsigned e) {
      const int j = (int)(e & LOCAL_MASK);
      const float4 gj = g32[j];
      float dx, dy, dz;
      const float r2 = entry_r2(gi, gj, shifts[e >> CODE_SHIFT], corr, dx, dy, dz);
      if (!(r2 >= rc2_lo && r2 < rc2_hi)) return;
      if (sub == 0) ++rechecks;
      if (!exact_inside_cold(&D, &S, i, S.atom_base + j, P.rc2)) return;
      if (SPECIES && !applies_to(P.spc_sum, ti, __float_as_int(gj.w))) return;
      float g, en;
      if (PC == PC_PAIR)
        lj_pair32(P, rcp_approx(r2), g, en);
      else  // the unscaled embedding factors of both atoms (rare path)
        eam_pair32_t<SCN, SCM>(P, r2, D.phif[i], D.phif[S.atom_base + j], g, en);
      const float fx = g * dx, fy = g * dy, fz = g * dz;
      if (sub == 0) {
        fqx.add_scaled32(fx);
        fqy.add_scaled32(fy);
        fqz.add_scaled32(fz);
        fqe.add_scaled26(0.5f * en);
        fqv.add_scaled26(-0.5f * (g * r2));
        bad |= fmaxf(fabsf(fx), fmaxf(fabsf(fy), fabsf(fz))) > 4000.0f;
      }
      stress[0] = fmaf(fx, dx, stress[0]);
      stress[1] = fmaf(fx, dy, stress[1]);
      stress[2] = fmaf(fx, dz, stress[2]);
      stress[3] = fmaf(fy, dy, stress[3]);
      stress[4] = fmaf(fy, dz, stress[4]);
      stress[5] = fmaf(fz, dz, stress[5]);
    };
    if (!more && (noted & (noted - 1)) == 0) {
      settle(__shfl_sync(mine, band_e, __ffs(noted) - 1));
    } else {
      for (int q = 0; q < ng; ++q) {
        const uint4 e4 = __ldg(L + (long long)q * na);
        const int rem = cnt - 4 * q;
        settle(e4.x);
        if (rem > 1) settle(e4.y);
        if (rem > 2) settle(e4.z);
        if (rem > 3) settle(e4.w);
      }
    }
  }
  lanes_sum<LANES>(fqx);
  lanes_sum<LANES>(fqy);
  lanes_sum<LANES>(fqz);
  if (sub == 0 && active) {
    fsum[0][slot] = fqx.value();
    fsum[1][slot] = fqy.value();
    fsum[2][slot] = fqz.value();
  }
  if (rechecks) atomicAdd(&D.sst[s].rechecks, (unsigned long long)rechecks);
  if (bad) atomicOr(&D.sst[s].error, ERR_FIXED);
  // energy and virial: every lane's own fixed-point partial (exact integer sums, whatever the lane
  // count); stress: the atom's sums (halved: full list), rounded once, from its first lane
  auto fix = [&](float t) { return fix64(sub == 0 ? t * (float)(-0.5 * FIX_E) : 0.0f); };
  long long v[8] = {fqe.value() * 64, fqv.value() * 64, fix(stress[0]), fix(stress[1]),
                    fix(stress[2]),   fix(stress[3]),   fix(stress[4]), fix(stress[5])};
  const long long t8 = warp_sums(v);
  if ((lane & 3) == 0) esum[w][lane >> 2] = t8;
  __syncthreads();
  unsigned long long* acc = D.sys_acc + (long long)s * SA_LEN;
  if (w == WARPS - 1 && lane < 11) {
    // energy, virial and the nine stress slots from the eight sums (in the last warp: the first ones
    // go on with the atoms)
    const int f = sum_of_slot(lane);
    long long t = 0;
    for (int k = 0; k < WARPS; ++k) t += esum[k][f];
    atomicAdd(acc + lane, (unsigned long long)t);
  }
  const int t = threadIdx.x;
  if (t >= ((B.count + 31) & ~31)) return;  // whole warps
  double ke = 0.0, px = 0.0, py = 0.0, pz = 0.0;
  float d2 = 0.0f;
  if (t < B.count) {
    const long long a = B.first + t, N = D.N;
    long long qx = fsum[0][t], qy = fsum[1][t], qz = fsum[2][t];
    if (!sp.first) {
      qx += D.facc[a];
      qy += D.facc[N + a];
      qz += D.facc[2 * N + a];
    }
    if (sp.last) {
      d2 = finish_atom<1>(D, S, a, (double)qx, (double)qy, (double)qz, sp, ke, px, py, pz);
    } else {
      D.facc[a] = qx;
      D.facc[N + a] = qy;
      D.facc[2 * N + a] = qz;
    }
  }
  track_displacement_warp(D, s, d2);
  if (sp.last) {
    const long long k = warp_kinetic_fix(ke, px, py, pz);
    if ((lane & 7) == 0) atomicAdd(acc + SA_KE + (lane >> 3), (unsigned long long)k);  // SA_P follows SA_KE
  }
}

// ------------------------------------------------------------------------------------------
// EAM density pass + embedding (FP64 embedding in both precisions).
// ------------------------------------------------------------------------------------------

// Mixed density pass over the Verlet list: FP32 rho_ij of each group of four entries
// (branch-free, out-of-range entries masked), the group sum added to the int64 fixed-point
// density; cutoff decisions in the guard band re-done in FP64 as in the force kernel.
template <int SCM, int FEED>
__device__ __forceinline__ void density32_tile(const Dev& D, const PotParams& P, const Blk32 B) {
  __shared__ __align__(16) uint4 ring_s[TILE / 32][RING][32];
  __shared__ __align__(8) unsigned long long bar_s[TILE / 32][RING];
  const int s = B.sys;
  const SysDev& S = D.sysd[s];
  if (!S.active) return;  // whole block: its atoms belong to one system
  __shared__ ShiftTable<> shifts;
  load_shifts(S, shifts);
  const ShiftCorr corr = shift_corr(S);
  const int li = B.first - (int)S.atom_base + (int)threadIdx.x;
  const long long i = S.atom_base + li;
  const bool active = (int)threadIdx.x < B.count;
  const float4* __restrict__ g32 = D.g32 + S.atom_base;
  const float4 gi = active ? g32[li] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float rc2_lo = P.f[12], rc2_hi = P.f[13];
  const int cnt = active ? D.ncount[i] : 0;
  const int ng = (cnt + 3) >> 2;
  Fix q;
  unsigned rechecks = 0;
  // guard-band entries are noted in the loop and decided in FP64 afterwards (as in k_force32)
  constexpr unsigned NO_BAND = 0xffffffffu;
  unsigned band_e = NO_BAND;
  bool band_more = false;
  auto term = [&](unsigned e, bool valid) -> float {
    const int j = (int)(e & LOCAL_MASK);
    float dx, dy, dz;
    const float r2 = entry_r2(gi, g32[j], shifts[e >> CODE_SHIFT], corr, dx, dy, dz);
    const bool in = valid && r2 < rc2_lo;
    if (valid && r2 >= rc2_lo && r2 < rc2_hi) {
      if (band_e == NO_BAND)
        band_e = e;
      else
        band_more = true;
    }
    const float v = eam_rho32_t<SCM>(P, r2);
    return in ? v : 0.0f;
  };
  const float scale = (float)FIX_RHO;
  // every lane of the warp takes part in the ring (lanes without an atom have no groups)
  const int w = threadIdx.x >> 5;
  const int wfirst = B.first - (int)S.atom_base + 32 * w;
  const int wcount = min(32, max(0, B.count - 32 * w));
  const int ngw = __reduce_max_sync(0xffffffffu, (unsigned)ng);
  auto row = [&](int g, const uint4& e4) {
    if (g < ng) {
      const int rem = cnt - 4 * g;
      const float part = ((term(e4.x, true) + term(e4.y, rem > 1)) + term(e4.z, rem > 2)) + term(e4.w, rem > 3);
      q.add(part * scale);
    }
  };
  bool waited = true;
  if constexpr (FEED == FEED_RING)
    waited = warp_list_ring2(D, S, wfirst, wcount, ngw, ring_s[w], bar_s[w], row);
  else
    warp_list_prefetch2(D, S, li, active, ngw, row);
  if (!waited) atomicOr(&D.sst[s].error, ERR_WAIT);
  if (band_e != NO_BAND) {
    auto settle = [&](unsigned e) {
      const int j = (int)(e & LOCAL_MASK);
      float dx, dy, dz;
      const float r2 = entry_r2(gi, g32[j], shifts[e >> CODE_SHIFT], corr, dx, dy, dz);
      if (!(r2 >= rc2_lo && r2 < rc2_hi)) return;
      ++rechecks;
      if (exact_inside_cold(&D, &S, i, S.atom_base + j, P.rc2)) q.add(eam_rho32_t<SCM>(P, r2) * scale);
    };
    if (!band_more) {
      settle(band_e);
    } else {
      const uint4* L = list_group(D, S, li, 0);
      for (int g = 0; g < ng; ++g) {
        const uint4 e4 = __ldg(L + (long long)g * S.natoms);
        const int rem = cnt - 4 * g;
        settle(e4.x);
        if (rem > 1) settle(e4.y);
        if (rem > 2) settle(e4.z);
        if (rem > 3) settle(e4.w);
      }
    }
  }
  if (rechecks) atomicAdd(&D.sst[s].rechecks, (unsigned long long)rechecks);
  double F = 0.0;
  if (active) {
    const double rho = (double)q.value() * (1.0 / FIX_RHO);
    double phi;
    eam_embed64(P, rho, F, phi);
    D.rho[i] = rho;
    D.phi[i] = phi;
    D.phif[i] = (float)phi;
    D.g32e[i] = make_float4(gi.x, gi.y, gi.z, (float)((double)P.f[14] * phi));
  }
  // FP64 embedding energies summed exactly as int64 fixed point (2^-32 eV per atom)
  long long v[1] = {active ? __double2ll_rn(F * FIX_E) : 0ll};
  long long t[1];
  block_sum<long long, 1>(v, t);
  if (threadIdx.x == 0) atomicAdd(D.sys_acc + (long long)s * SA_LEN + SA_EEMBED, (unsigned long long)t[0]);
}


template <int SCM, int FEED = FEED_REGS>
__global__ void GBMD_DENSITY_BOUNDS k_eam_density32(Dev D, PotParams P, const Blk32* blk) {
  density32_tile<SCM, FEED>(D, P, blk[blockIdx.x]);
}

// The same with LANES lanes per atom (see k_force32_lanes): densities bitwise those of one lane.
template <int SCM, int LANES>
__global__ void __launch_bounds__(lanes_threads(LANES), 8 * TILE / lanes_threads(LANES))
    k_eam_density32_lanes(Dev D, PotParams P, const Blk32* blk) {
  constexpr int APB = lanes_atoms(LANES);
  __shared__ ShiftTable<> shifts;
  __shared__ long long rsum[APB];
  const Blk32 B = blk[blockIdx.x];
  const SysDev& S = D.sysd[B.sys];
  if (!S.active) return;  // whole block: its atoms belong to one system
  load_shifts(S, shifts);
  const ShiftCorr corr = shift_corr(S);
  const int lane = threadIdx.x & 31;
  const int sub = threadIdx.x % LANES, slot = (int)threadIdx.x / LANES;
  const float4* __restrict__ g32 = D.g32 + S.atom_base;
  const float rc2_lo = P.f[12], rc2_hi = P.f[13];
  const float scale = (float)FIX_RHO;
  unsigned rechecks = 0;
  const bool active = slot < B.count;
  const int li = B.first - (int)S.atom_base + (active ? slot : 0);
  const long long i = S.atom_base + li;
  const float4 gi = active ? g32[li] : make_float4(0.f, 0.f, 0.f, 0.f);
  const int cnt = active ? D.ncount[i] : 0;
  const int ng = (cnt + 3) >> 2;
  Fix rho;
  const uint4* L = active ? list_group(D, S, li, 0) : nullptr;
  for (int q = sub; q < ng; q += LANES) {
    const uint4 cur = __ldg(L + (long long)q * S.natoms);
    const unsigned e[4] = {cur.x, cur.y, cur.z, cur.w};
    const int rem = cnt - 4 * q;
    float4 gj[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) gj[u] = g32[e[u] & LOCAL_MASK];
    float part = 0.f;
    bool band = false;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool valid = u == 0 || rem > u;
      float dx, dy, dz;
      const float r2 = entry_r2(gi, gj[u], shifts[e[u] >> CODE_SHIFT], corr, dx, dy, dz);
      band = band || (valid && r2 >= rc2_lo && r2 < rc2_hi);
      const float v = eam_rho32_t<SCM>(P, r2);
      const float t = valid && r2 < rc2_lo ? v : 0.0f;
      part = u == 0 ? t : part + t;
    }
    rho.add(part * scale);
    if (band) {  // exact FP64 cutoff decision for the group's guard-band entries
      for (int u = 0; u < 4 && u < rem; ++u) {
        const int j = (int)(e[u] & LOCAL_MASK);
        float dx, dy, dz;
        const float r2 = entry_r2(gi, g32[j], shifts[e[u] >> CODE_SHIFT], corr, dx, dy, dz);
        if (!(r2 >= rc2_lo && r2 < rc2_hi)) continue;
        ++rechecks;
        if (exact_inside_cold(&D, &S, i, S.atom_base + j, P.rc2)) rho.add(eam_rho32_t<SCM>(P, r2) * scale);
      }
    }
  }
  lanes_sum<LANES>(rho);
  if (sub == 0 && active) rsum[slot] = rho.value();
  if (rechecks) atomicAdd(&D.sst[B.sys].rechecks, (unsigned long long)rechecks);
  __syncthreads();
  const int t = threadIdx.x;
  if (t >= ((B.count + 31) & ~31)) return;  // whole warps
  long long f = 0;
  if (t < B.count) {
    const long long a = B.first + t;
    const double r = (double)rsum[t] * (1.0 / FIX_RHO);
    double F, phi;
    eam_embed64(P, r, F, phi);
    D.rho[a] = r;
    D.phi[a] = phi;
    D.phif[a] = (float)phi;
    const float4 g = g32[a - S.atom_base];
    D.g32e[a] = make_float4(g.x, g.y, g.z, (float)((double)P.f[14] * phi));
    f = __double2ll_rn(F * FIX_E);
  }
  f = warp_sum(f);
  if (lane == 0) atomicAdd(D.sys_acc + (long long)B.sys * SA_LEN + SA_EEMBED, (unsigned long long)f);
}


// ------------------------------------------------------------------------------------------
// Tail of an FP64 force evaluation: sums the partial records of the system's blocks in a fixed
// order, a slot per thread (coalesced rows of 16 doubles), writes the thermo record and, inside a
// step sequence, decides the next step's rebuild (as k_tail does).  The sums are FP64 additions at 2
// a clock and SM -- 14 us for the 3,400 rows of a 108k system on one SM -- so the rows of a large
// system are shared by several blocks (about THERMO_SHARE each, by the system's own count) and the
// last of them to finish adds their sums up.
// ------------------------------------------------------------------------------------------

constexpr int THERMO_ROWS = 32;
constexpr int THERMO_SHARE = 128;
__host__ __device__ inline int thermo_shares(int rows) {
  if (rows <= 2 * THERMO_SHARE) return 1;
  const int n = (rows + THERMO_SHARE - 1) / THERMO_SHARE;
  return n < 64 ? n : 64;
}
__global__ void __launch_bounds__(PART_D * THERMO_ROWS) k_thermo(Dev D, int count_step, int decide_next,
                                                                 unsigned long long cond_next) {
  __shared__ double sh[THERMO_ROWS][PART_D];
  __shared__ int last;
  const int s = blockIdx.x;
  const long long n = D.sys64[s].y;
  const int parts = thermo_shares((int)n);
  const bool active = D.sysd[s].active;
  if ((int)blockIdx.y >= parts || (!active && blockIdx.y != 0)) return;
  if (active) {
    const int k = threadIdx.x % PART_D, row = threadIdx.x / PART_D;
    auto sum_rows = [&](const double* t, int lo, int hi) {
      double v = 0.0;
#pragma unroll 4
      for (int r = lo + row; r < hi; r += THERMO_ROWS) v += __ldcg(t + (long long)r * PART_D + k);
      sh[row][k] = v;
      __syncthreads();
      for (int h = THERMO_ROWS / 2; h > 0; h >>= 1) {
        if (row < h) sh[row][k] += sh[row + h][k];
        __syncthreads();
      }
    };
    sum_rows(D.part64 + (long long)D.sys64[s].x * PART_D, (int)(n * blockIdx.y / parts),
             (int)(n * (blockIdx.y + 1) / parts));
    if (parts > 1) {
      double* mine = D.share64 + (long long)s * gridDim.y * PART_D;
      if (row == 0) {
        __stcg(mine + blockIdx.y * PART_D + k, sh[0][k]);
        __threadfence();
      }
      __syncthreads();
      if (threadIdx.x == 0) last = atomicAdd(D.ticket64 + s, 1u) == (unsigned)parts - 1u;
      __syncthreads();
      if (!last) return;
      __threadfence();
      sum_rows(mine, 0, parts);
      if (threadIdx.x == 0) D.ticket64[s] = 0u;
    }
  }
  if (threadIdx.x >= 32) return;
  if (active) thermo_record(D, s, sh[0], count_step);
  if (decide_next && decide_system(D, s, 2, 0) && cond_next && threadIdx.x == 0)
    cudaGraphSetConditional((cudaGraphConditionalHandle)cond_next, 1u);
}

}  // namespace gbmd
