// Pair forces of one small periodic system without any device allocation.
//
// The FP64 all-pairs pair-force pass (the minimum-image path of force64.cuh) rewritten so that its
// only scratch -- the per-block partial sums of energy, virial and stress -- lives in a fixed
// file-scope device array instead of the engine's allocated pools.  The caller brings the positions
// and receives forces and sums in device buffers it owns; this file allocates nothing, at set-up or
// per call.
//
// The first call on a device may load the module.  Calls from several host threads or streams share
// the one array per device and therefore must not overlap in time on the same device.

#include <cuda_runtime.h>

#include <string>

#include "../../include/gbmd.h"
#include "device.cuh"
#include "engine.h"
#include "pair64.cuh"

namespace gbmd {

namespace {

constexpr int ST_WARPS = 4;
constexpr int ST_MAX_ATOMS = GBMD_STATIC_MAX_ATOMS;
constexpr int ST_MAX_BLOCKS = 608;  // four for each of the 152 SMs
constexpr int ST_PART = 11;         // pair energy, virial, stress (9)

// Per-block partial sums.  Each call's force launch writes the slots of every block it runs before
// the reduction launch reads them, so nothing in the array has to start at zero and nothing is
// carried from one call to the next.
static __device__ __align__(256) double g_static_scratch[ST_MAX_BLOCKS * 8];

// One warp per atom (apw of them in turn): the lanes test 32 other atoms at a time in FP32, in index
// order, those that may be inside queue up, and every 32 of them go through the FP64 unit with all
// lanes at work.  The reference visits each pair once (j > i, plugins/minimumimage.cc:91) and applies
// the pair force to both atoms (liblpmd/simulation/pairpotential.cc:50-75); here each pair is seen
// from both ends, and the one with j > i adds energy and stress.  Bound by latency at a hundred
// atoms, by the FP32 tests of all pairs at thousands.  (One thread per atom, every candidate through
// the FP64 unit, on one SM per 128 atoms: 315 us a call for 108 atoms, 1,610 for 500; 14 and 19 so.)
__global__ void __launch_bounds__(32 * ST_WARPS)
    k_pair_forces_static(Pair64 c, double rc2, const double* __restrict__ pos, int n, int apw, double Lx, double Ly,
                         double Lz, double* __restrict__ force) {
  __shared__ int queue[ST_WARPS][64];
  __shared__ double red[ST_WARPS][8];
  const unsigned all = 0xffffffffu;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
  int* const q = queue[w];
  const long long hx = __double_as_longlong(0.5 * Lx), hy = __double_as_longlong(0.5 * Ly),
                  hz = __double_as_longlong(0.5 * Lz), rc2b = __double_as_longlong(rc2);
  const float fLx = (float)Lx, fLy = (float)Ly, fLz = (float)Lz, rc2up = (float)rc2 * 1.000002f;
  double ep = 0.0, sxx = 0.0, sxy = 0.0, sxz = 0.0, syy = 0.0, syz = 0.0, szz = 0.0;
  const int i0 = (blockIdx.x * ST_WARPS + w) * apw;
  for (int i = i0; i < min(i0 + apw, n); ++i) {
    const double xi = pos[3 * i], yi = pos[3 * i + 1], zi = pos[3 * i + 2];
    const float tx = trunc32(xi), ty = trunc32(yi), tz = trunc32(zi);
    double fx = 0.0, fy = 0.0, fz = 0.0;
    auto drain = [&](int m) {  // the queue's first m <= 32 entries
      __syncwarp();
      if (lane < m) {
        const int j = q[lane];
        double dx = dsub(pos[3 * j], xi), dy = dsub(pos[3 * j + 1], yi), dz = dsub(pos[3 * j + 2], zi);
        if (wraps_bits(dx, hx)) dx = dsub(dx, copysign(Lx, dx));
        if (wraps_bits(dy, hy)) dy = dsub(dy, copysign(Ly, dy));
        if (wraps_bits(dz, hz)) dz = dsub(dz, copysign(Lz, dz));
        // the reference's test: r^2 in its operation order, compared on the bit patterns
        const long long r2b = __double_as_longlong(ref_sq(dx, dy, dz));
        if (r2b >= 0 && r2b < rc2b) {
          const bool count = j > i;
          const double g = lj_body64(c, fma(dx, dx, fma(dy, dy, dz * dz)), count, ep);
          fx = fma(g, dx, fx);
          fy = fma(g, dy, fy);
          fz = fma(g, dz, fz);
          if (count) {
            const double gx = g * dx, gy = g * dy, gz = g * dz;
            sxx = fma(gx, dx, sxx);
            sxy = fma(gx, dy, sxy);
            sxz = fma(gx, dz, sxz);
            syy = fma(gy, dy, syy);
            syz = fma(gy, dz, syz);
            szz = fma(gz, dz, szz);
          }
        }
      }
      __syncwarp();
    };
    int nq = 0;
#pragma unroll 4
    for (int j0 = 0; j0 < n; j0 += 32) {
      const int j = j0 + lane;
      bool in = false;
      if (j < n && j != i) {
        const float dx = axis_bound(tx, trunc32(pos[3 * j]), fLx), dy = axis_bound(ty, trunc32(pos[3 * j + 1]), fLy),
                    dz = axis_bound(tz, trunc32(pos[3 * j + 2]), fLz);
        in = !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > rc2up);
      }
      const unsigned m = __ballot_sync(all, in);
      if (in) q[nq + __popc(m & below)] = j;
      nq += __popc(m);
      if (nq >= 32) {
        drain(32);
        const int rest = lane < nq - 32 ? q[32 + lane] : 0;
        __syncwarp();
        if (lane < nq - 32) q[lane] = rest;
        nq -= 32;
      }
    }
    if (nq > 0) drain(nq);
    const double f = atom_sum3(fx, fy, fz, lane, 32);
    if ((lane & 7) == 0 && lane < 24) force[3 * i + (lane >> 3)] = f;
  }
  double v[16] = {ep, sxx, sxy, sxz, syy, syz, szz, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  const double t = warp_sums(v);
  if ((lane & 1) == 0 && lane < 16) red[w][lane >> 1] = t;
  __syncthreads();
  if (threadIdx.x < 8) {
    double s = red[0][threadIdx.x];
    for (int k = 1; k < ST_WARPS; ++k) s += red[k][threadIdx.x];
    g_static_scratch[blockIdx.x * 8 + threadIdx.x] = s;
  }
}

// Sums the blocks' partials in a fixed order: 8 slots by 32 rows.
__global__ void __launch_bounds__(256) k_pair_sums_static(int nblocks, double* __restrict__ out) {
  __shared__ double sh[32][8];
  const int k = threadIdx.x & 7, row = threadIdx.x >> 3;
  double s = 0.0;
  for (int b = row; b < nblocks; b += 32) s += g_static_scratch[b * 8 + k];
  sh[row][k] = s;
  __syncthreads();
  for (int h = 16; h > 0; h >>= 1) {
    if (row < h) sh[row][k] += sh[row + h][k];
    __syncthreads();
  }
  if (threadIdx.x >= ST_PART) return;
  // energy, virial (the trace of the stress), stress
  constexpr signed char from[ST_PART] = {0, 0, 1, 2, 3, 2, 4, 5, 3, 5, 6};
  const double* t = sh[0];
  out[threadIdx.x] = threadIdx.x == 0 ? t[0] : threadIdx.x == 1 ? -(t[1] + t[4] + t[6]) : -t[from[threadIdx.x]];
}

}  // namespace

void pair_forces_static(const PotParams& P, const double* pos, int n, const double* box, double* force, double* out,
                        void* stream_handle) {
  cudaStream_t stream = (cudaStream_t)stream_handle;
  if (n < 1 || n > ST_MAX_ATOMS)
    throw Error(GBMD_ERR_INVALID, "gbmd_pair_forces_static: n = " + std::to_string(n) +
                                      " atoms is outside 1.." + std::to_string(ST_MAX_ATOMS) +
                                      ", the capacity of its fixed scratch array");
  if (P.kind != POT_LJ)
    throw Error(GBMD_ERR_INVALID, "gbmd_pair_forces_static: only pair potentials (lennardjones) are supported");
  for (int a = 0; a < 3; ++a)
    if (!(box[a] > 0.0)) throw Error(GBMD_ERR_INVALID, "gbmd_pair_forces_static: box lengths must be positive");
  // an atom a warp while the grid has blocks left for them
  const int apw = (n + ST_WARPS * ST_MAX_BLOCKS - 1) / (ST_WARPS * ST_MAX_BLOCKS);
  const int nblocks = (n + ST_WARPS * apw - 1) / (ST_WARPS * apw);
  k_pair_forces_static<<<nblocks, 32 * ST_WARPS, 0, stream>>>(pair64_constants(P), P.rc2, pos, n, apw, box[0], box[1],
                                                              box[2], force);
  k_pair_sums_static<<<1, 256, 0, stream>>>(nblocks, out);
  cudaError_t rc = cudaGetLastError();
  if (rc != cudaSuccess)
    throw Error(GBMD_ERR_CUDA, std::string("gbmd_pair_forces_static launch: ") + cudaGetErrorString(rc));
}

}  // namespace gbmd
