// force64.cuh -- the FP64 force and density passes (the plain path, every neighbour mode).
//
// What bounds them: GB300's FP64 unit takes 16 clocks per warp instruction and SM (2 lanes a
// clock), so the number of FP64 instructions a warp issues is the time; FP32, integer and memory
// work beside them is nearly free.  So
//   * candidates are tested in FP32 against a lower bound of their distance (list mode: the nearest
//     image from cell-relative offsets; stencil and all-pairs modes: truncated coordinates), and only
//     pairs that pass reach the FP64 unit, where the reference's own cutoff test decides those that
//     FP32 cannot.  FP32 can where a listed pair is inside by more than its error and every atom of the
//     system is in the box: the reference's distance is that of the image it reaches with a single
//     wrap, which for atoms outside may be box lengths further than the nearest;
//   * the passing pairs of an atom are queued in shared memory and shared out over the atom's
//     lanes, so that a warp's FP64 instructions run with nearly all lanes at work whatever the
//     lists' lengths (8 lanes an atom: an LJ liquid's 55 pairs fill 7 rounds of 8);
//   * energy and stress are summed from one end of each pair only (j > i), queued first, so that
//     the other half of the rounds leaves them out (18 FP64 instructions an LJ pair instead of 29);
//   * wraps and cutoff decisions compare bit patterns on the integer pipe, divisions and square
//     roots are one approximate start and one iteration, products feed fused multiply-adds, the
//     virial is the trace of the stress;
//   * small systems are cut into more blocks of fewer atoms, and into 32 lanes an atom, so that
//     every SM has work (a 864-atom system used to run on 7 SMs).
// How a system is cut depends on the system alone (plan64), so its sums have the same order in
// a batch and by itself.
//
// Measured on the GB300 against one thread per atom and every candidate in FP64: 54,743 copper
// atoms force 1553 -> 516 us, density 827 -> 277 us (FP64 unit 83 % busy while a block is resident);
// 31,899 atoms of LJ liquid 364 -> 134 us; 864 atoms, all pairs, 1243 -> 29 us a step (everything included).
#pragma once

#include "forces.cuh"
#include "pair64.cuh"

namespace gbmd {

constexpr int Q64_WARP = 1024;  // queue entries of a warp (split evenly over its atoms)
constexpr unsigned Q64_EXACT = 0x80000000u;

// x^n, n >= 0, by repeated squaring.
__device__ __forceinline__ double ipow64(double x, int n) {
  if (n == 0) return 1.0;
  while (!(n & 1)) {
    x *= x;
    n >>= 1;
  }
  double r = x;
  while (n >>= 1) {
    x *= x;
    if (n & 1) r *= x;
  }
  return r;
}

// ir^k for k > 0 from ir = 1/r and inv = 1/r^2.
__device__ __forceinline__ double ipow64_r(double ir, double inv, int k) {
  if (k & 1) return k == 1 ? ir : ipow64(inv, k >> 1) * ir;
  return ipow64(inv, k >> 1);
}

// x <= y for x, y >= 0 on the bit patterns.
__device__ __forceinline__ bool le_bits(double x, double y) {
  return __double_as_longlong(x) <= __double_as_longlong(y);
}

// rho_ij of the density pass; SCM = 6: Sutton-Chen with m = 6 without its a^m (applied to the sum).
template <int SCM>
__device__ __forceinline__ double rho_body64(const PotParams& P, const Pair64& c, double r2) {
  if (SCM == 6) {
    const double inv = rcp64(r2);
    return inv * inv * inv;
  }
  const double ir = rsqrt64(r2);
  if (P.kind == POT_SC) return P.am * (P.int_m >= 0 ? (P.int_m ? ipow64_r(ir, ir * ir, P.int_m) : 1.0) : pow(ir, P.p[3]));
  const double r = sqrt64(r2, ir);
  if (P.kind == POT_GUPTA) return exp(c.c1 * (r - P.p[1]));
  const double d = P.kind == POT_FS ? P.p[6] : P.p[8];
  if (!le_bits(r, d)) return 0.0;
  const double rd = r - d, t = rd * rd;
  return t * fma(c.c0, P.kind == POT_FS ? rd : t, 1.0);
}

// Pair and many-body force of a metal: g with F_i = g r_ij, the pair's energy added to ep
// if `count`.  phi: the sum of both atoms' embedding factors as the density pass
// stores them (times c.phi).  SCN = 9 or 12: Sutton-Chen with m = 6; 0: any.
template <int SCN>
__device__ __forceinline__ double eam_body64(const PotParams& P, const Pair64& c, double r2, double phi, bool count,
                                             double& ep) {
  if (SCN == 12) {  // even powers only
    const double inv = rcp64(r2);
    const double i2 = inv * inv, i4 = i2 * i2;  // r^-4, r^-8 = r^-(m+2)
    if (count) ep = fma(c.c0, i4 * i2, ep);
    return i4 * fma(c.c1, i2 * inv, phi);
  }
  const double ir = rsqrt64(r2);
  if (SCN == 9) {
    const double inv = ir * ir;
    const double i2 = inv * inv, i4 = i2 * i2;
    if (count) ep = fma(c.c0, i4 * ir, ep);
    return i4 * fma(c.c1, ir * inv, phi);
  }
  if (P.kind == POT_SC) {
    const double inv = ir * ir;
    const double pn = P.int_n >= 0 ? (P.int_n ? ipow64_r(ir, inv, P.int_n) : 1.0) : pow(ir, P.p[2]);
    const double pm = P.int_m >= 0 ? ipow64_r(ir, inv, P.int_m + 2) : pow(ir, P.p[3] + 2.0);
    if (count) ep = fma(c.c0, pn, ep);
    return fma(c.c1, pn * inv, phi * pm);
  }
  const double r = sqrt64(r2, ir);
  if (P.kind == POT_GUPTA) {
    const double dr = r - P.p[1];
    const double ex = exp(c.c0 * dr);
    if (count) ep = fma(P.p[0], ex, ep);
    return fma(c.c2, ex, phi * exp(c.c1 * dr)) * ir;
  }
  const bool fs = P.kind == POT_FS;
  const double rc = r - (fs ? P.p[5] : P.p[7]), rd = r - (fs ? P.p[6] : P.p[8]);
  double s = 0.0;
  if (rc <= 0.0) {
    double poly, dpoly;
    if (fs) {
      poly = fma(fma(P.p[2], r, P.p[1]), r, P.p[0]);
      dpoly = fma(c.c3, r, P.p[1]);
    } else {
      poly = fma(fma(fma(fma(P.p[4], r, P.p[3]), r, P.p[2]), r, P.p[1]), r, P.p[0]);
      dpoly = fma(fma(fma(4.0 * P.p[4], r, 3.0 * P.p[3]), r, c.c3), r, P.p[1]);
    }
    if (count) ep = fma(rc * rc, poly, ep);
    s = rc * fma(rc, dpoly, 2.0 * poly);
  }
  if (rd <= 0.0) s = fma(phi * rd, fma(c.c1, fs ? rd : rd * rd, 2.0), s);
  return s * ir;
}

// The candidates of one atom (the calling lane's), tested in FP32 and queued: entry = local index of
// j, plus Q64_EXACT where the FP64 test has to decide.  All lanes of the warp call this together; the
// lanes of an atom share its queue `q` of cap entries: those with j > i from the front, the others
// from the back.  drain(nf, nb) consumes the nf front and nb back entries of the atom; it is called
// whenever some atom's queue could overflow, and at the end.
template <int NB, class SH, class F>
__device__ __forceinline__ void scan64(const Dev& D, const SysDev& S, int s, int li, bool active, int lanes, int sub,
                                       unsigned* q, int cap, const SH& shifts, double rc2, float lo,
                                       float hi, int spc_sum, F&& drain) {
  const unsigned all = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int at = lane - sub;  // first lane of the atom
  const unsigned mine = (lanes == 32 ? all : ((1u << lanes) - 1u)) << at;
  const unsigned below = mine & ((1u << lane) - 1u);
  int nf = 0, nb = 0;
  auto push = [&](bool in, unsigned e) {
    const bool front = (int)(e & LOCAL_MASK) > li;
    const unsigned mf = __ballot_sync(all, in && front), mb = __ballot_sync(all, in && !front);
    if (in) q[front ? nf + __popc(mf & below) : cap - 1 - (nb + __popc(mb & below))] = e;
    nf += __popc(mf & mine);
    nb += __popc(mb & mine);
  };
  auto flush = [&](int room) {
    if (__any_sync(all, nf + nb + room > cap)) {
      __syncwarp();
      drain(nf, nb);
      __syncwarp();
      nf = nb = 0;
    }
  };
  const long long i = S.atom_base + li;
  const int ti = (spc_sum >= 0 && active) ? D.type[i] : 0;
  auto species_ok = [&](int j) { return spc_sum < 0 || ti + D.type[S.atom_base + j] == spc_sum; };
  if (NB == NB_LIST) {
    const ShiftCorr corr = shift_corr(S);
    const float4* __restrict__ g32 = D.g32 + S.atom_base;
    const float4 gi = active ? g32[li] : make_float4(0.f, 0.f, 0.f, 0.f);
    const int cnt = active ? D.ncount[i] : 0;
    // The entry's image was the nearest when the list was built; on the clock of an `each` manager it
    // need not be any more, so each component is folded once (exact where it does not fold).  A
    // component is off by at most tol: roundings of the two offsets (box lengths, for atoms far
    // outside), the shift, the box edge and their sums.
    const float Lx = (float)S.L[0], Ly = (float)S.L[1], Lz = (float)S.L[2];
    const float tol = 1e-6f * (fmaxf(fabsf(gi.x), fmaxf(fabsf(gi.y), fabsf(gi.z))) + fmaxf(Lx, fmaxf(Ly, Lz)));
    const float band = tol * fmaf(3.5f, sqrtf(hi), 3.0f * tol);  // (sqrt(hi) + sqrt(3) tol)^2 - hi
    const float near2 = D.outside[s] ? -1.0f : lo - band, far2 = hi + band;
    auto fold = [](float d, float L) { return fminf(fabsf(d), fabsf(fabsf(d) - L)); };
    const int ng = (cnt + 3) >> 2;
    const int ngw = (int)__reduce_max_sync(all, (unsigned)ng);
    const uint4* L = list_group(D, S, li, 0);
    for (int r = 0; r < ngw; r += lanes) {
      const int g = r + sub;
      const uint4 e4 = g < ng ? __ldg(L + (long long)g * S.natoms) : make_uint4(0u, 0u, 0u, 0u);
      const unsigned e[4] = {e4.x, e4.y, e4.z, e4.w};
      flush(4 * lanes);
      bool in[4];
      unsigned w[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const bool valid = 4 * g + u < cnt;
        const unsigned j = e[u] & LOCAL_MASK;
        const float4 gj = valid ? g32[j] : gi;
        float dx, dy, dz;
        entry_r2(gi, gj, shifts[e[u] >> CODE_SHIFT], corr, dx, dy, dz);
        dx = fold(dx, Lx);
        dy = fold(dy, Ly);
        dz = fold(dz, Lz);
        const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
        in[u] = valid && r2 < far2 && (spc_sum < 0 || applies_to(spc_sum, __float_as_int(gi.w), __float_as_int(gj.w)));
        w[u] = j | (r2 >= near2 ? Q64_EXACT : 0u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) push(in[u], w[u]);
    }
  } else {
    // lower bound of the reference's distance
    const double4_32a pi = active ? D.g64[i] : make_double4_32a(0., 0., 0., 0.);
    const float xi = trunc32(pi.x), yi = trunc32(pi.y), zi = trunc32(pi.z);
    const float Lx = (float)S.L[0], Ly = (float)S.L[1], Lz = (float)S.L[2];
    const float rc2up = (float)rc2 * 1.000002f;
    auto near = [&](const double4_32a& pj) {
      const float dx = axis_bound(xi, trunc32(pj.x), Lx), dy = axis_bound(yi, trunc32(pj.y), Ly),
                  dz = axis_bound(zi, trunc32(pj.z), Lz);
      return !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > rc2up);
    };
    if (NB == NB_CELLS) {
      // the reference stencil of LinkedCell (plugins/linkedcell.cc:221-240), duplicates included,
      // one stencil cell a lane
      const int h = active ? D.home[i] - S.cell_base : 0;
      const int cx = h % S.n[0], cy = (h / S.n[0]) % S.n[1], cz = h / (S.n[0] * S.n[1]);
      const int sd = S.lc_side, w = 2 * sd + 1, ncell = w * w * w;
      for (int c0 = 0; c0 < ncell; c0 += lanes) {
        const int c = c0 + sub;
        int b = 0, m = 0;
        if (active && c < ncell) {
          const int xc = wrap_around(cx + c % w - sd, S.n[0]), yc = wrap_around(cy + (c / w) % w - sd, S.n[1]),
                    zc = wrap_around(cz + c / (w * w) - sd, S.n[2]);
          const int g = S.cell_base + (zc * S.n[1] + yc) * S.n[0] + xc;
          b = D.cstart[g] - (int)S.atom_base;
          m = D.ccnt[g];
        }
        const int mw = (int)__reduce_max_sync(all, (unsigned)m);
        for (int k = 0; k < mw; ++k) {
          flush(lanes);
          const int j = b + k;
          push(k < m && j != li && near(D.g64[S.atom_base + j]) && species_ok(j), (unsigned)j | Q64_EXACT);
        }
      }
    } else {
      // four candidates a lane at a time: their loads overlap
      const int na = S.natoms;
      for (int j0 = 0; j0 < na; j0 += 4 * lanes) {
        flush(4 * lanes);
        double4_32a pj[4];
        bool in[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u * lanes + sub;
          in[u] = active && j < na && j != li;
          pj[u] = D.g64[S.atom_base + (j < na ? j : li)];
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) in[u] = in[u] && near(pj[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int j = j0 + u * lanes + sub;
          push(in[u] && species_ok(j), (unsigned)j | Q64_EXACT);
        }
      }
    }
  }
  __syncwarp();
  drain(nf, nb);
  __syncwarp();
}

// Entry k of a queue with nf front entries.
__device__ __forceinline__ unsigned queued64(const unsigned* q, int cap, int nf, int k) {
  return q[k < nf ? k : cap - 1 - (k - nf)];
}

// r_ij and its square in the reference's operation order or, where the pair is known to be inside,
// with fused multiply-adds.  (One more test of the wrapped components here, in place of the flag
// D.outside, cost 4 % of the force passes and 9 % of the density pass; the exact test of every pair
// on the bits of the fused r^2 14 % of the LJ force pass.)
__device__ __forceinline__ bool pair_geometry64(const double4_32a& pi, const double4_32a& pj, const SysDev& S,
                                                const long long (&lhb)[3], long long rc2b, bool exact, bool ref,
                                                double& dx, double& dy, double& dz, double& r2) {
  dx = dsub(pj.x, pi.x);
  dy = dsub(pj.y, pi.y);
  dz = dsub(pj.z, pi.z);
  const bool wx = wraps_bits(dx, lhb[0]), wy = wraps_bits(dy, lhb[1]), wz = wraps_bits(dz, lhb[2]);
  if (wx || wy || wz) {
    if (wx) dx = dsub(dx, copysign(S.L[0], dx));
    if (wy) dy = dsub(dy, copysign(S.L[1], dy));
    if (wz) dz = dsub(dz, copysign(S.L[2], dz));
  }
  if (exact) {
    r2 = ref_sq(dx, dy, dz);
    // r2 < rc2 on the bit patterns (both are >= 0; a NaN's bits are above any rc2)
    if (!(__double_as_longlong(r2) >= 0 && __double_as_longlong(r2) < rc2b)) return false;
    if (ref) return true;
  }
  r2 = ref ? ref_sq(dx, dy, dz) : fma(dx, dx, fma(dy, dy, dz * dz));
  return true;
}

template <int NB, int PC, int SCN>
__global__ void __launch_bounds__(TILE, 5) k_force64(Dev D, PotParams P, Pair64 c, StepParams sp) {
  __shared__ unsigned queue[TILE / 32][Q64_WARP];
  __shared__ double fs[3][TILE];
  __shared__ double red[TILE / 32][16];
  __shared__ ShiftTable<NB == NB_LIST ? 125 : 1> shifts;
  const Blk64 B = D.blk64[blockIdx.x];
  const SysDev& S = D.sysd[B.sys];
  if (!S.active) {
    if (sp.epi == EPI_KICK_DRIFT && sp.last) hold_range(D, S, B.first, B.count, true);
    return;
  }
  if constexpr (NB == NB_LIST) load_shifts(S, shifts);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lanes = B.lanes, sub = lane & (lanes - 1), slot = lane / lanes, per = 32 / lanes;
  const int cap = Q64_WARP / per;
  unsigned* const q = queue[w] + slot * cap;
  const long long lhb[3] = {__double_as_longlong(S.Lh[0]), __double_as_longlong(S.Lh[1]), __double_as_longlong(S.Lh[2])};
  const long long rc2b = __double_as_longlong(P.rc2);
  const bool tabulated = PC == PC_PAIR && P.kind == POT_FASTLJ;  // its bin needs the reference's r^2
  double ep = 0.0, sxx = 0.0, sxy = 0.0, sxz = 0.0, syy = 0.0, syz = 0.0, szz = 0.0;
  const int w0 = w * B.apw;                                // the warp's first atom within the block
  const int wn = min(B.apw, max(0, B.count - w0));         // and how many it has
  for (int g = 0; g < wn; g += per) {
    const bool active = g + slot < wn;
    const int li = B.first - (int)S.atom_base + w0 + (active ? g + slot : 0);
    const double4_32a pi = D.g64[S.atom_base + li];
    const double phi_i = PC == PC_EAM ? D.phi[S.atom_base + li] : 0.0;
    double fx = 0.0, fy = 0.0, fz = 0.0;
    scan64<NB>(D, S, B.sys, li, active, lanes, sub, q, cap, shifts, P.rc2, P.f[12], P.f[13], P.spc_sum, [&](int nf, int nb) {
      for (int k = sub; k < nf + nb; k += lanes) {
        const unsigned e = queued64(q, cap, nf, k);
        const long long j = S.atom_base + (e & LOCAL_MASK);
        double dx, dy, dz, r2;
        if (!pair_geometry64(pi, D.g64[j], S, lhb, rc2b, (e & Q64_EXACT) != 0u, tabulated, dx, dy, dz, r2)) continue;
        const bool count = k < nf;  // this end of the pair adds its energy and stress
        double gg;
        if (PC == PC_EAM) {
          gg = eam_body64<SCN>(P, c, r2, phi_i + D.phi[j], count, ep);
        } else if (tabulated) {
          double en;
          fastlj_pair64(P, r2, gg, en);
          if (count) ep += en;
        } else {
          gg = lj_body64(c, r2, count, ep);
        }
        fx = fma(gg, dx, fx);
        fy = fma(gg, dy, fy);
        fz = fma(gg, dz, fz);
        if (count) {
          const double gx = gg * dx, gy = gg * dy, gz = gg * dz;
          sxx = fma(gx, dx, sxx);
          sxy = fma(gx, dy, sxy);
          sxz = fma(gx, dz, sxz);
          syy = fma(gy, dy, syy);
          syz = fma(gy, dz, syz);
          szz = fma(gz, dz, szz);
        }
      }
    });
    const double f = atom_sum3(fx, fy, fz, sub, lanes);
    const int comp = sub / (lanes >> 2);
    if (active && comp < 3 && (sub & ((lanes >> 2) - 1)) == 0) fs[comp][w0 + g + slot] = f;
  }
  __syncthreads();
  // one thread per atom of the block, in as few warps as hold them
  double ke = 0.0, px = 0.0, py = 0.0, pz = 0.0;
  float d2 = 0.0f;
  const int t = threadIdx.x;
  if (t < B.count) {
    const long long i = B.first + t, N = D.N;
    double fx = fs[0][t], fy = fs[1][t], fz = fs[2][t];
    if (!sp.first) {
      fx += D.dacc[i];
      fy += D.dacc[N + i];
      fz += D.dacc[2 * N + i];
    }
    if (sp.last) {
      d2 = finish_atom<0>(D, S, i, fx, fy, fz, sp, ke, px, py, pz);
    } else {
      D.dacc[i] = fx;
      D.dacc[N + i] = fy;
      D.dacc[2 * N + i] = fz;
    }
  }
  track_displacement_warp(D, B.sys, d2);
  double v[16] = {ep, sxx, sxy, sxz, syy, syz, szz, ke, px, py, pz, 0.0, 0.0, 0.0, 0.0, 0.0};
  const double s = warp_sums(v);
  if ((lane & 1) == 0) red[w][lane >> 1] = s;
  __syncthreads();
  if (threadIdx.x < 11) {
    double x = red[0][threadIdx.x];
    for (int k = 1; k < TILE / 32; ++k) x += red[k][threadIdx.x];
    red[0][threadIdx.x] = x;
  }
  __syncthreads();
  if (threadIdx.x < PART_D) {
    // slots of the partial record and the sums they come from (the virial is the trace of the
    // stress)
    constexpr signed char from[PART_D] = {0, -1, -2, 1, 2, 3, 2, 4, 5, 3, 5, 6, 7, 8, 9, 10};
    const int k = (int)threadIdx.x;
    double* out = D.part64 + (long long)blockIdx.x * PART_D + k;
    double x = 0.0;
    if (k == PD_EPAIR)
      x = red[0][0];
    else if (k == PD_VIR)
      x = -(red[0][1] + red[0][4] + red[0][6]);
    else if (k >= PD_STRESS && k < PD_KE)
      x = -red[0][from[k]];
    if (k == PD_EEMBED) {
      // the density pass wrote it
    } else if (k < PD_KE) {
      *out = sp.first ? x : *out + x;
    } else if (sp.last) {
      *out = red[0][from[k]];
    }
  }
}

// FP64 density pass and embedding: rho_i over the atom's pairs, F(rho) and 1/sqrt(rho).
template <int NB, int SCM>
__global__ void __launch_bounds__(TILE, 8) k_eam_density(Dev D, PotParams P, Pair64 c, int first) {
  __shared__ unsigned queue[TILE / 32][Q64_WARP];
  __shared__ double rs[TILE];
  __shared__ ShiftTable<NB == NB_LIST ? 125 : 1> shifts;
  const Blk64 B = D.blk64[blockIdx.x];
  const SysDev& S = D.sysd[B.sys];
  if (!S.active) return;
  if constexpr (NB == NB_LIST) load_shifts(S, shifts);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lanes = B.lanes, sub = lane & (lanes - 1), slot = lane / lanes, per = 32 / lanes;
  const int cap = Q64_WARP / per;
  unsigned* const q = queue[w] + slot * cap;
  const long long lhb[3] = {__double_as_longlong(S.Lh[0]), __double_as_longlong(S.Lh[1]), __double_as_longlong(S.Lh[2])};
  const long long rc2b = __double_as_longlong(P.rc2);
  const int w0 = w * B.apw;
  const int wn = min(B.apw, max(0, B.count - w0));
  for (int g = 0; g < wn; g += per) {
    const bool active = g + slot < wn;
    const int li = B.first - (int)S.atom_base + w0 + (active ? g + slot : 0);
    const double4_32a pi = D.g64[S.atom_base + li];
    double rho = 0.0;
    scan64<NB>(D, S, B.sys, li, active, lanes, sub, q, cap, shifts, P.rc2, P.f[12], P.f[13], -1, [&](int nf, int nb) {
      for (int k = sub; k < nf + nb; k += lanes) {
        const unsigned e = queued64(q, cap, nf, k);
        double dx, dy, dz, r2;
        if (pair_geometry64(pi, D.g64[S.atom_base + (e & LOCAL_MASK)], S, lhb, rc2b, (e & Q64_EXACT) != 0u, false, dx, dy,
                            dz, r2))
          rho += rho_body64<SCM>(P, c, r2);
      }
    });
    for (int m = lanes >> 1; m > 0; m >>= 1) rho += __shfl_xor_sync(0xffffffffu, rho, m);
    if (active && sub == 0) rs[w0 + g + slot] = rho;
  }
  __syncthreads();
  double F = 0.0;
  if ((int)threadIdx.x < B.count) {
    const long long i = B.first + threadIdx.x;
    const double rho = SCM == 6 ? P.am * rs[threadIdx.x] : rs[threadIdx.x];
    double phi;
    eam_embed64(P, rho, F, phi);
    D.rho[i] = rho;
    D.phi[i] = c.phi * phi;
  }
  double v[1] = {F};
  double t[1];
  block_sum<double, 1>(v, t);
  if (threadIdx.x == 0) {
    double* td = D.part64 + (long long)blockIdx.x * PART_D;
    td[PD_EEMBED] = first ? t[0] : td[PD_EEMBED] + t[0];
  }
}

}  // namespace gbmd
