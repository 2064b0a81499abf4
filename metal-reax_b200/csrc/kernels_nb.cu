// Cell lists, full neighbor rows with the charge matrix, non-bonded forces, charge-equilibration CG, energy sums.
#include <cooperative_groups.h>

#include <type_traits>
#include <utility>

#include "device.cuh"
#include "kernels.hpp"

namespace cg = cooperative_groups;

namespace rx {

// ------------------------------------------------------------------------------------------------ Verlet check
// A system's Verlet rows stay valid while no atom of it has moved more than skin/2 since they were built (no pair can
// then have come from beyond nonb_cut + skin to within nonb_cut). Sets the system's rebuild flag otherwise.
__global__ void k_nbr_check(Dev d) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= d.na) return;
  // this evaluation's H-bond acceptor accumulators and per-atom energy tallies start from zero (the first kernel of an
  // evaluation: the bonded branch may start before the row filter)
  for (int c = 0; c < 3; ++c) d.fix_h[3 * static_cast<size_t>(a) + c] = 0ull;
  if (d.pe_on) d.pe_fix[a] = 0ull;
  const int s = d.sys_of[a];
  const int p = d.rank[a], ta = d.type[a];
  const double4 x = d.x[a];
  // the cell-ordered copies of the pair phase (a rebuild, which changes the order, writes them again: k_cell_start)
  d.xr[p] = ord_pack(x, ta, a);
  d.qr[p] = d.q[a];
  if (!(isfinite(x.x) && isfinite(x.y) && isfinite(x.z))) {
    atomicOr(d.status, ST_NONFINITE);
    return;
  }
  if (*reinterpret_cast<volatile const int*>(d.sys_flag + s)) return;
  const double4 r = d.xref[a];
  double dx = x.x - r.x, dy = x.y - r.y, dz = x.z - r.z;
  {   // positions handed in by a caller may sit in another periodic image than the engine's own (wrapped at the last
      // rebuild): the atom moves to the image nearest its reference position, so that the rows' lattice shifts hold
    const SysInfo& sy = d.sys[s];
    double n[3];
    bool shift = false;
    for (int k = 0; k < 3; ++k) {
      n[k] = sy.per[k] ? rint(sy.R[3 * k] * dx + sy.R[3 * k + 1] * dy + sy.R[3 * k + 2] * dz) : 0.0;
      shift = shift || n[k] != 0.0;
    }
    if (shift) {
      double4 y = x;
      y.x -= n[0] * sy.L[0] + n[1] * sy.L[3] + n[2] * sy.L[6];
      y.y -= n[0] * sy.L[1] + n[1] * sy.L[4] + n[2] * sy.L[7];
      y.z -= n[0] * sy.L[2] + n[1] * sy.L[5] + n[2] * sy.L[8];
      d.x[a] = y;
      d.xr[p] = ord_pack(y, ta, a);
      dx = y.x - r.x; dy = y.y - r.y; dz = y.z - r.z;
    }
  }
  if (dx * dx + dy * dy + dz * dz > d.half_skin2) atomicOr(d.sys_flag + s, 1);
}

// ------------------------------------------------------------------------------------------------ wrap + bin
// Atoms of systems being rebuilt are wrapped into the primary cell first (expand_images with wrap_owned,
// src/neighbor/neighbor.cpp:45-61), then binned into a uniform grid over the fractional coordinates of their system.
// Between rebuilds positions are never re-wrapped: the lattice shifts in the rows are relative to the positions of
// the last rebuild.
__global__ void k_wrap_bin(Dev d) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x;
  if (a >= d.na) return;
  const int sy = d.sys_of[a];
  if (!d.sys_flag[sy]) return;   // the atom keeps its key: its system's cells are not used this evaluation
  const SysInfo s = d.sys[sy];
  double4 x = d.x[a];
  double r[3] = {x.x, x.y, x.z};
  double f[3];
  for (int k = 0; k < 3; ++k) f[k] = s.R[3 * k] * (r[0] - s.origin[0]) + s.R[3 * k + 1] * (r[1] - s.origin[1]) + s.R[3 * k + 2] * (r[2] - s.origin[2]);
  bool moved = false;
  for (int k = 0; k < 3; ++k) {
    const double fl = floor(f[k]);
    if (fl != 0.0) {
      if (!s.per[k]) {   // never wrapped: the atom has left the extent the engine laid out for this direction
        atomicOr(d.status, ST_NONPERIODIC_ESCAPE);
        continue;
      }
      for (int c = 0; c < 3; ++c) r[c] -= fl * s.L[3 * k + c];
      moved = true;
    }
  }
  if (moved) {
    for (int k = 0; k < 3; ++k) f[k] = s.R[3 * k] * (r[0] - s.origin[0]) + s.R[3 * k + 1] * (r[1] - s.origin[1]) + s.R[3 * k + 2] * (r[2] - s.origin[2]);
    x.x = r[0]; x.y = r[1]; x.z = r[2];
    d.x[a] = x;
  }
  d.xref[a] = x;
  if (!(isfinite(r[0]) && isfinite(r[1]) && isfinite(r[2]))) atomicOr(d.status, ST_NONFINITE);
  int c[3];
  for (int k = 0; k < 3; ++k) {
    int v = static_cast<int>(floor(f[k] * s.nc[k]));
    v = v < 0 ? 0 : (v >= s.nc[k] ? s.nc[k] - 1 : v);
    c[k] = v;
  }
  d.cell_key[a] = s.cell_begin + (c[2] * s.nc[1] + c[1]) * s.nc[0] + c[0];
}

// Sets the captured evaluation's rebuild conditional: 1 when any system's Verlet rows are to be rebuilt (its flag set
// by k_nbr_check or by the host), 0 otherwise, so that the wrap/bin, sort, cell-start and row kernels are skipped.
__global__ void k_rebuild_flag(Dev d, cudaGraphConditionalHandle h) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  int mine = 0;
  for (int s = threadIdx.x; s < d.nsys; s += blockDim.x) mine |= d.sys_flag[s];
  if (mine) atomicOr(&any, 1);
  __syncthreads();
  if (threadIdx.x == 0) cudaGraphSetConditional(h, any ? 1u : 0u);
}

// cell_start[c] = first position in the sorted order whose key is >= c; the atoms' ranks and cell-ordered positions and
// charges; and positions relative to their system's origin and rounded to single precision (the candidate scan of the
// Verlet rows reads only these)
__global__ void k_cell_start(Dev d, const int* sorted_keys) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > d.na) return;
  const int prev = p == 0 ? -1 : sorted_keys[p - 1];
  const int cur = p == d.na ? d.ncell_total : sorted_keys[p];
  for (int c = prev + 1; c <= cur; ++c) d.cell_start[c] = p;
  if (p < d.na) {
    const int a = d.cell_atoms[p];
    const double4 x = d.x[a];
    d.rank[a] = p;
    d.xr[p] = ord_pack(x, d.type[a], a);
    d.qr[p] = d.q[a];
    const double* o = d.sys[d.sys_of[a]].origin;
    d.xs[p] = make_float4(static_cast<float>(x.x - o[0]), static_cast<float>(x.y - o[1]), static_cast<float>(x.z - o[2]),
                          static_cast<float>(d.type[a]));
  }
}

// ------------------------------------------------------------------------------------------------ neighbor rows
__device__ inline void taper_horner(const double* c, double r, double& Tap, double& dTap) {
  double t = c[7] * r + c[6];
  t = t * r + c[5]; t = t * r + c[4]; t = t * r + c[3]; t = t * r + c[2]; t = t * r + c[1]; t = t * r + c[0];
  double g = 7 * c[7] * r + 6 * c[6];
  g = g * r + 5 * c[5]; g = g * r + 4 * c[4]; g = g * r + 3 * c[3]; g = g * r + 2 * c[2];
  g += c[1] / r;
  Tap = t;
  dTap = g;
}

// Verlet rows (in cell order, entries by cell-order position), one warp per atom of a system being rebuilt: every image
// within nonb_cut + skin (a superset of the owned-row cut-off of build_far_list, src/neighbor/neighbor.cpp:180-212). The
// cells within `range` of the atom's cell are visited as runs of consecutive cells along x (one contiguous range of the cell-ordered atoms per run and periodic
// image), so the candidate loads are coalesced. Entries are written through a warp ballot in visiting order
// (deterministic). Rows only need to be supersets (every consumer re-tests its entries exactly in FP64 on the current
// positions), so candidates are tested in single precision against the system's thresholds SysInfo::vthr, which add
// the largest rounding error of that r^2 to the FP64 radii. The loops carry the wrapped cell and image of each row
// incrementally and prune with precomputed reciprocals: no division per run.
__global__ void __launch_bounds__(128, 6) k_neighbors(Dev d, DevFF ff) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= d.na) return;
  const int pi = warp, i = d.cell_atoms[warp];
  const int sy = d.sys_of[i];
  if (!d.sys_flag[sy]) return;
  const SysInfo& s = d.sys[sy];
  const int nc0 = s.nc[0], nc1 = s.nc[1], nc2 = s.nc[2];
  const int key = d.cell_key[i] - s.cell_begin;
  const int cx = key % nc0, cy = (key / nc0) % nc1, cz = key / (nc0 * nc1);
  const double4 xi = d.x[i];
  int count = 0, count_near = 0, count_acc = 0;
  const unsigned lt = (1u << lane) - 1u;
  const int center = (d.S * d.S * d.S - 1) / 2;
  const size_t rowbase = static_cast<size_t>(pi) * d.vcap;
  const bool hb_i = static_cast<int>(ff.sb[d.type[i] * SB_N + SB_P_HBOND]) == 1;
  const float tv = s.vthr[0], tn = s.vthr[1], ta = s.vthr[2];
  const int smax = d.smax, S = d.S, sbase = s.shift_base;
  const double oxi = xi.x - s.origin[0], oyi = xi.y - s.origin[1], ozi = xi.z - s.origin[2];
  // fractional coordinates of i: lower bounds of the distance to a cell slab prune whole runs and clip the x range
  double fi[3];
  for (int k = 0; k < 3; ++k) fi[k] = s.R[3 * k] * oxi + s.R[3 * k + 1] * oyi + s.R[3 * k + 2] * ozi;
  const double rc = sqrt(d.rv2) * (1.0 + 1e-9) + 1e-9;
  auto slab_gap = [&](int k, int c) {   // distance from i to the slab of cell index c (unwrapped) along direction k
    const double lo = static_cast<double>(c) * s.inv_nc[k], hi = static_cast<double>(c + 1) * s.inv_nc[k];
    const double g = fmax(0.0, fmax(lo - fi[k], fi[k] - hi));
    return fmax(0.0, g * s.h[k] - 1e-9 * s.h[k]);
  };
  auto advance = [](int& w, int& sh, int n) { if (++w == n) { w = 0; ++sh; } };
  int shz = floor_div(cz - s.range[2], nc2), wz = cz - s.range[2] - shz * nc2;
  const int shy0 = floor_div(cy - s.range[1], nc1), wy0 = cy - s.range[1] - shy0 * nc1;
  for (int zz = cz - s.range[2]; zz <= cz + s.range[2]; ++zz, advance(wz, shz, nc2)) {
    const double gz = slab_gap(2, zz);
    if (gz > rc) continue;
    int shy = shy0, wy = wy0;
    for (int yy = cy - s.range[1]; yy <= cy + s.range[1]; ++yy, advance(wy, shy, nc1)) {
      const double gy = slab_gap(1, yy);
      double rx;
      if (s.ortho) {
        const double g2 = gy * gy + gz * gz;
        if (g2 > rc * rc) continue;
        // single-precision square root widened past its rounding error: the x range only needs to be a superset
        rx = static_cast<double>(sqrtf(static_cast<float>(rc * rc - g2)) * 1.000001f) + 1e-6;
      } else {
        if (gy > rc) continue;
        rx = rc;
      }
      const int rowcell = s.cell_begin + (wz * nc1 + wy) * nc0;
      const double dfx = rx * s.inv_h[0];
      int xx = max(cx - s.range[0], static_cast<int>(floor((fi[0] - dfx) * nc0)));
      const int xend = min(cx + s.range[0], static_cast<int>(floor((fi[0] + dfx) * nc0)));
      if (xx > xend) continue;
      // wrapped cell and image of the first run; each further run starts a new image at cell 0
      int shx = __float2int_rd(static_cast<float>(xx) * s.inv_ncf0), wx0 = xx - shx * nc0;
      if (wx0 < 0) { wx0 += nc0; --shx; } else if (wx0 >= nc0) { wx0 -= nc0; ++shx; }
      for (; xx <= xend; wx0 = 0, ++shx) {
        const int len = min(nc0 - wx0, xend - xx + 1);
        xx += len;
        if (shx < -smax || shx > smax || shy < -smax || shy > smax || shz < -smax || shz > smax) {
          if (lane == 0) atomicOr(d.status, ST_SHIFT_RANGE);
          continue;
        }
        const int sidx = ((shx + smax) * S + (shy + smax)) * S + (shz + smax);
        const int c0 = d.cell_start[rowcell + wx0], c1 = d.cell_start[rowcell + wx0 + len];
        if (c0 >= c1) continue;
        // the run's image: separation = xs[p] + cimg, cimg = L s - (x_i - origin) in FP64 rounded once
        const double4 sh = d.shifts[sbase + sidx];
        const float3 cimg = make_float3(static_cast<float>(sh.x - oxi), static_cast<float>(sh.y - oyi), static_cast<float>(sh.z - ozi));
        for (int base = c0; base < c1; base += 32) {
          const int p = base + lane;
          bool ok = false;
          int j = 0;
          float r2 = 0.f, tj = 0.f;
          if (p < c1) {
            j = d.cell_atoms[p];
            const float4 xj = d.xs[p];
            tj = xj.w;
            if (!(p == pi && sidx == center)) {
              const float dx = xj.x + cimg.x, dy = xj.y + cimg.y, dz = xj.z + cimg.z;
              r2 = fmaf(dz, dz, fmaf(dy, dy, dx * dx));
              ok = r2 <= tv;
            }
          }
          const unsigned image = static_cast<unsigned>(sidx) << d.abits;
          const unsigned code = static_cast<unsigned>(j) | image;   // the bonded chain's rows name atoms
          const unsigned m = __ballot_sync(0xffffffffu, ok);
          if (ok) {
            const int pos = count + __popc(m & lt);
            if (pos < d.vcap) d.vrow[rowbase + pos] = static_cast<unsigned>(p) | image;
          }
          count += __popc(m);
          // the short Verlet rows of the bond and H-bond kernels (their own exact tests run on every evaluation)
          const bool nr = ok && r2 <= tn;
          const unsigned mn = __ballot_sync(0xffffffffu, nr);
          if (nr) {
            const int posn = count_near + __popc(mn & lt);
            if (posn < d.ncap_near) d.near[static_cast<size_t>(i) * d.ncap_near + posn] = code;
          }
          count_near += __popc(mn);
          if (hb_i) {   // warp-uniform
            const bool ac = ok && r2 <= ta && static_cast<int>(ff.sb[static_cast<int>(tj) * SB_N + SB_P_HBOND]) == 2;
            const unsigned ma = __ballot_sync(0xffffffffu, ac);
            if (ac) {
              const int posa = count_acc + __popc(ma & lt);
              if (posa < d.ncap_acc) d.acc[static_cast<size_t>(i) * d.ncap_acc + posa] = code;
            }
            count_acc += __popc(ma);
          }
        }
      }
    }
  }
  if (lane == 0) {
    d.vcnt[pi] = count;
    if (count > d.vcap) {
      atomicOr(d.status, ST_VERLET_OVERFLOW);
      atomicMax(d.status + 4, count);
    }
    d.near_cnt[i] = count_near;
    if (count_near > d.ncap_near) {
      atomicOr(d.status, ST_NEAR_OVERFLOW);
      atomicMax(d.status + 3, count_near);
    }
    d.acc_cnt[i] = count_acc;
    if (count_acc > d.ncap_acc) {
      atomicOr(d.status, ST_ACC_OVERFLOW);
      atomicMax(d.status + 5, count_acc);
    }
  }
}

// The rows of this evaluation, one warp per atom: the entries of the Verlet row within nonb_cut, in Verlet-row order,
// with the exact FP64 distance test of build_far_list (every cut-off decision is the reference's). Fused: the
// charge-matrix entry H = 14.4 Tap(r) / cbrt(r^3 + (gamma_i gamma_j)^-1.5) for r <= swb (ENGINE_SPEC 7; fix_qeq_reaxff
// compute_H) stored as hi + lo single-precision parts. Also clears the per-system rebuild flags for the next evaluation.
__global__ void __launch_bounds__(256) k_pairs(Dev d, DevFF ff, QeqParams qp) {
  const int gid = blockIdx.x * blockDim.x + threadIdx.x;
  if (gid < d.nsys) d.sys_flag[gid] = 0;
  const int warp = gid >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= d.na) return;
  if (warp_lists_failed(d)) {   // the evaluation is repeated: empty rows keep the kernels after this one inside the lists
    if (lane == 0) d.nbr_cnt[warp] = 0;
    return;
  }
  const SysInfo s = d.sys[d.sys_of[warp]];
  const double rc2 = ff.nonb_cut * ff.nonb_cut;
  const double4 xi = d.xr[warp];
  const int ti = ord_type(xi), i = ord_atom(xi);
  const double* shld_i = ff.shld + static_cast<size_t>(ti) * ff.nt;
  int count = 0;
  const unsigned lt = (1u << lane) - 1u;
  const size_t vbase = static_cast<size_t>(warp) * d.vcap, rowbase = static_cast<size_t>(warp) * d.ncap;
  const int nv = min(d.vcnt[warp], d.vcap);
  for (int base = 0; base < nv; base += 32) {
    const int e = base + lane;
    bool ok = false;
    unsigned code = 0;
    int tj = 0;
    double r2 = 0.0;
    if (e < nv) {
      code = d.vrow[vbase + e];
      const double4 xj = d.xr[code & d.amask];
      tj = ord_type(xj);
      double dv[3];
      pair_dvec_x(d, s, i, ord_atom(xj), static_cast<int>(code >> d.abits), xi, xj, dv);
      r2 = dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2];
      ok = r2 <= rc2;
    }
    const unsigned m = __ballot_sync(0xffffffffu, ok);
    if (ok) {
      const int pos = count + __popc(m & lt);
      if (pos < d.ncap) {
        d.nbr[rowbase + pos] = code;
        const double r = sqrt(r2);
        double h = 0.0;
        if (r <= qp.swb) {
          double Tap, dTap;
          taper_horner(qp.tap, r, Tap, dTap);
          const double a3 = r * r * r + shld_i[tj];
          // z = a3^(-1/3): single-precision seed, then two Newton steps z <- z + (z/3)(1 - a3 z^3), which
          // square the relative error each (1e-7 -> 1e-14 -> rounding level); no division
          double z = static_cast<double>(rcbrtf(static_cast<float>(a3)));
          for (int k = 0; k < 2; ++k) z = fma(z * (1.0 / 3.0), fma(-a3 * z, z * z, 1.0), z);
          h = Tap * 14.4 * z;
        }
        const float hi = static_cast<float>(h);
        d.hhi[rowbase + pos] = hi;
        d.hlo[rowbase + pos] = static_cast<float>(h - static_cast<double>(hi));
      }
    }
    count += __popc(m);
  }
  if (lane == 0) {
    d.nbr_cnt[warp] = min(count, d.ncap);
    if (count > d.ncap) {
      atomicOr(d.status, ST_NBR_OVERFLOW);
      atomicMax(d.status + 1, count);
    }
  }
}

// ------------------------------------------------------------------------------------------------ non-bonded
// The pair terms of one non-bonded entry at separation dvd (terms::nonbonded_pair, terms.hpp:282-323): returns CE with
// gradient -CE dvd on i and +CE dvd on the partner, and the pair's van der Waals and Coulomb energies.
__device__ __forceinline__ float nb_pair_terms(const DevFF& ff, int ti, int tj, float qi, float qj, const double* dvd,
                                               float p_vdW1, float p_vdW1i, float swa, float inv_dd, float& e_vdW,
                                               float& e_ele) {
  // the exact cut-off test was taken in FP64 when the row was filtered; the pair terms run in FP32, division-free:
  // 1/r from the reciprocal square root, reciprocals of the type-pair constants from the table, exp(a) as the square
  // of exp(a/2), and the Coulomb shielding through the reciprocal cube root z = (r^3 + gamma^-3)^(-1/3), whose cube
  // is 1/(r^3 + gamma^-3)
  const float r2f = static_cast<float>(dvd[0] * dvd[0] + dvd[1] * dvd[1] + dvd[2] * dvd[2]);
  const float inv_r = rsqrtf(r2f);
  const float r = r2f * inv_r;
  const float* pp = ff.nbf + (static_cast<size_t>(ti) * ff.nt + tj) * 12;
  float Tap, dTap;
  {   // taper_stable (include/reaxmetal/terms.hpp:268-272) in t = (r - swa)/(swb - swa)
    const float t = (r - swa) * inv_dd, t2 = t * t, t3 = t2 * t, t4 = t2 * t2;
    Tap = 1.f - t4 * (35.f - 84.f * t + 70.f * t2 - 20.f * t3);
    dTap = (t3 * (-140.f + 420.f * t - 420.f * t2 + 140.f * t3)) * (inv_dd * inv_r);
  }
  const float alpha = pp[0], D = pp[1], inv_rvdw = pp[10];
  float CEvd;
  e_vdW = 0.f;
  if (ff.vdw_type == 1 || ff.vdw_type == 3) {
    const float powr_vdW1 = exp2f(p_vdW1 * __log2f(r));   // r^p and (..)^(1/p) through the fast base-2 pair
    const float sum = powr_vdW1 + pp[3];
    const float fn13 = exp2f(p_vdW1i * __log2f(sum));
    const float exp2 = __expf(0.5f * alpha * (1.f - fn13 * inv_rvdw));
    const float exp1 = exp2 * exp2;
    const float evd = D * (exp1 - 2.f * exp2);
    e_vdW += Tap * evd;
    // (sum)^(1/p - 1) r^(p - 2) = fn13 / sum * powr / r^2
    const float dfn13 = __fdividef(fn13, sum) * (powr_vdW1 * inv_r * inv_r);
    CEvd = dTap * evd - Tap * D * (alpha * inv_rvdw) * (exp1 - exp2) * dfn13;
  } else {
    const float exp2 = __expf(0.5f * alpha * (1.f - r * inv_rvdw));
    const float exp1 = exp2 * exp2;
    const float evd = D * (exp1 - 2.f * exp2);
    e_vdW += Tap * evd;
    CEvd = dTap * evd - Tap * D * (alpha * inv_rvdw) * (exp1 - exp2) * inv_r;
  }
  if (ff.vdw_type == 2 || ff.vdw_type == 3) {
    const float ecore = pp[4], acore = pp[5], inv_rcore = pp[11];
    const float e_core = ecore * __expf(acore * (1.f - r * inv_rcore));
    e_vdW += Tap * e_core;
    const float de_core = -(acore * inv_rcore) * e_core;
    CEvd += dTap * e_core + Tap * de_core * inv_r;
    if (ff.lg) {
      const float r4 = r2f * r2f, r5 = r4 * r, r6 = r4 * r2f, re6 = pp[9];
      const float inv6 = __fdividef(1.f, r6 + re6);
      const float e_lg = -pp[8] * inv6;
      e_vdW += Tap * e_lg;
      const float de_lg = -6.f * e_lg * r5 * inv6;
      CEvd += dTap * e_lg + Tap * de_lg * inv_r;
    }
  }
  const float z = rcbrtf(r2f * r + pp[7]);
  const float cq = 332.06371f * (qi * qj);   // the same bits from both ends of the pair
  e_ele = cq * (Tap * z);
  const float CEclmb = cq * (dTap - Tap * r * (z * z * z)) * z;
  return CEvd + CEclmb;
}

// One warp per atom over its full row (FP32 pair arithmetic, FP64 accumulation). The gradient of atom i collects
// -CE * dvec from every entry of its own row, so no write ever touches another atom. Energies use the reference's
// counted pairs (owner-computes rule, classify_nonbonded_entry, src/neighbor/neighbor.cpp:295-310): an entry counts
// at i if it is owned-owned with j > i, or a periodic image with tag_i < tag_j or, for an image of i itself, the
// positive direction; each counted entry contributes its full pair energy (terms::nonbonded_pair, terms.hpp:282-323).
__global__ void k_nonbonded(Dev d, DevFF ff) {
  if (warp_lists_failed(d)) return;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= d.na) return;
  const SysInfo s = d.sys[d.sys_of[warp]];
  const double4 xi4 = d.xr[warp];
  const int ti = ord_type(xi4), i = ord_atom(xi4);
  const int cnt = d.nbr_cnt[warp];
  const float p_vdW1 = static_cast<float>(ff.gp[28]), p_vdW1i = 1.f / p_vdW1;
  const float swa = static_cast<float>(ff.nonb_low), inv_dd = static_cast<float>(1.0 / (ff.nonb_cut - ff.nonb_low));
  const double qd = d.qr[warp];
  const float qi = static_cast<float>(qd);
  const long long tag_i = d.tag[i];
  const int center = (d.S * d.S * d.S - 1) / 2;
  double gx = 0, gy = 0, gz = 0, ev = 0, ee = 0, ehalf = 0;
  float v0 = 0, v1 = 0, v2 = 0, v3 = 0, v4 = 0, v5 = 0;   // pair virial, half per directed entry (lane partials)
  int counted = 0;
  for (int e = lane; e < cnt; e += 32) {
    const unsigned code = d.nbr[static_cast<size_t>(warp) * d.ncap + e];
    const int pj = static_cast<int>(code & d.amask);
    const int sidx = static_cast<int>(code >> d.abits);
    const double4 xj = d.xr[pj];
    const int j = ord_atom(xj);
    double dvd[3];
    pair_dvec_x(d, s, i, j, sidx, xi4, xj, dvd);
    float e_vdW, e_ele;
    const float CE = nb_pair_terms(ff, ti, ord_type(xj), qi, static_cast<float>(d.qr[pj]), dvd, p_vdW1, p_vdW1i, swa, inv_dd, e_vdW, e_ele);
    const float dx = static_cast<float>(dvd[0]), dy = static_cast<float>(dvd[1]), dz = static_cast<float>(dvd[2]);
    gx -= static_cast<double>(CE * dx);
    gy -= static_cast<double>(CE * dy);
    gz -= static_cast<double>(CE * dz);
    {   // the gradient -CE dv on i and +CE dv on the partner: virial -CE dv (x) dv, half of it from each direction
      const float c = -0.5f * CE;
      v0 += c * dx * dx; v1 += c * dy * dy; v2 += c * dz * dz;
      v3 += c * dx * dy; v4 += c * dx * dz; v5 += c * dy * dz;
    }
    // owner-computes counting of the energy
    bool count = false;
    if (sidx == center) count = j > i;
    else {
      const long long tag_j = d.tag[j];
      if (tag_i < tag_j) count = true;
      else if (tag_i == tag_j) {
        const double SMALL = 1e-4;
        if (dvd[2] > SMALL) count = true;
        else if (fabs(dvd[2]) < SMALL) {
          if (dvd[1] > SMALL) count = true;
          else if (fabs(dvd[1]) < SMALL && dvd[0] > SMALL) count = true;
        }
      }
    }
    if (count) {
      ev += static_cast<double>(e_vdW);
      ee += static_cast<double>(e_ele);
      ++counted;
    }
    ehalf += 0.5 * (static_cast<double>(e_vdW) + static_cast<double>(e_ele));   // per-atom tally: half of every pair
  }
  gx = warp_sum(gx); gy = warp_sum(gy); gz = warp_sum(gz); ev = warp_sum(ev); ee = warp_sum(ee);
  const double w0 = warp_sum(static_cast<double>(v0)), w1 = warp_sum(static_cast<double>(v1)), w2 = warp_sum(static_cast<double>(v2));
  const double w3 = warp_sum(static_cast<double>(v3)), w4 = warp_sum(static_cast<double>(v4)), w5 = warp_sum(static_cast<double>(v5));
  if (d.pe_on) ehalf = warp_sum(ehalf);
  for (int o = 16; o > 0; o >>= 1) counted += __shfl_xor_sync(0xffffffffu, counted, o);
  if (lane == 0) {
    d.fnb[i] = make_double4(gx, gy, gz, 0.0);
    double* vi = d.vir_nb + static_cast<size_t>(i) * kVir;
    vi[0] = w0; vi[1] = w1; vi[2] = w2; vi[3] = w3; vi[4] = w4; vi[5] = w5;
    d.eatom[static_cast<size_t>(i) * kTerms + E_VDW] = ev;
    d.eatom[static_cast<size_t>(i) * kTerms + E_ELE] = ee;
    const double chi = ff.sb[ti * SB_N + SB_CHI], eta = ff.sb[ti * SB_N + SB_ETA];
    d.eatom[static_cast<size_t>(i) * kTerms + E_POL] = 23.02 * (chi * qd + (eta / 2.) * (qd * qd));
    if (d.pe_on) pe_add(d, i, ehalf + 23.02 * (chi * qd + (eta / 2.) * (qd * qd)));
    d.census[4 * d.na + i] = counted;
  }
}

// Each non-bonded pair once: the same terms as k_nonbonded over one entry of every pair, with the partner's gradient +CE dv
// added to its fixed-point accumulator (2^32 units: integer additions give the same sum in any order, so the result is
// deterministic). The entry taken is the one whose partner stands later in cell order (for an image of the atom itself,
// the one with the larger shift index): read off the code alone, where the reference's owner rule
// (classify_nonbonded_entry) would need the atoms' numbers and tags. The sums are over the same pairs; the census of
// that rule is k_count_pairs. The entries taken are gathered into a per-warp queue in row order, so every lane of a
// batch of 32 has a pair to compute. The pair virial goes whole to the owner; the per-atom split of energies and
// virials (RX_COMPUTE_PERATOM) takes k_nonbonded instead.
__global__ void __launch_bounds__(256) k_nonbonded_half(Dev d, DevFF ff) {
  if (warp_lists_failed(d)) return;
  __shared__ unsigned queue[8][64];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31, wb = threadIdx.x >> 5;
  if (warp >= d.na) return;
  const SysInfo s = d.sys[d.sys_of[warp]];
  const double4 xi4 = d.xr[warp];
  const int ti = ord_type(xi4), i = ord_atom(xi4);
  const int cnt = d.nbr_cnt[warp];
  const float p_vdW1 = static_cast<float>(ff.gp[28]), p_vdW1i = 1.f / p_vdW1;
  const float swa = static_cast<float>(ff.nonb_low), inv_dd = static_cast<float>(1.0 / (ff.nonb_cut - ff.nonb_low));
  const double qd = d.qr[warp];
  const float qi = static_cast<float>(qd);
  const int center = (d.S * d.S * d.S - 1) / 2;
  const unsigned lt = (1u << lane) - 1u;
  double gx = 0, gy = 0, gz = 0, ev = 0, ee = 0;
  float v0 = 0, v1 = 0, v2 = 0, v3 = 0, v4 = 0, v5 = 0;   // pair virials (lane partials)
  auto pair = [&](unsigned code) {
    const int pj = static_cast<int>(code & d.amask);
    const double4 xj = d.xr[pj];
    double dvd[3];
    pair_dvec_x(d, s, i, ord_atom(xj), static_cast<int>(code >> d.abits), xi4, xj, dvd);
    float e_vdW, e_ele;
    const float CE = nb_pair_terms(ff, ti, ord_type(xj), qi, static_cast<float>(d.qr[pj]), dvd, p_vdW1, p_vdW1i, swa, inv_dd,
                                   e_vdW, e_ele);
    const float dx = static_cast<float>(dvd[0]), dy = static_cast<float>(dvd[1]), dz = static_cast<float>(dvd[2]);
    const float fx = CE * dx, fy = CE * dy, fz = CE * dz;
    gx -= static_cast<double>(fx);
    gy -= static_cast<double>(fy);
    gz -= static_cast<double>(fz);
    unsigned long long* fj = d.fix_h + 3 * static_cast<size_t>(ord_atom(xj));
    fix_add(fj, static_cast<double>(fx));
    fix_add(fj + 1, static_cast<double>(fy));
    fix_add(fj + 2, static_cast<double>(fz));
    const float c = -CE;   // the pair virial -CE dv (x) dv, whole
    v0 += c * dx * dx; v1 += c * dy * dy; v2 += c * dz * dz;
    v3 += c * dx * dy; v4 += c * dx * dz; v5 += c * dy * dz;
    ev += static_cast<double>(e_vdW);
    ee += static_cast<double>(e_ele);
  };
  int qn = 0;   // entries waiting in this warp's queue (warp-uniform)
  for (int base = 0; base < cnt; base += 32) {
    const int e = base + lane;
    bool own = false;
    unsigned code = 0;
    if (e < cnt) {
      code = d.nbr[static_cast<size_t>(warp) * d.ncap + e];
      const int pj = static_cast<int>(code & d.amask);
      const int sidx = static_cast<int>(code >> d.abits);
      own = pj > warp || (pj == warp && sidx > center);
    }
    const unsigned m = __ballot_sync(0xffffffffu, own);
    if (own) queue[wb][qn + __popc(m & lt)] = code;
    qn += __popc(m);
    __syncwarp();
    if (qn >= 32) {   // a full batch: one pair per lane; the rest moves to the front of the queue
      const unsigned mine = queue[wb][lane];
      const unsigned rest = lane + 32 < qn ? queue[wb][lane + 32] : 0u;
      __syncwarp();
      if (lane + 32 < qn) queue[wb][lane] = rest;
      __syncwarp();
      qn -= 32;
      pair(mine);
    }
  }
  if (lane < qn) pair(queue[wb][lane]);
  double sums[16] = {gx, gy, gz, ev, ee, v0, v1, v2, v3, v4, v5, 0, 0, 0, 0, 0};
  const double total = warp_sums<16>(sums);
  if ((lane & 1) == 0) {   // lane 2 k holds sum k
    const int k = lane >> 1;
    double* ea = d.eatom + static_cast<size_t>(i) * kTerms;
    if (k < 3) reinterpret_cast<double*>(d.fnb + i)[k] = total;
    else if (k == 3) ea[E_VDW] = total;
    else if (k == 4) ea[E_ELE] = total;
    else if (k < 11) d.vir_nb[static_cast<size_t>(i) * kVir + k - 5] = total;
    else if (k == 11) {
      const double chi = ff.sb[ti * SB_N + SB_CHI], eta = ff.sb[ti * SB_N + SB_ETA];
      ea[E_POL] = 23.02 * (chi * qd + (eta / 2.) * (qd * qd));
    }
  }
}

// The counted non-bonded pairs of every atom (owner-computes rule, classify_nonbonded_entry,
// src/neighbor/neighbor.cpp:295-310, as in k_nonbonded) for the decision census
__global__ void k_count_pairs(Dev d) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= d.na) return;
  const int i = d.cell_atoms[warp], cnt = d.nbr_cnt[warp];
  const long long tag_i = d.tag[i];
  const int center = (d.S * d.S * d.S - 1) / 2;
  int counted = 0;
  for (int e = lane; e < cnt; e += 32) {
    const unsigned code = d.nbr[static_cast<size_t>(warp) * d.ncap + e];
    const int sidx = static_cast<int>(code >> d.abits);
    const int pj = static_cast<int>(code & d.amask), j = d.cell_atoms[pj];
    if (sidx == center) {
      counted += j > i;
      continue;
    }
    const long long tag_j = d.tag[j];
    if (tag_i != tag_j) {
      counted += tag_i < tag_j;
      continue;
    }
    double dv[3];   // an image of i itself: the positive direction
    pair_dvec_x(d, d.sys[d.sys_of[warp]], i, j, sidx, d.xr[warp], d.xr[pj], dv);
    const double SMALL = 1e-4;
    counted += dv[2] > SMALL || (fabs(dv[2]) < SMALL && (dv[1] > SMALL || (fabs(dv[1]) < SMALL && dv[0] > SMALL)));
  }
  for (int o = 16; o > 0; o >>= 1) counted += __shfl_xor_sync(0xffffffffu, counted, o);
  if (lane == 0) d.census[4 * d.na + i] = counted;
}

// ------------------------------------------------------------------------------------------------ ACKS2 pair terms
// The pair side of the ACKS2 charge model (src/cpu/acks2.cpp:11-63), FP64, one warp per atom over its full row, with
// the kinetic potentials s_kin of fix acks2/reaxff as input: the polarization coupling 23.02 q_i s_i, and over the
// entries within xcut = (bcut_i + bcut_j)/2 the bond-softness Coulomb E = -23.02/2 bs (s_i - s_j)^2,
// bs = softness d^3 (1 - d)^6, d = r / xcut (softness = gp[34]). The gradient of i takes every entry of its row; the
// energy takes the owner-computes counted entries, as k_nonbonded. Adds to the non-bonded branch's arrays (the same
// stream, after k_nonbonded).
__global__ void k_acks2(Dev d, DevFF ff, const double* s_kin) {
  if (warp_lists_failed(d)) return;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= d.na) return;
  const SysInfo s = d.sys[d.sys_of[warp]];
  const double4 xi4 = d.xr[warp];
  const int ti = ord_type(xi4), i = ord_atom(xi4);
  const int cnt = d.nbr_cnt[warp];
  const double softness = ff.gp[34];
  const double bcut_i = ff.sb[ti * SB_N + SB_BCUT_ACKS2], s_i = s_kin[i];
  const long long tag_i = d.tag[i];
  const int center = (d.S * d.S * d.S - 1) / 2;
  double gx = 0, gy = 0, gz = 0, ee = 0, eh2 = 0, v0 = 0, v1 = 0, v2 = 0, v3 = 0, v4 = 0, v5 = 0;
  for (int e = lane; e < cnt; e += 32) {
    const unsigned code = d.nbr[static_cast<size_t>(warp) * d.ncap + e];
    const double4 xj = d.xr[code & d.amask];
    const int j = ord_atom(xj);
    const int sidx = static_cast<int>(code >> d.abits);
    const double xcut = 0.5 * (bcut_i + ff.sb[ord_type(xj) * SB_N + SB_BCUT_ACKS2]);
    double dv[3];
    pair_dvec_x(d, s, i, j, sidx, xi4, xj, dv);
    const double dist = sqrt(dv[0] * dv[0] + dv[1] * dv[1] + dv[2] * dv[2]);
    if (!(dist <= xcut)) continue;
    const double dd = dist / xcut, om = 1.0 - dd, om2 = om * om;
    const double bs = softness * (dd * dd * dd) * (om2 * om2 * om2);
    if (!(bs > 0.0)) continue;
    const double effpot = s_i - s_kin[j];
    double dbs = softness * 3.0 / xcut * (dd * dd) * (om2 * om2 * om) * (1.0 - 3.0 * dd);
    dbs = 23.02 * (-0.5 * dbs * effpot * effpot) / dist;
    gx -= dbs * dv[0]; gy -= dbs * dv[1]; gz -= dbs * dv[2];
    const double c = -0.5 * dbs;
    v0 += c * dv[0] * dv[0]; v1 += c * dv[1] * dv[1]; v2 += c * dv[2] * dv[2];
    v3 += c * dv[0] * dv[1]; v4 += c * dv[0] * dv[2]; v5 += c * dv[1] * dv[2];
    bool count = false;
    if (sidx == center) count = j > i;
    else {
      const long long tag_j = d.tag[j];
      if (tag_i < tag_j) count = true;
      else if (tag_i == tag_j) {
        const double SMALL = 1e-4;
        if (dv[2] > SMALL) count = true;
        else if (fabs(dv[2]) < SMALL) {
          if (dv[1] > SMALL) count = true;
          else if (fabs(dv[1]) < SMALL && dv[0] > SMALL) count = true;
        }
      }
    }
    if (count) ee += -0.5 * 23.02 * bs * effpot * effpot;
    eh2 += 0.5 * (-0.5 * 23.02 * bs * effpot * effpot);
  }
  gx = warp_sum(gx); gy = warp_sum(gy); gz = warp_sum(gz); ee = warp_sum(ee);
  if (d.pe_on) eh2 = warp_sum(eh2);
  v0 = warp_sum(v0); v1 = warp_sum(v1); v2 = warp_sum(v2); v3 = warp_sum(v3); v4 = warp_sum(v4); v5 = warp_sum(v5);
  if (lane == 0) {
    double4 f = d.fnb[i];
    f.x += gx; f.y += gy; f.z += gz;
    d.fnb[i] = f;
    d.eatom[static_cast<size_t>(i) * kTerms + E_ELE] += ee;
    d.eatom[static_cast<size_t>(i) * kTerms + E_POL] += 23.02 * d.q[i] * s_i;
    if (d.pe_on) pe_add(d, i, eh2 + 23.02 * d.q[i] * s_i);
    double* vi = d.vir_nb + static_cast<size_t>(i) * kVir;
    vi[0] += v0; vi[1] += v1; vi[2] += v2; vi[3] += v3; vi[4] += v4; vi[5] += v5;
  }
}

// ------------------------------------------------------------------------------------------------ QEq CG
// The charge solve works in cell order throughout (vectors, rows, columns). Lanes take consecutive entries of a row, which
// mostly name consecutive positions (the Verlet rows list runs of consecutive cells), so the 32 gathers of a load
// touch a few cache lines instead of one each.
//
// (diag(eta) + H) v of one row in FP64 (hi + lo), in every lane
__device__ inline double2 row_mv(const Dev& d, int p, double eta, const double2* v) {
  const int lane = threadIdx.x & 31;
  const int cnt = d.nbr_cnt[p];
  const double2 vi = v[p];   // issued before the row so that its latency hides behind it
  const size_t base = static_cast<size_t>(p) * d.ncap;
  double y[2] = {0.0, 0.0};
  for (int e0 = lane; e0 < cnt; e0 += 128) {
    unsigned c[4];
    float hi[4], lo[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {   // past the row's end: weight 0 on the row's own vector entry
      const int e = e0 + 32 * k;
      const bool in = e < cnt;
      c[k] = in ? d.nbr[base + e] & d.amask : static_cast<unsigned>(p);
      hi[k] = in ? d.hhi[base + e] : 0.f;
      lo[k] = in ? d.hlo[base + e] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const double h = static_cast<double>(hi[k]) + static_cast<double>(lo[k]);
      const double2 vj = v[c[k]];
      y[0] += h * vj.x;
      y[1] += h * vj.y;
    }
  }
  const double t = warp_sums<2>(y);
  return make_double2(eta * vi.x + __shfl_sync(0xffffffffu, t, 0), eta * vi.y + __shfl_sync(0xffffffffu, t, 16));
}

// Row products of a warp's consecutive rows as one stream of 128-entry pieces. A row product alone is bound by latency:
// the entries come from L2 or HBM (600-1000 cycles) and only then can the vector be gathered. Here the entries are
// copied into a per-warp ring in shared memory several pieces ahead (cp.async: no registers, no waiting), and the gathers
// of one piece run beside the copies of the next ones.
static_assert(kRingBytes == 6 * 2 * 512 && kRingBytes == 4 * 3 * 512, "6 pieces of (column, hi), 4 of (column, hi, lo)");
__device__ __forceinline__ void copy16_async(unsigned dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory"); }

// y[r] = sum over row p0 + r of H v (without the diagonal) for r < nrows, by one warp; cnt[r] entries in row p0 + r; V is
// float2 (the FP32 copy of a vector, with the matrix's hi parts) or double2 (with hi + lo); products and sums FP64
//
// start() issues the first copies: before a grid barrier, so that the matrix is on its way while the blocks meet.
template <bool kF64>
struct RowStream {
  static constexpr int kStages = kF64 ? 4 : 6, kStage = (kF64 ? 3 : 2) * 512;
  const unsigned* col;
  const float* hi;
  const float* lo;
  const int* cnt;
  const char* ring;
  int nrows, ncap;
  int fr, fe, fn;       // the next piece to fetch: row, first entry, length of the row
  unsigned fo, wr, ring_at;

  __device__ __forceinline__ void next_row() {
    fe = 0;
    do {
      ++fr;
      fo += static_cast<unsigned>(ncap);
      fn = fr < nrows ? cnt[fr] : 1;
    } while (fn == 0);
  }
  __device__ __forceinline__ void fetch() {
    const int lane = threadIdx.x & 31;
    if (fr < nrows) {
      if (fe + 4 * lane < fn) {   // rows hold a multiple of 32 entries: 16 bytes from a multiple of 4 stay inside
        const unsigned o = fo + static_cast<unsigned>(fe);
        copy16_async(wr, col + o);
        copy16_async(wr + 512, hi + o);
        if (kF64) copy16_async(wr + 1024, lo + o);
      }
      fe += 128;
      if (fe >= fn) next_row();
    }
    copy_commit();   // an empty group past the end keeps the count of groups in step with the pieces
    wr = wr + kStage == ring_at + kStages * kStage ? ring_at : wr + kStage;
  }
  // rows p0 .. p0 + rows - 1 of the matrix, cnt_[r] entries in row p0 + r
  __device__ __forceinline__ void start(const Dev& d, int p0, int rows, const int* cnt_, const char* ring_) {
    const int lane = threadIdx.x & 31;
    const size_t base = static_cast<size_t>(p0) * d.ncap + 4 * lane;
    col = d.nbr + base;
    hi = d.hhi + base;
    lo = d.hlo + base;
    cnt = cnt_;
    ring = ring_;
    nrows = rows;
    ncap = d.ncap;
    ring_at = static_cast<unsigned>(__cvta_generic_to_shared(ring_)) + 16 * lane;
    fr = 0;
    fe = 0;
    fo = 0;
    wr = ring_at;
    fn = nrows > 0 ? cnt[0] : 0;
    if (nrows > 0 && fn == 0) next_row();
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) fetch();
  }
  // y[r] = sum over row p0 + r of H v (without the diagonal); V is float2 (the FP32 copy of a vector, with the matrix's hi
  // parts) or double2 (with hi + lo); products and sums FP64
  template <class V>
  __device__ __forceinline__ void run(unsigned amask, int p0, const V* v, double2* y) {
    const int lane = threadIdx.x & 31;
    unsigned rd = 0;
    for (int r = 0; r < nrows; ++r) {
      const int n = cnt[r];
      double acc[2] = {0.0, 0.0};
      auto piece = [&](int left, auto whole) {   // `left` entries of the row from here on; whole: 128 or more
        copy_wait<kStages - 2>();
        __syncwarp();
        const char* at = ring + rd + 4 * lane;
        unsigned c[4];
        float h[4], l[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          c[k] = *reinterpret_cast<const unsigned*>(at + 128 * k) & amask;
          h[k] = *reinterpret_cast<const float*>(at + 512 + 128 * k);
          if (kF64) l[k] = *reinterpret_cast<const float*>(at + 1024 + 128 * k);
          if (!decltype(whole)::value && lane + 32 * k >= left) {   // past the end: weight 0 on the row's own vector entry
            c[k] = static_cast<unsigned>(p0 + r);
            h[k] = 0.f;
            if (kF64) l[k] = 0.f;
          }
        }
        V w[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) w[k] = v[c[k]];
        fetch();   // into the piece read before this one (every lane has passed the barrier above since)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const double m = kF64 ? static_cast<double>(h[k]) + static_cast<double>(l[k]) : static_cast<double>(h[k]);
          acc[0] += m * static_cast<double>(w[k].x);
          acc[1] += m * static_cast<double>(w[k].y);
        }
        rd = rd + kStage == kStages * kStage ? 0u : rd + kStage;
      };
      int e = 0;
      for (; e + 128 <= n; e += 128) piece(128, std::true_type{});
      if (e < n) piece(n - e, std::false_type{});
      const double s = warp_sums<2>(acc);
      if ((lane & 15) == 0) reinterpret_cast<double*>(y + r)[lane >> 4] = s;
    }
    copy_wait<0>();
    __syncwarp();
  }
};

// deterministic block sum of NV doubles per thread into out[blockIdx.x * NV + k]
template <int NV>
__device__ inline void block_partials(double* v, double* out, double* sh) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const double t = warp_sums<NV>(v);
  if ((lane & (32 / NV - 1)) == 0) sh[wid * NV + lane / (32 / NV)] = t;
  __syncthreads();
  if (wid == 0) {
    double u[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) u[k] = lane < nw ? sh[lane * NV + k] : 0.0;
    const double s = warp_sums<NV>(u);
    if ((lane & (32 / NV - 1)) == 0) out[blockIdx.x * NV + lane / (32 / NV)] = s;
  }
}

// Sum of the per-block partials, the same in every block: each lane of the first warp sums a strided subset in order, then a
// fixed exchange (the order depends only on the number of blocks). Read around L1: another block wrote them. One warp
// per block reads them (the partials are a few cache lines: read by every warp of the grid they take 5 us more).
template <int NV>
__device__ inline void grid_totals(const double* part, int nblocks, double* tot, double* sh) {
  const int lane = threadIdx.x & 31;
  if (threadIdx.x < 32) {
    double v[NV];
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = 0.0;
    for (int b = lane; b < nblocks; b += 32) {
#pragma unroll
      for (int k = 0; k < NV; k += 2) {
        const double2 t = __ldcg(reinterpret_cast<const double2*>(part + b * NV + k));
        v[k] += t.x;
        v[k + 1] += t.y;
      }
    }
    const double t = warp_sums<NV>(v);
    if ((lane & (32 / NV - 1)) == 0) sh[lane / (32 / NV)] = t;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NV; ++k) tot[k] = sh[k];
}

// Persistent cooperative Jacobi-PCG for one system, s and t solved together: the loop of fix qeq/reaxff as reproduced in
// plugin/adapter/fix_qeq_reaxff_metal.cpp:89-123, each right-hand side stopping on its own test
// sqrt(r.M^-1 r)/|b| <= tol with at most imax-1 iterations; then calculate_Q: q = s - (sum s / sum t) t.
// Precision (the resident refinement of src/metal/metal_backend.mm:435-530, in FP64 instead of double-single): the
// iterations multiply the single-precision matrix (hi: 8 bytes per entry with its index) by an FP32 copy of the
// preconditioned residual (products and sums in FP64), the vectors and every dot product are FP64, and the residual is
// recomputed with the FP64 matrix (hi + lo) whenever the iterations have converged - or have reduced the residual by
// kRefineDrop, below which the single-precision matrix stops helping. The solve ends only on that FP64 residual, so the
// tolerance and the reported residuals are those of the FP64 system.
//
// Every block owns a contiguous range of cell-ordered rows and keeps their vectors in shared memory; other blocks read
// only the copy `df` of u = M^-1 r. The iteration is the form of Chronopoulos and Gear (J. Comput. Appl. Math. 25, 153
// (1989)): w = A u, then d = u + beta d and A d = w + beta (A d) by recurrence, so that only two grid barriers are
// needed per iteration (after the row products, carrying u.w, and after the vector update, carrying the new r.u)
// instead of three. Reductions are fixed-order, so the result is bitwise reproducible. Only the grid barrier waits; the
// kernel is launched cooperatively, with 256 to 1024 threads a block (hence the bound).
//
// Profiled (24,000 atoms of water, 512 threads): 30.8 us a matrix pass alone and cold, 27.9 MB from DRAM; stalls an issue:
// fixed latencies 2.8, barriers 2.4, shared memory and conversions 1.3, gathers 0.6; the conversions of the matrix take
// 28 % of their pipe, FP64 7 %. So it waits for instruction latencies and barriers with 16 warps an SM, not for memory.
constexpr double kRefineDrop = 1e-6;

__global__ void __launch_bounds__(1024, 1) k_cg_grid(Dev d, CgArgs a) {
  cg::grid_group g = cg::this_grid();
  // a ring per warp; then, when they fit, the six vectors and the row lengths of the block's rows (else in global memory)
  extern __shared__ double2 dyn[];
  __shared__ double sh[32 * 4];
  __shared__ double tot_sh[4];
  const int n = a.n, nb = static_cast<int>(gridDim.x), blk = static_cast<int>(blockIdx.x);
  const int r0 = static_cast<int>(static_cast<long long>(n) * blk / nb), r1 = static_cast<int>(static_cast<long long>(n) * (blk + 1) / nb);
  const int m = r1 - r0;
  const int wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const int w0 = m * wid / nw, w1 = m * (wid + 1) / nw;   // this warp's rows (within the block's)
  char* ring = reinterpret_cast<char*>(dyn) + wid * kRingBytes;
  double2* vec = dyn + nw * (kRingBytes / sizeof(double2));
  double* etas = reinterpret_cast<double*>(vec + 6 * static_cast<size_t>(a.smem_rows));
  int* cnts = reinterpret_cast<int*>(etas + a.smem_rows);
  const double* E = a.smem_rows ? etas : a.eta + r0;
  const int* cnt = a.smem_rows ? cnts : d.nbr_cnt + r0;
  double2* X = a.smem_rows ? vec : a.x + r0;
  double2* R = a.smem_rows ? vec + a.smem_rows : a.r + r0;
  double2* U = a.smem_rows ? vec + 2 * a.smem_rows : a.p + r0;
  double2* W = a.smem_rows ? vec + 3 * a.smem_rows : a.q + r0;
  double2* D = a.smem_rows ? vec + 4 * a.smem_rows : a.d + r0;
  double2* S = a.smem_rows ? vec + 5 * a.smem_rows : a.s + r0;
  double loc[4], tot[4];
  int phase = 0;
  auto partbuf = [&]() { return a.part + static_cast<size_t>(phase & 1) * nb * 4; };
  double bnorm_s = 0.0, bnorm_t = 0.0, sig_s = 0.0, sig_t = 0.0;
  bool act_s = true, act_t = true, breakdown = false;
  int it_s = 1, it_t = 1, nref = 0;
  for (int k = threadIdx.x; k < m; k += blockDim.x) {
    X[k] = a.x[r0 + k];
    if (a.smem_rows) {
      etas[k] = a.eta[r0 + k];
      cnts[k] = d.nbr_cnt[r0 + k];
    }
  }
  __syncthreads();
  RowStream<true> exact;
  RowStream<false> fast;
  exact.start(d, r0 + w0, w1 - w0, cnt + w0, ring);
  for (;;) {
    // ---- FP64 residual: r = b - A x ; u = M^-1 r ; r.u (and |b|^2 on the first pass)
    exact.run(d.amask, r0 + w0, a.x, W + w0);
    __syncthreads();
    loc[0] = loc[1] = loc[2] = loc[3] = 0.0;
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
      const double eta = E[k];
      const double2 b = a.b[r0 + k], x = X[k], y = W[k];
      const double2 r = make_double2(b.x - (eta * x.x + y.x), b.y - (eta * x.y + y.y));
      const double2 u = make_double2(r.x / eta, r.y / eta);
      R[k] = r;
      U[k] = u;
      a.df[r0 + k] = make_float2(static_cast<float>(u.x), static_cast<float>(u.y));
      loc[0] += b.x * b.x; loc[1] += b.y * b.y; loc[2] += r.x * u.x; loc[3] += r.y * u.y;
    }
    block_partials<4>(loc, partbuf(), sh);
    fast.start(d, r0 + w0, w1 - w0, cnt + w0, ring);
    g.sync();
    grid_totals<4>(partbuf(), nb, tot, tot_sh);
    ++phase;
    ++nref;
    if (nref == 1) { bnorm_s = sqrt(tot[0]); bnorm_t = sqrt(tot[1]); }
    if (act_s) sig_s = tot[2];
    if (act_t) sig_t = tot[3];
    act_s = act_s && (sqrt(sig_s) / bnorm_s > a.tol);
    act_t = act_t && (sqrt(sig_t) / bnorm_t > a.tol);
    if ((!act_s || it_s >= a.imax) && (!act_t || it_t >= a.imax)) break;
    const double stop_s = fmax(a.tol * bnorm_s, kRefineDrop * sqrt(sig_s));
    const double stop_t = fmax(a.tol * bnorm_t, kRefineDrop * sqrt(sig_t));
    // ---- single-precision-matrix iterations from this residual
    double beta_s = 0.0, beta_t = 0.0, alpha_s = 0.0, alpha_t = 0.0;
    for (bool fresh = true;; fresh = false) {
      const bool in_s = act_s && it_s < a.imax && sqrt(sig_s) > stop_s;
      const bool in_t = act_t && it_t < a.imax && sqrt(sig_t) > stop_t;
      if (!in_s && !in_t) break;
      // d.Ad = u.w - beta r.u / (the previous step length); beta is 0 on the first iteration from a residual
      const double bs = in_s ? beta_s : 0.0, bt = in_t ? beta_t : 0.0;
      const double less_s = fresh || !in_s ? 0.0 : bs * sig_s / alpha_s, less_t = fresh || !in_t ? 0.0 : bt * sig_t / alpha_t;
      // w = A u ; partial u.w
      fast.run(d.amask, r0 + w0, a.df, W + w0);
      __syncthreads();
      loc[0] = loc[1] = 0.0;
      for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const double eta = E[k];
        const double2 u = U[k];
        double2 w = W[k];
        w.x += eta * u.x; w.y += eta * u.y;
        W[k] = w;
        loc[0] += u.x * w.x; loc[1] += u.y * w.y;
      }
      block_partials<2>(loc, partbuf(), sh);
      g.sync();
      grid_totals<2>(partbuf(), nb, tot, tot_sh);
      ++phase;
      alpha_s = in_s ? sig_s / (tot[0] - less_s) : 0.0;
      alpha_t = in_t ? sig_t / (tot[1] - less_t) : 0.0;
      if (!(isfinite(alpha_s) && isfinite(alpha_t))) { breakdown = true; break; }
      // d = u + beta d ; Ad = w + beta Ad ; x += alpha d ; r -= alpha Ad ; u = M^-1 r ; partial r.u
      loc[0] = loc[1] = 0.0;
      for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const double eta = E[k];
        const double2 w = W[k];
        double2 u = U[k], dd = u, ss = w, x = X[k], r = R[k];
        if (!fresh) {   // a right-hand side that has stopped keeps beta = 0: its vectors stay finite, its step is 0
          const double2 o = D[k], q = S[k];
          dd.x += bs * o.x; dd.y += bt * o.y;
          ss.x += bs * q.x; ss.y += bt * q.y;
        }
        D[k] = dd;
        S[k] = ss;
        x.x += alpha_s * dd.x; x.y += alpha_t * dd.y;
        r.x -= alpha_s * ss.x; r.y -= alpha_t * ss.y;
        u = make_double2(r.x / eta, r.y / eta);
        X[k] = x;
        R[k] = r;
        U[k] = u;
        a.df[r0 + k] = make_float2(static_cast<float>(u.x), static_cast<float>(u.y));
        loc[0] += r.x * u.x; loc[1] += r.y * u.y;
      }
      block_partials<2>(loc, partbuf(), sh);
      auto token = g.barrier_arrive();
      fast.start(d, r0 + w0, w1 - w0, cnt + w0, ring);
      g.barrier_wait(std::move(token));
      grid_totals<2>(partbuf(), nb, tot, tot_sh);
      ++phase;
      if (in_s) { beta_s = tot[0] / sig_s; sig_s = tot[0]; ++it_s; }
      if (in_t) { beta_t = tot[1] / sig_t; sig_t = tot[1]; ++it_t; }
    }
    for (int k = threadIdx.x; k < m; k += blockDim.x) a.x[r0 + k] = X[k];
    if (breakdown) break;
    copy_wait<0>();   // the pieces of the pass that is not taken, before the ring is filled anew
    __syncwarp();
    exact.start(d, r0 + w0, w1 - w0, cnt + w0, ring);
    g.sync();   // the FP64 residual reads every block's solution
  }
  copy_wait<0>();
  // calculate_Q: q = s - (sum s / sum t) t
  loc[0] = loc[1] = 0.0;
  for (int k = threadIdx.x; k < m; k += blockDim.x) {
    const double2 x = X[k];
    loc[0] += x.x; loc[1] += x.y;
  }
  block_partials<2>(loc, partbuf(), sh);
  g.sync();
  grid_totals<2>(partbuf(), nb, tot, tot_sh);
  ++phase;
  const double u = tot[0] / tot[1];
  if (a.write_q)
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
      const double2 x = X[k];
      const double q = x.x - u * x.y;
      d.qr[r0 + k] = q;
      d.q[d.cell_atoms[r0 + k]] = q;
    }
  if (blk == 0 && threadIdx.x == 0) {
    if (a.out_brk) a.out_brk[0] = breakdown ? 1 : 0;
    a.out_iters[0] = it_s;
    a.out_iters[1] = it_t;
    a.out_rel[0] = sqrt(sig_s) / bnorm_s;
    a.out_rel[1] = sqrt(sig_t) / bnorm_t;
    if (a.out_nref) a.out_nref[0] = nref;
    if (breakdown) atomicOr(d.status, ST_CG_BREAKDOWN);
    if (!(a.out_rel[0] <= a.tol && a.out_rel[1] <= a.tol)) atomicOr(d.status, ST_CG_NOTCONV);
  }
}

// Jacobi-PCG of the systems of up to kClusterAtoms atoms, one thread-block cluster per system at a time (the clusters take
// systems off a list, the largest first): the loop and the stopping rule of fix qeq/reaxff
// (fix_qeq_reaxff_metal.cpp:89-123), s and t together, FP64 throughout (matrix hi + lo, vectors, dot products). The loop
// keeps its three meetings an iteration: the two-barrier form of k_cg_grid gained 6 us of 122 at 648 atoms and nothing
// on a batch. A solve over all SMs, however small the system, costs a grid barrier (5 us) or two
// for every matrix pass of a microsecond or so, and a batch iterates until its last system has converged; a cluster's
// hardware barrier costs about 1 us and each system stops on its own.
//
// A system's bits do not depend on the size of the cluster or on what else is in the batch: a row product depends on
// the row alone, and every dot product is summed over groups of eight consecutive rows (a fixed exchange), the groups'
// sums being handed to every block of the cluster and added up in one fixed order.
//
// Profiled (648 atoms on 16 blocks, 64 CHO systems on 120 blocks): 16 warps an SM, stalls an issue: fixed latencies 2.5,
// barriers 1.8-2.0, shared memory and conversions 1.6, gathers 0.6; FP64 pipe 8 %, conversions 12 %: too few warps to
// cover the latencies. A second block does not fit an SM (96 KB of rings and 24 KB of sums each); the bound of two keeps
// the registers at 64 a thread, so that half of them are left to the bonded terms that run beside the solve.
constexpr int kGroup = 8;   // rows whose terms are summed before they are handed over
__global__ void __launch_bounds__(512, 2) k_cg_cluster(Dev d, CgArgs a) {
  cg::cluster_group cl = cg::this_cluster();
  extern __shared__ double2 dyn[];   // a ring per warp; three sets of group sums; the vectors of this block's rows
  __shared__ int current;
  const int nw = blockDim.x >> 5, wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nb = static_cast<int>(cl.num_blocks()), rank = static_cast<int>(cl.block_rank());
  char* ring = reinterpret_cast<char*>(dyn) + wid * kRingBytes;
  double2* sums = dyn + nw * (kRingBytes / sizeof(double2));
  const int cap = a.smem_rows;
  double2* X = sums + 3 * kClusterAtoms / kGroup;
  double2 *R = X + cap, *P = R + cap, *Q = P + cap, *D = Q + cap;
  double* E = reinterpret_cast<double*>(D + cap);
  int* cnt = reinterpret_cast<int*>(E + cap);
  int flip = 0;
  cl.sync();   // every block of the cluster has started: before that its shared memory must not be written
  for (;;) {
    if (rank == 0 && threadIdx.x == 0) {
      const int t = atomicAdd(a.ticket, 1);
      const int s = t < a.nsmall ? (a.order ? a.order[t] : t) : -1;
      for (int q = 0; q < nb; ++q) *cl.map_shared_rank(&current, static_cast<unsigned>(q)) = s;
    }
    cl.sync();
    const int sy = current;
    if (sy < 0) break;
    const int i0 = d.sys[sy].begin, n = d.sys[sy].natoms;
    const int groups = (n + kGroup - 1) / kGroup;
    const int g0 = groups * rank / nb, g1 = groups * (rank + 1) / nb;
    const int r0 = g0 * kGroup, m = max(0, min(g1 * kGroup, n) - r0), p0 = i0 + r0;
    const int w0 = m * wid / nw, w1 = m * (wid + 1) / nw;   // this warp's rows (within the block's)
    // hand the sums over this block's groups of `term` (a value per row) to every block
    auto hand_over = [&](double2* set, auto term) {
      for (int k0 = 0; k0 < m; k0 += blockDim.x) {
        const int k = k0 + static_cast<int>(threadIdx.x);
        double2 t = k < m ? term(k) : make_double2(0.0, 0.0);
#pragma unroll
        for (int o = 1; o < kGroup; o <<= 1) {
          t.x += __shfl_xor_sync(0xffffffffu, t.x, o);
          t.y += __shfl_xor_sync(0xffffffffu, t.y, o);
        }
        if (k < m && (k & (kGroup - 1)) == 0)
          for (int q = 0; q < nb; ++q) cl.map_shared_rank(set, static_cast<unsigned>(q))[g0 + k / kGroup] = t;
      }
    };
    auto total = [&](const double2* set) {   // in every thread
      double v[2] = {0.0, 0.0};
      for (int k = lane; k < groups; k += 32) {
        v[0] += set[k].x;
        v[1] += set[k].y;
      }
      const double t = warp_sums<2>(v);
      return make_double2(__shfl_sync(0xffffffffu, t, 0), __shfl_sync(0xffffffffu, t, 16));
    };
    auto set_of = [&](int which) { return sums + which * (kClusterAtoms / kGroup); };
    RowStream<true> rows;
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
      X[k] = a.x[p0 + k];
      E[k] = a.eta[p0 + k];
      cnt[k] = d.nbr_cnt[p0 + k];
    }
    __syncthreads();
    // ---- r = b - A x, d = M^-1 r; |b|^2 and r.d; first stop test
    rows.start(d, p0 + w0, w1 - w0, cnt + w0, ring);
    rows.run(d.amask, p0 + w0, a.x, Q + w0);
    __syncthreads();
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
      const double eta = E[k];
      const double2 b = a.b[p0 + k], x = X[k], y = Q[k];
      const double2 r = make_double2(b.x - (eta * x.x + y.x), b.y - (eta * x.y + y.y));
      const double2 dd = make_double2(r.x / eta, r.y / eta);
      R[k] = r;
      D[k] = dd;
      a.d[p0 + k] = dd;
    }
    hand_over(set_of(2), [&](int k) {
      const double2 b = a.b[p0 + k];
      return make_double2(b.x * b.x, b.y * b.y);
    });
    hand_over(set_of(flip), [&](int k) { return make_double2(R[k].x * D[k].x, R[k].y * D[k].y); });
    rows.start(d, p0 + w0, w1 - w0, cnt + w0, ring);
    cl.sync();
    const double2 bb = total(set_of(2));
    double2 sig = total(set_of(flip));
    flip ^= 1;
    const double bnorm_s = sqrt(bb.x), bnorm_t = sqrt(bb.y);
    bool act_s = true, act_t = true, breakdown = false;
    int it_s = 1, it_t = 1;
    for (int it = 1; it < a.imax; ++it) {
      act_s = act_s && (sqrt(sig.x) / bnorm_s > a.tol);
      act_t = act_t && (sqrt(sig.y) / bnorm_t > a.tol);
      if (!act_s && !act_t) break;
      // ---- q = A d; d.q
      rows.run(d.amask, p0 + w0, a.d, Q + w0);
      __syncthreads();
      hand_over(set_of(flip), [&](int k) {
        const double eta = E[k];
        const double2 dd = D[k];
        double2 q = Q[k];
        q.x += eta * dd.x; q.y += eta * dd.y;
        Q[k] = q;
        return make_double2(dd.x * q.x, dd.y * q.y);
      });
      rows.start(d, p0 + w0, w1 - w0, cnt + w0, ring);
      cl.sync();
      const double2 dq = total(set_of(flip));
      flip ^= 1;
      const double alpha_s = act_s ? sig.x / dq.x : 0.0;
      const double alpha_t = act_t ? sig.y / dq.y : 0.0;
      if (!(isfinite(alpha_s) && isfinite(alpha_t))) { breakdown = true; break; }
      // ---- x += alpha d, r -= alpha q, p = M^-1 r; r.p
      hand_over(set_of(flip), [&](int k) {
        const double eta = E[k];
        const double2 dd = D[k], q = Q[k];
        double2 x = X[k], r = R[k];
        x.x += alpha_s * dd.x; x.y += alpha_t * dd.y;
        r.x -= alpha_s * q.x; r.y -= alpha_t * q.y;
        const double2 p = make_double2(r.x / eta, r.y / eta);
        X[k] = x;
        R[k] = r;
        P[k] = p;
        return make_double2(r.x * p.x, r.y * p.y);
      });
      cl.sync();
      const double2 rp = total(set_of(flip));
      flip ^= 1;
      const double beta_s = act_s ? rp.x / sig.x : 0.0, beta_t = act_t ? rp.y / sig.y : 0.0;
      if (act_s) { sig.x = rp.x; it_s = it + 1; }
      if (act_t) { sig.y = rp.y; it_t = it + 1; }
      // ---- d = p + beta d (only for the right-hand sides still iterating)
      for (int k = threadIdx.x; k < m; k += blockDim.x) {
        const double2 p = P[k];
        double2 dd = D[k];
        if (act_s) dd.x = p.x + beta_s * dd.x;
        if (act_t) dd.y = p.y + beta_t * dd.y;
        D[k] = dd;
        a.d[p0 + k] = dd;
      }
      cl.sync();
    }
    copy_wait<0>();   // the pieces of the pass that is not taken
    __syncwarp();
    // ---- calculate_Q: q = s - (sum s / sum t) t, the solution, the counts and residuals
    __syncthreads();
    hand_over(set_of(flip), [&](int k) { return X[k]; });
    cl.sync();
    const double2 sx = total(set_of(flip));
    flip ^= 1;
    const double c = sx.x / sx.y;
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
      const double2 x = X[k];
      a.x[p0 + k] = x;
      if (a.write_q) {
        const double q = x.x - c * x.y;
        d.qr[p0 + k] = q;
        d.q[d.cell_atoms[p0 + k]] = q;
      }
    }
    if (rank == 0 && threadIdx.x == 0) {
      const double rel_s = sqrt(sig.x) / bnorm_s, rel_t = sqrt(sig.y) / bnorm_t;
      if (a.out_brk) a.out_brk[sy] = breakdown ? 1 : 0;
      a.out_iters[2 * sy] = it_s;
      a.out_iters[2 * sy + 1] = it_t;
      a.out_rel[2 * sy] = rel_s;
      a.out_rel[2 * sy + 1] = rel_t;
      if (breakdown) atomicOr(d.status, ST_CG_BREAKDOWN);
      if (!(rel_s <= a.tol && rel_t <= a.tol)) atomicOr(d.status, ST_CG_NOTCONV);
    }
  }
}

// Segmented Jacobi-PCG: every system that k_cg_cluster does not take (those of more than a.cluster_max atoms), all of them
// at once on one cooperative grid, with the same algorithm and the same stopping rule per system, s and t separately, as the
// stock loop of fix qeq/reaxff (fix_qeq_reaxff_metal.cpp:89-123). Their rows are spread over all warps of the GPU.
// Every dot product is a per-row term written to rb0/rb1; the warp that brings the last row of a system to a pass
// sums that system's terms, so a system's result depends only on its own rows: it is bitwise the same alone and inside
// any batch. Row products and sums take the order of k_cg_cluster (groups of eight rows, then a lane-strided sum of the
// groups), so it is also bitwise the same whichever of the two kernels solves it. The iteration loop ends when no
// system is live; the live count is kept per iteration parity so that no block can see it change before every block
// has read it.
__device__ inline double2 sys_sum2(const double2* v, int i0, int n) {
  const int lane = threadIdx.x & 31, groups = (n + kGroup - 1) / kGroup;
  double s[2] = {0.0, 0.0};
  for (int g = lane; g < groups; g += 32) {
    double2 t[kGroup];
#pragma unroll
    for (int k = 0; k < kGroup; ++k) {
      const int row = g * kGroup + k;
      t[k] = row < n ? __ldcg(v + i0 + row) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int o = 1; o < kGroup; o <<= 1)   // the exchange of k_cg_cluster's hand-over, as its first lane sees it
#pragma unroll
      for (int k = 0; k < kGroup; k += 2 * o) {
        t[k].x += t[k + o].x;
        t[k].y += t[k + o].y;
      }
    s[0] += t[0].x;
    s[1] += t[0].y;
  }
  const double t = warp_sums<2>(s);
  return make_double2(__shfl_sync(0xffffffffu, t, 0), __shfl_sync(0xffffffffu, t, 16));
}

// lane 0 counts cnt rows of the system in (after every lane's writes are fenced); true in every lane of the warp that
// brought the system's last rows
__device__ inline bool arrive_last(SysCg* sc, int n, int cnt) {
  __threadfence();
  __syncwarp();
  bool last = false;
  if ((threadIdx.x & 31) == 0) last = atomicAdd(&sc->counter, static_cast<unsigned>(cnt)) == static_cast<unsigned>(n - cnt);
  last = __shfl_sync(0xffffffffu, last, 0);
  if (last) __threadfence();
  return last;
}

__global__ void __launch_bounds__(256, 4) k_cg_seg(Dev d, CgArgs a) {
  cg::grid_group g = cg::this_grid();
  const int lane = threadIdx.x & 31;
  const int gw = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int nw = gridDim.x * (blockDim.x >> 5);
  const int na = d.na;
  const double tol = a.tol;
  // matrix passes: warp per row, rows dealt round-robin over all warps (a system that is still iterating when most
  // have stopped keeps many warps busy); a warp counts its rows of one system in when it meets a different system
  // ---- r = b - A x, d = M^-1 r; |b|^2 and r.d per system; first stop test
  {
    int cur = -1, cnt = 0;
    auto finish = [&](int s, int c) {
      const SysInfo& si = d.sys[s];
      if (!arrive_last(a.sc + s, si.natoms, c)) return;
      const double2 bb = sys_sum2(a.rb0, si.begin, si.natoms);
      const double2 rd = sys_sum2(a.rb1, si.begin, si.natoms);
      if (lane == 0) {
        SysCg& c2 = a.sc[s];
        c2.counter = 0;
        c2.bnorm_s = sqrt(bb.x);
        c2.bnorm_t = sqrt(bb.y);
        c2.sig_s = rd.x;
        c2.sig_t = rd.y;
        c2.it_s = c2.it_t = 1;
        c2.breakdown = 0;
        c2.act_s = sqrt(c2.sig_s) / c2.bnorm_s > tol;
        c2.act_t = sqrt(c2.sig_t) / c2.bnorm_t > tol;
        c2.live = (c2.act_s || c2.act_t) && a.imax > 1;
        if (c2.live) atomicAdd(a.nlive + 1, 1);
      }
    };
    for (int i = gw; i < na; i += nw) {
      const int s = d.sys_of[i];
      if (s != cur) {
        if (cnt > 0) finish(cur, cnt);
        cur = s;
        cnt = 0;
      }
      if (d.sys[s].natoms <= a.cluster_max) continue;   // k_cg_cluster's (never live here)
      const double eta = a.eta[i];
      const double2 y = row_mv(d, i, eta, a.x);
      if (lane == 0) {
        const double2 b = a.b[i];
        const double2 rr = make_double2(b.x - y.x, b.y - y.y);
        a.r[i] = rr;
        const double2 dd = make_double2(rr.x / eta, rr.y / eta);
        a.d[i] = dd;
        a.rb0[i] = make_double2(b.x * b.x, b.y * b.y);
        a.rb1[i] = make_double2(rr.x * dd.x, rr.y * dd.y);
      }
      ++cnt;
    }
    if (cnt > 0) finish(cur, cnt);
  }
  g.sync();
  for (int it = 1; it < a.imax; ++it) {
    if (__ldcg(a.nlive + (it & 1)) == 0) break;
    if (blockIdx.x == 0 && threadIdx.x == 0) a.nlive[(it + 1) & 1] = 0;
    // ---- q = A d, d.q; alpha (or a breakdown, which ends this system)
    {
      int cur = -1, cnt = 0;
      bool live = false;
      auto finish = [&](int s, int c) {
        const SysInfo& si = d.sys[s];
        if (!arrive_last(a.sc + s, si.natoms, c)) return;
        const double2 dq = sys_sum2(a.rb0, si.begin, si.natoms);
        if (lane == 0) {
          SysCg& c2 = a.sc[s];
          c2.counter = 0;
          c2.alpha_s = c2.act_s ? c2.sig_s / dq.x : 0.0;
          c2.alpha_t = c2.act_t ? c2.sig_t / dq.y : 0.0;
          if (!(isfinite(c2.alpha_s) && isfinite(c2.alpha_t))) {
            c2.breakdown = 1;
            c2.live = 0;
          }
        }
      };
      for (int i = gw; i < na; i += nw) {
        const int s = d.sys_of[i];
        if (s != cur) {
          if (cnt > 0) finish(cur, cnt);
          cur = s;
          cnt = 0;
          live = __ldcg(&a.sc[s].live) != 0;
        }
        if (!live) continue;
        const double2 y = row_mv(d, i, a.eta[i], a.d);
        if (lane == 0) {
          a.q[i] = y;
          const double2 dd = a.d[i];
          a.rb0[i] = make_double2(dd.x * y.x, dd.y * y.y);
        }
        ++cnt;
      }
      if (cnt > 0) finish(cur, cnt);
    }
    g.sync();
    // ---- x += alpha d, r -= alpha q, p = M^-1 r, r.p; beta, the counts and the next stop test
    for (int i0 = gw * 32; i0 < na; i0 += nw * 32) {
      const int i = i0 + lane;
      int s = -1;
      bool on = false;
      if (i < na) {
        s = d.sys_of[i];
        on = __ldcg(&a.sc[s].live) != 0;
      }
      if (on) {
        const double alpha_s = __ldcg(&a.sc[s].alpha_s), alpha_t = __ldcg(&a.sc[s].alpha_t);
        const double2 dd = a.d[i], qq = a.q[i];
        double2 xx = a.x[i], rr = a.r[i];
        xx.x += alpha_s * dd.x; xx.y += alpha_t * dd.y;
        rr.x -= alpha_s * qq.x; rr.y -= alpha_t * qq.y;
        a.x[i] = xx;
        a.r[i] = rr;
        const double eta = a.eta[i];
        const double2 pp = make_double2(rr.x / eta, rr.y / eta);
        a.p[i] = pp;
        a.rb0[i] = make_double2(rr.x * pp.x, rr.y * pp.y);
      }
      __threadfence();
      __syncwarp();
      // one arrival per system present in this warp's 32 rows, by the lowest lane of that system
      const unsigned on_mask = __ballot_sync(0xffffffffu, on);
      const unsigned same = __match_any_sync(0xffffffffu, s) & on_mask;
      bool last = false;
      if (on && (__ffs(same) - 1) == lane) {
        const unsigned c = __popc(same);
        last = atomicAdd(&a.sc[s].counter, c) == static_cast<unsigned>(d.sys[s].natoms) - c;
      }
      unsigned m = __ballot_sync(0xffffffffu, last);
      if (m) __threadfence();
      while (m) {
        const int l = __ffs(m) - 1;
        m &= m - 1;
        const int ss = __shfl_sync(0xffffffffu, s, l);
        const SysInfo& si = d.sys[ss];
        const double2 rp = sys_sum2(a.rb0, si.begin, si.natoms);
        if (lane == 0) {
          SysCg& c = a.sc[ss];
          c.counter = 0;
          c.beta_s = c.act_s ? rp.x / c.sig_s : 0.0;
          c.beta_t = c.act_t ? rp.y / c.sig_t : 0.0;
          if (c.act_s) { c.sig_s = rp.x; c.it_s = it + 1; }
          if (c.act_t) { c.sig_t = rp.y; c.it_t = it + 1; }
          // the stop test of the next iteration; d below is updated only for the right-hand sides still active
          c.act_s = c.act_s && (sqrt(c.sig_s) / c.bnorm_s > tol);
          c.act_t = c.act_t && (sqrt(c.sig_t) / c.bnorm_t > tol);
          c.live = (c.act_s || c.act_t) && it + 1 < a.imax;
          if (c.live) atomicAdd(a.nlive + ((it + 1) & 1), 1);
        }
      }
    }
    g.sync();
    // ---- d = p + beta d
    for (int i = gw * 32 + lane; i < na; i += nw * 32) {
      const int s = d.sys_of[i];
      if (!__ldcg(&a.sc[s].live)) continue;
      const double beta_s = __ldcg(&a.sc[s].beta_s), beta_t = __ldcg(&a.sc[s].beta_t);
      const int act_s = __ldcg(&a.sc[s].act_s), act_t = __ldcg(&a.sc[s].act_t);
      const double2 pp = a.p[i];
      double2 dd = a.d[i];
      if (act_s) dd.x = pp.x + beta_s * dd.x;
      if (act_t) dd.y = pp.y + beta_t * dd.y;
      a.d[i] = dd;
    }
    g.sync();
  }
// ---- calculate_Q per system (warp per system): q = s - (sum s / sum t) t, the counts and residuals
  for (int s = gw; s < d.nsys; s += nw) {
    const SysInfo& si = d.sys[s];
    if (si.natoms <= a.cluster_max) continue;
    const double2 sum = sys_sum2(a.x, si.begin, si.natoms);
    const double u = sum.x / sum.y;
    if (a.write_q)
      for (int k = lane; k < si.natoms; k += 32) {
        const double2 xx = a.x[si.begin + k];
        const double qq = xx.x - u * xx.y;
        d.qr[si.begin + k] = qq;
        d.q[d.cell_atoms[si.begin + k]] = qq;
      }
    if (lane == 0) {
      const SysCg& c = a.sc[s];
      if (a.out_brk) a.out_brk[s] = c.breakdown;
      a.out_iters[2 * s] = c.it_s;
      a.out_iters[2 * s + 1] = c.it_t;
      a.out_rel[2 * s] = sqrt(c.sig_s) / c.bnorm_s;
      a.out_rel[2 * s + 1] = sqrt(c.sig_t) / c.bnorm_t;
      if (c.breakdown) atomicOr(d.status, ST_CG_BREAKDOWN);
      if (!(a.out_rel[2 * s] <= tol && a.out_rel[2 * s + 1] <= tol)) atomicOr(d.status, ST_CG_NOTCONV);
    }
  }
}


// Initial guesses from the histories (Q-23: s = 4(s0+s2) - (6 s1 + s3), t = t2 + 3(t0 - t1); index 0 = latest),
// right-hand sides b_s = -chi, b_t = -1, and the diagonal eta.
__global__ void k_qeq_prepare(Dev d, DevFF ff, CgArgs a, const double* s_hist, const double* t_hist) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;   // cell-order position
  if (i >= d.na) return;
  const int atom = d.cell_atoms[i], t = d.type[atom];
  const double* sh = s_hist + 4 * static_cast<size_t>(atom);
  const double* th = t_hist + 4 * static_cast<size_t>(atom);
  a.x[i] = make_double2(4 * (sh[0] + sh[2]) - (6 * sh[1] + sh[3]), th[2] + 3 * (th[0] - th[1]));
  a.b[i] = make_double2(-ff.sb[t * SB_N + SB_CHI], -1.0);
  a.eta[i] = ff.sb[t * SB_N + SB_ETA];
}

// A solve of given right-hand sides from given guesses (mtl::Context::qeq_solve, metal_backend.hpp:84-86): b and x0
// hold the s system for every atom, then the t system.
__global__ void k_qeq_prepare_given(Dev d, DevFF ff, CgArgs a, const double* b, const double* x0) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.na) return;
  const int atom = d.cell_atoms[i];
  a.x[i] = x0 ? make_double2(x0[atom], x0[d.na + atom]) : make_double2(0.0, 0.0);
  a.b[i] = make_double2(b[atom], b[d.na + atom]);
  a.eta[i] = ff.sb[d.type[atom] * SB_N + SB_ETA];
}

// the solve just finished becomes the newest history entry; not after a list overflow (the evaluation is repeated),
// nor after a failed solve (a breakdown, or a system above its tolerance in strict mode): the call then reports an
// error and leaves the histories as they were
__global__ void k_qeq_history(Dev d, const double2* x, double* s_hist, double* t_hist, int strict) {
  if (lists_failed(d)) return;
  const int st = *reinterpret_cast<volatile const int*>(d.status);
  if ((st & ST_CG_BREAKDOWN) || (strict && (st & ST_CG_NOTCONV))) return;
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= d.na) return;
  double* sh = s_hist + 4 * static_cast<size_t>(i);
  double* th = t_hist + 4 * static_cast<size_t>(i);
  for (int k = 3; k > 0; --k) { sh[k] = sh[k - 1]; th[k] = th[k - 1]; }
  const double2 xi = x[d.rank[i]];
  sh[0] = xi.x;
  th[0] = xi.y;
}

// y = (diag(eta) + H) v, owned rows (mtl::Context::qeq_matvec): v in cell order, y by atom
__global__ void k_qeq_matvec(Dev d, DevFF ff, const double2* v, double2* y) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (warp >= d.na) return;
  const double eta = ff.sb[ord_type(d.xr[warp]) * SB_N + SB_ETA];
  const double2 r = row_mv(d, warp, eta, v);
  if ((threadIdx.x & 31) == 0) y[ord_atom(d.xr[warp])] = r;
}

// per-atom values into cell order and back
__global__ void k_to_cell_order(Dev d, const double2* by_atom, double2* by_position) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < d.na) by_position[p] = by_atom[d.cell_atoms[p]];
}
__global__ void k_to_atom_order(Dev d, const double2* by_position, double2* by_atom) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < d.na) by_atom[d.cell_atoms[p]] = by_position[p];
}

// ------------------------------------------------------------------------------------------------ energy sums
// Per system: fixed-order sums of the 13 energy terms and the 6 virial components over the system's atoms, in two
// passes. k_energy_part: one block per (system, 256-atom chunk), a thread per atom, each of the 19 quantities summed by
// a fixed shuffle tree per warp and then over the warps in order; k_energy_final: per system, a warp per quantity over
// the chunk partials (lane-strided, then a fixed shuffle tree). Chunks start at the system's first atom, so a system's sums are the same alone or in a
// batch.
constexpr int kESum = kTerms + kVir;
__global__ void __launch_bounds__(256) k_energy_part(Dev d, double* part, int nchunk) {
  const int sidx = blockIdx.x, c = blockIdx.y;   // systems along x: any number of them
  const SysInfo& s = d.sys[sidx];
  if (c * 256 >= s.natoms) return;
  __shared__ double sh[8][kESum];
  const int r = c * 256 + threadIdx.x;
  double v[kESum];
  if (r < s.natoms) {
    const size_t a = static_cast<size_t>(s.begin + r);
#pragma unroll
    for (int t = 0; t < kTerms; ++t) v[t] = d.eatom[a * kTerms + t];
#pragma unroll
    for (int k = 0; k < kVir; ++k) {
      const size_t q = a * kVir + k;
      v[kTerms + k] = ((d.vir[q] + d.vir_h[q]) + d.vir_t[q]) + d.vir_nb[q];
    }
  } else {
#pragma unroll
    for (int t = 0; t < kESum; ++t) v[t] = 0.0;
  }
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
  for (int t = 0; t < kESum; ++t) {
    double x = v[t];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[w][t] = x;
  }
  __syncthreads();
  if (threadIdx.x < kESum) {
    double x = 0.0;
    for (int k = 0; k < 8; ++k) x += sh[k][threadIdx.x];
    part[(static_cast<size_t>(sidx) * nchunk + c) * kESum + threadIdx.x] = x;
  }
}

__global__ void k_energy_final(Dev d, const double* part, int nchunk, double* out, double* out_vir) {
  const int sidx = blockIdx.x, t = threadIdx.x >> 5, lane = threadIdx.x & 31;   // a warp per quantity
  if (t >= kESum) return;
  const int nc = (d.sys[sidx].natoms + 255) / 256;
  double x = 0.0;
  for (int c = lane; c < nc; c += 32) x += part[(static_cast<size_t>(sidx) * nchunk + c) * kESum + t];
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  if (lane == 0) {
    if (t < kTerms) out[sidx * kTerms + t] = x;
    else out_vir[sidx * kVir + (t - kTerms)] = x;
  }
}

}  // namespace rx
