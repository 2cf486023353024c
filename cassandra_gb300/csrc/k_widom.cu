// k_widom.cu -- batched CBMC Widom insertion on the GPU.
//
//   k_cell_count / k_cell_scan / k_cell_scatter / k_cell_place
//       per-box cell lists (counting sort, deterministic order inside a cell);
//       the GPU counterpart of Sector_Setup / CBMC_Cell_List_Setup
//       (sector_routines.f90:39-374).  Cells only accelerate the search:
//       every pair with r <= cutoff is visited exactly once, whatever the cell
//       count, so the energies are those of the molecule loop of
//       Compute_Molecule_Nonbond_Inter_Energy_Widom (energy_routines.f90:1266-1297).
//   k_vox_lists
//       neighbour lists on a grid of voxels, from the cell lists.
//   k_widom_f32 / k_widom_w (mixed / FP64)
//       a lane per Widom insertion: Build_Molecule with kappa_ins first-fragment
//       trials and Fragment_Placement with kappa_dih dihedral trials
//       (fragment_growth.f90:72-707, 1449-2132), then the full-cutoff energy,
//       intramolecular and bonded energies of the grown molecule
//       (widom_insert.f90:320-447); the neighbour queries of a warp's insertions
//       are worked through by the whole warp.  The CTA's box (cell-sorted atoms)
//       is staged in shared memory when it fits.
//   k_widom_fix
//       the FP64 cutoff decisions of the mixed path.
//   k_widom
//       FP64, one thread per insertion through the cell lists: CBMC options, the
//       molecule-pair cutoff, styles without a cutoff.
//   k_widom_recip
//       Update_System_Ewald_Reciprocal_Energy_Widom (energy_routines.f90:2500-2550)
//       for the insertions that survived, when the box carries an Ewald sum.
//   k_widom_finalize
//       widom_var = exp(-beta (dE - dE_frag) - ln_pbias) and the per-box sums
//       (widom_insert.f90:445-447, 538), in a fixed order.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <new>
#include <vector>

#include "cass_ctx.h"
#include "cass_cbmc.cuh"
#include "cass_cbmc_f.cuh"

namespace cassgpu {


struct BoxSrc {
  const double4_32a* p64;
  const float4* p32;
  const int4* meta;
};

// Per-insertion record: dE_intra, dE_inter (without reciprocal), dE_frag, ln_pbias.
using WRec = double4_32a;

// Widom cell edge rcut_cbmc / cells-per-cutoff, measured on the 64-box butane batch:
// with row-trimmed stencils, cells of a third of the cutoff visit 2.4x fewer
// candidates and the FP64 kernel runs 22 % faster than with cells of the cutoff.  The
// FP32 kernel searches cells only in boxes without voxel lists and while the lists are
// built: 15.2 ms at 1.25, 17.6 ms at 1.
constexpr double kCellsPerCutoffFP64 = 3.0;
constexpr double kCellsPerCutoffMixed = 1.25;
constexpr size_t kSmemMax = 227 * 1024;  // dynamic shared memory of a CTA
// voxels per cutoff of the neighbour lists: 2.6, 3.25 and 4 for the CBMC radius took
// 15.4, 15.2 and 15.8 ms, 3, 4 and 5 for the full one 15.2, 15.2 and 15.5 ms
constexpr double kVoxPerCutoffCbmc = 3.25;
constexpr double kVoxPerCutoffFull = 4.0;
// Most voxels per atom of a box: a voxel costs its search even where it is empty.  500
// atoms in a box of 400 A had 8e6 voxels of the CBMC radius: one FP64 insertion 1.62 ms,
// 0.37 ms now (1.30 ms without lists); 1e5 mixed ones, which went without lists, 2.70 ms,
// 1.09 ms now.  Liquids have 1 to 11.
constexpr double kVoxPerAtom = 16.0;
constexpr double kVoxMaxBytes = 4.0e9;      // most device memory for them, records and entries

__device__ __forceinline__ int wrapc(int c, int n) {
  c %= n;
  return c < 0 ? c + n : c;
}

// Periodic image of unwrapped cell c: the shift s (in box lengths) with
// c + s * n in [0, n); the division only runs outside one image either side
__device__ __forceinline__ int cell_image(int c, int n) {
  if (c >= 0 && c < n) return 0;
  if (c < 0 && c >= -n) return 1;
  if (c >= n && c < 2 * n) return -1;
  return (wrapc(c, n) - c) / n;
}

// ---------------------------------------------------------------------------
// K7: cell lists of the batch boxes
__device__ __forceinline__ int cell_index(const BoxDev& b, double x, double y, double z) {
  int c[3];
  double p[3] = {x, y, z};
  for (int d = 0; d < 3; ++d) {
    double w = p[d] - b.L[d] * floor((p[d] + b.hL[d]) / b.L[d]);  // wrapped into [-L/2, L/2)
    int k = (int)floor((w + b.hL[d]) * b.cell_inv[d]);
    c[d] = min(max(k, 0), b.nc[d] - 1);
  }
  return (c[2] * b.nc[1] + c[1]) * b.nc[0] + c[0];
}

__global__ void k_cell_count(const BoxSrc* src, const BoxDev* boxes, int* cell_of, int* count) {
  int k = blockIdx.y;
  const BoxDev& b = boxes[k];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.natoms) return;
  double4_32a p = src[k].p64[i];
  int c = cell_index(b, p.x, p.y, p.z);
  cell_of[b.atom_off + i] = c;
  atomicAdd(&count[b.cell_off + c], 1);
}

// exclusive scan of the box's cell counts; cstart holds local atom indices
__global__ void k_cell_scan(const BoxDev* boxes, const int* count, int* cstart, int* fill) {
  int k = blockIdx.x;
  const BoxDev& b = boxes[k];
  int nc = b.nc[0] * b.nc[1] * b.nc[2];
  __shared__ int carry;
  __shared__ int warp_tot[32];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  int* cs = cstart + b.cell_off + k;
  for (int base = 0; base < nc; base += blockDim.x) {
    int c = base + threadIdx.x;
    int v = c < nc ? count[b.cell_off + c] : 0;
    int x = v;
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, x, o);
      if ((threadIdx.x & 31) >= o) x += y;
    }
    if ((threadIdx.x & 31) == 31) warp_tot[threadIdx.x >> 5] = x;
    __syncthreads();
    if (threadIdx.x < 32) {
      int nw = blockDim.x >> 5;
      int t = threadIdx.x < nw ? warp_tot[threadIdx.x] : 0;
      for (int o = 1; o < 32; o <<= 1) {
        int y = __shfl_up_sync(0xffffffffu, t, o);
        if (threadIdx.x >= o) t += y;
      }
      if (threadIdx.x < nw) warp_tot[threadIdx.x] = t;
    }
    __syncthreads();
    int w = threadIdx.x >> 5;
    int excl = x - v + (w > 0 ? warp_tot[w - 1] : 0) + carry;
    if (c < nc) {
      cs[c] = excl;
      fill[b.cell_off + c] = 0;
    }
    __syncthreads();
    if (threadIdx.x == blockDim.x - 1) carry = excl + v;
    __syncthreads();
  }
  if (threadIdx.x == 0) cs[nc] = carry;
}

// the packed indices of each cell's atoms, in any order
__global__ void k_cell_scatter(const BoxDev* boxes, const int* cell_of, const int* cstart, int* fill, int* list) {
  int k = blockIdx.y;
  const BoxDev& b = boxes[k];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.natoms) return;
  int c = cell_of[b.atom_off + i];
  list[b.atom_off + cstart[b.cell_off + k + c] + atomicAdd(&fill[b.cell_off + c], 1)] = i;
}

// The cell-sorted copies: an atom stands in its cell behind those of smaller packed
// index, a deterministic order.  A thread per atom counts them; a thread per cell that
// sorted its cell took 281 us for the 27 cells of 256 waters.
__global__ void k_cell_place(const BoxSrc* src, const BoxDev* boxes, const int* cell_of, const int* cstart,
                             const int* list, double4_32a* c64, float4* c32, int* ctype, float* cq32, int* corig) {
  int k = blockIdx.y;
  const BoxDev& b = boxes[k];
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= b.natoms) return;
  const int c = cell_of[b.atom_off + i];
  const int first = cstart[b.cell_off + k + c], end = cstart[b.cell_off + k + c + 1];
  int rank = 0;
  for (int q = first; q < end; ++q) rank += list[b.atom_off + q] < i ? 1 : 0;
  const int g = b.atom_off + first + rank;
  // the copies hold the positions their cells were chosen from, wrapped into
  // [-L/2, L/2) (an atom of a molecule folded by its COM may stick out of the
  // box), so that a query's per-row image shift is the whole periodic shift
  double4_32a p = src[k].p64[i];
  p.x = p.x - b.L[0] * floor((p.x + b.hL[0]) / b.L[0]);
  p.y = p.y - b.L[1] * floor((p.y + b.hL[1]) / b.L[1]);
  p.z = p.z - b.L[2] * floor((p.z + b.hL[2]) / b.L[2]);
  c64[g] = p;
  const float4 q = src[k].p32[i];
  c32[g] = make_float4((float)p.x, (float)p.y, (float)p.z, q.w);
  ctype[g] = src[k].meta[i].y;
  cq32[g] = (float)p.w;
  corig[g] = i;
}

// ---------------------------------------------------------------------------
// box queries

struct BoxView {
  const BoxDev* b;          // shared-memory copy
  const double4_32a* p64;   // cell-sorted FP64 atoms (x, y, z, q) of this box (smem or global)
  const int* ptype;         // their types (smem or global)
  const int* cstart;        // cell starts, local atom indices (smem or global)
  const int* corig;         // packed index of each cell-sorted atom (global; molecule-pair boxes)
  double rc_cbmc, rc_full;
};

// The test molecule of one energy call as Check_MoleculePair_Cutoff sees it
// (energy_routines.f90:3027-3088): the COM and max_dcom of its existing atoms
struct QueryMol {
  double com[3];
  double dcom;
};

// Energy of one test atom at p against every box atom within the cutoff.
// Returns true on core overlap (r^2 < rcut_low^2), as Compute_MoleculePair_Energy
// (energy_routines.f90:1676-1679) does.
struct PairCount {
  unsigned long long visited = 0, in_cut = 0;
  double eabs = 0.0;  // sum of |pair energy| of the current query
};

// With qm (a box with a molecule-pair cutoff) a candidate atom counts only when
// its molecule passes Check_MoleculePair_Cutoff against the test molecule:
// |COM - COM_j| <= (rcut_cbmc or rcut_max) + max_dcom + max_dcom_j, as the
// molecule loop of Compute_Molecule_Nonbond_Inter_Energy_Widom applies it
// (energy_routines.f90:1266-1297) -- the overlap test included.
__device__ bool query_box(const BoxView& V, const PairTable& T, const double p[3], int qt, double qch, bool cbmc,
                          bool want_qq, double& eout, PairCount& pc, const QueryMol* qm = nullptr) {
  const BoxDev& b = *V.b;
  double rc = cbmc ? V.rc_cbmc : V.rc_full;
  // minimum-image charges count every pair of a molecule within the
  // molecule-pair cutoff, in CBMC calls too: the whole box is searched
  if (qm && cbmc && want_qq && b.charge_style == CASS_CHARGE_COUL && b.charge_sum_style == CASS_QQ_MINIMUM)
    rc = 1e30;
  const double rint0 = cbmc ? V.rc_cbmc : b.rcut_max;
  int lo[3], hi[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    double u = (p[d] + b.hL[d]) * b.cell_inv[d];
    double w = fmin(rc * b.cell_inv[d], 1.0e6);
    int l = (int)floor(u - w - 1e-6), h = (int)floor(u + w + 1e-6);
    if (h - l + 1 >= b.nc[d]) {
      l = 0;
      h = b.nc[d] - 1;
    }
    lo[d] = l;
    hi[d] = h;
  }
  const bool qq_on = want_qq && b.charge_style == CASS_CHARGE_COUL;
  const double4_32a* P = V.p64;
  double acc = 0.0, eabs = 0.0;
  // rows of the stencil trimmed to the cutoff sphere: the distance from p to a
  // row's y and z slabs (less a margin of 1e-6 cell) leaves a chord in x
  const double rc2 = rc * rc;
  const bool fully = hi[1] - lo[1] + 1 >= b.nc[1], fullz = hi[2] - lo[2] + 1 >= b.nc[2];
  double ch[3];
  for (int d = 0; d < 3; ++d) ch[d] = b.L[d] / (double)b.nc[d];
  auto slab_d2 = [&](int c, int d) {
    const double c0 = (double)c * ch[d] - b.hL[d];
    const double e = fmax(fmax(c0 - p[d], p[d] - (c0 + ch[d])) - 1.0e-6 * ch[d], 0.0);
    return e * e;
  };
  for (int cz = lo[2]; cz <= hi[2]; ++cz) {
    int wz = wrapc(cz, b.nc[2]);
    const double dz2 = fullz ? 0.0 : slab_d2(cz, 2);
    if (dz2 > rc2) continue;
    for (int cy = lo[1]; cy <= hi[1]; ++cy) {
      const double d2 = fully ? dz2 : dz2 + slab_d2(cy, 1);
      if (d2 > rc2) continue;
      int xlo, xhi;
      {
        const double u = (p[0] + b.hL[0]) * b.cell_inv[0];
        const double w = fmin(sqrt(rc2 - d2) * b.cell_inv[0], 1.0e6);
        xlo = (int)floor(u - w - 1e-6);
        xhi = (int)floor(u + w + 1e-6);
        if (xhi - xlo + 1 >= b.nc[0]) {
          xlo = 0;
          xhi = b.nc[0] - 1;
        }
      }
      int row = (wz * b.nc[1] + wrapc(cy, b.nc[1])) * b.nc[0];
      int cx = xlo;
      while (cx <= xhi) {
        int wx = wrapc(cx, b.nc[0]);
        int run = min(xhi - cx, b.nc[0] - 1 - wx) + 1;
        int j1 = V.cstart[row + wx + run];
        pc.visited += (unsigned long long)(j1 - V.cstart[row + wx]);
        for (int j = V.cstart[row + wx]; j < j1; ++j) {
          if (qm) {  // Check_MoleculePair_Cutoff
            const double4_32a mc = b.mcom[V.corig[j]];
            const double cx = fold(qm->com[0] - mc.x, b.hL[0], b.L[0]);
            const double cy = fold(qm->com[1] - mc.y, b.hL[1], b.L[1]);
            const double cz = fold(qm->com[2] - mc.z, b.hL[2], b.L[2]);
            if (sqrt(cx * cx + cy * cy + cz * cz) > rint0 + qm->dcom + mc.w) continue;
          }
          double4_32a a = P[j];
          double dx = fold(p[0] - a.x, b.hL[0], b.L[0]);
          double dy = fold(p[1] - a.y, b.hL[1], b.L[1]);
          double dz = fold(p[2] - a.z, b.hL[2], b.L[2]);
          double r2 = dx * dx + dy * dy + dz * dz;
          if (cbmc && b.sector && r2 < rmin2_pair(b, T.ntypes, qt, V.ptype[j])) return true;  // check_overlap
          if (cbmc && b.tab_res > 0) {  // Estimate_MoleculePair_Energy
            double et = 0.0;
            const int k = table_pair(b, T.ntypes, r2, qt, V.ptype[j], qch, a.w, et);
            if (k == 2) return true;
            if (k == 1) {
              ++pc.in_cut;
              acc += et;
              eabs += fabs(et);
            }
            continue;
          }
          if (r2 < b.rcut_lowsq) return true;
          int m = cutoff_mask(b, r2, cbmc);
          if (!qq_on) m &= 1;
          if (m) ++pc.in_cut;
          if (m & 1) {
            double ev = vdw_pair(T, b, qt, V.ptype[j], r2, 1.0);
            acc += ev;
            eabs += fabs(ev);
          }
          if (m & 2) {
            double eq = qq_pair_inter(b, qch * a.w, r2);
            acc += eq;
            eabs += fabs(eq);
          }
        }
        cx += run;
      }
    }
  }
  eout = acc;
  pc.eabs = eabs;
  return false;
}

// Compute_Max_COM_Distance (get_com.f90:220-295) over the atoms of `mask`
__device__ inline double max_dcom_of(const double* r, unsigned mask, const double com[3], int n) {
  double dmax = 0.0;
  for (int k = 0; k < n; ++k) {
    if (!((mask >> k) & 1u)) continue;
    const double dx = r[3 * k] - com[0], dy = r[3 * k + 1] - com[1], dz = r[3 * k + 2] - com[2];
    dmax = fmax(dmax, dx * dx + dy * dy + dz * dz);
  }
  return sqrt(dmax);
}

// ---------------------------------------------------------------------------
// K8: one Widom insertion per thread

__device__ void run_insertion(const WidomSpecies& S, const SpeciesPools& P, const PairTable& T, const BoxView& V,
                              const double* __restrict__ lib, Lfsr rng, WRec& rec, int& status, double* xyz_out,
                              CassWidomTrace* tr, PairCount& pc) {
  const BoxDev& b = *V.b;
  const SpeciesDevHdr& H = P.hdr[S.is0];
  const int n = S.natoms;
  const double beta = b.beta;
  double r[3 * kMaxAtoms];
  unsigned exist = 0u;
  double ln_pbias = 0.0, ln_pseq;
  double first_sum = 0.0;
  int selected = 0;
  bool cbmc_overlap = false;

  // Step 1: first fragment and growth order (fragment_growth.f90:218-253, 1317-1446)
  double u = rng.next();
  int fstart = 0;
  while (fstart < S.nfrag && !(u < S.cum_prob_ins[fstart])) ++fstart;
  if (fstart >= S.nfrag) fstart = S.nfrag - 1;
  ln_pseq = S.ln_prob_ins[fstart];
  int order[kMaxFrags];
  int norder = 1;
  order[0] = fstart;
  unsigned live = 1u << fstart;
  if (S.nfrag > 1) {
    int hang[kMaxFrags];
    int nh = 0;
    for (int k = 0; k < S.frag_nconnect[fstart]; ++k) {
      int f = S.frag_connect[fstart][k];
      if (!((live >> f) & 1u)) hang[nh++] = f;
    }
    while (nh > 0) {
      double prob[kMaxFrags], cum[kMaxFrags];
      for (int k = 0; k < nh; ++k) {
        prob[k] = (double)(S.frag_natoms[hang[k]] - 2);
        cum[k] = (k == 0 ? 0.0 : cum[k - 1]) + prob[k];
      }
      double tot = cum[nh - 1];
      for (int k = 0; k < nh; ++k) {
        prob[k] = prob[k] / tot;
        cum[k] = cum[k] / tot;
      }
      double uu = rng.next();
      int k = 0;
      while (k < nh && !(uu < cum[k])) ++k;
      if (k >= nh) k = nh - 1;
      int f = hang[k];
      ln_pseq = ln_pseq + log(prob[k]);
      order[norder++] = f;
      live |= 1u << f;
      for (int q = k; q + 1 < nh; ++q) hang[q] = hang[q + 1];
      --nh;
      for (int q = 0; q < S.frag_nconnect[f]; ++q) {
        int g = S.frag_connect[f][q];
        if (!((live >> g) & 1u) && nh < kMaxFrags) hang[nh++] = g;
      }
    }
  }

  // Step 2: library conformation of the first fragment (:274-304)
  const int nfa = S.frag_natoms[fstart];
  {
    int nconf = S.nconfig[fstart];
    int conf = (int)(rng.next() * nconf);
    if (conf >= nconf) conf = nconf - 1;
    const double* L0 = lib + S.lib_off[fstart] + (size_t)conf * nfa * 3;
    for (int i = 0; i < nfa; ++i) {
      int a = S.frag_atoms[fstart][i];
      r[3 * a] = L0[3 * i];
      r[3 * a + 1] = L0[3 * i + 1];
      r[3 * a + 2] = L0[3 * i + 2];
      exist |= 1u << a;
    }
  }

  // Step 3: Get_COM + Rotate_Molecule_Eulerian (rotation_routines.f90:41-137)
  double com[3];
  get_com(S, r, exist, com);
  {
    double theta = acos(1.0 - 2.0 * rng.next());
    double phi = (1.0 - 2.0 * rng.next()) * kPI;
    double psi = (1.0 - 2.0 * rng.next()) * kPI;
    double st, ct, sp, cp, ss, cs;
    sincos(theta, &st, &ct);
    sincos(phi, &sp, &cp);
    sincos(psi, &ss, &cs);
    double r11 = cs * cp - ct * sp * ss, r12 = cs * sp + ct * cp * ss, r13 = ss * st;
    double r21 = -ss * cp - ct * sp * cs, r22 = -ss * sp + ct * cp * cs, r23 = cs * st;
    double r31 = st * sp, r32 = -st * cp, r33 = ct;
    for (int i = 0; i < nfa; ++i) {
      int a = S.frag_atoms[fstart][i];
      double x = r[3 * a] - com[0], y = r[3 * a + 1] - com[1], z = r[3 * a + 2] - com[2];
      r[3 * a] = (r11 * x + r12 * y + r13 * z) + com[0];
      r[3 * a + 1] = (r21 * x + r22 * y + r23 * z) + com[1];
      r[3 * a + 2] = (r31 * x + r32 * y + r33 * z) + com[2];
    }
  }

  // Step 4: kappa_ins trial positions of the first fragment (:383-620)
  const int ki = S.kappa_ins;
  double nrg[kMaxKappa], w[kMaxKappa];
  unsigned ovm = 0u;
  double r0[3 * kMaxAtoms];
  for (int i = 0; i < 3 * n; ++i) r0[i] = r[i];
  const double com_old[3] = {com[0], com[1], com[2]};
  // molecule-pair cutoff boxes: the fragment at a trial centre has that COM
  // and the max_dcom of its atoms about it
  const bool mp = b.mcom != nullptr;
  QueryMol qm;
  qm.dcom = 0.0;
  if (mp) qm.dcom = max_dcom_of(r0, exist, com_old, n);
  Lfsr replay = rng;
  for (int it = 0; it < ki; ++it) {
    double ax = (0.5 - rng.next()) * b.L[0];
    double ay = (0.5 - rng.next()) * b.L[1];
    double az = (0.5 - rng.next()) * b.L[2];
    qm.com[0] = ax;
    qm.com[1] = ay;
    qm.com[2] = az;
    double e = 0.0;
    bool ov = false;
    for (int i = 0; i < nfa && !ov; ++i) {
      int a = S.frag_atoms[fstart][i];
      double p[3] = {r0[3 * a] - com_old[0] + ax, r0[3 * a + 1] - com_old[1] + ay, r0[3 * a + 2] - com_old[2] + az};
      double ea;
      ov = query_box(V, T, p, S.type[a], S.q[a], true, S.want_qq_cbmc != 0, ea, pc, mp ? &qm : nullptr);
      e += ea;
    }
    nrg[it] = e;
    w[it] = 0.0;
    if (ov) {
      ovm |= 1u << it;
    } else {
      double nk = beta * nrg[it];
      if (nk >= kMAX_KBT) {
        ovm |= 1u << it;
      } else {
        w[it] = exp(-nk);
        first_sum += nrg[it];
      }
    }
    if (it > 0) w[it] = w[it - 1] + w[it];
  }
  int sel = -1;
  if (ovm == ((ki >= 32) ? 0xffffffffu : ((1u << ki) - 1u))) {
    cbmc_overlap = true;
  } else {
    double rn = rng.next() * w[ki - 1];
    int i = 0;
    while (i < ki && !(rn < w[i])) ++i;
    if (i == ki) cbmc_overlap = true;
    else sel = i;
  }
  if (!cbmc_overlap) {
    ln_pbias = ln_pbias - beta * nrg[sel] - log(w[ki - 1]);
    double ax = 0, ay = 0, az = 0;
    for (int k = 0; k <= sel; ++k) {
      ax = (0.5 - replay.next()) * b.L[0];
      ay = (0.5 - replay.next()) * b.L[1];
      az = (0.5 - replay.next()) * b.L[2];
    }
    for (int i = 0; i < nfa; ++i) {
      int a = S.frag_atoms[fstart][i];
      r[3 * a] = r0[3 * a] - com_old[0] + ax;
      r[3 * a + 1] = r0[3 * a + 1] - com_old[1] + ay;
      r[3 * a + 2] = r0[3 * a + 2] - com_old[2] + az;
    }
    selected = sel + 1;
  }

  // Step 5: Fragment_Placement (:1449-2132)
  if (!cbmc_overlap && norder > 1) {
    double e_prev = dihedral_masked(H, P, r, exist);
    unsigned placed = 1u << fstart;
    const int kd = S.kappa_dih;
    double dn[kMaxKappa], dd[kMaxKappa];
    for (int oi = 1; oi < norder && !cbmc_overlap; ++oi) {
      const int f = order[oi];
      const int nf = S.frag_natoms[f];
      unsigned grown = exist;
      int nconf = S.nconfig[f];
      int cf = (int)(rng.next() * nconf);
      cf = (int)(rng.next() * nconf);  // the duplicated draw of fragment_growth.f90:1578,1584
      if (cf >= nconf) cf = nconf - 1;
      double cfg[3 * kMaxAtoms];
      const double* Lf = lib + S.lib_off[f] + (size_t)cf * nf * 3;
      for (int j = 0; j < nf; ++j) {
        int a = S.frag_atoms[f][j];
        exist |= 1u << a;
        cfg[3 * a] = Lf[3 * j];
        cfg[3 * a + 1] = Lf[3 * j + 1];
        cfg[3 * a + 2] = Lf[3 * j + 2];
      }
      const unsigned combined = exist, newex = combined & ~grown;
      int fc = -1;
      for (int q = 0; q < S.frag_nconnect[f]; ++q) {
        int g = S.frag_connect[f][q];
        if ((placed >> g) & 1u) {
          fc = g;
          break;
        }
      }
      if (fc < 0) {  // no placed neighbour: the fragment graph is not connected
        cbmc_overlap = true;
        break;
      }
      const int anc_i = S.frag_atoms[f][0], anc_c = S.frag_atoms[fc][0];
      int ids[kMaxAtoms], nid = 0;
      for (int j = 0; j < nf; ++j) {
        int a = S.frag_atoms[f][j];
        if (a != anc_i && a != anc_c) ids[nid++] = a;
      }
      unsigned idmask = 0u;
      for (int j = 0; j < nid; ++j) idmask |= 1u << ids[j];
      int atom_ifrag = nid > 0 ? ids[0] : S.frag_atoms[f][nf - 1];
      int atom_fc = S.frag_atoms[fc][S.frag_natoms[fc] - 1];
      for (int j = 0; j < S.frag_natoms[fc]; ++j) {
        int a = S.frag_atoms[fc][j];
        if (a != anc_i && a != anc_c) {
          atom_fc = a;
          break;
        }
      }
      double v1[3], v2[3], al_i[9], hg_i[9], al_c[9], hg_c[9];
      for (int d = 0; d < 3; ++d) {
        v1[d] = cfg[3 * anc_i + d] - cfg[3 * anc_c + d];
        v2[d] = cfg[3 * atom_ifrag + d] - cfg[3 * anc_c + d];
      }
      aligner_hanger(v1, v2, al_i, hg_i);
      for (int d = 0; d < 3; ++d) {
        v1[d] = r[3 * anc_i + d] - r[3 * anc_c + d];
        v2[d] = r[3 * atom_fc + d] - r[3 * anc_c + d];
      }
      aligner_hanger(v1, v2, al_c, hg_c);
      const double tx = cfg[3 * anc_c], ty = cfg[3 * anc_c + 1], tz = cfg[3 * anc_c + 2];
      for (int j = 0; j < nf; ++j) {
        int a = S.frag_atoms[f][j];
        double x = cfg[3 * a] - tx, y = cfg[3 * a + 1] - ty, z = cfg[3 * a + 2] - tz;
        cfg[3 * a] = x * al_i[0] + y * al_i[1] + z * al_i[2];
        cfg[3 * a + 1] = x * al_i[3] + y * al_i[4] + z * al_i[5];
        cfg[3 * a + 2] = x * al_i[6] + y * al_i[7] + z * al_i[8];
      }
      const double theta0 = kTWOPI * rng.next();
      const double dtheta = kTWOPI / (double)kd;
      unsigned dov = 0u;
      double dw[kMaxKappa];
      double theta = theta0;
      for (int ii = 0; ii < kd; ++ii) {
        if (ii > 0) theta = theta + dtheta;
        double sth, cth;
        sincos(theta, &sth, &cth);
        for (int j = 0; j < nid; ++j) {
          int a = ids[j];
          double x = cfg[3 * a], y = cfg[3 * a + 1], z = cfg[3 * a + 2];
          double yr = cth * y + sth * z, zr = -sth * y + cth * z;
          r[3 * a] = (x * hg_c[0] + yr * hg_c[1] + zr * hg_c[2]) + r[3 * anc_c];
          r[3 * a + 1] = (x * hg_c[3] + yr * hg_c[4] + zr * hg_c[5]) + r[3 * anc_c + 1];
          r[3 * a + 2] = (x * hg_c[6] + yr * hg_c[7] + zr * hg_c[8]) + r[3 * anc_c + 2];
        }
        dn[ii] = 0.0;
        dd[ii] = 0.0;
        exist &= ~idmask;
        double niv = 0.0, niq = 0.0, noq = 0.0;
        bool ov = false;
        for (int j = 0; j < nid; ++j) {
          exist |= 1u << ids[j];
          double eiv, eiq, eoq;
          if (atom_intra(H, P, b, T, ids[j], r, exist, eiv, eiq, eoq)) {
            ov = true;
            break;
          }
          niv += eiv;
          niq += eiq;
          noq += eoq;
        }
        if (ov) {
          dw[ii] = ii > 0 ? dw[ii - 1] : 0.0;
          dov |= 1u << ii;
          exist |= idmask;
          continue;
        }
        double einter = 0.0;
        if (mp) {  // the new atoms of the trial (fragment_growth.f90 Fragment_Placement energy call)
          get_com(S, r, newex, qm.com);
          qm.dcom = max_dcom_of(r, newex, qm.com, n);
        }
        for (int a = 0; a < n && !ov; ++a) {
          if (!((newex >> a) & 1u)) continue;
          double p[3] = {r[3 * a], r[3 * a + 1], r[3 * a + 2]};
          double ea;
          ov = query_box(V, T, p, S.type[a], S.q[a], true, S.want_qq_cbmc != 0, ea, pc, mp ? &qm : nullptr);
          einter += ea;
        }
        exist = combined;
        if (ov) {
          dw[ii] = 0.0;
          dov |= 1u << ii;
        } else {
          double ed = dihedral_masked(H, P, r, exist);
          dd[ii] = ed;
          dn[ii] = ed + niv + niq + einter + noq - e_prev;
          double nk = beta * dn[ii];
          if (nk >= kMAX_KBT) {
            dw[ii] = 0.0;
            dov |= 1u << ii;
          } else {
            dw[ii] = exp(-nk);
          }
        }
        if (ii > 0) dw[ii] = dw[ii - 1] + dw[ii];
      }
      if (dov == ((kd >= 32) ? 0xffffffffu : ((1u << kd) - 1u))) {
        cbmc_overlap = true;
        break;
      }
      double pp = rng.next() * dw[kd - 1];
      int trl = 0;
      while (trl < kd && !(pp < dw[trl])) ++trl;
      if (trl == kd) {
        cbmc_overlap = true;
        break;
      }
      ln_pbias = ln_pbias - beta * dn[trl] - log(dw[kd - 1]);
      theta = theta0;
      for (int ii = 1; ii <= trl; ++ii) theta = theta + dtheta;
      double sth, cth;
      sincos(theta, &sth, &cth);
      for (int j = 0; j < nid; ++j) {
        int a = ids[j];
        double x = cfg[3 * a], y = cfg[3 * a + 1], z = cfg[3 * a + 2];
        double yr = cth * y + sth * z, zr = -sth * y + cth * z;
        r[3 * a] = (x * hg_c[0] + yr * hg_c[1] + zr * hg_c[2]) + r[3 * anc_c];
        r[3 * a + 1] = (x * hg_c[3] + yr * hg_c[4] + zr * hg_c[5]) + r[3 * anc_c + 1];
        r[3 * a + 2] = (x * hg_c[6] + yr * hg_c[7] + zr * hg_c[8]) + r[3 * anc_c + 2];
      }
      e_prev = dd[trl];
      placed |= 1u << f;
    }
    if (!cbmc_overlap) get_com(S, r, exist, com);
  }

  // widom_insert.f90:350-447
  ln_pbias = ln_pbias + ln_pseq;
  ln_pbias = ln_pbias + S.ln_kappa_ins;
  ln_pbias = ln_pbias + S.ln_kappa_dih_term;
  if (tr) {
    tr->ln_pbias = ln_pbias;
    tr->e_first_trial_sum = first_sum;
    tr->selected_trial = selected;
    tr->e_inter = 0.0;
    tr->e_inter_abs = 0.0;
  }
  rec = make_double4_32a(0.0, 0.0, 0.0, ln_pbias);
  if (cbmc_overlap) {
    status = 1;
    return;
  }
  const unsigned all = (n >= 32) ? 0xffffffffu : ((1u << n) - 1u);
  exist = all;
  if (S.nfrag > 1) {  // Fold_Molecule, orthorhombic branch
    for (int d = 0; d < 3; ++d) {
      if (com[d] > b.hL[d]) {
        com[d] = com[d] - b.L[d];
        for (int a = 0; a < n; ++a) r[3 * a + d] -= b.L[d];
      } else if (com[d] < -b.hL[d]) {
        com[d] = com[d] + b.L[d];
        for (int a = 0; a < n; ++a) r[3 * a + d] += b.L[d];
      }
    }
  }
  double e_inter = 0.0, e_abs = 0.0;
  if (mp) {  // the whole molecule, folded
    get_com(S, r, exist, qm.com);
    qm.dcom = max_dcom_of(r, exist, qm.com, n);
  }
  for (int a = 0; a < n; ++a) {
    double p[3] = {r[3 * a], r[3 * a + 1], r[3 * a + 2]};
    double ea;
    if (query_box(V, T, p, S.type[a], S.q[a], false, true, ea, pc, mp ? &qm : nullptr)) {
      status = 2;
      return;
    }
    e_inter += ea;
    e_abs += pc.eabs;
  }
  IntraOut io = molecule_intra(P, S.is0, b, T, r);
  if (io.overlap) {
    status = 3;
    return;
  }
  e_inter = e_inter + io.pqq;
  double dE_inter = e_inter + b.e_inter_constant;
  double dE_intra = io.ivdw + io.iqq;
  dE_intra = dE_intra + io.bond + io.angle + io.dih + io.imp;
  rec = make_double4_32a(dE_intra, dE_inter, io.angle, ln_pbias);
  status = 0;
  if (tr) {
    tr->e_inter = e_inter;
    tr->e_inter_abs = e_abs;
  }
  if (xyz_out)
    for (int i = 0; i < 3 * n; ++i) xyz_out[i] = r[i];
}

// ---------------------------------------------------------------------------
// Mixed-precision Widom kernel: a lane per insertion, FP32 throughout.
//
// GB300 issues FP64 at 1/64 of its FP32 rate, so this kernel reads only FP32
// tables (species, box constants, fragment libraries, cell-sorted atoms) and
// keeps the test molecule, the trial energies and the Boltzmann weights in
// FP32; pair energies accumulate in compensated FP32 sums.  Only the
// per-insertion record is widened to FP64 (adding the box's FP64 constant
// E_lrc_diff + E_self - E_recip_old).  Cell stencils carry a per-row
// periodic image shift, so the minimum-image fold per pair is needed only in
// a dimension whose stencil spans the whole box.

// Cell-list view of the CTA's box
struct BoxViewF {
  const BoxF* f;
  const float4* p32;   // cell-sorted atoms (x, y, z, type bits), smem or global
  const double4_32a* p64;  // the same atoms in FP64 (global): cutoff decisions near a cutoff
  const float* q32;    // their charges (global)
  const int* cstart;   // cell starts, local atom indices, smem or global
  const float2* ljp;   // (eps, sigma^2) [kMaxTypes][kMaxTypes], smem
};

// A pair of the full-cutoff pass whose FP32 r^2 lies within the band of a
// cutoff (kind 0: rcut_vdw^2 or rcut_coul^2; kind 1: rcut_low^2) where the
// FP32 and the FP64 decisions can differ: box atom j, test atom `atom`
struct BandPair {
  int j;
  float r2;
  unsigned char atom, kind, pad0, pad1;
};
constexpr int kMaxBand = 4;

struct QueryAcc {
  KahanF e;
  float eabs = 0.0f;
  unsigned long long visited = 0, in_cut = 0;
  int nband = 0;
};

// r^2 to a stored atom, through the row's image shift (folded in full dimensions)
__device__ __forceinline__ float pair_r2(const BoxF& f, const bool (&full)[3], bool fold_any, float qx, float qy,
                                         float qz, const float4& a) {
  float dx = qx - a.x, dy = qy - a.y, dz = qz - a.z;
  if (fold_any) {
    if (full[0]) dx = fold(dx, f.hL[0], f.L[0]);
    if (full[1]) dy = fold(dy, f.hL[1], f.L[1]);
    if (full[2]) dz = fold(dz, f.hL[2], f.L[2]);
  }
  return fmaf(dx, dx, fmaf(dy, dy, dz * dz));
}

// r^2 of two stored atoms at once on the packed FP32x2 pipe (FFMA2, sm_100 and
// later): the same operations and rounding as pair_r2 without a fold,
// qx - a.x formed as fma(a.x, -1, qx)
__device__ __forceinline__ float2 pair_r2_x2(float qx0, float qx1, float qy, float qz, const float4& a0,
                                             const float4& a1) {
  const float2 m1 = make_float2(-1.0f, -1.0f);
  const float2 dx = __ffma2_rn(make_float2(a0.x, a1.x), m1, make_float2(qx0, qx1));
  const float2 dy = __ffma2_rn(make_float2(a0.y, a1.y), m1, make_float2(qy, qy));
  const float2 dz = __ffma2_rn(make_float2(a0.z, a1.z), m1, make_float2(qz, qz));
  return __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
}

// Squared distance from coordinate p to the slab of unwrapped cell c (edge h,
// cells numbered from -hL), less a margin of 1e-3 cell so that FP32 rounding
// never drops a cell that holds an atom within the cutoff.
__device__ __forceinline__ float slab_d2_f(int c, float h, float hl, float p) {
  const float c0 = (float)c * h - hl;
  const float d = fmaxf(fmaxf(c0 - p, p - (c0 + h)) - 1.0e-3f * h, 0.0f);
  return d * d;
}

// The x-cells of a stencil row whose y / z slabs lie at squared distance d2
// from the query: the chord of the cutoff sphere, rem = rc^2 - d2 >= 0.  A row
// chord spanning the whole box is visited once with the minimum-image fold.
__device__ __forceinline__ void row_x_cells_f(const BoxF& f, float px, float rem, int& lo, int& hi, bool& fullx) {
  const float w = fminf(sqrtf(rem) * f.cinv[0], 1.0e5f);
  const float u = (px + f.hL[0]) * f.cinv[0];
  const int l = (int)floorf(fminf(fmaxf(u - w - 1e-3f, -1.0e6f), 1.0e6f));
  const int h = (int)floorf(fminf(fmaxf(u + w + 1e-3f, -1.0e6f), 1.0e6f));
  fullx = h - l + 1 >= f.nc[0];
  lo = fullx ? 0 : l;
  hi = fullx ? f.nc[0] - 1 : h;
}

// FP64 minimum-image r^2 between p and cell-sorted atom j, as the FP64 query
// forms it (Minimum_Image_Separation, orthorhombic branch)
__device__ __noinline__ double exact_r2(const BoxF& f, const double4_32a* p64, int j, const double* p) {
  const double4_32a a = p64[j];
  const double dx = fold(p[0] - a.x, f.hL64[0], f.L64[0]);
  const double dy = fold(p[1] - a.y, f.hL64[1], f.L64[1]);
  const double dz = fold(p[2] - a.z, f.hL64[2], f.L64[2]);
  return dx * dx + dy * dy + dz * dz;
}

// Core overlap of the full-cutoff pass: an FP32 r^2 within band_low of
// rcut_low^2 is decided from the FP64 coordinates
__device__ __forceinline__ bool overlap_exact(const BoxViewF& V, float r2, int j, const double* p64) {
  const BoxF& f = *V.f;
  if (r2 < f.low2 - f.band_low) return true;
  if (r2 >= f.low2 + f.band_low) return false;
  return exact_r2(f, V.p64, j, p64) < f.low2d;
}

// LJ and real-space Ewald energy of one pair inside the selection radius.  An
// FP32 r^2 within a band of the vdW or Coulomb cutoff is compared with the cutoff
// in FP64, from the FP64 coordinates, so that the pair counts exactly when the
// FP64 energy counts it.
__device__ __forceinline__ void pair_energy_exact(const BoxViewF& V, QueryAcc& A, const float4& a, int j, float r2,
                                                  const float2* lrow, bool vdw_on, bool qq_on, float rv2, float rq2,
                                                  float qa, const double* p64) {
  const BoxF& f = *V.f;
  bool in_v = r2 <= rv2, in_q = r2 <= rq2;
  if (fabsf(r2 - rv2) <= f.band_v || fabsf(r2 - rq2) <= f.band_q) {
    const double d2 = exact_r2(f, V.p64, j, p64);
    in_v = d2 <= f.rv2d;
    in_q = d2 <= f.rq2d;
  }
  const int tj = __float_as_int(a.w);
  if (vdw_on && tj >= 0 && in_v) {
    const float2 es = lrow[tj];
    const float ev = lj_pair_f(es.x, es.y, r2);
    A.e.add(ev);
    A.eabs += fabsf(ev);
  }
  if (qq_on && in_q) {
    const float eq = qq_ewald_inter_f(f.alpha, qa * V.q32[j], r2);
    A.e.add(eq);
    A.eabs += fabsf(eq);
  }
}

// FP32 energy of one test atom at p against the box atoms within the full cutoff,
// added to A, the cutoff decisions within a band made in FP64 from the FP64
// coordinates p64 of the query atom.  Returns true on core overlap (r^2 <
// rcut_low^2), as Compute_MoleculePair_Energy (energy_routines.f90:1676-1679) does.
__device__ bool query_f_exact(const BoxViewF& V, QueryAcc& A, float px, float py, float pz, int ta, float qa,
                              const double* p64) {
  const BoxF& f = *V.f;
  const float rc = f.rc_full;
  const float p[3] = {px, py, pz};
  int lo[3], hi[3];
  bool full[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const float w = fminf(rc * f.cinv[d], 1.0e5f);
    const float ul = fminf(fmaxf((p[d] + f.hL[d]) * f.cinv[d] - w - 1e-3f, -1.0e6f), 1.0e6f);
    const float uh = fminf(fmaxf((p[d] + f.hL[d]) * f.cinv[d] + w + 1e-3f, -1.0e6f), 1.0e6f);
    const int l = (int)floorf(ul), h = (int)floorf(uh);
    full[d] = h - l + 1 >= f.nc[d];
    lo[d] = full[d] ? 0 : l;
    hi[d] = full[d] ? f.nc[d] - 1 : h;
  }
  const float rv2 = f.rv2;
  const float rq2 = f.rq2;
  const bool vdw_on = ta >= 0;
  const bool qq_on = f.charge_on && qa != 0.0f;
  // the selection and overlap radii, widened by the FP32 bands
  const float band = fmaxf(vdw_on ? f.band_v : 0.0f, qq_on ? f.band_q : 0.0f);
  const float rsel2 = fmaxf(vdw_on ? rv2 : -1.0f, qq_on ? rq2 : -1.0f) + band;
  const float low2q = f.low2 + f.band_low;
  const float rc2 = rc * rc;
  const float2* lrow = V.ljp + (vdw_on ? ta : 0) * kMaxTypes;
  const int nc0 = f.nc[0], nc1 = f.nc[1], nc2 = f.nc[2];
  for (int cz = lo[2]; cz <= hi[2]; ++cz) {
    const int sz = cell_image(cz, nc2);
    const int wz = cz + sz * nc2;
    const float qz = pz + (float)sz * f.L[2];
    const float dz2 = full[2] ? 0.0f : slab_d2_f(cz, f.ch[2], f.hL[2], pz);
    if (dz2 > rc2 || abs(sz) > 1) continue;  // a separation moves by one box edge at most
    for (int cy = lo[1]; cy <= hi[1]; ++cy) {
      const float d2 = full[1] ? dz2 : dz2 + slab_d2_f(cy, f.ch[1], f.hL[1], py);
      if (d2 > rc2 || abs(cell_image(cy, nc1)) > 1) continue;
      int xlo, xhi;
      bool fl[3] = {false, full[1], full[2]};
      row_x_cells_f(f, px, rc2 - d2, xlo, xhi, fl[0]);
      const bool fold_any = fl[0] || fl[1] || fl[2];
      const int sy = cell_image(cy, nc1);
      const int wy = cy + sy * nc1;
      const float qy = py + (float)sy * f.L[1];
      const int row = (wz * nc1 + wy) * nc0;
      int cx = xlo;
      while (cx <= xhi) {
        const int sx = cell_image(cx, nc0);
        const int wx = cx + sx * nc0;
        const int run = min(xhi - cx, nc0 - 1 - wx) + 1;
        const float qx = px + (float)sx * f.L[0];
        const int j0 = V.cstart[row + wx], j1 = abs(sx) <= 1 ? V.cstart[row + wx + run] : j0;
        for (int j = j0; j < j1; ++j) {
          const float4 a = V.p32[j];
          const float r2 = pair_r2(f, fl, fold_any, qx, qy, qz, a);
          if (r2 < low2q && overlap_exact(V, r2, j, p64)) return true;
          if (r2 <= rsel2) pair_energy_exact(V, A, a, j, r2, lrow, vdw_on, qq_on, rv2, rq2, qa, p64);
        }
        cx += run;
      }
    }
  }
  return false;
}

// ---------------------------------------------------------------------------
// Warp-wide neighbour queries of the mixed Widom kernel.
//
// A lane owns an insertion and does its serial steps (draws, geometry, weights);
// the queries of all lanes are put in a queue in shared memory and the warp
// works through them together, one (query, stencil row) per lane.  Rows of
// different queries fill the 32 lanes whatever the insertions' own states are:
// with a query per lane a warp instruction did the work of 7.6 lanes, because
// the insertions end their queries at different candidates.  A row's pairs
// within the selection radius are listed first and their energies formed
// afterwards, so that the energy code runs for full lists and not for the odd
// lane whose candidate happens to be near.
constexpr int kCoopItems = 128;  // rows of one batch of queries
constexpr int kCoopHits = 8;     // listed pairs per lane

// Scratch of one warp
struct CoopWarp {
  float4 pos[32];            // query point and type; then its sum (s, c, sum of |terms|)
  int2 st[32];               // first row (cy | cz << 16), rows per slab | slabs << 8 | full y, z << 16
  float q[32];               // charge of the query atom
  int own[32];               // owner lane | atom << 8
  int ov[32];                // core overlap met
  float2 part[kCoopItems];   // partial sum (s, c) of a (query, row)
  float pabs[kCoopItems];    // its sum of |terms|
  float2 hit[kCoopHits][32]; // r^2 and box atom of the listed pairs of a lane
  int nband[32];             // band pairs met by an owner's full-cutoff pass
  float band_r2[32][kMaxBand];  // the first of them: r^2, box atom, atom | kind << 7
  int band_j[32][kMaxBand];
  unsigned char band_at[32][kMaxBand];
};

// cells of dimension d within rc of p, as a query's stencil spans them
__device__ __forceinline__ void stencil_f(const BoxF& f, int d, float p, float rc, int& lo, int& n, bool& full) {
  const float w = fminf(rc * f.cinv[d], 1.0e5f);
  const float ul = fminf(fmaxf((p + f.hL[d]) * f.cinv[d] - w - 1e-3f, -1.0e6f), 1.0e6f);
  const float uh = fminf(fmaxf((p + f.hL[d]) * f.cinv[d] + w + 1e-3f, -1.0e6f), 1.0e6f);
  const int l = (int)floorf(ul), h = (int)floorf(uh);
  full = h - l + 1 >= f.nc[d];
  lo = full ? 0 : l;
  n = full ? f.nc[d] : h - l + 1;
}

// Neighbour lists on a grid of voxels: the atoms within the query radius plus half
// a voxel diagonal of a voxel's centre, so every query point in the voxel reads one
// contiguous list instead of the rows of a cell stencil (27 entries for 13 atoms
// within 6.5 A of the benchmark's fluid, against 65 visited through the cells).  An
// entry holds the atom and its periodic image.  The atoms that may lie within
// rcut_low come first.
struct VoxGrid {
  int nv[3];
  float inv[3];    // voxels per A
  float edge[3];
  float R2;        // list radius squared, about the voxel centre
  float near2;     // squared radius of the atoms that come first
  int off;         // first record of the box
  int on;
};
constexpr unsigned kVoxAtomBits = 23;
constexpr unsigned kVoxAtomMask = (1u << kVoxAtomBits) - 1u;
// An entry's image code is kImage0 + sx + 7 sy + 49 sz, a query point's own shift is added to
// it.  Minimum_Image_Separation (minimum_image_separation.f90:35-112) moves a separation by
// one box edge at most, so a sum beyond that is no pair: its shift is out of every reach.
constexpr int kImages = 343, kImage0 = 171;
constexpr float kNoImage = 1.0e15f;
__device__ __forceinline__ int image_of(int code, int d) {  // shift in dimension d, in box edges
  return (d == 0 ? code % 7 : d == 1 ? code / 7 % 7 : code / 49) - 3;
}
__device__ __forceinline__ bool image_valid(int code) {
  return abs(image_of(code, 0)) <= 1 && abs(image_of(code, 1)) <= 1 && abs(image_of(code, 2)) <= 1;
}

// Dynamic shared memory of a CTA: the head, one CoopWarp per warp, then (with
// SMEM) the box's cell starts and atoms at the offsets of its CoopBox.
struct CoopHead {
  BoxF f;
  VoxGrid vox[2];                     // neighbour lists of the CBMC and the full-cutoff radius
  float4 shift[kImages];              // (sx Lx, sy Ly, sz Lz) of an image code
  float2 ljp[kMaxTypes * kMaxTypes];  // (eps, sigma^2)
  double ec;
  int atom_off, cell_off, natoms;
  int rows_cbmc, rows_full;  // row slots of a query of either radius
};
struct CoopBox {
  const uint4* vrec;    // voxel records of the batch: first word of the list, near entries, entries
  const uint4* vlist;   // their entries, four to a word
  const float4* p32;  // global (SMEM false)
  const float* q32;
  const int* cstart;
  const double4_32a* c64;  // FP64 kernel
  const PairTable* T;
  unsigned off_cells, off_atoms;
};
extern __shared__ __align__(32) unsigned char smem[];
__device__ __forceinline__ CoopHead& coop_head() { return *reinterpret_cast<CoopHead*>(smem); }
constexpr unsigned kCoopHeadBytes = (sizeof(CoopHead) + 31) & ~31u;
__device__ __forceinline__ CoopWarp& coop_warp() {
  return reinterpret_cast<CoopWarp*>(smem + kCoopHeadBytes)[threadIdx.x >> 5];
}

// most cells a stencil of radius rc spans in dimension d
__device__ __forceinline__ int stencil_max(const BoxF& f, int d, float rc) {
  return min(f.nc[d], (int)floorf(fminf(2.0f * rc * f.cinv[d], 1.0e5f) + 4.0e-3f) + 2);
}

// a band pair of owner lane `own`, atom `atom` noted in W (all lanes of a warp may call it at once)
__device__ __forceinline__ void coop_note(CoopWarp& W, int own, int j, float r2, int kind) {
  const int lane = own & 0xff, s = atomicAdd(&W.nband[lane], 1);
  if (s >= kMaxBand) return;  // k_widom_fix redoes the pass
  W.band_r2[lane][s] = r2;
  W.band_j[lane][s] = j;
  W.band_at[lane][s] = (unsigned char)(own >> 8 | kind << 7);
}

// The energies of the nq queries of W (pos, q, own, st filled, ov cleared): sums
// left in pos, overlaps in ov.  rows: row slots per query.  DETECT: the
// full-cutoff pass with its band notes; OPT: a CBMC query with the CBMC options.
template <bool SMEM, bool COUNT, bool OPT, bool DETECT>
__device__ __noinline__ void coop_eval(const CoopBox B, int nq, bool want_qq, QueryAcc& cnt) {
  const CoopHead& H = coop_head();
  const BoxF& f = H.f;
  CoopWarp& W = coop_warp();
  const float4* p32;
  const int* cstart;
  if constexpr (SMEM) {
    p32 = reinterpret_cast<const float4*>(smem + B.off_atoms);
    cstart = reinterpret_cast<const int*>(smem + B.off_cells);
  } else {
    p32 = B.p32;
    cstart = B.cstart;
  }
  const int rows = DETECT ? H.rows_full : H.rows_cbmc;
  const int lane = threadIdx.x & 31;
  const float rc = DETECT ? f.rc_full : f.rc_cbmc;
  const float rv2 = DETECT ? f.rv2 : f.rcb2;
  const float rq2 = DETECT ? f.rq2 : f.rcb2;
  const float rc2 = rc * rc;
  const int nc0 = f.nc[0], nc1 = f.nc[1], nc2 = f.nc[2];
  const int rs = min(rows, kCoopItems);
  const int nbatch = kCoopItems / rs;  // queries of a batch
  const float inv_rs = 1.0f / (float)rs;
  for (int q0 = 0; q0 < nq; q0 += nbatch) {
    const int nb = min(nbatch, nq - q0);
    for (int base = 0; base < nb * rs; base += 32) {
      const int item = base + lane;
      const bool valid = item < nb * rs;
      const int ql = valid ? (int)(((float)item + 0.5f) * inv_rs) : 0;
      const int qi = q0 + ql, slot = item - ql * rs;
      const float4 p = W.pos[qi];
      const int2 st = W.st[qi];
      const int ta = __float_as_int(p.w);
      const float qa = W.q[qi];
      const bool vdw_on = ta >= 0;
      const bool qq_on = want_qq && f.charge_on && qa != 0.0f;
      const float band = DETECT ? fmaxf(vdw_on ? f.band_v : 0.0f, qq_on ? f.band_q : 0.0f) : 0.0f;
      const float rsel2 = fmaxf(vdw_on ? rv2 : -1.0f, qq_on ? rq2 : -1.0f) + band;
      const float low2q = DETECT ? f.low2 + f.band_low : f.low2;
      const float rlo = fminf(vdw_on ? rv2 : 3.0e38f, qq_on ? rq2 : 3.0e38f) - band;
      const float2* lrow = H.ljp + (vdw_on ? ta : 0) * kMaxTypes;
      const float* rmrow = f.rmin2 + (vdw_on ? ta : 0) * kMaxTypes;
      const float qicf = qa * (float)kCHARGE_FACTOR;
      const int ny = st.y & 0xff, nrow = ny * ((st.y >> 8) & 0xff);
      const bool fully = (st.y >> 16) & 1, fullz = (st.y >> 17) & 1;
      const int lo1 = (int)(short)(st.x & 0xffff), lo2 = st.x >> 16;
      KahanF e;
      float eabs = 0.0f;
      bool ov = false;
      int nh = 0;
      // energies of the listed pairs
      auto drain = [&]() {
        const int most = __reduce_max_sync(0xffffffffu, nh);
        for (int h = 0; h < most; ++h)
          if (h < nh) {
            const float2 hv = W.hit[h][lane];
            const int j = __float_as_int(hv.y);
            const float r2 = hv.x;
            if (DETECT && r2 >= rlo) coop_note(W, W.own[qi], j, r2, 0);
            if (COUNT) ++cnt.in_cut;
            const int tj = __float_as_int(p32[j].w);
            if (vdw_on && tj >= 0 && r2 <= rv2) {
              const float2 es = lrow[tj];
              const float ev = lj_pair_f(es.x, es.y, r2);
              e.add(ev);
              eabs += fabsf(ev);
            }
            if (qq_on && r2 <= rq2) {
              const float eq = qq_ewald_inter_f(f.alpha, qa * B.q32[j], r2);
              e.add(eq);
              eabs += fabsf(eq);
            }
          }
        nh = 0;
      };
      const int turns = (rows + rs - 1) / rs;  // one, but for stencils of more rows than a batch holds
      for (int turn = 0; turn < turns; ++turn) {
        const int rr = slot + turn * rs;
        // the row's candidates: up to two runs of cells, the second beyond the box edge
        int ja = 0, na = 0, jb = 0, n = 0;
        float qxa = 0.0f, qxb = 0.0f, qy = 0.0f, qz = 0.0f;
        bool fl[3] = {false, fully, fullz};
        if (valid && rr < nrow && !ov && !W.ov[qi]) {
          const int iz = (int)(((float)rr + 0.5f) * (1.0f / (float)ny));
          const int cz = lo2 + iz, cy = lo1 + rr - iz * ny;
          const float dz2 = fullz ? 0.0f : slab_d2_f(cz, f.ch[2], f.hL[2], p.z);
          const float d2 = fully ? dz2 : dz2 + slab_d2_f(cy, f.ch[1], f.hL[1], p.y);
          const int sz = cell_image(cz, nc2), sy = cell_image(cy, nc1);
          // a separation moves by one box edge at most
          if (dz2 <= rc2 && d2 <= rc2 && abs(sz) <= 1 && abs(sy) <= 1) {
            qz = p.z + (float)sz * f.L[2];
            qy = p.y + (float)sy * f.L[1];
            int xlo, xhi;
            row_x_cells_f(f, p.x, rc2 - d2, xlo, xhi, fl[0]);
            const int* cs = cstart + ((cz + sz * nc2) * nc1 + cy + sy * nc1) * nc0;
            const int sx = cell_image(xlo, nc0);
            const int wx = xlo + sx * nc0;
            const int run = min(xhi - xlo, nc0 - 1 - wx) + 1;
            qxa = p.x + (float)sx * f.L[0];
            ja = cs[wx];
            n = na = abs(sx) <= 1 ? cs[wx + run] - ja : 0;
            if (xlo + run <= xhi && abs(sx - 1) <= 1) {
              qxb = p.x + (float)(sx - 1) * f.L[0];
              jb = cs[0];
              n += cs[xhi + (sx - 1) * nc0 + 1] - jb;
            }
            if (COUNT) cnt.visited += (unsigned long long)n;
          }
        }
        const bool fold_any = fl[0] || fl[1] || fl[2];
        const int most = __reduce_max_sync(0xffffffffu, n);
        jb -= na;
        for (int t = 0; t < most; t += 2) {
          if (t < n) {
            const bool two = t + 1 < n;
            const int j0 = t < na ? ja + t : jb + t, j1 = two ? (t + 1 < na ? ja + t + 1 : jb + t + 1) : j0;
            const float4 a0 = p32[j0], a1 = p32[j1];
            const float qx0 = t < na ? qxa : qxb, qx1 = t + 1 < na ? qxa : qxb;
            float r20, r21;
            if (!fold_any) {
              const float2 r2 = pair_r2_x2(qx0, qx1, qy, qz, a0, a1);
              r20 = r2.x;
              r21 = r2.y;
            } else {
              r20 = pair_r2(f, fl, fold_any, qx0, qy, qz, a0);
              r21 = pair_r2(f, fl, fold_any, qx1, qy, qz, a1);
            }
            if (!two) r21 = 3.0e38f;
            if (OPT) {
              for (int s = 0; s < 2 && !ov; ++s) {
                if (s == 1 && !two) break;
                const float r2 = s ? r21 : r20;
                const int j = s ? j1 : j0, tj = __float_as_int(s ? a1.w : a0.w);
                if (f.sector && r2 < (vdw_on && tj >= 0 ? rmrow[tj] : f.low2)) {
                  ov = true;
                } else if (f.tab_res > 0) {
                  float et = 0.0f;
                  // the table's charges count whatever want_qq says (energy_routines.f90:1563-1583)
                  const int k = table_pair_f(f.tab_v, f.tab_f2, f.tab_res, f.tab_shift, f.tab_rcs, f.tab_step,
                                             f.tab_inv_step, f.ntypes, r2, ta, tj, qicf,
                                             f.charge_on ? B.q32[j] : 0.0f, et);
                  if (k == 2) ov = true;
                  if (k == 1) {
                    e.add(et);
                    eabs += fabsf(et);
                  }
                } else if (r2 < f.low2) {
                  ov = true;
                } else if (r2 <= rsel2) {
                  W.hit[nh++][lane] = make_float2(r2, __int_as_float(j));
                }
              }
            } else {
              if (fminf(r20, r21) < low2q) {
                if (!DETECT || fminf(r20, r21) < f.low2 - f.band_low) {
                  ov = true;
                } else {
                  if (r20 < low2q) coop_note(W, W.own[qi], j0, r20, 1);
                  if (r21 < low2q) coop_note(W, W.own[qi], j1, r21, 1);
                }
              }
              if (r20 <= rsel2) W.hit[nh++][lane] = make_float2(r20, __int_as_float(j0));
              if (r21 <= rsel2) W.hit[nh++][lane] = make_float2(r21, __int_as_float(j1));
            }
            if (ov) {  // the query's energy is not asked for any more
              n = 0;
              nh = 0;
            }
          }
          if (__any_sync(0xffffffffu, nh > kCoopHits - 2)) drain();
        }
      }
      if (ov) W.ov[qi] = 1;
      __syncwarp();
      if (W.ov[qi]) nh = 0;
      drain();
      if (valid) {
        W.part[item] = make_float2(e.s, e.c);
        if (DETECT) W.pabs[item] = eabs;
      }
    }
    __syncwarp();
    if (lane < nb) {  // the rows of a query added in their order
      KahanF e;
      float ea = 0.0f;
      for (int s = 0; s < rs; ++s) {
        const float2 v = W.part[lane * rs + s];
        e.add(v.x);
        e.c += v.y;
        if (DETECT) ea += W.pabs[lane * rs + s];
      }
      W.pos[q0 + lane] = make_float4(e.s, e.c, ea, 0.0f);
    }
    __syncwarp();
  }
}

// the voxel record of point (x, y, z); code: its own image shift, to be added to an entry's
__device__ __forceinline__ uint4 vox_record(const BoxF& f, const VoxGrid& g, const uint4* vrec, float x, float y,
                                            float z, int& code) {
  const float p[3] = {x, y, z};
  int w[3], s[3];
  bool far = false;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    const int i = (int)floorf(fminf(fmaxf((p[d] + f.hL[d]) * g.inv[d], -1.0e6f), 1.0e6f));
    s[d] = cell_image(i, g.nv[d]);
    w[d] = i + s[d] * g.nv[d];
    far = far || s[d] > 2 || s[d] < -2;
  }
  code = s[0] + 7 * s[1] + 49 * s[2];
  if (far) {  // no image of an atom is one box edge away
    code = 0;
    return make_uint4(0u, 0u, 0u, 0u);
  }
  return __ldg(&vrec[g.off + (w[2] * g.nv[1] + w[1]) * g.nv[0] + w[0]]);
}

// Core overlap of a CBMC query point of type ta: only the first entries of its list can be
// that near.  OPT: check_overlap (sector_routines.f90:160-233) and the energy table's rule.
template <bool SMEM, bool OPT>
__device__ __forceinline__ bool vox_overlap(const CoopBox& B, const CoopHead& H, float x, float y, float z, int ta) {
  const BoxF& f = H.f;
  const float4* p32;
  if constexpr (SMEM) p32 = reinterpret_cast<const float4*>(smem + B.off_atoms);
  else p32 = B.p32;
  int code;
  const uint4 rec = vox_record(H.f, H.vox[0], B.vrec, x, y, z, code);
  const unsigned* list = reinterpret_cast<const unsigned*>(B.vlist + rec.x);
  const int nnear = (int)rec.y;
  bool ov = false;
  for (int t = 0; t < nnear && !ov; ++t) {
    const unsigned e = __ldg(&list[t]);
    const float4 a = p32[e & kVoxAtomMask], sh = H.shift[(int)(e >> kVoxAtomBits) + code];
    const float dx = (x + sh.x) - a.x, dy = (y + sh.y) - a.y, dz = (z + sh.z) - a.z;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    ov = OPT && f.tab_res > 0 ? r2 - f.tab_shift < f.tab_step : r2 < f.low2;
    if (OPT && f.sector) {
      const int tj = __float_as_int(a.w);
      ov = ov || r2 < (ta >= 0 && tj >= 0 ? f.rmin2[ta * kMaxTypes + tj] : f.low2);
    }
  }
  return ov;
}

// A compensated sum of the even and the odd entries of a list, and its sum of |terms|
struct PairSum {
  float2 s = make_float2(0.0f, 0.0f), c = make_float2(0.0f, 0.0f);
  float a = 0.0f;
  __device__ __forceinline__ void first(float2 v) {  // the first term
    s = v;
    c = make_float2(0.0f, 0.0f);
  }
  __device__ __forceinline__ void add(float2 v) {  // TwoSum: the rounding error of the addition, exactly
    const float2 t = __fadd2_rn(s, v);
    const float2 m1 = make_float2(-1.0f, -1.0f);
    const float2 w = __ffma2_rn(s, m1, t);                      // t - s
    const float2 d = __fadd2_rn(__ffma2_rn(__ffma2_rn(w, m1, t), m1, s), __ffma2_rn(w, m1, v));
    c = __fadd2_rn(c, d);
    s = t;
  }
  __device__ __forceinline__ void add(const PairSum& o) {
    add(o.s);
    c = __fadd2_rn(c, o.c);
    a += o.a;
  }
  __device__ __forceinline__ PairSum down(int o, bool with_abs) const {  // that of the lane o further
    PairSum r;
    r.s.x = __shfl_down_sync(0xffffffffu, s.x, o);
    r.s.y = __shfl_down_sync(0xffffffffu, s.y, o);
    r.c.x = __shfl_down_sync(0xffffffffu, c.x, o);
    r.c.y = __shfl_down_sync(0xffffffffu, c.y, o);
    if (with_abs) r.a = __shfl_down_sync(0xffffffffu, a, o);
    return r;
  }
};

// coop_eval through the voxel lists: a query per lane, or per 2, 4 ... 32 lanes where
// the queue is short.  CBMC queries (not DETECT) come without an overlap.  Each word of a
// list (four entries) is summed by itself and the words in their order, whatever lanes
// have them: an insertion's bits do not depend on what else its warp works on.  A sum per
// lane and a tree over the lanes, whose order did, took 2 % less (64 boxes x 15,625
// insertions 13.06 ms against 13.39, 250 in one box 350 us against 356); all terms through
// one lane took 13.71 ms and 369 us.
template <bool SMEM, bool COUNT, bool OPT, bool DETECT>
__device__ __noinline__ void coop_eval_list(const CoopBox B, int nq, bool want_qq, QueryAcc& cnt) {
  const CoopHead& H = coop_head();
  const BoxF& f = H.f;
  CoopWarp& W = coop_warp();
  const float4* p32;
  if constexpr (SMEM) p32 = reinterpret_cast<const float4*>(smem + B.off_atoms);
  else p32 = B.p32;
  const int lane = threadIdx.x & 31;
  const int lb = 5 - (32 - __clz(nq - 1));  // log2 of the lanes per query (nq = 1: 5)
  const int qi = lane >> lb, sub = lane & ((1 << lb) - 1);
  const float rv2 = DETECT ? f.rv2 : f.rcb2;
  const float rq2 = DETECT ? f.rq2 : f.rcb2;
  const bool valid = qi < nq;
  const float4 p = W.pos[valid ? qi : 0];
  const int ta = __float_as_int(p.w);
  const float qa = W.q[valid ? qi : 0];
  const bool vdw_on = ta >= 0;
  const bool qq_on = want_qq && f.charge_on && qa != 0.0f;
  const float band = DETECT ? fmaxf(vdw_on ? f.band_v : 0.0f, qq_on ? f.band_q : 0.0f) : 0.0f;
  const float rsel2 = fmaxf(vdw_on ? rv2 : -1.0f, qq_on ? rq2 : -1.0f) + band;
  const float low2q = f.low2 + f.band_low;
  const float rlo = fminf(vdw_on ? rv2 : 3.0e38f, qq_on ? rq2 : 3.0e38f) - band;
  const float2* lrow = H.ljp + (vdw_on ? ta : 0) * kMaxTypes;
  float x = p.x, y = p.y, z = p.z;
  int code = 0, n = 0;
  const uint4* list = B.vlist;
  if (valid && W.st[qi].y != 1) {  // a slot without an atom has no rows
    const uint4 rec = vox_record(f, H.vox[DETECT ? 1 : 0], B.vrec, x, y, z, code);
    list += rec.x;
    n = (int)rec.z;
  }
  // half of the entries lie within the cutoff, so every entry's energy is formed, two
  // at a time on the packed FP32 pipe, and those outside add zero
  PairSum sum;
  bool ov = false;
  if (COUNT && sub == 0) cnt.visited += (unsigned long long)n;
  // with several lanes per query all go through the words of the longest list, one each
  const int most = lb > 0 ? __reduce_max_sync(0xffffffffu, (n + 3) >> 2) : 1;
  for (int g0 = 0; g0 < most; g0 += 1 << lb) {
    PairSum w;
    const int end = lb > 0 ? min(n, 4 * (g0 + (1 << lb))) : n;
    for (int g = g0 + sub; 4 * g < end && !ov; g += 1 << lb) {
      const uint4 E = __ldg(&list[g]);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int left = n - 4 * g - 2 * k;
        if (left <= 0) break;
        const unsigned e0 = k ? E.z : E.x, e1 = left > 1 ? (k ? E.w : E.y) : e0;
        const int j0 = (int)(e0 & kVoxAtomMask), j1 = (int)(e1 & kVoxAtomMask);
        const float4 a0 = p32[j0], a1 = p32[j1];
        const float4 s0 = H.shift[(int)(e0 >> kVoxAtomBits) + code], s1 = H.shift[(int)(e1 >> kVoxAtomBits) + code];
        const float2 m1 = make_float2(-1.0f, -1.0f);
        const float2 dx = __ffma2_rn(make_float2(a0.x, a1.x), m1, __fadd2_rn(make_float2(x, x), make_float2(s0.x, s1.x)));
        const float2 dy = __ffma2_rn(make_float2(a0.y, a1.y), m1, __fadd2_rn(make_float2(y, y), make_float2(s0.y, s1.y)));
        const float2 dz = __ffma2_rn(make_float2(a0.z, a1.z), m1, __fadd2_rn(make_float2(z, z), make_float2(s0.z, s1.z)));
        const float2 r2 = __ffma2_rn(dx, dx, __ffma2_rn(dy, dy, __fmul2_rn(dz, dz)));
        const bool in0 = r2.x <= rsel2, in1 = left > 1 && r2.y <= rsel2;
        if (COUNT) cnt.in_cut += (int)in0 + (int)in1;
        if (DETECT) {
          const float rmin = fminf(r2.x, left > 1 ? r2.y : r2.x);
          if (rmin < low2q) {
            if (rmin < f.low2 - f.band_low) {
              ov = true;  // a certain overlap
            } else {
              if (r2.x < low2q) coop_note(W, W.own[qi], j0, r2.x, 1);
              if (left > 1 && r2.y < low2q) coop_note(W, W.own[qi], j1, r2.y, 1);
            }
          }
          if (in0 && r2.x >= rlo) coop_note(W, W.own[qi], j0, r2.x, 0);
          if (in1 && r2.y >= rlo) coop_note(W, W.own[qi], j1, r2.y, 0);
        }
        if (OPT && f.tab_res > 0) {  // Estimate_MoleculePair_Energy, its charges whatever want_qq says
          const float qic = qa * (float)kCHARGE_FACTOR;
          float2 et = make_float2(0.0f, 0.0f);
          table_pair_f(f.tab_v, f.tab_f2, f.tab_res, f.tab_shift, f.tab_rcs, f.tab_step, f.tab_inv_step, f.ntypes, r2.x,
                       ta, __float_as_int(a0.w), qic, f.charge_on ? B.q32[j0] : 0.0f, et.x);
          if (left > 1)
            table_pair_f(f.tab_v, f.tab_f2, f.tab_res, f.tab_shift, f.tab_rcs, f.tab_step, f.tab_inv_step, f.ntypes, r2.y,
                         ta, __float_as_int(a1.w), qic, f.charge_on ? B.q32[j1] : 0.0f, et.y);
          if (k == 0) w.first(et);
          else w.add(et);
          continue;
        }
        if (vdw_on) {
          const int t0 = __float_as_int(a0.w), t1 = __float_as_int(a1.w);
          const float2 l0 = lrow[max(t0, 0)], l1 = lrow[max(t1, 0)];
          float2 ev = make_float2(lj_pair_f(l0.x, l0.y, r2.x), lj_pair_f(l1.x, l1.y, r2.y));
          if (!(t0 >= 0 && r2.x <= rv2)) ev.x = 0.0f;
          if (!(t1 >= 0 && left > 1 && r2.y <= rv2)) ev.y = 0.0f;
          if (k == 0) w.first(ev);
          else w.add(ev);
          if (DETECT) w.a += fabsf(ev.x) + fabsf(ev.y);
        }
        if (qq_on) {
          float2 eq = make_float2(0.0f, 0.0f);
          if (r2.x <= rq2) eq.x = qq_ewald_inter_f(f.alpha, qa * B.q32[j0], r2.x);
          if (left > 1 && r2.y <= rq2) eq.y = qq_ewald_inter_f(f.alpha, qa * B.q32[j1], r2.y);
          w.add(eq);
          if (DETECT) w.a += fabsf(eq.x) + fabsf(eq.y);
        }
      }
      if (lb == 0) {
        sum.add(w);
        w.a = 0.0f;
        if (!vdw_on) w.first(make_float2(0.0f, 0.0f));  // the next word's first term is a Coulomb one
      }
    }
    if (lb > 0) {  // the lanes' words in their order; those beyond a list's end are zero, which adds exactly
      sum.add(w);
      for (int o = 1; o < min(1 << lb, most - g0); ++o) sum.add(w.down(o, DETECT));
    }
  }
  if (DETECT && ov) W.ov[qi] = 1;
  KahanF e;
  e.s = sum.s.x;
  e.c = sum.c.x;
  e.add(sum.s.y);
  e.c += sum.c.y;
  __syncwarp();
  if (valid && sub == 0) W.pos[qi] = make_float4(e.s, e.c, sum.a, 0.0f);
  __syncwarp();
}

// Energy of the atoms ids[0..nat) (own numbers and positions per lane: r, shifted
// by sx, sy, sz) against the box for every lane that is `on`: added to A, ov set
// on core overlap.  The lanes' first atoms are queried together, then the next
// ones of the lanes without an overlap; with few lanes on, several atoms at once.
template <bool SMEM, bool COUNT, bool OPT, bool DETECT>
__device__ __forceinline__ void coop_atoms(const CoopBox& B, const SpeciesF& S, bool on, const float* r,
                                           const int* ids, int nat, float sx, float sy, float sz, bool want_qq,
                                           QueryAcc& A, bool& ov, QueryAcc& cnt) {
  const BoxF& f = coop_head().f;
  CoopWarp& W = coop_warp();
  const int lane = threadIdx.x & 31;
  const float rc = DETECT ? f.rc_full : f.rc_cbmc;
  const bool lists = coop_head().vox[DETECT ? 1 : 0].on;
  on = on && !ov;
  if (lists && !DETECT && on)  // the trials with a core overlap end here, before their energies
    for (int i = 0; i < nat && !ov; ++i) {
      const int at = ids[i];
      ov = vox_overlap<SMEM, OPT>(B, coop_head(), r[3 * at] + sx, r[3 * at + 1] + sy, r[3 * at + 2] + sz, S.type[at]);
    }
  const int most = __reduce_max_sync(0xffffffffu, on ? nat : 0);
  for (int i0 = 0; i0 < most;) {
    const bool mine = on && !ov && i0 < nat;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (!m) break;
    const int per = min(32 / __popc(m), most - i0);  // atoms of a lane in this batch
    const int s0 = __popc(m & ((1u << lane) - 1u)) * per;
    if (mine)
      for (int a = 0; a < per; ++a) {
        const int s = s0 + a;
        W.ov[s] = 0;
        W.st[s] = make_int2(0, 1);  // no rows
        W.pos[s] = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(-1));
        W.q[s] = 0.0f;
        if (i0 + a < nat) {
          const int at = DETECT ? i0 + a : ids[i0 + a];
          const float x = r[3 * at] + sx, y = r[3 * at + 1] + sy, z = r[3 * at + 2] + sz;
          int lo1 = 0, ny = 0, lo2 = 0, nz = 0;
          bool fy = false, fz = false;
          if (!lists) {
            stencil_f(f, 1, y, rc, lo1, ny, fy);
            stencil_f(f, 2, z, rc, lo2, nz, fz);
          }
          W.pos[s] = make_float4(x, y, z, __int_as_float(S.type[at]));
          W.st[s] = make_int2((lo1 & 0xffff) | (int)((unsigned)lo2 << 16), ny | nz << 8 | (int)fy << 16 | (int)fz << 17);
          W.q[s] = S.q[at];
          W.own[s] = lane | at << 8;
        }
      }
    __syncwarp();
    if (lists) coop_eval_list<SMEM, COUNT, OPT, DETECT>(B, __popc(m) * per, want_qq, cnt);
    else coop_eval<SMEM, COUNT, OPT, DETECT>(B, __popc(m) * per, want_qq, cnt);
    if (mine)
      for (int a = 0; a < per && i0 + a < nat; ++a) {
        const int s = s0 + a;
        if (W.ov[s]) ov = true;
        const float4 v = W.pos[s];
        A.e.add(v.x);
        A.e.c += v.y;
        A.eabs += v.z;
      }
    __syncwarp();
    i0 += per;
  }
}

// Record of one insertion (FP32 parts; the full-cutoff energy as a two-term sum)
struct RecF {
  float dE_intra, dE_frag, ln_pbias, e_abs, first_sum;
  double e_inter;
  int status, selected;
  bool fix;  // the full-cutoff pass met a band: k_widom_fix redoes it
};

// An insertion queued for k_widom_fix: its index in the box and the choices of
// its FP32 growth (growth order, first-fragment trial, dihedral trials)
struct FixEntry {
  int ins;
  unsigned char sel, norder, pad0, pad1;
  unsigned char order[kMaxFrags];
  unsigned char trl[kMaxFrags];
  int nband;                   // band pairs met (more than kMaxBand: the pass is redone)
  BandPair band[kMaxBand];
};

// Get_Aligner_Hanger with reciprocal square roots (row-major): the frame of
// aligner_hanger to a few ulps
__device__ inline void aligner_hanger_rs(double v1[3], double v2[3], double al[9], double hg[9]) {
  const double n1 = rsqrt(v1[0] * v1[0] + v1[1] * v1[1] + v1[2] * v1[2]);
  for (int i = 0; i < 3; ++i) v1[i] = v1[i] * n1;
  const double n2 = rsqrt(v2[0] * v2[0] + v2[1] * v2[1] + v2[2] * v2[2]);
  for (int i = 0; i < 3; ++i) v2[i] = v2[i] * n2;
  double p1[3] = {v1[1] * v2[2] - v1[2] * v2[1], -v1[0] * v2[2] + v1[2] * v2[0], v1[0] * v2[1] - v1[1] * v2[0]};
  const double np1 = rsqrt(p1[0] * p1[0] + p1[1] * p1[1] + p1[2] * p1[2]);
  for (int i = 0; i < 3; ++i) p1[i] = p1[i] * np1;
  double p2[3] = {v1[1] * p1[2] - v1[2] * p1[1], -v1[0] * p1[2] + v1[2] * p1[0], v1[0] * p1[1] - v1[1] * p1[0]};
  const double np2 = rsqrt(p2[0] * p2[0] + p2[1] * p2[1] + p2[2] * p2[2]);
  for (int i = 0; i < 3; ++i) p2[i] = p2[i] * np2;
  for (int i = 0; i < 3; ++i) {
    al[i] = v1[i];
    al[3 + i] = p2[i];
    al[6 + i] = p1[i];
    hg[i * 3 + 0] = v1[i];
    hg[i * 3 + 1] = p2[i];
    hg[i * 3 + 2] = p1[i];
  }
}

// The grown molecule again in FP64 (the arithmetic of run_insertion): the
// same lfsr258 stream from the insertion's first draw, the choices the FP32
// growth made (first fragment and order, selected first-fragment trial, the
// selected dihedral trial of each later fragment) and the FP64 fragment
// library.  Library conformations are taken with the same 32-bit rule as the
// FP32 growth; every geometry uniform is the full FP64 draw, and the angles'
// sines and cosines and the frames' normalisations agree with the FP64 path's
// to a few ulps, so the coordinates are those of the FP64 path for the same
// choices to about 1e-15 A.  Ends with
// Fold_Molecule (orthorhombic branch) as Widom_Insert does before the
// full-cutoff energy.
__device__ inline void replay_molecule_f64(const WidomSpecies& S, const BoxF& f, const double* __restrict__ lib,
                                           Lfsr g, const int* order, int norder, int sel, const int* trls,
                                           double* r) {
  const int n = S.natoms;
  for (int k = 0; k < norder; ++k) g.next_bits();  // first fragment, growth order
  const int f0 = order[0];
  const int nfa = S.frag_natoms[f0];
  unsigned exist = 0u;
  {
    const int conf = index_of(draw_u32(g), S.nconfig[f0]);
    const double* L0 = lib + S.lib_off[f0] + (size_t)conf * nfa * 3;
    for (int i = 0; i < nfa; ++i) {
      const int a = S.frag_atoms[f0][i];
      r[3 * a] = L0[3 * i];
      r[3 * a + 1] = L0[3 * i + 1];
      r[3 * a + 2] = L0[3 * i + 2];
      exist |= 1u << a;
    }
  }
  double com[3];
  get_com(S, r, exist, com);
  {
    // theta = acos(1 - 2u): cos theta = 1 - 2u, sin theta = 2 sqrt(u (1 - u));
    // phi, psi = (1 - 2u) pi through sincospi (the same angles to a few ulps)
    const double ut = g.next();
    const double ct = 1.0 - 2.0 * ut, st = 2.0 * sqrt(ut * (1.0 - ut));
    double sp, cp, ss, cs;
    sincospi(1.0 - 2.0 * g.next(), &sp, &cp);
    sincospi(1.0 - 2.0 * g.next(), &ss, &cs);
    const double r11 = cs * cp - ct * sp * ss, r12 = cs * sp + ct * cp * ss, r13 = ss * st;
    const double r21 = -ss * cp - ct * sp * cs, r22 = -ss * sp + ct * cp * cs, r23 = cs * st;
    const double r31 = st * sp, r32 = -st * cp, r33 = ct;
    for (int i = 0; i < nfa; ++i) {
      const int a = S.frag_atoms[f0][i];
      const double x = r[3 * a] - com[0], y = r[3 * a + 1] - com[1], z = r[3 * a + 2] - com[2];
      r[3 * a] = (r11 * x + r12 * y + r13 * z) + com[0];
      r[3 * a + 1] = (r21 * x + r22 * y + r23 * z) + com[1];
      r[3 * a + 2] = (r31 * x + r32 * y + r33 * z) + com[2];
    }
  }
  for (int k = 0; k < 3 * sel; ++k) g.next_bits();
  const double ax = (0.5 - g.next()) * f.L64[0];
  const double ay = (0.5 - g.next()) * f.L64[1];
  const double az = (0.5 - g.next()) * f.L64[2];
  for (int i = 0; i < nfa; ++i) {
    const int a = S.frag_atoms[f0][i];
    r[3 * a] = r[3 * a] - com[0] + ax;
    r[3 * a + 1] = r[3 * a + 1] - com[1] + ay;
    r[3 * a + 2] = r[3 * a + 2] - com[2] + az;
  }
  for (int k = 0; k < 3 * (S.kappa_ins - sel - 1) + 1; ++k) g.next_bits();  // later trials, selection
  unsigned placed = 1u << f0;
  const int kd = S.kappa_dih;
  for (int oi = 1; oi < norder; ++oi) {
    const int fr = order[oi];
    const int nf = S.frag_natoms[fr];
    g.next_bits();  // the duplicated draw of fragment_growth.f90:1578,1584
    const int cf = index_of(draw_u32(g), S.nconfig[fr]);
    double cfg[3 * kMaxAtoms];
    const double* Lf = lib + S.lib_off[fr] + (size_t)cf * nf * 3;
    for (int j = 0; j < nf; ++j) {
      const int a = S.frag_atoms[fr][j];
      exist |= 1u << a;
      cfg[3 * a] = Lf[3 * j];
      cfg[3 * a + 1] = Lf[3 * j + 1];
      cfg[3 * a + 2] = Lf[3 * j + 2];
    }
    int fc = 0;
    for (int q = 0; q < S.frag_nconnect[fr]; ++q) {
      const int gg = S.frag_connect[fr][q];
      if ((placed >> gg) & 1u) {
        fc = gg;
        break;
      }
    }
    const int anc_i = S.frag_atoms[fr][0], anc_c = S.frag_atoms[fc][0];
    int ids[kMaxAtoms], nid = 0;
    for (int j = 0; j < nf; ++j) {
      const int a = S.frag_atoms[fr][j];
      if (a != anc_i && a != anc_c) ids[nid++] = a;
    }
    const int atom_ifrag = nid > 0 ? ids[0] : S.frag_atoms[fr][nf - 1];
    int atom_fc = S.frag_atoms[fc][S.frag_natoms[fc] - 1];
    for (int j = 0; j < S.frag_natoms[fc]; ++j) {
      const int a = S.frag_atoms[fc][j];
      if (a != anc_i && a != anc_c) {
        atom_fc = a;
        break;
      }
    }
    double v1[3], v2[3], al_i[9], hg_i[9], al_c[9], hg_c[9];
    for (int d = 0; d < 3; ++d) {
      v1[d] = cfg[3 * anc_i + d] - cfg[3 * anc_c + d];
      v2[d] = cfg[3 * atom_ifrag + d] - cfg[3 * anc_c + d];
    }
    aligner_hanger_rs(v1, v2, al_i, hg_i);
    for (int d = 0; d < 3; ++d) {
      v1[d] = r[3 * anc_i + d] - r[3 * anc_c + d];
      v2[d] = r[3 * atom_fc + d] - r[3 * anc_c + d];
    }
    aligner_hanger_rs(v1, v2, al_c, hg_c);
    const double tx = cfg[3 * anc_c], ty = cfg[3 * anc_c + 1], tz = cfg[3 * anc_c + 2];
    // theta0 + trl (2 pi / kappa_dih), theta0 = 2 pi u, in units of pi
    const double t = 2.0 * g.next() + (double)trls[oi] * (2.0 / (double)kd);
    double sth, cth;
    sincospi(t, &sth, &cth);
    for (int j = 0; j < nid; ++j) {
      const int a = ids[j];
      const double x0 = cfg[3 * a] - tx, y0 = cfg[3 * a + 1] - ty, z0 = cfg[3 * a + 2] - tz;
      const double x = x0 * al_i[0] + y0 * al_i[1] + z0 * al_i[2];
      const double y = x0 * al_i[3] + y0 * al_i[4] + z0 * al_i[5];
      const double z = x0 * al_i[6] + y0 * al_i[7] + z0 * al_i[8];
      const double yr = cth * y + sth * z, zr = -sth * y + cth * z;
      r[3 * a] = (x * hg_c[0] + yr * hg_c[1] + zr * hg_c[2]) + r[3 * anc_c];
      r[3 * a + 1] = (x * hg_c[3] + yr * hg_c[4] + zr * hg_c[5]) + r[3 * anc_c + 1];
      r[3 * a + 2] = (x * hg_c[6] + yr * hg_c[7] + zr * hg_c[8]) + r[3 * anc_c + 2];
    }
    g.next_bits();  // trial selection
    placed |= 1u << fr;
  }
  if (S.nfrag > 1) {
    get_com(S, r, exist, com);
    for (int d = 0; d < 3; ++d) {
      const double sh = com[d] > f.hL64[d] ? -f.L64[d] : (com[d] < -f.hL64[d] ? f.L64[d] : 0.0);
      if (sh != 0.0)
        for (int a = 0; a < n; ++a) r[3 * a + d] += sh;
    }
  }
}

// One Widom insertion per lane that is `on`: Widom_Insert (widom_insert.f90:
// 250-447) with the CBMC growth of Build_Molecule (fragment_growth.f90:120-900)
// and Fragment_Placement (:1449-2132), in FP32.  The whole warp calls it; the
// neighbour queries are the warp's, everything else is a lane's own.
template <bool SMEM, bool COUNT, bool OPT>
__device__ RecF run_insertion_f(const WidomSpecies& S, const SpeciesF& SF, const CoopBox& B, bool on,
                                const float* __restrict__ lib, Lfsr rng, double* xyz_out, QueryAcc& cnt,
                                FixEntry& fe) {
  const CoopHead& H = coop_head();
  const BoxF& f = H.f;
  const int n = S.natoms;
  RecF out{0, 0, 0, 0, 0, 0.0, 0, 0, false};
  int sel_first = 0;
  int trls[kMaxFrags];
  float r[3 * kMaxAtoms];
  unsigned exist = 0u;
  float ln_pbias = 0.0f;
  bool cbmc_overlap = !on;

  // Step 1: first fragment and growth order (fragment_growth.f90:218-253, 1317-1446)
  const unsigned v0 = draw_u32(rng);
  int fstart = 0;
  while (fstart < S.nfrag && !((unsigned long long)v0 < SF.cumthr[fstart])) ++fstart;
  if (fstart >= S.nfrag) fstart = S.nfrag - 1;
  float ln_pseq = (float)S.ln_prob_ins[fstart];
  int order[kMaxFrags];
  int norder = 1;
  order[0] = fstart;
  unsigned live = 1u << fstart;
  if (S.nfrag > 1) {
    int hang[kMaxFrags];
    int nh = 0;
    for (int k = 0; k < S.frag_nconnect[fstart]; ++k) {
      const int g = S.frag_connect[fstart][k];
      if (!((live >> g) & 1u)) hang[nh++] = g;
    }
    while (nh > 0) {
      float tot = 0.0f;
      for (int k = 0; k < nh; ++k) tot += (float)(S.frag_natoms[hang[k]] - 2);
      const float uu = unit_of(draw_u32(rng));
      int k = 0;
      float cum = 0.0f;
      for (; k < nh; ++k) {
        cum += (float)(S.frag_natoms[hang[k]] - 2) / tot;
        if (uu < cum) break;
      }
      if (k >= nh) k = nh - 1;
      const int g = hang[k];
      if (nh > 1) ln_pseq += logf((float)(S.frag_natoms[g] - 2) / tot);
      order[norder++] = g;
      live |= 1u << g;
      for (int q = k; q + 1 < nh; ++q) hang[q] = hang[q + 1];
      --nh;
      for (int q = 0; q < S.frag_nconnect[g]; ++q) {
        const int h = S.frag_connect[g][q];
        if (!((live >> h) & 1u) && nh < kMaxFrags) hang[nh++] = h;
      }
    }
  }
  // Step 2: library conformation of the first fragment (:274-304)
  const int nfa = S.frag_natoms[fstart];
  int fa_ids[kMaxAtoms];
  {
    const int nconf = S.nconfig[fstart];
    const int conf = index_of(draw_u32(rng), nconf);
    const float* L0 = lib + S.lib_off[fstart] + (size_t)conf * nfa * 3;
    for (int i = 0; i < nfa; ++i) {
      const int a = S.frag_atoms[fstart][i];
      fa_ids[i] = a;
      r[3 * a] = L0[3 * i];
      r[3 * a + 1] = L0[3 * i + 1];
      r[3 * a + 2] = L0[3 * i + 2];
      exist |= 1u << a;
    }
  }
  // Step 3: random orientation about the COM (rotation_routines.f90:41-137);
  // the fragment is kept relative to its COM until a position is chosen
  float com[3];
  get_com_f(SF, r, exist, com);
  {
    const float theta = acosf(1.0f - 2.0f * unit_of(draw_u32(rng)));
    const float phi = (1.0f - 2.0f * unit_of(draw_u32(rng))) * (float)kPI;
    const float psi = (1.0f - 2.0f * unit_of(draw_u32(rng))) * (float)kPI;
    float st, ct, sp, cp, ss, cs;
    sincosf(theta, &st, &ct);
    sincosf(phi, &sp, &cp);
    sincosf(psi, &ss, &cs);
    const float r11 = cs * cp - ct * sp * ss, r12 = cs * sp + ct * cp * ss, r13 = ss * st;
    const float r21 = -ss * cp - ct * sp * cs, r22 = -ss * sp + ct * cp * cs, r23 = cs * st;
    const float r31 = st * sp, r32 = -st * cp, r33 = ct;
    for (int i = 0; i < nfa; ++i) {
      const int a = fa_ids[i];
      const float x = r[3 * a] - com[0], y = r[3 * a + 1] - com[1], z = r[3 * a + 2] - com[2];
      r[3 * a] = r11 * x + r12 * y + r13 * z;
      r[3 * a + 1] = r21 * x + r22 * y + r23 * z;
      r[3 * a + 2] = r31 * x + r32 * y + r33 * z;
    }
  }
  // Step 4: kappa_ins trial positions of the first fragment (:383-620)
  const int ki = S.kappa_ins;
  const bool cbmc_qq = S.want_qq_cbmc != 0;
  float nrg[kMaxKappa];
  unsigned ovm = 0u;
  const Lfsr replay = rng;
  for (int it = 0; it < ki; ++it) {
    const float ax = centre_of(draw_u32(rng), f.L[0], f.Llo[0]);
    const float ay = centre_of(draw_u32(rng), f.L[1], f.Llo[1]);
    const float az = centre_of(draw_u32(rng), f.L[2], f.Llo[2]);
    QueryAcc A;
    bool ov = false;
    coop_atoms<SMEM, COUNT, OPT, false>(B, SF, on, r, fa_ids, nfa, ax, ay, az, cbmc_qq, A, ov, cnt);
    const float e = A.e.s + A.e.c;
    ov = ov || e >= f.kmaxE;
    nrg[it] = e;
    if (ov) ovm |= 1u << it;
    else out.first_sum += e;
  }
  {
    float lnw = 0.0f;
    const int sel = select_trial_f(ki, nrg, ovm, f.beta, unit_of(draw_u32(rng)), &lnw);
    if (sel < 0 || !on) {
      cbmc_overlap = true;
    } else {
      ln_pbias = ln_pbias - f.beta * nrg[sel] - lnw;
      Lfsr rp = replay;
      float ax = 0, ay = 0, az = 0;
      for (int k = 0; k <= sel; ++k) {
        ax = centre_of(draw_u32(rp), f.L[0], f.Llo[0]);
        ay = centre_of(draw_u32(rp), f.L[1], f.Llo[1]);
        az = centre_of(draw_u32(rp), f.L[2], f.Llo[2]);
      }
      for (int i = 0; i < nfa; ++i) {
        const int a = fa_ids[i];
        r[3 * a] += ax;
        r[3 * a + 1] += ay;
        r[3 * a + 2] += az;
      }
      com[0] = ax;
      com[1] = ay;
      com[2] = az;
      out.selected = sel + 1;
      sel_first = sel;
    }
  }
  // Step 5: Fragment_Placement, kappa_dih dihedral trials per fragment
  if (S.nfrag > 1) {
    float e_prev = cbmc_overlap ? 0.0f : dihedral_f(SF, r, exist);
    unsigned placed = 1u << fstart;
    const int kd = S.kappa_dih;
    float dn[kMaxKappa], dd[kMaxKappa];
    for (int oi = 1; oi < S.nfrag; ++oi) {
      bool grow = !cbmc_overlap && oi < norder;  // this lane places a fragment
      if (!__any_sync(0xffffffffu, grow)) break;
      const int fr = order[grow ? oi : 0];
      const int nf = S.frag_natoms[fr];
      const unsigned grown = exist;
      const int nconf = S.nconfig[fr];
      if (grow) draw_u32(rng);  // the duplicated draw of fragment_growth.f90:1578,1584
      const int cf = grow ? index_of(draw_u32(rng), nconf) : 0;
      float cfg[3 * kMaxAtoms];
      const float* Lf = lib + S.lib_off[fr] + (size_t)cf * nf * 3;
      for (int j = 0; j < nf; ++j) {
        const int a = S.frag_atoms[fr][j];
        if (grow) exist |= 1u << a;
        cfg[3 * a] = Lf[3 * j];
        cfg[3 * a + 1] = Lf[3 * j + 1];
        cfg[3 * a + 2] = Lf[3 * j + 2];
      }
      const unsigned combined = exist;
      int fc = -1;
      for (int q = 0; q < S.frag_nconnect[fr]; ++q) {
        const int g = S.frag_connect[fr][q];
        if ((placed >> g) & 1u) {
          fc = g;
          break;
        }
      }
      if (fc < 0) {  // no placed neighbour: the fragment graph is not connected
        if (grow) cbmc_overlap = true;
        grow = false;
        fc = fr;
      }
      const int anc_i = S.frag_atoms[fr][0], anc_c = S.frag_atoms[fc][0];
      int ids[kMaxAtoms], nid = 0;
      for (int j = 0; j < nf; ++j) {
        const int a = S.frag_atoms[fr][j];
        if (a != anc_i && a != anc_c) ids[nid++] = a;
      }
      int newids[kMaxAtoms], nnew = 0;
      for (int a = 0; a < n; ++a)
        if (((combined & ~grown) >> a) & 1u) newids[nnew++] = a;
      unsigned idmask = 0u;
      for (int j = 0; j < nid; ++j) idmask |= 1u << ids[j];
      const int atom_ifrag = nid > 0 ? ids[0] : S.frag_atoms[fr][nf - 1];
      int atom_fc = S.frag_atoms[fc][S.frag_natoms[fc] - 1];
      for (int j = 0; j < S.frag_natoms[fc]; ++j) {
        const int a = S.frag_atoms[fc][j];
        if (a != anc_i && a != anc_c) {
          atom_fc = a;
          break;
        }
      }
      float v1[3], v2[3], al_i[9], hg_i[9], al_c[9], hg_c[9];
      for (int d = 0; d < 3; ++d) {
        v1[d] = cfg[3 * anc_i + d] - cfg[3 * anc_c + d];
        v2[d] = cfg[3 * atom_ifrag + d] - cfg[3 * anc_c + d];
      }
      aligner_hanger_f(v1, v2, al_i, hg_i);
      for (int d = 0; d < 3; ++d) {
        v1[d] = r[3 * anc_i + d] - r[3 * anc_c + d];
        v2[d] = r[3 * atom_fc + d] - r[3 * anc_c + d];
      }
      aligner_hanger_f(v1, v2, al_c, hg_c);
      const float tx = cfg[3 * anc_c], ty = cfg[3 * anc_c + 1], tz = cfg[3 * anc_c + 2];
      for (int j = 0; j < nid; ++j) {
        const int a = ids[j];
        const float x = cfg[3 * a] - tx, y = cfg[3 * a + 1] - ty, z = cfg[3 * a + 2] - tz;
        cfg[3 * a] = x * al_i[0] + y * al_i[1] + z * al_i[2];
        cfg[3 * a + 1] = x * al_i[3] + y * al_i[4] + z * al_i[5];
        cfg[3 * a + 2] = x * al_i[6] + y * al_i[7] + z * al_i[8];
      }
      const float theta0 = grow ? (float)kTWOPI * unit_of(draw_u32(rng)) : 0.0f;
      const float dtheta = (float)kTWOPI / (float)kd;
      unsigned dov = 0u;
      for (int ii = 0; ii < kd; ++ii) {
        float sth, cth;
        sincosf(theta0 + (float)ii * dtheta, &sth, &cth);
        for (int j = 0; grow && j < nid; ++j) {
          const int a = ids[j];
          const float x = cfg[3 * a], y = cfg[3 * a + 1], z = cfg[3 * a + 2];
          const float yr = cth * y + sth * z, zr = -sth * y + cth * z;
          r[3 * a] = (x * hg_c[0] + yr * hg_c[1] + zr * hg_c[2]) + r[3 * anc_c];
          r[3 * a + 1] = (x * hg_c[3] + yr * hg_c[4] + zr * hg_c[5]) + r[3 * anc_c + 1];
          r[3 * a + 2] = (x * hg_c[6] + yr * hg_c[7] + zr * hg_c[8]) + r[3 * anc_c + 2];
        }
        dn[ii] = 0.0f;
        dd[ii] = 0.0f;
        float niv = 0.0f, niq = 0.0f, noq = 0.0f;
        bool ov = !grow;
        if (grow) exist &= ~idmask;
        for (int j = 0; j < nid && !ov; ++j) {
          exist |= 1u << ids[j];
          float eiv, eiq, eoq;
          ov = atom_intra_f(SF, f, H.ljp, ids[j], r, exist, eiv, eiq, eoq);
          niv += eiv;
          niq += eiq;
          noq += eoq;
        }
        exist = combined;
        QueryAcc A;
        coop_atoms<SMEM, COUNT, OPT, false>(B, SF, grow, r, newids, nnew, 0.0f, 0.0f, 0.0f, cbmc_qq, A, ov, cnt);
        if (!ov) {
          const float ed = dihedral_f(SF, r, exist);
          dd[ii] = ed;
          dn[ii] = ed + niv + niq + (A.e.s + A.e.c) + noq - e_prev;
          ov = dn[ii] >= f.kmaxE;
        }
        if (ov) dov |= 1u << ii;
      }
      float lnw = 0.0f;
      if (!grow) continue;
      const int trl = select_trial_f(kd, dn, dov, f.beta, unit_of(draw_u32(rng)), &lnw);
      if (trl < 0) {
        cbmc_overlap = true;
        continue;
      }
      ln_pbias = ln_pbias - f.beta * dn[trl] - lnw;
      float sth, cth;
      sincosf(theta0 + (float)trl * dtheta, &sth, &cth);
      for (int j = 0; j < nid; ++j) {
        const int a = ids[j];
        const float x = cfg[3 * a], y = cfg[3 * a + 1], z = cfg[3 * a + 2];
        const float yr = cth * y + sth * z, zr = -sth * y + cth * z;
        r[3 * a] = (x * hg_c[0] + yr * hg_c[1] + zr * hg_c[2]) + r[3 * anc_c];
        r[3 * a + 1] = (x * hg_c[3] + yr * hg_c[4] + zr * hg_c[5]) + r[3 * anc_c + 1];
        r[3 * a + 2] = (x * hg_c[6] + yr * hg_c[7] + zr * hg_c[8]) + r[3 * anc_c + 2];
      }
      e_prev = dd[trl];
      trls[oi] = trl;
      placed |= 1u << fr;
    }
    if (!cbmc_overlap) get_com_f(SF, r, exist, com);
  }
  // widom_insert.f90:350-447
  ln_pbias = ln_pbias + ln_pseq + (float)S.ln_kappa_ins + (float)S.ln_kappa_dih_term;
  out.ln_pbias = ln_pbias;
  if (!cbmc_overlap && S.nfrag > 1) {  // Fold_Molecule, orthorhombic branch
    for (int d = 0; d < 3; ++d) {
      const float sh = com[d] > f.hL[d] ? -f.L[d] : (com[d] < -f.hL[d] ? f.L[d] : 0.0f);
      if (sh != 0.0f)
        for (int a = 0; a < n; ++a) r[3 * a + d] += sh;
    }
  }
  CoopWarp& W = coop_warp();
  const int lane = threadIdx.x & 31;
  W.nband[lane] = 0;
  __syncwarp();
  QueryAcc A;
  bool ov = false;
  coop_atoms<SMEM, COUNT, false, true>(B, SF, !cbmc_overlap, r, nullptr, n, 0.0f, 0.0f, 0.0f, true, A, ov, cnt);
  if (cbmc_overlap) {
    out.status = 1;
    return out;
  }
  A.nband = W.nband[lane];
  if (!ov && A.nband > 0) {  // pairs within FP32 rounding of a cutoff: k_widom_fix decides them in FP64
    out.fix = true;
    fe.nband = A.nband;
    for (int q = 0; q < A.nband && A.nband <= kMaxBand; ++q) {  // the notes, by atom and box atom
      const unsigned char ak = W.band_at[lane][q];
      const BandPair bp{W.band_j[lane][q], W.band_r2[lane][q], (unsigned char)(ak & 127), (unsigned char)(ak >> 7), 0, 0};
      int at = q;
      for (; at > 0 && (fe.band[at - 1].atom > bp.atom || (fe.band[at - 1].atom == bp.atom && fe.band[at - 1].j > bp.j)); --at)
        fe.band[at] = fe.band[at - 1];
      fe.band[at] = bp;
    }
    fe.sel = (unsigned char)sel_first;
    fe.norder = (unsigned char)norder;
    for (int k = 0; k < norder; ++k) {
      fe.order[k] = (unsigned char)order[k];
      fe.trl[k] = (unsigned char)(k > 0 ? trls[k] : 0);
    }
  }
  if (ov) {
    out.status = 2;
    return out;
  }
  const IntraF io = molecule_intra_f(SF, f, H.ljp, r);
  if (io.overlap) {
    out.status = 3;
    return out;
  }
  out.e_inter = (A.e.value() + (double)io.pqq);
  out.e_abs = A.eabs;
  out.dE_intra = (io.ivdw + io.iqq) + io.bond + io.angle + io.dih + io.imp;
  out.dE_frag = io.angle;
  out.status = 0;
  if (xyz_out)
    for (int i = 0; i < 3 * n; ++i) xyz_out[i] = (double)r[i];
  return out;
}

// 24 warps per CTA and one CTA per SM (80 registers), fewer where the staged box and
// the warps' scratch do not fit together.  On the 64-box butane batch 16, 24 and 32
// warps take 11.6, 11.5 and 11.3 ms, on 3,000 waters 1.33, 0.81 and 0.85 ms.
constexpr int kF32Threads = 768;
constexpr int kF32Waves = 64;  // at most this many CTAs per SM

// FP32 constants of box b (thread 0), the FP64 edges and squared cutoffs
// and the FP32 error bands of the full-cutoff pass
__device__ inline void widom_boxf(BoxF& sf, const BoxDev& b, double band_scale) {
  double lmax = 0.0;
  for (int d = 0; d < 3; ++d) {
    sf.L[d] = (float)b.L[d];
    sf.Llo[d] = (float)(b.L[d] - (double)sf.L[d]);
    sf.hL[d] = (float)b.hL[d];
    sf.cinv[d] = (float)b.cell_inv[d];
    sf.ch[d] = (float)(b.L[d] / (double)b.nc[d]);
    sf.nc[d] = b.nc[d];
    sf.L64[d] = b.L[d];
    sf.hL64[d] = b.hL[d];
    lmax = fmax(lmax, b.L[d]);
  }
  sf.rcb2 = (float)b.rcut_cbmcsq;
  sf.rv2 = (float)b.rcut_vdwsq;
  sf.rq2 = (float)b.rcut_coulsq;
  sf.low2 = (float)b.rcut_lowsq;
  sf.rc_cbmc = (float)sqrt(b.rcut_cbmcsq);
  sf.rc_full = (float)sqrt(fmax(b.rcut_vdwsq, b.rcut_coulsq));
  sf.beta = (float)b.beta;
  sf.kmaxE = (float)(kMAX_KBT / b.beta);
  sf.alpha = (float)b.alpha;
  sf.charge_on = b.charge_style == CASS_CHARGE_COUL;
  // |r2_32 - r2_64| <= 2 sqrt(3) r delta + the rounding of r^2, where delta
  // bounds the FP32 error of a coordinate difference: the FP32 growth of the
  // test molecule (its centre of mass rounded once, rotations of a few A), the
  // rounding of the stored box atom, of a row's image shift and of the
  // difference -- about 12 half-ulps of the largest coordinate, up to
  // L / 2 + rcut; delta = 5e-7 (L + 20 A) exceeds it by a factor of 2 or more
  const double delta = 5.0e-7 * (lmax + 20.0) * band_scale;
  auto band = [&](double rc2) { return (float)(3.5 * sqrt(rc2) * delta + 1.0e-6 * rc2); };
  sf.rv2d = b.rcut_vdwsq;
  sf.rq2d = b.rcut_coulsq;
  sf.low2d = b.rcut_lowsq;
  sf.band_v = band(b.rcut_vdwsq);
  sf.band_q = band(b.rcut_coulsq);
  sf.band_low = band(b.rcut_lowsq);
}

__device__ inline void widom_ljp(float2* s_ljp, const PairTable& T) {
  for (int i = threadIdx.x; i < kMaxTypes * kMaxTypes; i += blockDim.x) {
    const int a = i / kMaxTypes, c = i % kMaxTypes;
    const bool ok = a < T.ntypes && c < T.ntypes;
    s_ljp[i] = ok ? make_float2(T.epsf[a * T.ntypes + c], T.sig2f[a * T.ntypes + c]) : make_float2(0.f, 0.f);
  }
}

// The voxel lists of grid `which` (0 CBMC, 1 full) of every box of the batch: a thread
// per voxel counts its atoms through the cell lists, the CTA takes the room for its
// voxels' lists in one piece from the cursor, and each thread writes its own (padded
// to whole words).  Lists stand in no fixed order, the entries of each one do.
__global__ void __launch_bounds__(128) k_vox_lists(const BoxDev* boxes, const VoxGrid* vox, int which, const float4* c32,
                                                   const int* cstart, uint4* vrec, unsigned* vlist,
                                                   unsigned long long* cursor) {
  __shared__ int warp_sum[4];
  __shared__ unsigned long long base;
  const int k = blockIdx.y;
  const VoxGrid g = vox[2 * k + which];
  const int nvox = g.nv[0] * g.nv[1] * g.nv[2];
  if (!g.on || (int)(blockIdx.x * blockDim.x) >= nvox) return;
  const BoxDev& b = boxes[k];
  const int v = blockIdx.x * blockDim.x + threadIdx.x;
  const bool live = v < nvox;
  const float R = sqrtf(g.R2);
  const float4* p32 = c32 + b.atom_off;
  const int* cs = cstart + b.cell_off + k;
  float c[3], L[3], hL[3], ci[3], h[3];
  int lo[3], hi[3], nc[3];
  const int iv[3] = {v % g.nv[0], v / g.nv[0] % g.nv[1], v / (g.nv[0] * g.nv[1])};
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    L[d] = b.Lf[d];
    nc[d] = b.nc[d];
    hL[d] = b.hLf[d];
    ci[d] = (float)b.cell_inv[d];
    h[d] = L[d] / (float)nc[d];
    c[d] = ((float)iv[d] + 0.5f) * g.edge[d] - hL[d];
    lo[d] = (int)floorf((c[d] - R + hL[d]) * ci[d] - 1e-3f);
    hi[d] = (int)floorf((c[d] + R + hL[d]) * ci[d] + 1e-3f);
  }
  int total = 0, nnear = 0;
  unsigned* out = nullptr;
  // visits the atoms of the list: fn(atom, code, is near)
  auto visit = [&](auto fn) {
    for (int cz = lo[2]; cz <= hi[2]; ++cz) {
      const int sz = cell_image(cz, nc[2]);
      const float qz = c[2] + (float)sz * L[2];
      const float z0 = (float)cz * h[2] - hL[2];
      const float ez = fmaxf(fmaxf(z0 - c[2], c[2] - (z0 + h[2])) - 1e-3f * h[2], 0.0f);
      for (int cy = lo[1]; cy <= hi[1]; ++cy) {
        const float y0 = (float)cy * h[1] - hL[1];
        const float ey = fmaxf(fmaxf(y0 - c[1], c[1] - (y0 + h[1])) - 1e-3f * h[1], 0.0f);
        const float rem = g.R2 - ez * ez - ey * ey;
        if (rem < 0.0f) continue;
        const int sy = cell_image(cy, nc[1]);
        const float qy = c[1] + (float)sy * L[1];
        const int row = ((cz + sz * nc[2]) * nc[1] + cy + sy * nc[1]) * nc[0];
        const float w = sqrtf(rem);
        const int xlo = (int)floorf((c[0] - w + hL[0]) * ci[0] - 1e-3f);
        const int xhi = (int)floorf((c[0] + w + hL[0]) * ci[0] + 1e-3f);
        for (int cx = xlo; cx <= xhi;) {
          const int sx = cell_image(cx, nc[0]);
          const int wx = cx + sx * nc[0], run = min(xhi - cx, nc[0] - 1 - wx) + 1;
          const float qx = c[0] + (float)sx * L[0];
          const int code = kImage0 + sx + 7 * sy + 49 * sz;
          for (int j = cs[row + wx]; j < cs[row + wx + run]; ++j) {
            const float4 a = p32[j];
            const float dx = qx - a.x, dy = qy - a.y, dz = qz - a.z;
            const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
            if (r2 <= g.R2) fn(j, code, r2 <= g.near2);
          }
          cx += run;
        }
      }
    }
  };
  if (live) visit([&](int, int, bool near) {
    ++total;
    nnear += near ? 1 : 0;
  });
  const int need = live ? (total + 3) & ~3 : 0;
  int incl = need;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int o = 1; o < 32; o <<= 1) {
    const int t = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += t;
  }
  if (lane == 31) warp_sum[w] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int q = 0; q < (int)(blockDim.x >> 5); ++q) t += warp_sum[q];
    base = atomicAdd(cursor, t);
  }
  __syncthreads();
  unsigned long long at = base + (incl - need);
  for (int q = 0; q < w; ++q) at += warp_sum[q];
  if (!live) return;
  vrec[g.off + v] = make_uint4((unsigned)(at >> 2), (unsigned)nnear, (unsigned)total, 0u);
  out = vlist + at;
  int first = 0, last = total - 1;
  visit([&](int j, int code, bool near) { out[near ? first++ : last--] = (unsigned)j | (unsigned)code << kVoxAtomBits; });
}

// per_warp: insertions a warp works on at a time (a power of two up to 32)
template <bool SMEM, bool COUNT, bool OPT>
__global__ void __launch_bounds__(kF32Threads, 1) k_widom_f32(WidomSpecies S, SpeciesF SF, PairTable T, const BoxDev* boxes,
                                                   const int* box_ids, const float4* c32, const float* cq32,
                                                   const int* cstart, const float* __restrict__ libf, long long n_ins,
                                                   uint64_t seed, WRec* rec, signed char* status, double* xyz,
                                                   int want_xyz, CassWidomTrace* trace, FixEntry* fix_q,
                                                   int* fix_n, int per_warp,
                                                   const VoxGrid* vox, const uint4* vrec, const uint4* vlist,
                                                   double band_scale,
                                                   unsigned long long* pair_counts) {
  CoopHead& H = coop_head();
  const int k = blockIdx.y;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    const BoxDev& b = boxes[k];
    widom_boxf(H.f, b, band_scale);
    H.atom_off = b.atom_off;
    H.cell_off = b.cell_off;
    H.natoms = b.natoms;
    H.ec = b.e_inter_constant;
    H.rows_cbmc = stencil_max(H.f, 1, H.f.rc_cbmc) * stencil_max(H.f, 2, H.f.rc_cbmc);
    H.rows_full = stencil_max(H.f, 1, H.f.rc_full) * stencil_max(H.f, 2, H.f.rc_full);
  }
  if (OPT) boxf_options(H.f, boxes[k], T.ntypes);
  widom_ljp(H.ljp, T);
  if (threadIdx.x < 2) H.vox[threadIdx.x] = vox[2 * k + threadIdx.x];
  for (int q = threadIdx.x; q < kImages; q += blockDim.x)
    H.shift[q] = image_valid(q) ? make_float4((float)image_of(q, 0) * (float)boxes[k].L[0],
                                              (float)image_of(q, 1) * (float)boxes[k].L[1],
                                              (float)image_of(q, 2) * (float)boxes[k].L[2], 0.0f)
                                : make_float4(kNoImage, kNoImage, kNoImage, 0.0f);
  __syncthreads();
  const int ncell = H.f.nc[0] * H.f.nc[1] * H.f.nc[2];
  CoopBox B;
  B.vrec = vrec;
  B.vlist = vlist;
  B.q32 = cq32 + H.atom_off;
  B.p32 = c32 + H.atom_off;
  B.cstart = cstart + H.cell_off + k;
  B.off_cells = kCoopHeadBytes + (blockDim.x >> 5) * (unsigned)sizeof(CoopWarp);
  B.off_atoms = B.off_cells + (((ncell + 1) * (unsigned)sizeof(int) + 31) & ~31u);
  if (SMEM) {
    int* cs = reinterpret_cast<int*>(smem + B.off_cells);
    for (int c = threadIdx.x; c <= ncell; c += blockDim.x) cs[c] = B.cstart[c];
    float4* s32 = reinterpret_cast<float4*>(smem + B.off_atoms);
    for (int j = threadIdx.x; j < H.natoms; j += blockDim.x) s32[j] = B.p32[j];
    __syncthreads();
  }
  QueryAcc cnt;
  const long long warps = blockDim.x >> 5;
  for (long long first = (blockIdx.x * warps + (threadIdx.x >> 5)) * per_warp; first < n_ins;
       first += gridDim.x * warps * per_warp) {
    const long long i = first + lane;
    const bool on = lane < per_warp && i < n_ins;
    const size_t g = (size_t)k * n_ins + i;
    const Lfsr rng = seed_stream(seed, box_ids[k], i);
    FixEntry fe;
    const RecF o = run_insertion_f<SMEM, COUNT, OPT>(S, SF, B, on, libf, rng,
                                                     want_xyz && on ? xyz + g * 3 * S.natoms : nullptr, cnt, fe);
    __syncwarp();
    if (!on) continue;
    const double e_int = o.e_inter;
    rec[g] = make_double4_32a((double)o.dE_intra, e_int + H.ec, (double)o.dE_frag, (double)o.ln_pbias);
    status[g] = (signed char)o.status;
    if (trace) {
      CassWidomTrace& t = trace[g];
      t.ln_pbias = (double)o.ln_pbias;
      t.e_first_trial_sum = (double)o.first_sum;
      t.selected_trial = o.selected;
      t.e_inter = o.status == 0 ? e_int : 0.0;
      t.e_inter_abs = o.status == 0 ? (double)o.e_abs : 0.0;
      t.overlap = o.status;
    }
    if (o.fix) {
      fe.ins = (int)i;
      const int slot = atomicAdd(&fix_n[k], 1);  // < n_ins: one entry per insertion at most
      fix_q[(size_t)k * n_ins + slot] = fe;
    }
  }
  if (pair_counts) {
    atomicAdd(&pair_counts[0], cnt.visited);
    atomicAdd(&pair_counts[1], cnt.in_cut);
  }
}

// The insertions whose full-cutoff pass met pairs within a band of FP32
// rounding about a cutoff, one thread each: the selected molecule again in
// FP64 (replay_molecule_f64, the same choices), each band pair's r^2 in FP64
// from it (the FP64 path's r^2 to about 1e-15 A^2), and the FP64 decision:
// an overlap makes the insertion an overlap (status 2); a vdW or Coulomb term
// on the other side of its cutoff than in FP32 is added or removed (its FP32
// pair energy).  An insertion with more than kMaxBand band pairs has its whole
// full-cutoff pass redone from the FP64 coordinates (kQExact).  Record, status
// and trace are corrected in place; the box stays in global memory.
__global__ void __launch_bounds__(128) k_widom_fix(WidomSpecies S, SpeciesF SF, PairTable T, const BoxDev* boxes,
                                                   const int* box_ids, const float4* c32, const float* cq32,
                                                   const double4_32a* c64, const int* cstart,
                                                   const double* __restrict__ lib64, long long n_ins, uint64_t seed,
                                                   const FixEntry* fix_q, const int* fix_n, WRec* rec,
                                                   signed char* status, double* xyz, int want_xyz,
                                                   CassWidomTrace* trace, double band_scale) {
  __shared__ BoxF sf;
  __shared__ float2 s_ljp[kMaxTypes * kMaxTypes];
  __shared__ int s_atom_off, s_cell_off;
  __shared__ double s_ec;
  const int k = blockIdx.y;
  const int nq = fix_n[k];
  if ((long long)blockIdx.x * blockDim.x >= nq) return;  // nothing queued for this block
  if (threadIdx.x == 0) {
    const BoxDev& b = boxes[k];
    widom_boxf(sf, b, band_scale);
    s_atom_off = b.atom_off;
    s_cell_off = b.cell_off;
    s_ec = b.e_inter_constant;
  }
  widom_ljp(s_ljp, T);
  __syncthreads();
  BoxViewF V;
  V.f = &sf;
  V.p32 = c32 + s_atom_off;
  V.p64 = c64 + s_atom_off;
  V.q32 = cq32 + s_atom_off;
  V.cstart = cstart + s_cell_off + k;
  V.ljp = s_ljp;
  const int n = S.natoms;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < nq; e += gridDim.x * blockDim.x) {
    const FixEntry& fe = fix_q[(size_t)k * n_ins + e];
    const size_t g = (size_t)k * n_ins + fe.ins;
    int order[kMaxFrags], trls[kMaxFrags];
    const int norder = fe.norder;
    for (int q = 0; q < norder; ++q) {
      order[q] = fe.order[q];
      trls[q] = fe.trl[q];
    }
    double r64[3 * kMaxAtoms];
    replay_molecule_f64(S, sf, lib64, seed_stream(seed, box_ids[k], fe.ins), order, norder, fe.sel, trls, r64);
    const double lnp = rec[g].w;
    if (fe.nband > kMaxBand) {  // redo the pass from the FP64 coordinates
      float r[3 * kMaxAtoms];
      for (int i = 0; i < 3 * n; ++i) r[i] = (float)r64[i];
      QueryAcc A;
      bool ov = false;
      for (int a = 0; a < n && !ov; ++a)
        ov = query_f_exact(V, A, r[3 * a], r[3 * a + 1], r[3 * a + 2], SF.type[a], SF.q[a], r64 + 3 * a);
      int st = 2;
      double e_int = 0.0, e_abs = 0.0, dE_intra = 0.0, dE_frag = 0.0;
      if (!ov) {
        const IntraF io = molecule_intra_f(SF, sf, V.ljp, r);
        st = io.overlap ? 3 : 0;
        if (st == 0) {
          e_int = A.e.value() + (double)io.pqq;
          e_abs = (double)A.eabs;
          dE_intra = (double)((io.ivdw + io.iqq) + io.bond + io.angle + io.dih + io.imp);
          dE_frag = (double)io.angle;
        }
      }
      rec[g] = make_double4_32a(dE_intra, e_int + s_ec, dE_frag, lnp);
      status[g] = (signed char)st;
      if (trace) {
        trace[g].e_inter = e_int;
        trace[g].e_inter_abs = e_abs;
        trace[g].overlap = st;
      }
      if (want_xyz && st == 0)
        for (int i = 0; i < 3 * n; ++i) xyz[g * 3 * n + i] = r64[i];
      continue;
    }
    bool ov = false;
    double de = 0.0, dab = 0.0;
    for (int q = 0; q < fe.nband; ++q) {
      const BandPair bp = fe.band[q];
      const int a = bp.atom;
      const double d2 = exact_r2(sf, V.p64, bp.j, r64 + 3 * a);
      if (bp.kind == 1) {
        ov = ov || d2 < sf.low2d;
        continue;
      }
      const float4 at = V.p32[bp.j];
      const int ta = SF.type[a], tj = __float_as_int(at.w);
      if (ta >= 0 && tj >= 0 && (bp.r2 <= sf.rv2) != (d2 <= sf.rv2d)) {
        const float2 es = s_ljp[ta * kMaxTypes + tj];
        const double ev = (double)lj_pair_f(es.x, es.y, bp.r2);
        de += d2 <= sf.rv2d ? ev : -ev;
        dab += d2 <= sf.rv2d ? fabs(ev) : -fabs(ev);
      }
      const float qa = SF.q[a];
      if (sf.charge_on && qa != 0.0f && (bp.r2 <= sf.rq2) != (d2 <= sf.rq2d)) {
        const double eq = (double)qq_ewald_inter_f(sf.alpha, qa * V.q32[bp.j], bp.r2);
        de += d2 <= sf.rq2d ? eq : -eq;
        dab += d2 <= sf.rq2d ? fabs(eq) : -fabs(eq);
      }
    }
    if (ov) {
      rec[g] = make_double4_32a(0.0, s_ec, 0.0, lnp);
      status[g] = 2;
      if (trace) {
        trace[g].e_inter = 0.0;
        trace[g].e_inter_abs = 0.0;
        trace[g].overlap = 2;
      }
    } else if (status[g] == 0 && (de != 0.0 || dab != 0.0)) {
      rec[g].y += de;
      if (trace) {
        trace[g].e_inter += de;
        trace[g].e_inter_abs += dab;
      }
    }
  }
}

// FP64 kernel: one insertion per thread through the cell lists
template <bool SMEM>
__global__ void __launch_bounds__(128) k_widom(WidomSpecies S, PairTable T, SpeciesPools P, const BoxDev* boxes,
                                               const int* box_ids, const double4_32a* c64, const int* ctype,
                                               const int* corig, const int* cstart,
                                               const double* __restrict__ lib, long long n_ins,
                                               uint64_t seed, WRec* rec, signed char* status, double* xyz,
                                               int want_xyz, CassWidomTrace* trace, unsigned long long* pair_counts) {
  __shared__ BoxDev sb;
  const int k = blockIdx.y;
  if (threadIdx.x == 0) sb = boxes[k];
  __syncthreads();
  const int na = sb.natoms;
  const int ncell = sb.nc[0] * sb.nc[1] * sb.nc[2];
  BoxView V;
  V.b = &sb;
  V.rc_cbmc = sqrt(sb.rcut_cbmcsq);
  double rfull = sqrt(fmax(sb.rcut_vdwsq, sb.rcut_coulsq));
  if (sb.vdw_sum_style == CASS_VDW_SUM_MINIMUM || sb.vdw_sum_style == CASS_VDW_SUM_CHARMM ||
      (sb.charge_style == CASS_CHARGE_COUL && sb.charge_sum_style == CASS_QQ_MINIMUM))
    rfull = 1e30;
  if (sb.vdw_sum_style == CASS_VDW_SUM_CUT_SWITCH) rfull = fmax(rfull, sqrt(sb.roff_switch_sq));
  V.rc_full = rfull;
  V.corig = corig + sb.atom_off;
  if (SMEM) {
    int* cs = reinterpret_cast<int*>(smem);
    for (int c = threadIdx.x; c <= ncell; c += blockDim.x) cs[c] = cstart[sb.cell_off + k + c];
    size_t off = ((size_t)(ncell + 1) * sizeof(int) + 31) & ~(size_t)31;
    double4_32a* s64 = reinterpret_cast<double4_32a*>(smem + off);
    int* st = reinterpret_cast<int*>(smem + off + (size_t)na * sizeof(double4_32a));
    for (int j = threadIdx.x; j < na; j += blockDim.x) {
      s64[j] = c64[sb.atom_off + j];
      st[j] = ctype[sb.atom_off + j];
    }
    V.p64 = s64;
    V.ptype = st;
    V.cstart = cs;
    __syncthreads();
  } else {
    V.cstart = cstart + sb.cell_off + k;
    V.p64 = c64 + sb.atom_off;
    V.ptype = ctype + sb.atom_off;
  }
  const long long stride = (long long)gridDim.x * blockDim.x;
  PairCount pc;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_ins; i += stride) {
    size_t g = (size_t)k * n_ins + i;
    Lfsr rng = seed_stream(seed, box_ids[k], i);
    WRec rr;
    int st = 0;
    run_insertion(S, P, T, V, lib, rng, rr, st, want_xyz ? xyz + g * 3 * S.natoms : nullptr,
                  trace ? trace + g : nullptr, pc);
    rec[g] = rr;
    status[g] = (signed char)st;
    if (trace) trace[g].overlap = st;
  }
  if (pair_counts) {
    atomicAdd(&pair_counts[0], pc.visited);
    atomicAdd(&pair_counts[1], pc.in_cut);
  }
}

// ---------------------------------------------------------------------------
// Warp-wide queries of the FP64 kernel.
//
// GB300 takes 16 cycles of an SM for a warp's FP64 instruction however many lanes need
// it, so the FP64 work is done for full warps: a query's voxel list is gone through by
// all lanes in FP32 with a margin far above its rounding, the pairs that pass are
// queued, and 32 of them at a time are decided and evaluated in FP64.  (A thread per
// insertion had 8.5 of 32 lanes at work and formed every visited pair in FP64.)
constexpr int kHits64 = 256;  // queued pairs of a warp
constexpr unsigned kHitAtomBits = 17;  // a box on the FP64 lists has fewer than 2^17 atoms
constexpr int kThreads64 = 384;

struct Coop64 {
  double4_32a pos[32];  // query points and charges
  double sum[32], sabs[32];
  double e[kHits64];
  float4 posf[32];
  unsigned hit[kHits64];  // atom | image code << kHitAtomBits | query << 26 | image to be checked << 31
  int type[32], ov[32], first[33];
};
struct Head64 {
  BoxDev b;
  BoxF f;
  VoxGrid vox[2];
  float4 shift[kImages];
  double4_32a shift64[kImages];
  double2 lj[kMaxTypes * kMaxTypes];  // eps, sigma^2
  float pre[2];                       // FP32 bound of r^2 beyond the CBMC and the full cutoffs
  float low_sure, low_pre;            // FP32 r^2 below / above which a pair surely is / is not an overlap
  float edge_lo[3], edge_hi[3];       // |d| about half a box edge: surely this image / surely another
  int wide[2];                        // the cutoffs reach half a box edge: more than one image may be within them
};
__device__ __forceinline__ Head64& head64() { return *reinterpret_cast<Head64*>(smem); }
constexpr unsigned kHead64Bytes = (sizeof(Head64) + 31) & ~31u;
__device__ __forceinline__ Coop64& coop64() { return reinterpret_cast<Coop64*>(smem + kHead64Bytes)[threadIdx.x >> 5]; }

// FP64 separation of query point p and cell-sorted atom a through image code c
__device__ __forceinline__ double sep64(const Head64& H, const double4_32a& p, const double4_32a& a, int c, double d[3]) {
  const double4_32a sh = H.shift64[c];
  d[0] = (p.x - a.x) + sh.x;
  d[1] = (p.y - a.y) + sh.y;
  d[2] = (p.z - a.z) + sh.z;
  return d[0] * d[0] + d[1] * d[1] + d[2] * d[2];
}

// Core overlap of a CBMC query point, decided in FP64 where FP32 cannot tell
template <bool SMEM>
__device__ __forceinline__ bool vox_overlap64(const CoopBox& B, const Head64& H, const double4_32a* c64,
                                              const double4_32a& p) {
  const float4* p32;
  if constexpr (SMEM) p32 = reinterpret_cast<const float4*>(smem + B.off_atoms);
  else p32 = B.p32;
  if (!H.vox[0].on) return false;
  float x = (float)p.x, y = (float)p.y, z = (float)p.z;
  int code;
  const uint4 rec = vox_record(H.f, H.vox[0], B.vrec, x, y, z, code);
  const unsigned* list = reinterpret_cast<const unsigned*>(B.vlist + rec.x);
  bool ov = false;
  for (int t = 0; t < (int)rec.y && !ov; ++t) {
    const unsigned e = __ldg(&list[t]);
    const int j = (int)(e & kVoxAtomMask), c = (int)(e >> kVoxAtomBits) + code;
    const float4 a = p32[j], sh = H.shift[c];
    const float dx = (x + sh.x) - a.x, dy = (y + sh.y) - a.y, dz = (z + sh.z) - a.z;
    const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    if (r2 > H.low_pre) continue;
    double d[3];
    ov = r2 < H.low_sure || sep64(H, p, c64[j], c, d) < H.b.rcut_lowsq;
  }
  return ov;
}

// The energies of the nq queries of the warp's scratch, left in sum (sabs: of |terms|,
// FULL only) and ov (FULL only; CBMC queries come without an overlap)
template <bool SMEM, bool FULL>
__device__ __noinline__ void coop_eval64(const CoopBox B, int nq, bool want_qq, PairCount& pc) {
  const Head64& H = head64();
  const double4_32a* __restrict__ c64 = B.c64;
  const PairTable& T = *B.T;
  const BoxDev& b = H.b;
  Coop64& W = coop64();
  const float4* p32;
  if constexpr (SMEM) p32 = reinterpret_cast<const float4*>(smem + B.off_atoms);
  else p32 = B.p32;
  const int lane = threadIdx.x & 31;
  const VoxGrid& g = H.vox[FULL ? 1 : 0];
  const bool qq_on = want_qq && b.charge_style == CASS_CHARGE_COUL, lj = lj_plain_style(b);
  const bool ewald = b.charge_sum_style == CASS_QQ_EWALD;
  const float pre = H.pre[FULL ? 1 : 0];
  const bool wide = H.wide[FULL ? 1 : 0];
  if (lane < nq) W.sum[lane] = W.sabs[lane] = 0.0;
  int cnt = 0;
  double acc = 0.0, aabs = 0.0;  // FULL: this lane's share of the current query
  // queued pair h in FP64
  auto pair = [&](unsigned h, double& e, double& ea) {
    const int q = (int)(h >> 26) & 31, j = (int)(h & ((1u << kHitAtomBits) - 1u)), c = (int)(h >> kHitAtomBits) & 511;
    const double4_32a p = W.pos[q], a = c64[j];
    double d[3];
    const double r2 = sep64(H, p, a, c, d);
    e = 0.0;
    ea = 0.0;
    if (h >> 31) {  // the image that Minimum_Image_Separation takes, and no other
      const double d0[3] = {p.x - a.x, p.y - a.y, p.z - a.z};
      for (int k = 0; k < 3; ++k)
        if (image_of(c, k) != (d0[k] > b.hL[k] ? -1 : d0[k] < -b.hL[k] ? 1 : 0)) return;
    }
    if (FULL && r2 < b.rcut_lowsq) {
      W.ov[q] = 1;
      return;
    }
    int m = cutoff_mask(b, r2, !FULL);
    if (!qq_on) m &= 1;
    if (m) ++pc.in_cut;
    const int ta = W.type[q], tj = __float_as_int(p32[j].w);
    if ((m & 1) && ta >= 0 && tj >= 0) {
      double ev;
      if (lj) {
        const double2 es = H.lj[ta * kMaxTypes + tj];
        const double s2 = es.y * (1.0 / r2), s6 = s2 * s2 * s2;
        ev = 4.0 * es.x * (s6 * s6 - s6);
      } else {
        ev = vdw_pair(T, b, ta, tj, r2, 1.0);
      }
      e += ev;
      if (FULL) ea += fabs(ev);
    }
    if (m & 2) {
      double eq;
      if (ewald) {
        const double ri = rsqrt(r2);
        eq = p.w * a.w * kCHARGE_FACTOR * ri * erfc_as(b.alpha * (r2 * ri));
      } else {
        eq = qq_pair_inter(b, p.w * a.w, r2);
      }
      e += eq;
      if (FULL) ea += fabs(eq);
    }
  };
  // evaluates the queue; q: the query being listed
  auto flush = [&](int q) {
    __syncwarp();
    for (int t = lane; t < cnt; t += 32) {
      double e, ea;
      pair(W.hit[t], e, ea);
      if (FULL) {
        acc += e;
        aabs += ea;
      } else {
        W.e[t] = e;
      }
    }
    __syncwarp();
    if (!FULL && lane <= q) {  // each query's pairs stand together, in their order
      const int t1 = lane < q ? W.first[lane + 1] : cnt;
      double e = W.sum[lane];
      for (int t = W.first[lane]; t < t1; ++t) e += W.e[t];
      W.sum[lane] = e;
    }
    __syncwarp();
    if (!FULL && lane <= q) W.first[lane] = 0;
    cnt = 0;
    __syncwarp();
  };
  for (int q = 0; q < nq; ++q) {
    if (!FULL && lane == 0) W.first[q] = cnt;
    const float4 p = W.posf[q];
    float x = p.x, y = p.y, z = p.z;
    int code = 0, n = 0;
    const unsigned* list = nullptr;
    if (g.on) {
      const uint4 rec = vox_record(H.f, g, B.vrec, x, y, z, code);
      list = reinterpret_cast<const unsigned*>(B.vlist + rec.x);
      n = (int)rec.z;
    }
    if (lane == 0) pc.visited += (unsigned long long)n;
    for (int t0 = 0; t0 < n; t0 += 32) {
      bool hit = false;
      unsigned h = 0;
      if (t0 + lane < n) {
        const unsigned e = __ldg(&list[t0 + lane]);
        const int j = (int)(e & kVoxAtomMask), c = (int)(e >> kVoxAtomBits) + code;
        const float4 a = p32[j], sh = H.shift[c];
        const float dx = fabsf((x + sh.x) - a.x), dy = fabsf((y + sh.y) - a.y), dz = fabsf((z + sh.z) - a.z);
        hit = !(fmaf(dx, dx, fmaf(dy, dy, dz * dz)) > pre);
        unsigned check = 0u;
        if (wide) {  // a point outside the box may have its pairs through another image than the nearest
          hit = hit && (code != 0 || (dx <= H.edge_hi[0] && dy <= H.edge_hi[1] && dz <= H.edge_hi[2]));
          check = code != 0 || dx > H.edge_lo[0] || dy > H.edge_lo[1] || dz > H.edge_lo[2];
        }
        h = (unsigned)j | (unsigned)c << kHitAtomBits | (unsigned)q << 26 | check << 31;
      }
      const unsigned m = __ballot_sync(0xffffffffu, hit);
      if (hit) W.hit[cnt + __popc(m & ((1u << lane) - 1u))] = h;
      cnt += __popc(m);
      if (cnt > kHits64 - 32) flush(q);
    }
    if (FULL) {
      flush(q);
      for (int o = 16; o > 0; o >>= 1) {
        acc += __shfl_down_sync(0xffffffffu, acc, o);
        aabs += __shfl_down_sync(0xffffffffu, aabs, o);
      }
      if (lane == 0) {
        W.sum[q] = acc;
        W.sabs[q] = aabs;
      }
      acc = aabs = 0.0;
    }
  }
  if (!FULL) flush(nq - 1);
  __syncwarp();
}

// Energy of the atoms ids[0..nat) of every lane that is `on` (all atoms in order where
// ids is NULL) at r, or r - old + cen, against the box: added to e (and eabs), ov set on
// core overlap
template <bool SMEM, bool FULL>
__device__ __forceinline__ void coop_atoms64(const CoopBox& B, const WidomSpecies& S, bool on, const double* r,
                                             const signed char* ids, int nat, const double* old, const double* cen,
                                             bool want_qq, double& e, double* eabs, bool& ov, PairCount& pc) {
  const Head64& H = head64();
  Coop64& W = coop64();
  const int lane = threadIdx.x & 31;
  on = on && !ov;
  auto place = [&](int i) {
    const int a = ids ? ids[i] : i;
    double x = r[3 * a], y = r[3 * a + 1], z = r[3 * a + 2];
    if (old) {
      x = x - old[0] + cen[0];
      y = y - old[1] + cen[1];
      z = z - old[2] + cen[2];
    }
    return make_double4_32a(x, y, z, S.q[a]);
  };
  if (!FULL && on)
    for (int i = 0; i < nat && !ov; ++i) ov = vox_overlap64<SMEM>(B, H, B.c64, place(i));
  const int most = __reduce_max_sync(0xffffffffu, on ? nat : 0);
  for (int i0 = 0; i0 < most;) {
    const bool mine = on && !ov && i0 < nat;
    const unsigned m = __ballot_sync(0xffffffffu, mine);
    if (!m) break;
    const int per = min(32 / __popc(m), most - i0);  // atoms of a lane in this batch
    // the lanes' atoms that exist, packed
    const int cnt = mine ? min(per, nat - i0) : 0;
    int s0 = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(0xffffffffu, s0, o);
      if (lane >= o) s0 += t;
    }
    const int nq = __shfl_sync(0xffffffffu, s0, 31);
    s0 -= cnt;
    for (int k = 0; k < cnt; ++k) {
      const double4_32a p = place(i0 + k);
      W.pos[s0 + k] = p;
      W.posf[s0 + k] = make_float4((float)p.x, (float)p.y, (float)p.z, 0.0f);
      W.type[s0 + k] = S.type[ids ? ids[i0 + k] : i0 + k];
      W.ov[s0 + k] = 0;
    }
    __syncwarp();
    coop_eval64<SMEM, FULL>(B, nq, want_qq, pc);
    for (int k = 0; k < cnt; ++k) {
      if (W.ov[s0 + k]) ov = true;
      e += W.sum[s0 + k];
      if (eabs) *eabs += W.sabs[s0 + k];
    }
    __syncwarp();
    i0 += per;
  }
}

// One Widom insertion per lane that is `on`, as run_insertion in FP64: the queries are
// the warp's, everything else is a lane's own.  The whole warp calls it.
template <bool SMEM>
__device__ void run_insertion_w(const WidomSpecies& S, const SpeciesPools& P, const PairTable& T, const CoopBox& B,
                                bool on, const double* __restrict__ lib, Lfsr rng, WRec& rec, int& status,
                                double* xyz_out, CassWidomTrace* tr, PairCount& pc) {
  const BoxDev& b = head64().b;
  const SpeciesDevHdr& H = P.hdr[S.is0];
  const int n = S.natoms;
  const double beta = b.beta;
  double r[3 * kMaxAtoms];
  unsigned exist = 0u;
  double ln_pbias = 0.0, ln_pseq;
  double first_sum = 0.0;
  int selected = 0;
  bool cbmc_overlap = !on;

  // Step 1: first fragment and growth order (fragment_growth.f90:218-253, 1317-1446)
  double u = rng.next();
  int fstart = 0;
  while (fstart < S.nfrag && !(u < S.cum_prob_ins[fstart])) ++fstart;
  if (fstart >= S.nfrag) fstart = S.nfrag - 1;
  ln_pseq = S.ln_prob_ins[fstart];
  int order[kMaxFrags];
  int norder = 1;
  order[0] = fstart;
  unsigned live = 1u << fstart;
  if (S.nfrag > 1) {
    int hang[kMaxFrags];
    int nh = 0;
    for (int k = 0; k < S.frag_nconnect[fstart]; ++k) {
      int f = S.frag_connect[fstart][k];
      if (!((live >> f) & 1u)) hang[nh++] = f;
    }
    while (nh > 0) {
      double prob[kMaxFrags], cum[kMaxFrags];
      for (int k = 0; k < nh; ++k) {
        prob[k] = (double)(S.frag_natoms[hang[k]] - 2);
        cum[k] = (k == 0 ? 0.0 : cum[k - 1]) + prob[k];
      }
      double tot = cum[nh - 1];
      for (int k = 0; k < nh; ++k) {
        prob[k] = prob[k] / tot;
        cum[k] = cum[k] / tot;
      }
      double uu = rng.next();
      int k = 0;
      while (k < nh && !(uu < cum[k])) ++k;
      if (k >= nh) k = nh - 1;
      int f = hang[k];
      ln_pseq = ln_pseq + log(prob[k]);
      order[norder++] = f;
      live |= 1u << f;
      for (int q = k; q + 1 < nh; ++q) hang[q] = hang[q + 1];
      --nh;
      for (int q = 0; q < S.frag_nconnect[f]; ++q) {
        int g = S.frag_connect[f][q];
        if (!((live >> g) & 1u) && nh < kMaxFrags) hang[nh++] = g;
      }
    }
  }

  // Step 2: library conformation of the first fragment (:274-304)
  const int nfa = S.frag_natoms[fstart];
  {
    int nconf = S.nconfig[fstart];
    int conf = (int)(rng.next() * nconf);
    if (conf >= nconf) conf = nconf - 1;
    const double* L0 = lib + S.lib_off[fstart] + (size_t)conf * nfa * 3;
    for (int i = 0; i < nfa; ++i) {
      int a = S.frag_atoms[fstart][i];
      r[3 * a] = L0[3 * i];
      r[3 * a + 1] = L0[3 * i + 1];
      r[3 * a + 2] = L0[3 * i + 2];
      exist |= 1u << a;
    }
  }

  // Step 3: Get_COM + Rotate_Molecule_Eulerian (rotation_routines.f90:41-137)
  double com[3];
  get_com(S, r, exist, com);
  {
    double theta = acos(1.0 - 2.0 * rng.next());
    double phi = (1.0 - 2.0 * rng.next()) * kPI;
    double psi = (1.0 - 2.0 * rng.next()) * kPI;
    double st, ct, sp, cp, ss, cs;
    sincos(theta, &st, &ct);
    sincos(phi, &sp, &cp);
    sincos(psi, &ss, &cs);
    double r11 = cs * cp - ct * sp * ss, r12 = cs * sp + ct * cp * ss, r13 = ss * st;
    double r21 = -ss * cp - ct * sp * cs, r22 = -ss * sp + ct * cp * cs, r23 = cs * st;
    double r31 = st * sp, r32 = -st * cp, r33 = ct;
    for (int i = 0; i < nfa; ++i) {
      int a = S.frag_atoms[fstart][i];
      double x = r[3 * a] - com[0], y = r[3 * a + 1] - com[1], z = r[3 * a + 2] - com[2];
      r[3 * a] = (r11 * x + r12 * y + r13 * z) + com[0];
      r[3 * a + 1] = (r21 * x + r22 * y + r23 * z) + com[1];
      r[3 * a + 2] = (r31 * x + r32 * y + r33 * z) + com[2];
    }
  }

  // Step 4: kappa_ins trial positions of the first fragment (:383-620)
  const int ki = S.kappa_ins;
  double nrg[kMaxKappa], w[kMaxKappa];
  unsigned ovm = 0u;
  double r0[3 * kMaxAtoms];
  for (int i = 0; i < 3 * n; ++i) r0[i] = r[i];
  const double com_old[3] = {com[0], com[1], com[2]};
  Lfsr replay = rng;
  for (int it = 0; it < ki; ++it) {
    double ax = (0.5 - rng.next()) * b.L[0];
    double ay = (0.5 - rng.next()) * b.L[1];
    double az = (0.5 - rng.next()) * b.L[2];
    double e = 0.0;
    bool ov = false;
    const double cen[3] = {ax, ay, az};
    coop_atoms64<SMEM, false>(B, S, on, r0, S.frag_atoms[fstart], nfa, com_old, cen, S.want_qq_cbmc != 0, e, nullptr, ov,
                              pc);
    nrg[it] = e;
    w[it] = 0.0;
    if (ov) {
      ovm |= 1u << it;
    } else {
      double nk = beta * nrg[it];
      if (nk >= kMAX_KBT) {
        ovm |= 1u << it;
      } else {
        w[it] = exp(-nk);
        first_sum += nrg[it];
      }
    }
    if (it > 0) w[it] = w[it - 1] + w[it];
  }
  int sel = -1;
  if (!on || ovm == ((ki >= 32) ? 0xffffffffu : ((1u << ki) - 1u))) {
    cbmc_overlap = true;
  } else {
    double rn = rng.next() * w[ki - 1];
    int i = 0;
    while (i < ki && !(rn < w[i])) ++i;
    if (i == ki) cbmc_overlap = true;
    else sel = i;
  }
  if (!cbmc_overlap) {
    ln_pbias = ln_pbias - beta * nrg[sel] - log(w[ki - 1]);
    double ax = 0, ay = 0, az = 0;
    for (int k = 0; k <= sel; ++k) {
      ax = (0.5 - replay.next()) * b.L[0];
      ay = (0.5 - replay.next()) * b.L[1];
      az = (0.5 - replay.next()) * b.L[2];
    }
    for (int i = 0; i < nfa; ++i) {
      int a = S.frag_atoms[fstart][i];
      r[3 * a] = r0[3 * a] - com_old[0] + ax;
      r[3 * a + 1] = r0[3 * a + 1] - com_old[1] + ay;
      r[3 * a + 2] = r0[3 * a + 2] - com_old[2] + az;
    }
    selected = sel + 1;
  }

  // Step 5: Fragment_Placement (:1449-2132)
  if (S.nfrag > 1) {
    double e_prev = cbmc_overlap ? 0.0 : dihedral_masked(H, P, r, exist);
    unsigned placed = 1u << fstart;
    const int kd = S.kappa_dih;
    double dn[kMaxKappa], dd[kMaxKappa];
    for (int oi = 1; oi < S.nfrag; ++oi) {
      bool grow = !cbmc_overlap && oi < norder;  // this lane places a fragment
      if (!__any_sync(0xffffffffu, grow)) break;
      const int f = order[grow ? oi : 0];
      const int nf = S.frag_natoms[f];
      unsigned grown = exist;
      int nconf = S.nconfig[f];
      int cf = 0;
      if (grow) {
        rng.next();
        cf = (int)(rng.next() * nconf);  // the duplicated draw of fragment_growth.f90:1578,1584
        if (cf >= nconf) cf = nconf - 1;
      }
      double cfg[3 * kMaxAtoms];
      const double* Lf = lib + S.lib_off[f] + (size_t)cf * nf * 3;
      for (int j = 0; j < nf; ++j) {
        int a = S.frag_atoms[f][j];
        if (grow) exist |= 1u << a;
        cfg[3 * a] = Lf[3 * j];
        cfg[3 * a + 1] = Lf[3 * j + 1];
        cfg[3 * a + 2] = Lf[3 * j + 2];
      }
      const unsigned combined = exist;
      signed char newids[kMaxAtoms];
      int nnew = 0;
      for (int a = 0; a < n; ++a)
        if (((combined & ~grown) >> a) & 1u) newids[nnew++] = (signed char)a;
      int fc = -1;
      for (int q = 0; q < S.frag_nconnect[f]; ++q) {
        int g = S.frag_connect[f][q];
        if ((placed >> g) & 1u) {
          fc = g;
          break;
        }
      }
      if (fc < 0) {  // no placed neighbour: the fragment graph is not connected
        if (grow) cbmc_overlap = true;
        grow = false;
        fc = f;
      }
      const int anc_i = S.frag_atoms[f][0], anc_c = S.frag_atoms[fc][0];
      int ids[kMaxAtoms], nid = 0;
      for (int j = 0; j < nf; ++j) {
        int a = S.frag_atoms[f][j];
        if (a != anc_i && a != anc_c) ids[nid++] = a;
      }
      unsigned idmask = 0u;
      for (int j = 0; j < nid; ++j) idmask |= 1u << ids[j];
      int atom_ifrag = nid > 0 ? ids[0] : S.frag_atoms[f][nf - 1];
      int atom_fc = S.frag_atoms[fc][S.frag_natoms[fc] - 1];
      for (int j = 0; j < S.frag_natoms[fc]; ++j) {
        int a = S.frag_atoms[fc][j];
        if (a != anc_i && a != anc_c) {
          atom_fc = a;
          break;
        }
      }
      double v1[3], v2[3], al_i[9], hg_i[9], al_c[9], hg_c[9];
      for (int d = 0; d < 3; ++d) {
        v1[d] = cfg[3 * anc_i + d] - cfg[3 * anc_c + d];
        v2[d] = cfg[3 * atom_ifrag + d] - cfg[3 * anc_c + d];
      }
      aligner_hanger(v1, v2, al_i, hg_i);
      for (int d = 0; d < 3; ++d) {
        v1[d] = r[3 * anc_i + d] - r[3 * anc_c + d];
        v2[d] = r[3 * atom_fc + d] - r[3 * anc_c + d];
      }
      aligner_hanger(v1, v2, al_c, hg_c);
      const double tx = cfg[3 * anc_c], ty = cfg[3 * anc_c + 1], tz = cfg[3 * anc_c + 2];
      for (int j = 0; j < nf; ++j) {
        int a = S.frag_atoms[f][j];
        double x = cfg[3 * a] - tx, y = cfg[3 * a + 1] - ty, z = cfg[3 * a + 2] - tz;
        cfg[3 * a] = x * al_i[0] + y * al_i[1] + z * al_i[2];
        cfg[3 * a + 1] = x * al_i[3] + y * al_i[4] + z * al_i[5];
        cfg[3 * a + 2] = x * al_i[6] + y * al_i[7] + z * al_i[8];
      }
      const double theta0 = grow ? kTWOPI * rng.next() : 0.0;
      const double dtheta = kTWOPI / (double)kd;
      unsigned dov = 0u;
      double dw[kMaxKappa];
      double theta = theta0;
      for (int ii = 0; ii < kd; ++ii) {
        if (ii > 0) theta = theta + dtheta;
        double sth, cth;
        sincos(theta, &sth, &cth);
        for (int j = 0; grow && j < nid; ++j) {
          int a = ids[j];
          double x = cfg[3 * a], y = cfg[3 * a + 1], z = cfg[3 * a + 2];
          double yr = cth * y + sth * z, zr = -sth * y + cth * z;
          r[3 * a] = (x * hg_c[0] + yr * hg_c[1] + zr * hg_c[2]) + r[3 * anc_c];
          r[3 * a + 1] = (x * hg_c[3] + yr * hg_c[4] + zr * hg_c[5]) + r[3 * anc_c + 1];
          r[3 * a + 2] = (x * hg_c[6] + yr * hg_c[7] + zr * hg_c[8]) + r[3 * anc_c + 2];
        }
        dn[ii] = 0.0;
        dd[ii] = 0.0;
        double niv = 0.0, niq = 0.0, noq = 0.0;
        bool ov = !grow;
        if (grow) exist &= ~idmask;
        for (int j = 0; j < nid && !ov; ++j) {
          exist |= 1u << ids[j];
          double eiv, eiq, eoq;
          if (atom_intra(H, P, b, T, ids[j], r, exist, eiv, eiq, eoq)) {
            ov = true;
            break;
          }
          niv += eiv;
          niq += eiq;
          noq += eoq;
        }
        double einter = 0.0;
        coop_atoms64<SMEM, false>(B, S, grow, r, newids, nnew, nullptr, nullptr, S.want_qq_cbmc != 0, einter, nullptr, ov,
                                  pc);
        exist = combined;
        if (ov) {
          dw[ii] = 0.0;
          dov |= 1u << ii;
        } else {
          double ed = dihedral_masked(H, P, r, exist);
          dd[ii] = ed;
          dn[ii] = ed + niv + niq + einter + noq - e_prev;
          double nk = beta * dn[ii];
          if (nk >= kMAX_KBT) {
            dw[ii] = 0.0;
            dov |= 1u << ii;
          } else {
            dw[ii] = exp(-nk);
          }
        }
        if (ii > 0) dw[ii] = dw[ii - 1] + dw[ii];
      }
      if (!grow) continue;
      if (dov == ((kd >= 32) ? 0xffffffffu : ((1u << kd) - 1u))) {
        cbmc_overlap = true;
        continue;
      }
      double pp = rng.next() * dw[kd - 1];
      int trl = 0;
      while (trl < kd && !(pp < dw[trl])) ++trl;
      if (trl == kd) {
        cbmc_overlap = true;
        continue;
      }
      ln_pbias = ln_pbias - beta * dn[trl] - log(dw[kd - 1]);
      theta = theta0;
      for (int ii = 1; ii <= trl; ++ii) theta = theta + dtheta;
      double sth, cth;
      sincos(theta, &sth, &cth);
      for (int j = 0; j < nid; ++j) {
        int a = ids[j];
        double x = cfg[3 * a], y = cfg[3 * a + 1], z = cfg[3 * a + 2];
        double yr = cth * y + sth * z, zr = -sth * y + cth * z;
        r[3 * a] = (x * hg_c[0] + yr * hg_c[1] + zr * hg_c[2]) + r[3 * anc_c];
        r[3 * a + 1] = (x * hg_c[3] + yr * hg_c[4] + zr * hg_c[5]) + r[3 * anc_c + 1];
        r[3 * a + 2] = (x * hg_c[6] + yr * hg_c[7] + zr * hg_c[8]) + r[3 * anc_c + 2];
      }
      e_prev = dd[trl];
      placed |= 1u << f;
    }
    if (!cbmc_overlap) get_com(S, r, exist, com);
  }

  // widom_insert.f90:350-447
  ln_pbias = ln_pbias + ln_pseq;
  ln_pbias = ln_pbias + S.ln_kappa_ins;
  ln_pbias = ln_pbias + S.ln_kappa_dih_term;
  if (on && tr) {
    tr->ln_pbias = ln_pbias;
    tr->e_first_trial_sum = first_sum;
    tr->selected_trial = selected;
    tr->e_inter = 0.0;
    tr->e_inter_abs = 0.0;
  }
  rec = make_double4_32a(0.0, 0.0, 0.0, ln_pbias);
  if (!cbmc_overlap && S.nfrag > 1) {  // Fold_Molecule, orthorhombic branch
    for (int d = 0; d < 3; ++d) {
      if (com[d] > b.hL[d]) {
        com[d] = com[d] - b.L[d];
        for (int a = 0; a < n; ++a) r[3 * a + d] -= b.L[d];
      } else if (com[d] < -b.hL[d]) {
        com[d] = com[d] + b.L[d];
        for (int a = 0; a < n; ++a) r[3 * a + d] += b.L[d];
      }
    }
  }
  double e_inter = 0.0, e_abs = 0.0;
  bool ov = false;
  coop_atoms64<SMEM, true>(B, S, !cbmc_overlap, r, nullptr, n, nullptr, nullptr, true, e_inter, &e_abs, ov, pc);
  if (cbmc_overlap || ov) {
    status = cbmc_overlap ? 1 : 2;
    return;
  }
  IntraOut io = molecule_intra(P, S.is0, b, T, r);
  if (io.overlap) {
    status = 3;
    return;
  }
  e_inter = e_inter + io.pqq;
  double dE_inter = e_inter + b.e_inter_constant;
  double dE_intra = io.ivdw + io.iqq;
  dE_intra = dE_intra + io.bond + io.angle + io.dih + io.imp;
  rec = make_double4_32a(dE_intra, dE_inter, io.angle, ln_pbias);
  status = 0;
  if (tr) {
    tr->e_inter = e_inter;
    tr->e_inter_abs = e_abs;
  }
  if (xyz_out)
    for (int i = 0; i < 3 * n; ++i) xyz_out[i] = r[i];
}

// FP64 kernel, a lane per insertion and the warp's queries together (the reference's
// arithmetic); per_warp: insertions a warp works on at a time.
// 16 boxes x 1,000 butane insertions: 2.2 ms against 21.4 ms with a thread per
// insertion (k_widom, which remains for what the lists do not serve: CBMC options, the
// molecule-pair cutoff, styles without a cutoff).
template <bool SMEM>
__global__ void __launch_bounds__(kThreads64, 1) k_widom_w(const __grid_constant__ WidomSpecies S,
                                                        const __grid_constant__ PairTable T,
                                                        const __grid_constant__ SpeciesPools P, const BoxDev* boxes,
                                                        const int* box_ids, const double4_32a* c64, const float4* c32,
                                                        const VoxGrid* vox, const uint4* vrec, const uint4* vlist,
                                                        const double* __restrict__ lib, long long n_ins, uint64_t seed,
                                                        int per_warp, WRec* rec, signed char* status, double* xyz,
                                                        int want_xyz, CassWidomTrace* trace,
                                                        unsigned long long* pair_counts) {
  Head64& H = head64();
  const int k = blockIdx.y;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    H.b = boxes[k];
    const BoxDev& b = H.b;
    widom_boxf(H.f, b, 1.0);
    const double lmax = fmax(b.L[0], fmax(b.L[1], b.L[2]));
    auto above = [&](double r2) { return (float)(r2 * (1.0 + 1.0e-4) + 1.0e-3 + 2.0e-6 * lmax * sqrt(r2)); };
    H.pre[0] = above(fmax(b.rcut_cbmcsq, b.rcut_lowsq));
    double full = fmax(fmax(b.rcut_vdwsq, b.rcut_coulsq), b.rcut_lowsq);
    if (b.vdw_sum_style == CASS_VDW_SUM_CUT_SWITCH) full = fmax(full, b.roff_switch_sq);
    H.pre[1] = above(full);
    H.low_pre = above(b.rcut_lowsq);
    H.low_sure = (float)(2.0 * b.rcut_lowsq) - H.low_pre;
    for (int d = 0; d < 3; ++d) {
      H.edge_lo[d] = (float)(b.hL[d] * (1.0 - 1.0e-5));
      H.edge_hi[d] = (float)(b.hL[d] * (1.0 + 1.0e-5));
    }
    const float edge = fminf(H.edge_lo[0], fminf(H.edge_lo[1], H.edge_lo[2]));
    for (int w = 0; w < 2; ++w) H.wide[w] = !(H.pre[w] < edge * edge);
  }
  if (threadIdx.x < 2) H.vox[threadIdx.x] = vox[2 * k + threadIdx.x];
  for (int q = threadIdx.x; q < kImages; q += blockDim.x) {
    const double4_32a v = make_double4_32a(image_of(q, 0) * boxes[k].L[0], image_of(q, 1) * boxes[k].L[1],
                                           image_of(q, 2) * boxes[k].L[2], 0.0);
    H.shift64[q] = v;
    H.shift[q] = image_valid(q) ? make_float4((float)v.x, (float)v.y, (float)v.z, 0.0f)
                                : make_float4(kNoImage, kNoImage, kNoImage, 0.0f);
  }
  for (int i = threadIdx.x; i < kMaxTypes * kMaxTypes; i += blockDim.x) {
    const int a = i / kMaxTypes, c = i % kMaxTypes;
    const bool ok = a < T.ntypes && c < T.ntypes;
    H.lj[i] = ok ? make_double2(T.eps[pidx(a, c, T.ntypes)], T.sig2[pidx(a, c, T.ntypes)]) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  CoopBox B;
  B.vrec = vrec;
  B.vlist = vlist;
  B.p32 = c32 + H.b.atom_off;
  B.c64 = c64 + H.b.atom_off;
  B.T = &T;
  B.off_atoms = kHead64Bytes + (blockDim.x >> 5) * (unsigned)sizeof(Coop64);
  if (SMEM) {
    float4* s32 = reinterpret_cast<float4*>(smem + B.off_atoms);
    for (int j = threadIdx.x; j < H.b.natoms; j += blockDim.x) s32[j] = B.p32[j];
    __syncthreads();
  }
  PairCount pc;
  const long long warps = blockDim.x >> 5;
  for (long long first = (blockIdx.x * warps + (threadIdx.x >> 5)) * per_warp; first < n_ins;
       first += gridDim.x * warps * per_warp) {
    const long long i = first + lane;
    const bool on = lane < per_warp && i < n_ins;
    const size_t g = (size_t)k * n_ins + i;
    WRec rr;
    int st = 0;
    run_insertion_w<SMEM>(S, P, T, B, on, lib, seed_stream(seed, box_ids[k], i), rr, st,
                          want_xyz && on ? xyz + g * 3 * S.natoms : nullptr, trace && on ? trace + g : nullptr, pc);
    __syncwarp();
    if (!on) continue;
    rec[g] = rr;
    status[g] = (signed char)st;
    if (trace) trace[g].overlap = st;
  }
  if (pair_counts) {
    atomicAdd(&pair_counts[0], pc.visited);
    atomicAdd(&pair_counts[1], pc.in_cut);
  }
}

// an Ewald box of the batch (nv = 0: no reciprocal part)
struct RecipBox {
  const double4_32a* kvec;
  const int* kint;  // integers of the k-vectors (NULL: none)
  const double* cos_sum;
  const double* sin_sum;
  int nv, kn[3];  // kn: largest |n| + 1 per dimension
  double h1[3];   // 2 pi / L
};
constexpr int kRecipTab = 1024;
constexpr int kRecipThreads = 128;

// E_recip of each surviving insertion (absolute, as the reference computes it): a CTA per
// insertion, the phases products of tables of the powers of e^{i 2 pi x / L} of its atoms
// (8 FP64 operations per k-vector and atom).  959 k-vectors, 3,000 waters: 0.50 ms with a
// sincos per k-vector and atom, 0.21 ms now.
__global__ void __launch_bounds__(kRecipThreads) k_widom_recip(const RecipBox* boxes, long long n_ins, int na,
                                                               const double* q, const signed char* status,
                                                               const double* xyz, WRec* rec, CassWidomTrace* trace) {
  __shared__ double sh[kRecipThreads / 32];
  __shared__ double2 tab[kRecipTab];
  const long long gi = blockIdx.x;
  const RecipBox R = boxes[gi / n_ins];
  if (R.nv == 0 || status[gi] != 0) return;
  const double* r = xyz + (size_t)gi * 3 * na;
  const int nx = R.kn[0] * na, ny = R.kn[1] * na, nz = R.kn[2] * na;
  const bool tables = R.kint && nx + ny + nz <= kRecipTab;
  if (tables) {
    for (int e = threadIdx.x; e < nx + ny + nz; e += blockDim.x) {
      const int d = e < nx ? 0 : (e < nx + ny ? 1 : 2), f = e - (d > 0 ? nx : 0) - (d > 1 ? ny : 0);
      const int a = f / R.kn[d], k = f - a * R.kn[d];
      double sn, cs;
      sincos((double)k * R.h1[d] * r[3 * a + d], &sn, &cs);
      const double w = d == 0 ? q[a] : 1.0;
      tab[e] = make_double2(w * cs, w * sn);
    }
    __syncthreads();
  }
  double e = 0.0;
  for (int i = threadIdx.x; i < R.nv; i += blockDim.x) {
    const double4_32a h = R.kvec[i];
    double dc = 0.0, ds = 0.0;
    if (tables) {
      const int v = R.kint[i], kx = v & 1023, ky = ((v >> 10) & 1023) - 512, kz = ((v >> 20) & 1023) - 512;
      for (int a = 0; a < na; ++a) {
        const double2 x = tab[a * R.kn[0] + kx], y = tab[nx + a * R.kn[1] + abs(ky)],
                      z = tab[nx + ny + a * R.kn[2] + abs(kz)];
        const double ys = ky < 0 ? -y.y : y.y, zs = kz < 0 ? -z.y : z.y;
        const double c = y.x * z.x - ys * zs, sv = y.x * zs + ys * z.x;
        dc = fma(x.x, c, fma(-x.y, sv, dc));
        ds = fma(x.x, sv, fma(x.y, c, ds));
      }
    } else {
      for (int a = 0; a < na; ++a) {
        double hdotr = h.x * r[3 * a] + h.y * r[3 * a + 1] + h.z * r[3 * a + 2];
        double s, c;
        sincos(hdotr, &s, &c);
        dc += q[a] * c;
        ds += q[a] * s;
      }
    }
    const double c = R.cos_sum[i] + dc, s = R.sin_sum[i] + ds;
    e = e + h.w * (c * c + s * s);
  }
  for (int o = 16; o > 0; o >>= 1) e += __shfl_down_sync(0xffffffffu, e, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = e;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += sh[w];
    double er = t * kCHARGE_FACTOR;
    rec[gi].y = rec[gi].y + er;
    if (trace) trace[gi].e_inter += er;
  }
}

// widom_var and per-box sums; block per box, fixed-order reduction
__global__ void __launch_bounds__(256) k_widom_finalize(const BoxDev* boxes, long long n_ins, const WRec* rec,
                                                        const signed char* status, double* box_sum,
                                                        long long* box_ov, CassWidomTrace* trace) {
  __shared__ double shs[32];
  __shared__ long long sho[32];
  int k = blockIdx.x;
  double beta = boxes[k].beta, ec = boxes[k].e_inter_constant;
  double s = 0.0;
  long long nov = 0;
  for (long long i = threadIdx.x; i < n_ins; i += blockDim.x) {
    size_t g = (size_t)k * n_ins + i;
    double v = 0.0;
    if (status[g] == 0) {
      WRec r = rec[g];
      double dE = r.x + r.y;
      v = exp(-beta * (dE - r.z) - r.w);
      s += v;
    } else {
      ++nov;
    }
    if (trace) {
      trace[g].widom_var = v;
      if (status[g] == 0) trace[g].e_inter = rec[g].y - ec;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    s += __shfl_down_sync(0xffffffffu, s, o);
    nov += __shfl_down_sync(0xffffffffu, nov, o);
  }
  if ((threadIdx.x & 31) == 0) {
    shs[threadIdx.x >> 5] = s;
    sho[threadIdx.x >> 5] = nov;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    long long o = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      t += shs[w];
      o += sho[w];
    }
    box_sum[k] = t;
    box_ov[k] = o;
  }
}

}  // namespace cassgpu

using namespace cassgpu;

namespace {

double lrc_host(cass_ctx* c, const BoxH& B, const std::vector<double>& nb) {
  int nt = c->ntypes;
  double e = 0.0;
  if (B.desc.vdw_style == CASS_VDW_LJ) {
    for (int ia = 0; ia < nt; ++ia) {
      double eij = 0.0;
      for (int ja = 0; ja < nt; ++ja) {
        double eps = c->pt.eps[pidx(ia, ja, nt)], s2 = c->pt.sig2[pidx(ia, ja, nt)];
        double s6 = s2 * s2 * s2, s12 = s6 * s6;
        eij = eij + nb[ja] * 4.0 * eps * (s12 / (9.0 * B.rcut9) - (s6 / (3.0 * B.rcut3)));
      }
      e = e + nb[ia] * eij;
    }
    e = 2.0 * kPI * e / B.dev.volume;
  } else if (B.desc.vdw_style == CASS_VDW_MIE) {
    for (int ia = 0; ia < nt; ++ia) {
      double eij = 0.0;
      for (int ja = 0; ja < nt; ++ja) {
        int k = pidx(ia, ja, nt);
        double sor = std::sqrt(c->pt.sig2[k]) / B.desc.rcut_vdw;
        eij = eij + nb[ja] * c->pt.mie_c[k] * c->pt.eps[k] * std::pow(B.desc.rcut_vdw, 3.0) *
                        ((std::pow(sor, c->pt.mie_n[k]) / (3.0 - c->pt.mie_n[k])) +
                         (std::pow(sor, c->pt.mie_m[k]) / (c->pt.mie_m[k] - 3.0)));
      }
      e = e + nb[ia] * eij;
    }
    e = -2.0 * kPI * e / B.dev.volume;
  }
  return e;
}

}  // namespace

namespace cassgpu {
// FP32 copy of species s for the mixed kernels; false when a table exceeds the
// fixed capacities (the caller then runs the FP64 kernel)
bool species_f(const SpeciesH& s, SpeciesF& F) {
  memset(&F, 0, sizeof(F));
  const int n = s.natoms;
  const int nb = (int)s.bond_kind.size(), na = (int)s.angle_kind.size();
  const int nd = (int)(s.dih_atoms.size() / 4), ni = (int)(s.imp_atoms.size() / 4);
  if (n > kMaxAtoms || nb > kMaxBonded || na > kMaxBonded || nd > kMaxBonded || ni > kMaxBonded) return false;
  F.natoms = n;
  F.nbonds = nb;
  F.nangles = na;
  F.ndih = nd;
  F.nimp = ni;
  for (int a = 0; a < n; ++a) {
    F.q[a] = (float)s.q[a];
    F.mass[a] = (float)s.mass[a];
    F.type[a] = s.type[a];
    for (int b = 0; b < n; ++b) {
      F.vs[a * n + b] = (float)s.vscale[a * n + b];
      F.qs[a * n + b] = (float)s.qscale[a * n + b];
      if (s.bonded[a * n + b]) F.bonded[a] |= 1u << b;
    }
  }
  for (int k = 0; k < nb; ++k) {
    F.bond_atoms[k][0] = (signed char)s.bond_atoms[2 * k];
    F.bond_atoms[k][1] = (signed char)s.bond_atoms[2 * k + 1];
    F.bond_harm[k] = s.bond_kind[k] == CASS_BONDED_HARMONIC;
    F.bond_k[k] = (float)s.bond_param[2 * k];
    F.bond_l0[k] = (float)s.bond_param[2 * k + 1];
  }
  for (int k = 0; k < na; ++k) {
    for (int j = 0; j < 3; ++j) F.angle_atoms[k][j] = (signed char)s.angle_atoms[3 * k + j];
    F.angle_harm[k] = s.angle_kind[k] == CASS_BONDED_HARMONIC;
    F.angle_k[k] = (float)s.angle_param[2 * k];
    F.angle_t0[k] = (float)s.angle_param[2 * k + 1];
  }
  for (int k = 0; k < nd; ++k) {
    for (int j = 0; j < 4; ++j) F.dih_atoms[k][j] = (signed char)s.dih_atoms[4 * k + j];
    for (int j = 0; j < 6; ++j) F.rb[k][j] = (float)s.dih_rb[6 * k + j];
  }
  for (int k = 0; k < ni; ++k) {
    for (int j = 0; j < 4; ++j) F.imp_atoms[k][j] = (signed char)s.imp_atoms[4 * k + j];
    F.imp_k[k] = (float)s.imp_param[2 * k];
    F.imp_p0[k] = (float)s.imp_param[2 * k + 1];
  }
  for (int f = 0; f < s.nfrag; ++f) {
    F.cum_prob_ins[f] = (float)s.cum_prob_ins[f];
    const double c = f == s.nfrag - 1 ? 1.0 : std::min(1.0, s.cum_prob_ins[f]);
    F.cumthr[f] = (unsigned long long)std::floor(c * 4294967296.0);
  }
  return true;
}


// Growth tables of species s (0-based is0) for kernels that build molecules
void fill_growth_species(const SpeciesH& s, int is0, int kappa_ins, int kappa_dih, WidomSpecies& S) {
  memset(&S, 0, sizeof(S));
  S.natoms = s.natoms;
  S.nfrag = s.nfrag;
  S.is0 = is0;
  S.kappa_ins = kappa_ins;
  S.kappa_dih = s.nfrag > 1 ? kappa_dih : 0;
  S.want_qq_cbmc = s.l_coul_cbmc ? 1 : 0;
  S.ln_kappa_ins = std::log((double)kappa_ins);
  S.ln_kappa_dih_term = kappa_dih != 0 ? (double)(s.nfrag - 1) * std::log((double)kappa_dih) : 0.0;
  for (int a = 0; a < s.natoms; ++a) {
    S.mass[a] = s.mass[a];
    S.q[a] = s.q[a];
    S.type[a] = s.type[a];
  }
  for (int f = 0; f < s.nfrag; ++f) {
    S.frag_natoms[f] = (int)s.frag_atoms[f].size();
    for (size_t j = 0; j < s.frag_atoms[f].size(); ++j) S.frag_atoms[f][j] = (signed char)s.frag_atoms[f][j];
    S.frag_nconnect[f] = (int)s.frag_connect[f].size();
    for (size_t j = 0; j < s.frag_connect[f].size(); ++j) S.frag_connect[f][j] = (signed char)s.frag_connect[f][j];
    S.nconfig[f] = s.frag_nconfig[f];
    S.lib_off[f] = s.lib_off[f];
    S.prob_ins[f] = s.prob_ins[f];
    S.cum_prob_ins[f] = s.cum_prob_ins[f];
    S.ln_prob_ins[f] = std::log(s.prob_ins[f]);
  }
}

int ensure_pools(cass_ctx* c);
int pack_box_ext(cass_ctx* c, int ibox);
const std::vector<int>& members_ext(cass_ctx* c, int ibox);
}  // namespace cassgpu

namespace {

// The voxel grid `which` (0 CBMC, 1 full) of box b for queries of radius rc whose core
// overlaps lie within lowsq; room: entries it can need.  False where an
// entry cannot describe the box.
bool vox_grid(const BoxDev& b, int which, double rc, double lowsq, bool f32, VoxGrid& g, double& nvox,
              double& room) {
  memset(&g, 0, sizeof(g));
  if (b.natoms < 1 || b.natoms >= 1 << (f32 ? kVoxAtomBits : kHitAtomBits) || !(rc > 0.0)) return false;
  const double lmax = std::max(b.L[0], std::max(b.L[1], b.L[2])), lmin = std::min(b.L[0], std::min(b.L[1], b.L[2]));
  // a fraction of the radius; in a dilute box no more than kVoxPerAtom voxels an atom
  const double edge = std::max(rc / (which ? kVoxPerCutoffFull : kVoxPerCutoffCbmc),
                               std::min(std::cbrt(b.volume / (kVoxPerAtom * b.natoms)), 0.25 * lmin));
  double diag2 = 0.0, most = 1.0;
  nvox = 1.0;
  for (int d = 0; d < 3; ++d) {
    g.nv[d] = (int)std::min(1024.0, std::ceil(b.L[d] / edge));
    g.inv[d] = (float)(g.nv[d] / b.L[d]);
    g.edge[d] = (float)(b.L[d] / g.nv[d]);
    diag2 += (double)g.edge[d] * g.edge[d];
    nvox *= g.nv[d];
  }
  // half a diagonal, with a margin above the FP32 rounding of the coordinates
  const double half = 0.5 * std::sqrt(diag2) + 2.0e-3 + 4.0e-6 * lmax, R = rc + half;
  for (int d = 0; d < 3; ++d) most *= 2.0 * (R + half) / g.edge[d] + 1.0;
  // entries of an atom: at most the voxels in the sphere of R and another half diagonal
  const double per_atom = std::min(most, 4.18879021 * std::pow(R + half, 3.0) * nvox / b.volume);
  room = b.natoms * per_atom + 3.0 * nvox;
  g.R2 = (float)(R * R);
  const double near = std::sqrt(lowsq) + half;
  g.near2 = (float)(near * near);
  // images of the neighbouring boxes only; a list of 2e4 atoms is no neighbour list
  return R < 0.95 * lmin && nvox <= 1.0e8 && 4.18879021 * R * R * R * b.natoms / b.volume <= 2.0e4;
}

// Cells of a box in dimension d for the warp-wide kernels, or the thread-per-insertion one
int widom_cells(const cass_ctx* c, const BoxH& B, int d, bool warp_wide) {
  const double cpc = c->widom_cells > 0.0 ? c->widom_cells : (warp_wide ? kCellsPerCutoffMixed : kCellsPerCutoffFP64);
  double rcell = (B.desc.rcut_cbmc > 0.0 ? B.desc.rcut_cbmc : B.rcut_max) / cpc;
  // an atom a cell at least, for what goes through the cells of a dilute box
  if (warp_wide && !(c->widom_cells > 0.0)) rcell = std::max(rcell, std::cbrt(B.dev.volume / std::max(1, B.npacked)));
  return std::min(std::max(1, (int)std::floor(B.dev.L[d] / rcell)), 64);
}

double full_radius(const BoxDev& b) {
  double r2 = std::max(b.rcut_vdwsq, b.rcut_coulsq);
  if (b.vdw_sum_style == CASS_VDW_SUM_CUT_SWITCH) r2 = std::max(r2, b.roff_switch_sq);
  return std::sqrt(std::max(r2, b.rcut_lowsq));
}

// The lists of a box (g[w].on) and the device memory they may take.  FP64: both radii or
// none.  Mixed: each where a query's stencil never spans the box (the cell search then
// sees every pair through one image shift, as an entry does) and the insertions' queries
// are worth it: a list costs about as much as the cell search of a query, and 32 of an
// insertion's queries (4 full-cutoff ones) use them.  A matter of the box and of n_ins
// alone, so that an insertion does not depend on the other boxes of its call.
struct BoxLists {
  VoxGrid g[2];
  double nvox[2] = {0.0, 0.0}, room[2] = {0.0, 0.0};
  double bytes() const { return (room[0] + room[1]) * sizeof(unsigned) + (nvox[0] + nvox[1]) * sizeof(uint4); }
};
BoxLists box_lists(cass_ctx* c, const BoxH& B, bool f32, int64_t n_ins) {
  BoxLists P;
  memset(P.g, 0, sizeof(P.g));
  BoxDev b = B.dev;
  b.natoms = B.npacked;
  const double rfull2 = std::max(b.rcut_vdwsq, b.rcut_coulsq);
  // the mixed full-cutoff pass also looks at the pairs of the bands (widom_boxf) outside its cutoffs
  const double band = 3.5 * std::sqrt(rfull2) * 5.0e-7 * (std::max(b.L[0], std::max(b.L[1], b.L[2])) + 20.0) *
                          c->widom_band + 1.0e-6 * rfull2;
  const double rcs[2] = {std::sqrt(b.rcut_cbmcsq), f32 ? std::sqrt(rfull2 + band) : full_radius(b)};
  const bool opt = c->cbmc_opt.energy_table_res > 0 || c->cbmc_opt.sector_overlap;
  for (int w = 0; w < 2; ++w) {
    // check_overlap of the CBMC options reaches to r_min
    const double lowsq = opt && w == 0 ? std::max(b.rcut_lowsq, c->rminsq_most) : b.rcut_lowsq;
    VoxGrid g;
    double nvox, room;
    if (!vox_grid(b, w, rcs[w], lowsq, f32, g, nvox, room)) continue;
    if (f32) {
      bool open = (double)n_ins * (w ? 2.0 : 32.0) >= nvox;
      for (int d = 0; d < 3; ++d) {
        const int nc = widom_cells(c, B, d, true);
        open = open && std::floor(2.0 * rcs[w] * ((double)nc / b.L[d]) + 8.0e-3) + 2.0 < nc;
      }
      if (!open) continue;
    }
    if (P.bytes() + room * sizeof(unsigned) + nvox * sizeof(uint4) > kVoxMaxBytes) continue;
    P.g[w] = g;
    P.g[w].on = 1;
    P.nvox[w] = nvox;
    P.room[w] = room;
  }
  if (!f32 && !(P.g[0].on && P.g[1].on)) P = BoxLists(), memset(P.g, 0, sizeof(P.g));
  return P;
}

// True where the FP64 insertions into a box run on the voxel lists (k_widom_w): every
// style has a cutoff, no CBMC option and no molecule-pair cutoff asks for more than the
// atoms within it, and the box can be listed
bool lists64(cass_ctx* c, const BoxH& B) {
  const CassBoxDesc& d = B.desc;
  if (c->cbmc_opt.energy_table_res > 0 || c->cbmc_opt.sector_overlap || B.comcut ||
      (d.vdw_style != CASS_VDW_NONE &&
       (d.vdw_sum_style == CASS_VDW_SUM_MINIMUM || d.vdw_sum_style == CASS_VDW_SUM_CHARMM)) ||
      (d.charge_style == CASS_CHARGE_COUL && d.charge_sum_style == CASS_QQ_MINIMUM))
    return false;
  return B.npacked == 0 || (B.dev.rcut_cbmcsq >= B.dev.rcut_lowsq && box_lists(c, B, false, 1).g[0].on);
}

bool lists64(cass_ctx* c, int nboxes, const int32_t* iboxes) {
  for (int k = 0; k < nboxes; ++k)
    if (!lists64(c, c->box[iboxes[k] - 1])) return false;
  return true;
}

// True where the mixed kernel serves the call: LJ cut / cut_tail with no charges or Ewald
bool mixed_f32(cass_ctx* c, const SpeciesH& s, int nboxes, const int32_t* iboxes, SpeciesF& SF) {
  if (c->precision != CASS_PREC_MIXED || c->pt.ntypes > kMaxTypes) return false;
  for (int k = 0; k < nboxes; ++k) {
    const CassBoxDesc& d = c->box[iboxes[k] - 1].desc;
    if (d.vdw_style != CASS_VDW_LJ ||
        (d.vdw_sum_style != CASS_VDW_SUM_CUT && d.vdw_sum_style != CASS_VDW_SUM_CUT_TAIL) ||
        (d.charge_style != CASS_CHARGE_NONE && d.charge_sum_style != CASS_QQ_EWALD))
      return false;
  }
  return species_f(s, SF);
}

}  // namespace

static int widom_insert_impl(cass_ctx* c, int32_t is1, int32_t nboxes, const int32_t* iboxes, int64_t n_ins,
                                 int32_t kappa_ins, int32_t kappa_dih, uint64_t seed, CassWidomResult* out,
                                 CassWidomTrace* trace) {
  if (!c || is1 < 1 || is1 > c->nspecies || nboxes < 1 || !iboxes || !out || n_ins < 0)
    return set_error(CASS_EINVAL, "bad widom arguments");
  if (kappa_ins < 1 || kappa_ins > kMaxKappa) return set_error(CASS_EINVAL, "kappa_ins must be in 1..32");
  const SpeciesH& s = c->sp[is1 - 1];
  if (!s.defined) return set_error(CASS_ESTATE, "species not defined");
  if (s.nfrag < 1) return set_error(CASS_EINVAL, "species has no CBMC fragments");
  if (s.nfrag > 1 && (kappa_dih < 1 || kappa_dih > kMaxKappa)) return set_error(CASS_EINVAL, "kappa_dih must be in 1..32");
  if (s.natoms > kMaxAtoms) return set_error(CASS_ECAPACITY, "test species has more than 16 atoms");
  if (s.nfrag > kMaxFrags) return set_error(CASS_ECAPACITY, "test species has more than 8 fragments");
  for (int f = 0; f < s.nfrag; ++f) {
    if (s.frag_nconfig[f] < 1) return set_error(CASS_EINVAL, "fragment library is empty");
    if (s.frag_connect[f].size() > (size_t)kMaxFrags) return set_error(CASS_ECAPACITY, "too many fragment connections");
  }
  if (!c->pt_set) return set_error(CASS_ESTATE, "nonbond table not set");
  for (int k = 0; k < nboxes; ++k) {
    int ib = iboxes[k] - 1;
    if (ib < 0 || ib >= c->nboxes) return set_error(CASS_EINVAL, "box index out of range");
    if (!c->box[ib].energy_valid && !c->box[ib].frame_ready)
      return set_error(CASS_ESTATE, "system energy of box not computed");
  }
  int rc;
  CASS_CUDA(cudaSetDevice(c->device));
  if ((rc = ensure_pools(c))) return rc;
  if ((rc = ensure_cbmc(c))) return rc;
  const int is0 = is1 - 1;

  WidomSpecies S;
  fill_growth_species(s, is0, kappa_ins, kappa_dih, S);

  // per-box constants and cell grids
  std::vector<BoxDev> bd(nboxes);
  std::vector<BoxSrc> src(nboxes);
  std::vector<char> has_ew(nboxes, 0);
  int atom_off = 0, cell_off = 0, max_na = 0;
  size_t max_smem32 = 0, max_smem64 = 0;
  bool any_recip = false;
  for (int k = 0; k < nboxes; ++k)
    if ((rc = pack_box_ext(c, iboxes[k] - 1))) return rc;
  SpeciesF SF;
  const bool f32 = mixed_f32(c, s, nboxes, iboxes, SF);
  const bool warp64 = !f32 && lists64(c, nboxes, iboxes);
  for (int k = 0; k < nboxes; ++k) {
    int ib = iboxes[k] - 1;
    BoxH& B = c->box[ib];
    BoxDev v = B.dev;
    int ncell = 1;
    for (int d = 0; d < 3; ++d) {
      v.nc[d] = widom_cells(c, B, d, f32 || warp64);
      v.cell_inv[d] = (double)v.nc[d] / v.L[d];
      ncell *= v.nc[d];
    }
    v.atom_off = atom_off;
    v.natoms = B.npacked;
    v.cell_off = cell_off;
    v.mcom = B.comcut ? B.d_com.as<double4_32a>() : nullptr;  // built with the packed arrays
    v.rcut_max = B.rcut_max;
    // Widom_Insert set-up (widom_insert.f90:201-245)
    const std::vector<int>& mem = members_ext(c, ib);
    int nmols = 1;
    for (int slot : mem)
      if (c->slot_sp[slot] == is0) ++nmols;
    v.prefactor = v.volume / (double)nmols;
    double lrc_diff = 0.0;
    if (B.desc.vdw_sum_style == CASS_VDW_SUM_CUT_TAIL) {
      std::vector<double> nb(c->ntypes, 0.0);
      for (int slot : mem) {
        const SpeciesH& t = c->sp[c->slot_sp[slot]];
        for (int a = 0; a < t.natoms; ++a)
          if (t.type[a] >= 0) nb[t.type[a]] += 1.0;
      }
      for (int a = 0; a < s.natoms; ++a)
        if (s.type[a] >= 0) nb[s.type[a]] += 1.0;
      lrc_diff = lrc_host(c, B, nb) - B.energy.lrc;
    }
    double e_self = 0.0, e_recip_in = 0.0;
    if (B.desc.charge_style == CASS_CHARGE_COUL && s.has_charge) {
      double qq = 0.0;
      for (int a = 0; a < s.natoms; ++a) qq += s.q[a] * s.q[a];
      if (B.desc.charge_sum_style == CASS_QQ_EWALD) e_self = -qq * kCHARGE_FACTOR * v.alpha / kROOTPI;
      else if (B.desc.charge_sum_style == CASS_QQ_DSF)
        e_self = -qq * (v.alpha_dsf / kROOTPI + v.dsf_factor1 / 2.0) * kCHARGE_FACTOR;
      e_recip_in = B.energy.reciprocal;
    }
    v.e_inter_constant = lrc_diff + e_self - e_recip_in;
    if (B.desc.charge_style == CASS_CHARGE_COUL && B.desc.charge_sum_style == CASS_QQ_EWALD && s.has_charge &&
        B.nvecs > 0) {
      has_ew[k] = 1;
      any_recip = true;
    }
    bd[k] = v;
    src[k].p64 = B.d_p64.as<double4_32a>();
    src[k].p32 = B.d_p32.as<float4>();
    src[k].meta = B.d_meta.as<int4>();
    const size_t sm_cells = ((size_t)(ncell + 1) * sizeof(int) + 31) & ~(size_t)31;
    max_smem32 = std::max(max_smem32, sm_cells + (size_t)B.npacked * sizeof(float4));  // and the warps' scratch
    max_smem64 = std::max(max_smem64, sm_cells + (size_t)B.npacked * (sizeof(double4_32a) + sizeof(int)));
    max_na = std::max(max_na, B.npacked);
    atom_off += B.npacked;
    cell_off += ncell;
  }
  const int total_atoms = std::max(1, atom_off), total_cells = cell_off;
  // device buffers
  DevBuf& dbox = c->d_boxdev;
  if ((rc = dbox.reserve(nboxes * sizeof(BoxDev) + nboxes * sizeof(BoxSrc) + nboxes * sizeof(int) + 64))) return rc;
  BoxDev* d_bd = dbox.as<BoxDev>();
  BoxSrc* d_src = reinterpret_cast<BoxSrc*>(d_bd + nboxes);
  int* d_ids = reinterpret_cast<int*>(d_src + nboxes);
  if ((rc = c->d_c64.reserve((size_t)total_atoms * sizeof(double4_32a)))) return rc;
  if ((rc = c->d_c32.reserve((size_t)total_atoms * sizeof(float4) + (size_t)total_atoms * 2 * sizeof(int)))) return rc;
  if ((rc = c->d_cq32.reserve((size_t)total_atoms * sizeof(float)))) return rc;
  if ((rc = c->d_cell_start.reserve(((size_t)total_cells + nboxes) * sizeof(int)))) return rc;
  if ((rc = c->d_cell_count.reserve(((size_t)total_cells * 2 + 64) * sizeof(int)))) return rc;
  if ((rc = c->d_cell_of.reserve((size_t)total_atoms * 2 * sizeof(int)))) return rc;
  float4* d_c32 = c->d_c32.as<float4>();
  int* d_ctype = reinterpret_cast<int*>(d_c32 + total_atoms);
  int* d_corig = d_ctype + total_atoms;
  int* d_count = c->d_cell_count.as<int>();
  int* d_fill = d_count + total_cells;
  CASS_CUDA(h2d(c, d_bd, bd.data(), nboxes * sizeof(BoxDev)));
  CASS_CUDA(h2d(c, d_src, src.data(), nboxes * sizeof(BoxSrc)));
  CASS_CUDA(h2d(c, d_ids, iboxes, nboxes * sizeof(int)));
  CASS_CUDA(cudaEventRecord(c->ev[0], c->stream));
  CASS_CUDA(cudaMemsetAsync(d_count, 0, (size_t)std::max(1, total_cells) * sizeof(int), c->stream));
  // K7
  if (max_na > 0) {
    dim3 g((max_na + 255) / 256, nboxes);
    k_cell_count<<<g, 256, 0, c->stream>>>(d_src, d_bd, c->d_cell_of.as<int>(), d_count);
    k_cell_scan<<<nboxes, 1024, 0, c->stream>>>(d_bd, d_count, c->d_cell_start.as<int>(), d_fill);
    int* d_cell_of = c->d_cell_of.as<int>();
    k_cell_scatter<<<g, 256, 0, c->stream>>>(d_bd, d_cell_of, c->d_cell_start.as<int>(), d_fill, d_cell_of + total_atoms);
    k_cell_place<<<g, 256, 0, c->stream>>>(d_src, d_bd, d_cell_of, c->d_cell_start.as<int>(), d_cell_of + total_atoms,
                                           c->d_c64.as<double4_32a>(), d_c32, d_ctype, c->d_cq32.as<float>(), d_corig);
  } else {
    k_cell_scan<<<nboxes, 1024, 0, c->stream>>>(d_bd, d_count, c->d_cell_start.as<int>(), d_fill);
  }
  CASS_CUDA(cudaGetLastError());
  count_launch(c, max_na > 0 ? 4 : 1);
  // per-insertion records
  size_t nrec = (size_t)nboxes * (size_t)std::max<int64_t>(1, n_ins);
  DevBuf& drec = c->d_widom_out;
  if ((rc = drec.reserve(nrec * (sizeof(WRec) + 1) + 64))) return rc;
  WRec* d_rec = drec.as<WRec>();
  signed char* d_status = reinterpret_cast<signed char*>(d_rec + nrec);
  double* d_xyz = nullptr;
  if (any_recip) {
    if ((rc = c->d_widom_xyz.reserve(nrec * 3 * s.natoms * sizeof(double) + s.natoms * sizeof(double)))) return rc;
    d_xyz = c->d_widom_xyz.as<double>();
  }
  CassWidomTrace* d_trace = nullptr;
  if (trace) {
    if ((rc = c->d_trace.reserve(nrec * sizeof(CassWidomTrace)))) return rc;
    d_trace = c->d_trace.as<CassWidomTrace>();
  }
  if ((rc = c->d_box_sums.reserve((size_t)nboxes * (sizeof(double) + sizeof(long long)) + 2 * sizeof(long long))))
    return rc;
  double* d_bsum = c->d_box_sums.as<double>();
  long long* d_bov = reinterpret_cast<long long*>(d_bsum + nboxes);
  unsigned long long* d_pairs = c->count_pairs ? reinterpret_cast<unsigned long long*>(d_bov + nboxes) : nullptr;
  if (d_pairs) CASS_CUDA(cudaMemsetAsync(d_pairs, 0, 2 * sizeof(unsigned long long), c->stream));
  // K8 launch shape: 128-thread CTAs, enough CTAs per box to fill every SM;
  // the box is staged in shared memory when it fits
  const size_t max_smem = max_smem64;
  const bool use_smem = max_smem <= (size_t)200 * 1024;
  int dev_sms = 0;
  CASS_CUDA(cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, c->device));
  const int threads = 128;
  auto launch = [&](auto kern) -> int {
    if (use_smem) CASS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)max_smem));
    int per_sm = 1;
    CASS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, use_smem ? max_smem : 0));
    per_sm = std::max(per_sm, 1);
    long long want = ((long long)dev_sms * per_sm * 2 + nboxes - 1) / nboxes;
    long long need = (n_ins + threads - 1) / threads;
    int chunks = (int)std::max<long long>(1, std::min(want, need));
    dim3 g(chunks, nboxes);
    c->stats.widom_grid_x = chunks;
    c->stats.widom_grid_y = nboxes;
    c->stats.widom_block = threads;
    c->stats.widom_smem_bytes = use_smem ? (int)max_smem : 0;
    CASS_CUDA(cudaEventRecord(c->ev[1], c->stream));
    kern<<<g, threads, use_smem ? max_smem : 0, c->stream>>>(
        S, c->pt, c->pools, d_bd, d_ids, c->d_c64.as<double4_32a>(), d_ctype, d_corig, c->d_cell_start.as<int>(),
        s.d_library.as<double>(), (long long)n_ins, seed, d_rec, d_status, d_xyz, any_recip ? 1 : 0, d_trace, d_pairs);
    CASS_CUDA(cudaGetLastError());
    CASS_CUDA(cudaEventRecord(c->ev[2], c->stream));
    count_launch(c);
    return CASS_OK;
  };
  // FP32 kernel of the mixed path, then the FP64 fix-up of the insertions it
  // queued (both inside the kernel timing)
  int* d_fixn = nullptr;
  FixEntry* d_fixq = nullptr;
  // Voxel lists per box and radius
  std::vector<VoxGrid> vox(2 * nboxes);
  size_t vox_records = 0;
  double vox_entries = 0.0;
  int vox_most[2] = {0, 0};
  memset(vox.data(), 0, vox.size() * sizeof(VoxGrid));
  if ((f32 || warp64) && n_ins > 0)
    for (int k = 0; k < nboxes; ++k) {
      const BoxLists P = box_lists(c, c->box[iboxes[k] - 1], f32, n_ins);
      for (int w = 0; w < 2; ++w) {
        if (!P.g[w].on) continue;
        vox[2 * k + w] = P.g[w];
        vox[2 * k + w].off = (int)vox_records;
        vox_records += (size_t)P.nvox[w];
        vox_entries += P.room[w];
        vox_most[w] = std::max(vox_most[w], (int)P.nvox[w]);
      }
    }
  // their device arrays, built from the cell lists; `need`: an error where there is no room
  VoxGrid* d_vox = nullptr;
  uint4* d_vrec = nullptr;
  unsigned* d_vlist = nullptr;
  auto build_lists = [&](bool need) -> int {
    const size_t vox_head = ((2 * (size_t)nboxes * sizeof(VoxGrid) + sizeof(unsigned long long) + 255) & ~(size_t)255);
    const size_t vox_rec = (vox_records * sizeof(uint4) + 255) & ~(size_t)255;
    int rc2 = c->d_vox.reserve(vox_head + vox_rec + (size_t)vox_entries * sizeof(unsigned) + 256);
    if (rc2) {
      cudaGetLastError();  // no room for the lists: the cell search serves every query
      if (need) return rc2;
      for (VoxGrid& g : vox) g.on = 0;
      vox_most[0] = vox_most[1] = 0;
      if ((rc2 = c->d_vox.reserve(vox_head))) return rc2;
    }
    unsigned char* vb = c->d_vox.as<unsigned char>();
    d_vox = reinterpret_cast<VoxGrid*>(vb);
    unsigned long long* d_cursor = reinterpret_cast<unsigned long long*>(vb + 2 * (size_t)nboxes * sizeof(VoxGrid));
    d_vrec = reinterpret_cast<uint4*>(vb + vox_head);
    d_vlist = reinterpret_cast<unsigned*>(vb + vox_head + vox_rec);
    CASS_CUDA(h2d(c, d_vox, vox.data(), vox.size() * sizeof(VoxGrid)));
    CASS_CUDA(cudaMemsetAsync(d_cursor, 0, sizeof(unsigned long long), c->stream));
    CASS_CUDA(cudaEventRecord(c->ev[1], c->stream));
    for (int w = 0; w < 2; ++w)
      if (vox_most[w] > 0) {
        k_vox_lists<<<dim3((vox_most[w] + 127) / 128, nboxes), 128, 0, c->stream>>>(
            d_bd, d_vox, w, d_c32, c->d_cell_start.as<int>(), d_vrec, d_vlist, d_cursor);
        CASS_CUDA(cudaGetLastError());
        count_launch(c);
      }
    return CASS_OK;
  };
  // The launch of a warp-wide kernel: insertions per warp, as few as give every warp of
  // the GPU work at once (`waves` times), up to one per lane; then one group of insertions
  // per warp: a CTA is as long as its slowest warp and the hardware hands out the CTAs; in
  // very large calls several, to stage the box less often.  Cell rows fill the lanes
  // whatever a warp's insertions are, and a half-empty wave of long groups costs more than
  // the shorter ones: two waves where they serve (64 boxes of 180 x 1,000: 5.9 ms with one,
  // 4.2 with two, 4.0 with four; one box of 180 x 100,000: 4.4, 4.9, 5.8).
  int per_warp = 1, wthreads = 32;
  auto warp_grid = [&](int warps, int waves) {
    while (per_warp < 32 && (n_ins + per_warp - 1) / per_warp * nboxes > (long long)dev_sms * warps * waves) per_warp *= 2;
    const long long groups = (n_ins + per_warp - 1) / per_warp;
    wthreads = 32 * (int)std::min<long long>(warps, std::max<long long>(1, (groups * nboxes + dev_sms - 1) / dev_sms));
    const long long need = (groups + wthreads / 32 - 1) / (wthreads / 32);
    const long long most = std::max<long long>(1, (long long)dev_sms * kF32Waves / nboxes);
    const long long turns = (need + most - 1) / most;
    const int chunks = (int)std::max<long long>(1, (need + turns - 1) / turns);
    c->stats.widom_grid_x = chunks;
    c->stats.widom_grid_y = nboxes;
    c->stats.widom_block = wthreads;
    return dim3(chunks, nboxes);
  };
  // FP64 kernel on the lists; no room for them: a negative status, and the thread-per-insertion kernel serves the call
  auto launch_w64 = [&]() -> int {
    int rc2 = build_lists(true);
    if (rc2) return rc2;
    const size_t box = (size_t)std::max(1, max_na) * sizeof(float4);
    auto dyn_of = [&](int warps, bool staged) { return kHead64Bytes + warps * sizeof(Coop64) + (staged ? box : 0); };
    int warps = kThreads64 / 32;
    while (warps > 4 && dyn_of(warps, true) > kSmemMax) warps /= 2;
    const bool staged = dyn_of(warps, true) <= kSmemMax;
    if (!staged) warps = kThreads64 / 32;
    const size_t dyn = dyn_of(warps, staged);
    auto kern = staged ? k_widom_w<true> : k_widom_w<false>;
    CASS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    const dim3 g = warp_grid(warps, 1);
    c->stats.widom_smem_bytes = (int)dyn;
    kern<<<g, wthreads, dyn, c->stream>>>(S, c->pt, c->pools, d_bd, d_ids, c->d_c64.as<double4_32a>(), d_c32, d_vox,
                                          d_vrec, reinterpret_cast<const uint4*>(d_vlist), s.d_library.as<double>(),
                                          (long long)n_ins, seed, per_warp, d_rec, d_status, d_xyz, any_recip ? 1 : 0,
                                          d_trace, d_pairs);
    CASS_CUDA(cudaGetLastError());
    CASS_CUDA(cudaEventRecord(c->ev[2], c->stream));
    count_launch(c);
    return CASS_OK;
  };
  // warps per CTA: as many as fit beside the staged box
  auto smem_f32 = [&](int warps, bool box) { return kCoopHeadBytes + warps * sizeof(CoopWarp) + (box ? max_smem32 : 0); };
  int warps32 = kF32Threads / 32;
  while (warps32 > 4 && smem_f32(warps32, true) > kSmemMax) warps32 /= 2;
  const bool smem32 = smem_f32(warps32, true) <= kSmemMax;
  if (!smem32) warps32 = kF32Threads / 32;
  auto launch_f32 = [&](auto kern, const SpeciesF& SF) -> int {
    const size_t fix_off = ((size_t)nboxes * sizeof(int) + 63) & ~(size_t)63;
    int rc2 = c->d_widom_fix.reserve(fix_off + 64 + nrec * sizeof(FixEntry));
    if (rc2) return rc2;
    d_fixn = c->d_widom_fix.as<int>();
    d_fixq = reinterpret_cast<FixEntry*>(c->d_widom_fix.as<unsigned char>() + fix_off);
    CASS_CUDA(cudaMemsetAsync(d_fixn, 0, (size_t)nboxes * sizeof(int), c->stream));
    if ((rc2 = build_lists(false))) return rc2;
    const size_t dyn = smem_f32(warps32, smem32);
    CASS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dyn));
    bool rows = false;
    for (int k = 0; k < nboxes; ++k) rows = rows || !vox[2 * k].on || !vox[2 * k + 1].on;
    const dim3 g = warp_grid(warps32, rows ? 2 : 1);
    c->stats.widom_smem_bytes = (int)dyn;
    kern<<<g, wthreads, dyn, c->stream>>>(
        S, SF, c->pt, d_bd, d_ids, d_c32, c->d_cq32.as<float>(), c->d_cell_start.as<int>(), s.d_library_f.as<float>(),
        (long long)n_ins, seed, d_rec, d_status, d_xyz, any_recip ? 1 : 0, d_trace, d_fixq, d_fixn, per_warp,
        d_vox, d_vrec, reinterpret_cast<const uint4*>(d_vlist), c->widom_band, d_pairs);
    CASS_CUDA(cudaGetLastError());
    // one thread per queued insertion, the grid sized for 3 % of the
    // insertions (one to two per cent are queued; a longer queue is strided)
    const int fix_chunks = (int)std::max<long long>(1, std::min<long long>(64, (n_ins * 3 / 100 + 127) / 128));
    k_widom_fix<<<dim3(fix_chunks, nboxes), 128, 0, c->stream>>>(
        S, SF, c->pt, d_bd, d_ids, d_c32, c->d_cq32.as<float>(), c->d_c64.as<double4_32a>(), c->d_cell_start.as<int>(),
        s.d_library.as<double>(), (long long)n_ins, seed, d_fixq, d_fixn, d_rec, d_status, d_xyz, any_recip ? 1 : 0,
        d_trace, c->widom_band);
    CASS_CUDA(cudaGetLastError());
    CASS_CUDA(cudaEventRecord(c->ev[2], c->stream));
    count_launch(c, 2);
    return CASS_OK;
  };
  if (n_ins > 0) {
    const bool opt = c->cbmc_opt.energy_table_res > 0 || c->cbmc_opt.sector_overlap;  // no pair counts with options
    if (f32 && opt) rc = smem32 ? launch_f32(k_widom_f32<true, false, true>, SF) : launch_f32(k_widom_f32<false, false, true>, SF);
    else if (f32 && d_pairs) rc = smem32 ? launch_f32(k_widom_f32<true, true, false>, SF) : launch_f32(k_widom_f32<false, true, false>, SF);
    else if (f32) rc = smem32 ? launch_f32(k_widom_f32<true, false, false>, SF) : launch_f32(k_widom_f32<false, false, false>, SF);
    else if (warp64) rc = launch_w64();
    if (!f32 && (!warp64 || rc == CASS_ENOMEM)) rc = use_smem ? launch(k_widom<true>) : launch(k_widom<false>);
    if (rc) return rc;
    if (any_recip) {
      std::vector<RecipBox> rb(nboxes);
      for (int k = 0; k < nboxes; ++k) {
        const BoxH& B = c->box[iboxes[k] - 1];
        RecipBox& R = rb[k];
        memset(&R, 0, sizeof(R));
        if (!has_ew[k]) continue;
        R.kvec = B.d_kvec.as<double4_32a>();
        R.kint = B.kint_ok ? B.d_kint.as<int>() : nullptr;
        R.cos_sum = B.d_cos_sum.as<double>();
        R.sin_sum = B.d_sin_sum.as<double>();
        R.nv = B.nvecs;
        for (int d = 0; d < 3; ++d) {
          R.kn[d] = B.kn[d];
          R.h1[d] = kTWOPI / B.dev.L[d];
        }
      }
      if ((rc = c->d_partial.reserve(rb.size() * sizeof(RecipBox)))) return rc;
      RecipBox* d_rb = c->d_partial.as<RecipBox>();
      CASS_CUDA(h2d(c, d_rb, rb.data(), rb.size() * sizeof(RecipBox)));
      double* d_q = d_xyz + nrec * 3 * s.natoms;
      CASS_CUDA(h2d(c, d_q, s.q.data(), s.natoms * sizeof(double)));
      k_widom_recip<<<(unsigned)nrec, kRecipThreads, 0, c->stream>>>(d_rb, (long long)n_ins, s.natoms, d_q, d_status,
                                                                     d_xyz, d_rec, d_trace);
      CASS_CUDA(cudaGetLastError());
  count_launch(c);
    }
  }
  k_widom_finalize<<<nboxes, 256, 0, c->stream>>>(d_bd, (long long)n_ins, d_rec, d_status, d_bsum, d_bov, d_trace);
  CASS_CUDA(cudaGetLastError());
  count_launch(c);
  CASS_CUDA(cudaEventRecord(c->ev[3], c->stream));
  unsigned long long hpairs[2] = {0, 0};
  if (d_pairs) CASS_CUDA(d2h(c, hpairs, d_pairs, sizeof(hpairs)));
  std::vector<int> hfix(d_fixn ? nboxes : 0);
  if (d_fixn) CASS_CUDA(d2h(c, hfix.data(), d_fixn, nboxes * sizeof(int)));
  std::vector<double> hs(nboxes);
  std::vector<long long> ho(nboxes);
  CASS_CUDA(d2h(c, hs.data(), d_bsum, nboxes * sizeof(double)));
  CASS_CUDA(d2h(c, ho.data(), d_bov, nboxes * sizeof(long long)));
  if (trace)
    CASS_CUDA(d2h(c, trace, d_trace, nrec * sizeof(CassWidomTrace)));
  CASS_CUDA(cudaStreamSynchronize(c->stream));
  float ms_all = 0.0f, ms_k = 0.0f;
  CASS_CUDA(cudaEventElapsedTime(&ms_all, c->ev[0], c->ev[3]));
  if (n_ins > 0) CASS_CUDA(cudaEventElapsedTime(&ms_k, c->ev[1], c->ev[2]));
  c->stats.widom_ms = ms_all;
  c->stats.widom_kernel_ms = ms_k;
  c->stats.widom_pairs_visited = (int64_t)hpairs[0];
  c->stats.widom_pairs_in_cutoff = (int64_t)hpairs[1];
  c->stats.widom_fixups = 0;
  for (int v : hfix) c->stats.widom_fixups += v;
  for (int k = 0; k < nboxes; ++k) {
    out[k].widom_sum = hs[k] * bd[k].prefactor;
    out[k].prefactor = bd[k].prefactor;
    out[k].n_insertions = n_ins;
    out[k].n_overlaps = ho[k];
    out[k].n_trials = n_ins * (int64_t)(kappa_ins + (s.nfrag - 1) * (s.nfrag > 1 ? kappa_dih : 0));
  }
  return CASS_OK;
}

// The cell-edge autotuner of the thread-per-insertion FP64 kernel: the first call with a new batch
// signature (species, boxes, CBMC options, order of magnitude of the insertion count)
// times the kernel with each candidate edge on a sample of the insertions with its own
// seed (the faster of two runs after a first that sizes the buffers), keeps the faster
// one for the context, and then runs the call.  The edge changes neither the
// insertions' random streams nor the per-box sums (fixed order over insertions), only
// the order of each query's pair sum.  The mixed kernel has one shape: its queries
// hardly use the cells, and the lists' own edge does not matter within a tenth.
static int widom_insert_tuned(cass_ctx* c, int32_t is1, int32_t nboxes, const int32_t* iboxes, int64_t n_ins,
                              int32_t kappa_ins, int32_t kappa_dih, uint64_t seed, CassWidomResult* out,
                              CassWidomTrace* trace) {
  bool tune = c && c->precision != CASS_PREC_MIXED && iboxes && nboxes >= 1 && out && n_ins >= 64 && c->widom_autotune &&
              !(c->widom_cells > 0.0);
  for (int k = 0; tune && k < nboxes; ++k) tune = iboxes[k] >= 1 && iboxes[k] <= c->nboxes;
  for (int k = 0; tune && k < nboxes; ++k)
    if (pack_box_ext(c, iboxes[k] - 1)) tune = false;  // the call itself says why
  if (!tune || lists64(c, nboxes, iboxes))
    return widom_insert_impl(c, is1, nboxes, iboxes, n_ins, kappa_ins, kappa_dih, seed, out, trace);
  std::vector<long long> key = {is1, c->precision, kappa_ins, kappa_dih, c->cbmc_opt.energy_table_res,
                                c->cbmc_opt.sector_overlap, (long long)std::log2((double)n_ins)};
  for (int k = 0; k < nboxes; ++k) key.push_back(iboxes[k]);
  auto run_with = [&](double cells, int64_t n, uint64_t sd, CassWidomResult* o, CassWidomTrace* tr) {
    c->widom_cells = cells;
    const int rc = widom_insert_impl(c, is1, nboxes, iboxes, n, kappa_ins, kappa_dih, seed ^ sd, o, tr);
    c->widom_cells = 0.0;
    return rc;
  };
  for (const auto& e : c->widom_tuned)
    if (e.first == key) return run_with(e.second, n_ins, 0, out, trace);
  const double shapes[] = {3.0, 4.0};  // cells per rcut_cbmc
  const int64_t sample = std::min<int64_t>(n_ins, 4096);
  std::vector<CassWidomResult> tmp(nboxes);
  double best = shapes[0];
  float best_ms = -1.0f;
  for (double sh : shapes) {
    float ms = 0.0f;
    for (int rep = 0; rep < 3; ++rep) {  // the first run of a shape also sizes its buffers
      const int rc = run_with(sh, sample, 0x5bd1e995ULL, tmp.data(), nullptr);
      if (rc) return rc;
      if (rep == 1 || (rep == 2 && c->stats.widom_kernel_ms < ms)) ms = c->stats.widom_kernel_ms;
    }
    if (best_ms < 0.0f || ms < best_ms) {
      best_ms = ms;
      best = sh;
    }
  }
  c->widom_tuned.push_back({key, best});
  return run_with(best, n_ins, 0, out, trace);
}

// A batch whose lists need more than kVoxMaxBytes together is worked off in pieces, box
// after box as they fit; in FP64 the boxes without lists (k_widom) are a piece of their
// own, so that one of them does not send the others there (17 boxes x 1,000 butane
// insertions, one of them without lists: 20.1 ms together, 18.7 ms so, 16.5 ms of it the one).
extern "C" int cass_widom_insert(cass_ctx* c, int32_t is1, int32_t nboxes, const int32_t* iboxes, int64_t n_ins,
                                 int32_t kappa_ins, int32_t kappa_dih, uint64_t seed, CassWidomResult* out,
                                 CassWidomTrace* trace) {
  if (c) CASS_CUDA(cudaSetDevice(c->device));  // the boxes are packed to tell how they are worked off
  bool ok = c && iboxes && out && nboxes > 1 && is1 >= 1 && is1 <= c->nspecies && n_ins > 0;
  for (int k = 0; ok && k < nboxes; ++k) {
    const int ib = iboxes[k] - 1;
    ok = ib >= 0 && ib < c->nboxes && (c->box[ib].energy_valid || c->box[ib].frame_ready) && !pack_box_ext(c, ib);
  }
  std::vector<int> piece(ok ? nboxes : 0, 0);
  int npieces = 1;
  if (ok) {
    if (int rc = ensure_cbmc(c)) return rc;
    SpeciesF SF;
    const bool f32 = c->sp[is1 - 1].defined && mixed_f32(c, c->sp[is1 - 1], nboxes, iboxes, SF);
    double bytes = 0.0;
    bool any = false, rest = false;
    npieces = 0;
    for (int k = 0; k < nboxes; ++k) {
      const BoxH& B = c->box[iboxes[k] - 1];
      piece[k] = -1;
      if (!f32 && !lists64(c, B)) {
        rest = true;
        continue;
      }
      const double need = box_lists(c, B, f32, n_ins).bytes();
      if (!any || (bytes > 0.0 && bytes + need > kVoxMaxBytes)) {
        ++npieces;
        bytes = 0.0;
      }
      any = true;
      bytes += need;
      piece[k] = npieces - 1;
    }
    if (rest) ++npieces;  // the boxes without lists
    for (int& q : piece) q = q < 0 ? npieces - 1 : q;
  }
  if (npieces == 1)  // also whatever is wrong with the call: the reason comes from there
    return widom_insert_tuned(c, is1, nboxes, iboxes, n_ins, kappa_ins, kappa_dih, seed, out, trace);
  CassStats sum{};
  for (int p = 0; p < npieces; ++p) {
    std::vector<int> at;
    std::vector<int32_t> ids;
    for (int k = 0; k < nboxes; ++k)
      if (piece[k] == p) {
        at.push_back(k);
        ids.push_back(iboxes[k]);
      }
    std::vector<CassWidomResult> o(at.size());
    std::unique_ptr<CassWidomTrace[]> t;
    if (trace) {
      t.reset(new (std::nothrow) CassWidomTrace[at.size() * (size_t)n_ins]);
      if (!t) return set_error(CASS_ENOMEM, "no room for the records of a piece of the batch");
    }
    if (int rc = widom_insert_tuned(c, is1, (int)ids.size(), ids.data(), n_ins, kappa_ins, kappa_dih, seed, o.data(),
                                    t.get()))
      return rc;
    for (size_t q = 0; q < at.size(); ++q) {
      out[at[q]] = o[q];
      if (trace) memcpy(trace + (size_t)at[q] * n_ins, t.get() + q * n_ins, n_ins * sizeof(CassWidomTrace));
    }
    sum.widom_ms += c->stats.widom_ms;
    sum.widom_kernel_ms += c->stats.widom_kernel_ms;
    sum.widom_pairs_visited += c->stats.widom_pairs_visited;
    sum.widom_pairs_in_cutoff += c->stats.widom_pairs_in_cutoff;
    sum.widom_fixups += c->stats.widom_fixups;
  }
  c->stats.widom_ms = sum.widom_ms;
  c->stats.widom_kernel_ms = sum.widom_kernel_ms;
  c->stats.widom_pairs_visited = sum.widom_pairs_visited;
  c->stats.widom_pairs_in_cutoff = sum.widom_pairs_in_cutoff;
  c->stats.widom_fixups = sum.widom_fixups;
  return CASS_OK;
}
