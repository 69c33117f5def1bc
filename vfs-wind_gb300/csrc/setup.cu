// setup.cu -- grid metrics, dof numbering, operator assembly, right-hand
// side, pressure update, projection, divergence and the multigrid transfer
// operators.
//
// This translation unit is compiled with -fmad=false: every floating-point
// expression is rounded in the reference's source order, so these kernels
// reproduce the reference's arithmetic (restated in the oracle) bit for bit.
// Each kernel names the reference lines it follows.
#include "common.cuh"
#include "kernels.cuh"

namespace vfs {

static constexpr double kThr = 0.1;  // poisson_threshold, Source/main.c:124

// --------------------------------------------------------------------------
// FormMetrics (Source/metrics.c:12-1355; metrics.c:10 defines NEWMETRIC)
// --------------------------------------------------------------------------
#define CO(i, j, k, c) coor[g.at(i, j, k) * 3 + (c)]

// cell centres (metrics.c:89-108) and, for every interior cell, aj = 1/J and
// the cell metrics csi/eta/zet from the 8-node differences
// (metrics.c:194-256, the NEWMETRIC branch)
__global__ void k_metrics_cell(Grid g, const double *__restrict__ coor, MetricPtrs m) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= g.mx) return;
  size_t t = g.at(i, j, k);
  const int mx = g.mx, my = g.my, mz = g.mz;
  if (!(i >= 1 && i < mx - 1 && j >= 1 && j < my - 1 && k >= 1 && k < mz - 1)) return;
  for (int c = 0; c < 3; c++)
    m.cent[t * 3 + c] = 0.125 * (CO(i, j, k, c) + CO(i, j - 1, k, c) + CO(i, j, k - 1, c) + CO(i, j - 1, k - 1, c) +
                                 CO(i - 1, j, k, c) + CO(i - 1, j - 1, k, c) + CO(i - 1, j, k - 1, c) +
                                 CO(i - 1, j - 1, k - 1, c));
  double dc[3], de[3], dz[3];
  for (int c = 0; c < 3; c++) {
    dc[c] = 0.25 * (CO(i, j, k, c) + CO(i, j - 1, k, c) + CO(i, j, k - 1, c) + CO(i, j - 1, k - 1, c) -
                    CO(i - 1, j, k, c) - CO(i - 1, j - 1, k, c) - CO(i - 1, j, k - 1, c) - CO(i - 1, j - 1, k - 1, c));
    de[c] = 0.25 * (CO(i, j, k, c) + CO(i - 1, j, k, c) + CO(i, j, k - 1, c) + CO(i - 1, j, k - 1, c) -
                    CO(i, j - 1, k, c) - CO(i - 1, j - 1, k, c) - CO(i, j - 1, k - 1, c) - CO(i - 1, j - 1, k - 1, c));
    dz[c] = 0.25 * (CO(i, j, k, c) + CO(i, j - 1, k, c) + CO(i - 1, j, k, c) + CO(i - 1, j - 1, k, c) -
                    CO(i, j, k - 1, c) - CO(i, j - 1, k - 1, c) - CO(i - 1, j, k - 1, c) - CO(i - 1, j - 1, k - 1, c));
  }
  double det = dc[0] * (de[1] * dz[2] - de[2] * dz[1]) - dc[1] * (de[0] * dz[2] - de[2] * dz[0]) +
               dc[2] * (de[0] * dz[1] - de[1] * dz[0]);
  m.aj[t] = 1. / det;
  double *cs = &m.csi[t * 3], *et = &m.eta[t * 3], *ze = &m.zet[t * 3];
  cs[0] = de[1] * dz[2] - de[2] * dz[1];
  cs[1] = -de[0] * dz[2] + de[2] * dz[0];
  cs[2] = de[0] * dz[1] - de[1] * dz[0];
  et[0] = dz[1] * dc[2] - dz[2] * dc[1];
  et[1] = -dz[0] * dc[2] + dz[2] * dc[0];
  et[2] = dz[0] * dc[1] - dz[1] * dc[0];
  ze[0] = dc[1] * de[2] - dc[2] * de[1];
  ze[1] = -dc[0] * de[2] + dc[2] * de[0];
  ze[2] = dc[0] * de[1] - dc[1] * de[0];
}

// boundary mirror of csi, eta, zet and aj, one direction per launch, in the
// order x, y, z of metrics.c:262-342.
__global__ void k_metrics_mirror(Grid g, MetricPtrs m, int dir) {
  int u = blockIdx.x * blockDim.x + threadIdx.x, v = blockIdx.y;
  int nu = dir == 0 ? g.my : g.mx, nv = dir == 2 ? g.my : g.mz;
  if (u >= nu || v >= nv) return;
  for (int side = 0; side < 2; side++) {
    size_t t, s;
    if (dir == 0) { int i = side ? g.mx - 1 : 0; t = g.at(i, u, v); s = g.at(side ? i - 1 : 1, u, v); }
    else if (dir == 1) { int j = side ? g.my - 1 : 0; t = g.at(u, j, v); s = g.at(u, side ? j - 1 : 1, v); }
    else { int k = side ? g.mz - 1 : 0; t = g.at(u, v, k); s = g.at(u, v, side ? k - 1 : 1); }
    for (int c = 0; c < 3; c++) {
      m.csi[t * 3 + c] = m.csi[s * 3 + c];
      m.eta[t * 3 + c] = m.eta[s * 3 + c];
      m.zet[t * 3 + c] = m.zet[s * 3 + c];
    }
    m.aj[t] = m.aj[s];
  }
}

// periodic ghost copy: of the cell metrics before the face averages
// (metrics.c:360-397), of all sixteen arrays at the end (metrics.c:1227-1262).
// A source cell has every periodic coordinate inside 1..m-2, so it is never
// a target.
__global__ void k_metrics_periodic(Grid g, MetricPtrs m, int faces) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= g.mx) return;
  int a, b, c, fi, fj, fk;
  if (!g.remap(i, j, k, a, b, c, fi, fj, fk)) return;
  size_t s = g.at(a, b, c), t = g.at(i, j, k);
  double *v3[12] = {m.csi, m.eta, m.zet, m.icsi, m.ieta, m.izet, m.jcsi, m.jeta, m.jzet, m.kcsi, m.keta, m.kzet};
  double *v1[4] = {m.aj, m.iaj, m.jaj, m.kaj};
  const int n3 = faces ? 12 : 3, n1 = faces ? 4 : 1;
  for (int q = 0; q < n3; q++)
    for (int e = 0; e < 3; e++) v3[q][t * 3 + e] = v3[q][s * 3 + e];
  for (int q = 0; q < n1; q++) v1[q][t] = v1[q][s];
}

// NEWMETRIC face metrics (metrics.c:588-592, :696-700, :804-808): the
// arithmetic mean of the two adjacent cells' csi/eta/zet (AxByC,
// Source/momentum.c:40-45) and the harmonic mean of their aj; i faces
// i = 0..mx-2 of the interior j, k; j faces j = 0..my-2; k faces k = 0..mz-2.
__global__ void k_metrics_face(Grid g, MetricPtrs m, int dir) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  const int mx = g.mx, my = g.my, mz = g.mz;
  bool in;
  if (dir == 0) in = i < mx - 1 && j >= 1 && j < my - 1 && k >= 1 && k < mz - 1;
  else if (dir == 1) in = i >= 1 && i < mx - 1 && j < my - 1 && k >= 1 && k < mz - 1;
  else in = i >= 1 && i < mx - 1 && j >= 1 && j < my - 1 && k < mz - 1;
  if (!in) return;
  const size_t t = g.at(i, j, k);
  const size_t u = dir == 0 ? g.at(i + 1, j, k) : dir == 1 ? g.at(i, j + 1, k) : g.at(i, j, k + 1);
  double *fc = dir == 0 ? m.icsi : dir == 1 ? m.jcsi : m.kcsi;
  double *fe = dir == 0 ? m.ieta : dir == 1 ? m.jeta : m.keta;
  double *fz = dir == 0 ? m.izet : dir == 1 ? m.jzet : m.kzet;
  double *fa = dir == 0 ? m.iaj : dir == 1 ? m.jaj : m.kaj;
  for (int c = 0; c < 3; c++) {
    fc[t * 3 + c] = 0.5 * m.csi[t * 3 + c] + 0.5 * m.csi[u * 3 + c];
    fe[t * 3 + c] = 0.5 * m.eta[t * 3 + c] + 0.5 * m.eta[u * 3 + c];
    fz[t * 3 + c] = 0.5 * m.zet[t * 3 + c] + 0.5 * m.zet[u * 3 + c];
  }
  fa[t] = 2. / (1. / m.aj[t] + 1. / m.aj[u]);
}
#undef CO

// --------------------------------------------------------------------------
// Dof numbering, setup_lidx2 (Source/poisson.c:188-335)
// --------------------------------------------------------------------------
__device__ inline bool is_dof_cell(const Grid &g, const double *nvert, int i, int j, int k) {
  // poisson.c:244-251: interior and (int)nvert <= poisson_threshold
  if (i <= 0 || i >= g.mx - 1 || j <= 0 || j >= g.my - 1 || k <= 0 || k >= g.mz - 1) return false;
  return !((int)nvert[g.at(i, j, k)] > kThr);
}
// dof test of a possibly-ghost point, with the periodic aliasing of
// poisson.c:299-332 (Gid of a periodic ghost is its partner's Gid).
__device__ inline bool has_dof(const Grid &g, const double *nvert, int i, int j, int k) {
  int a, b, c, fi, fj, fk;
  g.remap(i, j, k, a, b, c, fi, fj, fk);
  return is_dof_cell(g, nvert, a, b, c);
}

// Four cells a thread, 1024 a block of the numbering: a dof's row type is not 0
// (assemble_cell), one byte a cell instead of eight of nvert; bit q of the result:
// cell c + q is a dof.
__device__ __forceinline__ uint32_t dof_bits(const uint8_t *__restrict__ rowtype, size_t c, size_t n) {
  uint32_t v = 0;
  if (c + 4 <= n) {
    v = *(const uint32_t *)(rowtype + c);  // (c is a multiple of four)
  } else {
    for (int q = 0; q < 4; q++)
      if (c + q < n) v |= (uint32_t)rowtype[c + q] << (8 * q);
  }
  return ((v & 0xffu) ? 1u : 0u) | ((v & 0xff00u) ? 2u : 0u) | ((v & 0xff0000u) ? 4u : 0u) | (v >> 24 ? 8u : 0u);
}
// per-block dof counts over the box order (k-j-i, the reference's loop order).
// 384x192x384: 0.086 ms with a byte a thread, 0.023 with four.
__global__ void __launch_bounds__(256) k_count_dofs(size_t n, const uint8_t *__restrict__ rowtype, int *block_count) {
  __shared__ int tot[8];
  const uint32_t f = dof_bits(rowtype, ((size_t)blockIdx.x * 256 + threadIdx.x) * 4, n);
  const int s = (int)__reduce_add_sync(0xffffffffu, (unsigned)__popc(f));
  if ((threadIdx.x & 31) == 0) tot[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int q = 0; q < 8; q++) t += tot[q];
    block_count[blockIdx.x] = t;
  }
}
// exclusive scan of the block counts by one block (sequential per thread
// chunk, then a scan over the 1024 chunk totals).
__global__ void k_scan_blocks(int *block_count, int nblocks, int *total) {
  __shared__ int part[32];
  int per = (nblocks + blockDim.x - 1) / blockDim.x;
  int lo = threadIdx.x * per, hi = min(nblocks, lo + per);
  int s = 0;
  for (int q = lo; q < hi; q++) s += block_count[q];
  // the totals' exclusive scan: a warp's by shuffles, 32 warps' by the first
  // (one thread over 1024 of them: 20 us)
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  auto scan = [&](int v) {
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += u;
    }
    return v;
  };
  const int inc = scan(s);
  if (lane == 31) part[w] = inc;
  __syncthreads();
  if (w == 0) {
    const int v = part[lane], t = scan(v);
    part[lane] = t - v;
    if (lane == 31) *total = t;
  }
  __syncthreads();
  int run = part[w] + inc - s;
  for (int q = lo; q < hi; q++) { int v = block_count[q]; block_count[q] = run; run += v; }
}
// The numbers go straight into the DA-layout Gid; its boundary layer holds -1
// since the handle was made, but for the periodic ghosts (k_gid_ghosts).
// 384x192x384: 0.158 ms with a cell a thread, whose warps added up to 31 totals
// one by one, 0.064 with four.
__global__ void __launch_bounds__(256) k_number_dofs(Grid g, Box b, const uint8_t *__restrict__ rowtype,
                                                     const int *block_off, int *gid_da) {
  __shared__ int tot[8];
  const size_t n = b.n(), c = ((size_t)blockIdx.x * 256 + threadIdx.x) * 4;
  const uint32_t f = dof_bits(rowtype, c, n);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, mine = __popc(f);
  int inc = mine;  // dofs of the warp's cells up to this thread's last
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  if (lane == 31) tot[w] = inc;
  __syncthreads();
  int num = block_off[blockIdx.x] + inc - mine;
  for (int q = 0; q < 7; q++)
    if (q < w) num += tot[q];
  if (c >= n) return;
  int i, j, k;
  box_ijk(b, c, i, j, k);
  for (int q = 0; q < 4 && c + q < n; q++) {
    gid_da[g.at(i + 1, j + 1, k + 1)] = (f >> q & 1) ? num++ : -1;
    if (++i == b.nx) {
      i = 0;
      if (++j == b.ny) { j = 0; k++; }
    }
  }
}
// (declared here for the ghost layers; defined with the other shell passes)
__device__ __forceinline__ bool shell_point(const Grid &g, size_t q, int &i, int &j, int &k);
__global__ void k_gid_ghosts(Grid g, int *gid_da) {
  int i, j, k, a, b, c, fi, fj, fk;
  if (!shell_point(g, (size_t)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
  g.remap(i, j, k, a, b, c, fi, fj, fk);
  gid_da[g.at(i, j, k)] = gid_da[g.at(a, b, c)];
}

// --------------------------------------------------------------------------
// PoissonLHSNew (Source/poisson.c:977-1688), level set off (r = 1)
// --------------------------------------------------------------------------
// g11..g33 at a face with the periodic source remap of poisson.c:1102-1138
__device__ inline double gface_at(const MetricPtrs &m, int q, size_t s) {
  const double *X, *Y, *AJ;
  switch (q) {
    case 0: X = m.icsi; Y = m.icsi; AJ = m.iaj; break;
    case 1: X = m.ieta; Y = m.icsi; AJ = m.iaj; break;
    case 2: X = m.izet; Y = m.icsi; AJ = m.iaj; break;
    case 3: X = m.jcsi; Y = m.jeta; AJ = m.jaj; break;
    case 4: X = m.jeta; Y = m.jeta; AJ = m.jaj; break;
    case 5: X = m.jzet; Y = m.jeta; AJ = m.jaj; break;
    case 6: X = m.kcsi; Y = m.kzet; AJ = m.kaj; break;
    case 7: X = m.keta; Y = m.kzet; AJ = m.kaj; break;
    default: X = m.kzet; Y = m.kzet; AJ = m.kaj; break;
  }
  return (X[s * 3] * Y[s * 3] + X[s * 3 + 1] * Y[s * 3 + 1] + X[s * 3 + 2] * Y[s * 3 + 2]) * AJ[s];
}
__device__ inline double gface(const Grid &g, const MetricPtrs &m, int q, int i, int j, int k) {
  int a, b, c, fi, fj, fk;
  g.remap(i, j, k, a, b, c, fi, fj, fk);
  const size_t s = g.at(a, b, c);
  return m.gface ? m.gface[(size_t)q * g.n() + s] : gface_at(m, q, s);
}
// the nine face coefficients of every DA point, as gface forms them (no FMA
// contraction in this unit: the same bits)
__global__ void k_face_coef(Grid g, MetricPtrs m, double *out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= g.mx) return;
  const size_t s = g.at(i, j, k), n = g.n();
#pragma unroll
  for (int q = 0; q < 9; q++) out[(size_t)q * n + s] = gface_at(m, q, s);
}

// mean (Source/level.c:2276-2280): the harmonic mean of two densities
__device__ inline double ls_mean(double A, double B) { return 2.0 * A * B / (A + B); }

// One row of the operator, accumulated in the reference's statement order.
// With a level set (ls.on) every face coefficient is divided by the face
// density and the Dirichlet top / bottom rows of poisson.c:1295-1554 apply.
template <bool LS>
__device__ void assemble_row_t(const Grid &g, const double *nvert, const MetricPtrs &m, int i, int j, int k,
                               double v[NSLOT], const LevelSet &ls) {
  // a face coefficient divided by the face density: without a level set
  // the density is exactly 1 and the division (exact there) is not issued
#define DR(x) (LS ? (x) / r : (x))
  const int mx = g.mx, my = g.my, mz = g.mz;
  const bool ip = g.px, jp = g.py, kp = g.pz;
  const double thr = kThr;
  double r = 1.0;
#define RHO(a, b, c) ls.rho[g.at(a, b, c)]
#define NV(a, b, c) nvert[g.at(a, b, c)]
#define G(q, a, b, c) gface(g, m, q, a, b, c)
  for (int s = 0; s < NSLOT; s++) v[s] = 0.;
  if (NV(i + 1, j, k) < thr && (i != mx - 2 || ip)) {  // poisson.c:1167-1230
    r = ls.on ? ls_mean(RHO(i + 1, j, k), RHO(i, j, k)) : 1.0;
    double g0 = G(0, i, j, k), g1 = G(1, i, j, k), g2 = G(2, i, j, k);
    v[CP] -= DR(g0); v[EP] += DR(g0);
    if ((j == my - 2 && !jp) || NV(i, j + 1, k) + NV(i + 1, j + 1, k) > thr) {
      if (NV(i, j - 1, k) + NV(i + 1, j - 1, k) < thr && j != 1) {
        v[CP] += DR(g1 * 0.5); v[EP] += DR(g1 * 0.5); v[SP] -= DR(g1 * 0.5); v[SE] -= DR(g1 * 0.5);
      }
    } else if ((j == 1 && !jp) || NV(i, j - 1, k) + NV(i + 1, j - 1, k) > thr) {
      if (NV(i, j + 1, k) + NV(i + 1, j + 1, k) < thr) {
        v[NP] += DR(g1 * 0.5); v[NE] += DR(g1 * 0.5); v[CP] -= DR(g1 * 0.5); v[EP] -= DR(g1 * 0.5);
      }
    } else {
      v[NP] += DR(g1 * 0.25); v[NE] += DR(g1 * 0.25); v[SP] -= DR(g1 * 0.25); v[SE] -= DR(g1 * 0.25);
    }
    if ((k == mz - 2 && !kp) || NV(i, j, k + 1) + NV(i + 1, j, k + 1) > thr) {
      if (NV(i, j, k - 1) + NV(i + 1, j, k - 1) < thr && k != 1) {
        v[CP] += DR(g2 * 0.5); v[EP] += DR(g2 * 0.5); v[BP] -= DR(g2 * 0.5); v[BE] -= DR(g2 * 0.5);
      }
    } else if ((k == 1 && !kp) || NV(i, j, k - 1) + NV(i + 1, j, k - 1) > thr) {
      if (NV(i, j, k + 1) + NV(i + 1, j, k + 1) < thr) {
        v[TP] += DR(g2 * 0.5); v[TE] += DR(g2 * 0.5); v[CP] -= DR(g2 * 0.5); v[EP] -= DR(g2 * 0.5);
      }
    } else {
      v[TP] += DR(g2 * 0.25); v[TE] += DR(g2 * 0.25); v[BP] -= DR(g2 * 0.25); v[BE] -= DR(g2 * 0.25);
    }
  }
  if (NV(i - 1, j, k) < thr && (i != 1 || ip)) {  // poisson.c:1233-1293
    r = ls.on ? ls_mean(RHO(i - 1, j, k), RHO(i, j, k)) : 1.0;
    double g0 = G(0, i - 1, j, k), g1 = G(1, i - 1, j, k), g2 = G(2, i - 1, j, k);
    v[CP] -= DR(g0); v[WP] += DR(g0);
    if ((j == my - 2 && !jp) || NV(i, j + 1, k) + NV(i - 1, j + 1, k) > thr) {
      if (NV(i, j - 1, k) + NV(i - 1, j - 1, k) < thr && j != 1) {
        v[CP] -= DR(g1 * 0.5); v[WP] -= DR(g1 * 0.5); v[SP] += DR(g1 * 0.5); v[SW] += DR(g1 * 0.5);
      }
    } else if ((j == 1 && !jp) || NV(i, j - 1, k) + NV(i - 1, j - 1, k) > thr) {
      if (NV(i, j + 1, k) + NV(i - 1, j + 1, k) < thr) {
        v[NP] -= DR(g1 * 0.5); v[NW] -= DR(g1 * 0.5); v[CP] += DR(g1 * 0.5); v[WP] += DR(g1 * 0.5);
      }
    } else {
      v[NP] -= DR(g1 * 0.25); v[NW] -= DR(g1 * 0.25); v[SP] += DR(g1 * 0.25); v[SW] += DR(g1 * 0.25);
    }
    if ((k == mz - 2 && !kp) || NV(i, j, k + 1) + NV(i - 1, j, k + 1) > thr) {
      if (NV(i, j, k - 1) + NV(i - 1, j, k - 1) < thr && k != 1) {
        v[CP] -= DR(g2 * 0.5); v[WP] -= DR(g2 * 0.5); v[BP] += DR(g2 * 0.5); v[BW] += DR(g2 * 0.5);
      }
    } else if ((k == 1 && !kp) || NV(i, j, k - 1) + NV(i - 1, j, k - 1) > thr) {
      if (NV(i, j, k + 1) + NV(i - 1, j, k + 1) < thr) {
        v[TP] -= DR(g2 * 0.5); v[TW] -= DR(g2 * 0.5); v[CP] += DR(g2 * 0.5); v[WP] += DR(g2 * 0.5);
      }
    } else {
      v[TP] -= DR(g2 * 0.25); v[TW] -= DR(g2 * 0.25); v[BP] += DR(g2 * 0.25); v[BW] += DR(g2 * 0.25);
    }
  }
  if (NV(i, j + 1, k) < thr && (j != my - 2 || jp || (ls.on && ls.bc3 == 4 && j == my - 2))) {  // poisson.c:1296-1361
    r = ls.on ? ls_mean(RHO(i, j + 1, k), RHO(i, j, k)) : 1.0;
    double g3 = G(3, i, j, k), g4 = G(4, i, j, k), g5 = G(5, i, j, k);
    if ((i == mx - 2 && !ip) || NV(i + 1, j, k) + NV(i + 1, j + 1, k) > thr) {
      if (NV(i - 1, j, k) + NV(i - 1, j + 1, k) < thr && i != 1) {
        v[CP] += DR(g3 * 0.5); v[NP] += DR(g3 * 0.5); v[WP] -= DR(g3 * 0.5); v[NW] -= DR(g3 * 0.5);
      }
    } else if ((i == 1 && !ip) || NV(i - 1, j, k) + NV(i - 1, j + 1, k) > thr) {
      if (NV(i + 1, j, k) + NV(i + 1, j + 1, k) < thr) {
        v[EP] += DR(g3 * 0.5); v[NE] += DR(g3 * 0.5); v[CP] -= DR(g3 * 0.5); v[NP] -= DR(g3 * 0.5);
      }
    } else {
      v[EP] += DR(g3 * 0.25); v[NE] += DR(g3 * 0.25); v[WP] -= DR(g3 * 0.25); v[NW] -= DR(g3 * 0.25);
    }
    if (ls.on && ls.bc3 == 4 && j == my - 2) v[CP] -= DR(g4 / 0.5);  // zero Dirichlet pressure, :1328
    else { v[CP] -= DR(g4); v[NP] += DR(g4); }
    if ((k == mz - 2 && !kp) || NV(i, j, k + 1) + NV(i, j + 1, k + 1) > thr) {
      if (NV(i, j, k - 1) + NV(i, j + 1, k - 1) < thr && k != 1) {
        v[CP] += DR(g5 * 0.5); v[NP] += DR(g5 * 0.5); v[BP] -= DR(g5 * 0.5); v[BN] -= DR(g5 * 0.5);
      }
    } else if ((k == 1 && !kp) || NV(i, j, k - 1) + NV(i, j + 1, k - 1) > thr) {
      if (NV(i, j, k + 1) + NV(i, j + 1, k + 1) < thr) {
        v[TP] += DR(g5 * 0.5); v[TN] += DR(g5 * 0.5); v[CP] -= DR(g5 * 0.5); v[NP] -= DR(g5 * 0.5);
      }
    } else {
      v[TP] += DR(g5 * 0.25); v[TN] += DR(g5 * 0.25); v[BP] -= DR(g5 * 0.25); v[BN] -= DR(g5 * 0.25);
    }
  }
  if (NV(i, j - 1, k) < thr && (j != 1 || jp)) {  // poisson.c:1364-1422
    r = ls.on ? ls_mean(RHO(i, j - 1, k), RHO(i, j, k)) : 1.0;
    double g3 = G(3, i, j - 1, k), g4 = G(4, i, j - 1, k), g5 = G(5, i, j - 1, k);
    if ((i == mx - 2 && !ip) || NV(i + 1, j, k) + NV(i + 1, j - 1, k) > thr) {
      if (NV(i - 1, j, k) + NV(i - 1, j - 1, k) < thr && i != 1) {
        v[CP] -= DR(g3 * 0.5); v[SP] -= DR(g3 * 0.5); v[WP] += DR(g3 * 0.5); v[SW] += DR(g3 * 0.5);
      }
    } else if ((i == 1 && !ip) || NV(i - 1, j, k) + NV(i - 1, j - 1, k) > thr) {
      if (NV(i + 1, j, k) + NV(i + 1, j - 1, k) < thr) {
        v[EP] -= DR(g3 * 0.5); v[SE] -= DR(g3 * 0.5); v[CP] += DR(g3 * 0.5); v[SP] += DR(g3 * 0.5);
      }
    } else {
      v[EP] -= DR(g3 * 0.25); v[SE] -= DR(g3 * 0.25); v[WP] += DR(g3 * 0.25); v[SW] += DR(g3 * 0.25);
    }
    v[CP] -= DR(g4); v[SP] += DR(g4);
    if ((k == mz - 2 && !kp) || NV(i, j, k + 1) + NV(i, j - 1, k + 1) > thr) {
      if (NV(i, j, k - 1) + NV(i, j - 1, k - 1) < thr && k != 1) {
        v[CP] -= DR(g5 * 0.5); v[SP] -= DR(g5 * 0.5); v[BP] += DR(g5 * 0.5); v[BS] += DR(g5 * 0.5);
      }
    } else if ((k == 1 && !kp) || NV(i, j, k - 1) + NV(i, j - 1, k - 1) > thr) {
      if (NV(i, j, k + 1) + NV(i, j - 1, k + 1) < thr) {
        v[TP] -= DR(g5 * 0.5); v[TS] -= DR(g5 * 0.5); v[CP] += DR(g5 * 0.5); v[SP] += DR(g5 * 0.5);
      }
    } else {
      v[TP] -= DR(g5 * 0.25); v[TS] -= DR(g5 * 0.25); v[BP] += DR(g5 * 0.25); v[BS] += DR(g5 * 0.25);
    }
  }
  if (NV(i, j, k + 1) < thr && (k != mz - 2 || kp || (ls.on && ls.bc5 == 4 && k == mz - 2))) {  // poisson.c:1425-1491
    r = ls.on ? ls_mean(RHO(i, j, k + 1), RHO(i, j, k)) : 1.0;
    double g6 = G(6, i, j, k), g7 = G(7, i, j, k), g8 = G(8, i, j, k);
    if ((i == mx - 2 && !ip) || NV(i + 1, j, k) + NV(i + 1, j, k + 1) > thr) {
      if (NV(i - 1, j, k) + NV(i - 1, j, k + 1) < thr && i != 1) {
        v[CP] += DR(g6 * 0.5); v[TP] += DR(g6 * 0.5); v[WP] -= DR(g6 * 0.5); v[TW] -= DR(g6 * 0.5);
      }
    } else if ((i == 1 && !ip) || NV(i - 1, j, k) + NV(i - 1, j, k + 1) > thr) {
      if (NV(i + 1, j, k) + NV(i + 1, j, k + 1) < thr) {
        v[EP] += DR(g6 * 0.5); v[TE] += DR(g6 * 0.5); v[CP] -= DR(g6 * 0.5); v[TP] -= DR(g6 * 0.5);
      }
    } else {
      v[EP] += DR(g6 * 0.25); v[TE] += DR(g6 * 0.25); v[WP] -= DR(g6 * 0.25); v[TW] -= DR(g6 * 0.25);
    }
    if ((j == my - 2 && !jp) || NV(i, j + 1, k) + NV(i, j + 1, k + 1) > thr) {
      if (NV(i, j - 1, k) + NV(i, j - 1, k + 1) < thr && j != 1) {
        v[CP] += DR(g7 * 0.5); v[TP] += DR(g7 * 0.5); v[SP] -= DR(g7 * 0.5); v[TS] -= DR(g7 * 0.5);
      }
    } else if ((j == 1 && !jp) || NV(i, j - 1, k) + NV(i, j - 1, k + 1) > thr) {
      if (NV(i, j + 1, k) + NV(i, j + 1, k + 1) < thr) {
        v[NP] += DR(g7 * 0.5); v[TN] += DR(g7 * 0.5); v[CP] -= DR(g7 * 0.5); v[TP] -= DR(g7 * 0.5);
      }
    } else {
      v[NP] += DR(g7 * 0.25); v[TN] += DR(g7 * 0.25); v[SP] -= DR(g7 * 0.25); v[TS] -= DR(g7 * 0.25);
    }
    if (ls.on && ls.bc5 == 4 && k == mz - 2) v[CP] -= DR(g8 / 0.5);  // :1482-1484
    else { v[CP] -= DR(g8); v[TP] += DR(g8); }
  }
  if (NV(i, j, k - 1) < thr &&
      (k != 1 || kp || (ls.on && ls.bc4 == 5000 && k == 1 && ls.level[g.at(i, j, k)] < 0))) {  // poisson.c:1494-1561
    r = ls.on ? (k == 1 ? RHO(i, j, k) : ls_mean(RHO(i, j, k - 1), RHO(i, j, k))) : 1.0;
    double g6 = G(6, i, j, k - 1), g7 = G(7, i, j, k - 1), g8 = G(8, i, j, k - 1);
    if ((i == mx - 2 && !ip) || NV(i + 1, j, k) + NV(i + 1, j, k - 1) > thr) {
      if (NV(i - 1, j, k) + NV(i - 1, j, k - 1) < thr && i != 1) {
        v[CP] -= DR(g6 * 0.5); v[BP] -= DR(g6 * 0.5); v[WP] += DR(g6 * 0.5); v[BW] += DR(g6 * 0.5);
      }
    } else if ((i == 1 && !ip) || NV(i - 1, j, k) + NV(i - 1, j, k - 1) > thr) {
      if (NV(i + 1, j, k) + NV(i + 1, j, k - 1) < thr) {
        v[EP] -= DR(g6 * 0.5); v[BE] -= DR(g6 * 0.5); v[CP] += DR(g6 * 0.5); v[BP] += DR(g6 * 0.5);
      }
    } else {
      v[EP] -= DR(g6 * 0.25); v[BE] -= DR(g6 * 0.25); v[WP] += DR(g6 * 0.25); v[BW] += DR(g6 * 0.25);
    }
    if ((j == my - 2 && !jp) || NV(i, j + 1, k) + NV(i, j + 1, k - 1) > thr) {
      if (NV(i, j - 1, k) + NV(i, j - 1, k - 1) < thr && j != 1) {
        v[CP] -= DR(g7 * 0.5); v[BP] -= DR(g7 * 0.5); v[SP] += DR(g7 * 0.5); v[BS] += DR(g7 * 0.5);
      }
    } else if ((j == 1 && !jp) || NV(i, j - 1, k) + NV(i, j - 1, k - 1) > thr) {
      if (NV(i, j + 1, k) + NV(i, j + 1, k - 1) < thr) {
        v[NP] -= DR(g7 * 0.5); v[BN] -= DR(g7 * 0.5); v[CP] += DR(g7 * 0.5); v[BP] += DR(g7 * 0.5);
      }
    } else {
      v[NP] -= DR(g7 * 0.25); v[BN] -= DR(g7 * 0.25); v[SP] += DR(g7 * 0.25); v[BS] += DR(g7 * 0.25);
    }
    if (ls.on && ls.bc4 == 5 && k == 1) v[CP] -= DR(g8 / 0.5);  // :1552-1554
    else { v[CP] -= DR(g8); v[BP] += DR(g8); }
  }
#undef RHO
#undef NV
#undef G
#undef DR
}
__device__ void assemble_row(const Grid &g, const double *nvert, const MetricPtrs &m, int i, int j, int k,
                             double v[NSLOT], const LevelSet &ls) {
  if (ls.on) assemble_row_t<true>(g, nvert, m, i, j, k, v, ls);
  else assemble_row_t<false>(g, nvert, m, i, j, k, v, ls);
}

// Assemble one level's operator into 19 box-layout planes.  filter: the
// reference's insertion test |v| > 1e-10 (poisson.c:1610-1614); scale: the
// aj row scaling of the poisson == -1 path (poisson.c:1563), used for the
// multigrid levels; split: store rows in the parity-split row layout of the
// multigrid levels (rowtype stays natural).  Slots whose column has no dof
// are zero (idx < 0).
__device__ __forceinline__ void assemble_cell(const Grid &g, const Box &b, const double *__restrict__ nvert,
                                              const MetricPtrs &m, int scale, int filter, int split, double *A,
                                              uint8_t *rowtype, const LevelSet &ls, int i, int j, int k) {
  const size_t n = b.n(), c = split ? b.at(split_pos(i, b.nx), j, k) : b.at(i, j, k);
  const size_t cr = b.at(i, j, k);
  const int I = i + 1, J = j + 1, K = k + 1;
  const size_t t = g.at(I, J, K);
  const bool dof = is_dof_cell(g, nvert, I, J, K);
  if (nvert[t] > 0.1 && dof) {  // identity row, poisson.c:1158-1160
    for (int s = 0; s < NSLOT; s++) A[s * n + c] = s == CP ? 1.0 : 0.0;
    rowtype[cr] = 2;
    return;
  }
  if (nvert[t] > kThr) {
    for (int s = 0; s < NSLOT; s++) A[s * n + c] = 0.0;
    rowtype[cr] = 0;
    return;
  }
  double v[NSLOT];
  assemble_row(g, nvert, m, I, J, K, v, ls);
  if (scale) {
    double a = m.aj[t];
    for (int s = 0; s < NSLOT; s++) v[s] *= a;
  }
  for (int s = 0; s < NSLOT; s++) {
    int di, dj, dk;
    slot_offset(s, di, dj, dk);
    bool keep = s == CP || (has_dof(g, nvert, I + di, J + dj, K + dk) && (!filter || fabs(v[s]) > 1.e-10));
    A[s * n + c] = keep ? v[s] : 0.0;
  }
  rowtype[cr] = 1;
}
__global__ void k_assemble(Grid g, Box b, const double *__restrict__ nvert, MetricPtrs m, int scale,
                           int filter, int split, double *A, uint8_t *rowtype, LevelSet ls) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= b.nx) return;
  assemble_cell(g, b, nvert, m, scale, filter, split, A, rowtype, ls, i, j, k);
}
// the same rows, only those listed (natural box indices rows[0 .. *nrows))
__global__ void k_assemble_rows(Grid g, Box b, const double *__restrict__ nvert, MetricPtrs m, int scale,
                                int filter, int split, double *A, uint8_t *rowtype, LevelSet ls,
                                const int *__restrict__ rows, const int *__restrict__ nrows) {
  const int nr = *nrows;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nr; w += gridDim.x * blockDim.x) {
    int i, j, k;
    box_ijk(b, (size_t)rows[w], i, j, k);
    assemble_cell(g, b, nvert, m, scale, filter, split, A, rowtype, ls, i, j, k);
  }
}

// The fine level's two assemblies from one evaluation of each row: the
// unscaled operator with the reference's insertion filter in the natural
// layout (A0, the FGMRES operator: k_assemble scale 0, filter 1, split 0)
// and the aj-scaled one without the filter in the parity-split layout (A1,
// the finest multigrid level: scale 1, filter 0, split 1); the same values
// as the two k_assemble passes.
__device__ __forceinline__ void assemble_fine_cell(const Grid &g, const Box &b, const double *__restrict__ nvert,
                                                   const MetricPtrs &m, double *A0, uint8_t *rowtype0, double *A1,
                                                   uint8_t *rowtype1, const LevelSet &ls, int i, int j, int k) {
  const size_t n = b.n(), c0 = b.at(i, j, k), c1 = b.at(split_pos(i, b.nx), j, k);
  const int I = i + 1, J = j + 1, K = k + 1;
  const size_t t = g.at(I, J, K);
  const bool dof = is_dof_cell(g, nvert, I, J, K);
  if ((nvert[t] > 0.1 && dof) || nvert[t] > kThr) {  // identity row (poisson.c:1158-1160) or no row
    const bool ident = nvert[t] > 0.1 && dof;
    for (int s = 0; s < NSLOT; s++) {
      const double v = ident && s == CP ? 1.0 : 0.0;
      A0[s * n + c0] = v;
      A1[s * n + c1] = v;
    }
    rowtype0[c0] = rowtype1[c0] = ident ? 2 : 0;
    return;
  }
  double v[NSLOT];
  assemble_row(g, nvert, m, I, J, K, v, ls);
  const double a = m.aj[t];
  for (int s = 0; s < NSLOT; s++) {
    int di, dj, dk;
    slot_offset(s, di, dj, dk);
    const bool col = s == CP || has_dof(g, nvert, I + di, J + dj, K + dk);
    A0[s * n + c0] = col && (s == CP || fabs(v[s]) > 1.e-10) ? v[s] : 0.0;
    A1[s * n + c1] = col ? v[s] * a : 0.0;
  }
  rowtype0[c0] = rowtype1[c0] = 1;
}
__global__ void k_assemble_fine(Grid g, Box b, const double *__restrict__ nvert, MetricPtrs m, double *A0,
                                uint8_t *rowtype0, double *A1, uint8_t *rowtype1, LevelSet ls) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= b.nx) return;
  assemble_fine_cell(g, b, nvert, m, A0, rowtype0, A1, rowtype1, ls, i, j, k);
}
// the same rows, only those listed (natural box indices rows[0 .. *nrows))
__global__ void k_assemble_fine_rows(Grid g, Box b, const double *__restrict__ nvert, MetricPtrs m, double *A0,
                                     uint8_t *rowtype0, double *A1, uint8_t *rowtype1, LevelSet ls,
                                     const int *__restrict__ rows, const int *__restrict__ nrows) {
  const int nr = *nrows;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nr; w += gridDim.x * blockDim.x) {
    int i, j, k;
    box_ijk(b, (size_t)rows[w], i, j, k);
    assemble_fine_cell(g, b, nvert, m, A0, rowtype0, A1, rowtype1, ls, i, j, k);
  }
}

// near[c]: some nvert within one point of cell c, or a periodic ghost's
// partner, has other bits than +0.  Elsewhere every sum of nvert is 0, every
// test of it is decided and every neighbour inside the box is a dof, so the
// kernels that follow the reference's blanking tests need no FP64 comparison
// there.  Formed once per mask from integer loads.
__device__ __forceinline__ bool nonzero_point(const Grid &g, const double *__restrict__ nvert, int i, int j, int k) {
  int a, b, c, fi, fj, fk;
  bool f = __double_as_longlong(nvert[g.at(i, j, k)]) != 0;
  if (g.remap(i, j, k, a, b, c, fi, fj, fk)) f |= __double_as_longlong(nvert[g.at(a, b, c)]) != 0;
  return f;
}
// a block takes 126 cells of a row: one thread per column ORs its 3 x 3
// points, the row's neighbours join in shared memory
__global__ void __launch_bounds__(128) k_near_body(Grid g, Box b, const double *__restrict__ nvert, uint8_t *near) {
  __shared__ uint8_t col[128];
  const int i = blockIdx.x * 126 + threadIdx.x, j = blockIdx.y + 1, k = blockIdx.z + 1;  // (DA indices)
  bool f = false;
  if (i < g.mx)
    for (int q = 0; q < 9; q++) f |= nonzero_point(g, nvert, i, j + q % 3 - 1, k + q / 3 - 1);
  col[threadIdx.x] = f;
  __syncthreads();
  const int x = threadIdx.x;
  if (x >= 1 && x < 127 && i < g.mx - 1) near[b.at(i - 1, j - 1, k - 1)] = col[x - 1] | col[x] | col[x + 1];
}
__global__ void k_near_body_rows(Grid g, Box b, const double *__restrict__ nvert, uint8_t *near,
                                 const int *__restrict__ rows, const int *__restrict__ nrows) {
  const int nr = *nrows;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nr; w += gridDim.x * blockDim.x) {
    int i, j, k;
    box_ijk(b, (size_t)rows[w], i, j, k);
    bool f = false;
    for (int q = 0; q < 27; q++) f |= nonzero_point(g, nvert, i + q % 3, j + (q / 3) % 3, k + q / 9);
    near[rows[w]] = f;
  }
}

// ---- incremental refill of the finest level on a new mask ----
// A row of the operator reads nvert within one point of its own (the
// one-sided differences and the neighbours' dof tests), where a periodic
// ghost neighbour's dof test reads its interior partner.  The rows to refill
// are those within two points of a point whose value changed, the periodic
// partners of ghost points included; every other row is the same as before.
// The changed points as bits, a word of 32 along i per warp (wpr words a row):
// dilating bits costs 1/8 of a byte a point and touches 32 at once (the three
// byte passes this replaces took 0.70 ms at 384x192x384, k_list_rows 0.024 ms).
// A ghost of a periodic i axis stands for its partner too.  src (the caller's
// mask) is copied to nvert on the way when they differ.
__global__ void __launch_bounds__(256) k_changed_bits(Grid g, int wpr, const double *src, double *nvert,
                                                      const double *__restrict__ prev, uint32_t *bits) {
  const int rows = g.my * g.mz, lane = threadIdx.x & 31;
  const long long *a = (const long long *)src, *p = (const long long *)prev;
  for (int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < rows * wpr; w += (gridDim.x * blockDim.x) >> 5) {
    const int row = w / wpr, i = (w - row * wpr) * 32 + lane;
    bool f = false;
    if (i < g.mx) {
      const size_t r = (size_t)row * g.mx, t = r + i;
      const long long v = a[t];
      f = v != p[t];
      if (src != nvert) ((long long *)nvert)[t] = v;
      if (g.px && i == 0) f |= a[r + g.mx - 2] != p[r + g.mx - 2];
      if (g.px && i == g.mx - 1) f |= a[r + 1] != p[r + 1];
    }
    const uint32_t m = __ballot_sync(0xffffffffu, f);
    if (lane == 0) bits[w] = m;
  }
}
// the interior rows within two points of a changed one along each axis
// (natural box indices, in no order), a ghost row of a periodic axis also
// standing for its partner, and the j-columns that hold one: a thread a word
__global__ void __launch_bounds__(256) k_list_rows(Grid g, Box b, int wpr, const uint32_t *__restrict__ bits,
                                                   int *rows, int *nrows, uint8_t *colflag) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x, total = b.ny * b.nz * wpr;
  uint32_t out = 0;
  int x = 0, j = 0, k = 0;
  if (w < total) {
    const int r = w / wpr;
    x = w - r * wpr;
    k = r / b.ny;
    j = r - k * b.ny + 1;
    k++;
    uint32_t L = 0, C = 0, R = 0;
    auto row = [&](int jj, int kk) {
      const uint32_t *q = bits + ((size_t)kk * g.my + jj) * wpr + x;
      C |= q[0];
      if (x > 0) L |= q[-1];
      if (x < wpr - 1) R |= q[1];
    };
    auto plane = [&](int kk) {
      for (int d = -2; d <= 2; d++) {
        const int q = min(max(j + d, 0), g.my - 1);
        row(q, kk);
        if (g.py && (q == 0 || q == g.my - 1)) row(q ? 1 : g.my - 2, kk);
      }
    };
    for (int d = -2; d <= 2; d++) {
      const int q = min(max(k + d, 0), g.mz - 1);
      plane(q);
      if (g.pz && (q == 0 || q == g.mz - 1)) plane(q ? 1 : g.mz - 2);
    }
    out = C | C << 1 | C << 2 | C >> 1 | C >> 2 | L >> 31 | L >> 30 | R << 31 | R << 30;
    const int first = x * 32;  // interior points 1 .. mx - 2 only
    if (first == 0) out &= ~1u;
    const int last = g.mx - 2 - first;
    if (last < 31) out &= last < 0 ? 0u : (2u << last) - 1u;
  }
  const int lane = threadIdx.x & 31, mine = __popc(out);
  int inc = mine;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  int at = 0;
  if (lane == 31 && inc) at = atomicAdd(nrows, inc);
  at = __shfl_sync(0xffffffffu, at, 31) + inc - mine;
  while (out) {
    const int i = x * 32 + __ffs(out) - 2;  // box index
    out &= out - 1;
    rows[at++] = (int)b.at(i, j - 1, k - 1);
    colflag[(size_t)(k - 1) * b.nx + i] = 1;
  }
}

// Per-face dot products S = a.b of the projection and the face aj, so that
// Projection can form (dpdc*S)*aj exactly as poisson.c:2828-2950 does.
__global__ void k_projection_coef(Grid g, Box b, MetricPtrs m, double *pc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= b.nx) return;
  size_t c = b.at(i, j, k), n = b.n(), s = g.at(i + 1, j + 1, k + 1);
#define DOT(A, B) (m.A[s * 3] * m.B[s * 3] + m.A[s * 3 + 1] * m.B[s * 3 + 1] + m.A[s * 3 + 2] * m.B[s * 3 + 2])
  pc[0 * n + c] = DOT(icsi, icsi); pc[1 * n + c] = DOT(ieta, icsi); pc[2 * n + c] = DOT(izet, icsi);
  pc[3 * n + c] = m.iaj[s];
  pc[4 * n + c] = DOT(jcsi, jeta); pc[5 * n + c] = DOT(jeta, jeta); pc[6 * n + c] = DOT(jzet, jeta);
  pc[7 * n + c] = m.jaj[s];
  pc[8 * n + c] = DOT(kcsi, kzet); pc[9 * n + c] = DOT(keta, kzet); pc[10 * n + c] = DOT(kzet, kzet);
  pc[11 * n + c] = m.kaj[s];
#undef DOT
}

// Box-layout masks of a level: row-active flag from the assembly, blanking
// (nvert > 0.1) and the restriction weight max(0, 1 - nvert)
// (MyRestriction, poisson.c:433-441), in both precisions.
__device__ __forceinline__ void level_mask_cell(const Grid &g, const Box &b, const double *nvert, uint8_t *blank,
                                                double *w64, float *w32, size_t c) {
  int i, j, k;
  box_ijk(b, c, i, j, k);
  double nv = nvert[g.at(i + 1, j + 1, k + 1)];
  double w = 1 - nv > 0. ? 1 - nv : 0.;
  blank[c] = nv > 0.1 ? 1 : 0;
  w64[c] = w;
  w32[c] = (float)w;
}
__global__ void k_level_masks(Grid g, Box b, const double *nvert, uint8_t *blank, double *w64, float *w32) {
  size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c < b.n()) level_mask_cell(g, b, nvert, blank, w64, w32, c);
}
// of the listed rows (the others' nvert is what it was)
__global__ void k_level_masks_rows(Grid g, Box b, const double *nvert, uint8_t *blank, double *w64, float *w32,
                                   const int *__restrict__ rows, const int *__restrict__ nrows) {
  const int nr = *nrows;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nr; w += gridDim.x * blockDim.x)
    level_mask_cell(g, b, nvert, blank, w64, w32, rows[w]);
}

// --------------------------------------------------------------------------
// Right-hand side: PoissonRHS2_hypre (Source/poisson_hypre.c:265-407) and
// Remove_Nullspace_Scale (:118-200)
// --------------------------------------------------------------------------
// The fluid test is the mask's byte plane and the sum of aj over the fluid,
// which the mask alone decides, is formed with it (k_fluid_mask): 7 FP64
// instructions per cell (the pipe that bounds this kernel) and 33 bytes,
// against 10 and 48.  256x192x256: 0.18 ms (0.26 ms before; at 40 registers
// the fixed grid did not fit the SMs in one wave).
__global__ void __launch_bounds__(256, 8) k_rhs(Grid g, Box b, const uint8_t *__restrict__ fluid,
                                                const double *__restrict__ ucont, double dt, double st, double coeff,
                                                double *__restrict__ rhs, double *partial) {
  pdl_trigger();
  pdl_wait();
  double sb = 0;
  const size_t n = b.n();
  const double f = -1.0 / dt * st * coeff;  // the reference's factor, formed once
  const int sj = 3 * g.mx, sk = 3 * g.mx * g.my;
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    double val = 0.;
    int i, j, k;
    box_ijk(b, c, i, j, k);
    const double *__restrict__ u = ucont + g.at(i + 1, j + 1, k + 1) * 3;
    // (loaded with the byte, not after it)
    const bool on = fluid[c];
    const double u0 = u[0], u1 = u[1], u2 = u[2], x0 = u[i == 0 && g.px ? 3 * (b.nx - 1) : -3],
                 y0 = u[1 + (j == 0 && g.py ? (b.ny - 1) * sj : -sj)],
                 z0 = u[2 + (k == 0 && g.pz ? (ptrdiff_t)(b.nz - 1) * sk : -(ptrdiff_t)sk)];
    if (on) {
      // (0 - U_i) + U_{i-1} as one subtraction: the same value
      val = x0 - u0;
      val -= u1;
      val += y0;
      val -= u2;
      val += z0;
      val *= f;
      sb += val;
    }
    rhs[c] = val;
  }
  const double tb = block_sum(sb);
  if (threadIdx.x == 0) partial[blockIdx.x] = tb;
}

// PoissonRHS2 (Source/poisson.c:1780-1906), the -poisson 0 / -1 variant:
// the same divergence on fluid cells, 0 on identity-row dofs, the aj row
// scaling for poisson == -1; block partials of the sum over every dof entry
// and of the fluid count for the unweighted mean removal.
__global__ void k_rhs2(Grid g, Box b, const double *__restrict__ nvert, const uint8_t *__restrict__ rowtype,
                       const double *__restrict__ ucont, const double *__restrict__ aj, double dt, double st,
                       double coeff, int poisson, double *rhs, double *partial) {
  double sb = 0, cnt = 0;
  const size_t n = b.n();
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    box_ijk(b, c, i, j, k);
    i++; j++; k++;
    size_t t = g.at(i, j, k);
    double val = 0.;
    if (nvert[t] < 0.1) {
#define U(a, bb, cc, q) ucont[g.at(a, bb, cc) * 3 + (q)]
      val -= U(i, j, k, 0);
      if (i == 1 && g.px) val += U(g.mx - 2, j, k, 0);
      else val += U(i - 1, j, k, 0);
      val -= U(i, j, k, 1);
      if (j == 1 && g.py) val += U(i, g.my - 2, k, 1);
      else val += U(i, j - 1, k, 1);
      val -= U(i, j, k, 2);
      if (k == 1 && g.pz) val += U(i, j, g.mz - 2, 2);
      else val += U(i, j, k - 1, 2);
#undef U
      val *= -1.0 / dt * st * coeff;
      if (poisson == -1) val *= aj[t];
      cnt += 1.;
    }
    if (rowtype[c]) sb += val;
    rhs[c] = val;
  }
  double tb = block_sum(sb);
  double tc = block_sum(cnt);
  if (threadIdx.x == 0) { partial[blockIdx.x] = tb; partial[gridDim.x + blockIdx.x] = tc; }
}
// the unweighted shift of PoissonRHS2 on fluid cells; for poisson == -1 the
// solver's (unscaled) right-hand side is B / aj on those rows
__global__ void k_rhs2_shift(Grid g, Box b, const double *__restrict__ nvert, const double *__restrict__ aj,
                             const double *sums, int poisson, double *rhs) {
  const double val = -sums[0] / (sums[1] > 0. ? sums[1] : 1.);
  const size_t n = b.n();
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    box_ijk(b, c, i, j, k);
    i++; j++; k++;
    size_t t = g.at(i, j, k);
    if (nvert[t] < 0.1) {
      rhs[c] += val;
      if (poisson == -1) rhs[c] = rhs[c] / aj[t];
    }
  }
}

// sums row blockIdx.x of `nb` block partials in a fixed tree order (launch
// one block per row)
__global__ void k_reduce_rows(const double *partial, int nb, int nrow, double *out) {
  pdl_trigger();
  pdl_wait();
  const int r = blockIdx.x;
  if (r >= nrow) return;
  double s = 0;
  for (int q = threadIdx.x; q < nb; q += blockDim.x) s += partial[(size_t)r * nb + q];
  s = block_sum(s);
  if (threadIdx.x == 0) out[r] = s;
}

// The reference's quotients by one divisor, correctly rounded (the bits of the
// division) without a division: with y = RN(1 / d) and a start q within 1 ulp
// of a / d, Markstein's correction RN(q + RN(a - q d) y), its remainder exact,
// is the correctly rounded quotient (P. Markstein, IBM J. Res. Dev. 34 (1990)
// 111-119).  Two starts reach 1 ulp:
//   RN(a y)             when delta = 1 - d y (exact by FMA) is at most 2^-54:
//                       a/d delta is then below half an ulp, and so is the rounding
//                       (three operations in all; 2^-54 holds for 1.5 and 3);
//   RN(a y + RN(a yl))  with yl = RN(delta y), the reciprocal's rest (1 / d to
//                       about 2^-105): the quotient to just over half an ulp (four).
// The remainder must not leave the normal range: the callers look at the numerator's
// exponent (k_rhs_nullspace at that of its factors, once for all cells).
__device__ __forceinline__ double markstein3(double a, double d, double y) {
  const double q = a * y;
  return fma(fma(-q, d, a), y, q);
}
__device__ __forceinline__ double markstein4(double a, double d, double y, double yl) {
  const double q = fma(a, y, a * yl);
  return fma(fma(-q, d, a), y, q);
}

// 256x192x256: 0.135 ms (0.196 with five operations and loads behind the byte's;
// the five operations left are 0.11 ms of the FP64 pipe).  Sums within 2^+-300
// keep numerator, quotient and remainder in the normal range for every aj down to
// 2^-400 (below, a quotient may be off in its last bit); other ones, infinities
// and NaN take the division.  A zero sum leaves rhs as it is (its quotients are -0).
__global__ void __launch_bounds__(256, 8) k_rhs_nullspace(Box b, const uint8_t *__restrict__ fluid,
                                                          const double *__restrict__ aj_box, const double *sums,
                                                          const double *fsum, double *__restrict__ rhs) {
  pdl_trigger();
  pdl_wait();
  const double sum = sums[0], sum_aj = fsum[0], y = 1.0 / sum_aj, delta = fma(-sum_aj, y, 1.0), yl = delta * y;
  const int es = (__double2hiint(sum) >> 20) & 0x7ff, ea = (__double2hiint(sum_aj) >> 20) & 0x7ff;
  const bool in = ea > 723 && ea < 1323, fast = in && es > 723 && es < 1323, three = fabs(delta) <= 0x1p-54;
  const size_t n = in && sum == 0. ? 0 : b.n();
  auto shift = [&](auto quotient_of) {
#pragma unroll 4
    for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
      const bool f = fluid[c];
      const double aj = aj_box[c], r = rhs[c];
      if (f) rhs[c] = r + quotient_of(-sum * aj);
    }
  };
  // (three loops: a choice inside one is computed all three ways)
  if (!fast) shift([&](double a) { return a / sum_aj; });
  else if (three) shift([&](double a) { return markstein3(a, sum_aj, y); });
  else shift([&](double a) { return markstein4(a, sum_aj, y, yl); });
}

// FullyBlocked (Source/poisson.c:1909-1993): per interior (i, j) column the
// first k (boundary layers included) with nvert > 0.1 into ksk[j mx + i]
// (-1 for none and on the boundary columns), and the count of interior
// columns without one (the multiple-null-space flag is that count == 0).
__global__ void k_fully_blocked(Grid g, const double *__restrict__ nvert, int *ksk, int *unblocked) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
  if (i >= g.mx) return;
  int first = -1;
  if (i >= 1 && i < g.mx - 1 && j >= 1 && j < g.my - 1) {
    for (int k = 0; k < g.mz; k++)
      if (nvert[g.at(i, j, k)] > 0.1) { first = k; break; }
    if (first < 0) atomicAdd(unblocked, 1);
  }
  ksk[(size_t)j * g.mx + i] = first;
}

// PoissonNullSpaceFunction_original (Source/poisson.c:757-943), first pass:
// block partials over the interior cells with nvert < 0.1 of the sum of x
// and the count, one pair of rows per region (multi: k below the column's
// first blocked k, then k at or above it; else the whole interior).
__global__ void k_nullspace_sums(Grid g, const double *__restrict__ nvert, const int *__restrict__ ksk, int multi,
                                 const double *__restrict__ x, double *partial) {
  double s[2] = {0., 0.}, c[2] = {0., 0.};
  const size_t n = (size_t)(g.mx - 2) * (g.my - 2) * (g.mz - 2);
  for (size_t q = (size_t)blockIdx.x * blockDim.x + threadIdx.x; q < n; q += (size_t)gridDim.x * blockDim.x) {
    const int i = 1 + (int)(q % (size_t)(g.mx - 2));
    const size_t r = q / (size_t)(g.mx - 2);
    const int j = 1 + (int)(r % (size_t)(g.my - 2)), k = 1 + (int)(r / (size_t)(g.my - 2));
    const size_t t = g.at(i, j, k);
    if (!(nvert[t] < 0.1)) continue;
    const int reg = multi && k >= ksk[(size_t)j * g.mx + i] ? 1 : 0;
    s[reg] += x[t];
    c[reg] += 1.;
  }
  for (int q = 0; q < 4; q++) {
    const double v = block_sum(q == 0 ? s[0] : q == 1 ? c[0] : q == 2 ? s[1] : c[1]);
    if (threadIdx.x == 0) partial[(size_t)q * gridDim.x + blockIdx.x] = v;
  }
}
// second pass: x += shift of its region on the interior cells with nvert <
// 0.1; the boundary layers and the cells with nvert > 0.1 become 0
__global__ void k_nullspace_apply(Grid g, const double *__restrict__ nvert, const int *__restrict__ ksk, int multi,
                                  double shift0, double shift1, double *x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= g.mx) return;
  const size_t t = g.at(i, j, k);
  const bool bnd = i == 0 || i == g.mx - 1 || j == 0 || j == g.my - 1 || k == 0 || k == g.mz - 1;
  const double nv = nvert[t];
  if (!bnd && nv < 0.1) x[t] += multi && k >= ksk[(size_t)j * g.mx + i] ? shift1 : shift0;
  if (bnd || nv > 0.1) x[t] = 0.;
}

// Remove_Nullspace (Source/poisson_hypre.c:202-263) on a box vector: sum and
// count over nvert < 0.1
__global__ void __launch_bounds__(256, 8) k_mean_partial(size_t n, const uint8_t *__restrict__ fluid,
                                                         const double *__restrict__ x, double *partial) {
  pdl_trigger();
  pdl_wait();
  double s = 0;
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x)
    if (fluid[c]) s += x[c];
  const double ts = block_sum(s);
  if (threadIdx.x == 0) partial[blockIdx.x] = ts;
}
// The fluid mask of a new nvert (nvert < 0.1), aj at the box cells, and the
// block partials of what the mask alone decides: the sum of aj over the
// fluid cells (row 0, Remove_Nullspace_Scale's sum_aj) and their count (row
// 1, Remove_Nullspace's).
__global__ void __launch_bounds__(256, 8) k_fluid_mask(Grid g, Box b, const double *__restrict__ nvert,
                                                       const double *__restrict__ aj, uint8_t *__restrict__ fluid,
                                                       double *__restrict__ aj_box, double *partial) {
  double sa = 0;
  int cnt = 0;
  const size_t n = b.n();
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    box_ijk(b, c, i, j, k);
    const size_t t = g.at(i + 1, j + 1, k + 1);
    const bool f = nvert[t] < 0.1;
    const double a = aj[t];
    fluid[c] = f ? 1 : 0;
    aj_box[c] = a;
    if (f) sa += a;
    cnt += f ? 1 : 0;
  }
  const double ta = block_sum(sa);
  const int tc = block_sum(cnt);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = ta;
    partial[gridDim.x + blockIdx.x] = (double)tc;
  }
}

// the same after a new mask that changed the listed rows only: their fluid
// bytes, then the sums from the byte and aj planes (9 bytes a cell for 33, in
// the same order)
__global__ void k_fluid_rows(Grid g, Box b, const double *__restrict__ nvert, uint8_t *fluid,
                             const int *__restrict__ rows, const int *__restrict__ nrows) {
  const int nr = *nrows;
  for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < nr; w += gridDim.x * blockDim.x) {
    int i, j, k;
    box_ijk(b, (size_t)rows[w], i, j, k);
    fluid[rows[w]] = nvert[g.at(i + 1, j + 1, k + 1)] < 0.1 ? 1 : 0;
  }
}
__global__ void __launch_bounds__(256, 8) k_fluid_sums(size_t n, const uint8_t *__restrict__ fluid,
                                                       const double *__restrict__ aj_box, double *partial) {
  double sa = 0;
  int cnt = 0;
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    const bool f = fluid[c];
    const double a = aj_box[c];
    if (f) sa += a;
    cnt += f ? 1 : 0;
  }
  const double ta = block_sum(sa);
  const int tc = block_sum(cnt);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = ta;
    partial[gridDim.x + blockIdx.x] = (double)tc;
  }
}

// Remove_Nullspace's shift, -sum / count, from the block partials of the
// fluid sum (in k_reduce_rows' order) and the mask's count; one block
__global__ void k_mean_shift(const double *partial, int nb, const double *fsum, double *shift) {
  pdl_trigger();
  pdl_wait();
  double s = 0;
  for (int q = threadIdx.x; q < nb; q += blockDim.x) s += partial[q];
  s = block_sum(s);
  if (threadIdx.x == 0) *shift = -s / fsum[1];
}

// Convert_Phi2_Phi (Source/poisson.c:98-186): box phi -> DA phi, zero on
// non-dof cells and non-periodic ghosts, partner values on periodic ghosts.
// With `shift` (device, one value), Remove_Nullspace's x += shift on the
// fluid cells (nvert < 0.1) is applied on the way (x itself is left as is).
// One thread per point in linear order (a row of 258 points would leave the
// third block of a row-wise launch nearly empty), the dof and fluid tests from
// byte planes: 18 bytes per point, 26 with the caller's copy (out).
__global__ void __launch_bounds__(256) k_box_to_da_phi(Grid g, Box b, const uint8_t *__restrict__ rowtype,
                                                       const uint8_t *__restrict__ fluid,
                                                       const double *__restrict__ x, double *__restrict__ phi,
                                                       const double *shift, double *__restrict__ out) {
  pdl_trigger();
  pdl_wait();
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.n()) return;
  int i, j, k, a, bb, c, fi, fj, fk;
  da_ijk(g, t, i, j, k);
  g.remap(i, j, k, a, bb, c, fi, fj, fk);
  double v = 0.;
  if (a >= 1 && a < g.mx - 1 && bb >= 1 && bb < g.my - 1 && c >= 1 && c < g.mz - 1) {
    const size_t q = b.at(a - 1, bb - 1, c - 1);
    if (rowtype[q]) {
      v = x[q];
      if (shift && fluid[q]) v += shift[0];
    }
  }
  phi[t] = v;
  if (out) out[t] = v;
}
// DA -> box copy of the interior (warm start / inspection input)
__global__ void k_da_to_box(Grid g, Box b, const double *da, double *x) {
  size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= b.n()) return;
  int i, j, k;
  box_ijk(b, c, i, j, k);
  i++; j++; k++;
  x[c] = da[g.at(i, j, k)];
}
__global__ void __launch_bounds__(256) k_box_to_da(Grid g, Box b, const double *__restrict__ x,
                                                   double *__restrict__ da) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.n()) return;
  int i, j, k;
  da_ijk(g, t, i, j, k);
  double v = 0.;
  if (i >= 1 && i < g.mx - 1 && j >= 1 && j < g.my - 1 && k >= 1 && k < g.mz - 1)
    v = x[b.at(i - 1, j - 1, k - 1)];
  da[t] = v;
}

// Periodic ghost points, one thread per point of the two boundary layers of
// each periodic axis (grid from shell_grid on the host: no pass over the
// whole array).  A point on the layers of two axes is visited twice with the
// same source, whose periodic coordinates all lie inside, so it is never a
// target.
__device__ __forceinline__ bool shell_point(const Grid &g, size_t q, int &i, int &j, int &k) {
  const uint32_t nx = g.px ? 2u * g.my * g.mz : 0u, ny = g.py ? 2u * g.mx * g.mz : 0u, nz = g.pz ? 2u * g.mx * g.my : 0u;
  uint32_t u = (uint32_t)q;
  if (u < nx) {
    i = (u & 1) ? g.mx - 1 : 0; u >>= 1;
    j = (int)(u % (uint32_t)g.my); k = (int)(u / (uint32_t)g.my);
    return true;
  }
  u -= nx;
  if (u < ny) {
    const uint32_t l = (uint32_t)g.mx * g.mz;
    j = u < l ? 0 : g.my - 1;
    if (u >= l) u -= l;
    i = (int)(u % (uint32_t)g.mx); k = (int)(u / (uint32_t)g.mx);
    return true;
  }
  u -= ny;
  if (u < nz) {
    const uint32_t l = (uint32_t)g.mx * g.my;
    k = u < l ? 0 : g.mz - 1;
    if (u >= l) u -= l;
    i = (int)(u % (uint32_t)g.mx); j = (int)(u / (uint32_t)g.mx);
    return true;
  }
  return false;
}
// UpdatePressure (Source/poisson.c:3137-3297): the interior update of p (in
// place) with phi copied to the handle's array on the way (phi_out; null when
// phi is that array), then the periodic ghosts of p and phi over the boundary
// layers alone.  One pass at its bytes (p in and out, phi in and out).
__global__ void __launch_bounds__(256) k_update_pressure(Grid g, const double *__restrict__ nvert,
                                                         const uint8_t *__restrict__ near,
                                                         const double *__restrict__ phi, double *__restrict__ p,
                                                         double *__restrict__ phi_out) {
  pdl_trigger();
  pdl_wait();
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= g.n()) return;
  int i, j, k;
  da_ijk(g, t, i, j, k);
  const double f = phi[t];
  if (phi_out) phi_out[t] = f;
  if (i < 1 || i >= g.mx - 1 || j < 1 || j >= g.my - 1 || k < 1 || k >= g.mz - 1) return;
  const size_t c = ((size_t)(k - 1) * (g.my - 2) + (j - 1)) * (g.mx - 2) + (i - 1);
  if (!near[c]) {
    p[t] += f;
    return;
  }
  if (nvert[t] < 0.1) p[t] += f;
  if (nvert[t] > 1.1) p[t] = 0;
}
__global__ void k_periodic_copy2(Grid g, double *p, double *phi, double *phi2) {
  pdl_trigger();
  pdl_wait();
  int i, j, k, a, b, c, fi, fj, fk;
  if (!shell_point(g, (size_t)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
  g.remap(i, j, k, a, b, c, fi, fj, fk);
  const size_t s = g.at(a, b, c), t = g.at(i, j, k);
  p[t] = p[s];
  phi[t] = phi[s];
  if (phi2) phi2[t] = phi2[s];
}

// Projection (Source/poisson.c:2700-3066).
// x * 2^-e (e = 1, 2) by the exponent field: the product's bits for results
// in the normal range, without an FP64 instruction (the FP64 pipe takes a
// warp's instruction over 16 cycles of the SM, an integer one over a quarter
// of a cycle); zeros, subnormals, infinities and NaN take the product.
__device__ __forceinline__ double scale_down(double x, int e) {
  const int hi = __double2hiint(x), ex = (hi >> 20) & 0x7ff;
  if (ex > e && ex < 0x7ff) return __hiloint2double(hi - (e << 20), __double2loint(x));
  return e == 1 ? x * 0.5 : x * 0.25;
}

// v * dt * st / coeff / r in the reference's left-to-right order.  A
// factor or divisor of exactly 1 leaves its operand unchanged, so those
// operations are skipped: the same bits.  The division by coeff is Markstein's
// (the quotient's bits in three or four operations) while quotient and
// remainders stay in the normal range.
template <bool LS>
__device__ __forceinline__ double proj_scale(double v, const ProjScale &ps, double r) {
  if (ps.ops & 1) v = v * ps.dt;
  if (ps.ops & 2) v = v * ps.st;
  if (ps.ops & 4) {
    const int ex = (__double2hiint(v) >> 20) & 0x7ff;
    if (ex > 200 && ex < 1900 && (ps.ops & 8))
      v = ps.ops & 16 ? markstein3(v, ps.coeff, ps.rcoeff) : markstein4(v, ps.coeff, ps.rcoeff, ps.rlow);
    else if ((ps.ops & 8) && ((__double2hiint(v) & 0x7fffffff) | __double2loint(v)) == 0)
      v = v * ps.rcoeff;  // a zero of the quotient's sign
    else
      v = v / ps.coeff;
  }
  if (LS && r != 1.0) v = v / r;
  return v;
}

// a + b against kThr and 5, without FP64 for the values masks hold (0, 1, 3:
// no two of them add up to 5)
struct MaskSum {
  bool above, below, five;
  __device__ MaskSum(double a, double b) {
    const int ha = __double2hiint(a), hb = __double2hiint(b);
    auto plain = [](int h) { return h == 0 || h == 0x3ff00000 || h == 0x40080000; };
    if ((__double2loint(a) | __double2loint(b)) == 0 && plain(ha) && plain(hb)) {
      above = (ha | hb) != 0;
      below = !above;
      five = false;
    } else {
      const double s = a + b;
      above = s > kThr;
      below = s < kThr;
      five = (int)s == 5;
    }
  }
};

// A tangential difference of a face (face offset f, tangential stride s):
// (P[t+op] + P[t+f+op] - P[t+om] - P[t+f+om]) 2^-e, central (op, om = s, -s;
// e = 2) or one-sided (op or om 0; e = 1); e = 0: none, the value 0.
struct Tangent {
  int op, om, e;
  // no nvert but 0 near the cell: only the box faces decide
  __device__ void plain(int c, int m, bool per, int s) {
    const bool top = c == m - 2 && !per, bot = c == 1 && !per;
    op = top ? 0 : s;
    om = bot && !top ? 0 : -s;
    e = top ? (c != 1 ? 1 : 0) : bot ? 1 : 2;
  }
  // the reference's tests (e.g. poisson.c:2773-2796), nv at the cell
  __device__ void masked(const double *__restrict__ nv, int f, int c, int m, bool per, int s) {
    const MaskSum np(nv[s], nv[f + s]), nm(nv[-s], nv[f - s]);
    op = s;
    om = -s;
    if ((c == m - 2 && !per) || np.above) {
      e = nm.below && c != 1 ? 1 : 0;
      op = 0;
    } else if ((c == 1 && !per) || nm.above) {
      e = np.below ? 1 : 0;
      om = 0;
    } else {
      e = 2;
    }
  }
  __device__ double diff(const double *__restrict__ P, int f) const {
    if (e == 0) return 0.;
    return scale_down(P[op] + P[f + op] - P[om] - P[f + om], e);
  }
};

// One thread per cell, its three upper faces (small boxes: one each); cells in linear order, so that
// no lane of the FP64 instructions idles on narrow boxes.  Bound by the FP64
// pipe (85 % busy, 69 instructions per cell with dt != 1 and coeff 1.5, of which
// the reference's roundings ask for 60; 78 with five for the quotient and FP64
// sums of the masks near bodies, about 150 with those everywhere: near says
// where they are needed).  256x192x256, dt != 1, coeff 1.5: 1.63 ms (1.83 and
// 3.42 ms before; the bytes alone would take 0.3 ms).
template <bool LS>
__device__ __forceinline__ void projection_body(Grid g, Box b, const double *__restrict__ nvert,
                                                const uint8_t *__restrict__ near, const double *__restrict__ phi,
                                                const double *__restrict__ pc, const ProjScale &ps, double *ucont,
                                                const MetricPtrs &m, const LevelSet &ls) {
  const size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x, n = b.n();
  if (c >= n) return;
  int i, j, k;
  box_ijk(b, c, i, j, k);
  i++; j++; k++;
  const int mx = g.mx, my = g.my, mz = g.mz;
  const bool ip = g.px, jp = g.py, kp = g.pz;
  const size_t t = g.at(i, j, k);
  const int sj = mx, sk = mx * my;
  const double *__restrict__ P = phi + t, *__restrict__ nv = nvert + t;
  double r1 = 1.0, r2 = 1.0, r3 = 1.0;
  if (LS) {  // poisson.c:2738-2749
    const double *rho = ls.rho;
    r1 = i == mx - 2 ? rho[t] : ls_mean(rho[t], rho[g.at(i + 1, j, k)]);
    r2 = j == my - 2 ? rho[t] : ls_mean(rho[t], rho[g.at(i, j + 1, k)]);
    r3 = k == mz - 2 ? rho[t] : ls_mean(rho[t], rho[g.at(i, j, k + 1)]);
  }
  const bool body = near[c];
  // a grid of three rows: a thread for each face (its loads and its chain of FP64
  // operations beside the other faces', where the SMs have room for them)
  const int faces = gridDim.y == 3 ? 1 << blockIdx.y : 7;
  Tangent a, e;
  if ((faces & 1) && (i < mx - 2 || ip)) {
    bool on = true;
    if (!body) {
      a.plain(j, my, jp, sj);
      e.plain(k, mz, kp, sk);
    } else {
      a.masked(nv, 1, j, my, jp, sj);
      e.masked(nv, 1, k, mz, kp, sk);
      on = MaskSum(nv[0], nv[1]).below;
    }
    if (on) {
      const double dpdc = P[i == mx - 2 ? 1 - i : 1] - P[0], dpde = a.diff(P, 1), dpdz = e.diff(P, 1);
      const double aj = pc[3 * n + c];
      ucont[t * 3 + 0] -= proj_scale<LS>(dpdc * pc[0 * n + c] * aj + dpde * pc[1 * n + c] * aj + dpdz * pc[2 * n + c] * aj,
                                         ps, r1);
    }
  }
  if ((faces & 2) && (j < my - 2 || jp || (LS && ls.bc3 == 4))) {
    bool on = true;
    if (!body) {
      a.plain(i, mx, ip, 1);
      e.plain(k, mz, kp, sk);
    } else {
      a.masked(nv, sj, i, mx, ip, 1);
      e.masked(nv, sj, k, mz, kp, sk);
      const MaskSum s(nv[0], nv[sj]);
      on = s.below || s.five;
    }
    if (on) {
      const double dpde = LS && ls.bc3 == 4 && j == my - 2 ? P[0] - P[-sj]
                                                           : P[j == my - 2 && jp ? (1 - j) * sj : sj] - P[0];
      const double dpdc = a.diff(P, sj), dpdz = e.diff(P, sj);
      const double aj = pc[7 * n + c];
      ucont[t * 3 + 1] -= proj_scale<LS>(dpdc * pc[4 * n + c] * aj + dpde * pc[5 * n + c] * aj + dpdz * pc[6 * n + c] * aj,
                                         ps, r2);
    }
  }
  if ((faces & 4) && (k < mz - 2 || kp || (LS && ls.bc5 == 4))) {
    bool on = true;
    if (!body) {
      a.plain(i, mx, ip, 1);
      e.plain(j, my, jp, sj);
    } else {
      a.masked(nv, sk, i, mx, ip, 1);
      e.masked(nv, sk, j, my, jp, sj);
      on = MaskSum(nv[0], nv[sk]).below;
    }
    if (on) {
      double dpdz;
      if (k == mz - 2 && kp) dpdz = P[(ptrdiff_t)(1 - k) * sk] - P[0];
      else if (LS && k == mz - 2 && ls.bc5 == 4) dpdz = P[0] - P[-sk];
      else dpdz = P[sk] - P[0];
      const double dpdc = a.diff(P, sk), dpde = e.diff(P, sk);
      const double aj = pc[11 * n + c];
      ucont[t * 3 + 2] -= proj_scale<LS>(dpdc * pc[8 * n + c] * aj + dpde * pc[9 * n + c] * aj + dpdz * pc[10 * n + c] * aj,
                                         ps, r3);
      if (LS && k == 1 && ls.bc4 == 5000 && ls.level[t] < 0) {  // poisson.c:2951-2956
        const size_t t0 = g.at(i, j, 0);
        const double *kz = &m.kzet[t0 * 3];
        ucont[t0 * 3 + 2] -= proj_scale<LS>(dpdz * (kz[0] * kz[0] + kz[1] * kz[1] + kz[2] * kz[2]) * m.kaj[t0], ps,
                                            ls.rho[t]);
      }
    }
  }
}
__global__ void __launch_bounds__(256) k_projection(Grid g, Box b, const double *nvert, const uint8_t *near,
                                                    const double *phi, const double *pc, ProjScale ps, double *ucont,
                                                    MetricPtrs m) {
  pdl_trigger();
  pdl_wait();
  projection_body<false>(g, b, nvert, near, phi, pc, ps, ucont, m, LevelSet{});
}
__global__ void __launch_bounds__(256) k_projection_ls(Grid g, Box b, const double *nvert, const uint8_t *near,
                                                       const double *phi, const double *pc, ProjScale ps,
                                                       double *ucont, MetricPtrs m, LevelSet ls) {
  pdl_trigger();
  pdl_wait();
  projection_body<true>(g, b, nvert, near, phi, pc, ps, ucont, m, ls);
}

// periodic face copy of Ucont (poisson.c:2996-3036)
__global__ void k_periodic_faces(Grid g, double *ucont) {
  pdl_trigger();
  pdl_wait();
  int i, j, k, a, b, c, fi, fj, fk;
  if (!shell_point(g, (size_t)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
  g.remap(i, j, k, a, b, c, fi, fj, fk);
  const size_t s = g.at(a, b, c), t = g.at(i, j, k);
  if (fi) ucont[t * 3 + 0] = ucont[s * 3 + 0];
  if (fj) ucont[t * 3 + 1] = ucont[s * 3 + 1];
  if (fk) ucont[t * 3 + 2] = ucont[s * 3 + 2];
}

// Divergence (Source/main.c:936-1074): block maxima of |div(Ucont) aj|.
// The seven-point blanking sum is formed only near a body; the running
// maximum compares bit patterns (non-negative doubles order like integers),
// leaving the difference and the product, six FP64 instructions per cell
// (256x192x256: 0.21 ms, 0.37 ms before; eight blocks per SM, so that the
// fixed grid is one wave: at 40 registers the sixth block of eight waited for
// a second one).  A NaN is passed over, as the comparison v > best passes it
// over.
__global__ void __launch_bounds__(256, 8) k_divergence(Grid g, Box b, const double *__restrict__ nvert, const uint8_t *__restrict__ near,
                             const double *__restrict__ ucont, const double *__restrict__ aj, double *partial) {
  pdl_trigger();
  pdl_wait();
  long long best = 0;
  const size_t n = b.n();
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    int i, j, k;
    box_ijk(b, c, i, j, k);
    i++; j++; k++;
    double v;
    if (near[c]) {
      v = divergence_cell(g, nvert, ucont, aj, i, j, k);
    } else {
      const size_t t = g.at(i, j, k);
      const double *__restrict__ u = ucont + t * 3;
      v = fabs((u[0] - u[-3] + u[1] - u[1 - 3 * (ptrdiff_t)g.mx] + u[2] - u[2 - 3 * (ptrdiff_t)g.mx * g.my]) * aj[t]);
    }
    const long long w = __double_as_longlong(v);
    if (w <= 0x7ff0000000000000ll && w > best) best = w;
  }
  double m = block_max(__longlong_as_double(best));
  if (threadIdx.x == 0) partial[blockIdx.x] = m;
}
__global__ void k_reduce_max(const double *partial, int nb, double *out) {
  pdl_trigger();
  pdl_wait();
  double m = 0.;
  for (int q = threadIdx.x; q < nb; q += blockDim.x) m = partial[q] > m ? partial[q] : m;
  m = block_max(m);
  if (threadIdx.x == 0) *out = m;
}

// --------------------------------------------------------------------------
// Multigrid hierarchy set-up and transfer operators
// --------------------------------------------------------------------------
// coarse nodes are every other fine node (Source/init.c:402-455 with
// GridRestriction, poisson.c:337-363)
__global__ void k_coarse_nodes(Grid gf, Grid gc, int cx, int cy, int cz, const double *cf, double *cc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= gc.mx) return;
  size_t t = gc.at(i, j, k);
  if (i > gc.mx - 2 || j > gc.my - 2 || k > gc.mz - 2) {
    cc[t * 3] = cc[t * 3 + 1] = cc[t * 3 + 2] = 0.;
    return;
  }
  size_t s = gf.at(cx ? 2 * i : i, cy ? 2 * j : j, cz ? 2 * k : k);
  cc[t * 3] = cf[s * 3]; cc[t * 3 + 1] = cf[s * 3 + 1]; cc[t * 3 + 2] = cf[s * 3 + 2];
}

// MyNvertRestriction (poisson.c:1995-2083), first pass: a coarse cell is
// blanked when the product of its children's nvert exceeds 0.1.
__global__ void k_nvert_restrict(Grid gh, Grid gc, int cx, int cy, int cz, const double *nh, double *nc) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
  if (i >= gc.mx || j >= gc.my) return;
  size_t t = gc.at(i, j, k);
  double v = 0.;
  if (i >= 1 && i < gc.mx - 1 && j >= 1 && j < gc.my - 1 && k >= 1 && k < gc.mz - 1) {
    const int ia = cx, ja = cy, ka = cz;
    int ih = cx ? 2 * i : i, jh = cy ? 2 * j : j, kh = cz ? 2 * k : k;
    const double q[8] = {nh[gh.at(ih, jh, kh)], nh[gh.at(ih - ia, jh, kh)], nh[gh.at(ih, jh - ja, kh)],
                         nh[gh.at(ih, jh, kh - ka)], nh[gh.at(ih - ia, jh - ja, kh)], nh[gh.at(ih - ia, jh, kh - ka)],
                         nh[gh.at(ih, jh - ja, kh - ka)], nh[gh.at(ih - ia, jh - ja, kh - ka)]};
    // (a zero among them decides without FP64: the product is 0, or NaN)
    bool any = true;
    for (int e = 0; e < 8; e++) any &= (__double_as_longlong(q[e]) << 1) != 0;
    if (any && q[0] * q[1] * q[2] * q[3] * q[4] * q[5] * q[6] * q[7] > 0.1) v = 1.;
  }
  nc[t] = v;
}
// second pass, isolated-cell fill.  The reference updates in place in k-j-i
// order; a cell is filled only when all six face neighbours are already
// blanked, so no fluid neighbour can change its decision and a parallel
// pass over a snapshot gives the same result.
__global__ void k_nvert_fill(Grid gc, const double *src, double *dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
  if (i >= gc.mx || j >= gc.my) return;
  size_t t = gc.at(i, j, k);
  // (src holds 0 and 1 only: a sum of two is above 1.1 when both are 1)
  const long long *q = (const long long *)src;
  double v = src[t];
  if (q[t] == 0 && i >= 1 && i < gc.mx - 1 && j >= 1 && j < gc.my - 1 && k >= 1 && k < gc.mz - 1) {
    if (q[gc.at(i + 1, j, k)] && q[gc.at(i - 1, j, k)] && q[gc.at(i, j + 1, k)] && q[gc.at(i, j - 1, k)] &&
        q[gc.at(i, j, k + 1)] && q[gc.at(i, j, k - 1)])
      v = 1.;
  }
  dst[t] = v;
}

// MyRestriction (poisson.c:365-472) on box vectors: the eight weighted
// children in the reference's order, times 1/8; zero on blanked coarse cells.
template <typename T>
__device__ __forceinline__ void restrict_body(Box bf, Box bc, int cx, int cy, int cz, const T *__restrict__ rf,
                                              const T *__restrict__ wf, const uint8_t *__restrict__ blank_c,
                                              T *bc_out) {
  pdl_trigger();
  pdl_wait();
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y * blockDim.y + threadIdx.y, k = blockIdx.z;
  if (i >= bc.nx || j >= bc.ny) return;
  size_t cc = bc.at(i, j, k);
  if (blank_c[cc]) { bc_out[cc] = (T)0; return; }
  int i1 = cx ? 2 * i + 1 : i, j1 = cy ? 2 * j + 1 : j, k1 = cz ? 2 * k + 1 : k;
  int i0 = i1 - cx, j0 = j1 - cy, k0 = k1 - cz;
#define X(a, b, c) (rf[bf.at(a, b, c)] * wf[bf.at(a, b, c)])
  T s = X(i1, j1, k1) + X(i0, j1, k1) + X(i1, j0, k1) + X(i1, j1, k0) + X(i0, j0, k1) + X(i1, j0, k0) +
        X(i0, j1, k0) + X(i0, j0, k0);
#undef X
  bc_out[cc] = (T)0.125 * s;
}

// MyInterpolation (poisson.c:527-670, GridInterpolation macro :474-507),
// added onto the fine vector (the V-cycle correction).  add = 0 writes.
// FSPLIT: the fine vector is in the parity-split row layout (the finest
// FP32 level under the checkerboard smoother); blank flags stay natural.
//
// FP32: a thread takes two rows by two planes of a column i: along a coarsened axis
// the points 2m and 2m + 1 (counted from 1), whose parents m and m + 1 are each
// other's neighbours, so that the four cells share the same eight coarse values
// and flags; along the others two points with their own.  Bound by its
// instructions where a cell loads and selects its own eight values (192x128x192
// onto 96x128x96: 27 us, 12 with the quad; the bytes are 6.5).
template <bool FSPLIT, bool CY, bool CZ>
__device__ __forceinline__ void prolong_quad(const Box &bf, const Box &bc, int cx, const float *__restrict__ xc,
                                             const uint8_t *__restrict__ blank_c, const uint8_t *__restrict__ blank_f,
                                             float *xf, int add) {
  using T = float;
  const int i = blockIdx.x * blockDim.x + threadIdx.x, m = blockIdx.y * blockDim.y + threadIdx.y, l = blockIdx.z;
  const int J0 = CY ? 2 * m : 2 * m + 1, K0 = CZ ? 2 * l : 2 * l + 1;
  if (i >= bf.nx || J0 > bf.ny) return;
  const int I = i + 1;
  int ic, ia;
  if (!cx) { ic = I; ia = 0; } else { ic = (I + 1) / 2; ia = (I - 2 * ic) == 0 ? 1 : -1; if (I == 1 || I == bf.nx) ia = 0; }
  // the coarse rows and planes of the two sides (beyond the box: the edge's, for
  // cells that do not exist or do not look there), as 32-bit offsets
  const int jc[2] = {max(CY ? m : J0, 1), min(CY ? m + 1 : J0 + 1, bc.ny)};
  const int kc[2] = {max(CZ ? l : K0, 1), min(CZ ? l + 1 : K0 + 1, bc.nz)};
  T X[2][2][2];  // [i side][row][plane]
  uint32_t blank[2][2][2], bfine[2][2], flags = 0;
  uint32_t cf[2][2];
  T xold[2][2];
  bool valid[2][2];
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const int a = q & 1, r = (q >> 1) & 1, p = q >> 2;
    const uint32_t at = (uint32_t)(((kc[p] - 1) * bc.ny + (jc[r] - 1)) * bc.nx + (ic - 1) + a * ia);
    X[a][r][p] = xc[at];
    blank[a][r][p] = blank_c[at];
    flags |= blank[a][r][p];
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int r = q & 1, p = q >> 1, J = J0 + r, K = K0 + p;
    valid[r][p] = J >= 1 && J <= bf.ny && K >= 1 && K <= bf.nz;
    const uint32_t row = (uint32_t)(((K - 1) * bf.ny + (J - 1)) * bf.nx);
    cf[r][p] = row + (FSPLIT ? split_pos(i, bf.nx) : i);
    bfine[r][p] = valid[r][p] ? blank_f[row + i] : 0;
    xold[r][p] = valid[r][p] && add ? xf[cf[r][p]] : (T)0;
    flags |= bfine[r][p] | (valid[r][p] ? 0u : 1u);
  }
  auto weigh = [](T x000, T x010, T x100, T x110, T x001, T x011, T x101, T x111) {
    return (x000 * (T)9 + x010 * (T)3 + x100 * (T)3 + x110) * (T)3. / (T)64. +
           (x001 * (T)9 + x011 * (T)3 + x101 * (T)3 + x111) / (T)64.;
  };
  const bool edge = (CY && (J0 < 2 || J0 + 1 >= bf.ny)) || (CZ && (K0 < 2 || K0 + 1 >= bf.nz));
  if (!flags && !edge) {
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int r = q & 1, p = q >> 1, rn = CY ? 1 - r : r, pn = CZ ? 1 - p : p;
      const T v = weigh(X[0][r][p], X[0][rn][p], X[1][r][p], X[1][rn][p], X[0][r][pn], X[0][rn][pn], X[1][r][pn],
                        X[1][rn][pn]);
      xf[cf[r][p]] = add ? xold[r][p] + v : v;
    }
    return;
  }
#pragma unroll
  for (int q = 0; q < 4; q++) {
    const int r = q & 1, p = q >> 1, rn = CY ? 1 - r : r, pn = CZ ? 1 - p : p, J = J0 + r, K = K0 + p;
    if (!valid[r][p]) continue;
    if (bfine[r][p]) { if (!add) xf[cf[r][p]] = (T)0; continue; }
    // the reference zeroes an offset whose coarse neighbour is blank and at
    // the box's edges: the centre's side instead, an axis at a time
    const bool ui = ia != 0 && !blank[1][r][p], uj = CY && J != 1 && J != bf.ny && !blank[0][rn][p],
               uk = CZ && K != 1 && K != bf.nz && !blank[0][r][pn];
    T Y[2][2][2];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const int a = e & 1, bb = (e >> 1) & 1, cc = e >> 2;
      const T lo0 = uj && bb ? X[0][rn][p] : X[0][r][p], lo1 = uj && bb ? X[1][rn][p] : X[1][r][p];
      const T hi0 = uj && bb ? X[0][rn][pn] : X[0][r][pn], hi1 = uj && bb ? X[1][rn][pn] : X[1][r][pn];
      const T s0 = uk && cc ? hi0 : lo0, s1 = uk && cc ? hi1 : lo1;
      Y[a][bb][cc] = ui && a ? s1 : s0;
    }
    const T v = weigh(Y[0][0][0], Y[0][1][0], Y[1][0][0], Y[1][1][0], Y[0][0][1], Y[0][1][1], Y[1][0][1], Y[1][1][1]);
    xf[cf[r][p]] = add ? xold[r][p] + v : v;
  }
}
template <bool FSPLIT>
__device__ __forceinline__ void prolong_body(const Box &bf, const Box &bc, int cx, int cy, int cz,
                                             const float *__restrict__ xc, const uint8_t *__restrict__ blank_c,
                                             const uint8_t *__restrict__ blank_f, float *xf, int add) {
  pdl_trigger();
  pdl_wait();
  if (cy && cz) prolong_quad<FSPLIT, true, true>(bf, bc, cx, xc, blank_c, blank_f, xf, add);
  else if (cy) prolong_quad<FSPLIT, true, false>(bf, bc, cx, xc, blank_c, blank_f, xf, add);
  else if (cz) prolong_quad<FSPLIT, false, true>(bf, bc, cx, xc, blank_c, blank_f, xf, add);
  else prolong_quad<FSPLIT, false, false>(bf, bc, cx, xc, blank_c, blank_f, xf, add);
}

// FP64: a cell's values each for itself, two rows a thread.  The FP64 pipe takes a
// warp's instruction over 64 cycles of its scheduler, so the quad's four cells in
// one thread run one after the other (72x40x56 solve: 5.55 ms with quads, 5.46).
__device__ __forceinline__ void prolong_rows(Box bf, Box bc, int cx, int cy, int cz, const double *__restrict__ xc,
                                             const uint8_t *__restrict__ blank_c, const uint8_t *__restrict__ blank_f,
                                             double *xf, int add) {
  using T = double;
  pdl_trigger();
  pdl_wait();
  // a thread takes a row j of the grid's and the one as many rows further on of
  // column i (when inside the box): all the loads of both cells first, then
  // both results
  const int i = blockIdx.x * blockDim.x + threadIdx.x, k = blockIdx.z;
  if (i >= bf.nx) return;
  const int mx = bf.nx + 2, my = bf.ny + 2, mz = bf.nz + 2;
  const int I = i + 1, K = k + 1;
  int ic, kc, ia, ka;
  if (!cx) { ic = I; ia = 0; } else { ic = (I + 1) / 2; ia = (I - 2 * ic) == 0 ? 1 : -1; if (I == 1 || I == mx - 2) ia = 0; }
  if (!cz) { kc = K; ka = 0; } else { kc = (K + 1) / 2; ka = (K - 2 * kc) == 0 ? 1 : -1; if (K == 1 || K == mz - 2) ka = 0; }
  size_t c[2];
  bool valid[2];
  int ja[2];
  uint8_t bf0[2], ni[2], nj[2], nk[2];
  T X[2][2][2][2], xold[2];  // [row][i side][j side][k side]
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int j = (blockIdx.y + r * gridDim.y) * blockDim.y + threadIdx.y;
    valid[r] = j < bf.ny;
    if (!valid[r]) continue;
    c[r] = bf.at(i, j, k);
    const int J = j + 1;
    int jc;
    if (!cy) { jc = J; ja[r] = 0; } else { jc = (J + 1) / 2; ja[r] = (J - 2 * jc) == 0 ? 1 : -1; if (J == 1 || J == my - 2) ja[r] = 0; }
    // every load in one round trip: the fine blank flag, the three coarse
    // neighbours' blank flags and the 8 coarse values at the unblanked
    // offsets (all inside the coarse box); a blanked neighbour then
    // selects the centre-side value, exactly the stencil the offsets
    // would give; 32-bit offsets into the coarse box (fewer than 2^31 cells)
    const int base = ((kc - 1) * bc.ny + (jc - 1)) * bc.nx + (ic - 1);
    const int oi = ia, oj = ja[r] * bc.nx, ok = ka * bc.nx * bc.ny;
    bf0[r] = blank_f[c[r]];
    nk[r] = blank_c[base + ok];
    nj[r] = blank_c[base + oj];
    ni[r] = blank_c[base + oi];
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int a = q & 1, bb = (q >> 1) & 1, cc = q >> 2;
      X[r][a][bb][cc] = xc[base + a * oi + bb * oj + cc * ok];
    }
    xold[r] = add ? xf[c[r]] : (T)0;
  }
#pragma unroll
  for (int r = 0; r < 2; r++) {
    if (!valid[r]) continue;
    if (bf0[r]) { if (!add) xf[c[r]] = (T)0; continue; }
    // the reference zeroes an offset whose coarse neighbour is blank; an
    // offset already 0 reads the centre (its test reads the centre cell,
    // which an unblanked fine cell's parent is not).  Collapse the zeroed
    // offsets one axis after the other (constant indices keep X in
    // registers).
    const bool zk = ka != 0 && nk[r], zj = ja[r] != 0 && nj[r], zi = ia != 0 && ni[r];
#pragma unroll
    for (int q = 0; q < 4; q++) X[r][1][q & 1][q >> 1] = zi ? X[r][0][q & 1][q >> 1] : X[r][1][q & 1][q >> 1];
#pragma unroll
    for (int q = 0; q < 4; q++) X[r][q & 1][1][q >> 1] = zj ? X[r][q & 1][0][q >> 1] : X[r][q & 1][1][q >> 1];
#pragma unroll
    for (int q = 0; q < 4; q++) X[r][q & 1][q >> 1][1] = zk ? X[r][q & 1][q >> 1][0] : X[r][q & 1][q >> 1][1];
    T v = (X[r][0][0][0] * (T)9 + X[r][0][1][0] * (T)3 + X[r][1][0][0] * (T)3 + X[r][1][1][0]) * (T)3. / (T)64. +
          (X[r][0][0][1] * (T)9 + X[r][0][1][1] * (T)3 + X[r][1][0][1] * (T)3 + X[r][1][1][1]) / (T)64.;
    if (add) xf[c[r]] = xold[r] + v;
    else xf[c[r]] = v;
  }
}

__global__ void k_restrict_f32(Box bf, Box bc, int cx, int cy, int cz, const float *rf, const float *wf,
                               const uint8_t *blank_c, float *out) {
  restrict_body<float>(bf, bc, cx, cy, cz, rf, wf, blank_c, out);
}
__global__ void k_restrict_f64(Box bf, Box bc, int cx, int cy, int cz, const double *rf, const double *wf,
                               const uint8_t *blank_c, double *out) {
  restrict_body<double>(bf, bc, cx, cy, cz, rf, wf, blank_c, out);
}
__global__ void k_prolong_f32(Box bf, Box bc, int cx, int cy, int cz, const float *xc, const uint8_t *blank_c,
                              const uint8_t *blank_f, float *xf, int add) {
  prolong_body<false>(bf, bc, cx, cy, cz, xc, blank_c, blank_f, xf, add);
}
__global__ void k_prolong_f32_split(Box bf, Box bc, int cx, int cy, int cz, const float *xc, const uint8_t *blank_c,
                                    const uint8_t *blank_f, float *xf, int add) {
  prolong_body<true>(bf, bc, cx, cy, cz, xc, blank_c, blank_f, xf, add);
}
__global__ void k_prolong_f64(Box bf, Box bc, int cx, int cy, int cz, const double *xc, const uint8_t *blank_c,
                              const uint8_t *blank_f, double *xf, int add) {
  prolong_rows(bf, bc, cx, cy, cz, xc, blank_c, blank_f, xf, add);
}

}  // namespace vfs

namespace vfs {

// ---- VolumeFlux (Source/poisson.c:3563-3903, immersed == 1) ----
// Faces between a fluid cell and an IB cell (0.1 < nvert < 1.1), visited
// once each from the cell below them in i, j or k: s = 0 the cell is fluid
// and the face's neighbour IB, s = 1 the reverse.
// 0: fluid, 1: IB, 2: neither, without FP64 for the values masks hold
__device__ __forceinline__ int mask_kind(double nv) {
  const int h = __double2hiint(nv);
  if (__double2loint(nv) == 0) {
    if (h == 0) return 0;
    if (h == 0x3ff00000) return 1;
    if (h == 0x40080000) return 2;
  }
  return nv < 0.1 ? 0 : nv > 0.1 && nv < 1.1 ? 1 : 2;
}
// f(flux, area, s) for each such face of cell (i, j, k), i before j before k
template <class F>
__device__ __forceinline__ void vflux_faces(const Grid &g, const double *__restrict__ nvert, const MetricPtrs &m,
                                            double *ucont, int i, int j, int k, F &&f) {
  const uint32_t t = (uint32_t)g.at(i, j, k);  // (fewer than 2^32 / 19 points)
  const double nv = nvert[t], n0 = nvert[t + 1], n1 = nvert[t + g.mx], n2 = nvert[t + g.mx * g.my];
  const int s = mask_kind(nv);
  if (s == 2) return;
  const uint32_t on = (i < g.mx - 2 && mask_kind(n0) == 1 - s ? 1u : 0u) |
                      (j < g.my - 2 && mask_kind(n1) == 1 - s ? 2u : 0u) |
                      (k < g.mz - 2 && mask_kind(n2) == 1 - s ? 4u : 0u);
  for (int q = 0; q < 3; q++) {
    if (!(on >> q & 1)) continue;
    const double *mm = (q == 0 ? m.csi : q == 1 ? m.eta : m.zet) + 3 * (size_t)t;
    f(ucont + 3 * (size_t)t + q, sqrt(mm[0] * mm[0] + mm[1] * mm[1] + mm[2] * mm[2]), s);
  }
}
// f(c) for this thread's cells of the near plane, in ascending order: the grid's
// stride apart, the bytes of eight cells loaded at a time (one after the other,
// each waits for the last one's latency)
template <class F>
__device__ __forceinline__ void near_cells(size_t n, const uint8_t *__restrict__ near, F &&f) {
  const uint32_t stride = gridDim.x * blockDim.x, end = (uint32_t)n;
  for (uint32_t c0 = blockIdx.x * blockDim.x + threadIdx.x; c0 < end; c0 += 8 * stride) {
    uint32_t hit = 0;
#pragma unroll
    for (int u = 0; u < 8; u++) {
      const uint32_t c = c0 + u * stride;
      hit |= (c < end && near[c] ? 1u : 0u) << u;
    }
    while (hit) {
      const int u = __ffs(hit) - 1;
      hit &= hit - 1;
      f(c0 + u * stride);
    }
  }
}

// Both passes look only at the cells of the near plane (elsewhere no face
// qualifies): one byte per cell instead of five nvert values and a 64-bit
// index division, the bytes of eight cells in flight, masks told apart without
// FP64, all blocks of the fixed grid resident.  256x192x256: 0.17 ms for the two
// passes (0.22 before those; 0.89 ms as three passes over every cell).
//
// First pass: zero |U| <= 1e-8 and sum flux, |U| (or |U| / area for flg 3)
// and area
__global__ void __launch_bounds__(256, 8) k_vflux_sum(Grid g, Box b, const double *__restrict__ nvert,
                                                   const uint8_t *__restrict__ near, MetricPtrs m, double *ucont,
                                                   int flg, double *partial) {
  double sf = 0, sab = 0, sa = 0;
  near_cells(b.n(), near, [&](size_t c) {
    int i, j, k;
    box_ijk(b, c, i, j, k);
    vflux_faces(g, nvert, m, ucont, i + 1, j + 1, k + 1, [&](double *pu, double area, int s) {
      const double u = *pu;
      if (fabs(u) > 1.e-8) {
        sf += s == 0 ? u : -u;
        sab += flg == 3 ? fabs(u) / area : fabs(u);
        sa += area;
      } else {
        *pu = 0.;
      }
    });
  });
  const double t0 = block_sum(sf), t1 = block_sum(sab), t2 = block_sum(sa);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = t0;
    partial[gridDim.x + blockIdx.x] = t1;
    partial[2 * gridDim.x + blockIdx.x] = t2;
  }
}
// The correction from the first pass's partials, rows summed in
// k_reduce_rows' order (one block; flg 4: the overload for immersed != 1,
// whose rows are flux and area).
__global__ void k_vflux_corr(const double *partial, int nb, int flg, double flux_intp_sum, double *corr) {
  double sums[3] = {0., 0., 0.};
  for (int r = 0; r < (flg == 4 ? 2 : 3); r++) {
    double s = 0;
    for (int q = threadIdx.x; q < nb; q += blockDim.x) s += partial[(size_t)r * nb + q];
    sums[r] = block_sum(s);
  }
  if (threadIdx.x) return;
  double v = 0.;
  if (flg == 4) {
    if (sums[1] > 1.e-15) v = sums[0] / sums[1];
  } else if (sums[2] > 1.e-15) {
    if (flg > 1) v = (sums[0] + flux_intp_sum) / sums[1];
    else if (flg) v = (sums[0] + flux_intp_sum) / sums[2];
    else v = sums[0] / sums[2];
  }
  *corr = v;
}

// Second pass: the correction, and the flux and area after it (each face
// belongs to one cell, so its new value is final)
__global__ void __launch_bounds__(256, 8) k_vflux_apply(Grid g, Box b, const double *__restrict__ nvert,
                                                     const uint8_t *__restrict__ near, MetricPtrs m, double *ucont,
                                                     int flg, const double *corr, double *partial) {
  const double cr = *corr;
  double sf = 0, sa = 0;
  near_cells(b.n(), near, [&](size_t c) {
    int i, j, k;
    box_ijk(b, c, i, j, k);
    vflux_faces(g, nvert, m, ucont, i + 1, j + 1, k + 1, [&](double *pu, double area, int s) {
      double u = *pu;
      if (fabs(u) > 1.e-8) {
        double dlt;
        if (flg == 3) dlt = cr * fabs(u) / area;
        else if (flg == 2) dlt = cr * fabs(u);
        else dlt = area * cr;
        u = s == 0 ? u - dlt : u + dlt;
        *pu = u;
      }
      sf += s == 0 ? u : -u;
      sa += area;
    });
  });
  const double t0 = block_sum(sf), t1 = block_sum(sa);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = t0;
    partial[gridDim.x + blockIdx.x] = t1;
  }
}

// ---- VolumeFlux, the overload for immersed != 1, 2 (Source/poisson.c:3299-3493) ----
// Faces between a fluid cell (nvert < 0.1) and a blanked one (nvert > 0.1),
// visited from the cell below them; the area term is the cell metric's norm.
struct VfluxFace {
  double *u;
  double a;
  int s;
};
__device__ inline int vflux0_faces(Grid g, const double *nvert, MetricPtrs m, double *ucont, int i, int j, int k,
                                   VfluxFace f[6]) {
  const size_t t = g.at(i, j, k);
  const size_t nb[3] = {g.at(i + 1, j, k), g.at(i, j + 1, k), g.at(i, j, k + 1)};
  const double *met[3] = {m.csi, m.eta, m.zet};
  int nf = 0;
  for (int s = 0; s < 2; s++) {
    if (s == 0 && !(nvert[t] < 0.1)) continue;
    if (s == 1 && !(nvert[t] > 0.1)) continue;
    for (int q = 0; q < 3; q++) {
      const double nn = nvert[nb[q]];
      if (s == 0 ? !(nn > 0.1) : !(nn < 0.1)) continue;
      const double *mm = &met[q][t * 3];
      f[nf].u = &ucont[t * 3 + q];
      f[nf].a = sqrt(mm[0] * mm[0] + mm[1] * mm[1] + mm[2] * mm[2]);
      f[nf].s = s;
      nf++;
    }
  }
  return nf;
}

// block partials of the flux (+U on the fluid side, -U on the blanked side)
// and of the area
__global__ void __launch_bounds__(256) k_vflux0_sum(Grid g, Box b, const double *__restrict__ nvert,
                                                    const uint8_t *__restrict__ near, MetricPtrs m, double *ucont,
                                                    double *partial) {
  double sf = 0, sa = 0;
  const size_t n = b.n();
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    if (!near[c]) continue;
    int i, j, k;
    box_ijk(b, c, i, j, k);
    VfluxFace f[6];
    const int nf = vflux0_faces(g, nvert, m, ucont, i + 1, j + 1, k + 1, f);
    for (int q = 0; q < nf; q++) {
      const double u = *f[q].u;
      sf += f[q].s == 0 ? u : -u;
      sa += f[q].a;
    }
  }
  const double t0 = block_sum(sf), t1 = block_sum(sa);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = t0;
    partial[gridDim.x + blockIdx.x] = t1;
  }
}

// the correction: off the fluid side, onto the blanked side; then the face
// is zeroed when `zero` (immersed 0 or 3); the flux and area after it
__global__ void __launch_bounds__(256) k_vflux0_apply(Grid g, Box b, const double *__restrict__ nvert,
                                                      const uint8_t *__restrict__ near, MetricPtrs m, double *ucont,
                                                      const double *corr, int zero, double *partial) {
  const double cr = *corr;
  double sf = 0, sa = 0;
  const size_t n = b.n();
  for (size_t c = (size_t)blockIdx.x * blockDim.x + threadIdx.x; c < n; c += (size_t)gridDim.x * blockDim.x) {
    if (!near[c]) continue;
    int i, j, k;
    box_ijk(b, c, i, j, k);
    VfluxFace f[6];
    const int nf = vflux0_faces(g, nvert, m, ucont, i + 1, j + 1, k + 1, f);
    for (int q = 0; q < nf; q++) {
      double u = *f[q].u;
      const double dlt = f[q].a * cr;
      u = zero ? 0. : (f[q].s == 0 ? u - dlt : u + dlt);
      *f[q].u = u;
      sf += f[q].s == 0 ? u : -u;
      sa += f[q].a;
    }
  }
  const double t0 = block_sum(sf), t1 = block_sum(sa);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = t0;
    partial[gridDim.x + blockIdx.x] = t1;
  }
}

// ---- Contra2Cart (Source/rhs.c:35-749), its change of basis ----
// periodic ghosts of a Cmpnts DA array take their partners' values
// the periodic ghosts of a Cmpnts array from their partners, in place
__global__ void k_periodic_cmpnts(Grid g, double *u) {
  int i, j, k, a, b, c, fi, fj, fk;
  if (!shell_point(g, (size_t)blockIdx.x * blockDim.x + threadIdx.x, i, j, k)) return;
  g.remap(i, j, k, a, b, c, fi, fj, fk);
  const size_t s = g.at(a, b, c), t = g.at(i, j, k);
  for (int q = 0; q < 3; q++) u[t * 3 + q] = u[s * 3 + q];
}

// What Contra2Cart takes from the grid alone: the nine minors of the cell
// metrics, their determinant, its reciprocal (0 where a quotient by it may leave
// the normal range) and the reciprocal's rest.
struct CellBasis {
  double q[9], det, y, yl;
  __device__ __forceinline__ void form(const MetricPtrs &m, size_t t) {
    const double *c0 = &m.csi[t * 3], *e0 = &m.eta[t * 3], *z0 = &m.zet[t * 3];
    const double m00 = c0[0], m01 = c0[1], m02 = c0[2], m10 = e0[0], m11 = e0[1], m12 = e0[2], m20 = z0[0],
                 m21 = z0[1], m22 = z0[2];
    q[0] = m11 * m22 - m12 * m21; q[1] = m01 * m22 - m02 * m21; q[2] = m01 * m12 - m02 * m11;
    q[3] = m10 * m22 - m12 * m20; q[4] = m00 * m22 - m02 * m20; q[5] = m00 * m12 - m02 * m10;
    q[6] = m10 * m21 - m11 * m20; q[7] = m00 * m21 - m01 * m20; q[8] = m00 * m11 - m01 * m10;
    det = m00 * q[0] - m01 * q[3] + m02 * q[6];
    const int ex = (__double2hiint(det) >> 20) & 0x7ff;
    y = ex > 700 && ex < 1300 ? 1.0 / det : 0.0;
    yl = fma(-det, y, 1.0) * y;
  }
};
// The 12 planes of them over the box, formed once per grid (where they fit).
__global__ void __launch_bounds__(256) k_contra2cart_coef(Grid g, Box b, MetricPtrs m, double *__restrict__ cc) {
  const size_t n = b.n(), c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  int i, j, k;
  box_ijk(b, c, i, j, k);
  CellBasis B;
  B.form(m, g.at(i + 1, j + 1, k + 1));
  for (int p = 0; p < 9; p++) cc[p * n + c] = B.q[p];
  cc[9 * n + c] = B.det;
  cc[10 * n + c] = B.y;
  cc[11 * n + c] = B.yl;
}

// a / d from y = RN(1 / d) and its rest yl: Markstein's quotient where a lies well inside the
// normal range (its remainders are then exact), a y where a is a zero (the
// quotient's sign), the division elsewhere and for y = 0.
__device__ __forceinline__ double quotient(double a, double d, double y, double yl) {
  const int hi = __double2hiint(a), ex = (hi >> 20) & 0x7ff;
  if (y != 0.0 && ex > 500 && ex < 1500) return markstein4(a, d, y, yl);
  if (y != 0.0 && ((hi & 0x7fffffff) | __double2loint(a)) == 0) return a * y;
  return a / d;
}

// (int)(nvert + 0.1) == 3, decided without FP64 for the values masks hold
__device__ __forceinline__ bool solid(double nv) {
  const long long v = __double_as_longlong(nv);
  if (v == 0x4008000000000000ll) return true;                // 3.0
  if (v == 0 || v == 0x3ff0000000000000ll) return false;     // 0.0, 1.0
  return (int)(nv + 0.1) == 3;
}

// Contra2Cart's change of basis by Cramer's rule, in place on ucat.  Bound by
// the FP64 pipe: with the minors and the reciprocal of the determinant from
// the grid (96 bytes more per cell) a cell takes 30 FP64 instructions instead
// of about 100, halves and comparisons go through the integer pipe.  zero:
// also clears solid cells, except on the two outermost layers (k_zero_rim
// follows once the periodic ghosts have been copied).
// 192x128x192: 0.72 -> 0.315 ms (77 % of the FP64 pipe; 0.34 ms with Markstein's
// second correction in place of the reciprocal's rest).  Without the planes
// (PLANES false) a cell forms them from its metrics, the same bits: 0.66 ms.
template <bool PLANES>
__device__ __forceinline__ void contra2cart_body(const Grid &g, const Box &b, const double *__restrict__ nvert,
                                                 const uint8_t *__restrict__ near, const double *__restrict__ cc,
                                                 const MetricPtrs &m, const double *__restrict__ u,
                                                 double *__restrict__ ucat, int zero) {
  const size_t n = b.n(), c = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= n) return;
  int i, j, k;
  box_ijk(b, c, i, j, k);
  const size_t t = g.at(i + 1, j + 1, k + 1);
  if (near[c]) {
    const double nv = nvert[t];
    if (!(nv < 0.1)) {
      const bool inner = i > 0 && i < b.nx - 1 && j > 0 && j < b.ny - 1 && k > 0 && k < b.nz - 1;
      if (zero && inner && solid(nv)) ucat[t * 3] = ucat[t * 3 + 1] = ucat[t * 3 + 2] = 0.;
      return;
    }
  }
  // (the ghost of a periodic axis is read in its partner)
  const size_t tx = i == 0 && g.px ? t + b.nx - 1 : t - 1,
               ty = j == 0 && g.py ? t + (size_t)(b.ny - 1) * g.mx : t - g.mx,
               tz = k == 0 && g.pz ? t + (size_t)(b.nz - 1) * g.mx * g.my : t - (size_t)g.mx * g.my;
  const double q0 = scale_down(u[tx * 3] + u[t * 3], 1), q1 = scale_down(u[ty * 3 + 1] + u[t * 3 + 1], 1),
               q2 = scale_down(u[tz * 3 + 2] + u[t * 3 + 2], 1);
  CellBasis B;
  if (PLANES) {
    B.det = __ldcs(&cc[9 * n + c]);
    B.y = __ldcs(&cc[10 * n + c]);
    B.yl = __ldcs(&cc[11 * n + c]);
#pragma unroll
    for (int p = 0; p < 9; p++) B.q[p] = __ldcs(&cc[p * n + c]);
  } else {
    B.form(m, t);
  }
  const double d0 = q0 * B.q[0] - q1 * B.q[1] + q2 * B.q[2];
  const double d1 = -q0 * B.q[3] + q1 * B.q[4] - q2 * B.q[5];
  const double d2 = q0 * B.q[6] - q1 * B.q[7] + q2 * B.q[8];
  ucat[t * 3 + 0] = quotient(d0, B.det, B.y, B.yl);
  ucat[t * 3 + 1] = quotient(d1, B.det, B.y, B.yl);
  ucat[t * 3 + 2] = quotient(d2, B.det, B.y, B.yl);
}
__global__ void __launch_bounds__(256) k_contra2cart(Grid g, Box b, const double *nvert, const uint8_t *near,
                                                     const double *cc, const double *u, double *ucat, int zero) {
  contra2cart_body<true>(g, b, nvert, near, cc, MetricPtrs{}, u, ucat, zero);
}
__global__ void __launch_bounds__(256) k_contra2cart_metrics(Grid g, Box b, const double *nvert, const uint8_t *near,
                                                             MetricPtrs m, const double *u, double *ucat, int zero) {
  contra2cart_body<false>(g, b, nvert, near, nullptr, m, u, ucat, zero);
}
// the solid points among the two outermost layers of every side
__global__ void k_zero_rim(Grid g, const double *__restrict__ nvert, double *ucat) {
  const uint32_t nx = 4u * g.my * g.mz, ny = 4u * g.mx * g.mz, nz = 4u * g.mx * g.my;
  uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
  auto layer = [](uint32_t l, int m) { return l < 2 ? min((int)l, m - 1) : max(m - 1 - (int)(l - 2), 0); };
  int i, j, k;
  if (u < nx) {
    i = layer(u & 3, g.mx);
    const uint32_t r = u >> 2;
    k = (int)(r / (uint32_t)g.my);
    j = (int)(r - (uint32_t)k * g.my);
  } else if ((u -= nx) < ny) {
    const uint32_t r = u / (uint32_t)g.mx;
    i = (int)(u - r * g.mx);
    j = layer(r & 3, g.my);
    k = (int)(r >> 2);
  } else if ((u -= ny) < nz) {
    const uint32_t r = u / (uint32_t)g.mx;
    i = (int)(u - r * g.mx);
    k = layer(r & 3, g.mz);
    j = (int)(r >> 2);
  } else {
    return;
  }
  const size_t t = g.at(i, j, k);
  if (solid(nvert[t])) ucat[t * 3] = ucat[t * 3 + 1] = ucat[t * 3 + 2] = 0.;
}

}  // namespace vfs

namespace vfs {

// A cell field (density, level set) on a coarse level: the average of the
// fine cells it covers (the children of MyNvertRestriction's mapping); a
// boundary-layer point takes the fine boundary-layer values it faces.
__global__ void k_cellfield_restrict(Grid gh, Grid gc, int cx, int cy, int cz, const double *fh, double *fc) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= gc.mx) return;
  int ia[2], ja[2], ka[2];
  auto kids = [](int c, int m, int mh, int coarsened, int o[2]) {
    if (c == 0) { o[0] = o[1] = 0; return; }
    if (c == m - 1) { o[0] = o[1] = mh - 1; return; }
    const int h = coarsened ? 2 * c : c;
    o[0] = h;
    o[1] = h - coarsened;
  };
  kids(i, gc.mx, gh.mx, cx, ia);
  kids(j, gc.my, gh.my, cy, ja);
  kids(k, gc.mz, gh.mz, cz, ka);
  double s = 0.;
  for (int q = 0; q < 8; q++) s += fh[gh.at(ia[q & 1], ja[(q >> 1) & 1], ka[q >> 2])];
  fc[gc.at(i, j, k)] = 0.125 * s;
}

}  // namespace vfs
