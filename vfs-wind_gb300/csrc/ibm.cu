// ibm.cu -- immersed-boundary node classification on the GPU: the blanking
// flags nvert of one body from its triangulated surface (ibm_search_advanced,
// Source/ibm.c:92-594, point_cell_advanced :1075-1200, randomdirection
// :59-91, intsect_triangle Source/compgeom.c:25-60).
//
// Compiled with -fmad=false (and host code with -ffp-contract=off) so that
// every ray-triangle test rounds exactly like the reference's C.
//
// Layout of the search structure: the reference hashes the triangles into a
// 40x40x40 grid over the body box and, for a cell centre in hash cell
// (ic,jc,kc), tests every triangle listed in the hash cells (ic,jc,k>=kc),
// each once.  Here each hash column (ic,jc) keeps one deduplicated list of
// its triangles sorted by the top hash cell they reach, so that the search
// of a cell is the prefix of its column list with top cell >= kc: the same
// triangle set without a per-thread "already searched" bitmap.
#include <climits>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "vfs_poisson.h"

namespace vfs {
void set_last_error(const std::string &msg);  // poisson.cu

int ibm_context(vfs_poisson *h, IbmContext *c);
}  // namespace vfs

using namespace vfs;

namespace {

constexpr int kHash = 40;       // ncx = ncy = ncz (ibm.c:111)
constexpr int kMaxTries = 64;   // rays per cell before giving up
constexpr int kMaxHits = 64;    // intersections kept per ray
constexpr int kAhead = 8;       // triangles whose FP32 tests go together

// First glibc rand() value after srand(seed) (TYPE_3 additive feedback
// generator r[i] = r[i-31] + r[i-3] mod 2^32, seeded by Park-Miller
// r[i] = 16807 r[i-1] mod 2^31-1, r[31..33] = r[0..2], 310 outputs dropped).
unsigned glibc_rand_first(unsigned seed) {
  int32_t r[345];
  r[0] = (int32_t)(seed == 0 ? 1 : seed);
  for (int i = 1; i < 31; i++) {
    long long hi = r[i - 1] / 127773, lo = r[i - 1] % 127773;
    long long word = 16807 * lo - 2836 * hi;
    if (word < 0) word += 2147483647;
    r[i] = (int32_t)word;
  }
  for (int i = 31; i < 34; i++) r[i] = r[i - 31];
  for (int i = 34; i < 345; i++) r[i] = (int32_t)((uint32_t)r[i - 31] + (uint32_t)r[i - 3]);
  return ((uint32_t)r[344]) >> 1;
}

struct HashBox {
  double xmin, ymin, zmin, xmax, ymax, zmax, dcx, dcy, dcz;
  // for the FP32 tests: the hash cells' sizes and reciprocals, the rays' end
  // height over zmin and the sum of the box's extents (infinite: no test drops)
  float fcx, fcy, fcz, rcx, rcy, rcz, fz, L;
};

// x > 0 without an FP64 comparison
__device__ __forceinline__ bool positive(double x) {
  const long long v = __double_as_longlong(x);
  return v > 0 && v <= 0x7ff0000000000000ll;
}
// floor(t / d) from FP32 where its error (below 40 * 2^-22) cannot matter
__device__ __forceinline__ int hash_cell(double t, double d, float r) {
  const float q = (float)t * r, k = floorf(q), f = q - k;
  return f > 1e-4f && f < 0.9999f ? (int)k : (int)floor(t / d);
}

// One cell centre: 4 if a ray from it crosses the surface an odd number of
// times, 0 if even, -1 if every ray met a singular (double) intersection or
// too many intersections.
//
// Nearly all triangles of a column are missed by far, and an FP64 test of
// some 45 instructions holds a quarter of the SM for 64 cycles each: a test in
// FP32 on coordinates relative to the box drops the triangles that the FP64
// test is certain to drop.  With u = 2^-24, L the sum of the box's extents and
// one-norms D, E1, E2 of the ray and the edges: FP32 has the ray d' = d + x with
// |x| <= 4 u L (L may be far more than D near a body's top) and t = p - v0 to
// 2 u L.  For a triangle that the ray meets, t = a e1 + w e2 - s d with a, w >= 0,
// a + w <= 1 and 0 < s <= 1 (the ray ends above the body), so that
//   t.(d' x e2) = a det' - s d'.(x x e2)     t.(d' x e2) and d'.(t x e1) within
//   d'.(t x e1) = w det' + s d'.(x x e1)     4 u L D E2 and 4 u L D E1 of a, w
//   e2.(t x e1) = s det                      times det', whatever its sign is
// and where det' has not the sign of det, |det| <= |x.(e2 x e1)| <= 4 u L E1 E2.  With
// the error of t and the roundings (24 u times the norms) that stays below the
// margins, 64 u times the norms with L added to that of t.  A triangle whose det'
// is 0 within its margin is kept, and every one where the box is so large
// (L > 10^12) that FP32 products might overflow: L is infinite then.  tf: v0,
// e1, e2, |e1|, |e2| per triangle.  A tower over 840 k cells: 674 -> 380 us, a
// rod over 48 k cells: 75 -> 58 us; with eight triangles' tests at a time, whose
// loads fly together, 210 and 30 us (one at a time is a chain of two loads each;
// four 5 % slower).
__device__ int point_cell(const double p[3], const double rel[3], int ip, int jp, int kp, const HashBox &H,
                          const int *col_start, const int *col_tri, const int *col_kmax, const double *tv,
                          const double *nf, const double *s_tab, const float4 *tf) {
  const int col = jp * kHash + ip;
  const int e0 = col_start[col], e1 = col_start[col + 1];
  const float px = (float)rel[0], py = (float)rel[1], pz = (float)rel[2];
  for (int tries = 1; tries <= kMaxTries; tries++) {
    const double s = s_tab[tries];
    const float fs = (float)s;
    const float dx = H.fcx * ((float)ip + 0.5f + fs) - px, dy = H.fcy * ((float)jp + 0.5f + fs) - py, dz = H.fz - pz;
    const float mD = 4e-6f * (fabsf(dx) + fabsf(dy) + fabsf(dz));
    bool aimed = false;
    double dir[3] = {0., 0., 0.};
    double dt[kMaxHits];
    int dn[kMaxHits];
    int nintp = 0;
    bool singular = false, overflow = false;
    // the FP32 tests of kAhead triangles at a time, their loads together (a
    // triangle's are two dependent ones), then the exact test of those that pass,
    // in the list's order
    bool more = true;
    for (int q0 = e0; q0 < e1 && more && !singular && !overflow; q0 += kAhead) {
      uint32_t pass = 0;
      int tri[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; u++) {
        const int q = min(q0 + u, e1 - 1);
        // (the list is sorted by top hash cell, descending)
        const bool on = q0 + u < e1 && col_kmax[q] - 1 >= kp;
        more &= on;
        const int e = tri[u] = col_tri[q];
        const float4 A = tf[3 * e], B = tf[3 * e + 1], C = tf[3 * e + 2];
        const float ax = A.w, ay = B.x, az = B.y, bx = B.z, by = B.w, bz = C.x, n1 = C.y, n2 = C.z;
        const float qx = dy * bz - dz * by, qy = dz * bx - dx * bz, qz = dx * by - dy * bx;
        const float det = ax * qx + ay * qy + az * qz, ad = fabsf(det), md = mD * n1 * n2;
        const float sg = det < 0.f ? -1.f : 1.f;
        const float tx = px - A.x, ty = py - A.y, tz = pz - A.z;
        const float T = fabsf(tx) + fabsf(ty) + fabsf(tz) + H.L;
        const float un = (tx * qx + ty * qy + tz * qz) * sg, mu = mD * n2 * T;
        const float rx = ty * az - tz * ay, ry = tz * ax - tx * az, rz = tx * ay - ty * ax;
        const float wn = (dx * rx + dy * ry + dz * rz) * sg, mw = mD * n1 * T;
        const bool out = ad > md && (un < -mu || un > ad + mu + md || wn < -mw || un + wn > ad + mu + mw + md ||
                                     (bx * rx + by * ry + bz * rz) * sg < -4e-6f * n1 * n2 * T);
        pass |= (on && !out ? 1u : 0u) << u;
      }
      while (pass && !singular) {
        const int at = __ffs(pass) - 1;
        pass &= pass - 1;
        int e = tri[0];
#pragma unroll
        for (int o = 1; o < kAhead; o++) e = at == o ? tri[o] : e;
        if (!aimed) {
          aimed = true;
          const double xpc = H.dcx * (ip + 0.5) + H.xmin, ypc = H.dcy * (jp + 0.5) + H.ymin;
          dir[0] = xpc + s * H.dcx - p[0];
          dir[1] = ypc + s * H.dcy - p[1];
          dir[2] = H.zmax + 0.2 - p[2];
          const double nrm = sqrt(dir[0] * dir[0] + dir[1] * dir[1] + dir[2] * dir[2]);
          dir[0] /= nrm; dir[1] /= nrm; dir[2] /= nrm;
        }
        const double *v = &tv[(size_t)e * 9];
        // intsect_triangle, compgeom.c:25-60
        const double EPS = 0.00000001;
        double e1v[3] = {v[3] - v[0], v[4] - v[1], v[5] - v[2]};
        double e2v[3] = {v[6] - v[0], v[7] - v[1], v[8] - v[2]};
        double pv[3] = {dir[1] * e2v[2] - dir[2] * e2v[1], dir[2] * e2v[0] - dir[0] * e2v[2],
                        dir[0] * e2v[1] - dir[1] * e2v[0]};
        double det = e1v[0] * pv[0] + e1v[1] * pv[1] + e1v[2] * pv[2];
        if (det > -EPS && det < EPS) continue;
        double inv = 1.0 / det;
        double tvv[3] = {p[0] - v[0], p[1] - v[1], p[2] - v[2]};
        double u = (tvv[0] * pv[0] + tvv[1] * pv[1] + tvv[2] * pv[2]) * inv;
        if (u < 0.0 || u > 1.0) continue;
        double qv[3] = {tvv[1] * e1v[2] - tvv[2] * e1v[1], tvv[2] * e1v[0] - tvv[0] * e1v[2],
                        tvv[0] * e1v[1] - tvv[1] * e1v[0]};
        double w = (dir[0] * qv[0] + dir[1] * qv[1] + dir[2] * qv[2]) * inv;
        if (w < 0.0 || u + w > 1.0) continue;
        double t = (e2v[0] * qv[0] + e2v[1] * qv[1] + e2v[2] * qv[2]) * inv;
        if (!(t > 0)) continue;
        if (nintp == kMaxHits) { overflow = true; break; }
        dt[nintp] = t;
        dn[nintp] = e;
        nintp++;
        for (int m = 0; m < nintp - 1; m++) {
          const double *a = &nf[(size_t)dn[m] * 3], *b = &nf[(size_t)e * 3];
          double ndotn = a[0] * b[0] + a[1] * b[1] + a[2] * b[2];
          if (fabs(t - dt[m]) < 1.e-8 && ndotn > -0.97) singular = true;
        }
      }
    }
    if (overflow) return -1;
    if (!singular) return (nintp % 2) ? 4 : 0;
  }
  return -1;
}

// The device copy of one body's surface.
struct Surface {
  HashBox H;
  const int *col_start, *col_tri, *col_kmax;
  const double *tv, *nf, *s_tab;
  const float4 *tf;
};

// Classification of one body (ibm_search_advanced, ibm.c:92-325) at DA point
// t of value nv: boundary points as they are, interior points whose centre
// lies in the body's hash box the larger of their value and the ray-parity
// test (4 inside); first: body 0 clears every value below 5 before.
__device__ __forceinline__ double classify_point(const Grid &g, const double *__restrict__ cent, bool first,
                                                 const Surface &S, int i, int j, int k, size_t t, double nv,
                                                 int *failed) {
  if (i < 1 || i >= g.mx - 1 || j < 1 || j >= g.my - 1 || k < 1 || k >= g.mz - 1) return nv;
  const HashBox &H = S.H;
  if (first && nv < 5.) nv = 0;
  const double p[3] = {cent[t * 3], cent[t * 3 + 1], cent[t * 3 + 2]};
  // (a difference has its exact sign)
  const double rel[3] = {p[0] - H.xmin, p[1] - H.ymin, p[2] - H.zmin};
  if (positive(rel[0]) && positive(H.xmax - p[0]) && positive(rel[1]) && positive(H.ymax - p[1]) &&
      positive(rel[2]) && positive(H.zmax - p[2])) {
    const int ic = hash_cell(rel[0], H.dcx, H.rcx), jc = hash_cell(rel[1], H.dcy, H.rcy),
              kc = hash_cell(rel[2], H.dcz, H.rcz);
    int val = point_cell(p, rel, ic, jc, kc, H, S.col_start, S.col_tri, S.col_kmax, S.tv, S.nf, S.s_tab, S.tf);
    if (val < 0) {
      atomicAdd(failed, 1);
      val = 0;
    }
    nv = nv > val ? nv : (double)val;
    if (nv < 0) nv = 0;
  }
  return nv;
}
// the dilation's test of a point as a neighbour, once per point instead of in
// each of its 27 neighbours
__device__ __forceinline__ uint8_t is_four(double nv) {
  if ((__double_as_longlong(nv) << 1) == 0) return 0;
  return (int)((nv < 0 ? 0. : nv) + 0.5) == 4;
}
// over every DA point (the search with IB node records; is4 null there)
__global__ void k_ibm_classify_from(Grid g, const double *__restrict__ cent, int first, Surface S, const double *src,
                                    double *dst, uint8_t *is4, int *failed) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= g.mx) return;
  const size_t t = g.at(i, j, k);
  const double nv = classify_point(g, cent, first, S, i, j, k, t, src[t], failed);
  dst[t] = nv;
  if (is4) is4[t] = is_four(nv);
}
// Body 0 clears every interior value below 5, in place (negative boundary
// values become 0, as the dilation leaves them); state[1]: a boundary point
// counts as a 4 for the dilation.
__global__ void k_ibm_clear(Grid g, double *nvert, int *state) {
  const size_t N = g.n();
  for (size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x; t < N; t += (size_t)gridDim.x * blockDim.x) {
    const double v = nvert[t];
    if (__double_as_longlong(v) == 0) continue;
    int i, j, k;
    da_ijk(g, t, i, j, k);
    if (i >= 1 && i < g.mx - 1 && j >= 1 && j < g.my - 1 && k >= 1 && k < g.mz - 1) {
      if (v < 5.) nvert[t] = 0;
    } else {
      if (v < 0) nvert[t] = 0;
      if (is_four(v)) state[1] = 1;
    }
  }
}
// A body changes only the cells whose centre lies in its hash box and, by the
// dilation, their neighbours (the earlier bodies' marks are finished: no 2 or
// 4 is left): both passes run on the index box of those cells (box: lower
// ends, upper ends; k_ibm_box_cells), grown by m points.  Body 0, too, once
// the mask is cleared: 28 M points 2.06 -> 0.50 ms.
struct Region {
  int lo[3], n[3];
  __device__ Region(const Grid &g, const int *box, int m) {
    const int hi[3] = {g.mx, g.my, g.mz};
    for (int q = 0; q < 3; q++) {
      lo[q] = max(box[q] - m, 0);
      n[q] = box[0] > box[3] ? 0 : min(box[3 + q] + m + 1, hi[q]) - lo[q];
    }
  }
};
// (the last factor keeps a warp on consecutive points of the box)
#define REGION_LOOP(R, i, j, k)                                                                              \
  for (uint32_t w = blockIdx.x * blockDim.x + threadIdx.x; w < (uint32_t)R.n[0] * R.n[1] * R.n[2];           \
       w += gridDim.x * blockDim.x)                                                                          \
    if (const uint32_t row = w / (uint32_t)R.n[0], kk = row / (uint32_t)R.n[1]; true)                       \
      if (const int i = R.lo[0] + (int)(w - row * R.n[0]), j = R.lo[1] + (int)(row - kk * R.n[1]),           \
          k = R.lo[2] + (int)kk;                                                                             \
          true)
__global__ void __launch_bounds__(128) k_ibm_classify(Grid g, const double *__restrict__ cent, Surface S,
                                                      const int *__restrict__ box, const double *__restrict__ src,
                                                      double *__restrict__ dst, uint8_t *is4, int *failed) {
  const Region R(g, box, 2);
  REGION_LOOP(R, i, j, k) {
    const size_t t = g.at(i, j, k);
    const double nv = classify_point(g, cent, false, S, i, j, k, t, src[t], failed);
    dst[t] = nv;
    is4[t] = is_four(nv);
  }
}

// The search of a body needs the index box of the interior
// cells whose centre lies strictly inside its hash box.  The centres are
// bounded per block of 8x8x8 interior cells once per grid (k_cent_blocks);
// a block whose bounds miss the hash box holds no such cell, so only the
// cells of the other blocks are tested, with the same strict comparisons.
constexpr int kCentBlock = 8;
__global__ void __launch_bounds__(512) k_cent_blocks(Grid g, const double *__restrict__ cent, int nbx, int nby,
                                                     double *bbox) {
  const int b = blockIdx.x;
  const int bi = b % nbx, bj = (b / nbx) % nby, bk = b / (nbx * nby);
  const int i = 1 + bi * kCentBlock + (threadIdx.x & 7), j = 1 + bj * kCentBlock + ((threadIdx.x >> 3) & 7),
            k = 1 + bk * kCentBlock + (threadIdx.x >> 6);
  double lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
  if (i < g.mx - 1 && j < g.my - 1 && k < g.mz - 1) {
    const size_t t = g.at(i, j, k);
    for (int q = 0; q < 3; q++) lo[q] = hi[q] = cent[t * 3 + q];
  }
  for (int q = 0; q < 3; q++)
    for (int o = 16; o > 0; o >>= 1) {
      lo[q] = fmin(lo[q], __shfl_xor_sync(0xffffffffu, lo[q], o));
      hi[q] = fmax(hi[q], __shfl_xor_sync(0xffffffffu, hi[q], o));
    }
  __shared__ double sh[16][6];
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0)
    for (int q = 0; q < 3; q++) { sh[w][q] = lo[q]; sh[w][3 + q] = hi[q]; }
  __syncthreads();
  if (threadIdx.x < 6) {
    double v = sh[0][threadIdx.x];
    for (int u = 1; u < 16; u++) v = threadIdx.x < 3 ? fmin(v, sh[u][threadIdx.x]) : fmax(v, sh[u][threadIdx.x]);
    bbox[(size_t)b * 6 + threadIdx.x] = v;
  }
}

// One thread tests one block's bounds and lists the block when they meet
// the hash box (box[6]: the count); then every thread block of a fixed grid
// takes listed blocks in turn and tests their cells, two per thread (box[0..5]:
// min/max of i, j, k), so that a large box's blocks spread over the
// whole GPU.
__global__ void __launch_bounds__(256) k_ibm_box_hits(const double *__restrict__ bbox, int nblocks, HashBox H,
                                                      int *box, int *hits) {
  const int b = blockIdx.x * blockDim.x + threadIdx.x;
  if (b >= nblocks) return;
  const double *q = bbox + (size_t)b * 6;
  if (q[3] > H.xmin && q[0] < H.xmax && q[4] > H.ymin && q[1] < H.ymax && q[5] > H.zmin && q[2] < H.zmax)
    hits[atomicAdd(&box[6], 1)] = b;
}
__global__ void __launch_bounds__(256) k_ibm_box_cells(Grid g, const double *__restrict__ cent, int nbx, int nby,
                                                       HashBox H, const int *__restrict__ hits, int *box) {
  const int nh = *(volatile int *)&box[6];
  int lo[3] = {INT_MAX, INT_MAX, INT_MAX}, hi[3] = {INT_MIN, INT_MIN, INT_MIN};
  for (int w = blockIdx.x; w < nh; w += gridDim.x) {
    const int bb = hits[w];
    const int bi = bb % nbx, bj = (bb / nbx) % nby, bk = bb / (nbx * nby);
    for (int c = threadIdx.x; c < kCentBlock * kCentBlock * kCentBlock; c += blockDim.x) {
      const int i = 1 + bi * kCentBlock + (c & 7), j = 1 + bj * kCentBlock + ((c >> 3) & 7),
                k = 1 + bk * kCentBlock + (c >> 6);
      if (i >= g.mx - 1 || j >= g.my - 1 || k >= g.mz - 1) continue;
      const size_t t = g.at(i, j, k);
      const double p0 = cent[t * 3], p1 = cent[t * 3 + 1], p2 = cent[t * 3 + 2];
      if (positive(p0 - H.xmin) && positive(H.xmax - p0) && positive(p1 - H.ymin) && positive(H.ymax - p1) &&
          positive(p2 - H.zmin) && positive(H.zmax - p2)) {
        lo[0] = min(lo[0], i); lo[1] = min(lo[1], j); lo[2] = min(lo[2], k);
        hi[0] = max(hi[0], i); hi[1] = max(hi[1], j); hi[2] = max(hi[2], k);
      }
    }
  }
  for (int q = 0; q < 3; q++) {  // six atomics a warp, not a cell
    const int l = __reduce_min_sync(0xffffffffu, lo[q]), u = __reduce_max_sync(0xffffffffu, hi[q]);
    if ((threadIdx.x & 31) == 0 && l <= u) {
      atomicMin(&box[q], l);
      atomicMax(&box[3 + q], u);
    }
  }
}

// near-boundary dilation over every DA point (ibm.c:326-348); a parallel pass
// over a snapshot equals the in-place loop because it only writes 2 and
// reads only the 4s.
__global__ void k_ibm_dilate(Grid g, const double *src, double *dst) {
  int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i >= g.mx) return;
  const size_t t = g.at(i, j, k);
  double v = src[t];
  if (v < 0) v = 0;
  if ((int)(v + 0.5) != 4) {
    const int ip = i < g.mx - 1 ? i + 1 : i, im = i > 0 ? i - 1 : i;
    const int jp = j < g.my - 1 ? j + 1 : j, jm = j > 0 ? j - 1 : j;
    const int kp = k < g.mz - 1 ? k + 1 : k, km = k > 0 ? k - 1 : k;
    for (int kk = km; kk <= kp; kk++)
      for (int jj = jm; jj <= jp; jj++)
        for (int ii = im; ii <= ip; ii++) {
          double w = src[g.at(ii, jj, kk)];
          if (w < 0) w = 0;
          if ((int)(w + 0.5) == 4) v = v > 2 ? v : 2;
        }
  }
  dst[t] = v;
}

// back to 3 / 1 and the wall rows of bctype -1 / -2 (ibm.c:514-543)
__device__ __forceinline__ double ibm_finish_value(const Grid &g, int b0, int b1, int b2, int b3, int b4, int b5,
                                                   int i, int j, int k, double v) {
  if ((int)(v + 0.5) == 2) v = 1;
  if ((int)(v + 0.5) == 4) v = 3;
  for (int q = -1; q >= -2; q--) {
    if (b0 == q && i == 1) v = 1;
    if (b1 == q && i == g.mx - 2) v = 1;
    if (b2 == q && j == 1) v = 1;
    if (b3 == q && j == g.my - 2) v = 1;
    if (b4 == q && k == 1) v = 1;
    if (b5 == q && k == g.mz - 2) v = 1;
  }
  return v;
}
__global__ void k_ibm_finish(Grid g, int b0, int b1, int b2, int b3, int b4, int b5, double *nvert) {
  int i = blockIdx.x * blockDim.x + threadIdx.x + 1, j = blockIdx.y + 1, k = blockIdx.z + 1;
  if (i >= g.mx - 1) return;
  const size_t t = g.at(i, j, k);
  nvert[t] = ibm_finish_value(g, b0, b1, b2, b3, b4, b5, i, j, k, nvert[t]);
}
// the dilation and the finishing pass in one (the search without IB node
// records, where nothing reads the dilated marks in between): the DA points
// get the dilation of src, the interior ones then their finished value
__device__ __forceinline__ void dilate_finish_point(const Grid &g, const int (&b)[6], const double *__restrict__ src,
                                                    const uint8_t *__restrict__ is4, double *__restrict__ dst, int i,
                                                    int j, int k) {
  const size_t t = g.at(i, j, k);
  double v = src[t];
  if (v < 0) v = 0;
  if (!is4[t]) {
    const int ip = i < g.mx - 1 ? i + 1 : i, im = i > 0 ? i - 1 : i;
    const int jp = j < g.my - 1 ? j + 1 : j, jm = j > 0 ? j - 1 : j;
    const int kp = k < g.mz - 1 ? k + 1 : k, km = k > 0 ? k - 1 : k;
    bool near = false;
    for (int kk = km; kk <= kp; kk++)
      for (int jj = jm; jj <= jp; jj++)
        for (int ii = im; ii <= ip; ii++) near |= is4[g.at(ii, jj, kk)] != 0;
    if (near) v = v > 2 ? v : 2;
  }
  if (i >= 1 && i < g.mx - 1 && j >= 1 && j < g.my - 1 && k >= 1 && k < g.mz - 1)
    v = ibm_finish_value(g, b[0], b[1], b[2], b[3], b[4], b[5], i, j, k, v);
  dst[t] = v;
}
struct Walls {
  int b[6];
};
__global__ void k_ibm_dilate_finish_all(Grid g, Walls W, const double *__restrict__ src,
                                        const uint8_t *__restrict__ is4, double *__restrict__ dst) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, k = blockIdx.z;
  if (i < g.mx) dilate_finish_point(g, W.b, src, is4, dst, i, j, k);
}
__global__ void __launch_bounds__(128) k_ibm_dilate_finish(Grid g, Walls W, const int *__restrict__ box,
                                                           const double *__restrict__ src,
                                                           const uint8_t *__restrict__ is4, double *__restrict__ dst) {
  const Region R(g, box, 1);
  REGION_LOOP(R, i, j, k) dilate_finish_point(g, W.b, src, is4, dst, i, j, k);
}

// ---- IB interpolation records (ibm.c:373-508) ----
// One thread per IB node: the nearest surface element (nearestcell1,
// :1373-1518), the interception of the normal ray with the 3x3 patches of
// neighbouring cell centres (InterceptionPoint, :1766-2258, ICP :1666-1764)
// and the boundary fallback (:423-505), in the reference's operation order
// (compiled without FMA contraction).
struct V3 {
  double x, y, z;
};
struct V2 {
  double x, y;
};
__device__ inline V3 vload(const double *a, size_t t) { return V3{a[3 * t], a[3 * t + 1], a[3 * t + 2]}; }
__device__ inline double vdist(V3 a, V3 b) {
  return sqrt((a.x - b.x) * (a.x - b.x) + (a.y - b.y) * (a.y - b.y) + (a.z - b.z) * (a.z - b.z));
}
// ISSameSide2D (compgeom.c:62-114)
__device__ inline int same_side(V2 p, V2 p1, V2 p2, V2 p3) {
  const double t1 = (p.x - p1.x) * (p2.y - p1.y) - (p.y - p1.y) * (p2.x - p1.x);
  const double t2 = (p3.x - p1.x) * (p2.y - p1.y) - (p3.y - p1.y) * (p2.x - p1.x);
  const double lt = sqrt((p1.x - p2.x) * (p1.x - p2.x) + (p1.y - p2.y) * (p1.y - p2.y));
  if (fabs(t1 / lt) < 1.e-10) return 1;
  if (t1 > 0) return t2 > 0 ? 1 : -1;
  return t2 < 0 ? 1 : -1;
}
// ISInsideTriangle2D / ISPointInTriangle (compgeom.c:116-166)
__device__ inline int point_in_triangle(V3 p, V3 p1, V3 p2, V3 p3, double nx, double ny, double nz) {
  V2 a, b, c, e;
  if (fabs(nz) >= fabs(nx) && fabs(nz) >= fabs(ny)) {
    a = {p.x, p.y}; b = {p1.x, p1.y}; c = {p2.x, p2.y}; e = {p3.x, p3.y};
  } else if (fabs(nx) >= fabs(ny) && fabs(nx) >= fabs(nz)) {
    a = {p.z, p.y}; b = {p1.z, p1.y}; c = {p2.z, p2.y}; e = {p3.z, p3.y};
  } else {
    a = {p.x, p.z}; b = {p1.x, p1.z}; c = {p2.x, p2.z}; e = {p3.x, p3.z};
  }
  int ls = same_side(a, b, c, e);
  if (ls < 0) return ls;
  ls = same_side(a, c, e, b);
  if (ls < 0) return ls;
  return same_side(a, e, b, c);
}
// Dis_P_Line (compgeom.c:168-194)
__device__ inline void dist_point_line(V3 p, V3 p1, V3 p2, V3 &po, double &d) {
  const double dx21 = p2.x - p1.x, dy21 = p2.y - p1.y, dz21 = p2.z - p1.z;
  const double dx31 = p.x - p1.x, dy31 = p.y - p1.y, dz31 = p.z - p1.z;
  const double t = (dx31 * dx21 + dy31 * dy21 + dz31 * dz21) / (dx21 * dx21 + dy21 * dy21 + dz21 * dz21);
  if (t < 0) {
    po = p1;
    d = sqrt(dx31 * dx31 + dy31 * dy31 + dz31 * dz31);
  } else if (t > 1) {
    po = p2;
    d = sqrt((p.x - po.x) * (p.x - po.x) + (p.y - po.y) * (p.y - po.y) + (p.z - po.z) * (p.z - po.z));
  } else {
    po = V3{p1.x + t * dx21, p1.y + t * dy21, p1.z + t * dz21};
    d = sqrt((p.x - po.x) * (p.x - po.x) + (p.y - po.y) * (p.y - po.y) + (p.z - po.z) * (p.z - po.z));
  }
}
// triangle_intp / triangle_intp2 (compgeom.c:196-230) on the plane the
// dominant normal component picks
__device__ inline void project_bary(V3 p, V3 p1, V3 p2, V3 p3, double nx, double ny, double nz, double w[3]) {
  V2 a, b, c, e;
  if (fabs(nx) >= fabs(ny) && fabs(nx) >= fabs(nz)) {
    a = {p.y, p.z}; b = {p1.y, p1.z}; c = {p2.y, p2.z}; e = {p3.y, p3.z};
  } else if (fabs(ny) >= fabs(nx) && fabs(ny) >= fabs(nz)) {
    a = {p.x, p.z}; b = {p1.x, p1.z}; c = {p2.x, p2.z}; e = {p3.x, p3.z};
  } else if (fabs(nz) >= fabs(ny) && fabs(nz) >= fabs(nx)) {
    a = {p.y, p.x}; b = {p1.y, p1.x}; c = {p2.y, p2.x}; e = {p3.y, p3.x};
  } else {
    return;
  }
  const double x13 = b.x - e.x, y13 = b.y - e.y, x23 = c.x - e.x, y23 = c.y - e.y;
  const double xp3 = a.x - e.x, yp3 = a.y - e.y;
  const double det = x13 * y23 - x23 * y13;
  w[0] = (y23 * xp3 - x23 * yp3) / det;
  w[1] = (-y13 * xp3 + x13 * yp3) / det;
  w[2] = 1. - w[0] - w[1];
}
__constant__ int kPatchTri[8][3] = {{0, 1, 4}, {1, 2, 4}, {2, 4, 5}, {4, 5, 8}, {4, 7, 8}, {4, 6, 7}, {3, 4, 6}, {3, 4, 0}};

// the cells of one body marked 2 (IB node) after the dilation, interior
// only: per 256-cell block, their count ...
__global__ void k_ibm_mark_count(Grid g, const double *nvert, int *bcount) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool mark = false;
  if (t < g.n()) {
    const int i = (int)(t % g.mx), j = (int)((t / g.mx) % g.my), k = (int)(t / ((size_t)g.mx * g.my));
    mark = i >= 1 && i < g.mx - 1 && j >= 1 && j < g.my - 1 && k >= 1 && k < g.mz - 1 &&
           (int)(nvert[t] + 0.5) == 2;
  }
  const int c = __syncthreads_count(mark);
  if (threadIdx.x == 0) bcount[blockIdx.x] = c;
}
// ... and their DA indices in order, from the blocks' exclusive offsets
__global__ void k_ibm_mark_scatter(Grid g, const double *nvert, const int *boff, int *list) {
  __shared__ int wsum[8];
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  bool mark = false;
  if (t < g.n()) {
    const int i = (int)(t % g.mx), j = (int)((t / g.mx) % g.my), k = (int)(t / ((size_t)g.mx * g.my));
    mark = i >= 1 && i < g.mx - 1 && j >= 1 && j < g.my - 1 && k >= 1 && k < g.mz - 1 &&
           (int)(nvert[t] + 0.5) == 2;
  }
  const unsigned ball = __ballot_sync(0xffffffffu, mark);
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
  if (lane == 0) wsum[wp] = __popc(ball);
  __syncthreads();
  int base = boff[blockIdx.x];
  for (int q = 0; q < wp; q++) base += wsum[q];
  if (mark) list[base + __popc(ball & ((1u << lane) - 1u))] = (int)t;
}

__global__ void k_ibm_nodes(Grid g, const double *__restrict__ cent, const int *__restrict__ list, int n_nodes,
                            int n_elmt, const double *__restrict__ tv, const double *__restrict__ nf,
                            const double *__restrict__ qv, const double *__restrict__ rad, vfs_ibm_node *out) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_nodes) return;
  const size_t t = (size_t)list[n];
  const int i = (int)(t % g.mx), j = (int)((t / g.mx) % g.my), k = (int)(t / ((size_t)g.mx * g.my));
  vfs_ibm_node nd;
  nd.i = i; nd.j = j; nd.k = k;
  const V3 p = vload(cent, t);
  // nearestcell1
  double dmin = 1.e20;
  int cell_min = -100;
  V3 pmin{0., 0., 0.};
  for (int e = 0; e < n_elmt; e++) {
    const V3 qe{qv[3 * e], qv[3 * e + 1], qv[3 * e + 2]};
    const double d_center = vdist(p, qe);
    if (!(d_center - rad[e] < dmin)) continue;
    const double *v = &tv[(size_t)e * 9];
    const V3 p1{v[0], v[1], v[2]}, p2{v[3], v[4], v[5]}, p3{v[6], v[7], v[8]};
    const double nfx = nf[3 * e], nfy = nf[3 * e + 1], nfz = nf[3 * e + 2];
    double tf = (p.x - p1.x) * nfx + (p.y - p1.y) * nfy + (p.z - p1.z) * nfz;
    if (fabs(tf) < 1.e-10) tf = 1.e-10;
    if (!(tf >= 0)) continue;
    const V3 pj{p.x - tf * nfx, p.y - tf * nfy, p.z - tf * nfz};
    if (point_in_triangle(pj, p1, p2, p3, nfx, nfy, nfz) == 1) {
      if (tf < dmin) { dmin = tf; pmin = pj; cell_min = e; }
    } else {
      V3 po;
      double d;
      dist_point_line(p, p1, p2, po, d);
      if (d < dmin) { dmin = d; pmin = po; cell_min = e; }
      dist_point_line(p, p2, p3, po, d);
      if (d < dmin) { dmin = d; pmin = po; cell_min = e; }
      dist_point_line(p, p3, p1, po, d);
      if (d < dmin) { dmin = d; pmin = po; cell_min = e; }
    }
  }
  nd.cell = cell_min;
  nd.pmin[0] = pmin.x; nd.pmin[1] = pmin.y; nd.pmin[2] = pmin.z;
  nd.d_s = dmin;
  nd.cs[0] = nd.cs[1] = nd.cs[2] = 0.;
  if (cell_min >= 0) {
    const double *v = &tv[(size_t)cell_min * 9];
    project_bary(pmin, V3{v[0], v[1], v[2]}, V3{v[3], v[4], v[5]}, V3{v[6], v[7], v[8]}, nf[3 * cell_min],
                 nf[3 * cell_min + 1], nf[3 * cell_min + 2], nd.cs);
  }
  // InterceptionPoint: the patches at i-1, i+1, j-1, j+1, k-1, k+1
  double nfx = p.x - pmin.x, nfy = p.y - pmin.y, nfz = p.z - pmin.z;
  const double dr = sqrt(nfx * nfx + nfy * nfy + nfz * nfz);
  nfx /= dr; nfy /= dr; nfz /= dr;
  nd.imode = -100;
  for (int s = 0; s < 3; s++) { nd.ip[s] = i; nd.jp[s] = j; nd.kp[s] = k; nd.cr[s] = 0.; }
  nd.d_i = 0.;
  for (int face = 0; face < 6 && nd.imode < 0; face++) {
    int ip[9], jp[9], kp[9];
    V3 pc[9];
    for (int s = 0; s < 9; s++) {
      const int a = s % 3 - 1, b = s / 3 - 1;
      switch (face) {
        case 0: ip[s] = i - 1; jp[s] = j + a; kp[s] = k + b; break;
        case 1: ip[s] = i + 1; jp[s] = j + a; kp[s] = k + b; break;
        case 2: ip[s] = i + a; jp[s] = j - 1; kp[s] = k + b; break;
        case 3: ip[s] = i + a; jp[s] = j + 1; kp[s] = k + b; break;
        case 4: ip[s] = i + a; jp[s] = j + b; kp[s] = k - 1; break;
        default: ip[s] = i + a; jp[s] = j + b; kp[s] = k + 1; break;
      }
      pc[s] = vload(cent, g.at(ip[s], jp[s], kp[s]));
    }
    for (int tr = 0; tr < 8; tr++) {  // ICP
      const V3 p1 = pc[kPatchTri[tr][0]], p2 = pc[kPatchTri[tr][1]], p3 = pc[kPatchTri[tr][2]];
      const double dx1 = p.x - p1.x, dy1 = p.y - p1.y, dz1 = p.z - p1.z;
      const double dx2 = p2.x - p1.x, dy2 = p2.y - p1.y, dz2 = p2.z - p1.z;
      const double dx3 = p3.x - p1.x, dy3 = p3.y - p1.y, dz3 = p3.z - p1.z;
      double d = (nfx * (dy2 * dz3 - dz2 * dy3) - nfy * (dx2 * dz3 - dz2 * dx3) + nfz * (dx2 * dy3 - dy2 * dx3));
      if (!(fabs(d) > 1.e-10)) continue;
      d = -(dx1 * (dy2 * dz3 - dz2 * dy3) - dy1 * (dx2 * dz3 - dz2 * dx3) + dz1 * (dx2 * dy3 - dy2 * dx3)) / d;
      if (!(d > 0)) continue;
      const V3 pint{p.x + d * nfx, p.y + d * nfy, p.z + d * nfz};
      const double rx1 = p2.x - p1.x, ry1 = p2.y - p1.y, rz1 = p2.z - p1.z;
      const double rx2 = p3.x - p1.x, ry2 = p3.y - p1.y, rz2 = p3.z - p1.z;
      const double nfxt = ry1 * rz2 - rz1 * ry2, nfyt = -rx1 * rz2 + rz1 * rx2, nfzt = rx1 * ry2 - ry1 * rx2;
      if (point_in_triangle(pint, p1, p2, p3, nfxt, nfyt, nfzt) >= 0) {
        double w[3] = {0., 0., 0.};
        project_bary(pint, p1, p2, p3, nfxt, nfyt, nfzt, w);
        nd.d_i = sqrt((pint.x - p.x) * (pint.x - p.x) + (pint.y - p.y) * (pint.y - p.y) +
                      (pint.z - p.z) * (pint.z - p.z));
        nd.imode = tr;
        for (int q = 0; q < 3; q++) {
          const int s = kPatchTri[tr][q];
          nd.ip[q] = ip[s]; nd.jp[q] = jp[s]; nd.kp[q] = kp[s];
          nd.cr[q] = w[q];
        }
        break;
      }
    }
  }
  nd.status = 0;
  if (nd.imode < 0) {
    int di = 0, dj = 0, dk = 0;
    if (i == 1 || i == g.mx - 2 || j == 1 || j == g.my - 2) {
      dk = (cell_min >= 0 && nf[3 * cell_min + 2] > 0) ? 1 : -1;
      nd.status = 1;
    } else if (k == 1 || k == g.mz - 2) {
      dj = 1;
      nd.status = 1;
    } else {
      nd.status = 2;
    }
    if (nd.status == 1) {
      const V3 c0 = p, c1 = vload(cent, g.at(i + di, j + dj, k + dk));
      nd.d_i = sqrt((c0.x - c1.x) * (c0.x - c1.x) + (c0.y - c1.y) * (c0.y - c1.y) + (c0.z - c1.z) * (c0.z - c1.z));
      nd.cr[0] = 1.; nd.cr[1] = 0.; nd.cr[2] = 0.;
      for (int q = 0; q < 3; q++) { nd.ip[q] = i + di; nd.jp[q] = j + dj; nd.kp[q] = k + dk; }
    }
  }
  out[n] = nd;
}

int fail(int code, const std::string &m) {
  set_last_error(m);
  return code;
}

bool on_device(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

}  // namespace

namespace {

// BoundingSphere (ibm.c:1282-1370): per element, a sphere through the
// longest edge's end points centred on the circumcentre side
void bounding_sphere(int n_elmt, const int32_t *tri, const std::vector<double> &x, const std::vector<double> &y,
                     const std::vector<double> &z, std::vector<double> &q, std::vector<double> &rad) {
  struct P { double x, y, z; };
  auto dist = [](P a, P b) {
    return std::sqrt((a.x - b.x) * (a.x - b.x) + (a.y - b.y) * (a.y - b.y) + (a.z - b.z) * (a.z - b.z));
  };
  const P p0{0., 0., 0.};
  q.assign((size_t)n_elmt * 3, 0.);
  rad.assign(n_elmt, 0.);
  for (int e = 0; e < n_elmt; e++) {
    const int n1 = tri[3 * e], n2 = tri[3 * e + 1], n3 = tri[3 * e + 2];
    const P p1{x[n1], y[n1], z[n1]}, p2{x[n2], y[n2], z[n2]}, p3{x[n3], y[n3], z[n3]};
    const double l12 = dist(p1, p2), l23 = dist(p2, p3), l31 = dist(p3, p1);
    P pa, pb, pc;
    if (l12 > l23) {
      if (l12 > l31) { pa = p1; pb = p2; pc = p3; } else { pa = p3; pb = p1; pc = p2; }
    } else {
      if (l31 < l23) { pa = p2; pb = p3; pc = p1; } else { pa = p3; pb = p1; pc = p2; }
    }
    const P pf{0.5 * (pa.x + pb.x), 0.5 * (pa.y + pb.y), 0.5 * (pa.z + pb.z)};
    const P pu{pa.x - pf.x, pa.y - pf.y, pa.z - pf.z}, pv{pc.x - pf.x, pc.y - pf.y, pc.z - pf.z};
    const P pt{pu.y * pv.z - pu.z * pv.y, pu.z * pv.x - pu.x * pv.z, pu.x * pv.y - pu.y * pv.x};
    const P pd{pt.y * pu.z - pt.z * pu.y, pt.z * pu.x - pt.x * pu.z, pt.x * pu.y - pt.y * pu.x};
    double gama = -(dist(pu, p0) * dist(pu, p0) - dist(pv, p0) * dist(pv, p0));
    const P pw{pv.x - pu.x, pv.y - pu.y, pv.z - pu.z};
    double lamda = 2 * (pd.x * pw.x + pd.y * pw.y + pd.z * pw.z);
    gama /= lamda;
    lamda = gama < 0 ? 0 : gama;
    const P qq{pf.x + lamda * pd.x, pf.y + lamda * pd.y, pf.z + lamda * pd.z};
    q[3 * e] = qq.x; q[3 * e + 1] = qq.y; q[3 * e + 2] = qq.z;
    rad[e] = dist(qq, pa);
  }
}

int ibm_search_impl(vfs_poisson *h, int ibi, int n_v, const double *xyz, int n_elmt, const int32_t *tri,
                    const int *bctype, double *nvert, int *n_failed, bool want_nodes, int *n_nodes) {
  if (!h || !xyz || !tri || !nvert || n_v < 3 || n_elmt < 1) return fail(VFS_EINVAL, "bad surface arguments");
  if (want_nodes && (ibi < 0 || ibi > 1023)) return fail(VFS_EINVAL, "body index out of range");
  IbmContext cx;
  int rc = ibm_context(h, &cx);
  if (rc != VFS_OK) return rc;
  const Grid g = cx.g;
  // the surface is small: it is prepared on the host (exact same double
  // operations as the reference's set-up loops)
  std::vector<double> x(n_v), y(n_v), z(n_v);
  for (int q = 0; q < n_v; q++) { x[q] = xyz[3 * q]; y[q] = xyz[3 * q + 1]; z[q] = xyz[3 * q + 2]; }
  for (int e = 0; e < 3 * n_elmt; e++)
    if (tri[e] < 0 || tri[e] >= n_v) return fail(VFS_EINVAL, "triangle vertex index out of range");
  HashBox H{1.e23, 1.e23, 1.e23, -1.e23, -1.e23, -1.e23, 0, 0, 0};
  for (int q = 0; q < n_v; q++) {
    H.xmin = std::min(H.xmin, x[q]); H.xmax = std::max(H.xmax, x[q]);
    H.ymin = std::min(H.ymin, y[q]); H.ymax = std::max(H.ymax, y[q]);
    H.zmin = std::min(H.zmin, z[q]); H.zmax = std::max(H.zmax, z[q]);
  }
  H.xmin -= 0.05; H.xmax += 0.05;
  H.ymin -= 0.05; H.ymax += 0.05;
  H.zmin -= 0.05; H.zmax += 0.05;
  H.dcx = (H.xmax - H.xmin) / (kHash - 1.);
  H.dcy = (H.ymax - H.ymin) / (kHash - 1.);
  H.dcz = (H.zmax - H.zmin) / (kHash - 1.);
  H.fcx = (float)H.dcx; H.fcy = (float)H.dcy; H.fcz = (float)H.dcz;
  H.rcx = (float)(1. / H.dcx); H.rcy = (float)(1. / H.dcy); H.rcz = (float)(1. / H.dcz);
  H.fz = (float)(H.zmax + 0.2 - H.zmin);
  const double extents = (H.xmax - H.xmin) + (H.ymax - H.ymin) + (H.zmax + 0.2 - H.zmin);
  H.L = extents <= 1e12 ? (float)extents : INFINITY;
  // everything the kernels read of the body in one buffer and one copy:
  // column starts, column entries (triangle and its top hash cell, sorted by
  // the latter, descending), vertices, normals, ray offsets, FP32 triangles
  std::vector<int> range((size_t)n_elmt * 5);  // hash columns of a triangle, its top cell
  std::vector<int> start(kHash * kHash + 1, 0);
  for (int e = 0; e < n_elmt; e++) {
    const int a = tri[3 * e], b = tri[3 * e + 1], c = tri[3 * e + 2];
    const double xv_min = std::min(std::min(x[a], x[b]), x[c]), xv_max = std::max(std::max(x[a], x[b]), x[c]);
    const double yv_min = std::min(std::min(y[a], y[b]), y[c]), yv_max = std::max(std::max(y[a], y[b]), y[c]);
    const double zv_max = std::max(std::max(z[a], z[b]), z[c]);
    int iv_min = (int)std::floor((xv_min - H.xmin) / H.dcx), iv_max = (int)std::floor((xv_max - H.xmin) / H.dcx) + 1;
    int jv_min = (int)std::floor((yv_min - H.ymin) / H.dcy), jv_max = (int)std::floor((yv_max - H.ymin) / H.dcy) + 1;
    int kv_max = (int)std::floor((zv_max - H.zmin) / H.dcz) + 1;
    iv_min = std::max(iv_min, 0); iv_max = std::min(iv_max, kHash);
    jv_min = std::max(jv_min, 0); jv_max = jv_max > kHash ? kHash : jv_max;
    kv_max = std::min(kv_max, kHash);
    const int r[5] = {iv_min, iv_max, jv_min, jv_max, kv_max};
    std::copy(r, r + 5, &range[(size_t)e * 5]);
    for (int jj = jv_min; jj < jv_max; jj++)
      for (int ii = iv_min; ii < iv_max; ii++) start[jj * kHash + ii + 1]++;
  }
  for (int q = 0; q < kHash * kHash; q++) start[q + 1] += start[q];
  const size_t entries = (size_t)start[kHash * kHash];
  size_t total = 0;
  auto place = [&](size_t bytes) {
    const size_t o = total;
    total += (std::max<size_t>(bytes, 1) + 15) & ~(size_t)15;
    return o;
  };
  const size_t o_start = place(start.size() * 4), o_tri = place(entries * 4), o_kmax = place(entries * 4),
               o_tv = place((size_t)n_elmt * 72), o_nf = place((size_t)n_elmt * 24), o_s = place((kMaxTries + 1) * 8),
               o_tf = place((size_t)n_elmt * 48);
  std::vector<double> pack((total + 7) / 8);
  unsigned char *pk = (unsigned char *)pack.data();
  int *col_tri = (int *)(pk + o_tri), *col_kmax = (int *)(pk + o_kmax);
  double *tv = (double *)(pk + o_tv), *nf = (double *)(pk + o_nf), *s_tab = (double *)(pk + o_s);
  float *tf = (float *)(pk + o_tf);
  std::copy(start.begin(), start.end(), (int *)(pk + o_start));
  // triangles by descending top cell, equal ones in their order (a stable
  // counting sort), dealt to their columns in that order
  {
    int first[kHash + 2] = {0};
    auto key = [&](int e) { return kHash - std::max(range[(size_t)e * 5 + 4], 0); };
    for (int e = 0; e < n_elmt; e++) first[key(e) + 1]++;
    for (int q = 0; q <= kHash; q++) first[q + 1] += first[q];
    std::vector<int> order(n_elmt), at(start.begin(), start.end());
    for (int e = 0; e < n_elmt; e++) order[first[key(e)]++] = e;
    for (int e : order) {
      const int *r = &range[(size_t)e * 5];
      for (int jj = r[2]; jj < r[3]; jj++)
        for (int ii = r[0]; ii < r[1]; ii++) {
          const int w = at[jj * kHash + ii]++;
          col_tri[w] = e;
          col_kmax[w] = r[4];
        }
    }
  }
  for (int e = 0; e < n_elmt; e++) {
    const int a = tri[3 * e], b = tri[3 * e + 1], c = tri[3 * e + 2];
    const double vv[9] = {x[a], y[a], z[a], x[b], y[b], z[b], x[c], y[c], z[c]};
    std::copy(vv, vv + 9, &tv[(size_t)e * 9]);
    // face normal as the UCD reader computes it (Source/ibm_io.c:997-1011)
    const double dx12 = x[b] - x[a], dy12 = y[b] - y[a], dz12 = z[b] - z[a];
    const double dx13 = x[c] - x[a], dy13 = y[c] - y[a], dz13 = z[c] - z[a];
    const double fx = dy12 * dz13 - dz12 * dy13, fy = -dx12 * dz13 + dz12 * dx13, fz = dx12 * dy13 - dy12 * dx13;
    const double dr = std::sqrt(fx * fx + fy * fy + fz * fz);
    nf[(size_t)e * 3] = fx / dr; nf[(size_t)e * 3 + 1] = fy / dr; nf[(size_t)e * 3 + 2] = fz / dr;
    const float f[12] = {(float)(x[a] - H.xmin), (float)(y[a] - H.ymin), (float)(z[a] - H.zmin),
                         (float)dx12, (float)dy12, (float)dz12, (float)dx13, (float)dy13, (float)dz13,
                         (float)(std::fabs(dx12) + std::fabs(dy12) + std::fabs(dz12)),
                         (float)(std::fabs(dx13) + std::fabs(dy13) + std::fabs(dz13)), 0.f};
    std::copy(f, f + 12, &tf[(size_t)e * 12]);
  }
  // (the offsets depend on nothing: formed once per process)
  static const std::vector<double> offsets = [] {
    std::vector<double> t(kMaxTries + 1, 0.);
    for (int q = 1; q <= kMaxTries; q++) t[q] = glibc_rand_first((unsigned)q) / ((double)2147483647 + 1) - 0.5;
    return t;
  }();
  std::copy(offsets.begin(), offsets.end(), s_tab);

  // device buffers of the handle's search (grown on demand): the body, two
  // masks, the is-4 bytes, and box[7], failed rays and the boundary flag
  const size_t N = g.n();
  IbmScratch &sc = *cx.scratch;
  void **buf = sc.buf;
  const int nbx = (g.mx - 2 + kCentBlock - 1) / kCentBlock, nby = (g.my - 2 + kCentBlock - 1) / kCentBlock,
            nbz = (g.mz - 2 + kCentBlock - 1) / kCentBlock, nblocks = nbx * nby * nbz;
  const bool dev = on_device(nvert);
  const size_t sizes[IbmScratch::kBufs] = {total, N * 8, dev && !want_nodes ? 0 : N * 8, N, 9 * 4,
                                           (size_t)nblocks * 6 * 8, (size_t)nblocks * 4};
  cudaStream_t st = cx.stream;
  for (int q = 0; q < IbmScratch::kBufs; q++)
    if (sc.cap[q] < sizes[q]) {
      if (buf[q]) {
        cudaStreamSynchronize(st);
        cudaFree(buf[q]);
      }
      buf[q] = nullptr;
      sc.cap[q] = 0;
      if (q == 5) sc.bbox_valid = false;
      if (cudaMalloc(&buf[q], sizes[q]) != cudaSuccess) {
        cudaGetLastError();
        buf[q] = nullptr;
        return fail(VFS_ENOMEM, "device allocation for the surface search failed");
      }
      sc.cap[q] = sizes[q];
    }
  cudaMemcpyAsync(buf[0], pk, total, cudaMemcpyHostToDevice, st);
  const unsigned char *db = (const unsigned char *)buf[0];
  const Surface S{H, (const int *)(db + o_start), (const int *)(db + o_tri), (const int *)(db + o_kmax),
                  (const double *)(db + o_tv), (const double *)(db + o_nf), (const double *)(db + o_s),
                  (const float4 *)(db + o_tf)};
  double *dnv = (double *)buf[1], *dtmp = (double *)buf[2], *bbox = (double *)buf[5];
  uint8_t *dis4 = (uint8_t *)buf[3];
  int *dbox = (int *)buf[4], *dfail = dbox + 7, *hits = (int *)buf[6];
  int b[6] = {0, 0, 0, 0, 0, 0};
  if (bctype)
    for (int q = 0; q < 6; q++) b[q] = bctype[q];
  Walls W;
  std::copy(b, b + 6, W.b);
  const dim3 gi((g.mx - 2 + 127) / 128, g.my - 2, g.mz - 2), gd((g.mx + 127) / 128, g.my, g.mz);
  int init[9] = {INT_MAX, INT_MAX, INT_MAX, INT_MIN, INT_MIN, INT_MIN, 0, 0, 0};
  cudaMemcpyAsync(dbox, init, sizeof(init), cudaMemcpyHostToDevice, st);
  if (!want_nodes) {
    // nvert is updated in place (a host array in its staged copy)
    double *nv = dev ? nvert : dtmp;
    if (!dev) cudaMemcpyAsync(dtmp, nvert, N * 8, cudaMemcpyHostToDevice, st);
    if (!sc.bbox_valid) {
      k_cent_blocks<<<nblocks, 512, 0, st>>>(g, cx.cent, nbx, nby, bbox);
      *cx.launches += 1;
      sc.bbox_valid = true;
    }
    int state[2] = {0, 0};
    auto read_state = [&] {
      cudaMemcpyAsync(state, dfail, sizeof(state), cudaMemcpyDeviceToHost, st);
      return cudaStreamSynchronize(st);
    };
    cudaError_t e = cudaSuccess;
    if (ibi == 0) {
      k_ibm_clear<<<152 * 8, 256, 0, st>>>(g, nv, dfail);
      *cx.launches += 1;
      e = read_state();
    }
    if (state[1]) {
      // a boundary point that counts as a 4 marks cells far from the body,
      // too: both passes over every point
      k_ibm_classify_from<<<gd, 128, 0, st>>>(g, cx.cent, 1, S, nv, dnv, dis4, dfail);
      k_ibm_dilate_finish_all<<<gd, 128, 0, st>>>(g, W, dnv, dis4, nv);
      *cx.launches += 2;
    } else {
      k_ibm_box_hits<<<(nblocks + 255) / 256, 256, 0, st>>>(bbox, nblocks, H, dbox, hits);
      k_ibm_box_cells<<<152 * 4, 256, 0, st>>>(g, cx.cent, nbx, nby, H, hits, dbox);
      k_ibm_classify<<<152 * 8, 128, 0, st>>>(g, cx.cent, S, dbox, nv, dnv, dis4, dfail);
      k_ibm_dilate_finish<<<152 * 8, 128, 0, st>>>(g, W, dbox, dnv, dis4, nv);
      *cx.launches += 4;
      if (ibi == 0 && std::any_of(b, b + 6, [](int v) { return v == -1 || v == -2; })) {
        k_ibm_finish<<<gi, 128, 0, st>>>(g, b[0], b[1], b[2], b[3], b[4], b[5], nv);
        *cx.launches += 1;
      }
    }
    if (e == cudaSuccess) e = read_state();
    if (e == cudaSuccess && !dev) e = cudaMemcpy(nvert, dtmp, N * 8, cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return fail(VFS_ECUDA, std::string("surface search: ") + cudaGetErrorString(e));
    }
    if (n_failed) *n_failed = state[0];
    if (n_nodes) *n_nodes = 0;
    return VFS_OK;
  }
  // with IB node records: every pass over all points (the classification
  // reads nvert where it lies; a host array is staged)
  const double *src = nvert;
  if (!dev) {
    cudaMemcpyAsync(dtmp, nvert, N * 8, cudaMemcpyHostToDevice, st);
    src = dtmp;
  }
  k_ibm_classify_from<<<gd, 128, 0, st>>>(g, cx.cent, ibi == 0, S, src, dnv, nullptr, dfail);
  k_ibm_dilate<<<gd, 128, 0, st>>>(g, dnv, dtmp);
  int nodes_found = 0;
  if (want_nodes) {  // the IB nodes (marked 2) and their interpolation records
    const int nb = (int)((N + 255) / 256);
    std::vector<double> q, rad;
    bounding_sphere(n_elmt, tri, x, y, z, q, rad);
    std::vector<int> bcount(nb), boff(nb + 1, 0);
    int *dcount = nullptr, *dlist = nullptr;
    double *dq = nullptr, *drad = nullptr;
    bool ok = cudaMalloc(&dcount, (size_t)nb * 4) == cudaSuccess;
    if (ok) {
      k_ibm_mark_count<<<nb, 256, 0, st>>>(g, dtmp, dcount);
      ok = cudaMemcpyAsync(bcount.data(), dcount, (size_t)nb * 4, cudaMemcpyDeviceToHost, st) == cudaSuccess &&
           cudaStreamSynchronize(st) == cudaSuccess;
    }
    if (ok) {
      for (int q2 = 0; q2 < nb; q2++) boff[q2 + 1] = boff[q2] + bcount[q2];
      nodes_found = boff[nb];
      ok = cudaMemcpyAsync(dcount, boff.data(), (size_t)nb * 4, cudaMemcpyHostToDevice, st) == cudaSuccess &&
           cudaMalloc(&dlist, (size_t)std::max(nodes_found, 1) * 4) == cudaSuccess &&
           cudaMalloc(&dq, q.size() * 8) == cudaSuccess && cudaMalloc(&drad, rad.size() * 8) == cudaSuccess;
    }
    IbmBody body;
    body.n_nodes = nodes_found;
    body.n_elmt = n_elmt;
    body.n_v = n_v;
    if (ok)
      ok = cudaMalloc(&body.nodes, (size_t)std::max(nodes_found, 1) * sizeof(vfs_ibm_node)) == cudaSuccess &&
           cudaMalloc(&body.tri, (size_t)n_elmt * 3 * 4) == cudaSuccess;
    if (ok) {
      cudaMemcpyAsync(dq, q.data(), q.size() * 8, cudaMemcpyHostToDevice, st);
      cudaMemcpyAsync(drad, rad.data(), rad.size() * 8, cudaMemcpyHostToDevice, st);
      cudaMemcpyAsync(body.tri, tri, (size_t)n_elmt * 3 * 4, cudaMemcpyHostToDevice, st);
      k_ibm_mark_scatter<<<nb, 256, 0, st>>>(g, dtmp, dcount, dlist);
      if (nodes_found > 0)
        k_ibm_nodes<<<(nodes_found + 127) / 128, 128, 0, st>>>(g, cx.cent, dlist, nodes_found, n_elmt,
                                                               S.tv, S.nf, dq, drad, body.nodes);
      *cx.launches += 3;
      ok = cudaStreamSynchronize(st) == cudaSuccess;
    }
    if (dcount) cudaFree(dcount);
    if (dlist) cudaFree(dlist);
    if (dq) cudaFree(dq);
    if (drad) cudaFree(drad);
    if (!ok) {
      cudaGetLastError();
      if (body.nodes) cudaFree(body.nodes);
      if (body.tri) cudaFree(body.tri);
      return fail(VFS_ECUDA, "IB node records: allocation or launch failed");
    }
    auto &B = *cx.bodies;
    if ((int)B.size() <= ibi) B.resize(ibi + 1);
    if (B[ibi].nodes) cudaFree(B[ibi].nodes);
    if (B[ibi].tri) cudaFree(B[ibi].tri);
    B[ibi] = body;
  }
  k_ibm_finish<<<gi, 128, 0, st>>>(g, b[0], b[1], b[2], b[3], b[4], b[5], dtmp);
  *cx.launches += 3;
  int nfail = 0;
  cudaMemcpyAsync(nvert, dtmp, N * 8, on_device(nvert) ? cudaMemcpyDeviceToDevice : cudaMemcpyDeviceToHost, st);
  cudaMemcpyAsync(&nfail, dfail, 4, cudaMemcpyDeviceToHost, st);
  cudaError_t e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    cudaGetLastError();
    return fail(VFS_ECUDA, std::string("surface search: ") + cudaGetErrorString(e));
  }
  if (n_failed) *n_failed = nfail;
  if (n_nodes) *n_nodes = nodes_found;
  return VFS_OK;
}

}  // namespace

extern "C" int vfs_poisson_ibm_search(vfs_poisson *h, int ibi, int n_v, const double *xyz, int n_elmt,
                                      const int32_t *tri, const int *bctype, double *nvert, int *n_failed) {
  return ibm_search_impl(h, ibi, n_v, xyz, n_elmt, tri, bctype, nvert, n_failed, false, nullptr);
}

extern "C" int vfs_poisson_ibm_search_nodes(vfs_poisson *h, int ibi, int n_v, const double *xyz, int n_elmt,
                                            const int32_t *tri, const int *bctype, double *nvert, int *n_failed,
                                            int *n_nodes) {
  return ibm_search_impl(h, ibi, n_v, xyz, n_elmt, tri, bctype, nvert, n_failed, true, n_nodes);
}

extern "C" int vfs_poisson_ibm_nodes(vfs_poisson *h, int ibi, vfs_ibm_node *nodes, int max_nodes, int *n_nodes) {
  if (!h || max_nodes < 0 || (max_nodes > 0 && !nodes)) return fail(VFS_EINVAL, "bad arguments");
  IbmContext cx;
  int rc = ibm_context(h, &cx);
  if (rc != VFS_OK) return rc;
  const auto &B = *cx.bodies;
  if (ibi < 0 || ibi >= (int)B.size() || !B[ibi].nodes) return fail(VFS_ESTATE, "no IB nodes for this body");
  const int n = B[ibi].n_nodes;
  if (n_nodes) *n_nodes = n;
  const int c = std::min(n, max_nodes);
  if (c > 0 && cudaMemcpy(nodes, B[ibi].nodes, (size_t)c * sizeof(vfs_ibm_node), cudaMemcpyDeviceToHost) !=
                   cudaSuccess) {
    cudaGetLastError();
    return fail(VFS_ECUDA, "copy of the IB node records failed");
  }
  return VFS_OK;
}

// ---- ibm_interpolation_advanced and IB_BC (launched by poisson.cu) ----
namespace vfs {

// noslip velocity and interpolated pressure at every IB node of one body
// (ibm.c:3405-3560, wallfunction.c:140-156), formed from lucat / lp, the arrays as
// they are (the reference's local copies), into val, four values a node: ucat and
// p are those arrays, and k_ibm_scatter writes them once every node has been read.
__global__ void k_ibm_gather(Grid g, const vfs_ibm_node *nodes, int n_nodes, const int *tri, const double *u_surf,
                             const double *nvert, const double *lucat, const double *lp, double *val) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_nodes) return;
  const vfs_ibm_node nd = nodes[n];
  const size_t t = g.at(nd.i, nd.j, nd.k);
  const size_t t1 = g.at(nd.ip[0], nd.jp[0], nd.kp[0]), t2 = g.at(nd.ip[1], nd.jp[1], nd.kp[1]),
               t3 = g.at(nd.ip[2], nd.jp[2], nd.kp[2]);
  const double sb = nd.d_s, sc = sb + nd.d_i;
  const double sk1 = nd.cr[0], sk2 = nd.cr[1], sk3 = nd.cr[2];
  double ua[3] = {0., 0., 0.};
  if (nd.cell >= 0 && u_surf) {
    const int v1 = tri[3 * nd.cell], v2 = tri[3 * nd.cell + 1], v3 = tri[3 * nd.cell + 2];
    for (int q = 0; q < 3; q++)
      ua[q] = u_surf[3 * v1 + q] * nd.cs[0] + u_surf[3 * v2 + q] * nd.cs[1] + u_surf[3 * v3 + q] * nd.cs[2];
  }
  if (nvert[t1] + nvert[t2] + nvert[t3] > 0.1 || nvert[t] > 2.9) {
    for (int q = 0; q < 3; q++) val[(size_t)n * 4 + q] = 0.;
  } else {
    for (int q = 0; q < 3; q++) {
      const double uc = (lucat[t1 * 3 + q] * sk1 + lucat[t2 * 3 + q] * sk2 + lucat[t3 * 3 + q] * sk3);
      const double uq = uc - ua[q];
      double v = sb / sc * uq;
      v += ua[q];
      val[(size_t)n * 4 + q] = v;
    }
  }
  val[(size_t)n * 4 + 3] = (lp[t1] * sk1 + lp[t2] * sk2 + lp[t3] * sk3);
}
__global__ void k_ibm_scatter(Grid g, const vfs_ibm_node *nodes, int n_nodes, const double *val, double *ucat,
                              double *p) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n >= n_nodes) return;
  const size_t t = g.at(nodes[n].i, nodes[n].j, nodes[n].k);
  for (int q = 0; q < 3; q++) ucat[t * 3 + q] = val[(size_t)n * 4 + q];
  p[t] = val[(size_t)n * 4 + 3];
}

__device__ inline double face_flux(const double *lu, size_t a, size_t b, const double *m) {
  const double ucx = (lu[a * 3] + lu[b * 3]) * 0.5;
  const double ucy = (lu[a * 3 + 1] + lu[b * 3 + 1]) * 0.5;
  const double ucz = (lu[a * 3 + 2] + lu[b * 3 + 2]) * 0.5;
  return ucx * m[0] + ucy * m[1] + ucz * m[2];
}

// the face fluxes around the IB nodes (ibm.c:3577-3630): every interior
// cell writes only its own three faces, so cells are independent.  A cell
// without a blanked point near has no such face: one byte of the 24 it would
// read of nvert, and no FP64.  u: ucat, whose periodic ghosts are read in
// their partners.
__global__ void k_ibm_faces(Grid g, Box b, const double *__restrict__ nvert, const uint8_t *__restrict__ near,
                            const double *__restrict__ lu, const double *icsi, const double *jeta, const double *kzet,
                            double f, int b0, int b1, int b2, int b3, int b4, int b5, double *ucont) {
  const size_t bc = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (bc >= b.n() || !near[bc]) return;
  int i, j, k;
  box_ijk(b, bc, i, j, k);
  i++, j++, k++;
  const size_t t = g.at(i, j, k), te = g.at(i + 1, j, k), tn = g.at(i, j + 1, k), tt = g.at(i, j, k + 1);
  const size_t ue = i == g.mx - 2 && g.px ? g.at(1, j, k) : te, un = j == g.my - 2 && g.py ? g.at(i, 1, k) : tn,
               ut = k == g.mz - 2 && g.pz ? g.at(i, j, 1) : tt;
  const bool wi0 = b0 == -1 || b0 == -2, wi1 = b1 == -1 || b1 == -2, wj0 = b2 == -1 || b2 == -2,
             wj1 = b3 == -1 || b3 == -2, wk0 = b4 == -1 || b4 == -2, wk1 = b5 == -1 || b5 == -2;
  if ((int)(nvert[t] + 0.5) == 1) {
    ucont[t * 3] = face_flux(lu, t, ue, &icsi[t * 3]) * f;
    ucont[t * 3 + 1] = face_flux(lu, un, t, &jeta[t * 3]) * f;
    ucont[t * 3 + 2] = face_flux(lu, ut, t, &kzet[t * 3]) * f;
    if (wi0 && i == 1) ucont[t * 3] = 0;
    if (wj0 && j == 1) ucont[t * 3 + 1] = 0;
    if (wk0 && k == 1) ucont[t * 3 + 2] = 0;
  }
  if ((int)(nvert[te] + 0.5) == 1) {
    ucont[t * 3] = face_flux(lu, t, ue, &icsi[t * 3]) * f;
    if (wi1 && i == g.mx - 3) ucont[t * 3] = 0;
  }
  if ((int)(nvert[tn] + 0.5) == 1) {
    ucont[t * 3 + 1] = face_flux(lu, un, t, &jeta[t * 3]) * f;
    if (wj1 && j == g.my - 3) ucont[t * 3 + 1] = 0;
  }
  if ((int)(nvert[tt] + 0.5) == 1) {
    ucont[t * 3 + 2] = face_flux(lu, ut, t, &kzet[t * 3]) * f;
    if (wk1 && k == g.mz - 3) ucont[t * 3 + 2] = 0;
  }
}

// IB_BC's interior loop (momentum.c:2114-2178): the IB faces from ucat
// ((int)nvert == 1), the immersed == 3 zeroing and the -1/-2 walls in i and
// j (the i == 1 / j == 1 rows write the face below them, which no other cell
// of this loop writes); the mask is looked at next to a body only
__global__ void k_ib_bc_faces(Grid g, Box b, const double *__restrict__ nvert, const uint8_t *__restrict__ near,
                              const double *lu, const double *icsi, const double *jeta, const double *kzet,
                              int immersed, int b0, int b1, int b2, int b3, double *ucont) {
  const size_t bc = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (bc >= b.n()) return;
  int i, j, k;
  box_ijk(b, bc, i, j, k);
  i++, j++, k++;
  const size_t t = g.at(i, j, k), te = g.at(i + 1, j, k), tn = g.at(i, j + 1, k), tt = g.at(i, j, k + 1);
  if (immersed && near[bc]) {
    const double f = immersed == 3 ? 0. : 1.;
    if ((int)nvert[t] == 1) {
      ucont[t * 3] = face_flux(lu, t, te, &icsi[t * 3]) * f;
      ucont[t * 3 + 1] = face_flux(lu, tn, t, &jeta[t * 3]) * f;
      ucont[t * 3 + 2] = face_flux(lu, tt, t, &kzet[t * 3]) * f;
    }
    if ((int)(nvert[te]) == 1) ucont[t * 3] = face_flux(lu, t, te, &icsi[t * 3]) * f;
    if ((int)(nvert[tn]) == 1) ucont[t * 3 + 1] = face_flux(lu, tn, t, &jeta[t * 3]) * f;
    if ((int)(nvert[tt]) == 1) ucont[t * 3 + 2] = face_flux(lu, tt, t, &kzet[t * 3]) * f;
    if (immersed == 3) {
      if ((nvert[te] + nvert[t]) > 1.1) ucont[t * 3] = 0;
      if ((nvert[tn] + nvert[t]) > 1.1) ucont[t * 3 + 1] = 0;
      if ((nvert[tt] + nvert[t]) > 1.1) ucont[t * 3 + 2] = 0;
    }
  }
  const bool wi0 = b0 == -1 || b0 == -2, wi1 = b1 == -1 || b1 == -2, wj0 = b2 == -1 || b2 == -2,
             wj1 = b3 == -1 || b3 == -2;
  if ((wi0 && i == 1) || (wi1 && i == g.mx - 2)) {
    if (i == 1) ucont[g.at(i - 1, j, k) * 3] = 0;
    else ucont[t * 3] = 0;
  }
  if ((wj0 && j == 1) || (wj1 && j == g.my - 2)) {
    if (j == 1) ucont[g.at(i, j - 1, k) * 3 + 1] = 0;
    else ucont[t * 3 + 1] = 0;
  }
}

// IB_BC's closing loop over every DA point (momentum.c:2180-2210): the slip
// (10) walls and the periodic faces.  The reference runs it in place in
// k, j, i order; a periodic copy there reads its partner before a slip rule
// of the same row could zero it, so every value follows from the values
// before the loop.  Component q changes at the ends of the lines along axis
// q only, and no other line reads it: one thread a line takes both partners
// before it writes, in place (the whole array was copied and rewritten
// before: 192x128x192 71 -> 3 us).
__global__ void k_ib_bc_edges(Grid g, int b0, int b1, int b2, int b3, int b4, int b5, double *ucont) {
  const uint32_t nx = (uint32_t)g.my * g.mz, ny = (uint32_t)g.mx * g.mz, nz = (uint32_t)g.mx * g.my;
  uint32_t u = blockIdx.x * blockDim.x + threadIdx.x;
  int q, m, per, lo, hi;
  size_t base, step;
  if (u < nx) {
    q = 0; m = g.mx; per = g.px; lo = b0; hi = b1;
    base = (size_t)u * g.mx;
    step = 1;
  } else if ((u -= nx) < ny) {
    q = 1; m = g.my; per = g.py; lo = b2; hi = b3;
    const uint32_t k = u / (uint32_t)g.mx;
    base = g.at((int)(u - k * g.mx), 0, (int)k);
    step = g.mx;
  } else if ((u -= ny) < nz) {
    q = 2; m = g.mz; per = g.pz; lo = b4; hi = b5;
    base = u;
    step = (size_t)g.mx * g.my;
  } else {
    return;
  }
  double *line = ucont + base * 3 + q;
  step *= 3;
  const double first = line[step], last = line[(m - 2) * step];
  if (per) {
    line[0] = last;
    line[(m - 1) * step] = first;
  }
  if (lo == 10) line[0] = 0;
  if (hi == 10) line[(m - 2) * step] = 0;
}

}  // namespace vfs
