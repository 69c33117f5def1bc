// vtail.cu -- the tail of the V-cycle: every level from the first small one
// to the coarsest and back, as one kernel of one thread-block cluster.
//
// A launch of a small level costs 3.5-4.5 us whatever its size (wait for the
// predecessor, one round trip to L2 for x, drain), and a level takes ten of
// them.  Here a phase (one colour of a sweep, a residual, a transfer) ends in
// a cluster barrier instead, x and the right-hand sides never leave shared
// memory, and the operator is read from global memory once per V-cycle.
// Planes of constant k are dealt to the CTAs in slabs, so that a j-line stays
// in one CTA and only the two planes next to a slab are foreign: the owner of
// a border plane stores new values into its neighbour's copy of the plane too
// (distributed shared memory), and every stencil read is local.  The
// restriction and the prolongation read the few foreign planes they need in
// their owner's memory.  What bounds a phase is latency: of 2.6 us at 16^3
// cells, 1.0 are a cell's residual (one warp a quarter of an SM), 0.8 the
// recurrences, 0.5 the stores, 0.3 the barrier.  Four levels from 24x16x24
// cells on take 46 us instead of 95, three from 16^3 on 40 instead of 72.
//
// The arithmetic is that of the kernels it replaces, operation for operation
// (k_residual16 / k_residual_f64, k_line_tri_*, k_restrict_*, k_prolong_*,
// k_coarsest_*), so that the V-cycle's result is the same bits.
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.cuh"

namespace cg = cooperative_groups;

namespace vfs {

namespace {

// products and sums that setup.cu's transfers round one by one
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }

extern __shared__ __align__(16) unsigned char sm[];

// n bytes from global to shared memory, asynchronously, W at a time
template <int W>
__device__ __forceinline__ void copy_async(uint32_t dst, const unsigned char *src, uint32_t n) {
  for (uint32_t e = threadIdx.x * W; e < n; e += kTailThreads * W) {
    if constexpr (W == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + e), "l"(src + e) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(dst + e), "l"(src + e), "n"(W) : "memory");
  }
}
// the same for any alignment: the widest copies the addresses allow (dst is
// aligned like src), bytes one by one where they allow none
__device__ __forceinline__ void copy_any(uint32_t dst, const void *from, uint32_t n) {
  const unsigned char *src = (const unsigned char *)from;
  const uint32_t al = (uint32_t)(uintptr_t)src | dst;
  const uint32_t m = (al & 15) == 0 ? n & ~15u : (al & 3) == 0 ? n & ~3u : 0u;
  if ((al & 15) == 0) copy_async<16>(dst, src, m);
  else if ((al & 3) == 0) copy_async<4>(dst, src, m);
  unsigned char *d = sm + (dst - (uint32_t)__cvta_generic_to_shared(sm));
#pragma unroll 4
  for (uint32_t e = m + threadIdx.x; e < n; e += kTailThreads) d[e] = src[e];
}
// a shared-memory address in CTA `rank` of the cluster, and accesses through one
__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void store_remote(uint32_t addr, float v) {
  asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ void store_remote(uint32_t addr, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void load_remote(uint32_t addr, float &v) {
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
}
__device__ __forceinline__ void load_remote(uint32_t addr, double &v) {
  asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(addr));
}

// planes of a level's operator in shared memory (words of 4 or 8 bytes):
// FP32: 10 packed couplings, D, S slot, inv, cp; FP64: 19 slots, inv, cp
template <typename T>
constexpr int kOpPlanes = sizeof(T) == 4 ? 14 : 21;

// One level as this CTA sees it (formed once per kernel, in shared memory):
// planes [k0, k1); lo, hi: the CTAs holding a copy of the first and of the
// last of them (-1: none); slab: words of a plane.
struct Slab {
  TailLevel l;
  int k0, k1, lo, hi, nh;
  uint32_t slab;

  __device__ void form(int rank) {
    const Box &b = l.b;
    nh = (b.nx + 1) >> 1;
    slab = (uint32_t)l.rs * b.ny;
    k0 = min(rank * l.q, b.nz);
    k1 = min(k0 + l.q, b.nz);
    lo = hi = -1;
    if (k0 < k1) {
      const int below = k0 > 0 ? k0 - 1 : (b.pz ? b.nz - 1 : 0), above = k1 < b.nz ? k1 : (b.pz ? 0 : b.nz - 1);
      if (below < k0 || below >= k1) lo = (int)l.dq.div(below);
      if (above < k0 || above >= k1) hi = (int)l.dq.div(above);
    }
  }
  __device__ __forceinline__ int planes() const { return k1 - k0; }
  // x-like vectors hold q + 2 planes: a copy of the plane below the slab, the slab, a copy of the plane above
  __device__ __forceinline__ uint32_t slot(int k) const { return (uint32_t)(k - k0 + 1) * slab; }
  __device__ __forceinline__ uint32_t slot_at(int m, uint32_t foreign) const {
    return m >= k0 && m < k1 ? slot(m) : foreign;
  }
};

// Operator pointers: element 0 is the first row of plane k0, rows rs apart,
// planes of coefficients st apart.
template <typename T>
struct Op {
  uint32_t st, rs;
  const __half2 *C;
  const T *D, *A, *S, *inv, *cp;
  __device__ __forceinline__ explicit Op(const Slab &v) {
    const TailLevel &l = v.l;
    if (l.res) {
      st = (uint32_t)l.q * v.slab;
      rs = l.rs;
      const T *o = (const T *)(sm + l.oA);
      if constexpr (sizeof(T) == 4) {
        C = (const __half2 *)o;
        D = o + 10 * st;
        S = o + 11 * st;
        inv = o + 12 * st;
        cp = o + 13 * st;
      } else {
        A = o;
        S = o + SP * st;
        inv = o + 19 * st;
        cp = o + 20 * st;
      }
    } else {
      const uint32_t plane = (uint32_t)l.b.nx * l.b.ny, base = (uint32_t)v.k0 * plane;
      st = plane * (uint32_t)l.b.nz;
      rs = l.b.nx;
      if constexpr (sizeof(T) == 4) {
        C = (const __half2 *)l.A + base;
        D = (const T *)l.D + base;
      } else {
        A = (const T *)l.A + base;
      }
      S = (const T *)l.Asp + base;
      inv = (const T *)l.inv + base;
      cp = (const T *)l.cp + base;
    }
  }
};

// Where the new values of a slab's border planes go besides the slab itself:
// the neighbours' copies of vector xd.
template <typename T>
struct Halo {
  uint32_t lo, hi;  // addresses of the plane's word 0 (0: no copy)
  __device__ __forceinline__ Halo(const Slab &v, const T *xd) {
    const uint32_t s = smem_addr(xd);
    lo = v.lo >= 0 ? map_rank(s + (uint32_t)(v.l.q + 1) * v.slab * (uint32_t)sizeof(T), v.lo) : 0u;
    hi = v.hi >= 0 ? map_rank(s, v.hi) : 0u;
  }
};

// The 19 values of cell (i, j, k) in slot order: columns of the parity of
// (i + k) from xo, the others from xn.
template <typename T>
__device__ __forceinline__ void stencil_values(const Slab &v, const T *xo, const T *xn, int i, int j, int k,
                                               T (&xs)[NSLOT]) {
  const Box &b = v.l.b;
  const int im = i > 0 ? i - 1 : (b.px ? b.nx - 1 : i), ip = i < b.nx - 1 ? i + 1 : (b.px ? 0 : i);
  const int km = k > 0 ? k - 1 : (b.pz ? b.nz - 1 : k), kp = k < b.nz - 1 ? k + 1 : (b.pz ? 0 : k);
  const int jm = j > 0 ? j - 1 : (b.py ? b.ny - 1 : j), jp = j < b.ny - 1 ? j + 1 : (b.py ? 0 : j);
  const int s0 = v.slot(k), sl = v.slot_at(km, 0u), su = v.slot_at(kp, (uint32_t)(v.l.q + 1) * v.slab);
  const int pc = (i & 1 ? v.nh : 0) + (i >> 1), pe = (ip & 1 ? v.nh : 0) + (ip >> 1), pw = (im & 1 ? v.nh : 0) + (im >> 1);
  const int r0 = j * v.l.rs, rm = jm * v.l.rs, rp = jp * v.l.rs;
  auto col = [&](int ii, int kk) { return ((ii + kk) ^ (i + k)) & 1 ? xn : xo; };
  const T *c = xo + s0 + pc, *e = col(ip, k) + s0 + pe, *w = col(im, k) + s0 + pw, *t = col(i, kp) + su + pc,
          *bt = col(i, km) + sl + pc;
  xs[CP] = c[r0];
  xs[EP] = e[r0];
  xs[WP] = w[r0];
  xs[NP] = c[rp];
  xs[SP] = c[rm];
  xs[TP] = t[r0];
  xs[BP] = bt[r0];
  xs[NE] = e[rp];
  xs[SE] = e[rm];
  xs[NW] = w[rp];
  xs[SW] = w[rm];
  xs[TN] = t[rp];
  xs[BN] = bt[rp];
  xs[TS] = t[rm];
  xs[BS] = bt[rm];
  xs[TE] = (col(ip, kp) + su + pe)[r0];
  xs[BE] = (col(ip, km) + sl + pe)[r0];
  xs[TW] = (col(im, kp) + su + pw)[r0];
  xs[BW] = (col(im, km) + sl + pw)[r0];
}

// rhs - A x of a cell from its 19 values; FP32: the difference form over the
// packed couplings, in the order of k_residual16.
__device__ __forceinline__ float row_residual(const Op<float> &o, uint32_t row, float rhs, const float (&xs)[NSLOT]) {
  const float xc = xs[CP];
  float s = 0.f;
#pragma unroll
  for (int m = 0; m < 9; m++) {
    const float2 f = __half22float2(o.C[m * o.st + row]);
    s = fmaf(f.x, xs[2 * m + 1] - xc, s);
    s = fmaf(f.y, xs[2 * m + 2] - xc, s);
  }
  s = fmaf(__low2float(o.C[9 * o.st + row]), xc, s);
  return fmaf(-o.D[row], s, rhs);
}
__device__ __forceinline__ double row_residual(const Op<double> &o, uint32_t row, double rhs,
                                               const double (&xs)[NSLOT]) {
  double s = 0.;
#pragma unroll
  for (int m = 0; m < NSLOT; m++) s = fma(o.A[m * o.st + row], xs[m], s);
  return rhs - s;
}

// What a phase does with the cells of one colour: a sweep's colour (from a
// zero guess: the residual is b), or the weighted residual that is restricted
// (kWeighted1: the other colour's is zero).
enum { kSweep, kSweepZero, kWeighted, kWeighted1 };

// FP32.  A unit is a chunk of 8 rows of 4 columns, one cell a lane: the
// operator rows (stride 4 times an odd number of words) and the columns'
// split positions make every read of the warp conflict-free, a unit's chunk
// recurrences run through shuffles of its 8 lanes, and only the joins of a
// column's chunks go through shared memory (ends).  One lane a chunk took
// 2.4 times as long: 8 cells' worth of straight-line code for one warp.
__device__ __noinline__ void phase32(const Slab &v, uint32_t oxo, uint32_t oxn, uint32_t oxd, float omega, int color,
                                     int mode, float2 *ends) {
  const TailLevel &l = v.l;
  const Op<float> o(v);
  const float *xo = (const float *)(sm + oxo), *xn = (const float *)(sm + oxn), *bb = (const float *)(sm + l.ob);
  float *own = (float *)(sm + (mode >= kWeighted ? l.orr : oxd + v.slab * 4u));
  const int nx = l.b.nx, ny = l.b.ny, P = l.P, rs = l.rs, nh = v.nh, k0 = v.k0;
  const int lane = threadIdx.x & 31, e = lane & 7, warp = threadIdx.x >> 5;
  const int units = (v.k1 - k0) * l.nq * P;
  struct Unit {
    int kl, k, t, m, par, j, ch;
  };
  const FastDiv dP = l.dP, dnq = l.dnq;
  const int nq = l.nq;
  auto unit = [&](int u) {
    Unit a;
    const int rest = (int)dP.div(u);
    a.ch = u - rest * P;
    a.kl = (int)dnq.div(rest);
    a.k = k0 + a.kl;
    a.t = (rest - a.kl * nq) * 4 + (lane >> 3);
    a.par = (color + a.k) & 1;
    a.m = a.par ? nx - nh : nh;
    a.j = a.ch * kLineChunk + e;
    return a;
  };
#pragma unroll 1
  for (int u = warp; u < units; u += kTailThreads / 32) {
    const Unit a = unit(u);
    const bool in = a.t < a.m && a.j < ny;
    // (a lane without a cell reads another one's)
    const int t = max(min(a.t, a.m - 1), 0), j = min(a.j, ny - 1), i = min(2 * t + a.par, nx - 1),
              p = min(a.par ? nh + t : t, nx - 1), row = a.kl * ny + j, at = row * rs + p;
    float y = bb[at];
    float w = 0.f;
    if (mode >= kWeighted) w = ((const float *)l.w)[(uint32_t)(k0 * ny + row) * nx + i];
    if (mode != kSweepZero) {
      float xs[NSLOT];
      stencil_values<float>(v, xo, xn, i, j, a.k, xs);
      y = row_residual(o, row * o.rs + p, y, xs);
    }
    if (mode >= kWeighted) y = mul_rn(y, w);
    if (in) own[at] = y;
    if (mode == kWeighted1 && a.j < ny && a.t < nx - a.m) own[row * rs + (a.par ? a.t : nh + a.t)] = 0.f;
  }
  if (mode >= kWeighted) return;
  constexpr int U = kTailUnits / (kTailThreads / 32);
  float y[U], g[U], c[U];
#pragma unroll
  for (int m = 0; m < U; m++) {
    const int u = warp + m * (kTailThreads / 32);
    if (u < units) {
      const Unit a = unit(u);
      const int t = max(min(a.t, a.m - 1), 0), j = min(a.j, ny - 1), p = min(a.par ? nh + t : t, nx - 1),
                row = a.kl * ny + j, at = row * o.rs + p;
      const float av = a.j > 0 ? o.S[at] : 0.f, iv = o.inv[at], r = own[row * rs + p];
      c[m] = a.j < ny - 1 ? o.cp[at] : 0.f;
      const float f = -av * iv;
      float Y = (r - av * 0.f) * iv, G = f;
#pragma unroll
      for (int s = 1; s < kLineChunk; s++) {
        const float yp = __shfl_up_sync(0xffffffffu, Y, 1, 8), gp = __shfl_up_sync(0xffffffffu, G, 1, 8);
        if (e == s) {
          Y = (r - av * yp) * iv;
          G = gp * f;
        }
      }
      y[m] = Y;
      g[m] = G;
      const int last = min(kLineChunk, ny - a.ch * kLineChunk) - 1;
      if (P > 1 && e == last) ends[u * 4 + (lane >> 3)] = make_float2(Y, G);
    }
  }
  if (P > 1) __syncthreads();
#pragma unroll
  for (int m = 0; m < U; m++) {
    const int u = warp + m * (kTailThreads / 32);
    if (u < units) {
      const int ch = u - (int)dP.div(u) * P, cnt = min(kLineChunk, ny - ch * kLineChunk);
      if (P > 1) {
        float Y = 0.f;
        for (int s = 0; s < ch; s++) {
          const float2 q = ends[(u - ch + s) * 4 + (lane >> 3)];
          Y = q.x + q.y * Y;
        }
        y[m] += g[m] * Y;
      }
      const float r = y[m];
      float X = r, H = -c[m];
#pragma unroll
      for (int s = kLineChunk - 2; s >= 0; s--) {
        const float xp = __shfl_down_sync(0xffffffffu, X, 1, 8), hp = __shfl_down_sync(0xffffffffu, H, 1, 8);
        if (e == s && s < cnt - 1) {
          X = r - c[m] * xp;
          H = hp * -c[m];
        }
      }
      y[m] = X;
      g[m] = H;
    }
  }
  if (P > 1) {
    __syncthreads();  // (ends is read above)
#pragma unroll
    for (int m = 0; m < U; m++) {
      const int u = warp + m * (kTailThreads / 32);
      if (u < units && e == 0) ends[u * 4 + (lane >> 3)] = make_float2(y[m], g[m]);
    }
    __syncthreads();
  }
  const Halo<float> halo(v, (const float *)(sm + oxd));
#pragma unroll
  for (int m = 0; m < U; m++) {
    const int u = warp + m * (kTailThreads / 32);
    if (u < units) {
      const Unit a = unit(u);
      if (P > 1) {
        float X = 0.f;
        for (int s = P - 1; s > a.ch; s--) {
          const float2 q = ends[(u - a.ch + s) * 4 + (lane >> 3)];
          X = q.x + q.y * X;
        }
        y[m] += g[m] * X;
      }
      if (a.t < a.m && a.j < ny) {
        const uint32_t pl = (uint32_t)(a.j * rs + (a.par ? nh + a.t : a.t)), at = a.kl * v.slab + pl;
        const float old = mode == kSweepZero ? 0.f : xo[v.slab + at], val = old + omega * y[m];
        own[at] = val;
        if (halo.lo && a.kl == 0) store_remote(halo.lo + pl * 4u, val);
        if (halo.hi && a.k == v.k1 - 1) store_remote(halo.hi + pl * 4u, val);
      }
    }
  }
}

// FP64.  A lane's FP64 operation holds its quarter of the SM for 64 cycles
// whether 32 lanes work or one: the residuals are spread over all warps, one
// lane a cell (r), and the lines over as few as hold them, one lane a chunk
// of 8 cells, the P chunks of a column in lanes ch cw + c of one warp and
// joined by shuffles.
__device__ __noinline__ void phase64(const Slab &v, uint32_t oxo, uint32_t oxn, uint32_t oxd, double omega, int color,
                                     int mode) {
  constexpr int M = kLineChunk;
  const TailLevel &l = v.l;
  const Op<double> o(v);
  const double *xo = (const double *)(sm + oxo), *xn = (const double *)(sm + oxn), *bb = (const double *)(sm + l.ob);
  double *r = (double *)(sm + l.orr);
  const int nx = l.b.nx, ny = l.b.ny, P = l.P, cw = l.cw, rs = l.rs, nh = v.nh, ncol = v.planes() * nh;
  if (mode != kSweepZero) {
    const uint32_t cells = (uint32_t)(v.planes() * ny * nh);
    for (uint32_t q = threadIdx.x; q < cells; q += kTailThreads) {
      const uint32_t row = l.dnh.div(q), kl = l.b.dy.div(row);
      const int t = (int)(q - row * nh), j = (int)(row - kl * ny), k = v.k0 + (int)kl, par = (color + k) & 1;
      if (t < (par ? nx - nh : nh)) {
        const uint32_t p = par ? nh + t : t, at = row * rs + p;
        double xs[NSLOT];
        stencil_values<double>(v, xo, xn, 2 * t + par, j, k, xs);
        double y = row_residual(o, row * o.rs + p, bb[at], xs);
        if (mode >= kWeighted) y = mul_rn(y, ((const double *)l.w)[(uint32_t)(v.k0 * ny + row) * nx + 2 * t + par]);
        r[at] = y;
      }
      if (mode == kWeighted1 && t < (par ? nh : nx - nh)) r[row * rs + (par ? t : nh + t)] = 0.;
    }
    if (mode >= kWeighted) return;
    __syncthreads();
  }
  const double *rhs = mode == kSweepZero ? bb : r;
  const int lane = threadIdx.x & 31, ch = (int)l.dcw.div((uint32_t)lane), c = lane - ch * cw, j0 = ch * M;
  const Halo<double> halo(v, (const double *)(sm + oxd));
  double *own = (double *)(sm + oxd);
  for (int c0 = (int)(threadIdx.x >> 5) * cw; c0 < ncol; c0 += (kTailThreads / 32) * cw) {
    const int col = min(c0 + c, ncol - 1), kl = (int)l.dnh.div((uint32_t)col), t = col - kl * nh, k = v.k0 + kl;
    const int par = (color + k) & 1, m = par ? nx - nh : nh;
    const int cnt = c0 + c < ncol && ch < P && t < m ? max(0, min(M, ny - j0)) : 0;
    // (a lane without a chunk reads in bounds and stores nothing)
    const int tt = max(min(t, m - 1), 0), p = min(par ? nh + tt : tt, nx - 1);
    double y[M], iv[M], f[M], g[M];
    double yp = 0., gp = 1.;
#pragma unroll
    for (int e = 0; e < M; e++) {
      const int row = kl * ny + min(j0 + e, ny - 1), at = row * o.rs + p;
      f[e] = j0 + e > 0 ? o.S[at] : 0.;
      iv[e] = o.inv[at];
      y[e] = rhs[row * rs + p];
    }
#pragma unroll
    for (int e = 0; e < M; e++) {
      if (e < cnt) {
        yp = (y[e] - f[e] * yp) * iv[e];
        gp = gp * (-f[e] * iv[e]);
      }
      y[e] = yp;
      g[e] = gp;
    }
    if (P > 1) {
      double Y = 0., in = 0.;
      for (int s = 0; s < P; s++) {
        const double ye = __shfl_sync(0xffffffffu, yp, s * cw + c), G = __shfl_sync(0xffffffffu, gp, s * cw + c);
        if (s == ch) in = Y;
        Y = ye + G * Y;
      }
#pragma unroll
      for (int e = 0; e < M; e++) y[e] += g[e] * in;
    }
#pragma unroll
    for (int e = 0; e < M; e++)
      f[e] = j0 + e < ny - 1 ? o.cp[(kl * ny + min(j0 + e, ny - 1)) * o.rs + p] : 0.;
    double xl = 0., hp = 1.;
#pragma unroll
    for (int e = M - 1; e >= 0; e--) {
      if (e < cnt) {
        xl = y[e] - f[e] * xl;
        hp = hp * (-f[e]);
      }
      y[e] = xl;
      g[e] = hp;
    }
    if (P > 1) {
      double X = 0., in = 0.;
      for (int s = P - 1; s >= 0; s--) {
        const double xe = __shfl_sync(0xffffffffu, xl, s * cw + c), H = __shfl_sync(0xffffffffu, hp, s * cw + c);
        if (s == ch) in = X;
        X = xe + H * X;
      }
#pragma unroll
      for (int e = 0; e < M; e++) y[e] += g[e] * in;
    }
    const bool lo = halo.lo && k == v.k0, hi = halo.hi && k == v.k1 - 1;
#pragma unroll
    for (int e = 0; e < M; e++) {
      if (e < cnt) {
        const uint32_t pl = (uint32_t)((j0 + e) * rs + p), at = v.slot(k) + pl;
        const double val = (mode == kSweepZero ? 0. : xo[at]) + omega * y[e];
        own[at] = val;
        if (lo) store_remote(halo.lo + pl * 8u, val);
        if (hi) store_remote(halo.hi + pl * 8u, val);
      }
    }
  }
}

// MyRestriction of the weighted residuals onto the next level's right-hand side
template <typename T>
__device__ __noinline__ void restrict_phase(const Slab &f, const Slab &c) {
  const TailLevel &l = f.l, &lc = c.l;
  T *bc = (T *)(sm + lc.ob);
  const int cny = lc.b.ny, cnx = lc.b.nx;
  const uint8_t *blank = sm + lc.obl + (uint32_t)(c.k0 * cny) * cnx;
  const uint32_t rf = smem_addr(sm) + l.orr, cells = (uint32_t)(c.planes() * cny * cnx);
  for (uint32_t e = threadIdx.x; e < cells; e += kTailThreads) {
    const uint32_t row = lc.b.dx.div(e), kl = lc.b.dy.div(row);
    const int i = (int)(e - row * cnx), j = (int)(row - kl * cny), k = c.k0 + (int)kl;
    const int i1 = l.cx ? 2 * i + 1 : i, j1 = l.cy ? 2 * j + 1 : j, k1 = l.cz ? 2 * k + 1 : k;
    const int i0 = i1 - l.cx, j0 = j1 - l.cy, k0 = k1 - l.cz;
    const uint32_t o1 = l.dq.div(k1), o0 = l.dq.div(k0);
    const uint32_t p1 = map_rank(rf, o1) + (k1 - o1 * l.q) * f.slab * (uint32_t)sizeof(T),
                   p0 = map_rank(rf, o0) + (k0 - o0 * l.q) * f.slab * (uint32_t)sizeof(T);
    const int q1 = split_pos(i1, l.b.nx), q0 = split_pos(i0, l.b.nx);
    const uint32_t a11 = (j1 * l.rs + q1) * sizeof(T), a01 = (j1 * l.rs + q0) * sizeof(T),
                   a10 = (j0 * l.rs + q1) * sizeof(T), a00 = (j0 * l.rs + q0) * sizeof(T);
    T v1, v2, v3, v4, v5, v6, v7, v8;
    load_remote(p1 + a11, v1);
    load_remote(p1 + a01, v2);
    load_remote(p1 + a10, v3);
    load_remote(p0 + a11, v4);
    load_remote(p1 + a00, v5);
    load_remote(p0 + a10, v6);
    load_remote(p0 + a01, v7);
    load_remote(p0 + a00, v8);
    const T s = add_rn(add_rn(add_rn(add_rn(add_rn(add_rn(add_rn(v1, v2), v3), v4), v5), v6), v7), v8);
    bc[row * lc.rs + split_pos(i, cnx)] = blank[e] ? (T)0 : mul_rn((T)0.125, s);
  }
}

// MyInterpolation of the next level's correction (byte offset oc), added onto
// x (byte offset ox); first: the fine level's flags are the CTA's planes'
template <typename T>
__device__ __noinline__ void prolong_phase(const Slab &f, const Slab &cs, bool first, uint32_t oc, uint32_t ox) {
  const TailLevel &l = f.l, &lc = cs.l;
  const Box &b = l.b, &cb = lc.b;
  T *x = (T *)(sm + ox);
  const Halo<T> halo(f, x);
  const int cnx = cb.nx, cnxy = cnx * cb.ny;
  const uint32_t xc = smem_addr(sm) + oc;
  const uint8_t *bf = sm + l.obl + (first ? 0u : (uint32_t)(f.k0 * b.ny) * b.nx), *bc = sm + lc.obl;
  const uint32_t cells = (uint32_t)(f.planes() * b.ny * b.nx);
  for (uint32_t e = threadIdx.x; e < cells; e += kTailThreads) {
    const uint32_t row = b.dx.div(e), kl = b.dy.div(row);
    const int I = (int)(e - row * b.nx) + 1, J = (int)(row - kl * b.ny) + 1, K = f.k0 + (int)kl + 1;
    int ic = I, jc = J, kc = K, ia = 0, ja = 0, ka = 0;
    if (l.cx) { ic = (I + 1) >> 1; ia = (I & 1) ? -1 : 1; if (I == 1 || I == b.nx) ia = 0; }
    if (l.cy) { jc = (J + 1) >> 1; ja = (J & 1) ? -1 : 1; if (J == 1 || J == b.ny) ja = 0; }
    if (l.cz) { kc = (K + 1) >> 1; ka = (K & 1) ? -1 : 1; if (K == 1 || K == b.nz) ka = 0; }
    const int base = (kc - 1) * cnxy + (jc - 1) * cnx + ic - 1;
    // (a blank fine cell keeps its value; a blanked neighbour's offset falls
    // back to the centre)
    const uint8_t nk = bc[base + ka * cnxy], nj = bc[base + ja * cnx], ni = bc[base + ia], skip = bf[e];
    const uint32_t pl = (uint32_t)((J - 1) * l.rs + split_pos(I - 1, b.nx)), at = (kl + 1) * f.slab + pl;
    const T old = x[at];
    if (nk) ka = 0;
    if (nj) ja = 0;
    if (ni) ia = 0;
    const uint32_t kA = kc - 1, kB = kA + ka, oA = lc.dq.div(kA), oB = lc.dq.div(kB);
    const int r0 = (jc - 1) * lc.rs, r1 = r0 + ja * lc.rs, c0 = split_pos(ic - 1, cnx), c1 = split_pos(ic - 1 + ia, cnx);
    const uint32_t pA = map_rank(xc, oA) + (kA - oA * lc.q + 1) * cs.slab * (uint32_t)sizeof(T),
                   pB = map_rank(xc, oB) + (kB - oB * lc.q + 1) * cs.slab * (uint32_t)sizeof(T);
    const uint32_t a0 = (r0 + c0) * sizeof(T), a1 = (r1 + c0) * sizeof(T), a2 = (r0 + c1) * sizeof(T),
                   a3 = (r1 + c1) * sizeof(T);
    T a00, a01, a10, a11, b00, b01, b10, b11;
    load_remote(pA + a0, a00);
    load_remote(pA + a1, a01);
    load_remote(pA + a2, a10);
    load_remote(pA + a3, a11);
    load_remote(pB + a0, b00);
    load_remote(pB + a1, b01);
    load_remote(pB + a2, b10);
    load_remote(pB + a3, b11);
    const T sa = add_rn(add_rn(add_rn(mul_rn(a00, (T)9), mul_rn(a01, (T)3)), mul_rn(a10, (T)3)), a11);
    const T sb = add_rn(add_rn(add_rn(mul_rn(b00, (T)9), mul_rn(b01, (T)3)), mul_rn(b10, (T)3)), b11);
    const T val = add_rn(old, add_rn(mul_rn(mul_rn(sa, (T)3), (T)0.015625), mul_rn(sb, (T)0.015625)));
    if (skip) continue;
    x[at] = val;
    if (halo.lo && K - 1 == f.k0) store_remote(halo.lo + pl * (uint32_t)sizeof(T), val);
    if (halo.hi && K == f.k1) store_remote(halo.hi + pl * (uint32_t)sizeof(T), val);
  }
}

// The coarsest level: every CTA gathers the right-hand side; the rows are
// dealt to the warps of all CTAs (FP64 sums: spread over the cluster) and
// each result goes to the CTA that holds the cell's plane.
template <typename T>
__device__ __noinline__ void coarsest_phase(const TailArgs &a, const Slab &v, int rank, int nranks) {
  const TailLevel &l = v.l;
  double *sb = (double *)(sm + a.osb);
  const int *didx = (const int *)(sm + a.odi), *dmap = didx + a.nd;
  const uint32_t bb = smem_addr(sm) + l.ob, x = smem_addr(sm) + l.ox;
  const int lane = threadIdx.x & 31, nd = a.nd, nm = (nd + 31) >> 5;
  // (a cell's word in its CTA, from plane `first` on)
  auto where = [&](uint32_t base, uint32_t c, uint32_t first) {
    const uint32_t row = l.b.dx.div(c), k = l.b.dy.div(row), o = l.dq.div(k);
    return map_rank(base, o) + ((k - o * l.q + first) * v.slab + (row - k * l.b.ny) * l.rs +
                                split_pos((int)(c - row * l.b.nx), l.b.nx)) * (uint32_t)sizeof(T);
  };
  const int step = nranks * (kTailThreads / 32);
  int e = (int)(threadIdx.x >> 5) * nranks + rank, row = e < a.nc ? dmap[e] : -1;
  constexpr int NL = kTailDofs / 32;
  double d[NL];
  auto coef = [&]() {
#pragma unroll
    for (int m = 0; m < NL; m++)
      if (m < nm && row >= 0) d[m] = a.dinv[(size_t)row * nd + min(lane + 32 * m, nd - 1)];
  };
  coef();
  for (int s = threadIdx.x; s < nd; s += kTailThreads) {
    T val;
    load_remote(where(bb, didx[s], 0u), val);
    sb[s] = (double)val;
  }
  __syncthreads();
  while (e < a.nc) {
    double s = 0.;
    if (row >= 0) {
#pragma unroll
      for (int m = 0; m < NL; m++)
        if (m < nm && lane + 32 * m < nd) s = fma(d[m], sb[lane + 32 * m], s);
      s = warp_sum(s);
    }
    if (lane == 0) store_remote(where(x, e, 1u), (T)s);
    e += step;
    row = e < a.nc ? dmap[e] : -1;
    coef();
  }
}

template <typename T>
__device__ __forceinline__ void clear(T *p, uint32_t n) {
  for (uint32_t e = threadIdx.x; e < n; e += kTailThreads) p[e] = (T)0;
}

// the operator of one level into shared memory, a plane of coefficients a warp
template <typename T>
__device__ __forceinline__ void copy_operator(const Slab &v) {
  constexpr int W = sizeof(T);
  const TailLevel &l = v.l;
  const int nx = l.b.nx, lane = threadIdx.x & 31, rows = v.planes() * l.b.ny;
  const size_t plane = (size_t)nx * l.b.ny, n = plane * l.b.nz;
  const bool wide = (nx * W) % 16 == 0;  // (rows then start and end at multiples of 16 bytes here and there)
  const uint32_t per = wide ? nx * W / 16 : nx, total = rows * per, st = (uint32_t)l.q * v.slab * W, rsb = l.rs * W;
  const uint32_t dst = smem_addr(sm) + l.oA;
  const FastDiv dr = l.dr4;
  for (int p = threadIdx.x >> 5; p < kOpPlanes<T>; p += kTailThreads / 32) {
    const T *src;
    if constexpr (W == 4)
      src = p < 10 ? (const T *)l.A + p * n : (const T *)(p == 10 ? l.D : p == 11 ? l.Asp : p == 12 ? l.inv : l.cp);
    else
      src = p < 19 ? (const T *)l.A + p * n : (const T *)(p == 19 ? l.inv : l.cp);
    const unsigned char *from = (const unsigned char *)(src + (size_t)v.k0 * plane);
    const uint32_t to = dst + p * st;
    for (uint32_t q = lane; q < total; q += 32) {
      const uint32_t row = dr.div(q), c = q - row * per;
      if (wide)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + row * rsb + c * 16), "l"(from + (size_t)q * 16));
      else
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(to + row * rsb + c * W), "l"(from + (size_t)q * W), "n"(W));
    }
  }
}

template <typename T>
__device__ __forceinline__ void vtail_body(const TailArgs &a) {
  __shared__ __align__(16) unsigned char slabs[kTailLevels * sizeof(Slab)];
  __shared__ float2 ends[sizeof(T) == 4 ? kTailUnits * 4 : 1];
  Slab *lv = (Slab *)slabs;
  auto cl = cg::this_cluster();
  const int rank = (int)cl.block_rank();
  pdl_trigger();
  {
    constexpr int NW = sizeof(TailLevel) / 4;
    const uint32_t *src = (const uint32_t *)a.lv;
    for (int w = threadIdx.x; w < a.nl * NW; w += kTailThreads) ((uint32_t *)&lv[w / NW].l)[w % NW] = src[w];
  }
  __syncthreads();
  if (threadIdx.x < a.nl) lv[threadIdx.x].form(rank);
  __syncthreads();
  // The operators (no kernel of the V-cycle writes them), the blank flags and
  // the coarsest level's indices: two groups of copies, the first level's and
  // the rest.
  if (lv[0].l.res) copy_operator<T>(lv[0]);
  asm volatile("cp.async.commit_group;" ::: "memory");
  for (int li = 1; li + 1 < a.nl; li++)
    if (lv[li].l.res) copy_operator<T>(lv[li]);
  const uint32_t s0 = smem_addr(sm);
  {
    const TailLevel &l = lv[0].l;
    const uint32_t plane = (uint32_t)l.b.nx * l.b.ny;
    copy_any(s0 + l.obl, l.blank + (uint32_t)lv[0].k0 * plane, (uint32_t)lv[0].planes() * plane);
    for (int li = 1; li < a.nl; li++) copy_any(s0 + lv[li].l.obl, lv[li].l.blank, (uint32_t)lv[li].l.b.n());
    copy_any(s0 + a.odi, a.didx, (uint32_t)a.nd * 4);
    for (int e = threadIdx.x; e < a.nc; e += kTailThreads) ((int *)(sm + a.odi))[a.nd + e] = a.dmap[e];
    asm volatile("cp.async.commit_group;" ::: "memory");
    clear((T *)(sm + l.ox), (uint32_t)(l.q + 2) * lv[0].slab);
    pdl_wait();
    T *b0 = (T *)(sm + l.ob);
    const T *src = (const T *)a.b + (uint32_t)lv[0].k0 * plane;
    const uint32_t cells = (uint32_t)lv[0].planes() * plane;
    for (uint32_t e = threadIdx.x; e < cells; e += kTailThreads) {
      const uint32_t row = l.b.dx.div(e);
      b0[row * l.rs + split_pos((int)(e - row * l.b.nx), l.b.nx)] = src[e];
    }
  }
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  cl.sync();
  const T omega = (T)a.omega;
  auto phase = [&](const Slab &v, uint32_t oxo, uint32_t oxn, uint32_t oxd, int color, int mode) {
    if constexpr (sizeof(T) == 4) phase32(v, oxo, oxn, oxd, omega, color, mode, ends);
    else phase64(v, oxo, oxn, oxd, omega, color, mode);
  };
  // one sweep of the vector at ox into the one at ot, which are then swapped
  auto smooth = [&](const Slab &v, uint32_t &ox, uint32_t &ot, bool zero) {
#pragma unroll 1
    for (int color = 0; color < 2; color++) {
      phase(v, ox, color ? ot : ox, ot, color, zero && !color ? kSweepZero : kSweep);
      cl.sync();
    }
    const uint32_t u = ox;
    ox = ot;
    ot = u;
  };
  for (int li = 0; li + 1 < a.nl; li++) {
    const Slab &v = lv[li], &c = lv[li + 1];
    uint32_t ox = v.l.ox, ot = v.l.ot;
    for (int s = 0; s < a.nu1; s++) smooth(v, ox, ot, s == 0);
    // (with omega 1 the second colour's lines were just solved: its residual
    // is zero)
    if (a.nu1 > 0 && omega == (T)1) {
      phase(v, ox, ox, 0u, 0, kWeighted1);
    } else {
      phase(v, ox, ox, 0u, 0, kWeighted);
      phase(v, ox, ox, 0u, 1, kWeighted);
    }
    clear((T *)(sm + c.l.ox), (uint32_t)(c.l.q + 2) * c.slab);
    if (li == 0) asm volatile("cp.async.wait_group 0;" ::: "memory");
    cl.sync();
    restrict_phase<T>(v, c);
    __syncthreads();
  }
  cl.sync();
  coarsest_phase<T>(a, lv[a.nl - 1], rank, (int)cl.num_blocks());
  cl.sync();
  for (int li = a.nl - 2; li >= 0; li--) {
    const Slab &v = lv[li], &c = lv[li + 1];
    // the buffer that holds a level's x after s sweeps
    auto at = [&](const TailLevel &m, int s) { return s & 1 ? m.ot : m.ox; };
    uint32_t ox = at(v.l, a.nu1), ot = at(v.l, a.nu1 + 1);
    prolong_phase<T>(v, c, li == 0, at(c.l, li + 2 == a.nl ? 0 : a.nu1 + a.nu2), ox);
    cl.sync();
    for (int s = 0; s < a.nu2; s++) smooth(v, ox, ot, false);
    if (li == 0) {
      const TailLevel &l = v.l;
      const T *x = (const T *)(sm + ox) + v.slab;
      const uint32_t plane = (uint32_t)l.b.nx * l.b.ny, cells = (uint32_t)v.planes() * plane;
      T *out = (T *)a.x + (uint32_t)v.k0 * plane;
      for (uint32_t e = threadIdx.x; e < cells; e += kTailThreads) {
        const uint32_t row = l.b.dx.div(e);
        out[e] = x[row * l.rs + split_pos((int)(e - row * l.b.nx), l.b.nx)];
      }
    }
  }
}

}  // namespace

__global__ void __launch_bounds__(kTailThreads, 1) k_vtail_f32(const __grid_constant__ TailArgs a) {
  vtail_body<float>(a);
}
__global__ void __launch_bounds__(kTailThreads, 1) k_vtail_f64(const __grid_constant__ TailArgs a) {
  vtail_body<double>(a);
}

}  // namespace vfs
