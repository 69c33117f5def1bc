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
// their owner's memory.  What bounds a phase is the latency of one warp's
// instructions (visit): 1.2-1.6 us, 0.3 of them the barrier.
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

// The coefficients of a lane's cell: FP32 in registers, FP64 read at use.
template <typename T>
struct Row;
template <>
struct Row<float> {
  __half2 h[10];
  float d;
  __device__ __forceinline__ void load(const Op<float> &o, uint32_t at) {
#pragma unroll
    for (int m = 0; m < 10; m++) h[m] = o.C[m * o.st + at];
    d = o.D[at];
  }
  __device__ __forceinline__ float residual(const Op<float> &, uint32_t, float rhs, const float (&xs)[NSLOT]) const {
    const float xc = xs[CP];
    float s = 0.f;
#pragma unroll
    for (int m = 0; m < 9; m++) {
      const float2 f = __half22float2(h[m]);
      s = fmaf(f.x, xs[2 * m + 1] - xc, s);
      s = fmaf(f.y, xs[2 * m + 2] - xc, s);
    }
    s = fmaf(__low2float(h[9]), xc, s);
    return fmaf(-d, s, rhs);
  }
};
template <>
struct Row<double> {
  __device__ __forceinline__ void load(const Op<double> &, uint32_t) {}
  __device__ __forceinline__ double residual(const Op<double> &o, uint32_t at, double rhs,
                                             const double (&xs)[NSLOT]) const {
    double s = 0.;
#pragma unroll
    for (int m = 0; m < NSLOT; m++) s = fma(o.A[m * o.st + at], xs[m], s);
    return rhs - s;
  }
};

// A lane's cell of one colour and what does not change during a stay on the
// level: its place in an x-like vector and that of the columns beside it, the
// right-hand side, the line's row (av, iv, cv), the products g, h of the line
// recurrences over the chunk, and the restriction weight.
template <typename T>
struct Cell {
  int pc, pe, pw;
  bool in, eo, wo;  // eo, wo: the column beside has the cell's colour
  T rhs, av, iv, cv, g, h, wt;
  Row<T> row;
};

// One stay on a level: `sweeps` sweeps from the vector at byte offset ox into
// the one at ot, swapped each time, then with `weigh` the residual times the
// restriction weight into r.
// A lane has one cell of each colour at most.  A unit of 8 rows of a column
// (a chunk of the line) takes 8 lanes, so that the chunk recurrences run
// through shuffles; up to 4 chunks a column (P <= 4) lie in one warp and are
// joined by shuffles, too, longer columns through shared memory (ends).
// Operator rows are a multiple of 4 times an odd number of words apart and
// columns at their split positions: reads of 8 rows of 4 columns meet no bank
// conflict.
// A phase costs the instructions that one warp needs for one cell, and the
// first pass through them fetches them from L2: everything that does not
// change is taken out of the loop (Cell), and the loop over phases holds one
// copy of the code, the two colours' cells changing places.
// A phase at 8^3 cells: 1.2 us (2.6 with addresses and coefficients formed in
// each phase, 3.7 with a lane per chunk).
template <typename T>
__device__ __noinline__ void visit(const Slab &v, uint32_t ox, uint32_t ot, int sweeps, bool zero, bool weigh, bool half,
                                   T omega, T *ends) {
  constexpr uint32_t W = sizeof(T);
  constexpr int NE = kTailThreads / 32 * 4;
  auto cl = cg::this_cluster();
  const TailLevel &l = v.l;
  const Box &b = l.b;
  const Op<T> o(v);
  const int nx = b.nx, ny = b.ny, nz = b.nz, P = l.P, rs = l.rs, nh = v.nh, slab = (int)v.slab;
  const int lane = threadIdx.x & 31, e = lane & 7, sub = lane >> 3, u = threadIdx.x >> 5;
  // the warp's unit(s): columns cpw of nu / (planes) groups; chunk 0 of the
  // lane's column in lanes 8 cb ..
  const bool inwarp = P <= 4, active = u < v.planes() * l.nu;
  const int cpw = inwarp ? 4 / P : 4, kl = active ? (int)l.dnu.div(u) : 0, k = v.k0 + kl, grp = u - kl * l.nu;
  const int quad = inwarp ? grp : (int)l.dP.div(grp), ci = !inwarp || P == 1 ? sub : P == 2 ? sub >> 1 : 0;
  const int cb = inwarp ? ci * P : 0, ch = inwarp ? min(sub - cb, P - 1) : grp - quad * P;
  const int t = sub >= cpw * (inwarp ? P : 1) ? nx : quad * cpw + ci;
  const int j = ch * kLineChunk + e, cnt = min(kLineChunk, ny - ch * kLineChunk), jc = min(j, ny - 1);
  const int at0 = slab + (kl * ny + jc) * rs;  // the cell's row in an x-like vector
  const int dm = ((jc > 0 ? jc - 1 : (b.py ? ny - 1 : jc)) - jc) * rs, dp = ((jc < ny - 1 ? jc + 1 : (b.py ? 0 : jc)) - jc) * rs;
  const int km = k > 0 ? k - 1 : (b.pz ? nz - 1 : k), kp = k < nz - 1 ? k + 1 : (b.pz ? 0 : k);
  const int dn = (int)v.slot_at(km, 0u) - (kl + 1) * slab, du = (int)v.slot_at(kp, (uint32_t)(l.q + 1) * v.slab) - (kl + 1) * slab;
  // a neighbour has the cell's colour where a side clamps it onto the cell
  // itself or an odd extent wraps
  const bool to = !((kp ^ k) & 1), bo = !((km ^ k) & 1);
  // the neighbours' copies, by byte offset in this CTA's memory: plane kl of
  // a vector is their plane q + 1 or 0
  const uint32_t base = smem_addr(sm);
  const bool lo = active && v.lo >= 0 && kl == 0, hi = active && v.hi >= 0 && k == v.k1 - 1;
  const uint32_t rlo = lo ? map_rank(base, v.lo) + (uint32_t)(l.q - kl) * v.slab * W : 0u,
                 rhi = hi ? map_rank(base, v.hi) - (uint32_t)(kl + 1) * v.slab * W : 0u;
  const uint32_t orow = (uint32_t)(kl * ny + jc) * o.rs;
  T *ys = ends, *gs = ends + NE, *hs = ends + NE * 3;  // of the chunks: y, g and h per colour
  Cell<T> A{}, B{};  // of the colour at work and of the other one
#pragma unroll 1
  for (int c = 0; c < 2; c++) {
    Cell<T> n{};
    const int par = (c + k) & 1, m = par ? nx - nh : nh, tt = max(min(t, m - 1), 0);
    n.in = active && t < m && j < ny;
    const int i = min(2 * tt + par, nx - 1), im = i > 0 ? i - 1 : (b.px ? nx - 1 : i), ip = i < nx - 1 ? i + 1 : (b.px ? 0 : i);
    const int p = split_pos(i, nx);
    n.pc = at0 + p;
    n.pe = at0 + split_pos(ip, nx);
    n.pw = at0 + split_pos(im, nx);
    n.eo = !((ip ^ i) & 1);
    n.wo = !((im ^ i) & 1);
    if (active) {
      const uint32_t at = orow + p;
      n.rhs = ((const T *)(sm + l.ob))[n.pc - slab];
      n.av = j > 0 ? o.S[at] : (T)0;
      n.iv = o.inv[at];
      n.cv = j < ny - 1 ? o.cp[at] : (T)0;
      n.row.load(o, at);
      if (weigh && (c == 0 || !half)) n.wt = ((const T *)l.w)[(uint32_t)((v.k0 + kl) * ny + jc) * nx + i];
      if (P > 1) {
        // (the way down leaves the products for the way up where they fit)
        T *keep = (T *)(sm + l.ogh) + ((size_t)c * l.q * l.nu * 32 + threadIdx.x) * 2;
        T G = -n.av * n.iv, H = -n.cv;
        if (l.ogh && !weigh) {
          G = keep[0];
          H = keep[1];
        } else {
          const T f = G;
#pragma unroll 1
          for (int s = 1; s < kLineChunk; s++) {  // (lane cnt - 1 starts h)
            const T gp = __shfl_up_sync(0xffffffffu, G, 1, 8), hp = __shfl_down_sync(0xffffffffu, H, 1, 8);
            if (e == s) G = gp * f;
            if (e == kLineChunk - 1 - s && e < cnt - 1) H = hp * -n.cv;
          }
          if (l.ogh) {
            keep[0] = G;
            keep[1] = H;
          }
        }
        n.g = G;
        n.h = H;
        if (!inwarp && e == cnt - 1) gs[c * NE + u * 4 + sub] = G;
        if (!inwarp && e == 0) hs[c * NE + u * 4 + sub] = H;
      }
    }
    A = B;
    B = n;
  }
  // 2 sweeps phases, then the weighted residuals of the colours
  const int phases = 2 * sweeps + (weigh ? 2 : 0);
#pragma unroll 1
  for (int ph = 0; ph < phases; ph++) {
    const int c = ph & 1;
    const bool solve = ph < 2 * sweeps, first = zero && ph == 0;
    T y = A.rhs;
    if (active && !first) {
      const uint32_t on = solve && c ? ot : ox;
      const T *xo = (const T *)(sm + ox), *xn = (const T *)(sm + on);
      const T *C = xo + A.pc, *E = (A.eo ? xo : xn) + A.pe, *Wt = (A.wo ? xo : xn) + A.pw,
              *Tp = (to ? xo : xn) + A.pc + du, *Bt = (bo ? xo : xn) + A.pc + dn;
      const T xs[NSLOT] = {C[0], E[0], Wt[0], C[dp], C[dm], Tp[0], Bt[0], E[dp], E[dm], Wt[dp], Wt[dm], Tp[dp], Bt[dp],
                           Tp[dm], Bt[dm], ((A.eo == to ? xo : xn) + A.pe + du)[0],
                           ((A.eo == bo ? xo : xn) + A.pe + dn)[0], ((A.wo == to ? xo : xn) + A.pw + du)[0],
                           ((A.wo == bo ? xo : xn) + A.pw + dn)[0]};
      y = A.row.residual(o, orow + (uint32_t)(A.pc - at0), A.rhs, xs);
    }
    if (!solve) {
      // (with omega 1 the second colour's lines were just solved: its residual
      // is zero)
      if (A.in) ((T *)(sm + l.orr))[A.pc - slab] = c && half ? (T)0 : mul_rn(y, A.wt);
    } else {
      if (active) {
        const T r = y;
        y = (r - A.av * (T)0) * A.iv;
#pragma unroll
        for (int q = 1; q < kLineChunk; q++) {
          const T yp = __shfl_up_sync(0xffffffffu, y, 1, 8);
          if (e == q) y = (r - A.av * yp) * A.iv;
        }
        if (inwarp) {
          T Y = (T)0;
          for (int q = 0; q < P - 1; q++) {
            const int w = ((cb + q) * 8 + kLineChunk - 1) & 31;
            const T ye = __shfl_sync(0xffffffffu, y, w), G = __shfl_sync(0xffffffffu, A.g, w);
            if (q < ch) Y = ye + G * Y;
          }
          if (P > 1) y += A.g * Y;
        } else if (e == cnt - 1) {
          ys[u * 4 + sub] = y;
        }
      }
      if (!inwarp) {
        __syncthreads();
        if (active) {
          T Y = (T)0;
          for (int q = 0; q < ch; q++) {
            const int w = (u - ch + q) * 4 + sub;
            Y = ys[w] + gs[c * NE + w] * Y;
          }
          y += A.g * Y;
        }
        __syncthreads();  // (ys is written again)
      }
      if (active) {
        const T r = y;
#pragma unroll
        for (int q = kLineChunk - 2; q >= 0; q--) {
          const T xp = __shfl_down_sync(0xffffffffu, y, 1, 8);
          if (e == q && q < cnt - 1) y = r - A.cv * xp;
        }
        if (inwarp) {
          T X = (T)0;
          for (int q = P - 1; q > 0; q--) {
            const int w = ((cb + q) * 8) & 31;
            const T xe = __shfl_sync(0xffffffffu, y, w), H = __shfl_sync(0xffffffffu, A.h, w);
            if (q > ch) X = xe + H * X;
          }
          if (P > 1) y += A.h * X;
        } else if (e == 0) {
          ys[u * 4 + sub] = y;
        }
      }
      if (!inwarp) {
        __syncthreads();
        if (active) {
          T X = (T)0;
          for (int q = P - 1; q > ch; q--) {
            const int w = (u - ch + q) * 4 + sub;
            X = ys[w] + hs[c * NE + w] * X;
          }
          y += A.h * X;
        }
      }
      if (A.in) {
        const T old = first ? (T)0 : ((const T *)(sm + ox))[A.pc], val = old + omega * y;
        const uint32_t at = ot + (uint32_t)A.pc * W;
        *(T *)(sm + at) = val;
        if (lo) store_remote(rlo + at, val);
        if (hi) store_remote(rhi + at, val);
      }
      cl.sync();
      if (c) {
        const uint32_t q = ox;
        ox = ot;
        ot = q;
      }
    }
    const Cell<T> q = A;
    A = B;
    B = q;
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
  __shared__ T ends[kTailThreads / 32 * 20];
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
  for (int li = 0; li + 1 < a.nl; li++) {
    const Slab &v = lv[li], &c = lv[li + 1];
    visit<T>(v, v.l.ox, v.l.ot, a.nu1, true, true, a.nu1 > 0 && omega == (T)1, omega, ends);
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
    const uint32_t ox = at(v.l, a.nu1);
    prolong_phase<T>(v, c, li == 0, at(c.l, li + 2 == a.nl ? 0 : a.nu1 + a.nu2), ox);
    cl.sync();
    visit<T>(v, ox, at(v.l, a.nu1 + 1), a.nu2, false, false, false, omega, ends);
    if (li == 0) {
      const TailLevel &l = v.l;
      const T *x = (const T *)(sm + at(l, a.nu1 + a.nu2)) + v.slab;
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
