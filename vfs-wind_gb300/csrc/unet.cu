// unet.cu -- the learned initial guess: a 3-level 3-D U-Net (16/32/64
// channels, 3x3x3 convolutions, ReLU, average-pool down, nearest up, skip
// concatenation, 1x1 head) with BF16 weights and activations on the tensor
// cores and FP32 accumulation, trained by its own forward, backward and
// Adam kernels.  No counterpart in the reference.
//
// Activations are channels-last BF16 tensors [z][y][x][C] over the interior
// box of a level (C a multiple of 16); gradients of activations are FP32.
// Convolutions are implicit GEMMs on mma.sync m16n8k16 (A = 16 voxels along
// x by 16 input channels of one tap, B = 16 input by 8 output channels):
//   * k_conv: a CTA computes a 16x8x4 (or 16x4x2) voxel tile for CT output
//     channels; the input tile with its one-voxel halo x 16 channels is
//     staged in shared memory one 16-channel group at a time, rows padded to
//     48 bytes so that ldmatrix rows fall in distinct banks; weights are
//     pre-packed in mma fragment order and read through L1.  The loader
//     fuses the skip concatenation (two sources) and the nearest-neighbour
//     upsampling (a half-resolution source); zero padding at the box edges.
//     The same kernel computes data gradients with flipped, transposed
//     weights and an FP32 epilogue.
//   * k_wgrad: weight gradients, A = input tile transposed (ldmatrix.trans),
//     B = pre-activation gradient tile; a warp owns one tap of a dz
//     plane, a CTA loops over voxel tiles and stores its sums.
// Every sum over voxels (weights, biases, head, loss) is a set of partials per
// CTA that one kernel adds in a fixed order (k_grad_reduce): a gradient of the
// mean squared error is the same bits every time.  ReLU's backward pass has no kernel of its own: what
// forms a gradient of an activation (a convolution's epilogue, the gradients
// of pooling, upsampling and the head) masks it, rounds it and sums the bias.
// All kernels are dependent launches (each waits for its predecessor first).
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <random>
#include <string>
#include <utility>
#include <vector>

#include "common.cuh"
#include "vfs_poisson.h"

namespace vfs {
void set_last_error(const std::string &msg);  // poisson.cu
}

namespace {

typedef __nv_bfloat16 bf16;
using vfs::pdl_trigger;
using vfs::pdl_wait;

constexpr int TX = 16, TY = 8, TZ = 4;                       // output tile
constexpr int HX = TX + 2, HY = TY + 2, HZ = TZ + 2;         // with halo
constexpr int HVOX = HX * HY * HZ;                           // 1080
constexpr int ROWB = 48;                                     // 16 ch + pad, bytes
constexpr int CONV_SMEM = HVOX * ROWB;                       // 51840
constexpr int CONV_SMALL = 2 * HX * 6 * 4 * ROWB;            // two stages of the 16x4x2 tile
constexpr int CONV_THREADS = 256;                            // 8 warps x 4 rows
constexpr int WGRAD_XT = HX * HY * TZ * ROWB;                // input tile of a weight gradient's dz plane

struct Src {
  const bf16 *p;  // channels-last tensor
  int c;          // its channel count
  int up;         // 1: half resolution, read at (x/2, y/2, z/2)
};

struct ConvGeom {
  int nx, ny, nz;  // output (and full-resolution input) dims
  Src s0, s1;      // concatenated input: s0 channels first
  int groups;      // (s0.c + s1.c) / 16
  int nt_tot;      // output channels / 8
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mma_bf16(float *c, const uint32_t *a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t *r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src));
}

// ldmatrix at a constant offset from a register
template <int OFF>
__device__ __forceinline__ void ldsm_x4_at(uint32_t *r, uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4 + %5];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr), "n"(OFF));
}
// The taps of a plane dz (dy, dx unrolled: every A row at a constant offset
// of the warp's row addresses).
template <int TAP, int HYV, int MT, int NT>
__device__ __forceinline__ void conv_taps(float (&acc)[MT][NT][4], const uint32_t (&row)[MT], const uint2 *wp,
                                          size_t tap_stride) {
  constexpr int dz = TAP / 9, dy = (TAP / 3) % 3, dx = TAP % 3;
  uint2 b[NT];
#pragma unroll
  for (int n = 0; n < NT; n++) b[n] = __ldg(wp + n * 32);
#pragma unroll
  for (int m = 0; m < MT; m++) {
    uint32_t a[4];
    ldsm_x4_at<((dz * HYV + dy) * HX + dx) * ROWB>(a, row[m]);
#pragma unroll
    for (int n = 0; n < NT; n++) mma_bf16(acc[m][n], a, b[n].x, b[n].y);
  }
  if constexpr (TAP < 26) conv_taps<TAP + 1, HYV, MT, NT>(acc, row, wp + tap_stride, tap_stride);
}

// Stage channel group g of the concatenated input around the output tile
// origin (x0, y0, z0) into `tile` (rows of HX voxels, HYV x HZV of them); zeros
// outside.  A warp takes whole rows, so that bounds in y and z and the row's
// address are formed once for its 36 copies; the copies are one group.
template <int HYV, int HZV, int WARPS = CONV_THREADS / 32>
__device__ __forceinline__ void load_rows(const ConvGeom &G, int g, int x0, int y0, int z0, unsigned char *tile) {
  const int g0 = G.s0.c / 16;
  const bool first = g < g0;
  const bf16 *p = first ? G.s0.p : G.s1.p;
  const int C = first ? G.s0.c : G.s1.c, up = first ? G.s0.up : G.s1.up, coff = (first ? g : g - g0) * 16;
  const int sx = up ? G.nx / 2 : G.nx, sy = up ? G.ny / 2 : G.ny, lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < HYV * HZV; r += WARPS) {
    const int hy = r % HYV, hz = r / HYV, gy = y0 - 1 + hy, gz = z0 - 1 + hz;
    const bool in = gy >= 0 && gz >= 0 && gy < G.ny && gz < G.nz;
    const bf16 *src = p + ((size_t)(gz >> up) * sy + (gy >> up)) * sx * C + coff;
    unsigned char *dst = tile + r * HX * ROWB;
    for (int q = lane; q < HX * 2; q += 32) {
      const int v = q >> 1, half = q & 1, gx = x0 - 1 + v;
      unsigned char *d = dst + v * ROWB + half * 16;
      if (!in || gx < 0 || gx >= G.nx) *reinterpret_cast<uint4 *>(d) = make_uint4(0, 0, 0, 0);
      else cp_async16(smem_u32(d), src + (size_t)(gx >> up) * C + half * 8);
    }
  }
  asm volatile("cp.async.commit_group;\n" ::);
}

// 3x3x3 convolution: forward (+ bias, ReLU, BF16 out); data gradient in FP32,
// split into two destinations at channel `split`; or data gradient of an
// activation `act` straight to the gradient before its ReLU (masked, BF16 out)
// with the CTA's sums of it per channel into part[CTA][cout].  Tiles of
// 16 x TYV x TZV voxels; STAGES 2: the next channel group is on its way while
// the present one is multiplied.
// Bound by issue: a tap of an m-tile is one ldmatrix and NT mma since their
// addresses are constants (with addresses formed at run time and a division
// per staged voxel a 16-channel layer of 64^3 voxels took 20.2 us, now 15.5: 234
// TFLOP/s, about what mma.sync gives here).
enum { kForward, kData, kMasked };
template <int CT, int MODE, int TYV, int TZV, int STAGES>
__global__ void __launch_bounds__(CONV_THREADS, CT == 16 ? 4 : 2) k_conv(ConvGeom G, const uint2 *__restrict__ wpk,
                                                          const float *__restrict__ bias,
                                                          const bf16 *__restrict__ act, bf16 *out_b, float *out0,
                                                          float *out1, int split, float *part) {
  extern __shared__ __align__(16) unsigned char tile[];
  pdl_trigger();
  pdl_wait();
  constexpr int NT = CT / 8, MT = TYV * TZV / (CONV_THREADS / 32), HYV = TYV + 2, HZV = TZV + 2;
  constexpr int TILE = HX * HYV * HZV * ROWB;
  const int tiles_x = (G.nx + TX - 1) / TX;
  const int x0 = (blockIdx.x % tiles_x) * TX, y0 = (blockIdx.x / tiles_x) * TYV, z0 = blockIdx.y * TZV;
  const int slice = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float acc[MT][NT][4];
#pragma unroll
  for (int m = 0; m < MT; m++)
#pragma unroll
    for (int n = 0; n < NT; n++) acc[m][n][0] = acc[m][n][1] = acc[m][n][2] = acc[m][n][3] = 0.f;
  const uint32_t tbase = smem_u32(tile);
  load_rows<HYV, HZV>(G, 0, x0, y0, z0, tile);
  for (int g = 0; g < G.groups; g++) {
    const int buf = STAGES == 2 ? g & 1 : 0;
    if (STAGES == 2 && g + 1 < G.groups) {
      load_rows<HYV, HZV>(G, g + 1, x0, y0, z0, tile + (buf ^ 1) * TILE);
      asm volatile("cp.async.wait_group 1;\n" ::);
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::);
    }
    __syncthreads();
    uint32_t row[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) {
      const int r = warp * MT + m, yy = r % TYV, zz = r / TYV;
      row[m] = tbase + buf * TILE + ((zz * HYV + yy) * HX + (lane & 15)) * ROWB + (lane >> 4) * 16;
    }
    conv_taps<0, HYV, MT, NT>(acc, row, wpk + ((size_t)g * G.nt_tot + slice * NT) * 32 + lane,
                              (size_t)G.groups * G.nt_tot * 32);
    if (g + 1 < G.groups) {
      __syncthreads();
      if (STAGES == 1) load_rows<HYV, HZV>(G, g + 1, x0, y0, z0, tile);
    }
  }
  // epilogue: rows lane/4 and lane/4 + 8 of each m-tile, channels pairs
  const int cout = G.nt_tot * 8;
  float sum[NT][2];
#pragma unroll
  for (int n = 0; n < NT; n++) sum[n][0] = sum[n][1] = 0.f;
#pragma unroll
  for (int m = 0; m < MT; m++) {
    const int r = warp * MT + m, y = y0 + r % TYV, z = z0 + r / TYV;
    if (y >= G.ny || z >= G.nz) continue;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int x = x0 + (lane >> 2) + h * 8;
      if (x >= G.nx) continue;
      const size_t v = ((size_t)z * G.ny + y) * G.nx + x;
#pragma unroll
      for (int n = 0; n < NT; n++) {
        const int co = slice * CT + n * 8 + (lane & 3) * 2;
        float c0 = acc[m][n][2 * h], c1 = acc[m][n][2 * h + 1];
        if (MODE == kForward) {
          c0 = fmaxf(c0 + bias[co], 0.f);
          c1 = fmaxf(c1 + bias[co + 1], 0.f);
          *reinterpret_cast<__nv_bfloat162 *>(out_b + v * cout + co) = __floats2bfloat162_rn(c0, c1);
        } else if (MODE == kMasked) {
          const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(act + v * cout + co));
          c0 = a.x > 0.f ? c0 : 0.f;
          c1 = a.y > 0.f ? c1 : 0.f;
          sum[n][0] += c0;
          sum[n][1] += c1;
          *reinterpret_cast<__nv_bfloat162 *>(out_b + v * cout + co) = __floats2bfloat162_rn(c0, c1);
        } else if (co < split) {
          *reinterpret_cast<float2 *>(out0 + v * split + co) = make_float2(c0, c1);
        } else {
          *reinterpret_cast<float2 *>(out1 + v * (cout - split) + co - split) = make_float2(c0, c1);
        }
      }
    }
  }
  if (MODE == kMasked) {
    __shared__ float sh[CONV_THREADS / 32][CT];
#pragma unroll
    for (int n = 0; n < NT; n++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        float t = sum[n][e];
        for (int o = 4; o < 32; o <<= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane < 4) sh[warp][n * 8 + lane * 2 + e] = t;
      }
    __syncthreads();
    if (threadIdx.x < CT) {
      float t = 0.f;
      for (int w = 0; w < CONV_THREADS / 32; w++) t += sh[w][threadIdx.x];
      part[(size_t)(blockIdx.x + gridDim.x * blockIdx.y) * cout + slice * CT + threadIdx.x] = t;
    }
  }
}

// Partial weight gradients: part[chunk][tap][ci][co] = sum over the chunk's
// voxel tiles of X[v + off(tap)][ci] * Gp[v][co] for input channel group
// blockIdx.y and the taps of plane dz = blockIdx.z - 1 (warp w: dy = w / 3 - 1,
// dx = w % 3 - 1), whose input tile needs no halo along z.  A chunk's products
// are one chain of FP32 accumulations in the tensor core, tile by tile
// (blockIdx.x, blockIdx.x + chunks, ...; wgrad_chunks): which tiles share a chain
// decides the gradient's last bits, and with them BF16 roundings of the next step.
// 16 x 16 channels of 64^3 voxels: 28.5 us (30.4 with the halo along z, and bounds
// and addresses formed for each voxel).  All 27 taps a CTA over 256 chunks takes 19,
// but its chains put the gradient of 48 x 16 channels 6e-6 off.
template <int COUT>
__global__ void __launch_bounds__(288, 2) k_wgrad(ConvGeom G, const bf16 *__restrict__ gpre, float *part) {
  extern __shared__ __align__(16) unsigned char smem[];
  pdl_trigger();
  pdl_wait();
  unsigned char *xt = smem;
  unsigned char *gt = smem + WGRAD_XT;
  constexpr int GROW = COUT * 2 + 16;  // bytes per voxel row of the gradient tile
  constexpr int NT = COUT / 8;
  const int g = blockIdx.y, dzi = blockIdx.z;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tiles_x = (G.nx + TX - 1) / TX, tiles_y = (G.ny + TY - 1) / TY, tiles_z = (G.nz + TZ - 1) / TZ;
  const int ntiles = tiles_x * tiles_y * tiles_z;
  float acc[NT][4];
#pragma unroll
  for (int n = 0; n < NT; n++) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.f;
  // A = X^T: rows ci, columns voxels; matrix i = lane / 8 holds (ci half
  // i & 1, voxel half i >> 1)
  const uint32_t xa = smem_u32(xt) + ((warp / 3) * HX + warp % 3 + ((lane >> 4) << 3) + (lane & 7)) * ROWB +
                      ((lane >> 3) & 1) * 16;
  // B = gradient rows (voxels) x 8 output channels; x4.trans covers (voxel
  // half i & 1, n-tile n + (i >> 1))
  const uint32_t ga = smem_u32(gt) + ((((lane >> 3) & 1) << 3) + (lane & 7)) * GROW + (lane >> 4) * 16;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int x0 = (t % tiles_x) * TX, y0 = ((t / tiles_x) % tiles_y) * TY, z0 = (t / (tiles_x * tiles_y)) * TZ;
    __syncthreads();
    // gradient tile (TX x TY x TZ voxels, COUT channels), zeros outside
    for (int q = threadIdx.x; q < TX * TY * TZ * (COUT / 8); q += blockDim.x) {
      const int v = q / (COUT / 8), c = q % (COUT / 8);
      const int x = x0 + v % TX, y = y0 + (v / TX) % TY, z = z0 + v / (TX * TY);
      unsigned char *dst = gt + v * GROW + c * 16;
      if (x >= G.nx || y >= G.ny || z >= G.nz)
        *reinterpret_cast<uint4 *>(dst) = make_uint4(0, 0, 0, 0);
      else
        cp_async16(smem_u32(dst), gpre + (((size_t)z * G.ny + y) * G.nx + x) * COUT + c * 8);
    }
    load_rows<HY, TZ, 9>(G, g, x0, y0, z0 + dzi, xt);
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
#pragma unroll 4
    for (int r = 0; r < TY * TZ; r++) {
      const uint32_t xr = xa + ((r / TY) * HY + r % TY) * HX * ROWB, gr = ga + r * TX * GROW;
      uint32_t b[NT / 2][4], a[4];
      ldsm_x4_t(a, xr);
#pragma unroll
      for (int n = 0; n < NT / 2; n++) ldsm_x4_t(b[n], gr + n * 32);
#pragma unroll
      for (int n = 0; n < NT / 2; n++) {
        mma_bf16(acc[2 * n], a, b[n][0], b[n][1]);
        mma_bf16(acc[2 * n + 1], a, b[n][2], b[n][3]);
      }
    }
  }
  const int cin = G.groups * 16;
  float *base = part + ((size_t)blockIdx.x * 27 + dzi * 9 + warp) * cin * COUT;
#pragma unroll
  for (int n = 0; n < NT; n++) {
    const int ci = g * 16 + (lane >> 2), co = n * 8 + (lane & 3) * 2;
    float *w = base + (size_t)ci * COUT + co;
    *reinterpret_cast<float2 *>(w) = make_float2(acc[n][0], acc[n][1]);
    *reinterpret_cast<float2 *>(w + 8 * COUT) = make_float2(acc[n][2], acc[n][3]);
  }
}

// The partials of one set of sums: parts rows of `cols` values, `stride` apart.
// A small set's first n sums go to dst, the next one to next (if set).
struct Sum {
  const float *src;
  float *dst;
  int cols, parts, stride, n;
  float *next;
};
constexpr int kSumBlocks = 152, kHeadBlocks = 304, kMaskBlocks = 608;
constexpr int kWeightSets = 10, kSmallSets = 11, kHeadCols = 32;
struct Sums {
  Sum w[kWeightSets], s[kSmallSets];  // weights (a block 32 values); biases and head (a block a set, cols divides 256)
  int first[kWeightSets + 1];         // blocks of the weight sets
};
// (a block's 8 warps share the partials of its values: a thread a value has up to 304
// loads in a row.  64^3 voxels: 36 MB of partials, 28 us)
__global__ void __launch_bounds__(256) k_grad_reduce(const __grid_constant__ Sums S) {
  pdl_trigger();
  pdl_wait();
  int b = blockIdx.x;
  if (b < kSmallSets) {
    __shared__ float sh[256];
    const Sum &s = S.s[b];
    const int col = threadIdx.x % s.cols, step = 256 / s.cols;
    float t = 0.f;
#pragma unroll 4
    for (int p = threadIdx.x / s.cols; p < s.parts; p += step) t += s.src[(size_t)p * s.stride + col];
    sh[threadIdx.x] = t;
    __syncthreads();
    if ((int)threadIdx.x < s.cols) {
      t = 0.f;
      for (int q = threadIdx.x; q < 256; q += s.cols) t += sh[q];
      if ((int)threadIdx.x < s.n) s.dst[threadIdx.x] = t;
      else if ((int)threadIdx.x == s.n && s.next) *s.next = t;
    }
    return;
  }
  b -= kSmallSets;
  int k = 0;
  while (b >= S.first[k + 1]) k++;
  const Sum &s = S.w[k];
  const int e = (b - S.first[k]) * 32 + (threadIdx.x & 31);  // (a multiple of 32 values a set)
  __shared__ float sh[8][32];
  float t = 0.f;
#pragma unroll 8
  for (int p = threadIdx.x >> 5; p < s.parts; p += 8) t += __ldg(s.src + (size_t)p * s.stride + e);
  sh[threadIdx.x >> 5][threadIdx.x & 31] = t;
  __syncthreads();
  if (threadIdx.x < 32) {
    t = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) t += sh[q][threadIdx.x];
    s.dst[e] = t;
  }
}

// Pack FP32 weights W[tap][ci][co] into mma B fragments: forward
// (k = ci, n = co) and data-gradient (tap flipped, k = co, n = ci).
struct PackLayer {
  int cin, cout;
  size_t w, pk, pkt;
};
struct PackLayers {
  PackLayer l[10];
};
__global__ void k_pack(const float *params, uint2 *frag, const __grid_constant__ PackLayers L) {
  pdl_trigger();
  pdl_wait();
  const PackLayer &l = L.l[blockIdx.y];
  const int cin = l.cin, cout = l.cout;
  const float *W = params + l.w;
  const int total = 27 * (cin / 16) * (cout / 8) * 32;
  const int total_t = 27 * (cout / 16) * (cin / 8) * 32;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total + total_t; e += gridDim.x * blockDim.x) {
    const bool tr = e >= total;
    const int q = tr ? e - total : e;
    const int lane = q & 31, rest = q >> 5;
    const int NTt = tr ? cin / 8 : cout / 8, Gt = tr ? cout / 16 : cin / 16;
    const int nt = rest % NTt, g = (rest / NTt) % Gt, tap = rest / (NTt * Gt);
    const int k0 = g * 16 + (lane & 3) * 2, n = nt * 8 + (lane >> 2);
    float w[4];
    for (int s = 0; s < 4; s++) {
      const int k = k0 + (s & 1) + (s >> 1) * 8;
      w[s] = tr ? W[((size_t)(26 - tap) * cin + n) * cout + k] : W[((size_t)tap * cin + k) * cout + n];
    }
    __nv_bfloat162 lo = __floats2bfloat162_rn(w[0], w[1]), hi = __floats2bfloat162_rn(w[2], w[3]);
    uint2 v;
    v.x = *reinterpret_cast<uint32_t *>(&lo);
    v.y = *reinterpret_cast<uint32_t *>(&hi);
    frag[(tr ? l.pkt : l.pk) + q] = v;
  }
}

// Network input: 4 FP32 feature planes (a sub-box of planes of dims
// (fx, fy, fz) starting at (ox, oy, oz)) -> BF16 [v][16], channels 4..15 zero.
__global__ void k_input(const float *feat, int fx, int fy, int fz, int ox, int oy, int oz, int nx, int ny, int nz,
                        bf16 *xin) {
  pdl_trigger();
  pdl_wait();
  const size_t n = (size_t)nx * ny * nz;
  const size_t plane = (size_t)fx * fy * fz;
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const uint32_t vr = (uint32_t)v / (uint32_t)nx;  // < 2^32 voxels
    const int x = (int)((uint32_t)v - vr * (uint32_t)nx), y = (int)(vr % (uint32_t)ny), z = (int)(vr / (uint32_t)ny);
    const size_t s = ((size_t)(z + oz) * fy + (y + oy)) * fx + (x + ox);
    __align__(16) bf16 row[16];
    for (int c = 0; c < 16; c++) row[c] = __float2bfloat16_rn(c < 4 ? feat[c * plane + s] : 0.f);
    uint4 *d = reinterpret_cast<uint4 *>(xin + v * 16);
    d[0] = reinterpret_cast<uint4 *>(row)[0];
    d[1] = reinterpret_cast<uint4 *>(row)[1];
  }
}

// 2x2x2 average pool of a BF16 tensor (fine dims nx, ny, nz), two channels a
// thread.
__global__ void __launch_bounds__(256) k_pool(const bf16 *__restrict__ in, int nx, int ny, int nz, int C, bf16 *out) {
  pdl_trigger();
  pdl_wait();
  const uint32_t cx = nx / 2, cy = ny / 2, half = C / 2, n = cx * cy * (nz / 2) * half;
  const __nv_bfloat162 *src = reinterpret_cast<const __nv_bfloat162 *>(in);
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const uint32_t v = e / half, c = e - v * half, row = v / cx, x = v - row * cx, z = row / cy, y = row - z * cy;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const size_t f = ((size_t)(2 * z + (q >> 2)) * ny + 2 * y + ((q >> 1) & 1)) * nx + 2 * x + (q & 1);
      const float2 a = __bfloat1622float2(src[f * half + c]);
      s0 += a.x;
      s1 += a.y;
    }
    reinterpret_cast<__nv_bfloat162 *>(out)[e] = __floats2bfloat162_rn(0.125f * s0, 0.125f * s1);
  }
}

// The gradient before a ReLU from the gradient of its output y, four channels a
// thread: masked, rounded to gp, its sums per channel into part[block][C].  C
// divides the grid's stride, so a thread keeps its channels.
__device__ __forceinline__ void masked(const float4 &g, const bf16 *__restrict__ y, bf16 *gp, uint32_t e, float4 &s) {
  const uint2 yy = reinterpret_cast<const uint2 *>(y)[e];
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&yy.x)),
               b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162 *>(&yy.y));
  const float4 v = make_float4(a.x > 0.f ? g.x : 0.f, a.y > 0.f ? g.y : 0.f, b.x > 0.f ? g.z : 0.f, b.y > 0.f ? g.w : 0.f);
  const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
  reinterpret_cast<uint2 *>(gp)[e] =
      make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
  s.x += v.x;
  s.y += v.y;
  s.z += v.z;
  s.w += v.w;
}
__device__ __forceinline__ void bias_part(const float4 &s, int C, float *part) {
  __shared__ float4 red[256];
  red[threadIdx.x] = s;
  __syncthreads();
  if ((int)threadIdx.x < C) {
    const float *r = reinterpret_cast<const float *>(red);
    float t = 0.f;
    for (int q = threadIdx.x; q < 1024; q += C) t += r[q];
    part[(size_t)blockIdx.x * C + threadIdx.x] = t;
  }
}
// of g plus the pool's gradient, 0.125 of the parent's
__global__ void __launch_bounds__(256) k_pool_relu_bwd(const float *__restrict__ g, const float *__restrict__ gc, int nx,
                                                       int ny, int nz, int C, const bf16 *__restrict__ y, bf16 *gp,
                                                       float *part) {
  pdl_trigger();
  pdl_wait();
  const uint32_t cx = nx / 2, cy = ny / 2, q = C / 4, n = (uint32_t)nx * ny * nz * q;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const uint32_t v = e / q, c = e - v * q, row = v / (uint32_t)nx, x = v - row * nx, z = row / (uint32_t)ny,
                   yy = row - z * ny;
    const float4 p = reinterpret_cast<const float4 *>(gc)[(((size_t)(z >> 1) * cy + (yy >> 1)) * cx + (x >> 1)) * q + c];
    float4 a = reinterpret_cast<const float4 *>(g)[e];
    a.x += 0.125f * p.x;
    a.y += 0.125f * p.y;
    a.z += 0.125f * p.z;
    a.w += 0.125f * p.w;
    masked(a, y, gp, e, s);
  }
  bias_part(s, C, part);
}
// of the nearest upsampling's gradient: the sum of the 8 children (fine dims
// nx, ny, nz)
__global__ void __launch_bounds__(256) k_up_relu_bwd(const float *__restrict__ gf, int nx, int ny, int nz, int C,
                                                     const bf16 *__restrict__ y, bf16 *gp, float *part) {
  pdl_trigger();
  pdl_wait();
  const uint32_t cx = nx / 2, cy = ny / 2, q = C / 4, n = cx * cy * (nz / 2) * q;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  for (uint32_t e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const uint32_t v = e / q, c = e - v * q, row = v / cx, x = v - row * cx, z = row / cy, yy = row - z * cy;
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      const size_t f = ((size_t)(2 * z + (k >> 2)) * ny + 2 * yy + ((k >> 1) & 1)) * nx + 2 * x + (k & 1);
      const float4 a = reinterpret_cast<const float4 *>(gf)[f * q + c];
      t.x += a.x;
      t.y += a.y;
      t.z += a.z;
      t.w += a.w;
    }
    masked(t, y, gp, e, s);
  }
  bias_part(s, C, part);
}

__device__ __forceinline__ float block_sum(float v, float *sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) sh[w] = v;
  __syncthreads();
  float t = 0.f;
  if (threadIdx.x < 32) {
    t = l < (int)(blockDim.x >> 5) ? sh[l] : 0.f;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  return t;  // valid in thread 0
}

// Sums of the loss weights of a sub-box (for the mean), per block.
__global__ void __launch_bounds__(256) k_weight_sum(const float *__restrict__ wt, int fx, int fy, int ox, int oy, int oz,
                                                    int nx, int ny, int nz, float *part) {
  __shared__ float sh[32];
  pdl_trigger();
  pdl_wait();
  const uint32_t n = (uint32_t)nx * ny * nz;
  float s = 0.f;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint32_t vr = v / (uint32_t)nx, x = v - vr * nx, z = vr / (uint32_t)ny, y = vr - z * ny;
    s += wt[((size_t)(z + oz) * fy + (y + oy)) * fx + (x + ox)];
  }
  s = block_sum(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}
// their total, in a fixed order, in every thread (block of 256)
__device__ __forceinline__ float weight_total(const float *__restrict__ part, float *sh) {
  const float s = block_sum(threadIdx.x < kSumBlocks ? part[threadIdx.x] : 0.f, sh);
  __shared__ float total;
  if (threadIdx.x == 0) total = s;
  __syncthreads();
  return total;
}

// 1x1 head: out = sum_c d[v][c] * wh[c] + bh.
__global__ void __launch_bounds__(256) k_head(const bf16 *__restrict__ d, size_t n, const float *__restrict__ wh,
                                              float *out) {
  pdl_trigger();
  pdl_wait();
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const uint4 *src = reinterpret_cast<const uint4 *>(d + v * 16);
    const uint4 q0 = src[0], q1 = src[1];
    const bf16 *h0 = reinterpret_cast<const bf16 *>(&q0), *h1 = reinterpret_cast<const bf16 *>(&q1);
    float o = wh[16];
    for (int c = 0; c < 16; c++) o += __bfloat162float(c < 8 ? h0[c] : h1[c - 8]) * wh[c];
    out[v] = o;
  }
}
// The head backwards from the weighted mean squared error (MSE: weights / their
// sum, its target tgt) or from the gradient gout of its output: the gradient
// before d's ReLU into gp (BF16); per block into part[block][kHeadCols] the
// sums of the head's parameter gradients (0..16) and of the loss (17), into
// bias[block][16] those of gp.  A fixed grid: the
// 34 sums of a block are as much work as the voxels of a thread.
template <bool MSE>
__global__ void __launch_bounds__(256) k_head_bwd(const bf16 *__restrict__ d, uint32_t n, const float *__restrict__ wh,
                                                  const float *__restrict__ gout, const float *__restrict__ tgt,
                                                  const float *__restrict__ wt, int fx, int fy, int ox, int oy, int oz,
                                                  int nx, int ny, const float *__restrict__ wpart, bf16 *gp,
                                                  float *part, float *bias) {
  __shared__ float sh[32], sums[8][34];
  pdl_trigger();
  pdl_wait();
  float lw[34], w[17];
#pragma unroll
  for (int c = 0; c < 34; c++) lw[c] = 0.f;
#pragma unroll
  for (int c = 0; c < 17; c++) w[c] = wh[c];
  const float inv = MSE ? 1.f / fmaxf(weight_total(wpart, sh), 1.f) : 0.f;
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < n; v += gridDim.x * blockDim.x) {
    const uint4 *src = reinterpret_cast<const uint4 *>(d + (size_t)v * 16);
    const uint4 q0 = src[0], q1 = src[1];
    const bf16 *h0 = reinterpret_cast<const bf16 *>(&q0), *h1 = reinterpret_cast<const bf16 *>(&q1);
    float dv[16], o = w[16];
#pragma unroll
    for (int c = 0; c < 16; c++) dv[c] = __bfloat162float(c < 8 ? h0[c] : h1[c - 8]);
#pragma unroll
    for (int c = 0; c < 16; c++) o += dv[c] * w[c];
    float go;
    if (MSE) {
      const uint32_t vr = v / (uint32_t)nx, x = v - vr * nx, z = vr / (uint32_t)ny, y = vr - z * ny;
      const size_t s = ((size_t)(z + oz) * fy + (y + oy)) * fx + (x + ox);
      const float ww = wt[s] * inv, e = o - tgt[s];
      go = 2.f * ww * e;
      lw[17] += ww * e * e;
    } else {
      go = gout[v];
    }
    __align__(16) bf16 row[16];
#pragma unroll
    for (int c = 0; c < 16; c++) {
      const float m = dv[c] > 0.f ? go * w[c] : 0.f;
      row[c] = __float2bfloat16_rn(m);
      lw[18 + c] += m;
      lw[c] += go * dv[c];
    }
    lw[16] += go;
    uint4 *dst = reinterpret_cast<uint4 *>(gp + (size_t)v * 16);
    dst[0] = reinterpret_cast<uint4 *>(row)[0];
    dst[1] = reinterpret_cast<uint4 *>(row)[1];
  }
  const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
#pragma unroll
  for (int c = 0; c < 34; c++) {
    float t = lw[c];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) sums[wp][c] = t;
  }
  __syncthreads();
  if (threadIdx.x < 34) {
    float t = 0.f;
    for (int k = 0; k < 8; k++) t += sums[k][threadIdx.x];
    if (threadIdx.x < 18) part[(size_t)blockIdx.x * kHeadCols + threadIdx.x] = t;
    else bias[(size_t)blockIdx.x * 16 + threadIdx.x - 18] = t;
  }
}

// Stencil offsets of the 19-point operator planes (slot order of the
// reference's PoissonLHSNew: C E W N S T B NE SE NW SW TN BN TS BS TE BE TW BW).
__constant__ int8_t c_off[19][3] = {{0, 0, 0},   {1, 0, 0},   {-1, 0, 0}, {0, 1, 0},  {0, -1, 0},
                                    {0, 0, 1},   {0, 0, -1},  {1, 1, 0},  {1, -1, 0}, {-1, 1, 0},
                                    {-1, -1, 0}, {0, 1, 1},   {0, 1, -1}, {0, -1, 1}, {0, -1, -1},
                                    {1, 0, 1},   {1, 0, -1},  {-1, 0, 1}, {-1, 0, -1}};

struct Crop {
  int fx, fy, fz, ox, oy, oz, nx, ny, nz;
  __device__ size_t glob(int x, int y, int z) const {
    return ((size_t)(z + oz) * fy + (y + oy)) * fx + (x + ox);
  }
  __device__ bool inner(int x, int y, int z) const {
    return x >= 1 && y >= 1 && z >= 1 && x < nx - 1 && y < ny - 1 && z < nz - 1;
  }
};

// Residual of the learned correction on the crop's inner cells (all 19
// neighbours inside the crop): res = f2 - s * (A out), A the row-scaled
// operator (19 planes over the feature grid), q = w res; acc[0] += w,
// acc[1] += w res^2.
__global__ void k_res_fwd(Crop cr, const float *__restrict__ op, const float *__restrict__ f2,
                          const float *__restrict__ wt, const float *__restrict__ out, float s, float *q,
                          float *acc) {
  __shared__ float sh[32];
  pdl_trigger();
  pdl_wait();
  const size_t n = (size_t)cr.nx * cr.ny * cr.nz, plane = (size_t)cr.fx * cr.fy * cr.fz;
  float sw = 0.f, sr = 0.f;
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(v % cr.nx), y = (int)((v / cr.nx) % cr.ny), z = (int)(v / ((size_t)cr.nx * cr.ny));
    float qv = 0.f;
    if (cr.inner(x, y, z)) {
      const size_t gv = cr.glob(x, y, z);
      const float w = wt[gv];
      if (w > 0.f) {
        float a = 0.f;
        for (int t = 0; t < 19; t++)
          a += op[t * plane + gv] * out[((size_t)(z + c_off[t][2]) * cr.ny + (y + c_off[t][1])) * cr.nx + x + c_off[t][0]];
        const float res = f2[gv] - s * a;
        qv = w * res;
        sw += w;
        sr += w * res * res;
      }
    }
    q[v] = qv;
  }
  sw = block_sum(sw, sh);
  if (threadIdx.x == 0) atomicAdd(acc, sw);
  sr = block_sum(sr, sh);
  if (threadIdx.x == 0) atomicAdd(acc + 1, sr);
}

// dLoss/dout = alpha * 2 w (out - t) / sum(w)  -  beta * 2 s A^T q / acc[0];
// the MSE part is added to the loss.
__global__ void k_res_bwd(Crop cr, const float *__restrict__ op, const float *__restrict__ q, const float *acc,
                          float s, float beta, const float *__restrict__ out, const float *__restrict__ tgt,
                          const float *__restrict__ wt, const float *wpart, float alpha, float *gout, float *loss) {
  __shared__ float sh[32];
  pdl_trigger();
  pdl_wait();
  const size_t n = (size_t)cr.nx * cr.ny * cr.nz, plane = (size_t)cr.fx * cr.fy * cr.fz;
  const float ir = acc[0] > 0.f ? 2.f * s * beta / acc[0] : 0.f;
  const float im = alpha / fmaxf(weight_total(wpart, sh), 1.f);
  float lm = 0.f;
  for (size_t v = blockIdx.x * (size_t)blockDim.x + threadIdx.x; v < n; v += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(v % cr.nx), y = (int)((v / cr.nx) % cr.ny), z = (int)(v / ((size_t)cr.nx * cr.ny));
    const size_t gv = cr.glob(x, y, z);
    float g = 0.f;
    if (alpha > 0.f) {
      const float w = wt[gv] * im, e = out[v] - tgt[gv];
      g += 2.f * w * e;
      lm += w * e * e;
    }
    float at = 0.f;
    for (int t = 0; t < 19; t++) {
      const int xi = x - c_off[t][0], yi = y - c_off[t][1], zi = z - c_off[t][2];
      if (!cr.inner(xi, yi, zi)) continue;
      at += op[t * plane + cr.glob(xi, yi, zi)] * q[((size_t)zi * cr.ny + yi) * cr.nx + xi];
    }
    gout[v] = g - ir * at;
  }
  lm = block_sum(lm, sh);
  if (threadIdx.x == 0) atomicAdd(loss, lm);
}

// Adam (bias-corrected; c1 = 1 - beta1^t, c2 = 1 - beta2^t).
__global__ void k_adam(float *p, const float *g, float *m, float *v, size_t n, float lr, float b1, float b2, float c1,
                       float c2, float eps) {
  pdl_trigger();
  pdl_wait();
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

int grid_for(size_t n, int threads = 256) {
  size_t b = (n + threads - 1) / threads;
  return (int)(b < 1 ? 1 : (b > 152 * 16 ? 152 * 16 : b));
}

int fail(int code, const std::string &m) {
  vfs::set_last_error(m);
  return code;
}

struct Conv {
  int cin, cout;     // cin = concatenated input channels
  int c0, c1, up0;   // concat split and upsampling of the first source
  size_t w, b;       // offsets of weights [27][cin][cout] and bias in params
  size_t pk, pkt;    // offsets of the packed fragments (uint2)
};

}  // namespace

// Layer table of the network (indices into the activation list below).
struct vfs_unet {
  int device = 0;
  cudaStream_t stream = nullptr;
  std::vector<Conv> conv;
  size_t nparams = 0, npk = 0, head = 0;
  float *params = nullptr, *grads = nullptr, *m = nullptr, *v = nullptr;
  uint2 *pk = nullptr;
  int64_t t = 0;
  bool packed = false;
  // activations for the current dims
  int nx = 0, ny = 0, nz = 0;
  bool train_bufs = false;
  std::vector<void *> bufs;
  bf16 *xin, *e0a, *e0b, *p0, *e1a, *e1b, *p1, *e2a, *e2b, *d1a, *d1b, *d0a, *d0b;
  bf16 *gp[2];  // gradients before a layer's ReLU: the present layer's and the one it passes on
  float *g_upd1b, *g_e0b, *g_upe2b, *g_e1b, *g_p1, *g_p0, *scal, *obuf, *qbuf, *gobuf;
  // partial sums: weights and biases per layer, the head's, the loss weights'
  float *wpart[10], *bpart[10], *hpart, *tpart;
  Sums sums;
  int64_t launches = 0;
};

namespace {

int setup_layers(vfs_unet *u) {
  // (cin, cout, c0, c1, up0): e0a e0b e1a e1b e2a e2b d1a d1b d0a d0b
  const int tab[10][5] = {{16, 16, 16, 0, 0}, {16, 16, 16, 0, 0}, {16, 32, 16, 0, 0}, {32, 32, 32, 0, 0},
                          {32, 64, 32, 0, 0}, {64, 64, 64, 0, 0}, {96, 32, 64, 32, 1}, {32, 32, 32, 0, 0},
                          {48, 16, 32, 16, 1}, {16, 16, 16, 0, 0}};
  size_t off = 0, pk = 0;
  for (auto &r : tab) {
    Conv c{r[0], r[1], r[2], r[3], r[4], 0, 0, 0, 0};
    c.w = off;
    off += (size_t)27 * c.cin * c.cout;
    c.b = off;
    off += c.cout;
    c.pk = pk;
    pk += (size_t)27 * (c.cin / 16) * (c.cout / 8) * 32;
    c.pkt = pk;
    pk += (size_t)27 * (c.cout / 16) * (c.cin / 8) * 32;
    u->conv.push_back(c);
  }
  u->head = off;
  off += 17;
  u->nparams = off;
  u->npk = pk;
  return 0;
}

void free_bufs(vfs_unet *u) {
  for (void *p : u->bufs) cudaFree(p);
  u->bufs.clear();
  u->nx = u->ny = u->nz = 0;
}

template <typename T>
int balloc(vfs_unet *u, T **p, size_t count) {
  if (cudaMalloc((void **)p, count * sizeof(T) + 16) != cudaSuccess) {
    cudaGetLastError();
    *p = nullptr;
    return fail(VFS_ENOMEM, "U-Net activation allocation failed");
  }
  u->bufs.push_back(*p);
  return VFS_OK;
}

// resolution of a layer's output: the box halved this many times
constexpr int kLayerLevel[10] = {0, 0, 1, 1, 2, 2, 1, 1, 0, 0};

// Tiles of 16x8x4 voxels and the widest channel slice while they fill the
// chip (two CTAs a SM), else tiles of 16x4x2 and slices of 16: eight times as
// many CTAs of a quarter of a warp's work (32^3 voxels of 32 channels had 64
// CTAs on 152 SMs, 16^3 of 64 had 16: the 11 such convolutions of a training
// step took 332 us, now 175).
struct ConvGrid {
  bool big;
  dim3 grid;
  ConvGrid(int nx, int ny, int nz, int cout) {
    const int tx = (nx + TX - 1) / TX;
    grid = dim3(tx * ((ny + TY - 1) / TY), (nz + TZ - 1) / TZ, cout / (cout % 32 == 0 ? 32 : 16));
    big = (size_t)grid.x * grid.y * grid.z >= 304;
    if (!big) grid = dim3(tx * ((ny + 3) / 4), (nz + 1) / 2, cout / 16);
  }
};

// Chunks of a layer's voxel tiles in the weight gradient: with the three dz
// planes and the channel groups two CTAs a SM.
int wgrad_chunks(const Conv &c, int nx, int ny, int nz) {
  const int ntiles = ((nx + TX - 1) / TX) * ((ny + TY - 1) / TY) * ((nz + TZ - 1) / TZ);
  return std::max(1, std::min(ntiles, 304 / (c.cin / 16 * 3)));
}

// Rows of the bias partials of layer li: the CTAs of what forms its gradient
// before the ReLU (the head for 9; the next layer's data gradient for 8, 6, 4,
// 2, 0, whose output has this layer's shape; a pooling or upsampling pass)
int bias_parts(int li, int nx, int ny, int nz) {
  if (li == 9) return kHeadBlocks;
  if (li % 2) return kMaskBlocks;
  const int cout[5] = {16, 32, 64, 32, 16};
  const ConvGrid g(nx, ny, nz, cout[li / 2]);
  return (int)(g.grid.x * g.grid.y);
}

int ensure_bufs(vfs_unet *u, int nx, int ny, int nz, bool train) {
  if (u->nx == nx && u->ny == ny && u->nz == nz && (u->train_bufs || !train)) return VFS_OK;
  free_bufs(u);
  const size_t n0 = (size_t)nx * ny * nz, n1 = n0 / 8, n2 = n0 / 64;
  int rc = VFS_OK;
#define A(p, n) \
  if ((rc = balloc(u, &u->p, n)) != VFS_OK) return rc;
  A(xin, n0 * 16) A(e0a, n0 * 16) A(e0b, n0 * 16) A(p0, n1 * 16) A(e1a, n1 * 32) A(e1b, n1 * 32) A(p1, n2 * 32)
  A(e2a, n2 * 64) A(e2b, n2 * 64) A(d1a, n1 * 32) A(d1b, n1 * 32) A(d0a, n0 * 16) A(d0b, n0 * 16) A(scal, 64)
  if (train) {
    A(gp[0], n0 * 16) A(gp[1], n0 * 16) A(g_upd1b, n0 * 32) A(g_e0b, n0 * 16) A(g_upe2b, n1 * 64) A(g_e1b, n1 * 32)
    A(g_p1, n2 * 32) A(g_p0, n1 * 16) A(obuf, n0) A(qbuf, n0) A(gobuf, n0)
    A(hpart, (size_t)kHeadBlocks * kHeadCols) A(tpart, kSumBlocks)
    Sums &S = u->sums;
    S = Sums{};
    for (int li = 0; li < 10; li++) {
      const Conv &c = u->conv[li];
      const int sh = kLayerLevel[li], lx = nx >> sh, ly = ny >> sh, lz = nz >> sh, w = 27 * c.cin * c.cout;
      const int chunks = wgrad_chunks(c, lx, ly, lz), parts = bias_parts(li, lx, ly, lz);
      A(wpart[li], (size_t)chunks * w) A(bpart[li], (size_t)parts * c.cout)
      S.w[li] = Sum{u->wpart[li], u->grads + c.w, w, chunks, w, 0, nullptr};
      S.first[li + 1] = S.first[li] + w / 32;
      S.s[li] = Sum{u->bpart[li], u->grads + c.b, c.cout, parts, c.cout, c.cout, nullptr};
    }
    S.s[10] = Sum{u->hpart, u->grads + u->head, kHeadCols, kHeadBlocks, kHeadCols, 17, u->scal + 1};
  }
#undef A
  u->nx = nx;
  u->ny = ny;
  u->nz = nz;
  u->train_bufs = train;
  return VFS_OK;
}

bool kernels_configured = false;
std::mutex cfg_mu;

template <typename K>
bool smem_attr(K kernel, int bytes) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) == cudaSuccess;
}

int configure_kernels() {
  std::lock_guard<std::mutex> lk(cfg_mu);
  if (kernels_configured) return VFS_OK;
  const int wg = WGRAD_XT + TX * TY * TZ * 16;  // + gradient tile rows of (2 COUT + 16) bytes
  bool ok = smem_attr(k_conv<16, kForward, TY, TZ, 1>, CONV_SMEM) && smem_attr(k_conv<32, kForward, TY, TZ, 1>, CONV_SMEM) &&
            smem_attr(k_conv<16, kData, TY, TZ, 1>, CONV_SMEM) && smem_attr(k_conv<32, kData, TY, TZ, 1>, CONV_SMEM) &&
            smem_attr(k_conv<16, kMasked, TY, TZ, 1>, CONV_SMEM) && smem_attr(k_conv<32, kMasked, TY, TZ, 1>, CONV_SMEM) &&
            smem_attr(k_wgrad<16>, wg + TX * TY * TZ * 32) && smem_attr(k_wgrad<32>, wg + TX * TY * TZ * 64) &&
            smem_attr(k_wgrad<64>, wg + TX * TY * TZ * 128);
  if (!ok) {
    cudaGetLastError();
    return fail(VFS_ECUDA, "cudaFuncSetAttribute failed for the U-Net kernels");
  }
  kernels_configured = true;
  return VFS_OK;
}

ConvGeom geom(const Conv &c, int nx, int ny, int nz, const bf16 *s0, const bf16 *s1) {
  ConvGeom G;
  G.nx = nx; G.ny = ny; G.nz = nz;
  G.s0 = Src{s0, c.c0, c.up0};
  G.s1 = Src{s1, c.c1, 0};
  G.groups = c.cin / 16;
  G.nt_tot = c.cout / 8;
  return G;
}

// A kernel as a dependent launch: its blocks may start while the previous
// kernel of the stream runs its last wave, and wait for it before they touch
// memory (the step's 60 launches left 2.9 us between kernels).
template <typename... P, typename... A>
void launch(vfs_unet *u, void (*kern)(P...), dim3 grid, int block, size_t smem, A &&...args) {
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = u->stream;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, std::forward<A>(args)...);
  u->launches++;
}

template <int MODE>
void launch_conv(vfs_unet *u, const ConvGeom &G, const uint2 *w, const float *bias, const bf16 *act, bf16 *out_b,
                 float *out0, float *out1, int split, float *part) {
  const int cout = G.nt_tot * 8;
  const ConvGrid g(G.nx, G.ny, G.nz, cout);
  const auto kern = !g.big ? k_conv<16, MODE, 4, 2, 2>
                           : cout % 32 == 0 ? k_conv<32, MODE, TY, TZ, 1> : k_conv<16, MODE, TY, TZ, 1>;
  launch(u, kern, g.grid, CONV_THREADS, g.big ? CONV_SMEM : CONV_SMALL, G, w, bias, act, out_b, out0, out1, split, part);
}

void conv_fwd(vfs_unet *u, int li, int nx, int ny, int nz, const bf16 *s0, const bf16 *s1, bf16 *out) {
  const Conv &c = u->conv[li];
  launch_conv<kForward>(u, geom(c, nx, ny, nz, s0, s1), u->pk + c.pk, u->params + c.b, (const bf16 *)nullptr, out,
                        nullptr, nullptr, 0, nullptr);
}

// data gradient of conv li: input gradient (gp, cout channels) -> FP32
// gradients of its sources (first c0 channels to d0, the rest to d1)
void conv_dgrad(vfs_unet *u, int li, int nx, int ny, int nz, const bf16 *gp, float *d0, float *d1) {
  const Conv &c = u->conv[li];
  Conv t{c.cout, c.cin, c.cout, 0, 0, 0, 0, 0, 0};
  launch_conv<kData>(u, geom(t, nx, ny, nz, gp, nullptr), u->pk + c.pkt, nullptr, (const bf16 *)nullptr, nullptr, d0,
                     d1, c.c0, nullptr);
}
// the same through the ReLU of its only source, layer li - 1's output act
void conv_dgrad_relu(vfs_unet *u, int li, int nx, int ny, int nz, const bf16 *gp, const bf16 *act, bf16 *out) {
  const Conv &c = u->conv[li];
  Conv t{c.cout, c.cin, c.cout, 0, 0, 0, 0, 0, 0};
  launch_conv<kMasked>(u, geom(t, nx, ny, nz, gp, nullptr), u->pk + c.pkt, nullptr, act, out, nullptr, nullptr, 0,
                       u->bpart[li - 1]);
}

void conv_wgrad(vfs_unet *u, int li, int nx, int ny, int nz, const bf16 *s0, const bf16 *s1, const bf16 *gp) {
  const Conv &c = u->conv[li];
  ConvGeom G = geom(c, nx, ny, nz, s0, s1);
  const dim3 grid(u->sums.w[li].parts, G.groups, 3);
  const int smem = WGRAD_XT + TX * TY * TZ * (c.cout * 2 + 16);
  launch(u, c.cout == 16 ? k_wgrad<16> : c.cout == 32 ? k_wgrad<32> : k_wgrad<64>, grid, 288, smem, G, gp, u->wpart[li]);
}

int pack(vfs_unet *u) {
  PackLayers L;
  for (int li = 0; li < 10; li++) {
    const Conv &c = u->conv[li];
    L.l[li] = PackLayer{c.cin, c.cout, c.w, c.pk, c.pkt};
  }
  launch(u, k_pack, dim3(48, 10), 256, 0, (const float *)u->params, u->pk, L);
  u->packed = true;
  return VFS_OK;
}

struct Box3 {
  const float *feat, *tgt, *wt;
  int fx, fy, fz, ox, oy, oz;
};

void forward(vfs_unet *u, const Box3 &b) {
  const int nx = u->nx, ny = u->ny, nz = u->nz;
  const int x1 = nx / 2, y1 = ny / 2, z1 = nz / 2, x2 = nx / 4, y2 = ny / 4, z2 = nz / 4;
  const size_t n0 = (size_t)nx * ny * nz, n1 = n0 / 8, n2 = n0 / 64;
  launch(u, k_input, grid_for(n0), 256, 0, b.feat, b.fx, b.fy, b.fz, b.ox, b.oy, b.oz, nx, ny, nz, u->xin);
  conv_fwd(u, 0, nx, ny, nz, u->xin, nullptr, u->e0a);
  conv_fwd(u, 1, nx, ny, nz, u->e0a, nullptr, u->e0b);
  launch(u, k_pool, grid_for(n1 * 8), 256, 0, (const bf16 *)u->e0b, nx, ny, nz, 16, u->p0);
  conv_fwd(u, 2, x1, y1, z1, u->p0, nullptr, u->e1a);
  conv_fwd(u, 3, x1, y1, z1, u->e1a, nullptr, u->e1b);
  launch(u, k_pool, grid_for(n2 * 16), 256, 0, (const bf16 *)u->e1b, x1, y1, z1, 32, u->p1);
  conv_fwd(u, 4, x2, y2, z2, u->p1, nullptr, u->e2a);
  conv_fwd(u, 5, x2, y2, z2, u->e2a, nullptr, u->e2b);
  conv_fwd(u, 6, x1, y1, z1, u->e2b, u->e1b, u->d1a);
  conv_fwd(u, 7, x1, y1, z1, u->d1a, nullptr, u->d1b);
  conv_fwd(u, 8, nx, ny, nz, u->d1b, u->e0b, u->d0a);
  conv_fwd(u, 9, nx, ny, nz, u->d0a, nullptr, u->d0b);
}

// from the gradient before layer 9's ReLU in gp[0]; every gradient into u->grads
void backward(vfs_unet *u) {
  const int nx = u->nx, ny = u->ny, nz = u->nz;
  const int x1 = nx / 2, y1 = ny / 2, z1 = nz / 2, x2 = nx / 4, y2 = ny / 4, z2 = nz / 4;
  bf16 *g0 = u->gp[0], *g1 = u->gp[1];
  auto up = [&](const float *gf, int x, int y, int z, int C, const bf16 *act, int li) {
    launch(u, k_up_relu_bwd, kMaskBlocks, 256, 0, gf, x, y, z, C, act, g0, u->bpart[li]);
  };
  auto pool = [&](const float *g, const float *gc, int x, int y, int z, int C, const bf16 *act, int li) {
    launch(u, k_pool_relu_bwd, kMaskBlocks, 256, 0, g, gc, x, y, z, C, act, g0, u->bpart[li]);
  };
  // d0b = relu(conv9(d0a)), d0a = relu(conv8(cat(up(d1b), e0b)))
  conv_wgrad(u, 9, nx, ny, nz, u->d0a, nullptr, g0);
  conv_dgrad_relu(u, 9, nx, ny, nz, g0, u->d0a, g1);
  conv_wgrad(u, 8, nx, ny, nz, u->d1b, u->e0b, g1);
  conv_dgrad(u, 8, nx, ny, nz, g1, u->g_upd1b, u->g_e0b);
  up(u->g_upd1b, nx, ny, nz, 32, u->d1b, 7);
  // d1b = relu(conv7(d1a)), d1a = relu(conv6(cat(up(e2b), e1b)))
  conv_wgrad(u, 7, x1, y1, z1, u->d1a, nullptr, g0);
  conv_dgrad_relu(u, 7, x1, y1, z1, g0, u->d1a, g1);
  conv_wgrad(u, 6, x1, y1, z1, u->e2b, u->e1b, g1);
  conv_dgrad(u, 6, x1, y1, z1, g1, u->g_upe2b, u->g_e1b);
  up(u->g_upe2b, x1, y1, z1, 64, u->e2b, 5);
  // e2b = relu(conv5(e2a)), e2a = relu(conv4(p1))
  conv_wgrad(u, 5, x2, y2, z2, u->e2a, nullptr, g0);
  conv_dgrad_relu(u, 5, x2, y2, z2, g0, u->e2a, g1);
  conv_wgrad(u, 4, x2, y2, z2, u->p1, nullptr, g1);
  conv_dgrad(u, 4, x2, y2, z2, g1, u->g_p1, nullptr);
  pool(u->g_e1b, u->g_p1, x1, y1, z1, 32, u->e1b, 3);
  // e1b = relu(conv3(e1a)), e1a = relu(conv2(p0))
  conv_wgrad(u, 3, x1, y1, z1, u->e1a, nullptr, g0);
  conv_dgrad_relu(u, 3, x1, y1, z1, g0, u->e1a, g1);
  conv_wgrad(u, 2, x1, y1, z1, u->p0, nullptr, g1);
  conv_dgrad(u, 2, x1, y1, z1, g1, u->g_p0, nullptr);
  pool(u->g_e0b, u->g_p0, nx, ny, nz, 16, u->e0b, 1);
  // e0b = relu(conv1(e0a)), e0a = relu(conv0(xin))
  conv_wgrad(u, 1, nx, ny, nz, u->e0a, nullptr, g0);
  conv_dgrad_relu(u, 1, nx, ny, nz, g0, u->e0a, g1);
  conv_wgrad(u, 0, nx, ny, nz, u->xin, nullptr, g1);
  launch(u, k_grad_reduce, kSmallSets + u->sums.first[kWeightSets], 256, 0, u->sums);
}

int check_dims(int nx, int ny, int nz) {
  if (nx < 4 || ny < 4 || nz < 4 || nx % 4 || ny % 4 || nz % 4)
    return fail(VFS_EINVAL, "U-Net box dims must be multiples of 4 (two 2x pooling levels)");
  return VFS_OK;
}

int cuda_status(const char *what) {
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail(VFS_ECUDA, std::string(what) + ": " + cudaGetErrorString(e));
  return VFS_OK;
}

// Loss and gradient of one sub-box (u->grads, copied to grad when set).
int loss_grad(vfs_unet *u, const vfs_unet_batch *bt, float *grad, double *loss) {
  int rc = check_dims(bt->nx, bt->ny, bt->nz);
  if (rc) return rc;
  if (bt->ox < 0 || bt->oy < 0 || bt->oz < 0 || bt->ox + bt->nx > bt->fx || bt->oy + bt->ny > bt->fy ||
      bt->oz + bt->nz > bt->fz)
    return fail(VFS_EINVAL, "sub-box outside the feature planes");
  if (bt->op && (bt->nx < 3 || bt->ny < 3 || bt->nz < 3)) return fail(VFS_EINVAL, "residual loss needs inner cells");
  if ((rc = ensure_bufs(u, bt->nx, bt->ny, bt->nz, true))) return rc;
  if (!u->packed) pack(u);
  Box3 b{bt->features, bt->target, bt->weight, bt->fx, bt->fy, bt->fz, bt->ox, bt->oy, bt->oz};
  const size_t n0 = (size_t)bt->nx * bt->ny * bt->nz;
  forward(u, b);
  launch(u, k_weight_sum, kSumBlocks, 256, 0, b.wt, b.fx, b.fy, b.ox, b.oy, b.oz, bt->nx, bt->ny, bt->nz, u->tpart);
  const bf16 *d = u->d0b;
  const float *wh = u->params + u->head;
  if (!bt->op) {
    launch(u, k_head_bwd<true>, kHeadBlocks, 256, 0, d, (uint32_t)n0, wh, (const float *)nullptr, b.tgt, b.wt, b.fx,
           b.fy, b.ox, b.oy, b.oz, bt->nx, bt->ny, (const float *)u->tpart, u->gp[0], u->hpart, u->bpart[9]);
  } else {
    // residual loss (+ optional MSE) through the row-scaled operator
    Crop cr{b.fx, b.fy, b.fz, b.ox, b.oy, b.oz, bt->nx, bt->ny, bt->nz};
    const size_t plane = (size_t)b.fx * b.fy * b.fz;
    cudaMemsetAsync(u->scal, 0, 64 * sizeof(float), u->stream);
    k_head<<<grid_for(n0), 256, 0, u->stream>>>(d, n0, wh, u->obuf);
    k_res_fwd<<<grid_for(n0), 256, 0, u->stream>>>(cr, bt->op, b.feat + 2 * plane, b.wt, u->obuf, bt->op_scale,
                                                  u->qbuf, u->scal + 2);
    k_res_bwd<<<grid_for(n0), 256, 0, u->stream>>>(cr, bt->op, u->qbuf, u->scal + 2, bt->op_scale, bt->res_weight,
                                                  u->obuf, b.tgt, b.wt, u->tpart, bt->mse_weight, u->gobuf,
                                                  u->scal + 4);
    u->launches += 3;
    launch(u, k_head_bwd<false>, kHeadBlocks, 256, 0, d, (uint32_t)n0, wh, (const float *)u->gobuf,
           (const float *)nullptr, (const float *)nullptr, 0, 0, 0, 0, 0, 1, 1, (const float *)nullptr, u->gp[0],
           u->hpart, u->bpart[9]);
  }
  backward(u);
  if (grad) cudaMemcpyAsync(grad, u->grads, u->nparams * 4, cudaMemcpyDefault, u->stream);
  float l[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
  cudaMemcpyAsync(l, u->scal, sizeof(l), cudaMemcpyDeviceToHost, u->stream);
  cudaError_t e = cudaStreamSynchronize(u->stream);
  if (e != cudaSuccess) return fail(VFS_ECUDA, std::string("U-Net step: ") + cudaGetErrorString(e));
  if (loss) *loss = bt->op ? l[4] + (l[2] > 0.f ? bt->res_weight * l[3] / l[2] : 0.f) : l[1];
  return cuda_status("U-Net step");
}

}  // namespace

extern "C" {

int vfs_unet_create(unsigned int seed, vfs_unet **out) {
  if (!out) return fail(VFS_EINVAL, "null argument");
  *out = nullptr;
  int rc = configure_kernels();
  if (rc) return rc;
  vfs_unet *u = new vfs_unet();
  cudaGetDevice(&u->device);
  setup_layers(u);
  auto al = [&](void **p, size_t bytes) {
    if (cudaMalloc(p, bytes) != cudaSuccess) { cudaGetLastError(); return false; }
    return true;
  };
  if (!al((void **)&u->params, u->nparams * 4) || !al((void **)&u->grads, u->nparams * 4) ||
      !al((void **)&u->m, u->nparams * 4) || !al((void **)&u->v, u->nparams * 4) ||
      !al((void **)&u->pk, u->npk * sizeof(uint2))) {
    vfs_unet_destroy(u);
    return fail(VFS_ENOMEM, "U-Net parameter allocation failed");
  }
  // He-uniform initialisation from a seeded generator; biases zero; the
  // head starts at zero so that the untrained network predicts no change.
  std::vector<float> p(u->nparams, 0.f);
  std::mt19937 gen(seed);
  for (const Conv &c : u->conv) {
    const float lim = std::sqrt(6.f / (27.f * c.cin));
    std::uniform_real_distribution<float> dist(-lim, lim);
    for (size_t i = 0; i < (size_t)27 * c.cin * c.cout; i++) p[c.w + i] = dist(gen);
  }
  cudaMemcpy(u->params, p.data(), u->nparams * 4, cudaMemcpyHostToDevice);
  cudaMemset(u->grads, 0, u->nparams * 4);
  cudaMemset(u->m, 0, u->nparams * 4);
  cudaMemset(u->v, 0, u->nparams * 4);
  rc = cuda_status("U-Net create");
  if (rc) {
    vfs_unet_destroy(u);
    return rc;
  }
  *out = u;
  return VFS_OK;
}

void vfs_unet_destroy(vfs_unet *u) {
  if (!u) return;
  free_bufs(u);
  cudaFree(u->params);
  cudaFree(u->grads);
  cudaFree(u->m);
  cudaFree(u->v);
  cudaFree(u->pk);
  delete u;
}

int vfs_unet_set_stream(vfs_unet *u, void *stream) {
  if (!u) return fail(VFS_EINVAL, "null argument");
  u->stream = (cudaStream_t)stream;
  return VFS_OK;
}

int64_t vfs_unet_num_params(vfs_unet *u) { return u ? (int64_t)u->nparams : 0; }

int vfs_unet_get_params(vfs_unet *u, float *out) {
  if (!u || !out) return fail(VFS_EINVAL, "null argument");
  cudaMemcpyAsync(out, u->params, u->nparams * 4, cudaMemcpyDefault, u->stream);
  if (cudaStreamSynchronize(u->stream) != cudaSuccess) return cuda_status("get_params");
  return VFS_OK;
}

int vfs_unet_set_params(vfs_unet *u, const float *in) {
  if (!u || !in) return fail(VFS_EINVAL, "null argument");
  cudaMemcpyAsync(u->params, in, u->nparams * 4, cudaMemcpyDefault, u->stream);
  u->packed = false;
  if (cudaStreamSynchronize(u->stream) != cudaSuccess) return cuda_status("set_params");
  return VFS_OK;
}

int vfs_unet_forward(vfs_unet *u, const vfs_unet_batch *bt, float *out) {
  if (!u || !bt || !bt->features || !out) return fail(VFS_EINVAL, "null argument");
  int rc = check_dims(bt->nx, bt->ny, bt->nz);
  if (rc) return rc;
  if (bt->ox < 0 || bt->oy < 0 || bt->oz < 0 || bt->ox + bt->nx > bt->fx || bt->oy + bt->ny > bt->fy ||
      bt->oz + bt->nz > bt->fz)
    return fail(VFS_EINVAL, "sub-box outside the feature planes");
  if ((rc = ensure_bufs(u, bt->nx, bt->ny, bt->nz, false))) return rc;
  if (!u->packed) pack(u);
  Box3 b{bt->features, nullptr, nullptr, bt->fx, bt->fy, bt->fz, bt->ox, bt->oy, bt->oz};
  forward(u, b);
  const size_t n0 = (size_t)bt->nx * bt->ny * bt->nz;
  launch(u, k_head, grid_for(n0), 256, 0, (const bf16 *)u->d0b, n0, (const float *)(u->params + u->head), out);
  return cuda_status("U-Net forward");
}

int vfs_unet_gradient(vfs_unet *u, const vfs_unet_batch *bt, float *grad, double *loss) {
  if (!u || !bt || !bt->features || !bt->target || !bt->weight) return fail(VFS_EINVAL, "null argument");
  const int rc = loss_grad(u, bt, grad, loss);
  if (rc) cudaMemsetAsync(u->grads, 0, u->nparams * 4, u->stream);
  return rc;
}

int vfs_unet_train_step(vfs_unet *u, const vfs_unet_batch *bt, double lr, double *loss) {
  if (!u || !bt || !bt->features || !bt->target || !bt->weight) return fail(VFS_EINVAL, "null argument");
  if (!(lr > 0)) return fail(VFS_EINVAL, "learning rate must be positive");
  const int rc = loss_grad(u, bt, nullptr, loss);
  if (rc) {
    cudaMemsetAsync(u->grads, 0, u->nparams * 4, u->stream);
    return rc;
  }
  return vfs_unet_adam(u, lr, 0.9, 0.999, 1e-8);
}

int vfs_unet_adam(vfs_unet *u, double lr, double beta1, double beta2, double eps) {
  if (!u) return fail(VFS_EINVAL, "null argument");
  u->t++;
  const float c1 = (float)(1.0 - std::pow(beta1, (double)u->t)), c2 = (float)(1.0 - std::pow(beta2, (double)u->t));
  launch(u, k_adam, grid_for(u->nparams), 256, 0, u->params, (const float *)u->grads, u->m, u->v, u->nparams, (float)lr,
         (float)beta1, (float)beta2, c1, c2, (float)eps);
  pack(u);
  return cuda_status("U-Net Adam step");
}

int vfs_unet_set_grads(vfs_unet *u, const float *grad) {
  if (!u || !grad) return fail(VFS_EINVAL, "null argument");
  cudaMemcpyAsync(u->grads, grad, u->nparams * 4, cudaMemcpyDefault, u->stream);
  if (cudaStreamSynchronize(u->stream) != cudaSuccess) return cuda_status("set_grads");
  return VFS_OK;
}

int64_t vfs_unet_kernel_launches(vfs_unet *u) { return u ? u->launches : 0; }

}  // extern "C"
