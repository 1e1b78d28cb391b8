// Learned stencil smoother (no counterpart in the reference).
//
// For a level whose dofs sit on an n1 x n1 x n1 node lattice (Q1 hexahedra)
// a small convolutional network maps each node's local operator -- its
// matrix row as a 27-point stencil normalised by the diagonal -- to a
// 27-point correction stencil W(x).  A smoothing step is then
//     x_i += omega * sum_k W_k(i) r_{i + o_k},   r = f - A x,
// one launch for the stencil after the residual (no colouring).  W depends
// only on the matrix, so the network runs once per assembly; per V-cycle the
// smoother costs two streaming passes per step.
//
// Network: three 3x3x3 convolutions with zero padding on the lattice,
// 27 -> 32 (ReLU) -> 32 (ReLU) -> 27 channels, BF16 weights and BF16
// activations (every layer's input is rounded to BF16), FP32 accumulation.
// The forward runs on the tensor cores as an implicit GEMM per brick of the
// lattice (mma.sync m16n8k16 BF16: rows = nodes, columns = output channels,
// reduction = 27 offsets x 32 input channels), and so does the backward: the
// activations and weights it multiplies with are BF16 already, and an FP32
// gradient is the sum of three BF16 numbers (its leading 8 bits, the next 8, the
// rest), so three BF16 products with FP32 accumulation give the FP32 product.
// Adam runs on FP32.  Training runs on the device through the pmg_learned_*
// entry points.
//
// Lattice order: node L = i + n1 (j + n1 k).  Activations are node-major BF16
// with the channels padded to 32 (L * 32 + c); gradients likewise, three such
// arrays one after the other.  Offsets: k = (di+1) + 3 (dj+1) + 9 (dk+1).
#include "pmg_internal.h"
#include <cuda_bf16.h>
#include <cmath>
#include <vector>

namespace pmg {

constexpr int NET_C0 = 27, NET_C1 = 32, NET_C2 = 32, NET_C3 = 27;
constexpr int NET_W1 = NET_C1 * NET_C0 * 27, NET_W2 = NET_C2 * NET_C1 * 27, NET_W3 = NET_C3 * NET_C2 * 27;
constexpr int NET_OFF_W1 = 0, NET_OFF_B1 = NET_W1, NET_OFF_W2 = NET_OFF_B1 + NET_C1, NET_OFF_B2 = NET_OFF_W2 + NET_W2,
              NET_OFF_W3 = NET_OFF_B2 + NET_C2, NET_OFF_B3 = NET_OFF_W3 + NET_W3, NET_NPARAM = NET_OFF_B3 + NET_C3;

int learned_num_params() { return NET_NPARAM; }

__device__ __forceinline__ int lat_nb(int L, int k, int n1) {
  const int i = L % n1, j = (L / n1) % n1, kk = L / (n1 * n1);
  const int a = i + (k % 3) - 1, b = j + (k / 3) % 3 - 1, c = kk + k / 9 - 1;
  if (a < 0 || b < 0 || c < 0 || a >= n1 || b >= n1 || c >= n1) return -1;
  return a + n1 * (b + n1 * c);
}

// ------------------------------------------------------------- features
// feature k of node L = a(i, nb_k(i)) / a(i,i) for an active row i at node L
// (0 elsewhere), rounded to BF16: xf[L * 32 + k] (channels 27..31 stay 0);
// dscale[L] = 1 / a(i,i) for active rows, 0 for Dirichlet rows.  The caller
// zeroes xf.
__global__ void k_features(int N, int Na, int n1, const int *__restrict__ rp, const int *__restrict__ kc,
                           const double *__restrict__ a, const int *__restrict__ dof_lat, __nv_bfloat16 *__restrict__ xf,
                           float *__restrict__ dscale) {
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= N) return;
  const int L = dof_lat[r];
  if (r >= Na) { dscale[L] = 0.0f; return; }
  double diag = 1.0;
  for (int p = rp[r]; p < rp[r + 1]; p++) if (kc[p] == r) diag = a[p];
  const int i = L % n1, j = (L / n1) % n1, kk = L / (n1 * n1);
  for (int p = rp[r]; p < rp[r + 1]; p++) {
    const int Lc = dof_lat[kc[p]];
    const int di = Lc % n1 - i, dj = (Lc / n1) % n1 - j, dk = Lc / (n1 * n1) - kk;
    if (di < -1 || di > 1 || dj < -1 || dj > 1 || dk < -1 || dk > 1) continue;  // not on a 27-point stencil
    const int k = (di + 1) + 3 * (dj + 1) + 9 * (dk + 1);
    xf[(size_t)L * 32 + k] = __float2bfloat16((float)(a[p] / diag));
  }
  dscale[L] = (float)(1.0 / diag);
}

// Weights of one layer, [co][ci][27] BF16, repacked for the tensor-core
// forward as [k][co][ci] with both channel counts padded to 32 by zeros.
__global__ void k_pack_weights(int cin, int cout, const __nv_bfloat16 *__restrict__ w, __nv_bfloat16 *__restrict__ wpk) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 27 * 32 * 32) return;
  const int k = t >> 10, co = (t >> 5) & 31, ci = t & 31;
  wpk[t] = (co < cout && ci < cin) ? w[((size_t)co * cin + ci) * 27 + k] : __float2bfloat16(0.0f);
}

// The same for the data gradient, whose input channels are the layer's outputs:
// dx[ci][L] = sum_{co,k} w[co][ci][k] dz[co][L - o_k] is a convolution with the
// offsets reversed (-o_k = o_{26-k}) and the channels exchanged.
__global__ void k_pack_weights_t(int cin, int cout, const __nv_bfloat16 *__restrict__ w,
                                 __nv_bfloat16 *__restrict__ wpk) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 27 * 32 * 32) return;
  const int k = t >> 10, ci = (t >> 5) & 31, co = t & 31;
  wpk[t] = (co < cout && ci < cin) ? w[((size_t)co * cin + ci) * 27 + 26 - k] : __float2bfloat16(0.0f);
}

// v = h + m + l, three BF16 numbers (exact: 3 x 8 significant bits, up to
// underflow).  An infinite v is h = v alone (v - h would be NaN), and the values
// that round to infinity in BF16 although finite are cut off instead.
__device__ __forceinline__ void split3(float v, __nv_bfloat16 &h, __nv_bfloat16 &m, __nv_bfloat16 &l) {
  h = fabsf(v) < 0x1.fep127f ? __float2bfloat16_rn(v) : __float2bfloat16_rz(v);
  const float r = isfinite(v) ? v - __bfloat162float(h) : 0.0f;
  m = __float2bfloat16(r);
  l = __float2bfloat16(r - __bfloat162float(m));
}

// ------------------------------------------------------------- tensor-core convolution
// One CTA (8 warps) owns a brick of CONV_BX x CONV_BY x CONV_BZ output nodes at
// a time (persistent over the bricks).  Shared memory holds the packed weights
// of the layer (27 x 32 x 32 BF16, loaded once) and the brick's input with a
// one-node halo (18 x 10 x 4 nodes x 64 bytes, zero outside the lattice).
// Warp w computes the nodes x = 0..15, y = w, z = 0..1 (two m16 tiles) for all
// 32 output channels (four n8 tiles): per offset and 16-channel chunk two
// ldmatrix.x4 for the activations, two for the weights and eight mma.
// Rows of 64 bytes are stored with their four 16-byte chunks permuted
// (chunk ^ ((row >> 1) & 3)), so the eight rows of one 8x8 ldmatrix read hit
// distinct banks.
constexpr int CONV_BX = 16, CONV_BY = 8, CONV_BZ = 2;
constexpr int CONV_HX = CONV_BX + 2, CONV_HY = CONV_BY + 2, CONV_HZ = CONV_BZ + 2;
constexpr int CONV_HALO = CONV_HX * CONV_HY * CONV_HZ;  // 720 nodes
constexpr int CONV_WROWS = 27 * 32;                     // weight rows [k][co]
constexpr int CONV_SMEM = (CONV_HALO + CONV_WROWS) * 64;  // 101,376 bytes: two CTAs per SM

__device__ __forceinline__ unsigned swz(int row, int chunk) {
  return (unsigned)(row * 64 + ((chunk ^ ((row >> 1) & 3)) << 4));
}

__device__ __forceinline__ void ldsm_x4(unsigned addr, unsigned (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}

// D += A (16x16, row) B (16x8, col), BF16 inputs, FP32 accumulators
__device__ __forceinline__ void mma_bf16(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// D = A B, the first of a chain
__device__ __forceinline__ void mma_bf16_first(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%10,%10,%10,%10};\n"
      : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}

// CONV_HIDDEN: xo = ReLU(conv + b) as BF16.
// CONV_STENCIL: the stencil W[co][L] = (conv + b)[co] * dscale[L], co < cout.
// CONV_GRAD: the data gradient: the input is a gradient in three BF16 parts
//   (accumulated one after the other), xo gets conv * (act > 0) in three parts, and
//   bsum[CTA][32] the CTA's sums of it per channel (the bias gradient's partials).
//   0.24 ms per 32 x 32 layer at 65^3 nodes (FP32 CUDA cores before: 0.81 ms).
enum { CONV_HIDDEN = 0, CONV_STENCIL = 1, CONV_GRAD = 2 };
template <int MODE>
__global__ void __launch_bounds__(256, 2)
    k_conv_tc(int n1, int cout, const __nv_bfloat16 *__restrict__ xi, const __nv_bfloat16 *__restrict__ wpk,
              const __nv_bfloat16 *__restrict__ bias, __nv_bfloat16 *__restrict__ xo, const float *__restrict__ dscale,
              float *__restrict__ Wst, const __nv_bfloat16 *__restrict__ act, float *__restrict__ bsum) {
  constexpr bool LAST = MODE == CONV_STENCIL, GRAD = MODE == CONV_GRAD;
  extern __shared__ __align__(128) unsigned char conv_sm[];
  const unsigned s_halo = (unsigned)__cvta_generic_to_shared(conv_sm);
  const unsigned s_w = s_halo + CONV_HALO * 64;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const size_t NL = (size_t)n1 * n1 * n1;
  // weights: 864 rows x 4 chunks
  for (int t = tid; t < CONV_WROWS * 4; t += blockDim.x) {
    const int row = t >> 2, ch = t & 3;
    const uint4 v = __ldg(reinterpret_cast<const uint4 *>(wpk) + t);
    *reinterpret_cast<uint4 *>(conv_sm + CONV_HALO * 64 + swz(row, ch)) = v;
  }
  float bv[4][2], bs[4][2];
#pragma unroll
  for (int nt = 0; nt < 4; nt++)
#pragma unroll
    for (int e = 0; e < 2; e++) {
      const int co = nt * 8 + 2 * (lane & 3) + e;
      bv[nt][e] = !GRAD && co < cout ? __bfloat162float(bias[co]) : 0.0f;
      bs[nt][e] = 0.0f;
    }
  const int nbx = (n1 + CONV_BX - 1) / CONV_BX, nby = (n1 + CONV_BY - 1) / CONV_BY, nbz = (n1 + CONV_BZ - 1) / CONV_BZ;
  const int nbricks = nbx * nby * nbz;
  // per-lane ldmatrix rows: A (activations) row within the m16 tile and chunk half;
  // B (weights) output channel within a pair of n8 tiles and chunk half
  const int a_row = (lane & 7) + 8 * ((lane >> 3) & 1), a_half = lane >> 4;
  const int b_co = 8 * (lane >> 4) + (lane & 7), b_half = (lane >> 3) & 1;
  for (int br = blockIdx.x; br < nbricks; br += gridDim.x) {
    const int bx = br % nbx, by = (br / nbx) % nby, bz = br / (nbx * nby);
    const int x0 = bx * CONV_BX, y0 = by * CONV_BY, z0 = bz * CONV_BZ;
    float acc[2][4][4], tot[GRAD ? 2 : 1][4][4];
#pragma unroll
    for (int m = 0; m < 2; m++)
#pragma unroll
      for (int nt = 0; nt < 4; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[m][nt][e] = tot[GRAD ? m : 0][nt][e] = 0.0f;
    // The tensor cores round every sum towards zero.  The gradient's smallest part
    // comes first (relative to a small sum that is little); the leading part's sums
    // leave the accumulators after every offset (2 mma) for FP32 sums in registers,
    // which round to nearest.  Without that the gradients of the first two layers
    // were 2 to 3 times as far from FP64 as with FP32 arithmetic throughout.
    auto flush = [&]() {
#pragma unroll
      for (int m = 0; m < 2; m++)
#pragma unroll
        for (int nt = 0; nt < 4; nt++)
#pragma unroll
          for (int e = 0; e < 4; e++) {
            tot[GRAD ? m : 0][nt][e] += acc[m][nt][e];
            acc[m][nt][e] = 0.0f;
          }
    };
    for (int part = GRAD ? 2 : 0; part >= 0; part--) {
      const __nv_bfloat16 *xp = xi + part * NL * 32;
      __syncthreads();  // the previous reads of the halo are done
      for (int t = tid; t < CONV_HALO * 4; t += blockDim.x) {
        const int node = t >> 2, ch = t & 3;
        const int hx = node % CONV_HX, hy = (node / CONV_HX) % CONV_HY, hz = node / (CONV_HX * CONV_HY);
        const int gx = x0 - 1 + hx, gy = y0 - 1 + hy, gz = z0 - 1 + hz;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (gx >= 0 && gy >= 0 && gz >= 0 && gx < n1 && gy < n1 && gz < n1) {
          const size_t L = (size_t)gx + (size_t)n1 * ((size_t)gy + (size_t)n1 * gz);
          v = __ldg(reinterpret_cast<const uint4 *>(xp + L * 32) + ch);
        }
        *reinterpret_cast<uint4 *>(conv_sm + swz(node, ch)) = v;
      }
      __syncthreads();
#pragma unroll 3
      for (int k = 0; k < 27; k++) {
        const int dx = k % 3, dy = (k / 3) % 3, dz = k / 9;
#pragma unroll
        for (int kc = 0; kc < 2; kc++) {
          unsigned a[2][4], b[2][4];
#pragma unroll
          for (int m = 0; m < 2; m++) {
            const int row = (a_row + dx) + CONV_HX * ((warp + dy) + CONV_HY * (m + dz));
            ldsm_x4(s_halo + swz(row, 2 * kc + a_half), a[m]);
          }
#pragma unroll
          for (int p = 0; p < 2; p++) {
            const int row = k * 32 + 16 * p + b_co;
            ldsm_x4(s_w + swz(row, 2 * kc + b_half), b[p]);
          }
#pragma unroll
          for (int m = 0; m < 2; m++)
#pragma unroll
            for (int p = 0; p < 2; p++) {
              mma_bf16(acc[m][2 * p], a[m], b[p][0], b[p][1]);
              mma_bf16(acc[m][2 * p + 1], a[m], b[p][2], b[p][3]);
            }
        }
        if (GRAD && part == 0) flush();
      }
      if (GRAD && part > 0) flush();
    }
    if (GRAD)
#pragma unroll
      for (int m = 0; m < 2; m++)
#pragma unroll
        for (int nt = 0; nt < 4; nt++)
#pragma unroll
          for (int e = 0; e < 4; e++) acc[m][nt][e] = tot[GRAD ? m : 0][nt][e];
    // epilogue: c0,c1 = (row g, channels 2q, 2q+1), c2,c3 = (row g+8, ...)
    const int g = lane >> 2, q = lane & 3;
    const int gy = y0 + warp;
#pragma unroll
    for (int m = 0; m < 2; m++) {
      const int gz = z0 + m;
#pragma unroll
      for (int hrow = 0; hrow < 2; hrow++) {
        const int gx = x0 + g + 8 * hrow;
        if (gx >= n1 || gy >= n1 || gz >= n1) continue;
        const size_t L = (size_t)gx + (size_t)n1 * ((size_t)gy + (size_t)n1 * gz);
        const float ds = LAST ? dscale[L] : 0.0f;
#pragma unroll
        for (int nt = 0; nt < 4; nt++) {
          const int co = nt * 8 + 2 * q;
          float v0 = acc[m][nt][2 * hrow] + bv[nt][0], v1 = acc[m][nt][2 * hrow + 1] + bv[nt][1];
          if (LAST) {
            if (co < cout) Wst[(size_t)co * NL + L] = v0 * ds;
            if (co + 1 < cout) Wst[(size_t)(co + 1) * NL + L] = v1 * ds;
          } else if (GRAD) {
            const __nv_bfloat162 x = *reinterpret_cast<const __nv_bfloat162 *>(act + L * 32 + co);
            if (!(__low2float(x) > 0.0f)) v0 = 0.0f;
            if (!(__high2float(x) > 0.0f)) v1 = 0.0f;
            bs[nt][0] += v0;
            bs[nt][1] += v1;
            __nv_bfloat162 h, mi, l;
            split3(v0, h.x, mi.x, l.x);
            split3(v1, h.y, mi.y, l.y);
            *reinterpret_cast<__nv_bfloat162 *>(xo + L * 32 + co) = h;
            *reinterpret_cast<__nv_bfloat162 *>(xo + (NL + L) * 32 + co) = mi;
            *reinterpret_cast<__nv_bfloat162 *>(xo + (2 * NL + L) * 32 + co) = l;
          } else {
            *reinterpret_cast<__nv_bfloat162 *>(xo + L * 32 + co) =
                __floats2bfloat162_rn(fmaxf(v0, 0.0f), fmaxf(v1, 0.0f));
          }
        }
      }
    }
  }
  if (GRAD) {
    // per channel: over the lanes of equal q, then over the warps
    __syncthreads();
    float *sb = reinterpret_cast<float *>(conv_sm);
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        float v = bs[nt][e];
        for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane < 4) sb[warp * 32 + nt * 8 + 2 * lane + e] = v;
      }
    __syncthreads();
    if (tid < 32) {
      double v = 0.0;
      for (int w = 0; w < 8; w++) v += sb[w * 32 + tid];
      bsum[blockIdx.x * 32 + tid] = (float)v;
    }
  }
}

// ------------------------------------------------------------- weight gradient
// gw[co][ci][k] = sum_L dz[co][L] x[ci][L + o_k] as 27 products 32 x NL x 32 on the
// tensor cores: the reduction runs over the nodes, so both operands are read
// transposed (ldmatrix.trans) from their node-major bricks -- dz (three BF16
// parts) of 16 x 8 nodes and x with its one-node halo -- in shared memory, the
// next brick on its way by cp.async meanwhile.  18 warps: warp w holds the
// accumulators of offsets 3 (w % 9) .. + 2 for 16 of the 32 channels co; per 16
// nodes 3 + 6 ldmatrix.x4 feed 36 mma.  The tensor cores round their sums towards
// zero, so nothing stays in them: the leading parts' products of 16 nodes are one
// mma from 0 (their sum mostly fits 24 bits), the two smaller parts' a chain of two,
// and both are added to FP32 sums in registers, which go to sums of their own in
// shared memory after every brick.  One CTA per
// SM; every CTA leaves its sums in part[CTA] and k_wgrad_sum adds those in order,
// so the result does not depend on the schedule.
// At 65^3 nodes 0.23 ms per layer (46 GFLOP in three parts, bound by the mma.sync
// and ldmatrix issue rate); the FP32 kernel before it read dz once per (ci, k)
// through L2, 864 times in all, and took 5.4 ms.  The error against FP64 with the
// same activations is 4e-8 to 7e-8 of the gradient (8 to 32 cells a side), with the
// FP32 kernel 6e-8 to 1.2e-7.
constexpr int WG_WARPS = 18, WG_NODES = CONV_BX * CONV_BY, WG_HALO = CONV_HX * CONV_HY * 3;
constexpr int WG_STAGE = (WG_HALO + 3 * WG_NODES) * 64;  // 59,136 bytes, two stages
constexpr int WG_SMEM = 2 * WG_STAGE + 48 * 32 * WG_WARPS * (int)sizeof(float);
__device__ __forceinline__ void ldsm_x4_t(unsigned addr, unsigned (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void cp_async16(unsigned dst, const void *src, bool on) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(on ? 16 : 0) : "memory");
}

__global__ void __launch_bounds__(32 * WG_WARPS, 1)
    k_conv_wgrad(int n1, const __nv_bfloat16 *__restrict__ dz, const __nv_bfloat16 *__restrict__ x,
                 float *__restrict__ part) {
  extern __shared__ __align__(128) unsigned char conv_sm[];
  const unsigned sm = (unsigned)__cvta_generic_to_shared(conv_sm);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wo = warp % 9, mt = warp / 9;
  const size_t NL = (size_t)n1 * n1 * n1;
  const int nbx = (n1 + CONV_BX - 1) / CONV_BX, nby = (n1 + CONV_BY - 1) / CONV_BY;
  const int nbricks = nbx * nby * n1;
  auto stage = [&](int br, int buf) {
    const int x0 = br % nbx * CONV_BX, y0 = br / nbx % nby * CONV_BY, z0 = br / (nbx * nby);
    const unsigned base = sm + buf * WG_STAGE;
    for (int t = tid; t < WG_HALO * 4; t += 32 * WG_WARPS) {
      const int node = t >> 2, ch = t & 3;
      const int gx = x0 - 1 + node % CONV_HX, gy = y0 - 1 + node / CONV_HX % CONV_HY,
                gz = z0 - 1 + node / (CONV_HX * CONV_HY);
      const bool on = gx >= 0 && gy >= 0 && gz >= 0 && gx < n1 && gy < n1 && gz < n1;
      const size_t L = on ? (size_t)gx + (size_t)n1 * ((size_t)gy + (size_t)n1 * gz) : 0;
      cp_async16(base + swz(node, ch), x + L * 32 + ch * 8, on);
    }
    for (int t = tid; t < 3 * WG_NODES * 4; t += 32 * WG_WARPS) {
      const int node = t >> 2, ch = t & 3, p = node / WG_NODES, i = node % WG_NODES;
      const int gx = x0 + i % CONV_BX, gy = y0 + i / CONV_BX;
      const bool on = gx < n1 && gy < n1;
      const size_t L = on ? (size_t)gx + (size_t)n1 * ((size_t)gy + (size_t)n1 * z0) : 0;
      cp_async16(base + WG_HALO * 64 + swz(node, ch), dz + ((size_t)p * NL + L) * 32 + ch * 8, on);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  float acc[3][4][4];
  float *own = reinterpret_cast<float *>(conv_sm + 2 * WG_STAGE) + tid;  // [48][threads]
#pragma unroll
  for (int o = 0; o < 3; o++)
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++) {
        acc[o][nt][e] = 0.0f;
        own[((o * 4 + nt) * 4 + e) * 32 * WG_WARPS] = 0.0f;
      }
  // lanes of ldmatrix.x4.trans: A tiles (nodes 0-7 | 8-15) x (co 0-7 | 8-15), the
  // node half in the tile index's high bit; B tiles the other way round
  const int ti = lane >> 3, tr = lane & 7;
  const int a_node = (ti >> 1) * 8 + tr, a_ch = 2 * mt + (ti & 1);
  const int b_node = (ti & 1) * 8 + tr, b_ch = ti >> 1;
  if (blockIdx.x < nbricks) stage(blockIdx.x, 0);
  int buf = 0;
  for (int br = blockIdx.x; br < nbricks; br += gridDim.x, buf ^= 1) {
    const int next = br + gridDim.x;
    if (next < nbricks) {
      stage(next, buf ^ 1);
      asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    }
    __syncthreads();
    const unsigned s_x = sm + buf * WG_STAGE, s_d = s_x + WG_HALO * 64;
#pragma unroll 1
    for (int ks = 0; ks < WG_NODES / 16; ks++) {
      unsigned a[3][4];
#pragma unroll
      for (int p = 0; p < 3; p++) ldsm_x4_t(s_d + swz(p * WG_NODES + ks * 16 + a_node, a_ch), a[p]);
#pragma unroll
      for (int o = 0; o < 3; o++) {
        const int k = 3 * wo + o, dx = k % 3, dy = k / 3 % 3, dzz = k / 9;
        const int row = b_node + dx + CONV_HX * (ks + dy + CONV_HY * dzz);
#pragma unroll
        for (int p = 0; p < 2; p++) {
          unsigned b[4];
          ldsm_x4_t(s_x + swz(row, 2 * p + b_ch), b);
          float t[2][4];
#pragma unroll
          for (int q = 1; q >= 0; q--) {
            if (q) {
              mma_bf16_first(t[0], a[2], b[0], b[1]);
              mma_bf16_first(t[1], a[2], b[2], b[3]);
              mma_bf16(t[0], a[1], b[0], b[1]);
              mma_bf16(t[1], a[1], b[2], b[3]);
            } else {
              mma_bf16_first(t[0], a[0], b[0], b[1]);
              mma_bf16_first(t[1], a[0], b[2], b[3]);
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
              acc[o][2 * p][e] += t[0][e];
              acc[o][2 * p + 1][e] += t[1][e];
            }
          }
        }
      }
    }
#pragma unroll
    for (int o = 0; o < 3; o++)
#pragma unroll
      for (int nt = 0; nt < 4; nt++)
#pragma unroll
        for (int e = 0; e < 4; e++) {
          own[((o * 4 + nt) * 4 + e) * 32 * WG_WARPS] += acc[o][nt][e];
          acc[o][nt][e] = 0.0f;
        }
    __syncthreads();  // this brick's reads are done before its buffer is filled again
  }
  const int g = lane >> 2, q = lane & 3;
  float *out = part + (size_t)blockIdx.x * 27 * 1024;
#pragma unroll
  for (int o = 0; o < 3; o++)
#pragma unroll
    for (int nt = 0; nt < 4; nt++)
#pragma unroll
      for (int e = 0; e < 4; e++)
        out[((3 * wo + o) * 32 + mt * 16 + g + 8 * (e >> 1)) * 32 + nt * 8 + 2 * q + (e & 1)] =
            own[((o * 4 + nt) * 4 + e) * 32 * WG_WARPS];
}

// gw[co][ci][k] += sum over the CTAs' partials; gb[co] likewise.  A block takes 64
// values, each in four runs of consecutive CTAs (more loads in flight), added
// in order.
__global__ void __launch_bounds__(256) k_wgrad_sum(int cin, int cout, int nw, const float *__restrict__ part, int nb,
                                                   const float *__restrict__ bsum, float *__restrict__ gw,
                                                   float *__restrict__ gb) {
  __shared__ double run[4][64];
  const int t = blockIdx.x * 64 + (threadIdx.x & 63), q = threadIdx.x >> 6;
  const bool weight = t < 27 * 1024;
  const int n = weight ? nw : nb, stride = weight ? 27 * 1024 : 32;
  const float *src = weight ? part + t : bsum + (t - 27 * 1024);
  double v = 0.0;
  if (weight || t < 27 * 1024 + 32) {
    const int per = (n + 3) / 4, c1 = min(n, (q + 1) * per);
#pragma unroll 8
    for (int c = q * per; c < c1; c++) v += src[(size_t)c * stride];
  }
  run[q][threadIdx.x & 63] = v;
  __syncthreads();
  if (q > 0) return;
  v = (run[0][threadIdx.x] + run[1][threadIdx.x]) + (run[2][threadIdx.x] + run[3][threadIdx.x]);
  if (weight) {
    const int k = t >> 10, co = t >> 5 & 31, ci = t & 31;
    if (co < cout && ci < cin) gw[((size_t)co * cin + ci) * 27 + k] += (float)v;
  } else if (t < 27 * 1024 + cout) {
    gb[t - 27 * 1024] += (float)v;
  }
}

// ------------------------------------------------------------- smoothing step
// x_i += omega sum_k W_k(L_i) r_{dof(nb_k(L_i))} on active dofs (dof order vectors)
template <typename T>
__global__ void __launch_bounds__(256) k_stencil_smooth(int Na, int n1, const int *__restrict__ dof_lat,
                                                        const int *__restrict__ lat_dof, const float *__restrict__ W,
                                                        const T *__restrict__ r, T *__restrict__ x, T omega) {
  pdl_wait();
  pdl_trigger();
  const int NL = n1 * n1 * n1;
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= Na) return;
  const int L = dof_lat[d];
  float s = 0.0f;
#pragma unroll
  for (int k = 0; k < 27; k++) {
    const int nb = lat_nb(L, k, n1);
    if (nb >= 0) s += W[(size_t)k * NL + L] * (float)r[lat_dof[nb]];
  }
  x[d] += omega * (T)s;
}

template <typename T>
int learned_smooth(cudaStream_t s, const Level &L, const T *r, T *x, double omega) {
  const int nb = (L.Na + 255) / 256;
  if (nb == 0) return PMG_OK;
  PMG_CUDA(launch_pdl(k_stencil_smooth<T>, dim3(nb), dim3(256), 0, s, L.Na, L.lat_n[0], (const int *)L.dof_ijk.p,
                      (const int *)L.lat_dof.p, (const float *)L.lw_stencil.p, r, x, (T)omega));
  count_launches(1);
  return PMG_OK;
}
template int learned_smooth<float>(cudaStream_t, const Level &, const float *, float *, double);
template int learned_smooth<double>(cudaStream_t, const Level &, const double *, double *, double);

// ------------------------------------------------------------- network driver
static int set_conv_attrs() {
  PMG_CUDA(func_smem(k_conv_tc<CONV_HIDDEN>, CONV_SMEM));
  PMG_CUDA(func_smem(k_conv_tc<CONV_STENCIL>, CONV_SMEM));
  PMG_CUDA(func_smem(k_conv_tc<CONV_GRAD>, CONV_SMEM));
  PMG_CUDA(func_smem(k_conv_wgrad, WG_SMEM));
  return PMG_OK;
}

// persistent grid of the tensor-core convolution: two CTAs per SM, at most one per brick
static int conv_grid(int n1, int num_sms) {
  const long nb = (long)((n1 + CONV_BX - 1) / CONV_BX) * ((n1 + CONV_BY - 1) / CONV_BY) * ((n1 + CONV_BZ - 1) / CONV_BZ);
  return (int)std::min<long>(nb, 2L * num_sms);
}

// forward pass on one level: features -> W (stencil, L.lw_stencil).  With train
// the layers' inputs stay in S.xa, S.xb, S.xc.
static int net_forward(cudaStream_t s, int num_sms, Level &L, const __nv_bfloat16 *wb, NetScratch &S, bool train) {
  const int n1 = L.lat_n[0], NL = n1 * n1 * n1;
  PMG_TRY(set_conv_attrs());
  PMG_TRY(S.alloc(NL, train));
  __nv_bfloat16 *xa = reinterpret_cast<__nv_bfloat16 *>(S.xa.p), *xb = reinterpret_cast<__nv_bfloat16 *>(S.xb.p);
  __nv_bfloat16 *xc = train ? reinterpret_cast<__nv_bfloat16 *>(S.xc.p) : xa;
  __nv_bfloat16 *wpk = reinterpret_cast<__nv_bfloat16 *>(S.wpk.p);
  const int WPK = 27 * 32 * 32;
  k_pack_weights<<<WPK / 256, 256, 0, s>>>(NET_C0, NET_C1, wb + NET_OFF_W1, wpk);
  k_pack_weights<<<WPK / 256, 256, 0, s>>>(NET_C1, NET_C2, wb + NET_OFF_W2, wpk + WPK);
  k_pack_weights<<<WPK / 256, 256, 0, s>>>(NET_C2, NET_C3, wb + NET_OFF_W3, wpk + 2 * WPK);
  PMG_CUDA(cudaMemsetAsync(xa, 0, sizeof(__nv_bfloat16) * 32 * (size_t)NL, s));
  PMG_CUDA(cudaMemsetAsync(S.dscale.p, 0, sizeof(float) * (size_t)NL, s));
  k_features<<<(L.N + 255) / 256, 256, 0, s>>>(L.N, L.Na, n1, L.rowptr.p, L.kcol.p, L.A.p, L.dof_ijk.p, xa, S.dscale.p);
  PMG_TRY(L.lw_stencil.alloc((size_t)27 * NL));
  const int g = conv_grid(n1, num_sms);
  k_conv_tc<CONV_HIDDEN><<<g, 256, CONV_SMEM, s>>>(n1, NET_C1, xa, wpk, wb + NET_OFF_B1, xb, nullptr, nullptr, nullptr,
                                                   nullptr);
  k_conv_tc<CONV_HIDDEN><<<g, 256, CONV_SMEM, s>>>(n1, NET_C2, xb, wpk + WPK, wb + NET_OFF_B2, xc, nullptr, nullptr,
                                                   nullptr, nullptr);
  k_conv_tc<CONV_STENCIL><<<g, 256, CONV_SMEM, s>>>(n1, NET_C3, xc, wpk + 2 * WPK, wb + NET_OFF_B3, nullptr, S.dscale.p,
                                                    L.lw_stencil.p, nullptr, nullptr);
  count_launches(7);
  PMG_CUDA(cudaGetLastError());
  return PMG_OK;
}

int learned_forward(Handle &h, Level &L) {
  if (!h.has_learned || L.lat_n[0] <= 0) {
    set_error("learned smoother: the forward needs weights and a lattice");
    return PMG_ERR_STATE;
  }
  PMG_TRY(net_forward(h.stream, h.num_sms, L, reinterpret_cast<const __nv_bfloat16 *>(h.lw_bf16.p), h.net_scratch, false));
  L.lw_fresh = true;
  return PMG_OK;
}

// network -> stencil on every level that has a lattice (after assembly)
int learned_prepare(Handle &h) {
  if (!h.has_learned) {
    set_error("learned smoother: no weights (pmg_set_learned_weights)");
    return PMG_ERR_STATE;
  }
  for (auto &L : h.lv) {
    if (L.lat_n[0] <= 0) {
      set_error("learned smoother: every level needs a lattice (pmg_set_level_lattice)");
      return PMG_ERR_STATE;
    }
    if (L.lw_fresh) continue;
    PMG_TRY(learned_forward(h, L));
  }
  return PMG_OK;
}

// ------------------------------------------------------------- training
// loss for one sample (e, r = A e) on a level:  c = S r, u = e - c, v = A u,
// loss = |v|^2 / |r|^2 ; gradients w.r.t. the FP32 master weights accumulate in g.
__global__ void k_lat_gather(int N, const int *__restrict__ dof_lat, const double *__restrict__ v, float *__restrict__ vl) {
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d < N) vl[dof_lat[d]] = (float)v[d];
}

// c[L] = sum_k W_k(L) r[nb_k(L)] (lattice order) ; u_dof = e_dof - c
__global__ void k_train_apply(int N, int Na, int n1, const int *__restrict__ dof_lat, const float *__restrict__ W,
                              const float *__restrict__ rl, const double *__restrict__ e, double *__restrict__ u) {
  const int NL = n1 * n1 * n1;
  const int d = blockIdx.x * blockDim.x + threadIdx.x;
  if (d >= N) return;
  if (d >= Na) { u[d] = e[d]; return; }
  const int L = dof_lat[d];
  float s = 0.0f;
  for (int k = 0; k < 27; k++) {
    const int nb = lat_nb(L, k, n1);
    if (nb >= 0) s += W[(size_t)k * NL + L] * rl[nb];
  }
  u[d] = e[d] - (double)s;
}

// y_i = sum_j A_ji z_j through the transposed-entry map (pattern is structurally symmetric)
__global__ void k_spmv_t(int N, const int *__restrict__ rp, const int *__restrict__ kc, const int *__restrict__ tpos,
                         const double *__restrict__ a, const double *__restrict__ z, double *__restrict__ y) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  double s = 0.0;
  for (int p = rp[i]; p < rp[i + 1]; p++) {
    const int t = tpos[p];
    if (t >= 0) s += a[t] * z[kc[p]];
  }
  y[i] = s;
}

// The loss's gradient at the last layer's output, dz[k][L] = -du[L] dscale[L] r[nb_k(L)]
// times 2 / |r|^2, in three BF16 parts (channels 27..31 are 0), and the blocks'
// sums per channel (bsum[block][32]); a thread takes 8 channels of a node at a time.
__global__ void __launch_bounds__(256) k_train_dout(int n1, const float *__restrict__ dul, const float *__restrict__ rl,
                                                    const float *__restrict__ dscale, const double *__restrict__ r2,
                                                    __nv_bfloat16 *__restrict__ dz, float *__restrict__ bsum) {
  __shared__ float sb[64][33];
  const int NL = n1 * n1 * n1, c8 = threadIdx.x & 3;
  const float f = (float)(2.0 / (*r2 > 0 ? *r2 : 1.0));
  float bs[8];
#pragma unroll
  for (int e = 0; e < 8; e++) bs[e] = 0.0f;
  for (int L = blockIdx.x * 64 + (threadIdx.x >> 2); L < NL; L += gridDim.x * 64) {
    const float g = -dul[L] * dscale[L];
    __align__(16) __nv_bfloat16 p[3][8];
#pragma unroll
    for (int e = 0; e < 8; e++) {
      const int k = c8 * 8 + e;
      const int nb = k < 27 ? lat_nb(L, k, n1) : -1;
      const float v = nb >= 0 ? g * rl[nb] * f : 0.0f;
      bs[e] += v;
      split3(v, p[0][e], p[1][e], p[2][e]);
    }
#pragma unroll
    for (int q = 0; q < 3; q++)
      *reinterpret_cast<uint4 *>(dz + ((size_t)q * NL + L) * 32 + c8 * 8) = *reinterpret_cast<const uint4 *>(p[q]);
  }
#pragma unroll
  for (int e = 0; e < 8; e++) sb[threadIdx.x >> 2][c8 * 8 + e] = bs[e];
  __syncthreads();
  if (threadIdx.x < 32) {
    double v = 0.0;
    for (int w = 0; w < 64; w++) v += sb[w][threadIdx.x];
    bsum[blockIdx.x * 32 + threadIdx.x] = (float)v;
  }
}

__global__ void k_adam(int n, float *__restrict__ p, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       float lr, float b1, float b2, float eps, float c1, float c2, __nv_bfloat16 *__restrict__ pb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1 - b1) * gi, vi = b2 * v[i] + (1 - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = pi;
  pb[i] = __float2bfloat16(pi);
}

}  // namespace pmg

using namespace pmg;

// Adam on the FP32 master weights (BF16 copy refreshed) from a host gradient
static int adam_step(pmg::Handle *h, const float *g, float lr) {
  using namespace pmg;
  cudaStream_t s = h->stream;
  PMG_CUDA(cudaMemcpyAsync(h->lw_grad.p, g, sizeof(float) * NET_NPARAM, cudaMemcpyHostToDevice, s));
  h->adam_t++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float c1 = 1.0f - powf(b1, (float)h->adam_t), c2 = 1.0f - powf(b2, (float)h->adam_t);
  k_adam<<<(NET_NPARAM + 255) / 256, 256, 0, s>>>(NET_NPARAM, h->lw_master.p, h->lw_grad.p, h->lw_m.p, h->lw_v.p, lr,
                                                   b1, b2, 1e-8f, c1, c2, reinterpret_cast<__nv_bfloat16 *>(h->lw_bf16.p));
  count_launches(1);
  PMG_CUDA(cudaGetLastError());
  PMG_CUDA(cudaStreamSynchronize(s));
  for (auto &Lv : h->lv) Lv.lw_fresh = false;
  return PMG_OK;
}

extern "C" {

int pmg_learned_num_params(int *n) {
  if (!n) return PMG_ERR_ARG;
  *n = NET_NPARAM;
  return PMG_OK;
}

int pmg_set_level_lattice(pmg_handle hh, int level, int nx, int ny, int nz, const int *dof_lat) {
  Handle *h = reinterpret_cast<Handle *>(hh);
  if (!h || level < 0 || level >= (int)h->lv.size() || !dof_lat) return PMG_ERR_ARG;
  Level &L = h->lv[level];
  if (!L.has_csr) { set_error("pmg_set_level_lattice: set the CSR first"); return PMG_ERR_STATE; }
  if (nx != ny || ny != nz || nx < 2 || (long)nx * nx * nx != L.N) {
    set_error("pmg_set_level_lattice: the learned smoother needs a cubic lattice with one dof per node");
    return PMG_ERR_UNSUPPORTED;
  }
  std::vector<int> inv((size_t)L.N, -1);
  for (int d = 0; d < L.N; d++) {
    if (dof_lat[d] < 0 || dof_lat[d] >= L.N || inv[dof_lat[d]] >= 0) {
      set_error("pmg_set_level_lattice: dof_lat is not a permutation of the lattice");
      return PMG_ERR_ARG;
    }
    inv[dof_lat[d]] = d;
  }
  PMG_TRY(L.dof_ijk.upload(dof_lat, L.N, h->stream));
  PMG_TRY(L.lat_dof.upload(inv.data(), inv.size(), h->stream));
  PMG_CUDA(cudaStreamSynchronize(h->stream));
  L.lat_n[0] = nx; L.lat_n[1] = ny; L.lat_n[2] = nz;
  L.lw_fresh = false;
  return PMG_OK;
}

int pmg_set_learned_weights(pmg_handle hh, const float *weights) {
  Handle *h = reinterpret_cast<Handle *>(hh);
  if (!h || !weights) return PMG_ERR_ARG;
  std::vector<__nv_bfloat16> wb(NET_NPARAM);
  for (int i = 0; i < NET_NPARAM; i++) {
    if (!std::isfinite(weights[i])) { set_error("pmg_set_learned_weights: non-finite weight"); return PMG_ERR_NONFINITE; }
    wb[i] = __float2bfloat16(weights[i]);
  }
  PMG_TRY(h->lw_bf16.upload(reinterpret_cast<const uint16_t *>(wb.data()), wb.size(), h->stream));
  PMG_TRY(h->lw_master.upload(weights, NET_NPARAM, h->stream));
  PMG_CUDA(cudaStreamSynchronize(h->stream));
  h->has_learned = true;
  for (auto &L : h->lv) L.lw_fresh = false;
  return PMG_OK;
}

int pmg_get_learned_weights(pmg_handle hh, float *weights) {
  Handle *h = reinterpret_cast<Handle *>(hh);
  if (!h || !weights || !h->lw_master.p) return PMG_ERR_STATE;
  PMG_CUDA(cudaMemcpy(weights, h->lw_master.p, sizeof(float) * NET_NPARAM, cudaMemcpyDeviceToHost));
  return PMG_OK;
}

// Stencil W of a level (27 x NL FP32, lattice order) for inspection / tests.
int pmg_learned_stencil(pmg_handle hh, int level, float *W_out) {
  Handle *h = reinterpret_cast<Handle *>(hh);
  if (!h || level < 0 || level >= (int)h->lv.size() || !W_out) return PMG_ERR_ARG;
  Level &L = h->lv[level];
  if (!L.assembled) { set_error("pmg_learned_stencil: assemble first"); return PMG_ERR_STATE; }
  PMG_TRY(learned_prepare(*h));
  PMG_CUDA(cudaMemcpyAsync(W_out, L.lw_stencil.p, sizeof(float) * 27 * (size_t)L.N, cudaMemcpyDeviceToHost, h->stream));
  PMG_CUDA(cudaStreamSynchronize(h->stream));
  return PMG_OK;
}

// One training step on `level` over n_samples pairs (e_s, r_s = A e_s) given as
// device arrays of n_samples x N doubles: loss = mean_s |A (e_s - S r_s)|^2 / |r_s|^2.
// lr > 0 applies one Adam step (beta 0.9 / 0.999) to the master weights;
// grad_out (host, n_params floats, may be NULL) receives the mean gradient.
int pmg_learned_train_step(pmg_handle hh, int level, int n_samples, const double *e_dev, const double *r_dev, float lr,
                           double *loss_out, float *grad_out) {
  Handle *h = reinterpret_cast<Handle *>(hh);
  if (!h || level < 0 || level >= (int)h->lv.size() || n_samples < 1 || !e_dev || !r_dev) return PMG_ERR_ARG;
  if (!h->has_learned) { set_error("pmg_learned_train_step: set initial weights first"); return PMG_ERR_STATE; }
  Level &L = h->lv[level];
  if (!L.assembled || L.lat_n[0] <= 0) { set_error("pmg_learned_train_step: level needs a matrix and a lattice"); return PMG_ERR_STATE; }
  cudaStream_t s = h->stream;
  const int n1 = L.lat_n[0], NL = n1 * n1 * n1, N = L.N;
  // transposed-entry map (once per pattern)
  if (L.tpos.n != (size_t)L.nnz) {
    std::vector<int> tp(L.nnz, -1);
    const std::vector<int> &rp = L.h_rowptr, &kc = L.h_kcol;
    for (int i = 0; i < N; i++)
      for (int p = rp[i]; p < rp[i + 1]; p++) {
        const int j = kc[p];
        int lo = rp[j], hi = rp[j + 1] - 1;
        while (lo <= hi) {
          int mid = (lo + hi) >> 1;
          if (kc[mid] == i) { tp[p] = mid; break; }
          if (kc[mid] < i) lo = mid + 1; else hi = mid - 1;
        }
      }
    PMG_TRY(L.tpos.upload(tp.data(), tp.size(), s));
  }
  NetScratch &S = h->net_scratch;
  PMG_TRY(net_forward(s, h->num_sms, L, reinterpret_cast<const __nv_bfloat16 *>(h->lw_bf16.p), S, true));
  PMG_TRY(h->lw_grad.alloc(NET_NPARAM));
  PMG_TRY(h->lw_m.alloc(NET_NPARAM));
  PMG_TRY(h->lw_v.alloc(NET_NPARAM));
  if (h->adam_t == 0) {
    PMG_CUDA(cudaMemsetAsync(h->lw_m.p, 0, sizeof(float) * NET_NPARAM, s));
    PMG_CUDA(cudaMemsetAsync(h->lw_v.p, 0, sizeof(float) * NET_NPARAM, s));
  }
  PMG_CUDA(cudaMemsetAsync(h->lw_grad.p, 0, sizeof(float) * NET_NPARAM, s));
  const int nw = h->num_sms, nb3 = std::min((NL + 63) / 64, 4 * h->num_sms), ngr = conv_grid(n1, h->num_sms);
  PMG_TRY(S.alloc_backward(NL, N, nw, std::max(nb3, ngr), n_samples));
  double *u = S.u.p, *v = S.v.p, *du = S.du.p, *nrm = S.nrm.p;
  const int gN = (N + 255) / 256, WPK = 27 * 32 * 32;
  float *gw = h->lw_grad.p, *part = S.part.p, *bsum = S.bsum.p;
  const __nv_bfloat16 *wb = reinterpret_cast<const __nv_bfloat16 *>(h->lw_bf16.p);
  const __nv_bfloat16 *x0 = reinterpret_cast<const __nv_bfloat16 *>(S.xa.p),
                      *x1 = reinterpret_cast<const __nv_bfloat16 *>(S.xb.p),
                      *x2 = reinterpret_cast<const __nv_bfloat16 *>(S.xc.p);
  __nv_bfloat16 *da = reinterpret_cast<__nv_bfloat16 *>(S.da.p), *db = reinterpret_cast<__nv_bfloat16 *>(S.db.p);
  __nv_bfloat16 *wt = reinterpret_cast<__nv_bfloat16 *>(S.wpk.p) + 3 * WPK;
  k_pack_weights_t<<<WPK / 256, 256, 0, s>>>(NET_C2, NET_C3, wb + NET_OFF_W3, wt);
  k_pack_weights_t<<<WPK / 256, 256, 0, s>>>(NET_C1, NET_C2, wb + NET_OFF_W2, wt + WPK);
  count_launches(2);
  const int gs = (WPK + 32 + 63) / 64;
  auto weights = [&](int cin, int cout, const __nv_bfloat16 *dz, const __nv_bfloat16 *x, int nb, int off_w, int off_b) {
    k_conv_wgrad<<<nw, 32 * WG_WARPS, WG_SMEM, s>>>(n1, dz, x, part);
    k_wgrad_sum<<<gs, 256, 0, s>>>(cin, cout, nw, part, nb, bsum, gw + off_w, gw + off_b);
  };
  for (int smp = 0; smp < n_samples; smp++) {
    const double *e = e_dev + (size_t)smp * N, *r = r_dev + (size_t)smp * N;
    PMG_CUDA(cudaMemsetAsync(S.rl.p, 0, sizeof(float) * NL, s));
    k_lat_gather<<<gN, 256, 0, s>>>(N, L.dof_ijk.p, r, S.rl.p);
    k_train_apply<<<gN, 256, 0, s>>>(N, L.Na, n1, L.dof_ijk.p, L.lw_stencil.p, S.rl.p, e, u);
    PMG_TRY(spmv<double>(s, L, L.A.p, u, v));
    PMG_TRY(dot(*h, v, v, N, nrm + 2 * smp));
    PMG_TRY(dot(*h, r, r, N, nrm + 2 * smp + 1));
    // dL/dv = 2 v / |r|^2 ; du = A^T dL/dv ; dL/dc = -du
    k_spmv_t<<<gN, 256, 0, s>>>(N, L.rowptr.p, L.kcol.p, L.tpos.p, L.A.p, v, du);
    PMG_CUDA(cudaMemsetAsync(S.dul.p, 0, sizeof(float) * NL, s));
    k_lat_gather<<<gN, 256, 0, s>>>(N, L.dof_ijk.p, du, S.dul.p);
    // layer 3 (no ReLU), layer 2, layer 1
    k_train_dout<<<nb3, 256, 0, s>>>(n1, S.dul.p, S.rl.p, S.dscale.p, nrm + 2 * smp + 1, da, bsum);
    weights(NET_C2, NET_C3, da, x2, nb3, NET_OFF_W3, NET_OFF_B3);
    k_conv_tc<CONV_GRAD><<<ngr, 256, CONV_SMEM, s>>>(n1, 0, da, wt, nullptr, db, nullptr, nullptr, x2, bsum);
    weights(NET_C1, NET_C2, db, x1, ngr, NET_OFF_W2, NET_OFF_B2);
    k_conv_tc<CONV_GRAD><<<ngr, 256, CONV_SMEM, s>>>(n1, 0, db, wt + WPK, nullptr, da, nullptr, nullptr, x1, bsum);
    weights(NET_C0, NET_C1, da, x0, ngr, NET_OFF_W1, NET_OFF_B1);
    count_launches(13);
    PMG_CUDA(cudaGetLastError());
  }
  std::vector<double> nr(2 * n_samples);
  PMG_CUDA(cudaMemcpyAsync(nr.data(), nrm, sizeof(double) * nr.size(), cudaMemcpyDeviceToHost, s));
  PMG_CUDA(cudaStreamSynchronize(s));
  double loss = 0;
  for (int smp = 0; smp < n_samples; smp++) loss += nr[2 * smp] / (nr[2 * smp + 1] > 0 ? nr[2 * smp + 1] : 1.0);
  loss /= n_samples;
  if (loss_out) *loss_out = loss;
  // mean over samples
  std::vector<float> g(NET_NPARAM);
  PMG_CUDA(cudaMemcpy(g.data(), gw, sizeof(float) * NET_NPARAM, cudaMemcpyDeviceToHost));
  for (auto &x : g) x /= (float)n_samples;
  if (grad_out) std::copy(g.begin(), g.end(), grad_out);
  if (lr > 0) PMG_TRY(adam_step(h, g.data(), lr));
  return PMG_OK;
}

int pmg_learned_apply_gradient(pmg_handle hh, const float *grad, float lr) {
  Handle *h = reinterpret_cast<Handle *>(hh);
  if (!h || !grad || !(lr > 0)) {
    set_error("pmg_learned_apply_gradient: bad arguments");
    return PMG_ERR_ARG;
  }
  if (!h->lw_master.p) {
    set_error("pmg_learned_apply_gradient: set the weights first");
    return PMG_ERR_STATE;
  }
  for (int k = 0; k < NET_NPARAM; k++)
    if (!std::isfinite(grad[k])) {
      set_error("pmg_learned_apply_gradient: non-finite gradient");
      return PMG_ERR_NONFINITE;
    }
  PMG_TRY(h->lw_grad.alloc(NET_NPARAM));
  PMG_TRY(h->lw_m.alloc(NET_NPARAM));
  PMG_TRY(h->lw_v.alloc(NET_NPARAM));
  if (h->adam_t == 0) {
    PMG_CUDA(cudaMemsetAsync(h->lw_m.p, 0, sizeof(float) * NET_NPARAM, h->stream));
    PMG_CUDA(cudaMemsetAsync(h->lw_v.p, 0, sizeof(float) * NET_NPARAM, h->stream));
  }
  return adam_step(h, grad, lr);
}

}  // extern "C"
