// Backward of the 3-D convolution of the learned-start network on the tensor
// cores: weight, bias and input gradients (psc_conv3d_bwd in unet.cu
// dispatches here).
//
// Both products contract an FP32 gradient with BF16 data, and the gradient
// must not lose bits.  So a brick of the gradient is staged as three BF16
// planes hi + mid + lo of 8 significant bits each, split by truncation (exact
// from 2^-110 up; below, bits under BF16's smallest subnormal, 2^-133, are
// cut), and every product is three mma.sync.m16n8k16 (BF16 operands, FP32
// accumulate) from the smallest plane up.  The split is made again for every
// brick: a pass that wrote the planes once needed 6 bytes per entry of context
// memory that overlapping calls shared and a stream capture could not allocate.  The tensor core's FP32
// accumulation does not round to nearest, so no accumulator runs through it
// for long: after the three MMAs of one 16-entry step the result is added to
// a register accumulator by an ordinary FP32 add (four adds per three MMAs).
// (tcgen05's accumulators live in tensor memory and cannot be promoted at
// that rate; its truncation over thousands of steps would cost 2e-5 of a
// gradient, 30 times this path's error.)
//
//   k_conv_prep  gradient through the activation into gm, and the bias
//                gradient's partial sums: one pass over the gradient
//   k_conv_dw    dW[tap][ci][co] = sum_v X[v s + tap - pad][ci] G[v][co].  A
//                CTA stages a brick of 8 x 4 x 4 output voxels: the input
//                with its halo once for all the taps (16 bytes = 8 channels
//                per voxel, so a tap is only another row address of
//                ldmatrix) and the three planes of the gradient.  The rows
//                of the product are units (channel octet, tap); each warp
//                owns MT pairs of units and all columns of the CTA's block of
//                output channels.  Chunks of bricks leave partial sums that
//                k_sum_chunks adds in order.
//   k_conv_dx    dvin[v][ci] = sum_{tap,co} G[o(v, tap)][co] W[tap][ci][co].
//                A CTA owns 8 x 8 x 4 voxels of one parity class (stride 2:
//                eight classes with 1 to 8 taps each, so that no product is
//                formed for a tap that the stride skips; stride 1: one class
//                of 27 taps) and a block of input channels; the gradient's
//                brick with its halo and the weights are staged 16 output
//                channels at a time.
//
// One training step's backward on 82^3 voxels (19 G multiply-adds for each
// product): weights 8.3 -> 0.80 ms, inputs 3.6 -> 0.95 ms against one thread
// per weight (two shared-memory loads per multiply-add) and one thread per
// voxel on the CUDA cores.  (0.10 and 0.48 ms of
// that were address arithmetic: a voxel's position is divided out once per
// brick, not once per 16-byte piece.)  What bounds them now is the
// mma.sync issue with its ldmatrix traffic (eight matrix loads per 24 MMAs)
// and, on the coarse levels, too few bricks for 148 SMs.  Relative errors
// against 64 bits over the network's layers: dW 7e-8 to 9e-8, input
// 8e-8 to 2.5e-7, bias 3e-8 to 8e-8 (before: up to 6e-7, 1e-6 and 3e-7).
//
// Infinities and NaNs.  The planes of an entry, the zeros staged for what lies
// outside the grid and the padding of a brick all turn an infinite factor into
// a NaN that the product of the two numbers would not give.  So a NaN in a
// result only says that an infinity or a NaN was at hand: its sum is taken
// again from the FP32 gradient, over the terms there are (dw_entry, dx_entry).
#include "psc_internal.cuh"
#include "../../include/psc.h"

#include "conv_geom.cuh"

#include <algorithm>

namespace {
constexpr int CBW_NT = 256;               // 8 warps
constexpr int BX = 8, BY = 4, BZ = 4;     // dW brick: output voxels
constexpr int BV = BX * BY * BZ;
constexpr int DX = 8, DY = 8, DZ = 4;     // dX brick: voxels of one class
constexpr int DH = (DX + 2) * (DY + 2) * (DZ + 2);   // with the halo of one
constexpr float CB_LEAK = 0.0625f;        // leaky-ReLU slope below zero

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(a));
}
__device__ __forceinline__ void ldsm2(uint32_t (&r)[2], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a));
}
__device__ __forceinline__ void ldsm2t(uint32_t (&r)[2], uint32_t a) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a));
}
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 8 BF16 values as one 16-byte word, whatever the alignment of p
__device__ __forceinline__ uint4 load8(const __nv_bfloat16* p, int aligned) {
  if (aligned) return __ldg(reinterpret_cast<const uint4*>(p));
  const unsigned short* h = reinterpret_cast<const unsigned short*>(p);
  uint32_t w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) w[j] = (uint32_t)h[2 * j] | ((uint32_t)h[2 * j + 1] << 16);
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// 8 FP32 values, whatever the alignment of p
__device__ __forceinline__ void load8f(const float* p, int aligned, float (&x)[8]) {
  if (aligned) {
    const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
    x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
    x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
  } else {
#pragma unroll
    for (int j = 0; j < 8; ++j) x[j] = p[j];
  }
}

// x - (its upper half)
__device__ __forceinline__ float split_rest(float x) {
  return x - __uint_as_float(__float_as_uint(x) & 0xffff0000u);
}

// x = hi + mid + lo: the upper half of x's bits, of the rest's, and of what
// is left, two values to a word (an infinity or NaN leaves NaNs)
__device__ __forceinline__ void split8(const float (&x)[8], uint4 (&plane)[3]) {
  uint32_t w[3][4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float a = x[2 * j], b = x[2 * j + 1];
#pragma unroll
    for (int t = 0; t < 3; ++t) {
      w[t][j] = __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632);
      a = split_rest(a);
      b = split_rest(b);
    }
  }
#pragma unroll
  for (int t = 0; t < 3; ++t) plane[t] = make_uint4(w[t][0], w[t][1], w[t][2], w[t][3]);
}
}  // namespace

// gm = gout act'(out) (gm may be gout), and part[CTA][Cout] = sums of gm over
// the CTA's voxels.  A thread owns one octet of channels and every R-th voxel
// of the CTA's range; the rows are added in order.
__global__ void __launch_bounds__(256)
k_conv_prep(const float* gout, const __nv_bfloat16* __restrict__ out, long nvo, int Cout, int act, int aligned,
            float* gm, long vchunk, float* __restrict__ part) {
  __shared__ float sh[256 * 8];
  const int oct = Cout / 8;
  const int R = 256 / oct;
  const int o = threadIdx.x % oct, r = threadIdx.x / oct;
  const long v0 = (long)blockIdx.x * vchunk, v1 = min(nvo, v0 + vchunk);
  const float below = act == 2 ? CB_LEAK : 0.0f;
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) s[j] = 0.0f;
  if (r < R)
    for (long v = v0 + r; v < v1; v += R) {
      const long e = v * oct + o;
      float x[8];
      if (aligned) {
        const float4* gp = reinterpret_cast<const float4*>(gout) + 2 * e;
        const float4 a = gp[0], b = gp[1];
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) x[j] = gout[8 * e + j];
      }
      if (act != 0) {
        const uint4 u = load8(out + 8 * e, aligned);
        const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float y = __uint_as_float(j & 1 ? w[j >> 1] & 0xffff0000u : w[j >> 1] << 16);
          if (!(y > 0.0f)) x[j] *= below;
        }
      }
      if (act != 0 || gm != gout) {
        if (aligned) {
          float4* gp = reinterpret_cast<float4*>(gm) + 2 * e;
          gp[0] = make_float4(x[0], x[1], x[2], x[3]);
          gp[1] = make_float4(x[4], x[5], x[6], x[7]);
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) gm[8 * e + j] = x[j];
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) s[j] += x[j];
    }
#pragma unroll
  for (int j = 0; j < 8; ++j) sh[threadIdx.x * 8 + j] = s[j];
  __syncthreads();
  for (int c = threadIdx.x; c < Cout; c += 256) {
    float t = 0.0f;
    for (int q = 0; q < R; ++q) t += sh[(q * oct + c / 8) * 8 + (c & 7)];
    part[(long)blockIdx.x * Cout + c] = t;
  }
}

// dB[c] = sum of the CTAs' partials, one warp per channel in a fixed order
__global__ void k_conv_bias(const float* __restrict__ part, int np, int Cout, float* __restrict__ dB) {
  const int c = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (c >= Cout) return;
  float s = 0.0f;
  for (int i = lane; i < np; i += 32) s += part[(long)i * Cout + c];
  s = psc_warp_sum(s);
  if (lane == 0) dB[c] = s;
}

struct DwArgs {
  const __nv_bfloat16* A;
  const __nv_bfloat16* S;
  const float* G;         // gradient through the activation [nvo][Cout]
  int g_aligned;          // G is 16-byte aligned
  ConvGeom g;
  int nbx, nby, nbz;      // bricks per axis
  int bricks_per_chunk;
  int hx, hy, hz;         // staged input extents of a brick
  int nc8;                // channel octets staged per CTA (at most)
  float* part;
};

// One entry's sum over the bricks b0 .. b1, term by term; a sum that has become
// NaN stays one.
__device__ __noinline__ float dw_entry(const DwArgs& P, int tap, int ci, int co, int b0, int b1) {
  const ConvGeom& g = P.g;
  const int pad = g.ksize / 2;
  const int dx = tap % g.ksize - pad, dy = (tap / g.ksize) % g.ksize - pad, dz = tap / (g.ksize * g.ksize) - pad;
  float s = 0.0f;
  for (int b = b0; b < b1; ++b)
    for (int v = 0; v < BV; ++v) {
      const int xo = (b % P.nbx) * BX + v % BX, yo = ((b / P.nbx) % P.nby) * BY + (v / BX) % BY,
                zo = (b / (P.nbx * P.nby)) * BZ + v / (BX * BY);
      if (xo >= g.nxo || yo >= g.nyo || zo >= g.nzo) continue;
      const int x = xo * g.stride + dx, y = yo * g.stride + dy, z = zo * g.stride + dz;
      if (x < 0 || y < 0 || z < 0 || x >= g.nxi || y >= g.nyi || z >= g.nzi) continue;
      const long vs = x + (long)g.nxi * (y + (long)g.nyi * z);
      const long va = g.up ? (x >> 1) + (long)g.nxa * ((y >> 1) + (long)g.nya * (z >> 1)) : vs;
      const __nv_bfloat16 xv = ci < g.Ca ? P.A[va * g.Ca + ci] : P.S[vs * g.Cs + (ci - g.Ca)];
      s = fmaf(__bfloat162float(xv), P.G[(xo + (long)g.nxo * (yo + (long)g.nyo * zo)) * g.Cout + co], s);
      if (s != s) return s;
    }
  return s;
}

template <int NT8, int MT>
__global__ void __launch_bounds__(CBW_NT)
k_conv_dw(const __grid_constant__ DwArgs P) {
  extern __shared__ __align__(128) unsigned char cb_sm[];
  const ConvGeom& g = P.g;
  const int taps = g.ksize * g.ksize * g.ksize, pad = g.ksize / 2;
  const int nu = (g.Cin / 8) * taps;
  constexpr int UC = 8 * MT * 2;                    // units per CTA
  const int u0 = blockIdx.y * UC;
  const int n0 = blockIdx.z * NT8 * 8;              // first output channel
  const int c8lo = u0 / taps;
  const int nc8 = (min(u0 + UC, nu) - 1) / taps - c8lo + 1;
  const int HV = P.hx * P.hy * P.hz;
  uint4* Xs = reinterpret_cast<uint4*>(cb_sm);      // [nc8][HV]
  uint4* Gs = Xs + (size_t)P.nc8 * HV;              // [3][NT8][BV]
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mi = lane >> 3, r = lane & 7;
  const uint32_t xbase = smem_u32(Xs), gbase = smem_u32(Gs);
  // this lane's row addresses: matrix mi of an A fragment is unit (mi & 1) of
  // the pair, voxels 8 (mi >> 1) + r of the step (two x rows of the brick)
  uint32_t aoff[MT];
#pragma unroll
  for (int m = 0; m < MT; ++m) {
    const int u = min(u0 + (warp * MT + m) * 2 + (mi & 1), nu - 1);
    const int tap = u % taps, c8 = u / taps - c8lo;
    const int dx = tap % g.ksize, dy = (tap / g.ksize) % g.ksize, dz = tap / (g.ksize * g.ksize);
    // (a unit past the end repeats the last one; it lies in a staged octet
    // only if that octet is this CTA's, which c8 < nc8 keeps true)
    const int c8s = min(max(c8, 0), nc8 - 1);
    aoff[m] = xbase + 16u * (uint32_t)(c8s * HV + dx + P.hx * (dy + P.hy * dz) +
                                       g.stride * (r + P.hx * (mi >> 1)));
  }
  float acc[MT][NT8][4];
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int j = 0; j < NT8; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[m][j][q] = 0.0f;

  const int nb = P.nbx * P.nby * P.nbz;
  const int b0 = blockIdx.x * P.bricks_per_chunk, b1 = min(nb, b0 + P.bricks_per_chunk);
  const int oct = g.Cout / 8;
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  for (int b = b0; b < b1; ++b) {
    const int bx = (b % P.nbx) * BX, by = ((b / P.nbx) % P.nby) * BY, bz = (b / (P.nbx * P.nby)) * BZ;
    __syncthreads();   // the previous brick is consumed
    // a voxel's position is worked out once for all its channel octets
    for (int w = threadIdx.x; w < HV; w += CBW_NT) {
      const int wy = w / P.hx, wz = wy / P.hy;
      const int x = bx * g.stride - pad + w - wy * P.hx, y = by * g.stride - pad + wy - wz * P.hy,
                z = bz * g.stride - pad + wz;
      const bool in = x >= 0 && y >= 0 && z >= 0 && x < g.nxi && y < g.nyi && z < g.nzi;
      const long va = g.up ? (x >> 1) + (long)g.nxa * ((y >> 1) + (long)g.nya * (z >> 1))
                           : x + (long)g.nxi * (y + (long)g.nyi * z);
      const long vs = x + (long)g.nxi * (y + (long)g.nyi * z);
      for (int c = 0; c < nc8; ++c) {
        const int ch = 8 * (c8lo + c);
        uint4 v = zero4;
        if (in) v = *reinterpret_cast<const uint4*>(ch < g.Ca ? P.A + va * g.Ca + ch : P.S + vs * g.Cs + (ch - g.Ca));
        Xs[c * HV + w] = v;
      }
    }
    {
      const int j = threadIdx.x % NT8;   // consecutive threads read a voxel's consecutive octets
#pragma unroll
      for (int q = 0; q < BV * NT8 / CBW_NT + (BV * NT8 < CBW_NT ? 1 : 0); ++q) {
        const int v = threadIdx.x / NT8 + q * (CBW_NT / NT8);
        if (v >= BV) break;
        const int x = bx + v % BX, y = by + (v / BX) % BY, z = bz + v / (BX * BY);
        const bool in = x < g.nxo && y < g.nyo && z < g.nzo && n0 / 8 + j < oct;
        uint4 pl[3] = {zero4, zero4, zero4};
        if (in) {
          float gv[8];
          load8f(P.G + (x + (long)g.nxo * (y + (long)g.nyo * z)) * g.Cout + n0 + 8 * j, P.g_aligned, gv);
          split8(gv, pl);
        }
#pragma unroll
        for (int t = 0; t < 3; ++t) Gs[(t * NT8 + j) * BV + v] = pl[t];
      }
    }
    __syncthreads();
#pragma unroll 1
    for (int s = 0; s < BV / 16; ++s) {
      const uint32_t vs = 16u * (uint32_t)(g.stride * P.hx * (2 * (s % (BY / 2)) + P.hy * (s / (BY / 2))));
      uint32_t bf[3][NT8][2];
#pragma unroll
      for (int t = 0; t < 3; ++t) {
        if constexpr (NT8 == 1) {
          uint32_t q[2];
          ldsm2t(q, gbase + 16u * (uint32_t)(t * BV + 16 * s + (lane & 15)));
          bf[t][0][0] = q[0];
          bf[t][0][1] = q[1];
        } else {
#pragma unroll
          for (int j = 0; j < NT8; j += 2) {
            uint32_t q[4];
            ldsm4t(q, gbase + 16u * (uint32_t)((t * NT8 + j + (mi >> 1)) * BV + 16 * s + 8 * (mi & 1) + r));
            bf[t][j][0] = q[0];
            bf[t][j][1] = q[1];
            bf[t][j + 1][0] = q[2];
            bf[t][j + 1][1] = q[3];
          }
        }
      }
#pragma unroll
      for (int m = 0; m < MT; ++m) {
        uint32_t a[4];
        ldsm4t(a, aoff[m] + vs);
#pragma unroll
        for (int j = 0; j < NT8; ++j) {
          float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          mma(d, a, bf[2][j][0], bf[2][j][1]);
          mma(d, a, bf[1][j][0], bf[1][j][1]);
          mma(d, a, bf[0][j][0], bf[0][j][1]);
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[m][j][q] += d[q];
        }
      }
    }
  }
  // fragment (row = channel of the unit, lane / 4; columns 2 (lane % 4) + {0, 1})
#pragma unroll
  for (int m = 0; m < MT; ++m)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int u = u0 + (warp * MT + m) * 2 + h;
      if (u >= nu) continue;
      const int tap = u % taps, ci = 8 * (u / taps) + (lane >> 2);
      float* row = P.part + (((long)blockIdx.x * taps + tap) * g.Cin + ci) * g.Cout;
#pragma unroll
      for (int j = 0; j < NT8; ++j) {
        const int co = n0 + 8 * j + 2 * (lane & 3);
        if (co < g.Cout) {
          float v0 = acc[m][j][2 * h], v1 = acc[m][j][2 * h + 1];
          if (v0 != v0) v0 = dw_entry(P, tap, ci, co, b0, b1);
          if (v1 != v1) v1 = dw_entry(P, tap, ci, co + 1, b0, b1);
          row[co] = v0;
          row[co + 1] = v1;
        }
      }
    }
}

struct DxArgs {
  const float* G;
  int g_aligned;
  const __nv_bfloat16* W;
  ConvGeom g;
  int nbx, nby, nbz;   // bricks per axis of the coarse (class) grid
  int co8;             // output-channel octets staged at a time (1 or 2)
  int ldo;             // floats per voxel of the target
  int acc;             // add to the target instead of overwriting it
  int w_aligned;       // W is 16-byte aligned
  int o_aligned;       // out is 8-byte aligned
  float* out;
};

// One entry of the input gradient, term by term (as dw_entry)
__device__ __noinline__ float dx_entry(const DxArgs& P, int x, int y, int z, int ci) {
  const ConvGeom& g = P.g;
  const int pad = g.ksize / 2;
  float s = 0.0f;
  for (int tap = 0; tap < g.ksize * g.ksize * g.ksize; ++tap) {
    const int ax = x + pad - tap % g.ksize, ay = y + pad - (tap / g.ksize) % g.ksize,
              az = z + pad - tap / (g.ksize * g.ksize);
    if (ax < 0 || ay < 0 || az < 0 || (g.stride == 2 && ((ax | ay | az) & 1))) continue;
    const int xo = ax / g.stride, yo = ay / g.stride, zo = az / g.stride;
    if (xo >= g.nxo || yo >= g.nyo || zo >= g.nzo) continue;
    const float* gp = P.G + (xo + (long)g.nxo * (yo + (long)g.nyo * zo)) * g.Cout;
    const __nv_bfloat16* wp = P.W + ((long)tap * g.Cin + ci) * g.Cout;
    for (int co = 0; co < g.Cout; ++co) s = fmaf(gp[co], __bfloat162float(wp[co]), s);
    if (s != s) return s;
  }
  return s;
}

template <int NT8>
__global__ void __launch_bounds__(CBW_NT)
k_conv_dx(const __grid_constant__ DxArgs P) {
  extern __shared__ __align__(128) unsigned char cb_sm[];
  const ConvGeom& g = P.g;
  constexpr int NC = NT8 * 8;
  const int pad = g.ksize / 2, st = g.stride;
  const int co8 = P.co8;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int mi = lane >> 3, r = lane & 7;
  const int nb = P.nbx * P.nby * P.nbz;
  const int cls = blockIdx.x / nb, b = blockIdx.x % nb;
  const int px = cls & 1, py = (cls >> 1) & 1, pz = cls >> 2;   // parities (stride 2)
  const int cx = (b % P.nbx) * DX, cy = ((b / P.nbx) % P.nby) * DY, cz = (b / (P.nbx * P.nby)) * DZ;
  const int ci0 = blockIdx.y * NC;
  // taps of this class: o = (v + pad - d) / stride, as an offset from the coarse coordinate
  __shared__ int s_tap[27], s_off[27];
  __shared__ int s_nt;
  uint4* Gs = reinterpret_cast<uint4*>(cb_sm);       // [3][co8][DH], then one zero row
  const int zrow = 3 * co8 * DH;
  uint4* Ws = Gs + zrow + 1;                         // [units][NC]
  if (threadIdx.x == 0) {
    int n = 0;
    for (int dz = 0; dz < g.ksize; ++dz)
      for (int dy = 0; dy < g.ksize; ++dy)
        for (int dx = 0; dx < g.ksize; ++dx) {
          const int ax = px + pad - dx, ay = py + pad - dy, az = pz + pad - dz;
          if (st == 2 && ((ax | ay | az) & 1)) continue;
          const int ox = st == 2 ? ax / 2 : ax, oy = st == 2 ? ay / 2 : ay, oz = st == 2 ? az / 2 : az;   // -1, 0 or 1
          s_tap[n] = dx + g.ksize * (dy + g.ksize * dz);
          s_off[n] = (ox + 1) + (DX + 2) * ((oy + 1) + (DY + 2) * (oz + 1));
          ++n;
        }
    s_nt = n;
    Gs[zrow] = make_uint4(0u, 0u, 0u, 0u);
  }
  __syncthreads();
  const int nt = s_nt;
  const int units = nt * co8, usteps = (units + 1) / 2;
  const int oct = g.Cout / 8;
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  const uint32_t gbase = smem_u32(Gs), wbase = smem_u32(Ws);
  // tiles 2 warp, 2 warp + 1: two x rows (y = 2 (tile % 4) + {0, 1}) of plane tile / 4
  int vpos[2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = 2 * warp + i;
    vpos[i] = r + (DX + 2) * ((2 * (t % (DY / 2)) + (mi & 1)) + (DY + 2) * (t / (DY / 2)));
  }
  float acc[2][NT8][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NT8; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0f;

  // the brick voxels this thread stages (the same for every group of output
  // channels): offsets into the gradient, -1 outside the grid
  const int lco = co8 - 1;   // log2 of co8 (1 or 2)
  const int sc = threadIdx.x & lco, sw = threadIdx.x >> lco;
  long goff[5];
#pragma unroll
  for (int q = 0; q < 5; ++q) {
    const int w = sw + q * (CBW_NT >> lco);
    const int x = cx - 1 + w % (DX + 2), y = cy - 1 + (w / (DX + 2)) % (DY + 2), z = cz - 1 + w / ((DX + 2) * (DY + 2));
    const bool in = w < DH && x >= 0 && y >= 0 && z >= 0 && x < g.nxo && y < g.nyo && z < g.nzo;
    goff[q] = in ? (x + (long)g.nxo * (y + (long)g.nyo * z)) * g.Cout + 8 * sc : -1;
  }
  for (int o0 = 0; o0 < oct; o0 += co8) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int w = sw + q * (CBW_NT >> lco);
      if (w >= DH) break;
      const bool in = goff[q] >= 0 && o0 + sc < oct;
      uint4 pl[3] = {zero4, zero4, zero4};
      if (in) {
        float gv[8];
        load8f(P.G + goff[q] + 8 * o0, P.g_aligned, gv);
        split8(gv, pl);
      }
#pragma unroll
      for (int t = 0; t < 3; ++t) Gs[(t * co8 + sc) * DH + w] = pl[t];
    }
    for (int e = threadIdx.x; e < 2 * usteps * NC; e += CBW_NT) {
      const int c = e & lco, n = (e >> lco) % NC, k = (e >> lco) / NC;   // unit k co8 + c
      const int u = k * co8 + c;
      if (u >= 2 * usteps) continue;
      const bool in = u < units && ci0 + n < g.Cin && o0 + c < oct;
      Ws[u * NC + n] = in ? load8(P.W + ((long)s_tap[k] * g.Cin + ci0 + n) * g.Cout + 8 * (o0 + c), P.w_aligned)
                          : zero4;
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < usteps; ++k) {
      const int u = 2 * k + (mi >> 1);   // this lane's unit of the step
      uint32_t bf[NT8][2];
#pragma unroll
      for (int j = 0; j + 1 < NT8; j += 2) {
        uint32_t q[4];
        ldsm4(q, wbase + 16u * (uint32_t)((2 * k + (mi & 1)) * NC + 8 * (j + (mi >> 1)) + r));
        bf[j][0] = q[0];
        bf[j][1] = q[1];
        bf[j + 1][0] = q[2];
        bf[j + 1][1] = q[3];
      }
      if constexpr (NT8 % 2 == 1) {
        uint32_t q[2];
        ldsm2(q, wbase + 16u * (uint32_t)((2 * k + (mi & 1)) * NC + 8 * (NT8 - 1) + r));
        bf[NT8 - 1][0] = q[0];
        bf[NT8 - 1][1] = q[1];
      }
      const bool real = u < units;
      const int c = real ? u & lco : 0;
      const int uo = real ? c * DH + s_off[u >> lco] : 0;
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        uint32_t a[3][4];
#pragma unroll
        for (int t = 0; t < 3; ++t)
          ldsm4(a[t], gbase + 16u * (uint32_t)(real ? t * co8 * DH + uo + vpos[i] : zrow));
#pragma unroll
        for (int j = 0; j < NT8; ++j) {
          float d[4] = {0.0f, 0.0f, 0.0f, 0.0f};
          mma(d, a[2], bf[j][0], bf[j][1]);
          mma(d, a[1], bf[j][0], bf[j][1]);
          mma(d, a[0], bf[j][0], bf[j][1]);
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[i][j][q] += d[q];
        }
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int t = 2 * warp + i;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int x = st * (cx + (lane >> 2)) + (st == 2 ? px : 0);
      const int y = st * (cy + 2 * (t % (DY / 2)) + h) + (st == 2 ? py : 0);
      const int z = st * (cz + t / (DY / 2)) + (st == 2 ? pz : 0);
      if (x >= g.nxi || y >= g.nyi || z >= g.nzi) continue;
      float* row = P.out + (x + (long)g.nxi * (y + (long)g.nyi * z)) * P.ldo;
#pragma unroll
      for (int j = 0; j < NT8; ++j) {
        const int ci = ci0 + 8 * j + 2 * (lane & 3);
        if (ci >= g.Cin) continue;
        float v0 = acc[i][j][2 * h], v1 = acc[i][j][2 * h + 1];
        if (v0 != v0) v0 = dx_entry(P, x, y, z, ci);
        if (v1 != v1) v1 = dx_entry(P, x, y, z, ci + 1);
        if (P.o_aligned) {
          float2* p = reinterpret_cast<float2*>(row + ci);
          if (P.acc) {
            const float2 old = *p;
            v0 = old.x + v0;
            v1 = old.y + v1;
          }
          *p = make_float2(v0, v1);
        } else {
          row[ci] = P.acc ? row[ci] + v0 : v0;
          row[ci + 1] = P.acc ? row[ci + 1] + v1 : v1;
        }
      }
    }
  }
}

// dW[e] = sum of the chunks' partials: a CTA takes 32 entries, warp w every
// eighth chunk from w on, and the eight sums are added in order
__global__ void __launch_bounds__(256)
k_sum_chunks(const float* __restrict__ part, int nchunk, long nw, float* __restrict__ dW) {
  __shared__ float sh[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long e = blockIdx.x * 32L + lane;
  float s = 0.0f;
  if (e < nw)
#pragma unroll 4
    for (int c = w; c < nchunk; c += 8) s += part[(long)c * nw + e];
  sh[w][lane] = s;
  __syncthreads();
  if (w == 0 && e < nw) {
#pragma unroll
    for (int q = 1; q < 8; ++q) s += sh[q][lane];
    dW[e] = s;
  }
}

template <int NT8, int MT>
static int launch_dw(psc_ctx* ctx, const DwArgs& P, dim3 grid, size_t smem, cudaStream_t st) {
  PSC_CUDA(ctx, psc_smem_optin(k_conv_dw<NT8, MT>));
  k_conv_dw<NT8, MT><<<grid, CBW_NT, smem, st>>>(P);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

template <int NT8>
static int launch_dx(psc_ctx* ctx, const DxArgs& P, dim3 grid, size_t smem, cudaStream_t st) {
  PSC_CUDA(ctx, psc_smem_optin(k_conv_dx<NT8>));
  k_conv_dx<NT8><<<grid, CBW_NT, smem, st>>>(P);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

// Gradient through the activation into gm, bias gradient dB and weight
// gradient dW; `work` holds the partial sums.
int psc_conv_bwd_weights(psc_ctx* ctx, const ConvGeom& g, const __nv_bfloat16* a, const __nv_bfloat16* s,
                         const float* gout, const __nv_bfloat16* out, int act, float* gm, float* dW, float* dB,
                         float* work, long work_floats, cudaStream_t st) {
  const int taps = g.ksize * g.ksize * g.ksize;
  const long nvo = (long)g.nxo * g.nyo * g.nzo;
  const long nw = (long)taps * g.Cin * g.Cout;
  PSC_REQUIRE(ctx, nw <= work_floats, "conv3d_bwd: work buffer too small");
  {
    const int rows = 256 / (g.Cout / 8);
    long nb = std::max<long>(1, std::min<long>(148 * 4, nvo / (4 * rows)));
    nb = std::max<long>(1, std::min<long>(nb, work_floats / g.Cout));
    const long vchunk = (nvo + nb - 1) / nb;
    nb = (nvo + vchunk - 1) / vchunk;
    const int aligned = ((reinterpret_cast<uintptr_t>(gout) | reinterpret_cast<uintptr_t>(gm) |
                          reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    k_conv_prep<<<(int)nb, 256, 0, st>>>(gout, out, nvo, g.Cout, act, aligned, gm, vchunk, work);
    PSC_LAUNCH_CHECK(ctx);
    k_conv_bias<<<psc_div_up(g.Cout, 8), 256, 0, st>>>(work, (int)nb, g.Cout, dB);
    PSC_LAUNCH_CHECK(ctx);
  }
  const int oct = g.Cout / 8, nu = (g.Cin / 8) * taps;
  const int nt8 = oct == 1 ? 1 : (oct == 2 ? 2 : 4);
  DwArgs P;
  P.A = a; P.S = s; P.G = gm; P.g = g; P.part = work;
  P.g_aligned = (reinterpret_cast<uintptr_t>(gm) & 15) == 0;
  P.nbx = psc_div_up(g.nxo, BX); P.nby = psc_div_up(g.nyo, BY); P.nbz = psc_div_up(g.nzo, BZ);
  P.hx = (BX - 1) * g.stride + g.ksize; P.hy = (BY - 1) * g.stride + g.ksize; P.hz = (BZ - 1) * g.stride + g.ksize;
  // units per CTA (16 MT): the split that pads least, a CTA's staging costing
  // about as much as 24 units of MMAs; 9 only with one column tile (registers)
  const int cand[4] = {1, 2, 4, 9};
  int mt = 1;
  size_t smem = 0;
  long best = -1;
  for (int q = 0; q < (nt8 == 1 ? 4 : 3); ++q) {
    const int uc = 16 * cand[q];
    const int nc8 = std::min(g.Cin / 8, (uc - 1 + taps - 1) / taps + 1);
    const size_t sm = ((size_t)nc8 * P.hx * P.hy * P.hz + 3 * (size_t)nt8 * BV) * 16;
    const long cost = (long)psc_div_up(nu, uc) * (uc + 24);
    if (sm <= 200 * 1024 && (best < 0 || cost <= best)) {
      best = cost;
      mt = cand[q];
      smem = sm;
      P.nc8 = nc8;
    }
  }
  PSC_REQUIRE(ctx, best >= 0, "conv3d_bwd: brick does not fit in shared memory");
  const int gy = psc_div_up(nu, 16 * mt), gz = psc_div_up(oct, nt8);
  const int nb = P.nbx * P.nby * P.nbz;
  long nchunk = std::max<long>(1, std::min<long>(nb, 148L * 6 / ((long)gy * gz)));
  nchunk = std::max<long>(1, std::min<long>(nchunk, work_floats / nw));
  P.bricks_per_chunk = psc_div_up(nb, nchunk);
  nchunk = psc_div_up(nb, P.bricks_per_chunk);
  const dim3 grid((unsigned)nchunk, gy, gz);
  int rc = 2;
#define PSC_DW(N, M) if (nt8 == N && mt == M) rc = launch_dw<N, M>(ctx, P, grid, smem, st);
  PSC_DW(1, 1) PSC_DW(1, 2) PSC_DW(1, 4) PSC_DW(1, 9) PSC_DW(2, 1) PSC_DW(2, 2) PSC_DW(2, 4) PSC_DW(4, 1)
  PSC_DW(4, 2) PSC_DW(4, 4)
#undef PSC_DW
  if (rc) return rc;
  k_sum_chunks<<<psc_div_up(nw, 32), 256, 0, st>>>(work, (int)nchunk, nw, dW);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

// Input gradient of all Cin channels into out (ldo floats per voxel, not
// overlapping gm), from the gm that psc_conv_bwd_weights left.
int psc_conv_bwd_input(psc_ctx* ctx, const ConvGeom& g, const __nv_bfloat16* w, const float* gm, float* out, int ldo,
                       int acc, cudaStream_t st) {
  DxArgs P;
  P.G = gm;
  P.g_aligned = (reinterpret_cast<uintptr_t>(gm) & 15) == 0;
  P.W = w; P.g = g; P.out = out; P.ldo = ldo; P.acc = acc;
  P.w_aligned = (reinterpret_cast<uintptr_t>(w) & 15) == 0;
  P.o_aligned = (reinterpret_cast<uintptr_t>(out) & 7) == 0;
  P.co8 = g.Cout >= 16 ? 2 : 1;
  const int cls = g.stride == 2 ? 8 : 1;
  P.nbx = psc_div_up(psc_div_up(g.nxi, g.stride), DX);
  P.nby = psc_div_up(psc_div_up(g.nyi, g.stride), DY);
  P.nbz = psc_div_up(psc_div_up(g.nzi, g.stride), DZ);
  const int c8 = g.Cin / 8;
  int nt8 = 4;
  for (int t : {1, 2, 5})   // the widest block among those that pad least
    if ((long)psc_div_up(c8, t) * t < (long)psc_div_up(c8, nt8) * nt8 ||
        ((long)psc_div_up(c8, t) * t == (long)psc_div_up(c8, nt8) * nt8 && t > nt8))
      nt8 = t;
  const int units = (g.stride == 2 ? 8 : g.ksize * g.ksize * g.ksize) * P.co8;   // most taps of a class
  const size_t smem = ((size_t)3 * P.co8 * DH + 1 + (size_t)((units + 1) / 2 * 2) * nt8 * 8) * 16;
  const dim3 grid(P.nbx * P.nby * P.nbz * cls, psc_div_up(c8, nt8));
  switch (nt8) {
    case 1: return launch_dx<1>(ctx, P, grid, smem, st);
    case 2: return launch_dx<2>(ctx, P, grid, smem, st);
    case 4: return launch_dx<4>(ctx, P, grid, smem, st);
    default: return launch_dx<5>(ctx, P, grid, smem, st);
  }
}
