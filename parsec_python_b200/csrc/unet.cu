// Learned initial density: BF16 3-D convolution forward with FP32
// accumulation on the CUDA cores, the C ABI of the convolutions (tensor-core
// forward: conv_tc.cu, backward: conv_bwd.cu), the loss and the Adam step.
//
// The reference only consumes a predicted density (it reads a file in
// V_ion/pseudoDiag_ML4Den_poisson.py:12-586 and renormalises it); the network
// that produces it is new here.  Activations are channels-last BF16 tensors
// [voxel][C] on a grid with x fastest (voxel = x + nx (y + ny z)), C a
// multiple of 8.  Weights are BF16 [tap][Cin][Cout] (tap = dx + 3 (dy + 3 dz)
// for 3x3x3 kernels, one tap for 1x1x1), biases FP32.  Gradients are FP32.
//
// One convolution reads a "virtual input" of Cin = Ca + Cs channels: the
// first Ca from tensor A -- nearest-neighbour upsampled x2 when `up` is set,
// which is how the decoder grows back to the finer grid -- and the last Cs
// from the skip tensor S at the virtual input's own resolution.  So the
// upsample and the concatenation of an encoder-decoder are never written out.
// Stride 2 halves the grid (output dims ceil(n/2)), padding is 1 for 3x3x3.
#include "psc_internal.cuh"
#include "../../include/psc.h"

#include <cuda_bf16.h>

#include "conv_geom.cuh"

#include <algorithm>

namespace {

__device__ __forceinline__ void unpack8(const uint4 u, float* f) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

constexpr int FWD_NT = 128;
constexpr float LEAK = 0.0625f;   // leaky-ReLU slope below zero
constexpr int WTILE = 256;   // weights staged per tap: input-chunk x output-chunk = 256 floats (27 KB for 27 taps)

}  // namespace

// ---------------------------------------------------------------------------
// forward: out[o][co] = act(b[co] + sum_tap sum_ci vin(o s + tap - pad)[ci] W[tap][ci][co])
// act: 0 identity, 1 ReLU, 2 leaky ReLU (slope 1/16 below zero).
// One thread per output voxel, COT output channels per CTA (blockIdx.y).
// ---------------------------------------------------------------------------
template <int COT>
__global__ void __launch_bounds__(FWD_NT)
k_conv_fwd(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ S,
           const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias, ConvGeom g, int act,
           __nv_bfloat16* __restrict__ out, float* __restrict__ out32) {
  constexpr int CIN_CHUNK = WTILE / COT;
  __shared__ __align__(16) float ws[27 * WTILE];
  const int taps = g.ksize * g.ksize * g.ksize;
  const int pad = g.ksize / 2;
  const int co0 = blockIdx.y * COT;
  const long nvo = (long)g.nxo * g.nyo * g.nzo;
  const long vo = (long)blockIdx.x * FWD_NT + threadIdx.x;
  const bool valid = vo < nvo;
  int xo = 0, yo = 0, zo = 0;
  if (valid) {
    xo = (int)(vo % g.nxo);
    const long r = vo / g.nxo;
    yo = (int)(r % g.nyo);
    zo = (int)(r / g.nyo);
  }
  float acc[COT];
#pragma unroll
  for (int j = 0; j < COT; ++j) acc[j] = bias[co0 + j];
  for (int cc = 0; cc < g.Cin; cc += CIN_CHUNK) {
    const int cn = min(CIN_CHUNK, g.Cin - cc);
    __syncthreads();
    for (int e = threadIdx.x; e < taps * cn * COT; e += FWD_NT) {
      const int co = e % COT;
      const int r = e / COT;
      const int ci = r % cn, tap = r / cn;
      ws[(tap * CIN_CHUNK + ci) * COT + co] =
          __bfloat162float(W[((long)tap * g.Cin + cc + ci) * g.Cout + co0 + co]);
    }
    __syncthreads();
    if (!valid) continue;
    for (int tap = 0; tap < taps; ++tap) {
      const int dx = tap % g.ksize, dy = (tap / g.ksize) % g.ksize, dz = tap / (g.ksize * g.ksize);
      const int xi = xo * g.stride + dx - pad, yi = yo * g.stride + dy - pad, zi = zo * g.stride + dz - pad;
      if (xi < 0 || yi < 0 || zi < 0 || xi >= g.nxi || yi >= g.nyi || zi >= g.nzi) continue;
      for (int c8 = 0; c8 < cn; c8 += 8) {
        float x[8];
        unpack8(conv_vin8(A, S, g, xi, yi, zi, cc + c8), x);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float* wr = ws + (tap * CIN_CHUNK + c8 + j) * COT;
#pragma unroll
          for (int co = 0; co < COT; co += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(wr + co);
            acc[co] = fmaf(x[j], w4.x, acc[co]);
            acc[co + 1] = fmaf(x[j], w4.y, acc[co + 1]);
            acc[co + 2] = fmaf(x[j], w4.z, acc[co + 2]);
            acc[co + 3] = fmaf(x[j], w4.w, acc[co + 3]);
          }
        }
      }
    }
  }
  if (!valid) return;
#pragma unroll
  for (int j = 0; j < COT; ++j) {
    const float a = acc[j];
    const float v = act == 1 ? fmaxf(a, 0.0f) : (act == 2 ? (a > 0.0f ? a : LEAK * a) : a);
    out[vo * g.Cout + co0 + j] = __float2bfloat16_rn(v);
    if (out32) out32[vo * g.Cout + co0 + j] = v;
  }
}

// ---------------------------------------------------------------------------
// forward of a stride-1 layer with 8 output channels per CTA (the full-grid
// layers).  Four voxels of one x row (8 apart, so that a warp's loads are
// consecutive) by 8 channels per thread: a weight fetched from shared memory
// serves four voxels, the products are packed pairs of channels, and the
// input brick with its halo is staged once for all the taps.  The plain
// kernel above fetches two weight vectors per input value for eight
// multiply-adds and reads the input 27 times through L1 (852 us for the three
// layers of a 90^3 pass); this one takes 450 us and is bound by the FP32 pipe.  Every output adds its terms in k_conv_fwd<8>'s order (32
// input channels at a time, taps, channels), so the results are the same
// bits.  A tap outside the grid adds a zero product here, which an infinite or
// NaN weight would turn into NaN: a thread that ends with a NaN takes its
// voxels' sums again without those taps (conv_fwd_point; 0.8 % of a 90^3 pass).
// ---------------------------------------------------------------------------
constexpr int F8_X = 32, F8_Y = 4, F8_Z = 4;   // voxels per CTA (128 threads)

// The taps of one staged chunk of NC channel octets.  Eight warps per SM do
// not hide the shared-memory latency by themselves, so the weights of the next
// input channel and the inputs of the next octet are loaded one step ahead of
// the products (the weights lie in the order they are used in, and 8 floats
// past the last ones belong to the CTA).
template <int KS, int NC>
__device__ __forceinline__ void fwd8_chunk(const uint4* x, int hx, int hxy, int hv, const float* wt,
                                           float2 (&acc)[4][4]) {
  float4 wa = *reinterpret_cast<const float4*>(wt), wb = *reinterpret_cast<const float4*>(wt + 4);
  uint4 xv[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) xv[i] = x[8 * i];
#pragma unroll 1
  for (int r = 0; r < KS * KS; ++r) {
    const uint4* xr = x + (r / KS) * hxy + (r % KS) * hx;
    const int rn = r + 1 < KS * KS ? r + 1 : 0;
    const uint4* xnext = x + (rn / KS) * hxy + (rn % KS) * hx;   // the row of taps after this one
#pragma unroll
    for (int dx = 0; dx < KS; ++dx)
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const uint4* xp = c + 1 < NC ? xr + (c + 1) * hv + dx : (dx + 1 < KS ? xr + dx + 1 : xnext);
        uint4 xn[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) xn[i] = xp[8 * i];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          wt += 8;
          const float4 na = *reinterpret_cast<const float4*>(wt);
          const float4 nb = *reinterpret_cast<const float4*>(wt + 4);
          const float2 w2[4] = {make_float2(wa.x, wa.y), make_float2(wa.z, wa.w), make_float2(wb.x, wb.y),
                                make_float2(wb.z, wb.w)};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const uint32_t word = j / 2 == 0 ? xv[i].x : (j / 2 == 1 ? xv[i].y : (j / 2 == 2 ? xv[i].z : xv[i].w));
            const float v = __uint_as_float(j & 1 ? word & 0xffff0000u : word << 16);
#pragma unroll
            for (int p = 0; p < 4; ++p) acc[i][p] = __ffma2_rn(make_float2(v, v), w2[p], acc[i][p]);
          }
          wa = na;
          wb = nb;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) xv[i] = xn[i];
      }
  }
}

// One output before the activation, taps outside the grid skipped; a sum that
// has become NaN stays one.
__device__ __noinline__ float conv_fwd_point(const __nv_bfloat16* A, const __nv_bfloat16* S, const __nv_bfloat16* W,
                                             float sum, const ConvGeom& g, int x, int y, int z, int co) {
  const int pad = g.ksize / 2, taps = g.ksize * g.ksize * g.ksize;
  for (int cc = 0; cc < g.Cin; cc += WTILE / 8) {
    const int cn = min(WTILE / 8, g.Cin - cc);
    for (int tap = 0; tap < taps; ++tap) {
      const int xi = x + tap % g.ksize - pad, yi = y + (tap / g.ksize) % g.ksize - pad,
                zi = z + tap / (g.ksize * g.ksize) - pad;
      if (xi < 0 || yi < 0 || zi < 0 || xi >= g.nxi || yi >= g.nyi || zi >= g.nzi) continue;
      for (int c = 0; c < cn; c += 8) {
        float v[8];
        unpack8(conv_vin8(A, S, g, xi, yi, zi, cc + c), v);
#pragma unroll
        for (int j = 0; j < 8; ++j)
          sum = fmaf(v[j], __bfloat162float(W[((long)tap * g.Cin + cc + c + j) * g.Cout + co]), sum);
      }
      if (sum != sum) return sum;
    }
  }
  return sum;
}

template <int KS>
__global__ void __launch_bounds__(FWD_NT)
k_conv_fwd8(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ S,
            const __nv_bfloat16* __restrict__ W, const float* __restrict__ bias, ConvGeom g, int act, int nbx, int nby,
            int aligned, __nv_bfloat16* __restrict__ out, float* __restrict__ out32) {
  extern __shared__ __align__(16) unsigned char f8_sm[];
  constexpr int PAD = KS / 2, TAPS = KS * KS * KS;
  constexpr int HX = F8_X + 2 * PAD, HY = F8_Y + 2 * PAD, HZ = F8_Z + 2 * PAD, HV = HX * HY * HZ;
  constexpr int CH = WTILE / 8;                        // input channels per chunk
  const int nc_max = min(CH, g.Cin) / 8;
  uint4* xs = reinterpret_cast<uint4*>(f8_sm);                      // [octet][HV]
  float* ws = reinterpret_cast<float*>(xs + (size_t)nc_max * HV);   // [tap][channel of the chunk][8]
  const int tx = threadIdx.x & 7, ty = (threadIdx.x >> 3) & 3, tz = threadIdx.x >> 5;
  const int b = blockIdx.x;
  const int x0 = (b % nbx) * F8_X, y0 = ((b / nbx) % nby) * F8_Y, z0 = (b / (nbx * nby)) * F8_Z;
  const int co0 = blockIdx.y * 8;
  float2 acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int p = 0; p < 4; ++p) acc[i][p] = make_float2(bias[co0 + 2 * p], bias[co0 + 2 * p + 1]);
  const uint4 zero4 = make_uint4(0u, 0u, 0u, 0u);
  for (int cc = 0; cc < g.Cin; cc += CH) {
    const int cn = min(CH, g.Cin - cc), nc = cn / 8;
    __syncthreads();
    for (int e = threadIdx.x; e < nc * HV; e += FWD_NT) {
      const int c = e / HV, w = e - c * HV;
      const int x = x0 - PAD + w % HX, y = y0 - PAD + (w / HX) % HY, z = z0 - PAD + w / (HX * HY);
      const bool in = x >= 0 && y >= 0 && z >= 0 && x < g.nxi && y < g.nyi && z < g.nzi;
      xs[e] = in ? conv_vin8(A, S, g, x, y, z, cc + 8 * c) : zero4;
    }
    for (int e = threadIdx.x; e < TAPS * cn * 8; e += FWD_NT) {
      const int co = e & 7, r = e >> 3, ci = r % cn, tap = r / cn;
      ws[(tap * cn + ci) * 8 + co] = __bfloat162float(W[((long)tap * g.Cin + cc + ci) * g.Cout + co0 + co]);
    }
    __syncthreads();
    const uint4* xt = xs + (tz * HY + ty) * HX + tx;
    switch (nc) {
      case 1: fwd8_chunk<KS, 1>(xt, HX, HX * HY, HV, ws, acc); break;
      case 2: fwd8_chunk<KS, 2>(xt, HX, HX * HY, HV, ws, acc); break;
      case 3: fwd8_chunk<KS, 3>(xt, HX, HX * HY, HV, ws, acc); break;
      default: fwd8_chunk<KS, 4>(xt, HX, HX * HY, HV, ws, acc); break;
    }
  }
  const int y = y0 + ty, z = z0 + tz;
  if (y >= g.nyo || z >= g.nzo) return;
  bool nan = false;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int p = 0; p < 4; ++p) nan |= acc[i][p].x != acc[i][p].x || acc[i][p].y != acc[i][p].y;
  if (nan) {
#pragma unroll 1
    for (int e = 0; e < 4 * 8; ++e) {
      const int x = x0 + tx + 8 * (e >> 3), co = co0 + (e & 7);
      if (x >= g.nxo) break;
      const float a = conv_fwd_point(A, S, W, bias[co], g, x, y, z, co);
      const float v = act == 1 ? fmaxf(a, 0.0f) : (act == 2 ? (a > 0.0f ? a : LEAK * a) : a);
      const long q = (x + (long)g.nxo * (y + (long)g.nyo * z)) * g.Cout + co;
      out[q] = __float2bfloat16_rn(v);
      if (out32) out32[q] = v;
    }
    return;
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int x = x0 + tx + 8 * i;
    if (x >= g.nxo) continue;
    const long vo = x + (long)g.nxo * (y + (long)g.nyo * z);
    float v[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const float a = j & 1 ? acc[i][j >> 1].y : acc[i][j >> 1].x;
      v[j] = act == 1 ? fmaxf(a, 0.0f) : (act == 2 ? (a > 0.0f ? a : LEAK * a) : a);
    }
    __nv_bfloat16* o = out + vo * g.Cout + co0;
    if (aligned) {
      uint4 pk;
      __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&pk);
#pragma unroll
      for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
      *reinterpret_cast<uint4*>(o) = pk;
      if (out32) {
        float4* q = reinterpret_cast<float4*>(out32 + vo * g.Cout + co0);
        q[0] = make_float4(v[0], v[1], v[2], v[3]);
        q[1] = make_float4(v[4], v[5], v[6], v[7]);
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        o[j] = __float2bfloat16_rn(v[j]);
        if (out32) out32[vo * g.Cout + co0 + j] = v[j];
      }
    }
  }
}

// Split the virtual-input gradient: dA (+)= pool(dvin[:, :Ca]) (sum over the
// 8 fine voxels of each coarse one when up), dS (+)= dvin[:, Ca:].
__global__ void k_split_grad_a(const float* __restrict__ dvin, ConvGeom g, int accumulate, float* __restrict__ dA) {
  const long na = (long)g.nxa * g.nya * g.nza * g.Ca;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < na; e += (long)gridDim.x * blockDim.x) {
    const int c = (int)(e % g.Ca);
    const long va = e / g.Ca;
    float s = 0.0f;
    if (g.up) {
      const int xa = (int)(va % g.nxa);
      const long r = va / g.nxa;
      const int ya = (int)(r % g.nya), za = (int)(r / g.nya);
      for (int d = 0; d < 8; ++d) {
        const int x = 2 * xa + (d & 1), y = 2 * ya + ((d >> 1) & 1), z = 2 * za + (d >> 2);
        if (x < g.nxi && y < g.nyi && z < g.nzi)
          s += dvin[(x + (long)g.nxi * (y + (long)g.nyi * z)) * g.Cin + c];
      }
    } else {
      s = dvin[va * g.Cin + c];
    }
    dA[e] = accumulate ? dA[e] + s : s;
  }
}

__global__ void k_split_grad_s(const float* __restrict__ dvin, ConvGeom g, int accumulate, float* __restrict__ dS) {
  const long ns = (long)g.nxi * g.nyi * g.nzi * g.Cs;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < ns; e += (long)gridDim.x * blockDim.x) {
    const int c = (int)(e % g.Cs);
    const long v = e / g.Cs;
    const float s = dvin[v * g.Cin + g.Ca + c];
    dS[e] = accumulate ? dS[e] + s : s;
  }
}

// MSE on channel 0 of a [n][C] FP32 prediction: per-CTA partial of sum (y-t)^2
// and the gradient 2 (y - t) / n on channel 0 (0 elsewhere).
__global__ void __launch_bounds__(256)
k_mse(const float* __restrict__ y, int C, const float* __restrict__ t, long n, float* __restrict__ grad,
      double* __restrict__ part) {
  __shared__ double sh[8];
  double s = 0.0;
  const float inv = 2.0f / (float)n;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float d = y[i * C] - t[i];
    s += (double)d * d;
    grad[i * C] = inv * d;
    for (int c = 1; c < C; ++c) grad[i * C + c] = 0.0f;
  }
  s = psc_block_sum<double, 256>(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void k_mse_final(const double* __restrict__ part, int np, long n, double* __restrict__ loss) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < np; ++i) s += part[i];
    *loss = s / (double)n;
  }
}

// Adam (Kingma & Ba 2015) on FP32 master weights; the BF16 copy used by the
// convolutions is refreshed in the same pass.
__global__ void k_adam(float* __restrict__ w, __nv_bfloat16* __restrict__ wb, const float* __restrict__ grad,
                       float* __restrict__ m, float* __restrict__ v, long n, float lr, float b1, float b2, float eps,
                       float c1, float c2) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float gi = grad[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    w[i] = wi;
    if (wb) wb[i] = __float2bfloat16_rn(wi);
  }
}

__global__ void k_f32_to_bf16(const float* __restrict__ x, __nv_bfloat16* __restrict__ y, long n) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    y[i] = __float2bfloat16_rn(x[i]);
}

// Network input: channels-last BF16 [n][8]: ch0 = a0 * x0, ch1 = a1 * x1, rest 0
__global__ void k_pack_input(const double* __restrict__ x0, const double* __restrict__ x1, long n, double a0,
                             double a1, __nv_bfloat16* __restrict__ out) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    out[i * 8] = __float2bfloat16_rn((float)(a0 * x0[i]));
    out[i * 8 + 1] = __float2bfloat16_rn((float)(a1 * x1[i]));
#pragma unroll
    for (int c = 2; c < 8; ++c) out[i * 8 + c] = __float2bfloat16_rn(0.0f);
  }
}

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
namespace {
int geom_from(psc_ctx* ctx, const int* gi, ConvGeom& g) {
  g.nxi = gi[0]; g.nyi = gi[1]; g.nzi = gi[2];
  g.nxa = gi[3]; g.nya = gi[4]; g.nza = gi[5];
  g.up = gi[6];
  g.Ca = gi[7]; g.Cs = gi[8];
  g.Cin = g.Ca + g.Cs;
  g.nxo = gi[9]; g.nyo = gi[10]; g.nzo = gi[11];
  g.stride = gi[12]; g.ksize = gi[13]; g.Cout = gi[14];
  PSC_REQUIRE(ctx, g.Ca > 0 && g.Ca % 8 == 0 && g.Cs >= 0 && g.Cs % 8 == 0 && g.Cout % 8 == 0 && g.Cout > 0,
              "conv3d: channel counts must be positive multiples of 8");
  PSC_REQUIRE(ctx, g.stride == 1 || g.stride == 2, "conv3d: stride must be 1 or 2");
  PSC_REQUIRE(ctx, g.ksize == 1 || g.ksize == 3, "conv3d: kernel size must be 1 or 3");
  PSC_REQUIRE(ctx, g.nxi > 0 && g.nyi > 0 && g.nzi > 0 && g.nxo > 0 && g.nyo > 0 && g.nzo > 0,
              "conv3d: empty grid");
  const int ex = g.stride == 1 ? g.nxi : (g.nxi + 1) / 2;
  const int ey = g.stride == 1 ? g.nyi : (g.nyi + 1) / 2;
  const int ez = g.stride == 1 ? g.nzi : (g.nzi + 1) / 2;
  PSC_REQUIRE(ctx, g.nxo == ex && g.nyo == ey && g.nzo == ez, "conv3d: output grid does not match stride");
  PSC_REQUIRE(ctx, g.ksize == 3 || g.stride == 1, "conv3d: 1x1x1 kernels take stride 1");
  PSC_REQUIRE(ctx, g.Cout <= 256, "conv3d: at most 256 output channels");
  if (g.up) {
    PSC_REQUIRE(ctx, g.nxa == (g.nxi + 1) / 2 && g.nya == (g.nyi + 1) / 2 && g.nza == (g.nzi + 1) / 2,
                "conv3d: A must be the virtual grid halved (rounded up) when up = 1");
  } else {
    PSC_REQUIRE(ctx, g.nxa == g.nxi && g.nya == g.nyi && g.nza == g.nzi, "conv3d: A must match the input grid");
  }
  return 0;
}
}  // namespace

extern "C" int psc_conv3d_fwd(psc_ctx* ctx, const int* geom, const void* A, const void* S, const void* W,
                              const float* bias, int act, void* out, float* out32, void* stream) {
  if (!ctx) return 2;
  ConvGeom g;
  if (int rc = geom_from(ctx, geom, g)) return rc;
  PSC_REQUIRE(ctx, act >= 0 && act <= 2, "conv3d_fwd: act must be 0 (identity), 1 (ReLU) or 2 (leaky ReLU)");
  PSC_REQUIRE(ctx, A && W && bias && out && (g.Cs == 0 || S), "conv3d_fwd: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const long nvo = (long)g.nxo * g.nyo * g.nzo;
  const auto* a = static_cast<const __nv_bfloat16*>(A);
  const auto* s = static_cast<const __nv_bfloat16*>(S);
  const auto* w = static_cast<const __nv_bfloat16*>(W);
  auto* o = static_cast<__nv_bfloat16*>(out);
  // the tensor cores where a layer has 32 or more output channels; with 8 (N
  // padded to 16) half of every MMA is padding and the gather costs as much as
  // for 16, so the full-grid layers are faster on the CUDA cores (90^3: 40 -> 8
  // channels 366 against 384 us, 8 -> 8 71 against 279).  Layers of stride 1 whose
  // channels are no multiple of 16 take the eight-channel brick kernel, the
  // rest (16 channels, stride 2) the plain one, whose 27 reads of a voxel hit L1.
  if (ctx->conv_tc == 2 || (ctx->conv_tc == 1 && g.Cout >= 32))
    return psc_conv_tc_forward(ctx, g, a, s, w, bias, act, o, out32, st);
  if (g.Cout % 16 != 0 && g.stride == 1) {
    const int nbx = psc_div_up(g.nxo, F8_X), nby = psc_div_up(g.nyo, F8_Y), nbz = psc_div_up(g.nzo, F8_Z);
    const int pad = g.ksize / 2, taps = g.ksize * g.ksize * g.ksize;
    const size_t hv = (size_t)(F8_X + 2 * pad) * (F8_Y + 2 * pad) * (F8_Z + 2 * pad);
    const int cn = std::min(WTILE / 8, g.Cin);
    const int smem = (int)((size_t)(cn / 8) * hv * 16 + ((size_t)taps * cn + 1) * 8 * sizeof(float));
    const int aligned = ((reinterpret_cast<uintptr_t>(o) | reinterpret_cast<uintptr_t>(out32)) & 15) == 0;
    const dim3 grid(nbx * nby * nbz, g.Cout / 8);
    auto kern = g.ksize == 3 ? k_conv_fwd8<3> : k_conv_fwd8<1>;
    PSC_CUDA(ctx, psc_smem_optin(kern));
    kern<<<grid, FWD_NT, smem, st>>>(a, s, w, bias, g, act, nbx, nby, aligned, o, out32);
  } else if (g.Cout % 16 == 0) {
    dim3 grid(psc_div_up(nvo, FWD_NT), g.Cout / 16);
    k_conv_fwd<16><<<grid, FWD_NT, 0, st>>>(a, s, w, bias, g, act, o, out32);
  } else {
    dim3 grid(psc_div_up(nvo, FWD_NT), g.Cout / 8);
    k_conv_fwd<8><<<grid, FWD_NT, 0, st>>>(a, s, w, bias, g, act, o, out32);
  }
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

extern "C" int psc_conv3d_bwd(psc_ctx* ctx, const int* geom, const void* A, const void* S, const void* W,
                              const float* gout, const void* out, int act, float* gm, float* dvin, float* dA,
                              int acc_a, float* dS, int acc_s, float* dW, float* dB, float* work, long work_floats,
                              void* stream) {
  if (!ctx) return 2;
  ConvGeom g;
  if (int rc = geom_from(ctx, geom, g)) return rc;
  PSC_REQUIRE(ctx, act >= 0 && act <= 2 && (act == 0 || out), "conv3d_bwd: bad activation arguments");
  PSC_REQUIRE(ctx, A && W && gout && gm && dW && dB && work && (g.Cs == 0 || S), "conv3d_bwd: NULL pointer");
  cudaStream_t st = (cudaStream_t)stream;
  const auto* a = static_cast<const __nv_bfloat16*>(A);
  const auto* s = static_cast<const __nv_bfloat16*>(S);
  const auto* w = static_cast<const __nv_bfloat16*>(W);
  // output gradient through the activation, weight and bias gradients
  int rc = psc_conv_bwd_weights(ctx, g, a, s, gout, static_cast<const __nv_bfloat16*>(out), act, gm, dW, dB, work,
                                work_floats, st);
  if (rc || !dvin) return rc;
  // input gradient: straight into dA when it is A's alone and dA lies clear of
  // gm (which is still read), else through dvin and split into dA and dS
  const long nvi = (long)g.nxi * g.nyi * g.nzi, nvo = (long)g.nxo * g.nyo * g.nzo;
  const bool clear = dA && (dA + nvi * g.Ca <= gm || gm + nvo * g.Cout <= dA);
  if (!g.up && g.Cs == 0 && clear) return psc_conv_bwd_input(ctx, g, w, gm, dA, g.Ca, acc_a, st);
  rc = psc_conv_bwd_input(ctx, g, w, gm, dvin, g.Cin, 0, st);
  if (rc) return rc;
  if (dA) {
    k_split_grad_a<<<148 * 8, 256, 0, st>>>(dvin, g, acc_a, dA);
    PSC_LAUNCH_CHECK(ctx);
  }
  if (dS && g.Cs > 0) {
    k_split_grad_s<<<148 * 8, 256, 0, st>>>(dvin, g, acc_s, dS);
    PSC_LAUNCH_CHECK(ctx);
  }
  return 0;
}

extern "C" int psc_mse_loss(psc_ctx* ctx, const float* y, int C, const float* target, long n, float* grad,
                            double* loss_dev, void* stream) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, y && target && grad && loss_dev && n > 0 && C >= 1, "mse: bad arguments");
  cudaStream_t st = (cudaStream_t)stream;
  double* part = ctx->red_partial;
  k_mse<<<PSC_RED_BLOCKS, 256, 0, st>>>(y, C, target, n, grad, part);
  PSC_LAUNCH_CHECK(ctx);
  k_mse_final<<<1, 32, 0, st>>>(part, PSC_RED_BLOCKS, n, loss_dev);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

extern "C" int psc_adam_step(psc_ctx* ctx, float* w, void* wb, const float* grad, float* m, float* v, long n,
                             float lr, float b1, float b2, float eps, int step, void* stream) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, w && grad && m && v && n > 0 && step >= 1, "adam: bad arguments");
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  k_adam<<<psc_div_up(n, 256), 256, 0, (cudaStream_t)stream>>>(w, static_cast<__nv_bfloat16*>(wb), grad, m, v, n,
                                                               lr, b1, b2, eps, c1, c2);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

extern "C" int psc_f32_to_bf16(psc_ctx* ctx, const float* x, void* y, long n, void* stream) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, x && y && n >= 0, "f32_to_bf16: bad arguments");
  if (n == 0) return 0;
  k_f32_to_bf16<<<psc_div_up(n, 256), 256, 0, (cudaStream_t)stream>>>(x, static_cast<__nv_bfloat16*>(y), n);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

extern "C" int psc_pack_input(psc_ctx* ctx, const double* x0, const double* x1, double a0, double a1, void* out,
                              void* stream) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, x0 && x1 && out, "pack_input: NULL pointer");
  k_pack_input<<<148 * 8, 256, 0, (cudaStream_t)stream>>>(x0, x1, ctx->n, a0, a1, static_cast<__nv_bfloat16*>(out));
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}
