// Multisecant Type-I potential mixing with group size 1 (Broyden's first
// method): Mixer/msecant1.py:40-175 with the parameters of
// Mixer/includemix.py:21-49 (mix 0.5, restart factor 0.1, EN_like 0).
//
// The secant history DX, DF (one n-vector per SCF iteration) stays in HBM.
// A call reads the history twice: once for the 3(m-1) dot products
// DF_i.df, DF_i.f1, DX_i.dx and once to form the new DX column, the new
// iterate and the group vector N.  The 1x1 quasi-inverse of
// Mixer/qinv.py:5-62 is 1/M (0 when M == 0).
#include "psc_internal.cuh"
#include "../../include/psc.h"

#include <algorithm>
#include <cmath>

__global__ void k_mix_first(const double* __restrict__ x1, const double* __restrict__ f1, double mix, long n,
                            double* __restrict__ dx0, double* __restrict__ df0, double* __restrict__ xn) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double x = x1[i], f = f1[i];
    dx0[i] = x;
    df0[i] = f;
    xn[i] = x + mix * f;
  }
}

__global__ void k_mix_restart(const double* __restrict__ xl, const double* __restrict__ fl, double mix, long n,
                              double* __restrict__ dx0, double* __restrict__ df0, double* __restrict__ xn) {
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double x = xl[i], f = fl[i];
    xn[i] = x + mix * f;
    dx0[i] = x;
    df0[i] = f;
  }
}

// dx = x1 - DX[m-1], df = f1 - DF[m-1], and |f1|^2 for the restart test (the
// last CTA sums the partials).  DF[m-1] itself is left alone: a restart reads
// it, and k_mix_final overwrites it otherwise.
__global__ void __launch_bounds__(256)
k_mix_diff(const double* __restrict__ x1, const double* __restrict__ f1, const double* __restrict__ dxl,
           const double* __restrict__ dfl, double* __restrict__ dx, double* __restrict__ df, long n,
           double* __restrict__ part, unsigned int* ticket, double* __restrict__ fnorm2) {
  __shared__ double sh[8];
  double s = 0.0;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const double f = f1[i];
    dx[i] = x1[i] - dxl[i];
    df[i] = f - dfl[i];
    s += f * f;
  }
  s = psc_block_sum<double, 256>(s, sh);
  if (threadIdx.x == 0) part[blockIdx.x] = s;
  if (!psc_last_block(ticket)) return;
  if (threadIdx.x < 32) {
    s = psc_warp_partials(part, gridDim.x);
    if (threadIdx.x == 0) *fnorm2 = s;
  }
}

// a_i = DF_i.df, b_i = DF_i.f1, c_i = DX_i.dx for i < mm.  A CTA takes a
// contiguous range of points (df, f1 and dx of it stay in L1 over the
// columns) and MD_G columns at a time, so that their loads are in flight
// together and one pair of barriers serves all 3 MD_G sums; the last CTA sums
// the partials, one warp per quantity.
constexpr int MD_NT = 512, MD_G = 4;
__global__ void __launch_bounds__(MD_NT)
k_mix_dots(const double* __restrict__ DX, const double* __restrict__ DF, const double* __restrict__ df,
           const double* __restrict__ f1, const double* __restrict__ dx, long n, int mm, double* __restrict__ part,
           unsigned int* ticket, double* __restrict__ coef) {
  __shared__ double sh[3 * MD_G * MD_NT / 32];
  const long chunk = (n + gridDim.x - 1) / gridDim.x;
  const long lo = chunk * blockIdx.x, hi = min(n, lo + chunk);
  for (int i0 = 0; i0 < mm; i0 += MD_G) {
    double v[3 * MD_G];
#pragma unroll
    for (int q = 0; q < 3 * MD_G; ++q) v[q] = 0.0;
    for (long p = lo + threadIdx.x; p < hi; p += MD_NT) {
      const double a = df[p], b = f1[p], c = dx[p];
#pragma unroll
      for (int g = 0; g < MD_G; ++g) {
        if (i0 + g >= mm) break;
        const double u = DF[(long)(i0 + g) * n + p];
        v[3 * g] += u * a;
        v[3 * g + 1] += u * b;
        v[3 * g + 2] += DX[(long)(i0 + g) * n + p] * c;
      }
    }
    psc_block_sums<MD_NT, 3 * MD_G>(v, sh);
    if (threadIdx.x == 0)
#pragma unroll
      for (int q = 0; q < 3 * MD_G; ++q)
        if (i0 + q / 3 < mm) part[(long)(3 * i0 + q) * PSC_RED_BLOCKS + blockIdx.x] = v[q];
  }
  if (!psc_last_block(ticket)) return;
  for (int s = threadIdx.x >> 5; s < 3 * mm; s += MD_NT / 32) {
    const double t = psc_warp_partials(part + (long)s * PSC_RED_BLOCKS, gridDim.x);
    if ((threadIdx.x & 31) == 0) coef[s] = t;
  }
}

// DX[m-1] = dx + mix df - sum DX_i a_i ; xn = x1 + mix f1 - sum DX_i b_i ;
// N = -mix dx + sum DF_i c_i ; s = [N.df, N.f1]
__global__ void __launch_bounds__(256)
k_mix_combine(double* __restrict__ DX, const double* __restrict__ DF, const double* __restrict__ x1,
              const double* __restrict__ f1, const double* __restrict__ dx, const double* __restrict__ df, long n,
              int m, double mix, const double* __restrict__ coef, double* __restrict__ xn, double* __restrict__ nv,
              double* __restrict__ part, unsigned int* ticket, double* __restrict__ s) {
  __shared__ double sh[2 * 8];
  __shared__ double cf[3 * 256];
  const int mm = m - 1;
  for (int i = threadIdx.x; i < 3 * mm; i += 256) cf[i] = coef[i];
  __syncthreads();
  double* dxl = DX + (long)mm * n;
  double v[2] = {0.0, 0.0};
  for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < n; p += (long)gridDim.x * blockDim.x) {
    const double dxp = dx[p], dfp = df[p], f = f1[p];
    double d = dxp + mix * dfp;
    double x = x1[p] + mix * f;
    double nn = -mix * dxp;
#pragma unroll 4
    for (int i = 0; i < mm; ++i) {
      const double hx = __ldcg(DX + (long)i * n + p);
      const double hf = __ldcg(DF + (long)i * n + p);
      d -= hx * cf[3 * i + 0];
      x -= hx * cf[3 * i + 1];
      nn += hf * cf[3 * i + 2];
    }
    dxl[p] = d;
    xn[p] = x;
    nv[p] = nn;
    v[0] += nn * dfp;
    v[1] += nn * f;
  }
  psc_block_sums<256, 2>(v, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v[0];
    part[PSC_RED_BLOCKS + blockIdx.x] = v[1];
  }
  if (!psc_last_block(ticket)) return;
  if (threadIdx.x < 64) {
    const int w = threadIdx.x >> 5;
    const double t = psc_warp_partials(part + (long)w * PSC_RED_BLOCKS, gridDim.x);
    if ((threadIdx.x & 31) == 0) s[w] = t;
  }
}

// C = qinv([M]) = 1/M (0 when M == 0); DF[m-1] = N C; xn -= DX[m-1] * (C * N.f1);
// append DX[m] = x1, DF[m] = f1
__global__ void k_mix_final(double* __restrict__ DX, double* __restrict__ DF, const double* __restrict__ x1,
                            const double* __restrict__ f1, const double* __restrict__ nv, long n, int m,
                            const double* __restrict__ s /* [M, N.f1] */, double* __restrict__ xn) {
  const double M = s[0];
  const double C = (M != 0.0) ? 1.0 / M : 0.0;
  const double g = C * s[1];
  double* dfl = DF + (long)(m - 1) * n;
  const double* dxl = DX + (long)(m - 1) * n;
  double* dxa = DX + (long)m * n;
  double* dfa = DF + (long)m * n;
  for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < n; p += (long)gridDim.x * blockDim.x) {
    dfl[p] = nv[p] * C;
    xn[p] -= dxl[p] * g;
    dxa[p] = x1[p];
    dfa[p] = f1[p];
  }
}

extern "C" int psc_mixer_reset(psc_ctx* ctx, int capacity) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, capacity >= 1 && capacity <= 255, "mixer: capacity must be 1..255");
  if (capacity > ctx->mix_cap) {
    psc_dfree(ctx->mix_dx); psc_dfree(ctx->mix_df); psc_dfree(ctx->mix_nv); psc_dfree(ctx->mix_tmp);
    psc_dfree(ctx->mix_ddf);
    psc_dfree(ctx->mix_coef); psc_dfree(ctx->mix_partial);
    ctx->mix_dx = ctx->mix_df = ctx->mix_nv = ctx->mix_tmp = ctx->mix_ddf = ctx->mix_coef = ctx->mix_partial =
        nullptr;
    const size_t n = ctx->n;
    PSC_CUDA(ctx, psc_dmalloc(&ctx->mix_dx, (size_t)(capacity + 1) * n * sizeof(double)));
    PSC_CUDA(ctx, psc_dmalloc(&ctx->mix_df, (size_t)(capacity + 1) * n * sizeof(double)));
    PSC_CUDA(ctx, psc_dmalloc(&ctx->mix_nv, n * sizeof(double)));
    PSC_CUDA(ctx, psc_dmalloc(&ctx->mix_tmp, n * sizeof(double)));
    PSC_CUDA(ctx, psc_dmalloc(&ctx->mix_ddf, n * sizeof(double)));
    PSC_CUDA(ctx, psc_dmalloc(&ctx->mix_coef, (3 * (size_t)capacity + 8) * sizeof(double)));
    PSC_CUDA(ctx, psc_dmalloc(&ctx->mix_partial, (3 * (size_t)capacity + 2) * PSC_RED_BLOCKS * sizeof(double)));
    ctx->mix_cap = capacity;
  }
  ctx->mix_m = 0;
  ctx->mix_slot = 0;
  return 0;
}

// x_new = mixer(x1, f1).  *m_used receives the number of secant equations
// (0 for the first call and after a restart), as Mixer/mixer.py:189-217.
extern "C" int psc_mixer_step(psc_ctx* ctx, const double* x1, const double* f1, double mix, double restart_factor,
                              double* x_new, int* m_used, void* stream) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, ctx->mix_cap > 0, "mixer: call psc_mixer_reset first");
  PSC_REQUIRE(ctx, x_new != x1 && x_new != f1, "mixer: output must not alias the inputs");
  cudaStream_t st = (cudaStream_t)stream;
  // the step's host state (history length, restart decision) cannot be replayed
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  PSC_CUDA(ctx, cudaStreamIsCapturing(st, &cap));
  PSC_REQUIRE(ctx, cap == cudaStreamCaptureStatusNone, "mixer: not available during stream capture");
  const long n = ctx->n;
  const int nb = (int)std::max<long>(1, std::min<long>(PSC_RED_BLOCKS, (n + 255) / 256));
  const int m = ctx->mix_m;
  // |f|^2 of the last accepted call sits in fn[mix_slot], this call's goes to
  // the other slot; the host reads them only when a restart is possible
  double* fn = ctx->scalars + 120;
  const int cur = ctx->mix_slot ^ 1;
  if (m == 0) {
    // (the first call's norm is never compared: a restart needs m >= 2)
    k_mix_first<<<nb, 256, 0, st>>>(x1, f1, mix, n, ctx->mix_dx, ctx->mix_df, x_new);
    PSC_LAUNCH_CHECK(ctx);
    ctx->mix_m = 1;
    if (m_used) *m_used = 0;
    return 0;
  }
  double* dxl = ctx->mix_dx + (long)(m - 1) * n;
  double* dfl = ctx->mix_df + (long)(m - 1) * n;
  k_mix_diff<<<nb, 256, 0, st>>>(x1, f1, dxl, dfl, ctx->mix_tmp, ctx->mix_ddf, n, ctx->mix_partial, psc_ticket(ctx),
                                 fn + cur);
  PSC_LAUNCH_CHECK(ctx);
  const int mm = m - 1;
  if (mm > 0) {
    // the history's dot products run while the host waits for the two norms
    // (they change nothing a restart reads)
    if (!ctx->mix_ev) PSC_CUDA(ctx, cudaEventCreateWithFlags(&ctx->mix_ev, cudaEventDisableTiming));
    PSC_CUDA(ctx, cudaMemcpyAsync(ctx->host_scalars + 120, fn, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
    PSC_CUDA(ctx, cudaEventRecord(ctx->mix_ev, st));
    const int nbd = (int)std::max<long>(1, std::min<long>(148, (n + MD_NT - 1) / MD_NT));
    k_mix_dots<<<nbd, MD_NT, 0, st>>>(ctx->mix_dx, ctx->mix_df, ctx->mix_ddf, f1, ctx->mix_tmp, n, mm,
                                      ctx->mix_partial, psc_ticket(ctx), ctx->mix_coef);
    PSC_LAUNCH_CHECK(ctx);
    PSC_CUDA(ctx, cudaEventSynchronize(ctx->mix_ev));
    const double fnorm = std::sqrt(ctx->host_scalars[120 + cur]);
    const double last = std::sqrt(ctx->host_scalars[120 + ctx->mix_slot]);
    if (last < restart_factor * fnorm) {
      k_mix_restart<<<nb, 256, 0, st>>>(dxl, dfl, mix, n, ctx->mix_dx, ctx->mix_df, x_new);
      PSC_LAUNCH_CHECK(ctx);
      ctx->mix_m = 1;
      if (m_used) *m_used = 0;
      return 0;
    }
  }
  PSC_REQUIRE(ctx, m + 1 <= ctx->mix_cap, "mixer: history capacity exceeded (raise it at reset)");
  double* sv = ctx->mix_coef + 3 * ctx->mix_cap;
  k_mix_combine<<<nb, 256, 0, st>>>(ctx->mix_dx, ctx->mix_df, x1, f1, ctx->mix_tmp, ctx->mix_ddf, n, m, mix,
                                    ctx->mix_coef, x_new, ctx->mix_nv, ctx->mix_partial, psc_ticket(ctx), sv);
  PSC_LAUNCH_CHECK(ctx);
  k_mix_final<<<nb, 256, 0, st>>>(ctx->mix_dx, ctx->mix_df, x1, f1, ctx->mix_nv, n, m, sv, x_new);
  PSC_LAUNCH_CHECK(ctx);
  ctx->mix_m = m + 1;
  ctx->mix_slot = cur;
  if (m_used) *m_used = m;
  return 0;
}

extern "C" int psc_mixer_history(psc_ctx* ctx, int* m_out) {
  if (!ctx) return 2;
  if (m_out) *m_out = ctx->mix_m;
  return 0;
}
