// Stencil step for grids whose planes the 16-byte bulk copies cannot address
// as they are (odd sides): Out = a (W In) + b In + g Prev, as in stencil.cu.
//
// The register-queue kernel of stencil.cu reads such grids with scalar loads
// that stall every plane (1.1 TB/s at 61 x 55 x 67, 31 FP64 columns).  Here a
// plane's window -- the CTA's 256 PPT consecutive xy points and R rows on each
// side -- is still one cp.async.bulk per plane into a ring of shared-memory
// slots: the copy starts at the 16-byte boundary at or below the window's
// first element and ends at the one at or above its last, and the plane's
// shift (its first element's position in that granule) is added to every
// shared-memory index.  What the rounding brings along lies outside the plane
// and is never used: x and y neighbours are selected by the point's distances
// to the edges, as in the register-queue kernel, whose order of arithmetic
// this kernel keeps.  A copy that would run past the block's last element is
// cut to the boundary below it and the remaining elements are stored by one
// thread before it arms the slot's barrier.
//
// H X at 61 x 55 x 67 with 31 columns: 124 -> 98 us, the step itself 101 -> 81.
// What is left is the chain of a plane's edge tests, loads and adds in 16 warps
// per SM and the unrolled loop's fetch: issue active 56 %, per issue 1.7 warps
// wait for a fixed latency and 1.1 for instructions, the shared-memory pipe is
// 43 % busy.
// Points of a thread are 256 apart, so shared-memory and global accesses of a
// warp are consecutive without any alignment.  Waits are bounded as in
// stencil_tma.cu (status word 3).
#include "psc_internal.cuh"
#include "../../include/psc.h"

#include <algorithm>
#include <cstdint>

namespace {
constexpr int BNT = 256;

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ bool try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, long limit) {
  for (long i = 0; i < limit; ++i)
    if (try_wait(bar, parity)) return true;
  return false;
}

template <typename T>
struct BulkArgs {
  const T* X;
  long ldx;
  const T* P;
  long ldp;
  T* Y;
  long ldy;
  const T* pot;
  int nx, ny, nz;
  long x_end;          // elements of X up to the end of the last column's grid
  const int4* sched;   // per CTA: column, slab, first plane, end plane
  T c0, c[4];
  const double* coef;
  double a, b, g;
  long wait_limit;
  int* status;
};
}  // namespace

template <typename T, int R, int PPT>
__global__ void __launch_bounds__(BNT, 2)
k_stencil_bulk(BulkArgs<T> A) {
  constexpr int S = BNT * PPT;
  constexpr int NBUF = R + 4;
  constexpr int Q = 2 * R + 1;
  constexpr int G = 16 / (int)sizeof(T);   // elements per 16-byte granule
  constexpr int SYNC = 2;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int nx = A.nx, ny = A.ny, nz = A.nz, nxy = nx * ny;
  const int H = R * nx;
  const int WS = (S + 2 * H + 4 * G) / G * G;
  T* ring = reinterpret_cast<T*>(smem_raw);                                // [NBUF][WS]
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + (size_t)NBUF * WS);  // [NBUF]
  __shared__ int s_fail;
  const int4 work = A.sched[blockIdx.x];
  const long col = work.x;
  const int slab0 = work.y * S, z0 = work.z, z1 = work.w;
  const int zlast = min(nz, z1 + R);
  const T* Xc = A.X + col * A.ldx;
  const T* Pc = A.P ? A.P + col * A.ldp : nullptr;
  T* Yc = A.Y + col * A.ldy;
  T a, b, g;
  if (A.coef) { a = (T)A.coef[0]; b = (T)A.coef[1]; g = (T)A.coef[2]; }
  else { a = (T)A.a; b = (T)A.b; g = (T)A.g; }

  const int w0 = slab0 - H;
  const int v0 = max(0, w0), v1 = min(nxy, slab0 + S + H);
  const int dst0 = (v0 - w0 + G - 1) / G * G;      // slot element of the copy's first granule
  const int lead = dst0 - (v0 - w0);               // window index w sits at slot[lead + shift + w]
  const int mis = (int)((col * A.ldx + v0) % G);   // shift of plane 0 (X itself is 16-byte aligned)
  const int mstep = nxy % G;
  auto shift_of = [&](int p) { return (mis + p * mstep) % G; };

  if (threadIdx.x == 0) {
    s_fail = 0;
    for (int i = 0; i < NBUF; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&bars[i])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  auto issue_x = [&](int p) {   // plane p into slot (p - z0) mod NBUF (thread 0)
    const int s = (p - z0) % NBUF;
    const int sh = shift_of(p);
    const long e0 = col * A.ldx + (long)p * nxy + v0 - sh;   // a multiple of G
    const int want = v1 - v0 + sh;                           // elements from e0
    int cnt = (want + G - 1) / G * G;
    T* dst = ring + (size_t)s * WS + dst0;
    if (e0 + cnt > A.x_end) {
      cnt = (int)((A.x_end - e0) / G * G);
      for (int i = cnt; i < want; ++i) dst[i] = A.X[e0 + i];
    }
    const uint32_t bytes = (uint32_t)(cnt * sizeof(T));
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&bars[s])), "r"(bytes)
                 : "memory");
    if (bytes)
      asm volatile(
          "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
              smem_u32(dst)),
          "l"(A.X + e0), "r"(bytes), "r"(smem_u32(&bars[s]))
          : "memory");
  };
  int issued = min(zlast, z0 + NBUF);
  if (threadIdx.x == 0)
    for (int p = z0; p < issued; ++p) issue_x(p);

  int q[PPT], xi[PPT], yi[PPT];
  bool own[PPT];
  T zq[PPT][Q];
#pragma unroll
  for (int v = 0; v < PPT; ++v) {
    q[v] = slab0 + threadIdx.x + BNT * v;
    own[v] = q[v] < nxy;
    xi[v] = own[v] ? q[v] % nx : 0;
    yi[v] = own[v] ? q[v] / nx : 0;
  }
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int zz = z0 - R + i;
#pragma unroll
    for (int v = 0; v < PPT; ++v) zq[v][i] = (own[v] && zz >= 0) ? Xc[(long)zz * nxy + q[v]] : T(0);
  }
  T np[PPT], nv[PPT];   // Prev and the potential of the next plane
  auto fetch = [&](int z) {
#pragma unroll
    for (int v = 0; v < PPT; ++v) {
      if (Pc) np[v] = own[v] ? Pc[(long)z * nxy + q[v]] : T(0);
      if (A.pot) nv[v] = own[v] ? A.pot[(long)z * nxy + q[v]] : T(0);
    }
  };
  fetch(z0);
  bool fail = false;
  int fail_plane = zlast;
  auto wait_plane = [&](int p) {
    if (!fail && !wait_for(&bars[(p - z0) % NBUF], ((p - z0) / NBUF) & 1, A.wait_limit)) {
      fail = true;
      fail_plane = p;
    }
  };
  auto at = [&](int p, int w) -> const T* {   // window index w of plane p
    return ring + (size_t)((p - z0) % NBUF) * WS + lead + shift_of(p) + w;
  };
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int p = z0 + i;
    if (p < nz) wait_plane(p);
#pragma unroll
    for (int v = 0; v < PPT; ++v) zq[v][R + i] = (p < nz && own[v]) ? *at(p, H + threadIdx.x + BNT * v) : T(0);
  }
#pragma unroll 1
  for (int zb = z0; zb < z1; zb += Q) {
#pragma unroll
    for (int u = 0; u < Q; ++u) {
      const int z = zb + u;
      if (z >= z1) break;
      const int pf = z + R;
      if (pf < nz) wait_plane(pf);
#pragma unroll
      for (int v = 0; v < PPT; ++v)
        zq[v][(u + 2 * R) % Q] = (pf < nz && own[v]) ? *at(pf, H + threadIdx.x + BNT * v) : T(0);
      T pv[PPT], vv[PPT];
#pragma unroll
      for (int v = 0; v < PPT; ++v) {
        pv[v] = np[v];
        vv[v] = nv[v];
      }
      if (z + 1 < z1) fetch(z + 1);
      const T* pl0 = at(z, H);
#pragma unroll
      for (int v = 0; v < PPT; ++v) {
        if (!own[v]) continue;
        const T* pl = pl0 + threadIdx.x + BNT * v;
        const T xc = zq[v][(u + R) % Q];
        T acc = A.c0 * xc;
#pragma unroll
        for (int d = 1; d <= R; ++d) {
          const T cd = A.c[d - 1];
          T sx = T(0), sy = T(0), sz = T(0);
          if (xi[v] - d >= 0) sx += pl[-d];
          if (xi[v] + d < nx) sx += pl[d];
          if (yi[v] - d >= 0) sy += pl[-d * nx];
          if (yi[v] + d < ny) sy += pl[d * nx];
          sz = zq[v][(u + R - d) % Q] + zq[v][(u + R + d) % Q];
          acc += cd * (sx + sy + sz);
        }
        if (A.pot) acc += vv[v] * xc;
        T out = a * acc + b * xc;
        if (Pc) out += g * pv[v];
        Yc[(long)z * nxy + q[v]] = out;
      }
      // every SYNC planes the slots of all planes <= z are free: the ring is
      // topped up to plane z + NBUF (the front z + R stays covered)
      if ((z - z0) % SYNC == SYNC - 1) {
        __syncthreads();
        if (threadIdx.x == 0 && !fail)
          for (; issued < zlast && issued <= z + NBUF; ++issued) issue_x(issued);
      }
    }
  }
  if (fail) s_fail = 1;
  // after a wait gave up: thread 0 drains the copies it issued (distinct slots)
  if (threadIdx.x == 0 && fail)
    for (int p = fail_plane; p < issued; ++p)
      wait_for(&bars[(p - z0) % NBUF], ((p - z0) / NBUF) & 1, PSC_DRAIN_WAIT);
  __syncthreads();
  if (threadIdx.x == 0 && s_fail) atomicExch(&A.status[3], 1);
}

// stencil_tma.cu: the cached work table of a launch shape
const int4* psc_stencil_sched(psc_ctx* ctx, int nslab, int k, int fill, int slots, int* n, cudaStream_t st);

template <typename T, int R>
static int launch_bulk(psc_ctx* ctx, const BulkArgs<T>& A0, int k, cudaStream_t st) {
  constexpr int PPT = 16 / (int)sizeof(T);   // 512 FP64 or 1024 FP32 points per CTA
  constexpr int G = 16 / (int)sizeof(T);
  BulkArgs<T> A = A0;
  const int S = BNT * PPT;
  const int nslab = (ctx->nx * ctx->ny + S - 1) / S;
  // The register-queue kernel keeps the calls too small to fill this one's
  // pipelines and the planes that leave a fifth of the slabs empty.  Measured
  // (us, register / bulk): FP64 45 x 47 x 49 at 4 columns 11.8 / 14.8, at 8 18.9 /
  // 16.9, at 64 142 / 84; 33 x 35 x 31 (slabs 75 % full) at 64 columns 36 / 47;
  // FP32 61 x 55 x 67 at 4 columns 15.7 / 19.0, at 8 25.3 / 23.0; 45 x 47 x 49 (69 %
  // full) at 64 columns 74 / 84.
  if (ctx->n * k < (sizeof(T) == 8 ? 800000 : 1800000) || 5L * ctx->nx * ctx->ny < 4L * nslab * S) return -1;
  const size_t ws = ((size_t)S + 2 * (size_t)R * ctx->nx + 4 * G) / G * G;
  const size_t smem = (R + 4) * ws * sizeof(T) + (R + 4) * sizeof(uint64_t);
  if (smem > 110 * 1024) return -1;   // two CTAs per SM, or the register-queue kernel
  int sms = 148, nwork = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  A.sched = psc_stencil_sched(ctx, nslab, k, R + 6, 2 * sms, &nwork, st);
  if (nwork == 0) return -1;   // no table yet, and none to be had during a stream capture
  PSC_REQUIRE(ctx, A.sched != nullptr, "stencil: work table allocation failed");
  auto kern = k_stencil_bulk<T, R, PPT>;
  PSC_CUDA(ctx, psc_smem_optin(kern));
  kern<<<nwork, BNT, smem, st>>>(A);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

// -1 if the path does not apply (X must start on a 16-byte boundary, so that
// no copy reaches below it, and the windows must fit)
template <typename T>
int psc_stencil_bulk(psc_ctx* ctx, int k, const T* X, long ldx, const T* P, long ldp, T* Y, long ldy, const T* pot,
                     const double* w, const double* coef, double a, double b, double g, cudaStream_t st) {
  if (reinterpret_cast<uintptr_t>(X) % 16) return -1;
  BulkArgs<T> A;
  A.X = X; A.ldx = ldx; A.P = P; A.ldp = ldp; A.Y = Y; A.ldy = ldy; A.pot = pot;
  A.nx = ctx->nx; A.ny = ctx->ny; A.nz = ctx->nz;
  A.x_end = (long)(k - 1) * ldx + ctx->n;
  A.sched = nullptr;
  A.c0 = (T)w[0];
  for (int i = 0; i < 4; ++i) A.c[i] = (T)w[1 + i];
  A.coef = coef; A.a = a; A.b = b; A.g = g;
  A.wait_limit = ctx->wait_limit;
  A.status = ctx->dev_status;
  switch (ctx->radius) {
    case 1: return launch_bulk<T, 1>(ctx, A, k, st);
    case 2: return launch_bulk<T, 2>(ctx, A, k, st);
    case 3: return launch_bulk<T, 3>(ctx, A, k, st);
    default: return launch_bulk<T, 4>(ctx, A, k, st);
  }
}

template int psc_stencil_bulk<double>(psc_ctx*, int, const double*, long, const double*, long, double*, long,
                                      const double*, const double*, const double*, double, double, double,
                                      cudaStream_t);
template int psc_stencil_bulk<float>(psc_ctx*, int, const float*, long, const float*, long, float*, long,
                                     const float*, const double*, const double*, double, double, double, cudaStream_t);
