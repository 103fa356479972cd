// TMA-fed stencil pipeline (sm_100a): the fused Chebyshev / H.X step
//   Out = a * (W In) + b * In + g * Prev,  W = c0 + sum_d c_d (shifts) [+ diag(pot)]
// with plane windows streamed into shared memory by 1-D bulk copies.
//
// A CTA owns S = 512 (FP64) or 1024 (FP32) consecutive flat xy points of one
// column and a chunk of z planes.  For every plane the points it needs -- its
// own S points plus R rows of y halo on each side -- are one contiguous range
// of the plane, so a single cp.async.bulk (no tensor map, no multicast) moves
// it into a slot of a ring of NBUF shared-memory windows, completing on the
// slot's mbarrier.  Each slot ends with one zero vector.
// The z neighbours of each point live in a register queue fed from the ring;
// x and y neighbours are read from the current plane's window with 16-byte
// loads (each thread owns a run of 2 FP64 or 4 FP32 points).  When the run
// cannot cross a row edge (2 | nx for FP64, 4 | nx for FP32) the x vectors
// outside the row are read from the zero vector, so the x terms need no
// per-point masks; otherwise each point masks its x neighbours by its
// distances to the row edges.
//
// The kernel is bound by instruction issue before it is bound by HBM (the
// FP32 step at 90^3, k = 307 moved 58 % of the copy rate at 62 % issue
// active with 320 instructions per thread and plane, half of them moves,
// selects and integer work), so everything around the 24 neighbour sums is
// made to cost nothing inside the z loop:
//   - the loop is unrolled by the queue length 2R + 1, so the queue rotates
//     by renaming; ring offsets, barrier addresses and parities run along and
//     wrap instead of being recomputed from the plane's number (opaque to the
//     compiler, which otherwise keeps every sum of the unrolled pass in
//     spilled registers);
//   - whether Prev and the potential exist is a template argument, and the
//     sphere mask of a point is an interval of planes found once;
//   - x sums at odd distances are scalar adds: a packed add would first have
//     to move both operands into aligned register pairs.
// Prev and pot are copied three planes ahead by per-thread 16-byte cp.async
// into a small ring that each thread reads back itself.  (Loading them, or
// only the potential, two planes ahead into registers instead saves a few
// instructions more and loses it all: 1.5 to 7.6 warps stalled on the loads
// per issue.  Under full HBM load two planes are not early enough.)
// With this a step at 90^3, k = 307 takes 635 us in FP32 and 1204 in FP64 (709
// and 1346 before; under the power cap of a long run FP64 takes 1265, 1358
// before), and 34.5 instead of 40.6 us at 52^3, k = 27.  The limit now is the
// shared-memory pipe, busy 77 % of the cycles: 24 neighbours of which the x and y
// ones are loads.  (Giving a thread several rows, so that most y neighbours are
// its own registers, cut the wavefronts by a fifth and was still slower: 1275 us
// in FP64, with 12 warps per SM instead of 16 and twice the unrolled code.)
// The order of the arithmetic of a point is fixed (shells from d = R down to
// 1 for FP32), whatever the path.
//
// Every mbarrier wait is bounded by the context's wait limit: on timeout the
// CTA records the failure in status[3], stops issuing copies and carries on
// without waiting (results are then garbage but the GPU is never hung).
// Every bulk copy issued is waited for before the CTA exits.
#include "psc_internal.cuh"
#include "../../include/psc.h"

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <type_traits>
#include <vector>

namespace {

#ifndef PSC_STENCIL_THREADS
#define PSC_STENCIL_THREADS 256
#endif
constexpr int TNT = PSC_STENCIL_THREADS;  // threads per CTA
#ifndef PSC_STENCIL_CTAS_PER_SM
#define PSC_STENCIL_CTAS_PER_SM 2   // resident CTAs per SM (registers and shared memory)
#endif
// Planes between block barriers.  At 90^3, k = 307: 651 / 635 / 714 us per FP32
// step for 2 / 3 / 4 (the ring runs dry), FP64 1203 / 1204 / 1303.
constexpr int SYNC_EVERY = 3;
// Planes of X in flight beyond the one consumed next (a template argument: the
// ring's length as a variable cost 2.5 % in FP32): 3, the least that SYNC_EVERY
// allows, or 5 for FP32 where that leaves room for two CTAs per SM (5 against 3
// planes: 635 against 657 us at 90^3, 194 against 197 at 74^3; FP64 at 90^3 has
// room for 3, and 2 cost 8 %).
constexpr int AHEAD = SYNC_EVERY, AHEAD_F32 = 5;
constexpr size_t SMEM_HALF = 113 * 1024;   // shared memory of one of two resident CTAs
constexpr int PP_SLOTS = 4;   // Prev and pot: the plane in use + three in flight

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// bounded wait; returns false on timeout
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, long limit) {
  for (long i = 0; i < limit; ++i)
    if (mbar_try_wait(bar, parity)) return true;
  return false;
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
          smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}

// Points per thread: 16-byte vectors (two FP64 or four FP32 points), or
// 8-byte vectors of two FP32 points when nx is only even (the runs then never
// cross a row, so the x terms need no per-point masks).
template <typename T, int VW>
struct VecOf;
template <>
struct VecOf<double, 2> {
  using type = double2;
};
template <>
struct VecOf<float, 4> {
  using type = float4;
};
template <>
struct VecOf<float, 2> {
  using type = float2;
};

template <int VW, typename T>
__device__ __forceinline__ void vload(const T* p, T* out) {
  using V = typename VecOf<T, VW>::type;
  const V v = *reinterpret_cast<const V*>(p);
  const T* e = reinterpret_cast<const T*>(&v);
#pragma unroll
  for (int j = 0; j < VW; ++j) out[j] = e[j];
}

template <int VW, typename T>
__device__ __forceinline__ void vstore(T* p, const T* in) {
  using V = typename VecOf<T, VW>::type;
  V v;
  T* e = reinterpret_cast<T*>(&v);
#pragma unroll
  for (int j = 0; j < VW; ++j) e[j] = in[j];
  *reinterpret_cast<V*>(p) = v;
}

// load VW consecutive values from an address aligned to A elements (A | VW)
template <typename T, int A, int VW>
__device__ __forceinline__ void vload_a(const T* p, T* out) {
  if constexpr (A == VW) {
    vload<VW>(p, out);
  } else if constexpr (A == 2) {
    using V2 = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
#pragma unroll
    for (int h = 0; h < VW / 2; ++h) {
      const V2 v = *reinterpret_cast<const V2*>(p + 2 * h);
      out[2 * h] = v.x;
      out[2 * h + 1] = v.y;
    }
  } else {
#pragma unroll
    for (int j = 0; j < VW; ++j) out[j] = p[j];
  }
}

// The y row at distance d from the run: the window offset of the run is a
// multiple of VW plus R nx, and R nx is a multiple of VW (a condition of the
// TMA path), so the row starts d nx away from a VW-aligned spot and is
// aligned to min(VW, YA 2^v) elements, 2^v the power of two in d (YA holds
// nx's).  d is a constant after unrolling, so the choice folds away.
template <typename T, int YA, int VW>
__device__ __forceinline__ void vload_row(const T* p, int d, T* out) {
  int a = YA;
  while (a < VW && (d & 1) == 0) {
    a *= 2;
    d >>= 1;
  }
  if (a >= VW)
    vload<VW>(p, out);
  else if (a >= 2)
    vload_a<T, 2, VW>(p, out);
  else
    vload_a<T, 1, VW>(p, out);
}

// per-thread asynchronous copy of one run (VW points) into shared memory
template <int BYTES>
__device__ __forceinline__ void cp_async_run(void* dst, const void* src) {
  if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

template <int VW>
__host__ __device__ constexpr int slab_points() {
  return VW * TNT;
}

template <typename T>
struct TmaArgs {
  const T* X;
  long ldx;
  const T* P;
  long ldp;
  T* Y;
  long ldy;
  const T* pot;
  int nx, ny, nz;
  const int4* sched;  // per CTA: column, slab, first plane, end plane
  T c0, c[4];
  T csr;              // FP32 weights: minus their sum-rule residual, (c0 + 6 sum_d c_d) in FP32 - in FP64
  const double* coef;
  double a, b, g;
  long wait_limit;    // polls of each mbarrier wait before the CTA gives up
  // sphere mask: outputs at points with (i h - cx)^2 + (j h - cy)^2 +
  // (l h - cz)^2 > mask_r2 are zero (mask_r2 = 0: the whole cube)
  double mask_r2, h, cx, cy, cz;
  int* status;
};

}  // namespace

// YA: alignment (in elements) of the y-neighbour rows, the largest of VW, 2, 1
// that divides nx; their loads are split to match.  PK (FP32): the arithmetic
// on packed pairs of points.  HASP / HASV: Prev / the potential exist.
// csr != 0 (FP32): sum-rule correction: with the weights rounded to FP32 the
// sum rule c0 + 6 sum_d c_d = 0 fails by their rounding errors (-6.1e-8 Ha at
// h = 0.47 bohr), a constant shift of every eigenvalue that the band energy
// multiplies by the electron count; one more term, -(that residual) x,
// removes it.  (Applying every weight as its FP32 value plus its rounding
// error moved the Rayleigh quotients of smooth fields by no more than this one
// term does.)
template <typename T, int R, int YA, int VW, bool PK, bool HASP, bool HASV, int DEEP>
__global__ void __launch_bounds__(TNT, PSC_STENCIL_CTAS_PER_SM)
k_stencil_tma(TmaArgs<T> A) {
  static_assert(!PK || (sizeof(T) == 4 && VW % 2 == 0), "packed pairs need FP32 runs of an even length");
  constexpr int TS = slab_points<VW>();    // points per slab (VW per thread)
  constexpr int NBUF = R + 1 + DEEP;       // X plane windows resident
  constexpr int Q = 2 * R + 1;             // z queue length, planes per unrolled pass
  static_assert(SYNC_EVERY <= DEEP, "barrier interval exceeds the ring");
  constexpr int NPP = (HASP ? 1 : 0) + (HASV ? 1 : 0);
  static_assert((TS & (TS - 1)) == 0 && (PP_SLOTS & (PP_SLOTS - 1)) == 0, "the Prev/pot ring wraps by masking");
  constexpr int HV = (R + VW - 1) / VW;    // x-halo vectors on each side
  constexpr int NPV = 2 * HV + 1;          // x vectors per row (the centre one comes from the queue)
  constexpr int OFF = HV * VW;             // xs index of the thread's first point
  extern __shared__ __align__(128) unsigned char smem_raw[];
  const int nx = A.nx, ny = A.ny, nz = A.nz;
  const int nxy = nx * ny;
  const int H = R * nx;
  const int WIN = TS + 2 * H;
  // slot stride: the window and one zero vector, rounded up to 16 bytes so
  // that every slot starts where a bulk copy may write
  constexpr int Q16 = 16 / (int)sizeof(T);
  const int WS = (WIN + VW + Q16 - 1) / Q16 * Q16;
  T* ring = reinterpret_cast<T*>(smem_raw);                          // [NBUF][WS]
  T* pring = ring + (size_t)NBUF * WS;                               // [PP_SLOTS][NPP][TS]: Prev, pot
  uint64_t* bars = reinterpret_cast<uint64_t*>(pring + PP_SLOTS * NPP * TS);  // [NBUF]
  __shared__ int s_fail;

  const int4 work = A.sched[blockIdx.x];
  const int slab0 = work.y * TS;
  const int z0 = work.z;
  const int z1 = work.w;
  if (work.x < 0) {
    // sphere mask: planes of this slab that hold no point inside the sphere;
    // the output is zero there and nothing is read
    const int loc0 = VW * threadIdx.x;
    if (loc0 < min(TS, nxy - slab0)) {
      T zv[VW];
#pragma unroll
      for (int j = 0; j < VW; ++j) zv[j] = T(0);
      T* Yz = A.Y + (long)(-1 - work.x) * A.ldy + slab0 + loc0;
      for (int z = z0; z < z1; ++z) vstore<VW>(Yz + (long)z * nxy, zv);
    }
    return;
  }
  const int zlast = min(nz, z1 + R);  // X planes needed: [z0 - R, z1 + R) within [0, nz)
  const long col = work.x;
  const T* Xc = A.X + col * A.ldx;
  const T* Pc = HASP ? A.P + col * A.ldp : nullptr;
  T* Yc = A.Y + col * A.ldy;

  T ca, cb, cg;
  if (A.coef) { ca = (T)A.coef[0]; cb = (T)A.coef[1]; cg = (T)A.coef[2]; }
  else { ca = (T)A.a; cb = (T)A.b; cg = (T)A.g; }

  // valid part of the window within the plane
  const int w0 = slab0 - H;
  const int v0 = max(0, w0), v1 = min(nxy, slab0 + TS + H);
  const uint32_t xbytes = (uint32_t)((v1 - v0) * sizeof(T));
  const int seff = min(TS, nxy - slab0);

  // zero the parts of every window that lie outside the plane and the pad
  // vector after it (neither is ever written by the copies)
  for (int s = 0; s < NBUF; ++s) {
    T* w = ring + (size_t)s * WS;
    for (int i = threadIdx.x; i < WS; i += TNT) {
      const int f = w0 + i;
      if (i >= WIN || f < v0 || f >= v1) w[i] = T(0);
    }
  }
  if (threadIdx.x == 0) {
    s_fail = 0;
    for (int i = 0; i < NBUF; ++i) mbar_init(&bars[i], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  __syncthreads();

  auto issue_x = [&](int p, int s) {  // plane p into slot s = (p - z0) mod NBUF; only z0 <= p < zlast
    uint64_t* bar = &bars[s];
    mbar_expect_tx(bar, xbytes);
    bulk_g2s(ring + (size_t)s * WS + (v0 - w0), Xc + (long)p * nxy + v0, xbytes, bar);
  };
  int issued = min(zlast, z0 + NBUF);  // next plane to copy (thread 0's count)
  if (threadIdx.x == 0) {
    for (int p = z0; p < issued; ++p) issue_x(p, p - z0);
  }

  // own run of VW points (it may cross a row boundary: every point has its own x)
  const int loc = VW * threadIdx.x;
  const bool own = loc < seff;
  const int q = slab0 + loc;
  const int s_c = H + loc;  // window offset of the run

  // Prev and pot of the run, PP_SLOTS - 1 planes ahead: each thread copies its
  // own run into slot (z - z0) mod PP_SLOTS and reads it back itself, so no
  // block-wide handshake is needed.  One commit group per plane (empty ones
  // too), so "at most PP_SLOTS - 1 groups pending" means plane z has landed.
  // (P may alias Y: plane z of P is read before this thread stores plane z of
  // Y.)
  constexpr int PSTEP = NPP * TS;
  auto copy_pp = [&](bool in, int slot, int e) {   // element e of the column into the slot's elements
    if (in) {
      if constexpr (HASP) cp_async_run<VW * sizeof(T)>(pring + slot + loc, Pc + e);
      if constexpr (HASV) cp_async_run<VW * sizeof(T)>(pring + slot + (HASP ? TS : 0) + loc, A.pot + e);
    }
    cp_async_commit();
  };
  if constexpr (NPP > 0)
    for (int i = 0; i < PP_SLOTS - 1; ++i) copy_pp(own && z0 + i < z1, i * PSTEP, (z0 + i) * nxy + q);

  // z queue: planes below the chunk from global memory, z0 .. z0+R-1 from the ring
  T zq[VW][Q];
#pragma unroll
  for (int i = 0; i < 2 * R; ++i) {
    const int zz = z0 - R + i;
#pragma unroll
    for (int j = 0; j < VW; ++j) zq[j][i] = T(0);
    if (zz < z0 && own && zz >= 0) {
      T v[VW];
      vload<VW>(Xc + (long)zz * nxy + q, v);
#pragma unroll
      for (int j = 0; j < VW; ++j) zq[j][i] = v[j];
    }
  }
  // A limit of 0 polls gives up at once.  The first poll is the whole cost of
  // a plane that has landed; the counted loop runs only when it has not.
  bool fail = A.wait_limit <= 0;
  int fail_plane = fail ? z0 : zlast;   // first plane whose wait this thread gave up on
  auto wait_plane = [&](int p, uint64_t* bar, uint32_t parity) {
    if (fail || mbar_try_wait(bar, parity)) return;
    if (!mbar_wait(bar, parity, A.wait_limit)) {
      fail = true;
      fail_plane = p;
    }
  };
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int p = z0 + i;
    if (p < nz) {
      wait_plane(p, &bars[i], 0u);
      if (own) {
        T v[VW];
        vload<VW>(ring + (size_t)i * WS + s_c, v);
#pragma unroll
        for (int j = 0; j < VW; ++j) zq[j][R + i] = v[j];
      }
    }
  }

  // When VW divides nx, a thread's run lies in one row and every aligned
  // x vector around it is either wholly in that row or wholly outside it:
  // the outside ones are read from the slot's zero pad, so the x terms need
  // no per-point masks.  Otherwise (FP32 runs crossing a row edge) each point
  // keeps its distances to the row edges, capped at R: a neighbour d > el
  // (left) or d > er (right) lies across the edge and gets weight 0.
  constexpr bool EXACT = (YA == VW);
  int xo[NPV];
#pragma unroll
  for (int v = 0; v < NPV; ++v) {
    const int xv = (own ? q % nx : 0) - OFF + v * VW;  // first x of vector v
    xo[v] = (xv >= 0 && xv + VW <= nx) ? s_c - OFF + v * VW : WIN;
  }
  int el[VW], er[VW];
#pragma unroll
  for (int j = 0; j < VW; ++j) {
    const int xj = own ? (q + j) % nx : 0;
    el[j] = min(R, xj);
    er[j] = min(R, nx - 1 - xj);
  }
  // Pair masks (FP32 4-point runs with packed arithmetic, nx = 2 mod 4):
  // the run's 12-value x window is six aligned pairs, none of which crosses
  // a row (nx is even), and the run itself splits into two pairs, A (points
  // 0, 1) and B (points 2, 3), each in one row.  A window pair is a valid x
  // neighbour of A's points iff it lies in A's row, likewise for B, so the
  // edge masks are twelve loop-invariant 0/1 factors (instead of a compare
  // and a select per point and distance in every plane).  mA[p], mB[p]:
  // pair p of the window (flat q - 4 + 2p) for owner A, B.
  constexpr bool PAIRM = (YA != VW) && PK && VW == 4 && YA == 2 && R <= 4;
  float mA[6], mB[6];
  if constexpr (PAIRM) {
    const int x0 = own ? q % nx : 0;
    const bool b_next = x0 + 2 > nx - 2;   // B starts the next row
#pragma unroll
    for (int p = 0; p < 6; ++p) {
      const int xp = x0 - 4 + 2 * p;       // x of the pair's first point, in A's row coordinates
      mA[p] = (xp >= 0 && xp <= nx - 2) ? 1.f : 0.f;
      mB[p] = b_next ? (xp >= nx ? 1.f : 0.f) : mA[p];
    }
  }
  // sphere mask: plane z of point j is inside iff zin[j] = lo | hi << 16 has
  // lo <= z <= hi.  x^2 + y^2 + z^2 > r^2 is decided in FP64 as written; it
  // grows with |z|, so the two ends are a square root and a step or two away.
  const bool masked = A.mask_r2 > 0.0;
  uint32_t zin[VW];
#pragma unroll
  for (int j = 0; j < VW; ++j) zin[j] = 0u;
  if (masked && own) {
#pragma unroll 1
    for (int j = 0; j < VW; ++j) {
      const int qq = q + j;
      const double xm = (qq % nx) * A.h - A.cx, ym = (qq / nx) * A.h - A.cy;
      const double mxy = xm * xm + ym * ym;
      auto inside = [&](int z) {
        const double zm = z * A.h - A.cz;
        return !(mxy + zm * zm > A.mask_r2);
      };
      const int zc = min(nz - 1, max(0, (int)(A.cz / A.h + 0.5)));   // the plane nearest the centre
      int lo = 1, hi = 0;
      if (inside(zc)) {
        const int span = (int)fmin(sqrt(fmax(0.0, A.mask_r2 - mxy)) / A.h, (double)nz);
        lo = max(0, zc - span);
        while (lo > 0 && inside(lo - 1)) --lo;
        while (lo < zc && !inside(lo)) ++lo;
        hi = min(nz - 1, zc + span);
        while (hi < nz - 1 && inside(hi + 1)) ++hi;
        while (hi > zc && !inside(hi)) --hi;
      }
      const uint32_t v = (uint32_t)lo | ((uint32_t)hi << 16);
#pragma unroll
      for (int i = 0; i < VW; ++i)
        if (i == j) zin[i] = v;
    }
  }
  const T c0 = A.c0;
  const bool comp = sizeof(T) == 4 && A.csr != T(0);
  // (a context's grid has fewer than 2^30 points)
  int o = z0 * nxy + q;             // element of plane z
  const int ring_end = NBUF * WS;
  int ro = 0;                       // element of plane z's slot
  int fo = R * WS;                  // of the queue front's slot (plane z + R; R < NBUF)
  int fs = R;                       // that slot's number and parity
  uint32_t fpar = 0;
  int po = 0;                       // of plane z's Prev/pot slot
  // at unrolled position u, plane z - R + i lies in zq[.][(u + i) % Q]
#pragma unroll 1
  for (int zb = z0; zb < z1; zb += Q) {
#pragma unroll
    for (int u = 0; u < Q; ++u) {
      const int z = zb + u;
      if (z >= z1) break;
      // queue front: plane z + R
      const int pf = z + R;
      {
        T f[VW];
#pragma unroll
        for (int j = 0; j < VW; ++j) f[j] = T(0);
        if (pf < nz) {
          wait_plane(pf, bars + fs, fpar);
          if (own) vload<VW>(ring + (fo + s_c), f);
        }
#pragma unroll
        for (int j = 0; j < VW; ++j) zq[j][(u + 2 * R) % Q] = f[j];
      }
      const T* pl = ring + ro;
      T pv[VW], pt[VW];
      if constexpr (NPP > 0) {
        copy_pp(own && z + PP_SLOTS - 1 < z1, (po + (PP_SLOTS - 1) * PSTEP) & (PP_SLOTS * PSTEP - 1),
                o + (PP_SLOTS - 1) * nxy);
        cp_async_wait<PP_SLOTS - 1>();
      }
      if (own) {
        if constexpr (HASP) vload<VW>(pring + po + loc, pv);
        if constexpr (HASV) vload<VW>(pring + po + (HASP ? TS : 0) + loc, pt);
        // x neighbours: the aligned vectors around the run (the run itself is
        // the queue's centre).  Row-aligned runs (EXACT) read the vectors
        // outside the row from the slot's zero pad; otherwise each point
        // masks its neighbours by its distances to the row edges.
        T xs[NPV * VW];
#pragma unroll
        for (int v = 0; v < NPV; ++v) {
          if (v == HV) {
#pragma unroll
            for (int j = 0; j < VW; ++j) xs[v * VW + j] = zq[j][(u + R) % Q];
          } else {
            vload<VW>(pl + (EXACT ? xo[v] : s_c - OFF + v * VW), xs + v * VW);
          }
        }
        auto xl = [&](int j, int d) -> T { return (EXACT || d <= el[j]) ? xs[OFF + j - d] : T(0); };
        auto xr = [&](int j, int d) -> T { return (EXACT || d <= er[j]) ? xs[OFF + j + d] : T(0); };
        // per point: acc = c0 x + sum_d c_d (((y-d + y+d) + (z-d + z+d)) + (x-d + x+d)).
        // FP32 sums the shells from d = R down to 1 and adds c0 x last: of
        // the orders tried this leaves the smallest bias in the Rayleigh
        // quotients of smooth fields (the low spectrum), about 3e-9 Ha.
        constexpr bool REV = sizeof(T) == 4;
        T out[VW];
        if constexpr (PK) {
          constexpr int NH = VW / 2;
          // the window masked for each owner pair (PAIRM)
          float xa[PAIRM ? NPV * VW : 1], xb[PAIRM ? NPV * VW : 1];
          if constexpr (PAIRM) {
#pragma unroll
            for (int i = 0; i < NPV * VW; ++i) {
              const int p = i >> 1;
              xa[i] = p == 2 ? xs[i] : xs[i] * mA[p];
              xb[i] = p == 3 ? xs[i] : xs[i] * mB[p];
            }
          }
          float2 acc[NH];
#pragma unroll
          for (int h = 0; h < NH; ++h) {
            const float2 xc = make_float2(xs[OFF + 2 * h], xs[OFF + 2 * h + 1]);
            acc[h] = REV ? make_float2(0.f, 0.f) : __fmul2_rn(make_float2(c0, c0), xc);
          }
#pragma unroll
          for (int dd = 0; dd < R; ++dd) {
            const int d = REV ? R - dd : dd + 1;
            T ym[VW], yp[VW];
            vload_row<T, YA, VW>(pl + s_c - d * nx, d, ym);
            vload_row<T, YA, VW>(pl + s_c + d * nx, d, yp);
            const float2 cd = make_float2(A.c[d - 1], A.c[d - 1]);
            const int sm = (u + R - d) % Q, sp = (u + R + d) % Q;
#pragma unroll
            for (int h = 0; h < NH; ++h) {
              const int j = 2 * h;
              const float2 yy = __fadd2_rn(make_float2(ym[j], ym[j + 1]), make_float2(yp[j], yp[j + 1]));
              const float2 zz = __fadd2_rn(make_float2(zq[j][sm], zq[j + 1][sm]), make_float2(zq[j][sp], zq[j + 1][sp]));
              float2 xx;
              if constexpr (PAIRM) {
                const float* xw = h == 0 ? xa : xb;
                if (d % 2 == 0)
                  xx = __fadd2_rn(make_float2(xw[OFF + j - d], xw[OFF + j + 1 - d]),
                                  make_float2(xw[OFF + j + d], xw[OFF + j + 1 + d]));
                else
                  xx = make_float2(xw[OFF + j - d] + xw[OFF + j + d], xw[OFF + j + 1 - d] + xw[OFF + j + 1 + d]);
              } else if (EXACT && d % 2 == 0) {
                xx = __fadd2_rn(make_float2(xl(j, d), xl(j + 1, d)), make_float2(xr(j, d), xr(j + 1, d)));
              } else {
                xx = make_float2(xl(j, d) + xr(j, d), xl(j + 1, d) + xr(j + 1, d));
              }
              const float2 t = __fadd2_rn(__fadd2_rn(yy, zz), xx);
              acc[h] = __ffma2_rn(cd, t, acc[h]);
            }
          }
#pragma unroll
          for (int h = 0; h < NH; ++h) {
            const int j = 2 * h;
            const float2 xc = make_float2(xs[OFF + j], xs[OFF + j + 1]);
            float2 a = acc[h];
            if constexpr (REV) a = __ffma2_rn(make_float2(c0, c0), xc, a);
            if (comp) a = __ffma2_rn(make_float2(A.csr, A.csr), xc, a);
            if constexpr (HASV) a = __ffma2_rn(make_float2(pt[j], pt[j + 1]), xc, a);
            float2 r = __ffma2_rn(make_float2(ca, ca), a, __fmul2_rn(make_float2(cb, cb), xc));
            if constexpr (HASP) r = __ffma2_rn(make_float2(cg, cg), make_float2(pv[j], pv[j + 1]), r);
            out[j] = r.x;
            out[j + 1] = r.y;
          }
        } else {
          T acc[VW];
#pragma unroll
          for (int j = 0; j < VW; ++j) acc[j] = REV ? T(0) : c0 * xs[OFF + j];
#pragma unroll
          for (int dd = 0; dd < R; ++dd) {
            const int d = REV ? R - dd : dd + 1;
            T ym[VW], yp[VW];
            vload_row<T, YA, VW>(pl + s_c - d * nx, d, ym);
            vload_row<T, YA, VW>(pl + s_c + d * nx, d, yp);
            const T cd = A.c[d - 1];
#pragma unroll
            for (int j = 0; j < VW; ++j) {
              const T t = ((ym[j] + yp[j]) + (zq[j][(u + R - d) % Q] + zq[j][(u + R + d) % Q])) +
                          (xl(j, d) + xr(j, d));
              acc[j] += cd * t;
            }
          }
#pragma unroll
          for (int j = 0; j < VW; ++j) {
            const T xc = xs[OFF + j];
            T a = acc[j];
            if constexpr (REV) a += c0 * xc;
            if (comp) a += A.csr * xc;
            if constexpr (HASV) a += pt[j] * xc;
            out[j] = ca * a + cb * xc;
            if constexpr (HASP) out[j] += cg * pv[j];
          }
        }
        if (masked) {
#pragma unroll
          for (int j = 0; j < VW; ++j)
            if (z < (int)(zin[j] & 0xffffu) || z > (int)(zin[j] >> 16)) out[j] = T(0);
        }
        vstore<VW>(Yc + o, out);
      }
      o += nxy;
      po = (po + PSTEP) & (PP_SLOTS * PSTEP - 1);
      ro = ro + WS == ring_end ? 0 : ro + WS;
      ++fs;
      fo += WS;
      if (fo == ring_end) {
        fo = 0;
        fs = 0;
        fpar ^= 1u;
      }
      asm volatile("" : "+r"(ro), "+r"(fo), "+r"(po));
      // every SYNC_EVERY planes, and at the end of the pass: the slots of the
      // planes since the last barrier are free, so the ring is topped up to
      // plane z + NBUF.  The queue front z + R stays covered while
      // SYNC_EVERY <= NBUF - R.
      if (u % SYNC_EVERY == SYNC_EVERY - 1 || u == Q - 1) {
        __syncthreads();
        if (threadIdx.x == 0 && !fail)
          for (; issued < zlast && issued <= z + NBUF; ++issued) issue_x(issued, (issued - z0) % NBUF);
      }
    }
  }
  if (fail) s_fail = 1;
  // Thread 0 issues every copy and waits for the planes in order; once it
  // has given up it issues no more, so the planes fail_plane .. issued-1 sit
  // in distinct slots.  Their copies are drained before the CTA exits.
  if (threadIdx.x == 0 && fail)
    for (int p = fail_plane; p < issued; ++p)
      mbar_wait(&bars[(p - z0) % NBUF], ((p - z0) / NBUF) & 1, PSC_DRAIN_WAIT);
  __syncthreads();
  if (threadIdx.x == 0 && s_fail) atomicExch(&A.status[3], 1);
}

// Alignment rules of the 1-D bulk copies: 16-byte aligned addresses and
// sizes, i.e. even (FP64) or multiple-of-4 (FP32) element offsets.
template <typename T>
static bool tma_ok(const psc_ctx* ctx, const void* X, long ldx, const void* P, long ldp, const void* Y, long ldy) {
  const long q = 16 / sizeof(T);
  const long nxy = (long)ctx->nx * ctx->ny;
  if (nxy % q || (ctx->radius * (long)ctx->nx) % q || ldx % q || (P && ldp % q) || ldy % q) return false;
  if (((uintptr_t)X | (uintptr_t)Y | (uintptr_t)P) % 16) return false;
  return true;
}

// Work table of one launch.  A CTA owns (column, slab, z range); the cost of a
// CTA is modelled as its planes plus a pipeline fill.  CTAs are dispatched
// about in order as resident slots free up, so the table puts whole-column
// (or half-column) items first and splits the last m (column, slab) pairs
// into smaller z chunks that fill the final wave.  The split is the one with
// the shortest simulated list-scheduling makespan over `slots` resident CTAs
// (every chunk of a split counted at its longest).
static void z_chunks(int nz, int c, std::vector<int2>& out) {
  const int zc = (nz + c - 1) / c;
  out.clear();
  for (int z = 0; z < nz; z += zc) out.push_back(make_int2(z, std::min(nz, z + zc)));
}

// End of a greedy schedule of nb items of cost cb, then ns items of cost cs, on
// `slots` equal workers.  After the first kind the workers are free at one of
// two times, a round apart, and the workers of a time stay together, so a
// schedule costs one step per round (item by item the candidates took 27 ms at
// 307 columns, on every new grid context).
static double makespan(long nb, double cb, long ns, double cs, int slots) {
  const long late = nb % slots;                        // workers with one more item of the first kind
  long n[2] = {slots - late, late};
  double t[2] = {(nb / slots) * cb, (nb / slots + 1) * cb};
  double end = late > 0 ? t[1] : t[0];
  while (ns > 0) {
    const int w = late > 0 && t[1] < t[0] ? 1 : 0;
    ns -= std::min(ns, n[w]);
    t[w] += cs;
    end = std::max(end, t[w]);
  }
  return end;
}

static std::vector<int4> stencil_schedule(int nslab, int nz, int k, int fill, int slots) {
  const long pairs = (long)nslab * k;
  const int cmax = std::max(1, nz / 8);  // chunks of at least 8 planes
  double best = 1e300;
  int bb = 1, bs = 1;
  long bm = 0;
  std::vector<int2> cb, cs;
  for (int b = 1; b <= std::min(2, cmax); ++b) {
    for (int sm = 1; sm <= 4; ++sm) {
      const int sc = std::min(cmax, b * sm);
      if (sm > 1 && sc == b) continue;
      z_chunks(nz, b, cb);
      z_chunks(nz, sc, cs);
      const long step = std::max(1L, pairs / 32);
      for (long m = 0; m <= pairs; m += step) {
        if (sc == b && m > 0) break;
        const double t = makespan((pairs - m) * (long)cb.size(), cb[0].y - cb[0].x + fill, m * (long)cs.size(),
                                  cs[0].y - cs[0].x + fill, slots);
        if (t < best - 1e-9) {
          best = t;
          bb = b;
          bs = sc;
          bm = m;
        }
      }
    }
  }
  z_chunks(nz, bb, cb);
  z_chunks(nz, bs, cs);
  std::vector<int4> out;
  for (long p = 0; p < pairs; ++p) {
    const int col = (int)(p / nslab), slab = (int)(p % nslab);
    for (const int2& c : (p < pairs - bm ? cb : cs)) out.push_back(make_int4(col, slab, c.x, c.y));
  }
  return out;
}

// Masked launches (sphere mode): per slab, the planes [zlo, zhi) that hold a
// point inside the sphere (one plane of margin each side) are computed, the
// rest only zero-filled.  Compute items are cut into chunks of at most lc
// planes and sorted longest first; the zero items (column stored as
// -1 - column) follow, at about a third of a plane's cost each.
static std::vector<int4> stencil_schedule_masked(const psc_ctx* ctx, int ts, int nslab, int k, int slots) {
  const int nx = ctx->nx, nxy = ctx->nx * ctx->ny, nz = ctx->nz;
  std::vector<int2> zr(nslab);
  long work = 0;
  for (int sl = 0; sl < nslab; ++sl) {
    double d2 = 1e300;
    for (int q = sl * ts; q < std::min(nxy, (sl + 1) * ts); ++q) {
      const double x = (q % nx) * ctx->h - ctx->mask_c[0], y = (q / nx) * ctx->h - ctx->mask_c[1];
      d2 = std::min(d2, x * x + y * y);
    }
    int lo = nz, hi = 0;
    if (d2 <= ctx->mask_r2) {
      const double half = std::sqrt(ctx->mask_r2 - d2);
      lo = std::max(0, (int)std::floor((ctx->mask_c[2] - half) / ctx->h) - 1);
      hi = std::min(nz, (int)std::ceil((ctx->mask_c[2] + half) / ctx->h) + 2);
    }
    zr[sl] = make_int2(lo, hi);
    if (hi > lo) work += hi - lo;
  }
  const int lc = std::max(8, (int)std::min<long>(nz, (work * (long)k + 2L * slots - 1) / (2L * slots)));
  std::vector<int4> comp, zero;
  for (int col = 0; col < k; ++col)
    for (int sl = 0; sl < nslab; ++sl) {
      const int lo = zr[sl].x, hi = zr[sl].y;
      if (hi > lo) {
        const int nch = (hi - lo + lc - 1) / lc;
        const int len = (hi - lo + nch - 1) / nch;
        for (int z = lo; z < hi; z += len) comp.push_back(make_int4(col, sl, z, std::min(hi, z + len)));
        if (lo > 0) zero.push_back(make_int4(-1 - col, sl, 0, lo));
        if (hi < nz) zero.push_back(make_int4(-1 - col, sl, hi, nz));
      } else {
        zero.push_back(make_int4(-1 - col, sl, 0, nz));
      }
    }
  std::stable_sort(comp.begin(), comp.end(), [](const int4& a, const int4& b) { return a.w - a.z > b.w - b.z; });
  comp.insert(comp.end(), zero.begin(), zero.end());
  return comp;
}

static long long sched_key(int nslab, int k, int fill, int slots, bool masked) {
  return ((long long)k << 32) | ((long long)nslab << 16) | ((long long)fill << 8) | (slots & 0x7f) |
         (masked ? PSC_SCHED_MASKED : 0);
}

// Cached per context: the table of a (k, slab count, fill, mask) combination
// is built and uploaded once.  The upload has ended before the table is handed
// out, since the next call may be on a stream that does not wait for st.
static const int4* stencil_sched(psc_ctx* ctx, int nslab, int k, int fill, int slots, bool masked, int ts, int* n) {
  const long long key = sched_key(nslab, k, fill, slots, masked);
  for (auto& e : ctx->st_sched)
    if (e.key == key) {
      *n = e.n;
      return reinterpret_cast<const int4*>(e.dev);
    }
  psc_ctx::StencilSched e;
  e.key = key;
  std::vector<int4> tab = masked ? stencil_schedule_masked(ctx, ts, nslab, k, slots)
                                 : stencil_schedule(nslab, ctx->nz, k, fill, slots);
  e.n = (int)tab.size();
  if (psc_dmalloc(&e.dev, tab.size() * sizeof(int4)) != cudaSuccess) return nullptr;
  if (cudaMemcpyAsync(e.dev, tab.data(), tab.size() * sizeof(int4), cudaMemcpyHostToDevice, cudaStreamLegacy) !=
          cudaSuccess ||
      cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {
    psc_dfree(e.dev);
    return nullptr;
  }
  ctx->st_sched.push_back(e);
  *n = e.n;
  return reinterpret_cast<const int4*>(e.dev);
}

// The unmasked table for another kernel with the same (column, slab, z range)
// items.  *n = 0 and NULL if it is not there yet and a capture of st forbids the
// allocation.
const int4* psc_stencil_sched(psc_ctx* ctx, int nslab, int k, int fill, int slots, int* n, cudaStream_t st) {
  *n = 0;
  const long long key = sched_key(nslab, k, fill, slots, false);
  bool cached = false;
  for (const auto& e : ctx->st_sched) cached = cached || e.key == key;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (!cached && (cudaStreamIsCapturing(st, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone)) return nullptr;
  *n = -1;
  return stencil_sched(ctx, nslab, k, fill, slots, false, 0, n);
}

template <typename T, int R, int YA, int VW, bool PK, bool HASP, bool HASV, int DEEP>
static int launch_tma_k(psc_ctx* ctx, const TmaArgs<T>& A, int nwork, size_t smem, cudaStream_t st) {
  auto kern = k_stencil_tma<T, R, YA, VW, PK, HASP, HASV, DEEP>;
  PSC_CUDA(ctx, psc_smem_optin(kern));
  kern<<<nwork, TNT, smem, st>>>(A);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

template <typename T, int R, int VW, bool PK, int DEEP>
static int launch_tma_t(psc_ctx* ctx, int k, const T* X, long ldx, const T* P, long ldp, T* Y, long ldy,
                        const T* pot, const double* w, const double* coef, double a, double b, double g,
                        bool masked, bool comp, cudaStream_t st) {
  const int nxy = ctx->nx * ctx->ny;
  constexpr int TS = slab_points<VW>();
  const int nslab = (nxy + TS - 1) / TS;
  constexpr size_t Q16 = 16 / sizeof(T);
  const size_t win = (TS + 2 * (size_t)R * ctx->nx + VW + Q16 - 1) / Q16 * Q16;   // window + zero pad, 16-byte slots
  const size_t npp = (P ? 1 : 0) + (pot ? 1 : 0);
  const size_t slot = win * sizeof(T) + sizeof(uint64_t), pp = PP_SLOTS * npp * TS * sizeof(T);
  const size_t smem = (R + 1 + DEEP) * slot + pp;
  if (DEEP > AHEAD && smem > SMEM_HALF) return -1;   // (the caller comes back with AHEAD)
  if (smem > 220 * 1024) return -1;  // window too wide: the register-queue kernel takes it
  // each CTA pays a pipeline fill of about R + DEEP planes; two CTAs per SM
  // are resident (registers and shared memory)
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, ctx->device);
  const int slots = PSC_STENCIL_CTAS_PER_SM * sms;
  const int fill = R + DEEP + 2;
  int nwork = 0;
  masked = masked && ctx->mask_r2 > 0.0;
  const int4* sched = stencil_sched(ctx, nslab, k, fill, slots, masked, TS, &nwork);
  PSC_REQUIRE(ctx, sched != nullptr, "stencil: work table allocation failed");
  TmaArgs<T> A;
  A.X = X; A.ldx = ldx; A.P = P; A.ldp = ldp; A.Y = Y; A.ldy = ldy; A.pot = pot;
  A.nx = ctx->nx; A.ny = ctx->ny; A.nz = ctx->nz; A.sched = sched;
  A.c0 = (T)w[0];
  // the sum rule c0 + 6 sum_d c_d = 0 holds for the FP64 weights; in the
  // stored type it is off by the weights' rounding errors, which the
  // correction term removes (FP32 only)
  double rs = (double)A.c0 - w[0];
  for (int i = 0; i < 4; ++i) {
    A.c[i] = (T)w[1 + i];
    rs += 6.0 * ((double)A.c[i] - w[1 + i]);
  }
  A.csr = comp ? (T)(-rs) : T(0);
  A.coef = coef; A.a = a; A.b = b; A.g = g; A.status = ctx->dev_status;
  A.wait_limit = ctx->wait_limit;
  A.mask_r2 = masked ? ctx->mask_r2 : 0.0;
  A.h = ctx->h;
  A.cx = ctx->mask_c[0]; A.cy = ctx->mask_c[1]; A.cz = ctx->mask_c[2];
#define PSC_TMA_PV(YAV)                                                                         \
  {                                                                                             \
    if (P)                                                                                      \
      return pot ? launch_tma_k<T, R, YAV, VW, PK, true, true, DEEP>(ctx, A, nwork, smem, st)         \
                 : launch_tma_k<T, R, YAV, VW, PK, true, false, DEEP>(ctx, A, nwork, smem, st);       \
    return pot ? launch_tma_k<T, R, YAV, VW, PK, false, true, DEEP>(ctx, A, nwork, smem, st)          \
               : launch_tma_k<T, R, YAV, VW, PK, false, false, DEEP>(ctx, A, nwork, smem, st);        \
  }
  if constexpr (sizeof(T) == 4) {
    // FP32 is the Hamiltonian's path alone, which always has a potential
    PSC_REQUIRE(ctx, pot != nullptr, "stencil: FP32 blocks need the potential");
#define PSC_TMA_P(YAV)                                                                       \
  return P ? launch_tma_k<T, R, YAV, VW, PK, true, true, DEEP>(ctx, A, nwork, smem, st)            \
           : launch_tma_k<T, R, YAV, VW, PK, false, true, DEEP>(ctx, A, nwork, smem, st);
    if (ctx->nx % VW == 0) { PSC_TMA_P(VW) }
    if constexpr (VW == 4) {   // (2-point runs are taken only where 2 divides nx)
      if (ctx->nx % 2 == 0) { PSC_TMA_P(2) }
      PSC_TMA_P(1)
    }
    return -1;
#undef PSC_TMA_P
  } else {
    if (ctx->nx % VW == 0) PSC_TMA_PV(VW)
    PSC_TMA_PV(1)
  }
#undef PSC_TMA_PV
}

// Returns -1 if the TMA path does not apply (caller uses the register kernel).
template <typename T>
int psc_stencil_tma(psc_ctx* ctx, int k, const T* X, long ldx, const T* P, long ldp, T* Y, long ldy, const T* pot,
                    const double* w, const double* coef, double a, double b, double g, bool masked,
                    cudaStream_t st) {
  if (!tma_ok<T>(ctx, X, ldx, P, ldp, Y, ldy)) return -1;
  if (masked && ctx->nz > 0xffff) return -1;   // the mask's intervals are 16-bit planes
  // FP32 takes 4-point runs with the arithmetic on packed pairs (measured
  // fastest, also where nx is only 2-aligned and the x terms need per-point
  // edge masks: 818 us per step at 90^3, k = 307, when it was chosen, against 995-1055 us for
  // 2-point runs and 894 us for scalar arithmetic); impl 2 / 3 ask for
  // 2-point runs when nx is even but not a multiple of 4, impl 3 / 4 for
  // scalar arithmetic
  const int impl = ctx->stencil_impl;
  const bool narrow = sizeof(T) == 4 && ctx->nx % 4 != 0 && ctx->nx % 2 == 0 && (impl == 2 || impl == 3);
  // the correction term in the kernel: weights mode 1, or mode 2 when this
  // call's potential is not the FP32 potential that carries it
  const bool comp = ctx->stencil_comp == 1 ||
                    (ctx->stencil_comp == 2 && (const void*)pot != (const void*)ctx->pot32);
  const bool pk = impl == 0 || impl == 2;
#define PSC_TMA_ARGS ctx, k, X, ldx, P, ldp, Y, ldy, pot, w, coef, a, b, g, masked, comp, st
#define PSC_TMA_R(RRV)                                                                                        \
  case RRV: {                                                                                                 \
    constexpr int RR = RRV;                                                                                   \
    if constexpr (sizeof(T) == 8)                                                                             \
      return launch_tma_t<T, RR, 2, false, AHEAD>(PSC_TMA_ARGS);                                              \
    else if (narrow)                                                                                          \
      return pk ? launch_tma_t<T, RR, 2, true, AHEAD>(PSC_TMA_ARGS)                                           \
                : launch_tma_t<T, RR, 2, false, AHEAD>(PSC_TMA_ARGS);                                         \
    else {                                                                                                    \
      if (!pk) return launch_tma_t<T, RR, 4, false, AHEAD>(PSC_TMA_ARGS);                                     \
      const int rc = launch_tma_t<T, RR, 4, true, AHEAD_F32>(PSC_TMA_ARGS);                                   \
      return rc >= 0 ? rc : launch_tma_t<T, RR, 4, true, AHEAD>(PSC_TMA_ARGS);                                \
    }                                                                                                         \
  }
  switch (ctx->radius) {
    PSC_TMA_R(1)
    PSC_TMA_R(2)
    PSC_TMA_R(3)
    PSC_TMA_R(4)
  }
#undef PSC_TMA_R
#undef PSC_TMA_ARGS
  return -1;
}

template int psc_stencil_tma<double>(psc_ctx*, int, const double*, long, const double*, long, double*, long,
                                     const double*, const double*, const double*, double, double, double, bool,
                                     cudaStream_t);
template int psc_stencil_tma<float>(psc_ctx*, int, const float*, long, const float*, long, float*, long,
                                    const float*, const double*, const double*, double, double, double, bool,
                                    cudaStream_t);
