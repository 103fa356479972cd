// Persistent conjugate-gradient kernel for the Hartree solve
// (Eigensolvers/pcg.py:7-85), one cooperative launch per solve.  Two forms:
// the grid in boxes (k_cg_box, below) wherever a cut of it fits, for cubes up to
// 84^3 (order 8, 148 SMs), and in flat ranges (k_cg_persistent) from there to
// 93^3.
//
// The flat form.
// The CG vectors of a whole grid fit in the shared memory of the GPU (a
// 78^3 grid needs 4 x 474,552 doubles = 15 MB against 148 x 227 KB), so each
// of G co-resident CTAs (one per SM) keeps x, r, p and Ap of a contiguous
// range [a, b) of flat grid points in shared memory for the entire solve.
// The only vector other CTAs read is r, mirrored to global memory after each
// update (read back with loads that bypass L1, since its owners rewrite it
// every iteration).
//
// Iteration it (same stop rule as the two-kernel CG in pcg.cu, including the
// reference's aliased first direction update):
//   A  s = A r: x and y neighbours from a shared-memory window of r over
//      [a - R nx, b + R nx), z neighbours straight from global r;
//      p = r + beta q and Ap = s + beta Aq with q = previous p (q = r in the
//      second iteration, p = r in the first) -- Ap by this recurrence rather
//      than a second stencil, the same quantity in exact arithmetic; partial
//      of p.Ap                                                 -> grid barrier
//   B  pAp from all partials (every CTA sums them in the same order), alpha,
//      x += alpha p, r -= alpha Ap; own r to global; partial of r.r
//                                                              -> grid barrier
//   C  ro1 from all partials; the stop decision and beta are then identical
//      in every CTA.
// The grid barrier is a monotone arrival counter with a bounded spin: a CTA
// that waits more than 4x the context's wait limit (2^26 polls by default)
// records status[4] and stops waiting, so a fault can never hang the GPU.  Every
// CTA takes the same number of barriers.  The arrival is one release reduction
// and the wait one acquire load (two fences around an atomic: 0.8 us more per
// iteration).
#include "psc_internal.cuh"
#include "../../include/psc.h"

#include <algorithm>

namespace {
constexpr int PNT = 1024;

__device__ __forceinline__ void grid_barrier(unsigned int* ctr, unsigned int target, int* status, bool& failed,
                                             long limit) {
  __syncthreads();
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
    if (!failed) {
      long spins = 0;
      while (true) {
        unsigned int v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
        if (v >= target) break;
        if (++spins > limit) {
          failed = true;
          atomicExch(&status[4], 1);
          break;
        }
      }
    }
  }
  __syncthreads();
}

// Sum of the G per-CTA partials part[0..G) by warp 0 in a fixed order, the
// same in every CTA; the result is broadcast through shared memory.
__device__ __forceinline__ double grid_sum(const double* part, int G, double* bc) {
  if (threadIdx.x < 32) {
    double s = 0.0;
    for (int t = threadIdx.x; t < G; t += 32) s += __ldcg(part + t);
    s = psc_warp_sum(s);
    if (threadIdx.x == 0) *bc = s;
  }
  __syncthreads();
  const double r = *bc;
  return r;
}
}  // namespace

template <int R>
__global__ void __launch_bounds__(PNT, 1)
k_cg_persistent(const double* __restrict__ rhs, double* __restrict__ xg, double* rg, int nx, int ny, int nz,
                double c0, double4 cw, int chunk, double* part, unsigned int* bar, int* status, double tol,
                int maxit, double* out, long bar_limit) {
  extern __shared__ double sm[];
  __shared__ double sh[PNT / 32];
  __shared__ double bc[2];
  __shared__ int s_failed;
  const int n = nx * ny * nz;
  const int nxy = nx * ny;
  const int G = gridDim.x;
  const int a = blockIdx.x * chunk;
  const int b = min(n, a + chunk);
  const int L = max(0, b - a);
  const int hw = R * nx;                 // window halo: the x and y neighbours
  const int W = chunk + 2 * hw;
  double* xs = sm;
  double* rs = sm + chunk;
  double* ps = sm + 2 * chunk;
  double* aps = sm + 3 * chunk;
  double* win = sm + 4 * chunk;          // win[w] = vector at flat a - hw + w (0 outside the grid)
  const double cd[4] = {cw.x, cw.y, cw.z, cw.w};
  unsigned int nbar = 0;
  bool failed = false;
  if (threadIdx.x == 0) s_failed = 0;

  // A v at own point t: x, y neighbours from the window, z neighbours from zsrc
  auto stencil = [&](int t, const double* zsrc) -> double {
    const int g = a + t;
    const int k = g / nxy;
    const int rem = g - k * nxy;
    const int j = rem / nx;
    const int i = rem - j * nx;
    const double* c = win + hw + t;
    double zv[2 * R];
#pragma unroll
    for (int d = 1; d <= R; ++d) {   // issue every z load before using any
      zv[2 * d - 2] = (k - d >= 0) ? __ldcg(zsrc + g - d * nxy) : 0.0;
      zv[2 * d - 1] = (k + d < nz) ? __ldcg(zsrc + g + d * nxy) : 0.0;
    }
    double acc = c0 * c[0];
#pragma unroll
    for (int d = 1; d <= R; ++d) {
      double s = zv[2 * d - 2] + zv[2 * d - 1];
      s += (i - d >= 0) ? c[-d] : 0.0;
      s += (i + d < nx) ? c[d] : 0.0;
      s += (j - d >= 0) ? c[-d * nx] : 0.0;
      s += (j + d < ny) ? c[d * nx] : 0.0;
      acc += cd[d - 1] * s;
    }
    return acc;
  };
  auto fill_window = [&](const double* own, const double* glob) {
    for (int w = threadIdx.x; w < W; w += PNT) {
      const int t = w - hw;
      const int g = a + t;
      double v = 0.0;
      if (t >= 0 && t < L) v = own[t];
      else if (g >= 0 && g < n) v = __ldcg(glob + g);
      win[w] = v;
    }
  };

  // ---- set-up: own x, r = rhs - A x, ro = r.r ----
  for (int t = threadIdx.x; t < L; t += PNT) xs[t] = xg[a + t];
  __syncthreads();
  fill_window(xs, xg);
  __syncthreads();
  double rr = 0.0;
  for (int t = threadIdx.x; t < L; t += PNT) {
    const double ri = rhs[a + t] - stencil(t, xg);
    rs[t] = ri;
    rg[a + t] = ri;
    rr += ri * ri;
  }
  rr = psc_block_sum<double, PNT>(rr, sh);
  if (threadIdx.x == 0) part[G + blockIdx.x] = rr;
  grid_barrier(bar, (++nbar) * G, status, failed, bar_limit);
  double ro = grid_sum(part + G, G, &bc[0]);
  const double tol1 = tol * tol * ro;
  int it = 0;
  bool active = maxit > 0 && ro > tol1;
  double beta = 0.0;
  while (active) {
    ++it;
    const bool alias = it <= 2;              // q = r in the first two iterations
    const double bt = it == 1 ? 0.0 : beta;  // p = r in the first
    // A: s = A r, direction, Ap, partial of p.Ap
    fill_window(rs, rg);
    __syncthreads();
    double pap = 0.0;
    for (int t = threadIdx.x; t < L; t += PNT) {
      const double sv = stencil(t, rg);
      const double rv = rs[t];
      const double pv = rv + bt * (alias ? rv : ps[t]);
      const double av = sv + bt * (alias ? sv : aps[t]);
      ps[t] = pv;
      aps[t] = av;
      pap += av * pv;
    }
    pap = psc_block_sum<double, PNT>(pap, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = pap;
    grid_barrier(bar, (++nbar) * G, status, failed, bar_limit);
    pap = grid_sum(part, G, &bc[0]);
    // B: alpha, updates, partial of r.r
    const double alp = ro / pap;
    rr = 0.0;
    for (int t = threadIdx.x; t < L; t += PNT) {
      xs[t] += alp * ps[t];
      const double ri = rs[t] - alp * aps[t];
      rs[t] = ri;
      rg[a + t] = ri;
      rr += ri * ri;
    }
    rr = psc_block_sum<double, PNT>(rr, sh);
    if (threadIdx.x == 0) part[G + blockIdx.x] = rr;
    grid_barrier(bar, (++nbar) * G, status, failed, bar_limit);
    // C: stop test and beta, identical in every CTA
    const double ro1 = grid_sum(part + G, G, &bc[1]);
    beta = ro1 / ro;
    ro = ro1;
    active = it < maxit && ro1 > tol1;
    if (threadIdx.x == 0 && failed) s_failed = 1;
    __syncthreads();
    if (s_failed) active = false;  // a barrier gave up: leave in step
  }
  for (int t = threadIdx.x; t < L; t += PNT) xg[a + t] = xs[t];
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    out[0] = (double)it;
    out[1] = ro;
  }
}

// ---------------------------------------------------------------------------
// The same iteration with the grid cut into boxes, one per CTA.  With flat
// ranges every z neighbour of a point belongs to another CTA: eight L2 loads
// per point made the stencil 10.4k of the 23.9k cycles of an iteration at
// 78^3.  A box of 20 x 13 x 13 points has 5.5k halo points against 26k.  r with
// its halo lies in shared memory (rows padded so that consecutive points of a
// warp fall into consecutive banks across rows); a thread owns a run of up to
// PT points along z, its z neighbours in registers, and keeps p and Ap of the
// run in registers for the whole solve (x, in shared memory, is touched once
// per iteration; with it in registers the run's state spilled, and a release
// waits for spilled stores too; runs of more than 8 points still spill 88 bytes).  The halo points inside the grid
// (an address and a slot each) are listed once; those outside stay zero.
// 200 iterations take 1913 us at 78^3 and 1307 at 52^3 (solves of 2460 and 1620 in
// flat ranges, 1985 and 1370 now).  Of an iteration's 9.6 and 6.5 us the two
// reductions with their grid-wide visibility take 5.9; the rest is bound by
// shared-memory loads (17 per point) and FP64 issue.  (Counters: 7.3 warps
// stalled at a barrier and 3.2 on shared memory per issue.)
// ---------------------------------------------------------------------------
constexpr int BOX_NT = 512;
constexpr int BOX_PAD = 16;   // row pitch - box width (>= 2 R, a multiple of the 16 8-byte banks)

struct BoxPlan {
  int px, py, pz;   // boxes per axis
  int zs;           // z segments per box
  int hmax;         // halo points of the largest box
  int xmax;         // x values of the largest box (whole runs)
};

namespace {
__host__ __device__ __forceinline__ int box_lo(int i, int p, int n) { return (int)((long)i * n / p); }
}  // namespace

// A double that travels with the number of its reduction: two 64-bit words,
// each half a value and the number, so that a reader needs no other ordering
// to know that both halves are of this reduction.
namespace {
__device__ __forceinline__ void put_tagged(unsigned long long* w, double v, unsigned int tag) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v), t = (unsigned long long)tag << 32;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w), "l"((b & 0xffffffffull) | t) : "memory");
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(w + 1), "l"((b >> 32) | t) : "memory");
}
__device__ __forceinline__ bool get_tagged(const unsigned long long* w, unsigned int tag, double* v) {
  unsigned long long a, b;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(a) : "l"(w) : "memory");
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(b) : "l"(w + 1) : "memory");
  *v = __longlong_as_double((long long)((a & 0xffffffffull) | (b << 32)));
  return (unsigned int)(a >> 32) == tag && (unsigned int)(b >> 32) == tag;
}

// Sum of v over the grid, in every thread; also a grid barrier, and with
// `publish` one behind which every CTA sees the others' writes.  Each CTA
// stores its tagged sum and counts itself in; when the count is complete, warp
// 0 of every CTA reads all sums and adds them in the same order.  The tags
// spare the reductions that publish nothing the wait for their sum's store
// before the arrival.  (Two forms without the counter lost: every CTA polling
// every sum, and CTA 0 collecting them and handing the total back, 1.2 us more
// per reduction.)
//
// A reduction that does not publish orders no memory access of other CTAs, so
// nothing may rely on it alone to keep a write behind an earlier read: whatever
// one CTA reads and another overwrites must have a publishing reduction in
// between.  At least every second one publishes.  words: the counter, from
// word 16 on two per CTA in each of four sets that take turns, so a sum is
// overwritten four reductions later; r alternates between two arrays (k_cg_box).
__device__ __forceinline__ double grid_reduce(double v, bool publish, unsigned long long* words, unsigned int tag,
                                              double* sh, double* bc, int* s_failed, long limit, int* status) {
  const int G = gridDim.x;
  asm volatile("" : "+l"(words));   // (opaque: nothing below is kept in registers between the calls)
  unsigned int* ctr = reinterpret_cast<unsigned int*>(words);
  unsigned long long* sums = words + 16 + (tag & 3u) * 2 * G;
  v = psc_block_sum<double, BOX_NT>(v, sh);
  if (threadIdx.x < 32) {
    bool ok = *s_failed == 0;   // (after a wait gave up there is no other)
    __syncwarp();
    if (threadIdx.x == 0) {
      put_tagged(sums + 2 * blockIdx.x, v, tag);
      if (publish) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
      else asm volatile("red.relaxed.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
      const unsigned int target = tag * (unsigned int)G;
      for (long i = 0; ok; ++i) {
        unsigned int c;
        if (publish) asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(ctr) : "memory");
        else asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(c) : "l"(ctr) : "memory");
        if (c >= target) break;
        if (i >= limit) ok = false;
      }
    }
    ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
    double s = 0.0;
#pragma unroll 1
    for (int t0 = 0; t0 < G; t0 += 32 * 5) {   // five sums per lane in flight
      double w[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
      bool in[5];
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        const int t = t0 + 32 * q + (int)threadIdx.x;
        in[q] = t >= G || get_tagged(sums + 2 * t, tag, &w[q]);
      }
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        const int t = t0 + 32 * q + (int)threadIdx.x;
        for (long i = 0; ok && !in[q] && i < limit; ++i) in[q] = get_tagged(sums + 2 * t, tag, &w[q]);
        if (!in[q]) ok = false;
        if (t < G) s += w[q];
      }
    }
    __syncwarp();
    s = psc_warp_sum(s);
    const bool all_ok = __all_sync(0xffffffffu, ok);
    if (threadIdx.x == 0) {
      *bc = s;
      if (!all_ok && *s_failed == 0) {
        *s_failed = 1;
        atomicExch(&status[4], 1);
      }
    }
  }
  __syncthreads();
  return *bc;
}
}  // namespace

template <int R, int PT>
__global__ void __launch_bounds__(BOX_NT, 1)
k_cg_box(const double* __restrict__ rhs, double* __restrict__ xg, double* rg0, double* rg1, int nx, int ny, int nz,
         BoxPlan P, double c0, double4 cw, unsigned long long* words, int* status, double tol, int maxit, double* out,
         long bar_limit) {
  extern __shared__ double sm[];
  __shared__ double sh[BOX_NT / 32];
  __shared__ double bc[2];
  __shared__ int s_failed, s_h;
  const int tid = threadIdx.x;
  const int bi = blockIdx.x % P.px, bj = blockIdx.x / P.px % P.py, bk = blockIdx.x / (P.px * P.py);
  const int x0 = box_lo(bi, P.px, nx), y0 = box_lo(bj, P.py, ny), z0 = box_lo(bk, P.pz, nz);
  const int bx = box_lo(bi + 1, P.px, nx) - x0, by = box_lo(bj + 1, P.py, ny) - y0, bz = box_lo(bk + 1, P.pz, nz) - z0;
  const int pitch = bx + BOX_PAD, plane = pitch * (by + 2 * R), nxy = nx * ny;
  const int slots = plane * (bz + 2 * R);
  double* v = sm;                                                        // the box of r with its halo
  double* xs = v + slots;                                                // [run point][thread] x
  int* hg = reinterpret_cast<int*>(xs + P.xmax);                         // [hmax] grid index
  unsigned short* hs = reinterpret_cast<unsigned short*>(hg + P.hmax);   // [hmax] slot
  const double cd[4] = {cw.x, cw.y, cw.z, cw.w};
  unsigned int nred = 0;
  if (tid == 0) s_failed = s_h = 0;
  for (int e = tid; e < slots; e += BOX_NT) v[e] = 0.0;
  __syncthreads();
  for (int e = tid; e < slots; e += BOX_NT) {
    const int k = e / plane - R, j = e / pitch % (by + 2 * R) - R, i = e % pitch - R;
    if (i >= bx + R) continue;   // the padding
    const int off = (i < 0 || i >= bx) + (j < 0 || j >= by) + (k < 0 || k >= bz);
    const int gx = x0 + i, gy = y0 + j, gz = z0 + k;
    if (off == 1 && gx >= 0 && gx < nx && gy >= 0 && gy < ny && gz >= 0 && gz < nz) {
      const int h = atomicAdd(&s_h, 1);
      hg[h] = gx + nx * gy + nxy * gz;
      hs[h] = (unsigned short)e;
    }
  }
  // this thread's run: points (x, y, zlo .. zlo + m - 1) of the box
  const int ncol = bx * by, zr = (bz + P.zs - 1) / P.zs;
  const int seg = tid / ncol, col = tid - seg * ncol;
  const int tx = col % bx, ty = col / bx, zlo = seg * zr;
  const int m = seg < P.zs ? max(0, min(zr, bz - zlo)) : 0;
  const int sb = (zlo + R) * plane + (ty + R) * pitch + tx + R;           // slot and grid index of its first point
  const int gb = x0 + tx + nx * (y0 + ty) + nxy * (z0 + zlo);
  __syncthreads();
  const int nh = s_h;

  auto fill_halo = [&](const double* src) {
    int h0 = tid;
    asm volatile("" : "+r"(h0));
    for (; h0 < nh; h0 += 8 * BOX_NT) {   // eight loads in flight per thread
      double t[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int h = h0 + q * BOX_NT;
        t[q] = h < nh ? __ldcg(src + hg[h]) : 0.0;
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int h = h0 + q * BOX_NT;
        if (h < nh) v[hs[h]] = t[q];
      }
    }
  };
  // A v along the run: f(i, A v, v) for its points in order
  auto along_run = [&](auto f) {
    double zc[PT + 2 * R];
    int o = sb - R * plane;   // (opaque: the solver's loop would keep every point's addresses in spilled registers)
    asm volatile("" : "+r"(o));
#pragma unroll
    for (int i = 0; i < 2 * R; ++i, o += plane) zc[i] = m > 0 ? v[o] : 0.0;
    o -= R * plane;
#pragma unroll
    for (int i = 0; i < PT; ++i) {
      if (i < m) {
        const double* c = v + o;
        zc[i + 2 * R] = c[R * plane];
        double acc = c0 * zc[R + i];
#pragma unroll
        for (int d = 1; d <= R; ++d) {
          double s = zc[R + i - d] + zc[R + i + d];
          s += c[-d];
          s += c[d];
          s += c[-d * pitch];
          s += c[d * pitch];
          acc += cd[d - 1] * s;
        }
        f(i, acc, zc[R + i]);
        o += plane;
        asm volatile("" : "+r"(o));
      }
    }
  };

  // ---- set-up: own x, r = rhs - A x, ro = r.r ----
  double p[PT], ap[PT];
  const int nu = ncol * P.zs;   // threads with a run
#pragma unroll
  for (int i = 0; i < PT; ++i) {
    p[i] = ap[i] = 0.0;
    if (i < m) {
      const double xi = xg[gb + i * nxy];
      xs[i * nu + tid] = xi;
      v[sb + i * plane] = xi;
    }
  }
  fill_halo(xg);
  __syncthreads();
  double rr = 0.0;
  along_run([&](int i, double av, double) {
    const double ri = rhs[gb + i * nxy] - av;
    ap[i] = ri;   // (until every thread has read x)
    rg0[gb + i * nxy] = ri;
    rr += ri * ri;
  });
  __syncthreads();
#pragma unroll
  for (int i = 0; i < PT; ++i)
    if (i < m) v[sb + i * plane] = ap[i];
  // (bc alternates: a total is read until the next reduction ends)
  double ro = grid_reduce(rr, true, words, ++nred, sh, &bc[1], &s_failed, bar_limit, status);
  const double tol1 = tol * tol * ro;
  int it = 0;
  bool active = maxit > 0 && ro > tol1;
  double beta = 0.0;
  while (active) {
    ++it;
    const bool alias = it <= 2;              // q = r in the first two iterations
    const double bt = it == 1 ? 0.0 : beta;  // p = r in the first
    // r for the neighbours: read from one array, written to the other.  The
    // one read here is written in the next iteration, behind this one's second
    // reduction, which publishes.
    const double* rin = it & 1 ? rg0 : rg1;
    fill_halo(rin);
    __syncthreads();
    double pap = 0.0;
    along_run([&](int i, double sv, double rv) {
      p[i] = rv + bt * (alias ? rv : p[i]);
      ap[i] = sv + bt * (alias ? sv : ap[i]);
      pap += ap[i] * p[i];
    });
    pap = grid_reduce(pap, false, words, ++nred, sh, &bc[0], &s_failed, bar_limit, status);
    const double alp = ro / pap;
    rr = 0.0;
    double* rout = it & 1 ? rg1 : rg0;
    int o = sb, g = gb, xo = tid;
    asm volatile("" : "+r"(o), "+r"(g), "+r"(xo));
#pragma unroll
    for (int i = 0; i < PT; ++i, o += plane, g += nxy, xo += nu)
      if (i < m) {
        xs[xo] += alp * p[i];
        const double ri = v[o] - alp * ap[i];
        v[o] = ri;
        rout[g] = ri;
        rr += ri * ri;
      }
    const double ro1 = grid_reduce(rr, true, words, ++nred, sh, &bc[1], &s_failed, bar_limit, status);
    beta = ro1 / ro;
    ro = ro1;
    active = it < maxit && ro1 > tol1;
    if (s_failed) active = false;  // a reduction gave up: leave (the others' waits run out too)
  }
#pragma unroll
  for (int i = 0; i < PT; ++i)
    if (i < m) xg[gb + i * nxy] = xs[i * nu + tid];
  if (blockIdx.x == 0 && tid == 0) {
    out[0] = (double)it;
    out[1] = ro;
  }
}

// The cut with the least work per iteration: about one cycle per point of the
// largest box (two threads' slots of a warp per cycle, whole warps) and a
// quarter per halo point, and a run's own latency (of equal cuts the one with more
// threads and shorter runs); false if none fits shared memory, threads and runs.
static bool box_plan(const psc_ctx* ctx, int sms, size_t lim, BoxPlan* best, int* pt, size_t* smem) {
  const int R = ctx->radius, nx = ctx->nx, ny = ctx->ny, nz = ctx->nz;
  double cost = 1e300;
  for (int px = 1; px <= std::min(sms, nx); ++px)
    for (int py = 1; px * py <= sms && py <= ny; ++py) {
      const int pz = std::min(sms / (px * py), nz);
      const int bx = (nx + px - 1) / px, by = (ny + py - 1) / py, bz = (nz + pz - 1) / pz;
      const int ncol = bx * by;
      if (ncol > BOX_NT) continue;
      const int zs = std::min(bz, BOX_NT / ncol), zr = (bz + zs - 1) / zs;
      if (zr > 12) continue;
      const long slots = (long)(bx + BOX_PAD) * (by + 2 * R) * (bz + 2 * R);
      const long halo = 2L * R * ((long)by * bz + (long)bx * bz + (long)bx * by);
      const long xn = (long)ncol * zs * zr;
      const size_t need = (slots + xn) * sizeof(double) + halo * (sizeof(int) + sizeof(unsigned short));
      if (slots > 65535 || need > lim) continue;
      const double c = (double)((ncol * zs + 31) / 32 * 32) * zr + 0.25 * halo + 40.0 * zr;
      if (c < cost) {
        cost = c;
        *best = BoxPlan{px, py, pz, zs, (int)((halo + 1) / 2 * 2), (int)xn};
        *pt = zr <= 4 ? 4 : (zr <= 8 ? 8 : 12);
        *smem = need + 16;
      }
    }
  return cost < 1e300;
}

// Persistent solve if the vectors fit in shared memory; returns -1 if not
// (the caller then uses the graph-replayed kernels).
int psc_pcg_persistent(psc_ctx* ctx, const double* rhs, double* x, int maxit, double tol, int* its_out,
                       cudaStream_t st) {
  if (ctx->cg_persistent == 0) return -1;
  int sms = 0, dev = ctx->device;
  PSC_CUDA(ctx, cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  int coop = 0;
  PSC_CUDA(ctx, cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
  if (!coop || sms <= 0) return -1;
  const long n = ctx->n;
  if (n >= (1L << 31) - 1) return -1;
  int G = sms;
  const int R = ctx->radius;
  const long chunk = (n + G - 1) / G;
  size_t smem = (5 * (size_t)chunk + 2 * (size_t)R * ctx->nx) * sizeof(double);
  int optin = 0;
  PSC_CUDA(ctx, cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
  // boxes where a cut fits, flat ranges above (cubes of 85^3 to 93^3 at order 8)
  BoxPlan plan;
  int pt = 0, threads = PNT;
  size_t box_smem = 0;
  const bool box = box_plan(ctx, sms, (size_t)optin - 2048, &plan, &pt, &box_smem);
  if (!box && smem + 2048 > (size_t)optin) return -1;
  void* fn = nullptr;
#define PSC_CG_FN(RR)                                                                               \
  fn = !box ? (void*)k_cg_persistent<RR>                                                            \
            : (pt == 4 ? (void*)k_cg_box<RR, 4> : (pt == 8 ? (void*)k_cg_box<RR, 8> : (void*)k_cg_box<RR, 12>))
  switch (R) {
    case 1: PSC_CG_FN(1); break;
    case 2: PSC_CG_FN(2); break;
    case 3: PSC_CG_FN(3); break;
    default: PSC_CG_FN(4); break;
  }
#undef PSC_CG_FN
  if (box) {
    smem = box_smem;
    threads = BOX_NT;
    G = plan.px * plan.py * plan.pz;
  }
  PSC_CUDA(ctx, psc_smem_optin(fn));
  int per_sm = 0;
  PSC_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem));
  if (per_sm < 1) return -1;
  if (!ctx->cg_r) PSC_CUDA(ctx, psc_dmalloc(&ctx->cg_r, n * sizeof(double)));
  // the arrival counter, or the box kernel's words: 16 and 8 per CTA
  const size_t bar_bytes = (16 + 8 * (size_t)sms) * sizeof(unsigned long long);
  if (!ctx->cg_bar) PSC_CUDA(ctx, psc_dmalloc(&ctx->cg_bar, bar_bytes));
  if (ctx->cg_part_cap < G) {
    psc_dfree(ctx->cg_part);
    ctx->cg_part = nullptr;
    PSC_CUDA(ctx, psc_dmalloc(&ctx->cg_part, 2 * (size_t)std::max(G, PSC_RED_BLOCKS) * sizeof(double)));
    ctx->cg_part_cap = std::max(G, PSC_RED_BLOCKS);
  }
  PSC_CUDA(ctx, cudaMemsetAsync(ctx->cg_bar, 0, bar_bytes, st));
  const double4 cw = make_double4(ctx->lap_c[0], ctx->lap_c[1], ctx->lap_c[2], ctx->lap_c[3]);
  double* out = ctx->scalars + 80;
  double* rg = ctx->cg_r;
  double* rg1 = ctx->cg_p;
  unsigned int* bar = ctx->cg_bar;
  auto* words = reinterpret_cast<unsigned long long*>(ctx->cg_bar);
  int* status = ctx->dev_status;
  int nx = ctx->nx, ny = ctx->ny, nz = ctx->nz;
  double c0 = ctx->lap_c0;
  int chunk_i = (int)chunk;
  double* part = ctx->cg_part;
  long bar_limit = 4 * ctx->wait_limit;   // grid barriers wait 4x longer than the mbarrier pipelines
  void* args[] = {(void*)&rhs, (void*)&x, (void*)&rg, (void*)&nx, (void*)&ny, (void*)&nz, (void*)&c0, (void*)&cw,
                  (void*)&chunk_i, (void*)&part, (void*)&bar, (void*)&status, (void*)&tol, (void*)&maxit, (void*)&out,
                  (void*)&bar_limit};
  void* box_args[] = {(void*)&rhs, (void*)&x, (void*)&rg, (void*)&rg1, (void*)&nx, (void*)&ny, (void*)&nz,
                      (void*)&plan, (void*)&c0, (void*)&cw, (void*)&words, (void*)&status, (void*)&tol,
                      (void*)&maxit, (void*)&out, (void*)&bar_limit};
  PSC_CUDA(ctx, cudaLaunchCooperativeKernel(fn, dim3(G), dim3(threads), box ? box_args : args, smem, st));
  PSC_LAUNCH_CHECK(ctx);
  PSC_CUDA(ctx, cudaMemcpyAsync(ctx->host_scalars + 80, out, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
  int* hflag = reinterpret_cast<int*>(ctx->host_scalars + 82);
  PSC_CUDA(ctx, cudaMemcpyAsync(hflag, status + 4, sizeof(int), cudaMemcpyDeviceToHost, st));
  PSC_CUDA(ctx, cudaStreamSynchronize(st));
  if (*hflag) {
    psc_set_error(ctx, "pcg: persistent CG grid barrier timed out (CTAs not co-resident?)");
    return 1;
  }
  if (its_out) *its_out = (int)ctx->host_scalars[80];
  return 0;
}
