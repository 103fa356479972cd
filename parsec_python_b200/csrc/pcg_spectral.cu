// Preconditioned Hartree solve (cg_prec = 1): conjugate gradients on
// A = -Lap_h with a spectral preconditioner, in the preconditioned form of
// Eigensolvers/pcg.py:7-85 (z = M r, p = z, ro = z.r, stop when
// z.r <= tol^2 z0.r0).
//
// The preconditioner.  On the nx x ny x nz box with zero values outside, the
// orthonormal discrete sine transform (DST-I) of each axis,
//   S[j][k] = sqrt(2 / (m + 1)) sin(pi (j + 1)(k + 1) / (m + 1)),
// diagonalises the same finite-difference stencil continued by odd
// reflection across the faces; its eigenvalues are the stencil's symbol,
//   Lambda = lap_c0 + sum_axes sum_d 2 lap_c[d] cos(d theta_axis),
//   theta = pi (k + 1) / (m + 1).
// For the 2nd-order stencil that operator is A itself; for wider stencils it
// differs from A only in the R planes next to each face (A reads zeros
// there, the reflected operator reads mirrored values), so
//   M = S_z S_y S_x Lambda^-1 S_x S_y S_z
// is a symmetric positive definite approximate inverse whose error is
// confined to the boundary layer.  S is symmetric and its own inverse.
//
// Mode k is even or odd about the middle of the axis as k is, so a transform
// is a butterfly (x_j + x_{m-1-j}, x_j - x_{m-1-j}) and two products of half
// the size: the even modes from the sums, the odd modes from the differences
// -- half the operations of the full product.  Spectral values are kept with
// the even modes first.  The way back is the transposed product and the same
// butterfly.
//
// The products run on the FP64 tensor cores (mma.sync m8n8k4), and an
// application is three launches:
//   k_spec_xy<fwd>  one CTA per xy plane: the plane in shared memory, along x,
//                   then along y
//   k_spec_z        32 neighbouring z lines per CTA: forward, 1 / Lambda, back
//   k_spec_xy<back> along y, then along x
// so the five passes of one transform each (16 lines by the full matrix,
// scalar FMAs fed from shared memory, 26 us each at 92^3) become three, and
// the CG's vector updates ride on them: x += alpha p, r -= alpha A p where
// the plane of r is loaded, z.r where the plane of z is stored.  The limit is
// the FP64 tensor rate of the CTAs at work: one plane per CTA leaves 148 - nz
// SMs idle, which still beats a second pass over the grid.
//
// The whole solve runs from device flags: the host queues iterations ahead
// and reads the state once per batch; kernels of iterations past convergence
// return at once.
//
// The reference's own cg_prec = 1 path has nothing to reproduce: its CPU
// branch passes the string "precLU" where pcg.py calls a function
// (rsdft_solver.py:339 into pcg.py:43) and its GPU twin ignores the
// preconditioner (pcg_gpu.py:38-41).
#include "psc_internal.cuh"
#include "../../include/psc.h"

#include <algorithm>
#include <cmath>
#include <vector>

constexpr int SP_MAXM = 128;
constexpr int XY_NT = 512;   // 16 warps: 4 row groups x 4 column groups
constexpr int XY_RB = 6;     // rows a warp loads or stores at a time
constexpr int Z_NT = 256;    // 8 warps: 2 parities x 4 row groups
constexpr int Z_W = 32;      // z lines per CTA
constexpr int Z_P = Z_W + 4; // pitch of the z tile (4 mod 16: two wavefronts per fragment load)

// One axis: m points, he even and ho odd modes; matrices [2][kp][pm] with
// M[part][j][a] = S[j][2 a + part], zero beyond; lam by stored mode.
struct SpecAxis {
  const double* M;
  const double* lam;
  int m, he, ho, kp, pm;
};

// scalars of a solve (device): ro, ro1, tol1, iterations, active
enum { SC_RO = 0, SC_RO1 = 1, SC_TOL1 = 2, SC_ITS = 3, SC_ACTIVE = 4 };

static int round_pitch(int n) {   // smallest pitch >= n that is 4 mod 16
  int p = (n + 3) / 4 * 4;
  while (p % 16 != 4) p += 4;
  return p;
}

namespace {
__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// acc[i][j] += sum over ks of A(i, ks) B(j, ks): fragment addresses come from
// the functors (lane included); nr x nc tiles of the 4 x 4 are live
template <int TR, int TC, typename FA, typename FB>
__device__ __forceinline__ void spec_mm(int nks, int nr, int nc, FA fa, FB fb, double (&acc)[TR][TC][2]) {
#pragma unroll
  for (int i = 0; i < TR; ++i)
#pragma unroll
    for (int j = 0; j < TC; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
  for (int ks = 0; ks < nks; ++ks) {
    double a[TR], b[TC];
#pragma unroll
    for (int i = 0; i < TR; ++i) a[i] = i < nr ? *fa(i, ks) : 0.0;
#pragma unroll
    for (int j = 0; j < TC; ++j) b[j] = j < nc ? *fb(j, ks) : 0.0;
#pragma unroll
    for (int i = 0; i < TR; ++i)
#pragma unroll
      for (int j = 0; j < TC; ++j)
        if (i < nr && j < nc) dmma(acc[i][j][0], acc[i][j][1], a[i], b[j]);
  }
}
}  // namespace

// What a forward pass does to r on its way in, and a backward pass with z on
// its way out.
struct XyArgs {
  const double* in;
  double* out;
  SpecAxis X, Y;
  int pd, rows;        // pitch and rows of the plane in shared memory
  int same;            // X.M == Y.M
  const double* sc;    // solve state (NULL: a plain application)
  // forward, in a solve: alpha = ro1 / sum(part); x += alpha p, r -= alpha ap, in = r
  double* r;
  double* x;
  const double* p;
  const double* ap;
  const double* part;
  int npart;
  // backward, in a solve: zr[plane] = sum of out r
  double* zr;
};

template <bool FWD>
__global__ void __launch_bounds__(XY_NT, 1)
k_spec_xy(XyArgs P) {
  extern __shared__ double sp_sm[];
  __shared__ double sh[XY_NT / 32];
  __shared__ double s_alp;
  const bool step = FWD && P.x != nullptr;
  if (P.sc && P.sc[SC_ACTIVE] == 0.0) return;
  const int nx = P.X.m, ny = P.Y.m, pd = P.pd;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int l4 = lane >> 2, lk = lane & 3;
  const int wr = warp >> 2, wc = warp & 3;
  double* D = sp_sm;                          // [rows][pd]
  double* M = sp_sm + (size_t)P.rows * pd;    // matrices of the axis at work
  const long base = (long)blockIdx.x * nx * ny;
  auto load_matrix = [&](const SpecAxis& A) {
    const int nm = 2 * A.kp * A.pm;
#pragma unroll 8
    for (int e = tid; e < nm; e += XY_NT) M[e] = A.M[e];
  };
  if (step) {
    double s = 0.0;
    for (int i = tid; i < P.npart; i += XY_NT) s += P.part[i];
    s = psc_block_sum<double, XY_NT>(s, sh);
    if (tid == 0) s_alp = P.sc[SC_RO1] / s;
    __syncthreads();
  }
  const double alp = step ? s_alp : 0.0;
  load_matrix(FWD ? P.X : P.Y);
  // the plane, zero beyond its sides: a warp takes whole rows, XY_RB of them
  // at a time so that their loads are in flight together
  for (int j0 = warp; j0 < P.rows; j0 += XY_RB * (XY_NT / 32))
    for (int i = lane; i < pd; i += 32) {
      double v[XY_RB];
#pragma unroll
      for (int u = 0; u < XY_RB; ++u) {
        const int j = j0 + u * (XY_NT / 32);
        const long g = base + i + (long)j * nx;
        v[u] = (i < nx && j < ny) ? (step ? P.r[g] - alp * P.ap[g] : P.in[g]) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < XY_RB; ++u) {
        const int j = j0 + u * (XY_NT / 32);
        if (j < P.rows) D[j * pd + i] = v[u];
        if (step && i < nx && j < ny) {
          const long g = base + i + (long)j * nx;
          P.r[g] = v[u];
          P.x[g] += alp * P.p[g];
        }
      }
    }
  __syncthreads();
  auto butterfly_x = [&]() {
    const int h = nx / 2;
    for (int j = warp; j < ny; j += XY_NT / 32)
      for (int i = lane; i < h; i += 32) {
        double* a = D + j * pd + i;
        double* b = D + j * pd + nx - 1 - i;
        const double p = *a, q = *b;
        *a = p + q;
        *b = p - q;
      }
  };
  auto butterfly_y = [&]() {
    const int h = ny / 2;
    for (int j = warp; j < h; j += XY_NT / 32)
      for (int i = lane; i < nx; i += 32) {
        double* a = D + j * pd + i;
        double* b = D + (ny - 1 - j) * pd + i;
        const double p = *a, q = *b;
        *a = p + q;
        *b = p - q;
      }
  };
  double acc[4][4][2];
  // along x: rows are grid rows (4 groups), columns the two parities (2 groups each)
  auto along_x = [&]() {
    const SpecAxis& A = P.X;
    const int part = wc >> 1, size = part ? A.ho : A.he;
    const double* Mp = M + (size_t)part * A.kp * A.pm;
    const int rt = P.rows / 8, rq = (rt + 3) / 4, r0 = wr * rq, nr = min(rq, rt - r0);
    const int ct = A.kp / 8, cq = (ct + 1) / 2, c0 = (wc & 1) * cq, nc = min(cq, ct - c0);
    const int nks = (size + 3) / 4;
    if (nr > 0 && nc > 0) {
      if constexpr (FWD)
        spec_mm<4, 4>(nks, nr, nc,
                      [&](int i, int ks) {
                        const int k = 4 * ks + lk;
                        return D + (8 * (r0 + i) + l4) * pd + (part ? max(0, nx - 1 - k) : k);
                      },
                      [&](int j, int ks) { return Mp + (4 * ks + lk) * A.pm + 8 * (c0 + j) + l4; }, acc);
      else
        spec_mm<4, 4>(nks, nr, nc,
                      [&](int i, int ks) { return D + (8 * (r0 + i) + l4) * pd + (part ? A.he : 0) + 4 * ks + lk; },
                      [&](int j, int ks) { return Mp + (8 * (c0 + j) + l4) * A.pm + 4 * ks + lk; }, acc);
    }
    __syncthreads();   // every read of D is done
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int row = 8 * (r0 + i) + l4, n = 8 * (c0 + j) + 2 * lk + h;
          if (i < nr && j < nc && row < ny && n < size)
            D[row * pd + (FWD ? (part ? A.he + n : n) : (part ? nx - 1 - n : n))] = acc[i][j][h];
        }
  };
  // along y: rows are the two parities (2 groups each), columns x positions (4 groups)
  auto along_y = [&]() {
    const SpecAxis& A = P.Y;
    const int part = wr >> 1, size = part ? A.ho : A.he;
    const double* Mp = M + (size_t)part * A.kp * A.pm;
    const int rt = A.kp / 8, rq = (rt + 1) / 2, r0 = (wr & 1) * rq, nr = min(rq, rt - r0);
    const int ct = (nx + 7) / 8, cq = (ct + 3) / 4, c0 = wc * cq, nc = min(cq, ct - c0);
    const int nks = (size + 3) / 4;
    if (nr > 0 && nc > 0) {
      if constexpr (FWD)
        spec_mm<4, 4>(nks, nr, nc,
                      [&](int i, int ks) { return Mp + (4 * ks + lk) * A.pm + 8 * (r0 + i) + l4; },
                      [&](int j, int ks) {
                        const int k = 4 * ks + lk;
                        return D + (part ? max(0, ny - 1 - k) : k) * pd + 8 * (c0 + j) + l4;
                      }, acc);
      else
        spec_mm<4, 4>(nks, nr, nc,
                      [&](int i, int ks) { return Mp + (8 * (r0 + i) + l4) * A.pm + 4 * ks + lk; },
                      [&](int j, int ks) { return D + ((part ? A.he : 0) + 4 * ks + lk) * pd + 8 * (c0 + j) + l4; },
                      acc);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int n = 8 * (r0 + i) + l4, col = 8 * (c0 + j) + 2 * lk + h;
          if (i < nr && j < nc && n < size && col < nx)
            D[(FWD ? (part ? A.he + n : n) : (part ? ny - 1 - n : n)) * pd + col] = acc[i][j][h];
        }
  };
  if constexpr (FWD) {
    butterfly_x();
    __syncthreads();
    along_x();
    if (!P.same) {
      __syncthreads();
      load_matrix(P.Y);
    }
    __syncthreads();
    butterfly_y();
    __syncthreads();
    along_y();
  } else {
    along_y();
    if (!P.same) {
      __syncthreads();
      load_matrix(P.X);
    }
    __syncthreads();
    butterfly_y();
    __syncthreads();
    along_x();
    __syncthreads();
    butterfly_x();
  }
  __syncthreads();
  double s = 0.0;
  for (int j0 = warp; j0 < ny; j0 += XY_RB * (XY_NT / 32))
    for (int i = lane; i < nx; i += 32) {
      double rv[XY_RB];
      if (!FWD && P.zr)
#pragma unroll
        for (int u = 0; u < XY_RB; ++u) {
          const int j = j0 + u * (XY_NT / 32);
          rv[u] = j < ny ? P.r[base + i + (long)j * nx] : 0.0;
        }
#pragma unroll
      for (int u = 0; u < XY_RB; ++u) {
        const int j = j0 + u * (XY_NT / 32);
        if (j < ny) {
          const double v = D[j * pd + i];
          P.out[base + i + (long)j * nx] = v;
          if (!FWD && P.zr) s += v * rv[u];
        }
      }
    }
  if (!FWD && P.zr) {
    s = psc_block_sum<double, XY_NT>(s, sh);
    if (tid == 0) P.zr[blockIdx.x] = s;
  }
}

// z lines q0 .. q0 + 31 of the plane's flat (stored-mode) index: forward,
// divide by the eigenvalue, back; out may be in (its solver's calls are): a CTA
// reads all of its lines before it writes them, and no other CTA's
__global__ void __launch_bounds__(Z_NT)
k_spec_z(const double* in, double* out, SpecAxis X, SpecAxis Y, SpecAxis A, int rows,
         const double* sc) {
  extern __shared__ double sp_sm[];
  if (sc && sc[SC_ACTIVE] == 0.0) return;
  const int nz = A.m, nx = X.m, nxy = X.m * Y.m;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int l4 = lane >> 2, lk = lane & 3;
  double* D = sp_sm;                        // [rows][Z_P]
  double* M = sp_sm + (size_t)rows * Z_P;   // [2][kp][pm]
  const int q0 = blockIdx.x * Z_W;
  const int q = q0 + (tid & 31);            // this thread's column in the loads and stores
#pragma unroll 8
  for (int e = tid; e < 2 * A.kp * A.pm; e += Z_NT) M[e] = A.M[e];
  for (int z0 = warp; z0 < rows; z0 += 8 * (Z_NT / 32)) {   // eight loads in flight per thread
    double v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int z = z0 + u * (Z_NT / 32);
      v[u] = (z < nz && q < nxy) ? in[(long)z * nxy + q] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int z = z0 + u * (Z_NT / 32);
      if (z < rows) D[z * Z_P + lane] = v[u];
    }
  }
  __syncthreads();
  auto butterfly = [&]() {
    for (int z = tid >> 5; z < nz / 2; z += Z_NT / 32) {
      double* a = D + z * Z_P + lane;
      double* b = D + (nz - 1 - z) * Z_P + lane;
      const double p = *a, r = *b;
      *a = p + r;
      *b = p - r;
    }
  };
  butterfly();
  __syncthreads();
  const int part = warp >> 2, size = part ? A.ho : A.he;
  const double* Mp = M + (size_t)part * A.kp * A.pm;
  const int rt = A.kp / 8, rq = (rt + 3) / 4, r0 = (warp & 3) * rq, nr = min(rq, rt - r0);
  const int nks = (size + 3) / 4;
  double acc[2][4][2];
  if (nr > 0)
    spec_mm<2, 4>(nks, nr, 4, [&](int i, int ks) { return Mp + (4 * ks + lk) * A.pm + 8 * (r0 + i) + l4; },
                  [&](int j, int ks) {
                    const int k = 4 * ks + lk;
                    return D + (part ? max(0, nz - 1 - k) : k) * Z_P + 8 * j + l4;
                  }, acc);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = 8 * (r0 + i) + l4, col = 8 * j + 2 * lk + h;
        if (i < nr && n < size) {
          const int c = part ? A.he + n : n;
          const int qq = min(q0 + col, nxy - 1);
          D[c * Z_P + col] = acc[i][j][h] / ((X.lam[qq % nx] + Y.lam[qq / nx]) + A.lam[c]);
        }
      }
  __syncthreads();
  if (nr > 0)
    spec_mm<2, 4>(nks, nr, 4, [&](int i, int ks) { return Mp + (8 * (r0 + i) + l4) * A.pm + 4 * ks + lk; },
                  [&](int j, int ks) { return D + ((part ? A.he : 0) + 4 * ks + lk) * Z_P + 8 * j + l4; }, acc);
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int n = 8 * (r0 + i) + l4;
        if (i < nr && n < size) D[(part ? nz - 1 - n : n) * Z_P + 8 * j + 2 * lk + h] = acc[i][j][h];
      }
  __syncthreads();
  butterfly();
  __syncthreads();
  if (q < nxy)
    for (int z = tid >> 5; z < nz; z += Z_NT / 32) out[(long)z * nxy + q] = D[z * Z_P + lane];
}

static int spec_setup(psc_ctx* ctx) {
  if (ctx->spec_S[0]) return 0;
  const int dims[3] = {ctx->nx, ctx->ny, ctx->nz};
  for (int a = 0; a < 3; ++a) {
    const int m = dims[a], he = (m + 1) / 2;
    const int kp = 8 * ((he + 7) / 8), pm = round_pitch(kp);
    std::vector<double> M(2 * (size_t)kp * pm, 0.0), lam(m);
    const double f = std::sqrt(2.0 / (m + 1));
    for (int part = 0; part < 2; ++part) {
      const int size = part ? m / 2 : he;
      for (int j = 0; j < size; ++j)
        for (int c = 0; c < size; ++c) {
          const int k = 2 * c + part;
          M[((size_t)part * kp + j) * pm + c] = f * std::sin(M_PI * (double)(j + 1) * (k + 1) / (m + 1));
        }
      for (int c = 0; c < size; ++c) {
        const double th = M_PI * (2 * c + part + 1) / (m + 1);
        double v = ctx->lap_c0 / 3.0;
        for (int d = 1; d <= 4; ++d) v += 2.0 * ctx->lap_c[d - 1] * std::cos(d * th);
        lam[part ? he + c : c] = v;
      }
    }
    PSC_CUDA(ctx, psc_dmalloc(&ctx->spec_lam[a], lam.size() * sizeof(double)));
    PSC_CUDA(ctx, cudaMemcpy(ctx->spec_lam[a], lam.data(), lam.size() * sizeof(double), cudaMemcpyHostToDevice));
    PSC_CUDA(ctx, psc_dmalloc(&ctx->spec_S[a], M.size() * sizeof(double)));
    PSC_CUDA(ctx, cudaMemcpy(ctx->spec_S[a], M.data(), M.size() * sizeof(double), cudaMemcpyHostToDevice));
  }
  if (!ctx->spec_tmp) PSC_CUDA(ctx, psc_dmalloc(&ctx->spec_tmp, ctx->n * sizeof(double)));
  return 0;
}

static SpecAxis spec_axis(const psc_ctx* ctx, int a) {
  SpecAxis s;
  s.m = a == 0 ? ctx->nx : (a == 1 ? ctx->ny : ctx->nz);
  s.he = (s.m + 1) / 2;
  s.ho = s.m / 2;
  s.kp = 8 * ((s.he + 7) / 8);
  s.pm = round_pitch(s.kp);
  s.M = ctx->spec_S[a];
  s.lam = ctx->spec_lam[a];
  return s;
}

// z = M r.  In a solve (sc): `x` set: the CG step is taken while r is loaded
// (r, x updated; part: the partials of p.Ap); zr: the planes' sums of z r.
static int spec_apply(psc_ctx* ctx, double* r, double* z, const double* sc, double* x, const double* p,
                      const double* ap, const double* part, int npart, double* zr, cudaStream_t st) {
  XyArgs P;
  P.X = spec_axis(ctx, 0);
  P.Y = spec_axis(ctx, 1);
  const SpecAxis Z = spec_axis(ctx, 2);
  P.same = ctx->nx == ctx->ny;
  if (P.same) P.Y.M = P.X.M;
  P.rows = 8 * ((ctx->ny + 7) / 8);
  P.pd = round_pitch(std::max(8 * ((ctx->nx + 7) / 8), P.X.kp));
  P.sc = sc;
  P.r = r; P.x = x; P.p = p; P.ap = ap; P.part = part; P.npart = npart; P.zr = nullptr;
  double* t = ctx->spec_tmp;
  const int xy_smem = (int)(((size_t)P.rows * P.pd +
                             2 * std::max((size_t)P.X.kp * P.X.pm, (size_t)P.Y.kp * P.Y.pm)) * sizeof(double));
  PSC_CUDA(ctx, psc_smem_optin(k_spec_xy<true>));
  PSC_CUDA(ctx, psc_smem_optin(k_spec_xy<false>));
  P.in = r;
  P.out = t;
  k_spec_xy<true><<<ctx->nz, XY_NT, xy_smem, st>>>(P);
  PSC_LAUNCH_CHECK(ctx);
  const int zrows = std::max(8 * ((ctx->nz + 7) / 8), Z.kp);
  const int z_smem = (int)(((size_t)zrows * Z_P + 2 * (size_t)Z.kp * Z.pm) * sizeof(double));
  PSC_CUDA(ctx, psc_smem_optin(k_spec_z));
  k_spec_z<<<psc_div_up((long)ctx->nx * ctx->ny, Z_W), Z_NT, z_smem, st>>>(t, t, P.X, P.Y, Z, zrows, sc);
  PSC_LAUNCH_CHECK(ctx);
  P.in = t;
  P.out = z;
  P.x = nullptr;
  P.zr = zr;
  k_spec_xy<false><<<ctx->nz, XY_NT, xy_smem, st>>>(P);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

extern "C" int psc_poisson_precond(psc_ctx* ctx, const double* r, double* z, void* stream) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, r && z && r != z, "poisson_precond: bad arguments");
  PSC_REQUIRE(ctx, ctx->nx <= SP_MAXM && ctx->ny <= SP_MAXM && ctx->nz <= SP_MAXM,
              "poisson preconditioner: grid dimension above 128");
  if (spec_setup(ctx)) return 1;
  return spec_apply(ctx, const_cast<double*>(r), z, nullptr, nullptr, nullptr, nullptr, nullptr, 0, nullptr,
                    (cudaStream_t)stream);
}

// ---------------------------------------------------------------------------
// preconditioned CG
// ---------------------------------------------------------------------------
constexpr int PCG_NT = 256;

// End of an iteration: ro1 = z.r from the planes' sums (every CTA adds them
// in the same order), p = z + (ro1 / ro) p, the iteration count and whether
// another iteration follows.  first: the start of the solve (p = z already;
// the tolerance is set).  sc is read by every CTA before the last one to
// finish writes it.
__global__ void __launch_bounds__(PCG_NT)
k_pcg_dir(const double* __restrict__ z, double* __restrict__ p, long n, const double* __restrict__ zr, int nz,
          int first, int maxit, double tol, double* sc, unsigned int* ticket) {
  __shared__ double sh[PCG_NT / 32];
  __shared__ double bc;
  // (read before the barriers below: the last CTA may write sc once every
  // CTA's first thread has passed them)
  const bool active = first || sc[SC_ACTIVE] != 0.0;
  const double ro = first ? 0.0 : sc[SC_RO1];
  double s = 0.0;
  if (active) {
    for (int i = threadIdx.x; i < nz; i += PCG_NT) s += zr[i];
    s = psc_block_sum<double, PCG_NT>(s, sh);
    if (threadIdx.x == 0) bc = s;
    __syncthreads();
    s = bc;
    if (!first) {
      const double bet = s / ro;
      for (long i = blockIdx.x * (long)PCG_NT + threadIdx.x; i < n; i += (long)gridDim.x * PCG_NT)
        p[i] = z[i] + bet * p[i];
    }
  }
  if (!active) return;   // the same in every CTA
  if (!psc_last_block(ticket)) return;
  if (threadIdx.x == 0) {
    const double its = first ? 0.0 : sc[SC_ITS] + 1.0;
    const double tol1 = first ? tol * tol * s : sc[SC_TOL1];
    sc[SC_RO] = ro;
    sc[SC_RO1] = s;
    sc[SC_TOL1] = tol1;
    sc[SC_ITS] = its;
    sc[SC_ACTIVE] = (its < maxit && s > tol1) ? 1.0 : 0.0;
  }
}

extern "C" int psc_pcg_poisson_prec(psc_ctx* ctx, const double* rhs, double* x, int maxit, double tol, int* its_out,
                                    void* stream) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, rhs && x && maxit >= 0, "pcg_prec: bad arguments");
  PSC_REQUIRE(ctx, ctx->nx <= SP_MAXM && ctx->ny <= SP_MAXM && ctx->nz <= SP_MAXM,
              "poisson preconditioner: grid dimension above 128");
  cudaStream_t st = (cudaStream_t)stream;
  if (spec_setup(ctx)) return 1;
  const long n = ctx->n;
  if (!ctx->cg_p2) PSC_CUDA(ctx, psc_dmalloc(&ctx->cg_p2, n * sizeof(double)));
  double* r = ctx->cg_r;
  double* p = ctx->cg_p;
  double* ap = ctx->cg_ap;
  double* z = ctx->cg_p2;
  double* sc = ctx->scalars + 88;      // this solve's state (SC_*)
  // partials of the fused stencil, one per block of its launch, then the planes' z.r
  const int nst = std::max(PSC_RED_BLOCKS, psc_stencil_blocks(ctx, 1));
  const int need = nst + SP_MAXM;
  if (2 * ctx->cg_part_cap < need) {
    psc_dfree(ctx->cg_part);
    ctx->cg_part = nullptr;
    ctx->cg_part_cap = 0;
    PSC_CUDA(ctx, psc_dmalloc(&ctx->cg_part, 2 * (size_t)need * sizeof(double)));
    ctx->cg_part_cap = need;
  }
  double* zr = ctx->cg_part + nst;
  const int nb = 148 * 4;
  // r = rhs - A x; z = M r; p = z; ro1 = z.r
  int rc = psc_laplacian_fused(ctx, x, rhs, r, -1.0, 0.0, 1.0, nullptr, nullptr, st);
  if (rc) return rc;
  rc = spec_apply(ctx, r, p, nullptr, nullptr, nullptr, nullptr, nullptr, 0, zr, st);
  if (rc) return rc;
  k_pcg_dir<<<1, PCG_NT, 0, st>>>(p, p, n, zr, ctx->nz, 1, maxit, tol, sc, psc_ticket(ctx));
  PSC_LAUNCH_CHECK(ctx);
  int queued = 0, its = 0;
  bool active = maxit > 0;
  while (active) {
    // these solves take two to four iterations: three are queued before the
    // state is first read, then two at a time (an iteration queued in vain
    // costs five empty launches, a read in between about as much as one more)
    const int batch = std::min(maxit - queued, queued == 0 ? 3 : 2);
    for (int b = 0; b < batch; ++b) {
      int nblk = 0;
      rc = psc_laplacian_fused(ctx, p, nullptr, ap, 1.0, 0.0, 0.0, ctx->cg_part, &nblk, st, sc + SC_ACTIVE);
      if (rc) return rc;
      rc = spec_apply(ctx, r, z, sc, x, p, ap, ctx->cg_part, nblk, zr, st);
      if (rc) return rc;
      k_pcg_dir<<<nb, PCG_NT, 0, st>>>(z, p, n, zr, ctx->nz, 0, maxit, tol, sc, psc_ticket(ctx));
      PSC_LAUNCH_CHECK(ctx);
    }
    queued += batch;
    PSC_CUDA(ctx, cudaMemcpyAsync(ctx->host_scalars + 88, sc, 5 * sizeof(double), cudaMemcpyDeviceToHost, st));
    PSC_CUDA(ctx, cudaStreamSynchronize(st));
    its = (int)ctx->host_scalars[88 + SC_ITS];
    active = ctx->host_scalars[88 + SC_ACTIVE] != 0.0;
  }
  if (maxit == 0) PSC_CUDA(ctx, cudaStreamSynchronize(st));
  if (its_out) *its_out = its;
  return 0;
}
