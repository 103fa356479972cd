// Kleinman-Bylander nonlocal term in factored form and its setup.
//
// V_nl = sum_a sum_m u_am u_am^T / xint_a  (V_ion/pseudoNL_original.py:187-206)
// is applied as  Y[idx] += alpha * sum_a sum_m u_am * (w_a * u_am . X[idx]),
// w_a = 1/xint_a = h^3 / Zvalue_a, never forming the n_a x n_a blocks.
//   project: one warp per (atom, column) reduces w_a * U_a^T X (3 values)
//            over the ball with a fixed shuffle tree;
//   scatter: one thread per (touched grid point, group of 8 columns) adds
//            the sum over the balls covering that point, in atom order.  No
//            atomics, so the result is bitwise reproducible.
#include "psc_internal.cuh"
#include "../../include/psc.h"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

// Projection: one CTA per (atom, group of NL_KC columns), one warp per
// column.  The ball's grid indices and u values are staged in shared memory
// NL_STAGE points at a time; lane l of a warp takes points l, l + 32, ...
// (NL_UNROLL gathers in flight), then a fixed shuffle tree sums the lanes,
// so the result is reproducible.  Many warps per SM keep enough gathers in
// flight for HBM, which a few threads per ball point could not.
constexpr int NL_KC = 16;       // columns (warps) per projection CTA
constexpr int NL_STAGE = 1024;  // ball points staged per pass
constexpr int NL_UNROLL = 4;

template <typename T>
__global__ void __launch_bounds__(NL_KC * 32)
k_nl_project(const T* __restrict__ X, long ldx, int k, const int* __restrict__ atom_off,
             const int* __restrict__ idx, const T* __restrict__ u, long npts, const double* __restrict__ w,
             double* __restrict__ proj) {
  __shared__ int s_idx[NL_STAGE];
  __shared__ T s_u[3][NL_STAGE];
  const int a = blockIdx.x;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int c = blockIdx.y * NL_KC + wid;
  const int lo = atom_off[a], hi = atom_off[a + 1];
  const T* Xc = X + (long)min(c, k - 1) * ldx;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  for (int b = lo; b < hi; b += NL_STAGE) {
    const int nb = min(NL_STAGE, hi - b);
    __syncthreads();
    for (int i = threadIdx.x; i < nb; i += NL_KC * 32) {
      s_idx[i] = idx[b + i];
      s_u[0][i] = u[b + i];
      s_u[1][i] = u[npts + b + i];
      s_u[2][i] = u[2 * npts + b + i];
    }
    __syncthreads();
    for (int i0 = lane; i0 < nb; i0 += 32 * NL_UNROLL) {
      double xv[NL_UNROLL];
#pragma unroll
      for (int r = 0; r < NL_UNROLL; ++r) {
        const int i = i0 + 32 * r;
        xv[r] = i < nb ? (double)Xc[s_idx[i]] : 0.0;
      }
#pragma unroll
      for (int r = 0; r < NL_UNROLL; ++r) {
        const int i = i0 + 32 * r;
        if (i < nb) {
          s0 += (double)s_u[0][i] * xv[r];
          s1 += (double)s_u[1][i] * xv[r];
          s2 += (double)s_u[2][i] * xv[r];
        }
      }
    }
  }
  s0 = psc_warp_sum(s0);
  s1 = psc_warp_sum(s1);
  s2 = psc_warp_sum(s2);
  if (lane == 0 && c < k) {
    const double wa = w[a];
    proj[((long)a * 3 + 0) * k + c] = wa * s0;
    proj[((long)a * 3 + 1) * k + c] = wa * s1;
    proj[((long)a * 3 + 2) * k + c] = wa * s2;
  }
}

// Scatter: one thread per (touched grid point, group of NL_SC columns); the
// entries covering the point and their u values are read once for every
// column of the group, the group's Y values are loaded before the sums and
// stored after them, and each column's sum runs over the entries in atom
// order (no atomics, so the result is bitwise reproducible).
constexpr int NL_SC = 8;
template <typename T>
__global__ void __launch_bounds__(256)
k_nl_scatter(T* __restrict__ Y, long ldy, int k, long ntouched, const int* __restrict__ t_idx,
             const int* __restrict__ t_off, const int* __restrict__ t_ent, const int* __restrict__ pt_atom,
             const T* __restrict__ u, long npts, const double* __restrict__ proj, const double* __restrict__ coef,
             double ha) {
  const int ngrp = (k + NL_SC - 1) / NL_SC;
  const long t = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (t >= ntouched * (long)ngrp) return;
  const double alpha = coef ? coef[0] : ha;
  const long pt = t % ntouched;
  const int c0 = (int)(t / ntouched) * NL_SC;
  const int nc = min(NL_SC, k - c0);
  T* yp = Y + (long)t_idx[pt] + (long)c0 * ldy;
  T yv[NL_SC];
#pragma unroll
  for (int c = 0; c < NL_SC; ++c) yv[c] = c < nc ? yp[(long)c * ldy] : T(0);
  double s[NL_SC];
#pragma unroll
  for (int c = 0; c < NL_SC; ++c) s[c] = 0.0;
  for (int e = t_off[pt]; e < t_off[pt + 1]; ++e) {
    const int p = t_ent[e];
    const double u0 = (double)u[p], u1 = (double)u[npts + p], u2 = (double)u[2 * npts + p];
    const double* pr = proj + (long)pt_atom[p] * 3 * k + c0;
#pragma unroll
    for (int c = 0; c < NL_SC; ++c)
      if (c < nc) s[c] += u0 * pr[c] + u1 * pr[k + c] + u2 * pr[2 * k + c];
  }
#pragma unroll
  for (int c = 0; c < NL_SC; ++c)
    if (c < nc) yp[(long)c * ldy] = (T)((double)yv[c] + alpha * s[c]);
}

int psc_ensure_proj(psc_ctx* ctx, int k) {
  size_t need = (size_t)std::max(ctx->nl_atoms, 1) * 3 * k * sizeof(double);
  if (need > ctx->nl_proj_bytes) {
    psc_dfree(ctx->nl_proj);
    ctx->nl_proj = nullptr;
    PSC_CUDA(ctx, psc_dmalloc(&ctx->nl_proj, need));
    ctx->nl_proj_bytes = need;
  }
  return 0;
}

int psc_nl_project(psc_ctx* ctx, int dtype, const void* X, long ldx, int k, cudaStream_t st) {
  if (psc_ensure_proj(ctx, k)) return 1;
  dim3 grid(ctx->nl_atoms, (k + NL_KC - 1) / NL_KC);
  if (dtype == PSC_F64)
    k_nl_project<double><<<grid, NL_KC * 32, 0, st>>>((const double*)X, ldx, k, ctx->nl_atom_off, ctx->nl_idx,
                                                       ctx->nl_u64, ctx->nl_points, ctx->nl_w,
                                                       (double*)ctx->nl_proj);
  else
    k_nl_project<float><<<grid, NL_KC * 32, 0, st>>>((const float*)X, ldx, k, ctx->nl_atom_off, ctx->nl_idx,
                                                      ctx->nl_u32, ctx->nl_points, ctx->nl_w,
                                                      (double*)ctx->nl_proj);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

int psc_nl_scatter(psc_ctx* ctx, int dtype, void* Y, long ldy, int k, const double* coef, double a,
                   cudaStream_t st) {
  const long total = ctx->nl_touched * (long)((k + NL_SC - 1) / NL_SC);
  if (total == 0) return 0;
  PSC_REQUIRE(ctx, (total + 255) / 256 <= INT32_MAX, "nl_scatter: too many touched points x columns");
  const int nb = (int)((total + 255) / 256);   // one (touched point, column group) per thread
  if (dtype == PSC_F64)
    k_nl_scatter<double><<<nb, 256, 0, st>>>((double*)Y, ldy, k, ctx->nl_touched, ctx->nl_t_idx,
                                              ctx->nl_t_off, ctx->nl_t_ent, ctx->nl_point_atom, ctx->nl_u64,
                                              ctx->nl_points, (const double*)ctx->nl_proj, coef, a);
  else
    k_nl_scatter<float><<<nb, 256, 0, st>>>((float*)Y, ldy, k, ctx->nl_touched, ctx->nl_t_idx, ctx->nl_t_off,
                                             ctx->nl_t_ent, ctx->nl_point_atom, ctx->nl_u32, ctx->nl_points,
                                             (const double*)ctx->nl_proj, coef, a);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

void psc_free_projectors(psc_ctx* ctx) {
  psc_dfree(ctx->nl_block); psc_dfree(ctx->nl_proj);
  ctx->nl_block = nullptr;
  ctx->nl_atom_off = ctx->nl_idx = ctx->nl_t_idx = ctx->nl_t_off = ctx->nl_t_ent = ctx->nl_point_atom = nullptr;
  ctx->nl_u64 = nullptr; ctx->nl_u32 = nullptr; ctx->nl_w = nullptr; ctx->nl_proj = nullptr;
  ctx->nl_proj_bytes = 0;
  ctx->nl_atoms = 0; ctx->nl_points = 0; ctx->nl_touched = 0;
}

int psc_nl_apply_mask(psc_ctx* ctx, cudaStream_t st);


// setup.cu
int psc_nl_box_distances(psc_ctx* ctx, int nbox, const int* box_dev /* [nbox][8] */, const double* xyz_dev,
                         const double* rcut_dev, long total, const long* box_start_dev, double radius,
                         unsigned char* mask_dev, cudaStream_t st);
int psc_nl_eval_u(psc_ctx* ctx, long npts, const int* idx_dev, const int* pt_atom_dev,
                  const int* atom_species_dev, const double* xyz_dev, double radius, double* u_dev,
                  cudaStream_t st);

// ---------------------------------------------------------------------------
// Building the tables on the device.  The ball points of an atom are the
// points of its window box that the mask keeps, in window order; the touched
// points are the distinct grid points in ascending order, each with its ball
// points in ascending (atom) order.  Both are compactions by prefix sums over
// blocks of SC_B values; the host only learns the boxes' counts and the two
// totals.  (On the host the compaction, the sort and the upload of the tables
// took 3 ms of a 7 ms setup.)
// ---------------------------------------------------------------------------
constexpr int SC_T = 256, SC_V = 8, SC_B = SC_T * SC_V;

// exclusive prefix sum of one int per thread over the CTA; *total = the sum
__device__ __forceinline__ int block_scan(int v, int* sh /* [SC_T / 32 + 1] */, int* total) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  __syncthreads();
  if (lane == 31) sh[w] = x;
  __syncthreads();
  int before = 0, sum = 0;
#pragma unroll
  for (int i = 0; i < SC_T / 32; ++i) {
    if (i < w) before += sh[i];
    sum += sh[i];
  }
  *total = sum;
  return before + x - v;
}

// per block of values: how many are positive, and their sum
template <typename V>
__global__ void __launch_bounds__(SC_T)
k_scan_count(const V* __restrict__ v, long n, int* __restrict__ pos, int* __restrict__ sum) {
  __shared__ int sh[SC_T / 32 + 1];
  const long i0 = blockIdx.x * (long)SC_B + threadIdx.x * SC_V;
  int p = 0, s = 0;
#pragma unroll
  for (int j = 0; j < SC_V; ++j)
    if (i0 + j < n) {
      const int x = (int)v[i0 + j];
      p += x > 0;
      s += x;
    }
  int tp, ts;
  block_scan(p, sh, &tp);
  block_scan(s, sh, &ts);
  if (threadIdx.x == 0) {
    pos[blockIdx.x] = tp;
    sum[blockIdx.x] = ts;
  }
}

// exclusive sums of the blocks' counts in place, totals at [nb] (one CTA)
__global__ void __launch_bounds__(SC_T) k_scan_top(int* pos, int* sum, int nb) {
  __shared__ int sh[SC_T / 32 + 1];
  int cp = 0, cs = 0;
  for (int b0 = 0; b0 < nb; b0 += SC_T) {
    const int b = b0 + threadIdx.x;
    const int p = b < nb ? pos[b] : 0, s = b < nb ? sum[b] : 0;
    int tp, ts;
    const int ep = block_scan(p, sh, &tp), es = block_scan(s, sh, &ts);
    if (b < nb) {
      pos[b] = cp + ep;
      sum[b] = cs + es;
    }
    cp += tp;
    cs += ts;
  }
  if (threadIdx.x == 0) {
    pos[nb] = cp;
    sum[nb] = cs;
  }
}

// ball points before each box (one warp per box; box_off[nbox] = all)
__global__ void k_box_offsets(const unsigned char* __restrict__ mask, const long* __restrict__ start, int nbox,
                              const int* __restrict__ pos, int nb, int* __restrict__ box_off) {
  const int b = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (b > nbox) return;
  int c = 0;
  if (b < nbox) {
    const long blk = start[b] / SC_B;
    for (long t = blk * SC_B + lane; t < start[b]; t += 32) c += mask[t] != 0;
    c = psc_warp_sum(c);
    c += pos[blk];
  } else {
    c = pos[nb];
  }
  if (lane == 0) box_off[b] = c;
}

// the kept points in window order: grid index, table atom, caller's atom
__global__ void __launch_bounds__(SC_T)
k_ball_points(const unsigned char* __restrict__ mask, long total, const int* __restrict__ pos, int nbox,
              const int* __restrict__ box, const long* __restrict__ start, const int* __restrict__ atom_of_box, int nx,
              int ny, int* __restrict__ idx, int* __restrict__ pt_atom, int* __restrict__ pt_orig) {
  __shared__ int sh[SC_T / 32 + 1];
  const long i0 = blockIdx.x * (long)SC_B + threadIdx.x * SC_V;
  unsigned int keep = 0;
#pragma unroll
  for (int j = 0; j < SC_V; ++j)
    if (i0 + j < total && mask[i0 + j]) keep |= 1u << j;
  int all;
  int at = pos[blockIdx.x] + block_scan(__popc(keep), sh, &all);
  for (int j = 0; j < SC_V; ++j) {
    if (!(keep >> j & 1u)) continue;
    const long t = i0 + j;
    int lo = 0, hi = nbox - 1;
    while (lo < hi) {   // last box whose start <= t
      const int mid = (lo + hi + 1) >> 1;
      if (start[mid] <= t) lo = mid;
      else hi = mid - 1;
    }
    const int* b = box + 8 * lo;
    const long li = t - start[lo];
    const int ni = b[1] - b[0] + 1, nj = b[3] - b[2] + 1;
    const int i = b[0] - 1 + (int)(li % ni), jj = b[2] - 1 + (int)((li / ni) % nj);
    const int k = b[4] - 1 + (int)(li / ((long)ni * nj));
    idx[at] = i + nx * (jj + k * ny);
    pt_atom[at] = atom_of_box[lo];
    pt_orig[at] = b[6];
    ++at;
  }
}

__global__ void k_cover_count(const int* __restrict__ idx, long npts, int* __restrict__ cover) {
  const long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (p < npts) atomicAdd(cover + idx[p], 1);
}

// touched points: grid index and first entry; cover[g] becomes that entry, the
// fill position of point g
__global__ void __launch_bounds__(SC_T)
k_touched(int* __restrict__ cover, long n, const int* __restrict__ pos, const int* __restrict__ sum, int nb,
          int* __restrict__ t_idx, int* __restrict__ t_off) {
  __shared__ int sh[SC_T / 32 + 1];
  const long i0 = blockIdx.x * (long)SC_B + threadIdx.x * SC_V;
  int c[SC_V], p = 0, s = 0;
#pragma unroll
  for (int j = 0; j < SC_V; ++j) {
    c[j] = i0 + j < n ? cover[i0 + j] : 0;
    p += c[j] > 0;
    s += c[j];
  }
  int all;
  int ti = pos[blockIdx.x] + block_scan(p, sh, &all);
  int off = sum[blockIdx.x] + block_scan(s, sh, &all);
#pragma unroll
  for (int j = 0; j < SC_V; ++j)
    if (c[j] > 0) {
      t_idx[ti] = (int)(i0 + j);
      t_off[ti] = off;
      cover[i0 + j] = off;
      ++ti;
      off += c[j];
    }
  if (blockIdx.x == 0 && threadIdx.x == 0) t_off[pos[nb]] = sum[nb];
}

__global__ void k_touched_fill(const int* __restrict__ idx, long npts, int* __restrict__ cover,
                               int* __restrict__ t_ent) {
  const long p = blockIdx.x * (long)blockDim.x + threadIdx.x;
  if (p < npts) t_ent[atomicAdd(cover + idx[p], 1)] = (int)p;
}

// each point's few entries in ascending order (the fill's order is arbitrary)
__global__ void k_touched_sort(const int* __restrict__ t_off, const int* __restrict__ ntouched,
                               int* __restrict__ t_ent) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= *ntouched) return;
  const int lo = t_off[t], hi = t_off[t + 1];
  for (int i = lo + 1; i < hi; ++i) {
    const int v = t_ent[i];
    int j = i - 1;
    for (; j >= lo && t_ent[j] > v; --j) t_ent[j + 1] = t_ent[j];
    t_ent[j + 1] = v;
  }
}

// Arrays gathered into one host block and uploaded by one copy; add() returns
// the array's offset (16-byte aligned) in the device block.
struct UploadBlock {
  std::vector<unsigned char> host;
  template <typename T>
  size_t add(const T* p, size_t count) {
    const size_t at = (host.size() + 15) & ~size_t(15);
    host.resize(at + count * sizeof(T));
    if (p && count) std::memcpy(host.data() + at, p, count * sizeof(T));
    return at;
  }
};

// device offsets of the arrays that only the device writes
struct Carve {
  size_t at;
  size_t take(size_t bytes) {
    at = (at + 15) & ~size_t(15);
    const size_t o = at;
    at += bytes;
    return o;
  }
};

// Build the projector tables for the atoms (species ids and coordinates in
// bohr, species-major order as in pseudoNL_original.py:60-115).
extern "C" int psc_projector_setup(psc_ctx* ctx, int natoms, const int* species, const double* xyz,
                                   double radius, void* stream) {
  if (!ctx) return 2;
  PSC_REQUIRE(ctx, natoms >= 0, "projector_setup: natoms < 0");
  cudaStream_t st = (cudaStream_t)stream;
  psc_free_projectors(ctx);
  if (natoms == 0) return 0;
  const double h = ctx->h;
  const int nx = ctx->nx, ny = ctx->ny, nz = ctx->nz;
  // per-atom window boxes (1-based inclusive ranges), pseudoNL_original.py:122-138
  std::vector<int> box;          // [imin, imax, jmin, jmax, kmin, kmax, atom, species]
  std::vector<long> start;
  long total = 0;
  for (int a = 0; a < natoms; ++a) {
    const int sp = species[a];
    PSC_REQUIRE(ctx, sp >= 0 && sp < (int)ctx->species.size() && ctx->species[sp].valid,
                "projector_setup: species table missing");
    const double R = ctx->species[sp].rcut;
    const double xa = xyz[3 * a], ya = xyz[3 * a + 1], za = xyz[3 * a + 2];
    // Python round() is round-half-even, as is nearbyint in the default mode.
    const int i0 = (int)std::nearbyint((xa + radius) / h + 1);
    const int j0 = (int)std::nearbyint((ya + radius) / h + 1);
    const int k0 = (int)std::nearbyint((za + radius) / h + 1);
    const int span = (int)std::nearbyint(R / h);
    int b[8] = {std::max(1, i0 - span), std::min(nx, i0 + span), std::max(1, j0 - span),
                std::min(ny, j0 + span), std::max(1, k0 - span), std::min(nz, k0 + span), a, sp};
    if (b[0] > b[1] || b[2] > b[3] || b[4] > b[5]) continue;
    box.insert(box.end(), b, b + 8);
    start.push_back(total);
    total += (long)(b[1] - b[0] + 1) * (b[3] - b[2] + 1) * (b[5] - b[4] + 1);
  }
  const int nbox = (int)start.size();
  if (nbox == 0) return 0;
  std::vector<double> rcut(nbox);
  for (int i = 0; i < nbox; ++i) rcut[i] = ctx->species[box[8 * i + 7]].rcut;
  UploadBlock in;
  const size_t o_box = in.add(box.data(), box.size()), o_start = in.add(start.data(), start.size());
  const size_t o_xyz = in.add(xyz, 3 * (size_t)natoms), o_asp = in.add(species, natoms);
  const size_t o_rc = in.add(rcut.data(), rcut.size());
  // scratch: the inputs, the mask, block counts of the mask and of the grid,
  // the boxes' offsets, the grid's cover counts
  const long n = ctx->n;
  const int nbm = psc_div_up(total, SC_B), nbg = psc_div_up(n, SC_B);
  Carve c{in.host.size()};
  const size_t o_mask = c.take(total), o_mpos = c.take((nbm + 1) * sizeof(int)), o_msum = c.take((nbm + 1) * sizeof(int));
  const size_t o_gpos = c.take((nbg + 1) * sizeof(int)), o_gsum = c.take((nbg + 1) * sizeof(int));
  const size_t o_boff = c.take((nbox + 1) * sizeof(int)), o_aob = c.take(nbox * sizeof(int));
  const size_t o_cover = c.take(n * sizeof(int));
  unsigned char* d = nullptr;
  PSC_CUDA(ctx, psc_dmalloc(&d, c.at));
  struct FreeLater {
    void* p = nullptr;
    ~FreeLater() { psc_dfree(p); }
  } scratch{d}, orig;
  PSC_CUDA(ctx, cudaMemcpyAsync(d, in.host.data(), in.host.size(), cudaMemcpyHostToDevice, st));
  const int* box_d = reinterpret_cast<const int*>(d + o_box);
  const long* start_d = reinterpret_cast<const long*>(d + o_start);
  const double* xyz_d = reinterpret_cast<const double*>(d + o_xyz);
  const int* asp_d = reinterpret_cast<const int*>(d + o_asp);
  unsigned char* mask_d = d + o_mask;
  auto ints = [&](size_t o) { return reinterpret_cast<int*>(d + o); };
  if (psc_nl_box_distances(ctx, nbox, box_d, xyz_d, reinterpret_cast<const double*>(d + o_rc), total, start_d, radius,
                           mask_d, st))
    return 1;
  k_scan_count<unsigned char><<<nbm, SC_T, 0, st>>>(mask_d, total, ints(o_mpos), ints(o_msum));
  PSC_LAUNCH_CHECK(ctx);
  k_scan_top<<<1, SC_T, 0, st>>>(ints(o_mpos), ints(o_msum), nbm);
  PSC_LAUNCH_CHECK(ctx);
  k_box_offsets<<<psc_div_up(nbox + 1, 8), 256, 0, st>>>(mask_d, start_d, nbox, ints(o_mpos), nbm, ints(o_boff));
  PSC_LAUNCH_CHECK(ctx);
  std::vector<int> box_off(nbox + 1);
  PSC_CUDA(ctx, cudaMemcpyAsync(box_off.data(), ints(o_boff), (nbox + 1) * sizeof(int), cudaMemcpyDeviceToHost, st));
  PSC_CUDA(ctx, cudaStreamSynchronize(st));
  // boxes without a kept point have no atom in the tables
  std::vector<int> atom_off{0}, atom_of_box(nbox, 0);
  std::vector<double> w;
  for (int bi = 0; bi < nbox; ++bi) {
    if (box_off[bi + 1] == box_off[bi]) continue;
    atom_of_box[bi] = (int)w.size();
    w.push_back(1.0 / (ctx->species[box[8 * bi + 7]].zvalue / (h * h * h)));
    atom_off.push_back(box_off[bi + 1]);
  }
  const int nla = (int)w.size();
  const long npts = box_off[nbox];
  if (nla == 0) return 0;
  UploadBlock tab;
  const size_t o_off = tab.add(atom_off.data(), atom_off.size()), o_w = tab.add(w.data(), w.size());
  Carve tc{tab.host.size()};
  const size_t ib = npts * sizeof(int);
  const size_t o_idx = tc.take(ib), o_pa = tc.take(ib), o_ti = tc.take(ib), o_to = tc.take(ib + sizeof(int));
  const size_t o_te = tc.take(ib), o_u64 = tc.take(3 * npts * sizeof(double)), o_u32 = tc.take(3 * npts * sizeof(float));
  unsigned char* blk = nullptr;
  PSC_CUDA(ctx, psc_dmalloc(&blk, tc.at));
  ctx->nl_block = blk;
  ctx->nl_atom_off = reinterpret_cast<int*>(blk + o_off);
  ctx->nl_idx = reinterpret_cast<int*>(blk + o_idx);
  ctx->nl_point_atom = reinterpret_cast<int*>(blk + o_pa);
  ctx->nl_w = reinterpret_cast<double*>(blk + o_w);
  ctx->nl_t_idx = reinterpret_cast<int*>(blk + o_ti);
  ctx->nl_t_off = reinterpret_cast<int*>(blk + o_to);
  ctx->nl_t_ent = reinterpret_cast<int*>(blk + o_te);
  ctx->nl_u64 = reinterpret_cast<double*>(blk + o_u64);
  ctx->nl_u32 = reinterpret_cast<float*>(blk + o_u32);
  PSC_CUDA(ctx, psc_dmalloc(&orig.p, ib));
  int* pt_orig = static_cast<int*>(orig.p);
  PSC_CUDA(ctx, cudaMemcpyAsync(blk, tab.host.data(), tab.host.size(), cudaMemcpyHostToDevice, st));
  PSC_CUDA(ctx, cudaMemcpyAsync(ints(o_aob), atom_of_box.data(), nbox * sizeof(int), cudaMemcpyHostToDevice, st));
  PSC_CUDA(ctx, cudaMemsetAsync(ints(o_cover), 0, n * sizeof(int), st));
  k_ball_points<<<nbm, SC_T, 0, st>>>(mask_d, total, ints(o_mpos), nbox, box_d, start_d, ints(o_aob), nx, ny,
                                      ctx->nl_idx, ctx->nl_point_atom, pt_orig);
  PSC_LAUNCH_CHECK(ctx);
  const int nbp = psc_div_up(npts, 256);
  k_cover_count<<<nbp, 256, 0, st>>>(ctx->nl_idx, npts, ints(o_cover));
  PSC_LAUNCH_CHECK(ctx);
  k_scan_count<int><<<nbg, SC_T, 0, st>>>(ints(o_cover), n, ints(o_gpos), ints(o_gsum));
  PSC_LAUNCH_CHECK(ctx);
  k_scan_top<<<1, SC_T, 0, st>>>(ints(o_gpos), ints(o_gsum), nbg);
  PSC_LAUNCH_CHECK(ctx);
  k_touched<<<nbg, SC_T, 0, st>>>(ints(o_cover), n, ints(o_gpos), ints(o_gsum), nbg, ctx->nl_t_idx, ctx->nl_t_off);
  PSC_LAUNCH_CHECK(ctx);
  k_touched_fill<<<nbp, 256, 0, st>>>(ctx->nl_idx, npts, ints(o_cover), ctx->nl_t_ent);
  PSC_LAUNCH_CHECK(ctx);
  k_touched_sort<<<nbp, 256, 0, st>>>(ctx->nl_t_off, ints(o_gpos) + nbg, ctx->nl_t_ent);
  PSC_LAUNCH_CHECK(ctx);
  int ntouched = 0;
  PSC_CUDA(ctx, cudaMemcpyAsync(&ntouched, ints(o_gpos) + nbg, sizeof(int), cudaMemcpyDeviceToHost, st));
  int rc = psc_nl_eval_u(ctx, npts, ctx->nl_idx, pt_orig, asp_d, xyz_d, radius, ctx->nl_u64, st);
  if (!rc) rc = psc_cast(ctx, PSC_F32, ctx->nl_u64, ctx->nl_u32, 3 * npts, st);
  PSC_CUDA(ctx, cudaStreamSynchronize(st));
  ctx->nl_atoms = nla;
  ctx->nl_points = npts;
  ctx->nl_touched = ntouched;
  if (!rc) rc = psc_nl_apply_mask(ctx, st);
  PSC_CUDA(ctx, cudaStreamSynchronize(st));
  return rc;
}

// Sphere mask: the projector functions vanish at ball points outside the
// sphere (their rows and columns of V_nl are those of masked points).
__global__ void k_nl_mask(double* u64, float* u32, const int* __restrict__ idx, long npts, int nx, int ny, double h,
                          double cx, double cy, double cz, double r2) {
  for (long p = blockIdx.x * (long)blockDim.x + threadIdx.x; p < npts; p += (long)gridDim.x * blockDim.x) {
    const long g = idx[p];
    const double x = (g % nx) * h - cx, y = ((g / nx) % ny) * h - cy, z = (g / ((long)nx * ny)) * h - cz;
    if (x * x + y * y + z * z > r2)
      for (int m = 0; m < 3; ++m) {
        u64[m * npts + p] = 0.0;
        u32[m * npts + p] = 0.0f;
      }
  }
}

int psc_nl_apply_mask(psc_ctx* ctx, cudaStream_t st) {
  if (ctx->mask_r2 <= 0.0 || ctx->nl_points == 0) return 0;
  const long npts = ctx->nl_points;
  k_nl_mask<<<(int)std::min<long>(148L * 8, (npts + 255) / 256), 256, 0, st>>>(
      ctx->nl_u64, ctx->nl_u32, ctx->nl_idx, npts, ctx->nx, ctx->ny, ctx->h, ctx->mask_c[0], ctx->mask_c[1],
      ctx->mask_c[2], ctx->mask_r2);
  PSC_LAUNCH_CHECK(ctx);
  return 0;
}

// Copy the projector tables out (for checks against the reference's V_nl).
extern "C" int psc_projector_export(psc_ctx* ctx, int* atom_off, int* idx, double* u, double* w) {
  if (!ctx) return 2;
  if (ctx->nl_atoms == 0) return 0;
  if (atom_off) PSC_CUDA(ctx, cudaMemcpy(atom_off, ctx->nl_atom_off, (ctx->nl_atoms + 1) * sizeof(int), cudaMemcpyDeviceToHost));
  if (idx) PSC_CUDA(ctx, cudaMemcpy(idx, ctx->nl_idx, ctx->nl_points * sizeof(int), cudaMemcpyDeviceToHost));
  if (u) PSC_CUDA(ctx, cudaMemcpy(u, ctx->nl_u64, 3 * ctx->nl_points * sizeof(double), cudaMemcpyDeviceToHost));
  if (w) PSC_CUDA(ctx, cudaMemcpy(w, ctx->nl_w, ctx->nl_atoms * sizeof(double), cudaMemcpyDeviceToHost));
  return 0;
}
