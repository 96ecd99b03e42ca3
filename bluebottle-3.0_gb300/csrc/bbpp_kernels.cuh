// bbpp_kernels.cuh -- general-form kernels on the unscaled operator (-A),
// templated on the vector type.  The PCG iteration itself runs on the scaled
// operator in bbpp_fast.cuh; these serve the kernel-level entry points
// (SpMV, residual, the context-free residual) and the checks.
//
//  k_axpy_x       x += alpha p (PP_update_solution, src/solver_kernel.cu:864-881).
//  k_resid        r = rhs - (-A) x with (r,z), (r,r), (rhs,rhs) partials
//                 (PP_update_residual after an SpMV of phi,
//                 src/solver_kernel.cu:883-904, src/cuda_solver.cu:209-224);
//                 with rhs == NULL it writes (-A) x (kernel-level SpMV).
//
// The last CTA of every reducing kernel finishes the global sum in block
// order and updates the device state (alpha; or beta and the stopping test),
// so no scalar crosses to the host inside an iteration.
#pragma once

#include "bbpp_dev.cuh"
#include "bbpp_fast.cuh"

namespace bbpp {

constexpr int TX = 32;  // tile width (x), one warp
constexpr int TY = 8;   // tile height (y)
constexpr int HX = TX + 2;
constexpr int HY = TY + 2;
constexpr int NT = TX * TY;  // 256 threads
constexpr int HPER = (HX * HY + NT - 1) / NT;  // halo elements per thread

enum ResidMode : int { RES_INIT = 0, RES_ITER = 1, RES_CONFIRM = 2, RES_PLAIN = 3 };

__device__ __forceinline__ void load_tab(const Geo &G, double *s_tab) {
  for (int e = threadIdx.x; e < 81; e += blockDim.x) s_tab[e] = G.tab[e];
}

template <typename T>
__global__ void __launch_bounds__(NT) k_axpy_x(const Geo G, T *__restrict__ x, const T *__restrict__ p,
                                               const DevState *st) {
  if (*(volatile const int *)&st->done) return;
  const T alpha = (T)(*(volatile const double *)&st->alpha);
  const unsigned int n = (unsigned int)G.n;
  for (unsigned int c = blockIdx.x * NT + threadIdx.x; c < n; c += gridDim.x * NT) x[c] = fma(alpha, p[c], x[c]);
}

// rz + w rd^2: a wall cell's part of (r,z), as a call (see nb_adds6)
__device__ __noinline__ static double wall_rz(double rz, double w, double rd) { return fma(rd, w * rd, rz); }

// ------------------------------------------------------------ residual -----
// r = rhs - (-A) x   (rhs != NULL), or r = (-A) x  (rhs == NULL, RES_PLAIN).
// TX: type of x and rhs; TR: type of r.  Partials: (r,z), (r,r), (rhs,rhs).
// xsum (FP64, cx == cy == cz): the six neighbours, zero across solid cells and
// walls, as one exact sum on the integer pipe (xsum6).
// Bound by the FP64 pipe with FP64 adds (13 instructions a cell; 426 us at 256^3);
// with the integer sums, (r,z) as (r,r) plus the wall cells' part, and a plane's
// loads in flight while the one before is computed it takes 300 us.
template <typename TXT, typename TR, bool MASK>
__global__ void __launch_bounds__(NT) k_resid(const Geo G, const TXT *__restrict__ xin,
                                              const TXT *__restrict__ rhs, TR *__restrict__ rout,
                                              const uint8_t *__restrict__ mask, DevState *st,
                                              double *partials, int kz, int mode, int xsum) {
  __shared__ double s_tab[81];
  __shared__ TXT sp[4][HY][HX];
  __shared__ uint8_t sm[4][HY][HX + 2];
  __shared__ double s_red[3 * NT / 32];
  if (mode == RES_ITER && *(volatile int *)&st->done) return;
  load_tab(G, s_tab);
  const int tid = threadIdx.x;
  const int tx = tid & (TX - 1), ty = tid / TX;
  const int x0 = blockIdx.x * TX, y0 = blockIdx.y * TY;
  const int z0 = blockIdx.z * kz;
  const int z1 = min(z0 + kz, G.nz);
  const int nx = G.nx, ny = G.ny, nz = G.nz;
  __syncthreads();

  // the tile of a plane plus halo: loaded into registers one plane ahead (issue),
  // written to shared memory the next plane (commit)
  long long eoff[HPER];  // offset in a plane, -1 outside a wall or the tile
#pragma unroll
  for (int k = 0; k < HPER; k++) {
    const int e = tid + k * NT, ly = e / HX, lx = e - ly * HX;
    const int hx = halo_index(x0 + lx - 1, nx, G.px), hy = halo_index(y0 + ly - 1, ny, G.py);
    eoff[k] = e < HX * HY && hx >= 0 && hy >= 0 ? hx + (long long)nx * hy : -1;
  }
  TXT pv[HPER];
  uint8_t pm[HPER];
  auto issue = [&](int zr) {
    const int gz = halo_index(zr, nz, G.pz);
#pragma unroll
    for (int k = 0; k < HPER; k++) {
      pv[k] = TXT(0);
      pm[k] = 0;
      if (gz >= 0 && eoff[k] >= 0) {
        const long long c = eoff[k] + (long long)nx * ny * gz;
        pv[k] = xin[c];
        if (MASK) pm[k] = mask[c];
      }
    }
  };
  auto commit = [&](int slot) {
#pragma unroll
    for (int k = 0; k < HPER; k++) {
      const int e = tid + k * NT;
      if (e >= HX * HY) continue;
      (&sp[slot][0][0])[e] = pv[k];
      const int ly = e / HX;
      sm[slot][ly][e - ly * HX] = pm[k];
    }
  };

  double rz = 0, rr = 0, bb = 0;
  issue(z0 - 1);
  commit(0);
  issue(z0);
  commit(1);
  issue(z0 + 1);
  const TXT cx = (TXT)G.cx, cy = (TXT)G.cy, cz = (TXT)G.cz;
  const int gx = x0 + tx, gy = y0 + ty;
  const bool mine = gx < nx && gy < ny;
  const int cls_xy = mine ? (wall_count(gx, nx, G.px) + 3 * wall_count(gy, ny, G.py)) : 0;
  for (int z = z0; z < z1; z++) {
    const int sb = (z - z0) & 3, sc = (z - z0 + 1) & 3, st_ = (z - z0 + 2) & 3;
    commit(st_);
    if (z + 2 <= z1) issue(z + 2);
    const long long c = gx + (long long)nx * (gy + (long long)ny * z);
    const TXT bv = rhs && mine ? rhs[c] : TXT(0);
    __syncthreads();
    if (mine) {
      TXT pc = sp[sc][ty + 1][tx + 1];
      TXT pe = sp[sc][ty + 1][tx + 2], pw = sp[sc][ty + 1][tx];
      TXT pn = sp[sc][ty + 2][tx + 1], ps = sp[sc][ty][tx + 1];
      TXT pt = sp[st_][ty + 1][tx + 1], pb = sp[sb][ty + 1][tx + 1];
      const int cls = cls_xy + 9 * wall_count(z, nz, G.pz);
      TXT d = (TXT)s_tab[cls];
      if (MASK) {
        const bool mc = sm[sc][ty + 1][tx + 1] != 0;
        pe = (mc || sm[sc][ty + 1][tx + 2]) ? TXT(0) : pe;
        pw = (mc || sm[sc][ty + 1][tx]) ? TXT(0) : pw;
        pn = (mc || sm[sc][ty + 2][tx + 1]) ? TXT(0) : pn;
        ps = (mc || sm[sc][ty][tx + 1]) ? TXT(0) : ps;
        pt = (mc || sm[st_][ty + 1][tx + 1]) ? TXT(0) : pt;
        pb = (mc || sm[sb][ty + 1][tx + 1]) ? TXT(0) : pb;
        d = mc ? (TXT)s_tab[54 + cls] : d;
      }
      TXT a;
      if (sizeof(TXT) == 8 && xsum) {
        a = fma(-cx, (TXT)nb_sum6(pe, pw, pn, ps, pt, pb, false), d * pc);
      } else {
        TXT s = cx * (pe + pw);
        s = fma(cy, pn + ps, s);
        s = fma(cz, pt + pb, s);
        a = fma(d, pc, -s);
      }
      if (rhs) {
        const TXT rv = bv - a;
        const TR ro = (TR)rv;
        rout[c] = ro;
        const double rd = (double)rv;
        rr = fma(rd, rd, rr);
        if (cls) rz = wall_rz(rz, s_tab[27 + cls] - s_tab[27], rd);
        bb = fma((double)bv, (double)bv, bb);
      } else {
        rout[c] = (TR)a;
      }
    }
  }
  if (mode == RES_PLAIN) return;
  double v[3] = {fma(s_tab[27], rr, rz), rr, bb}, tot[3];
  const unsigned int nb = gridDim.x * gridDim.y * gridDim.z;
  const unsigned int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
  if (last_cta_reduce<3>(v, partials, st, nb, bid, s_red, tot) && tid == 0) {
    const double rz1 = tot[0], rr1 = tot[1];
    if (mode == RES_INIT) {
      st->bb = tot[2];
      st->tol2bb = st->tol2bb * tot[2];  // host stores tol^2 here before the launch
      st->rz = rz1;
      st->rz_last = rz1;
      st->rr = rr1;
      st->iter = 0;
      st->first = 1;
      st->replacements = 0;
      if (tot[2] < 1e-16) st->done = DONE_TINY;
      else if (st->stop == 1 && rr1 <= st->tol2bb) st->done = DONE_CONVERGED;
      else st->done = RUNNING;
    } else if (mode == RES_ITER) {
      st->replacements += 1;
      finish_iteration(st, rz1, rr1, true);
    } else {  // RES_CONFIRM: explicit residual after a recursive convergence
      st->replacements += 1;
      st->rz_last = rz1;
      st->rr = rr1;
      if (rr1 <= st->tol2bb) {
        st->done = DONE_CONVERGED;
      } else if (isnan(rz1)) {
        st->done = DONE_NAN;
      } else {
        st->beta = rz1 / st->rz;
        st->rz = rz1;
        st->done = (st->iter > st->max_iter) ? DONE_MAX_ITER : RUNNING;
      }
    }
  }
}

}  // namespace bbpp
