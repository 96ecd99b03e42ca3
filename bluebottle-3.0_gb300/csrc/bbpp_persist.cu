// bbpp_persist.cu -- many PCG iterations in one launch, for grids whose search
// direction fits the chip's shared memory.
//
// One CTA per SM owns a box of cells and keeps the search direction of the box
// and of its six faces' neighbours in shared memory from iteration to
// iteration; r, Ap, x and the mask of the box stay there too as far as they
// fit, and in L2 otherwise.  In FP64 an iteration has two exchanges between the CTAs:
//   p = z + beta p on the box and its halo (the halo from the neighbours' z,
//   published by the previous exchange, and the halo's own p); Ap = L p;
//   exchange (p, Ap) -> alpha; r -= alpha Ap, x += alpha p, the z of the box's
//   surface to global memory; exchange (r, z), (r, r) -> beta, stopping test.
// In FP32 it has one (ONE below): all products of the iteration with (p, Ap), and
// the neighbours' Ap instead of their z, from which the halo's r follows.
// In an exchange every CTA stores its partial sums, counts itself in, and sums
// all CTAs' slots in the same order, so all take the same decisions.  The
// arithmetic per cell is that of k1_search2 and k2_update; the state at a
// checkpoint (every replace_every iterations) and at the end of a solve is
// theirs, so the residual replacement, the fold and the confirmation follow
// unchanged.
//
// Why: below ~3M cells the two-kernel iteration is bound by launches, by CTAs
// that are too few and by the length of their z march.  An iteration here takes
// its exchanges (2.5 us for (p, Ap), 4.5 us with the release of the surface) plus,
// in FP64, the FP64 and integer pipes.  Measured, us per iteration of a whole
// solve, kernel by kernel against resident: FP64 32^3 44.7 -> 10.8, 64^3 64 -> 16,
// 101x75x58 with walls 81 -> 23, 128^3 93 -> 53; FP32 128^3 39 -> 17 (20 with two
// exchanges), 200x144x106 with walls 69 -> 28 (31), 96^3 10.0 (13.2).
//
// A grid takes this path when p of its largest box fits a CTA's shared memory
// (about 3M cells in FP64, 6.8M in FP32); FP32 grids that can go in pairs do so
// from 4.2M cells on.
//
// Every wait is bounded (one second of globaltimer, or the state's wait_ns): a
// CTA whose wait runs out ends the solve with DONE_TIMEOUT and returns, and so
// does every CTA that waits for it.  The launch is cooperative: all CTAs are
// resident or the launch fails.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "bbpp_internal.h"
#include "bbpp_fast.cuh"

using namespace bbpp;

namespace {

constexpr int kMaxCtas = 256;          // one per SM
constexpr int kSmemCap = 227 * 1024;   // static and dynamic shared memory of a CTA

struct __align__(16) Slot {
  double v;
  unsigned long long epoch;
};

}  // namespace

struct bbpp_exchange {
  unsigned long long epoch;       // exchanges of the launches before; never reset
  unsigned long long base;        // `arrived` when the next launch starts
  unsigned long long pad[14];
  unsigned long long arrived;     // CTAs that have put their slots, over all exchanges
  unsigned long long pad2[15];
  Slot slot[2][7][kMaxCtas];      // by an exchange's parity and product
};

namespace {

// The split of the grid into boxes, and what of a box lives in shared memory:
// level 2: r, Ap, x and the mask; 1: r and Ap; 0: only p.
struct Boxes {
  int sx, sy, sz, nb;
  int one;                         // one exchange an iteration
  int level;
  int off_r, off_a, off_x, off_m, off_h, off_c;  // byte offsets in dynamic shared memory
  int smem;                        // dynamic shared memory of a CTA
};

__device__ __forceinline__ void slot_put(Slot *s, double v, unsigned long long e) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\t"
      "mov.b128 t, {%1, %2};\n\t"
      "st.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(s),
      "l"(__double_as_longlong(v)), "l"(e)
      : "memory");
}

__device__ __forceinline__ bool slot_get(const Slot *s, unsigned long long e, double &v) {
  long long lo, hi;
  asm volatile(
      "{\n\t.reg .b128 t;\n\t"
      "ld.relaxed.gpu.global.b128 t, [%2];\n\t"
      "mov.b128 {%0, %1}, t;\n\t}"
      : "=l"(lo), "=l"(hi)
      : "l"(s)
      : "memory");
  v = __longlong_as_double(lo);
  return (unsigned long long)hi == e;
}

__device__ __forceinline__ unsigned long long timer_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// L p of a cell away from walls, from its seven values (apply_L0's value)
template <typename T, bool ISO>
__device__ __forceinline__ T apply_box(const GeoL &G, T pc, T pe, T pw, T pn, T ps, T pt, T pb, bool skip) {
  if (ISO) {
    T s;
    if (sizeof(T) == 8 && G.xsum) s = (T)nb_sum6(pe, pw, pn, ps, pt, pb, skip);
    else s = ((pe + pw) + (pn + ps)) + (pt + pb);
    return fma(-gl_ax<T>(G), s, pc);
  } else {
    T s = gl_ax<T>(G) * (pe + pw);
    s = fma(gl_ay<T>(G), pn + ps, s);
    s = fma(gl_az<T>(G), pt + pb, s);
    return pc - s;
  }
}

__device__ __forceinline__ int div_m(int e, unsigned int m) { return m ? (int)__umulhi((unsigned int)e, m) : e; }
__device__ __forceinline__ unsigned int div_of(int d) { return d > 1 ? 0xffffffffu / (unsigned int)d + 1u : 0u; }

// Sum NV per-thread values over all CTAs; thread 0 of every CTA returns the
// totals, summed in the same order everywhere.  Exchange n puts this CTA's sums
// into its slots (value and epoch in one 16-byte store), adds one to the count
// of arrivals, waits until the count is `want` and reads all slots.  The slots
// carry their epoch because the count may overtake them; publish orders the
// CTA's earlier global writes before its arrival (a mailbox of tagged halo
// values, which needs no such fence, measured slower: 22 against 19 ms for a
// 128^3 FP32 solve).  s_bad is set when a wait ran out.
// Measured with 152 CTAs: 2.4 us; every CTA polling all slots instead of the
// count takes 4.6 us (152 x 19 lines polled at once), sums by groups 3.6 us.
template <int NV, int NTH>
__device__ __forceinline__ void exchange(const double (&v)[NV], double (&tot)[NV], bbpp_exchange *ex,
                                         Slot (*slots)[kMaxCtas], int nb, unsigned long long n,
                                         unsigned long long want, unsigned long long limit, bool publish, bool silent,
                                         double *s_part, double (*s_w)[8], int *s_bad) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
#pragma unroll
  for (int q = 0; q < NV; q++) s_part[q * NTH + tid] = v[q];
  __syncthreads();
  // an FP64 add occupies the pipe 16 cycles a warp: four warps sum the CTA's
  // values in fixed order, instead of shuffles in every warp
  if (tid < 128) {
    double a[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) {
      a[q] = s_part[q * NTH + tid];
#pragma unroll
      for (int k = 128; k < NTH; k += 128) a[q] += s_part[q * NTH + tid + k];
      a[q] = warp_sum(a[q]);
      if (lane == 0) s_w[q][warp] = a[q];
    }
    asm volatile("bar.sync 1, 128;" ::: "memory");
    if (tid == 0) {
      if (!silent) {
        if (publish) asm volatile("fence.acq_rel.gpu;" ::: "memory");
#pragma unroll
        for (int q = 0; q < NV; q++)
          slot_put(&slots[q][blockIdx.x], (s_w[q][0] + s_w[q][1]) + (s_w[q][2] + s_w[q][3]), n);
        asm volatile("red.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(&ex->arrived) : "memory");
      }
      unsigned long long have, t0 = 0;
      for (unsigned int k = 1;; k++) {
        if (publish) asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(have) : "l"(&ex->arrived) : "memory");
        else asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(have) : "l"(&ex->arrived) : "memory");
        if (have >= want) break;
        if ((k & 255u) == 0) {  // a look at the clock now and then
          const unsigned long long t = timer_ns();
          if (t0 == 0) t0 = t;
          else if (t - t0 > limit) {
            *s_bad = 1;
            break;
          }
        }
      }
    }
  }
  __syncthreads();
  const int nw = (nb + 31) >> 5;
  if (warp < nw) {
    const int b = warp * 32 + lane;
    const bool wait = *(volatile int *)s_bad == 0;
    double t[NV];
    bool got[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) {
      t[q] = 0.0;
      got[q] = b < nb ? slot_get(&slots[q][b], n, t[q]) : true;
    }
#pragma unroll
    for (int q = 0; q < NV; q++) {
      // the arrivals may be seen before the slot they follow: a few polls
      for (unsigned int k = 0; !got[q] && wait && k < (1u << 22); k++) got[q] = slot_get(&slots[q][b], n, t[q]);
      if (!got[q]) *s_bad = 1;
      t[q] = warp_sum(t[q]);
      if (lane == 0) s_w[q][warp] = t[q];
    }
  }
  __syncthreads();
  if (tid == 0) {
#pragma unroll
    for (int q = 0; q < NV; q++) {
      tot[q] = s_w[q][0];
      for (int w = 1; w < nw; w++) tot[q] += s_w[q][w];
    }
  }
}

// The same for the NV products of a one-exchange iteration (NV <= 7), each summed by a
// warp of its own: over the CTA's threads (sum_floats), then over the CTAs' slots, in
// fixed order.  Warp 7 counts the CTA in, its earlier global writes before it, and
// waits.  Totals in s_tot.
template <int NV, int NTH>
__device__ __forceinline__ void exchange_all(const float (&v)[NV], double *s_tot, bbpp_exchange *ex,
                                             Slot (*slots)[kMaxCtas], int nb, unsigned long long n,
                                             unsigned long long want, unsigned long long limit, bool silent,
                                             float *s_part, int *s_bad) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double a = 0.0;
#pragma unroll
  for (int q0 = 0; q0 < NV; q0 += 4) {  // four at a time, for less shared memory
    if (q0) __syncthreads();
#pragma unroll
    for (int q = q0; q < NV && q < q0 + 4; q++) s_part[(q - q0) * NTH + tid] = v[q];
    __syncthreads();
    if (warp >= q0 && warp < q0 + 4 && warp < NV) a = warp_sum(sum_floats(s_part + (warp - q0) * NTH, NTH, lane));
  }
  if (warp < NV) {
    if (lane == 0 && !silent) slot_put(&slots[warp][blockIdx.x], a, n);
  } else if (tid == 7 * 32) {
    if (!silent) {
      asm volatile("fence.acq_rel.gpu;" ::: "memory");
      asm volatile("red.relaxed.gpu.global.add.u64 [%0], 1;" ::"l"(&ex->arrived) : "memory");
    }
    unsigned long long have, t0 = 0;
    for (unsigned int k = 1;; k++) {
      asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(have) : "l"(&ex->arrived) : "memory");
      if (have >= want) break;
      if ((k & 255u) == 0) {  // a look at the clock now and then
        const unsigned long long t = timer_ns();
        if (t0 == 0) t0 = t;
        else if (t - t0 > limit) {
          *s_bad = 1;
          break;
        }
      }
    }
  }
  __syncthreads();
  if (warp < NV) {
    const bool wait = *(volatile int *)s_bad == 0;
    constexpr int K = kMaxCtas / 32;
    double t[K];
    bool got[K];
#pragma unroll
    for (int k = 0; k < K; k++) {
      t[k] = 0.0;
      got[k] = lane + 32 * k < nb ? slot_get(&slots[warp][lane + 32 * k], n, t[k]) : true;
    }
    a = 0.0;
#pragma unroll
    for (int k = 0; k < K; k++) {
      // the arrivals may be seen before a slot: a few polls
      for (unsigned int w = 0; !got[k] && wait && w < (1u << 20); w++)
        got[k] = slot_get(&slots[warp][lane + 32 * k], n, t[k]);
      if (!got[k]) *s_bad = 1;
      if (32 * k < nb) a += t[k];
    }
    a = warp_sum(a);
    if (lane == 0) s_tot[warp] = a;
  }
  __syncthreads();
}

}  // namespace

// A thread owns columns of the box: with at most NTH columns, one column and
// one of the segments of its z range; else the columns tid, tid + NTH, ...
// Along z the addresses advance by constants and the z neighbours of p are the
// values just read.  Loads go out U cells at a time ahead of the stores (the
// compiler cannot tell the box's arrays apart).
//
// ONE (FP32): one exchange an iteration.  (p,Ap) gives alpha; beta and the stopping
// test come from (r,z) - 2 alpha (Ap,z) + alpha^2 (Ap,Ap/dL), and (r,r) alike without
// dL, of products summed beside it.  The exact (r,z) of the next iteration restarts
// the expansion, so no error accumulates (as in the fused kernel).  r, x and p
// advance in one pass after it, the halo's r by the neighbours' Ap.  In FP64 the
// three more products a cell cost as much as the exchange saves from 64^3 on.
template <typename T, int NTH, int LEVEL, bool ONE, bool MASK, bool ISO>
__global__ void __launch_bounds__(NTH, 1) k_persist(const GeoL G, const Boxes B, T *p0,
                                                    T *p1, T *__restrict__ rg, T *__restrict__ ag,
                                                    T *__restrict__ xg, const uint8_t *__restrict__ mask,
                                                    DevState *st, bbpp_exchange *ex, int replace_every) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ T s_inv[27], s_im1[27], s_dm1[27];  // per class 1/dL, 1/dL - 1, dL - 1
  __shared__ __align__(16) unsigned char s_raw[ONE ? 4 * NTH * sizeof(T) : 2 * NTH * sizeof(double)];
  double *const s_part = reinterpret_cast<double *>(s_raw);
  __shared__ double s_w[2][8];
  __shared__ double s_tot[8];
  __shared__ double s_alpha, s_beta;
  __shared__ int s_bad, s_done, s_exact;
  constexpr int U = sizeof(T) == 8 ? 2 : 4;
  if (*(volatile int *)&st->done) return;
  unsigned long long epoch = *(volatile unsigned long long *)&ex->epoch;
  unsigned long long want = *(volatile unsigned long long *)&ex->base;
  const unsigned long long epoch0 = epoch;
  const int it0 = *(volatile int *)&st->iter;
  bool first = *(volatile int *)&st->first;
  const bool lag = !first && *(volatile int *)&st->dlag;
  const long long wl = *(volatile long long *)&st->wait_ns;
  const unsigned long long limit = wl > 0 ? (unsigned long long)wl : 1000000000ull;
  // test hooks, all of them in the last CTA
  const int inject = blockIdx.x == (unsigned)B.nb - 1u ? *(volatile int *)&st->inject : 0;
  const bool silent0 = inject == INJECT_EXCHANGE || (sizeof(T) == 4 && inject == INJECT_COPIES);
  const int tid = threadIdx.x;
  if (tid < 27) s_inv[tid] = sizeof(T) == 8 ? (T)G.invL[tid] : (T)G.finvL[tid];
  if (tid < 27) s_dm1[tid] = (sizeof(T) == 8 ? (T)G.dL[tid] : (T)G.fdL[tid]) - T(1);
  if (tid < 27) s_im1[tid] = (sizeof(T) == 8 ? (T)G.invL[tid] : (T)G.finvL[tid]) - T(1);
  if (tid == 0) {
    s_alpha = lag ? *(volatile double *)&st->alpha : 0.0;
    s_beta = first ? 0.0 : *(volatile double *)&st->beta;
    s_bad = 0;
    s_done = RUNNING;
    s_exact = 0;
  }
  // thread 0's copy of the solve's scalars
  double rz = *(volatile double *)&st->rz, rz_last = *(volatile double *)&st->rz_last,
         rr_last = *(volatile double *)&st->rr, pap = 0.0;
  const int stop = st->stop, max_iter = st->max_iter, trace_n = st->trace_n;
  const double tol2bb = st->tol2bb;
  double *const trace_a = blockIdx.x == 0 ? st->trace_a : nullptr;
  double *const trace_b = blockIdx.x == 0 ? st->trace_b : nullptr;

  // this CTA's box
  const int nx = G.nx, ny = G.ny, nz = G.nz;
  int ix = blockIdx.x;
  const int iz = ix / (B.sx * B.sy);
  ix -= iz * (B.sx * B.sy);
  const int iy = ix / B.sx;
  ix -= iy * B.sx;
  const int x0 = (int)((long long)ix * nx / B.sx), bx = (int)((long long)(ix + 1) * nx / B.sx) - x0;
  const int y0 = (int)((long long)iy * ny / B.sy), by = (int)((long long)(iy + 1) * ny / B.sy) - y0;
  const int z0 = (int)((long long)iz * nz / B.sz), bz = (int)((long long)(iz + 1) * nz / B.sz) - z0;
  const int PW = bx + 2, PP = PW * (by + 2);
  const unsigned int mbx = div_of(bx), mby = div_of(by);
  const unsigned int plane = (unsigned int)nx * (unsigned int)ny;
  const int ncol = bx * by;
  const int hz = ncol, hy = bx * bz, hx = by * bz, halo = 2 * (hz + hy + hx);
  // the box's faces at a wall (z low, z high, y low, y high, x low, x high)
  const int wf = (G.pz ? 0 : (int)(z0 == 0) | (int)(z0 + bz == nz) << 1) |
                 (G.py ? 0 : (int)(y0 == 0) << 2 | (int)(y0 + by == ny) << 3) |
                 (G.px ? 0 : (int)(x0 == 0) << 4 | (int)(x0 + bx == nx) << 5);
  // this thread's first column and its z range
  int col0 = tid, za = 0, zb = bz;
  if (ncol <= NTH) {
    const int nseg = NTH / ncol, seg = tid / ncol, len = (bz + nseg - 1) / nseg;
    col0 = seg < nseg ? tid - seg * ncol : ncol;
    za = min(bz, seg * len);
    zb = min(bz, za + len);
  }

  // between a launch's entry and exit p0 is free: it carries the z of the boxes'
  // surfaces to their neighbours
  T *const zg = p0;
  T *const sh = reinterpret_cast<T *>(smem_raw + B.off_h);  // ONE: r of the halo
  uint8_t *const sc = smem_raw + B.off_c;                   // ONE: its class
  // the halo has cells at a wall
  const bool near_wall = (!G.px && (x0 <= 1 || x0 + bx >= nx - 1)) || (!G.py && (y0 <= 1 || y0 + by >= ny - 1)) ||
                         (!G.pz && (z0 <= 1 || z0 + bz >= nz - 1));
  T *const sp = reinterpret_cast<T *>(smem_raw);
  T *const rs = reinterpret_cast<T *>(smem_raw + B.off_r);
  T *const as = reinterpret_cast<T *>(smem_raw + B.off_a);
  T *const xs = reinterpret_cast<T *>(smem_raw + B.off_x);
  uint8_t *const ms = smem_raw + B.off_m;

  // one column: its place in the box's arrays (e), in p's box (o) and in the
  // grid (g) at z = 0, with the steps per plane ncol, PP and plane
  struct Col {
    int e, o, lx, ly;
    unsigned int g;
  };
  auto column = [&](int col) {
    Col c;
    c.e = col;
    c.ly = div_m(col, mbx);
    c.lx = col - c.ly * bx;
    c.o = PP + (c.ly + 1) * PW + c.lx + 1;
    c.g = plane * (unsigned int)z0 + (unsigned int)nx * (unsigned int)(y0 + c.ly) + (unsigned int)(x0 + c.lx);
    return c;
  };
  // element q of face f: its coordinates in the box, one outside it in the
  // face's direction
  auto on_face = [&](int f, int q, int &lx, int &ly, int &lz) {
    if (f < 2) {
      ly = div_m(q, mbx);
      lx = q - ly * bx;
      lz = f ? bz : -1;
    } else if (f < 4) {
      lz = div_m(q, mbx);
      lx = q - lz * bx;
      ly = f == 3 ? by : -1;
    } else {
      lz = div_m(q, mby);
      ly = q - lz * by;
      lx = f == 5 ? bx : -1;
    }
  };
  // halo element h: its place in the box (o), its cell (g) and that cell's class;
  // false outside a wall, where p stays zero
  auto halo_cell = [&](int h, int &o, unsigned int &g, int &cls, auto classes) {
    int f = 0, lx, ly, lz;
    if (h >= 2 * (hz + hy)) {
      h -= 2 * (hz + hy);
      f = 4 + (int)(h >= hx);
      h -= f == 5 ? hx : 0;
    } else if (h >= 2 * hz) {
      h -= 2 * hz;
      f = 2 + (int)(h >= hy);
      h -= f == 3 ? hy : 0;
    } else {
      f = (int)(h >= hz);
      h -= f == 1 ? hz : 0;
    }
    on_face(f, h, lx, ly, lz);
    o = (lz + 1) * PP + (ly + 1) * PW + lx + 1;
    const int gx = halo_index(x0 + lx, nx, G.px), gy = halo_index(y0 + ly, ny, G.py),
              gz = halo_index(z0 + lz, nz, G.pz);
    g = plane * (unsigned int)gz + (unsigned int)nx * (unsigned int)gy + (unsigned int)gx;
    cls = decltype(classes)::value
              ? wall_count(gx, nx, G.px) + 3 * wall_count(gy, ny, G.py) + 9 * wall_count(gz, nz, G.pz)
              : 0;
    return ((wf >> f) & 1) == 0;
  };
  // fn(e, o, g, class) for every cell of the box at a wall, once.  The other
  // loops carry no class arithmetic: in FP64 even an instruction that no lane
  // takes occupies the pipe, and the boxes at a wall kept the others waiting
  auto wall_cells = [&](auto fn) {
    for (int f = 0; f < 6; f++) {
      if (!((wf >> f) & 1)) continue;
      const int n = f < 2 ? hz : (f < 4 ? hy : hx);
      for (int q = tid; q < n; q += NTH) {
        int lx, ly, lz;
        on_face(f, q, lx, ly, lz);
        lx = min(max(lx, 0), bx - 1);
        ly = min(max(ly, 0), by - 1);
        lz = min(max(lz, 0), bz - 1);
        const int hit = ((int)(lz == 0) | (int)(lz == bz - 1) << 1 | (int)(ly == 0) << 2 | (int)(ly == by - 1) << 3 |
                         (int)(lx == 0) << 4 | (int)(lx == bx - 1) << 5) &
                        wf;
        if (hit & ((1 << f) - 1)) continue;  // met on an earlier face
        fn(lx + bx * ly + ncol * lz, (lz + 1) * PP + (ly + 1) * PW + lx + 1,
           plane * (unsigned int)(z0 + lz) + (unsigned int)nx * (unsigned int)(y0 + ly) + (unsigned int)(x0 + lx),
           __popc(hit & 48) + 3 * __popc(hit & 12) + 9 * __popc(hit & 3));
      }
    }
  };
  __syncthreads();

  // the box's vectors; a step that the kernel before left pending goes into x
  {
    const T *po = (it0 & 1) ? p1 : p0;
    const T alpha = (T)s_alpha;
    for (int col = col0; col < ncol; col += NTH) {
      const Col c = column(col);
#pragma unroll 4
      for (int z = za; z < zb; z++) {
        const unsigned int g = c.g + plane * (unsigned int)z;
        const int e = c.e + ncol * z;
        const T p = first ? T(0) : po[g];
        sp[c.o + PP * z] = p;
        if (LEVEL >= 1) rs[e] = rg[g];
        if (LEVEL >= 2) xs[e] = lag ? fma(alpha, p, xg[g]) : xg[g];
        else if (lag) xg[g] = fma(alpha, p, xg[g]);
        if (MASK && LEVEL >= 2) ms[e] = mask[g];
      }
    }
    for (int h = tid; h < halo; h += NTH) {
      int o, cls;
      unsigned int g;
      const bool in = halo_cell(h, o, g, cls, std::false_type());
      sp[o] = in && !first ? po[g] : T(0);
      if (ONE && near_wall) sc[h] = 0;
    }
  }
  __syncthreads();

  int it = it0;
  // p = z + beta p on the box and its halo, z = r / dL.  The halo's z is in zg;
  // for a launch's first iteration it is formed from r.
  auto direction = [&]() {
    const T beta = (T)s_beta;
    // the halo first: its loads take longest
    if (it == it0 + 1) {
      for (int h = tid; h < halo; h += NTH) {
        int o, cls;
        unsigned int g;
        if (!halo_cell(h, o, g, cls, std::true_type())) continue;
        const T r = rg[g];
        if (ONE) {
          sh[h] = r;
          if (near_wall) sc[h] = (uint8_t)cls;
          sp[o] = fma(s_im1[cls], r, first ? r : fma(beta, sp[o], r));
          continue;
        }
        T z = r;
        if (cls) z *= s_inv[cls];
        sp[o] = first ? z : fma(beta, sp[o], z);
      }
    } else {
      constexpr int H = sizeof(T) == 8 ? 4 : 6;
      for (int h0 = tid; h0 < halo; h0 += H * NTH) {
        T z[H];
        int o[H];
#pragma unroll
        for (int k = 0; k < H; k++) {
          if (h0 + k * NTH >= halo) break;
          unsigned int g;
          int cls;
          if (!halo_cell(h0 + k * NTH, o[k], g, cls, std::false_type())) o[k] = -1;
          z[k] = o[k] >= 0 ? __ldcg(zg + g) : T(0);
        }
#pragma unroll
        for (int k = 0; k < H; k++) {
          if (h0 + k * NTH >= halo) break;
          if (o[k] >= 0) sp[o[k]] = fma(beta, sp[o[k]], z[k]);
        }
      }
    }
    for (int col = col0; col < ncol; col += NTH) {
      const Col c = column(col);
      for (int z = za; z < zb; z += 2 * U) {
        T v[2 * U], p[2 * U];
#pragma unroll
        for (int k = 0; k < 2 * U; k++) {
          const int zz = min(z + k, zb - 1);
          v[k] = LEVEL >= 1 ? rs[c.e + ncol * zz] : rg[c.g + plane * (unsigned int)zz];
          p[k] = sp[c.o + PP * zz];
        }
#pragma unroll
        for (int k = 0; k < 2 * U; k++)
          if (z + k < zb) sp[c.o + PP * (z + k)] = first ? v[k] : fma(beta, p[k], v[k]);
      }
    }
    if (wf) {
      __syncthreads();
      wall_cells([&](int e, int o, unsigned int g, int cls) {
        sp[o] = fma(s_im1[cls], LEVEL >= 1 ? rs[e] : rg[g], sp[o]);
      });
    }
  };
  // Ap = L p, (p, Ap)
  auto stencil = [&]() {
    typename Acc<T>::type acc = 0;
    for (int col = col0; col < ncol; col += NTH) {
      const Col c = column(col);
      const T *q = sp + c.o + PP * za;
      T pb = za < zb ? q[-PP] : T(0), pc = za < zb ? q[0] : T(0);
      for (int z = za; z < zb; z += U) {
        T t[U], e[U], w[U], n[U], s[U], a[U], cc[U];
        bool solid[U];
        const T *qz = sp + c.o + PP * z;
#pragma unroll
        for (int k = 0; k < U; k++) {
          const int kk = min(k, zb - 1 - z);
          const T *qk = qz + PP * kk;
          t[k] = qk[PP];
          e[k] = qk[1];
          w[k] = qk[-1];
          n[k] = qk[PW];
          s[k] = qk[-PW];
          solid[k] = MASK && (LEVEL >= 2 ? ms[c.e + ncol * (z + kk)]
                                         : __ldg(mask + c.g + plane * (unsigned int)(z + kk))) != 0;
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          cc[k] = pc;
          a[k] = apply_box<T, ISO>(G, pc, e[k], w[k], n[k], s[k], t[k], pb, solid[k]);
          if (solid[k]) a[k] = T(0);
          pb = pc;
          pc = t[k];
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          if (z + k >= zb) break;
          if (LEVEL >= 1) as[c.e + ncol * (z + k)] = a[k];
          else ag[c.g + plane * (unsigned int)(z + k)] = a[k];
          acc = fma(cc[k], a[k], acc);
        }
      }
    }
    if (wf) {
      __syncthreads();
      wall_cells([&](int e, int o, unsigned int g, int cls) {
        const T p = sp[o], q = s_dm1[cls] * p;  // the diagonal of L there is 1 + s_dm1
        T *a = LEVEL >= 1 ? as + e : ag + g;
        *a = *a + q;
        acc = fma(p, q, acc);
      });
    }
    return (double)acc;
  };
  // r -= alpha Ap, x += alpha p; (r, r) and the walls' part of (r, z)
  auto update = [&](double (&v)[2]) {
    typename Acc<T>::type rr = 0, corr = 0;
    const T alpha = (T)s_alpha;
    for (int col = col0; col < ncol; col += NTH) {
      const Col c = column(col);
      const bool side = c.lx == 0 || c.lx == bx - 1 || c.ly == 0 || c.ly == by - 1;
      for (int z = za; z < zb; z += U) {
        T r[U], a[U], x[U], p[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
          const int zz = min(z + k, zb - 1), e = c.e + ncol * zz;
          const unsigned int g = c.g + plane * (unsigned int)zz;
          x[k] = LEVEL >= 2 ? xs[e] : xg[g];
          r[k] = LEVEL >= 1 ? rs[e] : rg[g];
          a[k] = LEVEL >= 1 ? as[e] : ag[g];
          p[k] = sp[c.o + PP * zz];
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          if (z + k >= zb) break;
          const int e = c.e + ncol * (z + k);
          const unsigned int g = c.g + plane * (unsigned int)(z + k);
          const T rn = fma(-alpha, a[k], r[k]);
          const T xn = fma(alpha, p[k], x[k]);
          if (LEVEL >= 2) xs[e] = xn;
          else xg[g] = xn;
          if (LEVEL >= 1) rs[e] = rn;
          else rg[g] = rn;
          if (side || z + k == 0 || z + k == bz - 1) zg[g] = rn;  // the neighbours' halo
          rr = fma(rn, rn, rr);
        }
      }
    }
    if (wf) {
      __syncthreads();
      wall_cells([&](int e, int o, unsigned int g, int cls) {
        const T r = LEVEL >= 1 ? rs[e] : rg[g];
        zg[g] = r * s_inv[cls];
        corr = fma(s_im1[cls] * r, r, corr);
      });
    }
    v[0] = (double)rr + (double)corr;
    v[1] = (double)rr;
  };
  // ONE: Ap = L p with its products, Ap of the box's surface to wg; v: (p,Ap),
  // (r,r), (r,Ap), (Ap,Ap) and, of the last three with 1/dL, what the walls add
  auto stencil_all = [&](T *wg, T (&v)[7]) {
#pragma unroll
    for (int k = 0; k < 7; k++) v[k] = T(0);
    for (int col = col0; col < ncol; col += NTH) {
      const Col c = column(col);
      const bool side = c.lx == 0 || c.lx == bx - 1 || c.ly == 0 || c.ly == by - 1;
      const T *q = sp + c.o + PP * za;
      T pb = za < zb ? q[-PP] : T(0), pc = za < zb ? q[0] : T(0);
      for (int z = za; z < zb; z += U) {
        T t[U], e[U], w[U], n[U], s[U], a[U], cc[U], r[U];
        bool solid[U];
        const T *qz = sp + c.o + PP * z;
#pragma unroll
        for (int k = 0; k < U; k++) {
          const int kk = min(k, zb - 1 - z);
          const T *qk = qz + PP * kk;
          t[k] = qk[PP];
          e[k] = qk[1];
          w[k] = qk[-1];
          n[k] = qk[PW];
          s[k] = qk[-PW];
          r[k] = LEVEL >= 1 ? rs[c.e + ncol * (z + kk)] : rg[c.g + plane * (unsigned int)(z + kk)];
          solid[k] = MASK && (LEVEL >= 2 ? ms[c.e + ncol * (z + kk)]
                                         : __ldg(mask + c.g + plane * (unsigned int)(z + kk))) != 0;
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          cc[k] = pc;
          a[k] = apply_box<T, ISO>(G, pc, e[k], w[k], n[k], s[k], t[k], pb, solid[k]);
          if (solid[k]) a[k] = T(0);
          pb = pc;
          pc = t[k];
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          if (z + k >= zb) break;
          const unsigned int g = c.g + plane * (unsigned int)(z + k);
          if (LEVEL >= 1) as[c.e + ncol * (z + k)] = a[k];
          else ag[g] = a[k];
          if (side || z + k == 0 || z + k == bz - 1) wg[g] = a[k];
          v[0] = fma(cc[k], a[k], v[0]);
          v[1] = fma(r[k], r[k], v[1]);
          v[2] = fma(r[k], a[k], v[2]);
          v[3] = fma(a[k], a[k], v[3]);
        }
      }
    }
    if (wf) {
      __syncthreads();
      wall_cells([&](int e, int o, unsigned int g, int cls) {
        T *ap = LEVEL >= 1 ? as + e : ag + g;
        const T p = sp[o], q = s_dm1[cls] * p, a0 = *ap, a = a0 + q, r = LEVEL >= 1 ? rs[e] : rg[g];
        const T im = s_im1[cls];
        *ap = a;
        wg[g] = a;
        v[0] = fma(p, q, v[0]);
        v[2] = fma(r, q, v[2]);
        v[3] = fma(q, a + a0, v[3]);
        v[4] = fma(im * r, r, v[4]);
        v[5] = fma(im * r, a, v[5]);
        v[6] = fma(im * a, a, v[6]);
      });
    }
  };
  // ONE: r -= alpha Ap and p = z + beta p on the halo, with the roundings of the
  // boxes that own its cells
  auto turn_halo = [&](const T *wg) {
    const T alpha = (T)s_alpha, beta = (T)s_beta;
    constexpr int H = 6;
    for (int h0 = tid; h0 < halo; h0 += H * NTH) {
      T w[H];
      int o[H];
#pragma unroll
      for (int k = 0; k < H; k++) {
        if (h0 + k * NTH >= halo) break;
        unsigned int g;
        int cls;
        if (!halo_cell(h0 + k * NTH, o[k], g, cls, std::false_type())) o[k] = -1;
        w[k] = o[k] >= 0 ? __ldcg(wg + g) : T(0);
      }
#pragma unroll
      for (int k = 0; k < H; k++) {
        if (h0 + k * NTH >= halo) break;
        if (o[k] < 0) continue;
        const T r = fma(-alpha, w[k], sh[h0 + k * NTH]);
        sh[h0 + k * NTH] = r;
        sp[o[k]] = fma(beta, sp[o[k]], r);
      }
    }
    if (!near_wall) return;
#pragma unroll 1
    for (int h = tid; h < halo; h += NTH) {
      if (sc[h] == 0) continue;
      int o, cls;
      unsigned int g;
      halo_cell(h, o, g, cls, std::false_type());
      sp[o] = fma(s_im1[sc[h]], sh[h], sp[o]);
    }
  };
  // ONE: what 1 / dL adds to p at the walls
  auto turn_walls = [&]() {
    if (!wf) return;
    __syncthreads();
    wall_cells([&](int e, int o, unsigned int g, int cls) {
      sp[o] = fma(s_im1[cls], LEVEL >= 1 ? rs[e] : rg[g], sp[o]);
    });
  };
  // ONE: r -= alpha Ap, x += alpha p and, with `next`, the next p on the box and its halo
  auto advance = [&](const T *wg, bool next) {
    const T alpha = (T)s_alpha, beta = (T)s_beta;
    if (next) turn_halo(wg);
    for (int col = col0; col < ncol; col += NTH) {
      const Col c = column(col);
      for (int z = za; z < zb; z += U) {
        T r[U], a[U], x[U], p[U];
#pragma unroll
        for (int k = 0; k < U; k++) {
          const int zz = min(z + k, zb - 1), e = c.e + ncol * zz;
          const unsigned int g = c.g + plane * (unsigned int)zz;
          x[k] = LEVEL >= 2 ? xs[e] : xg[g];
          r[k] = LEVEL >= 1 ? rs[e] : rg[g];
          a[k] = LEVEL >= 1 ? as[e] : ag[g];
          p[k] = sp[c.o + PP * zz];
        }
#pragma unroll
        for (int k = 0; k < U; k++) {
          if (z + k >= zb) break;
          const int e = c.e + ncol * (z + k);
          const unsigned int g = c.g + plane * (unsigned int)(z + k);
          const T rn = fma(-alpha, a[k], r[k]);
          const T xn = fma(alpha, p[k], x[k]);
          if (LEVEL >= 2) xs[e] = xn;
          else xg[g] = xn;
          if (LEVEL >= 1) rs[e] = rn;
          else rg[g] = rn;
          if (next) sp[c.o + PP * (z + k)] = fma(beta, p[k], rn);
        }
      }
    }
    if (next) turn_walls();
  };

  bool checkpoint = false;
  if constexpr (ONE) {
    const bool walls = !(G.px && G.py && G.pz);
    // an exchange of NV sums into s_tot
    auto meet = [&](auto &v, bool silent) {
      constexpr int NV = sizeof(v) / sizeof(float);
      ++epoch;
      want += (unsigned long long)B.nb;
      exchange_all<NV, NTH>(v, s_tot, ex, ex->slot[epoch & 1], B.nb, epoch, want, limit, silent,
                            reinterpret_cast<float *>(s_raw), &s_bad);
    };
    // finish_iteration on thread 0's scalars
    auto finish = [&](double rz1, double rr1) {
      rz_last = rz1;
      rr_last = rr1;
      const bool conv = (stop == 0 ? rz1 : rr1) <= tol2bb;
      if (conv) {
        s_done = it > max_iter ? DONE_MAX_ITER : (stop == 0 ? DONE_CONVERGED : DONE_PENDING);
      } else if (isnan(rz1)) {
        s_done = DONE_NAN;
      } else {
        s_beta = rz1 / rz;
        trace_put(trace_b, trace_n, it - 1, s_beta);
        rz = rz1;
        if (it > max_iter) s_done = DONE_MAX_ITER;
      }
    };
    T v[7];
    auto meet_all = [&](bool silent) {
      if (walls) {
        meet(v, silent);
      } else {
        T u[4] = {v[0], v[1], v[2], v[3]};
        meet(u, silent);
      }
    };
    it++;
    direction();
    first = false;
    for (;;) {
      for (;; it++) {
        checkpoint = it % replace_every == 0;
        __syncthreads();
        // by the iteration's parity, as p is stored at the end: a slow neighbour may
        // still read the other buffer, which carries the iteration before's
        T *const wg = (it & 1) ? p1 : p0;
        stencil_all(wg, v);
        meet_all(silent0 && it == it0 + 1);
        if (tid == 0 && !s_bad) {
          const double wr = walls ? s_tot[4] : 0.0, wa = walls ? s_tot[5] : 0.0, waa = walls ? s_tot[6] : 0.0;
          const double rr = s_tot[1];
          rz = rr + wr;
          pap = s_tot[0];
          const double al = rz / pap;
          s_alpha = al;
          trace_put(trace_a, trace_n, it - 1, al);
          const double rz1 = rz - 2.0 * al * (s_tot[2] + wa) + al * al * (s_tot[3] + waa);
          const double rr1 = rr - 2.0 * al * s_tot[2] + al * al * s_tot[3];
          // what a step leaves of the residual is known to some 1e-7 of what was
          // there; where that is not enough (or is NaN), from the residual itself
          if (!checkpoint) {
            if (rz1 >= 0.03 * rz && rr1 >= 0.03 * rr) finish(rz1, rr1);
            else s_exact = 1;
          }
        }
        __syncthreads();
        if (s_bad || checkpoint || s_exact) break;
        const bool next = s_done == RUNNING;
        advance(wg, next);
        if (!next) break;
      }
      if (s_bad || !s_exact) break;
      // the step, the sums of the residual it leaves and the next p one by one
      const T alpha = (T)s_alpha;
      for (int k = 0; k < 7; k++) v[k] = T(0);
#pragma unroll 1
      for (int col = col0; col < ncol; col += NTH) {
        const Col c = column(col);
#pragma unroll 1
        for (int z = za; z < zb; z++) {
          const int e = c.e + ncol * z;
          const unsigned int g = c.g + plane * (unsigned int)z;
          T &r = LEVEL >= 1 ? rs[e] : rg[g], &x = LEVEL >= 2 ? xs[e] : xg[g];
          r = fma(-alpha, LEVEL >= 1 ? as[e] : ag[g], r);
          x = fma(alpha, sp[c.o + PP * z], x);
          v[1] = fma(r, r, v[1]);
        }
      }
      __syncthreads();
      if (wf)
        wall_cells([&](int e, int, unsigned int g, int cls) {
          const T r = LEVEL >= 1 ? rs[e] : rg[g];
          v[4] = fma(s_im1[cls] * r, r, v[4]);
        });
      meet_all(false);
      if (tid == 0) {
        s_exact = 0;
        if (!s_bad) finish(s_tot[1] + (walls ? s_tot[4] : 0.0), s_tot[1]);
      }
      __syncthreads();
      if (s_bad || s_done != RUNNING) break;
      const T beta = (T)s_beta;
      const T *const wg = (it & 1) ? p1 : p0;
#pragma unroll 1
      for (int h = tid; h < halo; h += NTH) {
        int o, cls;
        unsigned int g;
        if (!halo_cell(h, o, g, cls, std::true_type())) continue;
        const T r = fma(-alpha, __ldcg(wg + g), sh[h]);
        sh[h] = r;
        sp[o] = fma(s_im1[cls], r, fma(beta, sp[o], r));
      }
#pragma unroll 1
      for (int col = col0; col < ncol; col += NTH) {
        const Col c = column(col);
#pragma unroll 1
        for (int z = za; z < zb; z++) {
          T &p = sp[c.o + PP * z];
          p = fma(beta, p, LEVEL >= 1 ? rs[c.e + ncol * z] : rg[c.g + plane * (unsigned int)z]);
        }
      }
      turn_walls();
      it++;
    }
    __syncthreads();
  } else {
    for (;;) {
      it++;
      checkpoint = it % replace_every == 0;
      direction();
      first = false;
      __syncthreads();
      {
        const double v[1] = {stencil()};
        double tot[1];
        ++epoch;
        want += (unsigned long long)B.nb;
        exchange<1, NTH>(v, tot, ex, ex->slot[0], B.nb, epoch, want, limit, false, silent0 && it == it0 + 1, s_part, s_w, &s_bad);
        if (tid == 0 && !s_bad) {
          pap = tot[0];
          const double a = rz / pap;
          s_alpha = a;
          trace_put(trace_a, trace_n, it - 1, a);
        }
      }
      __syncthreads();
      if (s_bad || checkpoint) break;
      {
        double v[2], tot[2];
        update(v);
        ++epoch;
        want += (unsigned long long)B.nb;
        exchange<2, NTH>(v, tot, ex, ex->slot[0] + 1, B.nb, epoch, want, limit, true, false, s_part, s_w, &s_bad);
        if (tid == 0 && !s_bad) {
          // finish_iteration on the local scalars
          const double rz1 = tot[0], rr1 = tot[1];
          rz_last = rz1;
          rr_last = rr1;
          const bool conv = (stop == 0 ? rz1 : rr1) <= tol2bb;
          if (conv) {
            s_done = it > max_iter ? DONE_MAX_ITER : (stop == 0 ? DONE_CONVERGED : DONE_PENDING);
          } else if (isnan(rz1)) {
            s_done = DONE_NAN;
          } else {
            s_beta = rz1 / rz;
            trace_put(trace_b, trace_n, it - 1, s_beta);
            rz = rz1;
            if (it > max_iter) s_done = DONE_MAX_ITER;
          }
        }
      }
      __syncthreads();
      if (s_bad || s_done != RUNNING) break;
    }
  }

  if (inject == INJECT_LAST_WAIT && s_done != RUNNING) {
    if (tid == 0) s_bad = 1;
    __syncthreads();
  }
  if (!s_bad) {
    T *po = (it & 1) ? p1 : p0;
    for (int col = col0; col < ncol; col += NTH) {
      const Col c = column(col);
#pragma unroll 4
      for (int z = za; z < zb; z++) {
        const unsigned int g = c.g + plane * (unsigned int)z;
        const int e = c.e + ncol * z;
        po[g] = sp[c.o + PP * z];
        if (LEVEL >= 1) rg[g] = rs[e];
        if (LEVEL >= 2) xg[g] = xs[e];
        if (LEVEL >= 1 && checkpoint) ag[g] = as[e];
      }
    }
  }
  if (tid == 0) {
    if (s_bad) atomicExch(&st->done, (int)DONE_TIMEOUT);
    if (blockIdx.x == 0) {
      // after a wait that ran out: past every epoch the others may still write
      ex->epoch = epoch0 + 2ull * (unsigned long long)replace_every + 2ull;
      ex->base = want;
      if (!s_bad) {
        st->rz = rz;
        st->rz_last = rz_last;
        st->rz_next = rz_last;
        st->rr = rr_last;
        st->pAp = pap;
        st->alpha = s_alpha;
        st->beta = s_beta;
        st->first = 0;
        // at a checkpoint the iteration's step is still owed, to the update
        // or to the replacement that follows; otherwise x and r are current
        st->dlag = checkpoint ? 1 : 0;
        st->iter = checkpoint ? it - 1 : it;
        if (checkpoint) decide_replacement(st);
        // another CTA's wait may have run out in the last exchange: that stands
        else if (s_done != RUNNING) atomicCAS(&st->done, (int)RUNNING, s_done);
      }
    }
  }
}

// ------------------------------------------------------------------- host --
struct bbpp_persist_state {
  Boxes box[2];  // [FP32, FP64]
  bool ok[2] = {false, false};
  int nth[2] = {512, 512};
  bbpp_exchange *ex = nullptr;
  bool refused = false;  // the last launch
};

namespace {

constexpr size_t static_smem(int nth) { return 16 * (size_t)nth + 1024; }

// The split into at most `most` boxes that costs a thread least: the cells of
// its columns (see k_persist), and the halo cells at half a cell's cost (the x
// faces, whose cells lie in a sector each, at a cell's).  p of a box
// with its halo must fit `cap` bytes.
bool plan_boxes(const GeoL &G, int most, int elem, int nth, bool one, Boxes *out) {
  const size_t cap = kSmemCap - static_smem(nth);
  const bool walls = !(G.px && G.py && G.pz);
  // p of a box with its halo, and with one exchange the halo's r beside it
  auto fixed = [&](size_t bx, size_t by, size_t bz) {
    return (bx + 2) * (by + 2) * (bz + 2) * elem + (one ? 2 * (bx * by + bx * bz + by * bz) * (elem + walls) + 48 : 0);
  };
  double best = 1e300;
  for (int sx = 1; sx <= G.nx && sx <= most; sx++)
    for (int sy = 1; sy <= G.ny && sx * sy <= most; sy++) {
      const int sz0 = std::min(G.nz, most / (sx * sy));
      const int bz = (G.nz + sz0 - 1) / sz0, sz = (G.nz + bz - 1) / bz;
      const int bx = (G.nx + sx - 1) / sx, by = (G.ny + sy - 1) / sy;
      if (fixed(bx, by, bz) > cap) continue;
      const int ncol = bx * by, nseg = std::max(1, nth / ncol);
      const double steps = ncol <= nth ? (bz + nseg - 1) / nseg : (double)((ncol + nth - 1) / nth) * bz;
      const double cost = steps * nth + 1.0 * ((double)ncol + (double)bx * bz) + 2.0 * (double)by * bz;
      if (cost < best) {
        best = cost;
        out->sx = sx;
        out->sy = sy;
        out->sz = sz;
      }
    }
  if (best >= 1e300) return false;
  out->nb = out->sx * out->sy * out->sz;
  out->one = one;
  const size_t bx = (G.nx + out->sx - 1) / out->sx, by = (G.ny + out->sy - 1) / out->sy,
               bz = (G.nz + out->sz - 1) / out->sz;
  auto up = [](size_t v) { return (v + 15) / 16 * 16; };
  const size_t p0 = up((bx + 2) * (by + 2) * (bz + 2) * elem), vec = up(bx * by * bz * elem), m = up(bx * by * bz);
  out->off_h = (int)p0;
  const size_t halo = 2 * (bx * by + bx * bz + by * bz);
  out->off_c = (int)(p0 + up(halo * elem));
  const size_t p = p0 + (one ? up(halo * elem) + (walls ? up(halo) : 0) : 0);
  out->off_r = (int)p;
  out->off_a = (int)(p + vec);
  out->off_x = (int)(p + 2 * vec);
  out->off_m = (int)(p + 3 * vec);
  out->level = p + 3 * vec + m <= cap ? 2 : (p + 2 * vec <= cap ? 1 : 0);
  out->smem = (int)(p + (out->level + (out->level > 0)) * vec + (out->level == 2 ? m : 0));
  return true;
}

typedef void (*Kern64)(const GeoL, const Boxes, double *, double *, double *, double *, double *, const uint8_t *,
                       DevState *, bbpp_exchange *, int);
typedef void (*Kern32)(const GeoL, const Boxes, float *, float *, float *, float *, float *, const uint8_t *,
                       DevState *, bbpp_exchange *, int);
template <typename T> struct KernOf;
template <> struct KernOf<double> { typedef Kern64 type; };
template <> struct KernOf<float> { typedef Kern32 type; };

template <typename T, int NTH, int LEVEL, bool ONE>
typename KernOf<T>::type pick3(bool mask, bool iso) {
  if (mask) return iso ? k_persist<T, NTH, LEVEL, ONE, true, true> : k_persist<T, NTH, LEVEL, ONE, true, false>;
  return iso ? k_persist<T, NTH, LEVEL, ONE, false, true> : k_persist<T, NTH, LEVEL, ONE, false, false>;
}
// Small boxes (level 2 only) with 256 threads, the others with 512.
Kern32 pick(float, int nth, const Boxes &B, bool mask, bool iso) {
  if (!B.one) return pick3<float, 512, 0, false>(mask, iso);
  if (nth == 256) return pick3<float, 256, 2, true>(mask, iso);
  if (B.level == 2) return pick3<float, 512, 2, true>(mask, iso);
  return B.level == 1 ? pick3<float, 512, 1, true>(mask, iso) : pick3<float, 512, 0, true>(mask, iso);
}
Kern64 pick(double, int nth, const Boxes &B, bool mask, bool iso) {
  if (nth == 256) return pick3<double, 256, 2, false>(mask, iso);
  if (B.level == 2) return pick3<double, 512, 2, false>(mask, iso);
  return B.level == 1 ? pick3<double, 512, 1, false>(mask, iso) : pick3<double, 512, 0, false>(mask, iso);
}

}  // namespace

void bbpp_persist_init(bbpp_ctx *ctx) {
  bbpp_persist_state *t = new bbpp_persist_state();
  ctx->persist = t;
  const char *e = getenv("BBPP_PERSIST");
  if (e && e[0] == '0') return;
  int dev = 0, coop = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev);
  if (!coop) return;
  const int most = std::min(ctx->sms, kMaxCtas);
  for (int k = 0; k < 2; k++) {
    const int elem = k ? 8 : 4;
    Boxes &B = t->box[k];
    t->nth[k] = (ctx->GL.n + most - 1) / most <= 512 ? 256 : 512;
    bool ok = plan_boxes(ctx->GL, most, elem, t->nth[k], k == 0, &B);
    if (t->nth[k] == 256 && (!ok || B.level != 2)) {
      t->nth[k] = 512;
      ok = plan_boxes(ctx->GL, most, elem, 512, k == 0, &B);
    }
    // FP32: one exchange an iteration where the halo's r fits beside p
    if (!k && !ok) {
      ok = plan_boxes(ctx->GL, most, elem, 512, false, &B);
      B.level = 0;
    }
    t->ok[k] = ok;
  }
}

// The exchange lies behind the context's states, zeroed with them (an allocation and a
// memset of its own, and its release, took 30 us a context).
size_t bbpp_persist_bytes(const bbpp_ctx *ctx) {
  return ctx->persist->ok[0] || ctx->persist->ok[1] ? sizeof(bbpp_exchange) : 0;
}
void bbpp_persist_attach(bbpp_ctx *ctx, void *p) { ctx->persist->ex = static_cast<bbpp_exchange *>(p); }

void bbpp_persist_free(bbpp_ctx *ctx) {
  if (!ctx->persist) return;
  delete ctx->persist;
  ctx->persist = nullptr;
}

bool bbpp_one_step(const bbpp_ctx *ctx) { return ctx->fused == 0 || (ctx->fused == 1 && bbpp_tma_fused_ok(ctx)); }

// Profiling times kernels one by one, so it runs the kernels of one iteration.  FP32 with a checkpoint every
// iteration: only small grids without the tensor-map kernels gain by a launch an iteration (ms a solve, resident and
// one by one: 45x33x27 10.0 and 15.6, 90x75x58 31.4 and 35.4, 121x111x101 33.8 and 33.1).
bool bbpp_persist_ok(const bbpp_ctx *ctx, int elem, int replace_every) {
  if (elem == 4 && bbpp_one_step(ctx)) return false;
  if (elem == 4 && replace_every == 1 && (bbpp_tma_fused_ok(ctx) || ctx->GL.n > 1 << 19)) return false;
  return ctx->persist && ctx->persist->ok[elem == 8 ? 1 : 0] && !ctx->profiling;
}

// Before a solve's first resident kernel: its shared memory, and arrivals count from zero
// (a launch whose wait ran out leaves them uneven; epochs run on).  False: no resident
// kernel here.  The attribute is a per-function cap shared by all contexts, so it is the
// maximum, set once per device; only the kernel that runs is loaded for it (all of a
// context's, when it was made, took 5 ms of a process's first).
bool bbpp_persist_begin(bbpp_ctx *ctx, int elem, bool mask) {
  bbpp_persist_state *t = ctx->persist;
  const int k = elem == 8 ? 1 : 0, nth = t->nth[k];
  const Boxes &B = t->box[k];
  const bool iso = ctx->GL.iso != 0;
  static std::atomic<unsigned long long> ready[64];
  int dev = 0;
  cudaGetDevice(&dev);
  const unsigned long long bit =
      1ull << (32 * k + 16 * B.one + 4 * (nth == 256 ? 3 : B.level) + 2 * (int)mask + (int)iso);
  if (dev >= 64 || !(ready[dev].load() & bit)) {
    const void *f = k ? (const void *)pick(0.0, nth, B, mask, iso) : (const void *)pick(0.f, nth, B, mask, iso);
    const int all = kSmemCap - (int)static_smem(nth);
    int per_sm = 0;
    if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, all) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, f, nth, (size_t)all) != cudaSuccess || per_sm < 1) {
      cudaGetLastError();
      t->ok[k] = false;
      return false;
    }
    if (dev < 64) ready[dev].fetch_or(bit);
  }
  cudaError_t e = cudaMemsetAsync(&t->ex->base, 0, sizeof(t->ex->base), ctx->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(&t->ex->arrived, 0, sizeof(t->ex->arrived), ctx->stream);
  return e == cudaSuccess;  // the solve's next call reports it
}

// Was the resident launch refused (the last bbpp_persist, or, with e, the launch of a graph of it)?  Then the
// context makes no more of them.
bool bbpp_persist_refused(bbpp_ctx *ctx, int elem, cudaError_t e) {
  bbpp_persist_state *t = ctx->persist;
  if (!t->refused && e != cudaErrorCooperativeLaunchTooLarge && e != cudaErrorNotSupported) return false;
  cudaGetLastError();
  ctx->err.clear();
  t->refused = false;
  t->ok[elem == 8 ? 1 : 0] = false;
  return true;
}

template <typename T>
int bbpp_persist(bbpp_ctx *ctx, const uint8_t *mask, T *r, T *const p[2], T *Ap, T *x, DevState *st,
                 int replace_every) {
  const int k = sizeof(T) == 8 ? 1 : 0;
  const Boxes &B = ctx->persist->box[k];
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(B.nb);
  cfg.blockDim = dim3(ctx->persist->nth[k]);
  cfg.dynamicSmemBytes = (size_t)B.smem;
  cfg.stream = ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const cudaError_t e =
      ctx->inject == INJECT_REFUSED
          ? cudaErrorCooperativeLaunchTooLarge
          : cudaLaunchKernelEx(&cfg, pick(T(0), ctx->persist->nth[k], B, mask != nullptr, ctx->GL.iso != 0), ctx->GL,
                               B, p[0], p[1], r, Ap, x, mask, st, ctx->persist->ex, replace_every);
  if (e != cudaSuccess) {
    ctx->persist->refused = e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported;
    bbpp_record_error(ctx, e, "k_persist", __LINE__);
    return BBPP_CUDA_ERROR;
  }
  return 0;
}
template int bbpp_persist<float>(bbpp_ctx *, const uint8_t *, float *, float *const[2], float *, float *, DevState *,
                                 int);
template int bbpp_persist<double>(bbpp_ctx *, const uint8_t *, double *, double *const[2], double *, double *,
                                  DevState *, int);
