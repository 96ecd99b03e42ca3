// bbpp_pair.cu -- two FP32 PCG iterations in two kernels that read r and p
// twice and write them once (the s = 2 form of Chronopoulos and Gear's s-step
// conjugate gradients, J. Comput. Appl. Math. 25, 1989), for grids of whole
// 16-byte rows that do not fit the chip.
//
// The vectors are z = r / dL (dL the diagonal of L; r = z away from walls), p
// and x.  With w = L p, q = w / dL, t = L q, s = L z, two iterations need only
// the products (r,z), (r,r), (p,w), (z,w), (q,w), (z,s), (z,t), (q,t), (s,s/dL),
// (s,t/dL), (t,t/dL): they give alpha and beta of both iterations (pair_plan).
//   k_pair<false>  forms w, t and s on the fly and sums the products: reads z, p
//                  and the mask (9 B/cell), writes nothing;
//   k_pair<true>   forms them again and applies both steps: reads z, p, x and
//                  the mask, writes z, p, x (25 B/cell).
// 34 B/cell for two iterations, against 66 for two launches of a kernel that
// carries one iteration (r, Ap, p, x read and written).  The products of a pair are
// exact sums at its start, so no error of the expansions carries over; the
// iteration counts are those of the one-step form (644 against 643 at 256^3 and
// 1058 against 1057 at 512^3 to 1e-10).
//
// What bounds it: with the bytes halved, the three stencils that both kernels form
// a cell.  At 256^3 (1000 spheres) a pair takes 77 + 80 us, 78 us an iteration
// against 116 of the fused kernel (k1_fused); at 512^3 470 + 594 us, 573 an iteration
// against 938; on rows that the tensor-map kernels do not take (200x250x180, walls)
// 60 against 153.  Half of the issue slots are used, DRAM at 2 and 4.7 TB/s.  Two
// FP32 operations an instruction (add, fma .f32x2), two rows a thread, the vectors
// read again from the stages rather than held (no spills), and steps away from walls
// on constant stages took it there from 157 us.  Slabs of 14 rows at 256^3: 19 x 8 CTAs
// fill the 152 SMs; 6 rows with two CTAs an SM measured 85 us, 10 rows 102.
//
// A CTA owns TY whole rows and marches through its planes.  Slabs of rows are
// contiguous, so a plane of p (TY + 4 rows) and of z (TY + 2 rows) is one or
// two 1-D bulk copies into a ring of stages, each completing on an mbarrier.  A
// thread owns one float4 of two rows (the rows next to the slab included, for w
// there) and keeps its z neighbours of p, q and z in registers; y neighbours come
// from shared memory, x neighbours from shuffles.  w of plane c and t, s and the
// step of plane c - 1 are formed between two CTA barriers.  The dots kernel walks
// the planes in the reverse order of the step kernel, so that each starts on
// the planes the other touched last, still in L2.
//
// Every wait is bounded (one second of globaltimer, or the state's wait_ns): a
// CTA whose wait runs out marks itself, waits for its copies in flight with a
// bound ten times longer and ends the solve with DONE_TIMEOUT.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdlib>

#include "bbpp_internal.h"
#include "bbpp_fast.cuh"
#include "bbpp_pair_plan.cuh"

using namespace bbpp;

namespace {

constexpr int PNT = 512;      // threads of a CTA at most, two rows each
constexpr int NDOT = 11;
constexpr int kPairSmem = 225 * 1024;

__device__ __forceinline__ unsigned int smem_u32(const void *p) {
  return (unsigned int)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void bar_init(unsigned long long *b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(unsigned long long *b, unsigned int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool bar_try(unsigned long long *b, unsigned int parity) {
  unsigned int ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(b)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ bool bar_wait(unsigned long long *b, unsigned int parity, unsigned long long limit) {
  if (bar_try(b, parity)) return true;
  const unsigned long long t0 = now_ns();
  for (unsigned int k = 1;; k++) {
    if (bar_try(b, parity)) return true;
    if ((k & 255u) == 0 && now_ns() - t0 > limit) return false;
  }
}
// 1-D bulk copy, global to shared: 16-byte aligned, a multiple of 16 bytes
__device__ __forceinline__ void bulk_load(float *dst, const float *src, unsigned int bytes, unsigned long long *bar,
                                          unsigned long long pol) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::
          "r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar)), "l"(pol)
      : "memory");
}

constexpr int RING = 4;       // stages of p and of z
constexpr int XRING = 3;      // of x

struct PairShape {
  int ty, kz, nzc;  // own rows, planes per CTA, z chunks
  int smem;
};

// two FP32 operations an instruction (rounded as the scalar ones)
__device__ __forceinline__ float2 lo2(const float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(const float4 v) { return make_float2(v.z, v.w); }
__device__ __forceinline__ float4 join(const float2 a, const float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float4 add4(const float4 a, const float4 b) {
  return join(__fadd2_rn(lo2(a), lo2(b)), __fadd2_rn(hi2(a), hi2(b)));
}
__device__ __forceinline__ float4 fma4(const float2 a, const float4 b, const float4 c) {
  return join(__ffma2_rn(a, lo2(b), lo2(c)), __ffma2_rn(a, hi2(b), hi2(c)));
}

}  // namespace

// What the end of a dots kernel reads of the state, at once: one load after another,
// between the stores, would take an L2 latency each.
struct PairIn {
  int iter, stop, max_iter, fq, fresh, maxgap, last_rep, inject;
  double tol2bb, expected, rep_d2, rr_ref;
};
__device__ __forceinline__ PairIn pair_in(const DevState *st) {
  return {st->iter,     st->stop,    st->max_iter, st->fq,     st->pair_fresh, st->rep_maxgap,
          st->last_rep, st->inject,  st->tol2bb,  st->rz_next,  st->rep_d2, st->rr_ref};
}

// The end of a dots kernel: convergence of the residual at the pair's start,
// then the coefficients and the number of steps (1 also where a second would pass a
// checkpoint or the iteration limit).
__device__ static void pair_finish(DevState *st, const PairIn &in, const double *d, int replace_every) {
  const int it = in.iter;
  const double rz = d[0], rr = d[0] + d[1];
  st->rz_last = rz;
  st->rr = rr;
  st->rz = rz;
  if (isnan(rz)) {
    st->done = DONE_NAN;
    return;
  }
  if (it > 0 && (in.stop == 0 ? rz : rr) <= in.tol2bb) {
    st->done = it > in.max_iter ? DONE_MAX_ITER : (in.stop == 0 ? DONE_CONVERGED : DONE_PENDING);
    st->rz_next = rz;  // what a confirmation compares with
    return;
  }
  if (it > in.max_iter) {
    st->done = DONE_MAX_ITER;
    return;
  }
  const bool spoil = in.inject == INJECT_DIRECTION && in.fq % 6 == 5;
  const PairPlan o = pair_plan(d, in.fresh == in.fq, spoil ? 0.0 : in.expected);
  const int n = ((it + 1) % replace_every == 0 || it + 1 > in.max_iter) ? 1 : o.steps;
  st->pAp = d[2];
  st->pair[0] = o.a0;
  st->pair[1] = o.b0;
  st->pair[2] = o.a1;
  st->pair[3] = o.b1;
  st->pair_steps = n;
  st->pair_anew = o.anew ? in.fq : -1;
  st->rz_next = n == o.steps ? o.rz : rz * o.b0;
  st->iter = it + n;
  st->fq = in.fq + 1;
  if (o.fresh) st->pair_fresh = in.fq + 1;
  // a checkpoint after this pair: replace the residual?
  st->rep_now = (it + n) % replace_every == 0 &&
                ((in.rep_d2 <= 0.0) || (rr <= in.rep_d2 * in.rr_ref) || (it + n - in.last_rep >= in.maxgap));
}

// STEP: apply the steps; else sum the products.  WXY: walls in x or y (cells of
// a plane then differ in class).
template <bool STEP, bool MASK, bool ISO, bool WXY>
__global__ void __launch_bounds__(PNT, 1) k_pair(const GeoL G, const PairShape S, const float *__restrict__ zin,
                                                 const float *__restrict__ pin, float *__restrict__ zout,
                                                 float *__restrict__ pout, float *__restrict__ x,
                                                 const uint8_t *__restrict__ mask, DevState *st, double *partials,
                                                 int replace_every) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ float s_dL[27], s_inv[27];
  __shared__ unsigned long long s_bar[RING];  // the copies that a step waits for
  __shared__ float2 s_coef[6];
  __shared__ int s_last;
  __shared__ int s_piece[2][8][3], s_np[4];
  if (*(volatile int *)&st->done) return;
  // the first pair, and restarts (pair_plan, resid_finish): p = z
  const bool fresh = *(volatile int *)(STEP ? &st->pair_anew : &st->pair_fresh) == *(volatile int *)&st->fq - (STEP ? 1 : 0);
  const long long wl = *(volatile long long *)&st->wait_ns;
  const unsigned long long limit = wl > 0 ? (unsigned long long)wl : 1000000000ull;
  const bool skip_one = *(volatile int *)&st->inject == INJECT_COPIES && blockIdx.x == 0 && blockIdx.y == 0;
  load_tabs<float>(G, s_dL, s_inv);

  const int tid = threadIdx.x, lane = tid & 31;
  const int nx = G.nx, ny = G.ny, nz = G.nz, nxv = nx >> 2;
  const int y0 = blockIdx.x * S.ty, rows = min(S.ty, ny - y0);  // own rows
  const int z0 = blockIdx.y * S.kz, z1 = min(z0 + S.kz, nz);
  const unsigned int plane = (unsigned int)nx * (unsigned int)ny;
  const int prow = (S.ty + 4) * nx, zrow = (S.ty + 2) * nx;  // floats of a stage of p and of z (and q)
  float *const sp = reinterpret_cast<float *>(smem_raw);     // [RING][ty + 4][nx]: rows y0 - 2 ..
  float *const sz = sp + RING * prow;                          // [RING][ty + 2][nx]: rows y0 - 1 ..
  float *const sq = sz + RING * zrow;                          // [2][ty + 2][nx]
  float *const sx = sq + 2 * zrow;                             // STEP: [XRING][ty][nx]: the own rows of x
  const int xrow = S.ty * nx;

  if (tid == 0) {
    for (int k = 0; k < RING; k++) bar_init(&s_bar[k]);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // The rows y0 - h .. y0 + rows + h - 1 of a plane as contiguous pieces (more than
  // one where y wraps), the same for every plane: place in the stage, place in
  // the plane, bytes.
  auto pieces = [&](int h, int (*out)[3], int &count, int &bytes) {
    int y = y0 - h, left = rows + 2 * h, d = 0;
    if (!G.py && y < 0) {
      d = -y;
      left += y;
      y = 0;
    }
    if (!G.py) left = min(left, ny - y);
    count = bytes = 0;
    while (left > 0) {
      const int yy = G.py ? ((y % ny) + ny) % ny : y;
      const int n = min(left, ny - yy);
      out[count][0] = d * nx;
      out[count][1] = yy * nx;
      out[count][2] = n * nx * 4;
      bytes += n * nx * 4;
      count++;
      d += n;
      y += n;
      left -= n;
    }
  };
  if (STEP && tid < 6) {  // -a0, b0, -a1, b1, a0, a1, each twice
    const float c = (float)st->pair[tid < 4 ? tid : 2 * (tid - 4)] * (tid == 0 || tid == 2 ? -1.f : 1.f);
    s_coef[tid] = make_float2(c, c);
  }
  if (tid == 0) {
    pieces(2, s_piece[0], s_np[0], s_np[2]);
    pieces(1, s_piece[1], s_np[1], s_np[3]);
  }
  // stage rows outside a y wall are never copied: zero for the whole march
  if (!G.py) {
    for (int k = 0; k < 2 * RING; k++) {
      const int h = k < RING ? 2 : 1;
      float *b = k < RING ? sp + k * prow : sz + (k - RING) * zrow;
      for (int e = tid; e < (S.ty + 2 * h) * nx; e += blockDim.x) {
        const int y = y0 - h + e / nx;
        if (y < 0 || y >= ny) b[e] = 0.f;
      }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  __syncthreads();

  // step i = 0, 1, ..: centre plane of w in march order, from one plane before
  // the chunk to one after; the dots kernel marches down
  const int nsteps = z1 - z0 + 2;
  constexpr int dir = STEP ? 1 : -1;
  const int zfirst = STEP ? z0 - 1 : z1;
  // plane in march order -> plane of the grid, or -1 outside a z wall; z reaches
  // two planes past either end
  auto grid_plane = [&](int z) {
    if (z >= 0 && z < nz) return z;
    if (!G.pz) return -1;
    while (z < 0) z += nz;
    while (z >= nz) z -= nz;
    return z;
  };
  // Copy k of p is plane zfirst + dir (k - 1), copy k of z plane zfirst + dir k.
  // Step i reads p's copies i, i + 1 (centre) and i + 2 and z's copies i - 1 and i;
  // its barrier covers p's copy i + 2 and z's copy i (step 0's p's copies 0 and 1
  // too), both issued at the end of step i - 3, when all have read what was in
  // those stages.  One thread of the last warp, whose rows need no t, s and step,
  // issues them.
  const bool issuer = tid == (int)blockDim.x - 32;
  auto copy = [&](int k, int which, bool expect, unsigned int &bytes, unsigned long long *bar) {
    const int zp = grid_plane(zfirst + dir * (which ? k : k - 1));
    if (zp < 0) return;
    if (expect) {
      bytes += (unsigned int)s_np[2 + which];
      return;
    }
    float *dst = which ? sz + (k % RING) * zrow : sp + (k % RING) * prow;
    const float *src = (which || fresh ? zin : pin) + (size_t)plane * zp;
    for (int q = 0; q < s_np[which]; q++)
      bulk_load(dst + s_piece[which][q][0], src + s_piece[which][q][1], (unsigned int)s_piece[which][q][2], bar,
                l2_policy(0));
  };
  bool bad = false;  // a wait ran out: no further waits, and the issuer stops
  int last = -1;     // the last step issued
  auto issue = [&](int i) {  // what step i waits for
    if (i >= nsteps || bad || (skip_one && i == 2)) return;
    last = i;
    unsigned long long *bar = &s_bar[i % RING];
    unsigned int bytes = 0;
    for (int pass = 0; pass < 2; pass++) {
      if (pass) bar_expect(bar, bytes);
      if (i == 0) {
        copy(0, 0, !pass, bytes, bar);
        copy(1, 0, !pass, bytes, bar);
      }
      copy(i + 2, 0, !pass, bytes, bar);
      copy(i, 1, !pass, bytes, bar);
      if (STEP && i >= 2) {  // x of the own plane, streamed
        if (!pass) bytes += (unsigned int)(rows * nx * 4);
        else
          bulk_load(sx + (i % XRING) * xrow, x + ((size_t)plane * (zfirst + dir * (i - 1)) + (size_t)nx * y0),
                    (unsigned int)(rows * nx * 4), bar, l2_policy(1));
      }
    }
  };
  if (issuer) {  // p's copy 4 (step 2) takes the stage of copy 0: after step 0
    issue(0);
    issue(1);
  }

  // This thread's two float4: rows wr and wr + 1 of the rows y0 - 1 .. y0 + ty (from
  // 0), column c4.  Two rows share their y neighbours and the step's overhead
  // (one row a thread, 1024 threads of 64 registers, measured 87 us an iteration
  // at 256^3).
  const int pr = tid / nxv, c4 = tid - pr * nxv;
  const int nrow2 = (S.ty + 2) / 2;
  const int lr = 2 * min(pr, nrow2 - 1);  // a row to read at (idle threads stay in range)
  int ygrid[2];
  bool live[2], own[2];
  unsigned int grow[2];
#pragma unroll
  for (int r = 0; r < 2; r++) {
    const int wr = 2 * pr + r;
    ygrid[r] = pr < nrow2 && wr < rows + 2 ? halo_index(y0 - 1 + wr, ny, G.py) : -1;
    live[r] = ygrid[r] >= 0;                          // w is formed here
    own[r] = pr < nrow2 && wr >= 1 && wr <= rows;     // t, s and the step too
    grow[r] = (unsigned int)nx * (unsigned int)max(ygrid[r], 0) + 4u * (unsigned int)c4;
  }
  const bool wlive = __any_sync(0xffffffffu, live[0] || live[1]);
  const bool wown[2] = {(bool)__any_sync(0xffffffffu, own[0]), (bool)__any_sync(0xffffffffu, own[1])};
  const int oq = lr * nx + 4 * c4;  // in a stage of z or q; a row on in p's, a row back in x's
  // y neighbours of the two rows in a stage of z or q (in range for rows not owned)
  const int osq = max(lr - 1, 0) * nx + 4 * c4, onq = min(lr + 2, S.ty + 1) * nx + 4 * c4;
  // x neighbours across a warp's or a row's end come from shared memory
  const bool wmem = lane == 0 || c4 == 0, emem = lane == 31 || c4 == nxv - 1;
  const int wat = c4 > 0 ? -1 : nx - 1, eat = c4 < nxv - 1 ? 4 : 4 - nx;
  const bool wwall = WXY && !G.px && c4 == 0, ewall = WXY && !G.px && c4 == nxv - 1;
  // class of the thread's cells without z
  const int cy[2] = {WXY && live[0] ? 3 * wall_count(ygrid[0], ny, G.py) : 0,
                     WXY && live[1] ? 3 * wall_count(ygrid[1], ny, G.py) : 0};
  const int cx0 = WXY ? wall_count(4 * c4, nx, G.px) : 0, cx3 = WXY ? wall_count(4 * c4 + 3, nx, G.px) : 0;
  auto cell_class = [&](int r, int k, int wz) { return WXY ? cy[r] + wz + (k == 0 ? cx0 : (k == 3 ? cx3 : 0)) : wz; };
  auto ld4 = [](const float *v) { return *reinterpret_cast<const float4 *>(v); };

  // L v at row r's float4 from its centre c (at v in its stage) and its z (b, t) and
  // y (n, s) neighbours.  Plain: no cell of the plane is at a wall.
  auto stencil = [&](auto plain, int r, const float4 c, const float4 b, const float4 t, const float4 n,
                     const float4 s, const float *v, int wz) {
    float w = __shfl_up_sync(0xffffffffu, c.w, 1);
    float e = __shfl_down_sync(0xffffffffu, c.x, 1);
    if (wmem) w = v[wat];
    if (emem) e = v[eat];
    if (wwall) w = 0.f;
    if (ewall) e = 0.f;
    if (ISO) {
      const float4 ew = make_float4(c.y + w, c.z + c.x, c.w + c.y, e + c.z);
      const float4 sum = add4(add4(ew, add4(n, s)), add4(t, b));
      if (decltype(plain)::value) return fma4(make_float2(-G.fax, -G.fax), sum, c);
      return make_float4(fmaf(s_dL[cell_class(r, 0, wz)], c.x, -G.fax * sum.x),
                         fmaf(s_dL[cell_class(r, 1, wz)], c.y, -G.fax * sum.y),
                         fmaf(s_dL[cell_class(r, 2, wz)], c.z, -G.fax * sum.z),
                         fmaf(s_dL[cell_class(r, 3, wz)], c.w, -G.fax * sum.w));
    }
    const float4 ew = make_float4(G.fax * (c.y + w), G.fax * (c.z + c.x), G.fax * (c.w + c.y), G.fax * (e + c.z));
    const float4 sum = fma4(make_float2(G.faz, G.faz), add4(t, b), fma4(make_float2(G.fay, G.fay), add4(n, s), ew));
    if (decltype(plain)::value) return make_float4(c.x - sum.x, c.y - sum.y, c.z - sum.z, c.w - sum.w);
    return make_float4(fmaf(s_dL[cell_class(r, 0, wz)], c.x, -sum.x), fmaf(s_dL[cell_class(r, 1, wz)], c.y, -sum.y),
                       fmaf(s_dL[cell_class(r, 2, wz)], c.z, -sum.z), fmaf(s_dL[cell_class(r, 3, wz)], c.w, -sum.w));
  };
  auto over_dL = [&](int r, const float4 v, int wz) {
    return make_float4(v.x * s_inv[cell_class(r, 0, wz)], v.y * s_inv[cell_class(r, 1, wz)],
                       v.z * s_inv[cell_class(r, 2, wz)], v.w * s_inv[cell_class(r, 3, wz)]);
  };
  // zero where the mask word's byte is set
  auto fluid_only = [&](float4 &v, unsigned int m) {
    v = make_float4(m & 0xffu ? 0.f : v.x, m & 0xff00u ? 0.f : v.y, m & 0xff0000u ? 0.f : v.z,
                    m & 0xff000000u ? 0.f : v.w);
  };

  const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float acc[STEP ? 1 : NDOT];
#pragma unroll
  for (int k = 0; k < (STEP ? 1 : NDOT); k++) acc[k] = 0.f;
  const bool single = STEP && st->pair_steps == 1;

  // t, s and the steps (or products) of the own rows of a plane: p its p, q0 and v0
  // the plane before's q and z; qr, zr and z2r are the stages of its q, its z and
  // the next plane's z, q2 the next plane's q; xr its x, g its place in the grid.
  // Leaves its q and z in q0 and v0.
  auto finish = [&](auto plain, int wo, const float4 (&p)[2], float4 (&q0)[2], const float4 (&q2)[2], float4 (&v0)[2],
                    const float *qr, const float *zr, const float *z2r, const float *xr, const unsigned int (&m)[2],
                    const unsigned int (&g)[2]) {
    const float4 z[2] = {ld4(zr + oq), ld4(zr + oq + nx)}, q[2] = {ld4(qr + oq), ld4(qr + oq + nx)};
#pragma unroll
    for (int r = 0; r < 2; r++) {
      if (wown[r]) {
        const float4 zo = ld4(zr + (r ? onq : osq)), qo = ld4(qr + (r ? onq : osq));
        float4 s = stencil(plain, r, z[r], v0[r], ld4(z2r + oq + r * nx), r ? zo : z[1], r ? z[0] : zo,
                           zr + oq + r * nx, wo);
        float4 t = stencil(plain, r, q[r], q0[r], q2[r], r ? qo : q[1], r ? q[0] : qo, qr + oq + r * nx, wo);
        if (MASK) {
          fluid_only(t, m[r]);
          fluid_only(s, m[r]);
        }
        if (STEP) {
          if (!decltype(plain)::value) {
            t = over_dL(r, t, wo);
            s = over_dL(r, s, wo);
          }
          // z1 = z - a0 q, p1 = z1 + b0 p, w1 / dL = s - a0 t + b0 q; z2 = z1 - a1 w1 / dL,
          // p2 = z2 + b1 p1, x += a0 p + a1 p1
          if (own[r]) {
            float4 zw = fma4(s_coef[0], q[r], z[r]);
            float4 xo = fma4(s_coef[4], p[r], ld4(xr + oq + (r - 1) * nx));
            float4 pw = fma4(s_coef[1], p[r], zw);
            if (!single) {
              const float4 w1 = fma4(s_coef[1], q[r], fma4(s_coef[0], t, s));
              xo = fma4(s_coef[5], pw, xo);
              zw = fma4(s_coef[2], w1, zw);
              pw = fma4(s_coef[3], pw, zw);
            }
            *reinterpret_cast<float4 *>(zout + g[r]) = zw;
            *reinterpret_cast<float4 *>(pout + g[r]) = pw;
            __stcs(reinterpret_cast<float4 *>(x + g[r]), xo);
          }
        } else if (own[r]) {
          const float tv[4] = {t.x, t.y, t.z, t.w}, sv[4] = {s.x, s.y, s.z, s.w},
                      qv[4] = {q[r].x, q[r].y, q[r].z, q[r].w}, zv[4] = {z[r].x, z[r].y, z[r].z, z[r].w},
                      pv[4] = {p[r].x, p[r].y, p[r].z, p[r].w};
#pragma unroll
          for (int k = 0; k < 4; k++) {
            if (decltype(plain)::value) {  // r = z, w = q, s / dL = s, t / dL = t
              acc[0] = fmaf(zv[k], zv[k], acc[0]);
              acc[2] = fmaf(pv[k], qv[k], acc[2]);
              acc[3] = fmaf(zv[k], qv[k], acc[3]);
              acc[4] = fmaf(qv[k], qv[k], acc[4]);
              acc[8] = fmaf(sv[k], sv[k], acc[8]);
              acc[9] = fmaf(sv[k], tv[k], acc[9]);
              acc[10] = fmaf(tv[k], tv[k], acc[10]);
            } else {
              const float iv = s_inv[cell_class(r, k, wo)], dl = s_dL[cell_class(r, k, wo)];
              const float rv = zv[k] * dl, w = qv[k] * dl, si = sv[k] * iv, ti = tv[k] * iv;
              acc[0] = fmaf(rv, zv[k], acc[0]);
              acc[1] = fmaf(rv, rv - zv[k], acc[1]);  // (r, r) - (r, z)
              acc[2] = fmaf(pv[k], w, acc[2]);
              acc[3] = fmaf(zv[k], w, acc[3]);
              acc[4] = fmaf(qv[k], w, acc[4]);
              acc[8] = fmaf(sv[k], si, acc[8]);
              acc[9] = fmaf(sv[k], ti, acc[9]);
              acc[10] = fmaf(tv[k], ti, acc[10]);
            }
            acc[5] = fmaf(zv[k], sv[k], acc[5]);
            acc[6] = fmaf(zv[k], tv[k], acc[6]);
            acc[7] = fmaf(qv[k], tv[k], acc[7]);
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
      v0[r] = z[r];
      q0[r] = q[r];
    }
  };

  // What a thread carries from step to step: p, q and z of the plane before the
  // centre's neighbours (the rest is read again from the stages), the mask words of
  // the own plane and the centre (all set where w is zero for another reason).
  float4 p0[2] = {zero4, zero4}, q0[2] = {zero4, zero4}, v0[2] = {zero4, zero4};
  unsigned int mo[2] = {0u, 0u}, mc[2], mn[2];
  const unsigned int *const mask4 = reinterpret_cast<const unsigned int *>(mask);
  auto load_mask = [&](int zp, unsigned int (&m)[2]) {  // of plane zp of the grid
#pragma unroll
    for (int r = 0; r < 2; r++) {
      m[r] = live[r] ? 0u : ~0u;
      if (MASK && live[r] && zp >= 0) m[r] = __ldg(mask4 + ((plane * (unsigned int)zp + grow[r]) >> 2));
    }
  };
  load_mask(grid_plane(zfirst), mc);
  // step i: w and q of the centre plane, then t, s and the step of the plane before.
  // Any plane:
  auto step_any = [&](int i) {
    const int z = zfirst + dir * i;
    const int zg = grid_plane(z), zn = grid_plane(z + dir);
    load_mask(i + 1 < nsteps ? zn : -1, mn);
    if (!bad && !bar_wait(&s_bar[i % RING], (unsigned int)(i / RING) & 1u, limit)) bad = true;
    const float *pc = sp + ((i + 1) % RING) * prow + nx + oq, *pn = sp + ((i + 2) % RING) * prow + nx + oq;
    float4 p1[2] = {zero4, zero4}, q2[2] = {zero4, zero4};
    if (i == 0 && grid_plane(zfirst - dir) >= 0) {
      p0[0] = ld4(sp + nx + oq);
      p0[1] = ld4(sp + 2 * nx + oq);
    }
    if (zg >= 0) {
      p1[0] = ld4(pc);
      p1[1] = ld4(pc + nx);
    }
    if (wlive && zg >= 0) {
      const int wz = 9 * wall_count(zg, nz, G.pz);
      const float4 ps = ld4(pc - nx), pnn = ld4(pc + 2 * nx);
#pragma unroll
      for (int r = 0; r < 2; r++) {
        const float4 p2 = zn >= 0 ? ld4(pn + r * nx) : zero4;
        if (!WXY && wz == 0) {
          q2[r] = stencil(std::true_type(), r, p1[r], p0[r], p2, r ? pnn : p1[1], r ? p1[0] : ps, pc + r * nx, 0);
        } else {
          q2[r] = over_dL(r, stencil(std::false_type(), r, p1[r], p0[r], p2, r ? pnn : p1[1], r ? p1[0] : ps,
                                     pc + r * nx, wz), wz);
        }
        fluid_only(q2[r], mc[r]);
      }
    }
    if (pr < nrow2) {
      *reinterpret_cast<float4 *>(sq + (i & 1) * zrow + oq) = q2[0];
      *reinterpret_cast<float4 *>(sq + (i & 1) * zrow + oq + nx) = q2[1];
    }
    // z outside a wall (the last step's; no copy goes to that stage any more)
    float *z2r = sz + (i % RING) * zrow;
    if (i > 0 && zg < 0) {
#pragma unroll
      for (int r = 0; r < 2; r++)
        if (own[r]) *reinterpret_cast<float4 *>(z2r + oq + r * nx) = zero4;
    }
    if (i >= 2) {
      const int zo = z - dir;
      const float *qr = sq + ((i - 1) & 1) * zrow, *zr = sz + ((i - 1) % RING) * zrow, *xr = sx + (i % XRING) * xrow;
      const unsigned int g[2] = {plane * (unsigned int)zo + grow[0], plane * (unsigned int)zo + grow[1]};
      if (!WXY && (G.pz || (zo > 0 && zo < nz - 1)))
        finish(std::true_type(), 0, p0, q0, q2, v0, qr, zr, z2r, xr, mo, g);
      else
        finish(std::false_type(), 9 * wall_count(zo, nz, G.pz), p0, q0, q2, v0, qr, zr, z2r, xr, mo, g);
    } else if (i == 1) {  // the plane before the chunk
#pragma unroll
      for (int r = 0; r < 2; r++) {
        q0[r] = ld4(sq + oq + r * nx);
        if (grid_plane(zfirst) >= 0) v0[r] = ld4(sz + oq + r * nx);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; r++) {
      p0[r] = p1[r];
      mo[r] = mc[r];
      mc[r] = mn[r];
    }
    __syncthreads();
    if (issuer) {
      if (i == 0) issue(2);
      issue(i + 3);
    }
  };
  // the same away from walls and wraps: planes z - dir, z and z + dir lie inside the
  // grid (0 < z, z - dir < nz - 1 at z walls), 2 <= i, i + 1 < nsteps, i % RING = SL.
  // g: the thread's places in the centre plane
  const unsigned int gstep = STEP ? plane : 0u - plane;
  unsigned int g[2] = {0u, 0u}, par = 0;
  auto step_in = [&](auto slot, int i, int xs) {
    constexpr int SL = decltype(slot)::value;
    if (MASK) {
#pragma unroll
      for (int r = 0; r < 2; r++) mn[r] = live[r] ? __ldg(mask4 + ((g[r] + gstep) >> 2)) : ~0u;
    }
    if (!bar_try(&s_bar[SL], par)) {
      if (!bad && !bar_wait(&s_bar[SL], par, limit)) bad = true;
    }
    const float *pc = sp + ((SL + 1) % RING) * prow + nx + oq, *pn = sp + ((SL + 2) % RING) * prow + nx + oq;
    const float4 p1[2] = {ld4(pc), ld4(pc + nx)};
    float4 q2[2] = {zero4, zero4};
    if (wlive) {
      const float4 ps = ld4(pc - nx), pnn = ld4(pc + 2 * nx);
#pragma unroll
      for (int r = 0; r < 2; r++) {
        q2[r] = stencil(std::true_type(), r, p1[r], p0[r], ld4(pn + r * nx), r ? pnn : p1[1], r ? p1[0] : ps,
                        pc + r * nx, 0);
        fluid_only(q2[r], mc[r]);
      }
    }
    if (pr < nrow2) {
      *reinterpret_cast<float4 *>(sq + (SL & 1) * zrow + oq) = q2[0];
      *reinterpret_cast<float4 *>(sq + (SL & 1) * zrow + oq + nx) = q2[1];
    }
    const unsigned int gp[2] = {g[0] - gstep, g[1] - gstep};
    finish(std::true_type(), 0, p0, q0, q2, v0, sq + ((SL + 1) & 1) * zrow, sz + ((SL + RING - 1) % RING) * zrow,
           sz + SL * zrow, sx + xs * xrow, mo, gp);
#pragma unroll
    for (int r = 0; r < 2; r++) {
      p0[r] = p1[r];
      if (MASK) {
        mo[r] = mc[r];
        mc[r] = mn[r];
      }
      g[r] += gstep;
    }
    __syncthreads();
    if (issuer) issue(i + 3);
  };
  auto inside = [&](int i) {  // step_in's condition for steps i .. i + RING - 1
    if (WXY || i < 2 || i + RING >= nsteps) return false;
    const int a = zfirst + dir * (i - 1), b = zfirst + dir * (i + RING), lo = min(a, b), hi = max(a, b);
    return G.pz ? lo >= 0 && hi < nz : lo > 0 && hi < nz - 1;
  };
#pragma unroll 1
  for (int i = 0; i < nsteps;) {
    if (i % RING == 0 && inside(i)) {
#pragma unroll
      for (int r = 0; r < 2; r++) g[r] = plane * (unsigned int)(zfirst + dir * i) + grow[r];
      par = (unsigned int)(i / RING) & 1u;
      const int xs = i % XRING;
      step_in(std::integral_constant<int, 0>(), i, xs);
      step_in(std::integral_constant<int, 1>(), i + 1, xs == 2 ? 0 : xs + 1);
      step_in(std::integral_constant<int, 2>(), i + 2, xs == 0 ? 2 : xs - 1);
      step_in(std::integral_constant<int, 3>(), i + 3, xs);
      i += RING;
    } else {
      step_any(i);
      i++;
    }
  }

  if (__syncthreads_or(bad)) {
    if (issuer) {
      // the copies still in flight: the CTA must not exit while one writes its
      // shared memory
      for (int k = max(0, last - RING + 1); k <= last; k++)
        if (!(skip_one && k == 2)) bar_wait(&s_bar[k % RING], (unsigned int)(k / RING) & 1u, 10ull * limit);
      atomicExch(&st->done, (int)DONE_TIMEOUT);
    }
    return;
  }
  if (STEP) return;
  // The CTA's sums: per thread in FP32, across threads by sum_floats (FP64 adds for
  // 512 threads x 11 products would take the FP64 pipe 2.5 us a launch).
  float *sv = reinterpret_cast<float *>(smem_raw);  // [NDOT][threads]
  const int nth = blockDim.x;
#pragma unroll
  for (int k = 0; k < (STEP ? 1 : NDOT); k++) sv[k * nth + tid] = acc[k];
  __syncthreads();
  const unsigned int nb = gridDim.x * gridDim.y, bid = blockIdx.x + gridDim.x * blockIdx.y;
  for (int k = tid >> 5; k < NDOT; k += nth >> 5) {  // a warp a product
    const double v = warp_sum(sum_floats(sv + k * nth, nth, lane));
    if (lane == 0) partials[(size_t)k * nb + bid] = v;
  }
  __threadfence();
  __syncthreads();
  if (tid == 0) {
    const unsigned int t = atomicAdd(&st->ticket, 1u);
    s_last = t == nb - 1;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const PairIn in = pair_in(st);
  double *sd = reinterpret_cast<double *>(smem_raw);
  for (int k = tid >> 5; k < NDOT; k += nth >> 5) {
    double a = 0.0;
    for (unsigned int b0 = lane; b0 < nb; b0 += 256) {  // eight loads at once
      double v[8];
#pragma unroll
      for (int i = 0; i < 8; i++) v[i] = b0 + 32 * i < nb ? __ldcg(&partials[(size_t)k * nb + b0 + 32 * i]) : 0.0;
#pragma unroll
      for (int i = 0; i < 8; i++)
        if (b0 + 32 * i < nb) a += v[i];
    }
    a = warp_sum(a);
    if (lane == 0) sd[k] = a;
  }
  __syncthreads();
  if (tid == 0) {
    st->ticket = 0;
    pair_finish(st, in, sd, replace_every);
  }
}

// ------------------------------------------------------------------- host --
struct bbpp_pair_state {
  PairShape shape;
  int threads = 0;
  bool ok = false;
};

namespace {
typedef void (*PairKern)(const GeoL, const PairShape, const float *, const float *, float *, float *, float *,
                         const uint8_t *, DevState *, double *, int);
template <bool STEP, bool MASK>
PairKern pick2(bool iso, bool wxy) {
  if (iso) return wxy ? k_pair<STEP, MASK, true, true> : k_pair<STEP, MASK, true, false>;
  return wxy ? k_pair<STEP, MASK, false, true> : k_pair<STEP, MASK, false, false>;
}
PairKern pick_pair(bool step, bool mask, bool iso, bool wxy) {
  if (step) return mask ? pick2<true, true>(iso, wxy) : pick2<true, false>(iso, wxy);
  return mask ? pick2<false, true>(iso, wxy) : pick2<false, false>(iso, wxy);
}

// The kernel's shared memory cap, once per device and kernel; only the kernels that run
// are loaded for it (all sixteen, when a context was made, took 9 ms of a process's first).
bool pair_cap(const GeoL &G, bool step, bool mask) {
  static std::atomic<unsigned int> capped[64];
  const bool iso = G.iso != 0, wxy = !(G.px && G.py);
  const unsigned int bit = 1u << (8 * (int)step + 4 * (int)mask + 2 * (int)iso + (int)wxy);
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 64 && (capped[dev].load() & bit)) return true;
  if (cudaFuncSetAttribute(pick_pair(step, mask, iso, wxy), cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem) !=
      cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (dev < 64) capped[dev].fetch_or(bit);
  return true;
}
}  // namespace

void bbpp_pair_init(bbpp_ctx *ctx) {
  bbpp_pair_state *t = new bbpp_pair_state();
  ctx->pair = t;
  const char *e = getenv("BBPP_PAIR");
  if (e && e[0] == '0') return;
  const GeoL &G = ctx->GL;
  if (G.nx % 4 != 0 || G.nx > 1024) return;
  const int nxv = G.nx / 4;
  const char *ety = getenv("BBPP_PAIR_TY");
  int ty = std::min(2 * (PNT / nxv) - 2, (G.ny + 1) / 2 * 2);  // even
  if (ety) ty = std::max(2, std::min(ty, atoi(ety) / 2 * 2));
  if (ty < 2) return;
  const int threads = (nxv * (ty + 2) / 2 + 31) / 32 * 32;
  const size_t smem = ((size_t)RING * (ty + 4) + (size_t)(RING + 2) * (ty + 2) + (size_t)XRING * ty) * G.nx * 4;
  const size_t need = std::max(smem, sizeof(float) * NDOT * (size_t)threads);
  if (need > (size_t)kPairSmem) return;
  if (!pair_cap(G, true, true)) return;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, pick_pair(true, true, G.iso != 0, !(G.px && G.py)), threads,
                                                    need) != cudaSuccess ||
      per_sm < 1) {
    cudaGetLastError();
    return;
  }
  const int slabs = (G.ny + ty - 1) / ty;
  t->shape.ty = ty;
  t->shape.smem = (int)need;
  t->shape.nzc = bbpp_z_chunks(slabs, G.nz, (long long)ctx->sms * per_sm, 1, &t->shape.kz);
  t->threads = threads;
  t->ok = true;
}

void bbpp_pair_free(bbpp_ctx *ctx) {
  delete ctx->pair;
  ctx->pair = nullptr;
}

bool bbpp_pair_ok(const bbpp_ctx *ctx) { return ctx->pair && ctx->pair->ok; }

bool bbpp_pair_ready(const bbpp_ctx *ctx, bool mask) {
  return pair_cap(ctx->GL, false, mask) && pair_cap(ctx->GL, true, mask);
}

// CTAs x products over the three sums of a CTA that the context sizes by
size_t bbpp_pair_partials(const bbpp_ctx *ctx) {
  if (!bbpp_pair_ok(ctx)) return 0;
  const size_t slabs = (ctx->GL.ny + ctx->pair->shape.ty - 1) / ctx->pair->shape.ty;
  return (slabs * ctx->pair->shape.nzc * NDOT + 2) / 3;
}

// step false: the products of (zin, pin) and the coefficients; true: the steps
void bbpp_pair_launch(bbpp_ctx *ctx, bool step, const uint8_t *mask, const float *zin, const float *pin, float *zout,
                      float *pout, float *x, DevState *st, int replace_every) {
  const bbpp_pair_state *t = ctx->pair;
  const GeoL &G = ctx->GL;
  const dim3 grid((G.ny + t->shape.ty - 1) / t->shape.ty, t->shape.nzc);
  pick_pair(step, mask != nullptr, G.iso != 0, !(G.px && G.py))<<<grid, t->threads, t->shape.smem, ctx->stream>>>(
      G, t->shape, zin, pin, zout, pout, x, mask, st, ctx->partials, replace_every);
}
