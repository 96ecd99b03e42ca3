// bbpp_conv.cuh -- 3x3x3 convolutions of the learned initial guess as
// implicit GEMMs on BF16 tensor cores (mma.sync m16n8k16, FP32 accumulate).
//
// Activations are channels-last BF16 volumes, [volume][z][y][x][channel] with
// a channel stride `ld` and a channel offset, so a concatenation is two
// tensors writing disjoint channel ranges of one buffer.  Padding is periodic
// on the axes flagged periodic and zero otherwise.
//
//  k_conv3_fwd<CIN, COUT>   out = act(conv(in, W) + bias); a CTA computes a
//                           16x8xTZ tile of outputs (TZ = 8, 4, 2 for 16,
//                           32, 64 output channels) from a halo tile staged in
//                           shared memory 16 input channels at a time; the 27
//                           taps are 27 k16 steps whose A rows are shifted
//                           halo rows (ldmatrix gather).  dgrad uses the same
//                           kernel with the taps flipped and W transposed.
//  k_conv3_wgrad<CIN, COUT> dW[t] += sum_v g[v]^T in[v + t], all taps of 16 input
//                           channels per CTA over a range of tiles, warps split
//                           the taps.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace bbnet {

typedef __nv_bfloat16 bf16;

constexpr int CTX = 16, CTY = 8, CTZ = 2;                  // output tile of a CTA
constexpr int HTX = CTX + 2, HTY = CTY + 2, HTZ = CTZ + 2;  // with halo
constexpr int HVOX = HTX * HTY * HTZ;                      // 720 halo voxels
constexpr int RSB = 48;  // shared bytes per voxel row of a 16-channel chunk (32 + 16 pad)

struct ConvArgs {
  const bf16 *in;
  int ldi, ci_off;
  const bf16 *w;       // [27][COUT][CIN]
  const float *bias;   // [COUT] or null
  bf16 *out;
  int ldo, co_off;
  int nx, ny, nz, nb;  // volume, number of volumes
  int px, py, pz;      // periodic axes
  int relu;
};

struct WgradArgs {
  const bf16 *in;
  int ldi, ci_off;
  const bf16 *g;       // gradient of the conv output (after the activation gate)
  int ldg, cg_off;
  float *dW;           // [27][COUT][CIN], accumulated
  int nx, ny, nz, nb;
  int px, py, pz;
  int tiles_per_cta;
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void ldsm_x4(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3, const void *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_u32(p)));
}

__device__ __forceinline__ void ldsm_x4_t(uint32_t &r0, uint32_t &r1, uint32_t &r2, uint32_t &r3, const void *p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_u32(p)));
}

__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// index along one axis with periodic wrap or zero padding; false = padding
__device__ __forceinline__ bool pad_axis(int &g, int n, int periodic) {
  if (g >= 0 && g < n) return true;
  if (!periodic) return false;
  g = (g < 0) ? g + n : g - n;
  return g >= 0 && g < n;
}

// ------------------------------------------------------------- forward -----
// z planes of the forward kernel's output tile: deeper tiles reuse every
// weight fragment over more A fragments and cut the halo share, as long as
// the accumulators fit in registers
template <int COUT>
__host__ __device__ constexpr int fwd_tz() {
  return COUT <= 16 ? 8 : (COUT <= 32 ? 4 : 2);
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(256) k_conv3_fwd(const ConvArgs a) {
  static_assert(CIN % 16 == 0 && COUT % 16 == 0, "channels in multiples of 16");
  constexpr int TZ = fwd_tz<COUT>();
  constexpr int HVZ = HTX * HTY * (TZ + 2);  // halo voxels
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned char *s_in = smem;              // HVZ rows of RSB bytes
  unsigned char *s_w = smem + HVZ * RSB;   // 27 * COUT rows of RSB bytes
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int x0 = blockIdx.x * CTX, y0 = blockIdx.y * CTY;
  const int nzt = (a.nz + TZ - 1) / TZ;
  const int vb = blockIdx.z / nzt;
  const int z0 = (blockIdx.z - vb * nzt) * TZ;
  const long long vol = (long long)a.nx * a.ny * a.nz;
  const bf16 *inb = a.in + (long long)vb * vol * a.ldi + a.ci_off;

  float acc[TZ][COUT / 8][4];
#pragma unroll
  for (int i = 0; i < TZ; i++)
#pragma unroll
    for (int j = 0; j < COUT / 8; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[i][j][q] = 0.f;

  for (int c0 = 0; c0 < CIN; c0 += 16) {
    for (int idx = tid; idx < HVZ * 2; idx += 256) {
      const int e = idx >> 1, half = idx & 1;
      const int hx = e % HTX, t = e / HTX;
      const int hy = t % HTY, hz = t / HTY;
      int gx = x0 + hx - 1, gy = y0 + hy - 1, gz = z0 + hz - 1;
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (pad_axis(gx, a.nx, a.px) && pad_axis(gy, a.ny, a.py) && pad_axis(gz, a.nz, a.pz))
        v = *reinterpret_cast<const uint4 *>(inb + (((long long)gz * a.ny + gy) * a.nx + gx) * a.ldi + c0 + half * 8);
      *reinterpret_cast<uint4 *>(s_in + e * RSB + half * 16) = v;
    }
    for (int idx = tid; idx < 27 * COUT * 2; idx += 256) {
      const int row = idx >> 1, half = idx & 1;
      *reinterpret_cast<uint4 *>(s_w + row * RSB + half * 16) =
          *reinterpret_cast<const uint4 *>(a.w + (long long)row * CIN + c0 + half * 8);
    }
    __syncthreads();
#pragma unroll 1
    for (int tap = 0; tap < 27; tap++) {
      const int dz = tap / 9, dy = (tap / 3) % 3, dx = tap % 3;
      uint32_t bfr[COUT / 8][2];
#pragma unroll
      for (int j = 0; j < COUT / 8; j += 2) {
        const int n = tap * COUT + j * 8 + (lane & 7) + ((lane >> 4) << 3);
        ldsm_x4(bfr[j][0], bfr[j][1], bfr[j + 1][0], bfr[j + 1][1], s_w + n * RSB + ((lane >> 3) & 1) * 16);
      }
#pragma unroll
      for (int mi = 0; mi < TZ; mi++) {
        uint32_t afr[4];
        const int hv = ((mi + dz) * HTY + warp + dy) * HTX + (lane & 15) + dx;
        ldsm_x4(afr[0], afr[1], afr[2], afr[3], s_in + hv * RSB + (lane >> 4) * 16);
#pragma unroll
        for (int j = 0; j < COUT / 8; j++) mma16816(acc[mi][j], afr, bfr[j][0], bfr[j][1]);
      }
    }
    __syncthreads();
  }
  // epilogue: bias, activation, BF16 store
  const int y = y0 + warp;
  if (y >= a.ny) return;
  bf16 *outb = a.out + (long long)vb * vol * a.ldo + a.co_off;
#pragma unroll
  for (int mi = 0; mi < TZ; mi++) {
    const int z = z0 + mi;
    if (z >= a.nz) continue;
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int x = x0 + (lane >> 2) + 8 * h;
      if (x >= a.nx) continue;
      bf16 *o = outb + (((long long)z * a.ny + y) * a.nx + x) * a.ldo;
#pragma unroll
      for (int j = 0; j < COUT / 8; j++) {
        const int ch = j * 8 + (lane & 3) * 2;
        float v0 = acc[mi][j][2 * h], v1 = acc[mi][j][2 * h + 1];
        if (a.bias) {
          v0 += a.bias[ch];
          v1 += a.bias[ch + 1];
        }
        if (a.relu) {
          v0 = fmaxf(v0, 0.f);
          v1 = fmaxf(v1, 0.f);
        }
        *reinterpret_cast<__nv_bfloat162 *>(o + ch) = __floats2bfloat162_rn(v0, v1);
      }
    }
  }
}

template <int CIN, int COUT>
__host__ __device__ constexpr int conv_fwd_smem() {
  return HTX * HTY * (fwd_tz<COUT>() + 2) * RSB + 27 * COUT * RSB;
}

// --------------------------------------------------------------- wgrad -----
// dW[tap] += g^T (COUT x voxels) . in shifted by the tap (voxels x CIN), FP32.
// A CTA takes 16 input channels (blockIdx.y), a group of taps (blockIdx.z) and a
// run of tiles.  Per tile it stages the 256 voxels of g and the 720 halo voxels of
// the input once for all its taps: each warp owns WTAPS taps whole, so a g fragment
// serves them all, a tap is a shifted ldmatrix row, and no sums cross warps.  The
// next tile's copies (cp.async) are in flight while a tile is computed.  A plane's
// sums start from zero and are added to the CTA's in FP32: the tensor unit's
// accumulation loses a little at every step, and chains of whole tile runs gave
// up to ten times the error.
// One tap a CTA, as before, read g and the input 27 times over: 1435 us for 48 -> 16
// and 429 us for 16 -> 16 on four 64^3 volumes, against 189 and 70 us.
template <int COUT>
__host__ __device__ constexpr int wgrad_taps() {  // taps of a warp: its sums take 64 registers
  return 64 / COUT;
}
template <int COUT>
__host__ __device__ constexpr int wgrad_stage() {  // bytes of one tile's g and input
  return 256 * (COUT * 2 + 16) + HVOX * RSB;
}

// 16 bytes global to shared, zeros when !full
__device__ __forceinline__ void cp16(void *dst, const void *src, bool full) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(full ? 16 : 0)
               : "memory");
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(256) k_conv3_wgrad(const WgradArgs a) {
  constexpr int GRS = COUT * 2 + 16;  // shared bytes per voxel row of g
  constexpr int MT = COUT / 16;       // m tiles (output channels)
  constexpr int NTAP = wgrad_taps<COUT>();
  constexpr int STAGE = wgrad_stage<COUT>();
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int c0 = 16 * blockIdx.y, tap0 = 8 * NTAP * blockIdx.z + warp;  // taps tap0 + 8 i
  const int tx_n = (a.nx + CTX - 1) / CTX, ty_n = (a.ny + CTY - 1) / CTY, tz_n = (a.nz + CTZ - 1) / CTZ;
  const int ntiles = tx_n * ty_n * tz_n * a.nb;
  const long long vol = (long long)a.nx * a.ny * a.nz;
  const int t_begin = blockIdx.x * a.tiles_per_cta, t_end = min(t_begin + a.tiles_per_cta, ntiles);

  auto stage = [&](int tile, int slot) {  // g (zero outside the volume) and the halo of the input
    unsigned char *s_g = smem + slot * STAGE, *s_x = s_g + 256 * GRS;
    int tt = tile;
    const int bx = tt % tx_n * CTX;
    tt /= tx_n;
    const int by = tt % ty_n * CTY;
    tt /= ty_n;
    const int bz = tt % tz_n * CTZ;
    const long long vb = (long long)(tt / tz_n) * vol;
    {
      const int lx = tid % CTX, ly = (tid / CTX) % CTY, lz = tid / (CTX * CTY);
      const int ox = bx + lx, oy = by + ly, oz = bz + lz;
      const bool inside = ox < a.nx && oy < a.ny && oz < a.nz;
      const bf16 *src = a.g + a.cg_off + (inside ? (vb + ((long long)oz * a.ny + oy) * a.nx + ox) * a.ldg : 0);
#pragma unroll
      for (int q = 0; q < COUT / 8; q++) cp16(s_g + tid * GRS + q * 16, src + q * 8, inside);
    }
    for (int v = tid; v < HVOX; v += 256) {
      int gx = bx + v % HTX - 1, gy = by + (v / HTX) % HTY - 1, gz = bz + v / (HTX * HTY) - 1;
      const bool in = pad_axis(gx, a.nx, a.px) && pad_axis(gy, a.ny, a.py) && pad_axis(gz, a.nz, a.pz);
      const bf16 *src = a.in + a.ci_off + c0 + (in ? (vb + ((long long)gz * a.ny + gy) * a.nx + gx) * a.ldi : 0);
      cp16(s_x + v * RSB, src, in);
      cp16(s_x + v * RSB + 16, src + 8, in);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  float acc[NTAP][MT][2][4], sum[NTAP][MT][2][4];
#pragma unroll
  for (int i = 0; i < NTAP; i++)
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int n = 0; n < 2; n++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[i][m][n][q] = sum[i][m][n][q] = 0.f;
  int shift[NTAP];  // a tap's place in the halo; taps past the last repeat the first (not added)
#pragma unroll
  for (int i = 0; i < NTAP; i++) {
    const int tap = tap0 + 8 * i < 27 ? tap0 + 8 * i : 0;
    shift[i] = (tap / 9 * HTY + (tap / 3) % 3) * HTX + tap % 3;
  }
  if (t_begin < t_end) stage(t_begin, 0);
  for (int tile = t_begin; tile < t_end; tile++) {
    const int slot = (tile - t_begin) & 1;
    if (tile + 1 < t_end) {
      stage(tile + 1, slot ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
    const unsigned char *s_g = smem + slot * STAGE, *s_x = s_g + 256 * GRS;
    const int mi = lane >> 3, li = lane & 7;
#pragma unroll 1
    for (int lz = 0; lz < CTZ; lz++) {
#pragma unroll 2
    for (int row = lz * CTY; row < (lz + 1) * CTY; row++) {  // 16 voxels of a row (z, y) of the tile
      uint32_t af[MT][4];
#pragma unroll
      for (int m = 0; m < MT; m++)
        ldsm_x4_t(af[m][0], af[m][1], af[m][2], af[m][3],
                  s_g + (row * 16 + li + (mi >> 1) * 8) * GRS + (m * 16 + (mi & 1) * 8) * 2);
      const int hv = (row / CTY * HTY + row % CTY) * HTX + li + (mi & 1) * 8;
#pragma unroll
      for (int i = 0; i < NTAP; i++) {
        uint32_t b00, b01, b10, b11;  // input channels 0-7 and 8-15, k = 16 voxels
        ldsm_x4_t(b00, b01, b10, b11, s_x + (hv + shift[i]) * RSB + (mi >> 1) * 16);
#pragma unroll
        for (int m = 0; m < MT; m++) {
          mma16816(acc[i][m][0], af[m], b00, b01);
          mma16816(acc[i][m][1], af[m], b10, b11);
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NTAP; i++)
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int n = 0; n < 2; n++)
#pragma unroll
          for (int q = 0; q < 4; q++) {
            sum[i][m][n][q] += acc[i][m][n][q];
            acc[i][m][n][q] = 0.f;
          }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < NTAP; i++) {
    const int tap = tap0 + 8 * i;
    if (tap >= 27) continue;
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
      for (int n = 0; n < 2; n++)
#pragma unroll
        for (int q = 0; q < 4; q++) {
          const int co = m * 16 + (lane >> 2) + (q >> 1) * 8;
          const int ci = n * 8 + (lane & 3) * 2 + (q & 1);
          atomicAdd(&a.dW[((long long)tap * COUT + co) * CIN + c0 + ci], sum[i][m][n][q]);
        }
  }
}

template <int CIN, int COUT>
constexpr int conv_wgrad_smem() {
  return 2 * wgrad_stage<COUT>();
}

}  // namespace bbnet
