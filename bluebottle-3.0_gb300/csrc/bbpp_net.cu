// bbpp_net.cu -- the learned initial guess: a small 3D conv encoder-decoder
// on BF16 tensor cores, trained on the GPU with the library's own forward and
// backward kernels (bbpp_conv.cuh), and applied before the PCG.
//
// The network predicts the correction to a warm start: with p_prev the
// previous pressure and r = rhs - (-A) p_prev its residual (both computed from
// the inputs the guess is defined on: rhs, p_prev, mask),
//   p0 = p_prev + h^2 s_r^-1 OUT,    OUT ~ net(r / s_r, p_prev / s_p, mask)
// so that in grid units OUT approximates the unit-spacing inverse Laplacian of
// the normalised residual, a local relation that carries over between grid
// resolutions.  s_r, s_p: fluid RMS of r and p_prev.
// Network (channels-last BF16 activations, FP32 master weights, Adam):
//   X0  [V][16]  = (r / s_r, prev / s_p, mask, 0 ...)
//   E1  = relu(conv3(X0;  16 -> 16))      stored in CAT1[:, 32:48]
//   P1  = avgpool2(E1)                    [V/8][16]
//   E2  = relu(conv3(P1;  16 -> 32))      stored in CAT2[:, 64:96]
//   P2  = avgpool2(E2)                    [V/64][32]
//   E3  = relu(conv3(P2;  32 -> 64))      [V/64][64]
//   CAT2[:, 0:64] = up2(E3);  D2 = relu(conv3(CAT2; 96 -> 32))   [V/8][32]
//   CAT1[:, 0:32] = up2(D2);  D1 = relu(conv3(CAT1; 48 -> 16))   [V][16]
//   OUT = D1 . w_head + b_head  (FP32)
// Loss: mean over fluid cells of (OUT - (p* - p_prev) s_r / h^2)^2.
// Padding is periodic in x and y and zero in z (the workloads' boundaries).
// In a solve (bbpp_net_guess) the network runs, on large grids, on the
// problem restricted by 2 and its correction is interpolated back.  Forward
// convolutions on rows of 128 voxels (or 256 with 16 outputs) run on tcgen05
// with the x-taps stacked in N (bbpp_conv_tx.cuh); the others, the data
// gradients and the weight gradients on mma.sync (bbpp_conv.cuh).
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "../../include/bbpp.h"
#include "bbpp_conv.cuh"
#include "bbpp_conv_tc.cuh"
#include "bbpp_conv_tx.cuh"
#include "bbpp_internal.h"

using namespace bbnet;

#define NCK(call)                                                                                       \
  do {                                                                                                  \
    cudaError_t e_ = (call);                                                                            \
    if (e_ != cudaSuccess) {                                                                            \
      fprintf(stderr, "bbpp net: %s at %s:%d: %s\n", cudaGetErrorString(e_), __FILE__, __LINE__, #call); \
      return BBPP_CUDA_ERROR;                                                                           \
    }                                                                                                   \
  } while (0)

namespace {

// ------------------------------------------------------------ launchers ---
template <int CIN, int COUT>
cudaError_t conv_fwd_t(const ConvArgs &a, cudaStream_t s) {
  constexpr int smem = conv_fwd_smem<CIN, COUT>();
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(k_conv3_fwd<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  constexpr int TZ = fwd_tz<COUT>();
  dim3 grid((a.nx + CTX - 1) / CTX, (a.ny + CTY - 1) / CTY, a.nb * ((a.nz + TZ - 1) / TZ));
  k_conv3_fwd<CIN, COUT><<<grid, 256, smem, s>>>(a);
  return cudaGetLastError();
}

// tcgen05 path: error word of timed-out waits (bounded mbarrier waits)
__device__ int g_tc_err;
long long g_tc_launches = 0;  // tcgen05 convolutions launched by this process
int g_tc_max_ctas = 0;        // > 0: cap on the persistent grid (tests: longer z marches per CTA)
int g_tc_on = -1;             // -1: the environment decides (BBPP_CONV_TC, default 2)

typedef CUresult (*TmEncode)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                             const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                             CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// tensor maps of one (input, weights) pair, cached: the network calls the
// same few layers with the same buffers every time
struct TmKey {
  const void *in, *w;
  int ldi, nx, ny, nz, nb, cin, cout;
  bool operator==(const TmKey &o) const {
    return in == o.in && w == o.w && ldi == o.ldi && nx == o.nx && ny == o.ny && nz == o.nz && nb == o.nb &&
           cin == o.cin && cout == o.cout;
  }
};

bool tm_build(const TmKey &k, int rows, TmMaps *m) {
  TmEncode fn = reinterpret_cast<TmEncode>(bbpp_tensor_map_encoder());
  if (!fn) return false;
  const cuuint64_t e = 2;
  const cuuint64_t dim[5] = {(cuuint64_t)k.ldi, (cuuint64_t)k.nx, (cuuint64_t)k.ny, (cuuint64_t)k.nz,
                             (cuuint64_t)k.nb};
  const cuuint64_t str[4] = {k.ldi * e, k.nx * k.ldi * e, (cuuint64_t)k.ny * k.nx * k.ldi * e,
                             (cuuint64_t)k.nz * k.ny * k.nx * k.ldi * e};
  const cuuint32_t es[5] = {1, 1, 1, 1, 1};
  const cuuint32_t widths[3] = {144, 136, 128};
  const cuuint32_t box[5] = {8, 144, (cuuint32_t)rows, 1, 1};
  if (fn(&m->rows, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(k.in), dim, str, box, es,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  for (int i = 0; i < 3; i++) {
    const cuuint32_t box1[5] = {8, widths[i], 1, 1, 1};
    if (fn(&m->row[i], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(k.in), dim, str, box1, es,
           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return false;
  }
  const cuuint64_t wdim[3] = {(cuuint64_t)k.cin, (cuuint64_t)k.cout, 27};
  const cuuint64_t wstr[2] = {k.cin * e, (cuuint64_t)k.cout * k.cin * e};
  const cuuint32_t wbox[3] = {8, (cuuint32_t)k.cout, 27};
  return fn(&m->w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(k.w), wdim, wstr, wbox, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool tm_maps(const TmKey &k, int rows, TmMaps *out) {
  static std::vector<std::pair<TmKey, TmMaps>> cache;
  for (const auto &c : cache)
    if (c.first == k) {
      *out = c.second;
      return true;
    }
  TmMaps m;
  if (!tm_build(k, rows, &m)) return false;
  if (cache.size() >= 32) cache.erase(cache.begin());
  cache.emplace_back(k, m);
  *out = m;
  return true;
}

template <int CIN, int COUT>
cudaError_t conv_tc_t(const ConvArgs &a, cudaStream_t s) {
  constexpr int smem = tm_smem<CIN, COUT>();
  int dev = 0;
  cudaGetDevice(&dev);
  static unsigned long long attr = 0;  // per device
  if (dev < 64 && !(attr & (1ull << dev))) {
    cudaError_t e = cudaFuncSetAttribute(k_conv3_tm<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    attr |= 1ull << dev;
  }
  TmKey key{a.in, a.w, a.ldi, a.nx, a.ny, a.nz, a.nb, CIN, COUT};
  TmMaps maps;
  if (!tm_maps(key, tm_tyr<COUT>() + 2, &maps)) return cudaErrorNotSupported;  // the caller falls back
  TmGeo g;
  g.nxb = a.nx / 128;
  g.nyb = (a.ny + tm_tyr<COUT>() - 1) / tm_tyr<COUT>();
  g.units = (long long)a.nb * g.nyb * g.nxb * a.nz;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int cap = std::max(sms, 1);
  if (g_tc_max_ctas > 0) cap = std::min(cap, g_tc_max_ctas);
  const int grid = (int)std::min<long long>(cap, g.units);
  int *err = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void **)&err, g_tc_err);
  if (e != cudaSuccess) return e;
  k_conv3_tm<CIN, COUT><<<grid, TM_THREADS, smem, s>>>(a, maps, g, err);
  e = cudaGetLastError();
  if (e == cudaSuccess) g_tc_launches++;
  return e;
}

// the tx kernel: whole rows of 128 or 256 voxels, the three x-taps stacked in N
bool tx_build(const TmKey &k, int rows, TxMaps *m) {
  TmEncode fn = reinterpret_cast<TmEncode>(bbpp_tensor_map_encoder());
  if (!fn) return false;
  const cuuint64_t e = 2;
  const cuuint64_t dim[5] = {(cuuint64_t)k.ldi, (cuuint64_t)k.nx, (cuuint64_t)k.ny, (cuuint64_t)k.nz,
                             (cuuint64_t)k.nb};
  const cuuint64_t str[4] = {k.ldi * e, k.nx * k.ldi * e, (cuuint64_t)k.ny * k.nx * k.ldi * e,
                             (cuuint64_t)k.nz * k.ny * k.nx * k.ldi * e};
  const cuuint32_t es[5] = {1, 1, 1, 1, 1};
  const cuuint32_t box[5] = {8, (cuuint32_t)k.nx, (cuuint32_t)rows, 1, 1};
  const cuuint32_t box1[5] = {8, (cuuint32_t)k.nx, 1, 1, 1};
  if (fn(&m->rows, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(k.in), dim, str, box, es,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS ||
      fn(&m->row, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<void *>(k.in), dim, str, box1, es,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return false;
  const cuuint64_t wdim[3] = {(cuuint64_t)k.cin, (cuuint64_t)k.cout, 27};
  const cuuint64_t wstr[2] = {k.cin * e, (cuuint64_t)k.cout * k.cin * e};
  const cuuint32_t wbox[3] = {8, (cuuint32_t)k.cout, 27};
  return fn(&m->w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void *>(k.w), wdim, wstr, wbox, es,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

bool tx_maps(const TmKey &k, int rows, TxMaps *out) {
  static std::vector<std::pair<TmKey, TxMaps>> cache;
  for (const auto &c : cache)
    if (c.first == k) {
      *out = c.second;
      return true;
    }
  TxMaps m;
  if (!tx_build(k, rows, &m)) return false;
  if (cache.size() >= 32) cache.erase(cache.begin());
  cache.emplace_back(k, m);
  *out = m;
  return true;
}

template <int CIN, int COUT, int NXB>
cudaError_t conv_tx_t(const ConvArgs &a, cudaStream_t s) {
  // at least half an SM's shared memory: one CTA per SM (each holds all of tensor memory)
  constexpr int smem = std::max(tx_smem<CIN, COUT, NXB>(), 116 * 1024);
  constexpr int TYR = tx_tyr<COUT, NXB>();
  int dev = 0;
  cudaGetDevice(&dev);
  static unsigned long long attr = 0;  // per device
  if (dev < 64 && !(attr & (1ull << dev))) {
    cudaError_t e = cudaFuncSetAttribute(k_conv3_tx<CIN, COUT, NXB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem);
    if (e != cudaSuccess) return e;
    attr |= 1ull << dev;
  }
  TmKey key{a.in, a.w, a.ldi, a.nx, a.ny, a.nz, a.nb, CIN, COUT};
  TxMaps maps;
  if (!tx_maps(key, TYR + 2, &maps)) return cudaErrorNotSupported;  // the caller falls back
  TxGeo g;
  g.nyb = (a.ny + TYR - 1) / TYR;
  g.units = (long long)a.nb * g.nyb * a.nz;
  int sms = 0;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int cap = std::max(sms, 1);
  if (g_tc_max_ctas > 0) cap = std::min(cap, g_tc_max_ctas);
  const int grid = (int)std::min<long long>(cap, g.units);
  int *err = nullptr;
  cudaError_t e = cudaGetSymbolAddress((void **)&err, g_tc_err);
  if (e != cudaSuccess) return e;
  k_conv3_tx<CIN, COUT, NXB><<<grid, TX_THREADS, smem, s>>>(a, maps, g, err);
  e = cudaGetLastError();
  if (e == cudaSuccess) g_tc_launches++;
  return e;
}

// Forward convolution kernel: 0 = mma.sync, 1 = tcgen05 with x-shifted A tiles
// in tensor memory (k_conv3_tm), 2 = tcgen05 with the x-taps stacked in N
// (k_conv3_tx, the default; BBPP_CONV_TC=0 or 1 selects the others).  A
// tcgen05.mma of M = 128, K = 16 costs about the same whatever its N, so
// k_conv3_tm, with N = 16 or 32 output channels, is no faster than mma.sync;
// k_conv3_tx, with N = 48 or 96, is 1.6-2.3 times faster on these layers.
int conv_tc_mode() {
  if (g_tc_on < 0) {
    const char *v = getenv("BBPP_CONV_TC");
    return (v && (v[0] == '0' || v[0] == '1')) ? v[0] - '0' : 2;
  }
  return g_tc_on;
}

bool conv_tc_enabled() { return conv_tc_mode() != 0; }

// the tcgen05 kernel takes 128-voxel x blocks, 16-byte aligned channel runs and
// tensor maps (a driver with cuTensorMapEncodeTiled)
bool conv_tc_fits(const ConvArgs &a) {
  const auto al16 = [](const void *p) { return ((uintptr_t)p & 15u) == 0; };
  return conv_tc_enabled() && a.nx % 128 == 0 && a.ldi % 8 == 0 && a.ci_off % 8 == 0 && a.ldo % 8 == 0 &&
         a.co_off % 8 == 0 && al16(a.in) && al16(a.w) && al16(a.out) && bbpp_tensor_map_encoder() != nullptr;
}

// nonzero once a tcgen05 convolution gave up a wait; cleared by the read
int conv_tc_failed() {
  int v = 0;
  if (cudaMemcpyFromSymbol(&v, g_tc_err, sizeof(int)) != cudaSuccess) return 1;
  if (v) {
    const int zero = 0;
    cudaMemcpyToSymbol(g_tc_err, &zero, sizeof(int));
  }
  return v;
}

// rows of 128 voxels (and of 256 where COUT = 16); other widths fall back
template <int CIN, int COUT>
cudaError_t conv_tx_rows(const ConvArgs &a, cudaStream_t s) {
  if (a.nx == 128) return conv_tx_t<CIN, COUT, 1>(a, s);
  if constexpr (COUT == 16) {
    if (a.nx == 256) return conv_tx_t<CIN, COUT, 2>(a, s);
  }
  return cudaErrorNotSupported;
}

cudaError_t conv_fwd(int cin, int cout, const ConvArgs &a, cudaStream_t s) {
#define TCASE(CI, CO)                                                                     \
  if (cin == CI && cout == CO && conv_tc_fits(a)) {                                         \
    cudaError_t e_ = cudaErrorNotSupported;                                                 \
    if (conv_tc_mode() == 2) e_ = conv_tx_rows<CI, CO>(a, s);                               \
    else e_ = conv_tc_t<CI, CO>(a, s);                                                      \
    if (e_ != cudaErrorNotSupported) return e_;                                             \
  }
  TCASE(16, 16) TCASE(16, 32) TCASE(96, 32) TCASE(48, 16) TCASE(32, 16)
#undef TCASE
#define CASE(CI, CO) \
  if (cin == CI && cout == CO) return conv_fwd_t<CI, CO>(a, s);
  CASE(16, 16) CASE(16, 32) CASE(32, 64) CASE(96, 32) CASE(48, 16)  // forward layers
  CASE(16, 48) CASE(32, 96) CASE(64, 32) CASE(32, 16)               // dgrad of the layers
#undef CASE
  return cudaErrorInvalidValue;
}

template <int CIN, int COUT>
cudaError_t conv_wgrad_t(WgradArgs a, cudaStream_t s) {
  constexpr int smem = conv_wgrad_smem<CIN, COUT>();
  const long long ntiles = (long long)((a.nx + CTX - 1) / CTX) * ((a.ny + CTY - 1) / CTY) *
                           ((a.nz + CTZ - 1) / CTZ) * a.nb;
  if (ntiles >= (1ll << 31)) return cudaErrorInvalidValue;
  // one wave: every CTA adds its sums to dW once, so more CTAs are more atomics.  Asked of each device once (the
  // shared memory cap is a device's too).
  static std::atomic<int> waves[64];
  int dev = 0;
  cudaGetDevice(&dev);
  int wave = dev < 64 ? waves[dev].load() : 0;
  if (!wave) {
    cudaError_t e = cudaFuncSetAttribute(k_conv3_wgrad<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    int sms = 0, per_sm = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_conv3_wgrad<CIN, COUT>, 256, smem);
    wave = std::max(1, sms) * std::max(1, per_sm);
    if (dev < 64) waves[dev].store(wave);
  }
  constexpr int chunks = CIN / 16, groups = (27 + 8 * wgrad_taps<COUT>() - 1) / (8 * wgrad_taps<COUT>());
  // and more roundings: eight tiles a CTA at least, on small volumes
  int ctas = (int)std::min<long long>(std::min<long long>(ntiles, std::max<long long>(ntiles / 8, 16)),
                                      std::max(1, wave / (chunks * groups)));
  a.tiles_per_cta = (int)((ntiles + ctas - 1) / ctas);
  ctas = (int)((ntiles + a.tiles_per_cta - 1) / a.tiles_per_cta);
  dim3 grid(ctas, chunks, groups);
  k_conv3_wgrad<CIN, COUT><<<grid, 256, smem, s>>>(a);
  return cudaGetLastError();
}

cudaError_t conv_wgrad(int cin, int cout, const WgradArgs &a, cudaStream_t s) {
#define CASE(CI, CO) \
  if (cin == CI && cout == CO) return conv_wgrad_t<CI, CO>(a, s);
  CASE(16, 16) CASE(16, 32) CASE(32, 64) CASE(96, 32) CASE(48, 16)
#undef CASE
  return cudaErrorInvalidValue;
}

// W [27][cout][cin] -> Wt [27][cin][cout] with the taps reversed (the dgrad
// kernel of a 3x3x3 "same" convolution)
__global__ void k_wflip(const bf16 *__restrict__ w, bf16 *__restrict__ wt, int cin, int cout) {
  const int n = 27 * cin * cout;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x) {
    const int t = e / (cin * cout), r = e - t * cin * cout;
    const int ci = r / cout, co = r - ci * cout;
    wt[e] = w[((26 - t) * cout + co) * cin + ci];
  }
}

// ------------------------------------------------------- small kernels ---
__global__ void k_f32_to_bf16(const float *__restrict__ a, bf16 *__restrict__ b, int n) {
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < n; e += gridDim.x * blockDim.x)
    b[e] = __float2bfloat16_rn(a[e]);
}

// sum over fluid cells of v^2 for each volume (FP64 atomics, one per CTA)
template <typename T>
__global__ void k_fluid_sumsq(const T *__restrict__ v, const uint8_t *__restrict__ mask, long long vol, int nb,
                              double *out /* [nb][2]: sum v^2, count */) {
  __shared__ double s1[256], s2[256];
  const int b = blockIdx.y;
  double a = 0, c = 0;
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < vol; i += (long long)gridDim.x * 256) {
    if (mask && mask[i]) continue;
    const double x = (double)v[(long long)b * vol + i];
    a += x * x;
    c += 1;
  }
  s1[threadIdx.x] = a;
  s2[threadIdx.x] = c;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      s1[threadIdx.x] += s1[threadIdx.x + o];
      s2[threadIdx.x] += s2[threadIdx.x + o];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    atomicAdd(&out[2 * b], s1[0]);
    atomicAdd(&out[2 * b + 1], s2[0]);
  }
}

// scales[b] = (1/s_b, 1/s_p) from the sums; s = sqrt(sum/count), 1 if zero
__global__ void k_scales(const double *sb, const double *sp, int nb, float *scales) {
  for (int b = threadIdx.x; b < nb; b += blockDim.x) {
    const double rb = sb[2 * b + 1] > 0 ? sqrt(sb[2 * b] / sb[2 * b + 1]) : 0;
    const double rp = sp ? (sp[2 * b + 1] > 0 ? sqrt(sp[2 * b] / sp[2 * b + 1]) : 0) : 0;
    scales[2 * b] = rb > 0 ? (float)(1.0 / rb) : 1.f;
    scales[2 * b + 1] = rp > 0 ? (float)(1.0 / rp) : 1.f;
  }
}

// X0 = (rhs / s_b, prev / s_p, mask, 0 ...), 16 channels
template <typename T>
__global__ void k_prep(const T *__restrict__ rhs, const T *__restrict__ prev, const uint8_t *__restrict__ mask,
                       const float *__restrict__ scales, long long vol, int nb, bf16 *__restrict__ x0) {
  const long long n = vol * nb;
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < n; e += (long long)gridDim.x * 256) {
    const int b = (int)(e / vol);
    const long long i = e - (long long)b * vol;
    const bool solid = mask && mask[i];
    const float r = solid ? 0.f : (float)rhs[e] * scales[2 * b];
    const float p = (solid || !prev) ? 0.f : (float)prev[e] * scales[2 * b + 1];
    __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(x0 + e * 16);
    o[0] = __floats2bfloat162_rn(r, p);
    o[1] = __floats2bfloat162_rn(solid ? 1.f : 0.f, 0.f);
#pragma unroll
    for (int q = 2; q < 8; q++) o[q] = __floats2bfloat162_rn(0.f, 0.f);
  }
}

// The resampling kernels move 8 channels (16 bytes) per thread: C, the row
// strides and the channel offsets are multiples of 8.  Voxel indices are
// 32-bit (a batch holds fewer than 2^32 / 8 voxels).
__device__ __forceinline__ void bf8_unpack(const uint4 u, float (&f)[8]) {
  const __nv_bfloat162 *h = reinterpret_cast<const __nv_bfloat162 *>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const float2 t = __bfloat1622float2(h[i]);
    f[2 * i] = t.x;
    f[2 * i + 1] = t.y;
  }
}

__device__ __forceinline__ uint4 bf8_pack(const float (&f)[8]) {
  uint4 u;
  __nv_bfloat162 *h = reinterpret_cast<__nv_bfloat162 *>(&u);
#pragma unroll
  for (int i = 0; i < 4; i++) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return u;
}

// voxel index of child q (0..7) of the half-resolution voxel (x, y, z) of batch b
__device__ __forceinline__ unsigned int child_voxel(unsigned int b, unsigned int x, unsigned int y, unsigned int z,
                                                    int q, unsigned int nx, unsigned int ny, unsigned int nz) {
  return ((b * nz + 2 * z + (q >> 2)) * ny + 2 * y + ((q >> 1) & 1)) * nx + 2 * x + (q & 1);
}

// average pool 2x2x2: out[V/8][C] (ld C) from in (ld, off)
__global__ void k_pool_fwd(const bf16 *__restrict__ in, int ldi, int off, int C, int nx, int ny, int nz, int nb,
                           bf16 *__restrict__ out) {
  const unsigned int hx = nx / 2, hy = ny / 2, hz = nz / 2, cv = C / 8;
  const unsigned int n = hx * hy * hz * (unsigned int)nb * cv;
  for (unsigned int e = blockIdx.x * 256u + threadIdx.x; e < n; e += gridDim.x * 256u) {
    const unsigned int k = e % cv;
    unsigned int v = e / cv;
    const unsigned int x = v % hx;
    v /= hx;
    const unsigned int y = v % hy;
    v /= hy;
    const unsigned int z = v % hz, b = v / hz;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const unsigned int src = child_voxel(b, x, y, z, q, nx, ny, nz);
      float f[8];
      bf8_unpack(*reinterpret_cast<const uint4 *>(in + (size_t)src * ldi + off + 8 * k), f);
#pragma unroll
      for (int i = 0; i < 8; i++) s[i] += f[i];
    }
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] *= 0.125f;
    reinterpret_cast<uint4 *>(out)[e] = bf8_pack(s);
  }
}

// din[v][c] (ld C) = dskip[v][c] (ld, off; may be null) + dout[parent][c] / 8
__global__ void k_pool_bwd(const bf16 *__restrict__ dout, const bf16 *__restrict__ dskip, int lds, int offs, int C,
                           int nx, int ny, int nz, int nb, bf16 *__restrict__ din) {
  const unsigned int hx = nx / 2, hy = ny / 2, hz = nz / 2, cv = C / 8;
  const unsigned int n = (unsigned int)nx * ny * nz * nb * cv;
  for (unsigned int e = blockIdx.x * 256u + threadIdx.x; e < n; e += gridDim.x * 256u) {
    const unsigned int k = e % cv;
    const unsigned int v = e / cv;
    const unsigned int x = v % nx;
    unsigned int t = v / nx;
    const unsigned int y = t % ny;
    t /= ny;
    const unsigned int z = t % nz, b = t / nz;
    const unsigned int par = ((b * hz + z / 2) * hy + y / 2) * hx + x / 2;
    float g[8], d[8];
    bf8_unpack(reinterpret_cast<const uint4 *>(dout)[par * cv + k], g);
#pragma unroll
    for (int i = 0; i < 8; i++) g[i] *= 0.125f;
    if (dskip) {
      bf8_unpack(*reinterpret_cast<const uint4 *>(dskip + (size_t)v * lds + offs + 8 * k), d);
#pragma unroll
      for (int i = 0; i < 8; i++) g[i] += d[i];
    }
    reinterpret_cast<uint4 *>(din)[e] = bf8_pack(g);
  }
}

// nearest upsample x2: out[v][off + c] (ld) = in[parent][c] (ld C)
__global__ void k_up_fwd(const bf16 *__restrict__ in, int C, int nx, int ny, int nz, int nb, bf16 *__restrict__ out,
                         int ldo, int off) {
  const unsigned int hx = nx / 2, hy = ny / 2, hz = nz / 2, cv = C / 8;
  const unsigned int n = (unsigned int)nx * ny * nz * nb * cv;
  for (unsigned int e = blockIdx.x * 256u + threadIdx.x; e < n; e += gridDim.x * 256u) {
    const unsigned int k = e % cv;
    const unsigned int v = e / cv;
    const unsigned int x = v % nx;
    unsigned int t = v / nx;
    const unsigned int y = t % ny;
    t /= ny;
    const unsigned int z = t % nz, b = t / nz;
    const unsigned int par = ((b * hz + z / 2) * hy + y / 2) * hx + x / 2;
    *reinterpret_cast<uint4 *>(out + (size_t)v * ldo + off + 8 * k) = reinterpret_cast<const uint4 *>(in)[par * cv + k];
  }
}

// din[p][c] (ld C, at half resolution) = sum of the 8 children dout[v][off + c]
__global__ void k_up_bwd(const bf16 *__restrict__ dout, int ldo, int off, int C, int nx, int ny, int nz, int nb,
                         bf16 *__restrict__ din) {
  const unsigned int hx = nx / 2, hy = ny / 2, hz = nz / 2, cv = C / 8;
  const unsigned int n = hx * hy * hz * (unsigned int)nb * cv;
  for (unsigned int e = blockIdx.x * 256u + threadIdx.x; e < n; e += gridDim.x * 256u) {
    const unsigned int k = e % cv;
    unsigned int v = e / cv;
    const unsigned int x = v % hx;
    v /= hx;
    const unsigned int y = v % hy;
    v /= hy;
    const unsigned int z = v % hz, b = v / hz;
    float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const unsigned int ch = child_voxel(b, x, y, z, q, nx, ny, nz);
      float f[8];
      bf8_unpack(*reinterpret_cast<const uint4 *>(dout + (size_t)ch * ldo + off + 8 * k), f);
#pragma unroll
      for (int i = 0; i < 8; i++) s[i] += f[i];
    }
    reinterpret_cast<uint4 *>(din)[e] = bf8_pack(s);
  }
}

// ReLU backward: g = dout where the layer's output is positive, else 0 (g and dout
// dense, C = 16, 32 or 64 channels), and sums of g over the voxels for db (k_bias_out).
// Eight channels (16 bytes) a thread; a thread keeps its channels from voxel to voxel,
// so the bias sums stay in registers.  One pass: the gate and the bias gradient apart
// took 71 + 35 us for 16 channels of four 64^3 volumes.  The CTAs' sums meet in FP64:
// FP32 atomics on db, up to kGateCtas of them a channel, had up to six times the error
// of the two passes (now a tenth to a half of it).  kGateSums places a channel: on one,
// the CTAs wait for each other's atomics (4 us a layer).
constexpr int kGateCtas = 1216, kGateSums = 16;
__global__ void __launch_bounds__(256) k_gate_bias(const bf16 *__restrict__ dout, const bf16 *__restrict__ out,
                                                   int ldo, int off, int C, long long nvox, bf16 *__restrict__ g,
                                                   double *sum) {
  __shared__ float s[8][64];
  const int parts = C / 8, c8 = threadIdx.x % parts, per = 256 / parts;
  float a[8];
#pragma unroll
  for (int q = 0; q < 8; q++) a[q] = 0.f;
  for (long long v = blockIdx.x * (long long)per + threadIdx.x / parts; v < nvox; v += (long long)gridDim.x * per) {
    const uint4 du = *reinterpret_cast<const uint4 *>(dout + v * C + c8 * 8);
    const uint4 ou = *reinterpret_cast<const uint4 *>(out + v * ldo + off + c8 * 8);
    float d[8], o[8];
    bf8_unpack(du, d);
    bf8_unpack(ou, o);
#pragma unroll
    for (int q = 0; q < 8; q++) {
      d[q] = o[q] > 0.f ? d[q] : 0.f;
      a[q] += d[q];
    }
    *reinterpret_cast<uint4 *>(g + v * C + c8 * 8) = bf8_pack(d);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int o = 16; o >= parts; o >>= 1) {
#pragma unroll
    for (int q = 0; q < 8; q++) a[q] += __shfl_xor_sync(0xffffffffu, a[q], o);
  }
  if (lane < parts) {
#pragma unroll
    for (int q = 0; q < 8; q++) s[warp][lane * 8 + q] = a[q];
  }
  __syncthreads();
  if (threadIdx.x < (unsigned)C) {
    float t[8];
#pragma unroll
    for (int w = 0; w < 8; w++) t[w] = s[w][threadIdx.x];
    atomicAdd(&sum[blockIdx.x % kGateSums * 64 + threadIdx.x],
              (double)(((t[0] + t[1]) + (t[2] + t[3])) + ((t[4] + t[5]) + (t[6] + t[7]))));
  }
}

// db[c] += the sums of k_gate_bias, a layer a CTA
static_assert(kGateSums == 16, "four places in each quarter");
struct BiasOffsets {
  int off[5], n[5];
};
__global__ void __launch_bounds__(256) k_bias_out(const double *__restrict__ sums, const BiasOffsets L, float *grads) {
  __shared__ double s[4][64];
  const int c = threadIdx.x & 63, part = threadIdx.x >> 6;  // a quarter of the places
  const double *v = sums + (blockIdx.x * kGateSums + part * (kGateSums / 4)) * 64 + c;
  s[part][c] = (v[0] + v[64]) + (v[128] + v[192]);
  __syncthreads();
  if (part == 0 && c < L.n[blockIdx.x])
    grads[L.off[blockIdx.x] + c] += (float)((s[0][c] + s[1][c]) + (s[2][c] + s[3][c]));
}

// OUT[v] = D1[v] . w + b   (FP32)
__global__ void k_head_fwd(const bf16 *__restrict__ d1, const float *__restrict__ w, const float *__restrict__ b,
                           long long nvox, float *__restrict__ out) {
  for (long long v = blockIdx.x * 256LL + threadIdx.x; v < nvox; v += (long long)gridDim.x * 256) {
    float s = b[0];
    const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162 *>(d1 + v * 16);
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float2 f = __bfloat1622float2(p[q]);
      s = fmaf(f.x, w[2 * q], s);
      s = fmaf(f.y, w[2 * q + 1], s);
    }
    out[v] = s;
  }
}

// dD1[v][c] = dOUT[v] w[c];  dw[c] += sum_v dOUT[v] D1[v][c];  db += sum dOUT
__global__ void k_head_bwd(const float *__restrict__ dout, const bf16 *__restrict__ d1, const float *__restrict__ w,
                           long long nvox, bf16 *__restrict__ dd1, float *dw, float *db) {
  __shared__ float s[17][257];
  float a[17];
#pragma unroll
  for (int q = 0; q < 17; q++) a[q] = 0.f;
  for (long long v = blockIdx.x * 256LL + threadIdx.x; v < nvox; v += (long long)gridDim.x * 256) {
    const float g = dout[v];
    const __nv_bfloat162 *p = reinterpret_cast<const __nv_bfloat162 *>(d1 + v * 16);
    __nv_bfloat162 *o = reinterpret_cast<__nv_bfloat162 *>(dd1 + v * 16);
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const float2 f = __bfloat1622float2(p[q]);
      a[2 * q] += g * f.x;
      a[2 * q + 1] += g * f.y;
      o[q] = __floats2bfloat162_rn(g * w[2 * q], g * w[2 * q + 1]);
    }
    a[16] += g;
  }
#pragma unroll
  for (int q = 0; q < 17; q++) s[q][threadIdx.x] = a[q];
  __syncthreads();
  if (threadIdx.x < 17) {
    float t = 0.f;
    for (int i = 0; i < 256; i++) t += s[threadIdx.x][i];
    if (threadIdx.x < 16) atomicAdd(&dw[threadIdx.x], t);
    else atomicAdd(db, t);
  }
}

// loss = sum over volumes and fluid cells of (OUT - tgt / (s_r h^2))^2 / nfluid_total
// with tgt = p* - p_prev;  dOUT = 2 (OUT - tgt / (s_r h^2)) / nfluid_total on
// fluid cells, 0 on solid cells
__global__ void k_loss(const float *__restrict__ out, const float *__restrict__ tgt, const uint8_t *__restrict__ mask,
                       const float *__restrict__ scales, long long vol, int nb, double inv_n, float inv_h2,
                       float *__restrict__ dout, double *loss) {
  __shared__ double s[256];
  double a = 0;
  const long long n = vol * nb;
  for (long long e = blockIdx.x * 256LL + threadIdx.x; e < n; e += (long long)gridDim.x * 256) {
    const int b = (int)(e / vol);
    const long long i = e - (long long)b * vol;
    if (mask && mask[i]) {
      dout[e] = 0.f;
      continue;
    }
    const float d = out[e] - tgt[e] * (scales[2 * b] * inv_h2);
    a += (double)d * d;
    dout[e] = (float)(2.0 * inv_n) * d;
  }
  s[threadIdx.x] = a;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, s[0] * inv_n);
}

// p0 = p_prev + OUT h^2 / (1/s_r) on fluid cells, 0 on solid cells
__global__ void k_guess_out(const float *__restrict__ out, const double *__restrict__ prev,
                            const uint8_t *__restrict__ mask, const float *__restrict__ scales, double h2,
                            long long vol, double *__restrict__ x) {
  const double sr = h2 / (double)scales[0];
  for (long long i = blockIdx.x * 256LL + threadIdx.x; i < vol; i += (long long)gridDim.x * 256)
    x[i] = (mask && mask[i]) ? 0.0 : (prev ? prev[i] : 0.0) + (double)out[i] * sr;
}

// binary64 -> binary32 by truncating the significand (round toward zero): the
// exponent is rebiased (1023 -> 127) and the 52-bit fraction cut to its top 23
// bits.  Magnitudes below the binary32 normal range become a signed zero,
// finite magnitudes above it the largest finite binary32; infinities and NaNs
// stay so.  Integer operations only: a cvt runs on the FP64 pipe, which on
// this part has 1/64 of the FP32 rate, and the grid kernels of the guess
// convert several values per cell.
__device__ __forceinline__ float narrow_rz(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const unsigned int hi = (unsigned int)(b >> 32);
  const unsigned int sign = hi & 0x80000000u;
  const int e64 = (int)((hi >> 20) & 0x7ffu);
  const unsigned int frac = (unsigned int)(b >> 29) & 0x7fffffu;
  if (e64 == 0x7ff) return __uint_as_float(sign | 0x7f800000u | (frac ? 0x400000u : 0u));
  const int e = e64 - 1023 + 127;
  if (e <= 0) return __uint_as_float(sign);
  if (e >= 255) return __uint_as_float(sign | 0x7f7fffffu);
  return __uint_as_float(sign | ((unsigned int)e << 23) | frac);
}

// binary32 -> binary64, exact for normal numbers and zeros (exponent rebiased,
// fraction widened); binary32 subnormals become a signed zero, infinities and
// NaNs stay so.  Integer operations only, as narrow_rz.
__device__ __forceinline__ double widen(float f) {
  const unsigned int u = __float_as_uint(f);
  const unsigned long long sign = (unsigned long long)(u & 0x80000000u) << 32;
  const unsigned int e32 = (u >> 23) & 0xffu;
  const unsigned long long frac = (unsigned long long)(u & 0x7fffffu) << 29;
  if (e32 == 0) return __longlong_as_double((long long)sign);
  if (e32 == 0xffu) return __longlong_as_double((long long)(sign | 0x7ff0000000000000ull | frac));
  return __longlong_as_double((long long)(sign | ((unsigned long long)(e32 - 127u + 1023u) << 52) | frac));
}

// The warm start's residual r = rhs - (-A) p_prev, restricted by F (2 or 4) in
// the same pass (cell-centred: the means of the FxFxF children), with p_prev's
// means and the coarse solid cells (at least half the children solid).  The residual is
// formed as in the residual kernel (k_resid: neighbours of or across solid
// cells count 0, walls through the class diagonal) but in FP32 arithmetic, on
// inputs narrowed by truncation (narrow_rz): it only feeds the BF16 network.
// prev == NULL: r = rhs, p_prev = 0.
template <int F>
__global__ void __launch_bounds__(256) k_resid_restrict(const bbpp::Geo G, const double *__restrict__ rhs,
                                                        const double *__restrict__ prev,
                                                        const uint8_t *__restrict__ mask, double *__restrict__ rc,
                                                        double *__restrict__ pc, uint8_t *__restrict__ mc) {
  __shared__ float s_tab[81];
  for (int e = threadIdx.x; e < 81; e += blockDim.x) s_tab[e] = (float)G.tab[e];
  __syncthreads();
  const int nx = G.nx, ny = G.ny, nz = G.nz;
  const unsigned int cxn = (unsigned)nx / F, cyn = (unsigned)ny / F;
  const unsigned int nc = cxn * cyn * ((unsigned)nz / F);
  const float fx = (float)G.cx, fy = (float)G.cy, fz = (float)G.cz;
  // p_prev at a neighbour (0 outside a wall); solid: the neighbour is solid
  auto nb = [&](int xx, int yy, int zz, bool &solid) -> float {
    const int gx = bbpp::halo_index(xx, nx, G.px), gy = bbpp::halo_index(yy, ny, G.py),
              gz = bbpp::halo_index(zz, nz, G.pz);
    solid = false;
    if (gx < 0 || gy < 0 || gz < 0) return 0.f;
    const unsigned int c = (unsigned)gx + (unsigned)nx * ((unsigned)gy + (unsigned)ny * (unsigned)gz);
    if (mask) solid = mask[c] != 0;
    return narrow_rz(prev[c]);
  };
  for (unsigned int e = blockIdx.x * 256u + threadIdx.x; e < nc; e += gridDim.x * 256u) {
    const unsigned int i = e % cxn, t = e / cxn, j = t % cyn, k = t / cyn;
    float sr = 0.f, sp = 0.f;
    int sm = 0;
#pragma unroll 8
    for (int ch = 0; ch < F * F * F; ch++) {
      const int x = F * (int)i + ch % F, y = F * (int)j + (ch / F) % F, z = F * (int)k + ch / (F * F);
      const unsigned int c = (unsigned)x + (unsigned)nx * ((unsigned)y + (unsigned)ny * (unsigned)z);
      const bool ms = mask && mask[c] != 0;
      float r = narrow_rz(rhs[c]);
      if (prev) {
        const float pcv = narrow_rz(prev[c]);
        bool s0, s1, s2, s3, s4, s5;
        float pe = nb(x + 1, y, z, s0), pw = nb(x - 1, y, z, s1), pn = nb(x, y + 1, z, s2), ps = nb(x, y - 1, z, s3);
        float pt = nb(x, y, z + 1, s4), pb = nb(x, y, z - 1, s5);
        if (mask) {
          pe = (ms || s0) ? 0.f : pe;
          pw = (ms || s1) ? 0.f : pw;
          pn = (ms || s2) ? 0.f : pn;
          ps = (ms || s3) ? 0.f : ps;
          pt = (ms || s4) ? 0.f : pt;
          pb = (ms || s5) ? 0.f : pb;
        }
        const int cls = bbpp::wall_count(x, nx, G.px) + 3 * bbpp::wall_count(y, ny, G.py) +
                        9 * bbpp::wall_count(z, nz, G.pz);
        const float d = ms ? s_tab[54 + cls] : s_tab[cls];
        float s_ = fx * (pe + pw);
        s_ = fmaf(fy, pn + ps, s_);
        s_ = fmaf(fz, pt + pb, s_);
        r -= fmaf(d, pcv, -s_);
        sp += pcv;
      }
      sr += r;
      sm += ms ? 1 : 0;
    }
    constexpr double inv = 1.0 / (F * F * F);
    rc[e] = inv * (double)sr;
    pc[e] = inv * (double)sp;
    mc[e] = sm >= F * F * F / 2 ? 1 : 0;
  }
}

// the coarse correction p0c - pc (0 on coarse solid cells) in FP32: the
// prolongation interpolates it in FP32
__global__ void k_corr2(float *__restrict__ corr, const double *__restrict__ p0c, const double *__restrict__ pc,
                        const uint8_t *__restrict__ mc, unsigned int nc) {
  for (unsigned int e = blockIdx.x * 256u + threadIdx.x; e < nc; e += gridDim.x * 256u)
    corr[e] = mc[e] ? 0.f : (float)(p0c[e] - pc[e]);
}

// one axis of the cell-centred trilinear prolongation by F: fine cell a = F m + q
// lies at coarse coordinate m + (2q + 1 - F) / (2F), between coarse cells lo
// and hi, hi weighted w (F = 2: a/2 - 1/4)
template <int F>
__device__ __forceinline__ void prolong_axis(int a, int n, int periodic, int &lo, int &hi, float &w) {
  const int m = a / F, num = 2 * (a - m * F) + 1 - F;
  if (num < 0) {
    lo = m - 1;
    w = (float)(2 * F + num) / (float)(2 * F);
  } else {
    lo = m;
    w = (float)num / (float)(2 * F);
  }
  hi = lo + 1;
  if (periodic) {
    lo = lo < 0 ? lo + n : lo;
    hi = hi >= n ? hi - n : hi;
  } else {
    lo = max(lo, 0);
    hi = min(hi, n - 1);
  }
}

// x = p_prev + the trilinear interpolation of the coarse correction (FP32,
// widened exactly before the FP64 add); fine solid cells 0, as the guess on
// the grid itself
template <int F>
__global__ void __launch_bounds__(256) k_prolong(const float *__restrict__ corr, const double *__restrict__ prev,
                                                 const uint8_t *__restrict__ mask, int nx, int ny, int nz, int px,
                                                 int py, int pz, double *__restrict__ x) {
  const int cxn = nx / F, cyn = ny / F, czn = nz / F;
  const unsigned int n = (unsigned)nx * (unsigned)ny * (unsigned)nz;
  for (unsigned int f = blockIdx.x * 256u + threadIdx.x; f < n; f += gridDim.x * 256u) {
    if (mask && mask[f]) {
      x[f] = 0.0;
      continue;
    }
    const unsigned int t = f / (unsigned)nx;
    const int i = (int)(f - t * (unsigned)nx);
    const int k = (int)(t / (unsigned)ny), j = (int)(t - (unsigned)k * (unsigned)ny);
    int xl, xh, yl, yh, zl, zh;
    float wx, wy, wz;
    prolong_axis<F>(i, cxn, px, xl, xh, wx);
    prolong_axis<F>(j, cyn, py, yl, yh, wy);
    prolong_axis<F>(k, czn, pz, zl, zh, wz);
    const unsigned int r00 = ((unsigned)zl * cyn + yl) * cxn, r01 = ((unsigned)zl * cyn + yh) * cxn;
    const unsigned int r10 = ((unsigned)zh * cyn + yl) * cxn, r11 = ((unsigned)zh * cyn + yh) * cxn;
    const float a00 = (1.f - wx) * corr[r00 + xl] + wx * corr[r00 + xh];
    const float a01 = (1.f - wx) * corr[r01 + xl] + wx * corr[r01 + xh];
    const float a10 = (1.f - wx) * corr[r10 + xl] + wx * corr[r10 + xh];
    const float a11 = (1.f - wx) * corr[r11 + xl] + wx * corr[r11 + xh];
    const float v = (1.f - wz) * ((1.f - wy) * a00 + wy * a01) + wz * ((1.f - wy) * a10 + wy * a11);
    x[f] = prev ? prev[f] + widen(v) : widen(v);
  }
}

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m, float *__restrict__ v,
                       int n, float lr, float b1, float b2, float eps, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  }
}

int nblocks(long long n) { return (int)std::min<long long>(std::max<long long>((n + 255) / 256, 1), 4096); }

}  // namespace

// ------------------------------------------------------------- network ----
struct ConvLayer {
  int cin, cout;
  int woff, boff;  // offsets in the parameter vector
};

static const int NLAYER = 5;
static const ConvLayer kLayers[NLAYER] = {
    {16, 16, 0, 0}, {16, 32, 0, 0}, {32, 64, 0, 0}, {96, 32, 0, 0}, {48, 16, 0, 0}};

struct bbpp_net {
  int np = 0;                     // parameters
  ConvLayer L[NLAYER];
  int head_w = 0, head_b = 0;
  float *w = nullptr;             // FP32 master parameters
  float *g = nullptr;             // gradients
  float *m = nullptr, *v = nullptr;  // Adam moments
  bf16 *w16 = nullptr;            // BF16 copy of the parameters (conv weights used from it)
  bf16 *wt16 = nullptr;           // flipped/transposed conv weights (dgrad)
  int t = 0;                      // Adam step
  // workspace for one (nx, ny, nz, nb)
  int wx = 0, wy = 0, wz = 0, wb = 0;
  bool wgrad = false;
  bf16 *X0 = nullptr, *CAT1 = nullptr, *P1 = nullptr, *CAT2 = nullptr, *P2 = nullptr, *E3 = nullptr, *D2 = nullptr,
       *D1 = nullptr;
  float *OUT = nullptr, *dOUT = nullptr, *scales = nullptr;
  double *sums = nullptr, *lossd = nullptr;
  double *bsum = nullptr;  // bias gradients: the CTAs' sums of each layer
  bf16 *dD1 = nullptr, *G = nullptr, *dCAT1 = nullptr, *dD2 = nullptr, *dCAT2 = nullptr, *dE3 = nullptr,
       *dP2 = nullptr, *dE2 = nullptr, *dP1 = nullptr, *dE1 = nullptr;
  cudaStream_t stream = nullptr;
  long long launches = 0;  // kernels launched by inference / training
  // identity of this network and of its workspace, for captured guesses: a
  // graph holds the workspace's addresses, so it is keyed on both
  unsigned long long uid = 0, gen = 0;
};

static unsigned long long g_net_uid = 0;

static void free_work(bbpp_net *n) {
  n->gen++;
  void *ptrs[] = {n->X0, n->CAT1, n->P1, n->CAT2, n->P2, n->E3, n->D2, n->D1, n->OUT, n->dOUT, n->scales, n->sums,
                  n->lossd, n->dD1, n->G, n->dCAT1, n->dD2, n->dCAT2, n->dE3, n->dP2, n->dE2, n->dP1, n->dE1,
                  n->bsum};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  n->X0 = n->CAT1 = n->P1 = n->CAT2 = n->P2 = n->E3 = n->D2 = n->D1 = nullptr;
  n->OUT = n->dOUT = n->scales = nullptr;
  n->sums = n->lossd = nullptr;
  n->bsum = nullptr;
  n->dD1 = n->G = n->dCAT1 = n->dD2 = n->dCAT2 = n->dE3 = n->dP2 = n->dE2 = n->dP1 = n->dE1 = nullptr;
  n->wx = n->wy = n->wz = n->wb = 0;
}

static int ensure_work(bbpp_net *n, int nx, int ny, int nz, int nb, bool grads) {
  if (n->wx == nx && n->wy == ny && n->wz == nz && n->wb == nb && (n->wgrad || !grads)) return 0;
  free_work(n);
  const size_t V = (size_t)nx * ny * nz * nb, V2 = V / 8, V4 = V / 64;
  const size_t B = sizeof(bf16);
  NCK(cudaMalloc(&n->X0, V * 16 * B));
  NCK(cudaMalloc(&n->CAT1, V * 48 * B));
  NCK(cudaMalloc(&n->P1, V2 * 16 * B));
  NCK(cudaMalloc(&n->CAT2, V2 * 96 * B));
  NCK(cudaMalloc(&n->P2, V4 * 32 * B));
  NCK(cudaMalloc(&n->E3, V4 * 64 * B));
  NCK(cudaMalloc(&n->D2, V2 * 32 * B));
  NCK(cudaMalloc(&n->D1, V * 16 * B));
  NCK(cudaMalloc(&n->OUT, V * sizeof(float)));
  NCK(cudaMalloc(&n->scales, 2 * nb * sizeof(float)));
  NCK(cudaMalloc(&n->sums, 4 * nb * sizeof(double)));
  NCK(cudaMalloc(&n->lossd, sizeof(double)));
  if (grads) {
    NCK(cudaMalloc(&n->dOUT, V * sizeof(float)));
    NCK(cudaMalloc(&n->dD1, V * 16 * B));
    NCK(cudaMalloc(&n->G, V * 32 * B));  // largest gated gradient: [V][16] or [V/8][32] or [V/64][64]
    NCK(cudaMalloc(&n->dCAT1, V * 48 * B));
    NCK(cudaMalloc(&n->dD2, V2 * 32 * B));
    NCK(cudaMalloc(&n->dCAT2, V2 * 96 * B));
    NCK(cudaMalloc(&n->dE3, V4 * 64 * B));
    NCK(cudaMalloc(&n->dP2, V4 * 32 * B));
    NCK(cudaMalloc(&n->dE2, V2 * 32 * B));
    NCK(cudaMalloc(&n->dP1, V2 * 16 * B));
    NCK(cudaMalloc(&n->dE1, V * 16 * B));
    NCK(cudaMalloc(&n->bsum, NLAYER * 64 * kGateSums * sizeof(double)));
  }
  n->wx = nx;
  n->wy = ny;
  n->wz = nz;
  n->wb = nb;
  n->wgrad = grads;
  return 0;
}

static int check_dims(int nx, int ny, int nz) {
  if (nx < 4 || ny < 4 || nz < 4 || nx % 4 || ny % 4 || nz % 4) return BBPP_BAD_ARG;
  return 0;
}

static ConvArgs cargs(const bbpp_net *n, int nx, int ny, int nz, int nb, const bf16 *in, int ldi, int cio,
                      const bf16 *w, const float *bias, bf16 *out, int ldo, int coo, int relu) {
  ConvArgs a;
  a.in = in;
  a.ldi = ldi;
  a.ci_off = cio;
  a.w = w;
  a.bias = bias;
  a.out = out;
  a.ldo = ldo;
  a.co_off = coo;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.nb = nb;
  a.px = 1;
  a.py = 1;
  a.pz = 0;
  a.relu = relu;
  (void)n;
  return a;
}

static WgradArgs wargs(int nx, int ny, int nz, int nb, const bf16 *in, int ldi, int cio, const bf16 *g, int ldg,
                       float *dW) {
  WgradArgs a;
  a.in = in;
  a.ldi = ldi;
  a.ci_off = cio;
  a.g = g;
  a.ldg = ldg;
  a.cg_off = 0;
  a.dW = dW;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.nb = nb;
  a.px = 1;
  a.py = 1;
  a.pz = 0;
  a.tiles_per_cta = 1;
  return a;
}

// refresh the BF16 weight copies after a parameter change
static int sync_weights(bbpp_net *n) {
  cudaStream_t s = n->stream;
  k_f32_to_bf16<<<nblocks(n->np), 256, 0, s>>>(n->w, n->w16, n->np);
  for (int l = 0; l < NLAYER; l++) {
    const ConvLayer &L = n->L[l];
    k_wflip<<<nblocks(27 * L.cin * L.cout), 256, 0, s>>>(n->w16 + L.woff, n->wt16 + L.woff, L.cin, L.cout);
  }
  NCK(cudaGetLastError());
  return 0;
}

// Forward pass on X0 (already prepared) -> OUT.
static int forward(bbpp_net *n, int nx, int ny, int nz, int nb) {
  cudaStream_t s = n->stream;
  const int hx = nx / 2, hy = ny / 2, hz = nz / 2, qx = nx / 4, qy = ny / 4, qz = nz / 4;
  const long long V = (long long)nx * ny * nz * nb;
  const bf16 *W = n->w16;
  const float *Bf = n->w;
  const ConvLayer *L = n->L;
  cudaError_t e;
  // E1 -> CAT1[:, 32:48]
  e = conv_fwd(16, 16, cargs(n, nx, ny, nz, nb, n->X0, 16, 0, W + L[0].woff, Bf + L[0].boff, n->CAT1, 48, 32, 1), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  k_pool_fwd<<<nblocks(V / 8 * 16), 256, 0, s>>>(n->CAT1, 48, 32, 16, nx, ny, nz, nb, n->P1);
  // E2 -> CAT2[:, 64:96]
  e = conv_fwd(16, 32, cargs(n, hx, hy, hz, nb, n->P1, 16, 0, W + L[1].woff, Bf + L[1].boff, n->CAT2, 96, 64, 1), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  k_pool_fwd<<<nblocks(V / 64 * 32), 256, 0, s>>>(n->CAT2, 96, 64, 32, hx, hy, hz, nb, n->P2);
  e = conv_fwd(32, 64, cargs(n, qx, qy, qz, nb, n->P2, 32, 0, W + L[2].woff, Bf + L[2].boff, n->E3, 64, 0, 1), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  k_up_fwd<<<nblocks(V / 8 * 64), 256, 0, s>>>(n->E3, 64, hx, hy, hz, nb, n->CAT2, 96, 0);
  e = conv_fwd(96, 32, cargs(n, hx, hy, hz, nb, n->CAT2, 96, 0, W + L[3].woff, Bf + L[3].boff, n->D2, 32, 0, 1), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  k_up_fwd<<<nblocks(V * 32), 256, 0, s>>>(n->D2, 32, nx, ny, nz, nb, n->CAT1, 48, 0);
  e = conv_fwd(48, 16, cargs(n, nx, ny, nz, nb, n->CAT1, 48, 0, W + L[4].woff, Bf + L[4].boff, n->D1, 16, 0, 1), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  k_head_fwd<<<nblocks(V), 256, 0, s>>>(n->D1, n->w + n->head_w, n->w + n->head_b, V, n->OUT);
  n->launches += 10;
  NCK(cudaGetLastError());
  return 0;
}

// Backward pass from dOUT; accumulates into n->g (which the caller zeroes).
static int backward(bbpp_net *n, int nx, int ny, int nz, int nb) {
  cudaStream_t s = n->stream;
  const int hx = nx / 2, hy = ny / 2, hz = nz / 2, qx = nx / 4, qy = ny / 4, qz = nz / 4;
  const long long V = (long long)nx * ny * nz * nb, V2 = V / 8, V4 = V / 64;
  const ConvLayer *L = n->L;
  float *G32 = n->g;
  cudaError_t e;
  NCK(cudaMemsetAsync(n->bsum, 0, NLAYER * 64 * kGateSums * sizeof(double), s));
  k_head_bwd<<<nblocks(V), 256, 0, s>>>(n->dOUT, n->D1, n->w + n->head_w, V, n->dD1, G32 + n->head_w,
                                        G32 + n->head_b);
  // D1 = relu(conv(CAT1))
  k_gate_bias<<<std::min(nblocks(V * 2), kGateCtas), 256, 0, s>>>(n->dD1, n->D1, 16, 0, 16, V, n->G,
                                                                  n->bsum + 4 * 64 * kGateSums);
  e = conv_wgrad(48, 16, wargs(nx, ny, nz, nb, n->CAT1, 48, 0, n->G, 16, G32 + L[4].woff), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  e = conv_fwd(16, 48, cargs(n, nx, ny, nz, nb, n->G, 16, 0, n->wt16 + L[4].woff, nullptr, n->dCAT1, 48, 0, 0), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  // CAT1[:, 0:32] = up(D2)
  k_up_bwd<<<nblocks(V2 * 32), 256, 0, s>>>(n->dCAT1, 48, 0, 32, nx, ny, nz, nb, n->dD2);
  // D2 = relu(conv(CAT2))
  k_gate_bias<<<std::min(nblocks(V2 * 4), kGateCtas), 256, 0, s>>>(n->dD2, n->D2, 32, 0, 32, V2, n->G,
                                                                  n->bsum + 3 * 64 * kGateSums);
  e = conv_wgrad(96, 32, wargs(hx, hy, hz, nb, n->CAT2, 96, 0, n->G, 32, G32 + L[3].woff), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  e = conv_fwd(32, 96, cargs(n, hx, hy, hz, nb, n->G, 32, 0, n->wt16 + L[3].woff, nullptr, n->dCAT2, 96, 0, 0), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  // CAT2[:, 0:64] = up(E3)
  k_up_bwd<<<nblocks(V4 * 64), 256, 0, s>>>(n->dCAT2, 96, 0, 64, hx, hy, hz, nb, n->dE3);
  // E3 = relu(conv(P2))
  k_gate_bias<<<std::min(nblocks(V4 * 8), kGateCtas), 256, 0, s>>>(n->dE3, n->E3, 64, 0, 64, V4, n->G,
                                                                  n->bsum + 2 * 64 * kGateSums);
  e = conv_wgrad(32, 64, wargs(qx, qy, qz, nb, n->P2, 32, 0, n->G, 64, G32 + L[2].woff), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  e = conv_fwd(64, 32, cargs(n, qx, qy, qz, nb, n->G, 64, 0, n->wt16 + L[2].woff, nullptr, n->dP2, 32, 0, 0), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  // E2 (in CAT2[:, 64:96]): skip gradient dCAT2[:, 64:96] + pool backward of dP2
  k_pool_bwd<<<nblocks(V2 * 32), 256, 0, s>>>(n->dP2, n->dCAT2, 96, 64, 32, hx, hy, hz, nb, n->dE2);
  k_gate_bias<<<std::min(nblocks(V2 * 4), kGateCtas), 256, 0, s>>>(n->dE2, n->CAT2, 96, 64, 32, V2, n->G,
                                                                  n->bsum + 1 * 64 * kGateSums);
  e = conv_wgrad(16, 32, wargs(hx, hy, hz, nb, n->P1, 16, 0, n->G, 32, G32 + L[1].woff), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  e = conv_fwd(32, 16, cargs(n, hx, hy, hz, nb, n->G, 32, 0, n->wt16 + L[1].woff, nullptr, n->dP1, 16, 0, 0), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  // E1 (in CAT1[:, 32:48]): skip gradient dCAT1[:, 32:48] + pool backward of dP1
  k_pool_bwd<<<nblocks(V * 16), 256, 0, s>>>(n->dP1, n->dCAT1, 48, 32, 16, nx, ny, nz, nb, n->dE1);
  k_gate_bias<<<std::min(nblocks(V * 2), kGateCtas), 256, 0, s>>>(n->dE1, n->CAT1, 48, 32, 16, V, n->G,
                                                                  n->bsum + 0 * 64 * kGateSums);
  e = conv_wgrad(16, 16, wargs(nx, ny, nz, nb, n->X0, 16, 0, n->G, 16, G32 + L[0].woff), s);
  if (e != cudaSuccess) return BBPP_CUDA_ERROR;
  BiasOffsets B;
  for (int l = 0; l < NLAYER; l++) {
    B.off[l] = L[l].boff;
    B.n[l] = L[l].cout;
  }
  k_bias_out<<<NLAYER, 256, 0, s>>>(n->bsum, B, G32);
  NCK(cudaGetLastError());
  return 0;
}

// scales from rhs and (optionally) prev, then X0
template <typename T>
static int prepare(bbpp_net *n, int nx, int ny, int nz, int nb, const T *rhs, const T *prev, const uint8_t *mask) {
  cudaStream_t s = n->stream;
  const long long vol = (long long)nx * ny * nz;
  NCK(cudaMemsetAsync(n->sums, 0, 4 * nb * sizeof(double), s));
  dim3 g(std::min(nblocks(vol), 512), nb);
  k_fluid_sumsq<T><<<g, 256, 0, s>>>(rhs, mask, vol, nb, n->sums);
  if (prev) k_fluid_sumsq<T><<<g, 256, 0, s>>>(prev, mask, vol, nb, n->sums + 2 * nb);
  k_scales<<<1, 256, 0, s>>>(n->sums, prev ? n->sums + 2 * nb : nullptr, nb, n->scales);
  k_prep<T><<<nblocks(vol * nb), 256, 0, s>>>(rhs, prev, mask, n->scales, vol, nb, n->X0);
  n->launches += prev ? 4 : 3;
  NCK(cudaGetLastError());
  return 0;
}

// ------------------------------------------------------------------- ABI --
static unsigned long long rng_next(unsigned long long &v) {  // Ranq1 (src/rng.c:28-51)
  v ^= v >> 21;
  v ^= v << 35;
  v ^= v >> 4;
  return v * 2685821657736338717ULL;
}

extern "C" int bbpp_net_create(unsigned long long seed, bbpp_net **out) {
  if (!out) return BBPP_BAD_ARG;
  bbpp_net *n = new bbpp_net();
  n->uid = __atomic_add_fetch(&g_net_uid, 1ull, __ATOMIC_RELAXED);
  int off = 0;
  for (int l = 0; l < NLAYER; l++) {
    n->L[l] = kLayers[l];
    n->L[l].woff = off;
    off += 27 * n->L[l].cin * n->L[l].cout;
    n->L[l].boff = off;
    off += n->L[l].cout;
  }
  n->head_w = off;
  off += 16;
  n->head_b = off;
  off += 1;
  n->np = off;
  // He-uniform initialisation from Ranq1; biases zero; the real input
  // channels of the first layer are 3 of its 16
  std::vector<float> h(n->np, 0.f);
  unsigned long long v = 4101842887655102017ULL ^ seed;
  rng_next(v);
  for (int l = 0; l < NLAYER; l++) {
    const ConvLayer &L = n->L[l];
    const int fan_in = 27 * (l == 0 ? 3 : L.cin);
    const float bound = sqrtf(6.f / fan_in);
    for (int t = 0; t < 27; t++)
      for (int co = 0; co < L.cout; co++)
        for (int ci = 0; ci < L.cin; ci++) {
          const double u = 5.42101086242752217e-20 * (double)rng_next(v);
          const float val = (l == 0 && ci >= 3) ? 0.f : (float)((2 * u - 1) * bound);
          h[L.woff + (t * L.cout + co) * L.cin + ci] = val;
        }
  }
  for (int c = 0; c < 16; c++) {
    const double u = 5.42101086242752217e-20 * (double)rng_next(v);
    h[n->head_w + c] = (float)((2 * u - 1) * sqrtf(6.f / 16.f) * 0.1f);
  }
  cudaError_t e = cudaMalloc(&n->w, n->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&n->g, n->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&n->m, n->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&n->v, n->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMalloc(&n->w16, n->np * sizeof(bf16));
  if (e == cudaSuccess) e = cudaMalloc(&n->wt16, n->np * sizeof(bf16));
  if (e == cudaSuccess) e = cudaMemcpy(n->w, h.data(), n->np * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(n->g, 0, n->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(n->m, 0, n->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(n->v, 0, n->np * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(n->wt16, 0, n->np * sizeof(bf16));
  if (e != cudaSuccess) {
    fprintf(stderr, "bbpp_net_create: %s\n", cudaGetErrorString(e));
    bbpp_net_destroy(n);
    return BBPP_CUDA_ERROR;
  }
  int rc = sync_weights(n);
  if (rc) {
    bbpp_net_destroy(n);
    return rc;
  }
  cudaDeviceSynchronize();
  *out = n;
  return 0;
}

extern "C" int bbpp_net_destroy(bbpp_net *n) {
  if (!n) return BBPP_BAD_ARG;
  free_work(n);
  void *ptrs[] = {n->w, n->g, n->m, n->v, n->w16, n->wt16};
  for (void *p : ptrs)
    if (p) cudaFree(p);
  delete n;
  return 0;
}

extern "C" int bbpp_net_num_params(const bbpp_net *n) { return n ? n->np : 0; }

extern "C" int bbpp_net_get_params(const bbpp_net *n, float *host) {
  if (!n || !host) return BBPP_BAD_ARG;
  NCK(cudaMemcpy(host, n->w, n->np * sizeof(float), cudaMemcpyDeviceToHost));
  return 0;
}

extern "C" int bbpp_net_set_params(bbpp_net *n, const float *host) {
  if (!n || !host) return BBPP_BAD_ARG;
  NCK(cudaMemcpy(n->w, host, n->np * sizeof(float), cudaMemcpyHostToDevice));
  int rc = sync_weights(n);
  if (rc) return rc;
  NCK(cudaStreamSynchronize(n->stream));
  return 0;
}

// Forward (FP32 inputs), loss and gradients: loss to *loss, gradients to grads
// (host, np floats) when not null.  Volumes of nx*ny*nz stacked nb times;
// mask (one volume) may be null.  rhs holds the residual r of p_prev, target
// the correction p* - p_prev; h2 is the squared grid spacing.
extern "C" int bbpp_net_loss_grad(bbpp_net *n, int nx, int ny, int nz, int nb, double h2, const float *rhs,
                                  const float *prev, const float *target, const uint8_t *mask, double *loss,
                                  float *grads) {
  if (!n || !rhs || !target || nb < 1) return BBPP_BAD_ARG;
  int rc = check_dims(nx, ny, nz);
  if (rc) return rc;
  rc = ensure_work(n, nx, ny, nz, nb, true);
  if (rc) return rc;
  rc = prepare<float>(n, nx, ny, nz, nb, rhs, prev, mask);
  if (rc) return rc;
  rc = forward(n, nx, ny, nz, nb);
  if (rc) return rc;
  cudaStream_t s = n->stream;
  const long long vol = (long long)nx * ny * nz;
  // fluid count over all volumes
  long long nfl = vol;
  if (mask) {
    std::vector<uint8_t> hm(vol);
    NCK(cudaMemcpy(hm.data(), mask, vol, cudaMemcpyDeviceToHost));
    nfl = 0;
    for (long long i = 0; i < vol; i++) nfl += hm[i] == 0;
  }
  const double inv_n = 1.0 / std::max<long long>(1, nfl * nb);
  NCK(cudaMemsetAsync(n->lossd, 0, sizeof(double), s));
  k_loss<<<std::min(nblocks(vol * nb), 1024), 256, 0, s>>>(n->OUT, target, mask, n->scales, vol, nb, inv_n,
                                                            (float)(1.0 / h2), n->dOUT, n->lossd);
  NCK(cudaMemsetAsync(n->g, 0, n->np * sizeof(float), s));
  rc = backward(n, nx, ny, nz, nb);
  if (rc) return rc;
  if (loss) NCK(cudaMemcpyAsync(loss, n->lossd, sizeof(double), cudaMemcpyDeviceToHost, s));
  if (grads) NCK(cudaMemcpyAsync(grads, n->g, n->np * sizeof(float), cudaMemcpyDeviceToHost, s));
  NCK(cudaStreamSynchronize(s));
  return 0;
}

// Train on a device-resident set of nsamples volumes (FP32 rhs, prev, target;
// one shared mask): `steps` Adam steps on batches of `batch` volumes drawn
// with Ranq1.  loss_hist (host, steps) may be null.
extern "C" int bbpp_net_train(bbpp_net *n, int nx, int ny, int nz, int nsamples, double h2, const float *rhs,
                              const float *prev, const float *target, const uint8_t *mask, int steps, int batch,
                              float lr, unsigned long long seed, float *loss_hist) {
  if (!n || !rhs || !target || nsamples < 1 || batch < 1 || steps < 0) return BBPP_BAD_ARG;
  int rc = check_dims(nx, ny, nz);
  if (rc) return rc;
  const long long vol = (long long)nx * ny * nz;
  float *brhs = nullptr, *bprev = nullptr, *btgt = nullptr;
  NCK(cudaMalloc(&brhs, vol * batch * sizeof(float)));
  NCK(cudaMalloc(&bprev, vol * batch * sizeof(float)));
  NCK(cudaMalloc(&btgt, vol * batch * sizeof(float)));
  unsigned long long v = 4101842887655102017ULL ^ seed;
  rng_next(v);
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int it = 0; it < steps; it++) {
    for (int b = 0; b < batch; b++) {
      const int k = (int)(rng_next(v) % (unsigned long long)nsamples);
      NCK(cudaMemcpyAsync(brhs + b * vol, rhs + k * vol, vol * sizeof(float), cudaMemcpyDeviceToDevice, n->stream));
      if (prev)
        NCK(cudaMemcpyAsync(bprev + b * vol, prev + k * vol, vol * sizeof(float), cudaMemcpyDeviceToDevice,
                            n->stream));
      NCK(cudaMemcpyAsync(btgt + b * vol, target + k * vol, vol * sizeof(float), cudaMemcpyDeviceToDevice,
                          n->stream));
    }
    double loss = 0;
    rc = bbpp_net_loss_grad(n, nx, ny, nz, batch, h2, brhs, prev ? bprev : nullptr, btgt, mask, &loss, nullptr);
    if (rc) break;
    n->t++;
    const float c1 = 1.f / (1.f - powf(b1, (float)n->t)), c2 = 1.f / (1.f - powf(b2, (float)n->t));
    // cosine decay of the learning rate
    const float lrt = lr * 0.5f * (1.f + cosf(3.14159265f * (float)it / (float)std::max(1, steps)));
    k_adam<<<nblocks(n->np), 256, 0, n->stream>>>(n->w, n->g, n->m, n->v, n->np, lrt, b1, b2, eps, c1, c2);
    rc = sync_weights(n);
    if (rc) break;
    if (loss_hist) loss_hist[it] = (float)loss;
  }
  cudaStreamSynchronize(n->stream);
  cudaFree(brhs);
  cudaFree(bprev);
  cudaFree(btgt);
  return rc;
}

// Inference for one volume (FP64 r = rhs - (-A) p_prev and p_prev, as the
// solver holds them) into p0 = p_prev + h2 OUT / (1/s_r) (FP64), 0 on solid cells.
extern "C" int bbpp_net_infer(bbpp_net *n, int nx, int ny, int nz, double h2, const double *rhs,
                              const double *prev, const uint8_t *mask, double *p0) {
  if (!n || !rhs || !p0) return BBPP_BAD_ARG;
  int rc = check_dims(nx, ny, nz);
  if (rc) return rc;
  rc = ensure_work(n, nx, ny, nz, 1, false);
  if (rc) return rc;
  rc = prepare<double>(n, nx, ny, nz, 1, rhs, prev, mask);
  if (rc) return rc;
  rc = forward(n, nx, ny, nz, 1);
  if (rc) return rc;
  const long long vol = (long long)nx * ny * nz;
  k_guess_out<<<nblocks(vol), 256, 0, n->stream>>>(n->OUT, prev, mask, n->scales, h2, vol, p0);
  n->launches += 1;
  NCK(cudaGetLastError());
  return 0;
}

extern "C" int bbpp_net_set_stream(bbpp_net *n, void *stream) {
  if (!n) return BBPP_BAD_ARG;
  n->stream = (cudaStream_t)stream;
  return 0;
}

extern "C" int bbpp_net_save(const bbpp_net *n, const char *path) {
  if (!n || !path) return BBPP_BAD_ARG;
  std::vector<float> h(3 * (size_t)n->np);
  NCK(cudaMemcpy(h.data(), n->w, n->np * sizeof(float), cudaMemcpyDeviceToHost));
  NCK(cudaMemcpy(h.data() + n->np, n->m, n->np * sizeof(float), cudaMemcpyDeviceToHost));
  NCK(cudaMemcpy(h.data() + 2 * n->np, n->v, n->np * sizeof(float), cudaMemcpyDeviceToHost));
  FILE *f = fopen(path, "wb");
  if (!f) return BBPP_BAD_ARG;
  const char magic[8] = {'B', 'B', 'P', 'P', 'N', 'E', 'T', '1'};
  fwrite(magic, 1, 8, f);
  fwrite(&n->np, sizeof(int), 1, f);
  fwrite(&n->t, sizeof(int), 1, f);
  fwrite(h.data(), sizeof(float), h.size(), f);
  fclose(f);
  return 0;
}

extern "C" int bbpp_net_load(bbpp_net *n, const char *path) {
  if (!n || !path) return BBPP_BAD_ARG;
  FILE *f = fopen(path, "rb");
  if (!f) return BBPP_BAD_ARG;
  char magic[8];
  int np = 0, t = 0;
  std::vector<float> h(3 * (size_t)n->np);
  bool ok = fread(magic, 1, 8, f) == 8 && memcmp(magic, "BBPPNET1", 8) == 0 && fread(&np, sizeof(int), 1, f) == 1 &&
            np == n->np && fread(&t, sizeof(int), 1, f) == 1 && fread(h.data(), sizeof(float), h.size(), f) == h.size();
  fclose(f);
  if (!ok) return BBPP_BAD_ARG;
  NCK(cudaMemcpy(n->w, h.data(), n->np * sizeof(float), cudaMemcpyHostToDevice));
  NCK(cudaMemcpy(n->m, h.data() + n->np, n->np * sizeof(float), cudaMemcpyHostToDevice));
  NCK(cudaMemcpy(n->v, h.data() + 2 * n->np, n->np * sizeof(float), cudaMemcpyHostToDevice));
  n->t = t;
  int rc = sync_weights(n);
  if (rc) return rc;
  NCK(cudaDeviceSynchronize());
  return 0;
}

// Kernel-level entry points for tests: one 3x3x3 convolution (forward, or
// dgrad with `flip`), and a weight gradient, on BF16 channels-last volumes.
extern "C" int bbpp_conv3(int cin, int cout, const void *in, int ldi, int ci_off, const void *w, const float *bias,
                          void *out, int ldo, int co_off, int nx, int ny, int nz, int nb, int px, int py, int pz,
                          int relu) {
  ConvArgs a;
  a.in = (const bf16 *)in;
  a.ldi = ldi;
  a.ci_off = ci_off;
  a.w = (const bf16 *)w;
  a.bias = bias;
  a.out = (bf16 *)out;
  a.ldo = ldo;
  a.co_off = co_off;
  a.nx = nx;
  a.ny = ny;
  a.nz = nz;
  a.nb = nb;
  a.px = px;
  a.py = py;
  a.pz = pz;
  a.relu = relu;
  if (ldi % 8 || ci_off % 8 || ldo % 2 || co_off % 2 || nb < 1 || nx < 1 || ny < 1 || nz < 1) return BBPP_BAD_ARG;
  if (conv_fwd(cin, cout, a, 0) != cudaSuccess) return BBPP_BAD_ARG;
  NCK(cudaDeviceSynchronize());
  if (conv_tc_failed()) return BBPP_WAIT_TIMEOUT;
  return 0;
}

// Number of convolutions that ran on the tcgen05 kernel in this process.
extern "C" long long bbpp_conv3_tc_launches(void) { return g_tc_launches; }

// Kernel choice: mma.sync (0), k_conv3_tm (1), k_conv3_tx (2), or (-1) leave the
// choice to BBPP_CONV_TC; and cap the persistent grid (0: one CTA per SM).
extern "C" int bbpp_conv3_tc_config(int enable, int max_ctas) {
  if (enable < -1 || enable > 2 || max_ctas < 0) return BBPP_BAD_ARG;
  g_tc_on = enable;
  g_tc_max_ctas = max_ctas;
  return 0;
}

extern "C" int bbpp_conv3_wgrad(int cin, int cout, const void *in, int ldi, int ci_off, const void *g, int ldg,
                                float *dW, int nx, int ny, int nz, int nb, int px, int py, int pz) {
  WgradArgs a = wargs(nx, ny, nz, nb, (const bf16 *)in, ldi, ci_off, (const bf16 *)g, ldg, dW);
  a.px = px;
  a.py = py;
  a.pz = pz;
  if (ldi % 8 || ci_off % 8 || ldg % 8 || nb < 1) return BBPP_BAD_ARG;
  if (conv_wgrad(cin, cout, a, 0) != cudaSuccess) return BBPP_BAD_ARG;
  NCK(cudaDeviceSynchronize());
  return 0;
}

extern "C" int bbpp_conv3_wflip(int cin, int cout, const void *w, void *wt) {
  k_wflip<<<nblocks(27 * cin * cout), 256>>>((const bf16 *)w, (bf16 *)wt, cin, cout);
  NCK(cudaGetLastError());
  NCK(cudaDeviceSynchronize());
  return 0;
}

// ------------------------------------------------------ solver hook -------
// The guess's launches as a CUDA graph: one per (network, buffers, grid,
// restriction), captured the second time the same guess runs (the first run
// sizes the network's workspace and builds its tensor maps, which a capture
// must not do) and replayed after that.
struct GuessKey {
  unsigned long long net, gen;  // the network's identity and workspace generation
  const void *mask, *rhs, *prev, *x;
  int f, tc, tc_ctas;
  bool operator==(const GuessKey &o) const {
    return net == o.net && gen == o.gen && mask == o.mask && rhs == o.rhs && prev == o.prev && x == o.x &&
           f == o.f && tc == o.tc && tc_ctas == o.tc_ctas;
  }
};
struct GuessGraph {
  GuessKey key;
  cudaGraphExec_t exec = nullptr;  // null: seen once, not yet captured
  long long launches = 0;          // kernels in the graph
};

struct NetWork {
  double *prev0 = nullptr;  // zero "previous pressure" when none is given
  // the problem restricted by 2: r, p_prev, the network's p0; the solid cells
  double *rc = nullptr, *pc = nullptr, *p0c = nullptr;
  float *corr = nullptr;  // p0c - pc in FP32 (0 on coarse solid cells)
  uint8_t *mc = nullptr;
  long long ncap = 0;
  std::vector<GuessGraph> graphs;  // at most 4, oldest dropped first
};

static void drop_guess_graphs(NetWork *w) {
  for (auto &g : w->graphs)
    if (g.exec) cudaGraphExecDestroy(g.exec);
  w->graphs.clear();
}

// The learned guess of a solve.  coarsen F = 2 or 4: the network runs on the
// problem restricted by F (k_resid_restrict) with h^2 scaled by F^2, and its
// correction comes back by trilinear interpolation (k_prolong); at 256^3 and
// F = 2 this both costs 1/8 of the inference and gives a better guess (the
// network sees twice as far in fine cells).  F needs every extent a multiple
// of 4F (the network pools twice).  coarsen 0 picks 2 when every extent is a
// multiple of 8 and at least 128.
int bbpp_net_guess(bbpp_ctx *ctx, void *netp, const uint8_t *mask, const double *rhs, const double *prev, double *x,
                   int coarsen, double *ms) {
  bbpp_net *n = (bbpp_net *)netp;
  if (!n) return BBPP_BAD_ARG;
  const int nx = ctx->G.nx, ny = ctx->G.ny, nz = ctx->G.nz;
  auto fits = [&](int F) { return nx % (4 * F) == 0 && ny % (4 * F) == 0 && nz % (4 * F) == 0; };
  int f = coarsen;
  if (f == 0) f = (fits(2) && std::min(nx, std::min(ny, nz)) >= 128) ? 2 : 1;
  if (f != 1 && f != 2 && f != 4) return BBPP_BAD_ARG;
  if (f > 1 && !fits(f)) return BBPP_BAD_ARG;
  if (f > 1) {
    if (!ctx->net) ctx->net = new NetWork();
    NetWork *w = ctx->net;
    const long long nc = (long long)(nx / f) * (ny / f) * (nz / f);
    if (w->ncap < nc) {
      cudaFree(w->rc);
      cudaFree(w->pc);
      cudaFree(w->p0c);
      cudaFree(w->mc);
      cudaFree(w->corr);
      w->rc = w->pc = w->p0c = nullptr;
      w->corr = nullptr;
      w->mc = nullptr;
      w->ncap = 0;
      NCK(cudaMalloc(&w->rc, nc * sizeof(double)));
      NCK(cudaMalloc(&w->pc, nc * sizeof(double)));
      NCK(cudaMalloc(&w->p0c, nc * sizeof(double)));
      NCK(cudaMalloc(&w->mc, nc));
      NCK(cudaMalloc(&w->corr, nc * sizeof(float)));
      w->ncap = nc;
    }
  }
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  cudaStream_t saved = n->stream;
  n->stream = ctx->stream;
  cudaEventRecord(e0, ctx->stream);
  const double h2 = ctx->grid.dx * ctx->grid.dy;
  // the guess's launches: residual of the warm start (into the solver's free Ap
  // buffer; the coarse path forms it inside its restriction), network, and on
  // the coarse path the correction's interpolation; returns the kernels launched
  auto body = [&](long long *count) -> int {
    const long long l0 = n->launches;
    int rc_ = 0;
    const double *r = rhs;
    if (prev && f == 1) {
      rc_ = bbpp_residual_async(ctx, mask, rhs, prev, ctx->Ap);
      r = ctx->Ap;
    }
    if (f > 1) {
      NetWork *w = ctx->net;
      const long long nc = (long long)(nx / f) * (ny / f) * (nz / f);
      if (rc_ == 0) {
        if (f == 2)
          k_resid_restrict<2><<<nblocks(nc), 256, 0, ctx->stream>>>(ctx->G, rhs, prev, mask, w->rc, w->pc, w->mc);
        else
          k_resid_restrict<4><<<nblocks(nc), 256, 0, ctx->stream>>>(ctx->G, rhs, prev, mask, w->rc, w->pc, w->mc);
        if (cudaGetLastError() != cudaSuccess) rc_ = BBPP_CUDA_ERROR;
      }
      if (rc_ == 0)
        rc_ = bbpp_net_infer(n, nx / f, ny / f, nz / f, (double)(f * f) * h2, w->rc, w->pc, mask ? w->mc : nullptr,
                             w->p0c);
      if (rc_ == 0) {
        k_corr2<<<nblocks(nc), 256, 0, ctx->stream>>>(w->corr, w->p0c, w->pc, w->mc, (unsigned)nc);
        if (f == 2)
          k_prolong<2><<<nblocks(ctx->G.n), 256, 0, ctx->stream>>>(w->corr, prev, mask, nx, ny, nz, ctx->G.px,
                                                                   ctx->G.py, ctx->G.pz, x);
        else
          k_prolong<4><<<nblocks(ctx->G.n), 256, 0, ctx->stream>>>(w->corr, prev, mask, nx, ny, nz, ctx->G.px,
                                                                   ctx->G.py, ctx->G.pz, x);
        if (cudaGetLastError() != cudaSuccess) rc_ = BBPP_CUDA_ERROR;
      }
      *count = (n->launches - l0) + 3;
    } else {
      if (rc_ == 0) rc_ = bbpp_net_infer(n, nx, ny, nz, h2, r, prev, mask, x);
      *count = (n->launches - l0) + (prev ? 1 : 0);
    }
    return rc_;
  };
  int rc = 0;
  long long count = 0;
  const char *ge = getenv("BBPP_GUESS_GRAPH");
  if (!ctx->net) ctx->net = new NetWork();
  NetWork *gw = ctx->net;
  // the network's workspace for this grid exists before the key is taken
  if (!(ge && ge[0] == '0')) {
    const int wnx = nx / f, wny = ny / f, wnz = nz / f;
    if (!(n->wx == wnx && n->wy == wny && n->wz == wnz && n->wb == 1)) rc = ensure_work(n, wnx, wny, wnz, 1, false);
  }
  const GuessKey key = {n->uid, n->gen, mask, rhs, prev, x, f, conv_tc_mode(), g_tc_max_ctas};
  GuessGraph *hit = nullptr;
  for (auto &g : gw->graphs)
    if (g.key == key) hit = &g;
  if (rc) {
    // the workspace could not be made
  } else if (ge && ge[0] == '0') {
    rc = body(&count);
  } else if (hit && hit->exec) {
    if (cudaGraphLaunch(hit->exec, ctx->stream) != cudaSuccess) rc = BBPP_CUDA_ERROR;
    count = hit->launches;
  } else if (hit) {
    // second run with these buffers: capture, then replay the capture
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) {
      rc = BBPP_CUDA_ERROR;
    } else {
      rc = body(&count);
      const cudaError_t ec = cudaStreamEndCapture(ctx->stream, &graph);
      if (rc == 0 && ec != cudaSuccess) rc = BBPP_CUDA_ERROR;
      if (rc == 0 && cudaGraphInstantiate(&exec, graph, 0) != cudaSuccess) rc = BBPP_CUDA_ERROR;
      if (graph) cudaGraphDestroy(graph);
    }
    if (rc == 0) {
      hit->exec = exec;
      hit->launches = count;
      if (cudaGraphLaunch(exec, ctx->stream) != cudaSuccess) rc = BBPP_CUDA_ERROR;
    } else {
      cudaGetLastError();
      rc = body(&count);  // the capture failed: run the launches directly
    }
  } else {
    rc = body(&count);
    if (gw->graphs.size() >= 4) {
      if (gw->graphs.front().exec) cudaGraphExecDestroy(gw->graphs.front().exec);
      gw->graphs.erase(gw->graphs.begin());
    }
    GuessGraph g;
    g.key = key;
    gw->graphs.push_back(g);
  }
  ctx->launches += count;
  cudaEventRecord(e1, ctx->stream);
  n->stream = saved;
  if (rc == 0) {
    cudaEventSynchronize(e1);
    if (conv_tc_failed()) rc = BBPP_WAIT_TIMEOUT;
    float t = 0.f;
    cudaEventElapsedTime(&t, e0, e1);
    if (ms) *ms = t;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return rc;
}

void bbpp_net_ctx_free(bbpp_ctx *ctx) {
  if (ctx && ctx->net) {
    drop_guess_graphs(ctx->net);
    if (ctx->net->prev0) cudaFree(ctx->net->prev0);
    cudaFree(ctx->net->rc);
    cudaFree(ctx->net->pc);
    cudaFree(ctx->net->p0c);
    cudaFree(ctx->net->mc);
    cudaFree(ctx->net->corr);
    delete ctx->net;
    ctx->net = nullptr;
  }
}
