// Learned dispatcher: MLP kernels (forward, backward, Adam, dispatch) and the
// C-ABI around them and around the per-row-block data they learn from.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "context.h"
#include "gen.h"

namespace tb {
namespace {

constexpr int kNorm = 2 * kIn + 2 * kOut;  // in_mean, in_std, out_mean, out_std
constexpr int kModelThreads = 256;
constexpr char kMagic[8] = {'T', 'B', 'M', 'L', 'P', '0', '0', '1'};

__host__ __device__ __forceinline__ bool is_weight(int p) {
  return p < kB1 || (p >= kW2 && p < kB2) || (p >= kW3 && p < kB3);
}

// Rows a warp carries through the network together (one float4 of a row's
// features a lane: kRows * kIn / 4 lanes). A weight read from shared memory
// then serves kRows rows, and a unit's activations are read back four at a time
// as one broadcast. One row a warp, its activations passed by shuffles, was
// bound by the shuffles and weight reads: 65,521 rows predicted in 110 us, now
// 36; forward and backward 161, now 71. A batch that leaves the chip idle is
// better spread (forward_backward): a training step of 32 rows takes 22.9 us with
// a row a warp and 29 with eight, of 512 25.4 and 33, of 1,024 30 with two and 36
// with eight, of 4,096 60 either way, of 8,192 98 with one and 95 with eight.
constexpr int kRows = 8;
static_assert(kRows * kIn <= 4 * 32, "a warp loads its rows of features as one float4 a lane");
constexpr int kW2tStride = kH1 + 1;  // padded: transposing W2 writes 32 different banks

// Shared-memory image of a model: parameters, normalisation and, for the
// backward pass, W2 transposed; and each warp's activations.
struct SmemModel {
  float p[kNumParams + 1];
  float norm[kNorm + 2];
  float act[kModelThreads / 32][kRows * kH1];
};
struct SmemTrain {
  SmemModel m;
  float w2t[kH2 * kW2tStride];
};
static_assert((kNumParams + 1) % 4 == 0 && (kNorm + 2) % 4 == 0, "activations are read as float4");

__device__ void load_model(SmemModel& s, const float* __restrict__ eff, const float* __restrict__ norm, float* w2t) {
  for (int i = threadIdx.x; i < kNumParams; i += blockDim.x) s.p[i] = eff[i];
  for (int i = threadIdx.x; i < kNorm; i += blockDim.x) s.norm[i] = norm[i];
  if (w2t)
    for (int i = threadIdx.x; i < kH1 * kH2; i += blockDim.x) w2t[(i % kH2) * kW2tStride + i / kH2] = eff[kW2 + i];
  __syncthreads();
}

struct Acts {  // per-row activations kept for the weight gradients
  float* xn;   // B x kIn
  float* h1;   // B x kH1
  float* dz1;  // B x kH1
  float* h2;   // B x kH2
  float* dz2;  // B x kH2
  float* dy;   // B x kOut
};

// a[r], b[r] += sum over the K inputs of row r (at h + r * K, ascending) times
// columns lane and lane + 32 of w (rows of `stride` floats).
template <int K, int R>
__device__ __forceinline__ void dense(const float* __restrict__ w, int stride, const float* __restrict__ h,
                                      float (&a)[R], float (&b)[R]) {
  const int lane = threadIdx.x & 31;
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float4 x[R];
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = *reinterpret_cast<const float4*>(h + r * K + k);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float wa = w[(k + q) * stride + lane], wb = w[(k + q) * stride + lane + 32];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float v = q == 0 ? x[r].x : q == 1 ? x[r].y : q == 2 ? x[r].z : x[r].w;
        a[r] = fmaf(v, wa, a[r]);
        b[r] = fmaf(v, wb, b[r]);
      }
    }
  }
}

// Lane l's two units of every row into the warp's activations.
template <int R>
__device__ __forceinline__ void put_units(float* act, const float (&a)[R], const float (&b)[R]) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r) {
    act[r * kH1 + lane] = a[r];
    act[r * kH1 + lane + 32] = b[r];
  }
  __syncwarp();
}

// R rows a warp; lane l owns hidden units l and l + 32 of both layers.
// Computes the normalised predictions of the rows x(r), r < rows (the others
// repeat row 0 and are not stored); with Train also the backward pass for the
// MSE loss on normalised targets y(r) (scaled by inv_count), storing what the
// weight-gradient kernel needs in slots slot .. slot + rows and returning the
// rows' summed squared error.
template <bool Train, int R, class RowOf>
__device__ __forceinline__ float rows_pass(const SmemModel& s, const float* w2t, float* act, const float* __restrict__ X,
                                           const float* __restrict__ Y, const RowOf& row_of, int rows, float inv_count,
                                           float (&out)[R][kOut], const Acts* acts, uint32_t slot) {
  const int lane = threadIdx.x & 31;
  __syncwarp();
  if (lane < R * kIn / 4) {
    const int r = lane / (kIn / 4), q = (lane % (kIn / 4)) * 4;
    const float4 x = *reinterpret_cast<const float4*>(X + (size_t)row_of(r < rows ? r : 0) * kIn + q);
    const float4 v = make_float4((x.x - s.norm[q]) / s.norm[kIn + q], (x.y - s.norm[q + 1]) / s.norm[kIn + q + 1],
                                 (x.z - s.norm[q + 2]) / s.norm[kIn + q + 2],
                                 (x.w - s.norm[q + 3]) / s.norm[kIn + q + 3]);
    *reinterpret_cast<float4*>(act + r * kIn + q) = v;
    if (Train && r < rows) *reinterpret_cast<float4*>(acts->xn + (size_t)(slot + r) * kIn + q) = v;
  }
  __syncwarp();
  float a[R], b[R];  // the layer's pre-activations
#pragma unroll
  for (int r = 0; r < R; ++r) a[r] = s.p[kB1 + lane], b[r] = s.p[kB1 + lane + 32];
  dense<kIn, R>(s.p + kW1, kH1, act, a, b);
  uint32_t on1 = 0;  // bits 2r, 2r + 1: row r's two units are active
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (Train) on1 |= (a[r] > 0.f ? 1u << (2 * r) : 0u) | (b[r] > 0.f ? 2u << (2 * r) : 0u);
    a[r] = fmaxf(a[r], 0.f), b[r] = fmaxf(b[r], 0.f);
    if (Train && r < rows) {
      acts->h1[(size_t)(slot + r) * kH1 + lane] = a[r];
      acts->h1[(size_t)(slot + r) * kH1 + lane + 32] = b[r];
    }
  }
  put_units<R>(act, a, b);
#pragma unroll
  for (int r = 0; r < R; ++r) a[r] = s.p[kB2 + lane], b[r] = s.p[kB2 + lane + 32];
  dense<kH1, R>(s.p + kW2, kH2, act, a, b);
  uint32_t on2 = 0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    if (Train) on2 |= (a[r] > 0.f ? 1u << (2 * r) : 0u) | (b[r] > 0.f ? 2u << (2 * r) : 0u);
    const float h2a = fmaxf(a[r], 0.f), h2b = fmaxf(b[r], 0.f);
#pragma unroll
    for (int o = 0; o < kOut; ++o)
      out[r][o] = s.p[kB3 + o] + warp_sum(h2a * s.p[kW3 + lane * kOut + o] + h2b * s.p[kW3 + (lane + 32) * kOut + o]);
    if (Train && r < rows) {
      acts->h2[(size_t)(slot + r) * kH2 + lane] = h2a;
      acts->h2[(size_t)(slot + r) * kH2 + lane + 32] = h2b;
    }
  }
  if constexpr (!Train) return 0.f;
  float sq = 0.f;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    float dh2a = 0.f, dh2b = 0.f;
    const size_t yr = (size_t)row_of(r < rows ? r : 0) * kOut;
#pragma unroll
    for (int o = 0; o < kOut; ++o) {
      const float t = (Y[yr + o] - s.norm[2 * kIn + o]) / s.norm[2 * kIn + kOut + o];
      const float e = out[r][o] - t;
      const float dy = 2.f * e * inv_count;
      dh2a = fmaf(s.p[kW3 + lane * kOut + o], dy, dh2a);
      dh2b = fmaf(s.p[kW3 + (lane + 32) * kOut + o], dy, dh2b);
      if (r < rows) {
        sq += e * e;
        if (lane == o) acts->dy[(size_t)(slot + r) * kOut + o] = dy;
      }
    }
    a[r] = (on2 >> (2 * r)) & 1u ? dh2a : 0.f;
    b[r] = (on2 >> (2 * r)) & 2u ? dh2b : 0.f;
    if (r < rows) {
      acts->dz2[(size_t)(slot + r) * kH2 + lane] = a[r];
      acts->dz2[(size_t)(slot + r) * kH2 + lane + 32] = b[r];
    }
  }
  put_units<R>(act, a, b);
#pragma unroll
  for (int r = 0; r < R; ++r) a[r] = 0.f, b[r] = 0.f;
  dense<kH2, R>(w2t, kW2tStride, act, a, b);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r < rows) {
      acts->dz1[(size_t)(slot + r) * kH1 + lane] = (on1 >> (2 * r)) & 1u ? a[r] : 0.f;
      acts->dz1[(size_t)(slot + r) * kH1 + lane + 32] = (on1 >> (2 * r)) & 2u ? b[r] : 0.f;
    }
  return sq;
}

// Forward + backward over rows idx[r0 .. r0 + B) (idx null: identity), R a warp.
template <int R>
__global__ void __launch_bounds__(kModelThreads) k_fwd_bwd(const float* __restrict__ X, const float* __restrict__ Y,
                                                            const uint32_t* __restrict__ idx, uint32_t r0, uint32_t B,
                                                            const float* __restrict__ eff,
                                                            const float* __restrict__ norm, float inv_count, Acts acts,
                                                            double* loss) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmemTrain& st = *reinterpret_cast<SmemTrain*>(smem_raw);
  load_model(st.m, eff, norm, st.w2t);
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  float* act = st.m.act[threadIdx.x >> 5];
  // The warps' sums are added as they finish, in double: in float, the order of arrival
  // left up to 3e-6 of the loss.
  double sq = 0.0;
  for (uint64_t i = (uint64_t)warp * R; i < B; i += (uint64_t)nw * R) {
    const uint32_t base = r0 + (uint32_t)i;
    float out[R][kOut];
    sq += rows_pass<true, R>(st.m, st.w2t, act, X, Y, [&](int r) { return idx ? idx[base + r] : base + r; },
                             (int)min((uint64_t)R, B - i), inv_count, out, &acts, (uint32_t)i);
  }
  if ((threadIdx.x & 31) == 0 && sq != 0.0) atomicAdd(loss, sq);
}

// The weight gradients in two steps: CTA c sums rows [c R, c R + R) of the
// batch into part[c] (every parameter's sum in registers, rows staged kGradTile
// at a time), and k_wgrad_sum, or the step that uses them (k_adam), adds the CTAs' sums in
// order, so the result depends on the batch size alone. The 64 x 64 block is 4 x 4 sums a thread (two 16-byte
// shared reads for 16 products). One thread a parameter walking all rows left
// all but 22 CTAs of the chip idle, each step a pair of dependent L2 reads:
// 65,521 rows in 4,656 us, now 99. Sizes: wgrad_rows, wgrad_ctas.
__global__ void __launch_bounds__(256) k_wgrad(Acts a, uint32_t B, float* __restrict__ part) {
  __shared__ __align__(16) float xn[kGradTile][kIn], h1[kGradTile][kH1], z1[kGradTile][kH1], h2[kGradTile][kH2],
      z2[kGradTile][kH2], dy[kGradTile][kOut];
  const int t = threadIdx.x, ti = t >> 4, tj = (t & 15) * 4;
  const uint32_t R = wgrad_rows(B);
  const uint32_t c0 = blockIdx.x * R;
  const uint32_t c1 = (uint32_t)min((uint64_t)B, (uint64_t)c0 + R);
  float g1[4] = {0.f, 0.f, 0.f, 0.f}, g2[4][4] = {}, g3 = 0.f, gb = 0.f;
  auto stage = [&](float* dst, const float* src, uint32_t words) {  // words: a multiple of 4, but for dy
    if (words % 4 == 0)
      for (uint32_t i = t; i < words / 4; i += 256)
        reinterpret_cast<float4*>(dst)[i] = reinterpret_cast<const float4*>(src)[i];
    else
      for (uint32_t i = t; i < words; i += 256) dst[i] = src[i];
  };
  for (uint32_t r0 = c0; r0 < c1; r0 += kGradTile) {
    const uint32_t n = min(kGradTile, c1 - r0);
    __syncthreads();
    stage(&xn[0][0], a.xn + (size_t)r0 * kIn, n * kIn);
    stage(&h1[0][0], a.h1 + (size_t)r0 * kH1, n * kH1);
    stage(&z1[0][0], a.dz1 + (size_t)r0 * kH1, n * kH1);
    stage(&h2[0][0], a.h2 + (size_t)r0 * kH2, n * kH2);
    stage(&z2[0][0], a.dz2 + (size_t)r0 * kH2, n * kH2);
    stage(&dy[0][0], a.dy + (size_t)r0 * kOut, n * kOut);
    __syncthreads();
    for (uint32_t r = 0; r < n; ++r) {
      const float4 h = *reinterpret_cast<const float4*>(&h1[r][ti * 4]);
      const float4 z = *reinterpret_cast<const float4*>(&z2[r][tj]);
      const float4 d = *reinterpret_cast<const float4*>(&z1[r][tj]);
      const float x = xn[r][ti];
      const float hv[4] = {h.x, h.y, h.z, h.w}, zv[4] = {z.x, z.y, z.z, z.w}, dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        g1[i] = fmaf(x, dv[i], g1[i]);
#pragma unroll
        for (int j = 0; j < 4; ++j) g2[i][j] = fmaf(hv[i], zv[j], g2[i][j]);
      }
      if (t < kH2 * kOut) g3 = fmaf(h2[r][t / kOut], dy[r][t % kOut], g3);
      if (t < kH1)
        gb += z1[r][t];
      else if (t < kH1 + kH2)
        gb += z2[r][t - kH1];
      else if (t < kH1 + kH2 + kOut)
        gb += dy[r][t - kH1 - kH2];
    }
  }
  float* out = part + (size_t)blockIdx.x * kNumParams;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    out[kW1 + ti * kH1 + tj + i] = g1[i];
#pragma unroll
    for (int j = 0; j < 4; ++j) out[kW2 + (ti * 4 + i) * kH2 + tj + j] = g2[i][j];
  }
  if (t < kH2 * kOut) out[kW3 + t] = g3;
  if (t < kH1)
    out[kB1 + t] = gb;
  else if (t < kH1 + kH2)
    out[kB2 + t - kH1] = gb;
  else if (t < kH1 + kH2 + kOut)
    out[kB3 + t - kH1 - kH2] = gb;
}
static_assert(kIn == 16 && kH1 == 64 && kH2 == 64 && kH2 * kOut <= 256 && kH1 + kH2 + kOut <= 256,
              "k_wgrad's thread layout");

__device__ __forceinline__ float sum_parts(const float* __restrict__ part, uint32_t parts, int p) {
  float g = 0.f;
#pragma unroll 8
  for (uint32_t c = 0; c < parts; ++c) g += part[(size_t)c * kNumParams + p];
  return g;
}
__global__ void k_wgrad_sum(const float* __restrict__ part, uint32_t parts, float* __restrict__ grad) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < kNumParams) grad[p] = sum_parts(part, parts, p);
}

__device__ __forceinline__ float to_eff(int p, float w) {
  return is_weight(p) ? __bfloat162float(__float2bfloat16_rn(w)) : w;
}

__global__ void k_adam(float* __restrict__ master, float* __restrict__ eff, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ part, uint32_t parts, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= kNumParams) return;
  const float g = sum_parts(part, parts, p);
  const float mm = b1 * m[p] + (1.f - b1) * g;
  const float vv = b2 * v[p] + (1.f - b2) * g * g;
  m[p] = mm;
  v[p] = vv;
  const float w = master[p] - lr * (mm / c1) / (sqrtf(vv / c2) + eps);
  master[p] = w;
  eff[p] = to_eff(p, w);
}

__global__ void k_refresh(const float* __restrict__ master, float* __restrict__ eff) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < kNumParams) eff[p] = to_eff(p, master[p]);
}

// Denormalised predictions (log2 time per variant) for rows of X.
__global__ void __launch_bounds__(kModelThreads) k_predict(const float* __restrict__ X, uint32_t rows,
                                                            const float* __restrict__ eff,
                                                            const float* __restrict__ norm, float* __restrict__ Y) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmemModel& s = *reinterpret_cast<SmemModel*>(smem_raw);
  load_model(s, eff, norm, nullptr);
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (uint64_t i = (uint64_t)warp * kRows; i < rows; i += (uint64_t)nw * kRows) {
    const uint32_t base = (uint32_t)i, n = (uint32_t)min((uint64_t)kRows, rows - i);
    float out[kRows][kOut];
    rows_pass<false, kRows>(s, nullptr, s.act[threadIdx.x >> 5], X, nullptr, [&](int r) { return base + r; }, (int)n, 0.f, out,
                     nullptr, 0);
    float v = 0.f;  // lane r * kOut + o: output o of row r
#pragma unroll
    for (int q = 0; q < kRows * kOut; ++q)
      if (lane == q) v = out[q / kOut][q % kOut];
    const int o = lane % kOut;
    if (lane < (int)n * kOut)
      Y[(size_t)base * kOut + lane] = v * s.norm[2 * kIn + kOut + o] + s.norm[2 * kIn + o];
  }
}

// variant_of[rb] = argmin of the predicted (normalised-back) time.
__global__ void __launch_bounds__(kModelThreads) k_dispatch(const float* __restrict__ feat, uint32_t nrb,
                                                             const float* __restrict__ eff,
                                                             const float* __restrict__ norm,
                                                             uint8_t* __restrict__ variant_of) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  SmemModel& s = *reinterpret_cast<SmemModel*>(smem_raw);
  load_model(s, eff, norm, nullptr);
  const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
  const int lane = threadIdx.x & 31;
  for (uint64_t i = (uint64_t)warp * kRows; i < nrb; i += (uint64_t)nw * kRows) {
    const uint32_t base = (uint32_t)i, n = (uint32_t)min((uint64_t)kRows, nrb - i);
    float out[kRows][kOut];
    rows_pass<false, kRows>(s, nullptr, s.act[threadIdx.x >> 5], feat, nullptr, [&](int r) { return base + r; }, (int)n, 0.f,
                     out, nullptr, 0);
    float y[kOut] = {};  // lane r: the outputs of row r
#pragma unroll
    for (int r = 0; r < kRows; ++r)
#pragma unroll
      for (int o = 0; o < kOut; ++o)
        if (lane == r) y[o] = out[r][o];
    if (lane < (int)n) {
      // Bit tiles only where the block fits one tile (span of 1..kTileMaxK
      // column blocks); elsewhere the tile kernel would sweep the block's rows
      // one at a time on a single warp.
      const float span = feat[(size_t)(base + lane) * kIn + kFeatSpan];
      const bool tile_ok = span > 0.f && span <= log2f(1.f + (float)kTileMaxK) + 1e-4f;
      int best = -1;
      float bt = 0.f;
#pragma unroll
      for (int o = 0; o < kOut; ++o) {
        if (o == TRIBIT_VARIANT_MMA && !tile_ok) continue;
        const float t = y[o] * s.norm[2 * kIn + kOut + o] + s.norm[2 * kIn + o];
        if (best < 0 || t < bt) bt = t, best = o;
      }
      variant_of[base + lane] = (uint8_t)best;
    }
  }
}

void set_smem_attrs() {
  once_per_device<1>([] {
    TB_CUDA(cudaFuncSetAttribute(k_fwd_bwd<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemTrain)));
    TB_CUDA(cudaFuncSetAttribute(k_fwd_bwd<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemTrain)));
    TB_CUDA(cudaFuncSetAttribute(k_fwd_bwd<kRows>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemTrain)));
    TB_CUDA(cudaFuncSetAttribute(k_predict, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemModel)));
    TB_CUDA(cudaFuncSetAttribute(k_dispatch, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmemModel)));
  });
}

// CTAs for `rows` rows, `per` a warp at a time.
unsigned grid_warps(uint64_t rows, int per = kRows) {
  const uint64_t g = ceil_div<uint64_t>(rows, kModelThreads / 32 * (uint64_t)per);
  return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(g, 148ull * 3));
}

struct TrainBuffers {
  float* X = nullptr;
  float* Y = nullptr;
  uint32_t* idx = nullptr;
  double* loss = nullptr;
  float* part = nullptr;  // wgrad_parts(B) x kNumParams: the gradient's partial sums
  Acts acts{};
};

TrainBuffers layout_train(Arena& ar, uint64_t rows, uint32_t B) {
  TrainBuffers t;
  t.X = ar.take<float>(rows * kIn + 1);
  t.Y = ar.take<float>(rows * kOut + 1);
  t.idx = ar.take<uint32_t>(rows + 1);
  t.loss = ar.take<double>(1);
  t.acts.xn = ar.take<float>((uint64_t)B * kIn);
  t.acts.h1 = ar.take<float>((uint64_t)B * kH1);
  t.acts.dz1 = ar.take<float>((uint64_t)B * kH1);
  t.acts.h2 = ar.take<float>((uint64_t)B * kH2);
  t.acts.dz2 = ar.take<float>((uint64_t)B * kH2);
  t.acts.dy = ar.take<float>((uint64_t)B * kOut);
  t.part = ar.take<float>((uint64_t)wgrad_parts(B) * kNumParams);
  return t;
}

TrainBuffers stage_training(tribit_context* c, const float* X, const float* Y, uint64_t rows, uint32_t B) {
  Arena& ar = c->train_arena;
  ar.begin(true);
  layout_train(ar, rows, B);
  ar.reserve(ar.used());
  ar.begin(false);
  TrainBuffers t = layout_train(ar, rows, B);
  TB_CUDA(cudaMemcpyAsync(t.X, X, rows * kIn * sizeof(float), cudaMemcpyHostToDevice, c->st));
  if (Y) TB_CUDA(cudaMemcpyAsync(t.Y, Y, rows * kOut * sizeof(float), cudaMemcpyHostToDevice, c->st));
  return t;
}

// Forward and backward of the batch's B rows, from row (of idx) r0 on, into t.acts.
void forward_backward(const TrainBuffers& t, const uint32_t* idx, uint32_t r0, uint32_t B, const DeviceModel& m,
                      cudaStream_t st) {
  const float inv = 1.f / (float)(kOut * B);
  auto launch = [&](auto kernel, int per) {
    kernel<<<grid_warps(B, per), kModelThreads, sizeof(SmemTrain), st>>>(t.X, t.Y, idx, r0, B, m.eff, m.norm, inv, t.acts,
                                                                         t.loss);
    TB_LAUNCH_CHECK();
  };
  if (B <= kSmallBatch)
    launch(k_fwd_bwd<1>, 1);
  else if (B <= 4 * kSmallBatch)
    launch(k_fwd_bwd<2>, 2);
  else
    launch(k_fwd_bwd<kRows>, kRows);
}

// The gradient of the batch of B rows in t.acts (B at most the batch t was laid out for: an epoch's last batch is
// often shorter).
// In t.part, as the sums of so many parts (the result), to be added in order.
uint32_t weight_gradients(const TrainBuffers& t, uint32_t B, cudaStream_t st) {
  const uint32_t ctas = wgrad_ctas(B);
  k_wgrad<<<ctas, 256, 0, st>>>(t.acts, B, t.part);
  TB_LAUNCH_CHECK();
  return ctas;
}

void require_model(tribit_context* c) {
  if (!c->model.loaded) throw StatusError(TRIBIT_ERR_NO_MODEL, "no dispatcher model: load or initialise one first");
}

}  // namespace

void model_alloc(DeviceModel& m, cudaStream_t st) {
  if (m.master) return;
  float* base = nullptr;
  const size_t n = 5 * (size_t)kNumParams + kNorm;
  TB_CUDA(cudaMalloc(&base, n * sizeof(float)));
  // On the caller's stream: the uploads that follow are ordered after it.
  TB_CUDA(cudaMemsetAsync(base, 0, n * sizeof(float), st));
  m.master = base;
  m.eff = base + kNumParams;
  m.m = base + 2 * kNumParams;
  m.v = base + 3 * kNumParams;
  m.grad = base + 4 * kNumParams;
  m.norm = base + 5 * kNumParams;
}

void model_free(DeviceModel& m) {
  if (m.master) cudaFree(m.master);
  m = DeviceModel{};
}

void model_refresh_eff(DeviceModel& m, cudaStream_t st) {
  k_refresh<<<(kNumParams + 255) / 256, 256, 0, st>>>(m.master, m.eff);
  TB_LAUNCH_CHECK();
}

void model_dispatch(const DeviceModel& m, const float* features, uint32_t nrb, uint8_t* variant_of, cudaStream_t st) {
  if (nrb == 0) return;
  set_smem_attrs();
  k_dispatch<<<grid_warps(nrb), kModelThreads, sizeof(SmemModel), st>>>(features, nrb, m.eff, m.norm, variant_of);
  TB_LAUNCH_CHECK();
}

void apply_dispatch(tribit_context* c, cudaStream_t st) {
  const int mode = c->opts.dispatch;
  c->sched.piece_width = c->piece_width;
  c->sched.tile_min_nnz = c->tile_min_nnz;
  c->sched.merge_ratio = c->merge_ratio;
  c->sched.tile_engine = c->tile_engine;
  // Only merge blocks use the hub lists; the plain rule picks merge blocks
  // from the neighbour-side features, so it reads the full set too.
  c->sched.hubs = mode == TRIBIT_DISPATCH_LEARNED || mode == TRIBIT_DISPATCH_MERGE || mode == TRIBIT_DISPATCH_PLAIN;
  drop_graph(c);
  if (mode == TRIBIT_DISPATCH_LEARNED) {
    require_model(c);
    compute_features(c->prep.view, c->sched, TRIBIT_DISPATCH_PLAIN, true, st);
    model_dispatch(c->model, c->sched.features, c->sched.num_row_blocks, c->sched.variant_of, st);
  } else {
    compute_features(c->prep.view, c->sched, mode, mode == TRIBIT_DISPATCH_PLAIN, st);
  }
  // Both rules choose merge for the hub pass; a schedule taken without hub
  // lists (the rows tier under a small device budget) sweeps those blocks as
  // bitmaps instead (RMAT-24: 122 ms all-bitmap against 130 ms merge without
  // the hub pass).
  if (!c->sched.eflag && (mode == TRIBIT_DISPATCH_LEARNED || mode == TRIBIT_DISPATCH_PLAIN))
    merge_blocks_to_bitmap(c->sched, st);
  build_pieces(c->prep.view, c->sched, st);
}

}  // namespace tb

using tb::DeviceGuard;
using tb::guarded;
using tb::StatusError;

extern "C" {

uint32_t tribit_model_num_params(void) { return (uint32_t)tb::kNumParams; }

tribit_status tribit_model_init(tribit_context* c, uint64_t seed, const float* norm) {
  if (!c || !norm) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    DeviceGuard dg(c->device);
    tb::model_alloc(c->model, c->st);
    std::vector<float> p(tb::kNumParams, 0.f);
    auto fill = [&](int off, int fan_in, int count) {
      const double lim = std::sqrt(6.0 / fan_in);
      for (int i = 0; i < count; ++i) p[off + i] = (float)((2.0 * tb_unit(tb_rand(seed, off + i)) - 1.0) * lim);
    };
    fill(tb::kW1, tb::kIn, tb::kIn * tb::kH1);
    fill(tb::kW2, tb::kH1, tb::kH1 * tb::kH2);
    fill(tb::kW3, tb::kH2, tb::kH2 * tb::kOut);
    TB_CUDA(cudaMemcpyAsync(c->model.master, p.data(), p.size() * sizeof(float), cudaMemcpyHostToDevice, c->st));
    TB_CUDA(cudaMemsetAsync(c->model.m, 0, 2 * tb::kNumParams * sizeof(float), c->st));
    TB_CUDA(cudaMemcpyAsync(c->model.norm, norm, tb::kNorm * sizeof(float), cudaMemcpyHostToDevice, c->st));
    tb::model_refresh_eff(c->model, c->st);
    TB_CUDA(cudaStreamSynchronize(c->st));
    c->model.steps = 0;
    c->model.loaded = true;
  });
}

tribit_status tribit_model_get_params(tribit_context* c, float* out, int effective) {
  if (!c || !out) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    tb::require_model(c);
    DeviceGuard dg(c->device);
    TB_CUDA(cudaMemcpyAsync(out, effective ? c->model.eff : c->model.master, tb::kNumParams * sizeof(float),
                            cudaMemcpyDeviceToHost, c->st));
    TB_CUDA(cudaStreamSynchronize(c->st));
  });
}

tribit_status tribit_model_set_params(tribit_context* c, const float* in) {
  if (!c || !in) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    tb::require_model(c);
    DeviceGuard dg(c->device);
    TB_CUDA(cudaMemcpyAsync(c->model.master, in, tb::kNumParams * sizeof(float), cudaMemcpyHostToDevice, c->st));
    tb::model_refresh_eff(c->model, c->st);
    TB_CUDA(cudaStreamSynchronize(c->st));
  });
}

tribit_status tribit_model_predict(tribit_context* c, const float* x, uint64_t rows, float* y) {
  if (!c || (!x && rows) || (!y && rows)) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    tb::require_model(c);
    DeviceGuard dg(c->device);
    if (rows == 0) return;
    tb::set_smem_attrs();
    tb::TrainBuffers t = tb::stage_training(c, x, nullptr, rows, 1);
    tb::k_predict<<<tb::grid_warps(rows), tb::kModelThreads, sizeof(tb::SmemModel), c->st>>>(
        t.X, (uint32_t)rows, c->model.eff, c->model.norm, t.Y);
    TB_LAUNCH_CHECK();
    TB_CUDA(cudaMemcpyAsync(y, t.Y, rows * tb::kOut * sizeof(float), cudaMemcpyDeviceToHost, c->st));
    TB_CUDA(cudaStreamSynchronize(c->st));
  });
}

tribit_status tribit_model_gradients(tribit_context* c, const float* x, const float* y, uint64_t rows, float* grad,
                                     float* loss_out) {
  if (!c || !x || !y || !grad || rows == 0 || rows > 0xffffffffull) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    tb::require_model(c);
    DeviceGuard dg(c->device);
    tb::set_smem_attrs();
    tb::TrainBuffers t = tb::stage_training(c, x, y, rows, (uint32_t)rows);
    TB_CUDA(cudaMemsetAsync(t.loss, 0, sizeof(double), c->st));
    tb::forward_backward(t, nullptr, 0, (uint32_t)rows, c->model, c->st);
    const uint32_t parts = tb::weight_gradients(t, (uint32_t)rows, c->st);
    const float* sum = t.part;
    if (parts > 1) {
      tb::k_wgrad_sum<<<(tb::kNumParams + 63) / 64, 64, 0, c->st>>>(t.part, parts, c->model.grad);
      TB_LAUNCH_CHECK();
      sum = c->model.grad;
    }
    double loss = 0.0;
    TB_CUDA(cudaMemcpyAsync(grad, sum, tb::kNumParams * sizeof(float), cudaMemcpyDeviceToHost, c->st));
    TB_CUDA(cudaMemcpyAsync(&loss, t.loss, sizeof(double), cudaMemcpyDeviceToHost, c->st));
    TB_CUDA(cudaStreamSynchronize(c->st));
    if (loss_out) *loss_out = (float)(loss / (double)(tb::kOut * rows));
  });
}

tribit_status tribit_model_train(tribit_context* c, const float* x, const float* y, uint64_t rows, uint32_t epochs,
                                 uint32_t batch, float lr, uint64_t seed, float* loss_out) {
  if (!c || !x || !y || rows == 0 || rows > 0xffffffffull || batch == 0 || epochs == 0) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    tb::require_model(c);
    DeviceGuard dg(c->device);
    tb::set_smem_attrs();
    const uint32_t B = (uint32_t)std::min<uint64_t>(batch, rows);
    tb::TrainBuffers t = tb::stage_training(c, x, y, rows, B);
    std::vector<uint32_t> order(rows);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    double last = 0.0;
    for (uint32_t ep = 0; ep < epochs; ++ep) {
      for (uint64_t i = 0; i < rows; ++i) order[i] = (uint32_t)i;
      for (uint64_t i = rows - 1; i > 0; --i) std::swap(order[i], order[tb_rand(seed + ep, i) % (i + 1)]);
      TB_CUDA(cudaMemcpyAsync(t.idx, order.data(), rows * sizeof(uint32_t), cudaMemcpyHostToDevice, c->st));
      TB_CUDA(cudaMemsetAsync(t.loss, 0, sizeof(double), c->st));
      for (uint64_t r0 = 0; r0 < rows; r0 += B) {
        const uint32_t nb = (uint32_t)std::min<uint64_t>(B, rows - r0);
        tb::forward_backward(t, t.idx, (uint32_t)r0, nb, c->model, c->st);
        const uint32_t parts = tb::weight_gradients(t, nb, c->st);
        const int step = ++c->model.steps;
        tb::k_adam<<<(tb::kNumParams + 63) / 64, 64, 0, c->st>>>(
            c->model.master, c->model.eff, c->model.m, c->model.v, t.part, parts, lr, b1, b2, eps,
            1.f - std::pow(b1, (float)step), 1.f - std::pow(b2, (float)step));
        TB_LAUNCH_CHECK();
      }
      TB_CUDA(cudaMemcpyAsync(&last, t.loss, sizeof(double), cudaMemcpyDeviceToHost, c->st));
      TB_CUDA(cudaStreamSynchronize(c->st));
    }
    if (loss_out) *loss_out = (float)(last / (double)(tb::kOut * rows));
  });
}

tribit_status tribit_block_features(tribit_context* c, float* out, uint64_t cap, uint64_t* num_row_blocks) {
  if (!c || !num_row_blocks) return TRIBIT_ERR_INVALID_ARGUMENT;
  if (!c->prepared) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    DeviceGuard dg(c->device);
    const uint64_t nrb = c->sched.num_row_blocks;
    *num_row_blocks = nrb;
    if (!out) return;
    if (cap < nrb * tb::kIn) throw StatusError(TRIBIT_ERR_INVALID_ARGUMENT, "feature buffer too small");
    tb::compute_features(c->prep.view, c->sched, TRIBIT_DISPATCH_PLAIN, true, c->st);
    TB_CUDA(cudaMemcpyAsync(out, c->sched.features, nrb * tb::kIn * sizeof(float), cudaMemcpyDeviceToHost, c->st));
    tb::apply_dispatch(c, c->st);
    TB_CUDA(cudaStreamSynchronize(c->st));
  });
}

tribit_status tribit_block_times(tribit_context* c, int variant, float* cycles_out, uint64_t cap,
                                 uint64_t* triangles_out, float* variant_ms) {
  if (!c || !c->prepared || variant < 0 || variant >= TRIBIT_NUM_VARIANTS) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    DeviceGuard dg(c->device);
    const uint64_t nrb = c->sched.num_row_blocks;
    if (cycles_out && cap < nrb) throw StatusError(TRIBIT_ERR_INVALID_ARGUMENT, "timing buffer too small");
    // Per-block times, and the in-list rows the hub pieces charge their
    // cycles to (a one-piece schedule keeps no rows).
    tb::Arena& ar = c->timing_arena;
    const bool hub_rows = variant == TRIBIT_VARIANT_MERGE && c->sched.inl;
    ar.begin(true);
    ar.take<unsigned long long>(nrb + 1);
    if (hub_rows) ar.take<uint32_t>(c->sched.inl_cap);
    ar.reserve(ar.used());
    ar.begin(false);
    unsigned long long* ns = ar.take<unsigned long long>(nrb + 1);
    c->sched.inrow = hub_rows ? ar.take<uint32_t>(c->sched.inl_cap) : nullptr;
    TB_CUDA(cudaMemsetAsync(ns, 0, (nrb + 1) * sizeof(unsigned long long), c->st));
    if (nrb) TB_CUDA(cudaMemsetAsync(c->sched.variant_of, variant, nrb, c->st));
    c->sched.hubs = variant == TRIBIT_VARIANT_MERGE;
    c->sched.hub_rows = hub_rows;  // the hub pieces charge their cycles to their rows' blocks
    tb::build_pieces(c->prep.view, c->sched, c->st);
    c->sched.hub_rows = false;
    tb::CountConfig cfg = tb::count_config(c);
    cfg.block_ns = ns;
    cfg.variant_start = c->ev[0];
    cfg.variant_stop = c->ev[1];
    tb::launch_count(c->prep.view, c->sched, c->prep.stats, c->per_graph, cfg, c->st);
    std::vector<unsigned long long> h(nrb + 1);
    TB_CUDA(cudaMemcpyAsync(h.data(), ns, nrb * sizeof(unsigned long long), cudaMemcpyDeviceToHost, c->st));
    TB_CUDA(cudaMemcpyAsync(c->h_stats, c->prep.stats, sizeof(tb::DeviceStats), cudaMemcpyDeviceToHost, c->st));
    TB_CUDA(cudaStreamSynchronize(c->st));
    if (triangles_out) *triangles_out = c->h_stats->triangles;
    if (variant_ms) TB_CUDA(cudaEventElapsedTime(variant_ms, c->ev[0], c->ev[1]));
    if (cycles_out)
      for (uint64_t i = 0; i < nrb; ++i) cycles_out[i] = (float)h[i];
    c->sched.inrow = nullptr;
    tb::apply_dispatch(c, c->st);
    TB_CUDA(cudaStreamSynchronize(c->st));
  });
}

tribit_status tribit_model_save(tribit_context* c, const char* path) {
  if (!c || !path) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    tb::require_model(c);
    DeviceGuard dg(c->device);
    std::vector<float> p(tb::kNumParams), nrm(tb::kNorm);
    TB_CUDA(cudaMemcpyAsync(p.data(), c->model.master, p.size() * sizeof(float), cudaMemcpyDeviceToHost, c->st));
    TB_CUDA(cudaMemcpyAsync(nrm.data(), c->model.norm, nrm.size() * sizeof(float), cudaMemcpyDeviceToHost, c->st));
    TB_CUDA(cudaStreamSynchronize(c->st));
    FILE* f = std::fopen(path, "wb");
    if (!f) throw StatusError(TRIBIT_ERR_IO, "cannot write model file");
    const uint32_t dims[4] = {tb::kIn, tb::kH1, tb::kH2, tb::kOut};
    bool ok = std::fwrite(tb::kMagic, 1, 8, f) == 8 && std::fwrite(dims, 4, 4, f) == 4 &&
              std::fwrite(nrm.data(), 4, nrm.size(), f) == nrm.size() && std::fwrite(p.data(), 4, p.size(), f) == p.size();
    ok = (std::fclose(f) == 0) && ok;
    if (!ok) throw StatusError(TRIBIT_ERR_IO, "cannot write model file");
  });
}

tribit_status tribit_model_load(tribit_context* c, const char* path) {
  if (!c || !path) return TRIBIT_ERR_INVALID_ARGUMENT;
  return guarded(c, [&] {
    FILE* f = std::fopen(path, "rb");
    if (!f) throw StatusError(TRIBIT_ERR_IO, "cannot open model file");
    char magic[8];
    uint32_t dims[4];
    std::vector<float> p(tb::kNumParams), nrm(tb::kNorm);
    bool ok = std::fread(magic, 1, 8, f) == 8 && std::memcmp(magic, tb::kMagic, 8) == 0 &&
              std::fread(dims, 4, 4, f) == 4 && dims[0] == (uint32_t)tb::kIn && dims[1] == (uint32_t)tb::kH1 &&
              dims[2] == (uint32_t)tb::kH2 && dims[3] == (uint32_t)tb::kOut &&
              std::fread(nrm.data(), 4, nrm.size(), f) == nrm.size() &&
              std::fread(p.data(), 4, p.size(), f) == p.size();
    std::fclose(f);
    if (!ok) throw StatusError(TRIBIT_ERR_FORMAT, "not a tribit dispatcher model file");
    DeviceGuard dg(c->device);
    tb::model_alloc(c->model, c->st);
    TB_CUDA(cudaMemcpyAsync(c->model.master, p.data(), p.size() * sizeof(float), cudaMemcpyHostToDevice, c->st));
    TB_CUDA(cudaMemcpyAsync(c->model.norm, nrm.data(), nrm.size() * sizeof(float), cudaMemcpyHostToDevice, c->st));
    TB_CUDA(cudaMemsetAsync(c->model.m, 0, 2 * tb::kNumParams * sizeof(float), c->st));
    tb::model_refresh_eff(c->model, c->st);
    TB_CUDA(cudaStreamSynchronize(c->st));
    c->model.steps = 0;
    c->model.loaded = true;
  });
}

}  // extern "C"
