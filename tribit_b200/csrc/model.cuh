// Learned dispatcher: a 16 -> 64 -> 64 -> 3 MLP over row-block features that
// predicts, for each counting variant, log2 of the time the variant spends on
// the row block; dispatch picks the smallest. It changes scheduling only:
// every variant counts exactly, so the count never depends on the model.
//
// Weights are used in BF16 (rounded from FP32 master copies), activations and
// accumulation are FP32. Forward, backward and Adam are hand-written kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace tb {

constexpr int kIn = 16, kH1 = 64, kH2 = 64, kOut = 3;
constexpr int kW1 = 0;                      // [kIn][kH1]
constexpr int kB1 = kW1 + kIn * kH1;        // [kH1]
constexpr int kW2 = kB1 + kH1;              // [kH1][kH2]
constexpr int kB2 = kW2 + kH1 * kH2;        // [kH2]
constexpr int kW3 = kB2 + kH2;              // [kH2][kOut]
constexpr int kB3 = kW3 + kH2 * kOut;       // [kOut]
constexpr int kNumParams = kB3 + kOut;      // 5443

// The weight gradient's split: a CTA sums the rows of whole units, so a batch a
// little above kGradCtas units takes about half the CTAs of one just below (9,472
// rows 296 CTAs, 9,473 rows 149). The partial sums of a run of batches of up to
// B rows are therefore bounded by wgrad_parts(B), not by wgrad_ctas(B). Small
// batches are split finer, since a single tile keeps one CTA busy while the chip
// waits (a training step of 32 rows 22.9 us in one CTA, 18.9 in four).
constexpr uint32_t kSmallBatch = 512;
constexpr uint32_t kGradTile = 32;   // rows staged at a time
constexpr uint32_t kGradCtas = 296;  // two a multiprocessor
__host__ __device__ inline uint32_t wgrad_unit(uint32_t B) { return B <= kSmallBatch ? 8u : kGradTile; }
__host__ __device__ inline uint32_t wgrad_rows(uint32_t B) {  // rows a CTA sums: whole units
  const uint32_t per = (uint32_t)(((uint64_t)B + kGradCtas - 1) / kGradCtas), unit = wgrad_unit(B);
  return (per + unit - 1) / unit * unit;
}
__host__ __device__ inline uint32_t wgrad_ctas(uint32_t B) {
  const uint32_t R = wgrad_rows(B);
  return (uint32_t)(((uint64_t)B + R - 1) / R);
}
inline uint32_t wgrad_parts(uint32_t B) {  // at least wgrad_ctas(b) for every b <= B
  const uint32_t unit = wgrad_unit(B), units = (uint32_t)(((uint64_t)B + unit - 1) / unit);
  const uint32_t small = B <= kSmallBatch ? 0u : kSmallBatch / wgrad_unit(kSmallBatch);
  return units < small ? small : units < kGradCtas ? units : kGradCtas;
}

// Device-resident model. `eff` holds the parameters as the kernels use them:
// weights rounded to BF16 (stored as float), biases in FP32.
struct DeviceModel {
  float* master = nullptr;  // kNumParams, FP32
  float* eff = nullptr;     // kNumParams
  float* m = nullptr;       // Adam first moment
  float* v = nullptr;       // Adam second moment
  float* grad = nullptr;    // kNumParams
  float* norm = nullptr;    // in_mean[16], in_std[16], out_mean[3], out_std[3]
  int steps = 0;
  bool loaded = false;
};

void model_alloc(DeviceModel& m, cudaStream_t st);
void model_free(DeviceModel& m);
void model_refresh_eff(DeviceModel& m, cudaStream_t st);

// variant_of[rb] = argmin over variants of the predicted time, for row blocks
// with work; features are nrb x kIn.
void model_dispatch(const DeviceModel& m, const float* features, uint32_t nrb, uint8_t* variant_of, cudaStream_t st);

}  // namespace tb
