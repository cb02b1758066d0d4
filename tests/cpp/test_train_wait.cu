// The training kernel's waits run out: with no polls allowed the first wait (for the
// weights' bulk copies) expires at once. The kernel has to set the status, issue no
// products, wait for its copies and return; the next launch on the same device, with the
// ordinary limit, gives the gradient it gave before.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <vector>

#include "mlp_tc.cuh"

using namespace bbkde;
using namespace bbkde::mlp;

#define CHECK(x)                                                               \
  do {                                                                         \
    const cudaError_t e_ = (x);                                                \
    if (e_ != cudaSuccess) {                                                   \
      std::printf("FAILED %s: %s\n", #x, cudaGetErrorString(e_));              \
      return 1;                                                                \
    }                                                                          \
  } while (0)

int main() {
  int devices = 0;
  if (cudaGetDeviceCount(&devices) != cudaSuccess || devices == 0) {
    std::printf("no CUDA device\n");
    return 2;
  }
  constexpr int kBatch = 300, kBlocks = 3;
  std::vector<float> params(kParams), xy(2 * kBatch), target(kBatch);
  for (int i = 0; i < kParams; ++i) params[i] = 0.05f * std::sin(0.7f * (float)i);
  for (int i = 0; i < 2 * kBatch; ++i) xy[i] = std::cos(0.3f * (float)i);
  for (int i = 0; i < kBatch; ++i) target[i] = xy[2 * i] * xy[2 * i + 1];
  std::vector<__nv_bfloat16> w(2 * kH * kH);   // both matrices, canonical layout
  for (int m = 0; m < 2; ++m)
    for (int r = 0; r < kH; ++r)
      for (int k = 0; k < kH; ++k)
        w[m * kH * kH + ((k >> 3) * 2048 + (r >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2) / 2] =
            __float2bfloat16(params[(m ? kOffW3 : kOffW2) + r * kH + k]);
  float *dp = nullptr, *dxy = nullptr, *dt = nullptr, *grad = nullptr, *loss = nullptr;
  __nv_bfloat16 *dw = nullptr;
  int *status = nullptr;
  const size_t gbytes = (size_t)kBlocks * kPartStride * sizeof(float);
  CHECK(cudaMalloc(&dp, kParams * sizeof(float)));
  CHECK(cudaMalloc(&dxy, xy.size() * sizeof(float)));
  CHECK(cudaMalloc(&dt, target.size() * sizeof(float)));
  CHECK(cudaMalloc(&grad, gbytes));
  CHECK(cudaMalloc(&loss, kBlocks * sizeof(float)));
  CHECK(cudaMalloc(&dw, w.size() * sizeof(__nv_bfloat16)));
  CHECK(cudaMalloc(&status, sizeof(int)));
  CHECK(cudaMemcpy(dp, params.data(), kParams * sizeof(float), cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(dxy, xy.data(), xy.size() * sizeof(float), cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(dt, target.data(), target.size() * sizeof(float), cudaMemcpyHostToDevice));
  CHECK(cudaMemcpy(dw, w.data(), w.size() * sizeof(__nv_bfloat16), cudaMemcpyHostToDevice));
  CHECK(cudaFuncSetAttribute(k_mlp_train_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)TcTrainSmem::kBytes));
  TcTrainArgs a = {};
  a.t.params = dp;
  a.t.w2c = dw;
  a.t.w3c = dw + kH * kH;
  a.t.norm = Norm{0.f, 0.f, 1.f, 1.f, 0.f, 1.f};
  a.t.xy = reinterpret_cast<const float2 *>(dxy);
  a.t.target = dt;
  a.t.batch = kBatch;
  a.t.grad_part = grad;
  a.t.loss_part = loss;
  a.status = status;
  std::vector<float> g[3];
  const long long limits[3] = {kTcWaitLimit, 0, kTcWaitLimit};
  int st[3];
  for (int k = 0; k < 3; ++k) {
    CHECK(cudaMemset(status, 0, sizeof(int)));
    CHECK(cudaMemset(grad, 0x41, gbytes));
    a.limit = limits[k];
    k_mlp_train_tc<<<kBlocks, kTcTrainThreads, TcTrainSmem::kBytes>>>(a);
    CHECK(cudaGetLastError());
    CHECK(cudaDeviceSynchronize());
    g[k].resize(kBlocks * (size_t)kPartStride);
    CHECK(cudaMemcpy(g[k].data(), grad, gbytes, cudaMemcpyDeviceToHost));
    CHECK(cudaMemcpy(&st[k], status, sizeof(int), cudaMemcpyDeviceToHost));
  }
  if (st[0] != 0 || st[1] != 1 || st[2] != 0) {
    std::printf("FAILED status %d %d %d\n", st[0], st[1], st[2]);
    return 1;
  }
  if (std::memcmp(g[0].data(), g[2].data(), gbytes) != 0) {
    std::printf("FAILED gradient after the expired launch\n");
    return 1;
  }
  float untouched;
  std::memset(&untouched, 0x41, sizeof(untouched));
  for (int b = 0; b < kBlocks; ++b)
    for (int i = kOffW2; i < kOffB2; ++i)
      if (g[1][(size_t)b * kPartStride + i] != untouched ||
          g[0][(size_t)b * kPartStride + i] == untouched) {
        std::printf("FAILED dW2[%d] of block %d\n", i - kOffW2, b);
        return 1;
      }
  std::printf("ALL PASSED\n");
  return 0;
}
