// activation.cuh — the activations of the elementwise kernels and of the products that end in one, and their derivatives.
#pragma once

namespace sxb {
namespace ew {

enum Act : int { kIdentity = 0, kRelu = 1, kGelu = 2, kSilu = 3 };

__device__ __forceinline__ float act_fwd(float x, int act) {
  switch (act) {
    case kRelu: return fmaxf(x, 0.f);
    case kGelu: {
      const float k0 = 0.7978845608028654f, k1 = 0.044715f;
      return 0.5f * x * (1.f + tanhf(k0 * (x + k1 * x * x * x)));
    }
    case kSilu: return x / (1.f + __expf(-x));
    default: return x;
  }
}
__device__ __forceinline__ float act_bwd(float x, int act) {
  switch (act) {
    case kRelu: return x > 0.f ? 1.f : 0.f;
    case kGelu: {
      const float k0 = 0.7978845608028654f, k1 = 0.044715f;
      const float u = k0 * (x + k1 * x * x * x);
      const float t = tanhf(u);
      return 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k0 * (1.f + 3.f * k1 * x * x);
    }
    case kSilu: {
      const float s = 1.f / (1.f + __expf(-x));
      return s * (1.f + x * (1.f - s));
    }
    default: return 1.f;
  }
}

}  // namespace ew
}  // namespace sxb
