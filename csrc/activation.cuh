// activation.cuh — the activations of the elementwise kernels and of the products that end in one, and their derivatives.
#pragma once

namespace sxb {
namespace ew {

enum Act : int { kIdentity = 0, kRelu = 1, kGelu = 2, kSilu = 3 };

// FAST, for 16-bit results: SiLU by the hardware's reciprocal (two units of the last place in 32 bits) instead of a division with its
// correction steps, which bound the activation kernels by their instructions (4096 x 14336, with the walk without divisions: forward 76.8 -> 66.5 us,
// 54 at copy speed, backward 118 -> 99, 90).  The error against 64 bits is that of the 16-bit result (1.651e-3, 1.653e-3) either way.
template <bool FAST>
__device__ __forceinline__ float act_fwd(float x, int act) {
  switch (act) {
    case kRelu: return fmaxf(x, 0.f);
    case kGelu: {
      const float k0 = 0.7978845608028654f, k1 = 0.044715f;
      return 0.5f * x * (1.f + tanhf(k0 * (x + k1 * x * x * x)));
    }
    case kSilu: return FAST ? __fdividef(x, 1.f + __expf(-x)) : x / (1.f + __expf(-x));
    default: return x;
  }
}
// Value f and derivative b, what they share computed once.
template <bool FAST>
__device__ __forceinline__ void act_both(float x, int act, float& f, float& b) {
  switch (act) {
    case kRelu: f = fmaxf(x, 0.f), b = x > 0.f ? 1.f : 0.f; return;
    case kGelu: {
      const float k0 = 0.7978845608028654f, k1 = 0.044715f;
      const float t = tanhf(k0 * (x + k1 * x * x * x));
      f = 0.5f * x * (1.f + t);
      b = 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * k0 * (1.f + 3.f * k1 * x * x);
      return;
    }
    case kSilu: {
      const float y = 1.f + __expf(-x), s = FAST ? __fdividef(1.f, y) : 1.f / y;
      f = FAST ? x * s : x / y;
      b = s * (1.f + x * (1.f - s));
      return;
    }
    default: f = x, b = 1.f; return;
  }
}

}  // namespace ew
}  // namespace sxb
