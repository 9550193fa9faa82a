// elementwise.cu — RoPE, gated/bias activations, fused softmax-cross-entropy, embedding,
// dtype casts and scaled accumulation (sm_100a; all HBM-bound, 16-byte vector access).
//
// Reference behaviour:
//   gated activation  deepspeed/inference/v2/kernels/core_ops/gated_activations/gated_activation_kernels_cuda.cu:45
//   bias activation   deepspeed/inference/v2/kernels/core_ops/bias_activations/bias_activation_cuda.cu:52-92
//   rotary            deepspeed/sequence/layer.py:84-103, deepspeed/sequence/fpdt_layer.py:26-37
//   vocab-parallel CE deepspeed/sequence/cross_entropy.py:13-58
//   ragged embed      deepspeed/inference/v2/kernels/ragged_ops/embed/embed_cuda.cu:19-90
#include <cfloat>
#include "activation.cuh"
#include "sxb_common.cuh"

namespace sxb {
namespace ew {

constexpr int kThreads = 256;

template <typename T>
__device__ __forceinline__ void ld8(const T* p, float (&o)[8]) {
  uint4 t = *reinterpret_cast<const uint4*>(p);
  const T* h = reinterpret_cast<const T*>(&t);
#pragma unroll
  for (int i = 0; i < 8; ++i) o[i] = to_f32<T>(h[i]);
}
template <typename T>
__device__ __forceinline__ void st8(T* p, const float (&o)[8]) {
  uint4 t;
  T* h = reinterpret_cast<T*>(&t);
#pragma unroll
  for (int i = 0; i < 8; ++i) h[i] = from_f32<T>(o[i]);
  *reinterpret_cast<uint4*>(p) = t;
}

// The vectors that a thread takes of rows of `per` vectors, grid after grid: row and column go on by additions.  (For the rotary copy.  The
// activation kernels keep a division per vector: with it 4096 x 14336 took 76.8 us forward, with this walk 79.9.)
struct RowWalk {
  long long at, row, step, drow;
  int col, dcol, per;
  __device__ __forceinline__ explicit RowWalk(int per_) : per(per_) {
    at = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    step = (long long)gridDim.x * blockDim.x;
    row = at / per, col = (int)(at - row * per);
    drow = step / per, dcol = (int)(step - drow * per);
  }
  __device__ __forceinline__ void next() {
    at += step, row += drow, col += dcol;
    if (col >= per) col -= per, ++row;
  }
};

// ----------------------------------------------------------------------- RoPE
// x: [T, row_stride] with n_heads rotated heads of size D at the start of each row, `rest` columns behind them.
// cos/sin: [max_pos, D/2] fp32.  sign = +1 forward, -1 backward (inverse rotation).
// COPY: to y instead of in place, the other columns as they are (a gradient is not rotated in autograd's buffer: 13 us of copying
// for 4096 rows of 6144, and a launch).
template <typename T, bool COPY>
__global__ void __launch_bounds__(kThreads)
rope_kernel(T* x, T* y, const long long* __restrict__ pos, const float* __restrict__ cs,
            const float* __restrict__ sn, long long Ttok, int n_heads, int D, long long row_stride, int rest,
            float sign) {
  const int half = D >> 1;
  const int vec_per_head = half >> 3;  // 8 elements per thread-iteration
  auto turn = [&](long long t, int h, int v) {
    const long long p = pos ? pos[t] : t;
    const long long at = t * row_stride + (long long)h * D + v * 8;
    const T* base = x + at;
    T* to = (COPY ? y : x) + at;
    float a[8], b[8], c[8], s[8];
    ld8<T>(base, a);
    ld8<T>(base + half, b);
    const float4* cp = reinterpret_cast<const float4*>(cs + p * half + v * 8);
    const float4* sp = reinterpret_cast<const float4*>(sn + p * half + v * 8);
    float4 c0 = cp[0], c1 = cp[1], s0 = sp[0], s1 = sp[1];
    c[0] = c0.x; c[1] = c0.y; c[2] = c0.z; c[3] = c0.w; c[4] = c1.x; c[5] = c1.y; c[6] = c1.z; c[7] = c1.w;
    s[0] = s0.x; s[1] = s0.y; s[2] = s0.z; s[3] = s0.w; s[4] = s1.x; s[5] = s1.y; s[6] = s1.z; s[7] = s1.w;
    float oa[8], ob[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const float sk = sign * s[k];
      oa[k] = a[k] * c[k] - b[k] * sk;
      ob[k] = b[k] * c[k] + a[k] * sk;
    }
    st8<T>(to, oa);
    st8<T>(to + half, ob);
  };
  if constexpr (COPY) {
    const int turning = n_heads * vec_per_head, per = turning + rest / 16;
    for (RowWalk i(per); i.at < Ttok * per; i.next()) {
      if (i.col < turning) {
        turn(i.row, i.col / vec_per_head, i.col % vec_per_head);
      } else {
        const long long at = i.row * row_stride + (long long)n_heads * D + (i.col - turning) * 16;
        const uint4 a = *reinterpret_cast<const uint4*>(x + at), b = *reinterpret_cast<const uint4*>(x + at + 8);
        *reinterpret_cast<uint4*>(y + at) = a;
        *reinterpret_cast<uint4*>(y + at + 8) = b;
      }
    }
  } else {
    const long long total = Ttok * n_heads * vec_per_head;
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
      const long long th = i / vec_per_head;
      turn(th / n_heads, (int)(th % n_heads), (int)(i % vec_per_head));
    }
  }
}

// out[T,F] = act(in[:, :F] (+bias)) * (in[:, F:] (+bias))       (concatenated gate|up layout)
template <typename T>
__global__ void __launch_bounds__(kThreads)
gated_fwd_kernel(const T* in, const T* __restrict__ bias, T* __restrict__ out,
                 long long rows, int F, int act) {
  chain_next();
  chain_wait();
  const int vpr = F >> 3;
  const long long total = rows * vpr;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vpr;
    const int c = (int)(i % vpr) * 8;
    float g[8], u[8], o[8];
    ld8<T>(in + r * 2 * F + c, g);
    ld8<T>(in + r * 2 * F + F + c, u);
    if (bias) {
      float bg[8], bu[8];
      ld8<T>(bias + c, bg);
      ld8<T>(bias + F + c, bu);
#pragma unroll
      for (int k = 0; k < 8; ++k) { g[k] += bg[k]; u[k] += bu[k]; }
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = act_fwd(g[k], act) * u[k];
    st8<T>(out + r * F + c, o);
  }
}
// The same for the routed rows of an expert layer only: group g of `in` / `out` starts at row offsets[g] and holds counts[g]
// routed rows, the rest of its (256-row aligned) room is padding that nothing reads.  blockIdx.x counts the routed rows of
// all groups; rows behind them are left as they are.
template <typename T>
__global__ void __launch_bounds__(kThreads)
gated_groups_kernel(const T* __restrict__ in, T* __restrict__ out, const int* __restrict__ offsets,
                    const int* __restrict__ counts, int groups, int F, int act) {
  __shared__ int row_s;
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x, i = blockIdx.x;
    int base = 0, row = -1;
    for (int g0 = 0; g0 < groups; g0 += 32) {
      const int own = g0 + lane < groups ? counts[g0 + lane] : 0;
      int incl = own;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, base + incl > i);
      if (hit) {
        const int src = __ffs(hit) - 1;
        row = offsets[g0 + src] + i - base - (__shfl_sync(0xffffffffu, incl, src) - __shfl_sync(0xffffffffu, own, src));
        break;
      }
      base += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) row_s = row;
  }
  __syncthreads();
  const long long r = row_s;
  if (r < 0) return;
  for (int c = (blockIdx.y * kThreads + threadIdx.x) * 8; c < F; c += gridDim.y * kThreads * 8) {
    float g[8], u[8], o[8];
    ld8<T>(in + r * 2 * F + c, g);
    ld8<T>(in + r * 2 * F + F + c, u);
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = act_fwd(g[k], act) * u[k];
    st8<T>(out + r * F + c, o);
  }
}
template <typename T>
__global__ void __launch_bounds__(kThreads)
gated_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ in, T* __restrict__ din,
                 long long rows, int F, int act) {
  const int vpr = F >> 3;
  const long long total = rows * vpr;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vpr;
    const int c = (int)(i % vpr) * 8;
    float g[8], u[8], d[8], dg[8], du[8];
    ld8<T>(in + r * 2 * F + c, g);
    ld8<T>(in + r * 2 * F + F + c, u);
    ld8<T>(dy + r * F + c, d);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      dg[k] = d[k] * u[k] * act_bwd(g[k], act);
      du[k] = d[k] * act_fwd(g[k], act);
    }
    st8<T>(din + r * 2 * F + c, dg);
    st8<T>(din + r * 2 * F + F + c, du);
  }
}
// y = act(x + bias)  (in place allowed)
template <typename T>
__global__ void __launch_bounds__(kThreads)
bias_act_kernel(const T* __restrict__ x, const T* __restrict__ bias, T* __restrict__ y,
                long long rows, int C, int act) {
  const int vpr = C >> 3;
  const long long total = rows * vpr;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vpr;
    const int c = (int)(i % vpr) * 8;
    float v[8];
    ld8<T>(x + r * C + c, v);
    if (bias) {
      float b[8];
      ld8<T>(bias + c, b);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += b[k];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = act_fwd(v[k], act);
    st8<T>(y + r * C + c, v);
  }
}
// dx = dy * act'(x + bias)
template <typename T>
__global__ void __launch_bounds__(kThreads)
bias_act_bwd_kernel(const T* __restrict__ dy, const T* __restrict__ x, const T* __restrict__ bias,
                    T* __restrict__ dx, long long rows, int C, int act) {
  const int vpr = C >> 3;
  const long long total = rows * vpr;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long r = i / vpr;
    const int c = (int)(i % vpr) * 8;
    float v[8], d[8];
    ld8<T>(x + r * C + c, v);
    ld8<T>(dy + r * C + c, d);
    if (bias) {
      float b[8];
      ld8<T>(bias + c, b);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] += b[k];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) d[k] *= act_bwd(v[k], act);
    st8<T>(dx + r * C + c, d);
  }
}

// ------------------------------------------------------------- cross entropy
// One CTA per token row.  loss[row] = lse - logit[label]; logits are overwritten by
// dlogits = (softmax - onehot) * (*grad_scale) so the [T,V] tensor is touched twice
// and never duplicated.  Rows with label == ignore_index get loss 0 / grad 0.
// What bounds it: bytes under way.  A row's second reading comes from L2 (two CTAs per SM of 256 KB rows are 76 MB), so four
// words of a thread are asked for before the first is used (bf16, us with one word | four: 2048 rows of 128256 254 | 242,
// 1024 of 50304 61 | 55, 4096 of 32000 127 | 115, 2048 of 32000 72 | 64; one reading and one writing of the first
// take 158).
template <typename T, int THREADS, int CTAS, int U>
__global__ void __launch_bounds__(THREADS, CTAS)
xent_kernel(T* __restrict__ logits, const long long* __restrict__ labels,
            float* __restrict__ loss, float* __restrict__ lse_out, int V, long long ld,
            long long ignore_index, const float* __restrict__ grad_scale, int write_grad) {
  __shared__ float red[32];
  const long long row = blockIdx.x;
  T* lr = logits + row * ld;
  const long long label = labels[row];
  const int nvec = V >> 3;
  // a finite lowest value: -inf minus it is -inf, so words of masked columns alone leave a sum of 0, not NaN
  float mx = -FLT_MAX, sum = 0.f;
  for (int v0 = threadIdx.x; v0 < nvec; v0 += U * THREADS) {
    uint4 raw[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int vi = v0 + j * THREADS;
      if (vi < nvec) raw[j] = *reinterpret_cast<const uint4*>(lr + (long long)vi * 8);
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      if (v0 + j * THREADS >= nvec) break;
      const T* h = reinterpret_cast<const T*>(&raw[j]);
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) v[k] = to_f32<T>(h[k]);
      float lm = v[0];
#pragma unroll
      for (int k = 1; k < 8; ++k) lm = fmaxf(lm, v[k]);
      const float nm = fmaxf(mx, lm);
      float acc = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) acc += __expf(v[k] - nm);
      sum = sum * __expf(mx - nm) + acc;
      mx = nm;
    }
  }
  for (int j = (nvec << 3) + threadIdx.x; j < V; j += blockDim.x) {
    const float v = to_f32<T>(lr[j]);
    const float nm = fmaxf(mx, v);
    sum = sum * __expf(mx - nm) + __expf(v - nm);
    mx = nm;
  }
  const float gmx = block_max(mx, red);
  sum = block_sum(sum * __expf(mx - gmx), red);
  const float lse = gmx + __logf(sum);
  const bool ignored = (label == ignore_index);
  if (threadIdx.x == 0) {
    loss[row] = ignored ? 0.f : (lse - to_f32<T>(lr[label]));
    if (lse_out) lse_out[row] = lse;
  }
  if (!write_grad) return;
  __syncthreads();
  const float gs = ignored ? 0.f : (grad_scale ? *grad_scale : 1.f);
  for (int v0 = threadIdx.x; v0 < nvec; v0 += U * THREADS) {
    uint4 raw[U];
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int vi = v0 + j * THREADS;
      if (vi < nvec) raw[j] = *reinterpret_cast<const uint4*>(lr + (long long)vi * 8);
    }
#pragma unroll
    for (int j = 0; j < U; ++j) {
      const int vi = v0 + j * THREADS;
      if (vi >= nvec) break;
      const T* h = reinterpret_cast<const T*>(&raw[j]);
      float v[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        float pr = __expf(to_f32<T>(h[k]) - lse);
        if ((long long)(vi * 8 + k) == label) pr -= 1.f;
        v[k] = pr * gs;
      }
      st8<T>(lr + (long long)vi * 8, v);
    }
  }
  for (int j = (nvec << 3) + threadIdx.x; j < V; j += blockDim.x) {
    float pr = __expf(to_f32<T>(lr[j]) - lse);
    if (j == label) pr -= 1.f;
    lr[j] = from_f32<T>(pr * gs);
  }
}

// ------------------------------------------------------------------ embedding
template <typename T>
__global__ void __launch_bounds__(kThreads)
embed_fwd_kernel(const long long* __restrict__ ids, const T* __restrict__ table,
                 T* __restrict__ out, long long ntok, int H) {
  const int vpr = H >> 3;
  const long long total = ntok * vpr;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / vpr;
    const int c = (int)(i % vpr) * 8;
    *reinterpret_cast<uint4*>(out + t * H + c) =
        *reinterpret_cast<const uint4*>(table + ids[t] * H + c);
  }
}
// dtable[ids[t]] += dout[t]   (bf16x2 / half2 / float atomics)
template <typename T>
__global__ void __launch_bounds__(kThreads)
embed_bwd_kernel(const long long* __restrict__ ids, const T* __restrict__ dout,
                 T* __restrict__ dtable, long long ntok, int H) {
  const int ppr = H >> 1;
  const long long total = ntok * ppr;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / ppr;
    const int c = (int)(i % ppr) * 2;
    if constexpr (sizeof(T) == 4) {
      atomicAdd(reinterpret_cast<float*>(dtable) + ids[t] * H + c, to_f32<T>(dout[t * H + c]));
      atomicAdd(reinterpret_cast<float*>(dtable) + ids[t] * H + c + 1, to_f32<T>(dout[t * H + c + 1]));
    } else if constexpr (std::is_same<T, __nv_bfloat16>::value) {
      atomicAdd(reinterpret_cast<__nv_bfloat162*>(dtable + ids[t] * H + c),
                *reinterpret_cast<const __nv_bfloat162*>(dout + t * H + c));
    } else {
      atomicAdd(reinterpret_cast<__half2*>(dtable + ids[t] * H + c),
                *reinterpret_cast<const __half2*>(dout + t * H + c));
    }
  }
}

// ------------------------------------------------------------ cast / axpy
// dst = (accumulate ? dst : 0) + scale * src with independent dtypes.
template <typename TS, typename TD>
__global__ void __launch_bounds__(kThreads)
scale_cast_kernel(const TS* __restrict__ src, TD* __restrict__ dst, long long n, float scale,
                  int accumulate) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float v = scale * to_f32<TS>(src[i]);
    if (accumulate) v += to_f32<TD>(dst[i]);
    dst[i] = from_f32<TD>(v);
  }
}

// x *= *scale (rounded to the type of x first), nothing when it is one: the gradient of a loss that nobody has scaled costs a
// launch instead of a pass over the logits' gradient.
template <typename T>
__global__ void __launch_bounds__(kThreads)
scale_by_kernel(T* __restrict__ x, long long n8, const float* __restrict__ scale) {
  const float f = to_f32<T>(from_f32<T>(*scale));
  if (f == 1.f) return;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n8; i += (long long)gridDim.x * blockDim.x) {
    float v[8];
    ld8<T>(x + i * 8, v);
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] *= f;
    st8<T>(x + i * 8, v);
  }
}

static inline int grid_for(long long work) {
  long long b = (work + kThreads - 1) / kThreads;
  if (b < 1) b = 1;
  if (b > 148 * 16) b = 148 * 16;
  return (int)b;
}

}  // namespace ew
}  // namespace sxb

#include <type_traits>
using namespace sxb;
using namespace sxb::ew;

#define DISPATCH_16(dtype, CALL)                          \
  do {                                                    \
    if (dtype == kBF16) { using T = __nv_bfloat16; CALL; } \
    else if (dtype == kF16) { using T = __half; CALL; }   \
    else return SXB_ERR_BAD_ARG;                          \
  } while (0)

SXB_API int sxb_rope(void* x, const void* positions, const void* cos_tab, const void* sin_tab,
                     long long tokens, int n_heads, int head_dim, long long row_stride,
                     int inverse, int dtype, void* stream) {
  if (tokens <= 0 || n_heads <= 0) return SXB_OK;
  if (head_dim % 16) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  const long long work = tokens * n_heads * (head_dim / 16);
  DISPATCH_16(dtype, (rope_kernel<T, false><<<grid_for(work), kThreads, 0, s>>>(
                         (T*)x, nullptr, (const long long*)positions, (const float*)cos_tab,
                         (const float*)sin_tab, tokens, n_heads, head_dim, row_stride, 0,
                         inverse ? -1.f : 1.f)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}

// y = x with its first n_heads heads rotated, rows of `cols` columns one behind the other; -2 where the columns behind the heads are no
// multiple of 16.
SXB_API int sxb_rope_copy(const void* x, void* y, const void* positions, const void* cos_tab, const void* sin_tab, long long tokens,
                          int n_heads, int head_dim, int cols, int inverse, int dtype, void* stream) {
  if (tokens <= 0) return SXB_OK;
  const long long rest = cols - (long long)n_heads * head_dim;
  if (head_dim % 16 || cols % 8 || rest < 0 || rest % 16 ||
      ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15))
    return SXB_ERR_UNSUPPORTED;
  const long long work = tokens * (cols / 16);
  cudaStream_t s = (cudaStream_t)stream;
  DISPATCH_16(dtype, (rope_kernel<T, true><<<grid_for(work), kThreads, 0, s>>>(
                         (T*)x, (T*)y, (const long long*)positions, (const float*)cos_tab, (const float*)sin_tab, tokens, n_heads,
                         head_dim, cols, (int)rest, inverse ? -1.f : 1.f)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}

SXB_API int sxb_gated_act_fwd(const void* in, const void* bias, void* out, long long rows, int F,
                              int act, int dtype, void* stream) {
  if (rows <= 0) return SXB_OK;
  if (F % 8) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  int rc = SXB_OK;
  DISPATCH_16(dtype, rc = launch_chained(gated_fwd_kernel<T>, dim3(grid_for(rows * (F / 8))), kThreads, s, (const T*)in,
                                         (const T*)bias, (T*)out, rows, F, act));
  return rc;
}
// act(gate) * up for the routed rows of grouped expert rows: in [capacity, 2F], out [capacity, F]; offsets / counts int32
// [groups] (first row and routed rows of every group); n_rows = sum of the counts.  Other rows of out are not written.
SXB_API int sxb_gated_act_groups(const void* in, void* out, const void* offsets, const void* counts, int groups, int n_rows,
                                 int F, int act, int dtype, void* stream) {
  if (n_rows <= 0 || groups <= 0) return SXB_OK;
  if (F % 8) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  const int parts = (F / 8 + kThreads - 1) / kThreads;        // a word per thread while the rows are few
  const dim3 grid(n_rows, n_rows >= 16 * num_sms() ? 1 : parts);
  DISPATCH_16(dtype, (gated_groups_kernel<T><<<grid, kThreads, 0, s>>>((const T*)in, (T*)out, (const int*)offsets,
                                                                     (const int*)counts, groups, F, act)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}
SXB_API int sxb_gated_act_bwd(const void* dy, const void* in, void* din, long long rows, int F,
                              int act, int dtype, void* stream) {
  if (rows <= 0) return SXB_OK;
  if (F % 8) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  DISPATCH_16(dtype, (gated_bwd_kernel<T><<<grid_for(rows * (F / 8)), kThreads, 0, s>>>(
                         (const T*)dy, (const T*)in, (T*)din, rows, F, act)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}
SXB_API int sxb_bias_act(const void* x, const void* bias, void* y, long long rows, int C, int act,
                         int dtype, void* stream) {
  if (rows <= 0) return SXB_OK;
  if (C % 8) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  DISPATCH_16(dtype, (bias_act_kernel<T><<<grid_for(rows * (C / 8)), kThreads, 0, s>>>(
                         (const T*)x, (const T*)bias, (T*)y, rows, C, act)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}
SXB_API int sxb_bias_act_bwd(const void* dy, const void* x, const void* bias, void* dx,
                             long long rows, int C, int act, int dtype, void* stream) {
  if (rows <= 0) return SXB_OK;
  if (C % 8) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  DISPATCH_16(dtype, (bias_act_bwd_kernel<T><<<grid_for(rows * (C / 8)), kThreads, 0, s>>>(
                         (const T*)dy, (const T*)x, (const T*)bias, (T*)dx, rows, C, act)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}

// The ends of a mean cross entropy, one CTA each: inv[0] = 1 / max(1, labels that count), out[0] = inv[0] * sum of the rows' losses
// (summed in 64 bits).  They take the place of eleven launches of elementwise kernels and reductions around the loss kernel.
namespace sxb {
namespace ew {
template <typename V>
__device__ __forceinline__ V block_total(V v) {
  __shared__ V part[32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = v;
  __syncthreads();
  v = threadIdx.x < blockDim.x / 32 ? part[threadIdx.x] : V(0);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;                              // on the first warp
}
__global__ void __launch_bounds__(1024)
label_weight_kernel(const long long* __restrict__ labels, long long rows, long long ignore, float* __restrict__ inv) {
  long long n = 0;
#pragma unroll 4
  for (long long i = threadIdx.x; i < rows; i += 1024) n += labels[i] != ignore;
  n = block_total(n);
  if (threadIdx.x == 0) inv[0] = 1.f / (float)(n > 1 ? n : 1);
}
__global__ void __launch_bounds__(1024)
mean_loss_kernel(const float* __restrict__ loss, long long rows, const float* __restrict__ inv, float* __restrict__ out) {
  double a = 0.0;
#pragma unroll 4
  for (long long i = threadIdx.x; i < rows; i += 1024) a += loss[i];
  a = block_total(a);
  if (threadIdx.x == 0) out[0] = (float)a * inv[0];
}
}  // namespace ew
}  // namespace sxb

SXB_API int sxb_label_weight(const void* labels, long long rows, long long ignore_index, void* inv, void* stream) {
  label_weight_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>((const long long*)labels, rows, ignore_index, (float*)inv);
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}
SXB_API int sxb_mean_loss(const void* loss, long long rows, const void* inv, void* out, void* stream) {
  mean_loss_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>((const float*)loss, rows, (const float*)inv, (float*)out);
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}

// logits [rows, V] (row pitch ld) are overwritten with the gradient when write_grad != 0.
SXB_API int sxb_cross_entropy(void* logits, const void* labels, void* loss, void* lse,
                              long long rows, int V, long long ld, long long ignore_index,
                              const void* grad_scale, int write_grad, int dtype, void* stream) {
  if (rows <= 0) return SXB_OK;
  if (ld % 8 || (reinterpret_cast<uintptr_t>(logits) & 15)) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  // Rows of at most one word per thread have nothing to ask for ahead, and eight such CTAs fit an SM with the registers of one word
  // (1024 rows of 256 columns: 4.4 us, 6.5 with four words; 3000 rows: 8.5, 10.1).
  // Short rows: 256 threads.  Long ones 512, two CTAs per SM, so that one reads while the other waits in its reductions;
  // 1024 while no SM has more than one row (64 rows, 128256 columns: 24.6 us, 26.6 with 512; 512 rows: 77.8 and 73.7).
#define LAUNCH_XENT(THREADS, CTAS, U)                                                                                         \
  DISPATCH_16(dtype, (xent_kernel<T, THREADS, CTAS, U><<<(unsigned)rows, THREADS, 0, s>>>(                                       \
                         (T*)logits, (const long long*)labels, (float*)loss, (float*)lse, V, ld, ignore_index,                \
                         (const float*)grad_scale, write_grad)))
  if (V <= 256 * 8) LAUNCH_XENT(256, 8, 1);
  else if (V < 32768) LAUNCH_XENT(256, 4, 4);
  else if (rows > num_sms()) LAUNCH_XENT(512, 2, 4);
  else LAUNCH_XENT(1024, 1, 4);
#undef LAUNCH_XENT
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}

// x [n] (16-bit, n a multiple of 8, 16-byte aligned) *= *scale (fp32 on the device), in place.
SXB_API int sxb_scale_by(void* x, long long n, const void* scale, int dtype, void* stream) {
  if (n <= 0) return SXB_OK;
  if (n % 8 || (reinterpret_cast<uintptr_t>(x) & 15)) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  DISPATCH_16(dtype, (scale_by_kernel<T><<<grid_for(n / 8), kThreads, 0, s>>>((T*)x, n / 8, (const float*)scale)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}

SXB_API int sxb_embedding_fwd(const void* ids, const void* table, void* out, long long ntok, int H,
                              int dtype, void* stream) {
  if (ntok <= 0) return SXB_OK;
  if (H % 8) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  DISPATCH_16(dtype, (embed_fwd_kernel<T><<<grid_for(ntok * (H / 8)), kThreads, 0, s>>>(
                         (const long long*)ids, (const T*)table, (T*)out, ntok, H)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}
SXB_API int sxb_embedding_bwd(const void* ids, const void* dout, void* dtable, long long ntok,
                              int H, int dtype, void* stream) {
  if (ntok <= 0) return SXB_OK;
  if (H % 2) return SXB_ERR_UNSUPPORTED;
  cudaStream_t s = (cudaStream_t)stream;
  DISPATCH_16(dtype, (embed_bwd_kernel<T><<<grid_for(ntok * (H / 2)), kThreads, 0, s>>>(
                         (const long long*)ids, (const T*)dout, (T*)dtable, ntok, H)));
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}

SXB_API int sxb_scale_cast(const void* src, void* dst, long long n, int src_dtype, int dst_dtype,
                           float scale, int accumulate, void* stream) {
  if (n <= 0) return SXB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  const int g = grid_for(n);
#define SC(TS, TD) scale_cast_kernel<TS, TD><<<g, kThreads, 0, s>>>((const TS*)src, (TD*)dst, n, scale, accumulate)
  if (src_dtype == kBF16 && dst_dtype == kF32) SC(__nv_bfloat16, float);
  else if (src_dtype == kF32 && dst_dtype == kBF16) SC(float, __nv_bfloat16);
  else if (src_dtype == kF16 && dst_dtype == kF32) SC(__half, float);
  else if (src_dtype == kF32 && dst_dtype == kF16) SC(float, __half);
  else if (src_dtype == kF32 && dst_dtype == kF32) SC(float, float);
  else if (src_dtype == kBF16 && dst_dtype == kBF16) SC(__nv_bfloat16, __nv_bfloat16);
  else if (src_dtype == kF16 && dst_dtype == kF16) SC(__half, __half);
  else return SXB_ERR_BAD_ARG;
#undef SC
  SXB_CHECK_LAUNCH();
  return SXB_OK;
}
