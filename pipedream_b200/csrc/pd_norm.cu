// BatchNorm2d (training and inference) on padded-NHWC activations, for the ResNet-50 stages
// (runtime/image_classification/models/resnet50/gpus=4/stage0.py:12-55; cuDNN BN in the reference),
// with the residual add and the ReLU that follow the last normalisation of a bottleneck block
// (stage1.py forward: `out = out + identity; out = relu(out)`) folded into the same passes.
//
// The buffer is a [P, C] matrix, P = N*(H+2)*(W+2), whose border rows are zero; sums over all P rows are
// therefore sums over the N*H*W real pixels, and only the element count has to exclude the border.
//   forward : per-channel sum / sum of squares (two-level reduction, fixed order: deterministic), then
//             y = (x-mean)*invstd*gamma+beta (+ residual) (optional ReLU), border rows written as zero;
//             running statistics updated like torch.
//   backward: g = dy (zeroed where y <= 0 when the forward applied a ReLU); per-channel sum(g) and
//             sum(g*xhat); dx = gamma*invstd*(g - sum(g)/cnt - xhat*sum(g*xhat)/cnt), border rows zero;
//             g itself is the gradient of the residual input.
// All kernels are HBM-bound: tensors whose channel count is 8 times a power of two up to 256 (every ResNet-50
// layer) take a path with 16-byte accesses in which a thread keeps the same 8 channels for the whole launch;
// everything else takes the generic scalar path.  On the vector path the forward pass can leave one bit per
// value (y > 0) for the backward pass, which then reads 1/16 of the bytes that y itself takes in its two passes.
#include "pd_common.cuh"

namespace {

constexpr int kThreads = 256;
constexpr int kMaxColsPerThread = 8;      // generic path: C <= 2048

__device__ __forceinline__ bool is_border(int64_t row, int Hp, int Wp) {
  const int wp = (int)(row % Wp);
  const int hp = (int)((row / Wp) % Hp);
  return wp == 0 || wp == Wp - 1 || hp == 0 || hp == Hp - 1;
}

// Eight consecutive values of a channel group: 16 bytes of bf16, 32 bytes of fp32.
template <typename T> struct Vec8;
template <> struct Vec8<__nv_bfloat16> {
  uint4 u;
  __device__ __forceinline__ void zero() { u = make_uint4(0u, 0u, 0u, 0u); }
  __device__ __forceinline__ void load(const __nv_bfloat16* p, int64_t i) { u = reinterpret_cast<const uint4*>(p)[i]; }
  __device__ __forceinline__ void store(__nv_bfloat16* p, int64_t i) const { reinterpret_cast<uint4*>(p)[i] = u; }
  __device__ __forceinline__ void get(float* f) const {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 t = __bfloat1622float2(p[k]);
      f[2 * k] = t.x;
      f[2 * k + 1] = t.y;
    }
  }
  __device__ __forceinline__ void set(const float* f) {
    __nv_bfloat162* p = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int k = 0; k < 4; ++k) p[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
  }
};
template <> struct Vec8<float> {
  float4 a, b;
  __device__ __forceinline__ void zero() { a = b = make_float4(0.f, 0.f, 0.f, 0.f); }
  __device__ __forceinline__ void load(const float* p, int64_t i) {
    a = reinterpret_cast<const float4*>(p)[2 * i];
    b = reinterpret_cast<const float4*>(p)[2 * i + 1];
  }
  __device__ __forceinline__ void store(float* p, int64_t i) const {
    reinterpret_cast<float4*>(p)[2 * i] = a;
    reinterpret_cast<float4*>(p)[2 * i + 1] = b;
  }
  __device__ __forceinline__ void get(float* f) const {
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
  }
  __device__ __forceinline__ void set(const float* f) {
    a = make_float4(f[0], f[1], f[2], f[3]);
    b = make_float4(f[4], f[5], f[6], f[7]);
  }
};

// ------------------------------------------------------------------------------------------------
// generic path (channel counts the vector path does not take)
// ------------------------------------------------------------------------------------------------
// partial[block][0][C] = sum_r a(r,c), partial[block][1][C] = sum_r b(r,c) over the block's rows.
//   mode 0 (forward statistics): a = x, b = x*x
//   mode 1 (backward sums)     : g = dy (zeroed where y <= 0 when y != null); a = g, b = g * xhat
template <typename T>
__global__ void __launch_bounds__(kThreads)
bn_reduce_kernel(const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ y,
                 const float* __restrict__ mean, const float* __restrict__ invstd, int64_t rows, int C, int mode,
                 float* __restrict__ partial) {
  float a[kMaxColsPerThread], b[kMaxColsPerThread];
#pragma unroll
  for (int k = 0; k < kMaxColsPerThread; ++k) a[k] = b[k] = 0.f;
  const int64_t per = (rows + gridDim.x - 1) / gridDim.x;
  const int64_t r0 = (int64_t)blockIdx.x * per, r1 = min(rows, r0 + per);
  for (int64_t r = r0; r < r1; ++r) {
#pragma unroll
    for (int k = 0; k < kMaxColsPerThread; ++k) {
      const int c = threadIdx.x + k * kThreads;
      if (c < C) {
        const int64_t i = r * C + c;
        if (mode == 0) {
          const float v = pd_to_float(x[i]);
          a[k] += v; b[k] += v * v;
        } else {
          float g = pd_to_float(dy[i]);
          if (y != nullptr && !(pd_to_float(y[i]) > 0.f)) g = 0.f;
          a[k] += g;
          b[k] += g * (pd_to_float(x[i]) - mean[c]) * invstd[c];
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < kMaxColsPerThread; ++k) {
    const int c = threadIdx.x + k * kThreads;
    if (c < C) {
      partial[((int64_t)blockIdx.x * 2) * C + c] = a[k];
      partial[((int64_t)blockIdx.x * 2 + 1) * C + c] = b[k];
    }
  }
}

// The inference path hands over running variances (eps >= 0), the training path finished 1/sqrt(var + eps) (eps < 0).
__device__ __forceinline__ float scale_of(float v, float eps) { return eps < 0.f ? v : rsqrtf(v + eps); }

template <typename T>
__global__ void __launch_bounds__(kThreads)
bn_apply_kernel(const T* __restrict__ x, const T* __restrict__ res, const float* __restrict__ mean,
                const float* __restrict__ invstd, float eps, const T* __restrict__ gamma, const T* __restrict__ beta,
                int64_t rows, int C, int Hp, int Wp, int relu, T* __restrict__ y) {
  const int64_t total = rows * C;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const int64_t r = i / C;
    float v = 0.f;
    if (!is_border(r, Hp, Wp)) {
      v = (pd_to_float(x[i]) - mean[c]) * scale_of(invstd[c], eps) * pd_to_float(gamma[c]) + pd_to_float(beta[c]);
      if (res != nullptr) v += pd_to_float(res[i]);
      if (relu) v = fmaxf(v, 0.f);
    }
    y[i] = pd_from_float<T>(v);
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
bn_bwd_apply_kernel(const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ y,
                    const float* __restrict__ mean, const float* __restrict__ invstd, const T* __restrict__ gamma,
                    const float* __restrict__ sums, int64_t rows, int C, int Hp, int Wp, float inv_count,
                    T* __restrict__ dx, T* __restrict__ dres) {
  const int64_t total = rows * C;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int c = (int)(i % C);
    const int64_t r = i / C;
    float v = 0.f, g = 0.f;
    if (!is_border(r, Hp, Wp)) {
      g = pd_to_float(dy[i]);
      if (y != nullptr && !(pd_to_float(y[i]) > 0.f)) g = 0.f;
      const float xhat = (pd_to_float(x[i]) - mean[c]) * invstd[c];
      v = pd_to_float(gamma[c]) * invstd[c] * (g - sums[c] * inv_count - xhat * sums[C + c] * inv_count);
    }
    dx[i] = pd_from_float<T>(v);
    if (dres != nullptr) dres[i] = pd_from_float<T>(g);
  }
}

// ------------------------------------------------------------------------------------------------
// second level of the reductions (both paths): one block per 32 channels, 32 slices of the partials each
// (the loop over the partials is a chain of L2 round trips: short and wide beats long and narrow; 16 loads a thread
// are in flight at a time)
// ------------------------------------------------------------------------------------------------
__device__ __forceinline__ void sum_partials(const float* __restrict__ partial, int nblocks, int C, int c,
                                             float (*sh)[32][33], float& s, float& q) {
  s = q = 0.f;
  if (c < C) {
    for (int b0 = threadIdx.y; b0 < nblocks; b0 += 32 * 8) {
      float ps[8], pq[8];
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const int b = b0 + u * 32;
        ps[u] = b < nblocks ? partial[((int64_t)b * 2) * C + c] : 0.f;
        pq[u] = b < nblocks ? partial[((int64_t)b * 2 + 1) * C + c] : 0.f;
      }
#pragma unroll
      for (int u = 0; u < 8; ++u) { s += ps[u]; q += pq[u]; }
    }
  }
  sh[0][threadIdx.y][threadIdx.x] = s;
  sh[1][threadIdx.y][threadIdx.x] = q;
  __syncthreads();
  if (threadIdx.y == 0) {
    s = q = 0.f;
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      s += sh[0][j][threadIdx.x];
      q += sh[1][j][threadIdx.x];
    }
  }
}

// Forward: mean, invstd from the partial sums; running statistics (momentum, unbiased variance).
__global__ void __launch_bounds__(1024)
bn_stats_final_kernel(const float* __restrict__ partial, int nblocks, int C, float count, float eps, float momentum,
                      float* __restrict__ mean, float* __restrict__ invstd, float* __restrict__ running_mean,
                      float* __restrict__ running_var) {
  __shared__ float sh[2][32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s, q;
  sum_partials(partial, nblocks, C, c, sh, s, q);
  if (threadIdx.y != 0 || c >= C) return;
  const float m = s / count;
  const float var = fmaxf(q / count - m * m, 0.f);
  mean[c] = m;
  invstd[c] = rsqrtf(var + eps);
  if (running_mean != nullptr) {
    running_mean[c] = (1.f - momentum) * running_mean[c] + momentum * m;
    const float unbiased = count > 1.f ? var * count / (count - 1.f) : var;
    running_var[c] = (1.f - momentum) * running_var[c] + momentum * unbiased;
  }
}

// Backward: sums[0][C] = sum(g), sums[1][C] = sum(g*xhat); also the parameter gradients.
__global__ void __launch_bounds__(1024)
bn_bwd_final_kernel(const float* __restrict__ partial, int nblocks, int C, float* __restrict__ sums,
                    float* __restrict__ dgamma, float* __restrict__ dbeta, int accumulate) {
  __shared__ float sh[2][32][33];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s, q;
  sum_partials(partial, nblocks, C, c, sh, s, q);
  if (threadIdx.y != 0 || c >= C) return;
  sums[c] = s;
  sums[C + c] = q;
  if (dbeta != nullptr) dbeta[c] = accumulate ? dbeta[c] + s : s;
  if (dgamma != nullptr) dgamma[c] = accumulate ? dgamma[c] + q : q;
}

// ------------------------------------------------------------------------------------------------
// Vector path.  The matrix is read as nvec = P*C/8 vectors of 8 values; G = C/8 vectors per row, G a power of two
// <= 256, so a thread's channel group (index mod G) never changes.  MASK: where the forward pass applied a ReLU, what
// says that a value passed: 0 nothing to mask, 1 the output y, 2 one byte per vector that the forward pass left.
// ------------------------------------------------------------------------------------------------
template <typename T, int MASK>
struct Passed {
  Vec8<T> y;
  unsigned char bits;
  __device__ __forceinline__ void load(const T* yp, const unsigned char* mp, int64_t i, bool ok) {
    if (MASK == 1) { if (ok) y.load(yp, i); else y.zero(); }
    if (MASK == 2) bits = ok ? mp[i] : (unsigned char)0;
  }
  __device__ __forceinline__ void apply(float* g) const {
    if (MASK == 1) {
      float yf[8];
      y.get(yf);
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (!(yf[k] > 0.f)) g[k] = 0.f;
    }
    if (MASK == 2) {
#pragma unroll
      for (int k = 0; k < 8; ++k)
        if (!((bits >> k) & 1)) g[k] = 0.f;
    }
  }
};

template <typename T, int MODE, int MASK>
__global__ void __launch_bounds__(kThreads)
bn_reduce_v8_kernel(const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ y,
                    const unsigned char* __restrict__ mask, const float* __restrict__ mean,
                    const float* __restrict__ invstd, int64_t nvec, int G, int C, float* __restrict__ partial) {
  __shared__ float sh[kThreads][17];
  const int tid = threadIdx.x;
  const int cg = tid & (G - 1);
  float a[8], b[8], m[8], is[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    a[k] = b[k] = 0.f;
    if (MODE == 1) { m[k] = mean[cg * 8 + k]; is[k] = invstd[cg * 8 + k]; }
  }
  // contiguous chunk per block, a multiple of the block size so that the channel group stays put
  const int64_t per = (((nvec + gridDim.x - 1) / gridDim.x) + kThreads - 1) / kThreads * kThreads;
  const int64_t v0 = (int64_t)blockIdx.x * per;
  const int64_t v1 = min(nvec, v0 + per);
  constexpr int U = (MODE == 1 && (MASK == 1 || sizeof(T) == 4)) ? 2 : 4;
  for (int64_t base = v0 + tid; base < v1; base += (int64_t)kThreads * U) {
    Vec8<T> xv[U], gv[U];
    Passed<T, MASK> pass[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + (int64_t)u * kThreads;
      const bool ok = i < v1;
      if (ok) xv[u].load(x, i); else xv[u].zero();
      if (MODE == 1) {
        if (ok) gv[u].load(dy, i); else gv[u].zero();
        pass[u].load(y, mask, i, ok);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      float xf[8];
      xv[u].get(xf);
      if (MODE == 0) {
#pragma unroll
        for (int k = 0; k < 8; ++k) { a[k] += xf[k]; b[k] += xf[k] * xf[k]; }
      } else {
        float gf[8];
        gv[u].get(gf);
        pass[u].apply(gf);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          a[k] += gf[k];
          b[k] += gf[k] * (xf[k] - m[k]) * is[k];
        }
      }
    }
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) { sh[tid][k] = a[k]; sh[tid][8 + k] = b[k]; }
  __syncthreads();
  const int R = kThreads / G;
  for (int j = tid; j < 16 * G; j += kThreads) {
    const int g2 = j & (G - 1), k = j / G;
    float s = 0.f;
    for (int r = 0; r < R; ++r) s += sh[r * G + g2][k];
    partial[((int64_t)blockIdx.x * 2 + (k >> 3)) * C + g2 * 8 + (k & 7)] = s;
  }
}

__device__ __forceinline__ bool border_of_vec(int64_t i, int gshift, int Hp, int Wp) {
  const unsigned row = (unsigned)(i >> gshift);
  const unsigned q = row / (unsigned)Wp;
  const unsigned wp = row - q * (unsigned)Wp;
  const unsigned hp = q % (unsigned)Hp;
  return wp == 0 || wp == (unsigned)Wp - 1 || hp == 0 || hp == (unsigned)Hp - 1;
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
bn_apply_v8_kernel(const T* __restrict__ x, const T* __restrict__ res, const float* __restrict__ mean,
                   const float* __restrict__ invstd, float eps, const T* __restrict__ gamma,
                   const T* __restrict__ beta, int64_t nvec, int G, int gshift, int Hp, int Wp, int relu,
                   T* __restrict__ y, unsigned char* __restrict__ mask) {
  const int cg = threadIdx.x & (G - 1);
  float scale[8], shift[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int c = cg * 8 + k;
    scale[k] = scale_of(invstd[c], eps) * pd_to_float(gamma[c]);
    shift[k] = pd_to_float(beta[c]) - mean[c] * scale[k];
  }
  constexpr int U = sizeof(T) == 4 ? 2 : 4;
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  for (int64_t base = (int64_t)blockIdx.x * kThreads + threadIdx.x; base < nvec; base += stride * U) {
    Vec8<T> xv[U], rv[U];
    bool ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + (int64_t)u * stride;
      ok[u] = i < nvec && !border_of_vec(i, gshift, Hp, Wp);
      if (ok[u]) xv[u].load(x, i); else xv[u].zero();
      if (res != nullptr) { if (ok[u]) rv[u].load(res, i); else rv[u].zero(); }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + (int64_t)u * stride;
      if (i >= nvec) break;
      Vec8<T> out;
      out.zero();
      unsigned int bits = 0u;
      if (ok[u]) {
        float f[8], r[8];
        xv[u].get(f);
        if (res != nullptr) rv[u].get(r);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          float v = f[k] * scale[k] + shift[k];
          if (res != nullptr) v += r[k];
          f[k] = relu ? fmaxf(v, 0.f) : v;
        }
        out.set(f);
        if (mask != nullptr) {
          out.get(f);                      // as stored: what rounds to zero has not passed
#pragma unroll
          for (int k = 0; k < 8; ++k) bits |= f[k] > 0.f ? 1u << k : 0u;
        }
      }
      out.store(y, i);
      if (mask != nullptr) mask[i] = (unsigned char)bits;
    }
  }
}

template <typename T, int MASK>
__global__ void __launch_bounds__(kThreads)
bn_bwd_apply_v8_kernel(const T* __restrict__ x, const T* __restrict__ dy, const T* __restrict__ y,
                       const unsigned char* __restrict__ mask, const float* __restrict__ mean,
                       const float* __restrict__ invstd, const T* __restrict__ gamma, const float* __restrict__ sums,
                       int64_t nvec, int G, int gshift, int C, int Hp, int Wp, float inv_count, T* __restrict__ dx,
                       T* __restrict__ dres) {
  const int cg = threadIdx.x & (G - 1);
  // dx = k1 * (g - c1 - (x - mean) * c2),  k1 = gamma*invstd, c1 = sum(g)/cnt, c2 = invstd*sum(g*xhat)/cnt
  float k1[8], c1[8], c2[8], m[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int c = cg * 8 + k;
    const float is = invstd[c];
    k1[k] = pd_to_float(gamma[c]) * is;
    c1[k] = sums[c] * inv_count;
    c2[k] = is * sums[C + c] * inv_count;
    m[k] = mean[c];
  }
  constexpr int U = (MASK == 1 || sizeof(T) == 4) ? 2 : 4;
  const int64_t stride = (int64_t)gridDim.x * kThreads;
  for (int64_t base = (int64_t)blockIdx.x * kThreads + threadIdx.x; base < nvec; base += stride * U) {
    Vec8<T> xv[U], gv[U];
    Passed<T, MASK> pass[U];
    bool ok[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + (int64_t)u * stride;
      ok[u] = i < nvec && !border_of_vec(i, gshift, Hp, Wp);
      if (ok[u]) { xv[u].load(x, i); gv[u].load(dy, i); } else { xv[u].zero(); gv[u].zero(); }
      pass[u].load(y, mask, i, ok[u]);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t i = base + (int64_t)u * stride;
      if (i >= nvec) break;
      Vec8<T> out, gout;
      out.zero();
      gout.zero();
      if (ok[u]) {
        float xf[8], gf[8];
        xv[u].get(xf);
        gv[u].get(gf);
        pass[u].apply(gf);
#pragma unroll
        for (int k = 0; k < 8; ++k) xf[k] = k1[k] * (gf[k] - c1[k] - (xf[k] - m[k]) * c2[k]);
        out.set(xf);
        gout.set(gf);
      }
      out.store(dx, i);
      if (dres != nullptr) gout.store(dres, i);
    }
  }
}

int reduce_blocks() { return pd_num_sms() * 4; }
int apply_grid(int64_t total) {
  int64_t blocks = (total + kThreads - 1) / kThreads;
  int64_t cap = (int64_t)pd_num_sms() * 16;
  return (int)(blocks < cap ? (blocks < 1 ? 1 : blocks) : cap);
}
// vector path: grid capped at 8 blocks per SM, `per_thread` vectors per thread and pass
int vec_grid(int64_t nvec, int per_thread) {
  int64_t blocks = (nvec + (int64_t)kThreads * per_thread - 1) / ((int64_t)kThreads * per_thread);
  int64_t cap = (int64_t)pd_num_sms() * 8;
  return (int)(blocks < cap ? (blocks < 1 ? 1 : blocks) : cap);
}
// number of first-level blocks: one per 64 KB of input, at most reduce_blocks()
int reduce_grid(int64_t nvec) {
  int64_t blocks = (nvec * 16 + 65535) / 65536;
  int64_t cap = reduce_blocks();
  return (int)(blocks < cap ? (blocks < 1 ? 1 : blocks) : cap);
}
// Whole vectors in every row, a power of two of them, and the tensors on 16 bytes.
bool vector_path(int C, const void* a, const void* b, const void* c, const void* d) {
  if ((C % 8) != 0) return false;
  const int G = C / 8;
  const uintptr_t all = (uintptr_t)a | (uintptr_t)b | (uintptr_t)c | (uintptr_t)d;
  return G <= kThreads && (G & (G - 1)) == 0 && all % 16 == 0;
}
int log2i(int v) { int s = 0; while ((1 << s) < v) ++s; return s; }

}  // namespace

namespace {

template <typename T>
int bn_apply_any(const T* x, const T* res, int64_t rows, int Hp, int Wp, int C, const T* gamma, const T* beta,
                 const float* mean, const float* invstd, float eps, int relu, T* y, unsigned char* mask, bool vec,
                 cudaStream_t s) {
  if (vec) {
    const int64_t nvec = rows * C / 8;
    bn_apply_v8_kernel<T><<<vec_grid(nvec, sizeof(T) == 4 ? 2 : 4), kThreads, 0, s>>>(
        x, res, mean, invstd, eps, gamma, beta, nvec, C / 8, log2i(C / 8), Hp, Wp, relu, y, mask);
  } else {
    bn_apply_kernel<T><<<apply_grid(rows * C), kThreads, 0, s>>>(x, res, mean, invstd, eps, gamma, beta, rows, C, Hp, Wp,
                                                                 relu, y);
  }
  PD_LAUNCH_CHECK("bn_apply_kernel");
  return PD_OK;
}

template <typename T>
int bn_fwd_any(const T* x, const T* res, int64_t rows, float count, int Hp, int Wp, int C, const T* gamma, const T* beta,
               float eps, float momentum, int relu, float* mean, float* invstd, float* running_mean, float* running_var,
               T* y, unsigned char* mask, float* workspace, bool vec, cudaStream_t s) {
  const int64_t nvec = rows * C / 8;
  const int nb = vec ? reduce_grid(nvec * (int)sizeof(T) / 2) : reduce_blocks();
  if (vec)
    bn_reduce_v8_kernel<T, 0, 0><<<nb, kThreads, 0, s>>>(x, nullptr, nullptr, nullptr, nullptr, nullptr, nvec, C / 8, C, workspace);
  else
    bn_reduce_kernel<T><<<nb, kThreads, 0, s>>>(x, nullptr, nullptr, nullptr, nullptr, rows, C, 0, workspace);
  PD_LAUNCH_CHECK("bn_reduce_kernel");
  bn_stats_final_kernel<<<(C + 31) / 32, dim3(32, 32), 0, s>>>(workspace, nb, C, count, eps, momentum, mean, invstd,
                                                              running_mean, running_var);
  PD_LAUNCH_CHECK("bn_stats_final_kernel");
  return bn_apply_any<T>(x, res, rows, Hp, Wp, C, gamma, beta, mean, invstd, -1.f, relu, y, mask, vec, s);
}

template <typename T, int MASK>
int bn_bwd_vec(const T* x, const T* dy, const T* y, const unsigned char* mask, int64_t rows, float inv_count, int Hp,
               int Wp, int C, const T* gamma, const float* mean, const float* invstd, float* dgamma, float* dbeta,
               int accumulate, T* dx, T* dres, float* sums, float* workspace, cudaStream_t s) {
  const int64_t nvec = rows * C / 8;
  const int nb = reduce_grid(nvec * (int)sizeof(T) / 2);
  bn_reduce_v8_kernel<T, 1, MASK><<<nb, kThreads, 0, s>>>(x, dy, y, mask, mean, invstd, nvec, C / 8, C, workspace);
  PD_LAUNCH_CHECK("bn_reduce_kernel");
  bn_bwd_final_kernel<<<(C + 31) / 32, dim3(32, 32), 0, s>>>(workspace, nb, C, sums, dgamma, dbeta, accumulate);
  PD_LAUNCH_CHECK("bn_bwd_final_kernel");
  const int grid = vec_grid(nvec, (MASK == 1 || sizeof(T) == 4) ? 2 : 4);
  bn_bwd_apply_v8_kernel<T, MASK><<<grid, kThreads, 0, s>>>(x, dy, y, mask, mean, invstd, gamma, sums, nvec, C / 8,
                                                            log2i(C / 8), C, Hp, Wp, inv_count, dx, dres);
  PD_LAUNCH_CHECK("bn_bwd_apply_kernel");
  return PD_OK;
}

template <typename T>
int bn_bwd_any(const T* x, const T* dy, const T* y, const unsigned char* mask, int64_t rows, float inv_count, int Hp,
               int Wp, int C, const T* gamma, const float* mean, const float* invstd, float* dgamma, float* dbeta,
               int accumulate, T* dx, T* dres, float* sums, float* workspace, bool vec, cudaStream_t s) {
  if (vec && mask != nullptr)
    return bn_bwd_vec<T, 2>(x, dy, nullptr, mask, rows, inv_count, Hp, Wp, C, gamma, mean, invstd, dgamma, dbeta, accumulate,
                            dx, dres, sums, workspace, s);
  if (vec && y != nullptr)
    return bn_bwd_vec<T, 1>(x, dy, y, nullptr, rows, inv_count, Hp, Wp, C, gamma, mean, invstd, dgamma, dbeta, accumulate, dx,
                            dres, sums, workspace, s);
  if (vec)
    return bn_bwd_vec<T, 0>(x, dy, nullptr, nullptr, rows, inv_count, Hp, Wp, C, gamma, mean, invstd, dgamma, dbeta,
                            accumulate, dx, dres, sums, workspace, s);
  const int nb = reduce_blocks();
  bn_reduce_kernel<T><<<nb, kThreads, 0, s>>>(x, dy, y, mean, invstd, rows, C, 1, workspace);
  PD_LAUNCH_CHECK("bn_reduce_kernel");
  bn_bwd_final_kernel<<<(C + 31) / 32, dim3(32, 32), 0, s>>>(workspace, nb, C, sums, dgamma, dbeta, accumulate);
  PD_LAUNCH_CHECK("bn_bwd_final_kernel");
  bn_bwd_apply_kernel<T><<<apply_grid(rows * C), kThreads, 0, s>>>(x, dy, y, mean, invstd, gamma, sums, rows, C, Hp, Wp,
                                                                   inv_count, dx, dres);
  PD_LAUNCH_CHECK("bn_bwd_apply_kernel");
  return PD_OK;
}

}  // namespace

// workspace: fp32 scratch of at least pd_bn_workspace_bytes(C) bytes.
PD_EXPORT int64_t pd_bn_workspace_bytes(int C) { return (int64_t)reduce_blocks() * 2 * C * sizeof(float); }

// Bytes of the mask that pd_bn_fwd_masked writes for pd_bn_bwd_masked; 0: the shape has none (pass y instead).
PD_EXPORT int64_t pd_bn_mask_bytes(int N, int H, int W, int C) {
  return vector_path(C, nullptr, nullptr, nullptr, nullptr) ? (int64_t)N * (H + 2) * (W + 2) * (C / 8) : 0;
}

// Training forward.  x_pad/y_pad (and res_pad, the optional tensor added before the ReLU): [N,H+2,W+2,C];
// gamma/beta in `dtype`; mean/invstd: fp32 [C] (out, saved for backward); running_mean/var: fp32 [C],
// updated in place (may be NULL).  mask (may be NULL): pd_bn_mask_bytes bytes, one bit per value (y > 0).
PD_EXPORT int pd_bn_fwd_masked(int dtype, const void* x_pad, const void* res_pad, int N, int H, int W, int C,
                               const void* gamma, const void* beta, float eps, float momentum, int relu, float* mean,
                               float* invstd, float* running_mean, float* running_var, void* y_pad, void* mask,
                               void* workspace, int64_t workspace_bytes, void* stream) {
  int rc = pd_check_device();
  if (rc != PD_OK) return rc;
  PD_REQUIRE(x_pad && gamma && beta && mean && invstd && y_pad && workspace && N > 0 && H > 0 && W > 0 && C > 0,
             "pd_bn_fwd: bad arguments");
  PD_REQUIRE(dtype == PD_F32 || dtype == PD_BF16, "pd_bn_fwd: bad dtype");
  PD_REQUIRE(C <= kThreads * kMaxColsPerThread, "pd_bn_fwd: at most %d channels", kThreads * kMaxColsPerThread);
  PD_REQUIRE(workspace_bytes >= pd_bn_workspace_bytes(C), "pd_bn_fwd: workspace too small");
  const int Hp = H + 2, Wp = W + 2;
  const int64_t rows = (int64_t)N * Hp * Wp;
  PD_REQUIRE(rows < (1ll << 31), "pd_bn_fwd: too many rows");
  const float count = (float)((int64_t)N * H * W);
  const bool vec = vector_path(C, x_pad, res_pad, y_pad, nullptr);
  PD_REQUIRE(vec || mask == nullptr, "pd_bn_fwd: no mask for this shape or alignment");
  if (dtype == PD_F32)
    return bn_fwd_any<float>((const float*)x_pad, (const float*)res_pad, rows, count, Hp, Wp, C, (const float*)gamma,
                             (const float*)beta, eps, momentum, relu, mean, invstd, running_mean, running_var, (float*)y_pad,
                             (unsigned char*)mask, (float*)workspace, vec, (cudaStream_t)stream);
  using B = __nv_bfloat16;
  return bn_fwd_any<B>((const B*)x_pad, (const B*)res_pad, rows, count, Hp, Wp, C, (const B*)gamma, (const B*)beta, eps,
                       momentum, relu, mean, invstd, running_mean, running_var, (B*)y_pad, (unsigned char*)mask,
                       (float*)workspace, vec, (cudaStream_t)stream);
}

PD_EXPORT int pd_bn_fwd(int dtype, const void* x_pad, const void* res_pad, int N, int H, int W, int C, const void* gamma,
                        const void* beta, float eps, float momentum, int relu, float* mean, float* invstd,
                        float* running_mean, float* running_var, void* y_pad, void* workspace, int64_t workspace_bytes,
                        void* stream) {
  return pd_bn_fwd_masked(dtype, x_pad, res_pad, N, H, W, C, gamma, beta, eps, momentum, relu, mean, invstd, running_mean,
                          running_var, y_pad, nullptr, workspace, workspace_bytes, stream);
}

static int bn_infer(int dtype, const void* x_pad, const void* res_pad, int N, int H, int W, int C, const void* gamma,
                    const void* beta, const float* mean, const float* scale, float eps, int relu, void* y_pad, void* stream) {
  int rc = pd_check_device();
  if (rc != PD_OK) return rc;
  PD_REQUIRE(x_pad && gamma && beta && mean && scale && y_pad && N > 0 && H > 0 && W > 0 && C > 0, "pd_bn_apply: bad arguments");
  PD_REQUIRE(dtype == PD_F32 || dtype == PD_BF16, "pd_bn_apply: bad dtype");
  const int Hp = H + 2, Wp = W + 2;
  const int64_t rows = (int64_t)N * Hp * Wp;
  PD_REQUIRE(rows < (1ll << 31), "pd_bn_apply: too many rows");
  const bool vec = vector_path(C, x_pad, res_pad, y_pad, nullptr);
  if (dtype == PD_F32)
    return bn_apply_any<float>((const float*)x_pad, (const float*)res_pad, rows, Hp, Wp, C, (const float*)gamma,
                               (const float*)beta, mean, scale, eps, relu, (float*)y_pad, nullptr, vec, (cudaStream_t)stream);
  using B = __nv_bfloat16;
  return bn_apply_any<B>((const B*)x_pad, (const B*)res_pad, rows, Hp, Wp, C, (const B*)gamma, (const B*)beta, mean, scale, eps,
                         relu, (B*)y_pad, nullptr, vec, (cudaStream_t)stream);
}

// Inference forward: normalises with the given statistics (mean, invstd fp32 [C]).
PD_EXPORT int pd_bn_apply(int dtype, const void* x_pad, const void* res_pad, int N, int H, int W, int C, const void* gamma,
                          const void* beta, const float* mean, const float* invstd, int relu, void* y_pad, void* stream) {
  return bn_infer(dtype, x_pad, res_pad, N, H, W, C, gamma, beta, mean, invstd, -1.f, relu, y_pad, stream);
}

// The same from the running variance (eps >= 0): 1/sqrt(var + eps) is taken in the kernel, which spares the two
// launches per layer that made up 150 us of a 1.0 ms ResNet-50 forward pass over one image.
PD_EXPORT int pd_bn_apply_var(int dtype, const void* x_pad, const void* res_pad, int N, int H, int W, int C,
                              const void* gamma, const void* beta, const float* mean, const float* var, float eps, int relu,
                              void* y_pad, void* stream) {
  PD_REQUIRE(eps >= 0.f, "pd_bn_apply_var: eps has to be >= 0");
  return bn_infer(dtype, x_pad, res_pad, N, H, W, C, gamma, beta, mean, var, eps, relu, y_pad, stream);
}

// Training backward.  The forward applied a ReLU and dy is masked by (y > 0) first: y_pad != NULL, or mask != NULL (what
// pd_bn_fwd_masked left, taken instead of y).  dgamma/dbeta: fp32 [C] (stored, or added to when accumulate != 0).
// dres_pad (may be NULL): receives the masked dy, i.e. the gradient of the residual input.  sums_ws: fp32 [2*C] scratch.
PD_EXPORT int pd_bn_bwd_masked(int dtype, const void* x_pad, const void* dy_pad, const void* y_pad, const void* mask, int N,
                               int H, int W, int C, const void* gamma, const float* mean, const float* invstd, float* dgamma,
                               float* dbeta, int accumulate, void* dx_pad, void* dres_pad, float* sums_ws, void* workspace,
                               int64_t workspace_bytes, void* stream) {
  int rc = pd_check_device();
  if (rc != PD_OK) return rc;
  PD_REQUIRE(x_pad && dy_pad && gamma && mean && invstd && dx_pad && sums_ws && workspace && N > 0 && H > 0 && W > 0 && C > 0,
             "pd_bn_bwd: bad arguments");
  PD_REQUIRE(dtype == PD_F32 || dtype == PD_BF16, "pd_bn_bwd: bad dtype");
  PD_REQUIRE(C <= kThreads * kMaxColsPerThread, "pd_bn_bwd: at most %d channels", kThreads * kMaxColsPerThread);
  PD_REQUIRE(workspace_bytes >= pd_bn_workspace_bytes(C), "pd_bn_bwd: workspace too small");
  const int Hp = H + 2, Wp = W + 2;
  const int64_t rows = (int64_t)N * Hp * Wp;
  PD_REQUIRE(rows < (1ll << 31), "pd_bn_bwd: too many rows");
  const float inv_count = 1.f / (float)((int64_t)N * H * W);
  const uintptr_t grads = (uintptr_t)dy_pad | (uintptr_t)dx_pad;
  const bool vec = vector_path(C, x_pad, (const void*)grads, y_pad, dres_pad);
  PD_REQUIRE(vec || mask == nullptr, "pd_bn_bwd: no mask for this shape or alignment");
  if (dtype == PD_F32)
    return bn_bwd_any<float>((const float*)x_pad, (const float*)dy_pad, (const float*)y_pad, (const unsigned char*)mask, rows,
                             inv_count, Hp, Wp, C, (const float*)gamma, mean, invstd, dgamma, dbeta, accumulate, (float*)dx_pad,
                             (float*)dres_pad, sums_ws, (float*)workspace, vec, (cudaStream_t)stream);
  using B = __nv_bfloat16;
  return bn_bwd_any<B>((const B*)x_pad, (const B*)dy_pad, (const B*)y_pad, (const unsigned char*)mask, rows, inv_count, Hp, Wp,
                       C, (const B*)gamma, mean, invstd, dgamma, dbeta, accumulate, (B*)dx_pad, (B*)dres_pad, sums_ws,
                       (float*)workspace, vec, (cudaStream_t)stream);
}

PD_EXPORT int pd_bn_bwd(int dtype, const void* x_pad, const void* dy_pad, const void* y_pad, int N, int H, int W, int C,
                        const void* gamma, const float* mean, const float* invstd, float* dgamma, float* dbeta,
                        int accumulate, void* dx_pad, void* dres_pad, float* sums_ws, void* workspace,
                        int64_t workspace_bytes, void* stream) {
  return pd_bn_bwd_masked(dtype, x_pad, dy_pad, y_pad, nullptr, N, H, W, C, gamma, mean, invstd, dgamma, dbeta, accumulate,
                          dx_pad, dres_pad, sums_ws, workspace, workspace_bytes, stream);
}
