// fp32 contraction back end.  Same problem description as the bf16 path; fp32 operands and results, at the precision of
// fp32 sums (rounding the operands for the tensor cores would not meet the 1e-3 tolerance of the fp32 configuration
// after 20 training steps).  Two kinds of tiles: FMAs on CUDA cores, for problems too small for the other kind, and
// three-part bf16 products on the tensor cores (gemm_split_kernel below); pick_tile chooses by estimated time.
//
// The FMA tiles.
// Bound by the FMA pipe: 128 lanes per SM, 74 TFLOP/s at 1.965 GHz.  Every thread keeps an 8 x 8 block of outputs in
// registers, so that one k-step is 32 packed FMAs (fma.rn.f32x2, two lanes' worth per issue slot) on four 16-byte
// shared-memory reads; operands move from global memory to registers one chunk of 16 k ahead, and from there into the
// other half of a double-buffered shared tile, so a chunk costs one barrier.  Four tiles share the code: a block of 256
// threads is KG groups, and each group computes the whole BM x BN tile over its own 16 / KG of a chunk's k-steps; the
// groups' sums are added once at the end.  That keeps the 8 x 8 register blocks for tiles an eighth the size, which is
// what a problem with few output tiles (a 7 x 7 feature map, a weight gradient) needs to occupy the SMs.
// Measured: 48 to 52 TFLOP/s on 8192 x 4096 x 1024 (FMA pipe 72 % busy, shared memory 72 %), 40 to 47 on VGG-16's 3x3
// convolutions at batch 8, 12 to 28 on ResNet-50's at batch 7; a tile with 4 x 4 outputs per thread and no double
// buffering ran at 16 (VGG-16) and 10 (ResNet-50).
#include "pd_gemm.cuh"
#include "pd_sm100_ptx.cuh"
#include <mutex>

namespace {

constexpr int kThreads = 256;
constexpr int kSplitUnit = 32;                       // K slices start at multiples of this

struct SParams {
  const float* a; long long a_rows, lda; int a_major, a_vec;
  const float* b; long long b_rows, ldb; int b_major, b_vec;
  int M, N, K, num_taps;
  int a_row0, a_col0, b_row0, b_col0;
  int a_tap_row[PD_MAX_TAPS], a_tap_col[PD_MAX_TAPS];
  int b_tap_row[PD_MAX_TAPS], b_tap_col[PD_MAX_TAPS];
  int z_b_row[PD_MAX_TAPS]; long long z_out_col;
  int split_k, k_per_split;
  float* out; long long ldo; int atomic;
  const float* bias; int relu; int pad_hp, pad_wp;
  const float* relu_aux; long long ld_aux;
  int* err;
};

// Four neighbouring outputs of row m: bias, ReLU, masks, store or fp32 atomic add.
__device__ __forceinline__ void store4(const SParams& p, const float* v, int m, int n, int z, bool border) {
  float* o = p.out + (long long)m * p.ldo + (long long)z * p.z_out_col + n;
  float w[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float x = v[j];
    if (n + j < p.N) {
      if (p.bias) x += p.bias[n + j];
      if (p.relu) x = fmaxf(x, 0.f);
      if (p.relu_aux && !(p.relu_aux[(long long)m * p.ld_aux + n + j] > 0.f)) x = 0.f;
    }
    w[j] = border ? 0.f : x;
  }
  if (n + 4 <= p.N && (((uintptr_t)o) & 15) == 0) {
    if (p.atomic)
      asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(o), "f"(w[0]), "f"(w[1]), "f"(w[2]), "f"(w[3])
                   : "memory");
    else
      *reinterpret_cast<float4*>(o) = make_float4(w[0], w[1], w[2], w[3]);
  } else {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < p.N) {
        if (p.atomic) atomicAdd(o + j, w[j]);
        else o[j] = w[j];
      }
  }
}

__device__ __forceinline__ unsigned long long dup2(float a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
  return r;
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 halves(unsigned long long v) {
  float2 f;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
  return f;
}

// One operand's part of a chunk: ROWS (m or n) x BK (k) values, as ROWS * BK / 4 / 256 float4 per thread.  The smaller
// tiles do few FMAs per chunk and keep their addresses in registers from chunk to chunk (KEEP); the largest has no
// registers left for that and works them out anew, in the shadow of twice the FMAs.
template <int ROWS, int BK, bool KEEP>
struct Loader {
  static constexpr int kQuads = ROWS * BK / 4 / kThreads;
  float4 v[kQuads];
  const float* src[KEEP ? kQuads : 1];
  const float* base;
  long long ld, rows, first;      // first: row of the operand that row 0 (k-major) / k 0 (row-major) of the tile is
  int limit;                      // rows (k-major) / columns (row-major) of the tile that exist
  int have;                       // KEEP, k-major: bit q set = the row of quad q exists

  __device__ __forceinline__ static int krow(int q) { return ((threadIdx.x + q * kThreads) >> 1) % ROWS; }
  __device__ __forceinline__ static int kcol(int q) {
    const int id = threadIdx.x + q * kThreads;
    return (id & 1) * 4 + (id >> 1) / ROWS * 8;
  }
  __device__ __forceinline__ static int mrow(int q) { return (threadIdx.x + q * kThreads) / (ROWS / 4); }
  __device__ __forceinline__ static int mcol() { return (threadIdx.x % (ROWS / 4)) * 4; }

  __device__ __forceinline__ void tap(bool k_major, const float* from, long long ld_, long long rows_, long long first_,
                                      int limit_) {
    base = from; ld = ld_; rows = rows_; first = first_; limit = limit_;
    if constexpr (KEEP) {
      have = 0;
#pragma unroll
      for (int q = 0; q < kQuads; ++q) {
        if (k_major) {
          const long long gr = first + krow(q);
          if (krow(q) < limit && gr >= 0 && gr < rows) have |= 1 << q;
          src[q] = base + gr * ld + kcol(q);
        } else {
          src[q] = base + (first + mrow(q)) * ld + mcol();
        }
      }
    }
  }
  // k contiguous in memory: two neighbouring lanes read one 32-byte sector of a row; the transposed stores into
  // [k][row] (row stride ROWS + 4 floats) then hit 32 different banks.
  __device__ __forceinline__ void load_k(int k0, int k_end, int vec) {
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
      const int k = k0 + kcol(q);
      const float* s;
      bool ok;
      if constexpr (KEEP) {
        s = src[q] + k0;
        ok = (have >> q) & 1;
      } else {
        const long long gr = first + krow(q);
        ok = krow(q) < limit && gr >= 0 && gr < rows;
        s = base + gr * ld + k;
      }
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (ok) {
        if (vec && k + 4 <= k_end) {
          f = __ldg(reinterpret_cast<const float4*>(s));
        } else {
          if (k < k_end) f.x = s[0];
          if (k + 1 < k_end) f.y = s[1];
          if (k + 2 < k_end) f.z = s[2];
          if (k + 3 < k_end) f.w = s[3];
        }
      }
      v[q] = f;
    }
  }
  __device__ __forceinline__ void store_k(float (*tile)[ROWS + 4]) const {
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
      const int row = krow(q), k = kcol(q);
      tile[k][row] = v[q].x; tile[k + 1][row] = v[q].y; tile[k + 2][row] = v[q].z; tile[k + 3][row] = v[q].w;
    }
  }
  // rows contiguous in memory: 16-byte reads and stores along them
  __device__ __forceinline__ void load_m(int k0, int k_end, int vec) {
    const int m = mcol();
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
      const int k = k0 + mrow(q);
      const long long gr = first + k;
      const float* s;
      if constexpr (KEEP) s = src[q] + (long long)k0 * ld;
      else s = base + gr * ld + m;
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < k_end && gr >= 0 && gr < rows) {
        if (vec && m + 4 <= limit) {
          f = __ldg(reinterpret_cast<const float4*>(s));
        } else {
          if (m < limit) f.x = s[0];
          if (m + 1 < limit) f.y = s[1];
          if (m + 2 < limit) f.z = s[2];
          if (m + 3 < limit) f.w = s[3];
        }
      }
      v[q] = f;
    }
  }
  __device__ __forceinline__ void store_m(float (*tile)[ROWS + 4]) const {
#pragma unroll
    for (int q = 0; q < kQuads; ++q) *reinterpret_cast<float4*>(&tile[mrow(q)][mcol()]) = v[q];
  }
};

template <int BM, int BN, int BK>
struct Tiles {
  float a[2][BK][BM + 4];
  float b[2][BK][BN + 4];
};

template <int BM, int BN, int KG, int BK>
__global__ void __launch_bounds__(kThreads, 2)
gemm_simt_kernel(const __grid_constant__ SParams p) {
  static_assert(BM * BN * KG == 64 * kThreads, "8 x 8 outputs per thread");
  constexpr int kGroup = kThreads / KG;              // threads of a k-group
  constexpr int kTx = BN / 8;                        // threads across n
  extern __shared__ __align__(16) unsigned char smem[];
  Tiles<BM, BN, BK>& t = *reinterpret_cast<Tiles<BM, BN, BK>*>(smem);
  float* part = reinterpret_cast<float*>(smem);      // after the last chunk: one group's sums
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int z = blockIdx.z / p.split_k, split = blockIdx.z % p.split_k;
  const int k_begin = split * p.k_per_split;
  const int k_end = min(p.K, k_begin + p.k_per_split);
  const int chunks = (k_end - k_begin + BK - 1) / BK;
  const int total = chunks * p.num_taps;
  const int group = threadIdx.x / kGroup, lid = threadIdx.x % kGroup;
  // a warp covers 4 x 8 threads (or 8 x 4, in the narrowest tile): one shared-memory wavefront per operand read
  const int warp = lid >> 5, lane = lid & 31;
  constexpr int kLx = kTx < 8 ? kTx : 8, kLy = 32 / kLx, kWarpsX = kTx / kLx;
  const int tx = (warp % kWarpsX) * kLx + lane % kLx, ty = (warp / kWarpsX) * kLy + lane / kLx;

  unsigned long long acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

  Loader<BM, BK, (KG > 1)> la;
  Loader<BN, BK, (KG > 1)> lb;
  int tap = -1, chunk = chunks - 1;
  auto fetch = [&]() {
    if (++chunk == chunks) {
      chunk = 0;
      ++tap;
      const long long ar = (long long)p.a_row0 + p.a_tap_row[tap], br = (long long)p.b_row0 + p.b_tap_row[tap] + p.z_b_row[z];
      const int ac = p.a_col0 + p.a_tap_col[tap], bc = p.b_col0 + p.b_tap_col[tap];
      if (p.a_major == 0) la.tap(true, p.a + ac, p.lda, p.a_rows, ar + m0, p.M - m0);
      else la.tap(false, p.a + ac + m0, p.lda, p.a_rows, ar, p.M - m0);
      if (p.b_major == 0) lb.tap(true, p.b + bc, p.ldb, p.b_rows, br + n0, p.N - n0);
      else lb.tap(false, p.b + bc + n0, p.ldb, p.b_rows, br, p.N - n0);
    }
    const int k0 = k_begin + chunk * BK;
    if (p.a_major == 0) la.load_k(k0, k_end, p.a_vec); else la.load_m(k0, k_end, p.a_vec);
    if (p.b_major == 0) lb.load_k(k0, k_end, p.b_vec); else lb.load_m(k0, k_end, p.b_vec);
  };
  auto put = [&](int buf) {
    if (p.a_major == 0) la.store_k(t.a[buf]); else la.store_m(t.a[buf]);
    if (p.b_major == 0) lb.store_k(t.b[buf]); else lb.store_m(t.b[buf]);
  };

  fetch();
  put(0);
  __syncthreads();
  for (int it = 0; it < total; ++it) {
    const int buf = it & 1;
    if (it + 1 < total) fetch();
#pragma unroll
    for (int s = 0; s < BK / KG; ++s) {
      const int kk = group * (BK / KG) + s;
      const float4 a0 = *reinterpret_cast<const float4*>(&t.a[buf][kk][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&t.a[buf][kk][BM / 2 + ty * 4]);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&t.b[buf][kk][tx * 4]);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&t.b[buf][kk][BN / 2 + tx * 4]);
      const float av[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const unsigned long long d = dup2(av[i]);
        fma2(acc[i][0], d, b0.x);
        fma2(acc[i][1], d, b0.y);
        fma2(acc[i][2], d, b1.x);
        fma2(acc[i][3], d, b1.y);
      }
    }
    if (it + 1 < total) put(buf ^ 1);
    __syncthreads();
  }

  float v[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = halves(acc[i][j]);
      v[i][2 * j] = f.x;
      v[i][2 * j + 1] = f.y;
    }
  if constexpr (KG > 1) {
    for (int g = 1; g < KG; ++g) {
      if (group == g) {
#pragma unroll
        for (int i = 0; i < 64; ++i) part[i * kGroup + lid] = v[i >> 3][i & 7];
      }
      __syncthreads();
      if (group == 0) {
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i >> 3][i & 7] += part[i * kGroup + lid];
      }
      __syncthreads();
    }
    if (group != 0) return;
  }

#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const int m = m0 + (i >> 2) * (BM / 2) + ty * 4 + (i & 3);
    if (m >= p.M) continue;
    bool border = false;
    if (p.pad_wp > 0) {
      const int row = m / p.pad_wp, wp = m - row * p.pad_wp, hp = row % p.pad_hp;
      border = wp == 0 || wp == p.pad_wp - 1 || hp == 0 || hp == p.pad_hp - 1;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int n = n0 + h * (BN / 2) + tx * 4;
      if (n >= p.N) continue;
      store4(p, &v[i][h * 4], m, n, z, border);
    }
  }
}

// ---- tensor cores: three bf16 parts per fp32 value -------------------------------------------------------------------
// The FMA pipe ends at 74 TFLOP/s; the tensor pipe multiplies bf16 exactly into fp32 at twenty times that rate.  An fp32
// value is the sum of three bf16 values (8 + 8 + 8 significant bits), x = h + m + l, and a product of two such sums is
// taken as the six partial products hh, hm, mh, mm, hl, lh; what is left out (ml, lm, ll) is below 2^-25 of the product.
// The tensor core does not round its accumulator to nearest, so it never adds up more than one chunk of 64 k: chunk sums
// leave tensor memory and are added in registers, rounded to nearest.  Relative error against 64 bits (2-norm), FMA tiles
// -> this: K = 64 1.4e-7 -> 0.8e-7, 576 4.3e-7 -> 1.0e-7, 4608 1.2e-6 -> 1.8e-7, 25088 2.8e-6 -> 3.7e-7.  (A part below
// 2^-133, bf16's smallest step, is lost: values of less than 2^-109 are not held to all their bits.)
//
// One block per SM, a 128 x 128 tile: 8 warps read fp32 operands from global memory into registers, one chunk ahead,
// split them and store the six 128 x 64 planes (128-byte swizzle, either major order; 96 KB per stage, two stages); 8
// warps drain the accumulators, double-buffered, and two of them issue the MMAs, three products each into accumulators
// of their own.  Bound by the splitting warps' instructions (1.8 us per chunk, of which L2 takes 1.5 us: 64 KB a block at
// 6.2 TB/s).  Planes made by a pass of their own would save the splitting and load half as much again from L2.
// Measured: 4096 x 4096 x 4096 166 TFLOP/s (FMA tiles 50), VGG-16's 3x3 convolutions at batch 8 55 to 145 (40 to 47).
// A tile that meets a value of 2^127 or more, an infinity or a NaN (whose parts would multiply to NaN where fp32 keeps an
// infinity) is worked out again with plain FMAs.
constexpr int kSplitThreads = 16 * 32;               // warps 0-7 drain (0 and 4 also issue), 8-15 split: 128 registers each
constexpr uint32_t kPlane = 128 * 64 * 2;            // one part of one operand: 16 KiB
constexpr uint32_t kSplitStage = 6 * kPlane;
constexpr int kSplitSmem = 2 * kSplitStage + 1024;

// x = h + m + l, each rounded to nearest; l takes what is left, which has at most eight bits.
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ uint32_t round2(unsigned long long v) {
  const float2 f = halves(v);
  uint32_t r;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(f.y), "f"(f.x));
  return r;
}
__device__ __forceinline__ unsigned long long minus2(unsigned long long v, uint32_t h) {
  fma2(v, pack2(__uint_as_float(h << 16), __uint_as_float(h & 0xffff0000u)), pack2(-1.f, -1.f));
  return v;
}
__device__ __forceinline__ void split_pair(float x, float y, uint32_t& h, uint32_t& m, uint32_t& l) {
  unsigned long long v = pack2(x, y);
  h = round2(v);
  v = minus2(v, h);
  m = round2(v);
  l = round2(minus2(v, m));
}

// One operand's chunk: 128 rows x 64 k (k-major) or 64 k x 128 columns (row-major), eight float4 per thread.
struct SplitLoader {
  float4 v[8];
  const float* src;               // of the thread's first quad
  long long step, ld, first, rows;
  int have, limit;

  __device__ __forceinline__ void tap(int major, int tid, const float* from, long long ld_, long long rows_,
                                      long long first_, int limit_) {
    ld = ld_; rows = rows_; first = first_; limit = limit_;
    have = 0;
    if (major == 0) {             // 16 lanes read the 256 bytes of a row
      const int r0 = tid >> 4;
      src = from + (first + r0) * ld + (tid & 15) * 4;
      step = 16 * ld;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const long long gr = first + r0 + 16 * i;
        if (r0 + 16 * i < limit && gr >= 0 && gr < rows) have |= 1 << i;
      }
    } else {                      // a warp reads the 512 bytes of a k
      src = from + (first + (tid >> 5)) * ld + (tid & 31) * 4;
      step = 8 * ld;
    }
  }
  __device__ __forceinline__ void load(int major, int tid, int k0, int k_end, int vec) {
    if (major == 0) {
      const int k = k0 + (tid & 15) * 4;
      const float* s = src + k0;
      if (vec && k + 4 <= k_end) {
#pragma unroll
        for (int i = 0; i < 8; ++i, s += step)
          v[i] = (have >> i) & 1 ? __ldg(reinterpret_cast<const float4*>(s)) : make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i, s += step) {
          float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
          if ((have >> i) & 1) {
            if (k < k_end) f.x = s[0];
            if (k + 1 < k_end) f.y = s[1];
            if (k + 2 < k_end) f.z = s[2];
            if (k + 3 < k_end) f.w = s[3];
          }
          v[i] = f;
        }
      }
    } else {
      const int m = (tid & 31) * 4, kr = tid >> 5;
      const float* s = src + (long long)k0 * ld;
      // rows of this thread that exist: k below k_end, row inside the operand
      const long long lo = -(first + k0 + kr), hi = min((long long)(k_end - k0 - kr), rows - (first + k0 + kr));
      if (vec && m + 4 <= limit) {
#pragma unroll
        for (int i = 0; i < 8; ++i, s += step)
          v[i] = 8 * i >= lo && 8 * i < hi ? __ldg(reinterpret_cast<const float4*>(s)) : make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
#pragma unroll
        for (int i = 0; i < 8; ++i, s += step) {
          float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
          if (8 * i >= lo && 8 * i < hi) {
            if (m < limit) f.x = s[0];
            if (m + 1 < limit) f.y = s[1];
            if (m + 2 < limit) f.z = s[2];
            if (m + 3 < limit) f.w = s[3];
          }
          v[i] = f;
        }
      }
    }
  }
  // -> planes at `dst` (h), dst + 2 planes (m), dst + 4 planes (l); returns the largest |h| seen, as two bf16 halves.
  // A thread's rows are 16 (k-major) or 8 apart, so they share one swizzle pattern.
  template <int STEP>
  __device__ __forceinline__ uint32_t store_rows(uint32_t dst) const {
    uint32_t most = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      uint2 h, m, l;
      split_pair(v[i].x, v[i].y, h.x, m.x, l.x);
      split_pair(v[i].z, v[i].w, h.y, m.y, l.y);
      most = __vmaxu2(most, __vmaxu2(h.x & 0x7fff7fffu, h.y & 0x7fff7fffu));
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + i * STEP), "r"(h.x), "r"(h.y) : "memory");
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + i * STEP + 2 * kPlane), "r"(m.x), "r"(m.y) : "memory");
      asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + i * STEP + 4 * kPlane), "r"(l.x), "r"(l.y) : "memory");
    }
    return most;
  }
  __device__ __forceinline__ uint32_t store(int major, int tid, uint32_t dst) const {
    if (major == 0) {
      const int r = tid >> 4, c4 = tid & 15;
      return store_rows<16 * 128>(dst + (uint32_t)(r * 128 + (((c4 >> 1) ^ (r & 7)) << 4) + ((c4 & 1) << 3)));
    }
    const int r = tid >> 5, c4 = tid & 31;
    return store_rows<8 * 128>(dst + (uint32_t)((c4 >> 4) * (int)pd_sm100::kAtomBytes + r * 128 +
                                                ((((c4 & 15) >> 1) ^ (r & 7)) << 4) + ((c4 & 1) << 3)));
  }
};

__device__ __noinline__ float plain_sum(const SParams& p, int m, int n, int z, int k_begin, int k_end) {
  float x = 0.f;
  for (int tap = 0; tap < p.num_taps; ++tap) {
    const long long ar = (long long)p.a_row0 + p.a_tap_row[tap];
    const long long br = (long long)p.b_row0 + p.b_tap_row[tap] + p.z_b_row[z];
    const int ac = p.a_col0 + p.a_tap_col[tap], bc = p.b_col0 + p.b_tap_col[tap];
    for (int k = k_begin; k < k_end; ++k) {
      const long long ra = ar + (p.a_major ? k : m), rb = br + (p.b_major ? k : n);
      const float av = ra >= 0 && ra < p.a_rows ? p.a[ra * p.lda + ac + (p.a_major ? m : k)] : 0.f;
      const float bv = rb >= 0 && rb < p.b_rows ? p.b[rb * p.ldb + bc + (p.b_major ? n : k)] : 0.f;
      x = fmaf(av, bv, x);
    }
  }
  return x;
}

__device__ __forceinline__ void mbar_arrive_local(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

__global__ void __launch_bounds__(kSplitThreads, 1)
gemm_split_kernel(const __grid_constant__ SParams p) {
  using namespace pd_sm100;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ __align__(8) uint64_t full_bar[2], empty_bar[2], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_holder;
  __shared__ int plain;
  const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
  const uint32_t stage0 = (smem_u32(smem) + 1023u) & ~1023u;
  const int m0 = blockIdx.x * 128, n0 = blockIdx.y * 128;
  const int z = blockIdx.z / p.split_k, split = blockIdx.z % p.split_k;
  const int k_begin = split * p.k_per_split, k_end = min(p.K, k_begin + p.k_per_split);
  const int chunks = (k_end - k_begin + 63) / 64, total = chunks * p.num_taps;

  if (threadIdx.x == 0) {
    plain = 0;
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 8);
      mbar_init(smem_u32(&empty_bar[s]), 2);
      mbar_init(smem_u32(&acc_full[s]), 2);
      mbar_init(smem_u32(&acc_empty[s]), 8);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  if (warp == 8) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 ::"r"(smem_u32(&tmem_holder)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_holder;

  if (warp >= 8) {
    // ---------------------------------- operands ----------------------------------
    const int tid = threadIdx.x - 8 * 32;
    SplitLoader a, b;
    int tap = -1, chunk = chunks - 1;
    auto advance = [&]() {
      if (++chunk == chunks) {
        chunk = 0;
        ++tap;
        const long long ar = (long long)p.a_row0 + p.a_tap_row[tap];
        const long long br = (long long)p.b_row0 + p.b_tap_row[tap] + p.z_b_row[z];
        const int ac = p.a_col0 + p.a_tap_col[tap], bc = p.b_col0 + p.b_tap_col[tap];
        a.tap(p.a_major, tid, p.a + ac + (p.a_major ? m0 : 0), p.lda, p.a_rows, ar + (p.a_major ? 0 : m0), p.M - m0);
        b.tap(p.b_major, tid, p.b + bc + (p.b_major ? n0 : 0), p.ldb, p.b_rows, br + (p.b_major ? 0 : n0), p.N - n0);
      }
    };
    uint32_t most = 0u;              // largest magnitudes met, bf16 pair
    advance();
    a.load(p.a_major, tid, k_begin, k_end, p.a_vec);
    b.load(p.b_major, tid, k_begin, k_end, p.b_vec);
    for (int it = 0; it < total; ++it) {
      const int s = it & 1;
      if (!mbar_wait(smem_u32(&empty_bar[s]), ((uint32_t)(it >> 1) & 1u) ^ 1u, p.err, 1)) break;
      const uint32_t dst = stage0 + (uint32_t)s * kSplitStage;
      // the next chunk of one operand is on its way while the other one is split
      const bool more = it + 1 < total;
      most = __vmaxu2(most, a.store(p.a_major, tid, dst));
      if (more) advance();
      const int k0 = k_begin + chunk * 64;
      if (more) a.load(p.a_major, tid, k0, k_end, p.a_vec);
      most = __vmaxu2(most, b.store(p.b_major, tid, dst + kPlane));
      if (max(most & 0xffffu, most >> 16) >= 0x7f00u) plain = 1;
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_local(smem_u32(&full_bar[s]));
      if (more) b.load(p.b_major, tid, k0, k_end, p.b_vec);
    }
  } else {
    // ------------------------------- MMAs, drain, epilogue -------------------------------
    // planes: A h m l at 0, 2, 4, B h m l at 1, 3, 5.  Small products first, so that only the last four MMAs of a chunk
    // round at the size of the result.  Warps 0 and 4 issue the chunk after the one that they drain next.
    const bool issuer = (warp & 3) == 0;
    const int me = warp >> 2;
    const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(p.a_major ? 1 : 0) << 15) |
                           ((uint32_t)(p.b_major ? 1 : 0) << 16) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
    const uint64_t da = make_desc(stage0, p.a_major), db = make_desc(stage0, p.b_major);
    const uint32_t a_hi = (uint32_t)(da >> 32), b_hi = (uint32_t)(db >> 32);
    const uint32_t adv_a = p.a_major ? 128u : 2u, adv_b = p.b_major ? 128u : 2u;
    constexpr uint32_t P = kPlane >> 4;
    const uint32_t pa[3] = {me ? 4 * P : 0, 2 * P, 0};                        // lh, mh, hm  |  hl, mm, hh
    const uint32_t pb[3] = {me ? 1 * P : 5 * P, me ? 1 * P : 3 * P, me ? 3 * P : 1 * P};
    auto issue = [&](int it) {
      const int s = it & 1;
      const uint32_t par = (uint32_t)(it >> 1) & 1u;
      if (!mbar_wait_warp(smem_u32(&acc_empty[s]), par ^ 1u, p.err, 2)) return false;
      if (!mbar_wait_warp(smem_u32(&full_bar[s]), par, p.err, 2)) return false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + (uint32_t)(s * 256 + me * 128);
      const uint32_t so = (uint32_t)s * (kSplitStage >> 4);
      const uint32_t a_lo = (uint32_t)da + so, b_lo = (uint32_t)db + so;
#pragma unroll
      for (int q = 0; q < 3; ++q)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          if (q == 0 && kk == 0) umma_lo_elect<1, 0>(acc, a_lo + pa[q], a_hi, b_lo + pb[q], b_hi, idesc, 0u);
          else umma_lo_elect<1, 1>(acc, a_lo + pa[q] + kk * adv_a, a_hi, b_lo + pb[q] + kk * adv_b, b_hi, idesc, 1u);
        }
      umma_commit_elect(smem_u32(&empty_bar[s]));
      umma_commit_elect(smem_u32(&acc_full[s]));
      return true;
    };
    const int row = (warp & 3) * 32 + lane, col0 = (warp >> 2) * 64;
    float c[64];
#pragma unroll
    for (int j = 0; j < 64; ++j) c[j] = 0.f;
    bool ok = !issuer || issue(0);
    for (int it = 0; it < total && ok; ++it) {
      const int s = it & 1;
      if (issuer && it + 1 < total) ok = issue(it + 1);
      if (!ok) break;
      ok = mbar_wait_warp(smem_u32(&acc_full[s]), (uint32_t)(it >> 1) & 1u, p.err, 3);
      if (!ok) break;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t acc = tmem + (uint32_t)(s * 256 + col0) + ((uint32_t)((warp & 3) * 32) << 16);
#pragma unroll
      for (int h = 0; h < 4; ++h) {
        uint32_t r0[16], r1[16];
        tmem_ld16(acc + h * 16, r0);
        tmem_ld16(acc + 128 + h * 16, r1);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) c[h * 16 + j] += __uint_as_float(r0[j]) + __uint_as_float(r1[j]);
      }
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_local(smem_u32(&acc_empty[s]));
    }
    const int m = m0 + row;
    if (ok && m < p.M) {
      if (*(volatile int*)&plain) {
        for (int j = 0; j < 64 && n0 + col0 + j < p.N; ++j) {
          const float x = plain_sum(p, m, n0 + col0 + j, z, k_begin, k_end);
#pragma unroll
          for (int q = 0; q < 64; ++q)
            if (q == j) c[q] = x;
        }
      }
      bool border = false;
      if (p.pad_wp > 0) {
        const int r = m / p.pad_wp, wp = m - r * p.pad_wp, hp = r % p.pad_hp;
        border = wp == 0 || wp == p.pad_wp - 1 || hp == 0 || hp == p.pad_hp - 1;
      }
#pragma unroll
      for (int j = 0; j < 64; j += 4) {
        const int n = n0 + col0 + j;
        if (n < p.N) store4(p, &c[j], m, n, z, border);
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 8) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  }
}

// ---- a handful of rows: Linear forward and data gradient at a batch of at most eight --------------------------------
// The weights are the whole cost (411 MB for the first Linear layer of VGG-16, 64 us at the measured copy rate) and a
// 64-row tile would waste 7/8 of its FMAs and, with one block per 64 columns, most of the chip.  The weights are read
// once, straight into registers; the few rows of `a` come through the L1 cache.
constexpr int kFewRows = 8;

__device__ __forceinline__ float few_epilogue(const SParams& p, float x, int m, int n) {
  if (p.bias) x += p.bias[n];
  if (p.relu) x = fmaxf(x, 0.f);
  if (p.relu_aux && !(p.relu_aux[(long long)m * p.ld_aux + n] > 0.f)) x = 0.f;
  return x;
}

// out[m, n] = sum_k a[m, k] b[n, k]: a block owns eight rows of b, four per half of its warps; the four warps of a half
// take every fourth 128-wide piece of k.  4096 x 25088 weights: 1293 us with the tiles above.
__global__ void __launch_bounds__(kThreads, 2)
few_rows_nt_kernel(const __grid_constant__ SParams p) {
  constexpr int R = 4, S = 4;
  __shared__ float part[kThreads / 32][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n0 = (blockIdx.x * 2 + warp / S) * R;
  float acc[kFewRows][R];
#pragma unroll
  for (int m = 0; m < kFewRows; ++m)
#pragma unroll
    for (int r = 0; r < R; ++r) acc[m][r] = 0.f;
  const float* b[R];
#pragma unroll
  for (int r = 0; r < R; ++r) b[r] = p.b + (long long)min(n0 + r, p.N - 1) * p.ldb;
#pragma unroll 2
  for (int k = ((warp % S) * 32 + lane) * 4; k < p.K; k += S * 128) {
    float4 w[R];
#pragma unroll
    for (int r = 0; r < R; ++r) w[r] = __ldcs(reinterpret_cast<const float4*>(b[r] + k));
#pragma unroll
    for (int m = 0; m < kFewRows; ++m) {
      const float4 x = __ldg(reinterpret_cast<const float4*>(p.a + (long long)min(m, p.M - 1) * p.lda + k));
#pragma unroll
      for (int r = 0; r < R; ++r)
        acc[m][r] = fmaf(x.w, w[r].w, fmaf(x.z, w[r].z, fmaf(x.y, w[r].y, fmaf(x.x, w[r].x, acc[m][r]))));
    }
  }
#pragma unroll
  for (int m = 0; m < kFewRows; ++m)
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const float x = pd_warp_sum(acc[m][r]);
      if (lane == m * R + r) part[warp][lane] = x;
    }
  __syncthreads();
  if (warp % S == 0) {
    const int m = lane / R, n = n0 + lane % R;
    if (m < p.M && n < p.N) {
      float x = part[warp][lane];
#pragma unroll
      for (int w = 1; w < S; ++w) x += part[warp + w][lane];
      p.out[(long long)m * p.ldo + n] = few_epilogue(p, x, m, n);
    }
  }
}

// out[m, n] = sum_k a[m, k] b[k, n]: a block owns 32 columns, its 16 warps a sixteenth of k each.
__global__ void __launch_bounds__(512)
few_rows_nn_kernel(const __grid_constant__ SParams p) {
  constexpr int kWarps = 16;
  __shared__ float part[kWarps][kFewRows][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = blockIdx.x * 32 + lane;
  const int per = ((p.K + kWarps - 1) / kWarps + 3) / 4 * 4;
  const int k_begin = warp * per, k_end = min(p.K, k_begin + per);
  float acc[kFewRows];
#pragma unroll
  for (int m = 0; m < kFewRows; ++m) acc[m] = 0.f;
  const float* b = p.b + min(n, p.N - 1);
#pragma unroll 4
  for (int k = k_begin; k < k_end; k += 4) {         // K is a multiple of four
    float w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = __ldcs(b + (long long)(k + j) * p.ldb);
#pragma unroll
    for (int m = 0; m < kFewRows; ++m) {
      const float4 x = __ldg(reinterpret_cast<const float4*>(p.a + (long long)min(m, p.M - 1) * p.lda + k));
      acc[m] = fmaf(x.w, w[3], fmaf(x.z, w[2], fmaf(x.y, w[1], fmaf(x.x, w[0], acc[m]))));
    }
  }
#pragma unroll
  for (int m = 0; m < kFewRows; ++m) part[warp][m][lane] = acc[m];
  __syncthreads();
  if (warp < p.M && warp < kFewRows && n < p.N) {
    float x = 0.f;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) x += part[w][warp][lane];
    p.out[(long long)warp * p.ldo + n] = few_epilogue(p, x, warp, n);
  }
}

// 16-byte reads need every row start on a 16-byte boundary, tap and origin columns included.
int vectorised(const void* base, long long ld, int col0, const int* tap_col, int taps) {
  if (((uintptr_t)base & 15) || (ld & 3) || (col0 & 3)) return 0;
  for (int t = 0; t < taps; ++t)
    if (tap_col[t] & 3) return 0;
  return 1;
}

}  // namespace

namespace {

struct SimtTile {
  int bm, bn;
  double rate;                  // TFLOP/s of a problem that fills the chip with it (measured)
  int smem, threads;
  void (*kernel)(SParams);
};
template <int BM, int BN, int KG, int BK>
SimtTile simt_tile(double rate) {
  const int tiles = (int)sizeof(Tiles<BM, BN, BK>), part = KG > 1 ? BM * BN * 4 : 0;
  return {BM, BN, rate, tiles > part ? tiles : part, kThreads, gemm_simt_kernel<BM, BN, KG, BK>};
}
const SimtTile kTiles[5] = {{128, 128, 0., kSplitSmem, kSplitThreads, gemm_split_kernel},
                            simt_tile<128, 128, 1, 16>(49.), simt_tile<128, 64, 2, 16>(40.),
                            simt_tile<64, 64, 4, 32>(37.), simt_tile<64, 32, 8, 32>(28.)};
constexpr double kSplitChunkUs = 1.8, kSplitTileUs = 5.;        // measured, K from 576 to 25088
std::mutex g_simt_mu;
bool g_simt_ready[64];

// Estimated time in us of `blocks` blocks of a tile with k steps each: two of them share an SM; one alone gets three
// quarters of the SM's rate out of it (tensor-core tiles: one per SM, a fixed time per chunk); filling the pipeline and the epilogue cost about 3.6 us per block of an SM whatever
// the tile.  (Within a tenth of the measured times of ResNet-50's layers at batch 7, K from 64 to 4608.)  The smaller
// tiles lose to the larger ones on rate and win where the larger ones leave SMs idle in the last, often only, round.
double tile_time(const SimtTile& t, long long blocks, double k) {
  const long long sms = pd_num_sms(), n = (blocks + sms - 1) / sms;
  if (t.kernel == gemm_split_kernel) return (double)n * (kSplitChunkUs * ((k + 63.) / 64.) + kSplitTileUs);
  const double per_k = 2. * t.bm * t.bn / (t.rate * 1e6 / sms) * ((double)(n - n % 2) + (double)(n % 2) / 0.75);
  return per_k * k + 3.6 * n;
}
const SimtTile& pick_tile(int M, int N, long long outer, double k, double* time = nullptr) {
  const SimtTile* best = nullptr;
  double best_time = 0.;
  for (const SimtTile& t : kTiles) {
    const double e = tile_time(t, (long long)((M + t.bm - 1) / t.bm) * ((N + t.bn - 1) / t.bn) * outer, k);
    if (!best || e < best_time) { best = &t; best_time = e; }
  }
  if (time) *time = best_time;
  return *best;
}

}  // namespace

// K slices for a weight gradient of num_z outputs [M, N] over k units of 64: the count that takes the least time with the
// tile picked for it.  Slices of one output add up at the same addresses, which takes about 0.3 us a slice.
int pd_gemm_simt_split(int M, int N, int num_z, int units) {
  int best = 1;
  double best_time = 1e300;
  for (int s = 1; s <= 128 && s <= units; ++s) {
    const int per = (units + s - 1) / s, used = (units + per - 1) / per;
    if (used != s) continue;
    double time;
    pick_tile(M, N, (long long)num_z * used, 64. * per, &time);
    if (used > 1) time += 2. + 0.3 * used;
    if (time < best_time) { best_time = time; best = used; }
  }
  return best;
}

int pd_gemm_launch_simt(const PdGemm& g, cudaStream_t stream) {
  PD_REQUIRE(g.dtype == PD_F32 && g.out_dtype == PD_F32, "simt gemm: operands and output must be fp32");
  PD_REQUIRE(g.bias == nullptr || g.bias_dtype == PD_F32, "simt gemm: bias must be fp32");
  PD_REQUIRE(g.M > 0 && g.N > 0 && g.K > 0, "simt gemm: empty problem");
  PD_REQUIRE(g.num_taps >= 1 && g.num_taps <= PD_MAX_TAPS && g.num_z >= 1 && g.num_z <= PD_MAX_TAPS, "simt gemm: bad tap/z count");
  PD_REQUIRE(g.split_k >= 1 && (g.split_k == 1 || g.atomic), "simt gemm: split_k needs the atomic epilogue");
  SParams p;
  memset(&p, 0, sizeof(p));
  p.a = (const float*)g.a; p.a_rows = g.a_rows; p.lda = g.lda; p.a_major = g.a_major;
  p.b = (const float*)g.b; p.b_rows = g.b_rows; p.ldb = g.ldb; p.b_major = g.b_major;
  p.M = g.M; p.N = g.N; p.K = g.K; p.num_taps = g.num_taps;
  p.a_row0 = g.a_row0; p.a_col0 = g.a_col0; p.b_row0 = g.b_row0; p.b_col0 = g.b_col0;
  for (int t = 0; t < PD_MAX_TAPS; ++t) {
    p.a_tap_row[t] = g.a_tap_row[t]; p.a_tap_col[t] = g.a_tap_col[t];
    p.b_tap_row[t] = g.b_tap_row[t]; p.b_tap_col[t] = g.b_tap_col[t];
    p.z_b_row[t] = g.z_b_row[t];
  }
  p.a_vec = vectorised(g.a, g.lda, g.a_col0, g.a_tap_col, g.num_taps);
  p.b_vec = vectorised(g.b, g.ldb, g.b_col0, g.b_tap_col, g.num_taps);
  p.z_out_col = g.z_out_col;
  const int kblocks = (g.K + kSplitUnit - 1) / kSplitUnit;
  int split = g.split_k > kblocks ? kblocks : g.split_k;
  const int per = (kblocks + split - 1) / split;
  split = (kblocks + per - 1) / per;
  p.split_k = split; p.k_per_split = per * kSplitUnit;
  p.out = (float*)g.out; p.ldo = g.ldo; p.atomic = g.atomic;
  p.bias = (const float*)g.bias; p.relu = g.relu; p.pad_hp = g.pad_hp; p.pad_wp = g.pad_wp;
  p.relu_aux = (const float*)g.relu_aux; p.ld_aux = g.ld_aux;
  if (p.M <= kFewRows && !p.a_major && p.num_taps == 1 && g.num_z == 1 && split == 1 && !p.atomic && p.pad_wp == 0 &&
      p.a_row0 == 0 && p.b_row0 == 0 && p.a_col0 == 0 && p.b_col0 == 0 && p.a_tap_row[0] == 0 && p.b_tap_row[0] == 0 &&
      p.a_tap_col[0] == 0 && p.b_tap_col[0] == 0 && p.z_b_row[0] == 0 && p.a_vec && p.b_vec && p.K % 4 == 0 &&
      p.a_rows >= p.M && p.b_rows >= (p.b_major ? p.K : p.N)) {
    if (p.b_major) few_rows_nn_kernel<<<(p.N + 31) / 32, 512, 0, stream>>>(p);
    else few_rows_nt_kernel<<<(p.N + 7) / 8, kThreads, 0, stream>>>(p);
    PD_LAUNCH_CHECK("few_rows_kernel");
    return PD_OK;
  }
  const SimtTile& t = pick_tile(g.M, g.N, (long long)g.num_z * split, (double)p.num_taps * (p.k_per_split < p.K ? p.k_per_split : p.K));
  {
    int dev = 0;
    PD_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lk(g_simt_mu);
    if (dev >= 0 && dev < 64 && !g_simt_ready[dev]) {
      for (const SimtTile& k : kTiles)
        PD_CUDA(cudaFuncSetAttribute((const void*)k.kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, k.smem));
      g_simt_ready[dev] = true;
    }
  }
  dim3 grid((g.M + t.bm - 1) / t.bm, (g.N + t.bn - 1) / t.bn, g.num_z * split);
  PD_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "simt gemm: grid too large");
  {
    int rc = pd_gemm_error_word(&p.err);
    if (rc != PD_OK) return rc;
  }
  t.kernel<<<grid, t.threads, t.smem, stream>>>(p);
  PD_LAUNCH_CHECK("gemm_simt_kernel");
  return PD_OK;
}
