// fp32 contraction back end (CUDA cores).  Same problem description as the tcgen05 path; fp32 operands, products and sums
// throughout (tensor-core input rounding would not meet the 1e-3 tolerance of the fp32 configuration after 20 training
// steps).
//
// Bound by the FMA pipe: 128 lanes per SM, 74 TFLOP/s at 1.965 GHz.  Every thread keeps an 8 x 8 block of outputs in
// registers, so that one k-step is 32 packed FMAs (fma.rn.f32x2, two lanes' worth per issue slot) on four 16-byte
// shared-memory reads; operands move from global memory to registers one chunk of 16 k ahead, and from there into the
// other half of a double-buffered shared tile, so a chunk costs one barrier.  Three tiles share the code: a block of 256
// threads is KG groups, and each group computes the whole BM x BN tile over its own 16 / KG of a chunk's k-steps; the
// groups' sums are added once at the end.  That keeps the 8 x 8 register blocks for tiles a quarter the size, which is
// what a problem with few output tiles (a 7 x 7 feature map, a weight gradient) needs to occupy the SMs.
// The tile with 4 x 4 outputs per thread and no double buffering that this replaced ran at 16 TFLOP/s (VGG-16, batch 8).
#include "pd_gemm.cuh"

namespace {

constexpr int BK = 16, kThreads = 256;

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
};

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

// One operand's part of a chunk: ROWS (m or n) x 16 (k) values, as ROWS * 4 / 256 float4 per thread.
template <int ROWS>
struct Loader {
  static constexpr int kQuads = ROWS * 4 / kThreads;
  float4 v[kQuads];

  // k contiguous in memory: two neighbouring lanes read one 32-byte sector of a row; the transposed stores into
  // [k][row] (row stride ROWS + 4 floats) then hit 32 different banks.
  __device__ __forceinline__ void load_k(const float* base, long long ld, long long rows, long long row_first, int col,
                                         int limit, int k0, int k_end, int vec) {
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
      const int id = threadIdx.x + q * kThreads;
      const int row = (id >> 1) & (ROWS - 1), k = k0 + (id & 1) * 4 + (id >> 1) / ROWS * 8;
      const long long gr = row_first + row;
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < limit && gr >= 0 && gr < rows) {
        const float* src = base + gr * ld + col + k;
        if (vec && k + 4 <= k_end) {
          f = __ldg(reinterpret_cast<const float4*>(src));
        } else {
          if (k < k_end) f.x = src[0];
          if (k + 1 < k_end) f.y = src[1];
          if (k + 2 < k_end) f.z = src[2];
          if (k + 3 < k_end) f.w = src[3];
        }
      }
      v[q] = f;
    }
  }
  __device__ __forceinline__ void store_k(float (*tile)[ROWS + 4]) const {
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
      const int id = threadIdx.x + q * kThreads;
      const int row = (id >> 1) & (ROWS - 1), k = (id & 1) * 4 + (id >> 1) / ROWS * 8;
      tile[k][row] = v[q].x; tile[k + 1][row] = v[q].y; tile[k + 2][row] = v[q].z; tile[k + 3][row] = v[q].w;
    }
  }
  // rows contiguous in memory: 16-byte reads and stores along them
  __device__ __forceinline__ void load_m(const float* base, long long ld, long long rows, long long row_first, int col,
                                         int limit, int k0, int k_end, int vec) {
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
      const int id = threadIdx.x + q * kThreads;
      const int m = (id % (ROWS / 4)) * 4, k = k0 + id / (ROWS / 4);
      const long long gr = row_first + k;
      float4 f = make_float4(0.f, 0.f, 0.f, 0.f);
      if (k < k_end && gr >= 0 && gr < rows) {
        const float* src = base + gr * ld + col + m;
        if (vec && m + 4 <= limit) {
          f = __ldg(reinterpret_cast<const float4*>(src));
        } else {
          if (m < limit) f.x = src[0];
          if (m + 1 < limit) f.y = src[1];
          if (m + 2 < limit) f.z = src[2];
          if (m + 3 < limit) f.w = src[3];
        }
      }
      v[q] = f;
    }
  }
  __device__ __forceinline__ void store_m(float (*tile)[ROWS + 4]) const {
#pragma unroll
    for (int q = 0; q < kQuads; ++q) {
      const int id = threadIdx.x + q * kThreads;
      *reinterpret_cast<float4*>(&tile[id / (ROWS / 4)][(id % (ROWS / 4)) * 4]) = v[q];
    }
  }
};

template <int BM, int BN>
struct Tiles {
  float a[2][BK][BM + 4];
  float b[2][BK][BN + 4];
};

template <int BM, int BN, int KG>
__global__ void __launch_bounds__(kThreads, 2)
gemm_simt_kernel(const __grid_constant__ SParams p) {
  static_assert(BM * BN * KG == 64 * kThreads, "8 x 8 outputs per thread");
  constexpr int kGroup = kThreads / KG;              // threads of a k-group
  constexpr int kTx = BN / 8;                        // threads across n
  union Shared {
    Tiles<BM, BN> t;
    float part[KG > 1 ? kGroup * 64 : 1];
  };
  __shared__ __align__(16) Shared sh;
  const int m0 = blockIdx.x * BM, n0 = blockIdx.y * BN;
  const int z = blockIdx.z / p.split_k, split = blockIdx.z % p.split_k;
  const int k_begin = split * p.k_per_split;
  const int k_end = min(p.K, k_begin + p.k_per_split);
  const int chunks = (k_end - k_begin + BK - 1) / BK;
  const int total = chunks * p.num_taps;
  const int group = threadIdx.x / kGroup, lid = threadIdx.x % kGroup;
  // a warp covers 4 x 8 threads (32 m x 64 n of the tile): one shared-memory wavefront per operand read
  const int warp = lid >> 5, lane = lid & 31;
  constexpr int kWarpsX = kTx / 8;
  const int tx = (warp % kWarpsX) * 8 + (lane & 7), ty = (warp / kWarpsX) * 4 + (lane >> 3);

  unsigned long long acc[8][4];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

  Loader<BM> la;
  Loader<BN> lb;
  int tap = 0, chunk = 0;
  auto fetch = [&]() {
    const int k0 = k_begin + chunk * BK;
    if (p.a_major == 0)
      la.load_k(p.a, p.lda, p.a_rows, (long long)p.a_row0 + m0 + p.a_tap_row[tap], p.a_col0 + p.a_tap_col[tap], p.M - m0,
                k0, k_end, p.a_vec);
    else
      la.load_m(p.a, p.lda, p.a_rows, (long long)p.a_row0 + p.a_tap_row[tap], p.a_col0 + p.a_tap_col[tap] + m0, p.M - m0,
                k0, k_end, p.a_vec);
    const int zr = p.z_b_row[z];
    if (p.b_major == 0)
      lb.load_k(p.b, p.ldb, p.b_rows, (long long)p.b_row0 + n0 + p.b_tap_row[tap] + zr, p.b_col0 + p.b_tap_col[tap],
                p.N - n0, k0, k_end, p.b_vec);
    else
      lb.load_m(p.b, p.ldb, p.b_rows, (long long)p.b_row0 + p.b_tap_row[tap] + zr, p.b_col0 + p.b_tap_col[tap] + n0,
                p.N - n0, k0, k_end, p.b_vec);
    if (++chunk == chunks) { chunk = 0; ++tap; }
  };
  auto put = [&](int buf) {
    if (p.a_major == 0) la.store_k(sh.t.a[buf]); else la.store_m(sh.t.a[buf]);
    if (p.b_major == 0) lb.store_k(sh.t.b[buf]); else lb.store_m(sh.t.b[buf]);
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
      const float4 a0 = *reinterpret_cast<const float4*>(&sh.t.a[buf][kk][ty * 4]);
      const float4 a1 = *reinterpret_cast<const float4*>(&sh.t.a[buf][kk][BM / 2 + ty * 4]);
      const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&sh.t.b[buf][kk][tx * 4]);
      const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&sh.t.b[buf][kk][BN / 2 + tx * 4]);
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
        for (int i = 0; i < 64; ++i) sh.part[i * kGroup + lid] = v[i >> 3][i & 7];
      }
      __syncthreads();
      if (group == 0) {
#pragma unroll
        for (int i = 0; i < 64; ++i) v[i >> 3][i & 7] += sh.part[i * kGroup + lid];
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
      float* o = p.out + (long long)m * p.ldo + (long long)z * p.z_out_col + n;
      float w[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float x = v[i][h * 4 + j];
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

// Tile of an fp32 problem with `outer` independent outputs (z x K slices): the largest that still gives (nearly) every
// SM its two blocks; below that the tile that spreads the work over the most SMs (a block of the small tile takes a
// quarter of the large one's time).  Returns the tile's BM in *bm and BN in *bn.
static void pd_gemm_simt_tile(int M, int N, long long outer, int* bm, int* bn) {
  const long long full = 2ll * pd_num_sms() * 7 / 8;
  const auto tiles = [&](int tm, int tn) { return (long long)((M + tm - 1) / tm) * ((N + tn - 1) / tn) * outer; };
  if (N > 64 && M > 64 && tiles(128, 128) >= full) { *bm = 128; *bn = 128; return; }
  if (M > 64 && tiles(128, 64) >= full) { *bm = 128; *bn = 64; return; }
  *bm = 64; *bn = 64;
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
  int kblocks = (g.K + BK - 1) / BK;
  int split = g.split_k > kblocks ? kblocks : g.split_k;
  int per = (kblocks + split - 1) / split;
  split = (kblocks + per - 1) / per;
  p.split_k = split; p.k_per_split = per * BK;
  p.out = (float*)g.out; p.ldo = g.ldo; p.atomic = g.atomic;
  p.bias = (const float*)g.bias; p.relu = g.relu; p.pad_hp = g.pad_hp; p.pad_wp = g.pad_wp;
  p.relu_aux = (const float*)g.relu_aux; p.ld_aux = g.ld_aux;
  int bm, bn;
  pd_gemm_simt_tile(g.M, g.N, (long long)g.num_z * split, &bm, &bn);
  dim3 grid((g.M + bm - 1) / bm, (g.N + bn - 1) / bn, g.num_z * split);
  PD_REQUIRE(grid.y <= 65535 && grid.z <= 65535, "simt gemm: grid too large");
  if (bm == 128 && bn == 128) gemm_simt_kernel<128, 128, 1><<<grid, kThreads, 0, stream>>>(p);
  else if (bm == 128) gemm_simt_kernel<128, 64, 2><<<grid, kThreads, 0, stream>>>(p);
  else gemm_simt_kernel<64, 64, 4><<<grid, kThreads, 0, stream>>>(p);
  PD_LAUNCH_CHECK("gemm_simt_kernel");
  return PD_OK;
}
